"""The step kernel on folded fields (the default) against the tile kernel on plain ones.

A folded field pairs column x with column x + W and continues each half across the seam by three
copied columns.  Windows whose half-width, rows and absorbing layer are odd or barely larger than a
tile, sources and receivers in the seam's columns, at depth and several to a column, with and
without the free surface, one shot and several: seismograms, adjoint sources and gradients must be
the tile kernel's bit for bit (FWI_TX pins that kernel)."""
import dataclasses
import os

import numpy as np
import pytest

from fwiedu import engine as E
from fwiedu import models as M

pytestmark = pytest.mark.gpu

CASES = [  # nz, nx, pml, fs, nshot, receiver rows, precondition, path
    (31, 37, 10, 1, 3, (1,), 1, E.PATH_BATCHED),
    (45, 50, 7, 1, 2, (2, 9), 1, E.PATH_BATCHED),     # odd layer: the surface row is odd
    (40, 43, 3, 1, 4, (0,), 1, E.PATH_BATCHED),       # thinnest layer, receivers on the surface row
    (52, 61, 5, 0, 5, (3, 30), 0, E.PATH_BATCHED),    # no free surface, receivers at depth
    (12, 12, 4, 0, 2, (2,), 1, E.PATH_BATCHED),       # narrower than a tile
    (130, 95, 20, 1, 25, (1,), 1, E.PATH_BATCHED),    # several tiles of rows and chunks of shots
    (33, 64, 9, 1, 1, (1,), 1, E.PATH_BATCHED),
    (47, 58, 8, 1, 2, (1, 1), 1, E.PATH_PLAIN),       # two receivers in one cell, one shot per launch
]


def _run(case, pin, obs=None):
    nz, nx, pml, fs, nshot, rows, pre, path = case
    old = {k: os.environ.pop(k, None) for k in ("FWI_TX", "FWI_DEPTH")}
    if pin:
        os.environ.update(FWI_TX="16", FWI_DEPTH="1")
    try:
        water = 4
        vp = M.layered_model(nz, nx, seed=nz, water_rows=water, n_layers=4, anom_sigma=2.0)
        if obs is not None:
            vp = M.smooth_model(vp, 2.0, water_rows=water)
        rho = M.gardner(vp, water)
        nt, dt = 260, 0.001
        sv = M.line_survey(nz, nx, 10.0, 10.0, dt, nt, nshot, M.ricker(nt, dt, 18.0, 0.05))
        W = (nx + 2 * pml + 1) // 2
        seam = [x for x in range(W - 3 - pml, W + 4 - pml) if 0 <= x < nx]
        for k in range(nshot):  # sources in the seam's columns, one of them at depth
            sv.sx[k] = seam[k % len(seam)] if k % 2 == 0 else sv.sx[k]
            sv.sx[k] = min(max(sv.sx[k], 3), nx - 4)
            sv.sz[k] = nz // 2 if k == 2 else 2
            sv.gx[k] = np.concatenate([np.arange(3, nx - 3, dtype=np.int32) for _ in rows])
            sv.gz[k] = np.concatenate([np.full(nx - 6, r, np.int32) for r in rows])
            if not fs:
                sv.gz[k] = np.maximum(sv.gz[k], 3).astype(np.int32)
        shots = M.survey_shots(sv)
        ctx = E.Context(0)
        try:
            ctx.set_model(vp, rho, 10.0, 10.0, dt, nt, pml, fs)
            ctx.set_shots(shots)
            if obs is None:
                ctx.run(0, path=path)
                return [ctx.traces(i) for i in range(nshot)], None
            ctx.set_observed(obs)
            ctx.run(1, 12.0, 2, pre, path)
            return [ctx.traces(i) for i in range(nshot)], ctx.gradient()
        finally:
            ctx.close()
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}-pml{c[2]}-fs{c[3]}-{c[4]}")
def test_folded_fields_match_plain_fields(case):
    want, _ = _run(case, True)
    got, _ = _run(case, False)
    assert case[5] == (0,) or max(np.abs(t).max() for t in want) > 0  # the surface row records zeros
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    wadj, wgrad = _run(case, True, want)
    adj, grad = _run(case, False, want)
    assert all(np.array_equal(a, b) for a, b in zip(adj, wadj))
    assert np.array_equal(grad, wgrad, equal_nan=True)


@pytest.mark.parametrize("nshot,step,sr", [(4, 17, 1), (5, 0, 3), (50, 2, 1)], ids=["windows", "rates", "tables"])
def test_groups_in_one_launch_match_one_after_another(nshot, step, sr):
    """A moving spread (windows of their own, overlapping), one window recorded at two sample rates
    and more windows than one launch's table holds: the groups advance together, and every result
    equals the tile kernel's, which takes them one after another."""
    nz, nx, pml, nt, dt = 40, 170, 8, 151, 0.001
    old = {k: os.environ.pop(k, None) for k in ("FWI_TX", "FWI_DEPTH")}
    try:
        vp = M.layered_model(nz, nx, seed=3, water_rows=4, n_layers=4, anom_sigma=2.0)
        vp0 = M.smooth_model(vp, 2.0, water_rows=4)
        shots = []
        for k in range(nshot):
            rate = sr if k % 2 else 1
            sv = M.line_survey(nz, nx, 10.0, 10.0, dt, nt, 1, M.ricker(nt, dt, 18.0, 0.04), sample_rate=rate)
            sv.sx[0] = 40 + step * k
            sv.gx[0] = np.arange(sv.sx[0] - 7, sv.sx[0] + 8, dtype=np.int32)
            sv.gz[0] = np.full(15, 1, np.int32)
            shots += M.survey_shots(sv)

        def run(pin):
            for k in ("FWI_TX", "FWI_DEPTH"):
                os.environ.pop(k, None)
            if pin:
                os.environ.update(FWI_TX="16", FWI_DEPTH="1")
            ctx = E.Context(0)
            try:
                ctx.set_model(vp, M.gardner(vp, 4), 10.0, 10.0, dt, nt, pml, 1)
                ctx.set_shots(shots)
                ctx.run(0)
                obs = [ctx.traces(i) for i in range(nshot)]
                ctx.set_model(vp0, M.gardner(vp0, 4), 10.0, 10.0, dt, nt, pml, 1)
                ctx.set_observed(obs)
                ctx.run(1, 12.0, 2, 1)
                adj, grad = [ctx.traces(i) for i in range(nshot)], ctx.gradient()
                ctx.run(2, 12.0, 0, 1)
                return obs, adj, grad, [ctx.traces(i) for i in range(nshot)], ctx.pass_stats()["fwd_launches"]
            finally:
                ctx.close()

        want, got = run(True), run(False)
        for a, b in zip(got[:2] + got[3:4], want[:2] + want[3:4]):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))
        assert np.array_equal(got[2], want[2])
        assert got[4] == nt * (2 if nshot > 45 else 1)  # the groups shared their launches
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


def test_sample_rates_of_one_window_share_launches():
    """Shots of one window at three sample rates advance in the same launches, several to a block, each
    sampled at its own steps; a window that fills the GPU by itself is not split by rate either."""
    old = {k: os.environ.pop(k, None) for k in ("FWI_TX", "FWI_DEPTH", "FWI_CHUNK")}
    try:
        def run(nz, nx, nt, rates, pin):
            for k in ("FWI_TX", "FWI_DEPTH", "FWI_CHUNK"):
                os.environ.pop(k, None)
            os.environ.update({"FWI_TX": "16", "FWI_DEPTH": "1"} if pin else {"FWI_CHUNK": "4"})
            vp = M.layered_model(nz, nx, seed=9, water_rows=4, n_layers=4, anom_sigma=2.0)
            shots = []
            for k, r in enumerate(rates):
                sv = M.line_survey(nz, nx, 10.0, 10.0, 0.001, nt, 1, M.ricker(nt, 0.001, 30.0, 0.002), sample_rate=r)
                sv.sx[0] = 8 + 5 * k
                shots += M.survey_shots(sv)
                shots[-1].fpeak = 30.0  # a record of 13 samples has its spectrum's peak at 0 Hz
            ctx = E.Context(0)
            try:
                ctx.set_model(vp, M.gardner(vp, 4), 10.0, 10.0, 0.001, nt, 10, 1)
                ctx.set_shots(shots)
                ctx.run(0)
                return [ctx.traces(i) for i in range(len(shots))], ctx.pass_stats()["fwd_launches"]
            finally:
                ctx.close()

        for nz, nx, nt, rates in ((40, 60, 121, (2, 6, 4, 2, 1, 3, 6)), (1000, 3200, 13, (2, 1, 3))):
            want, _ = run(nz, nx, nt, rates, True)
            got, launches = run(nz, nx, nt, rates, False)
            assert launches == nt
            assert all(np.any(w) and np.array_equal(a, w) for a, w in zip(got, want))
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


@pytest.mark.parametrize("half,per,together", [(60, 1, True), (60, 4, True), (450, 1, False), (500, 3, False)])
def test_windows_share_launches_only_where_they_are_small(half, per, together):
    """Four windows of 130 or of 600 thousand and more cells, one or several shots each: small ones advance in
    the same launches, large ones in launches of their own; the seismograms are the tile kernel's."""
    nz, nt, ng, pml = 560, 9, 4, 20
    nx = 2 * half + 61 + 10 * ng
    old = {k: os.environ.pop(k, None) for k in ("FWI_TX", "FWI_DEPTH")}
    try:
        vp = M.layered_model(nz, nx, seed=2, water_rows=4, n_layers=4, anom_sigma=2.0)
        sv = M.line_survey(nz, nx, 10.0, 10.0, 0.001, nt, ng * per, M.ricker(nt, 0.001, 60.0, 0.002))
        for k in range(ng * per):
            mid = half + 31 + 10 * (k // per)
            sv.sx[k] = mid + k % per
            sv.gx[k] = np.arange(mid - half, mid + half, dtype=np.int32)
            sv.gz[k] = np.full(2 * half, 1, np.int32)
        shots = M.survey_shots(sv)
        for s in shots:
            s.fpeak = 60.0  # a record of 9 samples has its spectrum's peak at 0 Hz
        out = []
        for pin in (True, False):
            os.environ.update({"FWI_TX": "16", "FWI_DEPTH": "1"} if pin else {})
            ctx = E.Context(0)
            try:
                ctx.set_model(vp, M.gardner(vp, 4), 10.0, 10.0, 0.001, nt, pml, 1)
                ctx.set_shots(shots)
                ctx.run(0)
                out.append([ctx.traces(i) for i in range(ng * per)])
                launches = ctx.pass_stats()["fwd_launches"]
            finally:
                ctx.close()
            for k in ("FWI_TX", "FWI_DEPTH"):
                os.environ.pop(k, None)
        assert launches == nt * (1 if together else ng)
        assert all(np.any(w) and np.array_equal(a, w) for w, a in zip(*out))
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


@pytest.mark.parametrize("nz,nx,tile", [(60, 600, 8), (300, 900, 16), (1000, 3200, 8)])
def test_one_shot_launches_fold_windows_of_middle_size(nz, nx, tile):
    """One shot a launch on the plain path: windows of 50 thousand and 3 million cells take the kernel on
    plain fields (whose untuned tiles are 8 columns wide there), one of 0.3 million folded fields (always
    reported as 16).
    Alone, on either path, and two in one launch, on folded fields, a shot's seismogram is the same."""
    nt = 13
    old = {k: os.environ.pop(k, None) for k in ("FWI_TX", "FWI_DEPTH")}
    try:
        vp = M.layered_model(nz, nx, seed=4, water_rows=4, n_layers=4, anom_sigma=2.0)
        shots = M.survey_shots(M.line_survey(nz, nx, 10.0, 10.0, 0.001, nt, 2, M.ricker(nt, 0.001, 60.0, 0.002),
                                             first_cell=30))
        for s in shots:
            s.fpeak = 60.0  # a record of 13 samples has its spectrum's peak at 0 Hz
        ctx = E.Context(0)
        try:
            E.lib().fwi_ctx_set_autotune(ctx.h, 0)
            ctx.set_model(vp, M.gardner(vp, 4), 10.0, 10.0, 0.001, nt, 10, 1)
            ctx.set_shots(shots)
            ctx.run(0)
            want = [ctx.traces(i) for i in range(2)]
            ctx.run(0, path=E.PATH_PLAIN)
            assert ctx.launch_shape()["tile_columns"] == tile
            assert all(np.any(w) and np.array_equal(ctx.traces(i), w) for i, w in enumerate(want))
            ctx.set_shots(shots[1:])
            ctx.run(0)
            assert np.array_equal(ctx.traces(0), want[1])
        finally:
            ctx.close()
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


@pytest.mark.parametrize("limit_ms", [1, 20, 200])
def test_a_warps_bounded_wait_ends_alike_for_its_lanes(limit_ms):
    """Lanes whose time runs out before and after the phase completes all give up (FWI_ERR_STATE if not)."""
    ctx = E.Context(0)
    try:
        assert E.lib().fwi_ctx_selftest_wait(ctx.h, limit_ms) == E.FWI_ERR_CUDA
        assert b"did not complete" in E.lib().fwi_last_error()
    finally:
        ctx.close()


def test_more_shots_than_a_grid_has_rows():
    """33000 shots in each of two windows, more together than a grid dimension's 65535: the first and the
    last of either window record what they record alone."""
    nz, nx, pml, nt, per = 10, 30, 3, 8, 33000
    vp = M.layered_model(nz, nx, seed=1, water_rows=2, n_layers=2, anom_sigma=1.0)
    rho = M.gardner(vp, 2)
    sv = M.line_survey(nz, nx, 10.0, 10.0, 0.001, nt, 1, M.ricker(nt, 0.001, 80.0, 0.001))
    one = M.survey_shots(sv)[0]
    shots = []
    for lo in (0, 15):
        for k in range(per):
            s = dataclasses.replace(one, isx=3 + k % 7, igx=np.arange(3, 11, dtype=np.int32), igz=np.ones(8, np.int32),
                                    ix_min=lo, ix_max=lo + 14, fpeak=80.0)
            shots.append(s)
    ctx = E.Context(0)
    try:
        ctx.set_model(vp, rho, 10.0, 10.0, 0.001, nt, pml, 1)
        picks = [0, per - 1, per, 2 * per - 1]
        want = []
        for i in picks:
            ctx.set_shots([shots[i]])
            ctx.run(0)
            want.append(ctx.traces(0))
        ctx.set_shots(shots)
        ctx.run(0)
        for i, w in zip(picks, want):
            assert np.any(w) and np.array_equal(ctx.traces(i), w), i
    finally:
        ctx.close()


@pytest.mark.parametrize("nshot", [1, 3])
def test_paths_in_turn_on_one_context(nshot):
    """The batched path folds this window, the plain path does not: gradients and seismograms of runs that
    change layout on one context, a new model in between, are those of a context per run."""
    nz, nx, pml, nt, dt = 50, 90, 10, 121, 0.001
    shots = M.survey_shots(M.line_survey(nz, nx, 10.0, 10.0, dt, nt, nshot, M.ricker(nt, dt, 25.0, 0.04), first_cell=20))
    rng = np.random.default_rng(nshot)
    obs = [rng.standard_normal((len(s.igx), s.ns)).astype(np.float32) for s in shots]
    models = [M.layered_model(nz, nx, seed=k, water_rows=4, n_layers=4, anom_sigma=2.0) for k in (1, 2)]

    def run(ctx, vp, path):
        ctx.set_model(vp, M.gardner(vp, 4), 10.0, 10.0, dt, nt, pml, 1)
        if not ctx.shots:
            ctx.set_shots(shots)
        ctx.set_observed(obs)
        ctx.run(0, path=path)
        out = [ctx.traces(i) for i in range(nshot)]
        ctx.run(1, 20.0, 2, 1, path)
        return out + [ctx.traces(i) for i in range(nshot)] + [ctx.gradient()]

    steps = [(models[0], E.PATH_BATCHED), (models[0], E.PATH_PLAIN), (models[1], E.PATH_BATCHED),
             (models[1], E.PATH_PLAIN), (models[0], E.PATH_BATCHED)]
    one = E.Context(0)
    try:
        for vp, path in steps:
            got = run(one, vp, path)
            ctx = E.Context(0)
            try:
                want = run(ctx, vp, path)
            finally:
                ctx.close()
            assert all(np.any(w) and np.array_equal(a, w) for a, w in zip(got, want)), path
    finally:
        one.close()
