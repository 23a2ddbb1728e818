"""Copies of pageable host arrays by several threads, either side of the size from which they are used:
what arrives is what page-locked arrays, which are copied as they are, give, bit for bit."""
import ctypes as C
import threading
import time

import numpy as np
import pytest
import torch

from fwiedu import engine as E
from fwiedu import models as M

pytestmark = pytest.mark.gpu


def _shots(nshot, ntr, ns):
    sv = M.line_survey(61, ntr, 10.0, 10.0, 0.001, ns, nshot, M.ricker(ns, 0.001, 12.0, 0.1), spacing_cells=5,
                       first_cell=20)
    return M.survey_shots(sv)


@pytest.mark.parametrize("nshot,ntr,ns", [(4, 301, 5001), (5, 301, 4201), (7, 401, 4003)])
def test_misfit_and_step_length_of_pageable_gathers(nshot, ntr, ns):
    """24.1, 25.3 and 44.9 MB (the threshold is 24 * 2^20 = 25.2 MB) from four threads at once."""
    L = E.lib()
    L.calculate_objective_value.restype = C.c_float
    L.calculate_step_length.restype = C.c_float
    rng = np.random.default_rng(nshot)
    a = [rng.standard_normal((ntr, ns)).astype(np.float32) for _ in range(nshot)]
    b = [rng.standard_normal((ntr, ns)).astype(np.float32) for _ in range(nshot)]
    shots = _shots(nshot, ntr, ns)

    def run(x, y):
        keep = []
        rx, ry = E.make_records(shots, x, keep), E.make_records(shots, y, keep)
        return L.calculate_objective_value(rx, nshot), L.calculate_step_length(rx, ry, nshot)

    pin = [[torch.from_numpy(v).pin_memory() for v in side] for side in (a, b)]
    want = run(*[[t.numpy() for t in side] for side in pin])
    assert want[0] > 0
    got = [None] * 4

    def work(i):
        got[i] = run(a, b)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [want] * 4


@pytest.mark.parametrize("nshot", [4, 9])
def test_seismograms_into_pageable_gathers(nshot):
    """12.5 and 28.2 MB of seismograms through the drop-in call against one gather at a time."""
    nt = 2601
    shots = _shots(nshot, 301, nt)
    vp = M.layered_model(61, 301, seed=1)
    rho = M.gardner(vp)
    pre, _ = E.propagation(vp, rho, shots, 10.0, 10.0, 0.001, nt, 10, 1, 10.0, 2.0, 0, 0)
    ctx = E.Context(0)
    try:
        ctx.set_model(vp, rho, 10.0, 10.0, 0.001, nt, 10, 1)
        ctx.set_shots(shots)
        ctx.run(0)
        for i in range(nshot):
            want = ctx.traces(i)
            assert np.any(want) and np.array_equal(pre[i], want)
    finally:
        ctx.close()


def _big_gather(nz, nx, nshot, nt=21):
    """A survey whose first shot's record is long enough to be staged (28.8 MB), of a few steps."""
    shots = M.survey_shots(M.line_survey(nz, nx, 10.0, 10.0, 0.001, nt, nshot, M.ricker(nt, 0.001, 60.0, 0.002),
                                         first_cell=30))
    for s in shots:
        s.fpeak = 60.0  # a record of 21 samples has its spectrum's peak at 0 Hz
    shots[0].ns = 7200000 // shots[0].ntr
    vp = M.layered_model(nz, nx, seed=1)
    return shots, vp, M.gardner(vp), nt


def test_one_gather_down_in_pieces():
    """A gather above the threshold into a pageable array is what a page-locked one gets."""
    shots, vp, rho, nt = _big_gather(61, 301, 1)
    ctx = E.Context(0)
    try:
        ctx.set_model(vp, rho, 10.0, 10.0, 0.001, nt, 10, 1)
        ctx.set_shots(shots)
        obs = np.random.default_rng(3).standard_normal((301, shots[0].ns)).astype(np.float32)
        ctx.set_observed([obs])
        ctx.run(2, 30.0, 2, 0)  # the residual fills the record
        want = torch.empty((301, shots[0].ns), pin_memory=True)
        E._check(E.lib().fwi_ctx_get_traces(ctx.h, 0, E._ptr(want.numpy())))
        assert want.numpy().nbytes > 24 << 20
        # bits: what lies beyond the modelled steps is whatever the record's memory held
        assert np.any(want.numpy()) and np.array_equal(ctx.traces(0).view(np.uint32), want.numpy().view(np.uint32))
    finally:
        ctx.close()


def test_a_callers_copy_does_not_wait_for_another_ones_run():
    """Two callers with gathers above the threshold, one of whose streams still holds tens of
    milliseconds of step launches: the other's copy, on an idle stream, ends first."""
    shots, vp, rho, nt = _big_gather(1001, 3001, 60, 81)
    small, vp2, rho2, nt2 = _big_gather(61, 301, 1)
    ex, busy, idle = E.Executor(0), E.Context(0), E.Context(0)
    try:
        idle.set_model(vp2, rho2, 10.0, 10.0, 0.001, nt2, 10, 1)
        idle.set_shots(small)
        idle.run(0)
        idle.traces(0)
        busy.set_model(vp, rho, 10.0, 10.0, 0.001, nt, 20, 1)
        busy.set_shots(shots)
        end = {}

        def fetch(name, ctx):
            ctx.traces(0)
            end[name] = time.perf_counter()

        ex.add(busy, 0)
        assert ex.step(0) == 0  # issued, not finished
        t = threading.Thread(target=fetch, args=("busy", busy))
        t.start()
        time.sleep(0.005)
        fetch("idle", idle)
        t.join()
        assert ex.poll(busy) == (True, 0)
        assert end["idle"] < end["busy"] - 0.005
    finally:
        ex.close()
        busy.close()
        idle.close()
