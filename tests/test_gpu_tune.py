"""The autotuner's probes on records shorter than their usual number of launches: runs of one context with
several numbers of shots, launched directly and from graphs, ask for probe programs of different lengths
from the same few steps.  Gradients must be those of the untuned launches bit for bit."""
import numpy as np
import pytest

from fwiedu import engine as E
from fwiedu import models as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [13, 14, 17, 25])
def test_probes_of_short_records(nt):
    nz, nx, pml, dt = 21 + nt, 47, 9, 0.001  # a grid of its own per record length: each is tuned anew
    vp = M.layered_model(nz, nx, seed=nt, water_rows=4, n_layers=3, anom_sigma=2.0)
    rho = M.gardner(vp, 4)
    sv = M.line_survey(nz, nx, 10.0, 10.0, dt, nt, 3, M.ricker(nt, dt, 80.0, 0.004), first_cell=6)
    shots = M.survey_shots(sv)
    rng = np.random.default_rng(nt)
    obs = [rng.standard_normal((len(s.igx), s.ns)).astype(np.float32) for s in shots]

    def run(tune):
        out = []
        ctx = E.Context(0)
        try:
            E.lib().fwi_ctx_set_autotune(ctx.h, int(tune))
            ctx.set_model(vp, rho, 10.0, 10.0, dt, nt, pml, 1)
            for nshot, graphs in ((3, 0), (2, 1), (1, 1)):
                E.lib().fwi_ctx_set_graphs(ctx.h, graphs)
                ctx.set_shots(shots[:nshot])
                ctx.set_observed(obs[:nshot])
                ctx.run(1, 20.0, 2, 1)
                out += [ctx.traces(i) for i in range(nshot)] + [ctx.gradient()]
            return out
        finally:
            ctx.close()

    want, got = run(False), run(True)
    assert all(np.isfinite(w).all() and np.any(w) for w in want)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("nt", [1, 2, 3])
@pytest.mark.parametrize("path", [E.PATH_PLAIN, E.PATH_BATCHED])
def test_records_of_one_to_three_samples(port32, nt, path):
    """Probes stay within the record: seismograms of the smallest records are the oracle's."""
    nz, nx, pml, dt = 19, 33 + nt, 6, 0.001
    vp = M.layered_model(nz, nx, seed=nt, water_rows=3, n_layers=3, anom_sigma=2.0)
    rho = M.gardner(vp, 3)
    src = np.linspace(1.0, 2.0, nt).astype(np.float32)
    shots = M.survey_shots(M.line_survey(nz, nx, 10.0, 10.0, dt, nt, 2, src, first_cell=5))
    for s in shots:
        s.fpeak = 30.0
    ctx = E.Context(0)
    try:
        ctx.set_model(vp, rho, 10.0, 10.0, dt, nt, pml, 1)
        ctx.set_shots(shots)
        for _ in range(2):
            ctx.run(0, path=path)
            for i, s in enumerate(shots):
                assert np.array_equal(ctx.traces(i), port32.forward(s, vp, rho, 10.0, 10.0, dt, nt, pml, 1))
    finally:
        ctx.close()
