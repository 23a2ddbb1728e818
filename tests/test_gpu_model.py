"""Model arrays belong to the caller again once fwi_ctx_set_model returns, page-locked or not, however much
work the context's stream still holds."""
import numpy as np
import pytest
import torch

from fwiedu import engine as E
from fwiedu import models as M

pytestmark = pytest.mark.gpu


def test_page_locked_model_may_change_after_the_call():
    """Behind the zeroing of a 1 GB gather (a few hundred microseconds of stream work), a model in
    page-locked arrays is set and overwritten at once: the run models the one that was set."""
    nz, nx, pml, nt, dt = 40, 60, 8, 61, 0.001
    sv = M.line_survey(nz, nx, 10.0, 10.0, dt, nt, 2, M.ricker(nt, dt, 20.0, 0.02), first_cell=5)
    shots = M.survey_shots(sv)
    shots[1].ns = (1 << 28) // shots[1].ntr
    vp = M.layered_model(nz, nx, seed=5, water_rows=2, n_layers=4)
    rho = M.gardner(vp, 2)
    ctx = E.Context(0)
    try:
        ctx.set_model(vp, rho, 10.0, 10.0, dt, nt, pml, 1)
        ctx.set_shots(shots[:1])
        ctx.run(0)
        want = ctx.traces(0)
        pv, pr = torch.from_numpy(vp.copy()).pin_memory(), torch.from_numpy(rho.copy()).pin_memory()
        ctx.set_shots(shots)  # ends with the large gathers' memsets
        ctx.set_model(pv.numpy(), pr.numpy(), 10.0, 10.0, dt, nt, pml, 1)
        pv.fill_(3000.0)
        pr.fill_(2000.0)
        ctx.run(0)
        assert np.any(want) and np.array_equal(ctx.traces(0), want)
    finally:
        ctx.close()


def test_modelling_after_a_gradient_that_did_not_fit():
    """Under a budget that holds the modelling run's state but not the adjoint source (6000 receivers at
    every step, recorded at every 20th), the gradient is refused part of the way through its allocations;
    the seismograms of the run that follows on the same context are those of a context without a budget."""
    nz, nx, pml, nt, dt = 40, 100, 10, 2001, 0.001
    sv = M.line_survey(nz, nx, 10.0, 10.0, dt, nt, 1, M.ricker(nt, dt, 20.0, 0.06), sample_rate=20, first_cell=30)
    sv.gx[0], sv.gz[0] = np.repeat(sv.gx[0], 60), np.repeat(sv.gz[0], 60)
    shots = M.survey_shots(sv)
    vp = M.layered_model(nz, nx, seed=6, water_rows=4, anom_sigma=2.0)
    rho = M.gardner(vp, 4)
    got = []
    for budget in (0, 40 << 20):
        ctx = E.Context(0, budget)
        try:
            ctx.set_model(vp, rho, 10.0, 10.0, dt, nt, pml, 1)
            ctx.set_shots(shots)
            if budget:
                with pytest.raises(E.FwiError) as e:
                    ctx.run(1, 20.0, 2, 1)
                assert e.value.code == E.FWI_ERR_NOMEM and "budget exceeded" in str(e.value)
            ctx.run(0)
            got.append(ctx.traces(0))
        finally:
            ctx.close()
    assert np.any(got[0]) and np.array_equal(*got)
