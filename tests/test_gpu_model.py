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
