"""The coefficient set-up on the device (fwi_coef.cuh) against the oracle's, through seismograms that
must be bit for bit its: unequal spacings, thin and thick layers, windows too small for the interior
derivative of 1/rho, several windows and a second model on one context."""
import numpy as np
import pytest

from fwiedu import engine as E
from fwiedu import models as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,pml,fs,dx,dz", [(5, 5, 3, 1, 10.0, 10.0), (6, 11, 1, 0, 10.0, 8.0),
                                                (23, 40, 7, 1, 12.5, 9.0), (48, 37, 20, 0, 7.5, 10.0)])
def test_seismograms_equal_the_oracle(port32, nz, nx, pml, fs, dx, dz):
    nt, dt = 181, 0.0008
    rng = np.random.default_rng(nz)
    sv = M.line_survey(nz, nx, dx, dz, dt, nt, 2, M.ricker(nt, dt, 20.0, 0.05), first_cell=2)
    for k in range(2):
        sv.sx[k] = min(max(sv.sx[k], 2), nx - 3)
        sv.sz[k] = 2 if fs else 3
        # the second shot's window ends before the model does where the model is wide enough
        sv.gx[k] = np.arange(2, nx - 2 if k == 0 or nx < 40 else 6, dtype=np.int32)
        sv.gz[k] = np.full(len(sv.gx[k]), 2, np.int32)
    sv.sx[1] = 3
    shots = M.survey_shots(sv)
    ctx = E.Context(0)
    try:
        for _ in range(2):
            vp = rng.uniform(1500, 4000, (nx, nz)).astype(np.float32)
            rho = rng.uniform(1000, 2500, (nx, nz)).astype(np.float32)
            want = [port32.forward(s, vp, rho, dx, dz, dt, nt, pml, fs) for s in shots]
            ctx.set_model(vp, rho, dx, dz, dt, nt, pml, fs)
            if not ctx.shots:
                ctx.set_shots(shots)
            for path in (E.PATH_BATCHED, E.PATH_PLAIN):
                ctx.run(0, path=path)
                for i, w in enumerate(want):
                    assert np.array_equal(ctx.traces(i), w), (path, i)
    finally:
        ctx.close()


@pytest.mark.parametrize("nshot,nz,nx", [(2, 700, 1500), (1, 900, 1800)])
def test_a_window_holds_one_layout_of_its_planes(nshot, nz, nx):
    """Folded (two shots) or plain (one shot of more than 1.5 million cells): beside the model and the shots'
    scratch frames a window costs six planes (both layouts and the bulk modulus were thirteen).  Three
    more are allowed for gathers, tables and work space."""
    nt, pml = 16, 20
    shots = M.survey_shots(M.line_survey(nz, nx, 10.0, 10.0, 0.001, nt, nshot, M.ricker(nt, 0.001, 60.0, 0.002),
                                         first_cell=30))
    vp = M.layered_model(nz, nx, seed=2)
    ctx = E.Context(0)
    try:
        ctx.set_model(vp, M.gardner(vp), 10.0, 10.0, 0.001, nt, pml, 1)
        ctx.set_shots(shots)
        ctx.run(0)
        plane = 4 * (nx + 2 * pml + 12) * (nz + 2 * pml)  # folded: up to 12 columns wider
        frames = 4 * nshot
        held = ctx.stats()["device_bytes"]
        assert held <= 32 * nz * nx + (6 + frames + 3) * plane
    finally:
        ctx.close()
