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
