"""Copies of pageable host arrays by several threads, either side of the size from which they are used:
what arrives is what page-locked arrays, which are copied as they are, give, bit for bit."""
import ctypes as C
import threading

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
