"""The wavenumber filter's transforms at the lengths where their passes change: convolution sizes of
every leading radix and of the FP32 ones, odd and even padded sizes, odd and single columns, against
numpy's FFT in FP64.  The filtered field is float, formed from FP64 transforms whose intermediate
spectra are float: 1e-6 of its norm is asked (the reference's own FFT is FP32, 1e-5), 1e-5 where the
transforms are FP32 (more than 4096 padded samples)."""
import ctypes as C

import numpy as np
import pytest

from fwiedu import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,cells", [(1, 1, 1), (3, 1, 1), (2, 5, 1), (9, 6, 2), (31, 40, 5), (64, 33, 8),
                                         (40, 75, 20), (90, 41, 45), (30, 120, 100), (21, 37, 240)])
def test_lowpass2d_lengths(nz, nx, cells):
    """A pass wavenumber of 4 / `cells` per cell: a taper of `cells` samples and ten times that padding."""
    rng = np.random.default_rng(nz * nx)
    d = 10.0
    kpass = 4.0 / (cells * d)
    kcut = 2 * kpass
    s = rng.standard_normal((nx, nz)).astype(np.float32)
    y = np.zeros_like(s)
    E.lib().lowpass2d(E.rows(s), nz, nx, C.c_float(d), C.c_float(d), C.c_float(kpass), C.c_float(kcut), E.rows(y))
    pad = 10 * int(np.floor(4 / (np.float32(kpass) * d) + 0.5))
    f = np.pad(s.astype(np.float64), pad, mode="edge")  # s holds the tapered field now
    k = np.hypot(np.fft.fftfreq(f.shape[0], d)[:, None], np.fft.fftfreq(f.shape[1], d)[None, :])
    w = np.where(k < kpass, 1.0, np.where(k <= kcut, 0.5 * (1 + np.cos(np.pi * (k - kpass) / (kcut - kpass))), 0.0))
    want = np.fft.ifft2(np.fft.fft2(f) * w).real[pad:pad + nx, pad:pad + nz]
    tol = 1e-6 if max(f.shape) <= 4096 else 1e-5
    assert np.linalg.norm(y - want) <= tol * np.linalg.norm(want) + 1e-30


@pytest.mark.parametrize("nx", [4101, 4981, 5991])
def test_lowpass2d_rounding_of_fp32_transforms(nx):
    """Padded lengths of 4121, 5001 and 6011 (transforms of 16384 points kept in FP32) under a window that is
    one everywhere: the filter returns its input, up to the rounding of a transform and its inverse.  The
    transforms restated wholly in FP32, without fused operations and with every twiddle factor read from the
    table are off by 2.5e-7, 2.6e-7 and 2.8e-7 of the norm (twice as much with the factors' powers formed by
    multiplication), the float spectra between the stages by 3e-8 each: 3e-7 is asked."""
    nz, d = 12, 10.0
    s = np.random.default_rng(nx).standard_normal((nx, nz)).astype(np.float32)
    y = np.zeros_like(s)
    E.lib().lowpass2d(E.rows(s), nz, nx, C.c_float(d), C.c_float(d), C.c_float(4 / d), C.c_float(8 / d), E.rows(y))
    # s holds the tapered field now
    assert np.linalg.norm(y.astype(np.float64) - s) <= 3e-7 * np.linalg.norm(s.astype(np.float64))
