"""Statistics kernels at the edges of their work split: fewer points than one
block, sizes around the blocks' strides, values on bin edges and outside the
histogram, NaN and infinities, rows outside kM."""
import math

import numpy as np
import pytest

from oracle import nsve as O
from bfps_b200 import _lib, ic
from gpu_util import rel_err

pytestmark = pytest.mark.gpu


def _noalloc(r, me, nbins):
    import torch
    nz, ny, nx, _ = r.shape
    pad = np.full((nz, ny, 2 * (nx // 2 + 1), 3), np.nan, r.dtype)
    pad[:, :, :nx] = r
    f = torch.from_numpy(pad).cuda()
    mom = torch.zeros(40, dtype=torch.float64, device="cuda")
    hist = torch.zeros(nbins * 4, dtype=torch.int64, device="cuda")
    rc = _lib.lib().bfg_rspace_stats_noalloc(f.data_ptr(), nx, ny, nz, r.itemsize, me, nbins,
                                             mom.data_ptr(), hist.data_ptr(), None)
    assert rc == _lib.BFG_OK
    torch.cuda.synchronize()
    return mom.cpu().numpy().reshape(10, 4), hist.cpu().numpy().reshape(nbins, 4)


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 255), (3, 7, 37), (8, 37, 256), (5, 151, 101),
                                   (2, 74, 1025)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_moments_and_histogram_sizes(shape, dtype):
    r = np.random.default_rng(sum(shape)).standard_normal(shape + (3,)).astype(dtype)
    me, nbins = 2.0, 37
    mom, hist = _noalloc(r, me, nbins)
    wm, wh = O.rspace_stats(r.astype(np.float64), [me] * 3 + [me * math.sqrt(3)], nbins)
    # sums of at most 2e5 terms in FP64
    assert np.abs(mom - wm).max() <= 1e-12 * np.abs(wm).max()
    assert np.array_equal(hist, wh)


def test_values_on_and_outside_the_bins():
    """Multiples of the bin size (quotients that are whole numbers), values at
    and beyond the estimate, exact zeros: the same bins as the division."""
    me, nbins = 3.0, 30
    step = 2 * me / nbins
    vals = np.concatenate([np.arange(-nbins, nbins + 1) * step / 2, [me, -me, 1e9, -1e9, 1e300, 0.0],
                           np.nextafter(np.arange(-15, 16) * step, 10),
                           np.nextafter(np.arange(-15, 16) * step, -10)])
    r = np.stack([vals, vals[::-1], np.roll(vals, 7)], -1)[None, None]
    _, hist = _noalloc(r, me, nbins)
    with np.errstate(over="ignore", invalid="ignore"):
        want = np.zeros((nbins, 4), np.int64)
        mag = np.sqrt((r[..., 0] ** 2 + r[..., 1] ** 2) + r[..., 2] ** 2).ravel()
        for i in range(4):
            m = me * math.sqrt(3) if i == 3 else me
            q = mag * 2 / (2 * m / nbins) if i == 3 else (r[..., i].ravel() + m) / (2 * m / nbins)
            b = np.floor(q)
            b = b[(b >= 0) & (b < nbins)].astype(int)
            want[:, i] = np.bincount(b, minlength=nbins)
    assert np.array_equal(hist[:, :3], want[:, :3])
    # the magnitude's sum of squares may be fused: one count per edge value
    assert np.abs(hist[:, 3] - want[:, 3]).sum() <= 4


def test_nonfinite_values():
    """Infinities and NaN lie outside the histogram; infinities set the
    extrema, a NaN leaves them alone."""
    r = np.zeros((1, 1, 4, 3))
    r[0, 0, 1] = [np.inf, -np.inf, np.nan]
    r[0, 0, 2] = [1.0, -2.0, 0.5]
    mom, hist = _noalloc(r, 4.0, 8)
    assert np.isposinf(mom[9, 0]) and np.isneginf(mom[0, 1])
    assert mom[0, 2] == 0.0 and mom[9, 2] == 0.5
    assert hist[:, 0].sum() == 3 and hist[:, 1].sum() == 3
    assert hist[:, 2].sum() == 3 and hist[:, 3].sum() == 3


@pytest.mark.parametrize("n", [16, 64])
@pytest.mark.parametrize("dk", [(1.0, 1.0, 1.0), (0.7, 1.3, 1.0)])
def test_cospectrum_of_any_field(n, dk):
    """Every row (+-ky, +-kz), the zero and Nyquist lines included, for a field
    that fills the whole grid of modes and is not Hermitian."""
    from bfps_b200.solver import vorticity_equation
    import ctypes
    ve = vorticity_equation(n, n, n, *dk, precision="double")
    rng = np.random.default_rng(n)
    a = rng.standard_normal(ve.cshape) + 1j * rng.standard_normal(ve.cshape)
    kk = O.KSpace(n, n, n, *dk, O.SMOOTH)
    spec = np.zeros((kk.nshells, 3, 3))
    _lib.check(_lib.lib().bfg_field_stats(ve.handle, a.ctypes.data_as(ctypes.c_void_p), 1.0, 16,
                                          _lib.ptr(spec), None, None), ve.handle)
    assert rel_err(spec, kk.cospectrum(a, a)) < 1e-13
    assert np.array_equal(spec, spec.transpose(0, 2, 1))
    ve.close()
