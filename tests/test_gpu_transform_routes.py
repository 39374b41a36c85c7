"""field::ift / field::dft: the route that reads and writes the caller's device
arrays in place of copies, against the copying route (arrays off a 16-byte
boundary, host arrays) and against numpy."""
import numpy as np
import pytest

from oracle import nsve as O
from bfps_b200 import _lib

pytestmark = pytest.mark.gpu


def _off(count, real, shift):
    """`count` values of device memory starting `shift` values past a 256-byte boundary, NaN all over."""
    import torch
    return torch.full((count + shift,), float("nan"), dtype=real, device="cuda")[shift:]


def _put(values, real, shift):
    import torch
    flat = np.ascontiguousarray(values).view(values.real.dtype).reshape(-1)
    a = _off(flat.size, real, shift)
    a.copy_(torch.from_numpy(flat))
    return a


@pytest.mark.parametrize("n,precision", [(16, "single"), (32, "single"), (64, "single"), (128, "single"),
                                         (256, "single"), (512, "single"), (16, "double"), (64, "double"),
                                         (128, "double")])
def test_direct_route_matches_copies_and_numpy(n, precision):
    import torch
    from bfps_b200.solver import vorticity_equation
    ve = vorticity_equation(n, precision=precision)
    L = _lib.lib()
    rng = np.random.default_rng(n)
    real = torch.float32 if precision == "single" else torch.float64
    shift = 2 if precision == "single" else 1  # 8 bytes: not on a 16-byte boundary
    r = rng.standard_normal(ve.rshape).astype(ve.rdtype)  # garbage in the padding too
    out = []
    for s in (0, shift):
        din = _put(r, real, s)
        dout = _off(2 * int(np.prod(ve.cshape)), real, s)
        _lib.check(L.bfg_dft(ve.handle, din.data_ptr(), dout.data_ptr()), ve.handle)
        d = dout.cpu().numpy().view(ve.cdtype).reshape(ve.cshape)
        cin = _put(d, real, s)
        back = _off(r.size, real, s)
        _lib.check(L.bfg_ift(ve.handle, cin.data_ptr(), back.data_ptr()), ve.handle)
        out.append((d, back.cpu().numpy().reshape(ve.rshape)))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert np.all(out[0][1][:, :, n:] == 0)
    tol = 1e-13 if precision == "double" else 2e-6
    got = out[0][1][:, :, :n] / n ** 3
    assert np.abs(got - r[:, :, :n]).max() <= tol * np.abs(r).max()
    if n <= 128:
        want = O.dft(r[:, :, :n].astype(np.float64))
        assert np.abs(out[0][0] - want).max() <= tol * np.abs(want).max()
    ve.close()


@pytest.mark.parametrize("n,precision", [(32, "double"), (64, "single"), (512, "single")])
def test_in_place(n, precision):
    """in may equal out, as in the reference's in-place transforms."""
    import torch
    from bfps_b200.solver import vorticity_equation
    ve = vorticity_equation(n, precision=precision)
    L = _lib.lib()
    a = torch.randn(*ve.rshape, dtype=torch.float32 if precision == "single" else torch.float64, device="cuda")
    keep = a[:, :, :n].clone()
    other = torch.empty_like(a)
    _lib.check(L.bfg_dft(ve.handle, a.data_ptr(), other.data_ptr()), ve.handle)
    _lib.check(L.bfg_dft(ve.handle, a.data_ptr(), a.data_ptr()), ve.handle)
    assert torch.equal(a, other)
    _lib.check(L.bfg_ift(ve.handle, a.data_ptr(), a.data_ptr()), ve.handle)
    tol = 1e-13 if precision == "double" else 2e-6
    assert float((a[:, :, :n] / n ** 3 - keep).abs().max()) <= tol * float(keep.abs().max())
    ve.close()


def test_context_fields_survive():
    """The direct route leaves the state and the real velocity alone."""
    import torch
    from bfps_b200 import ic
    from bfps_b200.solver import vorticity_equation
    n = 64
    ve = vorticity_equation(n, precision="single")
    ve.set_cvorticity(ic.vorticity_ic(n, seed=3, dtype=np.complex64))
    ve.velocity_rspace()
    u, w = ve.get_rvelocity(), ve.get_cvorticity()
    a = torch.randn(*ve.rshape, dtype=torch.float32, device="cuda")
    _lib.check(_lib.lib().bfg_dft(ve.handle, a.data_ptr(), a.data_ptr()), ve.handle)
    _lib.check(_lib.lib().bfg_ift(ve.handle, a.data_ptr(), a.data_ptr()), ve.handle)
    assert np.array_equal(ve.get_rvelocity(), u) and np.array_equal(ve.get_cvorticity(), w)
    ve.close()
