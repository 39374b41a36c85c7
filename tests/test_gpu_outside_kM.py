"""The passes of a step leave out the modes outside kM (from 128^3 up): states
that are zero there and states that are not, both dealiasing rules, boxes with
unequal wavenumber spacings, stale values in every work buffer, ensembles of
unequal members."""
import ctypes

import numpy as np
import pytest

from oracle import nsve as O
from bfps_b200 import _lib, ic
from gpu_util import rel_err

pytestmark = pytest.mark.gpu

N = 128


def _field(seed, dk, dealias, full):
    """A random Hermitian field; zero outside kM unless `full`."""
    rng = np.random.default_rng(seed)
    w = O.dft(rng.standard_normal((N, N, N, 3))) / N ** 1.5
    kk = O.KSpace(N, N, N, *dk, dealias)
    w = w / (1.0 + kk.K2[..., None])
    if not full:
        w[kk.K2 >= kk.kM2] = 0
    return O.symmetrize(w)


def _solver(dk, dealias, precision="double"):
    from bfps_b200.solver import vorticity_equation
    ve = vorticity_equation(N, N, N, *dk, precision=precision, dealias_type=dealias)
    ref = O.VorticityEquation(N, N, N, *dk, dealias_type=dealias, workers=8)
    for o in (ve, ref):
        o.nu, o.forcing_type, o.famplitude, o.fk0, o.fk1 = 0.02, "linear", 0.5, 1.5, 3.0
    return ve, ref


def _poison(ve):
    """Large values without a pattern in the work buffers and both RK buffers.
    The statistics of white noise leave its modes in v1, its real values over all
    but the last N^2 * 8 / (N + 8) rows of v2 and its half-transformed ones in wb;
    the upload of the velocity then fills wa (and stages through wb)."""
    L = _lib.lib()
    rng = np.random.default_rng(77)
    big = np.empty(ve.cshape, ve.cdtype)
    big.real = 1e6 * rng.standard_normal(ve.cshape, dtype=np.float32)
    big.imag = 1e6 * rng.standard_normal(ve.cshape, dtype=np.float32)
    spec = np.zeros((ve.kspace()["nshells"], 3, 3))
    _lib.check(L.bfg_field_stats(ve.handle, big.ctypes.data_as(ctypes.c_void_p), 1.0, 16, _lib.ptr(spec),
                                 None, None), ve.handle)
    _lib.check(L.bfg_field_upload(ve.handle, _lib.FIELD_VELOCITY, big.ctypes.data), ve.handle)


@pytest.mark.parametrize("dealias", [O.SMOOTH, O.TWO_THIRDS])
@pytest.mark.parametrize("dk", [(1.0, 1.0, 1.0), (1.0, 0.5, 2.0), (0.7, 1.3, 1.0)])
@pytest.mark.parametrize("full", [False, True])
def test_step_matches_oracle(dealias, dk, full):
    ve, ref = _solver(dk, dealias)
    w0 = _field(3, dk, dealias, full)
    ve.set_cvorticity(w0)
    ref.cvorticity = w0.copy()
    for s in range(2):
        _poison(ve)
        ve.step(1e-3)
        ref.step(1e-3)
        got = ve.get_cvorticity()
        assert rel_err(got, ref.cvorticity) < 1e-12, s
        # outside kM: exactly what the state held, or zero
        out = ref.kk.K2 > ref.kk.kM2
        assert (np.abs(got[out]).max() > 0) == full
    st, want = ve.do_stats(2.0, 5.0, 32), O.nsve_do_stats(ref, 2.0, 5.0, 32)
    for name in ("velocity", "vorticity"):
        assert rel_err(st[name][0], want[name][0]) < 1e-12
        assert rel_err(st[name][1], want[name][1]) < 1e-10
    ve.velocity_rspace()
    ur = ref.ift(ref.compute_velocity(ref.cvorticity))
    assert rel_err(ve.get_rvelocity()[:, :, :N], ur) < 1e-12
    ve.close()


@pytest.mark.parametrize("dealias", [O.SMOOTH, O.TWO_THIRDS])
def test_single_precision_and_replaced_states(dealias):
    """Full state, then a zero-outside one, a checkpoint read of the full one
    and a reset on one FP32 context."""
    dk = (1.0, 1.0, 1.0)
    ve, ref = _solver(dk, dealias, "single")
    for full, read in ((True, False), (False, False), (True, True)):
        w0 = _field(11, dk, dealias, full).astype(np.complex64)
        _poison(ve)
        if read:
            ve.io_checkpoint_read(w0)
            ref.cvorticity = ref.read_checkpoint_semantics(w0.astype(np.complex128))
        else:
            ve.set_cvorticity(w0)
            ref.cvorticity = w0.astype(np.complex128)
        ve.step(1e-3, 2)
        ref.step(1e-3)
        ref.step(1e-3)
        assert rel_err(ve.get_cvorticity(), ref.cvorticity) < 2e-6, (full, read)
    ve.reset()
    ve.step(1e-3)
    assert np.abs(ve.get_cvorticity()).max() == 0.0
    ve.close()


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("dealias", [O.SMOOTH, O.TWO_THIRDS])
def test_upload_sees_single_values_outside(precision, dealias):
    """One value just outside kM (either part of any component, first and last
    rows and columns) is kept by a step, but for its part along k; a negative zero
    there is no value."""
    dk = (1.0, 1.0, 1.0)
    ve, ref = _solver(dk, dealias, precision)
    base = _field(5, dk, dealias, False).astype(ve.cdtype)
    K2, kM2 = ref.kk.K2, ref.kk.kM2
    m = int(np.sqrt(kM2))
    spots = [(0, 0, m + 1), (0, m + 1, 1), (N - 1, 0, m + 1), (N // 2, N // 2, N // 2), (N - m - 1, 0, 1),
             (m + 1, N - 1, 2)]
    for i, at in enumerate(spots):
        assert K2[at] > kM2
        k = np.array([at[2]] + [j if j <= N // 2 else j - N for j in at[:2]], float)
        for value in ((1e-3, 1e-3j)[i % 2], complex(-0.0, -0.0)):
            w = base.copy()
            w[at][(i + 1) % 3] = value
            ve.set_cvorticity(w)
            ve.step(1e-3)
            got = ve.get_cvorticity()
            want = w[at] - k * (k @ w[at]) / (k @ k)
            assert np.abs(got[at] - want).max() <= 1e-5 * abs(value), (at, value)
            got[at] = 0
            assert not got[K2 > kM2].any(), (at, value)
    ve.close()


@pytest.mark.parametrize("precision", ["single", "double"])
def test_ensemble_of_unequal_members(precision):
    """Members with different rules, boxes and states (one full, replaced while
    in the ensemble): bit-identical to stepping alone."""
    from bfps_b200.solver import ensemble
    mk = [((1.0, 1.0, 1.0), O.SMOOTH, False), ((1.0, 1.0, 1.0), O.TWO_THIRDS, False),
          ((1.0, 0.5, 2.0), O.SMOOTH, False)]
    fields = [_field(20 + i, dk, de, fu) for i, (dk, de, fu) in enumerate(mk)]
    replaced = _field(30, mk[1][0], mk[1][1], True)
    alone, ens, members = [], ensemble(), []
    for (dk, de, _), w in zip(mk, fields):
        for group in (alone, members):
            ve, _ = _solver(dk, de, precision)
            ve.set_cvorticity(w)
            group.append(ve)
        ens.add(members[-1], 1e-3)
    ens.step(2)
    members[1].set_cvorticity(replaced)
    ens.step(1)
    for i, ve in enumerate(alone):
        ve.step(1e-3, 2)
        if i == 1:
            ve.set_cvorticity(replaced)
        ve.step(1e-3)
    for a, b in zip(alone, members):
        assert np.array_equal(a.get_cvorticity(), b.get_cvorticity())
    ens.close()
    for ve in alone + members:
        ve.close()
