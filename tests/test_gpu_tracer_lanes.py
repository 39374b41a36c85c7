"""Lanes and lane groups of the tracer gather: tracer counts on both sides of
every change of the split (tracer_split: up to 37888 threads; 4 lanes a row in
FP64, 2 in FP32 and for n = 1) and of the form for many, all stencil widths,
stencils across the periodic boundary at every lane, values beside a stencil,
against the oracle; the same bits alone and batched."""
import numpy as np
import pytest

from oracle import nsve as O
from oracle import particles as P
from bfps_b200 import ic
from gpu_util import rel_err

pytestmark = pytest.mark.gpu

N = 32


def _positions(count, seed):
    pos = ic.tracer_ic(count, seed=seed)
    h = 2 * np.pi / N
    # a stencil starting at every offset of the row, and beyond both ends
    k = min(count, 2 * N)
    pos[:k, 0] = (np.arange(k) - 3) * h + 0.3 * h
    return pos


@pytest.fixture(scope="module")
def flow():
    w0 = ic.vorticity_ic(N, seed=1)
    ref = O.VorticityEquation(N)
    return w0, ref.ift(ref.compute_velocity(w0))


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("nm,count", [((1, 1), 1), ((1, 0), 2368), ((1, 2), 2369), ((2, 0), 33), ((2, 2), 1184),
                                      ((2, 1), 1185), ((3, 2), 1184), ((3, 0), 4737), ((4, 1), 2369),
                                      ((4, 0), 4736), ((5, 2), 65), ((5, 1), 9473),
                                      ((1, 1), 4736), ((1, 0), 9472), ((1, 2), 131072), ((1, 2), 131073),
                                      ((2, 0), 131072), ((2, 0), 131073)])
def test_sample_at_split_edges(flow, precision, nm, count):
    from bfps_b200.solver import vorticity_equation, particles_system
    w0, ur = flow
    ve = vorticity_equation(N, precision=precision)
    ve.set_cvorticity(w0)
    ve.velocity_rspace()
    pos = _positions(count, seed=count)
    ps = particles_system(ve, pos, nm[0], nm[1], nsteps=2)
    got = ps.sample_velocity()
    field = ur if precision == "double" else ve.get_rvelocity()[:, :, :N].astype(np.float64)
    want = P.sample(field, pos, nm[0], nm[1], P.Geometry(N, N, N))
    # FP64: sums of up to 12^3 products in another order; FP32: x weights and
    # row sums of up to 12 terms rounded to FP32
    tol = 1e-13 * 12 if precision == "double" else 2e-6
    assert np.abs(got - want).max() <= tol * np.abs(field).max()
    ps.close()
    ve.close()


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("nm,count", [((1, 1), 9), ((2, 0), 2500), ((3, 2), 40), ((4, 1), 40), ((5, 1), 9)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_beside_the_stencil_do_not_enter(flow, precision, nm, count, bad):
    """Not-finite planes of points right beside the stencil, at every alignment
    of the stencil's row, leave the sample as it is; inside, they reach it."""
    from bfps_b200.solver import vorticity_equation, particles_system
    _, ur = flow
    n = nm[0]
    ve = vorticity_equation(N, precision=precision)
    h = 2 * np.pi / N
    rng = np.random.default_rng(count)
    # cells 14..21 start their rows at every word of a vector (8 FP32, 4 FP64);
    # cell 1: across the boundary (n > 1)
    for cell in [1] + list(range(14, 22)):
        pos = rng.random((count, 3)) * 2 * np.pi
        pos[:, 0] = (cell + 0.1 + 0.8 * rng.random(count)) * h
        pos[-1, 0] -= h  # the last tracer's stencil holds the left plane
        field = np.zeros(ve.rshape, ve.rdtype)
        field[:, :, :N] = ur
        clean = field[:, :, :N].astype(np.float64)
        field[:, :, [(cell - n - 1) % N, (cell + n + 2) % N]] = bad
        ve.set_rvelocity(field)
        ps = particles_system(ve, pos, nm[0], nm[1], nsteps=2)
        got = ps.sample_velocity()
        ps.close()
        want = P.sample(clean, pos, nm[0], nm[1], P.Geometry(N, N, N))
        # as in test_sample_at_split_edges
        tol = 1e-13 * 12 if precision == "double" else 2e-6
        assert np.abs(got - want)[:-1].max() <= tol * np.abs(clean).max(), cell
        assert not np.isfinite(got[-1]).any()
    ve.close()


@pytest.mark.parametrize("precision,n", [("double", 2), ("single", 2), ("single", 1)])
def test_batched_systems_of_unequal_split(flow, precision, n):
    from bfps_b200.solver import NSVEparticles_step, ensemble, particles_system, vorticity_equation
    w0, _ = flow
    counts = [1, 7, 1184, 1185, 3000, 9473, 131073]
    ens, a, b = ensemble(), [], []
    for i, c in enumerate(counts):
        for group in (a, b):
            ve = vorticity_equation(N, precision=precision)
            ve.set_cvorticity(w0)
            group.append((ve, particles_system(ve, _positions(c, i), n, 0, nsteps=3)))
        ens.add(b[-1][0], 0.01, b[-1][1])
    ens.step(4)
    for (ve, ps), (ve2, ps2) in zip(a, b):
        NSVEparticles_step(ve, ps, 0.01, 4)
        for x, y in zip(ps.state(), ps2.state()):
            assert np.array_equal(x, y)
    ens.close()


@pytest.mark.parametrize("n", [16, 32, 64, 128])
@pytest.mark.parametrize("precision", ["double", "single"])
def test_launches_that_start_early_see_what_came_before(n, precision):
    """Passes of small grids are launched while the pass before them drains.  At the
    end of a step (inside, both sides launch alike): steps queued back to back give
    the bits of steps waited for one by one."""
    from bfps_b200.solver import NSVEparticles_step, particles_system, vorticity_equation
    out = []
    for wait in (True, False):
        ve = vorticity_equation(n, precision=precision)
        ve.nu, ve.forcing_type = 0.05, "linear"
        ve.set_cvorticity(ic.vorticity_ic(n, seed=9))
        ps = particles_system(ve, ic.tracer_ic(300, seed=2), 2, 0, nsteps=2)
        if wait:
            for _ in range(20):
                NSVEparticles_step(ve, ps, 0.002, 1)
                ve.last_step_ms()
        else:
            NSVEparticles_step(ve, ps, 0.002, 20)
        out.append((ve.get_cvorticity(), ps.state()[0]))
        ps.close()
        ve.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
