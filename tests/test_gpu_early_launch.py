"""Passes of short launches start while the pass before them drains (up to 2^22
grid points on a stream, up to 2^20 in the captured graphs of an ensemble of one size, IY of
16^3 for fewer than four members); the others wait for it.  Both give the same
bits."""
import numpy as np
import pytest

from bfps_b200 import _lib, ic

pytestmark = pytest.mark.gpu

STEPS = 12


def _member(n, precision, dealias, seed):
    from bfps_b200.solver import particles_system, vorticity_equation
    ve = vorticity_equation(n, precision=precision, dealias_type=dealias)
    ve.nu, ve.forcing_type = 0.05, "linear"
    ve.set_cvorticity(ic.vorticity_ic(n, seed=seed, dtype=ve.cdtype))
    return ve, particles_system(ve, ic.tracer_ic(300, seed=seed), 2, 0, nsteps=2)


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("n,precision,dealias", [(16, "single", _lib.SMOOTH), (32, "single", _lib.SMOOTH),
                                                 (64, "double", _lib.SMOOTH), (64, "single", _lib.SMOOTH),
                                                 (128, "single", _lib.SMOOTH), (128, "double", _lib.TWO_THIRDS)])
def test_early_and_waiting_launches_agree(n, precision, dealias, graphs):
    """One instance alone (early), two in an ensemble (early but for 128^3 in
    graphs) and the first two of one just above the limit (waiting; 16^3: a few
    members, whose IY waits)."""
    from bfps_b200.solver import NSVEparticles_step, ensemble
    many = 5 if n == 16 else (1 << (20 if graphs else 22)) // n ** 3 + 1
    many = max(many, 3)
    out = []
    for count in (1, 2, many):
        members = [_member(n, precision, dealias, seed) for seed in range(min(count, 2))]
        # the others are there for the size of the launches
        members += [_member(n, precision, dealias, 0) for _ in range(count - 2)]
        if count == 1:
            NSVEparticles_step(members[0][0], members[0][1], 0.002, STEPS)
        else:
            ens = ensemble()
            ens.use_graphs(graphs)
            for ve, ps in members:
                ens.add(ve, 0.002, ps)
            ens.step(STEPS)
            ens.close()
        out.append([(ve.get_cvorticity(), ps.state()[0]) for ve, ps in members[:2]])
        for ve, ps in members:
            ps.close()
            ve.close()
    alone, pair, group = out
    for got in (pair, group):
        assert np.array_equal(got[0][0], alone[0][0]) and np.array_equal(got[0][1], alone[0][1])
    assert np.array_equal(pair[1][0], group[1][0]) and np.array_equal(pair[1][1], group[1][1])
