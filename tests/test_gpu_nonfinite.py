"""An atom whose coordinate is not finite, mixed precision: it interacts with
nothing in real space, and the other atoms' energies and forces are those of
the system without its charge and its Lennard-Jones part -- also for the atom
that shares a list with it.  (The same sums in the two engines compared: FP32
rounding of other orders of summation, 1e-5 of the largest term.)
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gas(n, box, seed):
    rng = np.random.default_rng(seed)
    per = int(np.ceil(n ** (1 / 3)))
    a = box / per
    sites = (np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    pos = sites[rng.choice(len(sites), n, replace=False)] + rng.uniform(-0.05, 0.05, (n, 3))
    q = rng.uniform(-0.3, 0.3, n)
    e2, f2 = np.zeros((0, 2), np.int32), np.zeros((0, 2))
    return types.SimpleNamespace(
        n=n, pos=np.mod(pos, box), mass=np.full(n, 12.0), charge=q - q.mean(), sigma=rng.uniform(0.1, 0.2, n),
        epsilon=rng.uniform(0.1, 0.6, n), bonds=e2, bond_prm=f2, angles=np.zeros((0, 3), np.int32), angle_prm=f2,
        torsions=np.zeros((0, 4), np.int32), torsion_prm=f2, torsion_n=np.zeros(0, np.int32), cutoff=1.0,
        ewald_tol=5e-4, box=np.full(3, float(box)), grid=(24, 24, 24))


@pytest.mark.parametrize("switch", [0.0, 0.8])
@pytest.mark.parametrize("bad", [0, 1])
def test_nonfinite_coordinate_stays_with_its_atom(switch, bad):
    from nexusmd_gb300.engine import Engine
    s = _gas(900, 2.6, 5)
    kw = dict(precision=1, box="explicit", use_switch=int(switch > 0), switch_dist=switch)
    # the bad atom falls into cell (0, 0, 0): one of whose atoms is its
    # partner in a list when the others there are odd in number, so try both
    inside = np.flatnonzero((s.pos < 2.6 / 4).all(1))
    out = np.flatnonzero((s.pos > 1.0).all(1))
    if (len(inside) + bad) % 2 == 0:
        s.pos[inside[0]] += 1.3
    k = out[3]
    s.charge[k] = 0.0
    s.charge -= s.charge.sum() / (s.n - 1) * (np.arange(s.n) != k)
    s.epsilon[k] = 0.0
    eng = Engine(s, **kw)
    F0, E0 = eng.compute_forces(), eng.energies()
    pos = s.pos.copy()
    pos[k] = np.nan
    eng.set_positions(pos)
    F, E = eng.compute_forces(), eng.energies()
    eng.close()
    others = np.arange(s.n) != k
    print({t: (E[t], E0[t]) for t in ("coulomb", "vdw", "recip")}, np.abs(F - F0)[others].max())
    for t in ("coulomb", "vdw"):
        assert abs(E[t] - E0[t]) <= 1e-5 * max(abs(E0[u]) for u in ("coulomb", "vdw", "recip")) + 1e-6, t
    assert np.linalg.norm((F - F0)[others]) <= 1e-5 * np.linalg.norm(F0[others])
