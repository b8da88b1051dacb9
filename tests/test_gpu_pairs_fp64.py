"""FP64 pair kernel against the FP64 oracle where its parts meet: batches of 32
pairs that come out whole, one short and nearly empty, both ends of the Taylor
table of the Ewald terms and past it, a single row of it, and the switching
function.

Tolerance: both sides are sums of FP64 terms, each within a few 2^-53 of its
largest part; 1e-12 of the norm leaves room for sums of some hundred terms per
atom and the transform's log2 of the grid points.  Energies are sums of words
of 2^-28 kJ/mol, rounded once per warp.
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gas(n, box, seed, cutoff, tol):
    """n charged Lennard-Jones atoms, none closer than 0.14 nm, no bonds."""
    rng = np.random.default_rng(seed)
    per = int(np.ceil(n ** (1 / 3)))
    a = box / per
    assert a > 0.17
    sites = (np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    half = min(0.5 * (a - 0.14), 0.2)
    pos = sites[rng.choice(len(sites), n, replace=False)] + rng.uniform(-half / 2, half / 2, (n, 3))
    q = rng.uniform(-1, 1, n)
    e2, f2 = np.zeros((0, 2), np.int32), np.zeros((0, 2))
    return types.SimpleNamespace(
        n=n, pos=np.mod(pos, box), mass=np.full(n, 12.0), charge=q - q.mean(), sigma=rng.uniform(0.1, 0.2, n),
        epsilon=rng.uniform(0.05, 0.6, n), bonds=e2, bond_prm=f2, angles=np.zeros((0, 3), np.int32), angle_prm=f2,
        torsions=np.zeros((0, 4), np.int32), torsion_prm=f2, torsion_n=np.zeros(0, np.int32), cutoff=cutoff,
        ewald_tol=tol, box=np.full(3, float(box)), grid=(24, 27, 20))


@pytest.mark.parametrize("n,box,cutoff,tol,switch", [
    (2, 2.0, 1.0, 5e-4, 0.0),
    (33, 2.0, 1.0, 5e-4, 0.0),
    (700, 2.4, 1.0, 5e-4, 0.0),
    (700, 2.4, 1.0, 5e-4, 0.85),
    (700, 2.4, 1.1, 1e-19, 0.0),   # (alpha r)^2 up to 43, past the table
    (350, 2.4, 0.9, 0.49, 0.0),    # (alpha r)^2 below 0.03: one row
])
def test_fp64_pairs_match_oracle(oracle, n, box, cutoff, tol, switch):
    from nexusmd_gb300.engine import Engine
    s = _gas(n, box, 11 + n, cutoff, tol)
    lb, ub = np.zeros(3), s.box.copy()
    ob = oracle.box_explicit(lb, ub)
    off, lst = oracle.exclusions(s.n, s.bonds)
    d = oracle.describe(s, box_mode=1, lb=lb, ub=ub, use_switch=int(switch > 0), switch_dist=switch, switch_quirk=0)
    F0, E0 = oracle.forces(d, s.pos, ob, off, lst)
    eng = Engine(s, precision=0, box="explicit", use_switch=int(switch > 0), switch_dist=switch)
    F = eng.compute_forces()
    E = eng.energies()
    eng.close()
    err = np.linalg.norm(F - F0) / np.linalg.norm(F0)
    print(n, tol, switch, "force", err, {k: E[k] - E0[k] for k in ("coulomb", "vdw", "recip")})
    assert err <= 1e-12
    for k in ("coulomb", "vdw"):
        # the terms' own size, not the sum's: pairs of either sign cancel
        assert abs(E[k] - E0[k]) <= 1e-12 * n * 139.0 / 0.14 + 2.0 ** -28 * n, (k, E[k], E0[k])
