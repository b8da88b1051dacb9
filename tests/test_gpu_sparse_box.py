"""A few atoms in a large box: the neighbour lists take room by atoms, not by
the box's cells (most of them empty), and the pair set (FP64: the forces too)
is the oracle's.

2,000 atoms, 60 of them in a droplet, in a 40 nm box: 373,248 cells, whose
groups' span records (119 MB) and counters are all that may grow with the box;
a list place per two cells would be another 287 MB.
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _droplet(n, box, seed, drop=60):
    """`drop` atoms on a lattice in one place, the others spread over the box."""
    rng = np.random.default_rng(seed)
    k = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    tight = 11.0 + 0.2 * k[rng.permutation(len(k))[:drop]] + rng.uniform(-0.02, 0.02, (drop, 3))
    far = (np.stack(np.meshgrid(*[np.arange(20)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * (box / 20)
    far = far[(np.abs(far - 11.3) > 2.0).any(1)]
    far = far[rng.choice(len(far), n - drop, replace=False)] + rng.uniform(-0.4, 0.4, (n - drop, 3)) * (box / 20)
    pos = np.concatenate([tight, far])[rng.permutation(n)]
    q = rng.uniform(-0.5, 0.5, n)
    e2, f2 = np.zeros((0, 2), np.int32), np.zeros((0, 2))
    return types.SimpleNamespace(
        n=n, pos=np.mod(pos, box), mass=np.full(n, 12.0), charge=q - q.mean(), sigma=rng.uniform(0.1, 0.2, n),
        epsilon=rng.uniform(0.1, 0.6, n), bonds=e2, bond_prm=f2, angles=np.zeros((0, 3), np.int32), angle_prm=f2,
        torsions=np.zeros((0, 4), np.int32), torsion_prm=f2, torsion_n=np.zeros(0, np.int32), cutoff=1.0,
        ewald_tol=5e-4, box=np.full(3, float(box)), grid=(48, 48, 48))


@pytest.mark.parametrize("precision", [0, 1])
def test_sparse_box(oracle, precision):
    import torch

    from nexusmd_gb300.engine import Engine
    s = _droplet(2000, 40.0, 3)
    lb, ub = np.zeros(3), s.box.copy()
    ob = oracle.box_explicit(lb, ub)
    off, lst = oracle.exclusions(s.n, s.bonds)
    F0, _ = oracle.forces(oracle.describe(s, box_mode=1, lb=lb, ub=ub), s.pos, ob, off, lst)
    ref = oracle.neighbor_pairs(s.pos, ob, off, lst, s.cutoff)
    ref = ref[np.lexsort((ref[:, 1], ref[:, 0]))]
    small = _droplet(400, 24.0, 4)
    Engine(small, precision=precision, box="explicit").close()  # the process's own allocations
    before = torch.cuda.mem_get_info(0)[0]
    eng = Engine(s, precision=precision, box="explicit")
    F = eng.compute_forces()
    used = before - torch.cuda.mem_get_info(0)[0]
    pairs = eng.pairs()
    eng.close()
    print("context: %.0f MB" % (used / 1e6))
    assert used < 200e6
    assert np.array_equal(pairs, ref)
    if precision == 0:
        assert np.linalg.norm(F - F0) <= 1e-9 * np.linalg.norm(F0)
