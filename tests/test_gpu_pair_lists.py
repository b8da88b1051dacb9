"""Lists shared by pairs of atoms: the pair set and the forces where a list's
parts meet -- cells of one atom, of odd counts and of more than the in-warp
pairing takes, boxes in which the tile holds two images of an atom, exclusions
between and around the two atoms, and the switching function.

Tolerances: the pair set is equal; forces as everywhere (FP64 1e-9, mixed 1e-5
of the force norm; the gas here has no stiff bonds).
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, box, seed, cutoff, cluster=0, bonded=False):
    """n atoms no closer than 0.13 nm: `cluster` of them on a tight lattice in
    one corner, the rest on a jittered lattice over the box; `bonded`: threes
    of consecutive atoms are bonded in a row."""
    rng = np.random.default_rng(seed)
    corner = int(np.ceil(max(cluster, 1) ** (1 / 3)))
    tight = (np.stack(np.meshgrid(*[np.arange(corner)] * 3, indexing="ij"), -1).reshape(-1, 3)[:cluster] + 0.5) * 0.135
    per = int(np.ceil((n + 40) ** (1 / 3)))
    a = box / per
    assert a > 0.17
    sites = (np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    if cluster:
        sites = sites[(sites > corner * 0.135 + 0.1).any(1) & (sites < box - 0.12).all(1)]
    half = 0.5 * (a - 0.14)
    rest = sites[rng.choice(len(sites), n - cluster, replace=False)] + rng.uniform(-half, half, (n - cluster, 3))
    pos = np.concatenate([tight, rest])[rng.permutation(n)]
    q = rng.uniform(-1, 1, n)
    bonds = np.array([(k, k + 1) for k in range(0, n - 1) if k % 3 != 2], np.int32) if bonded else np.zeros((0, 2), np.int32)
    e2 = np.zeros((0, 2))
    return types.SimpleNamespace(
        n=n, pos=np.mod(pos, box), mass=np.full(n, 12.0), charge=q - q.mean(), sigma=rng.uniform(0.1, 0.16, n),
        epsilon=rng.uniform(0.05, 0.6, n), bonds=bonds, bond_prm=np.tile([0.2, 100.0], (len(bonds), 1)),
        angles=np.zeros((0, 3), np.int32), angle_prm=e2, torsions=np.zeros((0, 4), np.int32), torsion_prm=e2,
        torsion_n=np.zeros(0, np.int32), cutoff=cutoff, ewald_tol=5e-4, box=np.full(3, float(box)), grid=(24, 24, 24))


@pytest.mark.parametrize("n,box,cutoff,cluster,bonded,switch", [
    (1, 2.5, 1.0, 0, False, 0.0),      # one atom alone
    (3, 2.5, 1.0, 0, True, 0.0),       # nothing but exclusions
    (61, 3.0, 0.9, 0, False, 0.0),     # cells of none, one and two atoms
    (901, 2.2, 1.0, 0, True, 0.0),     # two images of an atom in the tile
    (1400, 2.9, 1.0, 0, True, 0.8),
    (1500, 4.5, 0.9, 64, True, 0.0),   # a cell at the in-warp pairing's limit
    (1500, 4.5, 0.9, 125, False, 0.0),  # and past it
])
@pytest.mark.parametrize("precision", [0, 1])
def test_pair_lists_match_oracle(oracle, n, box, cutoff, cluster, bonded, switch, precision):
    from nexusmd_gb300.engine import Engine
    s = _system(n, box, 5 + n, cutoff, cluster, bonded)
    lb, ub = np.zeros(3), s.box.copy()
    ob = oracle.box_explicit(lb, ub)
    off, lst = oracle.exclusions(s.n, s.bonds)
    d = oracle.describe(s, box_mode=1, lb=lb, ub=ub, use_switch=int(switch > 0), switch_dist=switch, switch_quirk=0)
    F0, _ = oracle.forces(d, s.pos, ob, off, lst)
    ref = oracle.neighbor_pairs(s.pos, ob, off, lst, cutoff)
    ref = ref[np.lexsort((ref[:, 1], ref[:, 0]))]
    eng = Engine(s, precision=precision, box="explicit", use_switch=int(switch > 0), switch_dist=switch)
    F = eng.compute_forces()
    pairs = eng.pairs()
    eng.close()
    assert np.array_equal(pairs, ref)
    norm = np.linalg.norm(F0)
    assert np.linalg.norm(F - F0) <= (1e-5 if precision else 1e-9) * norm + 1e-9
