"""The list build at its limits: an atom's capacity where a pair's union is
longer (accepted while each atom's own list fits, refused when one does not),
more entries excluded from one atom of a pair than are kept for the list's end,
and tiles whose shared memory lies between 43 and 48 KB in a process that has
launched nothing larger.

Tolerances as everywhere: the pair set is equal; forces FP64 1e-9, mixed 1e-5
of the norm.
"""
import os
import subprocess
import sys
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _gas(n, box, seed, cutoff, bonds=None):
    rng = np.random.default_rng(seed)
    per = int(np.ceil(n ** (1 / 3)))
    a = box / per
    sites = (np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    half = 0.5 * (a - 0.14)
    pos = sites[rng.choice(len(sites), n, replace=False)] + rng.uniform(-half, half, (n, 3))
    q = rng.uniform(-0.5, 0.5, n)
    bonds = np.zeros((0, 2), np.int32) if bonds is None else bonds
    return types.SimpleNamespace(
        n=n, pos=np.mod(pos, box), mass=np.full(n, 12.0), charge=q - q.mean(), sigma=rng.uniform(0.1, 0.16, n),
        epsilon=rng.uniform(0.05, 0.6, n), bonds=bonds, bond_prm=np.tile([0.3, 1.0], (len(bonds), 1)),
        angles=np.zeros((0, 3), np.int32), angle_prm=np.zeros((0, 2)), torsions=np.zeros((0, 4), np.int32),
        torsion_prm=np.zeros((0, 2)), torsion_n=np.zeros(0, np.int32), cutoff=cutoff, ewald_tol=5e-4,
        box=np.full(3, float(box)), grid=(24, 24, 24))


def _neighbours(s, radius):
    """Atoms within `radius` of each (minimum image)."""
    count = np.zeros(s.n, int)
    for i in range(s.n):
        d = s.pos - s.pos[i]
        d -= s.box * np.round(d / s.box)
        count[i] = ((d ** 2).sum(1) < radius * radius).sum() - 1
    return count


def _check(oracle, s, precision, depth=3, **kw):
    from nexusmd_gb300.engine import Engine
    lb, ub = np.zeros(3), s.box.copy()
    ob = oracle.box_explicit(lb, ub)
    off, lst = oracle.exclusions(s.n, s.bonds, depth)
    d = oracle.describe(s, box_mode=1, lb=lb, ub=ub, exclusion_depth=depth)
    F0, _ = oracle.forces(d, s.pos, ob, off, lst)
    ref = oracle.neighbor_pairs(s.pos, ob, off, lst, s.cutoff)
    ref = ref[np.lexsort((ref[:, 1], ref[:, 0]))]
    eng = Engine(s, precision=precision, box="explicit", exclusion_depth=depth, **kw)
    F = eng.compute_forces()
    pairs = eng.pairs()
    eng.close()
    assert np.array_equal(pairs, ref)
    assert np.linalg.norm(F - F0) <= (1e-5 if precision else 1e-9) * np.linalg.norm(F0)


@pytest.mark.parametrize("precision", [0, 1])
def test_capacity_is_an_atoms(oracle, precision):
    from nexusmd_gb300.engine import Engine, NxmError
    # 228 atoms in the mean, 245 at most, within the list radius of 1.1 nm: a
    # capacity of 256 holds every atom's list, and no union of two
    s = _gas(1200, 3.07, 21, 1.0)
    own = _neighbours(s, 1.1)
    assert 200 < own.mean() and own.max() < 256
    _check(oracle, s, precision, max_neighbors=256)
    # a denser box: some atoms have more than 256
    s = _gas(1500, 3.07, 22, 1.0)
    own = _neighbours(s, 1.1)
    assert own.max() > 270
    eng = Engine(s, precision=precision, box="explicit", max_neighbors=256)
    with pytest.raises(NxmError, match="capacity"):
        eng.compute_forces()
    eng.close()
    _check(oracle, s, precision, max_neighbors=512)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("leaves", [60, 70, 180])
def test_many_entries_excluded_from_one_atom(oracle, precision, leaves):
    # a hub bonded to `leaves` atoms all over the box: at depth 1 the hub
    # alone is excluded from them, the atom that shares its list is not
    n = 900
    hub = 450
    others = np.delete(np.arange(n), hub)
    leaf = np.random.default_rng(leaves).choice(others, min(5 * leaves, len(others)), replace=False)
    s = _gas(n, 2.7, 23, 1.0)
    d = s.pos[leaf] - s.pos[hub]
    d -= s.box * np.round(d / s.box)
    near = leaf[np.argsort((d ** 2).sum(1))][:leaves]
    s.bonds = np.stack([np.minimum(near, hub), np.maximum(near, hub)], 1).astype(np.int32)
    s.bond_prm = np.tile([0.5, 1.0], (leaves, 1))
    _check(oracle, s, precision, depth=1)


FRESH = """
import sys
sys.path.insert(0, %r); sys.path.insert(0, %r)
import numpy as np
import test_gpu_list_limits as t
from nexusmd_gb300.engine import Engine
from oracle.nxo import Oracle
s = t._gas(%d, %r, 31, 1.0)
eng = Engine(s, precision=%d, box="explicit")
lay = eng.layout()
eng.close()
print("hood", lay["hood_capacity"])
t._check(Oracle(), s, %d)
print("fresh process OK")
"""


@pytest.mark.parametrize("n,box", [(1250, 3.40), (2000, 3.40), (3000, 3.40)])
@pytest.mark.parametrize("precision", [0, 1])
def test_shared_memory_below_the_attribute_in_a_fresh_process(oracle, n, box, precision):
    # (dynamic shared memory of the list build, the mixed and the FP64 pair kernel)
    r = subprocess.run([sys.executable, "-c", FRESH % (ROOT, os.path.join(ROOT, "tests"), n, box, precision, precision)],
                       capture_output=True, text=True, timeout=300)
    print(r.stdout, r.stderr[-2000:])
    assert r.returncode == 0 and "fresh process OK" in r.stdout
