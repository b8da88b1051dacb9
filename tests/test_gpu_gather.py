"""The PME gather on either side of its rule (five lanes per atom below 9,728
atoms in a context, one thread above) and where a warp's six atoms do not come
out even: a system alone against the same system beside another in a batch
large enough for the other form.

Tolerance: both forms add 125 FP32 products q theta theta theta' phi (K / L) in
another order; 125 roundings of at most max|phi| each, weights below 1.
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gas(n, per, h, grid, seed):
    """Atoms on a lattice wider than the cutoff: no pair adds to the reciprocal force."""
    rng = np.random.default_rng(seed)
    sites = np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (sites[rng.choice(len(sites), n, replace=False)] + 0.5) * h + rng.uniform(-0.02, 0.02, (n, 3))
    e2, f2 = np.zeros((0, 2), np.int32), np.zeros((0, 2))
    return types.SimpleNamespace(
        n=n, pos=pos, mass=np.ones(n), charge=rng.uniform(-1.0, 1.0, n), sigma=np.full(n, 0.1), epsilon=np.zeros(n),
        bonds=e2, bond_prm=f2, angles=np.zeros((0, 3), np.int32), angle_prm=f2, torsions=np.zeros((0, 4), np.int32),
        torsion_prm=f2, torsion_n=np.zeros(0, np.int32), cutoff=0.25, ewald_tol=5e-4, box=np.full(3, per * h),
        grid=grid)


@pytest.mark.parametrize("n", [1, 5, 6, 7, 31, 1000])
def test_gather_forms_agree(n):
    from nexusmd_gb300.engine import Engine
    s = _gas(n, 12, 0.3, (24, 27, 20), n)
    other = _gas(9728, 22, 0.3, (64, 60, 54), 3)
    small = Engine(s, box="explicit")
    F = small.compute_forces()
    phi = small.pme_grids()[2]
    small.close()
    both = Engine([s, other], box="explicit")
    G = both.compute_forces()[:n]
    both.close()
    bound = 125 * 2.0 ** -24 * np.abs(s.charge)[:, None] * (np.array(s.grid) / s.box) * np.abs(phi).max()
    print(n, np.abs(F - G).max(), bound.max(), np.abs(F).max())
    assert (np.abs(F - G) <= bound).all()
