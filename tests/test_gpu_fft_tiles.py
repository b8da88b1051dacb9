"""The FFT's line path where its tiles end: axes of one, two, three and four
passes, fewer lines than a tile holds and one more, odd counts of real lines,
in both precisions, against numpy's transform of the engine's own charge grid.

Tolerance: a transform of n points rounds log2(n) times at most; forward and
inverse stay within 4 log2(n) 2^-24 (2^-53) of the norm, with a factor of 4 for
the twiddles' own rounding.
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(8, 8, 8), (5, 9, 10), (27, 5, 6), (50, 16, 81), (135, 9, 8), (12, 250, 15), (256, 10, 18)])
@pytest.mark.parametrize("precision", [0, 1])
def test_line_path_convolution_matches_numpy(grid, precision):
    from nexusmd_gb300.engine import Engine
    rng = np.random.default_rng(sum(grid))
    n = 40
    e2, f2 = np.zeros((0, 2), np.int32), np.zeros((0, 2))
    q = rng.uniform(-1, 1, n)
    s = types.SimpleNamespace(
        n=n, pos=rng.uniform(0, 3.0, (n, 3)), mass=np.ones(n), charge=q - q.mean(), sigma=np.full(n, 0.1),
        epsilon=np.full(n, 0.1), bonds=e2, bond_prm=f2, angles=np.zeros((0, 3), np.int32), angle_prm=f2,
        torsions=np.zeros((0, 4), np.int32), torsion_prm=f2, torsion_n=np.zeros(0, np.int32), cutoff=1.0,
        ewald_tol=5e-4, box=np.full(3, 3.0), grid=grid)
    eng = Engine(s, precision=precision, box="explicit", fft_path=1)
    eng.compute_forces()
    charge, influence, got = eng.pme_grids()
    eng.close()
    want = np.fft.irfftn(np.fft.rfftn(charge) * influence, s=grid, axes=(0, 1, 2), norm="forward")
    points = float(np.prod(grid))
    bound = 16 * np.log2(points) * (2.0 ** -24 if precision else 2.0 ** -53)
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    print(grid, precision, err, bound)
    assert err <= bound
