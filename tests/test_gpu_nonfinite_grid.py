"""Charge-grid indices of a coordinate that is not finite, on grids whose edges
are no powers of two (the least integer's remainder is then below zero): the
entry with static scratch gives the other atoms the forces they have without
that atom's charge, bit for bit, and the FP64 engine gives its first forces
again once the coordinate is put right.
"""
import ctypes as C
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAD = [np.nan, np.inf, -np.inf]


@pytest.mark.parametrize("bad", BAD)
def test_static_scratch_entry(bad):
    torch = pytest.importorskip("torch")
    from nexusmd_gb300.engine import load_library
    L = load_library()
    f = L.nxm_pme_reciprocal_noalloc
    f.restype = C.c_int
    rng = np.random.default_rng(9)
    n, k = 70, 5
    xyz, q = rng.uniform(0, 3.0, (n, 3)), rng.uniform(-1, 1, n)
    lb, ub, g = (C.c_double * 3)(0, 0, 0), (C.c_double * 3)(3.0, 3.0, 3.0), (C.c_int32 * 3)(27, 50, 45)

    def call(xyz, q):
        x, c = torch.tensor(xyz, device="cuda"), torch.tensor(q, device="cuda")
        F = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        e = torch.zeros(1, dtype=torch.float64, device="cuda")
        rc = f(C.c_void_p(x.data_ptr()), C.c_void_p(c.data_ptr()), C.c_int32(n), lb, ub, g, C.c_double(2.6),
               C.c_void_p(F.data_ptr()), C.c_void_p(e.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, L.nxm_last_error().decode()
        torch.cuda.synchronize()
        return F.cpu().numpy(), float(e)

    q0 = q.copy()
    q0[k] = 0.0
    F0, e0 = call(xyz, q0)
    wild = xyz.copy()
    wild[k] = bad
    F, e = call(wild, q)
    others = np.arange(n) != k
    assert np.array_equal(F[others], F0[others]) and e == e0
    again, e = call(xyz, q0)
    assert np.array_equal(again, F0) and e == e0


@pytest.mark.parametrize("bad", BAD)
def test_fp64_engine(bad):
    from nexusmd_gb300.engine import Engine
    rng = np.random.default_rng(10)
    box, per = 2.4, 9
    sites = (np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * (box / per)
    n = 500
    pos = sites[rng.choice(len(sites), n, replace=False)] + rng.uniform(-0.04, 0.04, (n, 3))
    q = rng.uniform(-1, 1, n)
    e2, f2 = np.zeros((0, 2), np.int32), np.zeros((0, 2))
    s = types.SimpleNamespace(
        n=n, pos=pos, mass=np.full(n, 12.0), charge=q - q.mean(), sigma=rng.uniform(0.1, 0.2, n),
        epsilon=rng.uniform(0.05, 0.6, n), bonds=e2, bond_prm=f2, angles=np.zeros((0, 3), np.int32), angle_prm=f2,
        torsions=np.zeros((0, 4), np.int32), torsion_prm=f2, torsion_n=np.zeros(0, np.int32), cutoff=1.0,
        ewald_tol=5e-4, box=np.full(3, box), grid=(27, 50, 45))
    eng = Engine(s, precision=0, box="explicit")
    F0 = eng.compute_forces()
    wild = pos.copy()
    wild[5] = bad
    eng.set_positions(wild)
    F = eng.compute_forces()
    eng.set_positions(pos)
    again = eng.compute_forces()
    eng.close()
    assert np.isfinite(F0).all() and not np.isfinite(F).all()
    assert np.linalg.norm(again - F0) <= 1e-12 * np.linalg.norm(F0)
