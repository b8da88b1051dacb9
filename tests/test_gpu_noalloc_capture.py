"""The no-allocation PME as links of a chain of launches: the same bits called
directly, back to back on a side stream, and replayed from a captured graph."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grid", [(1, (8, 8, 8)), (700, (32, 27, 50)), (5000, (64, 64, 64))])
def test_chained_launches_captured_and_repeated(n, grid):
    torch = pytest.importorskip("torch")
    from nexusmd_gb300.engine import load_library
    L = load_library()
    f = L.nxm_pme_reciprocal_noalloc
    f.restype = C.c_int
    rng = np.random.default_rng(n)
    xyz = torch.tensor(rng.uniform(0, 4.0, (n, 3)), dtype=torch.float64, device="cuda")
    q = torch.tensor(rng.uniform(-1, 1, n), dtype=torch.float64, device="cuda")
    lb, ub = (C.c_double * 3)(0, 0, 0), (C.c_double * 3)(4.0, 4.0, 4.0)
    g = (C.c_int32 * 3)(*grid)

    def call(F, e):
        rc = f(C.c_void_p(xyz.data_ptr()), C.c_void_p(q.data_ptr()), C.c_int32(n), lb, ub, g, C.c_double(2.6),
               C.c_void_p(F.data_ptr()), C.c_void_p(e.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, L.nxm_last_error().decode()

    def out():
        return torch.zeros((n, 3), dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")

    F0, e0 = out()
    call(F0, e0)
    torch.cuda.synchronize()
    assert bool(torch.isfinite(F0).all()) and float(e0) != 0.0
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        pairs = [out() for _ in range(3)]
        for F, e in pairs:
            call(F, e)
    torch.cuda.synchronize()
    for F, e in pairs:
        assert torch.equal(F, F0) and torch.equal(e, e0)
    F1, e1 = out()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(F1, e1)
    for _ in range(2):
        F1.zero_()
        e1.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(F1, F0) and torch.equal(e1, e0)
