"""Many-right-hand-side products and the batched solve where they change path: block rows shorter and
longer than the 32 slots a warp takes at once, every supported number of right-hand sides, vectors
that do not start on a 16-byte boundary, systems that converge at different iterations.

Product tolerance per entry: 2 (terms + 2) u sum |A| |x| with u = 2^-24 (FP32, the matrix rounded too) or
2^-53 -- any order of the sum stays within it."""
import ctypes

import numpy as np
import pytest
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["block", "fan"])
def system(request):
    if request.param == "block":
        P = F.hex_block(9, 7, 5, jitter=0.1, seed=3, fix="zmin")
    else:   # 40 elements around node 0: rows of 2 to ~120 blocks, no structure
        rng = np.random.default_rng(5)
        n = 130
        conn = np.stack([np.concatenate([[0], rng.choice(np.arange(1, n), 7, replace=False)]) for _ in range(40)])
        P = F.Physics(np.arange(1, n + 1), rng.random((n, 3)), conn.T.astype(np.int64), [[np.array([0]), [-1, -1, -1]]])
    M = F.Model("s", P, STEEL)
    rng = np.random.default_rng(1)
    K = torch.from_numpy(rng.standard_normal((M.mesh.nnzb, 3, 3))).cuda()
    S = F.DeviceSystem(M, K=K, F=torch.zeros(3 * P.Num_Node, dtype=torch.float64, device="cuda"))
    import scipy.sparse as sp
    A = sp.bsr_matrix((K.cpu().numpy(), np.asarray(P.ReNode), np.asarray(P.SmNode)), shape=(3 * P.Num_Node,) * 2).tocsr()
    return P, S, A


@pytest.mark.parametrize("nrhs", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("shift", [0, 1])
def test_product(system, nrhs, fp32, shift):
    P, S, A = system
    dt = torch.float32 if fp32 else torch.float64
    buf = torch.empty(3 * P.Num_Node * nrhs + 4, dtype=dt, device="cuda")
    x = buf[shift:shift + 3 * P.Num_Node * nrhs].view(3 * P.Num_Node, nrhs)
    x.copy_(torch.from_numpy(np.random.default_rng(nrhs).standard_normal((3 * P.Num_Node, nrhs))))
    S.K32()
    y = torch.full_like(x, float("nan"))
    for v in range(8 if nrhs == 1 else 1):
        _lib.check(S.lib.fem_bsr_spmv(ctypes.byref(S._A32 if fp32 else S.A64), nrhs, x.data_ptr(), y.data_ptr(), v,
                                      S.stream), "spmv")
        xd, yd = x.double().cpu().numpy(), y.double().cpu().numpy()
        terms = np.diff(A.indptr)[:, None] + 2
        u = 2.0 ** -24 if fp32 else 2.0 ** -53
        assert np.all(np.abs(yd - A @ xd) <= 2 * terms * u * (abs(A) @ np.abs(xd))), v


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("nrhs", [2, 4, 8, 32])
def test_systems_that_converge_at_different_iterations(mixed, nrhs):
    """Columns of very different difficulty (a smooth load, single nodes, zero): each right to 1e-8 of
    a direct solve, zero exactly zero; the caller's U off a 16-byte boundary."""
    import scipy.sparse.linalg as spla
    P = F.hex_block(11, 6, 5, jitter=0.1, seed=2, fix="zmin")
    M = F.Model("s", P, STEEL)
    S = F.DeviceSystem(M)
    rng = np.random.default_rng(0)
    Fm = np.zeros((3 * P.Num_Node, nrhs))
    free = np.nonzero(np.asarray(P.xyz)[:, 2] > 0)[0]
    for k in range(nrhs):
        if k % 3 == 0:
            Fm[3 * free + 2, k] = 1.0
        elif k % 3 == 1:
            Fm[3 * free[rng.integers(free.size)] + rng.integers(3), k] = 1.0
    lu = spla.splu(M.Get_MatrixKL().tocsc())
    U, st = S.solve(F=torch.from_numpy(Fm).cuda(), rtol=1e-11, mixed=mixed)
    assert st["status"] == 0, st
    Ur = lu.solve(Fm)
    for k in range(nrhs):
        u = U[:, k].cpu().numpy()
        if k % 3 == 2:
            assert np.all(u == 0.0)
        else:
            assert np.linalg.norm(u - Ur[:, k]) <= 1e-8 * np.linalg.norm(Ur[:, k])
    # the C entry with U shifted by one double: the same values
    buf = torch.zeros(3 * P.Num_Node * nrhs + 1, dtype=torch.float64, device="cuda")
    Ft = torch.from_numpy(Fm).cuda().contiguous()
    o = _lib.FemPcgOpts(nrhs, int(mixed), 1e-11, 50000, 1e-4, 20000, 40, 1, 16, 0, S.variant(True, nrhs) if mixed else 0,
                        _lib.RESIDUAL_FP64, 0)
    stt = _lib.FemPcgStats()
    ws = torch.empty(int(S.lib.fem_pcg_workspace_bytes(S.n, nrhs, int(mixed))), dtype=torch.uint8, device="cuda")
    _lib.check(S.lib.fem_pcg_solve(ctypes.byref(S.A64), ctypes.byref(S._A32) if mixed else None,
                                   S.block_jacobi().data_ptr(), Ft.data_ptr(), buf[1:].data_ptr(), ctypes.byref(o),
                                   ctypes.byref(stt), ws.data_ptr(), ws.numel(), S.stream), "solve")
    torch.cuda.synchronize()
    V = buf[1:].view(3 * P.Num_Node, nrhs)
    assert stt.status == 0
    assert float((V - U).abs().max()) <= 1e-9 * float(U.abs().max())
