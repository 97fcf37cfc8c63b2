"""Tall-skinny FP64 products at the edges of their tiles: row counts off the 16-, 32- and 64-row
steps, column counts around 32 and 256, every template width and one less, strided operands.
Tolerance: 4 (sum length) 2^-53 of the sums of absolute products (any order of n additions and
products stays within it)."""
import ctypes

import numpy as np
import pytest
import torch

from fem_taichi_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 33, 64, 1000, 20001])
@pytest.mark.parametrize("m,b", [(1, 1), (31, 4), (32, 5), (33, 8), (64, 10), (190, 12), (255, 15), (256, 16), (97, 23),
                                 (200, 32)])
def test_products(n, m, b):
    L, d = _lib.load(), "cuda"
    g = torch.Generator(device=d)
    g.manual_seed(n + m + b)
    Qs = torch.randn((n, m + 3), dtype=torch.float64, device=d, generator=g)
    Xs = torch.randn((n, b + 2), dtype=torch.float64, device=d, generator=g)
    Q, X = Qs[:, :m], Xs[:, :b]
    W = torch.randn((n, b + 1), dtype=torch.float64, device=d, generator=g)
    C = torch.full((m, b + 1), 7.0, dtype=torch.float64, device=d)
    ws = torch.empty(int(L.fem_ts_gemm_tn_workspace_bytes(n, m, b)), dtype=torch.uint8, device=d)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(L.fem_ts_gemm_tn(n, m, b, Q.data_ptr(), m + 3, X.data_ptr(), b + 2, C.data_ptr(), b + 1, ws.data_ptr(),
                                ws.numel(), st), "tn")
    q, x = Q.cpu().numpy(), X.cpu().numpy()
    c = C.cpu().numpy()
    assert np.all(c[:, b] == 7.0)
    c = np.ascontiguousarray(c[:, :b])
    eps = 2.0 ** -53
    assert np.all(np.abs(c - q.T @ x) <= 4 * n * eps * (np.abs(q.T) @ np.abs(x)))
    for alpha, beta in ((-1.0, 1.0), (0.5, 0.0), (2.0, -0.25)):
        V = W.clone()
        if beta == 0.0:
            V[:, :b] = float("nan")     # not read
        _lib.check(L.fem_ts_gemm_nn(n, m, b, Q.data_ptr(), m + 3, C.data_ptr(), b + 1, alpha, beta, V.data_ptr(),
                                    b + 1, st), "nn")
        v, w = V.cpu().numpy(), W.cpu().numpy()
        assert np.array_equal(v[:, b], w[:, b])
        ref = alpha * (q @ c) + (beta * w[:, :b] if beta else 0.0)
        bound = abs(alpha) * (np.abs(q) @ np.abs(c)) + abs(beta) * np.abs(w[:, :b])
        assert np.all(np.abs(v[:, :b] - ref) <= 4 * (m + 2) * eps * bound)
