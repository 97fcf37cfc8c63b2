"""FP32 products with many right-hand sides and an infinite entry in x: rows whose length is a multiple of 4
have no padding block, so what they give is the sum of their own products -- infinite where one product
is, not NaN from a zero times it -- whatever slots of the warp the row leaves empty."""
import ctypes

import numpy as np
import pytest
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [2, 4, 8, 16, 32])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_rows_without_padding(nrhs, value):
    P = F.hex_block(7, 5, 4, jitter=0.1, seed=3, fix="zmin")
    M = F.Model("s", P, STEEL)
    rng = np.random.default_rng(1)
    K = rng.uniform(0.5, 1.5, (M.mesh.nnzb, 3, 3))     # positive: one infinite product, infinite sum
    S = F.DeviceSystem(M, K=torch.from_numpy(K).cuda(), F=torch.zeros(3 * P.Num_Node, dtype=torch.float64, device="cuda"))
    S.K32()
    ptr, col = np.asarray(P.SmNode), np.asarray(P.ReNode)
    full = np.nonzero(np.diff(ptr) % 4 == 0)[0]
    assert {8, 12} <= set(np.diff(ptr)[full].tolist())
    for node in full[:: max(1, full.size // 12)]:
        x = torch.ones((3 * P.Num_Node, nrhs), dtype=torch.float32, device="cuda")
        x[3 * int(node) + 1, nrhs - 1] = value
        y = torch.empty_like(x)
        _lib.check(S.lib.fem_bsr_spmv(ctypes.byref(S._A32), nrhs, x.data_ptr(), y.data_ptr(), 0, S.stream), "spmv")
        y = y.cpu().numpy().reshape(P.Num_Node, 3, nrhs)
        for i in full:
            touched = node in col[ptr[i]:ptr[i + 1]]
            assert np.all(y[i, :, nrhs - 1] == value) if touched else np.isfinite(y[i]).all(), (node, i)
            assert np.isfinite(y[i, :, :-1]).all()
