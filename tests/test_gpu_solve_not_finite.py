"""A matrix with a NaN or infinite entry: no solve reports success.  The mixed solve ends in its first inner
solve with FEM_ERR_BREAKDOWN and U = 0 (its first residual is F, not F - K 0, which such a K makes NaN, and a
NaN norm would read as converged), and the residual it states is F's; the FP64 solve ends the same way."""
import numpy as np
import pytest
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 2, 32])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("mixed", [True, False])
def test_status(mixed, nrhs, value):
    P = F.hex_block(6, 5, 4, jitter=0.1, seed=3, fix="zmin", load_face="zmax", load=(0, 0, -1))
    M = F.Model("b", P, STEEL)
    K, _, _ = M.assemble(K=True, M=False, F=False)
    ptr, col = np.asarray(P.SmNode), np.asarray(P.ReNode)
    i = P.Num_Node - 1                      # a free node; a block off the diagonal, so that its inverse is finite
    slot = int(ptr[i] + np.nonzero(col[ptr[i]:ptr[i + 1]] != i)[0][-1])
    K[slot, 1, 2] = value
    b = torch.from_numpy(np.random.default_rng(nrhs).standard_normal((3 * P.Num_Node, nrhs))).cuda()
    S = F.DeviceSystem(M, K=K, F=b[:, 0])
    U, st = S.solve(F=b if nrhs > 1 else b[:, 0], rtol=1e-10, mixed=mixed)
    assert st["status"] == _lib.FEM_ERR_BREAKDOWN
    assert not U.any()
    assert not mixed or st["relres"] == 1.0
