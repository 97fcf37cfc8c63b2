"""FP32 iteration with one right-hand side, whose sums are formed by the kernels that use them: node
counts around a warp, a CTA and the nodes all CTAs hold at once, iterations launched in any number at a
time, and every way to end -- between two launches and inside one."""
import numpy as np
import pytest
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu


def _system(shape, seed=0, sign=1.0):
    """A well-conditioned SPD matrix on a block's pattern: 4 I + couplings -1/16 (27 at most)."""
    P = F.hex_block(*shape, jitter=0.0, seed=1, fix="zmin")
    M = F.Model("s", P, STEEL)
    ip, ix = (torch.from_numpy(np.asarray(a).astype(np.int64)).cuda() for a in (P.SmNode, P.ReNode))
    row = torch.repeat_interleave(torch.arange(P.Num_Node, device="cuda"), ip[1:] - ip[:-1])
    K = torch.full((ix.numel(), 1, 1), -1 / 16, dtype=torch.float64, device="cuda") * torch.eye(3, dtype=torch.float64, device="cuda")
    K[row == ix] = 4 * torch.eye(3, dtype=torch.float64, device="cuda")
    g = torch.Generator("cuda").manual_seed(seed)
    b = torch.randn(3 * P.Num_Node, dtype=torch.float64, device="cuda", generator=g)
    return F.DeviceSystem(M, K=(sign * K).contiguous(), F=b), b


def _relres(S, U, b):
    return float(torch.linalg.norm(b - S.spmv(U)) / torch.linalg.norm(b))


# 8 nodes; 27; 256 and 264 (one CTA's 8 warps, the next); more than 2 nodes for every thread of 152 CTAs
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 2, 2), (63, 1, 1), (65, 1, 1), (31, 7, 3), (160, 100, 20)])
def test_solves(shape):
    S, b = _system(shape)
    U, st = S.solve(rtol=1e-12)
    assert st["status"] == 0 and _relres(S, U, b) <= 1.01e-12


def test_iterations_launched_together_do_not_matter():
    S, b = _system((20, 15, 9))
    ref, s0 = S.solve(rtol=1e-12, unroll=16)
    for unroll, graph in ((1, True), (2, False), (3, True), (7, False), (64, True)):
        U, st = S.solve(rtol=1e-12, unroll=unroll, use_graph=graph)
        assert torch.equal(U, ref) and st["iterations"] == s0["iterations"] and st["outer"] == s0["outer"]


@pytest.mark.parametrize("cap", [1, 2, 7, 8, 9, 16])
def test_iteration_cap(cap):
    """Short of convergence, an inner solve takes exactly its cap, whether a launch ends there or not."""
    P = F.hex_block(12, 9, 7, jitter=0.1, seed=3, fix="zmin", load_face="zmax", load=(0, 0, -1))
    S = F.DeviceSystem(F.Model("c", P, STEEL))
    U, st = S.solve(rtol=1e-12, inner_rtol=1e-9, inner_maxit=cap, max_outer=1, unroll=8)
    V, s1 = S.solve(rtol=1e-12, inner_rtol=1e-9, inner_maxit=cap, max_outer=1, unroll=1)
    assert st["status"] != 0 and st["iterations"] == s1["iterations"] == cap and torch.equal(U, V)


def test_zero_load_and_indefinite_matrix():
    S, b = _system((9, 5, 3))
    U, st = S.solve(F=torch.zeros_like(b), rtol=1e-12)
    assert st["status"] == 0 and st["iterations"] == 0 and not U.any()
    S, b = _system((9, 5, 3), sign=-1.0)
    assert S.solve(rtol=1e-12)[1]["status"] == _lib.FEM_ERR_NOT_SPD
