"""Tangent / secant kernel at the edges of its tiles (8 elements per block, 4 per warp), with
element counts off every multiple, a wedge-degenerate element and large displacement gradients,
against the oracle.  Tolerance per scalar row: 1e-12 x the row's largest entry (the records between
the two kernels carry 48 bits: 2^-48 x ~64 contributions < 1e-12)."""
import numpy as np
import pytest

import fem_taichi_gb300 as F
from oracle import fem_oracle as O
from tests.fixtures import STEEL
from tests.test_gpu_assembly import assert_K_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 1), (5, 1, 1), (7, 1, 1), (2, 2, 2), (3, 3, 1), (17, 1, 1),
                                   (3, 11, 1)])
@pytest.mark.parametrize("amplitude", [0.03, 0.6])
def test_element_counts_off_the_tile(shape, amplitude):
    P = F.hex_block(*shape, jitter=0.1, seed=7, twist_deg=20, fix="xmin")
    P.Bounds[0][1] = [0, -1, 0]
    U = np.random.default_rng(1).uniform(-amplitude, amplitude, size=(P.Num_Node, 3))
    M = F.Model("t", P, STEEL)
    M.LDinit(U.reshape(-1))
    KT, KM = M.Get_MatrixKN()
    KTo, KMo = O.OracleModel(P, STEEL).Get_MatrixKN(U)
    assert_K_close(KT, KTo)
    assert_K_close(KM, KMo)


def test_bsr_and_csr_orders_hold_the_same_values():
    P = F.hex_block(4, 3, 3, jitter=0.1, seed=3, fix="zmin")
    M = F.Model("t", P, STEEL)
    M.LDinit(np.random.default_rng(2).uniform(-0.05, 0.05, size=3 * P.Num_Node))
    bsr = M.assemble_tangent(k_layout="bsr")
    csr = M.Get_MatrixKN()
    ptr, col = np.asarray(P.SmNode), np.asarray(P.ReNode)
    for V, A in zip(bsr, csr):
        V = V.cpu().numpy()
        for i in (0, P.Num_Node // 2, P.Num_Node - 1):
            for k in range(ptr[i], ptr[i + 1]):
                j = col[k]
                assert np.array_equal(V[k], A[3 * i:3 * i + 3, 3 * j:3 * j + 3].toarray())


def test_repeated_corner_node():
    """A wedge: two corners of one element are the same node."""
    b = F.mesh.block_arrays(3, 2, 1, jitter=0.0, seed=0, fix="zmin")
    elem = b["elem"].copy()
    elem[6, 1] = elem[5, 1]
    P = F.Physics(b["ids"], b["xyz"], elem, b["bounds"], [])
    U = np.random.default_rng(4).uniform(-0.02, 0.02, size=(P.Num_Node, 3))
    M = F.Model("w", P, STEEL)
    M.LDinit(U.reshape(-1))
    KT, KM = M.Get_MatrixKN()
    KTo, KMo = O.OracleModel(P, STEEL).Get_MatrixKN(U)
    assert_K_close(KT, KTo)
    assert_K_close(KM, KMo)
