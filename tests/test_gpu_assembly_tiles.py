"""FP64 element kernels at the edges of their tiles (a warp per element up to 16 elements an SM, 16
elements a block beyond) and where one takes over from the other: element counts off every multiple, the parts of a split assembly, far from the origin, an inverted element; K, M and F
against the oracle with the suite's tolerances (1e-12 of the row's / vector's largest entry)."""
import numpy as np
import pytest

import fem_taichi_gb300 as F
from oracle import fem_oracle as O
from tests.fixtures import STEEL
from tests.test_gpu_assembly import assert_K_close, assert_vec_close

pytestmark = pytest.mark.gpu


def _check(P, om=(30.0, -20.0, 80.0), **kw):
    M = F.Model("t", P, STEEL, Omegas=om, **kw)
    OM = O.OracleModel(P, STEEL, om)
    assert_K_close(M.Get_MatrixKL(), OM.Get_MatrixKL())
    assert_vec_close(M.Get_MatrixM().data, OM.Get_MatrixM().data)
    assert_vec_close(M.Get_VectorF(), OM.Get_VectorF())
    return M


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 1), (5, 1, 1), (15, 1, 1), (4, 4, 1), (17, 1, 1), (3, 11, 1), (7, 9, 1)])
def test_element_counts_off_the_tile(shape):
    _check(F.hex_block(*shape, jitter=0.1, seed=4, twist_deg=30, fix="xmin"))


@pytest.mark.parametrize("extra", [-1, 0, 1, 17])
def test_where_the_kernels_meet(extra):
    """16 x (SMs) elements and a few more or fewer, as a chain of bars of one element's section."""
    import torch
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    _check(F.hex_block(n, 1, 1, size=(float(n), 1.0, 1.0), jitter=0.0, seed=4, twist_deg=90, fix="xmin"))


@pytest.mark.parametrize("shape", [(9, 7, 5), (31, 13, 7)])
@pytest.mark.parametrize("parts", [1, 3, 50])
def test_parts_off_the_tile(shape, parts):
    P = F.hex_block(*shape, jitter=0.1, seed=4, origin=(500.0, -200.0, 0.0), fix="zmin")
    M = _check(P)
    K, Mm, Fv = M.assemble_host(n_parts=parts)
    K1, M1, F1 = M.assemble(k_layout="csr", m_layout="csr")
    assert np.array_equal(K, K1.cpu().numpy()) and np.array_equal(Mm, M1.cpu().numpy())
    assert np.array_equal(Fv, F1.reshape(-1).cpu().numpy())


def test_inverted_element_keeps_its_sign():
    """An element listed inside out has det < 0 at every Gauss point: its K, M and F enter negated."""
    P1 = F.hex_block(3, 2, 2, jitter=0.1, seed=4, fix="zmin")
    conn = P1.conn.copy()
    conn[5] = conn[5][[4, 5, 6, 7, 0, 1, 2, 3]]
    _check(F.Physics(P1.Node[0], P1.xyz, conn.T.astype(np.int64), P1.Bounds, []))
