"""The element kernel of large meshes (16 elements a block; a mesh of up to 16 elements an SM takes another) with
elements that are not well-formed hexahedra: listed inside out, collapsed to a wedge or a pyramid (repeated
corners), one of them in the last, partial block; element counts off the multiple of 16, jitter, far from the
origin.  K, M and F against the oracle with the suite's tolerances."""
import numpy as np
import pytest
import torch

import fem_taichi_gb300 as F
from tests.fixtures import STEEL
from tests.test_gpu_assembly_tiles import _check

pytestmark = pytest.mark.gpu


def _block(extra=0):
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    nx = n // 63 + 1 + extra
    nx += (63 * nx) % 16 == 0
    return F.hex_block(nx, 9, 7, size=(float(nx), 9.0, 7.0), jitter=0.1, seed=4, twist_deg=20, origin=(500.0, -200.0, 0.0),
                       fix="zmin")


def _with(P, conn):
    return F.Physics(P.Node[0], P.xyz, conn.T.astype(np.int64), P.Bounds, [])


def test_elements_listed_inside_out():
    P = _block()
    conn = P.conn.copy()
    for e in (5, 16, len(conn) - 1):
        conn[e] = conn[e][[4, 5, 6, 7, 0, 1, 2, 3]]
    _check(_with(P, conn))


@pytest.mark.parametrize("extra", [0, 1])
def test_repeated_corners(extra):
    P = _block(extra)
    conn = P.conn.copy()
    last = len(conn) - 1
    for e in (7, last):                       # wedge: one face collapsed to an edge
        conn[e][[5, 4]] = conn[e][[6, 7]]
    conn[40][[4, 5, 6, 7]] = conn[40][6]      # pyramid
    conn[last - 1][3] = conn[last - 1][2]     # one repeated corner
    _check(_with(P, conn))
