"""Device topology where its kernels change path: rows of up to 8 incident elements (sorted in
registers), of 9 to 128 (in shared memory), rows of more than 32 and 64 blocks, an unaligned
slot_map; every array bit-exact against the host build."""
import ctypes

import numpy as np
import pytest
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from tests.test_gpu_topology import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("valence", [1, 3, 7, 8, 9, 16, 17, 40, 128])
def test_node_shared_by_many_elements(valence):
    """`valence` elements around node 0, their other corners drawn at random (rows of 2 .. ~150
    blocks, repeated nodes among them)."""
    rng = np.random.default_rng(valence)
    n = min(3 * valence + 20, 200)   # a block row holds at most 256 blocks
    conn = np.stack([np.concatenate([[0], rng.choice(np.arange(1, n), 7, replace=False)]) for _ in range(valence)])
    if valence > 2:
        conn[1, 5] = conn[1, 4]
    conn = conn[:, rng.permutation(8)].astype(np.int32)
    P = F.Physics(np.arange(1, n + 1), rng.random((n, 3)), conn.T.astype(np.int64), [], [])
    _check(P)


def test_unaligned_slot_map():
    P = F.hex_block(5, 4, 3, seed=1)
    L, d = _lib.load(), "cuda"
    N, E = P.Num_Node, P.Num_Elem
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(d)  # noqa: E731
    conn, nep, nel, ip, ix = t(P.conn), t(P.ne_ptr), t(P.ne_list), t(P.SmNode), t(P.ReNode)
    ws = torch.empty(int(L.fem_topology_workspace_bytes(N, E)), dtype=torch.uint8, device=d)
    inv = torch.empty(8 * E, dtype=torch.int32, device=d)
    buf = torch.empty(64 * E + 8, dtype=torch.uint8, device=d)
    p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    nnzb = ctypes.c_int64(0)
    co = torch.empty(N, dtype=torch.int32, device=d)
    _lib.check(L.fem_topology_count_gpu(N, E, p(conn), p(nep), p(nel), p(co), p(ip), ctypes.byref(nnzb), p(ws),
                                        ws.numel(), st), "count")
    _lib.check(L.fem_topology_fill_gpu(N, E, p(conn), p(nep), p(nel), p(ip), p(ix), p(inv), p(buf[3:]), p(ws),
                                       ws.numel(), st), "fill")
    assert np.array_equal(buf[3:3 + 64 * E].cpu().numpy(), P.slot_map)
    assert np.array_equal(inv.cpu().numpy(), P.ne_inv)
