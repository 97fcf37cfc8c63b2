"""Device multigrid setup against the host setup, bit for bit, where its kernels change path: rows
shorter and longer than a warp's 32 sorted entries, rows beyond the shared-memory sort (1,024),
vectors shorter than and off the 256-element sum chunks, few and many coarse rows, small and
large aggregates."""
import types

import numpy as np
import pytest
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from fem_taichi_gb300.solve import AmgHierarchy, FEM_F64
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu


def _same(Hd, Hh, levels):
    ld, lh = Hd.levels(), Hh.levels()
    assert len(ld) == len(lh) >= levels
    for l, (a, b) in enumerate(zip(ld, lh)):
        assert {k: v for k, v in a.items() if k != "setup_s"} == {k: v for k, v in b.items() if k != "setup_s"}, l
        whats = [0] if l else []
        if l + 1 < len(ld):
            whats += [1, 2, 4, 6]
        for what in whats + [3]:
            x, y = Hd.export(l, what), Hh.export(l, what)
            for p, q in zip(x, y) if isinstance(x, tuple) else [(x, y)]:
                assert np.array_equal(p, q), (l, what)


@pytest.mark.parametrize("shape,stretch,opts", [
    ((3, 2, 2), 1.0, dict(max_coarse=20)),                       # 36 nodes: one partial chunk
    ((20, 18, 9), 4.0, dict(max_coarse=60)),                     # stretched: coarse rows of more than 64 blocks
    ((20, 18, 9), 4.0, dict(max_coarse=60, theta=0.0)),          # everything strong: the largest aggregates
    ((17, 5, 5), 1.0, dict(max_coarse=60, theta=0.25)),          # nothing strong: no coarse level
    ((26, 24, 6), 1.0, dict(max_coarse=100, smooth=0)),          # unsmoothed prolongator
])
def test_mesh_hierarchies(shape, stretch, opts):
    P = F.hex_block(*shape, size=(shape[0], shape[1], shape[2] * stretch), jitter=0.1, seed=6, fix="zmin")
    S = F.DeviceSystem(F.Model("b", P, STEEL))
    Hd, Hh = S.amg_variant(setup="device", **opts), S.amg_variant(setup="host", **opts)
    _same(Hd, Hh, 1 if opts.get("theta") == 0.25 else 2)
    Hd.close()
    Hh.close()


def test_rows_beyond_the_shared_memory_sort():
    """1,100 nodes in a line, every row full: neighbours couple strongly, the rest weakly."""
    n = 1100
    rng = np.random.default_rng(3)
    B = rng.standard_normal((n, n, 3, 3)) * 1e-4
    for i in range(n - 1):
        B[i, i + 1] -= np.diag([1.0, 0.7, 0.4])
    B = B + B.transpose(1, 0, 3, 2)
    B[np.arange(n), np.arange(n)] = np.diag([2.6, 2.1, 1.5]) + 0.01
    xyz = np.stack([np.arange(n), 0.1 * rng.standard_normal(n), 0.1 * rng.standard_normal(n)], 1).astype(float)
    ptr = (np.arange(n + 1) * n).astype(np.int32)
    col = np.tile(np.arange(n, dtype=np.int32), n)
    d = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in
         dict(ptr=ptr, col=col, val=B.reshape(-1), xyz=xyz).items()}
    S = types.SimpleNamespace(
        lib=_lib.load(), n=n, nnzb=n * n, device=torch.device("cuda"),
        stream=torch.cuda.current_stream().cuda_stream,
        A64=_lib.FemBsr(n, n * n, d["ptr"].data_ptr(), d["col"].data_ptr(), d["val"].data_ptr(), FEM_F64,
                        _lib.LAYOUT_BSR),
        model=types.SimpleNamespace(mesh=types.SimpleNamespace(xyz=d["xyz"]),
                                    Physics=types.SimpleNamespace(SmNode=ptr, ReNode=col)))
    opts = dict(max_coarse=600)
    Hd = AmgHierarchy.on_device(S, **opts)
    Hh = AmgHierarchy(S.lib, n, ptr, col, B.reshape(-1), xyz, **opts)
    _same(Hd, Hh, 2)
    Hd.close()
    Hh.close()
