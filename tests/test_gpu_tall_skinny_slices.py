"""W = Q C where the launch changes shape: row counts either side of the three rules (two warps a row group, one
or two columns a warp), odd and even column counts, column counts of Q around the tiles the two
warps take in turn.  A row's sum is the same tree whichever way, so the bits do not depend on how many
columns are asked for or how many rows there are."""
import ctypes

import pytest
import torch

from fem_taichi_gb300 import _lib

pytestmark = pytest.mark.gpu


def _nn(Q, C, W, alpha=1.0, beta=0.0):
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().fem_ts_gemm_nn(Q.shape[0], Q.shape[1], C.shape[1], Q.data_ptr(), Q.stride(0), C.data_ptr(),
                                          C.stride(0), alpha, beta, W.data_ptr(), W.stride(0), st), "nn")


@pytest.mark.parametrize("m", [1, 8, 32, 33, 64, 65, 96, 190, 256])
def test_same_bits_in_every_shape(m):
    parts = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    n = 32 * 9 * parts + 5          # one column already takes the widest form
    Q = torch.randn((n, m), dtype=torch.float64, device="cuda", generator=g)
    C = torch.randn((m, 32), dtype=torch.float64, device="cuda", generator=g)
    ref = torch.empty((n, 32), dtype=torch.float64, device="cuda")
    _nn(Q, C, ref)
    for b in (1, 2, 9, 10):
        for k in (0.05, 1.74, 1.76, 3.99, 4.01, 8.01):     # warps per sub-partition
            rows = min(n, max(1, int(k * parts / b) * 32 - 3))
            W = torch.full((rows, b + 1), 7.0, dtype=torch.float64, device="cuda")
            _nn(Q[:rows], C[:, :b], W)
            assert torch.equal(W[:, :b], ref[:rows, :b]) and bool((W[:, b] == 7.0).all()), (b, k)
