"""The forward's pre-activation stores: staged 16-byte rows where z1 and z2 allow it, single floats
where a caller's buffers do not start on 16 bytes -- the same values, at node counts off the 32-node
rows and the 128-node tiles, and nothing written past the last node."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import mlp_oracle as MO
from tests.test_gpu_learned import _random_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 31, 33, 127, 128, 129, 1000])
def test_aligned_and_unaligned_buffers_agree(n):
    net, _ = _random_net(3)
    Xf = MO.bf16_round(np.random.default_rng(n).standard_normal((n, 16)).astype(np.float32))
    X = torch.from_numpy(MO.bf16_bits(Xf).view(np.int16)).cuda()
    out, z1, z2 = net.forward(X, save=True)
    b1, b2 = (torch.full((64 * n + 64,), 7.0, device="cuda") for _ in range(2))
    out2 = torch.empty_like(out)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    mlp = net.net()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert net.lib.fem_mlp_forward(ctypes.byref(mlp), X.data_ptr(), n, out2.data_ptr(), b1[1:].data_ptr(),
                                   b2[3:].data_ptr(), err.data_ptr(), st) == 0
    assert int(err.item()) == 0
    assert torch.equal(out, out2)
    assert torch.equal(b1[1:1 + 64 * n].view(n, 64), z1) and torch.equal(b2[3:3 + 64 * n].view(n, 64), z2)
    assert float(b1[0]) == 7.0 and bool((b1[1 + 64 * n:] == 7.0).all()) and bool((b2[3 + 64 * n:] == 7.0).all())
