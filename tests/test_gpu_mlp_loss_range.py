"""Loss of many probes with large residuals: the sum of a node's squares passes FP32's largest number long
before one square does, and counts as FP64 does.  The residuals are prescribed (identity blocks, no
product), so the loss is a sum of exact squares; its bound is 60 roundings of 2^-53."""
import ctypes

import numpy as np
import pytest
import torch

from fem_taichi_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [113, 114, 128, 341, 1000])
@pytest.mark.parametrize("scale", [1e-11, 1.0, 3e17, 5.7e17, 9.9e17, 1.8e19])
def test_many_probes(R, scale):
    lib = _lib.load()
    n = 70
    rng = np.random.default_rng(R)
    z = (scale * rng.choice([-1.0, 1.0], (n, 3, R)) * rng.uniform(0.9, 1.0, (n, 3, R))).astype(np.float32)
    out, y, zd = (torch.from_numpy(a).cuda() for a in (np.zeros((n, 16), np.float32), np.zeros_like(z), z))
    d = torch.empty((n, 16), dtype=torch.float32, device="cuda")
    part, k = torch.empty(1024, dtype=torch.float64, device="cuda"), ctypes.c_int(0)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.fem_mlp_loss_grad(out.data_ptr(), y.data_ptr(), zd.data_ptr(), R, n, d.data_ptr(), part.data_ptr(),
                                 ctypes.byref(k), st) == 0
    got = float(part[:k.value].sum())
    want = float((z.astype(np.longdouble) ** 2).sum())
    assert abs(got - want) <= 60 * 2.0 ** -53 * want
