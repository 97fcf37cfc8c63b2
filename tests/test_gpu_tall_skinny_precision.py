"""Rounding error of W = Q C: no larger than a sum over 32 lanes and a butterfly leaves (rms error of the
sum over its rms, random terms, by emulation: 1.00, 1.22, 1.33, 1.45 and 1.52 x 10^-16 for 8, 33, 100, 190
and 256 columns; 5 % for the sample).  One chain of additions would leave 1.0, 1.9, 3.3, 4.6 and 5.3."""
import ctypes

import numpy as np
import pytest
import torch

from fem_taichi_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,bound", [(8, 1.00e-16), (33, 1.22e-16), (100, 1.33e-16), (190, 1.45e-16), (256, 1.52e-16)])
@pytest.mark.parametrize("b", [3, 10, 16, 32])
def test_rms_error(m, bound, b):
    L, n = _lib.load(), 8000 // b
    g = torch.Generator(device="cuda")
    g.manual_seed(m + b)
    Q, C = (torch.randn(s, dtype=torch.float64, device="cuda", generator=g) for s in ((n, m), (m, b)))
    W = torch.empty((n, b), dtype=torch.float64, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(L.fem_ts_gemm_nn(n, m, b, Q.data_ptr(), m, C.data_ptr(), b, 1.0, 0.0, W.data_ptr(), b, st), "nn")
    q, c = Q.cpu().numpy().astype(np.longdouble), C.cpu().numpy().astype(np.longdouble)
    want = np.stack([(q * c[:, k]).sum(1) for k in range(b)], 1)
    err = W.cpu().numpy() - want
    assert np.sqrt((err ** 2).sum() / (want ** 2).sum()) <= 1.05 * bound
