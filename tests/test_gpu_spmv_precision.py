"""Rounding error of the padded FP32 product against FP64: no larger than with the products of a block summed
and then added to the row's sum, which left (rms over the rms of y, this mesh and this x) 7.35, 7.71, 7.73,
7.47, 8.49 and 10.4 x 10^-8 for 1, 2, 4, 8, 16 and 32 right-hand sides.  One chain of products over a lane's
slots leaves 8.4."""
import ctypes

import pytest
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs,bound", [(1, 7.35e-8), (2, 7.71e-8), (4, 7.73e-8), (8, 7.47e-8), (16, 8.49e-8),
                                        (32, 10.4e-8)])
def test_rms_error(nrhs, bound):
    P = F.hex_block(24, 24, 12, size=(24.0, 24.0, 12.0), jitter=0.1, seed=2, fix="zmin")
    P.Bounds = [[P.Bounds[0][0], [-1, -1, -1]]]     # nothing held
    S = F.DeviceSystem(F.Model("m", P, STEEL))
    S.K32()
    g = torch.Generator("cuda").manual_seed(nrhs)
    x = 2 * torch.rand((3 * S.n, nrhs), device="cuda", generator=g) - 1
    y, x64 = torch.empty_like(x), x.double()
    y64 = torch.empty_like(x64)
    _lib.check(S.lib.fem_bsr_spmv(ctypes.byref(S.A64), nrhs, x64.data_ptr(), y64.data_ptr(), 0, S.stream), "FP64")
    for v in range(6 if nrhs == 1 else 1):          # the variants of at least eight lanes a row
        _lib.check(S.lib.fem_bsr_spmv(ctypes.byref(S._A32), nrhs, x.data_ptr(), y.data_ptr(), v, S.stream), "FP32")
        assert float(((y.double() - y64).square().sum() / y64.square().sum()).sqrt()) <= bound, v
