"""The single-load FP32 solve while another stream holds the SMs, so that its CTAs start at different
times: the same bits and the same number of iterations as alone, whatever the launches' timing."""
import pytest
import torch

import fem_taichi_gb300 as F
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 7, 5), (40, 30, 12)])
def test_same_bits_beside_another_stream(shape):
    P = F.hex_block(*shape, jitter=0.1, seed=3, fix="zmin", load_face="zmax", load=(0, 0, -1))
    S = F.DeviceSystem(F.Model("c", P, STEEL))
    ref, s0 = S.solve(rtol=1e-11, unroll=4)
    assert s0["status"] == 0
    side = torch.cuda.Stream()
    a = torch.randn(1 << 24, device="cuda")
    for n in (1 << 14, 1 << 18, 1 << 24):
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            for _ in range(400):
                a[:n].mul_(1.0)
        U, st = S.solve(rtol=1e-11, unroll=4)
        assert torch.equal(U, ref) and st["iterations"] == s0["iterations"] and st["outer"] == s0["outer"]
    torch.cuda.synchronize()
