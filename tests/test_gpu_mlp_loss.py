"""Loss and its gradient against FP64 on the host, in both access widths (probe counts that are and are
not multiples of 4, buffers off a 16-byte boundary) and where the residuals leave the range in which
their squares are summed in pairs of floats.  The loss sums FP64-exact squares of FP32 residuals: each
residual carries about 8 roundings of 2^-24 of the largest of its terms, so the bound is taken from
those terms; the gradient's is 40 roundings of the terms of its entry."""
import ctypes

import numpy as np
import pytest
import torch

from fem_taichi_gb300 import _lib

pytestmark = pytest.mark.gpu


def _run(out, y, z, R, shift=0):
    lib = _lib.load()
    n = out.shape[0]

    def dev(a):
        t = torch.empty(a.size + 4, dtype=torch.float32, device="cuda")
        v = t[shift:shift + a.size]
        v.copy_(torch.from_numpy(a.reshape(-1)))
        return v
    o, yd, zd, d = dev(out), dev(y), dev(z), dev(np.full((n, 16), 7, np.float32))
    part, k = torch.empty(1024, dtype=torch.float64, device="cuda"), ctypes.c_int(0)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.fem_mlp_loss_grad(o.data_ptr(), yd.data_ptr(), zd.data_ptr(), R, n, d.data_ptr(), part.data_ptr(),
                                 ctypes.byref(k), st) == 0
    return float(part[:k.value].sum()), d.cpu().numpy().reshape(n, 16)


def _host(out, y, z):
    """y, z: (n, 3, R)."""
    o, y, z = (a.astype(np.float64) for a in (out, y, z))
    L = np.zeros((len(o), 3, 3))
    for k, (r, c) in enumerate([(0, 0), (1, 1), (2, 2), (1, 0), (2, 0), (2, 1)]):
        L[:, r, c] = np.exp(o[:, k]) if k < 3 else o[:, k]
    C = L @ L.transpose(0, 2, 1)
    e = C @ y - z
    mag = np.abs(L) @ np.abs(L).transpose(0, 2, 1) @ np.abs(y) + np.abs(z)
    G, Gm = 2 * e @ y.transpose(0, 2, 1), 2 * mag @ np.abs(y).transpose(0, 2, 1)
    S, Sm = G + G.transpose(0, 2, 1), Gm + Gm.transpose(0, 2, 1)
    dL, dLm = S @ L, Sm @ np.abs(L)
    R = y.shape[2]
    pick = lambda A, f: np.stack([A[:, 0, 0] * f(0), A[:, 1, 1] * f(1), A[:, 2, 2] * f(2), A[:, 1, 0], A[:, 2, 0],
                                  A[:, 2, 1]], 1) / (len(o) * R)
    ex = lambda k: np.exp(o[:, k])
    u = 2.0 ** -24
    return (e ** 2).sum(), (2 * np.abs(e) * 8 * u * mag + (8 * u * mag) ** 2).sum(), pick(dL, ex), 40 * u * pick(dLm, ex)


@pytest.mark.parametrize("R", [1, 3, 4, 8, 12])
@pytest.mark.parametrize("n", [1, 255, 257, 1000])
def test_loss_and_gradient(n, R):
    rng = np.random.default_rng(n + R)
    out = (0.3 * rng.standard_normal((n, 16))).astype(np.float32)
    y, z = (rng.standard_normal((n, 3, R)).astype(np.float32) for _ in range(2))
    loss, tol, grad, gtol = _host(out, y, z)
    for shift in (0, 1, 2):
        got, d = _run(out, y, z, R, shift)
        assert abs(got - loss) <= tol
        assert (np.abs(d[:, :6] - grad) <= gtol).all()
        assert (d[:, 6:] == 0).all()


@pytest.mark.parametrize("scale", [1e-22, 1e-14, 1e-9, 1e17, 1e19])
def test_small_and_large_residuals(scale):
    """Squares below and above FP32's exponents count as FP64 does."""
    n, R = 300, 8
    rng = np.random.default_rng(5)
    out = (0.3 * rng.standard_normal((n, 16))).astype(np.float32)
    y, z = ((scale * rng.standard_normal((n, 3, R))).astype(np.float32) for _ in range(2))
    loss, tol, _, _ = _host(out, y, z)
    got, _ = _run(out, y, z, R)
    assert abs(got - loss) <= tol


def test_not_finite():
    n, R = 40, 8
    out = np.zeros((n, 16), np.float32)
    y, z = np.ones((n, 3, R), np.float32), np.zeros((n, 3, R), np.float32)
    z[7, 1, 3] = np.inf
    assert _run(out, y, z, R)[0] == np.inf
    z[7, 1, 3] = np.nan
    assert np.isnan(_run(out, y, z, R)[0])
