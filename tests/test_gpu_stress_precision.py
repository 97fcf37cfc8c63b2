"""Principal stresses of the FP64 node kernel against extended precision, from the kernel's own averaged
components.  The kernel finds the eigenvectors in FP32; its error is to be no larger than that of an
FP64 Jacobi iteration, whose rms over such fields is 1.03 x 10^-16 of the tensor's largest entry (1.25
for entries that are independent normals, the bound here)."""
import numpy as np
import pytest

import fem_taichi_gb300 as F
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu

L = np.longdouble


def _principal(c):
    """Descending eigenvalues of (n, 6) components xx, yy, zz, xy, yz, xz by cyclic Jacobi rotations."""
    A = c.astype(L)[:, [0, 3, 5, 3, 1, 4, 5, 4, 2]].reshape(-1, 3, 3).copy()
    for _ in range(10):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            e = A[:, p, q].copy()
            on = np.abs(e) > 1e-40 * np.abs(A).max(axis=(1, 2))
            th = (A[:, q, q] - A[:, p, p]) / 2 / np.where(on, e, 1)
            t = np.where(on, np.where(th < 0, -1, 1) / (np.abs(th) + np.sqrt(1 + th * th)), 0)
            k = 1 / np.sqrt(1 + t * t)
            x, y = A[:, p, r].copy(), A[:, q, r].copy()
            A[:, p, p] -= t * e
            A[:, q, q] += t * e
            A[:, p, q] = A[:, q, p] = 0
            A[:, p, r] = A[:, r, p] = k * x - t * k * y
            A[:, q, r] = A[:, r, q] = t * k * x + k * y
    return -np.sort(-np.stack([A[:, 0, 0], A[:, 1, 1], A[:, 2, 2]], 1), axis=1)


@pytest.mark.parametrize("field", ["random", "bending"])
def test_error_of_principal_values(field):
    P = F.hex_block(13, 11, 9, size=(13.0, 11.0, 18.0), jitter=0.1, seed=4, twist_deg=20, fix="zmin")
    if field == "random":
        u = np.random.default_rng(5).uniform(-1e-3, 1e-3, (P.Num_Node, 3))
    else:
        x = P.xyz
        u = 1e-4 * np.stack([x[:, 2] ** 2, 0.3 * x[:, 0] * x[:, 1], -2 * x[:, 0] * x[:, 2]], 1)
    S = F.Post("p", P, STEEL, u).Get_Stress()
    p = _principal(S[:, :6])
    size = np.abs(S[:, :6]).max(axis=1, keepdims=True)
    assert np.sqrt((((S[:, 6:9] - p) / size) ** 2).mean()) <= 1.25e-16
    vm = np.sqrt((p[:, 0] - p[:, 1]) ** 2 + 2 * (p[:, 1] - p[:, 2]) ** 2)
    # the differences of two such values, and three roundings
    assert np.sqrt((((S[:, 9] - vm) / size[:, 0]) ** 2).mean()) <= 3 * 1.25e-16
