"""Element stiffness of the FP64 assembly against extended precision, both element kernels, several
materials and shapes.  Disjoint elements, so that a block of K is one element's and nothing is
summed.  A block's value is eight terms of products of two rounded factors: 1.5 to 1.85 x 10^-16 rms is
what rounding noise alone gives for these elements (an emulation of the kernel's arithmetic, 16
materials); a constant or table entry that is off in one direction adds to that (2.0 to 2.5 x 10^-16)."""
import numpy as np
import pytest

import fem_taichi_gb300 as F

pytestmark = pytest.mark.gpu

L = np.longdouble
SX = np.array([1, -1, -1, 1, 1, -1, -1, 1], L)
SY = np.array([1, 1, -1, -1, 1, 1, -1, -1], L)
SZ = np.array([-1] * 4 + [1] * 4, L)
GS1 = L(0.57735026918962)


def _exact(x, EX, PO):
    """K of elements with corners x (n, 8, 3): (n, 8, 8, 3, 3)."""
    EX, PO = L(EX), L(PO)
    lam, mu = EX * PO / (1 + PO) / (1 - 2 * PO), EX / 2 / (1 + PO)
    K = 0
    for a in (-GS1, GS1):
        for b in (-GS1, GS1):
            for c in (-GS1, GS1):
                fx, fy, fz = 1 + a * SX, 1 + b * SY, 1 + c * SZ
                dn = np.stack([SX * fy * fz, fx * SY * fz, fx * fy * SZ], 1) / 8
                J = np.einsum("eai,ad->eid", x - x[:, :1], dn)
                A = np.stack([np.cross(J[:, 1], J[:, 2]), np.cross(J[:, 2], J[:, 0]), np.cross(J[:, 0], J[:, 1])], 2)
                det = (J[:, 0] * A[:, :, 0]).sum(-1)
                R = np.einsum("ad,edi->eai", dn, A)
                P = np.einsum("eap,ebq->eabpq", R, R) / det[:, None, None, None, None]
                K = K + lam * P + mu * P.swapaxes(-1, -2) + mu * np.einsum("eabrr->eab", P)[..., None, None] * np.eye(3, dtype=L)
    return K


# 2,600 elements: above the size up to which a warp takes an element
@pytest.mark.parametrize("n", [120, 2600])
@pytest.mark.parametrize("EX,PO,stretch", [(200000.0, 0.3, 1.0), (200000.0, 0.3, 2.7), (200000.0, 0.3, 4.0),
                                           (70000.0, 0.33, 1.0), (150000.0, 0.347, 3.4), (193000.0, 0.26, 3.5)])
def test_rounding_noise_only(n, EX, PO, stretch):
    rng = np.random.default_rng(7)
    base = np.stack([(SX + 1) / 2, (SY + 1) / 2, (SZ + 1) / 2 * stretch], 1).astype(float)
    x = base + rng.uniform(-0.1, 0.1, (n, 8, 3)) + 500.0 * rng.random((n, 1, 3))
    P = F.Physics(np.arange(1, 8 * n + 1), x.reshape(-1, 3), np.arange(8 * n).reshape(n, 8).T.astype(np.int64),
                  [[np.array([0]), [-1, -1, -1]]])   # nothing held
    M = F.Model("e", P, dict(DE=7.8e-9, EX=EX, PO=PO), algo="fp64")
    K, _, _ = M.assemble(K=True, M=False, F=False)
    m = 120
    K = K.cpu().numpy()[:64 * m].reshape(m, 8, 8, 3, 3)   # rows and columns of an element in corner order
    want = _exact(x[:m].astype(L), EX, PO)
    rms = float(np.sqrt(((K - want) ** 2).sum() / (want ** 2).sum()))
    assert rms <= 1.9e-16
