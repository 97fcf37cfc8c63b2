"""Principal stresses of the FP64 node kernel where its eigenvalue iteration changes path: equal and
nearly equal principal values, diagonal and plane states, magnitudes at and beyond the FP32
range, and element counts off the element kernel's tile.  One element per state: the nodes of a
uniform gradient all carry the same tensor.

Tolerances: p1 >= p2 >= p3 within 2e-14 of the tensor's largest entry against numpy's eigvalsh of
the kernel's own averaged components (both are backward stable; the iteration's measured error is
3e-15); components within the suite's 1e-10 per node of the oracle."""
import numpy as np
import pytest

import fem_taichi_gb300 as F
from oracle import fem_oracle as O
from tests.fixtures import STEEL

pytestmark = pytest.mark.gpu

LAM = STEEL["EX"] * STEEL["PO"] / (1 + STEEL["PO"]) / (1 - 2 * STEEL["PO"])
MU = STEEL["EX"] / 2 / (1 + STEEL["PO"])


def _strain(sig):
    """Symmetric strain whose stress is sig."""
    tr = np.trace(sig)
    return (sig - LAM / (3 * LAM + 2 * MU) * tr * np.eye(3)) / (2 * MU)


def _states():
    rng = np.random.default_rng(2)
    Q = np.linalg.qr(rng.standard_normal((3, 3)))[0]
    base = {"uniaxial": [1, 0, 0], "biaxial": [1, 1, 0], "hydrostatic": [1, 1, 1], "pure shear": [1, 0, -1],
            "near": [1, 1 + 1e-7, 1 - 3e-7], "graded": [1e4, 1, 1e-4], "general": [0.7, -0.2, 0.1]}
    out = []
    for name, d in base.items():
        for scale in (1.0, 1e-25, 1e25, 3.7e8):
            out.append((f"{name} x {scale:g}", scale * (Q * np.array(d, float)) @ Q.T))
            out.append((f"{name} axes x {scale:g}", scale * np.diag(np.array(d, float))))
    plane = np.array([[1.0, 0.4, 0], [0.4, -0.3, 0], [0, 0, 0]])
    out += [("plane", plane), ("zero", np.zeros((3, 3))), ("tiny off", np.diag([1.0, 2.0, 3.0]) + 1e-12)]
    return out


def test_principal_values_of_prescribed_states():
    states = _states()
    n = len(states)
    P1 = F.hex_block(1, 1, 1, fix=None)
    xyz = np.concatenate([P1.xyz + [3.0 * k, 0, 0] for k in range(n)])
    elem = np.concatenate([P1.conn + 8 * k for k in range(n)]).T
    P = F.Physics(np.arange(1, 8 * n + 1), xyz, elem)
    u = np.concatenate([(P1.xyz) @ _strain(s).T for _, s in states])
    S = F.Post("p", P, STEEL, u).Get_Stress()
    c = S[:, :6]
    T = np.stack([c[:, [0, 3, 5]], c[:, [3, 1, 4]], c[:, [5, 4, 2]]], 1)
    ref = np.linalg.eigvalsh(T)[:, ::-1]
    scale = np.abs(T).max(axis=(1, 2))
    for k in range(8 * n):
        assert np.all(np.abs(S[k, 6:9] - ref[k]) <= 2e-14 * scale[k]), (states[k // 8][0], S[k, 6:9], ref[k])
    assert np.all(S[:, 6] >= S[:, 7]) and np.all(S[:, 7] >= S[:, 8])
    vm = np.sqrt((S[:, 6] - S[:, 7]) ** 2 + 2 * (S[:, 7] - S[:, 8]) ** 2)
    assert np.all(np.abs(S[:, 9] - vm) <= 1e-14 * scale)


def test_infinite_and_nan_displacements_stay_not_finite():
    P = F.hex_block(3, 1, 1, fix=None)
    u = np.random.default_rng(0).uniform(-1e-3, 1e-3, (P.Num_Node, 3))
    u[0, 0], u[3, 1] = np.inf, np.nan
    S = F.Post("p", P, STEEL, u).Get_Stress()
    touched = np.zeros(P.Num_Node, bool)
    for e in P.conn:
        if not np.isfinite(u[e]).all():
            touched[e] = True
    assert np.all(np.isnan(S[touched][:, 6:])) and np.all(np.isfinite(S[~touched]))


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 1), (5, 3, 1), (17, 1, 1), (11, 3, 1)])
@pytest.mark.parametrize("mode", ["aliased", "written"])
def test_element_counts_off_the_tile(shape, mode):
    P = F.hex_block(*shape, jitter=0.1, seed=8, twist_deg=25, origin=(500.0, 0, 0), fix=None)
    u = np.random.default_rng(1).uniform(-1e-3, 1e-3, (P.Num_Node, 3))
    S = F.Post("p", P, STEEL, u, gmat_mode=mode).Get_Stress()
    So = O.oracle_stress(P, STEEL, u, gmat_mode=mode)
    assert np.all(np.abs(S - So) <= 1e-10 * np.abs(So).max(axis=1, keepdims=True))
