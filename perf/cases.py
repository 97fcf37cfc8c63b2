"""The workloads this package's speed is judged by: assembly, stress recovery, products with K,
static solves, the large-displacement tangent, the topology build, the modal solve's
reorthogonalisation and one training step of the learned preconditioner, each through the
entry point a program calls.

A case names a ``kind`` and its sizes; meshes are jittered structured hex blocks of the sizes
the package's configurations use (and odd ones), steel, with the centrifugal load.
"""
from __future__ import annotations

import copy
import ctypes

import numpy as np
import torch

import fem_taichi_gb300 as F
from fem_taichi_gb300 import _lib
from fem_taichi_gb300.learned import LearnedPreconditioner, NodeData, N_HID, N_IN, N_OUT, N_PARAMS
from fem_taichi_gb300.mesh import build_topology_gpu

OMEGA = (10.0, -20.0, 100.0)
GS1 = 0.57735026918962
NRHS = (1, 2, 4, 8, 16, 32)


def listed():
    return [
        # K, M and F of a small part on the device: a Newton or design loop's smallest call,
        # where launches and latency count
        dict(name="assemble-small", kind="assemble", nx=8, ny=8, nz=4, stretch=1.0, twist=0.0, fixed=True,
             algo="fp64", layout="bsr"),
        # K, M and F of the 1 M-node block on the device, no supports (a modal or an own-constraint
        # user): the largest ordinary assembly
        dict(name="assemble-large", kind="assemble", nx=200, ny=200, nz=24, stretch=1.0, twist=0.0, fixed=False,
             algo="fp64", layout="bsr"),
        # the reference's getters, host arrays in its CSR order, of a ragged mid-size part
        dict(name="getters-mid", kind="getters", nx=83, ny=61, nz=19, stretch=1.0, twist=20.0, fixed=False,
             algo="fp64"),
        # nodal stresses of the 1 M-node block from a displacement field
        dict(name="stress-large", kind="stress", nx=200, ny=200, nz=24, stretch=1.0, twist=0.0, algo="fp64",
             gmat="aliased"),
        # K X for 32 load cases in FP64: residuals of batched solves, Lanczos blocks
        dict(name="product-32", kind="product", nx=96, ny=80, nz=17, stretch=1.0, fp32=False, nrhs=32),
        # the reference's static solve, whole call, on the 4:1 stretched 214 k-node block
        dict(name="static-whole", kind="static", nx=100, ny=100, nz=20, stretch=4.0, precond="bj"),
        # the same part solved with the multigrid preconditioner, setup included
        dict(name="static-whole-amg", kind="static", nx=100, ny=100, nz=20, stretch=4.0, precond="amg"),
        # 32 load cases of a kept system in one batched solve
        dict(name="solve-32", kind="solve", nx=80, ny=80, nz=20, stretch=1.0, precond="bj", mixed=True, nrhs=32),
        # tangent and secant stiffness of one Newton step at large displacements
        dict(name="tangent-mid", kind="tangent", nx=64, ny=48, nz=15, stretch=1.0, twist=0.0, fixed=False,
             layout="bsr"),
        # block pattern, incidence and gather map of the 1 M-node block from its connectivity
        dict(name="topology-large", kind="topology", nx=200, ny=200, nz=24),
        # late reorthogonalisation of a block-Lanczos step: 21,853 nodes, 190 vectors, block of 10
        dict(name="reorth", kind="reorth", n=65559, m=190, b=10),
        # forward, loss and backward of the learned preconditioner on 214 k nodes (bf16 tensor cores)
        dict(name="train-step", kind="train", nx=100, ny=100, nz=20, stretch=1.0, probes=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def _block(rng, lo, hi, xy_max):
    """(nx, ny, nz) with lo .. hi elements in all, log-uniform, flat to cubic."""
    e = _log_int(rng, lo, hi)
    nz = max(2, min(30, int(round(e ** (1.0 / 3.0) * rng.uniform(0.3, 1.1)))))
    nx = max(2, min(xy_max, int(round((e / nz) ** 0.5 * rng.uniform(0.7, 1.4)))))
    ny = max(2, min(xy_max, e // (nx * nz)))
    return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "getters", "stress", "stress", "product", "static", "static", "solve",
                       "solve", "tangent", "topology", "reorth", "train"])
    stretch = round(rng.uniform(1.0, 4.0), 2)
    twist = rng.choice([0.0, 0.0, 15.0, 40.0])
    if kind == "assemble":
        return dict(kind=kind, **_block(rng, 60, 900000, 220), stretch=stretch, twist=twist, fixed=False,
                    algo=rng.choice(["fp64", "fp64", "fp64", "dd"]), layout=rng.choice(["bsr", "bsr", "csr"]))
    if kind == "getters":
        return dict(kind=kind, **_block(rng, 300, 90000, 120), stretch=stretch, twist=twist, fixed=False,
                    algo=rng.choice(["fp64", "fp64", "dd"]))
    if kind == "stress":
        return dict(kind=kind, **_block(rng, 60, 900000, 220), stretch=stretch, twist=twist,
                    algo=rng.choice(["fp64", "fp64", "fp64", "dd"]), gmat=rng.choice(["aliased", "aliased", "written"]))
    if kind == "product":
        return dict(kind=kind, **_block(rng, 500, 120000, 120), stretch=stretch, fp32=rng.choice([False, False, True]),
                    nrhs=rng.choice(NRHS))
    if kind == "static":
        return dict(kind=kind, **_block(rng, 2000, 120000, 110), stretch=round(rng.uniform(1.0, 3.0), 2),
                    precond=rng.choice(["bj", "amg"]))
    if kind == "solve":
        return dict(kind=kind, **_block(rng, 2000, 90000, 90), stretch=round(rng.uniform(1.0, 2.0), 2),
                    precond=rng.choice(["bj", "bj", "amg"]), mixed=rng.choice([True, True, False]),
                    nrhs=rng.choice(NRHS))
    if kind == "tangent":
        return dict(kind=kind, **_block(rng, 60, 45000, 70), stretch=stretch, twist=twist, fixed=False,
                    layout=rng.choice(["bsr", "csr"]))
    if kind == "topology":
        return dict(kind=kind, **_block(rng, 60, 900000, 220))
    if kind == "reorth":
        return dict(kind=kind, n=3 * _log_int(rng, 700, 21000), m=rng.randint(8, 190), b=rng.randint(1, 10))
    return dict(kind="train", **_block(rng, 2000, 190000, 110), stretch=stretch, probes=rng.choice([4, 8]))


# ---- inputs -----------------------------------------------------------------------------------
def _mesh(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    P = F.hex_block(nx, ny, nz, size=(float(nx), float(ny), nz * case.get("stretch", 1.0)), jitter=0.1, seed=seed,
                    twist_deg=case.get("twist", 0.0), fix="zmin", load_face="zmax", load=(0, 0, -1))
    if not case.get("fixed", True):
        P.Bounds = [[P.Bounds[0][0], [-1, -1, -1]]]   # no DOF of the group is held
    return P


def _loads(P, seed, nrhs):
    """(3N, nrhs): seeded random tractions on the top face, N(0, 1) per component and node."""
    rng = np.random.default_rng(seed)
    L = np.zeros((P.Num_Node, 3, nrhs))
    top = P.Forces[0][0]
    L[top] = rng.standard_normal((top.size, 3, nrhs))
    return torch.from_numpy(L.reshape(3 * P.Num_Node, nrhs)).cuda()


def _uniform(shape, seed, scale):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return scale * (2.0 * torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) - 1.0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "reorth":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        n, m, b = case["n"], case["m"], case["b"]
        Q = torch.randn((n, m), dtype=torch.float64, device="cuda", generator=g) / n ** 0.5
        X = torch.randn((n, b), dtype=torch.float64, device="cuda", generator=g)
        L = _lib.load()
        ws = torch.empty(int(L.fem_ts_gemm_tn_workspace_bytes(n, m, b)), dtype=torch.uint8, device="cuda")
        return dict(kind=kind, lib=L, n=n, m=m, b=b, Q=Q, X=X, W=X.clone(), ws=ws)
    if kind == "topology":
        P = _mesh(dict(case, stretch=1.0), 0)
        conn = np.ascontiguousarray(np.roll(P.conn, (7919 * seed) % P.Num_Elem, axis=0))   # elements in another order
        return dict(kind=kind, conn=conn, n=P.Num_Node)
    P = _mesh(case, seed)
    if kind == "stress":
        u = _uniform((P.Num_Node, 3), seed + 1, 1e-3)
        return dict(kind=kind, P=P, u=u, post=F.Post("part", P, F.STEEL, u, gmat_mode=case["gmat"], algo=case["algo"]))
    M = F.Model("part", P, F.STEEL, Omegas=OMEGA, algo=case.get("algo", "fp64"))
    s = dict(kind=kind, P=P, model=M, case=case)
    if kind == "product":
        s["system"] = F.DeviceSystem(M, *_free_K(M, P))
        s["x"] = _uniform((3 * P.Num_Node, case["nrhs"]), seed + 1, 1.0)
        if case["fp32"]:
            s["x"] = s["x"].float()
    elif kind == "solve":
        s["system"] = F.DeviceSystem(M)
        s["F"] = _loads(P, seed + 1, case["nrhs"])
        if case["precond"] == "amg":
            s["system"].amg()
    elif kind == "tangent":
        s["u"] = _uniform((P.Num_Node, 3), seed + 1, 0.03)
        M.LDinit(s["u"].cpu().numpy())
    elif kind == "train":
        S = F.DeviceSystem(M)
        s["data"] = NodeData(S, n_probes=case["probes"], seed=seed)
        s["net"] = LearnedPreconditioner(seed=seed)
        p = np.random.default_rng(seed).standard_normal(N_PARAMS)
        p[:N_HID * N_IN] *= N_IN ** -0.5
        p[N_HID * N_IN:N_PARAMS - N_OUT * (N_HID + 1)] *= 0.1
        p[N_PARAMS - N_OUT * (N_HID + 1):] *= 0.02          # a few hundred steps into the training
        s["net"].load_state_dict({"params": p.astype(np.float32)})
    return s


def _free_K(M, P):
    """K without held DOFs (penalty entries of 1e20 would hide every other value), and F."""
    held, M.fixed = M.fixed, torch.zeros_like(M.fixed)
    K, _, Fv = M.assemble(K=True, M=False, F=True)
    M.fixed = held
    return K, Fv


# ---- one pass ---------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "assemble":
        K, M, Fv = s["model"].assemble(k_layout=s["case"]["layout"], m_layout=s["case"]["layout"])
        return dict(K=K, M=M, F=Fv)
    if kind == "getters":
        m = s["model"]
        K, M, Fv = m.Get_MatrixKL(), m.Get_MatrixM(), m.Get_VectorF()
        return dict(K=K.data, M=M.data, F=Fv)
    if kind == "stress":
        return s["post"].stress_device()
    if kind == "product":
        return s["system"].spmv(s["x"], fp32=s["case"]["fp32"], nrhs=s["case"]["nrhs"])
    if kind == "static":
        solver = F.Static_solver(s["model"])
        if s["case"]["precond"] == "bj":
            return solver.Solve_cpu()
        return solver.Solve_gpu(rtol=1e-12, precond="amg")
    if kind == "solve":
        c = s["case"]
        U, _ = s["system"].solve(F=s["F"], rtol=1e-12, mixed=c["mixed"],
                                 precond="amg" if c["precond"] == "amg" else None)
        return U
    if kind == "tangent":
        KT, KM = s["model"].assemble_tangent(k_layout=s["case"]["layout"])
        return dict(KT=KT, KM=KM)
    if kind == "topology":
        return build_topology_gpu(s["conn"], s["n"])
    if kind == "reorth":
        C = torch.empty((s["m"], s["b"]), dtype=torch.float64, device="cuda")
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(s["lib"].fem_ts_gemm_tn(s["n"], s["m"], s["b"], s["Q"].data_ptr(), s["m"], s["X"].data_ptr(),
                                           s["b"], C.data_ptr(), s["b"], s["ws"].data_ptr(), s["ws"].numel(), st),
                   "fem_ts_gemm_tn")
        _lib.check(s["lib"].fem_ts_gemm_nn(s["n"], s["m"], s["b"], s["Q"].data_ptr(), s["m"], C.data_ptr(), s["b"],
                                           -1.0, 1.0, s["W"].data_ptr(), s["b"], st), "fem_ts_gemm_nn")
        return dict(C=C, W=s["W"])
    net, d = s["net"], s["data"]
    out, z1, z2 = net.forward(d.X, save=True)
    loss, dout = net.loss_and_grad(d, out)
    return dict(out=out, loss=loss, grad=net.backward(d.X, z1, z2, dout))


# ---- what a pass cannot do without --------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "reorth":
        n, m, b = case["n"], case["m"], case["b"]
        return {"bytes": 8.0 * (n * m + 3 * n * b + m * b), "flops": 4.0 * n * m * b}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    E = float(nx * ny * nz)
    N = float((nx + 1) * (ny + 1) * (nz + 1))
    B = float((3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1))    # 3x3 blocks of K
    mesh = 24 * N + 32 * E + 4 * (N + B)                       # coordinates, connectivity, pattern
    if kind == "assemble":
        full = case["layout"] == "csr"
        return {"bytes": mesh + 72 * B + (24 if full else 8) * B + 24 * N, "flops": 7500 * E}
    if kind == "getters":
        return {"bytes": mesh + 96 * B + 24 * N, "flops": 7500 * E}
    if kind == "stress":
        return {"bytes": 24 * N + 32 * E + 24 * N + 80 * N, "flops": 2400 * E + 300 * N}
    if kind == "product":
        v = 4 if case["fp32"] else 8
        return {"bytes": 9 * v * B + 4 * (B + N) + 2 * 3 * N * v * case["nrhs"], "flops": 18 * B * case["nrhs"]}
    if kind == "tangent":
        return {"bytes": mesh + 24 * N + 144 * B, "flops": 30000 * E}
    if kind == "topology":
        return {"bytes": 32 * E + 4 * (3 * N + B) + (32 + 32 + 64) * E, "flops": 0}
    if kind == "train":
        return {"bytes": N * (2 * N_IN + 4 * N_OUT + 24 * case["probes"]),
                "flops": 6 * N * (N_IN * N_HID + N_HID * N_HID + N_HID * N_OUT)}
    # solves: the iterations of one right-hand side grow like the diameter of the block; block Jacobi
    # takes about 12 products with the FP32 matrix per element across the longest side, multigrid 60 in all
    it = 60 if case["precond"] == "amg" else 12 * max(nx, ny) * case["stretch"] ** 0.5
    r = case.get("nrhs", 1)
    return {"bytes": it * (40 * B + 24 * N * r), "flops": it * 18 * B * r}


# ---- the same outputs in 64 bits, without this package's kernels --------------------------------
_SX = torch.tensor([1., -1, -1, 1, 1, -1, -1, 1], dtype=torch.float64)
_SY = torch.tensor([1., 1, -1, -1, 1, 1, -1, -1], dtype=torch.float64)
_SZ = torch.tensor([-1., -1, -1, -1, 1, 1, 1, 1], dtype=torch.float64)


def _shape(dev):
    """N (8, 8) and dN/dxi (8, 8, 3) at the Gauss points (zeta fastest) per corner."""
    s = (-GS1, GS1)
    pts = torch.tensor([[a, b, c] for a in s for b in s for c in s], dtype=torch.float64)
    fx, fy, fz = 1 + pts[:, :1] * _SX, 1 + pts[:, 1:2] * _SY, 1 + pts[:, 2:] * _SZ
    d = torch.stack([_SX * fy * fz, fx * _SY * fz, fx * fy * _SZ], -1)
    return (0.125 * fx * fy * fz).to(dev), (0.125 * d).to(dev)


def _geometry(x, dN):
    """dN/dx (e, 8 points, 8 corners, 3) and det of elements with corner coordinates x (e, 8, 3)."""
    J = torch.einsum("eai,gad->egid", x - x[:, :1], dN)
    c = torch.linalg.cross
    a0 = c(J[..., 1, :], J[..., 2, :])
    a1 = c(J[..., 2, :], J[..., 0, :])
    a2 = c(J[..., 0, :], J[..., 1, :])
    det = (J[..., 0, :] * a0).sum(-1)
    inv = torch.stack([a0, a1, a2], -1) / det[..., None, None]       # inv[d, i] = d xi_d / d x_i
    return torch.einsum("gad,egdi->egai", dN, inv), det


def _constants():
    E, nu = F.STEEL["EX"], F.STEEL["PO"]
    return F.STEEL["DE"], E * nu / (1 + nu) / (1 - 2 * nu), E / 2 / (1 + nu)


def _linear(G, det):
    """sum_g det (lam g_a g_b^T + mu g_b g_a^T + mu g_a.g_b I): (e, 8, 8, 3, 3)."""
    _, lam, mu = _constants()
    P = torch.einsum("egap,egbq,eg->eabpq", G, G, det)
    return lam * P + mu * P.transpose(-1, -2) + mu * P.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] * torch.eye(
        3, dtype=G.dtype, device=G.device)


def _tangent(G, det, u):
    """Tangent and secant blocks at corner displacements u (e, 8, 3); the stress of the geometric
    term is summed over the Gauss points so far and not reset (as the reference does)."""
    _, lam, mu = _constants()
    I = torch.eye(3, dtype=G.dtype, device=G.device)
    e = G.shape[0]
    KT = torch.zeros((e, 8, 8, 3, 3), dtype=G.dtype, device=G.device)
    KM = torch.zeros_like(KT)
    S = torch.zeros((e, 3, 3), dtype=G.dtype, device=G.device)
    for g in range(8):
        a, w = G[:, g], det[:, g]
        T = torch.einsum("eck,ecd->ekd", u, a)
        Fg = I + T
        strain = 0.5 * (T + T.transpose(1, 2) + T.transpose(1, 2) @ T)
        S = S + lam * strain.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None] * I + 2 * mu * strain
        X = torch.einsum("eap,ebq->eabpq", a, a)
        X = lam * X + mu * X.transpose(-1, -2) + mu * (a @ a.transpose(1, 2))[..., None, None] * I
        Y = Fg[:, None, None] @ X * w[:, None, None, None, None]
        Z = Y @ T.transpose(1, 2)[:, None, None]
        geo = w[:, None, None] * (a @ S @ a.transpose(1, 2))
        KT += Y + Z + geo[..., None, None] * I
        KM += Y + 0.5 * Z
    return KT, KM


def _pattern(conn, n):
    """Sorted block keys row * n + column, their block-row pointer, and each element's slots."""
    key = (conn[:, :, None] * n + conn[:, None, :]).reshape(-1)
    uniq = torch.unique(key)
    ptr = torch.searchsorted(uniq, torch.arange(n + 1, device=conn.device) * n)
    return uniq, ptr


def _to_csr(V, uniq, ptr, n):
    """Blocks (nnzb, r, c) in the scalar row order: row r of a block row holds its blocks' row r."""
    row = uniq // n
    rs, L = ptr[row], ptr[row + 1] - ptr[row]
    r, c = V.shape[1], V.shape[2]
    k = torch.arange(uniq.numel(), device=uniq.device)
    out = torch.empty(V.numel(), dtype=V.dtype, device=V.device)
    for p in range(r):
        for q in range(c):
            out[r * c * rs + p * c * L + c * (k - rs) + q] = V[:, p, q]
    return out


def _blocks(case, P, which, u=None):
    """(K, M, F) or (KT, KM, None) as blocks, with the pattern; held DOFs get 1e20."""
    dev = "cuda"
    n = P.Num_Node
    x = torch.from_numpy(P.xyz).to(dev)
    conn = torch.from_numpy(P.conn.astype(np.int64)).to(dev)
    Ns, dN = _shape(dev)
    uniq, ptr = _pattern(conn, n)
    A = torch.zeros((uniq.numel(), 3, 3), dtype=torch.float64, device=dev)
    B = torch.zeros((uniq.numel(), 3, 3) if which == "tangent" else (uniq.numel(),), dtype=torch.float64, device=dev)
    Fv = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    rho = F.STEEL["DE"]
    w = torch.tensor(OMEGA, dtype=torch.float64, device=dev)
    W = (w @ w) * torch.eye(3, dtype=torch.float64, device=dev) - torch.outer(w, w)
    for e0 in range(0, conn.shape[0], 60000):
        c = conn[e0:e0 + 60000]
        slot = torch.searchsorted(uniq, (c[:, :, None] * n + c[:, None, :]).reshape(-1))
        G, det = _geometry(x[c], dN)
        if which == "tangent":
            KT, KM = _tangent(G, det, u[c])
            A.index_add_(0, slot, KT.reshape(-1, 3, 3))
            B.index_add_(0, slot, KM.reshape(-1, 3, 3))
            continue
        A.index_add_(0, slot, _linear(G, det).reshape(-1, 3, 3))
        Me = rho * torch.einsum("eg,ga,gb->eab", det, Ns, Ns)
        B.index_add_(0, slot, Me.reshape(-1))
        Fv.index_add_(0, c.reshape(-1), (Me @ (x[c] @ W)).reshape(-1, 3))
    if case.get("fixed", True):
        d = torch.searchsorted(uniq, torch.from_numpy(P.Bounds[0][0]).to(dev) * (n + 1))
        for V in (A, B) if which == "tangent" else (A,):
            for p in range(3):
                V[d, p, p] = 1e20
    if which != "tangent":
        Fv[torch.from_numpy(P.Forces[0][0]).to(dev)] += torch.tensor([0., 0., -1.], dtype=torch.float64, device=dev)
    return A, B, Fv, uniq, ptr


def _solve(A, uniq, ptr, n, Fv):
    """K U = F by block-Jacobi conjugate gradients on torch's sparse product, restarted on the true
    residual until it is about 1e-14 or stops falling."""
    row = uniq // n
    L = ptr[1:] - ptr[:-1]
    crow = torch.zeros(3 * n + 1, dtype=torch.int64, device=A.device)
    crow[1:] = torch.cumsum(torch.repeat_interleave(3 * L, 3), 0)
    cols = (3 * (uniq % n)[:, None, None] + torch.arange(3, device=A.device)).expand(-1, 3, 3)
    K = torch.sparse_csr_tensor(crow, _to_csr(cols.contiguous(), uniq, ptr, n), _to_csr(A, uniq, ptr, n),
                                size=(3 * n, 3 * n))
    Minv = torch.linalg.inv(A[torch.searchsorted(uniq, torch.arange(n, device=A.device) * (n + 1))])
    b = Fv.reshape(3 * n, -1)
    r_ = b.shape[1]
    pre = lambda r: (Minv @ r.reshape(n, 3, r_)).reshape(3 * n, r_)  # noqa: E731
    norm = b.square().sum(0).sqrt()
    U = torch.zeros_like(b)
    last = float("inf")
    for _ in range(4):
        r = b - K @ U
        now = float((r.square().sum(0).sqrt() / norm).max())
        if now < 1e-14 or now > 0.3 * last:
            break
        last = now
        d = torch.zeros_like(b)
        z = pre(r)
        p, rz, r0 = z, (r * z).sum(0), r.square().sum(0)
        for it in range(6000):
            q = K @ p
            alpha = rz / (p * q).sum(0).clamp_min(1e-300)
            d = d + alpha * p
            r = r - alpha * q
            if it % 32 == 31 and float((r.square().sum(0) / r0).max()) < 1e-18:
                break
            z = pre(r)
            new = (r * z).sum(0)
            p = z + new / rz.clamp_min(1e-300) * p
            rz = new
        U = U + d
    return U


def _silu(z):
    return z * torch.sigmoid(z)


def exact(case, seed):
    kind = case["kind"]
    if kind == "topology":
        return None
    if kind == "reorth":
        s = prepare(case, seed)
        C = s["Q"].T @ s["X"]
        return dict(C=C, W=s["X"] - s["Q"] @ C)
    if kind == "train":
        return _exact_train(prepare(case, seed))
    P = _mesh(case, seed)
    n = P.Num_Node
    if kind == "stress":
        return _exact_stress(case, P, _uniform((n, 3), seed + 1, 1e-3))
    if kind == "tangent":
        KT, KM, _, uniq, ptr = _blocks(case, P, "tangent", _uniform((n, 3), seed + 1, 0.03))
        return dict(KT=KT, KM=KM) if case["layout"] == "bsr" else dict(KT=_to_csr(KT, uniq, ptr, n),
                                                                      KM=_to_csr(KM, uniq, ptr, n))
    K, M, Fv, uniq, ptr = _blocks(dict(case, fixed=False) if kind == "product" else case, P, "linear")
    if kind == "product":
        x = _uniform((3 * n, case["nrhs"]), seed + 1, 1.0)
        x = (x.float().double() if case["fp32"] else x).reshape(n, 3, -1)
        y = torch.zeros_like(x)
        for k0 in range(0, uniq.numel(), 1 << 20):
            u = uniq[k0:k0 + (1 << 20)]
            y.index_add_(0, u // n, K[k0:k0 + (1 << 20)] @ x[u % n])
        return y.reshape(3 * n, -1)
    if kind in ("static", "solve"):
        return _solve(K, uniq, ptr, n, Fv if kind == "static" else _loads(P, seed + 1, case["nrhs"])).reshape(
            (3 * n,) if kind == "static" else (3 * n, case["nrhs"]))
    M3 = M[:, None, None].expand(-1, 3, 1)
    if kind == "getters":
        return dict(K=_to_csr(K, uniq, ptr, n).cpu().numpy(), M=_to_csr(M3, uniq, ptr, n).cpu().numpy(),
                    F=Fv.reshape(-1).cpu().numpy())
    if case["layout"] == "csr":
        return dict(K=_to_csr(K, uniq, ptr, n), M=_to_csr(M3, uniq, ptr, n), F=Fv)
    return dict(K=K, M=M, F=Fv)


def _exact_stress(case, P, u):
    dev = "cuda"
    _, lam, mu = _constants()
    n = P.Num_Node
    x = torch.from_numpy(P.xyz).to(dev)
    conn = torch.from_numpy(P.conn.astype(np.int64)).to(dev)
    _, dN = _shape(dev)
    corner = [[a, b, c] for a in (-1, 1) for b in (-1, 1) for c in (-1, 1)]
    at = torch.tensor(corner if case["gmat"] == "written" else [corner[6 + (j & 1)] for j in range(8)],
                      dtype=torch.float64) / GS1
    Wt = (0.125 * (1 + at[:, :1] * _SX) * (1 + at[:, 1:2] * _SY) * (1 + at[:, 2:] * _SZ)).to(dev)
    S = torch.zeros((n, 6), dtype=torch.float64, device=dev)
    cnt = torch.zeros(n, dtype=torch.float64, device=dev)
    for e0 in range(0, conn.shape[0], 120000):
        c = conn[e0:e0 + 120000]
        G, _ = _geometry(x[c], dN)
        ue = u[c]
        H = torch.einsum("eak,egad->egkd", ue - ue[:, :1], G)
        tr = lam * H.diagonal(dim1=2, dim2=3).sum(-1)
        sg = torch.stack([tr + 2 * mu * H[..., 0, 0], tr + 2 * mu * H[..., 1, 1], tr + 2 * mu * H[..., 2, 2],
                          mu * (H[..., 0, 1] + H[..., 1, 0]), mu * (H[..., 1, 2] + H[..., 2, 1]),
                          mu * (H[..., 0, 2] + H[..., 2, 0])], -1)
        S.index_add_(0, c.reshape(-1), torch.einsum("jg,egc->ejc", Wt, sg).reshape(-1, 6))
        cnt.index_add_(0, c.reshape(-1), torch.ones(c.numel(), dtype=torch.float64, device=dev))
    S = S / cnt[:, None]
    T = S[:, [0, 3, 5, 3, 1, 4, 5, 4, 2]].reshape(n, 3, 3)
    p = torch.linalg.eigvalsh(T.cpu()).to(dev).flip(1) if n < 40000 else _eig3(T)
    vm = ((p[:, 0] - p[:, 1]).square() + 2 * (p[:, 1] - p[:, 2]).square()).sqrt()
    return torch.cat([S, p, vm[:, None]], 1)


def _eig3(A):
    """Eigenvalues, descending, of symmetric 3x3 matrices by cyclic Jacobi rotations."""
    A = A.clone()
    for _ in range(10):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            apq = A[:, p, q].clone()
            th = 0.5 * (A[:, q, q] - A[:, p, p]) / torch.where(apq == 0, torch.ones_like(apq), apq)
            t = torch.where(th < 0, -1.0, 1.0) / (th.abs() + (1 + th * th).sqrt())
            t = torch.where(apq == 0, torch.zeros_like(t), t)
            c = (1 + t * t).rsqrt()
            s = t * c
            x, y = A[:, p, r].clone(), A[:, q, r].clone()
            A[:, p, p] -= t * apq
            A[:, q, q] += t * apq
            A[:, p, q] = A[:, q, p] = 0.0
            A[:, p, r] = A[:, r, p] = c * x - s * y
            A[:, q, r] = A[:, r, q] = s * x + c * y
    return A.diagonal(dim1=1, dim2=2).sort(1, descending=True).values


def _exact_train(s):
    net, d = s["net"], s["data"]
    p = net.params.double().requires_grad_(True)
    o, parts = 0, []
    for shape in ((N_HID, N_IN), (N_HID,), (N_HID, N_HID), (N_HID,), (N_OUT, N_HID), (N_OUT,)):
        k = int(np.prod(shape))
        v = p[o:o + k].view(shape)
        if len(shape) == 2:      # the products take bf16 weights; the gradient is that of the rounded weights
            v = v + (v.detach().to(torch.bfloat16).double() - v.detach())
        parts.append(v)
        o += k
    W1, b1, W2, b2, W3, b3 = parts
    x = d.X.view(torch.bfloat16).double()
    h = _silu(_silu(x @ W1.T + b1) @ W2.T + b2)
    out = h @ W3.T + b3
    z0 = torch.zeros_like(out[:, 0])
    L = torch.stack([out[:, 0].exp(), z0, z0, out[:, 3], out[:, 1].exp(), z0, out[:, 4], out[:, 5], out[:, 2].exp()],
                    1).reshape(-1, 3, 3)
    e = L @ (L.transpose(1, 2) @ d.yhat.double()) - d.zhat.double()
    loss = e.square().sum() / (d.n * d.R)
    loss.backward()
    g = copy.copy(p.grad)
    return dict(out=out.detach(), loss=loss.detach(), grad=g)
