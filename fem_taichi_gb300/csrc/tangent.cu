// Large-displacement tangent and secant stiffness (Get_MatrixKN, FEM_model_bsr.py:134-145;
// UnitK :476-515, InslocalBN :544-592, MatrixS :517-525), FP64.
//
// With T = grad u, Fd = I + T and a_j = grad N_j at a Gauss point, the strain operators of
// InslocalBN are B1 + BN1 and B2 + BN2 = the linear ones with Fd^T applied to the node's
// displacement, so UnitK's products collapse to vectors pushed forward by Fd, A_j = Fd a_j:
//   (B+BN)_j^T D (B+BN)_k   = lam A_j A_k^T + mu A_k A_j^T + mu (a_j.a_k) Fd Fd^T
//   (B+BN)_j^T D (B+BN/2)_k = 1/2 [the above + lam A_j a_k^T + mu A_k a_j^T + mu (a_j.a_k) Fd]
// KT adds the geometric term (a_j . S a_k) I, S the second Piola-Kirchhoff stress of the Green
// strain T + T^T + T^T T, summed over the Gauss points so far and never reset (UnitK does the
// same: S of Gauss point g holds the points before it).
//
// k_hex8_tangent: 8 threads per element, an element's threads in one warp (no block barrier).
//   phase A (thread = Gauss point g): Jacobian and displacement gradient from trilinear
//     coefficients, T, Fd, S (prefix sum over the 8 lanes), and per corner a_j, A_j,
//     mu det a_j, mu det A_j, det S a_j into shared memory;
//   phase B (thread = corner pair j <= k): the five sums over g above, both matrices' blocks (j, k)
//     and (k, j), written as float pairs into the row-ordered chunks the double-float gather reads.
// Bound by the FP64 pipe (about 2,900 FP64 instructions per thread, conversions included).  The
// direct 3x3x3 products of UnitK, every (j, k, g) with its structural zeros, were about 16,000:
// KT and KM of 64 x 48 x 15 elements 15.25 -> 2.28 ms, the two gathers (0.21 ms) included.  The 28
// off-diagonal pairs are 3.5 per thread: the last four are shared by two threads, four Gauss points
// each, instead of idling half the lanes of a fourth round.
// Both matrices are then gathered (atomic-free, fixed order) with the penalty applied.
#include "fem_common.cuh"

namespace fem {
namespace {

constexpr int kEpcT = 8;
constexpr int kThreadsT = kEpcT * 8;
constexpr int kChunkT = 84;  // float pairs per (element, corner) chunk: 8 blocks x 10 + F 3 + pad
// Shared doubles per (Gauss point, corner): a, A, mu det a, mu det A, det S a.  An odd row keeps
// 8 corners in 8 different bank pairs; 8 more doubles per element move the second element of a
// half warp to the other 8.
constexpr int kRowT = 15;
constexpr int kElemT = 64 * kRowT + 8;

struct TangentParams {
    const double* xyz;
    const int4* conn4;
    const double* u;
    const int32_t* ne_inv;
    int64_t n_elem;
    float2* recT;
    float2* recM;
    double D0d, lam, mu;
    double lm;  // lam / mu = 2 PO / (1 - 2 PO)
    double dnr[8][8][3];
};

struct TangentSmem {
    double v[kEpcT][kElemT];
    double q[kEpcT][8][15];   // Fd Fd^T (00, 11, 22, 01, 02, 12), Fd (row-major)
    double cf[kEpcT][8][6];   // Walsh sums of the coordinates and displacements
    double dnr[8][25];
};

__device__ __forceinline__ float2 split(double x) {
    const float hi = __double2float_rn(x);
    return make_float2(hi, __double2float_rn(x - double(hi)));
}

// Block as 9 float pairs + a zero pair at dst (16-byte aligned).
__device__ __forceinline__ void split_block(const double (&v)[9], float2 (&w)[10]) {
#pragma unroll
    for (int i = 0; i < 9; ++i) w[i] = split(v[i]);
    w[9] = make_float2(0.f, 0.f);
}
template <bool kTranspose>
__device__ __forceinline__ void store_block(float2* dst, const float2 (&w)[10]) {
    float4* d = reinterpret_cast<float4*>(dst);
    auto at = [](int i) { return kTranspose && i < 9 ? 3 * (i % 3) + i / 3 : i; };
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const float2 x = w[at(2 * i)], y = w[at(2 * i + 1)];
        d[i] = make_float4(x.x, x.y, y.x, y.y);
    }
}

// The sums over Gauss points of one corner pair (j, k).
struct PairSums {
    double p1[9];   // sum mu det A_j A_k^T
    double pjk[9];  // sum mu det A_j a_k^T
    double pkj[9];  // sum mu det A_k a_j^T
    double sb[6];   // sum mu det (a_j.a_k) Fd Fd^T
    double sf[9];   // sum mu det (a_j.a_k) Fd
    double geo;     // sum det a_j . S a_k
};

template <bool kDiag>
__device__ __forceinline__ void pair_sums(const TangentSmem& s, int el, int j, int k, int g0, int ng, PairSums& r) {
#pragma unroll
    for (int i = 0; i < 9; ++i) r.p1[i] = r.pjk[i] = r.pkj[i] = r.sf[i] = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) r.sb[i] = 0.0;
    r.geo = 0.0;
#pragma unroll 1
    for (int g = g0; g < g0 + ng; ++g) {
        const double* vj = s.v[el] + (g * 8 + j) * kRowT;
        const double* vk = s.v[el] + (g * 8 + k) * kRowT;
        const double* q = s.q[el][g];
        const double ak[3] = {vk[0], vk[1], vk[2]};
        const double sc = fma(vj[8], ak[2], fma(vj[7], ak[1], vj[6] * ak[0]));   // mu det a_j . a_k
        r.geo = fma(vj[14], ak[2], fma(vj[13], ak[1], fma(vj[12], ak[0], r.geo)));
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const double Aj = vj[3 + p], Ak = vk[3 + p];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (!kDiag || c >= p) r.p1[3 * p + c] = fma(Aj, vk[9 + c], r.p1[3 * p + c]);
                r.pjk[3 * p + c] = fma(Aj, vk[6 + c], r.pjk[3 * p + c]);
                if (!kDiag) r.pkj[3 * p + c] = fma(Ak, vj[6 + c], r.pkj[3 * p + c]);
            }
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) r.sb[i] = fma(sc, q[i], r.sb[i]);
#pragma unroll
        for (int i = 0; i < 9; ++i) r.sf[i] = fma(sc, q[6 + i], r.sf[i]);
    }
}

// KT_jk, KM_jk and KM_kj of a pair (KT_kj is KT_jk transposed); lm = lam / mu.
template <bool kDiag>
__device__ __forceinline__ void pair_blocks(const PairSums& r, double lm, double (&KT)[9], double (&KM)[9],
                                            double (&KMt)[9]) {
    const double B[9] = {r.sb[0], r.sb[3], r.sb[4], r.sb[3], r.sb[1], r.sb[5], r.sb[4], r.sb[5], r.sb[2]};
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int i = 3 * p + c, t = 3 * c + p;
            if (kDiag) {
                const double x = c >= p ? r.p1[i] : r.p1[t];
                KT[i] = fma(lm, x, x + B[i]);
            } else {
                KT[i] = fma(lm, r.p1[i], r.p1[t] + B[i]);
            }
        }
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int i = 3 * p + c, t = 3 * c + p;
            if (kDiag) {
                KM[i] = 0.5 * (KT[i] + fma(lm, r.pjk[i], r.pjk[i] + r.sf[i]));
            } else {
                KM[i] = 0.5 * (KT[i] + fma(lm, r.pjk[i], r.pkj[i] + r.sf[i]));
                KMt[i] = 0.5 * (KT[t] + fma(lm, r.pkj[i], r.pjk[i] + r.sf[i]));
            }
        }
    KT[0] += r.geo;
    KT[4] += r.geo;
    KT[8] += r.geo;
}

// Off-diagonal pair q of 28 (j < k, row-major).
__device__ __forceinline__ void offdiag_pair(int q, int& j, int& k) {
    int a = 0, rem = q;
    while (rem >= 7 - a) {
        rem -= 7 - a;
        ++a;
    }
    j = a;
    k = a + 1 + rem;
}

__global__ void __launch_bounds__(kThreadsT) k_hex8_tangent(const TangentParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TangentSmem& s = *reinterpret_cast<TangentSmem*>(smem_raw);
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, el = tid >> 3, t = tid & 7;
    const int64_t e_raw = int64_t(blockIdx.x) * kEpcT + el;
    const bool valid = e_raw < p.n_elem;
    const int64_t e = valid ? e_raw : p.n_elem - 1;   // the lanes of absent elements repeat the last one
    for (int i = tid; i < 192; i += kThreadsT) s.dnr[i / 24][i % 24] = (&p.dnr[0][0][0])[i];
    const int64_t pos = __ldg(p.ne_inv + 8 * e + t);
    double c[6];
    {
        const int64_t node = __ldg(reinterpret_cast<const int*>(p.conn4) + 8 * e + t);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            c[i] = __ldg(p.xyz + 3 * node + i);
            c[3 + i] = __ldg(p.u + 3 * node + i);
        }
    }
    const int corner0 = tid & 24;  // lane of the element's corner 0
#pragma unroll
    for (int i = 0; i < 6; ++i) c[i] -= __shfl_sync(full, c[i], corner0);   // gradients need differences only
    // Walsh sums over the 8 corners, W_s = sum_a (-1)^popc(s & a) v_a on lane s.  With xi, eta, zeta
    // negative at corners {1,2,5,6}, {2,3,6,7}, {0,1,2,3}, the trilinear coefficients are xi: W_3,
    // eta: W_2, zeta: -W_4, xi eta: W_1, eta zeta: -W_6, xi zeta: -W_7, xi eta zeta: -W_5 (all / 8).
#pragma unroll
    for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double o = __shfl_xor_sync(full, c[i], m);
            c[i] = o + flip_sign(c[i], t & m);
        }
    const double eighth = (t & 4) ? -0.125 : 0.125;
#pragma unroll
    for (int i = 0; i < 6; ++i) s.cf[el][t][i] = eighth * c[i];
    __syncthreads();  // the shape table is shared by the two warps

    // ---- phase A: Gauss point g = t -----------------------------------------------------------
    {
        const int g = t;
        const double xi = (g & 4) ? kGS1 : -kGS1, et = (g & 2) ? kGS1 : -kGS1, ze = (g & 1) ? kGS1 : -kGS1;
        double J[3][3], G[3][3];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double c1 = s.cf[el][3][i], c2 = s.cf[el][2][i], c3 = s.cf[el][4][i], c4 = s.cf[el][1][i];
            const double c5 = s.cf[el][6][i], c6 = s.cf[el][7][i], c7 = s.cf[el][5][i];
            double* d = i < 3 ? J[i] : G[i - 3];
            const double m = fma(xi, c7, c5);
            d[0] = fma(ze, fma(et, c7, c6), fma(et, c4, c1));
            d[1] = fma(ze, m, fma(xi, c4, c2));
            d[2] = fma(et, m, fma(xi, c6, c3));
        }
        double A[3][3];  // adjugate, then the inverse
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
                A[j][i] = J[i1][j1] * J[i2][j2] - J[i2][j1] * J[i1][j2];
            }
        const double det = J[0][0] * A[0][0] + J[1][0] * A[0][1] + J[2][0] * A[0][2];
        const double inv = 1.0 / det;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) A[i][j] *= inv;
        double T[3][3];  // T[i][d] = du_i / dx_d
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int d = 0; d < 3; ++d) T[i][d] = fma(G[i][2], A[2][d], fma(G[i][1], A[1][d], G[i][0] * A[0][d]));
        double S[6];  // xx, yy, zz, yz, xz, xy of the Green strain's stress
        {
            double E[3], gm[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const double sq = fma(T[2][m], T[2][m], fma(T[1][m], T[1][m], T[0][m] * T[0][m]));
                E[m] = fma(0.5, sq, T[m][m]);
                const int a = (m + 1) % 3, b = (m + 2) % 3;   // m = 0: yz, 1: zx, 2: xy
                gm[m] = fma(T[2][a], T[2][b], fma(T[1][a], T[1][b], fma(T[0][a], T[0][b], T[a][b] + T[b][a])));
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                S[m] = fma(p.D0d, E[m], p.lam * (E[(m + 1) % 3] + E[(m + 2) % 3]));
                S[3 + m] = p.mu * gm[m];
            }
        }
#pragma unroll
        for (int off = 1; off < 8; off <<= 1)
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const double o = __shfl_up_sync(full, S[i], off, 8);
                if (t >= off) S[i] += o;
            }
        const double md = p.mu * det;
#pragma unroll
        for (int i = 0; i < 6; ++i) S[i] *= det;
        double* q = s.q[el][g];
        double Fd[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                Fd[i][d] = i == d ? 1.0 + T[i][d] : T[i][d];
                q[6 + 3 * i + d] = Fd[i][d];
            }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const int a = i < 3 ? i : (i == 5 ? 1 : 0), b = i < 3 ? i : (i == 3 ? 1 : 2);
            q[i] = fma(Fd[a][2], Fd[b][2], fma(Fd[a][1], Fd[b][1], Fd[a][0] * Fd[b][0]));
        }
#pragma unroll 2
        for (int j = 0; j < 8; ++j) {
            double* v = s.v[el] + (g * 8 + j) * kRowT;
            const double* dn = s.dnr[g] + 3 * j;
            double a[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) a[d] = fma(dn[2], A[2][d], fma(dn[1], A[1][d], dn[0] * A[0][d]));
            const double Sa[3] = {fma(S[4], a[2], fma(S[5], a[1], S[0] * a[0])),
                                  fma(S[3], a[2], fma(S[1], a[1], S[5] * a[0])),
                                  fma(S[2], a[2], fma(S[3], a[1], S[4] * a[0]))};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double Aj = fma(Fd[d][2], a[2], fma(Fd[d][1], a[1], Fd[d][0] * a[0]));
                v[d] = a[d];
                v[3 + d] = Aj;
                v[6 + d] = md * a[d];
                v[9 + d] = md * Aj;
                v[12 + d] = Sa[d];
            }
        }
    }
    __syncwarp();

    // ---- phase B: corner pairs ---------------------------------------------------------------
    const double lm = p.lm;
    const int base = tid & 24;
    auto chunk = [&](float2* rec, int row) { return rec + __shfl_sync(full, pos, base | row) * kChunkT; };
    PairSums r;
    double KT[9], KM[9], KMt[9];
    {
        pair_sums<true>(s, el, t, t, 0, 8, r);
        pair_blocks<true>(r, lm, KT, KM, KMt);
        float2 w[10];
        split_block(KT, w);
        if (valid) store_block<false>(p.recT + pos * kChunkT + 10 * t, w);
        split_block(KM, w);
        if (valid) store_block<false>(p.recM + pos * kChunkT + 10 * t, w);
    }
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const bool shared_pair = i == 3;   // the last four pairs: two threads, four Gauss points each
        int j, k;
        offdiag_pair(shared_pair ? 24 + (t >> 1) : 8 * i + t, j, k);
        pair_sums<false>(s, el, j, k, shared_pair ? 4 * (t & 1) : 0, shared_pair ? 4 : 8, r);
        if (shared_pair) {
#pragma unroll
            for (int m = 0; m < 9; ++m) {
                r.p1[m] += __shfl_xor_sync(full, r.p1[m], 1);
                r.pjk[m] += __shfl_xor_sync(full, r.pjk[m], 1);
                r.pkj[m] += __shfl_xor_sync(full, r.pkj[m], 1);
                r.sf[m] += __shfl_xor_sync(full, r.sf[m], 1);
            }
#pragma unroll
            for (int m = 0; m < 6; ++m) r.sb[m] += __shfl_xor_sync(full, r.sb[m], 1);
            r.geo += __shfl_xor_sync(full, r.geo, 1);
        }
        pair_blocks<false>(r, lm, KT, KM, KMt);
        float2* Tj = chunk(p.recT, j) + 10 * k;
        float2* Tk = chunk(p.recT, k) + 10 * j;
        float2* Mj = chunk(p.recM, j) + 10 * k;
        float2* Mk = chunk(p.recM, k) + 10 * j;
        const bool wT = valid && !(shared_pair && (t & 1)), wM = valid && !(shared_pair && !(t & 1));
        float2 w[10];
        split_block(KT, w);
        if (wT) store_block<false>(Tj, w);
        if (wT) store_block<true>(Tk, w);
        split_block(KM, w);
        if (wM) store_block<false>(Mj, w);
        split_block(KMt, w);
        if (wM) store_block<false>(Mk, w);
    }
}

}  // namespace

int launch_gather_dd(const fem_mesh* mesh, const fem_assembly_out* out, const void* workspace, cudaStream_t st,
                     int64_t row_begin, int64_t row_end);

}  // namespace fem

using namespace fem;

extern "C" size_t fem_tangent_workspace_bytes(int64_t n_elem) {
    if (n_elem <= 0) return 0;
    return 2 * ((size_t(n_elem) * 8 * kChunkT * sizeof(float2) + 255) / 256 * 256);
}

extern "C" int fem_assemble_tangent(const fem_mesh* mesh, const fem_material* mat, const double* u, int k_layout,
                                    double* KT, double* KM, const uint8_t* fixed, void* workspace,
                                    size_t workspace_bytes, void* stream) {
    FEM_REQUIRE(mesh && mat, "mesh/mat is NULL");
    FEM_REQUIRE(mesh->n_node >= 0 && mesh->n_elem >= 0 && mesh->nnzb >= 0, "negative mesh size");
    FEM_REQUIRE(mesh->n_elem < (int64_t(1) << 28), "n_elem too large");
    FEM_REQUIRE(mat->PO > -1.0 && mat->PO < 0.5, "Poisson ratio must lie in (-1, 0.5)");
    FEM_REQUIRE(k_layout == FEM_LAYOUT_BSR || k_layout == FEM_LAYOUT_CSR, "bad k_layout");
    if (mesh->n_node == 0) return FEM_OK;
    FEM_REQUIRE(KT && KM, "KT/KM is NULL");
    FEM_REQUIRE(mesh->indptr && mesh->ne_ptr && (mesh->nnzb == 0 || mesh->indices), "pattern arrays are NULL");
    const size_t need = fem_tangent_workspace_bytes(mesh->n_elem);
    if (mesh->n_elem) {
        FEM_REQUIRE(u && mesh->xyz && mesh->conn && aligned16(mesh->conn) && mesh->ne_inv && mesh->slot_map,
                    "u/xyz/conn/ne_inv/slot_map NULL or conn misaligned");
        if (workspace_bytes < need || !workspace) {
            set_error("workspace too small: need %zu bytes", need);
            return FEM_ERR_WORKSPACE;
        }
        FEM_REQUIRE(aligned16(workspace), "workspace not 16-byte aligned");
    }
    cudaStream_t st = as_stream(stream);
    float2* recT = static_cast<float2*>(workspace);
    float2* recM = reinterpret_cast<float2*>(static_cast<unsigned char*>(workspace) + need / 2);
    if (mesh->n_elem) {
        TangentParams tp;
        tp.xyz = mesh->xyz;
        tp.conn4 = reinterpret_cast<const int4*>(mesh->conn);
        tp.u = u;
        tp.ne_inv = mesh->ne_inv;
        tp.n_elem = mesh->n_elem;
        tp.recT = recT;
        tp.recM = recM;
        const double EX = mat->EX, PO = mat->PO;
        tp.D0d = EX * (1 - PO) / (1 + PO) / (1 - 2 * PO);  // FEM_model_bsr.py:435-449
        tp.lam = EX * PO / (1 + PO) / (1 - 2 * PO);
        tp.mu = EX / 2 / (1 + PO);
        tp.lm = 2 * PO / (1 - 2 * PO);
        const ShapeTables& T = shape_tables();
        for (int g = 0; g < 8; ++g)
            for (int a = 0; a < 8; ++a)
                for (int d = 0; d < 3; ++d) tp.dnr[g][a][d] = T.dnr[g][a][d];
        const size_t smem = sizeof(TangentSmem);
        FEM_CUDA(cudaFuncSetAttribute(k_hex8_tangent, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        const int64_t blocks = (mesh->n_elem + kEpcT - 1) / kEpcT;
        k_hex8_tangent<<<unsigned(blocks), kThreadsT, smem, st>>>(tp);
        FEM_LAUNCH_CHECK("k_hex8_tangent");
    } else {
        // no element: zero chunks are never read; both outputs still come from the gather
        recT = recM = nullptr;
    }
    fem_assembly_out o{};
    o.k_layout = k_layout;
    o.m_layout = FEM_LAYOUT_BSR;
    o.fixed = fixed;
    o.algo = FEM_ALGO_DD;
    o.K = KT;
    int rc = launch_gather_dd(mesh, &o, recT, st, 0, mesh->n_node);
    if (rc) return rc;
    o.K = KM;
    return launch_gather_dd(mesh, &o, recM, st, 0, mesh->n_node);
}
