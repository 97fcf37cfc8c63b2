// Hex8 K / M / F assembly for sm_103a.
//
// Two kernels, both deterministic and free of floating-point atomics:
//
//  1. k_hex8_element -- 8 threads per element, an element's threads in one warp (no block barrier
//     but for the shape table).  Thread t loads corner t; a Walsh transform over the 8 lanes gives
//     8 times the coefficients of the element's trilinear map x(xi) = sum_k c_k m_k(xi) (m = 1, xi,
//     eta, zeta, xi eta, eta zeta, xi zeta, xi eta zeta; c_k = 1/8 sum_a m_k(corner a) x_a); the powers of two
//     go into mu and DE.  Phase A: thread g handles Gauss point g (Jacobian from the coefficients --
//     a column d/dxi does not depend on xi, so the two lanes that share it split its three components
//     -- adjugate, determinant, the 8 scaled gradients R_a = dN_a/dxi . adj(J)); results are staged in
//     shared memory.  Phase B: the 36 node pairs (a <= b) are split across the 8 threads;
//     each accumulates the Gram matrix P_ab = mu sum_g R_a R_b^T / det_g and turns it into the
//     3x3 stiffness block  K_ab[p][q] = (lam/mu) P[p][q] + P[q][p],
//     K_ab[p][p] = (lam/mu + 1) P[p][p] + tr P, which equals sum_g det (B1_a^T D0 B1_b +
//     B2_a^T D1 B2_b) of the reference (FEM_model_bsr.py:262-274, 303-347) with a different
//     summation order.  The 28 off-diagonal pairs are 3.5 per thread: two threads share each of the
//     last four, four Gauss points a thread.  The consistent mass M_ab = DE sum_g det_g N_a N_b
//     (FEM_model_bsr.py:276-287) is sum-factorised: N_a(g) is a product of one 1D factor per
//     axis, so M_ab depends only on the per-axis class of (a, b) and the 8 det_g are contracted
//     axis by axis (27 classes, 114 FP64 operations per element instead of 288).  The centrifugal
//     load (FEM_model_bsr.py:229-245) is F_a = sum_g DE det_g N_a(g) W x(g); W x is linear and
//     the isoparametric map reproduces it at the Gauss points, W x(g) = sum_b N_b(g) W x_b, so
//     F_a = sum_b M_ab W x_b: the same quantity from the mass blocks, with no per-Gauss-point
//     load density.  Each element writes one 2,944-byte record: 28 off-diagonal pairs as
//     K (3x3) + M, 8 diagonal pairs as the 6 distinct values of the symmetric K + M (8-double
//     slots), 8 x F(3).  Bound by the FP64 pipe (one warp instruction per 16 cycles per SM): what
//     shuffles, sign flips and prescaled constants save shows in full.  960,000 elements: 8.85 ms with
//     a summed Jacobian per lane, lam and mu applied per block and half of a fourth round of pairs
//     idle; 7.4 ms in this form.
//
//  2. k_gather -- one warp per block row i.  Lane l owns slot l of the row (column node
//     indices[indptr[i] + l]).  The warp walks the incident (element, corner) list of
//     node i in ascending element order, and each lane adds the element block whose
//     column corner matches its column node.  The fixed order makes the sums
//     reproducible bit for bit.  The penalty (FEM_model_bsr.py:248-259) and nodal loads
//     (LoadF, :220-226) are applied in the same pass, and the row is written in either
//     the BSR block order or the reference's scalar-CSR order (FEM_model_csr.py:150-173).
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "fem_common.cuh"

namespace fem {
namespace {

constexpr int kEpc = 16;                 // elements per CTA in the element kernel
constexpr int kElemThreads = kEpc * 8;   // 8 threads per element
// Element record (FP64 kernels), 368 doubles = 2,944 bytes: for each corner a in turn, the
// diagonal pair (a, a) as the 6 distinct values of the symmetric K_aa (00, 11, 22, 01, 02, 12)
// + M_aa in an 8-double slot, then the pairs (a, b), b = a + 1..7, as K_ab (3x3) + M_ab; then
// F (8 x 3).  The blocks the 8 lanes of a row read for one incident entry, (a, a..7), stay
// contiguous; every block starts on a 16-byte boundary.
constexpr int kPairStride = 10;   // K (9) + M (1) of an off-diagonal pair
constexpr int kDiagStride = 8;    // K_aa (6) + M_aa + 1 unused
constexpr int kFOff = 8 * kDiagStride + 28 * kPairStride;  // 344: F block offset within a record
constexpr int kRec = kFOff + 24;  // 368 doubles per element record
constexpr int kRPad = 25;         // padded row (24 used) to spread smem banks

// record offset of pair (lo, hi), lo <= hi: 10 doubles per pair in upper-triangular order, less
// 2 for every diagonal slot before it
__host__ __device__ constexpr int pair_offset(int lo, int hi) {
    return kPairStride * (lo * 8 - (lo * (lo - 1)) / 2 + (hi - lo)) - 2 * (lo + (hi > lo ? 1 : 0));
}

struct ElemParams {
    const double* xyz;
    const int4* conn4;
    int64_t e_begin, e_end;  // elements [e_begin, e_end) of this launch
    double* rec;
    double lm;         // lam / mu
    double mu8;        // mu / 8 times the square of what dnr is divided by
    double wc[3][3];   // centrifugal operator: f = wc . x (UnitVectorF)
    double dnr[8][24]; // dN_a/dxi_i at Gauss point g at [g][3a+i], divided by the largest
    // tm[s][c]: product of the 1D shape factors of two corners along one axis at a Gauss point
    // on the negative (s = 0) or positive (s = 1) side: c = 0 both corners negative, 1 mixed,
    // 2 both positive; tmx the same times DE / 512 (x is contracted first)
    double tm[2][3], tmx[2][3];
};

struct ElemSmem {
    double dnr[8][kRPad];       // ElemParams::dnr; padded row: the 8 rows
                                // start in 8 different bank pairs (a 24-double row put every
                                // even g in one bank and every odd g in another)
    double cf[kEpc][8][3];      // Walsh sums of the element-local coordinates; later D1
    double wx[kEpc][8][3];      // W x_a: centrifugal density per unit mass at corner a
    double R[kEpc][8][kRPad];   // R_a(g)[i] (scaled as dnr, x 64) at [el][g][3a+i]
    double Rs[kEpc][8][kRPad];  // mu R_a(g)[i] / det_g, scaled so that the products have no factor
    double det[kEpc][8];        // x 512
    double d2[kEpc][18];        // second mass contraction
    double m[kEpc][36];         // mass by corner-pair class (27 used, DE included), see mass_class
};

// Class of the corner pair (a, b) for the mass: per axis 0 both corners on the negative side,
// 1 mixed, 2 both positive; M_ab depends only on it.  Corners on the negative side of xi: 1, 2, 5, 6 (mask
// 0x66), of eta: 2, 3, 6, 7 (0xCC), of zeta: 0-3 (0x0F).
__device__ __forceinline__ int mass_class(int a, int b) {
    const int nx = (0x66 >> a) & 1, ny = (0xCC >> a) & 1, nz = (0x0F >> a) & 1;
    const int mx = (0x66 >> b) & 1, my = (0xCC >> b) & 1, mz = (0x0F >> b) & 1;
    const int cx = nx != mx ? 1 : (nx ? 0 : 2), cy = ny != my ? 1 : (ny ? 0 : 2), cz = nz != mz ? 1 : (nz ? 0 : 2);
    return cx * 9 + cy * 3 + cz;
}

// Off-diagonal pair list (a < b), 28 entries.
__device__ __forceinline__ void offdiag_pair(int q, int& a, int& b) {
    // q -> (a, b) for row-major enumeration of a < b
    int aa = 0, rem = q;
    while (rem >= 7 - aa) {
        rem -= 7 - aa;
        ++aa;
    }
    a = aa;
    b = aa + 1 + rem;
}

// P += sum over Gauss points g0 .. g0 + ng - 1 of Rs_a R_b^T
__device__ __forceinline__ void gram(const ElemSmem& s, int el, int a, int b, int g0, int ng, double (&P)[9]) {
#pragma unroll
    for (int i = 0; i < 9; ++i) P[i] = 0.0;
#pragma unroll 4
    for (int g = g0; g < g0 + ng; ++g) {
        const double* q = s.Rs[el][g] + 3 * a;
        const double* r = s.R[el][g] + 3 * b;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) P[3 * i + j] = fma(q[i], r[j], P[3 * i + j]);
    }
}

__global__ void __launch_bounds__(kElemThreads, 48 / kEpc) k_hex8_element(const ElemParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ElemSmem& s = *reinterpret_cast<ElemSmem*>(smem_raw);
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x;
    const int el = tid >> 3;
    const int t = tid & 7;
    const int64_t e_raw = p.e_begin + int64_t(blockIdx.x) * kEpc + el;
    const bool valid = e_raw < p.e_end;
    const int64_t e = valid ? e_raw : p.e_end - 1;   // the lanes of absent elements repeat the last one

    for (int k = tid; k < 8 * 8 * 3; k += kElemThreads) s.dnr[k / 24][k % 24] = (&p.dnr[0][0])[k];
    double c[3];
    {
        const int64_t node = __ldg(reinterpret_cast<const int*>(p.conn4) + 8 * e + t);
#pragma unroll
        for (int i = 0; i < 3; ++i) c[i] = __ldg(p.xyz + 3 * node + i);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) s.wx[el][t][i] = p.wc[i][0] * c[0] + p.wc[i][1] * c[1] + p.wc[i][2] * c[2];
    // element-local coordinates (no offset to cancel), then Walsh sums over the corners,
    // W_s = sum_a (-1)^popc(s & a) x_a on lane s.  The natural coordinates are negative at corners
    // {1,2,5,6} (xi), {2,3,6,7} (eta), {0,1,2,3} (zeta) (FEM_model_bsr.py:371-382), so 8 c_k is W_3 for xi,
    // W_2 for eta, -W_4 for zeta, W_1 for xi eta, -W_6 for eta zeta, -W_7 for xi zeta, -W_5 for xi eta zeta.
#pragma unroll
    for (int i = 0; i < 3; ++i) c[i] -= __shfl_sync(full, c[i], tid & 24);
#pragma unroll
    for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double o = __shfl_xor_sync(full, c[i], m);
            c[i] = o + flip_sign(c[i], t & m);
        }
#pragma unroll
    for (int i = 0; i < 3; ++i) s.cf[el][t][i] = flip_sign(c[i], t & 4);
    __syncthreads();  // the shape table is shared by the block's warps

    // ---- phase A: Gauss point g = t ------------------------------------------------
    {
        const int g = t;
        // Gauss point coordinates in the reference's order (zeta fastest, FEM_model_bsr.py:425-432)
        const double xi = (g & 4) ? kGS1 : -kGS1, et = (g & 2) ? kGS1 : -kGS1, ze = (g & 1) ? kGS1 : -kGS1;
        const double(*f)[3] = s.cf[el];
        // 8 J: of the two lanes that share column d the one on the negative side of direction d forms
        // components 0 and 1, the other 2
        double J[3][3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int bit = d == 0 ? 4 : d == 1 ? 2 : 1;
            const bool up = (g & bit) != 0;
            double v[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i = up ? 2 : k;
                if (d == 0) v[k] = fma(ze, fma(et, f[5][i], f[7][i]), fma(et, f[1][i], f[3][i]));        // dx/dxi
                else if (d == 1) v[k] = fma(ze, fma(xi, f[5][i], f[6][i]), fma(xi, f[1][i], f[2][i]));   // dx/deta
                else v[k] = fma(et, fma(xi, f[5][i], f[6][i]), fma(xi, f[7][i], f[4][i]));               // dx/dzeta
            }
            const double o0 = __shfl_xor_sync(full, v[0], bit), o1 = __shfl_xor_sync(full, v[1], bit);
            J[0][d] = up ? o0 : v[0];
            J[1][d] = up ? o1 : v[1];
            J[2][d] = up ? v[0] : o0;
        }
        double A[3][3];  // adjugate: inverse(J) = A / det
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
                A[j][i] = J[i1][j1] * J[i2][j2] - J[i2][j1] * J[i1][j2];
            }
        const double det = J[0][0] * A[0][0] + J[1][0] * A[0][1] + J[2][0] * A[0][2];
        const double sc = p.mu8 / det;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double r = fma(s.dnr[g][3 * a + 2], A[2][i],
                                     fma(s.dnr[g][3 * a + 1], A[1][i], s.dnr[g][3 * a] * A[0][i]));
                s.R[el][g][3 * a + i] = r;
                s.Rs[el][g][3 * a + i] = r * sc;
            }
        s.det[el][g] = det;
    }
    __syncwarp();

    // ---- mass, M_ab = DE sum_g det_g N_a(g) N_b(g), by sum factorisation ------------------
    // N_a(g) is a product of one 1D factor per axis, so M_ab depends on the class of (a, b) per
    // axis only: contract the 8 det_g along x (D1: 3 classes x 4 (y, z) points), y (D2: 9 x 2),
    // z (D3: 27 classes), 114 FP64 operations instead of 36 pairs x 8 Gauss points.
    {
        double* D1 = &s.cf[el][0][0];
        double* D2 = s.d2[el];
        double* D3 = s.m[el];
        for (int i = t; i < 12; i += 8) {
            const int cx = i >> 2, gyz = i & 3;
            D1[i] = fma(s.det[el][4 + gyz], p.tmx[1][cx], s.det[el][gyz] * p.tmx[0][cx]);
        }
        __syncwarp();
        for (int i = t; i < 18; i += 8) {
            const int cx = i / 6, r = i - 6 * cx, cy = r >> 1, gz = r & 1;
            D2[i] = fma(D1[cx * 4 + 2 + gz], p.tm[1][cy], D1[cx * 4 + gz] * p.tm[0][cy]);
        }
        __syncwarp();
        for (int i = t; i < 27; i += 8) {
            const int cxy = i / 3, cz = i - 3 * cxy;
            D3[i] = fma(D2[cxy * 2 + 1], p.tm[1][cz], D2[cxy * 2] * p.tm[0][cz]);
        }
        __syncwarp();
    }

    // ---- phase B: node pairs -----------------------------------------------------------
    double* rec = p.rec + e * kRec;
    const double lm = p.lm, lm1 = p.lm + 1.0;
    // diagonal pair (t, t): P symmetric
    {
        const int a = t;
        double P00 = 0, P11 = 0, P22 = 0, P01 = 0, P02 = 0, P12 = 0;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            const double r0 = s.R[el][g][3 * a], r1 = s.R[el][g][3 * a + 1], r2 = s.R[el][g][3 * a + 2];
            const double q0 = s.Rs[el][g][3 * a], q1 = s.Rs[el][g][3 * a + 1], q2 = s.Rs[el][g][3 * a + 2];
            P00 = fma(q0, r0, P00);
            P11 = fma(q1, r1, P11);
            P22 = fma(q2, r2, P22);
            P01 = fma(q0, r1, P01);
            P02 = fma(q0, r2, P02);
            P12 = fma(q1, r2, P12);
        }
        const double tr = P00 + P11 + P22;
        if (valid) {
            double2* o = reinterpret_cast<double2*>(rec + kPairStride * pair_index(a, a) - 2 * a);  // pair_offset(a, a)
            o[0] = make_double2(fma(lm1, P00, tr), fma(lm1, P11, tr));
            o[1] = make_double2(fma(lm1, P22, tr), lm1 * P01);
            o[2] = make_double2(lm1 * P02, lm1 * P12);
            // the unused slot: whole 32-byte sectors written, none read back from DRAM
            o[3] = make_double2(s.m[el][mass_class(a, a)], 0.0);
        }
    }
    // off-diagonal pairs
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const bool shared_pair = i == 3;   // the last four pairs: two threads, four Gauss points each
        int a, b;
        offdiag_pair(shared_pair ? 24 + (t >> 1) : 8 * i + t, a, b);
        double P[9];
        if (shared_pair) {
            gram(s, el, a, b, 4 * (t & 1), 4, P);
#pragma unroll
            for (int k = 0; k < 9; ++k) P[k] += __shfl_xor_sync(full, P[k], 1);
        } else {
            gram(s, el, a, b, 0, 8, P);
        }
        const double tr = P[0] + P[4] + P[8];
        if (valid && !(shared_pair && (t & 1))) {
            double2* o = reinterpret_cast<double2*>(rec + kPairStride * pair_index(a, b) - 2 * (a + 1));  // pair_offset
            o[0] = make_double2(fma(lm1, P[0], tr), fma(lm, P[1], P[3]));
            o[1] = make_double2(fma(lm, P[2], P[6]), fma(lm, P[3], P[1]));
            o[2] = make_double2(fma(lm1, P[4], tr), fma(lm, P[5], P[7]));
            o[3] = make_double2(fma(lm, P[6], P[2]), fma(lm, P[7], P[5]));
            o[4] = make_double2(fma(lm1, P[8], tr), s.m[el][mass_class(a, b)]);
        }
    }
    // element load for corner t: F_t = sum_b M_tb W x_b (the mass blocks of the other threads'
    // pairs come through shared memory)
    if (valid) {
        double f0 = 0, f1 = 0, f2 = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const double mv = s.m[el][mass_class(t, b)];
            f0 = fma(mv, s.wx[el][b][0], f0);
            f1 = fma(mv, s.wx[el][b][1], f1);
            f2 = fma(mv, s.wx[el][b][2], f2);
        }
        rec[kFOff + 3 * t + 0] = f0;
        rec[kFOff + 3 * t + 1] = f1;
        rec[kFOff + 3 * t + 2] = f2;
    }
}

// The same records with a warp per element, for meshes too small to fill the SMs: one SMSP takes a
// FP64 warp instruction every 64 cycles, so the 566 of k_hex8_element are 18 us however few warps
// there are; spread over 32 lanes they are about 230 (the 28 off-diagonal pairs in one round; gradients,
// diagonal pairs and loads in quarters; the geometry of a Gauss point repeated by 4 lanes).  In total
// that is 1.6 times the work, so the rule of launch_hex8_element stops where the device is full.
// Lane = (quarter h, corner or Gauss point t).
constexpr int kWideEpc = 4;
constexpr int kWidePerSm = 16;   // elements per SM up to which it is taken (see launch_hex8_element)
struct WideSmem {
    double dnr[8][kRPad];
    double cf[kWideEpc][8][3];
    double wx[kWideEpc][8][3];
    double R[kWideEpc][8][kRPad];
    double Rs[kWideEpc][8][kRPad];
    double det[kWideEpc][8];
    double d1[kWideEpc][12], d2[kWideEpc][18];
    double m[kWideEpc][36];
};

__global__ void __launch_bounds__(kWideEpc * 32) k_hex8_element_wide(const ElemParams p) {
    __shared__ WideSmem s;
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, el = tid >> 5, lane = tid & 31, t = lane & 7, h = lane >> 3;
    const int64_t e_raw = p.e_begin + int64_t(blockIdx.x) * kWideEpc + el;
    const bool valid = e_raw < p.e_end;
    const int64_t e = valid ? e_raw : p.e_end - 1;
    for (int k = tid; k < 8 * 8 * 3; k += kWideEpc * 32) s.dnr[k / 24][k % 24] = (&p.dnr[0][0])[k];
    double c[3];
    {
        const int64_t node = __ldg(reinterpret_cast<const int*>(p.conn4) + 8 * e + t);
#pragma unroll
        for (int i = 0; i < 3; ++i) c[i] = __ldg(p.xyz + 3 * node + i);
    }
    if (h < 3) s.wx[el][t][h] = p.wc[h][0] * c[0] + p.wc[h][1] * c[1] + p.wc[h][2] * c[2];
#pragma unroll
    for (int i = 0; i < 3; ++i) c[i] -= __shfl_sync(full, c[i], lane & 24);
#pragma unroll
    for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double o = __shfl_xor_sync(full, c[i], m);
            c[i] = o + flip_sign(c[i], t & m);
        }
    if (h == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) s.cf[el][t][i] = flip_sign(c[i], t & 4);
    }
    __syncthreads();
    {
        const int g = t;
        const double xi = (g & 4) ? kGS1 : -kGS1, et = (g & 2) ? kGS1 : -kGS1, ze = (g & 1) ? kGS1 : -kGS1;
        const double(*f)[3] = s.cf[el];
        // 8 J: quarter h < 3 forms component h
        double d[3];
        {
            const int i = h < 3 ? h : 0;
            const double m = fma(xi, f[5][i], f[6][i]);
            d[0] = fma(ze, fma(et, f[5][i], f[7][i]), fma(et, f[1][i], f[3][i]));
            d[1] = fma(ze, m, fma(xi, f[1][i], f[2][i]));
            d[2] = fma(et, m, fma(xi, f[7][i], f[4][i]));
        }
        double J[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) J[i][k] = __shfl_sync(full, d[k], 8 * i + t);
        double A[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
                A[j][i] = J[i1][j1] * J[i2][j2] - J[i2][j1] * J[i1][j2];
            }
        const double det = J[0][0] * A[0][0] + J[1][0] * A[0][1] + J[2][0] * A[0][2];
        const double sc = p.mu8 / det;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int a = 2 * h + k;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double r = fma(s.dnr[g][3 * a + 2], A[2][i],
                                     fma(s.dnr[g][3 * a + 1], A[1][i], s.dnr[g][3 * a] * A[0][i]));
                s.R[el][g][3 * a + i] = r;
                s.Rs[el][g][3 * a + i] = r * sc;
            }
        }
        if (h == 0) s.det[el][g] = det;
    }
    __syncwarp();
    // mass by sum factorisation, as k_hex8_element
    if (lane < 12) {
        const int cx = lane >> 2, gyz = lane & 3;
        s.d1[el][lane] = fma(s.det[el][4 + gyz], p.tmx[1][cx], s.det[el][gyz] * p.tmx[0][cx]);
    }
    __syncwarp();
    if (lane < 18) {
        const int cx = lane / 6, r = lane - 6 * cx, cy = r >> 1, gz = r & 1;
        s.d2[el][lane] = fma(s.d1[el][cx * 4 + 2 + gz], p.tm[1][cy], s.d1[el][cx * 4 + gz] * p.tm[0][cy]);
    }
    __syncwarp();
    if (lane < 27) {
        const int cxy = lane / 3, cz = lane - 3 * cxy;
        s.m[el][lane] = fma(s.d2[el][cxy * 2 + 1], p.tm[1][cz], s.d2[el][cxy * 2] * p.tm[0][cz]);
    }
    __syncwarp();
    double* rec = p.rec + e * kRec;
    const double lm = p.lm, lm1 = p.lm + 1.0;
    // diagonal pair (t, t): two Gauss points a quarter
    {
        const int a = t;
        double P[6] = {0, 0, 0, 0, 0, 0};  // 00, 11, 22, 01, 02, 12
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double* r = s.R[el][2 * h + k] + 3 * a;
            const double* q = s.Rs[el][2 * h + k] + 3 * a;
            P[0] = fma(q[0], r[0], P[0]);
            P[1] = fma(q[1], r[1], P[1]);
            P[2] = fma(q[2], r[2], P[2]);
            P[3] = fma(q[0], r[1], P[3]);
            P[4] = fma(q[0], r[2], P[4]);
            P[5] = fma(q[1], r[2], P[5]);
        }
#pragma unroll
        for (int off = 8; off < 32; off <<= 1)
#pragma unroll
            for (int i = 0; i < 6; ++i) P[i] += __shfl_xor_sync(full, P[i], off);
        const double tr = P[0] + P[1] + P[2];
        if (valid && h == 0) {
            double2* o = reinterpret_cast<double2*>(rec + kPairStride * pair_index(a, a) - 2 * a);  // pair_offset(a, a)
            o[0] = make_double2(fma(lm1, P[0], tr), fma(lm1, P[1], tr));
            o[1] = make_double2(fma(lm1, P[2], tr), lm1 * P[3]);
            o[2] = make_double2(lm1 * P[4], lm1 * P[5]);
            o[3] = make_double2(s.m[el][mass_class(a, a)], 0.0);
        }
    }
    // element load for corner t: two corners b a quarter
    {
        double f[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int b = 2 * h + k;
            const double mv = s.m[el][mass_class(t, b)];
#pragma unroll
            for (int i = 0; i < 3; ++i) f[i] = fma(mv, s.wx[el][b][i], f[i]);
        }
#pragma unroll
        for (int off = 8; off < 32; off <<= 1)
#pragma unroll
            for (int i = 0; i < 3; ++i) f[i] += __shfl_xor_sync(full, f[i], off);
        if (valid && h < 3) rec[kFOff + 3 * t + h] = h == 0 ? f[0] : h == 1 ? f[1] : f[2];
    }
    if (valid && lane < 28) {
        int a, b;
        offdiag_pair(lane, a, b);
        double P[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) P[i] = 0.0;
#pragma unroll 4
        for (int g = 0; g < 8; ++g) {
            const double* q = s.Rs[el][g] + 3 * a;
            const double* r = s.R[el][g] + 3 * b;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) P[3 * i + j] = fma(q[i], r[j], P[3 * i + j]);
        }
        const double tr = P[0] + P[4] + P[8];
        double2* o = reinterpret_cast<double2*>(rec + kPairStride * pair_index(a, b) - 2 * (a + 1));  // pair_offset
        o[0] = make_double2(fma(lm1, P[0], tr), fma(lm, P[1], P[3]));
        o[1] = make_double2(fma(lm, P[2], P[6]), fma(lm, P[3], P[1]));
        o[2] = make_double2(fma(lm1, P[4], tr), fma(lm, P[5], P[7]));
        o[3] = make_double2(fma(lm, P[6], P[2]), fma(lm, P[7], P[5]));
        o[4] = make_double2(fma(lm1, P[8], tr), s.m[el][mass_class(a, b)]);
    }
}

// Block (a, b) of element e as 10 doubles (K row-major, then M), oriented for row corner a and
// column corner b: an off-diagonal pair is stored once (a < b) and transposed for a > b; a
// diagonal pair is stored as its 6 distinct values.  Every lane issues the same five 16-byte
// loads (a diagonal slot's last two land in the next block or in F and go unused) and picks
// its values with selects, so the lanes of a row do not diverge.
__device__ __forceinline__ void load_pair_block(const double* rec, int64_t e, int a, int b, double (&v)[kPairStride]) {
    const bool dg = a == b, tr = a > b;
    const int lo = min(a, b), hi = max(a, b);
    const double2* blk = reinterpret_cast<const double2*>(rec + e * kRec + pair_offset(lo, hi));
    double w[kPairStride];
#pragma unroll
    for (int q = 0; q < kPairStride / 2; ++q) {
        const double2 x = __ldg(blk + q);
        w[2 * q] = x.x;
        w[2 * q + 1] = x.y;
    }
    v[0] = w[0];
    v[1] = dg ? w[3] : (tr ? w[3] : w[1]);
    v[2] = dg ? w[4] : (tr ? w[6] : w[2]);
    v[3] = dg ? w[3] : (tr ? w[1] : w[3]);
    v[4] = dg ? w[1] : w[4];
    v[5] = dg ? w[5] : (tr ? w[7] : w[5]);
    v[6] = dg ? w[4] : (tr ? w[2] : w[6]);
    v[7] = dg ? w[5] : (tr ? w[5] : w[7]);
    v[8] = dg ? w[2] : w[8];
    v[9] = dg ? w[6] : w[9];
}

struct GatherParams {
    int64_t n_node;
    const int32_t* indptr;
    const int32_t* indices;
    const int32_t* ne_ptr;
    const int32_t* ne_list;
    const int4* conn4;
    const double* rec;
    int k_layout, m_layout;
    double* K;
    double* M;
    double* F;
    const uint8_t* fixed;
    const double* loads;
};

__device__ __forceinline__ unsigned corner_match(int col, const int4& c0, const int4& c1) {
    return unsigned(c0.x == col) | (unsigned(c0.y == col) << 1) | (unsigned(c0.z == col) << 2) |
           (unsigned(c0.w == col) << 3) | (unsigned(c1.x == col) << 4) | (unsigned(c1.y == col) << 5) |
           (unsigned(c1.z == col) << 6) | (unsigned(c1.w == col) << 7);
}

__global__ void __launch_bounds__(256) k_gather(const GatherParams p) {
    const int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= p.n_node) return;
    const int64_t rs = p.indptr[row];
    const int L = p.indptr[row + 1] - int(rs);
    const int ks = p.ne_ptr[row], ke = p.ne_ptr[row + 1];
    const unsigned fixed_bits = p.fixed ? p.fixed[row] : 0u;

    for (int base = 0; base < L; base += 32) {
        const int l = base + lane;
        const bool active = l < L;
        const int col = active ? __ldg(p.indices + rs + l) : -1;
        double acc[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[k] = 0.0;
        double accm = 0.0;
        for (int k = ks; k < ke; ++k) {
            const int ent = __ldg(p.ne_list + k);
            const int64_t e = ent >> 3;
            const int a = ent & 7;
            const int4 c0 = __ldg(p.conn4 + 2 * e), c1 = __ldg(p.conn4 + 2 * e + 1);
            unsigned mask = corner_match(col, c0, c1);
            while (mask) {
                const int b = __ffs(mask) - 1;
                mask &= mask - 1;
                double v[kPairStride];
                load_pair_block(p.rec, e, a, b, v);
#pragma unroll
                for (int k = 0; k < 9; ++k) acc[k] += v[k];
                accm += v[9];
            }
        }
        if (col == int(row)) {
#pragma unroll
            for (int d = 0; d < 3; ++d)
                if ((fixed_bits >> d) & 1u) acc[4 * d] = 1e20;
        }
        if (active) {
            if (p.K) {
                if (p.k_layout == FEM_LAYOUT_BSR) {
                    double* o = p.K + 9 * (rs + l);
#pragma unroll
                    for (int k = 0; k < 9; ++k) o[k] = acc[k];
                } else {
#pragma unroll
                    for (int pp = 0; pp < 3; ++pp) {
                        double* o = p.K + 9 * rs + int64_t(3 * pp) * L + 3 * l;
                        o[0] = acc[3 * pp];
                        o[1] = acc[3 * pp + 1];
                        o[2] = acc[3 * pp + 2];
                    }
                }
            }
            if (p.M) {
                if (p.m_layout == FEM_LAYOUT_BSR) {
                    p.M[rs + l] = accm;
                } else {
#pragma unroll
                    for (int pp = 0; pp < 3; ++pp) p.M[3 * rs + int64_t(pp) * L + l] = accm;
                }
            }
        }
    }
    if (p.F && lane < 3) {
        double f = 0.0;
        for (int k = ks; k < ke; ++k) {
            const int ent = __ldg(p.ne_list + k);
            f += __ldg(p.rec + int64_t(ent >> 3) * kRec + kFOff + 3 * (ent & 7) + lane);
        }
        if (p.loads) f += p.loads[3 * row + lane];
        p.F[3 * row + lane] = f;
    }
}

// ---- FP64 gather, lane = (row, element corner) -------------------------------------------------
//
// One warp per 4 block rows; lane (r, b) handles corner b of every element incident to row r.
// For incident entry k (ascending element index) it reads the element block of the pair
// (a, b) -- a = the row's corner in that element -- from the element record (transposed when
// a > b) and adds it into the row's shared-memory accumulator at the slot given by the
// element-to-block map (slot_map).  All 8 lanes of a row do useful FP64 work on every entry.
// The first contribution to a slot is stored instead of added (a per-row bit mask of the
// slots already holding a value), which saves the ~27 of ~64 block additions per interior
// row that would add into zero.  A repeated corner node of a degenerate element adds after
// the earlier corner.  The summation order (element by element, corners ascending) is fixed,
// so results are bitwise reproducible.  Rows with more than kG64MaxL blocks use the
// lane-per-slot path (same order).
constexpr int kG64Warps = 4;
constexpr int kG64Rows = 4;
// 27 slots: every row of a structured hex mesh (3 x 3 x 3 neighbour nodes).  A row's
// accumulator holds 29 positions of 10 doubles (2,320 bytes; 16 rows per CTA take 36 KB, so 6
// CTAs (24 warps) fit on an SM).  A row of 27 slots places slot s at kPos27(s): each element's 8
// corners hit a 2 x 2 x 2 sub-cube of the 3 x 3 x 3 neighbourhood, and the table gives the 8
// slots of every such sub-cube distinct positions mod 8, so the 16-byte accesses of a row's 8
// lanes fall in 8 different bank groups (in slot order, slots 8 apart collided).  No placement
// in 27 positions does that (the centre slot lies in all 8 sub-cubes, so its residue can hold
// nothing else); the table uses 29.  Other rows keep position = slot.  Any one-to-one placement
// gives the same sums; the table only removes bank conflicts.
constexpr int kG64MaxL = 27;
constexpr int kG64Pos = 29;
constexpr int kG64RowStride = kG64Pos * kPairStride;

// Position of slot s (0..26) in a row of 27 slots: 5 bits per slot, 12 slots per word.  The
// classes of equal position mod 8: {the 4 centres of the x edges}, 4 x {a face centre, the
// edge centre and 2 corners that complete its exact cover of the 8 sub-cubes}, 2 x {a z face
// centre, 2 edge centres}, {the centre}.
__device__ __forceinline__ int pos27(int s) {
    const unsigned long long w = s < 12 ? 0x048d9144ec575012ull : (s < 24 ? 0x0a99bc86964508e1ull : 0x671bull);
    return int((w >> (5 * (s - 12 * (s / 12)))) & 31ull);
}

struct Gather64Params {
    int64_t row_begin, row_end;  // block rows [row_begin, row_end) of this launch
    const int32_t* indptr;
    const int32_t* indices;
    const int32_t* ne_ptr;
    const int32_t* ne_list;
    const uint8_t* slot_map;
    int slot_map_aligned;  // slot_map on an 8-byte boundary: one 8-byte load per entry
    const int4* conn4;
    const double* rec;
    int k_layout, m_layout;
    double* K;
    double* M;
    double* F;
    const uint8_t* fixed;
    const double* loads;
};

struct Gather64Smem {
    double acc[kG64Warps][kG64Rows][kG64RowStride];
};

// Lane-per-slot path for one row of any length (K and M; F is summed by the caller).
__device__ void gather_row_long64(const Gather64Params& p, int64_t row, int lane) {
    const int64_t rs = p.indptr[row];
    const int L = p.indptr[row + 1] - int(rs);
    const int ks = p.ne_ptr[row], ke = p.ne_ptr[row + 1];
    const unsigned fixed_bits = p.fixed ? p.fixed[row] : 0u;
    for (int base = 0; base < L; base += 32) {
        const int l = base + lane;
        const bool active = l < L;
        double acc[kPairStride];
#pragma unroll
        for (int q = 0; q < kPairStride; ++q) acc[q] = 0.0;
        bool any = false;
        for (int k = ks; k < ke; ++k) {
            const int ent = __ldg(p.ne_list + k);
            for (int b = 0; b < 8; ++b) {
                if (int(__ldg(p.slot_map + 8 * int64_t(k) + b)) != l) continue;
                double v[kPairStride];
                load_pair_block(p.rec, ent >> 3, ent & 7, b, v);
#pragma unroll
                for (int q = 0; q < kPairStride; ++q) acc[q] = any ? acc[q] + v[q] : v[q];
                any = true;
            }
        }
        if (!active) continue;
        const bool diag = __ldg(p.indices + rs + l) == int(row);
        if (diag) {
#pragma unroll
            for (int d = 0; d < 3; ++d)
                if ((fixed_bits >> d) & 1u) acc[4 * d] = 1e20;
        }
        if (p.K) {
            if (p.k_layout == FEM_LAYOUT_BSR) {
#pragma unroll
                for (int q = 0; q < 9; ++q) p.K[9 * (rs + l) + q] = acc[q];
            } else {
#pragma unroll
                for (int q = 0; q < 9; ++q) p.K[9 * rs + int64_t(3 * (q / 3)) * L + 3 * l + (q % 3)] = acc[q];
            }
        }
        if (p.M) {
            if (p.m_layout == FEM_LAYOUT_BSR) p.M[rs + l] = acc[9];
            else
                for (int pp = 0; pp < 3; ++pp) p.M[3 * rs + int64_t(pp) * L + l] = acc[9];
        }
    }
}

__global__ void __launch_bounds__(kG64Warps * 32, 6) k_gather64(const Gather64Params p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Gather64Smem& S = *reinterpret_cast<Gather64Smem*>(smem_raw);
    const unsigned full = 0xffffffffu;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = lane >> 3, b = lane & 7;
    const int64_t row0 = p.row_begin + (int64_t(blockIdx.x) * kG64Warps + w) * kG64Rows;
    if (row0 >= p.row_end) return;  // uniform per warp
    const int64_t row = row0 + r;
    const bool vrow = row < p.row_end;
    const int64_t rs = vrow ? p.indptr[row] : 0;
    const int L = vrow ? p.indptr[row + 1] - int(rs) : 0;
    const int ks = vrow ? p.ne_ptr[row] : 0;
    const int cnt = vrow ? p.ne_ptr[row + 1] - ks : 0;

    // F of this row on lanes b < 3 (corner loads in element order, then the nodal loads) for
    // the warps that leave before the main path
    auto row_F = [&]() {
        if (p.F && vrow && b < 3) {
            double f = 0.0;
            for (int k = 0; k < cnt; ++k) {
                const int ent = __ldg(p.ne_list + ks + k);
                f += __ldg(p.rec + int64_t(ent >> 3) * kRec + kFOff + 3 * (ent & 7) + b);
            }
            if (p.loads) f += p.loads[3 * row + b];
            p.F[3 * row + b] = f;
        }
    };
    if (!p.K && !p.M) {
        row_F();
        return;
    }
    if (__any_sync(full, L > kG64MaxL)) {
        row_F();
        for (int rr = 0; rr < kG64Rows; ++rr)
            if (row0 + rr < p.row_end) gather_row_long64(p, row0 + rr, lane);
        return;
    }

    // the row's diagonal slot (-1 if the node is not its own neighbour), found by the 8 lanes
    int diag = -1;
    for (int l = b; l < L; l += 8)
        if (__ldg(p.indices + rs + l) == int(row)) diag = l;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) diag = max(diag, __shfl_xor_sync(full, diag, off));
    const bool full27 = L == kG64MaxL;
    double* accr = S.acc[w][r];

    int maxcnt = cnt;
#pragma unroll
    for (int off = 8; off < 32; off <<= 1) maxcnt = max(maxcnt, __shfl_xor_sync(full, maxcnt, off));

    // The row's incident entries, 8 at a time: lane (r, j) holds entry 8c + j of chunk c (its
    // ne_list value and its 8 slot_map bytes), and every lane of the row takes entry k from
    // lane (r, k mod 8) by a shuffle, so the element block loads of entry k + 1 issue without
    // first waiting for a load of ne_list.
    const int src = lane & ~7;
    int ent_reg = 0;
    unsigned long long sm_reg = 0ull;
    auto load_chunk = [&](int c) {
        const int j = 8 * c + b;
        ent_reg = j < cnt ? __ldg(p.ne_list + ks + j) : 0;
        if (j < cnt) {
            if (p.slot_map_aligned) {
                sm_reg = __ldg(reinterpret_cast<const unsigned long long*>(p.slot_map) + (ks + j));
            } else {
                sm_reg = 0ull;
                for (int q = 0; q < 8; ++q)
                    sm_reg |= (unsigned long long)__ldg(p.slot_map + 8 * int64_t(ks + j) + q) << (8 * q);
            }
        }
    };
    load_chunk(0);
    // F of this row on lanes b < 3: corner loads in element order, then the nodal loads.  Lane (r, j) loads
    // entry 8c + j's three values, so a chunk's loads are in flight together; the sums walk the lanes.
    if (p.F) {
        double f = 0.0;
        for (int c = 0; 8 * c < maxcnt; ++c) {
            if (c) load_chunk(c);
            double w[3] = {0.0, 0.0, 0.0};
            if (8 * c + b < cnt) {
                const double* q = p.rec + int64_t(ent_reg >> 3) * kRec + kFOff + 3 * (ent_reg & 7);
#pragma unroll
                for (int i = 0; i < 3; ++i) w[i] = __ldg(q + i);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const double w0 = __shfl_sync(full, w[0], src | j), w1 = __shfl_sync(full, w[1], src | j);
                const double w2 = __shfl_sync(full, w[2], src | j);
                if (8 * c + j < cnt) f += b == 0 ? w0 : b == 1 ? w1 : w2;
            }
        }
        if (maxcnt > 8) load_chunk(0);
        if (b < 3 && vrow) {
            if (p.loads) f += p.loads[3 * row + b];
            p.F[3 * row + b] = f;
        }
    }
    unsigned touched = 0;  // slots of row r holding a value (the same in the row's 8 lanes)
    double cur[kPairStride], nxt[kPairStride];
    int cur_slot = 0, nxt_slot = 0;
    if (maxcnt > 0) {
        const int ent = __shfl_sync(full, ent_reg, src);
        const unsigned long long wd = __shfl_sync(full, sm_reg, src);
        if (cnt > 0) {
            load_pair_block(p.rec, ent >> 3, ent & 7, b, cur);
            cur_slot = int((wd >> (8 * b)) & 0xffull);
        }
    }
    for (int k = 0; k < maxcnt; ++k) {
        const bool active = k < cnt;
        if (k + 1 < maxcnt) {  // uniform over the warp
            if (((k + 1) & 7) == 0) load_chunk((k + 1) >> 3);
            const int ent = __shfl_sync(full, ent_reg, src | ((k + 1) & 7));
            const unsigned long long wd = __shfl_sync(full, sm_reg, src | ((k + 1) & 7));
            if (k + 1 < cnt) {
                load_pair_block(p.rec, ent >> 3, ent & 7, b, nxt);
                nxt_slot = int((wd >> (8 * b)) & 0xffull);
            }
        }
        // a repeated corner node (degenerate element) maps two corners to one slot
        bool dup = false;
#pragma unroll
        for (int bp = 0; bp < 7; ++bp) {
            const int other = __shfl_sync(full, cur_slot, (lane & ~7) | bp);
            if (bp < b && other == cur_slot) dup = true;
        }
        const unsigned bit = 1u << cur_slot;
        double* a = accr + (full27 ? pos27(cur_slot) : cur_slot) * kPairStride;
        if (active && !dup) {
            if (touched & bit) {
#pragma unroll
                for (int q = 0; q < kPairStride; ++q) a[q] += cur[q];
            } else {
#pragma unroll
                for (int q = 0; q < kPairStride; ++q) a[q] = cur[q];
            }
        }
        if (__any_sync(full, active && dup)) {
            for (int bb = 1; bb < 8; ++bb) {
                __syncwarp();
                if (active && dup && b == bb) {
#pragma unroll
                    for (int q = 0; q < kPairStride; ++q) a[q] += cur[q];
                }
            }
        }
        unsigned nb = active ? bit : 0u;
        nb |= __shfl_xor_sync(full, nb, 1);
        nb |= __shfl_xor_sync(full, nb, 2);
        nb |= __shfl_xor_sync(full, nb, 4);
        touched |= nb;
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kPairStride; ++q) cur[q] = nxt[q];
        cur_slot = nxt_slot;
    }
    __syncwarp();

    // ---- write the four rows (all lanes, coalesced) -----------------------------------------
    for (int rr = 0; rr < kG64Rows; ++rr) {
        const int64_t rw = row0 + rr;
        if (rw >= p.row_end) break;
        const int64_t rrs = __shfl_sync(full, rs, rr * 8);
        const int LL = __shfl_sync(full, L, rr * 8);
        const unsigned tch = __shfl_sync(full, touched, rr * 8);
        const unsigned fixed_bits = p.fixed ? p.fixed[rw] : 0u;
        const int sd = __shfl_sync(full, diag, rr * 8);
        const bool has_diag = sd >= 0;
        const bool f27 = LL == kG64MaxL;
        const double* acc = S.acc[w][rr];
        auto value = [&](int s_, int q) -> double {
            if (!((tch >> s_) & 1u)) return 0.0;
            double v = acc[(f27 ? pos27(s_) : s_) * kPairStride + q];
            if (q < 9 && has_diag && s_ == sd && (q % 4 == 0) && ((fixed_bits >> (q / 4)) & 1u)) v = 1e20;
            return v;
        };
        if (p.K) {
            if (p.k_layout == FEM_LAYOUT_BSR) {
                for (int o = lane; o < 9 * LL; o += 32) {
                    const int s_ = o / 9;
                    p.K[9 * rrs + o] = value(s_, o - 9 * s_);
                }
            } else {
                for (int pp = 0; pp < 3; ++pp)
                    for (int idx = lane; idx < 3 * LL; idx += 32) {
                        const int s_ = idx / 3;
                        p.K[9 * rrs + int64_t(3 * LL) * pp + idx] = value(s_, 3 * pp + (idx - 3 * s_));
                    }
            }
        }
        if (p.M) {
            if (p.m_layout == FEM_LAYOUT_BSR) {
                for (int o = lane; o < LL; o += 32) p.M[rrs + o] = value(o, 9);
            } else {
                for (int o = lane; o < LL; o += 32) {
                    const double mv = value(o, 9);
                    p.M[3 * rrs + o] = mv;
                    p.M[3 * rrs + LL + o] = mv;
                    p.M[3 * rrs + 2 * LL + o] = mv;
                }
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_csr_index(int64_t n_node, const int32_t* __restrict__ indptr,
                                                   const int32_t* __restrict__ indices, int32_t* rowK,
                                                   int32_t* colK, int32_t* rowM, int32_t* colM) {
    const int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= n_node) return;
    const int64_t rs = indptr[row];
    const int L = indptr[row + 1] - int(rs);
    if (lane < 3) {
        // InstallIndexK / InstallIndexM: FEM_model_csr.py:167-173, 195-201
        if (rowK) rowK[3 * row + 1 + lane] = int32_t(L * 3 * (lane + 1) + rs * 9);
        if (rowM) rowM[3 * row + 1 + lane] = int32_t(L * (lane + 1) + rs * 3);
        if (row == 0) {
            if (rowK) rowK[0] = 0;
            if (rowM) rowM[0] = 0;
        }
    }
    for (int l = lane; l < L; l += 32) {
        const int col = indices[rs + l];
        for (int pp = 0; pp < 3; ++pp) {
            if (colK) {
                int32_t* o = colK + 9 * rs + int64_t(3 * pp) * L + 3 * l;
                o[0] = 3 * col;
                o[1] = 3 * col + 1;
                o[2] = 3 * col + 2;
            }
            if (colM) colM[3 * rs + int64_t(pp) * L + l] = 3 * col + pp;
        }
    }
}

int check_mesh(const fem_mesh* m) {
    FEM_REQUIRE(m != nullptr, "mesh is NULL");
    FEM_REQUIRE(m->n_node >= 0 && m->n_elem >= 0 && m->nnzb >= 0, "negative mesh size");
    FEM_REQUIRE(m->n_elem < (int64_t(1) << 28), "n_elem too large");
    FEM_REQUIRE(m->n_node < (int64_t(1) << 31) - 1, "n_node too large");
    FEM_REQUIRE(9 * m->nnzb < (int64_t(1) << 62), "nnzb too large");
    if (m->n_elem) FEM_REQUIRE(m->xyz && m->conn && aligned16(m->conn), "xyz/conn NULL or conn not 16-byte aligned");
    if (m->n_node) FEM_REQUIRE(m->indptr && m->ne_ptr && m->ne_list, "pattern/incidence arrays are NULL");
    if (m->nnzb) FEM_REQUIRE(m->indices != nullptr, "indices is NULL");
    return FEM_OK;
}

}  // namespace

}  // namespace fem

using namespace fem;

extern "C" size_t fem_assemble_workspace_bytes(int64_t n_elem) {
    // FEM_ALGO_FP64: one 2,944-byte record per element; FEM_ALGO_DD: eight 672-byte
    // row-ordered chunks per element.  The larger of the two serves both.
    return n_elem > 0 ? size_t(n_elem) * 8 * 672 : 0;
}

namespace {

int check_assembly_inputs(const fem_mesh* mesh, const fem_material* mat, void* workspace, size_t workspace_bytes) {
    int rc = check_mesh(mesh);
    if (rc) return rc;
    FEM_REQUIRE(mat != nullptr, "mat is NULL");
    FEM_REQUIRE(mat->PO > -1.0 && mat->PO < 0.5, "Poisson ratio must lie in (-1, 0.5)");
    if (workspace_bytes < fem_assemble_workspace_bytes(mesh->n_elem) || (mesh->n_elem && !workspace)) {
        set_error("workspace too small: need %zu bytes", fem_assemble_workspace_bytes(mesh->n_elem));
        return FEM_ERR_WORKSPACE;
    }
    FEM_REQUIRE(workspace == nullptr || aligned16(workspace), "workspace not 16-byte aligned");
    return FEM_OK;
}

}  // namespace

namespace fem {
namespace {

// Unevaluated sum of two doubles, for the constants of the FP64 element kernels.
struct Pair {
    double h, l;
};
Pair two_sum(double a, double b) {
    const double s = a + b, z = s - a;
    return {s, (a - (s - z)) + (b - z)};
}
Pair product(Pair a, Pair b) {
    const double p = a.h * b.h, e = std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h);
    const double s = p + e;
    return {s, e - (s - p)};
}
Pair quotient(Pair a, Pair b) {
    const double q = a.h / b.h, e = (std::fma(-q, b.h, a.h) + (a.l - q * b.l)) / b.h;
    const double s = q + e;
    return {s, e - (s - q)};
}
// a / b * c, correctly rounded but for ties
double rounded_quotient(double a, Pair b, Pair c) { return product(quotient({a, 0.0}, b), c).h; }

// The shape derivatives divided by the largest, (1 + g)^2 / 8, and the square of that.  A derivative is
// +-(1 + g)^2 / 8, (1 - g^2) / 8 or (1 - g)^2 / 8 (g = kGS1); rounded as they are, the first is high by 0.7 of
// its last place, everywhere it stands, and so were K's values: 1.3e-16 of themselves on average for
// steel.  As 1, t and t^2, t = (1 - g) / (1 + g), the ones that matter most are exact, and with mu and
// lam / mu rounded once K's error is rounding noise (100 jittered unit elements of steel: 1.7e-16 rms
// against 80-bit arithmetic, 2.1e-16 with the table as it is).
struct UnitShape {
    double dnr[8][24];
    Pair scale;
};
const UnitShape& unit_shape() {
    static const UnitShape u = [] {
        UnitShape v;
        const Pair far = two_sum(1.0, kGS1), near = two_sum(1.0, -kGS1);
        const Pair a = product(far, far), t = quotient(near, far), t2 = product(t, t);
        const double values[3] = {1.0, t.h, t2.h};
        const ShapeTables& s = shape_tables();
        for (int g = 0; g < 8; ++g)
            for (int k = 0; k < 24; ++k) {
                const double d = s.dnr[g][k / 3][k % 3], r = std::fabs(d) * 8 / a.h;   // one of the three, to rounding
                v.dnr[g][k] = std::copysign(values[r > 0.6 ? 0 : r > 0.15 ? 1 : 2], d);
            }
        v.scale = product(a, a);
        v.scale.h /= 64;
        v.scale.l /= 64;
        return v;
    }();
    return u;
}

}  // namespace

int sm_count();
int launch_hex8_element_dd(const fem_mesh* mesh, const fem_material* mat, void* workspace, cudaStream_t st,
                           int64_t e_begin, int64_t e_end);
int launch_gather_dd(const fem_mesh* mesh, const fem_assembly_out* out, const void* workspace, cudaStream_t st,
                     int64_t row_begin, int64_t row_end);
}  // namespace fem

namespace fem {
namespace {

int launch_hex8_element(const fem_mesh* mesh, const fem_material* mat, void* workspace, cudaStream_t st,
                        int64_t e_begin, int64_t e_end) {
    if (e_end <= e_begin) return FEM_OK;
    ElemParams ep;
    ep.xyz = mesh->xyz;
    ep.conn4 = reinterpret_cast<const int4*>(mesh->conn);
    ep.e_begin = e_begin;
    ep.e_end = e_end;
    ep.rec = static_cast<double*>(workspace);
    const double EX = mat->EX, PO = mat->PO;
    const UnitShape& us = unit_shape();
    std::memcpy(ep.dnr, us.dnr, sizeof(ep.dnr));
    // FEM_model_bsr.py:435-449: D0 = lam + 2 mu and lam, D1 = mu
    ep.lm = rounded_quotient(2 * PO, two_sum(1.0, -2 * PO), {1.0, 0.0});
    ep.mu8 = rounded_quotient(EX, two_sum(1.0, PO), us.scale) / 16;
    {
        const double w0 = mat->omega[0], w1 = mat->omega[1], w2 = mat->omega[2];
        const double wc[3][3] = {{w1 * w1 + w2 * w2, -w0 * w1, -w0 * w2},   // UnitVectorF, FEM_model_bsr.py:291-300
                                 {-w1 * w0, w0 * w0 + w2 * w2, -w1 * w2},
                                 {-w2 * w0, -w2 * w1, w1 * w1 + w0 * w0}};
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) ep.wc[i][j] = wc[i][j];
    }
    {
        // 1D shape factors (1 + s x) / 2 at x = +-kGS1: al for a corner on the Gauss point's
        // side, be for the other side
        const double al = 0.5 * (1.0 + kGS1), be = 0.5 * (1.0 - kGS1);
        const double tm[2][3] = {{al * al, al * be, be * be}, {be * be, al * be, al * al}};
        for (int sd = 0; sd < 2; ++sd)
            for (int c = 0; c < 3; ++c) {
                ep.tm[sd][c] = tm[sd][c];
                ep.tmx[sd][c] = mat->DE / 512 * tm[sd][c];
            }
    }
    // A warp per element up to 16 elements an SM (152 SMs): 12.3 against 26.7 us at 256 elements, 24.6
    // against 26.7 at 1,536, 39.5 against 41.1 at 2,560, 55.1 against 42.4 at 4,000.  By the whole mesh,
    // not the part: every split of an assembly gives the same bits.
    if (mesh->n_elem <= int64_t(kWidePerSm) * sm_count()) {
        const int64_t blocks = (e_end - e_begin + kWideEpc - 1) / kWideEpc;
        k_hex8_element_wide<<<unsigned(blocks), kWideEpc * 32, 0, st>>>(ep);
        FEM_LAUNCH_CHECK("k_hex8_element_wide");
        return FEM_OK;
    }
    const size_t smem = sizeof(ElemSmem);
    FEM_CUDA(cudaFuncSetAttribute(k_hex8_element, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    const int64_t blocks = (e_end - e_begin + kEpc - 1) / kEpc;
    k_hex8_element<<<unsigned(blocks), kElemThreads, smem, st>>>(ep);
    FEM_LAUNCH_CHECK("k_hex8_element");
    return FEM_OK;
}

// FP64 gather of block rows [row_begin, row_end); the lane-per-corner kernel needs the
// element-to-block map, the lane-per-slot kernel (whole mesh only) does not.
int launch_gather64(const fem_mesh* mesh, const fem_assembly_out* out, const void* workspace, cudaStream_t st,
                    int64_t row_begin, int64_t row_end) {
    if (row_end <= row_begin) return FEM_OK;
    if (!mesh->slot_map) {
        FEM_REQUIRE(row_begin == 0 && row_end == mesh->n_node, "a partial FP64 gather needs mesh->slot_map");
        GatherParams gp;
        gp.n_node = mesh->n_node;
        gp.indptr = mesh->indptr;
        gp.indices = mesh->indices;
        gp.ne_ptr = mesh->ne_ptr;
        gp.ne_list = mesh->ne_list;
        gp.conn4 = reinterpret_cast<const int4*>(mesh->conn);
        gp.rec = static_cast<const double*>(workspace);
        gp.k_layout = out->k_layout;
        gp.m_layout = out->m_layout;
        gp.K = out->K;
        gp.M = out->M;
        gp.F = out->F;
        gp.fixed = out->fixed;
        gp.loads = out->loads;
        const int64_t blocks = (mesh->n_node * 32 + 255) / 256;
        k_gather<<<unsigned(blocks), 256, 0, st>>>(gp);
        FEM_LAUNCH_CHECK("k_gather");
        return FEM_OK;
    }
    Gather64Params gp;
    gp.row_begin = row_begin;
    gp.row_end = row_end;
    gp.indptr = mesh->indptr;
    gp.indices = mesh->indices;
    gp.ne_ptr = mesh->ne_ptr;
    gp.ne_list = mesh->ne_list;
    gp.slot_map = mesh->slot_map;
    gp.slot_map_aligned = (reinterpret_cast<uintptr_t>(mesh->slot_map) & 7) == 0;
    gp.conn4 = reinterpret_cast<const int4*>(mesh->conn);
    gp.rec = static_cast<const double*>(workspace);
    gp.k_layout = out->k_layout;
    gp.m_layout = out->m_layout;
    gp.K = out->K;
    gp.M = out->M;
    gp.F = out->F;
    gp.fixed = out->fixed;
    gp.loads = out->loads;
    const size_t smem = sizeof(Gather64Smem);
    FEM_CUDA(cudaFuncSetAttribute(k_gather64, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    const int64_t rows_per_cta = int64_t(kG64Warps) * kG64Rows;
    const int64_t blocks = (row_end - row_begin + rows_per_cta - 1) / rows_per_cta;
    k_gather64<<<unsigned(blocks), kG64Warps * 32, smem, st>>>(gp);
    FEM_LAUNCH_CHECK("k_gather64");
    return FEM_OK;
}

}  // namespace
}  // namespace fem

extern "C" int fem_assemble_elements(const fem_mesh* mesh, const fem_material* mat, int algo, void* workspace,
                                     size_t workspace_bytes, void* stream) {
    int rc = check_assembly_inputs(mesh, mat, workspace, workspace_bytes);
    if (rc) return rc;
    FEM_REQUIRE(algo == FEM_ALGO_DD || algo == FEM_ALGO_FP64, "bad algo");
    if (mesh->n_elem == 0) return FEM_OK;
    FEM_REQUIRE(algo != FEM_ALGO_DD || (mesh->ne_inv && mesh->slot_map),
                "FEM_ALGO_DD needs mesh->ne_inv and mesh->slot_map (fem_gather_map)");
    if (algo == FEM_ALGO_DD) return launch_hex8_element_dd(mesh, mat, workspace, as_stream(stream), 0, mesh->n_elem);
    return launch_hex8_element(mesh, mat, workspace, as_stream(stream), 0, mesh->n_elem);
}

extern "C" int fem_assemble_gather(const fem_mesh* mesh, const fem_assembly_out* out, const void* workspace,
                                   size_t workspace_bytes, void* stream) {
    int rc = check_mesh(mesh);
    if (rc) return rc;
    FEM_REQUIRE(out != nullptr, "out is NULL");
    FEM_REQUIRE(out->k_layout == FEM_LAYOUT_BSR || out->k_layout == FEM_LAYOUT_CSR, "bad k_layout");
    FEM_REQUIRE(out->m_layout == FEM_LAYOUT_BSR || out->m_layout == FEM_LAYOUT_CSR, "bad m_layout");
    FEM_REQUIRE(out->algo == FEM_ALGO_DD || out->algo == FEM_ALGO_FP64, "bad algo");
    if (workspace_bytes < fem_assemble_workspace_bytes(mesh->n_elem) || (mesh->n_elem && !workspace)) {
        set_error("workspace too small: need %zu bytes", fem_assemble_workspace_bytes(mesh->n_elem));
        return FEM_ERR_WORKSPACE;
    }
    if (mesh->n_node == 0 || (!out->K && !out->M && !out->F)) return FEM_OK;
    if (out->algo == FEM_ALGO_DD) {
        FEM_REQUIRE(mesh->n_elem == 0 || mesh->slot_map, "FEM_ALGO_DD needs mesh->slot_map (fem_gather_map)");
        return launch_gather_dd(mesh, out, workspace, as_stream(stream), 0, mesh->n_node);
    }
    return launch_gather64(mesh, out, workspace, as_stream(stream), 0, mesh->n_node);
}

extern "C" int fem_assemble(const fem_mesh* mesh, const fem_material* mat, const fem_assembly_out* out,
                            void* workspace, size_t workspace_bytes, void* stream) {
    int rc = check_assembly_inputs(mesh, mat, workspace, workspace_bytes);
    if (rc) return rc;
    FEM_REQUIRE(out != nullptr, "out is NULL");
    FEM_REQUIRE(out->k_layout == FEM_LAYOUT_BSR || out->k_layout == FEM_LAYOUT_CSR, "bad k_layout");
    FEM_REQUIRE(out->m_layout == FEM_LAYOUT_BSR || out->m_layout == FEM_LAYOUT_CSR, "bad m_layout");
    if (mesh->n_node == 0) return FEM_OK;
    rc = fem_assemble_elements(mesh, mat, out->algo, workspace, workspace_bytes, stream);
    if (rc) return rc;
    return fem_assemble_gather(mesh, out, workspace, workspace_bytes, stream);
}

namespace fem {
namespace {

// fem_assemble_host; with `on_part`, the calling thread also waits for each part's copies in
// turn and calls on_part(q) while later parts are still being copied (then returns only when
// every copy and every on_part call is done).
template <typename OnPart>
int assemble_host_impl(const fem_mesh* mesh, const fem_material* mat, const fem_assembly_out* out,
                       const int64_t* row_split, const int64_t* elem_split, const int64_t* block_split, int n_parts,
                       double* K_host, double* M_host, double* F_host, void* workspace, size_t workspace_bytes,
                       void* stream, OnPart* on_part) {
    int rc = check_assembly_inputs(mesh, mat, workspace, workspace_bytes);
    if (rc) return rc;
    FEM_REQUIRE(out != nullptr, "out is NULL");
    FEM_REQUIRE(out->k_layout == FEM_LAYOUT_BSR || out->k_layout == FEM_LAYOUT_CSR, "bad k_layout");
    FEM_REQUIRE(out->m_layout == FEM_LAYOUT_BSR || out->m_layout == FEM_LAYOUT_CSR, "bad m_layout");
    FEM_REQUIRE(out->algo == FEM_ALGO_DD || out->algo == FEM_ALGO_FP64, "bad algo");
    FEM_REQUIRE((!K_host || out->K) && (!M_host || out->M) && (!F_host || out->F),
                "a host output needs the matching device output in out");
    FEM_REQUIRE(n_parts >= 1 && row_split && elem_split && block_split, "bad plan");
    FEM_REQUIRE(row_split[0] == 0 && row_split[n_parts] == mesh->n_node && elem_split[0] == 0 &&
                    elem_split[n_parts] == mesh->n_elem && block_split[0] == 0 && block_split[n_parts] == mesh->nnzb,
                "plan does not span the mesh (use fem_pipeline_plan)");
    for (int q = 0; q < n_parts; ++q)
        FEM_REQUIRE(row_split[q] <= row_split[q + 1] && elem_split[q] <= elem_split[q + 1] &&
                        block_split[q] <= block_split[q + 1],
                    "plan is not monotone");
    if (mesh->n_node == 0) return FEM_OK;
    FEM_REQUIRE(out->algo != FEM_ALGO_DD || mesh->n_elem == 0 || (mesh->ne_inv && mesh->slot_map),
                "FEM_ALGO_DD needs mesh->ne_inv and mesh->slot_map (fem_gather_map)");
    FEM_REQUIRE(out->algo == FEM_ALGO_DD || mesh->n_elem == 0 || mesh->slot_map || n_parts == 1,
                "a split FP64 assembly needs mesh->slot_map (fem_gather_map)");
    cudaStream_t st = as_stream(stream);
    const bool dd = out->algo == FEM_ALGO_DD;
    const int parts = n_parts;
    std::vector<cudaEvent_t> elems(parts, nullptr), done(parts, nullptr), copied(parts, nullptr);
    cudaStream_t cs = nullptr, gs = nullptr;
    cudaEvent_t start = nullptr, fin = nullptr;
    auto cleanup = [&] {
        for (auto* v : {&elems, &done, &copied})
            for (cudaEvent_t e : *v)
                if (e) cudaEventDestroy(e);
        if (start) cudaEventDestroy(start);
        if (fin) cudaEventDestroy(fin);
        if (cs) cudaStreamDestroy(cs);
        if (gs) cudaStreamDestroy(gs);
    };
    auto fail = [&](cudaError_t e, const char* what) {
        cleanup();
        return cuda_status(e, what);
    };
    int lo_prio = 0, hi_prio = 0;
    cudaError_t e = cudaDeviceGetStreamPriorityRange(&lo_prio, &hi_prio);
    if (e != cudaSuccess) return fail(e, "cudaDeviceGetStreamPriorityRange");
    if ((e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaStreamCreateWithPriority(&gs, cudaStreamNonBlocking, hi_prio)) != cudaSuccess)
        return fail(e, "stream creation");
    if ((e = cudaEventCreateWithFlags(&start, cudaEventDisableTiming)) != cudaSuccess ||
        (e = cudaEventRecord(start, st)) != cudaSuccess || (e = cudaStreamWaitEvent(gs, start, 0)) != cudaSuccess)
        return fail(e, "gather stream ordering");
    // All kernels first (a copy into pageable memory may block the host until it ends).  The
    // element parts run in order on the caller's stream and the gathers on a second,
    // highest-priority stream, gather q after element part q: the gather of part q fills the
    // partial last waves of element part q + 1 instead of waiting for them, and part q's copy
    // can start as soon as its gather ends.  Records of different parts never overlap, so the
    // results do not depend on how the two streams interleave.
    for (int q = 0; q < parts; ++q) {
        rc = dd ? launch_hex8_element_dd(mesh, mat, workspace, st, elem_split[q], elem_split[q + 1])
                : launch_hex8_element(mesh, mat, workspace, st, elem_split[q], elem_split[q + 1]);
        if (rc) {
            cleanup();
            return rc;
        }
        if ((e = cudaEventCreateWithFlags(&elems[q], cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventRecord(elems[q], st)) != cudaSuccess || (e = cudaStreamWaitEvent(gs, elems[q], 0)) != cudaSuccess)
            return fail(e, "element part event");
        rc = dd ? launch_gather_dd(mesh, out, workspace, gs, row_split[q], row_split[q + 1])
                : launch_gather64(mesh, out, workspace, gs, row_split[q], row_split[q + 1]);
        if (rc) {
            cleanup();
            return rc;
        }
        if ((e = cudaEventCreateWithFlags(&done[q], cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventRecord(done[q], gs)) != cudaSuccess)
            return fail(e, "cudaEventRecord");
    }
    const int64_t kq = 9, mq = out->m_layout == FEM_LAYOUT_BSR ? 1 : 3;
    for (int q = 0; q < parts; ++q) {
        const int64_t r0 = row_split[q], r1 = row_split[q + 1];
        const int64_t b0 = block_split[q], b1 = block_split[q + 1];
        if ((e = cudaStreamWaitEvent(cs, done[q], 0)) != cudaSuccess) return fail(e, "cudaStreamWaitEvent");
        if (K_host && b1 > b0 &&
            (e = cudaMemcpyAsync(K_host + kq * b0, out->K + kq * b0, sizeof(double) * kq * (b1 - b0),
                                 cudaMemcpyDeviceToHost, cs)) != cudaSuccess)
            return fail(e, "K device->host copy");
        if (M_host && b1 > b0 &&
            (e = cudaMemcpyAsync(M_host + mq * b0, out->M + mq * b0, sizeof(double) * mq * (b1 - b0),
                                 cudaMemcpyDeviceToHost, cs)) != cudaSuccess)
            return fail(e, "M device->host copy");
        if (F_host && r1 > r0 &&
            (e = cudaMemcpyAsync(F_host + 3 * r0, out->F + 3 * r0, sizeof(double) * 3 * (r1 - r0),
                                 cudaMemcpyDeviceToHost, cs)) != cudaSuccess)
            return fail(e, "F device->host copy");
        if (on_part && ((e = cudaEventCreateWithFlags(&copied[q], cudaEventDisableTiming)) != cudaSuccess ||
                        (e = cudaEventRecord(copied[q], cs)) != cudaSuccess))
            return fail(e, "copy event");
    }
    if (on_part)
        for (int q = 0; q < parts; ++q) {
            if ((e = cudaEventSynchronize(copied[q])) != cudaSuccess) return fail(e, "copy event wait");
            (*on_part)(q);
        }
    // the caller's stream is ordered after the last copy
    if ((e = cudaEventCreateWithFlags(&fin, cudaEventDisableTiming)) != cudaSuccess ||
        (e = cudaEventRecord(fin, cs)) != cudaSuccess || (e = cudaStreamWaitEvent(st, fin, 0)) != cudaSuccess)
        return fail(e, "copy completion event");
    cleanup();
    return FEM_OK;
}

}  // namespace
}  // namespace fem

extern "C" int fem_assemble_host(const fem_mesh* mesh, const fem_material* mat, const fem_assembly_out* out,
                                 const int64_t* row_split, const int64_t* elem_split, const int64_t* block_split,
                                 int n_parts, double* K_host, double* M_host, double* F_host, void* workspace,
                                 size_t workspace_bytes, void* stream) {
    struct NoPart {
        void operator()(int) const {}
    };
    return assemble_host_impl<NoPart>(mesh, mat, out, row_split, elem_split, block_split, n_parts, K_host, M_host,
                                      F_host, workspace, workspace_bytes, stream, nullptr);
}

extern "C" int fem_assemble_host_staged(const fem_mesh* mesh, const fem_material* mat, const fem_assembly_out* out,
                                        const int64_t* row_split, const int64_t* elem_split,
                                        const int64_t* block_split, int n_parts, const int32_t* indptr_host,
                                        double* K_host, double* M_host, double* F_host, double* M_stage,
                                        void* workspace, size_t workspace_bytes, void* stream) {
    FEM_REQUIRE(out != nullptr && mesh != nullptr, "NULL argument");
    if (!M_host || !M_stage || out->m_layout != FEM_LAYOUT_CSR)
        return fem_assemble_host(mesh, mat, out, row_split, elem_split, block_split, n_parts, K_host, M_host,
                                 F_host, workspace, workspace_bytes, stream);
    FEM_REQUIRE(indptr_host != nullptr && row_split != nullptr && n_parts >= 1, "NULL argument");
    // M leaves the device as one value per block (the BSR layout) into M_stage; the reference's
    // scalar CSR (3 copies of it per block row) is written on the host, part by part, while
    // the later parts are still being copied.
    fem_assembly_out o = *out;
    o.m_layout = FEM_LAYOUT_BSR;
    auto expand = [&](int q) {
        const int64_t r0 = row_split[q], r1 = row_split[q + 1];
#pragma omp parallel for schedule(dynamic, 512)
        for (int64_t i = r0; i < r1; ++i) {
            const int64_t rs = indptr_host[i], L = indptr_host[i + 1] - rs;
            const double* src = M_stage + rs;
            double* dst = M_host + 3 * rs;
            for (int pp = 0; pp < 3; ++pp)
                for (int64_t l = 0; l < L; ++l) dst[pp * L + l] = src[l];
        }
    };
    return assemble_host_impl(mesh, mat, &o, row_split, elem_split, block_split, n_parts, K_host, M_stage, F_host,
                              workspace, workspace_bytes, stream, &expand);
}

extern "C" int fem_csr_index(const fem_mesh* mesh, int32_t* rowK, int32_t* colK, int32_t* rowM, int32_t* colM,
                             void* stream) {
    FEM_REQUIRE(mesh != nullptr, "mesh is NULL");
    FEM_REQUIRE(mesh->n_node >= 0, "negative size");
    FEM_REQUIRE(9 * mesh->nnzb < (int64_t(1) << 31), "CSR column indices exceed int32");
    if (mesh->n_node == 0) return FEM_OK;
    FEM_REQUIRE(mesh->indptr && (mesh->nnzb == 0 || mesh->indices), "pattern arrays are NULL");
    const int64_t blocks = (mesh->n_node * 32 + 255) / 256;
    k_csr_index<<<unsigned(blocks), 256, 0, as_stream(stream)>>>(mesh->n_node, mesh->indptr, mesh->indices, rowK,
                                                                 colK, rowM, colM);
    FEM_LAUNCH_CHECK("k_csr_index");
    return FEM_OK;
}
