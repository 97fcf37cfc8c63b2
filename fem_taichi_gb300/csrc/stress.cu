// Nodal stress recovery for sm_103a (POST_process.py:72-99, 172-223).
//
//  1. k_stress_element -- 8 threads per element, an element's threads in one warp.  Thread t
//     loads corner t; a Walsh transform over the 8 lanes gives the trilinear coefficients of the
//     element-local coordinates and displacements (c_k = 1/8 sum_a m_k(corner a) v_a for the monomials
//     1, xi, eta, zeta, xi eta, eta zeta, xi zeta, xi eta zeta).  Thread g then evaluates J and
//     dU/dxi at Gauss point g -- d/dxi does not depend on xi, so the two lanes that share it compute
//     half of it each, and so for eta and zeta -- the displacement
//     gradient H = (sum_a u_a (x) dN_a/dxi) . adj(J) / det, and the
//     stresses  sigma_n = D0 (H00, H11, H22),  sigma_s = mu (H01+H10, H12+H21, H02+H20)
//     (components xy, yz, xz as UnitVectorS orders them, POST_process.py:190-209).
//     Corner j's extrapolated value is sum_k W[j][k] sigma(k) with the caller's 8x8 weight
//     table (get_NdSol / shapefunc_GS, POST_process.py:172-181, 212-223); the dot products of
//     the table's distinct rows are spread over the element's threads, and thread j writes
//     corner j's values to the per-element workspace.  Bound by the FP64 pipe (one warp instruction
//     per 16 cycles per SM), so shuffles and selects are spent to save FP64 instructions: about
//     130 per thread, 200 before (960,000 elements: 2.55 -> 1.76 ms, the pipe 90 % busy in both).
//  2. k_stress_node -- one thread per node: sums its incident (element, corner) values in
//     ascending element order (no atomics), divides by the element count (get_NdAve,
//     :183-187; one reciprocal, six products; an isolated node stays 0 * inf = NaN), then
//     computes the principal stresses (descending order; sym3_eig_desc) and the
//     reference's "VM" formula as written (:93-94).
#include <cstring>
#include <mutex>

#include "fem_common.cuh"
#include "fem_dd.cuh"

namespace fem {
namespace {

constexpr int kEpc = 16;
constexpr int kThreads = kEpc * 8;
constexpr int kSvPad = 7;

struct StressParams {
    const double* xyz;
    const int4* conn4;
    const double* u;
    int64_t n_elem;
    double* rec;  // [n_elem][8][6]
    double lm, mu;   // lam / mu, mu
    double W[8][8];  // the distinct rows of the caller's extrapolation table
    int nrow;        // how many
    int row_of[8];   // corner j -> its row of W
};

struct StressSmem {
    double W[8][8];
    double res[kEpc][8][6];  // extrapolated values of each distinct table row
    double cf[kEpc][8][7];   // Walsh sums of the coordinates and displacements
    double sv[kEpc][8][kSvPad];
};

__global__ void __launch_bounds__(kThreads) k_stress_element(const StressParams p) {
    __shared__ StressSmem s;
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x;
    const int el = tid >> 3;
    const int t = tid & 7;
    const int64_t e_raw = int64_t(blockIdx.x) * kEpc + el;
    const bool valid = e_raw < p.n_elem;
    const int64_t e = valid ? e_raw : p.n_elem - 1;   // the lanes of absent elements repeat the last one
    for (int k = tid; k < 64; k += kThreads) (&s.W[0][0])[k] = (&p.W[0][0])[k];
    double c[6];
    {
        const int64_t node = __ldg(reinterpret_cast<const int*>(p.conn4) + 8 * e + t);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            c[i] = __ldg(p.xyz + 3 * node + i);
            c[3 + i] = __ldg(p.u + 3 * node + i);
        }
    }
    // element-local values (corner 0 subtracted; the gradients depend on differences only), then
    // Walsh sums over the corners, W_s = sum_a (-1)^popc(s & a) v_a on lane s.  The natural
    // coordinates are negative at corners {1,2,5,6} (xi), {2,3,6,7} (eta), {0,1,2,3} (zeta), so the
    // coefficients are xi: W_3, eta: W_2, zeta: -W_4, xi eta: W_1, eta zeta: -W_6, xi zeta: -W_7,
    // xi eta zeta: -W_5 (POST_process.py:238-273 for the corner order).  The 1 / 8 of a coefficient
    // cancels in G adj(J) / det: J and G stay 8 times theirs.
#pragma unroll
    for (int i = 0; i < 6; ++i) c[i] -= __shfl_sync(full, c[i], tid & 24);
#pragma unroll
    for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double o = __shfl_xor_sync(full, c[i], m);
            c[i] = o + flip_sign(c[i], t & m);
        }
#pragma unroll
    for (int i = 0; i < 6; ++i) s.cf[el][t][i] = flip_sign(c[i], t & 4);
    __syncthreads();  // the weight table is shared by the block's warps
    {
        const int g = t;
        const double xi = (g & 4) ? kGS1 : -kGS1, et = (g & 2) ? kGS1 : -kGS1, ze = (g & 1) ? kGS1 : -kGS1;
        // J (components 0-2) and G = dU/dxi (3-5): column d is the same on the two lanes that differ
        // in direction d only; the lane on the negative side forms J's column, the other G's, and
        // they swap.
        const int hx = (g & 4) ? 3 : 0, he = (g & 2) ? 3 : 0, hz = (g & 1) ? 3 : 0;
        double J[3][3], G[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double(*f)[7] = s.cf[el];
            const double x0 = fma(ze, fma(et, f[5][hx + i], f[7][hx + i]), fma(et, f[1][hx + i], f[3][hx + i]));
            const double y0 = fma(ze, fma(xi, f[5][he + i], f[6][he + i]), fma(xi, f[1][he + i], f[2][he + i]));
            const double z0 = fma(et, fma(xi, f[5][hz + i], f[6][hz + i]), fma(xi, f[7][hz + i], f[4][hz + i]));
            const double x1 = __shfl_xor_sync(full, x0, 4);
            const double y1 = __shfl_xor_sync(full, y0, 2);
            const double z1 = __shfl_xor_sync(full, z0, 1);
            J[i][0] = hx ? x1 : x0;
            G[i][0] = hx ? x0 : x1;
            J[i][1] = he ? y1 : y0;
            G[i][1] = he ? y0 : y1;
            J[i][2] = hz ? z1 : z0;
            G[i][2] = hz ? z0 : z1;
        }
        double A[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
                A[j][i] = J[i1][j1] * J[i2][j2] - J[i2][j1] * J[i1][j2];
            }
        const double det = J[0][0] * A[0][0] + J[1][0] * A[0][1] + J[2][0] * A[0][2];
        const double mi = p.mu * (1.0 / det);
        // h = det times du_i/dx_i and du_i/dx_k + du_k/dx_i
        double h[6];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int k = (i + 1) % 3;
            h[i] = fma(G[i][2], A[2][i], fma(G[i][1], A[1][i], G[i][0] * A[0][i]));
            h[3 + i] = fma(G[k][2], A[2][i], fma(G[k][1], A[1][i], fma(G[k][0], A[0][i],
                       fma(G[i][2], A[2][k], fma(G[i][1], A[1][k], G[i][0] * A[0][k])))));
        }
        const double tr = p.lm * (h[0] + h[1] + h[2]);   // sigma = mu (2 H + (lam / mu) tr H I)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            s.sv[el][g][i] = mi * fma(2.0, h[i], tr);
            s.sv[el][g][3 + i] = mi * h[3 + i];
        }
    }
    __syncwarp();
    // Extrapolation: the table's distinct rows only (the reference's aliased GMat gives every
    // even corner one row and every odd corner another: 12 dot products per element instead of
    // 48), spread over the element's 8 threads; corner j then takes its row's values.
    const int nout = p.nrow * 6;
    for (int o0 = 0; o0 < nout; o0 += 8) {
        const bool half = nout - o0 == 4;   // the last four outputs: two threads each, four Gauss points a thread
        const int o = half ? o0 + (t >> 1) : o0 + t, k0 = half ? 4 * (t & 1) : 0;
        if (o >= nout) break;
        const int r = o / 6, cc = o - 6 * r;
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) acc = fma(s.W[r][k0 + k], s.sv[el][k0 + k][cc], acc);
        if (half) {
            acc += __shfl_xor_sync(full, acc, 1);
        } else {
#pragma unroll
            for (int k = 4; k < 8; ++k) acc = fma(s.W[r][k], s.sv[el][k][cc], acc);
        }
        s.res[el][r][cc] = acc;
    }
    __syncwarp();
    if (!valid) return;
    const double* r = s.res[el][p.row_of[t]];
    double2* o = reinterpret_cast<double2*>(p.rec + (e * 8 + t) * 6);
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = make_double2(r[2 * q], r[2 * q + 1]);
}

// Eigenvalues of the symmetric 3x3 [[a00,a01,a02],[a01,a11,a12],[a02,a12,a22]] by cyclic
// Jacobi rotations in Rutishauser's form (the rotated off-diagonal set to zero, the diagonal
// updated as a_pp - t a_pq and a_qq + t a_pq, the third row rotated with tau = s / (1 + c);
// Numerical Recipes, "jacobi"); from the second sweep on, an off-diagonal below the last bit of
// both diagonals (100 |a_pq| lost in |a_pp| and |a_qq|) is dropped instead of rotated -- its
// rotation would move the diagonal by about a_pq^2 / (a_qq - a_pp) -- which ends a 3 x 3 in
// about three sweeps instead of five; c = rsqrt(1 + t^2); capped at 32 sweeps; returned
// descending.
__device__ __noinline__ void sym3_eig_jacobi(double a00, double a11, double a22, double a01, double a12, double a02,
                              double& p1, double& p2, double& p3) {
    double d[3] = {a00, a11, a22};
    double o01 = a01, o02 = a02, o12 = a12;
    for (int sweep = 0; sweep < 32; ++sweep) {
        if (fabs(o01) + fabs(o02) + fabs(o12) == 0.0) break;
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {
            // (p, q, r): (0, 1, 2), (0, 2, 1), (1, 2, 0)
            const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
            double& apq = pq == 0 ? o01 : pq == 1 ? o02 : o12;
            double& apr = pq == 0 ? o02 : pq == 1 ? o01 : o01;   // (p, r)
            double& aqr = pq == 0 ? o12 : pq == 1 ? o12 : o02;   // (q, r)
            if (apq == 0.0) continue;
            const double g = 100.0 * fabs(apq);
            if (sweep > 0 && fabs(d[p]) + g == fabs(d[p]) && fabs(d[q]) + g == fabs(d[q])) {
                apq = 0.0;
                continue;
            }
            const double h = d[q] - d[p];
            double t;
            if (fabs(h) + g == fabs(h)) {
                t = apq / h;
            } else {
                const double theta = 0.5 * h / apq;
                t = 1.0 / (fabs(theta) + sqrt(1.0 + theta * theta));
                if (theta < 0.0) t = -t;
            }
            const double c = rsqrt(fma(t, t, 1.0)), sn = t * c, tau = sn / (1.0 + c);
            const double ht = t * apq;
            d[p] -= ht;
            d[q] += ht;
            apq = 0.0;
            const double x = apr, y = aqr;  // rotate (p, r) and (q, r)
            apr = x - sn * (y + x * tau);
            aqr = y + sn * (x - y * tau);
        }
    }
    double e0 = d[0], e1 = d[1], e2 = d[2], tmp;
    if (e0 < e1) tmp = e0, e0 = e1, e1 = tmp;
    if (e1 < e2) tmp = e1, e1 = e2, e2 = tmp;
    if (e0 < e1) tmp = e0, e0 = e1, e1 = tmp;
    p1 = e0;
    p2 = e1;
    p3 = e2;
}

// Eigenvalues, descending, of a symmetric 3x3 (the same entries as sym3_eig_jacobi) with few FP64
// instructions: the FP32 pipes find the eigenvectors, FP64 only applies and corrects them.
//  1. Cyclic Jacobi in FP32 accumulates its rotations in a quaternion q, rounded to multiples of 2^-22
//     so that the entries of R(q) are exact in FP64.
//  2. R(q) is |q|^2 times an orthogonal matrix whatever q is, so B = R^T A R / |q|^4 has A's
//     eigenvalues; its off-diagonals are FP32 noise, ~2e-7 |A|.  With theta_j the FP32 eigenvalues
//     (R^T R is diagonal), B_ij = theta_j delta_ij + R_i . (A - theta_j) R_j / |q|^4: the vectors are as
//     small as the off-diagonals, so of the two products only the first rounds at the size of A.
//  3. Jacobi rotations in FP64 with tan(phi) = t from FP32.  The rotation is orthogonal for any t
//     (c = 1 / sqrt(1 + t^2): from y, the same in FP32, and r = 1 - (1 + t^2) y^2, by the binomial series of
//     y (1 - r)^(-1/2) to second order; r is about 1e-7), and what an inexact t leaves is carried, not dropped:
//     each sweep takes the off-diagonals down by another ~1e-7, so one sweep serves separated
//     eigenvalues (the neglected shift e^2 / gap is below 1e-18 |A|) and two serve equal ones.
// About 160 FP64 instructions against 630 of the Jacobi form (no FP64 division or square root):
// k_stress_node on 1,010,025 nodes 1.37 -> 0.47 ms.  Rms error, of |A|, on random tensors 0.92e-16 (Jacobi
// 1.25e-16; 1.6e-16 with R rounded and B formed without theta), on uniaxial ones 0.74e-16 (0.68e-16).
// A matrix outside the FP32 range, or with an infinity or NaN, takes sym3_eig_jacobi.
__device__ __forceinline__ float tan_rotation(float h, float apq) {  // h = a_qq - a_pp
    const float theta = __fdividef(0.5f * h, apq);
    const float t = __fdividef(1.f, fabsf(theta) + __fsqrt_rn(fmaf(theta, theta, 1.f)));
    return fabsf(theta) < 1e18f ? copysignf(t, theta) : __fdividef(apq, h);
}

__device__ __forceinline__ void sym3_eig_desc(double a00, double a11, double a22, double a01, double a12, double a02,
                                              double& p1, double& p2, double& p3) {
    float f00 = float(a00), f11 = float(a11), f22 = float(a22), f01 = float(a01), f12 = float(a12), f02 = float(a02);
    const float m = fmaxf(fmaxf(fabsf(f00), fabsf(f11)), fmaxf(fabsf(f22), fmaxf(fabsf(f01), fmaxf(fabsf(f12), fabsf(f02)))));
    const float any = fabsf(f00) + fabsf(f11) + fabsf(f22) + fabsf(f01) + fabsf(f12) + fabsf(f02);
    if (!(m > 1e-18f && any < 1e18f)) {   // also NaN, and the zero matrix
        sym3_eig_jacobi(a00, a11, a22, a01, a12, a02, p1, p2, p3);
        return;
    }
    float qw = 1.f, qx = 0.f, qy = 0.f, qz = 0.f;
    for (int sweep = 0; sweep < 6; ++sweep) {
        const float off = fabsf(f01) + fabsf(f02) + fabsf(f12);
        if (!(off > 3e-8f * m)) break;
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {   // (p, q): (0, 1), (0, 2), (1, 2)
            float& apq = pq == 0 ? f01 : pq == 1 ? f02 : f12;
            float& app = pq == 2 ? f11 : f00;
            float& aqq = pq == 0 ? f11 : f22;
            float& x = pq == 0 ? f02 : f01;   // (p, r)
            float& y = pq == 2 ? f02 : f12;   // (q, r)
            if (fabsf(apq) <= 1e-9f * m) continue;
            const float t = tan_rotation(aqq - app, apq);
            const float c = rsqrtf(fmaf(t, t, 1.f)), sn = t * c;
            app = fmaf(-t, apq, app);
            aqq = fmaf(t, apq, aqq);
            apq = 0.f;
            const float x0 = x, y0 = y;
            x = c * x0 - sn * y0;
            y = sn * x0 + c * y0;
            // half angle; the new axes are p' = c p - sn q, q' = sn p + c q: a turn by -phi about
            // r for (0, 1) and (1, 2), by +phi for (0, 2)
            const float hc = __fsqrt_rn(0.5f * (1.f + c));
            const float hs = (pq == 1 ? 0.5f : -0.5f) * __fdividef(sn, hc);
            const float w0 = qw, u0 = qx, v0 = qy, z0 = qz;
            if (pq == 0) {          // q (hc + hs k)
                qw = w0 * hc - z0 * hs, qx = u0 * hc + v0 * hs, qy = v0 * hc - u0 * hs, qz = z0 * hc + w0 * hs;
            } else if (pq == 1) {   // q (hc + hs j)
                qw = w0 * hc - v0 * hs, qx = u0 * hc - z0 * hs, qy = v0 * hc + w0 * hs, qz = z0 * hc + u0 * hs;
            } else {                // q (hc + hs i)
                qw = w0 * hc - u0 * hs, qx = u0 * hc + w0 * hs, qy = v0 * hc + z0 * hs, qz = z0 * hc - v0 * hs;
            }
        }
    }
    double d0, d1, d2, e01, e02, e12;
    {
        // multiples of 2^-22 (the sums lie in [2, 4]): products and sums of four are exact in 53 bits
        auto grid = [](float v) { return __fsub_rn(__fadd_rn(v, 3.f), 3.f); };
        qw = grid(qw), qx = grid(qx), qy = grid(qy), qz = grid(qz);
        const double w = qw, x = qx, y = qy, z = qz, x2 = 2.f * qx, y2 = 2.f * qy, z2 = 2.f * qz;
        const double ww = w * w, xx = x * x, yy = y * y, zz = z * z;
        const double a = ww + xx, b = yy + zz, cd = ww - xx, dd = yy - zz;
        const double wz = w * z2, wy = w * y2, wx = w * x2;
        const double R[3][3] = {{a - b, fma(x, y2, -wz), fma(x, z2, wy)},
                                {fma(x, y2, wz), cd + dd, fma(y, z2, -wx)},
                                {fma(x, z2, -wy), fma(y, z2, wx), cd - dd}};
        const double eps = (a + b) - 1.0;                          // |q|^2 - 1
        const double f = fma(eps, fma(3.0, eps, -2.0), 1.0);       // |q|^-4
        const double th[3] = {f00, f11, f22};
        double C[3][3];   // (A - theta_j) R_j
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            C[0][j] = fma(a02, R[2][j], fma(a01, R[1][j], (a00 - th[j]) * R[0][j]));
            C[1][j] = fma(a12, R[2][j], fma(a01, R[0][j], (a11 - th[j]) * R[1][j]));
            C[2][j] = fma(a12, R[1][j], fma(a02, R[0][j], (a22 - th[j]) * R[2][j]));
        }
        auto dot = [&](int i, int j) { return fma(R[2][i], C[2][j], fma(R[1][i], C[1][j], R[0][i] * C[0][j])); };
        d0 = fma(f, dot(0, 0), th[0]), d1 = fma(f, dot(1, 1), th[1]), d2 = fma(f, dot(2, 2), th[2]);
        e01 = f * dot(0, 1), e02 = f * dot(0, 2), e12 = f * dot(1, 2);
    }
    const float rm = __fdividef(1.f, m);
    for (int sweep = 0; sweep < 4; ++sweep) {
        bool turned = false;
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {
            double& e = pq == 0 ? e01 : pq == 1 ? e02 : e12;
            double& dp = pq == 2 ? d1 : d0;
            double& dq = pq == 0 ? d1 : d2;
            double& x = pq == 0 ? e02 : e01;
            double& y = pq == 2 ? e02 : e12;
            const double h = dq - dp;
            const float ef = float(e), hf = float(h), en = ef * rm;
            if (!(en * en > 1e-18f * fabsf(hf * rm)) || fabsf(en) < 1e-16f) continue;
            turned = true;
            const float tf = tan_rotation(hf, ef), yf = rsqrtf(fmaf(tf, tf, 1.f));
            const double t = tf, y0 = yf, t2 = t * t;
            const double r = fma(-(t2 + 1.0), y0 * y0, 1.0);
            const double c = fma(y0 * r, fma(0.375, r, 0.5), y0), sn = t * c, c2 = c * c;
            const double dl = t * (c2 * fma(t, h, -2.0 * e));   // a_pp' - a_pp for any t
            e = c2 * fma(-t, h, fma(-t2, e, e));
            dp += dl;
            dq -= dl;
            const double x0 = x, y1 = y;
            x = fma(c, x0, -sn * y1);
            y = fma(sn, x0, c * y1);
        }
        if (!turned) break;
    }
    double tmp;
    if (d0 < d1) tmp = d0, d0 = d1, d1 = tmp;
    if (d1 < d2) tmp = d1, d1 = d2, d2 = tmp;
    if (d0 < d1) tmp = d0, d0 = d1, d1 = tmp;
    p1 = d0;
    p2 = d1;
    p3 = d2;
}

// 1 / k for the element counts of a hex mesh's nodes (the same quotients as the division)
__constant__ double kInverse[17] = {0.0,      1.0 / 1,  1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,
                                    1.0 / 6,  1.0 / 7,  1.0 / 8,  1.0 / 9,  1.0 / 10, 1.0 / 11,
                                    1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15, 1.0 / 16};

__global__ void __launch_bounds__(256) k_stress_node(int64_t n_node, const int32_t* __restrict__ ne_ptr,
                                                     const int32_t* __restrict__ ne_list,
                                                     const int32_t* __restrict__ co_elem,
                                                     const double* __restrict__ rec, double* __restrict__ out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_node) return;
    double v[6] = {0, 0, 0, 0, 0, 0};
    const int ks = ne_ptr[i], ke = ne_ptr[i + 1];
    if (ks < ke) {
        const double2* r = reinterpret_cast<const double2*>(rec + int64_t(__ldg(ne_list + ks)) * 6);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double2 x = __ldg(r + c);
            v[2 * c] = x.x;
            v[2 * c + 1] = x.y;
        }
    }
#pragma unroll 4
    for (int k = ks + 1; k < ke; ++k) {
        const double2* r = reinterpret_cast<const double2*>(rec + int64_t(__ldg(ne_list + k)) * 6);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double2 x = __ldg(r + c);
            v[2 * c] += x.x;
            v[2 * c + 1] += x.y;
        }
    }
    const int ce = co_elem[i];
    const double rce = ce > 0 && ce <= 16 ? kInverse[ce] : 1.0 / double(ce);
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] *= rce;
    double p1, p2, p3;
    // vector order [xx, yy, zz, xy, yz, xz] (POST_process.py:79-86)
    sym3_eig_desc(v[0], v[1], v[2], v[3], v[4], v[5], p1, p2, p3);
    double* o = out + 10 * i;   // the caller's: 8-byte alignment only
#pragma unroll
    for (int c = 0; c < 6; ++c) o[c] = v[c];
    o[6] = p1;
    o[7] = p2;
    o[8] = p3;
    const double d12 = p1 - p2, d23 = p2 - p3;
    o[9] = sqrt(fma(d12, d12, 2.0 * (d23 * d23)));
}

}  // namespace
}  // namespace fem

using namespace fem;

extern "C" size_t fem_stress_workspace_bytes(int64_t n_elem) {
    return n_elem > 0 ? size_t(n_elem) * 48 * sizeof(double) : 0;
}

namespace fem {
int launch_stress_dd(const fem_mesh* mesh, const fem_material* mat, const double* u, const int32_t* co_elem,
                     const double* extrap, double* out, void* workspace, cudaStream_t st);
}

extern "C" int fem_stress_ex(const fem_mesh* mesh, const fem_material* mat, const double* u, const int32_t* co_elem,
                             const double* extrap, double* out, void* workspace, size_t workspace_bytes, int algo,
                             void* stream) {
    FEM_REQUIRE(mesh && mat && extrap, "mesh/mat/extrap is NULL");
    FEM_REQUIRE(mesh->n_node >= 0 && mesh->n_elem >= 0, "negative mesh size");
    FEM_REQUIRE(mesh->n_elem < (int64_t(1) << 28), "n_elem too large");
    FEM_REQUIRE(mat->PO > -1.0 && mat->PO < 0.5, "Poisson ratio must lie in (-1, 0.5)");
    if (mesh->n_node == 0) return FEM_OK;
    FEM_REQUIRE(u && co_elem && out && mesh->ne_ptr && mesh->ne_list, "u/co_elem/out/incidence is NULL");
    if (mesh->n_elem) FEM_REQUIRE(mesh->xyz && mesh->conn && aligned16(mesh->conn), "xyz/conn NULL or misaligned");
    if (workspace_bytes < fem_stress_workspace_bytes(mesh->n_elem) || (mesh->n_elem && !workspace)) {
        set_error("workspace too small: need %zu bytes", fem_stress_workspace_bytes(mesh->n_elem));
        return FEM_ERR_WORKSPACE;
    }
    FEM_REQUIRE(algo == FEM_ALGO_DD || algo == FEM_ALGO_FP64, "bad algo");
    FEM_REQUIRE(workspace == nullptr || aligned16(workspace), "workspace not 16-byte aligned");
    cudaStream_t st = as_stream(stream);
    if (algo == FEM_ALGO_DD) return launch_stress_dd(mesh, mat, u, co_elem, extrap, out, workspace, st);
    if (mesh->n_elem) {
        StressParams sp;
        sp.xyz = mesh->xyz;
        sp.conn4 = reinterpret_cast<const int4*>(mesh->conn);
        sp.u = u;
        sp.n_elem = mesh->n_elem;
        sp.rec = static_cast<double*>(workspace);
        const double EX = mat->EX, PO = mat->PO;
        sp.lm = 2 * PO / (1 - 2 * PO);   // D0 of POST_process.py:292-302 = lam + 2 mu, lam; lam / mu
        sp.mu = EX / 2 / (1 + PO);       // :304-306
        // distinct rows of the table (exactly equal rows share one)
        std::memset(sp.W, 0, sizeof(sp.W));
        sp.nrow = 0;
        for (int j = 0; j < 8; ++j) {
            int r = 0;
            while (r < sp.nrow && std::memcmp(sp.W[r], extrap + 8 * j, sizeof(double) * 8) != 0) ++r;
            if (r == sp.nrow) {
                for (int k = 0; k < 8; ++k) sp.W[r][k] = extrap[8 * j + k];
                ++sp.nrow;
            }
            sp.row_of[j] = r;
        }
        const int64_t blocks = (mesh->n_elem + kEpc - 1) / kEpc;
        k_stress_element<<<unsigned(blocks), kThreads, 0, st>>>(sp);
        FEM_LAUNCH_CHECK("k_stress_element");
    }
    const int64_t blocks = (mesh->n_node + 255) / 256;
    k_stress_node<<<unsigned(blocks), 256, 0, st>>>(mesh->n_node, mesh->ne_ptr, mesh->ne_list, co_elem,
                                                    static_cast<const double*>(workspace), out);
    FEM_LAUNCH_CHECK("k_stress_node");
    return FEM_OK;
}

extern "C" int fem_stress(const fem_mesh* mesh, const fem_material* mat, const double* u, const int32_t* co_elem,
                          const double* extrap, double* out, void* workspace, size_t workspace_bytes, void* stream) {
    return fem_stress_ex(mesh, mat, u, co_elem, extrap, out, workspace, workspace_bytes, FEM_ALGO_FP64, stream);
}

// ---- allocation-free variant ------------------------------------------------------------------
// Some callers cannot allocate device memory at all: plug-ins living inside a host program that
// owns every device allocation and only lends them input/output buffers, or latency-critical
// loops where cudaMalloc/cudaFree are forbidden because they synchronise the device.  For them
// fem_stress_noalloc runs the same two stress kernels with their per-element scratch placed in
// this file-scope device array instead of a caller workspace.  The array is reserved on every
// GPU that loads this library and stays there until the process exits.
namespace {

static __device__ __align__(256) double g_stress_scratch[size_t(FEM_STRESS_NOALLOC_MAX_ELEMS) * 48];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
void* g_scratch_addr[kMaxDevices] = {};

// Device address of g_stress_scratch on the current device, looked up once per device (the
// host-side symbol is only a stand-in and must never be handed to a kernel).
int scratch_address(void** out) {
    int dev = 0;
    FEM_CUDA(cudaGetDevice(&dev));
    FEM_REQUIRE(dev >= 0 && dev < kMaxDevices, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        FEM_CUDA(cudaGetSymbolAddress(&p, g_stress_scratch));
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return FEM_OK;
}

}  // namespace

extern "C" int fem_stress_noalloc(const fem_mesh* mesh, const fem_material* mat, const double* u,
                                  const int32_t* co_elem, const double* extrap, double* out, void* stream) {
    FEM_REQUIRE(mesh != nullptr, "mesh is NULL");
    if (mesh->n_elem > FEM_STRESS_NOALLOC_MAX_ELEMS) {
        set_error("fem_stress_noalloc: %lld elements exceed the built-in scratch limit of %d elements; "
                  "use fem_stress with a caller-allocated workspace",
                  (long long)mesh->n_elem, FEM_STRESS_NOALLOC_MAX_ELEMS);
        return FEM_ERR_WORKSPACE;
    }
    void* scratch = nullptr;
    int rc = scratch_address(&scratch);
    if (rc) return rc;
    // Every element record is fully rewritten by the element kernel before the node kernel
    // reads it, so nothing in the shared scratch has to be cleared between calls.
    return fem_stress(mesh, mat, u, co_elem, extrap, out, scratch, sizeof(g_stress_scratch), stream);
}

// ---- double-float variant (FEM_ALGO_DD; fem_stress runs FEM_ALGO_FP64) ----------------------------
// Same two kernels and record size as above, with the FP64 arithmetic moved to double-float
// on the FP32 pipes (fem_dd.cuh): node coordinates and displacements are made element-local
// in FP64 first (the gradient only depends on differences), the corner values are stored as
// float pairs, and the node kernel sums, averages and diagonalises in double-float (cyclic
// Jacobi, threshold 2^-46 of the diagonal), forming the FP64 outputs at the end.
namespace fem {
namespace {

struct StressDdParams {
    const double* xyz;
    const int4* conn4;
    const double* u;
    int64_t n_elem;
    const int32_t* ne_inv;  // NULL: record of (e, j) at e*8+j; else at ne_inv[e*8+j] (row order)
    float2* rec;            // 8 * n_elem records of 6 float pairs
    float2 D0d, lam, mu;
    float2 dnr[8][8][3];
    float2 W[8][8];  // the distinct rows of the caller's extrapolation table
    int nrow;        // how many
    int row_of[8];   // corner j -> its row of W
};

struct StressDdSmem {
    float2 dnr[8][8][3];
    float2 W[8][8];
    float2 res[kEpc][8][6];  // extrapolated values of each distinct table row
    float2 x[kEpc][8][3];
    float2 u[kEpc][8][3];
    float2 sv[kEpc][8][kSvPad];
};

__device__ __forceinline__ dd ldp(const float2& v) { return dd{v.x, v.y}; }
__device__ __forceinline__ float2 stp(dd v) { return make_float2(v.hi, v.lo); }

__global__ void __launch_bounds__(kThreads) k_stress_element_dd(const StressDdParams p) {
    __shared__ StressDdSmem s;
    const int tid = threadIdx.x;
    const int el = tid >> 3;
    const int t = tid & 7;
    const int64_t e = int64_t(blockIdx.x) * kEpc + el;
    const bool valid = e < p.n_elem;
    for (int k = tid; k < 8 * 8 * 3; k += kThreads) (&s.dnr[0][0][0])[k] = (&p.dnr[0][0][0])[k];
    for (int k = tid; k < 64; k += kThreads) (&s.W[0][0])[k] = (&p.W[0][0])[k];
    if (valid) {
        const int* cn = reinterpret_cast<const int*>(p.conn4) + 8 * e;
        const int64_t node = __ldg(cn + t), node0 = __ldg(cn);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            s.x[el][t][i] = stp(dd_from_double(__ldg(p.xyz + 3 * node + i) - __ldg(p.xyz + 3 * node0 + i)));
            s.u[el][t][i] = stp(dd_from_double(__ldg(p.u + 3 * node + i) - __ldg(p.u + 3 * node0 + i)));
        }
    }
    __syncthreads();
    if (valid) {
        const int g = t;
        dd J[3][3], G[3][3];
        {
            dd_acc aj[3][3], ag[3][3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int d = 0; d < 3; ++d) aj[i][d] = ag[i][d] = acc_zero();
            // corner loop kept rolled: the unrolled form overflows the instruction cache
#pragma unroll 1
            for (int a = 0; a < 8; ++a) {
                dd c[3], xa[3], ua[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    c[i] = ldp(s.dnr[g][a][i]);
                    xa[i] = ldp(s.x[el][a][i]);
                    ua[i] = ldp(s.u[el][a][i]);
                }
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        acc_fma(aj[i][d], xa[i], c[d]);
                        acc_fma(ag[i][d], ua[i], c[d]);
                    }
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    J[i][d] = acc_value(aj[i][d]);
                    G[i][d] = acc_value(ag[i][d]);
                }
        }
        dd A[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
                dd_acc acc = acc_zero();
                acc_fma(acc, J[i1][j1], J[i2][j2]);
                acc_fma(acc, dd_neg(J[i2][j1]), J[i1][j2]);
                A[j][i] = acc_value(acc);
            }
        dd_acc da = acc_zero();
        acc_fma(da, J[0][0], A[0][0]);
        acc_fma(da, J[1][0], A[0][1]);
        acc_fma(da, J[2][0], A[0][2]);
        const dd inv = dd_rcp(acc_value(da));
        dd H[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                dd_acc acc = acc_zero();
                acc_fma(acc, G[i][0], A[0][k]);
                acc_fma(acc, G[i][1], A[1][k]);
                acc_fma(acc, G[i][2], A[2][k]);
                H[i][k] = dd_mul(acc_value(acc), inv);
            }
        const dd D0d = ldp(p.D0d), lam = ldp(p.lam), mu = ldp(p.mu);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            dd_acc acc = acc_zero();
            acc_fma(acc, D0d, H[i][i]);
            acc_fma(acc, lam, H[(i + 1) % 3][(i + 1) % 3]);
            acc_fma(acc, lam, H[(i + 2) % 3][(i + 2) % 3]);
            s.sv[el][g][i] = stp(acc_value(acc));
        }
        s.sv[el][g][3] = stp(dd_mul(mu, dd_add(H[0][1], H[1][0])));
        s.sv[el][g][4] = stp(dd_mul(mu, dd_add(H[1][2], H[2][1])));
        s.sv[el][g][5] = stp(dd_mul(mu, dd_add(H[0][2], H[2][0])));
    }
    __syncthreads();
    // the table's distinct rows only, spread over the element's threads (as the FP64 kernel)
    if (valid) {
        const int nout = p.nrow * 6;
        for (int o = t; o < nout; o += 8) {
            const int r = o / 6, c = o - 6 * r;
            dd_acc acc = acc_zero();
#pragma unroll
            for (int k = 0; k < 8; ++k) acc_fma(acc, ldp(s.W[r][k]), ldp(s.sv[el][k][c]));
            s.res[el][r][c] = stp(acc_value(acc));
        }
    }
    __syncthreads();
    if (!valid) return;
    const int j = t, r = p.row_of[j];
    const int64_t slot = p.ne_inv ? int64_t(__ldg(p.ne_inv + e * 8 + j)) : e * 8 + j;
    float2* o = p.rec + slot * 6;
#pragma unroll
    for (int c = 0; c < 6; ++c) o[c] = s.res[el][r][c];
}

// Cyclic Jacobi on a symmetric 3x3 in double-float; returns the eigenvalues descending.
__device__ void sym3_eig_desc_dd(dd (&a)[3][3], dd& p1, dd& p2, dd& p3) {
    for (int sweep = 0; sweep < 16; ++sweep) {
        const float off = fabsf(a[0][1].hi) + fabsf(a[0][2].hi) + fabsf(a[1][2].hi);
        const float dia = fabsf(a[0][0].hi) + fabsf(a[1][1].hi) + fabsf(a[2][2].hi);
        if (!(off > 0.f) || off <= 1.4210855e-14f * dia) break;  // 2^-46
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {
            const int pp = pq == 2 ? 1 : 0;
            const int qq = pq == 0 ? 1 : 2;
            const dd apq = a[pp][qq];
            if (apq.hi == 0.f) continue;
            const dd theta = dd_div(dd_sub(a[qq][qq], a[pp][pp]), dd_add(apq, apq));
            dd tt;
            if (fabsf(theta.hi) > 1e18f) {
                tt = dd_rcp(dd_add(theta, theta));
            } else {
                const dd r = dd_sqrt(dd_add(dd_mul(theta, theta), dd_from_float(1.f)));
                tt = dd_rcp(dd_add(dd_abs(theta), r));
                if (theta.hi < 0.f) tt = dd_neg(tt);
            }
            const dd c = dd_rcp(dd_sqrt(dd_add(dd_mul(tt, tt), dd_from_float(1.f))));
            const dd sn = dd_mul(tt, c);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const dd akp = a[k][pp], akq = a[k][qq];
                a[k][pp] = dd_sub(dd_mul(c, akp), dd_mul(sn, akq));
                a[k][qq] = dd_add(dd_mul(sn, akp), dd_mul(c, akq));
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const dd apk = a[pp][k], aqk = a[qq][k];
                a[pp][k] = dd_sub(dd_mul(c, apk), dd_mul(sn, aqk));
                a[qq][k] = dd_add(dd_mul(sn, apk), dd_mul(c, aqk));
            }
        }
    }
    dd e0 = a[0][0], e1 = a[1][1], e2 = a[2][2], tmp;
    if (dd_lt(e0, e1)) tmp = e0, e0 = e1, e1 = tmp;
    if (dd_lt(e1, e2)) tmp = e1, e1 = e2, e2 = tmp;
    if (dd_lt(e0, e1)) tmp = e0, e0 = e1, e1 = tmp;
    p1 = e0;
    p2 = e1;
    p3 = e2;
}

__global__ void __launch_bounds__(256) k_stress_node_dd(int64_t n_node, const int32_t* __restrict__ ne_ptr,
                                                        const int32_t* __restrict__ ne_list,
                                                        const int32_t* __restrict__ co_elem,
                                                        const float2* __restrict__ rec, int row_ordered,
                                                        double* __restrict__ out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_node) return;
    dd_acc acc[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] = acc_zero();
    const int ks = ne_ptr[i], ke = ne_ptr[i + 1];
    for (int k = ks; k < ke; ++k) {
        int64_t slot = k;  // row order: this node's corner records are contiguous
        if (!row_ordered) {
            const int ent = __ldg(ne_list + k);
            slot = int64_t(ent >> 3) * 8 + (ent & 7);
        }
        const float4* r = reinterpret_cast<const float4*>(rec + slot * 6);  // 48 bytes, 16-byte aligned
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float4 v = __ldg(r + q);
            acc_add(acc[2 * q], dd{v.x, v.y});
            acc_add(acc[2 * q + 1], dd{v.z, v.w});
        }
    }
    double* o = out + 10 * i;
    const int ce = co_elem[i];
    if (ce == 0) {  // 0 / 0 as the reference's average (POST_process.py:186)
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
#pragma unroll
        for (int c = 0; c < 10; ++c) o[c] = nan;
        return;
    }
    const dd inv = dd_rcp(dd_from_float(float(ce)));
    dd v[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] = dd_mul(acc_value(acc[c]), inv);
    // vector order [xx, yy, zz, xy, yz, xz] (POST_process.py:79-86)
    dd a[3][3] = {{v[0], v[3], v[5]}, {v[3], v[1], v[4]}, {v[5], v[4], v[2]}};
    dd p1, p2, p3;
    sym3_eig_desc_dd(a, p1, p2, p3);
    const dd d12 = dd_sub(p1, p2), d23 = dd_sub(p2, p3);
    // "VM" as written at POST_process.py:93-94: (p1-p2)^2 + (p2-p3)^2 + (p3-p2)^2
    const dd vm = dd_sqrt(dd_add(dd_mul(d12, d12), dd_add(dd_mul(d23, d23), dd_mul(d23, d23))));
#pragma unroll
    for (int c = 0; c < 6; ++c) o[c] = dd_to_double(v[c]);
    o[6] = dd_to_double(p1);
    o[7] = dd_to_double(p2);
    o[8] = dd_to_double(p3);
    o[9] = dd_to_double(vm);
}

void split2(double x, float2& o) {
    const float hi = float(x);
    o = make_float2(hi, float(x - double(hi)));
}

}  // namespace

int launch_stress_dd(const fem_mesh* mesh, const fem_material* mat, const double* u, const int32_t* co_elem,
                     const double* extrap, double* out, void* workspace, cudaStream_t st) {
    if (mesh->n_elem) {
        StressDdParams sp;
        sp.xyz = mesh->xyz;
        sp.conn4 = reinterpret_cast<const int4*>(mesh->conn);
        sp.u = u;
        sp.n_elem = mesh->n_elem;
        sp.ne_inv = mesh->ne_inv;
        sp.rec = static_cast<float2*>(workspace);
        const double EX = mat->EX, PO = mat->PO;
        split2(EX * (1 - PO) / (1 + PO) / (1 - 2 * PO), sp.D0d);  // POST_process.py:292-302
        split2(EX * PO / (1 + PO) / (1 - 2 * PO), sp.lam);
        split2(EX / 2 / (1 + PO), sp.mu);                          // :304-306
        const ShapeTables& T = shape_tables();
        for (int g = 0; g < 8; ++g)
            for (int a = 0; a < 8; ++a)
                for (int d = 0; d < 3; ++d) split2(T.dnr[g][a][d], sp.dnr[g][a][d]);
        // distinct rows of the table (exactly equal rows share one), split into float pairs
        std::memset(sp.W, 0, sizeof(sp.W));
        int first[8];  // the first corner of each distinct row
        sp.nrow = 0;
        for (int j = 0; j < 8; ++j) {
            int r = 0;
            while (r < sp.nrow && std::memcmp(extrap + 8 * first[r], extrap + 8 * j, sizeof(double) * 8) != 0) ++r;
            if (r == sp.nrow) {
                for (int k = 0; k < 8; ++k) split2(extrap[8 * j + k], sp.W[r][k]);
                first[r] = j;
                ++sp.nrow;
            }
            sp.row_of[j] = r;
        }
        const int64_t blocks = (mesh->n_elem + kEpc - 1) / kEpc;
        k_stress_element_dd<<<unsigned(blocks), kThreads, 0, st>>>(sp);
        FEM_LAUNCH_CHECK("k_stress_element_dd");
    }
    const int64_t blocks = (mesh->n_node + 255) / 256;
    k_stress_node_dd<<<unsigned(blocks), 256, 0, st>>>(mesh->n_node, mesh->ne_ptr, mesh->ne_list, co_elem,
                                                       static_cast<const float2*>(workspace),
                                                       mesh->ne_inv != nullptr, out);
    FEM_LAUNCH_CHECK("k_stress_node_dd");
    return FEM_OK;
}

}  // namespace fem
