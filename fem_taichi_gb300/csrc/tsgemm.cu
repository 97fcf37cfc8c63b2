// Tall-skinny FP64 products of the block-Lanczos modal solve (SOLVE_eigen.py:65-84):
// the reorthogonalisation w -= Q (Q^T M w) and the Ritz vectors X = Q V, with Q an n x m
// block of Lanczos vectors (n ~ 10^5..10^7 rows, m <= a few hundred columns) and w, M w
// n x b blocks (b <= 32).  No reference counterpart on the GPU (the reference runs these as
// numpy GEMMs on the host).
//
//  k_ts_tn_partial / k_ts_tn_reduce: C (m x b) = Q^T X, m <= 256.  CTA k of G takes the rows
//    [k n / G, (k + 1) n / G) -- the same number to within one, so no SM runs a chunk more than the
//    others -- in chunks of kChunk; it stages a chunk's X rows in shared memory and thread j
//    accumulates column j of Q (coalesced loads along a row of Q) against all b columns of X.  The
//    per-CTA partials are summed in a fixed order (deterministic): kSeg warps of a block each sum
//    a consecutive share of the CTAs for 32 outputs, loads running ahead, then the shares in order.
//  k_ts_nn: W = beta W + alpha Q C (C m x b staged in shared memory): one thread per row of Q and one
//    or two columns of W; a warp reads Q 32 x 32 values at a time, coalesced, into its own shared-memory
//    tile, the next tile's loads in flight.
// FP64 throughout and bound by the FP64 pipe (n m b FMAs each: 199 us at 65,559 x 190 x 10), so the
// column count of X is a template width close to b (4, 8, 10, 12, 16, 24, 32) rather than a power of
// two: padded columns would be FMAs on zeros.  At that size the products took 251 + 84 us (whole
// chunks per CTA: 4 on some SMs, 3 on others; one thread summing 513 partials) and 479 us (a warp per
// row, lanes over the columns: the butterfly adds of 10 sums were as many FP64 instructions as the FMAs);
// now 215 + 15 and 298 us.
#include <algorithm>
#include <type_traits>

#include "fem_common.cuh"

namespace fem {
int sm_count();
namespace {

constexpr int kChunk = 64;     // rows per step of the transposed product
constexpr int kTsThreads = 256;
constexpr int kMaxCols = 256;  // columns of Q per launch (one per thread)
constexpr int kSeg = 8;        // warps that share the sum over the CTAs of one output
constexpr int kNnThreads = 64;

template <int B>
__global__ void __launch_bounds__(kTsThreads) k_ts_tn_partial(int64_t n, int m, int b, const double* __restrict__ Q,
                                                                int64_t ldq, const double* __restrict__ X, int64_t ldx,
                                                                double* part) {
    __shared__ double xs[kChunk][B];
    const int j = threadIdx.x;  // column of Q (m <= kMaxCols)
    double acc[B];
#pragma unroll
    for (int c = 0; c < B; ++c) acc[c] = 0.0;
    const int64_t end = n * (int64_t(blockIdx.x) + 1) / gridDim.x;
    for (int64_t r0 = n * int64_t(blockIdx.x) / gridDim.x; r0 < end; r0 += kChunk) {
        const int rows = int(std::min<int64_t>(kChunk, end - r0));
        __syncthreads();
        for (int i = threadIdx.x; i < kChunk * B; i += kTsThreads) {
            const int r = i / B, c = i % B;
            xs[r][c] = (r < rows && c < b) ? X[(r0 + r) * ldx + c] : 0.0;
        }
        __syncthreads();
        if (j < m) {
            const double* q = Q + r0 * ldq + j;
#pragma unroll 4
            for (int r = 0; r < rows; ++r) {
                const double qv = __ldg(q + int64_t(r) * ldq);
#pragma unroll
                for (int c = 0; c < B; ++c) acc[c] = fma(qv, xs[r][c], acc[c]);
            }
        }
    }
    if (j < m) {
        double* o = part + (int64_t(blockIdx.x) * m + j) * B;
#pragma unroll
        for (int c = 0; c < B; ++c) o[c] = acc[c];
    }
}

// C[j][c] = sum over CTAs of the partials: warp w of a block adds the CTAs [w, w + 1) nblocks / kSeg in
// order for 32 consecutive outputs, then the kSeg sums are added in order.
template <int B>
__global__ void __launch_bounds__(kSeg * 32) k_ts_tn_reduce(int m, int b, int nblocks, const double* __restrict__ part,
                                                             double* C, int64_t ldc) {
    __shared__ double seg[kSeg][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t total = int64_t(m) * B, i = int64_t(blockIdx.x) * 32 + lane;
    double s = 0.0;
    if (i < total) {
        const int k1 = nblocks * (w + 1) / kSeg;
#pragma unroll 8
        for (int k = nblocks * w / kSeg; k < k1; ++k) s += __ldg(part + int64_t(k) * total + i);
    }
    seg[w][lane] = s;
    __syncthreads();
    const int j = int(i / B), c = int(i - int64_t(j) * B);
    if (w || i >= total || c >= b) return;
#pragma unroll
    for (int k = 1; k < kSeg; ++k) s += seg[k][lane];
    C[int64_t(j) * ldc + c] = s;
}

// Columns [B blockIdx.y, B (blockIdx.y + 1)) of W.  A row's sum over the m columns of Q is a tree down to
// chains of four, not one chain: with m = 190 random terms its rms error is 1.4e-16 of the sum, 4.6e-16 as
// a chain (1.45e-16 as 32 lanes and a butterfly).  The tree adds a quarter to the FP64 instructions.
// kSplit: the CTA's two warps share 32 rows, one takes every other tile of 32 columns; the two totals
// of a row are the same sums either way.
template <int B, bool kSplit>
__global__ void __launch_bounds__(kNnThreads) k_ts_nn(int64_t n, int m, int b, const double* __restrict__ Q,
                                                        int64_t ldq, const double* __restrict__ C, int64_t ldc,
                                                        double alpha, double beta, double* W, int64_t ldw) {
    extern __shared__ double cs[];  // [m rounded up to 8][B], then a 32 x 33 tile per warp
    const int m8 = (m + 7) & ~7, c0 = blockIdx.y * B, bs = min(B, b - c0);
    for (int i = threadIdx.x; i < m8 * B; i += kNnThreads) {
        const int j = i / B, c = i % B;
        cs[i] = j < m && c < bs ? C[int64_t(j) * ldc + c0 + c] : 0.0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* tile = cs + m8 * B + warp * (32 * 33);
    constexpr int kStep = kSplit ? 64 : 32, kRows = kSplit ? 32 : kNnThreads;   // a CTA's rows
    for (int64_t r0 = int64_t(blockIdx.x) * kRows + (kSplit ? 0 : 32 * warp); r0 < n; r0 += int64_t(gridDim.x) * kRows) {
        const int rows = int(std::min<int64_t>(32, n - r0));
        const int first = kSplit ? 32 * warp : 0;
        double even[B], odd[B], q[32];   // sums over every other tile of 32 columns
#pragma unroll
        for (int c = 0; c < B; ++c) even[c] = odd[c] = 0.0;
        auto load = [&](int j0) {
            const double* p = Q + r0 * ldq + j0 + lane;
#pragma unroll
            for (int r = 0; r < 32; ++r) q[r] = r < rows && j0 + lane < m ? __ldg(p + int64_t(r) * ldq) : 0.0;
        };
        load(first);
        for (int j0 = first; j0 < m; j0 += kStep) {
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 32; ++r) tile[r * 33 + lane] = q[r];
            __syncwarp();
            if (j0 + kStep < m) load(j0 + kStep);
            const double* cj = cs + j0 * B;
            const double* tl = tile + lane * 33;
            const int nj = min(32, m8 - j0);
            auto four = [&](int j, double (&s)[B]) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double qv = tl[j + k];
#pragma unroll
                    for (int c = 0; c < B; ++c) s[c] = k ? fma(qv, cj[(j + k) * B + c], s[c]) : qv * cj[j * B + c];
                }
            };
            double t[B];
#pragma unroll 1
            for (int h = 0; h < nj; h += 16) {
                double x[B], y[B];
                four(h, x);
                four(h + 4, y);
#pragma unroll
                for (int c = 0; c < B; ++c) x[c] += y[c];
                if (h + 8 < nj) {
                    double z[B];
                    four(h + 8, y);
                    four(h + 12, z);
#pragma unroll
                    for (int c = 0; c < B; ++c) x[c] += y[c] + z[c];
                }
#pragma unroll
                for (int c = 0; c < B; ++c) t[c] = h ? t[c] + x[c] : x[c];
            }
#pragma unroll
            for (int c = 0; c < B; ++c) {
                const double v = even[c] + t[c];
                even[c] = kSplit ? v : odd[c];
                odd[c] = kSplit ? 0.0 : v;
            }
        }
        if constexpr (kSplit) {   // warp 1's total to warp 0, through the front of its own tile
            __syncwarp();
            if (warp == 1)
#pragma unroll
                for (int c = 0; c < B; ++c) tile[c * 32 + lane] = even[c];
            __syncthreads();
            if (warp == 0)
#pragma unroll
                for (int c = 0; c < B; ++c) odd[c] = tile[32 * 33 + c * 32 + lane];
            __syncthreads();
        }
        if (lane < rows && !(kSplit && warp)) {
            double* w = W + (r0 + lane) * ldw + c0;
#pragma unroll
            for (int c = 0; c < B; ++c) {
                const double v = even[c] + odd[c];
                if (c < bs) w[c] = beta == 0.0 ? alpha * v : fma(alpha, v, beta * w[c]);
            }
        }
    }
}

int tn_grid(int64_t n) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // four CTAs an SM; short problems take CTAs of at least 16 rows
    return int(std::max<int64_t>(1, std::min<int64_t>((n + 15) / 16, int64_t(sms) * 4)));
}

template <int B>
int ts_tn(int64_t n, int m, int b, const double* Q, int64_t ldq, const double* X, int64_t ldx, double* C,
          int64_t ldc, double* ws, cudaStream_t st) {
    const int blocks = tn_grid(n);
    k_ts_tn_partial<B><<<unsigned(blocks), kTsThreads, 0, st>>>(n, m, b, Q, ldq, X, ldx, ws);
    FEM_LAUNCH_CHECK("k_ts_tn_partial");
    k_ts_tn_reduce<B><<<unsigned((int64_t(m) * B + 31) / 32), kSeg * 32, 0, st>>>(m, b, blocks, ws, C, ldc);
    FEM_LAUNCH_CHECK("k_ts_tn_reduce");
    return FEM_OK;
}

template <int B, bool kSplit>
int ts_nn(int64_t n, int m, int b, const double* Q, int64_t ldq, const double* C, int64_t ldc, double alpha,
          double beta, double* W, int64_t ldw, cudaStream_t st) {
    const size_t smem = (size_t((m + 7) & ~7) * B + (kNnThreads / 32) * 32 * 33) * sizeof(double);
    const int64_t rows = kSplit ? 32 : kNnThreads;
    const dim3 grid(unsigned(std::min<int64_t>((n + rows - 1) / rows, int64_t(1) << 20)), (b + B - 1) / B);
    k_ts_nn<B, kSplit><<<grid, kNnThreads, smem, st>>>(n, m, b, Q, ldq, C, ldc, alpha, beta, W, ldw);
    FEM_LAUNCH_CHECK("k_ts_nn");
    return FEM_OK;
}

int width(int b) { return b <= 4 ? 4 : b <= 8 ? 8 : b <= 10 ? 10 : b <= 12 ? 12 : b <= 16 ? 16 : b <= 24 ? 24 : 32; }

}  // namespace
}  // namespace fem

using namespace fem;

extern "C" size_t fem_ts_gemm_tn_workspace_bytes(int64_t n, int m, int b) {
    if (n <= 0 || m <= 0 || m > kMaxCols || b <= 0 || b > 32) return 0;
    return size_t(tn_grid(n)) * size_t(m) * width(b) * sizeof(double);
}

extern "C" int fem_ts_gemm_tn(int64_t n, int m, int b, const double* Q, int64_t ldq, const double* X, int64_t ldx,
                              double* C, int64_t ldc, void* workspace, size_t workspace_bytes, void* stream) {
    FEM_REQUIRE(n > 0 && m > 0 && m <= kMaxCols && b > 0 && b <= 32 && Q && X && C && workspace, "bad arguments");
    FEM_REQUIRE(ldq >= m && ldx >= b && ldc >= b, "leading dimensions too small");
    if (workspace_bytes < fem_ts_gemm_tn_workspace_bytes(n, m, b)) {
        set_error("workspace too small: need %zu bytes", fem_ts_gemm_tn_workspace_bytes(n, m, b));
        return FEM_ERR_WORKSPACE;
    }
    cudaStream_t st = as_stream(stream);
    double* ws = static_cast<double*>(workspace);
    auto run = [&](auto width_c) {
        return ts_tn<decltype(width_c)::value>(n, m, b, Q, ldq, X, ldx, C, ldc, ws, st);
    };
    switch (width(b)) {
        case 4: return run(std::integral_constant<int, 4>());
        case 8: return run(std::integral_constant<int, 8>());
        case 10: return run(std::integral_constant<int, 10>());
        case 12: return run(std::integral_constant<int, 12>());
        case 16: return run(std::integral_constant<int, 16>());
        case 24: return run(std::integral_constant<int, 24>());
        default: return run(std::integral_constant<int, 32>());
    }
}

extern "C" int fem_ts_gemm_nn(int64_t n, int m, int b, const double* Q, int64_t ldq, const double* C, int64_t ldc,
                              double alpha, double beta, double* W, int64_t ldw, void* stream) {
    FEM_REQUIRE(n > 0 && m > 0 && m <= kMaxCols && b > 0 && b <= 32 && Q && C && W, "bad arguments");
    FEM_REQUIRE(ldq >= m && ldc >= b && ldw >= b, "leading dimensions too small");
    cudaStream_t st = as_stream(stream);
    // An SM sub-partition takes one FP64 warp instruction every 64 cycles, so the time is that of the
    // sub-partition with the most (32 rows, column) warps, and of one warp's chain when there are few.  parts:
    // sub-partitions (608).  Two warps a row group (times in us, m = 190) at 2,100 x 16 (1.7 warps each) 22.8
    // against 24.9, at 4,200 x 10 (2.2) 33.1 against 28.9; two columns a warp at 8,400 x 8 (3.5) 41.3 against
    // 37.3, at 8,400 x 10 (4.3) 49.3 against 76.0 (a second wave of CTAs), at 65,559 x 10 298 against 312.  An odd
    // b pads a column: 65,559 x 3 127 against 115, but 13,000 x 9 (6.0) 67.9 against 78.0.  Wider columns were
    // slower throughout (65,559 x 10 in one: 340).
    const int64_t warps = (n + 31) / 32 * b, parts = 4 * int64_t(sm_count());
    if (4 * warps <= 7 * parts) return ts_nn<1, true>(n, m, b, Q, ldq, C, ldc, alpha, beta, W, ldw, st);
    if (warps <= 4 * parts || (b % 2 && warps > 8 * parts))
        return ts_nn<1, false>(n, m, b, Q, ldq, C, ldc, alpha, beta, W, ldw, st);
    return ts_nn<2, false>(n, m, b, Q, ldq, C, ldc, alpha, beta, W, ldw, st);
}
