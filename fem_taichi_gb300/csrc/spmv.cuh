// BSR (3x3 block) SpMV / SpMM device code shared by spmv.cu and pcg.cu.
//
// Vectors with nrhs right-hand sides are stored [n_brow][3][nrhs] (right-hand side
// fastest), so one block row's inputs/outputs for all RHS are contiguous.
//  * nrhs == 1: LPR lanes cooperate on one block row (lane = block slot), followed by an
//    xor-shuffle reduction of the three row sums; 32/LPR rows per warp.
//  * nrhs  > 1: lanes map to right-hand sides (32/nrhs rows per warp); each block's nine
//    values are loaded once per row group (broadcast) and applied to all RHS (the padded FP32
//    layout: spmm4_rows_epi).
// Rows are visited with a grid-stride loop so the grid can be sized in multiples of the SM
// count; a fixed grid gives a fixed row -> CTA mapping, hence deterministic partial sums.
#pragma once

#include "dot.cuh"
#include "fem_common.cuh"

namespace fem {

template <typename T>
struct BsrView {
    int64_t n;              // block rows
    const int32_t* indptr;  // [n+1]
    const int32_t* indices; // [nnzb]
    const T* vals;          // [nnzb][3][3] (BSR) or, per block row, [9][row length] (row-SoA)
    int rsoa;               // 1: row-SoA value layout; 2: row-SoA padded to 4-block multiples (FP32)
    int stream = 0;         // the values leave L2 first (value_stream; padded row-SoA only)
};

// Sum of d over the lanes of a warp that hold the same right-hand side (lane % R).  FP32 sums are joined on
// the FP32 pipes (the FP64 form's five adds and the conversions cost 16 FP64 cycles each per warp
// and SM).
template <int R>
__device__ __forceinline__ Dot<double> rhs_dot(Dot<double> d) {
#pragma unroll
    for (int off = 16; off >= R; off >>= 1) d.v += __shfl_xor_sync(0xffffffffu, d.v, off);
    return d;
}
template <int R>
__device__ __forceinline__ Dot<float> rhs_dot(Dot<float> d) {
#pragma unroll
    for (int off = 16; off >= R; off >>= 1)
        d.join(__shfl_xor_sync(0xffffffffu, d.s, off), __shfl_xor_sync(0xffffffffu, d.c, off),
               __shfl_xor_sync(0xffffffffu, d.d, off));
    return d;
}

// BsrView::rsoa for a fem_bsr layout code
inline int rsoa_kind(int layout) {
    return layout == FEM_LAYOUT_RSOA ? 1 : layout == FEM_LAYOUT_RSOA4 ? 2 : 0;
}

// address of value q (0..8) of the block in slot l of the row starting at rs with L blocks
template <typename T>
__device__ __forceinline__ const T* block_value(const BsrView<T>& A, int64_t rs, int L, int l, int q) {
    return A.rsoa ? A.vals + 9 * rs + int64_t(q) * L + l : A.vals + 9 * (rs + l) + q;
}

// (a0, a1, a2) += B x for the 3x3 block B whose values start at v (stride vs between them):
// nine chained fused multiply-adds, the product's only FP64 work (written as a sum of three
// products per row, it compiled to a multiply, two FMAs and an add: 12 instructions).
template <typename T>
__device__ __forceinline__ void block_fma3(const T* v, int64_t vs, T x0, T x1, T x2, T& a0, T& a1, T& a2) {
    a0 = fma(__ldg(v + 0 * vs), x0, a0);
    a1 = fma(__ldg(v + 3 * vs), x0, a1);
    a2 = fma(__ldg(v + 6 * vs), x0, a2);
    a0 = fma(__ldg(v + 1 * vs), x1, a0);
    a1 = fma(__ldg(v + 4 * vs), x1, a1);
    a2 = fma(__ldg(v + 7 * vs), x1, a2);
    a0 = fma(__ldg(v + 2 * vs), x2, a0);
    a1 = fma(__ldg(v + 5 * vs), x2, a1);
    a2 = fma(__ldg(v + 8 * vs), x2, a2);
}

// Sum over lanes l' with (l' / G) == (l / G) of a warp split into groups of G lanes.
template <int G, typename V>
__device__ __forceinline__ V group_sum(V v) {
#pragma unroll
    for (int off = G / 2; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Row epilogues.  The product kernels hand each finished row (and right-hand side k) to
// an epilogue: o is the index of the row's first component in the [n][3][R] vectors,
// `stride` = R, (a0, a1, a2) = (A x) of the row.

// y = A x, and dot += x_row . y_row when asked (PCG's p.q).
template <typename T>
struct StoreY {
    const T* x;
    T* y;
    bool want_dot;
    __device__ __forceinline__ void operator()(int64_t o, int stride, int, T a0, T a1, T a2, Dot<T>& dot) const {
        y[o] = a0;
        y[o + stride] = a1;
        y[o + 2 * stride] = a2;
        if (want_dot) {
            dot.add3(x[o], a0, x[o + stride], a1, x[o + 2 * stride], a2);
        }
    }
};

// The same with x of 4 floats a node (y of 3).
struct StoreYPad {
    const float* x;
    float* y;
    __device__ __forceinline__ void operator()(int64_t o, int, int, float a0, float a1, float a2, Dot<float>& dot) const {
        const float4 xr = __ldg(reinterpret_cast<const float4*>(x) + o / 3);
        y[o] = a0;
        y[o + 1] = a1;
        y[o + 2] = a2;
        dot.add3(xr.x, a0, xr.y, a1, xr.z, a2);
    }
};

// Whether A's values should be the first to leave L2 when it needs room.  An iteration reads them once and
// a handful of vectors several times; a matrix that does not fit pushes those out as well, one that fits
// would only be pushed out itself.  Microseconds an iteration of the FP32 solve with and without, one
// right-hand side: 65,000 nodes (63 MB of values) 25.9 and 22.9, 86,000 29.0 and 28.9, 97,000 30.6 and 33.7,
// 214,221 (200 MB) 50.5 and 58.3 (L2: 129 MB).  What else the iteration reads counts as well: at 65,000
// nodes 66.5 and 72.3 with eight right-hand sides, 353 and 372 with multigrid, whose transfers and
// coarse levels are about as large again.  The columns stay with the vectors: 52.3 with both streamed.
int value_stream(const fem_bsr* A, int nrhs, bool multigrid = false);

// The L2 policy of loads that are (first = 1) or are not the first to leave
__device__ __forceinline__ uint64_t l2_policy(int first) {
    uint64_t f, k;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(f));
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(k));
    return first ? f : k;
}
__device__ __forceinline__ float4 load_l2(const float4* p, uint64_t pol) {
    float4 v;
    asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "l"(pol));
    return v;
}

// Padded row-SoA FP32 product: each lane takes 4 consecutive slots of its row per step and
// reads each of the 9 values of those 4 blocks with one 16-byte load (rows, values and
// slot groups all start on 16-byte boundaries); padding blocks hold zeros.  kPad: x holds 4 floats a
// node, one 16-byte load per gather instead of three of 4 bytes.
// Bound by HBM once the row pointer, the columns and the gathers no longer wait for one another: the
// next row's columns and the pointer of the row after load while a row is summed (in line, 214,221 nodes took
// 45.6 us of 34 us of HBM time whatever the occupancy; the solve of which it is two thirds went from 69.5 to
// 66.3 us an iteration).
template <int LPR, bool kPad, typename Epi>
__device__ __forceinline__ Dot<float> spmv4_rows_epi(const BsrView<float>& A, const float* __restrict__ x,
                                                     const Epi& epi) {
    const int lane = threadIdx.x & 31;
    const int sub = lane / LPR, sl = lane % LPR;
    constexpr int RPW = 32 / LPR;
    const uint64_t pol = l2_policy(A.stream);
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t stride = ((int64_t(gridDim.x) * blockDim.x) >> 5) * RPW;
    Dot<float> dot;
    auto pointers = [&](int64_t row, int& rs, int& L) {
        rs = L = 0;
        if (row < A.n) {
            rs = __ldg(A.indptr + row);
            L = __ldg(A.indptr + row + 1) - rs;
        }
    };
    auto columns = [&](int rs, int L, int s) {
        return s < L ? __ldg(reinterpret_cast<const int4*>(A.indices + rs + s)) : make_int4(0, 0, 0, 0);
    };
    int rs, L, rs_next, L_next;
    int64_t row = warp * RPW + sub;
    pointers(row, rs, L);
    pointers(row + stride, rs_next, L_next);
    int4 c = columns(rs, L, 4 * sl);
    for (int64_t base = warp * RPW; base < A.n; base += stride, row += stride) {
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        auto step = [&](int s, const int4& cc4) {
            const float* v0 = A.vals + 9 * int64_t(rs) + s;
            const int cc[4] = {cc4.x, cc4.y, cc4.z, cc4.w};
            float4 w[9], xv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (kPad) {
                    xv[j] = __ldg(reinterpret_cast<const float4*>(x) + cc[j]);
                } else {
                    const float* xc = x + 3 * int64_t(cc[j]);
                    xv[j] = make_float4(xc[0], xc[1], xc[2], 0.f);
                }
            }
#pragma unroll
            for (int q = 0; q < 9; ++q) w[q] = load_l2(reinterpret_cast<const float4*>(v0 + int64_t(q) * L), pol);
            // the products of two slots in one chain, then added: with one chain over the row the product of
            // 8,125 rows is off by 8.5e-8 (rms), 6.7e-8 here (7.4e-8 with a sum per block added)
            return [=](float& b0, float& b1, float& b2) {
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    // component j of each value's float4 = slot s + j
                    auto pair = [&](int q, float b) {
                        const float v0 = j ? w[q].z : w[q].x, v1 = j ? w[q + 1].z : w[q + 1].x, v2 = j ? w[q + 2].z : w[q + 2].x;
                        const float u0 = j ? w[q].w : w[q].y, u1 = j ? w[q + 1].w : w[q + 1].y, u2 = j ? w[q + 2].w : w[q + 2].y;
                        float t = fmaf(v2, xv[j].z, fmaf(v1, xv[j].y, v0 * xv[j].x));
                        t = fmaf(u2, xv[j + 1].z, fmaf(u1, xv[j + 1].y, fmaf(u0, xv[j + 1].x, t)));
                        return b + t;
                    };
                    b0 = pair(0, b0);
                    b1 = pair(3, b1);
                    b2 = pair(6, b2);
                }
            };
        };
        int rs2, L2;
        int4 c_next;
        if (4 * sl < L) {
            const auto add = step(4 * sl, c);   // loads issued
            c_next = columns(rs_next, L_next, 4 * sl);
            pointers(row + 2 * stride, rs2, L2);
            add(a0, a1, a2);
        } else {
            c_next = columns(rs_next, L_next, 4 * sl);
            pointers(row + 2 * stride, rs2, L2);
        }
        for (int s = 4 * sl + 4 * LPR; s < L; s += 4 * LPR) step(s, columns(rs, L, s))(a0, a1, a2);
        a0 = group_sum<LPR>(a0);
        a1 = group_sum<LPR>(a1);
        a2 = group_sum<LPR>(a2);
        if (row < A.n && sl == 0) epi(3 * row, 1, 0, a0, a1, a2, dot);
        c = c_next;
        rs = rs_next;
        L = L_next;
        rs_next = rs2;
        L_next = L2;
    }
    return dot;
}

// One pass of A x over the rows assigned to this thread (LPR lanes per block row; one RHS);
// returns this lane's share of the epilogue's dot product.
template <typename T, int LPR, typename Epi>
__device__ __forceinline__ Dot<T> spmv1_rows_epi(const BsrView<T>& A, const T* __restrict__ x, const Epi& epi) {
    if constexpr (sizeof(T) == 4) {
        if (A.rsoa == 2) return spmv4_rows_epi<(LPR > 8 ? 8 : LPR), false>(A, x, epi);
    }
    const int lane = threadIdx.x & 31;
    const int sub = lane / LPR, sl = lane % LPR;
    constexpr int RPW = 32 / LPR;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    Dot<T> dot;
    for (int64_t base = warp * RPW; base < A.n; base += nwarps * RPW) {
        const int64_t row = base + sub;
        const bool valid = row < A.n;
        T a0 = 0, a1 = 0, a2 = 0;
        if (valid) {
            const int64_t rs = __ldg(A.indptr + row);
            const int L = __ldg(A.indptr + row + 1) - int(rs);
            const int64_t vs = A.rsoa ? int64_t(L) : 1;  // stride between the 9 values of a block
            for (int l = sl; l < L; l += LPR) {
                const int64_t c = __ldg(A.indices + rs + l);
                const T* v = block_value(A, rs, L, l, 0);
                const T x0 = x[3 * c], x1 = x[3 * c + 1], x2 = x[3 * c + 2];
                block_fma3(v, vs, x0, x1, x2, a0, a1, a2);
            }
        }
        a0 = group_sum<LPR>(a0);
        a1 = group_sum<LPR>(a1);
        a2 = group_sum<LPR>(a2);
        if (valid && sl == 0) epi(3 * row, 1, 0, a0, a1, a2, dot);
    }
    return dot;
}

// Many right-hand sides on the padded row-SoA FP32 copy, one block row per warp (256 threads a CTA).
// A row's values and columns are one contiguous piece each; cp.async brings them into the warp's
// shared-memory ring kStage - 1 rows ahead, so only the gathers of x wait on memory.  Lane = (slot group
// g of G, vector sub of LP): it takes 4 consecutive slots a step and V right-hand sides of them, so
// one load instruction fetches x of G blocks and one shared-memory load a value of 4 G slots.  At the end
// of a row the groups' sums are exchanged so that a lane adds only the right-hand sides it keeps
// (reduce-scatter), and right-hand side k's totals move to lane k.  A CTA takes eight consecutive rows
// at a time, for the x lines they share in L1.
// Bound by L1 (84 lines of x per 27-block row at R = 32) and the latency of the gathers.  Product of
// 137,781 rows at R = 32: 207 us with one right-hand side per lane and values loaded in line (1,188
// instructions a row, most of them addresses); 190 us with vectors of right-hand sides (560, every step
// waiting on values from HBM); 125 us staged, 119 us with the slot groups beyond a row's end left out.  L1
// capacity decides the rest: 2 rows staged and 2 CTAs an SM leave it 192 KB (3 rows: 156 us; 3 CTAs with
// p.q: 339 instead of 268 us an iteration of the solve);
// fewer right-hand sides gather less and take 3 CTAs (R = 8: 59 against 69 us).  V and G: 4-slot groups of a
// 28-slot row in 2 x 4 or 8 groups leave 1 in 8 idle, more groups would idle half.  kTwo: two sums a row
// and right-hand side, so that the chains are as short as block sums added were (8,125 rows against FP64:
// 7.1e-8 to 7.4e-8, 8.4e-8 with one; block sums 7.5e-8 to 8.5e-8, at R = 32, one group, 10.4e-8: there
// one is enough).  At R = 16 they leave V = 4 no third CTA: 84 us of 141,426 rows, 82 with V = 2.
template <int V>
struct alignas(4 * V) FloatVec {
    float v[V];
};
constexpr int kStage = 2;          // rows of a warp in shared memory
constexpr int kStageSlots = 32;    // longest staged row; longer ones are read in place
// CTAs per SM of the kernels around the products, for the compiler's registers (FP32: see spmm4_rows_epi,
// spmv4_rows_epi).  FP64 (bound by its pipe at 27 blocks a row): 4 for many right-hand sides with p.q, no bound
// otherwise.  With 1 it unrolls to 136 registers (product of 66,411 rows, 32 right-hand sides: 1.76 ms against
// 1.71); 65,331 rows, 8 right-hand sides: product 219 us without a bound and 222 with 4, solver iteration
// 299 and 287.
template <typename T, int R, bool kDot = false>
constexpr int spmm_ctas() {
    return sizeof(T) == 8 ? (kDot && R > 1 ? 4 : 0) : R == 1 ? 1 : R == 32 ? 2 : 3;
}

__device__ __forceinline__ void copy_async16(void* dst, const void* src, uint64_t pol) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(
                     unsigned(__cvta_generic_to_shared(dst))), "l"(src), "l"(pol) : "memory");
}
__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(unsigned(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

template <int R, typename Epi>
__device__ __forceinline__ Dot<float> spmm4_rows_epi(const BsrView<float>& A, const float* __restrict__ x, const Epi& epi) {
    constexpr int V = R >= 32 ? 4 : R >= 8 ? 2 : 1, LP = R / V, G = 32 / LP, CS = 4 * G;
    constexpr bool kTwo = R < 32;
    constexpr unsigned full = 0xffffffffu;
    constexpr int kWarps = 8;
    struct Stage {
        float val[9 * kStageSlots];
        int32_t col[kStageSlots];
    };
    __shared__ __align__(16) Stage ring[kWarps][kStage];
    using X = FloatVec<V>;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int g = lane / LP, sub = lane % LP;
    const uint64_t pol = l2_policy(A.stream);
    Dot<float> dot;
    const int64_t first = int64_t(blockIdx.x) * kWarps + wid, stride = int64_t(gridDim.x) * kWarps;
    const int steps = first < A.n ? int((A.n - first + stride - 1) / stride) : 0;

    int32_t rp = 0, rp1 = 0;  // row pointers of the warp's rows, 32 steps at a time
    int64_t rs[kStage];
    int len[kStage];
#pragma unroll
    for (int d = 0; d < kStage; ++d) rs[d] = 0, len[d] = 0;
    // row of step t into slot t % kStage of the ring; rs / len are shifted by the caller
    auto fetch = [&](int t, int64_t& r0, int& L) {
        r0 = 0;
        L = 0;
        if (t < steps) {
            if ((t & 31) == 0) {
                const int64_t row = first + stride * (t + lane);
                rp = rp1 = 0;
                if (row < A.n) {
                    rp = __ldg(A.indptr + row);
                    rp1 = __ldg(A.indptr + row + 1);
                }
            }
            r0 = __shfl_sync(full, rp, t & 31);
            L = __shfl_sync(full, rp1, t & 31) - int(r0);
            if (L <= kStageSlots) {
                Stage& st = ring[wid][t % kStage];
                const float* v = A.vals + 9 * r0;
#pragma unroll
                for (int i = 0; i < 9 * kStageSlots / 4; i += 32)
                    if (i + lane < 9 * L / 4) copy_async16(st.val + 4 * (i + lane), v + 4 * (i + lane), pol);
                if (lane < L / 4) copy_async16(st.col + 4 * lane, A.indices + r0 + 4 * lane);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int d = 0; d < kStage - 1; ++d) fetch(d, rs[d], len[d]);
    for (int t = 0; t < steps; ++t) {
        fetch(t + kStage - 1, rs[kStage - 1], len[kStage - 1]);
        asm volatile("cp.async.wait_group %0;" ::"n"(kStage - 1) : "memory");
        __syncwarp();   // every lane's copies of this row have landed
        const int64_t row = first + stride * t;
        const int Lp = len[0];
        const Stage& st = ring[wid][t % kStage];
        float acc[3][V], odd[3][V];   // kTwo: of slots 0, 1 and 2, 3 of every four
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < V; ++i) acc[j][i] = odd[j][i] = 0.f;
        // 4 slots, values and columns from `val` and `col`; the groups beyond the row's end sit out
        auto step = [&](int s, const float* val, const int32_t* col) {
            const int4 idx = *reinterpret_cast<const int4*>(col + s);
            X xv[4][3];
            const int cc[4] = {idx.x, idx.y, idx.z, idx.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float* xc = x + int64_t(cc[u]) * (3 * R) + sub * V;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    if constexpr (V == 4) {
                        const float4 f = __ldg(reinterpret_cast<const float4*>(xc + j * R));
                        xv[u][j].v[0] = f.x, xv[u][j].v[1] = f.y, xv[u][j].v[2] = f.z, xv[u][j].v[3] = f.w;
                    } else if constexpr (V == 2) {
                        const float2 f = __ldg(reinterpret_cast<const float2*>(xc + j * R));
                        xv[u][j].v[0] = f.x, xv[u][j].v[1] = f.y;
                    } else {
                        xv[u][j].v[0] = __ldg(xc + j * R);
                    }
                }
            }
            const float* vs = val + s;
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const float4 w = *reinterpret_cast<const float4*>(vs + (3 * j + c) * Lp);
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        acc[j][i] = fmaf(w.x, xv[0][c].v[i], acc[j][i]);
                        acc[j][i] = fmaf(w.y, xv[1][c].v[i], acc[j][i]);
                        float& a = kTwo ? odd[j][i] : acc[j][i];
                        a = fmaf(w.z, xv[2][c].v[i], a);
                        a = fmaf(w.w, xv[3][c].v[i], a);
                    }
                }
        };
        if (Lp <= kStageSlots) {
#pragma unroll 1
            for (int s = 4 * g; s < Lp; s += CS) step(s, st.val, st.col);
        } else {
#pragma unroll 1
            for (int s = 4 * g; s < Lp; s += CS) step(s, A.vals + 9 * rs[0], A.indices + rs[0]);
        }
        __syncwarp();   // the ring slot may be refilled
        if constexpr (kTwo) {
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int i = 0; i < V; ++i) acc[j][i] += odd[j][i];
        }
        // reduce-scatter: after a level with offset off, lane keeps half of its right-hand sides
        int off = LP;
#pragma unroll
        for (int keep = V / 2; keep >= 1; keep >>= 1, off <<= 1) {
            const bool hi = (lane & off) != 0;
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int i = 0; i < keep; ++i) {
                    const float send = hi ? acc[j][i] : acc[j][i + keep];
                    const float mine = hi ? acc[j][i + keep] : acc[j][i];
                    acc[j][i] = mine + __shfl_xor_sync(full, send, off);
                }
        }
        float a[3] = {acc[0][0], acc[1][0], acc[2][0]};
#pragma unroll
        for (; off < 32; off <<= 1)
#pragma unroll
            for (int j = 0; j < 3; ++j) a[j] += __shfl_xor_sync(full, a[j], off);
        // right-hand side k stays with vector k / V, on the lane whose scatter bits (high half first) are
        // the bits of k % V
        const int k = lane % R;
        if constexpr (V > 1) {
            const int src = (V == 4 ? ((k >> 1) & 1) + 2 * (k & 1) : k & 1) * LP + k / V;
#pragma unroll
            for (int j = 0; j < 3; ++j) a[j] = __shfl_sync(full, a[j], src);
        }
        if (lane < R) epi(3 * row * R + k, R, k, a[0], a[1], a[2], dot);
#pragma unroll
        for (int d = 0; d < kStage - 1; ++d) rs[d] = rs[d + 1], len[d] = len[d + 1];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    return dot;
}

// Many right-hand sides: lane = RHS (32 / R rows per warp), each block's values loaded once
// per row group and applied to every RHS.
template <typename T, int R, typename Epi>
__device__ __forceinline__ Dot<T> spmm_rows_epi(const BsrView<T>& A, const T* __restrict__ x, const Epi& epi) {
    if constexpr (sizeof(T) == 4) {
        // the vector loads of x need its rows on 16-byte boundaries (a caller's x may be a view)
        if (A.rsoa == 2 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0) return spmm4_rows_epi<R>(A, x, epi);
    }
    const int lane = threadIdx.x & 31;
    const int sub = lane / R, rhs = lane % R;
    constexpr int RPW = 32 / R;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    Dot<T> dot;
    for (int64_t base = warp * RPW; base < A.n; base += nwarps * RPW) {
        const int64_t row = base + sub;
        if (row >= A.n) continue;
        const int64_t rs = __ldg(A.indptr + row);
        const int L = __ldg(A.indptr + row + 1) - int(rs);
        T a0 = 0, a1 = 0, a2 = 0;
        const int64_t vs = A.rsoa ? int64_t(L) : 1;
#pragma unroll 3
        for (int l = 0; l < L; ++l) {
            const int64_t c = __ldg(A.indices + rs + l);
            const T* v = block_value(A, rs, L, l, 0);
            const T* xc = x + 3 * c * R + rhs;
            const T x0 = xc[0], x1 = xc[R], x2 = xc[2 * R];
            block_fma3(v, vs, x0, x1, x2, a0, a1, a2);
        }
        epi(3 * row * R + rhs, R, rhs, a0, a1, a2, dot);
    }
    return dot;
}

// y = A x forms of the three products (dot: sum_rows x_i . y_i when want_dot).
template <typename T, int LPR>
__device__ __forceinline__ Dot<T> spmv1_rows(const BsrView<T>& A, const T* __restrict__ x, T* __restrict__ y,
                                             bool want_dot) {
    return spmv1_rows_epi<T, LPR>(A, x, StoreY<T>{x, y, want_dot});
}

template <typename T, int R>
__device__ __forceinline__ Dot<T> spmm_rows(const BsrView<T>& A, const T* __restrict__ x, T* __restrict__ y,
                                            bool want_dot) {
    return spmm_rows_epi<T, R>(A, x, StoreY<T>{x, y, want_dot});
}

// SpMV launch variants picked by the autotuner (nrhs == 1): lanes per block row and CTA size.
struct SpmvVariant {
    int lpr;      // 32, 16 or 8 lanes per block row
    int threads;  // CTA size
    int ctas_per_sm;
};
constexpr int kNumSpmvVariants = 8;
__host__ __device__ inline SpmvVariant spmv_variant(int id) {
    const SpmvVariant v[kNumSpmvVariants] = {{32, 256, 8}, {16, 256, 8}, {8, 256, 8},  {32, 512, 4},
                                             {16, 128, 16}, {8, 512, 4},  {4, 256, 8}, {2, 256, 8}};
    return v[(id >= 0 && id < kNumSpmvVariants) ? id : 0];
}

int sm_count();
// CTAs of `kernel` resident on one SM with `threads` threads and `smem` bytes of dynamic shared
// memory (occupancy query, cached per kernel, CTA shape and device).
int resident_ctas(const void* kernel, int threads, size_t smem);
// Grid for a grid-stride kernel: min(need, cap, one wave of resident CTAs on every SM).
unsigned resident_grid(const void* kernel, int threads, int64_t need, int64_t cap);

}  // namespace fem
