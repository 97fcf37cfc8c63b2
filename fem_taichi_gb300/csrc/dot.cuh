// Dot-product accumulators of the solver.  Plain arithmetic on its own: a host compiler takes this file with
// the CUDA rounding intrinsics defined.
#pragma once

namespace fem {

// FP64 vectors: plain FP64 fused multiply-adds.
// FP32 vectors: every product is formed exactly (FMA error term) and summed with compensated two-sums in
// FP32 (add: pairs, about 48 significant bits), and becomes a double once per warp, so the
// per-element work stays on the FP32 pipes (GB300's FP64 pipe is ~64x slower) while the dot products
// keep FP64-class accuracy.  Sums of sums (join: over a thread's nodes, over the lanes of a warp) carry a
// third float, so that they lose less than FP64 additions would: with pairs only, the sum of 214,221
// nodes' products of mixed sign was off by 5.3e-15 of its value (rms), 1.5e-15 with join, the same as with
// each thread's pair converted and added in FP64.
template <typename T>
struct Dot {
    double v = 0.0;
    __device__ __forceinline__ void add(T a, T b) { v = fma(double(a), double(b), v); }
    // the three components of a node
    __device__ __forceinline__ void add3(T a0, T b0, T a1, T b1, T a2, T b2) {
        add(a0, b0);
        add(a1, b1);
        add(a2, b2);
    }
    __device__ __forceinline__ double value() const { return v; }
};
template <>
struct Dot<float> {
    float s = 0.f, c = 0.f, d = 0.f;
    __device__ __forceinline__ static float two_sum(float& s, float x) {  // s += x; returns the rounding error
        const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
        const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z));
        s = t;
        return e;
    }
    __device__ __forceinline__ void add(float a, float b) {
        const float pr = __fmul_rn(a, b);
        const float e = __fmaf_rn(a, b, -pr);
        const float err = two_sum(s, pr);
        c = __fadd_rn(c, __fadd_rn(err, e));
    }
    // += the sum (s2, c2, d2)
    __device__ __forceinline__ void join(float s2, float c2, float d2) {
        const float e1 = two_sum(s, s2), e2 = two_sum(c, c2), e3 = two_sum(c, e1);
        d = __fadd_rn(__fadd_rn(d, d2), __fadd_rn(e2, e3));
    }
    __device__ __forceinline__ void add3(float a0, float b0, float a1, float b1, float a2, float b2) {
        Dot n;
        n.s = __fmul_rn(a0, b0);
        n.c = __fmaf_rn(a0, b0, -n.s);
        n.add(a1, b1);
        n.add(a2, b2);
        join(n.s, n.c, 0.f);
    }
    __device__ __forceinline__ double value() const { return double(s) + (double(c) + double(d)); }
};

}  // namespace fem
