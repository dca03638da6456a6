// Single-precision arithmetic on pairs (sm_100a).
#pragma once

namespace ffcvb {

// Two floats per register pair, and two operations per instruction.
struct Two {
    static constexpr int width = 2;
    unsigned long long v;
    __device__ __forceinline__ Two() {}
    __device__ __forceinline__ Two(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
    __device__ __forceinline__ float lo() const { return half(0); }
    __device__ __forceinline__ float hi() const { return half(1); }
    __device__ __forceinline__ float half(int k) const {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        return k ? b : a;
    }
};
__device__ __forceinline__ Two fma_rn(Two a, Two b, Two c) {
    Two r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Two fma_rd(Two a, Two b, Two c) {
    Two r;
    asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Two add_rn(Two a, Two b) {
    Two r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Two sub_rn(Two a, Two b) {
    Two r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Two add_rd(Two a, Two b) {
    Two r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// One float, for what is written for either.
struct One {
    static constexpr int width = 1;
    float v;
    __device__ __forceinline__ One() {}
    __device__ __forceinline__ One(float lo, float) : v(lo) {}
    __device__ __forceinline__ float lo() const { return v; }
    __device__ __forceinline__ float hi() const { return v; }
};
__device__ __forceinline__ One fma_rn(One a, One b, One c) { return One(__fmaf_rn(a.v, b.v, c.v), 0.f); }
__device__ __forceinline__ One fma_rd(One a, One b, One c) { return One(__fmaf_rd(a.v, b.v, c.v), 0.f); }
__device__ __forceinline__ One add_rn(One a, One b) { return One(__fadd_rn(a.v, b.v), 0.f); }
__device__ __forceinline__ One add_rd(One a, One b) { return One(__fadd_rd(a.v, b.v), 0.f); }
__device__ __forceinline__ One mul_rn(One a, One b) { return One(__fmul_rn(a.v, b.v), 0.f); }
// (as a sum with zero: a product that is added next may be contracted into one rounding, which must not happen)
__device__ __forceinline__ Two mul_rn(Two a, Two b) { return fma_rn(a, b, Two(0.f, 0.f)); }

} // namespace ffcvb
