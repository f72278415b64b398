// Device helpers shared by the plain (lattice.cu) and the ordered (ordered.cu)
// filter.
#pragma once
#include "lattice.cuh"

namespace dcrf {

namespace {

constexpr int kRes = 10;         // RESOLUTION (include/permutohedral.h:41)
constexpr int kOrdW = 2 * kRes;  // lower + upper bins per (vertex, label)
constexpr int kLongList = 64;    // lists longer than this use the staged warp kernels
constexpr int kHugeList = 1024;  // lists longer than this get a block (plain) or the finest split (ordered splat)
constexpr int kTB = 256;         // threads per block of the element-wise kernels
constexpr int kSegPad = 4;       // entries past the splat lists' end that a paired load may touch

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp_async4(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// a + w x per half, the product and the sum each rounded: scalar products and
// a packed sum.  A packed product feeding a packed sum was measured to come
// out as one fused multiply-add (rounded once), which the reference's SSE2
// arithmetic does not do.
__device__ __forceinline__ unsigned long long add_mul2(unsigned long long a, float w, unsigned long long x) {
    const float2 f = unpack2(x);
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(pack2(fmul(w, f.x), fmul(w, f.y))));
    return r;
}

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}

// A splat list's entry is (pixel, weight bits).
__device__ __forceinline__ float entry_w(int2 e) { return __int_as_float(e.y); }

__device__ __forceinline__ float apply_epilogue(float v, long t, int i, int k, const SliceEpilogue& ep) {
    if (ep.potts) {
        if (ep.norm) v = fmul(v, ep.norm[i]);
        v = ep.scale_vec ? fmul(ep.scale_vec[k], v) : fmul(ep.scale, v);
    }
    if (ep.base) v = fadd(ep.base[t], fmul(ep.coef, v));
    else if (ep.zero_base) v = fadd(0.0f, fmul(ep.coef, v));
    return v;
}

// addSplitArray / sliceSplitArray bins (:548-589): the lower pass rounds
// q*10 in float, the upper pass (q - 1e-9)*10 in double.
// For q in [0, 1] these are the reference's indices; other values (which the
// reference rejects with an assert) are clamped to a valid bin so no access
// can leave the bin array.
__device__ __forceinline__ int bin_lower(float q) {
    int c = (int)floorf(fmul(q, (float)kRes));
    c = c < kRes - 1 ? c : kRes - 1;
    return c > 0 ? c : 0;
}
// floor((q - 1e-9) * 10) without double arithmetic: the product rounded down
// has the floor of the exact 10 q, and 10 q - 1e-8 falls into the bin below only
// where 10 q is an integer (0, 5 and 10: q = 0.5 here, the ends by the clamps);
// the next float above any n / 10 has 10 q - n > 1.4e-8.  Equal to the double
// expression for every float in [0, 1].
__device__ __forceinline__ int bin_upper(float q) {
    int c = (int)floorf(__fmul_rd(q, (float)kRes));
    c = q == 0.5f ? 4 : c;
    c = c < kRes - 1 ? c : kRes - 1;
    return c > 0 ? c : 0;
}

// Ordered bins of every (pixel, label), computed once per ordered filter
// (each pixel appears in d+1 splat lists and in the slice): the lower and
// upper bin indices, held as floats (exact small integers) because the splat
// compares them with float bin numbers.
__device__ __forceinline__ float2 ord_bin_pair(float q) {
    return make_float2((float)bin_lower(q), (float)bin_upper(q));
}
__device__ __forceinline__ int ord_lower_of(float2 b) { return (int)b.x; }
__device__ __forceinline__ int ord_upper_of(float2 b) { return (int)b.y; }

__host__ __device__ inline bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

}  // namespace dcrf
