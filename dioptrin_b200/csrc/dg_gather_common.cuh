// Pieces the gather kernels share (dg_gather.cu, dg_bins.cu): modes and their
// accumulators, pixel loads, the spread's origin, shared-memory copies and
// packed FP32 arithmetic.
#pragma once

#include <type_traits>

#include "dg_internal.h"

namespace dg {
namespace {

// kRaw: the per-frame-mask gather (entries {pixel, w, w*norm}); it sums
// S = sum w*s, V = sum w^2*max(s,0), N = sum w*norm and C = sum w over the
// entries whose pixel the frame's mask leaves unmasked.
enum Mode { kIntensity = 0, kErrors = 1, kSpread = 2, kRaw = 3 };

template <typename P>
constexpr bool is_float_px() {
    return std::is_same<P, float>::value || std::is_same<P, double>::value;
}

// Accumulators per (segment, frame): S = sum c*s, then V = sum c^2*max(s,0),
// then for the spread B = sum (c/n)*t^2 and A = sum c*t, then for float
// pixels the weight c*n and the count of non-finite pixels.
template <int MODE, typename P>
struct NAcc {
    static constexpr int value = MODE == kIntensity ? 1
                                 : MODE == kErrors  ? 2
                                 : MODE == kRaw     ? 4
                                                    : (is_float_px<P>() ? 6 : 4);
};
constexpr int kSpreadA = 3;  // index of A among the spread's accumulators
constexpr int kMaxAcc = 6;   // accumulators per (segment, frame), at most
static_assert(NAcc<kSpread, float>::value <= kMaxAcc && NAcc<kRaw, float>::value <= kMaxAcc,
              "partial sums are sized for kMaxAcc accumulators");

// Accumulators per frame of a mode, for sizing partial sums at run time.
inline int n_accumulators(int mode, bool float_px) {
    return mode == kIntensity ? 1 : mode == kErrors ? 2 : mode == kRaw ? 4 : (float_px ? 6 : 4);
}

template <typename P>
constexpr bool is_unsigned_px() {
    return std::is_same<P, uint16_t>::value || std::is_same<P, uint32_t>::value;
}

template <typename P>
__device__ __forceinline__ float load_px(const P *__restrict__ f, uint32_t i) {
    return float(__ldg(f + i));
}
template <>
__device__ __forceinline__ float load_px<double>(const double *__restrict__ f, uint32_t i) {
    return __double2float_rn(__ldg(f + i));
}

// Origin o = s/n of the spread's shift in this frame. The reference shifts
// by the row's first valid entry (azimuthal.rs:80-82); the spread does not
// depend on the shift, only its rounding does: the moments lose to
// cancellation about (mean - o)^2 / variance, so this build shifts by the
// row's heaviest valid entry (largest c*n, chosen at plan time), which sits
// at the mean of a bin dominated by one pixel. A float pixel that is not
// finite there hands the origin to the row's first valid finite entry
// (entries that are statically invalid carry c = 0).
template <typename P>
__device__ __forceinline__ float row_origin(const float4 *__restrict__ entry_std, int origin,
                                            int first, int row_end,
                                            const P *__restrict__ frame) {
    if (origin < 0) return 0.f;
    float4 e = entry_std[origin];
    float s = load_px<P>(frame, uint32_t(__float_as_int(e.x)));
    if (is_float_px<P>() && !isfinite(s)) {
        for (int k = first; k < row_end; ++k) {
            const float4 ek = entry_std[k];
            if (!(ek.y > 0.f)) continue;
            e = ek;
            s = load_px<P>(frame, uint32_t(__float_as_int(e.x)));
            if (isfinite(s)) break;
        }
    }
    return __fdiv_rn(s, e.z);
}

template <typename P>
using StagedPx = typename std::conditional<sizeof(P) == 4, P, float>::type;

__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
// The same with the shared-memory address as a 32-bit integer.
__device__ __forceinline__ void cp_async4_s(unsigned d, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
// A staged 4-byte pixel from its bits.
template <typename S>
__device__ __forceinline__ float staged_value(uint32_t b) {
    if constexpr (std::is_same<S, float>::value) return __uint_as_float(b);
    else if constexpr (std::is_same<S, int32_t>::value) return float(int32_t(b));
    else return float(b);
}

// Packed FP32x2 arithmetic (round to nearest, per element as the scalar
// operations).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 upk(f2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Packed FP32 partial sums (even entries in one half, odd in the other) folded
// into one FP64 sum, the even half then the odd: four registers, against six
// of a double-word FP32 sum.
struct AccP64 {
    f2 p;
    double d;
    __device__ __forceinline__ void zero() {
        p = 0ull;
        d = 0.0;
    }
    __device__ __forceinline__ void flush() {
        const float2 h = upk(p);
        d = __dadd_rn(__dadd_rn(d, double(h.x)), double(h.y));
        p = 0ull;
    }
    __device__ __forceinline__ double value() const { return d; }
};

// Row flip of a pixel index for frames stored bottom row first.
__device__ __forceinline__ int32_t flip_px(int32_t j, int rows, int cols) {
    const int32_t r = j / cols, c = j - r * cols;
    return (rows - 1 - r) * cols + c;
}

}  // namespace
}  // namespace dg
