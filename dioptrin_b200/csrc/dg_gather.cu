// Per-frame gather: CSR (bins x pixels) times a stack of frames.
//
// Three families of lane mappings, chosen per plan by timing (the
// autotuner): entry-lane units (k_gather, mappings 0-4, described first
// below), frame-lane units (k_gather_fl, 5-6) and bin tiles (k_gather_bins,
// 7-8). The first two leave per-segment partial sums that k_finalize folds;
// the bin tiles keep each bin's sums in registers for the whole batch and
// write the results themselves.
//
// Layout. The masked table is cut into segments: a segment is a run of one
// row's entries whose pixels lie in one strip of `strip_rows` detector rows
// (rows list pixels in ascending order, so this is a contiguous range), split
// further to at most kSegMax entries. Within a strip, the segments of
// neighbouring rows are grouped into units of at most kWarps segments and
// unit_cap entries. One CTA owns one unit: it stages the unit's packed entries
// in shared memory once and sweeps every frame of the call over them, so the
// table crosses HBM once per call however many frames there are. Neighbouring
// bins share most pixels (a split pixel falls in ~2.6 bins), and a unit's
// bins cover the same strip of the detector: warps take (segment, frame
// group) tasks in frame-major order, so at any time the CTA's warps read the
// same few kilobytes of the same frames and the repeats are served by L1
// instead of each costing an L2 sector.
//
// A task is (segment, group of kFrameLanes frames); lane (frame, slice)
// reads every kSlices-th staged entry (col, weight[, norm, weight/norm]) and
// gathers that pixel of its frame, kUnroll independent loads at a time; the
// kSlices lanes of a frame then fold their sums.
//
// Arithmetic. Sums are FP32 products accumulated in short plain-FP32 blocks
// (at most kFlush terms per lane) that are folded into a double-word (hi, lo)
// FP32 accumulator with TwoSum; each lane's double-word sum is exact in FP64,
// and lanes, then segments, are added in FP64 in a fixed order. The
// reduction order depends only on the table, never on how many frames a call
// carries, so one frame alone and the same frame inside a batch give
// bit-identical results.
//
// Azimuthal spread (azimuthal.rs:48-118): with x = s/n, w = c*n and origin
// o = x of one valid entry of the row, t = s - o*n gives w*(x - o) = c*t
// and w*(x - o)^2 = (c/n)*t*t, so the shifted moments A = sum c*t and
// B = sum (c/n)*t*t need no division per pixel, and the reference's second
// pass sum w*((x - o) - A/W)^2 equals m2 = B - A^2/W with W = sum w. The
// shift is exact to the last bit of t: n is kept as an FP32 pair
// (n_hi, n_lo) with n_hi + n_lo = n to 2^-48, t = (s - o*n_hi) - o*n_lo by
// two FMAs, and A is accumulated from the same t (forming it as S - o*W
// instead loses the products' rounding of S to the cancellation). Any
// constant origin gives the same m2 and o only has to be the same for every
// entry of a row, so its FP32 rounding is harmless; its distance from the
// mean sets the cancellation in m2, so o is the row's heaviest valid entry
// (row_origin) rather than the reference's first one.
#include <algorithm>
#include <climits>
#include <type_traits>

#include <array>
#include <atomic>
#include <memory>
#include <thread>

#include "dg_gather_common.cuh"

namespace dg {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kFlush = 16;  // terms per lane between double-word folds
// Gather lane mappings a plan chooses from (launch_gather). Entry-lane
// mappings, as (entry slices per frame group, frames per lane, entries per
// lane per step): 0 (32,4,4), 1 (32,2,8), 2 (8,2,4), 3 (4,1,8), 4 (16,4,2),
// and 9 (32,1,8), whose 32 lanes all take entries of one frame (the
// one-frame launches of the plain path); frame-lane mappings (k_gather_fl),
// 2 CTAs per SM (5) or 1 CTA per SM with the next frames prefetched while the
// current ones are summed (6); bin tiles (k_gather_bins: 7, one frame per
// lane; 8, two), which write the results themselves; row warps (k_rows, 10)
// for launches of a few frames, which write them too.
constexpr int kVariantCount = 11;
constexpr int kSegMax = 256;
constexpr int kUnitCap = 3008;  // 16-byte entries in the 48 KB default shared memory

// Double-word FP32 accumulator with a plain FP32 block in front.
struct AccDW {
    float p, hi, lo;
    __device__ __forceinline__ void zero() { p = hi = lo = 0.f; }
    __device__ __forceinline__ void fma(float a, float b) { p = __fmaf_rn(a, b, p); }
    __device__ __forceinline__ void add(float a) { p = __fadd_rn(p, a); }
    __device__ __forceinline__ void flush() {
        float s = __fadd_rn(hi, p);
        float bp = __fsub_rn(s, hi);
        float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(p, bp));
        hi = s;
        lo = __fadd_rn(lo, e);
        p = 0.f;
    }
    // (hi, lo) += (h2, l2), hi keeps the rounded sum.
    __device__ __forceinline__ void merge(float h2, float l2) {
        float s = __fadd_rn(hi, h2);
        if (!(fabsf(s) <= 3.40282347e+38f)) {  // inf or NaN: keep it
            hi = s;
            lo = 0.f;
            return;
        }
        float bp = __fsub_rn(s, hi);
        float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(h2, bp));
        float t = __fadd_rn(__fadd_rn(e, lo), l2);
        hi = __fadd_rn(s, t);
        lo = __fsub_rn(t, __fsub_rn(hi, s));
    }
};

// Reduce-scatter of V values (a power of two, <= 32) across the 32 lanes of
// a warp by a fixed butterfly: after the call, lanes 2i and 2i+1 (V = 16),
// or lanes with (lane >> log2(32/V)) == i in general, hold value i summed over
// all lanes. IEEE addition is commutative, so the result does not depend on
// which partner adds which.
template <int V>
__device__ __forceinline__ double reduce_scatter(double (&v)[V], int lane) {
    int cur = V;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        if (cur > 1) {
            const bool hi = (lane & m) != 0;
            const int half = cur / 2;
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
                if (i < half) {
                    const double send = hi ? v[i] : v[i + half];
                    const double keep = hi ? v[i + half] : v[i];
                    v[i] = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, m));
                }
            }
            cur = half;
        } else {
            v[0] = __dadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], m));
        }
    }
    return v[0];
}

// One CTA per unit; see the file comment. Template parameters choose the
// lane mapping: SLICES lanes split a segment's entries (lane sl takes entries
// sl, sl + SLICES, ...), 32 / SLICES lane groups take different frames, and
// each lane carries FPL frames, so a task is (segment, 32 / SLICES * FPL
// frames). U entries per lane per step have all their loads in flight.
// One unit of the entry-lane gather, run by the whole CTA (k_gather runs unit
// blockIdx.x; the work-queue gather runs the units it claims, several per
// CTA). It ends with a CTA barrier, so the next unit may restage the shared
// memory at once.
template <int MODE, typename P, int SLICES, int FPL, int U>
__device__ __forceinline__ void gather_unit(
    int unit, const int2 *__restrict__ units, const int4 *__restrict__ segs,
    const int2 *__restrict__ entry, const float4 *__restrict__ entry_std,
    const float *__restrict__ entry_nlo, const int32_t *__restrict__ first_valid,
    const int32_t *__restrict__ origin_entry, const P *__restrict__ frames, int64_t n_pixels,
    int n_frames, int n_segments, double *__restrict__ partial,
    const uint8_t *__restrict__ masks, int64_t mask_stride) {
    constexpr int NA = NAcc<MODE, P>::value;
    constexpr bool WIDE = MODE == kSpread || MODE == kRaw;  // 16-byte entries
    constexpr int GROUPS = 32 / SLICES;         // frame lane groups per warp
    constexpr int TASK_FRAMES = GROUPS * FPL;  // frames per task
    static_assert(kFlush % U == 0, "flush cadence must be a multiple of the unroll");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_off[kWarps + 1];
    const int2 un = units[unit];
    const int seg0 = un.x, nseg = un.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        int o = 0;
        for (int i = 0; i < nseg; ++i) {
            s_off[i] = o;
            const int4 sg = segs[seg0 + i];
            o += sg.z - sg.y;
        }
        s_off[nseg] = o;
    }
    __syncthreads();
    // Stage the unit's entries (16- or 8-byte vector copies, segment by segment).
    for (int i = 0; i < nseg; ++i) {
        const int4 sg = segs[seg0 + i];
        const int len = sg.z - sg.y, off = s_off[i];
        if (WIDE) {
            float4 *st = reinterpret_cast<float4 *>(smem) + off;
            for (int j = threadIdx.x; j < len; j += kThreads) st[j] = entry_std[sg.y + j];
        } else {
            int2 *st = reinterpret_cast<int2 *>(smem) + off;
            for (int j = threadIdx.x; j < len; j += kThreads) st[j] = entry[sg.y + j];
        }
    }
    __syncthreads();

    const int sl = lane % SLICES, fg = lane / SLICES;
    const int groups = (n_frames + TASK_FRAMES - 1) / TASK_FRAMES;
    int grp = 0, si = warp;
    // Frame-major task order: the CTA's warps work on the same frames at once.
    for (;; si += kWarps) {
        while (si >= nseg) {
            si -= nseg;
            ++grp;
        }
        if (grp >= groups) break;
        const int4 sg = segs[seg0 + si];
        const int row = sg.x, len = sg.z - sg.y, off = s_off[si];
        const int fbase = grp * TASK_FRAMES + fg * FPL;
        const P *fr[FPL];
        const uint8_t *mk[FPL];
        bool fv[FPL];
#pragma unroll
        for (int q = 0; q < FPL; ++q) {
            fv[q] = fbase + q < n_frames;
            fr[q] = frames + int64_t(fv[q] ? fbase + q : 0) * n_pixels;
            mk[q] = MODE == kRaw ? masks + int64_t(fv[q] ? fbase + q : 0) * mask_stride : nullptr;
        }
        float origin[FPL];
#pragma unroll
        for (int q = 0; q < FPL; ++q)
            origin[q] = MODE == kSpread ? row_origin<P>(entry_std, origin_entry[row],
                                                        first_valid[row], sg.w, fr[q])
                                        : 0.f;
        AccDW acc[FPL][NA];
#pragma unroll
        for (int q = 0; q < FPL; ++q)
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[q][a].zero();

        // One step: U entries of this lane, all loads issued before use.
        // CHECK is true only for the last, partial step, whose entries past
        // the segment end contribute zero without touching the frame.
        auto step = [&](int j0, auto check) {
            constexpr bool CHECK = decltype(check)::value;
            if (MODE == kRaw) {
                float4 e[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = j0 + SLICES * u;
                    if (CHECK)
                        e[u] = j < len ? reinterpret_cast<const float4 *>(smem)[off + j]
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
                    else
                        e[u] = reinterpret_cast<const float4 *>(smem)[off + j];
                }
                float sv[U][FPL];
                bool live[U][FPL];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int q = 0; q < FPL; ++q) {
                        const uint32_t col = uint32_t(__float_as_int(e[u].x));
                        const bool in = !CHECK || j0 + SLICES * u < len;
                        sv[u][q] = in ? load_px<P>(fr[q], col) : 0.f;
                        live[u][q] = in && __ldg(mk[q] + col) == 0;
                    }
#pragma unroll
                for (int u = 0; u < U; ++u) {
#pragma unroll
                    for (int q = 0; q < FPL; ++q) {
                        // a masked pixel adds nothing, whatever its value
                        const float c = live[u][q] ? e[u].y : 0.f;
                        const float cn = live[u][q] ? e[u].z : 0.f;
                        const float v = live[u][q] ? sv[u][q] : 0.f;
                        acc[q][0].fma(c, v);
                        acc[q][1].fma(__fmul_rn(c, c), is_unsigned_px<P>() ? v : fmaxf(v, 0.f));
                        acc[q][2].add(cn);
                        acc[q][3].add(c);
                    }
                }
            } else if (MODE == kSpread) {
                float4 e[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = j0 + SLICES * u;
                    if (CHECK)
                        e[u] = j < len ? reinterpret_cast<const float4 *>(smem)[off + j]
                                       : make_float4(0.f, 0.f, 1.f, 0.f);
                    else
                        e[u] = reinterpret_cast<const float4 *>(smem)[off + j];
                }
                float sv[U][FPL], nlo[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool in = !CHECK || j0 + SLICES * u < len;
                    nlo[u] = in ? __ldg(entry_nlo + sg.y + j0 + SLICES * u) : 0.f;
#pragma unroll
                    for (int q = 0; q < FPL; ++q)
                        sv[u][q] = in ? load_px<P>(fr[q], uint32_t(__float_as_int(e[u].x))) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float c = e[u].y, n = e[u].z, cr = e[u].w;
                    const float c2 = __fmul_rn(c, c);
#pragma unroll
                    for (int q = 0; q < FPL; ++q) {
                        const float v = sv[u][q];
                        if (is_float_px<P>() && !isfinite(v)) {
                            acc[q][NA - 2].add(__fmul_rn(c, n));
                            acc[q][NA - 1].add(c > 0.f ? 1.f : 0.f);
                            continue;
                        }
                        acc[q][0].fma(c, v);
                        acc[q][1].fma(c2, is_unsigned_px<P>() ? v : fmaxf(v, 0.f));
                        const float t = __fmaf_rn(-origin[q], nlo[u], __fmaf_rn(-origin[q], n, v));
                        acc[q][2].fma(__fmul_rn(cr, t), t);
                        acc[q][kSpreadA].fma(c, t);
                    }
                }
            } else {
                int2 e[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = j0 + SLICES * u;
                    if (CHECK)
                        e[u] = j < len ? reinterpret_cast<const int2 *>(smem)[off + j]
                                       : make_int2(0, 0);
                    else
                        e[u] = reinterpret_cast<const int2 *>(smem)[off + j];
                }
                float sv[U][FPL];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int q = 0; q < FPL; ++q)
                        sv[u][q] = !CHECK || j0 + SLICES * u < len
                                       ? load_px<P>(fr[q], uint32_t(e[u].x))
                                       : 0.f;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float c = __int_as_float(e[u].y);
                    const float c2 = __fmul_rn(c, c);
#pragma unroll
                    for (int q = 0; q < FPL; ++q) {
                        acc[q][0].fma(c, sv[u][q]);
                        if (MODE == kErrors)
                            acc[q][1].fma(c2, is_unsigned_px<P>() ? sv[u][q] : fmaxf(sv[u][q], 0.f));
                    }
                }
            }
        };
        int since = 0;
        const int full = len / (SLICES * U) * (SLICES * U);
        int j0 = sl;
        for (; j0 < full; j0 += SLICES * U) {
            step(j0, std::false_type{});
            since += U;
            if (since == kFlush) {
                since = 0;
#pragma unroll
                for (int q = 0; q < FPL; ++q)
#pragma unroll
                    for (int a = 0; a < NA; ++a) acc[q][a].flush();
            }
        }
        if (full < len) step(j0, std::true_type{});
#pragma unroll
        for (int q = 0; q < FPL; ++q)
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[q][a].flush();

        // Each lane's double-word sums are exact in FP64; the SLICES lanes of
        // a frame group are added by a fixed tree.
        if constexpr (SLICES == 32) {
            constexpr int V0 = FPL * NA;
            constexpr int V = V0 <= 1 ? 1 : V0 <= 2 ? 2 : V0 <= 4 ? 4 : V0 <= 8 ? 8 : V0 <= 16 ? 16 : 32;
            double d[V];
#pragma unroll
            for (int i = 0; i < V; ++i) d[i] = 0.0;
#pragma unroll
            for (int q = 0; q < FPL; ++q)
#pragma unroll
                for (int a = 0; a < NA; ++a)
                    d[q * NA + a] = double(acc[q][a].hi) + double(acc[q][a].lo);
            const double mine = reduce_scatter<V>(d, lane);
            const int idx = lane / (32 / V);
            if (lane % (32 / V) == 0 && idx < V0) {
                const int q = idx / NA, a = idx % NA;
                if (fbase + q < n_frames)
                    partial[(int64_t(seg0 + si) * NA + a) * n_frames + fbase + q] = mine;
            }
        } else {
            double d[FPL][NA];
#pragma unroll
            for (int q = 0; q < FPL; ++q)
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    double x = double(acc[q][a].hi) + double(acc[q][a].lo);
#pragma unroll
                    for (int o = SLICES / 2; o > 0; o >>= 1)
                        x = __dadd_rn(x, __shfl_down_sync(0xffffffffu, x, o));
                    d[q][a] = x;
                }
            if (sl == 0) {
#pragma unroll
                for (int q = 0; q < FPL; ++q) {
                    if (!fv[q]) continue;
#pragma unroll
                    for (int a = 0; a < NA; ++a)
                        partial[(int64_t(seg0 + si) * NA + a) * n_frames + fbase + q] = d[q][a];
                }
            }
        }
    }
    __syncthreads();
}

template <int MODE, typename P, int SLICES, int FPL, int U>
__global__ void __launch_bounds__(kThreads)
    k_gather(const int2 *__restrict__ units, const int4 *__restrict__ segs,
             const int2 *__restrict__ entry, const float4 *__restrict__ entry_std,
             const float *__restrict__ entry_nlo,
             const int32_t *__restrict__ first_valid, const int32_t *__restrict__ origin_entry,
             const P *__restrict__ frames, int64_t n_pixels, int n_frames, int n_segments,
             double *__restrict__ partial, const uint8_t *__restrict__ masks,
             int64_t mask_stride) {
    gather_unit<MODE, P, SLICES, FPL, U>(blockIdx.x, units, segs, entry, entry_std, entry_nlo,
                                         first_valid, origin_entry, frames, n_pixels, n_frames,
                                         n_segments, partial, masks, mask_stride);
}

// ---------------------------------------------------------------------------
// Row warps (lane mapping 10): launches of a few frames. A batch amortises
// the table over its frames; one frame reads every entry once, so what
// counts there is keeping enough loads in flight and doing nothing else: no
// staging, no partial sums, no second launch. A row of at most kRowsLong
// entries is one warp's (eight rows per CTA), one of at most kRowsTiny eight
// lanes' (32 per CTA), a longer one the whole CTA's, an eighth per warp
// (largest first, so the long rows start early), or in larger launches one
// warp's, eighth after eighth (rows_group). Lanes stride the entries
// (coalesced), kRowsU of them in flight each, load the pixels of F
// frames per entry and sum in FP64; a fixed butterfly adds the lanes' sums, and
// the eighths are added in order, so a row's bits do not depend on the launch.
// One thread writes the results (normalize_bin, prepared.rs:985-996; the spread's
// closing formulas, azimuthal.rs:96-104). The spread is shifted by the row's
// origin as in the other mappings, in FP64: t = s - o*n with n the entry's FP32
// pair.
//
// What bounds it: the latency of three dependent loads (row record, entry, pixel;
// 57 % of an Eiger-4M frame's warp cycles waited on them) with 28 to 64 warps per SM.
// So the record holds all of a row's plan data (it was an item, a row number and
// two row pointers, in a chain), and the loads past a row's end are made all the
// same, of its last entry with weight 0: as predicated loads the compiler finished
// each before it issued the next. Before and now, us: Eiger-4M with the spread, 1 /
// 2 / 4 / 64 frames 59.5 / 86.0 / 149.7 / 2148 and 53.0 / 69.6 / 121.6 / 1347; 1
// frame with errors 34.8 and 30.0; Eiger-4M cake 81.9 and 59.4; Eiger-9M
// intensities, 1 / 64 frames 36.4 / 745 and 29.8 / 596; Pilatus 1M 14.3 and 12.5.
// Clusters of eight CTAs that share eight rows' pixels in L1 (57 % hits against
// 6 %) were no faster for one frame (61.9), nor were loads of the next entries
// ahead (the registers cost a CTA per SM).
constexpr int kRowsLong = 512;
constexpr int kRowsTiny = 64;  // rows of at most this many entries take 8 lanes
constexpr int kRowsU = 4;  // entries in flight per thread (RowsForm takes fewer in one form)
constexpr int kRowsThreads = 256;

// Butterfly sum over the 32 lanes: every lane ends with the same value (IEEE
// addition is commutative, so partners compute the same sums).
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, m));
    return v;
}
// The same over each group of 8 lanes (the warp's four tiny rows).
__device__ __forceinline__ double group8_sum_d(double v) {
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, m));
    return v;
}

// Shared memory of a row-warp CTA: the warps' sums of long rows.
constexpr int kRowsWarps = kRowsThreads / 32;
using RowsRed = double[kRowsWarps][4 * kMaxAcc];

// Writes one row's results of one frame from its sums v.
template <int MODE, typename P>
__device__ __forceinline__ void rows_write(const QueuePlan &qp, int row, int frame, const double *v) {
    constexpr int NA = NAcc<MODE, P>::value;
    const int64_t oo = int64_t(frame) * qp.n_rows + row;
    if constexpr (MODE != kSpread) {
        const double n = qp.den[row];
        qp.out_i[oo] = n == 0.0 ? 0.0 : v[0] / n;
        if (MODE == kErrors) {
            const double s2 = n == 0.0 ? 0.0 : v[1] / (n * n);
            qp.out_s[oo] = sqrt(s2 > 0.0 ? s2 : 0.0);
        }
    } else {
        int valid = qp.valid_std[row];
        double sw = qp.den_std[row];
        if (NA == 6) {
            valid -= int(v[NA - 1] + 0.5);
            sw -= v[NA - 2];
        }
        if (valid <= 0 || !(sw > 0.0)) {
            qp.out_i[oo] = 0.0;
            if (qp.out_s) qp.out_s[oo] = 0.0;
            qp.out_d[oo] = __longlong_as_double(0x7ff8000000000000ll);
            return;
        }
        const double a1 = v[kSpreadA];
        qp.out_i[oo] = v[0] / sw;
        if (qp.out_s) qp.out_s[oo] = sqrt(v[1] > 0.0 ? v[1] : 0.0) / sw;
        const double mean = a1 / sw;
        const double q2 = (v[2] - mean * a1) / sw;
        // one valid contribution: its deviation from itself is exactly 0
        qp.out_d[oo] = valid == 1 ? 0.0 : sqrt(q2 > 0.0 ? q2 : 0.0);
    }
}

// The row's origin in frames f0 .. f0 + F - 1 (row_origin), 0 without the spread.
template <int MODE, typename P, int F>
__device__ __forceinline__ void rows_origin(const QueuePlan &qp, const int4 rec, int f0, double (&o)[F]) {
    const P *frames = static_cast<const P *>(qp.frames);
    const int fvalid = MODE == kSpread && is_float_px<P>() ? qp.first_valid[rec.x] : -1;
#pragma unroll
    for (int q = 0; q < F; ++q)
        o[q] = MODE == kSpread
                   ? double(row_origin<P>(qp.entry_std, rec.w, fvalid, rec.z,
                                          frames + int64_t(min(f0 + q, qp.n_frames - 1)) * qp.n_pixels))
                   : 0.0;
}

// This thread's sums of entries e0 + li, e0 + li + nl, ... < e1 of a row (rec:
// {row, first entry, end, origin}) in frames f0 .. f0 + F - 1.
template <int MODE, typename P, int F, int U = kRowsU>
__device__ __forceinline__ void rows_sum(const QueuePlan &qp, const int4 rec, int e0, int e1, int li,
                                         int nl, int f0, const double (&o)[F],
                                         double (&acc)[F][NAcc<MODE, P>::value]) {
    constexpr int NA = NAcc<MODE, P>::value;
    constexpr bool SPREAD = MODE == kSpread;
    const int2 *__restrict__ entry = qp.entry;
    const float2 *__restrict__ px_norm = qp.px_norm;
    const P *__restrict__ frames = static_cast<const P *>(qp.frames);
    const P *fr[F];
#pragma unroll
    for (int q = 0; q < F; ++q)
        fr[q] = frames + int64_t(min(f0 + q, qp.n_frames - 1)) * qp.n_pixels;
#pragma unroll
    for (int q = 0; q < F; ++q)
#pragma unroll
        for (int a = 0; a < NA; ++a) acc[q][a] = 0.0;
    for (int j0 = e0 + li; j0 < e1; j0 += nl * U) {
        // Loads past the end repeat the last entry with weight 0 and pixel 0: no
        // load waits behind a branch.
        float cw[U];
        [[maybe_unused]] float2 nn[U];
        P raw[U][F];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + nl * u;
            const int2 en = entry[min(j, e1 - 1)];
            const uint32_t col = uint32_t(en.x);
            cw[u] = j < e1 ? __int_as_float(en.y) : 0.f;
            if constexpr (SPREAD) nn[u] = px_norm[col];
#pragma unroll
            for (int q = 0; q < F; ++q) raw[u][q] = __ldg(fr[q] + col);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (is_float_px<P>() && j0 + nl * u >= e1) {
#pragma unroll
                for (int q = 0; q < F; ++q) raw[u][q] = P(0);
            }
            if constexpr (SPREAD) {
                // valid for the spread (azimuthal.rs:62-75): c > 0 and n
                // finite and > 0 ({0, 0} marks an invalid n); an invalid
                // entry adds nothing
                const float cf = cw[u];
                const bool ok = nn[u].x > 0.f && cf > 0.f && cf <= 3.40282347e+38f;
                const double c = ok ? double(cf) : 0.0;
                const double cr = ok ? double(__fdiv_rn(cf, nn[u].x)) : 0.0;
                const double n = ok ? __dadd_rn(double(nn[u].x), double(nn[u].y)) : 1.0;
                const double c2 = __dmul_rn(c, c);
#pragma unroll
                for (int q = 0; q < F; ++q) {
                    const double v = double(raw[u][q]);
                    if (is_float_px<P>() && !isfinite(v)) {
                        acc[q][NA - 2] = __dadd_rn(acc[q][NA - 2], __dmul_rn(c, n));
                        acc[q][NA - 1] = __dadd_rn(acc[q][NA - 1], c > 0.0 ? 1.0 : 0.0);
                        continue;
                    }
                    acc[q][0] = __fma_rn(c, v, acc[q][0]);
                    acc[q][1] = __fma_rn(c2, is_unsigned_px<P>() ? v : fmax(v, 0.0), acc[q][1]);
                    const double t = __fma_rn(-o[q], n, v);
                    acc[q][2] = __fma_rn(__dmul_rn(cr, t), t, acc[q][2]);
                    acc[q][kSpreadA] = __fma_rn(c, t, acc[q][kSpreadA]);
                }
            } else {
                const double c = cw[u];
                const double c2 = __dmul_rn(c, c);
#pragma unroll
                for (int q = 0; q < F; ++q) {
                    const double v = double(raw[u][q]);
                    acc[q][0] = __fma_rn(c, v, acc[q][0]);
                    if (MODE == kErrors)
                        acc[q][1] = __fma_rn(c2, is_unsigned_px<P>() ? v : fmax(v, 0.0), acc[q][1]);
                }
            }
        }
    }
}

// Warp w's eighth of a long row.
__device__ __forceinline__ int2 rows_eighth(const int4 rec, int w) {
    const int64_t n = rec.z - rec.y;
    return make_int2(rec.y + int(n * w / kRowsWarps), rec.y + int(n * (w + 1) / kRowsWarps));
}

// Row-warp item k of a plan's batch: a long row, eight rows of a warp each, or 32
// tiny ones (QueuePlan's n_long, n_mid, first_tiny); every thread of the CTA calls
// it. F frames, one pass over the entries.
template <int MODE, typename P, int F, int U = kRowsU>
__device__ __forceinline__ void rows_item(const QueuePlan &qp, int k, int fb, RowsRed &s_red) {
    constexpr int NA = NAcc<MODE, P>::value;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f0 = F * fb;  // frames [f0, f0 + F) of the batch
    double o[F], acc[F][NA];
    if (k < qp.n_long) {  // a long row for the whole CTA
        const int4 rec = qp.rows[k];
        const int2 e = rows_eighth(rec, warp);
        rows_origin<MODE, P, F>(qp, rec, f0, o);
        rows_sum<MODE, P, F, U>(qp, rec, e.x, e.y, lane, 32, f0, o, acc);
#pragma unroll
        for (int q = 0; q < F; ++q)
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                acc[q][a] = warp_sum_d(acc[q][a]);
                if (lane == 0) s_red[warp][q * NA + a] = acc[q][a];
            }
        __syncthreads();
        // the eighths' sums in order, a thread per sum
        const int t = int(threadIdx.x);
        if (t < F * NA) {
            double v = s_red[0][t];
#pragma unroll
            for (int w = 1; w < kRowsWarps; ++w) v = __dadd_rn(v, s_red[w][t]);
            s_red[0][t] = v;
        }
        __syncthreads();
        if (t < F && f0 + t < qp.n_frames) rows_write<MODE, P>(qp, rec.x, f0 + t, &s_red[0][t * NA]);
        __syncthreads();  // s_red is rewritten by the next item
        return;
    }
    // eight rows, one per warp, or 32 tiny rows, 8 lanes each (four per warp)
    const bool tiny = k >= qp.n_long + qp.n_mid;
    const int first = tiny ? qp.first_tiny + (k - qp.n_long - qp.n_mid) * 4 * kRowsWarps
                           : qp.n_long + (k - qp.n_long) * kRowsWarps;
    const int end = tiny ? qp.n_rows : qp.first_tiny;
    const int at = first + (tiny ? int(threadIdx.x) >> 3 : warp);
    if ((tiny ? first + 4 * warp : at) >= end) return;  // a warp whose rows are all past the end
    const bool live = at < end;                         // lanes past the end still shuffle
    const int4 rec = qp.rows[live ? at : first];
    const int li = tiny ? lane & 7 : lane;
    rows_origin<MODE, P, F>(qp, rec, f0, o);
    rows_sum<MODE, P, F, U>(qp, rec, rec.y, live ? rec.z : rec.y, li, tiny ? 8 : 32, f0, o, acc);
#pragma unroll
    for (int q = 0; q < F; ++q)
#pragma unroll
        for (int a = 0; a < NA; ++a)
            acc[q][a] = tiny ? group8_sum_d(acc[q][a]) : warp_sum_d(acc[q][a]);
    if (li == 0 && live) {
#pragma unroll
        for (int q = 0; q < F; ++q)
            if (f0 + q < qp.n_frames) rows_write<MODE, P>(qp, rec.x, f0 + q, acc[q]);
    }
}

// Eight neighbouring long rows, a warp each, which walks its row's eighths one
// after the other: the warps read the same pixels about the same time and share
// their sectors in L1. The sums are those of rows_item, bit for bit.
template <int MODE, typename P, int F>
__device__ __forceinline__ void rows_group(const QueuePlan &qp, int group, int fb, RowsRed &s_red) {
    constexpr int NA = NAcc<MODE, P>::value;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = group * kRowsWarps + warp;
    if (k >= qp.n_long) return;
    const int4 rec = qp.rows[k];
    const int f0 = F * fb;
    double o[F], acc[F][NA];
    rows_origin<MODE, P, F>(qp, rec, f0, o);
    for (int w = 0; w < kRowsWarps; ++w) {
        const int2 e = rows_eighth(rec, w);
        rows_sum<MODE, P, F>(qp, rec, e.x, e.y, lane, 32, f0, o, acc);
#pragma unroll
        for (int q = 0; q < F; ++q)
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                acc[q][a] = warp_sum_d(acc[q][a]);
                if (lane == 0) {
                    double &v = s_red[warp][q * NA + a];
                    v = w == 0 ? acc[q][a] : __dadd_rn(v, acc[q][a]);
                }
            }
    }
    __syncwarp();
    if (lane < F && f0 + lane < qp.n_frames)
        rows_write<MODE, P>(qp, rec.x, f0 + lane, &s_red[warp][lane * NA]);
}

// The rows' origin entries beside their ranges, so that a launch reads one record
// a row.
__global__ void k_row_origins(int4 *__restrict__ rows, const int32_t *__restrict__ origin, int n) {
    const int i = int(blockIdx.x * blockDim.x + threadIdx.x);
    if (i < n) rows[i].w = origin[rows[i].x];
}

// Lane mapping 10 for one plan's batch: one CTA per (item, frame block).
// Forms of the kernel without the spread: what hides the loads' latency is loads per
// thread where a launch leaves SMs with few CTAs, and CTAs per SM where it does not.
// The sums do not depend on the form.
enum RowsForm {
    kRowsFew,    // few CTAs per SM (launch_rows): the registers of all its loads
    kRowsMany,
    kRowsShort,  // many CTAs, most of them of rows of at most kRowsLong entries
};
// Resident CTAs per SM the compiler must allow for. us, graph-timed, Eiger-4M u32:
// four frames with errors, 3000 bins, 3 CTAs per SM 95.0, 4 100.7, unbounded 109.3;
// 1000 bins, intensities, 3 39.5, 4 36.3; two frames with errors, 3000 bins, 3 entries
// in flight and 4 CTAs 53.8, 4 and 4 62.4, 4 and 3 57.8; two float frames with the spread,
// 3000 bins, 3 CTAs 106, 4 (spilled) 128; an Eiger-4M cake, two frames of u16
// intensities, 6 CTAs 19.2, 4 21.7. One frame without the spread, 8 CTAs against 6:
// Eiger-4M cake 59.4 and 67.6. Four frames with the spread would spill (186 against
// 125 with 4 CTAs).
template <int MODE, typename P>
constexpr int rows_min_ctas(int f, RowsForm form) {
    if (MODE == kSpread) return f == 4 ? 1 : f == 2 && is_float_px<P>() ? 3 : 4;
    if (form == kRowsFew) return f == 1 ? 4 : 3;
    if (f == 1) return 8;
    if (f == 2) return form == kRowsShort ? 6 : 4;
    return MODE == kErrors && sizeof(P) >= 4 ? 3 : 4;
}
// Entries in flight per thread.
template <int MODE, typename P>
constexpr int rows_loads(int f, RowsForm form) {
    return MODE != kSpread && f == 2 && form == kRowsMany && !(MODE == kErrors && is_float_px<P>())
               ? 3
               : kRowsU;
}
template <int MODE, typename P, int F, RowsForm FORM>
__global__ void __launch_bounds__(kRowsThreads, rows_min_ctas<MODE, P>(F, FORM))
    k_rows(const QueuePlan q, const int groups) {
    __shared__ RowsRed s_red;
    int k = blockIdx.x;
    if constexpr (F == 4 && FORM == kRowsMany) {
        if (k < groups) return rows_group<MODE, P, F>(q, k, blockIdx.y, s_red);
        if (groups) k += q.n_long - groups;
    }
    rows_item<MODE, P, F, rows_loads<MODE, P>(F, FORM)>(q, k, blockIdx.y, s_red);
}

// Frames per pass (and per frame block) of a row-warp launch of nf frames.
__host__ __device__ constexpr int rows_pass_frames(int nf) { return nf <= 1 ? 1 : nf <= 2 ? 2 : 4; }

// Tiles a resident work-queue CTA claims at once (one atomic add per claim),
// and the most tiles a call runs as one CTA per tile.
constexpr int kQueueClaim = 4;
constexpr int64_t kQueueDirectTiles = int64_t(1) << 24;

// Work-queue gather over several plans (dg_multi_integrate). A persistent
// grid of row-warp CTAs claims (plan, row item, frame block) tiles from one
// counter until every plan's tiles are summed, so plans of very different
// sizes and batch sizes share one launch and the GPU stays full to the last
// tile. A plan's results are those
// of lane mapping 10 launched for that plan alone, bit for bit. No CTA waits
// on another: a claim is one atomic add, and a CTA that finds the counter
// past the end returns.
template <int MODE, typename P>
__global__ void __launch_bounds__(kRowsThreads)
    k_rows_queue(QueueHeader *__restrict__ hdr, const QueuePlan *__restrict__ plans) {
    __shared__ RowsRed s_red;
    __shared__ int s_item;
    const int n_plans = hdr->n_plans, total = hdr->total_items;
    // A grid that covers every tile takes tile blockIdx.x; a smaller one (a
    // batch beyond the grid limit) stays resident and claims tiles.
    const bool direct = int64_t(gridDim.x) >= int64_t(total);
    for (int pass = 0;; ++pass) {
        int first;
        if (direct) {
            first = int(blockIdx.x);
            if (pass > 0 || first >= total) return;
        } else {
            if (threadIdx.x == 0) s_item = atomicAdd(&hdr->counter, kQueueClaim);
            __syncthreads();
            first = s_item;
            __syncthreads();  // every thread has read s_item before it is claimed again
            if (first >= total) return;
        }
        // the last descriptor whose first tile is at most `first` (plans with
        // no tiles share the next one's prefix and are skipped)
        int lo = 0, hi = n_plans - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (plans[mid].item_first <= first) lo = mid;
            else hi = mid - 1;
        }
        const int last = direct ? first + 1 : min(first + kQueueClaim, total);
        for (int item = first; item < last; ++item) {
            while (lo + 1 < n_plans && plans[lo + 1].item_first <= item) ++lo;
            const QueuePlan &q = plans[lo];
            // (row item, frame block) tiles of the plan, the frame blocks of
            // an item one after another (its entries are still in L2 for the
            // next)
            const int local = item - q.item_first;
            const int k = local / q.frame_blocks, fb = local - k * q.frame_blocks;
            switch (rows_pass_frames(q.n_frames)) {
            case 1: rows_item<MODE, P, 1>(q, k, fb, s_red); break;
            case 2: rows_item<MODE, P, 2>(q, k, fb, s_red); break;
            default: rows_item<MODE, P, 4>(q, k, fb, s_red); break;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Frame-lane gather. Lane = frame: for 32 frames at a time, a unit's distinct
// pixels (at most kFlDCap, listed at plan time) are staged in shared memory,
// 4-byte pixel types by cp.async and the others converted to FP32 on the way,
// frame rows kFlStride words apart (odd, so the 32 lanes reading one pixel of
// their own frames hit 32 banks). Every lane of a warp walks the same entries
// against its own frame, so a frame's sums need no cross-lane reduction.
//
// Entries go in pairs, {index 0, index 1, c0, c1} and for the spread
// {n0, n1, c0/n0, c1/n1}, their columns rewritten at plan time as indices
// into the unit's pixel list; a segment of odd length ends with a padding
// entry of weight 0 whose index names column kFlDCap, which staging never
// writes and which holds 0. Sums use packed FP32x2 arithmetic: the even
// entries of a segment accumulate in one half, the odd ones in the other,
// each in a double-word accumulator folded every kFlFlushPairs pairs.
//
// A unit's pairs are cut into kWarps equal pieces, one per warp. A segment
// inside one piece is written straight to the partial sums; a piece's first
// and last segments go to shared-memory slots, and the slots of a segment
// cut by piece boundaries are added in warp order. Results depend on the
// table alone, not on the frames around them in a batch.

#ifndef DG_FL_DCAP
#define DG_FL_DCAP 384
#endif
constexpr int kFlSegs = 32;               // segments per frame-lane unit, at most
constexpr int kFlDCap = DG_FL_DCAP;       // distinct pixels per frame-lane unit (even)
constexpr int kFlECap = 2 * kFlDCap;      // entries per frame-lane unit before padding
constexpr int kFlPairCap = (kFlECap + kFlSegs) / 2;
constexpr int kFlStride = kFlDCap + 1;    // odd; column kFlDCap stays 0
constexpr int kFlSlots = 2 * kWarps;      // first and last segment of each piece
constexpr int kFlFlushPairs = 16;         // pairs per lane between double-word folds
constexpr int kFlSortMax = 2048;          // keys one unit sorts at plan time
static_assert(kFlECap + kFlSegs <= kFlSortMax, "frame-lane units must fit the plan-time sort");
static_assert(kFlSegs <= 32, "the unit set-up scans segment lengths in one warp");
static_assert(kSegMax <= kFlDCap, "a single segment must fit a frame-lane unit");

// Two double-word FP32 accumulators (even and odd entries) with a plain
// FP32 block in front; the fold is AccDW::flush on each half.
struct Acc2 {
    f2 p, hi, lo;
    __device__ __forceinline__ void zero() { p = hi = lo = 0ull; }
    __device__ __forceinline__ void flush() {
        const f2 s = add2(hi, p);
        const f2 bp = sub2(s, hi);
        const f2 e = add2(sub2(hi, sub2(s, bp)), sub2(p, bp));
        hi = s;
        lo = add2(lo, e);
        p = 0ull;
    }
    // Both halves' exact sums added in FP64 (even + odd).
    __device__ __forceinline__ double value() const {
        const float2 h = upk(hi), l = upk(lo);
        return __dadd_rn(double(h.x) + double(l.x), double(h.y) + double(l.y));
    }
};


// Dynamic shared memory of k_gather_fl: entry pairs, pixel list, one or
// (double-buffered) two sets of 32 frame rows, piece-boundary slots.
template <int MODE>
constexpr size_t fl_pair_bytes() {
    return MODE == kSpread ? 40 : 16;  // pair A, and B and C for the spread
}
template <int MODE, typename P, bool DB>
constexpr size_t fl_smem_bytes() {
    return size_t(kFlPairCap) * fl_pair_bytes<MODE>() + size_t(kFlDCap) * 4 +
           size_t(DB ? 64 : 32) * kFlStride * 4 + size_t(kFlSlots) * NAcc<MODE, P>::value * 32 * 8;
}

// CTAs per SM the frame-lane gather's shared memory allows (227 KB per CTA,
// 228 KB per SM with 1 KB reserved per CTA), for its launch bounds.
template <int MODE, typename P, bool DB>
constexpr int fl_ctas_per_sm() {
    return fl_smem_bytes<MODE, P, DB>() + 6 * 1024 <= 113 * 1024 ? 2 : 1;
}

template <int MODE, typename P, int U2, bool DB>
__global__ void __launch_bounds__(kThreads, (fl_ctas_per_sm<MODE, P, DB>()))
    k_gather_fl(const int4 *__restrict__ units, const int4 *__restrict__ segs,
                const int32_t *__restrict__ unit_px, const float4 *__restrict__ pair_a,
                const float4 *__restrict__ pair_b, const float2 *__restrict__ pair_c,
                const float4 *__restrict__ entry_std,
                const int32_t *__restrict__ first_valid, const int32_t *__restrict__ origin_entry,
                const int32_t *__restrict__ seg_org,
                const P *__restrict__ frames, int64_t n_pixels, int n_frames, int n_segments,
                double *__restrict__ partial) {
    using S = StagedPx<P>;
    constexpr int NA = NAcc<MODE, P>::value;
    constexpr bool SPREAD = MODE == kSpread;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_off[kFlSegs + 1], s_first[kFlSegs], s_rend[kFlSegs], s_oidx[kFlSegs],
        s_oent[kFlSegs];
    __shared__ float s_on[kFlSegs];
    __shared__ int s_sa[kWarps], s_sb[kWarps];
    __shared__ int s_nb, s_bseg[kFlSlots], s_bwlo[kFlSlots], s_bwhi[kFlSlots];
    float4 *s_pa = reinterpret_cast<float4 *>(smem);
    float4 *s_pb = s_pa + kFlPairCap;
    float2 *s_pc = reinterpret_cast<float2 *>(s_pb + kFlPairCap);
    int32_t *s_px = reinterpret_cast<int32_t *>(smem + size_t(kFlPairCap) * fl_pair_bytes<MODE>());
    S *s_buf = reinterpret_cast<S *>(s_px + kFlDCap);
    double *s_red = reinterpret_cast<double *>(s_buf + (DB ? 64 : 32) * kFlStride);

    const int4 un = units[blockIdx.x];
    const int seg0 = un.x, nseg = un.y, D = un.w;
    const int64_t poff = un.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp == 0) {
        int plen = 0;
        if (lane < nseg) {
            const int4 sg = segs[seg0 + lane];
            plen = (sg.z - sg.y + 1) & ~1;
            const int first = first_valid[sg.x], oe = origin_entry[sg.x];
            s_first[lane] = first;
            s_rend[lane] = sg.w;
            s_oent[lane] = oe;
            if (SPREAD) {
                s_oidx[lane] = seg_org[seg0 + lane];
                s_on[lane] = oe >= 0 ? entry_std[oe].z : 1.f;
            }
        }
        int inc = plen;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane < nseg) s_off[lane + 1] = inc;
        if (lane == 0) s_off[0] = 0;
    }
    __syncthreads();
    const int np = s_off[nseg] >> 1;
    for (int j = tid; j < np; j += kThreads) {
        s_pa[j] = pair_a[poff + j];
        if (SPREAD) {
            s_pb[j] = pair_b[poff + j];
            s_pc[j] = pair_c[poff + j];
        }
    }
    for (int j = tid; j < D; j += kThreads) s_px[j] = unit_px[int64_t(blockIdx.x) * kFlDCap + j];
    // Column kFlDCap of every frame row is read by padding entries and must
    // hold 0; staging writes columns below D <= kFlDCap only.
    for (int j = tid; j < (DB ? 64 : 32); j += kThreads) s_buf[j * kFlStride + kFlDCap] = S(0);
    // This warp's piece [lo, hi) (entries; pair aligned) and the segments
    // sa..sb it meets.
    const int lo = 2 * int(int64_t(warp) * np / kWarps);
    const int hi = 2 * int(int64_t(warp + 1) * np / kWarps);
    int sa = 0, sb = -1;
    if (lo < hi) {
        while (s_off[sa + 1] <= lo) ++sa;
        sb = sa;
        while (s_off[sb + 1] < hi) ++sb;
    }
    if (lane == 0) {
        s_sa[warp] = sa;
        s_sb[warp] = sb;
    }
    __syncthreads();
    if (tid == 0) {
        // Segments at piece boundaries, ascending, with their warps.
        int nb = 0;
        for (int w = 0; w < kWarps; ++w) {
            if (s_sb[w] < 0) continue;
            for (int e = 0; e < 2; ++e) {
                const int b = e == 0 ? s_sa[w] : s_sb[w];
                if (e == 1 && b == s_sa[w]) break;
                if (nb > 0 && s_bseg[nb - 1] == b) {
                    s_bwhi[nb - 1] = w;
                } else {
                    s_bseg[nb] = b;
                    s_bwlo[nb] = w;
                    s_bwhi[nb] = w;
                    ++nb;
                }
            }
        }
        s_nb = nb;
    }
    __syncthreads();

    // Stage pixel s_px[k] of frames f0.. into frame rows of `buf`; rows of
    // frames past the end keep stale values (their lanes are never written
    // out). 4-byte pixels are copied asynchronously as one commit group.
    auto stage = [&](int f0, S *buf) {
        const int nv = min(32, n_frames - f0);
        for (int k = tid; k < D; k += kThreads) {
            const P *src = frames + int64_t(f0) * n_pixels + s_px[k];
            S *dst = buf + k;
            if constexpr (sizeof(P) == 4) {
#pragma unroll 8
                for (int f = 0; f < nv; ++f) cp_async4(dst + f * kFlStride, src + int64_t(f) * n_pixels);
            } else {
#pragma unroll 8
                for (int f = 0; f < nv; ++f)
                    dst[f * kFlStride] = load_px<P>(src + int64_t(f) * n_pixels, 0u);
            }
        }
        if constexpr (sizeof(P) == 4) asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int groups = (n_frames + 31) / 32;
    if (DB) stage(0, s_buf);
    for (int g = 0; g < groups; ++g) {
        const int f0 = g * 32;
        const int nv = min(32, n_frames - f0);
        S *cur = DB && (g & 1) ? s_buf + 32 * kFlStride : s_buf;
        if (!DB) {
            stage(f0, cur);
            if constexpr (sizeof(P) == 4) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        } else if (g + 1 < groups) {
            // Prefetch the next group into the other buffer, last read by the
            // previous group's compute (finished at its closing barrier).
            stage(f0 + 32, (g & 1) ? s_buf : s_buf + 32 * kFlStride);
            if constexpr (sizeof(P) == 4) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            if constexpr (sizeof(P) == 4) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const S *px = cur + lane * kFlStride;

        for (int i = sa; i <= sb; ++i) {
            const int p0 = max(lo, s_off[i]) >> 1, p1 = min(hi, s_off[i + 1]) >> 1;
            // Origin o = s/n of the row's origin entry (row_origin): its pixel
            // is staged with the unit's; a non-finite float pixel there sends
            // the lane to the row's entries in global memory.
            float org = 0.f;
            if constexpr (SPREAD) {
                const float so = float(px[s_oidx[i]]);
                org = __fdiv_rn(so, s_on[i]);
                if (is_float_px<P>() && !isfinite(so)) {
                    const int fi = min(f0 + lane, n_frames - 1);
                    org = row_origin<P>(entry_std, s_oent[i], s_first[i], s_rend[i],
                                        frames + int64_t(fi) * n_pixels);
                }
            }
            const f2 norg = pk(-org, -org);
            Acc2 acc[NA];
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[a].zero();

            // UU pairs from p, all shared-memory reads issued before use.
            auto body = [&](int p, auto unroll) {
                constexpr int UU = decltype(unroll)::value;
                float4 ea[UU], eb[UU];
                f2 ec[UU];
#pragma unroll
                for (int u = 0; u < UU; ++u) {
                    ea[u] = s_pa[p + u];
                    if constexpr (SPREAD) {
                        eb[u] = s_pb[p + u];
                        ec[u] = reinterpret_cast<const f2 *>(s_pc)[p + u];
                    }
                }
                float v0[UU], v1[UU];
#pragma unroll
                for (int u = 0; u < UU; ++u) {
                    v0[u] = float(px[__float_as_int(ea[u].x)]);
                    v1[u] = float(px[__float_as_int(ea[u].y)]);
                }
#pragma unroll
                for (int u = 0; u < UU; ++u) {
                    const f2 c = pk(ea[u].z, ea[u].w);
                    if constexpr (SPREAD && is_float_px<P>()) {
                      if (!(isfinite(v0[u]) && isfinite(v1[u]))) {
                        // A non-finite pixel adds its weight c*n to the
                        // spread's excluded sums instead (azimuthal.rs:68-70).
                        const bool ok0 = isfinite(v0[u]), ok1 = isfinite(v1[u]);
                        const float x0 = ok0 ? v0[u] : 0.f, x1 = ok1 ? v1[u] : 0.f;
                        const f2 ce = pk(ok0 ? ea[u].z : 0.f, ok1 ? ea[u].w : 0.f);
                        const f2 x = pk(x0, x1), n = pk(eb[u].x, eb[u].y);
                        const f2 cre = pk(ok0 ? eb[u].z : 0.f, ok1 ? eb[u].w : 0.f);
                        acc[0].p = fma2(ce, x, acc[0].p);
                        acc[1].p = fma2(mul2(ce, ce), pk(fmaxf(x0, 0.f), fmaxf(x1, 0.f)), acc[1].p);
                        const f2 t = fma2(norg, ec[u], fma2(norg, n, x));
                        acc[2].p = fma2(mul2(cre, t), t, acc[2].p);
                        acc[kSpreadA].p = fma2(ce, t, acc[kSpreadA].p);
                        acc[NA - 2].p = add2(acc[NA - 2].p,
                                             pk(ok0 ? 0.f : __fmul_rn(ea[u].z, eb[u].x),
                                                ok1 ? 0.f : __fmul_rn(ea[u].w, eb[u].y)));
                        acc[NA - 1].p = add2(acc[NA - 1].p, pk(!ok0 && ea[u].z > 0.f ? 1.f : 0.f,
                                                               !ok1 && ea[u].w > 0.f ? 1.f : 0.f));
                        continue;
                      }
                    }
                    const f2 x = pk(v0[u], v1[u]);
                    acc[0].p = fma2(c, x, acc[0].p);
                    if constexpr (MODE != kIntensity) {
                        const f2 xp = is_unsigned_px<P>()
                                          ? x
                                          : pk(fmaxf(v0[u], 0.f), fmaxf(v1[u], 0.f));
                        acc[1].p = fma2(mul2(c, c), xp, acc[1].p);
                    }
                    if constexpr (SPREAD) {
                        const f2 n = pk(eb[u].x, eb[u].y), cr = pk(eb[u].z, eb[u].w);
                        const f2 t = fma2(norg, ec[u], fma2(norg, n, x));
                        acc[2].p = fma2(mul2(cr, t), t, acc[2].p);
                        acc[kSpreadA].p = fma2(c, t, acc[kSpreadA].p);
                    }
                }
            };
            int p = p0, since = 0;
            for (; p + U2 <= p1; p += U2) {
                body(p, std::integral_constant<int, U2>{});
                since += U2;
                if (since == kFlFlushPairs) {
                    since = 0;
#pragma unroll
                    for (int a = 0; a < NA; ++a) acc[a].flush();
                }
            }
            for (; p < p1; ++p) body(p, std::integral_constant<int, 1>{});
            double val[NA];
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                acc[a].flush();
                val[a] = acc[a].value();
            }
            if (i != sa && i != sb) {
                if (lane < nv) {
#pragma unroll
                    for (int a = 0; a < NA; ++a)
                        partial[(int64_t(seg0 + i) * NA + a) * n_frames + f0 + lane] = val[a];
                }
            } else {
                const int slot = 2 * warp + (i == sa ? 0 : 1);
#pragma unroll
                for (int a = 0; a < NA; ++a) s_red[(slot * NA + a) * 32 + lane] = val[a];
            }
        }
        __syncthreads();

        // Segments at piece boundaries: their pieces added in warp order.
        const int items = s_nb * NA * 32;
        for (int idx = tid; idx < items; idx += kThreads) {
            const int f = idx & 31, rest = idx >> 5;
            const int a = rest % NA, bi = rest / NA;
            const int b = s_bseg[bi];
            double v = 0.0;
            for (int w = s_bwlo[bi]; w <= s_bwhi[bi]; ++w) {
                if (s_sb[w] < 0) continue;  // an empty piece (units of < kWarps pairs)
                const int slot = 2 * w + (b == s_sa[w] ? 0 : 1);
                v = __dadd_rn(v, s_red[(slot * NA + a) * 32 + f]);
            }
            if (f < nv) partial[(int64_t(seg0 + b) * NA + a) * n_frames + f0 + f] = v;
        }
    }
}

// Frame-lane units at plan time: one CTA per unit sorts the unit's pixel
// indices and its segments' origin pixels (bitonic, kFlSortMax keys),
// writes each segment's origin index into seg_org (kFlDCap, the zero column,
// for a row without valid entries), counts the distinct ones into out_d
// and, with fill (and D <= kFlDCap), writes the distinct list and the
// unit's entry pairs: A {index 0, index 1, c0, c1} with the table's FP32
// weights, B {n0, n1, c0/n0, c1/n1}, C {n_lo 0, n_lo 1} and, when pair_as is
// given, A with the spread's weights (0 for entries the spread excludes).
// Each segment's origin pixel is its row's origin entry's.
__global__ void __launch_bounds__(256)
    k_fl_units(const int4 *__restrict__ units, const int4 *__restrict__ segs,
               const int32_t *__restrict__ col, const int32_t *__restrict__ origin_entry,
               int fill, int32_t *__restrict__ out_d, int32_t *__restrict__ unit_px,
               const int2 *__restrict__ entry, const float4 *__restrict__ entry_std,
               const float *__restrict__ entry_nlo, float4 *__restrict__ pair_a,
               float4 *__restrict__ pair_b, float2 *__restrict__ pair_c,
               float4 *__restrict__ pair_as, int32_t *__restrict__ seg_org) {
    constexpr int N = kFlSortMax, T = 256, PER = N / T;
    __shared__ int s_key[N];
    __shared__ int s_uniq[kFlDCap];
    __shared__ int s_off[kFlSegs + 1], s_poff[kFlSegs + 1];
    __shared__ int s_warp[T / 32 + 1];
    const int4 un = units[blockIdx.x];
    const int tid = threadIdx.x;
    if (tid == 0) {
        int o = 0, po = 0;
        for (int i = 0; i < un.y; ++i) {
            const int4 sg = segs[un.x + i];
            s_off[i] = o;
            s_poff[i] = po;
            o += sg.z - sg.y;
            po += (sg.z - sg.y + 1) & ~1;
        }
        s_off[un.y] = o;
        s_poff[un.y] = po;
    }
    __syncthreads();
    // Keys: the entries' pixels, then each segment's origin pixel (the
    // pixel of its row's first entry valid for the spread).
    const int E = s_off[un.y];
    for (int i = 0; i < un.y; ++i) {
        const int4 sg = segs[un.x + i];
        for (int j = tid; j < sg.z - sg.y; j += T) s_key[s_off[i] + j] = col[sg.y + j];
    }
    if (tid < un.y) {
        const int fv = origin_entry[segs[un.x + tid].x];
        s_key[E + tid] = fv >= 0 ? col[fv] : INT_MAX;
    }
    for (int j = E + un.y + tid; j < N; j += T) s_key[j] = INT_MAX;
    __syncthreads();
    for (int k = 2; k <= N; k <<= 1) {
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
            for (int i = tid; i < N; i += T) {
                const int ixj = i ^ jj;
                if (ixj > i) {
                    const int a = s_key[i], b = s_key[ixj];
                    const bool up = (i & k) == 0;
                    if ((a > b) == up) {
                        s_key[i] = b;
                        s_key[ixj] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    // Distinct keys: flags over PER consecutive keys per thread, block scan.
    int cnt = 0;
    for (int t = 0; t < PER; ++t) {
        const int i = tid * PER + t;
        const int key = s_key[i];
        cnt += key != INT_MAX && (i == 0 || key != s_key[i - 1]);
    }
    const int lane = tid & 31, w = tid >> 5;
    int inc = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int i = 0; i < T / 32; ++i) {
            const int x = s_warp[i];
            s_warp[i] = run;
            run += x;
        }
        s_warp[T / 32] = run;
    }
    __syncthreads();
    const int D = s_warp[T / 32];
    if (tid == 0) out_d[blockIdx.x] = D;
    if (!fill || D > kFlDCap) return;
    int pos = s_warp[w] + inc - cnt;
    for (int t = 0; t < PER; ++t) {
        const int i = tid * PER + t;
        const int key = s_key[i];
        if (key != INT_MAX && (i == 0 || key != s_key[i - 1])) {
            s_uniq[pos] = key;
            unit_px[int64_t(blockIdx.x) * kFlDCap + pos] = key;
            ++pos;
        }
    }
    __syncthreads();
    if (tid < un.y) {
        const int fv = origin_entry[segs[un.x + tid].x];
        int a = kFlDCap;
        if (fv >= 0) {
            const int cc = col[fv];
            int b = D;
            a = 0;
            while (a < b) {
                const int m = (a + b) >> 1;
                if (s_uniq[m] < cc) a = m + 1;
                else b = m;
            }
        }
        seg_org[un.x + tid] = a;
    }
    float *pa = reinterpret_cast<float *>(pair_a + un.z);
    float *pb = reinterpret_cast<float *>(pair_b + un.z);
    float *pc = reinterpret_cast<float *>(pair_c + un.z);
    float *ps = pair_as ? reinterpret_cast<float *>(pair_as + un.z) : nullptr;
    for (int i = 0; i < un.y; ++i) {
        const int4 sg = segs[un.x + i];
        const int len = sg.z - sg.y, padded = (len + 1) & ~1;
        for (int j = tid; j < padded; j += T) {
            const int p = s_poff[i] + j, rec = (p >> 1) * 4, h = p & 1;
            int idx = kFlDCap;
            float c = 0.f, cs = 0.f, n = 1.f, cr = 0.f, nlo = 0.f;
            if (j < len) {
                const int k = sg.y + j, cc = col[k];
                int a = 0, b = D;
                while (a < b) {
                    const int m = (a + b) >> 1;
                    if (s_uniq[m] < cc) a = m + 1;
                    else b = m;
                }
                idx = a;
                c = __int_as_float(entry[k].y);
                const float4 es = entry_std[k];
                cs = es.y;
                n = es.z;
                cr = es.w;
                nlo = entry_nlo[k];
            }
            pa[rec + h] = __int_as_float(idx);
            pa[rec + 2 + h] = c;
            pb[rec + h] = n;
            pb[rec + 2 + h] = cr;
            pc[(p >> 1) * 2 + h] = nlo;
            if (ps) {
                ps[rec + h] = __int_as_float(idx);
                ps[rec + 2 + h] = cs;
            }
        }
    }
}

// One thread per (frame, row): fold the row's segment partials in strip
// order in FP64 and normalise (normalize_bin, prepared.rs:985-996; the
// spread's closing formulas, azimuthal.rs:96-104).
constexpr int kFinRows = 8;  // rows per k_finalize CTA (x 32 frames)
// One tile of kFinRows rows from r0 and 32 frames from fb, by a CTA of 256
// threads: lanes run over frames while the partial sums are read
// (frame-contiguous), the results go through shared memory and are written
// row-contiguous for each frame. Ends with a CTA barrier, so the next tile
// may reuse the shared memory at once.
template <int MODE, typename P>
__device__ __forceinline__ void finalize_tile(
    int r0, int fb, const double *__restrict__ partial, const int32_t *__restrict__ row_seg,
    const int32_t *__restrict__ seg_ids, const double *__restrict__ den,
    const double *__restrict__ den_std, const int32_t *__restrict__ valid_std, int n_rows,
    int n_frames, double *__restrict__ out_i, double *__restrict__ out_s,
    double *__restrict__ out_d) {
    constexpr int NA = NAcc<MODE, P>::value;
    __shared__ double s_o[3][kFinRows][33];
    const int fl = threadIdx.x & 31, rl = threadIdx.x >> 5;
    const int r = r0 + rl, f = fb + fl;
    double ri = 0.0, rs = 0.0, rd = 0.0;
    if (r < n_rows && f < n_frames) {
        double v[NA];
        for (int a = 0; a < NA; ++a) v[a] = 0.0;
        const int k0 = row_seg[r], k1 = row_seg[r + 1];
        for (int k = k0; k < k1; ++k) {
            const double *p = partial + int64_t(seg_ids[k]) * NA * n_frames + f;
            for (int a = 0; a < NA; ++a) v[a] = __dadd_rn(v[a], p[int64_t(a) * n_frames]);
        }
        if (MODE == kRaw) {  // denominators of this frame's mask
            const double n = v[2];
            ri = n == 0.0 ? 0.0 : v[0] / n;
            const double q = n == 0.0 ? 0.0 : v[1] / (n * n);
            rs = sqrt(q > 0.0 ? q : 0.0);
        } else if (MODE != kSpread) {
            const double n = den[r];
            ri = n == 0.0 ? 0.0 : v[0] / n;
            if (MODE == kErrors) {
                const double q = n == 0.0 ? 0.0 : v[1] / (n * n);
                rs = sqrt(q > 0.0 ? q : 0.0);
            }
        } else {
            int valid = valid_std[r];
            double sw = den_std[r];
            if (NA == 6) {
                valid -= int(v[NA - 1] + 0.5);
                sw -= v[NA - 2];
            }
            if (valid <= 0 || !(sw > 0.0)) {
                rd = __longlong_as_double(0x7ff8000000000000ll);
            } else {
                const double a1 = v[kSpreadA];
                ri = v[0] / sw;
                rs = sqrt(v[1] > 0.0 ? v[1] : 0.0) / sw;
                const double mean = a1 / sw;
                const double m2 = v[2] - mean * a1;
                const double q = m2 / sw;
                // one valid contribution: its deviation from itself is exactly 0
                rd = valid == 1 ? 0.0 : sqrt(q > 0.0 ? q : 0.0);
            }
        }
    }
    s_o[0][rl][fl] = ri;
    s_o[1][rl][fl] = rs;
    s_o[2][rl][fl] = rd;
    __syncthreads();
    const int wr = threadIdx.x % kFinRows, wf = threadIdx.x / kFinRows;
    const int rr = r0 + wr, ff = fb + wf;
    if (rr < n_rows && ff < n_frames) {
        const int64_t o = int64_t(ff) * n_rows + rr;
        out_i[o] = s_o[0][wr][wf];
        if (MODE != kIntensity && out_s) out_s[o] = s_o[1][wr][wf];
        if (MODE == kSpread) out_d[o] = s_o[2][wr][wf];
    }
    __syncthreads();
}

template <int MODE, typename P>
__global__ void __launch_bounds__(256)
    k_finalize(const double *__restrict__ partial, const int32_t *__restrict__ row_seg,
               const int32_t *__restrict__ seg_ids, const double *__restrict__ den,
               const double *__restrict__ den_std, const int32_t *__restrict__ valid_std,
               int n_rows, int n_frames, double *__restrict__ out_i, double *__restrict__ out_s,
               double *__restrict__ out_d) {
    finalize_tile<MODE, P>(blockIdx.x * kFinRows, blockIdx.y * 32, partial, row_seg, seg_ids, den,
                           den_std, valid_std, n_rows, n_frames, out_i, out_s, out_d);
}

// Raw sums per (frame, row) (IntermediateResult1d, lut/integrate.rs:372-379):
// S and V from the partial sums; N and C from them too for the per-frame-mask
// gather, else the plan's strict FP64 denominator and weight sum.
template <int MODE>
__global__ void __launch_bounds__(256)
    k_finalize_raw(const double *__restrict__ partial, const int32_t *__restrict__ row_seg,
                   const int32_t *__restrict__ seg_ids, const double *__restrict__ den,
                   const double *__restrict__ cnt, int n_rows, int n_frames,
                   double *__restrict__ out_sig, double *__restrict__ out_norm,
                   double *__restrict__ out_var, double *__restrict__ out_cnt) {
    // Tiles of kFinRows rows x 32 frames, written row-contiguous per frame
    // through shared memory (as k_finalize).
    constexpr int NA = NAcc<MODE, float>::value;
    __shared__ double s_o[4][kFinRows][33];
    const int fl = threadIdx.x & 31, rl = threadIdx.x >> 5;
    const int r0 = blockIdx.x * kFinRows, fb = blockIdx.y * 32;
    const int r = r0 + rl, f = fb + fl;
    double v[NA];
    for (int a = 0; a < NA; ++a) v[a] = 0.0;
    if (r < n_rows && f < n_frames) {
        for (int k = row_seg[r]; k < row_seg[r + 1]; ++k) {
            const double *p = partial + int64_t(seg_ids[k]) * NA * n_frames + f;
            for (int a = 0; a < NA; ++a) v[a] = __dadd_rn(v[a], p[int64_t(a) * n_frames]);
        }
        s_o[0][rl][fl] = v[0];
        s_o[1][rl][fl] = NA > 1 ? v[1] : 0.0;
        s_o[2][rl][fl] = MODE == kRaw ? v[NA > 2 ? 2 : 0] : den[r];
        s_o[3][rl][fl] = MODE == kRaw ? v[NA > 3 ? 3 : 0] : cnt[r];
    }
    __syncthreads();
    const int wr = threadIdx.x % kFinRows, wf = threadIdx.x / kFinRows;
    const int rr = r0 + wr, ff = fb + wf;
    if (rr >= n_rows || ff >= n_frames) return;
    const int64_t o = int64_t(ff) * n_rows + rr;
    out_sig[o] = s_o[0][wr][wf];
    if (out_var) out_var[o] = s_o[1][wr][wf];
    out_norm[o] = s_o[2][wr][wf];
    out_cnt[o] = s_o[3][wr][wf];
}

// Rows of a table at plan time: T threads walk a row's entries together (32:
// eight rows per CTA; 256: a CTA per row), coalesced, and add their partial
// results in a fixed order. One thread per row read 8-byte words from 32 rows
// at once and left the chip idle (ten CTAs for 1250 rows): k_pack took 4.30 ms
// and the separate denominator pass 1.46 ms on the Pilatus-1M table (2.5 M
// entries); now one pass of 36 us for both.
constexpr int kPackThreads = 256;
// Rows of more than 256 entries on average take a CTA each; shorter ones (2D
// bins, about 70 entries) would leave most of its threads without one.
inline bool pack_cta_per_row(int64_t nnz, int64_t n_rows) { return nnz > 256 * n_rows; }

// Sum over the T threads of a row, in every thread (T = 32) or in thread 0 of
// the CTA (T = 256). Every thread of the warp (CTA) calls it.
template <int T>
__device__ __forceinline__ double row_sum(double v, double *s_red) {
    v = warp_sum_d(v);
    if constexpr (T > 32) {
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
        __syncthreads();
        v = 0.0;
        for (int w = 0; w < T / 32; ++w) v = __dadd_rn(v, s_red[w]);
        __syncthreads();
    }
    return v;
}

// Entries for the per-frame-mask gather, {pixel, w, w*norm} in FP32 (the
// product formed in FP64), and the FP64 weight sum of every row.
template <int T>
__global__ void __launch_bounds__(kPackThreads)
    k_pack_raw(const int64_t *__restrict__ row_ptr, int n_rows, const int32_t *__restrict__ col,
               const double *__restrict__ w, const double *__restrict__ norm,
               float4 *__restrict__ entry_raw, double *__restrict__ cnt, int flip_rows,
               int flip_cols) {
    __shared__ double s_red[kPackThreads / 32];
    const int r = blockIdx.x * (kPackThreads / T) + int(threadIdx.x) / T;
    const int li = int(threadIdx.x) % T;
    if (r >= n_rows) return;
    double sum = 0.0;
    for (int64_t k = row_ptr[r] + li; k < row_ptr[r + 1]; k += T) {
        const int32_t j = col[k];
        const double c = w[k];
        sum = __dadd_rn(sum, c);
        // the frame's pixel (rows flipped for InputOrder::FlipVertical)
        int32_t jf = j;
        if (flip_rows) {
            const int32_t rr = j / flip_cols;
            jf = (flip_rows - 1 - rr) * flip_cols + (j - rr * flip_cols);
        }
        entry_raw[k] = make_float4(__int_as_float(jf), __double2float_rn(c),
                                   __double2float_rn(c * norm[j]), 0.f);
    }
    sum = row_sum<T>(sum, s_red);
    if (li == 0) cnt[r] = sum;
}

// Packs the masked f64 table into the gather's entry formats and computes
// the spread's denominators over its valid entries (c > 0, n > 0, finite),
// its first valid entry and its origin entry (the heaviest valid, row_origin).
// The spread's n is stored as the pair (n_hi, n_lo): n_hi = FP32(n) in
// entry_std, n_lo = FP32(n - n_hi) in entry_nlo.
// Per-pixel norm as an FP32 pair for the row warps' spread, at frame
// storage index i: the detector pixel itself, or, for frames stored bottom row
// first (rows > 0), the pixel of the mirrored row.
__global__ void k_px_norm(const double *__restrict__ norm, int64_t n_px, int rows, int cols,
                          float2 *__restrict__ out) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n_px;
         i += int64_t(gridDim.x) * blockDim.x) {
        int64_t j = i;
        if (rows > 0) {
            const int64_t r = i / cols;
            j = (rows - 1 - r) * cols + (i - r * cols);
        }
        const double n = norm[j];
        const bool ok = isfinite(n) && n > 0.0;
        const float hi = ok ? __double2float_rn(n) : 0.f;
        out[i] = make_float2(hi, ok ? __double2float_rn(n - double(hi)) : 0.f);
    }
}

template <int T>
__global__ void __launch_bounds__(kPackThreads)
    k_pack(const int64_t *__restrict__ row_ptr, int n_rows, const int32_t *__restrict__ col,
           const double *__restrict__ w, const double *__restrict__ norm,
           int2 *__restrict__ entry, float4 *__restrict__ entry_std,
           float *__restrict__ entry_nlo, double *__restrict__ den,
           double *__restrict__ den_std, int32_t *__restrict__ valid_std,
           int32_t *__restrict__ first_valid, int32_t *__restrict__ origin) {
    __shared__ double s_red[kPackThreads / 32];
    __shared__ double s_heavy[kPackThreads / 32];
    __shared__ int s_int[3][kPackThreads / 32];
    const int r = blockIdx.x * (kPackThreads / T) + int(threadIdx.x) / T;
    const int li = int(threadIdx.x) % T;
    if (r >= n_rows) return;
    double all = 0.0, sw = 0.0, heaviest = 0.0;
    int valid = 0, first = INT_MAX, org = INT_MAX;
    for (int64_t k = row_ptr[r] + li; k < row_ptr[r + 1]; k += T) {
        int32_t j = col[k];
        double c = w[k], n = norm[j];
        double ww = __dmul_rn(c, n);
        all = __dadd_rn(all, ww);
        bool ok = isfinite(n) && n > 0.0 && isfinite(c) && c > 0.0 && isfinite(ww) && ww > 0.0;
        float cf = __double2float_rn(c);
        entry[k] = make_int2(j, __float_as_int(cf));
        float nf = __double2float_rn(n);
        entry_std[k] = make_float4(__int_as_float(j), ok ? cf : 0.f, ok ? nf : 1.f,
                                   ok ? __double2float_rn(c / n) : 0.f);
        entry_nlo[k] = ok ? __double2float_rn(n - double(nf)) : 0.f;
        if (ok) {
            sw = __dadd_rn(sw, ww);
            ++valid;
            first = min(first, int(k));
            if (ww > heaviest) {  // the first of equally heavy entries
                heaviest = ww;
                org = int(k);
            }
        }
    }
    all = row_sum<T>(all, s_red);
    sw = row_sum<T>(sw, s_red);
    auto heavier = [&](double h, int o) {
        if (h > heaviest || (h == heaviest && o < org)) {
            heaviest = h;
            org = o;
        }
    };
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        valid += __shfl_xor_sync(0xffffffffu, valid, m);
        first = min(first, __shfl_xor_sync(0xffffffffu, first, m));
        const double h = __shfl_xor_sync(0xffffffffu, heaviest, m);
        heavier(h, __shfl_xor_sync(0xffffffffu, org, m));
    }
    if constexpr (T > 32) {
        const int warp = int(threadIdx.x) >> 5;
        if ((threadIdx.x & 31) == 0) {
            s_heavy[warp] = heaviest;
            s_int[0][warp] = org;
            s_int[1][warp] = valid;
            s_int[2][warp] = first;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int q = 1; q < T / 32; ++q) {
                heavier(s_heavy[q], s_int[0][q]);
                valid += s_int[1][q];
                first = min(first, s_int[2][q]);
            }
    }
    if (li != 0) return;
    den[r] = all;
    den_std[r] = sw;
    valid_std[r] = valid;
    first_valid[r] = valid ? first : -1;
    origin[r] = valid ? org : -1;
}

// bounds[r * (n_strips + 1) + s]: first entry of row r whose pixel lies in
// strip s or later (columns within a row are ascending). A thread per (row,
// strip): the searches of one row by one thread ran one after another
// (0.30 ms for 1250 rows x 67 strips).
__global__ void k_strip_bounds(const int64_t *__restrict__ row_ptr, int n_rows,
                               const int32_t *__restrict__ col, int n_strips, int64_t strip_px,
                               int32_t *__restrict__ bounds) {
    const int64_t n = int64_t(n_rows) * (n_strips + 1);
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = i / (n_strips + 1), st = i - r * (n_strips + 1);
        int64_t key = st * strip_px, lo = row_ptr[r], hi = row_ptr[r + 1];
        while (lo < hi) {
            int64_t mid = (lo + hi) >> 1;
            if (int64_t(col[mid]) < key) lo = mid + 1;
            else hi = mid;
        }
        bounds[i] = int32_t(lo);
    }
}

template <int MODE, typename P, int U2, bool DB>
void launch_fl(const GatherTable &t, const P *fp, int64_t n_pixels, int nf, double *partial,
               cudaStream_t s) {
    if (t.fl_n_units <= 0)
        fail(DG_UNSUPPORTED, "the frame-lane gather is not available for this table");
    constexpr size_t smem = fl_smem_bytes<MODE, P, DB>();
    auto kern = k_gather_fl<MODE, P, U2, DB>;
    DG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    const float4 *pa = MODE == kSpread ? t.fl_pair_as : t.fl_pair_a.ptr;
    kern<<<t.fl_n_units, kThreads, smem, s>>>(t.fl_unit.ptr, t.seg.ptr, t.fl_px.ptr, pa,
                                              t.fl_pair_b.ptr, t.fl_pair_c.ptr, t.entry_std.ptr,
                                              t.first_valid.ptr, t.origin.ptr, t.fl_seg_org.ptr,
                                              fp, n_pixels, nf, t.n_segments, partial);
}

// Launches lane-mapping variant `variant` of the gather (kVariantCount) with
// its partial sums in `partial`.
template <int MODE, typename P>
void launch_finalize(const GatherTable &t, const double *partial, int nf, double *oi, double *os,
                     double *od, cudaStream_t s) {
    const dim3 grid(unsigned((t.n_rows + kFinRows - 1) / kFinRows), unsigned((nf + 31) / 32));
    k_finalize<MODE, P><<<grid, 32 * kFinRows, 0, s>>>(partial, t.row_seg.ptr, t.seg_ids.ptr,
                                                        t.den.ptr, t.den_std.ptr, t.valid_std.ptr,
                                                        t.n_rows, nf, oi, os, od);
    DG_CUDA(cudaGetLastError());
}

template <typename P>
constexpr int dtype_code() {
    return std::is_same<P, uint16_t>::value   ? DG_U16
           : std::is_same<P, uint32_t>::value ? DG_U32
           : std::is_same<P, int32_t>::value  ? DG_I32
           : std::is_same<P, float>::value    ? DG_F32
                                              : DG_F64;
}

// Row warps (mapping 10): F frames per pass over a row's entries, one CTA
// per (row item, block of F frames), so a launch of up to four frames reads
// every entry once and a larger one once per four frames.
template <int MODE, typename P>
void launch_rows(const GatherTable &t, const P *fp, int64_t n_pixels, int nf, double *oi,
                 double *os, double *od, cudaStream_t s) {
    const QueuePlan q = queue_plan(t, fp, n_pixels, nf, oi, os, od);
    // Long rows in groups of eight (rows_group): a group is a serial walk of eight
    // rows, so it pays once there are several groups per SM, the more the thicker
    // the rings (longer and fewer rows): a row then shares fewer sectors with its
    // neighbours. us, a CTA per row against groups: Eiger-9M u16, 1000 bins,
    // intensities, 32 / 64 frames (7 and 13 groups per SM, line at 11) 331 / 334 and
    // 653 / 594, with errors, 64 frames (line at 14) 677 / 764; 2000 bins with errors,
    // 16 / 24 frames (7 and 10, line at 6) 286 / 295 and 422 / 371; Eiger-4M u32 with
    // the spread, 1000 bins, 24 / 32 / 64 frames (5, 6 and 13, line at 6) 402 / 425, 532
    // / 532 and 1050 / 975, 2000 bins, 8 frames (3, line at 4) 228 / 177. A row much
    // longer than the others would hold its warp long after they are done.
    int groups = (q.n_long + kRowsWarps - 1) / kRowsWarps;
    if (rows_pass_frames(nf) < 4 || q.n_long == 0) {
        groups = 0;
    } else {
        const double mean = double(t.rw_long_entries) / q.n_long;
        const double per_sm = double(groups) * q.frame_blocks / sm_count();
        const double slope = MODE == kSpread ? 0.5 : MODE == kErrors ? 1.0 : 0.75;
        if (per_sm < 2.0 + slope * mean / q.n_long || t.rw_longest > 4.0 * mean) groups = 0;
    }
    const dim3 grid(unsigned(q.n_items - (groups ? q.n_long - groups : 0)), unsigned(q.frame_blocks));
    auto go = [&](auto frames, auto form) {
        k_rows<MODE, P, decltype(frames)::value, decltype(form)::value>
            <<<grid, kRowsThreads, 0, s>>>(q, groups);
    };
    using Few = std::integral_constant<RowsForm, kRowsFew>;
    using Many = std::integral_constant<RowsForm, kRowsMany>;
    using Short = std::integral_constant<RowsForm, kRowsShort>;
    const int f = rows_pass_frames(nf);
    // Where the lines between the forms lie (us, graph-timed, few against many): one
    // frame, u16 with errors, 6 CTAs per SM 11.2 / 12.4 and 13.9 / 16.0, 11 per SM 11.5 /
    // 10.4, 38 per SM (a cake) 19.3 / 16.4; two frames, u32 intensities, 2 per SM 17.9 /
    // 19.4, 7 per SM 23.8 / 22.0; four, 2 per SM 46.1 / 53.4, 7 per SM 39.5 / 36.3. Against
    // the kernel with predicated loads and no forms, two frames at 5 to 7 CTAs per SM
    // are up to 1.2 us (13 %) slower, all other forms as fast or faster.
    const bool few = MODE != kSpread && !groups && int64_t(grid.x) * grid.y <= (f == 1 ? 8 : 3) * sm_count();
    auto either = [&](auto frames) {
        if constexpr (MODE != kSpread)
            if (few) return go(frames, Few{});
        if constexpr (MODE != kSpread && decltype(frames)::value == 2)
            if (4 * q.n_long < 3 * q.n_items) return go(frames, Short{});
        go(frames, Many{});
    };
    if (f == 1) either(std::integral_constant<int, 1>{});
    else if (f == 2) either(std::integral_constant<int, 2>{});
    else either(std::integral_constant<int, 4>{});
    DG_CUDA(cudaGetLastError());
}

// Bin tiles offset a frame's 4-byte pixels by 32-bit byte counts. Larger frames go to
// the row warps, which leave no partial sums either (raw sums to an entry-lane
// mapping). 64-bit offsets in the copy loop took 1991 us against 1908 (Eiger-4M, 256
// frames with the spread), a loop of their own beside it 1301 against 1291 (128 float
// frames), 840 against 834 (per-frame masks).
bool bin_tiles_reach(int dtype, int64_t n_pixels) {
    return dtype == DG_U16 || dtype == DG_F64 || n_pixels <= int64_t(1) << 30;
}

// Launches lane mapping `variant`; returns true when the kernel wrote the
// normalised results to oi/os/od itself (mappings 7, 8, 10), false when it left
// partial sums for k_finalize. Those mappings need the outputs; callers without
// them (raw sums) get the frame-lane or an entry-lane mapping instead.
template <int MODE, typename P>
bool launch_gather(GatherTable &t, int variant, const P *fp, int64_t n_pixels, int nf,
                   double *partial, cudaStream_t s, const uint8_t *masks = nullptr,
                   int64_t mask_stride = 0, double *oi = nullptr, double *os = nullptr,
                   double *od = nullptr) {
    if constexpr (MODE == kRaw) {
        if ((variant >= 5 && variant <= 8) || variant == 10) variant = 2;  // entry-lane mappings only
    } else {
        if (variant == 10) {
            if (oi && t.rw_n_items > 0) {
                launch_rows<MODE, P>(t, fp, n_pixels, nf, oi, os, od, s);
                return true;
            }
            variant = 2;
        }
        if (variant == 7 || variant == 8) {
            if (oi && t.rw_n_items > 0 && !bin_tiles_reach(dtype_code<P>(), n_pixels)) {
                launch_rows<MODE, P>(t, fp, n_pixels, nf, oi, os, od, s);
                return true;
            }
            if (oi && t.bt[variant - 7].n_items > 0) {
                BinCall c{};
                c.frames = fp;
                c.dtype = dtype_code<P>();
                c.mode = MODE;
                c.n_pixels = n_pixels;
                c.n_frames = nf;
                c.out_i = oi;
                c.out_s = os;
                c.out_d = od;
                c.partial = partial;
                c.fixed = partial != t.partial.ptr;
                launch_bin_tiles(t, variant, c, s);
                return true;
            }
            variant = t.fl_n_units > 0 ? 5 : 2;
        }
        if (variant == 5 || variant == 6) {
            if (variant == 5) launch_fl<MODE, P, 4, false>(t, fp, n_pixels, nf, partial, s);
            else launch_fl<MODE, P, 4, true>(t, fp, n_pixels, nf, partial, s);
            DG_CUDA(cudaGetLastError());
            return false;
        }
    }
    const size_t smem = size_t(t.unit_cap) * (MODE == kSpread || MODE == kRaw ? 16 : 8);
    const float4 *wide = MODE == kRaw ? t.entry_raw.ptr : t.entry_std.ptr;
#define DG_GATHER_ARGS                                                                        \
    t.unit.ptr, t.seg.ptr, t.entry.ptr, wide, t.entry_nlo.ptr, t.first_valid.ptr, t.origin.ptr, fp, \
        n_pixels, nf, t.n_segments, partial, masks, mask_stride
    switch (variant) {
    case 0: k_gather<MODE, P, 32, 4, 4><<<t.n_units, kThreads, smem, s>>>(DG_GATHER_ARGS); break;
    case 1: k_gather<MODE, P, 32, 2, 8><<<t.n_units, kThreads, smem, s>>>(DG_GATHER_ARGS); break;
    case 2: k_gather<MODE, P, 8, 2, 4><<<t.n_units, kThreads, smem, s>>>(DG_GATHER_ARGS); break;
    case 3: k_gather<MODE, P, 4, 1, 8><<<t.n_units, kThreads, smem, s>>>(DG_GATHER_ARGS); break;
    case 9: k_gather<MODE, P, 32, 1, 8><<<t.n_units, kThreads, smem, s>>>(DG_GATHER_ARGS); break;
    default: k_gather<MODE, P, 16, 4, 2><<<t.n_units, kThreads, smem, s>>>(DG_GATHER_ARGS); break;
    }
#undef DG_GATHER_ARGS
    DG_CUDA(cudaGetLastError());
    return false;
}

template <typename P>
bool launch_typed(GatherTable &t, int variant, const void *frames, int64_t n_pixels,
                  int n_frames, int mode, double *partial, double *oi, double *os, double *od,
                  cudaStream_t s) {
    const P *fp = static_cast<const P *>(frames);
    if (mode == kSpread)
        return launch_gather<kSpread, P>(t, variant, fp, n_pixels, n_frames, partial, s, nullptr,
                                         0, oi, os, od);
    if (mode == kErrors)
        return launch_gather<kErrors, P>(t, variant, fp, n_pixels, n_frames, partial, s, nullptr,
                                         0, oi, os, od);
    return launch_gather<kIntensity, P>(t, variant, fp, n_pixels, n_frames, partial, s, nullptr,
                                        0, oi, os, od);
}

template <typename P>
void finalize_typed(const GatherTable &t, int mode, const double *partial, int nf, double *oi,
                    double *os, double *od, cudaStream_t s) {
    if (mode == kSpread) launch_finalize<kSpread, P>(t, partial, nf, oi, os, od, s);
    else if (mode == kErrors) launch_finalize<kErrors, P>(t, partial, nf, oi, os, od, s);
    else launch_finalize<kIntensity, P>(t, partial, nf, oi, os, od, s);
}

}  // namespace

int sm_count() {
    int dev = 0, sms = 0;
    DG_CUDA(cudaGetDevice(&dev));
    DG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return std::max(1, sms);
}

int gather_launches_per_call() { return 2; }

void gather_kernel_time(GatherTable &t, bool reset, double *ms, int64_t *gather_launches,
                        int64_t *launches) {
    double total = 0.0;
    EventPool &p = t.events;
    if (p.used) DG_CUDA(cudaEventSynchronize(p.events[p.used - 1].second));
    for (size_t i = 0; i < p.used; ++i) {
        float m = 0.f;
        DG_CUDA(cudaEventElapsedTime(&m, p.events[i].first, p.events[i].second));
        total += m;
    }
    if (ms) *ms = total;
    if (gather_launches) *gather_launches = int64_t(p.used);
    if (launches) *launches = t.launches;
    if (reset) {
        p.used = 0;
        t.launches = 0;
    }
}

namespace {
// Runs of consecutive segments of one strip, at most max_segs segments and
// `cap` entries each: emit(first segment, segments).
template <class Emit>
void group_segments(const std::vector<int4> &segs, const std::vector<int32_t> &strip_first, int cap,
                    int max_segs, Emit &&emit) {
    for (size_t st = 0; st + 1 < strip_first.size(); ++st) {
        int first = strip_first[st], entries = 0;
        for (int i = first; i < strip_first[st + 1]; ++i) {
            const int len = segs[size_t(i)].z - segs[size_t(i)].y;
            if (i - first == max_segs || entries + len > cap) {
                emit(first, i - first);
                first = i;
                entries = 0;
            }
            entries += len;
        }
        if (strip_first[st + 1] > first) emit(first, strip_first[st + 1] - first);
    }
}

__global__ void k_flip_rows(int2 *__restrict__ entry, float4 *__restrict__ entry_std, int64_t nnz,
                            int32_t *__restrict__ px, int64_t n_px, int rows, int cols);
}  // namespace

// Frame-lane units (k_gather_fl): runs of at most kFlSegs segments and
// kFlECap entries of one strip, split in halves by entries until each holds
// at most kFlDCap distinct pixels; then their pixel lists and entry pairs.
void build_fl_units(GatherTable &out, const DeviceCsr &table, const std::vector<int4> &segs,
                    std::vector<int4> fl, cudaStream_t s) {
    out.fl_n_units = 0;
    out.fl_pair_as = nullptr;
    if (segs.empty() || table.nnz > INT32_MAX) return;
    DeviceArray<int4> d_units;
    DeviceArray<int32_t> d_count;
    std::vector<int32_t> count;
    auto seg_len = [&](int i) { return segs[size_t(i)].z - segs[size_t(i)].y; };
    for (int pass = 0;; ++pass) {
        d_units.alloc(fl.size());
        d_count.alloc(fl.size());
        DG_CUDA(cudaMemcpyAsync(d_units.ptr, fl.data(), fl.size() * sizeof(int4),
                                cudaMemcpyHostToDevice, s));
        k_fl_units<<<unsigned(fl.size()), 256, 0, s>>>(
            d_units.ptr, out.seg.ptr, table.col.ptr, out.origin.ptr, 0, d_count.ptr, nullptr,
            nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
        DG_CUDA(cudaGetLastError());
        count.resize(fl.size());
        DG_CUDA(cudaMemcpyAsync(count.data(), d_count.ptr, count.size() * 4,
                                cudaMemcpyDeviceToHost, s));
        DG_CUDA(cudaStreamSynchronize(s));
        std::vector<int4> next;
        bool split = false;
        for (size_t u = 0; u < fl.size(); ++u) {
            const int4 un = fl[u];
            if (count[u] <= kFlDCap || un.y < 2) {
                next.push_back(make_int4(un.x, un.y, 0, count[u]));
                continue;
            }
            // Split where the first part's entries reach half the unit's.
            int total = 0;
            for (int i = 0; i < un.y; ++i) total += seg_len(un.x + i);
            int acc = 0, cut = 1;
            for (int i = 0; i < un.y - 1; ++i) {
                acc += seg_len(un.x + i);
                cut = i + 1;
                if (2 * acc >= total) break;
            }
            next.push_back(make_int4(un.x, cut, 0, 0));
            next.push_back(make_int4(un.x + cut, un.y - cut, 0, 0));
            split = true;
        }
        fl.swap(next);
        if (!split) break;
        if (pass > 8) fail(DG_DEVICE, "frame-lane units did not converge");
    }
    int64_t pairs = 0;
    for (auto &un : fl) {
        if (un.w > kFlDCap) fail(DG_DEVICE, "frame-lane unit exceeds its pixel cap");
        un.z = int(pairs);
        for (int i = 0; i < un.y; ++i) pairs += (seg_len(un.x + i) + 1) / 2;
    }
    // The spread needs its own weights only if it excludes some entry.
    std::vector<int32_t> valid(size_t(out.n_rows));
    if (!valid.empty())
        DG_CUDA(cudaMemcpyAsync(valid.data(), out.valid_std.ptr, valid.size() * 4,
                                cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaStreamSynchronize(s));
    int64_t n_valid = 0;
    for (int32_t v : valid) n_valid += v;
    const bool own_spread = n_valid != table.nnz;
    out.fl_unit.alloc(fl.size());
    out.fl_px.alloc(fl.size() * size_t(kFlDCap));
    out.fl_pair_a.alloc(size_t(std::max<int64_t>(pairs, 1)));
    out.fl_pair_b.alloc(size_t(std::max<int64_t>(pairs, 1)));
    out.fl_pair_c.alloc(size_t(std::max<int64_t>(pairs, 1)));
    if (own_spread) out.fl_pair_s.alloc(size_t(std::max<int64_t>(pairs, 1)));
    else out.fl_pair_s.release();
    DG_CUDA(cudaMemcpyAsync(out.fl_unit.ptr, fl.data(), fl.size() * sizeof(int4),
                            cudaMemcpyHostToDevice, s));
    out.fl_seg_org.alloc(segs.size());
    k_fl_units<<<unsigned(fl.size()), 256, 0, s>>>(
        out.fl_unit.ptr, out.seg.ptr, table.col.ptr, out.origin.ptr, 1, d_count.ptr,
        out.fl_px.ptr, out.entry.ptr, out.entry_std.ptr, out.entry_nlo.ptr, out.fl_pair_a.ptr,
        out.fl_pair_b.ptr, out.fl_pair_c.ptr, own_spread ? out.fl_pair_s.ptr : nullptr,
        out.fl_seg_org.ptr);
    DG_CUDA(cudaGetLastError());
    DG_CUDA(cudaStreamSynchronize(s));
    out.fl_pair_as = own_spread ? out.fl_pair_s.ptr : out.fl_pair_a.ptr;
    out.fl_n_units = int32_t(fl.size());
}

void make_gather_table(const DeviceCsr &table, const double *d_norm, int32_t dim1, int32_t dim2,
                       int32_t strip_rows, cudaStream_t s, GatherTable &out) {
    out.n_rows = int32_t(table.n_rows);
    out.nnz = table.nnz;
    out.unit_cap = kUnitCap;
    out.strip_rows = strip_rows;
    out.entry.alloc(size_t(table.nnz));
    out.entry_std.alloc(size_t(table.nnz));
    out.den.alloc(size_t(table.n_rows));
    out.den_std.alloc(size_t(table.n_rows));
    out.entry_nlo.alloc(size_t(table.nnz));
    out.valid_std.alloc(size_t(table.n_rows));
    out.first_valid.alloc(size_t(table.n_rows));
    out.origin.alloc(size_t(table.n_rows));
    const int64_t n_px = int64_t(dim1) * dim2;
    out.px_norm.alloc(size_t(std::max<int64_t>(n_px, 1)));
    if (n_px > 0)
        k_px_norm<<<unsigned(std::min<int64_t>((n_px + 255) / 256, 148 * 16)), 256, 0, s>>>(
            d_norm, n_px, 0, 0, out.px_norm.ptr);
    if (table.n_rows > 0) {
#define DG_PACK_ARGS                                                                          \
    table.row_ptr.ptr, int(table.n_rows), table.col.ptr, table.w.ptr, d_norm, out.entry.ptr,  \
        out.entry_std.ptr, out.entry_nlo.ptr, out.den.ptr, out.den_std.ptr, out.valid_std.ptr, \
        out.first_valid.ptr, out.origin.ptr
        if (pack_cta_per_row(table.nnz, table.n_rows))
            k_pack<256><<<unsigned(table.n_rows), kPackThreads, 0, s>>>(DG_PACK_ARGS);
        else
            k_pack<32><<<unsigned((table.n_rows + 7) / 8), kPackThreads, 0, s>>>(DG_PACK_ARGS);
#undef DG_PACK_ARGS
    }
    DG_CUDA(cudaGetLastError());

    // Segments: (row, strip) runs from per-row strip bounds found on the
    // device; grouped into units on the host (a few hundred thousand at most).
    const int n_strips = (dim1 + strip_rows - 1) / strip_rows;
    const int64_t nb = table.n_rows;
    DeviceArray<int32_t> bounds;
    bounds.alloc(size_t(nb * (n_strips + 1)));
    if (nb > 0)
        k_strip_bounds<<<unsigned(std::min<int64_t>((nb * (n_strips + 1) + 255) / 256, 148 * 64)), 256,
                         0, s>>>(table.row_ptr.ptr, int(nb), table.col.ptr, n_strips,
                                 int64_t(strip_rows) * dim2, bounds.ptr);
    DG_CUDA(cudaGetLastError());
    std::vector<int32_t> hb(size_t(nb * (n_strips + 1)));
    std::vector<int64_t> rp(size_t(nb) + 1);
    if (!hb.empty())
        DG_CUDA(cudaMemcpyAsync(hb.data(), bounds.ptr, hb.size() * 4, cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaMemcpyAsync(rp.data(), table.row_ptr.ptr, rp.size() * 8, cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaStreamSynchronize(s));

    std::vector<int4> segs;
    std::vector<int2> units;
    std::vector<int32_t> seg_count(size_t(nb), 0);
    std::vector<int32_t> strip_first(size_t(n_strips) + 1, 0);
    for (int st = 0; st < n_strips; ++st) {
        strip_first[size_t(st)] = int32_t(segs.size());
        for (int64_t r = 0; r < nb; ++r) {
            const int32_t *b = hb.data() + r * (n_strips + 1);
            for (int32_t lo = b[st]; lo < b[st + 1]; lo += kSegMax) {
                int32_t hi = std::min<int32_t>(lo + kSegMax, b[st + 1]);
                segs.push_back(make_int4(int(r), lo, hi, int(rp[size_t(r) + 1])));
                seg_count[size_t(r)]++;
            }
        }
    }
    strip_first[size_t(n_strips)] = int32_t(segs.size());
    group_segments(segs, strip_first, kUnitCap, kWarps,
                   [&](int first, int n) { units.push_back(make_int2(first, n)); });
    // Row -> its segments, in strip order (the finalize's fixed fold order).
    std::vector<int32_t> row_seg(size_t(nb) + 1, 0), seg_ids(segs.size());
    for (int64_t r = 0; r < nb; ++r) row_seg[size_t(r) + 1] = row_seg[size_t(r)] + seg_count[size_t(r)];
    std::vector<int32_t> fill(row_seg.begin(), row_seg.end() - 1);
    for (size_t i = 0; i < segs.size(); ++i) seg_ids[size_t(fill[size_t(segs[i].x)]++)] = int32_t(i);
    out.n_segments = int32_t(segs.size());
    out.n_units = int32_t(units.size());
    out.seg.alloc(std::max<size_t>(segs.size(), 1));
    out.unit.alloc(std::max<size_t>(units.size(), 1));
    out.seg_ids.alloc(std::max<size_t>(seg_ids.size(), 1));
    out.row_seg.alloc(row_seg.size());
    if (!segs.empty()) {
        DG_CUDA(cudaMemcpyAsync(out.seg.ptr, segs.data(), segs.size() * sizeof(int4),
                                cudaMemcpyHostToDevice, s));
        DG_CUDA(cudaMemcpyAsync(out.unit.ptr, units.data(), units.size() * sizeof(int2),
                                cudaMemcpyHostToDevice, s));
        DG_CUDA(cudaMemcpyAsync(out.seg_ids.ptr, seg_ids.data(), seg_ids.size() * 4,
                                cudaMemcpyHostToDevice, s));
    }
    DG_CUDA(cudaMemcpyAsync(out.row_seg.ptr, row_seg.data(), row_seg.size() * 4,
                            cudaMemcpyHostToDevice, s));
    // Row warps (mapping 10): long rows one to a CTA, longest first;
    // the others eight or 32 per CTA in row order.
    std::vector<int4> rw_rows;
    if (table.nnz <= INT32_MAX && nb > 0) {
        auto len = [&](int64_t r) { return rp[size_t(r) + 1] - rp[size_t(r)]; };
        auto take = [&](int64_t above, int64_t most) {  // rows of above < entries <= most
            for (int64_t r = 0; r < nb; ++r)
                if (len(r) > above && len(r) <= most)
                    rw_rows.push_back(make_int4(int(r), int(rp[size_t(r)]), int(rp[size_t(r) + 1]), -1));
            return int32_t(rw_rows.size());
        };
        out.rw_long = take(kRowsLong, INT64_MAX);
        for (const int4 &r : rw_rows) {
            out.rw_long_entries += r.z - r.y;
            out.rw_longest = std::max<int64_t>(out.rw_longest, r.z - r.y);
        }
        // neighbours stay together in groups of kRowsWarps, the longest rows first
        std::vector<int4> by_row(rw_rows);
        std::vector<std::pair<int64_t, size_t>> groups;
        for (size_t i = 0; i < by_row.size(); i += kRowsWarps) {
            int64_t n = 0;
            for (size_t j = i; j < std::min(by_row.size(), i + kRowsWarps); ++j) n += len(by_row[j].x);
            groups.push_back({by_row.size() - i < size_t(kRowsWarps) ? 0 : -n, i});
        }
        std::stable_sort(groups.begin(), groups.end());  // a group of fewer comes last
        rw_rows.clear();
        for (const auto &g : groups)
            for (size_t j = g.second; j < std::min(by_row.size(), g.second + kRowsWarps); ++j)
                rw_rows.push_back(by_row[j]);
        out.rw_tiny = take(kRowsTiny, kRowsLong);
        take(-1, kRowsTiny);
        out.rw_n_items = out.rw_long + (out.rw_tiny - out.rw_long + kRowsWarps - 1) / kRowsWarps +
                         int32_t((nb - out.rw_tiny + 4 * kRowsWarps - 1) / (4 * kRowsWarps));
        out.rw_rows.alloc(rw_rows.size());
        DG_CUDA(cudaMemcpyAsync(out.rw_rows.ptr, rw_rows.data(), rw_rows.size() * sizeof(int4),
                                cudaMemcpyHostToDevice, s));
        k_row_origins<<<unsigned((nb + 255) / 256), 256, 0, s>>>(out.rw_rows.ptr, out.origin.ptr,
                                                                 int(nb));
        DG_CUDA(cudaGetLastError());
    }
    DG_CUDA(cudaStreamSynchronize(s));
    out.strip_first = std::move(strip_first);
}

// Frame-lane units are built when mapping 5 or 6 is selected or timed, as the
// bin tiles are: a plan that runs neither (the default mapping, row warps, bin
// tiles) does not pay for them. Their build took 1.5 ms of device time, four
// launches with a host round trip each, of a Pilatus-1M plan's creation.
void ensure_fl_units(GatherTable &t, const DeviceCsr &table, cudaStream_t s) {
    if (t.fl_built) return;
    AllocScope alloc(s);  // s is synchronised before this returns
    std::vector<int4> segs(static_cast<size_t>(t.n_segments));
    if (!segs.empty()) {
        DG_CUDA(cudaMemcpyAsync(segs.data(), t.seg.ptr, segs.size() * sizeof(int4),
                                cudaMemcpyDeviceToHost, s));
        DG_CUDA(cudaStreamSynchronize(s));
    }
    std::vector<int4> fl;
    group_segments(segs, t.strip_first, kFlECap, kFlSegs,
                   [&](int first, int n) { fl.push_back(make_int4(first, n, 0, 0)); });
    build_fl_units(t, table, segs, std::move(fl), s);
    if (t.flip_rows && t.fl_px.ptr) {  // as flip_gather_rows did for the entries
        k_flip_rows<<<148 * 8, 256, 0, s>>>(nullptr, nullptr, 0, t.fl_px.ptr,
                                            int64_t(t.fl_px.count), t.flip_rows, t.flip_cols);
        DG_CUDA(cudaGetLastError());
        DG_CUDA(cudaStreamSynchronize(s));
    }
    t.fl_built = true;
}

bool gather_writes_results(const GatherTable &t) {
    if (t.variant == 10) return t.rw_n_items > 0;
    return (t.variant == 7 || t.variant == 8) && t.bt[t.variant - 7].n_items > 0;
}

int64_t partial_rows(const GatherTable &t) {
    if (t.n_units == 0) return 0;
    if (gather_writes_results(t)) return t.variant == 10 ? 0 : bin_tile_partials(t, t.variant);
    return std::max<int64_t>(1, t.n_segments);
}

void reserve_partials(GatherTable &t, int64_t n_frames, uint32_t flags, int dtype,
                      bool any_mapping) {
    if (n_frames <= 0) return;
    const int mode = (flags & DG_AZIMUTHAL_STD) ? kSpread : (flags & DG_ERRORS) ? kErrors
                                                                                : kIntensity;
    int64_t rows = partial_rows(t);
    if (any_mapping) {
        rows = std::max<int64_t>(1, t.n_segments);
        for (int v : {7, 8})
            if (t.bt[v - 7].n_items > 0) rows = std::max(rows, bin_tile_partials(t, v));
    }
    const int64_t need = rows * n_accumulators(mode, dtype == DG_F32 || dtype == DG_F64) *
                         std::min<int64_t>(256, (n_frames + 31) / 32 * 32);
    if (t.partial.count < size_t(need)) t.partial.alloc(size_t(need));
}

QueuePlan queue_plan(const GatherTable &t, const void *d_frames, int64_t n_pixels, int n_frames,
                     double *oi, double *os, double *od) {
    QueuePlan q{};
    q.rows = t.rw_rows.ptr;
    q.entry = t.entry.ptr;
    q.entry_std = t.entry_std.ptr;
    q.entry_nlo = t.entry_nlo.ptr;
    q.px_norm = t.px_norm.ptr;
    q.first_valid = t.first_valid.ptr;
    q.den = t.den.ptr;
    q.den_std = t.den_std.ptr;
    q.valid_std = t.valid_std.ptr;
    q.frames = d_frames;
    q.out_i = oi;
    q.out_s = os;
    q.out_d = od;
    q.n_pixels = n_pixels;
    q.n_frames = n_frames;
    q.n_rows = t.n_rows;
    q.n_items = n_frames > 0 ? t.rw_n_items : 0;
    q.n_long = t.rw_long;
    q.n_mid = (t.rw_tiny - t.rw_long + kRowsWarps - 1) / kRowsWarps;
    q.first_tiny = t.rw_tiny;
    q.frame_blocks = std::max(1, (n_frames + rows_pass_frames(n_frames) - 1) /
                                     rows_pass_frames(n_frames));
    return q;
}

namespace {

// Resident capacity of the work-queue gather: the CTAs the SMs hold at
// once, the grid of a call of more than kQueueDirectTiles tiles, whose CTAs
// stay resident and claim tiles until the queue is empty. Smaller calls run
// one CTA per tile (queue_grid).
template <int MODE, typename P>
int queue_capacity() {
    static int cap = 0;
    if (cap == 0) {
        int per_sm = 0, dev = 0, sms = 0;
        DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rows_queue<MODE, P>,
                                                              kRowsThreads, 0));
        DG_CUDA(cudaGetDevice(&dev));
        DG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        cap = std::max(1, per_sm) * std::max(1, sms);
    }
    return cap;
}

template <int MODE, typename P>
void queue_launch_typed(QueueHeader *hdr, const QueuePlan *plans, cudaStream_t s) {
    k_rows_queue<MODE, P><<<queue_capacity<MODE, P>(), kRowsThreads, 0, s>>>(hdr, plans);
    DG_CUDA(cudaGetLastError());
}

template <typename P>
int queue_capacity_mode(int mode) {
    if (mode == kSpread) return queue_capacity<kSpread, P>();
    if (mode == kErrors) return queue_capacity<kErrors, P>();
    return queue_capacity<kIntensity, P>();
}

template <typename P>
void queue_launch_mode(int mode, QueueHeader *hdr, const QueuePlan *plans, cudaStream_t s) {
    if (mode == kSpread) queue_launch_typed<kSpread, P>(hdr, plans, s);
    else if (mode == kErrors) queue_launch_typed<kErrors, P>(hdr, plans, s);
    else queue_launch_typed<kIntensity, P>(hdr, plans, s);
}

}  // namespace

int queue_grid(int dtype, uint32_t flags, int64_t total_tiles, bool resident) {
    // one CTA per tile (the hardware schedules them as CTAs retire, beside
    // other streams' kernels); a batch of more tiles than kQueueDirectTiles
    // runs the resident grid that claims them
    if (!resident && total_tiles <= kQueueDirectTiles)
        return int(std::max<int64_t>(1, total_tiles));
    const int mode = (flags & DG_AZIMUTHAL_STD) ? kSpread : (flags & DG_ERRORS) ? kErrors
                                                                                : kIntensity;
    int cap = 1;
    switch (dtype) {
    case DG_U16: cap = queue_capacity_mode<uint16_t>(mode); break;
    case DG_U32: cap = queue_capacity_mode<uint32_t>(mode); break;
    case DG_I32: cap = queue_capacity_mode<int32_t>(mode); break;
    case DG_F32: cap = queue_capacity_mode<float>(mode); break;
    case DG_F64: cap = queue_capacity_mode<double>(mode); break;
    default: fail(DG_INVALID_INPUT, "unknown pixel dtype");
    }
    const int64_t claims = (total_tiles + kQueueClaim - 1) / kQueueClaim;
    return int(std::max<int64_t>(1, std::min<int64_t>(claims, cap)));
}

void queue_launch(int dtype, uint32_t flags, QueueHeader *hdr, const QueuePlan *plans,
                  cudaStream_t s) {
    const int mode = (flags & DG_AZIMUTHAL_STD) ? kSpread : (flags & DG_ERRORS) ? kErrors
                                                                                : kIntensity;
    switch (dtype) {
    case DG_U16: queue_launch_mode<uint16_t>(mode, hdr, plans, s); break;
    case DG_U32: queue_launch_mode<uint32_t>(mode, hdr, plans, s); break;
    case DG_I32: queue_launch_mode<int32_t>(mode, hdr, plans, s); break;
    case DG_F32: queue_launch_mode<float>(mode, hdr, plans, s); break;
    case DG_F64: queue_launch_mode<double>(mode, hdr, plans, s); break;
    default: fail(DG_INVALID_INPUT, "unknown pixel dtype");
    }
}

void run_gather(GatherTable &t, const void *d_frames, int dtype, int64_t n_pixels,
                int64_t n_frames, uint32_t flags, int precision, double *d_i, double *d_sigma,
                double *d_std, cudaStream_t s, double *scratch, size_t scratch_doubles) {
    (void)precision;
    if (n_frames <= 0) return;
    if (dtype < DG_U16 || dtype > DG_F64) fail(DG_INVALID_INPUT, "unknown pixel dtype");
    const int mode = (flags & DG_AZIMUTHAL_STD) ? kSpread : (flags & DG_ERRORS) ? kErrors
                                                                                : kIntensity;
    // Frames per launch: 256, or fewer where the caller's fixed scratch holds
    // the partial sums of fewer frames (of the bin tiles, the pieces of cut tiles
    // alone leave any; the row warps none).
    int64_t chunk = 256;
    double *partial = nullptr;
    if (scratch) {
        const bool fpx = dtype == DG_F32 || dtype == DG_F64;
        const int64_t per_frame = partial_rows(t) * n_accumulators(mode, fpx);
        if (per_frame > 0) chunk = std::min<int64_t>(chunk, int64_t(scratch_doubles) / per_frame);
        if (chunk < 1)
            fail(DG_UNSUPPORTED, "this plan needs " + std::to_string(per_frame * 8) +
                                     " bytes of partial sums per frame; the fixed scratch holds " +
                                     std::to_string(scratch_doubles * 8) + " bytes");
        partial = scratch;
    } else {
        // [segment][accumulator][frame] for the largest launch of this call,
        // frames rounded up to 32 so that growing batches reallocate rarely;
        // mappings without partial sums do not allocate them
        if (partial_rows(t) > 0)
            reserve_partials(t, std::min<int64_t>(chunk, n_frames), flags, dtype);
        partial = t.partial.ptr;
    }
    // The plan's partial sums and the bin tiles' counts are shared by its calls;
    // row warps share nothing. Calls with a fixed scratch have counts of their own
    // and are ordered by their caller: an event of another stream would end a capture.
    const bool shared = !scratch && (gather_variant_needs_tiles(t.variant) || partial_rows(t) > 0);
    if (shared) t.scratch.wait(s);
    const size_t esize = dtype == DG_U16 ? 2 : dtype == DG_F64 ? 8 : 4;
    for (int64_t f0 = 0; f0 < n_frames; f0 += chunk) {
        const int nf = int(std::min<int64_t>(chunk, n_frames - f0));
        const void *fp = static_cast<const unsigned char *>(d_frames) + f0 * n_pixels * esize;
        double *oi = d_i + f0 * t.n_rows;
        double *os = d_sigma ? d_sigma + f0 * t.n_rows : nullptr;
        double *od = d_std ? d_std + f0 * t.n_rows : nullptr;
        bool done = false;  // results written by the gather itself (bin tiles)
        if (t.n_units > 0) {
            std::pair<cudaEvent_t, cudaEvent_t> *ev = nullptr;
            if (t.profile) {
                EventPool &p = t.events;
                if (p.used == p.events.size()) {
                    std::pair<cudaEvent_t, cudaEvent_t> e{};
                    DG_CUDA(cudaEventCreate(&e.first));
                    DG_CUDA(cudaEventCreate(&e.second));
                    p.events.push_back(e);
                }
                ev = &p.events[p.used++];
                DG_CUDA(cudaEventRecord(ev->first, s));
            }
            ++t.launches;
            switch (dtype) {
            case DG_U16: done = launch_typed<uint16_t>(t, t.variant, fp, n_pixels, nf, mode, partial, oi, os, od, s); break;
            case DG_U32: done = launch_typed<uint32_t>(t, t.variant, fp, n_pixels, nf, mode, partial, oi, os, od, s); break;
            case DG_I32: done = launch_typed<int32_t>(t, t.variant, fp, n_pixels, nf, mode, partial, oi, os, od, s); break;
            case DG_F32: done = launch_typed<float>(t, t.variant, fp, n_pixels, nf, mode, partial, oi, os, od, s); break;
            case DG_F64: done = launch_typed<double>(t, t.variant, fp, n_pixels, nf, mode, partial, oi, os, od, s); break;
            }
            if (ev) DG_CUDA(cudaEventRecord(ev->second, s));
        }
        if (t.n_rows > 0 && !done) {
            ++t.launches;
            switch (dtype) {
            case DG_U16: finalize_typed<uint16_t>(t, mode, partial, nf, oi, os, od, s); break;
            case DG_U32: finalize_typed<uint32_t>(t, mode, partial, nf, oi, os, od, s); break;
            case DG_I32: finalize_typed<int32_t>(t, mode, partial, nf, oi, os, od, s); break;
            case DG_F32: finalize_typed<float>(t, mode, partial, nf, oi, os, od, s); break;
            case DG_F64: finalize_typed<double>(t, mode, partial, nf, oi, os, od, s); break;
            }
        }
    }
    if (shared) t.scratch.mark(s);
}

namespace {

// Swaps detector rows r and rows - 1 - r of a per-pixel array.
__global__ void k_flip_px_norm(float2 *__restrict__ a, int rows, int cols) {
    const int64_t half = int64_t(rows / 2) * cols;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < half;
         i += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = i / cols, c = i - r * cols;
        const int64_t j = (rows - 1 - r) * cols + c;
        const float2 t = a[i];
        a[i] = a[j];
        a[j] = t;
    }
}

// InputOrder::FlipVertical: every pixel index the gathers load through,
// remapped in place (entry order, and so every sum, unchanged). Pixel-list
// slots past a unit's pixel count hold no index and may hold anything; values
// outside the frame are left alone.
__global__ void k_flip_rows(int2 *__restrict__ entry, float4 *__restrict__ entry_std, int64_t nnz,
                            int32_t *__restrict__ px, int64_t n_px, int rows, int cols) {
    const int64_t npix = int64_t(rows) * cols;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < nnz + n_px;
         i += int64_t(gridDim.x) * blockDim.x) {
        if (i < nnz) {
            entry[i].x = flip_px(entry[i].x, rows, cols);
            entry_std[i].x = __int_as_float(flip_px(__float_as_int(entry_std[i].x), rows, cols));
        } else {
            const int32_t v = px[i - nnz];
            if (v >= 0 && v < npix) px[i - nnz] = flip_px(v, rows, cols);
        }
    }
}

}  // namespace

void flip_gather_rows(GatherTable &t, int32_t dim1, int32_t dim2, cudaStream_t s) {
    t.flip_rows = dim1;
    t.flip_cols = dim2;
    // per-pixel norms to frame storage order: rows r and dim1 - 1 - r swapped
    const int64_t half = int64_t(dim1 / 2) * dim2;
    if (t.px_norm.ptr && half > 0)
        k_flip_px_norm<<<unsigned(std::min<int64_t>((half + 255) / 256, 148 * 16)), 256, 0, s>>>(
            t.px_norm.ptr, dim1, dim2);
    if (t.nnz > 0)
        k_flip_rows<<<148 * 8, 256, 0, s>>>(t.entry.ptr, t.entry_std.ptr, t.nnz, nullptr, 0, dim1,
                                            dim2);
    DG_CUDA(cudaGetLastError());
    // bin tiles and frame-lane units are built later and flipped then
}

void prepare_raw(GatherTable &t, const DeviceCsr &table, const double *d_norm, cudaStream_t s) {
    if (t.cnt.ptr) return;
    t.entry_raw.alloc(std::max<size_t>(size_t(table.nnz), 1));
    t.cnt.alloc(std::max<size_t>(size_t(table.n_rows), 1));
    if (table.n_rows > 0) {
#define DG_PACK_ARGS                                                                     \
    table.row_ptr.ptr, int(table.n_rows), table.col.ptr, table.w.ptr, d_norm,            \
        t.entry_raw.ptr, t.cnt.ptr, t.flip_rows, t.flip_cols
        if (pack_cta_per_row(table.nnz, table.n_rows))
            k_pack_raw<256><<<unsigned(table.n_rows), kPackThreads, 0, s>>>(DG_PACK_ARGS);
        else
            k_pack_raw<32><<<unsigned((table.n_rows + 7) / 8), kPackThreads, 0, s>>>(DG_PACK_ARGS);
#undef DG_PACK_ARGS
    }
    DG_CUDA(cudaGetLastError());
}

namespace {

// Per-frame masks on a mapping-8 plan (raw sums S, N, V, C, or the normalised
// results), and raw sums over the plan mask on a bin-tile plan: the tiles take them.
bool bin_tiles_take_raw(const GatherTable &t, int dtype, int64_t n_pixels, int mode, bool raw) {
    return bin_tiles_reach(dtype, n_pixels) &&
           (mode == kRaw ? t.variant == 8 && t.entry_raw.ptr
                         : raw && gather_variant_needs_tiles(t.variant)) &&
           t.bt[t.variant - 7].n_items > 0;
}

template <typename P>
bool launch_raw(GatherTable &t, const void *frames, int64_t n_pixels, int nf, int mode,
                const uint8_t *masks, int64_t mask_stride, cudaStream_t s, bool raw, double *o0,
                double *o1, double *o2, double *o3) {
    const P *fp = static_cast<const P *>(frames);
    if (bin_tiles_take_raw(t, dtype_code<P>(), n_pixels, mode, raw)) {
        BinCall c{};
        c.frames = frames;
        c.dtype = dtype_code<P>();
        c.mode = mode;
        c.n_pixels = n_pixels;
        c.n_frames = nf;
        c.out_i = o0;
        c.out_s = raw ? o2 : o1;
        c.out_d = raw ? o1 : nullptr;
        c.out_c = raw ? o3 : nullptr;
        c.raw = raw ? 1 : 0;
        c.masks = masks;
        c.mask_stride = mask_stride;
        c.partial = t.partial.ptr;
        launch_bin_tiles(t, t.variant, c, s);
        return true;
    }
    if (mode == kRaw)
        launch_gather<kRaw, P>(t, t.variant, fp, n_pixels, nf, t.partial.ptr, s, masks, mask_stride);
    else if (mode == kErrors)
        launch_gather<kErrors, P>(t, t.variant, fp, n_pixels, nf, t.partial.ptr, s);
    else
        launch_gather<kIntensity, P>(t, t.variant, fp, n_pixels, nf, t.partial.ptr, s);
    return false;
}

}  // namespace

void run_gather_raw(GatherTable &t, const void *d_frames, int dtype, int64_t n_pixels,
                    int64_t n_frames, const uint8_t *d_masks, int64_t mask_stride, uint32_t flags,
                    bool raw, double *o0, double *o1, double *o2, double *o3, cudaStream_t s) {
    if (n_frames <= 0) return;
    if (dtype < DG_U16 || dtype > DG_F64) fail(DG_INVALID_INPUT, "unknown pixel dtype");
    if (!t.cnt.ptr) fail(DG_DEVICE, "raw-sum entries were not prepared");
    const bool errors = (flags & DG_ERRORS) != 0;
    const int mode = d_masks ? kRaw : errors ? kErrors : kIntensity;
    const int64_t chunk = 256;
    // the partial sums of the mapping that runs
    const int64_t rows = bin_tiles_take_raw(t, dtype, n_pixels, mode, raw)
                             ? bin_tile_partials(t, t.variant)
                             : std::max<int64_t>(1, t.n_segments);
    const int64_t need = rows * n_accumulators(mode, dtype == DG_F32 || dtype == DG_F64) *
                         std::min<int64_t>(chunk, (n_frames + 31) / 32 * 32);
    if (t.partial.count < size_t(need)) t.partial.alloc(size_t(need));
    t.scratch.wait(s);
    const size_t esize = dtype == DG_U16 ? 2 : dtype == DG_F64 ? 8 : 4;
    for (int64_t f0 = 0; f0 < n_frames; f0 += chunk) {
        const int nf = int(std::min<int64_t>(chunk, n_frames - f0));
        const void *fp = static_cast<const unsigned char *>(d_frames) + f0 * n_pixels * esize;
        const uint8_t *mp = d_masks ? d_masks + f0 * mask_stride : nullptr;
        const int64_t off = f0 * t.n_rows;
        auto at = [&](double *o) { return o ? o + off : nullptr; };
        bool done = false;  // raw sums written by the bin tiles themselves
        if (t.n_units > 0) {
            std::pair<cudaEvent_t, cudaEvent_t> *ev = nullptr;
            if (t.profile) {
                EventPool &p = t.events;
                if (p.used == p.events.size()) {
                    std::pair<cudaEvent_t, cudaEvent_t> e{};
                    DG_CUDA(cudaEventCreate(&e.first));
                    DG_CUDA(cudaEventCreate(&e.second));
                    p.events.push_back(e);
                }
                ev = &p.events[p.used++];
                DG_CUDA(cudaEventRecord(ev->first, s));
            }
            ++t.launches;
            // raw: S, N, V, C; normalised (per-frame masks only): I, sigma
            double *r0 = at(o0), *r1 = at(o1), *r2 = raw && errors ? at(o2) : nullptr,
                   *r3 = raw ? at(o3) : nullptr;
            if (!raw && !errors) r1 = nullptr;
#define DG_RAW_CALL(T) \
    done = launch_raw<T>(t, fp, n_pixels, nf, mode, mp, mask_stride, s, raw, r0, r1, r2, r3)
            switch (dtype) {
            case DG_U16: DG_RAW_CALL(uint16_t); break;
            case DG_U32: DG_RAW_CALL(uint32_t); break;
            case DG_I32: DG_RAW_CALL(int32_t); break;
            case DG_F32: DG_RAW_CALL(float); break;
            case DG_F64: DG_RAW_CALL(double); break;
            }
#undef DG_RAW_CALL
            if (ev) DG_CUDA(cudaEventRecord(ev->second, s));
        }
        if (t.n_rows == 0 || done) continue;
        ++t.launches;
        const dim3 grid(unsigned((t.n_rows + kFinRows - 1) / kFinRows), unsigned((nf + 31) / 32));
        if (raw) {
#define DG_RAW_ARGS                                                                          \
    t.partial.ptr, t.row_seg.ptr, t.seg_ids.ptr, t.den.ptr, t.cnt.ptr, t.n_rows, nf, at(o0), \
        at(o1), errors ? at(o2) : nullptr, at(o3)
            if (mode == kRaw) k_finalize_raw<kRaw><<<grid, 32 * kFinRows, 0, s>>>(DG_RAW_ARGS);
            else if (mode == kErrors) k_finalize_raw<kErrors><<<grid, 32 * kFinRows, 0, s>>>(DG_RAW_ARGS);
            else k_finalize_raw<kIntensity><<<grid, 32 * kFinRows, 0, s>>>(DG_RAW_ARGS);
#undef DG_RAW_ARGS
            DG_CUDA(cudaGetLastError());
        } else {
            if (mode != kRaw) fail(DG_INVALID_INPUT, "normalised results need per-frame masks");
            double *oi = at(o0), *os = errors ? at(o1) : nullptr;
            launch_finalize<kRaw, float>(t, t.partial.ptr, nf, oi, os, nullptr, s);
        }
    }
    t.scratch.mark(s);
}

namespace {

// One integration with mapping `variant`: the gather and, unless it wrote the
// results itself, the finalize (the autotuner compares whole integrations).
template <typename P>
void launch_mode(GatherTable &t, int variant, int mode, const void *frames, int64_t n_pixels,
                 int nf, double *oi, double *os, double *od, cudaStream_t s) {
    if (!launch_typed<P>(t, variant, frames, n_pixels, nf, mode, t.partial.ptr, oi, os, od, s) &&
        t.n_rows > 0)
        finalize_typed<P>(t, mode, t.partial.ptr, nf, oi, os, od, s);
}

}  // namespace

int gather_variant_count() { return kVariantCount; }

bool gather_variant_available(const GatherTable &t, int variant) {
    if (variant < 0 || variant >= kVariantCount) return false;
    if (variant == 5 || variant == 6) return t.fl_n_units > 0;
    if (variant == 7 || variant == 8) return t.bt[variant - 7].n_items > 0;
    if (variant == 10) return t.rw_n_items > 0;
    return true;
}

int autotune_gather(GatherTable &t, const void *d_frames, int dtype, int64_t n_pixels,
                    int64_t n_frames, uint32_t flags, cudaStream_t s,
                    std::vector<double> *each) {
    if (dtype < DG_U16 || dtype > DG_F64) fail(DG_INVALID_INPUT, "unknown pixel dtype");
    if (n_frames <= 0) fail(DG_INVALID_INPUT, "autotuning needs at least one frame");
    const int mode = (flags & DG_AZIMUTHAL_STD) ? kSpread : (flags & DG_ERRORS) ? kErrors
                                                                                : kIntensity;
    const int nf = int(std::min<int64_t>(n_frames, 256));
    reserve_partials(t, nf, flags, dtype, true);
    t.scratch.wait(s);
    if (each) each->assign(size_t(kVariantCount), 0.0);
    if (t.n_units == 0) return t.variant;
    DeviceArray<double> outs;
    outs.alloc(size_t(std::max<int64_t>(1, int64_t(t.n_rows) * nf * 3)));
    double *oi = outs.ptr, *os = oi + int64_t(t.n_rows) * nf, *od = os + int64_t(t.n_rows) * nf;
    if (!(flags & DG_ERRORS)) os = nullptr;
    if (!(flags & DG_AZIMUTHAL_STD)) od = nullptr;
    cudaEvent_t a = nullptr, b = nullptr;
    DG_CUDA(cudaEventCreate(&a));
    DG_CUDA(cudaEventCreate(&b));
    int best = t.variant;
    float best_t = 3.4e38f;
    try {
        for (int v = 0; v < kVariantCount; ++v) {
            if (!gather_variant_available(t, v) ||
                (gather_variant_needs_tiles(v) && !bin_tiles_fill_gpu(t, v, n_frames))) {
                if (each) (*each)[size_t(v)] = -1.0;
                continue;
            }
            float vt = 3.4e38f;
            for (int rep = 0; rep < 4; ++rep) {
                DG_CUDA(cudaEventRecord(a, s));
                switch (dtype) {
                case DG_U16: launch_mode<uint16_t>(t, v, mode, d_frames, n_pixels, nf, oi, os, od, s); break;
                case DG_U32: launch_mode<uint32_t>(t, v, mode, d_frames, n_pixels, nf, oi, os, od, s); break;
                case DG_I32: launch_mode<int32_t>(t, v, mode, d_frames, n_pixels, nf, oi, os, od, s); break;
                case DG_F32: launch_mode<float>(t, v, mode, d_frames, n_pixels, nf, oi, os, od, s); break;
                case DG_F64: launch_mode<double>(t, v, mode, d_frames, n_pixels, nf, oi, os, od, s); break;
                }
                DG_CUDA(cudaEventRecord(b, s));
                DG_CUDA(cudaEventSynchronize(b));
                float ms = 0.f;
                DG_CUDA(cudaEventElapsedTime(&ms, a, b));
                if (rep > 0 && ms < vt) vt = ms;  // first launch warms caches
            }
            if (each) (*each)[size_t(v)] = vt;
            if (vt < best_t) {
                best_t = vt;
                best = v;
            }
        }
    } catch (...) {
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        throw;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    t.scratch.mark(s);
    t.variant = best;
    return best;
}

}  // namespace dg

// ---------------------------------------------------------------------------
// Fixed scratch of the allocation-free entry point (dg_integrate_device_noalloc
// in dg_api.cu).
//
// Some callers may not allocate device memory while they integrate: a
// real-time acquisition loop with a fixed memory budget, a host thread that
// must not enter the CUDA allocator, code running where cudaMalloc is not
// permitted. dg_integrate_device allocates its per-segment partial sums on
// first use; the allocation-free entry point keeps them in this one fixed
// array instead. It is a file-scope __device__ variable of
// kNoAllocScratchBytes, which every GPU that loads the library holds until
// the process exits. Host code cannot use its name as a device address (a
// kernel given the host-side name would fault or read the wrong memory), so
// its address is looked up with cudaGetSymbolAddress, with the device
// current, on every call: the lookup allocates nothing once the module is
// loaded, the first call on a device loads it (make that call before any
// stream capture), and an address never outlives a context that was reset.
namespace dg {
namespace {
constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;  // 32 MiB per device
static __device__ __align__(256) double g_noalloc_partial[kNoAllocScratchBytes / sizeof(double)];
}  // namespace

double *noalloc_scratch(size_t *n_doubles) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partial);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        fail(DG_DEVICE, std::string("cudaGetSymbolAddress of the fixed scratch array failed: ") +
                            cudaGetErrorString(e));
    }
    *n_doubles = kNoAllocScratchBytes / sizeof(double);
    return static_cast<double *>(p);
}

}  // namespace dg
