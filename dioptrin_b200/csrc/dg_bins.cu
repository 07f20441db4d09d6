// Bin-tile gathers (lane mappings 7 and 8): batches of frames over tiles of
// consecutive bins.
//
// A tile is ROWS consecutive rows (bins) of the table and 32 * F2 frames (lane
// = frame; F2 frames per lane, 32 apart). The tile's entries, merged over its
// rows in pixel order, are cut at plan time into chunks of at most DCAP
// distinct pixels and PCAP entry pairs; a row's entries inside a chunk are a
// contiguous run of its CSR row, taken in pairs (an odd run ends with a padding
// entry of weight 0). Consumer warp w owns row w of the tile and keeps its
// sums in registers: FP32 pairs of the row in plan order, folded every
// kBtFoldPairs pairs into FP64. Every row is summed in the same order for every
// frame and batch.
//
// Producers and consumers. The kernel is persistent, one CTA per SM, and runs
// its work items' chunks as one stream through a ring of BUFS shared-memory
// buffers. Producer warps stage a chunk: its pixels (4-byte pixel types by
// 4-byte cp.async, one instruction per 32 pixels of a frame; 2-byte ones alike, as
// the words that hold them; 8-byte ones by cp.async into a ring of the warp's own,
// then converted to FP32 and stored) into frame rows STRIDE words apart (odd, so
// the 32 lanes reading one pixel of their frames hit 32 banks), and by one thread's
// bulk copies its pair records and row offsets. Consumer warps only sum. "full"
// barriers count the producers' copies, "empty" barriers the
// consumer warps that have summed the buffer's chunk. When every warp staged a
// share of each chunk between its sums, 512 threads arrived three times per
// chunk on barriers in shared memory, the staging addresses took registers of
// the sums (114), each tile began with an empty pipeline, and a batch ended with
// its largest tile. Before and now, mapping 8, us: Eiger-4M uint32 with the
// spread, 256 / 128 / 64 frames 1857 / 1117 / 1099 and 1738 / 897 / 465; float32,
// 128 frames 1935 and 1218; per-frame masks, 64 frames 2024 and 837; Pilatus 1M,
// 256 / 50 frames 408 / 362 and 405 / 109. (256 Eiger frames draw the chip's full
// power; at the lower clock of a run of seconds they take 1900 and 1885.)
//
// Work items. Rings of large radius hold many times the entries of small ones,
// and a batch of one or two frame groups has fewer tiles than SMs, so a tile of
// many chunks is cut into pieces (kBtPieceMin), which CTAs claim largest first
// from one counter, neighbouring tiles' pieces one after the other (build_bin_tiles),
// all pieces for one frame group, then the next group. A row is cut where its FP32 sums are folded, so its sums round as in
// one piece; a piece leaves FP64 partial sums, and the CTA that finishes a
// tile's last piece adds them in piece order. A finished tile is normalised and
// written through shared memory, so that a frame's ROWS results are one run.
//
// 2-byte pixels went through the ring of the 8-byte ones, two instructions more per
// pixel for few warps and a memory latency per batch of frames; now the sums take
// their half of the word. Mapping 8, u16, us, through the ring and now: Pilatus 1M, 64
// / 256 frames with errors 212 / 665 and 155 / 482, with the spread 309 / 980 and 205 /
// 654; Eiger-4M, 256 frames with the spread 3616 and 2301, per-frame masks, 64 frames
// 1376 and 943.
//
// What bounds it. Four frame groups: DRAM, which reads every frame byte twice (256
// Eiger-4M frames with the spread 9.2 GB in 1764 us, 0.80 of the measured copy rate).
// One group: the load-store unit, whose data pipe is busy for 58 to 67 % of the
// cycles, more than any other unit (64 frames with the spread: DRAM at 48 % of its
// nominal rate, issue slots 47 %). A 4-byte cp.async of 32 pixels that lie in
// two or three short runs holds it for about 11 cycles (two per 32-byte sector);
// on the Eiger-4M table a chunk's 320 copies take 3670 cycles alone, its sums
// 3380, together 4400. 16-byte copies of the runs (rows on 16-byte boundaries,
// half the instructions) made as many sector requests and were no faster; TMA
// boxes take 6.3 cycles per frame row, more than cp.async; loads through
// registers hide too little latency.
//
// Every wait is bounded (kBtWaitNs); a warp that gives up stops reporting
// chunks, which ends the others' waits too, and sets a flag in mapped host
// memory that the host reports as DG_TIMEOUT.
//
// In mode kRaw the kernel applies per-frame masks: a word of frame bits per pixel
// (k_mask_words) is staged next to a chunk's pixels, and a masked entry adds
// nothing to S, V, N or C.
#include <algorithm>
#include <atomic>
#include <climits>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>

#include "dg_gather_common.cuh"

namespace dg {
namespace {

// Pairs of a row summed in plain FP32 (each half of a packed accumulator
// takes one entry per pair) before they are folded into FP64.
constexpr int kBtFoldPairs = 32;
// Chunks of a piece, at most: a 350th of the plan's chunks (two to three pieces
// per SM and frame group), between two bounds. A piece stages up to three chunks
// more than its share (where its rows end) and leaves partial sums; long pieces
// leave SMs idle at the end. Measured at 48 / 64 / 80 chunks: Pilatus-1M (6,640
// chunks), 256 frames 418 / 405 / 417 us, 50 frames 141 / 108 / 133; at 48 / 64 /
// 80 / 96: Eiger-4M (27,600), 256 frames 2030 / 1930 / 1873 / 1872 us, 64 frames
// 548 / 535 / 502 / 529 (before the pieces' sums were added in the kernel).
constexpr int kBtPieceMin = 64, kBtPieceMax = 96;

// Claimed items in flight between the claiming warp and the other producers: a
// producer is at most BUFS chunks, so at most BUFS + 1 items (every item has a
// chunk), behind it.
constexpr int kBtWork = 8;

// One bin-tile layout: rows per tile (= consumer warps), chunk capacities,
// frames per lane, pairs per step (the fold cadence counts whole steps) and
// buffers. Per-chunk record, fixed size: {pixels D, pairs, first pair, 0}, the
// rows' pair offsets (ROWS + 1, padded to a multiple of 4 words), then D pixel
// indices.
template <int ROWS, int DCAP, int PCAP, int F2, int U2, int BUFS>
struct BtCfg {
    static constexpr int kRows = ROWS;
    static constexpr int kU2 = U2;
    static_assert(BUFS + 2 <= kBtWork, "claimed items are not overwritten before they are read");
    static_assert(ROWS <= 32, "tile rows are packed in 5 bits at plan time");
    static constexpr int kDCap = DCAP;          // distinct pixels per chunk
    static constexpr int kStride = DCAP + 1;    // odd frame-row stride; column DCAP stays 0
    static constexpr int kPCap = PCAP;          // entry pairs per chunk
    static constexpr int kF2 = F2;              // frames per lane
    static constexpr int kFrames = 32 * F2;     // frames per CTA
    static constexpr int kMetaHead = (4 + ROWS + 1 + 3) / 4 * 4;
    static constexpr int kMetaWords = kMetaHead + DCAP;
    static_assert(kMetaWords % 4 == 0, "records are copied in 16-byte pieces");
    static_assert(kStride % 2 == 1, "frame rows must start in different banks");
    // Producer warps: two are too few to keep the copies of two buffers in flight
    // (Eiger-4M batch with the spread 2166 against 1908 us); eight leave the sums
    // of the spread 80 registers (2091), but the other modes need no more (Pilatus
    // batch 401 against 416 us; masks 845 against 1042).
    template <int MODE, typename P>
    static constexpr int producers() {
        return MODE == kSpread ? 4 : 8;
    }
    // Frames a producer's copy loop is unrolled by: bursts of copies hold the
    // load-store unit against the sums' loads.
    template <int MODE>
    static constexpr int copy_unroll() {
        return MODE == kSpread ? 2 : F2 == 1 ? 1 : 4;
    }
    template <int MODE, typename P>
    static constexpr int threads() {
        return (ROWS + producers<MODE, P>()) * 32;
    }
    // 8-byte pixels: a producer copies batches of raw_frames frames into a ring of its
    // own of two batches.
    static constexpr int kLaneSlots = (DCAP + 31) / 32;
    static constexpr int kRawFrames = kLaneSlots > 6 ? 1 : 2;
    template <int MODE, typename P>
    static constexpr size_t raw_bytes() {
        return sizeof(P) == 8 ? size_t(producers<MODE, P>()) * 2 * kRawFrames * kLaneSlots * 32 * 8 : 0;
    }
    template <typename P>
    static constexpr int bufs() {  // the ring of mapping 7 takes the third buffer's place
        return sizeof(P) != 8 || F2 == 2 ? BUFS : 2;
    }
    // A buffer: frame rows, pairs A, then B (spread, masks), C (spread), the
    // record's head, then a word of frame bits per slot (masks); every part
    // 16-byte aligned.
    static constexpr size_t kPairOff = size_t(kFrames) * kStride * 4;
    template <int MODE>
    static constexpr size_t head_off() {
        return kPairOff + size_t(PCAP) * (MODE == kSpread ? 40 : MODE == kRaw ? 32 : 16);
    }
    template <int MODE>
    static constexpr size_t buf_bytes() {
        return head_off<MODE>() + size_t(kMetaHead) * 4 +
               (MODE == kRaw ? size_t(DCAP + 2) / 2 * 16 : 0);
    }
    static_assert(kPairOff % 16 == 0 && PCAP % 2 == 0, "16-byte parts");
    // Results of a whole tile on their way out: [frame][row], odd row stride.
    static constexpr int kOutStride = ROWS + 1;
    template <int MODE, typename P>
    static constexpr size_t raw_off() {
        return size_t(bufs<P>()) * buf_bytes<MODE>();
    }
    template <int MODE, typename P>
    static constexpr size_t out_off() {
        return raw_off<MODE, P>() + raw_bytes<MODE, P>();
    }
    // Then the mbarriers full[BUFS], empty[BUFS], work[kBtWork], out, the claimed
    // items work[kBtWork] and each buffer's {item, group}.
    template <int MODE, typename P>
    static constexpr size_t bar_off() {
        return out_off<MODE, P>() + size_t(kFrames) * kOutStride * 8;
    }
    template <int MODE, typename P>
    static constexpr size_t work_off() {
        return bar_off<MODE, P>() + size_t(2 * BUFS + kBtWork + 1) * 8;
    }
    template <int MODE, typename P>
    static constexpr size_t smem_bytes() {
        return work_off<MODE, P>() + size_t(kBtWork) * 8 + size_t(BUFS) * 8;
    }
};
using Bt7 = BtCfg<24, 384, 640, 1, 4, 3>;  // mapping 7
using Bt8 = BtCfg<16, 160, 256, 2, 4, 3>;  // mapping 8
template <class CFG, typename P>
constexpr bool bt_fits() {
    return CFG::template smem_bytes<kSpread, P>() <= 227 * 1024 &&
           CFG::template smem_bytes<kErrors, P>() <= 227 * 1024 &&
           (CFG::kF2 == 1 || CFG::template smem_bytes<kRaw, P>() <= 227 * 1024);
}
static_assert(bt_fits<Bt7, float>() && bt_fits<Bt7, double>() && bt_fits<Bt7, uint16_t>() &&
                  bt_fits<Bt8, float>() && bt_fits<Bt8, double>() && bt_fits<Bt8, uint16_t>(),
              "bin tiles fit shared memory");

// Pairs per step of a mode: float pixels with the spread count in steps of two.
template <int MODE, typename P, class CFG>
constexpr int bt_step() {
    return MODE == kSpread && is_float_px<P>() && CFG::kU2 > 2 ? 2 : CFG::kU2;
}

// ------------------------------------------------- barriers and copies

__device__ __forceinline__ unsigned smem_addr(const void *p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(b), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(b) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(unsigned b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(b), "r"(bytes)
                 : "memory");
}
// Arrives (without raising the expected count) once all of this thread's
// earlier cp.async copies have landed.
__device__ __forceinline__ void mbar_arrive_copies(unsigned b) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(b) : "memory");
}
__device__ __forceinline__ void cp_async8_s(unsigned d, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
// One contiguous copy of `bytes` (a multiple of 16, both ends 16-byte aligned)
// counted on barrier b.
__device__ __forceinline__ void copy_bulk(unsigned dst, const void *src, unsigned bytes, unsigned b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
                 "[%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(b)
                 : "memory");
}
// Waits for the phase of the given parity to complete; gives up (false)
// after kBtWaitNs of global time, so a lost arrival cannot hang the GPU.
constexpr uint64_t kBtWaitNs = 1000000000ull;
__device__ __forceinline__ bool mbar_try(unsigned a, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    return now;
}
__device__ __forceinline__ bool mbar_wait(unsigned a, unsigned parity) {
    if (mbar_try(a, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try(a, parity))
        if (global_ns() - t0 > kBtWaitNs) return false;
    return true;
}
// 32-bit shared-memory load at a constant offset from a register.
template <int OFF>
__device__ __forceinline__ uint32_t lds32_at(unsigned a) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1+%2];\n" : "=r"(v) : "r"(a), "n"(OFF));
    return v;
}
__device__ __forceinline__ uint2 lds64(unsigned a) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}

// ------------------------------------------------------------- the kernel

struct BinArgs {
    const int4 *items;   // {first row, rows, first chunk, chunks}
    const int4 *spans;   // per (item, row) {chunk, pair} to start at and to end at; null: whole
    const int32_t *meta;
    const float4 *pair_a, *pair_b;
    const float2 *pair_c;
    const int4 *org;
    const float4 *entry_std;
    const double *den, *den_std;
    const int32_t *valid_std;
    const void *frames;
    int64_t n_pixels;
    int32_t n_frames, n_rows, n_items, groups;
    int32_t *counter;    // {next claim, CTAs done}, both 0 between launches
    double *out_i, *out_s, *out_d, *out_c;
    // With spans: partial sums [slot row][accumulator][frame], the slots of the
    // items, every row's slot rows (the table's in row_part), and the pieces done
    // per (tile, group), 0 between launches.
    double *partial;
    const int32_t *slot, *row_part, *part_ids;
    int32_t *tile_done;
    const double *raw_cnt;
    const uint64_t *mask_words;  // per group and pixel: bit f masks frame f of the group
    int *wait_err;
    int32_t raw, withhold;
};

template <int MODE, typename P, class CFG>
__global__ void __launch_bounds__(CFG::template threads<MODE, P>(), 1)
    k_gather_bins(const __grid_constant__ BinArgs a) {
    using S = StagedPx<P>;
    constexpr int NA = NAcc<MODE, P>::value;
    constexpr bool SPREAD = MODE == kSpread;
    constexpr bool WIDE = SPREAD || MODE == kRaw;  // pairs B
    constexpr bool FLOAT_SPREAD = SPREAD && is_float_px<P>();
    constexpr bool HALF = sizeof(P) == 2;                    // pixels as the words that hold them
    constexpr bool COPIES = sizeof(P) == 4 || HALF;          // pixels by cp.async
    constexpr bool ASYNC = COPIES || MODE == kRaw;           // some cp.async per chunk
    constexpr bool STORES = sizeof(P) != 4;                  // plain stores (2-byte: of a frame's ends)
    constexpr int F2 = CFG::kF2, STRIDE = CFG::kStride, DCAP = CFG::kDCap, PCAP = CFG::kPCap;
    constexpr int U2 = bt_step<MODE, P, CFG>();
    constexpr int NW = CFG::kRows, NP = CFG::template producers<MODE, P>(), NB = CFG::template bufs<P>();
    constexpr int NT = CFG::template threads<MODE, P>();
    constexpr int MH = CFG::kMetaHead, MW = CFG::kMetaWords;
    constexpr unsigned BUF = unsigned(CFG::template buf_bytes<MODE>());
    constexpr unsigned PAIRS = unsigned(CFG::kPairOff);
    constexpr unsigned HEAD = unsigned(CFG::template head_off<MODE>());
    constexpr unsigned MASKS = HEAD + unsigned(MH) * 4;
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned base = smem_addr(smem);
    const unsigned full = base + unsigned(CFG::template bar_off<MODE, P>()), empty = full + 8 * NB;
    const unsigned work = empty + 8 * NB, out_bar = work + 8 * kBtWork;
    volatile int2 *s_work = reinterpret_cast<volatile int2 *>(smem + CFG::template work_off<MODE, P>());
    // {item, frame group} of the chunk in a buffer; item -1: the end
    volatile int2 *s_info = s_work + kBtWork;
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31;
    // the warp's number, known to be the same in every lane
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

    if (tid == 0) {
        for (int b = 0; b < NB; ++b) {
            // one expect_tx, the copying threads, the storing warps
            mbar_init(full + 8 * b, 1 + (ASYNC ? NP * 32 : 0) + (STORES ? NP : 0));
            mbar_init(empty + 8 * b, NW);
        }
        for (int k = 0; k < kBtWork; ++k) mbar_init(work + 8 * k, 1);
        mbar_init(out_bar, NW);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // Column DCAP of a frame row is read by padding pairs and stays 0. Rows of frames
    // past the batch hold zeros or an earlier group's pixels: their sums go nowhere
    // (results and partial sums are stored for frames below nv alone).
    for (int b = 0; b < NB; ++b) {
        uint32_t *px = reinterpret_cast<uint32_t *>(smem + size_t(b) * BUF);
        for (int j = tid; j < CFG::kFrames * STRIDE; j += NT) px[j] = 0;
        if constexpr (MODE == kRaw) {
            uint64_t *mk = reinterpret_cast<uint64_t *>(smem + size_t(b) * BUF + MASKS);
            for (int j = tid; j <= DCAP; j += NT) mk[j] = 0;
        }
    }
    __syncthreads();

    const int total = a.n_items * a.groups;
    const P *__restrict__ frames = static_cast<const P *>(a.frames);
    unsigned b = 0, q = 0;  // ring buffer and its use count, continued over the items
    bool ok = true;

    if (warp >= NW) {
        // ------------------------------------------------------- producers
        constexpr int KSTEP = (DCAP + 31) / 32;
        const int pw = warp - NW;
        const bool claims = pw == 0 && lane == 0;
        int claim = claims ? atomicAdd(a.counter, 1) : 0;
        for (int n = 0; ok; ++n) {
            // the claiming thread hands the item it claimed an item ago to the
            // producers (a slot is read before it comes round again, kBtWork)
            const unsigned slot = unsigned(n) % kBtWork;
            if (claims) {
                // all items for one frame group, then the next group
                const int g = claim / a.n_items;
                s_work[slot].x = claim < total ? claim - g * a.n_items : -1;
                s_work[slot].y = g;
                mbar_arrive(work + 8 * slot);
                if (claim < total) claim = atomicAdd(a.counter, 1);
            }
            ok = mbar_wait(work + 8 * slot, unsigned(n) / kBtWork & 1u);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            const int item = s_work[slot].x, group = s_work[slot].y;
            if (item < 0) {
                // the end of the stream, in a buffer of its own
                if (q > 0) ok = mbar_wait(empty + 8 * b, (q - 1) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (claims) {
                    s_info[b].x = -1;
                    mbar_arrive(full + 8 * b);
                }
                if constexpr (ASYNC) mbar_arrive(full + 8 * b);
                if constexpr (STORES) {
                    if (lane == 0) mbar_arrive(full + 8 * b);
                }
                break;
            }
            const int4 it = a.items[item];
            // this warp's frames of the group, from fw on (nf may be <= 0): even shares,
            // but for 4-byte pixels fixed ones (with even ones a Pilatus batch of 256,
            // whose shares are the same, took 417 us against 399)
            const int gf = min(CFG::kFrames, a.n_frames - group * CFG::kFrames);
            const int per = sizeof(P) == 4 ? CFG::kFrames / NP : (gf + NP - 1) / NP, fw = pw * per;
            const int nf = min(per, gf - fw);
            const P *fbase = frames + int64_t(group * CFG::kFrames + fw) * a.n_pixels;
            const int32_t *rec = a.meta + int64_t(it.z) * MW;
            // the next chunk's record is read while this one's copies are issued
            int n_px = rec[0], n_pr = rec[1], first = rec[2];
            uint32_t ix[KSTEP];
#pragma unroll
            for (int i = 0; i < KSTEP; ++i) ix[i] = uint32_t(rec[MH + min(lane + 32 * i, DCAP - 1)]);
            for (int c = 0; c < it.w; ++c) {
                const int d = n_px, pr = n_pr, pr0 = first;
                uint32_t px[KSTEP];
#pragma unroll
                for (int i = 0; i < KSTEP; ++i) px[i] = ix[i];
                if (c + 1 < it.w) {
                    rec += MW;
                    n_px = rec[0];
                    n_pr = rec[1];
                    first = rec[2];
#pragma unroll
                    for (int i = 0; i < KSTEP; ++i)
                        ix[i] = uint32_t(rec[MH + min(lane + 32 * i, DCAP - 1)]);
                }
                if (q > 0) ok = mbar_wait(empty + 8 * b, (q - 1) & 1u);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
                const unsigned buf = base + b * BUF, bar = full + 8 * b;
                if (pw == 0 && lane == 0) {
                    s_info[b].x = item;
                    s_info[b].y = group;
                    const unsigned na = unsigned(pr) * 16u, nc = unsigned(pr + 1) / 2u * 16u;
                    mbar_arrive_tx(bar, unsigned(MH) * 4u + na + (WIDE ? na : 0u) + (SPREAD ? nc : 0u));
                    copy_bulk(buf + HEAD, a.meta + (int64_t(it.z) + c) * MW, unsigned(MH) * 4u, bar);
                    copy_bulk(buf + PAIRS, a.pair_a + pr0, na, bar);
                    if (WIDE) copy_bulk(buf + PAIRS + PCAP * 16u, a.pair_b + pr0, na, bar);
                    if (SPREAD) copy_bulk(buf + PAIRS + PCAP * 32u, a.pair_c + pr0, nc, bar);
                }
                bool in[KSTEP];
#pragma unroll
                for (int i = 0; i < KSTEP; ++i) in[i] = lane + 32 * i < d;
                unsigned dst = buf + unsigned(fw * STRIDE + lane) * 4u;
                const char *src = reinterpret_cast<const char *>(fbase);
                if constexpr (HALF) {
                    // 2-byte pixels as the aligned words that hold them, and the sums take
                    // their half; at the ends of a frame, where that word may reach outside
                    // the array, a word made of the pixel.
                    bool ends = false;
#pragma unroll
                    for (int i = 0; i < KSTEP; ++i) {
                        const bool end = in[i] && (px[i] == 0 || px[i] + 1 == a.n_pixels);
                        ends = ends || end;
                        in[i] = in[i] && !end;
                        px[i] *= 2u;
                    }
                    if (__any_sync(0xffffffffu, ends)) {
                        uint32_t *rows = reinterpret_cast<uint32_t *>(smem + b * BUF) + fw * STRIDE + lane;
#pragma unroll
                        for (int i = 0; i < KSTEP; ++i)
                            if (lane + 32 * i < d && !in[i])
                                for (int f = 0; f < nf; ++f) {
                                    const P *at = fbase + int64_t(f) * a.n_pixels + px[i] / 2u;
                                    rows[f * STRIDE + 32 * i] =
                                        uint32_t(__ldg(at)) << (unsigned(reinterpret_cast<uintptr_t>(at)) & 2u) * 8u;
                                }
                    }
                    constexpr int UNROLL = CFG::template copy_unroll<MODE>();
#pragma unroll UNROLL
                    for (int f = 0; f < nf; ++f) {
                        const unsigned low = unsigned(reinterpret_cast<uintptr_t>(src)) & 2u;
                        const char *fs = src - low;
#pragma unroll
                        for (int i = 0; i < KSTEP; ++i)
                            if (in[i]) cp_async4_s(dst + 128u * i, fs + ((px[i] + low) & ~3u));
                        dst += STRIDE * 4u;
                        src += a.n_pixels * 2;
                    }
                } else if constexpr (COPIES) {
#pragma unroll
                    for (int i = 0; i < KSTEP; ++i) px[i] *= 4u;
                    constexpr int UNROLL = CFG::template copy_unroll<MODE>();
#pragma unroll UNROLL
                    for (int f = 0; f < nf; ++f) {
#pragma unroll
                        for (int i = 0; i < KSTEP; ++i)
                            if (in[i]) cp_async4_s(dst + 128u * i, src + px[i]);
                        dst += STRIDE * 4u;
                        src += a.n_pixels * 4;
                    }
                } else {
                    // 8-byte pixels: FB frames' copies into half of this warp's ring
                    // while the other half is converted and stored. A lane reads back
                    // what it copied itself.
                    constexpr int FB = CFG::kRawFrames, SB = FB * KSTEP;
                    P *raw = reinterpret_cast<P *>(smem + CFG::template raw_off<MODE, P>()) +
                             pw * 2 * SB * 32 + lane;
                    const unsigned raw_a = smem_addr(raw);
                    const char *next = src;  // the next frame to copy
                    auto issue = [&](int f, int half) {
#pragma unroll
                        for (int g = 0; g < FB; ++g) {
                            if (f + g >= nf) break;
#pragma unroll
                            for (int i = 0; i < KSTEP; ++i)
                                if (in[i])
                                    cp_async8_s(raw_a + unsigned((half * SB + g * KSTEP + i) * 32) * 8u,
                                                next + size_t(px[i]) * 8u);
                            next += a.n_pixels * 8;
                        }
                        asm volatile("cp.async.commit_group;\n" ::: "memory");
                    };
                    float *rows = reinterpret_cast<float *>(smem + b * BUF) + fw * STRIDE + lane;
                    issue(0, 0);
                    int half = 0;
                    for (int f = 0; f < nf; f += FB) {
                        issue(f + FB, half ^ 1);
                        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
#pragma unroll
                        for (int g = 0; g < FB; ++g) {
                            if (f + g >= nf) break;
#pragma unroll
                            for (int i = 0; i < KSTEP; ++i) {
                                const float v = __double2float_rn(raw[(half * SB + g * KSTEP + i) * 32]);
                                if (in[i]) rows[(f + g) * STRIDE + 32 * i] = v;
                            }
                        }
                        half ^= 1;
                    }
                }
                if constexpr (MODE == kRaw) {
                    // the pixels' words of frame bits, shared out over the warps
                    const uint64_t *words = a.mask_words + int64_t(group) * a.n_pixels;
                    const int32_t *idx = a.meta + (int64_t(it.z) + c) * MW + MH;
                    for (int k = lane + 32 * pw; k < d; k += 32 * NP)
                        cp_async8_s(buf + MASKS + 8u * unsigned(k), words + idx[k]);
                }
                if constexpr (ASYNC) mbar_arrive_copies(bar);
                if constexpr (STORES) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar);
                }
                if (++b == NB) {
                    b = 0;
                    ++q;
                }
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (claims) {
            __threadfence();  // this CTA's claims are made before it counts as done
            if (atomicAdd(a.counter + 1, 1) + 1 == int(gridDim.x)) {
                // no CTA claims any more: the next launch starts at 0
                a.counter[0] = 0;
                a.counter[1] = 0;
            }
        }
        if (!ok && lane == 0) {
            *reinterpret_cast<volatile int *>(a.wait_err) = 1;
            __threadfence_system();
        }
        return;
    }

    // ----------------------------------------------------------- consumers
    const int r = warp;  // row of the tile
    // Failure-detection check (dg_plan_test_wait_timeout): warp 0 of the first
    // CTA never reports a chunk summed, so the waits for its buffers run out.
    const bool signal = !(a.withhold && blockIdx.x == 0 && warp == 0);
    double *s_out = reinterpret_cast<double *>(smem + CFG::template out_off<MODE, P>());
    // All consumer warps (a bounded barrier).
    unsigned out_phase = 0;
    auto consumers_meet = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(out_bar);
        return __all_sync(0xffffffffu, mbar_wait(out_bar, out_phase++ & 1u)) != 0;
    };
    for (;;) {
        // the first chunk of the next item, or the end of the stream
        if (ok) ok = mbar_wait(full + 8 * b, q & 1u);
        if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
        }
        const int item = s_info[b].x, group = s_info[b].y;
        if (item < 0) break;
        const int4 it = a.items[item];
        const int f0 = group * CFG::kFrames;
        const int nv = min(CFG::kFrames, a.n_frames - f0);
        const int row = it.x + r;
        const bool mine = r < it.y;
        int4 span = make_int4(0, 0, INT_MAX, 0);
        if (a.spans && mine) span = a.spans[int64_t(item) * NW + r];
        AccP64 acc[F2][NA - (FLOAT_SPREAD ? 2 : 0)];
#pragma unroll
        for (int h = 0; h < F2; ++h)
#pragma unroll
            for (int k = 0; k < NA - (FLOAT_SPREAD ? 2 : 0); ++k) acc[h][k].zero();
        // weight and count of the excluded non-finite pixels (rare)
        double ex_w[F2];
        int ex_n[F2];
#pragma unroll
        for (int h = 0; h < F2; ++h) {
            ex_w[h] = 0.0;
            ex_n[h] = 0;
        }
        int since = 0;
        // 2-byte pixels: the bytes of a word that hold an even pixel of this lane's frames
        // (alike for frames 32 apart), and the step to an odd one's, below the upper
        // bytes of 2^23: the float 2^23 + pixel, without a conversion's slow unit.
        [[maybe_unused]] unsigned sel_even = 0x7610u, sel_odd = 0x22u;
        if constexpr (HALF)
            if (reinterpret_cast<uintptr_t>(frames + int64_t(f0 + lane) * a.n_pixels) & 2u) {
                sel_even = 0x7632u;
                sel_odd = 0u - 0x22u;
            }
        // Origin of the spread's shift, per frame of the lane (row_origin).
        f2 norg[F2];
#pragma unroll
        for (int h = 0; h < F2; ++h) norg[h] = 0ull;
        if constexpr (SPREAD) {
            if (mine) {
                const int4 o = a.org[row];
#pragma unroll
                for (int h = 0; h < F2; ++h) {
                    const int fi = min(f0 + lane + 32 * h, a.n_frames - 1);
                    const float v =
                        -row_origin<P>(a.entry_std, o.x, o.y, o.z, frames + int64_t(fi) * a.n_pixels);
                    norg[h] = pk(v, v);
                }
            }
        }
        for (int c = 0; c < it.w; ++c) {
            if (c > 0) {
                ok = mbar_wait(full + 8 * b, q & 1u);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
            }
            if (mine) {
                const unsigned char *buf = smem + b * BUF;
                const int32_t *cp = reinterpret_cast<const int32_t *>(buf + HEAD) + 4;
                int p = cp[r], p1 = cp[r + 1];
                const int first = p;
                if (c <= span.x) p = c < span.x ? p1 : first + span.y;
                if (c >= span.z) p1 = c > span.z ? p : first + span.w;
                const unsigned pxa = base + b * BUF + unsigned(lane * STRIDE) * 4u;
                const float4 *s_pa = reinterpret_cast<const float4 *>(buf + PAIRS);
                const float4 *s_pb = s_pa + PCAP;
                const f2 *s_pc = reinterpret_cast<const f2 *>(buf + PAIRS + PCAP * 32u);
                [[maybe_unused]] const unsigned mk = base + b * BUF + MASKS;
                [[maybe_unused]] const unsigned my_bit = 1u << lane;
                auto body = [&](int p, auto unroll) {
                    constexpr int UU = decltype(unroll)::value;
                    float4 ea[UU];
                    [[maybe_unused]] float4 eb[UU];
                    [[maybe_unused]] f2 ec[UU];
#pragma unroll
                    for (int u = 0; u < UU; ++u) {
                        ea[u] = s_pa[p + u];
                        if constexpr (WIDE) eb[u] = s_pb[p + u];
                        if constexpr (SPREAD) ec[u] = s_pc[p + u];
                    }
                    // the pairs' pixels for this lane's frames
                    float v0[F2][UU], v1[F2][UU];
#pragma unroll
                    for (int u = 0; u < UU; ++u) {
                        // slot, and bit 30 (lost in the address): an odd pixel
                        const unsigned s0 = unsigned(__float_as_int(ea[u].x)), s1 = unsigned(__float_as_int(ea[u].y));
                        const unsigned a0 = pxa + 4u * s0, a1 = pxa + 4u * s1;
                        auto value = [&](uint32_t w, [[maybe_unused]] unsigned s) {
                            if constexpr (HALF)
                                return __fadd_rn(__uint_as_float(__byte_perm(
                                                     w, 0x4b000000u, sel_even + (s >> 30) * sel_odd)),
                                                 -8388608.f);
                            else
                                return staged_value<S>(w);
                        };
                        v0[0][u] = value(lds32_at<0>(a0), s0);
                        v1[0][u] = value(lds32_at<0>(a1), s1);
                        if constexpr (F2 == 2) {
                            v0[F2 - 1][u] = value(lds32_at<128 * STRIDE>(a0), s0);
                            v1[F2 - 1][u] = value(lds32_at<128 * STRIDE>(a1), s1);
                        }
                    }
                    if constexpr (MODE == kRaw) {
                        // {slot, slot, w, w}, {w*norm, w*norm, 0, 0}; a masked entry
                        // adds nothing to S, V, N or C, whatever its pixel holds
#pragma unroll
                        for (int h = 0; h < F2; ++h)
#pragma unroll
                            for (int u = 0; u < UU; ++u) {
                                const uint2 w0 = lds64(mk + 8u * unsigned(__float_as_int(ea[u].x)));
                                const uint2 w1 = lds64(mk + 8u * unsigned(__float_as_int(ea[u].y)));
                                const bool l0 = ((h ? w0.y : w0.x) & my_bit) == 0;
                                const bool l1 = ((h ? w1.y : w1.x) & my_bit) == 0;
                                const f2 cc = pk(l0 ? ea[u].z : 0.f, l1 ? ea[u].w : 0.f);
                                const float x0 = l0 ? v0[h][u] : 0.f, x1 = l1 ? v1[h][u] : 0.f;
                                const f2 x = pk(x0, x1);
                                acc[h][0].p = fma2(cc, x, acc[h][0].p);
                                const f2 xp = is_unsigned_px<P>()
                                                  ? x
                                                  : pk(fmaxf(x0, 0.f), fmaxf(x1, 0.f));
                                acc[h][1].p = fma2(mul2(cc, cc), xp, acc[h][1].p);
                                acc[h][2].p = add2(acc[h][2].p,
                                                   pk(l0 ? eb[u].x : 0.f, l1 ? eb[u].y : 0.f));
                                acc[h][3].p = add2(acc[h][3].p, cc);
                            }
                    } else {
                        if constexpr (FLOAT_SPREAD) {
                            // 0 * x summed over the step's pixels is not 0 when one of
                            // them is not finite; such a step is summed entry by entry
                            f2 z = 0ull;
#pragma unroll
                            for (int h = 0; h < F2; ++h)
#pragma unroll
                                for (int u = 0; u < UU; ++u) z = fma2(pk(v0[h][u], v1[h][u]), 0ull, z);
                            const float2 zz = upk(z);
                            if (!(zz.x + zz.y == 0.f)) {
#pragma unroll
                                for (int h = 0; h < F2; ++h)
#pragma unroll
                                    for (int u = 0; u < UU; ++u) {
                                        const bool ok0 = isfinite(v0[h][u]), ok1 = isfinite(v1[h][u]);
                                        const float x0 = ok0 ? v0[h][u] : 0.f, x1 = ok1 ? v1[h][u] : 0.f;
                                        const f2 ce = pk(ok0 ? ea[u].z : 0.f, ok1 ? ea[u].w : 0.f);
                                        const f2 x = pk(x0, x1), n = pk(eb[u].x, eb[u].y);
                                        const f2 cre = pk(ok0 ? eb[u].z : 0.f, ok1 ? eb[u].w : 0.f);
                                        acc[h][0].p = fma2(ce, x, acc[h][0].p);
                                        acc[h][1].p = fma2(mul2(ce, ce), pk(fmaxf(x0, 0.f), fmaxf(x1, 0.f)),
                                                           acc[h][1].p);
                                        const f2 t = fma2(norg[h], ec[u], fma2(norg[h], n, x));
                                        acc[h][2].p = fma2(mul2(cre, t), t, acc[h][2].p);
                                        acc[h][kSpreadA].p = fma2(ce, t, acc[h][kSpreadA].p);
                                        if (!ok0 && ea[u].z > 0.f) {
                                            ex_w[h] += double(__fmul_rn(ea[u].z, eb[u].x));
                                            ++ex_n[h];
                                        }
                                        if (!ok1 && ea[u].w > 0.f) {
                                            ex_w[h] += double(__fmul_rn(ea[u].w, eb[u].y));
                                            ++ex_n[h];
                                        }
                                    }
                                return;
                            }
                        }
#pragma unroll
                        for (int u = 0; u < UU; ++u) {
                            const f2 cc = pk(ea[u].z, ea[u].w);
#pragma unroll
                            for (int h = 0; h < F2; ++h) {
                                const f2 x = pk(v0[h][u], v1[h][u]);
                                acc[h][0].p = fma2(cc, x, acc[h][0].p);
                                if constexpr (MODE != kIntensity) {
                                    const f2 xp = is_unsigned_px<P>()
                                                      ? x
                                                      : pk(fmaxf(v0[h][u], 0.f), fmaxf(v1[h][u], 0.f));
                                    acc[h][1].p = fma2(mul2(cc, cc), xp, acc[h][1].p);
                                }
                                if constexpr (SPREAD) {
                                    const f2 n = pk(eb[u].x, eb[u].y), cr = pk(eb[u].z, eb[u].w);
                                    const f2 t = fma2(norg[h], ec[u], fma2(norg[h], n, x));
                                    acc[h][2].p = fma2(mul2(cr, t), t, acc[h][2].p);
                                    acc[h][kSpreadA].p = fma2(cc, t, acc[h][kSpreadA].p);
                                }
                            }
                        }
                    }
                };
                auto fold = [&]() {
#pragma unroll
                    for (int h = 0; h < F2; ++h)
#pragma unroll
                        for (int k = 0; k < NA - (FLOAT_SPREAD ? 2 : 0); ++k) acc[h][k].flush();
                };
                for (; p + U2 <= p1; p += U2) {
                    body(p, std::integral_constant<int, U2>{});
                    since += U2;
                    if (since >= kBtFoldPairs) {
                        since = 0;
                        fold();
                    }
                }
                for (; p < p1; ++p) {
                    body(p, std::integral_constant<int, 1>{});
                    if (++since >= kBtFoldPairs) {
                        since = 0;
                        fold();
                    }
                }
            }
            __syncwarp();
            if (lane == 0 && signal) mbar_arrive(empty + 8 * b);
            if (++b == NB) {
                b = 0;
                ++q;
            }
        }
        if (!ok) break;
        // This row's sums of each frame.
        double v[F2][NA];
#pragma unroll
        for (int h = 0; h < F2; ++h) {
#pragma unroll
            for (int k = 0; k < NA - (FLOAT_SPREAD ? 2 : 0); ++k) {
                acc[h][k].flush();
                v[h][k] = acc[h][k].value();
            }
            if constexpr (FLOAT_SPREAD) {
                v[h][NA - 2] = ex_w[h];
                v[h][NA - 1] = double(ex_n[h]);
            }
        }
        const int pieces = a.spans ? a.row_part[it.x + 1] - a.row_part[it.x] : 1;
        if (pieces > 1) {
            if (mine) {
                const int64_t slot = a.slot[item];
#pragma unroll
                for (int h = 0; h < F2; ++h) {
                    const int fl = lane + 32 * h;
                    if (fl >= nv) continue;
                    double *o = a.partial + (slot * NW + r) * NA * a.n_frames + f0 + fl;
#pragma unroll
                    for (int k = 0; k < NA; ++k) __stcg(o + int64_t(k) * a.n_frames, v[h][k]);
                }
            }
            __threadfence();
            if (!(ok = consumers_meet())) break;
            if (tid == 0) {
                int32_t *done = a.tile_done + it.x / NW * a.groups + group;
                const bool last = atomicAdd(done, 1) + 1 == pieces;
                if (last) *done = 0;
                s_last = last;
            }
            if (!(ok = consumers_meet())) break;
            if (!s_last) continue;
            __threadfence();
            if (mine) {
                const int32_t *ids = a.part_ids + a.row_part[row];
#pragma unroll
                for (int h = 0; h < F2; ++h) {
                    const int fl = min(lane + 32 * h, nv - 1);
#pragma unroll
                    for (int k = 0; k < NA; ++k) v[h][k] = 0.0;
                    for (int i = 0; i < pieces; ++i) {
                        const double *o = a.partial + int64_t(ids[i]) * NA * a.n_frames + f0 + fl;
#pragma unroll
                        for (int k = 0; k < NA; ++k)
                            v[h][k] = __dadd_rn(v[h][k], __ldcg(o + int64_t(k) * a.n_frames));
                    }
                }
            }
        }
        // A finished tile: normalise (normalize_bin, prepared.rs:985-996; the
        // spread's closing formulas, azimuthal.rs:96-104) as k_finalize does
        // from partial sums, or hand out the raw sums; then each output through
        // shared memory.
        double res[F2][4];
#pragma unroll
        for (int h = 0; h < F2; ++h) {
            double ri = 0.0, rs = 0.0, rd = 0.0, rc = 0.0;
            if (mine) {
                if (a.raw) {
                    // signal, variance, norm and weight sums (integrate1d_raw*,
                    // integrate.rs:682-797): the frame's own N and C with
                    // per-frame masks, else the row's
                    ri = v[h][0];
                    rs = NA > 1 ? v[h][NA > 1 ? 1 : 0] : 0.0;
                    rd = MODE == kRaw ? v[h][NA > 2 ? 2 : 0] : a.den[row];
                    rc = MODE == kRaw ? v[h][NA > 3 ? 3 : 0] : a.raw_cnt[row];
                } else if constexpr (SPREAD) {
                    int valid = a.valid_std[row];
                    double sw = a.den_std[row];
                    if (NA == 6) {
                        valid -= int(v[h][NA - 1] + 0.5);
                        sw -= v[h][NA - 2];
                    }
                    if (valid <= 0 || !(sw > 0.0)) {
                        rd = __longlong_as_double(0x7ff8000000000000ll);
                    } else {
                        const double a1 = v[h][kSpreadA];
                        ri = v[h][0] / sw;
                        rs = sqrt(v[h][1] > 0.0 ? v[h][1] : 0.0) / sw;
                        const double mean = a1 / sw;
                        const double m2 = v[h][2] - mean * a1;
                        const double var = m2 / sw;
                        // one valid contribution: its deviation from itself is exactly 0
                        rd = valid == 1 ? 0.0 : sqrt(var > 0.0 ? var : 0.0);
                    }
                } else {
                    const double n = MODE == kRaw ? v[h][NA > 2 ? 2 : 0] : a.den[row];
                    ri = n == 0.0 ? 0.0 : v[h][0] / n;
                    if (MODE != kIntensity) {
                        const double var = n == 0.0 ? 0.0 : v[h][NA > 1 ? 1 : 0] / (n * n);
                        rs = sqrt(var > 0.0 ? var : 0.0);
                    }
                }
            }
            res[h][0] = ri;
            res[h][1] = rs;
            res[h][2] = rd;
            res[h][3] = rc;
        }
        double *const outs[4] = {a.out_i, a.out_s, a.out_d, a.out_c};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (!outs[k]) continue;
#pragma unroll
            for (int h = 0; h < F2; ++h) s_out[(lane + 32 * h) * CFG::kOutStride + r] = res[h][k];
            ok = ok && consumers_meet();
            if (ok)
                for (int i = tid; i < nv * NW; i += NW * 32) {
                    const int f = i / NW, rr = i - f * NW;
                    if (rr < it.y)
                        outs[k][int64_t(f0 + f) * a.n_rows + it.x + rr] = s_out[f * CFG::kOutStride + rr];
                }
            ok = ok && consumers_meet();
        }
        if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
        }
    }
    if (!ok && lane == 0) {
        // A wait gave up: sums are incomplete. The host finds the flag (mapped
        // host memory) and reports the call as failed.
        *reinterpret_cast<volatile int *>(a.wait_err) = 1;
        __threadfence_system();
    }
}

// A pair's slot with bit 30 set where the pixel (as the frame stores it) is odd, which
// tells the half of a word of 2-byte pixels; the bit is lost in a slot's address (4 or
// 8 bytes a slot, 32 bits).
__device__ __forceinline__ float slot_of(int slot, int pixel) {
    return __int_as_float(slot | (pixel & 1) << 30);
}

// Bin-tile entry pairs from the plan-time layout: per pair {slot 0, slot 1,
// entry 0, entry 1} (entry -1: padding, slot = the zero column) to A {slot 0, slot 1,
// c0, c1} with the table's FP32 weights, AS the same with the spread's
// weights, B {n0, n1, c0/n0, c1/n1}.
__global__ void k_bt_fill(const int4 *__restrict__ desc, int64_t n_pairs,
                          const int2 *__restrict__ entry, const float4 *__restrict__ entry_std,
                          const float *__restrict__ entry_nlo, float4 *__restrict__ pair_a,
                          float4 *__restrict__ pair_as, float4 *__restrict__ pair_b,
                          float2 *__restrict__ pair_c) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n_pairs;
         i += int64_t(gridDim.x) * blockDim.x) {
        const int4 d = desc[i];
        float c[2] = {0.f, 0.f}, cs[2] = {0.f, 0.f}, n[2] = {1.f, 1.f}, cr[2] = {0.f, 0.f},
              nlo[2] = {0.f, 0.f};
        const int k[2] = {d.z, d.w};
        int px[2] = {0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (k[h] < 0) continue;
            px[h] = entry[k[h]].x;
            c[h] = __int_as_float(entry[k[h]].y);
            const float4 es = entry_std[k[h]];
            cs[h] = es.y;
            n[h] = es.z;
            cr[h] = es.w;
            nlo[h] = entry_nlo[k[h]];
        }
        const float s0 = slot_of(d.x, px[0]), s1 = slot_of(d.y, px[1]);
        pair_a[i] = make_float4(s0, s1, c[0], c[1]);
        pair_as[i] = make_float4(s0, s1, cs[0], cs[1]);
        pair_b[i] = make_float4(n[0], n[1], cr[0], cr[1]);
        pair_c[i] = make_float2(nlo[0], nlo[1]);
    }
}

// Pairs of the per-frame-mask bin tiles from the same layout: A {slot 0,
// slot 1, w0, w1} and B {w0*norm, w1*norm, 0, 0} with the raw entries'
// FP32 weights (k_pack_raw); padding entries are zero.
__global__ void k_bt_fill_raw(const int4 *__restrict__ desc, int64_t n_pairs,
                              const float4 *__restrict__ entry_raw, float4 *__restrict__ pair_a,
                              float4 *__restrict__ pair_b) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n_pairs;
         i += int64_t(gridDim.x) * blockDim.x) {
        const int4 d = desc[i];
        float w[2] = {0.f, 0.f}, wn[2] = {0.f, 0.f};
        const int k[2] = {d.z, d.w};
        int px[2] = {0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (k[h] < 0) continue;
            const float4 e = entry_raw[k[h]];
            px[h] = __float_as_int(e.x);
            w[h] = e.y;
            wn[h] = e.z;
        }
        pair_a[i] = make_float4(slot_of(d.x, px[0]), slot_of(d.y, px[1]), w[0], w[1]);
        pair_b[i] = make_float4(wn[0], wn[1], 0.f, 0.f);
    }
}

// InputOrder::FlipVertical: the pixel indices of bin-tile chunk records (D of
// them each), remapped to frames whose rows come in reverse order.
__global__ void k_flip_meta(int32_t *__restrict__ meta, int64_t n_rec, int words, int head,
                            int rows, int cols) {
    for (int64_t r = blockIdx.x; r < n_rec; r += gridDim.x) {
        int32_t *rec = meta + r * words;
        const int d = rec[0];
        for (int k = threadIdx.x; k < d; k += blockDim.x)
            rec[head + k] = flip_px(rec[head + k], rows, cols);
    }
}

// Per-frame masks as words: bit f of words[g][i] is set where frame 64 g + f masks
// pixel i. Reading the bytes once, in rows, replaces a byte load per (pixel,
// frame) of every tile that touches the pixel; a chunk then stages one word per
// pixel, and a lane reads its frames' bits of a slot in one shared-memory load.
__global__ void __launch_bounds__(256)
    k_mask_words(const uint8_t *__restrict__ masks, int64_t stride, int64_t n_px, int n_frames,
                 uint64_t *__restrict__ words) {
    const int f0 = int(blockIdx.y) * 64, nf = min(64, n_frames - f0);
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n_px;
         i += int64_t(gridDim.x) * blockDim.x) {
        const uint8_t *m = masks + int64_t(f0) * stride + i;
        uint64_t w = 0;
#pragma unroll 16
        for (int f = 0; f < nf; ++f) w |= uint64_t(m[int64_t(f) * stride] != 0) << f;
        words[int64_t(blockIdx.y) * n_px + i] = w;
    }
}

}  // namespace

// A tile on the host: runs of chunks, pixels and pairs are relative to it.
struct BinTile {
    std::vector<int4> chunks;      // {px offset, D, pair offset, pairs}
    std::vector<int32_t> cpair;    // per chunk kRows + 1
    std::vector<int32_t> px;
    std::vector<int4> pairs;       // {slot0, slot1, entry0, entry1}
    int64_t entries = 0;
};
// A piece of a tile: its chunks and, where the tile is cut, per fold cadence and
// row the {chunk, pair} to start and to end at, chunks relative to c0.
struct BinPiece {
    int64_t tile;
    int c0, n;
    std::vector<int4> spans[2];
};
// The tiles of a table and their pieces (items) in claim order.
struct BinLayout {
    std::vector<BinTile> tiles;
    std::vector<std::vector<BinPiece>> cut;
    std::vector<int64_t> first_chunk;         // per tile, then the number of chunks
    std::vector<int4> items;                  // {first row, rows, first chunk, chunks}
    bool split = false;                       // with the lists below
    std::vector<int4> spans[2];               // per item and row
    std::vector<int32_t> row_part, part_ids;  // every row's pieces (item * kRows + row), in order
    // Per item its slot among the pieces of cut tiles (-1: an uncut tile, which
    // leaves no partial sums), and the number of slots.
    std::vector<int32_t> slot;
    int32_t n_slots = 0;
};

// fn(0) .. fn(count - 1) over host threads, the caller's among them. The first
// exception is thrown on the caller's thread once all have stopped; where no more
// threads can be made, those that there are do the work.
template <class Fn>
void parallel(int64_t count, Fn &&fn) {
    const int nt = int(std::min<int64_t>(
        count, std::max(1u, std::min(16u, std::thread::hardware_concurrency()))));
    std::atomic<int64_t> next{0};
    std::mutex mu;
    std::exception_ptr error;
    auto run = [&]() {
        try {
            for (int64_t i; (i = next.fetch_add(1)) < count;) fn(i);
        } catch (...) {
            next = count;
            std::lock_guard<std::mutex> lock(mu);
            if (!error) error = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(size_t(std::max(nt, 1)));
    try {
        while (int(pool.size()) + 1 < nt) pool.emplace_back(run);
    } catch (const std::system_error &) {
    }
    run();
    for (auto &th : pool) th.join();
    if (error) std::rethrow_exception(error);
}

// Bin tiles (k_gather_bins) at plan time, on the host: for every run of
// CFG::kRows rows, the rows' entries merged in pixel order and cut into chunks of
// at most kBtDCap distinct pixels and kBtPCap pairs (a new pixel that would
// exceed either opens the next chunk, so a chunk is a pixel-index interval
// and each row's entries in it are a contiguous run of its CSR row). Tiles
// are cut into pieces (see the file comment). A chunk's first pair is even, so
// that its pairs C are copied from a 16-byte boundary.
template <class CFG>
void lay_out_bin_tiles(const int64_t *rp, const int32_t *col, int64_t nb, BinLayout &out) {
    constexpr int kBtDCap = CFG::kDCap, kBtPCap = CFG::kPCap, kBtRows = CFG::kRows;
    const int64_t n_items = (nb + kBtRows - 1) / kBtRows;
    std::vector<BinTile> &tiles = out.tiles;
    tiles.resize(static_cast<size_t>(n_items));
    auto build = [&](int64_t ti) {
        BinTile &T = tiles[size_t(ti)];
        const int64_t r0 = ti * kBtRows, r1 = std::min<int64_t>(nb, r0 + kBtRows);
        const int nr = int(r1 - r0);
        // Entries merged in pixel order, rows ascending within a pixel: keys
        // pixel << 32 | row << 27 | position in row; each row is sorted
        // already, so four rounds of pairwise merges order the tile.
        const int64_t n_e = rp[r1] - rp[r0];
        for (int64_t r = r0; r < r1; ++r)
            if (rp[r + 1] - rp[r] >= (int64_t(1) << 27))
                fail(DG_UNSUPPORTED, "a bin too large for bin tiles");
        std::vector<uint64_t> ka(static_cast<size_t>(n_e)), kb(static_cast<size_t>(n_e));
        std::vector<int64_t> bounds(static_cast<size_t>(kBtRows) + 1, 0);
        for (int j = 0; j < nr; ++j) {
            const int64_t b = rp[r0 + j], e = rp[r0 + j + 1];
            uint64_t *o = ka.data() + (b - rp[r0]);
            for (int64_t k = b; k < e; ++k)
                o[k - b] = (uint64_t(uint32_t(col[k])) << 32) | (uint64_t(j) << 27) |
                           uint64_t(k - b);
            bounds[size_t(j) + 1] = e - rp[r0];
        }
        for (int j = nr; j < kBtRows; ++j) bounds[size_t(j) + 1] = n_e;
        for (int width = 1; width < kBtRows; width *= 2) {
            for (int j = 0; j < kBtRows; j += 2 * width) {
                const int64_t a0 = bounds[size_t(j)], a1 = bounds[size_t(std::min(j + width, kBtRows))],
                              a2 = bounds[size_t(std::min(j + 2 * width, kBtRows))];
                std::merge(ka.begin() + a0, ka.begin() + a1, ka.begin() + a1, ka.begin() + a2,
                           kb.begin() + a0);
            }
            ka.swap(kb);
        }
        struct Ent {
            int32_t px, row, k;
        };
        std::vector<Ent> m(static_cast<size_t>(n_e));
        for (int64_t i = 0; i < n_e; ++i) {
            const uint64_t key = ka[size_t(i)];
            const int j = int((key >> 27) & 31u);
            m[size_t(i)] = {int32_t(key >> 32), j, int32_t(rp[r0 + j] + int64_t(key & ((1u << 27) - 1)))};
        }
        T.entries = n_e;
        T.pairs.reserve(size_t(n_e / 2 + 64));
        T.px.reserve(size_t(n_e / 2 + 64));
        std::vector<std::vector<std::pair<int32_t, int32_t>>> run(static_cast<size_t>(nr));  // (slot, entry)
        std::vector<int32_t> chunk_px;
        auto close = [&]() {
            if (chunk_px.empty()) return;
            int4 ch = make_int4(int(T.px.size()), int(chunk_px.size()), int(T.pairs.size()), 0);
            T.px.insert(T.px.end(), chunk_px.begin(), chunk_px.end());
            int po = 0;
            for (int j = 0; j < kBtRows; ++j) {
                T.cpair.push_back(po);
                if (j >= nr) continue;
                const auto &rv = run[size_t(j)];
                for (size_t e = 0; e < rv.size(); e += 2) {
                    const bool two = e + 1 < rv.size();
                    T.pairs.push_back(make_int4(rv[e].first, two ? rv[e + 1].first : kBtDCap,
                                                rv[e].second, two ? rv[e + 1].second : -1));
                    ++po;
                }
            }
            T.cpair.push_back(po);
            ch.w = po;
            if (po & 1)  // the next chunk's first pair is even
                T.pairs.push_back(make_int4(kBtDCap, kBtDCap, -1, -1));
            T.chunks.push_back(ch);
            chunk_px.clear();
            for (auto &rv : run) rv.clear();
        };
        int pairs = 0;
        for (size_t i = 0; i < m.size();) {
            size_t e = i;
            while (e < m.size() && m[e].px == m[i].px) ++e;
            // pairs after adding this pixel's entries
            int add = 0;
            for (size_t q = i; q < e; ++q) add += (run[size_t(m[q].row)].size() % 2 == 0) ? 1 : 0;
            if (!chunk_px.empty() &&
                (int(chunk_px.size()) + 1 > kBtDCap || pairs + add > kBtPCap)) {
                close();
                pairs = 0;
                add = int(e - i);
            }
            const int slot = int(chunk_px.size());
            chunk_px.push_back(m[i].px);
            for (size_t q = i; q < e; ++q) run[size_t(m[q].row)].push_back({slot, m[q].k});
            pairs += add;
            i = e;
        }
        close();
        if (T.chunks.empty()) {
            // rows without entries: a chunk of one pixel and no row's pairs, since
            // every item passes through the ring (and writes its rows)
            T.px.push_back(0);
            T.chunks.push_back(make_int4(0, 1, 0, 2));
            T.cpair.assign(size_t(kBtRows) + 1, 0);
            T.pairs.assign(2, make_int4(kBtDCap, kBtDCap, -1, -1));
        }
    };
    parallel(n_items, build);
    // Pieces: a tile of many chunks is cut at chunk boundaries, each row at the
    // first fold of its FP32 sums at or after the cut (spans). Both fold
    // cadences (steps of kU2 pairs, and of two for float pixels with the
    // spread) get their own spans; a piece's chunks cover both.
    int64_t all_chunks = 0;
    for (const BinTile &T : tiles) all_chunks += int64_t(T.chunks.size());
    const int piece = int(std::clamp<int64_t>(all_chunks / 350, kBtPieceMin, kBtPieceMax));
    // Neighbouring tiles whose pieces are claimed one after the other: they walk the
    // same rows at the same time and share the sectors at their common edges. Four
    // tiles where a table has more chunks than the shortest pieces take (22,750), two
    // where an even finish of few pieces counts more. us with two and with four:
    // Eiger-4M (27,619 chunks), 256 frames with the spread 1757 and 1731, with errors
    // 1526 and 1458, 64 frames with the spread 474 and 466; 2600 x 2500 pixels (40,128),
    // 128 frames with the spread 1325 and 1303; Eiger-9M (62,558), 128 frames with
    // errors 1697 and 1686, 192 with the spread 2906 and 2926; Pilatus 1M (6,639), 256
    // frames 405 and 415, 50 frames 117 and 119.
    const int64_t near = piece > kBtPieceMin ? 4 : 2;
    std::vector<std::vector<BinPiece>> &cut = out.cut;
    cut.resize(static_cast<size_t>(n_items));
    std::atomic<bool> any_cut{false};
    auto split = [&](int64_t ti) {
        const BinTile &T = tiles[size_t(ti)];
        const int nch = int(T.chunks.size());
        std::vector<int> at;  // first chunk of every piece
        int most = 0;  // neighbouring tiles are cut alike
        for (int64_t j = ti / near * near; j < std::min(n_items, (ti / near + 1) * near); ++j)
            most = std::max(most, int(tiles[size_t(j)].chunks.size()));
        const int parts = std::max(1, std::min(nch, (most + piece - 1) / piece));
        for (int q = 0; q < parts; ++q) at.push_back(int(int64_t(nch) * q / parts));
        const int k = int(at.size());
        at.push_back(nch);
        std::vector<BinPiece> &out_p = cut[size_t(ti)];
        out_p.resize(size_t(k));
        for (int i = 0; i < k; ++i) {
            out_p[size_t(i)].tile = ti;
            out_p[size_t(i)].c0 = at[size_t(i)];
            out_p[size_t(i)].n = at[size_t(i) + 1] - at[size_t(i)];
        }
        if (k == 1) return;
        const int nr = int(std::min<int64_t>(nb, (ti + 1) * kBtRows) - ti * kBtRows);
        // start[cadence][piece][row]: {chunk, pair of the row's run in it}
        std::vector<std::pair<int, int>> start[2];
        for (int s2 = 0; s2 < 2; ++s2) {
            const int step = s2 ? std::min(2, CFG::kU2) : CFG::kU2;
            start[s2].assign(size_t(k + 1) * kBtRows, {nch, 0});
            for (int r = 0; r < nr; ++r) {
                int since = 0, next = 1;  // the next cut to place
                start[s2][size_t(r)] = {0, 0};
                for (int c = 0; c < nch && next < k; ++c) {
                    const int32_t *cp = T.cpair.data() + size_t(c) * (kBtRows + 1);
                    const int n = cp[r + 1] - cp[r];
                    auto fold_at = [&](int p) {  // a fold before pair p of chunk c
                        const std::pair<int, int> at = p == n ? std::make_pair(c + 1, 0) : std::make_pair(c, p);
                        while (next < k && at.first >= out_p[size_t(next)].c0)
                            start[s2][size_t(next++) * kBtRows + size_t(r)] = at;
                    };
                    if (since == 0) fold_at(0);
                    for (int p = 0; p < n;) {
                        const int d = p + step <= n ? step : 1;
                        p += d;
                        since += d;
                        if (since >= kBtFoldPairs) {
                            since = 0;
                            fold_at(p);
                        }
                    }
                }
            }
        }
        for (int i = 0; i < k; ++i) {
            int lo = nch, hi = 0;
            for (int s2 = 0; s2 < 2; ++s2)
                for (int r = 0; r < nr; ++r) {
                    const auto a = start[s2][size_t(i) * kBtRows + size_t(r)];
                    const auto e = start[s2][size_t(i + 1) * kBtRows + size_t(r)];
                    if (a >= e) continue;
                    lo = std::min(lo, a.first);
                    hi = std::max(hi, e.second > 0 ? e.first + 1 : e.first);
                }
            BinPiece &p = out_p[size_t(i)];
            p.c0 = std::min(lo, hi);
            p.n = hi - p.c0;
            for (int s2 = 0; s2 < 2; ++s2) {
                p.spans[s2].assign(size_t(kBtRows), make_int4(0, 0, 0, 0));
                for (int r = 0; r < nr; ++r) {
                    const auto a = start[s2][size_t(i) * kBtRows + size_t(r)];
                    const auto e = start[s2][size_t(i + 1) * kBtRows + size_t(r)];
                    if (a < e)
                        p.spans[s2][size_t(r)] = make_int4(a.first - p.c0, a.second, e.first - p.c0, e.second);
                }
            }
        }
        // A piece in which no row folds holds nothing (a small tile cut like its
        // large neighbour): its neighbours' spans meet, and no warp would see it.
        out_p.erase(std::remove_if(out_p.begin(), out_p.end(), [](const BinPiece &p) { return p.n == 0; }),
                    out_p.end());
        if (out_p.size() > 1) {
            any_cut = true;
            return;
        }
        out_p.assign(1, {ti, 0, nch, {}});
    };
    parallel(n_items, split);
    std::vector<const BinPiece *> order;
    for (auto &v : cut)
        for (const BinPiece &p : v) order.push_back(&p);
    if (any_cut)  // largest first; whole tiles in tile order
    {
        // largest first, the pieces of neighbouring tiles side by side
        std::map<std::pair<int64_t, int>, int> size;
        auto key = [&](const BinPiece *p) {
            return std::make_pair(p->tile / near, int(p - cut[size_t(p->tile)].data()));
        };
        for (const BinPiece *p : order) {
            int &n = size[key(p)];
            n = std::max(n, p->n);
        }
        std::stable_sort(order.begin(), order.end(), [&](const BinPiece *a, const BinPiece *b) {
            const auto ka = key(a), kb = key(b);
            const int na = size[ka], nb2 = size[kb];
            if (na != nb2) return na > nb2;
            if (ka != kb) return ka < kb;
            return a->tile < b->tile;
        });
    }
    out.split = any_cut;
    out.first_chunk.assign(size_t(n_items) + 1, 0);
    for (int64_t i = 0; i < n_items; ++i)
        out.first_chunk[size_t(i) + 1] = out.first_chunk[size_t(i)] + int64_t(tiles[size_t(i)].chunks.size());
    if (out.first_chunk.back() > INT32_MAX) fail(DG_UNSUPPORTED, "table too large for bin tiles");
    out.items.resize(order.size());
    for (size_t i = 0; i < order.size(); ++i) {
        const BinPiece &p = *order[i];
        if (p.n < 1) fail(DG_DEVICE, "a bin-tile item without chunks");
        const int64_t r0 = p.tile * kBtRows;
        out.items[i] = make_int4(int(r0), int(std::min<int64_t>(nb, r0 + kBtRows) - r0),
                                 int(out.first_chunk[size_t(p.tile)]) + p.c0, p.n);
    }
    if (!out.split) return;
    // Spans per item and row, and the pieces of every row in tile order
    // (partial sums are kept per piece of a cut tile and row).
    std::vector<std::vector<int32_t>> pieces(static_cast<size_t>(n_items));
    for (int64_t ti = 0; ti < n_items; ++ti) pieces[size_t(ti)].resize(cut[size_t(ti)].size());
    for (size_t i = 0; i < order.size(); ++i) {
        const BinPiece &p = *order[i];
        out.slot.push_back(cut[size_t(p.tile)].size() > 1 ? out.n_slots++ : -1);
        pieces[size_t(p.tile)][size_t(order[i] - cut[size_t(p.tile)].data())] = int32_t(i);
        for (int s2 = 0; s2 < 2; ++s2) {
            if (p.spans[s2].empty())  // an uncut tile
                out.spans[s2].insert(out.spans[s2].end(), size_t(kBtRows), make_int4(0, 0, INT_MAX, 0));
            else
                out.spans[s2].insert(out.spans[s2].end(), p.spans[s2].begin(), p.spans[s2].end());
        }
    }
    out.row_part.assign(size_t(nb) + 1, 0);
    for (int64_t r = 0; r < nb; ++r) {
        for (int32_t i : pieces[size_t(r / kBtRows)])
            out.part_ids.push_back(i * kBtRows + int32_t(r % kBtRows));
        out.row_part[size_t(r) + 1] = int32_t(out.part_ids.size());
    }
}

// The bin tiles of a plan's table in device memory. Each row keeps {origin entry,
// first valid entry, row end} for the spread's origin (row_origin), read before
// the first chunk.
template <class CFG>
void build_bin_tiles(GatherTable &gt, BinTiles &out, const DeviceCsr &table, cudaStream_t s) {
    constexpr int kBtRows = CFG::kRows;
    constexpr int kBtMetaHead = CFG::kMetaHead, kBtMetaWords = CFG::kMetaWords;
    const int64_t nb = table.n_rows;
    out.n_items = 0;
    if (nb == 0 || table.nnz == 0) return;
    out.wait_err.alloc();
    std::vector<int64_t> rp(static_cast<size_t>(nb) + 1);
    DG_CUDA(cudaMemcpyAsync(rp.data(), table.row_ptr.ptr, rp.size() * 8, cudaMemcpyDeviceToHost, s));
    std::vector<int32_t> col(static_cast<size_t>(table.nnz)), fv(static_cast<size_t>(nb)),
        oe(static_cast<size_t>(nb));
    DG_CUDA(cudaMemcpyAsync(col.data(), table.col.ptr, col.size() * 4, cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaMemcpyAsync(fv.data(), gt.first_valid.ptr, fv.size() * 4, cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaMemcpyAsync(oe.data(), gt.origin.ptr, oe.size() * 4, cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaStreamSynchronize(s));
    BinLayout layout;
    lay_out_bin_tiles<CFG>(rp.data(), col.data(), nb, layout);
    std::vector<BinTile> &tiles = layout.tiles;
    out.split = layout.split;
    // Output offsets of every tile, then the tiles copied in parallel.
    const int64_t n_slots = int64_t(tiles.size());
    const std::vector<int64_t> &o_ch = layout.first_chunk;
    std::vector<int64_t> o_px(size_t(n_slots) + 1, 0), o_pr(size_t(n_slots) + 1, 0);
    for (int64_t i = 0; i < n_slots; ++i) {
        const BinTile &T = tiles[size_t(i)];
        o_px[size_t(i) + 1] = o_px[size_t(i)] + int64_t(T.px.size());
        o_pr[size_t(i) + 1] = o_pr[size_t(i)] + int64_t(T.pairs.size());
    }
    if (o_pr[size_t(n_slots)] > INT32_MAX || o_px[size_t(n_slots)] > INT32_MAX)
        fail(DG_UNSUPPORTED, "table too large for bin tiles");
    // default-initialised (not zeroed): every element is written below
    const size_t n_chunks = size_t(o_ch[size_t(n_slots)]), n_pairs = size_t(o_pr[size_t(n_slots)]);
    const std::vector<int4> &items = layout.items;
    std::vector<int4> org(static_cast<size_t>(nb));
    // per row {origin entry, first valid entry, row end, 0} (row_origin)
    for (int64_t r = 0; r < nb; ++r)
        org[size_t(r)] = make_int4(oe[size_t(r)], fv[size_t(r)], int(rp[size_t(r) + 1]), 0);
    std::unique_ptr<int32_t[]> meta(new int32_t[std::max<size_t>(n_chunks * kBtMetaWords, 1)]);
    std::unique_ptr<int4[]> pairs(new int4[std::max<size_t>(n_pairs, 1)]);
    auto flatten = [&](int64_t i) {
        BinTile &T = tiles[size_t(i)];
        const int64_t c0 = o_ch[size_t(i)], pr0 = o_pr[size_t(i)];
        for (size_t c = 0; c < T.chunks.size(); ++c) {
            const int4 ch = T.chunks[c];
            int32_t *rec = meta.get() + (size_t(c0) + c) * kBtMetaWords;
            rec[0] = ch.y;
            rec[1] = ch.w;
            rec[2] = int32_t(ch.z + pr0);
            rec[3] = 0;
            for (int j = 0; j < kBtMetaHead - 4; ++j)
                rec[4 + j] = j <= kBtRows ? T.cpair[c * (kBtRows + 1) + size_t(j)] : 0;
            std::copy(T.px.begin() + ch.x, T.px.begin() + ch.x + ch.y, rec + kBtMetaHead);
            std::fill(rec + kBtMetaHead + ch.y, rec + kBtMetaWords, 0);
        }
        std::copy(T.pairs.begin(), T.pairs.end(), pairs.get() + pr0);
        T = BinTile();
    };
    parallel(n_slots, flatten);
    out.n_items = int32_t(items.size());
    out.item.alloc(items.size());
    for (auto &n : out.counts) {
        n.claim.alloc(2);
        DG_CUDA(cudaMemsetAsync(n.claim.ptr, 0, n.claim.bytes(), s));
    }
    if (out.split) {
        const std::vector<int4>(&spans)[2] = layout.spans;
        const std::vector<int32_t> &row_part = layout.row_part;
        // the pieces' partial sums: slot * rows + row of the tile
        std::vector<int32_t> ids(layout.part_ids);
        for (int32_t &id : ids)
            id = std::max(0, layout.slot[size_t(id / kBtRows)]) * kBtRows + id % kBtRows;
        out.partial_rows = int64_t(layout.n_slots) * kBtRows;
        out.slot.alloc(layout.slot.size());
        DG_CUDA(cudaMemcpyAsync(out.slot.ptr, layout.slot.data(), layout.slot.size() * 4,
                                cudaMemcpyHostToDevice, s));
        for (int s2 = 0; s2 < 2; ++s2) {
            out.span[s2].alloc(spans[s2].size());
            DG_CUDA(cudaMemcpyAsync(out.span[s2].ptr, spans[s2].data(), spans[s2].size() * sizeof(int4),
                                    cudaMemcpyHostToDevice, s));
        }
        for (auto &n : out.counts) {
            n.tile_done.alloc(tiles.size() * size_t(256 / CFG::kFrames));
            DG_CUDA(cudaMemsetAsync(n.tile_done.ptr, 0, n.tile_done.bytes(), s));
        }
        out.row_part.alloc(row_part.size());
        out.part_ids.alloc(ids.size());
        DG_CUDA(cudaMemcpyAsync(out.row_part.ptr, row_part.data(), row_part.size() * 4,
                                cudaMemcpyHostToDevice, s));
        DG_CUDA(cudaMemcpyAsync(out.part_ids.ptr, ids.data(), ids.size() * 4, cudaMemcpyHostToDevice, s));
        DG_CUDA(cudaStreamSynchronize(s));  // ids is local
    }
    out.meta.alloc(std::max<size_t>(n_chunks * kBtMetaWords, 1));
    out.org.alloc(org.size());
    out.pair_a.alloc(std::max<size_t>(n_pairs, 1));
    out.pair_as.alloc(std::max<size_t>(n_pairs, 1));
    out.pair_b.alloc(std::max<size_t>(n_pairs, 1));
    out.pair_c.alloc(std::max<size_t>(n_pairs, 1));
    DeviceArray<int4> &desc = out.desc;  // kept for the per-frame-mask pairs
    desc.alloc(std::max<size_t>(n_pairs, 1));
    out.pair_ra.release();
    out.pair_rb.release();
    out.raw_built = false;
    DG_CUDA(cudaMemcpyAsync(out.item.ptr, items.data(), items.size() * sizeof(int4),
                            cudaMemcpyHostToDevice, s));
    if (n_chunks)
        DG_CUDA(cudaMemcpyAsync(out.meta.ptr, meta.get(), n_chunks * kBtMetaWords * 4,
                                cudaMemcpyHostToDevice, s));
    DG_CUDA(cudaMemcpyAsync(out.org.ptr, org.data(), org.size() * sizeof(int4),
                            cudaMemcpyHostToDevice, s));
    if (n_pairs) {
        DG_CUDA(cudaMemcpyAsync(desc.ptr, pairs.get(), n_pairs * sizeof(int4),
                                cudaMemcpyHostToDevice, s));
        k_bt_fill<<<148 * 8, 256, 0, s>>>(desc.ptr, int64_t(n_pairs), gt.entry.ptr,
                                         gt.entry_std.ptr, gt.entry_nlo.ptr, out.pair_a.ptr,
                                         out.pair_as.ptr, out.pair_b.ptr, out.pair_c.ptr);
        DG_CUDA(cudaGetLastError());
    }
    DG_CUDA(cudaStreamSynchronize(s));
    // Only mapping 8's tiles carry per-frame masks; the others drop the
    // descriptor once their pairs are filled.
    if (!std::is_same<CFG, Bt8>::value) desc.release();
}

void bin_items(int variant, int64_t n_rows, const int64_t *row_ptr, const int32_t *col,
               BinItems &out) {
    BinLayout layout;
    if (variant == 7) lay_out_bin_tiles<Bt7>(row_ptr, col, n_rows, layout);
    else if (variant == 8) lay_out_bin_tiles<Bt8>(row_ptr, col, n_rows, layout);
    else fail(DG_INVALID_INPUT, "bin tiles are lane mappings 7 and 8");
    out.rows = variant == 7 ? Bt7::kRows : Bt8::kRows;
    out.first_chunk = std::move(layout.first_chunk);
    out.items = std::move(layout.items);
    for (int s2 = 0; s2 < 2; ++s2) out.spans[s2] = std::move(layout.spans[s2]);
    out.row_part = std::move(layout.row_part);
    out.part_ids = std::move(layout.part_ids);
    out.partial_rows = int64_t(layout.n_slots) * out.rows;
}

bool bin_tile_wait_failed(const GatherTable &t) {
    bool failed = false;
    for (const BinTiles &bt : t.bt)
        if (bt.wait_err.host && *static_cast<volatile int *>(bt.wait_err.host)) {
            *bt.wait_err.host = 0;
            bt.counts[0].unfinished = bt.counts[1].unfinished = true;
            failed = true;
        }
    return failed;
}

void check_bin_tile_waits(const GatherTable &t) {
    if (bin_tile_wait_failed(t))
        fail(DG_TIMEOUT, "bin-tile gather: a chunk-pipeline wait gave up after 1 s; the "
                          "results of a launch on this plan since the last check are invalid");
}

void ensure_bin_tiles(GatherTable &t, const DeviceCsr &table, int variant, cudaStream_t s) {
    if (variant != 7 && variant != 8) return;
    BinTiles &bt = t.bt[variant - 7];
    if (bt.built) return;
    AllocScope alloc(s);  // s is synchronised before this returns
    int words = 0, head = 0;
    if (variant == 7) {
        build_bin_tiles<Bt7>(t, bt, table, s);
        words = Bt7::kMetaWords;
        head = Bt7::kMetaHead;
    } else {
        build_bin_tiles<Bt8>(t, bt, table, s);
        words = Bt8::kMetaWords;
        head = Bt8::kMetaHead;
    }
    if (t.flip_rows && bt.n_items > 0) {
        k_flip_meta<<<148 * 4, 256, 0, s>>>(bt.meta.ptr, int64_t(bt.meta.count) / words, words,
                                            head, t.flip_rows, t.flip_cols);
        DG_CUDA(cudaGetLastError());
        DG_CUDA(cudaStreamSynchronize(s));
    }
    bt.built = true;
}

bool gather_variant_needs_tiles(int variant) { return variant == 7 || variant == 8; }

bool bin_tiles_fill_gpu(const GatherTable &t, int variant, int64_t n_frames) {
    if (!gather_variant_needs_tiles(variant)) return false;
    const int64_t rows = variant == 7 ? Bt7::kRows : Bt8::kRows;
    const int64_t per = variant == 7 ? Bt7::kFrames : Bt8::kFrames;
    const int64_t nf = std::min<int64_t>(n_frames, 256);
    const int64_t ctas = (int64_t(t.n_rows) + rows - 1) / rows * ((nf + per - 1) / per);
    if (variant == 8 && 2 * nf >= per && bin_tiles_fill_gpu(t, 7, n_frames)) return true;
    return 2 * nf >= per && ctas >= 2 * 148;
}

namespace {

template <int MODE, typename P, class CFG>
void launch(const GatherTable &t, const BinTiles &bt, const BinCall &c, cudaStream_t s) {
    constexpr size_t smem = CFG::template smem_bytes<MODE, P>();
    auto kern = k_gather_bins<MODE, P, CFG>;
    DG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    BinArgs a{};
    a.items = bt.item.ptr;
    a.spans = bt.split ? bt.span[bt_step<MODE, P, CFG>() == CFG::kU2 ? 0 : 1].ptr : nullptr;
    a.meta = bt.meta.ptr;
    a.pair_a = MODE == kSpread ? bt.pair_as.ptr : MODE == kRaw ? bt.pair_ra.ptr : bt.pair_a.ptr;
    a.pair_b = MODE == kRaw ? bt.pair_rb.ptr : bt.pair_b.ptr;
    a.pair_c = bt.pair_c.ptr;
    a.org = bt.org.ptr;
    a.entry_std = t.entry_std.ptr;
    a.den = t.den.ptr;
    a.den_std = t.den_std.ptr;
    a.valid_std = t.valid_std.ptr;
    a.frames = c.frames;
    a.n_pixels = c.n_pixels;
    a.n_frames = c.n_frames;
    a.n_rows = t.n_rows;
    a.n_items = bt.n_items;
    a.groups = (c.n_frames + CFG::kFrames - 1) / CFG::kFrames;
    // Counts: a replay of a captured launch is ordered by its caller alone, and is
    // preceded by its own reset, since no call of the library comes before it.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    DG_CUDA(cudaStreamIsCapturing(s, &capture));
    const bool captured = capture != cudaStreamCaptureStatusNone;
    const BinTiles::Counts &counts = bt.counts[c.fixed || captured ? 1 : 0];
    a.counter = counts.claim.ptr;
    a.out_i = c.out_i;
    a.out_s = c.out_s;
    a.out_d = c.out_d;
    a.out_c = c.out_c;
    a.partial = c.partial;
    a.slot = bt.slot.ptr;
    a.row_part = bt.row_part.ptr;
    a.part_ids = bt.part_ids.ptr;
    a.tile_done = counts.tile_done.ptr;
    a.raw_cnt = t.cnt.ptr;
    a.raw = c.raw;
    a.mask_words = t.mask_words.ptr;
    a.wait_err = bt.wait_err.dev;
    a.withhold = t.withhold_test;
    if (int64_t(a.n_items) * a.groups > INT32_MAX)
        fail(DG_UNSUPPORTED, "too many bin tiles for one launch");
    check_bin_tile_waits(t);
    if (counts.unfinished || captured) {  // a launch that gave up left tiles partly done
        DG_CUDA(cudaMemsetAsync(counts.claim.ptr, 0, counts.claim.bytes(), s));
        if (bt.split)
            DG_CUDA(cudaMemsetAsync(counts.tile_done.ptr, 0, counts.tile_done.bytes(), s));
        if (!captured) counts.unfinished = false;
    }
    const int grid = std::min(a.n_items * a.groups, sm_count());
    kern<<<unsigned(grid), CFG::template threads<MODE, P>(), smem, s>>>(a);
    DG_CUDA(cudaGetLastError());
}

template <typename P, class CFG>
void launch_mode(const GatherTable &t, const BinTiles &bt, const BinCall &c, cudaStream_t s) {
    if (c.mode == kSpread) launch<kSpread, P, CFG>(t, bt, c, s);
    else if (c.mode == kErrors) launch<kErrors, P, CFG>(t, bt, c, s);
    else launch<kIntensity, P, CFG>(t, bt, c, s);
}

template <typename P>
void launch_typed(const GatherTable &t, int variant, const BinCall &c, cudaStream_t s) {
    const BinTiles &bt = t.bt[variant - 7];
    if (c.masks) launch<kRaw, P, Bt8>(t, bt, c, s);
    else if (variant == 7) launch_mode<P, Bt7>(t, bt, c, s);
    else launch_mode<P, Bt8>(t, bt, c, s);
}

}  // namespace

int64_t bin_tile_partials(const GatherTable &t, int variant) {
    return t.bt[variant - 7].partial_rows;
}

void launch_bin_tiles(GatherTable &t, int variant, const BinCall &c, cudaStream_t s) {
    BinTiles &bt = t.bt[variant - 7];
    if (c.masks && !bt.raw_built) {
        bt.pair_ra.alloc(bt.desc.count);
        bt.pair_rb.alloc(bt.desc.count);
        k_bt_fill_raw<<<148 * 8, 256, 0, s>>>(bt.desc.ptr, int64_t(bt.desc.count), t.entry_raw.ptr,
                                             bt.pair_ra.ptr, bt.pair_rb.ptr);
        DG_CUDA(cudaGetLastError());
        bt.raw_built = true;
    }
    if (c.masks) {
        const unsigned groups = unsigned((c.n_frames + 63) / 64);
        if (t.mask_words.count < size_t(groups) * size_t(c.n_pixels))
            t.mask_words.alloc(size_t(groups) * size_t(c.n_pixels));
        ++t.launches;
        const unsigned gx = unsigned(std::min<int64_t>((c.n_pixels + 255) / 256, 148 * 16));
        k_mask_words<<<dim3(gx, groups), 256, 0, s>>>(c.masks, c.mask_stride, c.n_pixels, c.n_frames,
                                                     t.mask_words.ptr);
        DG_CUDA(cudaGetLastError());
    }
    switch (c.dtype) {
    case DG_U16: launch_typed<uint16_t>(t, variant, c, s); break;
    case DG_U32: launch_typed<uint32_t>(t, variant, c, s); break;
    case DG_I32: launch_typed<int32_t>(t, variant, c, s); break;
    case DG_F32: launch_typed<float>(t, variant, c, s); break;
    case DG_F64: launch_typed<double>(t, variant, c, s); break;
    default: fail(DG_INVALID_INPUT, "unknown pixel dtype");
    }
}

}  // namespace dg
