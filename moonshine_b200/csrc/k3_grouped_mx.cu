// Ragged grouped GEMM on the block-scaled tensor-core path
// (tcgen05.mma kind::mxf8f6f4, scale_vec::1X) for layer-major prefill.
//
//   out[r, m] = sum_k W[g(r)][m, k] * x[r, k]      r: token rows grouped by expert
//
// Weights stay in their checkpoint form: packed E2M1 nibbles are expanded into
// the MMA's 8-bit containers by the TMA unit (tensor-map type 16U4_ALIGN16B) and
// the E8M0 scales go to tensor memory with tcgen05.st - no thread converts a
// weight.  Token rows are split once into two E4M3 terms with a shared E8M0
// scale per 32 columns, x = 2^s (hi + lo); bf16 carries 8 significant bits and
// each term 4, so every element within 2^10 of its block maximum is exact and
// the rest is held to 2^-17 of the block maximum.  Each K block of 32 issues two
// MMAs (hi and lo against the same weights and scales).
//
// Work item = two 128-row weight tiles x up to 160 token rows of one group over
// the whole K extent (gate+up with fused activation, or 256 rows of the down
// projection).  One CTA per SM, persistent; the item list is derived in-kernel from the
// group offsets and handed out by a global counter: the weight producer takes the next
// item with one atomicAdd and publishes it to the other roles through a mailbox in
// shared memory, so a CTA that drew short row tiles simply takes more of them.  Items
// are numbered with the row tiles of one (expert, weight tile) adjacent: CTAs that take
// neighbouring items stream the same weights at the same time and the second reader
// finds them in L2.  Warps: 0 TMA producer (weights), 2 TMA producer
// (token terms), 1 and 3 MMA issuers (one per weight tile), 4-7
// scale writers (global -> shared -> tensor memory, one lane quadrant each), 8-23
// epilogue.  All barrier waits are bounded.
#include "k3_grouped.h"
#include "k3_moe_ops.h"
#include "k3_tc_ptx.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

using namespace k3;
using namespace k3::tc;

namespace {

constexpr uint32_t BM = 128, KS = 128;                    // weight rows per tile, K per pipeline stage
constexpr uint32_t kATile = BM * 128u;                    // bytes in shared memory (8-bit containers)
constexpr uint32_t kATx = BM * 64u;                       // bytes the TMA transaction counts (packed)
constexpr uint32_t kBBox = 32u;                           // token rows per TMA box
constexpr uint32_t kEpilogueWarps = 16;
constexpr uint32_t kThreads = (8u + kEpilogueWarps) * 32u;   // 24 warps
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kMaxGroups = 1024;
constexpr uint32_t kItemSlots = 4;                        // mailbox of item numbers, producer -> other roles
constexpr uint32_t kItemLead = 16;                        // stages by which an item is published ahead of its stream
constexpr uint32_t kItemReaders = 7u + kEpilogueWarps;    // term producer, 2 issuers, 4 writers, epilogue warps
constexpr uint32_t kNoItem = 0xffffffffu;
constexpr uint32_t kBarBytes = 448;                       // barriers, then a few words, then the scan's warp totals
constexpr uint32_t kStackedRows = 64;

// The two instances.  Groups of up to 64 rows (kMany false): one row tile per group, the hi and the
// lo rows ONE N operand (lo from row `block` on) with accumulator columns of their own, so that a K
// block of 32 is one MMA per weight tile and the 8-bit weight containers are read from shared
// memory once.  Larger groups: row tiles of up to 160 rows, the hi and the lo MMA adding into the
// same columns.  A tile of 160 rows takes the weights through the copy unit once where a tile
// of 128 and a remainder took them twice: with 8192 tokens and a Zipf router bias most experts (573
// of 896) have 129 to 160 rows, and their remainders of a few rows were 29 % of the expert phase (with
// a uniform bias or four hot experts few have).  160 is what fits: three
// stages of 72 KB, two accumulators of 160 columns beside the scales (192 rows in two stages of
// 80 KB ran at 1250 useful TFLOP/s, 160 in three at 1300; both operand orders alike).  192 experts,
// whole calls back to back, tiles of 128 and a remainder / these: 129 rows 3579 / 2863 us, 146 3746 / 3148,
// 161 4014 / 3907, 176 4101 / 3995, 192 4250 / 4198, 193 4774 / 4367, 224 4928 / 4660, 256 5135 / 5099,
// 320 6660 / 6139.
// One accumulator for hi and lo has twice the additions of two, which a remainder of up to 64 rows had
// in the kernel with tiles of 128.  Against 64 bits, remainder rows of 18 group sizes, two / one: bf16
// activations on the wrong side of a rounding line 0.098 / 0.114 % at K = 7168 and 0.099 / 0.103 at 3584 (all
// other rows of such groups, both kernels: 0.123, 0.103), down products 0.61 / 0.61; the layer's rel-L2 to 64
// bits is 0.004097 with both (24 inputs of 3001 to 16384 tokens: -5e-6 to +1e-5 of itself, on average +2e-6).
template <bool kMany>
struct Cfg {
    static constexpr uint32_t kTileRows = kMany ? 160u : kStackedRows;
    static constexpr uint32_t kTermRows = kMany ? 160u : 2u * kStackedRows;      // rows of the N operand, at most
    static constexpr uint32_t kStages = kMany ? 3u : 4u;
    static constexpr uint32_t kStageBytes = 2u * kATile + 2u * kTileRows * 128u; // A0 | A1 | token terms
    static constexpr uint32_t kSfStages = kMany ? 2u : 4u;                       // stages per scale batch
    static constexpr uint32_t kSfSlots = kMany ? 2u : 4u;                        // scale ring in shared memory
    static constexpr uint32_t kSfAhead = kMany ? 2u : 3u;                        // batches under way to it
    static constexpr uint32_t kSfRow = 4u * kSfStages;                           // scale bytes of a row per batch
    static constexpr uint32_t kSfSlotBytes = (2u * BM + kTermRows) * kSfRow;     // SFA0 | SFA1 | SFB
    static constexpr uint32_t kSfBatches = kMany ? 6u : 3u;                      // scale ring in tensor memory
    static constexpr uint32_t kAccStride = kMany ? 160u : 128u;                  // tile 0 | tile 1
    static constexpr uint32_t kSftStage = kMany ? 8u : 4u;                       // token scale columns per stage
    static constexpr uint32_t kSfwCol = 2u * kAccStride;                         // weight scales: 8 columns per stage
    static constexpr uint32_t kSftCol = kSfwCol + 8u * kSfStages * kSfBatches;
    static constexpr uint32_t kSpan = kTileRows / 4u;                            // token rows of an epilogue warp, at most
    static constexpr uint32_t kSmemBytes =
        kStages * kStageBytes + kSfSlots * kSfSlotBytes + kBarBytes + (kMaxGroups + 1u) * 4u;
    static_assert(kSftCol + kSftStage * kSfStages * kSfBatches <= kTmemCols, "tensor memory");
    static_assert(kSmemBytes <= 227u * 1024u, "one CTA's shared memory");
    static_assert((2u * (kStages + kSfBatches + kSfSlots + 2u + kItemSlots)) * 8u + (3u + kItemSlots + kThreads / 32u) * 4u <= kBarBytes,
                  "barriers and words");
};

enum EMode : int { kEAct = 0, kEBf16 = 1 };

__device__ uint32_t g_gmx_status = 0;

K3_DEVINL void tmem_st_32x16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
K3_DEVINL void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
K3_DEVINL void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

K3_DEVINL void mma_mx(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                      uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n\t}" ::
            "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc)
        : "memory");
}

// UE8M0 scales, M = 128, K-major, byte 0 of the scale columns (kNextScaleByte: one further).
// A = weights (E2M1, 5), B = token terms (E4M3, 0).
constexpr uint32_t kNextScaleByte = (1u << 29) | (1u << 4);
K3_DEVINL uint32_t make_idesc_mx(uint32_t n) {
    return (5u << 7) | (0u << 10) | ((n >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24);
}

// Two-term E4M3 form of a block of 32 values held one per lane:
// v = 2^(scale_byte - 127) * (hi + lo).  The block exponent puts the largest
// magnitude in [128, 256), inside E4M3's finite range (448).  The terms saturate, so a block
// that holds an infinity or NaN gets E8M0's NaN as its scale: its row's results are NaN.
K3_DEVINL uint32_t block_scale_byte(uint32_t max_exponent) {
    return max_exponent == 0xffu ? 255u : min(max(max_exponent, 8u), 254u) - 7u;
}
struct SplitScale {
    float mult;             // 2^-(block exponent)
    uint32_t scale_byte;    // E8M0
};
K3_DEVINL SplitScale block_scale(float v) {
    const uint32_t mx = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(v)));
    const uint32_t max_exponent = mx >> 23;           // biased, of the block maximum
    const uint32_t be = min(max(max_exponent, 8u), 254u);
    SplitScale s;
    s.mult = __uint_as_float((261u - be) << 23);      // 2^(7 - (be - 127))
    s.scale_byte = block_scale_byte(max_exponent);
    return s;
}
// (hi0, hi1) in the low 16 bits, (lo0, lo1) in the high 16 bits
K3_DEVINL uint32_t split_pair(float a, float b) {
    const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(hi, __NV_E4M3);
    const float2 hf = __half22float2(__half2(hr));
    const __nv_fp8x2_storage_t lo =
        __nv_cvt_float2_to_fp8x2(make_float2(a - hf.x, b - hf.y), __NV_SATFINITE, __NV_E4M3);
    return (uint32_t)hi | ((uint32_t)lo << 16);
}

// bf16 of lo in the low half, of hi in the high half (round to nearest even)
K3_DEVINL uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

struct GmxArgs {
    const uint32_t *offsets;             // [groups+1]
    k3_group_parts parts;
    const uint8_t *sfa0, *sfa1;          // weight block scales [groups * w_rows, k / 32], tile 0 / tile 1
    const uint8_t *sfb;                  // token block scales [rows, k / 32]
    uint16_t *out;                       // bf16 [rows, out_width] (may be null in gate/up mode)
    uint8_t *act_hi, *act_lo, *act_sf;   // gate/up mode: E4M3 terms and block scales of the activation
    uint32_t groups, rows, row_floor, row_ceil, w_rows, k, out_width, m_items;   // groups of row_floor < rows <= row_ceil
    uint32_t *item_counter;              // zero before the launch; items are drawn from it
    int activation;
    float beta, linear_beta;
};

struct Item {
    uint32_t group, row_start, rows_valid, m_item;
};

// rows of the group in the whole pass
K3_DEVINL uint32_t pass_rows(const k3_group_parts &parts, uint32_t group, uint32_t rows) {
    return parts.table == nullptr ? rows : max(parts.table[group], rows);
}

// How a row tile's terms lie in shared memory: hi rows from row 0, lo rows from row `block` on; n
// rows of the N operand per MMA (hi and lo together where they are stacked).
struct TermLayout {
    uint32_t block, n;
};
template <bool kMany>
K3_DEVINL TermLayout term_layout(const Item &it) {
    const uint32_t n16 = (it.rows_valid + 15u) & ~15u;
    if (kMany) return {Cfg<true>::kTileRows, n16};
    const uint32_t block = it.rows_valid <= 32u ? 32u : kStackedRows;
    return {block, block + n16};
}

// Item w -> (group, weight tile, row tile).  prefix[g] = row tiles of the groups before
// g; group g owns items [prefix[g] * m_items, prefix[g + 1] * m_items), numbered with
// the row tile fastest.  A group's tiles are as even as multiples of 16 rows allow; none is
// empty, since their size is at most kTileRows and their number rows / kTileRows rounded up.
template <bool kMany>
K3_DEVINL Item decode_item(uint32_t w, const uint32_t *prefix, const GmxArgs &a) {
    Item it;
    const uint32_t nt = w / a.m_items;             // prefix[group] <= nt < prefix[group + 1]
    uint32_t lo = 0, hi = a.groups;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= nt) lo = mid; else hi = mid;
    }
    it.group = lo;
    const uint32_t tiles = prefix[lo + 1u] - prefix[lo];
    const uint32_t j = w - prefix[lo] * a.m_items;
    it.m_item = j / tiles;
    const uint32_t begin = a.offsets[lo], rows = a.offsets[lo + 1u] - begin, first = j % tiles *
        (kMany ? ((rows + tiles - 1u) / tiles + 15u) & ~15u : kStackedRows);
    it.row_start = begin + first;
    it.rows_valid = min(kMany ? ((rows + tiles - 1u) / tiles + 15u) & ~15u : kStackedRows, rows - first);
    return it;
}

// Accumulator columns [0, 256) of the instance for smaller groups as two buffers of 128: a row
// tile of at most 32 rows (N <= 64) takes one buffer (tile 0 in its first 64 columns, tile 1 in
// the other 64), so that its MMAs run while the epilogue still reads the item before; a larger
// tile takes both (tile 0 in [0, 128), tile 1 in [128, 256)), and so does every tile of the other
// instance.  Issuers and epilogue warps walk the items in the same order and keep the same books:
// uses per buffer (the barriers' phase) and whose turn it is.
template <bool kMany>
struct AccBuffers {
    uint32_t use0 = 0u, use1 = 0u;
    uint32_t turn = 0u;
    __device__ uint32_t uses(uint32_t b) const { return b == 0u ? use0 : use1; }
    __device__ bool small(const Item &it) const { return !kMany && it.rows_valid <= 32u; }
    __device__ uint32_t first(bool is_small) const { return is_small ? turn : 0u; }
    __device__ uint32_t column(bool is_small, uint32_t b0, uint32_t tile) const {
        return is_small ? b0 * 128u + tile * 64u : tile * Cfg<kMany>::kAccStride;
    }
    __device__ void advance(bool is_small, uint32_t b0) {
        if (is_small) {
            if (b0 == 0u) use0++; else use1++;
            turn ^= 1u;
        } else {
            use0++;
            use1++;
            turn = 0u;
        }
    }
};

struct GmxMaps {
    CUtensorMap a0, a1;        // packed E2M1 weights (4-bit elements, expanded by the copy)
    CUtensorMap bhi, blo;      // token terms, E4M3 bytes
};

// Weights and terms of a stage share their barriers.
template <int kE, bool kMany>
__global__ void __launch_bounds__(kThreads, 1)
grouped_mx_kernel(const __grid_constant__ GmxMaps maps, GmxArgs a) {
    using C = Cfg<kMany>;
    constexpr uint32_t kStages = C::kStages, kStageBytes = C::kStageBytes, kSfSlots = C::kSfSlots;
    constexpr uint32_t kSfBatches = C::kSfBatches, kSfStages = C::kSfStages;
    extern __shared__ __align__(1024) unsigned char base[];      // the swizzled stages start on multiples of 1024
    unsigned char *sf_smem = base + kStages * kStageBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sf_smem + kSfSlots * C::kSfSlotBytes);
    uint64_t *full = bars, *empty = full + kStages;
    uint64_t *sf_full = empty + kStages, *sf_empty = sf_full + kSfBatches;
    uint64_t *sfs_full = sf_empty + kSfBatches, *sfs_empty = sfs_full + kSfSlots;
    uint64_t *acc_full = sfs_empty + kSfSlots, *acc_empty = acc_full + 2;      // two accumulator buffers
    uint64_t *item_full = acc_empty + 2, *item_empty = item_full + kItemSlots;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(item_empty + kItemSlots);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    uint32_t *total_items_s = tmem_slot + 2;
    volatile uint32_t *item_box = tmem_slot + 3;          // [kItemSlots]
    uint32_t *warp_tot = tmem_slot + 3 + kItemSlots;      // [kThreads / kWarp]
    uint32_t *prefix = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(bars) + kBarBytes);
    const uint32_t warp = warp_index(), lane = threadIdx.x % kWarp;
    const uint32_t steps = a.k / KS;
    const uint32_t tile_rows = kE == kEAct ? BM : 2u * BM;     // weight rows one item advances

    if (threadIdx.x == 0) {
        *abort_flag = 0u;
        for (uint32_t s = 0; s < kStages; s++) {
            mbar_init(&full[s], 2);          // two producers arrive (weights, token terms)
            mbar_init(&empty[s], 2);         // both MMA issuers release a stage
        }
        for (uint32_t b = 0; b < kSfBatches; b++) {
            mbar_init(&sf_full[b], 4);
            mbar_init(&sf_empty[b], 2);
        }
        for (uint32_t b = 0; b < kSfSlots; b++) {
            mbar_init(&sfs_full[b], 4u * kWarp);     // every thread of the scale writers
            mbar_init(&sfs_empty[b], 4);
        }
        for (uint32_t b = 0; b < 2u; b++) {
            mbar_init(&acc_full[b], 2);
            mbar_init(&acc_empty[b], kEpilogueWarps);
        }
        for (uint32_t b = 0; b < kItemSlots; b++) {
            mbar_init(&item_full[b], 1);
            mbar_init(&item_empty[b], kItemReaders);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    // The kernel in front is the packed one or the other instance of this one.  It has waited for
    // everything before it, and nothing it writes is read here, so this kernel's blocks start as its
    // blocks leave and wait for it only before they end (so that who waits for this one waits for both).
    pdl_trigger();
    {   // exclusive prefix of the groups' row tiles (<= 1024 groups)
        uint32_t v[2], incl[2], run = 0;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t g = threadIdx.x * 2u + j;
            const uint32_t n = g < a.groups ? a.offsets[g + 1u] - a.offsets[g] : 0u;
            const uint32_t whole = n != 0u ? pass_rows(a.parts, g, n) : 0u;
            v[j] = whole > a.row_floor && whole <= a.row_ceil ? (n + C::kTileRows - 1u) / C::kTileRows : 0u;
            run += v[j];
            incl[j] = run;
        }
        uint32_t scan = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t n = __shfl_up_sync(0xffffffffu, scan, o);
            if (lane >= (uint32_t)o) scan += n;
        }
        if (lane == 31) warp_tot[warp] = scan;
        __syncthreads();
        uint32_t warp_base = 0;
        for (uint32_t wv = 0; wv < warp; wv++) warp_base += warp_tot[wv];
        const uint32_t excl = warp_base + scan - run;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t g = threadIdx.x * 2u + j;
            if (g < a.groups) prefix[g] = excl + incl[j] - v[j];
            if (g + 1u == a.groups) {
                prefix[a.groups] = excl + incl[j];
                *total_items_s = (excl + incl[j]) * a.m_items;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t total_items = *total_items_s;

    // Reader side of the item mailbox: the n-th call (of one thread, or of a warp) returns the n-th
    // item this CTA drew, kNoItem when there are no more.
    uint32_t item_seq = 0;
    auto next_item = [&]() -> uint32_t {
        const uint32_t slot = item_seq % kItemSlots, parity = (item_seq / kItemSlots) & 1u;
        item_seq++;
        uint32_t w = kNoItem;
        if (mbar_wait(&item_full[slot], parity, abort_flag)) {
            w = item_box[slot];
            mbar_arrive(&item_empty[slot]);
        }
        return w;
    };
    auto item_published = [&]() -> bool {                 // would next_item_warp() return at once?
        const bool ready = lane == 0 && mbar_test(&item_full[item_seq % kItemSlots], (item_seq / kItemSlots) & 1u);
        return __any_sync(0xffffffffu, ready);
    };
    auto next_item_warp = [&]() -> uint32_t {
        uint32_t w = kNoItem;
        if (lane == 0) w = next_item();
        return __shfl_sync(0xffffffffu, w, 0);
    };

    if (warp == 0) {
        // ================================ TMA producer: weights; draws the items
        // The next item is published kItemLead stages before this one's stream ends, so that the scale
        // writers can ask for its first scales while this one's last stages are multiplied.
        if (elect_one()) {
            prefetch_tensormap(&maps.a0);
            prefetch_tensormap(&maps.a1);
            uint32_t s = 0, ph = 0, seq = 0;
            auto publish = [&](uint32_t w) -> bool {
                const uint32_t slot = seq % kItemSlots, parity = (seq / kItemSlots) & 1u;
                seq++;
                if (!mbar_wait(&item_empty[slot], parity ^ 1u, abort_flag)) return false;
                item_box[slot] = w < total_items ? w : kNoItem;
                mbar_arrive(&item_full[slot]);
                return true;
            };
            const uint32_t draw_at = steps > kItemLead + 1u ? steps - kItemLead - 1u : 0u;
            uint32_t w = atomicAdd(a.item_counter, 1u);
            bool ok = publish(w);
            while (ok && w < total_items) {
                const Item it = decode_item<kMany>(w, prefix, a);
                const int32_t y0 = (int32_t)(it.group * a.w_rows + it.m_item * tile_rows);
                const int32_t y1 = kE == kEAct ? y0 : y0 + (int32_t)BM;
                for (uint32_t st = 0; st < steps; st++) {
                    if (st == draw_at) w = atomicAdd(a.item_counter, 1u);      // travels during this stage
                    if (st == draw_at + 1u && !publish(w)) { ok = false; break; }
                    if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
                    unsigned char *dst = base + s * kStageBytes;
                    const int32_t x = (int32_t)(st * KS);
                    mbar_arrive_expect_tx(&full[s], 2u * kATx);
                    tma_load_2d(dst, &maps.a0, &full[s], x, y0);
                    tma_load_2d(dst + kATile, &maps.a1, &full[s], x, y1);
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 2) {
        // ================================ TMA producer: token terms
        if (elect_one()) {
            prefetch_tensormap(&maps.bhi);
            prefetch_tensormap(&maps.blo);
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (uint32_t w = next_item(); ok && w != kNoItem; w = next_item()) {
                const Item it = decode_item<kMany>(w, prefix, a);
                const uint32_t boxes = (it.rows_valid + kBBox - 1u) / kBBox;
                const TermLayout t = term_layout<kMany>(it);
                for (uint32_t st = 0; st < steps; st++) {
                    if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
                    const int32_t x = (int32_t)(st * KS);
                    // only as many 32-row boxes as the tile has rows
                    mbar_arrive_expect_tx(&full[s], 2u * boxes * kBBox * 128u);
                    unsigned char *bh = base + s * kStageBytes + 2u * kATile, *bl = bh + t.block * 128u;
                    for (uint32_t b = 0; b < boxes; b++) {
                        const int32_t y = (int32_t)(it.row_start + b * kBBox);
                        tma_load_2d(bh + b * kBBox * 128u, &maps.bhi, &full[s], x, y);
                        tma_load_2d(bl + b * kBBox * 128u, &maps.blo, &full[s], x, y);
                    }
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1 || warp == 3) {
        // ==================================================== MMA issuers
        // One per weight tile; both commit to the same stage / scale / accumulator barriers (count 2).
        if (elect_one()) {
            const uint32_t q = warp == 1 ? 0u : 1u;
            uint32_t s = 0, ph = 0, sb = 0, sph = 0;
            AccBuffers<kMany> acc;
            bool ok = true;
            for (uint32_t w = next_item(); ok && w != kNoItem; w = next_item()) {
                const Item it = decode_item<kMany>(w, prefix, a);
                const TermLayout t = term_layout<kMany>(it);
                const uint32_t idesc = make_idesc_mx(t.n);
                const bool small = acc.small(it);
                const uint32_t b0 = acc.first(small);
                if (!mbar_wait(&acc_empty[b0], (acc.uses(b0) & 1u) ^ 1u, abort_flag) ||
                    (!small && !mbar_wait(&acc_empty[1], (acc.use1 & 1u) ^ 1u, abort_flag))) {
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + acc.column(small, b0, q);
                for (uint32_t st = 0; st < steps; st++) {
                    const uint32_t in_batch = st % kSfStages;
                    if (!mbar_wait(&full[s], ph, abort_flag) ||
                        (in_batch == 0u && !mbar_wait(&sf_full[sb], sph, abort_flag))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const unsigned char *src = base + s * kStageBytes;
                    const uint64_t dw = make_desc_sw128(smem_u32(src + q * kATile));
                    const uint64_t dhi = make_desc_sw128(smem_u32(src + 2u * kATile));
                    const uint32_t sfw = tmem + C::kSfwCol + (sb * kSfStages + in_batch) * 8u + 4u * q;
                    const uint32_t sft = tmem + C::kSftCol + (sb * kSfStages + in_batch) * C::kSftStage;
                    if (kMany) {
                        const uint64_t dlo = make_desc_sw128(smem_u32(src + 2u * kATile + C::kTileRows * 128u));
#pragma unroll
                        for (uint32_t j = 0; j < 4u; j++) {          // K blocks of 32 inside the stage
                            mma_mx(d, dw + 2u * j, dhi + 2u * j, idesc + j * kNextScaleByte, sfw, sft,
                                   (st | j) != 0u ? 1u : 0u);
                            mma_mx(d, dw + 2u * j, dlo + 2u * j, idesc + j * kNextScaleByte, sfw, sft, 1u);
                        }
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 4u; j++)
                            mma_mx(d, dw + 2u * j, dhi + 2u * j, idesc + j * kNextScaleByte, sfw, sft,
                                   (st | j) != 0u ? 1u : 0u);
                    }
                    mma_commit(&empty[s]);
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                    if (in_batch == kSfStages - 1u) {
                        mma_commit(&sf_empty[sb]);
                        if (++sb == kSfBatches) { sb = 0; sph ^= 1u; }
                    }
                }
                if (!ok) break;
                mma_commit(&acc_full[b0]);
                if (!small) mma_commit(&acc_full[1]);
                acc.advance(small, b0);
            }
        }
    } else if (warp < 8) {
        // ================== scale writers: global -> shared -> tensor memory
        // A scale column holds rows 32c .. 32c+31 (lane = row % 32), the same in every
        // lane quadrant; each warp fills its own quadrant.  One batch = kSfStages stages.  A thread
        // fetches the batch's scale bytes of one row of each table, kSfAhead batches
        // before they are stored: as TMA boxes of 128 rows x 16 bytes, issued with the
        // weights of the batch's first stage, they came late (the batch has three stages to get here)
        // and took a sixth of the rows that the copy unit moves (with the elected issue and, above 64
        // rows, still the terms as the A operand, both products of 192 experts, back to back: 128 rows
        // 1935 -> 1717 us, 64 rows 1288 -> 1196).  This kernel has not waited when it reads the token
        // scales, and the 8-byte copies go through L1 (they have no other form): both are safe because the
        // scales were complete before this kernel was launched.  The packed kernel, which is first
        // of a projection's launches, triggers only after its own wait for whoever wrote them.
        const uint32_t quad = warp & 3u;
        const uint32_t lane_base = (32u * quad) << 16;
        const uint32_t row = 32u * quad + lane, kb = a.k / 32u;
        uint32_t sb = 0, sph = 0, ss = 0, ssph = 0;
        uint32_t fs = 0, fph = 0, left = 0, pending = 0;       // fetching side: slot, batches left in its item
        const uint8_t *p0 = nullptr, *p1 = nullptr, *pt = nullptr, *pu = nullptr;
        bool ok = true, more = true;
        // One batch's copies.  While batches are pending it does not wait for an item that is not
        // published yet: the items in front would then wait for scales that this warp holds back.
        auto fetch = [&]() -> bool {
            if (left == 0u) {
                if (pending != 0u && !item_published()) return false;
                const uint32_t w = next_item_warp();
                if (w == kNoItem) { more = false; return false; }
                const Item it = decode_item<kMany>(w, prefix, a);
                const uint64_t y0 = (uint64_t)it.group * a.w_rows + it.m_item * tile_rows + row;
                p0 = a.sfa0 + y0 * kb;
                p1 = a.sfa1 + (kE == kEAct ? y0 : y0 + BM) * kb;
                // a stacked operand's lo rows have the scales of its hi rows; rows past the end repeat the last
                const uint32_t r = min(kMany ? row : row & (term_layout<kMany>(it).block - 1u), it.rows_valid - 1u);
                pt = a.sfb + (uint64_t)(it.row_start + r) * kb;
                if (kMany) pu = a.sfb + (uint64_t)(it.row_start + min(BM + lane, it.rows_valid - 1u)) * kb;
                left = steps / kSfStages;
            }
            if (!mbar_wait(&sfs_empty[fs], fph ^ 1u, abort_flag)) { ok = false; return false; }
            unsigned char *dst = sf_smem + fs * C::kSfSlotBytes + row * C::kSfRow;
            cp_async<C::kSfRow>(dst, p0);
            cp_async<C::kSfRow>(dst + BM * C::kSfRow, p1);
            cp_async<C::kSfRow>(dst + 2u * BM * C::kSfRow, pt);
            if (kMany && quad == 0u) {                       // token rows 128 .. 159
                cp_async<C::kSfRow>(dst + 3u * BM * C::kSfRow, pu);
                pu += C::kSfRow;
            }
            cp_async_arrive(&sfs_full[fs]);
            p0 += C::kSfRow;
            p1 += C::kSfRow;
            pt += C::kSfRow;
            left--;
            pending++;
            if (++fs == kSfSlots) { fs = 0; fph ^= 1u; }
            return true;
        };
        while (true) {
            while (ok && more && pending < C::kSfAhead && fetch()) {
            }
            if (!ok || pending == 0u) break;
            if (!mbar_wait(&sfs_full[ss], ssph, abort_flag)) break;
            const unsigned char *src = sf_smem + ss * C::kSfSlotBytes;
            const uint32_t wcol = tmem + lane_base + C::kSfwCol + sb * kSfStages * 8u;
            const uint32_t tcol = tmem + lane_base + C::kSftCol + sb * kSfStages * C::kSftStage;
            if constexpr (kMany) {
                auto at = [&](uint32_t r) { return *reinterpret_cast<const uint2 *>(src + r * 8u); };
                uint2 v0[4], v1[4];
#pragma unroll
                for (uint32_t c = 0; c < 4u; c++) {
                    v0[c] = at(32u * c + lane);
                    v1[c] = at(BM + 32u * c + lane);
                }
                if (!mbar_wait(&sf_empty[sb], sph ^ 1u, abort_flag)) break;
                tc_fence_after();
                const uint32_t w01[16] = {v0[0].x, v0[1].x, v0[2].x, v0[3].x, v1[0].x, v1[1].x, v1[2].x, v1[3].x,
                                          v0[0].y, v0[1].y, v0[2].y, v0[3].y, v1[0].y, v1[1].y, v1[2].y, v1[3].y};
                tmem_st_32x16(wcol, w01);
                uint2 v[5];
#pragma unroll
                for (uint32_t c = 0; c < 5u; c++) v[c] = at(2u * BM + 32u * c + lane);
                const uint32_t tok[16] = {v[0].x, v[1].x, v[2].x, v[3].x, v[4].x, 0u, 0u, 0u,
                                          v[0].y, v[1].y, v[2].y, v[3].y, v[4].y, 0u, 0u, 0u};
                tmem_st_32x16(tcol, tok);
            } else {
                auto rows_of = [&](uint32_t t, uint4 (&v)[4]) {
#pragma unroll
                    for (uint32_t c = 0; c < 4u; c++)
                        v[c] = *reinterpret_cast<const uint4 *>(src + (t * BM + 32u * c + lane) * 16u);
                };
                uint4 v0[4], v1[4];
                rows_of(0u, v0);
                rows_of(1u, v1);
                if (!mbar_wait(&sf_empty[sb], sph ^ 1u, abort_flag)) break;
                tc_fence_after();
                const uint32_t w01[16] = {v0[0].x, v0[1].x, v0[2].x, v0[3].x, v1[0].x, v1[1].x, v1[2].x, v1[3].x,
                                          v0[0].y, v0[1].y, v0[2].y, v0[3].y, v1[0].y, v1[1].y, v1[2].y, v1[3].y};
                tmem_st_32x16(wcol, w01);
                const uint32_t w23[16] = {v0[0].z, v0[1].z, v0[2].z, v0[3].z, v1[0].z, v1[1].z, v1[2].z, v1[3].z,
                                          v0[0].w, v0[1].w, v0[2].w, v0[3].w, v1[0].w, v1[1].w, v1[2].w, v1[3].w};
                tmem_st_32x16(wcol + 16u, w23);
                rows_of(2u, v0);
                const uint32_t tok[16] = {v0[0].x, v0[1].x, v0[2].x, v0[3].x, v0[0].y, v0[1].y, v0[2].y, v0[3].y,
                                          v0[0].z, v0[1].z, v0[2].z, v0[3].z, v0[0].w, v0[1].w, v0[2].w, v0[3].w};
                tmem_st_32x16(tcol, tok);
            }
            // The shared-memory slot is given back only now: the stores above consumed every
            // loaded register, so the loads have completed (an arrive right after issuing
            // them would not wait for that).
            __syncwarp();
            if (lane == 0) mbar_arrive(&sfs_empty[ss]);
            if (++ss == kSfSlots) { ss = 0; ssph ^= 1u; }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sf_full[sb]);
            if (++sb == kSfBatches) { sb = 0; sph ^= 1u; }
            pending--;
        }
        cp_async_wait_all();
    } else {
        // ======================================================== epilogue
        // Sixteen warps: quadrant = warp % 4 (tensor-memory lanes: weight rows), the accumulators'
        // columns (token rows) in four parts.  A warp takes its part of both accumulators out of
        // tensor memory at once, rounded to bf16 (which both modes do anyway) and packed in pairs, and
        // frees the accumulators before it computes anything: a tile of more than 32 rows has no
        // second buffer, so the MMAs of the next item wait for exactly this.
        const uint32_t quad = warp & 3u;
        const uint32_t part = (warp - 8u) >> 2;
        const uint32_t m = 32u * quad + lane;            // weight row inside the tile
        AccBuffers<kMany> acc;
        for (uint32_t w = next_item_warp(); w != kNoItem; w = next_item_warp()) {
            const Item it = decode_item<kMany>(w, prefix, a);
            const bool small = acc.small(it);
            const uint32_t b0 = acc.first(small);
            if (!mbar_wait(&acc_full[b0], acc.uses(b0) & 1u, abort_flag) ||
                (!small && !mbar_wait(&acc_full[1], acc.use1 & 1u, abort_flag))) {
                break;
            }
            acc.advance(small, b0);
            tc_fence_after();
            const uint32_t t0 = tmem + ((32u * quad) << 16) + acc.column(small, b0, 0u);
            const uint32_t tile1 = acc.column(small, b0, 1u) - acc.column(small, b0, 0u);
            const uint32_t col0 = it.m_item * tile_rows + m;
            const uint32_t col1 = kE == kEAct ? col0 : col0 + BM;
            const bool in0 = col0 < a.w_rows, in1 = col1 < a.w_rows;
            const TermLayout t = term_layout<kMany>(it);
            const uint32_t span = kMany ? (it.rows_valid + 31u) / 32u * 8u : t.block / 4u, c = span * part;   // this warp's token rows
            uint32_t pair[C::kSpan];                                     // bf16 of tile 0 | tile 1 << 16
#pragma unroll
            for (uint32_t i = 0; i < C::kSpan; i += 8u) {
                if (i >= span || c + i >= it.rows_valid) break;
                uint32_t r0[8], r1[8];
                tmem_ld_32x8(t0 + c + i, r0);
                tmem_ld_32x8(t0 + tile1 + c + i, r1);
                if (!kMany) {
                    uint32_t lo[8];
                    tmem_ld_32x8(t0 + t.block + c + i, lo);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t j = 0; j < 8u; j++)
                        r0[j] = __float_as_uint(__uint_as_float(r0[j]) + __uint_as_float(lo[j]));
                    tmem_ld_32x8(t0 + tile1 + t.block + c + i, lo);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t j = 0; j < 8u; j++)
                        r1[j] = __float_as_uint(__uint_as_float(r1[j]) + __uint_as_float(lo[j]));
                } else {
                    tmem_ld_wait();
                }
#pragma unroll
                for (uint32_t j = 0; j < 8u; j++)
                    pair[i + j] = pack_bf16x2(__uint_as_float(r0[j]), __uint_as_float(r1[j]));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&acc_empty[b0]);
                if (!small) mbar_arrive(&acc_empty[1]);
            }
            if (c >= it.rows_valid) continue;
            const uint32_t n_here = min(span, it.rows_valid - c);
            if (kE == kEAct) {
#pragma unroll
                for (uint32_t j = 0; j < C::kSpan; j += 2u) {
                    if (j >= n_here) break;                              // uniform across the warp
                    const uint64_t row = (uint64_t)(it.row_start + c + j);
                    float av[2];
#pragma unroll
                    for (uint32_t q = 0; q < 2u; q++) {
                        const uint16_t bits = float_to_bf16_bits(
                            activation(bf16_lo(pair[j + q]), bf16_hi(pair[j + q]), a.activation, a.beta, a.linear_beta));
                        av[q] = in0 ? bf16_bits_to_float(bits) : 0.f;
                        if (a.out != nullptr && in0 && j + q < n_here) a.out[(row + q) * a.out_width + col0] = bits;
                    }
                    const SplitScale s0 = block_scale(av[0]), s1 = block_scale(av[1]);
                    const uint32_t packed = split_pair(av[0] * s0.mult, av[1] * s1.mult);
                    if (in0) {
                        a.act_hi[row * a.w_rows + col0] = (uint8_t)packed;
                        a.act_lo[row * a.w_rows + col0] = (uint8_t)(packed >> 16);
                        if (lane == 0) a.act_sf[row * (a.w_rows / 32u) + col0 / 32u] = (uint8_t)s0.scale_byte;
                        if (j + 1u < n_here) {
                            a.act_hi[(row + 1u) * a.w_rows + col0] = (uint8_t)(packed >> 8);
                            a.act_lo[(row + 1u) * a.w_rows + col0] = (uint8_t)(packed >> 24);
                            if (lane == 0)
                                a.act_sf[(row + 1u) * (a.w_rows / 32u) + col0 / 32u] = (uint8_t)s1.scale_byte;
                        }
                    }
                }
            } else {
#pragma unroll
                for (uint32_t j = 0; j < C::kSpan; j++) {
                    if (j >= n_here) break;
                    const uint64_t row = (uint64_t)(it.row_start + c + j);
                    if (in0) a.out[row * a.out_width + col0] = (uint16_t)pair[j];
                    if (in1) a.out[row * a.out_width + col1] = (uint16_t)(pair[j] >> 16);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag != 0u) atomicExch(&g_gmx_status, 1u);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
    pdl_wait();
}

// 16 bf16 columns of one lane (two lanes share a block of 32) -> E4M3 terms and the block's scale.
struct SplitColumns {
    uint4 hi, lo;
    uint32_t scale_byte;
};
K3_DEVINL SplitColumns split_columns(const uint16_t *p) {
    const uint4 q0 = reinterpret_cast<const uint4 *>(p)[0], q1 = reinterpret_cast<const uint4 *>(p)[1];
    const uint32_t wv[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    uint32_t mx = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) mx = max(mx, max(wv[q] & 0x7fffu, (wv[q] >> 16) & 0x7fffu));   // bf16 magnitudes
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    const uint32_t be = min(max(mx >> 7, 8u), 254u);
    const float mult = __uint_as_float((261u - be) << 23);
    uint32_t h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t p0 = split_pair(bf16_lo(wv[2 * q]) * mult, bf16_hi(wv[2 * q]) * mult);
        const uint32_t p1 = split_pair(bf16_lo(wv[2 * q + 1]) * mult, bf16_hi(wv[2 * q + 1]) * mult);
        h[q] = (p0 & 0xffffu) | (p1 << 16);
        l[q] = (p0 >> 16) | (p1 & 0xffff0000u);
    }
    return {make_uint4(h[0], h[1], h[2], h[3]), make_uint4(l[0], l[1], l[2], l[3]), block_scale_byte(mx >> 7)};
}

// Product rows' E4M3 terms and block scales from the bf16 source rows (row r reads x[index[r]],
// or x[r]); a warp converts 512 columns per pass.  Rows of groups this path leaves to the other
// kernel are skipped.
__global__ void __launch_bounds__(256)
split_rows_kernel(uint8_t *__restrict__ hi, uint8_t *__restrict__ lo, uint8_t *__restrict__ sf,
                  const uint16_t *x, const uint32_t *index,
                  const uint32_t *offsets, k3_group_parts parts, uint32_t groups, uint32_t rows,
                  uint32_t k) {
    // launched behind a kernel that waited for the dispatch and shares nothing else with this one
    const uint32_t lane = threadIdx.x % kWarp;
    const uint32_t warps = (gridDim.x * blockDim.x) / kWarp;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp; r < rows; r += warps) {
        uint32_t g = 0, end = groups;                      // group of row r
        while (end - g > 1u) {
            const uint32_t mid = (g + end) >> 1;
            if (offsets[mid] <= r) g = mid; else end = mid;
        }
        if (pass_rows(parts, g, offsets[g + 1u] - offsets[g]) <= k3_mx4_rows) continue;
        const uint16_t *src = x + (uint64_t)(index ? index[r] : r) * k;
        for (uint32_t c = lane * 16u; c < k; c += 512u) {
            const SplitColumns t = split_columns(src + c);
            *reinterpret_cast<uint4 *>(hi + (uint64_t)r * k + c) = t.hi;
            *reinterpret_cast<uint4 *>(lo + (uint64_t)r * k + c) = t.lo;
            if ((lane & 1u) == 0u) sf[(uint64_t)r * (k / 32u) + c / 32u] = (uint8_t)t.scale_byte;
        }
    }
    pdl_wait();
}

// The same for tokens whose routes are known: a warp converts 512 columns of a token once and
// stores them to each of its product rows.  Bound by those stores (14 KB per row at 7168
// columns): 8192 tokens took 649 us when every product row was converted on its own.
__global__ void __launch_bounds__(256)
split_tokens_kernel(uint8_t *__restrict__ hi, uint8_t *__restrict__ lo, uint8_t *__restrict__ sf,
                    const uint16_t *x, const uint32_t *ids,
                    const uint32_t *inv_perm, const uint32_t *offsets, uint32_t top_k,
                    uint32_t tokens, uint32_t k) {
    const uint32_t lane = threadIdx.x % kWarp, passes = k / 512u;
    const uint64_t warps = (uint64_t)(gridDim.x * blockDim.x) / kWarp, jobs = (uint64_t)tokens * passes;
    for (uint64_t job = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp; job < jobs; job += warps) {
        const uint32_t token = (uint32_t)(job / passes), c = (uint32_t)(job % passes) * 512u + lane * 16u;
        uint32_t row = 0u;
        bool mine = false;
        if (lane < top_k) {
            const uint32_t e = ids[(uint64_t)token * top_k + lane];
            row = inv_perm[(uint64_t)token * top_k + lane];
            mine = offsets[e + 1u] - offsets[e] > k3_mx4_rows;
        }
        const SplitColumns t = split_columns(x + (uint64_t)token * k + c);
        for (uint32_t todo = __ballot_sync(0xffffffffu, mine); todo != 0u; todo &= todo - 1u) {
            const uint64_t r = __shfl_sync(0xffffffffu, row, __ffs((int)todo) - 1);
            *reinterpret_cast<uint4 *>(hi + r * k + c) = t.hi;
            *reinterpret_cast<uint4 *>(lo + r * k + c) = t.lo;
            if ((lane & 1u) == 0u) sf[r * (k / 32u) + c / 32u] = (uint8_t)t.scale_byte;
        }
    }
    pdl_wait();
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
        } else {
            (void)cudaGetLastError();
        }
    });
    return fn;
}

bool map_2d(CUtensorMap *map, const void *ptr, CUtensorMapDataType type, uint64_t rows, uint64_t inner,
            uint64_t pitch_bytes, uint32_t box_inner, uint32_t box_rows, CUtensorMapSwizzle swizzle,
            uint32_t align) {
    auto fn = encode_fn();
    if (!fn || (((uintptr_t)ptr) & (align - 1u)) != 0) return false;
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {pitch_bytes};
    const cuuint32_t box[2] = {box_inner, box_rows};
    const cuuint32_t es[2] = {1, 1};
    return fn(map, type, 2, const_cast<void *>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Operands {
    const void *a0, *a1;               // packed weights of tile 0 / tile 1
    const void *sfa0, *sfa1;           // their scale tables
    const uint8_t *bhi, *blo, *sfb;    // token terms and scales
};

// Tensor maps depend only on the tables, the term buffers and the shape: the sets of the most
// recent calls are kept (a model alternates between its layers' tables and a few row counts),
// so a steady-state pass encodes nothing; when the table is full it starts over.
struct MapKey {
    int device, mode;
    const void *p[4];
    uint32_t dims[4];
    bool operator<(const MapKey &o) const {
        if (device != o.device) return device < o.device;
        if (mode != o.mode) return mode < o.mode;
        const int c = memcmp(p, o.p, sizeof(p));
        return c != 0 ? c < 0 : memcmp(dims, o.dims, sizeof(dims)) < 0;
    }
};

template <int kE>
bool launch(const Operands &op, GmxArgs args, bool many, cudaStream_t stream) {
    constexpr size_t kCachedSets = 256;
    static std::mutex map_lock;
    static std::map<MapKey, GmxMaps> cached;
    MapKey key{};
    key.device = current_device();
    key.mode = kE;
    const void *ptrs[4] = {op.a0, op.a1, op.bhi, op.blo};
    memcpy(key.p, ptrs, sizeof(ptrs));
    args.sfa0 = (const uint8_t *)op.sfa0;
    args.sfa1 = (const uint8_t *)op.sfa1;
    args.sfb = op.sfb;
    key.dims[0] = args.groups; key.dims[1] = args.w_rows; key.dims[2] = args.k; key.dims[3] = args.rows;
    GmxMaps maps;
    {
        std::lock_guard<std::mutex> guard(map_lock);
        auto it = cached.find(key);
        if (it == cached.end()) {
            const uint64_t w_total = (uint64_t)args.groups * args.w_rows;
            const auto u4 = CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B;
            const auto u8 = CU_TENSOR_MAP_DATA_TYPE_UINT8;
            const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
            if (!map_2d(&maps.a0, op.a0, u4, w_total, args.k, args.k / 2u, 128, BM, sw, 32u) ||
                !map_2d(&maps.a1, op.a1, u4, w_total, args.k, args.k / 2u, 128, BM, sw, 32u) ||
                !map_2d(&maps.bhi, op.bhi, u8, args.rows, args.k, args.k, 128, kBBox, sw, 16u) ||
                !map_2d(&maps.blo, op.blo, u8, args.rows, args.k, args.k, 128, kBBox, sw, 16u)) {
                return false;
            }
            if (cached.size() >= kCachedSets) cached.clear();
            cached.emplace(key, maps);
        } else {
            maps = it->second;
        }
    }
    auto kernel = many ? grouped_mx_kernel<kE, true> : grouped_mx_kernel<kE, false>;
    const uint32_t smem = many ? Cfg<true>::kSmemBytes : Cfg<false>::kSmemBytes;
    if (!set_max_dynamic_smem((const void *)kernel, smem)) return false;
    return launch_chained(kernel, sm_count(), kThreads, smem, stream, maps, args);
}

inline size_t up256(size_t v) { return (v + 255u) & ~(size_t)255u; }

struct Scratch {
    uint8_t *x_hi, *x_lo, *x_sf;       // per product row
    uint8_t *a_hi, *a_lo, *a_sf;       // activation, per product row
    uint32_t *counters;                // item counters of the six launches (zeroed per call)
    void *few;                         // scratch of the kernel for few rows per group
    size_t total;
};

Scratch carve_scratch(const k3_moe_layer_desc *d, uint32_t rows, uint32_t source_rows, void *workspace) {
    const size_t H = d->hidden, I = d->expert_hidden, R = rows;
    uint8_t *p = (uint8_t *)(((uintptr_t)workspace + 255u) & ~(uintptr_t)255u);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        uint8_t *q = p + off;
        off += up256(bytes);
        return q;
    };
    Scratch s{};
    s.x_hi = take(R * H);
    s.x_lo = take(R * H);
    s.x_sf = take(R * (H / 32u));
    s.a_hi = take(R * I);
    s.a_lo = take(R * I);
    s.a_sf = take(R * (I / 32u));
    s.counters = (uint32_t *)take(256);
    s.few = take(k3_grouped_mx4_workspace_bytes(d, rows, source_rows ? source_rows : rows));
    s.total = off + 256u;
    return s;
}

}  // namespace

uint32_t k3_grouped_mx_status() {
    uint32_t v = 0xffffffffu;
    if (cudaMemcpyFromSymbol(&v, g_gmx_status, sizeof(v)) != cudaSuccess) (void)cudaGetLastError();
    return v;
}

bool k3_grouped_mx_status_clear() {
    const uint32_t zero = 0u;
    if (cudaMemcpyToSymbol(g_gmx_status, &zero, sizeof(zero)) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return true;
}

size_t k3_grouped_mx_workspace_bytes(const k3_moe_layer_desc *d, uint32_t rows, uint32_t source_rows) {
    return carve_scratch(d, rows, source_rows, nullptr).total;
}

bool k3_grouped_mx_supported(const k3_moe_layer_desc *d, uint32_t rows) {
    return rows >= 32u && d->hidden % 512u == 0 && d->expert_hidden % 512u == 0 &&
           d->local_expert_count >= 1u && d->local_expert_count <= kMaxGroups && encode_fn() != nullptr &&
           ((((uintptr_t)d->w1_packed) | ((uintptr_t)d->w3_packed) | ((uintptr_t)d->w2_packed)) & 31u) == 0 &&
           ((((uintptr_t)d->w1_scales) | ((uintptr_t)d->w3_scales) | ((uintptr_t)d->w2_scales)) & 15u) == 0;
}

// Which kernel a group goes to, by its rows (ms of a whole call with 192 experts at 7168 x 2048, back to
// back; the weights alone are 0.69 ms of HBM time):
//   rows                   1     8     16    17    24    32    48    64    65    96    128
//   packed                 0.69  0.80  0.97
//   two-term, 64 rows                        1.15  1.15  1.20  1.49  1.66
//   two-term, 160 rows                       1.24  1.32  1.38  1.62  1.81  1.91  2.24  2.70
// Both products alone, before the elected issue of TMA and MMA instructions: packed with 8 / 16 / 24 / 32
// rows 0.73 / 0.81 / 1.28 / 1.38, two-term for up to 64 rows 0.99 / 1.00 / 1.01 / 1.03.
constexpr uint32_t kFewRows = k3_mx4_rows, kSomeRows = kStackedRows;

// rows_in bf16 [source_rows, H]; product row r reads rows_in[index[r]] (or row r
// when index == nullptr, source_rows == 0).  `act` bf16 [rows, I] is written when
// not null; rows_out bf16 [rows, H].
//
// A group's kernel decides the order in which its rows' sums are added.  A caller that cuts a pass
// into parts and wants the pass's bits says with `pass` how many rows the groups have in the whole pass.
bool k3_grouped_mx_experts(const k3_moe_layer_desc *d, void *rows_out, void *act, const void *rows_in,
                           const void *index, uint32_t source_rows, const void *offsets, uint32_t rows,
                           void *workspace, cudaStream_t stream, const k3_token_routes *routes,
                           const k3_part_of_pass *pass) {
    // a token selects an expert at most once, so no group has more rows than there are tokens
    const uint32_t max_group_rows = routes ? source_rows : 0xffffffffu;
    const uint32_t H = d->hidden, I = d->expert_hidden;
    const Scratch s = carve_scratch(d, rows, index ? source_rows : 0u, workspace);
    const uint32_t conv_rows = index ? source_rows : rows;
    const bool few = max_group_rows > kFewRows, many = max_group_rows > kSomeRows;   // launches beyond the packed one
    const k3_group_parts parts{pass ? (const uint32_t *)pass->group_rows : nullptr};
    if (!k3_grouped_mx4_terms(d, rows_in, conv_rows, rows, routes ? routes->ids : nullptr, offsets, s.few, s.counters,
                              stream)) {
        return false;
    }
    if (few && routes) {
        const uint64_t jobs = (uint64_t)source_rows * (H / 512u);
        if (!launch_chained(split_tokens_kernel, (uint32_t)std::min<uint64_t>((jobs + 7u) / 8u, (uint64_t)sm_count() * 16u),
                            256, 0, stream, s.x_hi, s.x_lo, s.x_sf, (const uint16_t *)rows_in,
                            (const uint32_t *)routes->ids, (const uint32_t *)routes->inv_perm, (const uint32_t *)offsets,
                            d->top_k, source_rows, H)) {
            return false;
        }
    } else if (few && !launch_chained(split_rows_kernel, std::min<uint32_t>((rows + 7u) / 8u, (uint32_t)sm_count() * 16u),
                                      256, 0, stream, s.x_hi, s.x_lo, s.x_sf, (const uint16_t *)rows_in,
                                      (const uint32_t *)index, (const uint32_t *)offsets, parts, d->local_expert_count,
                                      rows, H)) {
        return false;
    }
    GmxArgs a{};
    a.offsets = (const uint32_t *)offsets;
    a.parts = parts;
    a.groups = d->local_expert_count;
    a.rows = rows;
    a.activation = d->activation;
    a.beta = d->beta;
    a.linear_beta = d->linear_beta;
    auto launches = [&](auto mode, const Operands &op, uint32_t *counters) {
        constexpr int kE = decltype(mode)::value;
        GmxArgs b = a;
        b.row_floor = kFewRows;
        b.row_ceil = kSomeRows;
        b.item_counter = counters;
        if (few && !launch<kE>(op, b, false, stream)) return false;
        b.row_floor = kSomeRows;
        b.row_ceil = 0xffffffffu;
        b.item_counter = counters + 8;
        return !many || launch<kE>(op, b, true, stream);
    };
    // gate/up + activation
    a.out = (uint16_t *)act;
    a.act_hi = s.a_hi;
    a.act_lo = s.a_lo;
    a.act_sf = s.a_sf;
    a.w_rows = I;
    a.k = H;
    a.out_width = I;
    a.m_items = (I + BM - 1u) / BM;
    const Operands gu{d->w1_packed, d->w3_packed, d->w1_scales, d->w3_scales, s.x_hi, s.x_lo, s.x_sf};
    if (!k3_grouped_mx4_gateup(d, act, index, conv_rows, offsets, rows, s.few, s.counters, parts, stream) ||
        !launches(std::integral_constant<int, kEAct>{}, gu, s.counters + 8)) {
        return false;
    }
    // down
    a.out = (uint16_t *)rows_out;
    a.act_hi = a.act_lo = a.act_sf = nullptr;
    a.w_rows = H;
    a.k = I;
    a.out_width = H;
    a.m_items = (H + 2u * BM - 1u) / (2u * BM);
    const Operands dn{d->w2_packed, d->w2_packed, d->w2_scales, d->w2_scales, s.a_hi, s.a_lo, s.a_sf};
    return k3_grouped_mx4_down(d, rows_out, offsets, rows, conv_rows, s.few, s.counters + 24, parts, stream) &&
           launches(std::integral_constant<int, kEBf16>{}, dn, s.counters + 32);
}
