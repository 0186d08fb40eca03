// Ragged grouped GEMM for experts with few rows, on the packed block-scaled tensor-core path
// (tcgen05.mma kind::mxf4, scale_vec::2X).
//
//   out[r, m] = sum_k W[g(r)][m, k] * x[r, k]      r: token rows grouped by expert
//
// An expert with few rows costs its weight bytes, so everything here is about streaming those
// at the memory system's rate: the packed nibbles stay packed in shared memory (a stage holds
// exactly the bytes HBM delivered, 32 KB of 48 KB; 128 KB of weights in flight per SM) and a
// K = 64 MMA consumes them.  The two-term E4M3 kernel (k3_grouped_mx.cu) expands weights to
// 8-bit containers (half the weight bytes in flight, twice the shared-memory traffic).
// Activations are sums of eight E2M1 terms with a block scale per term (k3_e2m1_terms.cuh,
// exact for bf16): the terms of a row are eight consecutive rows of the N operand and the
// epilogue adds eight accumulator columns, so the up to 16 token rows of a group are N = 128.
//
// Work item = two 128-row weight tiles (gate and up with the activation fused, or 256 rows of
// down) x the token rows of one group over the whole K extent.  One persistent CTA per SM draws
// items from a global counter.  Groups of more than 16 rows are left to the other kernel: the
// terms of a row are 4 bytes per column and cross from L2 once per weight tile, so from two row
// tiles on L2 bounds this form (24 rows per expert 1.28 ms, two-term form 1.01).  Warps: 0
// producer of weights and their scales, 2 term producer (one box of 8 term rows x 2 stages per
// token row, straight from the token's terms: no gather pass), 1 and 3 MMA issuers (one per
// weight tile), 4-7 scale writers (weight scales from shared memory, term scales from global
// memory -> tensor memory), 8-23 epilogue.  192 experts at 7168 x 2048 (4.5 GB) with 1, 8, 16
// rows each: 0.70, 0.73, 0.81 ms = 6.5, 6.2, 5.6 TB/s (the two-term kernel took 1.10, 1.11,
// 1.14).  All barrier waits are bounded.
#include "k3_e2m1_terms.cuh"
#include "k3_grouped.h"
#include "k3_tc_ptx.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>

using namespace k3;
using namespace k3::tc;

namespace {

constexpr uint32_t BM = 128, kTileRows = k3_mx4_rows, KS = 256;     // K per pipeline stage
constexpr uint32_t kStages = 4;
constexpr uint32_t kATile = BM * 128u;                     // 128 rows x 256 K, packed
constexpr uint32_t kBAtom = kTerms * 128u;                 // one token row: 8 term rows, one swizzle atom
constexpr uint32_t kStageBytes = 2u * kATile;              // weights; the terms have a ring of their own:
constexpr uint32_t kBSlots = 2;                            // slots of two stages (512 K) of up to 16 token rows
constexpr uint32_t kBSlotBytes = 2u * kTileRows * kBAtom;
constexpr uint32_t kEpilogueWarps = 16;
constexpr uint32_t kThreads = (8u + kEpilogueWarps) * 32u; // 24 warps
constexpr uint32_t kSfBatches = 4;                         // scale ring in tensor memory: batches of 2 stages
constexpr uint32_t kSfSlots = 4;                           // scale ring in shared memory
constexpr uint32_t kSfKind = BM * 16u;                     // 128 rows x 16 scale bytes (512 K)
constexpr uint32_t kSfSlotBytes = 2u * kSfKind;            // SFA0 | SFA1
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kSfa0Col = 256;                         // accumulators below; kSfBatches x 16 columns each
constexpr uint32_t kSfa1Col = kSfa0Col + 16u * kSfBatches;
constexpr uint32_t kSfbCol = kSfa1Col + 16u * kSfBatches;
constexpr uint32_t kMaxGroups = 1024;
constexpr uint32_t kItemSlots = 4;                         // mailbox of item numbers, producer -> other roles
constexpr uint32_t kItemReaders = 7u + kEpilogueWarps;     // term producer, 2 issuers, 4 writers, epilogue warps
constexpr uint32_t kNoItem = 0xffffffffu;
constexpr uint32_t kBarBytes = 512;
constexpr uint32_t kSmemBytes =
    kStages * kStageBytes + kBSlots * kBSlotBytes + kSfSlots * kSfSlotBytes + 1024u + kBarBytes + (kMaxGroups + 1u) * 4u;
static_assert(kSmemBytes <= 227u * 1024u, "one CTA's shared memory");

__device__ uint32_t g_mx4_status = 0;

K3_DEVINL void tmem_st_32x16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
K3_DEVINL void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
K3_DEVINL void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

K3_DEVINL void mma_mx4(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n\t}" ::
            "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc)
        : "memory");
}

// A = B = E2M1, UE8M0 scales, M = 128, K = 64, K-major; sf = first scale byte (0 or 2) of the column
K3_DEVINL uint32_t make_idesc_mx4(uint32_t n, uint32_t sf) {
    return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24) | (sf << 29) | (sf << 4);
}

// K-major 128-byte-swizzled operand whose 8-row atoms lie 2048 bytes apart (two stages interleaved)
K3_DEVINL uint64_t make_desc_sw128_pairs(uint32_t smem_addr) {
    return (make_desc_sw128(smem_addr) & ~(0x3FFFull << 32)) | ((uint64_t)(2048u >> 4) << 32);
}

// 3-D tiled load global -> shared of this CTA, completion on an mbarrier.
K3_DEVINL void tma_load_3d(void *dst, const void *map, uint64_t *bar, int32_t x, int32_t y, int32_t z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

K3_DEVINL float sum8(const uint32_t *r) {
    return ((__uint_as_float(r[0]) + __uint_as_float(r[1])) + (__uint_as_float(r[2]) + __uint_as_float(r[3]))) +
           ((__uint_as_float(r[4]) + __uint_as_float(r[5])) + (__uint_as_float(r[6]) + __uint_as_float(r[7])));
}

struct Mx4Args {
    const uint32_t *offsets;             // [groups+1]
    k3_group_parts parts;
    const uint32_t *index;               // term row block of product row r (null: r itself)
    const uint8_t *sfb;                  // term scales [term rows, K/32]
    uint16_t *out;                       // bf16 [rows, out_width] (may be null in gate/up mode)
    uint8_t *act_terms, *act_sf;         // gate/up mode: E2M1 terms [act rows * 8, w_rows / 2] and scales [.., w_rows / 32]
    bool act_by_group;                   // an activation row's place: 16 per group of this kernel, or the product row
    uint32_t groups, w_rows, k, out_width, m_items;
    uint32_t *item_counter;              // zero before the launch
    int activation;
    float beta, linear_beta;
};

struct Mx4Maps {
    CUtensorMap a0, a1;                  // packed weights as bytes [rows, K/2]
    CUtensorMap b;                       // E2M1 terms: 128 bytes of K x term rows x K/256
    CUtensorMap sfa0, sfa1;              // weight block scales [rows, K/32]
};

struct Item {
    uint32_t group, row_start, rows_valid, m_item;
    uint32_t act_row;                    // where the activation rows start
};

// Item w -> (group, weight tile); prefix[g] = groups this kernel takes before group g.
K3_DEVINL Item decode_item(uint32_t w, const uint32_t *prefix, const Mx4Args &a) {
    Item it;
    const uint32_t n = w / a.m_items;
    uint32_t lo = 0, hi = a.groups;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= n) lo = mid; else hi = mid;
    }
    it.group = lo;
    it.m_item = w - n * a.m_items;
    it.row_start = a.offsets[lo];
    it.rows_valid = a.offsets[lo + 1u] - it.row_start;
    it.act_row = a.act_by_group ? n * kTileRows : it.row_start;
    return it;
}

// Accumulator columns [0, 256): a tile of at most 8 rows (N <= 64) takes one of two halves, so
// that its MMAs run while the epilogue still reads the item before; a larger one takes both.
struct AccBuffers {
    uint32_t use0 = 0u, use1 = 0u, turn = 0u;
    __device__ uint32_t uses(uint32_t b) const { return b == 0u ? use0 : use1; }
    __device__ uint32_t first(bool small) const { return small ? turn : 0u; }
    __device__ uint32_t column(bool small, uint32_t b0, uint32_t tile) const {
        return small ? b0 * 128u + tile * 64u : tile * 128u;
    }
    __device__ void advance(bool small, uint32_t b0) {
        if (small) {
            if (b0 == 0u) use0++; else use1++;
            turn ^= 1u;
        } else {
            use0++;
            use1++;
            turn = 0u;
        }
    }
};

template <bool kAct>
__global__ void __launch_bounds__(kThreads, 1)
grouped_mx4_kernel(const __grid_constant__ Mx4Maps maps, Mx4Args a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char *b_smem = base + kStages * kStageBytes;
    unsigned char *sf_smem = b_smem + kBSlots * kBSlotBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sf_smem + kSfSlots * kSfSlotBytes);
    uint64_t *full = bars, *empty = full + kStages;
    uint64_t *sf_full = empty + kStages, *sf_empty = sf_full + kSfBatches;
    uint64_t *sfs_full = sf_empty + kSfBatches, *sfs_empty = sfs_full + kSfSlots;
    uint64_t *acc_full = sfs_empty + kSfSlots, *acc_empty = acc_full + 2;
    uint64_t *item_full = acc_empty + 2, *item_empty = item_full + kItemSlots;
    uint64_t *b_full = item_empty + kItemSlots, *b_empty = b_full + kBSlots;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(b_empty + kBSlots);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    uint32_t *total_items_s = tmem_slot + 2;
    volatile uint32_t *item_box = tmem_slot + 3;           // [kItemSlots]
    uint32_t *prefix = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(bars) + kBarBytes);
    const uint32_t warp = warp_index(), lane = threadIdx.x % kWarp;
    const uint32_t steps = a.k / KS;                       // even: K is a multiple of 512
    const uint32_t tile_rows = kAct ? BM : 2u * BM;        // weight rows one item advances

    if (threadIdx.x == 0) {
        *abort_flag = 0u;
        for (uint32_t s = 0; s < kStages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 2);                       // both MMA issuers release a stage
        }
        for (uint32_t s = 0; s < kBSlots; s++) {
            mbar_init(&b_full[s], 1);
            mbar_init(&b_empty[s], 2);
        }
        for (uint32_t b = 0; b < kSfBatches; b++) {
            mbar_init(&sf_full[b], 4);
            mbar_init(&sf_empty[b], 2);
        }
        for (uint32_t b = 0; b < kSfSlots; b++) {
            mbar_init(&sfs_full[b], 1);
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
    pdl_wait();
    pdl_trigger();                                         // the next kernel's blocks fit only when this one's leave
    {   // exclusive prefix of the groups this kernel takes (<= 1024 groups)
        __shared__ uint32_t warp_tot[kThreads / kWarp];
        uint32_t v[2], incl[2], run = 0;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t g = threadIdx.x * 2u + j;
            const uint32_t n = g < a.groups ? a.offsets[g + 1u] - a.offsets[g] : 0u;
            const uint32_t whole = a.parts.table != nullptr && g < a.groups ? max(a.parts.table[g], n) : n;
            v[j] = n != 0u && whole <= kTileRows ? 1u : 0u;
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

    // Reader side of the item mailbox: the n-th call (of one thread, or of a warp) returns
    // the n-th item this CTA drew.
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
    auto next_item_warp = [&]() -> uint32_t {
        uint32_t w = kNoItem;
        if (lane == 0) w = next_item();
        return __shfl_sync(0xffffffffu, w, 0);
    };

    if (warp == 0) {
        // ================================ TMA producer: weights and their scales; draws the items
        if (elect_one()) {
            prefetch_tensormap(&maps.a0);
            prefetch_tensormap(&maps.a1);
            prefetch_tensormap(&maps.sfa0);
            prefetch_tensormap(&maps.sfa1);
            const uint64_t stream_once = l2_policy_evict_first();
            uint32_t s = 0, ph = 0, ss = 0, ssph = 0, seq = 0;
            bool ok = true;
            uint32_t w = atomicAdd(a.item_counter, 1u);
            while (ok) {
                const uint32_t slot = seq % kItemSlots, parity = (seq / kItemSlots) & 1u;
                seq++;
                if (!mbar_wait(&item_empty[slot], parity ^ 1u, abort_flag)) break;
                const bool valid = w < total_items;
                item_box[slot] = valid ? w : kNoItem;
                mbar_arrive(&item_full[slot]);
                if (!valid) break;
                const Item it = decode_item(w, prefix, a);
                w = atomicAdd(a.item_counter, 1u);         // the next draw travels while this item streams
                const int32_t y0 = (int32_t)(it.group * a.w_rows + it.m_item * tile_rows);
                const int32_t y1 = kAct ? y0 : y0 + (int32_t)BM;
                for (uint32_t st = 0; st < steps; st++) {
                    if ((st & 1u) == 0u) {                 // scales, two stages at a time
                        if (!mbar_wait(&sfs_empty[ss], ssph ^ 1u, abort_flag)) { ok = false; break; }
                        unsigned char *sf = sf_smem + ss * kSfSlotBytes;
                        mbar_arrive_expect_tx(&sfs_full[ss], 2u * kSfKind);
                        tma_load_2d(sf, &maps.sfa0, &sfs_full[ss], (int32_t)(st * 8u), y0);
                        tma_load_2d(sf + kSfKind, &maps.sfa1, &sfs_full[ss], (int32_t)(st * 8u), y1);
                        if (++ss == kSfSlots) { ss = 0; ssph ^= 1u; }
                    }
                    if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
                    unsigned char *dst = base + s * kStageBytes;
                    const int32_t x = (int32_t)(st * 128u);
                    mbar_arrive_expect_tx(&full[s], 2u * kATile);
                    tma_load_2d_hint(dst, &maps.a0, &full[s], x, y0, stream_once);
                    tma_load_2d_hint(dst + kATile, &maps.a1, &full[s], x, y1, stream_once);
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 2) {
        // ================================ TMA producer: token terms; lane i brings row i of the tile
        if (lane == 0) prefetch_tensormap(&maps.b);
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (uint32_t w = next_item_warp(); ok && w != kNoItem; w = next_item_warp()) {
            const Item it = decode_item(w, prefix, a);
            const bool mine = lane < it.rows_valid;
            const uint32_t row = (kAct ? it.row_start : it.act_row) + lane;
            const int32_t y = mine ? (int32_t)(kTerms * (kAct && a.index ? a.index[row] : row)) : 0;
            for (uint32_t st = 0; st < steps; st += 2u) {
                if (lane == 0) {
                    ok = mbar_wait(&b_empty[s], ph ^ 1u, abort_flag);
                    if (ok) mbar_arrive_expect_tx(&b_full[s], it.rows_valid * 2u * kBAtom);
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1u : 0u, 0) != 0u;
                if (!ok) break;
                if (mine)
                    tma_load_3d(b_smem + s * kBSlotBytes + lane * 2u * kBAtom, &maps.b, &b_full[s], 0, y, (int32_t)st);
                if (++s == kBSlots) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == 1 || warp == 3) {
        // ==================================================== MMA issuers, one per weight tile
        if (elect_one()) {
            const uint32_t q = warp == 1 ? 0u : 1u;
            uint32_t s = 0, ph = 0, bs = 0, bph = 0, sb = 0, sph = 0;
            AccBuffers acc;
            bool ok = true;
            for (uint32_t w = next_item(); ok && w != kNoItem; w = next_item()) {
                const Item it = decode_item(w, prefix, a);
                // columns of a missing last row (odd counts) multiply whatever lies there; nothing reads them
                const uint32_t n = (kTerms * it.rows_valid + 15u) & ~15u;
                const uint32_t idesc[2] = {make_idesc_mx4(n, 0u), make_idesc_mx4(n, 2u)};
                const bool small = it.rows_valid <= 8u;
                const uint32_t b0 = acc.first(small);
                if (!mbar_wait(&acc_empty[b0], (acc.uses(b0) & 1u) ^ 1u, abort_flag) ||
                    (!small && !mbar_wait(&acc_empty[1], (acc.use1 & 1u) ^ 1u, abort_flag))) {
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + acc.column(small, b0, q);
                const uint32_t sfa_col = tmem + (q == 0u ? kSfa0Col : kSfa1Col);
                for (uint32_t st = 0; st < steps; st++) {
                    if (!mbar_wait(&full[s], ph, abort_flag) ||
                        ((st & 1u) == 0u && (!mbar_wait(&b_full[bs], bph, abort_flag) ||
                                             !mbar_wait(&sf_full[sb], sph, abort_flag)))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    unsigned char *src = base + s * kStageBytes;
                    const uint64_t da = make_desc_sw128(smem_u32(src + q * kATile));
                    const uint64_t db = make_desc_sw128_pairs(smem_u32(b_smem + bs * kBSlotBytes + (st & 1u) * kBAtom));
#pragma unroll
                    for (uint32_t j = 0; j < 4u; j++) {    // K blocks of 64 inside the stage
                        // a batch column group holds 128 K; MMA j takes scale bytes 2 (j & 1), 2 (j & 1) + 1
                        const uint32_t sfs = sb * 16u + (2u * (st & 1u) + (j >> 1)) * 4u;
                        mma_mx4(d, da + 2u * j, db + 2u * j, idesc[j & 1u], sfa_col + sfs, tmem + kSfbCol + sfs,
                                (st | j) != 0u ? 1u : 0u);
                    }
                    mma_commit(&empty[s]);
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                    if ((st & 1u) == 1u) {
                        mma_commit(&b_empty[bs]);
                        if (++bs == kBSlots) { bs = 0; bph ^= 1u; }
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
        // ================== scale writers: shared memory -> tensor memory (see k3_grouped_mx.cu)
        const uint32_t quad = warp & 3u;
        const uint32_t lane_base = (32u * quad) << 16;
        uint32_t sb = 0, sph = 0, ss = 0, ssph = 0;
        bool ok = true;
        for (uint32_t w = next_item_warp(); ok && w != kNoItem; w = next_item_warp()) {
            const Item it = decode_item(w, prefix, a);
            // this lane's term rows 32 c + lane: term lane % 8 of token row 4 c + lane / 8 (a row past
            // the tile's end repeats row 0: those accumulator columns are not read)
            const uint4 *term_sf[4];
            uint4 vb[4];
#pragma unroll
            for (uint32_t c = 0; c < 4u; c++) {
                const uint32_t i = 4u * c + lane / 8u;
                const uint32_t row = (kAct ? it.row_start : it.act_row) + (i < it.rows_valid ? i : 0u);
                const uint64_t term = (uint64_t)kTerms * (kAct && a.index ? a.index[row] : row) + lane % 8u;
                term_sf[c] = reinterpret_cast<const uint4 *>(a.sfb + term * (a.k / 32u));
            }
#pragma unroll
            for (uint32_t c = 0; c < 4u; c++) vb[c] = 4u * c < it.rows_valid ? *term_sf[c] : make_uint4(0u, 0u, 0u, 0u);
            for (uint32_t st = 0; st < steps; st += 2u) {
                if (!mbar_wait(&sfs_full[ss], ssph, abort_flag)) { ok = false; break; }
                const unsigned char *src = sf_smem + ss * kSfSlotBytes;
                uint4 v[3][4];
#pragma unroll
                for (uint32_t t = 0; t < 2u; t++)
#pragma unroll
                    for (uint32_t c = 0; c < 4u; c++)
                        v[t][c] = *reinterpret_cast<const uint4 *>(src + t * kSfKind + (32u * c + lane) * 16u);
#pragma unroll
                for (uint32_t c = 0; c < 4u; c++) {
                    v[2][c] = vb[c];
                    if (4u * c < it.rows_valid && st + 2u < steps) vb[c] = *++term_sf[c];   // two stages ahead
                }
                if (!mbar_wait(&sf_empty[sb], sph ^ 1u, abort_flag)) { ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (uint32_t t = 0; t < 3u; t++) {
                    const uint32_t cols[16] = {v[t][0].x, v[t][1].x, v[t][2].x, v[t][3].x,
                                               v[t][0].y, v[t][1].y, v[t][2].y, v[t][3].y,
                                               v[t][0].z, v[t][1].z, v[t][2].z, v[t][3].z,
                                               v[t][0].w, v[t][1].w, v[t][2].w, v[t][3].w};
                    tmem_st_32x16(tmem + lane_base + (t == 0 ? kSfa0Col : t == 1 ? kSfa1Col : kSfbCol) + sb * 16u, cols);
                }
                // only now: the stores above consumed every loaded register
                __syncwarp();
                if (lane == 0) mbar_arrive(&sfs_empty[ss]);
                if (++ss == kSfSlots) { ss = 0; ssph ^= 1u; }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sf_full[sb]);
                if (++sb == kSfBatches) { sb = 0; sph ^= 1u; }
            }
        }
    } else {
        // ======================================================== epilogue
        // Quadrant = warp % 4 (tensor-memory lanes); four token rows (32 columns) per warp, their
        // activations and term splits interleaved: one row after the other in eight warps, the
        // epilogue and not the stream bounded the gate/up launch at the latent shape (SiTU, K = 3584:
        // a 1021-token prompt 4.47 -> 4.2 ms).
        const uint32_t quad = warp & 3u, r0 = 4u * ((warp - 8u) >> 2);
        const uint32_t m = 32u * quad + lane;              // weight row inside the tile
        AccBuffers acc;
        for (uint32_t w = next_item_warp(); w != kNoItem; w = next_item_warp()) {
            const Item it = decode_item(w, prefix, a);
            const bool small = it.rows_valid <= 8u;
            const uint32_t b0 = acc.first(small);
            if (!mbar_wait(&acc_full[b0], acc.uses(b0) & 1u, abort_flag) ||
                (!small && !mbar_wait(&acc_full[1], acc.use1 & 1u, abort_flag))) {
                break;
            }
            tc_fence_after();
            const uint32_t t0 = tmem + ((32u * quad) << 16) + acc.column(small, b0, 0u);
            const uint32_t t1 = tmem + ((32u * quad) << 16) + acc.column(small, b0, 1u);
            acc.advance(small, b0);
            const uint32_t col0 = it.m_item * tile_rows + m, col1 = kAct ? col0 : col0 + BM;
            float v0[4], v1[4];
            if (r0 < it.rows_valid) {
#pragma unroll
                for (uint32_t c = 0; c < 2u; c++) {
                    uint32_t q0[16], q1[16];
                    tmem_ld_32x16(t0 + 8u * r0 + 16u * c, q0);
                    tmem_ld_32x16(t1 + 8u * r0 + 16u * c, q1);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t i = 0; i < 2u; i++) {
                        v0[2u * c + i] = sum8(q0 + 8u * i);
                        v1[2u * c + i] = sum8(q1 + 8u * i);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&acc_empty[b0]);
                if (!small) mbar_arrive(&acc_empty[1]);
            }
            if (r0 >= it.rows_valid) continue;
            const uint32_t n = min(4u, it.rows_valid - r0);
            const uint64_t row = it.row_start + r0;
            if (!kAct) {
#pragma unroll
                for (uint32_t i = 0; i < 4u; i++) {
                    if (i >= n) break;
                    a.out[(row + i) * a.out_width + col0] = float_to_bf16_bits(v0[i]);
                    a.out[(row + i) * a.out_width + col1] = float_to_bf16_bits(v1[i]);
                }
                continue;
            }
            float rest[4];                                 // what the terms so far leave of the activation
#pragma unroll
            for (uint32_t i = 0; i < 4u; i++) {
                // gate and up are rounded to bf16 before the activation
                const float g = bf16_bits_to_float(float_to_bf16_bits(v0[i]));
                const float u = bf16_bits_to_float(float_to_bf16_bits(v1[i]));
                const uint16_t bits = float_to_bf16_bits(activation(g, u, a.activation, a.beta, a.linear_beta));
                if (a.out != nullptr && i < n) a.out[(row + i) * a.out_width + col0] = bits;
                rest[i] = i < n ? bf16_bits_to_float(bits) : 0.f;
            }
            // eight E2M1 terms of the four rows' 32-column blocks (split_block_e2m1); a lane keeps the
            // packed word it stores: lane 8 w + j the columns 8 w .. 8 w + 7 of term j
            uint32_t word[4] = {0u, 0u, 0u, 0u}, scale[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (uint32_t j = 0; j < kTerms; j++) {
#pragma unroll
                for (uint32_t i = 0; i < 4u; i++) {
                    const uint32_t mx = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(rest[i])));
                    const uint32_t be = mx >> 23;
                    const bool none = be < 4u || be == 0xffu;
                    const uint32_t sb = be == 0xffu ? 255u : none ? 127u : be - 2u;     // 255: E8M0's NaN
                    uint32_t code = 0u;
                    if (!none) {                           // uniform across the warp
                        const float scaled = rest[i] * __uint_as_float((254u - sb) << 23);
                        code = (uint32_t)__nv_cvt_float_to_fp4(scaled, __NV_E2M1, cudaRoundNearest) & 0xfu;
                        const float back =
                            __half2float(__half(__nv_cvt_fp4_to_halfraw((__nv_fp4_storage_t)code, __NV_E2M1)));
                        rest[i] -= back * __uint_as_float(sb << 23);
                    }
                    uint32_t v = code << (4u * (lane & 7u));
                    v |= __shfl_xor_sync(0xffffffffu, v, 1);
                    v |= __shfl_xor_sync(0xffffffffu, v, 2);
                    v |= __shfl_xor_sync(0xffffffffu, v, 4);
                    if ((lane & 7u) == j) word[i] = v;
                    if (lane == j) scale[i] = sb;
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < 4u; i++) {
                if (i >= n) break;
                const uint64_t term = (uint64_t)(it.act_row + r0 + i) * kTerms;
                *reinterpret_cast<uint32_t *>(a.act_terms + (term + (lane & 7u)) * (a.w_rows / 2u) + (col0 & ~31u) / 2u +
                                              4u * (lane >> 3)) = word[i];
                if (lane < kTerms) a.act_sf[(term + lane) * (a.w_rows / 32u) + col0 / 32u] = (uint8_t)scale[i];
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag != 0u) atomicExch(&g_mx4_status, 1u);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// bf16 rows -> E2M1 terms and block scales: four lanes share a block of 32 columns (8 each), a
// warp converts 256 columns per pass and stores each term as 128 contiguous bytes.  The same
// values as split_block_e2m1 (one element per lane), a sixth of its instructions.  With `ids`, the
// experts of row r are ids[r * top_k ..], and a row none of whose experts is a group of this kernel
// is skipped.
__global__ void __launch_bounds__(256)
term_rows_kernel(uint8_t *__restrict__ terms, uint8_t *__restrict__ sf, const uint16_t *x,
                 uint32_t *__restrict__ counters, const uint32_t *ids,
                 const uint32_t *offsets, uint32_t top_k, uint32_t rows, uint32_t k) {
    pdl_wait();
    pdl_trigger();
    if (blockIdx.x == 0 && threadIdx.x < 64u) counters[threadIdx.x] = 0u;      // of the product launches
    const uint32_t lane = threadIdx.x % kWarp, passes = k / 256u;
    const uint64_t warps = (uint64_t)(gridDim.x * blockDim.x) / kWarp, jobs = (uint64_t)rows * passes;
    for (uint64_t job = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp; job < jobs; job += warps) {
        const uint32_t r = (uint32_t)(job / passes);
        if (ids != nullptr) {
            bool mine = false;
            if (lane < top_k) {
                const uint32_t e = ids[(uint64_t)r * top_k + lane];
                mine = offsets[e + 1u] - offsets[e] <= kTileRows;
            }
            if (!__any_sync(0xffffffffu, mine)) continue;
        }
        const uint32_t c = (uint32_t)(job % passes) * 256u + lane * 8u;
        const uint4 raw = *reinterpret_cast<const uint4 *>(x + (uint64_t)r * k + c);
        const uint32_t wv[4] = {raw.x, raw.y, raw.z, raw.w};
        float v[8];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[2 * q] = bf16_lo(wv[q]);
            v[2 * q + 1] = bf16_hi(wv[q]);
        }
#pragma unroll
        for (uint32_t j = 0; j < kTerms; j++) {
            uint32_t mx = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) mx = max(mx, __float_as_uint(fabsf(v[q])));
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const uint32_t be = mx >> 23;
            const bool none = be < 4u || be == 0xffu;      // nothing left in this block, or nothing finite
            // largest magnitude / 2^(sb - 127) in [4, 8); a block with an infinity or NaN gets the
            // scale 255, E8M0's NaN, so that its row's results are NaN
            const uint32_t sb = be == 0xffu ? 255u : none ? 127u : be - 2u;
            const float down = none ? 0.f : __uint_as_float((254u - sb) << 23), up = __uint_as_float(sb << 23);
            uint32_t word = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float2 s = none ? make_float2(0.f, 0.f) : make_float2(v[2 * q] * down, v[2 * q + 1] * down);
                const uint32_t p = (uint32_t)__nv_cvt_float2_to_fp4x2(s, __NV_E2M1, cudaRoundNearest) & 0xffu;
                const float2 back = __half22float2(__half2(__nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)p, __NV_E2M1)));
                v[2 * q] -= back.x * up;
                v[2 * q + 1] -= back.y * up;
                word |= p << (8 * q);
            }
            const uint64_t out_row = (uint64_t)r * kTerms + j;
            *reinterpret_cast<uint32_t *>(terms + out_row * (k / 2u) + c / 2u) = word;
            if ((lane & 3u) == 0u) sf[out_row * (k / 32u) + c / 32u] = (uint8_t)sb;
        }
    }
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

bool map_bytes(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t row_bytes, uint32_t box_bytes, uint32_t box_rows,
               CUtensorMapSwizzle swizzle) {
    auto fn = encode_fn();
    if (!fn || (((uintptr_t)ptr) & 15u) != 0 || row_bytes % 16u != 0) return false;
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_bytes, box_rows};
    const cuuint32_t es[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// terms: 128 bytes (256 K) x term rows x K/256, box = one token's 8 rows of two 256-K chunks, each
// chunk one swizzle atom
bool map_terms(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t row_bytes) {
    auto fn = encode_fn();
    if (!fn || (((uintptr_t)ptr) & 15u) != 0) return false;
    const cuuint64_t dims[3] = {128, rows, row_bytes / 128u};
    const cuuint64_t strides[2] = {row_bytes, 128};
    const cuuint32_t box[3] = {128, kTerms, 2};
    const cuuint32_t es[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(ptr), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Operands {
    const void *a0, *a1, *sfa0, *sfa1;   // packed weights of tile 0 / tile 1, their scale tables
    const uint8_t *terms, *sfb;          // terms and scales, kTerms rows per token row
    uint32_t term_rows;
};

// Tensor maps depend only on the tables, the term buffers and the shape: the sets of the most
// recent calls are kept; when the table is full it starts over.
struct MapKey {
    int device, mode;
    const void *p[5];
    uint32_t dims[4];
    bool operator<(const MapKey &o) const {
        if (device != o.device) return device < o.device;
        if (mode != o.mode) return mode < o.mode;
        const int c = memcmp(p, o.p, sizeof(p));
        return c != 0 ? c < 0 : memcmp(dims, o.dims, sizeof(dims)) < 0;
    }
};

template <bool kAct>
bool launch(const Operands &op, Mx4Args args, cudaStream_t stream) {
    args.sfb = op.sfb;
    constexpr size_t kCachedSets = 256;
    static std::mutex map_lock;
    static std::map<MapKey, Mx4Maps> cached;
    MapKey key{};
    key.device = current_device();
    key.mode = kAct;
    const void *ptrs[5] = {op.a0, op.a1, op.sfa0, op.sfa1, op.terms};
    memcpy(key.p, ptrs, sizeof(ptrs));
    key.dims[0] = args.groups; key.dims[1] = args.w_rows; key.dims[2] = args.k; key.dims[3] = op.term_rows;
    Mx4Maps maps;
    {
        std::lock_guard<std::mutex> guard(map_lock);
        auto it = cached.find(key);
        if (it == cached.end()) {
            const uint64_t w_total = (uint64_t)args.groups * args.w_rows, kb = args.k / 32u;
            const auto sw = CU_TENSOR_MAP_SWIZZLE_128B, none = CU_TENSOR_MAP_SWIZZLE_NONE;
            if (!map_bytes(&maps.a0, op.a0, w_total, args.k / 2u, 128, BM, sw) ||
                !map_bytes(&maps.a1, op.a1, w_total, args.k / 2u, 128, BM, sw) ||
                !map_terms(&maps.b, op.terms, op.term_rows, args.k / 2u) ||
                !map_bytes(&maps.sfa0, op.sfa0, w_total, kb, 16, BM, none) ||
                !map_bytes(&maps.sfa1, op.sfa1, w_total, kb, 16, BM, none)) {
                return false;
            }
            if (cached.size() >= kCachedSets) cached.clear();
            cached.emplace(key, maps);
        } else {
            maps = it->second;
        }
    }
    if (!set_max_dynamic_smem((const void *)grouped_mx4_kernel<kAct>, kSmemBytes)) return false;
    return launch_chained(grouped_mx4_kernel<kAct>, sm_count(), kThreads, kSmemBytes, stream, maps, args);
}

struct Scratch {
    uint8_t *x_terms, *x_sf;             // per source row
    uint8_t *a_terms, *a_sf;             // activation, per activation row
    uint32_t act_rows;
    bool act_by_group;
    size_t total;
};

Scratch carve_scratch(const k3_moe_layer_desc *d, uint32_t rows, uint32_t source_rows, void *workspace) {
    const size_t H = d->hidden, I = d->expert_hidden;
    uint8_t *p = (uint8_t *)(((uintptr_t)workspace + 255u) & ~(uintptr_t)255u);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        uint8_t *q = p + off;
        off += (bytes + 255u) & ~(size_t)255u;
        return q;
    };
    Scratch s{};
    s.x_terms = take((size_t)source_rows * kTerms * (H / 2u));
    s.x_sf = take((size_t)source_rows * kTerms * (H / 32u));
    // A row's terms are 4.25 bytes per column and at most kTileRows rows of a group come here, so
    // with many rows the activation is laid out by group: 125 MB instead of 2.3 GB for the
    // 262144 rows of 16384 tokens at 896 experts.  With few rows the product rows take less.
    s.act_by_group = (uint64_t)d->local_expert_count * kTileRows < rows;
    s.act_rows = s.act_by_group ? d->local_expert_count * kTileRows : rows;
    s.a_terms = take((size_t)s.act_rows * kTerms * (I / 2u));
    s.a_sf = take((size_t)s.act_rows * kTerms * (I / 32u));
    s.total = off + 256u;
    return s;
}

}  // namespace

uint32_t k3_grouped_mx4_status() {
    uint32_t v = 0xffffffffu;
    if (cudaMemcpyFromSymbol(&v, g_mx4_status, sizeof(v)) != cudaSuccess) (void)cudaGetLastError();
    return v;
}

bool k3_grouped_mx4_status_clear() {
    const uint32_t zero = 0u;
    if (cudaMemcpyToSymbol(g_mx4_status, &zero, sizeof(zero)) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return true;
}

size_t k3_grouped_mx4_workspace_bytes(const k3_moe_layer_desc *d, uint32_t rows, uint32_t source_rows) {
    return carve_scratch(d, rows, source_rows, nullptr).total;
}

bool k3_grouped_mx4_terms(const k3_moe_layer_desc *d, const void *rows_in, uint32_t source_rows, uint32_t rows,
                          const void *ids, const void *offsets, void *workspace, uint32_t *counters,
                          cudaStream_t stream) {
    const Scratch s = carve_scratch(d, rows, source_rows, workspace);
    const uint64_t jobs = (uint64_t)source_rows * (d->hidden / 256u);
    return launch_chained(term_rows_kernel, (uint32_t)std::min<uint64_t>((jobs + 7u) / 8u, (uint64_t)sm_count() * 16u), 256, 0,
                          stream, s.x_terms, s.x_sf, (const uint16_t *)rows_in, counters, (const uint32_t *)ids, (const uint32_t *)offsets,
                          d->top_k, source_rows, d->hidden);
}

bool k3_grouped_mx4_gateup(const k3_moe_layer_desc *d, void *act, const void *index, uint32_t source_rows,
                           const void *offsets, uint32_t rows, void *workspace, uint32_t *counter,
                           k3_group_parts parts, cudaStream_t stream) {
    const Scratch s = carve_scratch(d, rows, source_rows, workspace);
    Mx4Args a{};
    a.offsets = (const uint32_t *)offsets;
    a.parts = parts;
    a.index = (const uint32_t *)index;
    a.groups = d->local_expert_count;
    a.activation = d->activation;
    a.beta = d->beta;
    a.linear_beta = d->linear_beta;
    a.item_counter = counter;
    a.out = (uint16_t *)act;
    a.act_terms = s.a_terms;
    a.act_sf = s.a_sf;
    a.act_by_group = s.act_by_group;
    a.w_rows = d->expert_hidden;
    a.k = d->hidden;
    a.out_width = d->expert_hidden;
    a.m_items = d->expert_hidden / BM;
    const Operands op{d->w1_packed, d->w3_packed, d->w1_scales, d->w3_scales, s.x_terms, s.x_sf, source_rows * kTerms};
    return launch<true>(op, a, stream);
}

bool k3_grouped_mx4_down(const k3_moe_layer_desc *d, void *rows_out, const void *offsets, uint32_t rows,
                         uint32_t source_rows, void *workspace, uint32_t *counter,
                         k3_group_parts parts, cudaStream_t stream) {
    const Scratch s = carve_scratch(d, rows, source_rows, workspace);
    Mx4Args a{};
    a.offsets = (const uint32_t *)offsets;
    a.parts = parts;
    a.groups = d->local_expert_count;
    a.item_counter = counter;
    a.out = (uint16_t *)rows_out;
    a.w_rows = d->hidden;
    a.k = d->expert_hidden;
    a.out_width = d->hidden;
    a.m_items = d->hidden / (2u * BM);
    a.act_by_group = s.act_by_group;
    const Operands op{d->w2_packed, d->w2_packed, d->w2_scales, d->w2_scales, s.a_terms, s.a_sf, s.act_rows * kTerms};
    return launch<false>(op, a, stream);
}
