// MXFP4 rows against any number of bf16 vectors on mma.sync, for the operator entry points
// (one expert matrix per call, no workspace).
//
// Per output: the 32 products of a scale group are summed by two m16n8k16 MMAs from zero in
// fp32 (E2M1 is exact in bf16, the activations stay bf16), the E8M0 scale is applied with one
// fp32 FMA into a running sum - the reference's "dot per group, scale, accumulate"
// (k3_rocm_ops.cu:193-273) - and eight such sums over contiguous eighths of the row are added
// in ascending order.  Nothing of that depends on the number of vectors or on the tile, so
// batch == repeated single-row calls byte for byte.
//
// A warp takes 16 weight rows.  Lane (g, t) = (lane / 4, lane % 4) reads columns 8 t .. 8 t + 7
// of a group: one 32-bit word of row g and of row g + 8 (any 4-byte aligned base), 16 bytes of
// vector g of each 8-vector tile, and these are its MMA fragments as they lie: k slots
// {2t, 2t+1, 2t+8, 2t+9} of the first MMA are columns 8t .. 8t+3, of the second 8t+4 .. 8t+7.
//
#pragma once

#include "k3_common.cuh"

namespace k3 {

constexpr uint32_t kMxSplits = 8;

// Eight E2M1 nibbles (low nibble first) -> four bf16x2 registers.  Low and high byte of the bf16
// codes of 0, .5, 1, 1.5, 2, 3, 4, 6 come from two byte tables (PRMT looks up four at once).
K3_DEVINL void dequant_word_bf16(uint32_t w, uint32_t (&out)[4]) {
    const uint32_t sel = w & 0x77777777u, sel_hi = sel >> 16;
    const uint32_t l03 = __byte_perm(0xC0800000u, 0xC0804000u, sel), l47 = __byte_perm(0xC0800000u, 0xC0804000u, sel_hi);
    uint32_t h03 = __byte_perm(0x3F3F3F00u, 0x40404040u, sel), h47 = __byte_perm(0x3F3F3F00u, 0x40404040u, sel_hi);
    const uint32_t w4 = w << 4;
    h03 |= __byte_perm(w4, w, 0x5140u) & 0x80808080u;
    h47 |= __byte_perm(w4, w, 0x7362u) & 0x80808080u;
    out[0] = __byte_perm(l03, h03, 0x5140u);
    out[1] = __byte_perm(l03, h03, 0x7362u);
    out[2] = __byte_perm(l47, h47, 0x5140u);
    out[3] = __byte_perm(l47, h47, 0x7362u);
}

K3_DEVINL void mma_bf16_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
K3_DEVINL void mma_bf16_add(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Rows and vectors past the end read the last one; their sums are not stored.
struct MxRowPointers {
    const uint32_t *pa, *pb;
    const uint8_t *sa, *sb;
};
K3_DEVINL MxRowPointers mx_row_pointers(const uint8_t *packed, const uint8_t *scales, uint32_t row0, uint32_t rows,
                                        uint32_t k) {
    const uint32_t g = (threadIdx.x % kWarp) >> 2, t = threadIdx.x & 3u;
    const uint32_t row_a = min(row0 + g, rows - 1u), row_b = min(row0 + g + 8u, rows - 1u);
    return {reinterpret_cast<const uint32_t *>(packed + (uint64_t)row_a * (k / 2u)) + t,
            reinterpret_cast<const uint32_t *>(packed + (uint64_t)row_b * (k / 2u)) + t,
            scales + (uint64_t)row_a * (k / 32u), scales + (uint64_t)row_b * (k / 32u)};
}

// One scale group of 16 rows against one 8-vector tile.
K3_DEVINL void mx_group(float (&acc)[4], const uint32_t (&fa)[4], const uint32_t (&fb)[4], const uint4 &xq, float s_a,
                        float s_b) {
    float c[4];
    mma_bf16_zero(c, fa[0], fb[0], fa[1], fb[1], xq.x, xq.y);
    mma_bf16_add(c, fa[2], fb[2], fa[3], fb[3], xq.z, xq.w);
    acc[0] = fmaf(s_a, c[0], acc[0]);
    acc[1] = fmaf(s_a, c[1], acc[1]);
    acc[2] = fmaf(s_b, c[2], acc[2]);
    acc[3] = fmaf(s_b, c[3], acc[3]);
}

// Accumulators of one split and tile -> red[col][16 rows] (columns 2 t and 2 t + 1).
K3_DEVINL void mx_put(float *dst, const float (&acc)[4]) {
    const uint32_t g = (threadIdx.x % kWarp) >> 2, c0 = 2u * (threadIdx.x & 3u);
    dst[c0 * 16u + g] = acc[0];
    dst[(c0 + 1u) * 16u + g] = acc[1];
    dst[c0 * 16u + g + 8u] = acc[2];
    dst[(c0 + 1u) * 16u + g + 8u] = acc[3];
}

// red [row block][split][col][16] -> out: the eight split sums in ascending order.
template <int kCols, int kBlocks, int kThreads>
K3_DEVINL void mx_finish(uint16_t *out, const float *red, uint32_t row_base, uint32_t v0, uint32_t rows,
                         uint32_t vectors) {
    for (uint32_t i = threadIdx.x; i < kBlocks * kCols * 16u; i += kThreads) {
        // row fastest: 16 * kBlocks consecutive rows of one vector are stored together
        const uint32_t r = i % (16u * kBlocks), col = i / (16u * kBlocks);
        const float *src = red + ((size_t)(r / 16u) * kMxSplits * kCols + col) * 16u + (r & 15u);
        float total = src[0];
#pragma unroll
        for (uint32_t s = 1; s < kMxSplits; s++) total += src[(size_t)s * kCols * 16u];
        const uint32_t row = row_base + r, vec = v0 + col;
        if (row < rows && vec < vectors) out[(uint64_t)vec * rows + row] = float_to_bf16_bits(total);
    }
}

// Up to eight vectors: a block owns 16 rows, a warp one of the eight splits, everything straight
// from global memory.  Bound by launch and memory latency (a 3072 x 3584 matrix is 5.8 MB: 0.9 us
// of HBM time; 5.1 us in a chain of them, 8.2 before chained launches).  Through shared memory by
// asynchronous copies it is slower (6.2 us).  kWide: the vectors are 16-byte aligned.
template <bool kWide>
__global__ void __launch_bounds__(32 * kMxSplits)
mxfp4_rows_kernel(uint16_t *__restrict__ out, const uint8_t *packed, const uint8_t *scales,
                  const uint16_t *x, uint32_t vectors, uint32_t rows, uint32_t k) {
    __shared__ float red[kMxSplits * 8u * 16u];
    const uint32_t lane = threadIdx.x % kWarp, split = threadIdx.x / kWarp;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t groups = k / 32u, per = (groups + kMxSplits - 1u) / kMxSplits;
    const uint32_t row0 = blockIdx.x * 16u, v0 = blockIdx.y * 8u;
    if (blockIdx.y == 0 && threadIdx.x == 0) {
        const uint64_t n = min(16u, rows - row0);
        prefetch_l2(packed + (uint64_t)row0 * (k / 2u), n * (k / 2u));
        prefetch_l2(scales + (uint64_t)row0 * groups, n * groups);
    }
    pdl_wait();
    const MxRowPointers p = mx_row_pointers(packed, scales, row0, rows, k);
    const uint16_t *xv = x + (uint64_t)min(v0 + g, vectors - 1u) * k + 8u * t;
    const uint32_t begin = min(groups, split * per), end = min(groups, begin + per);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 7
    for (uint32_t grp = begin; grp < end; grp++) {
        const uint32_t wa = p.pa[4u * grp], wb = p.pb[4u * grp];
        const float s_a = e8m0_to_float(p.sa[grp]), s_b = e8m0_to_float(p.sb[grp]);
        const uint16_t *xp = xv + 32u * grp;
        const uint4 xq = kWide ? *reinterpret_cast<const uint4 *>(xp)
                               : make_uint4(xp[0] | (uint32_t)xp[1] << 16, xp[2] | (uint32_t)xp[3] << 16,
                                            xp[4] | (uint32_t)xp[5] << 16, xp[6] | (uint32_t)xp[7] << 16);
        uint32_t fa[4], fb[4];
        dequant_word_bf16(wa, fa);
        dequant_word_bf16(wb, fb);
        mx_group(acc, fa, fb, xq, s_a, s_b);
    }
    pdl_trigger();
    mx_put(red + (size_t)split * 8u * 16u, acc);
    __syncthreads();
    mx_finish<8, 1, 32 * kMxSplits>(out, red, row0, v0, rows, vectors);
}

// More vectors: kTiles 8-vector tiles x kBlocks 16-row blocks per block.  kTeams teams of kBlocks
// warps take the splits in turn; a team brings its vectors' next two scale groups into shared
// memory (three stages of asynchronous copies, one barrier of the team per stage), so they cross
// from L2 once per kBlocks row blocks.  Read straight from global memory by each warp, they came
// from L2 once per row block.  147 vectors of a 3072 x 3584 matrix: 27 us (387 us in the kernel
// before, which repeated the dequantisation for every two vectors and re-read the vectors).
// Bound by issue: per scale group 34 instructions dequantise, 7 per tile multiply and scale.
template <int kTiles, int kBlocks, int kTeams>
__global__ void __launch_bounds__(32 * kBlocks * kTeams)
mxfp4_tile_kernel(uint16_t *__restrict__ out, const uint8_t *packed, const uint8_t *scales,
                  const uint16_t *x, uint32_t vectors, uint32_t rows, uint32_t k) {
    constexpr uint32_t kCols = 8 * kTiles, kTeamThreads = 32 * kBlocks;
    constexpr uint32_t kStage = kCols * 128u;              // bytes: 64 columns of every vector
    extern __shared__ __align__(128) unsigned char smem_mx[];
    float *red = reinterpret_cast<float *>(smem_mx + kTeams * 3u * kStage);   // [kBlocks][kMxSplits][kCols][16]
    const uint32_t lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t team = warp / kBlocks, rb = warp % kBlocks, tid = threadIdx.x % kTeamThreads;
    const uint32_t groups = k / 32u, per = (groups + kMxSplits - 1u) / kMxSplits;
    const uint32_t row_base = blockIdx.x * kBlocks * 16u, v0 = blockIdx.y * kCols;
    if (blockIdx.y == 0 && team == 0 && lane == 0 && row_base + rb * 16u < rows) {
        const uint64_t first = row_base + rb * 16u, n = min(16u, rows - (uint32_t)first);
        prefetch_l2(packed + first * (k / 2u), n * (k / 2u));
    }
    pdl_wait();
    const MxRowPointers p = mx_row_pointers(packed, scales, row_base + rb * 16u, rows, k);
    unsigned char *ring = smem_mx + team * 3u * kStage;
    // this thread's 16-byte chunks of a stage: chunk tid % 8 of vectors tid / 8 + kTeamThreads / 8 * m
    constexpr uint32_t kCopies = (kCols * 8u + kTeamThreads - 1u) / kTeamThreads;
    const uint32_t chunk = tid & 7u, copy_row = tid >> 3;
    const uint16_t *src0[kCopies];
#pragma unroll
    for (uint32_t m = 0; m < kCopies; m++)
        src0[m] = x + (uint64_t)min(v0 + copy_row + kTeamThreads / 8u * m, vectors - 1u) * k + 8u * chunk;
    const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(ring) + copy_row * 128u + ((chunk ^ (copy_row & 1u) * 4u) * 16u);
    const uint32_t lds0 = g * 128u + ((t ^ (g & 1u) * 4u) * 16u), lds1 = lds0 ^ 64u;

    for (uint32_t split = team; split < kMxSplits; split += kTeams) {
        const uint32_t begin = min(groups, split * per), end = min(groups, begin + per);
        const uint32_t stages = (end - begin + 1u) / 2u;
        uint32_t fetched = 0, fetch_slot = 0;
        auto fetch = [&]() {
            if (fetched < stages) {
                // a half stage past the split's end is filled with zeros
                const uint32_t grp = begin + 2u * fetched, bytes = grp + chunk / 4u < end ? 16u : 0u;
#pragma unroll
                for (uint32_t m = 0; m < kCopies; m++) {
                    if (kCols * 8u % kTeamThreads != 0u && tid + kTeamThreads * m >= kCols * 8u) break;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                     dst0 + fetch_slot * kStage + kTeamThreads * 16u * m),
                                 "l"(bytes ? src0[m] + 32u * grp : x), "r"(bytes));
                }
                fetched++;
                fetch_slot = fetch_slot == 2u ? 0u : fetch_slot + 1u;
            }
            asm volatile("cp.async.commit_group;");
        };
        // the barrier of the previous split's last stage does not order its reads of slots 0 and 1
        asm volatile("bar.sync %0, %1;" ::"r"(team + 1u), "r"(kTeamThreads) : "memory");
        fetch();
        fetch();
        float acc[kTiles][4];
#pragma unroll
        for (int n = 0; n < kTiles; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[n][i] = 0.f;
        uint32_t wa[2], wb[2], ea[2], eb[2];               // weights and scales of the next stage
        const uint32_t *qa = p.pa + 4u * begin, *qb = p.pb + 4u * begin;
        const uint8_t *ca = p.sa + begin, *cb = p.sb + begin;
        uint32_t left = end - begin;                       // groups from the next stage on
        auto weights = [&]() {
#pragma unroll
            for (uint32_t j = 0; j < 2u; j++) {
                // zero weights and a finite scale where a split ends in half a stage
                const bool there = j < left;
                wa[j] = there ? qa[4u * j] : 0u;
                wb[j] = there ? qb[4u * j] : 0u;
                ea[j] = there ? ca[j] : 0u;
                eb[j] = there ? cb[j] : 0u;
            }
            qa += 8;
            qb += 8;
            ca += 2;
            cb += 2;
            left -= min(left, 2u);
        };
        weights();
        const unsigned char *src = ring;
        for (uint32_t stage = 0; stage < stages; stage++) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            asm volatile("bar.sync %0, %1;" ::"r"(team + 1u), "r"(kTeamThreads) : "memory");
            fetch();
            uint32_t fa[2][4], fb[2][4];
            float s_a[2], s_b[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                dequant_word_bf16(wa[j], fa[j]);
                dequant_word_bf16(wb[j], fb[j]);
                s_a[j] = e8m0_to_float(ea[j]);
                s_b[j] = e8m0_to_float(eb[j]);
            }
            weights();
#pragma unroll
            for (uint32_t j = 0; j < 2u; j++) {
#pragma unroll
                for (int n = 0; n < kTiles; n++) {
                    const uint4 xq = *reinterpret_cast<const uint4 *>(src + (j ? lds1 : lds0) + n * 1024);
                    mx_group(acc[n], fa[j], fb[j], xq, s_a[j], s_b[j]);
                }
            }
            src = src == ring + 2u * kStage ? ring : src + kStage;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int n = 0; n < kTiles; n++)
            mx_put(red + ((size_t)(rb * kMxSplits + split) * kCols + 8u * n) * 16u, acc[n]);
    }
    pdl_trigger();
    __syncthreads();
    mx_finish<kCols, kBlocks, 32 * kBlocks * kTeams>(out, red, row_base, v0, rows, vectors);
}

template <int kTiles, int kBlocks, int kTeams>
constexpr size_t mxfp4_tile_smem() {
    return (size_t)kTeams * 3u * 8u * kTiles * 128u + (size_t)kBlocks * kMxSplits * 8u * kTiles * 16u * sizeof(float);
}

}  // namespace k3
