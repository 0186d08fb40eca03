// Q8 products of a few token rows (fewer than the tcgen05 path takes) inside the layer: latent
// projections and shared expert of a decode batch.
//
//   out[v, r] = sum_blocks scale[r, block] * sum_{c in block} q[r, c] * x[v, c]
//
// Bound: the table's bytes.  The exact-order kernel of the operator interface
// (k3_exact_gemm.cuh) issues more than an instruction per multiply-add and runs at a fifth of the
// memory rate with 5 rows; here the 32 columns of a scale step go through two m16n8k16 MMAs
// from zero (int8 is exact in bf16, the products are exact, fp32 sums) and one fp32 FMA per
// step applies the scale - the arithmetic of the one-token kernels.  That rounds less than the
// exact-order kernel, which rounds every scaled weight.
//
// A block takes 16 weight rows; its warps share the columns step by step (8 splits, 16 from 4096
// columns on, added in ascending order).  The splits do not depend on the number of rows: a row has
// the same bits in any batch of 1 to 31.  Gate and up go together: half of the warps each, and the
// block applies the activation (one launch instead of three).  A block's table rows are requested
// into L2 before the wait for the kernel in front.  Tables from HBM: 2048 x 7168 with 5 / 24 / 31
// rows 9.6 / 14.6 / 15.5 us (exact order 15.3 / 40 / 50), 7168 x 2048 8.3 / 13.0 / 13.8 (20 / 56 /
// 73), 7168 x 3584 11.9 / 17.0 / 19.2 (30 / 83 / 109); one row 8.1 to 11.9 (6.8 to 12.7).  Against
// 64-bit results the error is that of the final rounding to bf16, as in the exact-order kernel:
// rel-L2 equal to six digits, and as many results on the wrong side of a rounding line (one in 5000).
#include "k3_grouped.h"
#include "k3_mxfp4_rows.cuh"

#include <cuda_fp16.h>

using namespace k3;

namespace {

constexpr uint32_t kRows = 16;

struct Q8FewArgs {
    const int8_t *q[2];
    const void *scales[2];
    const uint16_t *x;
    uint16_t *out, *gate, *up;           // gate, up: where a pair's two products go beside the activation
    uint32_t vectors, rows, columns, block;
    uint32_t per_block;                  // column steps per scale block, and 2^32 / per_block rounded up
    uint32_t reciprocal;                 //   (steps stay below 2^16, so the high word of a product is the quotient)
    int scale_f16, activation;
    float beta, linear_beta;
};

// Two bytes of `word` (by `selector`) as bf16: the low seven bits under the exponent of 128, minus
// 128 or (sign bit set) 256; both exact.
K3_DEVINL uint32_t int8_pair_to_bf16(uint32_t word, uint32_t selector) {
    const uint32_t v = __byte_perm(word, 0x43434343u, selector);       // 0x43, byte, 0x43, byte
    uint32_t r;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(v & 0x437f437fu), "r"(v & 0x43804380u));
    return r;
}
K3_DEVINL void int8_to_bf16(uint2 w, uint32_t (&out)[4]) {
    out[0] = int8_pair_to_bf16(w.x, 0x4140u);
    out[1] = int8_pair_to_bf16(w.x, 0x4342u);
    out[2] = int8_pair_to_bf16(w.y, 0x4140u);
    out[3] = int8_pair_to_bf16(w.y, 0x4342u);
}

// kTiles tiles of eight token rows; kDeep column steps' loads in flight; kSplits warps per table,
// each with kTurns of the kSplits * kTurns splits (step s belongs to split s mod that), so that a
// row's sum has the same order whatever the number of warps.
template <int kTiles, bool kPair, uint32_t kSplits, uint32_t kDeep, uint32_t kTurns>
__global__ void __launch_bounds__(32 * kSplits * (kPair ? 2 : 1))
q8_few_kernel(Q8FewArgs a) {
    constexpr uint32_t kTables = kPair ? 2u : 1u;
    __shared__ float red[kTables * kSplits][kTiles * 8u][kRows];
    const uint32_t lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp, g = lane >> 2, t = lane & 3u;
    const uint32_t split = warp % kSplits, table = warp / kSplits;
    const uint32_t row0 = blockIdx.x * kRows, per_row = a.columns / a.block, steps = a.columns / 32u;
    const int8_t *q = kPair && table != 0u ? a.q[1] : a.q[0];
    const void *scales = kPair && table != 0u ? a.scales[1] : a.scales[0];
    if (lane == 0 && split == 0) prefetch_l2(q + (uint64_t)row0 * a.columns, (uint64_t)min(kRows, a.rows - row0) * a.columns);
    pdl_wait();
    // rows and vectors past the end read the last one; their sums are not stored
    const uint32_t row_a = min(row0 + g, a.rows - 1u), row_b = min(row0 + g + 8u, a.rows - 1u);
    const int8_t *qa = q + (uint64_t)row_a * a.columns + 8u * t, *qb = q + (uint64_t)row_b * a.columns + 8u * t;
    const uint64_t sa = (uint64_t)row_a * per_row, sb = (uint64_t)row_b * per_row;
    auto scale = [&](uint64_t at) {
        return a.scale_f16 ? __half2float(reinterpret_cast<const __half *>(scales)[at])
                           : reinterpret_cast<const float *>(scales)[at];
    };
    const uint16_t *x[kTiles];
#pragma unroll
    for (int n = 0; n < kTiles; n++)
        x[n] = a.x + (uint64_t)min(8u * n + g, a.vectors - 1u) * a.columns + 8u * t;
    // the splits' sums in ascending order: first turn of every warp, then the second
    constexpr uint32_t kThreads = 32u * kSplits * kTables, kMine = (kTiles * 8u * kRows + kThreads - 1u) / kThreads;
    constexpr uint32_t kAll = kSplits * kTurns;
    float sums[kMine][kTables];
#pragma unroll
    for (uint32_t turn = 0; turn < kTurns; turn++) {
        float acc[kTiles][4];
#pragma unroll
        for (int n = 0; n < kTiles; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[n][i] = 0.f;
        for (uint32_t first = split + turn * kSplits; first < steps; first += kAll * kDeep) {
            uint2 wa[kDeep], wb[kDeep];
            float fa[kDeep], fb[kDeep];
            uint4 xq[kDeep][kTiles];
#pragma unroll
            for (uint32_t j = 0; j < kDeep; j++) {
                const uint32_t step = first + kAll * j, c = 32u * step;
                if (step >= steps) break;                                      // uniform across the warp
                wa[j] = *reinterpret_cast<const uint2 *>(qa + c);
                wb[j] = *reinterpret_cast<const uint2 *>(qb + c);
                const uint32_t at = a.per_block == 1u ? step : __umulhi(step, a.reciprocal);
                fa[j] = scale(sa + at);
                fb[j] = scale(sb + at);
#pragma unroll
                for (int n = 0; n < kTiles; n++) xq[j][n] = *reinterpret_cast<const uint4 *>(x[n] + c);
            }
#pragma unroll
            for (uint32_t j = 0; j < kDeep; j++) {
                if (first + kAll * j >= steps) break;
                uint32_t va[4], vb[4];
                int8_to_bf16(wa[j], va);
                int8_to_bf16(wb[j], vb);
#pragma unroll
                for (int n = 0; n < kTiles; n++) mx_group(acc[n], va, vb, xq[j][n], fa[j], fb[j]);
            }
        }
        if (turn + 1u == kTurns) pdl_trigger();
        if (turn != 0u) __syncthreads();
#pragma unroll
        for (int n = 0; n < kTiles; n++) mx_put(&red[warp][8 * n][0], acc[n]);
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < kMine; j++) {
            const uint32_t i = threadIdx.x + j * kThreads, r = i % kRows, v = i / kRows;
            if (i >= kTiles * 8u * kRows) break;
#pragma unroll
            for (uint32_t m = 0; m < kTables; m++) {
                float sum = turn != 0u ? sums[j][m] : red[m * kSplits][v][r];
#pragma unroll
                for (uint32_t s = turn != 0u ? 0u : 1u; s < kSplits; s++) sum += red[m * kSplits + s][v][r];
                sums[j][m] = sum;
            }
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < kMine; j++) {
        const uint32_t i = threadIdx.x + j * kThreads, r = i % kRows, v = i / kRows;
        if (i >= kTiles * 8u * kRows) break;
        const float(&sum)[kTables] = sums[j];
        if (row0 + r >= a.rows || v >= a.vectors) continue;
        const uint64_t at = (uint64_t)v * a.rows + row0 + r;
        uint16_t bits = float_to_bf16_bits(sum[0]);
        if (kPair) {
            const uint16_t up = float_to_bf16_bits(sum[kTables - 1u]);
            a.gate[at] = bits;
            a.up[at] = up;
            bits = float_to_bf16_bits(activation(bf16_bits_to_float(bits), bf16_bits_to_float(up), a.activation, a.beta,
                                                 a.linear_beta));
        }
        a.out[at] = bits;
    }
}

void set_block(Q8FewArgs &a, uint32_t block) {
    a.block = block;
    a.per_block = block / 32u;
    a.reciprocal = a.per_block == 1u ? 0u : (uint32_t)((0x100000000ull + a.per_block - 1u) / a.per_block);
}

template <bool kPair>
bool launch(const Q8FewArgs &a, cudaStream_t stream) {
    const uint32_t tiles = (a.vectors + 7u) / 8u;
    // Measured alone in a chain, tables from HBM: 2048 x 7168 and 5 rows 9.6 us with sixteen splits of
    // two steps (eight of four 14.1, of seven 11.9); 7168 x 2048 8.3 with eight of two (sixteen 9.6);
    // from 9 rows on eight splits of four (25 and more rows: three) steps are best or within 1 us
    // nearly everywhere (7168 x 2048 with 24 rows: 10.9 with four splits, 13.0).
    const bool deep = a.columns >= 4096u;
    // A row's order of sums must not depend on the rows beside it, so where up to 8 rows take sixteen
    // warps, more rows take sixteen splits as well, two per warp one after the other (sixteen warps would
    // run out of registers).  Shared expert of 7168 x 2048, all three products: 9 / 16 / 24 / 31 rows
    // 32.4 / 33.4 / 37.0 / 39.8 us; with eight splits there 31.7 / 32.8 / 36.6 / 37.5.
    const uint32_t warps = (tiles == 1u && deep ? 16u : 8u) * (kPair ? 2u : 1u);
    auto kernel = tiles == 1u   ? (deep ? q8_few_kernel<1, kPair, 16, 2, 1> : q8_few_kernel<1, kPair, 8, 2, 1>)
                  : tiles == 2u ? (deep ? q8_few_kernel<2, kPair, 8, 4, 2> : q8_few_kernel<2, kPair, 8, 4, 1>)
                  : tiles == 3u ? (deep ? q8_few_kernel<3, kPair, 8, 4, 2> : q8_few_kernel<3, kPair, 8, 4, 1>)
                                : (deep ? q8_few_kernel<4, kPair, 8, 2, 2> : q8_few_kernel<4, kPair, 8, 3, 1>);
    return launch_chained(kernel, (a.rows + kRows - 1u) / kRows, 32u * warps, 0, stream, a);
}

}  // namespace

// Up to 32 rows; whole column steps inside a scale block; 8-byte loads of the table, 16-byte loads
// of the rows.
bool k3_q8_few_supported(const void *q, const void *x, uint32_t vectors, uint32_t columns, uint32_t block) {
    return vectors >= 1u && vectors <= 32u && block != 0u && block % 32u == 0u && columns % block == 0u &&
           columns != 0u && columns / 32u < 65536u && (((uintptr_t)q) & 7u) == 0 && (((uintptr_t)x) & 15u) == 0;
}

bool k3_q8_few_product(void *out, const void *q, const void *scales, const void *x, uint32_t vectors, uint32_t rows,
                       uint32_t columns, uint32_t block, int scale_type, cudaStream_t stream) {
    Q8FewArgs a{};
    a.q[0] = (const int8_t *)q;
    a.scales[0] = scales;
    a.x = (const uint16_t *)x;
    a.out = (uint16_t *)out;
    a.vectors = vectors;
    a.rows = rows;
    a.columns = columns;
    set_block(a, block);
    a.scale_f16 = scale_type;
    return launch<false>(a, stream);
}

bool k3_q8_few_gateup(const k3_moe_layer_desc *d, void *act, void *gate, void *up, const void *x, uint32_t vectors,
                      cudaStream_t stream) {
    Q8FewArgs a{};
    a.q[0] = (const int8_t *)d->shared_gate_q;
    a.q[1] = (const int8_t *)d->shared_up_q;
    a.scales[0] = d->shared_gate_s;
    a.scales[1] = d->shared_up_s;
    a.x = (const uint16_t *)x;
    a.out = (uint16_t *)act;
    a.gate = (uint16_t *)gate;
    a.up = (uint16_t *)up;
    a.vectors = vectors;
    a.rows = d->shared_hidden;
    a.columns = d->hidden;
    set_block(a, d->q8_block);
    a.scale_f16 = d->q8_scale_type;
    a.activation = d->activation;
    a.beta = d->beta;
    a.linear_beta = d->linear_beta;
    return launch<true>(a, stream);
}
