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
#include "k3_exact_gemm.cuh"
#include "k3_grouped.h"
#include "k3_moe_ops.h"
#include "k3_mxfp4_rows.cuh"

#include <cuda_fp16.h>

using namespace k3;

namespace {

constexpr uint32_t kRows = 16;

struct Q8Table {
    const int8_t *q;
    const void *scales;
    const uint16_t *x;
    uint32_t columns, per_row;           // scale blocks per row
    uint32_t per_block;                  // column steps per scale block, and 2^32 / per_block rounded up
    uint32_t reciprocal;                 //   (steps stay below 2^16, so the high word of a product is the quotient)
};
struct Q8FewArgs {
    Q8Table table[2];
    uint16_t *out, *gate, *up;           // gate, up: where a pair's two products go beside the activation
    uint32_t vectors, rows;
    int scale_f16, activation;
    float beta, linear_beta;
};
// What becomes of a block's sums: one product; gate and up with the activation; the sum of two
// products, each rounded to bf16 first; one product's rows 0 .. 15 and 16 .. 31 of a block.
enum Form : int { kPlain = 0, kAct = 1, kAdd = 2, kTwin = 3 };

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
// row's sum has the same order whatever the number of warps.  `smem`: q8_few_smem_floats floats.
template <int kTiles, int kForm, uint32_t kSplits>
constexpr uint32_t q8_few_smem_floats() { return (kForm != kPlain ? 2u : 1u) * kSplits * kTiles * 8u * kRows; }

template <int kTiles, int kForm, uint32_t kSplits, uint32_t kDeep, uint32_t kTurns>
K3_DEVINL void q8_few_block(const Q8FewArgs &a, uint32_t block_index, float *smem) {
    constexpr uint32_t kTables = kForm != kPlain ? 2u : 1u;
    float(*red)[kTiles * 8u][kRows] = reinterpret_cast<float(*)[kTiles * 8u][kRows]>(smem);
    const uint32_t lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp, g = lane >> 2, t = lane & 3u;
    const uint32_t split = warp % kSplits, table = warp / kSplits;
    const bool second = kTables == 2u && kForm != kTwin && table != 0u;
    const uint32_t row0 = kForm == kTwin ? block_index * 2u * kRows + table * kRows : block_index * kRows;
    const uint32_t columns = second ? a.table[1].columns : a.table[0].columns, steps = columns / 32u;
    const uint32_t per_row = second ? a.table[1].per_row : a.table[0].per_row;
    const uint32_t per_block = second ? a.table[1].per_block : a.table[0].per_block;
    const uint32_t reciprocal = second ? a.table[1].reciprocal : a.table[0].reciprocal;
    const int8_t *q = second ? a.table[1].q : a.table[0].q;
    const void *scales = second ? a.table[1].scales : a.table[0].scales;
    const uint16_t *rows_x = second ? a.table[1].x : a.table[0].x;
    if (lane == 0 && split == 0 && row0 < a.rows)
        prefetch_l2(q + (uint64_t)row0 * columns, (uint64_t)min(kRows, a.rows - row0) * columns);
    pdl_wait();
    // rows and vectors past the end read the last one; their sums are not stored
    const uint32_t row_a = min(row0 + g, a.rows - 1u), row_b = min(row0 + g + 8u, a.rows - 1u);
    const int8_t *qa = q + (uint64_t)row_a * columns + 8u * t, *qb = q + (uint64_t)row_b * columns + 8u * t;
    const uint64_t sa = (uint64_t)row_a * per_row, sb = (uint64_t)row_b * per_row;
    auto scale = [&](uint64_t at) {
        return a.scale_f16 ? __half2float(reinterpret_cast<const __half *>(scales)[at])
                           : reinterpret_cast<const float *>(scales)[at];
    };
    const uint16_t *x[kTiles];
#pragma unroll
    for (int n = 0; n < kTiles; n++)
        x[n] = rows_x + (uint64_t)min(8u * n + g, a.vectors - 1u) * columns + 8u * t;
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
                const uint32_t at = per_block == 1u ? step : __umulhi(step, reciprocal);
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
        const uint32_t row = block_index * (kForm == kTwin ? 2u : 1u) * kRows + r;
        if (row >= a.rows || v >= a.vectors) continue;
        const uint64_t at = (uint64_t)v * a.rows + row;
        uint16_t bits = float_to_bf16_bits(sum[0]);
        const uint16_t other = float_to_bf16_bits(sum[kTables - 1u]);
        if (kForm == kAct) {
            a.gate[at] = bits;
            a.up[at] = other;
            bits = float_to_bf16_bits(activation(bf16_bits_to_float(bits), bf16_bits_to_float(other), a.activation, a.beta,
                                                 a.linear_beta));
        } else if (kForm == kAdd) {
            bits = float_to_bf16_bits(bf16_bits_to_float(bits) + bf16_bits_to_float(other));
        } else if (kForm == kTwin && row + kRows < a.rows) {
            a.out[at + kRows] = other;
        }
        a.out[at] = bits;
    }
}

template <int kTiles, int kForm, uint32_t kSplits, uint32_t kDeep, uint32_t kTurns>
__global__ void __launch_bounds__(32 * kSplits * (kForm != kPlain ? 2 : 1))
q8_few_kernel(Q8FewArgs a) {
    __shared__ float smem[q8_few_smem_floats<kTiles, kForm, kSplits>()];
    q8_few_block<kTiles, kForm, kSplits, kDeep, kTurns>(a, blockIdx.x, smem);
}

// What a batch of a few tokens computes from its rows alone, in one launch: the shared expert's gate
// and up with the activation, the latent projection (where there is one) and the router's
// logits.  By themselves each is bound by the latency of its loads, seven dependent rounds per
// warp at a fourth of the memory rate; together their blocks fill the chip once, two of 512 threads
// per SM for up to 8 rows.  Latent shape, one token: 39 us in three launches, 25 here (three column steps
// in flight spill: 27; one block per SM with four: 31); 24 tokens without the projection 56 -> 40.
// Whole latent layer with a launch each / joined (its last two products too): 1 token 115 / 102 us, 2
// 175 / 161, 5 282 / 273, 8 380 / 365, 9 420 / 411, 16 566 / 556, 24 697 / 684, 31 812 to 840 / 791 to 815.
// Every product keeps the order of sums of its own kernel, so it has the same bits.
struct FrontArgs {
    Q8FewArgs gateup, project;
    uint32_t gateup_blocks, project_blocks, router_blocks_x;
    float *logits;
    const uint16_t *router;
    uint32_t experts;
};
template <int kTiles, uint32_t kTurns, int kR, int kV>
__global__ void __launch_bounds__(512, kTiles == 1 ? 2 : 1)
few_front_kernel(FrontArgs f) {
    constexpr uint32_t kQ8 = q8_few_smem_floats<kTiles, kAct, 8>(), kRouter = exact_bf16_smem_floats<kR, kV, 8, 1>();
    constexpr uint32_t kDeep = kTiles == 1 || kTiles == 4 ? 2 : 4;
    __shared__ float smem[kQ8 > kRouter ? kQ8 : kRouter];
    uint32_t block = blockIdx.x;
    if (block < f.gateup_blocks) {
        q8_few_block<kTiles, kAct, 8, kDeep, kTurns>(f.gateup, block, smem);
        return;
    }
    block -= f.gateup_blocks;
    if (block < f.project_blocks) {
        q8_few_block<kTiles, kTwin, 8, kDeep, kTurns>(f.project, block, smem);
        return;
    }
    block -= f.project_blocks;
    exact_bf16_block<float, kR, kV, 8, 1>(f.logits, f.router, f.gateup.table[0].x, f.gateup.vectors, f.experts,
                                          f.gateup.table[0].columns, block % f.router_blocks_x, block / f.router_blocks_x,
                                          smem);
}

Q8Table table_of(const void *q, const void *scales, const void *x, uint32_t columns, uint32_t block) {
    const uint32_t per_block = block / 32u;
    return {(const int8_t *)q, scales, (const uint16_t *)x, columns, columns / block, per_block,
            per_block == 1u ? 0u : (uint32_t)((0x100000000ull + per_block - 1u) / per_block)};
}

// sixteen splits of a row's columns, or eight (see launch)
bool is_deep(uint32_t columns) { return columns >= 4096u; }

template <int kForm>
bool launch(const Q8FewArgs &a, cudaStream_t stream) {
    const uint32_t tiles = (a.vectors + 7u) / 8u;
    // Measured alone in a chain, tables from HBM: 2048 x 7168 and 5 rows 9.6 us with sixteen splits of
    // two steps (eight of four 14.1, of seven 11.9); 7168 x 2048 8.3 with eight of two (sixteen 9.6);
    // from 9 rows on eight splits of four (25 and more rows: three) steps are best or within 1 us
    // nearly everywhere (7168 x 2048 with 24 rows: 10.9 with four splits, 13.0).
    const bool deep = is_deep(a.table[0].columns);
    // A row's order of sums must not depend on the rows beside it, so where up to 8 rows take sixteen
    // warps, more rows take sixteen splits as well, two per warp one after the other (sixteen warps would
    // run out of registers).  Shared expert of 7168 x 2048, all three products: 9 / 16 / 24 / 31 rows
    // 32.4 / 33.4 / 37.0 / 39.8 us; with eight splits there 31.7 / 32.8 / 36.6 / 37.5.
    const uint32_t warps = (tiles == 1u && deep ? 16u : 8u) * (kForm != kPlain ? 2u : 1u);
    auto kernel = tiles == 1u   ? (deep ? q8_few_kernel<1, kForm, 16, 2, 1> : q8_few_kernel<1, kForm, 8, 2, 1>)
                  : tiles == 2u ? (deep ? q8_few_kernel<2, kForm, 8, 4, 2> : q8_few_kernel<2, kForm, 8, 4, 1>)
                  : tiles == 3u ? (deep ? q8_few_kernel<3, kForm, 8, 4, 2> : q8_few_kernel<3, kForm, 8, 4, 1>)
                                : (deep ? q8_few_kernel<4, kForm, 8, 2, 2> : q8_few_kernel<4, kForm, 8, 3, 1>);
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
    a.table[0] = table_of(q, scales, x, columns, block);
    a.out = (uint16_t *)out;
    a.vectors = vectors;
    a.rows = rows;
    a.scale_f16 = scale_type;
    return launch<kPlain>(a, stream);
}

static Q8FewArgs gateup_args(const k3_moe_layer_desc *d, void *act, void *gate, void *up, const void *x, uint32_t vectors) {
    Q8FewArgs a{};
    a.table[0] = table_of(d->shared_gate_q, d->shared_gate_s, x, d->hidden, d->q8_block);
    a.table[1] = table_of(d->shared_up_q, d->shared_up_s, x, d->hidden, d->q8_block);
    a.out = (uint16_t *)act;
    a.gate = (uint16_t *)gate;
    a.up = (uint16_t *)up;
    a.vectors = vectors;
    a.rows = d->shared_hidden;
    a.scale_f16 = d->q8_scale_type;
    a.activation = d->activation;
    a.beta = d->beta;
    a.linear_beta = d->linear_beta;
    return a;
}

bool k3_q8_few_gateup(const k3_moe_layer_desc *d, void *act, void *gate, void *up, const void *x, uint32_t vectors,
                      cudaStream_t stream) {
    return launch<kAct>(gateup_args(d, act, gate, up, x, vectors), stream);
}

bool k3_q8_few_front(const k3_moe_layer_desc *d, void *logits, void *act, void *gate, void *up, const void *x,
                     uint32_t vectors, void *latent, const void *down_q, const void *down_s, uint32_t latent_width,
                     cudaStream_t stream) {
    const uint32_t H = d->hidden;
    const bool known = d->q8_scale_type == K3_MOE_Q8_SCALE_F32 || d->q8_scale_type == K3_MOE_Q8_SCALE_F16;
    if (vectors > 31u || d->shared_hidden == 0u || !known || !d->shared_gate_q || !d->shared_gate_s || !d->shared_up_q ||
        !d->shared_up_s || !d->router_weight ||
        !k3_q8_few_supported(d->shared_gate_q, x, vectors, H, d->q8_block) ||
        !k3_q8_few_supported(d->shared_up_q, x, vectors, H, d->q8_block) ||
        (latent != nullptr && !k3_q8_few_supported(down_q, x, vectors, H, d->q8_block)) ||
        (((uintptr_t)d->router_weight) & 7u) != 0) {
        return false;
    }
    FrontArgs f{};
    f.gateup = gateup_args(d, act, gate, up, x, vectors);
    f.gateup_blocks = (d->shared_hidden + kRows - 1u) / kRows;
    if (latent != nullptr) {
        f.project.table[0] = table_of(down_q, down_s, x, H, d->q8_block);
        f.project.out = (uint16_t *)latent;
        f.project.vectors = vectors;
        f.project.rows = latent_width;
        f.project.scale_f16 = d->q8_scale_type;
        f.project_blocks = (latent_width + 2u * kRows - 1u) / (2u * kRows);
    }
    f.logits = (float *)logits;
    f.router = (const uint16_t *)d->router_weight;
    f.experts = d->expert_count;
    auto launch_front = [&](auto kernel, uint32_t r, uint32_t v) {
        f.router_blocks_x = (d->expert_count + 8u * r - 1u) / (8u * r);
        const uint32_t blocks = f.gateup_blocks + f.project_blocks + f.router_blocks_x * ((vectors + v - 1u) / v);
        return launch_chained(kernel, blocks, 512, 0, stream, f);
    };
    const uint32_t tiles = (vectors + 7u) / 8u;
    const bool deep = is_deep(H);
    if (vectors == 1u) return launch_front(deep ? few_front_kernel<1, 2, 2, 1> : few_front_kernel<1, 1, 2, 1>, 2, 1);
    if (tiles == 1u) return launch_front(deep ? few_front_kernel<1, 2, 1, 2> : few_front_kernel<1, 1, 1, 2>, 1, 2);
    if (tiles == 2u) return launch_front(deep ? few_front_kernel<2, 2, 2, 4> : few_front_kernel<2, 1, 2, 4>, 2, 4);
    if (tiles == 3u) return launch_front(deep ? few_front_kernel<3, 2, 2, 4> : few_front_kernel<3, 1, 2, 4>, 2, 4);
    return launch_front(deep ? few_front_kernel<4, 2, 2, 4> : few_front_kernel<4, 1, 2, 4>, 2, 4);
}

bool k3_q8_few_sum_of_two(void *out, const void *q0, const void *s0, const void *x0, uint32_t columns0, const void *q1,
                          const void *s1, const void *x1, uint32_t columns1, uint32_t vectors, uint32_t rows,
                          uint32_t block, int scale_type, cudaStream_t stream) {
    if (!q0 || !s0 || !x0 || !q1 || !s1 || !x1 || (scale_type != 0 && scale_type != 1) || vectors > 31u ||
        is_deep(columns0) != is_deep(columns1) || !k3_q8_few_supported(q0, x0, vectors, columns0, block) ||
        !k3_q8_few_supported(q1, x1, vectors, columns1, block)) {
        return false;
    }
    Q8FewArgs a{};
    a.table[0] = table_of(q0, s0, x0, columns0, block);
    a.table[1] = table_of(q1, s1, x1, columns1, block);
    a.out = (uint16_t *)out;
    a.vectors = vectors;
    a.rows = rows;
    a.scale_f16 = scale_type;
    return launch<kAdd>(a, stream);
}
