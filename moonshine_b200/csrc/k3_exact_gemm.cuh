// BF16 and Q8 products in the reference's summation order, any number of input rows.
//
// The order is part of the contract: 256 lanes per output (lane = column mod 256 for BF16,
// 8-column octet mod 256 for Q8), ascending within a lane with one fp32 fused multiply-add
// per term, then the binary tree 128, 64, ... 1.  So the work is fp32 FMAs on the vector
// pipes (72 TFLOP/s, measured) and what is left to choose is how little else is issued and
// moved around them.  A block computes a tile of weight rows x input rows out of register
// tiles (4 x 8 outputs per thread for Q8, 2 x 4 or 4 x 4 outputs x 4 columns for BF16): a weight is
// converted once per 8 input rows and an input once per 4 weight rows, where the one-row
// kernel these replace converted both again for every output and re-read each weight row
// from L2 for every four input rows.
//
// Bound: the issue rate.  Of the roughly 300 instructions of a 4 x 8 tile's Q8 octet step (256
// multiply-adds) 128 are packed FMAs, each for two input rows, 96 convert and scale the weights
// (byte -> float, the rounded scale product), 64 convert the inputs and about 20 load.  Before and
// after the packed FMAs: 200 rows of 3584 x 7168 517 -> 443 us, of 7168 x 3584 653 -> 541, 8 rows
// 26 -> 22 and 29 -> 25.  A BF16 step has no conversions, since the mixed-precision FMA takes bf16
// operands.
#pragma once

#include "k3_common.cuh"

#include <cuda_fp16.h>

namespace k3 {

// Two fp32 fused multiply-adds in one instruction (each rounds as fmaf does).
K3_DEVINL void fma_pair(float2 &acc, float a, float2 b) {
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "f"(a), "f"(b.x), "f"(b.y));
}

// acc + a * b for bf16 a, b: the product is exact in fp32, so this is fmaf(float(a), float(b), acc)
K3_DEVINL void fma_bf16(float &acc, uint16_t a, uint16_t b) {
    asm("fma.rn.f32.bf16 %0, %1, %2, %0;" : "+f"(acc) : "h"(a), "h"(b));
}

// ------------------------------------------------------------------------ Q8
// Warp i owns tree slot i: lanes 32 i .. 32 i + 31, i.e. octets 32 i + lane + 256 j.
// kDeep steps' loads are in flight at once (one or two input rows: the weights come from HBM).
template <int kR, int kV, int kDeep>
__global__ void __launch_bounds__(256)
exact_q8_kernel(uint16_t *__restrict__ out, const int8_t *q, const void *scales,
                const uint16_t *x, uint32_t vectors, uint32_t rows, uint32_t columns, uint32_t block,
                int scale_f16) {
    constexpr int kPhase = kV < 2 ? kV : 2;                // input rows reduced per pass over shared memory
    constexpr int kOut = kR * kPhase;
    __shared__ float red[kOut][8][32];
    const uint32_t lane = threadIdx.x % kWarp;
    const uint32_t slot = threadIdx.x / kWarp;
    const uint32_t octets = columns / 8u, per_row = columns / block;
    const uint32_t row0 = blockIdx.x * kR, v0 = blockIdx.y * kV;
    if (blockIdx.y == 0 && threadIdx.x == 0 && row0 < rows)
        prefetch_l2(q + (uint64_t)row0 * columns, (uint64_t)min((uint32_t)kR, rows - row0) * columns);
    pdl_wait();
    // rows and vectors past the end read the last one; their sums are not stored
    const int8_t *qr[kR];
    uint32_t sr[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const uint32_t row = min(row0 + (uint32_t)r, rows - 1u);
        qr[r] = q + (uint64_t)row * columns;
        sr[r] = row;
    }
    const uint16_t *xr[kV];
#pragma unroll
    for (int v = 0; v < kV; v++) xr[v] = x + (uint64_t)min(v0 + (uint32_t)v, vectors - 1u) * columns;
    constexpr int kPairs = (kV + 1) / 2;                   // input rows go in pairs through the packed FMA
    float2 acc[kR][kPairs];
#pragma unroll
    for (int r = 0; r < kR; r++)
#pragma unroll
        for (int v = 0; v < kPairs; v++) acc[r][v] = make_float2(0.f, 0.f);

    for (uint32_t first = 32u * slot + lane; first < octets; first += 256u * kDeep) {
        uint2 wq[kDeep][kR];
        float s[kDeep][kR];
        uint4 xq[kDeep][kV];
#pragma unroll
        for (int j = 0; j < kDeep; j++) {
            const uint32_t octet = min(first + 256u * j, octets - 1u);     // past the end: loaded, not used
            const uint32_t sidx = octet * 8u / block;
#pragma unroll
            for (int r = 0; r < kR; r++) wq[j][r] = *reinterpret_cast<const uint2 *>(qr[r] + (uint64_t)octet * 8u);
#pragma unroll
            for (int v = 0; v < kV; v++) xq[j][v] = *reinterpret_cast<const uint4 *>(xr[v] + (uint64_t)octet * 8u);
#pragma unroll
            for (int r = 0; r < kR; r++) {
                const uint64_t at = (uint64_t)sr[r] * per_row + sidx;
                s[j][r] = scale_f16 ? __half2float(reinterpret_cast<const __half *>(scales)[at])
                                    : reinterpret_cast<const float *>(scales)[at];
            }
        }
#pragma unroll
        for (int j = 0; j < kDeep; j++) {
            if (first + 256u * j >= octets) break;
#pragma unroll
            for (int b = 0; b < 8; b++) {
                float wf[kR];
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    // byte + 128 spliced under the exponent of 2^23, minus (2^23 + 128): exact
                    const uint32_t word = (b < 4 ? wq[j][r].x : wq[j][r].y) ^ 0x80808080u;
                    const float f = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7650u + (b & 3))) - 8388736.0f;
                    wf[r] = __fmul_rn(f, s[j][r]);
                }
                auto input = [&](int v) {
                    const uint4 &xv = xq[j][v];
                    const uint32_t pair = (b >> 1) == 0 ? xv.x : (b >> 1) == 1 ? xv.y : (b >> 1) == 2 ? xv.z : xv.w;
                    return (b & 1) ? bf16_hi(pair) : bf16_lo(pair);
                };
#pragma unroll
                for (int v = 0; v + 1 < kV; v += 2) {
                    const float2 xf = make_float2(input(v), input(v + 1));
#pragma unroll
                    for (int r = 0; r < kR; r++) fma_pair(acc[r][v / 2], wf[r], xf);
                }
                if constexpr (kV % 2 != 0) {
                    const float xf = input(kV - 1);
#pragma unroll
                    for (int r = 0; r < kR; r++) acc[r][kPairs - 1].x = fmaf(wf[r], xf, acc[r][kPairs - 1].x);
                }
            }
        }
    }
    pdl_trigger();
    // tree: widths 128, 64, 32 join slots, 16 .. 1 join lanes
#pragma unroll
    for (int p = 0; p < kV; p += kPhase) {
        if (p) __syncthreads();
#pragma unroll
        for (int r = 0; r < kR; r++)
#pragma unroll
            for (int v = 0; v < kPhase; v++) red[r * kPhase + v][slot][lane] = (p + v) % 2 ? acc[r][(p + v) / 2].y : acc[r][(p + v) / 2].x;
        __syncthreads();
        for (int o = (int)slot; o < kOut; o += 8) {
            const float(*a)[32] = red[o];
            float t0 = a[0][lane] + a[4][lane], t1 = a[1][lane] + a[5][lane];
            const float t2 = a[2][lane] + a[6][lane], t3 = a[3][lane] + a[7][lane];
            t0 += t2;
            t1 += t3;
            t0 += t1;
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) t0 += __shfl_down_sync(0xffffffffu, t0, w);
            const uint32_t row = row0 + (uint32_t)(o / kPhase), vec = v0 + (uint32_t)(p + o % kPhase);
            if (lane == 0 && row < rows && vec < vectors) out[(uint64_t)vec * rows + row] = float_to_bf16_bits(t0);
        }
    }
}

// ---------------------------------------------------------------------- BF16
// A pair of warps covers the 256 lanes of a 256-column step, four columns per thread:
// warp h of the pair holds lanes 128 h + 4 lane + i.  kSR x kSV pairs per block, each with
// its own kR weight rows and kV input rows.
template <int kR, int kV, int kSR, int kSV>
constexpr uint32_t exact_bf16_smem_floats() { return kSR * kSV * (kR * kV < 8 ? kR * kV : 8) * 4 * 32; }

// One block's work (64 * kSR * kSV threads): block_x along the weight rows, block_y along the input
// rows; `smem` holds exact_bf16_smem_floats floats.
template <typename Out, int kR, int kV, int kSR, int kSV>
K3_DEVINL void exact_bf16_block(Out *__restrict__ out, const uint16_t *w, const uint16_t *x, uint32_t vectors,
                                uint32_t rows, uint32_t columns, uint32_t block_x, uint32_t block_y, float *smem) {
    constexpr int kPhase = kR * kV < 8 ? kR * kV : 8;      // outputs whose halves meet per pass over shared memory
    float(*half_sum)[kPhase][4][32] = reinterpret_cast<float(*)[kPhase][4][32]>(smem);
    const uint32_t lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    const uint32_t h = warp & 1u, pair = warp >> 1;
    const uint32_t row0 = (block_x * kSR + pair % kSR) * kR, v0 = (block_y * kSV + pair / kSR) * kV;
    if (block_y == 0 && lane == 0 && h == 0 && row0 < rows)
        prefetch_l2(w + (uint64_t)row0 * columns, (uint64_t)min((uint32_t)kR, rows - row0) * columns * 2u);
    pdl_wait();
    const uint16_t *wr[kR];
    const uint16_t *xr[kV];
#pragma unroll
    for (int r = 0; r < kR; r++) wr[r] = w + (uint64_t)min(row0 + (uint32_t)r, rows - 1u) * columns;
#pragma unroll
    for (int v = 0; v < kV; v++) xr[v] = x + (uint64_t)min(v0 + (uint32_t)v, vectors - 1u) * columns;
    float acc[kR][kV][4];
#pragma unroll
    for (int r = 0; r < kR; r++)
#pragma unroll
        for (int v = 0; v < kV; v++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[r][v][i] = 0.f;
    // few outputs per thread: more steps in flight instead
    constexpr int kDeep = kR * kV <= 2 ? 8 : kR * kV <= 8 ? 4 : 1;
#pragma unroll kDeep
    for (uint32_t c = 128u * h + 4u * lane; c < columns; c += 256u) {
        uint2 wq[kR], xq[kV];
#pragma unroll
        for (int r = 0; r < kR; r++) wq[r] = *reinterpret_cast<const uint2 *>(wr[r] + c);
#pragma unroll
        for (int v = 0; v < kV; v++) xq[v] = *reinterpret_cast<const uint2 *>(xr[v] + c);
#pragma unroll
        for (int r = 0; r < kR; r++)
#pragma unroll
            for (int v = 0; v < kV; v++) {
                fma_bf16(acc[r][v][0], (uint16_t)wq[r].x, (uint16_t)xq[v].x);
                fma_bf16(acc[r][v][1], (uint16_t)(wq[r].x >> 16), (uint16_t)(xq[v].x >> 16));
                fma_bf16(acc[r][v][2], (uint16_t)wq[r].y, (uint16_t)xq[v].y);
                fma_bf16(acc[r][v][3], (uint16_t)(wq[r].y >> 16), (uint16_t)(xq[v].y >> 16));
            }
    }
    pdl_trigger();
    // tree: width 128 joins the two warps, 64 .. 4 join lanes (16 .. 1), 2 and 1 the four columns
#pragma unroll
    for (int p = 0; p < kR * kV; p += kPhase) {
        if (p) __syncthreads();
        if (h == 1u) {
#pragma unroll
            for (int o = p; o < p + kPhase; o++)
#pragma unroll
                for (int i = 0; i < 4; i++) half_sum[pair][o - p][i][lane] = acc[o / kV][o % kV][i];
        }
        __syncthreads();
        if (h == 1u) continue;
#pragma unroll
        for (int o = p; o < p + kPhase; o++) {
            float a[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = acc[o / kV][o % kV][i] + half_sum[pair][o - p][i][lane];
            // lanes 0-15 go on with columns 0 and 1, lanes 16-31 with 2 and 3 (lane l joins lane l + 16)
            const bool up = (lane & 16u) != 0u, up8 = (lane & 8u) != 0u;
            const float g0 = __shfl_xor_sync(0xffffffffu, up ? a[0] : a[2], 16);
            const float g1 = __shfl_xor_sync(0xffffffffu, up ? a[1] : a[3], 16);
            const float b0 = (up ? a[2] : a[0]) + g0, b1 = (up ? a[3] : a[1]) + g1;
            const float g = __shfl_xor_sync(0xffffffffu, up8 ? b0 : b1, 8);
            float t = (up8 ? b1 : b0) + g;               // lanes 0-7, 8-15, 16-23, 24-31: columns 0, 1, 2, 3
            t += __shfl_xor_sync(0xffffffffu, t, 4);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            t += __shfl_xor_sync(0xffffffffu, t, 16);    // columns m and m + 2
            t += __shfl_xor_sync(0xffffffffu, t, 8);     // and the last two
            const uint32_t row = row0 + (uint32_t)(o / kV), vec = v0 + (uint32_t)(o % kV);
            if (lane == 0 && row < rows && vec < vectors) {
                if constexpr (sizeof(Out) == 4) {
                    out[(uint64_t)vec * rows + row] = t;
                } else {
                    out[(uint64_t)vec * rows + row] = float_to_bf16_bits(t);
                }
            }
        }
    }
}

template <typename Out, int kR, int kV, int kSR, int kSV>
__global__ void __launch_bounds__(64 * kSR * kSV)
exact_bf16_kernel(Out *__restrict__ out, const uint16_t *w, const uint16_t *x,
                  uint32_t vectors, uint32_t rows, uint32_t columns) {
    __shared__ float smem[exact_bf16_smem_floats<kR, kV, kSR, kSV>()];
    exact_bf16_block<Out, kR, kV, kSR, kSV>(out, w, x, vectors, rows, columns, blockIdx.x, blockIdx.y, smem);
}

}  // namespace k3
