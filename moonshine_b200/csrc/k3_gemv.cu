// Matrix-vector / small-batch entry points: BF16 (router logits), Q8 block
// quantised (shared expert, static projections) and MXFP4 (routed experts).
// Signatures and argument checks follow the reference operator interface
// (k3_rocm_ops.h:45-182); kernels are new.
//
// Reduction order.  The BF16 and Q8 kernels reproduce the reference's
// 256-lane schedule exactly (lane = column mod 256, or 8-column octet mod 256,
// ascending within a lane, one fused multiply-add per term, then the binary
// tree 128, 64, ... 1), so their results equal the CPU oracle bit for bit.
// Batch entry points run the same code per input row, hence batch == repeated
// single-row calls byte for byte, and the batch_tile argument is validated
// but does not change any result.
#include "k3_exact_gemm.cuh"
#include "k3_mxfp4_rows.cuh"
#include "k3_moe_ops.h"

#include <algorithm>

using namespace k3;

namespace {

// ------------------------------------------------------------------- BF16
// Columns or bases that the register tiles (k3_exact_gemm.cuh) do not take, element by element: one
// warp per weight row.  Thread u keeps the partial sums of virtual lanes
// 8u..8u+7 (columns 256j + 8u + i).
template <typename Out, int VT>
__global__ void __launch_bounds__(256)
bf16_gemm_kernel(Out *__restrict__ out, const uint16_t *w,
                 const uint16_t *x, uint32_t vectors, uint32_t rows,
                 uint32_t columns) {
    pdl_wait();
    const uint32_t lane = threadIdx.x % kWarp;
    const uint32_t warps = (gridDim.x * blockDim.x) / kWarp;
    for (uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp; row < rows;
         row += warps) {
        const uint16_t *wr = w + (uint64_t)row * columns;
        for (uint32_t v0 = 0; v0 < vectors; v0 += VT) {
            float acc[VT][8];
#pragma unroll
            for (int v = 0; v < VT; v++)
#pragma unroll
                for (int i = 0; i < 8; i++) acc[v][i] = 0.f;
            for (uint32_t c0 = lane * 8u; c0 < columns; c0 += 256u) {
                float wf[8];
                uint32_t valid = min(8u, columns - c0);
#pragma unroll
                for (int i = 0; i < 8; i++)
                    wf[i] = (uint32_t)i < valid ? bf16_bits_to_float(wr[c0 + i]) : 0.f;
#pragma unroll
                for (int v = 0; v < VT; v++) {
                    if (v0 + v >= vectors) break;
                    const uint16_t *xr = x + (uint64_t)(v0 + v) * columns + c0;
                    float xf[8];
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        xf[i] = (uint32_t)i < valid ? bf16_bits_to_float(xr[i]) : 0.f;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if ((uint32_t)i < valid) acc[v][i] = fmaf(wf[i], xf[i], acc[v][i]);
                    }
                }
            }
#pragma unroll
            for (int v = 0; v < VT; v++) {
                if (v0 + v >= vectors) break;
                // tree over 256 virtual lanes t = 8u + i
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        acc[v][i] += __shfl_down_sync(0xffffffffu, acc[v][i], o);
                }
                float r0 = acc[v][0] + acc[v][4], r1 = acc[v][1] + acc[v][5];
                float r2 = acc[v][2] + acc[v][6], r3 = acc[v][3] + acc[v][7];
                r0 += r2; r1 += r3;
                r0 += r1;
                if (lane == 0) {
                    if constexpr (sizeof(Out) == 4) {
                        out[(uint64_t)(v0 + v) * rows + row] = r0;
                    } else {
                        out[(uint64_t)(v0 + v) * rows + row] = float_to_bf16_bits(r0);
                    }
                }
            }
        }
    }
}

template <typename Out, int kR, int kV, int kSR, int kSV>
bool launch_exact_bf16(void *output, const void *weights, const void *input, uint32_t vectors, uint32_t rows,
                       uint32_t columns, cudaStream_t stream) {
    const dim3 grid((rows + kR * kSR - 1u) / (kR * kSR), (vectors + kV * kSV - 1u) / (kV * kSV));
    return launch_chained(exact_bf16_kernel<Out, kR, kV, kSR, kSV>, grid, 64 * kSR * kSV, 0, stream, (Out *)output,
                          (const uint16_t *)weights, (const uint16_t *)input, vectors, rows, columns);
}

template <typename Out>
bool launch_bf16(void *output, const void *weights, const void *input, uint32_t vectors,
                 uint32_t rows, uint32_t columns, cudaStream_t stream) {
    if (columns % 4u != 0u || ((((uintptr_t)weights) | ((uintptr_t)input)) & 7u) != 0) {
        // ragged columns or odd bases: one warp per weight row, element by element where it must
        const uint32_t blocks = (uint32_t)std::min<uint64_t>(((uint64_t)rows + 7) / 8, (uint64_t)sm_count() * 8);
        auto kernel = vectors == 1u ? bf16_gemm_kernel<Out, 1> : bf16_gemm_kernel<Out, 4>;
        return launch_chained(kernel, blocks, 256, 0, stream, (Out *)output, (const uint16_t *)weights,
                              (const uint16_t *)input, vectors, rows, columns);
    }
    if (vectors == 1u) return launch_exact_bf16<Out, 1, 1, 4, 1>(output, weights, input, vectors, rows, columns, stream);
    if (vectors <= 6u) return launch_exact_bf16<Out, 1, 2, 4, 1>(output, weights, input, vectors, rows, columns, stream);
    // 2 x 4 outputs per thread fill the chip best with many blocks; between one wave of those (six
    // blocks of 128 threads per SM) and one wave of 4 x 4 (four per SM) the larger tile saves the
    // second wave.  896 x 7168, 2 x 4 against 4 x 4: 12 rows 8.2 / 11.6 us, 16 rows 14 / 12.5, 20 rows
    // 14.2 / 12.5, 24 rows 14.7 / 20, 200 rows 104 / 108 (blocks of 256 and 512 threads, as before:
    // 14.6, 14.7, 25.1, 25.2 and 123); six rows and fewer 1 x 2: 6.0 (8.0).
    const uint64_t sms = (uint64_t)sm_count(), passes = (vectors + 3u) / 4u;
    const bool one_wave_2x4 = (rows + 3u) / 4u * passes <= 6u * sms, one_wave_4x4 = (rows + 7u) / 8u * passes <= 4u * sms;
    if (!one_wave_2x4 && one_wave_4x4)
        return launch_exact_bf16<Out, 4, 4, 2, 1>(output, weights, input, vectors, rows, columns, stream);
    return launch_exact_bf16<Out, 2, 4, 2, 1>(output, weights, input, vectors, rows, columns, stream);
}

template <int kTiles, int kBlocks, int kTeams>
bool launch_mxfp4(void *output, const void *packed, const void *scales, const void *input, uint32_t vectors,
                  uint32_t rows, uint32_t columns, cudaStream_t stream) {
    constexpr size_t smem = mxfp4_tile_smem<kTiles, kBlocks, kTeams>();
    auto kernel = mxfp4_tile_kernel<kTiles, kBlocks, kTeams>;
    if (!set_max_dynamic_smem((const void *)kernel, smem)) return false;
    const dim3 grid((rows + 16u * kBlocks - 1u) / (16u * kBlocks), (vectors + 8u * kTiles - 1u) / (8u * kTiles));
    return launch_chained(kernel, grid, 32 * kBlocks * kTeams, smem, stream, (uint16_t *)output,
                          (const uint8_t *)packed, (const uint8_t *)scales, (const uint16_t *)input, vectors, rows,
                          columns);
}

template <int kR, int kV, int kDeep>
bool launch_exact_q8(void *output, const void *quantized, const void *scales, const void *input, uint32_t vectors,
                     uint32_t rows, uint32_t columns, uint32_t block, int scale_type, cudaStream_t stream) {
    const dim3 grid((rows + kR - 1u) / kR, (vectors + kV - 1u) / kV);
    return launch_chained(exact_q8_kernel<kR, kV, kDeep>, grid, 256, 0, stream, (uint16_t *)output, (const int8_t *)quantized,
                          scales, (const uint16_t *)input, vectors, rows, columns, block, scale_type);
}

}  // namespace

// ======================================================================= C ABI
extern "C" bool k3_rocm_bf16_gemm_tiled_f32(void *output, const void *weights, const void *input,
                                            uint32_t vector_count, uint32_t rows,
                                            uint32_t columns, uint32_t batch_tile, void *stream) {
    if (!output || !weights || !input || vector_count == 0u || vector_count > 65535u ||
        rows == 0u || columns == 0u) {
        return false;
    }
    if (batch_tile != 16u && batch_tile != 32u && batch_tile != 64u) return false;
    return launch_bf16<float>(output, weights, input, vector_count, rows, columns,
                              (cudaStream_t)stream);
}

extern "C" bool k3_rocm_bf16_gemm_f32(void *output, const void *weights, const void *input,
                                      uint32_t vector_count, uint32_t rows, uint32_t columns,
                                      void *stream) {
    return k3_rocm_bf16_gemm_tiled_f32(output, weights, input, vector_count, rows, columns, 16u,
                                       stream);
}

extern "C" bool k3_rocm_bf16_gemv_f32(void *output, const void *weights, const void *input,
                                      uint32_t rows, uint32_t columns, void *stream) {
    return k3_rocm_bf16_gemm_f32(output, weights, input, 1u, rows, columns, stream);
}

extern "C" bool k3_rocm_bf16_gemm_tiled_bf16(void *output, const void *weights,
                                             const void *input, uint32_t vector_count,
                                             uint32_t rows, uint32_t columns,
                                             uint32_t batch_tile, void *stream) {
    if (!output || !weights || !input || vector_count == 0u || vector_count > 65535u ||
        rows == 0u || columns == 0u) {
        return false;
    }
    if (batch_tile != 16u && batch_tile != 32u && batch_tile != 64u) return false;
    return launch_bf16<uint16_t>(output, weights, input, vector_count, rows, columns,
                                 (cudaStream_t)stream);
}

extern "C" bool k3_rocm_bf16_gemm_bf16(void *output, const void *weights, const void *input,
                                       uint32_t vector_count, uint32_t rows, uint32_t columns,
                                       void *stream) {
    return k3_rocm_bf16_gemm_tiled_bf16(output, weights, input, vector_count, rows, columns, 16u,
                                        stream);
}

extern "C" bool k3_rocm_bf16_gemv_bf16(void *output, const void *weights, const void *input,
                                       uint32_t rows, uint32_t columns, void *stream) {
    return k3_rocm_bf16_gemm_bf16(output, weights, input, 1u, rows, columns, stream);
}

extern "C" bool k3_moe_q8_gemm_bf16(void *output, const void *quantized, const void *scales,
                                    const void *input, uint32_t vector_count, uint32_t rows,
                                    uint32_t columns, uint32_t block, int scale_type,
                                    void *stream) {
    if (!output || !quantized || !scales || !input || vector_count == 0u ||
        vector_count > 65535u || rows == 0u || columns == 0u || block == 0u ||
        block % 8u != 0u || columns % block != 0u || (scale_type != 0 && scale_type != 1)) {
        return false;
    }
    if ((((uintptr_t)quantized) & 7u) != 0 || (((uintptr_t)input) & 15u) != 0) return false;
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t steps = (columns / 8u + 255u) / 256u;
    auto launch = vector_count > 4u    ? launch_exact_q8<4, 8, 1>
                  : vector_count > 2u  ? launch_exact_q8<4, 4, 1>
                  : vector_count == 2u ? (steps == 1u ? launch_exact_q8<4, 2, 1> : launch_exact_q8<4, 2, 4>)
                  : steps == 1u        ? launch_exact_q8<4, 1, 1>
                  : steps == 2u        ? launch_exact_q8<4, 1, 2>
                                       : launch_exact_q8<4, 1, 4>;
    return launch(output, quantized, scales, input, vector_count, rows, columns, block, scale_type, st);
}

extern "C" bool k3_rocm_q8_128_gemm_tiled_bf16(void *output, const void *quantized,
                                               const void *scales, const void *input,
                                               uint32_t vector_count, uint32_t rows,
                                               uint32_t columns, uint32_t batch_tile,
                                               void *stream) {
    if (columns % 128u != 0u) return false;
    if (batch_tile != 16u && batch_tile != 32u && batch_tile != 64u) return false;
    return k3_moe_q8_gemm_bf16(output, quantized, scales, input, vector_count, rows, columns,
                               128u, 0, stream);
}

extern "C" bool k3_rocm_q8_128_gemm_bf16(void *output, const void *quantized, const void *scales,
                                         const void *input, uint32_t vector_count, uint32_t rows,
                                         uint32_t columns, void *stream) {
    return k3_rocm_q8_128_gemm_tiled_bf16(output, quantized, scales, input, vector_count, rows,
                                          columns, 16u, stream);
}

extern "C" bool k3_rocm_q8_128_gemv_bf16(void *output, const void *quantized, const void *scales,
                                         const void *input, uint32_t rows, uint32_t columns,
                                         void *stream) {
    return k3_rocm_q8_128_gemm_bf16(output, quantized, scales, input, 1u, rows, columns, stream);
}

extern "C" bool k3_rocm_mxfp4_gemm_tiled_bf16(void *output, const void *packed,
                                              const void *scales, const void *input,
                                              uint32_t vector_count, uint32_t rows,
                                              uint32_t columns, uint32_t batch_tile,
                                              void *stream) {
    if (!output || !packed || !scales || !input || vector_count == 0u ||
        vector_count > 65535u || rows == 0u || columns == 0u || columns % 32u != 0u) {
        return false;
    }
    if (batch_tile != 16u && batch_tile != 32u && batch_tile != 64u) return false;
    if ((((uintptr_t)packed) & 7u) != 0) return false;   // the format guarantees 8 bytes
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t tiles = (vector_count + 7u) / 8u;
    const bool wide = (((uintptr_t)input) & 15u) == 0;
    if (tiles == 1u || !wide) {
        auto kernel = wide ? mxfp4_rows_kernel<true> : mxfp4_rows_kernel<false>;
        return launch_chained(kernel, dim3((rows + 15u) / 16u, tiles), 32 * kMxSplits, 0, st, (uint16_t *)output,
                              (const uint8_t *)packed, (const uint8_t *)scales, (const uint16_t *)input,
                              vector_count, rows, columns);
    }
    // Vectors in passes of equal width, at most seven tiles of accumulators: a block's time is
    // about tiles + 3 (the dequantisation), and what counts is that of the waves it takes.
    uint32_t best = 7u, best_cost = 0xffffffffu;
    for (uint32_t width = 2u; width <= 7u; width++) {
        const uint32_t block_rows = width <= 3u ? 32u : 64u;
        const uint64_t blocks = (uint64_t)((rows + block_rows - 1u) / block_rows) * ((tiles + width - 1u) / width);
        const uint64_t cost = (blocks + sm_count() - 1u) / sm_count() * (width + 3u);
        if (cost < best_cost) {
            best = width;
            best_cost = (uint32_t)std::min<uint64_t>(cost, 0xfffffffeu);
        }
    }
    switch (best) {
        case 2: return launch_mxfp4<2, 2, 8>(output, packed, scales, input, vector_count, rows, columns, st);
        case 3: return launch_mxfp4<3, 2, 8>(output, packed, scales, input, vector_count, rows, columns, st);
        case 4: return launch_mxfp4<4, 4, 4>(output, packed, scales, input, vector_count, rows, columns, st);
        case 5: return launch_mxfp4<5, 4, 4>(output, packed, scales, input, vector_count, rows, columns, st);
        case 6: return launch_mxfp4<6, 4, 4>(output, packed, scales, input, vector_count, rows, columns, st);
        default: return launch_mxfp4<7, 4, 4>(output, packed, scales, input, vector_count, rows, columns, st);
    }
}

extern "C" bool k3_rocm_mxfp4_gemm_bf16(void *output, const void *packed, const void *scales,
                                        const void *input, uint32_t vector_count, uint32_t rows,
                                        uint32_t columns, void *stream) {
    return k3_rocm_mxfp4_gemm_tiled_bf16(output, packed, scales, input, vector_count, rows,
                                         columns, 16u, stream);
}

extern "C" bool k3_rocm_mxfp4_gemv_bf16(void *output, const void *packed, const void *scales,
                                        const void *input, uint32_t rows, uint32_t columns,
                                        void *stream) {
    return k3_rocm_mxfp4_gemm_bf16(output, packed, scales, input, 1u, rows, columns, stream);
}
