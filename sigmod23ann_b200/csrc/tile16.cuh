// 16-bit operand tiles of the tensor-core products, filled straight from FP32
// rows in global memory: the neighbour-of-neighbour join's (FP16) and the
// precision form's (BF16).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "common.cuh"

namespace knng {

// 16-bit operand tiles, chunk-major: K padded to the MMA step of 16, a row held
// as KP / 8 chunks of 16 bytes (8 values), chunk c of row r at c * stride +
// r * 16.  The stride is one row more than the tile has, so that the lanes of
// a warp that hold consecutive pieces of one row write to different banks.
template <int D>
struct Tile16 {
    static constexpr int KP = (D + 15) / 16 * 16;
    static constexpr int CH = KP / 8;
    static constexpr int Q = D / 4;       // 16-byte pieces of an FP32 row
    static constexpr int R = kWarp / Q;   // rows a warp reads at once, a piece a lane
    static constexpr uint32_t stride(uint32_t rows) { return rows * 16 + 16; }
    static constexpr uint32_t bytes(uint32_t rows) { return CH * stride(rows); }
};

// Two FP32 values rounded to the 16-bit type, as one word.
template <class Half>
__device__ __forceinline__ uint32_t round2(float a, float b);
template <>
__device__ __forceinline__ uint32_t round2<__half>(float a, float b) {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
template <>
__device__ __forceinline__ uint32_t round2<__nv_bfloat16>(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Rows i * kWarps + warp (i < kRows / kWarps, below `count`) of a tile: the FP32
// row of point id_i (held by lane i) minus `centre` (this lane's four dimensions
// of it), rounded.  Consecutive lanes read consecutive pieces of a row, up to
// eight loads in flight each.
template <int D, int kRows, int kWarps, class Half>
__device__ __forceinline__ void tile_rows(const float* __restrict__ pts, int ld, uint32_t ids, uint32_t count,
                                          unsigned char* __restrict__ tile, uint32_t stride, float4 centre, int lane,
                                          int warp) {
    using T = Tile16<D>;
    constexpr int N = (kRows / kWarps + T::R - 1) / T::R, U = N < 8 ? N : 8;
    const int piece = lane % T::Q, sub = lane / T::Q;
    unsigned char* at = tile + (piece >> 1) * stride + (piece & 1) * 8;
    const float* from = pts + 4 * piece;
#pragma unroll
    for (int j = 0; j < N; j += U) {
        if (static_cast<uint32_t>(j * T::R * kWarps + warp) >= count) break;  // warp-uniform
        float4 x[U];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = (j + u) * T::R + sub;
            const uint32_t id = __shfl_sync(kFull, ids, i % kWarp);
            in[u] = sub < T::R && i < kRows / kWarps && static_cast<uint32_t>(i * kWarps + warp) < count;
            x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in[u]) x[u] = __ldg(reinterpret_cast<const float4*>(from + static_cast<size_t>(id) * ld));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = (j + u) * T::R + sub;
            const uint32_t a = round2<Half>(__fsub_rn(x[u].x, centre.x), __fsub_rn(x[u].y, centre.y));
            const uint32_t b = round2<Half>(__fsub_rn(x[u].z, centre.z), __fsub_rn(x[u].w, centre.w));
            if (in[u]) *reinterpret_cast<uint2*>(at + (i * kWarps + warp) * 16) = make_uint2(a, b);
        }
    }
}

}  // namespace knng
