// kvb_chunk_merge.cuh -- the last step of chunk attention: the partials of a row's key ranges become its output.
#pragma once

#include <climits>

#include "kvb_chunk_shape.hpp"
#include "kvb_common.cuh"
#include "kvb_ptx.cuh"

namespace kvb {
namespace {

constexpr int kNoRow = INT_MIN;     // position of a row of a tile that the chunk does not have (a row that sees no key: -1)

// Position of dim d inside its group of eight: order 0,4,1,5,2,6,3,7.
__device__ __forceinline__ int dim_slot(int d) { return (d & ~7) | ((d & 3) << 1) | ((d >> 2) & 1); }

// Merge the key ranges of one query row, normalise, undo the tile dim order (head_dim 128), rotate back, store -- or, for a cache
// that holds only a range of the sequence, export the merged partial instead (m in natural-log units, l, o in the
// rotated domain and natural dim order, not normalised).
// One CTA of 8 warps per row: warp w takes ranges w, w+8, ..; lane l owns dims l + 32 j.  The loop is pure load
// latency, so it is unrolled to keep several ranges in flight; the warp sums meet in shared memory.
template <int D, int kPer>  // kPer: ranges per warp, ksplit <= 8 kPer
__global__ void __launch_bounds__(256) prefill_merge_kernel(const float* __restrict__ ws_m, const float* __restrict__ ws_l,
                                                            const float* __restrict__ ws_o, int T, int q_heads, int kv_heads,
                                                            int mtiles, int ksplit, int dtype, uint16_t* __restrict__ out,
                                                            float* __restrict__ part_m, float* __restrict__ part_l,
                                                            float* __restrict__ part_o) {
    constexpr int R = D / 32;
    __shared__ float so[8][D];
    __shared__ float sl[8], smx[8];
    const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = q_heads / kv_heads, tq = row / q_heads, qh = row % q_heads, head = qh / G, mrow = tq * G + qh % G;
    const int64_t base = ((static_cast<int64_t>(head) * mtiles + mrow / kRowTile) * ksplit) * kRowTile + mrow % kRowTile;
    // Warp w merges ranges w, w + 8, .. (kPer of them; at most 16: ksplit <= 128) relative to their own maximum, every
    // load issued before the first use: one trip to memory for the whole row; the eight warp results meet in shared
    // memory.  kPer is a template parameter so that a chunk (a few ranges, tens of thousands of rows) keeps the
    // registers low and the occupancy high.
    float pm[kPer], pl[kPer], po[kPer][R];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int z = warp + 8 * k;
        const bool on = z < ksplit;
        const int64_t i = base + static_cast<int64_t>(on ? z : 0) * kRowTile;
        pm[k] = on ? ws_m[i] : -INFINITY;
        pl[k] = on ? ws_l[i] : 0.0f;
#pragma unroll
        for (int j = 0; j < R; ++j) po[k][j] = on ? ws_o[i * D + (D == 128 ? dim_slot(lane + 32 * j) : lane + 32 * j)] : 0.0f;
    }
    float mw = -INFINITY;
#pragma unroll
    for (int k = 0; k < kPer; ++k) mw = fmaxf(mw, pm[k]);
    float l = 0.0f, o[R] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (mw != -INFINITY) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const float w = fast_exp2(pm[k] - mw);  // 0 for a range that is not there
            l += w * pl[k];
#pragma unroll
            for (int j = 0; j < R; ++j) o[j] += w * po[k][j];
        }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) so[warp][lane + 32 * j] = o[j];
    if (lane == 0) { sl[warp] = l; smx[warp] = mw; }
    __syncthreads();
    if (warp != 0) return;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < 8; ++w) m = fmaxf(m, smx[w]);
    l = 0.0f;
#pragma unroll
    for (int j = 0; j < R; ++j) o[j] = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const float wt = smx[w] == -INFINITY ? 0.0f : fast_exp2(smx[w] - m);
        l += wt * sl[w];
#pragma unroll
        for (int j = 0; j < R; ++j) o[j] += wt * so[w][lane + 32 * j];
    }
    if (part_m != nullptr) {
        if (lane == 0) { part_m[row] = m * 0.6931471805599453f; part_l[row] = l; }
#pragma unroll
        for (int j = 0; j < R; ++j) part_o[static_cast<int64_t>(row) * D + lane + 32 * j] = o[j];
        return;
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
    for (int j = 0; j < R; ++j) o[j] *= inv;
    hadamard_warp<D>(o, lane);
#pragma unroll
    for (int j = 0; j < R; ++j)
        out[static_cast<int64_t>(row) * D + lane + 32 * j] = dtype == KVB_DTYPE_BF16 ? f32_to_out<true>(o[j]) : f32_to_out<false>(o[j]);
}

// The same for a chunk (tens of thousands of rows, at most 16 key ranges): one warp per row, eight rows a CTA.  Lane l owns
// dims 4 l .. 4 l + 3 of each 128 in the order they lie in the partials, so every load is a full 512-byte line; four ranges
// are in flight.  Bound by the partials' bytes.  Measured on B200 (a CTA per row, one load per warp in flight, in brackets):
// 24,576 rows of 256 dims in 3 ranges 18.1 us (67.1), 18,648 rows of 128 dims in 2 ranges 9.6 us (49.6, 3 ranges).
constexpr int kMergeWarps = 8, kMergeFew = 16;
template <int D>
__global__ void __launch_bounds__(32 * kMergeWarps) chunk_merge_kernel(const float* __restrict__ ws_m, const float* __restrict__ ws_l,
                                                                       const float* __restrict__ ws_o, int rows, int q_heads, int kv_heads,
                                                                       int mtiles, int ksplit, int dtype, uint16_t* __restrict__ out,
                                                                       float* __restrict__ part_m, float* __restrict__ part_l,
                                                                       float* __restrict__ part_o) {
    constexpr int R = D / 32, S = D / 128;
    __shared__ float4 so[kMergeWarps][D / 4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x * kMergeWarps + warp;
    if (row >= rows) return;
    const int G = q_heads / kv_heads, tq = row / q_heads, qh = row % q_heads, head = qh / G, mrow = tq * G + qh % G;
    const int64_t base = ((static_cast<int64_t>(head) * mtiles + mrow / kRowTile) * ksplit) * kRowTile + mrow % kRowTile;
    const float pm = lane < ksplit ? ws_m[base + static_cast<int64_t>(lane) * kRowTile] : -INFINITY;
    const float pl = lane < ksplit ? ws_l[base + static_cast<int64_t>(lane) * kRowTile] : 0.0f;
    float m = pm;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float wz = m == -INFINITY ? 0.0f : fast_exp2(pm - m);
    float l = wz * pl;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    float4 acc[S];
#pragma unroll
    for (int s = 0; s < S; ++s) acc[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (m != -INFINITY) {
        const float4* src = reinterpret_cast<const float4*>(ws_o + base * D) + lane;
#pragma unroll 4
        for (int z = 0; z < ksplit; ++z) {
            const float w = __shfl_sync(0xffffffffu, wz, z);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float4 v = src[static_cast<int64_t>(z) * (kRowTile * D / 4) + 32 * s];
                acc[s].x += w * v.x; acc[s].y += w * v.y; acc[s].z += w * v.z; acc[s].w += w * v.w;
            }
        }
    }
    const float inv = part_m != nullptr ? 1.0f : l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
    for (int s = 0; s < S; ++s) so[warp][32 * s + lane] = make_float4(acc[s].x * inv, acc[s].y * inv, acc[s].z * inv, acc[s].w * inv);
    __syncwarp();
    float o[R];
#pragma unroll
    for (int j = 0; j < R; ++j) o[j] = reinterpret_cast<const float*>(so[warp])[D == 128 ? dim_slot(lane + 32 * j) : lane + 32 * j];
    if (part_m != nullptr) {
        if (lane == 0) { part_m[row] = m * 0.6931471805599453f; part_l[row] = l; }
#pragma unroll
        for (int j = 0; j < R; ++j) part_o[static_cast<int64_t>(row) * D + lane + 32 * j] = o[j];
        return;
    }
    hadamard_warp<D>(o, lane);
#pragma unroll
    for (int j = 0; j < R; ++j)
        out[static_cast<int64_t>(row) * D + lane + 32 * j] = dtype == KVB_DTYPE_BF16 ? f32_to_out<true>(o[j]) : f32_to_out<false>(o[j]);
}

template <int D>
int launch_chunk_merge(const float* ws_m, const float* ws_l, const float* ws_o, int tokens, int q_heads, int kv_heads, int mtiles, int ksplit,
                       int dtype, void* out, float* part_m, float* part_l, float* part_o, cudaStream_t s) {
    const int rows = tokens * q_heads;
    if (ksplit <= kMergeFew) {  // a warp walks the ranges one after another: more of them are a CTA's work
        chunk_merge_kernel<D><<<(rows + kMergeWarps - 1) / kMergeWarps, 32 * kMergeWarps, 0, s>>>(
            ws_m, ws_l, ws_o, rows, q_heads, kv_heads, mtiles, ksplit, dtype, static_cast<uint16_t*>(out), part_m, part_l, part_o);
    } else {
        auto merge = ksplit <= 32 ? prefill_merge_kernel<D, 4> : ksplit <= 64 ? prefill_merge_kernel<D, 8> : prefill_merge_kernel<D, 16>;
        merge<<<rows, 256, 0, s>>>(ws_m, ws_l, ws_o, tokens, q_heads, kv_heads, mtiles, ksplit, dtype, static_cast<uint16_t*>(out), part_m, part_l,
                                   part_o);
    }
    KVB_CUDA_OK(cudaGetLastError());
    return KVB_OK;
}

}  // namespace
}  // namespace kvb
