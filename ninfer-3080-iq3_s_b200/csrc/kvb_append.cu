// kvb_append.cu -- quantise-append into the paged pool, and the tile decode used for verification.
//
// One launch covers any token count: the grid is (tile slot of the append, kv head, K|V x 128-dim slice).  A CTA rotates the
// new rows with 32 dims of a row a lane (Walsh-Hadamard in registers, shuffles last), keeps its slice of the 128-token tile in shared
// memory, and -- when the append completes the tile -- quantises it: per-row min/max -> fp16 scale / zero-point -> 4-bit
// codes, written to the two pages of the tile.  At head_dim 256 the slices are separate CTAs (each rotates the whole row:
// cheap beside the balancing of its slice).  There is no intermediate record and no bit-serial packing.
//
// Arithmetic that decides bytes (reference kvarn128_codec.cuh:188-217 == bee_oracle.cpp:328-341) is
// spelled with round-to-nearest intrinsics so that no multiply-add contraction can change a code:
//   scale = fmaxf((hi - lo) / 15, 1e-10f);  q = clamp(roundf((x - lo) / scale), 0, 15)
//   scale_axis = fp16(best_row * scale);  zp_axis = fp16(best_row * lo);  other_axis = fp16(best_col)
#include "kvb_common.cuh"
#include "kvb_ptx.cuh"

namespace kvb {
namespace {

constexpr int kThreads = 512;
constexpr int kRowStride = kSlice + 8;  // halves per staged row: the padding keeps 128-bit row reads conflict-free
constexpr int kRedStride = kSlice + 16;  // floats between the four partial results of an index: adjacent lanes write different ones
constexpr int kPer = 32;                 // elements of the slice matrix per thread, in either order

// Tile geometry of one append, derived on the device from the first and last position
// (reference kvarn128_launch.cu:53-77; positions are contiguous, single sequence).
struct AppendTile {
    int t0, tlast, tile, base, begin, end;
    bool in_range, sealed;
};

__device__ __forceinline__ AppendTile append_tile(int pos0, int last, int index) {
    AppendTile r;
    r.t0 = pos0 / kTile;
    r.tlast = last / kTile;
    r.tile = r.t0 + index;
    r.in_range = r.tile <= r.tlast;
    r.base = r.tile * kTile;
    r.begin = pos0 > r.base ? pos0 - r.base : 0;
    r.end = last + 1 < r.base + kTile ? last + 1 - r.base : kTile;
    r.sealed = r.base + kTile <= last + 1;
    return r;
}

struct AppendSmem {
    alignas(16) __half rows[kTile * kRowStride];  // rotated rows of the tile (the slice's dims), fp16 (what the stage holds)
    alignas(16) uint8_t codes[kTile * (kSlice / 2)];  // token-major code rows
    float red_lo[4 * kRedStride], red_hi[4 * kRedStride];  // partial sums / squares, minima / maxima
    alignas(16) float fac_dim[2][kSlice / 2 + 4];  // 1 / Sinkhorn factor per dim, even dims then odd dims
    alignas(16) float fac_tok[kTile];              // ... per token
    float best_col[kSlice], best_row[kSlice];      // the factors the codes are made with
    float4 extremes[kSlice / 32];                  // per warp: smallest / largest column, row deviation
    float2 state_dev[kSlice], state_fac[kSlice];   // a state of the balancing: column and row deviations, factors
    __half ax_scale[kSlice], ax_zp[kSlice], ax_other[kSlice];
};

// Two views of the slice matrix in registers, kPer elements per thread each:
//   by token: thread (token (tid / 2) % 128, dims 64 (tid / 256) + 2 e + tid % 2);
//   by dim:   thread (dim tid % 128, tokens 32 (tid / 128) + e).
// K has row = dim, col = token; V has row = token, col = dim (reference kvarn128_codec.cuh:366-379).
__device__ __forceinline__ void load_by_token(const AppendSmem& sm, float (&x)[kPer]) {
    const int par = threadIdx.x & 1, t = (threadIdx.x >> 1) & 127, hf = threadIdx.x >> 8;
    const uint4* row = reinterpret_cast<const uint4*>(&sm.rows[t * kRowStride + hf * 64]);
#pragma unroll
    for (int j = 0; j < kPer / 4; ++j) {
        const uint4 pk = row[j];
        const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) x[4 * j + e] = __half2float(__ushort_as_half(static_cast<uint16_t>(par ? w[e] >> 16 : w[e])));
    }
}
__device__ __forceinline__ void load_by_dim(const AppendSmem& sm, float (&x)[kPer]) {
    const int d = threadIdx.x & 127, c0 = (threadIdx.x >> 7) * kPer;
#pragma unroll
    for (int e = 0; e < kPer; ++e) x[e] = __half2float(sm.rows[(c0 + e) * kRowStride + d]);
}

// 1 / sqrt(x) and 1 / x for x > 0: the hardware's approximation and a step of Newton's method.
__device__ __forceinline__ float rsqrt_newton(float x) {
    const float y = rsqrtf(x), e = fmaf(-x * y, y, 1.0f);
    return fmaf(0.5f * y, e, y);
}
__device__ __forceinline__ float rcp_newton(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return fmaf(y, fmaf(-x, y, 1.0f), y);
}

// Sinkhorn variance balancing, `iters` rounds, in the reference's order of updates
// (kvarn128_codec.cuh:104-186 == bee_oracle.cpp:210-255): columns, rows, then "keep the best so far".
// iters > 0 is the tolerance-checked regime (the reference's own CUDA kernel does not reproduce its host oracle
// byte for byte there either), so the standard deviations are computed the fast way: every thread of the CTA
// takes part, x / (s_col * s_row) becomes x * (1/s_col) * (1/s_row) with the reciprocals taken once per update
// and the factor of the reduced-over axis pulled out of the sums, and partial sums meet in shared memory.
// Both views of the matrix stay in registers, so a pass reads only the 128 factors; a row update changes only the factor
// outside the row sums, so the deviations after it come from the sums before it.  Threads 0..127 own column i and row i and hold
// their factors; the reference's running sum of clamped logarithms is kept as the running product it stands for, clamped to the same
// range, which leaves a reciprocal square root, a few products and a reciprocal between the sums and the next factors.  Threads
// 128..255 rate the states meanwhile: the extremes of a state's deviations while the rows of the next are updated, the verdict while
// its columns are.  Two passes (in pairs of elements) and four barriers a round; bound by the chain pass, barrier, factors, barrier: 1.0
// us a round.  Measured on B200, 1,024 tokens, 4 heads of 256 dims, 16 rounds, calls in a row: 36.3 -> 31.8 us (logf and expf per round, the
// owners judging, single elements before).
template <bool kValue>
__device__ void sinkhorn(AppendSmem& sm, const float (&by_token)[kPer], const float (&by_dim)[kPer], int iters) {
    const int i = threadIdx.x, j = i & (kSlice - 1);
    const bool owner = i < kSlice, rater = i >= kSlice && i < 2 * kSlice;
    auto sums = [&](const float (&x)[kPer], const float* factors, int part, int index) {
        F2 s(0.0f, 0.0f), q(0.0f, 0.0f);
#pragma unroll
        for (int e = 0; e < kPer; e += 4) {
            const float4 f = *reinterpret_cast<const float4*>(factors + e);
            const F2 a = mul2(F2(x[e], x[e + 1]), F2(f.x, f.y)), b = mul2(F2(x[e + 2], x[e + 3]), F2(f.z, f.w));
            s = add2(s, a);
            q = fma2(a, a, q);
            s = add2(s, b);
            q = fma2(b, b, q);
        }
        const float2 s2 = s.get(), q2 = q.get();
        sm.red_lo[part * kRedStride + index] = s2.x + s2.y;
        sm.red_hi[part * kRedStride + index] = q2.x + q2.y;
    };
    auto sums_over_dims = [&]() { sums(by_token, &sm.fac_dim[i & 1][(i >> 8) * kPer], 2 * (i >> 8) + (i & 1), (i >> 1) & 127); };
    auto sums_over_tokens = [&]() { sums(by_dim, &sm.fac_tok[(i >> 7) * kPer], i >> 7, i & 127); };
    auto col_pass = [&]() { if constexpr (kValue) sums_over_tokens(); else sums_over_dims(); };
    auto row_pass = [&]() { if constexpr (kValue) sums_over_dims(); else sums_over_tokens(); };
    auto dim_factor = [&](float f) { sm.fac_dim[i & 1][i >> 1] = f; };
    auto set_col = [&](float f) { if constexpr (kValue) dim_factor(f); else sm.fac_tok[i] = f; };
    auto set_row = [&](float f) { if constexpr (kValue) sm.fac_tok[i] = f; else dim_factor(f); };
    auto total = [&](const float* red) { return (red[i] + red[kRedStride + i]) + (red[2 * kRedStride + i] + red[3 * kRedStride + i]); };
    auto deviation = [&]() {  // sample standard deviation of the 128 values summed last
        const float sum = total(sm.red_lo), sq = total(sm.red_hi), mean = sum * (1.0f / 128.0f);
        const float var = fmaxf((sq - 128.0f * mean * mean) * (1.0f / 127.0f), 0.0f);
        return var > 1e-30f && var < INFINITY ? var * rsqrt_newton(var) : sqrtf(var);
    };
    // exp of the reference's clamped sum of logarithms, -0.3 .. 10
    auto advance = [](float factor, float dev) { return fminf(fmaxf(factor * fminf(fmaxf(dev, 1e-3f), 1e3f), 0.74081822f), 22026.466f); };

    float cur_col = 1.0f, cur_row = 1.0f, rcp_col = 1.0f, rcp_row = 1.0f, dev_col = 0.0f, dev_row = 0.0f;
    float best_col = 1.0f, best_row = 1.0f, best = 3.402823466e+38f;
    auto hand_over = [&]() {  // the state the owners leave
        sm.state_dev[i] = make_float2(dev_col, dev_row);
        sm.state_fac[i] = make_float2(cur_col, cur_row);
    };
    auto look = [&]() {  // a state's extremes; deviations are >= 0, so their bits have their order
        const float2 d = sm.state_dev[j];
        const uint32_t c = __float_as_uint(d.x), r = __float_as_uint(d.y);
        const uint32_t cmin = __reduce_min_sync(0xffffffffu, c), cmax = __reduce_max_sync(0xffffffffu, c), rmin = __reduce_min_sync(0xffffffffu, r), rmax = __reduce_max_sync(0xffffffffu, r);
        if ((i & 31) == 0) sm.extremes[j >> 5] = make_float4(__uint_as_float(cmin), __uint_as_float(cmax), __uint_as_float(rmin), __uint_as_float(rmax));
    };
    float2 seen = make_float2(1.0f, 1.0f);  // the factors of the state that was looked at
    auto keep_best = [&]() {  // imbalance of that state; "<=" lets a later tie win
        float4 x = sm.extremes[0];
#pragma unroll
        for (int w = 1; w < kSlice / 32; ++w) {
            const float4 y = sm.extremes[w];
            x = make_float4(fminf(x.x, y.x), fmaxf(x.y, y.y), fminf(x.z, y.z), fmaxf(x.w, y.w));
        }
        const float imb = __fadd_rn(__fdiv_rn(x.y, fmaxf(x.x, 1e-8f)), __fdiv_rn(x.w, fmaxf(x.z, 1e-8f)));
        if (imb <= best) { best = imb; best_col = seen.x; best_row = seen.y; }
    };

    if (owner) { set_col(1.0f); set_row(1.0f); }
    __syncthreads();
    row_pass();
    __syncthreads();
    if (owner) dev_row = deviation();
    __syncthreads();
    col_pass();
    __syncthreads();
    for (int it = 0; it < iters; ++it) {
        if (owner) {
            dev_col = deviation() * rcp_col;
            hand_over();
            cur_col = advance(cur_col, dev_col);
            rcp_col = rcp_newton(cur_col);
            set_col(rcp_col);
        }
        if (rater && it > 0) keep_best();
        __syncthreads();
        row_pass();
        __syncthreads();
        if (owner) {
            const float dev = deviation();
            cur_row = advance(cur_row, dev * rcp_row);
            rcp_row = rcp_newton(cur_row);
            set_row(rcp_row);
            dev_row = dev * rcp_row;
        }
        if (rater) {
            look();
            seen = sm.state_fac[j];
        }
        __syncthreads();
        col_pass();
        __syncthreads();
    }
    if (owner) {
        dev_col = deviation() * rcp_col;
        hand_over();
    }
    if (rater && iters > 0) keep_best();
    __syncthreads();
    if (rater) {
        look();
        seen = sm.state_fac[j];
    }
    __syncthreads();
    if (rater) {
        keep_best();
        sm.best_col[j] = best_col;
        sm.best_row[j] = best_row;
    }
    __syncthreads();
}

__device__ __forceinline__ float quant_scale(float lo, float hi) {
    return fmaxf(__fdiv_rn(__fsub_rn(hi, lo), 15.0f), 1e-10f);
}
__device__ __forceinline__ uint32_t quant_code(float x, float lo, float scale) {
    return static_cast<uint32_t>(fminf(fmaxf(roundf(__fdiv_rn(__fsub_rn(x, lo), scale)), 0.0f), 15.0f));
}

__device__ __noinline__ uint32_t exact_codes8(float x0, float x1, float x2, float x3, float x4, float x5, float x6, float x7, float lo, float scale) {
    return quant_code(x0, lo, scale) | quant_code(x1, lo, scale) << 4 | quant_code(x2, lo, scale) << 8 | quant_code(x3, lo, scale) << 12 |
           quant_code(x4, lo, scale) << 16 | quant_code(x5, lo, scale) << 20 | quant_code(x6, lo, scale) << 24 | quant_code(x7, lo, scale) << 28;
}
// Eight codes, element e at bits 4 e.  The quotient's nearest integer by a product with the reciprocal, which is off by less than 2^-17;
// where it lies that close to the middle between two integers (or is not a number), the division and rounding that define the code.
__device__ __forceinline__ uint32_t quant_codes8(const float* x, float lo, float scale, float rcp) {
    uint32_t codes = 0;
    bool unsure = false;
    const F2 r2(rcp, rcp), lo2(lo, lo), magic(12582912.0f, 12582912.0f);  // 1.5 * 2^23
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
        const F2 d = sub2(F2(x[e], x[e + 1]), lo2), m = fma2(d, r2, magic);
        const float2 off = fma2(d, r2, sub2(magic, m)).get(), n = m.get();  // quotient less its nearest integer
        unsure = unsure || !(fabsf(off.x) <= 0.5f - 0x1p-16f) || !(fabsf(off.y) <= 0.5f - 0x1p-16f);
        codes |= (__float_as_uint(n.x) & 15u) << (4 * e) | (__float_as_uint(n.y) & 15u) << (4 * e + 4);
    }
    return unsure ? exact_codes8(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7], lo, scale) : codes;
}

// Quantise the slice from the view that runs along its rows (K: by dim, V: by token).  kSink = false is the iters == 0
// regime (all factors 1, x == v exactly); kSink = true divides by the Sinkhorn factors first.
template <bool kValue, bool kSink>
__device__ void quantize_slice(AppendSmem& sm, float (&x)[kPer]) {
    const int tid = threadIdx.x;
    // K: row = dim, elements are tokens 32 part + e.  V: row = token, elements are dims 64 (part / 2) + 2 e + part % 2.
    const int row = kValue ? (tid >> 1) & 127 : tid & 127, part = kValue ? 2 * (tid >> 8) + (tid & 1) : tid >> 7;
    float br = 1.0f;
    if constexpr (kSink) {
        br = sm.best_row[row];
#pragma unroll
        for (int e = 0; e < kPer; ++e)
            x[e] = __fdiv_rn(x[e], __fmul_rn(sm.best_col[kValue ? 64 * (part >> 1) + 2 * e + (part & 1) : kPer * part + e], br));
    }
    float lo = 3.402823466e+38f, hi = -3.402823466e+38f;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
        lo = fminf(lo, x[e]);
        hi = fmaxf(hi, x[e]);
    }
    sm.red_lo[part * kRedStride + row] = lo;
    sm.red_hi[part * kRedStride + row] = hi;
    __syncthreads();
    lo = fminf(fminf(sm.red_lo[row], sm.red_lo[kRedStride + row]), fminf(sm.red_lo[2 * kRedStride + row], sm.red_lo[3 * kRedStride + row]));
    hi = fmaxf(fmaxf(sm.red_hi[row], sm.red_hi[kRedStride + row]), fmaxf(sm.red_hi[2 * kRedStride + row], sm.red_hi[3 * kRedStride + row]));
    const float sc = quant_scale(lo, hi), rcp = rcp_newton(sc);
    uint32_t mine[kPer / 8], even[kPer / 8], odd[kPer / 8];  // eight codes a word
#pragma unroll
    for (int k = 0; k < kPer / 8; ++k) {
        mine[k] = quant_codes8(&x[8 * k], lo, sc, rcp);
        const uint32_t other = __shfl_xor_sync(0xffffffffu, mine[k], 1);  // the odd (even) dim of the same bytes
        even[k] = (tid & 1) ? other : mine[k];
        odd[k] = (tid & 1) ? mine[k] : other;
    }
    // the even lane of a pair writes the bytes of elements 0..15, the odd lane those of 16..31
    const int k0 = 2 * (tid & 1);
    uint32_t bytes[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // four bytes: elements 16 (tid & 1) + 4 k ..
        const uint32_t ev = ((k < 2 ? (k0 ? even[2] : even[0]) : (k0 ? even[3] : even[1])) >> (16 * (k & 1))) & 0xFFFFu;
        const uint32_t od = ((k < 2 ? (k0 ? odd[2] : odd[0]) : (k0 ? odd[3] : odd[1])) >> (16 * (k & 1))) & 0xFFFFu;
        bytes[k] = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) bytes[k] |= (((ev >> (4 * e)) & 15u) | (((od >> (4 * e)) & 15u) << 4)) << (8 * e);
    }
    if constexpr (kValue) {
        *reinterpret_cast<uint4*>(&sm.codes[row * 64 + (part >> 1) * 32 + 16 * (tid & 1)]) = make_uint4(bytes[0], bytes[1], bytes[2], bytes[3]);
    } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            sm.codes[(kPer * part + 16 * (tid & 1) + e) * 64 + (row >> 1)] = static_cast<uint8_t>(bytes[e >> 2] >> (8 * (e & 3)));
    }
    if (part == 0) {
        sm.ax_scale[row] = __float2half_rn(__fmul_rn(br, sc));
        sm.ax_zp[row] = __float2half_rn(__fmul_rn(br, lo));
    }
    if (tid < kSlice) sm.ax_other[tid] = __float2half_rn(kSink ? sm.best_col[tid] : 1.0f);
    __syncthreads();
}

// The new rows begin .. end - 1 of tile `base`, rotated (stages, order and roundings of hadamard_warp).  A lane holds 32 neighbouring
// dims of a row: D / 32 lanes a row, 1024 / D rows a warp at a time; the strides up to 16 stay inside a lane, in pairs of dims, those of
// 32 and more cross lanes, and rows are read and stored 16 bytes at a time.  A warp has up to 8 rows of the tile and reads them all before
// rotating any: it waits for global memory once.  `keep(row, d, x)` takes dims d .. d + 7 of the slice.  Measured on B200 against a
// warp a row with dims l + 32 r in lane l (five strides by shuffles, two bytes an access) and a division a code, us a call, graph replay of 1,024
// tokens: 128 dims 9.9 -> 7.0, 256 dims 12.5 -> 9.3; calls in a row: with 16 rounds of balancing 31.8 -> 27.1, a prompt of 777 tokens 32.6 -> 29.2.
// The rows start at 16-byte boundaries.
template <int D, bool kBf16, typename Keep>
__device__ __forceinline__ void rotate_rows(const uint16_t* __restrict__ src, int64_t row_stride, int begin, int end, int slice, Keep keep) {
    constexpr int kLanes = D / 32, kAtOnce = 32 / kLanes, kWarpsPerCta = kThreads / 32, kPasses = kTile / (kWarpsPerCta * kAtOnce);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, block = lane % kLanes;
    uint4 raw[kPasses][4];
#pragma unroll
    for (int u = 0; u < kPasses; ++u) {
        const int tt = begin + warp + kWarpsPerCta * (u * kAtOnce + lane / kLanes);
        const uint16_t* row = src + (tt - begin) * row_stride + 32 * block;
#pragma unroll
        for (int c = 0; c < 4; ++c) raw[u][c] = tt >= end ? make_uint4(0u, 0u, 0u, 0u) : reinterpret_cast<const uint4*>(row)[c];
    }
#pragma unroll
    for (int u = 0; u < kPasses; ++u) {
        if (begin + warp + kWarpsPerCta * u * kAtOnce >= end) break;  // no row left for any lane
        const int tt = begin + warp + kWarpsPerCta * (u * kAtOnce + lane / kLanes);
        F2 x[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t w[4] = {raw[u][c].x, raw[u][c].y, raw[u][c].z, raw[u][c].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {  // the stride of 1 lies inside a pair
                const float lo = in_to_f32<kBf16>(static_cast<uint16_t>(w[e])), hi = in_to_f32<kBf16>(static_cast<uint16_t>(w[e] >> 16));
                x[4 * c + e] = F2(__fadd_rn(lo, hi), __fsub_rn(lo, hi));
            }
        }
#pragma unroll
        for (int span = 1; span <= 8; span <<= 1)
#pragma unroll
            for (int b = 0; b < 16; b += 2 * span)
#pragma unroll
                for (int e = 0; e < span; ++e) {
                    const F2 lo = x[b + e], hi = x[b + e + span];
                    x[b + e] = add2(lo, hi);
                    x[b + e + span] = sub2(lo, hi);
                }
#pragma unroll
        for (int step = 1; step < kLanes; step <<= 1) {
            const float sign = (block & step) == 0 ? 1.0f : -1.0f;
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float2 y = x[e].get();
                const F2 peer(__shfl_xor_sync(0xffffffffu, y.x, step), __shfl_xor_sync(0xffffffffu, y.y, step));
                x[e] = fma2(x[e], F2(sign, sign), peer);
            }
        }
        if (tt >= end || block / 4 != slice) continue;
        constexpr float norm = D == 256 ? 0.0625f : 0.08838834764831845f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t h[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 y = mul2(x[4 * c + e], F2(norm, norm)).get();
                h[e] = pack_half2(y.x, y.y);
            }
            keep(tt, 32 * (block % 4) + 8 * c, make_uint4(h[0], h[1], h[2], h[3]));
        }
    }
}

// The same, a warp a row with dims l + 32 r in lane l: from any 2-byte boundary, up to 16 kBatch rows.  `keep(row, d, h)` takes dim d of the
// slice.
template <int D, bool kBf16, int kBatch, typename Keep>
__device__ __forceinline__ void rotate_rows_singly(const uint16_t* __restrict__ src, int64_t row_stride, int begin, int end, int slice, Keep keep) {
    constexpr int kWarpsPerCta = kThreads / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint16_t raw[kBatch][D / 32];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
        const int tt = begin + warp + u * kWarpsPerCta;
        if (tt < end) {
            const uint16_t* row = src + (tt - begin) * row_stride;
#pragma unroll
            for (int r = 0; r < D / 32; ++r) raw[u][r] = row[lane + 32 * r];
        }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
        const int tt = begin + warp + u * kWarpsPerCta;
        if (tt >= end) break;
        float val[D / 32];
#pragma unroll
        for (int r = 0; r < D / 32; ++r) val[r] = in_to_f32<kBf16>(raw[u][r]);
        hadamard_warp<D>(val, lane);
#pragma unroll
        for (int r = 0; r < 4; ++r) keep(tt, lane + 32 * r, __float2half_rn(D == 128 || slice == 0 ? val[r] : val[D / 32 - 4 + r]));
    }
}

// Whether the rows of a tile are rotated a warp each though they could go 32 dims a lane: up to 16 rows have a warp each either way, and a lane
// with 32 dims of one is the longer chain.  Measured on B200 in graph replay, us an append that completes no tile, 32 dims a lane / a warp a
// row, three rows a warp asked for at once: 128 dims 1 / 8 / 16 / 48 rows 1.9 2.3 2.9 3.0 / 1.8 1.8 1.9 2.6, at 64 rows 3.2 / 3.3 (eight at once); 256
// dims 1 / 8 / 16 / 32 rows 2.1 2.5 3.2 3.3 / 1.8 1.9 2.3 2.8, at 48 rows 3.4 / 3.7 (eight).  Rows off the 16-byte boundary (a warp a row: no
// other way reads them together): 1,024 tokens 7.7 and 10.3, by elements in the lanes that need them 10.7 and 16.6.
// Not in balanced caches of 128 dims, whose verify steps of two rows a warp take longer behind the shorter append (2 / 5 rows at 497 tokens 11.8 /
// 11.8 us a layer, a warp a row 12.1 / 12.3, the same and held up for as long 11.8 / 12.0: it is when the append ends that counts).
template <int D> __device__ __forceinline__ bool rotates_singly(int rows, bool wide, bool balanced) {
    return rows <= (D == 256 && wide ? 32 : 48) && !(D == 128 && wide && balanced);
}

// Rotate + stage + seal.
//
// Which tiles keep their rows in the stage: only the last two tiles of an append (one per slot) can be
// looked at again -- the open tile by attention and later appends, the one before it by a roll-back that
// re-opens it.  Earlier tiles of a long append would be overwritten within the same call anyway.  When the first tile
// begins inside (its earlier rows are read from the stage) and one of the last two, a different one, has the same slot, the
// first tile's CTA writes that tile's rows too, after it has read its own: no second launch, no order between CTAs.
template <int D, bool kBf16>
__global__ void __launch_bounds__(kThreads, 1) append_kernel(LayerView L, const uint16_t* __restrict__ k,
                                                             const uint16_t* __restrict__ v,
                                                             const int32_t* __restrict__ positions, int tokens) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AppendSmem& sm = *reinterpret_cast<AppendSmem*>(smem_raw);
    using G = Geo<D>;
    constexpr int S = G::S;
    grid_dependency_wait();  // launched while its predecessor still runs: nothing is read or written before it is over
    launch_dependents();
    const int pos0 = positions[0], last = positions[tokens - 1];
    if (pos0 < 0 || last - pos0 != tokens - 1) {  // positions must be contiguous and non-negative
        if (threadIdx.x == 0) L.flag(KVB_ERR_POSITIONS);
        return;
    }
    const AppendTile t = append_tile(pos0, last, blockIdx.x);
    if (!t.in_range) return;
    const int head = blockIdx.y, which = blockIdx.z / S, slice = blockIdx.z % S, slot = t.tile & 1;
    const bool inside = pos0 > t.t0 * kTile;  // the first tile has rows of earlier calls
    const bool write_stage = t.tile >= t.tlast - 1 && !(inside && t.tile >= t.t0 + 2 && ((t.tile ^ t.t0) & 1) == 0);
    const bool seal = t.sealed;
    if (!seal && !write_stage) return;

    // rows appended by earlier calls (first tile only) come from the stage
    if (seal && t.begin > 0) {
        const __half* src = L.stage_row(which, slot, head, 0) + slice * kSlice;
        for (int i = threadIdx.x; i < t.begin * (kSlice / 8); i += kThreads) {
            const int r = i / (kSlice / 8), c = i % (kSlice / 8);
            *reinterpret_cast<uint4*>(&sm.rows[r * kRowStride + c * 8]) =
                *reinterpret_cast<const uint4*>(src + static_cast<int64_t>(r) * D + c * 8);
        }
    }
    const int64_t row_stride = static_cast<int64_t>(L.kv_heads) * D;
    const uint16_t* src = (which ? v : k) + static_cast<int64_t>(head) * D;
    const bool wide = (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    // the new rows of a tile into shared memory and its stage rows, 16 bytes or one element at a time
    auto rotate = [&](const AppendTile& a, bool here, bool to_stage) {
        const uint16_t* const rows = src + (a.base + a.begin - pos0) * row_stride;
        __half* const stage = L.stage_row(which, a.tile & 1, head, 0) + slice * kSlice;
        auto keep = [&](int tt, int d, auto x) {
            using X = decltype(x);
            if (here) *reinterpret_cast<X*>(&sm.rows[tt * kRowStride + d]) = x;
            if (to_stage) *reinterpret_cast<X*>(&stage[tt * D + d]) = x;
        };
        if (rotates_singly<D>(a.end - a.begin, wide, L.iters > 0)) rotate_rows_singly<D, kBf16, 3>(rows, row_stride, a.begin, a.end, slice, keep);
        else if (wide) rotate_rows<D, kBf16>(rows, row_stride, a.begin, a.end, slice, keep);
        else rotate_rows_singly<D, kBf16, 8>(rows, row_stride, a.begin, a.end, slice, keep);
    };
    rotate(t, true, write_stage);
    if (!seal) return;
    __syncthreads();
    if (inside && t.tile == t.t0 && t.tlast >= t.t0 + 2) {
        const int later = ((t.tlast ^ t.t0) & 1) == 0 ? t.tlast : t.tlast - 1;  // of the last two tiles, the one with this slot
        if (later >= t.t0 + 2) rotate(append_tile(pos0, last, later - t.t0), false, true);
    }

    const int32_t* tbl = L.table();
    const int32_t page0 = L.page_of(tbl, 2 * t.tile), page1 = L.page_of(tbl, 2 * t.tile + 1);
    if (page0 < 0 || page1 < 0) return;  // error word already set; skip the tile instead of faulting

    float x[kPer];  // along the rows of the matrix
    if (which) load_by_token(sm, x);
    else load_by_dim(sm, x);
    if (L.iters > 0) {
        float y[kPer];  // along its columns
        if (which) {
            load_by_dim(sm, y);
            sinkhorn<true>(sm, x, y, L.iters);
            quantize_slice<true, true>(sm, x);
        } else {
            load_by_token(sm, y);
            sinkhorn<false>(sm, y, x, L.iters);
            quantize_slice<false, true>(sm, x);
        }
    } else {
        if (which) quantize_slice<true, false>(sm, x);
        else quantize_slice<false, false>(sm, x);
    }

    // code rows -> the two pages: 64 bytes of every token row
    uint8_t* code = which ? L.v_code : L.k_code;
    {
        static_assert(kThreads == kTile * 4, "one 16-byte store per thread");
        const int tok = threadIdx.x / 4, o = threadIdx.x % 4;
        uint8_t* dst = code + page_head_offset(G::kCodeLeading, L.kv_heads, tok < kPage ? page0 : page1, head) + (tok % kPage) * G::kCodeLeading + slice * 64;
        reinterpret_cast<uint4*>(dst)[o] = reinterpret_cast<const uint4*>(sm.codes + tok * 64)[o];
    }
    // scale pages: dim-axis entries go to both pages, token-axis entries to the page of the token; a slice owns the rows of its
    // dims and its column of the token entries
    const int SL = which ? G::kVScaleLeading : G::kKScaleLeading;
    constexpr int c = G::kAxisCols;
    __half* scale = which ? L.v_scale : L.k_scale;
    __half* dst0 = scale + page_head_offset(SL, L.kv_heads, page0, head);
    __half* dst1 = scale + page_head_offset(SL, L.kv_heads, page1, head);
    for (int i = threadIdx.x; i < 2 * kPage * SL; i += kThreads) {
        const int pg = i / (kPage * SL), r = (i / SL) % kPage, j = i % SL, tok = pg * kPage + r;
        __half h;
        bool mine;
        if (!which) {
            mine = j < 2 * c ? (c * r) / kSlice == slice : j - 2 * c == slice;
            if (j < c) h = sm.ax_scale[(c * r + j) % kSlice];
            else if (j < 2 * c) h = sm.ax_zp[(c * r + j - c) % kSlice];
            else h = sm.ax_other[tok];
        } else {
            mine = j < c ? (c * r) / kSlice == slice : (j - c) % S == slice;
            if (j < c) h = sm.ax_other[(c * r + j) % kSlice];
            else if (j < c + S) h = sm.ax_scale[tok];
            else h = sm.ax_zp[tok];
        }
        if (mine) (pg ? dst1 : dst0)[r * SL + j] = h;
    }
}

// One tile of one head -> rotated-domain fp16 [128][D]: val = (q * scale_axis + zp_axis) * other_axis,
// each step rounded (reference kvarn128_codec.cuh:314-350).
template <int D>
__global__ void __launch_bounds__(kThreads) decode_tile_kernel(LayerView L, int tile, int head, __half* out_k,
                                                               __half* out_v) {
    using G = Geo<D>;
    constexpr int c = G::kAxisCols, S = G::S;
    const int32_t* tbl = L.table();
    for (int i = threadIdx.x; i < kTile * D; i += kThreads) {
        const int tok = i / D, d = i % D, s = d / kSlice;
        const int32_t page = L.page_of(tbl, 2 * tile + tok / kPage);
        if (page < 0) continue;
        const int off = tok % kPage;
        const int64_t cb = page_head_offset(G::kCodeLeading, L.kv_heads, page, head) + off * G::kCodeLeading + d / 2;
        const int sh = (d & 1) * 4;
        const float qk = static_cast<float>((L.k_code[cb] >> sh) & 15), qv = static_cast<float>((L.v_code[cb] >> sh) & 15);
        const __half* ks = L.k_scale + page_head_offset(G::kKScaleLeading, L.kv_heads, page, head);
        const __half* vs = L.v_scale + page_head_offset(G::kVScaleLeading, L.kv_heads, page, head);
        const float ksa = __half2float(ks[G::kKScaleLeading * (d / c) + d % c]);
        const float kzp = __half2float(ks[G::kKScaleLeading * (d / c) + c + d % c]);
        const float koa = __half2float(ks[G::kKScaleLeading * off + 2 * c + s]);
        const float voa = __half2float(vs[G::kVScaleLeading * (d / c) + d % c]);
        const float vsa = __half2float(vs[G::kVScaleLeading * off + c + s]);
        const float vzp = __half2float(vs[G::kVScaleLeading * off + c + S + s]);
        out_k[i] = __float2half_rn(__fmul_rn(__fadd_rn(__fmul_rn(qk, ksa), kzp), koa));
        out_v[i] = __float2half_rn(__fmul_rn(__fadd_rn(__fmul_rn(qv, vsa), vzp), voa));
    }
}

template <int D, bool kBf16>
int launch_append(const LayerView& V, const void* k, const void* v, const int32_t* positions, int tokens,
                  cudaStream_t stream) {
    static_assert(sizeof(AppendSmem) <= 227 * 1024, "shared memory");
    static OncePerDevice opted;  // per template instance
    const int smem = static_cast<int>(sizeof(AppendSmem));
    KVB_CUDA_OK(allow_smem(opted, append_kernel<D, kBf16>, smem));
    const dim3 grid(tokens / kTile + 2, V.kv_heads, 2 * Geo<D>::S);
    KVB_CUDA_OK(launch_early(append_kernel<D, kBf16>, grid, dim3(kThreads), smem, stream, V, static_cast<const uint16_t*>(k), static_cast<const uint16_t*>(v),
                             positions, tokens));
    return KVB_OK;
}

}  // namespace
}  // namespace kvb

extern "C" int kvb_append(const kvb_layer* layer, const void* k, const void* v, const int32_t* positions_dev,
                          int tokens, void* stream) {
    using namespace kvb;
    if (tokens == 0) return KVB_OK;  // the reference returns silently for an empty append
    if (int st = check_layer(layer, "kvb_append")) return st;
    if (tokens < 0) return fail(KVB_EINVAL, "kvb_append: tokens = %d", tokens);
    if (k == nullptr || v == nullptr || positions_dev == nullptr)
        return fail(KVB_EINVAL, "kvb_append: null k / v / positions");
    if (layer->stage == nullptr) return fail(KVB_EINVAL, "kvb_append: layer has no stage buffer");
    const LayerView V = make_view(*layer);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool bf = layer->dtype == KVB_DTYPE_BF16;
    if (layer->head_dim == 128) return bf ? launch_append<128, true>(V, k, v, positions_dev, tokens, s)
                                          : launch_append<128, false>(V, k, v, positions_dev, tokens, s);
    return bf ? launch_append<256, true>(V, k, v, positions_dev, tokens, s)
              : launch_append<256, false>(V, k, v, positions_dev, tokens, s);
}

extern "C" int kvb_decode_tile(const kvb_layer* layer, int tile, int head, void* out_k, void* out_v, void* stream) {
    using namespace kvb;
    if (int st = check_layer(layer, "kvb_decode_tile")) return st;
    if (out_k == nullptr || out_v == nullptr) return fail(KVB_EINVAL, "kvb_decode_tile: null output");
    if (tile < 0 || head < 0 || head >= layer->kv_heads || 2 * tile + 1 >= layer->table_len)
        return fail(KVB_EINVAL, "kvb_decode_tile: tile %d / head %d out of range", tile, head);
    const LayerView V = make_view(*layer);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (layer->head_dim == 128)
        decode_tile_kernel<128><<<1, kThreads, 0, s>>>(V, tile, head, static_cast<__half*>(out_k), static_cast<__half*>(out_v));
    else
        decode_tile_kernel<256><<<1, kThreads, 0, s>>>(V, tile, head, static_cast<__half*>(out_k), static_cast<__half*>(out_v));
    KVB_CUDA_OK(cudaGetLastError());
    return KVB_OK;
}
