// kvb_chunk256.cu -- chunk attention over head_dim-256 caches (the reference engine's own geometry) on the
// 5th-generation tensor cores, at fp32 accuracy.
//
// A CTA owns 128 GQA-packed (token, q head) rows of one KV head and one range of 64-key pages.  Every operand of the two
// contractions is an fp32 value split into an fp16 high and low part (22 significant bits); a product takes three MMAs
// (low x high, high x low, high x high; the low x low term is below fp32's own rounding).  So that neither part runs
// into fp16's range, every query row, every page of K and the whole of V carry a power of two: rows and pages are scaled
// to a largest magnitude of 2^14 .. 2^15 and their exponents return in the logits (a thread owns a row), V follows the
// largest page seen so far and O is rescaled, exactly, when that grows.
//
// Roles (24 warps, one CTA per SM, registers re-divided by role):
//   warps 4-11   de-quantise K(i): code -> fp32 (code * scale + zp) * other -> high | low, 64 KB a page, in 128-byte-swizzled
//                tiles; thread = one key and 64 dims; codes and scales are fetched a page ahead;
//   warps 12-19  the same for V(i): two chains beside each other instead of one after the other;
//   warp 20      issues S(i) = Q K(i)^T, then O += P(i-1) V(i-1);
//   warps 0-3    softmax of S(i), thread = row: P (high | low) over S in tensor memory, O rescaled lazily.
// K(i+1) is written while P V(i-1) runs, V(i) while Q K(i+1)^T runs.  Tensor memory (512 columns): two S buffers of
// 64, the high part of Q (128, the A operand of two of the three Q K products), O (256).  The low part of Q stays in
// shared memory (64 KB), beside one K and one V buffer.
//
// Bound by the chain of a page: K is de-quantised (3,220 cycles), handed over (530), multiplied (48 MMAs of 128x64x16, 2,100 until
// the buffer is free; 3,100 with an election and a descriptor per MMA); P V, V and the softmax run beside it.  Measured on B200, 24 / 4
// heads, 1,024 tokens over a prefix of 16,384, balanced bf16 cache: 1.23 ms (346 TFLOP/s of attention) against 69.8 ms for
// one warp per key on fp32 FMAs, 1.40 ms with eight warps for K and V in turn, 1.38 ms with sixteen in turn.
// Accuracy: against float64 the un-normalised sums are off by 4e-7 .. 6e-6 (fp32 FMAs: 2e-7 .. 1.1e-5, sizes of 32 .. 65,576
// keys), the fp16 / bf16 outputs by their rounding alone (2.09e-4 and 1.70e-3, as before).
#include <climits>

#include "kvb_chunk_merge.cuh"
#include "kvb_common.cuh"
#include "kvb_tcgen05.cuh"

namespace kvb {
namespace {

constexpr int D = 256;
constexpr int kM = 128;   // query rows per CTA
constexpr int kN = 64;    // keys per step: one page
constexpr int kSoftWarps = 4, kDqWarps = 8, kMmaWarp = kSoftWarps + 2 * kDqWarps, kWarps = kMmaWarp + 4, kThreads = 32 * kWarps;
// Registers per thread: 80 at launch (61,440 a CTA), then by role 128 x 144 + 512 x 72 + 128 x 48 = 61,440.
constexpr int kSoftRegs = 144, kDqRegs = 72, kMmaRegs = 48;
constexpr int kKvBlock = kN * 128;       // one 64-dim block of a K or V tile: 64 rows of 128 bytes
constexpr int kKvTile = 4 * kKvBlock;
constexpr int kQBlock = kM * 128;        // one 64-dim block of the Q tile
// Per-page words handed to the softmax warps.  A writer is at most 3 pages ahead of a reader: the K role writes those of page i once
// S(i-2) is complete, which was issued after P V(i-4) but not after the softmax of page i-3.  No slot to spare.
constexpr int kSlotsMeta = 4;
constexpr uint32_t kTmemCols = 512, kColQ = 128, kColO = 256;  // S buffers at columns 0 and 64
constexpr int kTop = 14;                 // scaled operands reach 2^14 .. 2^15
constexpr float kPBoost = 4.0f;          // P is taken 2^4 above the row's reference point (and stays below 2^12): more bits of small weights survive

struct Chunk256Params {
    LayerView L;
    const uint16_t* q;         // [T][q_heads][D]
    const int32_t* pos;        // [T]
    const int32_t* total_pos;  // newest position in the cache
    int T, mtiles, ksplit;
    bool after_append;         // beside the append of the rows (kvb_step.hpp): only the readers of the planes and the stage wait for it first
    float scale_log2;
    float* ws_m;               // [H][mtiles][ksplit][128]
    float* ws_l;
    float* ws_o;               // [H][mtiles][ksplit][128][D]
};

struct __align__(1024) Chunk256Smem {
    uint8_t q_lo[4 * kQBlock];
    uint8_t k[2][kKvTile];     // high, low part; holds the high part of Q before the walk
    uint8_t v[2][kKvTile];
    float ks[2][D], kz[2][D], vo[2][D];  // per-dim factors by page parity; ks is divided by 16^(nibble position)
    alignas(16) uint2 red[2][2][kDqWarps];  // partial maxima (float bits) of K, of V: per-dim and per-key factors
    alignas(16) uint32_t poison[kSlotsMeta][kDqWarps];  // keys with a non-finite V (ballots of the warps)
    float k_unit[kSlotsMeta];            // page i: K = k_unit * (high + low)
    int v_exp[kSlotsMeta];               // exponent of V and O as of page i
    int bad_page[kSlotsMeta];
    int row_pos[kM];
    float row_unit[kM];                  // q' = row_unit * (high + low)
    uint64_t s_full[2], p_full[2], v_meta[2], k_full, v_full, o_done, drain;
    uint32_t tmem_base;
    int abort_flag;
};

// Largest power of two that keeps values of magnitude `bits` (a non-negative float) below 2^(kTop + 1): exponent of the
// scale that was taken out.  Zero and non-finite magnitudes: 0.
__device__ __forceinline__ int scale_exponent(uint32_t bits) {
    if (bits == 0u || bits >= 0x7F800000u) return 0;
    return max(static_cast<int>(bits >> 23) - 127, -100) - kTop;
}
__device__ __forceinline__ float pow2i(int e) { return __uint_as_float(static_cast<uint32_t>(e + 127) << 23); }  // |e| <= 126
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }

// x = high + low in fp16 (22 significant bits)
__device__ __forceinline__ void split2(F2 x, uint32_t& hi, uint32_t& lo) {
    const float2 f = x.get();
    hi = pack_half2(f.x, f.y);
    const float2 h = unpack_half2(hi);
    const float2 d = add2(x, F2(-h.x, -h.y)).get();
    lo = pack_half2(d.x, d.y);
}

// Eight fp32 values -> one 16-byte chunk of the high and of the low tile.
__device__ __forceinline__ void split_store(const F2 (&x)[4], uint8_t* hi_tile, uint8_t* lo_tile, uint32_t off) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split2(x[e], h[e], l[e]);
    *reinterpret_cast<uint4*>(hi_tile + off) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(lo_tile + off) = make_uint4(l[0], l[1], l[2], l[3]);
}
// Eight fp16 values of an un-quantised row, times `f`.
__device__ __forceinline__ void widen(const uint4& r, F2 f, F2 (&x)[4]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 h = unpack_half2(w[e]);
        x[e] = mul2(F2(h.x, h.y), f);
    }
}

// Eight codes of one word -> n * 16^p, p = 0 1 2 3 4 0 1 2: a nibble OR-ed under the exponent of 2^23 where it lies.
__device__ __forceinline__ void unpack_f32(uint32_t w, F2 (&n)[4]) {
    const uint32_t w5 = w >> 20;
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(lop3_and_or(e < 5 ? w : w5, 0xFu << (4 * (e < 5 ? e : e - 5)), 0x4B000000u));
#pragma unroll
    for (int e = 0; e < 4; ++e) n[e] = add2(F2(f[2 * e], f[2 * e + 1]), F2(-8388608.0f, -8388608.0f));
}
__device__ __forceinline__ constexpr int nibble_shift(int d) { return 4 * ((d & 7) < 5 ? (d & 7) : (d & 7) - 5); }

// One de-quantising role (eight warps, thread dt): K or V of the CTA's n pages p0 .. p1 - 1.
template <bool kValue>
__device__ __forceinline__ bool dequant_role(Chunk256Smem& sm, const LayerView& L, int head, int dt, int p0, int p1, int kv_total) {
    const int lane = dt & 31, dw = dt >> 5;                    // dt: also the dim whose factors this thread fetches
    const int quarter = dw & 3, key = 32 * (dw >> 2) + lane;   // 64 dims of one key of the page
    const int s = quarter >> 1, n = p1 - p0, sealed_pages = 2 * (kv_total / kTile);
    const uint32_t row_off = quarter * kKvBlock + key * 128;
    uint8_t (&tile)[2][kKvTile] = kValue ? sm.v : sm.k;
    const uint8_t* plane = kValue ? L.v_code : L.k_code;
    const int32_t* tbl = L.table();
    struct Meta {
        __half d0, d1, t0, t1;  // K: scale, zero point of the dim; other_K of the key.  V: other_V of the dim; scale, zero point of the key
        int32_t page;           // -1: unusable; the page is masked
        uint4 code[2];
    };
    int32_t entry = LayerView::kNoEntry;  // table entry of the page the next fetch asks for, requested a page earlier
    auto lookup = [&](int p) { entry = p < p1 && p < sealed_pages ? L.page_entry(tbl, p) : LayerView::kNoEntry; };
    auto fetch = [&](Meta& m) {
        m.page = L.checked_page(entry);
        m.d0 = m.d1 = m.t0 = m.t1 = __ushort_as_half(0);
        m.code[0] = m.code[1] = make_uint4(0u, 0u, 0u, 0u);
        if (m.page >= 0) {
            if constexpr (kValue) {
                const __half* vsp = L.v_scale + page_head_offset(8, L.kv_heads, m.page, head);
                m.d0 = vsp[8 * (dt >> 2) + (dt & 3)];
                m.t0 = vsp[8 * key + 4 + s];
                m.t1 = vsp[8 * key + 6 + s];
            } else {
                const __half* ksp = L.k_scale + page_head_offset(10, L.kv_heads, m.page, head);
                m.d0 = ksp[10 * (dt >> 2) + (dt & 3)];
                m.d1 = ksp[10 * (dt >> 2) + 4 + (dt & 3)];
                m.t0 = ksp[10 * key + 8 + s];
            }
            const uint4* src = reinterpret_cast<const uint4*>(plane + page_head_offset(128, L.kv_heads, m.page, head) + key * 128 + quarter * 32);
            m.code[0] = src[0];
            m.code[1] = src[1];
        }
    };
    Meta m, nxt;  // the next page's is requested at the top of a step: a step hides the trip to memory
    if (n > 0) {
        lookup(p0);
        fetch(nxt);
        lookup(p0 + 1);
    }
    bool failed = false;
    int v_run = INT_MIN;  // exponent of V so far
    for (int i = 0; i < n; ++i) {
        const int p = p0 + i, par = i & 1, slot = i & (kSlotsMeta - 1);
        const bool sealed = p < sealed_pages;
        m = nxt;
        fetch(nxt);
        lookup(p + 2);
        const __half* row = nullptr;  // open tile: this key's un-quantised row
        bool live = true;
        float d0 = __half2float(m.d0), t0 = __half2float(m.t0), t1 = __half2float(m.t1);
        // ---- per-dim tables of the page, and the largest magnitudes that decide its scale
        uint32_t db, tb;
        if constexpr (kValue) {
            db = abs_bits(d0);
            tb = max(abs_bits(t1), abs_bits(fmaf(15.0f, t0, t1)));
        } else {
            const float d1 = __half2float(m.d1);
            db = max(abs_bits(d1), abs_bits(fmaf(15.0f, d0, d1)));
            sm.ks[par][dt] = d0 * pow2i(-nibble_shift(dt));
            sm.kz[par][dt] = d1;
        }
        if (!sealed) {
            const int first = (p & 1) * kPage + key;
            row = L.stage_row(kValue ? 1 : 0, (kv_total / kTile) & 1, head, first) + 64 * quarter;
            live = p * kN + key < kv_total;
            uint32_t top = 0;
            if (live) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 a = reinterpret_cast<const uint4*>(row)[c];
                    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = unpack_half2(w[e]);
                        top = max(top, max(abs_bits(f.x), abs_bits(f.y)));
                    }
                }
            }
            if constexpr (kValue) {
                db = __float_as_uint(1.0f);
                tb = top;
            } else {
                db = top;
                t0 = 1.0f;
            }
        }
        if constexpr (kValue) {  // a key whose V is not finite is left out of the product, see the softmax
            const bool bad_key = tb >= 0x7F800000u;
            if (bad_key) { t0 = t1 = 0.0f; tb = 0u; live = false; }
            const uint32_t bad = __ballot_sync(0xffffffffu, bad_key);
            if (lane == 0) sm.poison[slot][dw] = bad;
            sm.vo[par][dt] = db >= 0x7F800000u ? 0.0f : d0;
        } else {
            tb = abs_bits(t0);
        }
        db = __reduce_max_sync(0xffffffffu, db);
        tb = __reduce_max_sync(0xffffffffu, tb);
        if (lane == 0) sm.red[par][kValue ? 1 : 0][dw] = make_uint2(db, tb);
        if (named_barrier_or(kValue ? 2 : 1, 32 * kDqWarps, failed)) return true;
#pragma unroll
        for (int w = 0; w < kDqWarps; w += 2) {
            const uint4 r = *reinterpret_cast<const uint4*>(&sm.red[par][kValue ? 1 : 0][w]);
            db = max(db, max(r.x, r.z));
            tb = max(tb, max(r.y, r.w));
        }
        float unit;  // 1 / scale of the page
        if constexpr (kValue) {
            const bool bad_dim = db >= 0x7F800000u;  // of every key
            const float top = __uint_as_float(tb) * (bad_dim ? 1.0f : __uint_as_float(db));
            if (top > 0.0f) v_run = max(v_run, scale_exponent(__float_as_uint(top)));
            const int v_exp = v_run == INT_MIN ? 0 : v_run;
            unit = pow2i(-v_exp);
            if (lane == 0) {
                if (dw == 0) sm.v_exp[slot] = v_exp;
                if (bad_dim) sm.poison[slot][dw] = 0xffffffffu;
                mbar_arrive(&sm.v_meta[par]);
            }
            // the buffer is free once P V(i-1) has completed
            if (i > 0 && !chunk_wait(&sm.o_done, (i - 1) & 1, &sm.abort_flag)) { failed = true; continue; }
        } else {
            const int k_exp = scale_exponent(__float_as_uint(__uint_as_float(db) * __uint_as_float(tb)));
            unit = t0 * pow2i(-k_exp);
            if (dt == 0) {
                sm.k_unit[slot] = pow2i(k_exp);
                sm.bad_page[slot] = sealed && m.page < 0;
            }
            // the buffer is free once S(i-1) has completed
            if (i > 0 && !chunk_wait(&sm.s_full[(i - 1) & 1], ((i - 1) >> 1) & 1, &sm.abort_flag)) { failed = true; continue; }
        }
        const F2 unit2(unit, unit);
        if (sealed) {
            const float z = t1 * unit, v0 = t0 * unit, v1 = v0 * 0.0625f, v2 = v1 * 0.0625f, v3 = v2 * 0.0625f, v4 = v3 * 0.0625f;
            const F2 z2(z, z), sc[4] = {F2(v0, v1), F2(v2, v3), F2(v4, v0), F2(v1, v2)};  // V: scale / 16^(nibble position)
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint4 cc = m.code[c >> 2];
                F2 x[4];
                unpack_f32((c & 3) == 0 ? cc.x : (c & 3) == 1 ? cc.y : (c & 3) == 2 ? cc.z : cc.w, x);
                const int at = 64 * quarter + 8 * c;
                if constexpr (kValue) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] = fma2(x[e], sc[e], z2);
                    const ulonglong2* ot = reinterpret_cast<const ulonglong2*>(&sm.vo[par][at]);
                    const ulonglong2 o0 = ot[0], o1 = ot[1];
                    x[0] = mul2(x[0], F2(o0.x)); x[1] = mul2(x[1], F2(o0.y));
                    x[2] = mul2(x[2], F2(o1.x)); x[3] = mul2(x[3], F2(o1.y));
                } else {
                    const ulonglong2* st = reinterpret_cast<const ulonglong2*>(&sm.ks[par][at]);
                    const ulonglong2* zt = reinterpret_cast<const ulonglong2*>(&sm.kz[par][at]);
                    const ulonglong2 s0 = st[0], s1 = st[1], z0 = zt[0], z1 = zt[1];
                    x[0] = mul2(fma2(x[0], F2(s0.x), F2(z0.x)), unit2); x[1] = mul2(fma2(x[1], F2(s0.y), F2(z0.y)), unit2);
                    x[2] = mul2(fma2(x[2], F2(s1.x), F2(z1.x)), unit2); x[3] = mul2(fma2(x[3], F2(s1.y), F2(z1.y)), unit2);
                }
                split_store(x, tile[0], tile[1], row_off + ((c ^ (key & 7)) << 4));
            }
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                F2 x[4];
                widen(live ? reinterpret_cast<const uint4*>(row)[c] : make_uint4(0u, 0u, 0u, 0u), unit2, x);
                split_store(x, tile[0], tile[1], row_off + ((c ^ (key & 7)) << 4));
            }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(kValue ? &sm.v_full : &sm.k_full);
    }
    return failed;
}

__global__ void __launch_bounds__(kThreads, 1) chunk256_kernel(const Chunk256Params P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Chunk256Smem& sm = *reinterpret_cast<Chunk256Smem*>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const LayerView& L = P.L;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mt = blockIdx.x, head = blockIdx.y, zs = blockIdx.z;
    const int G = L.q_heads / L.kv_heads;
    if (!P.after_append) grid_dependency_wait();
    const int kv_total = *P.total_pos + 1;

    if (warp == kMmaWarp) tc::tmem_alloc(&sm.tmem_base, kTmemCols);
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sm.s_full[b], 1);
            mbar_init(&sm.p_full[b], kSoftWarps);
            mbar_init(&sm.v_meta[b], kDqWarps);
        }
        mbar_init(&sm.k_full, kDqWarps);
        mbar_init(&sm.v_full, kDqWarps);
        mbar_init(&sm.o_done, 1);
        mbar_init(&sm.drain, 1);
        mbar_fence_init();
        sm.abort_flag = 0;
    }
    // ---- Q: rows rotated, scaled, split; one warp per row, lane l holds dims l + 32 j, the loads of four rows in flight
    constexpr int kQBatch = 4;
    for (int r0 = warp; r0 < kM; r0 += kQBatch * kWarps) {
        uint16_t raw[kQBatch][8];
        int rp[kQBatch];
#pragma unroll
        for (int u = 0; u < kQBatch; ++u) {
            const int r = r0 + u * kWarps, R = mt * kM + r, tq = R / G, gq = R % G;
            rp[u] = kNoRow;
#pragma unroll
            for (int j = 0; j < 8; ++j) raw[u][j] = 0;
            if (r < kM && tq < P.T) {
                const uint16_t* qrow = P.q + (static_cast<int64_t>(tq) * L.q_heads + head * G + gq) * D;
#pragma unroll
                for (int j = 0; j < 8; ++j) raw[u][j] = qrow[lane + 32 * j];
                rp[u] = max(P.pos[tq], -1);
            }
        }
#pragma unroll
        for (int u = 0; u < kQBatch; ++u) {
            const int r = r0 + u * kWarps;
            if (r >= kM) break;
            float v[8];
            uint32_t top = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = L.dtype == KVB_DTYPE_BF16 ? in_to_f32<true>(raw[u][j]) : in_to_f32<false>(raw[u][j]);
            hadamard_warp<D>(v, lane);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] *= P.scale_log2;
                top = max(top, abs_bits(v[j]));
            }
            const int e = scale_exponent(__reduce_max_sync(0xffffffffu, top));
            const float down = pow2i(-e);
            if (lane == 0) {
                sm.row_pos[r] = rp[u];
                sm.row_unit[r] = pow2i(e);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int d = lane + 32 * j;
                const uint32_t off = (d >> 6) * kQBlock + r * 128 + ((((d & 63) >> 3) ^ (r & 7)) << 4) + (d & 7) * 2;
                const float x = v[j] * down;
                const __half h = __float2half_rn(x);
                *reinterpret_cast<__half*>(sm.k[0] + off) = h;
                *reinterpret_cast<__half*>(sm.q_lo + off) = __float2half_rn(x - __half2float(h));
            }
        }
    }
    fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = sm.tmem_base;
    if (warp < kSoftWarps) {  // the high part of Q moves to tensor memory: thread = row, two dims per column
        const uint32_t lane_base = static_cast<uint32_t>(32 * warp) << 16;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            uint32_t w[32];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint4 x = *reinterpret_cast<const uint4*>(sm.k[0] + b * kQBlock + tid * 128 + ((c ^ (tid & 7)) << 4));
                w[4 * c] = x.x; w[4 * c + 1] = x.y; w[4 * c + 2] = x.z; w[4 * c + 3] = x.w;
            }
            tc::tmem_st32(tmem + kColQ + lane_base + 32 * b, w);
        }
        tc::tmem_st_wait();
    }
    int max_pos = -1, min_pos = INT_MAX;
#pragma unroll
    for (int i = 0; i < kM / 32; ++i) {
        const int p = sm.row_pos[lane + 32 * i];
        max_pos = max(max_pos, p);
        if (p != kNoRow) min_pos = min(min_pos, p);
    }
    max_pos = __reduce_max_sync(0xffffffffu, max_pos);
    min_pos = __reduce_min_sync(0xffffffffu, min_pos);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // pages this CTA walks: those a row of the tile can see, cut into ksplit ranges
    const int npages = max_pos < 0 ? 0 : min((kv_total + kN - 1) / kN, max_pos / kN + 1);
    const int p0 = static_cast<int>(static_cast<int64_t>(npages) * zs / P.ksplit);
    const int p1 = static_cast<int>(static_cast<int64_t>(npages) * (zs + 1) / P.ksplit);
    const int n = p1 - p0;
    bool failed = false;

    if (warp >= kSoftWarps && warp < kMmaWarp) {
        tc::regs_dec<kDqRegs>();
        if (P.after_append) grid_dependency_wait();
        const int dt = tid - 32 * kSoftWarps;
        if (dt < 32 * kDqWarps) failed = dequant_role<false>(sm, L, head, dt, p0, p1, kv_total);
        else failed = dequant_role<true>(sm, L, head, dt - 32 * kDqWarps, p0, p1, kv_total);
    } else if (warp >= kMmaWarp) {
        // =========================== MMA issue (one warp; the three beside it complete the warpgroup) ===========================
        tc::regs_dec<kMmaRegs>();
        if (warp == kMmaWarp) {
        constexpr uint32_t idesc_qk = tc::idesc_f16(kM, kN, false, false), idesc_pv = tc::idesc_f16(kM, D, false, true);
        const uint64_t q0 = tc::smem_desc(smem_u32(sm.q_lo), 16, 1024), k_hi = tc::smem_desc(smem_u32(sm.k[0]), 16, 1024), k_lo = tc::smem_desc(smem_u32(sm.k[1]), 16, 1024);
        const uint64_t v_hi = tc::smem_desc(smem_u32(sm.v[0]), kKvBlock, 1024), v_lo = tc::smem_desc(smem_u32(sm.v[1]), kKvBlock, 1024);
        for (int i = 0; i <= n && !failed; ++i) {
            if (i < n) {
                // S(i) goes where P(i-2) was: P V(i-2) has to be over
                if (!chunk_wait(&sm.k_full, i & 1, &sm.abort_flag) || (i > 1 && !chunk_wait(&sm.o_done, i & 1, &sm.abort_flag))) { failed = true; break; }
                tc::fence_after_sync();
                if (tc::elect_one()) {
                    const uint32_t s = tmem + 64 * (i & 1);
                    const uint64_t q = tc::desc_here(q0), kh = tc::desc_here(k_hi), kl = tc::desc_here(k_lo);
#pragma unroll
                    for (int b = 0; b < 4; ++b)  // 64 dims at a time
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            tc::mma_f16_ss(s, tc::desc_at(q, b * kQBlock + kk * 32), tc::desc_at(kh, b * kKvBlock + kk * 32), idesc_qk, b > 0 || kk > 0);
#pragma unroll
                    for (int b = 0; b < 4; ++b)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            tc::mma_f16_ts(s, tmem + kColQ + 32 * b + 8 * kk, tc::desc_at(kl, b * kKvBlock + kk * 32), idesc_qk, true);
#pragma unroll
                    for (int b = 0; b < 4; ++b)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            tc::mma_f16_ts(s, tmem + kColQ + 32 * b + 8 * kk, tc::desc_at(kh, b * kKvBlock + kk * 32), idesc_qk, true);
                    tc::commit(&sm.s_full[i & 1]);
                }
                __syncwarp();
            }
            if (i > 0) {
                const int j = i - 1;
                if (!chunk_wait(&sm.p_full[j & 1], (j >> 1) & 1, &sm.abort_flag) || !chunk_wait(&sm.v_full, j & 1, &sm.abort_flag)) { failed = true; break; }
                tc::fence_after_sync();
                if (tc::elect_one()) {
                    const uint32_t p = tmem + 64 * (j & 1);
                    const uint64_t vh = tc::desc_here(v_hi), vl = tc::desc_here(v_lo);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        tc::mma_f16_ts(tmem + kColO, p + 32 + 8 * kk, tc::desc_at(vh, kk * 2048), idesc_pv, j > 0 || kk > 0);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        tc::mma_f16_ts(tmem + kColO, p + 8 * kk, tc::desc_at(vl, kk * 2048), idesc_pv, true);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        tc::mma_f16_ts(tmem + kColO, p + 8 * kk, tc::desc_at(vh, kk * 2048), idesc_pv, true);
                    tc::commit(&sm.o_done);
                }
                __syncwarp();
            }
        }
        if (failed) {  // nothing of this CTA may still run when its tensor memory is given back
            if (tc::elect_one()) tc::commit(&sm.drain);
            __syncwarp();
            mbar_wait_bounded(&sm.drain, 0);
        }
        }
    } else {
        // =========================== softmax ===========================
        tc::regs_inc<kSoftRegs>();
        const uint32_t lane_base = static_cast<uint32_t>(32 * warp) << 16;
        const int my_pos = sm.row_pos[tid];
        const float row_unit = sm.row_unit[tid];
        const bool is_row = my_pos != kNoRow, warp_has_rows = __any_sync(0xffffffffu, is_row);
        float m_run = -INFINITY, l_run = 0.0f;
        int v_exp = 0;
        bool poisoned = false;
        for (int i = 0; i < n; ++i) {
            const int base = (p0 + i) * kN, slot = i & (kSlotsMeta - 1);
            if (!chunk_wait(&sm.v_meta[i & 1], (i >> 1) & 1, &sm.abort_flag) || !chunk_wait(&sm.s_full[i & 1], (i >> 1) & 1, &sm.abort_flag)) { failed = true; break; }
            tc::fence_after_sync();
            if (warp_has_rows) {
                const uint32_t ts = tmem + 64 * (i & 1) + lane_base;
                float s[kN];
                {
                    uint32_t r0[32], r1[32];
                    tc::tmem_ld32(ts, r0);
                    tc::tmem_ld32(ts + 32, r1);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        s[j] = __uint_as_float(r0[j]);
                        s[32 + j] = __uint_as_float(r1[j]);
                    }
                }
                const float unit = fmaxf(row_unit * sm.k_unit[slot], 1.175494351e-38f);  // > 0: a masked key stays at -inf
                const int v_new = sm.v_exp[slot];
                const bool bad_page = sm.bad_page[slot] != 0;
                if (base + kN - 1 > min_pos || base + kN > kv_total || bad_page) {
#pragma unroll
                    for (int j = 0; j < kN; ++j)
                        if (base + j > my_pos || base + j >= kv_total || bad_page) s[j] = -INFINITY;
                }
                {  // a key whose V is not finite was left out of the product: rows that see it end as NaN
                    const uint4 b0 = *reinterpret_cast<const uint4*>(&sm.poison[slot][0]), b1 = *reinterpret_cast<const uint4*>(&sm.poison[slot][4]);
                    const uint32_t lo = b0.x | b0.y | b0.z | b0.w, hi = b1.x | b1.y | b1.z | b1.w;
                    if ((lo | hi) != 0u && !bad_page) {
                        for (int j = 0; j < kN; ++j)
                            if (((j < 32 ? lo : hi) >> (j & 31) & 1u) && base + j <= my_pos && base + j < kv_total) poisoned = true;
                        __syncwarp();
                    }
                }
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int j = 0; j < kN; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], s[j]);
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * unit;
                constexpr float kLazy = 8.0f;  // the reference point moves only when the maximum has grown by more than 2^kLazy
                const bool grown = mx > m_run + kLazy || (m_run == -INFINITY && mx > -INFINITY);
                const float m_new = grown ? mx : m_run;
                const float m_use = m_new == -INFINITY ? 0.0f : m_new;
                float alpha = grown ? fast_exp2(m_run - m_use) : 1.0f;
                m_run = m_new;
                l_run *= alpha;
                bool moved = grown;
                if (v_new != v_exp) {  // the unit of V and O has grown: the sum so far is rescaled (powers of two: exact)
                    alpha *= pow2i(max(v_exp - v_new, -126));
                    v_exp = v_new;
                    moved = true;
                }
                const float off = kPBoost - m_use;
                const F2 unit2(unit, unit), off2(off, off);
                F2 sum[2] = {F2(0.0f, 0.0f), F2(0.0f, 0.0f)};
                uint32_t ph[32], pl[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const float2 e = fma2(F2(s[2 * j], s[2 * j + 1]), unit2, off2).get();
                    const F2 x(fast_exp2(e.x), fast_exp2(e.y));
                    sum[j & 1] = add2(sum[j & 1], x);
                    split2(x, ph[j], pl[j]);
                }
                tc::tmem_st32(ts, ph);
                tc::tmem_st32(ts + 32, pl);
                const float2 sum2 = add2(sum[0], sum[1]).get();
                l_run += sum2.x + sum2.y;
                if (i > 0 && __any_sync(0xffffffffu, moved)) {
                    if (!chunk_wait(&sm.o_done, (i - 1) & 1, &sm.abort_flag)) { failed = true; break; }
                    tc::fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < D / 32; ++c) {
                        uint32_t r[32];
                        tc::tmem_ld32(tmem + kColO + lane_base + 32 * c, r);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
                        tc::tmem_st32(tmem + kColO + lane_base + 32 * c, r);
                    }
                }
                tc::tmem_st_wait();
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_full[i & 1]);
        }
        // ---- partial of this (row tile, page range): m (log2 units), l, o
        // (P V(n-2) first: a parity wait must not be more than one phase ahead of its barrier)
        if (n > 1 && !failed && !chunk_wait(&sm.o_done, n & 1, &sm.abort_flag)) failed = true;
        if (n > 0 && !failed && !chunk_wait(&sm.o_done, (n - 1) & 1, &sm.abort_flag)) failed = true;
        tc::fence_after_sync();
        const bool have = n > 0 && !failed && __any_sync(0xffffffffu, m_run != -INFINITY), seen = have && m_run != -INFINITY;
        const int64_t idx = ((static_cast<int64_t>(head) * P.mtiles + mt) * P.ksplit + zs) * kM + tid;
        if (is_row) {
            P.ws_m[idx] = seen ? m_run - kPBoost : -INFINITY;
            P.ws_l[idx] = seen ? l_run : 0.0f;
        }
        const float unit = poisoned ? __uint_as_float(0x7FC00000u) : pow2i(v_exp);
        float* orow = P.ws_o + idx * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
            if (!warp_has_rows) break;
            __syncwarp();  // the load is the whole warp's: lanes without a row are back from the stores
            uint32_t r[32];
            if (have) {
                tc::tmem_ld32(tmem + kColO + lane_base + 32 * c, r);
                tc::tmem_ld_wait();
            }
            if (is_row) {
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4*>(orow + 32 * c + j) =
                        seen ? make_float4(__uint_as_float(r[j]) * unit, __uint_as_float(r[j + 1]) * unit, __uint_as_float(r[j + 2]) * unit, __uint_as_float(r[j + 3]) * unit)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    if (P.after_append) grid_dependency_wait();  // nobody leaves before the append is over: what waits for this grid finds both done
    if (failed && lane == 0) L.flag(KVB_ERR_WAIT_TIMEOUT);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) tc::tmem_dealloc(tmem, kTmemCols);
}

}  // namespace

// Chunk attention of `tokens` rows that are already appended, over a head_dim-256 cache.
int launch_chunk_attention_256(const kvb_layer* layer, const void* q, const int32_t* positions_dev, int tokens, float scale,
                               int kv_len_max, void* workspace, void* out, cudaStream_t s, float* part_m, float* part_l, float* part_o, const StepAppend* behind) {
    Chunk256Params P;
    P.L = make_view(*layer);
    P.q = static_cast<const uint16_t*>(q);
    P.pos = positions_dev;
    P.total_pos = positions_dev + (tokens - 1);
    P.T = tokens;
    const ChunkShape shape = chunk_shape_256(kv_len_max, layer->kv_heads, layer->q_heads, tokens, device_sm_count());
    P.mtiles = shape.mtiles;
    P.ksplit = shape.ksplit;
    P.scale_log2 = scale * 1.4426950408889634f;
    const size_t rows = static_cast<size_t>(layer->kv_heads) * P.mtiles * P.ksplit * kM;
    P.ws_m = workspace_base(workspace);
    P.ws_l = P.ws_m + rows;
    P.ws_o = P.ws_l + rows;
    P.after_append = starts_beside(behind, span_of(P.ws_m, partials_bytes(rows / kM, D)));
    const int smem = static_cast<int>(sizeof(Chunk256Smem)) + 1024;  // room to align the tiles to 1024 bytes
    static OncePerDevice opted;
    KVB_CUDA_OK(allow_smem(opted, chunk256_kernel, smem));
    const dim3 grid(P.mtiles, layer->kv_heads, P.ksplit);
    KVB_CUDA_OK(launch_early(chunk256_kernel, grid, dim3(kThreads), smem, s, P));
    return launch_chunk_merge<D>(P.ws_m, P.ws_l, P.ws_o, tokens, layer->q_heads, layer->kv_heads, P.mtiles, P.ksplit, layer->dtype, out,
                                 part_m, part_l, part_o, s);
}

}  // namespace kvb
