// kvb_prefill.cu -- chunk attention (prefill chunks, wide verify steps) over head_dim-128 caches on the 5th-generation
// tensor cores.
//
// The chunk's (token, q head) rows of one KV head are GQA-packed into row tiles of 128.  A CTA runs two streams, each with
// its own S, P and O in tensor memory and its own softmax warps, over 128-key tiles:
//   S = Q K^T   tcgen05.mma, A = Q tile and B = de-quantised K tile in shared memory (K-major, 128-byte swizzle),
//               accumulator S[128 x 128] fp32 in tensor memory;
//   softmax     thread r owns row r (= TMEM lane r): reads S in halves with tcgen05.ld, running max / sum in registers,
//               writes P (fp16) over the columns of S it has read, rescales O in tensor memory only when a row maximum moved;
//   O += P V    tcgen05.mma, A = P in tensor memory, B = de-quantised V tile (MN-major: one 128-byte row of 64 dims per key),
//               accumulator O[128 x 128] fp32 in tensor memory.
// kSplit false: the streams are two row tiles over the same keys (a de-quantised tile serves 256 rows).  kSplit true: one
// row tile, the streams take the even and the odd key tiles of the CTA's range.  A stream leaves a partial for the merge kernel, or,
// where the rows see one key range only, the CTA finishes them (finish_rows).
// One stream's MMAs run while the other's softmax does; each stream has a warp that issues them (one warp for both, which waited for one
// stream's hand-overs while the other's were due: 8-row verify step of a balanced cache of 100,003 tokens 62.0 us a layer, now 54.4).  With
// two row tiles a key tile is two parts of 64 keys, each with its own S and P: a stream's MMAs of one part run beside its softmax of the
// other (with one part and two issuing warps 1,024 tokens over 262,144 took 3.94 ms against 3.54).  Eight or sixteen warps de-quantise K and V
// straight from the planes into two-stage rings: nibbles -> fp16 with the exact unpack, then one fused multiply-add with the
// tile's per-dim (K) or the key's (V) fp16 scale and zero point.  Dims inside every group of eight are kept in the order the
// unpack yields (0,4,1,5,2,6,3,7); Q is written in the same order, so the contraction is unaffected, and what finishes a row
// (the merge kernel, finish_rows) puts the output dims back.  Keys of the open tile come un-quantised from the stage.
// Every wait on an mbarrier is bounded and also watches the CTA's abort flag; a wait that gives up sets
// KVB_ERR_WAIT_TIMEOUT and the CTA leaves through the normal exit (its MMAs are over, TMEM is freed).
#include <climits>

#include "kvb_chunk_merge.cuh"
#include "kvb_common.cuh"
#include "kvb_tcgen05.cuh"
#include "kvb_walk.hpp"

#include <cstddef>

namespace kvb {
namespace {

constexpr int D = 128;
constexpr int kM = 128;        // rows per row tile
constexpr int kN = 128;        // keys per step = one quantisation tile
constexpr int kStreams = 2;
// How the 28 warps are divided.  Two row tiles: the softmax is the longer part, its rows are cut into two column halves (a
// warp for each), eight warps de-quantise.  Split keys (a few rows): the de-quantising is, it gets sixteen warps.
template <bool kSplit> struct Roles {
    static constexpr int kHalves = kSplit ? 1 : 2;       // softmax warps per 32 rows of a stream, that share the columns of S and of O
    static constexpr int kParts = kSplit ? 1 : 2;        // parts of a key tile, each with its own S, P and hand-overs
    static constexpr int kSoft = 4 * kHalves;            // softmax warps per stream
    static constexpr int kDq = kSplit ? 8 : 4;           // for K, and again for V
    static constexpr int kDqWarp = kStreams * kSoft, kMmaWarp = kDqWarp + 2 * kDq;
    // Registers per thread: 72 at launch (64,512 a CTA), then by role 256 x 112 + 512 x 56 + 128 x 48 = 63,488 (split keys) or
    // 512 x 80 + 256 x 64 + 128 x 48 = 63,488.
    static constexpr int kSoftRegs = kSplit ? 112 : 80, kDqRegs = kSplit ? 56 : 64, kMmaRegs = 48;
};
constexpr int kWarps = 28, kThreads = 32 * kWarps;
constexpr int kTileBytes = kM * D * 2;
constexpr uint32_t kTmemCols = 512, kColO = 256;  // S of stream u at column 128 u, O at 256 + 128 u
constexpr int kSlotsMeta = 8;  // per-tile words handed to the softmax warps: a writer is at most six tiles ahead of a reader

struct PrefillParams {
    LayerView L;
    const uint16_t* q;         // [T][q_heads][D]
    const int32_t* pos;        // [T]
    const int32_t* total_pos;  // newest position in the cache
    int T, mtiles, ksplit;     // ksplit: partials per row
    bool after_append;         // beside the append of the rows (kvb_step.hpp): only the readers of the planes and the stage wait for it first
    float scale_log2;
    uint16_t* out;             // one key range: the finished rows [T][q_heads][D]; else null, and
    float* ws_m;               // [H][mtiles][ksplit][128]
    float* ws_l;
    float* ws_o;               // [H][mtiles][ksplit][128][D], dims in tile order
};

struct __align__(1024) PrefillSmem {
    uint8_t q[kStreams][kTileBytes];
    uint8_t k[2][kTileBytes];
    uint8_t v[2][kTileBytes];
    __half ks[2][D], kz[2][D], vo[2][D];  // per-dim factors by tile parity, in tile dim order
    uint32_t ko[2][kN];                   // other_K of the keys, twice
    uint64_t k_full[2], k_free[2], v_full[2], v_free[2], s_full[kStreams][2], p_full[kStreams][2], o_done[kStreams][2], drain[kStreams];  // [2]: part of a tile
    uint32_t tmem_base;
    int bad_tile[kSlotsMeta];
    int row_pos[kStreams][kM];
    float row_top[kStreams][2][2][kM];  // [part][half]: maximum of a row's columns, exchanged between its two softmax warps
    int abort_flag;
};

// Byte offset of element (row, col) in a [128 rows][128 cols] fp16 tile stored as two 64-column blocks of
// 128-byte rows, 8-row groups 1024 bytes apart, 16-byte chunks XOR-swizzled with the row (128-byte swizzle).
__device__ __forceinline__ uint32_t tile_off(int row, int col) {
    return (col >> 6) * 16384 + (row >> 3) * 1024 + (row & 7) * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4) + (col & 7) * 2;
}

__device__ __forceinline__ uint32_t hfma2_u32(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// What both de-quantising roles (kDqWarps warps each, thread dt) walk: the CTA's n tiles t0 .. t0 + n - 1, tile j into ring stage j & 1.
// Table entries are requested a tile before the fetch that needs them.
struct TilePages {
    const LayerView& L;
    const int32_t* tbl;
    int t0, n, sealed_tiles;
    int32_t ids[2];
    __device__ __forceinline__ TilePages(const LayerView& view, int first, int count, int kv_total)
        : L(view), tbl(view.table()), t0(first), n(count), sealed_tiles(kv_total / kN), ids{LayerView::kNoEntry, LayerView::kNoEntry} {}
    __device__ __forceinline__ bool sealed(int j) const { return t0 + j < sealed_tiles; }
    __device__ __forceinline__ void lookup(int j) {
        ids[0] = ids[1] = LayerView::kNoEntry;
        if (j < n && sealed(j)) {
            ids[0] = L.page_entry(tbl, 2 * (t0 + j));
            ids[1] = L.page_entry(tbl, 2 * (t0 + j) + 1);
        }
    }
};

// K: thread = the 16-byte chunk of eight dims dt % 16 of keys dt / 16, + kStep, ..: its dims' factors stay in registers for a tile, a warp
// reads the code rows of two keys at once and writes whole swizzled rows, and a store's address is a constant away from the last one's.
// Bound by its instructions (busy nine tenths of a step of split walks, three quarters with two row tiles).  Measured on B200 in graph replay against
// thread = key, which read both factors of every chunk from shared memory: 8 rows at 131,072 tokens 68.4 -> 62.6 us a layer, balanced at
// 100,003 54.4 -> 53.4; one call of 1,024 tokens over 262,144 3,465 -> 3,325 us.
// `other` (caches written with variance balancing): K is multiplied by the key's other_K, V by the per-dim other_V, reference
// kvarn128_codec.cuh:331-347; fp16 like the rest of this kernel.
template <bool kOther, int kDqWarps>
__device__ __forceinline__ bool dequant_k(PrefillSmem& sm, const LayerView& L, int head, int dt, int t0, int n, int kv_total) {
    constexpr int kStep = 2 * kDqWarps, kPer = kN / kStep, kPerPage = kPer / 2;
    const int lane = dt & 31, chunk = dt & 15, first = dt >> 4;
    TilePages T(L, t0, n, kv_total);
    struct Fetch {
        uint32_t code[kPer];
        __half d0, d1, t0;  // scale, zero point of dim dt; other_K of key dt
        bool bad;
    };
    const uint8_t* const code_at = L.k_code + page_head_offset(64, L.kv_heads, 0, head) + first * 64 + chunk * 4;
    const __half* const scales = L.k_scale + page_head_offset(5, L.kv_heads, 0, head);
    const __half* const tok_at = scales + (dt & 63) * 5 + 4;
    const __half* const dim_at = scales + ((dt & 127) >> 1) * 5 + (dt & 1);
    const int code_stride = 64 * kPage * L.kv_heads, scale_stride = 5 * kPage * L.kv_heads;
    auto fetch = [&](int j, Fetch& f) {
        const int32_t pg0 = L.checked_page(T.ids[0]), pg1 = L.checked_page(T.ids[1]);
        const bool here = pg0 >= 0 && pg1 >= 0;
        f.bad = !here && j < n && T.sealed(j);  // reported in the error word; the tile is masked
        f.d0 = f.d1 = f.t0 = __ushort_as_half(0);
        const uint8_t* src = code_at + static_cast<int64_t>(pg0) * code_stride;
        const uint8_t* src1 = code_at + static_cast<int64_t>(pg1) * code_stride;
#pragma unroll
        for (int i = 0; i < kPer; ++i) f.code[i] = here ? *reinterpret_cast<const uint32_t*>((i < kPerPage ? src : src1) + (i % kPerPage) * kStep * 64) : 0u;
        if (here && dt < D) {
            const __half* dim = dim_at + static_cast<int64_t>(pg0) * scale_stride;
            f.d0 = dim[0];
            f.d1 = dim[2];
            if constexpr (kOther) f.t0 = *(tok_at + static_cast<int64_t>(dt < kPage ? pg0 : pg1) * scale_stride);
        }
    };
    Fetch cur, nxt;
    if (n > 0) {
        T.lookup(0);
        fetch(0, nxt);
        T.lookup(1);
    }
    // chunk `chunk` of row `first` of a tile; the next row of this thread lies kStep / 8 groups of 1024 bytes further
    const uint32_t at = tile_off(first, 8 * chunk);
    bool failed = false;
    for (int j = 0; j < n; ++j) {
        const int st = j & 1;
        cur = nxt;
        fetch(j + 1, nxt);
        T.lookup(j + 2);
        if (dt < D) {
            sm.ks[st][dim_slot(dt)] = cur.d0;
            sm.kz[st][dim_slot(dt)] = cur.d1;
            if constexpr (kOther) sm.ko[st][dt] = __half_as_ushort(cur.t0) * 0x10001u;
        }
        if (dt == 0) sm.bad_tile[j & (kSlotsMeta - 1)] = cur.bad;
        if (named_barrier_or(1, 32 * kDqWarps, failed)) return true;
        // the stage is free once the MMAs of tile j - 2 have completed
        if (j > 1 && !chunk_wait(&sm.k_free[st], ((j >> 1) + 1) & 1, &sm.abort_flag)) {
            failed = true;
            continue;
        }
        uint8_t* const dst = sm.k[st] + at;
        if (T.sealed(j)) {
            const uint4 sc = *reinterpret_cast<const uint4*>(&sm.ks[st][8 * chunk]), zp = *reinterpret_cast<const uint4*>(&sm.kz[st][8 * chunk]);
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                uint32_t u[4];
                unpack8(cur.code[i], u);
                uint4 out = make_uint4(hfma2_u32(u[0], sc.x, zp.x), hfma2_u32(u[1], sc.y, zp.y), hfma2_u32(u[2], sc.z, zp.z), hfma2_u32(u[3], sc.w, zp.w));
                if constexpr (kOther) {
                    const uint32_t o2 = sm.ko[st][first + kStep * i];
                    out = make_uint4(hmul2_u32(out.x, o2), hmul2_u32(out.y, o2), hmul2_u32(out.z, o2), hmul2_u32(out.w, o2));
                }
                *reinterpret_cast<uint4*>(dst + i * (kStep / 8) * 1024) = out;
            }
        } else {  // un-quantised fp16 rows of the stage (dims re-ordered inside every group of eight)
            const int t = t0 + j;
            const __half* src = L.stage_row(0, t & 1, head, first) + 8 * chunk;
#pragma unroll 4
            for (int i = 0; i < kPer; ++i) {
                const uint4 r = t * kN + first + kStep * i < kv_total ? *reinterpret_cast<const uint4*>(src + i * kStep * D) : make_uint4(0u, 0u, 0u, 0u);
                *reinterpret_cast<uint4*>(dst + i * (kStep / 8) * 1024) =
                    make_uint4(prmt(r.x, r.z, 0x5410), prmt(r.x, r.z, 0x7632), prmt(r.y, r.w, 0x5410), prmt(r.y, r.w, 0x7632));
            }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.k_full[st]);
    }
    return failed;
}

// V: thread = a key (its scale and zero point in registers), 64 dims with eight warps, all 128 with four; threads 0 .. 127 also fetch the
// factor of dim dt.
template <bool kOther, int kDqWarps>
__device__ __forceinline__ bool dequant_v(PrefillSmem& sm, const LayerView& L, int head, int dt, int t0, int n, int kv_total) {
    constexpr int kWords = 64 / kDqWarps;  // 16-byte chunks of the tile row a thread writes
    const int lane = dt & 31, key = dt & 127, first = kDqWarps == 8 ? 64 * (dt >> 7) : 0;
    TilePages T(L, t0, n, kv_total);
    struct Fetch {
        uint4 code[kWords / 4];
        __half d0;    // other_V of the dim
        uint32_t sz;  // scale, zero point of the key
    };
    const uint8_t* const code_at = L.v_code + page_head_offset(64, L.kv_heads, 0, head) + (key & 63) * 64 + first / 2;
    const __half* const scales = L.v_scale + page_head_offset(4, L.kv_heads, 0, head);
    const __half* const tok_at = scales + (key & 63) * 4 + 2;
    const __half* const dim_at = scales + ((dt & 127) >> 1) * 4 + (dt & 1);
    const int code_stride = 64 * kPage * L.kv_heads, scale_stride = 4 * kPage * L.kv_heads;
    auto fetch = [&](Fetch& f) {
        const int32_t pg0 = L.checked_page(T.ids[0]), pg1 = L.checked_page(T.ids[1]), page = key < kPage ? pg0 : pg1;
        const bool here = pg0 >= 0 && pg1 >= 0;
        const uint4* src = reinterpret_cast<const uint4*>(code_at + static_cast<int64_t>(page) * code_stride);
#pragma unroll
        for (int c = 0; c < kWords / 4; ++c) f.code[c] = here ? src[c] : make_uint4(0u, 0u, 0u, 0u);
        f.sz = here ? *reinterpret_cast<const uint32_t*>(tok_at + static_cast<int64_t>(page) * scale_stride) : 0u;
        f.d0 = kOther && here && dt < D ? dim_at[static_cast<int64_t>(pg0) * scale_stride] : __ushort_as_half(0);
    };
    Fetch cur, nxt;
    if (n > 0) {
        T.lookup(0);
        fetch(nxt);
        T.lookup(1);
    }
    // row `key` of a tile, its 16-byte chunks exchanged as the 128-byte swizzle has them: chunk c lies at (at ^ 16 (c % 8)) in its block
    const uint32_t at = (key >> 3) * 1024 + (key & 7) * 128 + ((key & 7) << 4);
    bool failed = false;
    for (int j = 0; j < n; ++j) {
        const int st = j & 1;
        cur = nxt;
        fetch(nxt);
        T.lookup(j + 2);
        if constexpr (kOther) {
            if (dt < D) sm.vo[st][dim_slot(dt)] = cur.d0;
            if (named_barrier_or(2, 32 * kDqWarps, failed)) return true;
        }
        if (j > 1 && !chunk_wait(&sm.v_free[st], ((j >> 1) + 1) & 1, &sm.abort_flag)) {
            failed = true;
            if constexpr (!kOther) return true;
            continue;
        }
        uint8_t* const tile = sm.v[st] + (first >> 6) * 16384;
        auto put = [&](int c, uint4 x) { *reinterpret_cast<uint4*>(tile + (c >> 3) * 16384 + (at ^ ((c & 7) << 4))) = x; };
        if (T.sealed(j)) {
            const uint32_t s2 = prmt(cur.sz, cur.sz, 0x1010), z2 = prmt(cur.sz, cur.sz, 0x3232);
#pragma unroll
            for (int c = 0; c < kWords; ++c) {
                const uint4 cc = cur.code[c >> 2];
                uint32_t u[4];
                unpack8((c & 3) == 0 ? cc.x : (c & 3) == 1 ? cc.y : (c & 3) == 2 ? cc.z : cc.w, u);
                uint4 out = make_uint4(hfma2_u32(u[0], s2, z2), hfma2_u32(u[1], s2, z2), hfma2_u32(u[2], s2, z2), hfma2_u32(u[3], s2, z2));
                if constexpr (kOther) {
                    const uint4 ot = *reinterpret_cast<const uint4*>(&sm.vo[st][first + 8 * c]);
                    out = make_uint4(hmul2_u32(out.x, ot.x), hmul2_u32(out.y, ot.y), hmul2_u32(out.z, ot.z), hmul2_u32(out.w, ot.w));
                }
                put(c, out);
            }
        } else {
            const int t = t0 + j;
            const uint4* src = reinterpret_cast<const uint4*>(L.stage_row(1, t & 1, head, key) + first);
            const bool live = t * kN + key < kv_total;
#pragma unroll
            for (int c = 0; c < kWords; ++c) {
                const uint4 r = live ? src[c] : make_uint4(0u, 0u, 0u, 0u);
                put(c, make_uint4(prmt(r.x, r.z, 0x5410), prmt(r.x, r.z, 0x7632), prmt(r.y, r.w, 0x5410), prmt(r.y, r.w, 0x7632)));
            }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.v_full[st]);
    }
    return failed;
}

// One key range: the rows are finished here -- the two streams of a split walk merged, normalised, rotated back, stored --, no
// partials and no merge kernel (777 tokens alone, append included: 47.5 -> 35.9 us on B200; 19.4 MB of partials were written and
// read again, and a launch is gone).  Thread = row and a half of its dims (stream u of a split walk takes half u; `to`: the stream's O).
// The butterflies of strides 1 .. 16 run in registers, 32 dims at a time; those of 32 and 64 on values that meet in shared memory,
// [dim][row], where the K and V rings were.  Stages and roundings are those of hadamard_warp.
template <bool kSplit>
__device__ __forceinline__ void finish_rows(PrefillSmem& sm, const PrefillParams& P, uint32_t to, int u, int half, int row, int mt, int head, int G, bool is_row, bool seen,
                                            float m_run, float l_run, bool failed) {
    using Ro = Roles<kSplit>;
    constexpr int kFinishThreads = 32 * kStreams * Ro::kSoft;
    const int h = kSplit ? u : half;
    if constexpr (kSplit) {
        sm.row_top[u][0][0][row] = seen ? m_run : -INFINITY;
        sm.row_top[u][0][1][row] = seen ? l_run : 0.0f;
    }
    const int m = (kSplit ? mt : mt + u) * kM + row, tq = m / G, gq = m % G;
    uint16_t* const dst = P.out + (static_cast<int64_t>(tq) * P.L.q_heads + head * G + gq) * D + 16 * h;  // dims 16 h .. + 15 of every 32
    tc::fence_before_sync();
    // every P V of the CTA is over -- or a wait was given up: sums are missing, the de-quantising warps may still write where the
    // values would meet, and all rows of the CTA are zeros (the error word says why)
    if (named_barrier_or(11, kFinishThreads, failed)) {
#pragma unroll 1
        for (int c = 0; c < 8; ++c)
            if (is_row) *reinterpret_cast<uint4*>(dst + 8 * (c & 1) + 32 * (c >> 1)) = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    tc::fence_after_sync();
    float w[2] = {0.0f, 0.0f};  // weights of the streams' sums; a stream that saw no key has none
    bool used[2] = {seen, false};
    if constexpr (kSplit) {
        const float m0 = sm.row_top[0][0][0][row], m1 = sm.row_top[1][0][0][row], top = fmaxf(m0, m1);
        used[0] = m0 != -INFINITY;
        used[1] = m1 != -INFINITY;
        if (used[0]) w[0] = fast_exp2(m0 - top);
        if (used[1]) w[1] = fast_exp2(m1 - top);
        l_run = w[0] * sm.row_top[0][0][1][row] + w[1] * sm.row_top[1][0][1][row];
    } else {
        w[0] = 1.0f;
    }
    const float inv = l_run == 0.0f ? 0.0f : 1.0f / l_run;  // (a sum that is not a number stays one)
    w[0] *= inv;
    w[1] *= inv;
    const uint32_t o0 = (kSplit ? to - 128 * u : to) + 64 * h;
    float* const mine = reinterpret_cast<float*>(sm.k[0]) + (kSplit ? 0 : u) * (D * kM) + row;
    static_assert(sizeof(sm.k) + sizeof(sm.v) >= 2 * D * kM * 4 && offsetof(PrefillSmem, v) == offsetof(PrefillSmem, k) + sizeof(sm.k), "room for the rows");
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
        float v[32];
        {
            uint32_t r[32];
            __syncwarp();
            tc::tmem_ld32(o0 + 32 * c, r);
            tc::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = used[0] ? w[0] * __uint_as_float(r[e]) : 0.0f;  // (else columns no product was written to)
            if constexpr (kSplit) {
                tc::tmem_ld32(o0 + 128 + 32 * c, r);
                tc::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) v[e] += used[1] ? w[1] * __uint_as_float(r[e]) : 0.0f;
            }
        }
        float x[32];  // natural order
#pragma unroll
        for (int e = 0; e < 32; ++e) x[e] = v[(e & ~7) | ((e & 3) << 1) | ((e >> 2) & 1)];
#pragma unroll
        for (int span = 1; span <= 16; span <<= 1)
#pragma unroll
            for (int b = 0; b < 32; b += 2 * span)
#pragma unroll
                for (int e = 0; e < span; ++e) {
                    const float lo = x[b + e], hi = x[b + e + span];
                    x[b + e] = __fadd_rn(lo, hi);
                    x[b + e + span] = __fsub_rn(lo, hi);
                }
#pragma unroll
        for (int e = 0; e < 32; ++e) mine[(64 * h + 32 * c + e) * kM] = x[e];
    }
    named_barrier_sync(11, kFinishThreads);
    if (!is_row) return;
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {  // dims d .. d + 7 and those 32, 64, 96 further
        const int d = 16 * h + 8 * c;
        uint32_t o[4][4];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float a0 = mine[(d + e) * kM], a1 = mine[(d + e + 32) * kM], a2 = mine[(d + e + 64) * kM], a3 = mine[(d + e + 96) * kM];
            const float b0 = __fadd_rn(a0, a1), b1 = __fsub_rn(a0, a1), b2 = __fadd_rn(a2, a3), b3 = __fsub_rn(a2, a3);
            const float y[4] = {__fadd_rn(b0, b2), __fadd_rn(b1, b3), __fsub_rn(b0, b2), __fsub_rn(b1, b3)};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float z = __fmul_rn(y[k], 0.08838834764831845f);
                const uint32_t bits = P.L.dtype == KVB_DTYPE_BF16 ? f32_to_out<true>(z) : f32_to_out<false>(z);
                o[k][e >> 1] = e & 1 ? o[k][e >> 1] | bits << 16 : bits;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(dst + 8 * c + 32 * k) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
    }
}

template <bool kSplit, bool kOther>
__global__ void __launch_bounds__(kThreads, 1) chunk_kernel(const PrefillParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // the swizzled tiles need a 1024-byte aligned base; the launch reserves 1024 spare bytes for this
    PrefillSmem& sm = *reinterpret_cast<PrefillSmem*>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    using Ro = Roles<kSplit>;
    const LayerView& L = P.L;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int head = blockIdx.y, zs = blockIdx.z;
    constexpr int kDqWarps = Ro::kDq, kDqWarp = Ro::kDqWarp, kMmaWarp = Ro::kMmaWarp;
    static_assert(kMmaWarp + 4 == kWarps, "roles");
    constexpr int kRowTiles = kSplit ? 1 : 2;
    const int mt = kRowTiles * blockIdx.x;
    const int G = L.q_heads / L.kv_heads;
    if (!P.after_append) grid_dependency_wait();
    const int kv_total = *P.total_pos + 1;

    if (warp == kMmaWarp) tc::tmem_alloc(&sm.tmem_base, kTmemCols);
    if (tid == 0) {
        const int readers = !kSplit && (mt + 1) * kM < P.T * G ? 2 : 1;  // streams that read a tile
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sm.k_full[b], kDqWarps);
            mbar_init(&sm.v_full[b], kDqWarps);
            mbar_init(&sm.k_free[b], readers);
            mbar_init(&sm.v_free[b], readers);
            for (int h = 0; h < 2; ++h) {
                mbar_init(&sm.s_full[b][h], 1);
                mbar_init(&sm.p_full[b][h], Ro::kSoft);
                mbar_init(&sm.o_done[b][h], 1);
            }
            mbar_init(&sm.drain[b], 1);
        }
        mbar_fence_init();
        sm.abort_flag = 0;
    }
    // ---- Q: rows rotated, scaled, rounded to fp16, in tile dim order; rows beyond the chunk are zeros.  One warp per row, lane l
    //      holds dims l + 32 j, the loads of four rows in flight.
    constexpr int kQBatch = 4, kRows = kRowTiles * kM;
    for (int r0 = warp; r0 < kRows; r0 += kQBatch * kWarps) {
        uint16_t raw[kQBatch][4];
        int rp[kQBatch];
#pragma unroll
        for (int u = 0; u < kQBatch; ++u) {
            const int r = r0 + u * kWarps, R = mt * kM + r, tq = R / G, gq = R % G;
            rp[u] = kNoRow;
            raw[u][0] = raw[u][1] = raw[u][2] = raw[u][3] = 0;
            if (r < kRows && tq < P.T) {
                const uint16_t* qrow = P.q + (static_cast<int64_t>(tq) * L.q_heads + head * G + gq) * D;
#pragma unroll
                for (int j = 0; j < 4; ++j) raw[u][j] = qrow[lane + 32 * j];
                rp[u] = max(P.pos[tq], -1);
            }
        }
#pragma unroll
        for (int u = 0; u < kQBatch; ++u) {
            const int r = r0 + u * kWarps;
            if (r >= kRows) break;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = L.dtype == KVB_DTYPE_BF16 ? in_to_f32<true>(raw[u][j]) : in_to_f32<false>(raw[u][j]);
            if (rp[u] != kNoRow) hadamard_warp<D>(v, lane);  // warp-uniform: a row is real or not for the whole warp
            if (lane == 0) sm.row_pos[r >> 7][r & 127] = rp[u];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<__half*>(sm.q[r >> 7] + tile_off(r & 127, dim_slot(lane + 32 * j))) = __float2half_rn(v[j] * P.scale_log2);
        }
    }
    fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = sm.tmem_base;
    int max_pos = -1;
    for (int i = lane; i < kRows; i += 32) max_pos = max(max_pos, sm.row_pos[i >> 7][i & 127]);
    max_pos = __reduce_max_sync(0xffffffffu, max_pos);
    // key tiles this CTA walks: those a row can see, cut into ranges
    const int ranges = kSplit ? P.ksplit / 2 : P.ksplit;
    const int ntiles = max_pos < 0 ? 0 : min((kv_total + kN - 1) / kN, max_pos / kN + 1);
    const int t0 = static_cast<int>(static_cast<int64_t>(ntiles) * zs / ranges);
    const int n = static_cast<int>(static_cast<int64_t>(ntiles) * (zs + 1) / ranges) - t0;
    // stream u takes tiles u, u + 2, .. of the range (kSplit) or all of them for its row tile (none if it has no rows)
    auto steps_of = [&](int u) { return kSplit ? (n + 1 - u) / 2 : u == 0 || (mt + 1) * kM < P.T * G ? n : 0; };
    bool failed = false;

    if (warp >= kDqWarp && warp < kMmaWarp) {
        // =========================== de-quantise ===========================
        tc::regs_dec<Ro::kDqRegs>();
        if (P.after_append) grid_dependency_wait();
        const int dt = tid - 32 * kDqWarp;
        if (dt < 32 * kDqWarps) failed = dequant_k<kOther, kDqWarps>(sm, L, head, dt, t0, n, kv_total);
        else failed = dequant_v<kOther, kDqWarps>(sm, L, head, dt - 32 * kDqWarps, t0, n, kv_total);
    } else if (warp >= kMmaWarp) {
        // =========================== MMA issue (a warp a stream; the two beside them complete the warpgroup) ===========================
        tc::regs_dec<Ro::kMmaRegs>();
        const int u = warp - kMmaWarp;
        if (u < kStreams) {
            constexpr int kPart = kN / Ro::kParts;  // keys
            constexpr uint32_t idesc_qk = tc::idesc_f16(kM, kPart, false, false), idesc_pv = tc::idesc_f16(kM, D, false, true);
            const int steps = steps_of(u);
            const uint64_t q0 = tc::smem_desc(smem_u32(sm.q[kSplit ? 0 : u]), 16, 1024), k0 = tc::smem_desc(smem_u32(sm.k[0]), 16, 1024), v0 = tc::smem_desc(smem_u32(sm.v[0]), 16384, 1024);
            for (int i = 0; i <= steps && steps > 0 && !failed; ++i) {
                const int jk = kSplit ? 2 * i + u : i, jv = kSplit ? 2 * (i - 1) + u : i - 1;
                // V of step i - 1 and K of step i are there well before P: waited for first, off the chain P -> PV -> S
                if (i < steps && !chunk_wait(&sm.k_full[jk & 1], (jk >> 1) & 1, &sm.abort_flag)) { failed = true; break; }
                if (i > 0 && !chunk_wait(&sm.v_full[jv & 1], (jv >> 1) & 1, &sm.abort_flag)) { failed = true; break; }
#pragma unroll
                for (int h = 0; h < Ro::kParts; ++h) {
                    const uint32_t s = tmem + 128 * u + kPart * h;  // S of the part, then its P
                    if (i > 0) {  // O_u += P V of the stream's step i - 1
                        if (!chunk_wait(&sm.p_full[u][h], (i - 1) & 1, &sm.abort_flag)) { failed = true; break; }
                        tc::fence_after_sync();
                        if (tc::elect_one()) {
                            const uint64_t v = tc::desc_at(tc::desc_here(v0), (jv & 1) * kTileBytes + h * (kPart / 16) * 2048);
#pragma unroll
                            for (int kk = 0; kk < kPart / 16; ++kk)  // 16 keys = 8 columns of P
                                tc::mma_f16_ts(tmem + kColO + 128 * u, s + 8 * kk, tc::desc_at(v, kk * 2048), idesc_pv, i > 1 || h > 0 || kk > 0);
                            tc::commit(&sm.o_done[u][h]);
                            if (h == Ro::kParts - 1) tc::commit(&sm.v_free[jv & 1]);
                        }
                        __syncwarp();
                        // the next S_u is written over this P
                        if (!chunk_wait(&sm.o_done[u][h], (i - 1) & 1, &sm.abort_flag)) { failed = true; break; }
                    }
                    if (i < steps) {
                        tc::fence_after_sync();
                        if (tc::elect_one()) {
                            const uint64_t q = tc::desc_here(q0), k = tc::desc_at(tc::desc_here(k0), (jk & 1) * kTileBytes + h * kPart * 128);
#pragma unroll
                            for (int kk = 0; kk < 8; ++kk) {
                                const int o = (kk >> 2) * 16384 + (kk & 3) * 32;
                                tc::mma_f16_ss(s, tc::desc_at(q, o), tc::desc_at(k, o), idesc_qk, kk > 0);
                            }
                            tc::commit(&sm.s_full[u][h]);
                            if (h == Ro::kParts - 1) tc::commit(&sm.k_free[jk & 1]);
                        }
                        __syncwarp();
                    }
                }
            }
            if (failed) {  // nothing of this CTA may still run when its tensor memory is given back
                if (tc::elect_one()) tc::commit(&sm.drain[u]);
                __syncwarp();
                mbar_wait_bounded(&sm.drain[u], 0);
            }
        }
    } else {
        // =========================== softmax of stream u ===========================
        tc::regs_inc<Ro::kSoftRegs>();
        const int u = warp / Ro::kSoft, half = (warp % Ro::kSoft) >> 2, row = tid & 127;
        const uint32_t lane_base = static_cast<uint32_t>(32 * (warp & 3)) << 16;
        constexpr int kCols = D / Ro::kHalves;                     // columns of O this warp works on, from column kCols * half
        constexpr int kKeys = kN / Ro::kParts / Ro::kHalves;       // columns of S of a part, from kKeys * half
        const uint32_t to = tmem + kColO + 128 * u + kCols * half + lane_base;
        const int my_pos = kSplit ? sm.row_pos[0][row] : sm.row_pos[u][row];
        const bool is_row = my_pos != kNoRow, warp_has_rows = __any_sync(0xffffffffu, is_row);
        const int min_pos = __reduce_min_sync(0xffffffffu, is_row ? my_pos : INT_MAX);
        const int steps = steps_of(u);
        float m_run = -INFINITY, l_run = 0.0f;
        for (int i = 0; i < steps && !failed; ++i) {
            const int j = kSplit ? 2 * i + u : i;
#pragma unroll 1
            for (int h = 0; h < Ro::kParts; ++h) {
                const int base = (t0 + j) * kN + (kN / Ro::kParts) * h + kKeys * half;
                // P of the two warps lies side by side over S of the part, which both have read when they meet
                const uint32_t ts = tmem + 128 * u + (kN / Ro::kParts) * h + kKeys * half + lane_base, tp = ts - (Ro::kHalves == 2 ? kKeys / 2 * half : 0);
                if (leaves_alone<Ro::kHalves == 2>(failed, chunk_wait(&sm.s_full[u][h], i & 1, &sm.abort_flag), warp_has_rows)) break;
                tc::fence_after_sync();
                if (warp_has_rows) {
                    const bool bad_tile = sm.bad_tile[j & (kSlotsMeta - 1)] != 0;
                    const bool masked = base + kKeys - 1 > min_pos || base + kKeys > kv_total || bad_tile;
                    const int lim = bad_tile || !is_row ? -1 : min(my_pos, kv_total - 1) - base;  // last visible of this warp's keys
                    auto mask = [&](uint32_t (&s)[32], int first) {                    // keys the row may not see at -inf
                        if (masked) {
#pragma unroll
                            for (int e = 0; e < 32; ++e)
                                if (first + e > lim) s[e] = 0xFF800000u;
                        }
                    };
                    auto top = [&](const uint32_t (&s)[32]) {
                        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                        for (int e = 0; e < 32; ++e) mx[e & 3] = fmaxf(mx[e & 3], __uint_as_float(s[e]));
                        return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                    };
                    // With split keys a row of S is read twice, 32 columns at a time: for its maximum, and for the exponentials.  What is read
                    // last for the maximum stays in registers and is exponentiated first: P goes over columns already read.
                    uint32_t s0[32], s1[Ro::kHalves == 1 ? 32 : 1];
                    float mx;
                    if constexpr (Ro::kHalves == 1) {
                        tc::tmem_ld32(ts + 64, s0);
                        tc::tmem_ld32(ts + 96, s1);
                        tc::tmem_ld_wait();
                        mask(s0, 64);
                        mask(s1, 96);
                        mx = fmaxf(top(s0), top(s1));
                        tc::tmem_ld32(ts, s0);
                        tc::tmem_ld32(ts + 32, s1);
                        tc::tmem_ld_wait();
                        mask(s0, 0);
                        mask(s1, 32);
                        mx = fmaxf(mx, fmaxf(top(s0), top(s1)));
                    } else {
                        static_assert(Ro::kHalves == 1 || kKeys == 32, "columns of a warp");
                        tc::tmem_ld32(ts, s0);
                        tc::tmem_ld_wait();
                        mask(s0, 0);
                        mx = top(s0);
                        sm.row_top[u][h][half][row] = mx;
                        if (leaves_together(failed, named_barrier_or(3 + 4 * u + (warp & 3), 64, failed))) break;  // the two warps of these 32 rows
                        mx = fmaxf(mx, sm.row_top[u][h][half ^ 1][row]);
                    }
                    // The reference point of the row's exponentials follows the running maximum lazily: it moves only when the
                    // maximum has grown by more than 2^kLazy, so P stays below 2^kLazy (exact enough in fp16, whose precision is
                    // relative) and the O accumulator is rescaled a few times per walk instead of at every new maximum.
                    constexpr float kLazy = 8.0f;
                    const bool grown = mx > m_run + kLazy || (m_run == -INFINITY && mx > -INFINITY);
                    const float m_new = grown ? mx : m_run;
                    const float m_use = m_new == -INFINITY ? 0.0f : m_new;
                    const float alpha = grown ? fast_exp2(m_run - m_use) : 1.0f;
                    m_run = m_new;
                    F2 sum[2] = {F2(0.0f, 0.0f), F2(0.0f, 0.0f)};
                    const F2 off(-m_use, -m_use);
                    auto weights = [&](const uint32_t (&s)[32], int c) {  // exponentials of columns 32 c .. -> 16 columns of P
                        uint32_t pk[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            const float2 a = add2(F2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), off).get();
                            const float p0 = fast_exp2(a.x), p1 = fast_exp2(a.y);
                            sum[e & 1] = add2(sum[e & 1], F2(p0, p1));
                            pk[e] = pack_half2(p0, p1);
                        }
                        tc::tmem_st16(tp + 16 * c, pk);
                    };
                    weights(s0, 0);
                    if constexpr (Ro::kHalves == 1) {
                        weights(s1, 1);
#pragma unroll 1
                        for (int c = 2; c < 4; ++c) {  // (unrolled, the two loads cost spills)
                            tc::tmem_ld32(ts + 32 * c, s0);
                            tc::tmem_ld_wait();
                            mask(s0, 32 * c);
                            weights(s0, c);
                        }
                    }
                    const float2 sum2 = add2(sum[0], sum[1]).get();
                    l_run = l_run * alpha + (sum2.x + sum2.y);
                    if (i + h > 0 && __any_sync(0xffffffffu, grown)) {
                        // P V of step i - 1 completed before S of step i was issued; that of this step's first part may still run
                        if (h > 0) chunk_wait(&sm.o_done[u][0], i & 1, &sm.abort_flag);
                        if (Ro::kParts == 2 && h == 0) chunk_wait(&sm.o_done[u][1], (i - 1) & 1, &sm.abort_flag);
                        tc::fence_after_sync();
#pragma unroll 1
                        for (int c = 0; c < kCols / 32; ++c) {
                            uint32_t r[32];
                            tc::tmem_ld32(to + 32 * c, r);
                            tc::tmem_ld_wait();
#pragma unroll
                            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
                            tc::tmem_st32(to + 32 * c, r);
                        }
                    }
                    tc::tmem_st_wait();
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.p_full[u][h]);
            }
        }
        // ---- partial of this (row tile, key range): m (log2 units), l, o in tile dim order
        // (a wait ahead of a rescaling that was given up by a warp of this stream raised the flag before its last P was handed over)
#pragma unroll
        for (int h = 0; h < Ro::kParts; ++h)
            if (steps > 0 && !failed && !chunk_wait<Ro::kHalves == 2>(&sm.o_done[u][h], (steps - 1) & 1, &sm.abort_flag)) failed = true;
        tc::fence_after_sync();
        if constexpr (Ro::kHalves == 2) {  // a row's sum has two halves; a warp that gave up comes here too
            sm.row_top[u][0][half][row] = l_run;
            named_barrier_sync(3 + 4 * u + (warp & 3), 64);
            l_run += sm.row_top[u][0][half ^ 1][row];
        }
        const bool have = steps > 0 && !failed && __any_sync(0xffffffffu, m_run != -INFINITY), seen = have && m_run != -INFINITY;
        if (P.out != nullptr) {
            finish_rows<kSplit>(sm, P, to - kCols * half, u, half, row, mt, head, G, is_row, seen, m_run, l_run, failed);
        } else {
            const int tile = kSplit ? mt : mt + u, part = kSplit ? 2 * zs + u : zs;
            const int64_t idx = ((static_cast<int64_t>(head) * P.mtiles + tile) * P.ksplit + part) * kM + row;
            if (is_row && half == 0) {
                P.ws_m[idx] = seen ? m_run : -INFINITY;
                P.ws_l[idx] = seen ? l_run : 0.0f;
            }
            float* orow = P.ws_o + idx * D + kCols * half;
#pragma unroll 1
            for (int c = 0; c < kCols / 32; ++c) {
                if (!warp_has_rows) break;
                __syncwarp();  // the load is the whole warp's: lanes without a row are back from the stores
                uint32_t r[32];
                if (have) {
                    tc::tmem_ld32(to + 32 * c, r);
                    tc::tmem_ld_wait();
                }
                if (is_row) {
#pragma unroll
                    for (int e = 0; e < 32; e += 4)
                        *reinterpret_cast<float4*>(orow + 32 * c + e) =
                            seen ? make_float4(__uint_as_float(r[e]), __uint_as_float(r[e + 1]), __uint_as_float(r[e + 2]), __uint_as_float(r[e + 3]))
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
                }
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
}  // namespace kvb

namespace kvb {
// kvb_chunk256.cu: the same for head_dim 256
int launch_chunk_attention_256(const kvb_layer* layer, const void* q, const int32_t* positions_dev, int tokens, float scale,
                               int kv_len_max, void* workspace, void* out, cudaStream_t s, float* part_m, float* part_l, float* part_o, const StepAppend* behind);
}  // namespace kvb

extern "C" size_t kvb_prefill_workspace_bytes(int kv_len_max, int kv_heads, int q_heads, int head_dim, int tokens) {
    if (kv_heads < 1 || q_heads < kv_heads || tokens < 1) return 0;
    return kvb::partials_bytes(kvb::most_partials(head_dim, kv_len_max, kv_heads, q_heads, tokens, kvb::device_sm_count()), head_dim) + kvb::kWorkspaceSlack;
}

namespace kvb {
// Chunk attention of `tokens` rows that are already appended (shared by the prefill and the verify entry points).
int launch_chunk_attention(const kvb_layer* layer, const void* q, const int32_t* positions_dev, int tokens, float scale,
                           int kv_len_max, void* workspace, void* out, cudaStream_t s, float* part_m, float* part_l,
                           float* part_o, const int32_t* total_pos_dev, const StepAppend* behind) {
    PrefillParams P;
    P.L = make_view(*layer);
    P.q = static_cast<const uint16_t*>(q);
    P.pos = positions_dev;
    P.total_pos = total_pos_dev != nullptr ? total_pos_dev : positions_dev + (tokens - 1);
    P.T = tokens;
    const ChunkShape shape = chunk_shape_128(kv_len_max, layer->kv_heads, layer->q_heads, tokens, device_sm_count());
    P.mtiles = shape.mtiles;
    P.ksplit = shape.ksplit;
    P.scale_log2 = scale * 1.4426950408889634f;
    const size_t rows = static_cast<size_t>(layer->kv_heads) * P.mtiles * P.ksplit * kM;
    P.ws_m = workspace_base(workspace);
    P.ws_l = P.ws_m + rows;
    P.ws_o = P.ws_l + rows;
    // One key range needs no merge.  The rows are stored 16 bytes at a time, and while other CTAs still read q and the positions: an
    // output that starts elsewhere, or shares memory with them, takes the merge kernel's route.
    const size_t out_bytes = static_cast<size_t>(tokens) * layer->q_heads * D * sizeof(uint16_t);
    const bool finish = shape.ranges == 1 && part_m == nullptr && (reinterpret_cast<uintptr_t>(out) & 15u) == 0 &&
                        stores_beside(span_of(out, out_bytes), span_of(q, out_bytes), span_of(positions_dev, tokens * sizeof(int32_t)), span_of(P.total_pos, sizeof(int32_t)));
    P.out = finish ? static_cast<uint16_t*>(out) : nullptr;
    P.after_append = starts_beside(behind, finish ? span_of(out, out_bytes) : span_of(P.ws_m, partials_bytes(rows / kM, D)));
    const int smem = static_cast<int>(sizeof(PrefillSmem)) + 1024;  // room to align the tiles to 1024 bytes
    const bool other = layer->sinkhorn_iters > 0;
    const auto kernel = shape.split ? (other ? chunk_kernel<true, true> : chunk_kernel<true, false>) : (other ? chunk_kernel<false, true> : chunk_kernel<false, false>);
    static OncePerDevice opted[4];
    KVB_CUDA_OK(allow_smem(opted[2 * shape.split + other], kernel, smem));
    const dim3 grid(shape.split ? shape.mtiles : (shape.mtiles + 1) / 2, layer->kv_heads, shape.ranges);
    KVB_CUDA_OK(launch_early(kernel, grid, dim3(kThreads), smem, s, P));
    if (P.out != nullptr) return KVB_OK;
    return launch_chunk_merge<D>(P.ws_m, P.ws_l, P.ws_o, tokens, layer->q_heads, layer->kv_heads, P.mtiles, P.ksplit, layer->dtype, out,
                                 part_m, part_l, part_o, s);
}
}  // namespace kvb

extern "C" int kvb_attn_prefill(const kvb_layer* layer, const void* q, const void* k, const void* v,
                                const int32_t* positions_dev, int tokens, float scale, int kv_len_max, void* workspace,
                                void* out, void* stream) {
    using namespace kvb;
    if (int st = check_layer(layer, "kvb_attn_prefill")) return st;
    if (tokens < 1) return fail(KVB_EINVAL, "kvb_attn_prefill: tokens = %d", tokens);
    if (q == nullptr || workspace == nullptr || out == nullptr) return fail(KVB_EINVAL, "kvb_attn_prefill: null q / workspace / out");
    if (layer->stage == nullptr) return fail(KVB_EINVAL, "kvb_attn_prefill: layer has no stage buffer");
    if (tokens > 65535) return fail(KVB_ERANGE, "kvb_attn_prefill: %d tokens in one chunk (at most 65535)", tokens);
    if (int st = kvb_append(layer, k, v, positions_dev, tokens, stream)) return st;
    const StepAppend step = step_append(*layer, k, v, positions_dev, tokens);
    if (layer->head_dim != 128)
        return launch_chunk_attention_256(layer, q, positions_dev, tokens, scale, kv_len_max, workspace, out, static_cast<cudaStream_t>(stream),
                                          nullptr, nullptr, nullptr, &step);
    return launch_chunk_attention(layer, q, positions_dev, tokens, scale, kv_len_max, workspace, out, static_cast<cudaStream_t>(stream),
                                  nullptr, nullptr, nullptr, nullptr, &step);
}
