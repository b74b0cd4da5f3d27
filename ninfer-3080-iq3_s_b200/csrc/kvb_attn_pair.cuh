// kvb_attn_pair.cuh -- the CTA of decode and verify steps at head_dim 256: the loop of attn_cta (kvb_attn.cu, whose types and helpers
// this uses) with two warps a page, one for each 128-dim slice.
//
// Sixteen warps are eight pairs.  A pair streams its pages through one ring of two 8 KB slots; each warp multiplies the queries with its
// slice of K, the partial logits meet in shared memory, both warps work out the same weights, and each takes its slice of V.  Two
// barriers of the pair a page: where the logits meet (K has been read by both: its slot is refilled) and behind V.  A query element is
// 22-bit fixed point against the largest of its row and slice, a weight 23 bits against the page's largest scale of the slice (three
// bytes each, as much as the fp32 sums they enter keep).
//
// Bound by instruction issue (1,490 warp instructions a page and warp, 52 % of the issue slots at 131,072 tokens; next the fixed latencies
// and the pair's barriers).  One warp for both slices ran twice the straight-line code a page, on eight warps of 255 registers, and
// waited for instructions (21 .. 32 % of the issue slots).  Measured on B200 in graph replay, 24 / 4 heads, balanced bf16 cache, a layer,
// one warp a page against two: decode at 30,011 tokens 22.5 -> 21.4 us, at 131,072 46.2 -> 45.2, verify at 20,000 tokens of 2 / 4 / 5 rows
// 28.8 / 33.8 / 39.2 -> 25.8 / 30.2 / 35.5, 5 rows at 131,000 174 -> 157.  Sums of the MMAs that start at the bits of 2^23, which
// need no conversion, took 1 .. 4 % longer in the V products and 9 % in the K products (four moves for every MMA that starts a sum).
#pragma once

namespace kvb {
namespace {

constexpr int kPairs = 8, kPairWarps = 2 * kPairs;
struct Pair {
    static constexpr int kChunk = kPage * 128;  // the K or the V codes of one page
    static constexpr int kHdrV = 1024, kHdrK = 1280, kHdr = kHdrV + kHdrK;  // V scale rows of the page, then the K scale rows
    static constexpr int kSubs = 8, kSubBytes = kChunk / kSubs, kShift = 16;  // V: sub-blocks of 8 keys, each shifted further (bank groups, see VSlot)
    static constexpr int kSlot = (kChunk + (kSubs - 1) * kShift + 127) / 128 * 128;
    static constexpr int kTab = 256 + 8 * kTabPad;
    static constexpr float kQMax = 4194000.0f;   // largest query integer
    static constexpr float kPMagic = 8388608.0f;  // weights are >= 0: 2^23 leaves 23 bits
    static constexpr float kPMax = 8380000.0f;   // largest weight
    // Key of m-row g (+ 8: kKeyH further) of 16-key group grp: 8 g + key_grp(grp); see attn_cta.
    static constexpr int kKeyH = 1;
    static __device__ __forceinline__ constexpr int key_grp(int grp) { return 4 * (grp >> 1) + 2 * (grp & 1); }
};

struct __align__(128) PairRing {
    uint8_t slots[kSlots][Pair::kSlot];
    uint8_t hdr[kHdrs][Pair::kHdr];
    float scale_k[Pair::kTab], zp_k[Pair::kTab];  // per-dim scale / zero point of K for the tile in work: dim d at d + kTabPad * (d / 32)
};

struct __align__(128) PairSmem {
    PairRing ring[kPairs];       // in the end the merge buffer of the warps
    float4 swap[kPairs][2][4][32];     // logits over a slice: [pair][slice][16-key group][lane]; in the end the partial of a cluster's CTA
    uint64_t bars[kPairs][kSlots];     // outside the rings, see AttnSmem
    float4 qfrag[16][32];              // q' in per-lane fragment order: [8 slice + j][lane] = dims 128 slice + 32 t + 4 j .. + 3 of row g
    int row_pos[kRows];
    int poison[2][kRows];              // the row sees a key whose V (in this slice) is not finite
};
struct PairPart {  // the partial of a CTA whose cluster merges it
    float o[8][256];
    float m[8], l[8];
};
static_assert(sizeof(PairPart) <= sizeof(PairSmem::swap), "room for the partial");

// Values that are not finite.  A weight of zero does not keep an infinite V away from the rows that may not see its
// key: V enters the products clamped to finite values, and the rows that do see such a key are marked and end as NaN.
__device__ __forceinline__ bool nonfinite_half2(uint32_t w) { return (((w & 0x7C007C00u) + 0x04000400u) & 0x80008000u) != 0u; }
__device__ __forceinline__ uint32_t finite_half2(uint32_t w) {  // the same bits, or +-65504 in the place of an infinity or a NaN
    asm("max.f16x2 %0, %0, %1;" : "+r"(w) : "r"(0xFBFFFBFFu));
    asm("min.f16x2 %0, %0, %1;" : "+r"(w) : "r"(0x7BFF7BFFu));
    return w;
}
// Marks the rows that see one of the keys first + i, bit i of `keys`, i < 64.
__device__ __forceinline__ void poison_rows(int* poison, const int* row_pos, int lane, uint64_t keys, int first, int key_begin, int key_end) {
    if (lane >= kRows) return;
    const int lo = max(key_begin - first, 0), hi = min(min(key_end - 1, row_pos[lane]) - first, 63);
    if (lo <= hi && ((keys >> lo) << (63 - hi + lo)) != 0) poison[lane] = 1;
}
// The same for 16 V rows of the open tile (lanes 0 .. 15 look at slice 0, 16 .. 31 at slice 1).
__device__ __noinline__ void poison_stage_group(const __half* vrow, int (*poison)[kRows], const int* row_pos, int lane, int first, int kv_total, int key_begin, int key_end) {
    uint32_t keys[2] = {0u, 0u};
#pragma unroll 1
    for (int key = 0; key < 16 && first + key < kv_total; ++key) {
        const uint4 r = *reinterpret_cast<const uint4*>(vrow + key * 256 + 8 * lane);
        const uint32_t hit = __ballot_sync(0xffffffffu, nonfinite_half2(r.x) || nonfinite_half2(r.y) || nonfinite_half2(r.z) || nonfinite_half2(r.w));
        if (hit & 0x0000FFFFu) keys[0] |= 1u << key;
        if (hit & 0xFFFF0000u) keys[1] |= 1u << key;
    }
    for (int s = 0; s < 2; ++s) poison_rows(poison[s], row_pos, lane, keys[s], first, key_begin, key_end);
}

// Integer form of (q' * scale_K)^T of one slice, see QInt.  The third byte of an integer is signed.
struct PairQInt {
    uint32_t b[2][2][3][2];
    float f[2];   // row scale / 16 of the lane's rows 2t, 2t+1
    float qz[2];  // sum_d q'[row][d] * zp_K[d]
};
__device__ __forceinline__ void build_pair_qint(const PairSmem& sm, const PairRing& R, int s, int lane, PairQInt& f) {
    const int t = lane & 3;
    const float* const kt = &R.scale_k[(32 + kTabPad) * (4 * s + t)];
    const float* const zt = &R.zp_k[(32 + kTabPad) * (4 * s + t)];
    F2 qs[16], qz2(0.0f, 0.0f);
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float4 qv = sm.qfrag[8 * s + j][lane], ks = *reinterpret_cast<const float4*>(kt + 4 * j), kz = *reinterpret_cast<const float4*>(zt + 4 * j);
        const F2 q0(qv.x, qv.y), q1(qv.z, qv.w);
        qs[2 * j] = mul2(q0, F2(ks.x, ks.y));
        qs[2 * j + 1] = mul2(q1, F2(ks.z, ks.w));
        qz2 = fma2(q0, F2(kz.x, kz.y), qz2);
        qz2 = fma2(q1, F2(kz.z, kz.w), qz2);
        const float2 a = qs[2 * j].get(), b = qs[2 * j + 1].get();
        amax = fmaxf(fmaxf(amax, fmaxf(fabsf(a.x), fabsf(a.y))), fmaxf(fabsf(b.x), fabsf(b.y)));
    }
    float qz = qz2.get().x + qz2.get().y;
    qz += __shfl_xor_sync(0xffffffffu, qz, 1);
    qz += __shfl_xor_sync(0xffffffffu, qz, 2);  // every lane of group g now holds qz of row g
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float fr = amax > 0.0f ? amax * (1.0f / Pair::kQMax) : 1.0f, inv = amax > 0.0f ? Pair::kQMax / amax : 0.0f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {  // row 2t + j lives in lanes 4 * (2t + j) ..
        f.qz[j] = __shfl_sync(0xffffffffu, qz, 8 * t + 4 * j);
        f.f[j] = __shfl_sync(0xffffffffu, fr, 8 * t + 4 * j) * 0.0625f;
    }
    uint32_t x[32];
#pragma unroll
    for (int i = 0; i < 16; ++i) {  // low 22 bits: Qi (two's complement)
        const float2 y = fma2(qs[i], F2(inv, inv), F2(kMagic, kMagic)).get();
        x[2 * i] = __float_as_uint(y.x);
        x[2 * i + 1] = __float_as_uint(y.y);
    }
#pragma unroll
    for (int kb = 0; kb < 2; ++kb)
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
            for (int r = 0; r < 2; ++r) {  // b0: local dims 16 kb + 2j + part, b1: +8
                const int i0 = 16 * kb + 8 * r + part;
                const uint32_t t01 = prmt(x[i0], x[i0 + 2], 0x5140), t23 = prmt(x[i0 + 4], x[i0 + 6], 0x5140);  // [lo lo hi hi]
                f.b[kb][part][2][r] = prmt(t01, t23, 0x5410);
                f.b[kb][part][1][r] = prmt(t01, t23, 0x7632);
                // third byte: 0x40 + (Qi >> 16), made a signed byte (flip bit 6, copy it to bit 7)
                const uint32_t h01 = prmt(x[i0], x[i0 + 2], 0x0062), h23 = prmt(x[i0 + 4], x[i0 + 6], 0x0062);
                const uint32_t h = prmt(h01, h23, 0x5410) ^ 0x40404040u;
                f.b[kb][part][0][r] = h | ((h & 0x40404040u) << 1);
            }
}

// The V scale rows of a page (a key's row: other_V of four dims | its scales | its zero points), some of them of slice s not finite: such
// keys and dims of the slice leave the page.  A call: what happens never stays out of the loop's instructions and registers.
__device__ __noinline__ void sanitize_slice(uint8_t* rows, int s, int* poison, const int* row_pos, int lane, int first, int key_begin, int key_end) {
    key_end = min(key_end, first + kPage);
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        uint8_t* const row = rows + 16 * (lane + 32 * h);
        uint16_t* const scale = reinterpret_cast<uint16_t*>(row + 8) + s;  // zero point: two further
        const bool key = nonfinite_half2(scale[0]) || nonfinite_half2(scale[2]);
        if (key) scale[0] = scale[2] = 0;
        const uint32_t keys = __ballot_sync(0xffffffffu, key);
        poison_rows(poison, row_pos, lane, static_cast<uint64_t>(keys) << (32 * h), first, key_begin, key_end);
        if (h != s) continue;  // rows 32 s .. : dims of the slice
        uint2* const other = reinterpret_cast<uint2*>(row);
        const bool dims = nonfinite_half2(other->x) || nonfinite_half2(other->y);
        if (dims) *other = make_uint2(0u, 0u);
        if (__any_sync(0xffffffffu, dims)) poison_rows(poison, row_pos, lane, ~0ull, first, key_begin, key_end);
    }
    fence_proxy_async();
    __syncwarp();
}

// Split `split` of KV head `head`, row block `zb` (8 rows); the partial goes to rows pidx .. of the workspace, or (kCluster) stays in
// shared memory for the cluster.  The factors of balanced caches are always applied.
template <bool kCluster>
__device__ __forceinline__ void attn_pair_cta(const AttnParams& P, int split, int head, int zb, int64_t pidx) {
    constexpr int D = 256, kHdrV = Pair::kHdrV, kHdrK = Pair::kHdrK, kChunkBytes = Pair::kChunk, kORow = 128 + 4, kWarpFloats = 16 + 8 * kORow;
    static_assert(kPairWarps * kWarpFloats * 4 <= offsetof(PairSmem, swap), "the merge buffer ends before what else is in use");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    PairSmem& sm = *reinterpret_cast<PairSmem*>(smem_raw);
    const LayerView& L = P.L;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pair = warp >> 1, s = warp & 1;
    const int G = L.q_heads / L.kv_heads;
    PairRing& R = sm.ring[pair];
    uint64_t (&bars)[kSlots] = sm.bars[pair];
    const int pair_barrier = 1 + pair;
    // ---- the few bytes everything waits for go out first: positions, q rows (row w by warp w), page table entries
    uint16_t qraw[8];
    int qpos = INT_MAX;  // no such row: never masked, never stored
#pragma unroll
    for (int j = 0; j < 8; ++j) qraw[j] = 0;
    if (warp < 8) {
        const int Rr = zb * P.block_rows + warp, tq = Rr / G, gq = Rr % G;
        if (tq < P.T) {
            const uint16_t* qrow = P.q + (static_cast<int64_t>(tq) * L.q_heads + head * G + gq) * D;
#pragma unroll
            for (int j = 0; j < 8; ++j) qraw[j] = qrow[lane + 32 * j];
            qpos = P.pos[tq];
        }
    }
    const int pos0 = P.pos[0], kv_total = max(*P.total_pos + 1, 0);  // (a negative position: no key)
    const int key_end = min(P.key_end, kv_total), key_begin = max(P.key_begin, 0);
    const int sealed_pages = 2 * (kv_total / kTile);
    if (threadIdx.x < 2 * kRows) (&sm.poison[0][0])[threadIdx.x] = 0;
    if (threadIdx.x < kPairs) {
#pragma unroll
        for (int i = 0; i < kSlots; ++i) mbar_init(&sm.bars[threadIdx.x][i], 1);
        mbar_fence_init();
    }
    // pages of this CTA, then of this pair
    int w0, w1;
    {
        const int pb = min(key_begin / kPage, sealed_pages), pe = min((key_end + kPage - 1) / kPage, sealed_pages);
        int c0, c1;
        split_pages<kPairs, 2>(max(pe - pb, 0), kv_total % kTile, split, P.nsplit, P.by, c0, c1);
        const bool last_first = c1 - c0 < 3 * kPairs || split == P.nsplit - 1;
        w0 = pb + c0 + warp_pages<kPairs>(c1 - c0, pair, last_first);
        w1 = pb + c0 + warp_pages<kPairs>(c1 - c0, pair + 1, last_first);
        // the stage, and tiles from that of the first appended row on
        if (P.after_append && (split == P.nsplit - 1 || (pb + c1) * kPage > pos0 / kTile * kTile)) grid_dependency_wait();
    }
    const int npages = w1 - w0, nchunks = 2 * npages;
    // ---- the refill side of the ring (see attn_cta): both warps follow it; lane 0 of the first issues K, of the second V
    const int32_t* tbl = L.table();
    auto load_ids = [&](int base) -> int32_t { return base + lane < w1 ? L.page_of(tbl, base + lane) : -1; };
    int ids_base = w0;
    int32_t ids = npages > 0 ? load_ids(ids_base) : -1, ids_next = npages > 0 ? load_ids(ids_base + 32) : -1;
    const uint32_t code_stride = static_cast<uint32_t>(L.kv_heads) * kChunkBytes;
    const uint8_t* const kc = L.k_code + static_cast<size_t>(head) * kChunkBytes;
    const uint8_t* const vc = L.v_code + static_cast<size_t>(head) * kChunkBytes;
    const uint8_t* const ksr = reinterpret_cast<const uint8_t*>(L.k_scale) + static_cast<size_t>(head) * kHdrK;
    const uint8_t* const vsr = reinterpret_cast<const uint8_t*>(L.v_scale) + static_cast<size_t>(head) * kHdrV;
    uint32_t live = 0;
    int32_t issue_pid = -1;
    int n_issued = 0;
    auto issue_next = [&](int slot) {
        const int n = n_issued++;
        if ((n & 1) == 0) {
            const int lp = w0 + (n >> 1);
            if (lp - ids_base == 32) {
                ids = ids_next;
                ids_base += 32;
                ids_next = load_ids(ids_base + 32);
            }
            issue_pid = __shfl_sync(0xffffffffu, ids, lp - ids_base);
        }
        const int32_t pid = issue_pid;
        if (pid < 0) { live &= ~(1u << slot); return; }
        live |= 1u << slot;
        if (s == (n & 1) && lane == 0) {
            uint8_t* dst = R.slots[slot];
            if (n & 1) {
                const uint8_t* src = vc + static_cast<size_t>(pid) * code_stride;
                mbar_expect_tx(&bars[slot], kChunkBytes);
#pragma unroll
                for (int a = 0; a < Pair::kSubs; ++a) bulk_g2s(dst + a * (Pair::kSubBytes + Pair::kShift), src + a * Pair::kSubBytes, Pair::kSubBytes, &bars[slot]);
            } else {
                uint8_t* hdr = R.hdr[(n >> 1) % kHdrs];
                mbar_expect_tx(&bars[slot], kChunkBytes + kHdrV + kHdrK);
                bulk_g2s(dst, kc + static_cast<size_t>(pid) * code_stride, kChunkBytes, &bars[slot]);
                bulk_g2s(hdr, vsr + static_cast<size_t>(pid) * (static_cast<uint32_t>(L.kv_heads) * kHdrV), kHdrV, &bars[slot]);
                bulk_g2s(hdr + kHdrV, ksr + static_cast<size_t>(pid) * (static_cast<uint32_t>(L.kv_heads) * kHdrK), kHdrK, &bars[slot]);
            }
        }
    };
    __syncthreads();  // the barriers are ready
    while (n_issued < kSlots && n_issued < nchunks) issue_next(n_issued);

    // ---- q' = H q * scale * log2(e) for the rows of this block, stored in fragment order
    if (warp < 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = L.dtype == KVB_DTYPE_BF16 ? in_to_f32<true>(qraw[j]) : in_to_f32<false>(qraw[j]);
        hadamard_warp<D>(v, lane);  // rows beyond T are zeros and stay zeros
        if (lane == 0) sm.row_pos[warp] = qpos;
        float* dst = reinterpret_cast<float*>(sm.qfrag);
#pragma unroll
        for (int j = 0; j < 8; ++j)  // dim lane + 32 j -> lane' = row * 4 + (d%128)/32, slot j' = 8 slice + (d%32)/4, component d%4
            dst[((8 * (j >> 2) + (lane >> 2)) * 32 + warp * 4 + (j & 3)) * 4 + (lane & 3)] = v[j] * P.scale_log2;
    }
    if (warp == kPairWarps - 1) launch_dependents();  // the merge kernel may take its place on the SMs; it waits for this grid's completion
    __syncthreads();

    const int g = lane >> 2, t = lane & 3;
    const int row_lim[2] = {sm.row_pos[2 * t], sm.row_pos[2 * t + 1]};
    const int min_lim = __reduce_min_sync(0xffffffffu, sm.row_pos[lane & 7]);  // (a negative position: a row that sees no key)
    F2 o[4][2][2];  // [32-dim block of the slice][even, odd dims][c >> 1], see Acc
#pragma unroll
    for (int db = 0; db < 4; ++db)
#pragma unroll
        for (int xy = 0; xy < 2; ++xy) o[db][xy][0] = o[db][xy][1] = F2(0.0f, 0.0f);
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
    float4 (&swap)[2][4][32] = sm.swap[pair];
    auto rescale = [&](const float (&alpha)[2]) {
        const F2 a(alpha[0], alpha[1]);
#pragma unroll
        for (int db = 0; db < 4; ++db)
#pragma unroll
            for (int xy = 0; xy < 2; ++xy)
#pragma unroll
                for (int h = 0; h < 2; ++h) o[db][xy][h] = mul2(o[db][xy][h], a);
        l_run[0] *= alpha[0];
        l_run[1] *= alpha[1];
    };

    // ---- open tile (last split of the head): a 16-key group a pair, un-quantised, from the stage; the loads are in flight together with
    //      the first chunks of the ring
    if (split == P.nsplit - 1) {
        const int tile = kv_total / kTile, first = tile * kTile + 16 * pair;
        if (first < key_end && first + 16 > key_begin && first < kv_total) {
            const __half* const krow = L.stage_row(0, tile & 1, head, 16 * pair) + 128 * s;
            const __half* const vrow = L.stage_row(1, tile & 1, head, 16 * pair);
            float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // q' in fp16 high and low parts: the product keeps fp32 accuracy
                const uint4 a = *reinterpret_cast<const uint4*>(krow + g * D + 32 * t + 8 * i), b = *reinterpret_cast<const uint4*>(krow + (8 + g) * D + 32 * t + 8 * i);
                uint32_t hi[2][2], lo[2][2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float4 qv = sm.qfrag[8 * s + 2 * i + j][lane];
                    const float y[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        hi[j][h] = pack_half2(y[2 * h], y[2 * h + 1]);
                        const float2 hf = unpack_half2(hi[j][h]);
                        lo[j][h] = pack_half2(y[2 * h] - hf.x, y[2 * h + 1] - hf.y);
                    }
                }
                mma16816(x, a.x, b.x, a.y, b.y, hi[0][0], hi[0][1]);
                mma16816(x, a.z, b.z, a.w, b.w, hi[1][0], hi[1][1]);
                mma16816(x, a.x, b.x, a.y, b.y, lo[0][0], lo[0][1]);
                mma16816(x, a.z, b.z, a.w, b.w, lo[1][0], lo[1][1]);
            }
            swap[s][0][lane] = make_float4(x[0], x[1], x[2], x[3]);
            named_barrier_sync(pair_barrier, 64);
            const float4 other = swap[s ^ 1][0][lane];
            x[0] += other.x; x[1] += other.y; x[2] += other.z; x[3] += other.w;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int p = first + g + (e >> 1) * 8;
                if (p >= kv_total || p < key_begin || p >= key_end || p > row_lim[e & 1]) x[e] = -INFINITY;
            }
            float alpha[2], muse[2];
            bool moved = false;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float mx = fmaxf(x[j], x[2 + j]);
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float mnew = fmaxf(m_run[j], mx);
                moved |= mnew > m_run[j];
                muse[j] = mnew == -INFINITY ? 0.0f : mnew;
                alpha[j] = fast_exp2(m_run[j] - muse[j]);
                m_run[j] = mnew;
            }
            if (__any_sync(0xffffffffu, moved)) rescale(alpha);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] = fast_exp2(x[e] - muse[e & 1]);
                l_run[e & 1] += x[e];
            }
            const float2 h0 = unpack_half2(pack_half2(x[0], x[1])), h1 = unpack_half2(pack_half2(x[2], x[3]));
            const uint32_t b0 = movmatrix_trans(pack_half2(x[0], x[1])), b1 = movmatrix_trans(pack_half2(x[2], x[3]));  // -> (row g; keys 2t, 2t+1 | + 8)
            const uint32_t c0 = movmatrix_trans(pack_half2(x[0] - h0.x, x[1] - h0.y)), c1 = movmatrix_trans(pack_half2(x[2] - h1.x, x[3] - h1.y));
            // A = V^T, clamped to finite values (see finite_half2); keys at or beyond kv_total hold stale rows: zero
            uint32_t odd = 0;
#pragma unroll
            for (int db = 0; db < 4; ++db) {
                uint2 v[4];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const int key = 2 * t + (kk & 1) + (kk >> 1) * 8;
                    v[kk] = first + key < kv_total ? *reinterpret_cast<const uint2*>(vrow + key * D + 128 * s + 32 * db + 4 * g) : make_uint2(0u, 0u);
                    const uint2 f = make_uint2(finite_half2(v[kk].x), finite_half2(v[kk].y));
                    odd |= (f.x ^ v[kk].x) | (f.y ^ v[kk].y);
                    v[kk] = f;
                }
#pragma unroll
                for (int xy = 0; xy < 2; ++xy) {  // dims 4g, 4g+2 | 4g+1, 4g+3 of keys 2t, 2t+1 and 2t+8, 2t+9
                    const uint32_t sel = xy ? 0x7632 : 0x5410;
                    const float2 lo = o[db][xy][0].get(), hi = o[db][xy][1].get();
                    float d[4] = {lo.x, lo.y, hi.x, hi.y};
                    const uint32_t a0 = prmt(v[0].x, v[1].x, sel), a1 = prmt(v[0].y, v[1].y, sel), a2 = prmt(v[2].x, v[3].x, sel), a3 = prmt(v[2].y, v[3].y, sel);
                    mma16816(d, a0, a1, a2, a3, b0, b1);
                    mma16816(d, a0, a1, a2, a3, c0, c1);
                    o[db][xy][0] = F2(d[0], d[1]);
                    o[db][xy][1] = F2(d[2], d[3]);
                }
            }
            if (__any_sync(0xffffffffu, odd != 0u)) poison_stage_group(vrow, sm.poison, sm.row_pos, lane, first, kv_total, key_begin, key_end);
            named_barrier_sync(pair_barrier, 64);  // the logits of the first page go where these were
        }
    }

    // ---- sealed pages
    bool timed_out = false;
    int slot = 0;          // slot of the oldest chunk not yet released
    uint32_t phases = 0;   // bit i: parity the next wait on slot i expects
    auto wait_chunk = [&](int i, bool waits) {  // bounded; behind it the warp is together again (see attn_cta)
        if (!waits || (!__all_sync(0xffffffffu, mbar_try_wait(&bars[i], (phases >> i) & 1u)) && !mbar_wait_bounded(&bars[i], (phases >> i) & 1u))) timed_out = true;
    };
    auto release_chunk = [&](bool was_live) {  // the chunk in `slot` has been read by both warps: refill the slot, advance
        if (was_live) phases ^= 1u << slot;
        live &= ~(1u << slot);
        if (n_issued < nchunks) {
            if (lane == 0) fence_proxy_async();  // generic-proxy reads of the slot are ordered before the refill
            issue_next(slot);
        }
        slot ^= 1;
    };
    const int key_lo = 8 * g;
    constexpr int kKeyH = Pair::kKeyH;
    PairQInt qi;
    int cur_tile = -1;
    for (int pi = 0; pi < npages; ++pi) {
        const int lp = w0 + pi;
        if (!((live >> slot) & 1u)) {  // a page that could not be addressed: nothing was copied, nothing is read
            release_chunk(false);
            release_chunk(false);
            continue;
        }
        // ---- K chunk + header
        wait_chunk(slot, kStepWaitsK);
        uint8_t* const hdr = R.hdr[pi % kHdrs];
        uint32_t sc;  // the lane's largest scale of V
        {
            constexpr uint32_t kAbs = 0x7FFF7FFFu;
            const uint4* const rows = reinterpret_cast<const uint4*>(hdr);
            const uint2 a = *reinterpret_cast<const uint2*>(&rows[lane].z), b = *reinterpret_cast<const uint2*>(&rows[lane + 32].z), dims = *reinterpret_cast<const uint2*>(&rows[lane + 32 * s]);
            const uint32_t pick = s ? 0x7632 : 0x5410, sz0 = prmt(a.x, a.y, pick), sz1 = prmt(b.x, b.y, pick);  // scale, zero point
            const uint32_t both = __vmaxu2(sz0 & kAbs, sz1 & kAbs);
            sc = both & 0xFFFFu;
            if (__any_sync(0xffffffffu, nonfinite_half2(__vmaxu2(__vmaxu2(dims.x & kAbs, dims.y & kAbs), both)))) {
                sanitize_slice(hdr, s, sm.poison[s], sm.row_pos, lane, lp * kPage, key_begin, key_end);
                sc = max(*reinterpret_cast<const uint16_t*>(hdr + 16 * lane + 8 + 2 * s) & 0x7FFF, *reinterpret_cast<const uint16_t*>(hdr + 16 * (lane + 32) + 8 + 2 * s) & 0x7FFF);
            }
        }
        if ((lp >> 1) != cur_tile) {  // per-dim scale / zero point of K belong to the tile
            cur_tile = lp >> 1;
            __syncwarp();
            {  // scale row 32 s + lane: dims 4 lane .. of the slice
                const uint32_t* w = reinterpret_cast<const uint32_t*>(hdr + kHdrV + 20 * (32 * s + lane));
                const float2 s01 = unpack_half2(w[0]), s23 = unpack_half2(w[1]), z01 = unpack_half2(w[2]), z23 = unpack_half2(w[3]);
                const int at = 128 * s + 4 * lane + kTabPad * (4 * s + (lane >> 3));
                *reinterpret_cast<float4*>(&R.scale_k[at]) = make_float4(s01.x, s01.y, s23.x, s23.y);
                *reinterpret_cast<float4*>(&R.zp_k[at]) = make_float4(z01.x, z01.y, z23.x, z23.y);
            }
            __syncwarp();
            build_pair_qint(sm, R, s, lane, qi);
        }
        const int first = lp * kPage;
        const bool need_mask = first + kPage - 1 > min_lim || first < key_begin || first + kPage > key_end;
        // ---- QK over the slice: integer sums, then fp32 logits times the key's factor
        float sl[4][4];
        {
            const uint8_t* ch = R.slots[slot] + key_lo * 128 + 16 * t + 64 * s;
#pragma unroll
            for (int grp = 0; grp < 4; ++grp) {
                const int koff = Pair::key_grp(grp) * 128;
                const uint4 ka = *reinterpret_cast<const uint4*>(ch + koff), kb8 = *reinterpret_cast<const uint4*>(ch + koff + kKeyH * 128);
                const uint32_t wa[4] = {ka.x, ka.y, ka.z, ka.w}, wb[4] = {kb8.x, kb8.y, kb8.z, kb8.w};
                int ce[3][4], co[3][4];  // even dims, odd dims (x 16)
#pragma unroll
                for (int kb = 0; kb < 2; ++kb) {
                    const uint32_t l0 = wa[2 * kb] & 0x0F0F0F0Fu, l1 = wb[2 * kb] & 0x0F0F0F0Fu, l2 = wa[2 * kb + 1] & 0x0F0F0F0Fu, l3 = wb[2 * kb + 1] & 0x0F0F0F0Fu;
                    const uint32_t h0 = wa[2 * kb] & 0xF0F0F0F0u, h1 = wb[2 * kb] & 0xF0F0F0F0u, h2 = wa[2 * kb + 1] & 0xF0F0F0F0u, h3 = wb[2 * kb + 1] & 0xF0F0F0F0u;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const uint32_t(&be)[2] = qi.b[kb][0][d], (&bo)[2] = qi.b[kb][1][d];
                        if (d == 0) {
                            if (kb == 0) { imma_us0(ce[d], l0, l1, l2, l3, be[0], be[1]); imma_us0(co[d], h0, h1, h2, h3, bo[0], bo[1]); }
                            else { imma_us(ce[d], l0, l1, l2, l3, be[0], be[1]); imma_us(co[d], h0, h1, h2, h3, bo[0], bo[1]); }
                        } else {
                            if (kb == 0) { imma_uu0(ce[d], l0, l1, l2, l3, be[0], be[1]); imma_uu0(co[d], h0, h1, h2, h3, bo[0], bo[1]); }
                            else { imma_uu(ce[d], l0, l1, l2, l3, be[0], be[1]); imma_uu(co[d], h0, h1, h2, h3, bo[0], bo[1]); }
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {  // a key, rows 2t and 2t + 1
                    const float ok = __half2float(*reinterpret_cast<const __half*>(hdr + kHdrV + (key_lo + Pair::key_grp(grp) + kKeyH * h) * 20 + 16 + 2 * s));
                    float hi[2], lo[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int e = 2 * h + j;
                        hi[j] = static_cast<float>(ce[0][e] * 16 + co[0][e]);
                        // the two low bytes' sums stay below 2^31 together; the high byte's joins in fp32
                        lo[j] = static_cast<float>(((ce[1][e] * 16 + co[1][e]) << 8) + (ce[2][e] * 16 + co[2][e]));
                    }
                    const F2 sum = fma2(F2(hi[0], hi[1]), F2(65536.0f, 65536.0f), F2(lo[0], lo[1]));
                    const float2 y = mul2(fma2(sum, F2(qi.f[0], qi.f[1]), F2(qi.qz[0], qi.qz[1])), F2(ok, ok)).get();
                    sl[grp][2 * h] = y.x;
                    sl[grp][2 * h + 1] = y.y;
                }
                swap[s][grp][lane] = make_float4(sl[grp][0], sl[grp][1], sl[grp][2], sl[grp][3]);
            }
        }
        if (named_barrier_or(pair_barrier, 64, timed_out)) { timed_out = true; break; }  // the logits meet; K has been read by both
        release_chunk(true);
#pragma unroll
        for (int grp = 0; grp < 4; ++grp) {
            const float4 y = swap[s ^ 1][grp][lane];
            sl[grp][0] += y.x; sl[grp][1] += y.y; sl[grp][2] += y.z; sl[grp][3] += y.w;
        }
        if (need_mask) {  // keys a row may not see (causal limit, key range)
#pragma unroll
            for (int grp = 0; grp < 4; ++grp)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int p = first + key_lo + Pair::key_grp(grp) + kKeyH * (e >> 1);
                    if (p < key_begin || p >= key_end || p > row_lim[e & 1]) sl[grp][e] = -INFINITY;
                }
        }
        // ---- softmax of the page relative to its own row maxima; weights of the page against the running state
        uint32_t bw[3][4];  // weights as B fragments, one byte each: highest digit first
        F2 wq, zfull;       // per row: weight of the integer sums of this page; sum of p * zp_V, weighted like them
        {
            const float svmax = __half2float(__ushort_as_half(static_cast<uint16_t>(__reduce_max_sync(0xffffffffu, sc))));
            const float F = svmax > 0.0f ? Pair::kPMax / svmax : 0.0f, invF = svmax * (1.0f / Pair::kPMax);
            float alpha[2], wpass[2], cst[2];
            bool moved = false;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float mp = -INFINITY;
#pragma unroll
                for (int grp = 0; grp < 4; ++grp) mp = fmaxf(mp, fmaxf(sl[grp][j], sl[grp][2 + j]));
                mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, 4));
                mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, 8));
                mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, 16));
                const float mnew = fmaxf(m_run[j], mp);
                moved |= mnew > m_run[j];
                const float muse = mnew == -INFINITY ? 0.0f : mnew;
                alpha[j] = fast_exp2(m_run[j] - muse);
                wpass[j] = fast_exp2(mp - muse);
                m_run[j] = mnew;
                cst[j] = mp == -INFINITY ? 0.0f : -mp;
            }
            if (__any_sync(0xffffffffu, moved)) rescale(alpha);
            F2 lp_[2] = {F2(0.0f, 0.0f), F2(0.0f, 0.0f)}, zp_[2] = {F2(0.0f, 0.0f), F2(0.0f, 0.0f)};  // per row, the keys of m-rows g and g + 8
            const uint8_t* vs = hdr + key_lo * 16 + 8;  // V scale rows per key: 4 other_V, 2 scales, 2 zero points
            const uint32_t pick = s ? 0x7632 : 0x5410;
#pragma unroll
            for (int grp = 0; grp < 4; ++grp) {
                const int koff = Pair::key_grp(grp) * 16;
                const uint2 a = *reinterpret_cast<const uint2*>(vs + koff), b = *reinterpret_cast<const uint2*>(vs + koff + kKeyH * 16);
                const float2 sz0 = unpack_half2(prmt(a.x, a.y, pick)), sz1 = unpack_half2(prmt(b.x, b.y, pick));  // scale, zero point of m-rows g, g + 8
                const F2 sf = mul2(F2(sz0.x, sz1.x), F2(F, F)), zz(sz0.y, sz1.y);
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 d = add2(F2(sl[grp][j], sl[grp][2 + j]), F2(cst[j], cst[j])).get();  // masked keys stay at -inf
                    const F2 p(fast_exp2(d.x), fast_exp2(d.y));
                    lp_[j] = add2(lp_[j], p);
                    zp_[j] = fma2(p, zz, zp_[j]);
                    const float2 y = fma2(p, sf, F2(Pair::kPMagic, Pair::kPMagic)).get();
                    w[j] = __float_as_uint(y.x);
                    w[2 + j] = __float_as_uint(y.y);
                }
                // accumulator layout (m-row g; rows 2t, 2t+1) -> operand layout (row g; m-rows 2t, 2t+1 | 2t+8, 2t+9)
                const uint32_t y0 = movmatrix_trans(prmt(w[0], w[1], 0x5410)), y1 = movmatrix_trans(prmt(w[2], w[3], 0x5410));
                bw[2][grp] = prmt(y0, y1, 0x6420);
                bw[1][grp] = prmt(y0, y1, 0x7531);
                const uint32_t y2 = movmatrix_trans(prmt(prmt(w[0], w[2], 0x0062), prmt(w[1], w[3], 0x0062), 0x5410));  // the third bytes of both m-rows
                bw[0][grp] = prmt(y2, y2, 0x3120);
            }
            float zf[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float2 lp2 = lp_[j].get(), zp2 = zp_[j].get();
                l_run[j] = fmaf(lp2.x + lp2.y, wpass[j], l_run[j]);
                float zs = zp2.x + zp2.y;
                zs += __shfl_xor_sync(0xffffffffu, zs, 4);
                zs += __shfl_xor_sync(0xffffffffu, zs, 8);
                zs += __shfl_xor_sync(0xffffffffu, zs, 16);
                zf[j] = zs * wpass[j];
            }
            zfull = F2(zf[0], zf[1]);
            wq = F2(wpass[0] * invF, wpass[1] * invF);
        }
        // ---- PV on the int8 path, see attn_cta: key i' + 4c of each of the eight shifted sub-blocks
        wait_chunk(slot, kStepWaitsV);
        {
            const int vrow = lane & 7, vmat = lane >> 3;
            const uint8_t* ch = R.slots[slot] + (8 * vrow + vmat) * 128 + Pair::kShift * vrow + 64 * s;
            const F2 wn[2] = {wq, mul2(wq, F2(0.0625f, 0.0625f))};
#pragma unroll
            for (int db = 0; db < 4; ++db) {
                int ix[2][3][4];  // [xy][digit][c]
#pragma unroll
                for (int c = 0; c < 2; ++c) {  // 32-key halves of the page
                    uint32_t r[4];
                    ldsm_x4_trans(r, ch + c * 512 + 16 * db);
                    const uint32_t u0 = prmt(r[0], r[1], 0x6420), v0 = prmt(r[0], r[1], 0x7531), u1 = prmt(r[2], r[3], 0x6420), v1 = prmt(r[2], r[3], 0x7531);
                    const uint32_t ax0 = u0 & 0x0F0F0F0Fu, ax1 = v0 & 0x0F0F0F0Fu, ax2 = u1 & 0x0F0F0F0Fu, ax3 = v1 & 0x0F0F0F0Fu;
                    const uint32_t ay0 = u0 & 0xF0F0F0F0u, ay1 = v0 & 0xF0F0F0F0u, ay2 = u1 & 0xF0F0F0F0u, ay3 = v1 & 0xF0F0F0F0u;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        if (c == 0) {
                            imma_uu0(ix[0][d], ax0, ax1, ax2, ax3, bw[d][0], bw[d][1]);
                            imma_uu0(ix[1][d], ay0, ay1, ay2, ay3, bw[d][0], bw[d][1]);
                        } else {
                            imma_uu(ix[0][d], ax0, ax1, ax2, ax3, bw[d][2], bw[d][3]);
                            imma_uu(ix[1][d], ay0, ay1, ay2, ay3, bw[d][2], bw[d][3]);
                        }
                    }
                }
                // V scale row d / 4 starts with the other_V of its four dims
                const uint2 o4 = *reinterpret_cast<const uint2*>(hdr + (8 * (4 * s + db) + g) * 16);
                const float2 o01 = unpack_half2(o4.x), o23 = unpack_half2(o4.y);
                const float ov[2][2] = {{o01.x, o23.x}, {o01.y, o23.y}};  // [xy][h]
                // ---- integer sums of the page -> running fp32 accumulators: (sum p code scale_V + sum p zp_V) * other_V(dim)
#pragma unroll
                for (int xy = 0; xy < 2; ++xy)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float v[2], u[2];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const int c = 2 * h + j;
                            u[j] = static_cast<float>(ix[xy][0][c]);
                            v[j] = static_cast<float>((ix[xy][1][c] << 8) + ix[xy][2][c]);
                        }
                        const F2 vv = fma2(F2(u[0], u[1]), F2(65536.0f, 65536.0f), F2(v[0], v[1]));
                        o[db][xy][h] = fma2(fma2(vv, wn[xy], zfull), F2(ov[xy][h], ov[xy][h]), o[db][xy][h]);
                    }
            }
        }
        // V and the header have been read by both, or one has given it up: it is still on its way, and its slot stays as it is
        if (named_barrier_or(pair_barrier, 64, timed_out)) { timed_out = true; break; }
        release_chunk(true);
    }
    if (timed_out) {
        if (lane == 0) L.flag(KVB_ERR_WAIT_TIMEOUT);
        // copies already issued must land before the CTA's shared memory is released: one more bounded wait each
        for (int i = 0; i < kSlots; ++i)
            if ((live >> i) & 1u) mbar_wait_lane_bounded(&bars[i], (phases >> i) & 1u);
    }

    // ---- merge the pairs of the CTA (log-sum-exp), one partial per row; every slot has been consumed: the ring memory becomes the merge
    //      buffer
    __syncthreads();
    float* const mbuf = reinterpret_cast<float*>(sm.ring) + warp * kWarpFloats;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int k = 4; k <= 16; k <<= 1) l_run[j] += __shfl_xor_sync(0xffffffffu, l_run[j], k);
        if (g == 0) {
            mbuf[2 * t + j] = m_run[j];
            mbuf[8 + 2 * t + j] = l_run[j];
        }
    }
#pragma unroll
    for (int db = 0; db < 4; ++db) {
        const float2 a = o[db][0][0].get(), b = o[db][1][0].get(), c = o[db][0][1].get(), d = o[db][1][1].get();
        float* dst = mbuf + 16 + 2 * t * kORow + 32 * db + 4 * g;  // rows 2t, 2t + 1, dims 32 db + 4g .. +3
        *reinterpret_cast<float4*>(dst) = make_float4(a.x, b.x, c.x, d.x);
        *reinterpret_cast<float4*>(dst + kORow) = make_float4(a.y, b.y, c.y, d.y);
    }
    __syncthreads();
    {  // a thread: four dims of one row
        const float* const all = reinterpret_cast<const float*>(sm.ring);
        const int row = threadIdx.x >> 6, d = 4 * (threadIdx.x & 63), half = d >> 7;
        float m = -INFINITY, l = 0.0f;
#pragma unroll
        for (int p = 0; p < kPairs; ++p) m = fmaxf(m, all[2 * p * kWarpFloats + row]);
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (m != -INFINITY) {
#pragma unroll
            for (int p = 0; p < kPairs; ++p) {
                const float* const wb = all + (2 * p + half) * kWarpFloats;
                const float w = fast_exp2(wb[row] - m);  // exp2(-inf) = 0 for a pair that saw no key
                const float4 v = *reinterpret_cast<const float4*>(wb + 16 + row * kORow + (d & 127));
                l += w * wb[8 + row];
                x.x += w * v.x; x.y += w * v.y; x.z += w * v.z; x.w += w * v.w;
            }
        }
        if (sm.poison[half][row] != 0) x.x = x.y = x.z = x.w = __uint_as_float(0x7FC00000u);
        if constexpr (kCluster) {
            PairPart& part = *reinterpret_cast<PairPart*>(sm.swap);
            *reinterpret_cast<float4*>(&part.o[row][d]) = x;
            if (d == 0) { part.m[row] = m; part.l[row] = l; }
        } else {
            *reinterpret_cast<float4*>(P.ws_o + (pidx + row) * D + d) = x;
            if (d == 0) { P.ws_m[pidx + row] = m; P.ws_l[pidx + row] = l; }
        }
    }
}

__global__ void __launch_bounds__(kPairWarps * 32, 1) attn_pair_kernel(const AttnParams P) {
    if (!P.after_append) grid_dependency_wait();
    const int head = blockIdx.y, zb = blockIdx.z, split = blockIdx.x;
    attn_pair_cta<false>(P, split, head, zb, ((static_cast<int64_t>(head) * gridDim.z + zb) * P.nsplit + split) * kRows);
    if (P.after_append) grid_dependency_wait();  // nobody leaves before the append is over: what waits for this grid finds both done
}

}  // namespace
}  // namespace kvb
