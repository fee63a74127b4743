// Single-query (decode) attention with grouped queries, split over the KV length.
//
// Work item = (batch row, kv head, KV split); one CTA of four warps each (rows of
// different lengths: a share of all rows' tiles, see AttnSchedule).  The
// CTA streams its keys and values once, 64 keys per tile, through a 3-deep ring
// of shared-memory stages filled with 16-byte cp.async copies (zero-filled past
// the row's valid length, XOR-swizzled so that ldmatrix is conflict free).  The
// G query heads that share the kv head form the rows of a 16-row mma tile
// (rows >= G are zero), so every K/V byte is used by all G heads while it is on
// chip: S = Q K^T and O += P V both run on mma.sync m16n8k16 with fp32
// accumulation, soft-max statistics in fp32 in the exp2 domain.  Each warp owns
// 16 of the tile's 64 keys with its own running (max, sum, O); the four are
// merged in shared memory at the end, the split's (max, sum, O) goes to the
// workspace, and the CTA that finishes last for a (row, kv head) -- found with
// one atomic counter, no waiting -- folds the splits together in index order
// and writes the bf16 output.  No spin waits anywhere.
//
// Decode-layer mode (fuse_new_token): q, k, v of the token being decoded come
// straight from the fused QKV projection output; q and k get their RMSNorm over
// the head here (optionally with a weight and the rotary embedding, fp32 with one
// rounding), and the CTA whose split holds the token's cache slot (S-1, or the
// row's own length - 1 when per-row lengths are given) writes the new k and v
// into the cache and patches them into its shared-memory tile.
// The caches are contiguous [B, NKV, S, D] or page pools addressed through a page
// table (pages of a power-of-two number of keys >= 64, so a tile never straddles
// pages).
#include <atomic>

#include "launchers.h"

namespace ezb {

static constexpr int kAttnThreads = 128;
static constexpr int kTileKeys = 64;
static constexpr int kAttnStages = 3;
static constexpr int kSchedRows = 128;  // batch rows that the balanced schedule covers
// CTAs of the kernel that share an SM: bounded by registers at head_dim 64 (160 a thread), by shared memory at 128.
__host__ __device__ constexpr int attn_ctas_per_sm(int D) { return D <= 64 ? 3 : 2; }

struct AttnParams {
    const bf16* Q;
    long long q_bstride;
    const bf16* K;
    const bf16* V;
    bf16* Out;
    long long o_bstride;
    const int* seq_lens;
    int B, H, NKV, S, G;
    int chunk, nchunks, nqt;
    int min_tiles;  // balanced schedule: smallest split, in tiles
    int first;      // see pdl_open
    int early;      // the caches and lengths may be read before the dependency wait (see launch_attn_decode)
    float scale_log2e;
    float* part_o;   // [items][16][D]
    float* part_ml;  // [items][16][2]
    unsigned int* counters;
    int fuse_new_token;
    const bf16* qkv;
    long long qkv_bstride;
    int q_rows, kv_rows;
    bf16* K_cache_w;
    bf16* V_cache_w;
    float eps;
    const bf16* q_norm_w;
    const bf16* k_norm_w;
    const bf16* rope_cos;
    const bf16* rope_sin;
    int rope_by_len;  // 1: rope_cos / rope_sin are table bases, the row used is the token's slot (len-1)
    const int* page_table;  // null: contiguous caches [B, NKV, S, D]; else [B, max_pages] page ids into pools [pages, NKV, P, D]
    int page_shift;         // log2 of the page size P (a power of two >= 64, so a 64-key tile never straddles pages)
    int max_pages;
    int num_pages;          // pages in the pools: a table entry outside [0, num_pages) is reported, never dereferenced
    unsigned int* status;
    PrefetchList next;
    Trace trace;
};

// Head RMSNorm (+ optional weight, + optional rotate-half RoPE) of one head held by a warp:
// lane owns elements lane + 32*j, so the rotation partner (i +- D/2) is in the same lane.
// x: in/out fp32 values; returns them ready for the single bf16 rounding.
template <int D>
__device__ __forceinline__ void head_norm_rope(float (&x)[D / 32], float eps, const bf16* w, const bf16* cosr, const bf16* sinr,
                                               int lane) {
    constexpr int NJ = D / 32, HJ = NJ / 2;
    float ssq = 0.f;
#pragma unroll
    for (int j = 0; j < NJ; ++j) ssq += x[j] * x[j];
    ssq = warp_sum(ssq);
    const float r = 1.0f / sqrtf(ssq / (float)D + eps);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        x[j] = __fmul_rn(x[j], r);
        if (w) x[j] = __fmul_rn(x[j], __bfloat162float(w[lane + j * 32]));
    }
    if (cosr) {
#pragma unroll
        for (int j = 0; j < HJ; ++j) {
            const int i = lane + j * 32, i2 = i + D / 2;
            const float n1 = x[j], n2 = x[j + HJ];
            x[j] = __fadd_rn(__fmul_rn(n1, __bfloat162float(cosr[i])), __fmul_rn(-n2, __bfloat162float(sinr[i])));
            x[j + HJ] = __fadd_rn(__fmul_rn(n2, __bfloat162float(cosr[i2])), __fmul_rn(n1, __bfloat162float(sinr[i2])));
        }
    }
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ int warp_sum_int(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One CTA's share of one (batch row, kv head, query tile): tiles [t0, t1) of the row's keys.
struct AttnSegment {
    int b, kvh, qt;
    int t0, t1;
    int len;               // valid keys of the row
    int part, nparts;      // which of the group's parts this is
    long long rec0, rec1;  // records of part 0 and part 1; later parts follow `rec_step` behind one another
    int rec_step;
};

// Rows of different lengths (SCHED): the tiles of all groups - (row, kv head, query tile) - are dealt to the CTAs of one
// resident wave by their real lengths, which only the device knows.  Cutting every row on the grid of the longest one
// left most of 832 CTAs with nothing or one tile and ran them in three waves of pure latency (2B, 13 rows of 128..1024
// keys: 22 us for 5 us worth of bytes), or ended in a half-empty last wave (8B, 32 rows of 1024..8192 keys: 113 us for 92).
// Three ways, tried in this order:
//   chunks  all groups cut into pieces of at most `chunk` tiles, one piece per CTA, if some chunk within two tiles of the
//           even share fits the wave;
//   whole   groups short (four tiles or less on average): every CTA takes whole groups, cuts moved to group boundaries;
//   ranges  the tiles of all groups in one line, cut evenly: a CTA may finish one group and begin the next.  Coming to a
//           new group costs about as much as three tiles (merge, queries: 3.5 us of 1.3 us a tile), so each group has that
//           many units without a tile in front.
static constexpr int kGroupUnits = 3;
struct AttnSchedule {
    int end[kSchedRows];    // units (pieces or tiles) up to and including row b, over all its groups
    int tiles[kSchedRows];  // tiles of row b
    int len[kSchedRows];    // valid keys of row b
    int lead;               // units without a tile in front of each group
    int chunk;              // > 0: chunks
    int whole;
    int total;  // units of all rows
};

template <int D, bool SCHED>
__global__ void __launch_bounds__(kAttnThreads, attn_ctas_per_sm(D)) attn_decode_kernel(const AttnParams p) {
    constexpr int CPR = D / 8;                       // 16-byte chunks per key row
    constexpr int ROW_BYTES = D * 2;
    constexpr int TILE_BYTES = kTileKeys * ROW_BYTES;  // one K or V tile
    constexpr int STAGE_BYTES = 2 * TILE_BYTES;
    constexpr int QS = D + 8;                        // padded query row, elements
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* stages = smem;
    bf16* q_s = reinterpret_cast<bf16*>(smem + kAttnStages * STAGE_BYTES);
    bf16* kv_new_s = q_s + 16 * QS;  // [2][D]: the new token's k (normalised) and v, decode-layer mode
    bf16* rope_s = kv_new_s + 2 * D;  // [4][D]: q / k norm weights, cos and sin row of the token's slot
    AttnSchedule* sched = reinterpret_cast<AttnSchedule*>(rope_s + 4 * D);
    __shared__ int s_is_last;
    __shared__ float mrg_ml[128];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g4 = lane >> 2, t4 = lane & 3;
    const int G = p.G;
    const int cta = SCHED ? (int)blockIdx.x : (int)((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
    // Lengths and the first page ids may be read before the dependency wait (`early`): through L2, since a line that an
    // earlier kernel left in this SM's L1 is only known to be dropped behind that wait.
    auto row_len = [&](int b) { return p.seq_lens ? max(p.fuse_new_token ? 1 : 0, min(p.S, __ldcg(p.seq_lens + b))) : p.S; };

    unsigned long long* trec = (tid == 0) ? trace_open(p.trace, 9u, cta) : nullptr;
    pdl_open(p.first);
    // This kernel is latency-bound at small batch; meanwhile HBM can already pull
    // the next kernel's weights (immutable, so safe before the dependency wait).
    if (warp == 3) prefetch_next_operands(p.next, lane, cta, gridDim.x * gridDim.y * gridDim.z);
    // The KV cache is mutable state.  Inside a chain, however, nothing between the chain's first kernel - which began
    // after everything in front of it - and this one writes the keys read here: the new token's slot is patched from
    // shared memory.  Then (`early`) the schedule and the first tiles do not wait for the projection in front.
    if (!p.early) pdl_wait();

    // ---- this CTA's share ----
    int u0 = 0, u1 = 1;
    const int heads = p.NKV * p.nqt;
    if (SCHED) {
        if (warp == 0) {
            int t[kSchedRows / 32], sum = 0;
#pragma unroll
            for (int i = 0; i < kSchedRows / 32; ++i) {
                const int b = lane + 32 * i;
                t[i] = 0;
                if (32 * i >= p.B) continue;
                const int len = b < p.B ? row_len(b) : 0;
                t[i] = b < p.B ? max(1, (len + kTileKeys - 1) / kTileKeys) : 0;  // an empty row writes zeros
                sum += t[i];
                if (b < p.B) sched->tiles[b] = t[i], sched->len[b] = len;
            }
            const int total = warp_sum_int(sum) * heads;
            const int even = max(p.min_tiles, (int)((total + gridDim.x - 1) / gridDim.x));
            int chunk = 0;
            for (int c = even; c <= even + 2 && !chunk; ++c) {
                int n = 0;
#pragma unroll
                for (int i = 0; i < kSchedRows / 32; ++i)
                    if (32 * i < p.B) n += (t[i] + c - 1) / c;
                if (warp_sum_int(n) * heads <= (int)gridDim.x) chunk = c;
            }
            int carry = 0;
#pragma unroll
            for (int i = 0; i < kSchedRows / 32; ++i) {
                if (32 * i >= p.B) break;
                int v = t[i] == 0 ? 0 : (chunk ? (t[i] + chunk - 1) / chunk : t[i] + kGroupUnits) * heads;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += up;
                }
                sched->end[lane + 32 * i] = carry + v;
                carry += __shfl_sync(0xffffffffu, v, 31);
            }
            if (lane == 0)
                sched->chunk = chunk, sched->lead = chunk ? 0 : kGroupUnits, sched->total = carry,
                sched->whole = !chunk && total <= 4 * p.B * heads;
        }
        __syncthreads();
    }
    auto row_of = [&](int u) {  // the row that unit u belongs to
        int lo = 0, hi = p.B - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sched->end[mid] > u) hi = mid;
            else lo = mid + 1;
        }
        return lo;
    };
    auto first_unit = [&](int c) {  // of CTA c (ranges, whole)
        int u = (int)((long long)sched->total * c / gridDim.x);
        if (sched->whole && u < sched->total) {
            const int b = row_of(u), t = sched->tiles[b] + sched->lead, off = (u - (b ? sched->end[b - 1] : 0)) % t;
            u += 2 * off < t ? -off : t - off;
        }
        return u;
    };
    auto skip_lead = [&]() {  // u0 onto the next unit with a tile
        if (u0 >= u1) return;
        const int b = row_of(u0), off = (u0 - (b ? sched->end[b - 1] : 0)) % (sched->tiles[b] + sched->lead);
        if (off < sched->lead) u0 = min(u1, u0 + sched->lead - off);
    };
    if (SCHED) {
        if (sched->chunk) {
            u0 = cta, u1 = cta < sched->total ? cta + 1 : cta;
        } else {
            u0 = first_unit(cta), u1 = first_unit(cta + 1);
            skip_lead();
        }
    }
    if (u0 >= u1) {
        pdl_wait();
        trace_mark(trec, 3);
        trace_mark(trec, 5);
        return;
    }
    auto take_segment = [&]() {
        AttnSegment sg;
        if (SCHED) {
            sg.b = row_of(u0);
            const int start = sg.b ? sched->end[sg.b - 1] : 0, rem = u0 - start, t = sched->tiles[sg.b];
            int per;  // units of a group of this row
            if (sched->chunk) {
                per = (t + sched->chunk - 1) / sched->chunk;
                sg.part = rem % per, sg.nparts = per;
                sg.t0 = (int)((long long)t * sg.part / per), sg.t1 = (int)((long long)t * (sg.part + 1) / per);
                sg.rec0 = 2LL * (cta - sg.part), sg.rec1 = sg.rec0 + 2;
                u0 = u1;
            } else {
                const int lead = sched->lead;
                per = t + lead;
                sg.t0 = rem % per - lead, sg.t1 = min(t, sg.t0 + (u1 - u0));
                const int g_first = u0 - sg.t0, g_last = g_first + t - 1;  // the group's units with a tile
                // CTA c has the units from total * c / grid on; groups taken whole have one part
                const int c_first = sched->whole ? cta : (int)(((long long)(g_first + 1) * gridDim.x - 1) / sched->total);
                const int c_last = sched->whole ? cta : (int)(((long long)(g_last + 1) * gridDim.x - 1) / sched->total);
                sg.part = cta - c_first, sg.nparts = c_last - c_first + 1;
                // a CTA keeps the record of the group it began in the middle of (or exactly at) in slot 0, that of a
                // group it came to later in slot 1
                sg.rec0 = 2LL * c_first + (first_unit(c_first) < g_first - lead ? 1 : 0), sg.rec1 = 2LL * (c_first + 1);
                u0 += sg.t1 - sg.t0;
                skip_lead();
            }
            const int gi = rem / per;
            sg.kvh = gi / p.nqt, sg.qt = gi % p.nqt, sg.rec_step = 2, sg.len = sched->len[sg.b];
        } else {
            sg.part = blockIdx.x % p.nchunks, sg.nparts = p.nchunks, sg.qt = blockIdx.x / p.nchunks;
            sg.kvh = blockIdx.y, sg.b = blockIdx.z, sg.len = row_len(sg.b);
            const int ct = p.chunk / kTileKeys, all = (sg.len + kTileKeys - 1) / kTileKeys;
            sg.t0 = min(all, sg.part * ct), sg.t1 = min(all, sg.t0 + ct);
            sg.rec0 = (((long long)sg.b * p.NKV + sg.kvh) * p.nqt + sg.qt) * p.nchunks, sg.rec1 = sg.rec0 + 1, sg.rec_step = 1;
            u0 = u1;
        }
        return sg;
    };
    // Row (in units of D elements) of key `key` of a segment's (batch row, kv head) in the cache.
    // A page id outside the pools (a stale or "unallocated" -1 entry) sets ok = false and records a fault; the
    // caller then touches no memory for that key.
    auto cache_row = [&](const AttnSegment& sg, int key, bool& ok, bool before_wait) -> long long {
        ok = true;
        if (!p.page_table) return ((long long)sg.b * p.NKV + sg.kvh) * p.S + key;
        const int* entry = p.page_table + (long long)sg.b * p.max_pages + (key >> p.page_shift);
        const long long page = before_wait ? __ldcg(entry) : *entry;
        if (page < 0 || page >= p.num_pages) {
            report_fault(p.status, FAULT_PAGE_RANGE);
            ok = false;
            return 0;
        }
        return ((page * p.NKV + sg.kvh) << p.page_shift) + (key & ((1 << p.page_shift) - 1));
    };
    auto tiles_of = [&](const AttnSegment& sg) { return (max(0, min(sg.len, sg.t1 * kTileKeys) - sg.t0 * kTileKeys) + kTileKeys - 1) / kTileKeys; };
    // Tile t of a segment into ring stage `stage`; row0 is the cache row of its first key (a tile lies inside one page).
    auto load_tile = [&](const AttnSegment& sg, int t, int stage, long long row0, bool page_ok) {
        unsigned char* st = stages + stage * STAGE_BYTES;
        const int key0 = (sg.t0 + t) * kTileKeys, c1 = min(sg.len, sg.t1 * kTileKeys);
#pragma unroll
        for (int i = 0; i < (2 * kTileKeys * CPR) / kAttnThreads; ++i) {
            const int idx = tid + i * kAttnThreads;
            const int which = idx / (kTileKeys * CPR);
            const int rem = idx % (kTileKeys * CPR);
            const int r = rem / CPR, c = rem % CPR;
            const int key = key0 + r;
            const bool valid = page_ok && key < c1;  // a tile of a bad page is zero-filled, nothing is read
            const bf16* src = (which ? p.V : p.K) + (row0 + (valid ? r : 0)) * D + c * 8;
            const uint32_t dst = smem_u32(st) + which * TILE_BYTES + r * ROW_BYTES + ((c ^ (r & 7)) << 4);
            cp_async16(dst, src, valid);
        }
    };
    // A segment's start-up window: norm weights and rotary rows (inputs of the call), then its first two tiles; always
    // three commit groups.  In decode-layer mode slot len-1 still holds stale data when its tile is requested; the CTA
    // that owns it overwrites that row in shared memory once the tile has landed (see the loop below).
    auto open_segment = [&](const AttnSegment& sg, int ring, bool before_wait) {
        static_assert(kAttnStages == 3, "two tiles ahead, one stage for the merge");
        if (p.fuse_new_token && tid < 4 * CPR) {
            const int which = tid / CPR, c = tid % CPR;
            const bf16* src = which == 0 ? p.q_norm_w : (which == 1 ? p.k_norm_w : (which == 2 ? p.rope_cos : p.rope_sin));
            if (src) cp_async16(smem_u32(rope_s + which * D + c * 8), src + (which >= 2 && p.rope_by_len ? (long long)(sg.len - 1) * D : 0) + c * 8, true);
        }
        cp_async_commit();
        const int n = tiles_of(sg);
        bool ok0 = true, ok1 = true;
        const long long r0 = n > 0 ? cache_row(sg, sg.t0 * kTileKeys, ok0, before_wait) : 0;
        const long long r1 = n > 1 ? cache_row(sg, (sg.t0 + 1) * kTileKeys, ok1, before_wait) : 0;
        if (n > 0) load_tile(sg, 0, ring % kAttnStages, r0, ok0);
        cp_async_commit();
        if (n > 1) load_tile(sg, 1, (ring + 1) % kAttnStages, r1, ok1);
        cp_async_commit();
    };

    int ring = 0;  // tiles of the segments before this one: tile t of a segment lives in stage (ring + t) % 3
    AttnSegment sg = take_segment();
    open_segment(sg, ring, p.early);
    if (p.early) pdl_wait();
    trace_mark(trec, 3);

    for (;;) {
        const int kvh = sg.kvh, b = sg.b, qt = sg.qt, nparts = sg.nparts;
        const int g0 = qt * 16, gn = min(16, G - g0);
        // decode-layer mode: the token being decoded is the last valid key of the row (slot len-1;
        // with one length for all rows that is slot S-1, the reference layer's convention)
        const int new_slot = sg.len - 1;
        const int c0 = sg.t0 * kTileKeys;
        const int c1 = min(sg.len, sg.t1 * kTileKeys);
        const int ntiles = tiles_of(sg);
        const bool owns_new_slot = p.fuse_new_token && c0 <= new_slot && new_slot < c1;
        const bf16* q_norm_w = p.q_norm_w ? rope_s : nullptr;
        const bf16* k_norm_w = p.k_norm_w ? rope_s + D : nullptr;
        const bf16* rope_cos = p.rope_cos ? rope_s + 2 * D : nullptr;
        const bf16* rope_sin = p.rope_sin ? rope_s + 3 * D : nullptr;

        // ---- queries of this kv group into shared memory (rows >= gn are zero) ----
        {
            const bf16* qsrc = p.fuse_new_token ? p.qkv : p.Q;
            const long long qb = p.fuse_new_token ? p.qkv_bstride : p.q_bstride;
            constexpr int QV = (16 * CPR + kAttnThreads - 1) / kAttnThreads;
            uint4 qv[QV];
            bf16 knew[D / 32];  // warp 0: the new token's k, warp 1: its v (the CTA that holds its slot)
#pragma unroll
            for (int u = 0; u < QV; ++u) {  // loads first, stores after: one L2 round trip
                const int idx = tid + u * kAttnThreads;
                const int row = idx / CPR, c = idx % CPR;
                qv[u] = make_uint4(0, 0, 0, 0);
                if (idx < 16 * CPR && row < gn)
                    qv[u] = *reinterpret_cast<const uint4*>(qsrc + (long long)b * qb + (long long)(kvh * G + g0 + row) * D + c * 8);
            }
            if (owns_new_slot && warp < 2) {
                const bf16* src = p.qkv + (long long)b * p.qkv_bstride + p.q_rows + (warp ? p.kv_rows : 0) + kvh * D;
#pragma unroll
                for (int j = 0; j < D / 32; ++j) knew[j] = src[lane + j * 32];
            }
#pragma unroll
            for (int u = 0; u < QV; ++u) {
                const int idx = tid + u * kAttnThreads;
                if (idx < 16 * CPR) *reinterpret_cast<uint4*>(q_s + (idx / CPR) * QS + (idx % CPR) * 8) = qv[u];
            }
            cp_async_wait<2>();  // norm weights and rotary rows
            __syncthreads();
            if (p.fuse_new_token) {
                // unit-weight RMSNorm over the head, fp32 statistics, one rounding
                for (int row = warp; row < gn; row += 4) {
                    float x[D / 32];
#pragma unroll
                    for (int j = 0; j < D / 32; ++j) x[j] = __bfloat162float(q_s[row * QS + lane + j * 32]);
                    head_norm_rope<D>(x, p.eps, q_norm_w, rope_cos, rope_sin, lane);
#pragma unroll
                    for (int j = 0; j < D / 32; ++j) q_s[row * QS + lane + j * 32] = __float2bfloat16_rn(x[j]);
                }
                // new token's k (normalised) and v: kept in shared memory for the patch below and
                // written to cache slot S-1 (nobody reads that slot from memory in this kernel)
                if (owns_new_slot && warp < 2) {
                    bool slot_ok = true;
                    const long long slot = cache_row(sg, new_slot, slot_ok, false) * D;
                    const bool write_slot = slot_ok && qt == 0;  // a bad page: the new k / v are not written anywhere
                    if (warp == 0) {
                        float x[D / 32];
#pragma unroll
                        for (int j = 0; j < D / 32; ++j) x[j] = __bfloat162float(knew[j]);
                        head_norm_rope<D>(x, p.eps, k_norm_w, rope_cos, rope_sin, lane);
#pragma unroll
                        for (int j = 0; j < D / 32; ++j) {
                            const bf16 kn = __float2bfloat16_rn(x[j]);
                            kv_new_s[lane + j * 32] = kn;
                            if (write_slot) p.K_cache_w[slot + lane + j * 32] = kn;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < D / 32; ++j) {
                            kv_new_s[D + lane + j * 32] = knew[j];
                            if (write_slot) p.V_cache_w[slot + lane + j * 32] = knew[j];
                        }
                    }
                }
                __syncthreads();
            }
        }

        // ---- A fragments of Q: 16 rows x D, D/16 k-steps ----
        uint32_t qa[D / 16][4];
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            const bf16* base = q_s + kk * 16 + t4 * 2;
            qa[kk][0] = *reinterpret_cast<const uint32_t*>(base + g4 * QS);
            qa[kk][1] = *reinterpret_cast<const uint32_t*>(base + (g4 + 8) * QS);
            qa[kk][2] = *reinterpret_cast<const uint32_t*>(base + g4 * QS + 8);
            qa[kk][3] = *reinterpret_cast<const uint32_t*>(base + (g4 + 8) * QS + 8);
        }

        float o[D / 8][4];
#pragma unroll
        for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
        float m_run[2] = {-INFINITY, -INFINITY};
        float l_run[2] = {0.f, 0.f};

        // the cache row of the tile two ahead is looked up one iteration before its copy is issued
        bool ahead_ok = true;
        long long ahead = ntiles > 2 ? cache_row(sg, c0 + 2 * kTileKeys, ahead_ok, false) : 0;
        for (int t = 0; t < ntiles; ++t) {
            cp_async_wait<kAttnStages - 2>();
            __syncthreads();
            if (t == 0) trace_mark(trec, 4);
            if (t + 2 < ntiles) load_tile(sg, t + 2, (ring + t + 2) % kAttnStages, ahead, ahead_ok);
            cp_async_commit();
            if (t + 3 < ntiles) ahead = cache_row(sg, c0 + (t + 3) * kTileKeys, ahead_ok, false);
            if (owns_new_slot && t == ntiles - 1) {
                // overwrite the stale row of slot S-1 in this tile with the new token's k and v
                const int r = new_slot - (c0 + t * kTileKeys);
                if (tid < 2 * CPR) {
                    const int which = tid / CPR, c = tid % CPR;
                    unsigned char* dst = stages + ((ring + t) % kAttnStages) * STAGE_BYTES + which * TILE_BYTES + r * ROW_BYTES + ((c ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(kv_new_s + which * D + c * 8);
                }
                __syncthreads();
            }

            const unsigned char* st = stages + ((ring + t) % kAttnStages) * STAGE_BYTES;
            const uint32_t k_s = smem_u32(st), v_s = k_s + TILE_BYTES;
            const int kr0 = warp * 16;

            // ---- S = Q K^T for this warp's 16 keys ----
            float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            {
                const int mi = lane >> 3, rr = lane & 7;
                const int key_local = kr0 + (mi >> 1) * 8 + rr;
                const uint32_t row_addr = k_s + key_local * ROW_BYTES;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    const int chunk = kk * 2 + (mi & 1);
                    uint32_t b00, b01, b10, b11;
                    ldsm_x4(row_addr + ((chunk ^ (key_local & 7)) << 4), b00, b01, b10, b11);
                    mma_bf16_16816(s[0], qa[kk][0], qa[kk][1], qa[kk][2], qa[kk][3], b00, b01);
                    mma_bf16_16816(s[1], qa[kk][0], qa[kk][1], qa[kk][2], qa[kk][3], b10, b11);
                }
            }
            // ---- online soft-max (exp2 domain) ----
            const int key_base = c0 + t * kTileKeys + kr0 + t4 * 2;
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int key = key_base + j * 8 + (e & 1);
                    s[j][e] = (key < c1) ? s[j][e] * p.scale_log2e : -INFINITY;
                    mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
                }
            float alpha[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
                mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
                const float m_new = fmaxf(m_run[r], mx[r]);
                const float m_safe = (m_new == -INFINITY) ? 0.f : m_new;
                alpha[r] = fast_exp2(m_run[r] - m_safe);
                m_run[r] = m_new;
                float psum = 0.f;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    s[j][2 * r] = fast_exp2(s[j][2 * r] - m_safe);
                    s[j][2 * r + 1] = fast_exp2(s[j][2 * r + 1] - m_safe);
                    psum += s[j][2 * r] + s[j][2 * r + 1];
                }
                l_run[r] = l_run[r] * alpha[r] + psum;
            }
#pragma unroll
            for (int i = 0; i < D / 8; ++i) {
                o[i][0] *= alpha[0], o[i][1] *= alpha[0];
                o[i][2] *= alpha[1], o[i][3] *= alpha[1];
            }
            // ---- O += P V ----
            const uint32_t pa0 = pack_bf16(s[0][0], s[0][1]), pa1 = pack_bf16(s[0][2], s[0][3]);
            const uint32_t pa2 = pack_bf16(s[1][0], s[1][1]), pa3 = pack_bf16(s[1][2], s[1][3]);
            {
                const int mi = lane >> 3, rr = lane & 7;
                const int key_local = kr0 + (mi & 1) * 8 + rr;
                const uint32_t row_addr = v_s + key_local * ROW_BYTES;
#pragma unroll
                for (int dn = 0; dn < D / 16; ++dn) {
                    const int chunk = dn * 2 + (mi >> 1);
                    uint32_t v0, v1, v2, v3;
                    ldsm_x4_trans(row_addr + ((chunk ^ (key_local & 7)) << 4), v0, v1, v2, v3);
                    mma_bf16_16816(o[2 * dn], pa0, pa1, pa2, pa3, v0, v1);
                    mma_bf16_16816(o[2 * dn + 1], pa0, pa1, pa2, pa3, v2, v3);
                }
            }
        }
        cp_async_wait<0>();
        // The next segment's first tiles are on their way while this one is merged: every warp is past the tile before
        // last, so the two stages in front of the last tile's are free.
        ring += ntiles;
        const bool more = SCHED && u0 < u1;
        AttnSegment next = sg;
        if (more) {
            next = take_segment();
            open_segment(next, ring, false);
        }
        __syncthreads();

        // ---- merge the four warps (each saw a quarter of the keys) ----
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
            l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
        }
        float* mrg_m = mrg_ml;       // [4][16]
        float* mrg_l = mrg_ml + 64;  // [4][16]
        float* mrg_o = reinterpret_cast<float*>(stages + ((ring + 2) % kAttnStages) * STAGE_BYTES);  // [4][16][D]: one stage
        // columns are XORed with 8 * (row % 8): unswizzled, the eight rows of a store share their banks
        if (t4 == 0) {
            mrg_m[warp * 16 + g4] = m_run[0], mrg_m[warp * 16 + g4 + 8] = m_run[1];
            mrg_l[warp * 16 + g4] = l_run[0], mrg_l[warp * 16 + g4 + 8] = l_run[1];
        }
#pragma unroll
        for (int i = 0; i < D / 8; ++i) {
            float* dst = mrg_o + (warp * 16 + g4) * D + ((i ^ g4) * 8 + t4 * 2);
            *reinterpret_cast<float2*>(dst) = make_float2(o[i][0], o[i][1]);
            if (gn > 8) *reinterpret_cast<float2*>(dst + 8 * D) = make_float2(o[i][2], o[i][3]);
        }
        __syncthreads();

        const long long group = ((long long)b * p.NKV + kvh) * p.nqt + qt;
        auto rec_of = [&](int c) { return c == 0 ? sg.rec0 : sg.rec1 + (long long)(c - 1) * sg.rec_step; };
        const long long item = sg.part == 0 ? sg.rec0 : sg.rec1 + (long long)(sg.part - 1) * sg.rec_step;
        for (int idx = tid; idx < gn * (D / 4); idx += kAttnThreads) {
            const int row = idx / (D / 4), d = (idx % (D / 4)) * 4;
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < 4; ++w) M = fmaxf(M, mrg_m[w * 16 + row]);
            float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
            float L = 0.f;
            if (M != -INFINITY) {
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const float f = fast_exp2(mrg_m[w * 16 + row] - M);
                    const float4 v = *reinterpret_cast<const float4*>(mrg_o + (w * 16 + row) * D + (d ^ ((row & 7) * 8)));
                    O.x += f * v.x, O.y += f * v.y, O.z += f * v.z, O.w += f * v.w;
                    L += f * mrg_l[w * 16 + row];
                }
            }
            if (nparts == 1) {
                const bool any = L > 0.f;
                bf16* dst = p.Out + (long long)b * p.o_bstride + (long long)(kvh * G + g0 + row) * D + d;
                *reinterpret_cast<uint2*>(dst) = any ? make_uint2(pack_bf16(O.x / L, O.y / L), pack_bf16(O.z / L, O.w / L)) : make_uint2(0u, 0u);
            } else {
                *reinterpret_cast<float4*>(p.part_o + (item * 16 + row) * D + d) = O;
                if (d == 0) *reinterpret_cast<float2*>(p.part_ml + (item * 16 + row) * 2) = make_float2(M, L);
            }
        }
        bool fold = false;
        if (nparts > 1) {
            // ---- the last CTA of this (row, kv head, q tile) folds the splits together ----
            // One acq_rel atomic after the barrier both publishes this CTA's records (the
            // barrier orders the other threads' stores before it) and, for the CTA that
            // draws the last ticket, makes every other CTA's records visible.
            __syncthreads();
            if (tid == 0) {
                unsigned int prev;
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(p.counters + group) : "memory");
                s_is_last = (prev == (unsigned int)(nparts - 1));
            }
            __syncthreads();
            fold = s_is_last;
        }
        if (fold && nparts <= 32) {
            // Fast path: every thread owns four output dims of one head and issues all
            // its loads up front (32 split records + the first 16 partial vectors), so
            // the whole fold costs two L2 round trips.
            for (int idx = tid; idx < gn * (D / 4); idx += kAttnThreads) {
                const int row = idx / (D / 4), d = (idx % (D / 4)) * 4;
                const float* pm = p.part_ml + row * 2;
                const float* po = p.part_o + row * D + d;
                float2 ml[32];
                float4 v[16];
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    ml[c] = (c < nparts) ? __ldcg(reinterpret_cast<const float2*>(pm + rec_of(c) * 32)) : make_float2(-INFINITY, 0.f);
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    v[c] = (c < nparts) ? __ldcg(reinterpret_cast<const float4*>(po + rec_of(c) * 16 * D)) : make_float4(0.f, 0.f, 0.f, 0.f);
                float M = -INFINITY;
#pragma unroll
                for (int c = 0; c < 32; ++c) M = fmaxf(M, ml[c].x);
                float L = 0.f;
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    ml[c].x = (M != -INFINITY) ? fast_exp2(ml[c].x - M) : 0.f;
                    L += ml[c].x * ml[c].y;
                }
                const float inv = (L > 0.f) ? 1.0f / L : 0.f;
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    const float f = ml[c].x;
                    acc.x += f * v[c].x, acc.y += f * v[c].y, acc.z += f * v[c].z, acc.w += f * v[c].w;
                }
                if (nparts > 16) {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        v[c] = (c + 16 < nparts) ? __ldcg(reinterpret_cast<const float4*>(po + rec_of(c + 16) * 16 * D))
                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const float f = ml[c + 16].x;
                        acc.x += f * v[c].x, acc.y += f * v[c].y, acc.z += f * v[c].z, acc.w += f * v[c].w;
                    }
                }
                bf16* dst = p.Out + (long long)b * p.o_bstride + (long long)(kvh * G + g0 + row) * D + d;
                *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
            }
        } else if (fold) {
            // Any number of parts: statistics first, then the weighted sum, sixteen records in flight.
            for (int idx = tid; idx < gn * (D / 4); idx += kAttnThreads) {
                const int row = idx / (D / 4), d = (idx % (D / 4)) * 4;
                const float* pm = p.part_ml + row * 2;
                const float* po = p.part_o + row * D + d;
                float M = -INFINITY, L = 0.f;
                for (int c = 0; c < nparts; c += 16) {
                    float2 ml[16];
                    float m_new = M;
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        ml[u] = (c + u < nparts) ? __ldcg(reinterpret_cast<const float2*>(pm + rec_of(c + u) * 32)) : make_float2(-INFINITY, 0.f);
                        m_new = fmaxf(m_new, ml[u].x);
                    }
                    if (m_new == -INFINITY) continue;
                    L *= fast_exp2(M - m_new);
#pragma unroll
                    for (int u = 0; u < 16; ++u) L += fast_exp2(ml[u].x - m_new) * ml[u].y;
                    M = m_new;
                }
                const float inv = (L > 0.f) ? 1.0f / L : 0.f;
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int c = 0; c < nparts; c += 16) {
                    float4 v[16];
                    float f[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        f[u] = (c + u < nparts) ? __ldcg(pm + rec_of(c + u) * 32) : -INFINITY;
                        v[u] = (c + u < nparts) ? __ldcg(reinterpret_cast<const float4*>(po + rec_of(c + u) * 16 * D)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const float w = (M != -INFINITY) ? fast_exp2(f[u] - M) * inv : 0.f;
                        acc.x += w * v[u].x, acc.y += w * v[u].y, acc.z += w * v[u].z, acc.w += w * v[u].w;
                    }
                }
                bf16* dst = p.Out + (long long)b * p.o_bstride + (long long)(kvh * G + g0 + row) * D + d;
                *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(acc.x, acc.y), pack_bf16(acc.z, acc.w));
            }
        }
        if (fold && tid == 0) p.counters[group] = 0u;  // ready for the next call
        if (!more) break;
        __syncthreads();  // the merge stage is the next segment's third
        sg = next;
    }
    trace_mark(trec, 5);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// Rows of equal length are cut so that all CTAs are resident together, in ONE wave: as many splits per (row, kv
// head) as the resident slots allow, never more.  A second, partly filled wave costs a whole extra pass over a split
// (Qwen3-8B layer, KV 4096, batch 2 / 4 / 8 / 16 / 32: 94.5 / 110.5 / 126.8 / 147.1 / 191.4 us with splits sized for
// 1.5 waves, 89.5 / 107.4 / 124.6 / 141.2 / 181.6 with this rule; a sweep over every split length confirmed the
// optimum at ~256 CTAs for each).  Head dim 64 (32 heads over 8 kv heads; splits for four CTAs per SM, of which three are
// resident | this rule): 1 row of 8192 keys 13.5 | 10.3 us, 8 rows of 4096 16.2 | 13.4, 24 rows of 2048 21.8 | 18.6.
// Ragged batches get the balanced schedule (AttnSchedule) where launch_attn_instance says so.  Elsewhere, with more rows
// than it covers, or with EZB_TUNE_ATTN_WAVES > 0, they are cut into more, shorter splits, because every row is then cut on
// the grid of the longest row and short splits balance better.
int attn_chunk_keys(int B, int NKV, int S, bool ragged, int D) {
    const long long total = (long long)B * NKV * S;
    const int waves = tuning(ragged ? EZB_TUNE_ATTN_WAVES : EZB_TUNE_ATTN_WAVES_UNIFORM);
    long long chunk;
    if (!ragged && waves <= 0) {
        const long long slots = (long long)sm_count() * attn_ctas_per_sm(D);
        long long splits = slots / ((long long)B * NKV);
        if (splits < 1) splits = 1;
        chunk = (S + splits - 1) / splits;
    } else {
        const long long target = (long long)sm_count() * (waves > 0 ? waves : 8);
        chunk = (total + target - 1) / target;
    }
    chunk = (chunk + kTileKeys - 1) / kTileKeys * kTileKeys;
    long long floor_keys = max(kTileKeys, tuning(EZB_TUNE_ATTN_MIN_CHUNK) / kTileKeys * kTileKeys);
    if (chunk < floor_keys) chunk = floor_keys;
    const long long cap = ((long long)S + kTileKeys - 1) / kTileKeys * kTileKeys;
    if (chunk > cap) chunk = cap;
    while ((S + chunk - 1) / chunk > 256) chunk += kTileKeys;
    return (int)chunk;
}

static size_t counters_bytes(int B, int NKV, int nqt) { return ((size_t)B * NKV * nqt * 4 + 255) / 256 * 256; }

size_t attn_counters_bytes(int B, int H, int NKV) {
    const int G = H / NKV;
    return counters_bytes(B, NKV, (G + 15) / 16);
}

static bool balanced(int B, bool ragged) { return ragged && B <= kSchedRows && tuning(EZB_TUNE_ATTN_WAVES) <= 0; }

template <int D>
static constexpr size_t attn_smem_bytes() {
    return (size_t)kAttnStages * 2 * kTileKeys * D * 2 + 16 * (D + 8) * 2 + 6 * D * 2;
}

// CTAs of the balanced kernel that are resident together on the current device.
template <int D>
static int attn_slots() {
    static std::atomic<int> cache[64];
    int dev = 0;
    cudaGetDevice(&dev);
    const bool keep = dev >= 0 && dev < 64;
    if (keep)
        if (const int known = cache[dev].load(std::memory_order_relaxed)) return known;
    constexpr size_t smem = attn_smem_bytes<D>() + sizeof(AttnSchedule);
    int per_sm = 0;
    if (cudaFuncSetAttribute(attn_decode_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, attn_decode_kernel<D, true>, kAttnThreads, smem) != cudaSuccess || per_sm < 1)
        return sm_count();
    const int n = per_sm * sm_count();
    if (keep) cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

size_t attn_workspace_bytes(int B, int H, int NKV, int S, int D) {
    const int G = H / NKV, nqt = (G + 15) / 16;
    const int chunk = min(attn_chunk_keys(B, NKV, S, false, D), attn_chunk_keys(B, NKV, S, true, D));  // covers both cuts
    const int nchunks = (S + chunk - 1) / chunk;
    size_t items = (size_t)B * NKV * nqt * nchunks;
    // the balanced schedule keeps two records per CTA of its grid, which never exceeds the number of tiles
    const size_t tiles = (size_t)B * NKV * nqt * ((S + kTileKeys - 1) / kTileKeys);
    size_t slots = (size_t)sm_count() * attn_ctas_per_sm(D);
    if (slots > tiles) slots = tiles;
    if (B <= kSchedRows && 2 * slots > items) items = 2 * slots;
    return counters_bytes(B, NKV, nqt) + items * 16 * 2 * sizeof(float) + items * 16 * D * sizeof(float);
}

template <int D>
static cudaError_t launch_attn_instance(AttnParams& p, void* records, cudaStream_t stream) {
    bool sched = balanced(p.B, p.seq_lens != nullptr);
    int slots = 0;
    if (sched) {
        slots = attn_slots<D>();
        const int most = sm_count() * attn_ctas_per_sm(D);
        if (slots > most) slots = most;
        const long long tiles = (long long)p.B * p.NKV * p.nqt * ((p.S + kTileKeys - 1) / kTileKeys);
        if (slots > tiles) slots = (int)tiles;
        // If the wave holds the smallest splits of rows of full length, there is nothing to balance (0.6B, 4 rows of
        // 128..1024 keys, 28 layers: 858 us, 886 with the schedule computed in front of every layer's attention).
        const int cut = min(p.min_tiles * kTileKeys, (p.S + kTileKeys - 1) / kTileKeys * kTileKeys);
        const int n = (p.S + cut - 1) / cut;
        const long long groups = (long long)p.B * p.NKV * p.nqt;
        if (groups * n <= slots) sched = false, p.chunk = cut, p.nchunks = n;
        // Where the fixed grid does not cut a row either (a row is one split, or there are so many that each gets a CTA
        // of its own) the hardware hands out the groups one by one, which beats fixed shares of them: 64 rows of 13..100
        // keys 8.4 us on the grid, 15.5 by schedule; 128 rows of 48..384 keys 28 and 40; 45 rows of 112..900 keys and 32
        // kv heads 58 and 68; even from about 3000 keys on.
        else if (p.nchunks == 1) sched = false;
        // Head dim 64: a new group costs as much as at 128 but its tiles cost half, so the schedule gains only where groups
        // are few and long (11 rows of 512..4096 keys 17.3 us on the grid, 14.8 by schedule) and loses elsewhere (64 rows of
        // 64..512 keys 15.2 and 19.5).  Over 2000 shapes this rule is 11..14 % faster than the schedule wherever something
        // is cut, the grid everywhere 10..12 %.  Few and short groups leave the chip half empty anyway: one wave of splits
        // as for rows of one length (1 row of 8192 keys at most: 12.8 us in more, shorter splits, 10.6 so).
        else if (D <= 64 && (2 * groups > slots || tiles <= 4LL * slots)) {
            sched = false;
            if (2 * groups <= slots) p.chunk = max(p.chunk, attn_chunk_keys(p.B, p.NKV, p.S, false, D));
            p.nchunks = (p.S + p.chunk - 1) / p.chunk;
        }
    }
    const size_t items = sched ? 2 * (size_t)slots : (size_t)p.B * p.NKV * p.nqt * p.nchunks;
    p.part_ml = static_cast<float*>(records);
    p.part_o = p.part_ml + items * 16 * 2;
    if (sched)
        return launch_pdl(attn_decode_kernel<D, true>, dim3(slots), dim3(kAttnThreads), attn_smem_bytes<D>() + sizeof(AttnSchedule), stream, p);
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(attn_decode_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attn_smem_bytes<D>());
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    return launch_pdl(attn_decode_kernel<D, false>, dim3(p.nchunks * p.nqt, p.NKV, p.B), dim3(kAttnThreads), attn_smem_bytes<D>(), stream, p);
}

cudaError_t launch_attn_decode(const AttnArgs& a, cudaStream_t stream) {
    AttnParams p;
    p.Q = a.Q, p.q_bstride = a.q_bstride, p.K = a.K, p.V = a.V, p.Out = a.Out, p.o_bstride = a.o_bstride;
    p.seq_lens = a.seq_lens;
    p.B = a.B, p.H = a.H, p.NKV = a.NKV, p.S = a.S, p.G = a.H / a.NKV;
    p.nqt = (p.G + 15) / 16;
    p.chunk = attn_chunk_keys(a.B, a.NKV, a.S, a.seq_lens != nullptr, a.D);
    p.nchunks = (a.S + p.chunk - 1) / p.chunk;
    p.scale_log2e = 1.4426950408889634f / sqrtf((float)a.D);
    unsigned char* ws = reinterpret_cast<unsigned char*>(a.workspace);
    p.counters = reinterpret_cast<unsigned int*>(ws);
    p.min_tiles = max(1, tuning(EZB_TUNE_ATTN_MIN_CHUNK) / kTileKeys);
    // Inside a chain whose first kernel began after everything in front of it, the caches, the lengths and the page table
    // are complete before this kernel starts (not if calls may overlap).
    p.first = chain_waits_first();
    p.early = tuning(EZB_TUNE_PDL) && !tuning(EZB_TUNE_PDL_ACROSS_CALLS) && !chain_at_first();
    p.fuse_new_token = a.fuse_new_token;
    p.qkv = a.qkv, p.qkv_bstride = a.qkv_bstride;
    p.q_rows = a.H * a.D, p.kv_rows = a.NKV * a.D;
    p.K_cache_w = a.K_cache_w, p.V_cache_w = a.V_cache_w;
    p.eps = a.eps;
    p.q_norm_w = a.q_norm_w, p.k_norm_w = a.k_norm_w, p.rope_cos = a.rope_cos, p.rope_sin = a.rope_sin;
    p.rope_by_len = a.rope_by_len;
    p.page_table = a.page_table, p.page_shift = a.page_shift, p.max_pages = a.max_pages, p.num_pages = a.num_pages;
    p.status = status_ptr();
    if (!p.status) return cudaErrorUnknown;
    p.next = a.next;
    if (!tuning(EZB_TUNE_L2_PREFETCH)) p.next.plan[0].units = p.next.plan[1].units = 0;
    p.trace = trace_handle();
    void* records = ws + counters_bytes(a.B, a.NKV, p.nqt);
    if (a.D == 128) return launch_attn_instance<128>(p, records, stream);
    return launch_attn_instance<64>(p, records, stream);
}

}  // namespace ezb
