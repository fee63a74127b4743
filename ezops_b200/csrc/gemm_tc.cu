// Batched projections on the 5th-generation tensor cores:
//   Y[b, n] = epi( sum_k X[b, k] * W[n, k] ),   2 <= b <= 64,
// used once the batch turns the weight-streaming GEMV into a skinny GEMM.
//
// The weights are read from HBM exactly once and that is what bounds the kernel, so it is built like the GEMV (TMA
// ring, programmatic dependent launch) with the arithmetic on tcgen05:
//   * "swap AB": a tile is up to 128 weight rows (the MMA's M) by the whole batch (the MMA's N = 16, 32 or 64) and
//     walks K in blocks of 64 elements;
//   * one elected thread issues cp.async.bulk.tensor (2-D tiled TMA, 128-byte swizzle) for the W block [rows x 64]
//     and the X block [N x 64] of a stage; one elected thread issues tcgen05.mma (kind::f16, bf16 x bf16 -> fp32)
//     with the accumulator in tensor memory, and tcgen05.commit hands the stage back to the producer when the MMAs
//     that read it have retired; the accumulator is double buffered, so a tile's epilogue overlaps the next tile;
//   * K is split over the CTAs of a thread-block cluster (1, 2, 4 or 8).  A CTA writes the batch columns of its
//     partial tile that belong to CTA j straight from tensor memory into CTA j's shared memory (DSMEM), one mbarrier
//     arrival per warp and destination; CTA j adds the parts in cluster rank order (fixed order: results are
//     bit-reproducible) and applies the epilogue to its columns;
//   * the number of rows of a tile is free (the TMA box is encoded with it), so that the host can deal N rows evenly
//     to the clusters that fit on the chip (tc_plan below);
//   * a CTA takes at most half of an SM (shared memory, registers, tensor memory), so that the next kernel of a chain
//     can be resident while this one drains and already has its weight ring in flight when its input is complete.
//   * the LINK instance serves the fused tensor-parallel exchange (see TpLink).
// Every mbarrier wait is bounded; on a time-out the CTA records a fault, stops issuing work, waits (bounded) for
// copies in flight, frees its tensor memory and returns.
#include <cuda.h>

#include <atomic>
#include <mutex>

#include "launchers.h"
#include "map_table.h"

namespace ezb {

static constexpr int kTcRows = 128;     // MMA M; a tile holds at most this many weight rows
static constexpr int kTcBlockK = 64;    // k elements per stage: 128 bytes, one swizzle row
static constexpr int kTcEpiWarps = 8;
static constexpr int kTcThreads = 64 + 32 * kTcEpiWarps;  // TMA warp, MMA warp, epilogue warps
static constexpr int kTcMaxStages = 40;
static constexpr int kTcMaxCluster = 8;
static constexpr int kTcNormAt = 1024;     // scratch of the norm factors behind the barriers: 256 partial sums, 64 factors
static constexpr int kTcTailBytes = kTcNormAt + (256 + 64) * 4;

struct TcParams {
    int N, K, B;          // output units (rows, or gate/up pairs), reduction length, batch
    int tiles, kblocks;   // ceil(N / units), ceil(K / 64)
    int units;            // output units per tile (<= 128, or <= 64 pairs)
    int half_rows;        // pair: first row of the up block inside a tile (units rounded up to 8); else 0
    int a_rows;           // rows of the W block in a stage, a multiple of 8
    int log2c;            // log2 of the cluster size
    int cpc;              // batch columns that one CTA of the cluster finishes
    int nstages;
    int first;            // see pdl_open
    int pair;             // 1: a tile holds `units` gate rows and `units` up rows, SwiGLU epilogue
    int epilogue;
    const bf16* residual;
    long long ldres;
    void* out;
    long long ldout;
    unsigned int* status;
    // deferred RMSNorm (GemvArgs::ssq)
    const float* ssq_in;  // sums of squares of the input rows; their factor is applied to the products
    int ssq_parts;
    float inv_dim, eps;
    int cols_pad;       // cpc rounded up to a power of two
    float* ssq_out;     // sums of squares of the result rows, one part per tile and 32 rows
    bf16* xw_out;       // result * next_norm_w
    const bf16* next_norm_w;
    Trace trace;
    int trace_id;
    TpLink link;  // fused tensor-parallel exchange (world 0: none); only the push side lives in this kernel
};

// ---- tcgen05 / TMA wrappers -------------------------------------------------
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns: thread i of the warp gets lane (base lane + i)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major bf16 tile whose rows are 128
// bytes (64 elements) with the 128-byte swizzle that the tiled TMA wrote:
// start address / 16, stride between 8-row groups 1024 bytes, descriptor
// version 1 (sm_100), layout type 2 (128-byte swizzle).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

// Instruction descriptor, kind::f16: fp32 accumulator, bf16 A and B, both
// K-major, N in units of 8 at bit 17, M in units of 16 at bit 24.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ---- cluster wrappers -------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Relaxed: what the peers must see first is ordered otherwise (fence.mbarrier_init at the start; at the end every copy
// and arrival towards a peer has been waited for by that peer).  The release form waited for every store in flight.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// Address of `local` (a shared::cta address) in the shared memory of cluster CTA `rank`.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bulk copy from this CTA's shared memory into another CTA's of the cluster; the bytes are counted on that CTA's barrier.
__device__ __forceinline__ void bulk_s2cluster(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// As mbar_wait_bounded, for arrivals from other CTAs of the cluster.
__device__ __forceinline__ bool mbar_wait_bounded_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                          unsigned int* status, unsigned int fault_code) {
    const long long t0 = clock64();
    while (!mbar_try_wait_cluster(bar, parity)) {
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitLimitCycles) {
            *abort_flag = 1;
            report_fault(status, fault_code);
            return false;
        }
    }
    return true;
}

// One thread of a converged warp.  Unlike `lane == 0`, the compiler knows that exactly one thread enters the branch and
// keeps descriptors and addresses in uniform registers: four MMAs and their commit issue in 171 cycles instead of 264.
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}

// 32 lanes x 8 columns, see tmem_ld16
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// What bounds it: the weight stream.  A tile's parts meet in shared memory because the round trips of a reduction
// through L2 (park, ticket, read 4..19 parts in one CTA) cost 5..13 us at the end of every projection.
// Measured: Qwen3-8B layer, batch 32, KV 4096 187.9 -> 168.0 us; eight 2B layers, batch 13, paged 680 -> 488 us.
// A norm in front of a projection is left to its epilogue (ssq_in): the kernel that produced the rows has written their
// sums of squares and the rows times the norm weight, so no row kernel runs between two projections (3..6 us each; the
// 2B layers above 488 -> 438 us, 28 layers of 0.6B at batch 4 1008 -> 858 us).
// LINK: the instance for chains with the fused exchange: its epilogue can push fp32 results into the peers' inboxes (see
// TpLink), and its waits start behind the gather of the kernel in front.
template <int NB, bool LINK>
__global__ void __launch_bounds__(kTcThreads, 2)
gemm_tc_kernel(const __grid_constant__ CUtensorMap mapW0, const __grid_constant__ CUtensorMap mapW1,
               const __grid_constant__ CUtensorMap mapX, const TcParams p) {
    constexpr int B_BYTES = NB * kTcBlockK * 2;
    constexpr int TMEM_COLS = (2 * NB < 32) ? 32 : 2 * NB;  // two accumulators, power of two >= 32
    constexpr uint32_t IDESC = umma_idesc_bf16(kTcRows, NB);

    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    unsigned char* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);  // swizzled tiles need 1024-byte alignment
    const uint32_t a_bytes = (uint32_t)p.a_rows * (kTcBlockK * 2);
    const uint32_t stage_bytes = a_bytes + B_BYTES;
    unsigned char* stages = smem;
    unsigned char* tail = smem + (size_t)p.nstages * stage_bytes;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tail);
    uint64_t* empty_bar = full_bar + kTcMaxStages;
    uint64_t* acc_full = empty_bar + kTcMaxStages;  // [2] accumulator ready for the epilogue
    uint64_t* acc_empty = acc_full + 2;             // [2] accumulator drained
    uint64_t* recv_full = acc_empty + 2;            // the parts of all CTAs of the cluster have arrived in recv
    uint64_t* recv_free = recv_full + 1;            // all CTAs of the cluster have read what this CTA sent them
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(recv_free + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* norm_sum = reinterpret_cast<float*>(tail + kTcNormAt);                // [256 / cols_pad][cols_pad]
    float* norm_r = norm_sum + 256;                                             // norm factor of each column of this CTA
    const int RS = p.a_rows;                                                    // rows of a column of a partial tile
    float* mine = reinterpret_cast<float*>(tail + kTcTailBytes);                // [column][RS]: this CTA's part of the tile
    float* recv = mine + (size_t)(p.cpc << p.log2c) * RS;                       // [sender][column of this CTA][RS]

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int NS = p.nstages, KB = p.kblocks;
    const int C = 1 << p.log2c;
    const int rank = (int)cluster_rank();
    const int cluster = blockIdx.x >> p.log2c, n_clusters = gridDim.x >> p.log2c;
    const int kb0 = (int)((long long)KB * rank >> p.log2c), kb1 = (int)((long long)KB * (rank + 1) >> p.log2c);
    const int my_tiles = (p.tiles - cluster + n_clusters - 1) / n_clusters;

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&acc_full[a]), 1);
            mbar_init(smem_u32(&acc_empty[a]), kTcEpiWarps);
        }
        mbar_init(smem_u32(recv_full), 1);
        mbar_init(smem_u32(recv_free), kTcEpiWarps * C);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    unsigned long long* trec = (tid == 64) ? trace_open(p.trace, (unsigned)p.trace_id, blockIdx.x) : nullptr;
    pdl_open(p.first);
    // The barriers above are initialised: peers may write here once they have passed the wait.  (A launch without a
    // cluster leaves the cluster barrier alone: there its wait held the epilogue until every warp of the CTA had come.)
    if (C > 1) cluster_arrive();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            const int n_units = my_tiles * (kb1 - kb0);
            const int box_rows = p.pair ? 2 * p.units : p.units;
            const uint32_t tx = (uint32_t)box_rows * (kTcBlockK * 2) + B_BYTES;
            // Two cursors over (tile, k-block): the next unit whose weights / activations are requested.  The clusters
            // start their walk along K at different blocks: in step, all of them would ask the same few lines of X of
            // the L2 at the same time (a k-block took 270 ns however small its tile).
            const int k_first = kb0 + (int)((long long)(kb1 - kb0) * cluster / n_clusters);
            int wt = cluster, wkb = k_first, xkb = k_first;
            int stage = 0;
            uint32_t empty_parity = 1;  // a fresh barrier passes a wait on parity 1
            auto request_w = [&](int st) {
                const uint32_t bar = smem_u32(&full_bar[st]);
                mbar_arrive_expect_tx(bar, tx);
                const uint32_t a = smem_u32(stages) + (uint32_t)st * stage_bytes;
                tma_load_2d(a, &mapW0, wkb * kTcBlockK, wt * p.units, bar);
                if (p.pair) tma_load_2d(a + (uint32_t)p.half_rows * (kTcBlockK * 2), &mapW1, wkb * kTcBlockK, wt * p.units, bar);
                if (++wkb == kb1) wkb = kb0;
                if (wkb == k_first) wt += n_clusters;
            };
            auto request_x = [&](int st) {
                tma_load_2d(smem_u32(stages) + (uint32_t)st * stage_bytes + a_bytes, &mapX, xkb * kTcBlockK, 0, smem_u32(&full_bar[st]));
                if (++xkb == kb1) xkb = kb0;
            };
            // weights do not depend on the kernel in front: request them before the dependency wait
            const int npre = n_units < NS ? n_units : NS;
            for (int i = 0; i < npre; ++i) request_w(i);
            pdl_wait();
            for (int i = 0; i < npre; ++i) request_x(i);
            int issued = npre;
            stage = (npre == NS) ? 0 : npre;
            if (npre == NS) empty_parity = 0;
            for (int i = npre; i < n_units; ++i) {
                if (!mbar_wait_bounded(smem_u32(&empty_bar[stage]), empty_parity, abort_flag, p.status, FAULT_GEMV_EMPTY_WAIT)) break;
                request_w(stage);
                request_x(stage);
                if (++stage == NS) stage = 0, empty_parity ^= 1;
                issued = i + 1;
            }
            if (*abort_flag) {  // nothing may still be landing in this CTA's shared memory when it exits
                const int first = issued > NS ? issued - NS : 0;
                for (int i = first; i < issued; ++i) {
                    const long long t0 = clock64();
                    while (!mbar_try_wait(smem_u32(&full_bar[i % NS]), (uint32_t)((i / NS) & 1)))
                        if (clock64() - t0 > kWaitLimitCycles) {
                            report_fault(p.status, FAULT_GEMV_DRAIN);
                            break;
                        }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            // A stage is full only with the X block that the producer requests behind its own dependency wait.  Behind a
            // gather, which may wait for its peers for seconds and has released this kernel before, waiting here too keeps
            // that time out of the budget of the waits below.  (Elsewhere it only costs, even as a branch not taken: 30 ns
            // a projection.)
            if (LINK) pdl_wait();
            int stage = 0;
            uint32_t full_parity = 0;
            for (int i = 0; i < my_tiles && !(*abort_flag); ++i) {
                const int acc = i & 1;
                // wait until the epilogue has drained this accumulator (passes at once for its first use)
                if (!mbar_wait_bounded(smem_u32(&acc_empty[acc]), (uint32_t)(((i >> 1) & 1) ^ 1), abort_flag, p.status, FAULT_TC_ACC_WAIT))
                    break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * NB);
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait_bounded(smem_u32(&full_bar[stage]), full_parity, abort_flag, p.status, FAULT_GEMV_FULL_WAIT))
                        break;
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(stages) + (uint32_t)stage * stage_bytes;
                    const uint64_t adesc = umma_desc_sw128(a_addr);
                    const uint64_t bdesc = umma_desc_sw128(a_addr + a_bytes);
                    // A tile with fewer than 128 rows is multiplied as if it had 128: the rows behind it are whatever
                    // the shared memory holds, and the accumulator lanes they end up in are never read.
#pragma unroll
                    for (int k = 0; k < kTcBlockK / 16; ++k)  // 32 bytes along K per MMA: +2 in the 16-byte address field
                        tc_mma_bf16(d_tmem, adesc + 2 * k, bdesc + 2 * k, IDESC, (kb > kb0 || k > 0) ? 1u : 0u);
                    tc_commit(smem_u32(&empty_bar[stage]));  // stage reusable once these MMAs have read it
                    if (++stage == NS) stage = 0, full_parity ^= 1;
                }
                tc_commit(smem_u32(&acc_full[acc]));
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue warps
        const int q = warp & 3;            // tensor-memory lane quarter this warp may read
        const int row = q * 32 + lane;     // row of the tile held by this thread
        const int et = (warp - 2) * 32 + lane;
        constexpr int HC = NB / 2;         // two warps share a lane quarter: each drains half of the batch columns
        const int b_half = ((warp - 2) >> 2) * HC;
        const int cpc = p.cpc;  // batch columns per CTA of the cluster
        auto cols_of = [&](int r) { return max(0, min(cpc, p.B - r * cpc)); };
        const int b_first = rank * cpc, n_cols = cols_of(rank);
        // the threads that finish a tile: a row (or pair) each, every `groups`-th column
        const int frow = p.pair ? (et & 63) : (et & 127);
        const int cg = p.pair ? (et >> 6) : (et >> 7), groups = p.pair ? 4 : 2;
        if (C > 1) cluster_wait();
        pdl_wait();
        trace_mark(trec, 3);
        const unsigned int push_epoch = (LINK && p.link.world > 0 && p.link.push_inbox >= 0) ? tp_next_epoch(p.link, p.link.push_inbox) : 0u;
        const bool poisoned = LINK && p.link.world > 0 && tp_poisoned(p.status);  // see tp_poisoned: push nothing, advance nothing
        if (p.ssq_in) {
            // The norm factors of this CTA's columns, from the parts that the kernel in front left (fixed order), while
            // the products are being formed.
            const int c = et & (p.cols_pad - 1), j0 = et / p.cols_pad, per_col = 32 * kTcEpiWarps / p.cols_pad;
            float sum = 0.f;
            if (c < n_cols) {
                const float* src = p.ssq_in + b_first + c;
#pragma unroll 4
                for (int j = j0; j < p.ssq_parts; j += per_col) sum += __ldcg(src + (long long)j * kSsqStride);
            }
            norm_sum[c * per_col + j0] = sum;
            named_bar_sync(2, 32 * kTcEpiWarps);
            if (et < n_cols) {
                float tot = 0.f;
                for (int j = 0; j < per_col; ++j) tot += norm_sum[et * per_col + j];
                norm_r[et] = 1.0f / sqrtf(tot * p.inv_dim + p.eps);
            }
            named_bar_sync(2, 32 * kTcEpiWarps);
        }
        for (int i = 0; i < my_tiles; ++i) {
            const int tile = cluster + i * n_clusters;
            const int acc = i & 1;
            const int n = tile * p.units + frow;
            const bool live_row = frow < p.units && n < p.N;
            constexpr int CU = 4;  // columns in flight per thread
            // residual values of the first columns are fetched while the tile is still being multiplied
            float res[CU];
            auto fetch_residual = [&](int col) {
                const bf16* src = p.residual + (long long)(b_first + col) * p.ldres + n;
#pragma unroll
                for (int u = 0; u < CU; ++u) {
                    if (col + u * groups < n_cols) res[u] = __bfloat162float(*src);
                    src += groups * p.ldres;
                }
            };
            if (p.epilogue == EPI_RESIDUAL && live_row) fetch_residual(cg);
            const float next_w = (p.xw_out && live_row) ? __bfloat162float(p.next_norm_w[n]) : 0.f;
            mbar_wait_bounded(smem_u32(&acc_full[acc]), (uint32_t)((i >> 1) & 1), abort_flag, p.status, FAULT_TC_ACC_WAIT);
            if (i == 0) trace_mark(trec, 4);
            tc_fence_after();
            if (i > 0)  // the previous tile's parts have been read, here and by the CTAs they were sent to
                mbar_wait_bounded_cluster(smem_u32(recv_free), (uint32_t)((i - 1) & 1), abort_flag, p.status, FAULT_TC_ACC_WAIT);
            const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * NB + b_half);
            float* dst = mine + (size_t)b_half * RS + row;
            const int b_left = p.B - b_half;
            if constexpr (HC == 8) {
                float v[8];
                tmem_ld8(t_addr, v);
                tmem_ld_wait();
                if (row < RS) {
#pragma unroll
                    for (int e = 0; e < 8; ++e, dst += RS)
                        if (e < b_left) *dst = v[e];
                }
            } else {
#pragma unroll
                for (int c = 0; c < HC; c += 16) {
                    float v[16];
                    tmem_ld16(t_addr + (uint32_t)c, v);
                    tmem_ld_wait();
                    if (row < RS) {
#pragma unroll
                        for (int e = 0; e < 16; ++e, dst += RS)
                            if (c + e < b_left) *dst = v[e];
                    }
                }
            }
            tc_fence_before();
            fence_async_shared();
            named_bar_sync(2, 32 * kTcEpiWarps);
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
            if (C > 1) {
                if (warp == 2) {  // one lane per destination
                    if (lane == 0) mbar_arrive_expect_tx(smem_u32(recv_full), (uint32_t)((C - 1) * n_cols * RS * 4));
                    const uint32_t bytes = lane < C ? (uint32_t)(cols_of(lane) * RS * 4) : 0u;
                    if (lane != rank && bytes && !*abort_flag)
                        bulk_s2cluster(map_to_rank(smem_u32(recv + (size_t)rank * cpc * RS), lane), smem_u32(mine + (size_t)lane * cpc * RS), bytes,
                                       map_to_rank(smem_u32(recv_full), lane));
                    __syncwarp();
                }
                mbar_wait_bounded(smem_u32(recv_full), (uint32_t)(i & 1), abort_flag, p.status, FAULT_TC_ACC_WAIT);
            }
            // The parts of columns col, col + groups, ... of this thread's row, added in rank order
            auto gather = [&](int col, int first_row, float (&v)[CU]) {
#pragma unroll
                for (int u = 0; u < CU; ++u) v[u] = 0.f;
                for (int s = 0; s < C; ++s) {
                    const float* part = (s == rank ? mine : recv) + (size_t)(s * cpc + col) * RS + first_row;
#pragma unroll
                    for (int u = 0; u < CU; ++u)
                        if (col + u * groups < n_cols) v[u] += part[u * groups * RS];
                }
                if (p.ssq_in) {
#pragma unroll
                    for (int u = 0; u < CU; ++u)
                        if (col + u * groups < n_cols) v[u] *= norm_r[col + u * groups];
                }
            };
            if (p.ssq_out) {
                // Residual epilogue in front of a norm: the result, the result with the norm weight, and the sum of
                // squares of the warp's 32 rows of each column.
                const int q32 = (et & 127) >> 5, q32s = (p.units + 31) >> 5;
                if (!*abort_flag && q32 < q32s) {
                    for (int col = cg; col < n_cols; col += CU * groups) {
                        float v[CU];
                        gather(col, min(frow, RS - 1), v);
                        if (col != cg && live_row) fetch_residual(col);
#pragma unroll
                        for (int u = 0; u < CU; ++u) {
                            const int c = col + u * groups;
                            if (c < n_cols) {
                                float x = 0.f;
                                if (live_row) {
                                    const bf16 xb = __float2bfloat16_rn(res[u] + round_bf16(v[u]));
                                    x = __bfloat162float(xb);
                                    const long long o = (long long)(b_first + c) * p.ldout + n;
                                    reinterpret_cast<bf16*>(p.out)[o] = xb;
                                    if (p.xw_out) p.xw_out[(long long)(b_first + c) * p.N + n] = __float2bfloat16_rn(x * next_w);
                                }
                                const float sum = warp_sum(x * x);
                                if (lane == 0) p.ssq_out[(long long)(tile * q32s + q32) * kSsqStride + b_first + c] = sum;
                            }
                        }
                    }
                }
            } else if (!*abort_flag && live_row) {
                float v[CU];
                const long long step = (long long)groups * p.ldout;
                for (int col = cg; col < n_cols; col += CU * groups) {
                    const long long o = (long long)(b_first + col) * p.ldout + n;
                    gather(col, frow, v);
                    if (p.pair) {
                        float up[CU];
                        gather(col, frow + p.half_rows, up);
                        bf16* out = reinterpret_cast<bf16*>(p.out) + o;
#pragma unroll
                        for (int u = 0; u < CU; ++u, out += step)
                            if (col + u * groups < n_cols) *out = __float2bfloat16_rn(round_bf16(silu_f32(round_bf16(v[u]))) * round_bf16(up[u]));
                    } else if (p.epilogue == EPI_RESIDUAL) {
                        if (col != cg) fetch_residual(col);
                        bf16* out = reinterpret_cast<bf16*>(p.out) + o;
#pragma unroll
                        for (int u = 0; u < CU; ++u, out += step)
                            if (col + u * groups < n_cols) *out = __float2bfloat16_rn(res[u] + round_bf16(v[u]));
                    } else if (LINK && p.epilogue == EPI_PUSH_F32) {
#pragma unroll
                        for (int u = 0; u < CU; ++u)
                            if (!poisoned && col + u * groups < n_cols) tp_push(p.link, o + u * step, v[u], push_epoch);
                    } else if (p.epilogue == EPI_STORE_F32) {
                        float* out = reinterpret_cast<float*>(p.out) + o;
#pragma unroll
                        for (int u = 0; u < CU; ++u, out += step)
                            if (col + u * groups < n_cols) *out = v[u];
                    } else {
                        bf16* out = reinterpret_cast<bf16*>(p.out) + o;
#pragma unroll
                        for (int u = 0; u < CU; ++u, out += step)
                            if (col + u * groups < n_cols) *out = __float2bfloat16_rn(v[u]);
                    }
                }
            }
            if (i + 1 < my_tiles) {
                __syncwarp();
                if (lane < C) mbar_arrive_cluster(map_to_rank(smem_u32(recv_free), lane));
            }
        }
        trace_mark(trec, 5);
        if (LINK && p.link.world > 0 && p.link.bump_inbox >= 0 && blockIdx.x == 0 && et == 0 && !*abort_flag && !poisoned) tp_bump(p.link);
    }

    __syncwarp();
    if (C > 1 && warp < 2) cluster_wait();
    if (*abort_flag) __nanosleep(200000);  // copies towards the peers that may still be in flight
    // No CTA of the cluster leaves while another may still write to it or signal it.
    if (C > 1) {
        cluster_arrive();
        cluster_wait();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// 2-D bf16 row-major [rows, cols] with leading dimension ld; box = [64 cols, box_rows], 128-byte swizzle,
// out-of-range elements read as zero.
static bool encode_map(CUtensorMap* map, const bf16* base, long long rows, long long cols, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)kTcBlockK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A descriptor is a pure function of (address, shape, leading dimension, box), and a decode loop asks for the same ones
// over and over: five descriptors of its weights per layer, times the batch sizes that it alternates
// between (the box follows the batch), and the activation buffers of the workspace.  They are encoded once and kept in a
// table that holds the descriptors of a 64-layer model for four batch sizes (0.7 MB; an evicted one is encoded again).
struct MapKey {
    const void* base;
    long long rows, cols, ld;
    int box_rows;
    bool operator==(const MapKey& o) const {
        return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows;
    }
    uint64_t hash() const {
        uint64_t h = hash_mix((uint64_t)(uintptr_t)base, (uint64_t)rows);
        h = hash_mix(h, (uint64_t)cols);
        h = hash_mix(h, (uint64_t)ld);
        return hash_mix(h, (uint64_t)box_rows);
    }
};
static bool make_map(CUtensorMap* map, const bf16* base, long long rows, long long cols, long long ld, int box_rows) {
    using Table = MapTable<MapKey, CUtensorMap, 256>;
    static std::mutex mu;
    static Table* table = new Table;  // never freed: lives as long as the library
    const MapKey key = {base, rows, cols, ld, box_rows};
    std::lock_guard<std::mutex> lock(mu);
    if (const CUtensorMap* known = table->find(key)) {
        *map = *known;
        return true;
    }
    if (!encode_map(map, base, rows, cols, ld, box_rows)) return false;
    table->put(key, *map);
    return true;
}

static int tc_batch_tile(int B) { return B <= 16 ? 16 : (B <= 32 ? 32 : 64); }

bool gemm_tc_supported(int B, int K) { return B >= 2 && B <= 64 && K % 8 == 0 && encode_fn() != nullptr; }

static constexpr size_t kTcHalfSm = 113 * 1024;  // two CTAs of this size share an SM

// Clusters of 1 << log2c CTAs, one CTA per SM, that can be resident together (asked once per device): the clusters of
// eight leave SMs of a GPC over, 15 of them fit at a whole SM per CTA and 16 at half an SM; 33 of four, 74 of two.
template <int NB, bool LINK>
static int tc_resident_clusters(int dev, int log2c, bool half) {
    static std::atomic<int> cache[64][4][2];
    const bool keep = dev >= 0 && dev < 64;
    if (keep)
        if (const int known = cache[dev][log2c][half].load(std::memory_order_relaxed)) return known;
    auto ask = [&](size_t smem) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        cfg.gridDim = dim3(1u << log2c);
        cfg.blockDim = dim3(kTcThreads);
        cfg.dynamicSmemBytes = smem;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1u << log2c, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        return cudaOccupancyMaxActiveClusters(&n, gemm_tc_kernel<NB, LINK>, &cfg) == cudaSuccess ? n : 0;
    };
    int n = ask((size_t)max_smem_optin());
    if (half) {
        const int shared = ask(kTcHalfSm) / 2;
        if (shared > n) n = shared;
    }
    const int most = sm_count() >> log2c;
    if (n > most) n = most;
    if (n < 1) n = log2c == 0 ? 1 : 0;
    if (keep && n > 0) cache[dev][log2c][half].store(n, std::memory_order_relaxed);
    return n;
}

// How N output units and K are dealt out: cluster size, rows of a tile, rounds of tiles per cluster.  Few rows per CTA
// waste time per k-block and read X once per tile; large clusters leave SMs idle and exchange more; a second round adds
// an epilogue where the tile is short.  The estimate below (in ns) weighs these against each other; its constants were
// fitted to a sweep of every projection over all cluster sizes (Qwen3 0.6B / 2B / 8B / 32B, batch 2..64; e.g. 8B at batch
// 32, layer us with clusters of 1 | 2 | 4 | 8: gate/up 174.5 | 168.9 | 171.1 | 185.1, down 191.4 | 175.0 | 171.0 | 172.3;
// 0.6B o_proj 64.9 | 60.5 | 58.6 | 58.4).  A k-block costs 40 ns plus its bytes at a 148th of the HBM rate (never less
// than 150 ns: waiting for a stage and issuing its MMAs, which read 128 rows of A whatever the tile holds).
template <int NB, bool LINK>
static bool tc_plan(TcParams& p, int dev, int& clusters, size_t& smem) {
    double best = 0.;
    for (int log2c = 0; (1 << log2c) <= kTcMaxCluster && (1 << log2c) <= p.kblocks; ++log2c) {
        const int C = 1 << log2c, max_units = p.pair ? kTcRows / 2 : kTcRows;
        const int cpc = (p.B + C - 1) / C, nk = (p.kblocks + C - 1) / C;
        for (int half = 0; half < 2; ++half) {
            const int nc = tc_resident_clusters<NB, LINK>(dev, log2c, half != 0);
            if (nc < 1) continue;
            long long rounds = (p.N + (long long)nc * max_units - 1) / ((long long)nc * max_units);
            int units = (int)((p.N + nc * rounds - 1) / (nc * rounds));
            if (units < 8) units = 8;  // a TMA box no smaller than one swizzle group
            const int half_rows = p.pair ? (units + 7) / 8 * 8 : 0;
            const int a_rows = p.pair ? 2 * half_rows : (units + 7) / 8 * 8;
            const int tiles = (int)((p.N + units - 1) / units);
            const size_t stage = (size_t)(a_rows + NB) * kTcBlockK * 2;
            const size_t tail = kTcTailBytes + (size_t)(C > 1 ? 2 : 1) * cpc * C * a_rows * sizeof(float);
            // the MMA reads 128 rows from the start of every stage, whatever a_rows is
            const size_t a_read = (size_t)kTcRows * kTcBlockK * 2;
            const size_t behind = stage + tail < a_read ? a_read - stage : tail;
            const size_t cap = half ? kTcHalfSm : (size_t)max_smem_optin();
            if (cap < 1024 + behind + 2 * stage) continue;
            long long ns = (long long)((cap - 1024 - behind) / stage);
            if (ns > kTcMaxStages) ns = kTcMaxStages;
            const bool all = ns >= rounds * nk;  // the ring holds everything the CTA reads
            if (all) ns = rounds * nk < 2 ? 2 : rounds * nk;
            if (half && !all) continue;  // a long stream wants the deeper ring
            const double block = 40. + 2.6 * (p.pair ? 2 * units : units) + 0.9 * NB;
            const double tile = nk * (block < 150. ? 150. : block), epi = (C > 1 ? 1100. : 800.) + 60. * cpc;
            // The next tile's MMAs hide this one's epilogue, but an exchange keeps its buffers until every CTA of the cluster
            // has read them: 4 us from the last MMA on, whatever the batch.  Shorter tiles wait for it (N = 151936, K =
            // 1024, batch 16 | 32 | 64: 53 | 57 | 60 us on one CTA per tile, 66 | 72 | 74 on two, 95 | 105 | 122 on four).
            const double hidden = C > 1 && epi < 4000. ? 4000. : epi;
            const double cost = rounds * tile + (rounds - 1) * (hidden > tile ? hidden - tile : 0.) + epi;
            if (best > 0. && cost >= best) continue;
            best = cost;
            p.log2c = log2c, p.cpc = cpc, p.units = units, p.half_rows = half_rows, p.a_rows = a_rows, p.tiles = tiles;
            p.nstages = (int)ns;
            clusters = tiles < nc ? tiles : nc;
            smem = 1024 + (size_t)ns * stage + behind;
        }
    }
    return best > 0.;
}

template <int NB, bool LINK>
static cudaError_t launch_tc_instance(const GemvArgs& a, const bf16* x, long long ldx, TcParams& p, cudaStream_t stream) {
    auto kernel = gemm_tc_kernel<NB, LINK>;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem_optin());
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    int clusters = 0;
    size_t smem = 0;
    if (!tc_plan<NB, LINK>(p, dev, clusters, smem)) return cudaErrorInvalidConfiguration;
    if (a.tiling && a.prologue != PRO_SCALED) a.tiling->units = p.units, a.tiling->tiles = p.tiles;
    p.first = chain_waits_first();
    p.cols_pad = 1;
    while (p.cols_pad < p.cpc) p.cols_pad *= 2;
    alignas(64) CUtensorMap m0, m1, mx;
    if (!make_map(&m0, a.W0, a.N, a.K, a.ldw, p.units)) return cudaErrorInvalidValue;
    if (!make_map(&m1, p.pair ? a.W1 : a.W0, a.N, a.K, a.ldw, p.units)) return cudaErrorInvalidValue;
    if (!make_map(&mx, x, a.B, a.K, ldx, NB)) return cudaErrorInvalidValue;
    return launch_pdl_cluster(kernel, dim3((unsigned)clusters << p.log2c), dim3(kTcThreads), 1 << p.log2c, smem, stream, m0, m1, mx, p);
}

// x must already hold what the MMA consumes; the prologue is none or PRO_SCALED.
cudaError_t launch_gemm_tc(const GemvArgs& a, const bf16* x, long long ldx, cudaStream_t stream) {
    const bool pair = a.epilogue == EPI_SWIGLU;
    TcParams p;
    p.N = a.N, p.K = a.K, p.B = a.B;
    p.kblocks = (a.K + kTcBlockK - 1) / kTcBlockK;
    p.pair = pair ? 1 : 0;
    p.epilogue = a.epilogue;
    p.residual = a.residual, p.ldres = a.ldres;
    p.out = a.out, p.ldout = a.ldout;
    p.status = status_ptr();
    if (!p.status) return cudaErrorUnknown;
    p.trace = trace_handle();
    p.trace_id = a.trace_id;
    p.ssq_in = nullptr, p.ssq_parts = 0, p.inv_dim = 1.0f / (float)a.K, p.eps = a.eps;
    p.ssq_out = nullptr, p.xw_out = nullptr, p.next_norm_w = a.next_norm_w;
    if (a.prologue == PRO_SCALED) p.ssq_in = a.ssq, p.ssq_parts = a.tiling->parts();
    else if (a.ssq && a.epilogue == EPI_RESIDUAL) p.ssq_out = a.ssq, p.xw_out = a.next_norm_w ? a.xw_out : nullptr;
    p.link = a.link;
    if (a.link.world > 0 && (a.link.gather_inbox >= 0 || pair)) return cudaErrorNotSupported;  // only the push side lives here
    const int NB = tc_batch_tile(a.B);
    if (a.link.world > 0 || a.behind_gather) {
        switch (NB) {
            case 16: return launch_tc_instance<16, true>(a, x, ldx, p, stream);
            case 32: return launch_tc_instance<32, true>(a, x, ldx, p, stream);
            default: return launch_tc_instance<64, true>(a, x, ldx, p, stream);
        }
    }
    switch (NB) {
        case 16: return launch_tc_instance<16, false>(a, x, ldx, p, stream);
        case 32: return launch_tc_instance<32, false>(a, x, ldx, p, stream);
        default: return launch_tc_instance<64, false>(a, x, ldx, p, stream);
    }
}

}  // namespace ezb
