// bf16 GEMM with paired CTAs (tcgen05 cta_group::2): a cluster of two CTAs on
// neighbouring SMs computes one output tile of 256 x 256 (or, by the rule at
// ax_gemm_tc2_width, 192 or 128 columns).  Each CTA loads its own 128 rows of A and
// its own half of the columns of B (plain TMA tile loads — nothing is
// multicast; the pair shares B through the MMA unit, which reads both CTAs'
// shared memory), so a k-block costs 32 KB of L2->smem traffic per SM instead of
// the 48 KB of the single-CTA 128 x 256 tile, and half the smem operand reads
// per flop.  CTA 0 of the pair issues the MMAs (M = 256); accumulators live in
// both CTAs' TMEM (128 lanes x the tile's columns, double-buffered); completion is
// signalled to both CTAs with multicast commits; every CTA writes its own 128
// rows of C.
//
// Same operand layouts, epilogue and split-K scheme as the single-CTA kernel.
// All mbarrier waits are bounded.
#include <cuda_bf16.h>
#include <cstdio>
#include <cstdlib>

#include "common.cuh"
#include "gemm_epi.cuh"
#include "kernels.h"
#include "tc_common.cuh"

#define BM2 128            // rows per CTA (256 per pair)
#define BK2 64
#define STAGES2 6
#define STAT_GEMM2 0x400
#define A_BYTES2 (BM2 * BK2 * 2)
#define B_BYTES2 (128 * BK2 * 2)
#define STAGE_BYTES2 (A_BYTES2 + B_BYTES2)
#define STG_BYTES2 (4 * 2 * 4096)      // output staging: per epilogue warp two buffers of 32 rows x 128 B
#define SMEM2 (STAGES2 * STAGE_BYTES2 + STG_BYTES2 + 1024 + 512)

// What the epilogue does.  A kernel per kind: with all of them in one, the registers and the code of the computing ones
// (rotary rows, SwiGLU pairs) cost every plain product some per cent.
enum { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_SWB = 2, EPI_ROPE = 3 };
template <int EPI> struct EpiCfg {
    static constexpr int EW = EPI == EPI_SWB ? 8 : 4;               // epilogue warps
    static constexpr int NH = EW / 4;                               // of them per TMEM lane quarter
    static constexpr int THREADS = 64 + 32 * EW;                    // + TMA warp, MMA warp
};

// Bounded wait of a converged warp, with one answer for all of its lanes: a lane that left alone would be missed by the elect.sync of the others.
// It also ends when another role has given up; that flag is looked at only while the phase is not complete.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, const volatile int* abort_flag) {
    for (uint32_t i = 0; i < TC_SPIN_LIMIT; i++) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        if (__any_sync(0xffffffffu, *abort_flag)) return false;
    }
    return false;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// tile store from this CTA's shared memory (3-D map: column, row, split); bulk-group completion
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, uint32_t src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(m)), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void bulk_commit2() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_le2() { asm volatile("cp.async.bulk.wait_group.read 2;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void bulk_wait_read_le1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ uint32_t pack2_bf16(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
// tile loads by a converged warp (one elected lane issues), their completion counted on an mbarrier that may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_pair_e(uint32_t dst, const CUtensorMap* m, uint32_t bar_cluster, int x, int y) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair_e(uint32_t dst, const CUtensorMap* m, uint32_t bar_cluster, int x, int y, int z) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_e(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_mma_ss2(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// The same two for a converged warp: every lane executes the surrounding code (addresses and descriptor words stay
// warp-uniform and cheap to form), the elected lane issues.  A lone thread in a divergent branch needs about
// 45-50 cycles per MMA issue where this form needs 33 (measured on B200).
__device__ __forceinline__ void tc_mma_ss2_e(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_commit2_e(uint32_t bar, uint16_t mask) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
                 ::"r"(bar), "h"(mask) : "memory");
}
// Grouped launch: several GEMMs of one layer run as one persistent kernel.
//   mode 1: `count` problems share A; problem g has its own B (n[g] columns) and its own C — their column
//           tiles form one tile space (q/k/v or gate/up projections of the same input; their weight gradients).
//           With xkb > 0 every problem has an extra K-segment of its own behind the shared one: C_g = A B_g + A'_g B'_g
//           (xkb k-blocks; a low-rank adapter's contribution inside its projection's launch).
//   mode 2: one output accumulates over `count` (up to 6) K-segments, each with its own A and B (kb[s] k-blocks):
//           dX = dY0 W0^T + dY1 W1^T + ... without round trips of the partial sums through memory; an addend
//           (residual) may be fetched by TMA as in the plain GEMM.
//   mode 3: `count` independent problems of the same depth k, each with its own A, B, C, m[g] and n[g] (weight
//           gradients of different projections of a layer): their tiles form one tile space, so the second
//           problem fills the wave the first one leaves half empty.
//   mode 4: SwiGLU pair — gate and up projections of one input with the activation fused: a 256-wide pair tile holds
//           128 gate columns (B from problem 0, loaded by CTA 0) and the same 128 up columns (problem 1, CTA 1), so an
//           epilogue thread has g and u of its row side by side and writes g, u and h = silu(g) * u (three outputs).
//           With xkb > 0 the two projections have low-rank terms of their own: the segment of the gate's term multiplies
//           zeros in CTA 1 (a box outside the tensor) and the up projection's term zeros in CTA 0, so that one A operand
//           per k-block serves both column halves.
// EPI_SWB (mode 2): the sum over the K-segments is the gradient dh of h = silu(g) * u and never reaches memory; the
//           epilogue fetches g (tmD) and u (tmC2) and writes dg (tmC) and du (tmC1).
// Grouped launches write through TMA stores and do not split K; only mode 2 takes an addend.
// A launch of so few tiles that pairs would be left without one takes a cluster of S pairs to a tile (S 2 or 4): each sums its part of
// the depth, then gives the others, through distributed shared memory, their columns of its accumulator, and finishes its own.  A kernel of
// its own (SHARE): with S as a value in the one kernel, a launch that shares nothing took 0.6 us longer (0.4 with fp32 output), 7.3 us in place of
// 6.6 for 904 x 1704 x 128.
struct GemmGroup {
    int mode, count;
    int whole;               // M- and N-major operands have whole blocks of 64 along M and N: see map_mn
    int band;                // row tiles that are walked together, column by column (see band_of)
    int S;                   // pairs that share a tile's depth (1: a pair has tiles of its own)
    int n[3];
    int kb[6];
    int m[3];
    int xkb, xk_pad;
    // rotary embedding in the epilogue of a mode-1 launch with bf16 output: the outputs g whose bit is set in
    // rope_mask are [rows, heads * 64] projections (row = batch * rope_T + token); every 64-column piece of the
    // epilogue is one head, its columns i and i + 32 form a rotary pair (tables: fp32 [rope_T, 32])
    const float* rope_cos;
    const float* rope_sin;
    int rope_T, rope_mask;
};
static GemmGroup g_rope_req = {};        // rotary request for the next grouped launch (host side, one stream of launches)
void ax_gemm_group_rope(const float* cs, const float* sn, int T, int mask) {
    g_rope_req.rope_cos = cs; g_rope_req.rope_sin = sn; g_rope_req.rope_T = T; g_rope_req.rope_mask = mask;
}

// An N-major B comes in blocks of 64 columns by 64 rows (128-byte swizzle), of 32 (64-byte) where a CTA's columns are no multiple of 64
__host__ __device__ constexpr int b_block(int bn) { return bn / 2 % 64 ? 32 : 64; }

template <int A_MN, int B_MN, typename TO, int EPI, bool SHARE, int BN>
__global__ void __launch_bounds__(EpiCfg<EPI>::THREADS, 1)
k_gemm_tc2(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
           const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmD,
           const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmA2,
           const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmB2,
           const __grid_constant__ CUtensorMap tmC1, const __grid_constant__ CUtensorMap tmC2,
           const __grid_constant__ CUtensorMap tmEA0, const __grid_constant__ CUtensorMap tmEA1,
           const __grid_constant__ CUtensorMap tmEA2, const __grid_constant__ CUtensorMap tmEB0,
           const __grid_constant__ CUtensorMap tmEB1, const __grid_constant__ CUtensorMap tmEB2,
           const GemmGroup grp, int tma_out,
           TO* __restrict__ C, const TO* D, int m, int n, int k, float alpha, float beta, int* status,
           int ksplit, float* __restrict__ ws, long long* prof) {
    // tma_out != 0: the epilogue stages 32 x 128-byte pieces in shared memory (128-byte swizzle) and writes
    // them with TMA tile stores through tmC — {n, m, 1} over C, or {n, m, ksplit} over the fp32 split-K
    // workspace; the hardware clips pieces that overhang the matrix.  Otherwise threads store their rows.
    // tma_out == 2: the addend D is fetched the same way (TMA tile loads through tmD, two pieces ahead, into
    // the staging buffer where the result then replaces it); the operand ring then runs with five stages and
    // the sixth stage's memory doubles the staging area.
    // Epilogue warps: four (a warp per TMEM lane quarter), eight where the epilogue computes so much that four would
    // outlast the main loop of the next tile (SwiGLU backward); the two warps of a quarter then take the column pieces
    // in turn.  Eight for plain products gain 1 % in chains of one round (2000 x 1536 x 1536) and lose as much where rounds follow one another.
    // prof (only in builds with -DAXENG_PROF, otherwise null and every stamp compiles out): clock64 stamps of
    // pair 0's leader CTA — [0] entry, [1] set-up done, [2] predecessor grid finished, [3] first operands landed,
    // [4] last MMA issued, [5] last accumulator complete, [6] last tile stored, [7] exit
#ifdef AXENG_PROF
    const bool timing = prof != nullptr && blockIdx.x == 0;
#else
    constexpr bool timing = false;
#endif
    if (timing && threadIdx.x == 0) prof[0] = clock64();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES2 * STAGE_BYTES2 + STG_BYTES2);
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * STAGES2;
    const uint32_t bar_tfull = bar_empty + 8 * STAGES2, bar_tempty = bar_tfull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES2 + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t smem_base = smem_u32(smem);
    constexpr int NH = EpiCfg<EPI>::NH, EW = EpiCfg<EPI>::EW;
    constexpr bool swiglu = EPI == EPI_SWIGLU, swb = EPI == EPI_SWB;
    constexpr int B_BLK = b_block(BN);                             // columns of a block of an N-major B
    const bool wide_stg = swiglu || swb || tma_out == 2;           // 64 KB of staging instead of 32, five stages
    const int nst = wide_stg ? STAGES2 - 1 : STAGES2;              // operand stages in use
    const bool whole = grp.whole;
    const uint32_t bar_d = smem_u32(bars + 20);                    // [EW warps][16 / EW buffers] arrival barriers of fetched pieces

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Set-up: barriers, tensor memory and tensor maps by three warps at the same time, what each warp has to know about its tiles, and one barrier of the
    // cluster behind it (2560 cycles from the entry before, when one thread did it and two barriers followed; 1850 now: steps of small tiles 0.3 to 2 % shorter).
    static_assert(2 * STAGES2 + 4 == 16, "one barrier to a lane");
    if (warp == 0) {
        mbar_init(smem_u32(bars + (lane < 16 ? lane : lane + 4)), lane == 14 || lane == 15 ? 64 * EW : 1);
        if (lane == 0) *abort_flag = 0;
        mbar_fence_init();
    } else if (warp == 1) {
        tmem_alloc2(smem_u32(tmem_slot), 512);
        tmem_relinquish2();
    } else if (warp == 2 && lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        if (grp.count > 1) { tma_prefetch_desc(grp.mode == 2 ? &tmA1 : &tmC1); tma_prefetch_desc(&tmB1); }
        if (grp.count > 2) { tma_prefetch_desc(grp.mode == 2 ? &tmA2 : &tmC2); tma_prefetch_desc(&tmB2); }
        if (tma_out) tma_prefetch_desc(&tmC);
        if (tma_out == 2 || swb) tma_prefetch_desc(&tmD);
    }
    tc_fence_before();
    __syncwarp();
    const uint32_t crank = cluster_rank(), rank = crank & 1, lead = crank & ~1u;     // rank 0 of a pair leads it (issues the MMAs)
    const int S = SHARE ? grp.S : 1, part = SHARE ? crank >> 1 : 0;      // this pair's part of the depth
    const int pair = SHARE ? blockIdx.x / (2 * S) : blockIdx.x >> 1, npairs = SHARE ? gridDim.x / (2 * S) : gridDim.x >> 1;
    const uint16_t both = 3u << lead;                      // the pair's CTAs
    const int tiles_m = (m + 2 * BM2 - 1) / (2 * BM2);
    int tiles_n = (n + BN - 1) / BN, kblocks_all = (k + BK2 - 1) / BK2;
    const int kb_main = kblocks_all;                       // mode 1: k-blocks of the shared segment
    if (grp.mode == 1) {
        tiles_n = 0;
        for (int q = 0; q < grp.count; q++) tiles_n += (grp.n[q] + BN - 1) / BN;
        kblocks_all += grp.xkb;
    }
    if (grp.mode == 2) { kblocks_all = 0; for (int q = 0; q < grp.count; q++) kblocks_all += grp.kb[q]; }
    if (swiglu) { tiles_n = (n + 127) / 128; kblocks_all += 2 * grp.xkb; }
    int num_tiles = tiles_m * tiles_n;
    if (grp.mode == 3) {
        num_tiles = 0;
        for (int q = 0; q < grp.count; q++) num_tiles += ((grp.m[q] + 2 * BM2 - 1) / (2 * BM2)) * ((grp.n[q] + BN - 1) / BN);
    }
    // tile index -> problem g, row tile tm and column tile tl inside it (row tiles of a band fastest, bands slowest)
    auto locate = [&](int tile, int& tm, int& tl) -> int {
        int q = 0;
        if (grp.mode == 3) {
            int tmq = (grp.m[0] + 2 * BM2 - 1) / (2 * BM2);
            for (; q + 1 < grp.count; q++) {
                const int tq = tmq * ((grp.n[q] + BN - 1) / BN);
                if (tile < tq) break;
                tile -= tq;
                tmq = (grp.m[q + 1] + 2 * BM2 - 1) / (2 * BM2);
            }
            tm = tile % tmq; tl = tile / tmq;
            return q;
        }
        int b0 = 0, rows = tiles_m;
        if (grp.band < tiles_m) {
            b0 = tile / (grp.band * tiles_n) * grp.band;
            tile -= b0 * tiles_n;
            rows = min(grp.band, tiles_m - b0);
        }
        int tn = tile / rows;
        tm = b0 + tile - tn * rows;
        if (grp.mode == 1)
            for (; q + 1 < grp.count; q++) { const int tq = (grp.n[q] + BN - 1) / BN; if (tn < tq) break; tn -= tq; }
        tl = tn;
        return q;
    };
    const int kb_per = ksplit == 1 ? kblocks_all : (kblocks_all + ksplit - 1) / ksplit;
    const int kb_from = SHARE ? kblocks_all * part / S : 0, kb_to = SHARE ? kblocks_all * (part + 1) / S : kblocks_all;
    const int num_units = num_tiles * ksplit;

    // the CTA's own warps and the peer's: barriers are initialised and tensor memory is there
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t full_leader = map_to_cta(bar_full, lead);  // cluster address of the leader's full[0]
    const uint32_t tempty_leader = map_to_cta(bar_tempty, lead);
    // programmatic dependent launch: see the single-CTA kernel
    if (timing && threadIdx.x == 0) prof[1] = clock64();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (timing && threadIdx.x == 0) prof[2] = clock64();

    if (warp == 0) {
        // ── TMA producer (both CTAs): own 128 rows of A, own half of the tile's columns of B.  The whole warp runs the loop, one elected lane issues ──
        // This loop was the bound: as one thread of a divergent warp that chose its maps anew for each k-block it took 418 cycles and 61 for each
        // TMA instruction, 540 / 607 / 663 a k-block of 256 x 256 x 64 with both operands K-major / one / none (one pair alone, K 8192), where
        // the MMAs need 512.  Converged, with the choice made once for a run of k-blocks and one instruction for each operand, all three take 512 (that
        // is the tensor core's time).  8 launches in a row: 4096 x 1536 x 8192 (A^T B) 839 -> 746 us, 2000 x 1536 x 4096 (A B) 218 -> 201,
        // 2000 x 4096 x 1536 (A B^T) 178 -> 176.
        uint32_t it = 0, ph = 0;
        int s = 0;
        bool ok = true;
        for (int unit = pair; unit < num_units && ok; unit += npairs) {
            const int split = ksplit == 1 ? 0 : unit / num_tiles, tile = unit - split * num_tiles;
            const int kb0 = kb_from + split * kb_per, kb1 = min(kb_to, kb0 + kb_per);
            int tm, tl;
            const int g = locate(tile, tm, tl);
            const int row0 = tm * 2 * BM2 + rank * BM2, col0 = swiglu ? tl * 128 : tl * BN + rank * (BN / 2);
            // A run: k-blocks whose operands lie one behind the other in the same two tensors.  Modes 1 and 3 pick B by problem (mode 3 also A), mode 4
            // gives CTA 0 the gate weights and CTA 1 the up weights (same 128 columns).
            const CUtensorMap* pA = grp.mode == 3 ? (g == 0 ? &tmA : (g == 1 ? &tmA1 : &tmA2)) : &tmA;
            const CUtensorMap* pB = (grp.mode == 1 || grp.mode == 3) ? (g == 0 ? &tmB : (g == 1 ? &tmB1 : &tmB2))
                                    : (swiglu && rank == 1 ? &tmB1 : &tmB);
            int seg = 0, kl = kb0;                       // segment and k-block inside it
            for (int kb = kb0; kb < kb1 && ok;) {
                int run = kb1 - kb, yb = 0, ys = BK2;    // length; row of B when its rows run along K, and its step
                if (grp.mode == 2) {
                    while (seg + 1 < grp.count && kl >= grp.kb[seg]) kl -= grp.kb[seg++];
                    run = min(run, grp.kb[seg] - kl);
                    pA = seg == 0 ? &tmA : seg == 1 ? &tmA1 : seg == 2 ? &tmA2 : seg == 3 ? &tmEA0 : seg == 4 ? &tmEA1 : &tmEA2;
                    pB = seg == 0 ? &tmB : seg == 1 ? &tmB1 : seg == 2 ? &tmB2 : seg == 3 ? &tmEB0 : seg == 4 ? &tmEB1 : &tmEB2;
                } else if (kb < kb_main) {
                    run = min(run, kb_main - kb);
                } else if (grp.mode == 1) {              // the problem's own extra segment
                    kl = kb - kb_main;
                    pA = g == 0 ? &tmEA0 : (g == 1 ? &tmEA1 : &tmEA2);
                    pB = g == 0 ? &tmEB0 : (g == 1 ? &tmEB1 : &tmEB2);
                } else if (swiglu) {                     // gate term, then up term; the other CTA reads zeros
                    const int e = kb - kb_main >= grp.xkb;
                    kl = kb - kb_main - e * grp.xkb;
                    run = min(run, grp.xkb - kl);
                    pA = e ? &tmEA1 : &tmEA0;
                    pB = e ? &tmEB1 : &tmEB0;
                    if ((int)rank != e) { yb = grp.xk_pad; ys = 0; }
                }
                int x = kl * BK2;
                if (ys) yb = x;
                kb += run; kl += run;
                for (; run > 0; run--, it++, s = (s + 1 == nst ? 0 : s + 1), ph ^= (s == 0), x += BK2, yb += ys) {
                    if (it >= (uint32_t)nst && !mbar_wait_warp(bar_empty + 8 * s, ph ^ 1, abort_flag)) { ok = false; break; }
                    const uint32_t sa = smem_base + s * STAGE_BYTES2, sb = sa + A_BYTES2;
                    const uint32_t fb = full_leader + 8 * s;
                    if (rank == 0) mbar_expect_tx_e(bar_full + 8 * s, 2 * (A_BYTES2 + BN * BK2));   // both CTAs' bytes land on this barrier
                    if (A_MN) {
                        if (whole) tma_load_3d_pair_e(sa, pA, fb, 0, x, row0 >> 6);
                        else { tma_load_2d_pair_e(sa, pA, fb, row0, x); tma_load_2d_pair_e(sa + 8192, pA, fb, row0 + 64, x); }
                    } else {
                        tma_load_2d_pair_e(sa, pA, fb, x, row0);
                    }
                    if (B_MN) {
                        if (B_BLK == BN / 2) tma_load_2d_pair_e(sb, pB, fb, col0, yb);
                        else if (whole) tma_load_3d_pair_e(sb, pB, fb, 0, yb, col0 / B_BLK);
                        else {
#pragma unroll
                            for (int z = 0; z < BN / 2; z += B_BLK) tma_load_2d_pair_e(sb + z * BK2 * 2, pB, fb, col0 + z, yb);
                        }
                    } else {
                        tma_load_2d_pair_e(sb, pB, fb, x, col0);
                    }
                }
            }
        }
        __syncwarp();
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, STAT_GEMM2 | 1); }
    } else if (warp == 1 && rank == 0) {
        // ── MMA issuer (leader CTA only): the whole warp runs the loop converged, one elected lane issues ──
        constexpr uint32_t idesc = tc_idesc_bf16(256, BN, A_MN, B_MN);
        // descriptor words: the upper one is a constant (SBO 1024, 128-byte swizzle; 512 and 64 for blocks of 32 columns), the lower one is
        // (address >> 4) | (LBO >> 4) << 16; a k-step of 16 advances it by 2048 B (MN-major; 1024) or 32 B (K-major)
        constexpr bool b64 = B_MN && B_BLK == 32;
        constexpr uint32_t dhi = (1024u >> 4) | (1u << 14) | (2u << 29), dhi_b = b64 ? (512u >> 4) | (1u << 14) | (4u << 29) : dhi;
        constexpr uint32_t a_step = A_MN ? 128 : 2, b_step = B_MN ? (b64 ? 64 : 128) : 2;
        constexpr uint32_t a_lbo = (A_MN ? 8192u : 16u) >> 4, b_lbo = (B_MN ? B_BLK * BK2 * 2u : 16u) >> 4;
        uint32_t it = 0, tcount = 0, ph = 0;
        int s = 0;
        bool ok = true;
        for (int unit = pair; unit < num_units && ok; unit += npairs, tcount++) {
            const int split = ksplit == 1 ? 0 : unit / num_tiles;
            const int kb0 = kb_from + split * kb_per, kb1 = min(kb_to, kb0 + kb_per);
            const int acc = tcount & 1;
            const uint32_t aph = (tcount >> 1) & 1;
            if (tcount >= 2 && !mbar_wait_warp(bar_tempty + 8 * acc, aph ^ 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + acc * 256;
            for (int kb = kb0; kb < kb1; kb++, it++, s = (s + 1 == nst ? 0 : s + 1), ph ^= (s == 0)) {
                if (!mbar_wait_warp(bar_full + 8 * s, ph, abort_flag)) { ok = false; break; }
                tc_fence_after();
                if (timing && it == 0 && lane == 0) prof[3] = clock64();
                const uint32_t sa = smem_base + s * STAGE_BYTES2, sb = sa + A_BYTES2;
                const uint32_t a_lo = ((sa & 0x3FFFF) >> 4) | (a_lbo << 16), b_lo = ((sb & 0x3FFFF) >> 4) | (b_lbo << 16);
#pragma unroll
                for (int kk = 0; kk < BK2 / 16; kk++)
                    tc_mma_ss2_e(d_tmem, ((uint64_t)dhi << 32) | (a_lo + kk * a_step), ((uint64_t)dhi_b << 32) | (b_lo + kk * b_step),
                                 idesc, (kb != kb0) || (kk != 0));
                tc_commit2_e(bar_empty + 8 * s, both);       // frees the stage in both CTAs
            }
            if (ok) tc_commit2_e(bar_tfull + 8 * acc, both); // accumulator ready in both CTAs
            if (timing && lane == 0) prof[4] = clock64();
        }
        __syncwarp();
        if (lane != 0) ok = true;                      // one report is enough
        if (!ok) { *abort_flag = 1; atomicExch(status, STAT_GEMM2 | 2); }
    } else if (warp >= 2) {
        // ── epilogue (both CTAs): own 128 rows x 256 columns; of eight warps w and w + 4 share a lane quarter ──
        const int quad = warp & 3, ew = warp - 2, half = ew >> 2;
        uint32_t tcount = 0, pieces = 0;
        bool ok = true;
        const bool vec_ok = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (n % (16 / (int)sizeof(TO))) == 0 &&
                            (!D || (reinterpret_cast<uintptr_t>(D) & 15) == 0);
        const bool f32_out = ksplit > 1 || sizeof(TO) == 4;
        const float a_eff = ksplit > 1 ? 1.f : alpha;
        // staging of a warp: two 4 KB buffers behind the operand ring; with a stage less, whose memory adjoins, there is
        // twice the memory (four buffers of four warps, two of eight)
        const uint32_t nbuf = wide_stg ? 16 / EW : 2;
        const uint32_t stg_off = (wide_stg ? STAGES2 - 1 : STAGES2) * STAGE_BYTES2 + (EW == 4 ? quad : ew) * nbuf * 4096;
        uint8_t* stg = smem + stg_off;
        const uint32_t stg_u32 = smem_base + stg_off;
        const uint32_t my_bar_d = bar_d + 8 * (16 / EW) * (EW == 4 ? quad : ew);
        uint32_t dpar = 0;                                      // phase parity of each arrival barrier
        for (int unit = pair; unit < num_units && ok; unit += npairs, tcount++) {
            const int split = ksplit == 1 ? 0 : unit / num_tiles, tile = unit - split * num_tiles;
            int tm, tl;
            const int g = locate(tile, tm, tl);                  // grouped launch: which output, which tile of it
            const int tn = tl;
            const int acc = tcount & 1;
            const uint32_t aph = (tcount >> 1) & 1;
            const int row0 = tm * 2 * BM2 + rank * BM2 + quad * 32;
            const int row = row0 + lane;
            const int cw = f32_out ? 32 : 64;                   // columns per 128-byte piece
            const CUtensorMap* pC = g == 0 ? &tmC : (g == 1 ? &tmC1 : &tmC2);
            const int ncols = min(BN, ((grp.mode == 1 || grp.mode == 3) ? grp.n[g] : n) - tl * BN);
            const int m_g = grp.mode == 3 ? grp.m[g] : m;
            // pieces of this tile that this warp writes: half, half + NH, ...
            const int pw = swb ? 32 : cw;
            const int npt = (tma_out && !swiglu && row0 < m_g) ? (ncols + pw - 1) / pw : 0;
            const int j0 = SHARE ? part * (BN / cw / S) : 0;   // a shared tile: this part's 256 / S columns
            const int npc = SHARE ? max(0, min(npt - j0, BN / cw / S)) : (npt - half + NH - 1) / NH;
            const uint32_t pbase = pieces;
            const bool do_rope = EPI == EPI_ROPE && ((grp.rope_mask >> g) & 1);
            const int rope_t = do_rope ? (row < m_g ? row : 0) % grp.rope_T : 0;
            // lane 0: piece i of this warp of the addend, or of g and u, -> its buffer
            auto fetch_d = [&](int i) {
                const uint32_t bi = (pbase + i) & (nbuf - 1);
                const int x = tn * BN + (j0 + half + NH * i) * pw;
                mbar_expect_tx(my_bar_d + 8 * bi, 4096);
                tma_load_3d(stg_u32 + bi * 4096, &tmD, my_bar_d + 8 * bi, x, row0, 0);
                if (swb) tma_load_3d(stg_u32 + bi * 4096 + 2048, &tmC2, my_bar_d + 8 * bi, x, row0, 0);
            };
            if ((tma_out == 2 || swb) && lane == 0 && npc > 0) {         // the first two travel during the main loop
                if (swb) bulk_wait_read_all(); else bulk_wait_read_le2();
                fetch_d(0);
                if (npc > 1) fetch_d(1);
            }
            // rotary: the row's cos / sin values are the same for every head, so they are read once per tile, while the main
            // loop runs, and stay in registers
            float4 rc[8], rs[8];
            if (do_rope) {
                const float4* cr = reinterpret_cast<const float4*>(grp.rope_cos + (long long)rope_t * 32);
                const float4* sr = reinterpret_cast<const float4*>(grp.rope_sin + (long long)rope_t * 32);
#pragma unroll
                for (int q = 0; q < 8; q++) { rc[q] = __ldg(cr + q); rs[q] = __ldg(sr + q); }
            }
            if (!mbar_wait(bar_tfull + 8 * acc, aph) || *abort_flag) ok = false;
            tc_fence_after();
            if (timing && threadIdx.x == 64) prof[5] = clock64();
            const uint32_t taddr = tmem_base + acc * 256 + ((uint32_t)(quad * 32) << 16);
            const int own = 8 / S;                              // 32-column chunks of a part
            // sums of the other parts in this CTA's operand ring: [part][lane quarter][chunk][4 columns][row], 512 bytes in a row per warp
            auto part_at = [&](int from, int c) { return ((from - (from > part)) * 4 + quad) * own * 4096 + c * 4096 + lane * 16; };
            if (SHARE) {                                        // one tile per cluster: every warp comes by here once
                ok = __all_sync(0xffffffffu, ok);               // lanes may have seen the wait or the flag differently: TMEM is read by whole warps
                cluster_sync();                                 // no ring has a reader or a writer left
                if (ok)
                    for (int q = 1; q < S; q++) {
                        const int to = (part + q) & (S - 1);
                        const uint32_t dst = map_to_cta(smem_base + ((part - (part > to)) * 4 + quad) * own * 4096 + lane * 16, to * 2 + rank);
#pragma unroll 1
                        for (int c = 0; c < own; c++) {
                            uint32_t r[32];
                            tmem_ld32(taddr + (to * own + c) * 32, r);
                            tmem_ld_wait();
#pragma unroll
                            for (int z = 0; z < 8; z++)
                                asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + c * 4096 + z * 512), "r"(r[z * 4]), "r"(r[z * 4 + 1]),
                                             "r"(r[z * 4 + 2]), "r"(r[z * 4 + 3]) : "memory");
                        }
                    }
                cluster_sync();
            }
            if (!ok) break;
            auto part_add = [&](int c, uint32_t* r) {            // chunk c of this part, the parts in order behind the own sum
                if (!SHARE) return;
                for (int from = 0; from < S; from++) {
                    if (from == part) continue;
#pragma unroll
                    for (int z = 0; z < 8; z++) {
                        const float4 v = *reinterpret_cast<const float4*>(smem + part_at(from, c) + z * 512);
                        r[z * 4] = __float_as_uint(__uint_as_float(r[z * 4]) + v.x);
                        r[z * 4 + 1] = __float_as_uint(__uint_as_float(r[z * 4 + 1]) + v.y);
                        r[z * 4 + 2] = __float_as_uint(__uint_as_float(r[z * 4 + 2]) + v.z);
                        r[z * 4 + 3] = __float_as_uint(__uint_as_float(r[z * 4 + 3]) + v.w);
                    }
                }
            };
            if constexpr (swiglu) {
                // accumulator columns 0..127: gate, 128..255: up (same output columns tl*128 ..); per 64-column piece
                // three staged outputs g, u, h, each stored by its own bulk group so that the buffers rotate freely.
                // div_1p_exp: an IEEE division's slow-path branch serialised the 128 pairs of a thread (8192 x 1536 x 2 * 4096: 189 us
                // against 160 with an approximate quotient; its residual step costs 0.4 % more, 166.8 -> 167.5 us on another
                // box); eight warps instead of four gain nothing here (168 us against 160)
                const int vcols = min(128, n - tl * 128);
                const int np2 = row0 < m ? (vcols + 63) / 64 : 0;
#pragma unroll 1
                for (int j = 0; j < np2; j++) {
                    if (lane == 0) bulk_wait_read_le1();        // only the latest store may still be reading its buffer
                    __syncwarp();
                    uint8_t* bg = stg + ((pieces) & 3) * 4096 + lane * 128;
                    uint8_t* bu = stg + ((pieces + 1) & 3) * 4096 + lane * 128;
                    uint8_t* bh = stg + ((pieces + 2) & 3) * 4096 + lane * 128;
#pragma unroll 1
                    for (int half = 0; half < 2; half++) {
                        uint32_t rg[32], ru[32];
                        tmem_ld32(taddr + j * 64 + half * 32, rg);
                        tmem_ld32(taddr + 128 + j * 64 + half * 32, ru);
                        tmem_ld_wait();
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            float g8[8], u8[8], h8[8];
#pragma unroll
                            for (int e2 = 0; e2 < 8; e2++) {
                                g8[e2] = alpha * __uint_as_float(rg[q * 8 + e2]);
                                u8[e2] = alpha * __uint_as_float(ru[q * 8 + e2]);
                                h8[e2] = div_1p_exp(g8[e2], g8[e2]) * u8[e2];
                            }
                            const int sw = ((half * 4 + q) ^ (lane & 7)) << 4;
                            uint4 pk;
                            pk.x = pack2_bf16(g8[0], g8[1]); pk.y = pack2_bf16(g8[2], g8[3]); pk.z = pack2_bf16(g8[4], g8[5]); pk.w = pack2_bf16(g8[6], g8[7]);
                            *reinterpret_cast<uint4*>(bg + sw) = pk;
                            pk.x = pack2_bf16(u8[0], u8[1]); pk.y = pack2_bf16(u8[2], u8[3]); pk.z = pack2_bf16(u8[4], u8[5]); pk.w = pack2_bf16(u8[6], u8[7]);
                            *reinterpret_cast<uint4*>(bu + sw) = pk;
                            pk.x = pack2_bf16(h8[0], h8[1]); pk.y = pack2_bf16(h8[2], h8[3]); pk.z = pack2_bf16(h8[4], h8[5]); pk.w = pack2_bf16(h8[6], h8[7]);
                            *reinterpret_cast<uint4*>(bh + sw) = pk;
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        const int cx = tl * 128 + j * 64;
                        tma_store_3d(&tmC, stg_u32 + ((pieces) & 3) * 4096, cx, row0, 0); bulk_commit2();
                        tma_store_3d(&tmC1, stg_u32 + ((pieces + 1) & 3) * 4096, cx, row0, 0); bulk_commit2();
                        tma_store_3d(&tmC2, stg_u32 + ((pieces + 2) & 3) * 4096, cx, row0, 0); bulk_commit2();
                    }
                    pieces += 3;
                }
            } else if constexpr (swb) {
                // Bound: 268 MB of g, u, dg, du beside 103 GF at 8192 x 4096 x 1536 — 101 us in one launch against 141 us for the
                // product and the separate pass over memory; with four warps 120 us (div_1p_exp's residual step: 103.7 -> 106.1 us on another box).
                // dh stays in fp32 registers: dg = dh * u * s * (1 + g * (1 - s)), du = dh * g * s with s = sigmoid(g), written over
                // the fetched g and u; pieces of 32 columns (64-byte rows and swizzle), two in flight
#pragma unroll 1
                for (int i = 0; i < npc; i++) {
                    const uint32_t bi = (pbase + i) & (nbuf - 1);
                    uint8_t* buf = stg + bi * 4096 + lane * 64;
                    const int x = tn * BN + (half + NH * i) * 32;
                    uint32_t r[32];
                    tmem_ld32(taddr + (half + NH * i) * 32, r);
                    if (!mbar_wait(my_bar_d + 8 * bi, (dpar >> bi) & 1)) { ok = false; break; }
                    dpar ^= 1u << bi;
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        uint4* sg = reinterpret_cast<uint4*>(buf + ((q ^ ((lane >> 1) & 3)) << 4));
                        uint4* su = sg + 128;                       // 2 KB further: u
                        const uint4 gv = *sg, uv = *su;
                        const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
                        uint32_t og[4], ou[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            float dgv[2], duv[2];
#pragma unroll
                            for (int o = 0; o < 2; o++) {
                                const float g1 = __uint_as_float(o ? gw[e] & 0xffff0000u : gw[e] << 16);
                                const float u1 = __uint_as_float(o ? uw[e] & 0xffff0000u : uw[e] << 16);
                                const float dh = alpha * __uint_as_float(r[q * 8 + e * 2 + o]);
                                const float sig = div_1p_exp(1.f, g1);
                                dgv[o] = dh * u1 * (sig * (1.f + g1 * (1.f - sig)));
                                duv[o] = dh * (g1 * sig);
                            }
                            og[e] = pack2_bf16(dgv[0], dgv[1]); ou[e] = pack2_bf16(duv[0], duv[1]);
                        }
                        *sg = make_uint4(og[0], og[1], og[2], og[3]);
                        *su = make_uint4(ou[0], ou[1], ou[2], ou[3]);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_3d(&tmC, stg_u32 + bi * 4096, x, row0, 0);
                        tma_store_3d(&tmC1, stg_u32 + bi * 4096 + 2048, x, row0, 0);
                        bulk_commit2();
                        if (i + 2 < npc) { bulk_wait_read_all(); fetch_d(i + 2); }
                    }
                    pieces++;
                }
                if (!ok) break;
            } else if (tma_out) {
#pragma unroll 1
                for (int j = 0; j < npc && ok; j++) {
                    const int c = (j0 + j) * cw, cp = j * (cw / 32);     // first column; first chunk of the part
                    const uint32_t bi = pieces & (nbuf - 1);
                    uint8_t* buf = stg + bi * 4096 + lane * 128;
                    if (lane == 0) bulk_wait_read_le1();        // all but the latest store have read their buffers
                    if (tma_out == 2) {
                        if (lane == 0 && j + 2 < npc) fetch_d(j + 2);
                        if (!mbar_wait(my_bar_d + 8 * bi, (dpar >> bi) & 1)) { ok = false; break; }
                        dpar ^= 1u << bi;
                    }
                    __syncwarp();
                    uint32_t r[32];
                    tmem_ld32(taddr + c, r);
                    tmem_ld_wait();
                    part_add(cp, r);
                    if (f32_out) {
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            float4* slot = reinterpret_cast<float4*>(buf + ((q ^ (lane & 7)) << 4));
                            float4 f = make_float4(a_eff * __uint_as_float(r[q * 4]), a_eff * __uint_as_float(r[q * 4 + 1]),
                                                   a_eff * __uint_as_float(r[q * 4 + 2]), a_eff * __uint_as_float(r[q * 4 + 3]));
                            if (tma_out == 2) {
                                const float4 d = *slot;
                                f.x += beta * d.x; f.y += beta * d.y; f.z += beta * d.z; f.w += beta * d.w;
                            }
                            *slot = f;
                        }
                    } else if (do_rope) {
                        // the piece is one head: rotate the pairs (i, i + 32) in fp32, round once
                        uint32_t r2[32];
                        tmem_ld32(taddr + c + 32, r2);
                        tmem_ld_wait();
                        part_add(cp + 1, r2);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const float4 c0 = rc[2 * q], c1 = rc[2 * q + 1], s0 = rs[2 * q], s1 = rs[2 * q + 1];
                            const float cc[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
                            const float ss[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
                            float o1[8], o2[8];
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const float x1 = a_eff * __uint_as_float(r[q * 8 + e]), x2 = a_eff * __uint_as_float(r2[q * 8 + e]);
                                o1[e] = x1 * cc[e] - x2 * ss[e];
                                o2[e] = x1 * ss[e] + x2 * cc[e];
                            }
                            uint4 pk;
                            pk.x = pack2_bf16(o1[0], o1[1]); pk.y = pack2_bf16(o1[2], o1[3]); pk.z = pack2_bf16(o1[4], o1[5]); pk.w = pack2_bf16(o1[6], o1[7]);
                            *reinterpret_cast<uint4*>(buf + ((q ^ (lane & 7)) << 4)) = pk;
                            pk.x = pack2_bf16(o2[0], o2[1]); pk.y = pack2_bf16(o2[2], o2[3]); pk.z = pack2_bf16(o2[4], o2[5]); pk.w = pack2_bf16(o2[6], o2[7]);
                            *reinterpret_cast<uint4*>(buf + (((4 + q) ^ (lane & 7)) << 4)) = pk;
                        }
                    } else {
#pragma unroll
                        for (int half = 0; half < 2; half++) {
                            if (half) { tmem_ld32(taddr + c + 32, r); tmem_ld_wait(); part_add(cp + 1, r); }
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                uint4* slot = reinterpret_cast<uint4*>(buf + (((half * 4 + q) ^ (lane & 7)) << 4));
                                float f[8];
#pragma unroll
                                for (int e = 0; e < 8; e++) f[e] = a_eff * __uint_as_float(r[q * 8 + e]);
                                if (tma_out == 2) {
                                    const uint4 d = *slot;
                                    const uint32_t dw[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                                    for (int e = 0; e < 4; e++) {
                                        f[2 * e] += beta * __uint_as_float(dw[e] << 16);
                                        f[2 * e + 1] += beta * __uint_as_float(dw[e] & 0xffff0000u);
                                    }
                                }
                                uint4 pk;
                                pk.x = pack2_bf16(f[0], f[1]); pk.y = pack2_bf16(f[2], f[3]);
                                pk.z = pack2_bf16(f[4], f[5]); pk.w = pack2_bf16(f[6], f[7]);
                                *slot = pk;
                            }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_3d(pC, stg_u32 + bi * 4096, tl * BN + c, row0, ksplit > 1 ? split : 0);
                        bulk_commit2();
                    }
                    pieces++;
                }
                if (!ok) break;
            } else {
                TO* crow = C + (long long)row * n;
                const TO* drow = (D && beta != 0.f) ? D + (long long)row * n : nullptr;
                float* wrow = ws + ((long long)split * m + row) * n;
#pragma unroll 1
                for (int c = half * (BN / NH); c < (half + 1) * (BN / NH); c += 32) {
                    uint32_t r[32];
                    tmem_ld32(taddr + c, r);
                    tmem_ld_wait();
                    const int col0 = tn * BN + c;
                    if (row < m && col0 < n) {
                        if (ksplit > 1) epi_store<float>(wrow, nullptr, r, col0, n - col0, 1.f, 0.f, (n & 3) == 0);
                        else epi_store<TO>(crow, drow, r, col0, n - col0, alpha, beta, vec_ok);
                    }
                }
            }
            tc_fence_before();
            mbar_arrive_cluster(tempty_leader + 8 * acc);   // every epilogue thread of both CTAs frees the accumulator
            if (timing && threadIdx.x == 64) prof[6] = clock64();
        }
        if (tma_out && lane == 0) bulk_wait_read_all();       // staging stays valid until the last store has read it
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, STAT_GEMM2 | 3); }
    }
    if (SHARE && warp < 2) { cluster_sync(); cluster_sync(); }      // the two of the epilogue
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                        // nobody frees TMEM while the peer may still use the pair
    if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc2(tmem_base, 512); }
    if (timing && threadIdx.x == 0) prof[7] = clock64();
}

// ── host ────────────────────────────────────────────────────────────────────
extern float* ax_splitk_ws(size_t* bytes);
extern int ax_gemm_pdl(void);
extern int ax_gemm_mode(void);
extern int ax_gemm_tma_out(void);
extern bool ax_gemm_on_side(void);
extern bool ax_gemm_beside(void);
template <typename TO>
void ax_splitk_reduce_launch(const float* ws, int ksplit, TO* C, const TO* D, long long mn, float alpha, float beta, cudaStream_t st);

// co-resident clusters of S pairs of this kernel (0: none)
template <int A_MN, int B_MN, typename TO, int EPI = EPI_PLAIN, int S = 1, int BN = 256>
static int clusters_for() {
    static int g_max = -1;
    if (g_max < 0) {
        cudaFuncSetAttribute(k_gemm_tc2<A_MN, B_MN, TO, EPI, (S > 1), BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM2);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(AX_SMS / (2 * S) * 2 * S, 1, 1);
        cfg.blockDim = dim3(EpiCfg<EPI>::THREADS, 1, 1);
        cfg.dynamicSmemBytes = SMEM2;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 2 * S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, k_gemm_tc2<A_MN, B_MN, TO, EPI, (S > 1), BN>, &cfg) != cudaSuccess || nc < 1) { cudaGetLastError(); nc = 0; }
        g_max = nc;
    }
    return g_max;
}
static int g_share_max[2] = {0, 0};      // the least of that over the kernels that share a tile, for 2 and 4 pairs

// operand / output tensor maps of one problem.  An M- or N-major operand [k, e] is loaded as blocks of `blk` (64; 32: see b_block) elements by 64 rows, all of
// a CTA's `ext` elements with one instruction where its rows are whole blocks: as {blk, k, e / blk}.  (A block that reached past the end of a row
// would read the next one.)
static int map_mn(CUtensorMap* t, const void* p, int e, int k, bool whole, int ext, int blk) {
    uint64_t dims[3] = {(uint64_t)blk, (uint64_t)k, (uint64_t)e / blk}, strides[2] = {(uint64_t)e * 2, (uint64_t)blk * 2};
    uint32_t box[3] = {(uint32_t)blk, BK2, (uint32_t)(ext / blk)};
    whole = whole && ext > blk;
    if (!whole) dims[0] = e;
    return tc_make_tmap_bf16(t, p, whole ? 3 : 2, dims, strides, box, blk == 64 ? 128 : 64);
}
static int map_km(CUtensorMap* t, const void* p, int e, int k, int ext) {
    uint64_t dims[2] = {(uint64_t)k, (uint64_t)e}, strides[1] = {(uint64_t)k * 2};
    uint32_t box[2] = {BK2, (uint32_t)ext};
    return tc_make_tmap_bf16(t, p, 2, dims, strides, box, 128);
}
// {n, m, nz} tensor of osz-byte elements, pieces of 128 bytes (half_row: 64) x 32 rows
static int map_c(CUtensorMap* t, void* base, int m, int n, int nz, int osz, bool half_row = false) {
    PFN_tmapEncodeTiled enc = tc_encode_fn();
    if (!enc) return 2;
    cuuint64_t gd[3] = {(cuuint64_t)n, (cuuint64_t)m, (cuuint64_t)nz};
    cuuint64_t gs[2] = {(cuuint64_t)n * osz, (cuuint64_t)m * n * osz};
    cuuint32_t bx[3] = {(cuuint32_t)((half_row ? 64 : 128) / osz), 32, 1};
    cuuint32_t es[3] = {1, 1, 1};
    if (gs[1] % 16 != 0) gs[1] = (gs[1] + 15) / 16 * 16;     // only reached with nz == 1 (never indexed)
    const CUtensorMapDataType dtp = osz == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    return enc(t, dtp, 3, base, gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, half_row ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : 2;
}

// Pairs to a tile (GemmGroup::S) for a launch of `tiles` tiles of kb k-blocks (0.3 us each); *cost: the launch in k-blocks.  33 clusters of
// two pairs and 15 of four fit the GPU; two cluster barriers and the exchange of 64 or 96 KB per CTA cost what 8 and 12 k-blocks do.
// us with 1 / 2 / 4 pairs, tiles x k-blocks: 24 x 88 37.6 / 25.9, 24 x 44 with addend 21.8 / 17.4, 24 x 32 18.3 / 15.6, 20 x 24 13.3 / 13.2,
// 24 x 16 10.8 / 11.5 (there 16-deep products stay whole), 12 x 64 28.4 / 20.3 / 16.2, 12 x 32 17.8 / 14.2 / 13.1, 12 x 20 13.5 / 12.0 / 12.1, 12 x 12 9.5 / 9.8 / 10.8.
int ax_gemm_tc2_share(int tiles, int kb, double* cost) {
    int S = 1;
    double best = kb;
    for (int i = 0; i < 2; i++) {
        const int q = 2 << i;
        const double c = (double)((kb + q - 1) / q) + (i ? 12 : 8);
        if (tiles <= g_share_max[i] && c < best) { S = q; best = c; }
    }
    if (cost) *cost = best;
    return S;
}

// whether an output of n columns of osz bytes, and its addend if there is one, go by TMA (a shared tile needs that)
bool ax_gemm_tc2_by_tma(const void* C, const void* D, long long n, int osz) {
    return ax_gemm_tma_out() && ((uintptr_t)C & 15) == 0 && ((uintptr_t)D & 15) == 0 && n * osz % 16 == 0;
}

// Row tiles of a band.  74 pairs work on as many tiles at once.  While A stays in the L2 (126 MB, shared with B and the output), walking down
// all row tiles of a column reads A and B from memory once; when it does not, every two or three columns read all of A again, and a block of
// about 12 x 6 tiles reads the least.  us with one band / with bands of 12, by MB of A: 8192 x 4096 x 11008 (180) 575 / 545, 8192 x 32000 x 4096
// (67) 1610 / 1470, 8192 x 2 * 11008 x 4096 (67) 1225 / 1145, 32000 x 4096 x 8192 (524) 1944 / 1730, 50000 x 1536 x 3000 (300) 480 / 410,
// 8192 x 4096 x 3072 (50) 161 / 158; but 8192 x 32000 x 2048 (34) 770 / 805 and 6144 x 32000 x 3072 (38) 844 / 867, where bands read B again.
// Bands of 8 and 16 differ from 12 by 1 % either way.
static int band_of(int m, long long k) {
    const int tiles_m = (m + 255) / 256;
    return 2ll * m * k > 52000000ll && tiles_m > 12 ? 12 : tiles_m;
}

// Columns of a tile.  A launch is a set-up, a first load and the last tile's epilogue (f, and c for each tile of a round), a round's k-blocks (t each, by how many of the operands have rows that
// don't start on 32 bytes: every piece of 128 bytes is five sectors then), and for each further round of tiles over the pairs its k-blocks or, where they are few, the epilogue that they run under (e).
// Constants are fitted to 1172 seeded products, groups and sums that narrow tiles take, with rms of 3 to 5 %; f of the wide tile is 0.4 us above its fit, as narrow ones are to win by less than that.
// us of 256 / 192 / 128 columns in chains of launches: 2000 x 1536 x 1536 (48, 64, 96 tiles) 12.8 / 11.3 / 13.6, x 4096 24.8 / 21.8 / 28.1, 8192 x 768 x 2304 (96, 128, 192) 26.6 / 23.2 / 27.9,
// 1536 x 1024 x 1024 (24 shared by two pairs, 36, 48) 9.5 / 8.2 / 7.7, x 2816 15.3 / 14.8 / 13.0, x 5632 20.7 / 24.6 / 22.7, 2000 x 4096 x 1536 (128, 176, 256) 21.3 / 22.9 / 25.4.
// Few k-blocks: 2520 x 2920 x 104 (120, 160, 230) 9.9 / 11.5 / 12.9, 5720 x 816 x 128 (92, 115, 161) 7.9 / 8.2 / 9.2, 1544 x 2176 x 568 (63, 84, 119) 9.9 / 13.0 / 11.3, 768 x 2816 x
// 256 (33, 45, 66) 6.5 / 6.2 / 6.2.  Rows off 32 bytes, shared / 128: 1072 x 312 x (232 + 2456) 13.2 / 16.4, 1528 x (40, 168, 288) x 3304 17.7 / 21.2; 256 / 192: 888 x 2840 x 4360 31.2 / 33.5.
// Where the rule takes a narrow tile, 1055 of other seeded shapes, it has 0.867 of the time of the wide one, in 15 of them more than 4 % longer (0.874, 39 of 1172, when t knew no alignment).
// Only while a plan has queued nothing to another stream (see ax_gemm_plan_begin): products on the side stream fill the pairs that wide tiles leave, and
// the step of 8 x 1024 tokens at D 768 takes 5114 us with narrow ones throughout, 5037 without.  Steps with adapters are 1 to 2 % shorter, small ones up to 5.
// A shared or split depth stays one where the output is fp32, which narrow tiles would sum in one chain: the tensor core's accumulator loses with each step.  2-norm errors against float64 of
// fp32 outputs, shared by two or four / in one chain: 1040 x 720 x 2016 4.7e-7 / 2.1e-6, 2440 x 696 x 1880 9.1e-7 / 1.9e-6, 2248 x 584 x 3496 1.8e-6 / 3.7e-6; rounded to bf16 all are 1.7e-3.
// With three rounds or more the rounds even out and the wide tile, which moves the least, is the best under the power limit: 8192 x 1536 x 2560 (192, 256, 384)
// 48.6 / 49.5 / 58.4.
static int g_pairs = 0;                  // pairs that run at once
TileTimes ax_gemm_tc2_width(const long long* tiles /* of 256, 192, 128 columns */, int kb, bool may_share, int off32 /* operands, 0 to 2 */) {
    static const int width[3] = {256, 192, 128};
    static const double f[3] = {5.1, 4.1, 3.5}, t[3][3] = {{0.282, 0.290, 0.369}, {0.223, 0.304, 0.322}, {0.194, 0.222, 0.275}}, c[3] = {0.0163, 0.0248, 0.0250}, e[3] = {3.4, 3.2, 2.5};
    static const double t_shared[3] = {0.240, 0.255, 0.330};
    TileTimes best = {256, 0.0};
    for (int i = 0; i < 3; i++) {
        const long long rounds = g_pairs > 0 ? (tiles[i] + g_pairs - 1) / g_pairs : 1;
        const double round = t[i][off32] * kb;
        double us = f[i] + c[i] * (rounds > 1 ? g_pairs : tiles[i]) + round + (rounds - 1) * (round > e[i] ? round : e[i]);
        if (i == 0 && may_share && tiles[0] <= 33) {
            const int S = ax_gemm_tc2_share((int)tiles[0], kb, nullptr);
            if (S > 1) us = 7.7 + t_shared[off32] * ((kb + S - 1) / S) + 0.04 * S * tiles[0];
        }
        if (i == 0) best.us = us;
        else if (tiles[0] <= 2 * g_pairs && us < best.us) best = {width[i], us};
    }
    return best;
}

struct SwbArgs { const void* g; const void* u; void* du; };    // SwiGLU backward in the epilogue (C = dg)

// One launch.  grp.mode 0: the plain GEMM (A, B, C, D are element 0 of the arrays).  Grouped modes: see GemmGroup;
// n[] / k[] then hold the per-problem widths (mode 1) or per-segment depths (mode 2).
// Extra K-segments of a grouped launch: mode 1 — problem g adds XA[g] XB[g] (depth xk) to its output; mode 2 — they are
// appended to the launch's own segments (A, B, kv then hold count + xcount entries, at most 6).
template <int A_MN, int B_MN, typename TO, int EPI = EPI_PLAIN, int BN = 256>
static int gemm2_launch(int mode, int count, const void* const* A, const void* const* B, void* const* C, const void* D,
                        const int* mv, const int* nv, const int* kv, float alpha, float beta, int* status, int ksplit, cudaStream_t st,
                        const void* const* XA = nullptr, const void* const* XB = nullptr, int xk = 0, const SwbArgs* swb = nullptr) {
    constexpr bool CAN_SHARE = BN == 256 && (EPI == EPI_PLAIN || EPI == EPI_ROPE);
    const int maxp = clusters_for<A_MN, B_MN, TO, EPI, 1, BN>();
    if (maxp < 1) return -1;
    const int m = mv[0], n = nv[0], k = kv[0];
    GemmGroup grp = {};
    grp.mode = mode; grp.count = count;
    if (g_rope_req.rope_mask) {              // a rotary request is honoured by a mode-1 bf16 launch or refused
        grp.rope_cos = g_rope_req.rope_cos; grp.rope_sin = g_rope_req.rope_sin;
        grp.rope_T = g_rope_req.rope_T; grp.rope_mask = g_rope_req.rope_mask;
        g_rope_req.rope_mask = 0;
        if (mode != 1 || sizeof(TO) != 2 || grp.rope_T < 1 || !grp.rope_cos || !grp.rope_sin) return -1;
        for (int g = 0; g < count; g++) if (((grp.rope_mask >> g) & 1) && nv[g] % 64) return -1;
    }
    CUtensorMap tmA[3], tmB[3], tmC[3], tmD, tmEA[3], tmEB[3];
    grp.whole = 1;
    for (int g = 0; g < (mode == 1 || mode == 3 ? count : 1); g++) grp.whole = grp.whole && (!A_MN || mv[mode == 3 ? g : 0] % 64 == 0) && (!B_MN || nv[g] % b_block(BN) == 0);
    auto map_a = [&](CUtensorMap* t, const void* p, int e, int depth) { return A_MN ? map_mn(t, p, e, depth, grp.whole, 128, 64) : map_km(t, p, e, depth, 128); };
    auto map_b = [&](CUtensorMap* t, const void* p, int e, int depth) { return B_MN ? map_mn(t, p, e, depth, grp.whole, BN / 2, b_block(BN)) : map_km(t, p, e, depth, BN / 2); };
    bool have_x = false;
    int tiles_n = 0;
    if (mode == 0) {
        if (map_a(&tmA[0], A[0], m, k) || map_b(&tmB[0], B[0], n, k)) return 2;
        tiles_n = (n + BN - 1) / BN;
    } else if (mode == 1) {
        if (map_a(&tmA[0], A[0], m, k)) return 2;
        for (int g = 0; g < count; g++) {
            if (map_b(&tmB[g], B[g], nv[g], k)) return 2;
            grp.n[g] = nv[g];
            tiles_n += (nv[g] + BN - 1) / BN;
            if (XA && xk > 0) {
                if (map_a(&tmEA[g], XA[g], m, xk) || map_b(&tmEB[g], XB[g], nv[g], xk)) return 2;
                have_x = true;
            }
        }
        if (have_x) grp.xkb = (xk + BK2 - 1) / BK2;
    } else if (mode == 2) {
        if (count > 6) return -1;
        for (int g = 0; g < count; g++) {
            CUtensorMap* ta = g < 3 ? &tmA[g] : &tmEA[g - 3];
            CUtensorMap* tb_ = g < 3 ? &tmB[g] : &tmEB[g - 3];
            if (map_a(ta, A[g], m, kv[g]) || map_b(tb_, B[g], n, kv[g])) return 2;
            grp.kb[g] = (kv[g] + BK2 - 1) / BK2;
        }
        have_x = count > 3;
        tiles_n = (n + BN - 1) / BN;
    } else if (mode == 3) {
        for (int g = 0; g < count; g++) {
            if (map_a(&tmA[g], A[g], mv[g], k) || map_b(&tmB[g], B[g], nv[g], k)) return 2;
            grp.m[g] = mv[g]; grp.n[g] = nv[g];
        }
    } else {        // mode 4: gate and up weights of the same width n; outputs g, u, h
        if (sizeof(TO) != 2 || count != 2) return -1;
        if (map_a(&tmA[0], A[0], m, k) || map_b(&tmB[0], B[0], n, k) || map_b(&tmB[1], B[1], n, k)) return 2;
        if (XA && xk > 0) {                  // low-rank terms; the zeros come from rows of B behind the last
            for (int q = 0; q < 2; q++)
                if (map_a(&tmEA[q], XA[q], m, xk) || map_b(&tmEB[q], XB[q], n, xk)) return 2;
            have_x = true;
            grp.xkb = (xk + BK2 - 1) / BK2;
            grp.xk_pad = grp.xkb * BK2;
        }
    }
    const bool per_problem_c = mode == 1 || mode == 3;
    // output through TMA tile stores when the destination allows it: 1 = no addend to read, 2 = addend by TMA too
    int units = ((m + 255) / 256) * tiles_n;
    if (mode == 3) { units = 0; for (int g = 0; g < count; g++) units += ((mv[g] + 255) / 256) * ((nv[g] + BN - 1) / BN); }
    if (mode == 4) units = ((m + 255) / 256) * ((n + 127) / 128);
    int kb = (k + BK2 - 1) / BK2 + grp.xkb;
    if (mode == 2) { kb = 0; for (int g = 0; g < count; g++) kb += grp.kb[g]; }
    // (not beside the main chain, whose kernels fill the SMs and where a cluster waits for four or eight free ones in one place: a step of
    // 2 x 1536 tokens at D 1024 took 3522 us with the weight gradients shared, 3506 without)
    grp.S = CAN_SHARE && ksplit == 1 && !ax_gemm_on_side() ? ax_gemm_tc2_share(units, kb, nullptr) : 1;
    units *= ksplit;
    const int osz = ksplit > 1 ? 4 : (int)sizeof(TO);
    const bool has_d = D != nullptr && beta != 0.f && ksplit == 1;
    int tma_out = 0;
    bool c_ok = true;
    for (int g = 0; g < (per_problem_c ? count : (mode == 4 ? 3 : 1)); g++)
        c_ok = c_ok && ax_gemm_tc2_by_tma(C[g], has_d ? D : nullptr, nv[per_problem_c ? g : 0], osz);
    if (c_ok) tma_out = has_d ? 2 : 1;
    if (!tma_out) grp.S = 1;                 // (threads that store their rows write whole tiles)
    // grouped launches need the TMA-store epilogue; only the K-segment form takes an addend
    if (mode != 0 && (ksplit != 1 || !(tma_out == 1 || (tma_out == 2 && mode == 2)))) return -1;
    if (grp.rope_mask && tma_out != 1) return -1;
    if (tma_out) {
        size_t wsb0 = 0;
        if (per_problem_c) {
            for (int g = 0; g < count; g++) if (map_c(&tmC[g], C[g], mode == 3 ? mv[g] : m, nv[g], 1, osz)) return 2;
        } else if (mode == 4) {
            for (int g = 0; g < 3; g++) if (map_c(&tmC[g], C[g], m, n, 1, osz)) return 2;
        } else {
            void* base = ksplit > 1 ? (void*)ax_splitk_ws(&wsb0) : C[0];
            if (map_c(&tmC[0], base, m, n, ksplit > 1 ? ksplit : 1, osz)) return 2;
        }
        tmD = tmC[0];
        if (swb) {
            if (tma_out != 1 || sizeof(TO) != 2) return -1;
            if (map_c(&tmC[0], C[0], m, n, 1, 2, true) || map_c(&tmC[1], swb->du, m, n, 1, 2, true) ||
                map_c(&tmC[2], const_cast<void*>(swb->u), m, n, 1, 2, true) || map_c(&tmD, const_cast<void*>(swb->g), m, n, 1, 2, true)) return 2;
        }
        if (tma_out == 2 && map_c(&tmD, const_cast<void*>(D), m, n, 1, osz)) return 2;
    } else {
        tmC[0] = tmA[0]; tmD = tmA[0];
    }
    for (int g = 0; g < 3; g++) {           // unused slots carry valid (ignored) maps
        const bool used = (mode == 1 || mode == 4) ? (have_x && g < count) : (mode == 2 && g + 3 < count);
        if (!used) { tmEA[g] = tmA[0]; tmEB[g] = tmB[0]; }
    }
    for (int g = 1; g < 3; g++) {
        if ((mode != 2 && mode != 3) || g >= count) tmA[g] = tmA[0];
        if (mode == 0 || g >= count) tmB[g] = tmB[0];
        if (mode != 4 && !swb && (!per_problem_c || g >= count || !tma_out)) tmC[g] = tmC[0];
    }
    const int pairs = units < maxp ? units : maxp;
    grp.band = band_of(m, mode == 2 ? (long long)kb * BK2 : k);
    ax_gemm_parts = grp.S;
    size_t wsb = 0;
    float* ws = ax_splitk_ws(&wsb);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs * grp.S, 1, 1);
    cfg.blockDim = dim3(EpiCfg<EPI>::THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM2;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2 * grp.S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = ax_gemm_pdl() ? 2 : 1;
    TO* Cp = (TO*)C[0]; const TO* Dp = (const TO*)D;
    long long* prof = nullptr;
#ifdef AXENG_PROF       // debugging aid of instrumented builds: allocates, synchronises and prints per launch
    static const bool want_prof = getenv("AXENG_GEMM_PROF") != nullptr;
    if (want_prof && (cudaMalloc(&prof, 64) != cudaSuccess || cudaMemset(prof, 0, 64) != cudaSuccess)) prof = nullptr;
#endif
    auto launch = [&](auto kern) {
        return cudaLaunchKernelEx(&cfg, kern, tmA[0], tmB[0], tmC[0], tmD, tmA[1], tmA[2], tmB[1], tmB[2], tmC[1], tmC[2],
                                  tmEA[0], tmEA[1], tmEA[2], tmEB[0], tmEB[1], tmEB[2], grp, tma_out, Cp, Dp, m, n, k, alpha, beta, status, ksplit, ws, prof);
    };
    cudaError_t err;
    if constexpr (CAN_SHARE) err = grp.S > 1 ? launch(k_gemm_tc2<A_MN, B_MN, TO, EPI, true, BN>) : launch(k_gemm_tc2<A_MN, B_MN, TO, EPI, false, BN>);
    else err = launch(k_gemm_tc2<A_MN, B_MN, TO, EPI, false, BN>);
    if (err != cudaSuccess) return 3;
#ifdef AXENG_PROF
    if (prof) {
        long long h[8];
        cudaStreamSynchronize(st);
        cudaMemcpy(h, prof, 64, cudaMemcpyDeviceToHost);
        cudaFree(prof);
        fprintf(stderr, "gemm2 %dx%dx%d mode %d split %d pairs %d (cycles from entry): setup %lld dep %lld first_full %lld last_mma %lld last_acc %lld stored %lld exit %lld\n",
                m, n, k, mode, ksplit, pairs, h[1] - h[0], h[2] - h[0], h[3] - h[0], h[4] - h[0], h[5] - h[0], h[6] - h[0], h[7] - h[0]);
    }
#endif
    if (ksplit > 1) ax_splitk_reduce_launch<TO>(ws, ksplit, Cp, Dp, (long long)m * n, alpha, beta, st);
    return 0;
}

// Resolve the co-resident pair count of every variant up front (not while a graph is being captured).
int ax_gemm_tc2_init(void) {
    int worst = 1 << 30;
#define ALL_KERNELS(S) clusters_for<0, 1, bf16, EPI_PLAIN, S>(), clusters_for<0, 1, float, EPI_PLAIN, S>(), clusters_for<0, 0, bf16, EPI_PLAIN, S>(),      \
                       clusters_for<0, 0, float, EPI_PLAIN, S>(), clusters_for<1, 1, bf16, EPI_PLAIN, S>(), clusters_for<1, 1, float, EPI_PLAIN, S>(), \
                       clusters_for<0, 1, bf16, EPI_ROPE, S>()
    const int v[9] = {ALL_KERNELS(1), clusters_for<0, 1, bf16, EPI_SWIGLU>(), clusters_for<0, 0, bf16, EPI_SWB>()};
    const int v2[7] = {ALL_KERNELS(2)}, v4[7] = {ALL_KERNELS(4)};
#undef ALL_KERNELS
#define NARROW(W) clusters_for<0, 1, bf16, EPI_PLAIN, 1, W>(), clusters_for<0, 1, float, EPI_PLAIN, 1, W>(), clusters_for<0, 0, bf16, EPI_PLAIN, 1, W>(),      \
                  clusters_for<0, 0, float, EPI_PLAIN, 1, W>(), clusters_for<1, 1, bf16, EPI_PLAIN, 1, W>(), clusters_for<1, 1, float, EPI_PLAIN, 1, W>(), \
                  clusters_for<0, 1, bf16, EPI_ROPE, 1, W>(), clusters_for<0, 0, bf16, EPI_SWB, 1, W>()
    for (int x : {NARROW(192), NARROW(128)}) worst = x < worst ? x : worst;
#undef NARROW
    g_share_max[0] = g_share_max[1] = AX_SMS;
    for (int i = 0; i < 7; i++) {
        g_share_max[0] = v2[i] < g_share_max[0] ? v2[i] : g_share_max[0];
        g_share_max[1] = v4[i] < g_share_max[1] ? v4[i] : g_share_max[1];
    }
    for (int i = 0; i < 9; i++) worst = v[i] < worst ? v[i] : worst;
    g_pairs = worst;
    return worst;      // pairs that can run together (<= 0: the paired kernel is unavailable)
}

// Same argument meaning as ax_gemm_tc; returns -1 when the paired kernel cannot run here.
int ax_gemm_tc2(int out_bf16, int tb, const void* A, const void* B, void* C, const void* D,
                int m, int n, int k, float alpha, float beta, int* status, int ksplit, int bn, cudaStream_t st) {
    const void* Av[1] = {A}; const void* Bv[1] = {B}; void* Cv[1] = {C};
#define G2W(AM, BMj, T, W) gemm2_launch<AM, BMj, T, EPI_PLAIN, W>(0, 1, Av, Bv, Cv, D, &m, &n, &k, alpha, beta, status, ksplit, st)
#define G2T(AM, BMj, T) (bn == 256 ? G2W(AM, BMj, T, 256) : bn == 192 ? G2W(AM, BMj, T, 192) : G2W(AM, BMj, T, 128))
#define G2(AM, BMj) (out_bf16 ? G2T(AM, BMj, bf16) : G2T(AM, BMj, float))
    if (tb == 0) return G2(0, 1);
    if (tb == 1) return G2(0, 0);
    return G2(1, 1);
#undef G2
#undef G2T
#undef G2W
}

// Grouped launch (see GemmGroup).  mode 1: A[0] shared, B[g] / C[g] / n[g] per problem, m[0], k[0].  mode 2: A[s] / B[s] /
// k[s] per segment, C[0], m[0], n[0].  mode 3: A[g] / B[g] / C[g] / m[g] / n[g] per problem, k[0].  Returns -1 when this
// kernel cannot serve the request (the caller then runs the problems one by one).  mode 4: A[0], B[0] = gate weights,
// B[1] = up weights (both n[0] wide), C[0] = g, C[1] = u, C[2] = silu(g) * u; bf16 output only.  XA / XB / xk (mode 1):
// every problem's own extra K-segment.  Mode 2 takes up to 6 segments and an addend D (C = alpha * sum + beta * D).
int ax_gemm_tc2_group(int out_bf16, int tb, int mode, int count, const void* const* A, const void* const* B, void* const* C,
                      const int* m, const int* n, const int* k, float alpha, int* status, cudaStream_t st,
                      const void* const* XA, const void* const* XB, int xk, const void* D, float beta,
                      const void* swb_g, const void* swb_u, void* swb_du) {
    const int rope_mask = g_rope_req.rope_mask;
    const int maxc = mode == 2 ? 6 : 3;
    const SwbArgs swb_args = {swb_g, swb_u, swb_du};
    const SwbArgs* swb = swb_g ? &swb_args : nullptr;
    if (swb && (mode != 2 || !out_bf16 || tb != 1 || D || n[0] % 8 || !aligned16(swb_g) || !aligned16(swb_u) || !aligned16(swb_du))) { g_rope_req.rope_mask = 0; return -1; }
    if (count < (swb ? 1 : 2) || count > maxc || mode < 1 || mode > 4) { g_rope_req.rope_mask = 0; return -1; }
    if (mode == 4 && (!out_bf16 || tb != 0 || count != 2 || !aligned16(C[2]))) { g_rope_req.rope_mask = 0; return -1; }
    if (rope_mask && (mode != 1 || !out_bf16 || tb != 0)) { g_rope_req.rope_mask = 0; return -1; }
    if (XA && ((mode != 1 && mode != 4) || tb == 2 || xk < 8 || xk % 8)) { g_rope_req.rope_mask = 0; return -1; }
    if (D && (mode != 2 || !aligned16(D))) { g_rope_req.rope_mask = 0; return -1; }
    if (ax_gemm_mode() == 0) {
        const int rc = ax_gemm_small(out_bf16, tb, mode, count, A, B, C, m, n, k, alpha, st, XA, XB, xk, D, D ? beta : 0.f, swb_g, swb_u, swb_du,
                                     g_rope_req.rope_cos, g_rope_req.rope_sin, g_rope_req.rope_T, rope_mask);
        if (rc >= 0) { g_rope_req.rope_mask = 0; ax_variant = 0x26; return rc; }
    }
    for (int g = 0; g < count; g++) {
        bool bad = !aligned16(A[(mode == 2 || mode == 3) ? g : 0]) || !aligned16(B[g]);
        if (XA) bad = bad || !XA[g] || !XB[g] || !aligned16(XA[g]) || !aligned16(XB[g]);
        const int mg = m[mode == 3 ? g : 0], ng = n[(mode == 1 || mode == 3) ? g : 0], kg = k[mode == 2 ? g : 0];
        bad = bad || mg < 256 || ng < 8 || kg < 8;
        if (tb == 0) bad = bad || kg % 8 || ng % 8;
        else if (tb == 1) bad = bad || kg % 8;
        else bad = bad || mg % 8 || ng % 8;
        if (bad) { g_rope_req.rope_mask = 0; return -1; }
    }
    ax_variant = 0x23;
    // (a caller who forces this kernel gets the wide tiles, and what they share, as they are)
    int bn = 256;
    if (ax_gemm_mode() == 0 && !ax_gemm_beside() && (mode == 1 || mode == 2)) {
        long long tiles[3] = {0, 0, 0};
        int kb = mode == 1 && XA ? (xk + BK2 - 1) / BK2 : 0;
        for (int g = 0; g < (mode == 2 ? count : 1); g++) kb += (k[g] + BK2 - 1) / BK2;
        for (int i = 0; i < 3; i++)
            for (int g = 0; g < (mode == 1 ? count : 1); g++) tiles[i] += (long long)((m[0] + 255) / 256) * ((n[g] + 255 - 64 * i) / (256 - 64 * i));
        if (out_bf16 || ax_gemm_tc2_share((int)(tiles[0] < AX_SMS ? tiles[0] : AX_SMS), kb, nullptr) == 1) {
            int kk = k[0], nn = 0;           // the deepest segment, any problem
            for (int g = 1; mode == 2 && g < count; g++) kk = k[g] > kk ? k[g] : kk;
            for (int g = 0; g < (mode == 1 ? count : 1); g++) nn |= n[g];
            bn = ax_gemm_tc2_width(tiles, kb, !swb, ((tb == 2 ? m[0] : kk) % 16 != 0) + ((tb == 1 ? kk : nn) % 16 != 0)).width;
        }
    }
    ax_gemm_width = mode == 4 ? 256 : bn;
#define G2W(AM, BMj, T, EPI, W) gemm2_launch<AM, BMj, T, EPI, W>(mode, count, A, B, C, D, m, n, k, alpha, D ? beta : 0.f, status, 1, st, XA, XB, xk, swb)
#define G2X(AM, BMj, T, EPI) (bn == 256 ? G2W(AM, BMj, T, EPI, 256) : bn == 192 ? G2W(AM, BMj, T, EPI, 192) : G2W(AM, BMj, T, EPI, 128))
#define G2(AM, BMj) (out_bf16 ? G2X(AM, BMj, bf16, EPI_PLAIN) : G2X(AM, BMj, float, EPI_PLAIN))
    if (swb) return G2X(0, 0, bf16, EPI_SWB);
    if (mode == 4) return G2W(0, 1, bf16, EPI_SWIGLU, 256);
    if (rope_mask) return G2X(0, 1, bf16, EPI_ROPE);
    if (tb == 0) return G2(0, 1);
    if (tb == 1) return G2(0, 0);
    return G2(1, 1);
#undef G2X
#undef G2W
#undef G2
}
