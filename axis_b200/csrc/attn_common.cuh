// Device helpers shared by the tcgen05 attention kernels (head_dim 64 and 128).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"
#include "tc_common.cuh"

#define LOG2E 1.4426950408889634f
#define LN2 0.6931471805599453f

__device__ __forceinline__ void named_bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// max of three floats in one instruction (3-input max.f32 of sm_100)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// mbarrier wait that lets the hardware park the thread: try_wait with a suspend-time hint returns when the phase
// completes or the hint (in ns) runs out, so a waiting warp issues a handful of instructions per microsecond instead
// of spinning (a spinning warp is always eligible and takes issue slots from the warps that compute).  Bounded by
// elapsed SM cycles (about a second), then false.
__device__ __forceinline__ bool mbar_try_park(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(4000u) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_park(uint32_t bar, uint32_t parity) {
    if (mbar_try_park(bar, parity)) return true;
    const long long t0 = clock64();
    do {
        if (mbar_try_park(bar, parity)) return true;
    } while (clock64() - t0 < (1ll << 31));
    return false;
}
// Shared-memory descriptors of these kernels all use SBO = 1024 and 128-byte swizzle, so their upper
// word is one constant and the lower word is (address >> 4) | (LBO >> 4) << 16: the MMA-issuing thread
// keeps a few base words and adds tile offsets (in 16-byte units) instead of rebuilding descriptors.
#define DESC_HI ((1024u >> 4) | (1u << 14) | (2u << 29))
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr, uint32_t lbo_bytes) {
    return ((saddr & 0x3FFFF) >> 4) | ((lbo_bytes >> 4) << 16);
}
__device__ __forceinline__ uint64_t desc_of(uint32_t lo) { return ((uint64_t)DESC_HI << 32) | (uint64_t)lo; }
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* m, uint32_t src, int x, int y, int z, int w) {
    asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(m)), "r"(src), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// 1-D bulk copy global -> this CTA's shared memory (16-byte aligned addresses, size a multiple of 16), completion on an mbarrier
__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Issue forms for a converged warp: every lane executes the surrounding code (so addresses and descriptors stay
// warp-uniform and cheap to form) and the elected lane issues.  Measured on B200: a 128 x 64 x 16 MMA with A in
// TMEM issues every 32.6 cycles this way (its 32 cycles of math) against 45-50 from a lone thread in a divergent branch.
__device__ __forceinline__ void mma_ts_e(uint32_t d, uint32_t a, uint64_t bd, uint32_t id, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bd), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_ss_e(uint32_t d, uint64_t ad, uint64_t bd, uint32_t id, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(ad), "l"(bd), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void commit_e(uint32_t bar) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// two numbers each as the sum of two bf16 ones
__device__ __forceinline__ void split_bf16(float x, float y, uint32_t& hi, uint32_t& lo) {
    hi = pack_bf16(x, y);
    lo = pack_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}
// columns c0 .. c0 + 7 (a) and as many HALF further on (b) of a gradient row, times f, rotated back where the tables are given (a pair's columns are
// HALF apart): out1 = g1 c + g2 s, out2 = -g1 s + g2 c
template <int HALF = 32>
__device__ __forceinline__ void store_grad8(float* a, float* b, int c0, float f, const float* cr, const float* sr, bf16* row, int dh) {
#pragma unroll
    for (int z = 0; z < 8; z++) { a[z] *= f; b[z] *= f; }
    if (cr) {
#pragma unroll
        for (int z = 0; z < 8; z += 4) {
            const float4 c4 = *reinterpret_cast<const float4*>(cr + c0 + z), s4 = *reinterpret_cast<const float4*>(sr + c0 + z);
            const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int y = 0; y < 4; y++) {
                const float g1 = a[z + y], g2 = b[z + y];
                a[z + y] = g1 * cc[y] + g2 * ss[y];
                b[z + y] = g2 * cc[y] - g1 * ss[y];
            }
        }
    }
    if (c0 < dh) *reinterpret_cast<uint4*>(row + c0) = make_uint4(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7]));
    if (HALF + c0 < dh) *reinterpret_cast<uint4*>(row + HALF + c0) = make_uint4(pack_bf16(b[0], b[1]), pack_bf16(b[2], b[3]), pack_bf16(b[4], b[5]), pack_bf16(b[6], b[7]));
}

// Sixteen columns of a row of the sums that each CTA of a cluster has at `at` in its shared memory, added in rank order: eight, and eight HALF further on
template <int HALF>
__device__ __forceinline__ void cluster_sum16(uint32_t at, int S, float* a) {
#pragma unroll
    for (int z = 0; z < 16; z++) a[z] = 0.f;
    for (int q = 0; q < S; q++)
#pragma unroll
        for (int z = 0; z < 16; z += 4) {
            float4 x;
            asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t}"
                         : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(at + ((z & 7) + (z >> 3) * HALF) * 4), "r"(q) : "memory");
            a[z] += x.x; a[z + 1] += x.y; a[z + 2] += x.z; a[z + 3] += x.w;
        }
}
// CTAs that share the walk of a key tile of 128 in the backward kernels of whole tiles (clusters, whose dK and dV meet through distributed shared memory).  One
// CTA to a key tile and kv head is as long as its chain, the query tiles of all heads of the group; 74 clusters of two and 33 of four run at once.
// Backward in us with 1 / 2 / 4 (CTAs at 1, chain), head_dim 64 | 128 where a tile of the chain costs twice as much:
// B1 H8 KV2 T512 (8, 16) 39.9 / 27.5 / 23.2 | 72.3 / 44.6 / 34.1, B8 H16 KV4 T256 (64, 8) 30.7 / 26.2 / 40.1 | 51.6 / 38.2 / 54.5, B2 H16 KV4 T1024 (64, 32) 73.2 /
// 47.5 / 53.0 | 142 / 83.4 / 77.2, B1 H16 KV4 T2048 (64, 64) 130 / 76 / 67 | 262 / 144 / 107.  Short chains: B3 H8 KV4 T256 (24, 4) 17.6 / 17.2, B24 H2 KV1 T256
// (48, 4) 18.1 / 19.1, B8 H6 KV3 T384 (72, 6) 23.0 / 21.9 | B11 H4 KV2 T128 (22, 2) 19.1 / 18.8, B31 H2 KV2 T256 (62, 2) 19.6 / 20.6, B27 H6 KV2 T128 (54, 3) 26.4 / 25.6.
// A cluster that starts late is another set-up, first load and merge, 9 tiles of the chain at head_dim 64 and 4.5 at 128, behind the shortest walks of the first
// round: it pays where the walks of a head's key tiles differ enough.  Two CTAs, beyond 74 key tiles (CTAs, key tiles to a head, heads of a group): T128 (80, 1, 2)
// 17 / 30 | 23.9 / 38.3, (96, 1, 4) | 38.0 / 53.8, T256 (96, 2, 2) | 31.9 / 40.0, (88, 2, 4) | 51.2 / 53.1, T512 (96, 4, 3) 36.5 / 38.6, (84, 4, 2) | 46.1 / 39.7, T768
// (96, 6, 2) 38.1 / 36.7, T640 (100, 5, 3) | 75.2 / 58.7, T1536 (84, 12, 3) 78.3 / 50.4, (144, 12, 3) | 157 / 114, T4096 (128, 32, 3) 186 / 108; B4 H24 KV8 T768 (192, 6, 3)
// 54.0 / 72.6 | 104 / 117.  Four CTAs beyond 33 key tiles, 2 / 4: T2048 (64, 16, 16) 256 / 167, T1024 (64, 8, 8) 78.9 / 71.8, T256 (40, 2, 32) | 179 / 141; T128
// (36, 1, 48) 85 / 104 | (40, 1, 32) 121 / 141.
static inline int attn_tile_parts(int head_dim, long long ctas, int key_tiles /* of a head */, int rep) {
    const bool wide = head_dim > 64;
    const long long chain = (long long)rep * key_tiles;
    // Clusters of S, `fit` of which run at once, the longest first: twice S times what they take less than one CTA for each does, in tiles of the chain.  The last to
    // start in the second round waits for walk number 2 fit - ctas of the first.
    auto gain = [&](int S, int fit) {
        const long long late = ctas - fit, heads = ctas / key_tiles;
        if (late > fit) return -1ll;
        const long long first = (fit - late) / heads;
        return S * chain - rep * (key_tiles - first + 1);
    };
    int S = 1;
    if (ctas <= AX_SMS / 2 ? chain >= (wide ? 2 : 4) + (ctas <= 40 ? 0 : wide ? 1 : 2) : ctas <= AX_SMS && gain(2, AX_SMS / 2) > (wide ? 9 : 15)) S = 2;
    if (S == 2 && (ctas <= 33 ? chain >= 8 : ctas <= AX_SMS / 2 && key_tiles > 1 && chain >= (wide ? 32 : 48))) S = 4;
    return S;
}
// Launch of a kernel whose CTAs form clusters of S (1: none).  Up to half a CTA for each SM start while the grid in front of them ends (the step of two layers of 512
// tokens, D 256: 275 -> 259 us).  More would take SMs from what still runs, by side-stream products or by stacking the longest CTAs on the SMs that are free first:
// all of them early cost the step of 8192 tokens with adapters 1.2 %, one of 22 x 80 tokens 5 %.
template <typename... KA, typename... A>
static inline cudaError_t attn_launch(void (*kern)(KA...), long long grid, int block, size_t smem, int S, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(grid * S)); cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = grid * S <= AX_SMS / 2 && ax_gemm_pdl();
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = S; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = S > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KA>(args)...);
}
