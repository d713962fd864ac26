// General GEMM on CUDA cores: true fp32 FMA accumulation, any shape, stride or
// alignment, fp32 or bf16 operands and output, strided-batched.  k_gemm_f32 serves
// the fp32 parity mode, k_gemm_simt the bf16 shapes the tensor-core path does not take.
//
//   C[b][i,j] = alpha * sum_k A(i,k) * B(k,j) + beta * D[b][i,j]
//   tb = 0: A [m,k] row-major, B [k,n] row-major
//   tb = 1: A [m,k] row-major, B [n,k] row-major (C = A B^T)
//   tb = 2: A [k,m] row-major, B [k,n] row-major (C = A^T B)
#include "common.cuh"
#include "kernels.h"

#define GT 64      // C tile edge
#define GK 16      // k step

template <typename TI, typename TO>
__global__ void __launch_bounds__(256)
k_gemm_simt(const TI* __restrict__ A, const TI* __restrict__ B, TO* C, const TO* D,
            int m, int n, int k, long long as_m, long long as_k, long long bs_k, long long bs_n,
            long long sa, long long sb, long long sc, float alpha, float beta) {
    __shared__ float As[GK][GT + 4];
    __shared__ float Bs[GK][GT + 4];
    const int bz = blockIdx.z;
    A += (long long)bz * sa;
    B += (long long)bz * sb;
    C += (long long)bz * sc;
    if (D) D += (long long)bz * sc;
    const int i0 = blockIdx.y * GT, j0 = blockIdx.x * GT;
    const int tid = threadIdx.x;
    const int ty = tid >> 4, tx = tid & 15;
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] = 0.f;

    const bool a_kfast = as_k == 1;      // consecutive threads along k when k is contiguous
    const bool b_nfast = bs_n == 1;
    for (int k0 = 0; k0 < k; k0 += GK) {
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const int e = tid + l * 256;                 // 0..1023
            int ii, kk;
            if (a_kfast) { kk = e & (GK - 1); ii = e >> 4; } else { ii = e & (GT - 1); kk = e >> 6; }
            const int gi = i0 + ii, gk = k0 + kk;
            As[kk][ii] = (gi < m && gk < k) ? ldf(A, gi * as_m + gk * as_k) : 0.f;
            int jj, k2;
            if (b_nfast) { jj = e & (GT - 1); k2 = e >> 6; } else { k2 = e & (GK - 1); jj = e >> 4; }
            const int gj = j0 + jj, gk2 = k0 + k2;
            Bs[k2][jj] = (gj < n && gk2 < k) ? ldf(B, gk2 * bs_k + gj * bs_n) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GK; kk++) {
            float a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; q++) { a[q] = As[kk][ty * 4 + q]; b[q] = Bs[kk][tx * 4 + q]; }
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[p][q] = fmaf(a[p], b[q], acc[p][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const int gi = i0 + ty * 4 + p;
        if (gi >= m) continue;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int gj = j0 + tx * 4 + q;
            if (gj >= n) continue;
            const long long idx = (long long)gi * n + gj;
            float r = alpha * acc[p][q];
            if (beta != 0.f) r += beta * ldf(D, idx);
            stf(C, idx, r);
        }
    }
}

// ── fp32 operands: tiles through shared memory by cp.async, split over K inside the CTA and over a cluster ─────────
// The fp32 mode's products are small (a few hundred rows and columns): what bounds them is latency, not FMA rate.  A
// product of 512 x 256 x 256 is 32 tiles of 64 x 64 for 148 SMs, and a tile that walks its depth one 16-deep step after
// another pays a memory round trip per step.  So
//   * the depth travels in steps of 64 through a ring of cp.async stages that is filled before the first FMA;
//   * small tiles (64 x 32, 32 x 32) cut every step among four groups of 64 threads;
//   * where the tiles still leave SMs idle, a cluster of 2, 4 or 8 CTAs cuts the depth once more and adds its partial
//     tiles through distributed shared memory.
// 512 x 256 x 256 took 46 us with 64 x 64 tiles, 16-deep steps and no prefetch; what each tile takes now stands at f32_cut.
// All partial sums meet in a fixed order: run-to-run identical.  Operands keep their layout in shared memory: a
// K-major operand is read as 16-byte pieces along K (row pitch BK + 4: the rows of a warp fall in different banks), an
// M/N-major one as 16-byte pieces along M/N.
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, int bytes) {      // bytes < 16: the rest is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// rows x cols window (row pitch ld) at (r0, c0) of a matrix with R x C elements -> dst [rows][PITCH]; outside = 0
template <int ROWS, int COLS, int PITCH, bool VEC, int THREADS>
__device__ __forceinline__ void tile_cp(float* dst, const float* src, long long ld, int r0, int c0, int R, int C) {
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(dst);
    constexpr int W = VEC ? 4 : 1;
#pragma unroll
    for (int e = threadIdx.x; e < ROWS * COLS / W; e += THREADS) {
        const int r = e / (COLS / W), c = e % (COLS / W) * W;
        const int gr = r0 + r, gc = c0 + c;
        const int n = gr < R && gc < C ? min(W, C - gc) * 4 : 0;
        const float* p = n ? src + (long long)gr * ld + gc : src;
        if (VEC) cp16(base + (r * PITCH + c) * 4, p, n);
        else cp4(base + (r * PITCH + c) * 4, p, n);
    }
}
template <int BM, int BN, int BK, int KG, int TM, int TN, int ST, bool A_MN, bool B_KM>
struct F32Tile {
    static constexpr int THREADS = KG * (BM / TM) * (BN / TN);
    static constexpr int AP = (A_MN ? BM : BK) + 4, BP = (B_KM ? BK : BN) + 4;
    static constexpr int A_EL = (A_MN ? BK : BM) * AP, B_EL = (B_KM ? BN : BK) * BP;
    static constexpr int RED = KG * BM * (BN + 4);                  // partial tiles of the K groups (over the ring)
    static constexpr int EL = ST * (A_EL + B_EL) > RED ? ST * (A_EL + B_EL) : RED;
    static constexpr int SMEM = EL * 4;
};
// What one launch computes: up to three problems of one A-shape (their column tiles form one tile space), each the sum of its `nseg` segments
// seg[g * nseg ...]; the plain product is one problem of one segment.  A group is latency like a product of its size, its members one
// after the other are that many times as much.  With the tiles of `f32_gemm` the step of a 256-wide model of four layers, 512 tokens, takes 857 us
// in place of 987 (58 products of it had launches of their own, four activations and their backward too).
//   F32_SWIGLU: B and B2 are the gate and up weights; a tile holds BN / 2 columns of either; C = g, u, silu(g) * u
//   F32_SWB: the product is dh of h = silu(g) * u and stays in registers; C = dg, du
enum { F32_PLAIN, F32_SWIGLU, F32_SWB };
struct F32Seg { const float* A; const float* B; const float* B2; int k; };
struct F32Group {
    F32Seg seg[6];
    int nprob, nseg, n[3];
    float* C[3];
    const float* D;             // addend (one problem)
    const float* G; const float* U;
};
template <int BM, int BN, int BK, int KG, int TM, int TN, int ST, bool A_MN, bool B_KM, bool VEC, int EPI, bool ONE>
__global__ void __launch_bounds__(KG * (BM / TM) * (BN / TN))
k_gemm_f32(const __grid_constant__ F32Group a, int m, long long sa, long long sb, long long sc, int ksplit, float alpha, float beta) {
    using L = F32Tile<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM>;
    constexpr int TH = L::THREADS, TX = BN / TN, TY = BM / TM, GT_ = TX * TY, KS = BK / KG, W = EPI == F32_SWIGLU ? BN / 2 : BN;
    const int nprob = ONE ? 1 : a.nprob, nseg = ONE ? 1 : a.nseg;
    extern __shared__ __align__(16) float sm[];
    const int split = blockIdx.x % ksplit, i0 = blockIdx.y * BM;
    int tn = blockIdx.x / ksplit, g = 0;
    for (; g + 1 < nprob; g++) {
        const int t = (a.n[g] + W - 1) / W;
        if (tn < t) break;
        tn -= t;
    }
    const int n = a.n[g], j0 = tn * W;
    const F32Seg* seg = a.seg + g * nseg;
    const long long oa = blockIdx.z * sa, ob = blockIdx.z * sb, oc = blockIdx.z * sc;
    float* C = a.C[g] + oc;
    const float* D = a.D ? a.D + oc : nullptr;
    int steps_all = 0;
    for (int q = 0; q < nseg; q++) steps_all += (seg[q].k + BK - 1) / BK;
    const int per = (steps_all + ksplit - 1) / ksplit;
    const int s0 = split * per, s1 = min(steps_all, s0 + per), steps = max(s1 - s0, 0);
    const int grp = threadIdx.x / GT_, tid = threadIdx.x % GT_, ty = tid / TX, tx = tid % TX;
    int ls = 0, lk = s0;                                  // next step to load: segment and step inside it
    auto load = [&](int slot) {
        while (ls + 1 < nseg && lk >= (seg[ls].k + BK - 1) / BK) lk -= (seg[ls++].k + BK - 1) / BK;
        float* as = sm + slot * (L::A_EL + L::B_EL);
        float* bs = as + L::A_EL;
        const int k = seg[ls].k, k0 = lk++ * BK;
        const float* A = seg[ls].A + oa; const float* B = seg[ls].B + ob;
        if (A_MN) tile_cp<BK, BM, L::AP, VEC, TH>(as, A, m, k0, i0, k, m);
        else tile_cp<BM, BK, L::AP, VEC, TH>(as, A, k, i0, k0, m, k);
        if constexpr (EPI == F32_SWIGLU) {
            tile_cp<BK, BN / 2, L::BP, VEC, TH>(bs, B, n, k0, j0, k, n);
            tile_cp<BK, BN / 2, L::BP, VEC, TH>(bs + BN / 2, seg[ls].B2, n, k0, j0, k, n);
        }
        else if (B_KM) tile_cp<BN, BK, L::BP, VEC, TH>(bs, B, k, j0, k0, n, k);
        else tile_cp<BK, BN, L::BP, VEC, TH>(bs, B, n, k0, j0, k, n);
    };
    float acc[TM][TN];
#pragma unroll
    for (int p = 0; p < TM; p++)
#pragma unroll
        for (int q = 0; q < TN; q++) acc[p][q] = 0.f;
    pdl_enter();                                          // which tile this is comes from the arguments alone
#pragma unroll
    for (int st = 0; st < ST - 1; st++) {
        if (st < steps) load(st);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // rows of a thread: M-major operands in runs of four (16-byte reads along M), K-major ones TY apart; columns alike
    auto row_of = [&](int p) { return A_MN ? (p / 4) * (BM * 4 / TM) + ty * 4 + (p & 3) : ty + p * TY; };
    auto col_of = [&](int q) { return B_KM ? tx + q * TX : (q / 4) * (BN * 4 / TN) + tx * 4 + (q & 3); };
    for (int st = 0; st < steps; st++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();                                  // stage st has landed and everyone has left stage st - 1
        if (st + ST - 1 < steps) load((st + ST - 1) % ST);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = sm + (st % ST) * (L::A_EL + L::B_EL);
        const float* bs = as + L::A_EL;
#pragma unroll
        for (int kk = 0; kk < KS; kk += 4) {
            const int kb = grp * KS + kk;
            float a[4][TM], b[4][TN];
            if (A_MN) {
#pragma unroll
                for (int z = 0; z < 4; z++)
#pragma unroll
                    for (int p = 0; p < TM; p += 4) *reinterpret_cast<float4*>(&a[z][p]) = *reinterpret_cast<const float4*>(as + (kb + z) * L::AP + row_of(p));
            } else {
#pragma unroll
                for (int p = 0; p < TM; p++) {
                    const float4 v = *reinterpret_cast<const float4*>(as + row_of(p) * L::AP + kb);
                    a[0][p] = v.x; a[1][p] = v.y; a[2][p] = v.z; a[3][p] = v.w;
                }
            }
            if (B_KM) {
#pragma unroll
                for (int q = 0; q < TN; q++) {
                    const float4 v = *reinterpret_cast<const float4*>(bs + col_of(q) * L::BP + kb);
                    b[0][q] = v.x; b[1][q] = v.y; b[2][q] = v.z; b[3][q] = v.w;
                }
            } else {
#pragma unroll
                for (int z = 0; z < 4; z++)
#pragma unroll
                    for (int q = 0; q < TN; q += 4) *reinterpret_cast<float4*>(&b[z][q]) = *reinterpret_cast<const float4*>(bs + (kb + z) * L::BP + col_of(q));
            }
#pragma unroll
            for (int z = 0; z < 4; z++)
#pragma unroll
                for (int p = 0; p < TM; p++)
#pragma unroll
                    for (int q = 0; q < TN; q++) acc[p][q] = fmaf(a[z][p], b[z][q], acc[p][q]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                      // the ring becomes the exchange area
    constexpr int RP = BN + 4;
    float* red = sm + grp * BM * RP;
#pragma unroll
    for (int p = 0; p < TM; p++)
#pragma unroll
        for (int q = 0; q < TN; q += B_KM ? 1 : 4) {
            float* at = red + row_of(p) * RP + col_of(q);
            if (B_KM) *at = acc[p][q];
            else *reinterpret_cast<float4*>(at) = make_float4(acc[p][q], acc[p][q + (B_KM ? 0 : 1)], acc[p][q + (B_KM ? 0 : 2)], acc[p][q + (B_KM ? 0 : 3)]);
        }
    __syncthreads();
    if (ksplit > 1) {
        if (KG > 1) {                                     // this CTA's groups first, so that peers read one tile
            for (int e = threadIdx.x; e < BM * BN; e += TH) {
                const int o = (e / BN) * RP + e % BN;
                float t = sm[o];
#pragma unroll
                for (int g = 1; g < KG; g++) t += sm[g * BM * RP + o];
                sm[o] = t;
            }
        }
        cluster_sync();
    }
    // output rows: all of them, or this CTA's share of the cluster's tile
    const int rows = ksplit > 1 ? BM / ksplit : BM, rb = ksplit > 1 ? split * rows : 0;
    const uint32_t smb = (uint32_t)__cvta_generic_to_shared(sm);
    const bool v4 = VEC && (n & 3) == 0;
    auto total = [&](int r, int c, float* f) {            // four columns of the tile's sum, times alpha
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ksplit > 1) {
            for (int q = 0; q < ksplit; q++) {            // in rank order
                uint32_t ad;
                float4 v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ad) : "r"(smb + (r * RP + c) * 4), "r"(q));
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ad) : "memory");
                t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
            }
        } else {
#pragma unroll
            for (int q = 0; q < KG; q++) {
                const float4 v = *reinterpret_cast<const float4*>(sm + q * BM * RP + r * RP + c);
                t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
            }
        }
        f[0] = alpha * t.x; f[1] = alpha * t.y; f[2] = alpha * t.z; f[3] = alpha * t.w;
    };
    auto put = [&](float* dst, long long idx, int gj, const float* f) {
        if (v4) *reinterpret_cast<float4*>(dst + idx) = make_float4(f[0], f[1], f[2], f[3]);
        else for (int q = 0; q < 4 && gj + q < n; q++) dst[idx + q] = f[q];
    };
    auto get = [&](const float* src, long long idx, int gj, float* f) {
        if (v4) { const float4 v = *reinterpret_cast<const float4*>(src + idx); f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
        else for (int q = 0; q < 4; q++) f[q] = gj + q < n ? src[idx + q] : 0.f;
    };
    for (int e = threadIdx.x; e < rows * (W / 4); e += TH) {
        const int r = rb + e / (W / 4), c = e % (W / 4) * 4;
        const int gi = i0 + r, gj = j0 + c;
        float f[4];
        total(r, c, f);
        if constexpr (EPI == F32_SWIGLU) {
            float u[4], h[4];
            total(r, c + W, u);
            if (gi >= m || gj >= n) continue;
            const long long idx = (long long)gi * n + gj;
#pragma unroll
            for (int q = 0; q < 4; q++) h[q] = f[q] / (1.f + expf(-f[q])) * u[q];
            put(a.C[0], idx, gj, f); put(a.C[1], idx, gj, u); put(a.C[2], idx, gj, h);
        } else {
            if (gi >= m || gj >= n) continue;
            const long long idx = (long long)gi * n + gj;
            float d[4];
            if constexpr (EPI == F32_SWB) {
                float x[4], o[4];
                get(a.G, idx, gj, x); get(a.U, idx, gj, d);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float sig = 1.f / (1.f + expf(-x[q]));
                    o[q] = f[q] * d[q] * (sig * (1.f + x[q] * (1.f - sig)));
                    f[q] *= x[q] * sig;
                }
                put(a.C[0], idx, gj, o); put(a.C[1], idx, gj, f);
            } else {
                if (beta != 0.f) {
                    get(D, idx, gj, d);
#pragma unroll
                    for (int q = 0; q < 4; q++) f[q] += beta * d[q];
                }
                put(C, idx, gj, f);
            }
        }
    }
    if (ksplit > 1)                                       // nobody's shared memory goes away while a peer reads it
        cluster_sync();
}

template <int BM, int BN, int BK, int KG, int TM, int TN, int ST, bool A_MN, bool B_KM, bool VEC, int EPI, bool ONE>
static int f32_launch(const F32Group& a, int m, int batch, long long sa, long long sb, long long sc, int ksplit, float alpha, float beta, cudaStream_t st) {
    using L = F32Tile<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM>;
    constexpr int W = EPI == F32_SWIGLU ? BN / 2 : BN;
    auto kern = k_gemm_f32<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM, VEC, EPI, ONE>;
    static const cudaError_t attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (attr != cudaSuccess) return 125;
    int cols = 0;
    for (int g = 0; g < a.nprob; g++) cols += (a.n[g] + W - 1) / W;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cols * ksplit, (m + BM - 1) / BM, batch);
    if (cfg.gridDim.y > 65535 || cfg.gridDim.z > 65535) return 123;
    cfg.blockDim = dim3(L::THREADS); cfg.dynamicSmemBytes = L::SMEM; cfg.stream = st;
    cudaLaunchAttribute at[2];
    int na = 0;
    if (ksplit > 1) {
        at[na].id = cudaLaunchAttributeClusterDimension;
        at[na].val.clusterDim.x = ksplit; at[na].val.clusterDim.y = 1; at[na].val.clusterDim.z = 1;
        na++;
    }
    if (ax_gemm_pdl()) {
        at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg.attrs = at; cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, kern, a, m, sa, sb, sc, ksplit, alpha, beta) == cudaSuccess ? 0 : 126;
}
// How a launch is cut: tile, sums of a thread (rows), CTAs that share a tile's depth.  By the tiles that it would have, the 64-deep steps of its sums and whether rows are whole
// 16-byte pieces.
struct F32Cut { int rows, cols, sums, ctas; };
static F32Cut f32_cut(int tb, bool plain, long long t128, long long t64, long long t64x32, long long t32, int steps, long long depth, bool vec) {
    // A 128 x 128 tile has the most FMAs per shared-memory read, but fewer than 148 of them leave SMs without work, and so does a last round that is mostly empty (one CTA
    // to an SM; us there / with 64 x 64 tiles: 171 tiles, 1072 x 2360 x 944 238 / 160, 189 tiles, 2688 x 1152 x 376 85 / 71; 210 tiles, 1760 x 1848 x 112 28.2 / 28.7).
    // Rows that are no whole 16-byte pieces are copied by 4 bytes, once for each tile that reads them, which is all there is to a product of one step (2111 x 2267 x 12 16.9 / 22.6) and counts
    // most where both operands have short rows (A B^T: 1032 x 2085 x 13 11.5 / 16.4, 1675 x 1370 x 33 22.6 / 28.7, 2426 x 975 x 103 44.9 / 48.5, 1679 x 1771 x 237 87 / 94; but 1235 x 2108 x 701 234 / 219).
    if (t128 >= AX_SMS && (10 * t128 >= 7 * AX_SMS * ((t128 + AX_SMS - 1) / AX_SMS) || (!vec && depth <= (tb == 1 ? 256 : 20)))) return {128, 128, 8, 1};
    // Shallow products of many tiles are set-up, one load and the stores: 64 x 64 tiles of 4 x 4 sums with 32-deep steps, which leave an SM room for more CTAs.  us there / with 64 x 64
    // tiles of 8 x 8 sums or 32 x 32: 2232 x 368 x 24 4.8 / 6.9, 680 x 2792 x 32 7.9 / 10.0, 1184 x 960 x 24 5.8 / 9.2, 1968 x 912 x 16 8.2 / 10.7; A B^T 1992 x 1072 x 136 25.8 / 31.5,
    // 1552 x 1176 x 104 21.2 / 25.5; but 1008 x 656 x 40 7.2 / 6.3.
    if (plain && t64 >= AX_SMS && (depth <= 32 || (tb == 1 && steps <= 3 && t64 >= 2 * AX_SMS))) return {64, 64, 4, 1};
    // By 4-byte copies the 8 x 8 sums wait for their operands, 8 x 8 / 4 x 4: A B 1547 x 664 x 34 13.0 / 9.0, 1549 x 1025 x 73 26.9 / 18.6, 1453 x 1051 x 173 44.7 / 32.0; A B^T of 296 to 443 tiles
    // 1.07 / 0.96 of the time with 4 x 4 sums and no second depth group, of more 0.87 / 0.96; A^T B of 222 to 443 0.77 / 0.96, of more, 1455 x 1377 x 37, 15.2 / 14.8, 1146 x 1651 x 112 33.0 / 25.8.
    if (plain && !vec && (tb == 0 ? 2 * t64 >= 3 * AX_SMS : tb == 1 ? t64 >= 2 * AX_SMS && t64 < 3 * AX_SMS : t64 >= 3 * AX_SMS)) return {64, 64, 4, 1};
    // With 4 x 4 sums four CTAs fit an SM, with 8 x 8 two, whose second round of 1.5 to 2 then takes longer than all at once while the depth is short, 8 x 8 / 4 x 4: A^T B 1740 x 1188 x 76 19.0 / 15.1,
    // 2612 x 864 x 148 28.0 / 23.1, A B 2228 x 1012 x 140 27.5 / 24.4, A B^T 2636 x 856 x 328 61.7 / 50.7; but A^T B 2044 x 1004 x 764 93 / 97, and 364 tiles 12.2 / 14.9.
    if (plain && vec && t64 >= 3 * AX_SMS && t64 <= 4 * AX_SMS && steps <= 5) return {64, 64, 4, 1};
    if (t64 >= 2 * AX_SMS) return {64, 64, 8, 1};
    // Three steps of 32 are over before two of 64 where tiles are enough: A B 2732 x 316 x 88 8.9 / 10.6 on 32 x 32, A B^T 2392 x 444 x 92 12.2 / 14.6; but A B^T 300 x 1996 x 84, 160 tiles, 11.5 / 9.6.
    if (plain && vec && tb != 2 && depth > 64 && depth <= 96 && 4 * t64 >= 5 * AX_SMS) return {64, 64, 4, 1};
    // Below, a launch is the latency of its steps: 64 x 32 tiles (8 x 4 sums to a thread, 43 % of the FMA pipe with two CTAs on an SM, which is what
    // fits) with the depth cut over a cluster as far as two CTAs for each SM.  Where that leaves a third of the SMs idle or most with one CTA and some with two,
    // or takes a second round, 32 x 32 tiles spread better; a product of two steps is over before a larger tile pays.  us, 64 x 32 with 1 / 2 / 4 CTAs to a tile |
    // 32 x 32 alike: 512 x 256 x 256 8.6 / 7.9 / 6.2 | 8.8 / 7.6 / 10.1, 512 x 512 x 256 11.0 / 8.4 / 11.9 | 10.0 / 12.0 / 14.9, 512 x 256 x 688 21.1 / 16.4 / 10.8 | 20.2 / 14.8 /
    // 15.3, 512 x 1024 x 256 12.2 / 17.1 / 24.3 | 14.4 / 19.2 / 26.5, 512 x 688 x 256 12.2 / 16.6 / 18.2 | 10.8 / 12.9 / 20.3, 256 x 256 x 128 4.6 / 5.0 / 5.8 | 3.6 / 4.9 / 5.3,
    // 300 x 128 x 344 10.0 / 7.4 / 7.6 | 6.9 / 6.6 / 7.3; 1024 x 1536 x 512 58 | 60 and with 64 x 64 tiles of 8 x 8 sums 50.
    // Not where 64-row tiles are much larger than their rows (32 x 1656 x 144 5.8 / 7.1 | 4.4, 16 x 2208 x 320 7.9 / 9.2 / 7.9 | 5.8 / 6.0), where the steps do not go evenly into the
    // CTAs (704 x 192 x 176, 2 + 1 steps, 7.5 | 5.1; 856 x 142 x 348, 2 + 2 + 2 + 0, 11.7 | 14.0 / 10.6), nor for shared tiles of A B by 4-byte copies (215 x 569 x 2021 - / - / 47.9 | - / 37.3).
    int ks = 1, ks32 = 1;
    while (ks < 8 && t64x32 * ks * 2 <= 2 * AX_SMS && steps >= 2 * ks) ks *= 2;
    while (ks32 < 8 && t32 * ks32 * 2 <= AX_SMS * 5 / 2 && steps >= 4 * ks32) ks32 *= 2;
    // 70 clusters of four and 32 of eight run at once, a further one is a second round: 533 x 228 x 841, 72 of four, 27.7 us, 19.6 on 32 x 32; 220 x 258 x 958, 36 of eight, 18.1 and 13.1.
    const long long ctas = t64x32 * ks;
    const bool fit = ks < 4 || t64x32 <= (ks == 4 ? 70 : 32);
    if (fit && steps > 2 && 3 * ctas > 2 * AX_SMS && ctas <= 2 * AX_SMS && (ctas <= AX_SMS || 2 * ctas > 3 * AX_SMS) && 40 * t64x32 <= (ks > ks32 ? 28 : 23) * t32 &&
        (steps + ks - 1) / ks * ks * 100 <= steps * 127 && (vec || ks == 1 || tb)) return {64, 32, 8, ks};
    // 4-byte copies count for each CTA that reads a tile of an operand: 64 x 64 tiles from one for each SM on (1964 x 456 x 3179 296 | 385 us, 2196 x 412 x 402 41 | 58, 270 x 2271 x 220 25.0 | 28.2, 1115 x 687 x 51 9.4 | 11.0).
    if (plain && !vec && tb != 2 && (depth > 64 || tb == 0) && t64 >= AX_SMS) return {64, 64, 4, 1};
    return {32, 32, 4, ks32};
}
static int cut_code(const F32Cut& c) { return c.rows << 20 | c.cols << 8 | c.sums << 4 | c.ctas; }
int ax_f32_cut = 0;
// of one product of `batch`
int ax_gemm_f32_cut(int tb, int m, int n, int k, int batch, int aligned) {
    auto tiles = [&](int bm, int bn) { return (long long)((m + bm - 1) / bm) * ((n + bn - 1) / bn) * batch; };
    const bool vec = aligned && (tb != 2 || m % 4 == 0) && n % 4 == 0 && (tb == 2 || k % 4 == 0);
    return cut_code(f32_cut(tb, true, tiles(128, 128), tiles(64, 64), tiles(64, 32), tiles(32, 32), (k + 63) / 64, k, vec));
}

template <bool A_MN, bool B_KM, int EPI = F32_PLAIN, bool ONE = false>
static int f32_gemm(const F32Group& a, int m, int batch, long long sa, long long sb, long long sc, float alpha, float beta, cudaStream_t st) {
    // 16-byte copies need row pitches and starts on 16-byte boundaries
    bool vec = sa % 4 == 0 && sb % 4 == 0 && sc % 4 == 0 && (!A_MN || m % 4 == 0) && aligned16(a.D) && aligned16(a.G) && aligned16(a.U);
    for (const float* c : a.C) vec = vec && aligned16(c);
    for (int g = 0; g < a.nprob; g++) {
        vec = vec && a.n[g] % 4 == 0;
        for (const F32Seg* q = a.seg + g * a.nseg; q < a.seg + (g + 1) * a.nseg; q++)
            vec = vec && ((A_MN && !B_KM) || q->k % 4 == 0) && aligned16(q->A) && aligned16(q->B) && aligned16(q->B2);
    }
    auto tiles = [&](int bm, int bn) {
        long long cols = 0;
        const int w = EPI == F32_SWIGLU ? bn / 2 : bn;
        for (int g = 0; g < a.nprob; g++) cols += (a.n[g] + w - 1) / w;
        return (long long)((m + bm - 1) / bm) * cols * batch;
    };
#define F32L(BM, BN, BK, KG, TM, TN, ST, KSP)                                                                                  \
    (vec ? f32_launch<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM, true, EPI, ONE>(a, m, batch, sa, sb, sc, KSP, alpha, beta, st)        \
         : f32_launch<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM, false, EPI, ONE>(a, m, batch, sa, sb, sc, KSP, alpha, beta, st))
    int steps = 0;
    long long depth = 0;
    for (int q = 0; q < a.nseg; q++) { steps += (a.seg[q].k + 63) / 64; depth += a.seg[q].k; }
    const F32Cut c = f32_cut(A_MN ? 2 : B_KM, EPI == F32_PLAIN, tiles(128, 128), tiles(64, 64), tiles(64, 32), tiles(32, 32), steps, depth, vec);
    ax_f32_cut = cut_code(c);
    if (c.rows == 128) return F32L(128, 128, 16, 1, 8, 8, 3, 1);
    if constexpr (EPI == F32_PLAIN)
        if (c.cols == 64 && c.sums == 4) return F32L(64, 64, 32, 1, 4, 4, 3, 1);
    if (c.cols == 64) return F32L(64, 64, 32, 2, 8, 8, 4, 1);
    if (c.rows == 64) return F32L(64, 32, 64, 4, 8, 4, 3, c.ctas);
    return F32L(32, 32, 64, 4, 4, 4, 4, c.ctas);
#undef F32L
}

// Arguments as ax_gemm_tc2_group, fp32 operands and outputs (mode 0: one product).  -1: not for this kernel.
int ax_gemm_f32_group(int tb, int mode, int count, const void* const* A, const void* const* B, void* const* C, const int* m, const int* n,
                      const int* k, float alpha, const void* D, float beta, const void* swb_g, const void* swb_u, void* swb_du, cudaStream_t st) {
    if (count < 1 || count > (mode == 2 ? 6 : 3) || m[0] < 1 || (mode != 1 && mode != 2 && mode != 4) || (D && mode != 2) || (swb_g && (mode != 2 || tb != 1 || D))) return -1;
    F32Group a = {};
    a.nprob = mode == 1 ? count : 1;
    a.nseg = mode == 2 ? count : 1;
    auto f = [](const void* p) { return (const float*)p; };
    for (int g = 0; g < a.nprob; g++) { a.n[g] = n[g]; a.C[g] = (float*)C[g]; if (n[g] < 1) return -1; }
    for (int g = 0; g < (mode == 4 ? 1 : count); g++) {
        a.seg[g] = {f(A[mode == 2 ? g : 0]), f(B[g]), nullptr, k[mode == 2 ? g : 0]};
        if (a.seg[g].k < 1) return -1;
    }
    a.D = beta != 0.f ? f(D) : nullptr;
    if (!a.D) beta = 0.f;
    if (mode == 4) {
        if (tb != 0 || count != 2) return -1;
        a.seg[0].B2 = f(B[1]);
        a.C[1] = (float*)C[1]; a.C[2] = (float*)C[2];
        return f32_gemm<false, false, F32_SWIGLU>(a, m[0], 1, 0, 0, 0, alpha, 0.f, st);
    }
    if (swb_g) {
        a.G = f(swb_g); a.U = f(swb_u); a.C[1] = (float*)swb_du;
        return f32_gemm<false, true, F32_SWB>(a, m[0], 1, 0, 0, 0, alpha, 0.f, st);
    }
    if (tb == 0) return f32_gemm<false, false>(a, m[0], 1, 0, 0, 0, alpha, beta, st);
    if (tb == 1) return f32_gemm<false, true>(a, m[0], 1, 0, 0, 0, alpha, beta, st);
    return f32_gemm<true, false>(a, m[0], 1, 0, 0, 0, alpha, beta, st);
}

int ax_gemm_simt(int in_bf16, int out_bf16, int tb, const void* A, const void* B, void* C, const void* D,
                 int m, int n, int k, int batch, long long sa, long long sb, long long sc,
                 float alpha, float beta, cudaStream_t st) {
    if (m <= 0 || n <= 0) return 0;
    if (batch < 1) batch = 1;
    long long as_m, as_k, bs_k, bs_n;
    if (tb == 0) { as_m = k; as_k = 1; bs_k = n; bs_n = 1; }
    else if (tb == 1) { as_m = k; as_k = 1; bs_k = 1; bs_n = k; }
    else { as_m = 1; as_k = m; bs_k = n; bs_n = 1; }
    if (beta != 0.f && !D) D = C;
    if (!in_bf16 && !out_bf16) {
        F32Group a = {};
        a.seg[0] = {(const float*)A, (const float*)B, nullptr, k};
        a.nprob = a.nseg = 1; a.n[0] = n; a.C[0] = (float*)C; a.D = beta != 0.f ? (const float*)D : nullptr;
        if (tb == 0) return f32_gemm<false, false, F32_PLAIN, true>(a, m, batch, sa, sb, sc, alpha, beta, st);
        if (tb == 1) return f32_gemm<false, true, F32_PLAIN, true>(a, m, batch, sa, sb, sc, alpha, beta, st);
        return f32_gemm<true, false, F32_PLAIN, true>(a, m, batch, sa, sb, sc, alpha, beta, st);
    }
    dim3 grid((n + GT - 1) / GT, (m + GT - 1) / GT, batch);
    if (grid.y > 65535 || grid.z > 65535) return 123;
    if (in_bf16 && out_bf16)
        k_gemm_simt<bf16, bf16><<<grid, 256, 0, st>>>((const bf16*)A, (const bf16*)B, (bf16*)C, (const bf16*)D, m, n, k, as_m, as_k, bs_k, bs_n, sa, sb, sc, alpha, beta);
    else if (in_bf16)
        k_gemm_simt<bf16, float><<<grid, 256, 0, st>>>((const bf16*)A, (const bf16*)B, (float*)C, (const float*)D, m, n, k, as_m, as_k, bs_k, bs_n, sa, sb, sc, alpha, beta);
    else
        return 124;
    return 0;
}
