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
//   * small tiles (32 x 32) cut every step among four groups of 64 threads;
//   * where the tiles still leave SMs idle, a cluster of 2, 4 or 8 CTAs cuts the depth once more and adds its partial
//     tiles through distributed shared memory.
// 512 x 256 x 256, one cold launch: 46 us with 64 x 64 tiles, 16-deep steps and no prefetch, 7 us now; 512 x 512 x 256: 11 us.
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
template <int BM, int BN, int BK, int KG, int TM, int TN, int ST, bool A_MN, bool B_KM, bool VEC>
__global__ void __launch_bounds__(KG * (BM / TM) * (BN / TN))
k_gemm_f32(const float* __restrict__ A, const float* __restrict__ B, float* C, const float* D, int m, int n, int k,
           long long sa, long long sb, long long sc, int ksplit, float alpha, float beta) {
    using L = F32Tile<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM>;
    constexpr int TH = L::THREADS, TX = BN / TN, TY = BM / TM, GT_ = TX * TY, KS = BK / KG;
    extern __shared__ __align__(16) float sm[];
    pdl_enter();
    const int bz = blockIdx.z;
    A += (long long)bz * sa; B += (long long)bz * sb; C += (long long)bz * sc;
    if (D) D += (long long)bz * sc;
    const int split = blockIdx.x % ksplit, i0 = blockIdx.y * BM, j0 = (blockIdx.x / ksplit) * BN;
    const int steps_all = (k + BK - 1) / BK, per = (steps_all + ksplit - 1) / ksplit;
    const int s0 = split * per, s1 = min(steps_all, s0 + per), steps = max(s1 - s0, 0);
    const int grp = threadIdx.x / GT_, tid = threadIdx.x % GT_, ty = tid / TX, tx = tid % TX;
    auto load = [&](int st) {
        float* as = sm + (st % ST) * (L::A_EL + L::B_EL);
        float* bs = as + L::A_EL;
        const int k0 = (s0 + st) * BK;
        if (A_MN) tile_cp<BK, BM, L::AP, VEC, TH>(as, A, m, k0, i0, k, m);
        else tile_cp<BM, BK, L::AP, VEC, TH>(as, A, k, i0, k0, m, k);
        if (B_KM) tile_cp<BN, BK, L::BP, VEC, TH>(bs, B, k, j0, k0, n, k);
        else tile_cp<BK, BN, L::BP, VEC, TH>(bs, B, n, k0, j0, k, n);
    };
    float acc[TM][TN];
#pragma unroll
    for (int p = 0; p < TM; p++)
#pragma unroll
        for (int q = 0; q < TN; q++) acc[p][q] = 0.f;
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
        if (st + ST - 1 < steps) load(st + ST - 1);
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
        for (int q = 0; q < TN; q++) red[row_of(p) * RP + col_of(q)] = acc[p][q];
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
    for (int e = threadIdx.x; e < rows * (BN / 4); e += TH) {
        const int r = rb + e / (BN / 4), c = e % (BN / 4) * 4;
        const int gi = i0 + r, gj = j0 + c;
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
            for (int g = 0; g < KG; g++) {
                const float4 v = *reinterpret_cast<const float4*>(sm + g * BM * RP + r * RP + c);
                t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
            }
        }
        if (gi >= m || gj >= n) continue;
        const long long idx = (long long)gi * n + gj;
        float f[4] = {alpha * t.x, alpha * t.y, alpha * t.z, alpha * t.w};
        if (v4) {
            if (beta != 0.f) {
                const float4 d = *reinterpret_cast<const float4*>(D + idx);
                f[0] += beta * d.x; f[1] += beta * d.y; f[2] += beta * d.z; f[3] += beta * d.w;
            }
            *reinterpret_cast<float4*>(C + idx) = make_float4(f[0], f[1], f[2], f[3]);
        } else {
            for (int q = 0; q < 4 && gj + q < n; q++) {
                if (beta != 0.f) f[q] += beta * D[idx + q];
                C[idx + q] = f[q];
            }
        }
    }
    if (ksplit > 1)                                       // nobody's shared memory goes away while a peer reads it
        cluster_sync();
}

template <int BM, int BN, int BK, int KG, int TM, int TN, int ST, bool A_MN, bool B_KM, bool VEC>
static int f32_launch(const float* A, const float* B, float* C, const float* D, int m, int n, int k, int batch,
                      long long sa, long long sb, long long sc, int ksplit, float alpha, float beta, cudaStream_t st) {
    using L = F32Tile<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM>;
    auto kern = k_gemm_f32<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM, VEC>;
    static const cudaError_t attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (attr != cudaSuccess) return 125;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((n + BN - 1) / BN * ksplit, (m + BM - 1) / BM, batch);
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
    return cudaLaunchKernelEx(&cfg, kern, A, B, C, D, m, n, k, sa, sb, sc, ksplit, alpha, beta) == cudaSuccess ? 0 : 126;
}
template <bool A_MN, bool B_KM>
static int f32_gemm(const float* A, const float* B, float* C, const float* D, int m, int n, int k, int batch,
                    long long sa, long long sb, long long sc, float alpha, float beta, cudaStream_t st) {
    // 16-byte copies need row pitches and starts on 16-byte boundaries
    const bool vec = (A_MN ? m : k) % 4 == 0 && (B_KM ? k : n) % 4 == 0 && n % 4 == 0 && aligned16(A) && aligned16(B) && aligned16(C) &&
                     (!D || aligned16(D)) && sa % 4 == 0 && sb % 4 == 0 && sc % 4 == 0;
    auto tiles = [&](int bm, int bn) { return (long long)((m + bm - 1) / bm) * ((n + bn - 1) / bn) * batch; };
#define F32L(BM, BN, BK, KG, TM, TN, ST, KSP)                                                                                        \
    (vec ? f32_launch<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM, true>(A, B, C, D, m, n, k, batch, sa, sb, sc, KSP, alpha, beta, st)    \
         : f32_launch<BM, BN, BK, KG, TM, TN, ST, A_MN, B_KM, false>(A, B, C, D, m, n, k, batch, sa, sb, sc, KSP, alpha, beta, st))
    // the largest tile that still gives every SM one: a 128 x 128 tile has twice the FMAs per shared-memory read of a
    // 64 x 64 one, but fewer than 148 of them leave SMs without work
    if (tiles(128, 128) >= AX_SMS) return F32L(128, 128, 16, 1, 8, 8, 3, 1);
    if (tiles(64, 64) >= AX_SMS) return F32L(64, 64, 32, 1, 4, 4, 3, 1);
    // 32 x 32 tiles; a cluster splits the depth while CTAs are fewer than SMs and every CTA keeps two steps of 64
    int ks = 1;
    while (ks < 8 && tiles(32, 32) * ks * 2 <= AX_SMS * 2 && (k + 63) / 64 >= 4 * ks) ks *= 2;
    return F32L(32, 32, 64, 4, 4, 4, 4, ks);
#undef F32L
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
        const float* a = (const float*)A; const float* b = (const float*)B;
        float* c = (float*)C; const float* d = beta != 0.f ? (const float*)D : nullptr;
        if (tb == 0) return f32_gemm<false, false>(a, b, c, d, m, n, k, batch, sa, sb, sc, alpha, beta, st);
        if (tb == 1) return f32_gemm<false, true>(a, b, c, d, m, n, k, batch, sa, sb, sc, alpha, beta, st);
        return f32_gemm<true, false>(a, b, c, d, m, n, k, batch, sa, sb, sc, alpha, beta, st);
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
