// Causal grouped-query attention in bf16 with the probabilities held to 32-bit accuracy, for the shapes that the tcgen05
// kernels do not take (attn_tc.cu, attn_tc128.cu: whole 128-token tiles of head_dim 64 and 128; attn_tcs.cu: other lengths and head
// dims from 40 to 64, where there is work for all SMs and the line in that file says so): [B,T,H,DH] layout, DH a multiple of 8 up to 128, any T.
//
// The products that take P and dS as an operand need them in bf16, and eight bits are not what fp32 arithmetic on CUDA cores
// (attn_simt.cu) gives.  Here every P and dS enters as the sum of two bf16 numbers, hi = rn(x) and lo = rn(x - hi), in two MMAs
// with one accumulator: 16 bits and a sign, an error of at most 2^-17 of the element where the bf16 result is rounded at up to 2^-8.  Against
// float64 (T 200 to 2433, DH 32 to 128, N(0,1) inputs) the 2-norm errors are those of the CUDA-core kernels to 0.1 % either way,
// 1.57e-3 to 1.67e-3 for o and dv and 1.72e-3 to 1.90e-3 for dq and dk; with P and dS in one bf16 number o is at 1.92e-3 to
// 1.97e-3.  Under one per cent of the results round the other way.  No atomics, sums in a fixed order: the same bits on every run.
//
// A warp owns 16 rows (queries, or keys in the dK / dV kernel) and walks the other operand in steps of 32 rows; P and dS stay in
// registers, where the accumulator layout of one mma.sync is the operand layout of the next.  On tcgen05
// a tile of 64 columns is half empty for heads up to 32.  Heads above 64 have no such kernel yet: dV and dK of 128 columns and two S^T and dP^T of 64 each
// would fill TMEM, with K and V read from shared memory by the score products.  Bound by issue and by MMA latency: the MMA pipe (555 TFLOP/s by itself) is busy 49 / 57 / 52 % of the active cycles in
// the forward, dQ and dK / dV kernels (B2 H16 KV16 T1500 DH128: 119, 143 and 214 us), and the schedulers issue in 43 / 36 / 33 % of them (exponentials, splits,
// operand reads).  Times in us, forward / backward with the row dots,
// CUDA cores -> here (for comparison: tcgen05 with 8-bit P and dS; the first two and their like now run on attn_tcs.cu):
//   B3 H24 KV8 T1000 DH64    628 / 2080 ->  70 / 203   (31 / 77)      B4 H24 KV8 T500 DH64   247 / 790 ->  33 / 102   (21 / 51)
//   B2 H16 KV16 T1500 DH128 1439 / 3580 -> 122 / 347   (39 / 118)     B2 H8 KV4 T256 DH32    31.6 / 95 -> 11.2 / 22   (10.4 / 28)
#include "common.cuh"
#include "kernels.h"

#define MA_WARPS 4
#define MA_ROWS (MA_WARPS * 16)      // rows of a CTA, and rows of a shared-memory tile of the walked operand
#define MA_TH (MA_WARPS * 32)
#define MA_SUB 32                    // rows of the walked operand per step

__device__ __forceinline__ uint32_t ma_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ma_ld4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ma_ld4t(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ma_mma(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void ma_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void ma_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <bool B> struct MaFlag { __device__ constexpr operator bool() const { return B; } };

// A tile is MA_ROWS rows of DHP bf16; the 16-byte pieces of a row are exchanged by its number so that the eight rows of an
// ldmatrix fall in different banks.
template <int DHP> struct MaTile {
    static constexpr int BYTES = MA_ROWS * DHP * 2;
    static __device__ __forceinline__ uint32_t at(int row, int ch) {
        const int x = DHP == 32 ? (row >> 1) & 3 : row & 7;
        return row * DHP * 2 + ((ch ^ x) << 4);
    }
};
// MA_ROWS rows from r0 of a [T, DH] window with row stride `stride`; rows past T and columns past DH are zeros
template <int DHP, int TH = MA_TH>
__device__ __forceinline__ void ma_load(uint32_t dst, const bf16* src, long long stride, int r0, int T, int DH) {
    constexpr int CH = DHP / 8;
#pragma unroll
    for (int i = 0; i < MA_ROWS * CH / TH; i++) {
        const int e = threadIdx.x + i * TH, r = e / CH, ch = e % CH;
        const bool ok = r0 + r < T && ch * 8 < DH;
        const bf16* p = ok ? src + (long long)(r0 + r) * stride + ch * 8 : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + MaTile<DHP>::at(r, ch)), "l"(p), "r"(ok ? 16 : 0) : "memory");
    }
}
// operand fragments of one 16-wide step along the head dimension: 16 rows as A, 32 rows as B (four groups of eight)
template <int DHP> __device__ __forceinline__ void ma_a(uint32_t tile, int row0, int kk, uint32_t* a) {
    const int lane = threadIdx.x & 31;
    ma_ld4(tile + MaTile<DHP>::at(row0 + (lane & 15), kk * 2 + (lane >> 4)), a);
}
template <int DHP> __device__ __forceinline__ void ma_b(uint32_t tile, int row0, int kk, uint32_t (*b)[2]) {
    const int lane = threadIdx.x & 31, q = lane >> 3;
#pragma unroll
    for (int f = 0; f < 4; f += 2) {
        uint32_t r[4];
        ma_ld4(tile + MaTile<DHP>::at(row0 + f * 8 + (lane & 7) + ((q >> 1) << 3), kk * 2 + (q & 1)), r);
        b[f][0] = r[0]; b[f][1] = r[1]; b[f + 1][0] = r[2]; b[f + 1][1] = r[3];
    }
}
// s[16 rows of A, 32 rows of B] += A B^T over the head dimension
template <int DHP> __device__ __forceinline__ void ma_scores(uint32_t ta, int ra, uint32_t tb, int rb, float (*s)[4]) {
#pragma unroll
    for (int kk = 0; kk < DHP / 16; kk++) {
        uint32_t a[4], b[4][2];
        ma_a<DHP>(ta, ra, kk, a);
        ma_b<DHP>(tb, rb, kk, b);
#pragma unroll
        for (int j = 0; j < 4; j++) ma_mma(s[j], a, b[j]);
    }
}
__device__ __forceinline__ void ma_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 f = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - f.x, y - f.y);
    hi = reinterpret_cast<const uint32_t&>(h); lo = reinterpret_cast<const uint32_t&>(l);
}
// acc[16 rows, DHP] += p[16 rows, 32] * tile[row0 .. row0 + 31, DHP], p as hi + lo; the two MMAs of an accumulator stand
// eight (head_dim 32: four) apart
template <int DHP> __device__ __forceinline__ void ma_accumulate(const float (*p)[4], uint32_t tile, int row0, float (*acc)[4]) {
    constexpr int G = DHP < 64 ? DHP / 8 : 8;
    const int lane = threadIdx.x & 31, q = lane >> 3;
#pragma unroll
    for (int s = 0; s < 2; s++) {
        uint32_t hi[4], lo[4];
        ma_split(p[2 * s][0], p[2 * s][1], hi[0], lo[0]);
        ma_split(p[2 * s][2], p[2 * s][3], hi[1], lo[1]);
        ma_split(p[2 * s + 1][0], p[2 * s + 1][1], hi[2], lo[2]);
        ma_split(p[2 * s + 1][2], p[2 * s + 1][3], hi[3], lo[3]);
#pragma unroll
        for (int f0 = 0; f0 < DHP / 8; f0 += G) {
            uint32_t r[G / 2][4];
#pragma unroll
            for (int f = 0; f < G; f += 2) ma_ld4t(tile + MaTile<DHP>::at(row0 + s * 16 + (lane & 7) + ((q & 1) << 3), f0 + f + (q >> 1)), r[f / 2]);
#pragma unroll
            for (int f = 0; f < G; f++) ma_mma(acc[f0 + f], lo, r[f / 2] + (f & 1) * 2);
#pragma unroll
            for (int f = 0; f < G; f++) ma_mma(acc[f0 + f], hi, r[f / 2] + (f & 1) * 2);
        }
    }
}
// rows t and t + 8 of a warp's 16-row result
template <int DHP> __device__ __forceinline__ void ma_store(bf16* base, long long stride, int t, int T, int DH, const float (*acc)[4], float f0, float f1) {
    const int c = (threadIdx.x & 3) * 2;
#pragma unroll
    for (int f = 0; f < DHP / 8; f++) {
        if (f * 8 >= DH) break;
        if (t < T) *reinterpret_cast<__nv_bfloat162*>(base + t * stride + f * 8 + c) = __floats2bfloat162_rn(acc[f][0] * f0, acc[f][1] * f0);
        if (t + 8 < T) *reinterpret_cast<__nv_bfloat162*>(base + (t + 8) * stride + f * 8 + c) = __floats2bfloat162_rn(acc[f][2] * f1, acc[f][3] * f1);
    }
}

// The inverse rotary on rows t and t + 8 before they are rounded (head_dim DHP, tables fp32 [T, DHP / 2]): a pair's columns are DHP / 2
// apart, in one thread; out1 = g1 c + g2 s, out2 = -g1 s + g2 c
template <int DHP> __device__ __forceinline__ void ma_unrotate(float (*acc)[4], int t, int T, const float* __restrict__ cs, const float* __restrict__ sn) {
    constexpr int G = DHP / 16;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (t + r * 8 >= T) continue;
        const long long row = (long long)(t + r * 8) * (DHP / 2) + (threadIdx.x & 3) * 2;
#pragma unroll
        for (int f = 0; f < G; f++) {
            const float2 c = *reinterpret_cast<const float2*>(cs + row + f * 8), s = *reinterpret_cast<const float2*>(sn + row + f * 8);
            float& x0 = acc[f][r * 2]; float& x1 = acc[f][r * 2 + 1];
            float& y0 = acc[f + G][r * 2]; float& y1 = acc[f + G][r * 2 + 1];
            const float a0 = x0, a1 = x1;
            x0 = a0 * c.x + y0 * s.x; x1 = a1 * c.y + y1 * s.y;
            y0 = y0 * c.x - a0 * s.x; y1 = y1 * c.y - a1 * s.y;
        }
    }
}

#define MA_LOG2E 1.4426950408889634f
#define MA_LN2 0.6931471805599453f

// grid (H * B, query tiles): the longest rows first
template <int DHP>
__global__ void __launch_bounds__(MA_TH, DHP == 128 ? 2 : 3)
k_attn_fwd_mma(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v, bf16* __restrict__ o,
               float* __restrict__ lse, const AttnShape s) {
    extern __shared__ __align__(128) uint8_t ma_buf[];
    constexpr int TB = MaTile<DHP>::BYTES;
    const uint32_t Qs = ma_smem(ma_buf), Ks = Qs + TB, Vs = Ks + 2 * TB;       // K and V: two tiles each
    const int b = blockIdx.x / s.H, h = blockIdx.x % s.H, g = h / (s.H / s.KV);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = (gridDim.y - 1 - blockIdx.y) * MA_ROWS, t0 = r0 + warp * 16;
    const bf16* kb = k + b * s.kb + g * s.kh;
    const bf16* vb = v + b * s.kb + g * s.kh;
    const float c = s.scale * MA_LOG2E;                                        // scores and maxima in units of ln 2
    pdl_enter();
    ma_load<DHP>(Qs, q + b * s.qb + h * s.qh, s.qt, r0, s.T, s.DH);
    ma_load<DHP>(Ks, kb, s.kt, 0, s.T, s.DH);
    ma_load<DHP>(Vs, vb, s.kt, 0, s.T, s.DH);
    ma_commit();
    float acc[DHP / 8][4] = {}, m[2] = {-3.0e38f, -3.0e38f}, l[2] = {0.f, 0.f};       // l: this thread's share of the row sum
    const int ntiles = (min(r0 + MA_ROWS, s.T) - 1) / MA_ROWS + 1;
    for (int kt = 0; kt < ntiles; kt++) {
        ma_wait();
        __syncthreads();
        const uint32_t Kt = Ks + (kt & 1) * TB, Vt = Vs + (kt & 1) * TB;
        if (kt + 1 < ntiles) {
            ma_load<DHP>(Ks + (~kt & 1) * TB, kb, s.kt, (kt + 1) * MA_ROWS, s.T, s.DH);
            ma_load<DHP>(Vs + (~kt & 1) * TB, vb, s.kt, (kt + 1) * MA_ROWS, s.T, s.DH);
        }
        ma_commit();
#pragma unroll 1
        for (int sub = 0; sub < MA_ROWS; sub += MA_SUB) {
            const int k0 = kt * MA_ROWS + sub;
            if (k0 > t0 + 15) break;
            float sc[4][4] = {};
            ma_scores<DHP>(Qs, warp * 16, Kt, sub, sc);
            // a step that meets the diagonal masks its keys; one in front of it has none to mask
            auto softmax = [&](auto masked) {
                float corr[2];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int last = t0 + (lane >> 2) + r * 8 - k0 - (lane & 3) * 2;       // j * 8 + e of the row's own key
                    float mx = -3.0e38f;
#pragma unroll
                    for (int j = 0; j < 4; j++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            float& x = sc[j][r * 2 + e];
                            x = !masked || j * 8 + e <= last ? x * c : -3.0e38f;
                            mx = fmaxf(mx, x);
                        }
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    const float mn = fmaxf(m[r], mx);
                    corr[r] = exp2f(m[r] - mn);
                    m[r] = mn;
                    l[r] *= corr[r];
#pragma unroll
                    for (int j = 0; j < 4; j++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            float& x = sc[j][r * 2 + e];
                            x = !masked || j * 8 + e <= last ? exp2f(x - mn) : 0.f;
                            l[r] += x;
                        }
                }
                if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f))
#pragma unroll
                    for (int f = 0; f < DHP / 8; f++) { acc[f][0] *= corr[0]; acc[f][1] *= corr[0]; acc[f][2] *= corr[1]; acc[f][3] *= corr[1]; }
            };
            if (k0 + MA_SUB - 1 > t0) softmax(MaFlag<true>()); else softmax(MaFlag<false>());
            ma_accumulate<DHP>(sc, Vt, sub, acc);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        const int t = t0 + (lane >> 2) + r * 8;
        if (lse && t < s.T && (lane & 3) == 0) lse[((long long)b * s.H + h) * s.T + t] = m[r] * MA_LN2 + logf(l[r]);
    }
    ma_store<DHP>(o + b * s.qb + h * s.qh, s.qt, t0 + (lane >> 2), s.T, s.DH, acc, 1.f / l[0], 1.f / l[1]);
}

// dQ: a warp owns 16 queries and walks their keys.  grid as the forward
template <int DHP>
__global__ void __launch_bounds__(MA_TH, DHP == 128 ? 2 : 3)
k_attn_bwd_dq_mma(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v, const bf16* __restrict__ dO,
                  const float* __restrict__ lse, const float* __restrict__ Dv, bf16* __restrict__ dq, const AttnShape s,
                  const float* __restrict__ rope_cos, const float* __restrict__ rope_sin) {
    extern __shared__ __align__(128) uint8_t ma_buf[];
    constexpr int TB = MaTile<DHP>::BYTES;
    const uint32_t Qs = ma_smem(ma_buf), Gs = Qs + TB, Ks = Gs + TB, Vs = Ks + 2 * TB;
    const int b = blockIdx.x / s.H, h = blockIdx.x % s.H, g = h / (s.H / s.KV);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = (gridDim.y - 1 - blockIdx.y) * MA_ROWS, t0 = r0 + warp * 16;
    const bf16* kb = k + b * s.kb + g * s.kh;
    const bf16* vb = v + b * s.kb + g * s.kh;
    const float c = s.scale * MA_LOG2E;
    pdl_enter();
    ma_load<DHP>(Qs, q + b * s.qb + h * s.qh, s.qt, r0, s.T, s.DH);
    ma_load<DHP>(Gs, dO + b * s.qb + h * s.qh, s.qt, r0, s.T, s.DH);
    ma_load<DHP>(Ks, kb, s.kt, 0, s.T, s.DH);
    ma_load<DHP>(Vs, vb, s.kt, 0, s.T, s.DH);
    ma_commit();
    float L[2], D[2], acc[DHP / 8][4] = {};
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int t = t0 + (lane >> 2) + r * 8;
        L[r] = t < s.T ? lse[((long long)b * s.H + h) * s.T + t] * MA_LOG2E : 0.f;
        D[r] = t < s.T ? Dv[b * s.db + h * s.dh_ + t * s.dtk] : 0.f;
    }
    const int ntiles = (min(r0 + MA_ROWS, s.T) - 1) / MA_ROWS + 1;
    for (int kt = 0; kt < ntiles; kt++) {
        ma_wait();
        __syncthreads();
        const uint32_t Kt = Ks + (kt & 1) * TB, Vt = Vs + (kt & 1) * TB;
        if (kt + 1 < ntiles) {
            ma_load<DHP>(Ks + (~kt & 1) * TB, kb, s.kt, (kt + 1) * MA_ROWS, s.T, s.DH);
            ma_load<DHP>(Vs + (~kt & 1) * TB, vb, s.kt, (kt + 1) * MA_ROWS, s.T, s.DH);
        }
        ma_commit();
#pragma unroll 1
        for (int sub = 0; sub < MA_ROWS; sub += MA_SUB) {
            const int k0 = kt * MA_ROWS + sub;
            if (k0 > t0 + 15) break;
            float sc[4][4] = {}, dp[4][4] = {};
            ma_scores<DHP>(Qs, warp * 16, Kt, sub, sc);
            ma_scores<DHP>(Gs, warp * 16, Vt, sub, dp);
            auto grad = [&](auto masked) {
                const int last = t0 + (lane >> 2) - k0 - (lane & 3) * 2;
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float x = exp2f(fmaf(sc[j][e], c, -L[e >> 1])) * (dp[j][e] - D[e >> 1]);
                        sc[j][e] = !masked || j * 8 + (e & 1) <= last + (e >> 1) * 8 ? x : 0.f;
                    }
            };
            if (k0 + MA_SUB - 1 > t0) grad(MaFlag<true>()); else grad(MaFlag<false>());
            ma_accumulate<DHP>(sc, Kt, sub, acc);
        }
    }
    if (rope_cos) ma_unrotate<DHP>(acc, t0 + (lane >> 2), s.T, rope_cos, rope_sin);
    ma_store<DHP>(dq + b * s.qb + h * s.qh, s.qt, t0 + (lane >> 2), s.T, s.DH, acc, s.scale, s.scale);
}

// dK, dV: 16 keys of a kv head belong to two warps, which walk the group's query heads and their causal query tiles in order, each
// one half of a tile, and add their sums at the end — this is where the sum over the group happens.  The first key tiles meet the
// most queries and their chain is as long as the kernel: that is why it is two warps, and why a cluster of S CTAs takes the query
// tiles of a key tile in turn where one chain would outlast an even share of the work (see the launch).  The cluster's sums meet
// through distributed shared memory in rank order; half 0 finishes dK, half 1 dV.  grid (KV * B * S, key tiles).
// Queries past T need no mask: their Q and dO rows, lse and D are zeros, P is 1 and meets zeros, dS is zero.
#define MA_KV_TH (2 * MA_TH)
template <int DHP>
__global__ void __launch_bounds__(MA_KV_TH, DHP == 128 ? 1 : 2)
k_attn_bwd_dkv_mma(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v, const bf16* __restrict__ dO,
                   const float* __restrict__ lse, const float* __restrict__ Dv, bf16* __restrict__ dk, bf16* __restrict__ dv, const AttnShape s, int S,
                   const float* __restrict__ rope_cos, const float* __restrict__ rope_sin) {
    extern __shared__ __align__(128) uint8_t ma_buf[];
    constexpr int TB = MaTile<DHP>::BYTES;
    const uint32_t Ks = ma_smem(ma_buf), Vs = Ks + TB, Qs = Vs + TB, Gs = Qs + 2 * TB;
    float* stat = reinterpret_cast<float*>(ma_buf + 6 * TB);        // two tiles of lse, then of D
    const int part = blockIdx.x % S, gb = blockIdx.x / S, b = gb / s.KV, g = gb % s.KV, rep = s.H / s.KV;
    const int warp = (threadIdx.x >> 5) & (MA_WARPS - 1), half = threadIdx.x / MA_TH, lane = threadIdx.x & 31;
    const int r0 = blockIdx.y * MA_ROWS, j0 = r0 + warp * 16;
    const int qt0 = blockIdx.y, nq = gridDim.y - qt0, n_it = (rep * nq - part + S - 1) / S;       // this CTA: tiles part, part + S, ...
    const float c = s.scale * MA_LOG2E;
    auto load = [&](int it) {
        const int all = part + it * S, h = g * rep + all / nq, t = (qt0 + all % nq) * MA_ROWS;
        const long long hb = b * s.qb + h * s.qh;
        ma_load<DHP, MA_KV_TH>(Qs + (it & 1) * TB, q + hb, s.qt, t, s.T, s.DH);
        ma_load<DHP, MA_KV_TH>(Gs + (it & 1) * TB, dO + hb, s.qt, t, s.T, s.DH);
        if (threadIdx.x < 2 * MA_ROWS) {
            const int i = threadIdx.x % MA_ROWS, second = threadIdx.x / MA_ROWS;
            const bool ok = t + i < s.T;
            const float* p = second ? Dv + b * s.db + h * s.dh_ + (ok ? (t + i) * s.dtk : 0) : lse + ((long long)b * s.H + h) * s.T + (ok ? t + i : 0);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(ma_smem(stat + (second * 2 + (it & 1)) * MA_ROWS + i)), "l"(p), "r"(ok ? 4 : 0) : "memory");
        }
    };
    pdl_enter();
    ma_load<DHP, MA_KV_TH>(Ks, k + b * s.kb + g * s.kh, s.kt, r0, s.T, s.DH);
    ma_load<DHP, MA_KV_TH>(Vs, v + b * s.kb + g * s.kh, s.kt, r0, s.T, s.DH);
    if (n_it > 0) load(0);
    ma_commit();
    float ak[DHP / 8][4] = {}, av[DHP / 8][4] = {};
    for (int it = 0; it < n_it; it++) {
        ma_wait();
        __syncthreads();
        if (it + 1 < n_it) load(it + 1);
        ma_commit();
        const uint32_t Qt = Qs + (it & 1) * TB, Gt = Gs + (it & 1) * TB;
        const int sub = half * MA_SUB, q0 = (qt0 + (part + it * S) % nq) * MA_ROWS + sub;
        if (q0 + MA_SUB - 1 < j0 || q0 >= s.T) continue;
        const float* Ls = stat + (it & 1) * MA_ROWS + sub + (lane & 3) * 2;
        float sc[4][4] = {}, dp[4][4] = {};
        ma_scores<DHP>(Ks, warp * 16, Qt, sub, sc);
        ma_scores<DHP>(Vs, warp * 16, Gt, sub, dp);
        auto grad = [&](auto masked) {
            const int first = j0 + (lane >> 2) - q0 - (lane & 3) * 2;        // j * 8 + e of the key's own query
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 L = *reinterpret_cast<const float2*>(Ls + j * 8), D = *reinterpret_cast<const float2*>(Ls + 2 * MA_ROWS + j * 8);
                const float l2[2] = {L.x * MA_LOG2E, L.y * MA_LOG2E};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float p = exp2f(fmaf(sc[j][e], c, -l2[e & 1]));
                    sc[j][e] = !masked || j * 8 + (e & 1) >= first + (e >> 1) * 8 ? p : 0.f;
                    dp[j][e] = sc[j][e] * (dp[j][e] - ((e & 1) ? D.y : D.x));
                }
            }
        };
        if (q0 < j0 + 15) grad(MaFlag<true>()); else grad(MaFlag<false>());
        ma_accumulate<DHP>(sc, Gt, sub, av);
        ma_accumulate<DHP>(dp, Qt, sub, ak);
    }
    // the second half's sums through the ring's memory
    ma_wait();
    __syncthreads();
    float* xch = reinterpret_cast<float*>(ma_buf + 2 * TB) + (threadIdx.x & (MA_TH - 1));
    if (half) {
#pragma unroll
        for (int i = 0; i < DHP / 2; i++) { xch[i * MA_TH] = ak[i >> 2][i & 3]; xch[(DHP / 2 + i) * MA_TH] = av[i >> 2][i & 3]; }
    }
    __syncthreads();
    if (!half)
#pragma unroll
        for (int i = 0; i < DHP / 2; i++) { ak[i >> 2][i & 3] += xch[i * MA_TH]; av[i >> 2][i & 3] += xch[(DHP / 2 + i) * MA_TH]; }
    if (S > 1) {
        if (!half)                                          // a thread's own places again
#pragma unroll
            for (int i = 0; i < DHP / 2; i++) { xch[i * MA_TH] = ak[i >> 2][i & 3]; xch[(DHP / 2 + i) * MA_TH] = av[i >> 2][i & 3]; }
        cluster_sync();
        constexpr int HG = DHP / 16;                        // column groups of a half head; group f and f + HG are rotary pairs
        const uint32_t base = ma_smem(xch + half * (DHP / 2) * MA_TH);
        bf16* dst = (half ? dv : dk) + b * s.kb + g * s.kh;
        const int t0 = j0 + (lane >> 2), c2 = (lane & 3) * 2;
        const float fac = half ? 1.f : s.scale;
        for (int f = part * HG / S; f < (part + 1) * HG / S; f++) {
            float v[2][4] = {};
            for (int q = 0; q < S; q++)
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    float x;
                    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.f32 %0, [ra];\n\t}"
                                 : "=f"(x) : "r"(base + (((f + (e >> 2) * HG) * 4 + (e & 3)) * MA_TH) * 4), "r"(q) : "memory");
                    v[e >> 2][e & 3] += x;
                }
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int t = t0 + r * 8;
                if (t >= s.T) continue;
                float x0 = v[0][r * 2], x1 = v[0][r * 2 + 1], y0 = v[1][r * 2], y1 = v[1][r * 2 + 1];
                if (!half && rope_cos) {
                    const long long row = (long long)t * (DHP / 2) + f * 8 + c2;
                    const float2 cs = *reinterpret_cast<const float2*>(rope_cos + row), sn = *reinterpret_cast<const float2*>(rope_sin + row);
                    const float a0 = x0, a1 = x1;
                    x0 = a0 * cs.x + y0 * sn.x; x1 = a1 * cs.y + y1 * sn.y;
                    y0 = y0 * cs.x - a0 * sn.x; y1 = y1 * cs.y - a1 * sn.y;
                }
                bf16* o = dst + t * s.kt + f * 8 + c2;
                if (f * 8 < s.DH) *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(x0 * fac, x1 * fac);
                if ((f + HG) * 8 < s.DH) *reinterpret_cast<__nv_bfloat162*>(o + HG * 8) = __floats2bfloat162_rn(y0 * fac, y1 * fac);
            }
        }
        cluster_sync();   // peers have read
        return;
    }
    if (half) return;
    if (rope_cos) ma_unrotate<DHP>(ak, j0 + (lane >> 2), s.T, rope_cos, rope_sin);
    ma_store<DHP>(dk + b * s.kb + g * s.kh, s.kt, j0 + (lane >> 2), s.T, s.DH, ak, s.scale, s.scale);
    ma_store<DHP>(dv + b * s.kb + g * s.kh, s.kt, j0 + (lane >> 2), s.T, s.DH, av, 1.f, 1.f);
}

template <int DHP> static constexpr int ma_fwd_smem() { return 5 * MaTile<DHP>::BYTES; }
template <int DHP> static constexpr int ma_bwd_smem() { return 6 * MaTile<DHP>::BYTES + 4 * MA_ROWS * 4; }

template <int DHP> static int ma_attr() {
    int rc = (int)cudaFuncSetAttribute(k_attn_fwd_mma<DHP>, cudaFuncAttributeMaxDynamicSharedMemorySize, ma_fwd_smem<DHP>());
    rc |= (int)cudaFuncSetAttribute(k_attn_bwd_dq_mma<DHP>, cudaFuncAttributeMaxDynamicSharedMemorySize, ma_bwd_smem<DHP>());
    return rc | (int)cudaFuncSetAttribute(k_attn_bwd_dkv_mma<DHP>, cudaFuncAttributeMaxDynamicSharedMemorySize, ma_bwd_smem<DHP>());
}
int ax_attn_mma_init(void) { return ma_attr<32>() | ma_attr<64>() | ma_attr<128>(); }

// bf16 on the [B,T,H,DH] layout; the 16-byte copies need DH % 8 == 0 and aligned bases
static bool ma_served(const AttnShape& s) {
    return s.DH >= 8 && s.DH <= 128 && s.DH % 8 == 0 && s.B >= 1 && s.T >= 1 && s.KV >= 1 && s.H % s.KV == 0 && (long long)s.H * s.B * 4 <= 0x7fffffff && s.T <= 65535 * MA_ROWS &&
           s.qh == s.DH && s.kh == s.DH && s.qt == (long long)s.H * s.DH && s.kt == (long long)s.KV * s.DH;
}

int ax_attn_fwd_mma(const void* q, const void* k, const void* v, void* o, float* lse, const AttnShape& s, cudaStream_t st) {
    if (!ma_served(s) || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) return -1;
    const dim3 grid(s.H * s.B, (s.T + MA_ROWS - 1) / MA_ROWS);
    ax_variant = 0x82;
    auto go = [&](auto kern, int smem) {
        return ax_launch_chain(kern, grid, dim3(MA_TH), smem, st, (const bf16*)q, (const bf16*)k, (const bf16*)v, (bf16*)o, lse, s) == cudaSuccess ? 0 : 3;
    };
    if (s.DH <= 32) return go(k_attn_fwd_mma<32>, ma_fwd_smem<32>());
    if (s.DH <= 64) return go(k_attn_fwd_mma<64>, ma_fwd_smem<64>());
    return go(k_attn_fwd_mma<128>, ma_fwd_smem<128>());
}
int ax_attn_bwd_mma(const void* q, const void* k, const void* v, const void* dO, const float* lse, const float* Dv,
                    void* dq, void* dk, void* dv, const AttnShape& s, const float* rope_cos, const float* rope_sin, cudaStream_t st) {
    if (rope_cos && ((s.DH != 32 && s.DH != 64 && s.DH != 128) || !rope_sin || !aligned16(rope_cos) || !aligned16(rope_sin))) return -1;
    if (!ma_served(s) || !lse || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(dO) || !aligned16(dq) || !aligned16(dk) || !aligned16(dv)) return -1;
    const int tiles = (s.T + MA_ROWS - 1) / MA_ROWS;
    const dim3 gq(s.H * s.B, tiles);
    // dK / dV: the first key tile walks all query tiles of the group's heads, `chain` of them; an even share of the whole triangle over
    // the CTAs that fit the GPU (two per SM, one at head_dim above 64) is `share`.  A chain longer than that is cut over a
    // cluster of two or four.  Whole backward in us without / with clusters: B1 H12 KV4 T2500 DH64 392 / 225, B2 H16 KV4 T700 DH96
    // 181 / 118, B3 H24 KV8 T1000 DH64 240 / 203, B4 H24 KV8 T500 DH64 120 / 102, B8 H24 KV8 T320 DH64 90 / 85, B2 H8 KV4 T256 DH32 25.2 / 21.5.
    const long long chain = (long long)(s.H / s.KV) * tiles, share = (long long)s.H * s.B * tiles * (tiles + 1) / 2 / (AX_SMS * (s.DH > 64 ? 1 : 2));
    int S = 1;
    while (S < (s.DH <= 32 ? 2 : 4) && S * 2 <= chain && chain > S * share) S *= 2;
    ax_variant = 0x83 + 0x100 * S;
    auto go = [&](auto kq, auto kk, int smem) {
        if (ax_launch_chain(kq, gq, dim3(MA_TH), smem, st, (const bf16*)q, (const bf16*)k, (const bf16*)v, (const bf16*)dO, lse, Dv, (bf16*)dq, s, rope_cos, rope_sin) != cudaSuccess) return 3;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(s.KV * s.B * S, tiles); cfg.blockDim = dim3(MA_KV_TH); cfg.dynamicSmemBytes = smem; cfg.stream = st;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at; cfg.numAttrs = ax_gemm_pdl() ? 2 : 1;
        return cudaLaunchKernelEx(&cfg, kk, (const bf16*)q, (const bf16*)k, (const bf16*)v, (const bf16*)dO, lse, Dv, (bf16*)dk, (bf16*)dv, s, S,
                                  rope_cos, rope_sin) == cudaSuccess ? 0 : 3;
    };
    if (s.DH <= 32) return go(k_attn_bwd_dq_mma<32>, k_attn_bwd_dkv_mma<32>, ma_bwd_smem<32>());
    if (s.DH <= 64) return go(k_attn_bwd_dq_mma<64>, k_attn_bwd_dkv_mma<64>, ma_bwd_smem<64>());
    return go(k_attn_bwd_dq_mma<128>, k_attn_bwd_dkv_mma<128>, ma_bwd_smem<128>());
}
