// Causal grouped-query attention on CUDA cores with exact fp32 arithmetic —
// the general path (any head_dim <= 256, any T, any strides) for shapes that neither the
// tensor-core kernels nor attn_f32.cu (fp32 storage, head dims 12 to 64) take.  Layout is
// given by element strides, so [B,H,T,DH] and [B,T,H,DH] are both served.
// No atomics: dK/dV are accumulated per key row over the whole query group.
//
// Bound by shared-memory reads and, at the sizes of the parity mode (a few
// hundred tokens), by latency.  A warp owns AR = 4 rows (queries, or keys in
// the dK/dV kernel) and a lane one row of the other tile: a 16-byte read of the
// lane's row and four broadcast reads feed 16 FMAs, and the four probabilities
// of a lane go back to the warp as one 16-byte piece.  Tiles of the walked operand
// are double-buffered (cp.async for fp32), so the next tile's load runs under
// this one's arithmetic.  B2 H8 KV4 T256 DH32 fp32, one cold launch: forward 64 -> 23 us,
// dQ 65 -> 23 us, dK/dV 115 -> 54 us against one row per warp and scalar reads; with the walk cut over clusters 21, 17 and 22.
#include <initializer_list>

#include "common.cuh"
#include "kernels.h"

#define AW 8            // warps per block
#define AR 4            // rows per warp
#define ABLK (AW * AR)  // rows per block
#define AKT 32          // rows of the other operand per shared-memory tile (one per lane)
#define ATH (AW * 32)

// floats from row to row of a tile: whole 16-byte pieces, an odd number of them so that 8 lanes reading the same column of 8
// consecutive rows touch all 32 banks once
__host__ __device__ __forceinline__ int attn_ld(int dh) {
    const int d4 = (dh + 3) / 4 * 4;
    return d4 % 8 == 4 ? d4 : d4 + 4;
}

// AKT rows starting at r0 (row stride `stride` elements) -> dst [AKT][LD] as fp32; rows past T_ and the columns up to the next
// multiple of four are zeros.  vec: 16-byte (fp32) / 8-byte (bf16) accesses are aligned.
__device__ __forceinline__ void attn_tile(float* dst, const float* src, long long stride, int r0, int T_, int DH, int LD, int vec) {
    const int q4 = (DH + 3) / 4;
    for (int e = threadIdx.x; e < AKT * q4; e += ATH) {
        const int r = e / q4, d = (e - r * q4) * 4;
        const bool in = r0 + r < T_;
        const float* p = in ? src + (long long)(r0 + r) * stride + d : src;
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst + r * LD + d);
        if (vec) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(p), "r"(in ? 16 : 0) : "memory");
        else
            for (int q = 0; q < 4; q++) {
                const bool ok = in && d + q < DH;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(a + q * 4), "l"(ok ? p + q : src), "r"(ok ? 4 : 0) : "memory");
            }
    }
}
__device__ __forceinline__ void attn_tile(float* dst, const bf16* src, long long stride, int r0, int T_, int DH, int LD, int vec) {
    const int q4 = (DH + 3) / 4;
    for (int e = threadIdx.x; e < AKT * q4; e += ATH) {
        const int r = e / q4, d = (e - r * q4) * 4;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (r0 + r < T_) {
            const bf16* p = src + (long long)(r0 + r) * stride + d;
            if (vec) {
                const uint2 v = *reinterpret_cast<const uint2*>(p);
                f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
                f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
            } else
                for (int q = 0; q < 4; q++) if (d + q < DH) f[q] = __bfloat162float(p[q]);
        }
        *reinterpret_cast<float4*>(dst + r * LD + d) = make_float4(f[0], f[1], f[2], f[3]);
    }
}
__device__ __forceinline__ void attn_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void attn_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// out[r] = <rows[r], col> over q4 16-byte pieces
__device__ __forceinline__ void attn_dot(const float* rows, const float* col, int LD, int q4, float* out) {
#pragma unroll
    for (int r = 0; r < AR; r++) out[r] = 0.f;
    for (int d = 0; d < q4; d++) {
        const float4 k = *reinterpret_cast<const float4*>(col + d * 4);
#pragma unroll
        for (int r = 0; r < AR; r++) {
            const float4 q = *reinterpret_cast<const float4*>(rows + r * LD + d * 4);
            out[r] = fmaf(q.x, k.x, out[r]); out[r] = fmaf(q.y, k.y, out[r]);
            out[r] = fmaf(q.z, k.z, out[r]); out[r] = fmaf(q.w, k.w, out[r]);
        }
    }
}
// acc[r][i] += w[j].r * tile[j][lane + 32 i] over the AKT rows of the tile
template <int NJ>
__device__ __forceinline__ void attn_axpy(float (&acc)[AR][NJ], const float* w, const float* tile, int LD, int DH, int lane) {
#pragma unroll 4
    for (int j = 0; j < AKT; j++) {
        const float4 p = *reinterpret_cast<const float4*>(w + j * 4);
#pragma unroll
        for (int i = 0; i < NJ; i++) {
            const int d = lane + 32 * i;
            const float v = d < DH ? tile[j * LD + d] : 0.f;
            acc[0][i] = fmaf(p.x, v, acc[0][i]); acc[1][i] = fmaf(p.y, v, acc[1][i]);
            acc[2][i] = fmaf(p.z, v, acc[2][i]); acc[3][i] = fmaf(p.w, v, acc[3][i]);
        }
    }
}

// Where rows are few, a cluster of S CTAs takes the tiles that a block of rows walks in turn, and the sums meet through distributed
// shared memory: a unit is a warp's row of accumulators, [unit][i][thread], and each CTA finishes 1 / S of the units, in rank order.
// Kernels of their own (SHARE): with S as a value, walks that nobody shares took up to 20 % longer (B1 H8 KV8 T900 DH256,
// forward and backward: 1350 us so, 1650).
__device__ __forceinline__ float attn_peer(const float* p, int rank) {
    float x;
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.f32 %0, [ra];\n\t}"
                 : "=f"(x) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank) : "memory");
    return x;
}

template <typename T, int NJ, bool SHARE>
__global__ void __launch_bounds__(ATH)
k_attn_fwd_simt(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ o,
                float* __restrict__ lse, AttnShape s, int vec, int ctas) {
    extern __shared__ __align__(16) float smem[];
    const int DH = s.DH, LD = attn_ld(DH), q4 = (DH + 3) / 4, TILE = AKT * LD;
    float* Ks = smem;                    // two tiles each
    float* Vs = Ks + 2 * TILE;
    float* Qs = Vs + 2 * TILE;           // the block's rows
    float* Ps = Qs + TILE;               // [warp][key][AR]
    const int b = blockIdx.z, h = blockIdx.y, g = h / (s.H / s.KV);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = SHARE ? ctas : 1, part = SHARE ? blockIdx.x % S : 0, r0 = (gridDim.x / S - 1 - blockIdx.x / S) * ABLK, t0 = r0 + warp * AR;      // the longest rows first
    const T* kbase = k + b * s.kb + g * s.kh;
    const T* vbase = v + b * s.kb + g * s.kh;
    const int ntiles = min(r0 + ABLK - 1, s.T - 1) / AKT + 1;
    pdl_enter();
    attn_tile(Qs, q + b * s.qb + h * s.qh, s.qt, r0, s.T, DH, LD, vec);
    if (!SHARE || part < ntiles) {
        attn_tile(Ks, kbase, s.kt, part * AKT, s.T, DH, LD, vec);
        attn_tile(Vs, vbase, s.kt, part * AKT, s.T, DH, LD, vec);
    }
    attn_commit();
    float m[AR], l[AR], acc[AR][NJ];     // l: this lane's share of the row sum
#pragma unroll
    for (int r = 0; r < AR; r++) {
        m[r] = -3.0e38f; l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < NJ; i++) acc[r][i] = 0.f;
    }
    const float* myQ = Qs + warp * AR * LD;
    float* myP = Ps + warp * AKT * AR;
    for (int kt = part, it = 0; kt < ntiles; kt += S, it++) {
        attn_wait();
        __syncthreads();
        const int cur = it & 1, nxt = cur ^ 1;
        if (kt + S < ntiles) {
            attn_tile(Ks + nxt * TILE, kbase, s.kt, (kt + S) * AKT, s.T, DH, LD, vec);
            attn_tile(Vs + nxt * TILE, vbase, s.kt, (kt + S) * AKT, s.T, DH, LD, vec);
        }
        attn_commit();
        if (kt * AKT > t0 + AR - 1) continue;
        const int key = kt * AKT + lane;
        float sc[AR], p[AR];
        attn_dot(myQ, Ks + cur * TILE + lane * LD, LD, q4, sc);
#pragma unroll
        for (int r = 0; r < AR; r++) {
            const bool on = key <= t0 + r;
            sc[r] = on ? sc[r] * s.scale : -3.0e38f;
            const float mn = fmaxf(m[r], warp_max(sc[r]));
            p[r] = on ? expf(sc[r] - mn) : 0.f;
            const float corr = expf(m[r] - mn);
            l[r] = l[r] * corr + p[r];
            m[r] = mn;
#pragma unroll
            for (int i = 0; i < NJ; i++) acc[r][i] *= corr;
        }
        *reinterpret_cast<float4*>(myP + lane * AR) = make_float4(p[0], p[1], p[2], p[3]);
        __syncwarp();
        attn_axpy<NJ>(acc, myP, Vs + cur * TILE, LD, DH, lane);
        __syncwarp();
    }
    if (SHARE) {                         // merge: sums at the largest of the ranks' maxima
        attn_wait();
        __syncthreads();
        float* acc_x = smem + threadIdx.x;
        float* ml_x = smem + AR * NJ * ATH + warp * AR * 2;
#pragma unroll
        for (int r = 0; r < AR; r++) {
            const float ls = warp_sum(l[r]);
            if (lane == 0) { ml_x[r * 2] = m[r]; ml_x[r * 2 + 1] = ls; }
#pragma unroll
            for (int i = 0; i < NJ; i++) acc_x[(r * NJ + i) * ATH] = acc[r][i];
        }
        cluster_sync();
        for (int r = part * AR / S; r < (part + 1) * AR / S; r++) {
            const int t = t0 + r;
            if (t >= s.T) continue;
            float mx = -3.0e38f, ls = 0.f, a[NJ];
            for (int q = 0; q < S; q++) mx = fmaxf(mx, attn_peer(ml_x + r * 2, q));
#pragma unroll
            for (int i = 0; i < NJ; i++) a[i] = 0.f;
            for (int q = 0; q < S; q++) {
                const float f = expf(attn_peer(ml_x + r * 2, q) - mx);
                ls += attn_peer(ml_x + r * 2 + 1, q) * f;
#pragma unroll
                for (int i = 0; i < NJ; i++) a[i] += attn_peer(acc_x + (r * NJ + i) * ATH, q) * f;
            }
            T* orow = o + b * s.qb + h * s.qh + (long long)t * s.qt;
            const float il = 1.f / ls;
#pragma unroll
            for (int i = 0; i < NJ; i++)
                if (lane + 32 * i < DH) stf(orow, lane + 32 * i, a[i] * il);
            if (lse && lane == 0) lse[((long long)b * s.H + h) * s.T + t] = mx + logf(ls);
        }
        cluster_sync();             // peers have read
        return;
    }
#pragma unroll
    for (int r = 0; r < AR; r++) {
        const int t = t0 + r;
        const float ls = warp_sum(l[r]);
        if (t >= s.T) continue;
        T* orow = o + b * s.qb + h * s.qh + (long long)t * s.qt;
        const float il = 1.f / ls;
#pragma unroll
        for (int i = 0; i < NJ; i++) {
            const int d = lane + 32 * i;
            if (d < DH) stf(orow, d, acc[r][i] * il);
        }
        if (lse && lane == 0) lse[((long long)b * s.H + h) * s.T + t] = m[r] + logf(ls);
    }
}

// dQ: a warp owns AR query rows and walks the keys.
template <typename T, typename TO, int NJ, bool SHARE>
__global__ void __launch_bounds__(ATH)
k_attn_bwd_dq_simt(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                   const T* __restrict__ dO, const float* __restrict__ lse, const float* __restrict__ Dv,
                   TO* __restrict__ dq, AttnShape s, int vec, int ctas) {
    extern __shared__ __align__(16) float smem[];
    const int DH = s.DH, LD = attn_ld(DH), q4 = (DH + 3) / 4, TILE = AKT * LD;
    float* Ks = smem;
    float* Vs = Ks + 2 * TILE;
    float* Qs = Vs + 2 * TILE;
    float* Gs = Qs + TILE;               // dO rows
    float* Ps = Gs + TILE;
    const int b = blockIdx.z, h = blockIdx.y, g = h / (s.H / s.KV);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = SHARE ? ctas : 1, part = SHARE ? blockIdx.x % S : 0, r0 = (gridDim.x / S - 1 - blockIdx.x / S) * ABLK, t0 = r0 + warp * AR;
    const T* kbase = k + b * s.kb + g * s.kh;
    const T* vbase = v + b * s.kb + g * s.kh;
    pdl_enter();
    attn_tile(Qs, q + b * s.qb + h * s.qh, s.qt, r0, s.T, DH, LD, vec);
    attn_tile(Gs, dO + b * s.qb + h * s.qh, s.qt, r0, s.T, DH, LD, vec);
    const int ntiles = min(r0 + ABLK - 1, s.T - 1) / AKT + 1;
    if (!SHARE || part < ntiles) {
        attn_tile(Ks, kbase, s.kt, part * AKT, s.T, DH, LD, vec);
        attn_tile(Vs, vbase, s.kt, part * AKT, s.T, DH, LD, vec);
    }
    attn_commit();
    float L[AR], Dr[AR], acc[AR][NJ];
#pragma unroll
    for (int r = 0; r < AR; r++) {
        const int t = t0 + r;
        L[r] = t < s.T ? lse[((long long)b * s.H + h) * s.T + t] : 0.f;
        Dr[r] = t < s.T ? Dv[b * s.db + h * s.dh_ + (long long)t * s.dtk] : 0.f;
#pragma unroll
        for (int i = 0; i < NJ; i++) acc[r][i] = 0.f;
    }
    const float* myQ = Qs + warp * AR * LD;
    const float* myG = Gs + warp * AR * LD;
    float* myP = Ps + warp * AKT * AR;
    for (int kt = part, it = 0; kt < ntiles; kt += S, it++) {
        attn_wait();
        __syncthreads();
        const int cur = it & 1, nxt = cur ^ 1;
        if (kt + S < ntiles) {
            attn_tile(Ks + nxt * TILE, kbase, s.kt, (kt + S) * AKT, s.T, DH, LD, vec);
            attn_tile(Vs + nxt * TILE, vbase, s.kt, (kt + S) * AKT, s.T, DH, LD, vec);
        }
        attn_commit();
        if (kt * AKT > t0 + AR - 1) continue;
        const int key = kt * AKT + lane;
        float sc[AR], dp[AR], ds[AR];
        attn_dot(myQ, Ks + cur * TILE + lane * LD, LD, q4, sc);
        attn_dot(myG, Vs + cur * TILE + lane * LD, LD, q4, dp);
#pragma unroll
        for (int r = 0; r < AR; r++)
            ds[r] = key <= t0 + r && t0 + r < s.T ? expf(sc[r] * s.scale - L[r]) * (dp[r] - Dr[r]) * s.scale : 0.f;
        *reinterpret_cast<float4*>(myP + lane * AR) = make_float4(ds[0], ds[1], ds[2], ds[3]);
        __syncwarp();
        attn_axpy<NJ>(acc, myP, Ks + cur * TILE, LD, DH, lane);
        __syncwarp();
    }
    if (SHARE) {
        attn_wait();
        __syncthreads();
        float* acc_x = smem + threadIdx.x;
#pragma unroll
        for (int r = 0; r < AR; r++)
#pragma unroll
            for (int i = 0; i < NJ; i++) acc_x[(r * NJ + i) * ATH] = acc[r][i];
        cluster_sync();
        for (int r = part * AR / S; r < (part + 1) * AR / S; r++) {
            const int t = t0 + r;
            if (t >= s.T) continue;
            const long long roff = b * s.qb + h * s.qh + (long long)t * s.qt;
#pragma unroll
            for (int i = 0; i < NJ; i++) {
                float a = 0.f;
                for (int q = 0; q < S; q++) a += attn_peer(acc_x + (r * NJ + i) * ATH, q);
                if (lane + 32 * i < DH) stf(dq, roff + lane + 32 * i, a);
            }
        }
        cluster_sync();             // peers have read
        return;
    }
#pragma unroll
    for (int r = 0; r < AR; r++) {
        const int t = t0 + r;
        if (t >= s.T) continue;
        const long long roff = b * s.qb + h * s.qh + (long long)t * s.qt;
#pragma unroll
        for (int i = 0; i < NJ; i++) {
            const int d = lane + 32 * i;
            if (d < DH) stf(dq, roff + d, acc[r][i]);
        }
    }
}

// dK, dV: a warp owns AR key rows of a kv head and walks the group's query heads and their causal query tiles — this is
// where the GQA sum happens.
template <typename T, typename TO, int NJ, bool SHARE>
__global__ void __launch_bounds__(ATH)
k_attn_bwd_dkv_simt(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                    const T* __restrict__ dO, const float* __restrict__ lse, const float* __restrict__ Dv,
                    TO* __restrict__ dk, TO* __restrict__ dv, AttnShape s, int vec, int ctas) {
    extern __shared__ __align__(16) float smem[];
    const int DH = s.DH, LD = attn_ld(DH), q4 = (DH + 3) / 4, TILE = AKT * LD;
    float* Qs = smem;                    // two tiles each
    float* Gs = Qs + 2 * TILE;
    float* Kr = Gs + 2 * TILE;           // the block's rows
    float* Vr = Kr + TILE;
    float* Ps = Vr + TILE;               // [warp][query][AR]
    const int b = blockIdx.z, g = blockIdx.y, rep = s.H / s.KV;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = SHARE ? ctas : 1, part = SHARE ? blockIdx.x % S : 0, r0 = blockIdx.x / S * ABLK, j0 = r0 + warp * AR;       // the first key rows meet the most queries
    const int qt0 = r0 / AKT, nq = (s.T + AKT - 1) / AKT - qt0, n_it = rep * nq;
    pdl_enter();
    attn_tile(Kr, k + b * s.kb + g * s.kh, s.kt, r0, s.T, DH, LD, vec);
    attn_tile(Vr, v + b * s.kb + g * s.kh, s.kt, r0, s.T, DH, LD, vec);
    auto load = [&](int it, int cur) {
        const long long hb = b * s.qb + (long long)(g * rep + it / nq) * s.qh;
        const int t = (qt0 + it % nq) * AKT;
        attn_tile(Qs + cur * TILE, q + hb, s.qt, t, s.T, DH, LD, vec);
        attn_tile(Gs + cur * TILE, dO + hb, s.qt, t, s.T, DH, LD, vec);
    };
    if (!SHARE || part < n_it) load(part, 0);
    attn_commit();
    float ak[AR][NJ], av[AR][NJ];
#pragma unroll
    for (int r = 0; r < AR; r++)
#pragma unroll
        for (int i = 0; i < NJ; i++) { ak[r][i] = 0.f; av[r][i] = 0.f; }
    const float* myK = Kr + warp * AR * LD;
    const float* myV = Vr + warp * AR * LD;
    float* myP = Ps + warp * AKT * AR;
    for (int it = part, step = 0; it < n_it; it += S, step++) {
        const int cur = step & 1;
        const int h = g * rep + it / nq, t = (qt0 + it % nq) * AKT + lane;
        const bool live = t < s.T;
        const float L = live ? lse[((long long)b * s.H + h) * s.T + t] : 0.f;
        const float Dr = live ? Dv[b * s.db + h * s.dh_ + (long long)t * s.dtk] : 0.f;
        attn_wait();
        __syncthreads();
        if (it + S < n_it) load(it + S, cur ^ 1);
        attn_commit();
        const float* Qt = Qs + cur * TILE;
        const float* Gt = Gs + cur * TILE;
        float sc[AR], dp[AR], p[AR], ds[AR];
        attn_dot(myK, Qt + lane * LD, LD, q4, sc);
        attn_dot(myV, Gt + lane * LD, LD, q4, dp);
#pragma unroll
        for (int r = 0; r < AR; r++) {
            p[r] = live && t >= j0 + r ? expf(sc[r] * s.scale - L) : 0.f;
            ds[r] = p[r] * (dp[r] - Dr) * s.scale;
        }
        *reinterpret_cast<float4*>(myP + lane * AR) = make_float4(p[0], p[1], p[2], p[3]);
        __syncwarp();
        attn_axpy<NJ>(av, myP, Gt, LD, DH, lane);
        __syncwarp();
        *reinterpret_cast<float4*>(myP + lane * AR) = make_float4(ds[0], ds[1], ds[2], ds[3]);
        __syncwarp();
        attn_axpy<NJ>(ak, myP, Qt, LD, DH, lane);
        __syncwarp();
    }
    if (SHARE) {                         // units: dK rows, then dV rows
        attn_wait();
        __syncthreads();
        float* acc_x = smem + threadIdx.x;
#pragma unroll
        for (int r = 0; r < AR; r++)
#pragma unroll
            for (int i = 0; i < NJ; i++) { acc_x[(r * NJ + i) * ATH] = ak[r][i]; acc_x[((AR + r) * NJ + i) * ATH] = av[r][i]; }
        cluster_sync();
        for (int u = part * 2 * AR / S; u < (part + 1) * 2 * AR / S; u++) {
            const int j = j0 + u % AR;
            if (j >= s.T) continue;
            const long long koff = b * s.kb + g * s.kh + (long long)j * s.kt;
#pragma unroll
            for (int i = 0; i < NJ; i++) {
                float a = 0.f;
                for (int q = 0; q < S; q++) a += attn_peer(acc_x + (u * NJ + i) * ATH, q);
                if (lane + 32 * i < DH) stf(u < AR ? dk : dv, koff + lane + 32 * i, a);
            }
        }
        cluster_sync();             // peers have read
        return;
    }
#pragma unroll
    for (int r = 0; r < AR; r++) {
        const int j = j0 + r;
        if (j >= s.T) continue;
        const long long koff = b * s.kb + g * s.kh + (long long)j * s.kt;
#pragma unroll
        for (int i = 0; i < NJ; i++) {
            const int d = lane + 32 * i;
            if (d < DH) { stf(dk, koff + d, ak[r][i]); stf(dv, koff + d, av[r][i]); }
        }
    }
}

// Dynamic shared memory in bytes: the tiles and the warps' exchange area, or, where that is more (dK / dV of head dims up to 4), what
// the merge of a cluster puts in their place.
enum { ATTN_FWD, ATTN_DQ, ATTN_DKV };
static size_t attn_smem(int which, int DH) {
    const int nj = DH <= 32 ? 1 : DH <= 64 ? 2 : DH <= 128 ? 4 : 8;                          // columns of a row per lane
    const size_t walk = (size_t)(which == ATTN_FWD ? 5 : 6) * AKT * attn_ld(DH) + AW * AKT * AR;
    const size_t merge = (size_t)(which == ATTN_DKV ? 2 : 1) * AR * nj * ATH + (which == ATTN_FWD ? AW * AR * 2 : 0);
    return (walk > merge ? walk : merge) * 4;
}
long long ax_attn_simt_smem(int which, int DH) { return (long long)attn_smem(which, DH); }
template <typename K> static bool attn_smem_ok(size_t bytes, K kern) {
    if (bytes > 227 * 1024) return false;
    return bytes <= 48 * 1024 || cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
}
// whether every row piece of four elements starts on its natural boundary (dt: storage type)
static int attn_vec(int dt, const AttnShape& s, std::initializer_list<const void*> ptrs) {
    bool ok = s.DH % 4 == 0;
    for (long long st : {s.qb, s.qh, s.qt, s.kb, s.kh, s.kt}) ok = ok && st % 4 == 0;
    for (const void* p : ptrs) ok = ok && reinterpret_cast<uintptr_t>(p) % (dt == 1 ? 8 : 16) == 0;
    return ok;
}

// CTAs that fit the GPU, up to four per SM
static long long attn_slots(size_t smem) {
    const long long fit = (long long)(227 * 1024 / (smem + 1024));
    return (fit < 1 ? 1 : fit < 4 ? fit : 4) * AX_SMS;
}
// CTAs that share a block's walk of `chain` tiles: doubled up to four per SM, while each keeps half of `least` tiles; with more than one per SM one and
// a half, and with more than fit at once three (two fit: head dims above 64) or six (one fits: above 128).
// Gain of a doubling (484 shapes, DH 8 to 256, T 7 to 900, forward / backward) by the CTAs that it leads to and the tiles that it leaves to each:
// up to one per SM and one tile 1.16 / 1.11, two or three 1.31 / 1.18, four to seven 1.57 / 1.43; up to two per SM, where as many fit, one 1.07 / 0.90, two or
// three 1.23 / 1.10; up to four, where two fit, one 0.72 / 0.81, two or three 0.97 / 0.96, four to seven 1.08 / 1.05; up to two, where one fits, two or
// three 0.96 / 0.93, four to seven 1.12 / 0.99, eight to fifteen 1.34 / 1.20.
// fp32, forward / backward in us with 1 / 2 / 4 / (dK / dV) 8: B2 H8 KV4 T256 DH32 27, 21, 21 /
// 87, 79, 59, 47; B2 H4 KV2 T200 DH64 33, 24, 19 / 111, 73, 55, 44; B1 H8 KV8 T512 DH64 65, 45, 37 / 229, 130, 101, 107; B4 H8 KV4 T128 DH32
// 17, 15, 16 / 51, 49, 43, 36; B1 H4 KV1 T300 DH64 43, 28, 22 / 225, 126, 77, 56.
static int attn_share(long long ctas, int chain, int most, int least, size_t smem) {
    const long long slots = attn_slots(smem);
    int S = 1;
    for (; S < most; S *= 2) {
        const long long n = ctas * S * 2, half_tiles = n <= AX_SMS ? least : n <= slots ? 3 : 12 * AX_SMS / slots;
        if (n > 4 * AX_SMS || chain < half_tiles * S) break;
    }
    return S;
}
int ax_attn_simt_share(int which, const AttnShape& s) {
    const int blocks = (s.T + ABLK - 1) / ABLK, rep = s.H / s.KV;
    if (which == ATTN_DKV) return attn_share((long long)blocks * s.KV * s.B, blocks * rep, 8, 2, attn_smem(which, s.DH));
    return attn_share((long long)blocks * s.H * s.B, blocks, 4, 3, attn_smem(which, s.DH));
}

// the kernel of walks that CTAs share, or that of whole ones; early: its CTAs may start before the grid in front of it in the stream has finished
template <typename K, typename... A>
static int attn_launch(K shared, K whole, dim3 grid, size_t smem, int S, bool early, cudaStream_t st, A... args) {
    grid.x *= S;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(ATH); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = early && ax_gemm_pdl();
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = S; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = S > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, S > 1 ? shared : whole, args..., S) == cudaSuccess ? 0 : 3;
}

template <typename T, int NJ>
static int attn_fwd_launch(const void* q, const void* k, const void* v, void* o, float* lse, const AttnShape& s, int vec, cudaStream_t st) {
    const size_t smem = attn_smem(ATTN_FWD, s.DH);
    const auto shared = k_attn_fwd_simt<T, NJ, true>, whole = k_attn_fwd_simt<T, NJ, false>;
    const int S = ax_attn_simt_share(ATTN_FWD, s);
    if (!attn_smem_ok(smem, S > 1 ? shared : whole)) return 101;
    const dim3 grid((s.T + ABLK - 1) / ABLK, s.H, s.B);
    return attn_launch(shared, whole, grid, smem, S, true, st, (const T*)q, (const T*)k, (const T*)v, (T*)o, lse, s, vec);
}
template <typename T>
static int attn_fwd_nj(const void* q, const void* k, const void* v, void* o, float* lse, const AttnShape& s, int vec, cudaStream_t st) {
    if (s.DH <= 32) return attn_fwd_launch<T, 1>(q, k, v, o, lse, s, vec, st);
    if (s.DH <= 64) return attn_fwd_launch<T, 2>(q, k, v, o, lse, s, vec, st);
    if (s.DH <= 128) return attn_fwd_launch<T, 4>(q, k, v, o, lse, s, vec, st);
    return attn_fwd_launch<T, 8>(q, k, v, o, lse, s, vec, st);
}
int ax_attn_fwd_simt(int dt, const void* q, const void* k, const void* v, void* o, float* lse,
                     const AttnShape& s, cudaStream_t st) {
    if (s.DH > 256 || s.DH < 1 || s.KV < 1 || s.H % s.KV) return 101;
    if (s.B <= 0 || s.T <= 0) return 0;
    if (dt == 0) {
        const int rc = ax_attn_fwd_f32((const float*)q, (const float*)k, (const float*)v, (float*)o, lse, s, st);
        if (rc >= 0) return rc;
    }
    ax_variant = 0x86;
    const int vec = attn_vec(dt, s, {q, k, v});
    return dt == 1 ? attn_fwd_nj<bf16>(q, k, v, o, lse, s, vec, st) : attn_fwd_nj<float>(q, k, v, o, lse, s, vec, st);
}

template <typename T, typename TO, int NJ>
static int attn_bwd_launch(int part, const void* q, const void* k, const void* v, const void* dO, const float* lse,
                           const float* Dv, void* dq, void* dk, void* dv, const AttnShape& s, int vec, cudaStream_t st) {
    const size_t smem_q = attn_smem(ATTN_DQ, s.DH), smem_kv = attn_smem(ATTN_DKV, s.DH);
    const auto q_shared = k_attn_bwd_dq_simt<T, TO, NJ, true>, q_whole = k_attn_bwd_dq_simt<T, TO, NJ, false>;
    const auto kv_shared = k_attn_bwd_dkv_simt<T, TO, NJ, true>, kv_whole = k_attn_bwd_dkv_simt<T, TO, NJ, false>;
    const int Sq = ax_attn_simt_share(ATTN_DQ, s), Skv = ax_attn_simt_share(ATTN_DKV, s);
    if (!attn_smem_ok(smem_q, Sq > 1 ? q_shared : q_whole) || !attn_smem_ok(smem_kv, Skv > 1 ? kv_shared : kv_whole)) return 102;
    const dim3 g1((s.T + ABLK - 1) / ABLK, s.H, s.B), g2((s.T + ABLK - 1) / ABLK, s.KV, s.B);
    if (part == 0) return attn_launch(q_shared, q_whole, g1, smem_q, Sq, true, st, (const T*)q, (const T*)k, (const T*)v, (const T*)dO, lse, Dv, (TO*)dq, s, vec);
    // dK / dV comes early only as a quarter of a full GPU: the CTAs of its longest walks, the first, would be stacked on the SMs that dQ leaves first
    // (backward of B4 H8 KV4 T400 DH32 in us, in its turn / early: 130 / 159)
    const bool early = (long long)g2.x * g2.y * g2.z * Skv * 4 <= attn_slots(smem_kv);
    return attn_launch(kv_shared, kv_whole, g2, smem_kv, Skv, early, st, (const T*)q, (const T*)k, (const T*)v, (const T*)dO, lse, Dv, (TO*)dk, (TO*)dv, s, vec);
}
template <typename T, typename TO>
static int attn_bwd_nj(int part, const void* q, const void* k, const void* v, const void* dO, const float* lse,
                       const float* Dv, void* dq, void* dk, void* dv, const AttnShape& s, int vec, cudaStream_t st) {
    if (s.DH <= 32) return attn_bwd_launch<T, TO, 1>(part, q, k, v, dO, lse, Dv, dq, dk, dv, s, vec, st);
    if (s.DH <= 64) return attn_bwd_launch<T, TO, 2>(part, q, k, v, dO, lse, Dv, dq, dk, dv, s, vec, st);
    if (s.DH <= 128) return attn_bwd_launch<T, TO, 4>(part, q, k, v, dO, lse, Dv, dq, dk, dv, s, vec, st);
    return attn_bwd_launch<T, TO, 8>(part, q, k, v, dO, lse, Dv, dq, dk, dv, s, vec, st);
}
int ax_attn_bwd_simt(int dt, int out_dt, const void* q, const void* k, const void* v, const void* dO,
                     const float* lse, const float* Dv, void* dq, void* dk, void* dv,
                     const AttnShape& s, cudaStream_t st) {
    if (s.DH > 256 || s.DH < 1 || s.KV < 1 || s.H % s.KV) return 102;
    if (s.B <= 0 || s.T <= 0) return 0;
    if (dt == 0 && out_dt != 0) return 102;
    const int vec = attn_vec(dt, s, {q, k, v, dO});
    const bool f32 = dt == 0;
    bool there = false;
    for (int part = 0; part < 2; part++) {               // dQ, then dK / dV
        int rc = !f32 ? -1 : part == 0 ? ax_attn_dq_f32((const float*)q, (const float*)k, (const float*)v, (const float*)dO, lse, Dv, (float*)dq, s, st)
                                       : ax_attn_dkv_f32((const float*)q, (const float*)k, (const float*)v, (const float*)dO, lse, Dv, (float*)dk, (float*)dv, s, st);
        there = there || rc >= 0;
        if (rc < 0)
            rc = f32 ? attn_bwd_nj<float, float>(part, q, k, v, dO, lse, Dv, dq, dk, dv, s, vec, st) : out_dt == 1 ? attn_bwd_nj<bf16, bf16>(part, q, k, v, dO, lse, Dv, dq, dk, dv, s, vec, st)
                                                                                                          : attn_bwd_nj<bf16, float>(part, q, k, v, dO, lse, Dv, dq, dk, dv, s, vec, st);
        if (rc) return rc;
    }
    ax_variant = there ? 0x85 : 0x87;
    return 0;
}
