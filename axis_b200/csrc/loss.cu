// Index-based ops: embedding gather / scatter-add, valid-target count and
// token-mean cross-entropy with ignored targets (target < 0).
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "attn_common.cuh"

// ── embedding gather: o[r,:] = table[ids[r],:] ─────────────────────────────
// An id outside [0, rows) never reaches the table: its output row is zero-filled and the status word is set.
#define STAT_INDEX 0x400       // + 1 gather id, 2 scatter id, 3 cross-entropy target
template <typename T, typename I, int W>
__global__ void k_embed(const T* __restrict__ table, const I* __restrict__ ids, T* __restrict__ o,
                        int N, int Dw, int rows, int* status) {
    const long long total = (long long)N * Dw;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int r = (int)(i / Dw), j = (int)(i % Dw);
        const int id = (int)ids[r];
        if (id < 0 || id >= rows) {
            if (j == 0 && status) atomicExch(status, STAT_INDEX | 1);
            if (W == 1) o[i] = T(0.f);
            else reinterpret_cast<uint4*>(o)[i] = make_uint4(0, 0, 0, 0);
            continue;
        }
        const long long src = (long long)id * Dw + j;
        if (W == 1) o[i] = table[src];
        else reinterpret_cast<uint4*>(o)[i] = reinterpret_cast<const uint4*>(table)[src];
    }
}
template <typename T, typename I>
static void embed_launch(const void* table, const void* ids, void* o, int N, int D, int rows, int* status, cudaStream_t st) {
    constexpr int per = 16 / sizeof(T);
    if (D % per == 0 && aligned16(table) && aligned16(o))
        k_embed<T, I, per><<<ew_grid((long long)N * (D / per), 256), 256, 0, st>>>((const T*)table, (const I*)ids, (T*)o, N, D / per, rows, status);
    else
        k_embed<T, I, 1><<<ew_grid((long long)N * D, 256), 256, 0, st>>>((const T*)table, (const I*)ids, (T*)o, N, D, rows, status);
}
int ax_embed(int dt, const void* table, const void* ids, int ids_i32, void* o, int N, int D, int rows, int* status, cudaStream_t st) {
    if (N <= 0 || D <= 0) return 0;
    if (dt == 1) { if (ids_i32) embed_launch<bf16, int>(table, ids, o, N, D, rows, status, st); else embed_launch<bf16, float>(table, ids, o, N, D, rows, status, st); }
    else { if (ids_i32) embed_launch<float, int>(table, ids, o, N, D, rows, status, st); else embed_launch<float, float>(table, ids, o, N, D, rows, status, st); }
    return 0;
}

// ── scatter-add with fp32 atomics (reference ABI; summation order varies) ──
template <typename T>
__global__ void k_embed_bwd_atomic(const T* g, const float* ids, float* dT, int N, int D, int rows, int* status) {
    const long long total = (long long)N * D;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int r = (int)(i / D), j = (int)(i % D);
        const int id = (int)ids[r];
        if (id < 0 || id >= rows) {                     // the row is skipped, the table gradient untouched
            if (j == 0 && status) atomicExch(status, STAT_INDEX | 2);
            continue;
        }
        atomicAdd(&dT[(long long)id * D + j], ldf(g, i));
    }
}
int ax_embed_bwd_atomic(int g_bf16, const void* g, const float* ids, float* dT, int N, int D, int rows, int* status, cudaStream_t st) {
    if (N <= 0 || D <= 0) return 0;
    if (g_bf16) k_embed_bwd_atomic<bf16><<<ew_grid((long long)N * D, 256), 256, 0, st>>>((const bf16*)g, ids, dT, N, D, rows, status);
    else k_embed_bwd_atomic<float><<<ew_grid((long long)N * D, 256), 256, 0, st>>>((const float*)g, ids, dT, N, D, rows, status);
    return 0;
}

// ── ordered scatter-add without atomics ─────────────────────────────────────
// Block r acts only when row r is the first occurrence of its token; it then
// walks the later occurrences in row order and adds their gradient rows to
// dT[token] — the same order as a sequential scatter-add, every run.
template <typename T>
__global__ void k_embed_bwd_det(const T* __restrict__ g, const int* __restrict__ ids, float* dT, int N, int D, int rows, int* status) {
    __shared__ int s_flag;
    __shared__ int s_list[256];
    __shared__ int s_cnt;
    __shared__ int s_wcnt[8];
    for (int r = blockIdx.x; r < N; r += gridDim.x) {
        const int tok = ids[r];
        if (threadIdx.x == 0) s_flag = 0;
        __syncthreads();
        int seen = 0;
        for (int i = threadIdx.x; i < r; i += blockDim.x) seen |= (ids[i] == tok);
        if (seen) s_flag = 1;
        __syncthreads();
        const bool first = s_flag == 0;
        __syncthreads();
        if (tok >= rows && first && threadIdx.x == 0 && status) atomicExch(status, STAT_INDEX | 2);
        if (!first || tok < 0 || tok >= rows) continue;      // ids outside the table are skipped, nothing is written
        // gather the occurrences >= r in order, 256 at a time
        for (int base = r; base < N; base += 256) {
            if (threadIdx.x == 0) s_cnt = 0;
            __syncthreads();
            // ordered compaction of matches in [base, base+256)
            const int idx = base + (int)threadIdx.x;
            const int hit = (threadIdx.x < 256 && idx < N && ids[idx] == tok) ? 1 : 0;
            // ballot-based ordered positions (blockDim.x == 256 -> 8 warps)
            const unsigned bal = __ballot_sync(0xffffffffu, hit);
            const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
            if (!lane) s_wcnt[wp] = __popc(bal);
            __syncthreads();
            int off = 0;
            for (int q = 0; q < wp; q++) off += s_wcnt[q];
            if (hit) s_list[off + __popc(bal & ((1u << lane) - 1))] = idx;
            if (threadIdx.x == 0) { int t = 0; for (int q = 0; q < 8; q++) t += s_wcnt[q]; s_cnt = t; }
            __syncthreads();
            const int cnt = s_cnt;
            for (int j = threadIdx.x; j < D; j += blockDim.x) {
                float acc = 0.f;
                for (int q = 0; q < cnt; q++) acc += ldf(g, (long long)s_list[q] * D + j);
                if (cnt) dT[(long long)tok * D + j] += acc;
            }
            __syncthreads();
        }
    }
}

// The same for many rows.  The kernel above scans all ids once per row, N^2 / 2 reads: at 8192 rows that is 228 us (D 1536) beside
// 19 us for the memory it has to move.  Here one pass links the rows of every token into a list (last[tok] -> link[row] ->
// ...) and notes its first row; then the block of a first row takes the few others from the list, sorts them and adds
// their gradient rows in row order.  Tokens with more than EB_LIST rows are gathered by an ordered scan of the ids instead, so
// the order is always the row order and every run gives the same bits.
#define EB_LIST 16
#define EB_THREADS 256         // at most; a row of D columns takes as few slices of as many warps as it needs
__global__ void k_embed_link(const int* __restrict__ ids, unsigned* __restrict__ first, int* __restrict__ last, int* __restrict__ link,
                             int N, int rows, int* status) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        const int tok = ids[r];
        if (tok >= rows && status) atomicExch(status, STAT_INDEX | 2);
        if (tok < 0 || tok >= rows) continue;
        atomicMin(first + tok, (unsigned)r);
        link[r] = atomicExch(last + tok, r);
    }
}
// grid (rows of g, column slices of blockDim * VN columns); D is a multiple of VN, g rows and dT rows are 16-byte aligned.
// Bound by the chain of loads that depend on one another: the id, then its first and last row, then everything that a token with one row needs, its
// gradient row and the table's, at once; only tokens with more walk a list.  (With the list walked first and two slices of 128 threads for a row:
// N 8192 D 1536 V 32000 92 us, N 8192 D 768 V 32000 44 us; 56 and 15 now; the memory that it has to move takes 19 and 10.)
template <typename T, int PER>
__global__ void __launch_bounds__(EB_THREADS)
k_embed_bwd_list(const T* __restrict__ g, const int* __restrict__ ids, const unsigned* __restrict__ first, const int* __restrict__ last,
                 const int* __restrict__ link, float* __restrict__ dT, int N, int D, int rows) {
    constexpr int VN = Vec<T>::N;
    __shared__ int s_list[EB_THREADS], s_wcnt[2][EB_THREADS / 32];
    const int r = blockIdx.x, tok = ids[r];
    if (tok < 0 || tok >= rows) return;
    const unsigned head = first[tok];
    int e = last[tok];
    const int behind = link[r];
    if (head != (unsigned)r) return;
    const int col = (blockIdx.y * blockDim.x + threadIdx.x) * VN;
    float* dst = dT + (long long)tok * D + col;
    float old[VN], acc[VN];
#pragma unroll
    for (int q = 0; q < VN; q++) acc[q] = 0.f;
    if (col < D) {
#pragma unroll
        for (int q = 0; q < VN; q += 4) Vec<float>::ld(dst + q, old + q);
    }
    auto add_rows = [&](const int* list, int cnt) {
        if (col >= D) return;
#pragma unroll 4
        for (int i = 0; i < cnt; i++) {
            float f[VN];
            Vec<T>::ld(g + (long long)list[i] * D + col, f);
#pragma unroll
            for (int q = 0; q < VN; q++) acc[q] += f[q];
        }
    };
    if (e == r && behind < 0) {          // (the last to arrive may be the first row of several)
        add_rows(&r, 1);
    } else {
        // every thread walks the list (the same addresses); rows in descending order of arrival, sorted by insertion
        int list[EB_LIST], cnt = 0;
#pragma unroll
        for (int i = 0; i < EB_LIST; i++) {
            list[i] = 0x7fffffff;
            if (e >= 0) { list[i] = e; cnt++; e = link[e]; }
        }
        if (e < 0) {
            // odd-even transposition over the registers; unused places hold the largest value
#pragma unroll
            for (int p = 0; p < EB_LIST; p++) {
                if (p >= cnt) break;
#pragma unroll
                for (int i = 0; i + 1 < EB_LIST; i++)
                    if (((i ^ p) & 1) == 0 && list[i] > list[i + 1]) { const int t = list[i]; list[i] = list[i + 1]; list[i + 1] = t; }
            }
#pragma unroll
            for (int i = 0; i < EB_LIST; i++) if (threadIdx.x == i) s_list[i] = list[i];
            __syncthreads();
            add_rows(s_list, cnt);
        } else {
            const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, warps = blockDim.x >> 5;
            if (PER == 1) {
                for (int base = r; base < N; base += blockDim.x) {
                    const int idx = base + (int)threadIdx.x;
                    const bool hit = idx < N && ids[idx] == tok;
                    const unsigned bal = __ballot_sync(0xffffffffu, hit);
                    if (!lane) s_wcnt[0][wp] = __popc(bal);
                    __syncthreads();
                    int off = 0, n = 0;
                    for (int q = 0; q < warps; q++) { if (q < wp) off += s_wcnt[0][q]; n += s_wcnt[0][q]; }
                    if (hit) s_list[off + __popc(bal & ((1u << lane) - 1))] = idx;
                    __syncthreads();
                    add_rows(s_list, n);
                    __syncthreads();
                }
            }
            // Blocks of few warps, those of narrow rows: turns of some 256 ids all the same.  With an id to a thread the scan of one warp took three times as long as that
            // of the four warps that such rows had before (N 8000 D 128 V 1000 fp32, tokens of up to 31 rows: 30 us with four warps, 88 with one, 35 so).  Each warp has ids
            // of its own behind one another and does nothing where it finds none, which is most of the time.
            for (int base = r, turn = 0; PER > 1 && base < N; base += blockDim.x * PER, turn ^= 1) {
                const int mine = base + wp * 32 * PER + lane;
                unsigned hits = 0;
#pragma unroll
                for (int q = 0; q < PER; q++)
                    if (mine + q * 32 < N && ids[mine + q * 32] == tok) hits |= 1u << q;
                int cnt = 0;
                if (__any_sync(0xffffffffu, hits))
#pragma unroll
                    for (int q = 0; q < PER; q++) cnt += __popc(__ballot_sync(0xffffffffu, hits >> q & 1));
                if (!lane) s_wcnt[turn][wp] = cnt;
                __syncthreads();                           // (also: everyone has left the list of the turn before)
                int off = 0, n = 0;
                for (int w = 0; w < warps; w++) { if (w == wp) off = n; n += s_wcnt[turn][w]; }
                if (!n) continue;
                if (cnt)
#pragma unroll
                    for (int q = 0; q < PER; q++) {
                        const unsigned bal = __ballot_sync(0xffffffffu, hits >> q & 1);
                        if (hits >> q & 1) s_list[off + __popc(bal & ((1u << lane) - 1))] = mine + q * 32;
                        off += __popc(bal);
                    }
                __syncthreads();
                add_rows(s_list, n);
            }
        }
    }
    if (col < D) {
#pragma unroll
        for (int q = 0; q < VN; q += 4)
            *reinterpret_cast<float4*>(dst + q) = make_float4(old[q] + acc[q], old[q + 1] + acc[q + 1], old[q + 2] + acc[q + 2], old[q + 3] + acc[q + 3]);
    }
}
// ws: scratch for the lists, (2 * table rows + N) ints, or null.  The lists pay from about a thousand rows (512: 4 us scanned, 7 us
// with the two extra launches; 1536: 17 us scanned).
int ax_embed_bwd_det(int g_dt, const void* g, const int* ids, float* dT, int N, int D, int rows, int* status, void* ws, size_t ws_bytes,
                     cudaStream_t st) {
    if (N <= 0 || D <= 0) return 0;
    const int vn = g_dt >= 1 ? 8 : 4;
    if (ws && N >= 1024 && D % vn == 0 && aligned16(g) && aligned16(dT) && ((size_t)rows * 2 + N) * 4 <= ws_bytes) {
        unsigned* first = (unsigned*)ws;
        int* last = (int*)ws + rows;
        int* link = last + rows;
        if (cudaMemsetAsync(ws, 0xff, (size_t)rows * 8, st)) return 1;
        k_embed_link<<<(N + 255) / 256, 256, 0, st>>>(ids, first, last, link, N, rows, status);
        const int warps = (D / vn + 31) / 32, slices = (warps * 32 + EB_THREADS - 1) / EB_THREADS, threads = (warps + slices - 1) / slices * 32;
        const dim3 grid(N, slices);
        auto launch = [&](auto per) {                      // ids of a thread in a turn of the scan: some 256 a block
            constexpr int PER = decltype(per)::value;
            if (g_dt >= 1) k_embed_bwd_list<bf16, PER><<<grid, threads, 0, st>>>((const bf16*)g, ids, first, last, link, dT, N, D, rows);
            else k_embed_bwd_list<float, PER><<<grid, threads, 0, st>>>((const float*)g, ids, first, last, link, dT, N, D, rows);
        };
        if (threads <= 32) launch(std::integral_constant<int, 8>());
        else if (threads <= 64) launch(std::integral_constant<int, 4>());
        else if (threads < 128) launch(std::integral_constant<int, 2>());
        else launch(std::integral_constant<int, 1>());
        ax_variant = 0x71;
        return 0;
    }
    ax_variant = 0x70;
    const int grid = N < AX_SMS * 16 ? N : AX_SMS * 16;
    if (g_dt >= 1) k_embed_bwd_det<bf16><<<grid, 256, 0, st>>>((const bf16*)g, ids, dT, N, D, rows, status);
    else k_embed_bwd_det<float><<<grid, 256, 0, st>>>((const float*)g, ids, dT, N, D, rows, status);
    return 0;
}

// ── count of valid targets (float accumulator, exact below 2^24) ───────────
__global__ void k_countvalid(const float* tgt, float* acc, int N) {
    __shared__ float sh[40];
    float s = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += blockDim.x * gridDim.x) s += (tgt[i] >= 0.f) ? 1.f : 0.f;
    s = block_sum(s, sh);
    if (threadIdx.x == 0 && s != 0.f) atomicAdd(acc, s);
}
int ax_countvalid(const float* tgt, float* acc, int N, cudaStream_t st) {
    if (N <= 0) return 0;
    int blocks = (N + 255) / 256; if (blocks > 1024) blocks = 1024;
    k_countvalid<<<blocks, 256, 0, st>>>(tgt, acc, N);
    return 0;
}

// ── cross-entropy rows ──────────────────────────────────────────────────────
// One block per row.  Pass 1 keeps a running (max, sum) per thread — a single
// read of the row; pass 2 writes (softmax - onehot) * inv_count.  Safe in
// place (dlogits == logits): pass 2 starts after the block-wide reduction, and
// every element is re-read by the thread that overwrites it.
// Reference ABI (kind CE): fp32 targets, denom buffer optional, loss via one
// atomicAdd per row.
template <typename T, bool VEC>
__global__ void k_ce(const T* logits, const float* tgt, T* dlogits, float* loss, const float* denom, int Nrows, int V, int* status) {
    __shared__ float sh[40];
    __shared__ float s_xt;
    for (int r = blockIdx.x; r < Nrows; r += gridDim.x) {
        const T* lr = logits + (long long)r * V;
        T* dr = dlogits + (long long)r * V;
        int t = (int)tgt[r];
        if (t >= V) {                    // a target outside the vocabulary: the row counts as ignored
            if (threadIdx.x == 0 && status) atomicExch(status, STAT_INDEX | 3);
            t = -1;
        }
        if (t < 0) {
            for (int j = threadIdx.x; j < V; j += blockDim.x) stf(dr, j, 0.f);
            continue;
        }
        if (threadIdx.x == 0) s_xt = ldf(lr, t);       // before any in-place overwrite
        __syncthreads();
        const float inv = denom ? 1.f / denom[0] : 1.f / Nrows;
        constexpr int N = Vec<T>::N;
        float m = -3.0e38f, s = 0.f;
        if (VEC) {
            for (int j = threadIdx.x * N; j < V; j += blockDim.x * N) {
                float f[N];
                Vec<T>::ld(lr + j, f);
                float mx = f[0];
#pragma unroll
                for (int q = 1; q < N; q++) mx = fmaxf(mx, f[q]);
                if (mx > m) { s *= expf(m - mx); m = mx; }
#pragma unroll
                for (int q = 0; q < N; q++) s += expf(f[q] - m);
            }
        } else {
            for (int j = threadIdx.x; j < V; j += blockDim.x) {
                const float f = ldf(lr, j);
                if (f > m) { s *= expf(m - f); m = f; }
                s += expf(f - m);
            }
        }
        const float M = block_max(m, sh);
        s = (m > -3.0e38f) ? s * expf(m - M) : 0.f;
        const float S = block_sum(s, sh);
        const float invS = 1.f / S;
        if (VEC) {
            for (int j = threadIdx.x * N; j < V; j += blockDim.x * N) {
                float f[N];
                Vec<T>::ld(lr + j, f);
#pragma unroll
                for (int q = 0; q < N; q++) f[q] = (expf(f[q] - M) * invS - ((j + q) == t ? 1.f : 0.f)) * inv;
                Vec<T>::st(dr + j, f);
            }
        } else {
            for (int j = threadIdx.x; j < V; j += blockDim.x)
                stf(dr, j, (expf(ldf(lr, j) - M) * invS - (j == t ? 1.f : 0.f)) * inv);
        }
        if (threadIdx.x == 0) atomicAdd(loss, (logf(S) - (s_xt - M)) * inv);
        __syncthreads();
    }
}
int ax_ce(int dt, const void* logits, const float* tgt, void* dlogits, float* loss, const float* denom, int N, int V, int* status, cudaStream_t st) {
    if (N <= 0 || V <= 0) return 0;
    const int per = dt == 1 ? 8 : 4;
    const bool vec = V % per == 0 && aligned16(logits) && aligned16(dlogits);
    const int thr = V >= 4096 ? 512 : 256;
    const int grid = N < AX_SMS * 64 ? N : AX_SMS * 64;
    if (dt == 1) {
        if (vec) k_ce<bf16, true><<<grid, thr, 0, st>>>((const bf16*)logits, tgt, (bf16*)dlogits, loss, denom, N, V, status);
        else k_ce<bf16, false><<<grid, thr, 0, st>>>((const bf16*)logits, tgt, (bf16*)dlogits, loss, denom, N, V, status);
    } else {
        if (vec) k_ce<float, true><<<grid, thr, 0, st>>>((const float*)logits, tgt, (float*)dlogits, loss, denom, N, V, status);
        else k_ce<float, false><<<grid, thr, 0, st>>>((const float*)logits, tgt, (float*)dlogits, loss, denom, N, V, status);
    }
    return 0;
}

// ── fused, deterministic form ───────────────────────────────────────────────
// k_ce_prepare: one block counts the valid targets (integer), stores the count
// as float in denom[0], zeroes the done-counter and the count of rows handed out.  k_ce_rows: as k_ce, but the
// row keeps its loss term in rowloss[r]; the last block to finish adds the N
// terms in a fixed order and writes loss[0].
__global__ void k_ce_prepare(const int* tgt, float* denom, float* loss, unsigned int* counter, int N, int V) {
    __shared__ int sh_i[32];
    int c = 0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) c += tgt[i] >= 0 && tgt[i] < V;
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) sh_i[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) t += sh_i[q];
        denom[0] = (float)t;
        loss[0] = 0.f;
        counter[0] = counter[1] = 0u;
    }
}
template <typename T, bool VEC>
__global__ void k_ce_rows(const T* logits, const int* tgt, T* dlogits, float* loss, const float* denom,
                          float* rowloss, unsigned int* counter, int Nrows, int V, int ld, int* status) {
    // VEC: ld is a multiple of the vector, V need not be: the elements past V in a row's last vector count as -inf and
    // leave as zeros; the scalar form zeroes the same columns, as far as the row goes
    __shared__ float sh[40];
    __shared__ float s_xt;
    __shared__ bool s_last;
    constexpr int N = Vec<T>::N;
    const int pad_end = min(ld, (V + N - 1) / N * N);
    const float inv = 1.f / denom[0];
    for (int r = blockIdx.x; r < Nrows; r += gridDim.x) {
        const T* lr = logits + (long long)r * ld;
        T* dr = dlogits + (long long)r * ld;
        int t = tgt[r];
        if (t >= V) {
            if (threadIdx.x == 0 && status) atomicExch(status, STAT_INDEX | 3);
            t = -1;
        }
        if (t < 0) {
            if (VEC) {
                float z[N];
#pragma unroll
                for (int q = 0; q < N; q++) z[q] = 0.f;
                for (int j = threadIdx.x * N; j < V; j += blockDim.x * N) Vec<T>::st(dr + j, z);
            } else {
                for (int j = threadIdx.x; j < pad_end; j += blockDim.x) stf(dr, j, 0.f);
            }
            if (threadIdx.x == 0) rowloss[r] = 0.f;
            continue;
        }
        if (threadIdx.x == 0) s_xt = ldf(lr, t);
        __syncthreads();
        float m = -3.0e38f, s = 0.f;
        if (VEC) {
            for (int j = threadIdx.x * N; j < V; j += blockDim.x * N) {
                float f[N];
                Vec<T>::ld(lr + j, f);
                if (j + N > V) {
#pragma unroll
                    for (int q = 0; q < N; q++) if (j + q >= V) f[q] = -INFINITY;
                }
                float mx = f[0];
#pragma unroll
                for (int q = 1; q < N; q++) mx = fmaxf(mx, f[q]);
                if (mx > m) { s *= expf(m - mx); m = mx; }
#pragma unroll
                for (int q = 0; q < N; q++) s += expf(f[q] - m);
            }
        } else {
            for (int j = threadIdx.x; j < V; j += blockDim.x) {
                const float f = ldf(lr, j);
                if (f > m) { s *= expf(m - f); m = f; }
                s += expf(f - m);
            }
        }
        const float M = block_max(m, sh);
        s = (m > -3.0e38f) ? s * expf(m - M) : 0.f;
        const float S = block_sum(s, sh);
        const float invS = 1.f / S;
        if (VEC) {
            for (int j = threadIdx.x * N; j < V; j += blockDim.x * N) {
                float f[N];
                Vec<T>::ld(lr + j, f);
                if (j + N > V) {
#pragma unroll
                    for (int q = 0; q < N; q++) if (j + q >= V) f[q] = -INFINITY;
                }
#pragma unroll
                for (int q = 0; q < N; q++) f[q] = (expf(f[q] - M) * invS - ((j + q) == t ? 1.f : 0.f)) * inv;
                Vec<T>::st(dr + j, f);
            }
        } else {
            for (int j = threadIdx.x; j < V; j += blockDim.x)
                stf(dr, j, (expf(ldf(lr, j) - M) * invS - (j == t ? 1.f : 0.f)) * inv);
            for (int j = V + threadIdx.x; j < pad_end; j += blockDim.x) stf(dr, j, 0.f);
        }
        if (threadIdx.x == 0) rowloss[r] = logf(S) - (s_xt - M);
        __syncthreads();
    }
    // last block standing reduces the row terms in index order
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (s_last) {
        __threadfence();
        float acc = 0.f;
        for (int i = threadIdx.x; i < Nrows; i += blockDim.x) acc += __ldcg(rowloss + i);
        acc = block_sum(acc, sh);
        if (threadIdx.x == 0) loss[0] = acc * inv;
    }
}
// bf16 rows of up to TH * 8 * 8 logits (32768 with 512 threads, 65536 with 1024): the row is read from DRAM once into
// registers (8 packed 16-byte vectors per thread), reduced, and written back — one read and one write per element.
// F32: the registers keep the logits and the exponential of an element is taken twice in fp32; otherwise they keep it as fp16
// after the sum, whose small values (below 6e-5 of the row's largest) lose relative accuracy.  See the rule in ax_ce_fused.
// The rows of a block come by bulk copy into shared memory, each one while the row in front of it is worked on in registers: with loads
// straight into registers a block's memory traffic stood still during its reductions, and two blocks to an SM did not cover that
// (8192 x 32000, 1.05 GB, one launch: 262 us with the loads, 204 so, in turn on one box; behind the product that makes the logits as well).
// A block takes its next row when it has one, since rows without a loss take no time: in turn, 1500 x 65528 with nine in ten of them took
// 87 us against 71 with the loads, 64 so, and 8192 x 32000 with one in twenty 215 (204 so).  The terms of the loss are added in row order all the same.
#define CE_VPT 8
#define STAT_CE 0x800
template <int TH, bool F32>
__global__ void __launch_bounds__(TH, 1024 / TH)
k_ce_rows_reg(const bf16* logits, const int* __restrict__ tgt, bf16* dlogits, float* loss, const float* denom,
              float* rowloss, unsigned int* counter, int Nrows, int V, int ld, int* status) {
    __shared__ float sh[40];
    __shared__ float s_xt;
    __shared__ bool s_last;
    __shared__ uint64_t s_bar;
    __shared__ int s_next;
    extern __shared__ __align__(128) uint4 ce_row[];
    const float inv = 1.f / denom[0];
    const int nvec = (V + 7) >> 3;
    const uint32_t bar = smem_u32(&s_bar), row_at = smem_u32(ce_row);
    auto next_row = [&]() { return Nrows > (int)gridDim.x ? (int)(gridDim.x + atomicAdd(counter + 1, 1u)) : Nrows; };
    auto fetch = [&](int r) {                           // thread 0: the next row, unless it carries no loss
        if (r >= Nrows || tgt[r] < 0 || tgt[r] >= V) return;
        mbar_expect_tx(bar, nvec * 16);
        bulk_load_1d(row_at, logits + (long long)r * ld, nvec * 16, bar);
    };
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
        fetch(blockIdx.x);
    }
    __syncthreads();
    uint32_t par = 0;
    bool ok = true;
    for (int r = blockIdx.x; r < Nrows;) {
        bf16* dr = dlogits + (long long)r * ld;
        int t = tgt[r];
        if (t >= V) {
            if (threadIdx.x == 0 && status) atomicExch(status, STAT_INDEX | 3);
            t = -1;
        }
        if (t < 0) {
            const uint4 z = make_uint4(0, 0, 0, 0);
            for (int j = threadIdx.x; j < nvec; j += TH) reinterpret_cast<uint4*>(dr)[j] = z;
            __syncthreads();                             // everyone has taken r out of s_next
            if (threadIdx.x == 0) { rowloss[r] = 0.f; s_next = next_row(); fetch(s_next); }
            __syncthreads();
            r = s_next;
            continue;
        }
        ok = ok && mbar_wait(bar, par);                  // bounded; what follows a row that does not come is void, see below
        par ^= 1;
        uint4 pk[CE_VPT];
#pragma unroll
        for (int i = 0; i < CE_VPT; i++) {
            const int j = threadIdx.x + i * TH;
            pk[i] = j < nvec ? ce_row[j] : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);  // -inf
            if (j * 8 + 8 > V && j < nvec) {            // the row's last vector: what lies past V is -inf, too
                unsigned short* e = reinterpret_cast<unsigned short*>(&pk[i]);
#pragma unroll
                for (int q = 0; q < 8; q++) if (j * 8 + q >= V) e[q] = 0xff80;
            }
        }
        if (threadIdx.x == 0) s_xt = __bfloat162float(reinterpret_cast<const bf16*>(ce_row)[t]);
        float m = -3.0e38f;
#pragma unroll
        for (int i = 0; i < CE_VPT; i++) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&pk[i]);
#pragma unroll
            for (int q = 0; q < 4; q++) { const float2 f = __bfloat1622float2(h[q]); m = fmaxf(m, fmaxf(f.x, f.y)); }
        }
        const float M = block_max(m, sh);                // (everyone has read the row)
        if (threadIdx.x == 0) { s_next = next_row(); if (ok) fetch(s_next); }
        // !F32: one exponential per element, e = exp(x - M) replaces x in the same registers as packed fp16 (e <= 1,
        // 11-bit mantissa: finer than the bf16 the gradient is stored in); the sum uses the fp32 values
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < CE_VPT; i++) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&pk[i]);
            __half2 eh[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float2 f = __bfloat1622float2(h[q]);
                const float e0 = F32 ? expf(f.x - M) : __expf(f.x - M), e1 = F32 ? expf(f.y - M) : __expf(f.y - M);
                s += e0 + e1;
                if (!F32) eh[q] = __floats2half2_rn(e0, e1);
            }
            if (!F32) pk[i] = *reinterpret_cast<const uint4*>(eh);
        }
        const float S = block_sum(s, sh);
        const float sc = inv / S;
#pragma unroll
        for (int i = 0; i < CE_VPT; i++) {
            const int j = threadIdx.x + i * TH;
            if (j < nvec) {
                float f[8];
                if (F32) {
                    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&pk[i]);
#pragma unroll
                    for (int q = 0; q < 4; q++) { const float2 v = __bfloat1622float2(h[q]); f[2 * q] = expf(v.x - M); f[2 * q + 1] = expf(v.y - M); }
                } else {
                    const __half2* h = reinterpret_cast<const __half2*>(&pk[i]);
#pragma unroll
                    for (int q = 0; q < 4; q++) { const float2 v = __half22float2(h[q]); f[2 * q] = v.x; f[2 * q + 1] = v.y; }
                }
#pragma unroll
                for (int q = 0; q < 8; q++) f[q] = f[q] * sc - ((j * 8 + q) == t ? inv : 0.f);
                Vec<bf16>::st(dr + j * 8, f);
            }
        }
        if (threadIdx.x == 0) rowloss[r] = logf(S) - (s_xt - M);
        __syncthreads();
        r = s_next;                                      // (written again only behind the next row's barriers)
    }
    if (!ok) {                                           // (out here: in the loop it spills more of the row and takes 10 to 25 % longer)
        if (status) atomicExch(status, STAT_CE | 1);
        mbar_wait(bar, 0);                               // shared memory is not given up under a copy in flight (the phase that is over does not wait)
        mbar_wait(bar, 1);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (s_last) {
        __threadfence();
        float acc = 0.f;
        for (int i = threadIdx.x; i < Nrows; i += blockDim.x) acc += __ldcg(rowloss + i);
        acc = block_sum(acc, sh);
        if (threadIdx.x == 0) loss[0] = acc * inv;
    }
}

int ax_ce_fused(int dt, const void* logits, const int* tgt, void* dlogits, float* loss, float* denom,
                float* scratch, int N, int V, int ld, int* status, cudaStream_t st) {
    if (N <= 0 || V <= 0) return 0;
    unsigned int* counter = reinterpret_cast<unsigned int*>(scratch);
    float* rowloss = scratch + 8;
    k_ce_prepare<<<1, 1024, 0, st>>>(tgt, denom, loss, counter, N, V);
    const int per = dt == 1 ? 8 : 4;
    const bool vec = ld % per == 0 && aligned16(logits) && aligned16(dlogits);
    const int thr = V >= 4096 ? 512 : 256;
    const int grid = N < AX_SMS * 16 ? N : AX_SMS * 16;
    ax_variant = 0x10;
    if (dt == 1 && vec && V >= 2048 && V <= 1024 * 8 * CE_VPT) {
        const int per_sm = V > 512 * 8 * CE_VPT ? 1 : 2, g2 = N < AX_SMS * per_sm ? N : AX_SMS * per_sm;
        const size_t smem = (size_t)(V + 7) / 8 * 16;
        ax_variant = 0x11;
        // fp16 exponentials up to 32768 columns in whole vectors, the form these rows have always had; the others, which took
        // their exponentials in fp32 as streaming rows before they fitted the registers, keep them
#define CE_REG(TH, F32)                                                                                                                            \
    static const cudaError_t attr = cudaFuncSetAttribute(k_ce_rows_reg<TH, F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, TH * CE_VPT * 16); \
    if (attr != cudaSuccess) return 3;                                                                                                            \
    k_ce_rows_reg<TH, F32><<<g2, TH, smem, st>>>((const bf16*)logits, tgt, (bf16*)dlogits, loss, denom, rowloss, counter, N, V, ld, status)
        if (V > 512 * 8 * CE_VPT) { CE_REG(1024, true); }
        else if (V % 8) { CE_REG(512, true); }
        else { CE_REG(512, false); }
#undef CE_REG
        return 0;
    }
    if (dt == 1) {
        if (vec) k_ce_rows<bf16, true><<<grid, thr, 0, st>>>((const bf16*)logits, tgt, (bf16*)dlogits, loss, denom, rowloss, counter, N, V, ld, status);
        else k_ce_rows<bf16, false><<<grid, thr, 0, st>>>((const bf16*)logits, tgt, (bf16*)dlogits, loss, denom, rowloss, counter, N, V, ld, status);
    } else {
        if (vec) k_ce_rows<float, true><<<grid, thr, 0, st>>>((const float*)logits, tgt, (float*)dlogits, loss, denom, rowloss, counter, N, V, ld, status);
        else k_ce_rows<float, false><<<grid, thr, 0, st>>>((const float*)logits, tgt, (float*)dlogits, loss, denom, rowloss, counter, N, V, ld, status);
    }
    return 0;
}
