// Attention over a shared low-rank latent (multi-head latent attention), CUDA cores,
// everything after the loads in 32-bit.
//
// Per token the cache keeps one row of W = rank + rot elements for all heads: the latent c
// (RMS-normed down-projection) and one rotated key part r.  Head h's key is
// [Wuk_h c | r] and its value Wuv_h c; with q_h = [a_h | b_h] (b_h rotated)
//     s_hj = (a_h . Wuk_h c_j + b_h . r_j) * scale = ((Wuk_h^T a_h) . c_j + b_h . r_j) * scale
//     o_h  = Wuv_h (sum_j p_hj c_j)
// so the kernels here work on the cached rows themselves: the query is carried into the
// latent space first (`absorb`), the attention runs as many query heads over ONE key/value
// row per position (the value is the row's first `rank` elements), and the result is
// carried out through Wuv (`expand`).  Keys and values per head are never formed.
//
// Softmax: position i sees j with 0 <= i - j < window (window <= 0: all j <= i); the
// denominator also holds exp(sink_h) when sinks are given (a learned logit without key or
// value, not scaled).
//
// Kernels:
//   latent_prep    per token: c = rms(d[:rank]) * w, r = rotate(d[rank:]) at the token's
//                  position, the row [c | r] to a dense step buffer and (optionally) to the
//                  paged cache; the rotated part of every query head is rotated in place.
//   latent_store   rows of the step buffer to the paged cache (for a ring whose rows the
//                  step's own attention still had to read).
//   latent_absorb  qa[m, h] = [Wuk_h^T a_{m,h} | b_{m,h}] in float32.
//   latent_attn    the attention; a sequence's new tokens follow `seq_start[b]` positions in
//                  the cache (rows below the start are read from pages, the others from the
//                  step buffer), any mix of starts and counts in one launch.
//   latent_expand  o[m, h] = Wuv_h ol[m, h], times sigmoid(gate[m, h]) where a design gates its heads.
#include "common.cuh"
#include "attn_decode.cuh"
#include "tma.cuh"

#include <algorithm>

namespace {

struct LatentPages {
    void* pages;                 // [n_pages, page_size, W]
    const int* page_table; int table_width; int page_size; int ring_rows; int n_pages;
    const int* seq_len;          // each sequence's length after the step (for stores into a ring)
};

// sigmoid of a head's gate logit: logits [M, heads], row stride in elements
template <typename T>
__device__ __forceinline__ float head_gate(const T* gate, long long stride, size_t token, int head) {
    return ti_over(1.0f, 1.0f + expf(-to_f32(gate[token * stride + head])));
}

template <typename T>
__device__ __forceinline__ void store_row_to_pages(const LatentPages& kv, int slot, int seq, int pos, int W, const T* row_vals,
                                                   int tid, int nthreads) {
    // in a ring only the last ring_rows positions of the sequence are kept: an older row of this step
    // must not land on the place of a newer one, whichever block runs last
    if (kv.ring_rows > 0 && pos + kv.ring_rows < kv.seq_len[seq]) return;
    const int row = kv.ring_rows > 0 ? pos % kv.ring_rows : pos;
    const int pidx = row / kv.page_size;
    if (pidx >= kv.table_width) return;
    const int page = kv.page_table[(size_t)slot * kv.table_width + pidx];
    if (page < 0 || page >= kv.n_pages) return;
    T* dst = (T*)kv.pages + ((size_t)page * kv.page_size + row % kv.page_size) * W;
    for (int i = tid; i < W; i += nthreads) dst[i] = row_vals[i];
}

// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void latent_prep_body(float* sm, int m, const T* d, long long d_stride, T* q, long long q_stride,
                                                 int n_heads, int plain, int rank, int rot, const float* __restrict__ norm_w, float eps,
                                                 const float* __restrict__ cos_t, const float* __restrict__ sin_t, int max_pos,
                                                 const int* __restrict__ tok_pos, const int* __restrict__ tok_seq,
                                                 const int* __restrict__ seq_slot, T* __restrict__ lat, const LatentPages& kv) {
    const int W = rank + rot;
    float* vals = sm;                    // W floats, then 33, then W values of T
    float* red = sm + W;
    T* rounded = reinterpret_cast<T*>(red + 33);
    const int t = threadIdx.x, nt = blockDim.x;
    const int pos = min(max(tok_pos[m], 0), max_pos - 1);
    const int half = rot >> 1;
    const float* cs = cos_t + (size_t)pos * half;
    const float* sn = sin_t + (size_t)pos * half;
    const T* drow = d + (size_t)m * d_stride;
    // (loads in batches, so that several are on their way at a time, the weights and tables among them)
    constexpr int AHEAD = 8;
    float ss = 0.f, nw[AHEAD], c_r = 0.f, s_r = 0.f;
    for (int i0 = t; i0 < W; i0 += AHEAD * nt) {
        float x[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; j++) x[j] = i0 + j * nt < W ? to_f32(drow[i0 + j * nt]) : 0.f;
        if (i0 == t) {
#pragma unroll
            for (int j = 0; j < AHEAD; j++) nw[j] = t + j * nt < rank ? norm_w[t + j * nt] : 0.f;
            if (t < half) { c_r = cs[t]; s_r = sn[t]; }
        }
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            const int i = i0 + j * nt;
            if (i < W) vals[i] = x[j];
            if (i < rank) ss = fmaf(x[j], x[j], ss);
        }
    }
    ss = block_sum(ss, red);             // (also makes vals visible)
    const float inv = rsqrtf(ss / (float)rank + eps);
#pragma unroll
    for (int j = 0; j < AHEAD; j++)
        if (t + j * nt < rank) rounded[t + j * nt] = from_f32<T>(vals[t + j * nt] * inv * nw[j]);
    for (int i = t + AHEAD * nt; i < rank; i += nt) rounded[i] = from_f32<T>(vals[i] * inv * norm_w[i]);
    for (int i = t; i < half; i += nt) {
        const float u = vals[rank + i], v = vals[rank + i + half], c = i == t ? c_r : cs[i], s = i == t ? s_r : sn[i];
        rounded[rank + i] = from_f32<T>(u * c - v * s);
        rounded[rank + i + half] = from_f32<T>(v * c + u * s);
    }
    __syncthreads();
    if (lat)
        for (int i = t; i < W; i += nt) lat[(size_t)m * W + i] = rounded[i];
    if (kv.pages) store_row_to_pages<T>(kv, seq_slot[tok_seq[m]], tok_seq[m], tok_pos[m], W, rounded, t, nt);
    // the rotated part of every query head, in place
    if (q) {
        const int hd = plain + rot;
        for (int idx = t; idx < n_heads * half; idx += nt) {
            const int h = idx / half, i = idx - h * half;
            T* p = q + (size_t)m * q_stride + (size_t)h * hd + plain;
            const float u = to_f32(p[i]), v = to_f32(p[i + half]), c = cs[i], s = sn[i];
            p[i] = from_f32<T>(u * c - v * s);
            p[i + half] = from_f32<T>(v * c + u * s);
        }
    }
}

template <typename T>
__global__ void latent_prep_kernel(const T* __restrict__ d, long long d_stride, T* __restrict__ q, long long q_stride,
                                   int n_heads, int plain, int rank, int rot, const float* __restrict__ norm_w, float eps,
                                   const float* __restrict__ cos_t, const float* __restrict__ sin_t, int max_pos,
                                   const int* __restrict__ tok_pos, const int* __restrict__ tok_seq,
                                   const int* __restrict__ seq_slot, T* __restrict__ lat, LatentPages kv) {
    ti_pdl_trigger();
    extern __shared__ float sm[];
    ti_pdl_sync();
    d = ti_dependent(d); q = ti_dependent(q);
    latent_prep_body<T>(sm, blockIdx.x, d, d_stride, q, q_stride, n_heads, plain, rank, rot, norm_w, eps, cos_t, sin_t, max_pos, tok_pos, tok_seq,
                        seq_slot, lat, kv);
}

// For steps of few tokens: the work of latent_prep and latent_absorb in one launch.  Grid (tokens, heads + 1): block
// (m, h) with h < heads carries head h of token m into the latent space (the rotated part is rotated on the way, q itself
// stays as it is); block (m, heads) does the token's row.
constexpr int ABSORB_THREADS = 512;      // rows of Wuk that are on their way together: eight a thread, shared out over the block

template <typename T>
__global__ void __launch_bounds__(ABSORB_THREADS)
latent_prep_absorb_kernel(const T* __restrict__ d, long long d_stride, const T* __restrict__ q, long long q_stride,
                          int n_heads, int plain, int rank, int rot, const float* __restrict__ norm_w, float eps,
                          const float* __restrict__ cos_t, const float* __restrict__ sin_t, int max_pos,
                          const int* __restrict__ tok_pos, const int* __restrict__ tok_seq, const int* __restrict__ seq_slot,
                          T* __restrict__ lat, LatentPages kv, const T* __restrict__ uk, float* __restrict__ qa) {
    ti_pdl_trigger();
    extern __shared__ float sm[];
    ti_pdl_sync();
    d = ti_dependent(d); q = ti_dependent(q);
    if ((int)blockIdx.y == n_heads) {
        latent_prep_body<T>(sm, blockIdx.x, d, d_stride, (T*)nullptr, 0, n_heads, plain, rank, rot, norm_w, eps, cos_t, sin_t, max_pos, tok_pos,
                            tok_seq, seq_slot, lat, kv);
        return;
    }
    const int m = blockIdx.x, h = blockIdx.y, t = threadIdx.x;
    const int hd = plain + rot, W = rank + rot, half = rot >> 1;
    const T* qh = q + (size_t)m * q_stride + (size_t)h * hd;
    float* qs = sm;                      // [plain]
    for (int i = t; i < plain; i += blockDim.x) qs[i] = to_f32(qh[i]);
    float* dst = qa + ((size_t)m * n_heads + h) * W;
    if (rot) {
        const int pos = min(max(tok_pos[m], 0), max_pos - 1);
        for (int i = t; i < half; i += blockDim.x) {
            // (rounded to the engine's type as the rotation in place would have left it)
            const float u = to_f32(qh[plain + i]), v = to_f32(qh[plain + i + half]);
            const float c = cos_t[(size_t)pos * half + i], sn = sin_t[(size_t)pos * half + i];
            dst[rank + i] = to_f32(from_f32<T>(u * c - v * sn));
            dst[rank + i + half] = to_f32(from_f32<T>(v * c + u * sn));
        }
    }
    __syncthreads();
    const T* ukh = uk + (size_t)h * plain * rank;
    if (sizeof(T) == 2 && (rank & 7) == 0 && (reinterpret_cast<uintptr_t>(ukh) & 15) == 0) {
        // eight elements of a row a read, the rows shared out over as many groups of threads as a row leaves room for; a
        // group's sums meet in shared memory
        const int pieces = rank >> 3, lanes = min(pieces, (int)blockDim.x), groups = blockDim.x / lanes, grp = t / lanes;
        float* part = sm + plain;        // [groups][rank]
        for (int c0 = 0; c0 < pieces; c0 += lanes) {
            const int c = c0 + t - grp * lanes;
            if (grp < groups && c < pieces) {
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                const int n = (plain - grp + groups - 1) / groups;         // rows grp, grp + groups, ...
                for (int j0 = 0; j0 < n; j0 += 8) {
                    uint4 w[8];
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        w[j] = j0 + j < n ? reinterpret_cast<const uint4*>(ukh + (size_t)(grp + (j0 + j) * groups) * rank)[c] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float qv = j0 + j < n ? qs[grp + (j0 + j) * groups] : 0.f;
                        const bf16* wv = reinterpret_cast<const bf16*>(&w[j]);
#pragma unroll
                        for (int e = 0; e < 8; e++) acc[e] = fmaf(qv, to_f32(wv[e]), acc[e]);
                    }
                }
#pragma unroll
                for (int e = 0; e < 8; e++) part[grp * rank + c * 8 + e] = acc[e];
            }
        }
        __syncthreads();
        for (int r = t; r < rank; r += blockDim.x) {
            float x = 0.f;
            for (int k = 0; k < groups; k++) x += part[k * rank + r];
            dst[r] = x;
        }
        return;
    }
    for (int r0 = 0; r0 < rank; r0 += blockDim.x * 4) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int dd = 0; dd < plain; dd++) {
            const float qv = qs[dd];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int r = r0 + t + (int)blockDim.x * j;
                if (r < rank) acc[j] = fmaf(qv, to_f32(ukh[(size_t)dd * rank + r]), acc[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = r0 + t + (int)blockDim.x * j;
            if (r < rank) dst[r] = acc[j];
        }
    }
}

// A line towards L2.  Nothing is read into the program, so that this may run before the wait for the kernels before it whatever they
// write: L2 is where their writes arrive.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory"); }

// The same for several tokens at a time, bfloat16: a block takes one head, 64 elements of the latent and up to TOK tokens, so that an
// element of Wuk is read once for all of them (a block a token and head read a head's whole matrix for one token: 17 MB from L2 for 16
// tokens of 16 heads of 64 x 512; 9 us there, 6 so, and 31 -> 14 for 64 tokens).  A lane has two neighbouring elements, a warp every fourth row of Wuk; the four
// warps' sums meet in shared memory.  The blocks behind the heads' do the tokens' rows.
constexpr int AR_THREADS = 128, AR_COLS = 64;

template <int TOK> constexpr size_t absorb_rows_smem(int plain) { return (size_t)(plain * TOK + 4 * TOK * AR_COLS) * sizeof(float); }

template <int TOK>
__global__ void __launch_bounds__(AR_THREADS)
latent_absorb_rows_kernel(const bf16* __restrict__ d, long long d_stride, const bf16* __restrict__ q, long long q_stride,
                          int n_heads, int plain, int rank, int rot, const float* __restrict__ norm_w, float eps,
                          const float* __restrict__ cos_t, const float* __restrict__ sin_t, int max_pos,
                          const int* __restrict__ tok_pos, const int* __restrict__ tok_seq, const int* __restrict__ seq_slot,
                          bf16* __restrict__ lat, LatentPages kv, const bf16* __restrict__ uk, float* __restrict__ qa, int M, int chunks) {
    ti_pdl_trigger();
    extern __shared__ __align__(16) float sm[];
    if ((int)blockIdx.x < n_heads * chunks) {            // (into L2 only: see prefetch_l2)
        const bf16* from = uk + (size_t)(blockIdx.x / chunks) * plain * rank + blockIdx.x % chunks * AR_COLS;
        for (int e = threadIdx.x; e < plain; e += AR_THREADS) prefetch_l2(from + (size_t)e * rank);
    }
    ti_pdl_sync();
    d = ti_dependent(d); q = ti_dependent(q);
    const int m0 = blockIdx.y * TOK, n = min(TOK, M - m0);
    if ((int)blockIdx.x >= n_heads * chunks) {
        const int i = blockIdx.x - n_heads * chunks;
        if (i < n)
            latent_prep_body<bf16>(sm, m0 + i, d, d_stride, (bf16*)nullptr, 0, n_heads, plain, rank, rot, norm_w, eps, cos_t, sin_t, max_pos, tok_pos,
                                   tok_seq, seq_slot, lat, kv);
        return;
    }
    const int h = blockIdx.x / chunks, chunk = blockIdx.x - h * chunks, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int hd = plain + rot, W = rank + rot, half = rot >> 1, r = chunk * AR_COLS + 2 * lane;
    float* qs = sm;                      // [plain][TOK]
    float* part = sm + plain * TOK;      // [4][TOK][AR_COLS]
    // (loads in batches, so that several are on their way at a time: a warp every fourth token, a lane every 32nd element)
    for (int e0 = 0; e0 < plain; e0 += 64) {
        float x[TOK / 4][2];
#pragma unroll
        for (int i = 0; i < TOK / 4; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int tok = warp + 4 * i, e = e0 + lane + 32 * j;
                x[i][j] = tok < n && e < plain ? to_f32(q[(size_t)(m0 + tok) * q_stride + (size_t)h * hd + e]) : 0.f;
            }
#pragma unroll
        for (int i = 0; i < TOK / 4; i++)
#pragma unroll
            for (int j = 0; j < 2; j++)
                if (e0 + lane + 32 * j < plain) qs[(e0 + lane + 32 * j) * TOK + warp + 4 * i] = x[i][j];
    }
    // the rotated parts of the tokens chunk, chunk + chunks, ...
    for (int i = t; i < (n - chunk + chunks - 1) / chunks * half; i += AR_THREADS) {
        const int tok = chunk + i / half * chunks, e = i % half;
        if (tok >= n) continue;
        const bf16* qh = q + (size_t)(m0 + tok) * q_stride + (size_t)h * hd + plain;
        float* dst = qa + ((size_t)(m0 + tok) * n_heads + h) * W + rank;
        const int pos = min(max(tok_pos[m0 + tok], 0), max_pos - 1);
        // (rounded to the engine's type as the rotation in place would have left it)
        const float u = to_f32(qh[e]), v = to_f32(qh[e + half]), c = cos_t[(size_t)pos * half + e], sn = sin_t[(size_t)pos * half + e];
        dst[e] = to_f32(from_f32<bf16>(u * c - v * sn));
        dst[e + half] = to_f32(from_f32<bf16>(v * c + u * sn));
    }
    __syncthreads();
    float acc[TOK][2];
#pragma unroll
    for (int i = 0; i < TOK; i++) acc[i][0] = acc[i][1] = 0.f;
    const bf16* from = uk + (size_t)h * plain * rank + r;
    for (int e0 = warp; e0 < plain; e0 += 4 * 16) {
        uint32_t w[16];
#pragma unroll
        for (int j = 0; j < 16; j++) w[j] = e0 + 4 * j < plain && r < rank ? *reinterpret_cast<const uint32_t*>(from + (size_t)(e0 + 4 * j) * rank) : 0u;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            if (e0 + 4 * j >= plain) break;
            const float w0 = __uint_as_float(w[j] << 16), w1 = __uint_as_float(w[j] & 0xffff0000u);
#pragma unroll
            for (int i = 0; i < TOK; i += 4) {
                const float4 x = *reinterpret_cast<const float4*>(qs + (e0 + 4 * j) * TOK + i);
                acc[i][0] = fmaf(x.x, w0, acc[i][0]); acc[i][1] = fmaf(x.x, w1, acc[i][1]);
                acc[i + 1][0] = fmaf(x.y, w0, acc[i + 1][0]); acc[i + 1][1] = fmaf(x.y, w1, acc[i + 1][1]);
                acc[i + 2][0] = fmaf(x.z, w0, acc[i + 2][0]); acc[i + 2][1] = fmaf(x.z, w1, acc[i + 2][1]);
                acc[i + 3][0] = fmaf(x.w, w0, acc[i + 3][0]); acc[i + 3][1] = fmaf(x.w, w1, acc[i + 3][1]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TOK; i++) *reinterpret_cast<float2*>(part + (warp * TOK + i) * AR_COLS + 2 * lane) = make_float2(acc[i][0], acc[i][1]);
    __syncthreads();
    for (int i = t; i < n * AR_COLS; i += AR_THREADS) {
        const int tok = i / AR_COLS, e = i - tok * AR_COLS;
        if (chunk * AR_COLS + e < rank)
            qa[((size_t)(m0 + tok) * n_heads + h) * W + chunk * AR_COLS + e] =
                (part[i] + part[TOK * AR_COLS + i]) + (part[2 * TOK * AR_COLS + i] + part[3 * TOK * AR_COLS + i]);
    }
}

template <int TOK>
int launch_absorb_rows(const void* d, long long d_stride, const void* q, long long q_stride, int n_heads, int plain, int rank, int rot,
                       const float* norm_w, float eps, const float* cos_t, const float* sin_t, int max_pos, const int* tok_pos,
                       const int* tok_seq, const int* seq_slot, void* lat, const LatentPages& kv, const void* uk, float* qa, int M, size_t row,
                       cudaStream_t stream) {
    const int chunks = (rank + AR_COLS - 1) / AR_COLS;
    const size_t smem = std::max(row, absorb_rows_smem<TOK>(plain));
    // (below 48 KB: the entry takes heads of up to 512 elements here and refuses longer rows)
    TI_CUDA(ti_launch_class<2>(latent_absorb_rows_kernel<TOK>, dim3(n_heads * chunks + std::min(M, TOK), (M + TOK - 1) / TOK), dim3(AR_THREADS), smem, stream,
                               (const bf16*)d, d_stride, (const bf16*)q, q_stride, n_heads, plain, rank, rot, norm_w, eps, cos_t, sin_t, max_pos,
                               tok_pos, tok_seq, seq_slot, (bf16*)lat, kv, (const bf16*)uk, qa, M, chunks));
    TI_CHECK_LAUNCH("latent_prep_absorb");
    return 0;
}

// For steps of few tokens: the merge of the key splits and the way out through Wuv in one launch.  Block (token, head):
// the splits' unnormalised sums are weighed and added into the latent result (shared memory), then
// o[v] = sum_r uv[h, v, r] * result[r], a warp per output element, four elements at a time.
template <typename T>
__global__ void __launch_bounds__(512)
latent_merge_expand_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, const T* __restrict__ uv,
                           T* __restrict__ o, long long o_stride, int n_heads, int vdim, int rank, int n_splits,
                           const T* __restrict__ gate, long long gate_stride) {
    ti_pdl_trigger();
    extern __shared__ float res[];       // [rank], then [64] weights
    float* w_s = res + rank;
    if (sizeof(T) == 2)          // the head's Wuv towards L2 meanwhile, a part a token (see prefetch_l2)
        for (int i = ((int)blockIdx.x * blockDim.x + threadIdx.x) * 64; i < vdim * rank; i += gridDim.x * blockDim.x * 64) prefetch_l2(uv + (size_t)blockIdx.y * vdim * rank + i);
    ti_pdl_sync();
    part_o = ti_dependent(part_o); part_ml = ti_dependent(part_ml);
    const int b = blockIdx.x, h = blockIdx.y, t = threadIdx.x;
    const size_t base = ((size_t)b * n_heads + h) * n_splits;
    // every warp: the splits' maxima and denominators, two a lane (n_splits is at most 64)
    float ms[2], ls[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int s = (t & 31) + 32 * j;
        const float2 ml = s < n_splits ? *reinterpret_cast<const float2*>(part_ml + (base + s) * 2) : make_float2(-INFINITY, 0.f);
        ms[j] = ml.x; ls[j] = ml.y;
    }
    const float m = warp_max(fmaxf(ms[0], ms[1]));
    float l = 0.f;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const float w = ms[j] > -INFINITY ? expf(ms[j] - m) : 0.f;
        l += w > 0.f ? w * ls[j] : 0.f;
        if (t < 32) w_s[t + 32 * j] = w;
    }
    l = warp_sum(l);
    const unsigned some = __ballot_sync(0xffffffffu, ms[0] > -INFINITY), more = __ballot_sync(0xffffffffu, ms[1] > -INFINITY);
    const int last = more ? 64 - __clz(more) : 32 - __clz(some);      // (the splits behind are empty)
    __syncthreads();
    float inv = l > 0.f ? 1.f / l : 0.f;
    if (gate) inv *= head_gate(ti_dependent(gate), gate_stride, b, h);      // (the way out is linear)
    for (int e = t; e < rank; e += blockDim.x) {
        float acc = 0.f;
        for (int s0 = 0; s0 < last; s0 += 16) {          // sixteen splits' numbers on their way together
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; j++)         // (an empty split's numbers were never written)
                x[j] = s0 + j < last && w_s[s0 + j] > 0.f ? part_o[(base + s0 + j) * rank + e] : 0.f;
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (s0 + j < last) acc = fmaf(w_s[s0 + j], x[j], acc);
        }
        res[e] = acc * inv;
    }
    __syncthreads();
    const int warp = t >> 5, lane = t & 31, rows = (blockDim.x >> 5) * 4;
    if (sizeof(T) == 2 && (rank & 7) == 0 && (reinterpret_cast<uintptr_t>(uv) & 15) == 0) {
        // 16-byte pieces of four rows at a time: eight loads on their way per lane
        for (int v0 = warp * 4; v0 < vdim; v0 += rows) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
            for (int c = lane; c < (rank >> 3); c += 32) {
                uint4 w[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    w[j] = v0 + j < vdim ? reinterpret_cast<const uint4*>(uv + ((size_t)h * vdim + v0 + j) * rank)[c] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const bf16* wv = reinterpret_cast<const bf16*>(&w[j]);
#pragma unroll
                    for (int e = 0; e < 8; e++) acc[j] = fmaf(to_f32(wv[e]), res[c * 8 + e], acc[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float sum = warp_sum(acc[j]);
                if (lane == 0 && v0 + j < vdim) o[(size_t)b * o_stride + (size_t)h * vdim + v0 + j] = from_f32<T>(sum);
            }
        }
        return;
    }
    for (int v0 = warp * 4; v0 < vdim; v0 += rows) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int r = lane; r < rank; r += 32) {
            const float x = res[r];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (v0 + j < vdim) acc[j] = fmaf(to_f32(uv[((size_t)h * vdim + v0 + j) * rank + r]), x, acc[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float sum = warp_sum(acc[j]);
            if (lane == 0 && v0 + j < vdim) o[(size_t)b * o_stride + (size_t)h * vdim + v0 + j] = from_f32<T>(sum);
        }
    }
}

template <typename T>
__global__ void latent_store_kernel(const T* __restrict__ lat, int W, const int* __restrict__ tok_pos,
                                    const int* __restrict__ tok_seq, const int* __restrict__ seq_slot, LatentPages kv) {
    ti_pdl_trigger();
    ti_pdl_sync();
    lat = ti_dependent(lat);
    const int m = blockIdx.x;
    store_row_to_pages<T>(kv, seq_slot[tok_seq[m]], tok_seq[m], tok_pos[m], W, lat + (size_t)m * W, threadIdx.x, blockDim.x);
}

// ---------------------------------------------------------------------------
// qa[m, h, 0:rank] = sum_d q[m, h, d] * uk[h, d, 0:rank];  qa[m, h, rank:] = q[m, h, plain:]
// uk: [heads * plain, rank] (row (h, d)).  Grid (token tiles of TM, heads), 128 threads over the rank.
constexpr int ABS_TM = 8, ABS_THREADS = 128, ABS_RPT = 2;      // a block: 8 tokens, one head, 256 elements of the latent (grid.z)

template <typename T>
__global__ void __launch_bounds__(ABS_THREADS)
latent_absorb_kernel(const T* __restrict__ q, long long q_stride, const T* __restrict__ uk, float* __restrict__ qa,
                     int M, int n_heads, int plain, int rank, int rot) {
    ti_pdl_trigger();
    extern __shared__ float qs[];        // [TM][plain]
    ti_pdl_sync();
    q = ti_dependent(q);
    const int m0 = blockIdx.x * ABS_TM, h = blockIdx.y, t = threadIdx.x;
    const int hd = plain + rot, W = rank + rot;
    for (int idx = t; idx < ABS_TM * plain; idx += ABS_THREADS) {
        const int mm = idx / plain, dd = idx - mm * plain;
        qs[idx] = (m0 + mm < M) ? to_f32(q[(size_t)(m0 + mm) * q_stride + (size_t)h * hd + dd]) : 0.f;
    }
    for (int idx = t; idx < ABS_TM * rot && blockIdx.z == 0; idx += ABS_THREADS) {
        const int mm = idx / rot, dd = idx - mm * rot;
        if (m0 + mm < M)
            qa[((size_t)(m0 + mm) * n_heads + h) * W + rank + dd] = to_f32(q[(size_t)(m0 + mm) * q_stride + (size_t)h * hd + plain + dd]);
    }
    __syncthreads();
    const T* ukh = uk + (size_t)h * plain * rank;
    {
        const int r0 = blockIdx.z * ABS_THREADS * ABS_RPT;
        float acc[ABS_RPT][ABS_TM];
#pragma unroll
        for (int j = 0; j < ABS_RPT; j++)
#pragma unroll
            for (int mm = 0; mm < ABS_TM; mm++) acc[j][mm] = 0.f;
#pragma unroll 4
        for (int dd = 0; dd < plain; dd++) {
            float wv[ABS_RPT];
#pragma unroll
            for (int j = 0; j < ABS_RPT; j++) {
                const int r = r0 + t + j * ABS_THREADS;
                wv[j] = r < rank ? to_f32(ukh[(size_t)dd * rank + r]) : 0.f;
            }
#pragma unroll
            for (int mm = 0; mm < ABS_TM; mm++) {
                const float qv = qs[mm * plain + dd];
#pragma unroll
                for (int j = 0; j < ABS_RPT; j++) acc[j][mm] = fmaf(qv, wv[j], acc[j][mm]);
            }
        }
#pragma unroll
        for (int j = 0; j < ABS_RPT; j++) {
            const int r = r0 + t + j * ABS_THREADS;
            if (r < rank)
#pragma unroll
                for (int mm = 0; mm < ABS_TM; mm++)
                    if (m0 + mm < M) qa[((size_t)(m0 + mm) * n_heads + h) * W + r] = acc[j][mm];
        }
    }
}

// o[m, h, v] = sum_r uv[h, v, r] * ol[m, h, r].  uv: [heads * vdim, rank].  Grid (token tiles, heads);
// a warp per output element row v, lanes along the rank.
constexpr int EXP_TM = 8, EXP_THREADS = 128, EXP_VB = 16;      // a block: 8 tokens, one head, 16 output elements (grid.z)

template <typename T>
__global__ void __launch_bounds__(EXP_THREADS)
latent_expand_kernel(const float* __restrict__ ol, const T* __restrict__ uv, T* __restrict__ o, long long o_stride,
                     int M, int n_heads, int vdim, int rank, const T* __restrict__ gate, long long gate_stride) {
    ti_pdl_trigger();
    extern __shared__ float os[];        // [TM][rank]
    ti_pdl_sync();
    ol = ti_dependent(ol); gate = ti_dependent(gate);
    const int m0 = blockIdx.x * EXP_TM, h = blockIdx.y, t = threadIdx.x;
    for (int idx = t; idx < EXP_TM * rank; idx += EXP_THREADS) {
        const int mm = idx / rank, r = idx - mm * rank;
        os[idx] = (m0 + mm < M) ? ol[((size_t)(m0 + mm) * n_heads + h) * rank + r] : 0.f;
    }
    __syncthreads();
    const int warp = t >> 5, lane = t & 31;
    const int v_end = min(vdim, (int)(blockIdx.z + 1) * EXP_VB);
    for (int v = blockIdx.z * EXP_VB + warp; v < v_end; v += EXP_THREADS / 32) {
        const T* wrow = uv + ((size_t)h * vdim + v) * rank;
        float acc[EXP_TM];
#pragma unroll
        for (int mm = 0; mm < EXP_TM; mm++) acc[mm] = 0.f;
        for (int r = lane; r < rank; r += 32) {
            const float wv = to_f32(wrow[r]);
#pragma unroll
            for (int mm = 0; mm < EXP_TM; mm++) acc[mm] = fmaf(wv, os[mm * rank + r], acc[mm]);
        }
#pragma unroll
        for (int mm = 0; mm < EXP_TM; mm++) {
            const float s = warp_sum(acc[mm]);
            if (lane == 0 && m0 + mm < M)
                o[(size_t)(m0 + mm) * o_stride + (size_t)h * vdim + v] = from_f32<T>(gate ? s * head_gate(gate, gate_stride, m0 + mm, h) : s);
        }
    }
}

// ---------------------------------------------------------------------------
// Keys and values per head after all, for steps of whole prompts on the tensor cores: from the up-projection's output
// ku[m] = [Wuk c | Wuv c] (heads * plain, then heads * vdim) and the step's rows, the padded heads
//     Q[m, h] = [q plain | q rotated | 0],  K[m, h] = [Wuk_h c | r | 0],  V[m, h] = [Wuv_h c | 0]      (D elements each)
// that a plain multi-head attention kernel takes.  One block per token.
template <typename T>
__global__ void latent_pack_kernel(const T* __restrict__ q, long long q_stride, const T* __restrict__ ku, const T* __restrict__ lat,
                                   T* __restrict__ Qp, T* __restrict__ Kp, T* __restrict__ Vp, int n_heads, int plain, int rot,
                                   int vdim, int rank, int D) {
    ti_pdl_trigger();
    ti_pdl_sync();
    q = ti_dependent(q); ku = ti_dependent(ku); lat = ti_dependent(lat);
    const size_t m = blockIdx.x;
    const int hd = plain + rot, W = rank + rot;
    const T* qrow = q + m * q_stride;
    const T* krow = ku + m * ((size_t)n_heads * (plain + vdim));
    const T* vrow = krow + (size_t)n_heads * plain;
    const T* rrow = lat + m * W + rank;
    const T zero = from_f32<T>(0.f);
    for (int idx = threadIdx.x; idx < n_heads * D; idx += blockDim.x) {
        const int h = idx / D, e = idx - h * D;
        const size_t o = (m * n_heads + h) * D + e;
        Qp[o] = e < hd ? qrow[(size_t)h * hd + e] : zero;
        Kp[o] = e < plain ? krow[(size_t)h * plain + e] : e < hd ? rrow[e - plain] : zero;
        Vp[o] = e < vdim ? vrow[(size_t)h * vdim + e] : zero;
    }
}

// ---------------------------------------------------------------------------
// The attention.  A block works on 32 rows = QB consecutive queries of a sequence times HB heads
// (HB * QB == 32) against key tiles of 32 positions; thread t works on row t / 4, its 4 threads split
// a tile's keys (scores) and the latent's elements (output) between them.
constexpr int LQ = 32, LK = 32, LTHREADS = 128;

template <typename T, int MAXC>
__global__ void __launch_bounds__(LTHREADS)
latent_attn_kernel(const float* __restrict__ qa, const T* __restrict__ lat, float* __restrict__ ol,
                   const int* __restrict__ cu_new, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                   int n_heads, int hb, int rank, int rot, float scale, int window, const float* __restrict__ sink,
                   LatentPages kv, int n_splits, float* __restrict__ part_o, float* __restrict__ part_ml) {
    ti_pdl_trigger();
    extern __shared__ float sm[];
    ti_pdl_sync();
    qa = ti_dependent(qa); lat = ti_dependent(lat);
    const int W = rank + rot, ld = W + 1;
    float* Qs = sm;                       // [LQ][ld]
    float* Ks = Qs + LQ * ld;             // [LK][ld]
    float* Ps = Ks + LK * ld;             // [LQ][LK + 1]
    const int qb = LQ / hb;
    // with n_splits > 1 the key tiles of a block's queries are shared out over n_splits blocks, which leave their
    // unnormalised sums, maxima and denominators for the merging kernel
    const int split = blockIdx.x % n_splits;
    const int b = blockIdx.z, h0 = blockIdx.y * hb, q0 = (blockIdx.x / n_splits) * qb;
    const int tok0 = cu_new[b];
    const int n = cu_new[b + 1] - tok0;
    if (q0 >= n) return;
    const int start = seq_start[b], slot = seq_slot[b], end = start + n;
    const int t = threadIdx.x, r = t >> 2, c4 = t & 3;
    // row rr: query q0 + rr / hb, head h0 + rr % hb
    for (int idx = t; idx < LQ * W; idx += LTHREADS) {
        const int rr = idx / W, e = idx - rr * W;
        const int qq = q0 + rr / hb, hh = h0 + rr % hb;
        Qs[rr * ld + e] = (qq < n && hh < n_heads) ? qa[((size_t)(tok0 + qq) * n_heads + hh) * W + e] : 0.f;
    }
    const int my_q = q0 + r / hb, my_h = h0 + r % hb;
    const bool row_ok = my_q < n && my_h < n_heads;
    const int qi = start + my_q;
    float acc[MAXC];
#pragma unroll
    for (int c = 0; c < MAXC; c++) acc[c] = 0.f;
    // the sink stands in the denominator from the start: running maximum sink_h, running sum 1
    float m_run = -INFINITY, l_run = 0.f;
    if (sink && row_ok && split == 0) { m_run = sink[my_h]; l_run = 1.f; }
    const int nc = (rank + 3) >> 2;      // elements of the latent per thread (c4 + 4 c)
    const int last_q = start + min(q0 + qb, n) - 1;
    const int lo = window > 0 ? max(0, start + q0 - window + 1) : 0;
    const int kt_first = lo / LK, kt_last = last_q / LK;
    const int per = (kt_last - kt_first + n_splits) / n_splits;
    const int kt_a = kt_first + split * per, kt_b = min(kt_last, kt_a + per - 1);
    for (int kt = kt_a; kt <= kt_b; kt++) {
        const int k0 = kt * LK;
        __syncthreads();
        // a warp fetches whole rows: where a row lives is worked out once, then the lanes run along it
        for (int rr = t >> 5; rr < LK; rr += LTHREADS / 32) {
            const int p = k0 + rr;
            const T* src = nullptr;
            if (p >= start) {
                if (p < end) src = lat + (size_t)(tok0 + p - start) * W;
            } else if (p >= lo) {
                const int row = kv.ring_rows > 0 ? p % kv.ring_rows : p;
                const int pidx = row / kv.page_size;
                const int page = pidx < kv.table_width ? kv.page_table[(size_t)slot * kv.table_width + pidx] : -1;
                if (page >= 0 && page < kv.n_pages) src = (const T*)kv.pages + ((size_t)page * kv.page_size + row % kv.page_size) * W;
            }
            for (int e = t & 31; e < W; e += 32) Ks[rr * ld + e] = src ? to_f32(src[e]) : 0.f;
        }
        __syncthreads();
        float s[8];
#pragma unroll
        for (int c = 0; c < 8; c++) s[c] = 0.f;
        const float* qrow = Qs + r * ld;
        for (int e = 0; e < W; e++) {
            const float qv = qrow[e];
#pragma unroll
            for (int c = 0; c < 8; c++) s[c] = fmaf(qv, Ks[(c4 + 4 * c) * ld + e], s[c]);
        }
        float m_tile = -INFINITY;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int kj = k0 + c4 + 4 * c;
            const bool ok = row_ok && kj <= qi && kj < end && (window <= 0 || kj > qi - window);
            s[c] = ok ? s[c] * scale : -INFINITY;
            m_tile = fmaxf(m_tile, s[c]);
        }
        m_tile = fmaxf(m_tile, __shfl_xor_sync(0xffffffffu, m_tile, 1));
        m_tile = fmaxf(m_tile, __shfl_xor_sync(0xffffffffu, m_tile, 2));
        const float m_new = fmaxf(m_run, m_tile);
        float alpha = 1.f, l_tile = 0.f;
        if (m_new > -INFINITY) {
            alpha = expf(m_run - m_new);
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float p = expf(s[c] - m_new);
                Ps[r * (LK + 1) + c4 + 4 * c] = p;
                l_tile += p;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 8; c++) Ps[r * (LK + 1) + c4 + 4 * c] = 0.f;
        }
        l_tile += __shfl_xor_sync(0xffffffffu, l_tile, 1);
        l_tile += __shfl_xor_sync(0xffffffffu, l_tile, 2);
        l_run = l_run * alpha + l_tile;
        m_run = m_new;
        __syncwarp();
#pragma unroll
        for (int c = 0; c < MAXC; c++)
            if (c < nc) acc[c] *= alpha;
        const float* prow = Ps + r * (LK + 1);
        for (int j = 0; j < LK; j++) {
            const float p = prow[j];
            const float* vrow = Ks + j * ld + c4;
#pragma unroll
            for (int c = 0; c < MAXC; c++)
                if (c < nc) acc[c] = fmaf(p, vrow[4 * c], acc[c]);      // (an element past the rank is the rotated part: never stored)
        }
    }
    if (row_ok && n_splits > 1) {
        const size_t at = ((size_t)(tok0 + my_q) * n_heads + my_h) * n_splits + split;
        if (c4 == 0) { part_ml[at * 2] = m_run; part_ml[at * 2 + 1] = l_run; }
#pragma unroll
        for (int c = 0; c < MAXC; c++)
            if (c < nc && c4 + 4 * c < rank) part_o[at * rank + c4 + 4 * c] = acc[c];
    } else if (row_ok) {
        const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
        float* orow = ol + ((size_t)(tok0 + my_q) * n_heads + my_h) * rank;
#pragma unroll
        for (int c = 0; c < MAXC; c++)
            if (c < nc && c4 + 4 * c < rank) orow[c4 + 4 * c] = acc[c] * inv;
    }
}

// ---------------------------------------------------------------------------
// One query per sequence, bfloat16, on the tensor cores (`mma.sync m16n8k16`, float32 accumulation).  A block takes one
// sequence, 16 * MT heads and one share of the keys, 32 positions at a time: the rows [c | r] of a tile go to shared memory
// as they are; S = Qa L^T (every warp a quarter of a row's elements for all 32 keys; the quarters meet in shared memory), the softmax
// in 32-bit (a warp four heads of every 16), P rounded to bfloat16 as the second product's operand, O += P L[:, :rank] (the latent's
// columns shared out over the warps).  Unnormalised sums, maxima and denominators go to the merging kernel when the keys are split.
// Rows of a tile outside the query's reach are zeroed: a weight of zero times whatever stood there must stay zero.
//
// What bounds it: a tile's chain of steps.  A tile is on its way (a bulk copy a row) while the one before it is worked off, and two
// blocks share an SM where there is room; 16 sequences of 1,000 to 4,000 positions, 16 heads, rows of 512 + 64, us a tile of a block:
// the queue of copies and the look-up of the next tile's page 1.4 -> 0.2 (16-byte copies by all threads before, the page's number
// awaited at once), scores 0.9 -> 0.5 (queries in registers where they fit), softmax and its two barriers 0.5, values 0.65.  The longest
// sequence's blocks end last (7 tiles where the mean is 4): splits of equally many tiles over all sequences took 53.4 us for the layer's
// step where these take 59.2 (66.2 before), 196 and 312 for 32 sequences of up to 8,000 with 32 heads, but a sequence's results then
// changed by 0.0025 with the lengths of the others beside it.  The way into the latent before it 9 -> 6; the merge and the way out after
// it 12, bound by 34 MB of Wuv from L2 (a cluster of eight blocks that read it once, shared their results and took 13: not kept).
constexpr int DK = 32, D_THREADS = 128;

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ld_matrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ld_matrix4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

constexpr int Q_STEPS = 10;          // QREG: steps of 16 elements of a row that a warp has at most (rows of up to 640)

// Scores of a tile as the warps leave them: [shares][ROWS][pitch] floats, 32 keys a row; later a row's weights (bfloat16, in place) and,
// behind them, the factor of its sums so far.
constexpr int S_FACTOR = 16;         // where in a row of 32 floats that factor stands
struct DecodeShape { int tiles, shares, pitch; size_t smem; };
template <int MT, bool QREG> DecodeShape decode_mma_shape(int W) {
    auto bytes = [&](int tiles, int shares, int pitch) {
        return (size_t)((QREG ? 0 : 16 * MT) + tiles * DK) * (W + 8) * 2 + (size_t)shares * 16 * MT * pitch * 4;
    };
    DecodeShape s{2, 4, 40, 0};
    if (bytes(2, 4, 40) > 227 * 1024) s.tiles = 1;                                            // wide rows: one tile of them
    if (bytes(s.tiles, 4, 40) > 227 * 1024) { s.shares = 1; s.pitch = 32; }                  // the widest: the warps add to one place in turn
    s.smem = bytes(s.tiles, s.shares, s.pitch);
    return s;
}

// QREG: a warp's quarter of the queries stays in its registers (one tile of 16 heads, rows of up to 640 elements), else they lie in
// shared memory.
template <int MT, int NTW, bool QREG>
__global__ void __launch_bounds__(D_THREADS)
latent_decode_mma_kernel(const float* __restrict__ qa, const bf16* __restrict__ lat, float* __restrict__ ol,
                         const int* __restrict__ cu_new, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                         int n_heads, int rank, int rot, float scale, int window, const float* __restrict__ sink,
                         LatentPages kv, int n_splits, float* __restrict__ part_o, float* __restrict__ part_ml, int tiles,
                         int shares, int pitch, int* status) {
    ti_pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    constexpr int ROWS = 16 * MT;
    const int ahead = tiles - 1;                                   // (1, or 0: rows so wide that only one tile of them fits)
    const int W = rank + rot, LD = W + 8, steps = W >> 4;
    float* Sp = reinterpret_cast<float*>(smem_raw);
    bf16* Ls = reinterpret_cast<bf16*>(smem_raw + (size_t)shares * ROWS * pitch * 4);      // [tiles][DK][LD]
    // (the barriers stand in the 16 bytes between the first two rows, which nothing else uses: the widest rows leave no byte beside them)
    uint64_t* full = reinterpret_cast<uint64_t*>(Ls + W);
    if (tid == 0) { mbar_init(&full[0], 1); mbar_init(&full[1], 1); mbar_fence_init(); }
    __syncthreads();                     // (all warps wait on them below; here the meeting falls into the wait for the kernel before)
    ti_pdl_sync();
    qa = ti_dependent(qa); lat = ti_dependent(lat);
    bf16* Qs = Ls + tiles * DK * LD;                               // [ROWS][LD]
    const int split = blockIdx.z, h0 = blockIdx.y * ROWS, b = blockIdx.x;        // (the splits that are empty come last)
    const int tok = cu_new[b], tok_end = cu_new[b + 1], qi = seq_start[b], slot = seq_slot[b];
    if (tok_end - tok <= 0) return;
    const int lo = window > 0 ? max(0, qi - window + 1) : 0;
    const int kt_first = lo / DK, kt_last = qi / DK;
    // (equal parts of the sequence's own keys: where a split ends decides what its weights are rounded against, so that this must not
    // follow from the other sequences of the step)
    const int per = (kt_last - kt_first + n_splits) / n_splits;
    const int kt_a = kt_first + split * per, kt_b = min(kt_last, kt_a + per - 1);
    const int n_tiles8 = rank >> 3;
    if (kt_a > kt_last && part_o != nullptr) {                     // nothing is left for this split
        for (int r = tid; r < ROWS; r += D_THREADS)
            if (h0 + r < n_heads) {
                float* ml = part_ml + (((size_t)tok * n_heads + h0 + r) * n_splits + split) * 2;
                ml[0] = -INFINITY; ml[1] = 0.f;
            }
        return;
    }
    // The first warp brings the tiles, a lane a row: one bulk copy each, zeros where the row is out of the query's reach.  Where the
    // tiles lie is looked up for 32 of them at a time, a lane a tile (a tile lies inside one page): looked up tile by tile, the chain of
    // a load and its use cost the warp 1.4 us of every tile's 3.5.
    const bool whole = kv.page_size % DK == 0;                     // (else row by row)
    auto row_at = [&](int p) -> long long {                        // of position p among the cache's rows, or -1
        const int row = kv.ring_rows > 0 ? p % kv.ring_rows : p;
        const int pidx = row / kv.page_size;
        const int page = pidx < kv.table_width ? kv.page_table[(size_t)slot * kv.table_width + pidx] : -1;
        return page >= 0 && page < kv.n_pages ? (long long)page * kv.page_size + row % kv.page_size : -1;
    };
    long long tile_row = -1;                                       // of the first position of tile kt_a + 32 n + lane
    if (whole && warp == 0 && kt_a + lane <= kt_b) tile_row = row_at((kt_a + lane) * DK);
    uint32_t qf[QREG ? Q_STEPS : 1][4];
    float2 qx[QREG ? Q_STEPS : 1][4];
    if constexpr (QREG) {
        const float* q0 = qa + ((size_t)tok * n_heads + h0 + g) * W + 2 * t4;
        const bool ok0 = h0 + g < n_heads, ok1 = h0 + g + 8 < n_heads;
#pragma unroll
        for (int i = 0; i < Q_STEPS; i++) {
            const int ks = warp + 4 * i;
#pragma unroll
            for (int j = 0; j < 4; j++)          // (row g, k), (row g + 8, k), (row g, k + 8), (row g + 8, k + 8)
                qx[i][j] = ks < steps && (j & 1 ? ok1 : ok0) ? *reinterpret_cast<const float2*>(q0 + (size_t)(j & 1) * 8 * W + ks * 16 + (j >> 1) * 8) : make_float2(0.f, 0.f);
        }
    }
    auto fetch = [&](int kt) {                   // by the whole first warp
        const int nth = kt - kt_a, at = nth & ahead, p = kt * DK + lane;
        if (whole && nth > 0 && (nth & 31) == 0) tile_row = kt + lane <= kt_b ? row_at((kt + lane) * DK) : -1;
        long long row = whole ? __shfl_sync(0xffffffffu, tile_row, nth & 31) : -1;
        if (whole) row += row >= 0 ? lane : 0;
        else if (p >= lo && p < qi) row = row_at(p);
        const bf16* src = p == qi ? lat + (size_t)tok * W : p >= lo && p < qi && row >= 0 ? (const bf16*)kv.pages + (size_t)row * W : nullptr;
        bf16* to = Ls + (size_t)(at * DK + lane) * LD;
        const int live = __popc(__ballot_sync(0xffffffffu, src != nullptr));
        if (src == nullptr)
            for (int e = 0; e < W; e += 8) *reinterpret_cast<uint4*>(to + e) = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();             // (a place that held zeros is written by a copy next)
        if (lane == 0) { if (live) mbar_expect_tx(&full[at], (uint32_t)live * W * 2); else mbar_arrive(&full[at]); }
        __syncwarp();
        if (src != nullptr)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(to)), "l"(src), "r"(W * 2), "r"(smem_u32(&full[at])) : "memory");
    };
    const uint32_t ls0 = smem_u32(Ls), qs0 = smem_u32(Qs), sp0 = smem_u32(Sp);
    if (warp == 0) fetch(kt_a);
    if constexpr (QREG) {
#pragma unroll
        for (int i = 0; i < Q_STEPS; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const __nv_bfloat162 p = __floats2bfloat162_rn(qx[i][j].x, qx[i][j].y);
                qf[i][j] = *reinterpret_cast<const uint32_t*>(&p);
            }
    } else {
        // (global loads in batches, so that several are on their way at a time)
        const int per_row = W >> 2, total = ROWS * per_row;        // pieces of four floats
        for (int i0 = 0; i0 < total; i0 += 12 * D_THREADS) {
            float4 x[12];
#pragma unroll
            for (int u = 0; u < 12; u++) {
                const int idx = i0 + u * D_THREADS + tid, r = idx / per_row, e = idx - r * per_row;
                x[u] = (idx < total && h0 + r < n_heads) ? reinterpret_cast<const float4*>(qa + ((size_t)tok * n_heads + h0 + r) * W)[e]
                                                         : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < 12; u++) {
                const int idx = i0 + u * D_THREADS + tid, r = idx / per_row, e = idx - r * per_row;
                if (idx < total) {
                    const __nv_bfloat162 a = __floats2bfloat162_rn(x[u].x, x[u].y), c = __floats2bfloat162_rn(x[u].z, x[u].w);
                    *reinterpret_cast<uint2*>(Qs + r * LD + 4 * e) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&c));
                }
            }
        }
    }
    // The softmax: a warp has four rows of every 16, a lane four of a row's 32 keys.  The row's running maximum (the same in its eight
    // lanes) and this lane's share of the denominator:
    const int srow = warp * 4 + (lane >> 3), skey = (lane & 7) * 4;
    float m_run[MT], l_run[MT];
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        const int h = h0 + mt * 16 + srow;
        const bool with_sink = sink && split == 0 && h < n_heads;
        m_run[mt] = with_sink ? sink[h] : -INFINITY;
        l_run[mt] = with_sink && skey == 0 ? 1.f : 0.f;
    }
    float O[MT][NTW][4];
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int i = 0; i < NTW; i++)
#pragma unroll
            for (int c = 0; c < 4; c++) O[mt][i][c] = 0.f;
    bool ok = true;
    for (int kt = kt_a; kt <= kt_b; kt++) {
        const int nth = kt - kt_a;
        if (!mbar_wait(&full[nth & ahead], (uint32_t)((ahead ? nth >> 1 : nth) & 1))) { ti_report(status, TI_STATUS_TMA_WAIT); ok = false; }
        if (!__syncthreads_and(ok)) {            // (given up: not before the copies under way have arrived, or their wait has run out too)
            if (tid == 0) mbar_wait(&full[nth & ahead], (uint32_t)((ahead ? nth >> 1 : nth) & 1));
            __syncthreads();
            return;
        }                                // this tile is there (at first the queries too); the other place and the scores are no longer read
        if (ahead && kt < kt_b && warp == 0) fetch(kt + 1);
        const uint32_t ls = ls0 + (uint32_t)((nth & ahead) * DK * LD) * 2;
        // scores: this warp's steps of the rows' elements (every fourth) of all 32 keys
        {
            float c[MT][4][4] = {};
            const uint32_t kaddr = ls + (uint32_t)(((lane & 7) + ((lane >> 4) & 1) * 8) * LD + ((lane >> 3) & 1) * 8) * 2;
            const uint32_t qaddr = qs0 + (uint32_t)((lane & 15) * LD + (lane >> 4) * 8) * 2;
            auto step = [&](int ks, const uint32_t (&a)[MT][4]) {
                uint32_t k0[4], k1[4];       // keys 0-7 and 8-15, 16-23 and 24-31: two halves of the step each
                ld_matrix4(k0, kaddr + (uint32_t)(ks * 16) * 2);
                ld_matrix4(k1, kaddr + (uint32_t)(16 * LD + ks * 16) * 2);
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    mma_bf16_16816(c[mt][0], a[mt], k0[0], k0[1]);
                    mma_bf16_16816(c[mt][1], a[mt], k0[2], k0[3]);
                    mma_bf16_16816(c[mt][2], a[mt], k1[0], k1[1]);
                    mma_bf16_16816(c[mt][3], a[mt], k1[2], k1[3]);
                }
            };
            if constexpr (QREG) {
#pragma unroll
                for (int i = 0; i < Q_STEPS; i++)
                    if (warp + 4 * i < steps) {
                        const uint32_t a[1][4] = {{qf[i][0], qf[i][1], qf[i][2], qf[i][3]}};
                        step(warp + 4 * i, a);
                    }
            } else {
#pragma unroll 4
                for (int ks = warp; ks < steps; ks += 4) {
                    uint32_t a[MT][4];
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) ld_matrix4(a[mt], qaddr + (uint32_t)(mt * 16 * LD + ks * 16) * 2);
                    step(ks, a);
                }
            }
            for (int w = 0; w < 4; w++) {
                if (shares == 4 ? w == 0 : w == warp) {
                    float* mine = Sp + (size_t)(shares == 4 ? warp : 0) * ROWS * pitch + 2 * t4;
                    const bool add = shares == 1 && warp > 0;
#pragma unroll
                    for (int mt = 0; mt < MT; mt++)
#pragma unroll
                        for (int nt = 0; nt < 4; nt++)
#pragma unroll
                            for (int r = 0; r < 2; r++) {
                                float2* at = reinterpret_cast<float2*>(mine + (mt * 16 + g + 8 * r) * pitch + nt * 8);
                                const float2 had = add ? *at : make_float2(0.f, 0.f);
                                *at = make_float2(had.x + c[mt][nt][2 * r], had.y + c[mt][nt][2 * r + 1]);
                            }
                }
                __syncthreads();
                if (shares == 4) break;
            }
        }
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            float* row = Sp + (mt * 16 + srow) * pitch;
            float4 x = *reinterpret_cast<const float4*>(row + skey);
            if (shares == 4) {
                const float4 x1 = *reinterpret_cast<const float4*>(row + ROWS * pitch + skey), x2 = *reinterpret_cast<const float4*>(row + 2 * ROWS * pitch + skey);
                const float4 x3 = *reinterpret_cast<const float4*>(row + 3 * ROWS * pitch + skey);
                x = make_float4((x.x + x1.x) + (x2.x + x3.x), (x.y + x1.y) + (x2.y + x3.y), (x.z + x1.z) + (x2.z + x3.z), (x.w + x1.w) + (x2.w + x3.w));
            }
            const int p0 = kt * DK + skey;
            const bool head_ok = h0 + mt * 16 + srow < n_heads;
            float s[4] = {x.x, x.y, x.z, x.w}, mx = -INFINITY;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                s[e] = head_ok && p0 + e >= lo && p0 + e <= qi ? s[e] * scale : -INFINITY;
                mx = fmaxf(mx, s[e]);
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(mx, m_run[mt]), alpha = m_new > -INFINITY ? expf(m_run[mt] - m_new) : 1.f;
            m_run[mt] = m_new;
            float sum_e = 0.f;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                s[e] = s[e] == -INFINITY ? 0.f : expf(s[e] - m_new);
                sum_e += s[e];
            }
            l_run[mt] = l_run[mt] * alpha + sum_e;
            const __nv_bfloat162 p01 = __floats2bfloat162_rn(s[0], s[1]), p23 = __floats2bfloat162_rn(s[2], s[3]);
            __syncwarp();                // the row's scores have been read
            reinterpret_cast<uint2*>(row)[lane & 7] = make_uint2(*reinterpret_cast<const uint32_t*>(&p01), *reinterpret_cast<const uint32_t*>(&p23));
            if (skey == 0) row[S_FACTOR] = alpha;
        }
        __syncthreads();
        // O += P L: a warp has pairs of tiles of 8 columns of the latent, warp, warp + 4, ...
        uint32_t a[MT][2][4];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            const float f0 = Sp[(mt * 16 + g) * pitch + S_FACTOR], f1 = Sp[(mt * 16 + g + 8) * pitch + S_FACTOR];
            if (__any_sync(0xffffffffu, f0 != 1.f || f1 != 1.f)) {
#pragma unroll
                for (int i = 0; i < NTW; i++) {
                    O[mt][i][0] *= f0; O[mt][i][1] *= f0; O[mt][i][2] *= f1; O[mt][i][3] *= f1;
                }
            }
#pragma unroll
            for (int ks = 0; ks < 2; ks++) ld_matrix4(a[mt][ks], sp0 + (uint32_t)((mt * 16 + (lane & 15)) * pitch * 4 + ks * 32 + (lane >> 4) * 16));
        }
#pragma unroll
        for (int i = 0; i < NTW; i += 2) {
            const int nt = 2 * warp + 4 * i;                      // this tile and the next
            if (nt >= n_tiles8) continue;
            const int second = nt + 1 < n_tiles8 ? 8 : 0;         // (a latent of an odd number of tiles: the last one twice)
#pragma unroll
            for (int ks = 0; ks < 2; ks++) {
                uint32_t q[4];       // (keys 0-7, this tile), (keys 8-15, this), (keys 0-7, next), (keys 8-15, next), transposed on the way
                ld_matrix4_trans(q, ls + (uint32_t)((ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + nt * 8 + (lane >> 4) * second) * 2);
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    mma_bf16_16816(O[mt][i], a[mt][ks], q[0], q[1]);
                    mma_bf16_16816(O[mt][i + 1], a[mt][ks], q[2], q[3]);
                }
            }
        }
        if (!ahead && kt < kt_b) {
            __syncthreads();             // the one tile is no longer read
            if (warp == 0) fetch(kt + 1);
        }
    }
    if (part_o == nullptr) __syncthreads();
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        const int h = h0 + mt * 16 + srow;
        float l = l_run[mt];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (skey != 0) continue;
        if (part_o == nullptr) Sp[(mt * 16 + srow) * pitch + S_FACTOR] = l > 0.f ? 1.f / l : 0.f;
        else if (h < n_heads) {
            const size_t at = ((size_t)tok * n_heads + h) * n_splits + split;
            part_ml[at * 2] = m_run[mt]; part_ml[at * 2 + 1] = l;
        }
    }
    if (part_o == nullptr) __syncthreads();
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int r = mt * 16 + g + 8 * half, h = h0 + r;
            if (h >= n_heads) continue;
            float* dst = part_o != nullptr ? part_o + (((size_t)tok * n_heads + h) * n_splits + split) * rank : ol + ((size_t)tok * n_heads + h) * rank;
            const float f = part_o != nullptr ? 1.f : Sp[r * pitch + S_FACTOR];
#pragma unroll
            for (int i = 0; i < NTW; i++) {
                const int nt = 2 * warp + 4 * (i & ~1) + (i & 1);
                if (nt >= n_tiles8) continue;
                *reinterpret_cast<float2*>(dst + nt * 8 + 2 * t4) = make_float2(O[mt][i][2 * half] * f, O[mt][i][2 * half + 1] * f);
            }
        }
}

template <int MT, int NTW, bool QREG>
int launch_decode_form(const float* qa, const void* lat, float* ol, const int* cu_new, const int* seq_start, const int* seq_slot,
                       int n_seq, int n_heads, int rank, int rot, float scale, int window, const float* sink,
                       const LatentPages& kv, int n_splits, float* part_o, float* part_ml, cudaStream_t stream) {
    constexpr int ROWS = 16 * MT;
    const int W = rank + rot;
    const DecodeShape shape = decode_mma_shape<MT, QREG>(W);
    const size_t smem = shape.smem;
    int* status = ti_status_ptr();
    TI_REQUIRE(status != nullptr, "latent_attention: no status word");
    static size_t configured = 0;
    if (smem > 48 * 1024 && smem > configured) {
        TI_CUDA(cudaFuncSetAttribute(latent_decode_mma_kernel<MT, NTW, QREG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    dim3 grid(n_seq, (n_heads + ROWS - 1) / ROWS, n_splits);
    TI_CUDA(ti_launch_class<3>(latent_decode_mma_kernel<MT, NTW, QREG>, grid, dim3(D_THREADS), smem, stream, qa, (const bf16*)lat, ol, cu_new,
                               seq_start, seq_slot, n_heads, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, shape.tiles, shape.shares, shape.pitch, status));
    TI_CHECK_LAUNCH("latent_attention (one token, tensor cores)");
    return 0;
}

template <int MT, int NTW>
int launch_decode_mma(const float* qa, const void* lat, float* ol, const int* cu_new, const int* seq_start, const int* seq_slot,
                      int n_seq, int n_heads, int rank, int rot, float scale, int window, const float* sink,
                      const LatentPages& kv, int n_splits, float* part_o, float* part_ml, int n_tok, cudaStream_t stream,
                      const void* uv = nullptr, void* o = nullptr, long long o_stride = 0, int vdim = 0, const void* gate = nullptr,
                      long long gate_stride = 0) {
    int rc;
    if (MT == 1 && rank + rot <= 64 * Q_STEPS)
        rc = launch_decode_form<1, NTW, true>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, n_heads, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, stream);
    else
        rc = launch_decode_form<MT, NTW, false>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, n_heads, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, stream);
    if (rc) return rc;
    if (uv) {
        // (128 / 256 / 512 threads, us a layer of 16 sequences and 16 heads: a latent of 512 83 / 67 / 60, of 256 49 / 49 / 47; four
        // sequences, eight heads, a latent of 256 40 / 35 / 40)
        const size_t sm2 = (size_t)(rank + 64) * sizeof(float);
        TI_CUDA(ti_launch_class<4>(latent_merge_expand_kernel<bf16>, dim3(n_tok, n_heads), dim3(rank > 256 ? 512 : 256), sm2, stream, (const float*)part_o,
                                   (const float*)part_ml, (const bf16*)uv, (bf16*)o, o_stride, n_heads, vdim, rank, n_splits,
                                   (const bf16*)gate, gate_stride));
        TI_CHECK_LAUNCH("latent_merge_expand");
        return 0;
    }
    if (n_splits > 1) {
        int threads = ((rank + 3) / 4 + 31) / 32 * 32;
        TI_CUDA(ti_launch_class<4>(tiattn::attn_decode_combine_kernel<float>, dim3(n_tok, n_heads), dim3(threads), 0, stream,
                                   (const float*)part_o, (const float*)part_ml, ol, (long long)n_heads * rank, n_heads, rank, n_splits, (const bf16*)nullptr, 0LL));
        TI_CHECK_LAUNCH("latent_attention_combine");
    }
    return 0;
}

template <typename T, int MAXC>
int launch_attn(const float* qa, const void* lat, float* ol, const int* cu_new, const int* seq_start, const int* seq_slot,
                int n_seq, int max_new, int n_heads, int hb, int rank, int rot, float scale, int window, const float* sink,
                const LatentPages& kv, int n_splits, float* part_o, float* part_ml, int n_tok, cudaStream_t stream) {
    const int W = rank + rot;
    const size_t smem = ((size_t)(LQ + LK) * (W + 1) + (size_t)LQ * (LK + 1)) * sizeof(float);
    TI_REQUIRE(smem <= 227 * 1024, "latent_attention: rows of %d elements need %zu bytes of shared memory", W, smem);
    static size_t configured = 0;
    if (smem > configured) {
        TI_CUDA(cudaFuncSetAttribute(latent_attn_kernel<T, MAXC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    const int qb = LQ / hb;
    dim3 grid(((max_new + qb - 1) / qb) * n_splits, (n_heads + hb - 1) / hb, n_seq);
    TI_CUDA(ti_launch(latent_attn_kernel<T, MAXC>, grid, dim3(LTHREADS), smem, stream, qa, (const T*)lat, ol, cu_new, seq_start,
                      seq_slot, n_heads, hb, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml));
    TI_CHECK_LAUNCH("latent_attention");
    if (n_splits > 1) {
        // the splits' sums meet: one block per (token, head), the latent's elements over its threads
        int threads = ((rank + 3) / 4 + 31) / 32 * 32;
        TI_CUDA(ti_launch_class<4>(tiattn::attn_decode_combine_kernel<float>, dim3(n_tok, n_heads), dim3(threads), 0, stream,
                                   (const float*)part_o, (const float*)part_ml, ol, (long long)n_heads * rank, n_heads, rank, n_splits, (const bf16*)nullptr, 0LL));
        TI_CHECK_LAUNCH("latent_attention_combine");
    }
    return 0;
}

}  // namespace

// d[M, rank + rot] (row stride d_stride) is the down-projection's output; q[M, heads, plain + rot] or null;
// cos/sin: float32 [max_pos, rot / 2]; lat: [M, rank + rot] dense or null; pages null: no store.
extern "C" int ti_latent_prep(const void* d, long long d_stride, void* q, long long q_stride, int n_heads, int plain,
                              int rank, int rot, const float* norm_w, float eps, const float* cos_t, const float* sin_t,
                              int max_pos, const int* tok_pos, const int* tok_seq, const int* seq_slot, const int* seq_len,
                              void* lat, void* pages, const int* page_table, int table_width, int page_size, int ring_rows, int n_pages,
                              int M, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && rank > 0 && rot >= 0 && rot % 2 == 0 && plain >= 0, "latent_prep: bad sizes");
    TI_REQUIRE(rot == 0 || (cos_t && sin_t && max_pos > 0), "latent_prep: a rotated part needs cos and sin tables");
    TI_REQUIRE(!pages || (page_table && seq_len && page_size > 0 && table_width > 0 && n_pages > 0 && ring_rows % page_size == 0),
               "latent_prep: incomplete cache description");
    LatentPages kv{pages, page_table, table_width, page_size, ring_rows, n_pages, seq_len};
    const int W = rank + rot;
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        const size_t smem = (size_t)(W + 33) * sizeof(float) + (size_t)W * sizeof(T);
        TI_REQUIRE(smem <= 48 * 1024, "latent_prep: rows of %d elements are too long", W);
        TI_CUDA(ti_launch_class<2>(latent_prep_kernel<T>, dim3(M), dim3(128), smem, stream, (const T*)d, d_stride, (T*)q, q_stride,
                                   n_heads, plain, rank, rot, norm_w, eps, cos_t, sin_t, max_pos, tok_pos, tok_seq, seq_slot,
                                   (T*)lat, kv));
        TI_CHECK_LAUNCH("latent_prep");
        return 0;
    });
}

extern "C" int ti_latent_store(const void* lat, int W, const int* tok_pos, const int* tok_seq, const int* seq_slot,
                               const int* seq_len, void* pages, const int* page_table, int table_width, int page_size, int ring_rows, int n_pages,
                               int M, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(pages && page_table && seq_len && page_size > 0 && table_width > 0 && n_pages > 0 && ring_rows % page_size == 0,
               "latent_store: incomplete cache description");
    LatentPages kv{pages, page_table, table_width, page_size, ring_rows, n_pages, seq_len};
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        TI_CUDA(ti_launch_class<2>(latent_store_kernel<T>, dim3(M), dim3(128), 0, stream, (const T*)lat, W, tok_pos, tok_seq,
                                   seq_slot, kv));
        TI_CHECK_LAUNCH("latent_store");
        return 0;
    });
}

// A step of single tokens in two launches before and two after the projections... the latent's part of it: this one does
// latent_prep's and latent_absorb's work (q is left unrotated; qa gets the rotated part).
extern "C" int ti_latent_prep_absorb(const void* d, long long d_stride, const void* q, long long q_stride, int n_heads, int plain,
                                     int rank, int rot, const float* norm_w, float eps, const float* cos_t, const float* sin_t,
                                     int max_pos, const int* tok_pos, const int* tok_seq, const int* seq_slot, const int* seq_len,
                                     void* lat, void* pages, const int* page_table, int table_width, int page_size, int ring_rows,
                                     int n_pages, const void* uk, float* qa, int M, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && n_heads > 0 && n_heads < 65535 && rank > 0 && rot >= 0 && rot % 2 == 0 && plain >= 0 && q && uk && qa && lat,
               "latent_prep_absorb: bad arguments");
    TI_REQUIRE(rot == 0 || (cos_t && sin_t && max_pos > 0), "latent_prep_absorb: a rotated part needs cos and sin tables");
    TI_REQUIRE(!pages || (page_table && seq_len && page_size > 0 && table_width > 0 && n_pages > 0 && ring_rows % page_size == 0),
               "latent_prep_absorb: incomplete cache description");
    LatentPages kv{pages, page_table, table_width, page_size, ring_rows, n_pages, seq_len};
    const int W = rank + rot;
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        const size_t row = (size_t)(W + 33) * sizeof(float) + (size_t)W * sizeof(T);
        TI_REQUIRE(row <= 48 * 1024 && (size_t)plain * sizeof(float) <= 48 * 1024, "latent_prep_absorb: rows of %d elements are too long", W);
        if constexpr (sizeof(T) == 2)
            if (rank % 2 == 0 && ((uintptr_t)uk & 3) == 0 && plain <= 512 && (long long)n_heads * ((rank + AR_COLS - 1) / AR_COLS) < (1 << 24)) {
                auto go = M <= 4 ? launch_absorb_rows<4> : launch_absorb_rows<8>;
                return go(d, d_stride, q, q_stride, n_heads, plain, rank, rot, norm_w, eps, cos_t, sin_t, max_pos, tok_pos, tok_seq, seq_slot, lat, kv, uk,
                          qa, M, row, stream);
            }
        // (a head's query and its groups' sums: ABSORB_THREADS / (rank / 8) groups of `rank` sums, or a row's own)
        const size_t smem = std::max(row, (size_t)(plain + std::max(8 * ABSORB_THREADS, rank)) * sizeof(float));
        if (smem > 48 * 1024) TI_CUDA(cudaFuncSetAttribute(latent_prep_absorb_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        TI_CUDA(ti_launch_class<2>(latent_prep_absorb_kernel<T>, dim3(M, n_heads + 1), dim3(ABSORB_THREADS), smem, stream, (const T*)d, d_stride,
                                   (const T*)q, q_stride, n_heads, plain, rank, rot, norm_w, eps, cos_t, sin_t, max_pos, tok_pos, tok_seq,
                                   seq_slot, (T*)lat, kv, (const T*)uk, qa));
        TI_CHECK_LAUNCH("latent_prep_absorb");
        return 0;
    });
}

// Whether ti_latent_decode takes these sizes (bfloat16 only): rows in 16-element steps, a latent in 8-element tiles up to 512.
extern "C" int ti_latent_decode_takes(int rank, int rot) { return (rank + rot) % 16 == 0 && rank % 8 == 0 && rank <= 512; }

// One query per sequence, bfloat16, tensor cores; the key splits' merge and the way out through uv[heads * vdim, rank] in
// the second launch: o[n_seq, heads * vdim], head h times sigmoid(gate[., h]) where gate ([n_seq, heads], row stride
// gate_stride) is given.  part_o: float32 [n_seq, heads, n_splits, rank], part_ml: [n_seq, heads, n_splits, 2].
extern "C" int ti_latent_decode(const float* qa, const void* lat, const int* cu_new, const int* seq_start, const int* seq_slot,
                                int n_seq, int n_heads, int rank, int rot, float scale, int window, const float* sink,
                                const void* pages, const int* page_table, int table_width, int page_size, int ring_rows, int n_pages,
                                int n_splits, float* part_o, float* part_ml, const void* uv, void* o, long long o_stride, int vdim,
                                const void* gate, long long gate_stride, cudaStream_t stream) {
    if (n_seq == 0) return 0;
    TI_REQUIRE(n_seq > 0 && n_seq <= 65535 && n_heads > 0 && vdim > 0 && ti_latent_decode_takes(rank, rot), "latent_decode: sizes not taken");
    TI_REQUIRE(n_splits >= 1 && n_splits <= 64 && part_o && part_ml && uv && o, "latent_decode: bad arguments");
    TI_REQUIRE(pages && page_table && page_size > 0 && table_width > 0 && n_pages > 0 && ring_rows % page_size == 0,
               "latent_decode: incomplete cache description");
    TI_REQUIRE(ring_rows == 0 || (window > 0 && ring_rows >= window), "latent_decode: a ring of %d rows needs a window of at most as many", ring_rows);
    TI_REQUIRE((((uintptr_t)lat | (uintptr_t)pages | (uintptr_t)qa) & 15) == 0, "latent_decode: rows are not 16-byte aligned");
    LatentPages kv{const_cast<void*>(pages), page_table, table_width, page_size, ring_rows, n_pages, nullptr};
    const bool two = n_heads > 16;
#define TI_LATENT_DECODE(MT, NTW) launch_decode_mma<MT, NTW>(qa, lat, nullptr, cu_new, seq_start, seq_slot, n_seq, n_heads, rank, rot, scale, \
                                                            window, sink, kv, n_splits, part_o, part_ml, n_seq, stream, uv, o, o_stride, vdim, gate, gate_stride)
    if (rank <= 128) return two ? TI_LATENT_DECODE(2, 4) : TI_LATENT_DECODE(1, 4);
    if (rank <= 256) return two ? TI_LATENT_DECODE(2, 8) : TI_LATENT_DECODE(1, 8);
    return two ? TI_LATENT_DECODE(2, 16) : TI_LATENT_DECODE(1, 16);
#undef TI_LATENT_DECODE
}

extern "C" int ti_latent_pack(const void* q, long long q_stride, const void* ku, const void* lat, void* Qp, void* Kp, void* Vp,
                              int M, int n_heads, int plain, int rot, int vdim, int rank, int D, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && n_heads > 0 && plain >= 0 && rot >= 0 && vdim > 0 && rank > 0 && D >= plain + rot && D >= vdim,
               "latent_pack: heads of %d + %d and %d elements do not fit %d", plain, rot, vdim, D);
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        TI_CUDA(ti_launch_class<2>(latent_pack_kernel<T>, dim3(M), dim3(256), 0, stream, (const T*)q, q_stride, (const T*)ku,
                                   (const T*)lat, (T*)Qp, (T*)Kp, (T*)Vp, n_heads, plain, rot, vdim, rank, D));
        TI_CHECK_LAUNCH("latent_pack");
        return 0;
    });
}

extern "C" int ti_latent_absorb(const void* q, long long q_stride, const void* uk, float* qa, int M, int n_heads, int plain,
                                int rank, int rot, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && n_heads > 0 && n_heads <= 65535 && plain >= 0 && rank > 0 && rot >= 0, "latent_absorb: bad sizes");
    const size_t smem = (size_t)ABS_TM * (plain > 0 ? plain : 1) * sizeof(float);
    TI_REQUIRE(smem <= 48 * 1024, "latent_absorb: heads of %d unrotated elements are too long", plain);
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        const int zs = (rank + ABS_THREADS * ABS_RPT - 1) / (ABS_THREADS * ABS_RPT);
        TI_CUDA(ti_launch(latent_absorb_kernel<T>, dim3((M + ABS_TM - 1) / ABS_TM, n_heads, zs), dim3(ABS_THREADS), smem, stream,
                          (const T*)q, q_stride, (const T*)uk, qa, M, n_heads, plain, rank, rot));
        TI_CHECK_LAUNCH("latent_absorb");
        return 0;
    });
}

extern "C" int ti_latent_expand(const float* ol, const void* uv, void* o, long long o_stride, int M, int n_heads, int vdim,
                                int rank, const void* gate, long long gate_stride, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && n_heads > 0 && n_heads <= 65535 && vdim > 0 && rank > 0, "latent_expand: bad sizes");
    const size_t smem = (size_t)EXP_TM * rank * sizeof(float);
    TI_REQUIRE(smem <= 48 * 1024, "latent_expand: a latent of %d elements is too long", rank);
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        TI_CUDA(ti_launch(latent_expand_kernel<T>, dim3((M + EXP_TM - 1) / EXP_TM, n_heads, (vdim + EXP_VB - 1) / EXP_VB), dim3(EXP_THREADS), smem, stream, ol,
                          (const T*)uv, (T*)o, o_stride, M, n_heads, vdim, rank, (const T*)gate, gate_stride));
        TI_CHECK_LAUNCH("latent_expand");
        return 0;
    });
}

// qa: float32 [M, heads, rank + rot]; lat: the step's rows [M, rank + rot]; ol: float32 [M, heads, rank].
// hb: heads per block, a power of two up to 32.  sink: float32 [heads] or null.
extern "C" int ti_latent_attn(const float* qa, const void* lat, float* ol, const int* cu_new, const int* seq_start,
                              const int* seq_slot, int n_seq, int max_new, int n_heads, int hb, int rank, int rot, float scale,
                              int window, const float* sink, const void* pages, const int* page_table, int table_width,
                              int page_size, int ring_rows, int n_pages, int n_splits, float* part_o, float* part_ml, int n_tok,
                              int dtype, cudaStream_t stream) {
    if (n_seq == 0 || max_new == 0) return 0;
    TI_REQUIRE(n_seq > 0 && max_new > 0 && n_heads > 0 && rank > 0 && rot >= 0, "latent_attention: bad sizes");
    TI_REQUIRE(hb >= 1 && hb <= LQ && (hb & (hb - 1)) == 0, "latent_attention: %d heads per block (a power of two up to %d)", hb, LQ);
    TI_REQUIRE(n_seq <= 65535, "latent_attention: too many sequences for one launch");
    TI_REQUIRE(pages && page_table && page_size > 0 && table_width > 0 && n_pages > 0 && ring_rows % page_size == 0,
               "latent_attention: incomplete cache description");
    TI_REQUIRE(ring_rows == 0 || (window > 0 && ring_rows >= window),
               "latent_attention: a ring of %d rows needs a window of at most as many positions (got %d)", ring_rows, window);
    TI_REQUIRE(rank <= 1024, "latent_attention: a latent of %d elements is not supported (up to 1,024)", rank);
    TI_REQUIRE(n_splits >= 1 && (n_splits == 1 || (part_o && part_ml && n_tok > 0 && n_tok <= 65535 * 32768)),
               "latent_attention: %d splits need room for their partial results", n_splits);
    LatentPages kv{const_cast<void*>(pages), page_table, table_width, page_size, ring_rows, n_pages, nullptr};
    // every sequence brings one token, bfloat16, rows in 16-byte pieces: the tensor-core kernel
    if (dtype == TI_BF16 && max_new == 1 && n_tok == n_seq && (rank + rot) % 16 == 0 && rank % 8 == 0 && rank <= 512 &&
        ((uintptr_t)lat & 15) == 0 && ((uintptr_t)pages & 15) == 0) {
        const bool two = n_heads > 16;
#define TI_LATENT_DECODE(MT, NTW) launch_decode_mma<MT, NTW>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, n_heads, rank, rot, scale, \
                                                            window, sink, kv, n_splits, part_o, part_ml, n_tok, stream)
        if (rank <= 128) return two ? TI_LATENT_DECODE(2, 4) : TI_LATENT_DECODE(1, 4);
        if (rank <= 256) return two ? TI_LATENT_DECODE(2, 8) : TI_LATENT_DECODE(1, 8);
        return two ? TI_LATENT_DECODE(2, 16) : TI_LATENT_DECODE(1, 16);
#undef TI_LATENT_DECODE
    }
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        if (rank <= 64)
            return launch_attn<T, 16>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, max_new, n_heads, hb, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, n_tok, stream);
        if (rank <= 128)
            return launch_attn<T, 32>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, max_new, n_heads, hb, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, n_tok, stream);
        if (rank <= 256)
            return launch_attn<T, 64>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, max_new, n_heads, hb, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, n_tok, stream);
        if (rank <= 512)
            return launch_attn<T, 128>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, max_new, n_heads, hb, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, n_tok, stream);
        return launch_attn<T, 256>(qa, lat, ol, cu_new, seq_start, seq_slot, n_seq, max_new, n_heads, hb, rank, rot, scale, window, sink, kv, n_splits, part_o, part_ml, n_tok, stream);
    });
}
