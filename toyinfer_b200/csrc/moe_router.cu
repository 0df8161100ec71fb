// A mixture-of-experts router with independent (sigmoid) scores, and the sum that ends such a layer.
//
// moe_route_topk: from every token's router logits z [experts] (float32), the `top` experts with
// the largest logits (the sigmoid keeps the order; of equal logits the lower index wins) and for
// each pair p = m * top + j its score s = sigmoid(z) and s^2.  It counts the pairs of every expert
// and writes them out grouped by expert, as the grouped products read them: perm[i] is the pair at
// place i, off[e] .. off[e + 1] the places of expert e.  One block.
//
// moe_route_softmax: the same output for a router with softmax scores s = softmax(z) over all experts.  Experts are
// CHOSEN by s + correction (a float32 value per expert; without one by the logits themselves, which keep the order also
// where scores underflow; a bias per expert may be added to the logits first), only among the experts of the `keep` best of
// `n_groups` equal runs of neighbouring experts (a run's score is its largest choice score; n_groups <= 1: all
// experts), ties to the lower index; a pair's WEIGHT is its s divided by the sum of the token's chosen s (+ 1e-20),
// times `scale`.  Scores that are not allowed do not count as 0: choice scores may be negative.
//
// The experts of moe_route_topk act on the scaled input, expert(s x) = Wdown relu(Wup (s x))^2, which for s > 0
// is s^2 Wdown relu(Wup x)^2: the products run on x itself and
// moe_combine_gated: out[m] = sum_j s_p^2 z[place of pair p] + sigmoid(g_m) * shared[m]
// applies the squares at the end, with a shared expert's output behind a gate of its own logit
// (both optional).
#include "common.cuh"

#include <type_traits>

namespace {

constexpr int RT_THREADS = 1024, MAX_TOP = 16;

__global__ void moe_route_topk_kernel(const float* __restrict__ z, long long ldz, int n_experts, int top, int M,
                                      int* __restrict__ perm, int* __restrict__ off, int* __restrict__ pair_expert,
                                      float* __restrict__ pair_score, float* __restrict__ pair_score2) {
    ti_pdl_trigger();
    extern __shared__ int cnt[];         // [n_experts] counts, then [n_experts + 1] offsets, then [n_experts] cursors
    int* offs = cnt + n_experts;
    int* cur = offs + n_experts + 1;
    ti_pdl_sync();
    z = ti_dependent(z);
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) { cnt[e] = 0; cur[e] = 0; }
    __syncthreads();
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        const float* zr = z + (size_t)m * ldz;
        int chosen[MAX_TOP];
        for (int j = 0; j < top; j++) {
            int best = -1;
            float bz = 0.f;
            for (int e = 0; e < n_experts; e++) {
                bool taken = false;
                for (int i = 0; i < j; i++) taken |= chosen[i] == e;
                if (taken) continue;
                const float x = zr[e];
                if (best < 0 || x > bz) { best = e; bz = x; }      // a row of NaN keeps the lowest free index
            }
            chosen[j] = best;
            const int p = m * top + j;
            const float s = ti_over(1.0f, 1.0f + expf(-bz));
            pair_expert[p] = best;
            pair_score[p] = s;
            pair_score2[p] = s * s;
            atomicAdd(&cnt[best], 1);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0;
        for (int e = 0; e < n_experts; e++) { offs[e] = a; a += cnt[e]; }
        offs[n_experts] = a;
    }
    __syncthreads();
    for (int e = threadIdx.x; e <= n_experts; e += blockDim.x) off[e] = offs[e];
    const int P = M * top;
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        const int e = pair_expert[p];
        perm[offs[e] + atomicAdd(&cur[e], 1)] = p;
    }
}

// what both routers end with: the pairs of every expert counted in cnt[], written out grouped by expert
__device__ __forceinline__ void group_pairs(int* cnt, int* offs, int* cur, int n_experts, int P, const int* pair_expert,
                                            int* __restrict__ perm, int* __restrict__ off) {
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0;
        for (int e = 0; e < n_experts; e++) { offs[e] = a; a += cnt[e]; }
        offs[n_experts] = a;
    }
    __syncthreads();
    for (int e = threadIdx.x; e <= n_experts; e += blockDim.x) off[e] = offs[e];
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        const int e = pair_expert[p];
        perm[offs[e] + atomicAdd(&cur[e], 1)] = p;
    }
}

// The place of a pair among its expert's pairs: one atomic a warp and expert.  All lanes of the warp call it; those with e < 0
// have no pair.
__device__ __forceinline__ int place_among(int* cnt, int e) {
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    int first = 0;
    if (lane == leader && e >= 0) first = atomicAdd(&cnt[e], __popc(same));
    return __shfl_sync(0xffffffffu, first, leader) + __popc(same & ((1u << lane) - 1));
}

// Routers of up to E experts without runs of experts, E a compile-time bound: a token's logits are read once, into registers,
// and a pair's place among its expert's is known when it is counted, so that the pairs need no second count.  (One block, as
// above: 777 tokens, 16 experts, two per token
// 19 us with the logits read again for every choice, 11 so.)  32 is where a thread's 64 registers end: with 64 a token's logits and
// choices lie in local memory, and 777 tokens of 40 experts, two each, take 54 us where the kernel below takes 30 (64 experts, four
// each, 93 and 173).
// SOFT: weights by softmax (moe_route_softmax), else by sigmoid (moe_route_topk: pair_w the score, pair_w2 its square).
template <int E, bool SOFT>
__global__ void __launch_bounds__(RT_THREADS)
moe_route_few_kernel(const float* __restrict__ z, long long ldz, const float* __restrict__ logit_bias, const float* __restrict__ correction,
                     int n_experts, int top, float scale, int M, int* __restrict__ perm, int* __restrict__ off, int* __restrict__ pair_expert,
                     float* __restrict__ pair_w, float* __restrict__ pair_w2) {
    ti_pdl_trigger();
    __shared__ int cnt[E], offs[E + 1];
    ti_pdl_sync();
    z = ti_dependent(z);
    if (threadIdx.x < E) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int m0 = 0; m0 < M; m0 += RT_THREADS) {
        const int m = m0 + threadIdx.x;
        const bool live = m < M;
        const float* zr = z + (size_t)(live ? m : 0) * ldz;
        float l[E], c[E];
#pragma unroll
        for (int e = 0; e < E; e++) l[e] = e < n_experts ? zr[e] + (logit_bias ? logit_bias[e] : 0.f) : 0.f;
        float zmax = -INFINITY, sum = 0.f, inv = 1.f;
        if constexpr (SOFT) {
#pragma unroll
            for (int e = 0; e < E; e++) if (e < n_experts) zmax = fmaxf(zmax, l[e]);
#pragma unroll
            for (int e = 0; e < E; e++) if (e < n_experts) sum += expf(l[e] - zmax);
            inv = 1.0f / sum;
        }
#pragma unroll
        for (int e = 0; e < E; e++) c[e] = SOFT && correction && e < n_experts ? expf(l[e] - zmax) * inv + correction[e] : l[e];
        unsigned taken = 0;
        int chosen[MAX_TOP];
        float s_of[MAX_TOP], total = 0.f;
        for (int j = 0; j < top; j++) {
            int best = -1;
            float bc = 0.f, bl = 0.f;
#pragma unroll
            for (int e = 0; e < E; e++)
                if (e < n_experts && !(taken >> e & 1u) && (best < 0 || c[e] > bc)) { best = e; bc = c[e]; bl = l[e]; }     // a row of NaN keeps the lowest free index
            taken |= 1u << best;
            chosen[j] = best;
            s_of[j] = SOFT ? expf(bl - zmax) * inv : ti_over(1.0f, 1.0f + expf(-bl));
            total += s_of[j];
        }
        const float norm = SOFT ? scale / (total + 1e-20f) : 1.f;
        for (int j = 0; j < top; j++) {
            const int e = live ? chosen[j] : -1, at = place_among(cnt, e);
            if (live) {
                const int p = m * top + j;
                pair_expert[p] = e + at * E;                 // (E pairs' places per expert: P * E is below 2^31, see the entry)
                pair_w[p] = SOFT ? s_of[j] * norm : s_of[j];
                if (!SOFT) pair_w2[p] = s_of[j] * s_of[j];
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0;
        for (int e = 0; e < n_experts; e++) { offs[e] = a; a += cnt[e]; }
        offs[n_experts] = a;
    }
    __syncthreads();
    for (int e = threadIdx.x; e <= n_experts; e += blockDim.x) off[e] = offs[e];
    for (int p = threadIdx.x; p < M * top; p += blockDim.x) {
        const int x = pair_expert[p], e = x % E;
        perm[offs[e] + x / E] = p;
    }
}

template <bool SOFT>
int route_few(const float* z, long long ldz, const float* logit_bias, const float* correction, int n_experts, int top, float scale, int M,
              int* perm, int* off, int* pair_expert, float* pair_w, float* pair_w2, cudaStream_t stream) {
    auto go = [&](auto ec) -> int {
        TI_CUDA(ti_launch_class<1>(moe_route_few_kernel<decltype(ec)::value, SOFT>, dim3(1), dim3(RT_THREADS), 0, stream, z, ldz, logit_bias, correction,
                                   n_experts, top, scale, M, perm, off, pair_expert, pair_w, pair_w2));
        TI_CHECK_LAUNCH("moe_route (few experts)");
        return 0;
    };
    if (n_experts <= 8) return go(std::integral_constant<int, 8>());
    if (n_experts <= 16) return go(std::integral_constant<int, 16>());
    return go(std::integral_constant<int, 32>());
}

// A softmax router of up to 32 experts with its product: a block takes TOK tokens.  Its eight warps take every eighth expert's row
// each, lanes along the row (16 bytes, AHEAD pieces of every row on their way together), and then, a warp a token and a lane an
// expert, choose as moe_route_few_kernel does.  The choices go to moe_place_kernel, which counts and places the pairs.
// (The product alone, a tcgen05 tile of which 16 of 128 rows were used, took 12 us at 40 to 777 tokens, and the one-block router after
// it 7 us at one token and 9 at 777: what bounds both is a chain of dependent steps, not work.)
// Pieces on their way and blocks an SM so that nothing spills: 32 experts in bfloat16 with four pieces and three blocks took, rows of
// 2,048, 10.3, 19.4 and 22.9 us at 1, 296 and 777 tokens; with two and two 6.9, 8.6 and 13.4.
constexpr int RK_THREADS = 256;

// Smaller than every number's key: not a number.  Equal numbers (zeros of both signs too) have equal keys.
__device__ __forceinline__ unsigned order_key(float c) {
    if (c != c) return 0u;
    const unsigned b = __float_as_uint(c + 0.0f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}

template <typename T, int EPW, int TOK>
__global__ void __launch_bounds__(RK_THREADS, TOK == 1 || EPW * 16 / sizeof(T) > 16 ? 2 : 3)
moe_router_kernel(const T* __restrict__ x, long long ldx, const T* __restrict__ w, int K, const float* __restrict__ logit_bias,
                  const float* __restrict__ correction, int n_experts, int top, float scale, int M, int* __restrict__ pair_expert,
                  float* __restrict__ pair_w) {
    ti_pdl_trigger();
    constexpr int V = 16 / sizeof(T), AHEAD = TOK > 1 ? 1 : EPW * V > 16 ? 2 : 4;
    struct alignas(16) Pack { T v[V]; };
    __shared__ float logits[TOK][32];
    ti_pdl_sync();
    x = ti_dependent(x); w = ti_dependent(w);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, m0 = blockIdx.x * TOK;
    float acc[EPW][TOK];
#pragma unroll
    for (int i = 0; i < EPW; i++)
#pragma unroll
        for (int t = 0; t < TOK; t++) acc[i][t] = 0.f;
    for (int k0 = lane * V; k0 < K; k0 += 32 * V * AHEAD) {
        Pack px[AHEAD][TOK], pw[AHEAD][EPW];
#pragma unroll
        for (int u = 0; u < AHEAD; u++) {
            const int k = k0 + u * 32 * V;
            if (k >= K) break;
#pragma unroll
            for (int t = 0; t < TOK; t++) px[u][t] = *reinterpret_cast<const Pack*>(x + (size_t)min(m0 + t, M - 1) * ldx + k);
#pragma unroll
            for (int i = 0; i < EPW; i++)
                if (warp + 8 * i < n_experts) pw[u][i] = *reinterpret_cast<const Pack*>(w + (size_t)(warp + 8 * i) * K + k);
        }
#pragma unroll
        for (int u = 0; u < AHEAD; u++) {
            if (k0 + u * 32 * V >= K) break;
#pragma unroll
            for (int i = 0; i < EPW; i++)
                if (warp + 8 * i < n_experts) {
#pragma unroll
                    for (int t = 0; t < TOK; t++)
#pragma unroll
                        for (int j = 0; j < V; j++) acc[i][t] = fmaf(to_f32(px[u][t].v[j]), to_f32(pw[u][i].v[j]), acc[i][t]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < EPW; i++)
#pragma unroll
        for (int t = 0; t < TOK; t++) {
            const float s = warp_sum(acc[i][t]);
            if (lane == 0 && warp + 8 * i < n_experts) logits[t][warp + 8 * i] = s;
        }
    __syncthreads();
    const int m = m0 + warp;
    if (warp >= TOK || m >= M) return;
    const bool has = lane < n_experts;
    const float l = has ? logits[warp][lane] + (logit_bias ? logit_bias[lane] : 0.f) : -INFINITY;
    const float zmax = warp_max(l);
    const float ex = has ? expf(l - zmax) : 0.f;
    const float inv = 1.0f / warp_sum(ex);
    const float s = ex * inv, c = correction ? (has ? s + correction[lane] : 0.f) : l;
    const unsigned key = order_key(c);
    bool open = has;
    float mine = 0.f, total = 0.f;
    int rank = -1;
    for (int j = 0; j < top; j++) {
        // the lowest open index where that one is not a number (it is kept against every other), else the largest, lowest index first
        const int lowest = __ffs(__ballot_sync(0xffffffffu, open)) - 1;
        const unsigned most = __reduce_max_sync(0xffffffffu, open ? key : 0u);
        const int largest = __ffs(__ballot_sync(0xffffffffu, open && key == most)) - 1;
        const int best = __shfl_sync(0xffffffffu, key, lowest) == 0u ? lowest : largest;
        total += __shfl_sync(0xffffffffu, s, best);
        if (lane == best) { open = false; rank = j; mine = s; }
    }
    if (rank >= 0) {
        pair_expert[(size_t)m * top + rank] = lane;
        pair_w[(size_t)m * top + rank] = mine * (scale / (total + 1e-20f));
    }
}

// Counts the pairs of every expert (up to 32) and writes them out grouped by expert.  One block.  Without pad_src: perm and off.
// With it: the plan of moe_pad_plan (moe_grouped.cu) instead, every expert's places padded to whole tiles of 128.
__global__ void __launch_bounds__(RT_THREADS)
moe_place_kernel(int* __restrict__ pair_expert, int n_experts, int top, int P, int* __restrict__ perm, int* __restrict__ off,
                 int rows, int* __restrict__ pad_src, int* __restrict__ pad_of_pair, int* __restrict__ tile_group) {
    ti_pdl_trigger();
    __shared__ int cnt[32], offs[33];
    if (threadIdx.x < 32) cnt[threadIdx.x] = 0;
    ti_pdl_sync();
    pair_expert = ti_dependent(pair_expert);
    __syncthreads();
    if (pad_src) for (int i = threadIdx.x; i < rows; i += RT_THREADS) pad_src[i] = -1;
    constexpr int KEEP = 4;                    // pairs whose place a thread keeps in registers; further ones go back to pair_expert
    int e_of[KEEP], at_of[KEEP];
#pragma unroll
    for (int i = 0; i < KEEP; i++) {
        const int p = i * RT_THREADS + threadIdx.x;
        e_of[i] = p < P ? pair_expert[p] : -1;
    }
#pragma unroll
    for (int i = 0; i < KEEP; i++)
        if (i * RT_THREADS < P) at_of[i] = place_among(cnt, e_of[i]);
    for (int p0 = KEEP * RT_THREADS; p0 < P; p0 += RT_THREADS) {
        const int p = p0 + threadIdx.x, e = p < P ? pair_expert[p] : -1, at = place_among(cnt, e);
        if (p < P) pair_expert[p] = e + at * 32;                 // (P * 32 is below 2^31, see the entry)
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int n = (int)threadIdx.x < n_experts ? cnt[threadIdx.x] : 0;
        int upto = pad_src ? (n + 127) / 128 * 128 : n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, upto, o);
            if ((int)threadIdx.x >= o) upto += below;
        }
        offs[threadIdx.x + 1] = upto;
        if (threadIdx.x == 0) offs[0] = 0;
    }
    __syncthreads();
    auto put = [&](int p, int e, int at) {
        const int i = offs[e] + at;
        if (pad_src) { pad_src[i] = p / top; pad_of_pair[p] = i; }
        else perm[i] = p;
    };
#pragma unroll
    for (int i = 0; i < KEEP; i++)
        if (e_of[i] >= 0) put(i * RT_THREADS + threadIdx.x, e_of[i], at_of[i]);
    for (int p = KEEP * RT_THREADS + threadIdx.x; p < P; p += RT_THREADS) put(p, pair_expert[p] & 31, pair_expert[p] >> 5);
    if (!pad_src) {
        if ((int)threadIdx.x <= n_experts) off[threadIdx.x] = offs[threadIdx.x];
        return;
    }
    for (int t = threadIdx.x; t < rows / 128; t += RT_THREADS) {
        int g = -1;
        for (int e = 0; e < n_experts; e++)
            if (t * 128 >= offs[e] && t * 128 < offs[e + 1]) g = e;
        tile_group[t] = g;
    }
}

constexpr int MAX_GROUPS = 64;

__global__ void moe_route_softmax_kernel(const float* __restrict__ z, long long ldz, const float* __restrict__ logit_bias,
                                         const float* __restrict__ correction,
                                         int n_experts, int top, int n_groups, int keep, float scale, int M,
                                         int* __restrict__ perm, int* __restrict__ off, int* __restrict__ pair_expert,
                                         float* __restrict__ pair_w) {
    ti_pdl_trigger();
    extern __shared__ int cnt[];         // [n_experts] counts, then [n_experts + 1] offsets, then [n_experts] cursors
    int* offs = cnt + n_experts;
    int* cur = offs + n_experts + 1;
    ti_pdl_sync();
    z = ti_dependent(z);
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) { cnt[e] = 0; cur[e] = 0; }
    __syncthreads();
    const int per = n_groups > 1 ? n_experts / n_groups : n_experts;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        const float* zr = z + (size_t)m * ldz;
        auto logit = [&](int e) { return zr[e] + (logit_bias ? logit_bias[e] : 0.f); };
        float zmax = -INFINITY;
        for (int e = 0; e < n_experts; e++) zmax = fmaxf(zmax, logit(e));
        float sum = 0.f;
        for (int e = 0; e < n_experts; e++) sum += expf(logit(e) - zmax);
        const float inv = 1.0f / sum;
        auto score = [&](int e) { return expf(logit(e) - zmax) * inv; };
        auto choice = [&](int e) { return correction ? score(e) + correction[e] : logit(e); };
        unsigned long long open = ~0ull;                 // bit g: experts of run g may be chosen
        if (n_groups > 1 && keep < n_groups) {
            open = 0ull;
            for (int j = 0; j < keep; j++) {
                int best = -1;
                float bs = 0.f;
                for (int g = 0; g < n_groups; g++) {
                    if (open >> g & 1ull) continue;
                    float gs = -INFINITY;
                    for (int e = g * per; e < (g + 1) * per; e++) gs = fmaxf(gs, choice(e));
                    if (best < 0 || gs > bs) { best = g; bs = gs; }
                }
                open |= 1ull << best;
            }
        }
        int chosen[MAX_TOP];
        float s_of[MAX_TOP];
        float total = 0.f;
        for (int j = 0; j < top; j++) {
            int best = -1;
            float bc = 0.f;
            for (int e = 0; e < n_experts; e++) {
                if (n_groups > 1 && !(open >> (e / per) & 1ull)) continue;
                bool taken = false;
                for (int i = 0; i < j; i++) taken |= chosen[i] == e;
                if (taken) continue;
                const float c = choice(e);
                if (best < 0 || c > bc) { best = e; bc = c; }      // a row of NaN keeps the lowest free index
            }
            chosen[j] = best;
            s_of[j] = score(best);
            total += s_of[j];
        }
        const float norm = scale / (total + 1e-20f);
        for (int j = 0; j < top; j++) {
            const int p = m * top + j;
            pair_expert[p] = chosen[j];
            pair_w[p] = s_of[j] * norm;
            atomicAdd(&cnt[chosen[j]], 1);
        }
    }
    group_pairs(cnt, offs, cur, n_experts, M * top, pair_expert, perm, off);
}

template <typename T>
__global__ void moe_combine_gated_kernel(const T* __restrict__ z, const int* __restrict__ place_of_pair,
                                         const float* __restrict__ pair_w, const T* __restrict__ shared_out,
                                         const float* __restrict__ gate_logit, long long gate_stride, T* __restrict__ out, int H,
                                         int top) {
    ti_pdl_trigger();
    ti_pdl_sync();
    z = ti_dependent(z); place_of_pair = ti_dependent(place_of_pair); pair_w = ti_dependent(pair_w);
    shared_out = ti_dependent(shared_out); gate_logit = ti_dependent(gate_logit);
    const size_t m = blockIdx.x;
    const float g = (shared_out && gate_logit) ? ti_over(1.0f, 1.0f + expf(-gate_logit[m * gate_stride])) : 1.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float s = 0.f;
        for (int j = 0; j < top; j++) {
            const size_t p = m * top + j;
            const size_t at = place_of_pair ? (size_t)place_of_pair[p] : p;
            s = fmaf(pair_w ? pair_w[p] : 1.f, to_f32(z[at * H + i]), s);
        }
        if (shared_out) s = fmaf(g, to_f32(shared_out[m * H + i]), s);
        out[m * H + i] = from_f32<T>(s);
    }
}

// The same eight elements a thread, every source's in one read (bfloat16: one, float32: two).
template <typename T>
__global__ void moe_combine_gated_vec_kernel(const T* __restrict__ z, const int* __restrict__ place_of_pair,
                                             const float* __restrict__ pair_w, const T* __restrict__ shared_out,
                                             const float* __restrict__ gate_logit, long long gate_stride, T* __restrict__ out, int H, int top) {
    ti_pdl_trigger();
    ti_pdl_sync();
    z = ti_dependent(z); place_of_pair = ti_dependent(place_of_pair); pair_w = ti_dependent(pair_w);
    shared_out = ti_dependent(shared_out); gate_logit = ti_dependent(gate_logit);
    const size_t m = blockIdx.x;
    const float g = (shared_out && gate_logit) ? ti_over(1.0f, 1.0f + expf(-gate_logit[m * gate_stride])) : 1.f;
    struct alignas(16) Run { T v[8]; };
    for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
        float s[8] = {};
        for (int j0 = 0; j0 < top; j0 += 4) {        // four choices' rows on their way together
            Run x[4];
            float w[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j0 + j < top) {
                    const size_t p = m * top + j0 + j, at = place_of_pair ? (size_t)place_of_pair[p] : p;
                    w[j] = pair_w ? pair_w[p] : 1.f;
                    x[j] = *reinterpret_cast<const Run*>(z + at * H + i);
                }
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j0 + j < top) {
#pragma unroll
                    for (int e = 0; e < 8; e++) s[e] = fmaf(w[j], to_f32(x[j].v[e]), s[e]);
                }
        }
        if (shared_out) {
            const Run x = *reinterpret_cast<const Run*>(shared_out + m * H + i);
#pragma unroll
            for (int e = 0; e < 8; e++) s[e] = fmaf(g, to_f32(x.v[e]), s[e]);
        }
        Run y;
#pragma unroll
        for (int e = 0; e < 8; e++) y.v[e] = from_f32<T>(s[e]);
        *reinterpret_cast<Run*>(out + m * H + i) = y;
    }
}

}  // namespace

// z: float32 [M, >= n_experts] with row stride ldz; perm: int32 [M * top]; off: int32 [n_experts + 1]; pair_expert: int32
// scratch [M * top]; pair_score, pair_score2: float32 [M * top].
extern "C" int ti_moe_route_topk(const float* z, long long ldz, int n_experts, int top, int M, int* perm, int* off,
                                 int* pair_expert, float* pair_score, float* pair_score2, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && n_experts > 0 && top >= 1 && top <= n_experts && top <= MAX_TOP && ldz >= n_experts,
               "moe_route_topk: bad sizes (%d experts, %d per token; at most %d per token)", n_experts, top, MAX_TOP);
    if (n_experts <= 32 && (long long)M * top * 32 < (1LL << 31))
        return route_few<false>(z, ldz, nullptr, nullptr, n_experts, top, 1.f, M, perm, off, pair_expert, pair_score, pair_score2, stream);
    const size_t smem = (size_t)(3 * n_experts + 1) * sizeof(int);
    TI_REQUIRE(smem <= 48 * 1024, "moe_route_topk: %d experts are too many", n_experts);
    TI_CUDA(ti_launch_class<1>(moe_route_topk_kernel, dim3(1), dim3(RT_THREADS), smem, stream, z, ldz, n_experts, top, M, perm, off,
                               pair_expert, pair_score, pair_score2));
    TI_CHECK_LAUNCH("moe_route_topk");
    return 0;
}

// z: float32 [M, >= n_experts] with row stride ldz; logit_bias, correction: float32 [n_experts] or null; n_groups <= 1: no runs; perm: int32
// [M * top]; off: int32 [n_experts + 1]; pair_expert: int32 scratch [M * top]; pair_w: float32 [M * top].
extern "C" int ti_moe_route_softmax(const float* z, long long ldz, const float* logit_bias, const float* correction, int n_experts, int top, int n_groups,
                                    int keep, float scale, int M, int* perm, int* off, int* pair_expert, float* pair_w,
                                    cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && n_experts > 0 && top >= 1 && top <= n_experts && top <= MAX_TOP && ldz >= n_experts,
               "moe_route_softmax: bad sizes (%d experts, %d per token; at most %d per token)", n_experts, top, MAX_TOP);
    if (n_groups > 1)
        TI_REQUIRE(n_groups <= MAX_GROUPS && n_experts % n_groups == 0 && keep >= 1 && keep <= n_groups &&
                   (long long)keep * (n_experts / n_groups) >= top,
                   "moe_route_softmax: %d experts in %d runs of which %d stay, %d per token (at most %d runs)", n_experts, n_groups, keep,
                   top, MAX_GROUPS);
    if (n_groups <= 1 && n_experts <= 32 && (long long)M * top * 32 < (1LL << 31))
        return route_few<true>(z, ldz, logit_bias, correction, n_experts, top, scale, M, perm, off, pair_expert, pair_w, nullptr, stream);
    const size_t smem = (size_t)(3 * n_experts + 1) * sizeof(int);
    TI_REQUIRE(smem <= 48 * 1024, "moe_route_softmax: %d experts are too many", n_experts);
    TI_CUDA(ti_launch_class<1>(moe_route_softmax_kernel, dim3(1), dim3(RT_THREADS), smem, stream, z, ldz, logit_bias, correction, n_experts,
                               top, n_groups, keep, scale, M, perm, off, pair_expert, pair_w));
    TI_CHECK_LAUNCH("moe_route_softmax");
    return 0;
}

// The softmax router with its product, for up to 32 experts without runs: x [M, K] (row stride ldx), w [n_experts, K] dense, both of
// one type, rows on 16-byte boundaries.  pair_expert: int32 scratch [M * top]; pair_w: float32 [M * top].  With pad_src null: perm
// and off as ti_moe_route_softmax gives them; else pad_src [rows], pad_of_pair and tile_group as ti_moe_pad_plan does.
extern "C" int ti_moe_route_rows(const void* x, long long ldx, const void* w, int K, const float* logit_bias, const float* correction,
                                 int n_experts, int top, float scale, int M, int* pair_expert, float* pair_w, int* perm, int* off,
                                 int rows, int* pad_src, int* pad_of_pair, int* tile_group, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && K > 0 && n_experts > 0 && n_experts <= 32 && top >= 1 && top <= n_experts && top <= MAX_TOP && (long long)M * top * 32 < (1LL << 31),
               "moe_route_rows: bad sizes (%d experts, %d per token; at most 32 and %d)", n_experts, top, MAX_TOP);
    TI_REQUIRE(pad_src ? rows % 128 == 0 && rows >= M * top && pad_of_pair && tile_group : perm && off, "moe_route_rows: incomplete plan");
    const int code = ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        constexpr int V = 16 / sizeof(T);
        TI_REQUIRE(K % V == 0 && ldx % V == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0, "moe_route_rows: rows are not 16-byte aligned");
        auto go = [&](auto tok) -> int {
            constexpr int TOK = decltype(tok)::value;
            auto kernel = n_experts <= 8 ? moe_router_kernel<T, 1, TOK> : n_experts <= 16 ? moe_router_kernel<T, 2, TOK> : moe_router_kernel<T, 4, TOK>;
            TI_CUDA(ti_launch_class<1>(kernel, dim3((M + TOK - 1) / TOK), dim3(RK_THREADS), 0, stream, (const T*)x, ldx, (const T*)w, K, logit_bias,
                                       correction, n_experts, top, scale, M, pair_expert, pair_w));
            return 0;
        };
        // a token a block while all blocks fit the device at once
        const int rc = M <= 2 * ti_sm_count() ? go(std::integral_constant<int, 1>()) : go(std::integral_constant<int, 4>());
        if (rc) return rc;
        TI_CHECK_LAUNCH("moe_route_rows");
        return 0;
    });
    if (code) return code;
    // The tiles of some tens of bfloat16 places (moe_grouped.cu) read their operands through L1, of which the SMs have next to none as long
    // as kernels keep overlapping with one of large shared memory, the layer's own last product before this router among them.  There the
    // one block that places the pairs starts when the kernels before it have ended, so that the SMs come free: layers of 8 experts of 2,048 x 600
    // beside a shared one, 200 tokens, 122.9 us without, 98.5 so; 16 of 544, 98 tokens with four choices 123.0, 105.7.  Products from
    // registers and on tcgen05 gain nothing and would wait: one token of 16 experts 20.2, 21.0.
    const bool drained = !pad_src && dtype == TI_BF16 && M * top > 12 * n_experts;
    if (!drained)
        TI_CUDA(ti_launch_class<1>(moe_place_kernel, dim3(1), dim3(RT_THREADS), 0, stream, pair_expert, n_experts, top, M * top, perm, off, rows, pad_src,
                                   pad_of_pair, tile_group));
    else
        TI_CUDA(ti_launch_after(moe_place_kernel, dim3(1), dim3(RT_THREADS), 0, stream, pair_expert, n_experts, top, M * top, perm, off, rows, pad_src,
                                pad_of_pair, tile_group));
    TI_CHECK_LAUNCH("moe_route_rows (places)");
    return 0;
}

// z: [places, H] of the engine's type; place_of_pair: int32 [M * top] or null (pair p sits at row p); pair_w: float32
// [M * top] or null (ones); shared_out: [M, H] or null; gate_logit: float32, token m's at gate_logit[m * gate_stride], or null.
extern "C" int ti_moe_combine_gated(const void* z, const int* place_of_pair, const float* pair_w, const void* shared_out,
                                    const float* gate_logit, long long gate_stride, void* out, int M, int H, int top, int dtype,
                                    cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && H > 0 && top > 0, "moe_combine_gated: bad sizes");
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        if (H % 8 == 0 && ((reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(shared_out) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
            // (64 / 128 / 256 threads, us: 777 tokens of 2,048 5.4 / 3.5 / 3.5, eight 4.1 / 2.6 / 1.9, 777 of 1,024 3.1 / 2.2 / 3.2)
            const int threads = H >= 2048 ? 256 : H >= 1024 ? 128 : 64;
            TI_CUDA(ti_launch_class<1>(moe_combine_gated_vec_kernel<T>, dim3(M), dim3(threads), 0, stream, (const T*)z, place_of_pair,
                                       pair_w, (const T*)shared_out, gate_logit, gate_stride, (T*)out, H, top));
            TI_CHECK_LAUNCH("moe_combine_gated");
            return 0;
        }
        TI_CUDA(ti_launch_class<1>(moe_combine_gated_kernel<T>, dim3(M), dim3(H <= 256 ? 64 : 256), 0, stream, (const T*)z, place_of_pair,
                                   pair_w, (const T*)shared_out, gate_logit, gate_stride, (T*)out, H, top));
        TI_CHECK_LAUNCH("moe_combine_gated");
        return 0;
    });
}
