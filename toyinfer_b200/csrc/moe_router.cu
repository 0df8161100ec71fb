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
            const float s = 1.0f / (1.0f + expf(-bz));
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
            s_of[j] = SOFT ? expf(bl - zmax) * inv : 1.0f / (1.0f + expf(-bl));
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
    const float g = (shared_out && gate_logit) ? 1.0f / (1.0f + expf(-gate_logit[m * gate_stride])) : 1.f;
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
    const float g = (shared_out && gate_logit) ? 1.0f / (1.0f + expf(-gate_logit[m * gate_stride])) : 1.f;
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
