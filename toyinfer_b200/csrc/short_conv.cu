// A short causal convolution over time, one filter per channel, with the last inputs of every
// sequence kept as state.
//
// For channel c of a sequence whose inputs are x_0, x_1, ... (x_t = projection + input bias):
//     y_t = act(sum_{j < n} taps[c][j] * x_{t - (n - 1 - j)} + out_bias[c]),    x_s = 0 for s < 0,
// so the last column of `taps` weighs the current token.  The state of a sequence is its last
// n - 1 inputs, float32 [n - 1, C] (oldest first), zero when the sequence starts; a step reads it
// for its first tokens and leaves it holding the step's last inputs, however many tokens the
// step brings.  act: 0 none, 1 silu.
//
// short_conv: grid (token chunks of 64, channel groups, sequences); a thread owns one channel and
// walks its chunk's tokens with the window in registers.  A sequence whose new tokens fit one
// chunk gets its state updated by the same block; for longer ones short_conv_tail runs afterwards
// (other blocks still read the old state while the chunk with the last tokens is at work).
//
// short_conv_vec: the same for up to four taps and rows that can be read four channels at a time: a thread owns
// four channels and walks 16 tokens, eight rows on their way together.  2,048 tokens of 6,144 channels: 39 us a thread a channel
// (a wait for memory per token), 27 so (float32 47 and 32); 64 tokens 17 and 8.  Eight channels a thread: 162 registers, three
// blocks an SM, twice the time.
// Rows past the last sequence's are nobody's; they are set to zero.
#include "common.cuh"

#include <type_traits>

namespace {

constexpr int VEC_CHUNK = 16;       // tokens of a block of short_conv_vec
constexpr int CONV_CHUNK = 64, CONV_THREADS = 128, MAX_TAPS = 8;

__device__ __forceinline__ float conv_act(float z, int act) { return act == 1 ? ti_over(z, 1.0f + expf(-z)) : z; }

template <typename T, int N>
__global__ void __launch_bounds__(CONV_THREADS)
short_conv_kernel(const T* __restrict__ x, long long ldx, const float* __restrict__ in_bias, const float* __restrict__ taps,
                  const float* __restrict__ out_bias, int act, float* __restrict__ state, long long slot_stride,
                  T* __restrict__ out, long long ldo, const int* __restrict__ cu_new, const int* __restrict__ seq_slot, int C, int M) {
    ti_pdl_trigger();
    const int c = blockIdx.y * CONV_THREADS + threadIdx.x;
    float w[N];
    float ib = 0.f, ob = 0.f;
    if (c < C) {
#pragma unroll
        for (int j = 0; j < N; j++) w[j] = taps[(size_t)c * N + j];
        if (in_bias) ib = in_bias[c];
        if (out_bias) ob = out_bias[c];
    }
    ti_pdl_sync();
    x = ti_dependent(x);
    const int b = blockIdx.z;
    if (b == 0 && blockIdx.x == 0 && c < C)
        for (int m = cu_new[gridDim.z]; m < M; m++) out[(size_t)m * ldo + c] = from_f32<T>(0.f);
    const int tok0 = cu_new[b], n = cu_new[b + 1] - tok0;
    const int t0 = blockIdx.x * CONV_CHUNK;
    if (t0 >= n || c >= C) return;
    const int nt = min(CONV_CHUNK, n - t0);
    float* st = state + (size_t)seq_slot[b] * slot_stride;      // [N - 1, C]
    // win[j]: the input N - 1 - j tokens before the one at hand
    float win[N > 1 ? N - 1 : 1];
#pragma unroll
    for (int j = 0; j < N - 1; j++) {
        const int s = t0 - (N - 1 - j);                 // index among the step's tokens; negative: from the state
        win[j] = s >= 0 ? to_f32(x[(size_t)(tok0 + s) * ldx + c]) + ib : st[(size_t)(N - 1 + s) * C + c];
    }
    for (int t = 0; t < nt; t++) {
        const float cur = to_f32(x[(size_t)(tok0 + t0 + t) * ldx + c]) + ib;
        float a = ob;
#pragma unroll
        for (int j = 0; j < N - 1; j++) a = fmaf(w[j], win[j], a);
        a = fmaf(w[N - 1], cur, a);
        out[(size_t)(tok0 + t0 + t) * ldo + c] = from_f32<T>(conv_act(a, act));
#pragma unroll
        for (int j = 0; j + 1 < N - 1; j++) win[j] = win[j + 1];
        if constexpr (N > 1) win[N - 2] = cur;
    }
    if (n <= CONV_CHUNK) {
#pragma unroll
        for (int j = 0; j < N - 1; j++) st[(size_t)j * C + c] = win[j];
    }
}

template <typename T, int N>
__global__ void __launch_bounds__(CONV_THREADS)
short_conv_vec_kernel(const T* __restrict__ x, long long ldx, const float* __restrict__ in_bias, const float* __restrict__ taps,
                      const float* __restrict__ out_bias, int act, float* __restrict__ state, long long slot_stride,
                      T* __restrict__ out, long long ldo, const int* __restrict__ cu_new, const int* __restrict__ seq_slot, int C, int M) {
    ti_pdl_trigger();
    constexpr int V = 4, AHEAD = 8;
    using Run = std::conditional_t<sizeof(T) == 2, uint2, uint4>;       // four channels
    const int c = (blockIdx.y * CONV_THREADS + threadIdx.x) * V;
    if (c >= C) return;
    float w[V][N], ib[V], ob[V];
#pragma unroll
    for (int e = 0; e < V; e++) {
#pragma unroll
        for (int j = 0; j < N; j++) w[e][j] = taps[(size_t)(c + e) * N + j];
        ib[e] = in_bias ? in_bias[c + e] : 0.f;
        ob[e] = out_bias ? out_bias[c + e] : 0.f;
    }
    ti_pdl_sync();
    x = ti_dependent(x);
    const int b = blockIdx.z;
    if (b == 0 && blockIdx.x == 0)
        for (int m = cu_new[gridDim.z]; m < M; m++) *reinterpret_cast<Run*>(out + (size_t)m * ldo + c) = Run{};
    const int tok0 = cu_new[b], n = cu_new[b + 1] - tok0;
    const int t0 = blockIdx.x * VEC_CHUNK;
    if (t0 >= n) return;
    const int nt = min(VEC_CHUNK, n - t0);
    float* st = state + (size_t)seq_slot[b] * slot_stride;      // [N - 1, C]
    const T* xr = x + (size_t)(tok0 + t0) * ldx + c;
    // win[j]: the input N - 1 - j tokens before the one at hand
    float win[N > 1 ? N - 1 : 1][V];
#pragma unroll
    for (int j = 0; j < N - 1; j++) {
        const int s = t0 - (N - 1 - j);
        if (s >= 0) {
            const Run r = *reinterpret_cast<const Run*>(xr + ((long long)j - (N - 1)) * ldx);
#pragma unroll
            for (int e = 0; e < V; e++) win[j][e] = to_f32(reinterpret_cast<const T*>(&r)[e]) + ib[e];
        } else {
#pragma unroll
            for (int e = 0; e < V; e += 4) {
                const float4 r = *reinterpret_cast<const float4*>(st + (size_t)(N - 1 + s) * C + c + e);
                win[j][e] = r.x; win[j][e + 1] = r.y; win[j][e + 2] = r.z; win[j][e + 3] = r.w;
            }
        }
    }
    for (int u0 = 0; u0 < nt; u0 += AHEAD) {
        Run r[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; u++)
            if (u0 + u < nt) r[u] = *reinterpret_cast<const Run*>(xr + (size_t)(u0 + u) * ldx);
#pragma unroll
        for (int u = 0; u < AHEAD; u++) {
            if (u0 + u >= nt) break;
            Run y;
#pragma unroll
            for (int e = 0; e < V; e++) {
                const float cur = to_f32(reinterpret_cast<const T*>(&r[u])[e]) + ib[e];
                float a = ob[e];
#pragma unroll
                for (int j = 0; j < N - 1; j++) a = fmaf(w[e][j], win[j][e], a);
                a = fmaf(w[e][N - 1], cur, a);
                reinterpret_cast<T*>(&y)[e] = from_f32<T>(conv_act(a, act));
#pragma unroll
                for (int j = 0; j + 1 < N - 1; j++) win[j][e] = win[j + 1][e];
                if constexpr (N > 1) win[N - 2][e] = cur;
            }
            *reinterpret_cast<Run*>(out + (size_t)(tok0 + t0 + u0 + u) * ldo + c) = y;
        }
    }
    if (n <= VEC_CHUNK) {
#pragma unroll
        for (int j = 0; j < N - 1; j++)
#pragma unroll
            for (int e = 0; e < V; e += 4)
                *reinterpret_cast<float4*>(st + (size_t)j * C + c + e) = make_float4(win[j][e], win[j][e + 1], win[j][e + 2], win[j][e + 3]);
    }
}

// The state of the sequences with more than one chunk of new tokens: their last N - 1 inputs.
template <typename T, int N>
__global__ void short_conv_tail_kernel(const T* __restrict__ x, long long ldx, const float* __restrict__ in_bias,
                                       float* __restrict__ state, long long slot_stride, const int* __restrict__ cu_new,
                                       const int* __restrict__ seq_slot, int C, int chunk) {
    ti_pdl_trigger();
    ti_pdl_sync();
    x = ti_dependent(x);
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    const int tok0 = cu_new[b], n = cu_new[b + 1] - tok0;
    if (n <= chunk || c >= C) return;
    float* st = state + (size_t)seq_slot[b] * slot_stride;
    const float ib = in_bias ? in_bias[c] : 0.f;
#pragma unroll
    for (int j = 0; j < N - 1; j++) st[(size_t)j * C + c] = to_f32(x[(size_t)(tok0 + n - (N - 1) + j) * ldx + c]) + ib;
}

template <typename F>
int dispatch_taps(int n, F&& f) {
    switch (n) {
        case 1: return f(std::integral_constant<int, 1>());
        case 2: return f(std::integral_constant<int, 2>());
        case 3: return f(std::integral_constant<int, 3>());
        case 4: return f(std::integral_constant<int, 4>());
        case 5: return f(std::integral_constant<int, 5>());
        case 6: return f(std::integral_constant<int, 6>());
        case 7: return f(std::integral_constant<int, 7>());
        default: return f(std::integral_constant<int, 8>());
    }
}

}  // namespace

// x: [M, C] of the engine's type with row stride ldx; in_bias, out_bias: float32 [C] or null; taps: float32 [C, n];
// state: float32, sequence slot s at state + s * slot_stride holds [n - 1, C]; out: [M, C] with row stride ldo (rows past the last
// sequence's become zero).  launched: the number of kernels.
extern "C" int ti_short_conv(const void* x, long long ldx, const float* in_bias, const float* taps, const float* out_bias,
                             int act, float* state, long long slot_stride, void* out, long long ldo, const int* cu_new,
                             const int* seq_slot, int n_seq, int max_new, int M, int C, int n_taps, int* launched, int dtype, cudaStream_t stream) {
    *launched = 0;
    if (n_seq == 0 || max_new == 0) return 0;
    TI_REQUIRE(n_seq > 0 && n_seq <= 65535 && max_new > 0 && C > 0, "short_conv: bad sizes");
    TI_REQUIRE(n_taps >= 1 && n_taps <= MAX_TAPS, "short_conv: %d taps are not supported (1 to %d)", n_taps, MAX_TAPS);
    TI_REQUIRE(act == 0 || act == 1, "short_conv: unknown activation %d", act);
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        constexpr int V = 4;
        const bool vec = n_taps <= 4 && C % V == 0 && ldx % V == 0 && ldo % V == 0 && slot_stride % 4 == 0 &&
                         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & (V * sizeof(T) - 1)) == 0 &&
                         (reinterpret_cast<uintptr_t>(state) & 15) == 0;
        const int chunk = vec ? VEC_CHUNK : CONV_CHUNK, per_block = CONV_THREADS * (vec ? V : 1);
        const int chunks = (max_new + chunk - 1) / chunk, groups = (C + per_block - 1) / per_block;
        TI_REQUIRE(groups <= 65535, "short_conv: %d channels are too many for one launch", C);
        return dispatch_taps(n_taps, [&](auto nv) -> int {
            constexpr int N = decltype(nv)::value;
            if constexpr (N <= 4) {
                if (vec)
                    TI_CUDA(ti_launch(short_conv_vec_kernel<T, N>, dim3(chunks, groups, n_seq), dim3(CONV_THREADS), 0, stream, (const T*)x, ldx,
                                      in_bias, taps, out_bias, act, state, slot_stride, (T*)out, ldo, cu_new, seq_slot, C, M));
            }
            if (!vec)
                TI_CUDA(ti_launch(short_conv_kernel<T, N>, dim3(chunks, groups, n_seq), dim3(CONV_THREADS), 0, stream, (const T*)x, ldx,
                                  in_bias, taps, out_bias, act, state, slot_stride, (T*)out, ldo, cu_new, seq_slot, C, M));
            TI_CHECK_LAUNCH("short_conv");
            *launched = 1;
            if (chunks > 1 && N > 1) {
                TI_CUDA(ti_launch(short_conv_tail_kernel<T, N>, dim3((C + CONV_THREADS - 1) / CONV_THREADS, n_seq), dim3(CONV_THREADS), 0, stream,
                                  (const T*)x, ldx, in_bias, state, slot_stride, cu_new, seq_slot, C, chunk));
                TI_CHECK_LAUNCH("short_conv_tail");
                *launched = 2;
            }
            return 0;
        });
    });
}
