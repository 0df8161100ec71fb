// The grouped products of a mixture of experts straight from global memory into registers: every weight of a chosen expert is
// read once for up to 8 (bfloat16: 32) of its places.  Included by moe_grouped.cu, which holds the entry point and the rule.
//
// A place is a (token, choice) pair in the order grouped by expert; tile t of the walk over the groups is a run of at most TM
// places of one expert.  Every warp finds its tile itself: lanes read 32 experts' offsets at once and scan their tile counts (one
// thread walking the experts waited for memory 16 to 32 times in a row, some 10 us a kernel).
//
// With few places a product is a read of the chosen experts' matrices; with many the places' rows come from L1 and the
// weights, for the tiles after a group's first, from L2.
//
// Measured, a layer's step in us, against tiles of 32 places staged in shared memory: 32-bit, 11 tokens of 32 experts (one each,
// 1,024 x 392) 287 -> 27, 17 of 16 (two each, 2,048 x 600) some 500 -> 64, 300 of 16 (four each, 2,048 x 1,024) 1,170 -> 862 (17
// TFLOP/s; a place's piece from L1 feeds sixteen multiplications); bfloat16, 16 experts of 2,048 x 1,024, two each: one token
// 70 -> 25, eight 81 -> 43, forty 113 -> 58 (3.5 TB/s), 160 120 -> 97, the router's shorter chain included (moe_router.cu).
#pragma once

#include "common.cuh"
#include "mma_utils.cuh"

#include <type_traits>

namespace timoe {

struct RowsArgs {
    const void* a; long long lda;            // rows of K: the row of place i is a[gather ? perm[i] / top : i]
    const void* W; const void* W2;           // an expert's matrix [N, K]; W2: the second one of a pair, or null
    void* out; long long ldo;                // pair: out[i] = act(gate, up); else out[scatter ? perm[i] : i] = product * scale
    const int* perm; const int* off;
    int n_experts, N, K, top, gather, scatter;
    int relu2;                               // without a pair: every product through the squared ReLU instead of times `scale`
    float scale, limit, alpha, shift;
    long long w_estride;                     // elements from one expert's matrix to the next
};

// The whole warp: expert, first place and number of places of tile t (false: there are fewer tiles).
template <int TM>
__device__ __forceinline__ bool find_tile(const int* off, int n_experts, int t, int& expert, int& first, int& cnt) {
    const int lane = threadIdx.x & 31;
    for (int e0 = 0; e0 < n_experts; e0 += 32) {
        const int e = e0 + lane;
        const int lo = e < n_experts ? off[e] : 0, hi = e < n_experts ? off[e + 1] : 0;
        const int tiles = (hi - lo + TM - 1) / TM;
        int upto = tiles;                                        // tiles of this lane's expert and those before it
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += below;
        }
        const unsigned past = __ballot_sync(0xffffffffu, upto > t);
        if (past) {
            const int src = __ffs(past) - 1;
            const int at = t - __shfl_sync(0xffffffffu, upto - tiles, src);
            expert = e0 + src;
            first = __shfl_sync(0xffffffffu, lo, src) + at * TM;
            cnt = min(TM, __shfl_sync(0xffffffffu, hi, src) - first);
            return true;
        }
        t -= __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// the two products are rounded to the engine's type first, as a kernel after the product would find them
template <typename T>
__device__ __forceinline__ float pair_act(const RowsArgs& a, float gate, float up) {
    const float g = fminf(to_f32(from_f32<T>(gate)), a.limit);
    const float u = fminf(fmaxf(to_f32(from_f32<T>(up)), -a.limit), a.limit);
    return g * (ti_over(1.0f, 1.0f + expf(-a.alpha * g))) * (u + a.shift);
}

// a product without a pair, before it is stored
template <typename T>
__device__ __forceinline__ float single(int relu2, float scale, float x) {
    if (!relu2) return x * scale;
    return sizeof(T) == 2 ? ti_pointwise_bf16(x, 4) : ti_pointwise(x, 4);
}

// 32-bit arithmetic on the CUDA cores.  A warp takes four weight rows (two of each matrix of a pair) and eight places; its lanes
// lie along K, V elements each, two pieces of every weight row on their way together.  A piece of a place's row feeds four weight
// rows, a piece of a weight row eight places.  The 32 sums are added up over the lanes by exchanges that halve the sums each lane
// still holds (31 shuffles instead of 160).  PT warps of a block take the same weight rows for eight places each: groups of many
// places then read a weight from L2 once for 32 of them.  (Sixteen places a warp need 250 registers, one block an SM: 1,200 places
// of 16 experts, width 1,024, 2,048 elements, 1,370 us against 890 in eights.)
constexpr int ROWS_TM = 8, ROWS_THREADS = 256;

template <typename T, int V, int PT, bool PAIR>
__global__ void __launch_bounds__(ROWS_THREADS, 2) moe_rows_kernel(RowsArgs p) {
    ti_pdl_trigger();
    ti_pdl_sync();
    struct alignas(sizeof(T) * V) Pack { T v[V]; };
    constexpr int COLS = PAIR ? 2 : 4;                 // result columns of a warp
    constexpr int AHEAD = 2, TM = ROWS_TM;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int e, first, cnt;
    if (!find_tile<TM * PT>(p.off, p.n_experts, blockIdx.x, e, first, cnt)) return;
    first += warp % PT * TM;
    cnt = min(TM, cnt - warp % PT * TM);
    const int n0 = (blockIdx.y * (ROWS_THREADS / 32 / PT) + warp / PT) * COLS;
    if (n0 >= p.N || cnt <= 0) return;
    const T* w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int n = min(n0 + (PAIR ? (i & 1) : i), p.N - 1);      // rows past the end repeat the last; never stored
        w[i] = (const T*)(PAIR && i >= 2 ? p.W2 : p.W) + (size_t)e * p.w_estride + (size_t)n * p.K;
    }
    int src = 0;
    if (lane < cnt) src = p.gather ? p.perm[first + lane] / p.top : first + lane;
    const T* x[TM];
#pragma unroll
    for (int r = 0; r < TM; r++) x[r] = (const T*)p.a + (size_t)__shfl_sync(0xffffffffu, src, r) * p.lda;

    float acc[4 * TM];                                 // [weight row][place]
#pragma unroll
    for (int i = 0; i < 4 * TM; i++) acc[i] = 0.f;
    // more than half of the places: all eight rows are read (those past the end: row 0 of the matrix, never stored) without a branch
    // that would keep the loads from running ahead of the sums
    auto walk = [&](auto all) {
        for (int k0 = lane * V; k0 < p.K; k0 += 32 * V * AHEAD) {
            Pack pw[AHEAD][4];
#pragma unroll
            for (int u = 0; u < AHEAD; u++)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (k0 + u * 32 * V < p.K) pw[u][i] = *reinterpret_cast<const Pack*>(w[i] + k0 + u * 32 * V);
#pragma unroll
            for (int u = 0; u < AHEAD; u++) {
                const int k = k0 + u * 32 * V;
                if (k >= p.K) break;
#pragma unroll
                for (int r = 0; r < TM; r++) {
                    if (decltype(all)::value || r < cnt) {
                        const Pack px = *reinterpret_cast<const Pack*>(x[r] + k);
#pragma unroll
                        for (int i = 0; i < 4; i++)
#pragma unroll
                            for (int j = 0; j < V; j++) acc[i * TM + r] = fmaf(to_f32(pw[u][i].v[j]), to_f32(px.v[j]), acc[i * TM + r]);
                    }
                }
            }
        }
    };
    if (cnt > 4) walk(std::true_type()); else walk(std::false_type());
#pragma unroll
    for (int half = 16; half > 0; half >>= 1) {
        const bool upper = lane & half;
#pragma unroll
        for (int i = 0; i < half; i++) {
            const float keep = upper ? acc[i + half] : acc[i], give = upper ? acc[i] : acc[i + half];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    const float sum = acc[0];                          // of weight row lane / 8 and place lane % 8
    const float second = __shfl_xor_sync(0xffffffffu, sum, 16);
    const int r = lane & 7, n = n0 + (PAIR ? (lane >> 3 & 1) : lane >> 3);
    if (r >= cnt || n >= p.N || (PAIR && lane >= 16)) return;
    const size_t row = p.scatter ? (size_t)p.perm[first + r] : (size_t)(first + r);
    ((T*)p.out)[row * p.ldo + n] = from_f32<T>(PAIR ? pair_act<T>(p, sum, second) : single<T>(p.relu2, p.scale, sum));
}

// bfloat16 on mma.sync, as the dense product of a few tokens does it (gemm_skinny.cu): a warp owns 16 weight rows (8 of each
// matrix of a pair, so that a lane holds a gate and its up value), lane (g, t) loads 32 bytes of rows g and g + 8 and of place g at
// the same 16 t; the contraction's order is the same renaming on both operands.  NT tiles of 8 places; WPR warps share a row
// group, each a slice of K, and meet in shared memory.
constexpr int SK_WARPS = 8, SK_UNROLL = 2;

__device__ __forceinline__ uint4 load_weights(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

template <int NT, int WPR, bool PAIR>
__global__ void __launch_bounds__(SK_WARPS * 32, NT == 4 ? 2 : 3) moe_skinny_kernel(RowsArgs p) {
    ti_pdl_trigger();
    __shared__ float part[WPR > 1 ? SK_WARPS * NT * 4 * 32 : 1];
    ti_pdl_sync();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int group = warp / WPR, slice = warp % WPR;
    constexpr int R = PAIR ? 8 : 16;                   // result columns of a row group
    int e, first, cnt;
    if (!find_tile<8 * NT>(p.off, p.n_experts, blockIdx.x, e, first, cnt)) return;       // (the whole block leaves)
    const int n0 = (blockIdx.y * (SK_WARPS / WPR) + group) * R;
    const int n_lo = n0 + g, n_hi = PAIR ? n0 + g : n0 + g + 8;
    const bool lo_ok = n_lo < p.N, hi_ok = n_hi < p.N;
    const bf16* w_lo = (const bf16*)p.W + (size_t)e * p.w_estride + (size_t)min(n_lo, p.N - 1) * p.K + 16 * t;
    const bf16* w_hi = (const bf16*)(PAIR ? p.W2 : p.W) + (size_t)e * p.w_estride + (size_t)min(n_hi, p.N - 1) * p.K + 16 * t;
    const bf16* x[NT];
#pragma unroll
    for (int n = 0; n < NT; n++) {
        const int i = first + min(n * 8 + g, cnt - 1);          // places past the end repeat the last; never stored
        x[n] = (const bf16*)p.a + (size_t)(p.gather ? p.perm[i] / p.top : i) * p.lda + 16 * t;
    }
    const int steps = (p.K + 63) >> 6, per = (steps + WPR - 1) / WPR;
    const int s0 = slice * per, s1 = min(steps, s0 + per);
    float c[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.f;
    for (int s = s0; s < s1; s += SK_UNROLL) {
        uint4 wl[SK_UNROLL][2], wh[SK_UNROLL][2];
#pragma unroll
        for (int u = 0; u < SK_UNROLL; u++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int k = (s + u) * 64 + 8 * h;
                const bool ok = s + u < s1 && k + 16 * t < p.K;        // K is a multiple of 8: a piece is whole or absent
                wl[u][h] = ok && lo_ok ? load_weights(w_lo + k) : make_uint4(0, 0, 0, 0);
                wh[u][h] = ok && hi_ok ? load_weights(w_hi + k) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
        for (int n = 0; n < NT; n++) {
            if (n * 8 >= cnt) break;
            uint4 xv[SK_UNROLL][2];
#pragma unroll
            for (int u = 0; u < SK_UNROLL; u++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int k = (s + u) * 64 + 8 * h;
                    xv[u][h] = s + u < s1 && k + 16 * t < p.K ? *reinterpret_cast<const uint4*>(x[n] + k) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
            for (int u = 0; u < SK_UNROLL; u++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t a1[4] = {wl[u][h].x, wh[u][h].x, wl[u][h].y, wh[u][h].y};
                    const uint32_t a2[4] = {wl[u][h].z, wh[u][h].z, wl[u][h].w, wh[u][h].w};
                    mma_bf16(c[n], a1, xv[u][h].x, xv[u][h].y);
                    mma_bf16(c[n], a2, xv[u][h].z, xv[u][h].w);
                }
        }
    }
    if (WPR > 1) {
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) part[((warp * NT + n) * 4 + i) * 32 + lane] = c[n][i];
        __syncthreads();
        if (slice != 0) return;
#pragma unroll
        for (int q = 1; q < WPR; q++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) c[n][i] += part[(((warp + q) * NT + n) * 4 + i) * 32 + lane];
    }
    // c[n][0..1]: row g, places n*8 + 2t, 2t + 1;  c[n][2..3]: row g + 8 (pair: the up row of g), same places
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = n * 8 + 2 * t + i;
            if (r >= cnt) continue;
            const size_t row = p.scatter ? (size_t)p.perm[first + r] : (size_t)(first + r);
            bf16* out = (bf16*)p.out + row * p.ldo;
            if (PAIR) {
                if (lo_ok) out[n_lo] = from_f32<bf16>(pair_act<bf16>(p, c[n][i], c[n][i + 2]));
            } else {
                if (lo_ok) out[n_lo] = from_f32<bf16>(single<bf16>(p.relu2, p.scale, c[n][i]));
                if (hi_ok) out[n_hi] = from_f32<bf16>(single<bf16>(p.relu2, p.scale, c[n][i + 2]));
            }
        }
}

template <typename T, int V, int PT>
int launch_rows(const RowsArgs& p, int P, cudaStream_t stream) {
    const int cols = (p.W2 ? 2 : 4) * (ROWS_THREADS / 32 / PT), nblk = (p.N + cols - 1) / cols, tm = ROWS_TM * PT;
    TI_REQUIRE(nblk <= 65535, "moe_grouped: %d weight rows are too many for one launch", p.N);
    const dim3 grid((P + tm - 1) / tm + min(P, p.n_experts), nblk);
    if (p.W2) TI_CUDA(ti_launch(moe_rows_kernel<T, V, PT, true>, grid, dim3(ROWS_THREADS), 0, stream, p));
    else TI_CUDA(ti_launch(moe_rows_kernel<T, V, PT, false>, grid, dim3(ROWS_THREADS), 0, stream, p));
    TI_CHECK_LAUNCH("moe_grouped");
    return 0;
}

template <int NT, int WPR>
int launch_skinny_form(const RowsArgs& p, int P, cudaStream_t stream) {
    const int cols = (p.W2 ? 8 : 16) * (SK_WARPS / WPR), nblk = (p.N + cols - 1) / cols;
    TI_REQUIRE(nblk <= 65535, "moe_grouped: %d weight rows are too many for one launch", p.N);
    const dim3 grid((P + 8 * NT - 1) / (8 * NT) + min(P, p.n_experts), nblk);
    if (p.W2) TI_CUDA(ti_launch(moe_skinny_kernel<NT, WPR, true>, grid, dim3(SK_WARPS * 32), 0, stream, p));
    else TI_CUDA(ti_launch(moe_skinny_kernel<NT, WPR, false>, grid, dim3(SK_WARPS * 32), 0, stream, p));
    TI_CHECK_LAUNCH("moe_grouped");
    return 0;
}

template <int NT>
int launch_skinny(const RowsArgs& p, int P, cudaStream_t stream) {
    const int steps = (p.K + 63) / 64;
    int wpr = 1;
    while (wpr < 8 && steps >= wpr * 2 * SK_UNROLL) wpr *= 2;      // slices keep a turn's loads
    switch (wpr) {
        case 1: return launch_skinny_form<NT, 1>(p, P, stream);
        case 2: return launch_skinny_form<NT, 2>(p, P, stream);
        case 4: return launch_skinny_form<NT, 4>(p, P, stream);
        default: return launch_skinny_form<NT, 8>(p, P, stream);
    }
}

}  // namespace timoe
