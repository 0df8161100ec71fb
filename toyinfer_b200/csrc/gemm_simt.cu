// out[M, N] = x[M, K] * W[N, K]^T on the CUDA cores, 32-bit accumulation.
//
// Two kernels.  `gemm_tile_kernel` (128x128x16 tiles, 8x8 per thread, FFMA) is the product of
// more than 16 tokens whose rows do not start on 16-byte boundaries: what the tensor-core kernels
// (gemm_tcgen05.cu, and gemm_f32_split.cu for float32) cannot load.
// `gemv_rows_kernel` serves a handful of tokens (M <= 16): each warp streams R weight
// rows once and multiplies them with up to eight activation rows, so decode at a small
// batch is bound by the read of W.
//
// Sums of thousands of 32-bit products are kept short: the tiled kernel adds up 128
// consecutive k in one register and then moves that partial sum into a second one, so
// that rounding errors grow with the square root of K/128 + 128 rather than of K (with
// K = 9,728 a plain running sum alone put logits 1.5e-5 off the exact value; the few-row
// kernel's sums are short already: a lane's share of the row, then a tree over the warp).
//
// Same contraction as the reference's src/decode.cu:202-236 (one token) and
// src/prefill.cu:124-161 (one block per output element, W re-read for every token);
// weights are [out, in] row-major, no bias.
#include "common.cuh"

#include <type_traits>

// ---------------------------------------------------------------------------
// tiled kernel
// ---------------------------------------------------------------------------
namespace {
constexpr int BM = 128, BN = 128, BK = 16, PAD = 4, TILE_THREADS = 256;
constexpr int FLUSH_TILES = 8;      // partial sums over FLUSH_TILES * BK = 128 k are moved into the totals

template <typename T, typename OT>
__global__ void __launch_bounds__(TILE_THREADS)
gemm_tile_kernel(const T* __restrict__ X, const T* __restrict__ W, OT* __restrict__ out,
                 int M, int N, int K, long long ldx, long long ldw, long long ldo) {
    ti_pdl_trigger();
    __shared__ float As[BK][BM + PAD];
    __shared__ float Bs[BK][BN + PAD];
    ti_pdl_sync();
    X = ti_dependent(X);
    const int t = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int ty = t / 16, tx = t % 16;
    float acc[8][8], total[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = total[i][j] = 0.f;

    // loader mapping: 256 threads cover 64 rows x 4 groups of 4 k; two passes for 128 rows
    const int lr = t / 4, lk = (t % 4) * 4;
    int since_flush = 0;
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const int r = lr + p * 64;
            const int gm = m0 + r, gn = n0 + r;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int gk = k0 + lk + j;
                As[lk + j][r] = (gm < M && gk < K) ? to_f32(X[(size_t)gm * ldx + gk]) : 0.f;
                Bs[lk + j][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.f;
            }
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            float a[8], b[8];
            const float4 a0 = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4*>(&As[kk][64 + ty * 4]);
            const float4 b0 = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
            const float4 b1 = *reinterpret_cast<const float4*>(&Bs[kk][64 + tx * 4]);
            a[0] = a0.x; a[1] = a0.y; a[2] = a0.z; a[3] = a0.w; a[4] = a1.x; a[5] = a1.y; a[6] = a1.z; a[7] = a1.w;
            b[0] = b0.x; b[1] = b0.y; b[2] = b0.z; b[3] = b0.w; b[4] = b1.x; b[5] = b1.y; b[6] = b1.z; b[7] = b1.w;
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (++since_flush == FLUSH_TILES) {
            since_flush = 0;
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) { total[i][j] += acc[i][j]; acc[i][j] = 0.f; }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] += total[i][j];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int gm = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int gn = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + (j - 4));
            if (gn < N) out[(size_t)gm * ldo + gn] = from_f32<OT>(acc[i][j]);
        }
    }
}

// ---------------------------------------------------------------------------
// few rows: a warp takes R neighbouring weight rows and up to eight activation rows, its lanes along K
// ---------------------------------------------------------------------------
constexpr int GV_THREADS = 256, GV_WARPS = GV_THREADS / 32;
constexpr long long ROWS_LARGE = 1 << 19;      // weights from which several tokens take four rows a warp

// Four weight rows a warp: every piece of an activation row, read from L1, then feeds four of them (one row a warp was bound by those
// reads at eight tokens); one row, or a pair, where the matrix is small.  MR activation rows, 1, 2, 4 or 8 (those past the end repeat
// the last, without a branch that would keep their loads from running ahead).  KS > 1: the warps of a block share a group of rows,
// each a slice of K, and meet in shared memory: matrices of few rows would otherwise give every SM a few warps, each with a long chain
// of loads.  The sums are added up over the lanes by exchanges that halve the sums each lane still holds.
// PAIR: rows come in (gate, up) pairs, out is ti_gate_pair of them, [M, N / 2].
// us, one row a warp without slices / so, at 1, 4 and 8 tokens: 512 x 4,096 11.3, 18.3, 26 / 3.6, 4.3, 5.3; 2,048 x 2,048 8.1, 11.6, 15.6 /
// 4.7, 5.4, 6.7; 2,560 x 9,728 40, 80, 117 / 17, 27, 41; 19,456 x 2,560 41, 56, 83 / 32, 43, 68 (the read of the weights alone takes 30);
// 384 x 96 2.4, 2.7, 3.0 / 1.6, 1.8, 1.8; 1,024 x 400 at 8 tokens 5.1 / 3.0, gated 6.3 / 3.2.  Rows off the 16-byte boundary, elements one by
// one, at 1, 5 and 16 tokens: float32 2,048 x 2,045 17.4, 18.8, 22.7 / 3.2, 7.8, 13.9; bfloat16 9,728 x 2,559 50, 53, 108 / 21, 49, 74.
template <typename T, typename OT, int V, int R, int MR, int KS, bool PAIR>
__global__ void __launch_bounds__(GV_THREADS, R == 4 ? (MR >= 4 ? 2 : 3) : MR == 8 ? 2 : MR == 4 ? 3 : 4)
gemv_rows_kernel(const T* __restrict__ X, const T* __restrict__ W, OT* __restrict__ out,
                 int M, int N, int K, long long ldx, long long ldw, long long ldo, int kind, float limit) {
    ti_pdl_trigger();
    constexpr int AHEAD = V == 1 && MR == 8 && KS == 1 ? 8 : R == 4 ? (MR == 1 || MR == 4 ? 3 : 2) : R * MR >= 16 ? 2 : 4, SUMS = R * MR;
    __shared__ float part[KS > 1 ? GV_WARPS * 32 : 1];
    ti_pdl_sync();
    X = ti_dependent(X);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int mb = blockIdx.y * MR, rows = min(MR, M - mb);
    const int slice = warp % KS, n_groups = gridDim.x * (GV_WARPS / KS);
    constexpr int STEP = 32 * V;
    const int per = ((K + STEP - 1) / STEP + KS - 1) / KS * STEP, k_lo = slice * per, k_hi = min(K, k_lo + per);
    struct alignas(sizeof(T) * V) Pack { T v[V]; };
    for (int group = blockIdx.x * (GV_WARPS / KS) + warp / KS; KS > 1 || (long long)group * R < N; group += n_groups) {
        const int n0 = group * R;
        float acc[SUMS];                               // [weight row][activation row]
#pragma unroll
        for (int i = 0; i < SUMS; i++) acc[i] = 0.f;
        const T* wr[R];
#pragma unroll
        for (int i = 0; i < R; i++) wr[i] = W + (size_t)min(n0 + i, N - 1) * ldw;      // rows past the end repeat the last; never stored
        for (int k0 = k_lo + lane * V; k0 < k_hi; k0 += STEP * AHEAD) {
            Pack pw[AHEAD][R];
#pragma unroll
            for (int u = 0; u < AHEAD; u++)
#pragma unroll
                for (int i = 0; i < R; i++)
                    if (k0 + u * STEP < k_hi) pw[u][i] = *reinterpret_cast<const Pack*>(wr[i] + k0 + u * STEP);
#pragma unroll
            for (int u = 0; u < AHEAD; u++) {
                const int k = k0 + u * STEP;
                if (k >= k_hi) break;
#pragma unroll
                for (int r = 0; r < MR; r++) {
                    const Pack px = *reinterpret_cast<const Pack*>(X + (size_t)(mb + min(r, rows - 1)) * ldx + k);
#pragma unroll
                    for (int i = 0; i < R; i++)
#pragma unroll
                        for (int j = 0; j < V; j++) acc[i * MR + r] = fmaf(to_f32(pw[u][i].v[j]), to_f32(px.v[j]), acc[i * MR + r]);
                }
            }
        }
        // lane l: the sum number l mod SUMS (weight row l / MR, activation row l % MR)
#pragma unroll
        for (int half = SUMS / 2; half > 0; half >>= 1) {
            const bool upper = lane & half;
#pragma unroll
            for (int i = 0; i < half; i++) {
                const float keep = upper ? acc[i + half] : acc[i], give = upper ? acc[i] : acc[i + half];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
            }
        }
        float s = acc[0];
#pragma unroll
        for (int o = SUMS; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if constexpr (KS > 1) {
            part[warp * 32 + lane] = s;
            __syncthreads();
            if (slice == 0) {
#pragma unroll
                for (int q = 1; q < KS; q++) s += part[(warp + q) * 32 + lane];
            }
        }
        const int r = lane % MR, n = n0 + lane / MR;
        const float up = PAIR ? __shfl_xor_sync(0xffffffffu, s, MR) : 0.f;
        if ((KS == 1 || slice == 0) && lane < SUMS && r < rows && n < N) {
            if (PAIR) {
                if ((n & 1) == 0) out[(size_t)(mb + r) * ldo + (n >> 1)] = from_f32<OT>(ti_gate_pair(s, up, kind, limit));
            } else {
                out[(size_t)(mb + r) * ldo + n] = from_f32<OT>(s);
            }
        }
        if (KS > 1) return;
    }
}

template <typename T, typename OT, int V, int R, int MR, int KS, bool PAIR>
int launch_rows(const void* x, const void* w, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo, int kind, float limit,
                cudaStream_t stream) {
    const int groups = GV_WARPS / KS * R;           // weight rows of a block
    long long blocks = ((long long)N + groups - 1) / groups;
    if (KS == 1) blocks = blocks < 8LL * ti_sm_count() ? blocks : 8LL * ti_sm_count();
    const dim3 grid((unsigned)blocks, (M + MR - 1) / MR);
    TI_CUDA(ti_launch(gemv_rows_kernel<T, OT, V, R, MR, KS, PAIR>, grid, dim3(GV_THREADS), 0, stream, (const T*)x, (const T*)w, (OT*)out, M, N, K, ldx, ldw, ldo,
                      kind, limit));
    TI_CHECK_LAUNCH("linear (few rows)");
    return 0;
}

bool rows_aligned(const void* x, const void* w, int K, long long ldx, long long ldw, int V) {
    return K % V == 0 && ldx % V == 0 && ldw % V == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

// Four weight rows a warp, the contraction in as many slices as give the SMs warps.
template <typename T, typename OT, int V, int MR, bool PAIR>
int launch_rows_sliced(const void* x, const void* w, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo, int kind, float limit,
                       cudaStream_t stream) {
    const int groups = (N + 3) / 4, steps = (K + 32 * V - 1) / (32 * V);      // groups of four rows, turns of a warp over K
    int ks = 1;
    while (ks < 8 && groups * ks < 16 * ti_sm_count() && steps >= ks * 4) ks *= 2;
    switch (ks) {
        case 1: return launch_rows<T, OT, V, 4, MR, 1, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
        case 2: return launch_rows<T, OT, V, 4, MR, 2, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
        case 4: return launch_rows<T, OT, V, 4, MR, 4, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
        default: return launch_rows<T, OT, V, 4, MR, 8, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
    }
}

// 32-bit operands on 16-byte boundaries.
template <int MR, bool PAIR>
int launch_rows_f32(const void* x, const void* w, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo, int kind, float limit,
                    cudaStream_t stream) {
    constexpr int R1 = PAIR ? 2 : 1;
    if ((long long)N * K < ROWS_LARGE) return launch_rows<float, float, 4, R1, MR, 1, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
    return launch_rows_sliced<float, float, 4, MR, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
}
template <bool PAIR>
int launch_rows_f32(const void* x, const void* w, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo, int kind, float limit,
                    cudaStream_t stream) {
    if (M == 1) return launch_rows_f32<1, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
    if (M == 2) return launch_rows_f32<2, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
    if (M <= 4) return launch_rows_f32<4, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
    return launch_rows_f32<8, PAIR>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
}

template <typename T, typename OT>
int launch_simt(const void* x, const void* w, void* out, int M, int N, int K, long long ldx,
                long long ldw, long long ldo, cudaStream_t stream) {
    if (M <= 16) {
        if constexpr (sizeof(T) == 4)
            if (rows_aligned(x, w, K, ldx, ldw, 4)) return launch_rows_f32<false>(x, w, out, M, N, K, ldx, ldw, ldo, 0, 0.f, stream);
        // (bfloat16 comes here off the 16-byte boundary only: gemm_skinny.cu takes the rest)
        if (M == 1) return launch_rows_sliced<T, OT, 1, 1, false>(x, w, out, M, N, K, ldx, ldw, ldo, 0, 0.f, stream);
        if (M == 2) return launch_rows_sliced<T, OT, 1, 2, false>(x, w, out, M, N, K, ldx, ldw, ldo, 0, 0.f, stream);
        if (M <= 4) return launch_rows_sliced<T, OT, 1, 4, false>(x, w, out, M, N, K, ldx, ldw, ldo, 0, 0.f, stream);
        return launch_rows_sliced<T, OT, 1, 8, false>(x, w, out, M, N, K, ldx, ldw, ldo, 0, 0.f, stream);
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    TI_REQUIRE(grid.y <= 65535, "linear: %d rows exceed the tiled kernel's grid", M);
    TI_CUDA(ti_launch(gemm_tile_kernel<T, OT>, grid, dim3(TILE_THREADS), 0, stream, (const T*)x, (const T*)w, (OT*)out, M, N, K, ldx, ldw, ldo));
    TI_CHECK_LAUNCH("linear (tiled)");
    return 0;
}
}  // namespace

// dtype: element type of x and W.  out_f32 != 0: float32 output whatever dtype is.
extern "C" int ti_linear_simt(const void* x, const void* w, void* out, int M, int N, int K,
                              long long ldx, long long ldw, long long ldo, int dtype, int out_f32,
                              cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    TI_REQUIRE(M > 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    TI_REQUIRE(ldx >= K && ldw >= K && ldo >= N, "linear: a leading dimension is smaller than its row");
    if (dtype == TI_F32) return launch_simt<float, float>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    TI_REQUIRE(dtype == TI_BF16, "linear: unknown element type code %d", dtype);
    if (out_f32) return launch_simt<bf16, float>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    return launch_simt<bf16, bf16>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
}

// The same for up to 16 tokens of 32-bit operands on 16-byte boundaries whose weight rows come in (gate, up) pairs: out[M, N / 2] =
// ti_gate_pair (kind 1: silu, 2: gelu in the tanh form, 3: the clamped pair with its limit).
extern "C" int ti_linear_rows_gated(const void* x, const void* w, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo,
                                    int kind, float limit, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    TI_REQUIRE(M > 0 && M <= 16 && N > 0 && N % 2 == 0 && K > 0 && kind >= 1 && kind <= 3, "linear (few rows, gated): bad sizes M=%d N=%d K=%d, kind %d", M, N, K, kind);
    TI_REQUIRE(ldx >= K && ldw >= K && ldo >= N / 2, "linear (few rows, gated): a leading dimension is smaller than its row");
    TI_REQUIRE(rows_aligned(x, w, K, ldx, ldw, 4), "linear (few rows, gated): rows are not 16-byte aligned");
    return launch_rows_f32<true>(x, w, out, M, N, K, ldx, ldw, ldo, kind, limit, stream);
}
