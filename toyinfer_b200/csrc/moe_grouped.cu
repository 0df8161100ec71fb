// Mixture-of-experts feed-forward: tokens grouped by expert, one product kernel over all groups.
//
// A step has P = tokens * top (token, choice) pairs; pair p = m * top + j uses expert
// e_p.  `moe_route_table` takes e_p from a table indexed by the token's id (a router
// without arithmetic: table[id, j]), counts the pairs of every expert and writes them out
// grouped by expert: perm[i] is the pair at place i, off[e] .. off[e + 1] the places of expert e.
// The order inside a group is whatever the atomics gave; no result depends on it, since every
// pair's rows are computed for themselves.
//
// `moe_grouped` is the product, used twice:
//   first product   rows of x gathered by pair (token perm[i] / top), expert e's gate and up
//                   matrices, then the expert's activation, into y[i] (places, grouped)
//   second product  rows y[i], expert e's down matrix, result scattered to z[perm[i]] (pairs in
//                   the tokens' order), scaled by the pair's weight
// A tile of places lies inside one expert's group (groups are walked tile by tile: the grid has an upper bound of tiles,
// ceil(P / tile) + experts).  32-bit operands, and bfloat16 groups of few places, run from registers (moe_rows.cuh); bfloat16
// groups of some tens of places as shared-memory tiles on mma.sync (below), of many on tcgen05 (gemm_tcgen05_grouped.cu); rows off the
// 16-byte boundary with many places as shared-memory tiles on the CUDA cores (below).
//
// `moe_combine`: out[m] = sum_j z[m * top + j], summed in the order of j.
//
// The expert's activation (ACT_CLAMPED_SWISH): g' = min(g, limit), u' = clamp(u, -limit, limit),
// y = g' * sigmoid(alpha * g') * (u' + shift).  (limit = infinity, alpha = 1, shift = 0: silu(g) * u.)
// `relu2` (the dense feed-forward's activation, x -> max(x, 0)^2) is here as well.
#include "common.cuh"
#include "moe_rows.cuh"

namespace {

constexpr int RT_THREADS = 1024;

__global__ void moe_route_table_kernel(const int* __restrict__ ids, const int* __restrict__ table, int vocab, int top,
                                       int n_experts, int M, int* __restrict__ perm, int* __restrict__ off,
                                       int* __restrict__ pair_expert) {
    ti_pdl_trigger();
    extern __shared__ int cnt[];         // [n_experts] counts, then [n_experts + 1] offsets, then [n_experts] cursors
    int* offs = cnt + n_experts;
    int* cur = offs + n_experts + 1;
    ti_pdl_sync();
    ids = ti_dependent(ids);
    const int P = M * top;
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) { cnt[e] = 0; cur[e] = 0; }
    __syncthreads();
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        const int m = p / top, j = p - m * top;
        int id = ids[m];
        id = min(max(id, 0), vocab - 1);
        int e = table[(size_t)id * top + j];
        e = min(max(e, 0), n_experts - 1);
        pair_expert[p] = e;
        atomicAdd(&cnt[e], 1);
    }
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

constexpr int GM = 32, GN = 64, GK = 32, G_THREADS = 256;

// The product of rows off the 16-byte boundary with many places an expert, 32-bit arithmetic: tiles of 32 places x 64 weight rows staged in
// shared memory element by element.  Where such tiles fill the device they read a weight once for 32 places; the register form
// (moe_rows.cuh), whose loads are single elements there, once for 8, and it is bound by them: see staged_tiles below.
// out: PAIR -> out[i, n] = act(gate, up);  else out[(scatter ? perm[i] : i), n] = product * scale.
template <typename T, bool PAIR>
__global__ void __launch_bounds__(G_THREADS)
moe_staged_kernel(const T* __restrict__ a, long long lda, const T* __restrict__ W, const T* __restrict__ W2,
                   T* __restrict__ out, long long ldo, const int* __restrict__ perm, const int* __restrict__ off,
                   int n_experts, int N, int K, int top, int gather, int scatter, int relu2, float scale, float limit, float alpha, float shift,
                   long long w_estride) {
    ti_pdl_trigger();
    __shared__ float As[GK][GM + 1];
    __shared__ float Ws[GK][GN + 1];
    __shared__ float W2s[PAIR ? GK : 1][GN + 1];
    __shared__ int rows[GM];
    __shared__ int where[3];             // expert, first place, places in the tile
    ti_pdl_sync();
    a = ti_dependent(a); perm = ti_dependent(perm); off = ti_dependent(off);
    if (threadIdx.x < 32) {
        int found = -1, at = 0, n = 0;
        if (!timoe::find_tile<GM>(off, n_experts, blockIdx.x, found, at, n)) found = -1;
        if (threadIdx.x == 0) { where[0] = found; where[1] = at; where[2] = n; }
    }
    __syncthreads();
    const int e = where[0], first = where[1], cnt = where[2];
    if (e < 0) return;
    const int n0 = blockIdx.y * GN;
    if (threadIdx.x < GM) {
        const int i = first + threadIdx.x;
        int r = -1;
        if (threadIdx.x < cnt) r = gather ? perm[i] / top : i;
        rows[threadIdx.x] = r;
    }
    __syncthreads();
    const T* We = W + (size_t)e * w_estride;
    const T* W2e = PAIR ? W2 + (size_t)e * w_estride : nullptr;
    // thread (ty, tx): places ty, ty + 8, ty + 16, ty + 24; weight rows tx, tx + 32
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    float acc[4][2], acc2[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) { acc[i][j] = 0.f; acc2[i][j] = 0.f; }
    // (a step's 32 products are added up by themselves: sums of thousands one after another lose a digit)
    for (int k0 = 0; k0 < K; k0 += GK) {
        for (int idx = threadIdx.x; idx < GM * GK; idx += G_THREADS) {
            const int r = idx / GK, kk = idx - r * GK;
            const int src = rows[r];
            As[kk][r] = (src >= 0 && k0 + kk < K) ? to_f32(a[(size_t)src * lda + k0 + kk]) : 0.f;
        }
        for (int idx = threadIdx.x; idx < GN * GK; idx += G_THREADS) {
            const int r = idx / GK, kk = idx - r * GK;
            const bool ok = n0 + r < N && k0 + kk < K;
            Ws[kk][r] = ok ? to_f32(We[(size_t)(n0 + r) * K + k0 + kk]) : 0.f;
            if constexpr (PAIR) W2s[kk][r] = ok ? to_f32(W2e[(size_t)(n0 + r) * K + k0 + kk]) : 0.f;
        }
        __syncthreads();
        float part[4][2] = {}, part2[4][2] = {};
#pragma unroll 8
        for (int kk = 0; kk < GK; kk++) {
            float av[4], wv[2], w2v[2];
#pragma unroll
            for (int i = 0; i < 4; i++) av[i] = As[kk][ty + 8 * i];
#pragma unroll
            for (int j = 0; j < 2; j++) { wv[j] = Ws[kk][tx + 32 * j]; w2v[j] = PAIR ? W2s[kk][tx + 32 * j] : 0.f; }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    part[i][j] = fmaf(av[i], wv[j], part[i][j]);
                    if constexpr (PAIR) part2[i][j] = fmaf(av[i], w2v[j], part2[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) { acc[i][j] += part[i][j]; acc2[i][j] += part2[i][j]; }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = ty + 8 * i;
        if (r >= cnt) continue;
        const int place = first + r;
        const size_t orow = scatter ? (size_t)perm[place] : (size_t)place;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int n = n0 + tx + 32 * j;
            if (n >= N) continue;
            float y;
            if constexpr (PAIR) {
                // the two products are rounded to the engine's type first (as in moe_rows.cuh)
                const float g = fminf(to_f32(from_f32<T>(acc[i][j])), limit);
                const float u = fminf(fmaxf(to_f32(from_f32<T>(acc2[i][j])), -limit), limit);
                y = g * ti_over(1.0f, 1.0f + expf(-alpha * g)) * (u + shift);
            } else {
                y = timoe::single<T>(relu2, scale, acc[i][j]);
            }
            out[orow * ldo + n] = from_f32<T>(y);
        }
    }
}

// The product for bfloat16 groups of some tens of places: `mma.sync m16n8k16` with float32 accumulation.  Tiles of 32 places x
// 128 weight rows, contraction in steps of 64; 8 warps as 2 (places) x 4 (weight rows), a warp 16 x 32.  The tiles of the
// next step are fetched into registers while this step's are multiplied.  Rows in shared memory are padded by 16 bytes, so
// that the eight rows a fragment load touches fall into different banks.  Needs K, lda and the matrices' rows in multiples of
// 8 elements (16-byte loads).  With MI = 2 a tile has 64 places (a warp 32 x 32): every weight fragment then feeds two
// multiplications, which is what the shared memory's bandwidth allows the tensor cores; groups of few places take MI = 1.
constexpr int TN = 128, TK = 64, T_THREADS = 256, T_LD = TK + 8;
// Places an expert on average beyond which a block of the 32-bit product takes 32 of them (30 places, 1,024 x 600, 86 us a step
// against 102; at 5 they would leave three of four warps idle).
constexpr int ROWS_SMALL_PLACES = 12;

// How many tiles of eight places a warp of the bfloat16 product takes from registers (moe_rows.cuh), 0: shared-memory tiles on mma.sync.
// The register form reads an expert's weights once for 8 or 16 of its places (32: slower up to 18 places, where a second tile is the
// exception: 2,048 x 1,024 pairs, 64 experts of 9, 153 us against 117) and grows with its tiles; the tiles below read them once for 32
// and take the same from 1 place to 32, but no less than their chain of steps over K takes, however few experts there are.  So from
// registers with up to eight places, and beyond them as long as its tiles' reads (some 5 TB/s, most of them from L2) take less than that
// chain, 1.65 us a step of 64 (1.3 the shorter chains of a pair).  Weights and steps both grow with K, which cancels.
// us a product, registers / tiles, at 9, 16 and 24 places: 8 experts, 2,048 x 1,280 pairs 22, 28, 37 / 53; 16 experts 39, 53, 66 / 58;
// 32 experts 72, 96, 129 / 92; 64 experts 147, 204, 268 / 149; 64 experts of 1,024 x 256 23, 30, 40 / 31.
// Eight places a warp up to four an expert, us at 1, 2, 4, 6 and 8 places with eight a warp / sixteen: 16 experts, 2,048 x 1,024 pairs 18.7,
// 22.6, 24.6, 29.8, 31.5 / 20.7, 24.9, 27.6, 30.3, 30.9; 64 experts 59, 78, 93, 109, 127 / 64, 85, 100, 108, 114.
constexpr int SKINNY_MAX_PLACES = 24;
int skinny_tiles(int n_experts, int P, int N, int K, bool pair, int sms) {
    if (P <= 4 * n_experts) return 1;
    if (P <= 8 * n_experts) return 2;
    const long long tiles = P / 16 + n_experts / 2;
    if (P > SKINNY_MAX_PLACES * n_experts || tiles * N * (pair ? 2 : 1) > (long long)sms * (pair && K <= 1024 ? 340 : 432)) return 0;
    return P <= 18 * n_experts ? 2 : 4;
}

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool PAIR, int MI>
__global__ void __launch_bounds__(T_THREADS)
moe_grouped_mma_kernel(const bf16* __restrict__ a, long long lda, const bf16* __restrict__ W, const bf16* __restrict__ W2,
                       bf16* __restrict__ out, long long ldo, const int* __restrict__ perm, const int* __restrict__ off,
                       int n_experts, int N, int K, int top, int gather, int scatter, int relu2, float scale, float limit, float alpha, float shift,
                       long long w_estride) {
    ti_pdl_trigger();
    constexpr int TM = 32 * MI;
    __shared__ __align__(16) bf16 As[TM][T_LD];
    __shared__ __align__(16) bf16 Ws[TN][T_LD];
    __shared__ __align__(16) bf16 W2s[PAIR ? TN : 1][T_LD];
    __shared__ int rows[TM];
    __shared__ int where[3];
    ti_pdl_sync();
    a = ti_dependent(a); perm = ti_dependent(perm); off = ti_dependent(off);
    if (threadIdx.x < 32) {
        int found = -1, at = 0, n = 0;
        if (!timoe::find_tile<TM>(off, n_experts, blockIdx.x, found, at, n)) found = -1;
        if (threadIdx.x == 0) { where[0] = found; where[1] = at; where[2] = n; }
    }
    __syncthreads();
    const int e = where[0], first = where[1], cnt = where[2];
    if (e < 0) return;
    const int n0 = blockIdx.y * TN;
    if (threadIdx.x < TM) {
        const int i = first + threadIdx.x;
        rows[threadIdx.x] = threadIdx.x < cnt ? (gather ? perm[i] / top : i) : -1;
    }
    __syncthreads();
    const bf16* We = W + (size_t)e * w_estride;
    const bf16* W2e = PAIR ? W2 + (size_t)e * w_estride : nullptr;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 2, wn = warp & 3;             // the warp's 16 * MI places and 32 weight rows
    const int g = lane >> 2, t4 = lane & 3;
    // what this thread fetches per step: one 16-byte piece of the places' tile, four of each weight tile
    const int ar = tid >> 3, ac = (tid & 7) * 8;
    int a_src[MI];
#pragma unroll
    for (int i = 0; i < MI; i++) a_src[i] = rows[ar + 32 * i];
    uint4 ra[MI], rw[4], rw2[4];
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < MI; i++)
            ra[i] = (a_src[i] >= 0 && k0 + ac < K) ? *reinterpret_cast<const uint4*>(a + (size_t)a_src[i] * lda + k0 + ac) : zero;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = (tid >> 3) + 32 * i;
            const bool ok = n0 + r < N && k0 + ac < K;
            rw[i] = ok ? *reinterpret_cast<const uint4*>(We + (size_t)(n0 + r) * K + k0 + ac) : zero;
            if constexpr (PAIR) rw2[i] = ok ? *reinterpret_cast<const uint4*>(W2e + (size_t)(n0 + r) * K + k0 + ac) : zero;
        }
    };
    float acc[MI][4][4], acc2[MI][PAIR ? 4 : 1][4];
#pragma unroll
    for (int m = 0; m < MI; m++)
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) { acc[m][i][j] = 0.f; if constexpr (PAIR) acc2[m][i][j] = 0.f; }
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += TK) {
        __syncthreads();             // the last step's reads of the tiles are over
#pragma unroll
        for (int i = 0; i < MI; i++) *reinterpret_cast<uint4*>(&As[ar + 32 * i][ac]) = ra[i];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            *reinterpret_cast<uint4*>(&Ws[(tid >> 3) + 32 * i][ac]) = rw[i];
            if constexpr (PAIR) *reinterpret_cast<uint4*>(&W2s[(tid >> 3) + 32 * i][ac]) = rw2[i];
        }
        __syncthreads();
        if (k0 + TK < K) fetch(k0 + TK);
#pragma unroll
        for (int kk = 0; kk < TK; kk += 16) {
            uint32_t af[MI][4];
#pragma unroll
            for (int m = 0; m < MI; m++) {
                const int r0 = (wm * MI + m) * 16 + g;
                af[m][0] = *reinterpret_cast<const uint32_t*>(&As[r0][kk + 2 * t4]);
                af[m][1] = *reinterpret_cast<const uint32_t*>(&As[r0 + 8][kk + 2 * t4]);
                af[m][2] = *reinterpret_cast<const uint32_t*>(&As[r0][kk + 2 * t4 + 8]);
                af[m][3] = *reinterpret_cast<const uint32_t*>(&As[r0 + 8][kk + 2 * t4 + 8]);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int n = wn * 32 + j * 8 + g;
                const uint32_t b0 = *reinterpret_cast<const uint32_t*>(&Ws[n][kk + 2 * t4]);
                const uint32_t b1 = *reinterpret_cast<const uint32_t*>(&Ws[n][kk + 2 * t4 + 8]);
#pragma unroll
                for (int m = 0; m < MI; m++) mma_16816(acc[m][j], af[m], b0, b1);
                if constexpr (PAIR) {
                    const uint32_t c0 = *reinterpret_cast<const uint32_t*>(&W2s[n][kk + 2 * t4]);
                    const uint32_t c1 = *reinterpret_cast<const uint32_t*>(&W2s[n][kk + 2 * t4 + 8]);
#pragma unroll
                    for (int m = 0; m < MI; m++) mma_16816(acc2[m][j], af[m], c0, c1);
                }
            }
        }
    }
    // accumulator j: places g (elements 0, 1) and g + 8 (elements 2, 3) of the warp's 16, weight rows j * 8 + 2 t4, + 1
#pragma unroll
    for (int m = 0; m < MI; m++)
#pragma unroll
    for (int half = 0; half < 2; half++) {
        const int r = (wm * MI + m) * 16 + g + 8 * half;
        if (r >= cnt) continue;
        const int place = first + r;
        const size_t orow = scatter ? (size_t)perm[place] : (size_t)place;
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int n = n0 + wn * 32 + j * 8 + 2 * t4 + c;
                if (n >= N) continue;
                float y;
                if constexpr (PAIR) {
                    const float gt = fminf(to_f32(from_f32<bf16>(acc[m][j][2 * half + c])), limit);
                    const float u = fminf(fmaxf(to_f32(from_f32<bf16>(acc2[m][j][2 * half + c])), -limit), limit);
                    y = gt * (ti_over(1.0f, 1.0f + expf(-alpha * gt))) * (u + shift);
                } else {
                    y = timoe::single<bf16>(relu2, scale, acc[m][j][2 * half + c]);
                }
                out[orow * ldo + n] = from_f32<bf16>(y);
            }
    }
}

template <typename T>
__global__ void moe_combine_kernel(const T* __restrict__ z, T* __restrict__ out, int H, int top) {
    ti_pdl_trigger();
    ti_pdl_sync();
    z = ti_dependent(z);
    const size_t m = blockIdx.x;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float s = 0.f;
        for (int j = 0; j < top; j++) s += to_f32(z[(m * top + j) * H + i]);
        out[m * H + i] = from_f32<T>(s);
    }
}

// For the tcgen05 grouped product: every expert's places padded to whole tiles of 128.  pad_src[i] is the token row that
// padded place i takes its input from (-1: a padding row), pad_of_pair[p] the padded place of pair p, tile_group[t] the
// expert of tile t (-1: none).  One block.
__global__ void moe_pad_plan_kernel(const int* __restrict__ perm, const int* __restrict__ off, int n_experts, int P, int top,
                                    int rows, int* __restrict__ pad_src, int* __restrict__ pad_of_pair, int* __restrict__ tile_group) {
    ti_pdl_trigger();
    extern __shared__ int poff[];        // [n_experts + 1] padded offsets, then the offsets themselves
    int* uoff = poff + n_experts + 1;
    ti_pdl_sync();
    perm = ti_dependent(perm); off = ti_dependent(off);
    for (int e = threadIdx.x; e <= n_experts; e += blockDim.x) uoff[e] = off[e];
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0;
        for (int e = 0; e < n_experts; e++) { poff[e] = a; a += (uoff[e + 1] - uoff[e] + 127) / 128 * 128; }
        poff[n_experts] = a;
    }
    for (int i = threadIdx.x; i < rows; i += blockDim.x) pad_src[i] = -1;
    __syncthreads();
    for (int t = threadIdx.x; t < rows / 128; t += blockDim.x) {
        int g = -1;
        for (int e = 0; e < n_experts; e++)
            if (t * 128 >= poff[e] && t * 128 < poff[e + 1]) { g = e; break; }
        tile_group[t] = g;
    }
    // (all pairs in one sweep: an expert after another each waited for memory, 16 experts 9 us)
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        int lo = 0, hi = n_experts;          // the expert whose run holds place i
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (uoff[mid] <= i) lo = mid; else hi = mid;
        }
        const int p = perm[i], at = poff[lo] + i - uoff[lo];
        pad_src[at] = p / top;
        pad_of_pair[p] = at;
    }
}

template <typename T>
__global__ void moe_gather_rows_kernel(const T* __restrict__ x, long long ldx, const int* __restrict__ pad_src, T* __restrict__ xs, int H) {
    ti_pdl_trigger();
    ti_pdl_sync();
    x = ti_dependent(x); pad_src = ti_dependent(pad_src);
    const size_t i = blockIdx.x;
    const int src = pad_src[i];
    if ((H & 7) == 0 && sizeof(T) == 2) {
        const uint4* s4 = src >= 0 ? reinterpret_cast<const uint4*>(x + (size_t)src * ldx) : nullptr;
        uint4* d4 = reinterpret_cast<uint4*>(xs + i * H);
        for (int e = threadIdx.x; e < H / 8; e += blockDim.x) d4[e] = s4 ? s4[e] : make_uint4(0u, 0u, 0u, 0u);
    } else {
        for (int e = threadIdx.x; e < H; e += blockDim.x) xs[i * H + e] = src >= 0 ? x[(size_t)src * ldx + e] : from_f32<T>(0.f);
    }
}

// the same over 16-byte pieces of bfloat16 (ff a multiple of 8)
__global__ void moe_act_pair_vec_kernel(const bf16* __restrict__ gu, bf16* __restrict__ y, int ff8, long long total, float limit, float alpha, float shift) {
    ti_pdl_trigger();
    ti_pdl_sync();
    gu = ti_dependent(gu);
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
        const long long i = idx / ff8;
        const int c = (int)(idx - i * ff8);
        const uint4 g4 = reinterpret_cast<const uint4*>(gu)[i * 2 * ff8 + c], u4 = reinterpret_cast<const uint4*>(gu)[i * 2 * ff8 + ff8 + c];
        const bf16* gp = reinterpret_cast<const bf16*>(&g4);
        const bf16* up = reinterpret_cast<const bf16*>(&u4);
        uint4 o4;
        bf16* op = reinterpret_cast<bf16*>(&o4);
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const float g = fminf(to_f32(gp[e]), limit);
            const float u = fminf(fmaxf(to_f32(up[e]), -limit), limit);
            op[e] = from_f32<bf16>(g * (ti_over(1.0f, 1.0f + expf(-alpha * g))) * (u + shift));
        }
        reinterpret_cast<uint4*>(y)[idx] = o4;
    }
}

// an ungated activation (ti_pointwise) over 16-byte pieces of bfloat16
template <int KIND>
__global__ void pointwise_act_vec_kernel(const bf16* __restrict__ x, bf16* __restrict__ out, long long n8) {
    ti_pdl_trigger();
    ti_pdl_sync();
    x = ti_dependent(x);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
        const uint4 v4 = reinterpret_cast<const uint4*>(x)[i];
        const bf16* vp = reinterpret_cast<const bf16*>(&v4);
        uint4 o4;
        bf16* op = reinterpret_cast<bf16*>(&o4);
#pragma unroll
        for (int e = 0; e < 8; e++) {
            op[e] = from_f32<bf16>(ti_pointwise_bf16(to_f32(vp[e]), KIND));
        }
        reinterpret_cast<uint4*>(out)[i] = o4;
    }
}

// gu[i] = [gate (ff) | up (ff)] -> y[i] = g' sigmoid(alpha g') (u' + shift)
template <typename T>
__global__ void moe_act_pair_kernel(const T* __restrict__ gu, T* __restrict__ y, int ff, long long total, float limit, float alpha, float shift) {
    ti_pdl_trigger();
    ti_pdl_sync();
    gu = ti_dependent(gu);
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
        const long long i = idx / ff;
        const int f = (int)(idx - i * ff);
        const float g = fminf(to_f32(gu[i * 2 * ff + f]), limit);
        const float u = fminf(fmaxf(to_f32(gu[i * 2 * ff + ff + f]), -limit), limit);
        y[idx] = from_f32<T>(g * (ti_over(1.0f, 1.0f + expf(-alpha * g))) * (u + shift));
    }
}

// out[m] = sum_j z[pad_of_pair[m * top + j]] * weight, each term rounded as the scattering product would have stored it
template <typename T>
__global__ void moe_combine_indexed_kernel(const T* __restrict__ z, const int* __restrict__ pad_of_pair, T* __restrict__ out, int H,
                                           int top, float weight) {
    ti_pdl_trigger();
    ti_pdl_sync();
    z = ti_dependent(z); pad_of_pair = ti_dependent(pad_of_pair);
    const size_t m = blockIdx.x;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float s = 0.f;
        for (int j = 0; j < top; j++) {
            const float term = to_f32(from_f32<T>(to_f32(z[(size_t)pad_of_pair[m * top + j] * H + i]) * weight));
            s = j == 0 ? term : s + term;
        }
        out[m * H + i] = from_f32<T>(s);
    }
}

template <typename T, int KIND>
__global__ void pointwise_act_kernel(const T* __restrict__ x, T* __restrict__ out, long long n) {
    ti_pdl_trigger();
    ti_pdl_sync();
    x = ti_dependent(x);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = from_f32<T>(sizeof(T) == 2 ? ti_pointwise_bf16(to_f32(x[i]), KIND) : ti_pointwise(to_f32(x[i]), KIND));
}

}  // namespace

// ids: int32 [M]; table: int32 [vocab, top]; perm: int32 [M * top]; off: int32 [n_experts + 1];
// pair_expert: int32 scratch [M * top].
extern "C" int ti_moe_route_table(const int* ids, const int* table, int vocab, int top, int n_experts, int M, int* perm,
                                  int* off, int* pair_expert, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && top > 0 && n_experts > 0 && vocab > 0, "moe_route_table: bad sizes");
    const size_t smem = (size_t)(3 * n_experts + 1) * sizeof(int);
    TI_REQUIRE(smem <= 48 * 1024, "moe_route_table: %d experts are too many", n_experts);
    TI_CUDA(ti_launch_class<1>(moe_route_table_kernel, dim3(1), dim3(RT_THREADS), smem, stream, ids, table, vocab, top, n_experts, M,
                               perm, off, pair_expert));
    TI_CHECK_LAUNCH("moe_route_table");
    return 0;
}

// Whether a product of rows off the 16-byte boundary runs in staged tiles: with more than 48 places an expert, where the tiles are more
// than seven blocks an SM (a pair's counted twice, it reads two matrices).  us a product, registers / tiles, float32, 16 experts: pairs of 2,047 x 1,023, 40 places an
// expert 503 / 606, 80 942 / 799, 160 1,794 / 1,082, 320 3,462 / 1,829; 1,023 x 391, 80 places 176 / 230, 160 336 / 268; single matrices
// of 2,047 x 1,023, 40 places 265 / 330, 80 495 / 428; four experts of pairs of 2,047 x 1,023, 160 places 441 / 477, 320 860 / 567.
bool staged_tiles(int n_experts, int P, int N, bool pair, int sms) {
    return P > 48LL * n_experts && ((long long)P / GM + n_experts / 2) * ((N + GN - 1) / GN) * (pair ? 2 : 1) > 7LL * sms;
}

// skinny_tiles and staged_tiles above for the tests.
extern "C" int ti_moe_staged_tiles(int n_experts, int P, int N, int pair, int sms) { return staged_tiles(n_experts, P, N, pair != 0, sms); }
extern "C" int ti_moe_skinny_tiles(int n_experts, int P, int N, int K, int pair, int sms) { return skinny_tiles(n_experts, P, N, K, pair != 0, sms); }

// P places.  pair != 0: out[i, 0:N] = act(a_i W[e]^T, a_i W2[e]^T).  Else out[(scatter ? perm[i] : i)] = a_i W[e]^T * scale, or, pair 2
// without W2, the squared ReLU of a_i W[e]^T.
extern "C" int ti_moe_grouped(const void* a, long long lda, const void* W, const void* W2, void* out, long long ldo,
                              const int* perm, const int* off, int n_experts, int P, int N, int K, int top, int gather,
                              int scatter, int pair, float scale, float limit, float alpha, float shift, long long w_estride, int dtype,
                              cudaStream_t stream) {
    if (P == 0) return 0;
    if (w_estride <= 0) w_estride = (long long)N * K;          // elements from one expert's matrix to the next
    TI_REQUIRE(P > 0 && N > 0 && K > 0 && n_experts > 0 && top > 0, "moe_grouped: bad sizes");
    const int relu2 = pair == 2 && !W2;
    if (relu2) pair = 0;
    TI_REQUIRE(!pair || W2, "moe_grouped: the paired form needs a second matrix");
    const bool tensor_cores = dtype == TI_BF16 && K % 8 == 0 && lda % 8 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)W & 15) == 0 &&
                              (!W2 || ((uintptr_t)W2 & 15) == 0);
    timoe::RowsArgs r{a, lda, W, pair ? W2 : nullptr, out, ldo, perm, off, n_experts, N, K, top, gather, scatter, relu2, scale, limit, alpha, shift, w_estride};
    if (tensor_cores) switch (skinny_tiles(n_experts, P, N, K, pair != 0, ti_sm_count())) {
        case 1: return timoe::launch_skinny<1>(r, P, stream);
        case 2: return timoe::launch_skinny<2>(r, P, stream);
        case 4: return timoe::launch_skinny<4>(r, P, stream);
        default: break;
    }
    if (tensor_cores) {
        const bool big = P >= 48 * n_experts;         // groups of 48 places and more on average: tiles of 64
        const int tm = big ? 64 : 32;
        const int tiles = (P + tm - 1) / tm + n_experts;
        const int nblk = (N + TN - 1) / TN;
        TI_REQUIRE(nblk <= 65535, "moe_grouped: %d weight rows are too many for one launch", N);
#define TI_MOE_LAUNCH(PAIR, MI) TI_CUDA(ti_launch(moe_grouped_mma_kernel<PAIR, MI>, dim3(tiles, nblk), dim3(T_THREADS), 0, stream, (const bf16*)a, lda, \
                              (const bf16*)W, (const bf16*)W2, (bf16*)out, ldo, perm, off, n_experts, N, K, top, gather, scatter, relu2, scale, limit, alpha, shift, w_estride))
        if (pair) { if (big) TI_MOE_LAUNCH(true, 2); else TI_MOE_LAUNCH(true, 1); }
        else { if (big) TI_MOE_LAUNCH(false, 2); else TI_MOE_LAUNCH(false, 1); }
#undef TI_MOE_LAUNCH
        TI_CHECK_LAUNCH("moe_grouped");
        return 0;
    }
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        constexpr int V = 16 / sizeof(T);
        const bool vec = K % V == 0 && lda % V == 0 && w_estride % V == 0 && (((uintptr_t)a | (uintptr_t)W | (uintptr_t)r.W2) & 15) == 0;
        if constexpr (sizeof(T) == 4)
            if (vec) return P > ROWS_SMALL_PLACES * n_experts ? timoe::launch_rows<T, V, 4>(r, P, stream) : timoe::launch_rows<T, V, 1>(r, P, stream);
        if (!staged_tiles(n_experts, P, N, pair != 0, ti_sm_count())) return timoe::launch_rows<T, 1, 1>(r, P, stream);
        const dim3 grid((P + GM - 1) / GM + n_experts, (N + GN - 1) / GN);
        TI_REQUIRE(grid.y <= 65535, "moe_grouped: %d weight rows are too many for one launch", N);
#define TI_MOE_LAUNCH(PAIR) TI_CUDA(ti_launch(moe_staged_kernel<T, PAIR>, grid, dim3(G_THREADS), 0, stream, (const T*)a, lda, (const T*)W, (const T*)W2, (T*)out, ldo, \
                                              perm, off, n_experts, N, K, top, gather, scatter, relu2, scale, limit, alpha, shift, w_estride))
        if (pair) TI_MOE_LAUNCH(true); else TI_MOE_LAUNCH(false);
#undef TI_MOE_LAUNCH
        TI_CHECK_LAUNCH("moe_grouped");
        return 0;
    });
}

extern "C" int ti_moe_combine(const void* z, void* out, int M, int H, int top, int dtype, cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && H > 0 && top > 0, "moe_combine: bad sizes");
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        TI_CUDA(ti_launch_class<1>(moe_combine_kernel<T>, dim3(M), dim3(H <= 256 ? 64 : 256), 0, stream, (const T*)z, (T*)out, H, top));
        TI_CHECK_LAUNCH("moe_combine");
        return 0;
    });
}

extern "C" int ti_moe_pad_plan(const int* perm, const int* off, int n_experts, int P, int top, int rows, int* pad_src,
                               int* pad_of_pair, int* tile_group, cudaStream_t stream) {
    if (P == 0) return 0;
    TI_REQUIRE(P > 0 && n_experts > 0 && top > 0 && rows % 128 == 0 && rows >= P + 0, "moe_pad_plan: bad sizes");
    const size_t smem = (size_t)2 * (n_experts + 1) * sizeof(int);
    TI_REQUIRE(smem <= 96 * 1024, "moe_pad_plan: %d experts are too many", n_experts);
    if (smem > 48 * 1024) TI_CUDA(cudaFuncSetAttribute(moe_pad_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    TI_CUDA(ti_launch_class<1>(moe_pad_plan_kernel, dim3(1), dim3(1024), smem, stream, perm, off, n_experts, P, top, rows, pad_src,
                               pad_of_pair, tile_group));
    TI_CHECK_LAUNCH("moe_pad_plan");
    return 0;
}

extern "C" int ti_moe_gather_rows(const void* x, long long ldx, const int* pad_src, void* xs, int rows, int H, int dtype,
                                  cudaStream_t stream) {
    if (rows == 0) return 0;
    TI_REQUIRE(rows > 0 && H > 0, "moe_gather_rows: bad sizes");
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        TI_REQUIRE(sizeof(T) != 2 || (H & 7) || ((((uintptr_t)x | (uintptr_t)xs) & 15) == 0 && ldx % 8 == 0),
                   "moe_gather_rows: rows are not 16-byte aligned");
        TI_CUDA(ti_launch_class<1>(moe_gather_rows_kernel<T>, dim3(rows), dim3(128), 0, stream, (const T*)x, ldx, pad_src, (T*)xs, H));
        TI_CHECK_LAUNCH("moe_gather_rows");
        return 0;
    });
}

extern "C" int ti_moe_act_pair(const void* gu, void* y, long long rows, int ff, float limit, float alpha, float shift, int dtype, cudaStream_t stream) {
    if (rows == 0) return 0;
    TI_REQUIRE(rows > 0 && ff > 0, "moe_act_pair: bad sizes");
    if (dtype == TI_BF16 && ff % 8 == 0 && (((uintptr_t)gu | (uintptr_t)y) & 15) == 0) {
        const long long n = rows * (ff / 8);
        const long long want = (n + 255) / 256;
        TI_CUDA(ti_launch_class<1>(moe_act_pair_vec_kernel, dim3((unsigned)(want < 148 * 16 ? want : 148 * 16)), dim3(256), 0, stream,
                                   (const bf16*)gu, (bf16*)y, ff / 8, n, limit, alpha, shift));
        TI_CHECK_LAUNCH("moe_act_pair");
        return 0;
    }
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        const long long n = rows * ff;
        const long long want = (n + 255) / 256;
        TI_CUDA(ti_launch_class<1>(moe_act_pair_kernel<T>, dim3((unsigned)(want < 148 * 16 ? want : 148 * 16)), dim3(256), 0, stream,
                                   (const T*)gu, (T*)y, ff, n, limit, alpha, shift));
        TI_CHECK_LAUNCH("moe_act_pair");
        return 0;
    });
}

extern "C" int ti_moe_combine_indexed(const void* z, const int* pad_of_pair, void* out, int M, int H, int top, float weight, int dtype,
                                      cudaStream_t stream) {
    if (M == 0) return 0;
    TI_REQUIRE(M > 0 && H > 0 && top > 0, "moe_combine_indexed: bad sizes");
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        TI_CUDA(ti_launch_class<1>(moe_combine_indexed_kernel<T>, dim3(M), dim3(H <= 256 ? 64 : 256), 0, stream, (const T*)z, pad_of_pair,
                                   (T*)out, H, top, weight));
        TI_CHECK_LAUNCH("moe_combine_indexed");
        return 0;
    });
}

// out[i] = act(x[i]) in 32-bit with one rounding; kind 4: squared ReLU, 5: gelu (see ti_pointwise).
extern "C" int ti_pointwise_act(const void* x, void* out, long long n, int kind, int dtype, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(n > 0 && (kind == 4 || kind == 5), "pointwise_act: bad size or unknown activation %d", kind);
    if (dtype == TI_BF16 && n % 8 == 0 && (((uintptr_t)x | (uintptr_t)out) & 15) == 0) {
        const long long n8 = n / 8, want = (n8 + 255) / 256;
        auto kernel = kind == 4 ? pointwise_act_vec_kernel<4> : pointwise_act_vec_kernel<5>;
        TI_CUDA(ti_launch_class<1>(kernel, dim3((unsigned)(want < 148 * 16 ? want : 148 * 16)), dim3(256), 0, stream, (const bf16*)x, (bf16*)out,
                                   n8));
        TI_CHECK_LAUNCH("pointwise_act");
        return 0;
    }
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        const int threads = 256;
        const long long want = (n + threads - 1) / threads;
        const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
        auto kernel = kind == 4 ? pointwise_act_kernel<T, 4> : pointwise_act_kernel<T, 5>;
        TI_CUDA(ti_launch_class<1>(kernel, dim3(blocks), dim3(threads), 0, stream, (const T*)x, (T*)out, n));
        TI_CHECK_LAUNCH("pointwise_act");
        return 0;
    });
}
