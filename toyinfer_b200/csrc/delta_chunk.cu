// The gated delta rule over runs of tokens, in chunks of 32 (the recurrence and its inputs: delta_rule.cu, whose scan goes token
// by token and serves single tokens and sizes that this form does not take).
//
// Within a chunk, with D_ts = g_(s+1) ... g_t (per key channel or per head), G_t = D_t0 from the chunk's start, and S the state
// before it, the writes e_t obey  e_t = beta_t (v_t - (G_t k_t)^T S) - sum_(s<t) beta_t (k_t . D_ts k_s) e_s,  so that with
//     A_ts = beta_t (k_t . D_ts k_s)  (s < t),   T = (I + A)^-1,   P_ts = q_t . D_ts k_s  (s <= t),
//     R = beta v - (beta G k) S,   E = T R;      O = (G q) S + P E;      S <- G_32 S + (D_32,s k_s)^T E
// (Yang, Wang, Zhang, Shen and Kim, "Parallelizing Linear Transformers with the Delta Rule over Sequence Length").  All in
// float32, no further from 64 bits than the scan (operands as silu leaves them, heads of 64 and 128: outputs 0.79 to 1.00 times its
// error, states 0.65 to 0.99; operands of one sign, heads of 64: outputs up to 1.37 times, 1.1e-7 against 0.8e-7).  Decays are
// products of the tokens' own, never exponentials of differences of their sums, so that strong decays lose
// nothing; and R is formed before T, not U - W S with both multiplied by T first, which came out half as far off again as the scan.
//
// delta_chunk_prep_kernel makes T, P and the decayed queries and keys of all chunks at once: a block per (chunk, value head).
// delta_chunk_state_kernel walks a sequence's chunks: a block per (head, 16 columns of S), S kept in registers and, for the two
// products with it, transposed in shared memory; the next chunk's operands come by bulk copies into the parts of one buffer that
// are used up (the first kernel leaves them in the layout that this one reads).
//
// What bounds the second kernel: the shared memory that its multiply-adds read, 128 bytes a cycle whatever lanes share them.
// Hence tiles of 8 x 4 results a thread with the contraction shared out over neighbouring lanes (a thread reads 1.5 bytes a
// multiply-add where tiles of 4 x 4 and 4 x 2 read 2 and 3) and each lane left with its part of the sums after a few exchanges:
// a chunk takes 5,500 cycles, 2,000 of them the products with S.  2,048 tokens of 16 heads of 128 x 128, us, the scan / chunks:
// one decay per head 835 / 239, per key channel 986 / 312; heads of 64 x 64 472 / 174 and 781 / 197; a run of 32 tokens 21 /
// 15 and 24 / 23, of 16 tokens 14 / 15 and 15 / 21 (where the line lies: kernels/recurrent.py).
#include "tma.cuh"

#include <type_traits>

namespace {

constexpr int CH = 32, DC_THREADS = 256, DC_COLS = 16;      // tokens of a chunk; columns of S of a block
constexpr int P_PITCH = CH + 4;

__device__ __forceinline__ float dc_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }
// two multiply-adds in one instruction
__device__ __forceinline__ void fma2(float2& d, const float2& a, const float2& b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// A product of decays that is rounded once: what every multiplication rounds away goes along.  For one decay per head, where
// a factor that is off is off for the whole row: rounded token by token, outputs of heads of 64 came out 6 to 10 % further from 64
// bits than the scan's, whose roundings differ from element to element, and states up to 13 %.
struct Decay {
    float hi = 1.f, lo = 0.f;
    __device__ __forceinline__ void pass(float g) {
        const float p = hi * g;
        lo = fmaf(lo, g, fmaf(hi, g, -p));
        hi = p;
    }
    __device__ __forceinline__ float value() const { return hi + lo; }
};

// A chunk's operands of one head, side by side, as the second kernel has them in shared memory.
template <int D> struct Ops {
    static constexpr int PITCH = D + 4;
    static constexpr int k = 0;                         // [CH][PITCH] beta G k
    static constexpr int q = CH * PITCH;                // [CH][PITCH] G q
    static constexpr int d = 2 * CH * PITCH;            // [CH][PITCH] keys decayed to the chunk's end
    static constexpr int p = 3 * CH * PITCH;            // [CH][P_PITCH]
    static constexpr int t = p + CH * P_PITCH;          // [CH][P_PITCH]
    static constexpr int g = t + CH * P_PITCH;          // [D] G at the chunk's end
    static constexpr int floats = g + D;
};

struct DeltaChunkArgs {
    float* ops;                 // [chunks, heads][Ops<D>::floats]
    float* bv;                  // [chunks, heads, vdim / 16][CH][16] beta v
    const int* cu_new; const int* seq_slot;
    int n_heads, qk_heads, vdim;
    int least;                  // sequences of fewer new tokens are left to the scan
};

// A sequence's chunk c has the number tok0 / 32 + b + c: no two chunks of a step share one.
__device__ __forceinline__ size_t chunk_id(int tok0, int b, int c) { return (size_t)(tok0 / CH + b + c); }

// k, q; per channel: their decays, and the keys and queries as the dots of two blocks of tokens want them
template <int D, bool HEAD> constexpr int prep_smem_floats() {
    return 2 * CH * (D + 4) + (HEAD ? CH * P_PITCH : CH * D + 2 * CH * (D + 4)) + 2 * CH * P_PITCH + 2 * CH;
}

template <typename T, typename L, int D, bool HEAD>
__global__ void __launch_bounds__(DC_THREADS, 4)
delta_chunk_prep_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, long long q_stride, long long k_stride,
                        long long v_stride, const L* __restrict__ decay_logit, long long decay_stride, const float* __restrict__ dt_bias,
                        const float* __restrict__ rate, const T* __restrict__ beta_logit, long long beta_stride, DeltaChunkArgs a) {
    ti_pdl_trigger();
    constexpr int PITCH = D + 4;
    using O = Ops<D>;
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;                              // [CH][PITCH] unit keys
    float* qs = ks + CH * PITCH;                 // [CH][PITCH] unit queries times dim^-1/2
    float* gs = qs + CH * PITCH;                 // per channel: [CH][D] decays; per head: [CH][P_PITCH] the products D_ts
    float* kx = gs + CH * D;                     // (per channel) [CH][PITCH] keys, [CH][PITCH] queries, decayed to a block's border
    float* qx = kx + CH * PITCH;
    float* As = HEAD ? gs + CH * P_PITCH : qx + CH * PITCH;       // [CH][P_PITCH]
    float* Ps = As + CH * P_PITCH;               // [CH][P_PITCH]
    float* bs = Ps + CH * P_PITCH;               // [CH] betas
    float* gh = bs + CH;                         // [CH] decays of the head
    const int b = blockIdx.z, h = blockIdx.y, c = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    ti_pdl_sync();
    q = ti_dependent(q); k = ti_dependent(k); v = ti_dependent(v); decay_logit = ti_dependent(decay_logit); beta_logit = ti_dependent(beta_logit);
    const int tok0 = a.cu_new[b] + c * CH, n = min(CH, a.cu_new[b + 1] - tok0);
    if (n <= 0 || a.cu_new[b + 1] - a.cu_new[b] < a.least) return;
    const int hq = h / (a.n_heads / a.qk_heads), vdim = a.vdim;
    const float rt = rate[h];
    const size_t cid = chunk_id(a.cu_new[b], b, c) * a.n_heads + h;
    float* ops = a.ops + cid * O::floats;
    // rows past the sequence's end are zeros with a decay of one: they write nothing
    for (int t = warp; t < CH; t += 8) {
        float x[D / 32], y[D / 32], sk = 0.f, sq = 0.f;
#pragma unroll
        for (int i = 0; i < D / 32; i++) {
            const int e = lane + 32 * i;
            x[i] = t < n ? to_f32(k[(size_t)(tok0 + t) * k_stride + (size_t)hq * D + e]) : 0.f;
            y[i] = t < n ? to_f32(q[(size_t)(tok0 + t) * q_stride + (size_t)hq * D + e]) : 0.f;
            sk = fmaf(x[i], x[i], sk);
            sq = fmaf(y[i], y[i], sq);
        }
        const float ik = rsqrtf(warp_sum(sk) + 1e-6f), iq = rsqrtf(warp_sum(sq) + 1e-6f) * rsqrtf((float)D);
#pragma unroll
        for (int i = 0; i < D / 32; i++) {
            ks[t * PITCH + lane + 32 * i] = x[i] * ik;
            qs[t * PITCH + lane + 32 * i] = y[i] * iq;
        }
        if constexpr (!HEAD) {
#pragma unroll
            for (int i = 0; i < D / 32; i++) {
                const int e = lane + 32 * i;
                gs[t * D + e] = t < n ? expf(-rt * dc_softplus(to_f32(decay_logit[(size_t)(tok0 + t) * decay_stride + (size_t)h * D + e]) + dt_bias[(size_t)h * D + e])) : 1.f;
            }
        }
    }
    if (tid < CH) {
        bs[tid] = tid < n ? ti_over(1.0f, 1.0f + expf(-to_f32(beta_logit[(size_t)(tok0 + tid) * beta_stride + h]))) : 0.f;
        if constexpr (HEAD) gh[tid] = tid < n ? expf(-rt * dc_softplus(to_f32(decay_logit[(size_t)(tok0 + tid) * decay_stride + h]) + dt_bias[h])) : 1.f;
    }
    __syncthreads();
    for (int i = tid; i < CH * (vdim / 4); i += DC_THREADS) {       // four values of a row: [column group][token][16]
        const int e = i % 4 * 4, t = i / 4 % CH, grp = i / (4 * CH);
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        if (t < n) {
            const T* from = v + (size_t)(tok0 + t) * v_stride + (size_t)h * vdim + grp * DC_COLS + e;
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] = bs[t] * to_f32(from[j]);
        }
        *reinterpret_cast<float4*>(a.bv + cid * CH * vdim + 4 * i) = make_float4(x[0], x[1], x[2], x[3]);
    }
    if constexpr (HEAD) {
        if (warp == 0) {
            // D_ts for s = lane: 1 at t = s, zero before
            Decay d;
            for (int t = 0; t < CH; t++) {
                if (t > lane) d.pass(gh[t]);
                gs[t * P_PITCH + lane] = t >= lane ? d.value() : 0.f;
            }
        }
        __syncthreads();
        // A and P: two rows and two columns of either per thread
        const int t0 = (tid >> 4) * 2, s0 = (tid & 15) * 2;
        // (four sums a product, not one: a chain of all of a head's products was a good part of the error of outputs)
        float2 aa[2][2][2] = {}, pp[2][2][2] = {};
        if (s0 <= t0 + 1) {
#pragma unroll 4
            for (int e = 0; e < D; e += 4) {
                float4 kt[2], qt[2], kk[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    kt[i] = *reinterpret_cast<const float4*>(ks + (t0 + i) * PITCH + e);
                    qt[i] = *reinterpret_cast<const float4*>(qs + (t0 + i) * PITCH + e);
                    kk[i] = *reinterpret_cast<const float4*>(ks + (s0 + i) * PITCH + e);
                }
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        fma2(aa[i][j][0], make_float2(kt[i].x, kt[i].y), make_float2(kk[j].x, kk[j].y));
                        fma2(aa[i][j][1], make_float2(kt[i].z, kt[i].w), make_float2(kk[j].z, kk[j].w));
                        fma2(pp[i][j][0], make_float2(qt[i].x, qt[i].y), make_float2(kk[j].x, kk[j].y));
                        fma2(pp[i][j][1], make_float2(qt[i].z, qt[i].w), make_float2(kk[j].z, kk[j].w));
                    }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int t = t0 + i, s = s0 + j;
                const float d = gs[t * P_PITCH + s];
                const float2 *a2 = aa[i][j], *p2 = pp[i][j];
                As[t * P_PITCH + s] = s < t ? bs[t] * d * ((a2[0].x + a2[0].y) + (a2[1].x + a2[1].y)) : 0.f;
                Ps[t * P_PITCH + s] = s <= t ? d * ((p2[0].x + p2[0].y) + (p2[1].x + p2[1].y)) : 0.f;
            }
        __syncthreads();
    } else {
        for (int i = tid; i < 2 * CH * P_PITCH; i += DC_THREADS) As[i] = 0.f;
        // Pairs (t, s) in different blocks of 16, then of 8 tokens: with the keys of the earlier block decayed to its end and
        // keys and queries of the later one from there on, a pair is a plain dot product.
        for (int half = 16; half >= 8; half >>= 1) {
            for (int i = tid; i < D * (CH / half); i += DC_THREADS) {
                const int e = i % D, blk = i / D, first = blk * half;
                float run = 1.f;
                if (blk & 1) {          // the later block of its pair
                    for (int t = first; t < first + half; t++) {
                        run *= gs[t * D + e];
                        kx[t * PITCH + e] = ks[t * PITCH + e] * run;
                        qx[t * PITCH + e] = qs[t * PITCH + e] * run;
                    }
                } else {
                    for (int t = first + half - 1; t >= first; t--) {
                        kx[t * PITCH + e] = ks[t * PITCH + e] * run;
                        run *= gs[t * D + e];
                    }
                }
            }
            __syncthreads();
            // 256 pairs of a block pair of 16, or 64 in each of the two of 8 (two threads a pair then)
            const bool wide = half == 16;
            const int pair = wide ? tid : tid >> 1, e0 = wide ? 0 : (tid & 1) * 4, step = wide ? 4 : 8;
            const int within = wide ? pair : pair & 63, first = wide ? 0 : (pair >> 6) * 16;
            const int t = first + half + within / half, s = first + within % half;
            float2 xs[2] = {}, ys[2] = {};
#pragma unroll 8
            for (int e = e0; e < D; e += step) {
                const float4 kk = *reinterpret_cast<const float4*>(kx + s * PITCH + e);
                const float4 kt = *reinterpret_cast<const float4*>(kx + t * PITCH + e), qt = *reinterpret_cast<const float4*>(qx + t * PITCH + e);
                fma2(xs[0], make_float2(kt.x, kt.y), make_float2(kk.x, kk.y));
                fma2(xs[1], make_float2(kt.z, kt.w), make_float2(kk.z, kk.w));
                fma2(ys[0], make_float2(qt.x, qt.y), make_float2(kk.x, kk.y));
                fma2(ys[1], make_float2(qt.z, qt.w), make_float2(kk.z, kk.w));
            }
            float x = (xs[0].x + xs[0].y) + (xs[1].x + xs[1].y), y = (ys[0].x + ys[0].y) + (ys[1].x + ys[1].y);
            if (!wide) {
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                y += __shfl_xor_sync(0xffffffffu, y, 1);
            }
            if (wide || (tid & 1) == 0) {
                As[t * P_PITCH + s] = bs[t] * x;
                Ps[t * P_PITCH + s] = y;
            }
            __syncthreads();
        }
        // pairs within a block of 8: a warp per column s, its key decayed step by step (eight steps and less; four columns a warp,
        // at all four distances from their block's end together)
        for (int r = 0; r < 4; r++) {
            const int s = r * 8 + ((r & 1) ? 7 - warp : warp);
            float kw[D / 32];
#pragma unroll
            for (int i = 0; i < D / 32; i++) kw[i] = ks[s * PITCH + lane + 32 * i];
            for (int t = s; t < r * 8 + 8; t++) {
                float x = 0.f, y = 0.f;
#pragma unroll
                for (int i = 0; i < D / 32; i++) {
                    const int e = lane + 32 * i;
                    if (t > s) kw[i] *= gs[t * D + e];
                    x = fmaf(kw[i], ks[t * PITCH + e], x);
                    y = fmaf(kw[i], qs[t * PITCH + e], y);
                }
                // both sums at once: even lanes go on with A's, odd lanes with P's
                const bool odd = lane & 1;
                float z = (odd ? y : x) + __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
#pragma unroll
                for (int m = 2; m < 32; m <<= 1) z += __shfl_xor_sync(0xffffffffu, z, m);
                if (lane == 0 && t > s) As[t * P_PITCH + s] = bs[t] * z;
                if (lane == 1) Ps[t * P_PITCH + s] = z;
            }
        }
        __syncthreads();
    }
    if (warp == 0) {
        // T = (I + A)^-1, row by row: a lane per column
        float tr[CH];
#pragma unroll
        for (int t = 0; t < CH; t++) {
            float x = t == lane ? 1.f : 0.f, y = 0.f;
#pragma unroll
            for (int s = 0; s < t; s += 4) {
                const float4 w = *reinterpret_cast<const float4*>(As + t * P_PITCH + s);        // (zero from the diagonal on)
                x = fmaf(-w.x, tr[s], x);
                if (s + 1 < t) y = fmaf(-w.y, tr[s + 1], y);
                if (s + 2 < t) x = fmaf(-w.z, tr[s + 2], x);
                if (s + 3 < t) y = fmaf(-w.w, tr[s + 3], y);
            }
            tr[t] = x + y;
            ops[O::t + t * P_PITCH + lane] = tr[t];
        }
    } else if (warp == 1) {
        for (int t = 0; t < CH; t++) ops[O::p + t * P_PITCH + lane] = Ps[t * P_PITCH + lane];
    } else {
        // meanwhile: the decayed queries and keys, a channel a thread
        for (int e = tid - 64; e < D; e += DC_THREADS - 64) {
            float run = 1.f;
            Decay all;
#pragma unroll 8
            for (int t = 0; t < CH; t++) {
                if constexpr (HEAD) { all.pass(gh[t]); run = all.value(); } else run *= gs[t * D + e];
                const float key = ks[t * PITCH + e];
                ops[O::q + t * PITCH + e] = qs[t * PITCH + e] * run;
                ops[O::k + t * PITCH + e] = bs[t] * run * key;
                if constexpr (HEAD) ops[O::d + t * PITCH + e] = key * gs[(CH - 1) * P_PITCH + t];
            }
            ops[O::g + e] = run;
            if constexpr (!HEAD) {
                run = 1.f;
#pragma unroll 8
                for (int t = CH - 1; t >= 0; t--) {
                    ops[O::d + t * PITCH + e] = ks[t * PITCH + e] * run;
                    run *= gs[t * D + e];
                }
            }
        }
    }
}

constexpr int R_PITCH = DC_COLS + 4, E_PITCH = DC_COLS + 8;     // (eight, or four, rows side by side fall into different banks)

template <int D> constexpr int state_buf_floats() { return Ops<D>::floats + CH * DC_COLS; }
template <int D> constexpr size_t state_smem_bytes() {
    return (size_t)(state_buf_floats<D>() + DC_COLS * (D + 4) + CH * (R_PITCH + E_PITCH + DC_COLS)) * sizeof(float);
}

// x[0 .. 2 N) summed over the lanes whose numbers differ in bit `bit`: the lane with it set goes on with the upper half.
template <int N>
__device__ __forceinline__ void halve(const float* x, float* out, int bit) {
    const bool up = (threadIdx.x & bit) != 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const float keep = up ? x[N + i] : x[i], give = up ? x[i] : x[N + i];
        out[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
}

template <int D>
__global__ void __launch_bounds__(DC_THREADS, 2)
delta_chunk_state_kernel(DeltaChunkArgs a, float* __restrict__ o, int M, float* __restrict__ state, long long slot_stride, int* status) {
    ti_pdl_trigger();
    using O = Ops<D>;
    constexpr int PITCH = D + 4, BUF = state_buf_floats<D>();
    extern __shared__ __align__(16) float sm[];
    float* St = sm + BUF;                        // [DC_COLS][PITCH]: S transposed
    float* Rs = St + DC_COLS * PITCH;            // [CH][R_PITCH]
    float* Es = Rs + CH * R_PITCH;               // [CH][E_PITCH]
    float* Qs = Es + CH * E_PITCH;               // [CH][DC_COLS]: (G q) S
    __shared__ uint64_t ready[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int groups = a.vdim / DC_COLS, h = blockIdx.x / groups, grp = blockIdx.x - h * groups, col0 = grp * DC_COLS, b = blockIdx.y;
    if (tid == 0) { mbar_init(&ready[0], 1); mbar_init(&ready[1], 1); mbar_fence_init(); }
    ti_pdl_sync();
    if (b == 0)          // rows past the last sequence's are nobody's
        for (int m = a.cu_new[gridDim.y] + (tid >> 4); m < M; m += DC_THREADS / DC_COLS) o[((size_t)m * a.n_heads + h) * a.vdim + col0 + (tid & 15)] = 0.f;
    const int first = a.cu_new[b], n = a.cu_new[b + 1] - first;
    if (n <= 0 || n < a.least) return;
    const int H = a.n_heads, chunks = (n + CH - 1) / CH;
    const size_t id0 = chunk_id(first, b, 0);
    // One buffer, in two parts that come when what they replace is used up: the keys, queries and values of the next chunk once the
    // products with S are made, the rest of a chunk's operands while they are.
    auto copy = [&](uint64_t* bar, float* to, const float* from, int floats) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(to)), "l"(from), "r"(floats * 4), "r"(smem_u32(bar)) : "memory");
    };
    auto fetch_rows = [&](int c) {               // by one thread
        const size_t cid = (id0 + c) * H + h;
        mbar_expect_tx(&ready[0], (O::d + CH * DC_COLS) * 4);
        copy(&ready[0], sm, a.ops + cid * O::floats, O::d);
        copy(&ready[0], sm + O::floats, a.bv + (cid * groups + grp) * (CH * DC_COLS), CH * DC_COLS);
    };
    auto fetch_rest = [&](int c) {
        mbar_expect_tx(&ready[1], (O::floats - O::d) * 4);
        copy(&ready[1], sm + O::d, a.ops + ((id0 + c) * H + h) * O::floats + O::d, O::floats - O::d);
    };
    if (tid == 0) fetch_rows(0);
    // k^T E: tiles of 8 rows and 4 columns of S, a tile's tokens shared out over SG lanes; of its sums this thread keeps four
    // rows (d0 ..) and NC columns (sc ..), its piece of S
    constexpr int SG = D == 128 ? 4 : 8, NC = D == 128 ? 2 : 1;
    const int sg = lane & (SG - 1), tc = (lane / SG) & 3, td = D == 128 ? warp * 2 + (lane >> 4) : warp;
    const int d0 = td * 8 + (lane & (SG / 2) ? 4 : 0);
    const int sc = tc * 4 + (D == 128 ? (lane & 1) * 2 : ((lane & 2) | (lane & 1)));
    float* slot = state + (size_t)a.seq_slot[b] * slot_stride + (size_t)h * D * a.vdim + col0;
    float S[NC][4];
#pragma unroll
    for (int j = 0; j < NC; j++) {
#pragma unroll
        for (int i = 0; i < 4; i++) S[j][i] = slot[(size_t)(d0 + i) * a.vdim + sc + j];
        *reinterpret_cast<float4*>(St + (sc + j) * PITCH + d0) = make_float4(S[j][0], S[j][1], S[j][2], S[j][3]);
    }
    const int kq = lane & 7, ct = lane >> 3;
    bool ok = true;
    __syncthreads();
    const float* buf = sm;
    for (int c = 0; c < chunks; c++) {
        if (!mbar_wait(&ready[0], (uint32_t)(c & 1))) { ti_report(status, TI_STATUS_TMA_WAIT); ok = false; }
        if (!__syncthreads_and(ok)) {            // (given up: not before the copy under way has arrived, or its wait has run out too)
            if (tid == 0) mbar_wait(&ready[0], (uint32_t)(c & 1));
            __syncthreads();
            return;
        }                                        // this chunk's rows and S are there, the last one's operands are used up
        if (tid == 0) fetch_rest(c);
        // the products with S: 64 rows (32 keys, then 32 queries) x 16 columns; a warp has 8 rows, a lane 4 columns and an eighth of D
        float all[32];
        {
            float2 acc[8][4] = {};
            float4 x[2][8], y[2][4];             // the next step's operands are on their way while this one's are multiplied
            auto load = [&](int it) {
                const int e = it * 32 + kq * 4;
#pragma unroll
                for (int j = 0; j < 4; j++) y[it & 1][j] = *reinterpret_cast<const float4*>(St + (ct * 4 + j) * PITCH + e);
#pragma unroll
                for (int i = 0; i < 8; i++) x[it & 1][i] = *reinterpret_cast<const float4*>(buf + (warp * 8 + i) * PITCH + e);      // (queries follow keys)
            };
            load(0);
#pragma unroll
            for (int it = 0; it < D / 32; it++) {
                if (it + 1 < D / 32) load(it + 1);
                asm volatile("" ::: "memory");
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float4 &u = x[it & 1][i], &v = y[it & 1][j];
                        fma2(acc[i][j], make_float2(u.x, u.y), make_float2(v.x, v.y));
                        fma2(acc[i][j], make_float2(u.z, u.w), make_float2(v.z, v.w));
                    }
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) all[i * 4 + j] = acc[i][j].x + acc[i][j].y;
        }
        float half[16], quarter[8], mine[4];
        halve<16>(all, half, 4);
        halve<8>(half, quarter, 2);
        halve<4>(quarter, mine, 1);
        if (warp < 4) {
            const int t = warp * 8 + kq;
            const float4 u = *reinterpret_cast<const float4*>(buf + O::floats + t * DC_COLS + ct * 4);
            *reinterpret_cast<float4*>(Rs + t * R_PITCH + ct * 4) = make_float4(u.x - mine[0], u.y - mine[1], u.z - mine[2], u.w - mine[3]);
        } else {
            *reinterpret_cast<float4*>(Qs + ((warp - 4) * 8 + kq) * DC_COLS + ct * 4) = make_float4(mine[0], mine[1], mine[2], mine[3]);
        }
        if (!mbar_wait(&ready[1], (uint32_t)(c & 1))) { ti_report(status, TI_STATUS_TMA_WAIT); ok = false; }
        if (!__syncthreads_and(ok)) {
            if (tid == 0) mbar_wait(&ready[1], (uint32_t)(c & 1));
            __syncthreads();
            return;
        }                                        // R, (G q) S and the chunk's other operands are there, its rows are used up
        if (tid == 0 && c + 1 < chunks) fetch_rows(c + 1);
        {
            // E = T R: a warp has 4 rows, a lane 4 columns and the tokens kq, kq + 8, ...
            float acc[16] = {};
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const float4 r = *reinterpret_cast<const float4*>(Rs + (kq + 8 * m) * R_PITCH + ct * 4);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (kq + 8 * m > warp * 4 + i) continue;       // (a later token's is not looked at: zero times a NaN is one)
                    const float w = buf[O::t + (warp * 4 + i) * P_PITCH + kq + 8 * m];
                    acc[i * 4] = fmaf(w, r.x, acc[i * 4]);
                    acc[i * 4 + 1] = fmaf(w, r.y, acc[i * 4 + 1]);
                    acc[i * 4 + 2] = fmaf(w, r.z, acc[i * 4 + 2]);
                    acc[i * 4 + 3] = fmaf(w, r.w, acc[i * 4 + 3]);
                }
            }
            float half[8], quarter[4], mine[2];
            halve<8>(acc, half, 4);
            halve<4>(half, quarter, 2);
            halve<2>(quarter, mine, 1);
            *reinterpret_cast<float2*>(Es + (warp * 4 + (kq >> 1)) * E_PITCH + ct * 4 + (kq & 1) * 2) = make_float2(mine[0], mine[1]);
        }
        __syncthreads();
        {
            // S <- G S + k^T E
            float2 acc[4][4] = {};               // [column][pair of rows]
#pragma unroll
            for (int m = 0; m < CH / SG; m++) {
                const int s = sg + SG * m;
                const float4 x = *reinterpret_cast<const float4*>(buf + O::d + s * PITCH + td * 8);
                const float4 y = *reinterpret_cast<const float4*>(buf + O::d + s * PITCH + td * 8 + 4);
                const float4 e = *reinterpret_cast<const float4*>(Es + s * E_PITCH + tc * 4);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float w = j == 0 ? e.x : j == 1 ? e.y : j == 2 ? e.z : e.w;
                    const float2 ww = make_float2(w, w);
                    fma2(acc[j][0], make_float2(x.x, x.y), ww);
                    fma2(acc[j][1], make_float2(x.z, x.w), ww);
                    fma2(acc[j][2], make_float2(y.x, y.y), ww);
                    fma2(acc[j][3], make_float2(y.z, y.w), ww);
                }
            }
            float sums[32], half[16], quarter[8], eighth[4];
#pragma unroll
            for (int r = 0; r < 2; r++)           // rows 0-3 of all columns, then rows 4-7
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    sums[r * 16 + j * 4] = acc[j][2 * r].x;
                    sums[r * 16 + j * 4 + 1] = acc[j][2 * r].y;
                    sums[r * 16 + j * 4 + 2] = acc[j][2 * r + 1].x;
                    sums[r * 16 + j * 4 + 3] = acc[j][2 * r + 1].y;
                }
            halve<16>(sums, half, SG / 2);
            halve<8>(half, quarter, SG / 4);
            const float* left = quarter;
            if constexpr (SG == 8) { halve<4>(quarter, eighth, 1); left = eighth; }
            const float4 g = *reinterpret_cast<const float4*>(buf + O::g + d0);
#pragma unroll
            for (int j = 0; j < NC; j++) {
                S[j][0] = fmaf(S[j][0], g.x, left[j * 4]);
                S[j][1] = fmaf(S[j][1], g.y, left[j * 4 + 1]);
                S[j][2] = fmaf(S[j][2], g.z, left[j * 4 + 2]);
                S[j][3] = fmaf(S[j][3], g.w, left[j * 4 + 3]);
                *reinterpret_cast<float4*>(St + (sc + j) * PITCH + d0) = make_float4(S[j][0], S[j][1], S[j][2], S[j][3]);
            }
        }
        {
            // O = (G q) S + P E, as E = T R
            float acc[16] = {};
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const float4 e = *reinterpret_cast<const float4*>(Es + (kq + 8 * m) * E_PITCH + ct * 4);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (kq + 8 * m > warp * 4 + i) continue;
                    const float w = buf[O::p + (warp * 4 + i) * P_PITCH + kq + 8 * m];
                    acc[i * 4] = fmaf(w, e.x, acc[i * 4]);
                    acc[i * 4 + 1] = fmaf(w, e.y, acc[i * 4 + 1]);
                    acc[i * 4 + 2] = fmaf(w, e.z, acc[i * 4 + 2]);
                    acc[i * 4 + 3] = fmaf(w, e.w, acc[i * 4 + 3]);
                }
            }
            float half[8], quarter[4], mine[2];
            halve<8>(acc, half, 4);
            halve<4>(half, quarter, 2);
            halve<2>(quarter, mine, 1);
            const int r = warp * 4 + (kq >> 1), e = ct * 4 + (kq & 1) * 2, t = c * CH + r;
            const float2 q = *reinterpret_cast<const float2*>(Qs + r * DC_COLS + e);
            if (t < n) *reinterpret_cast<float2*>(o + ((size_t)(first + t) * H + h) * a.vdim + col0 + e) = make_float2(q.x + mine[0], q.y + mine[1]);
        }
    }
#pragma unroll
    for (int j = 0; j < NC; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) slot[(size_t)(d0 + i) * a.vdim + sc + j] = S[j][i];
}

template <typename T, typename L, int D, bool HEAD>
int run_chunks(const void* q, const void* k, const void* v, long long q_stride, long long k_stride, long long v_stride, const void* decay_logit,
               long long decay_stride, const float* dt_bias, const float* rate, const void* beta_logit, long long beta_stride, float* o,
               float* state, long long slot_stride, const DeltaChunkArgs& a, int n_seq, int max_new, int M, int sms, cudaStream_t stream) {
    constexpr size_t prep = prep_smem_floats<D, HEAD>() * sizeof(float), smem = state_smem_bytes<D>();
    constexpr size_t ALONE = 120 * 1024;        // shared memory of a block that shares its SM with no other
    int* status = ti_status_ptr();
    TI_REQUIRE(status != nullptr, "delta_rule: no status word");
    static bool configured = false;
    if (!configured) {
        TI_CUDA(cudaFuncSetAttribute(delta_chunk_prep_kernel<T, L, D, HEAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep));
        TI_CUDA(cudaFuncSetAttribute(delta_chunk_state_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem < ALONE ? ALONE : smem)));
        configured = true;
    }
    TI_CUDA(ti_launch(delta_chunk_prep_kernel<T, L, D, HEAD>, dim3((max_new + CH - 1) / CH, a.n_heads, n_seq), dim3(DC_THREADS), prep, stream,
                      (const T*)q, (const T*)k, (const T*)v, q_stride, k_stride, v_stride, (const L*)decay_logit, decay_stride, dt_bias, rate,
                      (const T*)beta_logit, beta_stride, a));
    TI_CHECK_LAUNCH("delta_rule (chunks)");
    // Blocks that have an SM each must not start two on the SM that the kernel before left first: the walk is a chain, and its
    // time is the slowest block's (64 blocks of 64 x 16: 245 us, spread out 169).  Two blocks of heads of 128 on an SM get 1.35 times one
    // block's work done, so that pays from the third round on: 384 blocks (500, 383 and 200 tokens) 86 us alone, 65 in pairs, but 256
    // (1,348 and 700) 176 and 183, where pairs of two long sequences' blocks end last.
    const long long blocks = (long long)a.n_heads * (a.vdim / DC_COLS) * n_seq;
    const size_t room = blocks <= (D == 128 ? 2 : 1) * (long long)sms && smem < ALONE ? ALONE : smem;
    TI_CUDA(ti_launch(delta_chunk_state_kernel<D>, dim3(a.n_heads * (a.vdim / DC_COLS), n_seq), dim3(DC_THREADS), room, stream, a, o, M, state,
                      slot_stride, status));
    TI_CHECK_LAUNCH("delta_rule (chunk states)");
    return 0;
}

}  // namespace

// Floats of scratch per chunk of 32 tokens and head (chunks of a step: M / 32 + n_seq at most).
extern "C" int ti_delta_chunk_floats(int dim, int vdim) { return (dim == 64 ? Ops<64>::floats : Ops<128>::floats) + CH * vdim; }

// As ti_delta_rule_scan (delta_rule.cu), for dim 64 or 128 and vdim a multiple of 16.  max_new: at least the most new tokens of
// a sequence.  Sequences of fewer than `least` new tokens are passed over (ti_delta_rule_scan takes those up to its `most`).
// sms: the device's SMs.  scratch: float32, 16-byte aligned, (M / 32 + n_seq) * heads * ti_delta_chunk_floats(dim, vdim) values.
extern "C" int ti_delta_rule_chunked(const void* q, const void* k, const void* v, long long q_stride, long long k_stride,
                                     long long v_stride, const void* decay_logit, long long decay_stride, int head_decay,
                                     const float* dt_bias, const float* rate, const void* beta_logit, long long beta_stride, float* o,
                                     float* state, long long slot_stride, float* scratch, const int* cu_new, const int* seq_slot, int n_seq,
                                     int max_new, int M, int n_heads, int qk_heads, int dim, int vdim, int least, int sms, int dtype,
                                     cudaStream_t stream) {
    if (n_seq == 0 || M == 0) return 0;
    TI_REQUIRE(n_seq > 0 && n_seq <= 65535 && M > 0 && max_new > 0 && n_heads > 0 && n_heads <= 65535 && qk_heads > 0 && n_heads % qk_heads == 0 && scratch,
               "delta_rule: bad sizes");
    TI_REQUIRE((dim == 64 || dim == 128) && vdim > 0 && vdim % DC_COLS == 0, "delta_rule: heads of %d x %d are not taken in chunks", dim, vdim);
    TI_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 15) == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0, "delta_rule: scratch and result must be 16-byte aligned");
    DeltaChunkArgs a;
    a.ops = scratch;
    a.bv = scratch + (size_t)(M / CH + n_seq) * n_heads * (dim == 64 ? Ops<64>::floats : Ops<128>::floats);
    a.cu_new = cu_new; a.seq_slot = seq_slot; a.n_heads = n_heads; a.qk_heads = qk_heads; a.vdim = vdim; a.least = least;
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        auto go = [&](auto dc) -> int {
            constexpr int D = decltype(dc)::value;
            if (head_decay)
                return run_chunks<T, T, D, true>(q, k, v, q_stride, k_stride, v_stride, decay_logit, decay_stride, dt_bias, rate, beta_logit, beta_stride, o,
                                                 state, slot_stride, a, n_seq, max_new, M, sms, stream);
            return run_chunks<T, float, D, false>(q, k, v, q_stride, k_stride, v_stride, decay_logit, decay_stride, dt_bias, rate, beta_logit, beta_stride, o,
                                                  state, slot_stride, a, n_seq, max_new, M, sms, stream);
        };
        return dim == 64 ? go(std::integral_constant<int, 64>()) : go(std::integral_constant<int, 128>());
    });
}
