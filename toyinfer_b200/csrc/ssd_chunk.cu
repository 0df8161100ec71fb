// The Mamba-2 recurrence over runs of bfloat16 tokens, in chunks of 128 on the tensor cores (the recurrence and its inputs:
// ssd_scan.cu, whose scan goes token by token and serves single tokens, the 32-bit engine and sizes that this form does not take).
//
// Within a chunk, with a_ts = a_(s+1) ... a_t, A_t = a_t0 from the chunk's start and S (vdim x N) the state before it:
//     y_t = sum_(s<=t) a_ts d_s (C_t . B_s) x_s + A_t S C_t + D x_t,       S <- A_128 S + sum_s a_(128,s) d_s x_s B_s^T
// (the state-space duality of Dao and Gu, "Transformers are SSMs").  Three kernels: what every chunk adds to the state; the
// states before all chunks, one after another; all outputs.
//
// x, B and C are bfloat16 as they come, so C . B is exact products summed in 32 bits.  Everything else stays 32-bit: weights,
// weighted x and states meet their bfloat16 partner as three bfloat16 parts (hi + mid + lo, which hold a float32 up to 2^-27),
// three MMAs a product.  Logarithms of the decays are summed in 64 bits and kept as two floats, so that the difference of two
// of them is as good as the sum of the logarithms between.
//
// What bounds it: the scan's two passes ran 20 multiply-adds a state value and token on the CUDA cores with a quarter of the
// warps an SM holds; here the MMAs (`mma.sync`: the operands are made in registers, weights from accumulators) and the making of
// the weights' parts share the issue slots about evenly (legacy tensor pipe 37 % active in the first and the last kernel).  2,048 tokens, 64
// heads of 64 x 128 in 8 groups, us: the scan in segments 387, this 105; 128 heads 738 / 204; 700 tokens of 64 heads of 32 x 64
// 106 / 27; a run of 96 tokens 28 / 22, of 80 24 / 22, of 64 20 / 22 (hence the scan below 80).  Error against 64 bits: outputs 0.81 to
// 0.98 times the scan's, on operands of one sign too, states 0.61 to 0.94 times.
#include "mma_utils.cuh"

#include <algorithm>
#include <type_traits>

namespace {

constexpr int SC = 128, SSD_THREADS = 256;          // tokens of a chunk

__device__ __forceinline__ float ssd_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

struct SsdArgs {
    const bf16* xbc; long long ld_xbc;
    const bf16* dt; long long ld_dt;
    const float* dt_bias; const float* rate; const float* skip;
    float* state; long long slot_stride;
    float* y;
    const int* cu_new; const int* seq_slot;
    int heads, groups, least;   // sequences of fewer than `least` new tokens are left to the scan
    float* scratch;             // [chunks, heads, vdim, N]: what a chunk adds, then the state before it
    float* decay;               // [chunks, heads]
};

// A sequence's chunk c has the number tok0 / 128 + b + c: no two chunks of a step share one.
__device__ __forceinline__ size_t ssd_chunk_id(int tok0, int b, int c) { return (size_t)(tok0 / SC + b + c); }

// Three bfloat16 parts of two values.
__device__ __forceinline__ void parts2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16(a, b);
    const float ra = a - __uint_as_float(hi << 16), rb = b - __uint_as_float(hi & 0xffff0000u);
    mid = pack_bf16(ra, rb);
    lo = pack_bf16(ra - __uint_as_float(mid << 16), rb - __uint_as_float(mid & 0xffff0000u));
}

// The decays of a chunk's tokens for one head, by one warp: per token its step size d and log2 of A_t as two floats; returns the
// logarithm at the chunk's end.  Tokens past the end: d 0, no decay.
__device__ __forceinline__ double chunk_decays(const SsdArgs& g, int tok0, int n, int h, float* ds, float* lh, float* ll) {
    const int lane = threadIdx.x & 31;
    const float hb = g.dt_bias[h], hr = g.rate[h];
    double own[4], sum = 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = lane * 4 + i;
        const float d = t < n ? ssd_softplus(to_f32(g.dt[(size_t)(tok0 + t) * g.ld_dt + h]) + hb) : 0.f;
        ds[t] = d;
        const float x = hr * d;         // the scan's exponent is this 32-bit product too; beyond 1,024 its decay is zero
        sum -= (double)(x > 1024.f ? 1024.f : x) * 1.4426950408889634;
        own[i] = sum;
    }
    double before = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += up;
    }
    const double all = __shfl_sync(0xffffffffu, before, 31);
    before -= sum;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const double v = before + own[i];
        const float hi = (float)v;
        lh[lane * 4 + i] = hi;
        ll[lane * 4 + i] = (float)(v - (double)hi);
    }
    return all;
}

__device__ __forceinline__ void async16(uint32_t to, const void* from, bool live) {
    const int bytes = live ? 16 : 0;            // the rest is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// acc += A B, rounded to nearest: the tensor core forms the 16 products' sum alone.  (A sum left in its accumulator is truncated
// at its own size with every MMA: over a state of 128 and a chunk of 128 tokens, outputs came out up to 2.6 times as far from 64
// bits as the scan's, 1.9 times on operands that have passed silu.)
__device__ __forceinline__ void mma_add(float (&acc)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float t[4];
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(t[0]), "=f"(t[1]), "=f"(t[2]), "=f"(t[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
#pragma unroll
    for (int e = 0; e < 4; e++) acc[e] += t[e];
}

// Bit 15 (31) of the result: the lower (upper) of two bfloat16 values is not finite.
__device__ __forceinline__ uint32_t not_finite2(uint32_t x) { return (x & 0x7f807f80u) + 0x00800080u; }

// Rows of COLS bfloat16 (64 or 128; or 32 in rows of 64) into the swizzled boxes of mma_utils.cuh, on their way until
// async_wait(); rows past the end are zeros.
template <int COLS>
__device__ __forceinline__ void load_rows(uint32_t to, const bf16* from, long long ld, int n) {
#pragma unroll
    for (int i = threadIdx.x; i < SC * (COLS / 8); i += SSD_THREADS) {
        const int t = i / (COLS / 8), e = (i % (COLS / 8)) * 8;
        async16(to + swizzled_offset<SC>(t, e), from + (size_t)(t < n ? t : 0) * ld + e, t < n);
    }
}

// U = sum_s a_(128,s) d_s x_s B_s^T of a chunk: a block per (chunk, run of heads of one group, sequence); a warp has a run of 16
// values of x and its share of N.  The heads share B; the next one's x is on its way while one is multiplied.
constexpr int STATE_RUN = 4;
template <int N, int V>
__global__ void __launch_bounds__(SSD_THREADS, 2)
ssd_chunk_state_kernel(SsdArgs g, int run) {
    ti_pdl_trigger();
    constexpr int X_BYTES = SC * 64 * 2;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ float ds[STATE_RUN][SC], lh[STATE_RUN][SC], ll[STATE_RUN][SC], w[STATE_RUN][SC];   // smem: B [SC][N], x [SC][V] twice (in rows of 64)
    const int c = blockIdx.x, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ti_pdl_sync();
    g.xbc = ti_dependent(g.xbc); g.dt = ti_dependent(g.dt);
    const int first = g.cu_new[b], tok0 = first + c * SC, n = min(SC, g.cu_new[b + 1] - tok0);
    if (n <= 0 || g.cu_new[b + 1] - first < g.least) return;
    const int inner = g.heads * V, per_group = g.heads / g.groups, runs = (per_group + run - 1) / run;
    const int grp = blockIdx.y / runs, h0 = grp * per_group + (blockIdx.y - grp * runs) * run, h1 = min(h0 + run, (grp + 1) * per_group);
    const bf16* row0 = g.xbc + (size_t)tok0 * g.ld_xbc;
    const uint32_t bs = (uint32_t)__cvta_generic_to_shared(smem), x0 = bs + SC * N * 2;
    load_rows<N>(bs, row0 + inner + grp * N, g.ld_xbc, n);
    load_rows<V>(x0, row0 + h0 * V, g.ld_xbc, n);
    async_commit();
    const size_t id0 = ssd_chunk_id(first, b, c) * g.heads;
    if (warp < h1 - h0) {
        const double all = chunk_decays(g, tok0, n, h0 + warp, ds[warp], lh[warp], ll[warp]);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int t = lane * 4 + i;
            const double x = all - (double)lh[warp][t] - (double)ll[warp][t];
            const float r = (float)x;           // (what the exponent loses here is put back: 2^x = 2^r (1 + ln 2 (x - r)))
            w[warp][t] = ds[warp][t] * (exp2f(r) * fmaf(0.6931472f, (float)(x - (double)r), 1.f));
        }
        if (lane == 0) g.decay[id0 + h0 + warp] = (float)exp2(all);
    }
    constexpr int VT = V / 16, NSPLIT = 8 / VT, NT = N / NSPLIT;        // warps side by side along N; columns of N of a warp
    const int v0 = (warp % VT) * 16, n0 = (warp / VT) * NT;
    for (int h = h0; h < h1; h++) {
        async_wait();
        __syncthreads();                        // this head's x is there; the other place is no longer read
        if (h + 1 < h1) {
            load_rows<V>(x0 + ((h + 1 - h0) & 1) * X_BYTES, row0 + (h + 1) * V, g.ld_xbc, n);
            async_commit();
        }
        const uint32_t xs = x0 + ((h - h0) & 1) * X_BYTES;
        const float* wh = w[h - h0];
        float acc[NT / 8][4] = {}, low[NT / 8][4] = {};     // (the small parts in sums of their own, where truncation costs nothing)
        for (int s0 = 0; s0 < SC; s0 += 16) {
            if (s0 >= n) break;
            // x transposed: matrices (v 0-7, s 0-7), (v 8-15, s 0-7), (v 0-7, s 8-15), (v 8-15, s 8-15)
            uint32_t a[4], hi[4], mid[4], lo[4];
            ldmatrix_x4_trans(a[0], a[1], a[2], a[3], xs + swizzled_offset<SC>(s0 + (lane & 7) + ((lane >> 4) << 3), v0 + (((lane >> 3) & 1) << 3)));
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 ww = *reinterpret_cast<const float2*>(wh + s0 + (i >> 1) * 8 + (lane & 3) * 2);
                parts2(__uint_as_float(a[i] << 16) * ww.x, __uint_as_float(a[i] & 0xffff0000u) * ww.y, hi[i], mid[i], lo[i]);
            }
#pragma unroll
            for (int j = 0; j < NT; j += 16) {
                uint32_t q[4];      // B: matrices (s 0-7, n 0-7), (s 8-15, n 0-7), (s 0-7, n 8-15), (s 8-15, n 8-15), transposed on the way
                ldmatrix_x4_trans(q[0], q[1], q[2], q[3], bs + swizzled_offset<SC>(s0 + (lane & 7) + (((lane >> 3) & 1) << 3), n0 + j + ((lane >> 4) << 3)));
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    mma_bf16(low[j / 8 + u], lo, q[2 * u], q[2 * u + 1]);
                    mma_bf16(low[j / 8 + u], mid, q[2 * u], q[2 * u + 1]);
                    mma_add(acc[j / 8 + u], hi, q[2 * u], q[2 * u + 1]);
                }
            }
        }
        float* to = g.scratch + (id0 + h) * (size_t)(V * N);
#pragma unroll
        for (int j = 0; j < NT / 8; j++) {
            const int v = v0 + (lane >> 2), e = n0 + j * 8 + (lane & 3) * 2;
            *reinterpret_cast<float2*>(to + (size_t)v * N + e) = make_float2(acc[j][0] + low[j][0], acc[j][1] + low[j][1]);
            *reinterpret_cast<float2*>(to + (size_t)(v + 8) * N + e) = make_float2(acc[j][2] + low[j][2], acc[j][3] + low[j][3]);
        }
    }
}

// The state before every chunk, in the place of what the chunk before it added, and the slot's state after the last.
__global__ void ssd_chunk_carry_kernel(SsdArgs g, int per_head) {
    ti_pdl_trigger();
    ti_pdl_sync();
    g.scratch = ti_dependent(g.scratch); g.decay = ti_dependent(g.decay);
    const int b = blockIdx.z, h = blockIdx.y, first = g.cu_new[b], n = g.cu_new[b + 1] - first;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (n <= 0 || n < g.least || i >= per_head) return;
    const int chunks = (n + SC - 1) / SC;
    float* slot = g.state + (size_t)g.seq_slot[b] * g.slot_stride + (size_t)h * per_head + i;
    const size_t id = ssd_chunk_id(first, b, 0) * g.heads + h;
    float* sc = g.scratch + id * per_head + i;
    const size_t step = (size_t)g.heads * per_head;
    float s[4] = {slot[0], slot[1], slot[2], slot[3]};
    constexpr int AHEAD = 8;                    // chunks whose parts are on their way together
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 u[AHEAD];
        float d[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; k++)
            if (c0 + k < chunks) {
                u[k] = *reinterpret_cast<const float4*>(sc + (c0 + k) * step);
                d[k] = g.decay[id + (size_t)(c0 + k) * g.heads];
            }
#pragma unroll
        for (int k = 0; k < AHEAD; k++)
            if (c0 + k < chunks) {
                *reinterpret_cast<float4*>(sc + (c0 + k) * step) = make_float4(s[0], s[1], s[2], s[3]);
                s[0] = fmaf(d[k], s[0], u[k].x);
                s[1] = fmaf(d[k], s[1], u[k].y);
                s[2] = fmaf(d[k], s[2], u[k].z);
                s[3] = fmaf(d[k], s[3], u[k].w);
            }
    }
#pragma unroll
    for (int e = 0; e < 4; e++) slot[e] = s[e];
}

// Outputs: a block per (chunk, run of heads of one group, sequence); a warp has 16 tokens.  C . B of the chunk is formed once and
// stays in registers for all of the block's heads, as does C.
template <int N, int V>
__global__ void __launch_bounds__(SSD_THREADS, 1)
ssd_chunk_out_kernel(SsdArgs g, int run, int M) {
    ti_pdl_trigger();
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int X_BYTES = SC * 64 * 2, PART = V * N * 2, RAW = 3 * PART;
    // S [V][N] in three parts and as it is in memory; x [SC][V] (in rows of 64) of this head and the next.  C and B are where the
    // parts of S are, and behind them, at first.
    unsigned char* st = smem;
    unsigned char* xt = smem + RAW + V * N * 4;
    __shared__ float ds[8][SC], lh[8][SC], ll[8][SC];
    __shared__ int spoilt_from[V];
    const int c = blockIdx.x, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    ti_pdl_sync();
    g.xbc = ti_dependent(g.xbc); g.dt = ti_dependent(g.dt); g.scratch = ti_dependent(g.scratch);
    const int first = g.cu_new[b], tok0 = first + c * SC, n = min(SC, g.cu_new[b + 1] - tok0);
    const int inner = g.heads * V, per_group = g.heads / g.groups, runs = (per_group + run - 1) / run;
    const int grp = blockIdx.y / runs, h0 = grp * per_group + (blockIdx.y - grp * runs) * run, h1 = min(h0 + run, (grp + 1) * per_group);
    if (b == 0 && c == 0) {      // rows past the last sequence's are nobody's (whether or not the first one brings tokens)
        const int cols = (h1 - h0) * V;
        for (int i = tid; i < (M - g.cu_new[gridDim.z]) * cols; i += SSD_THREADS)
            g.y[(size_t)(g.cu_new[gridDim.z] + i / cols) * inner + (size_t)h0 * V + i % cols] = 0.f;
    }
    if (n <= 0 || g.cu_new[b + 1] - first < g.least) return;
    const bf16* row0 = g.xbc + (size_t)tok0 * g.ld_xbc;
    const uint32_t ss = (uint32_t)__cvta_generic_to_shared(st), x0 = (uint32_t)__cvta_generic_to_shared(xt);
    auto fetch = [&](int h) {
        load_rows<V>(x0 + ((h - h0) & 1) * X_BYTES, row0 + h * V, g.ld_xbc, n);
        const float* from = g.scratch + (ssd_chunk_id(first, b, c) * g.heads + h) * (size_t)(V * N);
#pragma unroll
        for (int i = tid; i < V * N / 4; i += SSD_THREADS) async16(ss + RAW + i * 16, from + i * 4, true);
        async_commit();
    };
    const int tile = warp < 4 ? warp : 11 - warp;       // a scheduler's two warps see nine tiles of 16 tokens between them
    const int t0 = tile * 16, ra = lane >> 2, ca = (lane & 3) * 2;
    load_rows<N>(ss, row0 + inner + (g.groups + grp) * N, g.ld_xbc, n);                         // C, and B behind it
    load_rows<N>(ss + SC * N * 2, row0 + inner + grp * N, g.ld_xbc, n);
    async_commit();
    if (warp < h1 - h0) chunk_decays(g, tok0, n, h0 + warp, ds[warp], lh[warp], ll[warp]);      // (runs of up to 8 heads)
    async_wait();
    __syncthreads();
    uint32_t cf[N / 16][4];
#pragma unroll
    for (int k = 0; k < N / 16; k++)
        ldmatrix_x4(cf[k][0], cf[k][1], cf[k][2], cf[k][3], ss + swizzled_offset<SC>(t0 + (lane & 15), k * 16 + ((lane >> 4) << 3)));
    float cb[SC / 8][4] = {};                   // C_t . B_s; a warp's tokens see those up to their own
    const uint32_t bs = ss + SC * N * 2;
#pragma unroll
    for (int j = 0; j < SC / 16; j++) {
        if (j <= tile) {
#pragma unroll
            for (int k = 0; k < N / 16; k++) {
                uint32_t q[4];
                ldmatrix_x4(q[0], q[1], q[2], q[3], bs + swizzled_offset<SC>(j * 16 + (lane & 7) + ((lane >> 4) << 3), k * 16 + (((lane >> 3) & 1) << 3)));
                mma_add(cb[2 * j], cf[k], q[0], q[1]);
                mma_add(cb[2 * j + 1], cf[k], q[2], q[3]);
            }
        }
    }
    __syncthreads();                            // C and B are used up
    fetch(h0);
    for (int h = h0; h < h1; h++) {
        async_wait();
        __syncthreads();                        // this head's x and S are there; the parts of the head before are used up
#pragma unroll
        for (int i = tid; i < V * N / 8; i += SSD_THREADS) {
            const int v = i / (N / 8), e = (i % (N / 8)) * 8;
            const float4 p = *reinterpret_cast<const float4*>(st + RAW + i * 32), q = *reinterpret_cast<const float4*>(st + RAW + i * 32 + 16);
            uint4 hi, mid, lo;
            parts2(p.x, p.y, hi.x, mid.x, lo.x);
            parts2(p.z, p.w, hi.y, mid.y, lo.y);
            parts2(q.x, q.y, hi.z, mid.z, lo.z);
            parts2(q.z, q.w, hi.w, mid.w, lo.w);
            unsigned char* to = st + swizzled_offset<V>(v, e);
            *reinterpret_cast<uint4*>(to) = hi;
            *reinterpret_cast<uint4*>(to + PART) = mid;
            *reinterpret_cast<uint4*>(to + 2 * PART) = lo;
        }
        // Values of x that are not finite: a weight of zero would carry them to tokens before them.  They become zeros, and
        // every output of their channel from their token on becomes a NaN.
        unsigned char* xh = xt + ((h - h0) & 1) * X_BYTES;
        uint32_t any = 0;
#pragma unroll
        for (int i = tid; i < SC * (V / 8); i += SSD_THREADS) {
            const uint4 x = *reinterpret_cast<const uint4*>(xh + swizzled_offset<SC>(i / (V / 8), (i % (V / 8)) * 8));
            any |= not_finite2(x.x) | not_finite2(x.y) | not_finite2(x.z) | not_finite2(x.w);
        }
        const bool bad = __syncthreads_or((any & 0x80008000u) != 0);
        if (bad) {
            if (tid < V) {
                int at = SC;
                for (int t = SC - 1; t >= 0; t--) {
                    unsigned short* x = reinterpret_cast<unsigned short*>(xh + swizzled_offset<SC>(t, tid));
                    if ((*x & 0x7f80u) == 0x7f80u) { at = t; *x = 0; }
                }
                spoilt_from[tid] = at;
            }
            __syncthreads();
        }
        if (h + 1 < h1) fetch(h + 1);           // on its way while this head's outputs are formed
        const uint32_t xs = x0 + ((h - h0) & 1) * X_BYTES;
        const int hh = h - h0;
        // A_t S C_t
        float acc[V / 8][4] = {};
#pragma unroll
        for (int part = 2; part >= 0; part--)
#pragma unroll
            for (int k = 0; k < N / 16; k++)
#pragma unroll
                for (int j = 0; j < V / 16; j++) {
                    uint32_t q[4];
                    ldmatrix_x4(q[0], q[1], q[2], q[3], ss + part * PART + swizzled_offset<V>(j * 16 + (lane & 7) + ((lane >> 4) << 3), k * 16 + (((lane >> 3) & 1) << 3)));
                    if (part > 0) {
                        mma_bf16(acc[2 * j], cf[k], q[0], q[1]);
                        mma_bf16(acc[2 * j + 1], cf[k], q[2], q[3]);
                    } else {
                        mma_add(acc[2 * j], cf[k], q[0], q[1]);
                        mma_add(acc[2 * j + 1], cf[k], q[2], q[3]);
                    }
                }
        const float la = lh[hh][t0 + ra], la2 = ll[hh][t0 + ra], lb = lh[hh][t0 + ra + 8], lb2 = ll[hh][t0 + ra + 8];
        const float ea = exp2f(la + la2), eb = exp2f(lb + lb2);
#pragma unroll
        for (int j = 0; j < V / 8; j++) { acc[j][0] *= ea; acc[j][1] *= ea; acc[j][2] *= eb; acc[j][3] *= eb; }
        // the chunk's own tokens: weights from C . B (their small parts in sums of their own, as above)
        float low[V / 8][4] = {};
#pragma unroll
        for (int j = 0; j < SC / 16; j++) {
            if (j <= tile) {
                uint32_t hi[4], mid[4], lo[4];
#pragma unroll
                for (int u = 0; u < 2; u++) {   // columns s of this tile: 8 u + ca, + 1
                    const int s = j * 16 + u * 8 + ca;
                    float p[4];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const float lsh = lh[hh][s + e], lsl = ll[hh][s + e], d = ds[hh][s + e];
                        const float wa = exp2f((la - lsh) + (la2 - lsl)) * d, wb = exp2f((lb - lsh) + (lb2 - lsl)) * d;
                        p[e] = s + e <= t0 + ra ? cb[2 * j + u][e] * wa : 0.f;
                        p[2 + e] = s + e <= t0 + ra + 8 ? cb[2 * j + u][2 + e] * wb : 0.f;
                    }
                    parts2(p[0], p[1], hi[2 * u], mid[2 * u], lo[2 * u]);
                    parts2(p[2], p[3], hi[2 * u + 1], mid[2 * u + 1], lo[2 * u + 1]);
                }
#pragma unroll
                for (int v = 0; v < V / 16; v++) {
                    uint32_t q[4];
                    ldmatrix_x4_trans(q[0], q[1], q[2], q[3], xs + swizzled_offset<SC>(j * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), v * 16 + ((lane >> 4) << 3)));
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        mma_bf16(low[2 * v + u], lo, q[2 * u], q[2 * u + 1]);
                        mma_bf16(low[2 * v + u], mid, q[2 * u], q[2 * u + 1]);
                        mma_add(acc[2 * v + u], hi, q[2 * u], q[2 * u + 1]);
                    }
                }
            }
        }
        if (bad)
#pragma unroll
            for (int j = 0; j < V / 8; j++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (t0 + ra + (e >> 1) * 8 >= spoilt_from[j * 8 + ca + (e & 1)]) acc[j][e] = __int_as_float(0x7fffffff);
        const float skip = g.skip ? g.skip[h] : 0.f;
        float* yo = g.y + (size_t)(tok0 + t0) * inner + (size_t)h * V;
#pragma unroll
        for (int j = 0; j < V / 8; j++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int t = ra + 8 * r, v = j * 8 + ca;
                if (t0 + t < n) {
                    const uint32_t x = *reinterpret_cast<const uint32_t*>(xh + swizzled_offset<SC>(t0 + t, v));
                    *reinterpret_cast<float2*>(yo + (size_t)t * inner + v) =
                        make_float2(fmaf(skip, __uint_as_float(x << 16), acc[j][2 * r] + low[j][2 * r]),
                                    fmaf(skip, __uint_as_float(x & 0xffff0000u), acc[j][2 * r + 1] + low[j][2 * r + 1]));
                }
            }
    }
}

template <int N, int V>
int run_ssd_chunks(const SsdArgs& g, int n_seq, int max_new, int M, int sms, cudaStream_t stream) {
    constexpr size_t state_smem = (size_t)SC * N * 2 + 2 * SC * 64 * 2, out_smem = std::max<size_t>((size_t)SC * N * 4, (size_t)2 * SC * 64 * 2 + V * N * 10);
    static bool configured = false;
    if (!configured) {
        TI_CUDA(cudaFuncSetAttribute(ssd_chunk_state_kernel<N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)state_smem));
        TI_CUDA(cudaFuncSetAttribute(ssd_chunk_out_kernel<N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem));
        configured = true;
    }
    const int chunks = (max_new + SC - 1) / SC;
    const int per_group = g.heads / g.groups;
    // chunks that there can be: sequences that bring fewer tokens than the longest leave blocks of the grid without work
    const long long live = std::min((long long)chunks * n_seq, (long long)M / SC + std::min(n_seq, g.least > 0 ? M / g.least : n_seq)) * g.groups;
    int state_run = std::min(STATE_RUN, per_group);       // (heads share B, as long as most SMs have two blocks left)
    while (state_run > 1 && live * ((per_group + state_run - 1) / state_run) < 4 * sms / 3) state_run /= 2;
    TI_CUDA(ti_launch(ssd_chunk_state_kernel<N, V>, dim3(chunks, g.groups * ((per_group + state_run - 1) / state_run), n_seq), dim3(SSD_THREADS),
                      state_smem, stream, g, state_run));
    TI_CHECK_LAUNCH("ssd_scan (chunks' parts)");
    TI_CUDA(ti_launch(ssd_chunk_carry_kernel, dim3((V * N / 4 + 255) / 256, g.heads, n_seq), dim3(256), 0, stream, g, V * N));
    TI_CHECK_LAUNCH("ssd_scan (chunks' states)");
    // heads of a block, up to the eight that fit: forming C . B costs a block about as much as a head and a third does, and
    // blocks go round by round, one on an SM
    int run = 1;
    double best = 0.0;
    for (int r = 1; r <= std::min(8, per_group); r++) {
        const long long blocks = live * ((per_group + r - 1) / r);
        const double cost = (double)((blocks + sms - 1) / sms) * (1.3 + r);
        if (r == 1 || cost < best) { best = cost; run = r; }
    }
    TI_CUDA(ti_launch(ssd_chunk_out_kernel<N, V>, dim3(chunks, g.groups * ((per_group + run - 1) / run), n_seq), dim3(SSD_THREADS), out_smem, stream, g, run, M));
    TI_CHECK_LAUNCH("ssd_scan (chunks' outputs)");
    return 0;
}

}  // namespace

// As ti_ssd_scan (ssd_scan.cu), for bfloat16 tokens, N 64 or 128 and vdim 32 or 64; rows of xbc on 16-byte boundaries.  max_new:
// at least the most new tokens of a sequence.  Sequences of fewer than `least` are passed over (ti_ssd_scan takes those up to its
// `most`).  sms: the device's SMs.  scratch: float32, 16-byte aligned, (M / 128 + n_seq) * heads * (vdim * N + 1) values.
extern "C" int ti_ssd_chunked(const void* xbc, long long ld_xbc, const void* dt_raw, long long ld_dt, const float* dt_bias,
                              const float* rate, const float* skip, float* state, long long slot_stride, float* y, const int* cu_new,
                              const int* seq_slot, int n_seq, int max_new, int M, int heads, int groups, int N, int vdim, int least, int sms, float* scratch,
                              cudaStream_t stream) {
    if (n_seq == 0 || M == 0) return 0;
    TI_REQUIRE(n_seq > 0 && n_seq <= 65535 && M > 0 && max_new > 0 && heads > 0 && heads <= 65535 && groups > 0 && heads % groups == 0 && scratch,
               "ssd_scan: bad sizes");
    TI_REQUIRE((N == 64 || N == 128) && (vdim == 32 || vdim == 64), "ssd_scan: states of %d x %d are not taken in chunks", vdim, N);
    TI_REQUIRE(ld_xbc % 8 == 0 && (reinterpret_cast<uintptr_t>(xbc) & 15) == 0 && (reinterpret_cast<uintptr_t>(scratch) & 15) == 0 &&
               (reinterpret_cast<uintptr_t>(y) & 15) == 0, "ssd_scan: rows must start on 16-byte boundaries");
    SsdArgs g{(const bf16*)xbc, ld_xbc, (const bf16*)dt_raw, ld_dt, dt_bias, rate, skip, state, slot_stride, y, cu_new, seq_slot, heads, groups, least,
              scratch, scratch + (size_t)(M / SC + n_seq) * heads * vdim * N};
    if (N == 64) return vdim == 32 ? run_ssd_chunks<64, 32>(g, n_seq, max_new, M, sms, stream) : run_ssd_chunks<64, 64>(g, n_seq, max_new, M, sms, stream);
    return vdim == 32 ? run_ssd_chunks<128, 32>(g, n_seq, max_new, M, sms, stream) : run_ssd_chunks<128, 64>(g, n_seq, max_new, M, sms, stream);
}
