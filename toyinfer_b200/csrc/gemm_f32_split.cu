// out[M, N] = x[M, K] * W[N, K]^T in float32 on the tensor cores: the 32-bit engine's product of more than 16 tokens.
//
// A float32 value is the sum of three bfloat16 values, up to 2^-27 of itself: hi = bf16(v), mid = bf16(v - hi),
// lo = bf16(v - hi - mid) (both differences are exact).  Six of the nine products of two such sums are formed on the tensor
// cores (Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision
// Computations"); the three left out are below 2^-26 of the product.
//
// The tensor core's accumulator truncates: a contraction of 2,560 left in it comes out 2.3e-6 too small (9,728: 9.4e-6),
// where FFMA with partial sums of 128 is 1.1e-7 off (1.8e-7).  So nothing stays in it for longer than 32 steps of the
// contraction: a chunk of 32 is multiplied into one of two accumulators (the five small products first, then hi * hi, whose two
// MMAs are the only ones that truncate at the size of the result), and the epilogue warps add it to sums in registers,
// rounded to nearest, while the next chunk goes into the other.
// What the two large MMAs of a chunk cut off is left: results come out 4 to 5e-8 too small.  Error against 64 bits (2-norm) at
// contractions of 64 / 2,560 / 9,728, this and FFMA tiles: operands of mixed signs 0.6, 1.1, 1.4e-7 and 1.4, 2.2, 2.6e-7; of one sign,
// where every cut errs the same way, 0.6, 0.8, 1.0e-7 and 1.2, 0.7, 1.2e-7.  The few-row kernel, whose 9 to 16 tokens of a large
// matrix come here, is at 1.0 to 3.2e-7 on mixed signs (this 0.9 to 1.5e-7) and at 0.3 to 0.5e-7 on one sign (0.7 to 1.1e-7).
//
// What bounds it: six bfloat16 MMAs per product (a sixth of the bfloat16 rate); beside them, per chunk of a tile of 256 x 256
// on a pair of SMs (1,536 cycles of MMA), a block's issue slots are about a quarter splitting its 256 rows of operands and a
// fifth adding up accumulators, and its shared memory is busy moving operands in, parts out and both to the tensor cores (a
// block on its own would have to move half as much again: hence the pair).  Splitting in the kernel keeps the operands' reads
// at 4 bytes a value and needs no second copy of the weights.
// Roles of a block's 20 warps: 0-7 epilogue (128 sums a thread), 8-15 split operands, 16 of rank 0 issues the MMAs, 17 TMA.
//
// Weights are the MMA's 256 rows and tokens its columns (BN of 64, 128 or 256), so that the result of a few tokens wastes
// little.  The chunks of all tiles are dealt out to the pairs in equal runs; where a run ends inside a tile the pieces go to a
// workspace and a second kernel adds them in order.
//
// Infinite or not-a-number results (an operand that is, or whose bfloat16 part is, infinite) are formed again by FFMA from the
// operands themselves, so that they are what the CUDA-core kernel's sum gives.
#include "tcgen05.cuh"

#include <algorithm>

namespace {

constexpr int SPLIT_THREADS = 640, CHUNK = 32, WROWS = 128;      // contraction steps per chunk; weight rows of a block
constexpr int LAUNCH_REGS = 96, EPI_REGS = 160, CONV_REGS = 64, CTRL_REGS = 32;      // per thread: at launch, and after the split
static_assert(256 * EPI_REGS + 256 * CONV_REGS + 128 * CTRL_REGS <= SPLIT_THREADS * LAUNCH_REGS, "the split must fit what the block was launched with");

struct SplitArgs {
    const float* x; const float* w; float* out;
    int M, N, K;
    long long ldx, ldw, ldo;
    int units;                  // pairs of blocks
    float* workspace;
    int gated; float gate_limit;    // as in gemm_tcgen05.cuh: 1 to 3 gated pairs of weight rows, 4 and 5 pointwise
};

// A ring of chunks as they are in memory, filled by TMA, and a ring of chunks split into their parts.
template <int BN> constexpr int split_stage_bytes() { return (WROWS + BN / 2) * CHUNK * 2 * 3; }
template <int BN> constexpr int raw_stage_bytes() { return (WROWS + BN / 2) * CHUNK * 4; }
constexpr int PARTS = 3;
template <int BN> constexpr int raw_stages() { return (222 * 1024 - PARTS * split_stage_bytes<BN>()) / raw_stage_bytes<BN>(); }

__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
    for (uint32_t i = 0; i < TI_SPIN_LIMIT; i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// Descriptor of a K-major tile with rows of 64 bytes (32 bfloat16) under the 64-byte swizzle: groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

struct F8 { float v[8]; };

// Eight values as three runs of eight bfloat16.
__device__ __forceinline__ void split8(const F8& f, uint4& hi, uint4& mid, uint4& lo) {
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = f.v[2 * i], b = f.v[2 * i + 1];
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
        h[i] = *reinterpret_cast<const uint32_t*>(&h2);
        const float ra = a - __uint_as_float(h[i] << 16), rb = b - __uint_as_float(h[i] & 0xffff0000u);
        const __nv_bfloat162 m2 = __floats2bfloat162_rn(ra, rb);
        m[i] = *reinterpret_cast<const uint32_t*>(&m2);
        const __nv_bfloat162 l2 = __floats2bfloat162_rn(ra - __uint_as_float(m[i] << 16), rb - __uint_as_float(m[i] & 0xffff0000u));
        l[i] = *reinterpret_cast<const uint32_t*>(&l2);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    mid = make_uint4(m[0], m[1], m[2], m[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Whether a row holds a NaN; and a product of two rows by FFMA, which ends as soon as a sum has become one.  By a whole warp.
__device__ __forceinline__ bool row_has_nan(const float* a, int K) {
    for (int k0 = 0; k0 < K; k0 += 128) {
        bool any = false;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = k0 + u * 32 + (threadIdx.x & 31);
            any |= k < K && isnan(a[k < K ? k : 0]);
        }
        if (__any_sync(0xffffffffu, any)) return true;
    }
    return false;
}
__device__ __forceinline__ float plain_dot(const float* a, const float* b, int K) {
    float s = 0.f;
    for (int k0 = 0; k0 < K; k0 += 128) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = k0 + u * 32 + (threadIdx.x & 31);
            if (k < K) s = fmaf(a[k], b[k], s);
        }
        if (__any_sync(0xffffffffu, isnan(s))) return __int_as_float(0x7fffffff);
    }
    return warp_sum(s);
}

// Results of a warp (lane: weight row n; bit e of `bad`: token m0 + e) that are not finite.  Where an operand's row holds a NaN,
// so is the result, and the row is looked at once for all of them; the others (infinities, and values that only their
// bfloat16 parts make infinite) are formed again, a warp a result.  (A thread per result, every step of the contraction one
// after another, took 4.4 ms where a product of 256 x 1,024 x 1,024 of NaN takes 25 us otherwise.)  Called by whole warps.
__device__ __noinline__ void redo16(const SplitArgs& g, int m0, int n, unsigned bad, float* v) {
    const int lane = threadIdx.x & 31;
    const float nan = __int_as_float(0x7fffffff);
    for (int e = 0; e < 16; e++) {
        const unsigned who = __ballot_sync(0xffffffffu, bad >> e & 1u);
        if (__popc(who) < 2 || !row_has_nan(g.x + (size_t)(m0 + e) * g.ldx, g.K)) continue;
        if (bad >> e & 1u) v[e] = nan;
        bad &= ~(1u << e);
    }
    for (int l = 0; l < 32; l++) {
        unsigned left = __shfl_sync(0xffffffffu, bad, l);
        if (left == 0) continue;
        const float* w = g.w + (size_t)(n - lane + l) * g.ldw;
        const bool all = __popc(left) >= 2 && row_has_nan(w, g.K);
        for (; left != 0; left &= left - 1) {
            const int e = __ffs(left) - 1;
            const float s = all ? nan : plain_dot(g.x + (size_t)(m0 + e) * g.ldx, w, g.K);
            if (lane == l) v[e] = s;
        }
    }
}

// Stores sixteen results of a thread: tokens m0 .. m0 + 15 of weight row n (lanes are consecutive n).
__device__ __forceinline__ void put16(const SplitArgs& g, int m0, int n, float (&v)[16]) {
    const int live = min(16, g.M - m0);
    if (g.gated >= 1 && g.gated <= 3) {
        float* o = g.out + (size_t)m0 * g.ldo + (n >> 1);
        const bool mine = n < g.N && (n & 1) == 0;
#pragma unroll
        for (int e = 0; e < 16; e++) {
            const float other = __shfl_xor_sync(0xffffffffu, v[e], 1);
            // (the compiler's division: the branchless one made this code long enough to cost the ungated products of a few tokens 0.6 us
            // each, a float32 delta-rule step of 40 sequences 56.6 -> 58.1, and the gated ones gained nothing by it)
            if (mine && e < live) o[(size_t)e * g.ldo] = ti_gate_pair<false>(v[e], other, g.gated, g.gate_limit);
        }
        return;
    }
    if (n >= g.N) return;
    float* o = g.out + (size_t)m0 * g.ldo + n;
    if (g.gated >= 4) {
#pragma unroll
        for (int e = 0; e < 16; e++) v[e] = ti_pointwise(v[e], g.gated);
    }
#pragma unroll
    for (int e = 0; e < 16; e++)
        if (e < live) o[(size_t)e * g.ldo] = v[e];
}

// The same where one of a warp's results is not finite.
__device__ __noinline__ void store16_again(const SplitArgs& g, int m0, int n, float4 a, float4 b, float4 c, float4 d) {
    float v[16] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
    unsigned bad = 0;
#pragma unroll
    for (int e = 0; e < 16; e++)
        if (m0 + e < g.M && n < g.N && !isfinite(v[e])) bad |= 1u << e;
    redo16(g, m0, n, bad, v);
    put16(g, m0, n, v);
}

// All lanes of a warp call it together.  One copy of the code for all columns of a tile: written out for each of 128 columns it was
// fetched from L2 instruction by instruction, 40 us a tile.
__device__ __noinline__ void store16(const SplitArgs& g, int m0, int n, float4 a, float4 b, float4 c, float4 d) {
    float v[16] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
    float probe = 0.f;                  // not a number as soon as one of them is not finite
#pragma unroll
    for (int e = 0; e < 16; e++) probe = fmaf(v[e], 0.f, probe);
    if (__any_sync(0xffffffffu, probe != 0.f)) store16_again(g, m0, n, a, b, c, d);
    else put16(g, m0, n, v);
}

__host__ __device__ __forceinline__ long long unit_begin(long long total, int units, int u) { return total * u / units; }

// The pieces of work of a unit: runs of chunks inside one tile, in order.
struct SplitPiece { int tile, c0, c1, place; bool whole; };
struct SplitWalk {
    long long at, end, begin;
    int nk;
    __device__ SplitWalk(long long total, int nk_, int unit, int units) : nk(nk_) {
        begin = at = unit_begin(total, units, unit);
        end = unit_begin(total, units, unit + 1);
    }
    __device__ bool next(SplitPiece& p) {
        if (at >= end) return false;
        p.tile = (int)(at / nk);
        p.c0 = (int)(at - (long long)p.tile * nk);
        p.c1 = (int)min((long long)nk, p.c0 + (end - at));
        p.whole = p.c0 == 0 && p.c1 == nk;
        p.place = at == begin ? 0 : 1;
        at += p.c1 - p.c0;
        return true;
    }
};

template <int BN>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const SplitArgs g, int* status) {
    ti_pdl_trigger();
    constexpr int STAGES = PARTS, STAGE = split_stage_bytes<BN>(), RAW = raw_stage_bytes<BN>(), RAWS = raw_stages<BN>();
    constexpr int A_PART = WROWS * CHUNK * 2, B_PART = BN / 2 * CHUNK * 2;
    constexpr int ROWS = WROWS + BN / 2;                    // operand rows that this block splits
    constexpr int ITEMS = (ROWS * 4 + 127) / 128;           // runs of 8 values per splitting thread and chunk
    constexpr uint32_t ACC_COLS = BN, TMEM_COLS = 2 * ACC_COLS;
    constexpr int COLS = BN / 2;                            // columns of an epilogue warp: the two groups of four share a row's columns
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* raw = smem + STAGES * STAGE;
    __shared__ uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], raw_full[RAWS], raw_empty[RAWS];
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_rank(), unit = blockIdx.x >> 1;
    const int tiles_m = (g.M + BN - 1) / BN, tiles_n = (g.N + 2 * WROWS - 1) / (2 * WROWS);
    const int nk = (g.K + CHUNK - 1) / CHUNK;
    const long long total = (long long)tiles_m * tiles_n * nk;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(&full[s], 8); mbar_init(&empty[s], 1); }        // one group of splitting warps of either block
        for (int b = 0; b < 2; b++) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }    // epilogue warps of both blocks
        for (int s = 0; s < RAWS; s++) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 4); }  // one group of splitting warps
        mbar_fence_init();
    }
    __syncthreads();
    cluster_sync_all();             // the other block's barriers exist before anything arrives on them
    if (warp == 16) {
        __syncwarp();
        tmem_alloc_pair(&tmem_slot, TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    const int warp_u = warp_uniform();
    if (warp_u < 8) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPI_REGS));
        ti_pdl_sync();              // (a kernel before may still read what this one's results replace)
        const int q = warp_u & 3, half = warp_u >> 2;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        int it = 0;
        bool ok = true;
        SplitWalk walk(total, nk, unit, g.units);
        SplitPiece p;
        while (ok && walk.next(p)) {
            float sum[COLS];
#pragma unroll
            for (int c = 0; c < COLS; c++) sum[c] = 0.f;
            for (int kc = p.c0; kc < p.c1; kc++, it++) {
                const int buf = it & 1;
                if (!mbar_wait(&acc_full[buf], (uint32_t)((it >> 1) & 1))) { ti_report(status, TI_STATUS_MMA_WAIT); ok = false; }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr = tmem + buf * ACC_COLS + half * COLS + lanes;
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    float r[16];
                    tmem_ld16(taddr + c, r);
#pragma unroll
                    for (int e = 0; e < 16; e++) sum[c + e] += r[e];
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[buf], 0));
            }
            if (!ok) break;
            const int tn = p.tile / tiles_m, tm = p.tile - tn * tiles_m;
            const int n = tn * 2 * WROWS + rank * WROWS + q * 32 + lane, m0 = tm * BN + half * COLS;
            if (p.whole) {
#pragma unroll
                for (int c = 0; c < COLS; c += 16)
                    if (m0 + c < g.M)
                        store16(g, m0 + c, n, make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]), make_float4(sum[c + 4], sum[c + 5], sum[c + 6], sum[c + 7]),
                                make_float4(sum[c + 8], sum[c + 9], sum[c + 10], sum[c + 11]), make_float4(sum[c + 12], sum[c + 13], sum[c + 14], sum[c + 15]));
            } else {
                float* ws = g.workspace + (((size_t)unit * 2 + p.place) * 2 + rank) * (size_t)(BN * WROWS) + (size_t)(half * COLS) * WROWS + q * 32 + lane;
#pragma unroll
                for (int c = 0; c < COLS; c++) ws[(size_t)c * WROWS] = sum[c];
            }
        }
    } else if (warp_u < 16) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CONV_REGS));
        // two groups of four warps take the chunks in turn, so that one's waits and fences pass under the other's arithmetic
        const int t = threadIdx.x & 127, turn = (warp_u >> 2) & 1;
        const int grp = t & 3;                                  // this thread's run of 8 values within a row's 32
        const long long chunks = unit_begin(total, g.units, unit + 1) - unit_begin(total, g.units, unit);
        bool ok = true;
        for (int it = turn; it < chunks; it += 2) {
            const int s = it % STAGES, rs = it % RAWS;
            if (!mbar_wait(&raw_full[rs], (uint32_t)((it / RAWS) & 1))) { ti_report(status, TI_STATUS_TMA_WAIT); ok = false; }
            if (ok && !mbar_wait(&empty[s], (uint32_t)(((it / STAGES) & 1) ^ 1))) { ti_report(status, TI_STATUS_PIPE_WAIT); ok = false; }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            unsigned char* st = smem + (size_t)s * STAGE;
            const unsigned char* from = raw + (size_t)rs * RAW;
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const int row = (t >> 2) + 32 * i;
                if (32 * i + 32 > ROWS && row >= ROWS) continue;
                // a row's 128 bytes lie in pieces of 16 under the 128-byte swizzle
                const float4 u = *reinterpret_cast<const float4*>(from + row * 128 + (((2 * grp) ^ (row & 7)) << 4));
                const float4 v = *reinterpret_cast<const float4*>(from + row * 128 + (((2 * grp + 1) ^ (row & 7)) << 4));
                const F8 f = {{u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w}};
                uint4 hi, mid, lo;
                split8(f, hi, mid, lo);
                const bool is_w = i < WROWS / 32;
                const int r = is_w ? row : row - WROWS;
                unsigned char* base = st + (is_w ? 0 : 3 * A_PART) + r * 64 + ((grp ^ ((r >> 1) & 3)) << 4);
                const int part = is_w ? A_PART : B_PART;
                *reinterpret_cast<uint4*>(base) = hi;
                *reinterpret_cast<uint4*>(base + part) = mid;
                *reinterpret_cast<uint4*>(base + 2 * part) = lo;
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&raw_empty[rs]);
                mbar_arrive_cluster(cluster_addr(&full[s], 0));
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CTRL_REGS));
        const long long chunks = unit_begin(total, g.units, unit + 1) - unit_begin(total, g.units, unit);
        if (warp_u == 16 && rank == 0 && elect_one()) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            int it = 0;
            for (; it < chunks; it++) {
                const int s = it % STAGES, buf = it & 1;
                if (!mbar_wait_cluster(&acc_empty[buf], (uint32_t)(((it >> 1) & 1) ^ 1))) { ti_report(status, TI_STATUS_PIPE_WAIT); break; }
                if (!mbar_wait_cluster(&full[s], (uint32_t)((it / STAGES) & 1))) { ti_report(status, TI_STATUS_PIPE_WAIT); break; }
                fence_proxy_async();
                tc_fence_after();
                const uint32_t sa = smem_u32(smem + (size_t)s * STAGE);
                const uint64_t da = smem_desc_sw64(sa), db = smem_desc_sw64(sa + 3 * A_PART);
                const uint32_t acc = tmem + buf * ACC_COLS;
                // the products of the parts, smallest first; the last pair of MMAs is hi * hi
                constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                for (int j = 0; j < 6; j++)
#pragma unroll
                    for (int k = 0; k < CHUNK / 16; k++)
                        tc_mma_bf16_pair(acc, da + (uint64_t)((PA[j] * A_PART >> 4) + k * 2), db + (uint64_t)((PB[j] * B_PART >> 4) + k * 2), idesc,
                                         (j > 0 || k > 0) ? 1u : 0u);
                tc_commit_pair(&empty[s]);
                tc_commit_pair(&acc_full[buf]);
            }
            if (it < chunks && it > 0) mbar_wait(&acc_full[(it - 1) & 1], (uint32_t)(((it - 1) >> 1) & 1));      // (given up: the products under way end first)
        } else if (warp_u == 17 && elect_one()) {
            // TMA producer of this block: its 128 weight rows and BN / 2 tokens of every chunk.  The weights too are asked for after the
            // wait: a float32 matrix may be the work of the kernel before this one.
            ti_pdl_sync();
            SplitWalk walk(total, nk, unit, g.units);
            SplitPiece p;
            int it = 0;
            bool ok = true;
            while (ok && walk.next(p)) {
                const int tn = p.tile / tiles_m, tm = p.tile - tn * tiles_m;
                for (int kc = p.c0; kc < p.c1; kc++, it++) {
                    const int rs = it % RAWS;
                    unsigned char* to = raw + (size_t)rs * RAW;
                    if (it >= RAWS && !mbar_wait(&raw_empty[rs], (uint32_t)(((it / RAWS) & 1) ^ 1))) {
                        ti_report(status, TI_STATUS_PIPE_WAIT); ok = false; break;
                    }
                    mbar_expect_tx(&raw_full[rs], RAW);
                    tma_load_2d(to, &w_map, kc * CHUNK, tn * 2 * WROWS + rank * WROWS, &raw_full[rs]);
                    tma_load_2d(to + WROWS * 128, &x_map, kc * CHUNK, tm * BN + rank * (BN / 2), &raw_full[rs]);
                }
            }
            // not before every copy has arrived, also where the warps that wait for them have given up
            for (int k = max(0, it - RAWS); k < it; k++) mbar_wait(&raw_full[k % RAWS], (uint32_t)((k / RAWS) & 1));
        }
    }
    // neither block leaves, or gives back its tensor memory, while the other may still read its shared memory or arrive on its barriers
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 16) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc_pair(tmem, TMEM_COLS);
    }
}

// Adds the pieces of the tiles that a unit's run ended in, in the order of the contraction.  Block (boundary, rank, group of
// 32 tokens), 128 threads: a thread per weight row.  The first boundary inside a tile does the tile.
template <int BN>
__global__ void __launch_bounds__(WROWS)
gemm_f32_join_kernel(const SplitArgs g, int tiles_m, int nk, long long total) {
    ti_pdl_trigger();
    const int u = blockIdx.x + 1, rank = blockIdx.y, j0 = blockIdx.z * 32;
    const long long cut = unit_begin(total, g.units, u);
    const int tile = (int)(cut / nk);
    const long long t0 = (long long)tile * nk, t1 = t0 + nk;
    if (cut == t0 || unit_begin(total, g.units, u - 1) > t0) return;        // no cut inside, or not the first one
    int last = u;                                                           // the unit with the tile's last piece
    while (last + 1 < g.units && unit_begin(total, g.units, last + 1) < t1) last++;
    ti_pdl_sync();
    const int tn = tile / tiles_m, tm = tile - tn * tiles_m;
    const int n = tn * 2 * WROWS + rank * WROWS + threadIdx.x;
    float sum[32];
#pragma unroll
    for (int j = 0; j < 32; j++) sum[j] = 0.f;
    for (int v = u - 1; v <= last; v++) {
        const long long b = unit_begin(total, g.units, v);
        const int place = (b >= t0 ? 0 : 1);                                // the unit's run begins inside this tile, or before it
        const float* ws = ti_dependent(g.workspace) + (((size_t)v * 2 + place) * 2 + rank) * (size_t)(BN * WROWS) + (size_t)j0 * WROWS + threadIdx.x;
        float x[32];                    // (a piece's numbers all on their way together)
#pragma unroll
        for (int j = 0; j < 32; j++) x[j] = __ldcg(ws + (size_t)j * WROWS);
        asm volatile("" ::: "memory");
#pragma unroll
        for (int j = 0; j < 32; j++) sum[j] += x[j];
    }
#pragma unroll
    for (int c = 0; c < 32; c += 16)
        if (tm * BN + j0 + c < g.M)
            store16(g, tm * BN + j0 + c, n, make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]), make_float4(sum[c + 4], sum[c + 5], sum[c + 6], sum[c + 7]),
                    make_float4(sum[c + 8], sum[c + 9], sum[c + 10], sum[c + 11]), make_float4(sum[c + 12], sum[c + 13], sum[c + 14], sum[c + 15]));
}

// Whether a run of chunks ends inside a tile, so that pieces are left to be added.
bool split_cuts(long long total, int units, int nk) {
    for (int u = 1; u < units; u++)
        if (unit_begin(total, units, u) % nk != 0) return true;
    return false;
}

template <int BN>
int launch_split(const SplitArgs& g, cudaStream_t stream) {
    constexpr size_t smem = (size_t)PARTS * split_stage_bytes<BN>() + (size_t)raw_stages<BN>() * raw_stage_bytes<BN>() + 1024;
    static bool configured = false;
    if (!configured) {
        // the register split of the roles must fit what a block is launched with (an increase would wait for ever otherwise)
        cudaFuncAttributes a;
        TI_CUDA(cudaFuncGetAttributes(&a, gemm_f32_split_kernel<BN>));
        TI_REQUIRE(a.numRegs >= LAUNCH_REGS, "linear (float32): the kernel was built with %d registers a thread, its roles share %d", a.numRegs, LAUNCH_REGS);
        TI_CUDA(cudaFuncSetAttribute(gemm_f32_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = true;
    }
    int* status = ti_status_ptr();
    TI_REQUIRE(status != nullptr, "linear: no status word");
    CUtensorMap wm, xm;
    if (int rc = ti_make_tensor_map_2d_f32(&wm, g.w, (uint64_t)g.N, (uint64_t)g.K, (uint64_t)g.ldw * 4, WROWS, CHUNK)) return rc;
    if (int rc = ti_make_tensor_map_2d_f32(&xm, g.x, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.ldx * 4, BN / 2, CHUNK)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * g.units);
    cfg.blockDim = dim3(SPLIT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ti_pdl_enabled(5) ? 2 : 1;
    TI_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel<BN>, wm, xm, g, status));
    TI_CHECK_LAUNCH("linear (float32, tcgen05)");
    const int tiles_m = (g.M + BN - 1) / BN, tiles_n = (g.N + 2 * WROWS - 1) / (2 * WROWS), nk = (g.K + CHUNK - 1) / CHUNK;
    const long long total = (long long)tiles_m * tiles_n * nk;
    if (split_cuts(total, g.units, nk)) {
        TI_CUDA(ti_launch_class<5>(gemm_f32_join_kernel<BN>, dim3(g.units - 1, 2, BN / 32), dim3(WROWS), 0, stream, g, tiles_m, nk, total));
        TI_CHECK_LAUNCH("linear (float32, pieces)");
    }
    return 0;
}

// Tokens per tile: the narrowest that holds them all, then 256.
int split_bn(int M) { return M <= 64 ? 64 : M <= 128 ? 128 : 256; }

int split_units(int M, int N, int K, int sms) {
    const int bn = split_bn(M), nk = (K + CHUNK - 1) / CHUNK;
    const long long tiles = (long long)((M + bn - 1) / bn) * ((N + 2 * WROWS - 1) / (2 * WROWS));
    return (int)std::min<long long>(sms / 2, std::max(tiles, tiles * nk / 4));        // tiles are cut only into runs of four chunks and more
}

}  // namespace

// Pairs of blocks, floats of workspace and launches of a product.
extern "C" int ti_linear_f32_plan(int M, int N, int K, int sms, int* units, long long* workspace, int* launches) {
    TI_REQUIRE(M > 0 && N > 0 && K > 0 && sms >= 2, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    *units = split_units(M, N, K, sms);
    const int bn = split_bn(M), nk = (K + CHUNK - 1) / CHUNK;
    const bool cut = split_cuts((long long)((M + bn - 1) / bn) * ((N + 2 * WROWS - 1) / (2 * WROWS)) * nk, *units, nk);
    *launches = cut ? 2 : 1;
    *workspace = cut ? (long long)*units * 4 * split_bn(M) * WROWS : 0;
    return 0;
}

// x [M, K], w [N, K], out [M, N] (or [M, N / 2] when gated 1 to 3) float32; the leading dimensions multiples of 4, x and
// w on 16-byte boundaries.
extern "C" int ti_linear_f32_tc(const void* x, const void* w, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo,
                                int units, float* workspace, int gated, float gate_limit, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    TI_REQUIRE(M > 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    TI_REQUIRE(ldx % 4 == 0 && ldw % 4 == 0 && ldx >= K && ldw >= K && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0,
               "linear (float32): rows must start on 16-byte boundaries");
    TI_REQUIRE(units >= 1 && units <= 32767 && (workspace != nullptr || !split_cuts((long long)((M + split_bn(M) - 1) / split_bn(M)) *
               ((N + 2 * WROWS - 1) / (2 * WROWS)) * ((K + CHUNK - 1) / CHUNK), units, (K + CHUNK - 1) / CHUNK)), "linear (float32): %d units without room", units);
    TI_REQUIRE(gated >= 0 && gated <= 5 && (gated < 1 || gated > 3 || N % 2 == 0), "linear (float32): unknown activation %d", gated);
    SplitArgs g{(const float*)x, (const float*)w, (float*)out, M, N, K, ldx, ldw, ldo, units, workspace, gated, gate_limit};
    switch (split_bn(M)) {
        case 64: return launch_split<64>(g, stream);
        case 128: return launch_split<128>(g, stream);
        default: return launch_split<256>(g, stream);
    }
}
