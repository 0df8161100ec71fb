// One token per sequence through a recurrent layer's state: lightning attention (lightning.cu) and the gated delta rule
// (delta_rule.cu), whose scans serve every other step.  The recurrences are theirs:
//   lightning:  S <- decay S + k v^T;                                          o = S^T q     (entry function, k_scale)
//   delta:      S <- diag(g) S;  e = beta (v - S^T k);  S <- S + k e^T;        o = S^T q     (unit q and k, a decay per head or channel)
// Everything of the recurrence is 32-bit.
//
// What bounds it: reading and writing the state, 64 KB a head of 128 x 128.  A block takes a (sequence, head): a thread holds R
// rows of four columns, all of its reads on their way together, the sums over the rows meet in shared memory (once for
// lightning, twice for the delta rule), and the delta rule's unit vectors and decays are made by the block itself while the
// state is on its way, so the step has no kernel before this one.  32 sequences of 16 heads of 128 x 128 (67 MB of state read and
// written) through lightning attention, us: the scan, a thread a column with its 128 rows one read each, 42; this 17.
#include "common.cuh"

#include <type_traits>

namespace {

constexpr int ST_THREADS = 256;
enum { ST_LIGHTNING = 0, ST_DELTA_HEAD = 1, ST_DELTA_CHANNEL = 2 };

__device__ __forceinline__ float st_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

struct StepArgs {
    const void* q; const void* k; const void* v;
    long long q_stride, k_stride, v_stride;
    const void* decay; long long decay_stride;      // lightning: float32 [heads]; delta: logits
    const float* dt_bias; const float* rate; const void* beta; long long beta_stride;
    float* o; float* state; long long slot_stride;
    const int* cu_new; const int* seq_slot;
    int n_heads, qk_heads, M;
    int act; float k_scale;
};

// D rows, V columns, R = rows of a thread
template <typename T, int ALG, int D, int V>
__global__ void __launch_bounds__(ST_THREADS)
state_step_kernel(StepArgs a) {
    ti_pdl_trigger();
    constexpr int CQ = V / 4, RG = ST_THREADS / CQ, R = D / RG;
    __shared__ float ks[D], qs[D], gs[D], sums[RG][V], es[V];
    __shared__ float s_beta;
    const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cq = tid % CQ, rg = tid / CQ;
    ti_pdl_sync();
    const T* q = ti_dependent((const T*)a.q);
    const T* k = ti_dependent((const T*)a.k);
    const T* v = ti_dependent((const T*)a.v);
    if (b == 0 && ALG != ST_LIGHTNING)      // rows past the last sequence's are nobody's
        for (int i = tid; i < (a.M - a.cu_new[gridDim.y]) * V; i += ST_THREADS)
            a.o[((size_t)(a.cu_new[gridDim.y] + i / V) * a.n_heads + h) * V + i % V] = 0.f;
    const int tok = a.cu_new[b];
    if (a.cu_new[b + 1] <= tok) return;
    float4* S = reinterpret_cast<float4*>(a.state + (size_t)a.seq_slot[b] * a.slot_stride + (size_t)h * D * V) + (size_t)rg * CQ + cq;
    float4 s[R];
#pragma unroll
    for (int r = 0; r < R; r++) s[r] = S[(size_t)r * RG * CQ];      // rows rg, rg + RG, ...
    const int hq = h / (a.n_heads / a.qk_heads);
    const T* qr = q + (size_t)tok * a.q_stride + (size_t)hq * D;
    const T* kr = k + (size_t)tok * a.k_stride + (size_t)hq * D;
    float lam = 0.f;
    if constexpr (ALG == ST_LIGHTNING) {
        lam = ((const float*)a.decay)[h];
        for (int i = tid; i < D; i += ST_THREADS) {
            const float x = to_f32(kr[i]), y = to_f32(qr[i]);
            ks[i] = (a.act ? ti_over(x, 1.0f + expf(-x)) : x) * a.k_scale;
            qs[i] = a.act ? ti_over(y, 1.0f + expf(-y)) : y;
        }
        for (int i = tid; i < V; i += ST_THREADS) {
            const float x = to_f32(v[(size_t)tok * a.v_stride + (size_t)h * V + i]);
            es[i] = a.act ? ti_over(x, 1.0f + expf(-x)) : x;
        }
    } else {
        if (warp < 2) {         // unit key, unit query times dim^-1/2
            const T* from = warp == 0 ? kr : qr;
            float x[D / 32], ss = 0.f;
#pragma unroll
            for (int i = 0; i < D / 32; i++) { x[i] = to_f32(from[lane + 32 * i]); ss = fmaf(x[i], x[i], ss); }
            const float inv = rsqrtf(warp_sum(ss) + 1e-6f) * (warp == 0 ? 1.0f : rsqrtf((float)D));
            float* to = warp == 0 ? ks : qs;
#pragma unroll
            for (int i = 0; i < D / 32; i++) to[lane + 32 * i] = x[i] * inv;
        } else if (warp < 6) {
            const float rt = a.rate[h];
            for (int i = tid - 64; i < (ALG == ST_DELTA_CHANNEL ? D : 1); i += 128) {
                float l, dt;
                if constexpr (ALG == ST_DELTA_CHANNEL) {
                    l = ((const float*)a.decay)[(size_t)tok * a.decay_stride + (size_t)h * D + i];
                    dt = a.dt_bias[(size_t)h * D + i];
                } else {
                    l = to_f32(((const T*)a.decay)[(size_t)tok * a.decay_stride + h]);
                    dt = a.dt_bias[h];
                }
                gs[i] = expf(-rt * st_softplus(l + dt));
            }
        } else if (warp == 6) {
            if (lane == 0) s_beta = ti_over(1.0f, 1.0f + expf(-to_f32(((const T*)a.beta)[(size_t)tok * a.beta_stride + h])));
        }
    }
    __syncthreads();
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (ALG == ST_LIGHTNING) {
        const float4 e = *reinterpret_cast<const float4*>(es + 4 * cq);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float kv = ks[rg + r * RG], qv = qs[rg + r * RG];
            s[r].x = fmaf(lam, s[r].x, kv * e.x); s[r].y = fmaf(lam, s[r].y, kv * e.y);
            s[r].z = fmaf(lam, s[r].z, kv * e.z); s[r].w = fmaf(lam, s[r].w, kv * e.w);
            acc.x = fmaf(s[r].x, qv, acc.x); acc.y = fmaf(s[r].y, qv, acc.y);
            acc.z = fmaf(s[r].z, qv, acc.z); acc.w = fmaf(s[r].w, qv, acc.w);
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float g = ALG == ST_DELTA_CHANNEL ? gs[rg + r * RG] : gs[0], kv = ks[rg + r * RG];
            s[r].x *= g; s[r].y *= g; s[r].z *= g; s[r].w *= g;
            acc.x = fmaf(s[r].x, kv, acc.x); acc.y = fmaf(s[r].y, kv, acc.y);
            acc.z = fmaf(s[r].z, kv, acc.z); acc.w = fmaf(s[r].w, kv, acc.w);
        }
        *reinterpret_cast<float4*>(&sums[rg][4 * cq]) = acc;
        __syncthreads();
        for (int i = tid; i < V; i += ST_THREADS) {
            float d = 0.f;
#pragma unroll
            for (int j = 0; j < RG; j++) d += sums[j][i];
            es[i] = s_beta * (to_f32(v[(size_t)tok * a.v_stride + (size_t)h * V + i]) - d);
        }
        __syncthreads();
        const float4 e = *reinterpret_cast<const float4*>(es + 4 * cq);
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float kv = ks[rg + r * RG], qv = qs[rg + r * RG];
            s[r].x = fmaf(kv, e.x, s[r].x); s[r].y = fmaf(kv, e.y, s[r].y);
            s[r].z = fmaf(kv, e.z, s[r].z); s[r].w = fmaf(kv, e.w, s[r].w);
            acc.x = fmaf(s[r].x, qv, acc.x); acc.y = fmaf(s[r].y, qv, acc.y);
            acc.z = fmaf(s[r].z, qv, acc.z); acc.w = fmaf(s[r].w, qv, acc.w);
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++) S[(size_t)r * RG * CQ] = s[r];
    *reinterpret_cast<float4*>(&sums[rg][4 * cq]) = acc;
    __syncthreads();
    for (int i = tid; i < V; i += ST_THREADS) {
        float d = 0.f;
#pragma unroll
        for (int j = 0; j < RG; j++) d += sums[j][i];
        a.o[((size_t)tok * a.n_heads + h) * V + i] = d;
    }
}

template <typename T, int ALG>
int launch_step(const StepArgs& a, int n_seq, int dim, int vdim, cudaStream_t stream) {
    auto go = [&](auto dc, auto vc) -> int {
        TI_CUDA(ti_launch(state_step_kernel<T, ALG, decltype(dc)::value, decltype(vc)::value>, dim3(a.n_heads, n_seq), dim3(ST_THREADS), 0, stream, a));
        TI_CHECK_LAUNCH("state step");
        return 0;
    };
    using C64 = std::integral_constant<int, 64>;
    using C128 = std::integral_constant<int, 128>;
    if (dim == 64) return vdim == 64 ? go(C64(), C64()) : go(C64(), C128());
    return vdim == 64 ? go(C128(), C64()) : go(C128(), C128());
}

int check_step(const StepArgs& a, int n_seq, int dim, int vdim) {
    TI_REQUIRE(n_seq > 0 && n_seq <= 65535 && a.n_heads > 0 && a.qk_heads > 0 && a.n_heads % a.qk_heads == 0, "state step: bad sizes");
    TI_REQUIRE((dim == 64 || dim == 128) && (vdim == 64 || vdim == 128), "state step: heads of %d x %d are not taken", dim, vdim);
    TI_REQUIRE(a.slot_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(a.state) & 15) == 0, "state step: the state must lie on 16-byte boundaries");
    return 0;
}

}  // namespace

// As ti_lightning_scan (lightning.cu) where no sequence brings more than one token, for heads of 64 or 128 x 64 or 128.
extern "C" int ti_lightning_step(const void* q, const void* k, const void* v, long long q_stride, long long k_stride, long long v_stride,
                                 float* o, float* state, const float* decay, const int* cu_new, const int* seq_slot, int n_seq, int n_heads,
                                 int dim, int vdim, int act, float k_scale, int dtype, cudaStream_t stream) {
    if (n_seq == 0) return 0;
    StepArgs a{q, k, v, q_stride, k_stride, v_stride, decay, 0, nullptr, nullptr, nullptr, 0, o, state, (long long)n_heads * dim * vdim, cu_new, seq_slot,
               n_heads, n_heads, 0, act, k_scale};
    if (int rc = check_step(a, n_seq, dim, vdim)) return rc;
    return ti_dispatch_dtype(dtype, [&](auto t) -> int { return launch_step<decltype(t), ST_LIGHTNING>(a, n_seq, dim, vdim, stream); });
}

// As ti_delta_rule_scan (delta_rule.cu) where no sequence brings more than one token, for heads of 64 or 128 x 64 or 128.
extern "C" int ti_delta_step(const void* q, const void* k, const void* v, long long q_stride, long long k_stride, long long v_stride,
                             const void* decay_logit, long long decay_stride, int head_decay, const float* dt_bias, const float* rate,
                             const void* beta_logit, long long beta_stride, float* o, float* state, long long slot_stride, const int* cu_new,
                             const int* seq_slot, int n_seq, int M, int n_heads, int qk_heads, int dim, int vdim, int dtype, cudaStream_t stream) {
    if (n_seq == 0 || M == 0) return 0;
    StepArgs a{q, k, v, q_stride, k_stride, v_stride, decay_logit, decay_stride, dt_bias, rate, beta_logit, beta_stride, o, state, slot_stride, cu_new,
               seq_slot, n_heads, qk_heads, M, 0, 1.0f};
    if (int rc = check_step(a, n_seq, dim, vdim)) return rc;
    return ti_dispatch_dtype(dtype, [&](auto t) -> int {
        using T = decltype(t);
        return head_decay ? launch_step<T, ST_DELTA_HEAD>(a, n_seq, dim, vdim, stream) : launch_step<T, ST_DELTA_CHANNEL>(a, n_seq, dim, vdim, stream);
    });
}
