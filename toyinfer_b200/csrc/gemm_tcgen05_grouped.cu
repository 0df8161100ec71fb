// The tcgen05 matrix product over groups of rows that each meet a matrix of their own (the experts of a mixture):
// out[i, :] = a[i, :] W[group of i]^T.  The rows of a group stand together, every group padded to whole tiles of 128
// rows (the padding rows hold zeros), and `tile_group[t]` names the group of tile t (or -1: nothing to do).  The
// matrices are one tensor [groups * N, K]; a block's weight tile starts at row group * N + its column tile.  Otherwise
// the kernel is the one-block-per-tile product of gemm_tcgen05_tile.cu without the split contraction: TMA into an
// mbarrier ring, one elected thread issuing `tcgen05.mma`, accumulator in tensor memory, four epilogue warps.
// Which group a tile has is known only on the device, so nothing is requested before the wait for the earlier kernels.
//
// What bounds it: the operands' way into an SM (115 B/ns: 0.28 us a step of 32 KB), and with one block an SM the start and the end of
// every tile, in which nothing is on its way.  Two blocks of three stages each share an SM instead of one of six where there are tiles
// for it, and the activation of a gated pair is applied at the end (a tile of 64 gate and 64 up columns; a kernel of its own read and
// wrote the pairs again).  The whole layer, hidden 2,048, two choices a token, us before / with the activation inside
// / two blocks an SM too: 16 experts of 1,024, 3,000 tokens 176 / 168 / 149, 777 tokens with a shared expert 111 / 106 / 102.
// The gather and both products, one block an SM / two, at the tiles of the first and the second product that the rule counts: 8 experts
// of 1,000, 600 tokens with two choices (224, 224) 54.1 / 48.3; 16 of 640, 1,100 with one (170, 272) 52.0 / 45.5; 8 of 768, 512 with two
// (144, 192) 43.0 / 37.6; contractions of a few steps gain nothing, 16 of 512, hidden 1,024 (168, 168) 27.7 / 29.0, 8 of 1,280, hidden
// 1,024, one choice (240, 96) 30.0 / 30.5.  Where the tiles fit one round, two blocks lose: 8 of 1,000, 600 with one choice (144, 144)
// 35.1 / 44.3, 4 of 600, 150 with two (50, 80) 24.4 / 31.5.
#include "gemm_tcgen05.cuh"

namespace tigemm {
namespace {
constexpr int GBN = 128;

// What a gated pair's tile stores: g' sigmoid(alpha g') (u' + shift), g' = min(g, limit), u' = clamp(u, -limit, limit).  g and u are
// rounded to bfloat16 first, as the groups of fewer places have them (moe_rows.cuh, moe_grouped.cu): a token's result must not depend
// on how many others share its step.
struct PairAct { float limit, alpha, shift; };

template <int GSTAGES, bool PAIR>
__global__ void __launch_bounds__(THREADS, GSTAGES <= 3 ? 2 : 1)
gemm_tc_grouped_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b_map,
                       GemmArgs g, const int* __restrict__ tile_group, int rows_per_group, PairAct act, int* status) {
    ti_pdl_trigger();
    constexpr int A_BYTES = BM * BK * 2, B_BYTES = GBN * BK * 2;
    constexpr uint32_t TMEM_COLS = 128;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[GSTAGES], empty[GSTAGES], acc_ready;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_gave_up;
    if (threadIdx.x == 0) s_gave_up = *reinterpret_cast<volatile int*>(status);
    __syncthreads();
    if (s_gave_up) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int a0 = blockIdx.x * BM, b0 = blockIdx.y * (PAIR ? GBN / 2 : GBN);
    if (threadIdx.x == 0) {
        for (int s = 0; s < GSTAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&acc_ready, 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        __syncwarp();
        tmem_alloc(&tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    ti_pdl_sync();
    const int group = ti_dependent(tile_group)[blockIdx.x];
    const int n_iter = group >= 0 ? (g.K + BK - 1) / BK : 0;
    const int warp_u = warp_uniform();
    if (warp_u == 0) {
        if (elect_one()) {
            const int brow = group * rows_per_group + b0;
            for (int it = 0; it < n_iter; it++) {
                const int s = it % GSTAGES;
                if (it >= GSTAGES && !mbar_wait(&empty[s], (uint32_t)(((it / GSTAGES) & 1) ^ 1))) { ti_report(status, TI_STATUS_PIPE_WAIT); break; }
                unsigned char* sa = smem + (size_t)s * (A_BYTES + B_BYTES);
                mbar_expect_tx(&full[s], A_BYTES + B_BYTES);
                tma_load_2d(sa, &a_map, it * BK, a0, &full[s]);
                tma_load_2d(sa + A_BYTES, &b_map, it * BK, brow, &full[s]);
                if constexpr (PAIR) tma_load_2d(sa + A_BYTES + B_BYTES / 2, &b_map, it * BK, brow + (rows_per_group >> 1), &full[s]);
            }
        }
    } else if (warp_u == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = instr_desc<GBN>();
            bool ok = true;
            for (int it = 0; it < n_iter && ok; it++) {
                const int s = it % GSTAGES;
                if (!mbar_wait(&full[s], (uint32_t)((it / GSTAGES) & 1))) { ti_report(status, TI_STATUS_TMA_WAIT); ok = false; break; }
                tc_fence_after();
                const uint32_t sa = smem_u32(smem + (size_t)s * (A_BYTES + B_BYTES));
                const uint64_t da = smem_desc_sw128(sa), db = smem_desc_sw128(sa + A_BYTES);
#pragma unroll
                for (int k = 0; k < BK / 16; k++)
                    tc_mma_bf16(tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (it > 0 || k > 0) ? 1u : 0u);
                tc_commit(&empty[s]);
            }
            if (ok && n_iter > 0) tc_commit(&acc_ready);
        }
    } else {
        const int q = warp & 3;
        const int i = a0 + q * 32 + lane;
        bool ok = n_iter > 0;
        if (n_iter > 0) {
            if (!mbar_wait(&acc_ready, 0)) { ti_report(status, TI_STATUS_MMA_WAIT); ok = false; }
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
        }
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
        if (ok) {
#pragma unroll 1
            for (int c = 0; c < (PAIR ? GBN / 2 : GBN); c += 16) {
                float r[16];
                tmem_ld16(taddr + c, r);
                if constexpr (PAIR) {
                    float u[16];
                    tmem_ld16(taddr + GBN / 2 + c, u);
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        const __nv_bfloat162 gu = __floats2bfloat162_rn(r[e], u[e]);        // (both in one conversion)
                        const uint32_t both = *reinterpret_cast<const uint32_t*>(&gu);
                        const float gate = fminf(__uint_as_float(both << 16), act.limit);
                        const float up = fminf(fmaxf(__uint_as_float(both & 0xffff0000u), -act.limit), act.limit);
                        r[e] = gate * (ti_over(1.0f, 1.0f + expf(-act.alpha * gate))) * (up + act.shift);
                    }
                }
                store_chunk(g, i, b0, c, r, lane);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

template <int GSTAGES, bool PAIR>
int launch_grouped(dim3 grid, const CUtensorMap& am, const CUtensorMap& bm, const GemmArgs& g, const int* tile_group, int rows_per_group,
                   PairAct act, int* status, cudaStream_t stream) {
    constexpr size_t smem = (size_t)GSTAGES * (BM * BK * 2 + GBN * BK * 2) + 1024;
    static bool configured = false;
    if (!configured) {
        TI_CUDA(cudaFuncSetAttribute(gemm_tc_grouped_kernel<GSTAGES, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = true;
    }
    TI_CUDA(ti_launch_class<5>(gemm_tc_grouped_kernel<GSTAGES, PAIR>, grid, dim3(THREADS), smem, stream, am, bm, g, tile_group, rows_per_group, act, status));
    TI_CHECK_LAUNCH("linear_grouped (tcgen05)");
    return 0;
}
}  // namespace
}  // namespace tigemm

// a: bfloat16 [rows, K] dense, rows a multiple of 128 (groups padded to whole tiles); out: bfloat16 [rows, N] with row stride ld_out;
// tile_group: int32 [rows / 128] on the device.  act 0 or 4 (the squared ReLU of every value): W bfloat16 [groups, N, K] dense; act 1:
// W [groups, 2 N, K], a group's gate rows and then its up rows, and `out` holds their gated pairs (PairAct).
extern "C" int ti_linear_grouped_tc(const void* a, const void* W, void* out, const int* tile_group, int rows, int groups, int N,
                                    int K, long long ld_out, int act, float limit, float alpha, float shift, cudaStream_t stream) {
    using namespace tigemm;
    if (rows == 0) return 0;
    TI_REQUIRE(rows > 0 && rows % BM == 0 && groups > 0 && N > 0 && K > 0, "linear_grouped: bad sizes rows=%d groups=%d N=%d K=%d", rows, groups, N, K);
    TI_REQUIRE(K % 8 == 0, "linear_grouped: rows of %d elements are not whole 16-byte pieces", K);
    TI_REQUIRE(act == 0 || act == 1 || act == 4, "linear_grouped: unknown activation %d", act);
    const bool pair = act == 1;
    const int per_group = pair ? 2 * N : N, cols = pair ? GBN / 2 : GBN;
    CUtensorMap am, bm;
    if (int rc = ti_make_tensor_map_2d_bf16(&am, a, (uint64_t)rows, (uint64_t)K, (uint64_t)K * 2, BM, BK)) return rc;
    if (int rc = ti_make_tensor_map_2d_bf16(&bm, W, (uint64_t)groups * per_group, (uint64_t)K, (uint64_t)K * 2, cols, BK)) return rc;
    GemmArgs g = {};
    g.rows_a = rows; g.rows_b = N; g.K = K; g.out = out; g.ld_out = ld_out; g.out_f32 = 0; g.transposed = 0; g.splits = 1;
    g.gated = act == 4 ? 4 : 0;
    int* status = ti_status_ptr();
    TI_REQUIRE(status != nullptr, "linear_grouped: no status word");
    dim3 grid(rows / BM, (N + cols - 1) / cols);
    TI_REQUIRE(grid.y <= 65535, "linear_grouped: %d weight rows are too many for one launch", N);
    const PairAct pa{limit, alpha, shift};
    // Two blocks an SM where the tiles are more than one round of SMs (the groups' padding leaves half a tile each empty on average; how
    // many tiles hold rows is known on the device only); else one, with all its memory for the stages.
    const bool two = ((long long)grid.x - groups / 2) * grid.y > ti_sm_count();
    if (pair) return two ? launch_grouped<3, true>(grid, am, bm, g, tile_group, per_group, pa, status, stream)
                         : launch_grouped<6, true>(grid, am, bm, g, tile_group, per_group, pa, status, stream);
    return two ? launch_grouped<3, false>(grid, am, bm, g, tile_group, per_group, pa, status, stream)
               : launch_grouped<6, false>(grid, am, bm, g, tile_group, per_group, pa, status, stream);
}
