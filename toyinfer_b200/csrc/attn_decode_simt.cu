// Grouped-query attention of one new token per sequence over the paged cache,
// split along the keys, CUDA cores, 32-bit arithmetic.
//
// For sequence b with length L (the new token included, already stored) and query
// head h: keys at positions max(0, L - window) .. L-1 (all of them when window == 0),
// s_j = (q . k_j) * scale, softmax with the maximum subtracted, o = sum p_j v_j.
// Reference: src/decode.cu:401-432 (scores), :471-532 (softmax), :598-628 (values);
// it materialises all scores and clears max_seq_len-sized buffers every layer
// (src/decode.cu:703-744), here nothing is proportional to the capacity.
//
// Grid (sequences, kv heads x chunks of their query heads, splits), 256 threads.  A block takes up to six of the query
// heads that share its kv head, so every key and value is read once for all of them.  The tiles of 64 positions in range
// (a tile is one page of the cache) are dealt to the splits in contiguous runs, a split's keys to its eight warps in turn.
//
// What bounds it: on short sequences (one page) the chain of dependent loads, page table -> key -> score -> value sum; on
// long ones the read of the cache.  So nothing of a tile goes through shared memory and no barrier stands in the loop: the
// lanes of a warp lie along the head (four elements each, LPK lanes a key), a warp has 8 keys a lane group and their values
// in flight at once as 16-byte loads, the 8 dot products a head are added up over the lanes by exchanges that halve the keys
// each lane still sums (9 shuffles a head for 8 keys instead of 40), the softmax runs per warp, and the weights come back
// to the lanes by shuffles.  The warps meet once, at the end.
// Measured, a layer's step in us against the form that staged tiles in shared memory (one thread a score): 4 sequences of up to
// 589 positions, 32 heads of 128 over 8, 114 -> 52 (the attention 70 -> 12); 16 of up to 2,000, 40 over 8, 437 -> 185 (307 -> 57,
// 4.6 TB/s); one of 2,000, 24 over 4, 123 -> 42; heads of 32 at some twenty positions 12 -> 4 and no merging kernel.
// Up to CLUSTER_SPLITS splits are launched as one cluster and merge through distributed shared memory where all clusters find room
// (launch_form); else they go through global scratch and `attn_decode_combine_kernel`.  With one split the result is written directly.
#include "attn_decode.cuh"

#include <cooperative_groups.h>

namespace {
namespace cg = cooperative_groups;
using tiattn::DecodeArgs;
using tiattn::attn_decode_combine_kernel;
constexpr int TILE = 64, WARPS = 8, THREADS = 32 * WARPS, KEYS = 8;     // KEYS: per lane group and turn
constexpr int MAX_OUTPUTS = 4096, CLUSTER_SPLITS = 16;     // (above 8 a cluster must opt in)

// Elements 4 i .. 4 i + 3 of a row of hd elements, zero past its end.  VEC: the row starts on a boundary of four elements
// and hd is a multiple of four.
template <bool VEC>
__device__ __forceinline__ void load4(float (&x)[4], const float* row, int i, int hd) {
    if (VEC) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (4 * i < hd) v = *reinterpret_cast<const float4*>(row + 4 * i);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) x[e] = 4 * i + e < hd ? row[4 * i + e] : 0.f;
    }
}
template <bool VEC>
__device__ __forceinline__ void load4(float (&x)[4], const bf16* row, int i, int hd) {
    if (VEC) {
        uint2 v = make_uint2(0u, 0u);
        if (4 * i < hd) v = *reinterpret_cast<const uint2*>(row + 4 * i);
        x[0] = __uint_as_float(v.x << 16); x[1] = __uint_as_float(v.x & 0xffff0000u);
        x[2] = __uint_as_float(v.y << 16); x[3] = __uint_as_float(v.y & 0xffff0000u);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) x[e] = 4 * i + e < hd ? to_f32(row[4 * i + e]) : 0.f;
    }
}

// LPK lanes hold a key, NV runs of four elements each (run i of a lane: elements 4 (i LPK + lane) ..); G query heads.
template <typename T, int LPK, int NV, int G, bool VEC>
__global__ void __launch_bounds__(THREADS)
attn_decode_kernel(DecodeArgs a, int chunks, int in_cluster) {
    ti_pdl_trigger();
    extern __shared__ float sm[];
    __shared__ float warp_m[WARPS][G], warp_l[WARPS][G], block_ml[G][2];
    constexpr int GROUPS = 32 / LPK, BATCH = KEYS * GROUPS;
    const int hd = a.hd, g = a.n_heads / a.n_kv_heads;
    float* Wo = sm;                    // [WARPS][G][hd]
    const int b = blockIdx.x, kvh = blockIdx.y / chunks, chunk = blockIdx.y - kvh * chunks, split = blockIdx.z;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, sub = lane % LPK, grp = lane / LPK;
    const int h0 = kvh * g + chunk * G, live_heads = min(G, g - chunk * G);
    ti_pdl_sync();
    const int L = a.seq_len[b];
    const int slot = a.seq_slot[b];
    const int lo = a.window > 0 ? max(0, L - a.window) : 0;
    const int tile_lo = lo / TILE, tile_hi = (L - 1) / TILE;       // inclusive
    const int n_tiles = L > 0 ? tile_hi - tile_lo + 1 : 0;
    const int per = (n_tiles + a.n_splits - 1) / a.n_splits;
    const int my_lo = tile_lo + split * per;
    const int my_hi = min(my_lo + per, tile_lo + n_tiles);           // exclusive

    float q[G][NV][4];
#pragma unroll
    for (int h = 0; h < G; h++)
#pragma unroll
        for (int i = 0; i < NV; i++)
            load4<false>(q[h][i], (const T*)a.q + (size_t)b * a.q_stride + (size_t)(h0 + h) * hd, i * LPK + sub, h < live_heads ? hd : 0);
    float acc[G][NV][4], m[G], l[G];
#pragma unroll
    for (int h = 0; h < G; h++) {
        m[h] = -INFINITY; l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < NV; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[h][i][e] = 0.f;
    }

    const int end = min(my_hi * TILE, L);
    for (int p0 = my_lo * TILE + warp * BATCH; p0 < end; p0 += WARPS * BATCH) {
        if (p0 + BATCH <= lo) continue;
        const int row0 = a.ring_rows > 0 ? p0 % a.ring_rows : p0;      // (a batch lies inside one page)
        const int pidx = row0 / TILE;
        int page = pidx < a.table_width ? a.page_table[(size_t)slot * a.table_width + pidx] : 0;
        if (page < 0 || page >= a.n_pages) page = 0;
        const size_t first = (((size_t)page * a.n_kv_heads + kvh) * TILE + row0 % TILE) * hd;
        float kx[KEYS][NV][4], vx[KEYS][NV][4];
        auto values = [&]() {
#pragma unroll
            for (int k = 0; k < KEYS; k++) {
                const int r = k * GROUPS + grp, p = p0 + r;
                const int n = p >= lo && p < L ? hd : 0;
#pragma unroll
                for (int i = 0; i < NV; i++) load4<VEC>(vx[k][i], (const T*)a.v_pages + first + (size_t)r * hd, i * LPK + sub, n);
            }
        };
#pragma unroll
        for (int k = 0; k < KEYS; k++) {
            const int r = k * GROUPS + grp, p = p0 + r;
            const int n = p >= lo && p < L ? hd : 0;                     // a line outside the range may hold anything
#pragma unroll
            for (int i = 0; i < NV; i++) load4<VEC>(kx[k][i], (const T*)a.k_pages + first + (size_t)r * hd, i * LPK + sub, n);
        }
        if constexpr (NV < 4) values();                                  // (four runs: no registers for both; one head, scored first)
        // the key whose scores this lane ends up with, of its group's eight
        const int mine = sub / (LPK / 8), p_mine = p0 + mine * GROUPS + grp;
        const bool live = p_mine >= lo && p_mine < L;
#pragma unroll
        for (int h = 0; h < G; h++) {
            float s[KEYS];
#pragma unroll
            for (int k = 0; k < KEYS; k++) {
                s[k] = q[h][0][0] * kx[k][0][0];
#pragma unroll
                for (int i = 0; i < NV; i++)
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (i + e > 0) s[k] = fmaf(q[h][i][e], kx[k][i][e], s[k]);
            }
#pragma unroll
            for (int half = KEYS / 2, o = LPK / 2; half > 0; half >>= 1, o >>= 1) {
                const bool upper = sub & o;
#pragma unroll
                for (int k = 0; k < half; k++) {
                    const float keep = upper ? s[k + half] : s[k], give = upper ? s[k] : s[k + half];
                    s[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            }
            if constexpr (NV >= 4) values();
            float x = s[0];
#pragma unroll
            for (int o = LPK / 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            x = live ? x * a.scale : -INFINITY;
            float top = x;
#pragma unroll
            for (int o = LPK / 8; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_new = fmaxf(m[h], top);
            float p = 0.f;
            if (m_new > -INFINITY) {
                p = expf(x - m_new);
                if (m_new > m[h]) {                     // the same for all lanes
                    const float alpha = expf(m[h] - m_new);
                    l[h] *= alpha;
#pragma unroll
                    for (int i = 0; i < NV; i++)
#pragma unroll
                        for (int e = 0; e < 4; e++) acc[h][i][e] *= alpha;
                    m[h] = m_new;
                }
            }
            l[h] += p;
#pragma unroll
            for (int k = 0; k < KEYS; k++) {
                const float pk = __shfl_sync(0xffffffffu, p, grp * LPK + k * (LPK / 8));
#pragma unroll
                for (int i = 0; i < NV; i++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[h][i][e] = fmaf(pk, vx[k][i][e], acc[h][i][e]);
            }
        }
    }
    // the warp's sums: l over the lanes with different keys, the values over the lane groups
#pragma unroll
    for (int h = 0; h < G; h++) {
#pragma unroll
        for (int o = LPK / 8; o < 32; o <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);
#pragma unroll
        for (int i = 0; i < NV; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                float x = acc[h][i][e];
#pragma unroll
                for (int o = LPK; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                const int d = 4 * (i * LPK + sub) + e;
                if (grp == 0 && d < hd) Wo[(warp * G + h) * hd + d] = x;
            }
        if (lane == 0) { warp_m[warp][h] = m[h]; warp_l[warp][h] = l[h]; }
    }
    __syncthreads();
    const int n_out = live_heads * hd;
    for (int idx = t; idx < n_out; idx += THREADS) {
        const int h = idx / hd, d = idx - h * hd;
        float top = -INFINITY, sum = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; w++) top = fmaxf(top, warp_m[w][h]);
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
            const float mw = warp_m[w][h], e = mw > -INFINITY ? expf(mw - top) : 0.f;
            if (e > 0.f) { sum = fmaf(warp_l[w][h], e, sum); o = fmaf(Wo[(w * G + h) * hd + d], e, o); }
        }
        if (a.n_splits == 1) {
            ((T*)a.out)[(size_t)b * a.o_stride + (size_t)(h0 + h) * hd + d] = from_f32<T>(sum > 0.f ? o / sum : 0.f);
            continue;
        }
        const size_t part = ((size_t)b * a.n_heads + h0 + h) * a.n_splits + split;
        if (in_cluster) {
            Wo[h * hd + d] = o;          // warp 0's place: this thread alone has read it
            if (d == 0) { block_ml[h][0] = top; block_ml[h][1] = sum; }
        } else {
            a.part_o[part * hd + d] = o;
            if (d == 0) { a.part_ml[part * 2] = top; a.part_ml[part * 2 + 1] = sum; }
        }
    }
    if (!in_cluster) return;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int idx = split * THREADS + t; idx < n_out; idx += a.n_splits * THREADS) {
        const int h = idx / hd;
        float top = -INFINITY, sum = 0.f, o = 0.f;
#pragma unroll 4
        for (int r = 0; r < a.n_splits; r++) top = fmaxf(top, *cluster.map_shared_rank(&block_ml[h][0], r));
#pragma unroll 4
        for (int r = 0; r < a.n_splits; r++) {
            const float mr = *cluster.map_shared_rank(&block_ml[h][0], r), lr = *cluster.map_shared_rank(&block_ml[h][1], r);
            const float e = mr > -INFINITY ? expf(mr - top) : 0.f;
            if (e > 0.f) { sum = fmaf(lr, e, sum); o = fmaf(*cluster.map_shared_rank(Wo + idx, r), e, o); }
        }
        ((T*)a.out)[(size_t)b * a.o_stride + (size_t)h0 * hd + idx] = from_f32<T>(sum > 0.f ? o / sum : 0.f);
    }
    cluster.sync();        // nobody leaves while its shared memory may still be read
}

// How many clusters of n_splits blocks the device holds at once, asked once for each.
template <typename T, int LPK, int NV, int G, bool VEC>
int cluster_room(int n_splits, size_t smem, int* room) {
    static int known[64][CLUSTER_SPLITS + 1] = {};       // room + 1
    int dev = 0;
    TI_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && known[dev][n_splits] > 0) { *room = known[dev][n_splits] - 1; return 0; }
    auto* kernel = attn_decode_kernel<T, LPK, NV, G, VEC>;
    if (n_splits > 8) TI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, n_splits);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)n_splits;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TI_CUDA(cudaOccupancyMaxActiveClusters(room, kernel, &cfg));
    if (dev >= 0 && dev < 64) known[dev][n_splits] = *room + 1;
    return 0;
}

// kernels != null: nothing is launched, only the number of kernels that would be is left there.
//
// Clusters are placed whole, inside one part of the chip; those that find no room with the others wait for a whole one to end.  So
// they are taken only where all of them fit at once with some to spare (as the tensor-core kernel's plan asks, kernels/attention.py), else
// the splits meet through scratch memory.  us, as clusters / through scratch: 24 query heads of 128 over 4, four sequences of 2,000
// positions (16 clusters of 8) 27.9 / 17.2; 32 over 8, three of 7,000 (24 of 12) 57 / 38; 64 of 32 over 8, one of 2,000 (16 of 8) 13.7 /
// 8.1; where they fit: 32 of 128 over 8, one of 300 10.7 / 11.5, 16 of 32 over one, one of 300 5.7 / 7.1.
template <typename T, int LPK, int NV, int G, bool VEC>
int launch_form(const DecodeArgs& a, int n_seq, cudaStream_t stream, int* kernels) {
    const int g = a.n_heads / a.n_kv_heads, hd = a.hd, chunks = (g + G - 1) / G;
    const size_t smem = (size_t)WARPS * G * hd * sizeof(float);
    TI_REQUIRE((long long)a.n_kv_heads * chunks <= 65535, "attention_decode: %d kv heads with %d query heads each", a.n_kv_heads, g);
    static_assert(WARPS * G * LPK * NV * 4 * sizeof(float) <= 48 * 1024, "the warps' sums fit without a setting of the kernel's");
    int in_cluster = 0;
    if (a.n_splits > 1 && a.n_splits <= CLUSTER_SPLITS) {
        int room = 0;
        if (int rc = cluster_room<T, LPK, NV, G, VEC>(a.n_splits, smem, &room)) return rc;
        in_cluster = (long long)n_seq * a.n_kv_heads * chunks * 27 <= room * 25LL;
    }
    if (kernels) { *kernels = a.n_splits > 1 && !in_cluster ? 2 : 1; return 0; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_seq, a.n_kv_heads * chunks, a.n_splits);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (a.n_splits > 8 && in_cluster)
        TI_CUDA(cudaFuncSetAttribute(attn_decode_kernel<T, LPK, NV, G, VEC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (in_cluster) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = 1;
        attr[n_attr].val.clusterDim.y = 1;
        attr[n_attr++].val.clusterDim.z = (unsigned)a.n_splits;
    }
    if (ti_pdl_enabled(3)) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    TI_CUDA(cudaLaunchKernelEx(&cfg, attn_decode_kernel<T, LPK, NV, G, VEC>, a, chunks, in_cluster));
    TI_CHECK_LAUNCH("attention_decode");
    if (a.n_splits > 1 && !in_cluster) {
        dim3 cgrid(n_seq, a.n_heads);
        TI_CUDA(ti_launch(attn_decode_combine_kernel<T>, cgrid, dim3(hd < 128 ? 64 : 128), 0, stream, (const float*)a.part_o, (const float*)a.part_ml, (T*)a.out, a.o_stride, a.n_heads, hd, a.n_splits, (const bf16*)nullptr, 0LL));
        TI_CHECK_LAUNCH("attention_decode (combine)");
    }
    return 0;
}

// Query heads a block takes: all that share a kv head up to six (more registers leave one block on an SM), chunks of four
// beyond; wide heads, whose elements already fill the registers, one or two.
template <typename T, int LPK, bool VEC>
int launch_narrow(const DecodeArgs& a, int n_seq, cudaStream_t stream, int* kernels) {
    const int g = a.n_heads / a.n_kv_heads;
    if (!VEC || g == 1) return launch_form<T, LPK, 1, 1, VEC>(a, n_seq, stream, kernels);
    if (g == 2) return launch_form<T, LPK, 1, 2, true>(a, n_seq, stream, kernels);
    if (g == 5 || g == 6) return launch_form<T, LPK, 1, 6, true>(a, n_seq, stream, kernels);
    return launch_form<T, LPK, 1, 4, true>(a, n_seq, stream, kernels);
}

template <typename T, bool VEC>
int launch_width(const DecodeArgs& a, int n_seq, cudaStream_t stream, int* kernels) {
    const int hd = a.hd;
    if (hd <= 32) return launch_narrow<T, 8, VEC>(a, n_seq, stream, kernels);
    if (hd <= 64) return launch_narrow<T, 16, VEC>(a, n_seq, stream, kernels);
    if (hd <= 128) return launch_narrow<T, 32, VEC>(a, n_seq, stream, kernels);
    if (hd <= 256) return VEC && a.n_heads / a.n_kv_heads > 1 ? launch_form<T, 32, 2, 2, true>(a, n_seq, stream, kernels) : launch_form<T, 32, 2, 1, VEC>(a, n_seq, stream, kernels);
    return launch_form<T, 32, 4, 1, VEC>(a, n_seq, stream, kernels);
}

template <typename T>
int launch(const DecodeArgs& a, int n_seq, cudaStream_t stream, int* kernels) {
    const uintptr_t mask = 4 * sizeof(T) - 1;
    const bool vec = a.hd % 4 == 0 && ((uintptr_t)a.k_pages & mask) == 0 && ((uintptr_t)a.v_pages & mask) == 0;
    return vec ? launch_width<T, true>(a, n_seq, stream, kernels) : launch_width<T, false>(a, n_seq, stream, kernels);
}
}  // namespace

// part_o needs n_seq*n_heads*n_splits*head_dim floats and part_ml n_seq*n_heads*n_splits*2
// (both unused when n_splits == 1).
extern "C" int ti_attn_decode_simt(const void* q, long long q_stride, const void* k_pages, const void* v_pages,
                                   const int* page_table, int table_width, int page_size, int ring_rows,
                                   int n_pages, const int* seq_slot, const int* seq_len, int n_seq,
                                   int n_heads, int n_kv_heads, int head_dim, float scale, int window,
                                   int n_splits, void* out, long long o_stride, float* part_o,
                                   float* part_ml, int dtype, cudaStream_t stream) {
    if (n_seq == 0) return 0;
    TI_REQUIRE(n_seq > 0 && n_heads > 0 && n_kv_heads > 0 && n_heads % n_kv_heads == 0, "attention_decode: bad head counts");
    TI_REQUIRE(head_dim > 0 && head_dim <= 512, "attention_decode: head size %d not supported", head_dim);
    TI_REQUIRE(page_size == TILE, "attention_decode: pages of %d positions, this kernel works on %d", page_size, TILE);
    TI_REQUIRE(ring_rows % page_size == 0, "attention_decode: ring of %d rows is not whole pages", ring_rows);
    TI_REQUIRE(window == 0 || ring_rows == 0 || ring_rows >= window, "attention_decode: ring of %d rows is smaller than the window %d", ring_rows, window);
    TI_REQUIRE((n_heads / n_kv_heads) * head_dim <= MAX_OUTPUTS,
               "attention_decode: %d query heads per kv head of size %d exceed this kernel's %d outputs per kv head",
               n_heads / n_kv_heads, head_dim, MAX_OUTPUTS);
    // (kernels/attention.py refuses the same sizes before a model is built.  They are what a form of this kernel with a page of keys
    // and values in shared memory could hold; this one could take more, and no caller has more: heads of up to 449 elements pass)
    TI_REQUIRE(((long long)(n_heads / n_kv_heads) * (head_dim + TILE + 3) + TILE * (2LL * head_dim + 1)) * 4 <= 227 * 1024,
               "attention_decode: %d query heads per kv head of size %d are too many", n_heads / n_kv_heads, head_dim);
    TI_REQUIRE(n_splits >= 1 && n_splits <= 65535 && n_kv_heads <= 65535, "attention_decode: bad split count %d", n_splits);
    TI_REQUIRE(n_splits == 1 || (part_o && part_ml), "attention_decode: split results need scratch memory");
    DecodeArgs a;
    a.q = q; a.q_stride = q_stride; a.k_pages = k_pages; a.v_pages = v_pages; a.page_table = page_table;
    a.table_width = table_width; a.page_size = page_size; a.ring_rows = ring_rows; a.n_pages = n_pages;
    a.seq_slot = seq_slot; a.seq_len = seq_len; a.n_heads = n_heads; a.n_kv_heads = n_kv_heads; a.hd = head_dim;
    a.window = window; a.n_splits = n_splits; a.scale = scale; a.out = out; a.o_stride = o_stride;
    a.part_o = part_o; a.part_ml = part_ml;
    return ti_dispatch_dtype(dtype, [&](auto t) -> int { return launch<decltype(t)>(a, n_seq, stream, nullptr); });
}

// The kernels that ti_attn_decode_simt launches for these sizes (its pages at these addresses).
extern "C" int ti_attn_decode_simt_kernels(const void* k_pages, const void* v_pages, int n_seq, int n_heads, int n_kv_heads, int head_dim,
                                           int n_splits, int dtype, int* kernels) {
    TI_REQUIRE(n_seq > 0 && n_heads > 0 && n_kv_heads > 0 && n_heads % n_kv_heads == 0 && head_dim > 0 && head_dim <= 512 && n_splits >= 1 && kernels,
               "attention_decode: bad sizes");
    DecodeArgs a = {};
    a.k_pages = k_pages; a.v_pages = v_pages; a.n_heads = n_heads; a.n_kv_heads = n_kv_heads; a.hd = head_dim; a.n_splits = n_splits;
    return ti_dispatch_dtype(dtype, [&](auto t) -> int { return launch<decltype(t)>(a, n_seq, nullptr, kernels); });
}

// ---------------------------------------------------------------------------
// The same kernels with their scratch inside the library (see attn_decode_noalloc.h).
// ---------------------------------------------------------------------------
#include "attn_decode_noalloc.h"

// Partial outputs first, then the (maximum, sum) pairs.  In host code this name is only a
// handle for the runtime; the address kernels can use comes from cudaGetSymbolAddress.
static __device__ __align__(256) float g_noalloc_scratch[TI_NOALLOC_SCRATCH_FLOATS];

namespace {
float* g_noalloc_ptr[64] = {nullptr};   // per device, looked up at the first call on it

int noalloc_scratch(float** out) {
    int dev = 0;
    TI_CUDA(cudaGetDevice(&dev));
    TI_REQUIRE(dev >= 0 && dev < 64, "attention_decode (no allocation): device %d out of range", dev);
    if (!g_noalloc_ptr[dev]) {
        float* p = nullptr;
        TI_CUDA(cudaGetSymbolAddress((void**)&p, g_noalloc_scratch));
        TI_REQUIRE(p != nullptr, "attention_decode (no allocation): the scratch array has no device address");
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return 0;
}
}  // namespace

extern "C" int ti_attn_decode_noalloc(const void* q, long long q_stride, const void* k_pages, const void* v_pages,
                                      const int* page_table, int table_width, int page_size, int ring_rows,
                                      int n_pages, const int* seq_slot, const int* seq_len, int n_seq,
                                      int n_heads, int n_kv_heads, int head_dim, float scale, int window,
                                      int n_splits, void* out, long long o_stride, int dtype, cudaStream_t stream) {
    if (n_seq == 0) return 0;
    TI_REQUIRE(n_seq > 0 && n_heads > 0 && head_dim > 0 && n_splits >= 1, "attention_decode (no allocation): bad sizes");
    if (n_splits == 1)      // one split writes its result directly: no scratch is touched, and none is looked up
        return ti_attn_decode_simt(q, q_stride, k_pages, v_pages, page_table, table_width, page_size, ring_rows, n_pages,
                                   seq_slot, seq_len, n_seq, n_heads, n_kv_heads, head_dim, scale, window, 1, out,
                                   o_stride, nullptr, nullptr, dtype, stream);
    const long long need = (long long)n_seq * n_heads * n_splits * (head_dim + 2);
    TI_REQUIRE(need <= (long long)TI_NOALLOC_SCRATCH_FLOATS,
               "attention_decode (no allocation): %d sequences x %d heads x %d splits x head size %d need %lld floats of "
               "scratch, the library holds %d; use fewer splits or sequences per call, or the entry point that takes scratch",
               n_seq, n_heads, n_splits, head_dim, need, TI_NOALLOC_SCRATCH_FLOATS);
    float* scratch = nullptr;
    if (int rc = noalloc_scratch(&scratch)) return rc;
    float* part_o = scratch;
    float* part_ml = scratch + (size_t)n_seq * n_heads * n_splits * head_dim;
    return ti_attn_decode_simt(q, q_stride, k_pages, v_pages, page_table, table_width, page_size, ring_rows, n_pages,
                               seq_slot, seq_len, n_seq, n_heads, n_kv_heads, head_dim, scale, window, n_splits, out,
                               o_stride, part_o, part_ml, dtype, stream);
}
