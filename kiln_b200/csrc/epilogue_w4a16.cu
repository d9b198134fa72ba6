// Small kernels around the W4A16 GEMM's epilogue options.
//
//  * lora_down_kernel: t = scale * x * A^T, the rank-r projection of kiln's LoRA delta
//    (kiln-model/src/lora_loader.rs:213-233: delta = x @ A^T @ B^T * scale).  The GEMM kernel then adds t * B^T to its
//    fp32 sums before rounding, so the delta never exists as a matrix of its own.
//  * finish_kernel: for batch sizes beyond the decode kernel's range, where the options are not fused yet:
//    C = epilogue(base), base being the bf16 GEMM result in the workspace (LoRA delta added, SwiGLU applied).
#include <algorithm>
#include <atomic>

#include "w4a16_async.cuh"
#include "w4a16_common.cuh"

namespace kiln {
namespace {

__device__ __forceinline__ void store_t(void *t, size_t idx, float v, int bf16_out) {
    if (bf16_out)
        static_cast<__nv_bfloat16 *>(t)[idx] = __float2bfloat16(v);
    else
        static_cast<float *>(t)[idx] = v;
}

// Up to four rows of a short K and a small rank: one dot product per warp, fewer steps from the wait to the store than the tiles below have.
// grid = (ceil(r / 8), m), block = 256: warp w of a CTA computes t[row][8 * blockIdx.x + w].
__global__ void __launch_bounds__(256) lora_dot_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ a, float scale,
                                                       int k, int r, void *__restrict__ t, int bf16_out) {
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = blockIdx.y, j = blockIdx.x * 8 + warp;
    pdl_wait();  // x may be the previous kernel's output, and so may the adapter; t may still be read by it
    if (j >= r) return;
    const uint4 *xr = reinterpret_cast<const uint4 *>(x + static_cast<size_t>(row) * k);
    const uint4 *ar = reinterpret_cast<const uint4 *>(a + static_cast<size_t>(j) * k);
    float sum = 0.f;
    for (int i = lane; i < k / 8; i += 32) {
        const uint4 xv = ld_cg_v4(xr + i), av = ld_cg_v4(ar + i);
        const uint32_t xs[4] = {xv.x, xv.y, xv.z, xv.w}, as[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            sum += __uint_as_float(xs[e] << 16) * __uint_as_float(as[e] << 16) +
                   __uint_as_float(xs[e] & 0xFFFF0000u) * __uint_as_float(as[e] & 0xFFFF0000u);
    }
#pragma unroll
    for (int sh = 16; sh >= 1; sh >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sh);
    if (lane == 0) store_t(t, static_cast<size_t>(row) * r + j, sum * scale, bf16_out);
}

// Otherwise a small tensor-core GEMM, K split over the CTAs of a cluster and, for few rows, over the warps of a CTA.
//
// Bound: latency.  The operands are a few hundred KB (x 37 x 9216 and A 64 x 9216: 1.9 MB), so what counts is how many SMs load
// them at once and how short the chain from the grid-dependency wait to the last store is.  A lane loads 16 contiguous bytes of
// a row of x and of a row of A and uses them as the K slots {2qd, 2qd+1, 2qd+8, 2qd+9} of two m16n8k16 MMAs: the same K
// permutation on both sides, so no shared-memory staging and no ldmatrix.
// A CTA has WM row tiles of 16 and 8 / WM parts of its K range, one (row tile, part) per warp, and 8 NT adapter rows.  Small tiles
// nearly always (many CTAs, short chains: 64 rows, 9216 -> 2560 with its GEMM 21 -> 13 us against tiles of 64 x 32), large ones for
// very many rows (x is read once per 8 NT adapter rows).  The parts meet in shared memory; the cluster's partial tiles are pushed to
// the rank that owns the elements (st.async, counted on its barrier; two cluster barriers around reads took 0.7 us more; of the large tiles
// 16 bytes a push, with 4 bytes 2100 rows rank 64 512 -> 1024 16.9 -> 19.8 us) and added there in rank order: the result does not depend on timing.
// AHEAD: the first blocks of a warp whose loads are all in flight at once, and the adapter, cold in HBM in a model of many layers, is asked
// into L2 before the grid-dependency wait.  (Reading it before the wait would be another 2 % faster, but a caller may have written it: so
// no load of it is one that the compiler may move, as __ldg is.)
// By itself, us: 37 rows rank 64 K = 2560 3.0 -> 2.3, K = 9216 4.0 -> 3.0.  Against dot products, a warp each: 4 rows rank 64 K = 2560
// 2.35 -> 1.96, K = 9216 5.35 -> 2.5.  Four layers with it: 8 rows 254 -> 188, 37 rows 218 -> 188, 128 rows 301 -> 275.
template <int NT>
__device__ __forceinline__ void lora_mma_block(const uint4 &u, const uint4 &v, const uint4 (&w)[NT], float (&acc)[NT][4]) {
    const uint32_t lo[4] = {u.x, v.x, u.y, v.y}, hi[4] = {u.z, v.z, u.w, v.w};
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        mma_bf16_16816(acc[t], lo, w[t].x, w[t].y);
        mma_bf16_16816(acc[t], hi, w[t].z, w[t].w);
    }
}
template <int NT>
__device__ __forceinline__ void lora_mma_range(const uint4 *x0, const uint4 *x1, const uint4 *const (&a)[NT], int b0, int b1, float (&acc)[NT][4]) {
#pragma unroll 4
    for (int b = b0; b < b1; ++b) {
        const uint4 u = ld_cg_v4(x0 + b * 4), v = ld_cg_v4(x1 + b * 4);
        const uint32_t lo[4] = {u.x, v.x, u.y, v.y}, hi[4] = {u.z, v.z, u.w, v.w};
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const uint4 w = ld_v4(a[t] + b * 4);
            mma_bf16_16816(acc[t], lo, w.x, w.y);
            mma_bf16_16816(acc[t], hi, w.z, w.w);
        }
    }
}

// grid = (cluster size, ceil(r / (8 NT)), ceil(m / (16 WM))), cluster = (cluster size, 1, 1), block = 256.
// (bf16_out: t is a bf16 [m, r] matrix, the form the tcgen05 kernels read as an operand tile; fp32 otherwise.  test_missing: bytes that are
// announced to the exchange but never pushed.  ALONE: one CTA has a tile's whole K, and its threads store the sums of its parts at once.)
template <int WM, int NT>
constexpr int lora_smem() {
    return (8 * 16 * 8 * NT + 16 * WM * 8 * NT + 32) * static_cast<int>(sizeof(float));
}
template <int WM, int NT, int AHEAD, bool ALONE>
__global__ void __launch_bounds__(256) lora_down_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ a, float scale,
                                                        int m, int k, int r, void *__restrict__ t, int bf16_out, uint32_t *status,
                                                        unsigned long long wait_limit_ns, uint32_t test_missing, bool prefetch) {
    constexpr int kCols = 8 * NT, kRows = 16 * WM, kParts = 8 / WM, kTile = kRows * kCols;
    extern __shared__ __align__(16) float parts[];  // [kParts][kRows][kCols], then what the ranks push
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane >> 2, qd = lane & 3;
    const int wm = warp % WM, part = warp / WM;
    const int rank = ALONE ? 0 : blockIdx.x, size = ALONE ? 1 : gridDim.x;
    // A rank of the cluster owns `each` elements of the tile, the last ones fewer or none.  (armed before the wait; that every CTA runs is
    // checked before the first push)
    constexpr int kVec = kParts == 1 ? 4 : 1;  // floats of a push
    const int each = (kTile / kVec + size - 1) / size * kVec, own = max(0, min(each, kTile - rank * each));
    __shared__ __align__(8) unsigned long long exchange;
    __shared__ uint32_t gave_up;
    const uint32_t bar = smem_u32(&exchange);
    if (size > 1) {
        if (threadIdx.x == 0) {
            gave_up = 0;
            mbar_init(bar, 1);
            mbar_init_fence();
            mbar_arrive_expect_tx(bar, static_cast<uint32_t>((size - 1) * own) * 4u + test_missing);
        }
        __syncthreads();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    const int row0 = blockIdx.z * kRows + wm * 16, col0 = blockIdx.y * kCols;
    const int blocks = k / 32, slices = size * kParts, slice = rank * kParts + part;
    const int b0 = static_cast<int>(static_cast<long long>(blocks) * slice / slices), b1 = static_cast<int>(static_cast<long long>(blocks) * (slice + 1) / slices);
    float acc[NT][4];
    const uint4 *ap[NT];  // (rows past r or m repeat the last one: their sums are dropped)
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
        ap[i] = reinterpret_cast<const uint4 *>(a + static_cast<size_t>(min(col0 + 8 * i + c, r - 1)) * k) + qd;
    }
    const uint4 *x0 = reinterpret_cast<const uint4 *>(x + static_cast<size_t>(min(row0 + c, m - 1)) * k) + qd;
    const uint4 *x1 = reinterpret_cast<const uint4 *>(x + static_cast<size_t>(min(row0 + c + 8, m - 1)) * k) + qd;
    // The adapter's rows come to L2 before the wait, and are read after it: a kernel before this one may have written them.
    for (int b = b0; (AHEAD > 0 || (ALONE && prefetch)) && b < b1; ++b)
#pragma unroll
        for (int t = 0; t < NT; ++t) asm volatile("prefetch.global.L2 [%0];" ::"l"(ap[t] + b * 4));
    pdl_wait();  // x may be the previous kernel's output; t may still be read by it
    uint4 w[AHEAD + 1][NT], u[AHEAD + 1], v[AHEAD + 1];  // (the first blocks' loads are all in flight at once)
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
        if (b0 + i < b1) {
            u[i] = ld_cg_v4(x0 + (b0 + i) * 4), v[i] = ld_cg_v4(x1 + (b0 + i) * 4);
#pragma unroll
            for (int t = 0; t < NT; ++t) w[i][t] = ld_cg_v4(ap[t] + (b0 + i) * 4);
        }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
        if (b0 + i < b1) lora_mma_block<NT>(u[i], v[i], w[i], acc);
    lora_mma_range<NT>(x0, x1, ap, b0 + AHEAD, b1, acc);
    float *mine = parts + part * kTile + wm * 16 * kCols;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        *reinterpret_cast<float2 *>(mine + c * kCols + 8 * i + 2 * qd) = make_float2(acc[i][0], acc[i][1]);
        *reinterpret_cast<float2 *>(mine + (c + 8) * kCols + 8 * i + 2 * qd) = make_float2(acc[i][2], acc[i][3]);
    }
    __syncthreads();
    if (ALONE) {
        for (int e = threadIdx.x; e < kTile; e += 256) {
            float v = parts[e];
#pragma unroll
            for (int q = 1; q < kParts; ++q) v += parts[q * kTile + e];
            const int row = blockIdx.z * kRows + e / kCols, col = col0 + e % kCols;
            if (row < m && col < r) store_t(t, static_cast<size_t>(row) * r + col, v * scale, bf16_out);
        }
        return;
    }
    // Every CTA sums its parts and pushes each rank its share (counted on that rank's barrier), the owner adds the shares in rank order.
    float *recv = parts + kParts * kTile;  // [rank][each]
    if (size > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int e = kVec * threadIdx.x; e < kTile; e += kVec * 256) {
        const int owner = e / each;
        const uint32_t slot = smem_u32(recv + rank * each + e - owner * each);
        if constexpr (kVec == 4) {
            const float4 v = *reinterpret_cast<const float4 *>(parts + e);
            if (owner == rank)
                asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(slot), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
            else
                asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(map_to_cta(slot, owner)),
                             "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(map_to_cta(bar, owner))
                             : "memory");
        } else {
            float v = parts[e];
#pragma unroll
            for (int q = 1; q < kParts; ++q) v += parts[q * kTile + e];
            if (owner == rank)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(slot), "f"(v) : "memory");
            else
                asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(map_to_cta(slot, owner)), "f"(v),
                             "r"(map_to_cta(bar, owner))
                             : "memory");
        }
    }
    __syncthreads();
    if (size > 1 && !mbar_wait(bar, 0, &gave_up, status, 0xC00u, wait_limit_ns)) {
        mbar_wait_quiet(bar, 0, peers_limit_ns(wait_limit_ns));  // (a peer pushes into this CTA until it is through)
        return;
    }
    for (int i = threadIdx.x; i < own; i += 256) {
        float v = recv[i];
        for (int q = 1; q < size; ++q) v += recv[q * each + i];
        const int e = rank * each + i, row = blockIdx.z * kRows + e / kCols, col = col0 + e % kCols;
        if (row < m && col < r) store_t(t, static_cast<size_t>(row) * r + col, v * scale, bf16_out);
    }
}

__device__ __forceinline__ float lora_dot(const float *t, const __nv_bfloat16 *b, int r) {
    float d = 0.f;
    for (int j = 0; j < r; j += 2) {
        const uint32_t w = *reinterpret_cast<const uint32_t *>(b + j);
        d += t[j] * __uint_as_float(w << 16) + t[j + 1] * __uint_as_float(w & 0xFFFF0000u);
    }
    return d;
}

// One thread per output element of C ([m, n], or [m, n/2] with SwiGLU).
__global__ void __launch_bounds__(256) finish_kernel(const __nv_bfloat16 *__restrict__ base, __nv_bfloat16 *__restrict__ c, int m,
                                                     int n, const float *__restrict__ t, const __nv_bfloat16 *__restrict__ lb, int r,
                                                     int swiglu) {
    const int n_out = swiglu ? n / 2 : n;
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<size_t>(m) * n_out) return;
    const int row = static_cast<int>(idx / n_out), oc = static_cast<int>(idx - static_cast<size_t>(row) * n_out);
    auto value = [&](int col) {
        float v = __bfloat162float(base[static_cast<size_t>(row) * n + col]);
        if (r) v += lora_dot(t + static_cast<size_t>(row) * r, lb + static_cast<size_t>(col) * r, r);
        return v;
    };
    if (!swiglu) {
        c[idx] = __float2bfloat16(value(oc));
    } else {
        const int cg = (oc >> 5) * 64 + (oc & 31);  // gate column; its up column is 32 further
        const float g = value(cg), u = value(cg + 32);
        c[idx] = __float2bfloat16(g / (1.f + __expf(-g)) * u);
    }
}

}  // namespace

int launch_lora_down(const void *x, const void *lora_a, float scale, int m, int k, int r, void *t, int bf16_out, cudaStream_t stream) {
    const auto *xp = static_cast<const __nv_bfloat16 *>(x), *ap = static_cast<const __nv_bfloat16 *>(lora_a);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 1;
    // Dot products or tiles (us with the GEMM, rank 16, K = 640 / 1024 / 1280 / 1536 -> 512: one row 4.3 / 4.3 / 4.5 / 4.5 against 4.4 / 4.4 / 4.7 /
    // 4.5, four rows 4.4 / 4.3 / 4.6 / 4.7 against 4.4 / 4.4 / 4.9 / 4.6; four rows rank 64 1280 -> 2560 6.8 against 6.4).
    if (m <= 4 && m * r <= 128 && k <= 1280) {
        cfg.gridDim = dim3((r + 7) / 8, m);
        note_launch();
        return record_cuda_error(cudaLaunchKernelEx(&cfg, lora_dot_kernel, xp, ap, scale, k, r, t, bf16_out));
    }
    // Rows and adapter rows of a CTA: 16 x 16, or 128 x 64 for more than 1024 rows of a large rank, where reading x once per 16
    // adapter rows costs more than the longer chains of large tiles (2048 x 9216, rank 64, with its GEMM: 118 / 114 us; 1024 rows: 65 / 83).
    const int wm = m > 1024 && r > 32 ? 8 : 1, rows = 16 * wm, cols = wm == 1 ? 16 : 64, parts = 8 / wm;
    const int row_tiles = (m + rows - 1) / rows, col_tiles = (r + cols - 1) / cols;
    if (row_tiles > 65535) return KILN_W4A16_ERR_KERN_SHAPE;
    const int tiles = row_tiles * col_tiles;
    // K is split over as many CTAs as the tiles leave room for (four small ones to an SM: 768 x 9216, rank 64 57.6 -> 51.3 us against
    // one), while a warp keeps at least two 32-deep blocks.  Of the large ones, one to an SM for their 142 registers, all clusters have to
    // fit at once: not all SMs are in clusters of eight (2100 rows rank 64, 17 clusters where 15 of eight fit: 9216 -> 2560 128 us, six to a cluster 110).
    int size = std::min(8, std::max(1, (wm == 1 ? 4 : 1) * device_sm_count() / tiles));
    while (wm != 1 && size > 1 && smallm_clusters(size) < tiles) --size;
    size = std::max(1, std::min(size, k / 32 / (2 * parts)));
    cfg.gridDim = dim3(size, col_tiles, row_tiles);
    cfg.dynamicSmemBytes = wm == 1 ? lora_smem<1, 2>() : lora_smem<8, 8>();
    if (size > 1) {
        attrs[1].id = cudaLaunchAttributeClusterDimension;
        attrs[1].val.clusterDim.x = size;
        attrs[1].val.clusterDim.y = 1;
        attrs[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    uint32_t *status = size > 1 ? device_status_word() : nullptr;  // (of the exchange's wait)
    if (size > 1 && !status) return KILN_W4A16_ERR_CUDA;
    // The look-ahead takes 76 registers against 62, three CTAs to an SM: only where all are resident either way.  A projection whose
    // tiles have one CTA each has a short K and little to look ahead to, and its CTAs may have to start on the few SMs that the GEMM before
    // leaves free (256 rows rank 64 K = 512: 64 CTAs beside 128 of a GEMM; four to an SM 7.6 us with the next GEMM, three 8.6).  There it is for
    // a few tiles alone (8 x 512 -> 2560 rank 64 5.4 -> 5.1); the prefetch, which needs no register, stays.
    const bool few = size * tiles <= 3 * device_sm_count(), alone = size == 1;
    const auto kernel = wm != 1 ? lora_down_kernel<8, 8, 0, false>
                        : alone ? (tiles <= 8 ? lora_down_kernel<1, 2, 2, true> : lora_down_kernel<1, 2, 0, true>)
                                : (few ? lora_down_kernel<1, 2, 2, false> : lora_down_kernel<1, 2, 0, false>);
    if (wm != 1) {  // (its shared memory is beyond what a launch may have unasked)
        static std::atomic<bool> asked[64] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 64 || !asked[dev].load(std::memory_order_acquire)) {
            if (int rc = record_cuda_error(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lora_smem<8, 8>()))) return rc;
            if (dev < 64) asked[dev].store(true, std::memory_order_release);
        }
    }
    note_launch();
    const bool test = test_drop_a_load() == kTestShortExchange;  // (gives up well before a kernel that waits for this one does)
    return record_cuda_error(cudaLaunchKernelEx(&cfg, kernel, xp, ap, scale, m, k, r, t, bf16_out, status, current_wait_limit_ns() / (test ? 4 : 1), test ? 4u : 0u, wm == 1 && few));
}

int launch_finish(const void *base, void *c, int m, int n, const float *t, const void *lora_b, int r, int swiglu,
                  cudaStream_t stream) {
    const size_t total = static_cast<size_t>(m) * (swiglu ? n / 2 : n);
    const unsigned blocks = static_cast<unsigned>((total + 255) / 256);
    note_launch();
    finish_kernel<<<blocks, 256, 0, stream>>>(static_cast<const __nv_bfloat16 *>(base), static_cast<__nv_bfloat16 *>(c), m, n, t,
                                              static_cast<const __nv_bfloat16 *>(lora_b), r, swiglu);
    return record_cuda_error(cudaGetLastError());
}

}  // namespace kiln
