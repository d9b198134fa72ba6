// Native weight repacker: symmetric int4 quantiser + Marlin tile/fragment packing + scale
// reordering, on the host (multi-threaded inside one matrix) and on the device.
//
// Output is bit-identical to kiln's `pack::quantize_and_pack`
// (kiln-marlin-gemm/src/lib.rs:370-491) but computed directly: no k*n temporaries and no
// 1024-entry gather; every packed word is assembled from the eight weights the consuming lane
// owns (see the layout note in w4a16_common.cuh).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <thread>
#include <vector>

#include "pack_host.h"
#include "w4a16_common.cuh"

namespace kiln {
namespace {

constexpr int kMaxQ = 15;    // kiln-marlin-gemm/src/lib.rs:288
constexpr int kQOffset = 8;  // kiln-marlin-gemm/src/lib.rs:289

// (row, col) offsets of nibble i inside a lane's word, relative to (2*(lane%4), lane/4)
__host__ __device__ inline int nib_dr(int i) { return ((i >> 2) & 1) + 8 * (i & 1); }
__host__ __device__ inline int nib_dc(int i) { return 8 * ((i >> 1) & 1); }

// position of natural column `col` in the grouped scale order (lib.rs:333-341):
// out[8i + j] = in[i + 8j] within each 64 columns.
__host__ __device__ inline int scale_group_pos(int col) {
    const int c64 = col & 63;
    return (col & ~63) + 8 * (c64 & 7) + (c64 >> 3);
}

__host__ __device__ inline int quantize_one(float w, float s) {
    // lib.rs:422-423: f32 divide, round half away from zero, +8, clamp to [0,15]
    float r = roundf(w / s);
    // Rust `as i32` saturates and maps NaN to 0
    int raw;
    if (r != r) raw = 0;
    else if (r >= 2147483648.0f) raw = 2147483647;
    else if (r <= -2147483648.0f) raw = -2147483647 - 1;
    else raw = static_cast<int>(r);
    long long shifted = static_cast<long long>(raw) + kQOffset;
    if (shifted < 0) shifted = 0;
    if (shifted > kMaxQ) shifted = kMaxQ;
    return static_cast<int>(shifted);
}

// ---- host ---------------------------------------------------------------------------------

inline uint16_t host_f32_to_f16_bits(float f) {
    const __half h = __float2half_rn(f);  // host path of cuda_fp16: IEEE round-to-nearest-even
    uint16_t b;
    std::memcpy(&b, &h, 2);
    return b;
}
inline float host_f16_bits_to_f32(uint16_t b) {
    __half h;
    std::memcpy(&h, &b, 2);
    return __half2float(h);
}

template <class F>
void parallel_chunks(int chunks, int num_threads, F &&fn) {
    int nt = num_threads > 0 ? num_threads : static_cast<int>(std::thread::hardware_concurrency());
    if (nt < 1) nt = 1;
    nt = std::min(nt, chunks);
    if (nt <= 1) {
        for (int c = 0; c < chunks; ++c) fn(c);
        return;
    }
    std::vector<std::thread> pool;
    pool.reserve(nt);
    for (int t = 0; t < nt; ++t)
        pool.emplace_back([=, &fn] {
            for (int c = t; c < chunks; c += nt) fn(c);
        });
    for (auto &th : pool) th.join();
}

// fn(i) for i in [0, count), handed out one at a time (blocks differ in what the memory system has to do for them).
template <class F>
void parallel_units(int count, int num_threads, F &&fn) {
    int nt = num_threads > 0 ? num_threads : static_cast<int>(std::thread::hardware_concurrency());
    nt = std::max(1, std::min(nt, count));
    std::atomic<int> next{0};
    auto work = [&] {
        for (int i; (i = next.fetch_add(1, std::memory_order_relaxed)) < count;) fn(i);
    };
    std::vector<std::thread> pool;
    pool.reserve(nt - 1);
    for (int t = 1; t < nt; ++t) pool.emplace_back(work);
    work();
    for (auto &th : pool) th.join();
}

// Packs one 64-column chunk of a 16-row K-tile whose nibbles are in nib[16][64].
inline void pack_tile_host(const uint8_t (*nib)[64], int32_t *out128) {
    for (int lane = 0; lane < 32; ++lane) {
        const int r0 = 2 * (lane & 3), c = lane >> 2;
        for (int j = 0; j < 4; ++j) {
            uint32_t word = 0;
            for (int i = 0; i < 8; ++i)
                word |= static_cast<uint32_t>(nib[r0 + nib_dr(i)][16 * j + c + nib_dc(i)] & 0xF) << (4 * i);
            out128[lane * 4 + j] = static_cast<int32_t>(word);
        }
    }
}

int shape_ok(int k, int n, int groupsize, int *g_out) {
    if (k <= 0 || n <= 0) return KILN_W4A16_ERR_ARG;
    if (k % 128 != 0 || n % 256 != 0) return KILN_W4A16_ERR_PROB_SHAPE;  // lib.rs:377-378
    const int g = groupsize == -1 ? k : groupsize;
    if (g <= 0 || g % 16 != 0 || k % g != 0) return KILN_W4A16_ERR_PROB_SHAPE;  // lib.rs:385
    *g_out = g;
    return 0;
}

}  // namespace
}  // namespace kiln

using namespace kiln;

extern "C" {

void kiln_w4a16_build_weight_perm(int32_t *out) {
    // Derived from the fragment ownership rather than the reference's list construction:
    // output element e = word*8 + nibble of a 1024-element chunk takes the tiled element
    // 256*j + 16*row + col.
    for (int lane = 0; lane < 32; ++lane)
        for (int j = 0; j < 4; ++j)
            for (int i = 0; i < 8; ++i) {
                const int row = 2 * (lane & 3) + nib_dr(i), col = (lane >> 2) + nib_dc(i);
                out[(lane * 4 + j) * 8 + i] = 256 * j + 16 * row + col;
            }
}

void kiln_w4a16_build_scale_perm(int32_t *out) {
    for (int col = 0; col < 64; ++col) out[scale_group_pos(col)] = col;
}

void kiln_w4a16_build_scale_perm_single(int32_t *out) {
    for (int col = 0; col < 32; ++col) out[scale_single_pos(col)] = col;
}

kiln_w4a16_status_t kiln_w4a16_quantize_and_pack_host(const float *weight, int k, int n, int groupsize,
                                                      int32_t *b_packed, uint16_t *scales_f16,
                                                      float *dequant, int num_threads) {
    int g = 0;
    if (int rc = shape_ok(k, n, groupsize, &g)) return rc;
    if (!weight || !b_packed || !scales_f16) return KILN_W4A16_ERR_ARG;
    const int chunks = n / 64, ktiles_per_group = g / 16, num_groups = k / g;
    const size_t row_words = static_cast<size_t>(2) * n;
    if (pack_host_vectorised()) {
        int pos[64];
        for (int c = 0; c < 64; ++c) pos[c] = groupsize == -1 ? scale_single_pos(c) : scale_group_pos(c);
        const int col_blocks = n / kHostBlockCols;  // (n is a multiple of 256)
        parallel_units(col_blocks * num_groups, num_threads, [&](int u) {
            const int grp = u / col_blocks, cb = u - grp * col_blocks;
            pack_host_block(weight, n, grp * g, g, cb * kHostBlockCols, kHostBlockCols, b_packed, scales_f16 + static_cast<size_t>(grp) * n, pos,
                            dequant);
        });
        return KILN_W4A16_OK;
    }
    parallel_chunks(chunks, num_threads, [&](int ch) {
        const int c0 = ch * 64;
        float s[64];
        uint8_t nib[16][64];
        for (int grp = 0; grp < num_groups; ++grp) {
            // 1) scales for 64 columns of this group (lib.rs:393-413)
            float mx[64];
            for (int c = 0; c < 64; ++c) mx[c] = 0.f;
            for (int r = 0; r < g; ++r) {
                const float *wr = weight + static_cast<size_t>(grp * g + r) * n + c0;
                for (int c = 0; c < 64; ++c) {
                    const float v = std::fabs(wr[c]);
                    if (v > mx[c]) mx[c] = v;
                }
            }
            for (int c = 0; c < 64; ++c) {
                if (mx[c] == 0.f) mx[c] = 1.f;
                const uint16_t hb = host_f32_to_f16_bits((2.0f * mx[c]) / static_cast<float>(kMaxQ));
                s[c] = host_f16_bits_to_f32(hb);
                const int pos = groupsize == -1 ? scale_single_pos(c0 + c) : scale_group_pos(c0 + c);
                scales_f16[static_cast<size_t>(grp) * n + pos] = hb;
            }
            // 2-4) quantise and pack, one 16-row tile at a time
            for (int kt = 0; kt < ktiles_per_group; ++kt) {
                const int kb = grp * ktiles_per_group + kt;
                for (int r = 0; r < 16; ++r) {
                    const size_t off = static_cast<size_t>(kb * 16 + r) * n + c0;
                    for (int c = 0; c < 64; ++c) {
                        const int qv = quantize_one(weight[off + c], s[c]);
                        nib[r][c] = static_cast<uint8_t>(qv);
                        if (dequant) dequant[off + c] = static_cast<float>(qv - kQOffset) * s[c];
                    }
                }
                pack_tile_host(nib, b_packed + static_cast<size_t>(kb) * row_words + ch * 128);
            }
        }
    });
    return KILN_W4A16_OK;
}

kiln_w4a16_status_t kiln_w4a16_repack_host(const uint8_t *q, const uint16_t *scales, int k, int n,
                                           int groupsize, int32_t *b_packed, uint16_t *scales_perm,
                                           int num_threads) {
    int g = 0;
    if (k <= 0 || n <= 0) return KILN_W4A16_ERR_ARG;
    if (k % 16 != 0 || n % 64 != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    g = groupsize == -1 ? k : groupsize;
    if (g <= 0 || k % g != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    if (!q || !scales || !b_packed || !scales_perm) return KILN_W4A16_ERR_ARG;
    const int chunks = n / 64, num_groups = k / g;
    const size_t row_words = static_cast<size_t>(2) * n;
    parallel_chunks(chunks, num_threads, [&](int ch) {
        const int c0 = ch * 64;
        uint8_t nib[16][64];
        for (int kb = 0; kb < k / 16; ++kb) {
            for (int r = 0; r < 16; ++r)
                std::memcpy(nib[r], q + static_cast<size_t>(kb * 16 + r) * n + c0, 64);
            pack_tile_host(nib, b_packed + static_cast<size_t>(kb) * row_words + ch * 128);
        }
        for (int grp = 0; grp < num_groups; ++grp)
            for (int c = 0; c < 64; ++c) {
                const int pos = groupsize == -1 ? scale_single_pos(c0 + c) : scale_group_pos(c0 + c);
                scales_perm[static_cast<size_t>(grp) * n + pos] = scales[static_cast<size_t>(grp) * n + c0 + c];
            }
    });
    return KILN_W4A16_OK;
}


// GPTQ checkpoint tensors -> W4A16 layout without dequantising (kiln dequantises GPTQ to bf16 on the CPU,
// crates/kiln-model/src/quantized.rs:70-163, and the Marlin path then re-quantises that).  qweight int32 [k/8, n]
// (nibble i of a word = input row 8*row + i), qzeros int32 [k/g, n/8] (nibble j of a word = output column 8*col + j),
// scales fp16 [k/g, n].  GPTQ's value is (nibble - zero) * scale, this format's is (nibble - 8) * scale: the repack is
// exact when every zero-point is 8, and refused (KILN_W4A16_ERR_PROB_SHAPE, *asymmetric = how many are not) otherwise.
kiln_w4a16_status_t kiln_w4a16_repack_gptq_host(const int32_t *qweight, const int32_t *qzeros, const uint16_t *scales,
                                                int k, int n, int groupsize, int32_t *b_packed, uint16_t *scales_perm,
                                                uint32_t *asymmetric, int num_threads) {
    if (k <= 0 || n <= 0) return KILN_W4A16_ERR_ARG;
    if (k % 16 != 0 || n % 64 != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    const int g = groupsize == -1 ? k : groupsize;
    if (g <= 0 || k % g != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    if (!qweight || !qzeros || !scales || !b_packed || !scales_perm) return KILN_W4A16_ERR_ARG;
    const int num_groups = k / g;
    uint32_t bad = 0;
    for (size_t i = 0; i < static_cast<size_t>(num_groups) * (n / 8); ++i) {
        const uint32_t z = static_cast<uint32_t>(qzeros[i]);
        for (int j = 0; j < 8; ++j) bad += ((z >> (4 * j)) & 0xF) != static_cast<uint32_t>(kQOffset);
    }
    if (asymmetric) *asymmetric = bad;
    if (bad) return KILN_W4A16_ERR_PROB_SHAPE;
    const int chunks = n / 64;
    const size_t row_words = static_cast<size_t>(2) * n;
    parallel_chunks(chunks, num_threads, [&](int ch) {
        const int c0 = ch * 64;
        uint8_t nib[16][64];
        for (int kb = 0; kb < k / 16; ++kb) {
            for (int r = 0; r < 16; ++r) {
                const int32_t *row = qweight + static_cast<size_t>((kb * 16 + r) / 8) * n + c0;
                const int sh = 4 * ((kb * 16 + r) % 8);
                for (int c = 0; c < 64; ++c) nib[r][c] = static_cast<uint8_t>((static_cast<uint32_t>(row[c]) >> sh) & 0xF);
            }
            pack_tile_host(nib, b_packed + static_cast<size_t>(kb) * row_words + ch * 128);
        }
        for (int grp = 0; grp < num_groups; ++grp)
            for (int c = 0; c < 64; ++c) {
                const int pos = groupsize == -1 ? scale_single_pos(c0 + c) : scale_group_pos(c0 + c);
                scales_perm[static_cast<size_t>(grp) * n + pos] = scales[static_cast<size_t>(grp) * n + c0 + c];
            }
    });
    return KILN_W4A16_OK;
}

}  // extern "C"

// ---- device -------------------------------------------------------------------------------
namespace kiln {
namespace {

template <bool BF16>
__device__ __forceinline__ float load_w(const void *w, size_t idx) {
    if (BF16) return __bfloat162float(static_cast<const __nv_bfloat16 *>(w)[idx]);
    return static_cast<const float *>(w)[idx];
}

// One thread per column: max |w| over the group, f16 scale, written at its Marlin position.
// grid = (n/128, num_groups), block = 128.  `scales_nat` keeps the natural order for kernel 2.
template <bool BF16>
__global__ void pack_scales_kernel(const void *w, int n, int g, int per_column, uint16_t *scales_perm,
                                   float *scales_nat) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    const int grp = blockIdx.y;
    if (col >= n) return;
    float mx = 0.f;
    for (int r = 0; r < g; ++r) mx = fmaxf(mx, fabsf(load_w<BF16>(w, static_cast<size_t>(grp * g + r) * n + col)));
    if (mx == 0.f) mx = 1.f;
    const __half h = __float2half_rn(__fdiv_rn(2.0f * mx, 15.0f));
    const int pos = per_column ? scale_single_pos(col) : scale_group_pos(col);
    scales_perm[static_cast<size_t>(grp) * n + pos] = __half_as_ushort(h);
    scales_nat[static_cast<size_t>(grp) * n + col] = __half2float(h);
}

// One block per (16-row K-tile, 64-column chunk); thread (lane, j) assembles one packed word.
// grid = (n/64, k/16), block = 128.
template <bool BF16>
__global__ void pack_words_kernel(const void *w, int n, int g, const float *scales_nat, int32_t *b_packed,
                                  float *dequant) {
    __shared__ uint8_t nib[16][64];
    const int ch = blockIdx.x, kb = blockIdx.y, tid = threadIdx.x;
    const int grp = (kb * 16) / g;
    for (int e = tid; e < 16 * 64; e += blockDim.x) {
        const int r = e >> 6, c = e & 63;
        const size_t off = static_cast<size_t>(kb * 16 + r) * n + ch * 64 + c;
        const float s = scales_nat[static_cast<size_t>(grp) * n + ch * 64 + c];
        const float wv = load_w<BF16>(w, off);
        const int qv = quantize_one(wv, s);
        nib[r][c] = static_cast<uint8_t>(qv);
        if (dequant) dequant[off] = __fmul_rn(static_cast<float>(qv - kQOffset), s);
    }
    __syncthreads();
    const int lane = tid >> 2, j = tid & 3;
    const int r0 = 2 * (lane & 3), c = lane >> 2;
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        word |= static_cast<uint32_t>(nib[r0 + nib_dr(i)][16 * j + c + nib_dc(i)] & 0xF) << (4 * i);
    b_packed[static_cast<size_t>(kb) * 2 * n + ch * 128 + tid] = static_cast<int32_t>(word);
}

// ---- one pass over the weights, grouped (128 rows per scale) or per column --------------------------------------------
//
// One block per 128 rows x 64 columns.  A thread holds rows 2qd, 2qd+1, 2qd+8, 2qd+9 of one 16-row tile and eight neighbouring
// columns: half of the eight weights of each of eight packed words, whose other half (columns c + 8) is the neighbouring
// lane's.  So the weights go from 16-byte loads (128 contiguous bytes per row and eight lanes) to packed words in registers,
// with one shuffle per word; shared memory only carries the column maxima and the scales.
//
// Bound: HBM once the arithmetic is small.  With the IEEE division and roundf for every weight (about 30 instructions) the
// arithmetic took 40 us of a 2560 x 9216 weight's 44.  Here w / s is w * (1 / s): its error is below 4 units in the last place,
// 4e-6 at the largest quotient of 7.51, so rounding it to nearest gives what rounding the correctly rounded quotient half away
// from zero gives, unless it lies within 1e-5 of a tie.  One bf16 weight in a thousand does (few bits over few bits); those are
// divided exactly (quantize_near_tie).  NaN, and columns whose scale is zero, subnormal or infinite, take quantize_one.
// Measured: 2560 x 9216 bf16 44.8 -> 20.7 us per call (18 instructions per weight are what is left: the integer pipe), f32 45.2
// -> 24.7; per column, whose first version walked each column with one thread, 261 -> 31.

constexpr float kRoundMagic = 12582912.f;  // 1.5 * 2^23: adding it rounds to nearest, the integer sits in the low mantissa bits
constexpr uint32_t kRoundMagicBits = 0x4B400000u;

// two floats per instruction (sm_100)
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {  // NaN if either is
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

struct ColumnScale {
    float s, inv;  // inv = 0: no fast path for this column
};
__device__ __forceinline__ __half scale_of_max(float mx) {
    if (mx == 0.f) mx = 1.f;
    return __float2half_rn(__fdiv_rn(2.0f * mx, 15.0f));
}
__device__ __forceinline__ ColumnScale column_scale(__half h) {
    const float s = __half2float(h);
    return {s, s >= 6.2e-5f && s <= 65504.f ? __fdiv_rn(1.0f, s) : 0.f};
}

// The quantised weight where w / s may be a tie, without a division: Markstein's theorem (IBM J. Res. Dev. 34, 1990) makes
// q + (w - q s) * inv the correctly rounded quotient when inv is the correctly rounded 1 / s and q is within one unit in the
// last place, which the first of the two corrections sees to (s comes from fp16, so its mantissa is not all ones).
__device__ __forceinline__ uint32_t quantize_near_tie(float w, ColumnScale cs) {
    float q = w * cs.inv;
    q = fmaf(fmaf(-q, cs.s, w), cs.inv, q);
    q = fmaf(fmaf(-q, cs.s, w), cs.inv, q);
    float r = (q + kRoundMagic) - kRoundMagic;
    if (fabsf(q - r) == 0.5f) r = q + copysignf(0.5f, q);  // half away from zero
    return __float_as_uint(fminf(r, 7.f) + (kRoundMagic + 8.f)) & 0xFu;
}

// Four rows x eight columns of one thread, kept as they were loaded (bf16: two to a register, so that six blocks fit an SM).
template <bool BF16>
struct Rows {
    uint32_t x[4][BF16 ? 4 : 8];
    __device__ __forceinline__ void load(const void *w, size_t off, int n) {
        constexpr int kRow[4] = {0, 1, 8, 9};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint4 *p = reinterpret_cast<const uint4 *>(static_cast<const uint8_t *>(w) + (off + static_cast<size_t>(kRow[r]) * n) * (BF16 ? 2 : 4));
#pragma unroll
            for (int i = 0; i < (BF16 ? 1 : 2); ++i) {
                const uint4 raw = __ldg(p + i);
                x[r][4 * i] = raw.x;
                x[r][4 * i + 1] = raw.y;
                x[r][4 * i + 2] = raw.z;
                x[r][4 * i + 3] = raw.w;
            }
        }
    }
    __device__ __forceinline__ float at(int r, int c) const {
        if (!BF16) return __uint_as_float(x[r][c & (BF16 ? 3 : 7)]);
        return __uint_as_float((c & 1) ? (x[r][c >> 1] & 0xFFFF0000u) : (x[r][c >> 1] << 16));
    }
};

// Column maxima of the block's 128 x 64 weights -> part[warp][column]; the caller synchronises.
template <bool BF16>
__device__ __forceinline__ void block_column_max(const Rows<BF16> &v, float (*part)[64]) {
    const int warp = threadIdx.x >> 5, p8 = threadIdx.x & 7, qd = (threadIdx.x >> 3) & 3;
    if constexpr (BF16) {  // two columns at a time (the maximum of bf16 values is one of them: nothing is rounded)
#pragma unroll
        for (int c2 = 0; c2 < 4; ++c2) {
            auto bf = [](uint32_t u) { return __habs2(*reinterpret_cast<__nv_bfloat162 *>(&u)); };
            __nv_bfloat162 m = __hmax2(__hmax2(bf(v.x[0][c2]), bf(v.x[1][c2])), __hmax2(bf(v.x[2][c2]), bf(v.x[3][c2])));
            m = __hmax2(m, __shfl_xor_sync(0xFFFFFFFFu, m, 8));
            m = __hmax2(m, __shfl_xor_sync(0xFFFFFFFFu, m, 16));
            if (qd == 0) *reinterpret_cast<float2 *>(&part[warp][p8 * 8 + 2 * c2]) = make_float2(fmaxf(0.f, __low2float(m)), fmaxf(0.f, __high2float(m)));
        }
    } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            float m = fmaxf(fmaxf(fabsf(v.at(0, c)), fabsf(v.at(1, c))), fmaxf(fabsf(v.at(2, c)), fabsf(v.at(3, c))));
            m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 8));
            m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 16));
            if (qd == 0) part[warp][p8 * 8 + c] = fmaxf(0.f, m);  // (all four NaN: 0, as the reference's comparison leaves it)
        }
    }
}

// Per-column mode, first pass: maxima of every 128-row block, [k/128][n].  grid = (n/64, k/128), block = 256.
template <bool BF16>
__global__ void __launch_bounds__(256, BF16 ? 6 : 4) pack_max_kernel(const void *w, int n, float *block_max) {
    __shared__ float part[8][64];
    const int tid = threadIdx.x, p8 = tid & 7, qd = (tid >> 3) & 3, kt = tid >> 5;
    Rows<BF16> v;
    v.load(w, (static_cast<size_t>(blockIdx.y) * 128 + kt * 16 + 2 * qd) * n + blockIdx.x * 64 + p8 * 8, n);
    block_column_max(v, part);
    __syncthreads();
    if (tid < 64) {
        float mx = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, part[i][tid]);
        block_max[static_cast<size_t>(blockIdx.y) * n + blockIdx.x * 64 + tid] = mx;
    }
}

// Second pass: the maxima of a column's blocks -> its scale.  (The maxima wait in the buffer of the packed words, which the
// third pass overwrites; it only needs the scales.)  grid = n/64, block = 256: four threads per column.
__global__ void __launch_bounds__(256) pack_column_scales_kernel(const float *block_max, int n, int blocks, uint16_t *scales_perm) {
    __shared__ float part[4][64];
    const int c = threadIdx.x & 63, col = blockIdx.x * 64 + c;
    float mx = 0.f;
    for (int b = threadIdx.x >> 6; b < blocks; b += 4) mx = fmaxf(mx, block_max[static_cast<size_t>(b) * n + col]);
    part[threadIdx.x >> 6][c] = mx;
    __syncthreads();
    if (threadIdx.x < 64)
        scales_perm[scale_single_pos(col)] = __half_as_ushort(scale_of_max(fmaxf(fmaxf(part[0][c], part[1][c]), fmaxf(part[2][c], part[3][c]))));
}

// Grouped: scales from the block's own maxima.  Per column: scales from the second pass.  grid = (n/64, k/128), block = 256.
template <bool BF16>
__global__ void __launch_bounds__(256, BF16 ? 5 : 4) pack_group_kernel(const void *w, int n, int per_column, uint16_t *scales_perm,
                                                         int32_t *b_packed, float *dequant) {
    __shared__ float part[8][64];
    __shared__ ColumnScale col_scale[64];
    const int tid = threadIdx.x, p8 = tid & 7, qd = (tid >> 3) & 3, kt = tid >> 5;
    const int ch = blockIdx.x, grp = blockIdx.y;
    Rows<BF16> v;
    const size_t off = (static_cast<size_t>(grp) * 128 + kt * 16 + 2 * qd) * n + ch * 64 + p8 * 8;
    v.load(w, off, n);
    if (!per_column) {
        block_column_max(v, part);
        __syncthreads();
    }
    if (tid < 64) {
        const int col = ch * 64 + tid;
        __half h;
        if (!per_column) {
            float mx = part[0][tid];
#pragma unroll
            for (int i = 1; i < 8; ++i) mx = fmaxf(mx, part[i][tid]);
            h = scale_of_max(mx);
            scales_perm[static_cast<size_t>(grp) * n + scale_group_pos(col)] = __half_as_ushort(h);
        } else {
            h = __ushort_as_half(scales_perm[scale_single_pos(col)]);
        }
        col_scale[tid] = column_scale(h);
    }
    __syncthreads();
    // Half words: nibbles 0, 1, 4, 5 of the word of column c (rows 2qd, 2qd+8, 2qd+1, 2qd+9).
    uint32_t half[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const ColumnScale cs = col_scale[p8 * 8 + c];
        constexpr int kOrder[4] = {3, 1, 2, 0};  // rows of nibbles 5, 4, 1, 0: highest first
        uint32_t word = 0;
        float worst = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            const float2 q = f2_unpack(f2_mul(f2_pack(v.at(kOrder[i], c), v.at(kOrder[i + 1], c)), f2_pack(cs.inv, cs.inv)));
            const unsigned long long t = f2_pack(min_nan(q.x, 7.f), min_nan(q.y, 7.f));  // (above 7 the clamp decides)
            const unsigned long long r = f2_add(t, f2_pack(kRoundMagic, kRoundMagic));
            const float2 d = f2_unpack(f2_add(t, f2_fma(r, f2_pack(-1.f, -1.f), f2_pack(kRoundMagic, kRoundMagic))));  // t - rounded(t)
            worst = max_nan(worst, max_nan(fabsf(d.x), fabsf(d.y)));
            const float2 rr = f2_unpack(r);
            word = (word << (i == 2 ? 12 : 4)) + __float_as_uint(rr.x);
            word = (word << 4) + __float_as_uint(rr.y);
        }
        // each nibble came as magic + q: take the magic bits out and add the offset of 8
        constexpr uint32_t kAdd = 8u - kRoundMagicBits;
        word += kAdd * (1u + (1u << 4) + (1u << 16) + (1u << 20));
        if (!(worst < 0.49999f) || cs.inv == 0.f) {  // (NaN among them)
            const float sum = (v.at(0, c) + v.at(1, c)) + (v.at(2, c) + v.at(3, c));
            word = 0;
            if (cs.inv == 0.f || sum != sum) {
#pragma unroll 1
                for (int i = 0; i < 4; ++i) {
                    const float x = i == 0 ? v.at(3, c) : i == 1 ? v.at(1, c) : i == 2 ? v.at(2, c) : v.at(0, c);
                    word = (word << (i == 2 ? 12 : 4)) | static_cast<uint32_t>(quantize_one(x, cs.s));
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) word = (word << (i == 2 ? 12 : 4)) | quantize_near_tie(v.at(kOrder[i], c), cs);
            }
        }
        half[c] = word;
        if (dequant) {
            constexpr int kRow[4] = {0, 1, 8, 9}, kShift[4] = {0, 16, 4, 20};
#pragma unroll
            for (int r = 0; r < 4; ++r)
                dequant[off + static_cast<size_t>(kRow[r]) * n + c] =
                    __fmul_rn(static_cast<float>(static_cast<int>((word >> kShift[r]) & 0xF) - kQOffset), cs.s);
        }
    }
    // Lane p8 = 2j + e holds columns 16j + 8e + c.  The even lane finishes the words of c = 0..3, the odd one those of 4..7.
    const int e = p8 & 1, j = p8 >> 1;
    uint32_t *dst = reinterpret_cast<uint32_t *>(b_packed) + (static_cast<size_t>(grp) * 8 + kt) * 2 * n + ch * 128 + j;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, e ? half[i] : half[4 + i], 1);
        const uint32_t lo = e ? got : half[i], hi = e ? half[4 + i] : got;
        const int c = 4 * e + i;
        dst[(c * 4 + qd) * 4] = lo | (hi << 8);
    }
}

// Already-quantised input: q uint8 [k,n] -> packed words; scales moved to Marlin order.
__global__ void repack_words_kernel(const uint8_t *q, int n, int32_t *b_packed) {
    __shared__ uint8_t nib[16][64];
    const int ch = blockIdx.x, kb = blockIdx.y, tid = threadIdx.x;
    for (int e = tid; e < 16 * 16; e += blockDim.x) {  // 16 rows x 16 uint32 (4 nibble bytes each)
        const int r = e >> 4, c4 = e & 15;
        *reinterpret_cast<uint32_t *>(&nib[r][4 * c4]) =
            *reinterpret_cast<const uint32_t *>(q + static_cast<size_t>(kb * 16 + r) * n + ch * 64 + 4 * c4);
    }
    __syncthreads();
    const int lane = tid >> 2, j = tid & 3;
    const int r0 = 2 * (lane & 3), c = lane >> 2;
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        word |= static_cast<uint32_t>(nib[r0 + nib_dr(i)][16 * j + c + nib_dc(i)] & 0xF) << (4 * i);
    b_packed[static_cast<size_t>(kb) * 2 * n + ch * 128 + tid] = static_cast<int32_t>(word);
}

// GPTQ qweight int32 [k/8, n] -> packed words.  A thread takes one c of one 16-row tile and 64-column chunk: the two GPTQ words
// (rows 0-7 and 8-15 of the tile) of columns 16j + c and 16j + 8 + c give the words (c, qd) for every qd, byte qd of each being
// rows 2qd and 2qd + 1; the sixteen words of c are 64 contiguous bytes.  WIDE: b_packed is 16-byte aligned (an int32 buffer of a C caller
// need not be).  grid = (n/64, ceil(k/16/32)), block = 256.
// The scales and zero-points of a block's columns are dealt over the blocks that share them: scales to Marlin order, zero-points that are not
// 8 counted (count may be null).  One launch for the three: a call has 2 to 3 us of the host per launch, and waits for its end
// (1024 x 1024 27.5 -> 23.4 us, 2560 x 9216 38.6 -> 33.8).
template <bool WIDE>
__global__ void __launch_bounds__(256) repack_gptq_kernel(const int32_t *qweight, int n, int k_tiles, int32_t *b_packed, const uint16_t *scales,
                                                          const int32_t *qzeros, int rows, int per_column, uint16_t *scales_perm, uint32_t *count) {
    const int c = threadIdx.x & 7, kb = blockIdx.y * 32 + (threadIdx.x >> 3), ch = blockIdx.x;
    for (int r = blockIdx.y * 4 + (threadIdx.x >> 6); r < rows; r += 4 * gridDim.y) {
        const int col = ch * 64 + (threadIdx.x & 63);
        scales_perm[static_cast<size_t>(r) * n + (per_column ? scale_single_pos(col) : scale_group_pos(col))] = scales[static_cast<size_t>(r) * n + col];
    }
    if (count) {
        uint32_t bad = 0;
        for (int r = blockIdx.y * 32 + (threadIdx.x >> 3); r < rows; r += 32 * gridDim.y) {  // (one word = eight zero-points)
            const uint32_t z = static_cast<uint32_t>(qzeros[static_cast<size_t>(r) * (n / 8) + ch * 8 + c]);
#pragma unroll
            for (int j = 0; j < 8; ++j) bad += ((z >> (4 * j)) & 0xFu) != static_cast<uint32_t>(kQOffset);
        }
        if (bad) atomicAdd(count, bad);
    }
    if (kb >= k_tiles) return;
    const uint32_t *src = reinterpret_cast<const uint32_t *>(qweight) + static_cast<size_t>(kb) * 2 * n + ch * 64 + c;
    uint32_t in[2][8];  // [row half][8-column step]
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int t = 0; t < 8; ++t) in[r][t] = __ldg(src + static_cast<size_t>(r) * n + t * 8);
    int32_t *dst = b_packed + static_cast<size_t>(kb) * 2 * n + ch * 128 + c * 16;
#pragma unroll
    for (int qd = 0; qd < 4; ++qd) {
        uint32_t out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // bytes: low nibble = even row, high nibble = odd row
            const uint32_t a = (in[0][2 * j] >> (8 * qd)) & 0xFFu, b = (in[1][2 * j] >> (8 * qd)) & 0xFFu;
            const uint32_t a8 = (in[0][2 * j + 1] >> (8 * qd)) & 0xFFu, b8 = (in[1][2 * j + 1] >> (8 * qd)) & 0xFFu;
            const uint32_t x = a | (b << 8) | (a8 << 16) | (b8 << 24);  // nibbles: A0 A1 B0 B1 A'0 A'1 B'0 B'1
            const uint32_t ev = x & 0x0F0F0F0Fu, od = (x >> 4) & 0x0F0F0F0Fu;
            // even rows to nibbles 0..3, odd rows to nibbles 4..7
            const uint32_t e2 = (ev | (ev >> 4)) & 0x00FF00FFu, o2 = (od | (od >> 4)) & 0x00FF00FFu;
            out[j] = ((e2 | (e2 >> 8)) & 0xFFFFu) | ((o2 | (o2 >> 8)) << 16);
        }
        if constexpr (WIDE) {
            reinterpret_cast<uint4 *>(dst)[qd] = make_uint4(out[0], out[1], out[2], out[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[qd * 4 + j] = static_cast<int32_t>(out[j]);
        }
    }
}

__global__ void permute_scales_kernel(const uint16_t *scales, int n, int per_column, uint16_t *out) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x, grp = blockIdx.y;
    if (col >= n) return;
    const int pos = per_column ? scale_single_pos(col) : scale_group_pos(col);
    out[static_cast<size_t>(grp) * n + pos] = scales[static_cast<size_t>(grp) * n + col];
}

// The GEMM kernels are launched with programmatic stream serialisation and read the packed weights and scales BEFORE
// their grid-dependency wait (weights normally never depend on the kernel before a GEMM).  A GEMM enqueued right after a
// device pack would break that assumption, so every device pack entry point ends with this ordinary launch: it starts
// only when the pack kernels have completed and flushed, and it is what the next kernel's early part overlaps with.
__global__ void pack_fence_kernel() {}

}  // namespace
}  // namespace kiln

extern "C" {

kiln_w4a16_status_t kiln_w4a16_quantize_and_pack_device(const void *weight, int weight_is_bf16, int k, int n,
                                                        int groupsize, int32_t *b_packed,
                                                        uint16_t *scales_f16, float *dequant, void *stream) {
    int g = 0;
    if (int rc = shape_ok(k, n, groupsize, &g)) return rc;
    if (!weight || !b_packed || !scales_f16) return KILN_W4A16_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int num_groups = k / g;
    // The one-pass kernel: 16-byte loads, 128-row groups or the whole column.
    const bool aligned = (reinterpret_cast<uintptr_t>(weight) & 15) == 0;  // (n is a multiple of 64: rows stay 16-byte aligned)
    if (aligned && (groupsize == 128 || groupsize == -1)) {
        const dim3 grid(n / 64, k / 128);
        const int per_column = groupsize == -1;
        if (per_column) {
            float *block_max = reinterpret_cast<float *>(b_packed);  // (k/128 x n floats: a sixteenth of it)
            if (weight_is_bf16)
                pack_max_kernel<true><<<grid, 256, 0, st>>>(weight, n, block_max);
            else
                pack_max_kernel<false><<<grid, 256, 0, st>>>(weight, n, block_max);
            pack_column_scales_kernel<<<n / 64, 256, 0, st>>>(block_max, n, k / 128, scales_f16);
        }
        if (weight_is_bf16)
            pack_group_kernel<true><<<grid, 256, 0, st>>>(weight, n, per_column, scales_f16, b_packed, dequant);
        else
            pack_group_kernel<false><<<grid, 256, 0, st>>>(weight, n, per_column, scales_f16, b_packed, dequant);
        pack_fence_kernel<<<1, 32, 0, st>>>();
        note_launch(per_column ? 4 : 2);
        return record_cuda_error(cudaGetLastError());
    }
    float *scales_nat = nullptr;  // natural-order f32 scales, scratch for the second kernel
    if (int rc = record_cuda_error(cudaMallocAsync(&scales_nat, sizeof(float) * num_groups * n, st))) return rc;
    const dim3 g1(n / 128, num_groups), g2(n / 64, k / 16);
    if (weight_is_bf16) {
        pack_scales_kernel<true><<<g1, 128, 0, st>>>(weight, n, g, groupsize == -1, scales_f16, scales_nat);
        pack_words_kernel<true><<<g2, 128, 0, st>>>(weight, n, g, scales_nat, b_packed, dequant);
    } else {
        pack_scales_kernel<false><<<g1, 128, 0, st>>>(weight, n, g, groupsize == -1, scales_f16, scales_nat);
        pack_words_kernel<false><<<g2, 128, 0, st>>>(weight, n, g, scales_nat, b_packed, dequant);
    }
    pack_fence_kernel<<<1, 32, 0, st>>>();
    note_launch(3);
    int rc = record_cuda_error(cudaGetLastError());
    const int rc2 = record_cuda_error(cudaFreeAsync(scales_nat, st));
    return rc ? rc : rc2;
}

kiln_w4a16_status_t kiln_w4a16_repack_device(const uint8_t *q, const uint16_t *scales, int k, int n,
                                             int groupsize, int32_t *b_packed, uint16_t *scales_perm,
                                             void *stream) {
    if (k <= 0 || n <= 0) return KILN_W4A16_ERR_ARG;
    if (k % 16 != 0 || n % 64 != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    const int g = groupsize == -1 ? k : groupsize;
    if (g <= 0 || k % g != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    if (!q || !scales || !b_packed || !scales_perm) return KILN_W4A16_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(q) & 3) != 0) return KILN_W4A16_ERR_ALIGNMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    repack_words_kernel<<<dim3(n / 64, k / 16), 128, 0, st>>>(q, n, b_packed);
    permute_scales_kernel<<<dim3((n + 127) / 128, k / g), 128, 0, st>>>(scales, n, groupsize == -1, scales_perm);
    pack_fence_kernel<<<1, 32, 0, st>>>();
    note_launch(3);
    return record_cuda_error(cudaGetLastError());
}

// Device variant of kiln_w4a16_repack_gptq_host.  The symmetry check cannot refuse before the launch without a
// synchronisation, so it reports: *asymmetric (a DEVICE uint32, may be NULL) receives the number of zero-points that are
// not 8; the caller reads it (stream-ordered) and discards the output if it is not 0.
kiln_w4a16_status_t kiln_w4a16_repack_gptq_device(const int32_t *qweight, const int32_t *qzeros, const uint16_t *scales,
                                                  int k, int n, int groupsize, int32_t *b_packed, uint16_t *scales_perm,
                                                  uint32_t *asymmetric, void *stream) {
    if (k <= 0 || n <= 0) return KILN_W4A16_ERR_ARG;
    if (k % 16 != 0 || n % 64 != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    const int g = groupsize == -1 ? k : groupsize;
    if (g <= 0 || k % g != 0) return KILN_W4A16_ERR_PROB_SHAPE;
    if (!qweight || !qzeros || !scales || !b_packed || !scales_perm) return KILN_W4A16_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (asymmetric) {
        if (int rc = record_cuda_error(cudaMemsetAsync(asymmetric, 0, sizeof(uint32_t), st))) return rc;
    }
    const auto repack = (reinterpret_cast<uintptr_t>(b_packed) & 15) == 0 ? repack_gptq_kernel<true> : repack_gptq_kernel<false>;
    repack<<<dim3(n / 64, (k / 16 + 31) / 32), 256, 0, st>>>(qweight, n, k / 16, b_packed, scales, qzeros, k / g, groupsize == -1, scales_perm, asymmetric);
    pack_fence_kernel<<<1, 32, 0, st>>>();
    note_launch(2);
    return record_cuda_error(cudaGetLastError());
}

}  // extern "C"
