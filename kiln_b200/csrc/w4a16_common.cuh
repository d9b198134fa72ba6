// Shared device helpers and host-side declarations for the W4A16 kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/kiln_w4a16.h"

namespace kiln {

// ---- Marlin layout facts (what the packer of kiln-marlin-gemm/src/lib.rs:429-479 emits) ----
// b_packed is [k/16][n/64][32 lanes][4 words]: one 512-byte block per (16 K-rows, 64 N-cols).
// In a block, lane l (qd = l%4, c = l/4) owns four words, word j covering the 16-column tile
// j of the chunk.  Nibble i of a word holds q[kb*16 + r][chunk*64 + j*16 + cc] for
//   (r, cc) = (2qd, c) (2qd+8, c) (2qd, c+8) (2qd+8, c+8) (2qd+1, c) (2qd+9, c) (2qd+1, c+8) (2qd+9, c+8)
// so nibbles (0,4), (1,5), (2,6), (3,7) are the four bf16x2 B registers of two m16n8k16 MMAs.
// Grouped scales: within every 64 columns, position 8*i + j holds column i + 8*j.
constexpr int kGroup = 128;     // K elements per scale group
constexpr int kChunkCols = 64;  // N columns per 512-byte block


// Two packed nibbles -> (nibble - 8) * s * 2^-22 as bf16x2, in one AND and one fused multiply-add.
// Read as bf16, a nibble at bits 0..3 of a half word is the subnormal nibble * 2^-133, and one at bits 4..7, whose top bit is the
// exponent's lowest, is nibble * 2^-129: subnormals and the first normal binade are one linear scale.  So the fused multiply-add
// brings nibble * s - 8 s, rounded once, which is what subtracting 8 and multiplying by s in two steps gives.  s * 2^133 would be
// too large for bf16; with the factor of 2^-22 it is not, whatever the fp16 scale is (the largest rounds to 2^16).  The
// factor is a power of two, so it changes no rounding; what reads the sums takes it out (kWeightUnscale), in fp32: a product after
// the rounding to bf16 would round sums below 2^-104 as the subnormals that they are with it.
// An infinite scale gives NaN (without the factor, infinity except for a nibble of 8; a sum over a group of 128 was NaN either way unless no
// activation is 0, no nibble 8 and all products have one sign).  Sums in fp32 reach down to 2^-149 at the factor, so a sum has eight good
// bits from 2^-119 on (from 2^-126, where bf16's subnormals begin, without it).
// Nine instructions for a packed word's eight weights; OR-ing the nibbles into 128.0, subtracting 136 and multiplying took fifteen, and
// the dequantising warps bound every kernel that uses this up to a few hundred rows (37 rows 2560 -> 18432 10.4 -> 9.4 us, 9216 -> 2560
// 8.3 -> 7.6); above, it saves power (16384 x 9216 x 9216 2026 -> 1969 us).
constexpr uint32_t kNibMask = 0x000F000Fu, kHiNibMask = 0x00F000F0u;
constexpr float kWeightFactor = 1.f / 4194304.f, kWeightUnscale = 4194304.f;  // 2^-22
struct WeightScale {  // of two columns
    __nv_bfloat162 lo, hi, off;  // s * 2^111, s * 2^107, -8 s * 2^-22
};
__device__ __forceinline__ WeightScale weight_scale(uint32_t half2_bits) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&half2_bits));
    const __nv_bfloat162 s = __floats2bfloat162_rn(f.x, f.y);
    const uint32_t lo = 0x77007700u, hi = 0x75007500u, off = 0xB600B600u;  // bf16x2 2^111, 2^107, -2^-19
    return {__hmul2(s, *reinterpret_cast<const __nv_bfloat162 *>(&lo)), __hmul2(s, *reinterpret_cast<const __nv_bfloat162 *>(&hi)),
            __hmul2(s, *reinterpret_cast<const __nv_bfloat162 *>(&off))};
}
__device__ __forceinline__ uint32_t dequant_pair(uint32_t nibbles, __nv_bfloat162 mul, __nv_bfloat162 off) {
    const __nv_bfloat162 w = __hfma2(*reinterpret_cast<const __nv_bfloat162 *>(&nibbles), mul, off);
    return *reinterpret_cast<const uint32_t *>(&w);
}
// Two sums without the factor: one instruction, as a bf16x2 product is (256 rows 256 -> 2560 4.9 us; two FMULs 5.1).
__device__ __forceinline__ void unscale(float &a, float &b) {
    asm("{\n\t.reg .b64 x, f;\n\t"
        "mov.b64 x, {%0, %1};\n\t"
        "mov.b64 f, {%2, %2};\n\t"
        "mul.rn.f32x2 x, x, f;\n\t"
        "mov.b64 {%0, %1}, x;\n\t}"
        : "+f"(a), "+f"(b)
        : "f"(kWeightUnscale));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
// silu(g) * u of sums that still have the factor, g' = g 2^-22 and u' = u 2^-22: e^-g = 2^(-g log2 e) takes g's out in the product with
// log2 e, 1 / (2^-22 + 2^-22 e^-g) once more for the quotient, and u's goes last: no product on the way is larger than the result, so
// nothing overflows that the result does not.  (Taken out of u before the product, 300 rows 512 -> 9216 13.3 us; so 12.5.)
__device__ __forceinline__ float swiglu_scaled(float g, float u) {
    constexpr float kLog2e = 1.4426950408889634f;
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * (-kLog2e * kWeightUnscale)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaf(e, kWeightFactor, kWeightFactor)));
    return g * r * u * kWeightUnscale;
}
// the eight weights of a packed word: K 2qd, 2qd + 1 and 2qd + 8, 2qd + 9 of the first column (c), then of the second (c + 8)
__device__ __forceinline__ void dequant_word(uint32_t x, const WeightScale &s, uint32_t &k0, uint32_t &k8, uint32_t &second_k0, uint32_t &second_k8) {
    const uint32_t y = x >> 8;
    k0 = dequant_pair(x & kNibMask, __low2bfloat162(s.lo), __low2bfloat162(s.off));
    k8 = dequant_pair(x & kHiNibMask, __low2bfloat162(s.hi), __low2bfloat162(s.off));
    second_k0 = dequant_pair(y & kNibMask, __high2bfloat162(s.lo), __high2bfloat162(s.off));
    second_k8 = dequant_pair(y & kHiNibMask, __high2bfloat162(s.hi), __high2bfloat162(s.off));
}

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                               uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t smem_addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr));
}

// Weights are read exactly once: bypass L1.
__device__ __forceinline__ uint4 ld_stream_v4(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// Activations: cached in L2 only, so a buffer another kernel has just rewritten is never read from a stale L1 line.
__device__ __forceinline__ uint4 ld_cg_v4(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// (through L1, where CTAs on the same SM find it again)
__device__ __forceinline__ uint4 ld_v4(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Programmatic dependent launch: let the next kernel in the stream start its prologue,
// and wait for the previous kernel's memory before touching anything it may have written.
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_smem_addr, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(cta));
    return r;
}
// Position of natural column `col` inside the per-column (groupsize -1) scale order
// (kiln-marlin-gemm/src/lib.rs:348-357): within each 32, out[8i + j] = in[2i + {0,1,8,9,16,17,24,25}[j]].
__device__ __host__ __forceinline__ int scale_single_pos(int col) {
    int c32 = col & 31;
    return (col & ~31) + 8 * ((c32 & 7) >> 1) + 2 * (c32 >> 3) + (c32 & 1);
}

// per-column scales of an even column and the next one: neighbours in that order, one load of four bytes (S is 16-byte aligned)
__device__ __forceinline__ float2 scale_pair(const __half *S, int col) {
    return __half22float2(*reinterpret_cast<const __half2 *>(S + scale_single_pos(col)));
}

// ---- host side --------------------------------------------------------------------------
struct GemmArgs {
    const void *A;   // bf16 [m,k]
    const void *B;   // int32 [k/16, 2n]
    const void *S;   // fp16 [k/g, n]
    void *C;         // bf16 [m,n]
    int m, n, k;
    int groupsize;   // 128 or -1
    void *workspace;
    size_t workspace_bytes;
    cudaStream_t stream;
    // fused all-gather (prefill kernel only): store the result into the row-major [m, ldc] buffers of n_peers GPUs
    void *peer_c[8] = {};
    int n_peers = 0, ldc = 0, col0 = 0;
    // the same with one NVSwitch multicast address for the whole group instead of per-GPU pointers (multimem.st)
    void *mc_c = nullptr;
    // epilogue options.  LoRA delta C += lora_t * lora_b^T: lora_t [m, lora_r] = scale * x * A^T, fp32 for the decode kernel and the small-batch
    // kernel's fp32-scale variant, bf16 where it is an operand tile of a tcgen05 kernel; lora_b bf16 [n, lora_r].  swiglu: columns are gate / up
    // interleaved in runs of 32, C is [m, n/2] (decode kernel, small-batch kernel without a K split, pair kernel)
    bool no_scratch = false;  // the tcgen05 kernel may not use the workspace (legacy entry point: its caller's buffer is tiny)
    const void *lora_t = nullptr;
    const void *lora_b = nullptr;
    int lora_r = 0;
    int swiglu = 0;
};

// One GEMM of a grouped decode launch.
struct DecodeItem {
    const void *A, *B, *S;
    void *C;
    int m, n, k, groupsize;
    const void *lora_t, *lora_b;
    int lora_r, swiglu;
};

struct DecodeOverride {
    int cluster_k, warps_k, warps_n;
};

int device_sm_count();
void note_launch(unsigned n = 1);
int record_cuda_error(cudaError_t e);  // returns KILN_W4A16_ERR_CUDA if e != success else 0
uint32_t *device_status_word();        // per-device word written by bounded waits; nullptr on failure

int launch_decode(const GemmArgs &a, const DecodeOverride &ov);
void decode_plan(int m, int n, int k, const DecodeOverride &ov, int out[4]);
int launch_decode_list(const DecodeItem *items, int count, cudaStream_t stream, const DecodeOverride &ov);
int launch_lora_down(const void *x, const void *lora_a, float scale, int m, int k, int r, void *t, int bf16_out, cudaStream_t stream);
bool prefill_fuses_lora(int groupsize, int lora_r);
int launch_finish(const void *base, void *c, int m, int n, const float *t, const void *lora_b, int r, int swiglu, cudaStream_t stream);
int launch_prefill(const GemmArgs &a);
size_t prefill_workspace_bytes(int m, int n, int k);
void set_prefill_override(int bn, int splits, int mt, int stream_k);
void set_wait_limit_ns(unsigned long long ns);
unsigned long long current_wait_limit_ns();
void set_smallm_enabled(int on);
bool smallm_supported(int m, int n, int k, int groupsize, int splits);
int smallm_clusters(int splits);
bool smallm_takes(int m, int n, int k, int groupsize);
int launch_smallm(const GemmArgs &a, int splits, bool exact = false);
int launch_smallm_group(const GemmArgs *items, int count, int splits, bool exact);
int smallm_most_grouped();
bool exact_supported(int m, int n, int k, int groupsize, bool swiglu, int lora_r);
int launch_exact(const GemmArgs &a);
bool exact_group_pays(const GemmArgs *items, int count);
int launch_exact_group(const GemmArgs *items, int count);
int launch_plain_group(const GemmArgs *items, int count);
void set_test_drop_a_load(int k_step);
int test_drop_a_load();
constexpr int kTestShortExchange = -2;  // its value for the LoRA projection's exchange
void prefill_plan(int m, int n, int k, int out[4]);
bool prefill_supported(int m, int n, int k, int groupsize);
bool prefill_fuses_swiglu(int m, int n, int k);
bool prefill_swiglu_room(int m, int n, int k);
int static_status_read_clear(cudaStream_t st, uint32_t *out);
int decode_status_read_clear(cudaStream_t st, uint32_t *out);

}  // namespace kiln
