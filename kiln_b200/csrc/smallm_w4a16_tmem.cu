// W4A16 GEMM for at most 128 activation rows on sm_100a: the dequantised weights are the TENSOR-MEMORY operand of tcgen05.mma.
//
// The GEMM is issued transposed, C^T[n, m] = W^T[n, k] * X^T[k, m]: the 128 weight columns of a tile are the M = 128 rows of
// the MMA (TMEM lanes), dequantised straight into tensor memory, and the activations are the N operand (N = rows rounded up
// to 16), K-major 128B-swizzled tiles that TMA drops into shared memory.
//
//  * Packed words reach shared memory by TMA, 8 KB per 128 K (one scale group), up to twelve stages ahead, and all scales of
//    the CTA's K range in one copy.  One thread keeps the ring full, so the bytes in flight do not cost registers, and it
//    fills before the previous kernel in the stream has finished (weights never depend on it).
//  * A packed word of the kiln-marlin-gemm layout (kiln-marlin-gemm/src/lib.rs:262-357) gives lane (c, qd) of a warp two K pairs
//    of columns c and c + 8 of a 16-column tile.  That is the register layout of tcgen05.st.16x128b (register 0: TMEM lane
//    c, cell qd; register 1: lane c + 8; the next two: cells 4 + qd), so the four dequantised registers of a word are stored
//    as they are.  (A 32x32b store wants a lane per column: the packed bytes then have to be transposed within quads first,
//    8 of 39 instructions per 16 K, two of them shuffles in the dependent chain.)
//  * Four dequant teams of four warps take the stages in turn; a stage passes through one barrier on its way to the issuers
//    (activation bytes + one arrival per warp of the team) and one on its way back (a commit per issuer).  Every wait costs
//    ~90 cycles even when it need not wait, so the next ones are asked ahead (mbar_test) and there are few of them.
//  * The MMA issuers run with the whole warp and elect a lane around the instructions (elect_one).
//  * The bf16 tile is put together in shared memory and leaves through TMA.
//  * One (tile, K split) per CTA.  The CTAs of a tile's K splits are one thread-block cluster: each pushes its fp32 sums to
//    the CTA that owns the rows (st.async, counted on the owner's mbarrier), the owner adds them in split order.  No
//    workspace and no second kernel; the order is that of the general kernel's split-K reduction.
// Even and odd 64-deep halves of a stage have an MMA issuer and an accumulator of their own (as the general kernel's
// 128-column tiles; the epilogue adds the two), so the two kernels' results are bit-identical.
// Roles (640 threads): warp 0 packed words, warps 1 and 2 MMA issuers, warp 3 scales and activations, warps 4-19 dequant, then
// the epilogue.
// Warp x of a team owns TMEM lanes 32(x%4)..+31 = words 2h and 2h + 1 (h = x % 2) of chunk (x%4)/2, columns 32h..+31, which one
// 8-byte read per lane brings.  With SwiGLU, words h and h + 2 (of a 16-byte read): lanes 0..15 hold columns 16h + r, lanes 16..31
// columns 32 + 16h + r, so that with gate and up interleaved in runs of 32 columns a gate column and its up column are 16 lanes
// apart and meet through one shuffle.
// LoRA delta (grouped scales): an extra iteration at the start of a tile's K range, its tensor-memory operand the tile's rows of
// lora_b and its activation tile t = scale * x * A^T (bf16, written by the kernel launched just before).
// Every wait is bounded (w4a16_async.cuh).  Per-column scales (group size -1): the weights are dequantised unscaled and the
// scale multiplies the finished sums.
//
// What bounds it: about 0.25 us per 128 K and CTA up to 64 rows.  The dequant needs some 200 issue slots of every
// sub-partition (nine instructions per packed word), an MMA 32 cycles at 64 rows and 9 at 16, a barrier 160 cycles to answer beside
// them, and a launch has 2.5 to 3.4 us that no stage hides (the first words' latency after a CTA of the previous kernel has left the SM, the exchange, the
// exit).  CUDA graph over rotating weights, before (register-streamed words, quad transposes, split-K through global slabs and
// a second kernel) -> now: 64 rows 2560 -> 18432 14.0 -> 10.3 us, 2560 -> 4096 8.5 -> 5.3, 4096 -> 2560 8.9 -> 5.7, 2560 -> 8192
// 10.9 -> 7.1, 9216 -> 2560 12.0 -> 9.0; 128 rows 2560 -> 18432 16.0 -> 12.1.  EXACT, against the decode kernel: 16 rows
// 2560 -> 18432 12.2 -> 9.6, 2560 -> 4096 5.7 -> 4.5; 64 rows 2560 -> 512 5.8 -> 3.4.
#include <algorithm>

#include "w4a16_common.cuh"
#include "w4a16_umma.cuh"

namespace kiln {
namespace {

constexpr int kTileCols = 128;  // weight columns per tile = TMEM lanes = MMA M
constexpr int kMaxRows = 128;   // most activation rows = MMA N (rounded up to 16) the kernel takes
constexpr int kStageK = 128;    // K per stage of packed words: one scale group
constexpr int kAtomK = 64;      // K per 128B-swizzled activation tile: half a stage, four K = 16 MMAs
constexpr int kTmemCols = 512;
constexpr int kSlotCols = kStageK / 2;       // TMEM columns of one slot of weights (two bf16 per cell)
constexpr int kWSlotBytes = kStageK * kTileCols / 2;
constexpr int kScaleBytes = kTileCols * 2;   // scales of one stage
constexpr int kMaxStages = 96;               // K stages of one CTA: their scales are loaded at once
// A team asks for its next stage, kTeams further, when the slot's previous stage may only just have been asked for: a parity
// wait tells two neighbouring phases apart and no more, so the rings hold a multiple of kTeams stages (packed words: a slot's
// previous stage was this team's own) or, where the MMAs complete in order, at least kTeams (TMEM slots).
constexpr int kMaxWSlots = 12, kMaxSlots = 8;
constexpr int kTeamWarp0 = 4, kTeamWarps = 4, kTeams = 4;
constexpr int kTeamThreads = kTeams * kTeamWarps * 32;
constexpr int kThreads = kTeamWarp0 * 32 + kTeamThreads;
static_assert(kMaxWSlots % kTeams == 0, "see above");

constexpr int kExactRows = 16;  // rows of a CTA of the EXACT variant (see the kernel)

// barriers: [wfull][wempty] x kMaxWSlots, [full][empty] x kMaxSlots, done, exchange, scales
constexpr int kBarWFull = 0, kBarWEmpty = kMaxWSlots, kBarFull = 2 * kMaxWSlots, kBarEmpty = kBarFull + kMaxSlots,
              kBarDone = kBarEmpty + kMaxSlots, kBarExchange = kBarDone + 1, kBarScales = kBarExchange + 1, kBars = kBarScales + 1;
constexpr int kBarrierBytes = (kBars * 8 + 8 + 127) / 128 * 128;

struct SmallMParams {
    const __half *S;
    __nv_bfloat16 *C;
    uint32_t *status;
    int m, n, splits, k_stages, npad;
    int scale_rows;                  // most stages of a CTA
    int w_slots;                     // depth of the ring of packed words, in stages
    int recv_over_rings;             // the receive buffer of a K split lies over the rings (more than 64 rows)
    int off_x, off_scale, off_recv, off_lora;  // shared memory: packed words at 0, then these (bytes from the 1024-byte aligned base)
    int quads;                       // groups of four rows
    int quads_per_rank, rank_magic;  // K splits: those owned by one rank; x / quads_per_rank = (x * rank_magic) >> 16
    // LoRA delta C += t * lora_b^T: t = scale * x * A^T is bf16 [m, lora_r], lora_b bf16 [n, lora_r], lora_r a multiple of 8 up to 128
    const float *lora_t;  // EXACT: the fp32 projection [m, lora_r]
    const __nv_bfloat16 *lora_b;
    int lora_r;
    int per_column;  // one fp16 scale per column (group size -1): dequantised unscaled, the scale applied to the sums
    unsigned long long wait_limit_ns;
};

__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// 16 TMEM lanes x 16 cells: two K tiles of 16 of sixteen columns
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
                 "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_32x32b_x4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
__device__ __forceinline__ uint2 lds_v2(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ float lds_half(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void st_shared_bf16(uint32_t addr, __nv_bfloat16 v) {
    asm volatile("st.shared.b16 [%0], %1;" ::"r"(addr), "h"(__bfloat16_as_ushort(v)) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: A = 128 lanes x 8 cells (16 K as bf16 pairs), B = K-major tile of N rows
__device__ __forceinline__ void umma_bf16_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// four floats into a peer's shared memory; their bytes count on the peer's mbarrier when they have landed
__device__ __forceinline__ void st_async_v4(uint32_t cluster_addr, float a, float b, float c, float d, uint32_t cluster_mbar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(cluster_addr),
                 "f"(a), "f"(b), "f"(c), "f"(d), "r"(cluster_mbar)
                 : "memory");
}

__device__ __forceinline__ void sts_v4(uint32_t addr, float a, float b, float c, float d) {
    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// One packed word -> the four bf16x2 registers {column c: K pair qd, column c + 8: K pair qd, c: K pair 4 + qd, c + 8: K pair
// 4 + qd}.
__device__ __forceinline__ void dequant_word(uint32_t x, const WeightScale &s, uint32_t *r) { dequant_word(x, s, r[0], r[2], r[1], r[3]); }

// Further GEMMs of one launch, which have the rows, the K, the group size and the K splits of the first in common: blockIdx.y runs over the
// tiles of all of them.  (A template parameter, because what a launch passes and looks up for them costs a single GEMM a few per cent.)
constexpr int kMaxGroup = 4;
template <bool GROUP>
struct SmallMGroup {};
template <>
struct SmallMGroup<true> {
    CUtensorMap w[kMaxGroup], s[kMaxGroup], x[kMaxGroup], c[kMaxGroup];
    const __half *S[kMaxGroup];
    __nv_bfloat16 *C[kMaxGroup];
    int n[kMaxGroup], tile0[kMaxGroup];
    int count;
};

// Stages in flight: TMEM slots of weights, and activation slots in shared memory
template <int R>
constexpr int slots() {
    return (kTmemCols - 2 * R) / kSlotCols;  // 6 for R = 64, 4 for R = 128
}

// EXACT: the weights go to tensor memory unscaled, as the integers -8..7.  A stage, which is one scale group, has an
// accumulator of its own, one of four like the teams; before a team hands its next stage to the issuers, and once more at the end, it
// adds the finished one, times the fp32 group scale of the lane's column, to sums in registers.  That is the decode kernel's
// arithmetic (exact products, the scale applied once per group, in fp32), so the batches that were the decode kernel's lose no
// precision here.  The teams' sums meet in tensor memory, and a LoRA delta is added to them in fp32 from the fp32 projection.  More than
// sixteen rows are so many more CTAs (blockIdx.z): for projections of few columns, which leave the GPU empty otherwise.
// R: most rows.  SWIGLU is a template parameter so that the plain epilogue is compiled on its own.
template <int R, bool SWIGLU, bool EXACT, bool GROUP = false>
__global__ void __launch_bounds__(kThreads, 1)
w4a16_smallm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_s, const __grid_constant__ CUtensorMap tmap_x,
                    const __grid_constant__ CUtensorMap tmap_t, const __grid_constant__ CUtensorMap tmap_c,
                    const __grid_constant__ SmallMParams p, const __grid_constant__ SmallMGroup<GROUP> g) {
    constexpr int kSlots = slots<R>();
    static_assert(kSlots >= kTeams && kSlots <= kMaxSlots, "see kMaxWSlots");
    static_assert(!EXACT || (kTeams <= kSlots && kTeams * kExactRows <= R && kExactRows == 4 * kTeams), "see above");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    __shared__ __align__(128) uint8_t bar_mem[kBarrierBytes];
    const uint32_t bar_base = smem_u32(bar_mem);
    auto bar = [&](int i) { return bar_base + 8u * i; };
    auto full = [&](int s) { return bar(kBarFull + s); };    // activation bytes + one arrival per warp of the dequant team
    auto empty = [&](int s) { return bar(kBarEmpty + s); };  // one commit per issuer
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(bar_mem + 8 * kBars);
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(bar_mem + 8 * kBars + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int tile = blockIdx.y, width = p.n;
    const CUtensorMap *map_w = &tmap_w, *map_s = &tmap_s, *map_x = &tmap_x, *map_c = &tmap_c;
    const __half *scales = p.S;
    __nv_bfloat16 *result = p.C;
    if constexpr (GROUP) {
        int i = 0;
#pragma unroll
        for (int j = 1; j < kMaxGroup; ++j)
            if (j < g.count && tile >= g.tile0[j]) i = j;
        tile -= g.tile0[i];
        width = g.n[i];
        map_w = &g.w[i], map_s = &g.s[i], map_x = &g.x[i], map_c = &g.c[i];
        scales = g.S[i];
        result = g.C[i];
    }
    const int rank = blockIdx.x, nt = tile, m0 = EXACT ? blockIdx.z * kExactRows : 0;  // K split (= rank in the cluster), tile, first row
    const int ks0 = rank * p.k_stages / p.splits, ks1 = (rank + 1) * p.k_stages / p.splits, n_st = ks1 - ks0;
    const int lora_it = (!EXACT && rank == 0 && p.lora_r > 0) ? 1 : 0;  // the CTA that starts the tile's K range begins with the LoRA iteration
    const int n_it = n_st + lora_it;

    pdl_launch_dependents();
    if (warp == 0) {
        for (int i = lane; i < kBars; i += 32) {
            const int count = i < kBarWEmpty ? 1 : i < kBarFull ? kTeamWarps : i < kBarEmpty ? 1 + kTeamWarps : i <= kBarDone ? 2 : 1;
            mbar_init(bar(i), count);
        }
        if (lane == 0) *abort_flag = 0;
        mbar_init_fence();
        __syncwarp();
        if (lane == 0 && p.splits > 1) {
            const int own = max(0, min(p.quads_per_rank, p.quads - rank * p.quads_per_rank));
            mbar_arrive_expect_tx(bar(kBarExchange), static_cast<uint32_t>((p.splits - 1) * own) * kTileCols * 16u);
        }
    } else if (warp == 3 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(map_s) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(map_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(map_c) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t *>(tmem_ptr_slot))),
                     "r"(static_cast<uint32_t>(kTmemCols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_slot;
    // (a CTA may be written through distributed shared memory once it runs and its barriers stand; checked before the first push)
    if (p.splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int x_bytes = p.npad * 128;  // one 64-deep activation tile; a stage has two

    if (warp == 0) {
        // ---------------- packed words and scales ----------------
        // (the stream starts before the previous kernel in the stream has finished: it depends on nothing)
        if (lane == 0) {
            bool ok = true;
            int i = 0, s = 0, ph = 1;
            for (; i < n_st; ++i) {
                if (i == p.w_slots) pdl_wait();  // (park until the consumers run)
                if (i >= p.w_slots && !(ok = mbar_wait(bar(kBarWEmpty + s), ph, abort_flag, p.status, 0xA00u | s, p.wait_limit_ns))) break;
                mbar_arrive_expect_tx(bar(kBarWFull + s), kWSlotBytes);
                tma_load_2d(smem_base + s * kWSlotBytes, map_w, nt * (2 * kTileCols), (ks0 + i) * (kStageK / 16), bar(kBarWFull + s));
                if (++s == p.w_slots) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (!ok)  // drain: wait (bounded, ignoring the abort flag) for copies already issued
                for (int j = max(0, i - p.w_slots); j < i; ++j) mbar_wait_quiet(bar(kBarWFull + j % p.w_slots), (j / p.w_slots) & 1);
        }
    } else if (warp == 3) {
        // ---------------- activations ----------------
        if (lane == 0) {
            if (!p.per_column) {  // the scales of all stages (rows past the CTA's last one are not used)
                mbar_arrive_expect_tx(bar(kBarScales), p.scale_rows * kScaleBytes);
                tma_load_2d(smem_base + p.off_scale, map_s, nt * kTileCols, ks0, bar(kBarScales));
            }
            pdl_wait();  // the activations may be the previous kernel's output
            bool ok = true;
            int it = 0, s = 0, ph = 1;
            for (; it < n_it; ++it) {
                if (it >= kSlots && !(ok = mbar_wait(empty(s), ph, abort_flag, p.status, 0xA80u | s, p.wait_limit_ns))) break;
                mbar_arrive_expect_tx(full(s), 2 * x_bytes);  // (rows past m are zero-filled and counted)
                const uint32_t dst = smem_base + p.off_x + s * 2 * x_bytes;
                if (it < lora_it) {  // (columns of t past lora_r read zero)
                    tma_load_2d(dst, &tmap_t, 0, 0, full(s));
                    tma_load_2d(dst + x_bytes, &tmap_t, kAtomK, 0, full(s));
                } else {
                    tma_load_3d(dst, map_x, 0, m0, (ks0 + it - lora_it) * 2, full(s));
                }
                if (++s == kSlots) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (!ok)  // drain: wait (bounded, ignoring the abort flag) for copies already issued
                for (int j = max(0, it - kSlots); j < it; ++j) mbar_wait_quiet(full(j % kSlots), (j / kSlots) & 1);
        }
    } else if (warp < 3) {
        // ---------------- MMA issuers: half t of every stage into accumulator t ----------------
        const int t = warp - 1;
        pdl_wait();
        const bool issue = elect_one();
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(p.npad >> 3) << 17) |
                               (static_cast<uint32_t>(kTileCols >> 4) << 24);  // D fp32, A/B bf16, K-major, N = npad, M = 128
        const uint32_t d_tmem = tmem_base + t * R;
        const uint64_t desc0 = make_smem_desc(smem_base + p.off_x + t * x_bytes);
        int s = 0, ph = 0;
        bool ok = true, ready = false;
        int it = 0;
        for (; it < n_it; ++it) {
            if (!ready && !(ok = mbar_wait(full(s), ph, abort_flag, p.status, 0xB00u | s, p.wait_limit_ns))) break;
            tc_fence_after();
            const uint64_t b_desc = desc0 + static_cast<uint64_t>((s * 2 * x_bytes) >> 4);
            const uint32_t a_tmem = tmem_base + 2 * R + s * kSlotCols + t * (kAtomK / 2);
            if (issue) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    umma_bf16_tmem_a(d_tmem + (EXACT ? it % kTeams * kExactRows : 0), a_tmem + j * 8, b_desc + 2 * j, idesc,
                                     ((!EXACT && it > 0) || j > 0) ? 1u : 0u);
                umma_commit(empty(s));
            }
            if (++s == kSlots) {
                s = 0;
                ph ^= 1;
            }
            ready = mbar_test(full(s), ph);
        }
        if (!EXACT && ok && issue) umma_commit(bar(kBarDone));
        if (!ok && it > 0) mbar_wait_quiet(empty((it - 1) % kSlots), ((it - 1) / kSlots) & 1);  // the MMAs it has issued
    } else {
        // ---------------- dequant: packed int4 -> bf16 pairs in tensor memory ----------------
        // team u takes every fourth iteration, from iteration u
        const int u = (warp - kTeamWarp0) / kTeamWarps;
        const int quarter = warp & 3, ch = quarter >> 1, h = quarter & 1;
        const int c = lane >> 2;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        const int col_in_tile = 64 * ch + (SWIGLU ? 16 * h + (lane & 15) + 32 * (lane >> 4) : 32 * h + lane);  // of TMEM lane `lane` of this warp
        bool ok = true;
        int it = u;
        if (lora_it && it == 0) {
            // LoRA iteration: this tile's rows of lora_b, one row per TMEM lane, K = lora_r padded with zeros.  A weight like any
            // other: it is read without waiting for the previous kernel.  (The first iteration of a slot waits for nobody.)
            const uint4 *row = reinterpret_cast<const uint4 *>(p.lora_b + (static_cast<size_t>(nt) * kTileCols + col_in_tile) * p.lora_r);
#pragma unroll 2
            for (int kt = 0; kt < kStageK / 16; ++kt) {
                uint4 lw[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) lw[i] = 16 * kt + 8 * i + 8 <= p.lora_r ? ld_stream_v4(row + 2 * kt + i) : make_uint4(0u, 0u, 0u, 0u);
                const uint32_t r[8] = {lw[0].x, lw[0].y, lw[0].z, lw[0].w, lw[1].x, lw[1].y, lw[1].z, lw[1].w};
                tmem_st_32x32b_x8(t_lane + 2 * R + kt * 8, r);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(full(0));
            it = kTeams;
        }
        // scales of the lane's four columns c and c + 8 of its two words: word w has them at positions 8c + 2w + {0, 1} of the
        // chunk's scale order (position 8i + j holds column 8j + i)
        const uint32_t sc_addr = smem_base + p.off_scale + (ch * 64 + 8 * c + (SWIGLU ? 2 : 4) * h) * 2;
        const uint32_t w_addr = smem_base + ch * 512 + lane * 16;
        int s = it % kSlots, ph = (it / kSlots & 1) ^ 1;                               // slot of the iteration
        int ws = (it - lora_it) % p.w_slots, wph = ((it - lora_it) / p.w_slots) & 1;  // slot of its packed words
        bool w_ready = false, t_ready = false;  // the next waits, asked ahead
        if (it < n_it && !p.per_column) ok = warp_all(mbar_wait(bar(kBarScales), 0, abort_flag, p.status, 0xEC0u, p.wait_limit_ns));
        // EXACT: the CTA's part of the LoRA rank (the K splits share it), and its values of lora_b for the tile's columns, a weight that
        // is there before it is needed; 16 bytes more per row keep the reads off each other's banks
        const int lora_0 = 8 * (rank * (p.lora_r / 8) / p.splits), lora_n = 8 * ((rank + 1) * (p.lora_r / 8) / p.splits) - lora_0;
        const int lora_pitch = lora_n * 2 + 16;
        const uint32_t lora_b_addr = smem_base + p.off_lora, lora_t_addr = lora_b_addr + kTileCols * lora_pitch;
        if (EXACT && p.lora_r > 0) {
            const int pieces = lora_n / 8, x = (warp - kTeamWarp0) * 32 + lane;
            for (int i = x; i < kTileCols * pieces; i += kTeamThreads) {
                const int col = i / pieces, piece = i - col * pieces;
                cp_async_16(lora_b_addr + col * lora_pitch + piece * 16,
                            p.lora_b + (static_cast<size_t>(nt) * kTileCols + col) * p.lora_r + lora_0 + 8 * piece);
            }
        }
        // EXACT: sums of the lane's column, and the step that adds the stage j of this team
        float y[EXACT ? kExactRows : 1] = {};
        const int col_in_chunk = col_in_tile & 63;
        const uint32_t exact_sc = smem_base + p.off_scale + (ch * 64 + 8 * (col_in_chunk & 7) + (col_in_chunk >> 3)) * 2;
        auto add_stage = [&](int j, int s, int ph) {
            if (ok && !mbar_test(empty(s), ph)) ok = mbar_wait(empty(s), ph, abort_flag, p.status, 0xF00u | s, p.wait_limit_ns);
            __syncwarp();
            tc_fence_after();
            const float scale = p.per_column ? kWeightUnscale : lds_half(exact_sc + j * kScaleBytes) * kWeightUnscale;
            uint32_t a[kExactRows], b[kExactRows];
            tmem_ld_32x32b_x16(t_lane + u * kExactRows, a);
            tmem_ld_32x32b_x16(t_lane + R + u * kExactRows, b);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < (EXACT ? kExactRows : 1); ++i) y[i] = fmaf(scale, __uint_as_float(a[i]) + __uint_as_float(b[i]), y[i]);
        };
        int s0 = 0, ph0 = 0;  // slot of the team's previous stage, and the phase that ends with it
        for (; it < n_it; it += kTeams) {  // (to the end, whatever a wait says: see warp_all)
            if (it >= kSlots && it < kSlots + kTeams) pdl_wait();  // (park until the MMAs may run)
            if (ok && !w_ready) ok = mbar_wait(bar(kBarWFull + ws), wph, abort_flag, p.status, 0xE00u | ws, p.wait_limit_ns);
            uint32_t wa[8], wb[8];  // the two words of the eight K tiles
#pragma unroll
            for (int kt = 0; kt < 8; ++kt) {
                if (SWIGLU) {
                    const uint4 v = lds_v4(w_addr + ws * kWSlotBytes + kt * 1024);
                    wa[kt] = h ? v.y : v.x;
                    wb[kt] = h ? v.w : v.z;
                } else {
                    const uint2 v = lds_v2(w_addr + 8 * h + ws * kWSlotBytes + kt * 1024);
                    wa[kt] = v.x;
                    wb[kt] = v.y;
                }
            }
            WeightScale sc[2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
                sc[i] = weight_scale(EXACT || p.per_column ? 0x3C003C00u : lds_u32(sc_addr + (it - lora_it) * kScaleBytes + (SWIGLU ? 8 : 4) * i));
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(bar(kBarWEmpty + ws));  // the stage's words are in registers: its slot can load again
            if (it >= kSlots && ok && !t_ready) ok = mbar_wait(empty(s), ph, abort_flag, p.status, 0xE80u | s, p.wait_limit_ns);
            tc_fence_after();
            const uint32_t dst = t_lane + 2 * R + s * kSlotCols;
#pragma unroll
            for (int k4 = 0; k4 < 2; ++k4) {  // four K tiles of 16 at a time
                uint32_t r[16];
#pragma unroll
                for (int i = 0; i < 4; ++i) dequant_word(wa[4 * k4 + i], sc[0], r + 4 * i);
                tmem_st_16x128b_x8(dst + k4 * 32, r);
#pragma unroll
                for (int i = 0; i < 4; ++i) dequant_word(wb[4 * k4 + i], sc[1], r + 4 * i);
                tmem_st_16x128b_x8(dst + (16u << 16) + k4 * 32, r);
            }
            if (EXACT && it >= kTeams) {
                if (it < 2 * kTeams) pdl_wait();  // (as above)
                add_stage(it - kTeams, s0, ph0);
            }
            const uint32_t done = full(s);
            s0 = s;
            ph0 = ph ^ 1;  // (the producer side of a slot waits for the phase before)
            if ((s += kTeams) >= kSlots) {
                s -= kSlots;
                ph ^= 1;
            }
            ws += kTeams;
            while (ws >= p.w_slots) {
                ws -= p.w_slots;
                wph ^= 1;
            }
            w_ready = mbar_test(bar(kBarWFull + ws), wph);
            t_ready = mbar_test(empty(s), ph);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(done);
        }
        if constexpr (EXACT) {
            pdl_wait();
            if (p.lora_r > 0) {  // this CTA's part of the fp32 projection (rows past m are not stored: any row will do for them)
                const int pieces = lora_n / 4, x = (warp - kTeamWarp0) * 32 + lane;
                for (int i = x; i < kExactRows * pieces; i += kTeamThreads) {
                    const int row = i / pieces, piece = i - row * pieces;
                    cp_async_16(lora_t_addr + i * 16, p.lora_t + static_cast<size_t>(min(m0 + row, p.m - 1)) * p.lora_r + lora_0 + 4 * piece);
                }
            }
            if (it > u) add_stage(it - kTeams, s0, ph0);
#pragma unroll
            for (int r8 = 0; r8 < kExactRows; r8 += 8) {
                uint32_t r[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(y[r8 + i]);
                tmem_st_32x32b_x8(t_lane + u * kExactRows + r8, r);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            // the four warps with this quarter of the lanes; all stages are through when they meet
            asm volatile("bar.sync %0, %1;" ::"r"(2 + quarter), "n"(kTeams * 32) : "memory");
            if (p.lora_r > 0) {
                cp_async_wait_all();
                asm volatile("bar.sync 1, %0;" ::"n"(kTeamThreads) : "memory");
            }
            ok = warp_all(ok && *abort_flag == 0);
        }
        // ---------------- epilogue: a thread owns one output column; team u takes every fourth block of 16 rows (EXACT: of 4) ----------------
        if (!EXACT) pdl_wait();  // (park until the MMAs may run)
        if (!EXACT) ok = warp_all(ok && mbar_wait(bar(kBarDone), 0, abort_flag, p.status, 0xD00u, p.wait_limit_ns));
        tc_fence_after();
        const int col = nt * kTileCols + col_in_tile;
        float v4[4] = {};  // EXACT: rows 4u..4u + 3
        if (EXACT) {
#pragma unroll
            for (int w = 0; w < kTeams; ++w) {
                uint32_t r[4];
                tmem_ld_32x32b_x4(t_lane + w * kExactRows + 4 * u, r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 4; ++i) v4[i] += __uint_as_float(r[i]);
            }
            if (p.lora_r > 0) {
                const uint32_t lb = lora_b_addr + col_in_tile * lora_pitch, t = lora_t_addr + 4 * u * lora_n * 4;
                for (int r = 0; r < lora_n; r += 8) {
                    const uint4 w4 = lds_v4(lb + r * 2);
                    const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 t0 = lds_v4(t + (i * lora_n + r) * 4), t1 = lds_v4(t + (i * lora_n + r) * 4 + 16);
                        const uint32_t tv[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            v4[i] = fmaf(__uint_as_float(tv[e]), __uint_as_float(e & 1 ? w[e / 2] & 0xFFFF0000u : w[e / 2] << 16), v4[i]);
                    }
                }
            }
        }
        auto drain = [&] {  // a wait of the teams has run out: copies that may be in flight though no wait of the loading warps has
            if (!p.per_column) mbar_wait_quiet(bar(kBarScales), 0);
            for (int j = max(0, n_st - p.w_slots); j < n_st; ++j) mbar_wait_quiet(bar(kBarWFull + j % p.w_slots), (j / p.w_slots) & 1);
            for (int j = max(0, n_it - kSlots); j < n_it; ++j) mbar_wait_quiet(full(j % kSlots), (j / kSlots) & 1);
        };
        if (p.splits == 1) {
            // The bf16 tile is put together in shared memory (over the rings, which are spent) and leaves through TMA: two-byte
            // stores from registers cost 8 cycles of the SM's load / store unit each.
            const float cs = (p.per_column ? __half2float(scales[scale_single_pos(col)]) : 1.f) * (EXACT ? 1.f : kWeightUnscale);
            const int ocol = SWIGLU ? ch * 32 + 16 * h + (lane & 15) : col_in_tile;  // output column within the tile
            const uint32_t stage = smem_base + (ocol >> 6) * x_bytes + (ocol & 7) * 2;
            const uint32_t chunk16 = (ocol & 63) >> 3;  // 16-byte chunk of a 128-byte row, XORed with row % 8
            if constexpr (EXACT) {
                const bool up = lane >= 16;
#pragma unroll
                for (int i = 0; i < 4; ++i) v4[i] *= cs;  // (before the exchange: the partner's column has a scale of its own)
#pragma unroll
                for (int i = 0; i < (SWIGLU ? 2 : 4); ++i) {
                    int row = 4 * u + i;
                    float out = v4[i];
                    if constexpr (SWIGLU) {  // (as below)
                        const float other = __shfl_xor_sync(0xFFFFFFFFu, up ? v4[2 * i] : v4[2 * i + 1], 16);
                        row = 4 * u + 2 * i + (up ? 1 : 0);
                        // (the division is slow for a dividend of zero, which rows past m would have)
                        const float g = m0 + row < p.m ? (up ? other : v4[2 * i]) : 1.f, w = up ? v4[2 * i + 1] : other;
                        out = g / (1.f + __expf(-g)) * w;  // (as the decode kernel divides: __fdividef gives 0 for a divisor above 2^126)
                    }
                    st_shared_bf16(stage + row * 128 + ((chunk16 ^ (row & 7)) << 4), __float2bfloat16_rn(out));
                }
            } else if (ok)
#pragma unroll 1
                for (int r0 = 16 * u; r0 < p.npad; r0 += 16 * kTeams) {
#pragma unroll
                    for (int r8 = 0; r8 < 16; r8 += 8) {
                        uint32_t a[8], b[8];
                        tmem_ld_32x32b_x8(t_lane + r0 + r8, a);
                        tmem_ld_32x32b_x8(t_lane + R + r0 + r8, b);
                        tmem_ld_wait();
                        float v[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] = (__uint_as_float(a[i]) + __uint_as_float(b[i])) * cs;
                        if constexpr (SWIGLU) {
                            // lanes 0..15 hold gate columns, lanes 16..31 their up columns: the former finish the even rows, the
                            // latter the odd ones
                            const bool up = lane >= 16;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float other = __shfl_xor_sync(0xFFFFFFFFu, up ? v[2 * i] : v[2 * i + 1], 16);
                                const float g = up ? other : v[2 * i], w = up ? v[2 * i + 1] : other;
                                const int row8 = 2 * i + (up ? 1 : 0);
                                st_shared_bf16(stage + (r0 + r8 + row8) * 128 + ((chunk16 ^ row8) << 4),
                                               __float2bfloat16_rn(__fdividef(g, 1.f + __expf(-g)) * w));
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                st_shared_bf16(stage + (r0 + r8 + i) * 128 + ((chunk16 ^ i) << 4), __float2bfloat16_rn(v[i]));
                        }
                    }
                }
            fence_proxy_async_smem();
            asm volatile("bar.sync 1, %0;" ::"n"(kTeamThreads) : "memory");  // (every warp of the teams comes here, whatever happened)
            if (ok && warp == kTeamWarp0 && lane == 0) {
                tma_store_2d(map_c, smem_base, nt * (SWIGLU ? kTileCols / 2 : kTileCols), m0);  // (rows past m are clipped)
                if (!SWIGLU) tma_store_2d(map_c, smem_base + x_bytes, nt * kTileCols + 64, m0);
                bulk_commit_group();
                bulk_wait_group_read0();  // (the end of the grid completes them)
            } else if (!ok && warp == kTeamWarp0 && lane == 0) {
                drain();
            }
        }
        if (p.splits > 1) {
            const uint32_t recv = smem_base + p.off_recv;
            __syncwarp();
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA of the cluster runs
            if (R > 64 && p.recv_over_rings) cluster_sync_all();  // ... and its rings, which the receive buffer lies over, are spent
            // (a quad of rows of this CTA's own goes straight to the buffer: the network between SMs bounds the exchange of many rows)
            auto push = [&](int quad, float a, float b, float c, float d) {
                const int owner = (quad * p.rank_magic) >> 16, slot = quad - owner * p.quads_per_rank;
                const uint32_t addr = recv + static_cast<uint32_t>((rank * p.quads_per_rank + slot) * kTileCols + col_in_tile) * 16u;
                if (owner == rank)
                    sts_v4(addr, a, b, c, d);
                else
                    st_async_v4(map_to_cta(addr, owner), a, b, c, d, map_to_cta(bar(kBarExchange), owner));
            };
            // A CTA that has given up pushes all the same, whatever its sums are (the status word tells what the results are worth): every CTA stays
            // until it has everything, so a push always finds its owner there.
            if constexpr (EXACT) {
                if (u < p.quads) push(u, v4[0], v4[1], v4[2], v4[3]);
            } else {
#pragma unroll 1
                for (int r0 = 8 * u; r0 < 4 * p.quads; r0 += 8 * kTeams) {
                    uint32_t a[8], b[8];
                    tmem_ld_32x32b_x8(t_lane + r0, a);
                    tmem_ld_32x32b_x8(t_lane + R + r0, b);
                    tmem_ld_wait();
                    float v[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(a[i]) + __uint_as_float(b[i]);
                    push(r0 / 4, v[0], v[1], v[2], v[3]);
                    if (r0 / 4 + 1 < p.quads) push(r0 / 4 + 1, v[4], v[5], v[6], v[7]);
                }
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kTeamThreads) : "memory");  // (the rows of its own; every warp of the teams comes here)
            if (ok) {
                ok = mbar_wait(bar(kBarExchange), 0, abort_flag, p.status, 0xD80u, p.wait_limit_ns);
            }
            if (ok) {
                if constexpr (EXACT || R <= 64) {
                    const int own = min(p.quads_per_rank, p.quads - rank * p.quads_per_rank);
                    const int x = (warp - kTeamWarp0) * 32 + lane, cc = x & (kTileCols - 1);
                    const int gcol = nt * kTileCols + cc;
                    const float cs = (p.per_column ? __half2float(scales[scale_single_pos(gcol)]) : 1.f) * (EXACT ? 1.f : kWeightUnscale);
                    for (int slot = x >> 7; slot < own; slot += kTeamThreads / kTileCols) {
                        const uint32_t src = recv + static_cast<uint32_t>(slot * kTileCols + cc) * 16u;
                        const uint4 v0 = lds_v4(src);
                        float v[4] = {__uint_as_float(v0.x), __uint_as_float(v0.y), __uint_as_float(v0.z), __uint_as_float(v0.w)};
                        for (int r = 1; r < p.splits; ++r) {
                            const uint4 u = lds_v4(src + static_cast<uint32_t>(r * p.quads_per_rank) * kTileCols * 16u);
                            v[0] += __uint_as_float(u.x);
                            v[1] += __uint_as_float(u.y);
                            v[2] += __uint_as_float(u.z);
                            v[3] += __uint_as_float(u.w);
                        }
                        const int row0 = m0 + (rank * p.quads_per_rank + slot) * 4;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (row0 + i < p.m) result[static_cast<size_t>(row0 + i) * width + gcol] = __float2bfloat16_rn(v[i] * cs);
                    }
                } else {
                    // A warp finishes a quad of rows, four adjacent columns a lane, and stores 256 contiguous bytes of each row: two-byte
                    // stores cost 8 cycles of the load / store unit each (128 rows, 2560 -> 4096 8.0 -> 7.6 us).  Up to 64 rows a CTA owns few
                    // quads, and a column a thread, whose chain of reads is shorter, is as fast or faster (16 rows 4.4 against 4.6).  The
                    // lanes read their columns in turned order, so that eight of them hit all banks.
                    const int own = min(p.quads_per_rank, p.quads - rank * p.quads_per_rank), turn = (lane >> 1) & 3;
                    const int gcol = nt * kTileCols + 4 * lane;
                    for (int slot = warp - kTeamWarp0; slot < own; slot += kTeams * kTeamWarps) {
                        float v[4][4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint4 x = lds_v4(recv + static_cast<uint32_t>(slot * kTileCols + 4 * lane + ((j + turn) & 3)) * 16u);
                            v[j][0] = __uint_as_float(x.x), v[j][1] = __uint_as_float(x.y), v[j][2] = __uint_as_float(x.z), v[j][3] = __uint_as_float(x.w);
                        }
                        for (int r = 1; r < p.splits; ++r) {
                            const uint32_t src = recv + static_cast<uint32_t>((r * p.quads_per_rank + slot) * kTileCols + 4 * lane) * 16u;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const uint4 x = lds_v4(src + ((j + turn) & 3) * 16u);
                                v[j][0] += __uint_as_float(x.x), v[j][1] += __uint_as_float(x.y), v[j][2] += __uint_as_float(x.z), v[j][3] += __uint_as_float(x.w);
                            }
                        }
                        const int row0 = m0 + (rank * p.quads_per_rank + slot) * 4;
                        float cs[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) cs[j] = (p.per_column ? __half2float(scales[scale_single_pos(gcol + j)]) : 1.f) * kWeightUnscale;
                        __nv_bfloat16 *dst = result + static_cast<size_t>(row0) * width + gcol;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float a0 = turn & 1 ? v[3][i] : v[0][i], a1 = turn & 1 ? v[0][i] : v[1][i], a2 = turn & 1 ? v[1][i] : v[2][i],
                                        a3 = turn & 1 ? v[2][i] : v[3][i];
                            const float c0 = turn & 2 ? a2 : a0, c1 = turn & 2 ? a3 : a1, c2 = turn & 2 ? a0 : a2, c3 = turn & 2 ? a1 : a3;
                            __nv_bfloat162 lo = __floats2bfloat162_rn(c0 * cs[0], c1 * cs[1]), hi = __floats2bfloat162_rn(c2 * cs[2], c3 * cs[3]);
                            if (row0 + i < p.m)
                                *reinterpret_cast<uint2 *>(dst + static_cast<size_t>(i) * width) =
                                    make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
                        }
                    }
                }
            } else {
                if (warp == kTeamWarp0 && lane == 0) drain();
                mbar_wait_quiet(bar(kBarExchange), 0, peers_limit_ns(p.wait_limit_ns));  // peers push into this CTA until they are through or have given up
            }
        }
        tc_fence_before();
    }

    if (R > 64 && p.recv_over_rings && warp < kTeamWarp0) {  // (the other warps' part in the barrier above)
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }

    // ---------------- teardown ----------------
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(static_cast<uint32_t>(kTmemCols))
                     : "memory");
    }
}

}  // namespace

// Problems this kernel takes with that many K splits (the dispatcher decides from which row count it pays).
bool smallm_supported(int m, int n, int k, int groupsize, int splits) {
    return m >= 1 && m <= kMaxRows && (groupsize == 128 || groupsize == -1) && n % kTileCols == 0 && n / kTileCols <= 65535 && k % kStageK == 0 &&
           splits >= 1 && splits <= 8 && splits <= k / kStageK && (k / kStageK + splits - 1) / splits <= kMaxStages;
}

// Clusters of `splits` (1..8) CTAs that the device holds at once: what a GPC has left over does not make a cluster (without a device,
// those of a B200 with 148 SMs).
int smallm_clusters(int splits) {
    static const int b200[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    static int cached[64][9] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return b200[splits];
    if (!cached[dev][splits]) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(splits, 64);
        cfg.blockDim = dim3(kThreads);
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = splits;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;  // (one CTA per SM, whatever its shared memory: registers)
        if (cudaOccupancyMaxActiveClusters(&n, w4a16_smallm_kernel<64, false, false>, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = b200[splits];
        }
        cached[dev][splits] = n;
    }
    return cached[dev][splits];
}

// C = A * dequant(B) with `splits` K splits (one cluster per tile), for up to kMaxGroup GEMMs that share rows, K and group size (several:
// no epilogue options).  exact: group scales applied in fp32.
int launch_smallm_group(const GemmArgs *items, int count, int splits, bool exact) {
    const GemmArgs &a = items[0];
    EncodeTiledFn enc = encode_fn();
    if (!enc) return KILN_W4A16_ERR_CUDA;
    uint32_t *status = device_status_word();
    if (!status) return KILN_W4A16_ERR_CUDA;
    const int rows = exact ? std::min(a.m, kExactRows) : a.m;  // of a CTA
    if (!smallm_supported(rows, a.n, a.k, a.groupsize, splits) || (a.swiglu && splits != 1)) return KILN_W4A16_ERR_KERN_SHAPE;

    if (count < 1 || count > kMaxGroup) return KILN_W4A16_ERR_ARG;
    int tiles = a.n / kTileCols;
    for (int i = 1; i < count; ++i) {
        const GemmArgs &b = items[i];
        if (b.m != a.m || b.k != a.k || b.groupsize != a.groupsize || b.n % kTileCols != 0) return KILN_W4A16_ERR_KERN_SHAPE;
        tiles += b.n / kTileCols;
    }
    if (tiles > 65535) return KILN_W4A16_ERR_KERN_SHAPE;

    const int npad = (rows + 15) & ~15, stages = (a.k / kStageK + splits - 1) / splits;
    auto encode = [&](CUtensorMap *map, const void *ptr, int cols) {  // boxes of 64 columns x all rows, 128-byte swizzle
        const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(a.m)}, strides[1] = {static_cast<cuuint64_t>(cols) * 2};
        const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(npad)}, estr[2] = {1, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    // Tensor maps of one GEMM: packed words, scales (unused with per-column scales), activations (unless x has those of the same ones already),
    // result (unused when K is split).  A map takes 0.1 us of the host, as much as a tenth of a launch.
    auto encode_maps = [&](const GemmArgs &q, CUtensorMap *w, CUtensorMap *s, CUtensorMap *x, CUtensorMap *c, bool same_x) {
        {  // packed words: [k/16][2n] int32, boxes of one tile x eight rows (128 K)
            const cuuint64_t dims[2] = {2ull * q.n, static_cast<cuuint64_t>(q.k / 16)}, strides[1] = {8ull * q.n};
            const cuuint32_t box[2] = {2 * kTileCols, kStageK / 16}, estr[2] = {1, 1};
            if (enc(w, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void *>(q.B), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return false;
        }
        *s = *w;
        if (q.groupsize != -1) {  // scales [k/128][n] fp16, boxes of one tile x the most stages a CTA has (rows past the matrix read zero)
            const cuuint64_t dims[2] = {static_cast<cuuint64_t>(q.n), static_cast<cuuint64_t>(q.k / kStageK)}, strides[1] = {2ull * q.n};
            const cuuint32_t box[2] = {kTileCols, static_cast<cuuint32_t>(stages)}, estr[2] = {1, 1};
            if (enc(s, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(q.S), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return false;
        }
        if (!same_x) {  // activations [m, k] seen as [k/64][m][64], so that one copy brings both 64-deep tiles of a stage
            const cuuint64_t dims[3] = {kAtomK, static_cast<cuuint64_t>(q.m), static_cast<cuuint64_t>(q.k / kAtomK)};
            const cuuint64_t strides[2] = {static_cast<cuuint64_t>(q.k) * 2, kAtomK * 2};
            // (test hook: boxes of eight rows less than the kernel announces, so that its waits for them run out)
            const cuuint32_t box[3] = {kAtomK, static_cast<cuuint32_t>(test_drop_a_load() >= 0 ? npad - 8 : npad), 2}, estr[3] = {1, 1, 1};
            if (enc(x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(q.A), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return false;
        }
        *c = *x;
        return splits != 1 || encode(c, q.C, q.swiglu ? q.n / 2 : q.n);
    };
    CUtensorMap tmap_w, tmap_s, tmap_x, tmap_t, tmap_c;
    if (!encode_maps(a, &tmap_w, &tmap_s, &tmap_x, &tmap_c, false)) return KILN_W4A16_ERR_CUDA;
    tmap_t = tmap_x;  // (unused without a LoRA delta)
    const bool lora = a.lora_r > 0 && a.lora_t && a.lora_b;
    if (lora) {
        if (a.groupsize == -1 || a.lora_r % 8 != 0 || a.lora_r > 128) return KILN_W4A16_ERR_KERN_SHAPE;
        if (!exact && !encode(&tmap_t, a.lora_t, a.lora_r)) return KILN_W4A16_ERR_CUDA;
    }
    if (count > 1 && (lora || a.swiglu)) return KILN_W4A16_ERR_KERN_SHAPE;

    SmallMParams p{};
    p.S = static_cast<const __half *>(a.S);
    p.C = static_cast<__nv_bfloat16 *>(a.C);
    p.status = status;
    p.m = a.m;
    p.n = a.n;
    p.splits = splits;
    p.k_stages = a.k / kStageK;
    p.npad = npad;
    p.quads = (rows + 3) / 4;
    p.quads_per_rank = (p.quads + splits - 1) / splits;
    p.rank_magic = (65536 + p.quads_per_rank - 1) / p.quads_per_rank;  // (exact for the at most 32 quads)
    p.per_column = a.groupsize == -1;
    p.lora_b = lora ? static_cast<const __nv_bfloat16 *>(a.lora_b) : nullptr;
    p.lora_t = lora ? static_cast<const float *>(a.lora_t) : nullptr;
    p.lora_r = lora ? a.lora_r : 0;
    p.wait_limit_ns = current_wait_limit_ns();

    // Shared memory: the activation ring mirrors the TMEM slots; packed words take the rest, up to twelve stages (eight, 64 KB
    // in flight, cover the latency of HBM at an SM's share of its bandwidth) or as many as the CTA has.  The receive buffer of a K
    // split lies behind them, or, above 64 rows and where it would leave fewer than those eight, over them: that costs a barrier of the
    // cluster between the last MMA and the exchange.
    constexpr int kMostSmem = 226 * 1024 - kBarrierBytes;
    const int recv = splits > 1 ? splits * p.quads_per_rank * kTileCols * 16 : 0;
    const int x_stages = std::min(stages + (lora && !exact ? 1 : 0), rows <= 64 ? slots<64>() : slots<128>());
    const int lora_part = lora && exact ? (a.lora_r / 8 + splits - 1) / splits * 8 : 0;  // most of the rank that a CTA has
    const int lora_bytes = lora_part ? kTileCols * (2 * lora_part + 16) + kExactRows * lora_part * 4 : 0;
    const int fixed = 2 * x_stages * npad * 128 + (p.per_column ? 0 : stages * kScaleBytes) + lora_bytes + 1024;
    p.scale_rows = stages;
    auto w_slots = [&](int bytes) {  // beside the rest and that many bytes
        int slots = kMaxWSlots;
        while (slots > kTeams && fixed + slots * kWSlotBytes + bytes > kMostSmem) slots -= kTeams;
        return std::min(stages, slots);
    };
    p.w_slots = w_slots(recv);
    p.recv_over_rings = rows > 64 && recv > 0 && (p.w_slots < std::min(stages, 8) || fixed + p.w_slots * kWSlotBytes + recv > kMostSmem);
    if (p.recv_over_rings) p.w_slots = w_slots(0);
    p.off_x = p.w_slots * kWSlotBytes;
    p.off_scale = p.off_x + 2 * x_stages * npad * 128;
    p.off_recv = p.recv_over_rings ? 0 : p.off_scale + (p.per_column ? 0 : stages * kScaleBytes);
    p.off_lora = p.off_recv + recv;
    const int smem = std::max(p.w_slots * kWSlotBytes + fixed, p.off_lora + lora_bytes + 1024);
    if (smem > kMostSmem) return KILN_W4A16_ERR_KERN_SHAPE;

    static bool attr_set[9][64] = {};  // per kernel variant and device: the shared-memory attribute is set once
    int dev = 0;
    cudaGetDevice(&dev);
    auto launch = [&](auto kernel, int variant, const auto &group) -> int {
        if (dev < 64 && !attr_set[variant][dev]) {
            if (int rc = record_cuda_error(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem))) return rc;
            attr_set[variant][dev] = true;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(splits, tiles, exact ? (a.m + kExactRows - 1) / kExactRows : 1);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = a.stream;
        cudaLaunchAttribute attrs[2];
        attrs[0] = pdl_attribute();
        attrs[1].id = cudaLaunchAttributeClusterDimension;
        attrs[1].val.clusterDim.x = splits;
        attrs[1].val.clusterDim.y = 1;
        attrs[1].val.clusterDim.z = 1;
        cfg.attrs = attrs;
        cfg.numAttrs = splits > 1 ? 2 : 1;
        note_launch();
        return record_cuda_error(cudaLaunchKernelEx(&cfg, kernel, tmap_w, tmap_s, tmap_x, tmap_t, tmap_c, p, group));
    };
    if (count > 1) {
        SmallMGroup<true> g;
        int tile0 = 0;
        g.count = count;
        for (int i = 0; i < count; ++i) {
            const GemmArgs &q = items[i];
            g.x[i] = tmap_x;
            if (i == 0)
                g.w[0] = tmap_w, g.s[0] = tmap_s, g.c[0] = tmap_c;
            else if (!encode_maps(q, &g.w[i], &g.s[i], &g.x[i], &g.c[i], q.A == a.A))
                return KILN_W4A16_ERR_CUDA;
            g.S[i] = static_cast<const __half *>(q.S);
            g.C[i] = static_cast<__nv_bfloat16 *>(q.C);
            g.n[i] = q.n;
            g.tile0[i] = tile0;
            tile0 += q.n / kTileCols;
        }
        if (exact) return launch(w4a16_smallm_kernel<64, false, true, true>, 8, g);
        return rows <= 64 ? launch(w4a16_smallm_kernel<64, false, false, true>, 6, g) : launch(w4a16_smallm_kernel<128, false, false, true>, 7, g);
    }
    const SmallMGroup<false> none;
    if (exact) return a.swiglu ? launch(w4a16_smallm_kernel<64, true, true>, 5, none) : launch(w4a16_smallm_kernel<64, false, true>, 4, none);
    if (a.swiglu) return a.m <= 64 ? launch(w4a16_smallm_kernel<64, true, false>, 2, none) : launch(w4a16_smallm_kernel<128, true, false>, 3, none);
    return a.m <= 64 ? launch(w4a16_smallm_kernel<64, false, false>, 0, none) : launch(w4a16_smallm_kernel<128, false, false>, 1, none);
}
int launch_smallm(const GemmArgs &a, int splits, bool exact) { return launch_smallm_group(&a, 1, splits, exact); }
int smallm_most_grouped() { return kMaxGroup; }

}  // namespace kiln
