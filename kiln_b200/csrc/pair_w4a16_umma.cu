// Prefill-shape W4A16 GEMM on CTA pairs (tcgen05.mma.cta_group::2): tiles of 256 rows x 256 or 128 columns, 64 K per pipeline stage.
//
// The kernel of single CTAs (prefill_w4a16_umma.cu) dequantises a weight once per 256 rows by giving a CTA two 128-row tiles.
// That costs it shared memory (per 256 x 256 x 64 it reads 96 KB of operands and writes 64 KB: 1250 cycles at 128 bytes a cycle
// against 1024 cycles of MMAs) and tensor memory (both accumulators belong to one tile, so its epilogue, 14,000 of 59,000 cycles
// at K = 2560, hides under nothing).  Here two SMs share the tile: each holds 128 rows of the activations and dequantises 128
// of the 256 weight columns (64 of 128), every MMA multiplies both halves, and an SM's tensor memory holds two accumulators of 128 x 256.
// Per SM and 64 K that is 32 KB read and 32 KB written in 512 cycles of MMAs, and the epilogue of a tile runs under the next one.
//
// Cluster of two CTAs; CTA 0 (the leader) issues the MMAs.  Per stage:
//  * full (leader's): the activation bytes of both CTAs (TMA loads of either count on it) + one arrival per dequant warp of both;
//  * empty (each CTA's own): the commit of the stage's MMAs, multicast to both.
// Per accumulator: full (each CTA's own, multicast commit), empty (leader's): one arrival per epilogue warp of both.
// Roles (608 threads): warp 0 TMA of the activations, warp 1 MMA issuer (leader) and the TMEM allocation, warps 2-5 epilogue, warp 6 TMA of the
// packed words and scales, warps 7-18 dequant in three teams that take the stages in turn.  Work distribution, K splits and the hybrid stream-K are those of the other kernel, a
// worker being a pair.  Dequantisation, LoRA steps, SwiGLU and per-column scales as there: same roundings.
// Every wait is bounded (w4a16_async.cuh).  When one runs out, its CTA tells the other one, lets what is in flight land, and the two leave
// together (see the teardown).
// No load is multicast.
#include "w4a16_prefill.cuh"

namespace kiln {
namespace {

constexpr int kTileM = 256;                      // rows of a tile
constexpr int kHalf = 128;                       // ... per CTA
constexpr int kABytes = kHalf * BK * 2;          // a stage's activations, per CTA
constexpr int kWordWarp = 6, kDequantWarp0 = 7, kTeams = 3, kTeamWarps = 4;
constexpr int kThreads = (kDequantWarp0 + kTeams * kTeamWarps) * 32;
// A dequant team asks for its next stage of words, kTeams further, knowing only its own last one: a parity wait tells neighbouring
// phases apart and no more, so the previous user of a slot has to be the team itself.
constexpr int kWordSlots = 6;
static_assert(kWordSlots % kTeams == 0, "see above");
constexpr int kBarrierBytes = 1024;              // (the staging tiles behind them are 1024-byte aligned)

// TN columns per tile, half of them dequantised by each CTA.
template <int TN>
struct Cfg {
    static constexpr int kCols = TN / 2;                                  // columns of B per CTA
    static constexpr int kBBytes = kCols * BK * 2, kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = TN == 256 ? 5 : 6;
    static constexpr int kTmemCols = 2 * TN;                              // two accumulators
    static constexpr int kWordBytes = kCols * BK / 2, kScaleBytes = kCols * 2, kWordSlotBytes = kWordBytes + 256;
    static constexpr int kSmemBytes = kStages * kStageBytes + kBarrierBytes + 4 * 2 * kEpiWarpBytes + kWordSlots * kWordSlotBytes + 1024;  // + alignment slack
    static constexpr int kBlocks = kCols / 64 * 4 / kTeamWarps;           // 512-byte packed blocks per dequant warp and stage
    // D fp32, A/B bf16, both K-major, N = TN, M = 256
    static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(TN >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
};

__device__ __forceinline__ void arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// a load into this CTA's shared memory that counts on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t cluster_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(cluster_bar)
                 : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives at the barrier at this offset in both CTAs when the MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<unsigned short>(3))
                 : "memory");
}

__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// One 512-byte packed block (16 K x 64 columns) -> the K-major 128B-swizzled tile: row (column of B) 8t + c at row_base + 1024 t, its
// two 16-byte chunks of the block at sw_lo and sw_hi.
__device__ __forceinline__ void dequant_block(const uint4 &w, const WeightScale (&sc)[4], uint32_t row_base, uint32_t sw_lo, uint32_t sw_hi) {
    const uint32_t xs[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t v[4];
        dequant_word(xs[j], sc[j], v[0], v[1], v[2], v[3]);
        const uint32_t r_lo = row_base + static_cast<uint32_t>(16 * j) * 128u, r_hi = r_lo + 8u * 128u;
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_lo + sw_lo), "r"(v[0]) : "memory");
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_lo + sw_hi), "r"(v[1]) : "memory");
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_hi + sw_lo), "r"(v[2]) : "memory");
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_hi + sw_hi), "r"(v[3]) : "memory");
    }
}

template <int TN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
w4a16_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_s,
                  const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_p, const __grid_constant__ CUtensorMap tmap_t,
                  const __grid_constant__ CUtensorMap tmap_lb, const __grid_constant__ PrefillParams p) {
    using C = Cfg<TN>;
    constexpr int kStages = C::kStages, kStageBytes = C::kStageBytes, kCols = C::kCols;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + kStages * kStageBytes;
    auto full = [&](int s) { return bar_base + 8u * s; };
    auto empty = [&](int s) { return bar_base + 8u * (kStages + s); };
    auto tmem_full = [&](int a) { return bar_base + 8u * (2 * kStages + a); };
    auto tmem_empty = [&](int a) { return bar_base + 8u * (2 * kStages + 2 + a); };
    auto word_full = [&](int s) { return bar_base + 8u * (2 * kStages + 4 + s); };
    auto word_empty = [&](int s) { return bar_base + 8u * (2 * kStages + 4 + kWordSlots + s); };
    constexpr int kBars = 2 * kStages + 4 + 2 * kWordSlots;
    const uint32_t epi_base = bar_base + kBarrierBytes, word_base = epi_base + 4 * 2 * kEpiWarpBytes;
    uint8_t *bar_gen = smem_gen + kStages * kStageBytes;
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(bar_gen + 8 * kBars);
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(bar_gen + 8 * kBars + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_ctarank());  // 0: leader
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full(s), 1 + 2 * kTeamWarps);
            mbar_init(empty(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tmem_full(a), 1);
            mbar_init(tmem_empty(a), 2 * 4);
        }
        for (int s = 0; s < kWordSlots; ++s) {
            mbar_init(word_full(s), 1);
            mbar_init(word_empty(s), kTeamWarps);
        }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) {  // (both CTAs of the pair take part)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t *>(tmem_ptr_slot))),
                     "r"(static_cast<uint32_t>(C::kTmemCols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the other CTA's barriers stand
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_slot;
    pdl_launch_dependents();

    int mt, nt, sp, ki0, ki1, slab;
    WorkIter wi(p, pair, pairs);

    if (warp == 0) {
        // ---------------- TMA: this CTA's 128 rows of the activations ----------------
        if (lane == 0) {
            pdl_wait();  // the activations may be the previous kernel's output
            bool ok = true;
            int s = 0;
            uint32_t ph = 1;
            while (ok && wi.next(mt, nt, sp, ki0, ki1, slab)) {
                const int ki1e = ki1 + (ki0 == 0 ? p.lora_steps : 0);
                for (int ki = ki0; ki < ki1e; ++ki) {
                    if (!(ok = mbar_wait(empty(s), ph, abort_flag, p.status, 0x100u | s, p.wait_limit_ns))) break;
                    const uint32_t leader_full = map_to_cta(full(s), 0), dst = smem_base + s * kStageBytes;
                    const bool lora = ki >= ki1;  // both operand tiles come by TMA (rows past m, columns past r read zero)
                    if (rank == 0) mbar_arrive_expect_tx(full(s), 2 * (lora ? kStageBytes : kABytes));
                    if (lora) {
                        tma_load_2d_pair(dst, &tmap_t, (ki - ki1) * BK, mt * kTileM + rank * kHalf, leader_full);
                        tma_load_2d_pair(dst + kABytes, &tmap_lb, (ki - ki1) * BK, nt * TN + rank * kCols, leader_full);
                    } else {
                        tma_load_2d_pair(dst, &tmap_a, ki * BK, mt * kTileM + rank * kHalf, leader_full);
                    }
                    if (++s == kStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (rank == 0) {
            const bool issue = elect_one();
            uint32_t tile = 0, ph = 0;
            int s = 0;
            bool ok = true, ready = false;
            for (; ok && wi.next(mt, nt, sp, ki0, ki1, slab); ++tile) {
                const uint32_t acc = tile & 1, acc_ph = (tile >> 1) & 1;
                const int ki1e = ki1 + (ki0 == 0 ? p.lora_steps : 0);
                if (!(ok = mbar_wait(tmem_empty(acc), acc_ph ^ 1, abort_flag, p.status, 0x200u | acc, p.wait_limit_ns))) break;
                for (int ki = ki0; ki < ki1e; ++ki) {
                    if (!ready && !(ok = mbar_wait(full(s), ph, abort_flag, p.status, 0x300u | s, p.wait_limit_ns))) break;
                    tc_fence_after();
                    const uint64_t a_desc = make_smem_desc(smem_base + s * kStageBytes), b_desc = make_smem_desc(smem_base + s * kStageBytes + kABytes);
                    if (issue) {
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j) umma_pair(tmem_base + acc * TN, a_desc + 2 * j, b_desc + 2 * j, C::kIdesc, (ki > ki0 || j > 0) ? 1u : 0u);
                        umma_commit_pair(empty(s));
                        if (ki == ki1e - 1) umma_commit_pair(tmem_full(acc));
                    }
                    if (++s == kStages) {
                        s = 0;
                        ph ^= 1;
                    }
                    ready = mbar_test(full(s), ph);
                }
            }
        }
    } else if (warp < kWordWarp) {
        // ---------------- epilogue: this CTA's 128 rows, all 256 columns ----------------
        const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 are the ones this warp may read
        pdl_wait();                    // C (or the workspace) may still be read or written by the previous kernel
        const uint32_t epi_tma0 = epi_base + static_cast<uint32_t>(warp - 2) * (2 * kEpiWarpBytes);  // two 1024-byte aligned staging tiles
        uint32_t tile = 0;
        bool ok = true;
        for (; ok && wi.next(mt, nt, sp, ki0, ki1, slab); ++tile) {
            const uint32_t acc = tile & 1, acc_ph = (tile >> 1) & 1;
            if (!(ok = warp_all(mbar_wait(tmem_full(acc), acc_ph, abort_flag, p.status, 0x500u | acc, p.wait_limit_ns)))) break;
            tc_fence_after();
            const int row = mt * kTileM + rank * kHalf + quarter * 32 + lane;
            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * TN;
            const uint32_t leader_empty = map_to_cta(tmem_empty(acc), 0);
            auto release = [&] {  // every column of the accumulator is in registers or shared memory
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_cluster(leader_empty);
            };
            if (slab >= 0 || p.splits > 1) {
                // fp32 piece of a split tile, 32 x 32 at a time through a swizzled staging tile and TMA: a stream-K piece to its
                // tile-shaped slab, a K split to its slab of C (rows past m are clipped)
#pragma unroll 1
                for (int q = 0; q < TN / 32; ++q) {
                    const uint32_t stage = epi_tma0 + static_cast<uint32_t>(q & 1) * kEpiWarpBytes;
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(t_row + q * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int v = 0; v < 8; ++v)
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(stage + lane * 128 + ((v ^ (lane & 7)) << 4)), "r"(r[4 * v]),
                                     "r"(r[4 * v + 1]), "r"(r[4 * v + 2]), "r"(r[4 * v + 3])
                                     : "memory");
                    if (q == TN / 32 - 1) release();
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (slab >= 0)
                            tma_store_3d(&tmap_p, stage, q * 32, rank * kHalf + quarter * 32, slab);
                        else
                            tma_store_3d(&tmap_p, stage, nt * TN + q * 32, mt * kTileM + rank * kHalf + quarter * 32, sp);
                        bulk_commit_group();
                        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the other staging tile has been read
                    }
                    __syncwarp();
                }
                continue;
            }
            uint32_t ra[32], rb[32];
            tmem_ld_32x32b_x32(t_row, ra);
            tmem_ld_32x32b_x32(t_row + 32, rb);
            if (p.swiglu) {
                // a 64-column run is 32 gate columns and their 32 up columns, i.e. the two register buffers of a round
                __nv_bfloat16 *crow = p.C + static_cast<size_t>(row) * (p.n >> 1) + ((nt * TN) >> 1);
#pragma unroll 1
                for (int pp = 0; pp < TN / 64; ++pp) {
                    tmem_ld_wait();
                    uint4 *dst = reinterpret_cast<uint4 *>(crow + pp * 32);
#pragma unroll
                    for (int v = 0; v < 4; ++v) {  // eight output columns at a time: their registers die with the store
                        uint32_t o[4];
#pragma unroll
                        for (int e2 = 0; e2 < 4; ++e2) {
                            const int e = 4 * v + e2;
                            float ga = __uint_as_float(ra[2 * e]), gb = __uint_as_float(ra[2 * e + 1]);
                            float ua = __uint_as_float(rb[2 * e]), ub = __uint_as_float(rb[2 * e + 1]);
                            if (p.per_column) {
                                const float2 sg = scale_pair(p.S, nt * TN + pp * 64 + 2 * e), su = scale_pair(p.S, nt * TN + pp * 64 + 32 + 2 * e);
                                ga *= sg.x;
                                gb *= sg.y;
                                ua *= su.x;
                                ub *= su.y;
                            }
                            o[e2] = pack_bf16x2(swiglu_scaled(ga, ua), swiglu_scaled(gb, ub));
                        }
                        if (row < p.m) dst[v] = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                    if (pp + 1 < TN / 64) {
                        tmem_ld_32x32b_x32(t_row + (pp + 1) * 64, ra);
                        tmem_ld_32x32b_x32(t_row + (pp + 1) * 64 + 32, rb);
                    } else {
                        release();
                    }
                }
                continue;
            }
#pragma unroll 1
            for (int pp = 0; pp < TN / 64; ++pp) {
                const uint32_t epi_tma = epi_tma0 + static_cast<uint32_t>(pp & 1) * kEpiWarpBytes;
                tmem_ld_wait();
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int col = nt * TN + pp * 64 + half * 32;
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float x0 = __uint_as_float(half ? rb[8 * v + 2 * e] : ra[8 * v + 2 * e]);
                            float x1 = __uint_as_float(half ? rb[8 * v + 2 * e + 1] : ra[8 * v + 2 * e + 1]);
                            if (p.per_column) {
                                const float2 s = scale_pair(p.S, col + 8 * v + 2 * e);
                                x0 *= s.x * kWeightUnscale;
                                x1 *= s.y * kWeightUnscale;
                            } else {
                                unscale(x0, x1);
                            }
                            o[e] = pack_bf16x2(x0, x1);
                        }
                        // 128-byte rows, 16-byte chunk index XOR (row % 8): the layout of the 128B-swizzled tensor map
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(epi_tma + lane * 128 + (((half * 4 + v) ^ (lane & 7)) << 4)), "r"(o[0]),
                                     "r"(o[1]), "r"(o[2]), "r"(o[3])
                                     : "memory");
                    }
                }
                if (pp + 1 < TN / 64) {
                    tmem_ld_32x32b_x32(t_row + (pp + 1) * 64, ra);
                    tmem_ld_32x32b_x32(t_row + (pp + 1) * 64 + 32, rb);
                } else {
                    release();
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {  // (rows past m are clipped by the tensor map)
                    tma_store_2d(&tmap_c, epi_tma, nt * TN + pp * 64, mt * kTileM + rank * kHalf + quarter * 32);
                    bulk_commit_group();
                    // the other tile, written two rounds ago, has been read
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                }
                __syncwarp();
            }
        }
        if (lane == 0) bulk_wait_group0();  // this warp's TMA stores are complete before the CTA may exit
    } else if (warp == kWordWarp) {
        // ---------------- TMA: packed words and scales of this CTA's 128 columns (they depend on no kernel before) ----------------
        if (lane == 0) {
            bool ok = true;
            int s = 0;
            uint32_t ph = 1;
            while (ok && wi.next(mt, nt, sp, ki0, ki1, slab)) {
                const int ki1e = ki1 + (ki0 == 0 ? p.lora_steps : 0), col = nt * TN + rank * kCols;
                for (int ki = ki0; ki < ki1e; ++ki) {
                    if (!(ok = mbar_wait(word_empty(s), ph, abort_flag, p.status, 0x800u | s, p.wait_limit_ns))) break;
                    const uint32_t dst = word_base + s * C::kWordSlotBytes;
                    if (ki >= ki1) {  // a LoRA step has no words; its slot passes through the ring empty
                        mbar_arrive(word_full(s));
                    } else {
                        mbar_arrive_expect_tx(word_full(s), C::kWordBytes + (p.per_column ? 0 : C::kScaleBytes));
                        tma_load_2d(dst, &tmap_w, 2 * col, ki * (BK / 16), word_full(s));
                        if (!p.per_column) tma_load_2d(dst + C::kWordBytes, &tmap_s, col, ki >> 1, word_full(s));
                    }
                    if (++s == kWordSlots) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else {
        // ---------------- dequant: this CTA's 128 columns, packed int4 -> bf16 B tile ----------------
        const int team = (warp - kDequantWarp0) % kTeams, dw = (warp - kDequantWarp0) / kTeams;  // warp `dw` of team `team`
        const int qd = lane & 3, c = lane >> 2;
        // 64-column chunk and first 16-row K tile of a stage: two chunks, K tiles kt0 and kt0 + 2, or one chunk and one K tile
        const int ch = TN == 256 ? dw & 1 : 0, kt0 = TN == 256 ? dw >> 1 : dw;
        // row (= column of B) 64 ch + 8t + c, 128 B per row; 16-byte chunk (2 kt + half) ^ c
        const uint32_t row0 = smem_base + kABytes + static_cast<uint32_t>(ch * 64 + c) * 128u + 4u * qd;
        const uint32_t words = word_base + kt0 * (kCols * 8) + ch * 512 + lane * 16, scales = word_base + C::kWordBytes + ch * 128 + c * 16;
        const uint32_t leader_full0 = map_to_cta(full(0), 0);
        int skip = team;  // steps until this team's next one
        int s = team, ws = team;
        uint32_t ph = 1, wph = 0;
        bool ok = true, w_ready = false, s_ready = false;  // the next waits, asked ahead
        while (wi.next(mt, nt, sp, ki0, ki1, slab)) {
            const int ki1e = ki1 + (ki0 == 0 ? p.lora_steps : 0);
            int ki = ki0 + skip;
            for (; ki < ki1e; ki += kTeams) {  // (to the end, whatever a wait says: see warp_all)
                if (ok && !w_ready) ok = mbar_wait(word_full(ws), wph, abort_flag, p.status, 0x900u | ws, p.wait_limit_ns);
                uint4 w[C::kBlocks], sc = make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);  // (per-column scales come in the epilogue)
                WeightScale s2[4];  // of columns 16j + c, 16j + 8 + c
                if (ki < ki1) {
#pragma unroll
                    for (int b = 0; b < C::kBlocks; ++b) w[b] = lds_v4(words + ws * C::kWordSlotBytes + b * (2 * kCols * 8));
                    if (!p.per_column) sc = lds_v4(scales + ws * C::kWordSlotBytes);
                    s2[0] = weight_scale(sc.x), s2[1] = weight_scale(sc.y), s2[2] = weight_scale(sc.z), s2[3] = weight_scale(sc.w);
                }
                __syncwarp();
                if (ok && lane == 0) mbar_arrive(word_empty(ws));  // in registers: the slot can load again
                if (ok && !s_ready) ok = mbar_wait(empty(s), ph, abort_flag, p.status, 0x600u | s, p.wait_limit_ns);
                if (ki < ki1) {
#pragma unroll
                    for (int b = 0; b < C::kBlocks; ++b) {
                        const int kt = kt0 + 2 * b;
                        dequant_block(w[b], s2, row0 + s * kStageBytes, static_cast<uint32_t>((2 * kt) ^ c) << 4, static_cast<uint32_t>((2 * kt + 1) ^ c) << 4);
                    }
                }
                fence_proxy_async_smem();  // every thread publishes its own stores to the async proxy
                __syncwarp();
                if (ok && lane == 0) arrive_cluster(leader_full0 + 8u * s);
                if ((s += kTeams) >= kStages) {
                    s -= kStages;
                    ph ^= 1;
                }
                if ((ws += kTeams) >= kWordSlots) {
                    ws -= kWordSlots;
                    wph ^= 1;
                }
                w_ready = mbar_test(word_full(ws), wph);
                s_ready = mbar_test(empty(s), ph);
            }
            skip = ki - ki1e;
        }
    }

    __syncwarp();
    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // A wait has run out, and every warp of this CTA has given up.  The other one would learn of it by its own limit.  Copies and MMAs that have
        // been issued take microseconds, in whatever state the rings are, and land during this pause; neither CTA leaves before it.
        st_cluster_u32(map_to_cta(smem_u32(const_cast<uint32_t *>(abort_flag)), cluster_ctarank() ^ 1), 1u);
        pause_ns(20ull * 1000 * 1000);
    }
    __syncwarp();
    cluster_sync_all();  // nothing of the pair is in flight any more: MMAs, arrivals, tensor memory
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(static_cast<uint32_t>(C::kTmemCols)) : "memory");
    }
}

}  // namespace

// Where the MMAs need 512 cycles per 64 K of a tile of 256 columns, the kernel takes about 540 (16384 x 9216 x 9216: 1367 TFLOP/s at
// the 1.17 GHz that the power cap leaves; single CTAs 1056).  Writing the dequantised weight out first and feeding both operands by
// TMA reaches 515 cycles, at 1.10 GHz: the bytes through L2 cost more power than the arithmetic saves (2380 us against 2036).
// Tiles of 128 columns are for problems that have too few of the wide ones (per 64 K 0.19 us against 0.28).
int launch_pair(const GemmArgs &a, PrefillParams p, int tile_n, const CUtensorMap &tmap_c, const CUtensorMap &tmap_p) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return KILN_W4A16_ERR_CUDA;
    auto encode = [&](CUtensorMap *map, CUtensorMapDataType type, int elem, const void *ptr, long long cols, int rows, int box_cols, int box_rows,
                      CUtensorMapSwizzle swizzle) {
        const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)}, strides[1] = {static_cast<cuuint64_t>(cols) * elem};
        const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)}, estr[2] = {1, 1};
        return enc(map, type, 2, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    auto operand = [&](CUtensorMap *map, const void *ptr, int cols, int rows, int box_rows) {
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, cols, rows, BK, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    const int cols = tile_n / 2;  // columns per CTA
    CUtensorMap tmap_a, tmap_w, tmap_s, tmap_t, tmap_lb;
    // (test hook: boxes of eight rows less than the kernel announces, so that its waits for them run out)
    if (!operand(&tmap_a, a.A, a.k, a.m, p.test_drop_a_load >= 0 ? kHalf - 8 : kHalf) ||
        !encode(&tmap_w, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, a.B, 2ll * a.n, a.k / 16, 2 * cols, BK / 16, CU_TENSOR_MAP_SWIZZLE_NONE))
        return KILN_W4A16_ERR_CUDA;
    tmap_s = tmap_w;  // (unused with per-column scales)
    if (!p.per_column && !encode(&tmap_s, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, a.S, a.n, a.k / 128, cols, 1, CU_TENSOR_MAP_SWIZZLE_NONE))
        return KILN_W4A16_ERR_CUDA;
    tmap_t = tmap_lb = tmap_a;  // (unused without a LoRA delta)
    if (p.lora_steps > 0 && (!operand(&tmap_t, a.lora_t, a.lora_r, a.m, kHalf) || !operand(&tmap_lb, a.lora_b, a.lora_r, a.n, cols)))
        return KILN_W4A16_ERR_CUDA;
    const bool wide = tile_n == 256;
    const auto kernel = wide ? w4a16_pair_kernel<256> : w4a16_pair_kernel<128>;
    const int smem = wide ? Cfg<256>::kSmemBytes : Cfg<128>::kSmemBytes;
    static bool attr_set[2][64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !attr_set[wide][dev]) {
        if (int rc = record_cuda_error(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))) return rc;
        attr_set[wide][dev] = true;
    }
    const int units = p.m_tiles * p.n_tiles * p.splits, pairs = device_sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (p.stream_k || units > pairs ? pairs : units));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = a.stream;
    cudaLaunchAttribute attr = pdl_attribute();
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    note_launch();
    return record_cuda_error(cudaLaunchKernelEx(&cfg, kernel, tmap_a, tmap_w, tmap_s, tmap_c, tmap_p, tmap_t, tmap_lb, p));
}

}  // namespace kiln
