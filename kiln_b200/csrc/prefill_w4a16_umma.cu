// Prefill-shape W4A16 GEMM for sm_100a: TMA-fed tcgen05 (UMMA) GEMM with TMEM accumulators
// and the int4 -> bf16 dequant fused into the shared-memory staging of the B operand.
//
// Replaces the reference's `Marlin<256,{1..4},16,4,4,8>` path
// (kiln-marlin-gemm/csrc/marlin_kernel.cu:197-700, dispatch :784-816: 64-row m-tiles,
// mma.sync, host loop over M) with a persistent, warp-specialised kernel:
//
//   warp 0      TMA producer: activation tiles A[128 x 64] bf16 -> 128B-swizzled smem
//   warp 1      MMA issuer: tcgen05.mma 128 x BN x 16, fp32 accumulators in TMEM (two buffers);
//               also owns the TMEM allocation
//   warps 2-5   epilogue: tcgen05.ld TMEM -> registers -> bf16 -> global (or fp32 split-K slabs)
//   warps 6-13  dequant: packed int4 words (16 B per lane, straight from global/L2) ->
//               bf16 (nib-8)*scale -> the K-major 128B-swizzled B tile the MMA reads
//
// The Marlin fragment layout maps onto the swizzled K-major tile with conflict-free 4-byte
// stores: lane (qd, c) owns K-pairs (2qd, 2qd+1), (2qd+8, 2qd+9) of column 8t + c, and the
// 128B swizzle XORs the 16-byte chunk index with (column % 8) = c.
//
// Most prefill runs on CTA pairs (pair_w4a16_umma.cu), which shares the tile walk, the reduction and the fix-up with this kernel.
// It keeps what pairs do not pay for or do not take: few row tiles of few columns, the fused all-gather, and problems of at most
// 128 rows that the small-batch kernel does not take.  This file also holds the planner that picks between the three.
//
// Every wait in the kernel is bounded: a wait that runs out records an error code in the
// device status word, raises a CTA-wide abort flag that every other wait polls, and the CTA
// drains its outstanding TMA copies, frees its TMEM and returns.
#include <algorithm>
#include <mutex>

#include "w4a16_prefill.cuh"

namespace kiln {
namespace {

constexpr int kDequantWarp0 = 6;
constexpr int kNumEpilogueThreads = 4 * 32;

// MT = M-tiles of 128 rows that share one dequantised B stage.  With MT = 2 every weight is dequantised
// once per 256 rows instead of once per 128, which halves the dequant work per MMA flop; the two
// accumulators then take both TMEM buffers, so the epilogue only partly overlaps the next tile.
// DG = dequant groups: the DW dequant warps are split into DG teams that fill alternate stages, so the
// dequant of stage s+1 runs beside that of stage s instead of after it.
// KP = MMA issuers per M-tile: with KP = 2 (128-column tiles of one M-tile, which are bound by the ~105 cycles one thread
// needs per tcgen05.mma) a second warp issues the upper two of a K-step's four MMAs into an accumulator of its own, and
// the epilogue adds the two accumulators.
// KS = 64-deep K atoms per pipeline stage: with KS = 2 a stage holds 128 K-elements (one scale group), which halves the
// barrier round trips, waits and commits per K of the small tiles that are bound by them.
// AR = activation rows that a stage holds per 64-deep atom: 128 (a whole M-tile), or 64 when the problem has at most 64
// rows.  The MMA still reads 128 rows; rows 64..127 then alias whatever follows the atom in the stage (the next atom or
// the weight tile: finite or not, they only reach accumulator rows that are never stored).  The 8 KB saved per atom buy
// a deeper pipeline (4 stages of 48 KB instead of 3 of 64 KB), and these problems are bound by the round trip
// stage free -> TMA load / dequant -> MMA -> commit, not by any throughput.
template <int BN, int MT = 1, int DW = 8, int DG = 2, int KP = 1, int KS = 1, int AR = BM>
struct Cfg {
    static_assert(KP == 1 || (KP == 2 && MT == 1 && BN == 128), "K-parity issuers: one M-tile of 128 columns only");
    static_assert(KS == 1 || KS == 2, "one or two 64-deep atoms per stage");
    static_assert(AR == BM || (AR == 64 && MT == 1), "half-height activation atoms: one M-tile only");
    static constexpr int kAAtomBytes = MT * AR * BK * 2;  // one 64-deep atom of the activation tile(s)
    static constexpr int kBAtomBytes = BN * BK * 2;
    static constexpr int kIssuers = MT == 2 ? 2 : KP;
    static constexpr int kGroupWarps = DW / DG;
    // producer, MMA, 4 epilogue and DW dequant warps (16 dequant warps were measured no faster than 8)
    // MT == 2 adds a second MMA-issuing warp (the last one): each issuer owns one M-tile of the pair
    static constexpr int kMmaWarp2 = 6 + DW;
    static constexpr int kThreads = (6 + DW + (kIssuers == 2 ? 1 : 0)) * 32;
    static constexpr int kABytes = kAAtomBytes * KS;  // 16 KB per M-tile and atom
    static constexpr int kBBytes = kBAtomBytes * KS;  // 32 / 16 KB per atom
    static constexpr int kStages = (192 * 1024) / (kABytes + kBBytes);
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kTmemCols = 2 * BN * KP;
    static constexpr int kBlocksPerStage = (BN / 64) * 4 * KS;  // 512-byte packed blocks per stage
    static constexpr int kBlocksPerWarp = kBlocksPerStage / kGroupWarps;
    static_assert(kBlocksPerStage % kGroupWarps == 0 && kGroupWarps % (BN / 64) == 0,
                  "a dequant team must divide the packed blocks of a stage and keep one chunk per warp");
    static constexpr int kBarrierBytes = 1024;
    static constexpr int kSmemBytes = kStages * kStageBytes + kBarrierBytes + 4 * 2 * kEpiWarpBytes + 1024;  // + alignment slack
    // instruction descriptor: D fp32, A/B bf16, both K-major, N = BN, M = 128
    static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(BN >> 3) << 17) |
                                       (static_cast<uint32_t>(BM >> 4) << 24);
};

template <int NBLK>
struct DequantRegs {
    uint4 w[NBLK];
};

template <int BN, int MT, int DW, int DG, int KP, int KS, int AR>
__global__ void __launch_bounds__((6 + DW + ((MT == 2 || KP == 2) ? 1 : 0)) * 32, 1)
w4a16_prefill_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_c,
                     const __grid_constant__ CUtensorMap tmap_p, const __grid_constant__ CUtensorMap tmap_t,
                     const __grid_constant__ CUtensorMap tmap_lb, const PrefillParams p) {
    using C = Cfg<BN, MT, DW, DG, KP, KS, AR>;
    using Regs = DequantRegs<C::kBlocksPerWarp>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + C::kStages * C::kStageBytes;
    auto full_a = [&](int s) { return bar_base + 8u * s; };
    auto full_b = [&](int s) { return bar_base + 8u * s; };  // same barrier as full_a: one wait per K-step for the issuer
    auto empty = [&](int s) { return bar_base + 8u * (2 * C::kStages + s); };
    auto tmem_full = [&](int a) { return bar_base + 8u * (3 * C::kStages + a); };
    auto tmem_empty = [&](int a) { return bar_base + 8u * (3 * C::kStages + 2 + a); };
    const uint32_t epi_base = bar_base + C::kBarrierBytes;
    uint8_t *bar_gen = smem_gen + C::kStages * C::kStageBytes;
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(bar_gen + 8 * (3 * C::kStages + 4));
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(bar_gen + 8 * (3 * C::kStages + 4) + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            // one "stage full" barrier: the TMA producer (1 arrival + the tile's bytes) and the threads of the dequant team
            mbar_init(full_a(s), 1 + C::kGroupWarps * 32);
            mbar_init(empty(s), C::kIssuers);  // one tcgen05.commit per MMA issuer
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tmem_full(a), KP);  // one tcgen05.commit per issuer that writes into this buffer
            mbar_init(tmem_empty(a), kNumEpilogueThreads);
        }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t *>(tmem_ptr_slot))),
                     "r"(static_cast<uint32_t>(C::kTmemCols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_slot;
    // Programmatic dependent launch: the next kernel in the stream may start on SMs this grid has left (or never used) and
    // run its prologue and its weight stream there.  In this kernel only the activation loads and every global write
    // order themselves after the previous kernel (griddepcontrol.wait); the packed weights and scales never depend on it.
    pdl_launch_dependents();

    const int chunks_n = p.n >> 6;
    int mt, nt, sp, ki0, ki1, slab;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            pdl_wait();  // the activations may be the previous kernel's output
            uint32_t it = 0;
            bool ok = true;
            WorkIter wi(p, blockIdx.x, gridDim.x);
            while (ok && wi.next(mt, nt, sp, ki0, ki1, slab)) {
                const int ki1e = ki1 + ((KS == 1 && ki0 == 0) ? p.lora_steps : 0);  // + the LoRA steps of the tile
                for (int ki = ki0; ki < ki1e; ++ki, ++it) {
                    const int s = it % C::kStages;
                    const uint32_t ph = (it / C::kStages) & 1;
                    if (!(ok = mbar_wait(empty(s), ph ^ 1, abort_flag, p.status, 0x100u | s, p.wait_limit_ns))) break;
                    if (ki >= ki1) {  // LoRA step: both operand tiles come by TMA (rows past m, columns past r read zero)
                        mbar_arrive_expect_tx(full_a(s), C::kAAtomBytes + C::kBAtomBytes);
                        tma_load_2d(smem_base + s * C::kStageBytes, &tmap_t, (ki - ki1) * BK, mt * (BM * MT), full_a(s));
                        tma_load_2d(smem_base + s * C::kStageBytes + C::kABytes, &tmap_lb, (ki - ki1) * BK, nt * BN, full_a(s));
                        continue;
                    }
                    mbar_arrive_expect_tx(full_a(s), C::kABytes);
                    if (static_cast<int>(it) != p.test_drop_a_load)
#pragma unroll
                        for (int at = 0; at < KS; ++at)
                            tma_load_2d(smem_base + s * C::kStageBytes + at * C::kAAtomBytes, &tmap_a, (ki * KS + at) * BK, mt * (BM * MT),
                                        full_a(s));
                }
            }
            if (!ok) {
                // drain: wait (bounded, ignoring the abort flag) for copies already issued
                const uint32_t first = it >= static_cast<uint32_t>(C::kStages) ? it - C::kStages : 0;
                for (uint32_t j = first; j < it; ++j) {
                    const int s = j % C::kStages;
                    const uint32_t ph = (j / C::kStages) & 1;
                    mbar_wait_quiet(full_a(s), ph);
                }
            }
        }
    } else if (warp == 1 || (C::kIssuers == 2 && warp == C::kMmaWarp2)) {
        // ---------------- MMA issuer(s) ----------------
        // One thread issues about one tcgen05.mma per ~105 cycles and spends ~400 more per K-step on the
        // barrier waits and the commit, which is more than the 1024 cycles the eight 128 x 256 x 16 MMAs of a
        // pair execute in.  With MT == 2 the two M-tiles therefore have one issuer each (warp 1: tile 0, the
        // last warp: tile 1); their MMAs go to different accumulators and need no order between them.  With
        // KP == 2 (one M-tile of 128 columns, whose four MMAs per K-step execute in 256 cycles) the two issuers
        // share the K-step instead: warp 1 issues MMAs 0 and 1, the last warp MMAs 2 and 3, each into an
        // accumulator of its own, and the epilogue adds the two (gate+up M=64: 20.6 -> 18.7 us).
        if (lane == 0) {
            const int h0 = (MT == 2 && warp != 1) ? 1 : 0, h1 = MT == 2 ? h0 + 1 : 1;
            const int q = (KP == 2 && warp != 1) ? 1 : 0;  // K-parity issuer: MMAs 2q, 2q+1 of every K-step, accumulator q
            uint32_t it = 0, tile = 0;
            bool ok = true;
            WorkIter wi(p, blockIdx.x, gridDim.x);
            for (; ok && wi.next(mt, nt, sp, ki0, ki1, slab); ++tile) {
                // MT == 1: the two TMEM buffers alternate between tiles.  MT == 2: buffer h holds M-tile h of the pair.
                const uint32_t acc0 = MT == 1 ? (tile & 1) : 0u, acc_ph = MT == 1 ? ((tile >> 1) & 1) : (tile & 1);
                const int ki1e = ki1 + ((KS == 1 && ki0 == 0) ? p.lora_steps : 0);  // + the LoRA steps of the tile
                for (int ki = ki0; ki < ki1e; ++ki, ++it) {
                    const int s = it % C::kStages;
                    const uint32_t ph = (it / C::kStages) & 1;
                    if (!(ok = mbar_wait(full_a(s), ph, abort_flag, p.status, 0x300u | s, p.wait_limit_ns))) break;
                    tc_fence_after();
                    for (int h = h0; h < h1; ++h) {
                        const uint32_t acc = acc0 + h;
                        if (ki == ki0) {  // first write into this accumulator: the epilogue must have drained it
                            if (!(ok = mbar_wait(tmem_empty(acc), acc_ph ^ 1, abort_flag, p.status, 0x200u | acc, p.wait_limit_ns))) break;
                            tc_fence_after();
                        }
                        constexpr int kPer = (BK / 16) * KS / KP;  // MMAs of this issuer per stage and M-tile
#pragma unroll
                        for (int j = 0; j < kPer; ++j) {
                            const int kg = q * kPer + j, at = kg >> 2, kw = kg & 3;  // 64-deep atom, 16-deep slice in it
                            const uint64_t a_desc = make_smem_desc(smem_base + s * C::kStageBytes + at * C::kAAtomBytes + h * (BM * BK * 2));
                            const uint64_t b_desc = make_smem_desc(smem_base + s * C::kStageBytes + C::kABytes + at * C::kBAtomBytes);
                            umma_bf16(tmem_base + (acc * KP + q) * BN, a_desc + 2 * kw, b_desc + 2 * kw, C::kIdesc,
                                      (ki > ki0 || j > 0) ? 1u : 0u);
                        }
                        if (ki == ki1e - 1) umma_commit(tmem_full(acc));  // accumulator h is complete
                    }
                    if (!ok) break;
                    umma_commit(empty(s));  // this issuer's MMAs have read the stage; the slot is free after all issuers'
                }
            }
        }
    } else if (warp < kDequantWarp0) {
        // ---------------- epilogue ----------------
        const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 are the ones this warp may read
        pdl_wait();  // C (or the workspace) may still be read or written by the previous kernel
        uint32_t tile = 0;
        bool ok = true;
        WorkIter wi(p, blockIdx.x, gridDim.x);
        for (; ok && wi.next(mt, nt, sp, ki0, ki1, slab); ++tile) {
            const uint32_t acc0 = MT == 1 ? (tile & 1) : 0u, acc_ph = MT == 1 ? ((tile >> 1) & 1) : (tile & 1);
#pragma unroll 1
            for (int h = 0; h < MT && ok; ++h) {
            const uint32_t acc = acc0 + h;
            if (!(ok = warp_all(mbar_wait(tmem_full(acc), acc_ph, abort_flag, p.status, 0x500u | acc, p.wait_limit_ns)))) break;
            tc_fence_after();
            const int row = (mt * MT + h) * BM + quarter * 32 + lane;
            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * KP * BN;
            if (slab < 0 && p.splits == 1) {
                // bf16 result, 64 columns per round.  A thread owns one row of the accumulator; the 128-byte pieces go
                // through a per-warp shared-memory tile so that the global (or peer, over NVLink) stores are 128
                // contiguous bytes per row and four rows per instruction instead of 16 scattered bytes.  The TMEM loads
                // of round i+1 are issued as soon as the registers of round i are in shared memory, so their latency
                // hides behind the stores, and the accumulator is handed back to the MMA issuer right after the
                // last load has landed, not after the last store.
                // This GPU's own copy of the result (the only copy when the all-gather is not fused) leaves through one
                // asynchronous TMA store of the 32 x 64 tile per round; copies for other GPUs (fused all-gather) are read
                // back from the same tile and stored over NVLink, 128 contiguous bytes of four rows per instruction, or
                // once through the NVSwitch multicast address.
                const bool tma_out = (p.n_peers == 0 && !p.mc_c) || p.self_peer >= 0;
                const bool remote_out = p.mc_c || p.n_peers > (p.self_peer >= 0 ? 1 : 0);
                // two staging tiles per warp, used in turn: the TMA store of one round reads its tile while the next round fills the other
                const uint32_t epi_tma0 = epi_base + static_cast<uint32_t>(warp - 2) * (2 * kEpiWarpBytes);  // 1024-byte aligned swizzle atoms
                const int x0_out = (p.n_peers > 0 ? p.col0 : 0) + nt * BN;  // first column of the tile in the output buffer
                uint32_t ra[32], rb[32];
                if constexpr (KP == 2) {
                    // two accumulators (one per K-parity issuer) to add: 32 columns of each per half-round; the loads of the
                    // next half-round are in flight while a finished 64-column tile is stored
                    tmem_ld_32x32b_x32(t_row, ra);
                    tmem_ld_32x32b_x32(t_row + BN, rb);
#pragma unroll 1
                    for (int hh = 0; hh < BN / 32; ++hh) {
                        const int pp = hh >> 1, half = hh & 1;
                        const uint32_t epi_tma = epi_tma0 + static_cast<uint32_t>(pp & 1) * kEpiWarpBytes;
                        const int col = nt * BN + hh * 32;
                        tmem_ld_wait();
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            uint32_t o[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                float x0 = __uint_as_float(ra[8 * v + 2 * e]) + __uint_as_float(rb[8 * v + 2 * e]);
                                float x1 = __uint_as_float(ra[8 * v + 2 * e + 1]) + __uint_as_float(rb[8 * v + 2 * e + 1]);
                                if (p.per_column) {
                                    const float2 s = scale_pair(p.S, col + 8 * v + 2 * e);
                                    x0 *= s.x * kWeightUnscale;
                                    x1 *= s.y * kWeightUnscale;
                                } else {
                                    unscale(x0, x1);
                                }
                                o[e] = pack_bf16x2(x0, x1);
                            }
                            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(
                                             epi_tma + lane * 128 + (((half * 4 + v) ^ (lane & 7)) << 4)),
                                         "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3])
                                         : "memory");
                        }
                        if (hh + 1 < BN / 32) {
                            tmem_ld_32x32b_x32(t_row + (hh + 1) * 32, ra);
                            tmem_ld_32x32b_x32(t_row + BN + (hh + 1) * 32, rb);
                        } else {
                            tc_fence_before();
                            mbar_arrive(tmem_empty(acc));  // every column of both accumulators is in registers or shared memory
                        }
                        if (half == 0) continue;
                        if (tma_out) fence_proxy_async_smem();
                        __syncwarp();
                        if (tma_out && lane == 0) {
                            tma_store_2d(&tmap_c, epi_tma, x0_out + pp * 64, (mt * MT + h) * BM + quarter * 32);
                            bulk_commit_group();
                        }
                        if (remote_out) {
                            const int piece = lane & 7;
                            const int col_out = p.col0 + nt * BN + pp * 64 + piece * 8;
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const int rl = i * 4 + (lane >> 3);
                                const int grow = (mt * MT + h) * BM + quarter * 32 + rl;
                                uint4 val;
                                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                             : "=r"(val.x), "=r"(val.y), "=r"(val.z), "=r"(val.w)
                                             : "r"(epi_tma + rl * 128 + ((piece ^ (rl & 7)) << 4)));
                                if (grow < p.m) {
                                    if (p.mc_c) {
                                        asm volatile("multimem.st.weak.global.v4.bf16x2 [%0], {%1,%2,%3,%4};" ::"l"(
                                                         p.mc_c + static_cast<size_t>(grow) * p.ldc + col_out),
                                                     "r"(val.x), "r"(val.y), "r"(val.z), "r"(val.w)
                                                     : "memory");
                                    } else {
                                        for (int pe = 0; pe < p.n_peers; ++pe)
                                            if (pe != p.self_peer)
                                                *reinterpret_cast<uint4 *>(p.peer_c[pe] + static_cast<size_t>(grow) * p.ldc + col_out) = val;
                                    }
                                }
                            }
                        }
                        if (tma_out && lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        __syncwarp();
                    }
                    continue;  // the accumulators were released above
                }
                tmem_ld_32x32b_x32(t_row, ra);
                tmem_ld_32x32b_x32(t_row + 32, rb);
#pragma unroll 1
                for (int pp = 0; pp < BN / 64; ++pp) {
                    const uint32_t epi_tma = epi_tma0 + static_cast<uint32_t>(pp & 1) * kEpiWarpBytes;
                    tmem_ld_wait();
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int col = nt * BN + pp * 64 + half * 32;
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
                            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(
                                             epi_tma + lane * 128 + (((half * 4 + v) ^ (lane & 7)) << 4)),
                                         "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3])
                                         : "memory");
                        }
                    }
                    if (pp + 1 < BN / 64) {
                        tmem_ld_32x32b_x32(t_row + (pp + 1) * 64, ra);
                        tmem_ld_32x32b_x32(t_row + (pp + 1) * 64 + 32, rb);
                    } else {
                        tc_fence_before();
                        mbar_arrive(tmem_empty(acc));  // every column of this accumulator is in registers or shared memory
                    }
                    if (tma_out) fence_proxy_async_smem();
                    __syncwarp();
                    if (tma_out && lane == 0) {
                        // (full 128-byte lines, no load back from shared memory; rows past m are clipped by the tensor map)
                        tma_store_2d(&tmap_c, epi_tma, x0_out + pp * 64, (mt * MT + h) * BM + quarter * 32);
                        bulk_commit_group();
                    }
                    if (remote_out) {
                        const int piece = lane & 7;
                        const int col_out = p.col0 + nt * BN + pp * 64 + piece * 8;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int rl = i * 4 + (lane >> 3);
                            const int grow = (mt * MT + h) * BM + quarter * 32 + rl;
                            uint4 val;
                            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                         : "=r"(val.x), "=r"(val.y), "=r"(val.z), "=r"(val.w)
                                         : "r"(epi_tma + rl * 128 + ((piece ^ (rl & 7)) << 4)));
                            if (grow < p.m) {
                                if (p.mc_c) {
                                    asm volatile("multimem.st.weak.global.v4.bf16x2 [%0], {%1,%2,%3,%4};" ::"l"(
                                                     p.mc_c + static_cast<size_t>(grow) * p.ldc + col_out),
                                                 "r"(val.x), "r"(val.y), "r"(val.z), "r"(val.w)
                                                 : "memory");
                                } else {
                                    // column-parallel all-gather fused into the epilogue: plain stores into the other GPUs' buffers
                                    for (int pe = 0; pe < p.n_peers; ++pe)
                                        if (pe != p.self_peer)
                                            *reinterpret_cast<uint4 *>(p.peer_c[pe] + static_cast<size_t>(grow) * p.ldc + col_out) = val;
                                }
                            }
                        }
                    }
                    // this tile is rewritten two rounds from now: the TMA store of the round before this one has read the
                    // other tile (the next round's TMEM loads are already in flight), and every lane is done with this one
                    if (tma_out && lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    __syncwarp();
                }
                continue;  // the accumulator was released above
            }
#pragma unroll 1
            for (int cc = 0; cc < BN / 32; ++cc) {
                uint32_t r[32];
                tmem_ld_32x32b_x32(t_row + cc * 32, r);
                if constexpr (KP == 2) {  // add the second K-parity accumulator
                    uint32_t r2[32];
                    tmem_ld_32x32b_x32(t_row + BN + cc * 32, r2);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(r2[i]));
                }
                tmem_ld_wait();
                // fp32 piece of a split tile, 32 x 32 at a time through a swizzled staging tile and TMA: a stream-K piece to its
                // tile-shaped slab, a K split to its slab of C (rows past m are clipped)
                const uint32_t stage = epi_base + static_cast<uint32_t>(warp - 2) * (2 * kEpiWarpBytes) + static_cast<uint32_t>(cc & 1) * kEpiWarpBytes;
#pragma unroll
                for (int v = 0; v < 8; ++v)
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(stage + lane * 128 + ((v ^ (lane & 7)) << 4)), "r"(r[4 * v]), "r"(r[4 * v + 1]),
                                 "r"(r[4 * v + 2]), "r"(r[4 * v + 3])
                                 : "memory");
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (slab >= 0)
                        tma_store_3d(&tmap_p, stage, cc * 32, h * BM + quarter * 32, slab);
                    else
                        tma_store_3d(&tmap_p, stage, nt * BN + cc * 32, (mt * MT + h) * BM + quarter * 32, sp);
                    bulk_commit_group();
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the other staging tile has been read
                }
                __syncwarp();
            }
            tc_fence_before();
            mbar_arrive(tmem_empty(acc));
            }
        }
        if (lane == 0) bulk_wait_group0();  // this warp's TMA stores are complete before the CTA may exit
    } else {
        // ---------------- dequant: packed int4 -> bf16 B tile ----------------
        const int dw = (warp - kDequantWarp0) / DG, team = (warp - kDequantWarp0) % DG;  // warp `dw` of team `team`
        const int qd = lane & 3, c = lane >> 2;
        constexpr int kChunksPerTile = BN / 64;
        uint32_t it_base = 0;  // stages issued before this piece of work (all teams count alike)
        bool ok = true;
        int cur_group = -1;
        WeightScale s2[4];  // of columns 16j + c, 16j + 8 + c of this warp's chunk
        WorkIter wi(p, blockIdx.x, gridDim.x);
        while (ok && wi.next(mt, nt, sp, ki0, ki1, slab)) {
            cur_group = -1;
            auto load_regs = [&](Regs &d, int ki) {
#pragma unroll
                for (int b = 0; b < C::kBlocksPerWarp; ++b) {
                    const int blk = dw + C::kGroupWarps * b;
                    const int ch = blk % kChunksPerTile, kt = blk / kChunksPerTile;
                    const size_t idx =
                        (static_cast<size_t>(ki * (4 * KS) + kt) * chunks_n + nt * kChunksPerTile + ch) * 32 + lane;
                    d.w[b] = ld_stream_v4(p.B + idx);
                }
            };
            auto group_of = [](int ki) { return KS == 2 ? ki : (ki >> 1); };  // scale group of a stage (KS == 2: a stage is a group)
            auto load_scales = [&](int g) {
                return ld_stream_v4(reinterpret_cast<const uint4 *>(
                    p.S + static_cast<size_t>(g) * p.n + (nt * kChunksPerTile + dw % kChunksPerTile) * 64 + 8 * c));
            };
            // this team's K-steps of the piece: those whose stage number is congruent to `team`
            const int kf = ki0 + static_cast<int>((static_cast<uint32_t>(team) + DG - it_base % DG) % DG);
            // Packed words and scales of this team's next three K-steps are always in flight, each step's in registers of
            // its own: the loop below is unrolled three times so that no register with a pending load is ever copied (a
            // copy would wait for the load and shrink the three round trips in flight to one).
            Regs rw[3];
            uint4 rs[3];
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                rs[u] = make_uint4(0, 0, 0, 0);
                if (kf + u * DG < ki1) {
                    load_regs(rw[u], kf + u * DG);
                    if (!p.per_column) rs[u] = load_scales(group_of(kf + u * DG));
                }
            }
            for (int kb = kf; kb < ki1 && ok; kb += 3 * DG) {
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const int ki = kb + u * DG;
                if (ki >= ki1) break;
                Regs &r0 = rw[u];
                const uint32_t it = it_base + static_cast<uint32_t>(ki - ki0);
                const int s = it % C::kStages;
                const uint32_t ph = (it / C::kStages) & 1;
                // scales of this K-step's group (all blocks of a warp share one chunk: blk % kChunksPerTile == dw % ..)
                const int g = p.per_column ? 0 : group_of(ki);
                if (g != cur_group) {
                    cur_group = g;
                    // (per-column scales are applied in the epilogue)
                    const uint4 sw = p.per_column ? make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u) : rs[u];
                    s2[0] = weight_scale(sw.x), s2[1] = weight_scale(sw.y), s2[2] = weight_scale(sw.z), s2[3] = weight_scale(sw.w);
                }
                if (!(ok = mbar_wait(empty(s), ph ^ 1, abort_flag, p.status, 0x600u | s, p.wait_limit_ns))) break;
                const uint32_t b_tile = smem_base + s * C::kStageBytes + C::kABytes;
#pragma unroll
                for (int b = 0; b < C::kBlocksPerWarp; ++b) {
                    const int blk = dw + C::kGroupWarps * b;
                    const int ch = blk % kChunksPerTile, ktb = blk / kChunksPerTile;  // 16-row K tile of the stage: 0 .. 4*KS-1
                    const int at = ktb >> 2, kt = ktb & 3;                            // 64-deep atom, K tile inside it
                    const uint32_t xs[4] = {r0.w[b].x, r0.w[b].y, r0.w[b].z, r0.w[b].w};
                    // row (= column of B) n_local = ch*64 + 8t + c, 128 B per row; 16-byte chunk (2kt + half) ^ c
                    const uint32_t row_base = b_tile + static_cast<uint32_t>(at * C::kBAtomBytes) + static_cast<uint32_t>(ch * 64 + c) * 128u + 4u * qd;
                    const uint32_t sw_lo = static_cast<uint32_t>((2 * kt) ^ c) << 4;
                    const uint32_t sw_hi = static_cast<uint32_t>((2 * kt + 1) ^ c) << 4;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t v[4];
                        dequant_word(xs[j], s2[j], v[0], v[1], v[2], v[3]);
                        const uint32_t r_lo = row_base + static_cast<uint32_t>(16 * j) * 128u;
                        const uint32_t r_hi = r_lo + 8u * 128u;
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_lo + sw_lo), "r"(v[0]) : "memory");
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_lo + sw_hi), "r"(v[1]) : "memory");
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_hi + sw_lo), "r"(v[2]) : "memory");
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(r_hi + sw_hi), "r"(v[3]) : "memory");
                    }
                }
                // every thread publishes its own stores to the async proxy and arrives itself (one arrival per
                // warp behind a __syncwarp was measured slower: 1154 vs 1217 TFLOP/s on gate+up M=8192)
                fence_proxy_async_smem();
                mbar_arrive(full_b(s));
                if (ki + 3 * DG < ki1) {
                    load_regs(rw[u], ki + 3 * DG);
                    if (!p.per_column) rs[u] = load_scales(group_of(ki + 3 * DG));
                }
            }
            }
            it_base += static_cast<uint32_t>(ki1 - ki0);
            // LoRA steps of the tile: the weight-side tile comes by TMA; the team that owns a stage only owes its barrier the arrivals
            if (KS == 1 && ki0 == 0 && p.lora_steps > 0) {
                for (int e = 0; e < p.lora_steps && ok; ++e, ++it_base) {
                    if (it_base % DG != static_cast<uint32_t>(team)) continue;
                    const int s = it_base % C::kStages;
                    const uint32_t ph = (it_base / C::kStages) & 1;
                    if (!(ok = mbar_wait(empty(s), ph ^ 1, abort_flag, p.status, 0x700u | s, p.wait_limit_ns))) break;
                    mbar_arrive(full_b(s));
                }
            }
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(static_cast<uint32_t>(C::kTmemCols))
                     : "memory");
    }
}

// complete sums of four columns, times the factor that the weights were formed at -> bf16
__device__ __forceinline__ uint2 finish4(float4 v, const __half *S, int col, int per_column) {
    v.x *= kWeightUnscale, v.y *= kWeightUnscale, v.z *= kWeightUnscale, v.w *= kWeightUnscale;
    if (per_column) {
        const float2 s0 = scale_pair(S, col), s1 = scale_pair(S, col + 2);
        v.x *= s0.x, v.y *= s0.y, v.z *= s1.x, v.w *= s1.y;
    }
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    return make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
}
__device__ __forceinline__ void add4(float4 &a, const float4 &v) {
    a.x += v.x;
    a.y += v.y;
    a.z += v.z;
    a.w += v.w;
}

// out[m][n] = bf16(sum_s partial[s][m][n]) (* per-column scale).  Four sums per thread, whose loads (at most eight) are all in
// flight at once: the kernel is a few round trips to L2 long and no more.  grid = ceil(m n / 1024), block = 256.
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float *partial, __nv_bfloat16 *C, const __half *S, int m, int n,
                                                            int splits, int per_column) {
    pdl_launch_dependents();
    const size_t slab4 = static_cast<size_t>(m) * n / 4, i = blockIdx.x * static_cast<size_t>(256) + threadIdx.x;
    pdl_wait();  // the partial sums come from the kernel launched just before
    if (i >= slab4) return;
    float4 v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
        if (s < splits) v[s] = reinterpret_cast<const float4 *>(partial)[i + s * slab4];
#pragma unroll
    for (int s = 1; s < 8; ++s)
        if (s < splits) add4(v[0], v[s]);
    reinterpret_cast<uint2 *>(C)[i] = finish4(v[0], S, per_column ? static_cast<int>((i * 4) % n) : 0, per_column);
}

// Stream-K fix-up: finds out which workers covered only a part of the tile's K-steps (the same arithmetic as WorkIter), sums their
// slabs in worker order and writes bf16.  A tile that one worker covered completely was already written by it.  Four sums per
// thread.  (With sixteen blocks per tile and the slabs loaded one after another this pass took 20 us for six tiles.)
// grid = (tiles of the remainder, tile elements / 1024), block = 256.
__global__ void __launch_bounds__(256) streamk_fixup_kernel(const float *partial, __nv_bfloat16 *C, const __half *S, int m, int n, int m_tiles,
                                                            int n_tiles, int group_m, int k_iters, int tile_rows, int bn, int ctas, long long total,
                                                            int first_tile, int per_column) {
    __shared__ int slabs[64];  // (a tile has at most 39 candidates)
    __shared__ int count;
    pdl_launch_dependents();
    const int tr = blockIdx.x, lane = threadIdx.x;
    if (threadIdx.x < 32) {
        const long long t0 = static_cast<long long>(tr) * k_iters, t1 = t0 + k_iters;
        const int r_lo = max(0, static_cast<int>(t0 * ctas / total) - 1), r_hi = min(ctas - 1, static_cast<int>(t1 * ctas / total) + 1);
        int ns = 0;
        for (int r0 = r_lo; r0 <= r_hi; r0 += 32) {
            const int r = r0 + lane;
            const long long g0 = total * r / ctas, g1 = total * (r + 1) / ctas;
            const long long a = g0 > t0 ? g0 : t0, b = g1 < t1 ? g1 : t1;
            const bool part = r <= r_hi && a < b, whole = part && a == t0 && b == t1;
            const unsigned mask = __ballot_sync(0xFFFFFFFFu, part);
            if (part) slabs[ns + __popc(mask & ((1u << lane) - 1))] = 2 * r + (a == g0 ? 0 : 1);
            ns += __popc(mask);
            if (__any_sync(0xFFFFFFFFu, whole)) {
                ns = 0;
                break;
            }
        }
        if (lane == 0) count = ns;
    }
    __syncthreads();
    const int ns = count;
    pdl_wait();  // the slabs come from the kernel launched just before
    int mt, nt;
    tile_of(first_tile + tr, m_tiles, n_tiles, group_m, mt, nt);
    const int vec_per_row = bn / 4, i = blockIdx.y * 256 + threadIdx.x;
    const int rl = i / vec_per_row, cv = i % vec_per_row, row = mt * tile_rows + rl;
    if (ns == 0 || row >= m) return;
    const float *src = partial + static_cast<size_t>(rl) * bn + 4 * cv;
    const size_t tile_elems = static_cast<size_t>(tile_rows) * bn;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = 0; j0 < ns; j0 += 8) {
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j0 + j < ns) v[j] = *reinterpret_cast<const float4 *>(src + slabs[j0 + j] * tile_elems);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j0 + j < ns) add4(acc, v[j]);
    }
    const int col = nt * bn + 4 * cv;
    *reinterpret_cast<uint2 *>(C + static_cast<size_t>(row) * n + col) = finish4(acc, S, col, per_column);
}

// ---- host -----------------------------------------------------------------------------------

struct PrefillConfig {
    int bn, splits, mt, stream_k;
};

// Cost model of one launch for everything that runs on CTA pairs or single CTAs above 128 rows, least-squares fitted (mean error 5 %)
// to 2700 timed launches (CUDA graph over rotating weights; 12 shapes K = 512..9216 x N = 512..18432, M = 137..8192, every tiling
// considered; on them the model's choice takes 0.9 % more time than the best one, geometric mean).  Microseconds:
//   launch + waves * (K-steps per unit * step + tile) + work * (K-steps of all tiles per worker)
//   + [K split: fixed + per MB of fp32 slab traffic]  or  [stream-K: 2 * tile + per MB of remainder tiles + per slab piece]
// `work` is what a step costs beyond its time in a wave that leaves part of the chip idle: the power cap lowers the clock.
struct TileCost {
    double step, tile, work;
};
TileCost tile_cost(int bn, int mt) {
    if (mt == 2) return bn == 256 ? TileCost{0.276, 1.11, 0.074} : TileCost{0.186, 0.38, 0.069};
    return TileCost{0.224, 0.61, 0.071};  // (bn = 128; 256-column tiles of one M-tile were never the fastest)
}
constexpr double kCostLaunch = 4.17, kCostSplitFixed = 1.14, kCostSplitPerMB = 0.212, kCostSkPerMB = 0.75, kCostSkPerPiece = 0.044;
// Stream-K keeps every SM busy to the end, which the power cap takes back under a sustained load: it has to win by this factor.
constexpr double kSkMargin = 1.04;

// The model for single CTAs alone (the no-allocation entry, the fused all-gather), and for the K splits that size the workspace
// up to 128 rows: launch + waves * (K-steps per unit * step + tile) [+ split-K: fixed + per MB of slab traffic].
struct SingleCost {
    double step, tile;
};
SingleCost single_cost(int bn, int mt) {
    if (mt == 2) return bn == 256 ? SingleCost{0.584, 11.26} : SingleCost{0.463, 3.83};
    return bn == 256 ? SingleCost{0.489, 4.85} : SingleCost{0.301, 2.10};
}
constexpr double kSingleLaunch = 7.02, kSingleSplitFixed = 4.21, kSingleSplitPerMB = 0.332;

// Stream-K split of `tiles` tiles over `grid` CTAs: the tiles of the whole waves are dealt round-robin, the K-steps of
// the rest go in equal shares to `ctas` CTAs.  A share is at least 8 K-steps and at least 1/36 of a tile, so that no tile
// is spread over more slabs than the fix-up kernel sums (40).
struct StreamKPlan {
    int first_tile, ctas;
};
StreamKPlan streamk_plan(int tiles, int k_iters, int grid) {
    StreamKPlan pl;
    pl.first_tile = tiles / grid * grid;
    const long long total = static_cast<long long>(tiles - pl.first_tile) * k_iters;
    const int min_share = k_iters / 36 + 1 > 8 ? k_iters / 36 + 1 : 8;
    long long c = total / min_share;
    pl.ctas = static_cast<int>(c > grid ? grid : (c < 1 ? 1 : c));
    return pl;
}

// Rows of tiles in a band (tile_of): about 2048 rows of the problem, in bands of equal height.
int band_rows(int m_tiles, int mt) {
    const int most = 2048 / (BM * mt), bands = (m_tiles + most - 1) / most;
    return (m_tiles + bands - 1) / bands;
}

PrefillConfig g_prefill_override{0, 0, 0, 0};
unsigned long long g_wait_limit_ns = kWaitLimitNs;
int g_test_drop_a_load = -1;
int g_smallm_enabled = 1;

// K splits of the small-batch kernel.  Its time in microseconds, fitted to 570 timed launches (CUDA graph over rotating weights;
// K = 1024..9216 x N = 512..18432 x 9..128 rows x every split; the splits it picked were within 2% of the best.  Dequantisation and
// exchange have become cheaper since, which it does not know).  While its clusters
// take at most half the GPU, consecutive launches run side by side and only the chain from the grid-dependency wait to the exit
// counts; above that a launch starts on the SMs the one before leaves.  A further wave of CTAs repeats that start; how many clusters
// fit decides when there is one (4096 x 6144 has 48 tiles, and 3 splits need 48 clusters of 3 where 45 fit: 12.2 us, 2 splits 7.9).
// The exchange is bound by what a CTA sends to the others.
double smallm_cost(int m, int n, int k, int splits) {
    const int tiles = n / 128, clusters = smallm_clusters(splits), waves = (tiles + clusters - 1) / clusters;
    const double stages = (k / 128 + splits - 1) / splits, rows = (m + 15) / 16 * 16;
    const double over = ((tiles < clusters ? tiles : clusters) / static_cast<double>(clusters) - 0.5) * device_sm_count();
    double start = 1.86, step = 0.221 + 0.00092 * rows + (m > 64 ? 0.0091 : 0.0), exchange = 0.0;
    if (over > 0) {
        start = 2.55 + 0.0228 * over;
        step += 0.0433 + (m > 64 ? 0.00044 * over : 0.0);
    }
    if (splits > 1) exchange = 0.22 + 0.0174 * rows * (splits - 1) / splits + (m > 64 ? 0.65 : 0.0);
    return start + waves * step * stages + (waves - 1) * 2.73 + exchange;
}

// The models are asked several times per call with the same sizes and take 0.3 to 0.6 us each, as long as a quarter of a launch:
// a thread keeps what they said for the sizes it met last.  (They depend on sizes and device alone.)
template <class T>
struct PlanMemo {
    static constexpr int kEntries = 64;
    struct Entry {
        int dev = -1, m = 0, n = 0, k = 0;
        T plan{};
    } entry[kEntries];
    template <class F>
    T get(int m, int n, int k, F &&model) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return model();
        const unsigned hash = (static_cast<unsigned>(m) * 31u + static_cast<unsigned>(n >> 7)) * 31u + static_cast<unsigned>(k >> 7);
        Entry &e = entry[(hash * 2654435761u) >> 26];
        if (e.dev != dev || e.m != m || e.n != n || e.k != k) {
            e.plan = model();
            e.dev = dev;
            e.m = m;
            e.n = n;
            e.k = k;
        }
        return e.plan;
    }
};

int choose_smallm_splits(int m, int n, int k) {
    static thread_local PlanMemo<int> memo;
    return memo.get(m, n, k, [=] {
        int best = 1;
        double best_t = smallm_cost(m, n, k, 1);
        for (int s : {2, 3, 4, 6, 8}) {
            if (s > k / 128) break;
            const double t = smallm_cost(m, n, k, s);
            if (t < best_t) {
                best_t = t;
                best = s;
            }
        }
        return best;
    });
}

// Tilings of single CTAs.
PrefillConfig choose_single(int m, int n, int k, bool narrow, bool allow_pairs, bool allow_scratch, size_t max_split_bytes) {
    const int sms = device_sm_count(), k_iters = k / BK;
    PrefillConfig best{narrow ? 128 : 256, 1, 1, 0};
    double best_t = 1e30;
    for (int mt = 1; mt <= (allow_pairs && m > BM ? 2 : 1); ++mt)
        for (int bn = narrow ? 128 : 256; bn >= 128; bn /= 2)
            for (int s : {1, 2, 3, 4, 6, 8}) {
                if (k_iters / s < 8) continue;
                if (s > 1 && (!allow_scratch || static_cast<size_t>(s) * m * n * sizeof(float) > max_split_bytes)) continue;
                const long long units = static_cast<long long>((m + BM * mt - 1) / (BM * mt)) * (n / bn) * s;
                const double waves = static_cast<double>((units + sms - 1) / sms);
                const SingleCost tc = single_cost(bn, mt);
                double t = kSingleLaunch + waves * (static_cast<double>(k_iters) / s * tc.step + tc.tile);
                if (s > 1) t += kSingleSplitFixed + kSingleSplitPerMB * (static_cast<double>(s) + 0.5) * m * static_cast<double>(n) * 4.0 / 1.0e6;
                if (t < best_t) {
                    best_t = t;
                    best = PrefillConfig{bn, s, mt, 0};
                }
            }
    return best;
}

// Tilings of CTA pairs (two M-tiles of 128 rows) and of single CTAs of one M-tile and 128 columns.
PrefillConfig choose_any(int m, int n, int k, bool allow_scratch, bool pairs_only = false) {
    const int k_iters = k / BK;
    PrefillConfig best{128, 1, 1, 0};
    double best_t = 1e30;
    for (int mt = m > BM ? 2 : 1; mt >= (pairs_only ? 2 : 1); --mt)
        for (int bn = mt == 2 ? 256 : 128; bn >= 128; bn /= 2) {
            const TileCost tc = tile_cost(bn, mt);
            const int workers = device_sm_count() / mt;
            const long long tiles = static_cast<long long>((m + BM * mt - 1) / (BM * mt)) * (n / bn);
            const double base = kCostLaunch + tc.work * static_cast<double>(tiles) * k_iters / workers;
            for (int s : {1, 2, 3, 4, 6, 8}) {
                if (s > 1 && (!allow_scratch || k_iters / s < 4)) continue;
                const double waves = static_cast<double>((tiles * s + workers - 1) / workers);
                double t = base + waves * (((k_iters + s - 1) / s) * tc.step + tc.tile);
                if (s > 1) t += kCostSplitFixed + kCostSplitPerMB * (s + 0.5) * m * static_cast<double>(n) * 4.0 / 1.0e6;
                if (t < best_t) {
                    best_t = t;
                    best = PrefillConfig{bn, s, mt, 0};
                }
            }
            if (!allow_scratch || mt == 1) continue;
            const StreamKPlan pl = streamk_plan(static_cast<int>(tiles), k_iters, workers);
            const double rem = static_cast<double>(tiles - pl.first_tile);
            if (rem == 0) continue;
            const double share = rem * k_iters / pl.ctas;
            const double t = kSkMargin * (base + static_cast<double>(pl.first_tile / workers) * (k_iters * tc.step + tc.tile) + share * tc.step + 2.0 * tc.tile +
                                          kCostSkPerMB * rem * BM * mt * bn * 4.0 / 1.0e6 + kCostSkPerPiece * rem * k_iters / share);
            if (t < best_t) {
                best_t = t;
                best = PrefillConfig{bn, 1, mt, 1};
            }
        }
    return best;
}

// single: the launch has to run on single CTAs (fused all-gather).  !allow_pairs: one M-tile per CTA as well (the no-allocation entry,
// which has no fix-up pass either).
PrefillConfig choose_prefill(int m, int n, int k, bool allow_pairs = true, bool allow_scratch = true,
                             size_t max_split_bytes = ~static_cast<size_t>(0), bool single = false) {
    const int k_iters = k / BK;
    {  // tuning hook (kiln_w4a16_set_prefill_override): taken when it is legal for this problem, else the rule below
        const PrefillConfig &o = g_prefill_override;
        const bool legal = (o.bn == 128 || o.bn == 256) && n % o.bn == 0 && (o.mt == 1 || (o.mt == 2 && allow_pairs && m > BM)) &&
                           o.splits >= 1 && o.splits <= 8 && k_iters / o.splits >= 1 && (o.stream_k == 0 || o.stream_k == 1) &&
                           !(o.stream_k && o.splits != 1) && (allow_scratch || (o.splits == 1 && !o.stream_k));
        // (a forced split larger than max_split_bytes is returned as it is: the no-allocation entry then refuses the call)
        if (legal) return o;
    }
    if (!allow_pairs || single) return choose_single(m, n, k, false, allow_pairs, allow_scratch, max_split_bytes);
    if (!allow_scratch) return choose_any(m, n, k, false);
    static thread_local PlanMemo<PrefillConfig> memo;
    return memo.get(m, n, k, [=] {
        if (m > BM) return choose_any(m, n, k, true);
        // At most 128 rows: 128-column tiles, which the small-batch kernel shares; it may run fewer splits (exec_splits).
        PrefillConfig c = choose_single(m, n, k, true, true, true, ~static_cast<size_t>(0));
        c.splits = std::max(c.splits, choose_smallm_splits(m, n, k));
        return c;
    });
}

// The K splits that a plain problem of at most 128 rows runs with, in the small-batch kernel and, when that is switched off, in the
// general one (so that both give the same bits); `c` is the planner's tiling, whose splits size the workspace and are no fewer.
int exec_splits(const PrefillConfig &c, int m, int n, int k) {
    const PrefillConfig &o = g_prefill_override;
    if (m > BM || (o.bn == c.bn && o.splits == c.splits && o.mt == c.mt && o.stream_k == c.stream_k)) return c.splits;
    return std::min(c.splits, choose_smallm_splits(m, n, k));
}

// Tensor map of the bf16 result [m, n] for the epilogue's TMA stores: boxes of 32 rows x 64 columns, 128-byte swizzle.
bool encode_c_map(EncodeTiledFn enc, CUtensorMap *map, void *c, int m, int n) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(n), static_cast<cuuint64_t>(m)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(n) * 2};
    const cuuint32_t box[2] = {64, 32};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map of the fp32 pieces of split tiles: [slabs][rows][cols], boxes of 32 x 32, 128-byte swizzle.
bool encode_partial_map(EncodeTiledFn enc, CUtensorMap *map, float *partial, int cols, int rows, int slabs) {
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(slabs)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols) * 4, static_cast<cuuint64_t>(cols) * rows * 4};
    const cuuint32_t box[3] = {32, 32, 1}, estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, partial, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int MT = 1, int DW = 8, int DG = 2, int KP = 1, int KS = 1, int AR = BM>
int launch_bn(const CUtensorMap &tmap, const CUtensorMap &tmap_c, const CUtensorMap &tmap_p, PrefillParams p, cudaStream_t stream,
              const CUtensorMap *tmap_t = nullptr, const CUtensorMap *tmap_lb = nullptr) {
    using C = Cfg<BN, MT, DW, DG, KP, KS, AR>;
    p.k_iters /= KS;  // the kernel counts pipeline stages of KS atoms (k is a multiple of 128)
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !attr_set[dev]) {
        if (int rc = record_cuda_error(cudaFuncSetAttribute(w4a16_prefill_kernel<BN, MT, DW, DG, KP, KS, AR>,
                                                            cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes)))
            return rc;
        attr_set[dev] = true;
    }
    const int units = p.m_tiles * p.n_tiles * p.splits;
    const int grid = p.stream_k ? device_sm_count() : (units < device_sm_count() ? units : device_sm_count());
    note_launch();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(C::kThreads);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr = pdl_attribute();
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    static const CUtensorMap kNoMap = {};  // (never dereferenced when p.lora_steps == 0)
    if (!tmap_t || !tmap_lb || KS != 1) p.lora_steps = 0;
    return record_cuda_error(cudaLaunchKernelEx(&cfg, w4a16_prefill_kernel<BN, MT, DW, DG, KP, KS, AR>, tmap, tmap_c, tmap_p,
                                                tmap_t ? *tmap_t : kNoMap, tmap_lb ? *tmap_lb : kNoMap, p));
}

}  // namespace

// whether the small-batch kernel runs a plain problem that the planner tiled as `c`
static bool smallm_takes(const PrefillConfig &c, int m, int n, int k, int groupsize) {
    return g_smallm_enabled && c.bn == 128 && c.mt == 1 && !c.stream_k &&
           smallm_supported(m, n, k, groupsize, exec_splits(c, m, n, k));
}

// The small-batch kernel by itself, for a plain problem: no workspace.
bool smallm_takes(int m, int n, int k, int groupsize) { return m <= BM && smallm_takes(choose_prefill(m, n, k), m, n, k, groupsize); }

// The small-batch kernel's variant that applies the group scales in fp32 (the decode kernel's arithmetic): 16 rows a CTA.
static int exact_splits(int m, int n, int k, bool swiglu) { return swiglu ? 1 : choose_smallm_splits(16, n * ((m + 15) / 16), k); }
bool exact_supported(int m, int n, int k, int groupsize, bool swiglu, int lora_r) {
    return g_smallm_enabled && m <= 256 && (lora_r == 0 || (groupsize != -1 && lora_r <= 128)) &&
           smallm_supported(std::min(m, 16), n, k, groupsize, exact_splits(m, n, k, swiglu));
}
int launch_exact(const GemmArgs &a) { return launch_smallm(a, exact_splits(a.m, a.n, a.k, a.swiglu), true); }
// GEMMs of the same rows, K and group size, in launches of as many as one takes.  The K splits are those of one GEMM with all columns, but
// no fewer than a CTA's most stages ask for: more columns want fewer splits, and each member by itself may need the splits that it has.
struct GroupLaunch {
    int end, n, splits;  // the members before `end`, their columns
};
static GroupLaunch group_launch(const GemmArgs *items, int i, int count, bool exact) {
    const GemmArgs &a = items[i];
    GroupLaunch g{i + 1, a.n, 1};
    for (; g.end < count && g.end < i + smallm_most_grouped() && static_cast<long long>(g.n) + items[g.end].n <= 65535LL * 128; ++g.end) g.n += items[g.end].n;
    g.splits = exact ? exact_splits(a.m, g.n, a.k, false) : choose_smallm_splits(a.m, g.n, a.k);
    for (int s : {2, 3, 4, 6, 8})
        if (s > g.splits && !smallm_supported(exact ? std::min(a.m, 16) : a.m, a.n, a.k, a.groupsize, g.splits)) g.splits = s;
    return g;
}
static int launch_groups(const GemmArgs *items, int count, bool exact) {
    for (int i = 0; i < count;) {
        const GroupLaunch g = group_launch(items, i, count, exact);
        if (int rc = launch_smallm_group(items + i, g.end - i, g.splits, exact)) return rc;
        i = g.end;
    }
    return 0;
}
// Whether a group of decode-sized GEMMs that the fp32-scale variant could run is faster there than in one launch of the decode kernel.  Measured
// from 4 to 32 rows for K = 128 .. 12288 and 512 .. 25600 columns in all (weights cold in HBM); us, decode kernel / this one:
//  * up to 8 rows, one block of the decode kernel: while the tiles take half the GPU (8 x 512 x 8192 4.7 / 2.7, 5 x 512 x 12288 3.6 / 3.8), four rows
//    only between the shortest K and eight groups (4 x 512 x 8192 3.6 / 2.6, 4 x 128 x 1024 2.2 / 2.3, 4 x 1024 x 6144 3.1 / 3.5);
//  * in one wave of CTAs always (16 x 2560 x 5120 6.4 / 5.7, 32 x 4096 x 4864 12.3 / 7.0), but for the widest of a short K (9 x 256 x 18944 3.5 / 4.2);
//  * a further wave repeats a CTA's start, which only a long K makes up for, where the decode kernel dequantises twice (from 17 rows; from 13 above
//    5120): whole tiles or many from 2560 (17 x 2560 x 10240 16.9 / 15.1, 17 x 4864 x 13824 41 / 28; 17 x 4608 x 10240, split, 20.6 / 24.9, 17 x 2304 x 10240
//    12.4 / 14.1, 17 x 256 x 24576 5.4 / 10.8), around 12288 columns from 1408 (17 x 1792 x 13568 14.5 / 12.4, x 18432 14.2 / 14.7), all above 5120
//    (17 x 6144 x 10240 37.6 / 29.2, 16 x 8192 x 9728 22.6 / 19.7; 9 x 12288 x 11008 24.4 / 25.8);
//  * a second launch, for more than four members, under the same condition (five of 3840 columns, 17 rows: K = 1408 6.0 / 7.5, 6144 22.1 / 13.1).
bool exact_group_pays(const GemmArgs *items, int count) {
    const int m = items[0].m, k = items[0].k;
    if (count > smallm_most_grouped() && (m < 17 || k <= 5120)) return false;
    for (int i = 0; i < count;) {
        const GroupLaunch g = group_launch(items, i, count, true);
        const int tiles = g.n / 128, units = tiles * ((m + 15) / 16);
        bool pays;
        if (m <= 8)
            pays = 2 * tiles <= device_sm_count() && (m > 4 || (k > 128 && (k < 1024 || g.n <= 4096)));
        else if (units <= smallm_clusters(g.splits))
            pays = k > 512 || g.n <= 16384;
        else if (k > 5120)
            pays = m >= 13;
        else
            pays = m >= 17 && (k >= 2560 ? g.splits == 1 || g.n > 12288 : k >= 1408 && g.n >= 12288 && g.n <= 16384);
        if (!pays) return false;
        i = g.end;
    }
    return true;
}
int launch_exact_group(const GemmArgs *items, int count) { return launch_groups(items, count, true); }
int launch_plain_group(const GemmArgs *items, int count) { return launch_groups(items, count, false); }

// SwiGLU is fused into an epilogue that sees whole tiles: the small-batch kernel's without a K split, or the pair kernel's.  A second
// pass over the bf16 result takes about 4 us, more than a K split saves a SwiGLU-sized projection, except for a long K and few columns.
constexpr double kCostSwigluPass = 4.0;
PrefillConfig swiglu_config(int m, int n, int k) {
    const PrefillConfig c = choose_prefill(m, n, k);
    return m <= BM || (c.splits == 1 && !c.stream_k && c.mt == 2) ? c : choose_any(m, n, k, false, true);
}
bool prefill_fuses_swiglu(int m, int n, int k) {
    if (m > BM) return true;
    const PrefillConfig c = choose_prefill(m, n, k);
    const int splits = exec_splits(c, m, n, k);
    if (!smallm_takes(c, m, n, k, 128)) return false;
    return splits == 1 || (smallm_supported(m, n, k, 128, 1) && smallm_cost(m, n, k, 1) < smallm_cost(m, n, k, splits) + kCostSwigluPass);
}
// Whether a SwiGLU call reserves room for the bf16 result that a second pass would read: unless the planned tiling writes whole tiles.
bool prefill_swiglu_room(int m, int n, int k) {
    const PrefillConfig c = choose_prefill(m, n, k);
    return m <= BM ? !(c.splits == 1 && smallm_takes(c, m, n, k, 128)) : !(c.splits == 1 && !c.stream_k && c.mt == 2 && c.bn == 256);
}

// The LoRA delta can ride in the tcgen05 kernel as extra K-steps unless the scales are per column (those are applied to
// the whole accumulator in the epilogue and would scale the delta too).
bool prefill_fuses_lora(int groupsize, int lora_r) { return groupsize == 128 && lora_r > 0 && lora_r <= 128 && lora_r % 8 == 0; }

void set_wait_limit_ns(unsigned long long ns) { g_wait_limit_ns = ns ? ns : kWaitLimitNs; }
unsigned long long current_wait_limit_ns() { return g_wait_limit_ns; }
void set_smallm_enabled(int on) { g_smallm_enabled = on; }
void set_test_drop_a_load(int k_step) { g_test_drop_a_load = k_step; }
int test_drop_a_load() { return g_test_drop_a_load; }

void set_prefill_override(int bn, int splits, int mt, int stream_k) {
    g_prefill_override = PrefillConfig{bn, splits, mt, stream_k};
}

void prefill_plan(int m, int n, int k, int out[4]) {
    const PrefillConfig c = choose_prefill(m, n, k);
    out[0] = c.bn;
    out[1] = c.splits;
    out[2] = c.mt;
    out[3] = c.stream_k;
}

bool prefill_supported(int m, int n, int k, int groupsize) {
    (void)groupsize;
    return m >= 1 && n % 256 == 0 && k % 128 == 0 && k / BK >= 2;
}

size_t workspace_for(const PrefillConfig &c, int m, int n) {
    if (c.stream_k) return static_cast<size_t>(2) * device_sm_count() * (BM * c.mt) * c.bn * sizeof(float);
    return c.splits > 1 ? static_cast<size_t>(c.splits) * m * n * sizeof(float) : 0;
}

size_t prefill_workspace_bytes(int m, int n, int k) { return workspace_for(choose_prefill(m, n, k), m, n); }

int launch_prefill(const GemmArgs &a) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return KILN_W4A16_ERR_CUDA;
    uint32_t *status = device_status_word();
    if (!status) return KILN_W4A16_ERR_CUDA;
    const bool fused = a.n_peers > 0 || a.mc_c;  // the peer-store epilogue needs whole tiles: no split-K, no stream-K
    // At most 128 rows: the kernel that keeps the dequantised weights in tensor memory; its K splits need no workspace
    if (!fused && a.m <= BM && (a.lora_r == 0 || (a.lora_t && a.lora_b && prefill_fuses_lora(a.groupsize, a.lora_r)))) {
        const PrefillConfig sc = choose_prefill(a.m, a.n, a.k);
        const int splits = exec_splits(sc, a.m, a.n, a.k);
        if (smallm_takes(sc, a.m, a.n, a.k, a.groupsize)) return launch_smallm(a, a.swiglu ? 1 : splits);
    }
    PrefillConfig c = a.swiglu ? swiglu_config(a.m, a.n, a.k) : choose_prefill(a.m, a.n, a.k, true, !fused && !a.no_scratch, ~static_cast<size_t>(0), fused);
    c.splits = exec_splits(c, a.m, a.n, a.k);
    if (a.swiglu && (fused || c.splits != 1 || c.stream_k || c.mt == 1)) return KILN_W4A16_ERR_KERN_SHAPE;  // (callers ask prefill_fuses_swiglu first)
    CUtensorMap tmap;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(a.k), static_cast<cuuint64_t>(a.m)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(a.k) * 2};
    // at most 64 rows in 128-column tiles of one M-tile: half-height activation atoms (AR = 64)
    const bool half_a = a.m <= 64 && c.mt == 1 && c.bn == 128;
    const cuuint32_t box[2] = {BK, static_cast<cuuint32_t>(half_a ? 64 : BM * c.mt)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(&tmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(a.A), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return KILN_W4A16_ERR_CUDA;
    // Which of the fused all-gather's buffers lives on this GPU: that copy leaves through the TMA-store path.
    int self_peer = -1;
    if (a.n_peers > 0) {
        int dev = -1, found = 0;
        cudaGetDevice(&dev);
        for (int i = 0; i < a.n_peers && i < 8; ++i) {
            cudaPointerAttributes at;
            if (cudaPointerGetAttributes(&at, a.peer_c[i]) == cudaSuccess && at.type == cudaMemoryTypeDevice && at.device == dev) {
                self_peer = i;
                ++found;
            }
        }
        cudaGetLastError();  // (an unregistered pointer only means "not ours")
        if (found != 1) self_peer = -1;  // ambiguous: every copy goes through the store path of the remote copies
    }
    CUtensorMap tmap_c;  // this GPU's own C: [m, n], or its [m, ldc] buffer of the fused all-gather
    if (self_peer >= 0) {
        if (!encode_c_map(enc, &tmap_c, a.peer_c[self_peer], a.m, a.ldc)) return KILN_W4A16_ERR_CUDA;
    } else if (!encode_c_map(enc, &tmap_c, a.C, a.m, a.swiglu ? a.n / 2 : a.n)) {
        return KILN_W4A16_ERR_CUDA;
    }

    PrefillParams p{};
    p.B = static_cast<const uint4 *>(a.B);
    p.S = static_cast<const __half *>(a.S);
    p.C = static_cast<__nv_bfloat16 *>(a.C);
    p.partial = static_cast<float *>(a.workspace);
    p.status = status;
    p.m = a.m;
    p.n = a.n;
    p.k = a.k;
    p.m_tiles = (a.m + BM * c.mt - 1) / (BM * c.mt);
    p.n_tiles = a.n / c.bn;
    p.splits = c.splits;
    p.group_m = band_rows(p.m_tiles, c.mt);
    p.k_iters = a.k / BK;
    p.per_column = a.groupsize == -1;
    p.n_peers = a.n_peers;
    p.ldc = a.ldc;
    p.col0 = a.col0;
    p.self_peer = self_peer;
    p.swiglu = a.swiglu;
    // LoRA delta fused as extra K-steps: t = scale * x * A^T (bf16 [m, r], written by the kernel launched just before) and
    // lora_b (bf16 [n, r]) are operand tiles like any other; columns past r read zero
    CUtensorMap tmap_t, tmap_lb;
    const bool lora = a.lora_r > 0 && a.lora_t && a.lora_b;
    if (lora) {
        if (a.groupsize == -1 || a.lora_r % 8 != 0 || a.lora_r > 128) return KILN_W4A16_ERR_KERN_SHAPE;  // (callers ask prefill_fuses_lora first)
        const cuuint64_t td[2] = {static_cast<cuuint64_t>(a.lora_r), static_cast<cuuint64_t>(a.m)};
        const cuuint64_t ld[2] = {static_cast<cuuint64_t>(a.lora_r), static_cast<cuuint64_t>(a.n)};
        const cuuint64_t st[1] = {static_cast<cuuint64_t>(a.lora_r) * 2};
        const cuuint32_t tb[2] = {BK, static_cast<cuuint32_t>(half_a ? 64 : BM * c.mt)}, lb[2] = {BK, static_cast<cuuint32_t>(c.bn)};
        if (enc(&tmap_t, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(a.lora_t), td, st, tb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
            enc(&tmap_lb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(a.lora_b), ld, st, lb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return KILN_W4A16_ERR_CUDA;
        p.lora_steps = (a.lora_r + BK - 1) / BK;
    }
    const CUtensorMap *pt = lora ? &tmap_t : nullptr, *plb = lora ? &tmap_lb : nullptr;
    p.mc_c = static_cast<__nv_bfloat16 *>(a.mc_c);
    for (int i = 0; i < a.n_peers && i < 8; ++i) p.peer_c[i] = static_cast<__nv_bfloat16 *>(a.peer_c[i]);
    p.stream_k = c.stream_k;
    p.wait_limit_ns = g_wait_limit_ns;
    p.test_drop_a_load = g_test_drop_a_load;
    // tiles of 256 rows run on CTA pairs (the fused all-gather stays on single CTAs)
    const bool pair = c.mt == 2 && !fused;
    const StreamKPlan plan = streamk_plan(p.m_tiles * p.n_tiles, p.k_iters, pair ? device_sm_count() / 2 : device_sm_count());
    p.sk_first_tile = plan.first_tile;
    p.sk_ctas = plan.ctas;
    const size_t need = workspace_for(c, a.m, a.n);
    if (need > 0 && (!a.workspace || a.workspace_bytes < need)) return KILN_W4A16_ERR_WORKSPACE;

    CUtensorMap tmap_p = tmap_c;  // (unused when no tile is split)
    if (c.stream_k ? !encode_partial_map(enc, &tmap_p, p.partial, c.bn, BM * c.mt, 2 * plan.ctas)
                   : c.splits > 1 && !encode_partial_map(enc, &tmap_p, p.partial, a.n, a.m, c.splits))
        return KILN_W4A16_ERR_CUDA;

    int rc;
    if (pair)
        rc = launch_pair(a, p, c.bn, tmap_c, tmap_p);
    else if (c.mt == 2)
        rc = c.bn == 256 ? launch_bn<256, 2>(tmap, tmap_c, tmap_p, p, a.stream, pt, plb) : launch_bn<128, 2>(tmap, tmap_c, tmap_p, p, a.stream, pt, plb);
    else
        // (128-column tiles of one M-tile are bound by the MMA issue rate: two issuers, each with an accumulator of its own)
        // ... and 128-deep pipeline stages, which halve their barrier round trips per K (not with stream-K, whose fix-up pass
        // counts 64-deep steps, nor when a split would be left without a whole stage)
        if (c.bn == 256)
            rc = launch_bn<256, 1>(tmap, tmap_c, tmap_p, p, a.stream, pt, plb);
        else if (c.stream_k || a.k / 128 < c.splits || lora)  // (the LoRA steps are 64 deep)
            rc = half_a ? launch_bn<128, 1, 8, 2, 2, 1, 64>(tmap, tmap_c, tmap_p, p, a.stream, pt, plb)
                        : launch_bn<128, 1, 8, 2, 2, 1>(tmap, tmap_c, tmap_p, p, a.stream, pt, plb);
        else
            rc = half_a ? launch_bn<128, 1, 8, 2, 2, 2, 64>(tmap, tmap_c, tmap_p, p, a.stream)
                        : launch_bn<128, 1, 8, 2, 2, 2>(tmap, tmap_c, tmap_p, p, a.stream);
    if (rc) return rc;
    if (c.splits > 1) {
        const unsigned blocks = static_cast<unsigned>((static_cast<size_t>(a.m) * a.n / 4 + 255) / 256);
        note_launch();
        rc = record_cuda_error(launch_pdl(splitk_reduce_kernel, dim3(blocks), dim3(256), a.stream, p.partial, p.C, p.S, a.m, a.n,
                                          c.splits, static_cast<int>(p.per_column)));
    }
    if (c.stream_k && p.m_tiles * p.n_tiles > plan.first_tile) {
        const int rem = p.m_tiles * p.n_tiles - plan.first_tile;
        const long long total = static_cast<long long>(rem) * p.k_iters;
        note_launch();
        rc = record_cuda_error(launch_pdl(streamk_fixup_kernel, dim3(rem, BM * c.mt * c.bn / 1024), dim3(256), a.stream, p.partial, p.C, p.S, a.m, a.n,
                                          p.m_tiles, p.n_tiles, p.group_m, p.k_iters, BM * c.mt, c.bn, plan.ctas, total, plan.first_tile,
                                          static_cast<int>(p.per_column)));
    }
    return rc;
}

}  // namespace kiln

// ---- the entry point that allocates nothing ---------------------------------------------------
//
// Some callers of this library cannot allocate device memory at call time and have no buffer to
// lend either: an inference server that hands every remaining byte of HBM to its KV-cache pool at
// start-up, or a serving loop that cannot afford the device-wide synchronisation a cudaMalloc or
// cudaFree implies.  For them the split-K scratch of the prefill kernel lives in a fixed array in
// the library's own device image.  Every GPU that loads the library holds these 16 MiB until the
// process exits.
namespace kiln {
namespace {

static __device__ __align__(256) float g_static_scratch[KILN_W4A16_NOALLOC_SCRATCH_BYTES / sizeof(float)];
static __device__ __align__(256) uint32_t g_static_status[64];

struct StaticDeviceState {
    float *scratch = nullptr;
    uint32_t *status = nullptr;
};

// In host code `g_static_scratch` is only a handle for the symbol, not a device address: the
// address has to be asked for, once per device, with that device current.
int static_state(StaticDeviceState **out) {
    static StaticDeviceState per_device[64];
    static std::mutex mu;
    int dev = 0;
    if (int rc = record_cuda_error(cudaGetDevice(&dev))) return rc;
    if (dev < 0 || dev >= 64) return KILN_W4A16_ERR_ARG;
    std::lock_guard<std::mutex> lock(mu);
    StaticDeviceState &st = per_device[dev];
    if (!st.scratch) {
        void *p_scratch = nullptr, *p_status = nullptr;
        if (int rc = record_cuda_error(cudaGetSymbolAddress(&p_scratch, g_static_scratch))) return rc;
        if (int rc = record_cuda_error(cudaGetSymbolAddress(&p_status, g_static_status))) return rc;
        st.status = static_cast<uint32_t *>(p_status);
        st.scratch = static_cast<float *>(p_scratch);
    }
    *out = &st;
    return 0;
}

PrefillConfig noalloc_config(int m, int n, int k) {
    return choose_prefill(m, n, k, /*allow_pairs=*/false, /*allow_scratch=*/true, KILN_W4A16_NOALLOC_SCRATCH_BYTES);
}

}  // namespace

// Reads and clears the status word of the no-allocation entry's launches on the current device (0 if that entry has
// never run there).  No allocation: the word lives in the library image.
int static_status_read_clear(cudaStream_t st, uint32_t *out) {
    *out = 0;
    int dev = 0;
    if (int rc = record_cuda_error(cudaGetDevice(&dev))) return rc;
    if (dev < 0 || dev >= 64) return 0;
    StaticDeviceState *state = nullptr;
    if (int rc = static_state(&state)) return rc;
    if (int rc = record_cuda_error(cudaMemcpyAsync(out, state->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, st))) return rc;
    if (int rc = record_cuda_error(cudaStreamSynchronize(st))) return rc;
    if (*out != 0) {
        if (int rc = record_cuda_error(cudaMemsetAsync(state->status, 0, sizeof(uint32_t), st))) return rc;
        if (int rc = record_cuda_error(cudaStreamSynchronize(st))) return rc;
    }
    return 0;
}
}  // namespace kiln

extern "C" void kiln_w4a16_noalloc_plan(int m, int n, int k, int out[4]) {
    if (!out || m <= 0 || n <= 0 || k <= 0) return;
    const kiln::PrefillConfig c = kiln::noalloc_config(m, n, k);
    out[0] = c.bn;
    out[1] = c.splits;
    out[2] = c.mt;
    out[3] = c.stream_k;
}

extern "C" kiln_w4a16_status_t kiln_w4a16_gemm_bf16_noalloc(const void *A, const void *B, void *C, const void *s,
                                                            int m, int n, int k, int groupsize, void *stream) {
    using namespace kiln;
    if (m < 0 || n < 0 || k < 0) return KILN_W4A16_ERR_ARG;
    if (k % 128 != 0 || n % 256 != 0 || !(groupsize == -1 || groupsize == 128)) return KILN_W4A16_ERR_PROB_SHAPE;
    if (m == 0 || n == 0 || k == 0) return KILN_W4A16_OK;
    if (!A || !B || !C || !s) return KILN_W4A16_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
         reinterpret_cast<uintptr_t>(s)) & 15)
        return KILN_W4A16_ERR_ALIGNMENT;
    if (!prefill_supported(m, n, k, groupsize)) return KILN_W4A16_ERR_KERN_SHAPE;

    // the best tiling whose split-K slabs fit the array (a tiling without a split always does); only a tiling forced
    // through the tuning hook can still ask for more
    const PrefillConfig c = noalloc_config(m, n, k);
    const size_t need = c.splits > 1 ? static_cast<size_t>(c.splits) * m * n * sizeof(float) : 0;
    if (need > KILN_W4A16_NOALLOC_SCRATCH_BYTES) return KILN_W4A16_ERR_STATIC_SCRATCH;

    StaticDeviceState *st = nullptr;
    if (int rc = static_state(&st)) return rc;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return KILN_W4A16_ERR_CUDA;

    CUtensorMap tmap;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(m)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2};
    const cuuint32_t box[2] = {BK, BM};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&tmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(A), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return KILN_W4A16_ERR_CUDA;

    PrefillParams p{};
    p.B = static_cast<const uint4 *>(B);
    p.S = static_cast<const __half *>(s);
    p.C = static_cast<__nv_bfloat16 *>(C);
    // Nothing in the scratch has to start at zero: every split writes its whole [m, n] slab before the
    // reduction reads it, so what the previous call left behind is simply overwritten.
    p.partial = st->scratch;
    p.status = st->status;
    p.m = m;
    p.n = n;
    p.k = k;
    p.m_tiles = (m + BM - 1) / BM;
    p.n_tiles = n / c.bn;
    p.splits = c.splits;
    p.group_m = band_rows(p.m_tiles, 1);
    p.k_iters = k / BK;
    p.per_column = groupsize == -1;
    p.wait_limit_ns = g_wait_limit_ns;
    p.test_drop_a_load = -1;
    p.self_peer = -1;
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    CUtensorMap tmap_c;
    if (!encode_c_map(enc, &tmap_c, C, m, n)) return KILN_W4A16_ERR_CUDA;
    CUtensorMap tmap_p = tmap_c;  // (unused when no tile is split)
    if (c.splits > 1 && !encode_partial_map(enc, &tmap_p, p.partial, n, m, c.splits)) return KILN_W4A16_ERR_CUDA;
    int rc = c.bn == 256 ? launch_bn<256>(tmap, tmap_c, tmap_p, p, cs) : launch_bn<128>(tmap, tmap_c, tmap_p, p, cs);
    if (rc) return rc;
    if (c.splits > 1) {
        const unsigned blocks = static_cast<unsigned>((static_cast<size_t>(m) * n / 4 + 255) / 256);
        note_launch();
        rc = record_cuda_error(launch_pdl(splitk_reduce_kernel, dim3(blocks), dim3(256), cs, p.partial, p.C, p.S, m, n, c.splits,
                                          static_cast<int>(p.per_column)));
    }
    return rc;
}
