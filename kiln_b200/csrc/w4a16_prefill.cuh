// Work description and distribution shared by the two prefill kernels (prefill_w4a16_umma.cu, pair_w4a16_umma.cu).
#pragma once

#include "w4a16_umma.cuh"

namespace kiln {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr uint32_t kEpiWarpBytes = 4096;  // per epilogue warp: 32 rows x 64 columns of bf16, 128B-swizzled (four 1024-byte atoms)

struct PrefillParams {
    const uint4 *B;
    const __half *S;
    __nv_bfloat16 *C;
    float *partial;  // fp32 [splits][m][n] when splits > 1
    uint32_t *status;
    int m, n, k;
    int m_tiles, n_tiles, splits, k_iters;  // k_iters = k / 64
    int per_column;
    // fused all-gather epilogue: n_peers > 0 -> every finished tile row segment is stored to the row-major
    // [m, ldc] buffer of each peer GPU (peer_c[i], plain peer-mapped pointers) at column offset col0
    __nv_bfloat16 *peer_c[8];
    int n_peers, ldc, col0;
    int self_peer;  // index in peer_c of the buffer that lives on this GPU (written through the TMA store), or -1
    int swiglu;     // columns hold gate and up interleaved in runs of 32; C is [m, n/2] = silu(gate) * up (pair kernel, whole tiles)
    // LoRA delta as extra K-steps: the piece of work that starts a tile's K range appends lora_steps (1 or 2) 64-deep steps
    // whose operands are bf16 tiles of t = scale * x * A^T [m, r] and of lora_b [n, r], both fetched by TMA (KS == 1 only)
    int lora_steps;
    // mc_c != nullptr: one multimem.st per piece to the group's multicast address instead (the switch replicates
    // the store into every GPU's buffer, this GPU's included, so each tile leaves this GPU once)
    __nv_bfloat16 *mc_c;
    int stream_k;     // 1: whole waves of tiles round-robin, then the remaining tiles' (tile, K-step) space in equal shares
    int sk_first_tile;  // stream-K: tiles below this index are dealt whole (a multiple of the grid size)
    int sk_ctas;        // stream-K: CTAs that share the remaining tiles (<= grid size)
    int group_m;        // tiles are dealt in bands of this many rows of tiles (tile_of)
    unsigned long long wait_limit_ns;  // every bounded wait of the launch gives up after this long
    int test_drop_a_load;  // test hook: the activation tile of this K-step (counted per CTA) is announced but never copied; -1 = off
};

// Tile t of the launch: bands of group_m rows of tiles, column by column inside a band.  The CTAs of a wave then work on a few rows
// and a few columns of tiles at once, whose operands stay in L2, also where the activations as a whole do not fit (16384 x 9216:
// 302 MB, read once per column of tiles when the tiles were dealt row by row).
__host__ __device__ __forceinline__ void tile_of(int t, int m_tiles, int n_tiles, int group_m, int &mt, int &nt) {
    const int band = t / (group_m * n_tiles), r = t - band * group_m * n_tiles;
    const int rows = m_tiles - band * group_m < group_m ? m_tiles - band * group_m : group_m;
    nt = r / rows;
    mt = band * group_m + (r - nt * rows);
}

// Hands a CTA (or a CTA pair) its work.  Default: units (tile, K-split) dealt round-robin.  Stream-K (hybrid): the flattened (tile,
// K-step) space of the tiles that do not fill a whole wave of the grid is cut into sk_ctas equal contiguous ranges, so no SM idles in
// a last partial wave; a range covers the tail of one tile, whole tiles, and the head of another.  They come first, so that the
// fp32 pieces drain under the main loops of the other tiles, which are dealt round-robin.  Whole tiles are written straight to C; the at most
// two partial pieces of a CTA go to fp32 slabs 2*cta and 2*cta+1 of the workspace and are summed per tile, in
// CTA order, by `streamk_fixup_kernel`.  No CTA waits for another.
struct WorkIter {
    int me, mode, u, units, stride, splits, m_tiles, n_tiles, group_m, k_iters, first_tile;
    long long cur, begin, end;
    // worker `index` of `workers` (a CTA of the grid, or a pair of CTAs)
    __device__ WorkIter(const PrefillParams &p, int index, int workers)
        : me(index), mode(p.stream_k), u(index), units(p.m_tiles * p.n_tiles * p.splits), stride(workers), splits(p.splits),
          m_tiles(p.m_tiles), n_tiles(p.n_tiles), group_m(p.group_m), k_iters(p.k_iters), first_tile(p.sk_first_tile) {
        if (mode) {
            units = first_tile;  // whole tiles of the full waves (splits == 1 in this mode)
            const long long total = static_cast<long long>(p.m_tiles * p.n_tiles - first_tile) * p.k_iters;
            const long long c = index, n = p.sk_ctas;
            begin = cur = c < n ? total * c / n : 0;
            end = c < n ? total * (c + 1) / n : 0;
        } else {
            begin = cur = end = 0;
        }
    }
    // slab: -1 = the piece is a whole tile (or an ordinary split) and goes where `sp` says; >= 0 = stream-K slab index
    __device__ bool next(int &mt, int &nt, int &sp, int &ki0, int &ki1, int &slab) {
        if (cur < end) {
            const int tr = static_cast<int>(cur / k_iters);  // tile within the remainder
            ki0 = static_cast<int>(cur - static_cast<long long>(tr) * k_iters);
            const long long left = end - cur;
            ki1 = left < k_iters - ki0 ? ki0 + static_cast<int>(left) : k_iters;
            const int t = first_tile + tr;
            tile_of(t, m_tiles, n_tiles, group_m, mt, nt);
            sp = 0;
            slab = (ki0 == 0 && ki1 == k_iters) ? -1 : 2 * me + (cur == begin ? 0 : 1);
            cur += ki1 - ki0;
            return true;
        }
        if (u >= units) return false;
        sp = u % splits;
        const int t = u / splits;
        tile_of(t, m_tiles, n_tiles, group_m, mt, nt);
        ki0 = static_cast<int>(static_cast<long long>(k_iters) * sp / splits);
        ki1 = static_cast<int>(static_cast<long long>(k_iters) * (sp + 1) / splits);
        slab = -1;
        u += stride;
        return true;
    }
};

// The kernel of CTA pairs: tiles of 256 x tile_n (128 or 256; m_tiles, n_tiles count those), no fused all-gather.  tmap_p: the fp32
// pieces of split tiles (encode_partial_map).
int launch_pair(const GemmArgs &a, PrefillParams p, int tile_n, const CUtensorMap &tmap_c, const CUtensorMap &tmap_p);

}  // namespace kiln
