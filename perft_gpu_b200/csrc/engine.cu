// B200 perft engine: level-synchronous tree expansion with a fused,
// count-only last ply.
//
// What it replaces in the reference (ankan-ban/perft_gpu):
//   perft_bb_gpu_simple / _hash BFS drivers (perft_bb.h:1027-1138,
//   1242-1589), the per-level kernels makemove_and_count_moves_single_level
//   (perft_bb.h:601-625), generate_moves_single_level (perft_bb.h:983-996),
//   the leaf pass makeMove_and_perft_single_level_indices (perft_bb.h:412-446)
//   and moderngpu's ScanD + IntervalExpandDGenValues (perft_bb.h:1088-1124).
//
// Design (B200-first):
//   * Boards are side-relative (movegen.cuh), so no kernel branches on the
//     side to move.
//   * A level is a structure-of-arrays buffer in HBM: the boards as three
//     arrays of 16-byte plane pairs (128-bit loads and stores), plus the move
//     count and root id of each node.  Every node of a level has
//     the same remaining depth (roots are grouped by depth).
//   * One exclusive scan of the move counts turns a level into a flat list
//     of (parent, move) items.  Items are cut into fixed tiles of TILE_CAP;
//     the scan also records the first parent of every tile, so the tile
//     kernel needs no search and no parent-index expansion buffer.
//   * The tile kernel is persistent (one wave of CTAs sized by occupancy)
//     and steals tiles from an atomic counter.  Per tile it stages the
//     parents in shared memory, generates their moves into a compact shared
//     item list (only the moves inside the tile window), then every thread
//     takes items: make the move, count the child's legal moves, write the
//     child (coalesced: item order is child order) and its count.
//   * The last ply writes nothing: its kernel sums the replies to quiet moves
//     from the parent alone, makes and counts only the other moves, and sums
//     per root in a shared-memory accumulator with one global atomic per run.
//   * Equal nodes of a level are merged before it is expanded.
//   * When a level does not fit the HBM arena, its item range is split at
//     tile boundaries and the chunks are expanded depth-first.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../../include/perft_b200.h"
#include "movegen.cuh"

namespace pg {
void build_tables();
}  // namespace pg

using namespace pg;

namespace {

// ------------------------------------------------------------- constants
#ifndef PG_TILE_CAP_LOG2
#define PG_TILE_CAP_LOG2 13
#endif
#ifndef PG_TILE_MINB
#define PG_TILE_MINB 3
#endif
#ifndef PG_ONE_RUN_VOTE
#define PG_ONE_RUN_VOTE 1  // one block vote for windows whose parents share one root
#endif
#ifndef PG_MIRRORED_STAGE
#define PG_MIRRORED_STAGE 1  // parents staged mirrored: children are made in their own frame
#endif
#ifndef PG_KNOWN_KINGS
#define PG_KNOWN_KINGS 1  // (with mirrored staging) the count gets both king squares from the parent
#endif
#ifndef PG_KNOWN_OCC
#define PG_KNOWN_OCC 1  // (with known kings) and the occupancy and opponent set from make-move
#endif
#ifndef PG_TILE_NT
#define PG_TILE_NT 256
#endif
constexpr int TILE_NT = PG_TILE_NT;  // threads per tile CTA
constexpr int TILE_CAP_LOG2 = PG_TILE_CAP_LOG2;  // largest tile: 2^TILE_CAP_LOG2 items
constexpr int TILE_CAP = 1 << TILE_CAP_LOG2;
constexpr int TILE_MIN_LOG2 = 10;  // small levels use tiles down to 1024 items to fill every SM
constexpr u64 MAX_TILES_PER_NODE_DIV = 1ull << TILE_MIN_LOG2;
constexpr int TILE_MAXP = TILE_NT;
// The count-only ply: CTA size and resident CTAs, and the item list, which
// holds the listed moves of LEAF_NT parents or all moves of LEAF_FEW.  Large
// CTAs in step fetch each instruction for more warps; the L1 that shared
// memory leaves holds the move tables.  With 24 items per parent the list
// overflowed where half the moves are listed (exposed kings) and the unit was
// generated again in parts: depth 6 of one such position 0.61 -> 0.57 ms, two
// table positions 220 -> 198 ms with 32; 40 takes 1% more (less L1).
#ifndef PG_LEAF_NT
#define PG_LEAF_NT 256
#endif
#ifndef PG_LEAF_MINB
#define PG_LEAF_MINB 3
#endif
constexpr int LEAF_NT = PG_LEAF_NT;
constexpr int LEAF_MINB = PG_LEAF_MINB;
constexpr u32 LEAF_ITEMS = 32 * LEAF_NT;
constexpr int LEAF_FEW = LEAF_NT / 64;
static_assert(LEAF_FEW * MAX_ANY_MOVES <= LEAF_ITEMS, "a few parents always fit, whatever their pieces");
// A CTA takes LEAF_NT parents at a time, or fewer (down to this) while some
// CTA would get none: 100 positions at depth 2 take 95 us with 16, 104 with
// 32, 110 with 4 or always LEAF_NT.
constexpr int LEAF_MIN_UNIT = 16;
constexpr int TILE_MINB = PG_TILE_MINB;          // resident CTAs per SM the register budget targets
constexpr int MAX_LEGAL_MOVES = 218;

constexpr int SCAN_NT = 512;
// (16 nodes per thread: the same on large levels, but one position at depth 6
// takes 0.633 ms instead of 0.620, its scans in fewer blocks)
constexpr int SCAN_IPT = 8;
constexpr int SCAN_CHUNK = SCAN_NT * SCAN_IPT;
constexpr int SCAN_TOP_NT = 1024;

// Entries of the index that holds the first parent of each tile of a level of
// n nodes: MAX_LEGAL_MOVES items per node in the smallest tiles.  Placements
// that no game reaches have more moves (never more than MAX_ANY_MOVES); their
// levels use tiles large enough for the index (tile_log2_for).
__host__ __device__ constexpr u64 tile_index_len(u64 n) { return (n * MAX_LEGAL_MOVES) / MAX_TILES_PER_NODE_DIV + 2; }
static_assert((u64)MAX_ANY_MOVES << TILE_MIN_LOG2 <= (u64)MAX_LEGAL_MOVES << TILE_CAP_LOG2,
              "the largest tiles always fit the index");
__host__ __device__ inline int tile_log2_for(u64 total, u64 n, int capLog2)
{
    while (capLog2 < TILE_CAP_LOG2 && (total >> capLog2) >= tile_index_len(n)) capLog2++;
    return capLog2;
}

constexpr u32 DERR_GEN_MISMATCH = 1u;
constexpr u32 DERR_BAD_ITEM = 2u;
constexpr u32 DERR_BAD_POSITION = 4u;

enum { MODE_EXPAND = 0, MODE_LEAF = 1 };

// Bytes of one level node: 6 planes + count + root + scan entry, plus its
// share of the tile index (4 B per TILE_CAP items, up to 218 items a node)
// and of the scan's block sums, rounded up.
constexpr u64 NODE_BYTES = 6 * 8 + 4 + 4 + 8 + 1;  // (tile index sized for the smallest tile: < 1 B/node)
// With merged transpositions a node also has a path weight, and the level's
// set takes MERGE_SLOTS 8-byte slots per node until the scan (whose entries
// and tile index reuse that memory).
constexpr u64 MERGE_SLOTS = 2;
constexpr u64 NODE_BYTES_MERGE = 6 * 8 + 4 + 4 + 8 + 8 * MERGE_SLOTS + 1;
// Plies from the root at which merging starts: two plies reach almost no
// position twice, the third brings the first a-x-b = b-x-a pairs.
constexpr int MERGE_MIN_PLIES = 3;
// Share of a merged level's nodes predicted to stay; predictions only choose
// the path and the grids.  The third and fourth plies keep 0.58-0.61 of their
// children, in openings and in 8-30-ply playouts alike, the initial position's
// fifth 0.46: the deeper the level, the more it is below the prediction.
constexpr double MERGE_KEPT = 0.7;

// ------------------------------------------------------- level node boards
// A level's boards in HBM are a structure of arrays of plane pairs: pair j of
// node g (planes 2j and 2j+1: mine/pawns, knights/bq, rq/kings) is one
// 16-byte vector at pp[j * stride + g].  A node is written with three 128-bit
// stores and read with three 128-bit loads, and a warp's 32 consecutive nodes
// touch 512 contiguous bytes per pair.  48 bytes per node, as six u64 planes.
__device__ __forceinline__ void level_put(u64 *planes, u64 stride, u64 g, const Board &b)
{
    ulonglong2 *pp = reinterpret_cast<ulonglong2 *>(planes);
    pp[g] = make_ulonglong2(b.mine, b.pawns);
    pp[stride + g] = make_ulonglong2(b.knights, b.bq);
    pp[2 * stride + g] = make_ulonglong2(b.rq, b.kings);
}

__device__ __forceinline__ Board level_get(const u64 *planes, u64 stride, u64 g)
{
    const ulonglong2 *pp = reinterpret_cast<const ulonglong2 *>(planes);
    const ulonglong2 a = pp[g], c = pp[stride + g], d = pp[2 * stride + g];
    return Board{a.x, a.y, c.x, c.y, d.x, d.y};
}

// --------------------------------------------------------- block helpers
template <int NT>
__device__ __forceinline__ u64 block_excl_scan_u64(u64 v, u64 *sw, u64 &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    u64 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        u64 y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sw[w] = x;
    __syncthreads();
    if (w == 0) {
        u64 t = lane < NT / 32 ? sw[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            u64 y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < NT / 32) sw[lane] = t;
    }
    __syncthreads();
    const u64 warpOff = w ? sw[w - 1] : 0;
    total = sw[NT / 32 - 1];
    __syncthreads();
    return warpOff + x - v;
}

// Adds every thread's v to a statistics counter: one atomic per block.  Every
// thread of the block must call it.
__device__ __forceinline__ void block_add_stat(unsigned long long *ctr, u32 v)
{
    __shared__ u32 sCount;
    if (threadIdx.x == 0) sCount = 0;
    __syncthreads();
    const u32 sum = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&sCount, sum);
    __syncthreads();
    if (threadIdx.x == 0 && sCount) atomicAdd(ctr, (unsigned long long)sCount);
    __syncthreads();
}

// Exclusive count of set flags over the block; total returned in *total.
template <int NT>
__device__ __forceinline__ int block_excl_count(bool flag, int *sw, int &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned b = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) sw[w] = __popc(b);
    __syncthreads();
    int off = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; i++) {
        off += (i < w) ? sw[i] : 0;
        tot += sw[i];
    }
    __syncthreads();
    total = tot;
    return off + __popc(b & ((1u << lane) - 1u));
}

// ------------------------------------------------------------------ scan
// Exclusive scan of u32 move counts into u64 item offsets (the entry after
// the last parent's is the total), plus the first parent of every tile.
//
// With COMPACT only the nodes that have items become parents: `live` lists
// them in order and the offsets are theirs.  In merged and table levels
// about 40% of the nodes have none (copies of another node, table hits);
// left in place they held 40% of the tile kernel's parent slots, so a tile
// took two staging rounds and generated moves with 40% of its threads idle.
// Without COMPACT every node is a parent, at its own index.
// Measured with compaction: depth 7 from a middlegame position 6.7 -> 6.05 ms,
// the 4096-position batch 5% less; with results staged in shared memory the
// offsets of 100 M nodes take 0.7 ms instead of 0.94.
struct ScanSums {
    u64 items, live;
};

// A chunk's items and live nodes in one word: at most SCAN_CHUNK nodes of at
// most MAX_LEGAL_MOVES moves each.
constexpr int SCAN_LIVE_SHIFT = 32;

__device__ __forceinline__ u64 scan_pack(u32 c) { return (u64)c | ((u64)(c != 0) << SCAN_LIVE_SHIFT); }

// Sums of chunk b into bsum[b].
__device__ __forceinline__ void scan_reduce_chunk(const u32 *__restrict__ cnt, u64 n, u64 b, ScanSums *bsum, u64 *sw)
{
    const u64 base = b * SCAN_CHUNK;
    u64 s = 0;
    for (int i = threadIdx.x; i < SCAN_CHUNK; i += SCAN_NT) {
        const u64 k = base + i;
        if (k < n) s += scan_pack(cnt[k]);
    }
    u64 total;
    block_excl_scan_u64<SCAN_NT>(s, sw, total);
    if (threadIdx.x == 0) bsum[b] = ScanSums{(u32)total, total >> SCAN_LIVE_SHIFT};
}

// Exclusive scan of the chunk sums in place (one block); returns the totals.
__device__ __forceinline__ ScanSums scan_top_block(ScanSums *bsum, u64 nb, u64 *sw)
{
    const u64 per = (nb + SCAN_TOP_NT - 1) / SCAN_TOP_NT;
    const u64 b0 = min(per * threadIdx.x, nb), b1 = min(b0 + per, nb);
    ScanSums s{0, 0}, total;
    for (u64 i = b0; i < b1; i++) {
        s.items += bsum[i].items;
        s.live += bsum[i].live;
    }
    ScanSums run;
    run.items = block_excl_scan_u64<SCAN_TOP_NT>(s.items, sw, total.items);
    run.live = block_excl_scan_u64<SCAN_TOP_NT>(s.live, sw, total.live);
    for (u64 i = b0; i < b1; i++) {
        const ScanSums v = bsum[i];
        bsum[i] = run;
        run.items += v.items;
        run.live += v.live;
    }
    return total;
}

// Marks the tiles whose first item belongs to parent `idx`, whose items are
// [run, run + c).  The count-only ply has no tiles (null).
__device__ __forceinline__ void scan_tiles(u32 *tileFirst, int capLog2, u64 run, u32 c, u64 idx)
{
    if (!tileFirst) return;
    const u64 t0 = (run + (1ull << capLog2) - 1) >> capLog2;
    const u64 t1 = (run + c - 1) >> capLog2;
    for (u64 t = t0; t <= t1; t++) tileFirst[t] = (u32)idx;
}

// Offsets, parent list and tile index of chunk b.  The chunk's results are
// placed in shared memory first, so that global writes are coalesced.
struct ScanShared {
    u32 c[SCAN_CHUNK];    // counts, then the parents' offsets within the chunk
    uint16_t at[SCAN_CHUNK];  // the parents' places within the chunk
    u64 sw[SCAN_NT / 32];
};

template <bool COMPACT>
__device__ __forceinline__ void scan_apply_chunk(const u32 *__restrict__ cnt, u64 n, u64 b, const ScanSums *bsum,
                                                 u64 *__restrict__ scan, u32 *__restrict__ live,
                                                 u32 *__restrict__ tileFirst, int capLog2, ScanShared &S)
{
    const u64 base = b * SCAN_CHUNK;
    for (int i = threadIdx.x; i < SCAN_CHUNK; i += SCAN_NT) {
        const u64 k = base + i;
        S.c[i] = k < n ? cnt[k] : 0u;
    }
    __syncthreads();
    u32 c[SCAN_IPT];
    u64 local = 0;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; k++) {
        c[k] = S.c[threadIdx.x * SCAN_IPT + k];
        local += scan_pack(c[k]);
    }
    u64 total;
    const u64 run0 = block_excl_scan_u64<SCAN_NT>(local, S.sw, total);  // (its barriers also end the reads of S.c)
    const ScanSums B = bsum[b];
    u32 run = (u32)run0;
    u32 place = COMPACT ? (u32)(run0 >> SCAN_LIVE_SHIFT) : threadIdx.x * SCAN_IPT;
    const u64 first = COMPACT ? B.live : base;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; k++) {
        if (!COMPACT || c[k]) {
            S.c[place] = run;
            if (COMPACT) S.at[place] = (uint16_t)(threadIdx.x * SCAN_IPT + k);
            if (c[k]) scan_tiles(tileFirst, capLog2, B.items + run, c[k], first + place);
            place++;
        }
        run += c[k];
    }
    __syncthreads();
    const u32 m = COMPACT ? (u32)(total >> SCAN_LIVE_SHIFT) : (u32)min((u64)SCAN_CHUNK, n - base);
    for (u32 i = threadIdx.x; i < m; i += SCAN_NT) {
        scan[first + i] = B.items + S.c[i];
        if (COMPACT) live[first + i] = (u32)(base + S.at[i]);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(SCAN_NT) k_scan_reduce(const u32 *__restrict__ cnt, u64 n,
                                                         ScanSums *__restrict__ bsum)
{
    __shared__ u64 sw[SCAN_NT / 32];
    scan_reduce_chunk(cnt, n, blockIdx.x, bsum, sw);
}

// totalOut[0]: items, totalOut[1]: live nodes.
__global__ void __launch_bounds__(SCAN_TOP_NT) k_scan_top(ScanSums *__restrict__ bsum, u64 nb,
                                                          u64 *__restrict__ totalOut)
{
    __shared__ u64 sw[SCAN_TOP_NT / 32];
    const ScanSums t = scan_top_block(bsum, nb, sw);
    if (threadIdx.x == 0) {
        totalOut[0] = t.items;
        totalOut[1] = t.live;
    }
}

template <bool COMPACT>
__global__ void __launch_bounds__(SCAN_NT) k_scan_apply(const u32 *__restrict__ cnt, u64 n,
                                                        const ScanSums *__restrict__ bsum,
                                                        const u64 *__restrict__ totals, u64 *__restrict__ scan,
                                                        u32 *__restrict__ live, u32 *__restrict__ tileFirst,
                                                        int capLog2)
{
    __shared__ ScanShared S;
    if (blockIdx.x == 0 && threadIdx.x == 0) scan[COMPACT ? totals[1] : n] = totals[0];
    scan_apply_chunk<COMPACT>(cnt, n, blockIdx.x, bsum, scan, live, tileFirst, capLog2, S);
}

// ----------------------------------------------------------------- roots
__global__ void k_init_roots(const u64 *__restrict__ pos48, const u32 *__restrict__ ids, u32 n,
                             u64 *__restrict__ planes, u64 stride, u32 *__restrict__ cnt,
                             u32 *__restrict__ root, unsigned long long *__restrict__ weight, int depth,
                             unsigned long long *__restrict__ rootCounts, u32 *err)
{
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const u32 id = ids[i];
    u64 p[6];
#pragma unroll
    for (int k = 0; k < 6; k++) p[k] = pos48[6 * (u64)id + k];
    u32 c = 0;
    Board b = from_pos48(p);
    if (validate_pos48(p) != 0) {
        atomicOr(err, DERR_BAD_POSITION);
    } else {
        c = count_moves<SV_KOGGE>(b);
    }
    level_put(planes, stride, i, b);
    cnt[i] = c;
    root[i] = id;
    if (weight) weight[i] = 1ull;
    if (depth == 0) rootCounts[id] = 1ull;
    if (depth == 1) rootCounts[id] = c;
}

// ------------------------------------------- device-driven level pipeline
// The scan of level k runs with a fixed grid (grid-stride over chunks), its
// top block computes the total and bump-allocates level k+1 and that
// level's scan buffers from a device-resident plan.  No host round trip
// separates the plies, so a whole perft is one captured CUDA graph.  If the
// region is exhausted the plan's overflow flag is raised, every following
// level is empty, and the host reruns the batch on the host-driven path.
// A level whose sizes and buffers are decided on the device (device-driven
// pipeline, no host round trip between plies).
struct LevelDesc {
    u64 *planes;
    u64 stride;
    u32 *cnt;
    u32 *root;
    unsigned long long *weight;  // merged runs: paths that reach the node
    unsigned long long *set;     // merged levels: the set's slots (transient), null when they do not fit
    u64 n;        // nodes: the previous ply's children, then the roots joining here
    u64 nChild;   // children written by the previous ply's tile kernel
    u32 *live;  // merged levels: the nodes with items, in order (null: all nodes are parents)
    u64 *pscan;
    u32 *tileFirst;
    ScanSums *bsum;
    u64 total;
    int capLog2;  // tile size of this level's items
};

struct TileParams {
    const u64 *ppl;   // parent planes, plane i at ppl + i * pstride
    u64 pstride;
    const u64 *pscan; // nParents + 1 item offsets
    const u32 *live;  // node index of each parent; null: the parent's own index
    const u32 *proot;  // root id of each parent; null: sums go to the parent's own slot
    const unsigned long long *pweight;  // paths that reach each parent; null: one each
    u64 nParents;
    const u32 *tileFirst;  // indexed by absolute tile number
    u64 itemBase;     // first item of this launch (multiple of the tile size)
    u64 itemEnd;      // one past the last item
    int capLog2;      // tile size of this level (the scan's tileFirst granularity)
    u32 *tileCounter; // work-stealing cursor, zeroed before launch
    // interior ply outputs (child index = item - itemBase)
    u64 *cpl;
    u64 cstride;
    u32 *ccnt;
    u32 *croot;
    unsigned long long *cweight;  // null: not kept
    u32 uncounted;    // the children are the count-only ply's parents: every count is written as 1
    // last ply output
    unsigned long long *rootCounts;
    unsigned long long *moves;  // statistics: moves of the parents (null: not kept)
    u32 *err;
    // serving: pending-node counter of each query slot (TRACK kernels only)
    unsigned long long *pending;
    // device-driven DD_SHARED launches: the plan's entry for this launch
    const struct TileParams *planEntry;
};


// The nodes of one root in a level (they are contiguous).
struct MergeSeg {
    u32 begin, end;
};

constexpr int DD_MAX_LEVELS = 24;
// Largest predicted tree (bytes of materialised plies) run as a graph, on top
// of the arena check: no limit unless PERFT_DD_MAX_GB sets one.
constexpr double DD_MAX_BYTES_DEFAULT = 1e30;
// Plies predicted to have fewer items than this read their launch
// parameters through shared memory instead of a constant-bank copy node.
constexpr double DD_CONST_MIN_ITEMS = double(1u << 22);
struct DevPlan {
    char *base;
    u64 cap;
    u64 bump;
    u32 overflow;
    unsigned long long leafMoves;  // moves of the count-only ply's parents
    u32 tileTarget;  // smallest tile count a level should have (2 x resident CTAs)
    LevelDesc lv[DD_MAX_LEVELS];
    // roots that join level k (their depth is the level's remaining depth)
    u32 joinN[DD_MAX_LEVELS];
    const u32 *joinIds[DD_MAX_LEVELS];
    int capMax[DD_MAX_LEVELS];  // largest tile (log2 items) for the items of level k (interior plies)
    int lastLv;                    // the count-only ply's level
    int weighted;                  // levels carry path weights (some level is merged)
    int mergeLv[DD_MAX_LEVELS];    // level k's transpositions are merged
    MergeSeg *segs;                // per root: its nodes in the level being merged
    const uint8_t *rootDepth;
    // the tile launch of level k's items, completed on the device by the scan
    // (level pointers and sizes) and copied into c_ddTile before that launch
    TileParams tp[DD_MAX_LEVELS];
    u32 *tileCounter;  // the tile launches' work-stealing cursor, reset by each scan
};

// The parameters of the device-driven tile launch about to run.  A graph
// copies the plan's entry for the level here (a device-to-device copy node)
// before each tile launch, so the kernel reads them from the constant bank,
// as a plain launch reads its parameters, instead of holding plan pointers
// in registers or shared memory.  Only the device-driven graphs use it, and
// they run one at a time on the engine's stream.
__constant__ TileParams c_ddTile;

// Nodes of a level as the scans see it.  Once the plan has overflowed every
// level is empty: buffers of levels that were planned but not written hold
// whatever an earlier call left there.
__device__ __forceinline__ u64 dd_nodes(const DevPlan *plan, const LevelDesc &L) { return plan->overflow ? 0 : L.n; }

__device__ __forceinline__ void *dd_take(DevPlan *plan, u64 bytes)
{
    const u64 a = (plan->bump + 255) & ~255ULL;
    if (a + bytes > plan->cap) {
        plan->overflow = 1;
        return nullptr;
    }
    plan->bump = a + bytes;
    return plan->base + a;
}

__global__ void __launch_bounds__(SCAN_NT) k_dd_scan_reduce(DevPlan *plan, int lv)
{
    __shared__ u64 sw[SCAN_NT / 32];
    const LevelDesc &L = plan->lv[lv];
    const u64 n = dd_nodes(plan, L), nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    for (u64 b = blockIdx.x; b < nb; b += gridDim.x) scan_reduce_chunk(L.cnt, n, b, L.bsum, sw);
}

__device__ void dd_plan_level(DevPlan *plan, int lv, int last, ScanSums total);

__global__ void __launch_bounds__(SCAN_TOP_NT) k_dd_scan_top(DevPlan *plan, int lv, int last)
{
    __shared__ u64 sw[SCAN_TOP_NT / 32];
    LevelDesc &L = plan->lv[lv];
    const ScanSums total = scan_top_block(L.bsum, (dd_nodes(plan, L) + SCAN_CHUNK - 1) / SCAN_CHUNK, sw);
    if (threadIdx.x == 0) dd_plan_level(plan, lv, last, total);
}

// Whole-level scan in one block: the total, the tile size and the next level
// (dd_plan_level), then the offsets and tile index, 4096 nodes per pass.
// Used for levels predicted small, where three launches (each with its own
// latency) would cost more than the work; correct for any size.  A level of
// one pass takes its total from the pass's own scan.
__global__ void __launch_bounds__(1024) k_dd_scan_small(DevPlan *plan, int lv, int last)
{
    constexpr int IPT = 4, PASS = 1024 * IPT;
    __shared__ u64 sw[32];
    __shared__ int sCap;
    LevelDesc &L = plan->lv[lv];
    const u64 n = dd_nodes(plan, L);
    const u32 *cnt = L.cnt;
    u32 c[IPT];
    u64 x, tot;  // this thread's place in the pass's scan, and the pass's sums
    auto scan_pass = [&](u64 c0) {
        u64 local = 0;
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const u64 i = c0 + (u64)threadIdx.x * IPT + k;
            c[k] = i < n ? cnt[i] : 0u;
            local += scan_pack(c[k]);
        }
        x = block_excl_scan_u64<1024>(local, sw, tot);
    };
    if (n > PASS) {
        u64 s = 0, a = 0;
        for (u64 i = threadIdx.x; i < n; i += 1024) {
            const u32 v = cnt[i];
            s += v;
            a += v != 0;
        }
        ScanSums total;
        block_excl_scan_u64<1024>(s, sw, total.items);
        block_excl_scan_u64<1024>(a, sw, total.live);
        if (threadIdx.x == 0) dd_plan_level(plan, lv, last, total);
        scan_pass(0);
    } else {
        scan_pass(0);
        if (threadIdx.x == 0) dd_plan_level(plan, lv, last, ScanSums{(u32)tot, tot >> SCAN_LIVE_SHIFT});
    }
    if (threadIdx.x == 0) sCap = L.capLog2;
    __syncthreads();
    const int cl = sCap;
    u64 *pscan = L.pscan;
    u32 *live = L.live;
    u32 *tileFirst = L.tileFirst;
    u64 base = 0, place0 = 0;
    for (u64 c0 = 0;;) {
        u64 run = base + (u32)x, place = place0 + (x >> SCAN_LIVE_SHIFT);
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const u64 i = c0 + (u64)threadIdx.x * IPT + k;
            const u64 at = live ? place : i;
            if (live ? c[k] != 0 : i < n) {
                pscan[at] = run;
                if (live) live[at] = (u32)i;
                if (c[k]) scan_tiles(tileFirst, cl, run, c[k], at);
            }
            run += c[k];
            place += c[k] != 0;
        }
        base += (u32)tot;
        place0 += tot >> SCAN_LIVE_SHIFT;
        c0 += PASS;
        if (c0 >= n) break;
        scan_pass(c0);
    }
}

// Top-of-scan bookkeeping of a device-driven level (one thread): the level's
// total and tile size, then the next level's buffers from the plan's bump
// allocator (children plus the roots joining there).
__device__ void dd_plan_level(DevPlan *plan, int lv, int last, ScanSums sums)
{
    LevelDesc &L = plan->lv[lv];
    const u64 n = dd_nodes(plan, L);
    const u64 total = sums.items;
    const u64 nParents = L.live ? sums.live : n;
    if (n) L.pscan[nParents] = total;
    L.total = total;  // (0 when the plan has overflowed: the sums are those of no nodes)
    int cap = TILE_CAP_LOG2;
    if (!last) {  // (the count-only ply has no tiles)
        cap = plan->capMax[lv];
        while (cap > TILE_MIN_LOG2 && (total >> cap) < plan->tileTarget) cap--;
        cap = tile_log2_for(total, n, cap);
    }
    L.capLog2 = cap;
    *plan->tileCounter = 0;  // the next launch is this level's tile launch
    TileParams &T = plan->tp[lv];  // host fields (cursor, outputs, error word) come from the template
    T.ppl = L.planes;
    T.pstride = L.stride;
    T.pscan = L.pscan;
    T.proot = L.root;
    T.pweight = L.weight;
    T.live = L.live;
    T.nParents = nParents;
    T.tileFirst = L.tileFirst;
    T.itemBase = 0;
    T.itemEnd = L.total;
    T.capLog2 = cap;
    if (last) return;
    LevelDesc &C = plan->lv[lv + 1];
    const u64 m = L.total + plan->joinN[lv + 1];
    C.n = m;
    C.nChild = L.total;
    C.stride = (m + 31) & ~31ULL;
    C.total = 0;
    C.planes = (u64 *)dd_take(plan, 48 * C.stride);
    C.cnt = (u32 *)dd_take(plan, 4 * C.stride);
    C.root = (u32 *)dd_take(plan, 4 * C.stride);
    C.weight = plan->weighted ? (unsigned long long *)dd_take(plan, 8 * C.stride) : nullptr;
    C.live = plan->mergeLv[lv + 1] ? (u32 *)dd_take(plan, 4 * C.stride) : nullptr;
    C.pscan = (u64 *)dd_take(plan, 8 * (m + 1));
    C.tileFirst = lv + 1 < plan->lastLv
                      ? (u32 *)dd_take(plan, 4 * tile_index_len(m))
                      : nullptr;
    C.bsum = (ScanSums *)dd_take(plan, sizeof(ScanSums) * ((m + SCAN_CHUNK - 1) / SCAN_CHUNK + 1));
    if (plan->overflow) {
        C.n = 0;
        L.total = 0;  // nothing is expanded into a level that does not exist
        T.nParents = 0;
    }
    // The merge set lies above the bump mark: it is done with before the next
    // level's buffers are placed there.  A set that does not fit leaves the
    // level unmerged.
    const u64 setAt = (plan->bump + 255) & ~255ULL;
    C.set = plan->mergeLv[lv + 1] && !plan->overflow && setAt + 8 * MERGE_SLOTS * m <= plan->cap
                ? (unsigned long long *)(plan->base + setAt)
                : nullptr;
    T.itemEnd = L.total;
    T.cpl = C.planes;
    T.cstride = C.stride;
    T.ccnt = C.cnt;
    T.croot = C.root;
    T.cweight = C.weight;
}

template <bool COMPACT>
__global__ void __launch_bounds__(SCAN_NT) k_dd_scan_apply(DevPlan *plan, int lv)
{
    __shared__ ScanShared S;
    const LevelDesc &L = plan->lv[lv];
    const u64 n = dd_nodes(plan, L), nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    for (u64 b = blockIdx.x; b < nb; b += gridDim.x)
        scan_apply_chunk<COMPACT>(L.cnt, n, b, L.bsum, L.pscan, L.live, L.tileFirst, L.capLog2, S);
}

// Roots joining level lv of a device-driven run: written behind the
// children, from the position array (as k_init_roots does).  Nothing is
// written into a level that overflowed the plan.
__global__ void k_dd_join(DevPlan *plan, int lv, const u64 *__restrict__ pos48, u32 *err)
{
    const LevelDesc &C = plan->lv[lv];
    const u32 nj = plan->joinN[lv];
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nj || dd_nodes(plan, C) == 0) return;
    const u32 id = plan->joinIds[lv][i];
    u64 p[6];
#pragma unroll
    for (int k = 0; k < 6; k++) p[k] = pos48[6 * (u64)id + k];
    u32 c = 0;
    const Board b = from_pos48(p);
    if (validate_pos48(p) != 0) atomicOr(err, DERR_BAD_POSITION);
    else c = count_moves<SV_KOGGE>(b);
    const u64 g = C.nChild + i;
    level_put(C.planes, C.stride, g, b);
    C.cnt[g] = c;
    C.root[g] = id;
    if (C.weight) C.weight[g] = 1ull;
}

// ------------------------------------------------- merged transpositions
// Different move orders reach the same position.  From the third ply below a
// root on, a level therefore holds many equal nodes (about 40% of the third
// ply's children and again 40% of the fourth's, in openings and in 8-30-ply
// playouts), and each copy's whole subtree would be searched again.  Before a level is scanned,
// equal nodes of one root are merged: one of them, the owner, keeps its
// moves and takes over the others' path weights; the others lose theirs
// (cnt = 0).  A node's weight is the number of move paths from its root that
// reach it, children inherit their parent's, and the count-only ply adds
// weight x moves, so the root's count is the same.  Nodes are merged only
// when their boards (state included) are equal in all 48 bytes: the hash
// only picks the slot.
//
// The set is open addressed, MERGE_SLOTS 8-byte slots {hash tag, node} per
// node.  Each root's nodes use the slots at their own place in the set, so a
// batch works on one small region of the set and of the boards at a time
// and most of its random accesses stay in L2.  Which of several equal nodes
// becomes the owner depends on timing; the sums do not.
// Bound by the latency of its chain of dependent accesses (segment, slot,
// owner's board): one node per thread, and enough CTAs to fill every SM.
// Measured: 4096 playouts of depths 4-6 1588 -> 671 ms, one middlegame
// position at depth 7 34.2 -> 6.8 ms, an opening at depth 8 365 -> 35 ms.
constexpr unsigned long long MERGE_EMPTY = ~0ULL;
constexpr int MERGE_MAX_PROBES = 64;
// One node per thread wherever the grid can be that large: blocks then start
// in level order and work on one root's region at a time.  512 positions of
// depths 4-6, 100 M nodes: 4.05 ms; with 64 blocks per SM striding through the
// level 5.2, 16 per SM 7.6, one resident wave 10.4.
constexpr int MERGE_CTAS = 5;  // resident per SM

struct MergeLevel {
    const u64 *planes;
    u64 stride, n;
    u32 *cnt;
    const u32 *root;
    unsigned long long *weight;
    unsigned long long *set;
    MergeSeg *segs;
    const uint8_t *rootDepth;  // null: every root is deep enough
    int remaining;  // plies left below the level
    bool initWeight;  // the weights are not set yet: one path each
    // linked levels (below): each node's owner, and the subtree sums to clear
    u32 *alias;
    unsigned long long *acc;
    unsigned long long *merged;  // statistics: nodes merged
};

// Owner links.  Levels whose subtree sums flow up node by node (with a
// transposition table, or with related roots) are merged over all roots: a
// copy remembers its owner in `alias` and takes the owner's sum when the
// level is finished (k_tt_finish), instead of handing over its weight.
constexpr u32 ALIAS_HIT = 0xFFFFFFFFu;     // final value in acc: from the table, or no moves
constexpr u32 ALIAS_NOSLOT = 0xFFFFFFFEu;  // searched by itself (no slot found in the set)

// Multiplies each word by an odd constant and finishes with xor-shifts.  The
// constants are known 64-bit hash multipliers: 2^64 / golden ratio, two of
// xxHash64's primes (the second and third), degski's 64-bit mixer's multiplier
// and two of wyhash's defaults.
__device__ __forceinline__ u64 board_hash(const Board &b)
{
    u64 h = b.mine * 0x9E3779B97F4A7C15ULL + b.pawns * 0xC2B2AE3D27D4EB4FULL + b.knights * 0x165667B19E3779F9ULL +
            b.bq * 0xD6E8FEB86659FD93ULL + b.rq * 0xA0761D6478BD642FULL + b.kings * 0xE7037ED1A0B428DBULL;
    h ^= h >> 32;
    h *= 0xD6E8FEB86659FD93ULL;
    h ^= h >> 29;
    h *= 0x9E3779B97F4A7C15ULL;
    return h ^ (h >> 32);
}

// Clears the set and finds every root's nodes.  Roots fewer than
// MERGE_MIN_PLIES above the level get an empty segment: nothing to merge.
__device__ __forceinline__ void merge_prepare(const MergeLevel &M)
{
    const u64 t0 = (u64)blockIdx.x * blockDim.x + threadIdx.x, step = (u64)gridDim.x * blockDim.x;
    ulonglong2 *set2 = reinterpret_cast<ulonglong2 *>(M.set);
    for (u64 i = t0; i < M.n; i += step) {
        set2[i] = make_ulonglong2(MERGE_EMPTY, MERGE_EMPTY);
        if (M.initWeight) M.weight[i] = 1ull;
        const u32 r = M.root[i];
        const bool deep = !M.rootDepth || M.rootDepth[r] >= M.remaining + MERGE_MIN_PLIES;
        if (i == 0 || M.root[i - 1] != r) M.segs[r].begin = deep ? (u32)i : 0u;
        if (i + 1 == M.n || M.root[i + 1] != r) M.segs[r].end = deep ? (u32)(i + 1) : 0u;
    }
}

template <bool LINKED>
__device__ __forceinline__ void merge_nodes(const MergeLevel &M)
{
    const u64 t0 = (u64)blockIdx.x * blockDim.x + threadIdx.x, step = (u64)gridDim.x * blockDim.x;
    u32 nMerged = 0;
    for (u64 i = t0; i < M.n; i += step) {
        u32 link = ALIAS_HIT;
        if (LINKED) M.acc[i] = 0;
        if (M.cnt[i]) {  // (no moves: nothing below to search)
            link = ALIAS_NOSLOT;
            MergeSeg sg{0, (u32)M.n};
            if (!LINKED) sg = M.segs[M.root[i]];
            if (!LINKED && sg.end - sg.begin < 2) continue;
            Board b = level_get(M.planes, M.stride, i);
            // nodes of different roots may differ in the real side to move,
            // which no count depends on
            if (LINKED) b.pawns &= ~SIDE_BIT;
            const u64 h = board_hash(b);
            const u64 nSlots = MERGE_SLOTS * (u64)(sg.end - sg.begin);
            unsigned long long *slots = M.set + MERGE_SLOTS * (u64)sg.begin;
            const unsigned long long mine = (h << 32) | (u32)i;
            u64 at = __umul64hi(h, nSlots);
            for (int k = 0; k < MERGE_MAX_PROBES; k++) {
                unsigned long long v = *(volatile unsigned long long *)(slots + at);
                if (v == MERGE_EMPTY) {
                    v = atomicCAS(slots + at, MERGE_EMPTY, mine);
                    if (v == MERGE_EMPTY) {  // this node owns its position
                        link = (u32)i;
                        break;
                    }
                }
                if ((v >> 32) == (u32)h) {
                    const u32 o = (u32)v;
                    Board ob = level_get(M.planes, M.stride, o);
                    if (LINKED) ob.pawns &= ~SIDE_BIT;
                    if (((ob.mine ^ b.mine) | (ob.pawns ^ b.pawns) | (ob.knights ^ b.knights) | (ob.bq ^ b.bq) |
                         (ob.rq ^ b.rq) | (ob.kings ^ b.kings)) == 0) {
                        if (!LINKED) atomicAdd(M.weight + o, M.weight[i]);
                        M.cnt[i] = 0;
                        link = o;
                        nMerged++;
                        break;
                    }
                }
                if (++at == nSlots) at = 0;
            }
        }
        if (LINKED) M.alias[i] = link;
    }
    if (LINKED) block_add_stat(M.merged, nMerged);
}

__global__ void __launch_bounds__(256) k_merge_prepare(const MergeLevel M) { merge_prepare(M); }
__global__ void __launch_bounds__(256, MERGE_CTAS) k_merge_nodes(const MergeLevel M) { merge_nodes<false>(M); }
__global__ void __launch_bounds__(256, MERGE_CTAS) k_merge_linked(const MergeLevel M) { merge_nodes<true>(M); }

// The same for a device-driven level.
__device__ __forceinline__ MergeLevel dd_merge_level(const DevPlan *plan, int lv, int remaining)
{
    const LevelDesc &C = plan->lv[lv];
    return MergeLevel{C.planes, C.stride, C.set ? dd_nodes(plan, C) : 0, C.cnt, C.root, C.weight, C.set,
                      plan->segs, plan->rootDepth, remaining, false, nullptr, nullptr, nullptr};
}
__global__ void __launch_bounds__(256) k_dd_merge_prepare(const DevPlan *plan, int lv, int remaining)
{
    merge_prepare(dd_merge_level(plan, lv, remaining));
}
__global__ void __launch_bounds__(256, MERGE_CTAS) k_dd_merge_nodes(const DevPlan *plan, int lv, int remaining)
{
    merge_nodes<false>(dd_merge_level(plan, lv, remaining));
}

// ------------------------------------------------------------ tile kernel



// Emits a parent's moves, keeping only those whose global item index falls
// inside [lo, hi): the window of the current tile.
// Positions are relative to the window start: a parent starts at most
// MAX_LEGAL_MOVES items before it and a window holds at most TILE_CAP items,
// so 32 bits hold them and one unsigned compare does the bounds test.
struct WindowSink {
    u32 *items;
    int rel;  // next move's position relative to the window start
    u32 n;    // window length
    u32 tag;
    __device__ __forceinline__ void operator()(u32 m)
    {
        if ((u32)rel < n) items[rel] = tag | m;
        ++rel;
    }
};

// Makes an item's move on its (mirrored) parent and counts the child's moves.
template <int SV>
__device__ __forceinline__ u32 tile_make_count(const Board &b, u32 it, int kO, int kS, Board &ch)
{
    if (PG_KNOWN_KINGS && PG_MIRRORED_STAGE && PG_KNOWN_OCC) {
        int tk;
        u64 occ, theirs;
        ch = make_child_mirrored(b, it, &tk, kS, &occ, &theirs);
        return count_moves_ko<SV>(ch, kO, tk, occ, theirs);
    }
    if (PG_KNOWN_KINGS && PG_MIRRORED_STAGE) {
        int tk;
        ch = make_child_mirrored(b, it, &tk, kS);
        return count_moves_k<SV>(ch, kO, tk);
    }
    ch = PG_MIRRORED_STAGE ? make_child_mirrored(b, it) : make_child<PG_MOVER_BITS>(b, it);
    return count_moves<SV>(ch);
}

// TRACK (serving): besides the counts, every root run also accumulates the
// change of its query's pending-node counter: +1 per child written, -1 when
// a parent's last item is processed.  The counter reaching zero means the
// query's subtree is fully counted.
// DD: 0 for plain launches (parameters in the parameter bank); DD_SHARED or
// DD_CONST for the device-driven graph's launches (below).
enum { DD_NONE = 0, DD_SHARED = 1, DD_CONST = 2 };
template <int SV, bool TRACK = false, int DD = DD_NONE>
__global__ void __launch_bounds__(TILE_NT, TILE_MINB) k_tile(const TileParams Pin)
{
    // Device-driven launches take the level pointers and sizes from the plan:
    //  * DD_CONST reads them from the constant bank (c_ddTile, which the graph
    //    fills by a copy node before the launch), exactly as a plain launch
    //    reads its parameter bank.  Used for large plies: held in registers
    //    across the make-and-count loop the pointers compete with the count at
    //    the 80-register cap (5% slower), and read from shared memory they
    //    still cost 1.3%; from the constant bank the count-only launch of the
    //    4096-position batch takes the same time as a plain launch.
    //  * DD_SHARED reads the plan entry into shared memory at the start of the
    //    launch.  Used for small plies, where the copy node's few microseconds
    //    would cost more than they save.
    __shared__ TileParams sP;
    if (DD == DD_SHARED) {
        if (threadIdx.x == 0) sP = *Pin.planEntry;
        __syncthreads();
    }
    const TileParams &P = DD == DD_CONST ? c_ddTile : (DD == DD_SHARED ? sP : Pin);
    __shared__ u64 sb[6][TILE_MAXP];
    // king squares in the children's frame: the side to move there (the
    // parent's opponent) and the parent's mover
    __shared__ uint8_t skO[PG_KNOWN_KINGS ? TILE_MAXP : 1], skS[PG_KNOWN_KINGS ? TILE_MAXP : 1];
    __shared__ u64 sqEnd[TRACK ? TILE_MAXP : 1];
    __shared__ int sdelta[TRACK ? TILE_MAXP : 1];
    __shared__ u32 sroot[TILE_MAXP];
    __shared__ unsigned long long sweight[TILE_MAXP];  // paths that reach each parent
    __shared__ u32 srun[TRACK ? TILE_MAXP : 1];
    __shared__ u32 srunRoot[TRACK ? TILE_MAXP : 1];
    extern __shared__ __align__(16) u32 sitems[];  // TILE_CAP items (dynamic: may exceed 48 KB)
    __shared__ int swarp[TILE_NT / 32];
    __shared__ u32 sTile;

    const int tid = threadIdx.x, lane = tid & 31;
    const int capLog2 = P.capLog2;
    const u64 tile0 = P.itemBase >> capLog2;
    const u64 nTiles = (P.itemEnd - P.itemBase + (1ull << capLog2) - 1) >> capLog2;

    for (;;) {
        if (tid == 0) sTile = atomicAdd(P.tileCounter, 1u);
        __syncthreads();
        const u64 tl = sTile;
        if (tl >= nTiles) break;
        const u64 iBeg = P.itemBase + (tl << capLog2);
        const u64 iEnd = min(iBeg + ((u64)1 << capLog2), P.itemEnd);
        u64 p = P.tileFirst[tile0 + tl];

        for (;;) {
            // ---- stage the parents that own items of this window
            const u64 q = p + tid;
            u64 qBeg = 0, qEnd = 0;
            bool valid = false;
            if (q < P.nParents) {
                qBeg = P.pscan[q];
                valid = qBeg < iEnd;
            }
            const int nP = __syncthreads_count(valid);
            if (valid) {
                qEnd = P.pscan[q + 1];
                if (TRACK) sqEnd[tid] = qEnd;
                const u64 node = P.live ? P.live[q] : q;
                // mirrored staging: the per-parent flips here replace six
                // byte swaps per child in make-move
                const Board lb = level_get(P.ppl, P.pstride, node);
                const Board pb = PG_MIRRORED_STAGE ? flip_board(lb) : lb;
                sb[0][tid] = pb.mine;
                sb[1][tid] = pb.pawns;
                sb[2][tid] = pb.knights;
                sb[3][tid] = pb.bq;
                sb[4][tid] = pb.rq;
                sb[5][tid] = pb.kings;
                if (PG_KNOWN_KINGS && PG_MIRRORED_STAGE) {
                    skO[tid] = (uint8_t)ctz(pb.kings & ~pb.mine);
                    skS[tid] = (uint8_t)ctz(pb.kings & pb.mine);
                }
                sroot[tid] = P.proot ? P.proot[node] : (u32)node;  // no root array: account to the parent itself
                sweight[tid] = P.pweight ? P.pweight[node] : 1ull;
            }
            const u64 sBeg = max(P.pscan[p], iBeg);
            const u64 sEnd = min(P.pscan[p + nP], iEnd);
            __syncthreads();

            int nRuns = 0;
            if (TRACK) {
                // parents are ordered by root: number the runs of equal roots.
                // Usually the whole window belongs to one root, which one
                // block vote settles without the two-barrier run count.
                if (PG_ONE_RUN_VOTE && nP > 0 && __syncthreads_and(!valid || sroot[tid] == sroot[0])) {
                    nRuns = 1;
                    if (valid) srun[tid] = 0;
                    if (tid == 0) {
                        srunRoot[0] = sroot[0];
                        sdelta[0] = 0;
                    }
                } else {
                    const bool head = valid && (tid == 0 || sroot[tid] != sroot[tid - 1]);
                    const int r = block_excl_count<TILE_NT>(head, swarp, nRuns);
                    if (valid) srun[tid] = head ? r : r - 1;
                    if (head) {
                        srunRoot[r] = sroot[tid];
                        sdelta[r] = 0;
                    }
                }
            }

            // ---- generate the window's moves into the shared item list
            // parents without items (none legal, or answered by the table) generate nothing
            if (valid && qEnd > qBeg && qEnd > sBeg && qBeg < sEnd) {
                const Board sbt{sb[0][tid], sb[1][tid], sb[2][tid], sb[3][tid], sb[4][tid], sb[5][tid]};
                const Board b = PG_MIRRORED_STAGE ? flip_board(sbt) : sbt;
                WindowSink sink{sitems, (int)((long long)qBeg - (long long)sBeg), (u32)(sEnd - sBeg), (u32)tid << 16};
                gen_moves<SV, PG_MOVER_BITS>(b, sink);  // items carry the mover's planes
                if ((long long)sink.rel != (long long)qEnd - (long long)sBeg) atomicOr(P.err, DERR_GEN_MISMATCH);
            }
            __syncthreads();

            // ---- every thread takes items: make, count, write
            const int nItems = (int)(sEnd - sBeg);
            for (int j0 = 0; j0 < nItems; j0 += TILE_NT) {
                const int j = j0 + tid;
                const bool act = j < nItems;
                int pl = 0;
                if (act) {
                    const u32 it = sitems[j];  // move (bits 0-15), parent slot (16-23), mover planes (24-28)
                    pl = (int)((it >> 16) & 0xFFu);
                    if (pl < nP) {
                        const Board b{sb[0][pl], sb[1][pl], sb[2][pl], sb[3][pl], sb[4][pl], sb[5][pl]};
                        Board ch;
                        // The count-only ply needs no move counts of its parents, and
                        // 42% of these children are merged away; without the counts
                        // depth 7 takes 3.96 -> 3.67 ms, a batch 41.5 -> 39.4.
                        u32 cnt = 1;
                        if (P.uncounted)
                            ch = PG_MIRRORED_STAGE ? make_child_mirrored(b, it) : make_child<PG_MOVER_BITS>(b, it);
                        else
                            cnt = tile_make_count<SV>(b, it, skO[PG_KNOWN_KINGS ? pl : 0], skS[PG_KNOWN_KINGS ? pl : 0],
                                                      ch);
                        const u64 g = sBeg + (u64)j - P.itemBase;
                        level_put(P.cpl, P.cstride, g, ch);
                        P.ccnt[g] = cnt;
                        P.croot[g] = sroot[pl];
                        if (P.cweight) P.cweight[g] = sweight[pl];
                    } else {
                        atomicOr(P.err, DERR_BAD_ITEM);
                        pl = 0;
                    }
                }
                if (TRACK) {
                    const u32 key = act ? srun[pl] : 0xFFFFFFFFu;
                    const unsigned peers = __match_any_sync(0xffffffffu, key);
                    const bool lastOfParent = act && (sBeg + (u64)j + 1 == sqEnd[pl]);
                    const int d = (act ? 1 : 0) - (lastOfParent ? 1 : 0);
                    const int dsum = __reduce_add_sync(peers, d);
                    if (act && lane == __ffs(peers) - 1 && dsum) atomicAdd(&sdelta[key], dsum);
                }
            }
            __syncthreads();
            if (TRACK && tid < nRuns && sdelta[tid])
                atomicAdd(&P.pending[srunRoot[tid]], (unsigned long long)(long long)sdelta[tid]);
            if (sEnd >= iEnd || p + nP >= P.nParents) break;
            p += nP;
            __syncthreads();
        }
        __syncthreads();
    }
}

// -------------------------------------------------------- count-only last ply
// Counts the replies to every move of a level's parents (remaining depth 2)
// and adds weight x replies per root.  One thread generates a parent's moves;
// the replies to its quiet moves, about two thirds, are summed from the
// position alone (movegen.cuh, QuietCtx) without making the moves, and only
// the rest go to the shared item list, where every thread takes items, makes
// the move and counts.  CTAs take LEAF_NT consecutive parents at a time.
//
// Bound by the integer pipes (ALU 74% busy) and by instruction fetch: a
// counted item issues about 950 thread instructions, a parent's generation
// and analysis about 5000, so counting a quarter of the 33 items is a third of
// counting all of them.  Measured against making and counting every item:
// 4096 playouts of depths 4-6 656 -> 452 ms with two thirds counted as sets,
// tiles of 8192 items and straight-line analysis; per item of that ply then
// (depth 7 of a middlegame position / a batch / an opening at depth 8)
//   straight-line analysis, tiles of 8192 items   23.4 / 22.4 / 19.7 ps
//   loops over lines, pieces and pawn moves       21.8 / 21.8 / 17.8
//   units of LEAF_NT parents (a tile of 8192 items had 240-300 parents, the
//   part beyond 256 in a round of its own)        18.5 / 20.3 / 15.0
//   attacks told apart by line, exact king lines  16.5 / 18.5 / 14.3
//   replies added per parent in shared memory (before: per root, grouped in
//   each warp, weight by weight)                  15.3 / 17.3 / 13.3
// and with a sum for every parent (table levels) 22.9 -> 19.3.
// Slower: 128-thread CTAs, 6 per SM (26.4 / 25.7 / 22.5 against 21.8 / 21.8 /
// 17.8) and warps that work by themselves without barriers (34.7 / 37.3 /
// 29.0): warps at different places fetch each instruction again.  384 threads,
// 2 per SM: the same within 1%.
struct LeafSink {
    u32 *items;
    u32 *count;
    u32 at, tag, n;
    __device__ __forceinline__ void room(int k)
    {
        at = atomicAdd(count, (u32)k);
        n += (u32)k;
    }
    __device__ __forceinline__ void operator()(u32 m)
    {
        if (at < LEAF_ITEMS) items[at] = tag | m;
        ++at;
    }
};

template <int SV, bool TRACK = false, int DD = DD_NONE>
__global__ void __launch_bounds__(LEAF_NT, LEAF_MINB) k_leaf(const TileParams Pin)
{
    __shared__ TileParams sP;  // (see k_tile)
    if (DD == DD_SHARED) {
        if (threadIdx.x == 0) sP = *Pin.planEntry;
        __syncthreads();
    }
    const TileParams &P = DD == DD_CONST ? c_ddTile : (DD == DD_SHARED ? sP : Pin);
    __shared__ u64 sb[6][LEAF_NT];
    __shared__ uint8_t skO[LEAF_NT], skS[LEAF_NT];  // king squares in the children's frame (see k_tile)
    __shared__ u32 sroot[LEAF_NT];
    __shared__ unsigned long long sweight[LEAF_NT];  // paths that reach each parent
    __shared__ u32 sreplies[LEAF_NT];  // to each parent's listed moves
    __shared__ uint16_t scounted[LEAF_NT];  // each parent's moves as the level counted them
    __shared__ unsigned long long ssum;
    __shared__ u32 smoves;
    __shared__ int sdone;
    extern __shared__ __align__(16) u32 sitems[];  // LEAF_ITEMS
    __shared__ u32 sUnit, sCount;

    const int tid = threadIdx.x, lane = tid & 31;
    // small levels: fewer parents per unit, so that every CTA gets some
    int perUnit = LEAF_NT;
    while (perUnit > LEAF_MIN_UNIT && P.nParents < (u64)perUnit * gridDim.x) perUnit >>= 1;
    const u64 nUnits = (P.nParents + perUnit - 1) / perUnit;

    for (;;) {
        if (tid == 0) sUnit = atomicAdd(P.tileCounter, 1u);
        __syncthreads();
        if (sUnit >= nUnits) break;
        // ---- stage the unit's parents (serving: those whose first item is in the step).
        // The level's counts say only which nodes have items (see `uncounted`).
        const u64 q = (u64)sUnit * perUnit + tid;
        const bool inUnit = tid < perUnit && q < P.nParents;
        bool active = false;
        sreplies[tid] = 0;
        if (tid == 0) {
            sCount = 0;
            ssum = 0;
            smoves = 0;
            sdone = 0;
        }
        if (inUnit) {
            const u64 beg = P.pscan[q], end = P.pscan[q + 1];
            active = beg >= P.itemBase && beg < P.itemEnd && end != beg;
            scounted[tid] = (uint16_t)(end - beg);
            const u64 node = P.live ? P.live[q] : q;
            sroot[tid] = P.proot ? P.proot[node] : (u32)node;  // no root array: account to the parent itself
            sweight[tid] = P.pweight ? P.pweight[node] : 1ull;
            const Board pb = flip_board(level_get(P.ppl, P.pstride, node));  // mirrored (see k_tile)
            sb[0][tid] = pb.mine;
            sb[1][tid] = pb.pawns;
            sb[2][tid] = pb.knights;
            sb[3][tid] = pb.bq;
            sb[4][tid] = pb.rq;
            sb[5][tid] = pb.kings;
            skO[tid] = (uint8_t)ctz(pb.kings & ~pb.mine);
            skS[tid] = (uint8_t)ctz(pb.kings & pb.mine);
        }
        if (!__syncthreads_or(active)) continue;

        // usually the whole unit belongs to one root (parents are ordered by root)
        const bool oneRoot = __syncthreads_and(!inUnit || sroot[tid] == sroot[0]);

        u32 quietReplies = 0;
        for (int g = 0, step = LEAF_NT; g < LEAF_NT;) {
            // ---- generate: quiet moves are counted here, the rest is listed.
            // Should the list overflow, fewer parents take turns.
            u32 replies = 0;
            u32 nMoves = 0;
            if (active && tid >= g && tid < g + step) {
                const Board f{sb[0][tid], sb[1][tid], sb[2][tid], sb[3][tid], sb[4][tid], sb[5][tid]};
                QuietCtx qc;
                quiet_setup(f, qc);
                quiet_flip(qc);
                LeafSink sink{sitems, &sCount, 0u, (u32)tid << 16, 0u};
                gen_moves_quiet<SV>(flip_board(f), qc, sink, nMoves, replies);
                nMoves += sink.n;
            }
            __syncthreads();
            const u32 listed = sCount;
            if (listed > LEAF_ITEMS && step > LEAF_FEW) {
                __syncthreads();
                if (tid == 0) sCount = 0;
                __syncthreads();
                step >>= 1;
                continue;
            }
            quietReplies += replies;
            if (active && tid >= g && tid < g + step && !moves_as_counted(scounted[tid], nMoves))
                atomicOr(P.err, DERR_GEN_MISMATCH);
            nMoves = __reduce_add_sync(0xffffffffu, nMoves);
            if (lane == 0) atomicAdd(&smoves, nMoves);
            if (listed > LEAF_ITEMS && tid == 0) atomicOr(P.err, DERR_BAD_ITEM);

            // ---- every thread takes listed items: make, count, add to the parent's
            for (int j = tid; j < (int)min(listed, LEAF_ITEMS); j += LEAF_NT) {
                const u32 it = sitems[j];
                const int pl = (int)(it >> 16);
                const Board b{sb[0][pl], sb[1][pl], sb[2][pl], sb[3][pl], sb[4][pl], sb[5][pl]};
                Board ch;
                atomicAdd(&sreplies[pl], tile_make_count<SV>(b, it, skO[pl], skS[pl], ch));
            }
            g += step;
            if (g < LEAF_NT) {
                __syncthreads();
                if (tid == 0) sCount = 0;
                __syncthreads();
            }
        }

        __syncthreads();
        // ---- weight x replies into the roots' sums
        unsigned long long s = inUnit ? (quietReplies + sreplies[tid]) * sweight[tid] : 0ull;
        const unsigned done = __ballot_sync(0xffffffffu, active);
        if (tid == 0 && P.moves) atomicAdd(P.moves, (unsigned long long)smoves);
        if (oneRoot) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0 && s) atomicAdd(&ssum, s);
            if (TRACK && lane == 0 && done) atomicAdd(&sdone, __popc(done));
            __syncthreads();
            if (tid == 0) {
                if (ssum) atomicAdd(&P.rootCounts[sroot[0]], ssum);
                if (TRACK && sdone) atomicAdd(&P.pending[sroot[0]], (unsigned long long)(-(long long)sdone));
            }
        } else {
            // segmented sums over the warp's runs of equal roots
            const u32 root = inUnit ? sroot[tid] : 0xFFFFFFFFu;
            const unsigned run = __match_any_sync(0xffffffffu, root);
            if (P.proot) {
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long y = __shfl_down_sync(0xffffffffu, s, o);
                    if (lane + o < 32 && ((run >> (lane + o)) & 1)) s += y;
                }
            }
            const bool first = !P.proot || lane == __ffs(run) - 1;
            if (inUnit && first && s) atomicAdd(&P.rootCounts[root], s);
            if (TRACK && inUnit && first && (run & done))
                atomicAdd(&P.pending[root], (unsigned long long)(-(long long)__popc(run & done)));
        }
        __syncthreads();
    }
}

// ============================================================ small trees
// Positions of small depth in one launch, with no level buffers: one position
// of depth 2..5, or a batch of up to SMALL_BATCH positions of depth 0..4.
// The level pipeline spends such trees' time on per-ply latency: a scan and a
// tile launch per ply, each a few microseconds on a handful of busy SMs.  Here
// each position has some CTAs (its slices), and each CTA counts whole subtrees
// rooted `depth - 3` plies below the position in shared memory.  Two steps
// alternate, each with a whole CTA's threads on it:
//   * small_process: one thread per move makes the child and counts the
//     child's moves; the count also yields what the child's moves depend on
//     (MoveCtx);
//   * small_list: the moves of some positions into the CTA's item list, each
//     warp taking one part of the generation (gen_part) of 32 positions, so
//     that no thread generates a whole position and no warp diverges by part.
// Bound by latency, not throughput: a handful of dependent steps per ply.
// The steps replace one thread generating a position's moves from scratch
// while the CTA waits (5-6.5 us each, three in a row at depth 5).  Both steps
// are single out-of-line functions, since every further inlined copy is
// fetched cold on every launch.
// Tried: a thread per (position, piece) and the n-th move found by a search in
// the scanned move counts instead of a list.  As fast for one position, but
// 32 positions took 8-20 us against 4: every thread paid for all eight slider
// directions.
// Measured per call, before and after: opening at depth 5 84 -> 62 us, depth 3
// 52 -> 26 us (the kernel 12 us of it), 61 positions of depths 1-4 217 -> 88 us
// (as a replayed graph of the level pipeline before; on new depths 500 -> 94).
// Every CTA finds its subtree roots for itself, so no CTA waits for another;
// the last CTA to finish hands the sums over and clears them for the next
// launch.  The make-move and count are the level pipeline's own functions.
constexpr int SMALL_NT = 128;  // threads per CTA: small CTAs put more subtrees in flight
constexpr int SMALL_MINB = 4;
constexpr int SMALL_MAX_DEPTH = 5;
// Largest batch: at depth 4 alone one launch and a replayed graph of levels
// meet here (64 positions 216 us in one launch, 220 as levels; 32 positions 117
// and 211).  Shallower and mixed batches still gain at this size (64 of depths
// 1-4 90 and 221 us, and 451 in the first call with a new mix).  A depth-5
// position fills the device by itself (smallGrid CTAs), so batches of them are
// left to the levels.
constexpr int SMALL_BATCH = 64;
constexpr int SMALL_BATCH_DEPTH = 4;
constexpr u32 SMALL_LIST_CAP = 4096;  // most subtree roots of a depth-5 position (larger trees: level pipeline)
constexpr u32 SMALL_PART = 256;
constexpr u32 SMALL_ITEMS = 2048 + MAX_LEGAL_MOVES;  // the item list: whole positions up to 2048 moves and one more
constexpr int SMALL_SLICES = 48;      // subtree roots of a depth-4 position handled at the same time (few positions have more moves)
constexpr u32 SMALL_OVERFLOW = 1u << 8;  // not counted: too many subtree roots, moves or pieces

// The launch's parameters, positions included, so that host positions need no copy.
template <int N>
struct SmallParams {
    const u64 *dPos;  // positions on the device; null: pos below
    u64 *dOut;        // device results (may be null)
    struct SmallResult *host;  // mapped host memory
    struct SmallState *state;
    u32 n, listCap;
    uint16_t unit0[N + 1];  // first CTA of each position
    uint8_t depth[N];
    uint8_t split[N];  // CTAs that share one subtree
    u64 pos[6 * N];
};
struct SmallResult {
    u64 count[SMALL_BATCH];
    u32 flags;  // 0, SMALL_OVERFLOW or DERR_BAD_POSITION
};
struct SmallState {  // all zero between launches
    unsigned long long sum[SMALL_BATCH];
    u32 done;   // CTAs finished
    u32 flags;  // raised by any CTA
};

// Places of the positions a CTA holds.
constexpr int SMALL_CHILD0 = 0;                     // the current subtree root's children
constexpr int SMALL_SUB = MAX_LEGAL_MOVES;          // the current subtree root
constexpr int SMALL_ROOT = SMALL_SUB + 1;           // the CTA's position
constexpr int SMALL_FIRST0 = SMALL_ROOT + 1;        // its children
constexpr int SMALL_PLACES = SMALL_FIRST0 + MAX_LEGAL_MOVES;
struct SmallShared {
    Board b[SMALL_PLACES];
    MoveCtx c[SMALL_PLACES];
    u32 items[SMALL_ITEMS];  // (place << 16) | move
    u32 nItems;
    u32 nPart[GEN_PARTS];  // one position's list: its parts' moves, each part at its own SMALL_PART items
    u32 first[MAX_LEGAL_MOVES];  // first item below each child of the position, or of the subtree root
    uint8_t cnt[SMALL_PLACES];  // move counts (at most MAX_LEGAL_MOVES, else flagged)
    u32 sw[SMALL_NT / 32];
    u32 flags;
    bool last;
};
constexpr size_t SMALL_DYN_SMEM = sizeof(SmallShared);

// Exclusive block sum of one u32 per thread; `total` gets the block's sum.
template <int NT>
__device__ __forceinline__ u32 block_excl_sum(u32 v, u32 *sw, u32 &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    u32 inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) sw[w] = inc;
    __syncthreads();
    u32 off = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; i++) {
        off += (i < w) ? sw[i] : 0u;
        tot += sw[i];
    }
    __syncthreads();
    total = tot;
    return off + inc - v;
}

// Exclusive sums of the move counts at places p0 .. p0 + n - 1 into S.first
// (n <= MAX_LEGAL_MOVES); returns the total.
__device__ __forceinline__ u32 small_first(SmallShared &S, int p0, int n)
{
    static_assert(2 * SMALL_NT >= MAX_LEGAL_MOVES, "two positions per thread");
    const int t = 2 * threadIdx.x;
    const u32 a = t < n ? S.cnt[p0 + t] : 0u, b = t + 1 < n ? S.cnt[p0 + t + 1] : 0u;
    u32 total;
    const u32 x = block_excl_sum<SMALL_NT>(a + b, S.sw, total);
    if (t < n) S.first[t] = x;
    if (t + 1 < n) S.first[t + 1] = x + a;
    __syncthreads();
    return total;
}

// Lists run by run at the list's cursor, or (one position) part by part.
template <bool SHARED>
struct SmallSink {
    SmallShared &S;
    u32 at, tag;
    __device__ __forceinline__ void room(int n)
    {
        if (SHARED && n) at = atomicAdd(&S.nItems, (u32)n);
    }
    __device__ __forceinline__ void operator()(u32 m)
    {
        if (at < SMALL_ITEMS) S.items[at] = tag | m;
        at++;
    }
};

// Lists the moves of the positions at places p0 .. p0 + w - 1.  One
// position's list has the same order in every CTA (slices pick their moves by
// number); a list of several positions is in no particular order.
__device__ __noinline__ void small_list(SmallShared &S, int p0, int w)
{
    static_assert(SMALL_NT == 32 * GEN_PARTS, "a warp per part");
    const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) S.nItems = 0;
    __syncthreads();
    if (w == 1) {
        if (lane == 0) {
            SmallSink<false> sink{S, (u32)part * SMALL_PART, (u32)p0 << 16};
            gen_part(S.b[p0], S.c[p0], part, sink);
            S.nPart[part] = sink.at - (u32)part * SMALL_PART;
        }
        __syncthreads();
        return;
    }
    for (int p = p0 + lane; p < p0 + w; p += 32) {
        if (!S.cnt[p]) continue;
        SmallSink<true> sink{S, 0u, (u32)p << 16};
        gen_part(S.b[p], S.c[p], part, sink);
    }
    __syncthreads();
    if (threadIdx.x < GEN_PARTS) S.nPart[threadIdx.x] = threadIdx.x ? 0u : min(S.nItems, SMALL_ITEMS);
    __syncthreads();
}

// Makes the listed moves j0, j0 + step, ... below j1 (one per thread) and
// counts the children's moves; keeps the children at places keep, keep + 1,
// ... when keep >= 0 (at most MAX_LEGAL_MOVES of them).  Returns this
// thread's sum of counts.  A kept position with more moves than any game's
// flags the tree.
__device__ __noinline__ u32 small_process(SmallShared &S, u32 j0, u32 j1, u32 step, int keep)
{
    u32 sum = 0;
    const u32 c0 = S.nPart[0], c1 = S.nPart[1], c2 = S.nPart[2], c3 = S.nPart[3];
    j1 = min(j1, c0 + c1 + c2 + c3);
    for (u32 i = threadIdx.x; j0 + i * step < j1; i += SMALL_NT) {
        u32 j = j0 + i * step;
        if (j >= c0) {  // (a list of several positions is all in the first part)
            j -= c0;
            u32 at = SMALL_PART;
            if (j >= c1) {
                j -= c1;
                at += SMALL_PART;
                if (j >= c2) {
                    j -= c2;
                    at += SMALL_PART;
                }
            }
            j += at;
        }
        const u32 it = S.items[j];
        const Board b = make_child<false>(S.b[it >> 16], it & 0xFFFFu);
        MoveCtx c;
        const u32 n = count_moves_fused<SV_KOGGE>(b, -1, -1, 0, 0, &c);
        sum += n;
        if (keep >= 0) {
            S.b[keep + i] = b;
            S.c[keep + i] = c;
            S.cnt[keep + i] = (uint8_t)n;
            if (n > (u32)MAX_LEGAL_MOVES) atomicOr(&S.flags, SMALL_OVERFLOW);
        }
    }
    return sum;
}

template <int N>
__global__ void __launch_bounds__(SMALL_NT, SMALL_MINB) k_small_trees(const __grid_constant__ SmallParams<N> P)
{
    extern __shared__ __align__(16) unsigned char smallShared[];
    SmallShared &S = *reinterpret_cast<SmallShared *>(smallShared);
    const int tid = threadIdx.x, lane = tid & 31;

    // this CTA's position, and its slice of it
    int lo = 0, hi = N == 1 ? 1 : (int)P.n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (P.unit0[mid] <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    const int at = lo;
    const int depth = P.depth[at];
    const u32 split = P.split[at], unit = blockIdx.x - P.unit0[at];
    const u32 nSlices = (u32)(P.unit0[at + 1] - P.unit0[at]) / split;
    const u32 slice = unit / split, part = unit % split;

    if (tid == 0) S.flags = 0;
    __syncthreads();
    // the position's count and its check at the same time (no count without
    // both kings: the move tables are indexed by their squares)
    if (tid == 0 || tid == 32) {
        u64 p[6];
#pragma unroll
        for (int k = 0; k < 6; k++) p[k] = P.dPos ? P.dPos[6 * at + k] : P.pos[6 * at + k];
        if (tid == 32) {
            if (validate_pos48(p) != 0) atomicOr(&S.flags, DERR_BAD_POSITION);
        } else if (one_king_each(p)) {
            const Board b = from_pos48(p);
            MoveCtx c;
            const u32 n = count_moves_fused<SV_KOGGE>(b, -1, -1, 0, 0, &c);
            S.b[SMALL_ROOT] = b;
            S.c[SMALL_ROOT] = c;
            S.cnt[SMALL_ROOT] = (uint8_t)n;
            if (n > (u32)MAX_LEGAL_MOVES && depth >= 2) atomicOr(&S.flags, SMALL_OVERFLOW);
            S.nItems = n;
        }
    }
    __syncthreads();
    unsigned long long acc = 0;
    const u32 n1 = S.nItems;
    if (!S.flags && tid == 0 && depth < 2) acc = depth == 0 ? 1u : n1;
    if (depth >= 2 && !S.flags && n1) {
        // the subtrees: this CTA's share of them
        u32 s = slice, nSub = 1;
        __syncthreads();  // every thread has read S.nItems and S.flags
        small_list(S, SMALL_ROOT, 1);
        if (depth == 4) {  // roots: the position's children
            nSub = n1;
            small_process(S, slice, n1, nSlices, SMALL_FIRST0);
            __syncthreads();
        } else if (depth == 5) {  // roots: its grandchildren
            small_process(S, 0, n1, 1, SMALL_FIRST0);
            __syncthreads();
            nSub = small_first(S, SMALL_FIRST0, (int)n1);
            if (tid == 0 && nSub > P.listCap) S.flags |= SMALL_OVERFLOW;
            __syncthreads();
        }
        // (flags are only read between two barriers with no position stored
        // in between, so that every thread sees the same)
        for (; s < nSub; s += nSlices) {
            const bool stop = S.flags != 0;
            __syncthreads();
            if (stop) break;
            int sub = SMALL_ROOT;
            if (depth == 4) sub = SMALL_FIRST0 + (int)((s - slice) / nSlices);
            if (depth == 5) {
                // the s-th grandchild: the child it is below, and that child's moves
                if (s != slice) small_first(S, SMALL_FIRST0, (int)n1);  // (the last subtree used the array)
                int c = 0, e = (int)n1;
                while (e - c > 1) {
                    const int mid = (c + e) >> 1;
                    if (S.first[mid] <= s) c = mid;
                    else e = mid;
                }
                const u32 k = s - S.first[c];
                small_list(S, SMALL_FIRST0 + c, 1);
                small_process(S, k, k + 1, 1, SMALL_SUB);
                __syncthreads();
                if (S.flags) break;  // (the next position is stored behind small_list's barriers)
                sub = SMALL_SUB;
            }
            const u32 T = sub == SMALL_ROOT ? n1 : S.cnt[sub];
            if (sub != SMALL_ROOT) small_list(S, sub, 1);
            if (depth == 2) {
                acc += small_process(S, 0, T, 1, -1);
                continue;
            }
            const u32 lo3 = part * T / split, hi3 = (part + 1) * T / split;
            small_process(S, lo3, hi3, 1, SMALL_CHILD0);
            __syncthreads();
            // the children's moves, as many whole children at a time as the list holds
            const int nC = (int)(hi3 - lo3);
            const u32 all = small_first(S, SMALL_CHILD0, nC);
            for (int w0 = 0; w0 < nC;) {
                int w = nC - w0;
                if (all - S.first[w0] > SMALL_ITEMS) {
                    w = 1;
                    while (S.first[w0 + w] + S.cnt[SMALL_CHILD0 + w0 + w] - S.first[w0] <= SMALL_ITEMS) w++;
                }
                small_list(S, SMALL_CHILD0 + w0, w);
                acc += small_process(S, 0, ~0u, 1, -1);
                __syncthreads();
                w0 += w;
            }
        }
    }

    // the CTA's sum into its position's; the last CTA hands everything over
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0 && acc) atomicAdd(&P.state->sum[at], acc);
    __syncthreads();
    if (tid == 0) {
        if (S.flags) atomicOr(&P.state->flags, S.flags);
        __threadfence();
        S.last = atomicAdd(&P.state->done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!S.last) return;
    __threadfence();
    const u32 flags = __ldcg(&P.state->flags);
    for (int i = tid; i < (int)P.n; i += SMALL_NT) {
        const u64 c = __ldcg(&P.state->sum[i]);
        P.host->count[i] = c;
        if (P.dOut && !flags) P.dOut[i] = c;
        P.state->sum[i] = 0;
    }
    __syncthreads();
    if (tid == 0) {
        P.host->flags = flags;
        P.state->flags = 0;
        P.state->done = 0;
    }
}

// The first two plies of a single-root graph in one launch: a CTA per root
// move writes that move's children to level 2.  As two plies of the level
// pipeline (root, scan, tile launch, scan, tile launch) they took 75 us, most
// of it the latency of launches with a handful of busy warps; one position at
// depth 6 takes 571 -> 537 us with this.  The graph's plan
// has level 2's buffers; a root or child with more moves than any game's
// raises the overflow flag (the host-driven path then runs).  Every CTA makes
// all of the root's children, so all see the same flags before they write:
// level 2 has nodes only when every CTA writes its share of them.
constexpr int FRONT_LEVEL = 2;
constexpr u64 FRONT_NODES = (u64)MAX_LEGAL_MOVES * MAX_LEGAL_MOVES;
__global__ void __launch_bounds__(SMALL_NT, SMALL_MINB) k_dd_front(DevPlan *plan, const u64 *__restrict__ pos48, u32 *err)
{
    extern __shared__ __align__(16) unsigned char smallShared[];
    SmallShared &S = *reinterpret_cast<SmallShared *>(smallShared);
    const int tid = threadIdx.x;
    if (tid == 0) S.flags = 0;
    __syncthreads();
    if (tid == 0 || tid == 32) {
        u64 p[6];
#pragma unroll
        for (int k = 0; k < 6; k++) p[k] = pos48[k];
        if (tid == 32) {
            if (validate_pos48(p) != 0) atomicOr(&S.flags, DERR_BAD_POSITION);
        } else if (one_king_each(p)) {
            const Board b = from_pos48(p);
            MoveCtx c;
            const u32 n = count_moves_fused<SV_KOGGE>(b, -1, -1, 0, 0, &c);
            S.b[SMALL_ROOT] = b;
            S.c[SMALL_ROOT] = c;
            S.cnt[SMALL_ROOT] = (uint8_t)n;
            if (n > (u32)MAX_LEGAL_MOVES) atomicOr(&S.flags, SMALL_OVERFLOW);
        }
    }
    __syncthreads();
    if (!S.flags) {  // (uniform: no position is stored before the barriers of small_list)
        const int n1 = S.cnt[SMALL_ROOT];
        if ((int)blockIdx.x >= n1) return;
        small_list(S, SMALL_ROOT, 1);
        small_process(S, 0, (u32)n1, 1, SMALL_FIRST0);
        __syncthreads();
        const u32 total = small_first(S, SMALL_FIRST0, n1);
        LevelDesc &L = plan->lv[FRONT_LEVEL];
        if (!S.flags) {
            const int c = (int)blockIdx.x;
            if (c == 0 && tid == 0) L.n = L.nChild = total;
            const u32 at = S.first[c], m = S.cnt[SMALL_FIRST0 + c];
            small_list(S, SMALL_FIRST0 + c, 1);
            small_process(S, 0, m, 1, SMALL_CHILD0);
            __syncthreads();
            for (u32 i = tid; i < m; i += SMALL_NT) {
                level_put(L.planes, L.stride, at + i, S.b[SMALL_CHILD0 + i]);
                L.cnt[at + i] = S.cnt[SMALL_CHILD0 + i];
                L.root[at + i] = 0;
                if (L.weight) L.weight[at + i] = 1ull;
            }
        }
    }
    if (tid == 0 && S.flags) {
        if (S.flags & DERR_BAD_POSITION) atomicOr(err, DERR_BAD_POSITION);
        if (S.flags & SMALL_OVERFLOW) plan->overflow = 1;
    }
}

// ====================================================== transposition table
// Lockless table of 16-byte entries {verify ^ value, value} at the slot the
// slot key picks: a torn or foreign entry fails the XOR check (the
// reference's scheme, perft_bb.h:759-764, whose 128-bit hash is here two
// independent 64-bit hashes).  Both are Zobrist hashes of the side-relative
// board (two sets of 781 seeded keys: 12 piece kinds x 64 squares, 4 castling
// rights, 8 en-passant files, one spare) XOR a per-remaining-depth key, so
// one table holds every depth ("per-depth slots").  Perft is invariant under the
// colour mirror, so a position and its mirror may share an entry.
constexpr int ZOB_KEYS = 781;
constexpr int ZOB_DEPTH_KEYS = 32;
// Two independent key sets (x, y): the x hash picks the table slot, the y
// hash verifies.  A verification key that shares
// no bits with the index keeps false hits at 2^-64 per probe; with one 64-bit
// hash doing both, only the bits above the index are checked, and searches
// with ~1e12 probes (perft 12 of the initial position) did see false hits.
__device__ ulonglong2 d_zobrist[ZOB_KEYS + ZOB_DEPTH_KEYS];

struct TTStats {
    unsigned long long probes, hits, aliases, stores;
};

__device__ __forceinline__ void zx(ulonglong2 &h, const ulonglong2 &z)
{
    h.x ^= z.x;
    h.y ^= z.y;
}

// Both Zobrist hashes of a side-relative board (one 16-byte key read from
// shared memory per piece).
__device__ __forceinline__ ulonglong2 zobrist_rel(const Board &b, const ulonglong2 *keys)
{
    const u64 pawns = b.pawns & RANKS2TO7;
    const u64 occ = pawns | b.knights | b.bq | b.rq | b.kings;
    const u64 theirs = occ ^ b.mine;
    const u64 sets[6] = {pawns, b.knights, b.bq & ~b.rq, b.rq & ~b.bq, b.bq & b.rq, b.kings};
    ulonglong2 h = make_ulonglong2(0, 0);
#pragma unroll
    for (int pc = 0; pc < 6; pc++) {
        for_each_bit(sets[pc] & b.mine, [&](int sq) { zx(h, keys[pc * 64 + sq]); });
        for_each_bit(sets[pc] & theirs, [&](int sq) { zx(h, keys[(6 + pc) * 64 + sq]); });
    }
    const u32 st = (u32)(b.pawns & 0xFF);
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (st & (1u << k)) zx(h, keys[768 + k]);
    if (st >> 4) zx(h, keys[772 + (st >> 4) - 1]);
    return h;
}

// Block-aggregated increment of a statistics counter: warp ballots summed
// in shared memory, then one global atomic per block.  Per-warp atomics on
// the same few counters serialised in L2 and cost a large part of the table
// kernels' time.  Every thread of the block must call it.
__device__ __forceinline__ void count_stat(unsigned long long *ctr, bool hit)
{
    __shared__ unsigned sCount;
    if (threadIdx.x == 0) sCount = 0;
    __syncthreads();
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(&sCount, (unsigned)__popc(m));
    __syncthreads();
    if (threadIdx.x == 0 && sCount) atomicAdd(ctr, (unsigned long long)sCount);
}

// Hashes and probes the nodes that stand for themselves after the level was
// merged (owners, and nodes the set had no slot for).  Hits take the table's
// value and lose their children; their alias is ALIAS_HIT.
// The keys are read from shared memory: a warp's 32 scattered 16-byte reads
// per piece took one L1 pass each from global memory and bound the kernel.
// Persistent blocks, so that the 13 KB of keys are loaded once per block.
// Merging first (exact, by the boards) halves the nodes hashed.  Two table
// positions at depth 8: 261 -> 255 ms.
__global__ void __launch_bounds__(256) k_tt_probe(const u64 *__restrict__ planes, u64 stride, u64 n, int remaining,
                                                  u64 keyMask, u32 *__restrict__ cnt, u64 *__restrict__ hash,
                                                  u64 *__restrict__ hash2, unsigned long long *__restrict__ acc,
                                                  u32 *__restrict__ alias, const ulonglong2 *tt, u64 ttMask,
                                                  TTStats *ts)
{
    __shared__ ulonglong2 keys[ZOB_KEYS];
    for (int k = threadIdx.x; k < ZOB_KEYS; k += 256) keys[k] = d_zobrist[k];
    const ulonglong2 depthKey = d_zobrist[ZOB_KEYS + remaining];
    __syncthreads();
    u32 probes = 0, hits = 0;
    for (u64 i = (u64)blockIdx.x * 256 + threadIdx.x; i < n; i += (u64)gridDim.x * 256) {
        const u32 a = alias[i];
        if (a != (u32)i && a != ALIAS_NOSLOT) continue;
        ulonglong2 z = zobrist_rel(level_get(planes, stride, i), keys);
        zx(z, depthKey);
        const u64 h = z.x & keyMask;  // slot key (table index)
        hash[i] = h;
        hash2[i] = z.y;               // verification key
        const ulonglong2 e = tt[h & ttMask];
        probes++;
        if ((e.x ^ e.y) == z.y) {
            hits++;
            acc[i] = e.y;
            cnt[i] = 0;
            alias[i] = ALIAS_HIT;
        }
    }
    block_add_stat(&ts->probes, probes);
    block_add_stat(&ts->hits, hits);
}

// After a level's subtrees are summed into acc: copy owners' values into
// their duplicates, store owners in the table, and add every value into the
// parent level (nodes are ordered by parent: segmented warp sums, then one
// atomic per parent run).  At level 0 the values go to the roots' results.
__global__ void __launch_bounds__(256) k_tt_finish(u64 n, bool store, const u64 *__restrict__ hash,
                                                   const u64 *__restrict__ hash2,
                                                   unsigned long long *__restrict__ acc, const u32 *__restrict__ alias,
                                                   const u32 *__restrict__ parent, unsigned long long *parentAcc,
                                                   ulonglong2 *tt, u64 ttMask, TTStats *ts)
{
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    unsigned long long v = 0;
    u32 key = 0xFFFFFFFFu;
    bool stored = false;
    if (i < n) {
        const u32 a = alias[i];
        v = acc[i];
        if (a != ALIAS_HIT && a != ALIAS_NOSLOT && a != (u32)i) {
            v = acc[a];  // the owner is final: its subtree finished before this kernel
        } else if (a != ALIAS_HIT && store) {
            tt[hash[i] & ttMask] = make_ulonglong2(hash2[i] ^ v, v);
            stored = true;
        }
        key = parent[i];
    }
    count_stat(&ts->stores, stored);
    if (!parentAcc) return;  // level 0: k_tt_roots writes the results
    // segmented inclusive sum over runs of equal parent within the warp
    unsigned long long sum = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, sum, o);
        const u32 ky = __shfl_up_sync(0xffffffffu, key, o);
        if (lane >= o && ky == key) sum += y;
    }
    const u32 knext = __shfl_down_sync(0xffffffffu, key, 1);
    const bool last = (lane == 31) || knext != key;
    if (i < n && last && key != 0xFFFFFFFFu) atomicAdd(&parentAcc[key], sum);
}

// Level 0 of a TT run: each root's value (own, owner's, or table's) is its result.
__global__ void k_tt_roots(u64 n, const unsigned long long *__restrict__ acc, const u32 *__restrict__ alias,
                           const u32 *__restrict__ root, unsigned long long *__restrict__ out)
{
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const u32 a = alias[i];
    out[root[i]] = (a != ALIAS_HIT && a != ALIAS_NOSLOT && a != (u32)i) ? acc[a] : acc[i];
}

// ================================================================ host side
struct DeviceLevel {
    u64 *planes;
    u64 stride;
    u32 *cnt;
    u32 *root;  // root id (no TT) or parent index in the previous level (TT)
    u64 n;
    unsigned long long *weight = nullptr;  // merged runs: paths that reach each node
    // transposition-table runs only
    u64 *hash = nullptr;   // slot key
    u64 *hash2 = nullptr;  // verification key
    unsigned long long *acc = nullptr;  // perft of each node's subtree
    u32 *alias = nullptr;               // owner index, ALIAS_HIT or ALIAS_NOSLOT
};

// Bytes of one TT level node: the plain node plus two hashes, subtree sum, alias,
// and the transient merge set (it is released before the scan, so this
// over-counts).
constexpr u64 NODE_BYTES_TT = NODE_BYTES + 8 + 8 + 8 + 4 + 30;
// Without a table (related roots): the plain node plus sum, alias and set.
constexpr u64 NODE_BYTES_LINKED = NODE_BYTES + 8 + 4 + 8 * MERGE_SLOTS;

class Engine {
public:
    int init(const perft_config &cfg);
    void shutdown();
    // trySmall: small trees try the one-launch kernel first (false when the
    // caller already tried it)
    // related: the roots are a few moves apart from each other (related_roots)
    int run_batch(const u64 *dPos, const uint8_t *depths, u32 n, u64 *dOut, bool trySmall = true,
                  bool related = false);
    // Host buffers: staged through engine-owned device buffers that persist
    // across calls (no per-call allocation; stable addresses let replayed
    // graphs be reused).
    int run_batch_host(const u64 *pos, const uint8_t *depths, u32 n, u64 *out);
    u64 *ioPos = nullptr, *ioOut = nullptr;
    u32 ioCap = 0;

    perft_stats stats{};
    std::mutex mu;
    bool ready = false;
    std::string lastCudaError;

private:
    int device = 0;
    int nsm = 0;
    cudaStream_t stream = nullptr;
    char *arena = nullptr;
    u64 arenaCap = 0, arenaTop = 0, arenaPeak = 0;
    u32 *dCounter = nullptr;  // tile cursor
    u32 *dErr = nullptr;
    u64 *hPinned = nullptr;   // small read-backs
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int svExpand = SV_KOGGE, svLeaf = SV_KOGGE;
    int gridTile[2][SV_COUNT] = {};
    bool trace = false;  // PERFT_TRACE=1: one stderr line per tile launch

public:
    // Launch configuration per (ply kind, remaining depth of the parent level):
    // slider variant, largest tile (log2 items; interior plies) and resident CTAs
    // per SM.  The count-only ply always has remaining depth 2; interior plies have 3..20
    // and use the entry of the nearest calibrated depth.
    struct TuneCfg {
        int sv = SV_KOGGE;
        int cap = TILE_CAP_LOG2;
        int ctas = 0;  // 0: as many as fit
        double ms = 0;  // calibration time of this key (median of the timed runs)
    };
    static constexpr int TUNE_MAX_R = 20;
    TuneCfg tuneTab[2][TUNE_MAX_R + 1];
    int tunedMaxR = 3;

private:
    bool tuning = false;  // autotune running: launch times accumulate per key
    double tuneAccMs[2][TUNE_MAX_R + 1] = {};
    const TuneCfg &cfg_for(int mode, int r) const
    {
        if (mode == MODE_LEAF) return tuneTab[MODE_LEAF][2];
        return tuneTab[MODE_EXPAND][std::max(3, std::min(r, tunedMaxR))];
    }
    int grid_for(int mode, const TuneCfg &c) const
    {
        const int occ = gridTile[mode][c.sv];
        return c.ctas > 0 ? std::min(occ, c.ctas * nsm) : occ;
    }
    int max_ctas(int mode, int sv) const { return std::max(1, gridTile[mode][sv] / std::max(1, nsm)); }
    void fill_tune(int svL, int svE)
    {
        for (int r = 0; r <= TUNE_MAX_R; r++) {
            tuneTab[MODE_LEAF][r] = TuneCfg{svL, TILE_CAP_LOG2, 0, 0};
            tuneTab[MODE_EXPAND][r] = TuneCfg{svE, TILE_CAP_LOG2, 0, 0};
        }
        tunedMaxR = 3;
    }

    // A scanned level: its parents, their items and the tiles of those.
    struct ParentIndex {
        u64 *pscan = nullptr;
        u32 *live = nullptr;  // null: every node is a parent
        u32 *tileFirst = nullptr;
        u64 nParents = 0, total = 0;
        int capLog2 = TILE_CAP_LOG2;
    };
    void *alloc(u64 bytes)
    {
        const u64 a = (arenaTop + 255) & ~255ULL;
        if (a + bytes > arenaCap) return nullptr;
        arenaTop = a + bytes;
        arenaPeak = std::max(arenaPeak, arenaTop);
        return arena + a;
    }
    u64 arena_free() const { return arenaCap > arenaTop ? arenaCap - arenaTop : 0; }
    bool alloc_level(DeviceLevel &L, u64 n, bool weighted = false);
    int scan(const u32 *cnt, u64 n, int remaining, bool compact, ParentIndex &out);
    int launch_tile(int mode, int remaining, const DeviceLevel &parents, const ParentIndex &ix, u64 itemBase,
                    u64 itemEnd, DeviceLevel *children, unsigned long long *rootCounts);
    // Roots that join the search at a given remaining depth: their ids (device
    // array) and count, indexed by depth.  A root of depth d enters the level
    // whose nodes have d plies left, behind that level's children.
    struct Joiners {
        const u64 *dPos = nullptr;
        const u32 *ids[21] = {};
        u32 n[21] = {};
        // merged runs (else null): every root's depth, and its nodes in the level being merged
        const uint8_t *depths = nullptr;
        MergeSeg *segs = nullptr;
        int maxDepth = 0;
    };
    int merge_level(const Joiners &J, const DeviceLevel &C, int remaining);
    int run_levels(const u64 *dPos, const uint8_t *depths, u32 n, unsigned long long *rootCounts, bool merge);
    bool mergeEnabled = true;
    int process_level(const DeviceLevel &L, int remaining, unsigned long long *rootCounts,
                      const Joiners *join = nullptr);
    int init_joiners(const Joiners &J, int depth, DeviceLevel &C, u64 at, unsigned long long *rootCounts);
    int process_level_tt(const DeviceLevel &L, int remaining, unsigned long long *parentAcc,
                         unsigned long long *rootOut);
    bool alloc_level_tt(DeviceLevel &L, u64 n);

public:
    // A long-lived block at the top of the arena (the server's memory);
    // per-call allocations stack above it.
    char *reserve_block(u64 bytes)
    {
        blockMark = arenaTop;
        char *p = (char *)alloc(bytes);
        if (!p) arenaTop = blockMark;
        return p;
    }
    void release_block() { arenaTop = blockMark; }
    u64 free_bytes() const { return arena_free(); }
    int device_id() const { return device; }
    int leaf_sliders() const { return svLeaf; }
    bool merge_enabled() const { return mergeEnabled; }
    u64 blockMark = 0;
    // The transposition table as the server sees it (null table: none configured).
    struct TTView {
        ulonglong2 *table;
        u64 mask, keyMask;
    };
    TTView tt_view() const { return TTView{tt, ttMask, ttKeyMask}; }
    int tt_clear();
    void read_tt_stats()
    {
        TTStats t{};
        if (dTTStats && cudaMemcpy(&t, dTTStats, sizeof t, cudaMemcpyDeviceToHost) == cudaSuccess) {
            stats.tt_probes = t.probes;
            stats.tt_hits = t.hits;
            stats.tt_duplicates = t.aliases;
            stats.tt_stores = t.stores;
        }
        stats.tt_entries = tt ? ttMask + 1 : 0;
    }
    void zero_tt_stats()
    {
        if (dTTStats) cudaMemset(dTTStats, 0, sizeof(TTStats));
    }

private:
    ulonglong2 *tt = nullptr;
    u64 ttMask = 0;
    u64 ttKeyMask = ~0ULL;
    TTStats *dTTStats = nullptr;
    int ttMinDepth = 2;
    int check(cudaError_t e, const char *what);
    int sync_and_check_errors();
    int autotune(bool leaf, bool expand);

    // device-driven runs captured as CUDA graphs (small single-depth batches)
    struct DDGraph {
        int depth = 0;                // deepest root
        std::vector<uint8_t> depths;  // every root's depth (the graph's plan depends on the mix)
        u32 n = 0;
        const u64 *dPos = nullptr;
        u64 *dOut = nullptr;
        u64 top = 0;
        int svL = 0, svE = 0;
        bool overflowed = false;  // the plan did not fit: later calls go host-driven at once
        cudaEvent_t evLeaf0 = nullptr, evLeaf1 = nullptr;  // recorded around the count-only ply
        std::vector<double> predLv;  // predicted nodes per level (empty: no prediction)
        u64 otherLaunches = 0;       // root, scan and join kernels per replay
        u64 expandLaunches = 0;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        DevPlan *hTemplate = nullptr;  // pinned
        u32 *hIds = nullptr;           // pinned
        u64 *hFlags = nullptr;         // pinned: overflow, device error, leaf items
    };
    std::vector<DDGraph> ddCache;
    // one-launch small trees (k_small_trees)
    SmallState *dSmall = nullptr;
    SmallResult *hSmall = nullptr;  // mapped
    int smallGrid = 0;
    bool smallEnabled = true;
    u32 smallListCap = SMALL_LIST_CAP;
    // batches replay one captured launch whose parameters each call sets: 24.5 us
    // for 2 positions of depth 2, 34.4 us for 64 of depth 3, against 31.1 and
    // 36.7 as a plain launch of the same kernel
    SmallParams<SMALL_BATCH> smallBatch;
    cudaGraph_t smallGraph = nullptr;
    cudaGraphExec_t smallExec = nullptr;
    cudaGraphNode_t smallNode = nullptr;
    int run_small(const u64 *dPos, const u64 *pos, const uint8_t *depths, u32 n, u64 *dOut, u64 *hOut, bool &handled);
    template <int N>
    u32 small_params(SmallParams<N> &P, const u64 *dPos, const u64 *pos, const uint8_t *depths, u32 n, u64 *dOut);
    bool ddEnabled = true;
    bool ddForce = false;  // PERFT_DD_FORCE=1: skip the size estimate (tests the overflow fallback)
    double ddMaxBytes = DD_MAX_BYTES_DEFAULT;
    int ddGridScan = 0;
    int run_dd(const u64 *dPos, const uint8_t *depths, u32 n, u64 *dOut, bool &handled);
    int build_dd(DDGraph &G);
    void drop_dd();
};

int Engine::check(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return PERFT_OK;
    char buf[256];
    snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
    lastCudaError = buf;
    return e == cudaErrorMemoryAllocation ? PERFT_ERR_OUT_OF_MEMORY : PERFT_ERR_CUDA;
}

#define ENG_TRY(expr)                                   \
    do {                                                \
        int rc_ = check((expr), #expr);                 \
        if (rc_ != PERFT_OK) return rc_;                \
    } while (0)

constexpr size_t TILE_DYN_SMEM = sizeof(u32) * TILE_CAP;
constexpr size_t LEAF_DYN_SMEM = sizeof(u32) * LEAF_ITEMS;
constexpr size_t tile_dyn_smem(int mode) { return mode == MODE_LEAF ? LEAF_DYN_SMEM : TILE_DYN_SMEM; }

// Most CTAs of the count-only ply that get parents.
constexpr u64 leaf_units(u64 nParents) { return (nParents + LEAF_MIN_UNIT - 1) / LEAF_MIN_UNIT; }
constexpr int tile_threads(int mode) { return mode == MODE_LEAF ? LEAF_NT : TILE_NT; }

template <int MODE, int SV, bool TRACK = false, int DD = DD_NONE>
constexpr void (*tile_kernel())(const TileParams)
{
    if constexpr (MODE == MODE_LEAF) return k_leaf<SV, TRACK, DD>;
    else return k_tile<SV, TRACK, DD>;
}

// Allows the item list's dynamic shared memory on one instantiation and
// returns its resident-CTA grid (SMs x CTAs per SM).
template <int MODE, int SV, bool TRACK = false>
int occupancy_grid(int nsm)
{
    const auto fn = tile_kernel<MODE, SV, TRACK>();
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_dyn_smem(MODE));
    int perSm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, tile_threads(MODE), tile_dyn_smem(MODE)) != cudaSuccess ||
        perSm < 1)
        perSm = 1;
    return perSm * nsm;
}

template <int MODE>
void launch_tile_variant(int sv, int grid, cudaStream_t st, const TileParams &P)
{
    constexpr size_t smem = tile_dyn_smem(MODE);
    switch (sv) {
    case SV_MAGIC: tile_kernel<MODE, SV_MAGIC>()<<<grid, tile_threads(MODE), smem, st>>>(P); break;
    case SV_KOGGE_FMA: tile_kernel<MODE, SV_KOGGE_FMA>()<<<grid, tile_threads(MODE), smem, st>>>(P); break;
    case SV_KOGGE_SPLIT: tile_kernel<MODE, SV_KOGGE_SPLIT>()<<<grid, tile_threads(MODE), smem, st>>>(P); break;
    case SV_HYBRID: tile_kernel<MODE, SV_HYBRID>()<<<grid, tile_threads(MODE), smem, st>>>(P); break;
    default: tile_kernel<MODE, SV_KOGGE>()<<<grid, tile_threads(MODE), smem, st>>>(P); break;
    }
}

// A device-driven tile launch: the two graph variants (Kogge-Stone, split
// shifts) x the two parameter modes (constant bank for large plies, shared
// memory for small ones).
template <int MODE>
void launch_dd_tile(int sv, bool constParams, int grid, cudaStream_t st, const TileParams &P)
{
    constexpr size_t smem = tile_dyn_smem(MODE);
    const bool split = sv == SV_KOGGE_SPLIT;
    if (constParams && split)
        tile_kernel<MODE, SV_KOGGE_SPLIT, false, DD_CONST>()<<<grid, tile_threads(MODE), smem, st>>>(P);
    else if (constParams) tile_kernel<MODE, SV_KOGGE, false, DD_CONST>()<<<grid, tile_threads(MODE), smem, st>>>(P);
    else if (split) tile_kernel<MODE, SV_KOGGE_SPLIT, false, DD_SHARED>()<<<grid, tile_threads(MODE), smem, st>>>(P);
    else tile_kernel<MODE, SV_KOGGE, false, DD_SHARED>()<<<grid, tile_threads(MODE), smem, st>>>(P);
}

const char *slider_name(int sv)
{
    switch (sv) {
    case SV_KOGGE: return "kogge";
    case SV_MAGIC: return "magic";
    case SV_KOGGE_FMA: return "kogge_fma";
    case SV_KOGGE_SPLIT: return "kogge_split";
    case SV_HYBRID: return "hybrid";
    default: return "?";
    }
}

int Engine::init(const perft_config &cfg)
{
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return PERFT_ERR_NO_DEVICE;
    if (cfg.device < 0 || cfg.device >= ndev) return PERFT_ERR_INVALID_ARG;
    device = cfg.device;
    trace = getenv("PERFT_TRACE") && getenv("PERFT_TRACE")[0] == '1';
    ENG_TRY(cudaSetDevice(device));
    cudaDeviceProp prop;
    ENG_TRY(cudaGetDeviceProperties(&prop, device));
    nsm = prop.multiProcessorCount;

    build_tables();
    ENG_TRY(cudaMemcpyToSymbol(d_tables, &h_tables, sizeof(Tables)));
    ENG_TRY(cudaMemcpyToSymbol(d_magic, h_magic, sizeof(h_magic)));
    u32 pow2[32];
    for (int k = 0; k < 32; k++) pow2[k] = 1u << k;
    ENG_TRY(cudaMemcpyToSymbol(c_pow2, pow2, sizeof pow2));

    // A blocking stream: it orders against the legacy default stream, where
    // callers (and torch) usually produce device-resident inputs.
    ENG_TRY(cudaStreamCreate(&stream));
    ENG_TRY(cudaEventCreate(&ev0));
    ENG_TRY(cudaEventCreate(&ev1));
    ENG_TRY(cudaMalloc(&dCounter, 64));
    ENG_TRY(cudaMalloc(&dErr, 64));
    ENG_TRY(cudaMallocHost(&hPinned, 64));

    // Zobrist keys (splitmix64 of the seed) and the transposition table
    {
        ulonglong2 keys[ZOB_KEYS + ZOB_DEPTH_KEYS];
        u64 x = cfg.zobrist_seed;
        auto next = [&x]() {
            x += 0x9E3779B97F4A7C15ULL;
            u64 z = x;
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
            return z ^ (z >> 31);
        };
        for (int k = 0; k < ZOB_KEYS + ZOB_DEPTH_KEYS; k++) keys[k].x = next();
        for (int k = 0; k < ZOB_KEYS + ZOB_DEPTH_KEYS; k++) keys[k].y = next();
        ENG_TRY(cudaMemcpyToSymbol(d_zobrist, keys, sizeof keys));
        // PERFT_TT_INDEX_KEY_BITS=b keeps only the low b bits of the slot key:
        // a test setting that makes different positions share table slots,
        // which the verification key must then tell apart
        ttKeyMask = ~0ULL;
        if (const char *kb = getenv("PERFT_TT_INDEX_KEY_BITS")) {
            const int bits = atoi(kb);
            if (bits >= 1 && bits < 64) ttKeyMask = (1ULL << bits) - 1;
        }
    }
    ENG_TRY(cudaMalloc(&dTTStats, sizeof(TTStats)));
    ENG_TRY(cudaMemset(dTTStats, 0, sizeof(TTStats)));
    if (cfg.tt_log2_entries > 0) {
        if (cfg.tt_log2_entries < 10 || cfg.tt_log2_entries > 34) return PERFT_ERR_INVALID_ARG;
        const u64 entries = 1ULL << cfg.tt_log2_entries;
        ENG_TRY(cudaMalloc(&tt, entries * sizeof(ulonglong2)));
        ENG_TRY(cudaMemset(tt, 0, entries * sizeof(ulonglong2)));
        ttMask = entries - 1;
    }

    size_t freeB = 0, totalB = 0;
    ENG_TRY(cudaMemGetInfo(&freeB, &totalB));
    u64 want = cfg.arena_bytes ? cfg.arena_bytes : (u64)(freeB * 0.85);
    if (want > freeB) return PERFT_ERR_OUT_OF_MEMORY;
    ENG_TRY(cudaMalloc(&arena, want));
    arenaCap = want;

    gridTile[MODE_EXPAND][SV_KOGGE] = occupancy_grid<MODE_EXPAND, SV_KOGGE>(nsm);
    gridTile[MODE_EXPAND][SV_MAGIC] = occupancy_grid<MODE_EXPAND, SV_MAGIC>(nsm);
    gridTile[MODE_EXPAND][SV_KOGGE_FMA] = occupancy_grid<MODE_EXPAND, SV_KOGGE_FMA>(nsm);
    gridTile[MODE_EXPAND][SV_KOGGE_SPLIT] = occupancy_grid<MODE_EXPAND, SV_KOGGE_SPLIT>(nsm);
    gridTile[MODE_LEAF][SV_KOGGE] = occupancy_grid<MODE_LEAF, SV_KOGGE>(nsm);
    gridTile[MODE_LEAF][SV_MAGIC] = occupancy_grid<MODE_LEAF, SV_MAGIC>(nsm);
    gridTile[MODE_LEAF][SV_KOGGE_FMA] = occupancy_grid<MODE_LEAF, SV_KOGGE_FMA>(nsm);
    gridTile[MODE_LEAF][SV_KOGGE_SPLIT] = occupancy_grid<MODE_LEAF, SV_KOGGE_SPLIT>(nsm);
    gridTile[MODE_EXPAND][SV_HYBRID] = occupancy_grid<MODE_EXPAND, SV_HYBRID>(nsm);
    gridTile[MODE_LEAF][SV_HYBRID] = occupancy_grid<MODE_LEAF, SV_HYBRID>(nsm);

    for (auto fn : {(const void *)k_leaf<SV_KOGGE, false, DD_CONST>, (const void *)k_leaf<SV_KOGGE_SPLIT, false, DD_CONST>,
                    (const void *)k_leaf<SV_KOGGE, false, DD_SHARED>,
                    (const void *)k_leaf<SV_KOGGE_SPLIT, false, DD_SHARED>})
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LEAF_DYN_SMEM);
    for (auto fn : {(const void *)k_tile<SV_KOGGE, false, DD_CONST>, (const void *)k_tile<SV_KOGGE_SPLIT, false, DD_CONST>,
                    (const void *)k_tile<SV_KOGGE, false, DD_SHARED>,
                    (const void *)k_tile<SV_KOGGE_SPLIT, false, DD_SHARED>})
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_DYN_SMEM);
    ddGridScan = 4 * nsm;
    {
        ENG_TRY(cudaMalloc(&dSmall, sizeof(SmallState)));
        ENG_TRY(cudaMemset(dSmall, 0, sizeof(SmallState)));
        ENG_TRY(cudaHostAlloc(&hSmall, sizeof(SmallResult), cudaHostAllocMapped));
        ENG_TRY(cudaFuncSetAttribute(k_small_trees<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)SMALL_DYN_SMEM));
        ENG_TRY(cudaFuncSetAttribute(k_dd_front, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMALL_DYN_SMEM));
        ENG_TRY(cudaFuncSetAttribute(k_small_trees<SMALL_BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)SMALL_DYN_SMEM));
        int perSm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_small_trees<1>, SMALL_NT, SMALL_DYN_SMEM) !=
                cudaSuccess ||
            perSm < 1)
            perSm = 1;
        smallGrid = perSm * nsm;
        ENG_TRY(cudaGraphCreate(&smallGraph, 0));
        cudaKernelNodeParams kp = {};
        void *args[] = {&smallBatch};
        memset(&smallBatch, 0, sizeof smallBatch);
        kp.func = (void *)k_small_trees<SMALL_BATCH>;
        kp.gridDim = dim3(1);
        kp.blockDim = dim3(SMALL_NT);
        kp.sharedMemBytes = (unsigned)SMALL_DYN_SMEM;
        kp.kernelParams = args;
        ENG_TRY(cudaGraphAddKernelNode(&smallNode, smallGraph, nullptr, 0, &kp));
        ENG_TRY(cudaGraphInstantiate(&smallExec, smallGraph, 0));
        smallEnabled = !(getenv("PERFT_SMALL_TREE") && getenv("PERFT_SMALL_TREE")[0] == '0');
        // PERFT_SMALL_LIST_CAP=k lists at most k depth-5 subtree roots per CTA:
        // a test setting that sends ordinary positions down the fallback
        smallListCap = SMALL_LIST_CAP;
        if (const char *c = getenv("PERFT_SMALL_LIST_CAP")) {
            const long v = atol(c);
            if (v >= 1 && v <= (long)SMALL_LIST_CAP) smallListCap = (u32)v;
        }
    }
    mergeEnabled = !(getenv("PERFT_NO_MERGE") && getenv("PERFT_NO_MERGE")[0] == '1');
    ddEnabled = !(getenv("PERFT_NO_GRAPHS") && getenv("PERFT_NO_GRAPHS")[0] == '1');
    ddForce = getenv("PERFT_DD_FORCE") && getenv("PERFT_DD_FORCE")[0] == '1';
    ddMaxBytes = DD_MAX_BYTES_DEFAULT;
    if (const char *g = getenv("PERFT_DD_MAX_GB")) ddMaxBytes = atof(g) * (double)(1ull << 30);

    auto pick = [](int v) { return (v >= 0 && v < SV_COUNT) ? v : SV_KOGGE; };
    svExpand = pick(cfg.sliders_expand);
    svLeaf = pick(cfg.sliders_leaf);
    fill_tune(svLeaf, svExpand);
    ready = true;
    const bool tuneLeaf = cfg.sliders_leaf == PERFT_SLIDERS_AUTO;
    const bool tuneExpand = cfg.sliders_expand == PERFT_SLIDERS_AUTO;
    if (tuneLeaf || tuneExpand) {
        const int rc = autotune(tuneLeaf, tuneExpand);
        if (rc != PERFT_OK) {
            ready = false;
            return rc;
        }
    }
    memset(&stats, 0, sizeof stats);
    stats.sliders_expand = svExpand;
    stats.sliders_leaf = svLeaf;
    stats.arena_bytes = arenaCap;
    return PERFT_OK;
}

void Engine::shutdown()
{
    if (!ready) return;
    cudaSetDevice(device);
    cudaStreamSynchronize(stream);
    drop_dd();
    if (ioPos) cudaFree(ioPos);
    if (ioOut) cudaFree(ioOut);
    ioPos = ioOut = nullptr;
    ioCap = 0;
    cudaFree(arena);
    if (tt) cudaFree(tt);
    tt = nullptr;
    ttMask = 0;
    if (dTTStats) cudaFree(dTTStats);
    dTTStats = nullptr;
    cudaFree(dCounter);
    cudaFree(dErr);
    if (smallExec) cudaGraphExecDestroy(smallExec);
    if (smallGraph) cudaGraphDestroy(smallGraph);
    smallExec = nullptr;
    smallGraph = nullptr;
    if (dSmall) cudaFree(dSmall);
    dSmall = nullptr;
    if (hSmall) cudaFreeHost(hSmall);
    hSmall = nullptr;
    cudaFreeHost(hPinned);
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    cudaStreamDestroy(stream);
    arena = nullptr;
    ready = false;
}

bool Engine::alloc_level(DeviceLevel &L, u64 n, bool weighted)
{
    L.n = n;
    L.stride = (n + 31) & ~31ULL;
    L.planes = (u64 *)alloc(6 * 8 * L.stride);
    L.cnt = (u32 *)alloc(4 * L.stride);
    L.root = (u32 *)alloc(4 * L.stride);
    L.weight = weighted ? (unsigned long long *)alloc(8 * L.stride) : nullptr;
    return L.planes && L.cnt && L.root && (L.weight || !weighted);
}

// Merges the equal nodes of a level with `remaining` plies left.
int Engine::merge_level(const Joiners &J, const DeviceLevel &C, int remaining)
{
    if (!C.weight || C.n < 2 || J.maxDepth < remaining + MERGE_MIN_PLIES) return PERFT_OK;
    const u64 mark = arenaTop;
    unsigned long long *set = (unsigned long long *)alloc(8 * MERGE_SLOTS * C.n);
    arenaTop = mark;  // free again once the merge has run (stream order)
    if (!set) return PERFT_OK;  // the level stays unmerged
    const MergeLevel M{C.planes, C.stride, C.n,       C.cnt,     C.root,  C.weight, set,
                       J.segs,   J.depths, remaining, false,   nullptr, nullptr,  nullptr};
    const u64 blocks = (C.n + 255) / 256;
    k_merge_prepare<<<(unsigned)std::min<u64>(blocks, 64ull * nsm), 256, 0, stream>>>(M);
    k_merge_nodes<<<(unsigned)blocks, 256, 0, stream>>>(M);
    stats.other_launches += 2;
    return check(cudaGetLastError(), "k_merge_nodes");
}

// `remaining`: remaining depth of the level scanned; its items go to the
// count-only ply when it is 2, to an interior ply otherwise.
int Engine::scan(const u32 *cnt, u64 n, int remaining, bool compact, ParentIndex &ix)
{
    const u64 nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    const bool tiles = remaining > 2;
    ix.pscan = (u64 *)alloc(8 * (n + 1));
    ix.live = compact ? (u32 *)alloc(4 * n) : nullptr;
    ix.tileFirst = tiles ? (u32 *)alloc(4 * tile_index_len(n)) : nullptr;
    ScanSums *bsum = (ScanSums *)alloc(sizeof(ScanSums) * (nb + 1));
    if (!ix.pscan || (tiles && !ix.tileFirst) || !bsum || (compact && !ix.live)) return PERFT_ERR_OUT_OF_MEMORY;
    u64 *totals = (u64 *)(bsum + nb);
    k_scan_reduce<<<(unsigned)nb, SCAN_NT, 0, stream>>>(cnt, n, bsum);
    k_scan_top<<<1, SCAN_TOP_NT, 0, stream>>>(bsum, nb, totals);
    ENG_TRY(cudaGetLastError());
    ENG_TRY(cudaMemcpyAsync(hPinned, totals, 16, cudaMemcpyDeviceToHost, stream));
    ENG_TRY(cudaStreamSynchronize(stream));
    ix.total = hPinned[0];
    ix.nParents = compact ? hPinned[1] : n;
    // tile size: the tuned largest tile for this ply, made smaller while some
    // resident CTA would get no second tile
    if (tiles) {
        const TuneCfg &tc = cfg_for(MODE_EXPAND, remaining);
        ix.capLog2 = tc.cap;
        while (ix.capLog2 > TILE_MIN_LOG2 && (ix.total >> ix.capLog2) < 2ull * grid_for(MODE_EXPAND, tc)) ix.capLog2--;
        ix.capLog2 = tile_log2_for(ix.total, n, ix.capLog2);
    }
    if (compact)
        k_scan_apply<true><<<(unsigned)nb, SCAN_NT, 0, stream>>>(cnt, n, bsum, totals, ix.pscan, ix.live,
                                                                            ix.tileFirst, ix.capLog2);
    else
        k_scan_apply<false><<<(unsigned)nb, SCAN_NT, 0, stream>>>(cnt, n, bsum, totals, ix.pscan, nullptr,
                                                                             ix.tileFirst, ix.capLog2);
    stats.other_launches += 3;
    ENG_TRY(cudaGetLastError());
    return PERFT_OK;
}

int Engine::launch_tile(int mode, int remaining, const DeviceLevel &parents, const ParentIndex &ix, u64 itemBase,
                        u64 itemEnd, DeviceLevel *children, unsigned long long *rootCounts)
{
    const int capLog2 = ix.capLog2;
    TileParams P;
    memset(&P, 0, sizeof P);
    P.ppl = parents.planes;
    P.pstride = parents.stride;
    P.pscan = ix.pscan;
    P.live = ix.live;
    P.proot = parents.root;
    P.pweight = parents.weight;
    P.nParents = ix.nParents;
    P.tileFirst = ix.tileFirst;
    P.itemBase = itemBase;
    P.itemEnd = itemEnd;
    P.capLog2 = capLog2;
    P.tileCounter = dCounter;
    if (children) {
        P.cpl = children->planes;
        P.cstride = children->stride;
        P.ccnt = children->cnt;
        P.croot = children->root;
        P.cweight = children->weight;
    }
    P.rootCounts = rootCounts;
    P.moves = (unsigned long long *)(dCounter + 8);
    P.uncounted = remaining == 3;
    P.err = dErr;

    const u64 units = mode == MODE_LEAF ? leaf_units(ix.nParents)
                                        : (itemEnd - itemBase + (1ull << capLog2) - 1) >> capLog2;
    const TuneCfg &tc = cfg_for(mode, remaining);
    const int sv = tc.sv;
    const int grid = (int)std::min<u64>((u64)grid_for(mode, tc), units);
    ENG_TRY(cudaMemsetAsync(dCounter, 0, 64, stream));
    ENG_TRY(cudaEventRecord(ev0, stream));
    if (mode == MODE_LEAF) launch_tile_variant<MODE_LEAF>(sv, grid, stream, P);
    else launch_tile_variant<MODE_EXPAND>(sv, grid, stream, P);
    ENG_TRY(cudaGetLastError());
    ENG_TRY(cudaEventRecord(ev1, stream));
    if (mode == MODE_LEAF) ENG_TRY(cudaMemcpyAsync(hPinned + 2, P.moves, 8, cudaMemcpyDeviceToHost, stream));
    ENG_TRY(cudaStreamSynchronize(stream));
    float ms = 0.f;
    ENG_TRY(cudaEventElapsedTime(&ms, ev0, ev1));
    if (trace)
        fprintf(stderr, "perft-trace %s sv=%s parents=%llu items=%llu..%llu grid=%d ms=%.4f\n",
                mode == MODE_LEAF ? "leaf" : "expand", slider_name(sv), (unsigned long long)ix.nParents,
                (unsigned long long)itemBase, (unsigned long long)itemEnd, grid, ms);
    if (tuning) tuneAccMs[mode][mode == MODE_LEAF ? 2 : std::min(remaining, (int)TUNE_MAX_R)] += ms;
    if (mode == MODE_LEAF) {
        stats.leaf_launches++;
        stats.leaf_items += hPinned[2];
        stats.leaf_parents += ix.nParents;
        stats.leaf_ms += ms;
    } else {
        stats.expand_launches++;
        stats.expand_items += itemEnd - itemBase;
        stats.expand_ms += ms;
    }
    return PERFT_OK;
}

// L holds the nodes of one level, all with `remaining` plies left (>= 2).
// Writes the roots that join at remaining depth `depth` into C from index `at`.
int Engine::init_joiners(const Joiners &J, int depth, DeviceLevel &C, u64 at, unsigned long long *rootCounts)
{
    const u32 nj = J.n[depth];
    if (!nj) return PERFT_OK;
    k_init_roots<<<(nj + 127) / 128, 128, 0, stream>>>(J.dPos, J.ids[depth], nj, C.planes + 2 * at, C.stride,
                                                        C.cnt + at, C.root + at, C.weight ? C.weight + at : nullptr,
                                                        depth, rootCounts, dErr);
    stats.other_launches++;
    return check(cudaGetLastError(), "k_init_roots");
}

// L holds the nodes of one level, all with `remaining` plies left (>= 2).
// With `join`, the roots of depth remaining - 1 are appended to the children
// (to the last chunk when the children are chunked), so every depth group of
// a batch shares one launch per ply: the deepest roots start the search and
// shallower ones join the level whose remaining depth equals theirs.
int Engine::process_level(const DeviceLevel &L, int remaining, unsigned long long *rootCounts, const Joiners *join)
{
    const u32 nJoin = (join && remaining - 1 >= 2) ? join->n[remaining - 1] : 0;
    if (L.n == 0 && nJoin == 0) return PERFT_OK;
    const u64 mark = arenaTop;
    ParentIndex ix;
    const bool merged = L.weight && join && join->maxDepth >= remaining + MERGE_MIN_PLIES;
    int rc = L.n ? scan(L.cnt, L.n, remaining, merged, ix) : PERFT_OK;
    if (rc != PERFT_OK) return rc;
    const u64 total = ix.total;
    if (remaining == 2) {
        if (total) rc = launch_tile(MODE_LEAF, 2, L, ix, 0, total, nullptr, rootCounts);
        arenaTop = mark;
        return rc;
    }
    if (total == 0 && nJoin == 0) {
        arenaTop = mark;
        return PERFT_OK;
    }
    // interior ply: children fit whole, or in tile-aligned chunks
    const u64 slack = std::min<u64>(64ull << 20, arenaCap / 16);
    const u64 freeB = arena_free() > slack ? arena_free() - slack : 0;
    const bool weighted = L.weight != nullptr;
    u64 budgetNodes = freeB / (weighted ? NODE_BYTES_MERGE : NODE_BYTES);
    if (remaining > 3) budgetNodes /= 2;  // leave room for the plies below
    budgetNodes = budgetNodes > nJoin ? budgetNodes - nJoin : 0;
    // whole level when it fits; otherwise tile-aligned chunks
    u64 chunk = total <= budgetNodes ? total : (budgetNodes & ~(u64)(TILE_CAP - 1));
    if (chunk == 0 && total) return PERFT_ERR_OUT_OF_MEMORY;
    if (chunk < total) stats.chunked_levels++;
    const u64 nChunks = total ? (total + chunk - 1) / chunk : 1;
    for (u64 k = 0; k < nChunks; k++) {
        const u64 lo = k * chunk, hi = std::min(total, lo + chunk);
        const bool last = k + 1 == nChunks;
        const u64 cm = arenaTop;
        DeviceLevel C;
        if (!alloc_level(C, (hi - lo) + (last ? nJoin : 0), weighted)) return PERFT_ERR_OUT_OF_MEMORY;
        if (hi > lo) {
            rc = launch_tile(MODE_EXPAND, remaining, L, ix, lo, hi, &C, nullptr);
            if (rc != PERFT_OK) return rc;
        }
        if (last && nJoin) {
            rc = init_joiners(*join, remaining - 1, C, hi - lo, rootCounts);
            if (rc != PERFT_OK) return rc;
        }
        if (join) {
            rc = merge_level(*join, C, remaining - 1);
            if (rc != PERFT_OK) return rc;
        }
        rc = process_level(C, remaining - 1, rootCounts, join);
        if (rc != PERFT_OK) return rc;
        arenaTop = cm;
    }
    arenaTop = mark;
    return PERFT_OK;
}

// Per-depth autotuner.  A seeded calibration batch (32 playouts of 10-30
// plies at depth 6: interior plies with remaining depth 6..3, then the
// count-only ply) is run under candidate launch configurations, one warm-up
// and three timed runs each; every tile launch's CUDA-event time is charged
// to its (ply kind, remaining depth) key, and each key keeps the median of
// its three runs.  Coordinate search, every key at once:
//   1. slider variant (all five), largest tiles, all resident CTAs;
//   2. interior plies: largest tile 2^13 / 2^12 / 2^11 items with each key's variant;
//   3. resident CTAs per SM: all that fit, or one fewer.
// A candidate replaces a key's current choice only when it is more than 1%
// faster, so near-ties resolve to the same (earlier) choice on every run.
// These are the reference's compile-time knobs (switches.h:13-26: block size,
// memory) chosen per depth on the device at hand.  Results are kept per
// device for the life of the process (PERFT_RETUNE=1 times again).
int Engine::autotune(bool leaf, bool expand)
{
    struct Cached {
        TuneCfg tab[2][TUNE_MAX_R + 1];
        int maxR;
    };
    static std::mutex cacheMu;
    static std::map<std::pair<int, int>, Cached> cache;
    const std::pair<int, int> key{device, (leaf ? 2 : 0) | (expand ? 1 : 0)};
    const bool retune = getenv("PERFT_RETUNE") && getenv("PERFT_RETUNE")[0] == '1';
    auto adopt = [&]() {
        svLeaf = tuneTab[MODE_LEAF][2].sv;
        svExpand = tuneTab[MODE_EXPAND][3].sv;
    };
    {
        std::lock_guard<std::mutex> lk(cacheMu);
        auto it = cache.find(key);
        if (!retune && it != cache.end()) {
            for (int m = 0; m < 2; m++) {
                for (int r = 0; r <= TUNE_MAX_R; r++) {
                    // a mode that is not tuned keeps the caller's variant
                    if ((m == MODE_LEAF && !leaf) || (m == MODE_EXPAND && !expand)) continue;
                    tuneTab[m][r] = it->second.tab[m][r];
                }
            }
            tunedMaxR = it->second.maxR;
            adopt();
            return PERFT_OK;
        }
    }

    constexpr u32 N = 32;
    constexpr int CAL_DEPTH = 6;
    std::vector<perft_pos48> pos(N);
    int rc = perft_random_playouts(0xA070707EULL, N, 10, 30, pos.data());
    if (rc != PERFT_OK) return rc;
    std::vector<uint8_t> depths(N, CAL_DEPTH);
    const u64 mark = arenaTop;
    u64 *dPos = (u64 *)alloc(48ull * N);
    u64 *dOut = (u64 *)alloc(8ull * N);
    if (!dPos || !dOut) return PERFT_ERR_OUT_OF_MEMORY;
    ENG_TRY(cudaMemcpyAsync(dPos, pos.data(), 48ull * N, cudaMemcpyHostToDevice, stream));
    ulonglong2 *keepTT = tt;
    tt = nullptr;  // time the kernels, not table hits
    const bool keepDD = ddEnabled;
    ddEnabled = false;  // the host-driven path times each launch
    struct Restore {
        Engine &e;
        ulonglong2 *t;
        bool dd;
        u64 mark;
        ~Restore()
        {
            e.tt = t;
            e.ddEnabled = dd;
            e.tuning = false;
            e.arenaTop = mark;
        }
    } restore{*this, keepTT, keepDD, mark};
    tunedMaxR = CAL_DEPTH;

    // median over the timed runs of each key's time under the current table
    double med[2][TUNE_MAX_R + 1];
    auto measure = [&]() -> int {
        std::vector<double> reps[2][TUNE_MAX_R + 1];
        for (int rep = 0; rep < 4; rep++) {
            memset(tuneAccMs, 0, sizeof tuneAccMs);
            tuning = true;
            const perft_stats keep = stats;
            const int r = run_batch(dPos, depths.data(), N, dOut);
            stats = keep;  // calibration runs stay out of the statistics
            tuning = false;
            if (r != PERFT_OK) return r;
            if (rep == 0) continue;  // warms caches and clocks
            for (int m = 0; m < 2; m++)
                for (int k = 0; k <= TUNE_MAX_R; k++) reps[m][k].push_back(tuneAccMs[m][k]);
        }
        for (int m = 0; m < 2; m++)
            for (int k = 0; k <= TUNE_MAX_R; k++) {
                std::sort(reps[m][k].begin(), reps[m][k].end());
                med[m][k] = reps[m][k][reps[m][k].size() / 2];
            }
        return PERFT_OK;
    };
    auto keys = [&](auto fn) {  // every tuned (mode, r) key of the calibration
        if (leaf) fn(MODE_LEAF, 2);
        if (expand)
            for (int r = 3; r <= CAL_DEPTH; r++) fn(MODE_EXPAND, r);
    };
    double best[2][TUNE_MAX_R + 1];
    TuneCfg chosen[2][TUNE_MAX_R + 1];
    auto apply = [&](int m, int r, const TuneCfg &c) {
        if (m == MODE_LEAF) {
            for (int k = 0; k <= TUNE_MAX_R; k++) tuneTab[MODE_LEAF][k] = c;
        } else {
            tuneTab[MODE_EXPAND][r] = c;
            if (r == 3)
                for (int k = 0; k < 3; k++) tuneTab[MODE_EXPAND][k] = c;
            if (r == CAL_DEPTH)
                for (int k = CAL_DEPTH + 1; k <= TUNE_MAX_R; k++) tuneTab[MODE_EXPAND][k] = c;
        }
    };
    // stage 1: slider variant
    for (int v = 0; v < SV_COUNT; v++) {
        keys([&](int m, int r) { apply(m, r, TuneCfg{v, TILE_CAP_LOG2, 0, 0}); });
        if ((rc = measure()) != PERFT_OK) return rc;
        keys([&](int m, int r) {
            if (v == 0 || med[m][r] < 0.99 * best[m][r]) {
                best[m][r] = med[m][r];
                chosen[m][r] = TuneCfg{v, TILE_CAP_LOG2, 0, med[m][r]};
            }
        });
    }
    // stage 2: largest tile (interior plies; the count-only ply has none)
    for (int cap = TILE_CAP_LOG2 - 1; expand && cap >= TILE_CAP_LOG2 - 2 && cap >= TILE_MIN_LOG2; cap--) {
        keys([&](int m, int r) { apply(m, r, m == MODE_LEAF ? chosen[m][r] : TuneCfg{chosen[m][r].sv, cap, 0, 0}); });
        if ((rc = measure()) != PERFT_OK) return rc;
        keys([&](int m, int r) {
            if (m != MODE_LEAF && med[m][r] < 0.99 * best[m][r]) {
                best[m][r] = med[m][r];
                chosen[m][r] = TuneCfg{chosen[m][r].sv, cap, 0, med[m][r]};
            }
        });
    }
    // stage 3: one resident CTA per SM fewer
    keys([&](int m, int r) {
        const TuneCfg &c = chosen[m][r];
        apply(m, r, TuneCfg{c.sv, c.cap, std::max(1, max_ctas(m, c.sv) - 1), 0});
    });
    if ((rc = measure()) != PERFT_OK) return rc;
    keys([&](int m, int r) {
        if (med[m][r] < 0.99 * best[m][r]) {
            best[m][r] = med[m][r];
            chosen[m][r] = TuneCfg{chosen[m][r].sv, chosen[m][r].cap, std::max(1, max_ctas(m, chosen[m][r].sv) - 1),
                                   med[m][r]};
        }
    });
    keys([&](int m, int r) { apply(m, r, chosen[m][r]); });
    adopt();
    {
        std::lock_guard<std::mutex> lk(cacheMu);
        Cached &c = cache[key];
        memcpy(c.tab, tuneTab, sizeof tuneTab);
        c.maxR = tunedMaxR;
    }
    return PERFT_OK;
}

bool Engine::alloc_level_tt(DeviceLevel &L, u64 n)
{
    if (!alloc_level(L, n)) return false;
    if (tt) {
        L.hash = (u64 *)alloc(8 * L.stride);
        L.hash2 = (u64 *)alloc(8 * L.stride);
        if (!L.hash || !L.hash2) return false;
    }
    L.acc = (unsigned long long *)alloc(8 * L.stride);
    L.alias = (u32 *)alloc(4 * L.stride);
    return L.acc && L.alias;
}

int Engine::tt_clear()
{
    if (tt) ENG_TRY(cudaMemsetAsync(tt, 0, (ttMask + 1) * sizeof(ulonglong2), stream));
    ENG_TRY(cudaMemsetAsync(dTTStats, 0, sizeof(TTStats), stream));
    ENG_TRY(cudaStreamSynchronize(stream));
    return PERFT_OK;
}

// Transposition-table version of process_level.  L (remaining plies
// `remaining`) is merged over all its roots, and the nodes that stay are
// hashed and probed; hits and copies are not expanded.  Subtree sums accumulate in L.acc: directly from the
// count-only last ply, or from the child levels' finish pass.  When L is
// done, owners are stored, duplicates copy their owner's value, and the
// values are added into parentAcc (or written to the roots' results).
int Engine::process_level_tt(const DeviceLevel &L, int remaining, unsigned long long *parentAcc,
                             unsigned long long *rootOut)
{
    if (L.n == 0) return PERFT_OK;
    const u64 mark = arenaTop;
    const unsigned nb = (unsigned)((L.n + 255) / 256);
    const bool useTT = tt != nullptr && remaining >= ttMinDepth;

    unsigned long long *set = (unsigned long long *)alloc(8 * MERGE_SLOTS * L.n);
    if (!set) return PERFT_ERR_OUT_OF_MEMORY;
    ENG_TRY(cudaMemsetAsync(set, 0xFF, 8 * MERGE_SLOTS * L.n, stream));
    const MergeLevel M{L.planes, L.stride, L.n,     L.cnt, nullptr, nullptr, set,
                       nullptr,  nullptr,  remaining, false, L.alias, L.acc, &dTTStats->aliases};
    k_merge_linked<<<nb, 256, 0, stream>>>(M);
    if (useTT)
        k_tt_probe<<<(unsigned)std::min<u64>(nb, 8ull * nsm), 256, 0, stream>>>(
            L.planes, L.stride, L.n, remaining, ttKeyMask, L.cnt, L.hash, L.hash2, L.acc, L.alias, tt, ttMask,
            dTTStats);
    stats.other_launches += 1 + useTT;
    ENG_TRY(cudaGetLastError());
    arenaTop = mark;  // the set is no longer needed

    ParentIndex ix;
    int rc = scan(L.cnt, L.n, remaining, true, ix);
    if (rc != PERFT_OK) return rc;
    const u64 total = ix.total;
    DeviceLevel self = L;
    self.root = nullptr;  // tile sums and child links point at the parent itself
    if (total > 0) {
        if (remaining == 2) {
            rc = launch_tile(MODE_LEAF, 2, self, ix, 0, total, nullptr, L.acc);
            if (rc != PERFT_OK) return rc;
        } else {
            const u64 slack = std::min<u64>(64ull << 20, arenaCap / 16);
            const u64 freeB = arena_free() > slack ? arena_free() - slack : 0;
            u64 budgetNodes = freeB / (tt ? NODE_BYTES_TT : NODE_BYTES_LINKED);
            if (remaining > 3) budgetNodes /= 2;
            const u64 chunk = total <= budgetNodes ? total : (budgetNodes & ~(u64)(TILE_CAP - 1));
            if (chunk == 0) return PERFT_ERR_OUT_OF_MEMORY;
            if (chunk < total) stats.chunked_levels++;
            for (u64 lo = 0; lo < total; lo += chunk) {
                const u64 hi = std::min(total, lo + chunk);
                const u64 cm = arenaTop;
                DeviceLevel C;
                if (!alloc_level_tt(C, hi - lo)) return PERFT_ERR_OUT_OF_MEMORY;
                rc = launch_tile(MODE_EXPAND, remaining, self, ix, lo, hi, &C, nullptr);
                if (rc != PERFT_OK) return rc;
                rc = process_level_tt(C, remaining - 1, L.acc, nullptr);
                if (rc != PERFT_OK) return rc;
                arenaTop = cm;
            }
        }
    }
    arenaTop = mark;
    k_tt_finish<<<nb, 256, 0, stream>>>(L.n, useTT, L.hash, L.hash2, L.acc, L.alias, L.root,
                                        parentAcc, tt,
                                        ttMask, dTTStats);
    stats.other_launches++;
    if (rootOut) {
        k_tt_roots<<<nb, 256, 0, stream>>>(L.n, L.acc, L.alias, L.root, rootOut);
        stats.other_launches++;
    }
    ENG_TRY(cudaGetLastError());
    return PERFT_OK;
}

void Engine::drop_dd()
{
    for (DDGraph &G : ddCache) {
        if (G.exec) cudaGraphExecDestroy(G.exec);
        if (G.graph) cudaGraphDestroy(G.graph);
        cudaFreeHost(G.hTemplate);
        cudaFreeHost(G.hIds);
        cudaFreeHost(G.hFlags);
        if (G.evLeaf0) cudaEventDestroy(G.evLeaf0);
        if (G.evLeaf1) cudaEventDestroy(G.evLeaf1);
    }
    ddCache.clear();
}

// Captures one device-driven perft of G.n roots of any depth mix.  The
// deepest roots form level 0; a root of depth d joins level G.depth - d
// (behind that level's children), so every ply of the whole batch is one
// scan and one tile launch.  Roots of depth 0 and 1 are answered by
// k_init_roots.  Every buffer the graph reads is re-initialised inside it
// (plan, root ids, outputs), so the region above the arena top may be reused
// by other calls between replays.
int Engine::build_dd(DDGraph &G)
{
    const u64 n = G.n;
    const int d = G.depth;
    std::vector<u32> order;
    order.reserve(n);
    u32 nAt[DD_MAX_LEVELS + 2] = {};
    u64 offAt[DD_MAX_LEVELS + 2] = {};
    for (int dd = d; dd >= 0; dd--) {
        offAt[dd] = order.size();
        for (u32 i = 0; i < n; i++)
            if (G.depths[i] == dd) order.push_back(i);
        nAt[dd] = (u32)(order.size() - offAt[dd]);
    }
    const u64 off0 = (arenaTop + 255) & ~255ULL;
    char *base = arena + off0;
    const u64 cap = arenaCap - off0;
    u64 bump = 0;
    auto place = [&](u64 bytes) -> char * {
        const u64 a = (bump + 255) & ~255ULL;
        bump = a + bytes;
        return base + a;
    };
    DevPlan *dPlan = (DevPlan *)place(sizeof(DevPlan));
    u32 *dIds = (u32 *)place(4 * n);
    // merged transpositions (levels at least MERGE_MIN_PLIES below some root)
    const bool merge = mergeEnabled && d - 2 >= MERGE_MIN_PLIES;
    uint8_t *dDepths = merge ? (uint8_t *)place(n) : nullptr;
    MergeSeg *dSegs = merge ? (MergeSeg *)place(sizeof(MergeSeg) * n) : nullptr;
    const u64 n0 = nAt[d];
    LevelDesc L0{};
    L0.n = n0;
    L0.nChild = 0;
    L0.stride = (n0 + 31) & ~31ULL;
    L0.planes = (u64 *)place(48 * L0.stride);
    L0.cnt = (u32 *)place(4 * L0.stride);
    L0.root = (u32 *)place(4 * L0.stride);
    L0.weight = merge ? (unsigned long long *)place(8 * L0.stride) : nullptr;
    L0.pscan = (u64 *)place(8 * (n0 + 1));
    L0.tileFirst = (u32 *)place(4 * tile_index_len(n0));
    L0.bsum = (ScanSums *)place(sizeof(ScanSums) * ((n0 + SCAN_CHUNK - 1) / SCAN_CHUNK + 1));
    // scratch level for the roots of depth 0 and 1 (counts only)
    const u64 nShallow = std::max<u64>(nAt[0], nAt[1]);
    const u64 sStride = (nShallow + 31) & ~31ULL;
    u64 *sPlanes = (u64 *)place(48 * std::max<u64>(sStride, 32));
    u32 *sCnt = (u32 *)place(4 * std::max<u64>(sStride, 32));
    u32 *sRoot = (u32 *)place(4 * std::max<u64>(sStride, 32));
    // a single root's first two plies are one launch (k_dd_front)
    const bool front = n == 1 && d - 2 > FRONT_LEVEL && smallEnabled;
    LevelDesc L2{};
    if (front) {
        L2.stride = (FRONT_NODES + 31) & ~31ULL;
        L2.planes = (u64 *)place(48 * L2.stride);
        L2.cnt = (u32 *)place(4 * L2.stride);
        L2.root = (u32 *)place(4 * L2.stride);
        L2.weight = merge ? (unsigned long long *)place(8 * L2.stride) : nullptr;
        L2.pscan = (u64 *)place(8 * (FRONT_NODES + 1));
        L2.tileFirst = (u32 *)place(4 * tile_index_len(FRONT_NODES));
        L2.bsum = (ScanSums *)place(sizeof(ScanSums) * ((FRONT_NODES + SCAN_CHUNK - 1) / SCAN_CHUNK + 1));
    }
    if (bump > cap) return PERFT_ERR_OUT_OF_MEMORY;

    ENG_TRY(cudaMallocHost(&G.hTemplate, sizeof(DevPlan)));
    ENG_TRY(cudaMallocHost(&G.hIds, 5 * n));  // root ids, then every root's depth
    ENG_TRY(cudaMallocHost(&G.hFlags, 64));
    ENG_TRY(cudaEventCreate(&G.evLeaf0));
    ENG_TRY(cudaEventCreate(&G.evLeaf1));
    memset(G.hTemplate, 0, sizeof(DevPlan));
    G.hTemplate->base = base;
    G.hTemplate->cap = cap;
    G.hTemplate->bump = bump;
    G.hTemplate->tileTarget = 2 * gridTile[MODE_LEAF][G.svL];
    G.hTemplate->tileCounter = dCounter;
    G.hTemplate->lastLv = d - 2;
    G.hTemplate->weighted = merge;
    G.hTemplate->segs = dSegs;
    G.hTemplate->rootDepth = dDepths;
    for (int lv = MERGE_MIN_PLIES; lv <= d - 2; lv++) G.hTemplate->mergeLv[lv] = merge;
    G.hTemplate->lv[0] = L0;
    if (front) G.hTemplate->lv[FRONT_LEVEL] = L2;
    for (int dd = 2; dd < d; dd++) {
        G.hTemplate->joinN[d - dd] = nAt[dd];
        G.hTemplate->joinIds[d - dd] = dIds + offAt[dd];
    }
    // per ply: the tuned variant (one of the two graph instantiations) and largest tile
    auto ddSv = [](int v) { return (v == SV_KOGGE || v == SV_KOGGE_SPLIT) ? v : (int)SV_KOGGE; };
    int lvSv[DD_MAX_LEVELS] = {}, lvGrid[DD_MAX_LEVELS] = {};
    for (int lv = 0; lv <= d - 2; lv++) {
        const int r = d - lv, mode = r == 2 ? MODE_LEAF : MODE_EXPAND;
        const bool last = lv == d - 2;
        TuneCfg c = cfg_for(mode, r);
        c.sv = ddSv(c.sv);
        lvSv[lv] = c.sv;
        lvGrid[lv] = grid_for(mode, c);
        if (!last) G.hTemplate->capMax[lv] = c.cap;
        TileParams &T = G.hTemplate->tp[lv];  // the scan fills the level fields on the device
        T.tileCounter = dCounter;
        T.rootCounts = (unsigned long long *)G.dOut;
        T.moves = &dPlan->leafMoves;
        T.uncounted = r == 3;
        T.err = dErr;
        // A ply predicted to have few tiles gets a grid of four CTAs per
        // predicted tile (at least 8) instead of one CTA per resident slot:
        // the tile kernel is persistent, so any grid is correct, and the
        // CTAs that would find no tile cost launch and exit time.
        if ((int)G.predLv.size() > lv + 1) {
            const double items = last ? G.predLv[lv] * 32.0 : G.predLv[lv + 1];
            const double tiles = items / (double)(1u << TILE_MIN_LOG2) + 1.0;
            if (4.0 * tiles < (double)lvGrid[lv]) lvGrid[lv] = std::max(8, (int)(4.0 * tiles));
        }
    }
    memcpy(G.hIds, order.data(), 4 * n);
    memcpy(G.hIds + n, G.depths.data(), n);

    ENG_TRY(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    cudaMemcpyAsync(dPlan, G.hTemplate, sizeof(DevPlan), cudaMemcpyHostToDevice, stream);
    cudaMemcpyAsync(dIds, G.hIds, 4 * n, cudaMemcpyHostToDevice, stream);
    if (merge) cudaMemcpyAsync(dDepths, G.hIds + n, n, cudaMemcpyHostToDevice, stream);
    cudaMemsetAsync(G.dOut, 0, 8 * n, stream);
    cudaMemsetAsync(dErr, 0, 4, stream);
    G.otherLaunches = (nAt[0] ? 1 : 0) + (nAt[1] ? 1 : 0) + (d >= 2 ? 1 : 0);
    for (int dd = 0; dd <= 1; dd++)
        if (nAt[dd])
            k_init_roots<<<(nAt[dd] + 127) / 128, 128, 0, stream>>>(G.dPos, dIds + offAt[dd], nAt[dd], sPlanes,
                                                                   sStride, sCnt, sRoot, nullptr, dd,
                                                                   (unsigned long long *)G.dOut, dErr);
    if (front)
        k_dd_front<<<MAX_LEGAL_MOVES, SMALL_NT, SMALL_DYN_SMEM, stream>>>(dPlan, G.dPos, dErr);
    else if (d >= 2)
        k_init_roots<<<(unsigned)((n0 + 127) / 128), 128, 0, stream>>>(G.dPos, dIds + offAt[d], (u32)n0,
                                                                      L0.planes, L0.stride, L0.cnt, L0.root,
                                                                      L0.weight, d,
                                                                      (unsigned long long *)G.dOut, dErr);
    const int lv0 = front ? FRONT_LEVEL : 0;
    G.expandLaunches = d > 2 ? d - 2 - lv0 : 0;
    for (int lv = lv0; lv <= d - 2; lv++) {
        const int last = lv == d - 2;
        // levels predicted small take one single-block scan launch instead of three
        if ((int)G.predLv.size() > lv && G.predLv[lv] <= 32768.0) {
            k_dd_scan_small<<<1, 1024, 0, stream>>>(dPlan, lv, last);
            G.otherLaunches += 1;
        } else {
            // grid-stride scans: large predicted levels get up to one block
            // per chunk (64 per SM at most), like the host-driven scan
            int sg = ddGridScan;
            if ((int)G.predLv.size() > lv)
                sg = (int)std::min<double>(64.0 * nsm, std::max<double>(ddGridScan, G.predLv[lv] / SCAN_CHUNK));
            k_dd_scan_reduce<<<sg, SCAN_NT, 0, stream>>>(dPlan, lv);
            G.otherLaunches += 3;
            k_dd_scan_top<<<1, SCAN_TOP_NT, 0, stream>>>(dPlan, lv, last);
            if (G.hTemplate->mergeLv[lv]) k_dd_scan_apply<true><<<sg, SCAN_NT, 0, stream>>>(dPlan, lv);
            else k_dd_scan_apply<false><<<sg, SCAN_NT, 0, stream>>>(dPlan, lv);
        }
        // (the scan reset the tile cursor)
        // Large plies read their launch parameters (completed by the scan)
        // from the constant bank, copied there by a copy node; small ones
        // from the plan, through shared memory (no copy node).
        const bool big = !((int)G.predLv.size() > lv + 1 &&
                           (last ? G.predLv[lv] * 32.0 : G.predLv[lv + 1]) < DD_CONST_MIN_ITEMS);
        if (big)
            cudaMemcpyToSymbolAsync(c_ddTile, &dPlan->tp[lv], sizeof(TileParams), 0, cudaMemcpyDeviceToDevice,
                                    stream);
        TileParams P;
        memset(&P, 0, sizeof P);
        P.planEntry = &dPlan->tp[lv];
        const int sv = lvSv[lv];
        const int grid = lvGrid[lv];
        if (last) {
            // external records: event record nodes in the graph (a plain
            // record during capture only orders the capture)
            cudaEventRecordWithFlags(G.evLeaf0, stream, cudaEventRecordExternal);
            launch_dd_tile<MODE_LEAF>(sv, big, grid, stream, P);
            cudaEventRecordWithFlags(G.evLeaf1, stream, cudaEventRecordExternal);
        } else {
            launch_dd_tile<MODE_EXPAND>(sv, big, grid, stream, P);
            const u32 nj = G.hTemplate->joinN[lv + 1];
            if (nj) {
                k_dd_join<<<(nj + 127) / 128, 128, 0, stream>>>(dPlan, lv + 1, G.dPos, dErr);
                G.otherLaunches += 1;
            }
            if (G.hTemplate->mergeLv[lv + 1]) {
                // grid-stride: any grid is correct; a block per 256 predicted nodes, up
                // to 512 blocks per SM.  The prediction takes 0.7 of a merged level to
                // remain; deep levels keep less, and most of its blocks would find no
                // node (an opening at depth 8 7.16 -> 6.74 ms, 512 positions at depths
                // 4-6 38.7 -> 38.3 ms; 128, 256 and 1024 blocks per SM: 6.82, 6.80 and
                // 6.75 ms).
                double mg = 64.0 * nsm;
                if ((int)G.predLv.size() > lv + 1) mg = std::max(8.0, G.predLv[lv + 1] / 256.0);
                k_dd_merge_prepare<<<(unsigned)std::min(mg, 64.0 * nsm), 256, 0, stream>>>(dPlan, lv + 1, d - (lv + 1));
                k_dd_merge_nodes<<<(unsigned)std::min(mg, 512.0 * nsm), 256, 0, stream>>>(dPlan, lv + 1, d - (lv + 1));
                G.otherLaunches += 2;
            }
        }
    }
    cudaMemcpyAsync(&G.hFlags[0], &dPlan->overflow, 4, cudaMemcpyDeviceToHost, stream);
    cudaMemcpyAsync(&G.hFlags[1], dErr, 4, cudaMemcpyDeviceToHost, stream);
    if (d >= 2) {
        cudaMemcpyAsync(&G.hFlags[2], &dPlan->leafMoves, 8, cudaMemcpyDeviceToHost, stream);
        cudaMemcpyAsync(&G.hFlags[3], &dPlan->tp[d - 2].nParents, 8, cudaMemcpyDeviceToHost, stream);
    }
    const cudaError_t ce = cudaStreamEndCapture(stream, &G.graph);
    if (ce != cudaSuccess) {
        cudaGetLastError();
        return check(ce, "capture of the device-driven perft");
    }
    ENG_TRY(cudaGraphInstantiate(&G.exec, G.graph, 0));
    return PERFT_OK;
}

// Batches whose predicted tree fits the arena run as one replayed graph,
// whatever their depth mix: the launch sequence is fixed and the sizes live
// on the device, so the host only waits once.  The prediction charges each
// root its own move count times 32 per further ply (times MERGE_KEPT from the
// third ply on, where levels are merged) and 72 bytes per node of every
// materialised ply (planes, count, root, scan entry, tile index; 92 with path
// weights, live list and merge set), against 85% of the free arena.  `handled`
// stays false when the batch is not eligible or the device plan overflowed; the caller
// then runs the host-driven path.
int Engine::run_dd(const u64 *dPos, const uint8_t *depths, u32 n, u64 *dOut, bool &handled)
{
    handled = false;
    if (!ddEnabled || tt || n == 0) return PERFT_OK;
    int d = 0;
    for (u32 i = 0; i < n; i++) d = std::max<int>(d, depths[i]);
    if (d > DD_MAX_LEVELS) return PERFT_OK;
    // the graph path has the two Kogge-Stone instantiations; another tuned
    // variant runs there as plain Kogge-Stone (same counts)
    auto ddSv = [](int v) { return (v == SV_KOGGE || v == SV_KOGGE_SPLIT) ? v : (int)SV_KOGGE; };
    const int ddL = ddSv(svLeaf), ddE = ddSv(svExpand);
    DDGraph *G = nullptr;
    for (DDGraph &g : ddCache)
        if (g.depth == d && g.n == n && g.dPos == dPos && g.dOut == dOut && g.top == arenaTop && g.svL == ddL &&
            g.svE == ddE && memcmp(g.depths.data(), depths, n) == 0)
            G = &g;
    if (G && G->overflowed) return PERFT_OK;
    std::vector<double> predLv;
    if (!G && !ddForce) {
        // (The measured mean is about 30 moves.)  The positions are read back
        // once, when the graph is built; a replay needs no prediction.
        std::vector<u64> hp(6ull * n);
        ENG_TRY(cudaMemcpyAsync(hp.data(), dPos, 48ull * n, cudaMemcpyDeviceToHost, stream));
        ENG_TRY(cudaStreamSynchronize(stream));
        double est = 0;
        predLv.assign(DD_MAX_LEVELS, 0.0);
        for (u32 i = 0; i < n; i++) {
            if (depths[i] < 2 || validate_pos48(&hp[6ull * i]) != 0) continue;
            const int join = d - depths[i];  // the level this root enters
            predLv[join] += 1.0;
            double nodes = (double)count_moves<SV_KOGGE>(from_pos48(&hp[6ull * i])), sum = 0;
            for (int k = 1; k <= (int)depths[i] - 2; k++) {
                sum += nodes;
                predLv[join + k] += nodes;
                nodes *= 32.0;
                if (mergeEnabled && k >= MERGE_MIN_PLIES) nodes *= MERGE_KEPT;
            }
            est += sum * (mergeEnabled && d - 2 >= MERGE_MIN_PLIES ? 92.0 : 72.0);
        }
        if (est > 0.85 * (double)arena_free()) return PERFT_OK;
        if (est > ddMaxBytes) return PERFT_OK;
    }
    if (!G) {
        if (ddCache.size() >= 16) {
            DDGraph &old = ddCache.front();
            if (old.exec) cudaGraphExecDestroy(old.exec);
            if (old.graph) cudaGraphDestroy(old.graph);
            cudaFreeHost(old.hTemplate);
            cudaFreeHost(old.hIds);
            cudaFreeHost(old.hFlags);
            if (old.evLeaf0) cudaEventDestroy(old.evLeaf0);
            if (old.evLeaf1) cudaEventDestroy(old.evLeaf1);
            ddCache.erase(ddCache.begin());
        }
        ddCache.emplace_back();
        G = &ddCache.back();
        G->depth = d;
        G->depths.assign(depths, depths + n);
        G->n = n;
        G->dPos = dPos;
        G->dOut = dOut;
        G->top = arenaTop;
        G->svL = ddL;
        G->svE = ddE;
        G->predLv = predLv;
        const int rc = build_dd(*G);
        if (rc != PERFT_OK) {
            drop_dd();
            return rc == PERFT_ERR_OUT_OF_MEMORY ? PERFT_OK : rc;
        }
    }
    G->hFlags[2] = G->hFlags[3] = 0;
    ENG_TRY(cudaGraphLaunch(G->exec, stream));
    ENG_TRY(cudaStreamSynchronize(stream));
    stats.other_launches += G->otherLaunches;
    stats.expand_launches += G->expandLaunches;
    stats.leaf_launches += d >= 2 ? 1 : 0;
    stats.graph_launches += 1;
    if ((u32)G->hFlags[0]) {  // overflow: rerun host-driven, now and on later calls
        G->overflowed = true;
        return PERFT_OK;
    }
    const u32 e = (u32)G->hFlags[1];
    if (e & DERR_BAD_POSITION) return PERFT_ERR_INVALID_ARG;
    if (e) return PERFT_ERR_INTERNAL;
    stats.leaf_items += G->hFlags[2];
    stats.leaf_parents += G->hFlags[3];
    if (d >= 2) {
        float ms = 0.f;  // the count-only ply's device time, from the events recorded in the graph
        if (cudaEventElapsedTime(&ms, G->evLeaf0, G->evLeaf1) == cudaSuccess) stats.leaf_ms += ms;
        else cudaGetLastError();  // a statistic only: leave no error behind for the caller
    }
    handled = true;
    return PERFT_OK;
}

// Fills the launch's parameters; returns the grid.  A depth-4 position has
// SMALL_SLICES CTAs' worth of subtree roots and a depth-5 position fills the
// device; subtrees are shared by more CTAs while the grid stays one wave.
template <int N>
u32 Engine::small_params(SmallParams<N> &P, const u64 *dPos, const u64 *pos, const uint8_t *depths, u32 n, u64 *dOut)
{
    P.dPos = dPos;
    P.dOut = dOut;
    P.host = hSmall;
    P.state = dSmall;
    P.n = n;
    P.listCap = smallListCap;
    u32 base = 0, n3 = 0, n4 = 0;
    for (u32 i = 0; i < n; i++) {
        n3 += depths[i] == 3;
        n4 += depths[i] == 4;
        base += depths[i] < 3;
    }
    auto total = [&](u32 k) { return base + n3 * k + n4 * k * SMALL_SLICES; };
    u32 split = 1;
    while (split < 8 && total(2 * split) <= (u32)smallGrid) split *= 2;
    u32 grid = 0;
    for (u32 i = 0; i < n; i++) {
        P.unit0[i] = (uint16_t)grid;
        P.depth[i] = depths[i];
        P.split[i] = (uint8_t)(depths[i] == 3 || depths[i] == 4 ? split : 1);
        grid += depths[i] == 5 ? (u32)smallGrid : depths[i] == 4 ? split * SMALL_SLICES : depths[i] == 3 ? split : 1;
    }
    P.unit0[n] = (uint16_t)grid;
    if (!dPos) memcpy(P.pos, pos, 48ull * n);
    return grid;
}

// One position of depth 2..5, or a batch of small ones: all trees in one
// k_small_trees launch, positions passed as launch parameters when they are
// on the host (dPos null), counts and flags written to mapped host memory.
// Not handled (the level pipeline runs it) when disabled, when depths or
// sizes are outside that, or when a position has more depth-5 subtree roots,
// moves or pieces than the kernel holds.
int Engine::run_small(const u64 *dPos, const u64 *pos, const uint8_t *depths, u32 n, u64 *dOut, u64 *hOut,
                      bool &handled)
{
    handled = false;
    if (!smallEnabled) return PERFT_OK;
    if (n == 1) {
        if (depths[0] < 2 || depths[0] > SMALL_MAX_DEPTH) return PERFT_OK;
        SmallParams<1> P;
        const u32 grid = small_params(P, dPos, pos, depths, 1, dOut);
        k_small_trees<1><<<grid, SMALL_NT, SMALL_DYN_SMEM, stream>>>(P);
        ENG_TRY(cudaGetLastError());
    } else {
        if (n > (u32)SMALL_BATCH || tt || !ddEnabled) return PERFT_OK;
        for (u32 i = 0; i < n; i++)
            if (depths[i] > SMALL_BATCH_DEPTH) return PERFT_OK;
        cudaKernelNodeParams kp = {};
        void *args[] = {&smallBatch};
        kp.func = (void *)k_small_trees<SMALL_BATCH>;
        kp.gridDim = dim3(small_params(smallBatch, dPos, pos, depths, n, dOut));
        kp.blockDim = dim3(SMALL_NT);
        kp.sharedMemBytes = (unsigned)SMALL_DYN_SMEM;
        kp.kernelParams = args;
        ENG_TRY(cudaGraphExecKernelNodeSetParams(smallExec, smallNode, &kp));
        ENG_TRY(cudaGraphLaunch(smallExec, stream));
    }
    ENG_TRY(cudaStreamSynchronize(stream));
    const u32 flags = hSmall->flags;
    if (flags & DERR_BAD_POSITION) return PERFT_ERR_INVALID_ARG;
    if (flags) return PERFT_OK;
    if (hOut) memcpy(hOut, hSmall->count, 8ull * n);
    if (n == 1) {
        stats.small_launches += 1;
    } else {
        stats.graph_launches += 1;
        stats.other_launches += 1;
    }
    handled = true;
    return PERFT_OK;
}

// Whether a batch's trees meet often enough to be searched as one: positions
// of one depth whose occupied squares differ in at most RELATED_SQUARES from
// the first one's, as the boards of a divided or host-split search do (five
// plies move at most ten squares; unrelated middlegames differ in 20-30), and
// enough work to pay for the linked levels' host round trips.  Measured,
// searched together against root by root, by predicted parents of the
// count-only ply: 0.4 M 0.91 / 0.78 ms, 0.54 M 0.52 / 0.37, 0.9 M 0.94 / 1.14
// and 1.30 / 2.13, 5.6 M 3.2 / 5.2, 12 M 15.4 / 61.7 ms.  Unrelated openings of
// up to 3 plies qualify too: 1000 of depth 4 (0.9 M) 0.41 / 0.29 ms, 100 of
// depth 5 (2.7 M) 0.60 / 0.48, 400 of depth 5 (11 M) 0.97 / 1.30, 30 and 60 of
// depth 6 (24 and 49 M) 1.58 / 1.66 and 1.90 / 2.82 (openings of 4-8 plies did
// not qualify).
constexpr int RELATED_SQUARES = 12;
constexpr double RELATED_MIN_NODES = double(3u << 18);
bool related_roots(const u64 *pos, const uint8_t *depths, u32 n)
{
    if (n < 2 || depths[0] < 4) return false;
    double nodes = n;
    for (int k = 2; k < depths[0]; k++) nodes *= 30.0;
    if (nodes < RELATED_MIN_NODES) return false;
    auto occ = [&](u32 i) {
        const u64 *p = pos + 6ull * i;
        return (p[1] & RANKS2TO7) | p[2] | p[3] | p[4] | p[5];
    };
    const u64 occ0 = occ(0);
    for (u32 i = 1; i < n; i++)
        if (depths[i] != depths[0] || popc(occ(i) ^ occ0) > RELATED_SQUARES) return false;
    return true;
}

int Engine::run_batch_host(const u64 *pos, const uint8_t *depths, u32 n, u64 *out)
{
    ENG_TRY(cudaSetDevice(device));  // the staging buffers and the stream belong to the engine's device
    bool handled = false;
    const int rcSmall = run_small(nullptr, pos, depths, n, nullptr, out, handled);
    if (rcSmall != PERFT_OK || handled) return rcSmall;
    if (n > ioCap) {
        if (ioPos) cudaFree(ioPos);
        if (ioOut) cudaFree(ioOut);
        ioPos = ioOut = nullptr;
        ioCap = 0;
        u32 cap = 1024;
        while (cap < n) cap *= 2;
        ENG_TRY(cudaMalloc(&ioPos, 48ull * cap));
        ENG_TRY(cudaMalloc(&ioOut, 8ull * cap));
        ioCap = cap;
        drop_dd();
    }
    ENG_TRY(cudaMemcpyAsync(ioPos, pos, 48ull * n, cudaMemcpyHostToDevice, stream));
    const int rc = run_batch(ioPos, depths, n, ioOut, false, related_roots(pos, depths, n));
    if (rc != PERFT_OK) return rc;
    ENG_TRY(cudaMemcpyAsync(out, ioOut, 8ull * n, cudaMemcpyDeviceToHost, stream));
    ENG_TRY(cudaStreamSynchronize(stream));
    return PERFT_OK;
}

int Engine::sync_and_check_errors()
{
    ENG_TRY(cudaMemcpyAsync(hPinned + 1, dErr, 4, cudaMemcpyDeviceToHost, stream));
    ENG_TRY(cudaStreamSynchronize(stream));
    const u32 e = (u32)hPinned[1];
    if (e & DERR_BAD_POSITION) return PERFT_ERR_INVALID_ARG;
    if (e) return PERFT_ERR_INTERNAL;
    return PERFT_OK;
}

// Batch without a table, host-driven.  All depth groups share their plies:
// the deepest roots start, the others join the level of their remaining
// depth, so the batch takes one launch per ply (chunked only where a level
// does not fit the arena).  Roots of depth 0 and 1 are answered by
// k_init_roots alone.  With `merge`, levels from the third ply below a root
// on are merged.
int Engine::run_levels(const u64 *dPos, const uint8_t *depths, u32 n, unsigned long long *rootCounts, bool merge)
{
    std::map<int, std::vector<u32>, std::greater<int>> groups;
    for (u32 i = 0; i < n; i++) groups[depths[i]].push_back(i);
    const int dmax = groups.begin()->first;
    std::vector<u32> order;
    order.reserve(n);
    Joiners J;
    J.dPos = dPos;
    u32 *dIds = (u32 *)alloc(4ull * n);
    if (!dIds) return PERFT_ERR_OUT_OF_MEMORY;
    for (auto &g : groups) {
        J.ids[g.first] = dIds + order.size();
        J.n[g.first] = (u32)g.second.size();
        order.insert(order.end(), g.second.begin(), g.second.end());
    }
    ENG_TRY(cudaMemcpyAsync(dIds, order.data(), 4ull * n, cudaMemcpyHostToDevice, stream));
    merge = merge && dmax - 2 >= MERGE_MIN_PLIES;
    if (merge) {
        uint8_t *dDepths = (uint8_t *)alloc(n);
        J.segs = (MergeSeg *)alloc(sizeof(MergeSeg) * (u64)n);
        if (!dDepths || !J.segs) return PERFT_ERR_OUT_OF_MEMORY;
        ENG_TRY(cudaMemcpyAsync(dDepths, depths, n, cudaMemcpyHostToDevice, stream));
        J.depths = dDepths;
        J.maxDepth = dmax;
    }
    // the shallow roots (depth 0, 1) in one scratch level each
    for (int d = 0; d <= 1; d++) {
        if (!J.n[d]) continue;
        const u64 gm = arenaTop;
        DeviceLevel S;
        if (!alloc_level(S, J.n[d])) return PERFT_ERR_OUT_OF_MEMORY;
        const int rc = init_joiners(J, d, S, 0, rootCounts);
        if (rc != PERFT_OK) return rc;
        arenaTop = gm;
    }
    if (dmax < 2) return PERFT_OK;
    DeviceLevel L0;
    if (!alloc_level(L0, J.n[dmax], merge)) return PERFT_ERR_OUT_OF_MEMORY;
    int rc = init_joiners(J, dmax, L0, 0, rootCounts);
    if (rc == PERFT_OK) rc = sync_and_check_errors();
    if (rc == PERFT_OK) rc = process_level(L0, dmax, rootCounts, &J);
    return rc;
}

int Engine::run_batch(const u64 *dPos, const uint8_t *depths, u32 n, u64 *dOut, bool trySmall, bool related)
{
    ENG_TRY(cudaSetDevice(device));
    if (trySmall) {
        bool handled = false;
        const int rc = run_small(dPos, nullptr, depths, n, dOut, nullptr, handled);
        if (rc != PERFT_OK || handled) return rc;
    }
    related = related && mergeEnabled;
    if (!related) {
        bool handled = false;
        const int rc = run_dd(dPos, depths, n, dOut, handled);
        if (rc != PERFT_OK || handled) return rc;
    }
    const u64 mark0 = arenaTop;
    unsigned long long *rootCounts = (unsigned long long *)dOut;
    ENG_TRY(cudaMemsetAsync(rootCounts, 0, 8ull * n, stream));
    ENG_TRY(cudaMemsetAsync(dErr, 0, 4, stream));

    int rc = PERFT_OK;
    if (!tt && !related) {
        rc = run_levels(dPos, depths, n, rootCounts, mergeEnabled);
        // path weights and the merge set cost memory: an arena too small for
        // them still runs what it ran without
        if (rc == PERFT_ERR_OUT_OF_MEMORY && mergeEnabled) {
            arenaTop = mark0;
            ENG_TRY(cudaMemsetAsync(rootCounts, 0, 8ull * n, stream));
            rc = run_levels(dPos, depths, n, rootCounts, false);
        }
    }
    // With a table, or related roots: levels merged over all roots.  Roots are
    // grouped by depth: every node of a level then has the same remaining depth.
    std::map<int, std::vector<u32>, std::greater<int>> groups;
    if (tt || related)
        for (u32 i = 0; i < n; i++) groups[depths[i]].push_back(i);
    for (auto &g : groups) {
        const int depth = g.first;
        const std::vector<u32> &ids = g.second;
        const u64 gm = arenaTop;
        u32 *dIds = (u32 *)alloc(4ull * ids.size());
        DeviceLevel L0;
        if (!dIds || !alloc_level_tt(L0, ids.size())) {
            rc = PERFT_ERR_OUT_OF_MEMORY;
            break;
        }
        ENG_TRY(cudaMemcpyAsync(dIds, ids.data(), 4ull * ids.size(), cudaMemcpyHostToDevice, stream));
        const u32 nb = (u32)((ids.size() + 127) / 128);
        k_init_roots<<<nb, 128, 0, stream>>>(dPos, dIds, (u32)ids.size(), L0.planes, L0.stride, L0.cnt,
                                              L0.root, nullptr, depth, rootCounts, dErr);
        stats.other_launches++;
        ENG_TRY(cudaGetLastError());
        rc = sync_and_check_errors();
        if (rc != PERFT_OK) break;
        if (depth >= 2) rc = process_level_tt(L0, depth, nullptr, rootCounts);
        arenaTop = gm;
        if (rc != PERFT_OK) break;
    }
    arenaTop = mark0;
    if (rc != PERFT_OK) {
        cudaStreamSynchronize(stream);
        // (a linked node takes more memory than a plain one)
        if (rc == PERFT_ERR_OUT_OF_MEMORY && related && !tt) return run_batch(dPos, depths, n, dOut, false, false);
        return rc;
    }
    rc = sync_and_check_errors();
    stats.peak_arena_bytes = std::max<u64>(stats.peak_arena_bytes, arenaPeak);
    return rc;
}

// ================================================================ C ABI glue
Engine g_engine;

}  // namespace

#include "serve.cuh"

namespace pg {
// Shared with host.cpp: run a batch on the process-wide engine (host buffers).
int engine_batch_host(const u64 *pos, const uint8_t *depths, u32 n, u64 *out);
}

int pg::engine_batch_host(const u64 *pos, const uint8_t *depths, u32 n, u64 *out)
{
    Engine &E = g_engine;
    std::lock_guard<std::mutex> lk(E.mu);
    if (!E.ready) return PERFT_ERR_NOT_INITIALIZED;
    if (n == 0) return PERFT_OK;
    for (u32 i = 0; i < n; i++) {
        if (validate_pos48(pos + 6ull * i) != 0) return PERFT_ERR_INVALID_ARG;
        if (depths[i] > 20) return PERFT_ERR_INVALID_ARG;
    }
    return E.run_batch_host(pos, depths, n, out);
}

extern "C" {

void perft_config_default(perft_config *cfg)
{
    if (!cfg) return;
    memset(cfg, 0, sizeof *cfg);
    cfg->device = 0;
    cfg->arena_bytes = 0;
    cfg->sliders_expand = PERFT_SLIDERS_AUTO;
    cfg->sliders_leaf = PERFT_SLIDERS_AUTO;
    cfg->tt_log2_entries = 0;
    cfg->zobrist_seed = 0x5EED0781ULL;
}

int perft_init(const perft_config *cfg)
{
    perft_config c;
    if (cfg) c = *cfg;
    else perft_config_default(&c);
    if (g_server.running) perft_serve_stop();
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (g_engine.ready) g_engine.shutdown();
    return g_engine.init(c);
}

int perft_shutdown(void)
{
    if (g_server.running) perft_serve_stop();
    std::lock_guard<std::mutex> lk(g_engine.mu);
    g_engine.shutdown();
    return PERFT_OK;
}

void perft_serve_config_default(perft_serve_config *cfg)
{
    if (!cfg) return;
    memset(cfg, 0, sizeof *cfg);
    cfg->memory_bytes = 0;
    cfg->step_items = 1ull << 27;
    cfg->max_in_flight = 4096;
    cfg->use_tt = 1;
}

int perft_serve_start(const perft_serve_config *cfg)
{
    perft_serve_config c;
    if (cfg) c = *cfg;
    else perft_serve_config_default(&c);
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (!g_engine.ready) return PERFT_ERR_NOT_INITIALIZED;
    if (g_server.running) return PERFT_ERR_INVALID_ARG;
    const u64 fixed = 256ull << 20;  // slot tables, staging, scratch
    u64 bytes = c.memory_bytes ? c.memory_bytes + fixed : (u64)(g_engine.free_bytes() * 0.9);
    if (bytes > g_engine.free_bytes()) return PERFT_ERR_OUT_OF_MEMORY;
    char *block = g_engine.reserve_block(bytes);
    if (!block) return PERFT_ERR_OUT_OF_MEMORY;
    const int rc = g_server.start(c, block, bytes, g_engine.device_id());
    if (rc != PERFT_OK) g_engine.release_block();
    return rc;
}

int perft_serve_stop(void)
{
    const bool was = g_server.running;
    const int rc = g_server.stop();
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (was && g_engine.ready) g_engine.release_block();
    return rc;
}

int perft_serve_submit(const perft_pos48 *pos, uint32_t depth, uint64_t *ticket)
{
    if (!pos || !ticket) return PERFT_ERR_INVALID_ARG;
    if (!g_server.running) return PERFT_ERR_NOT_INITIALIZED;
    return g_server.submit(pos->bb, depth, ticket);
}

int perft_serve_poll(uint64_t ticket, uint64_t *count, double *latency_s)
{
    return g_server.poll(ticket, count, latency_s, false, 0.0);
}

int perft_serve_wait(uint64_t ticket, double timeout_s, uint64_t *count, double *latency_s)
{
    return g_server.poll(ticket, count, latency_s, true, timeout_s);
}

int perft_serve_get_stats(perft_serve_stats *out)
{
    if (!out) return PERFT_ERR_INVALID_ARG;
    memset(out, 0, sizeof *out);
    g_server.get_stats(out);
    return PERFT_OK;
}

const char *perft_status_string(int status)
{
    switch (status) {
    case PERFT_OK: return "ok";
    case PERFT_ERR_INVALID_ARG: return "invalid argument";
    case PERFT_ERR_NOT_INITIALIZED: return "engine not initialized (call perft_init)";
    case PERFT_ERR_CUDA: return "CUDA error";
    case PERFT_ERR_OUT_OF_MEMORY: return "out of device memory";
    case PERFT_ERR_INTERNAL: return "internal consistency check failed on the device";
    case PERFT_ERR_BAD_FEN: return "malformed FEN";
    case PERFT_ERR_NO_DEVICE: return "no CUDA device";
    case PERFT_ERR_ILLEGAL_MOVE: return "illegal move";
    case PERFT_ERR_TIMEOUT: return "timed out";
    case PERFT_ERR_NOT_FOUND: return "not found";
    case PERFT_ERR_IO: return "file I/O error";
    case PERFT_ERR_OVERFLOW: return "count does not fit 64 bits";
    default: return "unknown status";
    }
}

int perft(const perft_pos48 *pos, uint32_t depth, uint64_t *out)
{
    if (!pos || !out || depth > 255) return PERFT_ERR_INVALID_ARG;
    uint8_t d = (uint8_t)depth;
    return pg::engine_batch_host(pos->bb, &d, 1, out);
}

int perft_batch(const perft_pos48 *pos, const uint8_t *depths, uint32_t n, uint64_t *out)
{
    if ((!pos || !depths || !out) && n) return PERFT_ERR_INVALID_ARG;
    return pg::engine_batch_host(pos ? pos->bb : nullptr, depths, n, out);
}

int perft_batch_device(const perft_pos48 *d_pos, const uint8_t *depths, uint32_t n, uint64_t *d_out)
{
    if ((!d_pos || !depths || !d_out) && n) return PERFT_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (!g_engine.ready) return PERFT_ERR_NOT_INITIALIZED;
    for (u32 i = 0; i < n; i++)
        if (depths[i] > 20) return PERFT_ERR_INVALID_ARG;
    if (n == 0) return PERFT_OK;
    return g_engine.run_batch(d_pos->bb, depths, n, d_out);
}

int perft_get_stats(perft_stats *out)
{
    if (!out) return PERFT_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (g_engine.ready) g_engine.read_tt_stats();
    *out = g_engine.stats;
    return PERFT_OK;
}

int perft_get_tuning(perft_tune_entry *out, uint32_t cap, uint32_t *n)
{
    if (!n || (!out && cap)) return PERFT_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (!g_engine.ready) return PERFT_ERR_NOT_INITIALIZED;
    uint32_t k = 0;
    auto put = [&](int leaf, int r) {
        const Engine::TuneCfg &c = g_engine.tuneTab[leaf ? MODE_LEAF : MODE_EXPAND][r];
        if (k < cap) out[k] = perft_tune_entry{leaf, r, c.sv, c.cap, c.ctas, c.ms};
        k++;
    };
    put(1, 2);
    for (int r = 3; r <= g_engine.tunedMaxR; r++) put(0, r);
    *n = k;
    return k <= cap ? PERFT_OK : PERFT_ERR_INVALID_ARG;
}

int perft_tt_clear(void)
{
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (!g_engine.ready) return PERFT_ERR_NOT_INITIALIZED;
    return g_engine.tt_clear();
}

int perft_reset_stats(void)
{
    std::lock_guard<std::mutex> lk(g_engine.mu);
    if (g_engine.ready) g_engine.zero_tt_stats();
    perft_stats keep = g_engine.stats;
    memset(&g_engine.stats, 0, sizeof g_engine.stats);
    g_engine.stats.sliders_expand = keep.sliders_expand;
    g_engine.stats.sliders_leaf = keep.sliders_leaf;
    g_engine.stats.arena_bytes = keep.arena_bytes;
    return PERFT_OK;
}

}  // extern "C"

// ======================================================= allocation-free entry
// perft_batch_noalloc: the batched perft for callers that cannot allocate
// device memory — processes whose HBM is already reserved by another
// allocator (a serving framework or torch's caching allocator holding the
// device), and latency-critical callers for which cudaMalloc's implicit
// device-wide synchronisation is unacceptable.  It runs the interior and
// count-only kernels of perft_batch_device, but every level buffer, scan, tile
// index and counter lives in one fixed scratch array compiled into this
// library, so the call allocates nothing.  The scratch has no room for merge
// sets: equal nodes are not merged, every move path is searched.  Trees whose levels do not fit the scratch are refused
// (PERFT_ERR_OUT_OF_MEMORY); the arena engine handles those by chunking.
//
// The scratch is a file-scope __device__ array: every GPU that loads this
// library holds NOALLOC_SCRATCH_BYTES of it until the process exits.  All
// calls on a device share it and it keeps the previous call's contents, so
// each call clears its counters and outputs first.  Two calls whose GPU work
// overlapped would corrupt each other: this entry point takes a process-wide
// lock and waits for its stream before returning, on error paths too, so its
// own calls never overlap.  The first call on a device uploads the
// move-generator tables and looks up the scratch address
// (cudaGetSymbolAddress) with that device current; make that first call
// before any stream capture.
static __device__ __align__(256) unsigned char g_noallocScratch[PERFT_NOALLOC_SCRATCH_BYTES];

namespace {

constexpr int NOALLOC_MAX_DEVICES = 64;

struct NoallocDevice {
    bool ready = false;
    unsigned char *scratch = nullptr;  // device address of g_noallocScratch
    int gridLeaf = 0, gridExpand = 0;
};

std::mutex g_noallocMu;
NoallocDevice g_noallocDev[NOALLOC_MAX_DEVICES];

// Writes, in order, the indices of the roots whose depth equals `depth`.
__global__ void __launch_bounds__(1024) k_noalloc_group_ids(const uint8_t *__restrict__ depths, u32 n,
                                                            int depth, u32 *__restrict__ ids,
                                                            u32 *__restrict__ count)
{
    __shared__ int sw[32];
    u32 base = 0;
    for (u32 c0 = 0; c0 < n; c0 += 1024) {
        const u32 i = c0 + threadIdx.x;
        const bool hit = i < n && depths[i] == depth;
        int tot = 0;
        const int r = block_excl_count<1024>(hit, sw, tot);
        if (hit) ids[base + r] = i;
        base += (u32)tot;
    }
    if (threadIdx.x == 0) *count = base;
}

// Looks up the scratch address with `dev` current, on every call: the lookup
// allocates nothing and is cheap.  If the address differs from the one cached
// (first call on the device, or the device's primary context was destroyed and
// created again, e.g. by cudaDeviceReset), the move tables are uploaded into
// the current context before the address is trusted.
int noalloc_setup(int dev)
{
    NoallocDevice &D = g_noallocDev[dev];
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noallocScratch) != cudaSuccess || p == nullptr) return PERFT_ERR_CUDA;
    if (D.ready && D.scratch == (unsigned char *)p) return PERFT_OK;
    D.ready = false;
    build_tables();
    if (cudaMemcpyToSymbol(d_tables, &h_tables, sizeof(Tables)) != cudaSuccess) return PERFT_ERR_CUDA;
    if (cudaMemcpyToSymbol(d_magic, h_magic, sizeof(h_magic)) != cudaSuccess) return PERFT_ERR_CUDA;
    u32 pow2[32];
    for (int k = 0; k < 32; k++) pow2[k] = 1u << k;
    if (cudaMemcpyToSymbol(c_pow2, pow2, sizeof pow2) != cudaSuccess) return PERFT_ERR_CUDA;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return PERFT_ERR_CUDA;
    D.scratch = (unsigned char *)p;
    D.gridLeaf = occupancy_grid<MODE_LEAF, SV_KOGGE>(prop.multiProcessorCount);
    D.gridExpand = occupancy_grid<MODE_EXPAND, SV_KOGGE>(prop.multiProcessorCount);
    D.ready = true;
    return PERFT_OK;
}

// One call's bump allocator over the static scratch, and the level loop
// without chunking.
struct NoallocRun {
    unsigned char *base;
    u64 top = 0;
    cudaStream_t st;
    u32 *counter = nullptr, *err = nullptr;
    int gridLeaf = 0, gridExpand = 0;

    void *take(u64 bytes)
    {
        const u64 a = (top + 255) & ~255ULL;
        if (a + bytes > PERFT_NOALLOC_SCRATCH_BYTES) return nullptr;
        top = a + bytes;
        return base + a;
    }

    bool level(DeviceLevel &L, u64 n)
    {
        L.n = n;
        L.stride = (n + 31) & ~31ULL;
        L.planes = (u64 *)take(6 * 8 * L.stride);
        L.cnt = (u32 *)take(4 * L.stride);
        L.root = (u32 *)take(4 * L.stride);
        return L.planes && L.cnt && L.root;
    }

    int read_u64(const u64 *src, u64 &v)
    {
        if (cudaMemcpyAsync(&v, src, 8, cudaMemcpyDeviceToHost, st) != cudaSuccess) return PERFT_ERR_CUDA;
        return cudaStreamSynchronize(st) == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
    }

    int scan(const u32 *cnt, u64 n, bool tiles, u64 *&scanOut, u32 *&tileFirst, u64 &total)
    {
        const u64 nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
        const u64 maxTiles = (n * MAX_LEGAL_MOVES + TILE_CAP - 1) / TILE_CAP + 1;
        scanOut = (u64 *)take(8 * (n + 1));
        tileFirst = tiles ? (u32 *)take(4 * maxTiles) : nullptr;
        const u64 mark = top;
        ScanSums *bsum = (ScanSums *)take(sizeof(ScanSums) * (nb + 1));
        if (!scanOut || (tiles && !tileFirst) || !bsum) return PERFT_ERR_OUT_OF_MEMORY;
        u64 *totals = (u64 *)(bsum + nb);
        k_scan_reduce<<<(unsigned)nb, SCAN_NT, 0, st>>>(cnt, n, bsum);
        k_scan_top<<<1, SCAN_TOP_NT, 0, st>>>(bsum, nb, totals);
        if (cudaGetLastError() != cudaSuccess) return PERFT_ERR_CUDA;
        const int rc = read_u64(totals, total);
        if (rc != PERFT_OK) return rc;
        const u64 nTiles = (total + TILE_CAP - 1) / TILE_CAP;
        if (tiles && nTiles > maxTiles) {  // more moves than any game's: an index of its own size
            tileFirst = (u32 *)take(4 * nTiles);
            if (!tileFirst) return PERFT_ERR_OUT_OF_MEMORY;
        } else {
            top = mark;  // the block sums are done with before the next level is written (stream order)
        }
        k_scan_apply<false><<<(unsigned)nb, SCAN_NT, 0, st>>>(cnt, n, bsum, totals, scanOut, nullptr,
                                                                        tileFirst, TILE_CAP_LOG2);
        return cudaGetLastError() == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
    }

    int tile(int mode, const DeviceLevel &par, const u64 *pscan, const u32 *tileFirst, u64 total,
             DeviceLevel *ch, bool uncounted, unsigned long long *rootCounts)
    {
        TileParams P;
        memset(&P, 0, sizeof P);
        P.ppl = par.planes;
        P.pstride = par.stride;
        P.pscan = pscan;
        P.proot = par.root;
        P.nParents = par.n;
        P.tileFirst = tileFirst;
        P.itemBase = 0;
        P.itemEnd = total;
        P.capLog2 = TILE_CAP_LOG2;
        P.tileCounter = counter;
        if (ch) {
            P.cpl = ch->planes;
            P.cstride = ch->stride;
            P.ccnt = ch->cnt;
            P.croot = ch->root;
        }
        P.rootCounts = rootCounts;
        P.uncounted = uncounted;
        P.err = err;
        const u64 nTiles = (total + TILE_CAP - 1) / TILE_CAP;
        if (cudaMemsetAsync(counter, 0, 4, st) != cudaSuccess) return PERFT_ERR_CUDA;
        if (mode == MODE_LEAF)
            launch_tile_variant<MODE_LEAF>(SV_KOGGE, (int)std::min<u64>(gridLeaf, leaf_units(par.n)), st, P);
        else
            launch_tile_variant<MODE_EXPAND>(SV_KOGGE, (int)std::min<u64>(gridExpand, nTiles), st, P);
        return cudaGetLastError() == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
    }

    int process(const DeviceLevel &L, int remaining, unsigned long long *rootCounts)
    {
        if (L.n == 0) return PERFT_OK;
        u64 *pscan = nullptr;
        u32 *tileFirst = nullptr;
        u64 total = 0;
        int rc = scan(L.cnt, L.n, remaining > 2, pscan, tileFirst, total);
        if (rc != PERFT_OK || total == 0) return rc;
        if (remaining == 2) return tile(MODE_LEAF, L, pscan, tileFirst, total, nullptr, false, rootCounts);
        const u64 mark = top;
        DeviceLevel C;
        if (!level(C, total)) return PERFT_ERR_OUT_OF_MEMORY;
        rc = tile(MODE_EXPAND, L, pscan, tileFirst, total, &C, remaining == 3, nullptr);
        if (rc == PERFT_OK) rc = process(C, remaining - 1, rootCounts);
        top = mark;
        return rc;
    }
};

}  // namespace

extern "C" int perft_batch_noalloc(const perft_pos48 *d_pos, const uint8_t *depths, uint32_t n,
                                   uint64_t *d_out, void *stream)
{
    if ((!d_pos || !depths || !d_out) && n) return PERFT_ERR_INVALID_ARG;
    for (uint32_t i = 0; i < n; i++)
        if (depths[i] > 20) return PERFT_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lk(g_noallocMu);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return PERFT_ERR_NO_DEVICE;
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return PERFT_ERR_INVALID_ARG;
    int rc = noalloc_setup(dev);
    if (rc != PERFT_OK || n == 0) return rc;

    NoallocRun R;
    R.base = g_noallocDev[dev].scratch;
    R.st = (cudaStream_t)stream;
    R.gridLeaf = g_noallocDev[dev].gridLeaf;
    R.gridExpand = g_noallocDev[dev].gridExpand;
    u32 *words = (u32 *)R.take(12);  // tile cursor, error flags, group size
    R.counter = words;
    R.err = words + 1;
    u32 *dIds = (u32 *)R.take(4ull * n);
    uint8_t *dDepths = (uint8_t *)R.take(n);
    u32 *dGroupCount = words + 2;
    if (!words || !dIds || !dDepths) return PERFT_ERR_OUT_OF_MEMORY;

    // From the first queued operation on, every return goes through the
    // stream synchronisation at the end, so the call never returns with work
    // of its own still queued on the shared scratch (a failed call included).
    unsigned long long *rootCounts = (unsigned long long *)d_out;
    if (cudaMemsetAsync(R.err, 0, 4, R.st) != cudaSuccess ||
        cudaMemsetAsync(rootCounts, 0, 8ull * n, R.st) != cudaSuccess ||
        cudaMemcpyAsync(dDepths, depths, n, cudaMemcpyHostToDevice, R.st) != cudaSuccess)
        rc = PERFT_ERR_CUDA;

    // Group roots by depth without host allocation: the depths go to the
    // scratch and a kernel compacts the ids of one depth group in order.
    u32 perDepth[21] = {0};
    for (u32 i = 0; i < n; i++) perDepth[depths[i]]++;
    for (int depth = 20; depth >= 0 && rc == PERFT_OK; depth--) {
        const u32 cnt = perDepth[depth];
        if (!cnt) continue;
        const u64 mark = R.top;
        DeviceLevel L0;
        if (!R.level(L0, cnt)) {
            rc = PERFT_ERR_OUT_OF_MEMORY;
            break;
        }
        k_noalloc_group_ids<<<1, 1024, 0, R.st>>>(dDepths, n, depth, dIds, dGroupCount);
        k_init_roots<<<(cnt + 127) / 128, 128, 0, R.st>>>(d_pos->bb, dIds, cnt, L0.planes, L0.stride,
                                                           L0.cnt, L0.root, nullptr, depth, rootCounts, R.err);
        if (cudaGetLastError() != cudaSuccess) {
            rc = PERFT_ERR_CUDA;
            break;
        }
        if (depth >= 2) rc = R.process(L0, depth, rootCounts);
        R.top = mark;
    }
    u32 e = 0;
    const bool readOk = cudaMemcpyAsync(&e, R.err, 4, cudaMemcpyDeviceToHost, R.st) == cudaSuccess;
    const bool syncOk = cudaStreamSynchronize(R.st) == cudaSuccess;
    if (rc != PERFT_OK) return rc;
    if (!readOk || !syncOk) return PERFT_ERR_CUDA;
    if (e & DERR_BAD_POSITION) return PERFT_ERR_INVALID_ARG;
    return e ? PERFT_ERR_INTERNAL : PERFT_OK;
}
