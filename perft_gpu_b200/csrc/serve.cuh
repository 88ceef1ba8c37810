// Continuous-batching perft server (included by engine.cu: it drives the
// same kernels).
//
// Queries of mixed depth arrive at any time.  Each admitted query owns a
// slot; its frontier lives in HBM as level buffers, kept in pools by
// remaining depth, and the levels of different queries with the same
// remaining depth are advanced by the same kernels.  One scheduler iteration:
//   1. admit queued queries while slots are free and the predicted
//      level-buffer memory of all admitted queries fits the budget;
//   2. advance every pool, the count-only last ply first, each level by at
//      most `step_items` (tile-aligned; the count-only ply by as many parents
//      as have about that many moves, see advance), so a large level never
//      blocks the small levels of newer queries for more than one step;
//   3. read back the per-query pending-node counters (maintained on the
//      device by the tracking tile kernels) and complete every query whose
//      counter reached zero.
// Work of different queries therefore overlaps on the device, queries that
// arrive while others run join at the next iteration, and no query waits for
// another to finish.  A query's count is the same alone or in the mix: it
// is a sum of exact per-item counts, only the grouping into launches varies.
//
// Transposition table: with an engine table and use_tt, every level two or
// three plies above the leaves (remaining depth 2 or 3) is hashed and probed
// before its scan, exactly as the engine's own table levels are: identical
// nodes of the level are searched once (k_merge_linked), and the others that
// hit the table take the stored count and generate nothing (k_tt_probe).
// Levels further above the leaves are not merged then; without a table every
// level is, within each query (merge_level).  Table levels' counts flow up per
// node, not per query:
//   * a remaining-depth-3 level expands without pending-count tracking; each
//     child level (remaining depth 2) it produces sums its leaf ply per node
//     and, when done, stores its nodes and adds each node's count into its
//     parent's sum (the engine's k_tt_finish);
//   * once a remaining-depth-3 level is fully expanded and all its child
//     levels are done, it is finished like a remaining-depth-2 level of a
//     depth-2 query: its searched nodes are stored, duplicates take their
//     owner's count, and every node's count goes to its query, whose pending
//     count drops by one per node (k_serve_tt_finish).
// The table lives in the engine for the life of the process, so it is shared
// by all queries and keeps its entries across queries.
#pragma once

#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <thread>
#include <unordered_map>

namespace {

constexpr u32 SERVE_MAX_SLOTS = 1u << 16;
constexpr int SERVE_MAX_R = 21;
// Memory of the server's block that no level of items takes: new queries' roots
// and the copies of their positions (under 180 bytes for each of 65536), and
// room for the free ranges being split.
constexpr u64 SERVE_MARGIN = 16ull << 20;
constexpr u64 SERVE_MOVES_PER_PARENT = 32;  // in round numbers: step_items in parents of the count-only ply

__global__ void k_serve_admit(const u64 *__restrict__ stagePos, const u32 *__restrict__ slots,
                              const uint8_t *__restrict__ depths, u32 n, u64 *__restrict__ posBySlot,
                              unsigned long long *__restrict__ pending, unsigned long long *__restrict__ counts)
{
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const u32 s = slots[i];
#pragma unroll
    for (int k = 0; k < 6; k++) posBySlot[6ull * s + k] = stagePos[6ull * i + k];
    counts[s] = 0;
    pending[s] = depths[i] >= 2 ? 1ull : 0ull;
}

// Parents without items (no legal move, or merged into an equal node) end
// their branch at scan time.  One atomic per warp and query: a merged level
// has hundreds of thousands of them.
__global__ void k_serve_zero_parents(const u32 *__restrict__ cnt, const u32 *__restrict__ root, u64 n,
                                     unsigned long long *pending)
{
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const bool zero = i < n && cnt[i] == 0;
    const u32 key = zero ? root[i] : 0xFFFFFFFFu;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (zero && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
        atomicAdd(&pending[key], (unsigned long long)(-(long long)__popc(peers)));
}

struct ServeQuery {
    u64 ticket = 0;
    u64 pos[6];
    u32 depth = 0;
    int slot = -1;
    int state = 0;  // 0 queued, 1 running, 2 done
    double tSubmit = 0, tAdmit = 0, tDone = 0;
    u64 predicted = 0;
    u64 result = 0;
};

// Last step of a table level: owners (and nodes not de-duplicated) store
// their subtree count, duplicates take their owner's, and every node's count
// goes to its query with the node's pending mark removed (warp-aggregated per
// run of equal query slot: the nodes of a level are ordered by query).
__global__ void __launch_bounds__(256) k_serve_tt_finish(u64 n, const u64 *__restrict__ hash,
                                                         const u64 *__restrict__ hash2,
                                                         const unsigned long long *__restrict__ acc,
                                                         const u32 *__restrict__ alias, const u32 *__restrict__ slot,
                                                         unsigned long long *counts, unsigned long long *pending,
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
            v = acc[a];  // the owner's subtree finished with this level's last launch
        } else if (a != ALIAS_HIT) {
            tt[hash[i] & ttMask] = make_ulonglong2(hash2[i] ^ v, v);
            stored = true;
        }
        key = slot[i];
    }
    count_stat(&ts->stores, stored);
    // a count three plies deep is below 218^3 < 2^24, so 32 of them sum in 32 bits
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const unsigned long long sum = __reduce_add_sync(peers, (unsigned)v);
    if (i < n && lane == __ffs(peers) - 1) {
        atomicAdd(&counts[key], sum);
        atomicAdd(&pending[key], (unsigned long long)(-(long long)__popc(peers)));
    }
}

struct ServeLevel {
    DeviceLevel L;
    int r = 0;
    int depth = 0;  // of its queries (a level's queries all have one depth)
    bool scanned = false;
    bool tt = false;  // a table level: per-node sums, finished by k_serve_tt_finish
    // a remaining-depth-2 level expanded from a table level of remaining depth
    // 3: its root array holds parent indices into that level, its counts go
    // into the parent's sums (k_tt_finish)
    struct ServeLevel *parent = nullptr;
    int outstanding = 0;  // (table levels of remaining depth 3) child levels not yet finished
    std::vector<std::pair<u64, u64>> ttMem;  // its hashes, sums and aliases
    u64 *pscan = nullptr;
    u32 *live = nullptr;  // merged and table levels: the nodes with items
    u32 *liveMem = nullptr;  // where they are listed, should the level be merged
    u32 *tileFirst = nullptr;
    // until the level is scanned: the scan's block sums, and a table level's merge set
    ScanSums *bsum = nullptr;
    unsigned long long *set = nullptr;
    std::vector<std::pair<u64, u64>> scanMem;
    u64 nParents = 0, total = 0, next = 0;
    std::vector<std::pair<u64, u64>> mem;  // (offset, bytes) in the server block
};

double now_s()
{
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

class Server {
public:
    int start(const perft_serve_config &cfg, char *block, u64 bytes, int device);
    int stop();
    int submit(const u64 pos[6], u32 depth, u64 *ticket);
    int poll(u64 ticket, u64 *count, double *latency, bool wait, double timeoutS);
    void get_stats(perft_serve_stats *out);
    bool running = false;
    char *blockBase = nullptr;

private:
    // ---- device-memory first-fit allocator over the server's arena block
    u64 blockBytes = 0;
    std::map<u64, u64> freeRanges;  // offset -> size
    u64 inUse = 0, peakInUse = 0;
    void *take(u64 bytes, std::vector<std::pair<u64, u64>> &owner);
    void give_back(std::vector<std::pair<u64, u64>> &owner);

    void loop();
    int admit();
    int advance();
    int complete();
    template <class Take>
    bool level_memory(ServeLevel &S, u64 n, bool weighted, Take take);
    bool take_level(ServeLevel &S, u64 n, bool weighted);
    u64 reserve_below(int r);
    bool table_level(int r) const { return tt && (r == 2 || r == 3); }
    int scan_level(ServeLevel &S);
    int launch(int mode, ServeLevel &S, u64 lo, u64 hi, DeviceLevel *child);
    int probe_level(ServeLevel &S);
    int merge_level(ServeLevel &S);
    int finish_level(ServeLevel &S);
    int retire(ServeLevel *S);
    std::vector<ServeLevel *> waiting;  // table levels fully expanded, waiting for their child levels

    std::thread worker;
    std::mutex mu;
    std::condition_variable cvWork, cvDone;
    bool stopping = false;
    std::deque<ServeQuery *> queue;
    std::unordered_map<u64, ServeQuery *> byTicket;
    std::vector<ServeQuery *> bySlot;
    std::vector<u32> freeSlots;
    u64 nextTicket = 1;

    int dev = 0;
    cudaStream_t st = nullptr;
    u32 *dErr = nullptr, *dCounter = nullptr;
    u64 *posBySlot = nullptr;
    unsigned long long *pending = nullptr, *counts = nullptr;
    MergeSeg *segs = nullptr;  // per slot: its nodes in the level being merged
    bool mergeEnabled = true;
    u64 *hostPending = nullptr, *hostCounts = nullptr, *hostTotal = nullptr;  // pinned
    u64 *stagePos = nullptr;   // pinned
    u32 *stageSlots = nullptr; // pinned
    uint8_t *stageDepths = nullptr;
    std::vector<std::pair<u64, u64>> fixedMem;
    std::vector<ServeLevel *> pools[SERVE_MAX_R + 1];
    u64 budget = 0, reserved = 0, stepItems = 0;
    u32 maxInFlight = 0, inFlight = 0, maxSlotUsed = 0;
    int gridLeaf = 0, gridExpand = 0, gridLeafAcc = 0, gridExpandTT = 0;
    bool leafSplit = false;
    unsigned nsm = 1;
    // the engine's transposition table, when the server uses it
    ulonglong2 *tt = nullptr;
    u64 ttMask = 0, ttKeyMask = ~0ULL;
    TTStats *dTTStats = nullptr;
    TTStats *hostTTStats = nullptr;  // pinned
    int idleIterations = 0;
    // statistics
    u64 submitted = 0, completed = 0, iterations = 0, launches = 0, admittedBatches = 0;
    int lastError = PERFT_OK;
};

void *Server::take(u64 bytes, std::vector<std::pair<u64, u64>> &owner)
{
    bytes = (bytes + 255) & ~255ULL;
    for (auto it = freeRanges.begin(); it != freeRanges.end(); ++it) {
        if (it->second < bytes) continue;
        const u64 off = it->first, rest = it->second - bytes;
        freeRanges.erase(it);
        if (rest) freeRanges[off + bytes] = rest;
        owner.push_back({off, bytes});
        inUse += bytes;
        peakInUse = std::max(peakInUse, inUse);
        return blockBase + off;
    }
    return nullptr;
}

// Returns every range of `owner`; later launches on the same stream may
// reuse it, which stream order makes safe.
void Server::give_back(std::vector<std::pair<u64, u64>> &owner)
{
    for (auto &r : owner) {
        u64 off = r.first, size = r.second;
        inUse -= size;
        auto nx = freeRanges.lower_bound(off);
        if (nx != freeRanges.end() && off + size == nx->first) {
            size += nx->second;
            nx = freeRanges.erase(nx);
        }
        if (nx != freeRanges.begin()) {
            auto pv = std::prev(nx);
            if (pv->first + pv->second == off) {
                pv->second += size;
                continue;
            }
        }
        freeRanges[off] = size;
    }
    owner.clear();
}

// Everything that a level with n nodes needs until its items are taken from
// it, each piece through take(bytes, owner): its nodes, the scan's arrays, and
// a table level's hashes, sums and merge set.  Taken together when the level
// is made, so that a level that exists can always be scanned.
template <class Take>
bool Server::level_memory(ServeLevel &S, u64 n, bool weighted, Take take)
{
    const u64 nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    const bool table = table_level(S.r), merges = mergeEnabled && !tt && S.r + MERGE_MIN_PLIES <= S.depth;
    S.L.n = n;
    S.L.stride = (n + 31) & ~31ULL;
    bool ok = (S.L.planes = (u64 *)take(48 * S.L.stride, S.mem)) && (S.L.cnt = (u32 *)take(4 * S.L.stride, S.mem)) &&
              (S.L.root = (u32 *)take(4 * S.L.stride, S.mem)) && (S.pscan = (u64 *)take(8 * (n + 1), S.mem)) &&
              (S.bsum = (ScanSums *)take(sizeof(ScanSums) * (nb + 1), S.scanMem));
    if (ok && weighted) ok = (S.L.weight = (unsigned long long *)take(8 * S.L.stride, S.mem));
    if (ok && (table || merges)) ok = (S.liveMem = (u32 *)take(4 * n, S.mem));
    if (ok && S.r > 2) ok = (S.tileFirst = (u32 *)take(4 * tile_index_len(n), S.mem));  // (the count-only ply has no tiles)
    if (ok && table)
        ok = (S.L.hash = (u64 *)take(8 * S.L.stride, S.ttMem)) && (S.L.hash2 = (u64 *)take(8 * S.L.stride, S.ttMem)) &&
             (S.L.acc = (unsigned long long *)take(8 * S.L.stride, S.ttMem)) &&
             (S.L.alias = (u32 *)take(4 * S.L.stride, S.ttMem)) &&
             (S.set = (unsigned long long *)take(8 * MERGE_SLOTS * n, S.scanMem));
    return ok;
}

bool Server::take_level(ServeLevel &S, u64 n, bool weighted)
{
    if (level_memory(S, n, weighted, [this](u64 b, std::vector<std::pair<u64, u64>> &o) { return take(b, o); }))
        return true;
    give_back(S.mem);
    give_back(S.ttMem);
    give_back(S.scanMem);
    return false;
}

// What must stay free when a level r plies above the leaves has been made: a
// smallest step of items for each ply below it.  Every level of items leaves
// this much, so the level nearest the leaves always finds memory for its next
// step, whatever else is admitted: a small budget makes work wait, and never
// stops it.  Without this rule 13 of 145 combinations of a budget of 1 MB to
// 2 GB and queries of depths 3-7 ended in advance()'s out-of-memory error, and
// 60 with a table; with it none, at the same times where memory is ample.
u64 Server::reserve_below(int r)
{
    u64 bytes = SERVE_MARGIN;
    for (int k = 2; k < r; k++) {
        ServeLevel S;
        S.r = k;
        S.depth = SERVE_MAX_R;
        auto add = [&bytes](u64 b, std::vector<std::pair<u64, u64>> &) {
            bytes += (b + 255) & ~255ULL;
            return (void *)&bytes;  // (only counted)
        };
        level_memory(S, TILE_CAP, mergeEnabled && !tt, add);
    }
    return bytes;
}

int Server::start(const perft_serve_config &cfg, char *block, u64 bytes, int device)
{
    dev = device;
    blockBase = block;
    blockBytes = bytes;
    freeRanges.clear();
    freeRanges[0] = bytes;
    inUse = peakInUse = 0;
    stepItems = cfg.step_items ? ((cfg.step_items + TILE_CAP - 1) & ~(u64)(TILE_CAP - 1)) : (1ull << 27);
    maxInFlight = cfg.max_in_flight ? std::min(cfg.max_in_flight, SERVE_MAX_SLOTS) : 4096;
    if (cudaSetDevice(dev) != cudaSuccess) return PERFT_ERR_CUDA;
    if (cudaStreamCreate(&st) != cudaSuccess) return PERFT_ERR_CUDA;
    posBySlot = (u64 *)take(48ull * SERVE_MAX_SLOTS, fixedMem);
    pending = (unsigned long long *)take(8ull * SERVE_MAX_SLOTS, fixedMem);
    counts = (unsigned long long *)take(8ull * SERVE_MAX_SLOTS, fixedMem);
    segs = (MergeSeg *)take(sizeof(MergeSeg) * SERVE_MAX_SLOTS, fixedMem);
    mergeEnabled = g_engine.merge_enabled();
    dCounter = (u32 *)take(256, fixedMem);
    dErr = (u32 *)take(256, fixedMem);
    dTTStats = (TTStats *)take(256, fixedMem);
    if (!posBySlot || !pending || !counts || !segs || !dCounter || !dErr || !dTTStats) return PERFT_ERR_OUT_OF_MEMORY;
    if (cudaMemsetAsync(dErr, 0, 4, st) != cudaSuccess) return PERFT_ERR_CUDA;
    if (cudaMemsetAsync(dTTStats, 0, sizeof(TTStats), st) != cudaSuccess) return PERFT_ERR_CUDA;
    {
        const Engine::TTView v = g_engine.tt_view();
        tt = cfg.use_tt ? v.table : nullptr;
        ttMask = v.mask;
        ttKeyMask = v.keyMask;
    }
    budget = std::min<u64>(cfg.memory_bytes ? cfg.memory_bytes : bytes, blockBytes - inUse);
    if (cudaMallocHost(&hostPending, 8ull * SERVE_MAX_SLOTS) != cudaSuccess ||
        cudaMallocHost(&hostCounts, 8ull * SERVE_MAX_SLOTS) != cudaSuccess ||
        cudaMallocHost(&hostTotal, 64) != cudaSuccess ||
        cudaMallocHost(&stagePos, 48ull * SERVE_MAX_SLOTS) != cudaSuccess ||
        cudaMallocHost(&stageSlots, 4ull * SERVE_MAX_SLOTS) != cudaSuccess ||
        cudaMallocHost(&stageDepths, SERVE_MAX_SLOTS) != cudaSuccess ||
        cudaMallocHost(&hostTTStats, sizeof(TTStats)) != cudaSuccess)
        return PERFT_ERR_OUT_OF_MEMORY;
    memset(hostTTStats, 0, sizeof(TTStats));
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return PERFT_ERR_CUDA;
    nsm = (unsigned)prop.multiProcessorCount;
    // the count-only ply follows the engine's tuned leaf variant when it is
    // the split-shift Kogge-Stone one; every other choice uses plain Kogge-Stone
    leafSplit = g_engine.leaf_sliders() == SV_KOGGE_SPLIT;
    gridLeaf = leafSplit ? occupancy_grid<MODE_LEAF, SV_KOGGE_SPLIT, true>(prop.multiProcessorCount)
                         : occupancy_grid<MODE_LEAF, SV_KOGGE, true>(prop.multiProcessorCount);
    gridExpand = occupancy_grid<MODE_EXPAND, SV_KOGGE, true>(prop.multiProcessorCount);
    // table levels' last ply: the engine's per-node-sum leaf kernel
    gridLeafAcc = leafSplit ? occupancy_grid<MODE_LEAF, SV_KOGGE_SPLIT>(prop.multiProcessorCount)
                            : occupancy_grid<MODE_LEAF, SV_KOGGE>(prop.multiProcessorCount);
    gridExpandTT = occupancy_grid<MODE_EXPAND, SV_KOGGE>(prop.multiProcessorCount);
    bySlot.assign(SERVE_MAX_SLOTS, nullptr);
    freeSlots.clear();
    for (u32 s = SERVE_MAX_SLOTS; s-- > 0;) freeSlots.push_back(s);
    submitted = completed = iterations = launches = admittedBatches = 0;
    reserved = 0;
    inFlight = 0;
    maxSlotUsed = 0;
    stopping = false;
    running = true;
    worker = std::thread([this] { loop(); });
    return PERFT_OK;
}

int Server::stop()
{
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!running) return PERFT_OK;
        stopping = true;
    }
    cvWork.notify_all();
    worker.join();
    cudaSetDevice(dev);
    cudaStreamSynchronize(st);
    for (int r = 0; r <= SERVE_MAX_R; r++) {
        for (ServeLevel *S : pools[r]) delete S;
        pools[r].clear();
    }
    for (ServeLevel *S : waiting) delete S;
    waiting.clear();
    for (auto &kv : byTicket) delete kv.second;
    byTicket.clear();
    queue.clear();
    cudaFreeHost(hostPending);
    cudaFreeHost(hostCounts);
    cudaFreeHost(hostTotal);
    cudaFreeHost(stagePos);
    cudaFreeHost(stageSlots);
    cudaFreeHost(stageDepths);
    cudaFreeHost(hostTTStats);
    cudaStreamDestroy(st);
    running = false;
    cvDone.notify_all();
    return PERFT_OK;
}

int Server::submit(const u64 pos[6], u32 depth, u64 *ticket)
{
    if (validate_pos48(pos) != 0 || depth > 20) return PERFT_ERR_INVALID_ARG;
    ServeQuery *q = new ServeQuery();
    memcpy(q->pos, pos, 48);
    q->depth = depth;
    q->tSubmit = now_s();
    // predicted peak frontier: root branching ^ (depth - 2) nodes of the last
    // materialised ply, 65 bytes each, with a safety margin that also covers a
    // merged level's weights, list and set (28 bytes a node, of 0.6 times the
    // nodes).  It decides how many queries run at once; a query that takes
    // more makes others wait (reserve_below).
    const Board b = from_pos48(pos);
    double bf = std::min(45.0, std::max(20.0, (double)count_moves<SV_KOGGE>(b)));
    double nodes = 1.0;
    for (u32 k = 2; k < depth; k++) nodes *= bf;
    q->predicted = (u64)(nodes * NODE_BYTES * 1.5) + (1ull << 20);
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!running || stopping) {
            delete q;
            return PERFT_ERR_NOT_INITIALIZED;
        }
        q->ticket = nextTicket++;
        byTicket[q->ticket] = q;
        queue.push_back(q);
        submitted++;
        *ticket = q->ticket;
    }
    cvWork.notify_one();
    return PERFT_OK;
}

int Server::poll(u64 ticket, u64 *count, double *latency, bool wait, double timeoutS)
{
    std::unique_lock<std::mutex> lk(mu);
    auto it = byTicket.find(ticket);
    if (it == byTicket.end()) return PERFT_ERR_NOT_FOUND;
    ServeQuery *q = it->second;
    if (q->state != 2 && wait) {
        const auto deadline = std::chrono::steady_clock::now() + std::chrono::duration<double>(timeoutS);
        cvDone.wait_until(lk, deadline, [&] { return q->state == 2 || !running; });
    }
    if (q->state != 2) return (wait ? PERFT_ERR_TIMEOUT : PERFT_PENDING);
    if (count) *count = q->result;
    if (latency) *latency = q->tDone - q->tSubmit;
    byTicket.erase(it);
    delete q;
    return PERFT_OK;
}

void Server::get_stats(perft_serve_stats *o)
{
    std::lock_guard<std::mutex> lk(mu);
    o->submitted = submitted;
    o->completed = completed;
    o->in_flight = inFlight;
    o->queued = queue.size();
    o->iterations = iterations;
    o->launches = launches;
    o->memory_budget = budget;
    o->memory_reserved = reserved;
    o->memory_peak = peakInUse;
    o->last_error = lastError;
    o->tt_probes = hostTTStats ? hostTTStats->probes : 0;
    o->tt_hits = hostTTStats ? hostTTStats->hits : 0;
    o->tt_merged = hostTTStats ? hostTTStats->aliases : 0;
    o->tt_stores = hostTTStats ? hostTTStats->stores : 0;
}

int Server::admit()
{
    std::vector<ServeQuery *> batch;
    {
        std::lock_guard<std::mutex> lk(mu);
        while (!queue.empty() && inFlight < maxInFlight && !freeSlots.empty()) {
            ServeQuery *q = queue.front();
            // always admit into an idle server, so one huge query cannot starve
            if (inFlight > 0 && reserved + q->predicted > budget) break;
            queue.pop_front();
            q->slot = (int)freeSlots.back();
            freeSlots.pop_back();
            q->state = 1;
            q->tAdmit = now_s();
            reserved += q->predicted;
            inFlight++;
            bySlot[q->slot] = q;
            maxSlotUsed = std::max(maxSlotUsed, (u32)q->slot + 1);
            batch.push_back(q);
        }
    }
    if (batch.empty()) return PERFT_OK;
    admittedBatches++;
    const u32 n = (u32)batch.size();
    // group by depth: every node of a level has the same remaining depth
    std::stable_sort(batch.begin(), batch.end(), [](ServeQuery *a, ServeQuery *b) { return a->depth > b->depth; });
    for (u32 i = 0; i < n; i++) {
        memcpy(stagePos + 6ull * i, batch[i]->pos, 48);
        stageSlots[i] = (u32)batch[i]->slot;
        stageDepths[i] = (uint8_t)batch[i]->depth;
    }
    std::vector<std::pair<u64, u64>> tmp;
    u64 *dPos = (u64 *)take(48ull * n, tmp);
    u32 *dSlots = (u32 *)take(4ull * n, tmp);
    uint8_t *dDepths = (uint8_t *)take(n, tmp);
    if (!dPos || !dSlots || !dDepths) {
        give_back(tmp);
        return PERFT_ERR_OUT_OF_MEMORY;
    }
    if (cudaMemcpyAsync(dPos, stagePos, 48ull * n, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(dSlots, stageSlots, 4ull * n, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(dDepths, stageDepths, n, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return PERFT_ERR_CUDA;
    k_serve_admit<<<(n + 127) / 128, 128, 0, st>>>(dPos, dSlots, dDepths, n, posBySlot, pending, counts);
    launches++;
    u32 i0 = 0;
    while (i0 < n) {
        const u32 depth = batch[i0]->depth;
        u32 i1 = i0;
        while (i1 < n && batch[i1]->depth == depth) i1++;
        ServeLevel *S = new ServeLevel();
        S->r = S->depth = (int)depth;
        const u64 cnt = i1 - i0;
        if (!take_level(*S, cnt, false)) {
            delete S;
            give_back(tmp);
            return PERFT_ERR_OUT_OF_MEMORY;
        }
        k_init_roots<<<(unsigned)((cnt + 127) / 128), 128, 0, st>>>(posBySlot, dSlots + i0, (u32)cnt, S->L.planes,
                                                                     S->L.stride, S->L.cnt, S->L.root, nullptr, depth,
                                                                     counts, dErr);
        launches++;
        if (depth >= 2) pools[depth].push_back(S);
        else {
            give_back(S->mem);
            give_back(S->scanMem);
            delete S;
        }
        i0 = i1;
    }
    give_back(tmp);  // reused only by later launches on this stream
    return cudaGetLastError() == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
}

// Merges a level two or three plies above the leaves over all its queries, then
// hashes and probes the nodes that stay; copies and hits get no items.  The
// level keeps the hashes, per-node sums and aliases until it is finished.
int Server::probe_level(ServeLevel &S)
{
    const u64 n = S.L.n;
    const unsigned nb = (unsigned)((n + 255) / 256);
    if (cudaMemsetAsync(S.set, 0xFF, 8 * MERGE_SLOTS * n, st) != cudaSuccess) return PERFT_ERR_CUDA;
    const MergeLevel M{S.L.planes, S.L.stride, n,   S.L.cnt,   nullptr, nullptr, S.set,
                       nullptr,    nullptr,    S.r, false,     S.L.alias, S.L.acc, &dTTStats->aliases};
    k_merge_linked<<<nb, 256, 0, st>>>(M);
    k_tt_probe<<<std::min(nb, 8u * nsm), 256, 0, st>>>(S.L.planes, S.L.stride, n, S.r, ttKeyMask, S.L.cnt, S.L.hash,
                                                       S.L.hash2, S.L.acc, S.L.alias, tt, ttMask, dTTStats);
    launches += 2;
    S.live = S.liveMem;  // hits and copies make no parents
    S.tt = true;
    return cudaGetLastError() == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
}

// Merges the equal nodes of each query's part of a level, as the engine's
// levels do: nodes at least MERGE_MIN_PLIES below their query's position.
// Small levels stay as they are (two launches would cost more than their
// copies), and so do levels while less than a quarter of the server's memory
// is free, or where weights and set would take what the plies below need:
// merging must not displace admitted work.  A server with a
// table merges its table levels instead (probe_level).
// 200 queries of depths 3-6 submitted at once: 66.1 -> 28.5 ms.
constexpr u64 SERVE_MERGE_MIN = 4096;
int Server::merge_level(ServeLevel &S)
{
    const u64 n = S.L.n;
    if (!mergeEnabled || tt || S.r + MERGE_MIN_PLIES > S.depth || n < SERVE_MERGE_MIN ||
        blockBytes - inUse < blockBytes / 4)
        return PERFT_OK;  // (no liveMem where the level is not deep enough)
    std::vector<std::pair<u64, u64>> tmp, own;
    const bool init = S.L.weight == nullptr;
    unsigned long long *weight = init ? (unsigned long long *)take(8 * S.L.stride, own) : S.L.weight;
    unsigned long long *set = (unsigned long long *)take(8 * MERGE_SLOTS * n, tmp);
    if (!weight || !set || blockBytes - inUse < reserve_below(S.r)) {
        give_back(tmp);
        give_back(own);
        return PERFT_OK;
    }
    S.mem.insert(S.mem.end(), own.begin(), own.end());
    S.L.weight = weight;
    S.live = S.liveMem;
    const MergeLevel M{S.L.planes, S.L.stride,  n,   S.L.cnt, S.L.root, weight, set,
                       segs,       nullptr,     S.r, init,    nullptr,  nullptr, nullptr};
    const unsigned blocks = (unsigned)((n + 255) / 256);
    k_merge_prepare<<<std::min(blocks, 64u * nsm), 256, 0, st>>>(M);
    k_merge_nodes<<<blocks, 256, 0, st>>>(M);
    launches += 2;
    give_back(tmp);  // reused only by later launches on this stream
    return cudaGetLastError() == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
}

int Server::finish_level(ServeLevel &S)
{
    const u64 n = S.L.n;
    const unsigned nb = (unsigned)((n + 255) / 256);
    if (S.parent)  // into the parent level's per-node sums
        k_tt_finish<<<nb, 256, 0, st>>>(n, true, S.L.hash, S.L.hash2, S.L.acc, S.L.alias, S.L.root, S.parent->L.acc,
                                        tt, ttMask, dTTStats);
    else           // into the queries' counts
        k_serve_tt_finish<<<nb, 256, 0, st>>>(n, S.L.hash, S.L.hash2, S.L.acc, S.L.alias, S.L.root, counts,
                                               pending, tt, ttMask, dTTStats);
    launches++;
    return cudaGetLastError() == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
}

// A level whose items are all processed: finish it (table levels), free it,
// and finish a waiting parent whose last child level this was.  A table
// level of remaining depth 3 with child levels still running waits.
int Server::retire(ServeLevel *S)
{
    if (S->tt && S->outstanding > 0) {
        waiting.push_back(S);
        return PERFT_OK;
    }
    if (S->tt) {
        const int rc = finish_level(*S);
        if (rc != PERFT_OK) return rc;
    }
    ServeLevel *parent = S->parent;
    give_back(S->mem);
    give_back(S->ttMem);
    delete S;
    if (parent && --parent->outstanding == 0 && parent->scanned && parent->next >= parent->total) {
        auto it = std::find(waiting.begin(), waiting.end(), parent);
        if (it != waiting.end()) {
            waiting.erase(it);
            return retire(parent);
        }
    }
    return PERFT_OK;
}

int Server::scan_level(ServeLevel &S)
{
    const int rcMerge = table_level(S.r) ? probe_level(S) : merge_level(S);
    if (rcMerge != PERFT_OK) return rcMerge;
    const u64 n = S.L.n;
    const u64 nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    ScanSums *bsum = S.bsum;
    k_scan_reduce<<<(unsigned)nb, SCAN_NT, 0, st>>>(S.L.cnt, n, bsum);
    u64 *totals = (u64 *)(bsum + nb);
    k_scan_top<<<1, SCAN_TOP_NT, 0, st>>>(bsum, nb, totals);
    if (S.live)
        k_scan_apply<true><<<(unsigned)nb, SCAN_NT, 0, st>>>(S.L.cnt, n, bsum, totals, S.pscan, S.live,
                                                                       S.tileFirst, TILE_CAP_LOG2);
    else
        k_scan_apply<false><<<(unsigned)nb, SCAN_NT, 0, st>>>(S.L.cnt, n, bsum, totals, S.pscan, nullptr,
                                                                        S.tileFirst, TILE_CAP_LOG2);
    launches += 3;
    // a table level's nodes leave the pending count in its finish pass
    if (!S.tt) {
        k_serve_zero_parents<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(S.L.cnt, S.L.root, n, pending);
        launches++;
    }
    const bool readOk = cudaMemcpyAsync(hostTotal, totals, 16, cudaMemcpyDeviceToHost, st) == cudaSuccess;
    give_back(S.scanMem);  // reused only by later launches on this stream
    if (!readOk || cudaStreamSynchronize(st) != cudaSuccess) return PERFT_ERR_CUDA;
    S.total = hostTotal[0];
    S.nParents = S.live ? hostTotal[1] : n;
    S.scanned = true;
    return PERFT_OK;
}

int Server::launch(int mode, ServeLevel &S, u64 lo, u64 hi, DeviceLevel *child)
{
    TileParams P;
    memset(&P, 0, sizeof P);
    P.ppl = S.L.planes;
    P.pstride = S.L.stride;
    P.pscan = S.pscan;
    P.proot = S.L.root;
    P.live = S.live;
    P.pweight = S.L.weight;
    P.nParents = S.nParents;
    P.tileFirst = S.tileFirst;
    P.itemBase = lo;
    P.itemEnd = hi;
    P.capLog2 = TILE_CAP_LOG2;
    P.tileCounter = dCounter;
    if (child) {
        P.cpl = child->planes;
        P.cstride = child->stride;
        P.ccnt = child->cnt;
        P.croot = child->root;
        P.cweight = child->weight;
    }
    P.uncounted = S.r == 3;
    P.rootCounts = counts;
    P.pending = pending;
    P.err = dErr;
    const u64 nTiles = mode == MODE_LEAF ? leaf_units(S.nParents) : (hi - lo + TILE_CAP - 1) / TILE_CAP;
    if (cudaMemsetAsync(dCounter, 0, 4, st) != cudaSuccess) return PERFT_ERR_CUDA;
    if (mode == MODE_LEAF && S.tt) {
        // sums per node (the parent's own slot of acc), as the engine's table levels do
        P.proot = nullptr;
        P.rootCounts = S.L.acc;
        P.pending = nullptr;
        launch_tile_variant<MODE_LEAF>(leafSplit ? SV_KOGGE_SPLIT : SV_KOGGE,
                                       (int)std::min<u64>(gridLeafAcc, nTiles), st, P);
    } else if (mode == MODE_EXPAND && S.tt) {
        // a table level expands without pending tracking; the children's
        // root entries are parent indices (their counts flow into its sums)
        P.proot = nullptr;
        P.pending = nullptr;
        launch_tile_variant<MODE_EXPAND>(SV_KOGGE, (int)std::min<u64>(gridExpandTT, nTiles), st, P);
    } else if (mode == MODE_LEAF && leafSplit)
        k_leaf<SV_KOGGE_SPLIT, true><<<(int)std::min<u64>(gridLeaf, nTiles), LEAF_NT, LEAF_DYN_SMEM, st>>>(P);
    else if (mode == MODE_LEAF)
        k_leaf<SV_KOGGE, true><<<(int)std::min<u64>(gridLeaf, nTiles), LEAF_NT, LEAF_DYN_SMEM, st>>>(P);
    else
        k_tile<SV_KOGGE, true><<<(int)std::min<u64>(gridExpand, nTiles), TILE_NT, TILE_DYN_SMEM, st>>>(P);
    launches++;
    return cudaGetLastError() == cudaSuccess ? PERFT_OK : PERFT_ERR_CUDA;
}

int Server::advance()
{
    const u64 launchesBefore = launches;
    for (int r = 2; r <= SERVE_MAX_R; r++) {
        std::vector<ServeLevel *> keep;
        std::vector<ServeLevel *> work;
        work.swap(pools[r]);
        for (size_t li = 0; li < work.size(); li++) {
            ServeLevel *S = work[li];
            if (!S->scanned) {
                const int rc = scan_level(*S);
                if (rc != PERFT_OK) return rc;
            }
            // The count-only ply's parents count as one item each (see k_tile), but
            // the positions of depth-2 queries as their moves.  At least 8192 of them:
            // the launch is most of a smaller step's time, so that no query gets
            // done sooner.  200 queries of depths 3-6 with step_items 8192: a tenth
            // done after 2.0 ms and all after 0.72 s; in steps of 256 parents 2.5 ms
            // and 4.4 s.
            const u64 step = r == 2 ? std::max<u64>(stepItems / SERVE_MOVES_PER_PARENT, TILE_CAP) : stepItems;
            u64 lo = S->next, hi = std::min(S->total, lo + step);
            if (lo < hi) {
                if (r == 2) {
                    int rc = launch(MODE_LEAF, *S, lo, hi, nullptr);
                    if (rc != PERFT_OK) return rc;
                } else {
                    ServeLevel *C = nullptr;
                    for (;;) {  // shrink the step until the children fit
                        C = new ServeLevel();
                        C->r = r - 1;
                        C->depth = S->depth;
                        if (take_level(*C, hi - lo, S->L.weight != nullptr)) {
                            if (blockBytes - inUse >= reserve_below(C->r)) break;
                            give_back(C->mem);
                            give_back(C->ttMem);
                            give_back(C->scanMem);
                        }
                        delete C;
                        C = nullptr;
                        if (hi - lo <= (u64)TILE_CAP) break;
                        hi = lo + (((hi - lo) / 2 + TILE_CAP - 1) & ~(u64)(TILE_CAP - 1));
                    }
                    if (!C) {  // no memory this iteration
                        keep.push_back(S);
                        continue;
                    }
                    int rc = launch(MODE_EXPAND, *S, lo, hi, &C->L);
                    if (rc != PERFT_OK) return rc;
                    if (S->tt) {
                        C->parent = S;
                        S->outstanding++;
                    }
                    pools[r - 1].push_back(C);
                }
                S->next = hi;
            }
            if (S->next >= S->total) {
                const int rc = retire(S);
                if (rc != PERFT_OK) return rc;
            } else {
                keep.push_back(S);
            }
        }
        for (ServeLevel *S : keep) pools[r].push_back(S);
    }
    // Levels that cannot get memory wait for others to finish; if nothing at
    // all could run for many iterations the budget is too small for the
    // admitted work: fail loudly instead of spinning.
    bool pendingWork = !waiting.empty();
    for (int r = 2; r <= SERVE_MAX_R; r++) pendingWork |= !pools[r].empty();
    idleIterations = (launches == launchesBefore && pendingWork) ? idleIterations + 1 : 0;
    return idleIterations > 200 ? PERFT_ERR_OUT_OF_MEMORY : PERFT_OK;
}

int Server::complete()
{
    if (!maxSlotUsed) return PERFT_OK;
    if (cudaMemcpyAsync(hostPending, pending, 8ull * maxSlotUsed, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(hostCounts, counts, 8ull * maxSlotUsed, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        (tt && cudaMemcpyAsync(hostTTStats, dTTStats, sizeof(TTStats), cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return PERFT_ERR_CUDA;
    const double t = now_s();
    bool any = false;
    {
        std::lock_guard<std::mutex> lk(mu);
        for (u32 s = 0; s < maxSlotUsed; s++) {
            ServeQuery *q = bySlot[s];
            if (!q || hostPending[s] != 0) continue;
            q->result = hostCounts[s];
            q->state = 2;
            q->tDone = t;
            bySlot[s] = nullptr;
            freeSlots.push_back(s);
            reserved -= q->predicted;
            inFlight--;
            completed++;
            any = true;
        }
        while (maxSlotUsed && !bySlot[maxSlotUsed - 1]) maxSlotUsed--;
    }
    if (any) cvDone.notify_all();
    return PERFT_OK;
}

void Server::loop()
{
    cudaSetDevice(dev);
    for (;;) {
        {
            std::unique_lock<std::mutex> lk(mu);
            cvWork.wait_for(lk, std::chrono::milliseconds(50),
                            [&] { return stopping || !queue.empty() || inFlight > 0; });
            if (stopping) break;
            if (queue.empty() && inFlight == 0) continue;
        }
        int rc = admit();
        if (rc == PERFT_OK) rc = advance();
        if (rc == PERFT_OK) rc = complete();
        iterations++;
        if (rc != PERFT_OK) {
            std::lock_guard<std::mutex> lk(mu);
            lastError = rc;
            break;
        }
    }
}

Server g_server;

}  // namespace
