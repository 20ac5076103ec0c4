// grz_ccbfs.cu -- Connected Components and Breadth-First Search: edge-pull, edge-push on a
// compacted frontier, vertex (frontier) phase, and the engine-switching driver loops.
//
// Reference semantics (paths in the Grazelle tree):
//   CC pull   source/phase_edge_pull_cc.asm:50-392   label[d] = min(label[d], min over valid sources)
//   CC push   source/phase_edge_push_cc.asm:51-573   for sources in HasInfo: CAS-min into label[dst]
//   BFS pull  source/phase_edge_pull_bfs.asm:53-211  for dst in WantsInfo: parent = max HasInfo source
//                                                    of the first vector that holds one
//   BFS push  source/phase_edge_push_bfs.asm:53-202  for sources in HasInfo: visit dst in WantsInfo
//   vertex    source/phase_vertex_{cc,bfs}.asm:37-46 zero HasInfo* after the pointer swap
//   driver    source/execution_cc.c:94-268, source/execution_bfs.c:120-276
//   vote      include/phasehelpers.inc:388-399       1 + outdeg per changed vertex
//
// GPU form:
//   * Labels and parents live on the device as uint32 (IDs are below 2^32).  The reference's
//     double props are produced only when the result is read back.  Entry V of the label
//     array is a permanent +infinity that invalid lanes gather.
//   * Pull: one thread per vector, a warp-segmented reduction per destination, one atomic per
//     (warp, destination).  Labels are updated in place, as the reference's CAS loop does, so
//     a later vector may already see a lowered label.
//   * Push: HasInfo is compacted, in vertex order block by block, into a list of active sources that have
//     out-edges, with the offset of each one's vectors among all of theirs.  The concatenation of
//     their vector ranges is expanded in tiles of one vector per thread over the whole grid, so
//     neither threads nor blocks wait on high-degree sources.
//   * Each changed vertex is counted once per iteration: the first setter of its HasInfo* bit
//     adds 1 + outdeg to the vote.  The reference can count a destination that straddles two
//     work units twice.  The vote only steers the engine choice.
//   * BFS parent rules are deterministic, so parents equal the single-thread reference: pull
//     keeps the largest HasInfo source of the lowest-indexed vector that holds one (a 64-bit
//     atomicMin on (vector index, ~source)); push keeps the smallest HasInfo source (atomicMin).
//     A vertex's BFS level is the iteration that visits it, so levels are exact by construction.
#include <cooperative_groups.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "grz_internal.cuh"
#include "grz_switch.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int T = 256;
constexpr uint32_t INF = 0xffffffffu;
// BFS visit: sweep all vertices instead of the touched list when more than V / this were touched
constexpr uint64_t VISIT_DENSE_RATIO = 128;
// tiles of T vectors per step of the BFS pull kernel
constexpr int BFS_PULL_TILES = 4;
// bitmap words (64 destinations each) a warp of the first-vector passes owns, and their blocks per SM
#ifndef GRZ_BFS_FW
#define GRZ_BFS_FW 2
#endif
#ifndef GRZ_BFS_MINB
#define GRZ_BFS_MINB 8
#endif
constexpr int FW = GRZ_BFS_FW;

unsigned blocks_for(uint64_t n) { return (unsigned)((n + T - 1) / T); }

__device__ __forceinline__ bool bit_of(const unsigned long long* bm, uint32_t v) { return (bm[v >> 6] >> (v & 63)) & 1ull; }

// sets bit v; true if this call set it (it was clear)
__device__ __forceinline__ bool bit_set_first(unsigned long long* bm, uint32_t v)
{
    const unsigned long long m = 1ull << (v & 63);
    return !(atomicOr(bm + (v >> 6), m) & m);
}

__device__ __forceinline__ void vote_add(unsigned long long* vote, unsigned long long x)
{
    // one add per block (the callers aggregate the block first), spread over the vote slots
    if (x) atomicAdd(vote + (blockIdx.x & (GRZ_VOTE_SLOTS - 1)) * GRZ_VOTE_STRIDE, x);
}

__device__ __forceinline__ unsigned long long block_sum_u64(unsigned long long x, unsigned long long* red)
{
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    x = 0;
    if (threadIdx.x < 32) {
        x = (threadIdx.x < T / 32) ? red[threadIdx.x] : 0ull;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    }
    return x;
}

// Appends `val` to the BFS touched list for the lanes with `pred`, one atomicAdd per warp (all 32
// lanes call it together; the callers' loops are warp-uniform), until the list holds
// V / VISIT_DENSE_RATIO + 1 entries.  From there on k_bfs_visit sweeps all vertices instead of
// reading the list (the count only grows), so further appends are skipped: a plain load of the
// counter replaces the atomic, and a large iteration no longer queues millions of atomics on one
// address.  Each destination is first-touched once per phase, so the list never outgrows V.
__device__ __forceinline__ bool touched_full(const uint32_t* count, uint32_t V)
{
    return *(volatile const uint32_t*)count >= (uint32_t)((uint64_t)V / VISIT_DENSE_RATIO + 1);
}

// `full`: touched_full as the caller last read it (once per tile or step, warp-uniform); the
// count can pass the bound between two reads, which only lets a few more appends through
__device__ __forceinline__ void touched_append(bool pred, uint32_t val, uint32_t* __restrict__ list, uint32_t* __restrict__ count,
                                               bool full)
{
    if (full) return;
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) list[base + __popc(m & ((1u << lane) - 1u))] = val;
}

// The same for four values per lane, in one atomicAdd.  Looks at the count only when there is something to
// append (GB300, a push to few open destinations, of a million vectors: 53 us with a look for every vector, so
// 32); returns whether the list was full.
__device__ __forceinline__ bool touched_append4(const bool (&pred)[4], const uint32_t (&val)[4], uint32_t* __restrict__ list,
                                                uint32_t* __restrict__ count, uint32_t V)
{
    unsigned m[4];
    uint32_t n = 0;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        m[l] = __ballot_sync(0xffffffffu, pred[l]);
        n += __popc(m[l]);
    }
    if (!n) return false;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t base = 0;
    bool full = false;
    if (lane == 0) {
        full = touched_full(count, V);
        if (!full) base = atomicAdd(count, n);
    }
    if (__shfl_sync(0xffffffffu, full, 0)) return true;
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (pred[l]) list[base + __popc(m[l] & ((1u << lane) - 1u))] = val[l];
        base += __popc(m[l]);
    }
    return false;
}

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct VoteCfg {
    const uint32_t* degree;
    int without_count, without_outdeg;
    __device__ __forceinline__ unsigned long long of(uint32_t v) const
    {
        return (without_count ? 0ull : 1ull) + (without_outdeg ? 0ull : (unsigned long long)degree[v]);
    }
};

// ---------------------------------------------------------------------------------------------
// CC pull

// Smallest label written by a CC iteration, for the next iteration's converged-destination
// skip.  Iteration k adds ((k << 32) | ~m) into word k & 1 with atomicMax, m the smallest label
// it wrote; the words are never reset: a tag other than k - 1 means "unknown" and the reader
// does not skip.  Why the skip is exact: after a complete iteration (a pull over the
// whole list, or a push from the whole frontier) every destination d holds at most the labels
// its sources had when d was last evaluated, so only a source that changed since can lower d.
// Every such change happened in iteration k - 1 (earlier ones were evaluated or pushed in
// k - 1) or happens during iteration k (recorded in HasInfo*, handled in k + 1).  A change in
// k - 1 wrote a label >= m(k - 1); so if label[d] <= m(k - 1), iteration k cannot lower d.
// Iteration 1 follows the initial state, in which every vertex counts as changed: no skip.
__device__ __forceinline__ bool cc_prev_min(const unsigned long long* __restrict__ chg, uint32_t k, uint32_t* m)
{
    if (k < 2) return false;
    const unsigned long long w = chg[(k - 1) & 1];
    if ((uint32_t)(w >> 32) != k - 1) return false;
    *m = ~(uint32_t)w;
    return true;
}

// block-wide minimum of one value per thread, then one tagged atomicMax (threadIdx.x 0 only)
template <int BT>
__device__ __forceinline__ void cc_record_min(uint32_t my_min, uint32_t* red32, unsigned long long* __restrict__ chg, uint32_t k)
{
    my_min = __reduce_min_sync(0xffffffffu, my_min);
    if ((threadIdx.x & 31) == 0) red32[threadIdx.x >> 5] = my_min;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t x = threadIdx.x < BT / 32 ? red32[threadIdx.x] : INF;
        x = __reduce_min_sync(0xffffffffu, x);
        if (threadIdx.x == 0 && x != INF) atomicMax(chg + (k & 1), ((unsigned long long)k << 32) | (unsigned long long)(~x));
    }
}

// Persistent, BT threads per block, one thread per vector per tile of BT vectors.  The labels
// of the first `ncache` hub slots are copied into shared memory when the block starts; lanes
// that name them read shared memory instead of gathering through L1 (in a power-law graph most
// lanes).  Those copies may fall behind the in-place updates of this phase, which the
// reference's asynchronous CAS loop allows as well: a label only ever decreases, every value
// read is one the source really had, and an iteration that changes nothing is still a fixpoint.
// Iteration k (epoch_dev, else epoch) skips destinations whose label is at most the smallest
// label written in iteration k - 1 (cc_prev_min; only with use_prev, i.e. when k - 1 was a
// complete iteration): it reads their destination and label, not their vectors.  R-MAT's
// hubs have the smallest IDs, so after the first iteration most of the giant component holds
// label 0 and the second pull reads little more than the destinations.
// tiles whose destination and label loads the skip mode issues together
constexpr int SKIP_TILES = 4;

// double-buffered staging of the edge stream in shared memory (the bulk-copy form)
template <int BT>
struct CCStage {
    uint4 nbr[2][BT];
    uint32_t dst[2][BT];
    unsigned long long bar[2];
};
struct CCNoStage {};

template <int BT, bool BULK>
__global__ void __launch_bounds__(BT) k_cc_pull(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv, uint64_t first,
                                                uint64_t nvec, uint32_t V, uint32_t* __restrict__ label,
                                                const uint32_t* __restrict__ hub_vid, uint32_t nhub, uint32_t ncache,
                                                unsigned long long* __restrict__ has_next, VoteCfg vc,
                                                unsigned long long* __restrict__ vote, unsigned long long* __restrict__ chg,
                                                uint32_t epoch, const uint32_t* __restrict__ epoch_dev, int use_prev,
                                                unsigned* __restrict__ err)
{
    extern __shared__ uint32_t s_hub[];
    __shared__ unsigned long long red[BT / 32];
    __shared__ uint32_t red32[BT / 32];
    __shared__ __align__(16) typename std::conditional<BULK, CCStage<BT>, CCNoStage>::type stg;
    for (uint32_t k = threadIdx.x; k < ncache; k += BT) s_hub[k] = label[__ldg(hub_vid + k)];
    const uint32_t ep = epoch_dev ? *epoch_dev : epoch;
    uint32_t mprev = 0;
    bool skip = use_prev && cc_prev_min(chg, ep, &mprev);
    // use_prev 2: a source-segment pass, which runs only when the skip is off (the full pass);
    // use_prev 3: the pass over the whole list that runs only when it is on (the grid agrees)
    if ((use_prev == 2 && skip) || (use_prev == 3 && !skip)) return;
    // use_prev 4: after k_cc_pull_first, which ran because the skip is off: the destinations
    // whose label is already 0, the smallest there is, need none of their vectors
    // use_prev 5: the same, but only then (a later iteration is left to the open-destination pass)
    if (use_prev == 5 && skip) return;
    if ((use_prev == 4 || use_prev == 5) && !skip) {
        skip = true;
        mprev = 0;
    }
    const int lane = threadIdx.x & 31;
    unsigned long long my_vote = 0;
    uint32_t my_min = INF;
    const uint64_t ntiles = (nvec + BT - 1) / BT;
    const uint64_t nfull = nvec / BT;  // tiles the bulk copies serve (whole tiles only)
    // The bulk form copies each whole tile's vectors and destinations into shared memory on the
    // copy engine, two tiles ahead, so the SM's load path serves only the label gathers.  Not in
    // skip mode (it reads most vectors' destinations only) nor for a vector sub-range.
    const bool bulk = BULK && !skip && first == 0;
    unsigned par = 0u;  // bit j: the parity stage j waits for next
    if constexpr (BULK) {
        if (bulk && threadIdx.x == 0) {
            mbar_init(&stg.bar[0], 1);
            mbar_init(&stg.bar[1], 1);
            mbar_fence_init();
            for (int j = 0; j < 2; ++j) {
                const uint64_t t = blockIdx.x + (uint64_t)j * gridDim.x;
                if (t < nfull) {
                    mbar_arrive_expect_tx(&stg.bar[j], BT * (sizeof(uint4) + sizeof(uint32_t)));
                    bulk_copy_g2s(stg.nbr[j], nbr + t * BT, BT * sizeof(uint4), &stg.bar[j]);
                    bulk_copy_g2s(stg.dst[j], dstv + t * BT, BT * sizeof(uint32_t), &stg.bar[j]);
                }
            }
        }
    }
    __syncthreads();
    // one tile's reduction and updates, once its destinations (key), their labels if known (labd,
    // skip mode) and its vectors (staged, or loaded here when needed) are at hand
    auto finish = [&](uint64_t v, bool live, uint32_t key, uint32_t labd, bool need, bool staged, uint4 sv) {
        uint32_t m = INF;
        if (need) {
            const uint4 s4 = staged ? sv : ld_stream(nbr + v);
            const uint32_t x[4] = { s4.x, s4.y, s4.z, s4.w };
            auto fetch = [&](uint32_t xl) -> uint32_t {
                const uint32_t sl = xl - GRZ_HUB_BASE;
                if (sl < ncache) return s_hub[sl];
                // labels change in place during the phase: plain (coherent) loads
                const uint32_t id = sl < nhub ? __ldg(hub_vid + sl) : min(xl, V);
                return ld_label(label + id);
            };
            // A vector's lanes hold its sources in ascending order, so lane 0 is the
            // smallest-ID source: in a power-law graph often a hub whose label is already 0.
            // Then the minimum is 0 and the other three gathers are not issued.
            m = fetch(x[0]);
            if (m != 0) m = min(m, min(min(fetch(x[1]), fetch(x[2])), fetch(x[3])));
        }
        const uint32_t prevkey = __shfl_up_sync(0xffffffffu, key, 1);
        const uint32_t nextkey = __shfl_down_sync(0xffffffffu, key, 1);
        const bool head = lane == 0 || key != prevkey;
        const bool tail = lane == 31 || key != nextkey;
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        const int segstart = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
        const int maxlen = __reduce_max_sync(0xffffffffu, (unsigned)(lane - segstart + 1));
        for (int off = 1; off < maxlen; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, m, off);
            if (lane - off >= segstart) m = min(m, o);
        }
        if (live && tail && m != INF && m < (skip ? labd : label[key])) {
            const uint32_t old = atomicMin(label + key, m);
            if (m < old) {
                my_min = min(my_min, m);
                if (bit_set_first(has_next, key)) my_vote += vc.of(key);
            }
        }
    };
    if (skip) {
        // Skip mode: a vector is read only if its destination's label can still drop.  Each
        // block takes SKIP_TILES consecutive tiles at a time and issues all their destination
        // loads, then all their label loads, before any tile goes on: the chain destination ->
        // label -> vector is latency-bound, so this keeps SKIP_TILES times more loads in flight.
        constexpr int U = SKIP_TILES;
        for (uint64_t t0 = (uint64_t)blockIdx.x * U; t0 < ntiles; t0 += (uint64_t)gridDim.x * U) {
            uint32_t keys[U], labs[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint64_t i = (t0 + u) * BT + threadIdx.x;
                keys[u] = i < nvec ? ld_stream(dstv + first + i) : INF;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) labs[u] = keys[u] != INF ? ld_label(label + keys[u]) : INF;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint64_t i = (t0 + u) * BT + threadIdx.x;
                const bool live = i < nvec;
                const bool need = live && labs[u] > mprev;
                if (!__any_sync(0xffffffffu, need)) continue;  // warp-uniform
                finish(first + i, live, keys[u], labs[u], need, false, make_uint4(INF, INF, INF, INF));
            }
        }
    } else {
        uint64_t j = 0;
        for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x, ++j) {
            const uint64_t i = t * BT + threadIdx.x;
            const uint64_t v = first + i;
            const bool live = i < nvec;
            uint32_t key = INF;
            bool staged = false;
            uint4 sv = make_uint4(INF, INF, INF, INF);
            if constexpr (BULK) {
                if (bulk && t < nfull) {
                    const int st = (int)(j & 1);
                    const bool ok = mbar_wait_bounded(&stg.bar[st], (par >> st) & 1u);
                    if (__syncthreads_or(!ok)) {
                        if (threadIdx.x == 0) atomicExch(err, 1u);
                        return;
                    }
                    par ^= 1u << st;
                    sv = stg.nbr[st][threadIdx.x];
                    key = stg.dst[st][threadIdx.x];
                    staged = true;
                    __syncthreads();  // every thread has read the stage
                    const uint64_t tn = t + 2ull * gridDim.x;
                    if (threadIdx.x == 0 && tn < nfull) {
                        fence_proxy_async_smem();
                        mbar_arrive_expect_tx(&stg.bar[st], BT * (sizeof(uint4) + sizeof(uint32_t)));
                        bulk_copy_g2s(stg.nbr[st], nbr + tn * BT, BT * sizeof(uint4), &stg.bar[st]);
                        bulk_copy_g2s(stg.dst[st], dstv + tn * BT, BT * sizeof(uint32_t), &stg.bar[st]);
                    }
                }
            }
            if (live && !staged) key = ld_stream(dstv + v);
            finish(v, live, key, INF, live, staged, sv);
        }
    }
    for (int o = 16; o > 0; o >>= 1) my_vote += __shfl_down_sync(0xffffffffu, my_vote, o);
    if (lane == 0) red[threadIdx.x >> 5] = my_vote;
    cc_record_min<BT>(my_min, red32, chg, ep);  // (contains the __syncthreads the vote sum needs)
    if (threadIdx.x < 32) {
        unsigned long long x = threadIdx.x < BT / 32 ? red[threadIdx.x] : 0ull;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (threadIdx.x == 0) vote_add(vote, x);
    }
}

// CC pull, first-vector pass of an iteration without a usable previous minimum (the first pull of
// a run).  Each destination's first vector holds its smallest-ID sources; in a power-law graph
// one of them is usually a hub whose label is 0 by the time it is read (in place, as the full
// pass reads them), and then the destination's label is final for this iteration: 0 cannot be
// lowered.  This pass evaluates every destination's first vector (lane 0 first, as in
// k_cc_pull), one destination per thread, and writes the new labels.  What follows reads the
// other vectors of the destinations still above 0, so the iteration's result is the full pull's:
// in the default form (GRZ_TUNE_CC_PULL_FIRST 4) the compaction of the destinations this pass
// marks in `unres` (open_all: every one still above 0) and k_cc_pull_expand over all their
// vectors; in form 2 the same for the remaining vectors of those with more than one; in forms 1
// and 3 the pass over the whole list (k_cc_pull with use_prev 4 or 5) that skips the
// destinations at 0.  A warp owns CFW bitmap words (64 destinations each), so it writes their
// HasInfo* and `unres` bits without atomics; the pass records its smallest label written for the
// next iteration's skip, and sets *gate to 1 in an iteration it runs, 0 in one it leaves to the
// later-pull kernels.
#ifndef GRZ_CC_FW
#define GRZ_CC_FW 1
#endif
// bitmap words a warp of k_cc_pull_first owns (GB300, R-MAT 24 sym: 1 word 0.42 ms for the first pull,
// 2 words 0.46 ms, with 60 bytes of spills at 32 registers)
constexpr int CFW = GRZ_CC_FW;

__global__ void __launch_bounds__(T, 8) k_cc_pull_first(const uint32_t* __restrict__ rowptr, const uint4* __restrict__ nbr,
                                                      uint32_t V, uint64_t W, uint32_t* __restrict__ label,
                                                      const uint32_t* __restrict__ hub_vid, uint32_t nhub,
                                                      unsigned long long* __restrict__ has_next, VoteCfg vc,
                                                      unsigned long long* __restrict__ vote, unsigned long long* __restrict__ chg,
                                                      uint32_t epoch, const uint32_t* __restrict__ epoch_dev,
                                                      unsigned long long* __restrict__ unres, uint32_t* __restrict__ gate,
                                                      int open_all)
{
    __shared__ unsigned long long red[T / 32];
    __shared__ uint32_t red32[T / 32];
    const uint32_t ep = epoch_dev ? *epoch_dev : epoch;
    uint32_t mprev = 0;
    const bool skip_iteration = cc_prev_min(chg, ep, &mprev);  // the same on every thread
    if (gate && blockIdx.x == 0 && threadIdx.x == 0) *gate = skip_iteration ? 0u : 1u;
    if (skip_iteration) return;  // the skip pass does this iteration alone
    constexpr int Q = 2 * CFW;
    const int lane = threadIdx.x & 31;
    unsigned long long my_vote = 0;
    uint32_t my_min = INF;
    auto fetch = [&](uint32_t xl) -> uint32_t {
        const uint32_t sl = xl - GRZ_HUB_BASE;
        const uint32_t id = sl < nhub ? __ldg(hub_vid + sl) : min(xl, V);
        return ld_label(label + id);
    };
    const uint64_t nwarps = (uint64_t)gridDim.x * (T / 32);
    // row pointers of a group of destinations (a and b: start and end of each slot's range)
    auto rows = [&](uint64_t w, uint32_t* a, uint32_t* b) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const uint64_t v = 64 * w + 32 * (uint64_t)q + lane;
            a[q] = b[q] = 0;
            if (w < W && v < V) {
                a[q] = rowptr[v];
                b[q] = rowptr[v + 1];
            }
        }
    };
    uint64_t w0 = ((uint64_t)blockIdx.x * (T / 32) + (threadIdx.x >> 5)) * CFW;
    uint32_t ra[Q], rb[Q];
    rows(w0, ra, rb);
    for (; w0 < W; w0 += nwarps * CFW) {  // warp-uniform
        uint32_t r0[Q], n[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            r0[q] = ra[q];
            n[q] = rb[q] - ra[q];
        }
        uint4 sv[Q];
        uint32_t cur[Q];  // the destinations' own labels, loaded with their first vectors
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            sv[q] = n[q] ? ld_stream(nbr + r0[q]) : make_uint4(INF, INF, INF, INF);
            cur[q] = n[q] ? ld_label(label + (uint32_t)(64 * w0 + 32 * (uint64_t)q + lane)) : 0u;
        }
        uint32_t m[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) m[q] = n[q] ? fetch(sv[q].x) : INF;
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (m[q] != 0 && n[q]) m[q] = min(m[q], min(min(fetch(sv[q].y), fetch(sv[q].z)), fetch(sv[q].w)));
#pragma unroll
        for (int f = 0; f < CFW; ++f) {
            // word w0 + f: new labels of its 64 destinations, then its HasInfo* bits (set by lane 0;
            // a destination counts in the vote if its bit was clear)
            unsigned long long hn = 0ull, un = 0ull;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int q = 2 * f + h;
                const uint32_t v = (uint32_t)(64 * w0 + 32 * (uint64_t)q + lane);
                bool ch = false, more = false;
                if (n[q]) {
                    // this thread is the destination's only writer in this pass, so its label read
                    // with the vector is still current
                    if (m[q] < cur[q]) {
                        label[v] = m[q];
                        my_min = min(my_min, m[q]);
                        ch = true;
                    }
                    // still open: its other vectors (open_all: all of them again) are read next
                    more = (open_all || n[q] > 1) && min(m[q], cur[q]) != 0;
                }
                hn |= (unsigned long long)__ballot_sync(0xffffffffu, ch) << (32 * h);
                un |= (unsigned long long)__ballot_sync(0xffffffffu, more) << (32 * h);
            }
            if (unres && lane == 0 && w0 + f < W) unres[w0 + f] = un;
            if (!hn) continue;  // warp-uniform
            unsigned long long old = 0ull;
            if (lane == 0) {
                old = has_next[w0 + f];
                has_next[w0 + f] = old | hn;
            }
            const unsigned long long fresh = hn & ~__shfl_sync(0xffffffffu, old, 0);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if ((fresh >> (32 * h + lane)) & 1ull) my_vote += vc.of((uint32_t)(64 * (w0 + f) + 32 * h + lane));
        }
        // the next group's row pointers (issuing them at the top of the step instead, to overlap
        // this group's chain, needed more registers than the 32 of 8 blocks per SM and measured no
        // faster on GB300; loading the destinations' own labels with their first vectors, one
        // dependent round trip less, took the first pull at R-MAT 24 sym from 0.33 to 0.32 ms)
        rows(w0 + nwarps * CFW, ra, rb);
    }
    my_vote = block_sum_u64(my_vote, red);
    if (threadIdx.x == 0) vote_add(vote, my_vote);
    __syncthreads();
    cc_record_min<T>(my_min, red32, chg, ep);
}

// CC pull of an iteration with a usable previous minimum m (the skip of k_cc_pull): marks in
// `unres` the destinations with in-vectors whose label is above m, the only ones the iteration can
// lower, for the compaction and k_cc_pull_expand; *gate = 1.  In an iteration without a usable
// minimum it only sets *gate = 0.  A warp per bitmap word: each lane reads two labels.
__global__ void __launch_bounds__(T) k_cc_mark_open(const uint32_t* __restrict__ label, const unsigned long long* __restrict__ nonempty,
                                                    uint64_t V, uint64_t W, const unsigned long long* __restrict__ chg, uint32_t epoch,
                                                    const uint32_t* __restrict__ epoch_dev, unsigned long long* __restrict__ unres,
                                                    uint32_t* __restrict__ gate)
{
    const uint32_t ep = epoch_dev ? *epoch_dev : epoch;
    uint32_t mprev = 0;
    const bool skip_iteration = cc_prev_min(chg, ep, &mprev);
    if (gate && blockIdx.x == 0 && threadIdx.x == 0) *gate = skip_iteration ? 1u : 0u;
    if (!skip_iteration) return;
    const int lane = threadIdx.x & 31;
    const uint64_t nwarps = (uint64_t)gridDim.x * (T / 32);
    for (uint64_t w = (uint64_t)blockIdx.x * (T / 32) + (threadIdx.x >> 5); w < W; w += nwarps) {  // warp-uniform
        const uint64_t v0 = 64 * w + lane, v1 = v0 + 32;
        const bool o0 = v0 < V && ld_label(label + v0) > mprev;
        const bool o1 = v1 < V && ld_label(label + v1) > mprev;
        const unsigned long long m = (unsigned long long)__ballot_sync(0xffffffffu, o0) |
                                     ((unsigned long long)__ballot_sync(0xffffffffu, o1) << 32);
        if (lane == 0) unres[w] = m & nonempty[w];
    }
}

// ---------------------------------------------------------------------------------------------
// BFS pull

// BFS pull (phase_edge_pull_bfs.asm:53-211), persistent over tiles of T vectors.  For a
// wanted destination, a vector's candidate is (vector index, ~largest HasInfo source); the
// smallest candidate per destination wins: the reference's parent rule (the largest frontier
// source of the first vector that has one).  Vectors of one destination are reduced within
// the warp first, so only one atomicMin per (warp, destination) reaches memory.
__global__ void __launch_bounds__(T) k_bfs_pull(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv, uint64_t first,
                                                uint64_t nvec, uint32_t V, const unsigned long long* __restrict__ has,
                                                const unsigned long long* __restrict__ wants,
                                                unsigned long long* __restrict__ cand, uint32_t* __restrict__ touched,
                                                uint32_t* __restrict__ ntouched, const uint32_t* __restrict__ hub_vid, uint32_t nhub,
                                                unsigned long long* __restrict__ has_next)
{
    // U tiles per step: their destination loads, then their WantsInfo loads, are issued together
    // (enough bytes in flight per SM to cover DRAM latency);
    // late in a BFS most destinations are visited and a warp without a wanted one skips its tile
    constexpr int U = BFS_PULL_TILES;
    const int lane = threadIdx.x & 31;
    const uint64_t ntiles = (nvec + T - 1) / T;
    for (uint64_t t0 = (uint64_t)blockIdx.x * U; t0 < ntiles; t0 += (uint64_t)gridDim.x * U) {
        uint32_t keys[U];
        bool want[U];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const uint64_t i = (t0 + j) * T + threadIdx.x;
            keys[j] = i < nvec ? __ldcs(dstv + first + i) : INF;
        }
#pragma unroll
        for (int j = 0; j < U; ++j) want[j] = keys[j] != INF && bit_of(wants, keys[j]);  // strong check
        const bool full = __shfl_sync(0xffffffffu, lane == 0 ? touched_full(ntouched, V) : false, 0);
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (!__ballot_sync(0xffffffffu, want[j])) continue;  // warp-uniform
            const uint64_t v = first + (t0 + j) * T + threadIdx.x;
            const uint32_t key = keys[j];
            unsigned long long k = ~0ull;
            if (want[j]) {
                const uint4 s = __ldcs(nbr + v);
                const uint32_t ids[4] = { grz_hub_decode(s.x, hub_vid, nhub), grz_hub_decode(s.y, hub_vid, nhub),
                                          grz_hub_decode(s.z, hub_vid, nhub), grz_hub_decode(s.w, hub_vid, nhub) };
                uint32_t best = 0;
                bool any = false;
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    const uint32_t id = ids[l];
                    if (id < V && bit_of(has, id)) {  // weak check on the source
                        best = any ? max(best, id) : id;
                        any = true;
                    }
                }
                if (any) k = ((unsigned long long)v << 32) | (unsigned long long)(~best);
            }
            // segmented min of k over runs of equal keys within the warp
            const uint32_t prevkey = __shfl_up_sync(0xffffffffu, key, 1);
            const uint32_t nextkey = __shfl_down_sync(0xffffffffu, key, 1);
            const bool head = lane == 0 || key != prevkey;
            const bool tail = lane == 31 || key != nextkey;
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            const int segstart = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
            const int maxlen = __reduce_max_sync(0xffffffffu, (unsigned)(lane - segstart + 1));
            for (int off = 1; off < maxlen; off <<= 1) {
                const unsigned long long o = __shfl_up_sync(0xffffffffu, k, off);
                if (lane - off >= segstart) k = min(k, o);
            }
            bool first_touch = false;
            if (tail && k != ~0ull && k < cand[key]) {
                first_touch = atomicMin(cand + key, k) == ~0ull;
                if (first_touch) atomicOr(has_next + (key >> 6), 1ull << (key & 63));
            }
            touched_append(first_touch, key, touched, ntouched, full);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Push: frontier compaction and edge-balanced expansion.
//
// The active sources that have out-vectors are compacted, each with the offset
// of its first vector in the concatenation of their vector ranges.  The expansion then splits
// that concatenation into tiles of PUSH_TILE vectors spread over the grid, so a hub's vectors
// are spread over many blocks.  tile_first[t] is the frontier entry that owns the first vector
// of tile t.  Passes: k_fr_compact (frontier entries, their vector offsets and the tile owners),
// k_push_expand.
//
// A tile is one vector per thread: a long tile's vectors would wait for each other, and small frontiers
// would leave most of the chip idle.  GB300, tiles of 1024, 512 and 256 vectors: the pushes of 8 BFS runs
// on an R-MAT graph of 2^24 vertices 815, 743 and 687 us, CC of 4096 vertices 148, 140 and 136 us.

constexpr uint32_t PUSH_TILE = T;

// Each warp takes WORDS consecutive 32-vertex words of the two bitmaps, one per lane
// (HasInfo and out-vectors for push; WantsInfo, or the destinations a first pass left open, and
// in-vectors for the pulls); a block with nothing selected returns after reading its words.  A warp
// then walks its words with a lane per vertex, so row pointers and entries are read and written
// coalesced: once to count its vectors, and, after one 64-bit atomic per block has given the block
// its place (selected vertices in the high half, their vectors in the low half, so the two stay in
// step), once more to write.  The list is in vertex order inside a block's part only, which is all
// its readers need: a vertex's vectors stay consecutive and offsets ascend along the list.
// Before: a count kernel, a one-block scan and a write kernel with 32 vertices per thread.  GB300,
// whole runs, three kernels -> one: 8 BFS at R-MAT 24 9.67 -> 9.15 ms, a BFS of 1400 levels on a mesh of
// 250k vertices 33.4 -> 30.6 ms.
// Words of a warp: its passes over them are a chain of loads, FR_STEP words at a time, so a graph that would
// give few blocks takes fewer words per warp (GB300, 4096 vertices: 32 words 8 to 13 us, 4 words 2 us); with
// more blocks the adds to the one counter cost more than the chain.
constexpr int FR_WORDS = 32, FR_WORDS_SMALL = 4;
constexpr uint64_t FR_SMALL_V = 1ull << 19;
constexpr int FR_STEP = 4;  // words whose row pointers are loaded together

// `counters`[2] = vectors, [3] = selected vertices (zero before the launch).
// frontier[i] = a selected vertex, voff[i] = offset of its first vector among the selected
// vertices' vectors, vdelta[i] = its first vector's index in the list minus voff[i] (mod 2^32);
// tile_first[t] for the tiles that start in its range.  `skip` leaves out the first vectors of
// every selected vertex (each selected one has more).  A zero gate selects nothing (the bitmaps
// were not written in this phase).  The words from `word0` on.
template <int WORDS>
__global__ void __launch_bounds__(T) k_fr_compact(const unsigned long long* __restrict__ bm1, const unsigned long long* __restrict__ bm2,
                                                  uint64_t V, const uint32_t* __restrict__ rowptr, uint32_t skip,
                                                  const uint32_t* __restrict__ gate, uint32_t* __restrict__ counters,
                                                  uint32_t* __restrict__ frontier, uint32_t* __restrict__ voff,
                                                  uint32_t* __restrict__ vdelta, uint32_t* __restrict__ tile_first, uint64_t word0)
{
    __shared__ uint32_t sn[T / 32], sv[T / 32];
    __shared__ unsigned long long s_base;
    if (gate && *gate == 0u) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t first = word0 + ((uint64_t)blockIdx.x * (T / 32) + warp) * WORDS, word = first + lane;  // bits of vertices [32 word, 32 word + 32)
    uint32_t bits = 0;
    if (lane < WORDS && 32 * word < V) bits = reinterpret_cast<const uint32_t*>(bm1)[word] & reinterpret_cast<const uint32_t*>(bm2)[word];
    if (32 * word + 32 > V && bits) bits &= (1u << (V - 32 * word)) - 1u;
    if (!__syncthreads_or(bits)) return;
    const uint32_t vbase = (uint32_t)(32 * first) + lane;  // this lane's vertex of the warp's word 0
    const unsigned words = __ballot_sync(0xffffffffu, bits != 0);
    // vectors of this lane's vertices in words j .. j + FR_STEP - 1 (0 if not selected), their first in r0
    auto rows = [&](int j, uint32_t* r0, uint32_t* cnt) {
#pragma unroll
        for (int q = 0; q < FR_STEP; ++q) {
            const uint32_t v = vbase + 32u * (j + q);
            r0[q] = cnt[q] = 0;
            if ((__shfl_sync(0xffffffffu, bits, j + q) >> lane) & 1u) {
                r0[q] = rowptr[v];
                cnt[q] = rowptr[v + 1];
            }
        }
#pragma unroll
        for (int q = 0; q < FR_STEP; ++q)
            if (cnt[q]) {
                r0[q] += skip;
                cnt[q] -= r0[q];
            }
    };
    const uint32_t n = __reduce_add_sync(0xffffffffu, (unsigned)__popc(bits));
    uint32_t vec = 0;
    for (int j = 0; j < WORDS; j += FR_STEP) {
        if (!((words >> j) & ((1u << FR_STEP) - 1u))) continue;  // warp-uniform
        uint32_t r0[FR_STEP], cnt[FR_STEP];
        rows(j, r0, cnt);
#pragma unroll
        for (int q = 0; q < FR_STEP; ++q) vec += cnt[q];
    }
    vec = __reduce_add_sync(0xffffffffu, vec);
    if (lane == 0) { sn[warp] = n; sv[warp] = vec; }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t an = 0, av = 0;
        for (int w = 0; w < T / 32; ++w) {
            const uint32_t tn = sn[w], tv = sv[w];
            sn[w] = an; sv[w] = av;
            an += tn; av += tv;
        }
        s_base = atomicAdd(reinterpret_cast<unsigned long long*>(counters + 2), ((unsigned long long)an << 32) | av);
    }
    __syncthreads();
    uint32_t pos = (uint32_t)(s_base >> 32) + sn[warp], vo = (uint32_t)s_base + sv[warp];
    for (int j = 0; j < WORDS; j += FR_STEP) {
        if (!((words >> j) & ((1u << FR_STEP) - 1u))) continue;
        uint32_t r0[FR_STEP], cnt[FR_STEP];
        rows(j, r0, cnt);
#pragma unroll
        for (int q = 0; q < FR_STEP; ++q) {
            const uint32_t b = __shfl_sync(0xffffffffu, bits, j + q);
            if (!b) continue;  // warp-uniform
            uint32_t x = cnt[q];
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            const uint32_t p = pos + __popc(b & ((1u << lane) - 1u)), o = vo + x - cnt[q];
            uint32_t t0 = 0, t1 = 0;  // tiles whose first vector is the entry's
            if ((b >> lane) & 1u) {
                frontier[p] = vbase + 32u * (j + q);
                voff[p] = o;
                vdelta[p] = r0[q] - o;
                t0 = (uint32_t)(((uint64_t)o + PUSH_TILE - 1) / PUSH_TILE);
                t1 = (uint32_t)(((uint64_t)o + cnt[q] + PUSH_TILE - 1) / PUSH_TILE);
                if (t1 - t0 <= 4)
                    for (; t0 < t1; ++t0) tile_first[t0] = p;
            }
            for (unsigned hubs = __ballot_sync(0xffffffffu, t0 < t1); hubs; hubs &= hubs - 1) {  // the warp writes a hub's
                const int h = __ffs(hubs) - 1;
                const uint32_t hp = __shfl_sync(0xffffffffu, p, h), h1 = __shfl_sync(0xffffffffu, t1, h);
                for (uint32_t t = __shfl_sync(0xffffffffu, t0, h) + lane; t < h1; t += 32) tile_first[t] = hp;
            }
            pos += __popc(b);
            vo += __shfl_sync(0xffffffffu, x, 31);
        }
    }
}

// Expand the compacted frontier, one tile of PUSH_TILE vectors at a time (grid-stride over
// tiles; the totals stay on the device).  The tile's owners are staged in shared memory and
// each vector finds its owner by a binary search there.
// Bound by the latency of the random loads and atomics, so those of a vector's four destinations are
// issued together, and the touched list's counter, one address for the whole chip, gets one add per warp
// and vector.  GB300, R-MAT of 2^24 vertices, the largest push of a run
// (with tiles of 1024 vectors before): 422 us one destination after the other, 177 us so.
template <bool IsBfs>
__global__ void __launch_bounds__(T) k_push_expand(const uint32_t* __restrict__ frontier, const uint32_t* __restrict__ voff,
                                                   const uint32_t* __restrict__ vdelta, const uint32_t* __restrict__ tile_first,
                                                   const uint32_t* __restrict__ counters, const uint4* __restrict__ nbr,
                                                   uint32_t V, uint32_t* __restrict__ label,
                                                   unsigned long long* __restrict__ has_next, const unsigned long long* __restrict__ wants,
                                                   uint32_t* __restrict__ cand32, uint32_t* __restrict__ touched,
                                                   uint32_t* __restrict__ ntouched, VoteCfg vc, unsigned long long* __restrict__ vote,
                                                   unsigned long long* __restrict__ chg, uint32_t epoch,
                                                   const uint32_t* __restrict__ epoch_dev)
{
    __shared__ uint32_t s_src[PUSH_TILE];
    __shared__ uint32_t red32[T / 32];
    uint32_t my_min = INF;  // CC: the smallest label written (cc_prev_min of the next iteration)
    __shared__ uint32_t s_off[PUSH_TILE];
    __shared__ uint32_t s_delta[PUSH_TILE];
    __shared__ unsigned long long red[T / 32];
    const uint32_t nf = counters[3], total = counters[2];
    const uint32_t ntiles = (total + PUSH_TILE - 1) / PUSH_TILE;
    unsigned long long my_vote = 0;
    // a tile has at most as many owners as threads: each thread holds one of the next tile's, loaded while
    // this tile is expanded (GB300, 8 BFS by pushes alone on 2^24 vertices 16.56 -> 16.36 ms)
    static_assert(PUSH_TILE == T, "one owner per thread");
    uint32_t first = blockIdx.x < ntiles ? tile_first[blockIdx.x] : nf;
    uint32_t after = (uint64_t)blockIdx.x + gridDim.x < ntiles ? tile_first[blockIdx.x + gridDim.x] : nf;
    uint32_t n_off = 0, n_src = 0, n_delta = 0;
    auto owners = [&](uint32_t from) {
        if (threadIdx.x < nf - from) {
            n_off = voff[from + threadIdx.x];
            n_src = frontier[from + threadIdx.x];
            n_delta = vdelta[from + threadIdx.x];
        }
    };
    owners(first);
    bool full = false;  // BFS: the touched list, as the warp last saw it (it only grows)
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t t0 = tile * PUSH_TILE;
        const uint32_t tend = min(total, t0 + PUSH_TILE);
        // entries first .. first+nw-1 own every vector of the tile (each owns at least one)
        const uint32_t nw = min(PUSH_TILE, nf - first);
        if (threadIdx.x < nw) {
            s_off[threadIdx.x] = n_off;
            s_src[threadIdx.x] = n_src;
            s_delta[threadIdx.x] = n_delta;
        }
        first = after;
        owners(first);
        after = (uint64_t)tile + 2ull * gridDim.x < ntiles ? tile_first[tile + 2 * gridDim.x] : nf;
        __syncthreads();
        for (uint32_t base = t0; base < tend; base += T) {  // warp-uniform trip count
            const uint32_t gv = base + threadIdx.x;
            const bool live = gv < tend;
            uint32_t u = 0;
            uint4 s = make_uint4(INF, INF, INF, INF);
            if (live) {
                int lo = 0, hi = (int)nw - 1;  // last entry with s_off <= gv
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s_off[mid] <= gv) lo = mid; else hi = mid - 1;
                }
                u = s_src[lo];
                s = __ldcs(nbr + (uint32_t)(gv + s_delta[lo]));
            }
            const uint32_t ids[4] = { s.x, s.y, s.z, s.w };
            // the loads, then the atomics, of the four destinations together
            bool ok[4];
            uint32_t old[4];
            if (IsBfs) {
#pragma unroll
                for (int l = 0; l < 4; ++l) ok[l] = ids[l] < V && bit_of(wants, ids[l]);
#pragma unroll
                for (int l = 0; l < 4; ++l) old[l] = ok[l] ? cand32[ids[l]] : 0u;
#pragma unroll
                for (int l = 0; l < 4; ++l) old[l] = u < old[l] ? atomicMin(cand32 + ids[l], u) : 0u;
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    ok[l] = old[l] == INF;  // the first touch
                    if (ok[l]) atomicOr(has_next + (ids[l] >> 6), 1ull << (ids[l] & 63));
                }
                if (!full) full = touched_append4(ok, ids, touched, ntouched, V);
            } else if (live) {
                const uint32_t msg = label[u];
#pragma unroll
                for (int l = 0; l < 4; ++l) old[l] = ids[l] < V ? label[ids[l]] : 0u;
#pragma unroll
                for (int l = 0; l < 4; ++l) old[l] = msg < old[l] ? atomicMin(label + ids[l], msg) : 0u;
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    ok[l] = msg < old[l];
                    if (ok[l]) {
                        my_min = min(my_min, msg);
                        ok[l] = bit_set_first(has_next, ids[l]);
                    }
                }
#pragma unroll
                for (int l = 0; l < 4; ++l)
                    if (ok[l]) my_vote += vc.of(ids[l]);
            }
        }
        __syncthreads();
    }
    if (!IsBfs) {
        my_vote = block_sum_u64(my_vote, red);
        if (threadIdx.x == 0) vote_add(vote, my_vote);
        cc_record_min<T>(my_min, red32, chg, epoch_dev ? *epoch_dev : epoch);
    }
}

// BFS pull over the compacted wanted destinations (WantsInfo and in-vectors): only their vectors
// are read, in tiles of pull_tile vectors.  The vectors of one destination are consecutive in the
// concatenation, so the per-destination minimum candidate (the reference's parent rule, as in
// k_bfs_pull) is reduced within the warp before one atomicMin.
// Early exit: the candidate is (first vector with a frontier source, ~largest such source), so
// once a destination has a candidate, its later vectors cannot win.  Blocks take their first tile
// by number and the next from a queue, asked for while the tile before is worked on (balanced, and a long
// destination's tiles are processed roughly in order; runs of 2, 4 and 8 tiles: CC of 4096 vertices 136,
// 139 and 149 us, single ones 124), and a vector past its destination's first LONG_RUN vectors is
// skipped (no neighbour or frontier reads) when the candidate already names an earlier vector.
// In R-MAT the sources of a destination ascend and the hubs have small IDs, so a long
// destination next to a frontier hub stops after its first vectors.
constexpr uint32_t LONG_RUN = 32;

// Vectors of a tile of the pulls' expansions: one per thread, or four where that still gives every block several
// tiles, for a tile costs a trip to the queue and three barriers whatever its size.  GB300, CC's first pull, tiles of
// 256 / 512 / 1024 / 2048 vectors (of 1024 and two at a time before): uniform 1M vertices of degree 60 341 / 297 / 287 /
// 473 us (305), 3.8M of 42 965 / 801 / 746 / 1252 (810), R-MAT of 2^24 316 / 324 / 317 / 440 (328).
constexpr uint32_t PULL_TILE = 4 * PUSH_TILE;
constexpr uint32_t PULL_MANY = 2;
__device__ __forceinline__ uint32_t pull_tile(uint32_t total, uint32_t blocks)
{
    return total / (PULL_MANY * PULL_TILE) >= blocks ? PULL_TILE : PUSH_TILE;
}

__global__ void __launch_bounds__(T) k_bfs_pull_expand(const uint32_t* __restrict__ dests, const uint32_t* __restrict__ voff,
                                                       const uint32_t* __restrict__ vdelta, const uint32_t* __restrict__ tile_first,
                                                       const uint32_t* __restrict__ counters, const uint4* __restrict__ nbr,
                                                       uint32_t V, const unsigned long long* __restrict__ has,
                                                       unsigned long long* __restrict__ cand, uint32_t* __restrict__ touched,
                                                       uint32_t* __restrict__ ntouched, const uint32_t* __restrict__ hub_vid,
                                                       uint32_t nhub, unsigned long long* __restrict__ has_next,
                                                       uint32_t* __restrict__ queue)
{
    __shared__ uint32_t s_dst[PULL_TILE];
    __shared__ uint32_t s_off[PULL_TILE];
    __shared__ uint32_t s_delta[PULL_TILE];
    __shared__ uint32_t s_tile;
    __shared__ bool s_full;  // the touched list is long enough for the visit to sweep (read per tile)
    const uint32_t nd = counters[3], total = counters[2], span = pull_tile(total, gridDim.x);
    const uint32_t ntiles = (total + span - 1) / span;
    const int lane = threadIdx.x & 31;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile = s_tile) {
        uint32_t next = 0;
        if (threadIdx.x == 0) next = atomicAdd(queue, 1u) + gridDim.x;
        const uint32_t t0 = tile * span, first = tile_first[t0 / PUSH_TILE];
        const uint32_t tend = min(total, t0 + span);
        const uint32_t nw = min(span, nd - first);
        for (uint32_t i = threadIdx.x; i < nw; i += T) {
            s_off[i] = voff[first + i];
            s_dst[i] = dests[first + i];
            s_delta[i] = vdelta[first + i];
        }
        if (threadIdx.x == 0) s_full = touched_full(ntouched, V);
        __syncthreads();
        for (uint32_t base = t0; base < tend; base += T) {  // warp-uniform trip count
            const uint32_t gv = base + threadIdx.x;
            uint32_t key = INF;
            unsigned long long k = ~0ull;
            if (gv < tend) {
                int lo = 0, hi = (int)nw - 1;  // last entry with s_off <= gv
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s_off[mid] <= gv) lo = mid; else hi = mid - 1;
                }
                key = s_dst[lo];
                const uint32_t vec = gv + s_delta[lo];
                bool skip = false;
                if (gv >= s_off[lo] + LONG_RUN) {
                    const unsigned long long c = __ldcg(cand + key);  // atomics of other blocks land in L2
                    skip = c != ~0ull && (uint32_t)(c >> 32) < vec;
                }
                if (!skip) {
                    const uint4 s = __ldcs(nbr + vec);
                    const uint32_t ids[4] = { grz_hub_decode(s.x, hub_vid, nhub), grz_hub_decode(s.y, hub_vid, nhub),
                                              grz_hub_decode(s.z, hub_vid, nhub), grz_hub_decode(s.w, hub_vid, nhub) };
                    uint32_t best = 0;
                    bool any = false;
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        const uint32_t id = ids[l];
                        if (id < V && bit_of(has, id)) {
                            best = any ? max(best, id) : id;
                            any = true;
                        }
                    }
                    if (any) k = ((unsigned long long)vec << 32) | (unsigned long long)(~best);
                }
            }
            if (!__any_sync(0xffffffffu, k != ~0ull)) continue;  // no frontier source in the warp's vectors
            const uint32_t prevkey = __shfl_up_sync(0xffffffffu, key, 1);
            const uint32_t nextkey = __shfl_down_sync(0xffffffffu, key, 1);
            const bool head = lane == 0 || key != prevkey;
            const bool tail = lane == 31 || key != nextkey;
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            const int segstart = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
            const int maxlen = __reduce_max_sync(0xffffffffu, (unsigned)(lane - segstart + 1));
            for (int off = 1; off < maxlen; off <<= 1) {
                const unsigned long long o = __shfl_up_sync(0xffffffffu, k, off);
                if (lane - off >= segstart) k = min(k, o);
            }
            bool first_touch = false;
            if (tail && k != ~0ull && k < cand[key]) {
                first_touch = atomicMin(cand + key, k) == ~0ull;
                if (first_touch) atomicOr(has_next + (key >> 6), 1ull << (key & 63));
            }
            touched_append(first_touch, key, touched, ntouched, s_full);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_tile = next;
        __syncthreads();
    }
}

// CC pull over the remaining vectors of the destinations k_cc_pull_first left open (label above 0
// after their first vector), compacted with their vector ranges as the BFS pull's are (the same
// tiles, queue and binary search as k_bfs_pull_expand).  A vector whose destination reached 0
// meanwhile needs no gathers; the others take the minimum of their lanes' labels (lane 0 first),
// reduced per destination within the warp, and the run's last lane lowers the label in place.
__global__ void __launch_bounds__(T) k_cc_pull_expand(const uint32_t* __restrict__ dests, const uint32_t* __restrict__ voff,
                                                      const uint32_t* __restrict__ vdelta, const uint32_t* __restrict__ tile_first,
                                                      const uint32_t* __restrict__ counters, const uint4* __restrict__ nbr,
                                                      uint32_t V, uint32_t* __restrict__ label, const uint32_t* __restrict__ hub_vid,
                                                      uint32_t nhub, unsigned long long* __restrict__ has_next, VoteCfg vc,
                                                      unsigned long long* __restrict__ vote, unsigned long long* __restrict__ chg,
                                                      uint32_t epoch, const uint32_t* __restrict__ epoch_dev,
                                                      uint32_t* __restrict__ queue, unsigned long long* __restrict__ work)
{
    __shared__ uint32_t s_dst[PULL_TILE];
    __shared__ uint32_t s_off[PULL_TILE];
    __shared__ uint32_t s_delta[PULL_TILE];
    __shared__ uint32_t s_tile;
    __shared__ unsigned long long red[T / 32];
    __shared__ uint32_t red32[T / 32];
    const uint32_t ep = epoch_dev ? *epoch_dev : epoch;
    const uint32_t nd = counters[3], total = counters[2], span = pull_tile(total, gridDim.x);
    const uint32_t ntiles = (total + span - 1) / span;
    const int lane = threadIdx.x & 31;
    unsigned long long my_vote = 0, my_vecs = 0;
    uint32_t my_min = INF;
    auto fetch = [&](uint32_t xl) -> uint32_t {
        const uint32_t sl = xl - GRZ_HUB_BASE;
        const uint32_t id = sl < nhub ? __ldg(hub_vid + sl) : min(xl, V);
        return ld_label(label + id);
    };
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile = s_tile) {
        uint32_t next = 0;
        if (threadIdx.x == 0) next = atomicAdd(queue, 1u) + gridDim.x;
        const uint32_t t0 = tile * span, first = tile_first[t0 / PUSH_TILE];
        const uint32_t tend = min(total, t0 + span);
        const uint32_t nw = min(span, nd - first);
        for (uint32_t i = threadIdx.x; i < nw; i += T) {
            s_off[i] = voff[first + i];
            s_dst[i] = dests[first + i];
            s_delta[i] = vdelta[first + i];
        }
        __syncthreads();
        for (uint32_t base = t0; base < tend; base += T) {  // warp-uniform trip count
            const uint32_t gv = base + threadIdx.x;
            uint32_t key = INF, m = INF;
            if (gv < tend) {
                int lo = 0, hi = (int)nw - 1;  // last entry with s_off <= gv
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s_off[mid] <= gv) lo = mid; else hi = mid - 1;
                }
                key = s_dst[lo];
                if (ld_label(label + key) != 0) {
                    ++my_vecs;
                    const uint4 sv = ld_stream(nbr + (uint32_t)(gv + s_delta[lo]));
                    m = fetch(sv.x);
                    if (m != 0) m = min(m, min(min(fetch(sv.y), fetch(sv.z)), fetch(sv.w)));
                }
            }
            if (!__any_sync(0xffffffffu, m != INF)) continue;
            const uint32_t prevkey = __shfl_up_sync(0xffffffffu, key, 1);
            const uint32_t nextkey = __shfl_down_sync(0xffffffffu, key, 1);
            const bool head = lane == 0 || key != prevkey;
            const bool tail = lane == 31 || key != nextkey;
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            const int segstart = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
            const int maxlen = __reduce_max_sync(0xffffffffu, (unsigned)(lane - segstart + 1));
            for (int off = 1; off < maxlen; off <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, m, off);
                if (lane - off >= segstart) m = min(m, o);
            }
            if (tail && m != INF && m < ld_label(label + key)) {
                const uint32_t old = atomicMin(label + key, m);
                if (m < old) {
                    my_min = min(my_min, m);
                    if (bit_set_first(has_next, key)) my_vote += vc.of(key);
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) s_tile = next;
        __syncthreads();
    }
    my_vote = block_sum_u64(my_vote, red);
    if (threadIdx.x == 0) vote_add(vote, my_vote);
    __syncthreads();
    if (work) {  // profiling: vectors read, by kind of iteration
        uint32_t mp = 0;
        const int slot = cc_prev_min(chg, ep, &mp) ? 1 : 0;
        my_vecs = block_sum_u64(my_vecs, red);
        if (threadIdx.x == 0 && my_vecs) atomicAdd(work + slot, my_vecs);
        __syncthreads();
    }
    cc_record_min<T>(my_min, red32, chg, ep);
}

// BFS pull, early-exit pass.  Every in-neighbour of a wanted (unvisited) destination that has been
// visited is in the frontier (it was visited in the previous iteration, else it would have
// visited the destination already), so in the big pull iterations most wanted destinations find
// a frontier source in their first vector.  Each wanted destination reads its first `first_n`
// vectors in order and stops at the first one with a frontier source; that vector's largest
// frontier source is its parent, which is the full scan's rule (smallest vector index, then
// largest source) because no earlier vector has one.  A destination decided here is visited here
// (parent, level, WantsInfo cleared, HasInfo* set, vote), so it needs no candidate word and no
// place in the touched list, whose single counter would serialise millions of appends.  One
// still undecided that has more vectors is marked in `unres`, and the tiled pass
// (k_bfs_pull_expand, then k_bfs_visit) reads the rest of its vectors.  A warp owns FW whole
// bitmap words (64 destinations each; lane l of slot q holds destination 64 w0 + 32 q + l), so
// it writes their WantsInfo, HasInfo* and unres words without atomics, and the first-vector
// loads of its 2 FW slots are issued together.  Where at most 32 of the 64 FW destinations are
// wanted, each lane takes one of them instead (late pulls: bound by instructions spent on empty
// slots).  GB300, R-MAT of 2^24 vertices, the pulls of one run: 156, 65 and 42 us with slots only,
// 154, 45 and 22 us so.  The first is near what its row pointers, first vectors, degrees, parents and
// levels take at the memory's rate (106 us); probing the frontier bits in two or four steps, loading a
// word ahead, and 1 or 4 words per warp gave nothing.

__global__ void __launch_bounds__(T, GRZ_BFS_MINB) k_bfs_pull_first(unsigned long long* __restrict__ wants,
                                                      const unsigned long long* __restrict__ nonempty,
                                                      const uint32_t* __restrict__ rowptr, const uint4* __restrict__ nbr,
                                                      uint32_t V, uint64_t W, const unsigned long long* __restrict__ has,
                                                      const uint32_t* __restrict__ hub_vid, uint32_t nhub,
                                                      unsigned long long* __restrict__ has_next,
                                                      unsigned long long* __restrict__ unres, uint32_t first_n,
                                                      uint32_t* __restrict__ parent, uint32_t* __restrict__ level,
                                                      uint32_t iter_host, const uint32_t* __restrict__ iter_dev, VoteCfg vc,
                                                      unsigned long long* __restrict__ vote)
{
    __shared__ unsigned long long red[T / 32];
    __shared__ uint8_t s_bit[T / 32][32];
    constexpr int Q = 2 * FW;
    const int lane = threadIdx.x & 31;
    uint8_t* const bit_at = s_bit[threadIdx.x >> 5];
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t iter = iter_dev ? *iter_dev : iter_host;
    unsigned long long my_vote = 0;
    // the largest frontier source of vector `vec`, or INF without one
    auto vec_best = [&](uint32_t vec) -> uint32_t {
        const uint4 s = __ldcs(nbr + vec);
        const uint32_t ids[4] = { grz_hub_decode(s.x, hub_vid, nhub), grz_hub_decode(s.y, hub_vid, nhub),
                                  grz_hub_decode(s.z, hub_vid, nhub), grz_hub_decode(s.w, hub_vid, nhub) };
        bool in[4];
#pragma unroll
        for (int l = 0; l < 4; ++l) in[l] = ids[l] < V && bit_of(has, ids[l]);
        // (the sources of a list that is only grouped come in any order)
        uint32_t best = 0;  // source + 1
#pragma unroll
        for (int l = 0; l < 4; ++l) best = max(best, in[l] ? ids[l] + 1 : 0u);
        return best - 1;
    };
    auto visit = [&](uint32_t v, uint32_t p) {
        parent[v] = p;
        level[v] = iter;
        my_vote += vc.of(v);
    };
    const uint64_t nwarps = (uint64_t)gridDim.x * (T / 32);
    for (uint64_t w0 = ((uint64_t)blockIdx.x * (T / 32) + (threadIdx.x >> 5)) * FW; w0 < W; w0 += nwarps * FW) {  // warp-uniform
        // bit `lane` of word q: destination 64 w0 + 32 q + lane (words past the bitmap are empty)
        uint32_t sel[Q], total = 0;
#pragma unroll
        for (int f = 0; f < FW; ++f) {
            const unsigned long long x = w0 + f < W ? wants[w0 + f] & nonempty[w0 + f] : 0ull;
            sel[2 * f] = (uint32_t)x;
            sel[2 * f + 1] = (uint32_t)(x >> 32);
            total += __popcll(x);
        }
        uint32_t hn[Q], un[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) hn[q] = un[q] = 0u;
        if (total > 32) {
            uint32_t r0[Q], n[Q], p[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const uint64_t v = 64 * w0 + 32 * (uint64_t)q + lane;
                n[q] = 0;
                if ((sel[q] >> lane) & 1u) {
                    r0[q] = rowptr[v];
                    n[q] = rowptr[v + 1] - r0[q];
                }
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) p[q] = n[q] ? vec_best(r0[q]) : INF;
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const uint32_t m = min(n[q], first_n);
                for (uint32_t j = 1; j < m && p[q] == INF; ++j) p[q] = vec_best(r0[q] + j);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const bool hit = p[q] != INF;
                if (hit) visit((uint32_t)(64 * w0 + 32 * (uint64_t)q + lane), p[q]);
                hn[q] = __ballot_sync(0xffffffffu, hit);
                un[q] = __ballot_sync(0xffffffffu, !hit && n[q] > first_n);
            }
        } else if (total) {
            // few: lane i takes the i-th
            uint32_t base = 0;
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                if ((sel[q] >> lane) & 1u) bit_at[base + __popc(sel[q] & below)] = (uint8_t)(32 * q + lane);
                base += __popc(sel[q]);
            }
            __syncwarp();
            uint32_t bit = 0, p = INF, n = 0;
            if (lane < total) {
                bit = bit_at[lane];
                const uint32_t v = (uint32_t)(64 * w0) + bit, r0 = rowptr[v];
                n = rowptr[v + 1] - r0;
                const uint32_t m = min(n, first_n);
                for (uint32_t j = 0; j < m && p == INF; ++j) p = vec_best(r0 + j);
                if (p != INF) visit(v, p);
            }
            const bool hit = p != INF, open = !hit && n > first_n;
            if (__any_sync(0xffffffffu, hit || open)) {
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const uint32_t m = (int)(bit >> 5) == q ? 1u << (bit & 31u) : 0u;
                    hn[q] = __reduce_or_sync(0xffffffffu, hit ? m : 0u);
                    un[q] = __reduce_or_sync(0xffffffffu, open ? m : 0u);
                }
            }
        }
        if (lane == 0) {
#pragma unroll
            for (int f = 0; f < FW; ++f) {
                if (w0 + f >= W) break;
                const unsigned long long h = (unsigned long long)hn[2 * f + 1] << 32 | hn[2 * f];
                unres[w0 + f] = (unsigned long long)un[2 * f + 1] << 32 | un[2 * f];
                if (h) {
                    has_next[w0 + f] |= h;
                    wants[w0 + f] &= ~h;
                }
            }
        }
        __syncwarp();
    }
    my_vote = block_sum_u64(my_vote, red);
    if (threadIdx.x == 0) vote_add(vote, my_vote);
}

// Calls f(vertex, whether it is marked, load(vertex) if it is, half) for the vertices of every nonzero word
// word(i), i < W, a warp per word, first the lower then the upper 32 vertices (f is called by whole warps);
// g(word, bits) once after each.  A warp looks at `span` words and takes MARK_WORDS nonzero ones at a time,
// whose vertices it loads for first (one after the other, each a trip to memory, the pass after a run of
// small iterations that had marked most of 100k vertices took 27.6 us, so 4.4 us; 2 words keep more warps
// resident than 4).  A map of few words is spread over more warps; a large one is nearly empty, and 32 words
// are one load.
constexpr int MARK_WORDS = 2;
constexpr uint64_t MARK_SPAN_W = 1u << 15;
__host__ __device__ constexpr int mark_span(uint64_t W) { return W < MARK_SPAN_W ? 4 : 32; }
template <typename M, typename C, typename F, typename G>
__device__ __forceinline__ void for_marked(M word, uint64_t W, C load, F f, G g)
{
    const int lane = threadIdx.x & 31, span = mark_span(W);
    const uint64_t nwarps = (uint64_t)gridDim.x * (T / 32);
    for (uint64_t w0 = span * ((uint64_t)blockIdx.x * (T / 32) + (threadIdx.x >> 5)); w0 < W; w0 += span * nwarps) {
        const unsigned long long mine = lane < span && w0 + lane < W ? word(w0 + lane) : 0ull;
        unsigned nz = __ballot_sync(0xffffffffu, mine != 0);
        while (nz) {  // warp-uniform
            unsigned long long bits[MARK_WORDS], c[2 * MARK_WORDS];
            uint32_t at[MARK_WORDS];
#pragma unroll
            for (int j = 0; j < MARK_WORDS; ++j) {
                const int i = nz ? __ffs(nz) - 1 : 0;
                bits[j] = __shfl_sync(0xffffffffu, mine, i);
                if (!nz) bits[j] = 0ull;
                at[j] = (uint32_t)(w0 + i);
                nz &= nz - 1;
            }
#pragma unroll
            for (int j = 0; j < 2 * MARK_WORDS; ++j)
                c[j] = (bits[j / 2] >> (32 * (j & 1) + lane)) & 1ull ? load(64 * at[j / 2] + 32 * (j & 1) + lane) : 0ull;
#pragma unroll
            for (int j = 0; j < 2 * MARK_WORDS; ++j) {
                if (!bits[j / 2]) break;
                f(64 * at[j / 2] + 32 * (j & 1) + lane, ((bits[j / 2] >> (32 * (j & 1) + lane)) & 1ull) != 0, c[j], j & 1);
                if ((j & 1) && lane == 0) g(at[j / 2], bits[j / 2]);
            }
        }
    }
}

// BFS: visit the touched destinations (pull: decode the winning (vector, source) key; push: the
// smallest source), in one pass over the touched list
template <bool FromPull>
__global__ void __launch_bounds__(T) k_bfs_visit(const uint32_t* __restrict__ touched, const uint32_t* __restrict__ ntouched,
                                                 unsigned long long* __restrict__ cand64, uint32_t* __restrict__ cand32,
                                                 uint32_t* __restrict__ parent, uint32_t* __restrict__ level, uint32_t iter_host,
                                                 const uint32_t* __restrict__ iter_dev,
                                                 unsigned long long* __restrict__ wants, const unsigned long long* __restrict__ has_next,
                                                 VoteCfg vc, unsigned long long* __restrict__ vote, uint32_t V)
{
    __shared__ unsigned long long red[T / 32];
    const uint32_t n = *ntouched;
    const uint32_t iter = iter_dev ? *iter_dev : iter_host;
    unsigned long long my_vote = 0;
    auto visit = [&](uint32_t d) {
        uint32_t p;
        if (FromPull) {
            p = ~(uint32_t)(cand64[d] & 0xffffffffull);
            cand64[d] = ~0ull;
        } else {
            p = cand32[d];
            cand32[d] = INF;
        }
        parent[d] = p;
        level[d] = iter;
        my_vote += vc.of(d);
    };
    if ((uint64_t)n * VISIT_DENSE_RATIO <= V) {
        // few: the touched list (first-touch order)
        for (uint32_t i = blockIdx.x * T + threadIdx.x; i < n; i += gridDim.x * T) {
            const uint32_t d = touched[i];
            visit(d);
            atomicAnd(wants + (d >> 6), ~(1ull << (d & 63)));
        }
    } else {
        // many: every word of vertices.  A vertex was touched in this call when its HasInfo* bit is set
        // (at first touch) and its WantsInfo bit still is (a caller's earlier vector range of this
        // iteration visited and cleared its own).  Its candidate and out-degree are loaded together.
        // GB300, R-MAT of 2^24 vertices, a run's large visit until the next kernel starts: 37.8 us with a look
        // at every vertex, 26.9 us over the nonzero words.
        for_marked(
            [&](uint64_t w) { return has_next[w] & wants[w]; }, (uint64_t)V / 64 + 1,
            [&](uint32_t d) {
                const uint32_t p = FromPull ? ~(uint32_t)cand64[d] : cand32[d];
                return (unsigned long long)(vc.without_outdeg ? 0u : vc.degree[d]) << 32 | p;
            },
            [&](uint32_t d, bool marked, unsigned long long c, int) {
                if (!marked) return;
                if (FromPull) cand64[d] = ~0ull; else cand32[d] = INF;
                parent[d] = (uint32_t)c;
                level[d] = iter;
                my_vote += (vc.without_count ? 0ull : 1ull) + (c >> 32);
            },
            [&](uint64_t w, unsigned long long bits) { wants[w] &= ~bits; });
    }
    my_vote = block_sum_u64(my_vote, red);
    if (threadIdx.x == 0) vote_add(vote, my_vote);
}

// ---------------------------------------------------------------------------------------------
// Small iterations, many per launch.
//
// A frontier of a few hundred vertices leaves the chip idle: an iteration of the run graph costs
// about 21 us in kernel starts whatever its size, and a road network or any long tail has a
// thousand of them.  One cluster of 16 blocks runs such iterations back to back, with the frontier's
// vectors listed in its shared memory, until the frontier is empty or too large (GRZ_HOP_VOTE),
// the policy chooses an engine it does not stand in for, or a bound of the run is reached; the last
// iteration is left to the decision kernel, as if the engine's kernels had run it.  A cluster,
// because one SM takes one gather per clock, and a frontier of 10k edges needs four for each.  GB300, BFS of 764 levels on a mesh of 250k
// vertices (7 kernels per level -> one block -> this): 29 -> 4.0 -> 2.2 ms.
//
// An iteration is one pass over the listed vectors and one cluster barrier.  BFS: a destination's
// candidate is (iteration << 33 | pull << 32 | source), lowered by atomicMin in cand64.  The
// iteration number makes the candidates of earlier iterations win, so a destination keeps its first
// iteration and, within it, the smallest source; no visit pass separates the iterations.  The
// destination whose candidate was empty is new: its vectors are listed for the next iteration, in the
// shared memory of the block that found it (when a list outgrows one step of its block, the next
// iteration shares all lists evenly, reading the other blocks').  That source is the push engine's parent.  A pull visits the same
// destinations (every unvisited one with a frontier source), so a small pull runs the same way, and
// only the parent differs: the largest frontier source of the first vector that holds one.  Where
// sources ascend along the list that vector is the smallest frontier source's, found by a binary
// search once all levels are known (k_hop_visit, k_hop_parents).  CC: labels are lowered in place,
// as k_push_expand does, and a lowered destination is listed once per iteration (the first to lower
// its stamp, cand32, to the iteration's); a pull is left to the pull kernels.  Votes, engine choice,
// iteration numbers and the smallest label written are those of single iterations.  The vertices
// that were listed are marked in `map`, from which k_hop_visit / k_hop_labels write what outlives the
// launch (the last frontier's HasInfo* among it) and empty the scratch arrays.
//
// What an iteration waits for is a chain of round trips (GB300, clocks: L2 300-450, an atomic 500-850,
// shared memory of another block 400, cluster barrier 480), so a thread takes one edge, not a
// vector of four whose branches would wait in turn, and nothing that is not needed is outstanding
// when the barrier is reached: its release waits for every write to arrive, and with reductions to
// global memory on their way it takes 2200 clocks instead of 480.  The marks are therefore set by
// the iteration after, at its start.
constexpr int HOP_CTAS = 16;
constexpr int HOP_T = 512;
constexpr uint32_t HOP_CAP = 8192;  // listed vectors per block: twice an even share
constexpr uint32_t HOP_STEP = HOP_T / 4;  // vectors a block takes in one step
constexpr size_t HOP_SMEM = sizeof(uint32_t) * HOP_CAP * 4;  // two lists of vectors and their sources

struct HopIn {
    const uint4* nbr;                   // push list
    const uint32_t* rowptr;
    const uint32_t* degree;
    uint32_t V;
    double dV, dE, max_degree;
    const unsigned long long* wants;    // BFS
    unsigned long long* cand64;         // BFS: all ~0 before, and again after the kernels that follow
    uint32_t* cand32;                   // CC: likewise
    uint32_t* label;                    // CC
    unsigned long long* map;            // all zero before, and again after the kernels that follow
    const uint32_t* list;               // the frontier's vertices (ctl->hop_n of them)
    unsigned long long* vote;
    unsigned long long* chg;            // CC
    grz_runctl* ctl;
    int pulls;                          // small pulls run here too (BFS over ascending lists)
};

// an iteration's totals
struct __align__(16) HopPart {
    uint32_t vote_lo, vote_hi;  // vote = vote_lo + 2^16 vote_hi
    uint32_t verts;             // vertices of the next frontier
    uint32_t flags;             // HOP_OVER, HOP_LATE
    uint32_t min;               // CC: smallest label written
    uint32_t items;             // vectors the block has listed
    uint32_t pad[2];
};
constexpr uint32_t HOP_OVER = 1u, HOP_LATE = 2u;
constexpr uint32_t HOP_FIRST = 0x80000000u;  // of a listed source: this vector marks it in `map`
constexpr uint32_t HOP_NOVEC = 0xffffffffu;  // a vertex without vectors, listed to be marked

// the warp's totals of every lane's x, in all lanes
__device__ __forceinline__ HopPart hop_reduce(HopPart x)
{
    x.vote_lo = __reduce_add_sync(0xffffffffu, x.vote_lo);
    x.vote_hi = __reduce_add_sync(0xffffffffu, x.vote_hi);
    x.verts = __reduce_add_sync(0xffffffffu, x.verts);
    x.flags = __reduce_or_sync(0xffffffffu, x.flags);
    x.min = __reduce_min_sync(0xffffffffu, x.min);
    return x;
}

__device__ __forceinline__ HopPart hop_zero()
{
    HopPart x;
    x.vote_lo = x.vote_hi = x.verts = x.flags = x.items = 0;
    x.min = INF;
    return x;
}

// the cluster's totals of every thread's x, after a cluster barrier; s_block (zeroed) and s_part are not
// those of the call before.  s_part[r].items = *items of block r.
__device__ __forceinline__ HopPart hop_exchange(cg::cluster_group& cl, HopPart x, const uint32_t* items, HopPart* s_block, HopPart* s_part)
{
    const int lane = threadIdx.x & 31;
    if (__any_sync(0xffffffffu, x.vote_lo != 0 || x.vote_hi != 0 || x.flags != 0 || x.min != INF)) {
        x = hop_reduce(x);
        if (lane == 0) {
            atomicAdd(&s_block->vote_lo, x.vote_lo & 0xffffu);
            atomicAdd(&s_block->vote_hi, x.vote_hi + (x.vote_lo >> 16));
            atomicAdd(&s_block->verts, x.verts);
            if (x.flags) atomicOr(&s_block->flags, x.flags);
            if (x.min != INF) atomicMin(&s_block->min, x.min);
        }
    }
    __syncthreads();
    if (threadIdx.x < HOP_CTAS) {
        HopPart y = *s_block;
        y.items = *items;
        *cl.map_shared_rank(s_part + cl.block_rank(), threadIdx.x) = y;
    }
    cl.sync();
    return hop_reduce(lane < HOP_CTAS ? s_part[lane] : hop_zero());
}

// (started by the decision kernel when the next iteration's vote is at most GRZ_HOP_VOTE)
// Vectors of a vertex that its lane lists by itself; its warp lists more.  A hub's thousands of vectors listed
// by one lane held up all 16 blocks: GB300, first small iterations of a BFS on 2^24 R-MAT vertices 58 -> 10 us.
constexpr uint32_t HOP_NARROW = 4;
// Vectors of a vertex of the starting frontier that its thread lists by itself; all blocks share the listing
// of more.  A run of 32 takes about 1 us, and a root's 16000 vectors one after the other took longer than the
// iteration they saved: GB300, BFS from a root of degree 64722 on 2^20 R-MAT
// vertices 499 -> 208 us (285 without k_hop).
constexpr uint32_t HOP_WIDE = 128;
constexpr uint32_t HOP_MAX_WIDE = GRZ_HOP_VOTE / (4 * HOP_WIDE);  // more than 128 full vectors each, but for the last

template <bool IsBfs>
__global__ void __cluster_dims__(HOP_CTAS, 1, 1) __launch_bounds__(HOP_T, 1) k_hop(const HopIn in)
{
    extern __shared__ uint32_t s_mem[];
    __shared__ uint32_t s_items[4];  // vectors listed for an iteration, by its number mod 4
    __shared__ HopPart s_block[2], s_part[2][HOP_CTAS];
    __shared__ uint32_t s_nwide, s_wide[HOP_MAX_WIDE];  // (block 0's)
    __shared__ int s_pull;
    __shared__ float s_f[NF], s_par[MLP_WARP_FLOATS];
    cg::cluster_group cl = cg::this_cluster();
    grz_runctl* const ctl = in.ctl;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t rank = cl.block_rank();
    const uint32_t n0 = ctl->hop_n;
    if (tid < 4) s_items[tid] = 0;
    if (tid == 0) s_nwide = 0;
    if (tid < 2) s_block[tid] = hop_zero();
    const uint32_t level0 = ctl->level, max_level = ctl->max_level, mode0 = ctl->engine;
    const int force = ctl->force;
    const float* params = ctl->params;
    const double threshold = ctl->threshold;
    const unsigned long long t0 = ctl->t0_ns, limit = ctl->limit_ns, unvisited = ctl->unvisited;
    if (params) mlp_stage(params, s_par, tid, HOP_T);
    cl.sync();
    // The starting frontier's vectors, spread over the blocks in runs of at most 32, a full list's over
    // the next ones: they are fewer than the vote, which is half of what the lists hold.
    HopPart sum = hop_zero();
    auto place = [&](uint32_t d, uint32_t r, uint32_t k, uint32_t to) {
        for (int tries = 0; tries < 64; ++tries, to = (to + 1) & (HOP_CTAS - 1)) {
            const uint32_t at = atomicAdd(cl.map_shared_rank(&s_items[0], to), k);
            uint32_t* vec = cl.map_shared_rank(s_mem, to);
            if (at + k <= HOP_CAP) {
                for (uint32_t q = 0; q < k; ++q) { vec[at + q] = r + q; vec[HOP_CAP + at + q] = d; }
                return;
            }
            for (uint32_t q = at; q < HOP_CAP; ++q) { vec[q] = HOP_NOVEC; vec[HOP_CAP + q] = 0; }  // the places no one takes
        }
    };
    for (uint32_t i = rank + HOP_CTAS * tid; i < n0; i += HOP_CTAS * HOP_T) {
        const uint32_t d = in.list[i], r0 = __ldg(in.rowptr + d), n = __ldg(in.rowptr + d + 1) - r0;
        if (n > HOP_WIDE) {
            const uint32_t w = atomicAdd(cl.map_shared_rank(&s_nwide, 0), 1u);
            if (w < HOP_MAX_WIDE) {
                *cl.map_shared_rank(s_wide + w, 0) = d;
                continue;
            }
        }
        for (uint32_t j = 0, to = rank + tid; j < n; j += 32, ++to) place(d, r0 + j, min(32u, n - j), to & (HOP_CTAS - 1));
    }
    cl.sync();  // other blocks have added to this one's list
    const uint32_t nwide = min(*cl.map_shared_rank(&s_nwide, 0), HOP_MAX_WIDE);
    if (nwide) {
        for (uint32_t w = tid >> 5; w < nwide; w += HOP_T / 32) {  // a warp of every block, a lane per run
            const uint32_t d = *cl.map_shared_rank(s_wide + w, 0), r0 = __ldg(in.rowptr + d), n = __ldg(in.rowptr + d + 1) - r0;
            for (uint32_t j = 32 * (((rank - w) & (HOP_CTAS - 1)) + HOP_CTAS * lane); j < n; j += 32 * HOP_CTAS * 32)
                place(d, r0 + j, min(32u, n - j), rank);
        }
        cl.sync();
    }
    hop_exchange(cl, sum, &s_items[0], &s_block[1], s_part[1]);
    // lists the vectors [r0, r0 + n) of the lanes' vertices d that are `fresh` in this block's list q (by
    // whole warps, which share the writing of long ranges); false for those that it has no room for
    auto append = [&](int q, int slot, bool fresh, uint32_t d, uint32_t r0, uint32_t n) -> bool {
        const uint32_t k = fresh ? max(n, 1u) : 0u, at = fresh ? atomicAdd(&s_items[slot], k) : 0u;
        uint32_t* vec = s_mem + q * 2 * HOP_CAP;
        const bool fits = at <= HOP_CAP && k <= HOP_CAP - at;
        if (fresh && !fits) {
            atomicOr(in.map + (d >> 6), 1ull << (d & 63));
            for (uint32_t i = at; i < HOP_CAP; ++i) vec[HOP_CAP + i] = 0;  // places no one takes carry no mark
        }
        const bool wide = fresh && fits && k > HOP_NARROW;
        if (fresh && fits && !wide)
            for (uint32_t i = 0; i < k; ++i) {
                vec[at + i] = n ? r0 + i : HOP_NOVEC;
                vec[HOP_CAP + at + i] = i == 0 ? d | HOP_FIRST : d;
            }
        for (unsigned todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1) {
            const int h = __ffs(todo) - 1;
            const uint32_t hk = __shfl_sync(0xffffffffu, k, h), ha = __shfl_sync(0xffffffffu, at, h);
            const uint32_t hr = __shfl_sync(0xffffffffu, r0, h), hd = __shfl_sync(0xffffffffu, d, h);
            for (uint32_t i = lane; i < hk; i += 32) {
                vec[ha + i] = hr + i;
                vec[HOP_CAP + ha + i] = i == 0 ? hd | HOP_FIRST : hd;
            }
        }
        return fits;
    };
    uint32_t it = 0, mode = mode0, pulls = 0;     // iterations finished, this one's engine, pulls before it
    unsigned long long left = unvisited, vote;    // BFS: vertices not visited yet
    for (;; ++it) {
        const int p = it & 1, nxt = (it + 1) & 3;
        const uint32_t level = level0 + it;
        // this block's share: its own list, or every 16th vector of all lists when one is longer than a step
        const uint32_t theirs = lane < HOP_CTAS ? min(s_part[p ^ 1][lane].items, HOP_CAP) : 0u;
        const bool own = __reduce_max_sync(0xffffffffu, theirs) <= HOP_STEP;
        uint32_t m = __shfl_sync(0xffffffffu, theirs, (int)rank), before = theirs;
        if (!own) {
            for (int o = 1; o < HOP_CTAS; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += y;  // vectors of the lists up to this lane's
            }
            m = __shfl_sync(0xffffffffu, before, HOP_CTAS - 1);
        }
        if (tid == 0) {
            s_items[(it + 2) & 3] = 0;
            s_block[p ^ 1] = hop_zero();
        }
        sum = hop_zero();
        // a timer read is slow
        if (rank == 0 && tid == 0 && (it & 15) == 0 && now_ns() - t0 > limit) sum.flags = HOP_LATE;
        const uint32_t l = tid & 3;  // this thread's lane of its vectors
        const uint32_t every = own ? 1 : HOP_CTAS, shift = own ? 0 : rank;
        for (uint32_t k0 = (tid - lane) >> 2; k0 * every < m; k0 += HOP_STEP) {  // warp-uniform
            uint32_t at = (k0 + (lane >> 2)) * every + shift, from = rank;
            const bool in_list = at < m;
            if (!own) {  // the list that holds vector `at` of all
                from = 0;
#pragma unroll
                for (int r = 0; r < HOP_CTAS - 1; ++r) from += at >= __shfl_sync(0xffffffffu, before, r);
                const uint32_t b = __shfl_sync(0xffffffffu, before, from ? (int)from - 1 : 0);
                if (from) at -= b;
            }
            uint32_t u = 0, d = INF;
            if (in_list) {
                const uint32_t* vec = cl.map_shared_rank(s_mem + p * 2 * HOP_CAP, from);
                const uint32_t us = vec[HOP_CAP + at], v = vec[at];
                u = us & ~HOP_FIRST;
                if ((us & HOP_FIRST) && l == 0) atomicOr(in.map + (u >> 6), 1ull << (u & 63));
                if (v != HOP_NOVEC) d = __ldg(reinterpret_cast<const uint32_t*>(in.nbr) + 4 * (uint64_t)v + l);
            }
            bool fresh = false;
            uint32_t r0 = 0, r1 = 0, deg = 0;
            // the row pointers and degree are loaded while the atomic that decides is on its way
            if (d < in.V) {
                if (IsBfs) {
                    const unsigned long long key = ((unsigned long long)level << 33) | ((unsigned long long)mode << 32) | u;
                    const unsigned long long c = __ldcg(in.cand64 + d);
                    const bool w = (__ldg(in.wants + (d >> 6)) >> (d & 63)) & 1ull;
                    if (w && key < c) {
                        const unsigned long long old = atomicMin(in.cand64 + d, key);
                        r0 = __ldg(in.rowptr + d);
                        r1 = __ldg(in.rowptr + d + 1);
                        deg = __ldg(in.degree + d);
                        fresh = old == ~0ull;
                    }
                } else {
                    const uint32_t msg = __ldcg(in.label + u);
                    if (msg < __ldcg(in.label + d)) {
                        const uint32_t old = atomicMin(in.label + d, msg);
                        r0 = __ldg(in.rowptr + d);
                        r1 = __ldg(in.rowptr + d + 1);
                        deg = __ldg(in.degree + d);
                        if (msg < old) {
                            sum.min = min(sum.min, msg);
                            fresh = atomicMin(in.cand32 + d, ~level) > ~level;
                        }
                    }
                }
            }
            if (fresh) {
                const unsigned long long x = 1ull + deg + sum.vote_lo;
                sum.vote_lo = (uint32_t)(x & 0xffffu);
                sum.vote_hi += (uint32_t)(x >> 16);
                sum.verts += 1;
            }
            if (__any_sync(0xffffffffu, fresh) && !append(p ^ 1, nxt, fresh, d, r0, r1 - r0) && fresh) sum.flags |= HOP_OVER;
        }
        sum = hop_exchange(cl, sum, &s_items[nxt], &s_block[p], s_part[p]);
        // every thread of the cluster takes the same decision from the iteration's totals
        vote = sum.vote_lo + ((unsigned long long)sum.vote_hi << 16);
        if (IsBfs) left -= sum.verts;
        if (vote == 0 || vote > GRZ_HOP_VOTE || sum.flags || level >= max_level) break;
        int pull;
        if (force >= 0) {
            pull = force;
        } else if (params) {
            if (tid < 32) {
                FeatIn fe;
                fe.V = in.dV;
                fe.E = in.dE;
                fe.max_degree = in.max_degree;
                fe.iter = level + 1;
                fe.app_bfs = IsBfs;
                fe.last_engine = (int)mode;
                if (lane < NF) s_f[lane] = feature(lane, fe, (float)(unsigned long long)sum.verts, IsBfs ? (float)left : 0.f, (float)vote);
                __syncwarp();
                const float z = mlp_logit_warp(MlpShared{ s_par }, s_f, lane);
                if (lane == 0) s_pull = z > 0.f ? 1 : 0;
            }
            __syncthreads();
            pull = s_pull;
        } else {
            pull = (double)vote > threshold ? 1 : 0;
        }
        if (pull && !in.pulls) break;
        pulls += mode;
        mode = (uint32_t)pull;
    }
    // the last frontier's marks
    const uint32_t* last = s_mem + ((it & 1) ^ 1) * 2 * HOP_CAP + HOP_CAP;
    for (uint32_t i = tid; i < min(s_items[(it + 1) & 3], HOP_CAP); i += HOP_T) {
        const uint32_t u = last[i];
        if (u & HOP_FIRST) atomicOr(in.map + ((u & ~HOP_FIRST) >> 6), 1ull << (u & 63));
    }
    // iteration `it` is the last: the decision kernel counts it and reads its vote from the slots
    if (tid == 0 && rank == 0) {
        const uint32_t level = level0 + it;
        in.vote[0] = vote;
        if (!IsBfs && sum.min != INF)
            atomicMax(in.chg + (level & 1), ((unsigned long long)level << 32) | (unsigned long long)(~sum.min));
        ctl->level = level;
        ctl->engine = mode;
        ctl->npull += pulls;
        ctl->npush += it - pulls;
        ctl->hop_pulls = pulls + mode;
        ctl->hop_levels[0] += it + 1 - pulls - mode;
        ctl->hop_levels[1] += pulls + mode;
        ctl->hop_runs += 1;
    }
}

// BFS, after k_hop: levels, WantsInfo and the last frontier's HasInfo* of the marked vertices, and the
// parents of those that a push visited, whose candidates it empties.  `clear`: no k_hop_parents follows.
__global__ void __launch_bounds__(T) k_hop_visit(const grz_runctl* __restrict__ ctl, unsigned long long* __restrict__ map, uint64_t W,
                                                 unsigned long long* __restrict__ cand64, uint32_t* __restrict__ parent,
                                                 uint32_t* __restrict__ level, unsigned long long* __restrict__ wants,
                                                 unsigned long long* __restrict__ has_next, int clear)
{
    const uint32_t last = ctl->level;
    unsigned long long in_last = 0ull;
    for_marked(
        [&](uint64_t w) { return map[w]; }, W, [&](uint32_t d) { return cand64[d]; },
        [&](uint32_t d, bool marked, unsigned long long c, int half) {
            bool l = false;
            if (marked) {
                const uint32_t lv = (uint32_t)(c >> 33);
                level[d] = lv;
                l = lv == last;
                if (!((c >> 32) & 1ull)) {
                    parent[d] = (uint32_t)c;
                    cand64[d] = ~0ull;
                }
            }
            const unsigned long long m = __ballot_sync(0xffffffffu, l);
            in_last = half ? in_last | (m << 32) : m;
        },
        [&](uint64_t w, unsigned long long bits) {
            wants[w] &= ~bits;
            has_next[w] = in_last;
            if (clear) map[w] = 0ull;
        });
}

// BFS: parents of the marked vertices that a pull visited.  The candidate's source is the smallest in
// the frontier; its vector is the last one that starts below it, or, when that one ends before it, the
// next (repeated edges can fill the end of one vector and the start of the next: the first that holds
// the source counts).  The parent is the largest source there that was visited one iteration earlier.
__global__ void __launch_bounds__(T) k_hop_parents(const grz_runctl* __restrict__ ctl, unsigned long long* __restrict__ map, uint64_t W,
                                                   unsigned long long* __restrict__ cand64, uint32_t* __restrict__ parent,
                                                   const uint32_t* __restrict__ level, uint32_t V, const uint4* __restrict__ nbr,
                                                   const uint32_t* __restrict__ rowptr, const uint32_t* __restrict__ hub_vid, uint32_t nhub)
{
    if (!ctl->hop_pulls) {
        for_marked([&](uint64_t w) { return map[w]; }, W, [](uint32_t) { return 0ull; }, [](uint32_t, bool, unsigned long long, int) {},
                   [&](uint64_t w, unsigned long long) { map[w] = 0ull; });
        return;
    }
    for_marked(
        [&](uint64_t w) { return map[w]; }, W, [&](uint32_t d) { return cand64[d]; },
        [&](uint32_t d, bool marked, unsigned long long c, int) {
            if (!marked || c == ~0ull) return;  // a push visited it
            cand64[d] = ~0ull;
            const uint32_t u = (uint32_t)c, before = (uint32_t)(c >> 33) - 1;
            uint32_t lo = __ldg(rowptr + d), hi = __ldg(rowptr + d + 1) - 1;
            const uint32_t last = hi;
            while (lo < hi) {
                const uint32_t mid = lo + (hi - lo + 1) / 2;
                if (grz_hub_decode(__ldg(&nbr[mid].x), hub_vid, nhub) < u) lo = mid; else hi = mid - 1;
            }
            uint32_t id[4];
            auto sources = [&](uint32_t vec) {
                const uint4 s = __ldg(nbr + vec);
                id[0] = grz_hub_decode(s.x, hub_vid, nhub);
                id[1] = grz_hub_decode(s.y, hub_vid, nhub);
                id[2] = grz_hub_decode(s.z, hub_vid, nhub);
                id[3] = grz_hub_decode(s.w, hub_vid, nhub);
            };
            sources(lo);
            if (lo < last && id[3] < u) sources(lo + 1);  // (a vector before the last is full)
            uint32_t best = u;
#pragma unroll
            for (int l = 0; l < 4; ++l)
                if (id[l] < V && id[l] > best && level[id[l]] == before) best = id[l];
            parent[d] = best;
        },
        [&](uint64_t w, unsigned long long) { map[w] = 0ull; });
}

// CC, after k_hop: the last frontier's HasInfo*; empties the stamps
__global__ void __launch_bounds__(T) k_hop_labels(const grz_runctl* __restrict__ ctl, unsigned long long* __restrict__ map, uint64_t W,
                                                  uint32_t* __restrict__ cand32, unsigned long long* __restrict__ has_next)
{
    const uint32_t last = ctl->level;
    unsigned long long in_last = 0ull;
    for_marked(
        [&](uint64_t w) { return map[w]; }, W, [&](uint32_t d) { return (unsigned long long)cand32[d]; },
        [&](uint32_t d, bool marked, unsigned long long c, int half) {
            bool l = false;
            if (marked) {
                l = (uint32_t)c == ~last;
                cand32[d] = INF;
            }
            const unsigned long long m = __ballot_sync(0xffffffffu, l);
            in_last = half ? in_last | (m << 32) : m;
        },
        [&](uint64_t w, unsigned long long) {
            has_next[w] = in_last;
            map[w] = 0ull;
        });
}

// ---------------------------------------------------------------------------------------------
// init / output

// The starting state of a run, in one launch: CC labels (execution_initialize_vertex_prop_cc: the ID) or
// BFS parents and levels (INF, the root's level 0), entry V = +inf; HasInfo and WantsInfo (CC all,
// execution_cc.c:66-73; BFS the root, and all but the root), HasInfo* empty; the words of cc_prev_min
// (before iteration 1 every vertex counts as changed, the smallest label being 0); the vote slots; and
// a graph run's control block (`ctl` not null).  Four vertices per thread with 16-byte stores (the
// arrays are 256-byte aligned), the last few one by one; bitmap bits at and beyond V stay clear.
__global__ void __launch_bounds__(T) k_frontier_init(uint32_t* __restrict__ label, uint32_t* __restrict__ level,
                                                     unsigned long long* __restrict__ has, unsigned long long* __restrict__ wants,
                                                     unsigned long long* __restrict__ has_next, uint64_t V, uint64_t W, int bfs, uint32_t root,
                                                     unsigned long long* __restrict__ chg, unsigned* __restrict__ err,
                                                     unsigned long long* __restrict__ vote, grz_runctl* __restrict__ ctl,
                                                     const __grid_constant__ grz_runctl c)
{
    const uint64_t q = (uint64_t)blockIdx.x * T + threadIdx.x;
    const uint64_t v = 4 * q;
    if (v <= V) {
        uint32_t a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a[j] = bfs || v + j >= V ? INF : (uint32_t)(v + j);
            b[j] = v + j == root ? 0u : INF;
        }
        if (v + 3 <= V) {
            reinterpret_cast<uint4*>(label)[q] = make_uint4(a[0], a[1], a[2], a[3]);
            if (bfs) reinterpret_cast<uint4*>(level)[q] = make_uint4(b[0], b[1], b[2], b[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (v + j <= V) {
                    label[v + j] = a[j];
                    if (bfs) level[v + j] = b[j];
                }
        }
    }
    if (q < W) {
        const unsigned long long all = 64 * q + 64 <= V ? ~0ull : (64 * q < V ? (1ull << (V - 64 * q)) - 1ull : 0ull);
        const unsigned long long r = bfs && q == root >> 6 ? 1ull << (root & 63) : 0ull;
        has[q] = bfs ? r : all;
        wants[q] = all & ~r;
        has_next[q] = 0ull;
    }
    if (q < GRZ_VOTE_SLOTS * GRZ_VOTE_STRIDE) vote[q] = 0ull;
    if (q == 0) {
        chg[0] = 0x00000000ffffffffull;
        chg[1] = 0ull;
        *err = 0u;
        if (ctl) *ctl = c;
    }
}

// bitmap of vertices that own at least one vector in a list: a thread per vertex, a warp per
// 32-bit half of a bitmap word (the words are little-endian), all `words` words written
__global__ void k_nonempty(const uint32_t* __restrict__ rowptr, uint64_t V, unsigned long long* __restrict__ bm, uint64_t words)
{
    const uint64_t v = (uint64_t)blockIdx.x * T + threadIdx.x;
    const bool in = v < 64 * words;  // uniform per warp: 64 words is a multiple of 32
    const bool bit = in && v < V && rowptr[v + 1] > rowptr[v];
    const unsigned m = __ballot_sync(0xffffffffu, bit);
    if (in && (threadIdx.x & 31) == 0) reinterpret_cast<uint32_t*>(bm)[v >> 5] = m;
}

// reference-format output: CC labels as double; BFS parents as double with -1 for unvisited
// vertices and the root (source/execution_bfs.c:113-116)
__global__ void k_u32_to_double(const uint32_t* __restrict__ x, uint64_t V, double* __restrict__ out, int bfs)
{
    const uint64_t v = (uint64_t)blockIdx.x * T + threadIdx.x;
    if (v >= V) return;
    const uint32_t a = x[v];
    out[v] = (bfs && a == INF) ? -1.0 : (double)a;
}

__global__ void k_levels_out(const uint32_t* __restrict__ level, uint64_t V, int64_t* __restrict__ out)
{
    const uint64_t v = (uint64_t)blockIdx.x * T + threadIdx.x;
    if (v < V) out[v] = level[v] == INF ? -1 : (int64_t)level[v];
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// host side

static uint64_t words_of(uint64_t V) { return (V >> 6) + 2; }
static int frontier_list_state(grz_graph* g);

// tile_first with room for `tiles`
static int tiles_alloc(grz_graph* g, uint64_t tiles)
{
    grz_frontier_state& f = g->fr;
    if (tiles <= f.tile_cap) return GRZ_OK;
    GRZ_CK(g, cudaFree(f.tile_first));
    f.tile_first = nullptr;
    f.tile_cap = 0;
    GRZ_CK(g, cudaMalloc((void**)&f.tile_first, sizeof(uint32_t) * tiles));
    f.tile_cap = tiles;
    return GRZ_OK;
}

static int ensure_frontier_state(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    if (f.label && !f.lists_changed) return GRZ_OK;
    const uint64_t V = g->V, W = words_of(V);
    const uint64_t tiles = std::max(g->push.nvec, g->pull.nvec) / PUSH_TILE + 2;
    if (f.label) {
        // kept from the graph loaded before, which had the same V
        if (f.alloc_V != V) return grz_set_error(g, GRZ_ERR_STATE, "frontier buffers sized for another graph");
        GRZ_TRY(tiles_alloc(g, tiles));
        f.lists_changed = 0;
        return frontier_list_state(g);
    }
    f.alloc_V = V;
    // One allocation (and tile_first, which a reload may make larger): twenty were a part of a small graph's
    // first run.  But above half a GB the driver can let it, and the small one after it, wait for what was freed
    // before, 0.9 ms each; then there are three, the randomly read arrays still together (in allocations of their
    // own they read slower: CC on a uniform graph of 16.8M vertices 3.62 and 3.86 ms).  GB300, what a first pass takes
    // beyond the next, twenty / one / three: CC of 4096 vertices 310 / 260 / - us, 2^20 660 / 380 / -, 2^23 920 / 450 / -, 12M
    // 950 / 510 / 570, R-MAT of 2^24 (590 MB) 1070 / 1430 / 790 (one, and the control block after it: 2290).
    const size_t v4 = sizeof(uint32_t) * (V + 1), v8 = sizeof(unsigned long long) * (V + 1), w8 = sizeof(unsigned long long) * W;
    const grz_part part[] = {
        { (void**)&f.label, v4 }, { (void**)&f.level, v4 }, { (void**)&f.has, w8 }, { (void**)&f.has_next, w8 }, { (void**)&f.wants, w8 },
        { (void**)&f.nonempty_push, w8 }, { (void**)&f.nonempty_pull, w8 }, { (void**)&f.unres, w8 }, { (void**)&f.hop_map, w8 },
        { (void**)&f.hop_buf, sizeof(uint32_t) * GRZ_HOP_VOTE }, { (void**)&f.counters, sizeof(uint32_t) * 8 },
        { (void**)&f.digest, sizeof(unsigned long long) * 4 }, { (void**)&f.vote, sizeof(unsigned long long) * GRZ_VOTE_SLOTS * GRZ_VOTE_STRIDE },
        { (void**)&f.chg, sizeof(unsigned long long) * 2 }, { (void**)&f.dev_err, sizeof(unsigned) }, { (void**)&f.ctl, sizeof(grz_runctl) },
        { (void**)&f.frontier, v4 }, { (void**)&f.voff, v4 }, { (void**)&f.vdelta, v4 }, { (void**)&f.touched, v4 },
        { (void**)&f.cand64, v8 }, { (void**)&f.cand32, v4 } };
    constexpr int N = sizeof(part) / sizeof(part[0]), SECOND = N - 6, THIRD = N - 2;
    size_t total = 0;
    for (const grz_part& p : part) total += p.bytes;
    GRZ_TRY(tiles_alloc(g, tiles));
    const bool one = total <= (512u << 20);
    cudaError_t e = grz_alloc_arrays(part, one ? N : SECOND, &f.mem[0]);
    if (!one && e == cudaSuccess) e = grz_alloc_arrays(part + SECOND, THIRD - SECOND, &f.mem[1]);
    if (!one && e == cudaSuccess) e = grz_alloc_arrays(part + THIRD, N - THIRD, &f.mem[2]);
    if (e != cudaSuccess) {
        for (void*& m : f.mem) { cudaFree(m); m = nullptr; }
        f.label = nullptr;  // no state
        return grz_cuda_check(g, e, "frontier arrays");
    }
    GRZ_CK(g, cudaMemsetAsync(f.hop_map, 0, w8, g->stream));
    GRZ_CK(g, cudaMemsetAsync(f.digest, 0, sizeof(unsigned long long) * 4, g->stream));
    return frontier_list_state(g);
}

// the state that depends on the loaded lists, and the scratch values the kernels expect
static int frontier_list_state(grz_graph* g)
{
    const uint64_t V = g->V, W = words_of(V);
    grz_frontier_state& f = g->fr;
    GRZ_CK(g, cudaMemsetAsync(f.vote, 0, sizeof(unsigned long long) * GRZ_VOTE_SLOTS * GRZ_VOTE_STRIDE, g->stream));
    GRZ_CK(g, cudaMemsetAsync(f.cand64, 0xff, sizeof(unsigned long long) * (V + 1), g->stream));
    GRZ_CK(g, cudaMemsetAsync(f.cand32, 0xff, sizeof(uint32_t) * (V + 1), g->stream));
    GRZ_CK(g, cudaMemsetAsync(f.nonempty_push, 0, sizeof(unsigned long long) * W, g->stream));
    GRZ_CK(g, cudaMemsetAsync(f.nonempty_pull, 0, sizeof(unsigned long long) * W, g->stream));
    if (g->pull.rowptr && V) {
        k_nonempty<<<blocks_for(64 * W), T, 0, g->stream>>>(g->pull.rowptr, V, f.nonempty_pull, W); GRZ_COUNT_LAUNCH(g);
        GRZ_CK(g, cudaGetLastError());
    }
    if (g->push.rowptr && V) {
        k_nonempty<<<blocks_for(64 * W), T, 0, g->stream>>>(g->push.rowptr, V, f.nonempty_push, W); GRZ_COUNT_LAUNCH(g);
        GRZ_CK(g, cudaGetLastError());
    }
    return GRZ_OK;
}

static VoteCfg vote_cfg(const grz_graph* g)
{
    VoteCfg vc;
    vc.degree = g->degree;
    vc.without_count = (g->fr.flags & GRZ_FLAG_WITHOUT_COUNT) ? 1 : 0;
    vc.without_outdeg = (g->fr.flags & GRZ_FLAG_WITHOUT_OUTDEG) ? 1 : 0;
    return vc;
}

// Everything of an initialisation but the device state, which frontier_reset writes.  Leaves the
// starting vote in fr.vote_host, for BFS without the root's out-degree.
int grz_frontier_prepare(grz_graph* g, int app, int flags, uint32_t root)
{
    if (!g->outdeg) return grz_set_error(g, GRZ_ERR_STATE, "no graph loaded");
    int rc = ensure_frontier_state(g);
    if (rc) return rc;
    if (app == GRZ_APP_CONNECTED_COMPONENTS && g->tune.cc_segments == 2) {
        rc = grz_pr_ensure_segments(g, 1);
        if (rc) return rc;
    }
    grz_frontier_state& f = g->fr;
    f.app = app;
    f.flags = flags;
    f.root = root;
    f.iter = 0;
    f.npull = f.npush = 0;
    f.last_engine = 1;
    f.next_pull = 1;
    f.cc_partial = 0;
    f.vote_host = 0;
    if (app == GRZ_APP_CONNECTED_COMPONENTS) {
        if (!(flags & GRZ_FLAG_WITHOUT_OUTDEG)) f.vote_host += g->E;     // execution_cc.c:106-112
        if (!(flags & GRZ_FLAG_WITHOUT_COUNT)) f.vote_host += g->V;
    } else {
        if (root >= g->V) return grz_set_error(g, GRZ_ERR_ARG, "root %u >= V", root);
        if (!(flags & GRZ_FLAG_WITHOUT_COUNT)) f.vote_host += 1;         // execution_bfs.c:132-137
    }
    return GRZ_OK;
}

// the device state of the prepared run; `c`: also a graph run's control block
static int frontier_reset(grz_graph* g, const grz_runctl* c)
{
    grz_frontier_state& f = g->fr;
    const uint64_t V = g->V, W = words_of(V);
    const uint64_t n = std::max<uint64_t>(std::max<uint64_t>(V / 4 + 1, W), GRZ_VOTE_SLOTS * GRZ_VOTE_STRIDE);
    grz_runctl none;
    memset(&none, 0, sizeof(none));
    k_frontier_init<<<blocks_for(n), T, 0, g->stream>>>(f.label, f.level, f.has, f.wants, f.has_next, V, W, f.app == GRZ_APP_BREADTH_FIRST_SEARCH,
                                                        f.root, f.chg, f.dev_err, f.vote, c ? f.ctl : nullptr, c ? *c : none); GRZ_COUNT_LAUNCH(g);
    return grz_cuda_check(g, cudaGetLastError(), "k_frontier_init");
}

int grz_frontier_init(grz_graph* g, int app, int flags, uint32_t root)
{
    GRZ_TRY(grz_frontier_prepare(g, app, flags, root));
    GRZ_TRY(frontier_reset(g, nullptr));
    if (app == GRZ_APP_BREADTH_FIRST_SEARCH && !(flags & GRZ_FLAG_WITHOUT_OUTDEG)) {
        uint32_t deg = 0;
        GRZ_CK(g, cudaMemcpyAsync(&deg, g->degree + root, sizeof(deg), cudaMemcpyDeviceToHost, g->stream));
        GRZ_CK(g, cudaStreamSynchronize(g->stream));
        g->fr.vote_host += deg;
    }
    return GRZ_OK;
}

// the reference's threshold engine choice (execution_bfs.c:146-168, execution_cc.c:120-142)
int grz_engine_threshold(const grz_graph* g, uint64_t vote)
{
    const int flags = g->fr.flags;
    if (flags & GRZ_FLAG_FORCE_PULL) return 1;
    if (flags & GRZ_FLAG_FORCE_PUSH) return 0;
    const uint64_t thr = (flags & GRZ_FLAG_WITHOUT_OUTDEG) ? g->V / 2 : g->E / 5;
    return vote > thr ? 1 : 0;
}

// BFS visit grid: full occupancy (8 blocks of 256 per SM), fewer for small graphs
static unsigned visit_grid(const grz_graph* g)
{
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(blocks_for((g->V + 3) / 4), (uint64_t)g->num_sms * 8));
}

// Whether the CC pull's full pass reads the source-segmented lists (built by grz_pr_init, or by
// grz_frontier_init under GRZ_TUNE_CC_SEGMENTS = 2); they need a pull list without hub encoding.
static bool cc_use_segments(const grz_graph* g)
{
    return g->tune.cc_segments != 1 && g->seg_nbr && g->nseg && g->pull.nhub == 0 && !g->tune.cc_pull_first;
}

// kernels one segmented CC pull launches per source segment (the empty segments are skipped)
static uint64_t cc_segment_launches(const grz_graph* g)
{
    uint64_t n = 0;
    for (uint32_t sg = 0; sg < g->nseg; ++sg) n += g->seg_first[sg + 1] > g->seg_first[sg];
    return n;
}

// Shared-memory opt-in and resident blocks per SM of the CC pull kernel, per device, block size
// and staging form.
template <int BT, bool BULK>
static int cc_pull_config(grz_graph* g, size_t smem, int* resident)
{
    static int configured[64] = {};
    const int bit = (BT == 256 ? 1 : (BT == 512 ? 2 : 4)) << (BULK ? 3 : 0);
    if (g->device < 0 || g->device >= 64) return GRZ_ERR_ARG;
    if (!(configured[g->device] & bit)) {
        cudaFuncAttributes fa;
        int optin = 0;
        GRZ_CK(g, cudaFuncGetAttributes(&fa, k_cc_pull<BT, BULK>));
        GRZ_CK(g, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, g->device));
        GRZ_CK(g, cudaFuncSetAttribute(k_cc_pull<BT, BULK>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes));
        configured[g->device] |= bit;
    }
    GRZ_CK(g, cudaOccupancyMaxActiveBlocksPerMultiprocessor(resident, k_cc_pull<BT, BULK>, BT, smem));
    if (*resident < 1) return grz_set_error(g, GRZ_ERR_ARG, "CC pull: %d threads with %zu bytes of shared memory do not fit", BT, smem);
    return GRZ_OK;
}

template <int BT>
static int cc_pull_config_any(grz_graph* g, size_t smem, int* resident)
{
    return g->tune.pull_staging ? cc_pull_config<BT, true>(g, smem, resident) : cc_pull_config<BT, false>(g, smem, resident);
}

// blocks of the kernels that go through compacted vectors by tiles (their number is on the device)
static unsigned tile_grid(const grz_graph* g, const grz_list& l)
{
    return (unsigned)std::min<uint64_t>(l.nvec / PUSH_TILE + 1, (uint64_t)g->num_sms * 8);
}

// Compacts the vertices selected by bm1 & bm2 (defined below)
static void compact(grz_graph* g, const unsigned long long* bm1, const unsigned long long* bm2, const uint32_t* rowptr,
                    uint32_t skip = 0, const uint32_t* gate = nullptr, bool lowest_first = false);

template <int BT, bool BULK>
static int launch_cc_pull_bt(grz_graph* g, uint64_t first, uint64_t count, const VoteCfg& vc)
{
    grz_frontier_state& f = g->fr;
    const uint32_t ncache = std::min<uint32_t>(g->tune.cc_cache, g->pull.nhub);
    const size_t smem = sizeof(uint32_t) * ncache;
    int resident = 0;
    int rc = cc_pull_config<BT, BULK>(g, smem, &resident);
    if (rc) return rc;
    const uint64_t tiles = (count + BT - 1) / BT;
    uint64_t grid = g->tune.cc_grid ? g->tune.cc_grid : (uint64_t)g->num_sms * resident;
    grid = std::max<uint64_t>(1, std::min<uint64_t>(grid, tiles));
    // the skip needs every earlier iteration to have been complete (the whole list, or the whole
    // frontier): true for the driver loops, not once a phases.h call covered part of the list
    const bool whole = !f.cc_partial && first == 0 && count == g->pull.nvec;
    if (whole && g->tune.cc_pull_first) {
        // Each destination's first vector (k_cc_pull_first, which decides on the device whether
        // this is an iteration without a usable previous minimum and otherwise returns at once).
        // Form 1: the whole list without the destinations at 0.  Form 2: the destinations it left
        // open are compacted with their remaining vectors and pulled (gated, empty in a skip
        // iteration), and the skip pass over the whole list runs only in a skip iteration; its
        // first pull is shorter, but it propagates less in place and the runs take one iteration
        // more (GB300, R-MAT 24 sym: 0.81 against 0.76 ms per run).
        const bool open_list = g->tune.cc_pull_first == 2;
        uint32_t* gate = f.counters + 6;
        const uint64_t W = words_of(g->V), groups = (W + CFW - 1) / CFW;
        const unsigned fgrid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((groups + T / 32 - 1) / (T / 32),
                                                                                   (uint64_t)g->num_sms * 8));
        const bool open_all = g->tune.cc_pull_first == 4;
        k_cc_pull_first<<<fgrid, T, 0, g->stream>>>(g->pull.rowptr, g->pull.nbr, (uint32_t)g->V, W, f.label, g->pull.hub_vid,
                                                     g->pull.nhub, f.has_next, vc, f.vote, f.chg, f.iter, f.level_dev,
                                                     (open_list || open_all) ? f.unres : nullptr, gate, open_all ? 1 : 0); GRZ_COUNT_LAUNCH(g);
        unsigned long long* work = nullptr;
        if (g->prof && g->prof->on) {
            if (!g->prof_work) {
                GRZ_CK(g, cudaMalloc((void**)&g->prof_work, sizeof(unsigned long long) * 2));
                GRZ_CK(g, cudaMemsetAsync(g->prof_work, 0, sizeof(unsigned long long) * 2, g->stream));
            }
            work = g->prof_work;
        }
        auto expand = [&]() {
            k_cc_pull_expand<<<tile_grid(g, g->pull), T, 0, g->stream>>>(f.frontier, f.voff, f.vdelta, f.tile_first, f.counters,
                                                                           g->pull.nbr, (uint32_t)g->V, f.label, g->pull.hub_vid,
                                                                           g->pull.nhub, f.has_next, vc, f.vote, f.chg, f.iter,
                                                                           f.level_dev, f.counters + 5, work); GRZ_COUNT_LAUNCH(g);
        };
        if (open_all) {
            // form 4: every pull over the open destinations only, marked by the first-vector pass
            // (first iteration: every vector of those still above 0) or by k_cc_mark_open (later
            // iterations); one of the two writes the whole bitmap in each iteration
            const unsigned mgrid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((W + T / 32 - 1) / (T / 32),
                                                                                       (uint64_t)g->num_sms * 8));
            k_cc_mark_open<<<mgrid, T, 0, g->stream>>>(f.label, f.nonempty_pull, g->V, W, f.chg, f.iter, f.level_dev, f.unres,
                                                        nullptr); GRZ_COUNT_LAUNCH(g);
            compact(g, f.unres, f.nonempty_pull, g->pull.rowptr, 0, nullptr);
            expand();
            return GRZ_OK;
        }
        if (open_list) {
            compact(g, f.unres, f.unres, g->pull.rowptr, 1, gate);
            expand();
        }
        // form 3: the whole list only in the first iteration; in a skip iteration the destinations
        // above the previous minimum are marked, compacted and pulled instead of the whole list
        const bool open_skip = g->tune.cc_pull_first == 3;
        k_cc_pull<BT, BULK><<<(unsigned)grid, BT, smem, g->stream>>>(g->pull.nbr, g->pull.shared, first, count, (uint32_t)g->V, f.label,
                                                                    g->pull.hub_vid, g->pull.nhub, ncache, f.has_next, vc, f.vote, f.chg,
                                                                    f.iter, f.level_dev, open_list ? 3 : (open_skip ? 5 : 4),
                                                                    f.dev_err); GRZ_COUNT_LAUNCH(g);
        if (open_skip) {
            uint32_t* gate2 = f.counters + 7;
            const unsigned mgrid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((W + T / 32 - 1) / (T / 32),
                                                                                       (uint64_t)g->num_sms * 8));
            k_cc_mark_open<<<mgrid, T, 0, g->stream>>>(f.label, f.nonempty_pull, g->V, W, f.chg, f.iter, f.level_dev, f.unres,
                                                        gate2); GRZ_COUNT_LAUNCH(g);
            compact(g, f.unres, f.nonempty_pull, g->pull.rowptr, 0, gate2);
            expand();
        }
        return GRZ_OK;
    }
    if (whole && cc_use_segments(g)) {
        // The full pass (no skip yet) reads the source-segmented lists, so that each segment's
        // labels stay in L2 while its edges stream; the pass with the skip reads the whole list
        // (it reads destinations, not sources).  Which of them does the work is decided on the
        // device, so one captured run graph holds both.
        for (uint32_t sg = 0; sg < g->nseg; ++sg) {
            const uint64_t a = g->seg_first[sg], n = g->seg_first[sg + 1] - a;
            if (n == 0) continue;
            const uint64_t sgrid = std::max<uint64_t>(1, std::min<uint64_t>(grid, (n + BT - 1) / BT));
            k_cc_pull<BT, false><<<(unsigned)sgrid, BT, 0, g->stream>>>(g->seg_nbr, g->seg_dst, a, n, (uint32_t)g->V, f.label,
                                                                       g->pr_hot_vid, g->seg_nhot, 0u, f.has_next, vc, f.vote, f.chg, f.iter, f.level_dev, 2,
                                                                       f.dev_err); GRZ_COUNT_LAUNCH(g);
        }
        k_cc_pull<BT, BULK><<<(unsigned)grid, BT, smem, g->stream>>>(g->pull.nbr, g->pull.shared, first, count, (uint32_t)g->V, f.label,
                                                                    g->pull.hub_vid, g->pull.nhub, ncache, f.has_next, vc, f.vote, f.chg,
                                                                    f.iter, f.level_dev, 3, f.dev_err); GRZ_COUNT_LAUNCH(g);
        return GRZ_OK;
    }
    k_cc_pull<BT, BULK><<<(unsigned)grid, BT, smem, g->stream>>>(g->pull.nbr, g->pull.shared, first, count, (uint32_t)g->V, f.label,
                                                                g->pull.hub_vid, g->pull.nhub, ncache, f.has_next, vc, f.vote, f.chg,
                                                                f.iter, f.level_dev, whole ? 1 : 0, f.dev_err); GRZ_COUNT_LAUNCH(g);
    return GRZ_OK;
}

static int launch_cc_pull(grz_graph* g, uint64_t first, uint64_t count, const VoteCfg& vc)
{
    const bool b = g->tune.pull_staging != 0;
    switch (g->tune.cc_threads) {
    case 256: return b ? launch_cc_pull_bt<256, true>(g, first, count, vc) : launch_cc_pull_bt<256, false>(g, first, count, vc);
    case 1024: return b ? launch_cc_pull_bt<1024, true>(g, first, count, vc) : launch_cc_pull_bt<1024, false>(g, first, count, vc);
    default: return b ? launch_cc_pull_bt<512, true>(g, first, count, vc) : launch_cc_pull_bt<512, false>(g, first, count, vc);
    }
}

// Compacts the vertices selected by bm1 & bm2, with their vector ranges in `rowptr`, into
// fr.frontier / voff / vdelta / tile_first (counts on the device in counters[3], [2], which are zero).
// lowest_first: in a large graph the first 1/256 of the vertices come before the others.  CC's push wants that:
// labels are vertex IDs, so the lowest have the smallest labels, which spread in place while the rest of
// the list is pushed and spare it its atomics.  GB300, R-MAT, forced pushes, a whole run with the list in vertex
// order by three kernels / any order / this: 2^20 vertices 428 / 437 / 386 us, 2^21 709 / - / 671, 2^23 2408 / 2780 /
// 2418, uniform 3M 1202 / - / 1014.
constexpr uint64_t FR_LOWEST = 256;
static bool compact_twice(const grz_graph* g, bool lowest_first) { return lowest_first && g->V >= FR_SMALL_V; }
static void compact(grz_graph* g, const unsigned long long* bm1, const unsigned long long* bm2, const uint32_t* rowptr,
                    uint32_t skip, const uint32_t* gate, bool lowest_first)
{
    grz_frontier_state& f = g->fr;
    auto launch = [&](auto kernel, unsigned nb, uint64_t word0) {
        kernel<<<nb, T, 0, g->stream>>>(bm1, bm2, g->V, rowptr, skip, gate, f.counters, f.frontier, f.voff, f.vdelta, f.tile_first, word0);
        GRZ_COUNT_LAUNCH(g);
    };
    if (g->V < FR_SMALL_V) {
        launch(k_fr_compact<FR_WORDS_SMALL>, (unsigned)(g->V / (T * FR_WORDS_SMALL) + 1), 0);
        return;
    }
    // blocks of FR_WORDS words per warp; the first part's words are spread over more blocks
    const unsigned nb = (unsigned)(g->V / (T * FR_WORDS) + 1), lowest = compact_twice(g, lowest_first) ? (unsigned)((nb + FR_LOWEST - 1) / FR_LOWEST) : 0u;
    if (lowest) launch(k_fr_compact<FR_WORDS_SMALL>, lowest * (FR_WORDS / FR_WORDS_SMALL), 0);
    if (nb > lowest) launch(k_fr_compact<FR_WORDS>, nb - lowest, (uint64_t)lowest * (T / 32) * FR_WORDS);
}

// One edge phase on a vector range of the pull (pull=1) or push list.  Leaves the vote of the
// phase in fr.vote[0] on the device.  The push engine always expands the whole compacted frontier.
static int edge_phase(grz_graph* g, int pull, uint64_t first, uint64_t count)
{
    grz_frontier_state& f = g->fr;
    const uint32_t V = (uint32_t)g->V;
    const uint64_t W = words_of(g->V);
    cudaStream_t st = g->stream;
    const VoteCfg vc = vote_cfg(g);
    const bool bfs = f.app == GRZ_APP_BREADTH_FIRST_SEARCH;
    // in a captured run the decision before the phase cleared the counters
    if (!f.level_dev) GRZ_CK(g, cudaMemsetAsync(f.counters, 0, sizeof(uint32_t) * 8, st));
    if (pull) {
        if (!g->pull.nbr) return grz_set_error(g, GRZ_ERR_STATE, "pull list not loaded");
        if (count == 0) return GRZ_OK;
        const bool compacted = bfs && first == 0 && count == g->pull.nvec && !g->tune.bfs_pull_scan;
        const uint32_t first_n = g->tune.bfs_pull_first;
        if (compacted && first_n) {
            // the whole list: each wanted destination's first vectors up to the first frontier
            // source, then the remaining vectors of those left undecided
            if (g->stats_on) {  // the work counted is the reference's: every vector of the wanted destinations
                compact(g, f.wants, f.nonempty_pull, g->pull.rowptr);
                GRZ_TRY(grz_stats_count_selected(g, &g->pull, f.frontier, f.counters));
                GRZ_CK(g, cudaMemsetAsync(f.counters, 0, sizeof(uint32_t) * 8, st));  // the compaction below counts anew
            }
            grz_prof_begin(g, GRZ_PROF_BFS_PULL);
            const uint64_t pgroups = (W + FW - 1) / FW;
            const unsigned fgrid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((pgroups + T / 32 - 1) / (T / 32),
                                                                                       (uint64_t)g->num_sms * GRZ_BFS_MINB));
            k_bfs_pull_first<<<fgrid, T, 0, st>>>(f.wants, f.nonempty_pull, g->pull.rowptr, g->pull.nbr, V, W, f.has,
                                                  g->pull.hub_vid, g->pull.nhub, f.has_next, f.unres, first_n, f.label, f.level,
                                                  f.iter, f.level_dev, vc, f.vote); GRZ_COUNT_LAUNCH(g);
            compact(g, f.unres, f.unres, g->pull.rowptr, first_n);
            k_bfs_pull_expand<<<tile_grid(g, g->pull), T, 0, st>>>(f.frontier, f.voff, f.vdelta, f.tile_first, f.counters,
                                                                     g->pull.nbr, V, f.has, f.cand64, f.touched, f.counters + 1,
                                                                     g->pull.hub_vid, g->pull.nhub, f.has_next, f.counters + 5); GRZ_COUNT_LAUNCH(g);
        } else if (compacted) {
            // the whole list: only the vectors of wanted destinations
            grz_prof_begin(g, GRZ_PROF_PUSH_COMPACT);
            compact(g, f.wants, f.nonempty_pull, g->pull.rowptr);
            grz_prof_end(g);
            GRZ_TRY(grz_stats_count_selected(g, &g->pull, f.frontier, f.counters));
            grz_prof_begin(g, GRZ_PROF_BFS_PULL);
            k_bfs_pull_expand<<<tile_grid(g, g->pull), T, 0, st>>>(f.frontier, f.voff, f.vdelta, f.tile_first, f.counters,
                                                                     g->pull.nbr, V, f.has, f.cand64, f.touched, f.counters + 1,
                                                                     g->pull.hub_vid, g->pull.nhub, f.has_next, f.counters + 5); GRZ_COUNT_LAUNCH(g);
        } else {
            GRZ_TRY(grz_stats_count_range(g, &g->pull, first, count));
            grz_prof_begin(g, bfs ? GRZ_PROF_BFS_PULL : GRZ_PROF_CC_PULL);
        }
        if (bfs && !compacted) {
            const unsigned pgrid = (unsigned)std::min<uint64_t>(blocks_for(count), (uint64_t)g->num_sms * 8);
            k_bfs_pull<<<pgrid, T, 0, st>>>(g->pull.nbr, g->pull.shared, first, count, V, f.has, f.wants, f.cand64,
                                                       f.touched, f.counters + 1, g->pull.hub_vid, g->pull.nhub, f.has_next); GRZ_COUNT_LAUNCH(g);
        }
        if (bfs) {
            grz_prof_end(g);
            grz_prof_begin(g, GRZ_PROF_BFS_VISIT);
            k_bfs_visit<true><<<visit_grid(g), T, 0, st>>>(f.touched, f.counters + 1, f.cand64, f.cand32, f.label, f.level,
                                                            f.iter, f.level_dev, f.wants, f.has_next, vc, f.vote, V); GRZ_COUNT_LAUNCH(g);
        } else {
            int rc = launch_cc_pull(g, first, count, vc);
            if (rc) return rc;
        }
        grz_prof_end(g);
    } else {
        if (!g->push.nbr) return grz_set_error(g, GRZ_ERR_STATE, "push list not loaded");
        grz_prof_begin(g, GRZ_PROF_PUSH_COMPACT);
        compact(g, f.has, f.nonempty_push, g->push.rowptr, 0, nullptr, !bfs);
        grz_prof_end(g);
        GRZ_TRY(grz_stats_count_selected(g, &g->push, f.frontier, f.counters));
        grz_prof_begin(g, bfs ? GRZ_PROF_BFS_PUSH : GRZ_PROF_CC_PUSH);
        const unsigned grid = tile_grid(g, g->push);
        if (bfs) {
            k_push_expand<true><<<grid, T, 0, st>>>(f.frontier, f.voff, f.vdelta, f.tile_first, f.counters, g->push.nbr, V, f.label,
                                                    f.has_next, f.wants, f.cand32, f.touched, f.counters + 1, vc, f.vote,
                                                    nullptr, 0, nullptr); GRZ_COUNT_LAUNCH(g);
            grz_prof_end(g);
            grz_prof_begin(g, GRZ_PROF_BFS_VISIT);
            k_bfs_visit<false><<<visit_grid(g), T, 0, st>>>(f.touched, f.counters + 1, f.cand64, f.cand32, f.label, f.level,
                                                             f.iter, f.level_dev, f.wants, f.has_next, vc, f.vote, V); GRZ_COUNT_LAUNCH(g);
        } else {
            k_push_expand<false><<<grid, T, 0, st>>>(f.frontier, f.voff, f.vdelta, f.tile_first, f.counters, g->push.nbr, V, f.label,
                                                     f.has_next, f.wants, f.cand32, f.touched, f.counters + 1, vc, f.vote,
                                                     f.chg, f.iter, f.level_dev); GRZ_COUNT_LAUNCH(g);
        }
        grz_prof_end(g);
    }
    return grz_cuda_check(g, cudaGetLastError(), "edge phase");
}

// perform_vertex_phase_{cc,bfs}: HasInfo <- HasInfo*, HasInfo* <- 0 (pointer swap + clear)
int grz_frontier_vertex_phase(grz_graph* g, uint64_t first, uint64_t count)
{
    (void)first;
    (void)count;
    grz_frontier_state& f = g->fr;
    if (!grz_frontier_live(g)) return grz_set_error(g, GRZ_ERR_STATE, "frontier state not initialised for the loaded graph");
    unsigned long long* t = f.has;
    f.has = f.has_next;
    f.has_next = t;
    GRZ_CK(g, cudaMemsetAsync(f.has_next, 0, sizeof(unsigned long long) * words_of(g->V), g->stream));
    return GRZ_OK;
}

// the phases.h entry points: one edge phase with a fresh vote, counted into the iteration total
int grz_cc_phase(grz_graph* g, int pull, uint64_t first_vec, uint64_t count)
{
    if (!grz_frontier_live(g) || g->fr.app != GRZ_APP_CONNECTED_COMPONENTS) {
        int rc = grz_frontier_init(g, GRZ_APP_CONNECTED_COMPONENTS, 0, 0);
        if (rc) return rc;
    }
    // An edge phase per call, numbered like the driver loops' iterations.  A pull over part of
    // the list leaves the converged-destination skip off for the rest of this state (the tag
    // 2^32 - 1 never matches; grz_frontier_init starts over).
    grz_frontier_state& f = g->fr;
    const bool whole = !pull || (first_vec == 0 && count == g->pull.nvec);
    if (!whole) f.cc_partial = 1;
    f.iter++;
    const int rc = edge_phase(g, pull, first_vec, count);
    if (rc) return rc;
    if (f.cc_partial) GRZ_CK(g, cudaMemsetAsync(f.chg, 0xff, 2 * sizeof(unsigned long long), g->stream));
    return GRZ_OK;
}

int grz_bfs_phase(grz_graph* g, int pull, uint64_t first_vec, uint64_t count)
{
    if (!grz_frontier_live(g) || g->fr.app != GRZ_APP_BREADTH_FIRST_SEARCH) {
        int rc = grz_frontier_init(g, GRZ_APP_BREADTH_FIRST_SEARCH, 0, 0);
        if (rc) return rc;
    }
    grz_frontier_state& f = g->fr;
    f.iter++;  // a BFS level per edge phase; the root is level 0
    return edge_phase(g, pull, first_vec, count);
}

// Runs one iteration: engine choice from the current vote (or the caller's choice), the edge
// phase, the vote read-back and, unless converged, the vertex phase.  Returns 1 while not
// converged, 0 when the vote is 0, negative on error.  *engine_out = 1 pull / 0 push.
int grz_frontier_step(grz_graph* g, int engine, int* engine_out, uint64_t* vote_out)
{
    grz_frontier_state& f = g->fr;
    const bool learned = f.policy == GRZ_POLICY_LEARNED && f.mlp;
    int rc;
    if (engine < 0 && learned && f.iter == 0) {
        // first iteration: decide from the initial frontier and the initial vote
        uint64_t v0 = 0;
        rc = grz_switch_decide(g, f.has, f.vote_host, 1, &v0, &f.next_pull, f.last_features);
        if (rc) return rc;
    }
    const bool forced = (f.flags & (GRZ_FLAG_FORCE_PULL | GRZ_FLAG_FORCE_PUSH)) != 0;
    const int pull = engine >= 0 ? engine : ((learned && !forced) ? f.next_pull : grz_engine_threshold(g, f.vote_host));
    if (engine_out) *engine_out = pull;
    GRZ_CK(g, cudaMemsetAsync(f.vote, 0, sizeof(unsigned long long) * GRZ_VOTE_SLOTS * GRZ_VOTE_STRIDE, g->stream));
    f.iter++;
    if (f.time_edges) GRZ_CK(g, cudaEventRecord(f.ev[0], g->stream));
    rc = edge_phase(g, pull, 0, pull ? g->pull.nvec : g->push.nvec);
    if (rc) return rc;
    if (f.time_edges) GRZ_CK(g, cudaEventRecord(f.ev[1], g->stream));
    if (pull) f.npull++; else f.npush++;
    f.last_engine = pull;
    uint64_t v = 0;
    if (learned) {
        // the vote and the next engine in one read-back; the next frontier is HasInfo*
        rc = grz_switch_decide(g, f.has_next, ~0ull, f.iter + 1, &v, &f.next_pull, f.last_features);
    } else {
        rc = grz_read_vote(g, &v);
    }
    if (rc) return rc;
    if (f.time_edges) {
        GRZ_CK(g, cudaEventSynchronize(f.ev[1]));
        GRZ_CK(g, cudaEventElapsedTime(&f.last_edge_ms, f.ev[0], f.ev[1]));
    }
    f.vote_host = v;
    if (vote_out) *vote_out = v;
    if (v == 0) return 0;
    rc = grz_frontier_vertex_phase(g, 0, g->V);
    return rc ? rc : 1;
}

// GRZ_ERR_TIMEOUT if a bounded device-side wait of an edge phase gave up since grz_frontier_init
// (synchronises the stream)
int grz_frontier_check_waits(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    if (!f.dev_err) return GRZ_OK;
    unsigned e = 0;
    GRZ_CK(g, cudaMemcpyAsync(&e, f.dev_err, sizeof(e), cudaMemcpyDeviceToHost, g->stream));
    GRZ_CK(g, cudaStreamSynchronize(g->stream));
    if (e) return grz_set_error(g, GRZ_ERR_TIMEOUT, "an edge phase's wait for its staged vectors ran out");
    return GRZ_OK;
}

// the pinned host buffer the per-iteration read-backs go through
int grz_frontier_mail(grz_graph* g)
{
    if (!g->fr.mail) GRZ_CK(g, cudaMallocHost(&g->fr.mail, sizeof(unsigned long long) * GRZ_VOTE_SLOTS * GRZ_VOTE_STRIDE));
    return GRZ_OK;
}

// sum of the vote slots (synchronises the stream)
int grz_read_vote(grz_graph* g, uint64_t* out)
{
    const int rc = grz_frontier_mail(g);
    if (rc) return rc;
    const size_t bytes = sizeof(unsigned long long) * GRZ_VOTE_SLOTS * GRZ_VOTE_STRIDE;
    GRZ_CK(g, cudaMemcpyAsync(g->fr.mail, g->fr.vote, bytes, cudaMemcpyDeviceToHost, g->stream));
    GRZ_CK(g, cudaStreamSynchronize(g->stream));
    const unsigned long long* slots = (const unsigned long long*)g->fr.mail;
    uint64_t v = 0;
    for (int i = 0; i < GRZ_VOTE_SLOTS; ++i) v += slots[i * GRZ_VOTE_STRIDE];
    *out = v;
    return GRZ_OK;
}

// digest of a CC/BFS result: out[0] = reached vertices (BFS: level set; CC: label == own id,
// i.e. components), out[1] = sum of out-degrees of the reached vertices (BFS), out[2] = an
// order-independent checksum of the labels and levels: sum over v of (value(v) + 1) * odd(v)
// mod 2^64, where value is the BFS level or the CC label (unreached = 2^32 - 1)
// A read of the levels and degrees (or labels): four vertices per thread and step, one atomic per block and
// sum; the last block writes the sums to `out` (page-locked host memory) and leaves `acc` zero for the next
// call.  GB300, the whole call after a BFS of 2^24 vertices and of 100k: 79 and 28 us with one vertex per step,
// an atomic per warp and the sums allocated, cleared and copied on each call; 37 and 16 us so.
__global__ void __launch_bounds__(T) k_digest(const uint32_t* __restrict__ label, const uint32_t* __restrict__ level,
                                              const uint32_t* __restrict__ degree, uint64_t V, int bfs,
                                              unsigned long long* __restrict__ acc, unsigned long long* __restrict__ out)
{
    __shared__ unsigned long long red[T / 32];
    unsigned long long sum[3] = { 0, 0, 0 };  // reached, their out-degrees, hash
    const uint32_t* const value = bfs ? level : label;
    auto add = [&](uint64_t v, uint32_t x, uint32_t deg) {
        const bool reached = bfs ? x != INF : x == (uint32_t)v;
        sum[0] += reached;
        if (bfs && reached) sum[1] += deg;
        sum[2] += ((unsigned long long)x + 1ull) * ((v * 0x9E3779B97F4A7C15ull) | 1ull);
    };
    const uint64_t stride = (uint64_t)gridDim.x * T, tid = (uint64_t)blockIdx.x * T + threadIdx.x;
    for (uint64_t q = tid; q < V / 4; q += stride) {
        const uint4 x = __ldcs(reinterpret_cast<const uint4*>(value) + q);
        const uint4 d = bfs ? __ldg(reinterpret_cast<const uint4*>(degree) + q) : make_uint4(0, 0, 0, 0);
        add(4 * q, x.x, d.x);
        add(4 * q + 1, x.y, d.y);
        add(4 * q + 2, x.z, d.z);
        add(4 * q + 3, x.w, d.w);
    }
    if (tid < V % 4) {
        const uint64_t v = V - 1 - tid;
        add(v, value[v], bfs ? degree[v] : 0u);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        sum[k] = block_sum_u64(sum[k], red);
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    for (int k = 0; k < 3; ++k) atomicAdd(acc + k, sum[k]);
    __threadfence();
    if (atomicAdd(acc + 3, 1ull) != gridDim.x - 1) return;
    __threadfence();
    for (int k = 0; k < 3; ++k) out[k] = atomicExch(acc + k, 0ull);
    acc[3] = 0;
}

int grz_frontier_digest(grz_graph* g, uint64_t* out3)
{
    grz_frontier_state& f = g->fr;
    if (!grz_frontier_live(g)) return grz_set_error(g, GRZ_ERR_STATE, "no CC/BFS result for the loaded graph");
    int rc = grz_frontier_mail(g);
    if (rc) return rc;
    uint64_t* const out = (uint64_t*)f.mail;
    if (g->V) {
        const unsigned grid = (unsigned)std::min<uint64_t>(blocks_for((g->V + 3) / 4), (uint64_t)g->num_sms * 8);
        k_digest<<<grid, T, 0, g->stream>>>(f.label, f.level, g->degree, g->V, f.app == GRZ_APP_BREADTH_FIRST_SEARCH, f.digest,
                                            (unsigned long long*)f.mail); GRZ_COUNT_LAUNCH(g);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
        if (e != cudaSuccess) return grz_cuda_check(g, e, "digest");
    } else {
        out[0] = out[1] = out[2] = 0;
    }
    memcpy(out3, out, 3 * sizeof(uint64_t));
    return GRZ_OK;
}

// the props (CC labels, BFS parents) as doubles, into device or mapped host memory
int grz_frontier_props(grz_graph* g, double* out)
{
    grz_frontier_state& f = g->fr;
    if (!grz_frontier_live(g)) return grz_set_error(g, GRZ_ERR_STATE, "no CC/BFS result for the loaded graph");
    k_u32_to_double<<<blocks_for(g->V), T, 0, g->stream>>>(f.label, g->V, out, f.app == GRZ_APP_BREADTH_FIRST_SEARCH); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    return GRZ_OK;
}

// the BFS levels (-1 unreached) as int64, into device or mapped host memory
int grz_frontier_levels(grz_graph* g, int64_t* out)
{
    if (!g->V) return GRZ_OK;
    k_levels_out<<<blocks_for(g->V), T, 0, g->stream>>>(g->fr.level, g->V, out); GRZ_COUNT_LAUNCH(g);
    return grz_cuda_check(g, cudaGetLastError(), "k_levels_out");
}

void grz_frontier_park(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    // the captured run names the old lists
    if (f.run_exec) cudaGraphExecDestroy(f.run_exec);
    f.run_exec = nullptr;
    f.run_bm[0] = f.run_bm[1] = nullptr;
    f.lists_changed = 1;
}

void grz_frontier_free(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    for (void* p : { f.mem[0], f.mem[1], f.mem[2], (void*)f.tile_first, f.sw_out, f.snap }) cudaFree(p);
    if (f.ev[0]) { cudaEventDestroy(f.ev[0]); cudaEventDestroy(f.ev[1]); }
    if (f.mail) cudaFreeHost(f.mail);
    if (f.run_exec) cudaGraphExecDestroy(f.run_exec);
    grz_mlp* keep_mlp = f.mlp;
    const int keep_policy = f.policy;
    memset(&f, 0, sizeof(f));
    f.mlp = keep_mlp;
    f.policy = keep_policy;
}

// ---------------------------------------------------------------------------------------------
// A whole CC/BFS run as one CUDA graph.
//
//   k_run_decide (initial: sets engine0)  ->  WHILE (loop) {
//       SWITCH (engine0) { pull edge phase | push edge phase | k_hop, even roles;
//                          each then k_run_decide (next HasInfo = B, clears A; sets engine1, loop) }
//       SWITCH (engine1) { the same, odd roles (next HasInfo = A, clears B; sets engine0, loop) }
//   }
//
// The decision ends each branch instead of following the SWITCH: a kernel after a conditional node starts
// about 5 us after it, one after a kernel about 1.  GB300, CC of 4096 vertices 133 -> 128 us, BFS of 100k
// vertices 256 -> 248 us.
//
// Even iterations read HasInfo from buffer A and write HasInfo* into B; odd ones the reverse,
// which is the reference's pointer swap (source/execution_cc.c:245-250) without a host step.
// The decision kernel sets the conditional handles, so the engine choice, the convergence test
// and the iteration count never leave the device: one launch, and the last decision writes the
// control block to page-locked memory (a copy behind the graph took the run of 4096 vertices 8 us longer).  The iterations, engines and results are those of the host loop (grz_frontier_step).

static int capture_begin(grz_graph* g, cudaStream_t cs, cudaGraph_t graph, const cudaGraphNode_t* deps, size_t ndeps)
{
    GRZ_CK(g, cudaStreamBeginCaptureToGraph(cs, graph, deps, nullptr, ndeps, cudaStreamCaptureModeThreadLocal));
    return GRZ_OK;
}

// ends a capture into an existing graph; *sink = the captured work's last node
static int capture_end(grz_graph* g, cudaStream_t cs, cudaGraphNode_t* sink)
{
    cudaStreamCaptureStatus st;
    const cudaGraphNode_t* deps = nullptr;
    size_t n = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(cs, &st, nullptr, nullptr, &deps, nullptr, &n);
    cudaGraphNode_t last = (e == cudaSuccess && n == 1) ? deps[0] : nullptr;
    cudaGraph_t out = nullptr;
    const cudaError_t e2 = cudaStreamEndCapture(cs, &out);
    if (e != cudaSuccess) return grz_cuda_check(g, e, "capture info");
    if (e2 != cudaSuccess) return grz_cuda_check(g, e2, "end capture");
    if (sink) {
        if (!last) return grz_set_error(g, GRZ_ERR_STATE, "captured work does not end in one node");
        *sink = last;
    }
    return GRZ_OK;
}

// a conditional node with `size` bodies (a SWITCH runs the one its handle names, or none)
static int add_conditional(grz_graph* g, cudaGraph_t graph, const cudaGraphNode_t* deps, size_t ndeps, cudaGraphConditionalHandle h,
                           cudaGraphConditionalNodeType type, unsigned size, cudaGraphNode_t* node, cudaGraph_t* bodies)
{
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = type;
    p.conditional.size = size;
    GRZ_CK(g, cudaGraphAddNode(node, graph, deps, nullptr, ndeps, &p));
    for (unsigned i = 0; i < size; ++i) bodies[i] = p.conditional.phGraph_out[i];
    return GRZ_OK;
}

// whether small pulls go through k_hop as well
static bool hop_pulls(const grz_graph* g)
{
    return g->fr.hop_list && g->fr.app == GRZ_APP_BREADTH_FIRST_SEARCH && g->pull.ascending;
}

// k_hop and what writes its results, captured as a body of its own
static int hop_phase(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    const bool bfs = f.app == GRZ_APP_BREADTH_FIRST_SEARCH;
    HopIn in;
    memset(&in, 0, sizeof(in));
    in.nbr = g->push.nbr;
    in.rowptr = g->push.rowptr;
    in.degree = g->degree;
    in.V = (uint32_t)g->V;
    in.dV = (double)g->V;
    in.dE = (double)(g->E ? g->E : 1);
    in.max_degree = (double)g->max_degree;
    in.wants = f.wants;
    in.cand64 = f.cand64;
    in.cand32 = f.cand32;
    in.label = f.label;
    in.map = f.hop_map;
    in.list = f.hop_list;
    in.vote = f.vote;
    in.chg = f.chg;
    in.ctl = f.ctl;
    in.pulls = hop_pulls(g);
    const uint64_t W = words_of(g->V);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(W / (mark_span(W) * (T / 32)) + 1, (uint64_t)g->num_sms * 8));
    if (bfs) {
        k_hop<true><<<HOP_CTAS, HOP_T, HOP_SMEM, g->stream>>>(in);
        k_hop_visit<<<grid, T, 0, g->stream>>>(f.ctl, f.hop_map, W, f.cand64, f.label, f.level, f.wants, f.has_next, !in.pulls);
        if (in.pulls)
            k_hop_parents<<<grid, T, 0, g->stream>>>(f.ctl, f.hop_map, W, f.cand64, f.label, f.level, (uint32_t)g->V, g->pull.nbr, g->pull.rowptr,
                                                     g->pull.hub_vid, g->pull.nhub);
    } else {
        k_hop<false><<<HOP_CTAS, HOP_T, HOP_SMEM, g->stream>>>(in);
        k_hop_labels<<<grid, T, 0, g->stream>>>(f.ctl, f.hop_map, W, f.cand32, f.has_next);
    }
    return grz_cuda_check(g, cudaGetLastError(), "k_hop");
}

static bool hop_fits(const grz_graph* g)
{
    static int known[64] = {};  // per device: 1 fits, 2 does not
    if (g->device < 0 || g->device >= 64 || (g->tune.withhold & GRZ_WITHHOLD_CLUSTERS)) return false;
    if (!known[g->device])
        known[g->device] = grz_clusters_fit((const void*)k_hop<true>, HOP_CTAS, HOP_T, HOP_SMEM) &&
                           grz_clusters_fit((const void*)k_hop<false>, HOP_CTAS, HOP_T, HOP_SMEM) ? 1 : 2;
    return known[g->device] == 1;
}

// Whether a run's small iterations go through k_hop: its frontiers are bounded by the vote, so the
// vote has to count vertices and out-edges (the default; forced engines included).  Where its cluster does
// not fit (a cluster of 16 blocks needs the opt-in, and a GPC that can hold it), the engines' kernels run every
// iteration.
static void hop_prepare(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    f.hop_list = nullptr;
    if ((f.flags & (GRZ_FLAG_WITHOUT_COUNT | GRZ_FLAG_WITHOUT_OUTDEG)) || g->V >= 0x80000000ull) return;  // (31-bit iteration numbers)
    if (hop_fits(g)) f.hop_list = f.hop_buf;
}

static int build_run_graph(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    if (f.run_exec) {
        cudaGraphExecDestroy(f.run_exec);
        f.run_exec = nullptr;
    }
    unsigned long long* A = f.has;
    unsigned long long* B = f.has_next;
    cudaStream_t user = g->stream;
    cudaStream_t cs = nullptr;
    GRZ_CK(g, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t top = nullptr;
    int rc = grz_cuda_check(g, cudaGraphCreate(&top, 0), "graph create");
    // one handle per conditional node: the loop, and the engine of the even and odd halves
    cudaGraphConditionalHandle hloop = 0, hengine[2] = { 0, 0 };
    if (!rc) rc = grz_cuda_check(g, cudaGraphConditionalHandleCreate(&hloop, top, 1, cudaGraphCondAssignDefault), "handle");
    for (int p = 0; p < 2 && !rc; ++p)
        rc = grz_cuda_check(g, cudaGraphConditionalHandleCreate(&hengine[p], top, GRZ_RUN_NONE, cudaGraphCondAssignDefault), "handle");
    g->stream = cs;
    f.level_dev = &f.ctl->level;
    cudaGraphNode_t n0 = nullptr, wnode = nullptr;
    cudaGraph_t body = nullptr;
    if (!rc) rc = capture_begin(g, cs, top, nullptr, 0);
    if (!rc) {
        rc = grz_switch_launch_run_decide(g, A, nullptr, 1, hloop, hengine[0], hop_pulls(g));
        const int rc2 = capture_end(g, cs, &n0);
        if (!rc) rc = rc2;
    }
    if (!rc) rc = add_conditional(g, top, &n0, 1, hloop, cudaGraphCondTypeWhile, 1, &wnode, &body);
    cudaGraphNode_t prev = nullptr;
    for (int parity = 0; parity < 2 && !rc; ++parity) {
        f.has = parity ? B : A;
        f.has_next = parity ? A : B;
        cudaGraphNode_t nengine = nullptr;
        cudaGraph_t engine[3] = { nullptr, nullptr, nullptr };  // GRZ_RUN_PULL, _PUSH, _HOP
        rc = add_conditional(g, body, prev ? &prev : nullptr, prev ? 1 : 0, hengine[parity], cudaGraphCondTypeSwitch, f.hop_list ? 3 : 2,
                             &nengine, engine);
        for (int e = 0; e < (f.hop_list ? 3 : 2) && !rc; ++e) {
            rc = capture_begin(g, cs, engine[e], nullptr, 0);
            if (rc) break;
            rc = e == GRZ_RUN_PULL ? edge_phase(g, 1, 0, g->pull.nvec) : (e == GRZ_RUN_PUSH ? edge_phase(g, 0, 0, g->push.nvec) : hop_phase(g));
            // decides the other half's engine
            if (!rc) rc = grz_switch_launch_run_decide(g, f.has_next, f.has, 0, hloop, hengine[1 - parity], hop_pulls(g));
            const int rc2 = capture_end(g, cs, nullptr);
            if (!rc) rc = rc2;
        }
        prev = nengine;
    }
    f.has = A;
    f.has_next = B;
    f.level_dev = nullptr;
    g->stream = user;
    if (!rc) rc = grz_cuda_check(g, cudaGraphInstantiate(&f.run_exec, top, 0), "graph instantiate");
    if (top) cudaGraphDestroy(top);
    cudaStreamDestroy(cs);
    if (rc) {
        f.run_exec = nullptr;
        return rc;
    }
    f.run_bm[0] = A;
    f.run_bm[1] = B;
    f.run_key[0] = f.app;
    f.run_key[1] = f.flags;
    f.run_tune = g->tune;
    f.run_seg = cc_use_segments(g) ? g->seg_nbr : nullptr;
    f.run_seg_gen = g->seg_gen;
    return GRZ_OK;
}

// Before a graph run: puts the HasInfo buffers back in the roles the cached graph has.
void grz_frontier_run_prepare(grz_graph* g)
{
    grz_frontier_state& f = g->fr;
    if (f.run_exec && f.has == f.run_bm[1] && f.has_next == f.run_bm[0]) {
        f.has = f.run_bm[0];
        f.has_next = f.run_bm[1];
    }
}

// Runs the prepared CC/BFS state (grz_frontier_prepare) to convergence: one kernel for the starting state
// and the control block, and one graph launch.  `started` is recorded between the two.  *launches:
// kernels the graph ran.
int grz_frontier_run_graph(grz_graph* g, cudaEvent_t started, uint64_t* launches)
{
    grz_frontier_state& f = g->fr;
    if (!grz_frontier_live(g)) return grz_set_error(g, GRZ_ERR_STATE, "frontier state not initialised for the loaded graph");
    if (!g->pull.nbr || !g->push.nbr || !g->pull.nvec || !g->push.nvec)
        return grz_set_error(g, GRZ_ERR_STATE, "the graph run needs both edge lists");
    int rc = grz_frontier_mail(g);
    if (rc) return rc;
    rc = grz_switch_max_degree(g);
    if (rc) return rc;
    const bool same = f.run_exec && f.run_bm[0] == f.has && f.run_bm[1] == f.has_next && f.run_key[0] == f.app &&
                      f.run_key[1] == f.flags && !memcmp(&f.run_tune, &g->tune, sizeof(g->tune)) &&
                      f.run_seg == (cc_use_segments(g) ? g->seg_nbr : nullptr) && f.run_seg_gen == g->seg_gen;
    if (!same) {
        int resident = 0;
        const size_t smem = sizeof(uint32_t) * std::min<uint32_t>(g->tune.cc_cache, g->pull.nhub);
        rc = g->tune.cc_threads == 256 ? cc_pull_config_any<256>(g, smem, &resident)
             : (g->tune.cc_threads == 1024 ? cc_pull_config_any<1024>(g, smem, &resident) : cc_pull_config_any<512>(g, smem, &resident));
        if (rc) return rc;
        hop_prepare(g);
        GRZ_TRY(build_run_graph(g));
    }
    grz_runctl c;
    memset(&c, 0, sizeof(c));
    c.running = 1;
    c.level = f.iter + 1;
    c.last_engine = (uint32_t)f.last_engine;
    c.vote = f.vote_host;
    const bool bfs = f.app == GRZ_APP_BREADTH_FIRST_SEARCH;
    if (bfs && !(f.flags & GRZ_FLAG_WITHOUT_OUTDEG)) c.root_degree = g->degree + f.root;
    const uint64_t max_it = g->tune.run_max_iterations ? g->tune.run_max_iterations : std::min<uint64_t>(g->V + 2, 0xfffffff0ull);
    c.max_level = (uint32_t)std::min<uint64_t>(max_it + f.iter, 0xfffffff0ull);
    c.limit_ns = g->tune.run_limit_us ? (unsigned long long)g->tune.run_limit_us * 1000ull : 300ull * 1000000000ull;
    grz_switch_policy_ctl(g, &c);
    GRZ_TRY(frontier_reset(g, &c));
    GRZ_CK(g, cudaEventRecord(started, g->stream));
    GRZ_CK(g, cudaGraphLaunch(f.run_exec, g->stream));
    GRZ_CK(g, cudaStreamSynchronize(g->stream));
    memcpy(&c, f.mail, sizeof(c));  // written by the last decision
    if (c.overrun) {
        // the loop stopped before convergence: the state is left as the last iteration made it
        // (a later grz_frontier_begin, grz_cc_run or grz_bfs_run starts over)
        f.iter += c.npull + c.npush;
        f.npull += c.npull;
        f.npush += c.npush;
        if (c.bodies % 2 == 0 && c.bodies > 0) {
            unsigned long long* t = f.has;
            f.has = f.has_next;
            f.has_next = t;
        }
        if (c.overrun == 1) return grz_set_error(g, GRZ_ERR_TIMEOUT, "no convergence within %u iterations", c.max_level);
        return grz_set_error(g, GRZ_ERR_TIMEOUT, "run stopped by its time bound (%llu us)", c.limit_ns / 1000ull);
    }
    const uint32_t n = c.npull + c.npush;
    f.iter += n;
    f.npull += c.npull;
    f.npush += c.npush;
    f.vote_host = c.vote;
    f.last_engine = (int)c.last_engine;
    f.next_pull = (int)c.engine;
    memcpy(f.last_features, c.features, sizeof(f.last_features));
    // iteration k of the loop (1-based within the launch) read HasInfo from A when k is odd
    if (c.bodies % 2 == 0 && c.bodies > 0) {
        unsigned long long* t = f.has;
        f.has = f.has_next;
        f.has_next = t;
    }
    // kernels of one pull iteration: BFS scan + visit, or (first pass,) compaction, expand, visit;
    // CC one pull launch, or one per source segment plus the whole-list one
    const uint64_t per_pull = bfs ? (g->tune.bfs_pull_scan ? 2 : (g->tune.bfs_pull_first ? 4 : 3))
                                  : (f.run_seg ? cc_segment_launches(g) + 1 : (g->tune.cc_pull_first == 2 ? 4 : (g->tune.cc_pull_first == 3 ? 5 : (g->tune.cc_pull_first == 4 ? 4 : (g->tune.cc_pull_first ? 2 : 1)))));
    const uint64_t per_push = bfs ? 3 : 2 + compact_twice(g, true);
    // decisions, iterations by an engine's kernels, and k_hop's launches
    const uint64_t k = 1 + c.bodies + (uint64_t)(c.npull - c.hop_levels[1]) * per_pull + (uint64_t)(c.npush - c.hop_levels[0]) * per_push +
                       (uint64_t)c.hop_runs * (2 + hop_pulls(g));
    g->nlaunch += k;
    if (launches) *launches = k;
    return GRZ_OK;
}
