// grz_batch.cu -- many personalized-PageRank and multi-source BFS instances over many graphs
// of uneven size, each run as one CUDA graph launch.
//
// The reference has no batching and no personalized PageRank.  PPR here is the reference's
// PageRank vertex phase (source/phase_vertex_pr.asm:75-134) with the teleport term and the
// dangling mass sent to the seed instead of spread over all vertices:
//   accum[v]   = sum over v's in-edges (u, v) of prop[u]        (edge-pull, phase_edge_pull_pr.asm)
//   S          = sum over v of accum[v]
//   rank'[v]   = d * accum[v] + [v == seed] * (d * (1 - S) + (1 - d))
//   prop'[v]   = rank'[v] / deg'(v)                              (deg' as the reference: V if 0)
// starting from rank = one-hot(seed).  Ranks sum to 1 in every iteration.
//
// GB300 design:
//   * The graphs become one block-diagonal union graph: each graph's vertex IDs are offset by
//     the vertices of the graphs before it, and the union is loaded as one grz_graph.  Kernels
//     never need to know where one graph ends; only the per-graph sums S do.
//   * Up to GRZ_BATCH_K (8) instances per graph share one pass over the edges.  Props are stored
//     [vertex][instance] packed in 8 bytes (pk_to_fx), so the 8 lanes that serve one vector's
//     instances read one aligned 64-byte row per source: the random gather costs one line for 8
//     instances instead of 8 lines.
//   * PPR iteration: one kernel gathers and applies.  S only enters at the seed and is the sum of
//     deg(u) * prop(u) of the props being gathered, so it is known before the iteration, and a
//     destination whose sum is complete gets its new prop at once: the accumulators of the
//     destinations that one slot sums alone never reach memory.  A warp is 4 slots of 8 lanes (lane =
//     8 * slot + instance), and each slot walks a contiguous range of vectors, two at a time.  The
//     destinations that the ranges cut are added with exact u128 atomics and finished by a second,
//     small kernel, which also serves the seeds without in-edges (every other vertex without
//     in-edges keeps a prop of zero).  The next S is summed in registers per graph, then per block
//     in shared memory.  Sums are exact, so results do not depend on the launch shape.
//   * Multi-source BFS: bit-parallel, 8 roots per graph.  visited / frontier are one byte per
//     vertex (bit i = instance i).  Pull: a vector's new bits are the OR of its sources'
//     frontier bytes, reduced per destination within the warp, minus the visited bits; the
//     vertex pass sets level = iteration for each new bit.  Levels are exact (level-synchronous).
//   * The PPR iteration loop (fixed count) and the BFS loop (WHILE until no new bit, decided on
//     the device) are each captured once as a CUDA graph and replayed.
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

#include "grz_internal.cuh"
#include "../../include/grazelle_gb300.h"

namespace {

constexpr int K = GRZ_BATCH_K;  // instances per graph (8)
constexpr int GT = 256;         // threads per block
constexpr int MIN_V = 32;       // vertices of the smallest graph
constexpr uint32_t NONE = 0xffffffffu;
constexpr int MAX_GRAPHS = 1024;

typedef unsigned long long pk_t;  // a packed prop (pk_to_fx)

// graph of union vertex v (voff: G+1 ascending offsets)
__device__ __forceinline__ uint32_t graph_of(const uint32_t* voff, uint32_t G, uint32_t v)
{
    uint32_t lo = 0, hi = G - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (voff[mid] <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// initial PPR state: prop = one-hot(seed) / deg'; S = deg(seed) * prop(seed) per (graph, instance).
// The props and ranks are zero elsewhere (and in the buffer the first iteration writes).
__global__ void k_ppr_init(const uint32_t* __restrict__ seeds, uint32_t G, const double* __restrict__ inv_deg,
                           const uint32_t* __restrict__ degree, pk_t* __restrict__ prop, u128* __restrict__ S, u128* __restrict__ S_next)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= G * K) return;
    const uint32_t s = seeds[t];
    u128 v = u128_zero();
    if (s != NONE) {
        const pk_t w = pk_from_double(inv_deg[s]);
        prop[(uint64_t)s * K + t % K] = w;
        v = u128_mul32(pk_to_fx(w), degree[s]);
    }
    S[t] = v;
    S_next[t] = u128_zero();
}

// what finishing a destination needs
struct PprApply {
    const double* inv_deg;
    const uint32_t* degree;
    const uint32_t* voff;    // [G + 1]
    uint32_t G;
    const uint32_t* seeds;   // [G][K]
    double damping;
    const u128* S;           // [G][K]: sum of deg * prop of the props being gathered
    u128* S_next;            // the same of the props being written
    pk_t* prop_out;          // [vertex][K]
    double* rank_out;        // last iteration, or null
};

// d * (1 - S) + (1 - d): the seed's teleport and dangling mass
__device__ __forceinline__ double ppr_teleport(const PprApply& ap, uint32_t g, int inst)
{
    const double S = fx_to_double(ap.S[g * K + inst]);
    return __dadd_rn(__dmul_rn(ap.damping, 1.0 - S), 1.0 - ap.damping);
}

// rank' = fma(accum, d, [v == seed] * teleport) and prop' = rank' / deg' of one vertex and instance;
// returns deg * prop'.  Two FP64 operations: the FP64 pipe is the narrowest of the chip (one warp
// instruction in 16 clocks per SM).
__device__ __forceinline__ u128 ppr_finish(const PprApply& ap, uint32_t v, int inst, u128 x, double teleport)
{
    const double rank = __fma_rn(fx_to_double(x), ap.damping, teleport);
    // (rounding can leave 1 - S below zero at damping 1; props are taken without sign)
    const pk_t w = pk_from_double(__dmul_rn(rank, __ldg(ap.inv_deg + v)));
    ap.prop_out[(uint64_t)v * K + inst] = w;
    if (ap.rank_out) ap.rank_out[(uint64_t)v * K + inst] = rank;
    return u128_mul32(pk_to_fx(w), __ldg(ap.degree + v));
}

constexpr int APPLY_SLOTS = 64;  // graphs whose next S a block sums in shared memory (beyond: global atomics)
constexpr uint32_t PQ = 16;      // ring of the complete sums a warp holds: 3 left over and 8 of a step at most
constexpr int PPR_RESIDENT = 4;  // blocks per SM the launch bounds fit

// Ranges of the slots: bnd[4 w + s] is the first vector of slot s of warp w (a multiple of 4), bnd[4 nwarps]
// = nvec.  The warps' ranges are equal in PPR_WV per vector + PPR_WD per vertex up to their destinations, about
// the instructions k_ppr_step has for each; a warp's slots have the same number of vectors.  All ranges run at
// once, so the longest sets the time: 8-graph batch of 1.04M vertices, 8 instances x 20 iterations, ranges of
// equal vectors 4.46 ms.  Weights 1:1 / 4:5 / 2:3 / 4:7 / 1:2, PPR alone: that batch 3.42 / 3.47 / 3.55 / 3.64 / 3.75 ms, 6 graphs
// of 2.2M vectors 2.86 / 2.87 / 2.91 / 2.94 / 2.97, one of 10^6 vertices and 1.2M vectors 1.96 / 2.06 / 1.99 / 2.06 / 2.15, three of
// 5.3M 2.54 / 2.50 / 2.63 / 2.51 / 2.55.
constexpr uint32_t PPR_WV = 4, PPR_WD = 5;

__global__ void k_ppr_bounds(const uint32_t* __restrict__ dstv, uint32_t nvec, uint32_t V, uint32_t nwarps, uint32_t* __restrict__ bnd)
{
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w > nwarps) return;
    const uint64_t total = (uint64_t)PPR_WV * nvec + (uint64_t)PPR_WD * V;
    uint32_t at[2];
    for (int e = 0; e < 2; ++e) {
        const uint64_t goal = total * (w + e) / nwarps;
        uint32_t lo = 0, hi = (nvec + 3) / 4;  // in groups of 4 vectors
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if ((uint64_t)PPR_WV * 4 * mid + (uint64_t)PPR_WD * dstv[4 * mid] < goal) lo = mid + 1;
            else hi = mid;
        }
        at[e] = w + e >= nwarps ? (nvec + 3) / 4 : lo;
    }
    const uint32_t q = (at[1] - at[0] + 3) / 4;
    for (uint32_t s = 0; s < 4 && w < nwarps; ++s) bnd[4 * w + s] = min(4 * min(at[0] + s * q, at[1]), nvec);
    if (w == nwarps) bnd[4 * w] = nvec;
}

// cut[r]: the destination that the start of range r cuts, once per destination; NONE elsewhere
__global__ void k_ppr_cuts(const uint32_t* __restrict__ dstv, const uint32_t* __restrict__ bnd, uint32_t nranges, uint32_t* __restrict__ cut)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nranges) return;
    const uint32_t lo = bnd[r];
    uint32_t v = NONE;
    if (lo > 0 && lo < bnd[r + 1] && dstv[lo - 1] == dstv[lo]) {
        v = dstv[lo];
        uint32_t p = r;  // the range before that is not empty
        while (bnd[p] == lo) --p;
        if (bnd[p] > 0 && dstv[bnd[p] - 1] == v) v = NONE;
    }
    cut[r] = v;
}

// pk_to_fx of a prop of at least 2^-60 (s < 64), or zero
__device__ __forceinline__ u128 pk_to_fx_near(pk_t w)
{
    const uint32_t s = (uint32_t)w & 63u;
    const pk_t x = w & ~127ull;
    u128 r;
    r.hi = x >> s;
    r.lo = shl64_clamp(x, 64u - s);
    return r;
}

// block sums of the next S in shared memory
__device__ __forceinline__ void ppr_add_S(u128* s_part, const PprApply& ap, uint32_t g, int inst, u128 m)
{
    if ((m.lo | m.hi) == 0) return;
    if (g < (uint32_t)APPLY_SLOTS) u128_atomic_add(s_part + g * K + inst, m);
    else u128_atomic_add(ap.S_next + (uint64_t)g * K + inst, m);
}

__device__ __forceinline__ void ppr_flush_S(const u128* s_part, uint32_t nslots, const PprApply& ap)
{
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < nslots; k += GT) {
        const u128 y = s_part[k];
        if (y.lo | y.hi) u128_atomic_add(ap.S_next + k, y);
    }
}

// One PPR iteration but for the cut destinations (see the file comment).  Block 0 clears S_clear for the
// iteration after.  prop row V is zero: empty lanes gather it.
//
// Bound by the ALU pipe (shifts, logic and additions of the 128-bit sums: 53% of its peak over the whole
// launch, memory below 35%).  So the slots walk ranges of their own, which needs no scan across lanes (a scan
// over the slots: 722 instructions per 16 vectors and 206 us, without 535 and 160 us); props of 2^-60 and
// more, nearly all, are unpacked by a shorter form when all of a warp's are; and complete sums wait in shared
// memory to be finished four at a time with all lanes, for FP64 instructions cost the same for one lane.
//
// GB300, 8 graphs of 1.04M vertices and 10.5M edges in all, 8 instances, us per iteration: a gather of
// 16-byte fixed-point rows and an apply over all vertices 224; this and k_ppr_rest 175.  32 graphs of 245M
// edges, 20 iterations: 89.9 ms and 71.8 ms.
__global__ void __launch_bounds__(GT, PPR_RESIDENT) k_ppr_step(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv,
                                                              const uint32_t* __restrict__ bnd, uint32_t nvec, uint32_t V,
                                                              const pk_t* __restrict__ prop, u128* __restrict__ rowacc,
                                                              u128* __restrict__ S_clear, const PprApply ap)
{
    __shared__ uint32_t voff[MAX_GRAPHS + 1];
    __shared__ u128 s_part[APPLY_SLOTS * K];
    __shared__ u128 s_sum[GT / 32][PQ * K];
    __shared__ uint32_t s_vid[GT / 32][PQ];
    u128* const qsum = s_sum[threadIdx.x >> 5];
    uint32_t* const qvid = s_vid[threadIdx.x >> 5];
    const uint32_t nslots = (ap.G < (uint32_t)APPLY_SLOTS ? ap.G : (uint32_t)APPLY_SLOTS) * K;
    for (uint32_t k = threadIdx.x; k <= ap.G; k += GT) voff[k] = ap.voff[k];
    for (uint32_t k = threadIdx.x; k < nslots; k += GT) s_part[k] = u128_zero();
    if (blockIdx.x == 0)
        for (uint32_t k = threadIdx.x; k < ap.G * K; k += GT) S_clear[k] = u128_zero();
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int slot = lane / K, inst = lane % K;
    const uint32_t below = (1u << (slot * K)) - 1u;
    const uint32_t range = 4 * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) + slot;
    const uint32_t lo = __ldg(bnd + range), hi = __ldg(bnd + range + 1);
    const uint32_t steps = __reduce_max_sync(0xffffffffu, (hi - lo + 1) / 2);
    const uint32_t kbefore = lo > 0 && lo < hi ? __ldg(dstv + lo - 1) : NONE - 1;
    const uint32_t kafter = lo < hi && hi < nvec ? __ldg(dstv + hi) : NONE;
    // the graph of the destinations this lane is finishing
    uint32_t g = 0, gbeg = 0, gend = 0, seed = NONE;
    double teleport = 0.0;
    u128 acc = u128_zero();
    auto finish = [&](uint32_t v, u128 x) {
        if (v < gbeg || v >= gend) {
            ppr_add_S(s_part, ap, g, inst, acc);
            acc = u128_zero();
            g = graph_of(voff, ap.G, v);
            gbeg = voff[g];
            gend = voff[g + 1];
            seed = ap.seeds[g * K + inst];
            teleport = seed != NONE ? ppr_teleport(ap, g, inst) : 0.0;
        }
        if (seed != NONE) acc = u128_add(acc, ppr_finish(ap, v, inst, x, v == seed ? teleport : 0.0));
    };
    auto cut = [&](uint32_t v, u128 x) {  // a part of a destination that other ranges share
        if (x.lo | x.hi) u128_atomic_add(rowacc + (uint64_t)v * K + inst, x);
    };
    const pk_t* const row = prop + inst;
    uint32_t ids[8];
    uint2 nk;
    auto load = [&](uint32_t v) {  // the slot's two vectors from v on, the same in its 8 lanes
        uint4 x = make_uint4(NONE, NONE, NONE, NONE), y = x;
        nk = make_uint2(NONE, NONE);
        if (v + 1 < hi) {
            x = __ldg(nbr + v);
            y = __ldg(nbr + v + 1);
            nk = __ldg(reinterpret_cast<const uint2*>(dstv + v));
        } else if (v < hi) {
            x = __ldg(nbr + v);
            nk.x = __ldg(dstv + v);
        }
        ids[0] = x.x; ids[1] = x.y; ids[2] = x.z; ids[3] = x.w;
        ids[4] = y.x; ids[5] = y.y; ids[6] = y.z; ids[7] = y.w;
    };
    load(lo);
    u128 sum = u128_zero();     // of the destination being read
    uint32_t qh = 0, nq = 0;    // complete sums waiting
    for (uint32_t i = 0, v = lo; i < steps; ++i, v += 2) {
        const uint2 k = nk;
        u128 x[2];
        pk_t p[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) p[j] = __ldg(row + (uint64_t)min(ids[j], V) * K);
        load(v + 2);
        const uint32_t far = (uint32_t)(p[0] | p[1] | p[2] | p[3] | p[4] | p[5] | p[6] | p[7]) & 64u;
        if (!__any_sync(0xffffffffu, far)) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
                x[j] = u128_add(u128_add(pk_to_fx_near(p[4 * j]), pk_to_fx_near(p[4 * j + 1])),
                                u128_add(pk_to_fx_near(p[4 * j + 2]), pk_to_fx_near(p[4 * j + 3])));
        } else {
#pragma unroll
            for (int j = 0; j < 2; ++j)
                x[j] = u128_add(u128_add(pk_to_fx(p[4 * j]), pk_to_fx(p[4 * j + 1])), u128_add(pk_to_fx(p[4 * j + 2]), pk_to_fx(p[4 * j + 3])));
        }
        const uint32_t key[3] = {k.x, k.y, v + 2 < hi ? nk.x : kafter};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            sum = u128_add(sum, x[j]);
            const bool ends = key[j] != key[j + 1] && key[j] != NONE;
            const bool whole = ends && key[j] != kbefore;
            const uint32_t m = __ballot_sync(0xffffffffu, whole) & 0x01010101u;
            if (ends) {
                if (whole) {
                    const uint32_t at = (qh + nq + __popc(m & below)) % PQ;
                    qsum[at * K + inst] = sum;
                    if (inst == 0) qvid[at] = key[j];
                } else {
                    cut(key[j], sum);
                }
                sum = u128_zero();
            }
            nq += __popc(m);
        }
        __syncwarp();
        for (; nq >= 4; nq -= 4, qh += 4) finish(qvid[(qh + slot) % PQ], qsum[(qh + slot) % PQ * K + inst]);
        __syncwarp();
    }
    if ((uint32_t)slot < nq) finish(qvid[(qh + slot) % PQ], qsum[(qh + slot) % PQ * K + inst]);
    if (kafter != NONE) cut(kafter, sum);  // nothing is left of a destination that ended
    ppr_add_S(s_part, ap, g, inst, acc);
    ppr_flush_S(s_part, nslots, ap);
}

// The rest of an iteration: the cut destinations, whose accumulators are emptied, and the seeds without
// in-edges.
__global__ void __launch_bounds__(GT) k_ppr_rest(const uint32_t* __restrict__ cuts, uint32_t nranges, const uint32_t* __restrict__ rowptr,
                                                 u128* __restrict__ rowacc, const PprApply ap)
{
    __shared__ u128 s_part[APPLY_SLOTS * K];
    const uint32_t nslots = (ap.G < (uint32_t)APPLY_SLOTS ? ap.G : (uint32_t)APPLY_SLOTS) * K;
    for (uint32_t k = threadIdx.x; k < nslots; k += GT) s_part[k] = u128_zero();
    __syncthreads();
    const uint32_t t = blockIdx.x * GT + threadIdx.x, item = t / K;
    const int inst = t % K;
    uint32_t v = NONE;
    u128 x = u128_zero();
    if (item < nranges) {
        v = __ldg(cuts + item);
        if (v != NONE) {
            u128* a = rowacc + (uint64_t)v * K + inst;
            x = *a;
            *a = u128_zero();
        }
    } else if (item - nranges < ap.G) {
        v = ap.seeds[(item - nranges) * K + inst];
        if (v != NONE && __ldg(rowptr + v + 1) > __ldg(rowptr + v)) v = NONE;
    }
    if (v != NONE) {
        const uint32_t g = graph_of(ap.voff, ap.G, v), seed = ap.seeds[g * K + inst];
        if (seed != NONE) ppr_add_S(s_part, ap, g, inst, ppr_finish(ap, v, inst, x, v == seed ? ppr_teleport(ap, g, inst) : 0.0));
    }
    ppr_flush_S(s_part, nslots, ap);
}

// ----------------------------------------------------------------------------------------------
// multi-source BFS

__global__ void k_msbfs_init(const uint32_t* __restrict__ roots, uint32_t n, uint8_t* __restrict__ visited,
                             uint8_t* __restrict__ frontier, int32_t* __restrict__ level, uint32_t* __restrict__ iter)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0 && iter) *iter = 1;  // the first iteration
    if (t >= n) return;
    const uint32_t r = roots[t];
    if (r == NONE) return;
    const uint32_t bit = 1u << (t % K);
    // several instances may share a root: byte-wise OR through the containing word
    atomicOr(reinterpret_cast<unsigned*>(visited) + (r >> 2), bit << (8 * (r & 3)));
    atomicOr(reinterpret_cast<unsigned*>(frontier) + (r >> 2), bit << (8 * (r & 3)));
    level[(uint64_t)r * K + t % K] = 0;
}

// pull: new bits of each destination = OR of its sources' frontier bytes, minus its visited bits
__global__ void __launch_bounds__(256) k_msbfs_pull(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv, uint64_t nvec,
                                                    uint32_t V, const uint8_t* __restrict__ frontier,
                                                    const uint8_t* __restrict__ visited, unsigned* __restrict__ next_words)
{
    const int lane = threadIdx.x & 31;
    const uint64_t ntiles = (nvec + 255) / 256;
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint64_t v = t * 256 + threadIdx.x;
        uint32_t key = NONE, m = 0;
        if (v < nvec) {
            key = __ldcs(dstv + v);
            if (visited[key] != 0xffu) {
                const uint4 s = __ldcs(nbr + v);
                const uint32_t ids[4] = { s.x, s.y, s.z, s.w };
#pragma unroll
                for (int l = 0; l < 4; ++l)
                    if (ids[l] < V) m |= frontier[ids[l]];
            }
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
            if (lane - off >= segstart) m |= o;
        }
        if (tail && key != NONE) {
            const uint32_t nb = m & ~(uint32_t)visited[key] & 0xffu;
            if (nb) atomicOr(next_words + (key >> 2), nb << (8 * (key & 3)));
        }
    }
}

// vertex pass: four vertices (one word) per thread; counts the new bits
__global__ void __launch_bounds__(256) k_msbfs_vertex(unsigned* __restrict__ next_words, unsigned* __restrict__ visited_words,
                                                      unsigned* __restrict__ frontier_words, int32_t* __restrict__ level,
                                                      uint32_t V, const uint32_t* __restrict__ iter,
                                                      unsigned long long* __restrict__ changed)
{
    const uint32_t W = (V + 3) / 4;
    const uint32_t k = *iter;
    unsigned long long cnt = 0;
    for (uint32_t w = blockIdx.x * 256 + threadIdx.x; w < W; w += gridDim.x * 256) {
        const unsigned nx = next_words[w];
        const unsigned vis = visited_words[w];
        const unsigned nb = nx & ~vis;
        frontier_words[w] = nb;
        if (nx) next_words[w] = 0;
        if (nb) {
            visited_words[w] = vis | nb;
            cnt += __popc(nb);
            for (int b = 0; b < 4; ++b) {
                unsigned bits = (nb >> (8 * b)) & 0xffu;
                const uint32_t v = w * 4 + b;
                while (bits) {
                    const int i = __ffs(bits) - 1;
                    bits &= bits - 1;
                    level[(uint64_t)v * K + i] = (int32_t)k;
                }
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(changed, cnt);
}

// %globaltimer into *out (one thread): the branch timers of the combined PPR + BFS graph
__global__ void k_stamp(unsigned long long* __restrict__ out)
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    *out = t;
}

// end of a BFS iteration: stop when no bit changed or the bound is reached; next iteration number
__global__ void k_msbfs_decide(unsigned long long* __restrict__ ctl, uint32_t* __restrict__ iter, uint32_t max_iter,
                               cudaGraphConditionalHandle loop)
{
    // ctl[0] changed in this iteration, ctl[1] iterations with a change, ctl[2] bound hit
    // (1: iterations, 2: time), ctl[3] %globaltimer of the first decision
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (ctl[3] == 0) ctl[3] = now;
    const unsigned long long c = ctl[0];
    ctl[0] = 0;
    unsigned run = c != 0;
    if (run) ctl[1] += 1;
    if (run && *iter >= max_iter) { run = 0; ctl[2] = 1; }
    if (run && now - ctl[3] > 120ull * 1000000000ull) { run = 0; ctl[2] = 2; }
    if (run) *iter += 1;
    cudaGraphSetConditional(loop, run);
}

}  // namespace

// ----------------------------------------------------------------------------------------------

struct grz_batch {
    int device;
    cudaStream_t stream;
    int own_stream;
    grz_graph* u;                        // the union graph
    std::vector<uint32_t> voff;          // G+1 vertex offsets
    std::vector<uint64_t> Vg, Eg;
    std::vector<std::vector<uint64_t>> pairs;  // pending pull pairs per graph (until build)
    uint32_t* d_voff;
    uint32_t* d_seeds;                   // [G][K] union vertex IDs or NONE
    // PPR
    pk_t* prop[2];                       // [V + 1][instance], packed; row V zero
    int ppr_props;                       // tuning, kept for callers: the props are packed whatever it says
    double* rank;
    u128* rowacc;                        // [V][instance]: sums of the cut destinations, zero between iterations
    uint32_t* ppr_bnd;                   // ranges of k_ppr_step (k_ppr_bounds) and the destinations they cut
    uint32_t* ppr_cut;
    void *ppr_mem, *bfs_mem;             // the allocations that hold the PPR and the BFS arrays
    u128* S[3];                          // of the props gathered, written, and of the iteration after
    cudaGraphExec_t ppr_exec;
    uint32_t ppr_iters;
    double ppr_damping;
    // BFS
    uint8_t* visited;
    uint8_t* frontier;
    unsigned* next_words;
    int32_t* level;
    unsigned long long* ctl;             // changed, iterations, bound hit
    uint32_t* iter;
    cudaGraphExec_t bfs_exec;
    // PPR and BFS together: one graph whose two branches run the two loops side by side
    uint32_t* d_roots;                   // [G][K] BFS roots of the combined run
    cudaGraphExec_t run_exec;
    uint32_t run_iters;
    double run_damping;
    unsigned long long* stamps;          // PPR start / end, BFS start / end (%globaltimer, written inside the graph)
    int ppr_blocks, bfs_blocks;          // resident blocks per SM of the persistent kernels
    void* mail;                          // pinned host read-back
    char err[256];
};

static int bset(grz_batch* b, int code, const char* msg)
{
    snprintf(b->err, sizeof(b->err), "%s", msg);
    return code;
}

static int bck(grz_batch* b, cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return GRZ_OK;
    cudaGetLastError();
    snprintf(b->err, sizeof(b->err), "%s: %s", what, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? GRZ_ERR_NOMEM : GRZ_ERR_CUDA;
}
#define BCK(b, x) do { int rc_ = bck((b), (x), #x); if (rc_) return rc_; } while (0)

static unsigned persistent_grid(const grz_batch* b, uint64_t work_blocks, int per_sm)
{
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(work_blocks, (uint64_t)b->u->num_sms * per_sm));
}

extern "C" int grz_batch_create(grz_batch** out, int device, void* stream)
{
    if (!out) return GRZ_ERR_ARG;
    *out = nullptr;
    grz_batch* b = new (std::nothrow) grz_batch();
    if (!b) return GRZ_ERR_NOMEM;
    b->device = device;
    int rc = grz_graph_create(&b->u, device, stream);
    if (rc) { delete b; return rc; }
    b->stream = b->u->stream;
    b->voff.push_back(0);
    b->ppr_blocks = 8;
    b->bfs_blocks = 8;
    *out = b;
    return GRZ_OK;
}

static void free_state(grz_batch* b)
{
    void* p[] = { b->d_voff, b->d_seeds, b->d_roots, b->stamps, b->ppr_mem, b->bfs_mem };
    for (void* x : p) cudaFree(x);
    b->d_voff = b->d_seeds = b->d_roots = nullptr;
    b->stamps = nullptr;
    b->ppr_mem = b->bfs_mem = nullptr;
    b->prop[0] = b->prop[1] = nullptr;
    b->rank = nullptr;
    b->rowacc = b->S[0] = b->S[1] = b->S[2] = nullptr;
    b->ppr_bnd = b->ppr_cut = nullptr;
    b->visited = b->frontier = nullptr;
    b->next_words = nullptr;
    b->level = nullptr;
    b->ctl = nullptr;
    b->iter = nullptr;
    if (b->ppr_exec) cudaGraphExecDestroy(b->ppr_exec);
    if (b->bfs_exec) cudaGraphExecDestroy(b->bfs_exec);
    if (b->run_exec) cudaGraphExecDestroy(b->run_exec);
    b->ppr_exec = b->bfs_exec = b->run_exec = nullptr;
}

extern "C" void grz_batch_destroy(grz_batch* b)
{
    if (!b) return;
    cudaSetDevice(b->device);
    free_state(b);
    if (b->mail) cudaFreeHost(b->mail);

    grz_graph_destroy(b->u);
    delete b;
}

extern "C" const char* grz_batch_last_error(const grz_batch* b) { return b ? b->err : ""; }

// Adds one graph: V vertices, E edges as interleaved (src, dst) pairs sorted by (dst, src) (the
// -pull order, source/graphdata.c:957).  Copied; the union is built by grz_batch_build.
extern "C" int grz_batch_add_graph(grz_batch* b, uint64_t V, uint64_t E, const uint64_t* pull_pairs)
{
    if (!b || V == 0 || (E > 0 && !pull_pairs)) return GRZ_ERR_ARG;
    if (b->voff.size() > MAX_GRAPHS) return bset(b, GRZ_ERR_RANGE, "too many graphs");
    if (V < MIN_V) return bset(b, GRZ_ERR_RANGE, "a batched graph needs at least 32 vertices");
    const uint64_t base = b->voff.back();
    if (base + V >= GRZ_HUB_BASE) return bset(b, GRZ_ERR_RANGE, "the union exceeds 2^31 vertices");
    std::vector<uint64_t> p(2 * E);
    for (uint64_t e = 0; e < E; ++e) {
        const uint64_t s = pull_pairs[2 * e], d = pull_pairs[2 * e + 1];
        if (s >= V || d >= V) return bset(b, GRZ_ERR_RANGE, "vertex ID out of range");
        if (e > 0) {
            const uint64_t ps = pull_pairs[2 * e - 2], pd = pull_pairs[2 * e - 1];
            if (d < pd || (d == pd && s < ps)) return bset(b, GRZ_ERR_UNSORTED, "pairs are not in (dst, src) order");
        }
        p[2 * e] = s + base;
        p[2 * e + 1] = d + base;
    }
    b->pairs.push_back(std::move(p));
    b->Vg.push_back(V);
    b->Eg.push_back(E);
    b->voff.push_back((uint32_t)(base + V));
    return GRZ_OK;
}

extern "C" int grz_batch_build(grz_batch* b)
{
    if (!b || b->pairs.empty()) return GRZ_ERR_ARG;
    BCK(b, cudaSetDevice(b->device));
    free_state(b);
    uint64_t E = 0;
    for (uint64_t e : b->Eg) E += e;
    std::vector<uint64_t> all;
    all.reserve(2 * E);
    for (auto& p : b->pairs) all.insert(all.end(), p.begin(), p.end());
    const uint64_t V = b->voff.back();
    int rc = grz_graph_load_pairs(b->u, V, E, E ? all.data() : nullptr, nullptr);
    if (rc) return bset(b, rc, grz_graph_last_error(b->u));
    const uint32_t G = (uint32_t)b->Vg.size();
    BCK(b, cudaMalloc((void**)&b->d_voff, sizeof(uint32_t) * (G + 1)));
    BCK(b, cudaMemcpy(b->d_voff, b->voff.data(), sizeof(uint32_t) * (G + 1), cudaMemcpyHostToDevice));
    BCK(b, cudaMalloc((void**)&b->d_seeds, sizeof(uint32_t) * G * K));
    BCK(b, cudaMalloc((void**)&b->d_roots, sizeof(uint32_t) * G * K));
    if (!b->mail) BCK(b, cudaMallocHost(&b->mail, 64));
    return GRZ_OK;
}

extern "C" int grz_batch_info(const grz_batch* b, uint64_t* graphs, uint64_t* vertices, uint64_t* edges, uint64_t* vectors)
{
    if (!b) return GRZ_ERR_ARG;
    if (graphs) *graphs = b->Vg.size();
    if (vertices) *vertices = b->voff.back();
    if (edges) *edges = b->u->E;
    if (vectors) *vectors = b->u->pull.nvec;
    return GRZ_OK;
}

static int upload_seeds(grz_batch* b, const uint32_t* local, uint32_t k, uint32_t* dst = nullptr)
{
    if (!dst) dst = b->d_seeds;
    const uint32_t G = (uint32_t)b->Vg.size();
    std::vector<uint32_t> s((size_t)G * K, NONE);
    for (uint32_t g = 0; g < G; ++g)
        for (uint32_t i = 0; i < k; ++i) {
            const uint32_t x = local[(size_t)g * k + i];
            if (x == NONE) continue;
            if (x >= b->Vg[g]) return bset(b, GRZ_ERR_ARG, "seed or root outside its graph");
            s[(size_t)g * K + i] = b->voff[g] + x;
        }
    BCK(b, cudaMemcpyAsync(dst, s.data(), sizeof(uint32_t) * s.size(), cudaMemcpyHostToDevice, b->stream));
    BCK(b, cudaStreamSynchronize(b->stream));
    return GRZ_OK;
}

// Blocks of k_ppr_step: a step of 16 vectors per warp at least, in lists that would fill the chip so, two: shorter
// ranges cut more destinations, and the BFS beside it waits for the registers.  GB300, PPR alone / with BFS, one and
// two steps at least: 3k vectors 136 / 171 and 157 / 193 us, 29k 89 / 158 and 93 / 158, 41k 95 / 162 and 97 / 155, 74k 356 / 402
// and 339 / 388, 117k 125 / 278 and 128 / 260, 210k 261 / 346 and 261 / 349.
static unsigned ppr_grid(const grz_batch* b)
{
    const uint64_t nvec = b->u->pull.nvec, least = nvec < (1u << 15) ? 16 : 32, steps = (nvec + least - 1) / least;
    return persistent_grid(b, (steps + GT / 32 - 1) / (GT / 32), std::min(b->ppr_blocks, PPR_RESIDENT));
}

// the ranges of k_ppr_step, before its graph is captured: a graph's launches have the grid of its capture,
// and a change of ppr_blocks drops the captured graphs
static int ppr_ranges(grz_batch* b)
{
    grz_graph* u = b->u;
    const uint32_t nwarps = ppr_grid(b) * (GT / 32), nranges = 4 * nwarps;
    k_ppr_bounds<<<nwarps / 256 + 1, 256, 0, b->stream>>>(u->pull.shared, (uint32_t)u->pull.nvec, (uint32_t)u->V, nwarps, b->ppr_bnd);
    k_ppr_cuts<<<(nranges + 255) / 256, 256, 0, b->stream>>>(u->pull.shared, b->ppr_bnd, nranges, b->ppr_cut);
    return bck(b, cudaGetLastError(), "ppr ranges");
}

// Enqueues the PPR's initial state and its fixed-length loop (k_ppr_step, k_ppr_rest per iteration) on cs.
static int enqueue_ppr(grz_batch* b, cudaStream_t cs, uint32_t iterations, double damping)
{
    grz_graph* u = b->u;
    const uint32_t V = (uint32_t)u->V, G = (uint32_t)b->Vg.size(), nvec = (uint32_t)u->pull.nvec;
    // the props and the ranks, neighbours in memory (ppr_alloc)
    BCK(b, cudaMemsetAsync(b->prop[0], 0, (size_t)((char*)(b->rank + (uint64_t)V * K) - (char*)b->prop[0]), cs));
    k_ppr_init<<<(G * K + 255) / 256, 256, 0, cs>>>(b->d_seeds, G, u->inv_deg, u->degree, b->prop[0], b->S[0], b->S[1]);
    const unsigned grid = ppr_grid(b);
    const uint32_t nranges = 4 * grid * (GT / 32);
    PprApply ap;
    ap.inv_deg = u->inv_deg;
    ap.degree = u->degree;
    ap.voff = b->d_voff;
    ap.G = G;
    ap.seeds = b->d_seeds;
    ap.damping = damping;
    for (uint32_t it = 0; it < iterations; ++it) {
        ap.S = b->S[it % 3];
        ap.S_next = b->S[(it + 1) % 3];
        ap.prop_out = b->prop[(it & 1) ^ 1];
        ap.rank_out = it + 1 == iterations ? b->rank : nullptr;
        k_ppr_step<<<grid, GT, 0, cs>>>(u->pull.nbr, u->pull.shared, b->ppr_bnd, nvec, V, b->prop[it & 1], b->rowacc, b->S[(it + 2) % 3],
                                       ap);
        k_ppr_rest<<<(unsigned)(((uint64_t)(nranges + G) * K + GT - 1) / GT), GT, 0, cs>>>(b->ppr_cut, nranges, u->pull.rowptr, b->rowacc, ap);
    }
    return bck(b, cudaGetLastError(), "ppr launch");
}

// a PPR run as one CUDA graph
static int build_ppr_graph(grz_batch* b, uint32_t iterations, double damping)
{
    if (b->ppr_exec) { cudaGraphExecDestroy(b->ppr_exec); b->ppr_exec = nullptr; }
    const int rr = ppr_ranges(b);
    if (rr) return rr;
    cudaStream_t cs = nullptr;
    BCK(b, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    int rc = bck(b, cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal), "begin capture");
    if (!rc) rc = enqueue_ppr(b, cs, iterations, damping);
    const cudaError_t e = cudaStreamEndCapture(cs, &graph);
    if (!rc) rc = bck(b, e, "end capture");
    if (!rc) rc = bck(b, cudaGraphInstantiate(&b->ppr_exec, graph, 0), "instantiate");
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(cs);
    if (rc) { b->ppr_exec = nullptr; return rc; }
    b->ppr_iters = iterations;
    b->ppr_damping = damping;
    return GRZ_OK;
}

// the PPR state (props, ranks, accumulators), allocated on first use, in one call (GB300, what a batch's first run takes
// beyond the next, nine and one: three graphs of 1400 vertices in all 215 and 190 us, eight of 1.04M 770 and 610 us)
static int ppr_alloc(grz_batch* b)
{
    const uint64_t V = b->u->V;
    const uint32_t G = (uint32_t)b->Vg.size();
    if (b->prop[0]) return GRZ_OK;
    const uint64_t max_ranges = 4ull * (GT / 32) * b->u->num_sms * PPR_RESIDENT;
    const size_t s = sizeof(u128) * G * K;
    const grz_part part[] = { { (void**)&b->prop[0], sizeof(pk_t) * (V + 1) * K }, { (void**)&b->prop[1], sizeof(pk_t) * (V + 1) * K },
                              { (void**)&b->rank, sizeof(double) * V * K }, { (void**)&b->rowacc, sizeof(u128) * V * K },
                              { (void**)&b->S[0], s }, { (void**)&b->S[1], s }, { (void**)&b->S[2], s },
                              { (void**)&b->ppr_bnd, sizeof(uint32_t) * (max_ranges + 1) }, { (void**)&b->ppr_cut, sizeof(uint32_t) * max_ranges } };
    BCK(b, grz_alloc_arrays(part, sizeof(part) / sizeof(part[0]), &b->ppr_mem));
    for (pk_t* p : b->prop) BCK(b, cudaMemsetAsync(p + V * K, 0, sizeof(pk_t) * K, b->stream));
    BCK(b, cudaMemsetAsync(b->rowacc, 0, sizeof(u128) * V * K, b->stream));
    return GRZ_OK;
}

// k seeds per graph (local vertex IDs, NONE = unused instance), `iterations` PPR iterations;
// ranks out as [union vertex][k] (graph g's vertex v at row voff[g] + v)
extern "C" int grz_batch_ppr(grz_batch* b, const uint32_t* seeds, uint32_t k, uint32_t iterations, double damping,
                             double* ranks_out, grz_run_stats_t* stats)
{
    if (!b || !seeds || k == 0 || k > (uint32_t)K || iterations == 0 || !(damping >= 0.0 && damping <= 1.0)) return GRZ_ERR_ARG;
    if (!b->d_seeds) return bset(b, GRZ_ERR_STATE, "grz_batch_build not called");
    BCK(b, cudaSetDevice(b->device));
    grz_graph* u = b->u;
    const uint64_t V = u->V;
    int rc = ppr_alloc(b);
    if (rc) return rc;
    rc = upload_seeds(b, seeds, k);
    if (rc) return rc;
    if (!b->ppr_exec || b->ppr_iters != iterations || b->ppr_damping != damping) {
        rc = build_ppr_graph(b, iterations, damping);
        if (rc) return rc;
    }
    cudaEvent_t e0, e1;
    BCK(b, cudaEventCreate(&e0));
    BCK(b, cudaEventCreate(&e1));
    cudaStream_t st = b->stream;
    rc = bck(b, cudaEventRecord(e0, st), "event");
    if (!rc) rc = bck(b, cudaGraphLaunch(b->ppr_exec, st), "graph launch");
    if (!rc) rc = bck(b, cudaEventRecord(e1, st), "event");
    if (!rc && ranks_out) {
        if (k == (uint32_t)K) {
            rc = bck(b, cudaMemcpyAsync(ranks_out, b->rank, sizeof(double) * V * K, cudaMemcpyDeviceToHost, st), "D2H");
        } else {
            rc = bck(b, cudaMemcpy2DAsync(ranks_out, sizeof(double) * k, b->rank, sizeof(double) * K, sizeof(double) * k, V,
                                          cudaMemcpyDeviceToHost, st), "D2H");
        }
    }
    if (!rc) rc = bck(b, cudaStreamSynchronize(st), "run");
    if (!rc && stats) {
        memset(stats, 0, sizeof(*stats));
        stats->iterations = iterations;
        stats->pull_iterations = iterations;
        cudaEventElapsedTime(&stats->ms, e0, e1);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    u->nlaunch += 1 + 2ull * iterations;
    return rc;
}

// Adds to `graph`, after `deps`, the BFS loop: WHILE (a bit changed) { pull; vertex pass; decide }.
static int add_bfs_loop(grz_batch* b, cudaGraph_t graph, const cudaGraphNode_t* deps, size_t ndeps, cudaGraphNode_t* node_out)
{
    grz_graph* u = b->u;
    const uint32_t V = (uint32_t)u->V;
    cudaGraphConditionalHandle loop = 0;
    int rc = bck(b, cudaGraphConditionalHandleCreate(&loop, graph, 1, cudaGraphCondAssignDefault), "handle");
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = loop;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node = nullptr;
    if (!rc) rc = bck(b, cudaGraphAddNode(&node, graph, deps, nullptr, ndeps, &p), "while node");
    cudaStream_t cs = nullptr;
    if (!rc) rc = bck(b, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "stream");
    if (!rc) rc = bck(b, cudaStreamBeginCaptureToGraph(cs, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                      cudaStreamCaptureModeThreadLocal), "capture");
    if (!rc) {
        const unsigned pgrid = persistent_grid(b, (u->pull.nvec + 255) / 256, b->bfs_blocks);
        const unsigned vgrid = persistent_grid(b, ((V + 3) / 4 + 255) / 256, b->bfs_blocks);
        k_msbfs_pull<<<pgrid, 256, 0, cs>>>(u->pull.nbr, u->pull.shared, u->pull.nvec, V, b->frontier, b->visited, b->next_words);
        k_msbfs_vertex<<<vgrid, 256, 0, cs>>>(b->next_words, reinterpret_cast<unsigned*>(b->visited),
                                              reinterpret_cast<unsigned*>(b->frontier), b->level, V, b->iter, b->ctl);
        k_msbfs_decide<<<1, 1, 0, cs>>>(b->ctl, b->iter, V + 1, loop);
        rc = bck(b, cudaGetLastError(), "bfs launch");
        cudaGraph_t g2 = nullptr;
        const cudaError_t e = cudaStreamEndCapture(cs, &g2);
        if (!rc) rc = bck(b, e, "end capture");
    }
    if (cs) cudaStreamDestroy(cs);
    *node_out = node;
    return rc;
}

// the BFS loop as one CUDA graph
static int build_bfs_graph(grz_batch* b)
{
    if (b->bfs_exec) { cudaGraphExecDestroy(b->bfs_exec); b->bfs_exec = nullptr; }
    cudaGraph_t top = nullptr;
    BCK(b, cudaGraphCreate(&top, 0));
    cudaGraphNode_t node = nullptr;
    int rc = add_bfs_loop(b, top, nullptr, 0, &node);
    if (!rc) rc = bck(b, cudaGraphInstantiate(&b->bfs_exec, top, 0), "instantiate");
    cudaGraphDestroy(top);
    if (rc) b->bfs_exec = nullptr;
    return rc;
}

// the multi-source BFS state, allocated on first use
static int bfs_alloc(grz_batch* b)
{
    const uint64_t V = b->u->V;
    const uint64_t Vw = (V + 3) / 4 * 4;
    if (!b->visited) {
        const grz_part part[] = { { (void**)&b->visited, Vw }, { (void**)&b->frontier, Vw }, { (void**)&b->next_words, Vw },
                                  { (void**)&b->ctl, sizeof(unsigned long long) * 4 }, { (void**)&b->iter, sizeof(uint32_t) },
                                  { (void**)&b->level, sizeof(int32_t) * V * K } };
        BCK(b, grz_alloc_arrays(part, sizeof(part) / sizeof(part[0]), &b->bfs_mem));
    }
    return GRZ_OK;
}

// no vertex visited, no level: the bitmaps and the control words are neighbours in memory (bfs_alloc)
static int bfs_clear(grz_batch* b, cudaStream_t st)
{
    BCK(b, cudaMemsetAsync(b->visited, 0, (size_t)((char*)(b->ctl + 4) - (char*)b->visited), st));
    BCK(b, cudaMemsetAsync(b->level, 0xff, sizeof(int32_t) * b->u->V * K, st));
    return GRZ_OK;
}

// the last node of the work captured so far on cs (one node), then ends the capture
static int end_capture_sink(grz_batch* b, cudaStream_t cs, cudaGraphNode_t* sink)
{
    cudaStreamCaptureStatus st;
    const cudaGraphNode_t* deps = nullptr;
    size_t n = 0;
    const cudaError_t e = cudaStreamGetCaptureInfo(cs, &st, nullptr, nullptr, &deps, nullptr, &n);
    const cudaGraphNode_t last = (e == cudaSuccess && n == 1) ? deps[0] : nullptr;
    cudaGraph_t out = nullptr;
    const cudaError_t e2 = cudaStreamEndCapture(cs, &out);
    if (e != cudaSuccess) return bck(b, e, "capture info");
    if (e2 != cudaSuccess) return bck(b, e2, "end capture");
    if (sink) {
        if (!last) return bset(b, GRZ_ERR_STATE, "captured work does not end in one node");
        *sink = last;
    }
    return GRZ_OK;
}

// PPR and multi-source BFS as one CUDA graph with two independent branches, each from its initial
// state to its results: branch 1 the PPR loop (d_seeds), branch 2 the BFS loop (d_roots).  Event
// records at both ends of each branch time them inside the one launch.
static int build_run_graph(grz_batch* b, uint32_t iterations, double damping)
{
    if (b->run_exec) { cudaGraphExecDestroy(b->run_exec); b->run_exec = nullptr; }
    if (!b->stamps) BCK(b, cudaMalloc((void**)&b->stamps, 4 * sizeof(unsigned long long)));
    const int rr = ppr_ranges(b);
    if (rr) return rr;
    grz_graph* u = b->u;
    const uint64_t V = u->V;
    const uint32_t G = (uint32_t)b->Vg.size();
    cudaGraph_t top = nullptr;
    BCK(b, cudaGraphCreate(&top, 0));
    cudaStream_t cs = nullptr;
    int rc = bck(b, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "stream");
    // branch 1: PPR
    if (!rc) rc = bck(b, cudaStreamBeginCaptureToGraph(cs, top, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal), "capture");
    if (!rc) {
        k_stamp<<<1, 1, 0, cs>>>(b->stamps + 0);
        rc = enqueue_ppr(b, cs, iterations, damping);
        k_stamp<<<1, 1, 0, cs>>>(b->stamps + 1);
        const int rc2 = end_capture_sink(b, cs, nullptr);
        if (!rc) rc = rc2;
    }
    // branch 2: BFS (no dependency on branch 1)
    cudaGraphNode_t init = nullptr, loop = nullptr;
    if (!rc) rc = bck(b, cudaStreamBeginCaptureToGraph(cs, top, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal), "capture");
    if (!rc) {
        k_stamp<<<1, 1, 0, cs>>>(b->stamps + 2);
        rc = bfs_clear(b, cs);
        k_msbfs_init<<<(G * K + 255) / 256, 256, 0, cs>>>(b->d_roots, G * K, b->visited, b->frontier, b->level, b->iter);
        if (!rc) rc = bck(b, cudaGetLastError(), "bfs init");
        const int rc2 = end_capture_sink(b, cs, &init);
        if (!rc) rc = rc2;
    }
    if (!rc) rc = add_bfs_loop(b, top, &init, 1, &loop);
    if (!rc) rc = bck(b, cudaStreamBeginCaptureToGraph(cs, top, &loop, nullptr, 1, cudaStreamCaptureModeThreadLocal), "capture");
    if (!rc) {
        k_stamp<<<1, 1, 0, cs>>>(b->stamps + 3);
        rc = bck(b, cudaGetLastError(), "stamp");
        const int rc2 = end_capture_sink(b, cs, nullptr);
        if (!rc) rc = rc2;
    }
    if (cs) cudaStreamDestroy(cs);
    if (!rc) rc = bck(b, cudaGraphInstantiate(&b->run_exec, top, 0), "instantiate");
    cudaGraphDestroy(top);
    if (rc) { b->run_exec = nullptr; return rc; }
    b->run_iters = iterations;
    b->run_damping = damping;
    return GRZ_OK;
}

// k roots per graph (local IDs, NONE = unused instance); levels out as [union vertex][k]
// (-1 = unreached)
extern "C" int grz_batch_msbfs(grz_batch* b, const uint32_t* roots, uint32_t k, int32_t* levels_out, grz_run_stats_t* stats)
{
    if (!b || !roots || k == 0 || k > (uint32_t)K) return GRZ_ERR_ARG;
    if (!b->d_seeds) return bset(b, GRZ_ERR_STATE, "grz_batch_build not called");
    BCK(b, cudaSetDevice(b->device));
    grz_graph* u = b->u;
    const uint64_t V = u->V;
    const uint32_t G = (uint32_t)b->Vg.size();
    int rc = bfs_alloc(b);
    if (rc) return rc;
    rc = upload_seeds(b, roots, k);
    if (rc) return rc;
    if (!b->bfs_exec) {
        rc = build_bfs_graph(b);
        if (rc) return rc;
    }
    cudaStream_t st = b->stream;
    cudaEvent_t e0, e1;
    BCK(b, cudaEventCreate(&e0));
    BCK(b, cudaEventCreate(&e1));
    const uint32_t one = 1;
    rc = bck(b, cudaEventRecord(e0, st), "event");
    if (!rc) rc = bfs_clear(b, st);
    if (!rc) {
        memcpy(b->mail, &one, sizeof(one));
        rc = bck(b, cudaMemcpyAsync(b->iter, b->mail, sizeof(uint32_t), cudaMemcpyHostToDevice, st), "H2D");
    }
    if (!rc) {
        k_msbfs_init<<<(G * K + 255) / 256, 256, 0, st>>>(b->d_seeds, G * K, b->visited, b->frontier, b->level, nullptr);
        rc = bck(b, cudaGetLastError(), "bfs init");
    }
    if (!rc) rc = bck(b, cudaGraphLaunch(b->bfs_exec, st), "graph launch");
    if (!rc) rc = bck(b, cudaEventRecord(e1, st), "event");
    if (!rc) rc = bck(b, cudaMemcpyAsync(b->mail, b->ctl, sizeof(unsigned long long) * 3, cudaMemcpyDeviceToHost, st), "D2H");
    if (!rc && levels_out) {
        if (k == (uint32_t)K)
            rc = bck(b, cudaMemcpyAsync(levels_out, b->level, sizeof(int32_t) * V * K, cudaMemcpyDeviceToHost, st), "D2H");
        else
            rc = bck(b, cudaMemcpy2DAsync(levels_out, sizeof(int32_t) * k, b->level, sizeof(int32_t) * K, sizeof(int32_t) * k, V,
                                          cudaMemcpyDeviceToHost, st), "D2H");
    }
    if (!rc) rc = bck(b, cudaStreamSynchronize(st), "run");
    unsigned long long c[3];
    memcpy(c, b->mail, sizeof(c));
    if (!rc && c[2] == 1) rc = bset(b, GRZ_ERR_TIMEOUT, "BFS did not converge within V + 1 iterations");
    if (!rc && c[2] == 2) rc = bset(b, GRZ_ERR_TIMEOUT, "BFS stopped by its time bound");
    if (!rc && stats) {
        memset(stats, 0, sizeof(*stats));
        stats->iterations = (uint32_t)c[1] + 1;  // the last iteration found nothing new
        stats->pull_iterations = stats->iterations;
        cudaEventElapsedTime(&stats->ms, e0, e1);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    u->nlaunch += 1 + 3ull * (c[1] + 1);
    return rc;
}

// PPR (seeds, k per graph, `iterations`) and multi-source BFS (roots, kb per graph) in one CUDA
// graph launch: the two loops run side by side as independent branches of one graph, each from
// its initial state.  Results and per-branch device times as grz_batch_ppr / grz_batch_msbfs;
// *total_ms is the launch's device time.
extern "C" int grz_batch_run(grz_batch* b, const uint32_t* seeds, uint32_t k, uint32_t iterations, double damping,
                             const uint32_t* roots, uint32_t kb, double* ranks_out, int32_t* levels_out,
                             grz_run_stats_t* ppr_stats, grz_run_stats_t* bfs_stats, float* total_ms)
{
    if (!b || !seeds || !roots || k == 0 || k > (uint32_t)K || kb == 0 || kb > (uint32_t)K || iterations == 0 ||
        !(damping >= 0.0 && damping <= 1.0))
        return GRZ_ERR_ARG;
    if (!b->d_seeds) return bset(b, GRZ_ERR_STATE, "grz_batch_build not called");
    BCK(b, cudaSetDevice(b->device));
    grz_graph* u = b->u;
    const uint64_t V = u->V;
    int rc = ppr_alloc(b);
    if (!rc) rc = bfs_alloc(b);
    if (!rc) rc = upload_seeds(b, seeds, k, b->d_seeds);
    if (!rc) rc = upload_seeds(b, roots, kb, b->d_roots);
    if (rc) return rc;
    if (!b->run_exec || b->run_iters != iterations || b->run_damping != damping) {
        rc = build_run_graph(b, iterations, damping);
        if (rc) return rc;
    }
    cudaStream_t st = b->stream;
    cudaEvent_t e0, e1;
    BCK(b, cudaEventCreate(&e0));
    BCK(b, cudaEventCreate(&e1));
    rc = bck(b, cudaEventRecord(e0, st), "event");
    if (!rc) rc = bck(b, cudaGraphLaunch(b->run_exec, st), "graph launch");
    if (!rc) rc = bck(b, cudaEventRecord(e1, st), "event");
    if (!rc) rc = bck(b, cudaMemcpyAsync(b->mail, b->ctl, sizeof(unsigned long long) * 3, cudaMemcpyDeviceToHost, st), "D2H");
    if (!rc) rc = bck(b, cudaMemcpyAsync((unsigned long long*)b->mail + 4, b->stamps, 4 * sizeof(unsigned long long),
                                         cudaMemcpyDeviceToHost, st), "D2H");
    if (!rc && ranks_out) {
        if (k == (uint32_t)K) {
            rc = bck(b, cudaMemcpyAsync(ranks_out, b->rank, sizeof(double) * V * K, cudaMemcpyDeviceToHost, st), "D2H");
        } else {
            rc = bck(b, cudaMemcpy2DAsync(ranks_out, sizeof(double) * k, b->rank, sizeof(double) * K, sizeof(double) * k, V,
                                          cudaMemcpyDeviceToHost, st), "D2H");
        }
    }
    if (!rc && levels_out) {
        if (kb == (uint32_t)K)
            rc = bck(b, cudaMemcpyAsync(levels_out, b->level, sizeof(int32_t) * V * K, cudaMemcpyDeviceToHost, st), "D2H");
        else
            rc = bck(b, cudaMemcpy2DAsync(levels_out, sizeof(int32_t) * kb, b->level, sizeof(int32_t) * K, sizeof(int32_t) * kb, V,
                                          cudaMemcpyDeviceToHost, st), "D2H");
    }
    if (!rc) rc = bck(b, cudaStreamSynchronize(st), "run");
    unsigned long long c[3];
    memcpy(c, b->mail, sizeof(c));
    if (!rc && c[2] == 1) rc = bset(b, GRZ_ERR_TIMEOUT, "BFS did not converge within V + 1 iterations");
    if (!rc && c[2] == 2) rc = bset(b, GRZ_ERR_TIMEOUT, "BFS stopped by its time bound");
    if (!rc) {
        const unsigned long long* ts = (const unsigned long long*)b->mail + 4;
        if (ppr_stats) {
            memset(ppr_stats, 0, sizeof(*ppr_stats));
            ppr_stats->iterations = ppr_stats->pull_iterations = iterations;
            ppr_stats->ms = (float)((double)(ts[1] - ts[0]) * 1e-6);
        }
        if (bfs_stats) {
            memset(bfs_stats, 0, sizeof(*bfs_stats));
            bfs_stats->iterations = bfs_stats->pull_iterations = (uint32_t)c[1] + 1;
            bfs_stats->ms = (float)((double)(ts[3] - ts[2]) * 1e-6);
        }
        if (total_ms) cudaEventElapsedTime(total_ms, e0, e1);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    u->nlaunch += 2 + 2ull * iterations + 1 + 3ull * (c[1] + 1);
    return rc;
}

extern "C" int grz_batch_tune_set(grz_batch* b, int param, int64_t value)
{
    if (!b) return GRZ_ERR_ARG;
    if (param == GRZ_BATCH_TUNE_PPR_PROPS) {
        if (value < 0 || value > 2) return bset(b, GRZ_ERR_RANGE, "PPR props must be 0, 1 or 2");
        b->ppr_props = (int)value;
        return GRZ_OK;
    }
    if (value < 1 || value > 32) return bset(b, GRZ_ERR_RANGE, "blocks per SM must be 1..32");
    int* slot = param == GRZ_BATCH_TUNE_PPR_BLOCKS ? &b->ppr_blocks : (param == GRZ_BATCH_TUNE_BFS_BLOCKS ? &b->bfs_blocks : nullptr);
    if (!slot) return bset(b, GRZ_ERR_ARG, "unknown batch tuning parameter");
    if (*slot != (int)value) {
        *slot = (int)value;
        // the captured loops bake the grid in: capture again at the next run
        cudaSetDevice(b->device);
        if (param == GRZ_BATCH_TUNE_PPR_BLOCKS && b->ppr_exec) { cudaGraphExecDestroy(b->ppr_exec); b->ppr_exec = nullptr; }
        if (param == GRZ_BATCH_TUNE_BFS_BLOCKS && b->bfs_exec) { cudaGraphExecDestroy(b->bfs_exec); b->bfs_exec = nullptr; }
        if (b->run_exec) { cudaGraphExecDestroy(b->run_exec); b->run_exec = nullptr; }
    }
    return GRZ_OK;
}

extern "C" int grz_batch_tune_get(const grz_batch* b, int param, int64_t* value)
{
    if (!b || !value) return GRZ_ERR_ARG;
    if (param == GRZ_BATCH_TUNE_PPR_BLOCKS) *value = b->ppr_blocks;
    else if (param == GRZ_BATCH_TUNE_BFS_BLOCKS) *value = b->bfs_blocks;
    else if (param == GRZ_BATCH_TUNE_PPR_PROPS) *value = b->ppr_props;
    else return GRZ_ERR_ARG;
    return GRZ_OK;
}

extern "C" unsigned long long grz_batch_launch_count(const grz_batch* b) { return b ? b->u->nlaunch : 0ull; }
