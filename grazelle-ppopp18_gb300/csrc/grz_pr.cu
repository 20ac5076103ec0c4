// grz_pr.cu -- PageRank edge-pull and vertex phases on the vector-sparse layout.
//
// Reference semantics (source/phase_edge_pull_pr.asm:45-171, source/phase_vertex_pr.asm:27-134):
//   accum[v] = sum over v's in-edge vectors of the props of the valid source lanes
//   S        = sum of all accumulators (the "PageRank sum" of the reduce buffer)
//   prop[v]  = ((accum[v] + (1 - S)/V) * d + (1 - d)/V) / (outdeg[v] == 0 ? V : outdeg[v])
//
// GB300 design:
//   * Accumulation is exact in unsigned 4.124 fixed point (u128).  The gathered values are the
//     props converted exactly from double.  Integer addition is associative, so each sum is the
//     exact sum of the reference's double inputs, rounded once to double.  The result is
//     independent of tile shape, thread count and scheduling.  GB300's FP64 pipe runs at ~1/58
//     of its integer rate, so FP64 adds per edge would bound the kernel.
//   * The gathers bound the iteration: about one line request per SM clock.  The iterations of
//     grz_pr_iterate therefore gather 8-byte packed props (pk_to_fx), and take those of the sources
//     with the highest out-degrees from shared memory (k_pr_gather_pk): in a power-law graph 20000
//     sources are more than half of the edges at R-MAT 20.  Each thread sums four consecutive vectors, a
//     warp-segmented scan joins the threads, and a warp walks a contiguous range of the list, so
//     only the destinations cut by the ends of a range are combined with exact u128 atomics, in any
//     order.  This replaces the reference's work-unit merge buffer (source/phases.c:41-70); no
//     thread ever waits on another.
//   * The apply kernel is the vertex phase.  It also accumulates S_{k+1} = sum_u outdeg[u] *
//     prop_{k+1}[u] exactly, which equals iteration k+1's sum of accumulators, so an iteration is
//     two kernels with no host round trip.
//   * The vertex formula is fma(acc, d, G*d + (1-d)/V) times a precomputed 1/deg'.  It stays
//     within a few roundings of the reference's ((acc + G)*d + (1-d)/V) / deg': two FP64 ops
//     per vertex instead of three plus a division, on a part whose FP64 rate is low.
#include <cooperative_groups.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "grz_internal.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int PR_THREADS = 256;

// The gathers and applies of grz_pr_iterate start while the kernel before them ends (programmatic
// dependent launch): pdl_start lets the next kernel of the stream begin, pdl_wait holds until the one
// before has completed and its writes are visible.  What a kernel reads before pdl_wait (the lists,
// the degrees) no kernel of the chain writes.  What the chain does write (props, hot table, sums,
// accumulators, the iteration's constant) comes through the coherent path and through pointers taken
// after the wait (after_wait): the read-only path asks for data that stays the same for the whole kernel, and
// a load through a pointer known before may be moved above the wait.  GB300, us per iteration, plain launches -> these: R-MAT of 4096
// vertices 10.3 -> 7.3, of 50k 12.4 -> 9.8, of 2^20 59 -> 56.
__device__ __forceinline__ void pdl_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename T>
__device__ __forceinline__ T* after_wait(T* p)
{
    asm volatile("" : "+l"(p) : : "memory");
    return p;
}

template <typename... P, typename... A>
cudaError_t pdl_launch(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

__device__ __forceinline__ u128 ld_fx(const u128* p, uint32_t i)
{
#if GRZ_GATHER_LD == 1
    u128 r;
    asm("ld.global.nc.L1::evict_last.v2.u64 {%0, %1}, [%2];" : "=l"(r.lo), "=l"(r.hi) : "l"(p + i));
    return r;
#else
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p) + i);
    u128 r;
    r.lo = v.x;
    r.hi = v.y;
    return r;
#endif
}

// a gathered prop as fixed point: stored so (16 bytes), or packed (8 bytes: half the gathered
// working set, the same sums)
typedef unsigned long long pk_t;
__device__ __forceinline__ u128 ld_prop(const u128* p, uint32_t i) { return ld_fx(p, i); }
__device__ __forceinline__ u128 ld_prop(const pk_t* p, uint32_t i) { return pk_to_fx(__ldg(p + i)); }

// a packed prop through the coherent path, L1-cached (nothing writes the props while they are read)
__device__ __forceinline__ pk_t ld_l1(const pk_t* p)
{
    pk_t x;
    asm("ld.global.u64 %0, [%1];" : "=l"(x) : "l"(p));
    return x;
}

// The same through the coherent path (ld.global, L1-cached): for the persistent kernel, whose
// apply phase rewrites the props that a later gather phase of the same launch reads, which the
// read-only (non-coherent) path does not allow.
__device__ __forceinline__ u128 ld_prop_coh(const u128* p, uint32_t i)
{
    u128 r;
    asm volatile("ld.global.v2.u64 {%0, %1}, [%2];" : "=l"(r.lo), "=l"(r.hi) : "l"(p + i));
    return r;
}
__device__ __forceinline__ u128 ld_prop_coh(const pk_t* p, uint32_t i)
{
    pk_t x;
    asm volatile("ld.global.u64 %0, [%1];" : "=l"(x) : "l"(p + i));
    return pk_to_fx(x);
}

// per-iteration constants handed from the gather kernel to the apply kernel
struct PRConst {
    const u128* part_in;  // per-block partial sums whose total is S_k (exact)
    uint32_t nparts;
    double* K_out;        // G*d + (1-d)/V
    double damping, c, nverts;
};

__device__ __forceinline__ u128 u128_shfl_up(u128 v, int off)
{
    u128 r;
    r.lo = __shfl_up_sync(0xffffffffu, v.lo, off);
    r.hi = __shfl_up_sync(0xffffffffu, v.hi, off);
    return r;
}

// Edge-pull gather: one thread per vector.  Each vector's four source props are summed exactly
// in the reference's lane order (g2+g3)+(g0+g1) (phase_edge_pull_pr.asm:146-149); integer
// addition makes the order immaterial anyway.  A warp-segmented inclusive scan over the
// destination keys then sums the vectors of each destination within the warp.  A destination
// whose vectors all lie in this warp is stored with one plain store.  One that continues into a
// neighbouring warp is combined across the block and stored once; only a destination whose
// vectors straddle the block's tile edge is added with exact u128 atomics, so only those
// accumulators must be zero on entry (the fused apply clears exactly those, marked in pr_cut).
// A destination with no in-edges is never touched and stays 0.  The loads of nbr/dst are
// streamed once (evict-first); the prop gathers go through L1.  P is the gathered props' type:
// u128 fixed point, or packed.  This is the general form: the phases.h calls (any vector range),
// hub-encoded lists, and 16-byte props when asked for; grz_pr_iterate's packed props go through
// k_pr_gather_pk.
__device__ __forceinline__ u128 block_reduce_u128(u128 s, u128* red);

// shared memory of the gather's block combine
struct GatherSmem {
    static constexpr int NW = PR_THREADS / 32;
    uint32_t key[2][NW];
    u128 sum[2][NW];
    uint32_t flag[2][NW];  // bit0 present, bit1 head real, bit2 tail real
    u128 red[NW];
};

// once per iteration (block 0 of the gather): S_k from the previous apply's per-block partials,
// then K = G*d + (1-d)/V with G = (1 - S_k)/V
__device__ __forceinline__ void pr_publish_K(const PRConst& pc, u128* red)
{
    u128 S = u128_zero();
    for (uint32_t b = threadIdx.x; b < pc.nparts; b += PR_THREADS) S = u128_add(S, pc.part_in[b]);
    S = block_reduce_u128(S, red);
    if (threadIdx.x == 0) *pc.K_out = __fma_rn((1.0 - fx_to_double(S)) / pc.nverts, pc.damping, pc.c);
}

// A destination's sum.  ADD: the accumulators already hold the sums of earlier launches (source
// segments); a destination owned by one warp is added by a plain read-modify-write, one cut by the
// edge of a range atomically.
__device__ __forceinline__ void rowacc_put(u128* rowacc, uint32_t key, u128 val, bool add)
{
    ulonglong2* p = reinterpret_cast<ulonglong2*>(rowacc) + key;
    if (add) {
        const ulonglong2 o = __ldcg(p);
        u128 a;
        a.lo = o.x;
        a.hi = o.y;
        val = u128_add(val, a);
    }
    __stcg(p, make_ulonglong2(val.lo, val.hi));
}

// The gather over tiles blockIdx.x, blockIdx.x + nblocks, ... of PR_THREADS vectors.
template <typename P, bool COH>
__device__ __forceinline__ void pr_gather_tiles(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv, uint64_t first,
                                                uint64_t nvec, uint64_t list_nvec, const P* __restrict__ prop_fx, uint32_t V,
                                                u128* __restrict__ rowacc, const uint32_t* __restrict__ hub_vid, uint32_t nhub,
                                                uint32_t block, uint32_t nblocks, GatherSmem& sm)
{
    constexpr int NW = GatherSmem::NW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // vector indices stay below 2^32 (the lists' limit), so the index arithmetic is 32-bit
    const uint32_t ntiles = (uint32_t)((nvec + PR_THREADS - 1) / PR_THREADS);
    const uint32_t first32 = (uint32_t)first, nvec32 = (uint32_t)nvec, list32 = (uint32_t)list_nvec;
    for (uint32_t tile = block; tile < ntiles; tile += nblocks) {
        if (lane < 2) sm.flag[lane][warp] = 0;
        const uint32_t i = tile * PR_THREADS + threadIdx.x;
        const uint32_t v = first32 + i;
        const bool live = i < nvec32;
        uint32_t key = 0xffffffffu;
        u128 val = u128_zero();
        if (live) {
            const uint4 s = ld_stream(nbr + v);
            key = ld_stream(dstv + v);
            const uint32_t i0 = min(grz_hub_decode(s.x, hub_vid, nhub), V), i1 = min(grz_hub_decode(s.y, hub_vid, nhub), V);
            const uint32_t i2 = min(grz_hub_decode(s.z, hub_vid, nhub), V), i3 = min(grz_hub_decode(s.w, hub_vid, nhub), V);
            const u128 g0 = COH ? ld_prop_coh(prop_fx, i0) : ld_prop(prop_fx, i0);
            const u128 g1 = COH ? ld_prop_coh(prop_fx, i1) : ld_prop(prop_fx, i1);
            const u128 g2 = COH ? ld_prop_coh(prop_fx, i2) : ld_prop(prop_fx, i2);
            const u128 g3 = COH ? ld_prop_coh(prop_fx, i3) : ld_prop(prop_fx, i3);
            val = u128_add(u128_add(g2, g3), u128_add(g0, g1));
        }
        uint32_t prevkey = __shfl_up_sync(0xffffffffu, key, 1);
        uint32_t nextkey = __shfl_down_sync(0xffffffffu, key, 1);
        // neighbours across the warp edge come from the whole list, so a destination cut by the edge of
        // a caller's vector range is also added atomically, from both sides
        if (lane == 0) prevkey = (live && v > 0) ? __ldg(dstv + v - 1) : 0xfffffffeu;
        if (lane == 31) nextkey = (live && v + 1 < list32) ? __ldg(dstv + v + 1) : 0xfffffffeu;
        const bool head = key != prevkey;  // the previous vector has another destination
        const bool tail = key != nextkey;  // the next vector has another destination
        const unsigned real_heads = __ballot_sync(0xffffffffu, head);
        const unsigned seg_heads = real_heads | 1u;  // warp-local segments
        const int segstart = 31 - __clz(seg_heads & (0xffffffffu >> (31 - lane)));
        const int maxlen = __reduce_max_sync(0xffffffffu, (unsigned)(lane - segstart + 1));
        for (int off = 1; off < maxlen; off <<= 1) {
            const u128 o = u128_shfl_up(val, off);
            if (lane - off >= segstart) val = u128_add(val, o);
        }
        __syncwarp();
        if (live && (tail || lane == 31)) {
            const bool head_real = (real_heads >> segstart) & 1u;
            if (tail && head_real) {
                // every vector of this destination is in this warp
                rowacc_put(rowacc, key, val, false);
            } else {
                // open on the left (slot 0) or on the right only (slot 1): combined across the block below
                const int slot = (segstart == 0 && !head_real) ? 0 : 1;
                sm.key[slot][warp] = key;
                sm.sum[slot][warp] = val;
                sm.flag[slot][warp] = 1u | (head_real ? 2u : 0u) | (tail ? 4u : 0u);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // Walk the warps' open pieces in order.  A destination that starts and ends inside the
            // block is stored once.  Only destinations that cross the block edge (at most the first
            // and the last) are added to global memory atomically.
            bool open = false, open_head = false;
            uint32_t ok = 0;
            u128 os = u128_zero();
            for (int w = 0; w < NW; ++w) {
                const uint32_t f0 = sm.flag[0][w];
                if (f0 & 1u) {
                    if (!open) { open = true; open_head = false; ok = sm.key[0][w]; os = u128_zero(); }
                    os = u128_add(os, sm.sum[0][w]);
                    if (f0 & 4u) {
                        if (open_head) rowacc_put(rowacc, ok, os, false);
                        else if (os.lo | os.hi) u128_atomic_add(rowacc + ok, os);
                        open = false;
                    }
                }
                const uint32_t f1 = sm.flag[1][w];
                if (f1 & 1u) { open = true; open_head = (f1 & 2u) != 0; ok = sm.key[1][w]; os = sm.sum[1][w]; }
            }
            if (open && (os.lo | os.hi)) u128_atomic_add(rowacc + ok, os);
        }
        __syncthreads();  // the walk has read this tile's pieces
    }
}

// 8 resident blocks per SM asked of the compiler: 32 registers, the most gathers in flight (a
// 16-byte spill in the fixed-point form).  Unbounded, the compiler takes 80 registers (3 blocks
// per SM), which measured 47% slower at R-MAT 20.
constexpr int PR_GATHER_MIN_BLOCKS = 8;

template <typename P>
__global__ void __launch_bounds__(PR_THREADS, PR_GATHER_MIN_BLOCKS) k_pr_gather(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv,
                                                          uint64_t first, uint64_t nvec, uint64_t list_nvec,
                                                          const P* __restrict__ prop_fx, uint32_t V, u128* __restrict__ rowacc,
                                                          const uint32_t* __restrict__ hub_vid, uint32_t nhub, const PRConst pc)
{
    __shared__ GatherSmem sm;
    if (pc.K_out && blockIdx.x == 0) pr_publish_K(pc, sm.red);
    pr_gather_tiles<P, false>(nbr, dstv, first, nvec, list_nvec, prop_fx, V, rowacc, hub_vid, nhub, blockIdx.x, gridDim.x, sm);
}

// ---------------------------------------------------------------------------------------------
// The gather of grz_pr_iterate over packed props.
//
// A random gather costs an L1 tag lookup per line, one per SM clock, and a miss about 1.9 clocks of
// the SM's path to L2 (GB300: 160 G misses/s, at R-MAT 20 and on a uniform graph alike), whatever
// its width.  So what helps is fewer gathers through L1 and fewer instructions around them:
//   * HOT: the props of up to GRZ_PR_HOT_MAX sources of the highest out-degrees are copied into
//     shared memory when the block starts, and lanes that name one
//     (GRZ_HUB_BASE + slot in the encoded list) read them there.  The other gathers of a whole list then
//     hardly hit L1 (3% at R-MAT 20) and go past it (GB300, through L1 / past it: R-MAT of 2^21 vertices 88 /
//     84 us, 2^24 828 / 765; in segments 4449 / 4471 at 2^26, and without a table 146 / 286 on a uniform
//     graph: those stay).
//   * A thread owns four consecutive vectors (two 32-byte loads and one of four destinations, the
//     next group's issued before this one's sums): it joins vectors of one destination in registers,
//     so the u128 scan over the warp runs once per 128 vectors, not once per 32.
//   * A warp walks a contiguous range of `per` vectors and carries the open destination's sum from
//     group to group.  There is no barrier, and only the two destinations cut by the range's ends
//     are added atomically (the apply clears exactly those, marked in pr_cut).
// One block of 768 threads per SM: 80 registers hold a thread's 16 gathers without spills, and the
// table is copied once per SM.  GB300, gather per iteration (16-byte props, a thread per vector,
// 2048 threads per SM -> this kernel): R-MAT 20 83 -> 43 us, R-MAT 24 1550 -> 810 us, uniform graph of
// 3M vertices and 36M edges 200 -> 148 us.
constexpr int PK_THREADS = 768;
constexpr uint32_t PK_GROUP = 128;    // vectors a warp sums at a time
constexpr uint32_t PK_MIN_RANGE = 32; // fewest vectors per warp: a small list spreads over the SMs

struct PkVec8 {
    uint32_t a[8];  // two vectors' sources
};

// two consecutive vectors, read once (32-byte aligned)
__device__ __forceinline__ PkVec8 ld_vec8(const uint4* p)
{
    PkVec8 r;
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r.a[0]), "=r"(r.a[1]), "=r"(r.a[2]), "=r"(r.a[3]), "=r"(r.a[4]), "=r"(r.a[5]), "=r"(r.a[6]), "=r"(r.a[7])
                 : "l"(p));
    return r;
}

__device__ __forceinline__ u128 u128_shfl(u128 v, int src)
{
    u128 r;
    r.lo = __shfl_sync(0xffffffffu, v.lo, src);
    r.hi = __shfl_sync(0xffffffffu, v.hi, src);
    return r;
}

// Sums a warp's group of vectors by destination.  k, v0..v3: the destinations and sums of the lane's four
// consecutive vectors (GRZ_INVALID_ID past the range).  carry, ckey: the sum so far of the
// destination that the group before left open.  after: the destination after lane `last`'s vectors,
// the group's last ones.  put(destination, sum): a destination that ends in this group; open(...):
// one that goes on past the range, whose last group this is (`ends`).
template <typename Put, typename Open>
__device__ __forceinline__ void pk_group(uint4 k, u128 v0, u128 v1, u128 v2, u128 v3, uint32_t after, bool ends, int last, u128& carry,
                                         uint32_t& ckey, Put put, Open open)
{
    const int lane = threadIdx.x & 31;
    uint32_t kp = __shfl_up_sync(0xffffffffu, k.w, 1), kn = __shfl_down_sync(0xffffffffu, k.x, 1);
    if (lane == 0) kp = ckey;
    if (lane == last) kn = after;
    // the thread's vectors: the first destination's sum if it ends here (`head`), destinations that
    // start and end here (put at once), and the last destination's sum (`cur`)
    u128 cur = v0, head = u128_zero();
    bool closed = false;
    if (k.y == k.x) cur = u128_add(cur, v1);
    else { head = cur; closed = true; cur = v1; }
    if (k.z == k.y) cur = u128_add(cur, v2);
    else { if (closed) put(k.y, cur); else { head = cur; closed = true; } cur = v2; }
    if (k.w == k.z) cur = u128_add(cur, v3);
    else { if (closed) put(k.z, cur); else { head = cur; closed = true; } cur = v3; }
    if (lane == 0 && !closed && kp == k.x) cur = u128_add(cur, carry);
    // segmented inclusive scan of `cur` over the threads
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || closed || kp != k.x);
    const int segstart = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    const int maxlen = __reduce_max_sync(0xffffffffu, (unsigned)(lane - segstart + 1));
    for (int off = 1; off < maxlen; off <<= 1) {
        const u128 o = u128_shfl_up(cur, off);
        if (lane - off >= segstart) cur = u128_add(cur, o);
    }
    u128 before = u128_shfl_up(cur, 1);
    if (lane == 0) before = carry;
    if (closed) {
        if (kp == k.x) head = u128_add(head, before);
        put(k.x, head);
    }
    if (k.w != kn) put(k.w, cur);
    carry = u128_shfl(cur, 31);
    ckey = __shfl_sync(0xffffffffu, k.w, 31);
    if (ends && lane == last && k.w == kn && k.w != GRZ_INVALID_ID) open(k.w, cur);
}

// The vectors [first, end) of a list whose first vector is at a multiple of 16 bytes of `dstv`.
// `base` is `first` rounded down to a multiple of 4 (vectors before `first` count as empty), so that
// the wide loads are aligned; ranges are [base + w * per, base + (w + 1) * per), per a multiple of 4.
template <bool HOT, bool ADD>
__global__ void __launch_bounds__(PK_THREADS, 1) k_pr_gather_pk(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv,
                                                                uint32_t first, uint32_t end, uint32_t per,
                                                                const pk_t* props, uint32_t V, const pk_t* hot, uint32_t nhot,
                                                                u128* rowacc, const PRConst pc)
{
    extern __shared__ __align__(16) pk_t s_hot[];
    const int lane = threadIdx.x & 31;
    const uint32_t nwarps = gridDim.x * (PK_THREADS / 32);
    const uint32_t wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // neighbouring ranges on different SMs
    pdl_start();
    const uint32_t base = first & ~3u;
    const uint64_t lo64 = (uint64_t)base + (uint64_t)wid * per;
    const uint32_t lo = (uint32_t)(lo64 < end ? lo64 : end);
    const uint32_t hi = (uint32_t)(lo64 + per < end ? lo64 + per : end);
    PkVec8 na, nb;
    uint4 nk;
    const uint32_t pad = HOT ? (GRZ_HUB_BASE | nhot) : GRZ_INVALID_ID;
    auto load = [&](uint64_t v) {  // the lane's four vectors from v on
        if (v >= first && v + 3 < hi) {
            na = ld_vec8(nbr + v);
            nb = ld_vec8(nbr + v + 2);
            nk = __ldcs(reinterpret_cast<const uint4*>(dstv + v));
        } else {
            uint4 x[4];
            uint32_t k[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool in = v + j >= first && v + j < hi;
                x[j] = in ? __ldcs(nbr + v + j) : make_uint4(pad, pad, pad, pad);
                k[j] = in ? __ldcs(dstv + v + j) : GRZ_INVALID_ID;
            }
            na.a[0] = x[0].x; na.a[1] = x[0].y; na.a[2] = x[0].z; na.a[3] = x[0].w;
            na.a[4] = x[1].x; na.a[5] = x[1].y; na.a[6] = x[1].z; na.a[7] = x[1].w;
            nb.a[0] = x[2].x; nb.a[1] = x[2].y; nb.a[2] = x[2].z; nb.a[3] = x[2].w;
            nb.a[4] = x[3].x; nb.a[5] = x[3].y; nb.a[6] = x[3].z; nb.a[7] = x[3].w;
            nk = make_uint4(k[0], k[1], k[2], k[3]);
        }
    };
    uint32_t kbefore = GRZ_INVALID_ID - 1;  // destination of the vector before the range
    if (lo < hi) {
        load((uint64_t)lo + 4 * lane);
        if (lo > first) kbefore = __ldg(dstv + lo - 1);
    }
    pdl_wait();
    props = after_wait(props);
    hot = after_wait(hot);
    rowacc = after_wait(rowacc);
    if (HOT) {
        // 16 bytes per thread and step, all steps' loads in flight (the table ends in zeros)
        const uint32_t n16 = (nhot + 2) / 2;
#pragma unroll
        for (uint32_t j = 0; j < (GRZ_PR_HOT_MAX / 2 + PK_THREADS) / PK_THREADS; ++j) {
            const uint32_t i = j * PK_THREADS + threadIdx.x;
            if (i < n16) reinterpret_cast<ulonglong2*>(s_hot)[i] = __ldcg(reinterpret_cast<const ulonglong2*>(hot) + i);
        }
    }
    // the iteration's constant (pr_publish_K), by the warp of the last range, which is usually empty
    if (pc.K_out && wid == nwarps - 1) {
        u128 S = u128_zero();
        const u128* const part_in = after_wait(pc.part_in);
        for (uint32_t b = lane; b < pc.nparts; b += 32) S = u128_add(S, part_in[b]);
        for (int o = 16; o > 0; o >>= 1) S = u128_add(S, u128_shfl_down(S, o));
        if (lane == 0) *pc.K_out = __fma_rn((1.0 - fx_to_double(S)) / pc.nverts, pc.damping, pc.c);
    }
    if (HOT) __syncthreads();
    auto get = [&](uint32_t id) -> pk_t {
        if (HOT) {
            if ((int)id < 0) return s_hot[id & (GRZ_HUB_BASE - 1)];
            return ADD ? ld_l1(props + id) : __ldcg(props + id);
        }
        return ld_l1(props + min(id, V));  // entry V is zero
    };
    auto put = [&](uint32_t key, u128 v) {
        if (key == GRZ_INVALID_ID) return;
        if (key != kbefore) rowacc_put(rowacc, key, v, ADD);
        else u128_atomic_add(rowacc + key, v);  // cut by the start of the range
    };
    u128 carry = u128_zero();  // sum so far of the destination the previous group left open
    uint32_t ckey = GRZ_INVALID_ID - 1;
    for (uint64_t v = lo; v < hi; v += PK_GROUP) {  // warp-uniform
        const uint4 k = nk;
        u128 v0, v1, v2, v3;
        {
            pk_t p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) p[j] = get(na.a[j]);
            v0 = u128_add(u128_add(pk_to_fx(p[0]), pk_to_fx(p[1])), u128_add(pk_to_fx(p[2]), pk_to_fx(p[3])));
            v1 = u128_add(u128_add(pk_to_fx(p[4]), pk_to_fx(p[5])), u128_add(pk_to_fx(p[6]), pk_to_fx(p[7])));
#pragma unroll
            for (int j = 0; j < 8; ++j) p[j] = get(nb.a[j]);
            if (v + PK_GROUP < hi) {
                load(v + PK_GROUP + 4 * lane);
            } else {
                nk.x = hi < end ? __ldg(dstv + hi) : GRZ_INVALID_ID;  // the next range's first destination
            }
            v2 = u128_add(u128_add(pk_to_fx(p[0]), pk_to_fx(p[1])), u128_add(pk_to_fx(p[2]), pk_to_fx(p[3])));
            v3 = u128_add(u128_add(pk_to_fx(p[4]), pk_to_fx(p[5])), u128_add(pk_to_fx(p[6]), pk_to_fx(p[7])));
        }
        const uint32_t after = __shfl_sync(0xffffffffu, nk.x, 0);
        const bool ends = v + PK_GROUP >= hi;  // the range's last group: its last vectors may not fill the warp
        pk_group(k, v0, v1, v2, v3, after, ends, ends ? (int)((hi - (uint32_t)v + 3) / 4) - 1 : 31, carry, ckey, put,
                 [&](uint32_t key, u128 x) { u128_atomic_add(rowacc + key, x); });
    }
}

__device__ __forceinline__ u128 block_reduce_u128(u128 s, u128* red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = u128_add(s, u128_shfl_down(s, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    s = u128_zero();
    if (threadIdx.x < 32) {
        s = (threadIdx.x < PR_THREADS / 32) ? red[threadIdx.x] : u128_zero();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = u128_add(s, u128_shfl_down(s, o));
    }
    return s;
}

// Vertex phase fused with reading the accumulators (phase_vertex_pr.asm:75-134):
//   prop[v] = (acc[v]*d + G*d + (1-d)/V) / deg'[v],  G = (1 - S)/V
// computed as fma + multiply by the precomputed 1/deg'.  It writes the new props in fixed point,
// or packed when the next gather reads them packed (and then the hot sources' once more, into the
// table of the next gather), plus the reference-format doubles when asked, and accumulates S' = sum deg[v]*prop[v] exactly; S' is the next
// iteration's sum of accumulators.  Of the accumulators it clears only those the next gather
// adds to atomically (bit set in `cut`); the others are overwritten by the next gather's stores.
// The grid strides over the vertices, PR_APPLY_U vertices per thread at a time whose
// accumulators are loaded before anything is stored; one partial of S' per block.  GB300 sweep of
// vertices in flight per thread x blocks per SM: 8 x 3 (80 registers) 16.7 us at V = 2^20 and
// 2.08 ms at V = 2^27; 4 x 4 14.5 us; 2 x 6 14.5 us and 1.25 ms; 1 x 8 (31 registers) 14.5 us and
// 1.15 ms (5.2 TB/s of 44V bytes).  Occupancy hides the latency better than loads in flight.
#ifndef GRZ_PR_APPLY_U
#define GRZ_PR_APPLY_U 1
#endif
#ifndef GRZ_PR_APPLY_MINB
#define GRZ_PR_APPLY_MINB 8
#endif
constexpr int PR_APPLY_U = GRZ_PR_APPLY_U;
constexpr int PR_APPLY_RESIDENT = GRZ_PR_APPLY_MINB;  // blocks per SM that the launch bounds fit

// vertex v's packed prop also into its slot of the hot table, if it has one (slots ascend by vertex)
__device__ __forceinline__ void hot_put(const uint2* __restrict__ hotmap, pk_t* __restrict__ hot, uint64_t v, pk_t w)
{
    const uint2 m = __ldg(hotmap + (v >> 5));
    const uint32_t bit = (uint32_t)v & 31u;
    if ((m.x >> bit) & 1u) hot[m.y + __popc(m.x & ((1u << bit) - 1u))] = w;
}

// the apply over vertices block*PR_THREADS + tid, strided by nblocks*PR_THREADS, U vertices per
// thread loaded before any is stored; returns the block's partial of S' (valid in thread 0;
// every thread of the block must call it)
template <int U>
__device__ __forceinline__ u128 pr_apply_range(u128* rowacc, const uint32_t* __restrict__ cut, bool clear_all,
                                               const double* __restrict__ inv_deg, const uint32_t* __restrict__ degree, uint64_t V,
                                               double sK, double damping, u128* __restrict__ prop_fx, pk_t* __restrict__ prop_pk,
                                               double* __restrict__ prop_out, const uint2* __restrict__ hotmap, pk_t* __restrict__ hot,
                                               uint32_t block, uint32_t nblocks, u128* red)
{
    const uint64_t stride = (uint64_t)nblocks * PR_THREADS;
    u128 s = u128_zero();
    for (uint64_t base = (uint64_t)block * PR_THREADS + threadIdx.x; base < V; base += stride * U) {
        ulonglong2 a[U];
        uint32_t cw[U];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const uint64_t v = base + (uint64_t)j * stride;
            a[j] = make_ulonglong2(0ull, 0ull);
            cw[j] = 0;
            if (v < V) {
                a[j] = __ldcs(reinterpret_cast<const ulonglong2*>(rowacc) + v);
                cw[j] = clear_all ? 0u : __ldg(cut + (v >> 5));
            }
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const uint64_t v = base + (uint64_t)j * stride;
            if (v >= V) break;
            if ((a[j].x | a[j].y) && (clear_all || ((cw[j] >> (v & 31)) & 1u)))
                *(reinterpret_cast<ulonglong2*>(rowacc) + v) = make_ulonglong2(0ull, 0ull);
            u128 acc;
            acc.lo = a[j].x;
            acc.hi = a[j].y;
            const double p = __dmul_rn(__fma_rn(fx_to_double(acc), damping, sK), __ldg(inv_deg + v));
            u128 pf;
            if (prop_pk) {
                const pk_t w = pk_from_double(p);
                pf = pk_to_fx(w);
                __stcg(prop_pk + v, w);
                if (hotmap) hot_put(hotmap, hot, v, w);
            } else {
                pf = fx_from_double(p);
                __stcg(reinterpret_cast<ulonglong2*>(prop_fx) + v, make_ulonglong2(pf.lo, pf.hi));
            }
            if (prop_out) prop_out[v] = p;
            s = u128_add(s, u128_mul32(pf, __ldg(degree + v)));
        }
    }
    return block_reduce_u128(s, red);
}

__global__ void __launch_bounds__(PR_THREADS, PR_APPLY_RESIDENT) k_pr_apply(u128* rowacc, const uint32_t* __restrict__ cut,
                                                                            int clear_all, const double* __restrict__ inv_deg,
                                                                            const uint32_t* __restrict__ degree, uint64_t V,
                                                                            const double* Kp, u128* __restrict__ part_out,
                                                                            double damping, u128* __restrict__ prop_fx,
                                                                            pk_t* __restrict__ prop_pk, double* __restrict__ prop_out,
                                                                            const uint2* __restrict__ hotmap, pk_t* __restrict__ hot)
{
    __shared__ u128 red[PR_THREADS / 32];
    pdl_start();
    pdl_wait();
    const u128 s = pr_apply_range<PR_APPLY_U>(after_wait(rowacc), cut, clear_all != 0, inv_deg, degree, V, *after_wait(Kp), damping, prop_fx, prop_pk, prop_out, hotmap, hot, blockIdx.x,
                                  gridDim.x, red);
    if (threadIdx.x == 0) part_out[blockIdx.x] = s;  // summed by the next gather kernel's block 0
}

// ---------------------------------------------------------------------------------------------
// Persistent form: all iterations in one cooperative launch, gather and apply separated by a
// grid-wide barrier (the reference's pull phase -> threads_barrier -> perform_vertex_phase_pr,
// source/phase_vertex_pr.asm:190-285, barrier source/threads.asm:181-204).  Every wait of the
// barrier is bounded: past the deadline (%globaltimer) a block sets the error word and every
// block returns at its next barrier, so a launch always ends and the host reads the error.

struct PRBar {
    unsigned int count;     // arrivals at the current barrier
    unsigned int gen;       // barriers completed
    unsigned int err;       // 1: a wait ran out
    unsigned int where;     // the barrier (1-based) whose wait ran out
    unsigned long long gather_ns[64];  // per iteration, block 0's view: gather phase (the barrier included)
    unsigned long long apply_ns[64];   // apply phase
};

constexpr unsigned long long PR_BAR_SPIN_MAX = 1ull << 26;  // iteration bound of one wait (besides the deadline)

__device__ __forceinline__ unsigned long long pr_now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// true when every block arrived; false when a wait gave up (or another block's did).
// `withhold` leaves this block's arrival out (host-side fault injection for the tests).
__device__ __forceinline__ bool pr_grid_barrier(PRBar* bar, unsigned nblocks, unsigned long long limit_ns, unsigned idx, bool withhold)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        volatile unsigned int* vgen = &bar->gen;
        volatile unsigned int* verr = &bar->err;
        const unsigned int g0 = *vgen;
        __threadfence();
        if (*verr) {
            ok = 0;
        } else if (!withhold && atomicAdd(&bar->count, 1u) + 1u == nblocks) {
            bar->count = 0u;
            __threadfence();
            atomicAdd(&bar->gen, 1u);
        } else {
            const unsigned long long t0 = pr_now_ns();
            for (unsigned long long spin = 0; *vgen == g0; ++spin) {
                if (*verr) { ok = 0; break; }
                if (spin >= PR_BAR_SPIN_MAX || pr_now_ns() - t0 > limit_ns) {
                    if (atomicExch(&bar->err, 1u) == 0u) bar->where = idx;
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

struct PRPersist {
    const uint4* nbr;
    const uint32_t* dstv;
    uint64_t nvec;
    uint32_t V;
    const uint32_t* hub_vid;
    uint32_t nhub;
    u128* rowacc;
    const uint32_t* cut;
    const double* inv_deg;
    const uint32_t* degree;
    u128* fx[2];            // props, fixed point (ping-pong)
    pk_t* pk[2];            // props, packed (ping-pong; gathered in packed mode)
    int pkmode;
    int cur;                // which buffer holds the current props
    u128* sum[2];           // per-block partials of S (ping-pong)
    uint32_t nparts0;       // partials in sum[sum_cur] at the start
    int sum_cur;
    double* K;
    double damping, c, nverts;
    uint32_t iters;
    double* prop_out;       // reference-format doubles after the last iteration, or null
    PRBar* bar;
    unsigned long long limit_ns;
    int withhold_block;     // -1: none
    int time_phases;        // block 0 records the phase durations into bar
};

// registers bounded so that MINB blocks of 256 threads stay resident per SM (the gather wants as
// many random loads in flight as possible: 6 leaves the apply unspilled, 8 is the two-kernel
// gather's occupancy); the apply loads 2 vertices per thread ahead
constexpr int PR_PERSIST_APPLY_U = 2;

template <typename P, int MINB>
__global__ void __launch_bounds__(PR_THREADS, MINB) k_pr_persistent(const PRPersist q)
{
    __shared__ GatherSmem sm;
    const unsigned nb = gridDim.x;
    unsigned bi = 0;
    int cur = q.cur, sc = q.sum_cur;
    uint32_t nparts = q.nparts0;
    for (uint32_t it = 0; it < q.iters; ++it) {
        const unsigned long long t0 = (q.time_phases && blockIdx.x == 0 && threadIdx.x == 0) ? pr_now_ns() : 0ull;
        if (blockIdx.x == 0) {
            PRConst pc;
            pc.part_in = q.sum[sc];
            pc.nparts = nparts;
            pc.K_out = q.K;
            pc.damping = q.damping;
            pc.c = q.c;
            pc.nverts = q.nverts;
            pr_publish_K(pc, sm.red);
        }
        const P* props = q.pkmode ? (const P*)q.pk[cur] : (const P*)q.fx[cur];
        pr_gather_tiles<P, true>(q.nbr, q.dstv, 0, q.nvec, q.nvec, props, q.V, q.rowacc, q.hub_vid, q.nhub, blockIdx.x, nb, sm);
        if (!pr_grid_barrier(q.bar, nb, q.limit_ns, ++bi, (int)blockIdx.x == q.withhold_block)) return;
        const unsigned long long t1 = (q.time_phases && blockIdx.x == 0 && threadIdx.x == 0) ? pr_now_ns() : 0ull;
        const double sK = *(volatile double*)q.K;
        const u128 s = pr_apply_range<PR_PERSIST_APPLY_U>(q.rowacc, q.cut, false, q.inv_deg, q.degree, q.V, sK, q.damping, q.fx[cur ^ 1],
                                      q.pkmode ? q.pk[cur ^ 1] : nullptr, it + 1 == q.iters ? q.prop_out : nullptr, nullptr, nullptr,
                                      blockIdx.x, nb, sm.red);
        if (threadIdx.x == 0) q.sum[sc ^ 1][blockIdx.x] = s;
        if (!pr_grid_barrier(q.bar, nb, q.limit_ns, ++bi, false)) return;
        if (q.time_phases && blockIdx.x == 0 && threadIdx.x == 0 && it < 64) {
            const unsigned long long t2 = pr_now_ns();
            q.bar->gather_ns[it] = t1 - t0;
            q.bar->apply_ns[it] = t2 - t1;
        }
        cur ^= 1;
        sc ^= 1;
        nparts = nb;
    }
}

// ---------------------------------------------------------------------------------------------
// All iterations of a small graph in one launch.
//
// Two kernels per iteration cost about 10 us in starts however small the graph.  Here one cluster of 16
// blocks runs every iteration.  Each block owns a range of vertices (an even share of vectors and
// vertices) with their vectors, and holds a copy of all packed props in shared memory, so a gather is
// a shared-memory read.  It sums its vectors as k_pr_gather_pk does, a contiguous range per warp; the
// destinations cut by the ranges are pieced together by the thread that owns the vertex, which knows
// the pieces from the start (no atomics: a 64-bit one on shared memory is a loop).  It writes its
// vertices' new props and its part of the next S to memory; one cluster barrier ends the iteration,
// and every block copies all new props, which is 1900 clocks for 32 KB.  (Writing them into the other
// blocks' shared memory instead took 4800: it moves 7 bytes per clock.)  Sums and formulas are those
// of the two kernels, bit for bit.  A block's vectors past PS_CAP, when a few destinations hold most of
// the list, are read from memory each time.  The bounds (PS_MAX_V, PS_MAX_VEC) lie where the two kernels
// overtake it.  GB300, us per iteration (16 in a launch), two kernels / this: 1000 vertices and 20k edges
// 6.2 / 4.6, R-MAT of 4096 and 53k 7.3 / 5.3, of 4096 and 65k 7.2 / 6.9, uniform 6000 and 72k 6.9 / 5.9;
// past the bounds, uniform 8192 and 49k 5.8 / 6.0, R-MAT of 8192 and 111k 6.5 / 7.8, 12000 and 48k 5.9 / 6.8.
constexpr int PS_CTAS = 16;
constexpr int PS_T = 512;
constexpr int PS_WARPS = PS_T / 32;
constexpr uint32_t PS_MAX_V = 6144;
constexpr uint32_t PS_MAX_VEC = 24576;
constexpr uint32_t PS_CAP = PS_MAX_VEC / 8;  // vectors a block keeps in shared memory: twice an even share
// a block's vertices: at most twice an even share, PS_OWN per thread
constexpr uint32_t PS_ACC = PS_MAX_V / 8 + 32;
constexpr int PS_OWN = (PS_ACC + PS_T - 1) / PS_T;

struct PRSmall {
    const uint4* nbr;
    const uint32_t* dstv;
    const uint32_t* rowptr;
    uint32_t V, nvec;
    const double* inv_deg;
    const uint32_t* degree;
    pk_t* props0;            // in; after an even number of iterations, out (entry V is zero)
    pk_t* props1;            // after an odd number
    const u128* part_in;     // partials of S
    uint32_t nparts;
    u128* parts;             // [2][PS_CTAS]: each block's part of S, by iteration parity
    u128* part_out;          // the last S
    double damping, c, nverts;
    uint32_t iters;
};

constexpr size_t ps_smem(uint32_t V)
{
    return sizeof(u128) * PS_ACC + sizeof(pk_t) * ((V + 2) & ~1u) + (sizeof(ushort4) + sizeof(uint16_t)) * PS_CAP;
}

__global__ void __cluster_dims__(PS_CTAS, 1, 1) __launch_bounds__(PS_T, 1) k_pr_small(const PRSmall q)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ u128 s_red[PS_WARPS], s_piece[2 * PS_WARPS];
    __shared__ uint32_t s_v[2], s_cut[2 * PS_WARPS];
    __shared__ double s_K;
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = cl.block_rank(), V = q.V;
    u128* const s_acc = reinterpret_cast<u128*>(s_raw);
    pk_t* const s_prop = reinterpret_cast<pk_t*>(s_raw + sizeof(u128) * PS_ACC);
    ushort4* const s_vec = reinterpret_cast<ushort4*>(s_prop + ((V + 2) & ~1u));
    uint16_t* const s_dst = reinterpret_cast<uint16_t*>(s_vec + PS_CAP);
    // This block's vertices: those whose weight, rowptr[v] * V + v * nvec, lies in its share.  All vectors
    // together weigh as much as all vertices, so a block has at most twice an even share of either
    // (and the vectors of its last destination).  The first vertex at or past each end, by all threads.
    const uint64_t total = 2ull * q.nvec * V;
    if (tid < 2) s_v[tid] = V;
    __syncthreads();
    for (uint32_t v = tid; v < V; v += PS_T) {
        const uint64_t w = (uint64_t)__ldg(q.rowptr + v) * V + (uint64_t)v * q.nvec;
        const uint64_t before = v ? (uint64_t)__ldg(q.rowptr + v - 1) * V + (uint64_t)(v - 1) * q.nvec : 0;
#pragma unroll
        for (uint32_t e = 0; e < 2; ++e) {
            const uint64_t want = total * (rank + e) / PS_CTAS;
            if (rank + e < PS_CTAS && w >= want && (v == 0 || before < want)) s_v[e] = v;
        }
        s_prop[v] = q.props0[v];
    }
    if (tid == 0) s_prop[V] = 0ull;  // empty lanes gather it
    for (uint32_t i = tid; i < PS_ACC; i += PS_T) s_acc[i] = u128_zero();
    if (tid < 2 * PS_WARPS) s_cut[tid] = GRZ_INVALID_ID;
    __syncthreads();
    const uint32_t v0 = s_v[0], nv = s_v[1] - v0;
    const uint32_t r0 = __ldg(q.rowptr + v0), m = __ldg(q.rowptr + v0 + nv) - r0;
    auto vec_of = [&](uint32_t i) -> ushort4 {
        const uint4 x = __ldg(q.nbr + r0 + i);
        return make_ushort4((unsigned short)min(x.x, V), (unsigned short)min(x.y, V), (unsigned short)min(x.z, V), (unsigned short)min(x.w, V));
    };
    for (uint32_t i = tid; i < min(m, PS_CAP); i += PS_T) {
        s_vec[i] = vec_of(i);
        s_dst[i] = (uint16_t)(__ldg(q.dstv + r0 + i) - v0);
    }
    // S of the first iteration, summed by every warp
    u128 S = u128_zero();
    for (uint32_t b = lane; b < q.nparts; b += 32) S = u128_add(S, q.part_in[b]);
    for (int o = 16; o > 0; o >>= 1) S = u128_add(S, u128_shfl_down(S, o));
    S = u128_shfl(S, 0);
    __syncthreads();
    auto dst_of = [&](uint32_t i) -> uint32_t { return i < PS_CAP ? s_dst[i] : __ldg(q.dstv + r0 + i) - v0; };
    const uint32_t per = ((m + PS_WARPS - 1) / PS_WARPS + 3) & ~3u;
    const uint32_t lo = min(m, warp * per), hi = min(m, lo + per);
    // the destinations cut by the start and the end of the warp's range: their pieces are s_piece[warp]
    // and s_piece[PS_WARPS + warp] (one that fills the whole range is a piece at the end)
    const uint32_t kbefore = lo > 0 && lo < hi ? dst_of(lo - 1) : GRZ_INVALID_ID - 1;
    const uint32_t after = lo < hi && hi < m ? dst_of(hi) : GRZ_INVALID_ID;
    if (lane == 0 && lo < hi) {
        const uint32_t first = dst_of(lo), last = dst_of(hi - 1);
        if (last == after) s_cut[PS_WARPS + warp] = last;
        if (first == kbefore && !(first == last && last == after)) s_cut[warp] = first;
    }
    __syncthreads();
    // of each vertex this thread owns: its pieces, 1/deg' and degree (a cluster barrier empties L1)
    uint32_t pieces[PS_OWN], deg[PS_OWN];
    double inv[PS_OWN];
#pragma unroll
    for (int j = 0; j < PS_OWN; ++j) {
        const uint32_t i = tid + j * PS_T;
        inv[j] = i < nv ? __ldg(q.inv_deg + v0 + i) : 0.0;
        deg[j] = i < nv ? __ldg(q.degree + v0 + i) : 0u;
        pieces[j] = 0;
        for (int k = 0; k < 2 * PS_WARPS; ++k)
            if (s_cut[k] == (uint32_t)(tid + j * PS_T)) pieces[j] |= 1u << k;
    }
    for (uint32_t it = 0; it < q.iters; ++it) {
        // one thread: 512 FP64 divisions would take 3500 clocks of the SM's two FP64 lanes
        if (tid == PS_T - 1) s_K = __fma_rn((1.0 - fx_to_double(S)) / q.nverts, q.damping, q.c);
        u128 carry = u128_zero();
        uint32_t ckey = GRZ_INVALID_ID - 1;
        for (uint32_t v = lo; v < hi; v += PK_GROUP) {  // warp-uniform
            uint32_t k[4];
            u128 x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t i = v + 4 * lane + j;
                k[j] = GRZ_INVALID_ID;
                x[j] = u128_zero();
                if (i < hi) {
                    k[j] = dst_of(i);
                    const ushort4 s = i < PS_CAP ? s_vec[i] : vec_of(i);
                    x[j] = u128_add(u128_add(pk_to_fx(s_prop[s.x]), pk_to_fx(s_prop[s.y])), u128_add(pk_to_fx(s_prop[s.z]), pk_to_fx(s_prop[s.w])));
                }
            }
            const bool ends = v + PK_GROUP >= hi;
            pk_group(
                make_uint4(k[0], k[1], k[2], k[3]), x[0], x[1], x[2], x[3], ends ? after : dst_of(v + PK_GROUP), ends,
                ends ? (int)((hi - v + 3) / 4) - 1 : 31, carry, ckey,
                [&](uint32_t key, u128 y) {
                    if (key == GRZ_INVALID_ID) return;
                    if (key != kbefore) s_acc[key] = y;
                    else s_piece[warp] = y;
                },
                [&](uint32_t, u128 y) { s_piece[PS_WARPS + warp] = y; });
        }
        __syncthreads();
        const double K = s_K;
        pk_t* const out = it & 1 ? q.props0 : q.props1;
        u128 s = u128_zero();
#pragma unroll
        for (int j = 0; j < PS_OWN; ++j) {
            const uint32_t i = tid + j * PS_T;
            if (i < nv) {
                u128 a = s_acc[i];
                for (uint32_t k = pieces[j]; k; k &= k - 1) a = u128_add(a, s_piece[__ffs(k) - 1]);
                const double p = __dmul_rn(__fma_rn(fx_to_double(a), q.damping, K), inv[j]);
                const pk_t w = pk_from_double(p);
                __stcg(out + v0 + i, w);
                s = u128_add(s, u128_mul32(pk_to_fx(w), deg[j]));
            }
        }
        for (int o = 16; o > 0; o >>= 1) s = u128_add(s, u128_shfl_down(s, o));
        if (lane == 0) s_red[warp] = s;
        __syncthreads();
        u128* const parts = q.parts + (it & 1) * PS_CTAS;
        if (warp == 0) {
            s = lane < PS_WARPS ? s_red[lane] : u128_zero();
            for (int o = 8; o > 0; o >>= 1) s = u128_add(s, u128_shfl_down(s, o));
            if (lane == 0) __stcg(reinterpret_cast<ulonglong2*>(parts + rank), make_ulonglong2(s.lo, s.hi));
        }
        cl.sync();
        // all new props (this block's gathers of the old ones are done) and S
        for (uint32_t v = 2 * tid; v < V; v += 2 * PS_T)  // (entry V is zero)
            *reinterpret_cast<ulonglong2*>(s_prop + v) = __ldcg(reinterpret_cast<const ulonglong2*>(out + v));
        S = u128_zero();
        if (lane < PS_CTAS) {
            const ulonglong2 x = __ldcg(reinterpret_cast<const ulonglong2*>(parts + lane));
            S.lo = x.x;
            S.hi = x.y;
        }
        for (int o = 8; o > 0; o >>= 1) S = u128_add(S, u128_shfl_down(S, o));
        S = u128_shfl(S, 0);
        __syncthreads();
    }
    if (tid == 0 && rank == 0) *q.part_out = S;
}

// bit j of word t: vertex 32t + j has pull vectors in two or more of the gather's ranges of `per`
// vectors (its accumulator is summed with atomics)
__global__ void k_pr_cutbits(const uint32_t* __restrict__ rowptr, uint64_t V, uint32_t per, uint32_t* __restrict__ cut)
{
    const uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool c = false;
    if (v < V) {
        const uint32_t r0 = rowptr[v], r1 = rowptr[v + 1];
        c = r1 > r0 && r0 / per != (r1 - 1) / per;
    }
    const unsigned m = __ballot_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && v < V) cut[v >> 5] = m;
}

// ---------------------------------------------------------------------------------------------
// Source-segmented pull lists.  A destination's in-edges are its vectors' lanes in order, sorted
// by source (the -pull order), so the edges from source segment s form one run of lanes
// [a_s, b_s).  Segment s's list has ceil((b_s - a_s) / 4) vectors per destination, grouped by
// destination in ascending order; the segment lists are concatenated in segment order.
//
// Both passes over the list run a thread per vector, so a hub's lanes are spread over the grid and
// every read is coalesced (GB300, R-MAT 26 in 4 segments, against a thread per destination that
// searched its lanes for each segment's run: 20.9 -> 9.3 ms of device time, hot
// encoding included).

// a code of the gathered list: the slot of a hot source, the zero slot of an empty lane, else the ID
__device__ __forceinline__ uint32_t hot_code(uint32_t id, const uint2* __restrict__ hotmap, uint32_t nhot)
{
    if (id == GRZ_INVALID_ID) return GRZ_HUB_BASE | nhot;
    const uint2 m = __ldg(hotmap + (id >> 5));
    const uint32_t bit = id & 31u;
    return (m.x >> bit) & 1u ? GRZ_HUB_BASE | (m.y + __popc(m.x & ((1u << bit) - 1u))) : id;
}

// the source after vector v's lanes in its destination's order, or GRZ_INVALID_ID if v is its last
__device__ __forceinline__ uint32_t seg_next_src(const uint4* __restrict__ nbr, uint32_t v, uint32_t r1)
{
    return v + 1 < r1 ? __ldg(&nbr[v + 1].x) : GRZ_INVALID_ID;
}

// start and end lane of the run of every (segment, destination) pair: [s * (V + 1) + d], both 0 for
// a pair without edges
__global__ void __launch_bounds__(PR_THREADS) k_seg_bounds(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv,
                                                           const uint32_t* __restrict__ rowptr, uint64_t nvec, uint64_t V, uint32_t bits,
                                                           uint32_t* __restrict__ start, uint32_t* __restrict__ end)
{
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (v >= nvec) return;
    const uint32_t d = __ldg(dstv + v), r0 = __ldg(rowptr + d), r1 = __ldg(rowptr + d + 1);
    const uint4 x = __ldg(nbr + v);
    const uint32_t id[5] = { x.x, x.y, x.z, x.w, seg_next_src(nbr, (uint32_t)v, r1) };
    const uint32_t pos = 4 * ((uint32_t)v - r0);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (id[l] == GRZ_INVALID_ID) break;
        const uint32_t sg = id[l] >> bits;
        if (id[l + 1] != GRZ_INVALID_ID && id[l + 1] >> bits == sg) continue;
        end[(uint64_t)sg * (V + 1) + d] = pos + l + 1;
        if (id[l + 1] != GRZ_INVALID_ID) start[(uint64_t)(id[l + 1] >> bits) * (V + 1) + d] = pos + l + 1;
    }
}

// vectors of every pair, in place of its end
__global__ void __launch_bounds__(PR_THREADS) k_seg_sizes(const uint32_t* __restrict__ start, uint32_t* __restrict__ end, uint64_t n)
{
    for (uint64_t i = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x; i < n; i += (uint64_t)gridDim.x * PR_THREADS)
        end[i] = (end[i] - start[i] + 3) / 4;
}

// every lane to its place: the lane of rank r in its run goes to lane r % 4 of vector r / 4 of the
// pair, whose vectors start at seg_first[s] + off[s][d]; the run's last lane also fills the vector
struct SegFirst {
    uint64_t at[GRZ_PR_MAX_SEGMENTS + 1];
};
__global__ void __launch_bounds__(PR_THREADS) k_seg_emit(const uint4* __restrict__ nbr, const uint32_t* __restrict__ dstv,
                                                         const uint32_t* __restrict__ rowptr, uint64_t nvec, uint64_t V, uint32_t bits,
                                                         const uint32_t* __restrict__ start, const uint32_t* __restrict__ off,
                                                         const __grid_constant__ SegFirst first, const uint2* __restrict__ hotmap, uint32_t nhot,
                                                         uint32_t* __restrict__ out_nbr, uint32_t* __restrict__ out_dst)
{
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (v >= nvec) return;
    const uint32_t d = __ldg(dstv + v), r0 = __ldg(rowptr + d), r1 = __ldg(rowptr + d + 1);
    const uint4 x = __ldg(nbr + v);
    const uint32_t id[5] = { x.x, x.y, x.z, x.w, seg_next_src(nbr, (uint32_t)v, r1) };
    const uint32_t pos = 4 * ((uint32_t)v - r0);
    const uint32_t pad = hotmap ? GRZ_HUB_BASE | nhot : GRZ_INVALID_ID;
    uint32_t sg = 0xffffffffu, a = 0;
    uint64_t o = 0;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (id[l] == GRZ_INVALID_ID) break;
        if (id[l] >> bits != sg) {
            sg = id[l] >> bits;
            a = __ldg(start + (uint64_t)sg * (V + 1) + d);
            o = first.at[sg] + __ldg(off + (uint64_t)sg * (V + 1) + d);
        }
        const uint32_t r = pos + l - a;
        const uint64_t at = 4 * o + r;
        out_nbr[at] = hotmap ? hot_code(id[l], hotmap, nhot) : id[l];
        if ((r & 3u) == 0) out_dst[at >> 2] = d;
        if (id[l + 1] == GRZ_INVALID_ID || id[l + 1] >> bits != sg)
            for (uint64_t q = at + 1; q & 3u; ++q) out_nbr[q] = pad;
    }
}

// Edge-pull phase alone (the phases.h boundary): accumulators as doubles plus their exact sum
// into the global accumulator; clears rowacc.
__global__ void __launch_bounds__(PR_THREADS) k_pr_accum_out(u128* __restrict__ rowacc, uint64_t V, double* __restrict__ accum,
                                                             u128* __restrict__ glob)
{
    __shared__ u128 red[PR_THREADS / 32];
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    u128 s = u128_zero();
    if (v < V) {
        s = rowacc[v];
        rowacc[v] = u128_zero();
        accum[v] = fx_to_double(s);
    }
    s = block_reduce_u128(s, red);
    if (threadIdx.x == 0) u128_slot_add(glob, s);
}

// perform_vertex_phase_pr over [first, first+count): double accumulators -> props (double and fixed)
__global__ void k_pr_vertex(const double* __restrict__ accum, const double* __restrict__ inv_deg,
                            double* __restrict__ prop, u128* __restrict__ prop_fx, uint64_t first, uint64_t count,
                            double damping, double K)
{
    const uint64_t i = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (i >= count) return;
    const uint64_t v = first + i;
    const double p = __dmul_rn(__fma_rn(accum[v], damping, K), inv_deg[v]);
    prop[v] = p;
    prop_fx[v] = fx_from_double(p);
}

// execution_initialize_vertex_prop_pr (source/execution_pr.c:85-88): c / deg' with c = 1/V, in the
// form the first gather reads (packed with the hot table, or fixed point).  The division is one
// Newton step on the reciprocal 1/deg' (Markstein 1990): q0 = c * inv, r = c - q0 * deg' exactly by
// one fma, q = q0 + r * inv.  That is the division's result for every degree below 2^32: r is a multiple
// of ulp(q0) below 2^34 of them, so it is exact; q0 + r * inv before its one rounding is within 2^-51 ulp of
// the quotient; and the quotient of a 53-bit significand by a 32-bit integer is a number of 53 bits or at
// least 2^-33 ulp from every rounding boundary.  3 FP64 operations instead of a division's; the grid strides, with one partial of S_0 per block.  GB300, with
// the accumulators' clearing (a division per vertex, props also written as doubles and in fixed point
// -> now): V = 2^24 512 -> 171 us, 2^20 52 -> 24 us.
__global__ void __launch_bounds__(PR_THREADS, 8) k_pr_init(const double* __restrict__ inv_deg, const uint32_t* __restrict__ degree, uint64_t V,
                                                           double c, double* __restrict__ accum, u128* __restrict__ prop_fx, pk_t* __restrict__ prop_pk,
                                                           const uint2* __restrict__ hotmap, pk_t* __restrict__ hot, u128* __restrict__ part0)
{
    __shared__ u128 red[PR_THREADS / 32];
    u128 s = u128_zero();
    for (uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x; v < V; v += (uint64_t)gridDim.x * PR_THREADS) {
        const uint32_t deg = __ldg(degree + v);
        const double inv = __ldg(inv_deg + v), d = deg ? (double)deg : (double)V;
        const double q0 = __dmul_rn(c, inv);
        const double p = __fma_rn(__fma_rn(-q0, d, c), inv, q0);
        u128 pf;
        if (prop_pk) {
            const pk_t w = pk_from_double(p);
            pf = pk_to_fx(w);
            prop_pk[v] = w;
            if (hotmap) hot_put(hotmap, hot, v, w);
        } else {
            pf = fx_from_double(p);
            prop_fx[v] = pf;
        }
        accum[v] = 0.0;
        s = u128_add(s, u128_mul32(pf, deg));
    }
    if (blockIdx.x == 0 && threadIdx.x < 8) accum[V + threadIdx.x] = 0.0;
    s = block_reduce_u128(s, red);
    if (threadIdx.x == 0) part0[blockIdx.x] = s;
}

__global__ void k_fx_to_double(const u128* __restrict__ fx, uint64_t V, double* __restrict__ out)
{
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (v < V) out[v] = fx_to_double(fx[v]);
}

// packed props -> fixed point, or the doubles they are
__global__ void k_pk_unpack(const pk_t* __restrict__ pk, uint64_t V, u128* __restrict__ fx, double* __restrict__ out)
{
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (v >= V) return;
    const u128 f = pk_to_fx(pk[v]);
    if (fx) fx[v] = f;
    if (out) out[v] = fx_to_double(f);
}

// fixed-point props (each the conversion of a double) -> packed, and the hot table
__global__ void k_pk_pack(const u128* __restrict__ fx, uint64_t V, pk_t* __restrict__ pk, const uint2* __restrict__ hotmap,
                          pk_t* __restrict__ hot)
{
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (v >= V) return;
    const pk_t w = pk_from_double(fx_to_double(fx[v]));
    pk[v] = w;
    if (hotmap) hot_put(hotmap, hot, v, w);
}

// ---------------------------------------------------------------------------------------------
// Hot sources: the vertices of the highest out-degrees, at most GRZ_PR_HOT_MAX of them, cut where a
// degree bin ends (32 bins per octave above 64, exact below).

constexpr uint32_t HOT_BINS = 64 + 26 * 32;

__device__ __forceinline__ uint32_t hot_bin(uint32_t d)
{
    if (d < 64u) return d;
    const uint32_t e = 31u - (uint32_t)__clz(d);
    return 64u + (e - 6u) * 32u + ((d >> (e - 5u)) & 31u);
}

// vertices and out-edges per bin, of the vertices with out-degree `dmin` or more
__global__ void __launch_bounds__(PR_THREADS) k_hot_hist(const uint32_t* __restrict__ degree, uint64_t V, uint32_t dmin,
                                                         unsigned long long* __restrict__ hist)
{
    __shared__ uint32_t cnt[HOT_BINS];
    __shared__ unsigned long long edges[HOT_BINS];
    for (uint32_t b = threadIdx.x; b < HOT_BINS; b += PR_THREADS) { cnt[b] = 0; edges[b] = 0; }
    __syncthreads();
    for (uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x; v < V; v += (uint64_t)gridDim.x * PR_THREADS) {
        const uint32_t d = __ldg(degree + v);
        if (d < dmin) continue;
        const uint32_t b = hot_bin(d);
        atomicAdd(cnt + b, 1u);
        atomicAdd(edges + b, (unsigned long long)d);
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < HOT_BINS; b += PR_THREADS)
        if (cnt[b]) {
            atomicAdd(hist + b, (unsigned long long)cnt[b]);
            atomicAdd(hist + HOT_BINS + b, edges[b]);
        }
}

// out[0] = the lowest bin whose vertices and all above are at most `cap`, out[1] = how many they
// are, out[2] = their out-edges.  One block, thread t has the t-th bin from the top.
constexpr int HOT_PICK_T = (HOT_BINS + 31) / 32 * 32;

__global__ void __launch_bounds__(HOT_PICK_T) k_hot_pick(const unsigned long long* __restrict__ hist, uint32_t cap,
                                                         unsigned long long* __restrict__ out)
{
    __shared__ unsigned long long sn[HOT_PICK_T / 32], se[HOT_PICK_T / 32];
    const int t = threadIdx.x, lane = t & 31;
    unsigned long long n = t < (int)HOT_BINS ? hist[HOT_BINS - 1 - t] : 0ull;
    unsigned long long e = t < (int)HOT_BINS ? hist[2 * HOT_BINS - 1 - t] : 0ull;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long yn = __shfl_up_sync(0xffffffffu, n, o), ye = __shfl_up_sync(0xffffffffu, e, o);
        if (lane >= o) { n += yn; e += ye; }
    }
    if (lane == 31) { sn[t >> 5] = n; se[t >> 5] = e; }
    __syncthreads();
    for (int w = 0; w < t >> 5; ++w) { n += sn[w]; e += se[w]; }
    // the running counts ascend, so the bins within the cap are the first `fit`
    const int fit = __syncthreads_count(t < (int)HOT_BINS && n <= cap);
    if (t == 0) { out[0] = HOT_BINS - (uint32_t)fit; }
    if (fit == 0 && t == 0) { out[1] = 0; out[2] = 0; }
    if (t == fit - 1) { out[1] = n; out[2] = e; }
}

// the hot bits of 32 vertices per warp, and how many there are (words: (V + 31) / 32)
__global__ void __launch_bounds__(PR_THREADS) k_hot_mark(const uint32_t* __restrict__ degree, uint64_t V, uint32_t dmin, uint32_t bin,
                                                         uint2* __restrict__ hotmap, uint32_t* __restrict__ count)
{
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    const uint32_t d = v < V ? __ldg(degree + v) : 0u;
    const unsigned m = __ballot_sync(0xffffffffu, d >= dmin && hot_bin(d) >= bin);
    if ((threadIdx.x & 31) == 0 && v < V) {
        hotmap[v >> 5].x = m;
        count[v >> 5] = __popc(m);
    }
}

// the slot of each word's first hot vertex, and the vertex of each slot
__global__ void k_hot_base(const uint32_t* __restrict__ base, uint64_t words, uint2* __restrict__ hotmap, uint32_t* __restrict__ vid)
{
    const uint64_t w = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (w >= words) return;
    uint32_t b = base[w];
    hotmap[w].y = b;
    for (uint32_t m = hotmap[w].x; m; m &= m - 1) vid[b++] = (uint32_t)(32 * w) + (uint32_t)(__ffs(m) - 1);
}

// the list with its hot sources as GRZ_HUB_BASE + slot and its empty lanes as the slot after the
// last, which is zero
__global__ void __launch_bounds__(PR_THREADS) k_hot_encode(const uint4* __restrict__ nbr, uint64_t nvec, const uint2* __restrict__ hotmap,
                                                           uint32_t nhot, uint4* __restrict__ out)
{
    const uint64_t v = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (v >= nvec) return;
    const uint4 s = __ldcs(nbr + v);
    __stcs(out + v, make_uint4(hot_code(s.x, hotmap, nhot), hot_code(s.y, hotmap, nhot), hot_code(s.z, hotmap, nhot), hot_code(s.w, hotmap, nhot)));
}

unsigned blocks_for(uint64_t n) { return (unsigned)((n + PR_THREADS - 1) / PR_THREADS); }

}  // namespace

// The current props live in pr_fx[pr_cur] (fixed point) or, after fused iterations that gather
// packed props, in pr_pk[pr_cur]; each form is brought up to date from the other before a path that
// reads it.
static int pr_sync_fx(grz_graph* g)
{
    if (!g->pr_fx_stale) return GRZ_OK;
    k_pk_unpack<<<blocks_for(g->V), PR_THREADS, 0, g->stream>>>(g->pr_pk[g->pr_cur], g->V, g->pr_fx[g->pr_cur], nullptr); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    g->pr_fx_stale = 0;
    return GRZ_OK;
}

// whether the packed gather takes hot sources from the table: some were chosen, and the list it reads names them
static bool pr_hot_on(const grz_graph* g) { return g->pr_nhot && (g->pr_segmode || g->pr_hot_nbr); }

static int pr_sync_pk(grz_graph* g)
{
    if (!g->pr_pk_stale) return GRZ_OK;
    k_pk_pack<<<blocks_for(g->V), PR_THREADS, 0, g->stream>>>(g->pr_fx[g->pr_cur], g->V, g->pr_pk[g->pr_cur],
                                                             pr_hot_on(g) ? g->pr_hotmap : nullptr, g->pr_hot[g->pr_cur]); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    g->pr_pk_stale = 0;
    return GRZ_OK;
}

// The phase-API gathers and the push phase add into every accumulator: after fused iterations,
// which leave the accumulators of non-straddling destinations holding their last sums, clear all.
int grz_pr_rowacc_clean(grz_graph* g)
{
    if (g->pr_rowacc && g->pr_rowacc_stale) {
        GRZ_CK(g, cudaMemsetAsync(g->pr_rowacc, 0, sizeof(u128) * (g->V + 1), g->stream));
        g->pr_rowacc_stale = 0;
    }
    return GRZ_OK;
}

// Marks the destinations cut by the gather's ranges of `per` vectors.  When the ranges change, the
// accumulators that the old marks left uncleared are cleared.
static int pr_cut_for(grz_graph* g, uint32_t per)
{
    if (g->pr_cut_vec == per || !g->V) return GRZ_OK;
    GRZ_TRY(grz_pr_rowacc_clean(g));
    k_pr_cutbits<<<blocks_for(g->V), PR_THREADS, 0, g->stream>>>(g->pull.rowptr, g->V, per, g->pr_cut); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    g->pr_cut_vec = per;
    return GRZ_OK;
}

// Chooses the hot sources of the loaded lists.  Once per loaded lists; one read-back.  Worth it
// when the hot sources are at least a tenth of the edges.  GB300, us per iteration without / with the table,
// uniform graphs with that share of the edges moved to 20000 sources: 3M vertices, degree 12, 5% 167 / 166, 10%
// 167 / 160, 30% 166 / 138; 2^20, degree 16, 5% 77.3 / 78.5, 10% 77.2 / 76.3; 2^22, degree 16, 2% 289 / 291, 10%
// 289 / 274; R-MAT of 2^20 67.4 / 51.8.  (Only a thin rest of 8M to 12M vertices is better without: 10M, degree 8, 10%
// 472 / 567.)  Lists below 2^21 vectors stay as they are: R-MAT of 0.5M vectors 13.7 / 14.8, 1.0M 19.2 / 18.8, 2.0M
// 27.6 / 24.1, and choosing and encoding take 120 us there, the gain of 35 iterations.
constexpr uint64_t PR_HOT_MIN_VECTORS = 1ull << 21;
static int pr_hot_choose(grz_graph* g)
{
    const uint64_t V = g->V;
    if (g->pr_hot_known) return GRZ_OK;
    cudaStream_t st = g->stream;
    const uint64_t words = (V + 31) / 32;
    g->pr_nhot = 0;
    if (g->pull.nvec < PR_HOT_MIN_VECTORS || V >= GRZ_HUB_BASE) {
        g->pr_hot_known = 1;
        return GRZ_OK;
    }
    const uint32_t dmin = (uint32_t)std::min<uint64_t>(g->E / V + 1, 0xffffffffull);
    unsigned long long* hist = nullptr;
    uint32_t* cnt = nullptr;
    unsigned long long pick[3] = { 0, 0, 0 };
    int rc = grz_dev_alloc(g, (void**)&hist, sizeof(unsigned long long) * (2 * HOT_BINS + 3));
    if (!rc) rc = grz_cuda_check(g, cudaMemsetAsync(hist, 0, sizeof(unsigned long long) * (2 * HOT_BINS + 3), st), "memset");
    if (!rc) {
        const unsigned grid = (unsigned)std::min<uint64_t>(blocks_for(V), (uint64_t)g->num_sms * 8);
        k_hot_hist<<<grid, PR_THREADS, 0, st>>>(g->degree, V, dmin, hist); GRZ_COUNT_LAUNCH(g);
        k_hot_pick<<<1, HOT_PICK_T, 0, st>>>(hist, V < GRZ_PR_HOT_MAX_V ? GRZ_PR_HOT_MAX : GRZ_PR_HOT_FEW, hist + 2 * HOT_BINS); GRZ_COUNT_LAUNCH(g);
        rc = grz_cuda_check(g, cudaGetLastError(), "k_hot_pick");
    }
    if (!rc) rc = grz_cuda_check(g, cudaMemcpyAsync(pick, hist + 2 * HOT_BINS, sizeof(pick), cudaMemcpyDeviceToHost, st), "D2H");
    if (!rc) rc = grz_cuda_check(g, cudaStreamSynchronize(st), "hot sources");
    if (!rc && pick[1] && pick[2] * 10 >= g->E) {
        rc = grz_dev_alloc(g, (void**)&g->pr_hotmap, sizeof(uint2) * words);
        if (!rc) rc = grz_dev_alloc(g, (void**)&cnt, sizeof(uint32_t) * words);
        if (!rc) rc = grz_dev_alloc(g, (void**)&g->pr_hot_vid, sizeof(uint32_t) * pick[1]);
        if (!rc) {
            k_hot_mark<<<blocks_for(V), PR_THREADS, 0, st>>>(g->degree, V, dmin, (uint32_t)pick[0], g->pr_hotmap, cnt); GRZ_COUNT_LAUNCH(g);
            rc = grz_cuda_check(g, cudaGetLastError(), "k_hot_mark");
        }
        if (!rc) rc = grz_exclusive_sum_u32_on(g, cnt, cnt, words, nullptr, st);
        if (!rc) {
            k_hot_base<<<blocks_for(words), PR_THREADS, 0, st>>>(cnt, words, g->pr_hotmap, g->pr_hot_vid); GRZ_COUNT_LAUNCH(g);
            rc = grz_cuda_check(g, cudaGetLastError(), "k_hot_base");
        }
        for (int i = 0; i < 2 && !rc; ++i) {
            rc = grz_dev_alloc(g, (void**)&g->pr_hot[i], sizeof(pk_t) * (GRZ_PR_HOT_MAX + 2));
            // the slots past the last stay zero
            if (!rc) rc = grz_cuda_check(g, cudaMemsetAsync(g->pr_hot[i], 0, sizeof(pk_t) * (GRZ_PR_HOT_MAX + 2), st), "memset");
        }
    }
    grz_dev_free(g, hist);
    grz_dev_free(g, cnt);
    if (rc) {
        for (void* p : { (void*)g->pr_hotmap, (void*)g->pr_hot_vid, (void*)g->pr_hot[0], (void*)g->pr_hot[1] }) grz_dev_free(g, p);
        g->pr_hotmap = nullptr;
        g->pr_hot_vid = nullptr;
        g->pr_hot[0] = g->pr_hot[1] = nullptr;
        return rc;
    }
    if (g->pr_hotmap) g->pr_nhot = (uint32_t)pick[1];
    g->pr_hot_known = 1;
    return GRZ_OK;
}

// The pull list encoded for the packed gather (source segments are encoded as they are built).
static int pr_hot_encode(grz_graph* g)
{
    if (!g->pr_nhot || g->pr_hot_nbr) return GRZ_OK;
    if (g->tune.withhold & GRZ_WITHHOLD_HOT_LIST) return GRZ_ERR_NOMEM;
    GRZ_TRY(grz_dev_alloc(g, (void**)&g->pr_hot_nbr, sizeof(uint4) * g->pull.nvec));
    k_hot_encode<<<blocks_for(g->pull.nvec), PR_THREADS, 0, g->stream>>>(g->pull.nbr, g->pull.nvec, g->pr_hotmap, g->pr_nhot, g->pr_hot_nbr);
    GRZ_COUNT_LAUNCH(g);
    return grz_cuda_check(g, cudaGetLastError(), "k_hot_encode");
}

static int pr_build_segments(grz_graph* g, uint32_t bits);

// Sources per segment (log2) of the segmented lists, 0 for none: the tuned size, else by the size
// of the packed props (8V bytes) against L2; never more than GRZ_PR_MAX_SEGMENTS segments.  GB300
// (128 MB of L2), ms per iteration unsegmented / with 2^24 / 2^23 sources per segment, and the first
// grz_pr_init's extra ms for the lists:
//   hot sources (R-MAT): 2^25 vertices 2.16 / 2.39 / 2.45; 40M 2.78 / 2.50 / 2.58 (+8.1); 50M 2.95 /
//     2.06 / 2.17 (+6.5); 2^26 7.85 / 5.07 / 5.31 (+13): from 2.75 times L2 on, where the lists pay
//     for themselves within a run of 8 iterations, in segments of 1.25 times L2
//   none (uniform): 8.4M 0.59 / - / 0.62; 10M, degree 16 0.89 / - / 0.80, degree 6 0.45 / - / 0.53; 13M
//     1.65 / - / 1.04 and 0.75 / - / 0.68; 17M 2.71 / 2.81 / 1.45; 30M 7.04 / 4.86 / 3.25; 40M 3.26 /
//     3.01 / 3.21; 60M 10.2 / 7.37 / 7.74 (+0.8 to +2.6): from 3/4 of L2 on, in segments of 5/8 of
//     L2 while that gives at most four, else of twice that
// (`force`: for the CC pull, before the hot sources are known.)
static uint32_t pr_segment_bits(const grz_graph* g, int force)
{
    const uint64_t V = g->V;
    uint32_t bits = 0;
    const uint32_t sb = g->tune.pr_segment_bits;
    if (sb >= 8) {
        bits = sb;
    } else if (sb == 0) {
        const uint64_t props = (uint64_t)sizeof(pk_t) * V, l2 = (uint64_t)g->l2_bytes;
        const bool hot = force || g->pr_nhot;
        if (force || props * 4 > l2 * (hot ? 11 : 3)) {
            bits = 8;
            while ((8ull << (bits + 1)) <= l2 * 5 / (hot ? 4 : 8)) ++bits;
            if (!hot && ((V + (1ull << bits) - 1) >> bits) > 4) ++bits;
        }
    }
    while (bits && ((V + (1ull << bits) - 1) >> bits) > GRZ_PR_MAX_SEGMENTS) ++bits;
    return bits;
}

int grz_pr_ensure_segments(grz_graph* g, int force)
{
    const uint32_t bits = pr_segment_bits(g, force);
    if (!bits || g->pull.nhub || !g->pull.nvec || !g->pull.ascending) return GRZ_OK;
    return pr_build_segments(g, bits);
}

// The PageRank arrays of V vertices, with those of the packed props if `pk`.
static int pr_arrays(grz_graph* g, bool pk)
{
    // together (GB300, the first grz_pr_init of a graph of 300k vertices 338 us with eight allocations, 119 in one; 16
    // iterations on R-MAT of 2^20 vertices with it 1380 and 1148 us)
    const uint64_t V = g->V;
    const grz_part part[] = { { (void**)&g->pr_fx[0], sizeof(u128) * (V + 1) }, { (void**)&g->pr_fx[1], sizeof(u128) * (V + 1) },
                              { (void**)&g->pr_rowacc, sizeof(u128) * (V + 1) }, { (void**)&g->pr_pk[0], pk ? sizeof(pk_t) * (V + 1) : 0 },
                              { (void**)&g->pr_pk[1], pk ? sizeof(pk_t) * (V + 1) : 0 }, { (void**)&g->pr_sum, sizeof(u128) * 2 * (blocks_for(V) + 1) },
                              { (void**)&g->pr_cut, sizeof(uint32_t) * ((V + 31) / 32 + 1) }, { (void**)&g->pr_K, sizeof(double) * 2 },
                              { (void**)&g->pr_small_parts, sizeof(u128) * 2 * PS_CTAS } };
    if (pk && (g->tune.withhold & GRZ_WITHHOLD_PACKED)) return GRZ_ERR_NOMEM;
    GRZ_CK(g, grz_alloc_arrays(part, sizeof(part) / sizeof(part[0]), &g->pr_mem));
    g->pr_pk_own = 0;
    g->pr_lists_changed = 1;
    return GRZ_OK;
}

// the packed props by themselves, where the other arrays came without them
static int pr_packed_arrays(grz_graph* g)
{
    if (g->tune.withhold & GRZ_WITHHOLD_PACKED) return GRZ_ERR_NOMEM;
    const size_t half = (sizeof(pk_t) * (g->V + 1) + 255) & ~(size_t)255;
    GRZ_CK(g, cudaMalloc((void**)&g->pr_pk[0], 2 * half));
    g->pr_pk[1] = g->pr_pk[0] + half / sizeof(pk_t);
    g->pr_pk_own = 1;
    GRZ_CK(g, cudaMemsetAsync(g->pr_pk[0], 0, 2 * half, g->stream));
    return GRZ_OK;
}

// Packed props, segments and the encoded list only make the iterations faster: where the memory for one of
// them cannot be had, the graph runs without it.
static int pr_or_without(int rc) { return rc == GRZ_ERR_NOMEM ? GRZ_OK : rc; }

int grz_pr_prepare(grz_graph* g)
{
    const uint64_t V = g->V;
    if (!g->pr_fx[0]) {
        int rc = pr_arrays(g, g->tune.pr_props != 1);
        if (rc == GRZ_ERR_NOMEM && g->tune.pr_props != 1) rc = pr_arrays(g, false);
        if (rc) return rc;
    }
    if (g->pr_lists_changed) {
        // (also after a reload with the same V, which kept the arrays)
        g->pr_rowacc_stale = 0;
        g->pr_cut_vec = 0;
        // the sums, and the props: entry V of both prop arrays is a permanent zero that invalid lanes gather
        // (from pr_fx[0] to the end of pr_rowacc, or of pr_pk[1], in one piece)
        const bool pk = g->pr_pk[0] && !g->pr_pk_own;
        const char* const end = pk ? (const char*)(g->pr_pk[1] + V + 1) : (const char*)(g->pr_rowacc + V + 1);
        GRZ_CK(g, cudaMemsetAsync(g->pr_fx[0], 0, (size_t)(end - (const char*)g->pr_fx[0]), g->stream));
        if (g->pr_pk_own) GRZ_CK(g, cudaMemsetAsync(g->pr_pk[0], 0, (size_t)((char*)(g->pr_pk[1] + V + 1) - (char*)g->pr_pk[0]), g->stream));
        g->pr_lists_changed = 0;
    }
    // Packed props (8 bytes) unless 16-byte fixed point is asked for: half the gathered working set
    // for a few integer instructions per edge (GB300, a thread per vector, gather per iteration, 16 ->
    // 8 bytes: R-MAT 20 71 -> 63 us, R-MAT 24 1089 -> 938 us, uniform 3M vertices 153 -> 145 us).
    g->pr_pkmode = g->tune.pr_props != 1;
    if (!g->pull.nhub && V) GRZ_TRY(pr_or_without(pr_hot_choose(g)));
    // Source segments (pr_segment_bits): each segment's props mostly stay in L2 while its edges
    // stream, instead of one random DRAM sector per gathered prop.  They need sources in ascending
    // order along each destination's lanes: not a hub-encoded list, nor one that is only grouped.
    const uint32_t bits = pr_segment_bits(g, 0);
    g->pr_segmode = 0;
    if (bits && g->pull.nhub == 0 && g->pull.nvec && g->pull.ascending) {
        const int rc = pr_build_segments(g, bits);
        GRZ_TRY(pr_or_without(rc));
        if (!rc) g->pr_segmode = g->pr_pkmode = 1;  // the segments gather the props packed
    }
    if (g->pr_pkmode && !g->pr_pk[0]) {
        GRZ_TRY(pr_or_without(pr_packed_arrays(g)));
        if (!g->pr_pk[0]) g->pr_segmode = g->pr_pkmode = 0;
    }
    if (g->pr_pkmode && !g->pr_segmode && !g->pull.nhub && V) GRZ_TRY(pr_or_without(pr_hot_encode(g)));
    return GRZ_OK;
}

// Builds the source-segmented pull lists with 2^bits sources per segment (once per lists, bits and
// encoding: with the hot sources as codes when there are any).
static int pr_build_segments(grz_graph* g, uint32_t bits)
{
    if (g->seg_nbr && g->seg_bits == bits && g->seg_nhot == g->pr_nhot) return GRZ_OK;
    if (g->tune.withhold & GRZ_WITHHOLD_SEGMENTS) return GRZ_ERR_NOMEM;
    grz_dev_free(g, g->seg_nbr);
    grz_dev_free(g, g->seg_dst);
    g->seg_nbr = nullptr;
    g->seg_dst = nullptr;
    g->seg_bits = 0;
    const uint64_t V = g->V, n = g->pull.nvec;
    const uint32_t nseg = (uint32_t)((V + (1ull << bits) - 1) >> bits);
    if (nseg == 0 || nseg > GRZ_PR_MAX_SEGMENTS) return grz_set_error(g, GRZ_ERR_RANGE, "%u source segments (at most %d)", nseg, GRZ_PR_MAX_SEGMENTS);
    cudaStream_t st = g->stream;
    uint32_t *start = nullptr, *off = nullptr, *tot = nullptr;
    const uint64_t npair = (uint64_t)nseg * (V + 1);
    int rc = grz_dev_alloc(g, (void**)&start, sizeof(uint32_t) * npair);
    if (!rc) rc = grz_dev_alloc(g, (void**)&off, sizeof(uint32_t) * npair);
    if (!rc) rc = grz_dev_alloc(g, (void**)&tot, sizeof(uint32_t) * (nseg + 1));
    if (!rc) rc = grz_cuda_check(g, cudaMemsetAsync(start, 0, sizeof(uint32_t) * npair, st), "memset");
    if (!rc) rc = grz_cuda_check(g, cudaMemsetAsync(off, 0, sizeof(uint32_t) * npair, st), "memset");
    if (!rc) {
        k_seg_bounds<<<blocks_for(n), PR_THREADS, 0, st>>>(g->pull.nbr, g->pull.shared, g->pull.rowptr, n, V, bits, start, off); GRZ_COUNT_LAUNCH(g);
        const unsigned grid = (unsigned)std::min<uint64_t>(blocks_for(npair), (uint64_t)g->num_sms * 8);
        k_seg_sizes<<<grid, PR_THREADS, 0, st>>>(start, off, npair); GRZ_COUNT_LAUNCH(g);
        rc = grz_cuda_check(g, cudaGetLastError(), "k_seg_bounds");
    }
    for (uint32_t sg = 0; sg < nseg && !rc; ++sg)
        rc = grz_exclusive_sum_u32_on(g, off + (uint64_t)sg * (V + 1), off + (uint64_t)sg * (V + 1), V + 1, tot + sg, st);
    std::vector<uint32_t> th(nseg);
    if (!rc) rc = grz_cuda_check(g, cudaMemcpyAsync(th.data(), tot, sizeof(uint32_t) * nseg, cudaMemcpyDeviceToHost, st), "D2H");
    if (!rc) rc = grz_cuda_check(g, cudaStreamSynchronize(st), "segment counts");
    SegFirst first;
    uint64_t total = 0;
    if (!rc) {
        for (uint32_t sg = 0; sg < nseg; ++sg) {
            g->seg_first[sg] = first.at[sg] = total;
            total += th[sg];
        }
        g->seg_first[nseg] = total;
        if (total >= 0xffffffffull) rc = grz_set_error(g, GRZ_ERR_RANGE, "segmented lists of %llu vectors", (unsigned long long)total);
    }
    if (!rc) rc = grz_dev_alloc(g, (void**)&g->seg_nbr, sizeof(uint4) * std::max<uint64_t>(total, 1));
    if (!rc) rc = grz_dev_alloc(g, (void**)&g->seg_dst, sizeof(uint32_t) * std::max<uint64_t>(total, 1));
    if (!rc) {
        k_seg_emit<<<blocks_for(n), PR_THREADS, 0, st>>>(g->pull.nbr, g->pull.shared, g->pull.rowptr, n, V, bits, start, off, first,
                                                         g->pr_nhot ? g->pr_hotmap : nullptr, g->pr_nhot,
                                                         reinterpret_cast<uint32_t*>(g->seg_nbr), g->seg_dst); GRZ_COUNT_LAUNCH(g);
        rc = grz_cuda_check(g, cudaGetLastError(), "k_seg_emit");
    }
    for (void* q : { (void*)start, (void*)off, (void*)tot }) grz_dev_free(g, q);
    if (rc) {
        grz_dev_free(g, g->seg_nbr);
        grz_dev_free(g, g->seg_dst);
        g->seg_nbr = nullptr;
        g->seg_dst = nullptr;
        return rc;
    }
    g->seg_bits = bits;
    g->seg_nhot = g->pr_nhot;
    g->seg_gen++;
    g->nseg = nseg;
    return GRZ_OK;
}

// PageRank initial state (props, zero accumulators, S_0)
int grz_pr_init_state(grz_graph* g, double damping)
{
    int rc = grz_pr_prepare(g);
    if (rc) {
        g->pr_lists_changed = 1;  // no state to iterate
        return rc;
    }
    g->pr_damping = damping;
    g->pr_cur = 0;
    g->pr_fx_stale = g->pr_pkmode;
    g->pr_pk_stale = g->pr_pk[0] && !g->pr_pkmode;
    g->pr_sum_cur = 0;
    g->pr_iters_done = 0;
    if (g->V) {
        const unsigned grid = (unsigned)std::min<uint64_t>(blocks_for(g->V), (uint64_t)g->num_sms * 8);
        k_pr_init<<<grid, PR_THREADS, 0, g->stream>>>(g->inv_deg, g->degree, g->V, 1.0 / (double)g->V, g->accum, g->pr_fx[0],
                                                      g->pr_pkmode ? g->pr_pk[0] : nullptr, pr_hot_on(g) ? g->pr_hotmap : nullptr,
                                                      g->pr_hot[0], g->pr_sum); GRZ_COUNT_LAUNCH(g);
        GRZ_CK(g, cudaGetLastError());
        g->pr_nparts[0] = grid;
    }
    return GRZ_OK;
}

// resident blocks per SM of the general gather kernel (its grid is persistent: SMs x resident)
template <typename P>
static int pr_gather_resident(grz_graph* g)
{
    static int resident[64] = {};
    if (g->device < 0 || g->device >= 64) return 1;
    if (!resident[g->device]) {
        int r = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_pr_gather<P>, PR_THREADS, 0) != cudaSuccess || r < 1) {
            cudaGetLastError();
            r = 1;
        }
        resident[g->device] = r;
    }
    return resident[g->device];
}

// the general gather over vectors [first, first + count) of the pull list
template <typename P>
static int pr_gather(grz_graph* g, uint64_t first, uint64_t count, const PRConst& pc, const P* props)
{
    if (count == 0) return GRZ_OK;
    grz_prof_begin(g, GRZ_PROF_PR_GATHER);
    const uint64_t want = g->tune.pr_grid ? g->tune.pr_grid : (uint64_t)g->num_sms * pr_gather_resident<P>(g);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(blocks_for(count), want));
    k_pr_gather<P><<<grid, PR_THREADS, 0, g->stream>>>(g->pull.nbr, g->pull.shared, first, count, g->pull.nvec, props, (uint32_t)g->V,
                                                       g->pr_rowacc, g->pull.hub_vid, g->pull.nhub, pc);
    GRZ_COUNT_LAUNCH(g);
    grz_prof_end(g);
    return grz_cuda_check(g, cudaGetLastError(), "k_pr_gather");
}

// shared-memory opt-in of the packed gather with a hot table, once per device
static int pr_gather_pk_config(grz_graph* g)
{
    static bool done[64] = {};
    if (g->device >= 0 && g->device < 64 && done[g->device]) return GRZ_OK;
    const int bytes = (int)(sizeof(pk_t) * (GRZ_PR_HOT_MAX + 2));
    GRZ_CK(g, cudaFuncSetAttribute(k_pr_gather_pk<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    GRZ_CK(g, cudaFuncSetAttribute(k_pr_gather_pk<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (g->device >= 0 && g->device < 64) done[g->device] = true;
    return GRZ_OK;
}

static unsigned pr_gather_pk_grid(const grz_graph* g, uint64_t nvec)
{
    const uint64_t want = g->tune.pr_grid ? g->tune.pr_grid : (uint64_t)g->num_sms;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((nvec + PK_MIN_RANGE - 1) / PK_MIN_RANGE, want));
}

// vectors of a warp's range: an even share of the list, a multiple of 4
static uint32_t pr_gather_pk_range(uint64_t nvec, unsigned grid)
{
    const uint64_t nwarps = (uint64_t)grid * (PK_THREADS / 32);
    const uint64_t share = ((nvec + nwarps - 1) / nwarps + 3) & ~3ull;
    return (uint32_t)std::max<uint64_t>(share, PK_MIN_RANGE);
}

// the packed gather over vectors [first, end) of `nbr` (encoded when there are hot sources)
template <bool ADD>
static int pr_gather_pk(grz_graph* g, const uint4* nbr, const uint32_t* dstv, uint64_t first, uint64_t end, const PRConst& pc)
{
    const uint64_t span = end - (first & ~3ull);
    const unsigned grid = pr_gather_pk_grid(g, span);
    const uint32_t per = pr_gather_pk_range(span, grid);
    const pk_t* props = g->pr_pk[g->pr_cur];
    cudaError_t e;
    if (pr_hot_on(g)) {
        GRZ_TRY(pr_gather_pk_config(g));
        const size_t smem = sizeof(pk_t) * 2 * ((g->pr_nhot + 2) / 2);
        e = pdl_launch(k_pr_gather_pk<true, ADD>, grid, PK_THREADS, smem, g->stream, nbr, dstv, (uint32_t)first, (uint32_t)end, per, props,
                       (uint32_t)g->V, (const pk_t*)g->pr_hot[g->pr_cur], g->pr_nhot, g->pr_rowacc, pc);
    } else {
        e = pdl_launch(k_pr_gather_pk<false, ADD>, grid, PK_THREADS, 0, g->stream, nbr, dstv, (uint32_t)first, (uint32_t)end, per, props,
                       (uint32_t)g->V, (const pk_t*)nullptr, 0u, g->pr_rowacc, pc);
    }
    GRZ_COUNT_LAUNCH(g);
    return grz_cuda_check(g, e, "k_pr_gather_pk");
}

// The gather over the source segments in order, each adding into the accumulators (which the
// apply of segmented iterations leaves all zero).  One profiler record spans all segments.
static int pr_gather_segments(grz_graph* g, const PRConst& pc0)
{
    grz_prof_begin(g, GRZ_PROF_PR_GATHER);
    bool first = true;
    int rc = GRZ_OK;
    for (uint32_t sg = 0; sg < g->nseg && !rc; ++sg) {
        const uint64_t a = g->seg_first[sg], b = g->seg_first[sg + 1];
        if (a == b) continue;
        PRConst pc = pc0;
        if (!first) pc.K_out = nullptr;  // the iteration's constant once
        first = false;
        rc = pr_gather_pk<true>(g, g->seg_nbr, g->seg_dst, a, b, pc);
    }
    // no edges at all: the constant still has to be published
    if (first && !rc) rc = pr_gather_pk<true>(g, g->seg_nbr, g->seg_dst, 0, 0, pc0);
    grz_prof_end(g);
    return rc;
}

// one PageRank iteration: edge-pull gather + vertex phase (two kernels)
int grz_pr_fused_iteration(grz_graph* g, int write_double_props)
{
    if (g->V == 0) return GRZ_OK;
    const int k = g->pr_sum_cur;
    const double dV = (double)g->V;
    const uint32_t stride = blocks_for(g->V) + 1;  // each half of pr_sum holds up to blocks_for(V) partials
    PRConst pc;
    pc.part_in = g->pr_sum + (size_t)k * stride;
    pc.nparts = g->pr_nparts[k];
    pc.K_out = g->pr_K;
    pc.damping = g->pr_damping;
    pc.c = (1.0 - g->pr_damping) / dV;
    pc.nverts = dV;
    // hot sources are chosen by grz_pr_init for a list without hub encoding
    const bool packed = g->pr_pkmode && !g->pull.nhub;
    const uint64_t n = g->pull.nvec;
    int rc = g->pr_pkmode ? pr_sync_pk(g) : pr_sync_fx(g);
    if (rc) return rc;
    if (g->pr_segmode) {
        GRZ_TRY(grz_pr_rowacc_clean(g));  // (unsegmented iterations came before)
        rc = pr_gather_segments(g, pc);
    } else if (packed) {
        rc = pr_cut_for(g, pr_gather_pk_range(n, pr_gather_pk_grid(g, n)));
        if (rc) return rc;
        grz_prof_begin(g, GRZ_PROF_PR_GATHER);
        rc = pr_gather_pk<false>(g, pr_hot_on(g) ? g->pr_hot_nbr : g->pull.nbr, g->pull.shared, 0, n, pc);
        grz_prof_end(g);
    } else {
        rc = pr_cut_for(g, PR_THREADS);
        if (!rc) rc = g->pr_pkmode ? pr_gather(g, 0, n, pc, (const pk_t*)g->pr_pk[g->pr_cur]) : pr_gather(g, 0, n, pc, (const u128*)g->pr_fx[g->pr_cur]);
    }
    if (rc) return rc;
    const bool hot = g->pr_pkmode && pr_hot_on(g);
    grz_prof_begin(g, GRZ_PROF_PR_APPLY);
    const uint64_t agrid = std::max<uint64_t>(1, std::min<uint64_t>((g->V + (uint64_t)PR_THREADS * PR_APPLY_U - 1) /
                                                                        ((uint64_t)PR_THREADS * PR_APPLY_U),
                                                                    (uint64_t)g->num_sms * PR_APPLY_RESIDENT));
    const cudaError_t ae = pdl_launch(k_pr_apply, (unsigned)agrid, PR_THREADS, 0, g->stream, g->pr_rowacc, (const uint32_t*)g->pr_cut, g->pr_segmode,
                                      (const double*)g->inv_deg, (const uint32_t*)g->degree, g->V, (const double*)g->pr_K,
                                      g->pr_sum + (size_t)(k ^ 1) * stride, g->pr_damping, g->pr_fx[g->pr_cur ^ 1],
                                      g->pr_pkmode ? g->pr_pk[g->pr_cur ^ 1] : (pk_t*)nullptr, write_double_props ? g->prop : (double*)nullptr,
                                      hot ? (const uint2*)g->pr_hotmap : (const uint2*)nullptr, g->pr_hot[g->pr_cur ^ 1]); GRZ_COUNT_LAUNCH(g);
    grz_prof_end(g);
    GRZ_CK(g, ae);
    g->pr_nparts[k ^ 1] = (uint32_t)agrid;
    g->pr_fx_stale = g->pr_pkmode;  // the new props are only in pr_pk
    g->pr_rowacc_stale = !g->pr_segmode;  // the apply of segmented iterations clears all
    g->pr_cur ^= 1;
    g->pr_sum_cur = k ^ 1;
    g->pr_iters_done++;
    return GRZ_OK;
}

// resident blocks per SM of the persistent kernel (a cooperative launch needs them all resident)
template <typename P, int MINB>
static int pr_persistent_resident(grz_graph* g)
{
    static int resident[64] = {};
    if (g->device < 0 || g->device >= 64) return 1;
    if (!resident[g->device]) {
        int r = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_pr_persistent<P, MINB>, PR_THREADS, 0) != cudaSuccess || r < 1) {
            cudaGetLastError();
            r = 1;
        }
        resident[g->device] = r;
    }
    return resident[g->device];
}

// Whether grz_pr_iterate runs its iterations in one persistent launch.  Measured on GB300 (R-MAT
// 20, 16 iterations): two kernels 93 us per iteration, the persistent kernel (6 blocks per SM)
// 109 us: its gather must read the props through the coherent path (its apply rewrites them in
// the same launch) and holds fewer blocks per SM.  Two kernels stay the default.
int grz_pr_use_persistent(const grz_graph* g) { return g->tune.pr_persistent >= 2 && !g->pr_segmode; }

// `iters` PageRank iterations (gather + apply each) in one cooperative launch.  Synchronises the
// graph's stream to read the barrier's error word.  A wait that runs out returns GRZ_ERR_TIMEOUT
// and leaves the PageRank state uninitialised (grz_pr_init starts over).
int grz_pr_persistent_iterations(grz_graph* g, uint32_t iters)
{
    if (iters == 0 || g->V == 0) return GRZ_OK;
    if (!g->pr_bar) {
        GRZ_CK(g, cudaMalloc(&g->pr_bar, sizeof(PRBar)));
        GRZ_CK(g, cudaMallocHost(&g->pr_bar_host, sizeof(PRBar)));
    }
    int rc = g->pr_pkmode ? pr_sync_pk(g) : pr_sync_fx(g);
    if (!rc) rc = pr_cut_for(g, PR_THREADS);
    if (rc) return rc;
    const bool eight = g->tune.pr_persistent == 3;
    const int resident = eight ? (g->pr_pkmode ? pr_persistent_resident<pk_t, 8>(g) : pr_persistent_resident<u128, 8>(g))
                               : (g->pr_pkmode ? pr_persistent_resident<pk_t, 6>(g) : pr_persistent_resident<u128, 6>(g));
    uint64_t want = g->tune.pr_grid ? g->tune.pr_grid : (uint64_t)g->num_sms * resident;
    want = std::min<uint64_t>(want, (uint64_t)g->num_sms * resident);  // co-resident
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, blocks_for(g->V)));  // partial slots
    const uint32_t stride = blocks_for(g->V) + 1;
    const bool timing = g->prof && g->prof->on;
    PRPersist q;
    memset(&q, 0, sizeof(q));
    q.nbr = g->pull.nbr;
    q.dstv = g->pull.shared;
    q.nvec = g->pull.nvec;
    q.V = (uint32_t)g->V;
    q.hub_vid = g->pull.hub_vid;
    q.nhub = g->pull.nhub;
    q.rowacc = g->pr_rowacc;
    q.cut = g->pr_cut;
    q.inv_deg = g->inv_deg;
    q.degree = g->degree;
    q.fx[0] = g->pr_fx[0];
    q.fx[1] = g->pr_fx[1];
    q.pk[0] = g->pr_pk[0];
    q.pk[1] = g->pr_pk[1];
    q.pkmode = g->pr_pkmode;
    q.cur = g->pr_cur;
    q.sum[0] = g->pr_sum;
    q.sum[1] = g->pr_sum + stride;
    q.sum_cur = g->pr_sum_cur;
    q.nparts0 = g->pr_nparts[g->pr_sum_cur];
    q.K = g->pr_K;
    q.damping = g->pr_damping;
    q.nverts = (double)g->V;
    q.c = (1.0 - g->pr_damping) / q.nverts;
    q.iters = iters;
    q.prop_out = nullptr;
    q.bar = (PRBar*)g->pr_bar;
    q.limit_ns = (unsigned long long)(g->tune.pr_wait_limit_us ? g->tune.pr_wait_limit_us : 2000000u) * 1000ull;
    q.withhold_block = (int)g->tune.pr_withhold - 1;
    q.time_phases = timing ? 1 : 0;
    GRZ_CK(g, cudaMemsetAsync(g->pr_bar, 0, 4 * sizeof(unsigned int), g->stream));
    void* args[] = { &q };
    const void* fn = eight ? (g->pr_pkmode ? (const void*)k_pr_persistent<pk_t, 8> : (const void*)k_pr_persistent<u128, 8>)
                           : (g->pr_pkmode ? (const void*)k_pr_persistent<pk_t, 6> : (const void*)k_pr_persistent<u128, 6>);
    GRZ_CK(g, cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(PR_THREADS), args, 0, g->stream));
    GRZ_COUNT_LAUNCH(g);
    const size_t rb = timing ? sizeof(PRBar) : 4 * sizeof(unsigned int);
    GRZ_CK(g, cudaMemcpyAsync(g->pr_bar_host, g->pr_bar, rb, cudaMemcpyDeviceToHost, g->stream));
    GRZ_CK(g, cudaStreamSynchronize(g->stream));
    const PRBar* hb = (const PRBar*)g->pr_bar_host;
    if (hb->err) {
        // the iteration stopped part-way: the accumulators and props are inconsistent
        GRZ_CK(g, cudaMemsetAsync(g->pr_rowacc, 0, sizeof(u128) * (g->V + 1), g->stream));
        g->pr_rowacc_stale = 0;
        g->pr_lists_changed = 1;
        return grz_set_error(g, GRZ_ERR_TIMEOUT, "PageRank grid barrier %u: a wait ran out after %u us", hb->where,
                             g->tune.pr_wait_limit_us ? g->tune.pr_wait_limit_us : 2000000u);
    }
    if (timing)
        for (uint32_t i = 0; i < iters && i < 64; ++i) {
            grz_prof_direct(g, GRZ_PROF_PR_GATHER, (float)(hb->gather_ns[i] * 1e-6));
            grz_prof_direct(g, GRZ_PROF_PR_APPLY, (float)(hb->apply_ns[i] * 1e-6));
        }
    if (iters & 1) {
        g->pr_cur ^= 1;
        g->pr_sum_cur ^= 1;
    }
    g->pr_nparts[g->pr_sum_cur] = grid;
    g->pr_fx_stale = g->pr_pkmode;
    if (pr_hot_on(g)) {
        // the persistent form does not keep the hot table: packed again before the next fused iteration
        GRZ_TRY(pr_sync_fx(g));
        g->pr_pk_stale = 1;
    }
    g->pr_rowacc_stale = 1;
    g->pr_iters_done += iters;
    return GRZ_OK;
}

static bool pr_small_fits(const grz_graph* g)
{
    static int known[64] = {};  // per device: 1 fits, 2 does not
    if (g->device < 0 || g->device >= 64 || (g->tune.withhold & GRZ_WITHHOLD_CLUSTERS)) return false;
    if (!known[g->device]) known[g->device] = grz_clusters_fit((const void*)k_pr_small, PS_CTAS, PS_T, ps_smem(PS_MAX_V)) ? 1 : 2;
    return known[g->device] == 1;
}

// Whether a graph's iterations run in one cluster (k_pr_small): packed props of a small graph, unless a
// form or grid of the two kernels is asked for, or their times, or the device cannot hold the cluster.
static bool pr_use_small(const grz_graph* g)
{
    return g->pr_pkmode && !g->pr_segmode && !g->pull.nhub && !g->pr_nhot && g->tune.pr_persistent == 0 && g->tune.pr_grid == 0 &&
           !(g->prof && g->prof->on) && g->V && g->V <= PS_MAX_V && g->pull.nvec <= PS_MAX_VEC && pr_small_fits(g);
}

static int pr_small_iterations(grz_graph* g, uint32_t iters)
{
    GRZ_TRY(pr_sync_pk(g));
    const uint32_t stride = blocks_for(g->V) + 1;
    const int k = g->pr_sum_cur, cur = g->pr_cur ^ (int)(iters & 1);
    PRSmall q;
    q.nbr = g->pull.nbr;
    q.rowptr = g->pull.rowptr;
    q.V = (uint32_t)g->V;
    q.nvec = (uint32_t)g->pull.nvec;
    q.inv_deg = g->inv_deg;
    q.degree = g->degree;
    q.dstv = g->pull.shared;
    q.props0 = g->pr_pk[g->pr_cur];
    q.props1 = g->pr_pk[g->pr_cur ^ 1];
    q.parts = g->pr_small_parts;
    q.part_in = g->pr_sum + (size_t)k * stride;
    q.nparts = g->pr_nparts[k];
    q.part_out = g->pr_sum + (size_t)(k ^ 1) * stride;
    q.damping = g->pr_damping;
    q.nverts = (double)g->V;
    q.c = (1.0 - g->pr_damping) / q.nverts;
    q.iters = iters;
    k_pr_small<<<PS_CTAS, PS_T, ps_smem((uint32_t)g->V), g->stream>>>(q); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    g->pr_cur = cur;
    g->pr_sum_cur = k ^ 1;
    g->pr_nparts[k ^ 1] = 1;
    g->pr_fx_stale = 1;
    g->pr_iters_done += iters;
    return GRZ_OK;
}

// `iterations` PageRank iterations in the form that suits the graph
int grz_pr_iterations(grz_graph* g, uint32_t iterations)
{
    if (grz_pr_use_persistent(g)) return grz_pr_persistent_iterations(g, iterations);
    if (iterations && pr_use_small(g)) return pr_small_iterations(g, iterations);
    for (uint32_t i = 0; i < iterations; ++i) GRZ_TRY(grz_pr_fused_iteration(g, 0));
    return GRZ_OK;
}

// Edge-pull phase alone, over vectors [first, first+count).  Slices of the list (the reference's
// per-NUMA-node lists) may come in separate calls, in list order.  The call whose slice ends the
// list publishes the double accumulators and their exact sum into g->glob.
int grz_pr_edge_pull(grz_graph* g, uint64_t first, uint64_t count)
{
    if (g->V == 0) return GRZ_OK;
    int rc = grz_pr_rowacc_clean(g);
    if (rc == GRZ_OK) rc = pr_sync_fx(g);
    if (rc) return rc;
    PRConst pc;
    memset(&pc, 0, sizeof(pc));
    rc = pr_gather(g, first, count, pc, (const u128*)g->pr_fx[g->pr_cur]);
    if (rc) return rc;
    if (first + count < g->pull.nvec) return GRZ_OK;
    k_pr_accum_out<<<blocks_for(g->V), PR_THREADS, 0, g->stream>>>(g->pr_rowacc, g->V, g->accum, g->glob); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    return GRZ_OK;
}

// vertex phase over [first, first+count) with S from the reduce buffer
int grz_pr_vertex(grz_graph* g, uint64_t first, uint64_t count, double S)
{
    if (first >= g->V) return GRZ_OK;
    if (first + count > g->V) count = g->V - first;
    const double dV = (double)g->V;
    const double G = (1.0 - S) / dV;
    const double c = (1.0 - g->pr_damping) / dV;
    const double K = fma(G, g->pr_damping, c);
    int rc = pr_sync_fx(g);
    if (rc) return rc;
    g->pr_pk_stale = g->pr_pk[0] != nullptr;  // the props change in the fixed-point form only
    // the props being gathered are rewritten in place: the boundary path keeps one live copy
    k_pr_vertex<<<blocks_for(count), PR_THREADS, 0, g->stream>>>(g->accum, g->inv_deg, g->prop, g->pr_fx[g->pr_cur],
                                                                 first, count, g->pr_damping, K); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    return GRZ_OK;
}

// reference-format props (double) from the current fixed-point props, into device or mapped host memory
int grz_pr_props_to_double(grz_graph* g, double* out)
{
    if (g->V == 0) return GRZ_OK;
    if (g->pr_fx_stale) {
        k_pk_unpack<<<blocks_for(g->V), PR_THREADS, 0, g->stream>>>(g->pr_pk[g->pr_cur], g->V, nullptr, out); GRZ_COUNT_LAUNCH(g);
    } else {
        k_fx_to_double<<<blocks_for(g->V), PR_THREADS, 0, g->stream>>>(g->pr_fx[g->pr_cur], g->V, out); GRZ_COUNT_LAUNCH(g);
    }
    GRZ_CK(g, cudaGetLastError());
    return GRZ_OK;
}

// ---------------------------------------------------------------------------------------------
// PageRank push (EDGE_FORCE_PUSH): source/phase_edge_push_pr.asm:42-354.  Each valid lane adds
// the source's prop to the destination's accumulator.  Here the accumulator is an exact u128
// (two 64-bit atomics with carry), so push and pull give bit-identical sums, in any order.

namespace {

__global__ void k_pr_push(const uint4* __restrict__ nbr, const uint32_t* __restrict__ shared, uint64_t first,
                          uint64_t count, const u128* __restrict__ prop_fx, u128* __restrict__ acc_fx,
                          u128* __restrict__ glob)
{
    __shared__ u128 red[PR_THREADS / 32];
    const uint64_t i = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    u128 s = u128_zero();
    if (i < count) {
        const uint64_t v = first + i;
        const uint4 n = __ldg(nbr + v);
        const u128 msg = ld_fx(prop_fx, shared[v]);
        const uint32_t ids[4] = { n.x, n.y, n.z, n.w };
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (ids[l] == GRZ_INVALID_ID) continue;
            u128_atomic_add(&acc_fx[ids[l]], msg);
            s = u128_add(s, msg);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = u128_add(s, u128_shfl_down(s, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = (threadIdx.x < PR_THREADS / 32) ? red[threadIdx.x] : u128_zero();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = u128_add(s, u128_shfl_down(s, o));
        if (threadIdx.x == 0) u128_slot_add(glob, s);
    }
}

// accumulators (exact) -> double accumulators, then reset (phase_vertex_pr.asm:101-106)
__global__ void k_pr_push_accum_out(u128* __restrict__ acc_fx, double* __restrict__ accum, uint64_t first, uint64_t count)
{
    const uint64_t i = (uint64_t)blockIdx.x * PR_THREADS + threadIdx.x;
    if (i >= count) return;
    const uint64_t v = first + i;
    accum[v] = fx_to_double(acc_fx[v]);
    acc_fx[v] = u128_zero();
}

}  // namespace

int grz_pr_push_phase(grz_graph* g, uint64_t first_vec, uint64_t count)
{
    if (!g->push.nbr) return grz_set_error(g, GRZ_ERR_STATE, "push list not loaded");
    if (count == 0) return GRZ_OK;
    // the pull accumulators double as the push accumulators (all zero between uses)
    int rc = grz_pr_rowacc_clean(g);
    if (rc == GRZ_OK) rc = pr_sync_fx(g);
    if (rc) return rc;
    k_pr_push<<<blocks_for(count), PR_THREADS, 0, g->stream>>>(g->push.nbr, g->push.shared, first_vec, count,
                                                               g->pr_fx[g->pr_cur], g->pr_rowacc, g->glob); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    k_pr_push_accum_out<<<blocks_for(g->V), PR_THREADS, 0, g->stream>>>(g->pr_rowacc, g->accum, 0, g->V); GRZ_COUNT_LAUNCH(g);
    GRZ_CK(g, cudaGetLastError());
    return GRZ_OK;
}
