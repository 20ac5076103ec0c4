// grz_switch.cuh -- the engine decision's device code: the state's features and the MLP's forward pass
// of one sample.  Shared by the decision kernels (grz_switch.cu) and the kernel that runs many small
// push iterations in one launch (grz_ccbfs.cu), so that both choose alike, bit for bit.
#pragma once

#include "grz_internal.cuh"

#define NF GRZ_MLP_FEATURES
#define NH GRZ_MLP_HIDDEN

namespace {

// parameter layout (floats): W1[NH][NF] b1[NH] W2[NH][NH] b2[NH] W3[NH] b3
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + NH * NF;
constexpr int OFF_W2 = OFF_B1 + NH;
constexpr int OFF_B2 = OFF_W2 + NH * NH;
constexpr int OFF_W3 = OFF_B2 + NH;
constexpr int OFF_B3 = OFF_W3 + NH;
constexpr int NP = OFF_B3 + 1;
static_assert(NP == GRZ_MLP_PARAMS, "parameter count");

__device__ __forceinline__ float relu(float x) { return x > 0.f ? x : 0.f; }

// features of the state the next iteration will start from (computed before the frontier swap:
// has_next is the next HasInfo)
struct FeatIn {
    const unsigned long long* frontier;
    unsigned long long vote_override;  // ~0: read the vote slots
    const unsigned long long* wants;
    const unsigned long long* vote_slots;
    uint64_t words;
    double V, E, max_degree;
    uint32_t iter;
    int app_bfs;
    int last_engine;
};

// MLP forward pass of one sample by one warp, lane j computing hidden unit j.  Same operation
// order as mlp_forward, so the logit equals grz_mlp_predict's.  f: NF features, h: NH scratch
// (both shared); every lane returns the logit.
// One warp, lane j = hidden unit j, the weights in registers: lane j loads its own rows of W1 and
// W2 straight from global memory (all loads issued together, one L2 round trip), and the hidden
// activations pass between lanes by shuffles.  The operation order is mlp_forward's, so the
// logit equals grz_mlp_predict's bit for bit.
// Weights: from global memory, or staged in shared memory for a warp that decides again and again (lane
// j's rows as columns: no bank conflicts).
struct MlpGlobal {
    const float* p;
    __device__ __forceinline__ float w1(int lane, int k) const { return __ldg(p + OFF_W1 + lane * NF + k); }
    __device__ __forceinline__ float w2(int lane, int k) const { return __ldg(p + OFF_W2 + lane * NH + k); }
    __device__ __forceinline__ float rest(int off) const { return __ldg(p + off); }
};
constexpr int MLP_WARP_FLOATS = NP;
struct MlpShared {
    const float* p;
    __device__ __forceinline__ float w1(int lane, int k) const { return p[OFF_W1 + k * NH + lane]; }
    __device__ __forceinline__ float w2(int lane, int k) const { return p[OFF_W2 + k * NH + lane]; }
    __device__ __forceinline__ float rest(int off) const { return p[off]; }
};
__device__ __forceinline__ void mlp_stage(const float* __restrict__ params, float* s, int tid, int nthreads)
{
    for (int i = tid; i < NP; i += nthreads) {
        int to = i;
        if (i < OFF_B1) to = OFF_W1 + (i % NF) * NH + i / NF;
        else if (i >= OFF_W2 && i < OFF_B2) to = OFF_W2 + ((i - OFF_W2) % NH) * NH + (i - OFF_W2) / NH;
        s[to] = __ldg(params + i);
    }
}

// a lane's share of the weights, so that they can be loaded long before the features are known
struct MlpLane {
    float w1[NF], w2[NH], b1, b2, w3, b3;
    template <typename W>
    __device__ __forceinline__ void load(const W w, int lane)
    {
#pragma unroll
        for (int k = 0; k < NF; ++k) w1[k] = w.w1(lane, k);
#pragma unroll
        for (int k = 0; k < NH; ++k) w2[k] = w.w2(lane, k);
        b1 = w.rest(OFF_B1 + lane);
        b2 = w.rest(OFF_B2 + lane);
        w3 = w.rest(OFF_W3 + lane);
        b3 = w.rest(OFF_B3);
    }
    __device__ __forceinline__ float logit(const float* f) const
    {
        float s = b1;
#pragma unroll
        for (int k = 0; k < NF; ++k) s = fmaf(w1[k], f[k], s);
        const float h1 = relu(s);
        s = b2;
#pragma unroll
        for (int k = 0; k < NH; ++k) s = fmaf(w2[k], __shfl_sync(0xffffffffu, h1, k), s);
        const float h2 = relu(s);
        float z = b3;
#pragma unroll
        for (int k = 0; k < NH; ++k) z = fmaf(__shfl_sync(0xffffffffu, w3, k), __shfl_sync(0xffffffffu, h2, k), z);
        return z;
    }
};

template <typename W>
__device__ __forceinline__ float mlp_logit_warp(const W w, const float* f, int lane)
{
    MlpLane m;
    m.load(w, lane);
    return m.logit(f);
}

// Feature k of the state, lane k computing it: every feature is a quotient, of a number or its logarithm, so
// the lanes select operands and then all take one path.  (As a switch, its cases ran one after the other,
// each with its own logarithms and division: GB300, a BFS of 764 small iterations with the learned policy 3.58 ms,
// so 2.70 ms; a CC run on 4096 vertices, four decisions, 125 us, so 118.)
__device__ __forceinline__ float feature(int k, const FeatIn& in, float F, float U, float vote)
{
    const float V = (float)in.V, E = (float)in.E;
    // log2f(frontier + 1) / log2f(V + 1); frontier / V; vote / E; log2f(vote + 1) / log2f(E + 1)
    float num = k < 2 || k == 11 ? F : vote;
    float den = k == 0 || k == 1 ? V : (k == 11 ? 32.f : E);
    bool log_num = k == 0 || k == 3 || k == 11, log_den = k == 0 || k == 3;
    // BFS: unvisited / V, else 0; iteration / 32; log2f(E / V + 1) / 8; log2f(V) / 32
    if (k == 4) { num = in.app_bfs ? U : 0.f; den = V; }
    if (k == 5) { num = (float)in.iter; den = 32.f; }
    if (k == 6) { num = E / V; den = 8.f; log_num = true; }
    if (k == 7) { num = V; den = 32.f; log_num = true; }
    // log2f(largest degree + 1) / log2f(E + 1); BFS; the last engine; log2f(frontier + 1) / 32 (k == 11, above)
    if (k == 8) { num = (float)in.max_degree; log_num = log_den = true; }
    if (k == 9) { num = in.app_bfs ? 1.f : 0.f; den = 1.f; }
    if (k == 10) { num = in.last_engine ? 1.f : 0.f; den = 1.f; }
    const float lnum = log2f(k == 7 ? num : num + 1.f), lden = log2f(den + 1.f);
    return (log_num ? lnum : num) / (log_den ? lden : den);
}

}  // namespace
