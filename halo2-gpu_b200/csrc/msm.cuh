// Internal MSM interface shared by the C-ABI launchers and the batched /
// no-allocation entry points.
#pragma once
#include <cstdint>
#include "abi.cuh"
#include "curve.cuh"

namespace h2b {

// Entries per accumulation chunk: `fixed` if set, else the fewest whole waves
// of `threads` chunks of at most `cap` entries, evened out.
struct MsmChunk {
    uint32_t fixed, threads, cap;
};

constexpr int MSM_FOLD_PASSES = 6;

struct MsmPlan {
    uint64_t n;
    int c;           // window bits
    int W;           // windows
    uint32_t H;      // buckets per window = 2^(c-1)
    uint64_t NB;     // Wr * H
    uint64_t nv;     // virtual (GLV half) scalars = 2n
    uint64_t max_entries;
    MsmChunk chunk;
    uint64_t max_chunks;
    uint32_t fix_lanes;  // lanes that sum a bucket's chunk heads
    uint32_t fix_limit;  // heads beyond which a bucket is listed instead
    uint64_t max_dense;  // capacity of that list
    uint64_t max_items;  // and of the list of its pieces
    int passes;      // passes of the bucket reduction
    int fold[MSM_FOLD_PASSES];  // index bits that each folds
    uint64_t leaves; // Wr c: the points the last step doubles and adds up
    uint64_t tn;     // points per window slice of a precomputed table (0: plain bases)
    int Wr;          // windows in the bucket reduction (W; with a table 1, or one per merged job)
};

struct MsmScratch {
    G1Affine* bases_stage;
    Fr* scalar_stage;
    Fr* canon;
    uint32_t* counts;
    uint32_t* offsets;
    uint32_t* cursor;
    uint32_t* scan_tmp;
    uint32_t* sorted;
    G1Xyzz* buckets;
    G1Xyzz* heads;
    uint32_t* dense;
    uint2* items;
    G1Xyzz* fold[2];     // outputs of the reduction passes, alternating
    uint32_t* tailctr;   // arrival counters of the last reduction step
    G1Jac* result;
    Fq* phix;            // plain bases: x of phi(P_i) (form 0: P_i, then phi(P_i), as points x 2^261)
};

// Plan for an MSM that runs beside `concurrent` - 1 others (batches): same
// results; the accumulation's chunk size assumes the others share the SMs.
MsmPlan msm_plan_shared(uint64_t n, uint64_t tn, uint32_t concurrent);
MsmPlan msm_plan(uint64_t n);
// Plan for an MSM of n <= tn points over a precomputed window table built for
// tn points (window width chosen by tn; all windows share one bucket set).
MsmPlan msm_plan_table(uint64_t n, uint64_t tn);
void msm_plan_scratch(const MsmPlan& p, ScratchPlan& sp, bool scalar_host, bool bases_host);
MsmScratch msm_carve(const MsmPlan& p, ScratchArena& ar, bool scalar_host, bool bases_host);
RustError msm_run(const MsmPlan& p, const MsmScratch& s, const Fr* d_scalars, const G1Affine* d_bases,
                  cudaStream_t st);
// Merged runs: up to MSM_MERGE_MAX MSMs over one window table of tn points
// (n_total scalars in all) sorted, accumulated and reduced together, job j in
// bucket set j; each job's 96-byte result goes to outs[j].
constexpr uint32_t MSM_MERGE_MAX = 64;
MsmPlan msm_plan_merged(uint64_t n_total, uint64_t tn, uint32_t J);
// Bucket offsets, scatter cursors and chunk starts count sorted entries in 32
// bits, and an entry names its point in 31.
inline bool msm_plan_fits(const MsmPlan& p)
{
    return p.n < (1ull << 30) && p.max_entries < (1ull << 32) && p.tn < (1ull << 30) &&
           2 * (uint64_t)p.W * p.tn < (1ull << 31);
}
RustError msm_run_merged(const MsmPlan& p, const MsmScratch& s, uint32_t J, const Fr* const* scalars,
                         const uint64_t* ns, const G1Affine* table, G1Jac* const* outs, cudaStream_t st);
void msm_set_tuning(int window_bits, int chunk);

} // namespace h2b
