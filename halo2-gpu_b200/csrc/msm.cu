// Pippenger G1 MSM behind Params::commit / commit_lagrange
// (halo2_proofs/src/poly/kzg/commitment.rs:456-575) and the reference entry
// points `_halo2_multiexp{,_device_bases,_device_scalars_device_bases}`
// (halo2_proofs/cuda/src/multiexp.cu:260-525, declared at
// halo2_proofs/src/cuda/culib.rs:30-70).
//
// Pipeline (all stream-ordered, no host round trip until the 96-byte result):
//  1. split:   each scalar leaves Montgomery form and is split by the GLV
//              endomorphism into two signed halves below 2^127 (glv.cuh), so
//              n points become 2n virtual points P_i, phi(P_i) with 128-bit
//              scalars: half the windows, half the buckets and half the
//              final doubling chain of a 254-bit Pippenger.  The caller's
//              scalars are never mutated.
//  2. digits:  signed c-bit windows, digits in [-(2^(c-1)-1), 2^(c-1)], so a
//              window needs 2^(c-1) buckets; a negative digit (or a negative
//              half) adds -P.
//  3. sort:    counting sort of (window, bucket) keys -- warp-aggregated
//              histogram, exclusive scan to bucket offsets, warp-aggregated
//              scatter of point indices (sign in bit 31).
//  4. accumulate: the sorted entry list is cut into equal chunks of K entries,
//              one chunk per thread, so dense buckets (e.g. every scalar == 1
//              landing in one bucket) cost the same as sparse ones.  A chunk
//              writes finished buckets directly and the partial sum of the
//              bucket it started in the middle of to a per-chunk slot.
//  5. fixup:   each bucket adds the per-chunk partials it spans; buckets that
//              span many chunks get warps of their own.
//  6. reduce:  per window, the buckets are folded bit by bit of their index
//              into c - 1 bit sums and a total; every one of them is doubled
//              by its whole weight on its own SM, and they are added up.
//  7. output:  XYZZ -> the reference's Jacobian image {x, y, 1} (or (0,1,0)).
#include <algorithm>
#include "abi.cuh"
#include "curve.cuh"
#include "msm.cuh"
#include "prof.cuh"
#include "glv.cuh"
#include "scan_u32.cuh"

extern "C" RustError h2b_exec_fork(cudaStream_t parent, uint32_t n, cudaStream_t* out);  // exec.cu

namespace h2b {

static constexpr int GLV_BITS = 127;
// longest MSM: 2 halves x 8 windows x n entries stay below 2^32 (msm_plan_fits)
static constexpr uint64_t MSM_MAX_LENGTH = 1ull << 27;
static constexpr uint32_t SIGN_BIT = 0x80000000u;
// widest window the tuning override accepts (22 bits: 6 windows per GLV half)
static constexpr int MSM_MAX_WINDOW = 22;
static constexpr uint32_t FOLD_THREADS = 320;     // most threads of a reduction CTA
// accumulation threads resident at once: 148 SMs x 4 CTAs x 128
static constexpr uint32_t ACC_RESIDENT = 148u * 4u * 128u;
static constexpr uint32_t ACC_MIN_K = 4;          // smallest chunk
// Largest chunk of an MSM that runs alone: larger ones leave fewer heads to the
// fixup, smaller ones even out the ends of the accumulation (2^22 witness mix
// 8.14 ms at 64, 8.07 at 96 and 128, 8.12 at 192).
static constexpr uint32_t ACC_MAX_K = 96;
static constexpr uint32_t ACC_MAX_K_SHARED = 128; // and of one of several that run at once
// Lanes that the fixup spreads few buckets over (2^16 table, one MSM: 0.60 ms at
// 2^15, 0.72 ms at 2^17 lanes; 2^20: 3.37 and 3.42 ms).
static constexpr uint64_t FIX_THREADS = 32768;
static constexpr uint32_t HEADS_PIECE = 32;       // chunk heads per warp of a long bucket
static constexpr uint32_t HEADS_PIECES_MAX = 1024;
static constexpr uint64_t MSM_PIPE_MIN = 1ull << 18;  // host scalars from here on are copied in pieces
static constexpr int MSM_PIPE_PIECES = 8;

static int g_msm_window_override = 0;
static int g_msm_acc_variant = 6;  // form of the accumulation kernel: 6 or 0

uint64_t fq_batch_invert_scratch(uint64_t n);
int tune_value(int param, int log_n);  // tune.cu
RustError fq_batch_invert(Fq* d, uint64_t n, void* scratch, uint64_t scratch_bytes, cudaStream_t st);

static int g_msm_chunk_override = 0;
static uint32_t g_msm_prefetch = 2;   // entries ahead whose point the accumulation prefetches into L2 (0: none)

void msm_set_tuning(int window_bits, int chunk)
{
    g_msm_window_override = window_bits;
    g_msm_chunk_override = chunk;
}

static int floor_log2(uint64_t n)
{
    int lg = 0;
    while ((1ull << (lg + 1)) <= n) lg++;
    return lg;
}

// Windows of c bits over the GLV halves (magnitudes < 2^GLV_BITS); the top one
// must leave room for the signed-digit carry (its width <= c - 1).
static int window_count(int c)
{
    const int W = (GLV_BITS + c - 1) / c;
    return GLV_BITS - c * (W - 1) > c - 1 ? W + 1 : W;
}

// The width an MSM over n points would like, before widen_c.  `plain`: over
// plain bases, whose window width may come from the per-size tuning table; a
// window table's width is fixed when it is built.
static int wanted_c(uint64_t n, bool plain = false)
{
    const int lg = floor_log2(n);
    if (g_msm_window_override >= 4 && g_msm_window_override <= MSM_MAX_WINDOW) return g_msm_window_override;
    if (plain) {
        const int tuned = tune_value(0, lg);
        if (tuned) return tuned;
        // Plain-base widths, measured on B200 (uniform / witness-mix scalars, us).
        // What is left over for the top window matters as much as the width:
        // 7, 9 and 14 bits leave one bit of the 127, whose one or two buckets
        // hold half of all entries each.
        //   1000 points:  8 bits 387 / 442, 10 bits 452 / 462
        //   2^13: 8 bits 464 / 514, 13 bits 514 / 526
        //   2^16: 13 bits 751 / 685, 12 bits 803 / 716, 16 bits 929 / 944
        //   2^18: 13 bits 1522 / 1138, 16 bits 1527 / 1302
        //   2^19: 16 bits 2267 / 1755, 13 bits 2553 / 1761
        if (lg >= 19) return 16;
        if (lg >= 14) return 13;
        return 8;
    }
    // Window tables: every window's digits land in one bucket set of 2^(c-1)
    // buckets, so a narrow window makes few, long buckets (2^18 points at 13
    // bits: 4096 buckets of about 1300 entries).
    // Widths from a sweep of c in 10..18 on B200 (bench.py --case
    // table_widths; uniform / witness-mix scalars, n = table size, ms):
    //   2^12: 10 bits 0.29 / 0.29, 13 bits 0.30 / 0.34
    //   2^13: 13 bits 0.32 / 0.36, 10 bits 0.34 / 0.38
    //   2^16: 13 bits 0.58 / 0.53, 10 bits 0.99 / 0.82, 16 bits 0.49 / 0.52
    //   2^17: 16 bits 0.69 / 0.63, 13 bits 0.84 / 0.71
    //   2^20: 16 bits 3.26 / 2.19, 13 bits 4.62 / 2.93
    // (16 bits would serve 2^15 and 2^16 too; a table's layout follows this
    // rule, and a caller may hold tables of the present one.)
    if (lg >= 17) return 16;
    if (lg >= 13) return 13;
    if (lg >= 10) return 10;
    return 7;
}

// A width set by hand can be too narrow for the 32-bit entry count (4 bits
// from 2^26 points on): plain bases then take the next one that fits.  A table
// keeps the width it was built with, at which table_fits holds.
static int choose_c(uint64_t n, bool plain = false)
{
    int c = wanted_c(n, plain);
    while (plain && c < MSM_MAX_WINDOW && 2 * n * (uint64_t)window_count(c) >= (1ull << 32)) c++;
    return c;
}

// tn > 0: precomputed window table of tn points per window; all windows then
// share one bucket set and the reduction has a single window (one per job of
// a merged run).
static MsmPlan plan_core(uint64_t n, int c, uint64_t tn, uint32_t concurrent = 1, uint32_t jobs = 1)
{
    MsmPlan p;
    p.n = n;
    p.tn = tn;
    p.c = c;
    p.W = window_count(c);
    p.H = 1u << (c - 1);
    p.Wr = tn ? (int)jobs : p.W;
    p.NB = (uint64_t)p.Wr * p.H;
    p.nv = 2 * n;
    p.max_entries = p.nv * (uint64_t)p.W;
    // Entries per accumulation chunk (one thread walks a chunk; chunk_entries
    // below fixes it on the device from the entries that are really there): a
    // tuned or overriding size as it is, else the fewest whole waves of
    // resident threads whose chunks stay within the cap.  MSMs that run
    // `concurrent` at a time share the resident threads and take larger
    // chunks, whose fewer heads cost the fixup less.  A tuned size applies to
    // a plain-base MSM that runs alone.
    const bool alone_plain = concurrent <= 1 && tn == 0;
    const int tuned_k = alone_plain ? tune_value(1, floor_log2(n)) : 0;
    p.chunk.fixed = g_msm_chunk_override > 0 ? (uint32_t)g_msm_chunk_override : (uint32_t)std::max(tuned_k, 0);
    p.chunk.threads = std::max<uint32_t>(ACC_RESIDENT / std::max(concurrent, 1u), 128u);
    p.chunk.cap = concurrent <= 1 ? ACC_MAX_K : ACC_MAX_K_SHARED;
    // more entries never make fewer chunks than one wave less: the bound over
    // every entry count up to max_entries
    p.max_chunks = p.chunk.fixed ? p.max_entries / p.chunk.fixed + 2
                                 : std::min<uint64_t>(p.max_entries / ACC_MIN_K,
                                                      (p.max_entries / ((uint64_t)p.chunk.threads * p.chunk.cap) + 1) *
                                                          p.chunk.threads) + 2;
    // Bits folded by each pass of the bucket reduction: nine at first (one CTA
    // of 256 threads per 512 buckets), then as many as keep a pass's first
    // step within one addition per thread (FOLD_THREADS).
    p.passes = 0;
    int arrays = 1, left = c - 1;
    do {
        int m = std::min(left, 9);
        while (m > 1 && (uint32_t)arrays << (m - 1) > FOLD_THREADS) m--;
        p.fold[p.passes++] = m;
        arrays += m;
        left -= m;
    } while (left > 0);
    p.leaves = (uint64_t)p.Wr * c;                     // c - 1 bit sums and the total per window
    // Lanes per bucket that sum its chunk heads: enough to occupy the GPU when
    // the buckets are few, no more than the heads an average bucket has.  A
    // bucket with more than `limit` heads goes to warps of its own instead.
    const uint64_t avg = p.max_chunks / p.NB + 1;
    p.fix_lanes = 1;
    while (p.fix_lanes < 32 && p.NB * p.fix_lanes < FIX_THREADS && p.fix_lanes < avg) p.fix_lanes *= 2;
    p.fix_limit = p.fix_lanes * (uint32_t)std::max<uint64_t>(2 * avg / p.fix_lanes + 2, 4);
    p.max_dense = p.max_chunks / p.fix_limit + 1;
    p.max_items = p.max_chunks / HEADS_PIECE + p.max_dense + 1;
    return p;
}

MsmPlan msm_plan(uint64_t n) { return plan_core(n, choose_c(n, true), 0); }

MsmPlan msm_plan_table(uint64_t n, uint64_t tn) { return plan_core(n, choose_c(tn), tn); }

MsmPlan msm_plan_shared(uint64_t n, uint64_t tn, uint32_t concurrent)
{
    return tn ? plan_core(n, choose_c(tn), tn, concurrent) : plan_core(n, choose_c(n, true), 0, concurrent);
}

// J MSMs over one window table of tn points, n_total scalars in all, as one
// run: job j's entries go to bucket set j (J bucket sets of H buckets), so
// the sort, the accumulation and the bucket reduction run once for all jobs.
MsmPlan msm_plan_merged(uint64_t n_total, uint64_t tn, uint32_t J)
{
    MsmPlan p = plan_core(n_total, choose_c(tn), tn, 1, J);
    return p;
}

// Points that the even (k = 0) or odd passes of the bucket reduction write at
// most: 1 + (bits folded so far) arrays of one element per block left.
static uint64_t msm_fold_points(const MsmPlan& p, int k)
{
    uint64_t most = 0;
    int done = 0;
    for (int i = 0; i < p.passes; i++) {
        done += p.fold[i];
        if ((i & 1) == k) most = std::max<uint64_t>(most, (uint64_t)p.Wr * (1 + done) * (p.H >> done));
    }
    return most;
}

void msm_plan_scratch(const MsmPlan& p, ScratchPlan& sp, bool scalar_host, bool bases_host)
{
    if (bases_host) sp.add(p.n * sizeof(G1Affine));
    if (scalar_host) sp.add(p.n * sizeof(Fr));       // host scalars staged here
    sp.add(p.n * sizeof(Fr));                         // canonical scalars
    sp.add_n<uint32_t>(p.NB);                         // counts
    sp.add_n<uint32_t>(p.NB + 1);                     // offsets
    sp.add_n<uint32_t>(p.NB);                         // cursor
    sp.add_n<uint32_t>(scan_u32_tiles(p.NB) + 1);     // scan tiles
    sp.add_n<uint32_t>(p.max_entries);                // sorted entries
    sp.add_n<G1Xyzz>(p.NB);                           // bucket sums
    sp.add_n<G1Xyzz>(p.max_chunks);                   // chunk head partials
    sp.add_n<uint32_t>(p.max_dense + 2);              // long buckets, their count, their pieces' count
    sp.add_n<uint2>(p.max_items);                     // their pieces
    for (int k = 0; k < 2; k++) sp.add_n<G1Xyzz>(msm_fold_points(p, k));  // outputs of the reduction passes
    sp.add_n<uint32_t>(p.leaves);                     // counters of the last reduction step
    sp.add_n<G1Jac>(1);                               // result
    if (p.tn == 0) sp.add_n<Fq>((g_msm_acc_variant == 6 ? 1 : 4) * p.n);  // x of phi(P_i); form 0: P_i, phi(P_i) x 2^261
}

MsmScratch msm_carve(const MsmPlan& p, ScratchArena& ar, bool scalar_host, bool bases_host)
{
    MsmScratch s;
    s.bases_stage = bases_host ? (G1Affine*)ar.take(p.n * sizeof(G1Affine)) : nullptr;
    s.scalar_stage = scalar_host ? (Fr*)ar.take(p.n * sizeof(Fr)) : nullptr;
    s.canon = (Fr*)ar.take(p.n * sizeof(Fr));
    s.counts = ar.take_n<uint32_t>(p.NB);
    s.offsets = ar.take_n<uint32_t>(p.NB + 1);
    s.cursor = ar.take_n<uint32_t>(p.NB);
    s.scan_tmp = ar.take_n<uint32_t>(scan_u32_tiles(p.NB) + 1);
    s.sorted = ar.take_n<uint32_t>(p.max_entries);
    s.buckets = ar.take_n<G1Xyzz>(p.NB);
    s.heads = ar.take_n<G1Xyzz>(p.max_chunks);
    s.dense = ar.take_n<uint32_t>(p.max_dense + 2);
    s.items = ar.take_n<uint2>(p.max_items);
    for (int k = 0; k < 2; k++) s.fold[k] = ar.take_n<G1Xyzz>(msm_fold_points(p, k));
    s.tailctr = ar.take_n<uint32_t>(p.leaves);
    s.result = ar.take_n<G1Jac>(1);
    s.phix = p.tn == 0 ? ar.take_n<Fq>((g_msm_acc_variant == 6 ? 1 : 4) * p.n) : nullptr;
    return s;
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------

// Virtual scalars: vs[2i] = k1, vs[2i+1] = k2 of the GLV split of scalar i
// (128-bit magnitudes, sign in bit 127), so entry v stands for point i = v/2,
// taken as P_i (v even) or phi(P_i) (v odd).
__global__ void k_msm_glv(const Fr* __restrict__ sc, uint4* __restrict__ vs, uint64_t n)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint4 a, b;
        glv::decompose(from_mont(ldg(&sc[i])), a, b);
        vs[2 * i] = a;
        vs[2 * i + 1] = b;
    }
}

__device__ __forceinline__ uint32_t window_bits(const uint4& s, int bit, int c)
{
    const uint32_t w[5] = {s.x, s.y, s.z, s.w & 0x7fffffffu, 0u};
    int li = bit >> 5, sh = bit & 31;
    uint64_t v = ((uint64_t)w[li] | ((uint64_t)w[li + 1] << 32)) >> sh;
    return (uint32_t)(v & ((1ull << c) - 1));
}

// Signed digit w of a virtual scalar (carry in/out through `carry`) and its
// bucket key w*H + |d| - 1, or ~0 for a zero digit or an invalid lane.
// With a window table every window shares one bucket set, based at `kb`
// (the job's bucket set in a merged run, 0 otherwise).  The histogram and
// the scatter both take their keys from here, so their counts agree.
__device__ __forceinline__ uint32_t digit_key(const uint4& s, int w, int c, uint32_t H, uint32_t& carry, bool valid,
                                              uint64_t tn, uint32_t kb, int32_t& d)
{
    const uint32_t v = window_bits(s, w * c, c) + carry;
    if (v > H) { d = (int32_t)v - (int32_t)(1u << c); carry = 1; }
    else { d = (int32_t)v; carry = 0; }
    return (valid && d != 0) ? (tn ? kb : (uint32_t)w * H) + (uint32_t)(d < 0 ? -d : d) - 1u : 0xffffffffu;
}

// Warp-aggregated count of one key per lane (all 32 lanes call it together).
__device__ __forceinline__ void hist_key(uint32_t key, uint32_t* __restrict__ counts)
{
    const unsigned lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (key != 0xffffffffu && (int)lane == __ffs(peers) - 1) atomicAdd(&counts[key], __popc(peers));
}

// For each digit: key = w*H + |d| - 1 (or ~0 for zero digits); the entry's
// sign is the digit's sign flipped by the virtual scalar's sign.
// Virtual points v0 <= i < n.
template <bool SCATTER>
__global__ void k_msm_sort(const uint4* __restrict__ vsc, uint64_t v0, uint64_t n, int c, int W, uint32_t H,
                           uint32_t* __restrict__ counts_or_cursor, uint32_t* __restrict__ sorted, uint64_t tn,
                           uint32_t kb)
{
    const unsigned lane = threadIdx.x & 31;
    for (uint64_t base = v0 + blockIdx.x * (uint64_t)blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t i = base + threadIdx.x;
        bool valid = i < n;
        uint4 s = valid ? vsc[i] : make_uint4(0u, 0u, 0u, 0u);
        const bool sneg = (s.w >> 31) != 0;
        uint32_t carry = 0;
        for (int w = 0; w < W; w++) {
            int32_t d;
            const uint32_t key = digit_key(s, w, c, H, carry, valid, tn, kb, d);
            unsigned peers = __match_any_sync(0xffffffffu, key);
            int leader = __ffs(peers) - 1;
            if (!SCATTER) {
                if (key != 0xffffffffu && (int)lane == leader) atomicAdd(&counts_or_cursor[key], __popc(peers));
            } else {
                uint32_t b = 0;
                if (key != 0xffffffffu && (int)lane == leader) b = atomicAdd(&counts_or_cursor[key], __popc(peers));
                b = __shfl_sync(0xffffffffu, b, leader);
                if (key != 0xffffffffu) {
                    uint32_t rank = __popc(peers & ((1u << lane) - 1u));
                    // with a window table the entry names table point w * tn + i/2
                    const uint32_t v = (uint32_t)(i + 2 * (uint64_t)w * tn);
                    sorted[b + rank] = v | (((d < 0) != sneg) ? SIGN_BIT : 0u);
                }
            }
        }
    }
}

// The GLV split of each scalar and, over plain bases, the x coordinate beta x of
// phi(P) = (beta x, y), fused with the digit
// histogram of k_msm_sort<false> for the two halves of each scalar: the
// histogram's atomics overlap the split's memory traffic, and the halves are
// counted from registers instead of re-read.  Loops are block-uniform so
// that every lane reaches the warp-wide match.
__global__ void k_msm_glv_hist(const Fr* __restrict__ sc, uint4* __restrict__ vs, uint64_t lo, uint64_t hi,
                               const G1Affine* __restrict__ bases, Fq* __restrict__ phix, int c, int W, uint32_t H,
                               uint32_t* __restrict__ counts, uint64_t tn)
{
    const Fq beta = glv::beta();
    for (uint64_t base = lo + blockIdx.x * (uint64_t)blockDim.x; base < hi; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = base + threadIdx.x;
        const bool valid = i < hi;
        uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
        if (valid) {
            glv::decompose(from_mont(ldg(&sc[i])), a, b);
            vs[2 * i] = a;
            vs[2 * i + 1] = b;
            if (phix) st(&phix[i], ldg(&bases[i].x) * beta);   // infinity (0, 0) stays (0, 0)
        }
        uint32_t ca = 0, cb = 0;
        for (int w = 0; w < W; w++) {
            int32_t d;
            hist_key(digit_key(a, w, c, H, ca, valid, tn, 0u, d), counts);
            hist_key(digit_key(b, w, c, H, cb, valid, tn, 0u, d), counts);
        }
    }
}


// Bases (affine, memory image x 2^256 mod p) -> canonical x 2^261 mod p, the
// form the lazy accumulation reads; infinity (0, 0) stays (0, 0).
__global__ void k_to_r261(const G1Affine* in, G1Affine* out, uint64_t n, G1Affine* phi)  // in may equal out
{
    const Fq beta = glv::beta();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const G1Affine a = ld_affine(&in[i]);
        G1Affine r;
        r.x = to_r261(a.x);
        r.y = to_r261(a.y);
        if (phi) {
            st(&phi[i].x, to_r261(a.x * beta));   // phi(P) = (beta x, y); infinity stays (0, 0)
            st(&phi[i].y, r.y);
        }
        st(&out[i].x, r.x);
        st(&out[i].y, r.y);
    }
}

// Entries per chunk for M sorted entries (MsmChunk: the plan's rule).
__device__ __forceinline__ uint32_t chunk_entries(const MsmChunk& k, uint32_t M)
{
    if (k.fixed) return k.fixed;
    const uint32_t wave = k.threads * k.cap;               // entries of one wave of the largest chunks
    const uint32_t waves = M / wave + (M % wave != 0);
    const uint32_t threads = k.threads * (waves ? waves : 1u);
    const uint32_t n = M / threads + (M % threads != 0);
    return n < ACC_MIN_K ? ACC_MIN_K : n;
}

// The accumulation in the lazy form (curve.cuh, lazy.cuh): same chunking,
// bucket boundaries and outputs as k_msm_accumulate, over bases in the
// x 2^261 form.  The accumulator's additions and subtractions are one-step
// carry passes with no conditional correction; results are converted back
// to the canonical memory image when a bucket or chunk head is stored.
// phi(P) of the point at bases[j] is stored at bases[phi_off + j] (plain
// bases: phi_off = n; window tables: W n, after all slices).
__global__ void __launch_bounds__(128, 3) k_msm_accumulate_z(const uint32_t* __restrict__ sorted,
                                                             const uint32_t* __restrict__ offsets, uint64_t NB,
                                                             const MsmChunk kc, const G1Affine* __restrict__ bases,
                                                             uint64_t phi_off, G1Xyzz* __restrict__ buckets,
                                                             G1Xyzz* __restrict__ heads)
{
    const FqZ one = fz_from_words(to_r261(Fq::one()));           // 1 in the lazy form (2^261 mod p)
    const FqZ r256 = fz_from_words(Fq::one());                    // 2^256 mod p, for the stores
    const uint32_t M = offsets[NB];
    const uint32_t K = chunk_entries(kc, M);
    const uint64_t nchunks = (M + (uint64_t)K - 1) / K;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < nchunks;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t start = (uint32_t)(t * K);
        const uint32_t end = ((uint64_t)start + K < (uint64_t)M) ? start + K : M;
        uint64_t lo = 0, hi = NB;  // offsets[lo] <= start < offsets[hi]
        while (hi - lo > 1) {
            uint64_t mid = (lo + hi) >> 1;
            if (offsets[mid] <= start) lo = mid; else hi = mid;
        }
        uint64_t b = lo;
        uint32_t next = offsets[b + 1];
        bool head = offsets[b] < start;
        G1XyzzZ acc = xyzzz_inf();
        for (uint32_t e = start; e < end; e++) {
            if (e == next) {
                st_xyzzz(head ? &heads[t] : &buckets[b], acc, r256);
                acc = xyzzz_inf();
                head = false;
                do { b++; next = offsets[b + 1]; } while (next == e);
            }
            const uint32_t ent = sorted[e];
            const uint32_t v = ent & ~SIGN_BIT;
            const bool phi = (v & 1u) != 0;
            const G1Affine P = ld_affine(&bases[(v >> 1) + (phi ? phi_off : 0)]);    // phi(P) precomputed
            if (is_inf(P)) continue;
            FqZ qx = fz_from_words(P.x);                                   // < p
            FqZ qy = fz_from_words(P.y);                                   // < p
            if (ent & SIGN_BIT) qy = fz_sub<FqCfg, 2>(fz_zero<FqCfg>(), qy);  // 2p - y < 2p

            xyzzz_madd(acc, qx, qy, one);
        }
        st_xyzzz(head ? &heads[t] : &buckets[b], acc, r256);
    }
}

// x 2^261 mod p (canonical) -> x 2^256 mod p, canonical: v / 32 mod p as
// (v + t p) / 32 with t = -v / p mod 32.
__device__ __forceinline__ Fq from_r261(const Fq& v)
{
    const uint32_t t = (v.v[0] * FqCfg::N0) & 31u;
    const uint32_t p[8] = {FqCfg::M0, FqCfg::M1, FqCfg::M2, FqCfg::M3, FqCfg::M4, FqCfg::M5, FqCfg::M6, FqCfg::M7};
    uint32_t w[8];
    uint64_t c = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        c += (uint64_t)t * p[i] + v.v[i];
        w[i] = (uint32_t)c;
        c >>= 32;
    }
    Fq r;
#pragma unroll
    for (int i = 0; i < 7; i++) r.v[i] = __funnelshift_r(w[i], w[i + 1], 5);
    r.v[7] = w[7] >> 5;                  // v + 31 p < 2^5 p < 2^259: the carry c joins the top word
    r.v[7] |= (uint32_t)c << 27;
    return r;
}

// The accumulation with coordinates in [0, 2p) on the even/odd product (default).
// TABLE: points in a window table's x 2^261 form, divided by 32 on load, phi(P)
// at phi_off; else the caller's bases as they are, with the x coordinate of
// phi(P) from phix (its y is P's).  Buckets leave in the canonical memory image.
// Ten products an addition (two of them squares, two sharing a reduction) bound
// it: 2^22 witness mix (39.7 M additions) 5.8 ms, against 8.6 ms with the FP64
// form; 128 registers, 16 warps per SM (three CTAs measured 6.18 against 6.09 ms).
template <bool TABLE>
__global__ void __launch_bounds__(128, 4) k_msm_accumulate_e(const uint32_t* __restrict__ sorted,
                                                             const uint32_t* __restrict__ offsets, uint64_t NB,
                                                             const MsmChunk kc, const G1Affine* __restrict__ bases,
                                                             uint64_t phi_off, const Fq* __restrict__ phix,
                                                             G1Xyzz* __restrict__ buckets, G1Xyzz* __restrict__ heads,
                                                             uint32_t pf)
{
    const uint32_t M = offsets[NB];
    const uint32_t K = chunk_entries(kc, M);
    const uint64_t nchunks = (M + (uint64_t)K - 1) / K;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < nchunks;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t start = (uint32_t)(t * K);
        const uint32_t end = ((uint64_t)start + K < (uint64_t)M) ? start + K : M;
        uint64_t lo = 0, hi = NB;  // offsets[lo] <= start < offsets[hi]
        while (hi - lo > 1) {
            uint64_t mid = (lo + hi) >> 1;
            if (offsets[mid] <= start) lo = mid; else hi = mid;
        }
        uint64_t b = lo;
        uint32_t next = offsets[b + 1];
        bool head = offsets[b] < start;
        G1Xyzz acc = xyzz_inf();
        for (uint32_t e = start; e < end; e++) {
            if (e == next) {
                st_xyzze(head ? &heads[t] : &buckets[b], acc);
                acc = xyzz_inf();
                head = false;
                do { b++; next = offsets[b + 1]; } while (next == e);
            }
            if (pf && e + pf < end) {   // bring the point pf entries ahead into L2 (no registers held)
                const uint32_t vn = sorted[e + pf] & ~SIGN_BIT;
                const G1Affine* pn = &bases[(vn >> 1) + (TABLE && (vn & 1u) ? phi_off : 0)];
                asm volatile("prefetch.global.L2 [%0];" ::"l"(pn));
                if (!TABLE && (vn & 1u)) asm volatile("prefetch.global.L2 [%0];" ::"l"(&phix[vn >> 1]));
            }
            const uint32_t ent = sorted[e];
            const uint32_t v = ent & ~SIGN_BIT;
            const bool phi = (v & 1u) != 0;
            G1Affine P;
            if (TABLE) {
                P = ld_affine(&bases[(v >> 1) + (phi ? phi_off : 0)]);
            } else {
                P.x = ldg(phi ? &phix[v >> 1] : &bases[v >> 1].x);
                P.y = ldg(&bases[v >> 1].y);
            }
            if (is_inf(P)) continue;
            const Fq qx = TABLE ? from_r261(P.x) : P.x;
            Fq qy = TABLE ? from_r261(P.y) : P.y;
            if (ent & SIGN_BIT) qy = qsub(Fq::zero(), qy);
            xyzze_madd<true>(acc, qx, qy);
        }
        st_xyzze(head ? &heads[t] : &buckets[b], acc);
    }
}

// pieces of a long bucket with m chunk heads (one warp each)
__device__ __forceinline__ uint32_t head_pieces(uint32_t m)
{
    const uint32_t n = (m + HEADS_PIECE - 1) / HEADS_PIECE;
    return n < HEADS_PIECES_MAX ? n : HEADS_PIECES_MAX;
}

// Adds the chunk heads of each bucket to what the bucket's first chunk left
// in it, G lanes per bucket (a serial share each, then a tree).  A bucket with
// more than `limit` heads is listed instead, with its pieces, for
// k_msm_heads.  Latency-bound unless the buckets are many: one lane per bucket
// took 161 us for 4096 buckets of 19 heads.
template <int G>
__global__ void __launch_bounds__(128, 4) k_msm_fixup(const uint32_t* __restrict__ offsets, uint64_t NB, const MsmChunk kc,
                                                   G1Xyzz* __restrict__ buckets, const G1Xyzz* __restrict__ heads,
                                                   uint32_t limit, uint32_t* __restrict__ dense, uint64_t max_dense,
                                                   uint2* __restrict__ items, uint64_t max_items)
{
    __shared__ G1Xyzz red[G > 1 ? 128 : 1];
    const uint32_t K = chunk_entries(kc, offsets[NB]);
    const uint32_t lane = threadIdx.x & 31, j = lane % G;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    constexpr uint32_t PER = 32 / G;                 // buckets per warp
    for (uint64_t base = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * PER; base < NB;
         base += warps * PER) {                      // uniform within the warp
        const uint64_t gb = base + lane / G;
        uint32_t t0 = 0, t1 = 0;
        bool take = false;
        if (gb < NB) {
            const uint32_t s = offsets[gb], e = offsets[gb + 1];
            if (s == e) {
                if (j == 0) st_xyzz(&buckets[gb], xyzz_inf());
            } else {
                t0 = s / K;
                t1 = (e - 1) / K;
                if (t1 - t0 > limit) {
                    if (j == 0) {
                        const uint32_t n = head_pieces(t1 - t0), at = atomicAdd(&dense[max_dense + 1], n);
                        dense[atomicAdd(&dense[max_dense], 1u)] = (uint32_t)gb;
                        for (uint32_t p = 0; p < n && at + p < max_items; p++) items[at + p] = make_uint2((uint32_t)gb, p);
                    }
                } else {
                    take = t1 > t0;
                }
            }
        }
        G1Xyzz acc = xyzz_inf();
        if (take) {
            if (j == 0) acc = ld_xyzz(&buckets[gb]);
            for (uint32_t t = t0 + 1 + j; t <= t1; t += G) xyzze_add<false>(acc, ld_xyzz(&heads[t]));
        }
        if (G > 1) {
            red[threadIdx.x] = acc;
#pragma unroll 1
            for (int h = G / 2; h > 0; h >>= 1) {
                __syncwarp();
                if (take && j < (uint32_t)h) {
                    xyzze_add<false>(acc, red[threadIdx.x + h]);
                    red[threadIdx.x] = acc;
                }
            }
            __syncwarp();
        }
        if (take && j == 0) st_xyzze(&buckets[gb], acc);
    }
}

// One warp per piece of a long bucket: the sum of its slice of chunk heads,
// left in place of the slice's first head (or added to the bucket when the
// piece is the only one).
__global__ void __launch_bounds__(128) k_msm_heads(const uint32_t* __restrict__ offsets, uint64_t NB, const MsmChunk kc,
                                                   G1Xyzz* __restrict__ buckets, G1Xyzz* heads,
                                                   const uint32_t* __restrict__ dense, uint64_t max_dense,
                                                   const uint2* __restrict__ items)
{
    __shared__ G1Xyzz red[128];
    const uint32_t n = dense[max_dense + 1];
    if (blockIdx.x * (blockDim.x >> 5) >= n) return;
    const uint32_t K = chunk_entries(kc, offsets[NB]);
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t it = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < n;
         it += gridDim.x * (blockDim.x >> 5)) {
        const uint2 item = items[it];
        const uint32_t t0 = offsets[item.x] / K, t1 = (offsets[item.x + 1] - 1) / K, m = t1 - t0;
        const uint32_t P = head_pieces(m);
        const uint32_t b0 = (uint32_t)((uint64_t)m * item.y / P), b1 = (uint32_t)((uint64_t)m * (item.y + 1) / P);
        G1Xyzz acc = xyzz_inf();
        for (uint32_t i = b0 + lane; i < b1; i += 32) xyzze_add<false>(acc, ld_xyzz(&heads[t0 + 1 + i]));
        red[threadIdx.x] = acc;
#pragma unroll 1
        for (int h = 16; h > 0; h >>= 1) {
            __syncwarp();
            if (lane < (uint32_t)h) {
                xyzze_add<false>(acc, red[threadIdx.x + h]);
                red[threadIdx.x] = acc;
            }
        }
        if (lane == 0) {
            if (P > 1) {
                st_xyzze(&heads[t0 + 1 + b0], acc);
            } else {
                xyzze_add<false>(acc, ld_xyzz(&buckets[item.x]));
                st_xyzze(&buckets[item.x], acc);
            }
        }
        __syncwarp();
    }
}

// CTA-wide tree sum of n XYZZ values produced by get(i); result valid in
// thread 0 (coordinates below 2p).
template <class Get>
__device__ G1Xyzz block_sum_xyzz(uint64_t n, Get get)
{
    __shared__ G1Xyzz red[256];
    G1Xyzz acc = xyzz_inf();
    for (uint64_t i = threadIdx.x; i < n; i += blockDim.x) xyzze_add<false>(acc, get(i));
    red[threadIdx.x] = acc;
    __syncthreads();
    int h = blockDim.x >> 1;
    while (h > 1 && (uint64_t)h >= n) h >>= 1;         // no sums above n
    for (; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            G1Xyzz a = red[threadIdx.x];
            xyzze_add<false>(a, red[threadIdx.x + h]);
            red[threadIdx.x] = a;
        }
        __syncthreads();
    }
    G1Xyzz r = red[0];
    __syncthreads();
    return r;
}

// One CTA per long bucket of more than one piece: the pieces' sums into the bucket.
__global__ void __launch_bounds__(256) k_msm_heads_merge(const uint32_t* __restrict__ offsets, uint64_t NB,
                                                         const MsmChunk kc, G1Xyzz* __restrict__ buckets,
                                                         const G1Xyzz* __restrict__ heads,
                                                         const uint32_t* __restrict__ dense, uint64_t max_dense)
{
    const uint32_t cnt = dense[max_dense];
    if (blockIdx.x >= cnt) return;
    const uint32_t K = chunk_entries(kc, offsets[NB]);
    for (uint32_t i = blockIdx.x; i < cnt; i += gridDim.x) {
        const uint32_t gb = dense[i];
        const uint32_t t0 = offsets[gb] / K, m = (offsets[gb + 1] - 1) / K - t0, P = head_pieces(m);
        if (P <= 1) continue;
        G1Xyzz r = block_sum_xyzz(P, [&](uint64_t p) {
            return ld_xyzz(&heads[t0 + 1 + (uint32_t)((uint64_t)m * p / P)]);
        });
        if (threadIdx.x == 0) {
            xyzze_add<false>(r, ld_xyzz(&buckets[gb]));
            st_xyzze(&buckets[gb], r);
        }
        __syncthreads();
    }
}

// Bucket reduction, W_w = sum_{j<H} (j+1) B_{w,j} = sum_j B_j + sum_k 2^k T_k
// with T_k the sum of the buckets whose index has bit k set.
// Folding the top index bit of an array y of n sums gives its T as the upper
// half of y and a new y of the pairwise sums of both halves; every T array
// found so far is halved by the same step.  A pass folds `m` bits: CTA (w, blk)
// takes 2^m consecutive elements of each of the `arrays` arrays of window w
// (array 0 is y, the others are T arrays; `len` elements each) and writes one
// element of each of the arrays + m arrays that result.
// Two additions per bucket, all of them in parallel within a step, so the
// depth is the number of bits: running sums over 8-bucket segments and then
// per-bit sums of the segments (16 and 16 additions one after the other at
// c = 16) took 146 + 212 us for 8 windows of 2^15 buckets and 104 + 210 us for
// one; the two passes here 245 + 61 and 81 + 60 us (two CTAs per SM; one, at 150
// registers, made the first pass 333 us).  A CTA of the first pass whose buckets
// hold no entry writes infinities and leaves (2^20 points, scalars all zero 281 ->
// 212 us, all one 703 -> 653 us; full bucket sets as before).
template <int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS) k_msm_fold(const G1Xyzz* __restrict__ in, uint32_t arrays, uint32_t len,
                                                           int m, G1Xyzz* __restrict__ out, uint32_t* __restrict__ ctr,
                                                           uint32_t nctr, const uint32_t* __restrict__ offsets)
{
    extern __shared__ uint4 fold_smem[];
    G1Xyzz* sm = reinterpret_cast<G1Xyzz*>(fold_smem);
    const uint32_t t = threadIdx.x;
    const uint32_t blocks = len >> m, w = blockIdx.x / blocks, blk = blockIdx.x % blocks;
    if (blockIdx.x == 0)
        for (uint32_t i = t; i < nctr; i += blockDim.x) ctr[i] = 0;
    const G1Xyzz* src = in + (uint64_t)w * arrays * len + ((uint64_t)blk << m);
    if (offsets) {                                     // the first pass (arrays == 1): no entry in any of its buckets
        const uint64_t b0 = (uint64_t)w * len + ((uint64_t)blk << m);
        if (offsets[b0] == offsets[b0 + (1ull << m)]) {
            if (t <= (uint32_t)m) st_xyzz(&out[((uint64_t)w * (m + 1) + t) * blocks + blk], xyzz_inf());
            return;
        }
    }
    uint32_t A = arrays;
#pragma unroll 1
    for (int step = 0; step < m; step++) {
        const int lh = m - 1 - step;                   // log2 of the halved length
        const uint32_t half = 1u << lh, a = t >> lh, i = t & (half - 1);
        const bool active = t < A << lh;
        G1Xyzz x, y;
        if (active) {
            if (step == 0) {
                x = ld_xyzz(&src[(uint64_t)a * len + i]);
                y = ld_xyzz(&src[(uint64_t)a * len + i + half]);
            } else {
                x = sm[(a << (lh + 1)) + i];
                y = sm[(a << (lh + 1)) + i + half];
            }
        }
        __syncthreads();
        if (active) {
            if (a == 0) sm[(A << lh) + i] = y;         // the folded bit's T array
            xyzze_add<false>(x, y);
            sm[(a << lh) + i] = x;
        }
        __syncthreads();
        A++;
    }
    if (t < A) st_xyzze(&out[((uint64_t)w * A + t) * blocks + blk], sm[t]);
}

// A merged run over a window table: window j of the reduction is job j's
// whole sum (the table already holds the window multiples), so each job has
// its own result; otherwise all windows of a run sum into one.
struct MsmOuts {
    G1Jac* p[MSM_MERGE_MAX];
};

// bits folded by each pass of the reduction
struct MsmFold {
    int passes, bits[MSM_FOLD_PASSES];
};

// The reduction's last step: result = sum over windows w of
// 2^(c w) (sum_j B_{w,j} + sum_k 2^k T_{w,k}), `per` points a window.  One warp
// (one CTA) takes one of them, doubles it by its whole weight on the x coordinate alone
// (sl_dbl_many: the chain of a bit sum of the top window is as long as the
// window doublings it replaces, but all of them run at once on their own SMs)
// and the points are then added up pairwise: of two siblings the CTA that
// arrives second adds the other's point and goes on, so no CTA waits for
// another.  The last one of a group converts to the affine image.
// Node i of a level stands at leaf i << level; a pair's counter is its right
// child's leaf index.  Counters start at zero (k_msm_fold).
// The chain is bound by product latency, two per doubling.  Measured at
// c = 16, 8 windows: Horner over bit sums per window, then the window
// doublings with one warp per window on one SM, 567 us; this kernel 214 us.
__global__ void __launch_bounds__(32) k_msm_tail(G1Xyzz* sums, uint32_t per, MsmFold f, int c, uint32_t leaves,
                                                 uint32_t* ctr, const __grid_constant__ MsmOuts outs)
{
    __shared__ __align__(16) Fq sl[20];   // read and written as uint4
    const int lane = (int)threadIdx.x;
    const uint32_t group = blockIdx.x / leaves;
    uint32_t i = blockIdx.x % leaves;
    G1Xyzz* pts = sums + (uint64_t)group * leaves;
    uint32_t* gctr = ctr + (uint64_t)group * leaves;
    // leaf (w, a): the window's total (a = 0) or a bit sum; a pass appends its bits from the highest down
    int dbl = c * (int)(i / per), a = (int)(i % per), base = 0;
    for (int k = 0; k < f.passes && a > 0; k++) {
        if (a <= f.bits[k]) dbl += base + f.bits[k] - a;
        a -= f.bits[k];
        base += f.bits[k];
    }
    // the four coordinates of a point are consecutive: lane j < 4 moves coordinate j
    if (lane < 4) st(&sl[lane], ld(&pts[i].X + lane));
    __syncwarp();
    if (!sl_get(sl, 2).is_zero()) sl_dbl_many(sl, dbl);
    uint32_t cnt = leaves;
    for (int level = 0; cnt > 1; level++) {
        const uint32_t sib = i ^ 1u;
        if (sib < cnt) {
            if (lane < 4) st(&pts[i << level].X + lane, sl_get(sl, lane));
            __threadfence();
            __syncwarp();
            uint32_t old = 0;
            if (lane == 0) old = atomicAdd(&gctr[(i | 1u) << level], 1u);
            old = __shfl_sync(0xffffffffu, old, 0);
            if (old == 0) return;               // the sibling's CTA will take this point
            __threadfence();
            if (lane < 4) {
                const uint4* q = reinterpret_cast<const uint4*>(&pts[sib << level].X + lane);
                uint4* d = reinterpret_cast<uint4*>(&sl[4 + lane]);
                d[0] = __ldcg(q);
                d[1] = __ldcg(q + 1);
            }
            __syncwarp();
            sl_add(sl);
        }
        i >>= 1;
        cnt = (cnt + 1) >> 1;
    }
    if (lane == 0) {
        G1Xyzz r;
        r.X = sl[0]; r.Y = sl[1]; r.ZZ = sl[2]; r.ZZZ = sl[3];
        const G1Jac j = xyzz_to_jac_affine(xyzze_canonical(r));
        G1Jac* out = outs.p[group];
        st(&out->X, j.X);
        st(&out->Y, j.Y);
        st(&out->Z, j.Z);
    }
}

__global__ void k_write_inf(G1Jac* out)
{
    if (threadIdx.x == 0) {
        st(&out->X, Fq::zero());
        st(&out->Y, Fq::one());
        st(&out->Z, Fq::zero());
    }
}

// The first reduction pass takes 64 KB of shared memory (opt-in above 48 KB;
// the attribute is the device's, so it is set on every call).
static cudaError_t fold_smem_ready()
{
    return cudaFuncSetAttribute(k_msm_fold<256, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 512 * (int)sizeof(G1Xyzz));
}

// Steps 5 to 7 from the accumulated buckets: chunk heads, bucket reduction, and
// the results, one per group of `group_windows` reduction windows.
static RustError msm_reduce(const MsmPlan& p, const MsmScratch& s, int group_windows, int c, const MsmOuts& outs,
                            cudaStream_t st)
{
    const unsigned sm_cap = 148u * 16u;
    const unsigned fix_grid = grid_for(p.NB * p.fix_lanes, 128, sm_cap);
    switch (p.fix_lanes) {
#define FIX(G)                                                                                                        \
    case G:                                                                                                           \
        k_msm_fixup<G><<<fix_grid, 128, 0, st>>>(s.offsets, p.NB, p.chunk, s.buckets, s.heads, p.fix_limit, s.dense,  \
                                                 p.max_dense, s.items, p.max_items);                                  \
        break;
        FIX(1) FIX(2) FIX(4) FIX(8) FIX(16) FIX(32)
#undef FIX
    }
    H2B_LAUNCHED("k_msm_fixup");
    k_msm_heads<<<148 * 8, 128, 0, st>>>(s.offsets, p.NB, p.chunk, s.buckets, s.heads, s.dense, p.max_dense, s.items);
    H2B_LAUNCHED("k_msm_heads");
    k_msm_heads_merge<<<148 * 4, 256, 0, st>>>(s.offsets, p.NB, p.chunk, s.buckets, s.heads, s.dense, p.max_dense);
    H2B_LAUNCHED("k_msm_heads_merge");
    const G1Xyzz* in = s.buckets;
    uint32_t arrays = 1, len = p.H;
    MsmFold f;
    f.passes = p.passes;
    for (int k = 0; k < p.passes; k++) {
        const int m = p.fold[k];
        f.bits[k] = m;
        const uint32_t tasks = std::max(arrays << (m - 1), arrays + (uint32_t)m);
        const size_t smem = sizeof(G1Xyzz) * ((size_t)(arrays + 1) << (m - 1));
        H2B_CUDA(fold_smem_ready());
        const auto fold = k == 0 ? k_msm_fold<256, 2> : k_msm_fold<(int)FOLD_THREADS, 1>;
        fold<<<(unsigned)p.Wr * (len >> m), (tasks + 31) / 32 * 32, smem, st>>>(
            in, arrays, len, m, s.fold[k & 1], s.tailctr, k == 0 ? (uint32_t)p.leaves : 0u,
            k == 0 ? s.offsets : nullptr);
        H2B_LAUNCHED("k_msm_fold");
        in = s.fold[k & 1];
        arrays += (uint32_t)m;
        len >>= m;
    }
    k_msm_tail<<<(unsigned)p.leaves, 32, 0, st>>>(s.fold[(p.passes - 1) & 1], (uint32_t)p.c, f, c,
                                                  (uint32_t)group_windows * (uint32_t)p.c, s.tailctr, outs);
    H2B_LAUNCHED("k_msm_tail");
    return ok();
}

// Runs steps 1-7 on device buffers; result (96 bytes) lands in s.result.
// Phases of one MSM on `st`: msm_begin clears the histogram, msm_split takes
// points [lo, hi) through the GLV split (and base conversion) and the
// histogram -- callers may feed the points in pieces as they arrive --, and
// msm_finish sorts, accumulates and reduces.
static RustError msm_begin(const MsmPlan& p, const MsmScratch& s, cudaStream_t st)
{
    prof_begin(PROF_MSM_TOTAL, st);
    H2B_CUDA(cudaMemsetAsync(s.counts, 0, p.NB * sizeof(uint32_t), st));
    H2B_CUDA(cudaMemsetAsync(s.dense + p.max_dense, 0, 2 * sizeof(uint32_t), st));
    return ok();
}

static RustError msm_split(const MsmPlan& p, const MsmScratch& s, const Fr* d_scalars, const G1Affine* d_bases,
                           uint64_t lo, uint64_t hi, cudaStream_t st)
{
    if (hi <= lo) return ok();
    const unsigned sm_cap = 148u * 16u;
    uint4* vsc = reinterpret_cast<uint4*>(s.canon);  // 2n x 16 B in the n x 32 B slot
    k_msm_glv_hist<<<grid_for(hi - lo, 256, sm_cap), 256, 0, st>>>(
        d_scalars, vsc, lo, hi, d_bases, p.tn == 0 && g_msm_acc_variant == 6 ? s.phix : nullptr, p.c, p.W, p.H,
        s.counts, p.tn);
    H2B_LAUNCHED("k_msm_glv_hist");
    return ok();
}

// The bucket accumulation over a window table (p.tn > 0) or plain bases.
static RustError msm_accumulate(const MsmPlan& p, const MsmScratch& s, const G1Affine* pts, cudaStream_t st)
{
    const unsigned grid = grid_for(p.max_chunks, 128, 148u * 32u);
    const uint64_t phi = (uint64_t)p.W * p.tn;
    if (g_msm_acc_variant == 6) {
        if (p.tn)
            k_msm_accumulate_e<true><<<grid, 128, 0, st>>>(s.sorted, s.offsets, p.NB, p.chunk, pts, phi, nullptr,
                                                           s.buckets, s.heads, g_msm_prefetch);
        else
            k_msm_accumulate_e<false><<<grid, 128, 0, st>>>(s.sorted, s.offsets, p.NB, p.chunk, pts, 0, s.phix,
                                                            s.buckets, s.heads, g_msm_prefetch);
        H2B_LAUNCHED("k_msm_accumulate");
        return ok();
    }
    G1Affine* rb = (G1Affine*)s.phix;
    if (!p.tn) {
        k_to_r261<<<grid_for(p.n, 256, 148u * 8u), 256, 0, st>>>(pts, rb, p.n, rb + p.n);
        H2B_LAUNCHED("k_to_r261");
    }
    k_msm_accumulate_z<<<grid, 128, 0, st>>>(s.sorted, s.offsets, p.NB, p.chunk, p.tn ? pts : rb, p.tn ? phi : p.n,
                                             s.buckets, s.heads);
    H2B_LAUNCHED("k_msm_accumulate");
    return ok();
}

static RustError msm_finish(const MsmPlan& p, const MsmScratch& s, const G1Affine* d_bases, cudaStream_t st)
{
    const unsigned sm_cap = 148u * 16u;
    const uint4* vsc = reinterpret_cast<const uint4*>(s.canon);
    H2B_CUDA(scan_u32(s.counts, p.NB, s.offsets, s.scan_tmp, st));
    H2B_CUDA(cudaMemcpyAsync(s.cursor, s.offsets, p.NB * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    k_msm_sort<true><<<grid_for(p.nv, 256, sm_cap), 256, 0, st>>>(vsc, 0, p.nv, p.c, p.W, p.H, s.cursor,
                                                                    s.sorted, p.tn, 0u);
    H2B_LAUNCHED("k_msm_sort<scatter>");
    prof_begin(PROF_MSM_ACCUMULATE, st);
    H2B_TRY(msm_accumulate(p, s, d_bases, st));
    prof_end(PROF_MSM_ACCUMULATE, st);
    MsmOuts o;
    o.p[0] = s.result;
    H2B_TRY(msm_reduce(p, s, p.Wr, p.c, o, st));
    prof_end(PROF_MSM_TOTAL, st);
    return ok();
}

RustError msm_run(const MsmPlan& p, const MsmScratch& s, const Fr* d_scalars, const G1Affine* d_bases, cudaStream_t st)
{
    if (p.n == 0) {
        k_write_inf<<<1, 32, 0, st>>>(s.result);
        H2B_LAUNCHED("k_write_inf");
        return ok();
    }
    H2B_TRY(msm_begin(p, s, st));
    H2B_TRY(msm_split(p, s, d_scalars, d_bases, 0, p.n, st));
    return msm_finish(p, s, d_bases, st);
}

RustError msm_run_merged(const MsmPlan& p, const MsmScratch& s, uint32_t J, const Fr* const* scalars,
                         const uint64_t* ns, const G1Affine* table, G1Jac* const* outs, cudaStream_t st)
{
    if (J == 0) return ok();
    if (J > (uint32_t)MSM_MERGE_MAX || p.tn == 0 || (uint32_t)p.Wr != J)
        return err(cudaErrorInvalidValue, "msm_run_merged: plan does not match the jobs");
    const unsigned sm_cap = 148u * 16u;
    uint4* vsc = reinterpret_cast<uint4*>(s.canon);
    prof_begin(PROF_MSM_TOTAL, st);
    H2B_CUDA(cudaMemsetAsync(s.counts, 0, p.NB * sizeof(uint32_t), st));
    H2B_CUDA(cudaMemsetAsync(s.dense + p.max_dense, 0, 2 * sizeof(uint32_t), st));
    uint64_t at = 0;   // job j's virtual scalars start at vsc + 2 * at
    for (uint32_t j = 0; j < J; j++) {
        if (ns[j] == 0) continue;
        k_msm_glv<<<grid_for(ns[j], 256, sm_cap), 256, 0, st>>>(scalars[j], vsc + 2 * at, ns[j]);
        H2B_LAUNCHED("k_msm_glv");
        k_msm_sort<false><<<grid_for(2 * ns[j], 256, sm_cap), 256, 0, st>>>(vsc + 2 * at, 0, 2 * ns[j], p.c, p.W,
                                                                              p.H, s.counts, nullptr, p.tn, j * p.H);
        H2B_LAUNCHED("k_msm_sort<hist>");
        at += ns[j];
    }
    H2B_CUDA(scan_u32(s.counts, p.NB, s.offsets, s.scan_tmp, st));
    H2B_CUDA(cudaMemcpyAsync(s.cursor, s.offsets, p.NB * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    at = 0;
    for (uint32_t j = 0; j < J; j++) {
        if (ns[j] == 0) continue;
        k_msm_sort<true><<<grid_for(2 * ns[j], 256, sm_cap), 256, 0, st>>>(vsc + 2 * at, 0, 2 * ns[j], p.c, p.W, p.H,
                                                                             s.cursor, s.sorted, p.tn, j * p.H);
        H2B_LAUNCHED("k_msm_sort<scatter>");
        at += ns[j];
    }
    prof_begin(PROF_MSM_ACCUMULATE, st);
    H2B_TRY(msm_accumulate(p, s, table, st));
    prof_end(PROF_MSM_ACCUMULATE, st);
    MsmOuts o;
    for (uint32_t j = 0; j < J; j++) o.p[j] = outs[j];
    H2B_TRY(msm_reduce(p, s, 1, 0, o, st));
    prof_end(PROF_MSM_TOTAL, st);
    return ok();
}

} // namespace h2b

using namespace h2b;

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------

static uint64_t msm_ws(uint64_t length, bool scalar_host, bool bases_host)
{
    MsmPlan p = msm_plan(length);
    ScratchPlan sp;
    msm_plan_scratch(p, sp, scalar_host, bases_host);
    return sp.used;
}

extern "C" uint64_t _halo2_msm_max_length(uint64_t free_bytes)
{
    for (int lg = 27; lg > 0; lg--) {
        if (msm_ws(1ull << lg, true, true) < free_bytes) return 1ull << lg;
    }
    return 0;
}

extern "C" uint64_t _halo2_multiexp_workspace_size(uint64_t length) { return msm_ws(length, true, true); }
extern "C" uint64_t _halo2_multiexp_device_bases_workspace_size(uint64_t length) { return msm_ws(length, true, false); }
extern "C" uint64_t _halo2_multiexp_device_scalars_device_bases_workspace_size(uint64_t length)
{
    return msm_ws(length, false, false);
}

static RustError msm_entry(const void* scalars, bool scalar_host, const void* bases, bool bases_host, void* h_out,
                           uint64_t length, void* scratch, uint64_t scratch_bytes, cudaStream_t st, const char* who)
{
    if (length > MSM_MAX_LENGTH) return err(cudaErrorInvalidValue, "MSM length above 2^27 points");
    MsmPlan p = msm_plan(length);
    uint64_t need = msm_ws(length, scalar_host, bases_host);
    if (scratch_bytes < need) return scratch_too_small(who, scratch_bytes, need);
    ScratchArena ar(scratch, scratch_bytes);
    MsmScratch s = msm_carve(p, ar, scalar_host, bases_host);
    if (!ar.good()) return scratch_too_small(who, scratch_bytes, need);
    const Fr* d_sc = (const Fr*)scalars;
    const G1Affine* d_b = (const G1Affine*)bases;
    if (length > 0 && bases_host) {
        H2B_CUDA(cudaMemcpyAsync(s.bases_stage, bases, length * sizeof(G1Affine), cudaMemcpyHostToDevice, st));
        d_b = s.bases_stage;
    }
    if (length >= MSM_PIPE_MIN && scalar_host) {
        // Host scalars arrive in MSM_PIPE_PIECES pieces on a forked copy stream;
        // the split and histogram of each piece run while the next one copies.
        cudaStream_t cs;
        H2B_TRY(h2b_exec_fork(st, 1, &cs));
        cudaEvent_t ev[MSM_PIPE_PIECES];
        for (int i = 0; i < MSM_PIPE_PIECES; i++) H2B_CUDA(cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming));
        RustError e = msm_begin(p, s, st);
        for (int i = 0; i < MSM_PIPE_PIECES && e.code == 0; i++) {
            const uint64_t lo = length * i / MSM_PIPE_PIECES, hi = length * (i + 1) / MSM_PIPE_PIECES;
            cudaError_t c = cudaMemcpyAsync(s.scalar_stage + lo, (const Fr*)scalars + lo, (hi - lo) * sizeof(Fr),
                                            cudaMemcpyHostToDevice, cs);
            if (c == cudaSuccess) c = cudaEventRecord(ev[i], cs);
            if (c == cudaSuccess) c = cudaStreamWaitEvent(st, ev[i], 0);
            e = c == cudaSuccess ? msm_split(p, s, s.scalar_stage, d_b, lo, hi, st) : cuda_err(c, who);
        }
        for (int i = 0; i < MSM_PIPE_PIECES; i++) cudaEventDestroy(ev[i]);
        H2B_TRY(e);
        H2B_TRY(msm_finish(p, s, d_b, st));
    } else {
        if (length > 0 && scalar_host) {
            H2B_CUDA(cudaMemcpyAsync(s.scalar_stage, scalars, length * sizeof(Fr), cudaMemcpyHostToDevice, st));
            d_sc = s.scalar_stage;
        }
        H2B_TRY(msm_run(p, s, d_sc, d_b, st));
    }
    H2B_CUDA(cudaMemcpyAsync(h_out, s.result, sizeof(G1Jac), cudaMemcpyDeviceToHost, st));
    H2B_CUDA(cudaStreamSynchronize(st));
    return ok();
}

extern "C" RustError _halo2_multiexp(const FFITraitObject* scalar, const FFITraitObject* point,
                                     const FFITraitObject* output, uint64_t length, void* scratch,
                                     uint64_t scratch_bytes, cudaStream_t stream)
{
    return msm_entry(scalar->ptr, true, point->ptr, true, output->ptr, length, scratch, scratch_bytes, stream,
                     "_halo2_multiexp");
}

extern "C" RustError _halo2_multiexp_device_bases(const FFITraitObject* h_scalar, const void* d_bases,
                                                  const FFITraitObject* h_output, uint64_t length, void* scratch,
                                                  uint64_t scratch_bytes, cudaStream_t stream)
{
    return msm_entry(h_scalar->ptr, true, d_bases, false, h_output->ptr, length, scratch, scratch_bytes, stream,
                     "_halo2_multiexp_device_bases");
}

extern "C" RustError _halo2_multiexp_device_scalars_device_bases(const void* d_scalar, const void* d_bases,
                                                                 const FFITraitObject* h_output, uint64_t length,
                                                                 void* scratch, uint64_t scratch_bytes,
                                                                 cudaStream_t stream)
{
    return msm_entry(d_scalar, false, d_bases, false, h_output->ptr, length, scratch, scratch_bytes, stream,
                     "_halo2_multiexp_device_scalars_device_bases");
}

// Device-output, sync-free variant: the 96-byte Jacobian image is written to
// d_out on `stream`.  Same scratch size as the device-scalars entry point.
extern "C" RustError h2b_msm_device(const void* d_scalar, const void* d_bases, void* d_out, uint64_t length,
                                    void* scratch, uint64_t scratch_bytes, cudaStream_t stream)
{
    if (length > MSM_MAX_LENGTH) return err(cudaErrorInvalidValue, "MSM length above 2^27 points");
    MsmPlan p = msm_plan(length);
    uint64_t need = msm_ws(length, false, false);
    if (scratch_bytes < need) return scratch_too_small("h2b_msm_device", scratch_bytes, need);
    ScratchArena ar(scratch, scratch_bytes);
    MsmScratch s = msm_carve(p, ar, false, false);
    H2B_TRY(msm_run(p, s, (const Fr*)d_scalar, (const G1Affine*)d_bases, stream));
    H2B_CUDA(cudaMemcpyAsync(d_out, s.result, sizeof(G1Jac), cudaMemcpyDeviceToDevice, stream));
    return ok();
}

// ---- precomputed window tables (SRS kept resident with its window multiples) --
// A table for n bases holds W slices of n affine points, slice w being
// [2^(c w)] P_i (c and W from the n-point plan).  An MSM over the table puts
// the digits of every window into one bucket set, so the bucket reduction
// covers one window and the final 2^(c w) doubling chain disappears; the
// entry count (bucket additions) is unchanged.  Slice w + 1 is c doublings of
// slice w, made affine with one batch inversion per slice.

namespace h2b {

__global__ void k_table_double(const G1Affine* __restrict__ prev, uint64_t n, int c, G1Xyzz* __restrict__ tmp,
                               Fq* __restrict__ den)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const G1Affine P = ld_affine(&prev[i]);
        if (is_inf(P)) {
            st_xyzz(&tmp[i], xyzz_inf());
            st(&den[i], Fq::zero());
            continue;
        }
        G1Xyzz X = xyzz_dbl_affine(P);
        for (int k = 1; k < c; k++) X = xyzz_dbl(X);
        st_xyzz(&tmp[i], X);
        st(&den[i], X.ZZ * X.ZZZ);
    }
}

// den_inv[i] = 1 / (ZZ ZZZ): x = X ZZZ / (ZZ ZZZ), y = Y ZZ / (ZZ ZZZ); zero -> infinity (0, 0).
__global__ void k_table_affine(const G1Xyzz* __restrict__ tmp, const Fq* __restrict__ den_inv, uint64_t n,
                               G1Affine* __restrict__ out)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const Fq d = ld(&den_inv[i]);
        G1Affine a;
        if (d.is_zero()) {
            a.x = Fq::zero();
            a.y = Fq::zero();
        } else {
            const G1Xyzz X = ld_xyzz(&tmp[i]);
            a.x = X.X * (d * X.ZZZ);
            a.y = X.Y * (d * X.ZZ);
        }
        st(&out[i].x, a.x);
        st(&out[i].y, a.y);
    }
}

// Layout of a window table for tn bases: the untuned window width, which
// msm_plan_table also uses, so tuning never changes a table's meaning.
static MsmPlan table_layout_plan(uint64_t tn) { return plan_core(tn, choose_c(tn), 0); }

// Entries encode the table point as 2 (w tn + i) + half in 31 bits.
static bool table_fits(uint64_t tn)
{
    const MsmPlan p = table_layout_plan(tn);
    return tn > 0 && tn <= MSM_MAX_LENGTH && 2 * (uint64_t)p.W * tn < (1ull << 31);
}

} // namespace h2b

// W window slices of n points, then the same W slices under phi (x -> beta x).
extern "C" uint64_t h2b_msm_table_points(uint64_t n)
{
    if (!table_fits(n)) return 0;
    return 2 * (uint64_t)table_layout_plan(n).W * n;
}

extern "C" uint64_t h2b_msm_table_precompute_workspace_size(uint64_t n)
{
    if (!table_fits(n)) return 0;
    ScratchPlan sp;
    sp.add_n<G1Xyzz>(n);
    sp.add_n<Fq>(n);
    sp.add(fq_batch_invert_scratch(n));
    return sp.used;
}

// d_table receives h2b_msm_table_points(n) affine points; d_bases is not modified.
extern "C" RustError h2b_msm_table_precompute(const void* d_bases, uint64_t n, void* d_table, void* scratch,
                                              uint64_t scratch_bytes, cudaStream_t stream)
{
    if (!table_fits(n)) return err(cudaErrorInvalidValue, "h2b_msm_table_precompute: n out of range");
    const MsmPlan p = table_layout_plan(n);
    ScratchArena ar(scratch, scratch_bytes);
    G1Xyzz* tmp = ar.take_n<G1Xyzz>(n);
    Fq* den = ar.take_n<Fq>(n);
    const uint64_t inv_bytes = fq_batch_invert_scratch(n);
    void* inv_scratch = ar.take(inv_bytes);
    if (!ar.good())
        return scratch_too_small("h2b_msm_table_precompute", scratch_bytes, h2b_msm_table_precompute_workspace_size(n));
    G1Affine* table = (G1Affine*)d_table;
    H2B_CUDA(cudaMemcpyAsync(table, d_bases, n * sizeof(G1Affine), cudaMemcpyDeviceToDevice, stream));
    for (int w = 1; w < p.W; w++) {
        k_table_double<<<grid_for(n, 128, 148u * 16u), 128, 0, stream>>>(table + (uint64_t)(w - 1) * n, n, p.c, tmp,
                                                                         den);
        H2B_LAUNCHED("k_table_double");
        H2B_TRY(fq_batch_invert(den, n, inv_scratch, inv_bytes, stream));
        k_table_affine<<<grid_for(n, 256), 256, 0, stream>>>(tmp, den, n, table + (uint64_t)w * n);
        H2B_LAUNCHED("k_table_affine");
    }
    // the accumulation reads the table in the lazy x 2^261 form, with the
    // phi images of all slices after them
    const uint64_t pts = (uint64_t)p.W * n;
    k_to_r261<<<grid_for(pts, 256, 148u * 8u), 256, 0, stream>>>(table, table, pts, table + pts);
    H2B_LAUNCHED("k_to_r261");
    return ok();
}

extern "C" uint64_t h2b_msm_table_workspace_size(uint64_t n, uint64_t table_n)
{
    if (n > table_n || !table_fits(table_n)) return 0;
    const MsmPlan p = msm_plan_table(n, table_n);
    ScratchPlan sp;
    msm_plan_scratch(p, sp, false, false);
    return sp.used;
}

// MSM of n <= table_n device scalars over a table built for table_n bases
// (its first n points of every slice are used); result to d_out (96 B, device).
extern "C" RustError h2b_msm_device_table(const void* d_scalars, const void* d_table, uint64_t table_n, void* d_out,
                                          uint64_t n, void* scratch, uint64_t scratch_bytes, cudaStream_t stream)
{
    if (n > table_n || !table_fits(table_n))
        return err(cudaErrorInvalidValue, "h2b_msm_device_table: n above the table size, or table size out of range");
    const MsmPlan p = msm_plan_table(n, table_n);
    const uint64_t need = h2b_msm_table_workspace_size(n, table_n);
    if (scratch_bytes < need) return scratch_too_small("h2b_msm_device_table", scratch_bytes, need);
    ScratchArena ar(scratch, scratch_bytes);
    MsmScratch s = msm_carve(p, ar, false, false);
    H2B_TRY(msm_run(p, s, (const Fr*)d_scalars, (const G1Affine*)d_table, stream));
    H2B_CUDA(cudaMemcpyAsync(d_out, s.result, sizeof(G1Jac), cudaMemcpyDeviceToDevice, stream));
    return ok();
}

extern "C" void h2b_msm_set_tuning(int window_bits, int chunk) { msm_set_tuning(window_bits, chunk); }

// Form of the bucket-accumulation kernel: 6 = coordinates in [0, 2p) on the
// even/odd product (default), 0 = the lazy R = 2^261 form of 29-bit limbs with
// one-step carries.  Measured at 2^22 with the witness-like scalar mix, the
// whole MSM: 6 7.57 ms, 0 13.6 ms.  Results are identical; only speed differs.
// Any other value leaves the setting unchanged (read it back with
// h2b_msm_get_accumulate_variant).
extern "C" void h2b_msm_set_accumulate_variant(int v)
{
    if (v == 0 || v == 6) g_msm_acc_variant = v;
}

extern "C" int h2b_msm_get_accumulate_variant(void) { return g_msm_acc_variant; }

// Distance (sorted entries ahead, 0..64) at which the accumulation
// prefetches the next points into L2; 0 turns it off.  Same results.
extern "C" void h2b_msm_set_prefetch(int distance)
{
    if (distance >= 0 && distance <= 64) g_msm_prefetch = (uint32_t)distance;
}
extern "C" int h2b_msm_get_prefetch(void) { return (int)g_msm_prefetch; }

// Batch-affine pairing rounds before the XYZZ accumulation are not built (0.5 ns
// per addition against 0.15 ns for an XYZZ mixed addition): the setting stays 0.
extern "C" int h2b_msm_get_pair_rounds(void) { return 0; }
extern "C" void h2b_msm_set_pair_rounds(int) {}

// Number of nonzero signed window digits (= sorted entries = bucket
// additions) the MSM of these scalars performs; written to *d_count (u64).
// Used by the benchmark for its algorithmic work count, untimed.
namespace h2b {
__global__ void k_msm_count(const Fr* __restrict__ sc, uint64_t n, int c, int W, uint32_t H,
                            unsigned long long* __restrict__ cnt)
{
    unsigned long long local = 0;
    const uint32_t full = 1u << c;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint4 half[2];
        glv::decompose(from_mont(ldg(&sc[i])), half[0], half[1]);
        for (int h = 0; h < 2; h++) {
            uint32_t carry = 0;
            for (int w = 0; w < W; w++) {
                uint32_t v = window_bits(half[h], w * c, c) + carry;
                int32_t d = (v > H) ? (int32_t)v - (int32_t)full : (int32_t)v;
                carry = (v > H) ? 1u : 0u;
                if (d != 0) local++;
            }
        }
    }
    atomicAdd(cnt, local);
}
} // namespace h2b

extern "C" RustError h2b_msm_count_entries(const void* d_scalars, uint64_t n, void* d_count, cudaStream_t stream)
{
    MsmPlan p = msm_plan(n);
    H2B_CUDA(cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), stream));
    if (n == 0) return ok();
    k_msm_count<<<grid_for(n, 256, 148u * 8u), 256, 0, stream>>>((const Fr*)d_scalars, n, p.c, p.W, p.H,
                                                                (unsigned long long*)d_count);
    H2B_LAUNCHED("k_msm_count");
    return ok();
}

extern "C" int h2b_msm_window_bits(uint64_t n) { return msm_plan(n).c; }
