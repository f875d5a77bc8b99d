// Neighbour-of-neighbour pass: SolutionKmeans::topUpSingle
// (src/SolutionKmeans.hpp:480-555).
//
// Snapshot: every set's k slot ids, sorted ascending, unfilled slots included
// (as the point set's first id, 0 for a single set) -- the reference reads all
// 100 current_ids (:494).  Per point p, the candidates are the union of the
// snapshot lists of p's snapshot list, minus p, each offered with the exact
// distance when dist < bound.
//
// The reference iterates its candidate set in hash order; this pass offers
// them in ascending id order.  The order can only matter between candidates
// that beat the bound p had when its pass started, so the pass collects every
// such survivor (dist < starting bound), sorts each point's survivors by id and
// replays them in that order through the sequential set update.
//
// Two ways to collect the survivors, with the same result:
//   * the local join (k_join, the default): per point q, the rows R(q) (points
//     whose list holds q) against the columns S(q) (q's list) as one block; a
//     tcgen05 tile of centred dot products (FP16 operands, FP32 accumulation)
//     rules out the pairs that provably cannot beat bound(p) and leaves, per
//     edge p -> q, the bits of the columns that may; k_apply then takes p's
//     candidates from its lists' bits, drops members and repeats, computes the
//     exact FP32 distances, sorts and replays;
//   * one warp per point (k_refine): the warp walks its candidates (one lane per
//     candidate, rows gathered from HBM/L2) with a shared-memory seen-set, keeps
//     the survivors in shared memory (or a per-warp global region of k*k
//     entries) and replays them.  It serves as the cross-check of the join
//     (environment KNNG_REFINE=pointwise), as the pass for points with more
//     candidates than a CTA's tables hold, where the budget has no room for the
//     join's bits, and behind the allocation-free entry point.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "context.hpp"
#include "dispatch.hpp"
#include "tc.cuh"
#include "tile16.cuh"

namespace knng {
namespace {

constexpr int kSnapWarps = 8;
constexpr int kRefWarps = 4;
constexpr int kSurvCap = 256;

constexpr int kSeenSlots = 2048;  // per-warp open-addressing set of candidate ids
constexpr int kSeenProbes = 32;

// Inserts id into the warp's seen-set; true if it was not there.  When the
// probe limit is reached the id is reported new: a repeated offer is harmless
// (the set update rejects it), only slower.
__device__ __forceinline__ bool seen_insert(uint32_t* seen, uint32_t id) {
    uint32_t h = (id * 0x9E3779B1u) >> (32 - 11);
    for (int probe = 0; probe < kSeenProbes; ++probe) {
        const uint32_t prev = atomicCAS(&seen[h], kNone, id);
        if (prev == kNone) return true;
        if (prev == id) return false;
        h = (h + 1) & (kSeenSlots - 1);
    }
    return true;
}

__host__ __device__ uint32_t pow2_at_least(uint32_t v) {
    uint32_t p = 2;
    while (p < v) p <<= 1;
    return p;
}

// Words of a point's old-entry mask (one bit per snapshot entry).
constexpr int kOldWords = kMaxK / kWarp;  // 4

// Each point's sorted list of its set's k slot ids.  With `snap_d` also the
// distance of each entry (NaN for an empty slot's).  With `prev` (the sorted
// lists of the previous pass) also old[p * kOldWords + i / 32] bit i % 32 =
// entry i of the new list is in the point's previous list.
//
// A warp per point sorts (id, slot) in registers, four entries a lane, so that
// an entry's slot tells its distance and, of equal ids, a member comes before
// the empty slots.  Bound by the network's shuffles, not by memory (3.2 GB a
// pass at 2,000,000 points): in shared memory, with each distance's place found
// by bisection, a pass took 4.1 ms; in registers 3.9 with 64-bit keys, 2.4 with
// 32-bit ones.
//
// Key is a 64-bit id << 32 | slot, or for ids below kShortIds a 32-bit id << 7 |
// slot (one shuffle, minimum and maximum an exchange in place of two shuffles
// and a pair of compares and selects).
constexpr uint32_t kShortIds = 1u << 25;
template <class Key>
__global__ void __launch_bounds__(kSnapWarps * kWarp)
    k_snapshot(const uint32_t* __restrict__ set_id, const float* __restrict__ set_dist,
               const uint32_t* __restrict__ set_size, uint32_t n, int K, uint32_t* __restrict__ snap,
               float* __restrict__ snap_d, const uint32_t* __restrict__ prev, uint32_t* __restrict__ old) {
    __shared__ uint32_t prev_s[kSnapWarps][kMaxK];
    __shared__ float dist_s[kSnapWarps][kMaxK];
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    constexpr int kShift = sizeof(Key) == 8 ? 32 : 7;
    static_assert(kMaxK <= 1 << 7, "a slot takes seven bits");
    uint32_t* pl = prev_s[warp];
    float* dl = dist_s[warp];
    int top = 1;  // largest power of two <= K (branch-free lower bound)
    while (top * 2 <= K) top *= 2;
    for (uint32_t p = blockIdx.x * kSnapWarps + warp; p < n; p += gridDim.x * kSnapWarps) {
        const size_t base = static_cast<size_t>(p) * K;
        Key key[kSlotsPerLane];
        const int size = snap_d ? static_cast<int>(set_size[p]) : 0;
#pragma unroll
        for (int r = 0; r < kSlotsPerLane; ++r) {
            const int slot = r * kWarp + lane;
            key[r] = slot < K ? (static_cast<Key>(set_id[base + slot]) << kShift) | static_cast<Key>(slot) : ~Key(0);
            if (snap_d) dl[slot] = slot < size ? set_dist[base + slot] : __int_as_float(0x7fc00000);
            if (prev && slot < K) pl[slot] = prev[base + slot];
        }
        warp_sort_lanes<kSlotsPerLane>(key, lane);
        uint32_t id[kSlotsPerLane];
#pragma unroll
        for (int r = 0; r < kSlotsPerLane; ++r) id[r] = static_cast<uint32_t>(key[r] >> kShift);
        store_lane_run(snap + base, K, lane, id);
        __syncwarp();
        if (snap_d) {
            float dist[kSlotsPerLane];
#pragma unroll
            for (int r = 0; r < kSlotsPerLane; ++r) dist[r] = dl[static_cast<uint32_t>(key[r]) & (kMaxK - 1)];
            store_lane_run(snap_d + base, K, lane, dist);
        }
        if (prev) {
            uint32_t bits = 0;  // of the eight lanes that hold a word's entries
#pragma unroll
            for (int r = 0; r < kSlotsPerLane; ++r) {
                int pos = 0;  // first entry of the previous list >= id
                for (int step = top; step > 0; step >>= 1)
                    if (pos + step <= K && pl[pos + step - 1] < id[r]) pos += step;
                const int i = kSlotsPerLane * lane + r;
                if (i < K && pos < K && pl[pos] == id[r]) bits |= 1u << (i % kWarp);
            }
#pragma unroll
            for (int j = 1; j < kWarp / kSlotsPerLane; j <<= 1) bits |= __shfl_xor_sync(kFull, bits, j);
            if (lane % (kWarp / kSlotsPerLane) == 0)
                old[static_cast<size_t>(p) * kOldWords + lane / (kWarp / kSlotsPerLane)] = bits;
        }
        __syncwarp();
    }
}

template <int D>
__global__ void __launch_bounds__(kRefWarps * kWarp)
    k_refine(const uint32_t* __restrict__ snap, const float* __restrict__ pts, int ld, float* __restrict__ set_dist,
             uint32_t* __restrict__ set_id, uint32_t* __restrict__ set_size, uint32_t* __restrict__ set_maxslot,
             float* __restrict__ set_bound, int K, uint32_t n, const uint32_t* __restrict__ plist, uint32_t first,
             unsigned long long* __restrict__ scratch_keys, uint32_t warp_capacity,
             uint32_t* __restrict__ changed_count) {
    constexpr int Q = D / 4;
    __shared__ float4 rowp_s[kRefWarps][Q];
    __shared__ unsigned long long surv_s[kRefWarps][kSurvCap];
    __shared__ uint32_t seen_s[kRefWarps][kSeenSlots];
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    const uint32_t gw = blockIdx.x * kRefWarps + warp;
    const uint32_t nw = gridDim.x * kRefWarps;
    unsigned long long* gbuf = scratch_keys + static_cast<size_t>(gw) * warp_capacity;
    const unsigned lt_mask = (1u << lane) - 1u;
    for (uint32_t w = gw; w < n; w += nw) {
        const uint32_t p = plist ? plist[w] : first + w;
        for (int q = lane; q < Q; q += kWarp)
            rowp_s[warp][q] = __ldg(reinterpret_cast<const float4*>(pts + static_cast<size_t>(p) * ld) + q);
        WarpSet s;
        set_load(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
        // Seen-set: p itself and p's current members are pre-inserted, so
        // candidates that could only be rejected (self, already a member, or a
        // repeat from another list) skip the row gather and the distance.
        uint32_t* seen = seen_s[warp];
        for (int t = lane; t < kSeenSlots; t += kWarp) seen[t] = kNone;
        __syncwarp();
        if (lane == 0) seen_insert(seen, p);
#pragma unroll
        for (int r = 0; r < kSlotsPerLane; ++r)
            if (lane + r * kWarp < static_cast<int>(s.size)) seen_insert(seen, s.id[r]);
        __syncwarp();
        const float bound0 = s.bound;
        uint32_t S = 0;
        uint32_t prev_q = kNone;
        const uint32_t* mine = snap + static_cast<size_t>(p) * K;
        for (int a = 0; a < K; ++a) {
            const uint32_t q = mine[a];
            if (q == prev_q) continue;  // the list is sorted: repeats are adjacent
            prev_q = q;
            const uint32_t* theirs = snap + static_cast<size_t>(q) * K;
            for (int b0 = 0; b0 < K; b0 += kWarp) {
                const int bb = b0 + lane;
                const uint32_t c = bb < K ? theirs[bb] : p;
                const bool valid = c != p && seen_insert(seen, c);
                float d = 0.0f;
                if (valid)
                    d = canonical_distance4<D>(reinterpret_cast<const float4*>(pts + static_cast<size_t>(c) * ld),
                                               rowp_s[warp]);
                const bool pass = valid && d < bound0;
                const unsigned m = __ballot_sync(kFull, pass);
                if (pass) gbuf[S + __popc(m & lt_mask)] = (static_cast<unsigned long long>(c) << 32) | __float_as_uint(d);
                S += __popc(m);
            }
        }
        __syncwarp();
        // Sort the survivors by (id, dist); equal ids carry equal distances.
        const uint32_t P2 = pow2_at_least(S);
        unsigned long long* buf = gbuf;
        if (P2 <= kSurvCap) {
            buf = surv_s[warp];
            for (uint32_t t = lane; t < P2; t += kWarp) buf[t] = t < S ? gbuf[t] : ~0ull;
        } else {
            for (uint32_t t = S + lane; t < P2; t += kWarp) buf[t] = ~0ull;
        }
        __syncwarp();
        if (S > 1) warp_bitonic_sort(buf, P2, lane);
        uint32_t changed = 0;
        for (uint32_t t0 = 0; t0 < S; t0 += kWarp) {
            const uint32_t t = t0 + lane;
            const unsigned long long key = t < S ? buf[t] : ~0ull;
            const unsigned long long prev = (t > 0 && t < S) ? buf[t - 1] : ~0ull;
            const uint32_t cid = static_cast<uint32_t>(key >> 32);
            const float d = __uint_as_float(static_cast<uint32_t>(key & 0xFFFFFFFFu));
            const bool valid = t < S && (t == 0 || static_cast<uint32_t>(prev >> 32) != cid);
            changed += set_offer_batch(s, cid, d, valid, K, lane);
        }
        set_store(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
        if (changed && lane == 0) atomicAdd(changed_count, 1u);
        __syncwarp();
    }
}

// ------------------------------------------------------------ local join
//
// The same pass, reorganised around the shared point q: p's candidates are
// the lists S(q) of every q in S(p), so for each q the block
// R(q) x S(q) (R(q) = the points whose list holds q) carries every candidate
// pair that goes through q.  Each block reads |R(q)| + |S(q)| rows instead of
// one row per (p, candidate), and its dot products run on the tensor cores:
//
//   1. k_rev_count / scan / k_rev_fill   R(q) as a CSR (counting sort; the
//                 points visited in leaf order so that the scattered writes
//                 meet in L2) of edges: (p, position of q in p's list).  After a
//                 first pass, an entry whose edge was already in p's previous
//                 list carries bit 31.
//   2. k_join     three persistent CTAs per SM take the points q in leaf order
//                 and write, per edge p -> q, the bits of q's list entries that
//                 may beat bound(p): a tcgen05 tile of centred dot products
//                 rules the others out by a proven error bound.
//   3. k_apply    per p: the entries left of its K lists, minus p's members and
//                 repeats, get the exact FP32 distance; survivors are sorted by
//                 id and replayed through the sequential set update in ascending
//                 id order -- the same offers, in the same order, as the
//                 per-point pass (one warp up to 800 candidates, k_apply_big up
//                 to 8,192).
//   Points with more candidates are redone by k_refine.  When the budget has no
//   room for every edge's bits, the pass goes over ranges of points p (1 to 3
//   for each range; the snapshot, and so the result, is the same).

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int kScanTile = kScanThreads * kScanPer;

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const uint32_t* __restrict__ in, uint64_t n,
                                                              unsigned long long* __restrict__ tile_sum) {
    __shared__ unsigned long long ws[kScanThreads / kWarp];
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanPer;
    unsigned long long s = 0;
#pragma unroll
    for (int u = 0; u < kScanPer; ++u)
        if (base + u < n) s += in[base + u];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    if (threadIdx.x % kWarp == 0) ws[threadIdx.x / kWarp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < kScanThreads / kWarp; ++w) t += ws[w];
        tile_sum[blockIdx.x] = t;
    }
}

// Exclusive scan of the tile sums in place (one CTA; by warps, where one thread
// adding the 1,024 partial sums took 7.7 us of its launch, now 2.4).
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(unsigned long long* __restrict__ tile_sum, uint32_t nt) {
    __shared__ unsigned long long ws[kScanThreads / kWarp];
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    const uint32_t per = (nt + kScanThreads - 1) / kScanThreads;
    const uint32_t b = threadIdx.x * per, e = min(nt, b + per);
    unsigned long long s = 0;
    for (uint32_t i = b; i < e; ++i) s += tile_sum[i];
    unsigned long long incl = s;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == kWarp - 1) ws[warp] = incl;
    __syncthreads();
    unsigned long long run = incl - s;
    for (int w = 0; w < warp; ++w) run += ws[w];
    for (uint32_t i = b; i < e; ++i) {
        const unsigned long long v = tile_sum[i];
        tile_sum[i] = run;
        run += v;
    }
}

// out[i] = sum of in[0..i); out[n] = total.
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const uint32_t* __restrict__ in, uint64_t n,
                                                             const unsigned long long* __restrict__ tile_off,
                                                             unsigned long long* __restrict__ out) {
    __shared__ unsigned long long ws[kScanThreads / kWarp];
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanPer;
    uint32_t v[kScanPer];
    unsigned long long mine = 0;
#pragma unroll
    for (int u = 0; u < kScanPer; ++u) {
        v[u] = base + u < n ? in[base + u] : 0u;
        mine += v[u];
    }
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == kWarp - 1) ws[warp] = incl;
    __syncthreads();
    unsigned long long wbase = 0;
    for (int w = 0; w < warp; ++w) wbase += ws[w];
    unsigned long long run = tile_off[blockIdx.x] + wbase + incl - mine;
#pragma unroll
    for (int u = 0; u < kScanPer; ++u) {
        if (base + u < n) out[base + u] = run;
        run += v[u];
        if (base + u + 1 == n) out[n] = run;
    }
}

// One warp per point p of [lo, hi): every distinct q of S(p) counts / receives
// the edge p -> q.
__global__ void k_rev_count(const uint32_t* __restrict__ snap, uint32_t lo, uint32_t hi, int K,
                            uint32_t* __restrict__ cnt) {
    const int lane = threadIdx.x % kWarp;
    for (uint32_t p = lo + (blockIdx.x * blockDim.x + threadIdx.x) / kWarp; p < hi;
         p += gridDim.x * blockDim.x / kWarp) {
        const uint32_t* row = snap + static_cast<size_t>(p) * K;
        for (int a = lane; a < K; a += kWarp) {
            const uint32_t q = row[a];
            if (a == 0 || row[a - 1] != q) atomicAdd(&cnt[q], 1u);
        }
    }
}

// Bit 31 of a reverse-list entry: the edge p -> q was already in p's list of
// the previous pass (edge numbers are below 2^31).
constexpr uint32_t kOldEdge = 0x80000000u;

// Points are visited in `order` when given (the last repetition's leaf
// order): neighbouring points fill the same reverse lists close in time, so
// their 4-byte writes meet in L2 instead of each moving a DRAM sector.
__global__ void k_rev_fill(const uint32_t* __restrict__ snap, uint32_t n, uint32_t lo, uint32_t hi, int K,
                           const unsigned long long* __restrict__ off, uint32_t* __restrict__ cursor,
                           uint32_t* __restrict__ rev, const uint32_t* __restrict__ old,
                           const uint32_t* __restrict__ order) {
    const int lane = threadIdx.x % kWarp;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp; w < n; w += gridDim.x * blockDim.x / kWarp) {
        const uint32_t p = order ? order[w] : w;
        if (p < lo || p >= hi) continue;
        const uint32_t* row = snap + static_cast<size_t>(p) * K;
        // A lane's edges together: their lookups overlap (2,000,000 x 100 edges: 5.4 ms
        // one after the other, 4.7 so).
        uint32_t q[kSlotsPerLane], at[kSlotsPerLane];
        unsigned long long first[kSlotsPerLane];
        bool has[kSlotsPerLane];
#pragma unroll
        for (int r = 0; r < kSlotsPerLane; ++r) {
            const int a = r * kWarp + lane;
            q[r] = a < K ? row[a] : 0u;
            has[r] = a < K && (a == 0 || row[a - 1] != q[r]);
        }
#pragma unroll
        for (int r = 0; r < kSlotsPerLane; ++r) {
            if (!has[r]) continue;
            at[r] = atomicAdd(&cursor[q[r]], 1u);
            first[r] = off[q[r]];
        }
#pragma unroll
        for (int r = 0; r < kSlotsPerLane; ++r) {
            if (!has[r]) continue;
            const int a = r * kWarp + lane;
            const bool was = old && ((old[static_cast<size_t>(p) * kOldWords + r] >> lane) & 1u);
            rev[first[r] + at[r]] = ((p - lo) * static_cast<uint32_t>(K) + a) | (was ? kOldEdge : 0u);
        }
    }
}

constexpr int kJoinThreads = 256;
constexpr int kJoinWarps = kJoinThreads / kWarp;  // 8
constexpr int kJoinPerSm = 3;                     // CTAs per SM: one's waits overlap the others' work
constexpr int kTile = 128;                        // MMA M: rows of R(q) per chunk
constexpr int kGroupCols = 64;                    // columns one thread filters (2 groups of 64)
constexpr uint32_t kJoinBatch = 4;                // points a CTA takes from the work counter at a time

// Columns of the B tile: the MMA takes N in steps of 16.
__host__ __device__ constexpr uint32_t join_cols(uint32_t K) { return K <= 16 ? 16u : (K + 15) / 16 * 16; }

__host__ __device__ inline uint32_t join_smem(int D, uint32_t K) {
    const uint32_t chunks = (static_cast<uint32_t>(D) + 15) / 16 * 2;
    return chunks * (kTile * 16 + 16) + chunks * (join_cols(K) * 16 + 16);
}

// The filter's error terms.  A pair is left out only when
//   approx - margin >= bound(p),  approx = |x'|^2 + |y'|^2 - 2 x'.y',
//   margin = (2^-8 + 2^-14) (|x'|^2 + |y'|^2) + 2^-19 (|x'| + |y'|) + 2^-20 bound(p)
// (x', y' the rows centred on q, their dot product from FP16 operands).  The
// margin covers FP16 rounding of both operands (2^-11 relative, 2^-25 absolute
// in the subnormal range), FP32 accumulation, the rounding of the centring, of
// the squared norms (the edges' own FP32 distances) and of the reference's
// summation, and the rounding of the test itself, which compares the
// accumulator with a sum of a row's term and a column's:
//   left out  <=>  half_gap(row) - bound(p) / 2 + half_gap(column) >= x'.y'.
constexpr float kNormKeep = 1.0f - 0.00390625f - 6.103515625e-05f;
__device__ __forceinline__ float half_gap(float norm) {
    return 0.5f * (norm * kNormKeep - 1.9073486328125e-06f * sqrtf(norm));
}
// Squared norms from which a value might not fit FP16 (or that are no number):
// the filter keeps every pair of such a row or column.
__device__ __forceinline__ bool norm_unfit(float norm) { return !(norm < 1.0e9f); }

// The local join of one neighbour-of-neighbour pass, for the points p in
// [lo, lo + range).  For every point q (taken in `order`, the last
// repetition's leaf order, through the work counter): the rows R(q) (points of
// the range whose snapshot list holds q), in chunks of 128, against the columns
// S(q) (q's snapshot list, by position).  masks[e] of the edge e = (p - lo) K +
// (position of q in p's list) receives the columns that p has to look at: all
// but those whose distance certainly is at least bound(p), the repeats in an
// unfilled list, and (with `old_marks`) the pairs whose two edges were both in
// the previous pass's lists.
//
// Per chunk: every warp reads its rows of R(q) (and, for a new q, of S(q))
// straight into centred FP16 tiles; one thread issues the tcgen05.mma
// (kind::f16, FP32 accumulate) into TMEM; every thread compares 64 accumulator
// columns of its TMEM lane with the sum of its row's and the columns' terms and
// writes the comparison bits.  One barrier a chunk.  The squared norms are the
// edges' own distances, kept with the snapshot.
//
// What bounds it: the rows (800 bytes a member of S(q) and R(q), mostly L2
// hits) and the latency of a q's dependent steps (point, list, rows, product),
// which three CTAs an SM overlap.  Everything that needs a pair one at a time
// -- members, repeats, exact distances -- is the replay's, where p's own list
// is at hand and a candidate reached through several q is met once.  Doing it
// here took per q 100 staged lists and 200 staged rows (bulk copies, about 70
// cycles each) and an exact distance for every repeat: 495 ms for the two passes
// of a 2M x 100 build and 14.9 ms for the one of a 100k build, now 107 and 2.5.
template <int D>
__global__ void __launch_bounds__(kJoinThreads, kJoinPerSm)
    k_join(const uint32_t* __restrict__ snap, const float* __restrict__ snap_d,
           const unsigned long long* __restrict__ rev_off, const uint32_t* __restrict__ rev,
           const float* __restrict__ pts, int ld, const float* __restrict__ bound, uint32_t K, uint32_t n, uint32_t lo,
           uint2* __restrict__ masks, uint32_t* __restrict__ error_flag, unsigned long long* __restrict__ counters,
           const uint32_t* __restrict__ order, uint32_t* __restrict__ work, const uint32_t* __restrict__ old_marks) {
    using T = Tile16<D>;
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t NB = join_cols(K);
    unsigned char* tile_a = smem;
    unsigned char* tile_b = smem + T::bytes(kTile);
    __shared__ __align__(16) float col_s[2][kTile];  // half_gap of the columns (two q in flight at most)
    __shared__ uint32_t valid_s[2][kOldWords], unfit_s[2][kOldWords];
    __shared__ uint64_t mma_bar;
    __shared__ uint32_t tmem_slot, failed_s, work_s[2];
    const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
    // The tiles' padding (dimensions past D) stays zero; rows past a chunk's
    // count hold earlier rows, whose products nobody reads.
    for (uint32_t f = tid; f < (T::bytes(kTile) + T::bytes(NB)) / 16; f += kJoinThreads)
        reinterpret_cast<uint4*>(smem)[f] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) tc::tmem_alloc(&tmem_slot, kTile);
    if (tid == 0) {
        failed_s = 0;
        tc::mbar_init(&mma_bar, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = tc::idesc_f16(kTile, NB);
    const int quarter = warp % 4, group = warp / 4;
    const int row = quarter * kWarp + lane;  // TMEM lane / tile row this thread filters
    const uint32_t piece = lane % T::Q;
    uint32_t phase = 0, buf = 0;
    unsigned long long n_pairs = 0, n_pass = 0;
    for (uint32_t it = 0;; ++it) {
        if (tid == 0) work_s[it & 1u] = atomicAdd(work, kJoinBatch);
        __syncthreads();
        const uint32_t base = work_s[it & 1u];
        if (failed_s || base >= n) break;
        uint32_t qs = 0;
        unsigned long long rbs = 0, res = 0;
        if (lane < kJoinBatch && base + lane < n) {
            qs = order ? order[base + lane] : base + lane;
            rbs = rev_off[qs];
            res = rev_off[qs + 1];
        }
        for (uint32_t i = 0; i < kJoinBatch; ++i) {
            const uint32_t q = __shfl_sync(kFull, qs, i);
            const unsigned long long rb = __shfl_sync(kFull, rbs, i), re = __shfl_sync(kFull, res, i);
            if (rb == re) continue;
            buf ^= 1u;
            const size_t sq = static_cast<size_t>(q) * K;
            const float4 centre = __ldg(reinterpret_cast<const float4*>(pts + static_cast<size_t>(q) * ld) + piece);
            for (unsigned long long cb = rb; cb < re; cb += kTile) {
                const uint32_t m = static_cast<uint32_t>(min(static_cast<unsigned long long>(kTile), re - cb));
                // Point of tile row lane * 8 + warp (lanes below 16), and this
                // thread's filter row with its term.
                const uint32_t mine = lane * kJoinWarps + warp;
                const uint32_t a_id =
                    lane < kTile / kJoinWarps && mine < m ? lo + (rev[cb + mine] & ~kOldEdge) / K : 0u;
                const bool live = row < static_cast<int>(m);
                const uint32_t edge = live ? rev[cb + row] : 0u;
                const uint32_t e = edge & ~kOldEdge;
                float na = 0.0f, bp = 0.0f;
                if (live) {
                    na = snap_d[static_cast<size_t>(lo) * K + e];
                    bp = bound[lo + e / K];
                }
                tile_rows<D, kTile, kJoinWarps, __half>(pts, ld, a_id, m, tile_a, T::stride(kTile), centre, lane, warp);
                if (cb == rb) {  // uniform over the CTA
                    const uint32_t b_id = lane < kTile / kJoinWarps && mine < K ? snap[sq + mine] : 0u;
                    tile_rows<D, kTile, kJoinWarps, __half>(pts, ld, b_id, K, tile_b, T::stride(NB), centre, lane, warp);
                    if (warp < kOldWords) {
                        const uint32_t c = tid;  // column
                        const bool in = c < K;
                        const uint32_t id = in ? snap[sq + c] : 0u;
                        const float nb = in ? snap_d[sq + c] : 0.0f;
                        // Repeats: the empty slots of an unfilled set.
                        const bool valid = in && (c == 0 || snap[sq + c - 1] != id);
                        const bool unfit = norm_unfit(nb);
                        col_s[buf][c] = unfit ? 0.0f : half_gap(nb);
                        const unsigned bv = __ballot_sync(kFull, valid), bu = __ballot_sync(kFull, valid && unfit);
                        if (lane == 0) {
                            valid_s[buf][warp] = bv;
                            unfit_s[buf][warp] = bu;
                        }
                    }
                }
                tc::fence_proxy_async();
                tc::fence_before_sync();
                __syncthreads();
                if (tid == 0) {
                    tc::fence_after_sync();
                    tc::issue_tile_strided(tmem, tc::smem_u32(tile_a), tc::smem_u32(tile_b), T::stride(kTile),
                                           T::stride(NB), T::KP, idesc);
                    tc::mma_commit(&mma_bar);
                }
                if (!tc::mbar_wait_limited(&mma_bar, phase)) {
                    // Recorded; the launch ends at the next batch, after this
                    // product has had the full limit to complete.
                    atomicExch(error_flag, 1u);
                    failed_s = 1u;
                    tc::mbar_wait(&mma_bar, phase);
                }
                __syncwarp();
                phase ^= 1u;
                tc::fence_after_sync();
                const bool keep_all = norm_unfit(na) || !(bp == bp);
                const float gap = half_gap(na) - 0.5f * (bp + 9.5367431640625e-07f * bp);
                uint32_t word[2] = {0u, 0u};
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const int c0 = group * kGroupCols + w * kWarp;
                    if (c0 >= static_cast<int>(NB)) break;  // warp-uniform
                    const uint32_t at = tmem + (static_cast<uint32_t>(quarter * kWarp) << 16) + c0;
                    uint32_t bits = 0;
#pragma unroll
                    for (int h = 1; h >= 0; --h) {
                        if (c0 + 16 * h >= static_cast<int>(NB)) continue;  // warp-uniform
                        float g[16];
                        tc::tmem_ld16(at + 16 * h, g);
                        const float4* cs = reinterpret_cast<const float4*>(&col_s[buf][c0 + 16 * h]);
                        float t[16];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float4 c = cs[u];
                            t[4 * u + 0] = gap + c.x;
                            t[4 * u + 1] = gap + c.y;
                            t[4 * u + 2] = gap + c.z;
                            t[4 * u + 3] = gap + c.w;
                        }
                        tc::tmem_wait_ld();
                        // The sign of (row's term + column's term) - product, highest column first.
#pragma unroll
                        for (int u = 15; u >= 0; --u)
                            bits = __funnelshift_l(__float_as_uint(t[u] - g[u]), bits, 1);
                    }
                    const uint32_t valid = valid_s[buf][c0 / kWarp];
                    bits = keep_all ? valid : (bits | unfit_s[buf][c0 / kWarp]) & valid;
                    // A pair whose two edges (p -> q and q -> c) were both in the
                    // previous pass's lists was offered then: every offer of it
                    // now is rejected (c is in S(p), or at least as far as a
                    // bound that has only fallen since).
                    if (old_marks && (edge & kOldEdge)) bits &= ~old_marks[static_cast<size_t>(q) * kOldWords + c0 / kWarp];
                    word[w] = bits;
                    if (live) n_pairs += __popc(valid);
                }
                if (live) {
                    n_pass += __popc(word[0]) + __popc(word[1]);
                    masks[static_cast<size_t>(e) * 2 + group] = make_uint2(word[0], word[1]);
                }
                // The accumulator is read before the next chunk's product.
                tc::fence_before_sync();
            }
        }
    }
    atomicAdd(&counters[0], n_pairs);
    atomicAdd(&counters[1], n_pass);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, kTile);
    }
}

// ---------------------------------------------------------------- replay
//
// Per point p: the columns that the join left of each of p's K lists, minus
// p's members and the repeats (a hash set in shared memory), are sorted by id and
// offered in that order with their exact FP32 distances -- the offers of the
// per-point pass, in its order.  One warp per point up to kWarpCands candidates, then
// one CTA up to kCtaCands, then the per-point pass.

constexpr int kApplyWarps = 5;
constexpr int kApplyPerSm = 4;
constexpr uint32_t kWarpCands = 800;    // candidates of a point that one warp handles
constexpr uint32_t kWarpTable = 1024;   // its hash slots (members, p, candidates and what a step adds past the cap)
constexpr uint32_t kWarpList = 1024;    // mask bits expanded at a time
constexpr int kBigThreads = 256;
constexpr uint32_t kCtaCands = 8192;
constexpr uint32_t kCtaTable = 16384;

// Inserts id (below 2^31) into a table of `buckets` (a power of two) buckets of
// four ids, never full; `mark` (kMember or 0) goes in with it.  Returns the mark
// it was found with, or kFresh.  A bucket is one 16-byte load and fills from its
// front, so nearly every id -- most are there already -- takes one step (with
// single slots a warp waited for its longest probe chain).
constexpr uint32_t kMember = 0x80000000u;
constexpr uint32_t kFresh = 1u;
__device__ __forceinline__ uint32_t table_insert(uint32_t* table, uint32_t buckets, uint32_t id, uint32_t mark) {
    uint32_t h = (id * 0x9E3779B1u) >> (__clz(buckets) + 1);
    for (uint32_t probe = 0; probe < 8 * buckets; ++probe) {
        uint4 v;
        asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(tc::smem_u32(table + 4 * h))
                     : "memory");
        uint32_t hit = kFresh;  // the entry found, without its id's bits
        hit = ((v.x ^ id) & ~kMember) == 0 ? v.x & kMember : hit;
        hit = ((v.y ^ id) & ~kMember) == 0 ? v.y & kMember : hit;
        hit = ((v.z ^ id) & ~kMember) == 0 ? v.z & kMember : hit;
        hit = ((v.w ^ id) & ~kMember) == 0 ? v.w & kMember : hit;
        if (hit != kFresh) return hit;
        if (v.w == kNone) {
            const uint32_t slot = v.x == kNone ? 0u : v.y == kNone ? 1u : v.z == kNone ? 2u : 3u;
            if (atomicCAS(&table[4 * h + slot], kNone, id | mark) == kNone) return kFresh;
            // Another lane took the slot: the bucket is read again.
        } else {
            h = (h + 1) & (buckets - 1);
        }
    }
    return 0u;
}

// canonical_distance4 of two rows held by the eight lanes of the group whose
// first lane is g0; every lane of the group returns it.  All 32 lanes call it.
template <int D>
__device__ __forceinline__ float group_distance(const ChainRow<D>& a, const ChainRow<D>& b, int g0) {
    constexpr int M = ChainRow<D>::M;
    static_assert(D - M == 0 || D - M == 4, "tail of 0 or 4 dims");
    float chain = 0.0f;
#pragma unroll
    for (int i = 0; i < M / 8; ++i) {
        const float d = __fsub_rn(a.c[i], b.c[i]);
        chain = __fmaf_rn(d, d, chain);
    }
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = __fadd_rn(acc, __shfl_sync(kFull, chain, g0 + j));
    if constexpr (D > M) {
        float d = __fsub_rn(a.tail.x, b.tail.x);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
        d = __fsub_rn(a.tail.y, b.tail.y);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
        d = __fsub_rn(a.tail.z, b.tail.z);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
        d = __fsub_rn(a.tail.w, b.tail.w);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
    }
    return acc;
}

// snap_d[p K + i] = distance of p and entry i of its list: the squared norms of
// the join where the sets' distances did not come from this context's kernels
// (sets handed over or read from a file hold what their writer put there).
template <int D>
__global__ void __launch_bounds__(256)
    k_edge_distances(const uint32_t* __restrict__ snap, const float* __restrict__ pts, int ld, uint32_t n, uint32_t K,
                     float* __restrict__ snap_d) {
    const int lane = threadIdx.x % kWarp, l = lane & 7, g = lane >> 3;
    for (uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp; p < n; p += gridDim.x * blockDim.x / kWarp) {
        ChainRow<D> mine;
        load_chain_row<D>(mine, pts + static_cast<size_t>(p) * ld, l);
        const size_t base = static_cast<size_t>(p) * K;
        for (uint32_t i0 = 0; i0 < K; i0 += 4) {
            const uint32_t i = i0 + g;
            ChainRow<D> row;
            load_chain_row<D>(row, pts + static_cast<size_t>(snap[base + (i < K ? i : i0)]) * ld, l);
            const float d = group_distance<D>(row, mine, lane & ~7);
            if (i < K && l == 0) snap_d[base + i] = d;
        }
    }
}

// Ascending sort of ids[0 .. U), U <= 32 E, by one warp.
template <int E>
__device__ __forceinline__ void warp_sort_ids(uint32_t* ids, uint32_t U, int lane) {
    uint32_t x[E];
#pragma unroll
    for (int r = 0; r < E; ++r) x[r] = lane * E + r < static_cast<int>(U) ? ids[lane * E + r] : kNone;
    warp_sort_lanes<E>(x, lane);
#pragma unroll
    for (int r = 0; r < E; ++r)
        if (lane * E + r < static_cast<int>(U)) ids[lane * E + r] = x[r];
    __syncwarp();
}

// Offers a point's candidates ids[0 .. U) (sorted, each once, none a member), 32
// at a time, with their exact distances; returns the number of changes.  One
// warp.  (A candidate is offered when its distance is below the bound it meets;
// the bound p had when its pass started rules nothing else out.)
template <int D>
__device__ __forceinline__ uint32_t offer_sorted(WarpSet& s, const uint32_t* ids, uint32_t U, uint32_t p,
                                                 const float* __restrict__ pts, int ld, int K, int lane) {
    ChainRow<D> mine;
    load_chain_row<D>(mine, pts + static_cast<size_t>(p) * ld, lane & 7);
    uint32_t changed = 0;
    for (uint32_t t0 = 0; t0 < U; t0 += kWarp) {
        const uint32_t id = ids[min(t0 + lane, U - 1)];
        const float d = warp_distances<D, 4>(mine, id, pts, ld, lane);
        changed += set_offer_new_batch(s, id, d, t0 + lane < U, K, lane);
    }
    return changed;
}

// Shared memory of one warp of k_apply: the hash table, the candidates, the
// expanded mask bits, p's own list.
struct ApplyWarpSmem {
    uint32_t table[kWarpTable];
    uint32_t cands[kWarpTable];  // a power of two, for the sort
    uint16_t list[kWarpList];
    uint32_t mine[kMaxK];
};

// Points of [lo, hi), in `order` when given.  What bounds it: per point some 200
// candidate rows and 2,300 list entries gathered from L2 (5 TB/s at 2M points,
// where gathers alone reach 9), behind chains of dependent steps that few warps
// hide, so shared memory and registers are cut to 20 warps an SM: 15 warps with
// tables twice the size took 113 ms for the two passes of a 2M build, 25 with a
// cap of 512 candidates 144 (the points past it are slow), this 98; it was 111
// with the distances first, 64-bit keys sorted in shared memory and single-slot
// probes.
template <int D>
__global__ void __launch_bounds__(kApplyWarps * kWarp, kApplyPerSm)
    k_apply(const uint32_t* __restrict__ snap, const uint4* __restrict__ masks, const float* __restrict__ pts, int ld,
            uint32_t n, uint32_t lo, uint32_t hi, int K, uint32_t cap, const uint32_t* __restrict__ order,
            const uint32_t* __restrict__ error_flag, float* __restrict__ set_dist, uint32_t* __restrict__ set_id,
            uint32_t* __restrict__ set_size, uint32_t* __restrict__ set_maxslot, float* __restrict__ set_bound,
            uint32_t* __restrict__ big, uint32_t* __restrict__ big_n, uint32_t* __restrict__ changed_count,
            unsigned long long* __restrict__ counters) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    ApplyWarpSmem& sm = reinterpret_cast<ApplyWarpSmem*>(smem)[warp];
    const unsigned lt = (1u << lane) - 1u;
    unsigned long long n_member = 0, n_record = 0, n_exact = 0;
    uint32_t n_changed = 0;
    if (*error_flag) return;  // the join gave up: the sets stay as they are
    for (uint32_t w = blockIdx.x * kApplyWarps + warp; w < n; w += gridDim.x * kApplyWarps) {
        const uint32_t p = order ? order[w] : w;
        if (p < lo || p >= hi) continue;
        __syncwarp();  // the last point's candidates are read
        const uint32_t* list = snap + static_cast<size_t>(p) * K;
        const uint4* mask = masks + static_cast<size_t>(p - lo) * K;
        for (int a = lane; a < K; a += kWarp) sm.mine[a] = list[a];
        for (uint32_t t = lane; t < kWarpTable / 4; t += kWarp)
            reinterpret_cast<uint4*>(sm.table)[t] = make_uint4(kNone, kNone, kNone, kNone);
        WarpSet s;
        set_load(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
        __syncwarp();
        // p and its members first: they are never candidates.
        if (lane == 0) table_insert(sm.table, kWarpTable / 4, p, kMember);
#pragma unroll
        for (int r = 0; r < kSlotsPerLane; ++r)
            if (lane + r * kWarp < static_cast<int>(s.size)) table_insert(sm.table, kWarpTable / 4, s.id[r], kMember);
        __syncwarp();
        uint32_t U = 0, records = 0, members = 0;
        bool fits = true;
        // Expands the bits `word` (of the columns col0 ..) of each lane's list
        // a and inserts their ids.
        for (int a0 = 0; a0 < K && fits; a0 += kWarp) {
            const int a = a0 + lane;
            uint4 m = make_uint4(0u, 0u, 0u, 0u);
            if (a < K && (a == 0 || sm.mine[a - 1] != sm.mine[a])) m = mask[a];
            const uint32_t bits = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
            const uint32_t all = __reduce_add_sync(kFull, bits);
            if (all == 0) continue;
            // All four words at once when they fit the list, else a word at a time
            // (32 lanes' 32 bits fill it at most).
            const int steps = all <= kWarpList ? 1 : 4;
            for (int step = 0; step < steps && fits; ++step) {
                uint32_t w[4] = {m.x, m.y, m.z, m.w};
                if (steps > 1) {
#pragma unroll
                    for (int x = 0; x < 4; ++x) w[x] = step == x ? w[x] : 0u;
                }
                const uint32_t have = __popc(w[0]) + __popc(w[1]) + __popc(w[2]) + __popc(w[3]);
                uint32_t incl = have;
#pragma unroll
                for (int o = 1; o < kWarp; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += y;
                }
                const uint32_t T = __shfl_sync(kFull, incl, kWarp - 1);
                uint32_t at = incl - have;
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    for (uint32_t b = w[x]; b; b &= b - 1)
                        sm.list[at++] = static_cast<uint16_t>(a << 7 | (x * kWarp + __ffs(b) - 1));
                __syncwarp();
                // Entry t of the list: its id, four steps ahead of its insertion.
                auto entry = [&](uint32_t t) {
                    if (t >= T) return kNone;
                    const uint32_t x = sm.list[t];
                    return __ldg(snap + static_cast<size_t>(sm.mine[x >> 7]) * K + (x & 127u));
                };
                uint32_t c0 = entry(lane), c1 = entry(kWarp + lane), c2 = entry(2 * kWarp + lane), c3 = entry(3 * kWarp + lane);
                for (uint32_t t0 = 0; t0 < T && fits; t0 += kWarp) {
                    const uint32_t c = c0;
                    c0 = c1;
                    c1 = c2;
                    c2 = c3;
                    c3 = entry(t0 + 4 * kWarp + lane);
                    const uint32_t found = c != kNone ? table_insert(sm.table, kWarpTable / 4, c, 0u) : 0u;
                    const bool fresh = found == kFresh;
                    members += found == kMember ? 1u : 0u;
                    const unsigned b = __ballot_sync(kFull, fresh);
                    const uint32_t at2 = U + __popc(b & lt);
                    if (fresh) sm.cands[at2] = c;  // at most a step past the cap
                    U += __popc(b);
                    fits = U <= cap;
                }
                __syncwarp();
                records += T;
            }
        }
        if (!fits) {
            if (lane == 0) big[atomicAdd(big_n, 1u)] = p;
            continue;
        }
        n_member += members;
        n_record += lane == 0 ? records : 0u;
        n_exact += lane == 0 ? U : 0u;
        if (U == 0) continue;
        if (U <= 4 * kWarp)
            warp_sort_ids<4>(sm.cands, U, lane);
        else if (U <= 8 * kWarp)
            warp_sort_ids<8>(sm.cands, U, lane);
        else if (U <= 16 * kWarp)
            warp_sort_ids<16>(sm.cands, U, lane);
        else {
            for (uint32_t t = U + lane; t < kWarpTable; t += kWarp) sm.cands[t] = kNone;
            __syncwarp();
            warp_bitonic_sort(sm.cands, kWarpTable, lane);
        }
        if (offer_sorted<D>(s, sm.cands, U, p, pts, ld, K, lane)) {
            set_store(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
            ++n_changed;
        }
    }
    if (n_member) atomicAdd(&counters[2], n_member);
    if (lane == 0) {
        if (n_changed) atomicAdd(changed_count, n_changed);
        atomicAdd(&counters[3], n_exact);
        atomicAdd(&counters[4], n_record);
    }
}

// The queued points, one CTA each, with larger tables; those with more than
// `cap` candidates are queued on `lost` for the per-point pass.
struct ApplyBigSmem {
    uint32_t table[kCtaTable];
    uint32_t cands[kCtaCands];
    uint32_t mine[kMaxK];
};

template <int D>
__global__ void __launch_bounds__(kBigThreads)
    k_apply_big(const uint32_t* __restrict__ big, const uint32_t* __restrict__ big_n, const uint32_t* __restrict__ snap,
                const uint4* __restrict__ masks, const float* __restrict__ pts, int ld, uint32_t lo, int K, uint32_t cap,
                float* __restrict__ set_dist, uint32_t* __restrict__ set_id, uint32_t* __restrict__ set_size,
                uint32_t* __restrict__ set_maxslot, float* __restrict__ set_bound, uint32_t* __restrict__ changed_count,
                uint32_t* __restrict__ lost, uint32_t* __restrict__ lost_n, unsigned long long* __restrict__ counters) {
    extern __shared__ __align__(1024) unsigned char smem[];
    ApplyBigSmem& sm = *reinterpret_cast<ApplyBigSmem*>(smem);
    __shared__ uint32_t found_s;
    constexpr int kWarps = kBigThreads / kWarp;
    const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
    const uint32_t total = *big_n;
    for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
        const uint32_t p = big[w];
        const uint32_t* list = snap + static_cast<size_t>(p) * K;
        const uint4* mask = masks + static_cast<size_t>(p - lo) * K;
        for (uint32_t t = tid; t < kCtaTable / 4; t += kBigThreads)
            reinterpret_cast<uint4*>(sm.table)[t] = make_uint4(kNone, kNone, kNone, kNone);
        for (int a = tid; a < K; a += kBigThreads) sm.mine[a] = list[a];
        if (tid == 0) found_s = 0;
        __syncthreads();
        if (tid == 0) table_insert(sm.table, kCtaTable / 4, p, kMember);
        for (uint32_t t = tid; t < set_size[p]; t += kBigThreads)
            table_insert(sm.table, kCtaTable / 4, set_id[static_cast<size_t>(p) * K + t], kMember);
        __syncthreads();
        uint32_t members = 0, records = 0;
        for (int a = warp; a < K; a += kWarps) {
            if (a > 0 && sm.mine[a - 1] == sm.mine[a]) continue;
            const uint4 m = mask[a];
            const uint32_t part[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (part[x] == 0) continue;
                // The table has room for what the warps can add past the cap.  One
                // lane reads the count and the others take its word: other warps
                // add to it meanwhile, and the votes below need the whole warp.
                uint32_t so_far = 0;
                if (lane == 0) so_far = *static_cast<volatile uint32_t*>(&found_s);
                if (__shfl_sync(kFull, so_far, 0) > cap) continue;
                uint32_t c = 0, found = 0;
                if ((part[x] >> lane) & 1u) {
                    c = __ldg(snap + static_cast<size_t>(sm.mine[a]) * K + x * kWarp + lane);
                    found = table_insert(sm.table, kCtaTable / 4, c, 0u);
                }
                members += found == kMember ? 1u : 0u;
                records += __popc(part[x]);
                const unsigned b = __ballot_sync(kFull, found == kFresh);
                if (b == 0) continue;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&found_s, static_cast<uint32_t>(__popc(b)));
                at = __shfl_sync(kFull, at, 0) + __popc(b & ((1u << lane) - 1u));
                if (found == kFresh && at < kCtaCands) sm.cands[at] = c;
            }
        }
        __syncthreads();
        const uint32_t U = found_s;
        if (U > cap) {  // uniform over the CTA
            if (tid == 0) lost[atomicAdd(lost_n, 1u)] = p;
            __syncthreads();
            continue;
        }
        if (members) atomicAdd(&counters[2], static_cast<unsigned long long>(members));
        if (lane == 0) atomicAdd(&counters[4], static_cast<unsigned long long>(records));
        if (tid == 0) atomicAdd(&counters[3], static_cast<unsigned long long>(U));
        const uint32_t P2 = pow2_at_least(U);
        for (uint32_t t = U + tid; t < P2; t += kBigThreads) sm.cands[t] = kNone;
        __syncthreads();
        for (uint32_t k = 2; k <= P2; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t t = tid; t < P2 / 2; t += kBigThreads) {
                    const uint32_t i = 2 * t - (t & (j - 1));  // 2 j (t / j) + t % j, j a power of two
                    const uint32_t partner = i + j;
                    const bool up = (i & k) == 0;
                    const uint32_t a = sm.cands[i], b = sm.cands[partner];
                    if ((a > b) == up) {
                        sm.cands[i] = b;
                        sm.cands[partner] = a;
                    }
                }
                __syncthreads();
            }
        }
        // Every warp its share of the distances (the table's space takes them),
        // then the first one makes the offers.
        float* dists = reinterpret_cast<float*>(sm.table);
        ChainRow<D> row;
        load_chain_row<D>(row, pts + static_cast<size_t>(p) * ld, lane & 7);
        for (uint32_t t0 = warp * kWarp; t0 < U; t0 += kBigThreads) {
            const float d = warp_distances<D, 4>(row, sm.cands[min(t0 + lane, U - 1)], pts, ld, lane);
            if (t0 + lane < U) dists[t0 + lane] = d;
        }
        __syncthreads();
        if (warp == 0) {
            WarpSet s;
            set_load(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
            uint32_t changed = 0;
            for (uint32_t t0 = 0; t0 < U; t0 += kWarp) {
                const uint32_t t = min(t0 + lane, U - 1);
                changed += set_offer_new_batch(s, sm.cands[t], dists[t], t0 + lane < U, K, lane);
            }
            if (changed) {
                set_store(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
                if (lane == 0) atomicAdd(changed_count, 1u);
            }
        }
        __syncthreads();  // the distances are read before the next point's table
    }
}

// One 128 x 128 tile of the join's filter: a(m x D) . b(n x D)^T with both
// operands rounded to FP16 and FP32 accumulation (rows past m / n are zero);
// the diagnostic behind knng_debug_tile_gram.
template <int D>
__global__ void __launch_bounds__(kJoinThreads, 1)
    k_tile_gram(const float* __restrict__ a, uint32_t m, const float* __restrict__ b, uint32_t n,
                float* __restrict__ out, uint32_t* __restrict__ error_flag) {
    using T = Tile16<D>;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* tile_a = smem;
    unsigned char* tile_b = smem + T::bytes(kTile);
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
    for (uint32_t f = tid; f < 2 * T::bytes(kTile) / 16; f += kJoinThreads)
        reinterpret_cast<uint4*>(smem)[f] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) tc::tmem_alloc(&tmem_slot, kTile);
    if (tid == 0) {
        tc::mbar_init(&mbar, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t id = lane < kTile / kJoinWarps ? lane * kJoinWarps + warp : 0u;
    tile_rows<D, kTile, kJoinWarps, __half>(a, D, id, m, tile_a, T::stride(kTile), zero, lane, warp);
    tile_rows<D, kTile, kJoinWarps, __half>(b, D, id, n, tile_b, T::stride(kTile), zero, lane, warp);
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
        tc::fence_after_sync();
        tc::issue_tile_strided(tmem, tc::smem_u32(tile_a), tc::smem_u32(tile_b), T::stride(kTile), T::stride(kTile),
                               T::KP, tc::idesc_f16(kTile, kTile));
        tc::mma_commit(&mbar);
    }
    const bool done = tc::mbar_wait(&mbar, 0);
    if (__syncthreads_or(!done)) {
        if (tid == 0) atomicExch(error_flag, 1u);
        tc::mbar_wait(&mbar, 0);
    } else {
        tc::fence_after_sync();
        const int quarter = warp % 4, group = warp / 4, row = quarter * kWarp + lane;
        for (int hh = 0; hh < kGroupCols / 16; ++hh) {
            const int j0 = group * kGroupCols + 16 * hh;
            float g[16];
            tc::tmem_ld16(tmem + (static_cast<uint32_t>(quarter * kWarp) << 16) + j0, g);
            tc::tmem_wait_ld();
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (static_cast<uint32_t>(row) < m && static_cast<uint32_t>(j0 + u) < n)
                    out[static_cast<size_t>(row) * n + j0 + u] = g[u];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, kTile);
    }
}

void device_scan(Context& c, const uint32_t* in, uint64_t n, unsigned long long* out) {
    const uint32_t tiles = static_cast<uint32_t>((n + kScanTile - 1) / kScanTile);
    auto* tsum = static_cast<unsigned long long*>(scratch(c, "scan_tiles", (tiles + 1) * sizeof(unsigned long long)));
    k_scan_reduce<<<tiles, kScanThreads, 0, c.stream>>>(in, n, tsum);
    k_scan_tiles<<<1, kScanThreads, 0, c.stream>>>(tsum, tiles);
    k_scan_apply<<<tiles, kScanThreads, 0, c.stream>>>(in, n, tsum, out);
    c.launches += 3;
    KNNG_CUDA(cudaGetLastError());
}

}  // namespace

void set_refine_wait_limit(uint32_t polls) { KNNG_CUDA(cudaMemcpyToSymbol(tc::g_wait_limit, &polls, sizeof(polls))); }

void run_tile_gram(Context& c, uint32_t d, const float* d_a, uint32_t m, const float* d_b, uint32_t n, float* d_out) {
    auto* err = static_cast<uint32_t*>(scratch(c, "gram_error", sizeof(uint32_t)));
    KNNG_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), c.stream));
    KNNG_DISPATCH_D(d, {
        const size_t smem = join_smem(D, kTile);
        auto kern = k_tile_gram<D>;
        allow_max_smem(c, kern);
        kern<<<1, kJoinThreads, smem, c.stream>>>(d_a, m, d_b, n, d_out, err);
    });
    ++c.launches;
    KNNG_CUDA(cudaGetLastError());
    uint32_t h = 0;
    download(c, &h, err, 1);
    if (h) fail(KNNG_ERR_CUDA, "tensor-core tile: the MMA completion wait gave up");
}

namespace {

// Survivor keys of one block's warps in the per-point pass (k * k candidates a
// warp, as a power of two for the sort), and that pass's scratch for `blocks`.
uint64_t pointwise_block_bytes(const Context& c) {
    return static_cast<uint64_t>(kRefWarps) * pow2_at_least(c.k * c.k) * sizeof(unsigned long long);
}
struct PointwiseScratch {
    unsigned long long* keys;
    uint32_t* changed;
};
PointwiseScratch pointwise_scratch(Context& c, uint32_t blocks) {
    return {static_cast<unsigned long long*>(spare_take(c, kSpareKeys, blocks * pointwise_block_bytes(c))),
            static_cast<uint32_t*>(scratch(c, "refine_changed", sizeof(uint32_t)))};
}

}  // namespace

// The per-point pass over the points of d_list, or first .. first + count - 1.
uint64_t run_refine_pointwise(Context& c, const uint32_t* snap, const uint32_t* d_list, uint32_t count,
                              uint32_t first = 0) {
    const int K = static_cast<int>(c.k);
    const uint32_t cap = pow2_at_least(static_cast<uint32_t>(K * K));
    uint32_t blocks = std::max<uint32_t>(1, std::min<uint32_t>((count + kRefWarps - 1) / kRefWarps, 148 * 5));
    // Each block's warps need cap survivor keys; fewer blocks (a longer grid
    // stride) when the budget leaves less room.
    const uint64_t per_block = pointwise_block_bytes(c);
    spare_done(c, kSpareKeys, kSpareKeys);
    const uint64_t held_other = c.held - spare_bytes(c);
    const uint64_t room = c.budget > held_other + (16ull << 20) ? c.budget - held_other - (16ull << 20) : 0;
    blocks = static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>(blocks, room / per_block)));
    const auto [keys, changed] = pointwise_scratch(c, blocks);
    KNNG_CUDA(cudaMemsetAsync(changed, 0, sizeof(uint32_t), c.stream));
    KNNG_DISPATCH_D(c.d, {
        k_refine<D><<<blocks, kRefWarps * kWarp, 0, c.stream>>>(snap, c.points, c.ld, c.set_dist, c.set_id,
                                                               c.set_size, c.set_maxslot, c.set_bound, K, count,
                                                               d_list, first, keys, cap, changed);
    });
    ++c.launches;
    KNNG_CUDA(cudaGetLastError());
    uint32_t h = 0;
    download(c, &h, changed, 1);
    return h;
}

namespace {

// The lists of a join pass.  A join takes up to all of the budget for them, so
// they are spare buffers: the finished lists or the next pass's snapshot, for
// instance, may have their room.  This object gives them back at a pass's end.
struct PassLists {
    static constexpr int kFirst = kSpareSnapD, kLast = kSpareLost;
    Context& c;
    explicit PassLists(Context& ctx) : c(ctx) {}
    ~PassLists() { spare_done(c, kSpareSnapD, kSpareKeys); }
    // Keeps those of the last pass that are large enough, unless (its ranges may
    // have been larger) they would leave less than `reserve` of the budget.
    void take(const uint64_t (&need)[kLast - kFirst + 1], uint64_t reserve) {
        uint64_t all = 0;
        for (int i = kFirst; i <= kLast; ++i) {
            if (c.spare[i].bytes < need[i - kFirst]) spare_free(c, static_cast<SpareBuffer>(i));
            all += std::max<uint64_t>(c.spare[i].bytes, need[i - kFirst]);
        }
        if (c.held - spare_bytes(c) + all + reserve > c.budget)
            for (int i = kFirst; i <= kLast; ++i) spare_free(c, static_cast<SpareBuffer>(i));
        for (int i = kFirst; i <= kLast; ++i) c.spare_in_use |= 1u << i;
        for (int i = kFirst; i <= kLast; ++i) spare_take(c, static_cast<SpareBuffer>(i), need[i - kFirst]);
    }
    template <class T>
    T* list(SpareBuffer which) const {
        return static_cast<T*>(c.spare[which].ptr);
    }
};

}  // namespace

uint64_t run_refine(Context& c) {
    if (c.n == 0) return 0;
    PassLists lists(c);
    c.last_refine = {};  // a pass that goes point by point has no join to report
    const int K = static_cast<int>(c.k);
    const uint32_t n = c.n;
    const size_t entries = static_cast<size_t>(n) * K;
    // Points a range of the join takes beside `more` bytes: their edges' bits (16
    // bytes) and reverse entries (4) have to fit what the rest leaves of the
    // budget, and edge numbers 31 bits.  The reserve holds the other scratch, the
    // per-point pass's least among it.
    const uint64_t fixed = entries * 4 + static_cast<uint64_t>(n) * 24;
    const uint64_t reserve =
        std::max<uint64_t>(std::min<uint64_t>(256ull << 20, c.budget / 8), pointwise_block_bytes(c) + (64u << 10));
    auto fit_beside = [&](uint64_t more) {
        const uint64_t used = c.held - spare_bytes(c) + more + fixed + reserve;
        const uint64_t room = c.budget > used ? c.budget - used : 0;
        return std::min<uint64_t>({n, room / (20ull * K), ((1ull << 31) - 1) / K});
    };
    // A budget without room for a 64th of the points leaves the pass to the
    // per-point kernel.
    const uint64_t fit_least = (n + 63) / 64;
    // The join skips pairs the previous join pass offered (both edges in that
    // pass's lists): the snapshot is made in one of two buffers in turn, the
    // other holding the previous pass's lists, and marks each entry that was
    // already there.  (Not where that would cost more than half a range.)
    const size_t old_bytes = static_cast<size_t>(n) * kOldWords * 4;
    static const char* const snap_names[2] = {"refine_snap", "refine_snap_other"};
    const char* other = snap_names[c.snap_flip ^ 1u];
    const uint64_t more = (scratch_bytes(c, other) >= entries * 4 ? 0 : entries * 4) +
                          (scratch_bytes(c, "refine_old") >= old_bytes ? 0 : old_bytes);
    const bool marks = c.refine_mode == 0 && c.refine_skip_old && c.snap_prev_valid &&
                       fit_beside(more) >= std::max(fit_least, fit_beside(0) / 2);
    c.snap_prev_valid = false;  // valid again once this pass completes
    const uint32_t* prev = nullptr;
    uint32_t* old = nullptr;
    if (marks) {
        prev = static_cast<const uint32_t*>(scratch(c, snap_names[c.snap_flip], entries * 4));
        old = static_cast<uint32_t*>(scratch(c, "refine_old", old_bytes));
        c.snap_flip ^= 1u;
    }
    uint32_t* snap = static_cast<uint32_t*>(scratch(c, snap_names[c.snap_flip], entries * 4));
    const uint32_t sblocks = std::min<uint32_t>((n + kSnapWarps - 1) / kSnapWarps, 148 * 8);
    auto snapshot = [&](float* snap_d) {
        auto kernel = n <= kShortIds ? k_snapshot<uint32_t> : k_snapshot<unsigned long long>;
        kernel<<<sblocks, kSnapWarps * kWarp, 0, c.stream>>>(c.set_id, c.set_dist, c.set_size, n, K, snap, snap_d, prev, old);
        ++c.launches;
        KNNG_CUDA(cudaGetLastError());
    };
    auto pointwise = [&] {
        prev = nullptr;
        old = nullptr;
        snapshot(nullptr);
        return run_refine_pointwise(c, snap, nullptr, n);
    };
    if (c.refine_mode == 1) return pointwise();

    const uint64_t fit = fit_beside(0);
    if (fit < fit_least) return pointwise();
    const uint32_t rounds = static_cast<uint32_t>((n + fit - 1) / fit);
    const uint32_t step = (n + rounds - 1) / rounds;

    // With several ranges a later one may have to go to the per-point pass after
    // the sets have begun to change: what that needs is taken now.
    if (rounds > 1) pointwise_scratch(c, 1);

    const uint32_t wblocks = std::min<uint32_t>((n + 7) / 8, 148 * 16);
    Context::RefineRecord rec;
    cudaEvent_t ev[4];
    for (auto& e : ev) KNNG_CUDA(cudaEventCreate(&e));
    KNNG_CUDA(cudaEventRecord(ev[0], c.stream));
    const uint64_t point = static_cast<uint64_t>(n) + 1, edges = static_cast<uint64_t>(step) * K;
    lists.take({entries * sizeof(float), point * sizeof(uint32_t), point * sizeof(uint32_t),
                point * sizeof(unsigned long long), edges * sizeof(uint32_t), edges * sizeof(uint4),
                step * sizeof(uint32_t), step * sizeof(uint32_t)},
               reserve);
    auto* snap_d = lists.list<float>(kSpareSnapD);
    auto* cnt = lists.list<uint32_t>(kSpareRevCount);
    auto* cur = lists.list<uint32_t>(kSpareRevCursor);
    auto* off = lists.list<unsigned long long>(kSpareRevOffsets);
    auto* rev = lists.list<uint32_t>(kSpareRevIds);
    auto* masks = lists.list<uint4>(kSpareMasks);
    auto* big = lists.list<uint32_t>(kSpareBig);
    auto* lost = lists.list<uint32_t>(kSpareLost);
    snapshot(c.dists_own ? snap_d : nullptr);
    if (!c.dists_own) {
        KNNG_DISPATCH_D(c.d, {
            k_edge_distances<D><<<wblocks, 256, 0, c.stream>>>(snap, c.points, c.ld, n, static_cast<uint32_t>(K), snap_d);
        });
        ++c.launches;
        KNNG_CUDA(cudaGetLastError());
    }
    // What the pass's kernels count, and its error word.
    struct Counts {
        unsigned long long join[5];  // pairs, filter-passing, members, exact distances, candidate records
        uint32_t error, changed, big, lost, work, pad;
    };
    auto* counts = static_cast<Counts*>(scratch(c, "refine_counts", sizeof(Counts)));

    const uint32_t join_bytes = join_smem(static_cast<int>(c.d), static_cast<uint32_t>(K));
    // CTAs per SM from the SM's shared memory and registers (the kernel's
    // launch bounds ask for three).
    int sms = 0, smem_sm = 0, smem_reserved = 0, regs_sm = 0;
    KNNG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
    KNNG_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c.device));
    KNNG_CUDA(cudaDeviceGetAttribute(&smem_reserved, cudaDevAttrReservedSharedMemoryPerBlock, c.device));
    KNNG_CUDA(cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, c.device));
    cudaFuncAttributes fa{};
    KNNG_DISPATCH_D(c.d, {
        auto kern = k_join<D>;
        allow_max_smem(c, kern);
        allow_max_smem(c, k_apply<D>);
        allow_max_smem(c, k_apply_big<D>);
        KNNG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       static_cast<int>(cudaSharedmemCarveoutMaxShared)));
        KNNG_CUDA(cudaFuncGetAttributes(&fa, kern));
    });
    const size_t per_cta_smem = join_bytes + fa.sharedSizeBytes + static_cast<size_t>(smem_reserved);
    const int by_smem = static_cast<int>(static_cast<size_t>(smem_sm) / per_cta_smem);
    const int by_regs = fa.numRegs > 0 ? regs_sm / (fa.numRegs * kJoinThreads) : 2;
    const int per_sm = std::min({by_smem, by_regs, kJoinPerSm});
    if (per_sm < 1) fail(KNNG_ERR_UNSUPPORTED, "the join kernel does not fit on an SM");
    const uint32_t join_blocks = static_cast<uint32_t>(sms) * static_cast<uint32_t>(per_sm);
    // Points in the leaf order of the last repetition (c.indices), unless the
    // context was created with KNNG_JOIN_ORDER=id.
    const uint32_t* order = c.join_order_ids ? nullptr : c.indices;
    const uint32_t warp_cap = c.refine_slots >= 0 ? std::min<uint32_t>(c.refine_slots, kWarpCands) : kWarpCands;
    const uint32_t cta_cap =
        c.refine_pool >= 0 ? static_cast<uint32_t>(std::min<int64_t>(c.refine_pool, kCtaCands)) : kCtaCands;
    auto elapsed = [](cudaEvent_t a, cudaEvent_t b) {
        float ms = 0.f;
        KNNG_CUDA(cudaEventElapsedTime(&ms, a, b));
        return ms;
    };
    uint64_t changed = 0;
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t lo = r * step, hi = std::min(n, lo + step);
        if (lo >= hi) break;
        if (r > 0) KNNG_CUDA(cudaEventRecord(ev[0], c.stream));
        KNNG_CUDA(cudaMemsetAsync(cnt, 0, static_cast<size_t>(n) * sizeof(uint32_t), c.stream));
        KNNG_CUDA(cudaMemsetAsync(cur, 0, static_cast<size_t>(n) * sizeof(uint32_t), c.stream));
        KNNG_CUDA(cudaMemsetAsync(counts, 0, sizeof(Counts), c.stream));
        k_rev_count<<<wblocks, 256, 0, c.stream>>>(snap, lo, hi, K, cnt);
        device_scan(c, cnt, n, off);
        k_rev_fill<<<wblocks, 256, 0, c.stream>>>(snap, n, lo, hi, K, off, cur, rev, old, order);
        c.launches += 2;
        KNNG_CUDA(cudaGetLastError());
        KNNG_CUDA(cudaEventRecord(ev[1], c.stream));
        KNNG_DISPATCH_D(c.d, {
            k_join<D><<<join_blocks, kJoinThreads, join_bytes, c.stream>>>(
                snap, snap_d, off, rev, c.points, c.ld, c.set_bound, static_cast<uint32_t>(K), n, lo,
                reinterpret_cast<uint2*>(masks), &counts->error, counts->join, order, &counts->work, old);
        });
        KNNG_CUDA(cudaGetLastError());
        if (c.join_fails_in == static_cast<int>(r))  // as a wait that gives up leaves it
            KNNG_CUDA(cudaMemsetAsync(&counts->error, 1, sizeof(uint32_t), c.stream));
        KNNG_CUDA(cudaEventRecord(ev[2], c.stream));
        KNNG_DISPATCH_D(c.d, {
            k_apply<D><<<std::min<uint32_t>((n + kApplyWarps - 1) / kApplyWarps, kApplyPerSm * sms), kApplyWarps * kWarp,
                         kApplyWarps * sizeof(ApplyWarpSmem), c.stream>>>(
                snap, masks, c.points, c.ld, n, lo, hi, K, warp_cap, order, &counts->error, c.set_dist, c.set_id,
                c.set_size, c.set_maxslot, c.set_bound, big, &counts->big, &counts->changed, counts->join);
            k_apply_big<D><<<2 * sms, kBigThreads, sizeof(ApplyBigSmem), c.stream>>>(
                big, &counts->big, snap, masks, c.points, c.ld, lo, K, cta_cap, c.set_dist, c.set_id, c.set_size,
                c.set_maxslot, c.set_bound, &counts->changed, lost, &counts->lost, counts->join);
        });
        c.launches += 3;
        ++rec.join_launches;
        KNNG_CUDA(cudaGetLastError());
        KNNG_CUDA(cudaEventRecord(ev[3], c.stream));
        Counts h{};
        download(c, &h, counts, 1);
        // A pass is whole or not started.  The first range's join gave up: no set
        // has changed, and the pass fails.  A later one's: the points from here on
        // take the per-point pass, which waits for nothing, to the same sets.
        if (h.error && r == 0) {
            for (auto& e : ev) cudaEventDestroy(e);
            fail(KNNG_ERR_CUDA, "tensor-core join: an MMA completion wait gave up");
        }
        const uint32_t redo = h.error ? n - lo : h.lost;
        const float ms_all = elapsed(ev[0], ev[3]), ms_join = elapsed(ev[1], ev[2]), ms_apply = elapsed(ev[2], ev[3]);
        rec.ms_join += ms_join;
        rec.ms_apply += ms_apply;
        rec.ms_prep += std::max(0.f, ms_all - ms_join - ms_apply);
        // Points with too many candidates: the one-warp-per-point pass over
        // their list.
        if (redo > 0) {
            KNNG_CUDA(cudaEventRecord(ev[0], c.stream));
            changed += run_refine_pointwise(c, snap, h.error ? nullptr : lost, redo, lo);
            KNNG_CUDA(cudaEventRecord(ev[1], c.stream));
            KNNG_CUDA(cudaEventSynchronize(ev[1]));
            rec.ms_fallback += elapsed(ev[0], ev[1]);
        }
        changed += h.changed;
        rec.pairs += h.join[0];
        rec.filter_pass += h.join[1];
        rec.member_skip += h.join[2];
        rec.exact += h.join[3];
        rec.emits += h.join[4] - h.join[2];
        rec.overflow += h.big;
        rec.lost += redo;
        if (h.error) break;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    c.last_refine = rec;
    // This pass offered every pair of its lists; the next one may skip them.
    c.snap_prev_valid = c.refine_skip_old;
    return changed;
}

}  // namespace knng

// ------------------------------------------------------------------------
// Allocation-free neighbour-of-neighbour pass.
//
// Some callers cannot allocate device memory while they call into this
// library: code that runs inside another framework's memory pool or under a
// strict memory budget, code that only receives device pointers from a host
// application, and code paths where a cudaMalloc would synchronise the device
// at the wrong moment.  knng_refine_pointwise_noalloc serves them: it runs the
// one-warp-per-point pass on buffers the caller passes in, and keeps its only
// scratch -- each warp's survivor records -- in the fixed device array below,
// which every GPU that loads the library holds until the process exits.
//
// The array is cut into one region per warp of pow2(k*k) records (a point has
// at most k*k candidates), so the launch is as wide as the array allows for
// the caller's k: 256 warps at k = 100, 1024 at k <= 64, up to 2,368 (16 per
// SM) at k <= 32.
namespace {

constexpr uint64_t kNoAllocRecords = 1ull << 22;  // 32 MiB of 8-byte survivor records
constexpr uint32_t kNoAllocMaxWarps = 148 * 16;
static __device__ __align__(256) unsigned long long g_noalloc_survivors[kNoAllocRecords];

// The device address of that array differs per CUDA context, and a context
// handle can be reused after its context is destroyed, so the cache is keyed on
// the context's unique id (cuCtxGetId), resolved through the runtime's driver
// entry points (no link-time dependence on the driver library).
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

struct NoAllocEntry {
    unsigned long long ctx_id;
    void* addr;
};

std::mutex g_noalloc_mutex;
std::vector<NoAllocEntry> g_noalloc_cache;
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;

cudaError_t current_context_id(unsigned long long* id) {
    if (!g_ctx_get_current || !g_ctx_get_id) {
        void* f = nullptr;
        void* g = nullptr;
        cudaDriverEntryPointQueryResult q1, q2;
        cudaError_t e = cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q1);
        if (e != cudaSuccess) return e;
        e = cudaGetDriverEntryPoint("cuCtxGetId", &g, cudaEnableDefault, &q2);
        if (e != cudaSuccess) return e;
        if (q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f || !g)
            return cudaErrorNotSupported;
        g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(g);
    }
    CUcontext ctx = nullptr;
    if (g_ctx_get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr) return cudaErrorDeviceUninitialized;
    return g_ctx_get_id(ctx, id) == CUDA_SUCCESS ? cudaSuccess : cudaErrorDeviceUninitialized;
}

// Device address of the scratch array in the current context, looked up with
// cudaGetSymbolAddress the first time a context calls (the array's name in host
// code is a host-side stand-in, not a device address).
cudaError_t noalloc_scratch(unsigned long long** out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    unsigned long long id = 0;
    cudaError_t e = current_context_id(&id);
    if (e == cudaErrorDeviceUninitialized) {
        // No context is current yet: the lookup below makes the device's
        // primary context current, then its id is taken.
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_survivors);
        if (e != cudaSuccess) return e;
        e = current_context_id(&id);
    }
    if (e != cudaSuccess) return e;
    for (const NoAllocEntry& c : g_noalloc_cache) {
        if (c.ctx_id == id) {
            *out = static_cast<unsigned long long*>(c.addr);
            return cudaSuccess;
        }
    }
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_survivors);
    if (e != cudaSuccess) return e;
    g_noalloc_cache.push_back({id, p});
    *out = static_cast<unsigned long long*>(p);
    return cudaSuccess;
}

}  // namespace

extern "C" knng_status knng_refine_pointwise_noalloc(const float* d_points, uint32_t n, uint32_t d, uint32_t k,
                                                     uint32_t* d_snapshot, float* d_dist, uint32_t* d_ids,
                                                     uint32_t* d_size, uint32_t* d_maxslot, float* d_bound,
                                                     uint32_t* d_changed, void* stream) {
    using namespace knng;
    // A point has at most k*k candidates; the set capacity is at most 128.
    if (k == 0 || k > static_cast<uint32_t>(kMaxK)) return KNNG_ERR_UNSUPPORTED;
    if (!dim_supported(d)) return KNNG_ERR_UNSUPPORTED;
    if (n == 0) return KNNG_OK;
    if (!d_points || !d_snapshot || !d_dist || !d_ids || !d_size || !d_maxslot || !d_bound || !d_changed)
        return KNNG_ERR_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(d_points) % 16 != 0) return KNNG_ERR_INVALID_ARGUMENT;
    unsigned long long* scratch_keys = nullptr;
    if (noalloc_scratch(&scratch_keys) != cudaSuccess) {
        cudaGetLastError();
        return KNNG_ERR_CUDA;
    }
    // One region of pow2(k*k) records per warp; whole blocks of kRefWarps.
    const uint32_t region = pow2_at_least(k * k);
    const uint64_t fit = kNoAllocRecords / region;
    const uint32_t warps = static_cast<uint32_t>(std::min<uint64_t>(fit, kNoAllocMaxWarps)) / kRefWarps * kRefWarps;
    const uint32_t need = (n + kRefWarps - 1) / kRefWarps * kRefWarps;
    const uint32_t blocks = std::max<uint32_t>(1, std::min(warps, need) / kRefWarps);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int K = static_cast<int>(k);
    if (cudaMemsetAsync(d_changed, 0, sizeof(uint32_t), s) != cudaSuccess) {
        cudaGetLastError();
        return KNNG_ERR_CUDA;
    }
    const uint32_t sblocks = std::min<uint32_t>((n + kSnapWarps - 1) / kSnapWarps, 148 * 8);
    // The caller's ids are not bounded by n in its empty slots: the wide keys.
    k_snapshot<unsigned long long><<<sblocks, kSnapWarps * kWarp, 0, s>>>(d_ids, nullptr, nullptr, n, K, d_snapshot, nullptr,
                                                                          nullptr, nullptr);
    try {
        KNNG_DISPATCH_D(d, {
            k_refine<D><<<blocks, kRefWarps * kWarp, 0, s>>>(d_snapshot, d_points, static_cast<int>(d), d_dist,
                                                             d_ids, d_size, d_maxslot, d_bound, K, n, nullptr, 0,
                                                             scratch_keys, region, d_changed);
        });
    } catch (const Error& e) {
        return e.status;
    }
    if (cudaGetLastError() != cudaSuccess) return KNNG_ERR_CUDA;
    return KNNG_OK;
}
