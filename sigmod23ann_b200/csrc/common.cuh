// Device-side building blocks shared by the k-NN graph kernels.
//
//  * canonical_distance4 / canonical_dot: the reference's FP32 evaluation order
//    (src/LinearAlgebra.hpp:53-77 and :179-200): eight lanes, lane l an FMA
//    chain over dims l, l+8, ... below the largest multiple of 8 <= D, lanes
//    summed left to right into 0.0f, then each tail dim added as a separately
//    rounded product.  Written with __f*_rn intrinsics so nvcc cannot contract
//    or reorder them.
//  * Warp-resident neighbour sets: lane l holds slots l, l+32, l+64, l+96 of a
//    set of capacity K <= 128; warp_argmax reproduces the slot that
//    KnnSetScannableSimd::getMaxIdx (src/KnnSets.hpp:82-111) selects.
//  * mix64 / counter_position: the counter-based RNG of the device-seeded build.
#pragma once

#include <cfloat>
#include <cstdint>
#include <cstring>

namespace knng {

constexpr int kWarp = 32;
constexpr int kMaxK = 128;
constexpr int kSlotsPerLane = kMaxK / kWarp;
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr unsigned kFull = 0xFFFFFFFFu;

// ---------------------------------------------------------------- arithmetic

template <int D>
__device__ __forceinline__ float canonical_dot(const float* __restrict__ a, const float* __restrict__ b) {
    constexpr int M = D / 8 * 8;
    float lane[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) lane[l] = 0.0f;
#pragma unroll
    for (int base = 0; base < M; base += 8) {
#pragma unroll
        for (int l = 0; l < 8; ++l) lane[l] = __fmaf_rn(b[base + l], a[base + l], lane[l]);
    }
    float acc = 0.0f;
#pragma unroll
    for (int l = 0; l < 8; ++l) acc = __fadd_rn(acc, lane[l]);
#pragma unroll
    for (int i = M; i < D; ++i) acc = __fadd_rn(acc, __fmul_rn(a[i], b[i]));
    return acc;
}

// Rows read as float4 (16-byte aligned, D % 4 == 0).
template <int D>
__device__ __forceinline__ float canonical_distance4(const float4* __restrict__ a, const float4* __restrict__ b) {
    static_assert(D % 4 == 0, "float4 path needs D % 4 == 0");
    constexpr int M = D / 8 * 8;
    float lane[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) lane[l] = 0.0f;
#pragma unroll
    for (int q = 0; q < M / 4; ++q) {
        float4 x = a[q];
        float4 y = b[q];
        const int l0 = (q & 1) * 4;
        float d0 = __fsub_rn(x.x, y.x), d1 = __fsub_rn(x.y, y.y), d2 = __fsub_rn(x.z, y.z), d3 = __fsub_rn(x.w, y.w);
        lane[l0 + 0] = __fmaf_rn(d0, d0, lane[l0 + 0]);
        lane[l0 + 1] = __fmaf_rn(d1, d1, lane[l0 + 1]);
        lane[l0 + 2] = __fmaf_rn(d2, d2, lane[l0 + 2]);
        lane[l0 + 3] = __fmaf_rn(d3, d3, lane[l0 + 3]);
    }
    float acc = 0.0f;
#pragma unroll
    for (int l = 0; l < 8; ++l) acc = __fadd_rn(acc, lane[l]);
#pragma unroll
    for (int q = M / 4; q < D / 4; ++q) {
        float4 x = a[q];
        float4 y = b[q];
        float d0 = __fsub_rn(x.x, y.x), d1 = __fsub_rn(x.y, y.y), d2 = __fsub_rn(x.z, y.z), d3 = __fsub_rn(x.w, y.w);
        acc = __fadd_rn(acc, __fmul_rn(d0, d0));
        acc = __fadd_rn(acc, __fmul_rn(d1, d1));
        acc = __fadd_rn(acc, __fmul_rn(d2, d2));
        acc = __fadd_rn(acc, __fmul_rn(d3, d3));
    }
    return acc;
}

// ------------------------------------------------- distances by warp groups

// A row as lane l of a group of eight holds it for the reference's distance
// order: FMA chain l's dimensions l, l + 8, ..., and the tail.
template <int D>
struct ChainRow {
    static constexpr int M = D / 8 * 8;
    float c[M / 8];
    float4 tail;
};

template <int D>
__device__ __forceinline__ void load_chain_row(ChainRow<D>& r, const float* __restrict__ row, int l) {
    constexpr int M = ChainRow<D>::M;
#pragma unroll
    for (int i = 0; i < M / 8; ++i) r.c[i] = __ldg(row + 8 * i + l);
    r.tail = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (D > M) r.tail = __ldg(reinterpret_cast<const float4*>(row + M));
}

// A load that stays where it is written (the compiler otherwise puts a row's
// loads next to their uses, and each row waits for its own latency).
__device__ __forceinline__ float load_now(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// canonical_distance4 of `mine` (p's row) and the rows of 32 points, lane t's
// point id t; every lane returns its own.  A group of eight lanes reads its
// eight rows one after the other, a lane a chain (32 bytes of each row a load);
// the chains are then exchanged within the group, so that each lane sums the
// eight of its own point and adds its tail.
template <int D, int V>
__device__ __forceinline__ float warp_distances(const ChainRow<D>& mine, uint32_t id, const float* __restrict__ pts,
                                                int ld, int lane) {
    constexpr int M = ChainRow<D>::M;
    static_assert(D - M == 0 || D - M == 4, "tail of 0 or 4 dims");
    const int l = lane & 7, g0 = lane & ~7;
    float4 tail = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (D > M) tail = __ldg(reinterpret_cast<const float4*>(pts + static_cast<size_t>(id) * ld + M));
    // V rows' loads in flight, then their chains.
    float x[8];
#pragma unroll
    for (int v0 = 0; v0 < 8; v0 += V) {
        float y[V][M / 8];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const float* row = pts + static_cast<size_t>(__shfl_sync(kFull, id, g0 + v0 + v)) * ld + l;
#pragma unroll
            for (int i = 0; i < M / 8; ++i) y[v][i] = load_now(row + 8 * i);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            float chain = 0.0f;
#pragma unroll
            for (int i = 0; i < M / 8; ++i) {
                const float d = __fsub_rn(y[v][i], mine.c[i]);
                chain = __fmaf_rn(d, d, chain);
            }
            x[v0 + v] = chain;
        }
    }
#pragma unroll
    for (int s = 1; s < 8; s <<= 1) {
        const bool high = (l & s) != 0;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            if (a & s) continue;
            const float got = __shfl_xor_sync(kFull, high ? x[a] : x[a | s], s);
            if (high) x[a] = got; else x[a | s] = got;
        }
    }
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = __fadd_rn(acc, x[j]);
    if constexpr (D > M) {
        float d = __fsub_rn(tail.x, mine.tail.x);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
        d = __fsub_rn(tail.y, mine.tail.y);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
        d = __fsub_rn(tail.z, mine.tail.z);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
        d = __fsub_rn(tail.w, mine.tail.w);
        acc = __fadd_rn(acc, __fmul_rn(d, d));
    }
    return acc;
}

// ---------------------------------------------------------- neighbour sets
//
// Tie order of getMaxIdx: among slots holding the maximum distance, the one
// with the smallest (slot % 8), then the smallest (slot / 8).

struct WarpSet {
    float dist[kSlotsPerLane];
    uint32_t id[kSlotsPerLane];
    uint32_t size;     // warp-uniform
    uint32_t maxslot;  // warp-uniform
    float bound;       // warp-uniform
};

// Loads point p's set from the slot arrays (row stride K) into the warp.
__device__ __forceinline__ void set_load(WarpSet& s, const float* __restrict__ dist, const uint32_t* __restrict__ ids,
                                         const uint32_t* __restrict__ sizes, const uint32_t* __restrict__ maxslot,
                                         const float* __restrict__ bounds, uint32_t p, int K, int lane) {
    const size_t base = static_cast<size_t>(p) * K;
#pragma unroll
    for (int r = 0; r < kSlotsPerLane; ++r) {
        const int slot = lane + r * kWarp;
        s.dist[r] = slot < K ? dist[base + slot] : 0.0f;
        s.id[r] = slot < K ? ids[base + slot] : 0u;
    }
    s.size = sizes[p];
    s.maxslot = maxslot[p];
    s.bound = bounds[p];
}

__device__ __forceinline__ void set_store(const WarpSet& s, float* __restrict__ dist, uint32_t* __restrict__ ids,
                                          uint32_t* __restrict__ sizes, uint32_t* __restrict__ maxslot,
                                          float* __restrict__ bounds, uint32_t p, int K, int lane) {
    const size_t base = static_cast<size_t>(p) * K;
#pragma unroll
    for (int r = 0; r < kSlotsPerLane; ++r) {
        const int slot = lane + r * kWarp;
        if (slot < K) {
            dist[base + slot] = s.dist[r];
            ids[base + slot] = s.id[r];
        }
    }
    if (lane == 0) {
        sizes[p] = s.size;
        maxslot[p] = s.maxslot;
        bounds[p] = s.bound;
    }
}

// Slot of the maximum distance over K filled slots, in getMaxIdx's tie order;
// sets s.maxslot and s.bound (warp-uniform).  Distances are sums of squares
// (+0 or positive), so their bit patterns order like their values: one warp
// max reduction finds the largest distance, a second one, over the slots
// holding it, the winner of the tie order (smallest slot % 8, then slot / 8,
// encoded so that the preferred slot has the largest key).
__device__ __forceinline__ void warp_argmax(WarpSet& s, int K, int lane) {
    uint32_t vb = 0;
#pragma unroll
    for (int r = 0; r < kSlotsPerLane; ++r) {
        const uint32_t slot = lane + r * kWarp;
        if (slot < static_cast<uint32_t>(K)) vb = max(vb, __float_as_uint(s.dist[r]));
    }
    const uint32_t top = __reduce_max_sync(kFull, vb);
    uint32_t tk = 0;  // 128 - (slot % 8 * 16 + slot / 8) for slots holding `top`, else 0
#pragma unroll
    for (int r = 0; r < kSlotsPerLane; ++r) {
        const uint32_t slot = lane + r * kWarp;
        if (slot < static_cast<uint32_t>(K) && __float_as_uint(s.dist[r]) == top)
            tk = max(tk, 128u - (((slot & 7u) << 4) | (slot >> 3)));
    }
    const uint32_t t = 128u - __reduce_max_sync(kFull, tk);
    s.maxslot = (t & 15u) * 8u + (t >> 4);
    s.bound = __uint_as_float(top);
}

__device__ __forceinline__ bool set_contains(const WarpSet& s, uint32_t cand, int lane) {
    bool hit = false;
#pragma unroll
    for (int r = 0; r < kSlotsPerLane; ++r) {
        const uint32_t slot = lane + r * kWarp;
        hit |= (slot < s.size) && (s.id[r] == cand);
    }
    return __any_sync(kFull, hit);
}

__device__ __forceinline__ void set_write_slot(WarpSet& s, uint32_t slot, uint32_t cand, float d, int lane) {
#pragma unroll
    for (int r = 0; r < kSlotsPerLane; ++r) {
        if (slot == static_cast<uint32_t>(lane + r * kWarp)) {
            s.dist[r] = d;
            s.id[r] = cand;
        }
    }
}

// addCandidateLessThan (src/KnnSets.hpp:39-57) for a warp-uniform offer that
// already passed d < s.bound.  Returns true if the set changed.
__device__ __forceinline__ bool set_offer(WarpSet& s, uint32_t cand, float d, int K, int lane) {
    if (set_contains(s, cand, lane)) return false;
    if (s.size < static_cast<uint32_t>(K)) {
        set_write_slot(s, s.size, cand, d, lane);
        s.size += 1;
        if (s.size == static_cast<uint32_t>(K)) warp_argmax(s, K, lane);
        return true;
    }
    set_write_slot(s, s.maxslot, cand, d, lane);
    warp_argmax(s, K, lane);
    return true;
}

// Offers the warp's 32 candidates (lane j holds (cand_j, d_j), valid_j) in lane
// order, with the sequential semantics of the reference's inner loop.
__device__ __forceinline__ uint32_t set_offer_batch(WarpSet& s, uint32_t cand, float d, bool valid, int K, int lane) {
    uint32_t changed = 0;
    unsigned pending = __ballot_sync(kFull, valid && d < s.bound);
    while (pending) {
        const int src = __ffs(pending) - 1;
        pending &= pending - 1;
        const float dj = __shfl_sync(kFull, d, src);
        const uint32_t cj = __shfl_sync(kFull, cand, src);
        if (dj < s.bound) changed += set_offer(s, cj, dj, K, lane) ? 1u : 0u;
        // The bound only decreases: drop the candidates it now excludes.
        pending &= __ballot_sync(kFull, valid && d < s.bound);
    }
    return changed;
}

// set_offer_batch for candidates that are not in the set and that are offered
// once: the containment check falls away.  (A caller leaves out the members of
// the set as it found it; one that is evicted later is at least as far as every
// later bound, so leaving it out is what offering it would do.)
//
// Offers that only fill free slots are placed together, by rank; `scratch` is 32
// bytes of shared memory for that (null: one by one).  A full set's arg-max
// takes the common case first: the lanes whose largest slot is the maximum are
// found by one vote, and if there is one such lane its first slot holding it is
// the answer (slots of one lane share slot % 8); ties between lanes go through
// the full order.  The slot stays with its lane (its number there in `mine`)
// until the batch is done.
__device__ __forceinline__ uint32_t set_offer_new_batch(WarpSet& s, uint32_t cand, float d, bool valid, int K, int lane,
                                                        uint8_t* scratch = nullptr) {
    static_assert(kSlotsPerLane == 4, "four slots a lane");
    unsigned pending = __ballot_sync(kFull, valid && d < s.bound);
    if (pending == 0) return 0;
    uint32_t changed = 0;
    if (s.size < static_cast<uint32_t>(K)) {
        const uint32_t count = __popc(pending);
        if (scratch && s.size + count <= static_cast<uint32_t>(K)) {
            if ((pending >> lane) & 1u) scratch[__popc(pending & ((1u << lane) - 1u))] = static_cast<uint8_t>(lane);
            __syncwarp();
            const uint32_t rank = (lane - s.size) % kWarp;  // of the slot this lane gets
            const bool gets = rank < count;
            const int src = gets ? scratch[rank] : 0;
            const float dj = __shfl_sync(kFull, d, src);
            const uint32_t cj = __shfl_sync(kFull, cand, src);
            const uint32_t at = (s.size + rank) / kWarp;
#pragma unroll
            for (uint32_t r = 0; r < kSlotsPerLane; ++r) {
                if (gets && at == r) {
                    s.dist[r] = dj;
                    s.id[r] = cj;
                }
            }
            s.size += count;
            if (s.size == static_cast<uint32_t>(K)) warp_argmax(s, K, lane);
            __syncwarp();  // the scratch is read
            return count;
        }
        while (pending && s.size < static_cast<uint32_t>(K)) {
            const int src = __ffs(pending) - 1;
            pending &= pending - 1;
            const float dj = __shfl_sync(kFull, d, src);
            const uint32_t cj = __shfl_sync(kFull, cand, src);
            set_write_slot(s, s.size, cj, dj, lane);
            s.size += 1;
            ++changed;
        }
        if (s.size < static_cast<uint32_t>(K)) return changed;
        warp_argmax(s, K, lane);
        pending &= __ballot_sync(kFull, d < s.bound);
    }
    if (pending == 0) return changed;
    int owner = s.maxslot % kWarp;
    uint32_t mine = s.maxslot / kWarp;
    do {
        const int src = __ffs(pending) - 1;
        pending &= pending - 1;
        const float dj = __shfl_sync(kFull, d, src);
        const uint32_t cj = __shfl_sync(kFull, cand, src);
        const bool here = lane == owner;
#pragma unroll
        for (uint32_t r = 0; r < kSlotsPerLane; ++r) {
            if (here && mine == r) {
                s.dist[r] = dj;
                s.id[r] = cj;
            }
        }
        ++changed;
        const uint32_t b0 = __float_as_uint(s.dist[0]), b1 = __float_as_uint(s.dist[1]);
        const uint32_t b2 = __float_as_uint(s.dist[2]), b3 = __float_as_uint(s.dist[3]);
        const uint32_t most = max(max(b0, b1), max(b2, b3));  // slots past K hold 0
        const uint32_t top = __reduce_max_sync(kFull, most);
        const unsigned holders = __ballot_sync(kFull, most == top);
        mine = b0 == most ? 0u : b1 == most ? 1u : b2 == most ? 2u : 3u;
        owner = 31 - __clz(holders);
        s.bound = __uint_as_float(top);
        if (holders != (1u << owner)) {
            warp_argmax(s, K, lane);
            owner = s.maxslot % kWarp;
            mine = s.maxslot / kWarp;
        }
        // The bound only decreases: drop the candidates it now excludes.
        pending &= __ballot_sync(kFull, d < s.bound);
    } while (pending);
    s.maxslot = __shfl_sync(kFull, mine * kWarp + lane, owner);
    return changed;
}

// Ascending sort of a warp's 32 E unsigned keys, E (a power of two) registers a
// lane, element lane * E + r of the result in x[r]: a bitonic network.  Strides
// below E stay in a lane; the lanes whose block a level sorts downwards hold its
// keys complemented, so that every exchange is a minimum and a maximum.
template <int E, class Key>
__device__ __forceinline__ void warp_sort_lanes(Key (&x)[E], int lane) {
#pragma unroll
    for (int k = 2; k <= E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
            for (int r = 0; r < E; ++r) {
                if (r & j) continue;
                // Direction of element lane * E + r at level k: within the lane
                // below E, the lane's own bit at E.
                const bool up = k < E ? (r & k) == 0 : (lane & 1) == 0;
                const Key lo = min(x[r], x[r | j]), hi = max(x[r], x[r | j]);
                x[r] = up ? lo : hi;
                x[r | j] = up ? hi : lo;
            }
        }
    }
    Key flip = 0;
#pragma unroll
    for (int k = 2; k <= kWarp; k <<= 1) {  // level k * E: blocks of k lanes; the last sorts upwards everywhere
        const Key want = (lane & k) ? ~Key(0) : Key(0);
#pragma unroll
        for (int r = 0; r < E; ++r) x[r] ^= flip ^ want;
        flip = want;
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const bool low = (lane & j) == 0;
#pragma unroll
            for (int r = 0; r < E; ++r) {
                const Key o = __shfl_xor_sync(kFull, x[r], j);
                x[r] = low ? min(x[r], o) : max(x[r], o);
            }
        }
#pragma unroll
        for (int j = E >> 1; j > 0; j >>= 1) {
#pragma unroll
            for (int r = 0; r < E; ++r) {
                if (r & j) continue;
                const Key lo = min(x[r], x[r | j]), hi = max(x[r], x[r | j]);
                x[r] = lo;
                x[r | j] = hi;
            }
        }
    }
}

// A warp writes out[0 .. K): entries 4 lane .. 4 lane + 3 from each lane, as one
// 16-byte store where the row's address allows it (k not a multiple of 4, or a
// caller's array, may leave it anywhere).
template <class T>
__device__ __forceinline__ void store_lane_run(T* out, int K, int lane, const T (&x)[4]) {
    static_assert(sizeof(T) == 4, "four entries are one 16-byte store");
    const int i = 4 * lane;
    if (i + 3 < K && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
        uint4 v;
        memcpy(&v, x, sizeof(v));
        *reinterpret_cast<uint4*>(out + i) = v;
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (i + r < K) out[i + r] = x[r];
    }
}

// Ascending bitonic sort of n (power of two, n >= 2) unsigned keys by one
// warp; keys may live in shared or global memory.
template <class Key>
__device__ __forceinline__ void warp_bitonic_sort(Key* keys, uint32_t n, int lane) {
    for (uint32_t k = 2; k <= n; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t t = lane; t < n / 2; t += kWarp) {
                const uint32_t i = 2 * t - (t & (j - 1));  // 2 j (t / j) + t % j, j a power of two
                const uint32_t partner = i + j;
                const bool up = (i & k) == 0;
                const Key a = keys[i], b = keys[partner];
                if ((a > b) == up) {
                    keys[i] = b;
                    keys[partner] = a;
                }
            }
            __syncwarp();
        }
    }
}

// --------------------------------------------------------------- randomness

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z) {
    // splitmix64 finaliser (Steele, Lea, Flood 2014).
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

// Draw t of node [start, end) at the given attempt: a position in [start, end).
__host__ __device__ __forceinline__ uint32_t counter_position(uint64_t seed, uint32_t rep, uint32_t start, uint32_t end,
                                                              uint32_t attempt, uint32_t t) {
    uint64_t h = mix64(seed + 0x9e3779b97f4a7c15ULL * (static_cast<uint64_t>(rep) + 1));
    h = mix64(h ^ ((static_cast<uint64_t>(start) << 32) | end));
    h = mix64(h ^ ((static_cast<uint64_t>(attempt) << 32) | t));
    const uint64_t n = end - start;
    return start + static_cast<uint32_t>(((h >> 32) * n) >> 32);
}

}  // namespace knng
