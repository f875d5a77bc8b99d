// Precision form of the bucket pass (KNNG_PRECISION_BF16_RERANK): the
// reference's addCandidatesLessThan (src/KnnSets.hpp:131-160) offers every
// other bucket member to a point's set with its exact FP32 distance.  Here the
// bucket's distances are first estimated on the tensor cores and only each
// point's 128 best candidates are offered, with exact distances:
//
//   1. the bucket's rows, centred on its first point, are rounded to BF16 and
//      multiplied on the tensor cores (tcgen05.mma kind::f16, FP32
//      accumulation): approx(i, j) = |x_i'|^2 + |x_j'|^2 - 2 bf16(x_i').bf16(x_j'),
//      with the norms of the FP32 centred rows; a block of 32 rows against a
//      tile of 128 columns at a time lands in TMEM and goes to shared memory;
//   2. one warp per row keeps the 128 smallest (estimate, bucket position)
//      keys seen so far, in bucket order: with a tile's 128 new keys there are
//      at most 256, eight a lane, and the bound between the 128 smallest and the
//      rest is found by bisection on the estimates' bits;
//   3. each kept candidate gets the exact FP32 distance in the reference's
//      order and is offered to the point's set in bucket position order (the
//      order of the FP32 form), through the same warp-resident set update.
//
// Buckets of at most 1024 points (max_leaf <= 1025).  The result differs from
// the FP32 form only where a candidate outside a point's 128 best estimates
// would have entered its set.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "context.hpp"
#include "dispatch.hpp"
#include "tc.cuh"
#include "tile16.cuh"

namespace knng {
namespace {

constexpr int kBfThreads = 512;
constexpr int kBfWarps = kBfThreads / kWarp;  // 16
constexpr int kBfPerSm = 2;
constexpr int kBfRows = 32;    // rows per block, two a warp
constexpr int kBfCols = 128;   // MMA N: columns per tile
constexpr int kBfTile = 128;   // MMA M
constexpr int kKeep = 128;     // candidates re-ranked per point
constexpr int kBfMaxBucket = 1024;
constexpr int kEstStride = kBfCols + 4;  // whole 16-byte stores, rows in different banks

template <int D>
struct BfLayout {
    using T = Tile16<D>;
    // A tile (the block's rows; the MMA's other 96 rows read on into what
    // follows, and nobody reads their products), B tile, estimates of a tile,
    // kept estimates and positions per row, member marks per row, norms and ids
    // of the bucket.
    static constexpr uint32_t a = 0;
    static constexpr uint32_t b = a + T::bytes(kBfRows);
    static constexpr uint32_t est = b + T::bytes(kBfCols);
    static constexpr uint32_t kept_v = est + kBfRows * kEstStride * 4;
    static constexpr uint32_t kept_j = kept_v + kBfRows * kKeep * 4;
    static constexpr uint32_t marks = kept_j + kBfRows * kKeep * 2;
    static constexpr uint32_t norms = marks + kBfRows * (kBfMaxBucket / kWarp) * 4;
    static constexpr uint32_t ids = norms + kBfMaxBucket * 4;
    static constexpr uint32_t bytes = ids + kBfMaxBucket * 4;
    static_assert((T::CH - 1) * T::stride(kBfRows) + kBfTile * 16 <= est, "the MMA's last rows stay in the tiles");
};

// norms[position] = squared norm of the bucket row at that position minus the
// bucket's first row, in FP32, dimensions in order.  A CTA per bucket.
template <int D>
__global__ void __launch_bounds__(256)
    k_bf16_norms(const uint32_t* __restrict__ starts, const uint32_t* __restrict__ ends, uint32_t count,
                 const uint32_t* __restrict__ dcount, const uint32_t* __restrict__ idx, const float* __restrict__ pts,
                 int ld, float* __restrict__ norms) {
    __shared__ __align__(16) float centre[D];
    if (dcount) count = *dcount;
    for (uint32_t leaf = blockIdx.x; leaf < count; leaf += gridDim.x) {
        const uint32_t s = starts[leaf], b = ends[leaf] - s;
        if (b < 2 || b - 1 <= static_cast<uint32_t>(kKeep)) continue;  // uniform: no estimates are made
        __syncthreads();  // the last bucket's centre is read
        for (int k = threadIdx.x; k < D; k += blockDim.x) centre[k] = pts[static_cast<size_t>(idx[s]) * ld + k];
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < b; t += blockDim.x) {
            const float4* row = reinterpret_cast<const float4*>(pts + static_cast<size_t>(idx[s + t]) * ld);
            float sum = 0.f;
#pragma unroll 5
            for (int q = 0; q < D / 4; ++q) {
                const float4 x = __ldg(row + q);
                const float4 m = reinterpret_cast<const float4*>(centre)[q];
                float v = __fsub_rn(x.x, m.x);
                sum = __fmaf_rn(v, v, sum);
                v = __fsub_rn(x.y, m.y);
                sum = __fmaf_rn(v, v, sum);
                v = __fsub_rn(x.z, m.z);
                sum = __fmaf_rn(v, v, sum);
                v = __fsub_rn(x.w, m.w);
                sum = __fmaf_rn(v, v, sum);
            }
            norms[s + t] = sum;
        }
    }
}

// Merges a tile's columns cb .. (below b, not i) into a row's kept list
// (kv, kj)[0 .. n) of estimates and positions, ascending by position: keeps the
// kKeep smallest (estimate, position) of both; returns the new count.  One warp.
__device__ __forceinline__ uint32_t keep_smallest(uint32_t* __restrict__ kv, uint16_t* __restrict__ kj, uint32_t n,
                                                  const float* __restrict__ est, uint32_t cb, uint32_t b, uint32_t i,
                                                  int lane) {
    constexpr int KR = kKeep / kWarp, NR = kBfCols / kWarp;  // registers of kept and of new keys
    const unsigned lt = (1u << lane) - 1u;
    uint32_t v[KR + NR], j[KR + NR];
    bool in[KR + NR];
#pragma unroll
    for (int r = 0; r < KR; ++r) {
        const uint32_t t = r * kWarp + lane;
        in[r] = t < n;
        v[r] = in[r] ? kv[t] : ~0u;
        j[r] = in[r] ? kj[t] : 0u;
    }
    uint32_t total = n;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const uint32_t c = r * kWarp + lane;
        j[KR + r] = cb + c;
        in[KR + r] = cb + c < b && cb + c != i;
        v[KR + r] = in[KR + r] ? __float_as_uint(est[c]) : ~0u;
        total += __popc(__ballot_sync(kFull, in[KR + r]));
    }
    __syncwarp();  // the list is read before it is rewritten
    // Keep v < limit, and the first `ties` of v == limit.
    uint32_t limit = ~0u, ties = 0;
    bool all = total <= static_cast<uint32_t>(kKeep);
    if (!all) {
        uint32_t lo = ~0u, hi = 0;
#pragma unroll
        for (int r = 0; r < KR + NR; ++r) {
            lo = min(lo, v[r]);
            hi = max(hi, in[r] ? v[r] : 0u);
        }
        lo = __reduce_min_sync(kFull, lo);
        hi = __reduce_max_sync(kFull, hi) + 1u;  // estimates are at most infinity
        // count(v < lo) <= kKeep < count(v < hi)
        uint32_t below = 0;
        for (;;) {
            if (hi - lo <= 1u) {
                limit = lo;
                ties = kKeep - below;
                break;
            }
            const uint32_t mid = lo + (hi - lo) / 2;
            uint32_t c = 0;
#pragma unroll
            for (int r = 0; r < KR + NR; ++r) c += v[r] < mid ? 1u : 0u;
            c = __reduce_add_sync(kFull, c);
            if (c == static_cast<uint32_t>(kKeep)) {
                limit = mid;
                break;
            }
            if (c < static_cast<uint32_t>(kKeep)) {
                lo = mid;
                below = c;
            } else {
                hi = mid;
            }
        }
    }
    uint32_t at = 0;
#pragma unroll
    for (int r = 0; r < KR + NR; ++r) {
        bool keep = in[r] && (all || v[r] < limit);
        if (ties > 0) {  // warp-uniform
            const bool tie = in[r] && v[r] == limit;
            const unsigned m = __ballot_sync(kFull, tie);
            keep = keep || (tie && static_cast<uint32_t>(__popc(m & lt)) < ties);
            ties -= min(ties, static_cast<uint32_t>(__popc(m)));
        }
        const unsigned m = __ballot_sync(kFull, keep);
        if (keep) {
            const uint32_t to = at + __popc(m & lt);
            kv[to] = v[r];
            kj[to] = static_cast<uint16_t>(j[r]);
        }
        at += __popc(m);
    }
    __syncwarp();
    return at;
}

// A persistent grid takes blocks of 32 rows of the buckets from the work
// counter.  `own`: the sets hold distances of these points, so their members
// (marked beforehand by bucket position, `pos`) are left out of the offers.
//
// What bounds it: issue slots, shared by the offers, the exact distances of 128
// candidates a point (rows from L1 and L2) and the selection (some 300
// instructions a row and tile).  A thread per row with a 128-key heap in shared
// memory took 52.9 ms for the eight passes of a 100k x 100 build (buckets of up
// to 256), this 6.4.
template <int D>
__global__ void __launch_bounds__(kBfThreads, kBfPerSm)
    k_leaf_bf16(const uint32_t* __restrict__ starts, const uint32_t* __restrict__ ends,
                const uint32_t* __restrict__ idx, const uint32_t* __restrict__ pos, const float* __restrict__ norms_g,
                const float* __restrict__ pts, int ld, float* __restrict__ set_dist, uint32_t* __restrict__ set_id,
                uint32_t* __restrict__ set_size, uint32_t* __restrict__ set_maxslot, float* __restrict__ set_bound, int K,
                bool own, uint32_t* __restrict__ error_flag, LeafItems items,
                const uint32_t* __restrict__ n_items, uint32_t* __restrict__ work) {
    using L = BfLayout<D>;
    using T = Tile16<D>;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* A = smem + L::a;
    unsigned char* B = smem + L::b;
    float* est = reinterpret_cast<float*>(smem + L::est);
    uint32_t* kept_v = reinterpret_cast<uint32_t*>(smem + L::kept_v);
    uint16_t* kept_j = reinterpret_cast<uint16_t*>(smem + L::kept_j);
    uint32_t* marks = reinterpret_cast<uint32_t*>(smem + L::marks);
    float* norms = reinterpret_cast<float*>(smem + L::norms);
    uint32_t* ids = reinterpret_cast<uint32_t*>(smem + L::ids);
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ uint32_t next_s;
    __shared__ uint8_t place_s[kBfWarps][kWarp];
    constexpr int P = kBfRows / kBfWarps;
    constexpr uint32_t kMarkWords = kBfMaxBucket / kWarp;
    const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
    // The tiles' padding (dimensions past D) stays zero.
    for (uint32_t f = tid; f < L::est / 16; f += kBfThreads) reinterpret_cast<uint4*>(smem)[f] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) tc::tmem_alloc(&tmem_slot, kBfCols);
    if (tid == 0) {
        tc::mbar_init(&mbar, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    uint32_t phase = 0;
    bool healthy = true;
    const uint32_t idesc = tc::idesc_bf16(kBfTile, kBfCols);
    const uint32_t total = *n_items;
    while (healthy) {
        if (tid == 0) next_s = atomicAdd(work, 1u);
        __syncthreads();
        const int64_t w = next_s;
        if (w >= total) break;
        const uint32_t leaf = items.leaf[-w], rb = items.row[-w];
        const uint32_t s0 = starts[leaf], b = ends[leaf] - s0;
        // Buckets of at most 129 points keep every other member: no estimates.
        const bool keep_all = b - 1 <= static_cast<uint32_t>(kKeep);
        for (uint32_t t = tid; t < b; t += kBfThreads) {
            ids[t] = idx[s0 + t];
            if (!keep_all) norms[t] = norms_g[s0 + t];
        }
        __syncthreads();
        const uint32_t cnt = min(static_cast<uint32_t>(kBfRows), b - rb);
        uint32_t kept[P];
#pragma unroll
        for (int u = 0; u < P; ++u) kept[u] = 0;
        if (keep_all) {
#pragma unroll
            for (int u = 0; u < P; ++u) {
                const uint32_t row = warp * P + u, i = rb + row;
                if (row < cnt) {
                    for (uint32_t t = lane; t + 1 < b; t += kWarp)
                        kept_j[row * kKeep + t] = static_cast<uint16_t>(t < i ? t : t + 1);
                    kept[u] = b - 1;
                }
            }
        } else {
            float4 centre = make_float4(0.f, 0.f, 0.f, 0.f);
            centre = __ldg(reinterpret_cast<const float4*>(pts + static_cast<size_t>(ids[0]) * ld) + lane % T::Q);
            const uint32_t a_row = lane * kBfWarps + warp;
            tile_rows<D, kBfRows, kBfWarps, __nv_bfloat16>(pts, ld, lane < P && a_row < cnt ? ids[rb + a_row] : 0u, cnt,
                                                           A, T::stride(kBfRows), centre, lane, warp);
            for (uint32_t cb = 0; cb < b; cb += kBfCols) {
                const uint32_t cols = min(static_cast<uint32_t>(kBfCols), b - cb);
                const uint32_t b_row = lane * kBfWarps + warp;
                tile_rows<D, kBfCols, kBfWarps, __nv_bfloat16>(
                    pts, ld, lane < kBfCols / kBfWarps && b_row < cols ? ids[cb + b_row] : 0u, cols, B,
                    T::stride(kBfCols), centre, lane, warp);
                tc::fence_proxy_async();
                tc::fence_before_sync();
                __syncthreads();
                if (tid == 0) {
                    tc::fence_after_sync();
                    tc::issue_tile_strided(tmem, tc::smem_u32(A), tc::smem_u32(B), T::stride(kBfRows),
                                           T::stride(kBfCols), T::KP, idesc);
                    tc::mma_commit(&mbar);
                }
                const bool done = tc::mbar_wait(&mbar, phase);
                phase ^= 1u;
                if (__syncthreads_or(!done)) {
                    if (tid == 0) atomicExch(error_flag, 1u);
                    tc::mbar_wait(&mbar, phase ^ 1u);
                    healthy = false;
                    break;
                }
                tc::fence_after_sync();
                // The warps whose TMEM quarter holds the block's rows: 32 columns each.
                if (warp % 4 == 0) {
                    const float na = rb + lane < b ? norms[rb + lane] : 0.f;
                    const uint32_t c0 = warp / 4 * kWarp;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float g[16];
                        tc::tmem_ld16(tmem + c0 + 16 * h, g);
                        tc::tmem_wait_ld();
                        float* out = est + lane * kEstStride + c0 + 16 * h;
#pragma unroll
                        for (int u = 0; u < 16; u += 4) {
                            float e[4];
#pragma unroll
                            for (int x = 0; x < 4; ++x) {
                                const uint32_t j = cb + c0 + 16 * h + u + x;
                                e[x] = fmaxf(0.f, na + (j < b ? norms[j] : 0.f) - 2.0f * g[u + x]);
                            }
                            *reinterpret_cast<float4*>(out + u) = make_float4(e[0], e[1], e[2], e[3]);
                        }
                    }
                }
                tc::fence_before_sync();
                __syncthreads();
#pragma unroll
                for (int u = 0; u < P; ++u) {
                    const uint32_t row = warp * P + u;
                    if (row < cnt)
                        kept[u] = keep_smallest(kept_v + row * kKeep, kept_j + row * kKeep, kept[u],
                                                est + row * kEstStride, cb, b, rb + row, lane);
                }
            }
            if (!healthy) break;
        }
        __syncwarp();
        // Offers: each warp its rows' kept candidates, 32 at a time, in bucket order.
#pragma unroll 1
        for (int u = 0; u < P; ++u) {
            const uint32_t row = warp * P + u;
            if (row >= cnt) break;
            const uint32_t p = ids[rb + row];
            const uint32_t nk = u == 0 ? kept[0] : kept[P - 1];
            WarpSet s;
            set_load(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
            uint32_t* mark = marks + row * kMarkWords;
            if (own) {
                for (uint32_t t = lane; t < kMarkWords; t += kWarp) mark[t] = 0u;
                __syncwarp();
#pragma unroll
                for (int r = 0; r < kSlotsPerLane; ++r) {
                    if (lane + r * kWarp < static_cast<int>(s.size)) {
                        const uint32_t at = pos[s.id[r]] - s0;
                        if (at < b) atomicOr(&mark[at / kWarp], 1u << (at % kWarp));
                    }
                }
                __syncwarp();
            }
            ChainRow<D> mine;
            load_chain_row<D>(mine, pts + static_cast<size_t>(p) * ld, lane & 7);
            for (uint32_t t0 = 0; t0 < nk; t0 += kWarp) {
                const bool valid = t0 + lane < nk;
                const uint32_t j = kept_j[row * kKeep + min(t0 + lane, nk - 1)];
                const uint32_t cand = ids[j];
                const float d = warp_distances<D, 2>(mine, cand, pts, ld, lane);
                if (own)
                    set_offer_new_batch(s, cand, d, valid && !((mark[j / kWarp] >> (j % kWarp)) & 1u), K, lane,
                                        place_s[warp]);
                else
                    set_offer_batch(s, cand, d, valid, K, lane);
            }
            set_store(s, set_dist, set_id, set_size, set_maxslot, set_bound, p, K, lane);
        }
        __syncthreads();  // everyone is done with ids, the tiles and the work word
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, kBfCols);
    }
}

// One 128 x 128 BF16 tile of a(m x D) . b(n x D)^T with FP32 accumulation
// (rows past m / n are zero); the diagnostic behind knng_debug_tile_gram_bf16.
template <int D>
__global__ void __launch_bounds__(kBfThreads, 1)
    k_tile_gram_bf16(const float* __restrict__ a, uint32_t m, const float* __restrict__ b, uint32_t n,
                     float* __restrict__ out, uint32_t* __restrict__ error_flag) {
    using T = Tile16<D>;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* A = smem;
    unsigned char* B = smem + T::bytes(kBfTile);
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
    for (uint32_t f = tid; f < 2 * T::bytes(kBfTile) / 16; f += kBfThreads)
        reinterpret_cast<uint4*>(smem)[f] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) tc::tmem_alloc(&tmem_slot, kBfCols);
    if (tid == 0) {
        tc::mbar_init(&mbar, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t id = lane < kBfTile / kBfWarps ? lane * kBfWarps + warp : 0u;
    tile_rows<D, kBfTile, kBfWarps, __nv_bfloat16>(a, D, id, m, A, T::stride(kBfTile), zero, lane, warp);
    tile_rows<D, kBfTile, kBfWarps, __nv_bfloat16>(b, D, id, n, B, T::stride(kBfTile), zero, lane, warp);
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
        tc::fence_after_sync();
        tc::issue_tile_strided(tmem, tc::smem_u32(A), tc::smem_u32(B), T::stride(kBfTile), T::stride(kBfTile), T::KP,
                               tc::idesc_bf16(kBfTile, kBfCols));
        tc::mma_commit(&mbar);
    }
    const bool done = tc::mbar_wait(&mbar, 0);
    if (__syncthreads_or(!done)) {
        if (tid == 0) atomicExch(error_flag, 1u);
    } else if (warp < 4) {
        tc::fence_after_sync();
        const uint32_t row = static_cast<uint32_t>(warp * kWarp + lane);
        for (uint32_t j0 = 0; j0 < kBfCols; j0 += 16) {
            float g[16];
            tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * kWarp) << 16) + j0, g);
            tc::tmem_wait_ld();
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (row < m && j0 + u < n) out[static_cast<size_t>(row) * n + j0 + u] = g[u];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, kBfCols);
    }
}

}  // namespace

void run_tile_gram_bf16(Context& c, uint32_t d, const float* d_a, uint32_t m, const float* d_b, uint32_t n,
                        float* d_out) {
    auto* err = static_cast<uint32_t*>(scratch(c, "gram_error", sizeof(uint32_t)));
    KNNG_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), c.stream));
    KNNG_DISPATCH_D(d, {
        auto kern = k_tile_gram_bf16<D>;
        allow_max_smem(c, kern);
        kern<<<1, kBfThreads, 2 * Tile16<D>::bytes(kBfTile), c.stream>>>(d_a, m, d_b, n, d_out, err);
    });
    ++c.launches;
    KNNG_CUDA(cudaGetLastError());
    uint32_t h = 0;
    download(c, &h, err, 1);
    if (h) fail(KNNG_ERR_CUDA, "BF16 tile: the MMA completion wait gave up");
}

namespace {

// The pass over the buckets [0, count) or [0, *dcount): its items and norms, then
// a persistent grid.  *n_items and *work start at 0.
void enqueue_bf16(Context& c, uint32_t count, const uint32_t* d_starts, const uint32_t* d_ends, const uint32_t* dcount,
                  LeafItems items, uint32_t* n_items, uint32_t* work, float* norms, uint32_t* d_error) {
    uint32_t* pos = launch_leaf_items(c, count, d_starts, d_ends, dcount, kBfRows, items, n_items);
    KNNG_DISPATCH_D(c.d, {
        k_bf16_norms<D><<<c.sms * 8, 256, 0, c.stream>>>(d_starts, d_ends, count, dcount, c.indices, c.points, c.ld, norms);
        auto kern = k_leaf_bf16<D>;
        allow_max_smem(c, kern);
        kern<<<kBfPerSm * c.sms, kBfThreads, BfLayout<D>::bytes, c.stream>>>(
            d_starts, d_ends, c.indices, pos, norms, c.points, c.ld, c.set_dist, c.set_id, c.set_size, c.set_maxslot,
            c.set_bound, static_cast<int>(c.k), c.dists_own, d_error, items, n_items, work);
    });
    c.launches += 2;
    KNNG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_leaves_bf16(Context& c, uint32_t count, const uint32_t* d_starts, const uint32_t* d_ends,
                        uint32_t max_bucket) {
    if (count == 0) return;
    if (max_bucket > static_cast<uint32_t>(kBfMaxBucket))
        fail(KNNG_ERR_INVALID_ARGUMENT, "the BF16 bucket pass takes buckets of at most 1024 points");
    // Item count, work counter, error word; the items; the norms.
    const size_t cap = c.n / kBfRows + static_cast<size_t>(count) + 1;
    auto* lists = static_cast<uint32_t*>(spare_take(c, kSpareLeafLists, (3 + 2 * cap + c.n) * sizeof(uint32_t)));
    spare_done(c, kSpareLeafLists, kSpareLeafLists);  // nothing is allocated before the pass is on the stream
    KNNG_CUDA(cudaMemsetAsync(lists, 0, 3 * sizeof(uint32_t), c.stream));
    enqueue_bf16(c, count, d_starts, d_ends, nullptr, {lists + 2 + cap, lists + 2 + 2 * cap}, lists, lists + 1,
                 reinterpret_cast<float*>(lists + 3 + 2 * cap), lists + 2);
    uint32_t h = 0;
    download(c, &h, lists + 2, 1);
    if (h) fail(KNNG_ERR_CUDA, "BF16 bucket pass: the MMA completion wait gave up");
}

void prepare_leaves_bf16_list(Context& c) {
    KNNG_DISPATCH_D(c.d, { allow_max_smem(c, k_leaf_bf16<D>); });
}

void launch_leaves_bf16_list(Context& c, uint32_t* d_starts, uint32_t* d_ends, uint32_t cap, const uint32_t* d_count,
                             uint32_t* d_n_items, uint32_t* d_work, float* d_norms, uint32_t* d_error) {
    enqueue_bf16(c, 0, d_starts, d_ends, d_count, {d_starts + cap - 1, d_ends + cap - 1}, d_n_items, d_work, d_norms,
                 d_error);
}

}  // namespace knng
