// Neighbour search of the DFSPH step: ParticleSearch::FindNeighbors
// (Simulation/DFSPH/ParticleSearch/ParticleSearch.h:80-93, ParticleSearch.cu:29-195,
// ParticleSearchKernels.cu:40-193) rebuilt for GB300:
//   * the grid (bounds, dimensions, Morton meta-grid keys) is computed on the
//     device, per scene, with the reference's float arithmetic (IEEE-rounded
//     intrinsics, no contraction), so no host round trip is needed;
//   * the counting sort is deterministic: within a cell, particles are ordered
//     by original index (the reference's atomicAdd rank allows any order);
//   * the carried state is gathered into cell order (coalesced float4 rows for
//     every later kernel) instead of being read through an index;
//   * neighbour lists are rows of kRow slots per particle (row-major), capped at 70
//     in the reference's z, y, x cell order; one pass, no count/scan/query split.
#include "dfsph_common.cuh"
#include "dfsph_halo.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace vfd {

constexpr uint32_t kScanItems = 1024u;  // cells per scan block (256 threads x 4)

__device__ __forceinline__ bool aborted(const Dev& d) { return is_aborted(d); }

// Cell of edge h around x; false (with the status set) when x is not finite.
__device__ __forceinline__ bool position_cell(const Dev& d, SceneDev& S, float3 x, int* c) {
    if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z))) {
        atomicOr(&S.flags, 0x10u);
        atomicOr(d.status, 0x10u);
        atomicExch(d.status + 1, 1u);
        return false;
    }
    const float p[3] = {x.x, x.y, x.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float q = floorf(__fdiv_rn(p[k], S.h));
        // positions beyond +-2^30 cells cannot be gridded; flag them.
        const bool in = fabsf(q) < 1.0e9f;
        if (!in) { atomicOr(d.status, 0x20u); atomicExch(d.status + 1, 1u); }
        c[k] = in ? (int)q : 0;
    }
    return true;
}

// Search-grid key of a position (N2), or kNoKey with the status set.
constexpr uint32_t kNoKey = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t position_key(const Dev& d, const SceneDev& S, float3 x, uint32_t total) {
    const float p[3] = {x.x, x.y, x.z};
    int c[3];
#pragma unroll
    for (int k = 0; k < 3; k++) c[k] = (int)__fmul_rn(__fsub_rn(p[k], S.gridMin[k]), S.gridDelta[k]);
    const uint32_t key = S.cellBase + cell_key(S, c[0], c[1], c[2]);
    if (key >= total || c[0] < 0 || c[1] < 0 || c[2] < 0) {  // cannot happen for finite input
        atomicOr(d.status, 0x20u);
        atomicExch(d.status + 1, 1u);
        return kNoKey;
    }
    return key;
}

// N1: ComputeMinMaxKernel (ParticleSearchKernels.cu:40-62) on the current positions.
__global__ void __launch_bounds__(kBlock) k_minmax(Dev d) {
    VFD_COUNT_LAUNCH(d);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < d.n;
    const uint32_t sid = valid ? scene_of(d, i) : 0u;
    int c[3] = {INT_MAX, INT_MAX, INT_MAX};
    int cmax[3] = {INT_MIN, INT_MIN, INT_MIN};
    if (valid) {
        const float4 x4 = d.XN[i];
        const float3 x = abs_pos(d, d.scenes[sid], x4);
        if (position_cell(d, d.scenes[sid], x, c))
            for (int k = 0; k < 3; k++) cmax[k] = c[k];
    }
    const uint32_t s0 = __shfl_sync(0xffffffffu, sid, 0);
    const bool uniform = __all_sync(0xffffffffu, !valid || sid == s0);
    const uint32_t bucket = blockIdx.x % kBuckets;
    if (uniform) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int mn = __reduce_min_sync(0xffffffffu, c[k]);
            const int mx = __reduce_max_sync(0xffffffffu, cmax[k]);
            if ((threadIdx.x & 31u) == 0 && mn != INT_MAX) {
                atomicMin(mm_bucket(d, s0, k, bucket), mn);
                atomicMax(mm_bucket(d, s0, 3 + k, bucket), mx);
            }
        }
    } else if (valid) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            atomicMin(mm_bucket(d, sid, k, bucket), c[k]);
            atomicMax(mm_bucket(d, sid, 3 + k, bucket), cmax[k]);
        }
    }
}

// ComputeCellInformation of a scene whose cell bounds are known.
__device__ void scene_grid(SceneDev& S) {
    const float R = S.h;
    uint32_t cells = 1u;
    bool ok = S.count > 0;
    for (int k = 0; k < 3; k++) {
        const float bmin = __fmul_rn((float)S.minCell[k], R);
        const float bmax = __fmul_rn((float)(S.maxCell[k] + 1), R);
        const float size = __fsub_rn(bmax, bmin);
        const float q = ceilf(__fdiv_rn(size, R));
        const uint32_t dim = (ok && q >= 0.0f && q < 1.0e7f) ? (uint32_t)q + 4u : 4u;
        S.dim[k] = dim;
        S.gridMin[k] = __fsub_rn(bmin, __fmul_rn(R, 2.0f));
        S.meta[k] = (uint32_t)ceilf(__fdiv_rn((float)dim, 8.0f));
        const float gs = __fmul_rn((float)dim, R);
        S.gridDelta[k] = __fdiv_rn((float)dim, gs);
        cells = (cells > 0xFFFFFFFFu / 8u) ? 0xFFFFFFFFu : cells * S.meta[k];
    }
    S.cellCount = (!ok) ? 0u : ((cells > 0xFFFFFFFFu / 512u) ? 0xFFFFFFFFu : cells * 512u);
}

// ParticleSearch::ComputeMinMax tail + ComputeCellInformation (ParticleSearch.cu:50-86),
// per scene, then the scene cell bases (exclusive scan) and the capacity check. With one
// scene the first warp folds the N1 buckets (lane b takes bucket b, an xor butterfly of
// min / max) instead of one thread walking them: 192 dependent L2 round trips were ~27 us,
// most of a small scene's search.
__global__ void k_grid(Dev d) {
    VFD_COUNT_LAUNCH(d);
    __shared__ uint32_t total;
    __shared__ int foldMin[3], foldMax[3];
    const bool one = d.nscenes == 1;
    if (one && threadIdx.x < 32u) {
        const uint32_t b = threadIdx.x;
        for (int k = 0; k < 3; k++) {  // fold the N1 buckets, reset them for the next step
            int32_t* qa = mm_bucket(d, 0, k, b);
            int32_t* qb = mm_bucket(d, 0, 3 + k, b);
            int mn = *qa, mx = *qb;
            *qa = INT_MAX;
            *qb = INT_MIN;
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            if (b == 0) {
                foldMin[k] = mn;
                foldMax[k] = mx;
            }
        }
        *max_bucket(d, 0, 1, b) = 0u;
    }
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < d.nscenes; s += blockDim.x) {
        SceneDev& S = d.scenes[s];
        if (one) {
            for (int k = 0; k < 3; k++) {
                S.minCell[k] = foldMin[k];
                S.maxCell[k] = foldMax[k];
            }
        } else {
            for (int k = 0; k < 3; k++) {  // fold the N1 buckets, reset them for the next step
                int mn = INT_MAX, mx = INT_MIN;
                for (uint32_t b = 0; b < kBuckets; b++) {
                    int32_t* qa = mm_bucket(d, s, k, b);
                    int32_t* qb = mm_bucket(d, s, 3 + k, b);
                    mn = min(mn, *qa);
                    mx = max(mx, *qb);
                    *qa = INT_MAX;
                    *qb = INT_MIN;
                }
                S.minCell[k] = mn;
                S.maxCell[k] = mx;
            }
            for (uint32_t b = 0; b < kBuckets; b++) *max_bucket(d, s, 1, b) = 0u;
        }
        scene_grid(S);
        S.flags = 0u;
        if (halo_on(d)) d.haloScene[s] = make_uint2(0xFFFFFFFFu, 0u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint64_t acc = 0;
        for (uint32_t s = 0; s < d.nscenes; s++) {
            d.scenes[s].cellBase = (uint32_t)min(acc, (uint64_t)0xFFFFFFFFu);
            acc += d.scenes[s].cellCount;
        }
        total = (uint32_t)min(acc, (uint64_t)0xFFFFFFFFu);
        d.status[2] = total;
        if (halo_on(d))
            for (int k = 0; k < 6; k++) d.haloInfo[k] = 0u;
        if (acc > d.cellCap) {
            atomicOr(d.status, 0x20u);
            atomicExch(d.status + 1, 1u);
        }
    }
}

__global__ void __launch_bounds__(256) k_clear_cells(Dev d) {
    VFD_COUNT_LAUNCH(d);
    if (aborted(d)) return;
    const uint32_t total = d.status[2];
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
        d.CELL_COUNT[c] = 0u;
        d.FILL[c] = 0u;
    }
}

// N2: InsertParticlesMortonKernel (ParticleSearchKernels.cu:64-78), count part.
__global__ void __launch_bounds__(kBlock) k_keys(Dev d) {
    VFD_COUNT_LAUNCH(d);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n || aborted(d)) return;
    const SceneDev& S = d.scenes[scene_of(d, i)];
    const float3 x = abs_pos(d, S, d.XN[i]);
    const uint32_t key = position_key(d, S, x, d.status[2]);
    if (key == kNoKey) return;
    d.KEY[i] = key;
    atomicAdd(d.CELL_COUNT + key, 1u);
}

// N3: exclusive scan of the cell counts (thrust::exclusive_scan, ParticleSearch.cu:111-115),
// three phases over the device-known number of cells. With staged tiles the same phases count
// and list the non-empty tiles in cell order (a thread owns four consecutive cells, so a
// tile is a run of kTileLanes lanes).
constexpr uint32_t kTileLanes = kHaloTileCells / 4u;
static_assert(kTileLanes <= 32u && kScanItems % kHaloTileCells == 0u, "a tile lies in one warp's cells");

__global__ void __launch_bounds__(256) k_scan_reduce(Dev d) {
    VFD_COUNT_LAUNCH(d);
    if (aborted(d)) return;
    const uint32_t total = d.status[2];
    const uint32_t base = blockIdx.x * kScanItems;
    if (base >= total) return;
    uint32_t s = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4u; k++) {
        const uint32_t c = base + threadIdx.x * 4u + k;
        if (c < total) s += d.CELL_COUNT[c];
    }
    const uint32_t filled = __ballot_sync(0xffffffffu, s > 0u);
    s = __reduce_add_sync(0xffffffffu, s);
    __shared__ uint32_t ws[8], wt[8];
    if ((threadIdx.x & 31u) == 0) {
        uint32_t tiles = 0;
#pragma unroll
        for (uint32_t k = 0; k < 32u; k += kTileLanes) tiles += (filled >> k & ((1u << kTileLanes) - 1u)) ? 1u : 0u;
        ws[threadIdx.x >> 5] = s;
        wt[threadIdx.x >> 5] = tiles;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0, n = 0;
        for (int w = 0; w < 8; w++) {
            t += ws[w];
            n += wt[w];
        }
        d.SCAN[blockIdx.x] = t;
        if (halo_on(d)) d.haloScan[blockIdx.x] = n;
    }
}

__device__ __forceinline__ uint32_t block_exclusive_scan_1024(uint32_t v, uint32_t& blockTotal) {
    // 1024 threads; returns the exclusive prefix of v within the block
    __shared__ uint32_t ws[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += y;
        }
        ws[lane] = w;
    }
    __syncthreads();
    const uint32_t warpPrefix = warp ? ws[warp - 1] : 0u;
    blockTotal = ws[31];
    __syncthreads();
    return warpPrefix + x - v;
}

__global__ void __launch_bounds__(1024) k_scan_top(Dev d) {
    VFD_COUNT_LAUNCH(d);
    if (aborted(d)) return;
    const uint32_t total = d.status[2];
    const uint32_t nb = (total + kScanItems - 1) / kScanItems;
    uint32_t carry = 0, tiles = 0;
    for (uint32_t base = 0; base < nb; base += 1024u) {
        const uint32_t k = base + threadIdx.x;
        const uint32_t v = k < nb ? d.SCAN[k] : 0u;
        uint32_t tot;
        const uint32_t ex = block_exclusive_scan_1024(v, tot);
        if (k < nb) d.SCAN[k] = carry + ex;
        carry += tot;
        if (halo_on(d)) {
            const uint32_t n = k < nb ? d.haloScan[k] : 0u;
            const uint32_t before = block_exclusive_scan_1024(n, tot);
            if (k < nb) d.haloScan[k] = tiles + before;
            tiles += tot;
        }
    }
    if (halo_on(d) && threadIdx.x == 0) d.haloInfo[0] = tiles;
}

__global__ void __launch_bounds__(256) k_scan_down(Dev d) {
    VFD_COUNT_LAUNCH(d);
    if (aborted(d)) return;
    const uint32_t total = d.status[2];
    const uint32_t base = blockIdx.x * kScanItems;
    if (base >= total) return;
    __shared__ uint32_t ws[8];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // each thread owns 4 consecutive cells
    uint32_t v[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t c = base + threadIdx.x * 4u + k;
        v[k] = c < total ? d.CELL_COUNT[c] : 0u;
        s += v[k];
    }
    uint32_t x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    uint32_t wp = 0;
    for (uint32_t w = 0; w < warp; w++) wp += ws[w];
    uint32_t run = d.SCAN[blockIdx.x] + wp + x - s;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t c = base + threadIdx.x * 4u + k;
        if (c < total) d.CELL_START[c] = run;
        run += v[k];
    }
    if (!halo_on(d)) return;
    // the tile of this thread's lanes, listed by its first lane after the tiles before it
    const uint32_t mask = ((1u << kTileLanes) - 1u) << (lane & ~(kTileLanes - 1u));
    const uint32_t filled = __ballot_sync(0xffffffffu, s > 0u);
    uint32_t inTile = s, before = 0, mine = 0;
#pragma unroll
    for (uint32_t o = kTileLanes / 2u; o > 0u; o >>= 1) inTile += __shfl_xor_sync(0xffffffffu, inTile, o);
#pragma unroll
    for (uint32_t k = 0; k < 32u; k += kTileLanes) {
        const uint32_t full = (filled >> k & ((1u << kTileLanes) - 1u)) ? 1u : 0u;
        mine += full;
        if (k < (lane & ~(kTileLanes - 1u))) before += full;
    }
    __shared__ uint32_t wt[8], rounds[2];  // of a block's threads over the tiles, narrow and wide
    if (lane == 0) wt[warp] = mine;
    if (threadIdx.x < 2u) rounds[threadIdx.x] = 0u;
    __syncthreads();
    for (uint32_t w = 0; w < warp; w++) before += wt[w];
    if (lane % kTileLanes == 0u && (filled & mask)) {
        const uint32_t at = d.haloScan[blockIdx.x] + before, first = run - s;
        HaloTile T = {};
        T.cell0 = base + threadIdx.x * 4u;
        T.first = first;
        T.last = first + inTile;
        T.scene = scene_of(d, first);
        d.haloTiles[at] = T;
        atomicMin(&d.haloScene[T.scene].x, at);
        atomicAdd(&d.haloScene[T.scene].y, 1u);
        atomicAdd(&rounds[0], halo_rounds(inTile, kHaloThreads));
        atomicAdd(&rounds[1], halo_rounds(inTile, kHaloWideThreads));
    }
    __syncthreads();
    if (threadIdx.x == 0 && rounds[0] > 0u) {
        HaloCounts* all = halo_counts(d);
        atomicAdd(&all->narrow, rounds[0]);
        atomicAdd(&all->wide, rounds[1]);
    }
}

// N4 (first half): CountingSortIndicesKernel's slot, here through a per-cell fill counter.
__global__ void __launch_bounds__(kBlock) k_slots(Dev d) {
    VFD_COUNT_LAUNCH(d);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n || aborted(d)) return;
    const uint32_t key = d.KEY[i];
    const uint32_t s = atomicAdd(d.FILL + key, 1u);
    d.TMP[d.CELL_START[key] + s] = i;
}

// N4 (second half): the deterministic in-cell rank (ascending original index) and the
// gather of the carried state into the new cell order.
__global__ void __launch_bounds__(kBlock) k_rank_gather(Dev d) {
    VFD_COUNT_LAUNCH(d);
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= d.n || aborted(d)) return;
    const uint32_t i = d.TMP[p];
    const uint32_t key = d.KEY[i];
    const uint32_t start = d.CELL_START[key], cnt = d.CELL_COUNT[key];
    const uint32_t pid = d.PIDc[i];
    uint32_t rank = 0;
    for (uint32_t q = start; q < start + cnt; q++) rank += (d.PIDc[d.TMP[q]] < pid) ? 1u : 0u;
    const uint32_t dst = start + rank;
    d.X[dst] = d.XN[i];
    d.V[dst] = d.Vc[i];
    d.DV[dst] = d.DVc[i];
    d.DK[dst] = d.DKc[i];
    d.PID[dst] = pid;
    d.KEYS[dst] = key;
}

// N1 to N4 of one small scene in one launch: a cluster of kSmallBlocks blocks, with a barrier
// of the cluster where the kernels above end. A thread keeps its particles' positions, keys and
// places in registers. Bound by latency: a round trip to the L2 and a barrier that waits for the
// stores before it take 1.3 to 2 us a phase, 15.8 us in all for 4,096 particles where the nine
// kernels take 35.3 (each timed alone).
constexpr uint32_t kSmallThreads = 1024u, kSmallPer = kSearchSmallMax / (kSmallBlocks * kSmallThreads);
static_assert(kSmallPer * kSmallBlocks * kSmallThreads == kSearchSmallMax && kSmallBlocks <= 8u, "portable clusters");
__global__ void __cluster_dims__(kSmallBlocks, 1, 1) __launch_bounds__(kSmallThreads) k_search_small(Dev d) {
    VFD_COUNT_LAUNCH(d);
    const cg::cluster_group cluster = cg::this_cluster();
    constexpr uint32_t T = kSmallBlocks * kSmallThreads;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t rank = cluster.block_rank(), t = rank * kSmallThreads + threadIdx.x;
    __shared__ int bounds[6];                                // of the block's particles
    __shared__ int warpBounds[6][kSmallThreads / 32u];
    __shared__ uint32_t blockCells;                          // particles in the block's cells
    __shared__ uint32_t before, stop;
    __shared__ __align__(16) unsigned char gridBytes[sizeof(SceneDev)];
    SceneDev& G = *reinterpret_cast<SceneDev*>(gridBytes);   // the scene's grid, as d.scenes[0] gets it
    SceneDev& S = d.scenes[0];

    float3 x[kSmallPer];
    int c[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
#pragma unroll
    for (uint32_t u = 0; u < kSmallPer; u++) {
        const uint32_t i = u * T + t;
        if (i >= d.n) break;
        x[u] = abs_pos(d, S, d.XN[i]);
        int q[3];
        if (!position_cell(d, S, x[u], q)) continue;
        for (int k = 0; k < 3; k++) {
            c[k] = min(c[k], q[k]);
            c[3 + k] = max(c[3 + k], q[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const int v = k < 3 ? __reduce_min_sync(0xffffffffu, c[k]) : __reduce_max_sync(0xffffffffu, c[k]);
        if (lane == 0) warpBounds[k][warp] = v;
    }
    __syncthreads();
    if (warp < 6u) {
        const int v = warpBounds[warp][lane];
        const int w = warp < 3u ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
        if (lane == 0) bounds[warp] = w;
    }
    cluster.sync();
    if (warp == 0) {
        int m[6];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const int v = cluster.map_shared_rank(bounds, lane % kSmallBlocks)[k];
            m[k] = k < 3 ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
        }
        if (lane == 0) {
            G.h = S.h;
            G.count = S.count;
            G.cellBase = 0u;
            for (int k = 0; k < 3; k++) {
                G.minCell[k] = m[k];
                G.maxCell[k] = m[3 + k];
            }
            scene_grid(G);
            // every block decides alike: the status changes again only behind the next barrier
            stop = (__ldcg(d.status + 1) != 0u || G.cellCount > d.cellCap) ? 1u : 0u;
        }
        if (rank == 0u) *max_bucket(d, 0, 1, lane) = 0u;
    }
    __syncthreads();
    const uint32_t total = G.cellCount;
    if (!stop)
        for (uint32_t i = t; i < total; i += T) d.CELL_COUNT[i] = 0u;
    cluster.sync();
    if (t == 0u) {
        for (int k = 0; k < 3; k++) {
            S.minCell[k] = G.minCell[k];
            S.maxCell[k] = G.maxCell[k];
            S.dim[k] = G.dim[k];
            S.meta[k] = G.meta[k];
            S.gridMin[k] = G.gridMin[k];
            S.gridDelta[k] = G.gridDelta[k];
        }
        S.cellCount = total;
        S.cellBase = 0u;
        S.flags = 0u;
        d.status[2] = total;
        if (total > d.cellCap) {
            atomicOr(d.status, 0x20u);
            atomicExch(d.status + 1, 1u);
        }
    }
    if (stop) return;

    uint32_t key[kSmallPer], at[kSmallPer];
#pragma unroll
    for (uint32_t u = 0; u < kSmallPer; u++) {
        key[u] = kNoKey;
        if (u * T + t >= d.n) break;
        key[u] = position_key(d, G, x[u], total);
        if (key[u] != kNoKey) at[u] = atomicAdd(d.CELL_COUNT + key[u], 1u);
    }
    cluster.sync();
    if (threadIdx.x == 0) stop = __ldcg(d.status + 1);

    // a run of whole groups of four cells per thread
    const uint32_t per = (total + 4u * T - 1u) / (4u * T), first = t * per, groups = total / 4u;
    const uint4* counts = reinterpret_cast<const uint4*>(d.CELL_COUNT);
    uint32_t sum = 0;
    for (uint32_t g = first; g < min(first + per, groups); g++) {
        const uint4 v = __ldcg(counts + g);
        sum += v.x + v.y + v.z + v.w;
    }
    uint32_t inBlock;
    uint32_t run = block_exclusive_scan_1024(sum, inBlock);
    if (threadIdx.x == 0) blockCells = inBlock;
    cluster.sync();
    if (stop) return;
    if (warp == 0) {
        const uint32_t v = lane < rank ? *cluster.map_shared_rank(&blockCells, lane) : 0u;
        const uint32_t w = __reduce_add_sync(0xffffffffu, v);
        if (lane == 0) before = w;
    }
    __syncthreads();
    run += before;
    for (uint32_t g = first; g < min(first + per, groups); g++) {
        const uint4 v = __ldcg(counts + g);
        reinterpret_cast<uint4*>(d.CELL_START)[g] = make_uint4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
        run += v.x + v.y + v.z + v.w;
    }
    cluster.sync();

    uint32_t start[kSmallPer], pid[kSmallPer];
#pragma unroll
    for (uint32_t u = 0; u < kSmallPer; u++) {
        const uint32_t i = u * T + t;
        if (i >= d.n) break;
        start[u] = __ldcg(d.CELL_START + key[u]);
        pid[u] = d.PIDc[i];
        d.TMP[start[u] + at[u]] = pid[u];
    }
    cluster.sync();
#pragma unroll
    for (uint32_t u = 0; u < kSmallPer; u++) {
        const uint32_t i = u * T + t;
        if (i >= d.n) break;
        const uint32_t count = __ldcg(d.CELL_COUNT + key[u]);
        uint32_t dst = start[u];
        for (uint32_t q = start[u]; q < start[u] + count; q++) dst += __ldcg(d.TMP + q) < pid[u] ? 1u : 0u;
        d.X[dst] = d.XN[i];
        d.V[dst] = d.Vc[i];
        d.DV[dst] = d.DVc[i];
        d.DK[dst] = d.DKc[i];
        d.PID[dst] = pid[u];
        d.KEYS[dst] = key[u];
    }
}

// N6-N8: ComputeCountsKernel + NeighborhoodQueryWithCountsKernel (ParticleSearchKernels.cu:93-193)
// in one pass, one warp per cell. The particles of a cell share their 27 candidate cells,
// so the warp walks that candidate set once, 32 candidates per round (lane j < 27 holds
// cell j's range, a prefix over the lanes flattens them), and tests each candidate
// against every particle of the cell, whose positions sit in shared memory. A ballot per
// particle appends its hits in candidate order, so each row keeps the reference's order
// (z, y, x cells, then cell order) and its cap of 70. The squared distance is computed
// without contraction, x^2 + y^2 + z^2 left to right, as the FP32 oracle does. The
// cell's grid coordinates come from its first particle by the same formula a
// per-particle search would use on each of them (they agree: it is how they were binned).
// Each hit also goes into the particle's NBRC row (when kept) as its stencil position: the
// candidates of cells 3w, 3w + 1, 3w + 2 (an x-run) are positions 0.. of run w, and the entry
// is (w << 6) | position. A cell with an x-run of more than 64 candidates gets no NBRC rows;
// its particles are flagged kRowPath.
// Bound by instructions: the tests of up to kNbrRounds rounds leave only their ballots, and the
// warp then writes the hits, its lanes shared out over the particles: 332 us for 1M particles
// (442 with each test's hits written at once and each candidate's cell sought by its lane), 301
// for 48 scenes of 18,000 (375), the same for 4,096.
constexpr uint32_t kNbrRounds = 8u;
template <bool REL>
__global__ void __launch_bounds__(kBlock) k_neighbors(Dev d) {
    VFD_COUNT_LAUNCH(d);
    if (aborted(d)) return;
    struct Warp {
        float4 x[32];                    // the cell's particles
        uint32_t slot[kNbrRounds][32];   // candidates
        uint32_t place[kNbrRounds][32];  // their staged place and stencil position, 16 bits each
        uint32_t hits[kNbrRounds][32];   // per particle: candidates in range
        uint32_t first[kNbrRounds][32];  // per particle: row entries before them
    };
    __shared__ Warp warpData[kBlock / 32u];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    Warp& W = warpData[w];
    const uint32_t total = d.status[2];
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < total; c += warps) {
        const uint32_t cnt = d.CELL_COUNT[c];
        if (cnt == 0u) continue;
        const uint32_t start = d.CELL_START[c];
        const uint32_t sid = scene_of(d, start);
        const SceneDev& S = d.scenes[sid];
        const float3 xa = abs_pos(d, S, d.X[start]);
        const float pos[3] = {xa.x, xa.y, xa.z};
        int gc[3];
#pragma unroll
        for (int k = 0; k < 3; k++) gc[k] = (int)floorf(__fmul_rn(__fsub_rn(pos[k], S.gridMin[k]), S.gridDelta[k]));
        // lane j < 27: candidate cell j (dz, dy, dx = j / 9, j / 3 % 3, j % 3, each minus 1)
        uint32_t cs = 0u, cc = 0u;
        if (lane < 27u) {
            const int fx = gc[0] + (int)(lane % 3u) - 1, fy = gc[1] + (int)(lane / 3u % 3u) - 1,
                      fz = gc[2] + (int)(lane / 9u) - 1;
            if (fx >= 0 && fy >= 0 && fz >= 0 && fx < (int)S.dim[0] && fy < (int)S.dim[1] && fz < (int)S.dim[2]) {
                const uint32_t key = S.cellBase + cell_key(S, fx, fy, fz);
                cs = d.CELL_START[key];
                cc = d.CELL_COUNT[key];
            }
        }
        uint32_t incl = cc;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const uint32_t ncand = __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t excl = incl - cc;
        const float h2 = S.h2;
        // x-run w (lanes 3w, 3w + 1, 3w + 2): its candidate total decides whether masks fit
        const uint32_t runEnd = __shfl_sync(0xffffffffu, incl, min(3u * lane + 2u, 31u));
        const uint32_t runBeg = __shfl_sync(0xffffffffu, excl, min(3u * lane, 31u));
        const bool want = d.NBRC != nullptr && d.compactRows != 0u;
        const bool compact = want && !__any_sync(0xffffffffu, lane < 9u && runEnd - runBeg > kRunMax);
        const uint32_t rowFlag = (want && !compact) ? kRowPath : 0u;
        // staged place of candidate i of cell j: i + (the cell's first place - the candidates before it)
        uint32_t place = 0u;
        const bool halo = halo_on(d);
        if (halo && lane < 27u)
            place = d.haloBase[(size_t)(c / kHaloTileCells) * kHaloCells +
                               halo_cell(c, lane % 3u, lane / 3u % 3u, lane / 9u)] - excl;
        // stencil position of candidate i of cell j: its x-run and place in the run, entry + i
        const uint32_t entry = (lane / 3u << 6) - __shfl_sync(0xffffffffu, excl, lane / 3u * 3u);
        uint32_t mx = 0u;
        for (uint32_t k0 = 0; k0 < cnt; k0 += 32u) {
            const uint32_t kk = min(32u, cnt - k0);
            // lanes that share a particle when the hits are written: lane mod `width` is its number
            const uint32_t width = kk > 1u ? 1u << (32 - __clz(kk - 1u)) : 1u, shares = 32u / width;
            const uint32_t kw = lane & (width - 1u), share = lane / width;
            __syncwarp();
            if (lane < kk) W.x[lane] = d.X[start + k0 + lane];
            uint32_t found = 0u;  // neighbours so far of particle start + k0 + lane
            for (uint32_t base0 = 0; base0 < ncand; base0 += 32u * kNbrRounds) {
                const uint32_t rounds = min(kNbrRounds, (ncand - base0 + 31u) / 32u);
                // every lane lists its cell's candidates of these rounds
                for (uint32_t i = max(excl, base0); i < min(incl, base0 + 32u * kNbrRounds); i++) {
                    (&W.slot[0][0])[i - base0] = cs + (i - excl);
                    (&W.place[0][0])[i - base0] = (place + i) << 16 | (entry + i & 0xFFFFu);
                }
                __syncwarp();
                for (uint32_t r = 0; r < rounds; r++) {
                    const bool valid = base0 + 32u * r + lane < ncand;
                    const uint32_t q = checked_index(d.status, valid ? W.slot[r][lane] : 0u, d.n);
                    const float4 xq = valid ? d.X[q] : make_float4(0.f, 0.f, 0.f, 0.f);
                    uint32_t mine = 0u;
#pragma unroll 4
                    for (uint32_t k = 0; k < kk; k++) {
                        const float3 e = pair_r<REL>(d, xq, W.x[k]);
                        const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(e.x, e.x), __fmul_rn(e.y, e.y)), __fmul_rn(e.z, e.z));
                        const uint32_t bits = __ballot_sync(0xffffffffu, valid && d2 < h2 && d2 > 0.0f);
                        if (lane == k) mine = bits;
                    }
                    W.hits[r][lane] = mine;
                    W.first[r][lane] = found;
                    found += __popc(mine);
                }
                __syncwarp();
                if (kw < kk) {
                    const size_t p = start + k0 + kw;
                    for (uint32_t r = share; r < rounds; r += shares) {
                        uint32_t at = W.first[r][kw];
                        for (uint32_t m = W.hits[r][kw]; m != 0u && at < kMaxNeighbors; m &= m - 1u, at++) {
                            const uint32_t b = __ffs(m) - 1u;
                            const uint32_t both = W.place[r][b];
                            d.NBR[p * kRow + at] = W.slot[r][b];
                            if (compact) d.NBRC[p * kRow + at] = (uint16_t)both;
                            if (halo) d.haloRow[halo_row_at((uint32_t)p, at)] = (uint16_t)(both >> 16);
                        }
                    }
                }
                __syncwarp();
            }
            const uint32_t count = min(found, kMaxNeighbors);
            if (lane < kk) {
                d.NCNT[start + k0 + lane] = count | rowFlag;
                if (count == kMaxNeighbors) atomicOr(&d.scenes[sid].flags, 0x8u);
            }
            mx = max(mx, __reduce_max_sync(0xffffffffu, lane < kk ? count : 0u));
        }
        if (lane == 0) atomicMax(max_bucket(d, sid, 1, blockIdx.x % kBuckets), mx);
    }
}

// ---------------------------------------------------------------- launchers
// `profiled` = false launches without the per-kernel profiler hook (the allocation-free
// search must not create CUDA events, whatever another thread is profiling).
#define SEARCH_LAUNCH(name, ...)                 \
    do {                                         \
        if (profiled) VFD_LAUNCH(name, s, __VA_ARGS__); \
        else { __VA_ARGS__; }                    \
    } while (0)
void launch_neighbors(const Dev& d, cudaStream_t s, bool profiled) {
    // a warp per cell, a fixed grid striding over the cells the device counted
    const uint32_t nbrBlocks = 4u * d.batchBlocks;
    if (d.cellRel) SEARCH_LAUNCH("k_neighbors", k_neighbors<true><<<nbrBlocks, kBlock, 0, s>>>(d));
    else SEARCH_LAUNCH("k_neighbors", k_neighbors<false><<<nbrBlocks, kBlock, 0, s>>>(d));
}
// Cells and (with staged tiles) tiles of the current positions; then the order and the rows.
void launch_search_cells(const Dev& d, cudaStream_t s, bool profiled) {
    const uint32_t nb = blocks_for(d.n);
    SEARCH_LAUNCH("k_minmax", k_minmax<<<nb, kBlock, 0, s>>>(d));
    SEARCH_LAUNCH("k_grid", k_grid<<<1, 256, 0, s>>>(d));
    SEARCH_LAUNCH("k_clear_cells", k_clear_cells<<<1216, 256, 0, s>>>(d));
    SEARCH_LAUNCH("k_keys", k_keys<<<nb, kBlock, 0, s>>>(d));
    SEARCH_LAUNCH("k_scan_reduce", k_scan_reduce<<<d.scanBlocks, 256, 0, s>>>(d));
    SEARCH_LAUNCH("k_scan_top", k_scan_top<<<1, 1024, 0, s>>>(d));
    SEARCH_LAUNCH("k_scan_down", k_scan_down<<<d.scanBlocks, 256, 0, s>>>(d));
    if (halo_on(d)) launch_halo_build(d, s);
}
void launch_search_rows(const Dev& d, cudaStream_t s, bool profiled) {
    const uint32_t nb = blocks_for(d.n);
    SEARCH_LAUNCH("k_slots", k_slots<<<nb, kBlock, 0, s>>>(d));
    SEARCH_LAUNCH("k_rank_gather", k_rank_gather<<<nb, kBlock, 0, s>>>(d));
    launch_neighbors(d, s, profiled);
}
void launch_search(const Dev& d, cudaStream_t s, bool profiled) {
    if (search_small(d)) {
        SEARCH_LAUNCH("k_search_small", k_search_small<<<kSmallBlocks, kSmallThreads, 0, s>>>(d));
        launch_neighbors(d, s, profiled);
        return;
    }
    launch_search_cells(d, s, profiled);
    launch_search_rows(d, s, profiled);
}
#undef SEARCH_LAUNCH

uint32_t scan_block_count(uint32_t cellCap) { return (cellCap + kScanItems - 1) / kScanItems; }

}  // namespace vfd
