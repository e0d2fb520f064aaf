// Neighbour loops of large scenes over staged cell tiles.
//
// The row kernels of dfsph_physics.cu gather each neighbour's position and field through
// L1, two 16-byte gathers a pair, and wait on them (73 % of the L1 pipe busy, 35 % of DRAM
// bandwidth, at 1M particles). Here a block takes a tile of 4x4x2 Morton cells, brings the
// positions and the pass's field of the tile grown by one cell on every side (its halo, in z,
// y, x cell order) to shared memory with asynchronous copies, and walks each particle's
// neighbours there. A pair costs 6 bytes of DRAM: its 16-bit place in the staged halo and the
// 32-bit gradient factor gradW / r; the gathers read shared memory.
//   * Once a step, after the counting sort: the non-empty tiles are listed in cell order
//     (k_scan_down), k_halo_build writes each one's halo as a list of slots and the staged
//     place of each halo cell's first particle, the search writes the 16-bit rows and the
//     density pass the gradient factors.
//   * A tile whose halo outgrows the shared memory walks its slot rows (NBR) instead.
//   * A thread takes a particle: 32 consecutive rows are interleaved so that its eight entries
//     of a load are 16 bytes from consecutive addresses of the warp. It keeps eight partial
//     sums, those of the row kernels' eight lanes, and adds them as their shuffle tree does, so
//     a particle's sums have the same bits on either path.
// What bounds it: shared-memory gathers (ncu, 512k particles: the data pipe 78 % busy while an
// SM is active, 2.4 wavefronts of bank conflict each; DRAM 260 bytes a particle, a third of
// its bandwidth). Per launch at 1M particles on a lattice, row kernels with eight lanes, with
// four, and tiles (narrow form): Jacobi update 147 / 131 / 101 us, pressure acceleration 83 / 89 /
// 68, viscosity product 179 / 148 / 110; after 300 steps rows with four lanes and the wide form:
// 160 / 139, 106 / 100, 178 / 162 (and the density pass 285 / 316). Tried and left out: four lanes a particle (124 us for
// the Jacobi update; the same gathers, more instructions), 4x4x4 tiles (102), two halo buffers
// (164: half the resident warps), and bulk copies of the halo's runs of 8 to 16 particles by
// the TMA unit (213: about 80 cycles a copy and SM), and tiles drawn by an atomic ticket instead of
// strided (103, and 2 % at 8M; 1 % less for 48 scenes), and part-filled rounds with two or four
// threads a particle (after 300 steps 184 us for the Jacobi update, 155 with idle threads).
#include "dfsph_common.cuh"
#include "dfsph_passes.cuh"
#include "dfsph_halo.cuh"
#include "dfsph_sim.h"

namespace vfd {
// ---------------------------------------------------------------- tile lists
// Cost of a step's passes on tiles, in units of the row kernels' time for a particle; a step runs on
// the cheapest form (k_tile_form). A round of a tile costs its block about the same however few
// particles it has, so sparse fluid runs on rows. A wave of blocks lasts for its slowest tile, and
// the last, part-filled one costs half of what it lacks. One halo beyond the shared memory makes a
// pass wait for that block. Fitted to steps of ten iterations a solver over 198 states (lattices,
// thinned ones, clumps, squeezed ones, dams after 15 to 400 steps, batches; 104,000 to 3M
// particles): the mean step 0.1 % above the best of rows, narrow and wide tiles, the worst 4 %, none
// slower than rows with eight lanes. (Narrow up to a quarter of the tiles beyond it, else wide, as
// before: up to 1.76 times the rows' time, at 40 particles a tile.)
__device__ __forceinline__ float rounds_cost(const Dev& d, uint32_t tiles, uint32_t rounds, uint32_t blocks, float round,
                                             uint32_t rows, float wait, float row) {
    const uint32_t resident = blocks * (d.batchBlocks / (2048u / kBlock));
    const float waves = (float)((tiles + resident - 1u) / resident) * (float)resident;
    const float full = waves * fminf(2.0f, 2.0f * (float)rounds / (float)tiles - 1.0f);
    return round * 0.5f * ((float)rounds + full) + (rows ? wait + row * (float)rows : 0.0f);
}
__device__ __forceinline__ float narrow_cost(const Dev& d, uint32_t tiles, uint32_t rounds, uint32_t rows) {
    return 50000.0f + rounds_cost(d, tiles, rounds, 4u, 110.0f, rows, 300000.0f, 350.0f);
}
__device__ __forceinline__ float wide_cost(const Dev& d, uint32_t tiles, uint32_t rounds, uint32_t rows) {
    return rounds_cost(d, tiles, rounds, 3u, 170.0f, rows, 250000.0f, 900.0f);
}
// Of the allowed forms (bit 1 << form; rows always).
__device__ __forceinline__ uint32_t cheapest_form(const Dev& d, uint32_t tiles, uint32_t narrow, uint32_t narrowRows,
                                                  uint32_t wide, uint32_t wideRows, uint32_t forms) {
    if (tiles == 0u) return 0u;
    const float n = narrow_cost(d, tiles, narrow, narrowRows), w = wide_cost(d, tiles, wide, wideRows);
    uint32_t form = 0u;
    float best = (float)d.n;
    if ((forms >> kHaloNarrow & 1u) && n < best) form = kHaloNarrow, best = n;
    if ((forms >> kHaloWide & 1u) && w < best) form = kHaloWide;
    return form;
}

// One block per tile: its halo's slots into haloList and the staged place of each halo
// cell's first particle into haloBase. The list space is handed out in any order (the lists'
// contents do not depend on it); a particle lies in at most eight halos (two tiles an axis).
__global__ void __launch_bounds__(256) k_halo_build(Dev d) {
    VFD_COUNT_LAUNCH(d);
    if (is_aborted(d)) return;
    __shared__ uint32_t warpSum[8], base[kHaloCells], start[kHaloCells], offset;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t nt = d.haloInfo[0];
    // where rows are cheaper than either form with all halos staged, nothing is listed
    HaloCounts* all = halo_counts(d);
    if (d.formChoice && cheapest_form(d, nt, all->narrow, 0u, all->wide, 0u, d.formChoice) == 0u) return;
    uint32_t narrowRows = 0u, wideRows = 0u;  // in thread 0: rounds over tiles that outgrow the shared memory
    for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
        HaloTile& T = d.haloTiles[t];
        const SceneDev& S = d.scenes[T.scene];
        const uint32_t kl = T.cell0 - S.cellBase, meta = kl >> 9, low = kl & 511u;
        const uint32_t myz = meta / S.meta[0];
        const int ox = (int)((meta % S.meta[0]) * 8u + compact3(low)) - 1;
        const int oy = (int)((myz % S.meta[1]) * 8u + compact3(low >> 1)) - 1;
        const int oz = (int)((myz / S.meta[1]) * 8u + compact3(low >> 2)) - 1;
        uint32_t cs = 0u, cc = 0u;
        if (threadIdx.x < kHaloCells) {
            const uint32_t c = threadIdx.x;
            const int cx = ox + (int)(c % kHaloX), cy = oy + (int)(c / kHaloX % kHaloY), cz = oz + (int)(c / (kHaloX * kHaloY));
            if (cx >= 0 && cy >= 0 && cz >= 0 && cx < (int)S.dim[0] && cy < (int)S.dim[1] && cz < (int)S.dim[2]) {
                const uint32_t key = S.cellBase + cell_key(S, cx, cy, cz);
                cs = d.CELL_START[key];
                cc = d.CELL_COUNT[key];
            }
        }
        uint32_t x = cc;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31u) warpSum[w] = x;
        __syncthreads();
        uint32_t pre = 0u, total = 0u;
        for (uint32_t k = 0; k < 8u; k++) {
            if (k < w) pre += warpSum[k];
            total += warpSum[k];
        }
        if (threadIdx.x < kHaloCells) {
            base[threadIdx.x] = pre + x - cc;
            start[threadIdx.x] = cs;
            d.haloBase[(size_t)(T.cell0 / kHaloTileCells) * kHaloCells + threadIdx.x] = (uint16_t)(pre + x - cc);
        }
        if (threadIdx.x == 0) {
            const bool fits = total <= kHaloWideCap;
            const uint32_t at = fits ? atomicAdd(d.haloInfo + 1, total) : 0u;
            offset = fits ? at : 0xFFFFFFFFu;
            T.list = at;
            T.staged = total;
            if (total > kHaloCap) narrowRows += halo_rounds(T.last - T.first, kHaloThreads);
            if (total > kHaloWideCap) wideRows += halo_rounds(T.last - T.first, kHaloWideThreads);
        }
        __syncthreads();
        if (offset != 0xFFFFFFFFu)
            for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) {
                uint32_t c = 0u;  // the last cell whose first place is <= i
#pragma unroll
                for (uint32_t step = 128u; step > 0u; step >>= 1)
                    if (c + step < kHaloCells && base[c + step] <= i) c += step;
                d.haloList[(size_t)offset + i] = start[c] + (i - base[c]);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (narrowRows) atomicAdd(&all->narrowRows, narrowRows);
        if (wideRows) atomicAdd(&all->wideRows, wideRows);
    }
}

// The form that this step runs on, of Dev::formChoice and rows.
__global__ void k_tile_form(Dev d) {
    VFD_COUNT_LAUNCH(d);
    const HaloCounts c = *halo_counts(d);
    const uint32_t form =
        is_aborted(d) ? 0u : cheapest_form(d, d.haloInfo[0], c.narrow, c.narrowRows, c.wide, c.wideRows, d.formChoice);
    d.status[14] = form;
    // the graph's branches: rows, then the allowed forms
    if (d.formHandle)
        cudaGraphSetConditional((cudaGraphConditionalHandle)d.formHandle, form ? __popc(d.formChoice & ((2u << form) - 1u)) : 0u);
}

// ---------------------------------------------------------------- the tile loop
__device__ __forceinline__ void copy_async16(void* smem, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}
__device__ __forceinline__ void copy_async4(void* smem, const void* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

enum HaloField { kNoField = 0, kScalarField = 1, kVectorField = 4 };  // floats staged beside the position
enum HaloGrad { kReadGrad = 0, kWriteGrad = 1 };

// Threads and resident blocks of a pass, and the particles it can stage, in the narrow and the wide form.
template <class Op, bool WIDE>
struct HaloShape {
    static constexpr uint32_t kThreads = WIDE ? Op::kWideThreads : kHaloThreads, kCap = WIDE ? kHaloWideCap : kHaloCap;
    static constexpr uint32_t kBlocks = kThreads == kHaloThreads ? Op::kBlocks : Op::kBlocks >= 4u ? 3u : 2u;
    static constexpr bool kAhead = Op::kAhead && kThreads == kHaloThreads;
    static constexpr size_t kSmem = (size_t)kCap * (16u + 4u * (size_t)Op::kField);
};

// FP32-pair sums of a pass's K reduction terms over a block's tiles, added to the scene's
// FP64 buckets when the scene changes and at the end.
template <int K, uint32_t THREADS>
struct HaloSum {
    float hi[K], lo[K];
    int scene = -1;
    __device__ __forceinline__ HaloSum() {
#pragma unroll
        for (int k = 0; k < K; k++) hi[k] = lo[k] = 0.0f;
    }
    // all threads of the block, with the same scene
    __device__ void flush(const Dev& d, const int* slot) {
        __shared__ float2 part[THREADS / 32u][K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            float h = hi[k], l = lo[k];
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
                const float h2 = __shfl_xor_sync(0xffffffffu, h, o);
                const float l2 = __shfl_xor_sync(0xffffffffu, l, o);
                pair_add(h, l, h2, l2);
            }
            if ((threadIdx.x & 31u) == 0u) part[threadIdx.x >> 5][k] = make_float2(h, l);
        }
        __syncthreads();
        if (threadIdx.x < (uint32_t)K && scene >= 0) {
            float a = 0.0f, b = 0.0f;
            for (uint32_t w = 0; w < THREADS / 32u; w++) pair_add(a, b, part[w][threadIdx.x].x, part[w][threadIdx.x].y);
            const double t = pair_value(make_float2(a, b));
            if (t != 0.0) atomicAdd(acc_bucket(d, (uint32_t)scene, slot[threadIdx.x], blockIdx.x % kBuckets), t);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; k++) hi[k] = lo[k] = 0.0f;
    }
};

template <uint32_t THREADS>
struct HaloSum<0, THREADS> {
    int scene = -1;
    float hi[1], lo[1];
    __device__ __forceinline__ void flush(const Dev&, const int*) {}
};

// Starts the copies of a tile's halo into shared memory.
template <int FIELD, uint32_t THREADS, uint32_t CAP>
__device__ __forceinline__ void halo_fetch(const Dev& d, const HaloTile& T, const void* field, float4* sx) {
    if (T.staged <= CAP) {
        const uint32_t* list = d.haloList + T.list;
#pragma unroll 2
        for (uint32_t i = threadIdx.x; i < T.staged; i += THREADS) {
            const uint32_t q = checked_index(d.status, __ldg(list + i), d.n);
            copy_async16(sx + i, d.X + q);
            if (FIELD == kVectorField) copy_async16(sx + CAP + i, reinterpret_cast<const float4*>(field) + q);
            if (FIELD == kScalarField)
                copy_async4(reinterpret_cast<float*>(sx + CAP) + i, reinterpret_cast<const float*>(field) + q);
        }
    }
}

// Eight row entries: staged places and gradient factors.
struct HaloEntries {
    uint4 e;
    float4 g0, g1;
};
template <int GRAD>
__device__ __forceinline__ void halo_entries(const Dev& d, uint32_t p, uint32_t k, HaloEntries& x) {
    x.e = __ldcs(reinterpret_cast<const uint4*>(d.haloRow + halo_row_at(p, k)));
    if (GRAD == kReadGrad) {
        x.g0 = __ldcs(reinterpret_cast<const float4*>(d.haloGrad + halo_grad_at(p, k)));
        x.g1 = __ldcs(reinterpret_cast<const float4*>(d.haloGrad + halo_grad_at(p, k + 4u)));
    }
}

// A pass over the tiles, a thread a particle. What it supplies (static members of Op):
//   kField, kGrad          staged field; whether the pass reads or writes the gradient factors
//   kTerms, slots()        reduction terms of finish() and their accumulators
//   kLoop                  solver loop whose active scenes it walks, or -1
//   active(S)              whether scene S runs the pass
//   field(d)               the staged array (float4 or float)
//   Own, load()            the particle's own data
//   pair(d, o, xq, fq, gs, ok, acc)  one neighbour's term, added when ok (gs written by a
//                          kWriteGrad pass)
//   Acc                    the pair sums: eight a thread, added with += as the rows' lanes meet
//   finish(d, p, S, o, acc, ncnt, term)  writes the outputs, sets the terms
template <class Op, bool WIDE>
__device__ __forceinline__ void halo_pass(const Dev& d) {
    using Shape = HaloShape<Op, WIDE>;
    constexpr uint32_t kThreads = Shape::kThreads, kCap = Shape::kCap;
    constexpr bool kAhead = Shape::kAhead;
    extern __shared__ float4 haloSmem[];
    float4* const sx = haloSmem;
    float4* const sv = haloSmem + kCap;                            // kVectorField
    float* const ss = reinterpret_cast<float*>(haloSmem + kCap);   // kScalarField
    if (is_aborted(d)) return;
    HaloSum<Op::kTerms, kThreads> sum;
    const uint32_t nt = halo_tile_total(d, Op::kLoop);
    for (uint32_t v = blockIdx.x; v < nt; v += gridDim.x) {
        const HaloTile T = d.haloTiles[halo_tile_at(d, Op::kLoop, v)];
        const SceneDev& S = d.scenes[T.scene];
        if (!Op::active(S)) continue;
        if (Op::kTerms > 0 && (int)T.scene != sum.scene) {
            if (sum.scene >= 0) sum.flush(d, Op::slots());
            sum.scene = (int)T.scene;
        }
        const bool fits = T.staged <= kCap;
        halo_fetch<Op::kField, kThreads, kCap>(d, T, Op::field(d), sx);
        bool waiting = true;
        for (uint32_t pb = T.first; pb < T.last; pb += kThreads) {
            const bool live = pb + threadIdx.x < T.last;
            const uint32_t p = live ? pb + threadIdx.x : T.first;
            const uint32_t ncnt = d.NCNT[p];
            const uint32_t cnt = live ? ncnt & kCountMask : 0u;
            HaloEntries x;
            halo_entries<Op::kGrad>(d, p, 0u, x);
            typename Op::Own own;
            Op::load(d, p, S, own);
            if (waiting) {
                copy_async_wait();
                __syncthreads();
                waiting = false;
            }
            // partial sums of the row kernels' eight lanes, met as their shuffle tree meets
            typename Op::Acc acc[8] = {};
            if (fits) {
                for (uint32_t k = 0; k < cnt; k += 8u) {
                    HaloEntries y;
                    if (kAhead && k + 8u < cnt) halo_entries<Op::kGrad>(d, p, k + 8u, y);
                    if (!kAhead && k > 0u) halo_entries<Op::kGrad>(d, p, k, x);
                    const uint32_t ee[4] = {x.e.x, x.e.y, x.e.z, x.e.w};
                    float gg[8] = {x.g0.x, x.g0.y, x.g0.z, x.g0.w, x.g1.x, x.g1.y, x.g1.z, x.g1.w};
#pragma unroll
                    for (uint32_t u = 0; u < 8u; u++) {
                        const bool ok = k + u < cnt;
                        const uint32_t at = checked_index(d.status, ok ? (ee[u >> 1] >> (16u * (u & 1u))) & 0xFFFFu : 0u, T.staged);
                        float4 fq = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (Op::kField == kVectorField) fq = sv[at];
                        if (Op::kField == kScalarField) fq.x = ss[at];
                        Op::pair(d, own, sx[at], fq, gg[u], ok, acc[u]);
                    }
                    if (Op::kGrad == kWriteGrad) {
                        __stcs(reinterpret_cast<float4*>(d.haloGrad + halo_grad_at(p, k)), make_float4(gg[0], gg[1], gg[2], gg[3]));
                        __stcs(reinterpret_cast<float4*>(d.haloGrad + halo_grad_at(p, k + 4u)), make_float4(gg[4], gg[5], gg[6], gg[7]));
                    }
                    if (kAhead) x = y;
                }
            } else {
                for (uint32_t k = 0; k < cnt; k += 8u)
#pragma unroll
                    for (uint32_t u = 0; u < 8u; u++) {
                        const uint32_t j = k + u;
                        if (j >= cnt) continue;
                        const uint32_t q = checked_index(d.status, __ldg(d.NBR + (size_t)p * kRow + j), d.n);
                        float4 fq = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (Op::kField == kVectorField) fq = reinterpret_cast<const float4*>(Op::field(d))[q];
                        if (Op::kField == kScalarField) fq.x = reinterpret_cast<const float*>(Op::field(d))[q];
                        float gs = Op::kGrad == kReadGrad ? d.haloGrad[halo_grad_at(p, j)] : 0.0f;
                        Op::pair(d, own, d.X[q], fq, gs, true, acc[u]);
                        if (Op::kGrad == kWriteGrad) d.haloGrad[halo_grad_at(p, j)] = gs;
                    }
            }
#pragma unroll
            for (uint32_t o = 4u; o > 0u; o >>= 1)
#pragma unroll
                for (uint32_t u = 0; u < o; u++) acc[u] += acc[u + o];
            if (live) {
                float term[Op::kTerms > 0 ? Op::kTerms : 1];
                Op::finish(d, p, S, own, acc[0], ncnt, term);
#pragma unroll
                for (int k = 0; k < Op::kTerms; k++) pair_add(sum.hi[k], sum.lo[k], term[k], 0.0f);
            }
        }
        __syncthreads();  // the next tile overwrites the halo
    }
    if (Op::kTerms > 0) sum.flush(d, Op::slots());
}

// ---------------------------------------------------------------- the passes
// Parts shared by the passes that reduce nothing or walk every scene.
template <int FIELD, int GRAD = kReadGrad, uint32_t BLOCKS = 3u, int TERMS = 0, int LOOP = -1>
struct HaloOp {
    static constexpr int kField = FIELD, kGrad = GRAD, kTerms = TERMS, kLoop = LOOP;
    // Blocks per SM that the registers allow, and whether the next eight row entries are loaded
    // ahead. The passes of the solver loops run best with four blocks and nothing ahead (at 1M
    // particles 67, 100 and 110 us for the pressure acceleration, the Jacobi update and the
    // product, against 75, 107 and 118 with three and 73, 106 and 125 with three and entries
    // ahead); the others, with more sums a particle, with three and entries ahead.
    static constexpr uint32_t kBlocks = BLOCKS;
    static constexpr uint32_t kWideThreads = kHaloWideThreads;
    static constexpr bool kAhead = BLOCKS < 4u;
    __device__ static bool active(const SceneDev&) { return true; }
    __device__ static const void* field(const Dev&) { return nullptr; }
    __device__ static const int* slots() { return nullptr; }
};
__device__ constexpr int kSlots01[2] = {0, 1};

// K2 + K3 + K4 (k_density_factor with DIV).
template <bool REL>
struct HaloDensity : HaloOp<kVectorField, kWriteGrad> {
    struct Own {
        float4 xi;
        float3 vi;
        float V;
        bool div;
    };
    using Acc = DensitySums;
    __device__ static const void* field(const Dev& d) { return d.V; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, Own& o) {
        o.xi = d.X[p];
        o.V = S.volume;
        o.div = S.enableDiv != 0;
        o.vi = o.div ? f3(d.V[p]) : make_float3(0.f, 0.f, 0.f);
    }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 fq, float& gs, bool ok, Acc& a) {
        const float3 r = pair_r<REL>(d, o.xi, xq);
        float w;
        kernel_wg(d, r, w, gs);
        if (!ok) return;
        a.add(o.V, w, gs, r, o.div, o.vi - f3(fq));
    }
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const Own& o, const Acc& a, uint32_t ncnt,
                                  float*) {
        density_finish(d, p, S, f3(o.xi), o.vi, o.div, a, ncnt);
    }
};

// The pair sum of the pressure acceleration (K5 / K7 / K18 / K20): kappa rides in X.w, or is
// staged beside cell-relative positions.
template <bool DIV, bool REL, int LOOP>
struct HaloPressure : HaloOp<REL ? kScalarField : kNoField, kReadGrad, 4u, 0, LOOP> {
    struct Own {
        float4 xi;
        float ki, V;
    };
    using Acc = float3;
    __device__ static const void* field(const Dev& d) { return DIV ? d.KAPPAV : d.KAPPA; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, Own& o) {
        o.xi = d.X[p];
        o.ki = (DIV ? d.KAPPAV : d.KAPPA)[p];
        o.V = S.volume;
    }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 fq, float& gs, bool ok, Acc& a) {
        const float sum = o.ki + (REL ? fq.x : xq.w);
        const float3 r = pair_r<REL>(d, o.xi, xq);
        add_pressure(a, sum, o.V, gs, r, ok);
    }
    __device__ static float3 total(const Dev& d, uint32_t p, const Own& o, float3 a, uint32_t ncnt) {
        if (fabsf(o.ki) > kEps && (ncnt & kHasBoundary)) a += o.ki * (-f3(d.GB[p]));
        return a;
    }
};
template <bool DIV, bool REL>
struct HaloPressureAccel : HaloPressure<DIV, REL, DIV ? kLoopDiv : kLoopPres> {  // K5 / K18
    using Base = HaloPressure<DIV, REL, DIV ? kLoopDiv : kLoopPres>;
    __device__ static bool active(const SceneDev& S) { return (DIV ? S.div.active : S.pres.active) != 0u; }
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev&, const typename Base::Own& o, float3 a,
                                  uint32_t ncnt, float*) {
        d.AP[p] = f4(Base::total(d, p, o, a, ncnt), 0.0f);
    }
};
template <bool REL>
struct HaloDivFinish : HaloPressure<true, REL, -1> {  // K7 + K8
    using Base = HaloPressure<true, REL, -1>;
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const typename Base::Own& o, float3 a,
                                  uint32_t ncnt, float*) {
        if (S.enableDiv) div_finish_item(d, p, S, Base::total(d, p, o, a, ncnt));
        d.A[p] = make_float4(S.g[0], S.g[1], S.g[2], 0.0f);
    }
};
template <bool REL>
struct HaloPresFinish : HaloPressure<false, REL, -1> {  // K20 + K21
    using Base = HaloPressure<false, REL, -1>;
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const typename Base::Own& o, float3 a,
                                  uint32_t ncnt, float*) {
        pres_finish_item(d, p, S, Base::total(d, p, o, a, ncnt));
    }
};

// K6 / K19.
template <bool DIV, bool REL>
struct HaloJacobi : HaloOp<kVectorField, kReadGrad, 4u, 1, DIV ? kLoopDiv : kLoopPres> {
    using Base = JacobiOp<DIV, REL>;
    using Own = typename Base::Own;
    using Acc = float;
    __device__ static bool active(const SceneDev& S) { return Base::active(S); }
    __device__ static const void* field(const Dev& d) { return d.AP; }
    __device__ static const int* slots() { return kSlots01; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, Own& o) { Base::load(d, p, S, o); }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 aq, float& gs, bool ok, Acc& f) {
        const float3 r = pair_r<REL>(d, o.xi, xq);
        const float t = dot3(o.ai - f3(aq), gs * r);
        if (ok) f += t;
    }
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const Own& o, Acc f, uint32_t ncnt, float* term) {
        term[0] = Base::finish(d, p, S, o, f, ncnt);
    }
};

// K17.
template <bool REL>
struct HaloPresInit : HaloOp<kVectorField> {
    static constexpr uint32_t kWideThreads = kHaloThreads;  // the registers of more threads would spill
    struct Own {
        float4 xi;
        float3 vi;
    };
    using Acc = float;
    __device__ static const void* field(const Dev& d) { return d.V; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev&, Own& o) {
        o.xi = d.X[p];
        o.vi = f3(d.V[p]);
    }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 vq, float& gs, bool ok, Acc& s) {
        const float3 r = pair_r<REL>(d, o.xi, xq);
        const float t = dot3(o.vi - f3(vq), gs * r);
        if (ok) s += t;
    }
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const Own& o, Acc s, uint32_t ncnt, float*) {
        s *= S.volume;
        if (ncnt & kHasBoundary) s += dot3(o.vi, f3(d.GB[p]));
        pres_init_finish(d, p, S, s);
    }
};

// K12 + K13.
template <bool REL>
struct HaloPrecond : HaloOp<kScalarField, kReadGrad, 2u> {
    static constexpr uint32_t kWideThreads = kHaloThreads;  // the registers of more threads would spill
    struct Own {
        float4 xi;
        float eps2, cmu, mass;
    };
    using Acc = Mat3;
    __device__ static bool active(const SceneDev& S) { return S.enableVisc != 0; }
    __device__ static const void* field(const Dev& d) { return d.RHO; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, Own& o) {
        o.xi = d.X[p];
        o.eps2 = 0.01f * S.h2;
        o.cmu = 10.0f * S.dynVisc;
        o.mass = S.mass;
    }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 rho, float& gs, bool ok, Acc& m) {
        const float3 r = pair_r<REL>(d, o.xi, xq);
        if (!ok) return;
        const float3 g = gs * r;
        const float c = __fdividef(o.cmu * __fdividef(o.mass, rho.x), dot3(r, r) + o.eps2);
        add_outer(m, c, r, g);
    }
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const Own& o, const Acc& m, uint32_t ncnt,
                                  float*) {
        precond_finish(d, p, S, f3(o.xi), m, ncnt);
    }
};

// K14 on the first guess (the initial residual) and on the CG direction.
template <bool REL, int LOOP>
struct HaloMatvec : HaloOp<kVectorField, kReadGrad, 4u, LOOP < 0 ? 2 : 1, LOOP> {
    using Own = typename SpmvOp<REL>::Own;
    using Acc = float3;
    __device__ static const int* slots() { return kSlots01; }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 vq, float& gs, bool ok, Acc& acc) {
        const float3 r = pair_r<REL>(d, o.xi, xq);
        add_viscous(acc, o.cmu * vq.w, o.vi - f3(vq), o.eps2, gs, r, ok);
    }
};
template <bool REL>
struct HaloSetup : HaloMatvec<REL, -1> {
    using Base = HaloMatvec<REL, -1>;
    __device__ static bool active(const SceneDev& S) { return S.enableVisc != 0; }
    __device__ static const void* field(const Dev& d) { return d.CG; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, typename Base::Own& o) {
        SpmvOp<REL>::load(d, p, S, o);
        o.vi = f3(d.CG[p]);
    }
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const typename Base::Own& o, float3 acc,
                                  uint32_t ncnt, float* term) {
        const float3 b = f3(d.CB[p]);
        const float3 r = b - visc_product<false>(d, p, S, o.vi, acc, ncnt);
        d.CR[p] = f4(r, 0.0f);
        term[0] = dot_term(b, b);
        term[1] = dot_term(r, r);
    }
};
template <bool REL>
struct HaloSpmv : HaloMatvec<REL, kLoopCG> {
    using Base = HaloMatvec<REL, kLoopCG>;
    __device__ static bool active(const SceneDev& S) { return S.cgActive != 0u; }
    __device__ static const void* field(const Dev& d) { return d.CP; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, typename Base::Own& o) {
        SpmvOp<REL>::load(d, p, S, o);
    }
    __device__ static void finish(const Dev& d, uint32_t p, const SceneDev& S, const typename Base::Own& o, float3 acc,
                                  uint32_t ncnt, float* term) {
        const float3 ap = visc_product<true>(d, p, S, o.vi, acc, ncnt);
        d.CAP[p] = f4(ap, 0.0f);
        term[0] = dot_term(o.vi, ap);
    }
};

// One kernel name per pass, for profilers.
#define HALO_KERNEL(NAME, OP)                                                          \
    template <bool REL, bool WIDE>                                                     \
    __global__ void __launch_bounds__(HaloShape<OP HALO_COMMA WIDE>::kThreads, HaloShape<OP HALO_COMMA WIDE>::kBlocks) \
        NAME(Dev d) {                                                                  \
        VFD_COUNT_LAUNCH(d);                                                           \
        halo_pass<OP HALO_COMMA WIDE>(d);                                              \
    }
#define HALO_COMMA ,
HALO_KERNEL(k_density_factor_halo, HaloDensity<REL>)
HALO_KERNEL(k_pressure_accel_halo_d, HaloPressureAccel<true HALO_COMMA REL>)
HALO_KERNEL(k_pressure_accel_halo_p, HaloPressureAccel<false HALO_COMMA REL>)
HALO_KERNEL(k_jacobi_iter_halo_d, HaloJacobi<true HALO_COMMA REL>)
HALO_KERNEL(k_jacobi_iter_halo_p, HaloJacobi<false HALO_COMMA REL>)
HALO_KERNEL(k_div_finish_halo, HaloDivFinish<REL>)
HALO_KERNEL(k_pres_init_halo, HaloPresInit<REL>)
HALO_KERNEL(k_pres_finish_halo, HaloPresFinish<REL>)
HALO_KERNEL(k_visc_precond_halo, HaloPrecond<REL>)
HALO_KERNEL(k_visc_setup_halo, HaloSetup<REL>)
HALO_KERNEL(k_cg_spmv_halo, HaloSpmv<REL>)

// ---------------------------------------------------------------- launches
// Grid of a pass: the blocks that are resident at once (found by prepare_halo_kernels, which
// also raises the shared-memory limit, before any capture).
constexpr int kMaxDevices = 64;
inline int current_device() {
    int device = 0;
    cudaGetDevice(&device);
    return device < kMaxDevices ? device : 0;
}
template <void (*K)(Dev)>
int& halo_resident() {
    static int resident[kMaxDevices] = {};
    return resident[current_device()];
}
template <void (*K)(Dev)>
cudaError_t prepare_halo(uint32_t threads, size_t smem) {
    if (halo_resident<K>() > 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int n = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, K, (int)threads, smem);
    if (e == cudaSuccess) halo_resident<K>() = n > 0 ? n : 1;
    return e;
}
template <void (*K)(Dev)>
void launch_halo(const Dev& d, uint32_t threads, size_t smem, const char* name, cudaStream_t s) {
    const uint32_t sms = d.batchBlocks / (2048u / kBlock);
    VFD_LAUNCH(name, s, K<<<sms * (uint32_t)halo_resident<K>(), threads, smem, s>>>(d));
}

#define HALO_PASSES(ACT)                                                     \
    ACT(kHaloDensity, "k_density_factor", k_density_factor_halo, HaloDensity<REL>)                                  \
    ACT(kHaloPAccelD, "k_pressure_accel", k_pressure_accel_halo_d, HaloPressureAccel<true HALO_COMMA REL>)          \
    ACT(kHaloPAccelP, "k_pressure_accel", k_pressure_accel_halo_p, HaloPressureAccel<false HALO_COMMA REL>)         \
    ACT(kHaloJacobiD, "k_jacobi_iter", k_jacobi_iter_halo_d, HaloJacobi<true HALO_COMMA REL>)                       \
    ACT(kHaloJacobiP, "k_jacobi_iter", k_jacobi_iter_halo_p, HaloJacobi<false HALO_COMMA REL>)                      \
    ACT(kHaloDivFinish, "k_div_finish", k_div_finish_halo, HaloDivFinish<REL>)                                      \
    ACT(kHaloPresInit, "k_pres_init", k_pres_init_halo, HaloPresInit<REL>)                                          \
    ACT(kHaloPresFinish, "k_pres_finish", k_pres_finish_halo, HaloPresFinish<REL>)                                  \
    ACT(kHaloPrecond, "k_visc_precond", k_visc_precond_halo, HaloPrecond<REL>)                                      \
    ACT(kHaloSetup, "k_visc_setup", k_visc_setup_halo, HaloSetup<REL>)                                              \
    ACT(kHaloSpmv, "k_cg_spmv", k_cg_spmv_halo, HaloSpmv<REL>)

template <bool REL, bool WIDE>
cudaError_t prepare_halo_kernels() {
    cudaError_t e = cudaSuccess;
#define HALO_PREPARE(ID, NAME, K, ...)                                  \
    if (e == cudaSuccess) {                                             \
        using Shape = HaloShape<__VA_ARGS__, WIDE>;                     \
        e = prepare_halo<K<REL, WIDE>>(Shape::kThreads, Shape::kSmem);  \
    }
    HALO_PASSES(HALO_PREPARE)
    return e;
}
cudaError_t prepare_halo_kernels() {
    cudaError_t e = prepare_halo_kernels<false, false>();
    if (e == cudaSuccess) e = prepare_halo_kernels<true, false>();
    if (e == cudaSuccess) e = prepare_halo_kernels<false, true>();
    return e == cudaSuccess ? prepare_halo_kernels<true, true>() : e;
}

template <bool REL, bool WIDE>
void launch_halo_pass(const Dev& d, HaloPass pass, cudaStream_t s) {
    switch (pass) {
#define HALO_LAUNCH(ID, NAME, K, ...)                                                   \
    case ID: {                                                                          \
        using Shape = HaloShape<__VA_ARGS__, WIDE>;                                     \
        launch_halo<K<REL, WIDE>>(d, Shape::kThreads, Shape::kSmem, NAME, s);           \
        break;                                                                          \
    }
        HALO_PASSES(HALO_LAUNCH)
    }
}
void launch_halo_pass(const Dev& d, HaloPass pass, cudaStream_t s) {
    const bool wide = d.haloOn == kHaloWide;
    if (d.cellRel) wide ? launch_halo_pass<true, true>(d, pass, s) : launch_halo_pass<true, false>(d, pass, s);
    else wide ? launch_halo_pass<false, true>(d, pass, s) : launch_halo_pass<false, false>(d, pass, s);
}

void launch_halo_build(const Dev& d, cudaStream_t s) {
    VFD_LAUNCH("k_halo_build", s, k_halo_build<<<d.batchBlocks / 2u, 256, 0, s>>>(d));
}
void launch_tile_form(const Dev& d, cudaStream_t s) {
    VFD_LAUNCH("k_tile_form", s, k_tile_form<<<1, 1, 0, s>>>(d));
}

}  // namespace vfd
