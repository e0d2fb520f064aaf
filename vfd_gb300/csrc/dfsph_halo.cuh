// Shapes of the staged-tile passes (dfsph_halo.cu) and the device helpers that the search and
// the loop controllers share with them.
#pragma once

#include "dfsph_common.cuh"

namespace vfd {

constexpr uint32_t kHaloLog2 = 5u;                        // 2^5 Morton cells a tile: 4x4x2
constexpr uint32_t kHaloTileCells = 1u << kHaloLog2;
constexpr uint32_t kHaloX = (1u << ((kHaloLog2 + 2u) / 3u)) + 2u, kHaloY = (1u << ((kHaloLog2 + 1u) / 3u)) + 2u,
                   kHaloZ = (1u << (kHaloLog2 / 3u)) + 2u, kHaloCells = kHaloX * kHaloY * kHaloZ;
// Two forms (Dev::haloOn). A lattice at the particles' diameter holds eight particles a cell, 256
// a tile and 1,152 a halo; a fluid at rest density ten, 320 and 1,440. The narrow form takes the
// first in one round of its threads with four blocks an SM, and spills over into a second,
// nearly empty one in the other; the wide form takes both, with three. Mean step of the viscous
// dam at 1M particles: 6.9 ms narrow and 7.7 wide from the lattice, 8.2 and 7.7 after 300 steps
// (row kernels 8.2 and 8.2), where halos above the cap walk their rows: 12.3 with the narrow one.
constexpr uint32_t kHaloNarrow = 1u, kHaloWide = 2u;
constexpr uint32_t kHaloThreads = 256u, kHaloWideThreads = 384u;
constexpr uint32_t kHaloCap = 1408u, kHaloWideCap = 1760u;
// Rounds of a block's threads over a tile's particles.
__device__ __forceinline__ uint32_t halo_rounds(uint32_t particles, uint32_t threads) {
    return (particles + threads - 1u) / threads;
}
__device__ __forceinline__ HaloCounts* halo_counts(const Dev& d) { return reinterpret_cast<HaloCounts*>(d.haloInfo + 2); }
constexpr uint32_t kHaloRow = 96u;                        // row length: kMaxNeighbors rounded up to 32

// Layouts that have staged tiles; each step chooses whether it runs on them (k_tile_form). Against
// the row kernels with four lanes a particle, a step of a viscous drop (graph) took 1374 us against 1184 at 33,000 particles, 1795 against 1732 at
// 66,000, 2180 against 2199 at 100,000 and 2705 against 3027 at 260,000; below the line there
// are too few tiles for the SMs. List places fit 32 bits up to the other. The wide form is
// chosen from a line further up: 50 steps to 350 of a viscous dam took
// 1.7 to 2.2 ms a step against 1.7 to 2.0 by rows at 157,000 particles, 2.5 to 2.8 against 2.5 to 2.6
// at 262,000, 4.0 to 4.7 against 3.7 to 4.8 at 512,000 and 7.4 to 7.7 against 8.0 to 8.3 at 1M.
constexpr uint32_t kHaloMinParticles = 100000u, kHaloMaxParticles = 1u << 28, kHaloWideMinParticles = 700000u;
// Where row entry j of slot p lies: the rows of 32 consecutive slots are interleaved, eight
// places (four gradient factors) of a slot at a time, so that a warp with a particle a lane
// loads 16 bytes a lane from consecutive addresses.
__device__ __forceinline__ size_t halo_row_at(uint32_t p, uint32_t j) {
    return ((size_t)(p >> 5) * (kHaloRow / 8u) + (j >> 3)) * 256u + (p & 31u) * 8u + (j & 7u);
}
__device__ __forceinline__ size_t halo_grad_at(uint32_t p, uint32_t j) {
    return ((size_t)(p >> 5) * (kHaloRow / 4u) + (j >> 2)) * 128u + (p & 31u) * 4u + (j & 3u);
}
// Halo cell of the stencil cell (dx, dy, dz in 0..2) around a cell of the tile.
__device__ __forceinline__ uint32_t halo_cell(uint32_t cell, uint32_t dx, uint32_t dy, uint32_t dz) {
    const uint32_t m = cell % kHaloTileCells;
    return ((compact3(m >> 2) + dz) * kHaloY + compact3(m >> 1) + dy) * kHaloX + compact3(m) + dx;
}

// Tiles of a pass: all of them, or (batches) those of the scenes still in solver loop `loop`,
// whose work list holds the prefix sums of their tile counts and their first tiles.
__device__ __forceinline__ uint32_t halo_tile_total(const Dev& d, int loop) {
    if (loop < 0 || d.nscenes == 1) return __ldg(d.haloInfo);
    return __ldg(work_list(d, loop) + 2u + 2u * d.nscenes);
}
__device__ __forceinline__ uint32_t halo_tile_at(const Dev& d, int loop, uint32_t v) {
    if (loop < 0 || d.nscenes == 1) return v;
    const uint32_t* w = work_list(d, loop);
    const uint32_t* pre = w + 3u + 2u * d.nscenes;
    const uint32_t* beg = pre + d.nscenes;
    uint32_t lo = 0, hi = __ldg(w + 1) - 1u;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (__ldg(pre + mid) <= v) lo = mid;
        else hi = mid - 1u;
    }
    return __ldg(beg + lo) + (v - __ldg(pre + lo));
}

enum HaloPass {
    kHaloDensity, kHaloPAccelD, kHaloPAccelP, kHaloJacobiD, kHaloJacobiP, kHaloDivFinish, kHaloPresInit, kHaloPresFinish,
    kHaloPrecond, kHaloSetup, kHaloSpmv
};
void launch_halo_pass(const Dev& d, HaloPass pass, cudaStream_t s);
void launch_halo_build(const Dev& d, cudaStream_t s);
void launch_tile_form(const Dev& d, cudaStream_t s);
cudaError_t prepare_halo_kernels();

}  // namespace vfd
