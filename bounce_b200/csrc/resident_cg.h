// Shapes and launches of the on-chip MPCG (resident_cg.cuh, resident_cg.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "cloth_dev.cuh"

namespace b3g {

constexpr int kResMaxThreads = 512;
constexpr int kResMaxTeam = 8;    // CTAs of a cluster
constexpr int kResMaxGrid = 160;  // CTAs of a cooperative launch
constexpr int kResWideSlots = 32; // widest row
constexpr int kResSlots = 16;     // widest row with more than one row a thread, and in a batch
constexpr int kResFewSlots = 8;   // widest row of the forms for few blocks a row
constexpr int kResMaxWords = 128; // warps of a team
constexpr int kResBatchRows = 4;  // most rows a thread in a batch
constexpr int kResMaxSlices = kResBatchRows * kResMaxThreads / 32;  // of a CTA
constexpr int kResLine = 8;       // 16-byte words between two partials of a grid
constexpr int kResHalo = 4;       // halo rows a thread
constexpr uint32_t kResHeader = 4736;
constexpr uint32_t kResBatchStatic = 2048;  // static shared memory of the batch's kernel
constexpr uint32_t kResSmemLimit = 227 * 1024;

// Rows whose direction a CTA of `chunk` rows keeps: its own and the band's, or
// (listed != 0) its own and the halo rows it lists, `listed` at most.
__host__ __device__ inline uint32_t res_window(uint32_t n, uint32_t chunk, uint32_t band)
{
    const uint64_t w = (uint64_t)chunk + 2ull * band;
    return w < n ? (uint32_t)w : n;
}
__host__ __device__ inline uint32_t res_rows(uint32_t n, uint32_t chunk, uint32_t band, uint32_t listed)
{
    return listed ? chunk + listed : res_window(n, chunk, band);
}
// Byte offset of the resident blocks in shared memory.
__host__ __device__ inline uint32_t res_block_offset(uint32_t rows, uint32_t z_bytes)
{
    return (kResHeader + 12u * rows + z_bytes + 127u) & ~127u;
}
// Whether a CTA's band holds more halo rows than its threads.
__host__ __device__ inline bool res_wide(uint32_t n, uint32_t chunk, uint32_t band, uint32_t threads)
{
    return res_window(n, chunk, band) > (chunk < n ? chunk : n) + (uint32_t)kResHalo * threads;
}

struct ResShape {
    bool grid = false;       // cooperative launch, else one cluster
    uint32_t listed = 0;     // most halo rows of a CTA that lists them; 0: by band
    uint32_t ctas = 0;       // 0: the cloth does not fit the on-chip form
    uint32_t threads = 0, chunk = 0, rows_per_thread = 0, smem = 0;
};
// Bytes of a grid's tagged partials: two alternating sets of two sums.
constexpr size_t kResPartialBytes = (size_t)2 * 2 * kResMaxGrid * kResLine * 16;
// The shape of cloth c's solve on the current device.
ResShape resident_shape(const ClothDev& c);
// CTAs of a system of n rows on one cluster, and its rows a CTA there or on
// the grid of a 148-SM device.
uint32_t resident_team(uint32_t n);
uint32_t resident_chunk(uint32_t n, bool grid);

// Fills c.halo_team and c.halo_grid where the band is too wide for the
// threads of a CTA: the most rows outside a CTA's chunk that its rows touch.
// each(i, f): f(column) for every column of row i.  Counting ends where a CTA
// already touches more than the threads of any shape hold.
template <class Each>
void resident_halos(ClothDev& c, Each&& each)
{
    c.halo_team = c.halo_grid = 0;
    for (int grid = 0; grid < 2; ++grid) {
        const uint32_t n = c.n, chunk = resident_chunk(n, grid != 0);
        if (!chunk || !res_wide(n, chunk, c.band, kResMaxThreads)) continue;
        std::vector<uint32_t> seen(n, ~0u);
        uint32_t most = 0;
        const uint32_t bound = kResHalo * kResMaxThreads;
        for (uint32_t r0 = 0; r0 < n && most <= bound; r0 += chunk) {
            uint32_t count = 0;
            for (uint32_t i = r0; i < r0 + chunk && i < n && count <= bound; ++i)
                each(i, [&](uint32_t j) {
                    if (j - r0 >= chunk && seen[j] != r0) seen[j] = r0, ++count;
                });
            if (count > most) most = count;
        }
        (grid ? c.halo_grid : c.halo_team) = (most + 31u) & ~31u;
    }
}
// by_blocks: a cluster sums in the order of the per-iteration kernels, else in
// the cooperative CG's.
cudaError_t launch_resident_cg(const ClothDev& c, const ResShape& s, int dot, bool by_blocks, cudaStream_t st);

}  // namespace b3g
