// Shapes and launches of the on-chip MPCG (resident_cg.cuh, resident_cg.cu).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "cloth_dev.cuh"

namespace b3g {

constexpr int kResMaxThreads = 512;
constexpr int kResMaxTeam = 8;    // CTAs of a cluster
constexpr int kResMaxGrid = 160;  // CTAs of a cooperative launch
constexpr int kResSlots = 16;     // widest row
constexpr int kResFewSlots = 8;   // widest row of the forms for few blocks a row
constexpr int kResMaxWords = 128; // warps of a team
constexpr int kResBatchRows = 4;  // most rows a thread in a batch
constexpr int kResLine = 8;       // 16-byte words between two partials of a grid
constexpr int kResHalo = 4;       // halo rows a thread
constexpr uint32_t kResHeader = 4224;
constexpr uint32_t kResBatchStatic = 2048;  // static shared memory of the batch's kernel
constexpr uint32_t kResSmemLimit = 227 * 1024;

// Rows whose direction a CTA of `chunk` rows keeps: its own and the band's.
__host__ __device__ inline uint32_t res_window(uint32_t n, uint32_t chunk, uint32_t band)
{
    const uint64_t w = (uint64_t)chunk + 2ull * band;
    return w < n ? (uint32_t)w : n;
}
// Byte offset of the resident blocks in shared memory.
__host__ __device__ inline uint32_t res_block_offset(uint32_t n, uint32_t chunk, uint32_t band, bool z_in_smem,
                                                         bool wide)
{
    const uint32_t b =
        kResHeader + (wide ? 15u : 12u) * res_window(n, chunk, band) + (z_in_smem ? 12u * chunk : 0u);
    return (b + 127u) & ~127u;
}

// Whether a CTA's halo is wider than its threads hold.
__host__ __device__ inline bool res_wide(uint32_t n, uint32_t chunk, uint32_t band, uint32_t threads)
{
    return res_window(n, chunk, band) > (chunk < n ? chunk : n) + (uint32_t)kResHalo * threads;
}

struct ResShape {
    bool grid = false;       // cooperative launch, else one cluster
    bool wide = false;       // the window is listed: its halo is wider than the threads can hold
    uint32_t ctas = 0;       // 0: the cloth does not fit the on-chip form
    uint32_t threads = 0, chunk = 0, rows_per_thread = 0, smem = 0;
};
// Bytes of a grid's tagged partials: two alternating sets of two sums.
constexpr size_t kResPartialBytes = (size_t)2 * 2 * kResMaxGrid * kResLine * 16;
// The shape of cloth c's solve on the current device.
ResShape resident_shape(const ClothDev& c);
cudaError_t launch_resident_cg(const ClothDev& c, const ResShape& s, int dot, cudaStream_t st);

}  // namespace b3g
