// Persistent whole-GPU MPCG of one cloth (grid_cg.cu).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "cloth_dev.cuh"
#include "resident_cg.h"

namespace b3g {

// Software grid barrier state; its first kBarrierClear bytes are zero before
// each launch of the counter kernels.
struct GridBarrier {
    uint32_t count;       // CTA arrivals since the launch began
    uint32_t error;
    uint32_t spin_limit;  // polls before a waiting CTA gives up; 0: the built-in limit
    uint32_t arrivals;    // the on-chip CG: value of `arrived` when a launch begins
    uint32_t pad0[28];
    uint32_t arrived;     // its count of arrivals, in a line of its own
    uint32_t pad1[31];
    uint32_t nonce;       // tags it has used up; never cleared
};
constexpr size_t kBarrierClear = 12;                            // bytes cleared before a launch
constexpr size_t kBarrierReset = offsetof(GridBarrier, nonce);  // bytes cleared after a wait gave up

// Upper bound on the CTAs of one persistent CG launch; the cloth's partials
// buffer holds 8 values of the widest dot type (8 bytes) per CTA: two
// alternating sets of up to four sums.
constexpr int kMaxGridCgBlocks = 1024;
constexpr size_t kGridCgCounterBytes = (size_t)kMaxGridCgBlocks * 64;
// ... followed by the on-chip CG's tagged partials.
constexpr size_t kGridCgPartialBytes = kGridCgCounterBytes + kResPartialBytes;

struct GridCgShape {
    int blocks, threads;
};
GridCgShape grid_cg_shape(uint32_t n, int device, bool fused);
// Cooperative launch over the current device, shaped by grid_cg_shape():
// two grid reductions per iteration.
cudaError_t launch_grid_cg(const ClothDev& c, int dot, GridBarrier* bar, cudaStream_t st);
// The fused form, one grid reduction per iteration; slot 0 of every row must
// hold the row's diagonal block (it multiplies the row's own direction,
// formed in registers).  `rec`: device scratch
// of grid_cg_fused_rec_bytes(n) bytes, 16-byte aligned (the per-vertex
// records of two consecutive iterations).
cudaError_t launch_grid_cg_fused(const ClothDev& c, int dot, GridBarrier* bar, float4* rec, cudaStream_t st);
inline size_t grid_cg_fused_rec_bytes(uint32_t n) { return 2 * 3 * sizeof(float4) * (size_t)n; }


}  // namespace b3g
