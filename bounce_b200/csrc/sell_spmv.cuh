// One row of y = A q for the SELL-32 block matrix of a cloth.
//
// The row's column indices are loaded first (up to W at a time), then all
// its blocks and the gathered q values, so a thread has the whole row's
// loads in flight together instead of one block's at a time.  Blocks are
// still summed in slot order, acc = acc + A_k q_k, with A q evaluated like
// b3Mat33 * b3Vec3 (include/bounce/common/math/mat33.h:129-132).
#pragma once

#include "cloth_dev.cuh"
#include "vec.cuh"

namespace b3g {

// L2ONLY: q is rewritten by other SMs during the same launch, so its loads
// go around L1 (ld.global.cg).  W: blocks whose loads are issued together
// (16 covers a whole row of a cloth with bending; 8 keeps kernels that must
// stay at 64 registers free of spills).
template <bool L2ONLY, int W = 16>
__device__ __forceinline__ f3 sell_row_times(const ClothDev& c, uint32_t row, const float* q)
{
    const uint32_t base = c.slice_off[row >> 5] + (row & 31u);
    const uint32_t deg = c.row_deg[row];
    const uint32_t n = c.n, E = c.E;
    const float* v = c.vals;
    f3 acc = zero3();
    for (uint32_t k0 = 0; k0 < deg; k0 += W) {
        uint32_t cl[W];
#pragma unroll
        for (int k = 0; k < W; ++k) cl[k] = (k0 + k < deg) ? c.cols[base + 32u * (k0 + k)] : 0u;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            if (k0 + k < deg) {
                const uint32_t idx = base + 32u * (k0 + k);
                const m3 a{f3{v[idx], v[E + idx], v[2 * E + idx]}, f3{v[3 * E + idx], v[4 * E + idx], v[5 * E + idx]},
                           f3{v[6 * E + idx], v[7 * E + idx], v[8 * E + idx]}};
                const uint32_t j = cl[k];
                const f3 qj = L2ONLY ? f3{__ldcg(q + j), __ldcg(q + n + j), __ldcg(q + 2 * n + j)}
                                     : f3{q[j], q[n + j], q[2 * n + j]};
                acc = acc + a * qj;
            }
        }
    }
    return acc;
}

// Walks a warp's slices q, q + step, ... of a matrix that comes from HBM in
// every pass, one slice ahead of their use: next() brings the following slice's
// blocks and columns into L2, one bulk prefetch a value plane.  The 16 warps an
// SM has room for keep, with loads alone, less in flight than HBM delivers (at
// 1024^2 DRAM 35 % busy and 19.5 cycles of long scoreboard an issue); the
// two-phase CG there went from 146 to 121 us an iteration.  Two slices ahead is
// too many (151 us): they leave L2 again before they are read.  The offsets are
// themselves loaded a slice before their prefetch, so nothing waits for them.
// ON = false: nothing.
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
template <bool ON>
struct SliceAhead {
    uint32_t q, step, so, len;
    __device__ __forceinline__ void fetch(const ClothDev& c)
    {
        q += step;
        so = len = 0u;
        if (q < c.nslices) so = c.slice_off[q], len = c.slice_off[q + 1] - so;
    }
    __device__ __forceinline__ SliceAhead(const ClothDev& c, uint32_t first, uint32_t step_)
        : q(first), step(step_), so(0), len(0)
    {
        if (ON) fetch(c);
    }
    __device__ __forceinline__ void next(const ClothDev& c)
    {
        if (!ON) return;
        const uint32_t lane = threadIdx.x & 31u;
        if (len && lane < 9u) prefetch_l2(c.vals + (size_t)lane * c.E + so, 4u * len);
        else if (len && lane == 9u) prefetch_l2(c.cols + so, 4u * len);
        fetch(c);
    }
};

}  // namespace b3g
