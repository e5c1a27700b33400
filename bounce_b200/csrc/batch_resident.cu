// Batched MPCG on chip: the cloths of a batch whose systems (mostly) fit the
// shared memory of their team (resident_cg.cuh), in one persistent launch of
// one CTA an SM.  Teams take cloths from a queue as in batch_cg.cu; the other
// cloths run there.
//
// Bound: the streaming kernel reads every matrix from HBM in every iteration
// (128 cloths of 16^2..128^2: 230 MB a sweep, 2.1 ms a solve at 17 iterations
// a cloth); here a matrix is read once, and a team of eight holds 1.6 MB of
// it.  What does not fit (from about 85^2 on a team of eight) comes from L2,
// which holds the 15 matrices in flight.  Measured (FP64 dots, tuned
// schedules, streaming and on chip): 128 cloths of 16^2..128^2, 2,322
// iterations, 2.42 and 1.50 ms; 400 of 16^2..30^2, 6,282 iterations, 0.50 and
// 0.30 ms; 64 of 120^2..128^2, 1,234 iterations, 3.03 and 1.72 ms.
#include <algorithm>

#include "batch.cuh"
#include "resident_cg.cuh"

namespace b3g {

namespace {

template <int DOT>
__device__ __forceinline__ void batch_solve(const ClothDev& c, TeamScope& team, char* smem, uint32_t smem_bytes,
                                            uint32_t& phase)
{
    const uint32_t slices = (c.n + 31u) >> 5, per = (slices + team.size - 1u) / team.size;
    const uint32_t chunk = 32u * per;
    team.parity = 0u;
    team.by_blocks = true;
    team.zs = reinterpret_cast<float*>(smem + kResHeader) + 3u * (size_t)res_window(c.n, chunk, c.band);
    if (per <= (uint32_t)kResMaxWarps)
        resident_solve<DOT, 1, kResSlots>(c, team, smem, chunk, 0u, smem_bytes, phase);
    else if (per <= 2u * kResMaxWarps)
        resident_solve<DOT, 2, kResFewSlots>(c, team, smem, chunk, 0u, smem_bytes, phase);
    else
        resident_solve<DOT, kResBatchRows, kResFewSlots>(c, team, smem, chunk, 0u, smem_bytes, phase);
}

// A task is one cloth split over the cluster (count 0) or up to one cloth
// for each of its CTAs.
template <int DOT>
__global__ void __launch_bounds__(kResMaxThreads, 1)
    k_batch_resident(const __grid_constant__ BatchCgArgs a, uint32_t smem_bytes)
{
    extern __shared__ __align__(128) char smem[];
    __shared__ uint32_t item;
    // the cloth's descriptor: its pointers are read from here all along
    __shared__ __align__(16) uint32_t desc[sizeof(ClothDev) / 4];
    static_assert(sizeof(ClothDev) % 4 == 0 && sizeof(ClothDev) + 64 <= kResBatchStatic, "descriptor in shared memory");
    ResShared* sh = reinterpret_cast<ResShared*>(smem);
    rcg::cluster_group cl = rcg::this_cluster();
    const uint32_t rank = cl.block_rank(), size = cl.num_blocks();
    uint32_t phase = 0u;
    res_init_copy_barrier(sh);
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) item = atomicAdd(a.next, 1u);
        cl.sync();
        const uint32_t k = *cl.map_shared_rank(&item, 0);
        cl.sync();  // also: nobody writes the shared memory of a CTA still in the last task
        if (k >= a.ntasks) break;
        const uint2 task = a.tasks[k];
        const bool split = task.y == 0;
        if (!split && rank >= task.y) continue;
        TeamScope team;
        team.sh = sh;
        team.rank = split ? rank : 0u;
        team.size = split ? size : 1u;
        const uint32_t* d = reinterpret_cast<const uint32_t*>(a.descs + a.order[split ? task.x : task.x + rank]);
        for (uint32_t i = threadIdx.x; i < sizeof(ClothDev) / 4u; i += blockDim.x) desc[i] = d[i];
        __syncthreads();
        const ClothDev& c = *reinterpret_cast<const ClothDev*>(desc);
        if constexpr (DOT >= 0) {
            batch_solve<DOT>(c, team, smem, smem_bytes, phase);
        } else {  // a batch that mixes dot precisions: each cloth's own
            const int dot = c.sc->dot;
            if (dot == 2) batch_solve<2>(c, team, smem, smem_bytes, phase);
            else if (dot == 1) batch_solve<1>(c, team, smem, smem_bytes, phase);
            else batch_solve<0>(c, team, smem, smem_bytes, phase);
        }
        __syncthreads();  // the descriptor is written again
    }
}

const void* kernel_for(int dot)
{
    switch (dot) {
        case 0: return (const void*)k_batch_resident<0>;
        case 1: return (const void*)k_batch_resident<1>;
        case 2: return (const void*)k_batch_resident<2>;
        default: return (const void*)k_batch_resident<-1>;
    }
}

}  // namespace

bool batch_on_chip(const ClothDev& c, int team)
{
    return resident_in_batch({c.n, c.E, c.max_deg, c.band, 0u, 0u}, (uint32_t)team);
}

cudaError_t launch_batch_resident(const BatchCgArgs& a, int team, int dot, cudaStream_t st)
{
    if (!a.ntasks) return cudaSuccess;
    const void* fn = kernel_for(dot);
    const uint32_t smem = kResSmemLimit - kResBatchStatic;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(team);
    cfg.blockDim = dim3(kResMaxThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = team;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3((unsigned)(team * std::max(1, std::min(clusters, (int)a.ntasks))));
    uint32_t bytes = smem;
    void* args[2] = {const_cast<BatchCgArgs*>(&a), &bytes};
    e = cudaLaunchKernelExC(&cfg, fn, args);
    count_launches(1);
    return e;
}

}  // namespace b3g
