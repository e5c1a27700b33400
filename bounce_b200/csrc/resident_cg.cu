// Launches of the on-chip MPCG (resident_cg.cuh) for one cloth.
#include "resident_cg.h"

#include "resident_cg.cuh"

namespace b3g {

namespace {

template <int DOT, int RPT, int SLOTS>
__global__ void __launch_bounds__(kResMaxThreads, 1)
    k_resident_team(const __grid_constant__ ClothDev c, uint32_t chunk, uint32_t listed, uint32_t by_blocks,
                    uint32_t smem_bytes)
{
    extern __shared__ __align__(128) char smem[];
    ResShared* sh = reinterpret_cast<ResShared*>(smem);
    TeamScope team;
    team.by_blocks = by_blocks != 0u;
    team.size = gridDim.x;  // one cluster
    team.rank = blockIdx.x;
    team.parity = 0u;
    team.sh = sh;
    team.zs = reinterpret_cast<float*>(smem + kResHeader) + 3u * (size_t)res_rows(c.n, chunk, c.band, listed);
    uint32_t phase = 0u;
    res_init_copy_barrier(sh);
    team.barrier();  // every CTA runs before another writes into it
    resident_solve<DOT, RPT, SLOTS>(c, team, smem, chunk, listed, smem_bytes, phase);
    team.barrier();  // no CTA leaves while another may still write into it
}

template <int DOT, int RPT, int SLOTS>
__global__ void __launch_bounds__(kResMaxThreads, 1)
    k_resident_grid(const __grid_constant__ ClothDev c, uint32_t chunk, uint32_t listed, uint32_t, uint32_t smem_bytes)
{
    extern __shared__ __align__(128) char smem[];
    ResShared* sh = reinterpret_cast<ResShared*>(smem);
    GridScope team;
    team.size = gridDim.x;
    team.rank = blockIdx.x;
    team.epoch = 0u;
    team.sh = sh;
    team.bar = c.bar;
    team.part = reinterpret_cast<ulonglong2*>(static_cast<char*>(c.partials) + kGridCgCounterBytes);
    team.base = *(volatile uint32_t*)&c.bar->nonce;
    const uint32_t withheld = *(volatile uint32_t*)&c.bar->count;
    team.mute = withheld == kResWithholdAll;
    team.mute_rows = withheld != 0u;
    team.row_lost = false;
    team.limit = c.bar->spin_limit ? c.bar->spin_limit : kResSpinLimit;
    team.zt = reinterpret_cast<float4*>(c.p);  // p and s, 6 n floats, are free here
    team.arrivals = *(volatile uint32_t*)&c.bar->arrivals;
    uint32_t phase = 0u;
    res_init_copy_barrier(sh);
    const bool good = resident_solve<DOT, RPT, SLOTS>(c, team, smem, chunk, listed, smem_bytes, phase);
    if (threadIdx.x == 0 && !good) {
        c.sc->status = kResTimeout;
        c.sc->cont = 0;
    }
    // the next launch's tags differ from this one's (a CTA that gave up may
    // be a reduction behind the others)
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *(volatile uint32_t*)&c.bar->arrivals = team.arrivals + team.epoch * team.size;
        *(volatile uint32_t*)&c.bar->nonce = team.base + team.epoch + 8u;
    }
}

template <int DOT, int RPT, int SLOTS>
const void* kernel_of(bool grid)
{
    return grid ? (const void*)k_resident_grid<DOT, RPT, SLOTS> : (const void*)k_resident_team<DOT, RPT, SLOTS>;
}
template <int DOT>
const void* kernel_for(bool grid, uint32_t rpt, uint32_t deg)
{
    if (rpt == 1)
        return deg <= (uint32_t)kResSlots ? kernel_of<DOT, 1, kResSlots>(grid) : kernel_of<DOT, 1, kResWideSlots>(grid);
    return deg <= (uint32_t)kResFewSlots ? kernel_of<DOT, 2, kResFewSlots>(grid) : kernel_of<DOT, 2, kResSlots>(grid);
}

}  // namespace

ResShape resident_shape(const ClothDev& c)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return resident_shape_on({c.n, c.E, c.max_deg, c.band, c.halo_team, c.halo_grid}, sms);
}

cudaError_t launch_resident_cg(const ClothDev& c, const ResShape& s, int dot, bool by_blocks, cudaStream_t st)
{
    const void* fn = dot == 2 ? kernel_for<2>(s.grid, s.rows_per_thread, c.max_deg)
                   : dot == 1 ? kernel_for<1>(s.grid, s.rows_per_thread, c.max_deg)
                              : kernel_for<0>(s.grid, s.rows_per_thread, c.max_deg);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmemLimit);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s.ctas);
    cfg.blockDim = dim3(s.threads);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (s.grid) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    } else {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = s.ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    uint32_t chunk = s.chunk, listed = s.listed, blocks = by_blocks ? 1u : 0u, bytes = s.smem;
    void* args[5] = {const_cast<ClothDev*>(&c), &chunk, &listed, &blocks, &bytes};
    e = cudaLaunchKernelExC(&cfg, fn, args);
    count_launches(1);
    return e;
}

}  // namespace b3g
