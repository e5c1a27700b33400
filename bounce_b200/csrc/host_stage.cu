#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "cloth_dev.cuh"
#include "host_stage.h"

namespace b3g {

namespace {

constexpr uint32_t kTile = 768;        // words a CTA moves: 256 xyz triples
constexpr uint32_t kHalfTiles = 170;   // tiles of half a block (510 KiB)
constexpr size_t kHalfWords = (size_t)kTile * kHalfTiles;
constexpr size_t kKept = 4;
// the largest calls that go through the stage, in tiles of all arrays
constexpr uint32_t kWriteTiles = 256;  // 768 KiB
constexpr uint32_t kReadTiles = 8192;  // 24 MiB

struct Block {
    int device = 0;
    float* mem = nullptr;
    cudaEvent_t done[2] = {};
};

struct Pool {
    std::mutex m;
    size_t users = 0;
    std::vector<Block> idle;
};

Pool& pool()
{
    static Pool* p = new Pool;  // not destroyed at exit: the driver may be gone by then
    return *p;
}

void free_block(Block& b)
{
    if (b.mem) cudaFreeHost(b.mem);
    for (cudaEvent_t e : b.done)
        if (e) cudaEventDestroy(e);
    b = Block();
}

bool take_block(Block& b)
{
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return false;
    {
        Pool& p = pool();
        std::lock_guard<std::mutex> lock(p.m);
        for (Block& q : p.idle)
            if (q.device == device) {
                b = q;
                q = p.idle.back();
                p.idle.pop_back();
                return true;
            }
    }
    b.device = device;
    if (cudaMallocHost(&b.mem, 2 * kHalfWords * sizeof(float)) == cudaSuccess &&
        cudaEventCreateWithFlags(&b.done[0], cudaEventDisableTiming) == cudaSuccess &&
        cudaEventCreateWithFlags(&b.done[1], cudaEventDisableTiming) == cudaSuccess)
        return true;
    free_block(b);
    cudaGetLastError();
    return false;
}

void give_block(Block& b)
{
    {
        Pool& p = pool();
        std::lock_guard<std::mutex> lock(p.m);
        if (p.users && p.idle.size() < kKept) {
            p.idle.push_back(b);
            return;
        }
    }
    free_block(b);
}

struct StageCopy {
    float* dev[kStageArrays];
    uint32_t words[kStageArrays];
    uint32_t planes[kStageArrays];
    uint32_t end[kStageArrays];  // tiles of this array and those before it
};

// CTA b moves tile first + b of the arrays, tiles counted array after array.
// The bus is what bounds it, so a warp's accesses to the host side are always
// whole 128-byte lines; triples are transposed through shared memory (stride 3:
// no bank is met twice).
template <bool TO_HOST>
__global__ void __launch_bounds__(256) k_stage_copy(const __grid_constant__ StageCopy a, float* half, uint32_t first)
{
    __shared__ float tile[kTile];
    uint32_t q = first + blockIdx.x, k = 0;
    while (q >= a.end[k]) ++k;
    if (k) q -= a.end[k - 1];
    const uint32_t t = threadIdx.x, n = a.planes[k], count = min(kTile, a.words[k] - q * kTile);
    float* dev = a.dev[k];
    float* host = half + (size_t)blockIdx.x * kTile;
    if (n == 0) {
        dev += (size_t)q * kTile;
        for (uint32_t w = t; w < count; w += 256) {
            if (TO_HOST) host[w] = dev[w];
            else dev[w] = host[w];
        }
        return;
    }
    const uint32_t i = q * (kTile / 3) + t;
    if (TO_HOST) {
        if (i < n)
            for (uint32_t c = 0; c < 3; ++c) tile[3 * t + c] = dev[(size_t)c * n + i];
        __syncthreads();
        for (uint32_t w = t; w < count; w += 256) host[w] = tile[w];
    } else {
        for (uint32_t w = t; w < count; w += 256) tile[w] = host[w];
        __syncthreads();
        if (i < n)
            for (uint32_t c = 0; c < 3; ++c) dev[(size_t)c * n + i] = tile[3 * t + c];
    }
}

// The host's part of the tiles first .. last, one copy an array.
void host_part(const StageCopy& a, char* const (&host)[kStageArrays], int used, uint32_t first, uint32_t last,
               float* half, bool to_host)
{
    for (int k = 0; k < used; ++k) {
        const uint32_t begin = k ? a.end[k - 1] : 0u;
        const uint32_t lo = std::max(first, begin), hi = std::min(last, a.end[k]);
        if (lo >= hi) continue;
        const size_t w0 = (size_t)(lo - begin) * kTile, w1 = std::min((size_t)(hi - begin) * kTile, (size_t)a.words[k]);
        float* at = half + (size_t)(lo - first) * kTile;
        if (to_host) std::memcpy(host[k] + 4 * w0, at, 4 * (w1 - w0));
        else std::memcpy(at, host[k] + 4 * w0, 4 * (w1 - w0));
    }
}

cudaError_t launch_part(const StageCopy& a, float* half, uint32_t first, uint32_t last, bool to_host, cudaStream_t st)
{
    if (to_host) k_stage_copy<true><<<last - first, 256, 0, st>>>(a, half, first);
    else k_stage_copy<false><<<last - first, 256, 0, st>>>(a, half, first);
    count_launches(1);
    return cudaGetLastError();
}

// Whether the runtime has not heard of `p`: ordinary host memory.
bool pageable(const void* p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

}  // namespace

HostStageUse::HostStageUse()
{
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.m);
    ++p.users;
}

HostStageUse::~HostStageUse()
{
    Pool& p = pool();
    std::vector<Block> idle;
    {
        std::lock_guard<std::mutex> lock(p.m);
        if (--p.users == 0) idle.swap(p.idle);
    }
    for (Block& b : idle) free_block(b);
}

cudaError_t host_stage_copy(const StageArray (&arrays)[kStageArrays], bool to_host, cudaStream_t st, bool* taken)
{
    *taken = false;
    StageCopy a{};
    char* host[kStageArrays] = {};
    uint32_t tiles = 0;
    int used = 0;
    for (const StageArray& s : arrays) {
        if (!s.host || !s.words) continue;
        if (!pageable(s.host)) return cudaSuccess;
        a.dev[used] = s.dev;
        a.words[used] = s.words;
        a.planes[used] = s.planes;
        host[used] = (char*)s.host;
        tiles += s.words / kTile + (s.words % kTile != 0);
        a.end[used++] = tiles;
    }
    if (!used || tiles > (to_host ? kReadTiles : kWriteTiles)) return cudaSuccess;
    Block b;
    if (!take_block(b)) return cudaSuccess;
    *taken = true;
    const uint32_t parts = (tiles + kHalfTiles - 1) / kHalfTiles;
    auto half = [&](uint32_t k) { return b.mem + (k & 1u) * kHalfWords; };
    auto first = [&](uint32_t k) { return std::min(k * kHalfTiles, tiles); };
    cudaError_t e = cudaSuccess;
    if (to_host) {
        auto launch = [&](uint32_t k) {
            if (e == cudaSuccess) e = launch_part(a, half(k), first(k), first(k + 1), true, st);
            if (e == cudaSuccess && k + 1 < parts) e = cudaEventRecord(b.done[k & 1u], st);
        };
        launch(0);
        for (uint32_t k = 0; k < parts && e == cudaSuccess; ++k) {
            if (k + 1 < parts) {
                launch(k + 1);
                if (e == cudaSuccess) e = cudaEventSynchronize(b.done[k & 1u]);
            } else {
                e = cudaStreamSynchronize(st);
            }
            if (e == cudaSuccess) host_part(a, host, used, first(k), first(k + 1), half(k), true);
        }
    } else {
        for (uint32_t k = 0; k < parts && e == cudaSuccess; ++k) {
            if (k >= 2 && (e = cudaEventSynchronize(b.done[k & 1u])) != cudaSuccess) break;
            host_part(a, host, used, first(k), first(k + 1), half(k), false);
            e = launch_part(a, half(k), first(k), first(k + 1), false, st);
            if (e == cudaSuccess && k + 2 < parts) e = cudaEventRecord(b.done[k & 1u], st);
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) cudaStreamSynchronize(st);  // nothing of the block is in use when it goes back
    give_block(b);
    return e;
}

}  // namespace b3g
