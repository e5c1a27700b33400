// Shapes of the on-chip MPCG (resident_cg.cuh): which systems fit, on how many
// CTAs and threads, and how much shared memory.  Host arithmetic only, so that
// it can be checked without a GPU; the device code shares its constants and
// offsets.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define B3G_HD __host__ __device__
#else
#define B3G_HD
#endif

namespace b3g {

constexpr int kResMaxThreads = 512;
constexpr int kResMaxTeam = 8;    // CTAs of a cluster
constexpr int kResMaxGrid = 160;  // CTAs of a cooperative launch
constexpr int kResWideSlots = 32; // widest row
constexpr int kResSlots = 16;     // widest row with more than one row a thread, and in a batch
constexpr int kResFewSlots = 8;   // widest row of the forms for few blocks a row
constexpr int kResMaxWords = 128; // warps of a team
constexpr int kResBatchRows = 4;  // most rows a thread in a batch
constexpr int kResMaxWarps = kResMaxThreads / 32;
constexpr int kResMaxSlices = kResBatchRows * kResMaxThreads / 32;  // of a CTA
constexpr int kResLine = 8;       // 16-byte words between two partials of a grid
constexpr int kResHalo = 4;       // halo rows a thread
constexpr uint32_t kResHeader = 4736;
constexpr uint32_t kResBatchStatic = 2048;  // static shared memory of the batch's kernel
constexpr uint32_t kResSmemLimit = 227 * 1024;
// GridBarrier::count of a launch that withholds what others wait for (the
// diagnostic of the bounded waits): everything, or the rows of z.
constexpr uint32_t kResWithholdAll = 0x80000000u, kResWithholdRows = 1u;
// Bytes of a grid's tagged partials: two alternating sets of two sums.
constexpr size_t kResPartialBytes = (size_t)2 * 2 * kResMaxGrid * kResLine * 16;

// Rows whose direction a CTA of `chunk` rows keeps: its own and the band's, or
// (listed != 0) its own and the halo rows it lists, `listed` at most.
B3G_HD inline uint32_t res_window(uint32_t n, uint32_t chunk, uint32_t band)
{
    const uint64_t w = (uint64_t)chunk + 2ull * band;
    return w < n ? (uint32_t)w : n;
}
B3G_HD inline uint32_t res_rows(uint32_t n, uint32_t chunk, uint32_t band, uint32_t listed)
{
    return listed ? chunk + listed : res_window(n, chunk, band);
}
// Byte offset of the resident blocks in shared memory.
B3G_HD inline uint32_t res_block_offset(uint32_t rows, uint32_t z_bytes)
{
    return (kResHeader + 12u * rows + z_bytes + 127u) & ~127u;
}
// The most halo rows a CTA's band holds.  Not the window less a chunk: a last
// CTA of few rows has up to a chunk more of them once the window is the whole
// system.
inline uint32_t res_halo(uint32_t n, uint32_t chunk, uint32_t band)
{
    uint32_t most = 0;
    for (uint64_t r0 = 0; chunk && r0 < n; r0 += chunk) {
        const uint32_t below = (uint32_t)r0, above = n - (uint32_t)std::min<uint64_t>(n, r0 + chunk);
        most = std::max(most, std::min(below, band) + std::min(above, band));
    }
    return most;
}
// Whether that is more than `threads` threads hold.
inline bool res_wide(uint32_t n, uint32_t chunk, uint32_t band, uint32_t threads)
{
    return res_halo(n, chunk, band) > (uint32_t)kResHalo * threads;
}

// What the shape depends on: rows, blocks, widest row, widest |row - column|,
// and where that band is too wide the halo rows a CTA lists (resident_halos).
struct ResSystem {
    uint32_t n, E, max_deg, band, halo_team, halo_grid;
};

struct ResShape {
    bool grid = false;       // cooperative launch, else one cluster
    uint32_t listed = 0;     // most halo rows of a CTA that lists them; 0: by band
    uint32_t ctas = 0;       // 0: the cloth does not fit the on-chip form
    uint32_t threads = 0, chunk = 0, rows_per_thread = 0, smem = 0;
};

// CTAs of a system of n rows on one cluster, and its rows a CTA there or on
// the grid of a 148-SM device, a B200's.  (Halos are counted for that grid, when
// a cloth is laid out; with another number of SMs a system whose band is too
// wide is left to the cooperative kernels.)
inline uint32_t resident_team(uint32_t n)
{
    if (n > (uint32_t)(kResMaxTeam * kResMaxThreads)) return 0u;
    uint32_t t = 1;
    while (n > 256u && t < (uint32_t)kResMaxTeam && n > t * 128u) t *= 2;
    return t;
}
inline uint32_t resident_chunk(uint32_t n, bool grid)
{
    const uint32_t slices = (n + 31u) / 32u, ctas = grid ? 148u : resident_team(n);
    return ctas ? 32u * ((slices + ctas - 1u) / ctas) : 0u;
}

// The shape on a device of `sms` SMs.
inline ResShape resident_shape_on(const ResSystem& c, int sms)
{
    ResShape s;
    if (c.max_deg > (uint32_t)kResWideSlots || c.n == 0) return s;
    const uint32_t n = c.n, slices = (n + 31u) / 32u;
    auto shape = [&](bool grid, uint32_t ctas) {
        ResShape r;
        const uint32_t per = (slices + ctas - 1u) / ctas, most = (uint32_t)kResMaxThreads;
        r.grid = grid;
        r.chunk = 32u * per;
        r.ctas = grid ? (n + r.chunk - 1u) / r.chunk : ctas;
        r.rows_per_thread = r.chunk <= most ? 1u : 2u;
        const uint32_t own = 32u * ((per + r.rows_per_thread - 1u) / r.rows_per_thread);
        // threads without rows of their own help with the halo
        const bool wide = res_wide(n, r.chunk, c.band, most);
        if (wide && r.chunk == resident_chunk(n, grid)) r.listed = grid ? c.halo_grid : c.halo_team;
        const uint32_t halo = wide ? r.listed : res_halo(n, r.chunk, c.band);
        r.threads = std::max(own, 32u * ((halo + 32u * kResHalo - 1u) / (32u * kResHalo)));
        if (grid) r.threads = std::max(r.threads, 32u * ((r.ctas + 31u) / 32u));  // a thread a partial
        const uint64_t off = res_block_offset(res_rows(n, r.chunk, c.band, r.listed),
                                              !grid && ctas > 1u ? 12u * r.chunk : 0u);
        // (listing needs two words a 32 rows and one a halo row beside the window)
        const uint64_t all = off + std::max<uint64_t>((uint64_t)r.chunk * c.max_deg * 36u,
                                            r.listed ? 8ull * slices + 4ull * r.listed : 0ull);
        r.smem = (uint32_t)std::min<uint64_t>(all, kResSmemLimit);
        if ((wide && !r.listed) || r.threads > most) r.ctas = 0;
        // at least half of the blocks resident, on average
        if (off + (uint64_t)per * (c.E / slices) * 18u > kResSmemLimit) r.ctas = 0;
        if (r.listed && off + 8ull * slices + 4ull * r.listed > kResSmemLimit) r.ctas = 0;
        if (r.rows_per_thread > 1u && c.max_deg > (uint32_t)kResSlots) r.ctas = 0;
        return r;
    };
    // One CTA to 256 rows, then clusters of up to 8 CTAs of 128 to 512 rows,
    // then the grid.  Measured per iteration (FP64 dots, 7 blocks a row): 256
    // rows 2.6 us on one CTA and 2.9 on two; 1,024 rows 3.3 on eight CTAs, 4.2
    // on two; 4,096 rows 4.5 on eight and 6.2 on the grid; 8,281 rows (13
    // blocks) 8.5 on a cluster of 16 and 5.4 on the grid.
    if (const uint32_t t = resident_team(n)) {
        s = shape(false, t);
        if (s.ctas) return s;
    }
    return shape(true, (uint32_t)std::min(sms, kResMaxGrid));
}

// Whether a batch's team of `team` CTAs of kResMaxThreads threads solves the
// system on chip.  A window of more than half of the shared memory leaves too
// little for the blocks; more than one row a thread is for rows of up to
// kResFewSlots blocks.
inline bool resident_in_batch(const ResSystem& c, uint32_t team)
{
    const uint32_t slices = (c.n + 31u) / 32u, per = (slices + team - 1u) / team;
    if (per > (uint32_t)(kResBatchRows * kResMaxWarps)) return false;
    if (c.max_deg > (uint32_t)(per > (uint32_t)kResMaxWarps ? kResFewSlots : kResSlots)) return false;
    return !res_wide(c.n, 32u * per, c.band, kResMaxThreads) &&
           res_block_offset(res_window(c.n, 32u * per, c.band), 12u * 32u * per) <= kResSmemLimit / 2u;
}

// Fills c.halo_team and c.halo_grid where the band is too wide for the
// threads of a CTA: the most rows outside a CTA's chunk that its rows touch.
// each(i, f): f(column) for every column of row i.  Counting ends where a CTA
// already touches more than the threads of any shape hold.
template <class System, class Each>
void resident_halos(System& c, Each&& each)
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

}  // namespace b3g
