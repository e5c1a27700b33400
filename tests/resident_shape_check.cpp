// Host check of the on-chip CG's shapes (resident_shape.h), built by
// tests/test_resident_shape.py with g++.
//
// A replay of the kernel's index arithmetic (resident_cg.cuh, resident_solve):
// CTA k owns the rows from k chunk on; by band its halo is the rows within
// `band` of them on both sides, thread t takes the halo rows t, t + threads,
// ..., kResHalo of them, and a halo row's direction lies in the window from
// r0 - band on; listed, the halo is the rows its columns name.  Checked:
//   * every row is owned once, with a thread for it;
//   * every halo row has a thread (a row without one is read but never written);
//   * the window, z and the blocks' start lie inside the shared memory;
//   * listed shapes hold the rows the columns name, counted here by themselves.
// For one cloth (team and grid), for a batch's teams of 1 to 8, over all sizes a
// team takes and narrow, medium and full bands, and for closed tubes and grids
// in random numbering.
#include <cstdio>
#include <random>
#include <set>

#include "../bounce_b200/csrc/resident_shape.h"

using namespace b3g;

static int fail(const char* what, const ResSystem& c, const ResShape& s, uint32_t cta)
{
    std::printf("FAIL n %u band %u deg %u: grid %d ctas %u threads %u chunk %u listed %u, CTA %u: %s\n", c.n, c.band,
                c.max_deg, (int)s.grid, s.ctas, s.threads, s.chunk, s.listed, cta, what);
    return 1;
}

static int check_by_band(const ResSystem& c, const ResShape& s)
{
    if ((uint64_t)s.ctas * s.chunk < c.n) return fail("rows without a CTA", c, s, 0);
    if (s.threads > (uint32_t)kResMaxThreads || s.threads % 32u) return fail("threads", c, s, 0);
    if (s.chunk > s.threads * s.rows_per_thread) return fail("rows without a thread", c, s, 0);
    if (res_block_offset(res_rows(c.n, s.chunk, c.band, s.listed), s.grid ? 0u : 12u * s.chunk) > kResSmemLimit)
        return fail("shared memory", c, s, 0);
    for (uint32_t k = 0; k < s.ctas && !s.listed; ++k) {
        const uint32_t r0 = std::min(c.n, k * s.chunk), r1 = std::min(c.n, r0 + s.chunk);
        if (r0 == r1) continue;
        const uint32_t w0 = r0 > c.band ? r0 - c.band : 0u, w1 = std::min(c.n, r1 + c.band);
        const uint32_t halo = (r0 - w0) + (w1 - r1);
        if (halo > (uint32_t)kResHalo * s.threads) return fail("halo rows without a thread", c, s, k);
        if (w1 - w0 > res_window(c.n, s.chunk, c.band)) return fail("window", c, s, k);
    }
    return 0;
}

static int check_sizes()
{
    for (uint32_t n = 1; n <= 4096; ++n) {
        const uint32_t bands[] = {0, 1, 33, n / 3, n / 2, n - n / 8, n - 1 - (n > 1), n - 1};
        for (uint32_t band : bands) {
            const ResSystem c{n, 7u * ((n + 31u) / 32u) * 32u, 7u, std::min(band, n - 1), 0u, 0u};
            const ResShape s = resident_shape_on(c, 148);
            if (s.ctas && check_by_band(c, s)) return 1;
            for (uint32_t team = 1; team <= 8; team *= 2) {
                if (!resident_in_batch(c, team)) continue;
                const uint32_t per = ((n + 31u) / 32u + team - 1u) / team;
                ResShape b;
                b.ctas = team;
                b.chunk = 32u * per;
                b.threads = (uint32_t)kResMaxThreads;
                b.rows_per_thread = per <= 16u ? 1u : per <= 32u ? 2u : 4u;
                if (check_by_band(c, b)) return 1;
            }
        }
    }
    std::mt19937 rng(1);
    for (int q = 0; q < 20000; ++q) {
        const uint32_t n = 4097u + rng() % 160000u, deg = q % 2 ? 7u : 13u;
        const uint32_t band = rng() % (q % 3 ? 3000u : n);
        const ResSystem c{n, deg * ((n + 31u) / 32u) * 32u, deg, band, 0u, 0u};
        const ResShape s = resident_shape_on(c, 148);
        if (s.ctas && check_by_band(c, s)) return 1;
    }
    return 0;
}

// Systems that the tests of the cooperative kernels rely on: not solved on chip.
static int check_refused()
{
    const ResSystem hub{1201, 41u * 1216u, 41, 1200, 0, 0};  // a row of 41 blocks
    if (resident_shape_on(hub, 148).ctas) return fail("on chip after all", hub, ResShape(), 0);
    return 0;
}

// A grid of rows x side vertices, its triangles' couplings; closed: the last
// row is coupled to the first one; shuffled: in random numbering.
static int check_mesh(uint32_t rows, uint32_t side, bool closed, bool shuffled, bool refused = false)
{
    const uint32_t n = rows * side;
    std::vector<uint32_t> id(n);
    for (uint32_t i = 0; i < n; ++i) id[i] = i;
    std::mt19937 rng(n);
    if (shuffled) std::shuffle(id.begin(), id.end(), rng);
    std::vector<std::set<uint32_t>> nb(n);
    ResSystem c{n, 7u * ((n + 31u) / 32u) * 32u, 7u, 0u, 0u, 0u};
    auto couple = [&](uint32_t a, uint32_t b) {
        a = id[a], b = id[b];
        nb[a].insert(b), nb[b].insert(a);
        c.band = std::max(c.band, a > b ? a - b : b - a);
    };
    for (uint32_t i = 0; i < rows; ++i)
        for (uint32_t j = 0; j < side; ++j) {
            const uint32_t down = i + 1 < rows ? i + 1 : closed ? 0u : rows;
            if (j + 1 < side) couple(i * side + j, i * side + j + 1);
            if (down < rows) couple(i * side + j, down * side + j);
            if (down < rows && j + 1 < side) couple(i * side + j, down * side + j + 1);
        }
    resident_halos(c, [&](uint32_t i, auto&& f) {
        for (uint32_t j : nb[i]) f(j);
    });
    const ResShape s = resident_shape_on(c, 148);
    if (refused) return s.ctas ? fail("on chip after all", c, s, 0) : 0;
    if (!s.ctas) return 0;
    if (check_by_band(c, s)) return 1;
    for (uint32_t k = 0; k < s.ctas && s.listed; ++k) {
        std::set<uint32_t> halo;
        const uint32_t r0 = std::min(n, k * s.chunk), r1 = std::min(n, r0 + s.chunk);
        for (uint32_t i = r0; i < r1; ++i)
            for (uint32_t j : nb[i])
                if (j < r0 || j >= r1) halo.insert(j);
        if (halo.size() > s.listed || halo.size() > (size_t)kResHalo * s.threads)
            return fail("listed rows without a thread", c, s, k);
    }
    std::printf("%u x %u%s%s: %s, %u CTAs of %u threads, %u listed\n", rows, side, closed ? " closed" : "",
                shuffled ? " shuffled" : "", s.grid ? "grid" : "team", s.ctas, s.threads, s.listed);
    return 0;
}

int main()
{
    if (check_sizes() || check_refused()) return 1;
    for (uint32_t side : {240u, 268u, 300u})
        if (check_mesh(side, side, false, true, true)) return 1;
    const uint32_t sides[][2] = {{27, 27}, {33, 32}, {46, 46}, {34, 34}, {40, 40}, {48, 48}, {64, 64}, {91, 91}, {200, 128}};
    for (const auto& s : sides)
        for (int form = 0; form < 4; ++form)
            if (check_mesh(s[0], s[1], form & 1, form & 2)) return 1;
    std::printf("ok\n");
    return 0;
}
