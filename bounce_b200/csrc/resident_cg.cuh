// The MPCG of one cloth with its system held on chip: device code shared by
// the single-cloth launches (resident_cg.cu) and the batch (batch_resident.cu).
//
// A team of CTAs owns the cloth's rows in contiguous chunks, at most RPT rows
// a thread.  For the whole solve a CTA keeps in shared memory
//  * its rows' blocks, copied once by bulk copies in the SELL layout (a slice's
//    component q is one contiguous run of 128 bytes a slot), as many slices as
//    fit; the rest are read from L2 in every product;
//  * the direction p of its window: its own rows and every row within `band`
//    of them (band = the widest |row - column| of the matrix) or, where few
//    rows of so wide a band are needed, those it lists at the start; so a
//    product gathers p from shared memory only.
// x, r, z, p and P^-1 of its own rows and their column indices stay in
// registers (with more than two rows a thread, x and P^-1 in L2, z in shared memory
// and p in its window).  Per iteration only z of the window's halo crosses CTAs: the
// halo's p = z + beta p_old is formed where it is needed, from the same float
// expression as its owner's.
//
// An iteration (b3SolveMPCG, src/bounce/cloth/cloth_force_solver.cpp:61-136):
//   A: p = z + beta p_old, s = S A p, p.s                     -> alpha
//   B: x += alpha p, r -= alpha s, z = S P^-1 r, r.z          -> delta', beta
// Each phase ends in a team reduction; B's also publishes z.
//
// Two kinds of team:
//  * TeamScope: one CTA, or a cluster whose CTAs store their partials into
//    each other's shared memory; one cluster barrier a reduction, z read from
//    the owner's shared memory.
//  * GridScope: the CTAs of a cooperative launch.  Partials and rows of z are
//    published as 16-byte words that carry a tag of the launch and the
//    reduction, so that a reader knows whether it has them: no fence (one a
//    phase costs 0.75 us), only a count of arrivals.
#pragma once

#include <cooperative_groups.h>

#include "cg_common.cuh"
#include "cloth_dev.cuh"
#include "grid_cg.cuh"
#include "resident_cg.h"
#include "vec.cuh"

namespace b3g {

namespace {

namespace rcg = cooperative_groups;

constexpr uint32_t kResSpinLimit = 1u << 24;
constexpr uint32_t kResTimeout = 7;  // B3G_ERR_TIMEOUT

// The fixed part of the shared memory.
struct ResShared {
    double wsum[2][2][kResMaxWords];  // [parity][value][warp of the team]
    unsigned long long mbar;
    int lost;
    uint32_t copied;               // blocks made resident
    uint32_t len[kResMaxSlices];   // per slice of the CTA: its blocks,
    uint32_t at[kResMaxSlices];    // and where they lie (~0: in L2)
};
static_assert(sizeof(ResShared) <= kResHeader, "fixed shared memory of the resident CG");

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- sums -------------------------------------------------------------------

template <class T>
__device__ __forceinline__ unsigned long long pack8(T a)
{
    unsigned long long u = 0ull;
    memcpy(&u, &a, sizeof(T));
    return u;
}
template <class T>
__device__ __forceinline__ T unpack8(unsigned long long u)
{
    T a;
    memcpy(&a, &u, sizeof(T));
    return a;
}

template <class D>
__device__ __forceinline__ typename D::T warp_sum(typename D::T v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = D::combine(v, D::shfl(v, off));
    return v;
}

// The sum of `count` 8-byte words in shared memory, a warp's sum each, in the
// order of the kernels these solves stand in for, so that FP32 sums come out
// the same.  by_blocks: block_reduce and grid_reduce (cg_common.cuh) over
// blocks of eight warps, a tree over each eight and a tree over the blocks;
// else the cooperative CG's (grid_cg.cu) for one-warp CTAs: lane l adds words
// l, l + 32, ... and a shuffle tree adds the lanes.  Up to 16 words by one
// thread, else by a warp with the sum in lane 0.
template <class D>
__device__ __forceinline__ typename D::T words_sum(const double* w, uint32_t count, bool by_blocks)
{
    typedef typename D::T T;
    T a[kResMaxWarps];
#pragma unroll
    for (uint32_t k = 0; k < (uint32_t)kResMaxWarps; ++k)
        a[k] = k < count ? *reinterpret_cast<const T*>(w + k) : D::zero();
    if (by_blocks) {
#pragma unroll
        for (int step = 4; step > 0; step >>= 1)
#pragma unroll
            for (int k = 0; k < step; ++k) {
                a[k] = D::combine(a[k], a[k + step]);
                a[k + 8] = D::combine(a[k + 8], a[k + 8 + step]);
            }
        return D::combine(a[0], a[8]);
    }
#pragma unroll
    for (int step = kResMaxWarps / 2; step > 0; step >>= 1)
#pragma unroll
        for (int k = 0; k < step; ++k) a[k] = D::combine(a[k], a[k + step]);
    return a[0];
}
template <class D>
__device__ __forceinline__ typename D::T words_sum_warp(const double* w, uint32_t count, bool by_blocks)
{
    typedef typename D::T T;
    const uint32_t lane = threadIdx.x & 31u;
    T a[kResMaxWords / 32];
#pragma unroll
    for (uint32_t m = 0; m < (uint32_t)kResMaxWords / 32u; ++m) {
        const uint32_t i = lane + 32u * m;
        a[m] = i < count ? *reinterpret_cast<const T*>(w + i) : D::zero();
        if (by_blocks && 32u * m < count)
#pragma unroll
            for (int off = 4; off > 0; off >>= 1) a[m] = D::combine(a[m], D::shfl(a[m], off));
    }
    if (!by_blocks) {
#pragma unroll
        for (uint32_t m = 1; m < (uint32_t)kResMaxWords / 32u; ++m)
            if (lane + 32u * m < count) a[0] = D::combine(a[0], a[m]);
        return warp_sum<D>(a[0]);
    }
    // blocks 4 m + lane / 8: a tree over sixteen
    if (count > 32u) {
        a[0] = D::combine(a[0], a[2]);
        a[1] = D::combine(a[1], a[3]);
        a[0] = D::combine(a[0], a[1]);
    }
    a[0] = D::combine(a[0], D::shfl(a[0], 16));
    return D::combine(a[0], D::shfl(a[0], 8));
}

// One CTA (size 1) or the CTAs of a thread-block cluster.
struct TeamScope {
    static constexpr bool kGrid = false;
    uint32_t rank, size, parity;
    uint32_t word, words;  // this warp's word of the sums (kResMaxWords: none), and how many there are
    bool by_blocks;        // the order of the sums (words_sum)
    ResShared* sh;
    float* zs;  // 3 planes of `chunk`: z of this CTA's rows, read by the team

    __device__ void barrier() const
    {
        if (size == 1) __syncthreads();
        else rcg::this_cluster().sync();
    }

    // The team's sums, the same in every thread: every warp stores its sum
    // into each CTA of the team, one barrier, and every thread adds them up.
    // A buffer is written again only two reductions later, after the barrier
    // in between.
    template <class D, int NV>
    __device__ bool sum(typename D::T (&v)[NV])
    {
        typedef typename D::T T;
        const uint32_t lane = threadIdx.x & 31u;
        parity ^= 1u;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const unsigned long long u = __shfl_sync(0xffffffffu, pack8(warp_sum<D>(v[k])), 0);
            double* mine = &sh->wsum[parity][k][word];
            if (lane < size && word < (uint32_t)kResMaxWords) {
                double* to = size == 1 ? mine : rcg::this_cluster().map_shared_rank(mine, lane);
                *reinterpret_cast<unsigned long long*>(to) = u;
            }
        }
        barrier();
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const double* w = sh->wsum[parity][k];
            if (words <= (uint32_t)kResMaxWarps) v[k] = words_sum<D>(w, words, by_blocks);
            else v[k] = unpack8<T>(__shfl_sync(0xffffffffu, pack8(words_sum_warp<D>(w, words, by_blocks)), 0));
        }
        return true;
    }
    __device__ void put_z(const ClothDev&, uint32_t, uint32_t local, uint32_t chunk, f3 z) const
    {
        if (size > 1) st3(zs, chunk, local, z);
    }
    __device__ f3 get_z(const ClothDev&, uint32_t row, uint32_t chunk, uint32_t) const
    {
        const uint32_t owner = row / chunk;
        return ld3(rcg::this_cluster().map_shared_rank(zs, owner), chunk, row - owner * chunk);
    }
};

// The CTAs of a cooperative launch.
struct GridScope {
    static constexpr bool kGrid = true;
    uint32_t rank, size, epoch, base, arrivals;
    ResShared* sh;
    GridBarrier* bar;
    ulonglong2* part;  // [parity][value][rank], a line each
    float4* zt;        // z of every row and a tag of the reduction that follows it
    uint32_t limit;
    bool mute, mute_rows;  // the diagnostic of the bounded waits: nothing, or no row of z, is published
    bool row_lost;         // this thread gave up on a row

    static __device__ void put(ulonglong2* p, unsigned long long v, unsigned long long tag)
    {
        asm volatile("{.reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t;}" ::"l"(p), "l"(v),
                     "l"(tag)
                     : "memory");
    }
    static __device__ void get(const ulonglong2* p, unsigned long long& v, unsigned long long& tag)
    {
        asm volatile("{.reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t;}"
                     : "=l"(v), "=l"(tag)
                     : "l"(p)
                     : "memory");
    }
    __device__ bool failed() const { return *(volatile uint32_t*)&bar->error == base + 1u; }
    __device__ void fail() const { *(volatile uint32_t*)&bar->error = base + 1u; }

    // A row's z travels with its tag in one 16-byte word, so whoever reads
    // the tag has the row: no fence, and the reduction that follows moves no
    // data but its partials.  The tag is a NaN that no arithmetic makes.
    __device__ uint32_t z_tag() const { return 0xffc00000u | ((base + epoch) & 0x3fffffu); }
    __device__ void put_z(const ClothDev&, uint32_t row, uint32_t, uint32_t, f3 z) const
    {
        if (mute_rows) return;
        put(reinterpret_cast<ulonglong2*>(zt + row),
            (unsigned long long)__float_as_uint(z.x) | ((unsigned long long)__float_as_uint(z.y) << 32),
            (unsigned long long)__float_as_uint(z.z) | ((unsigned long long)z_tag() << 32));
    }
    // Row `row` as published under `tag`; the wait is bounded.  Giving up shows in
    // the next reduction: at once, another thread still at the end of the last
    // one might see it there and leave the block's barriers by itself.
    __device__ f3 get_z(const ClothDev&, uint32_t row, uint32_t, uint32_t tag)
    {
        unsigned long long a, b;
        for (uint32_t spins = 0;; ++spins) {
            get(reinterpret_cast<const ulonglong2*>(zt + row), a, b);
            if ((uint32_t)(b >> 32) == tag) break;
            if (out_of_time(spins)) {
                row_lost = true;
                break;
            }
        }
        return f3{__uint_as_float((uint32_t)a), __uint_as_float((uint32_t)(a >> 32)), __uint_as_float((uint32_t)b)};
    }

    // The grid's sums.  Each CTA counts itself in and publishes its partial as
    // one tagged 16-byte word in a line of its own; once the count is full,
    // thread r of every CTA reads rank r's partial, and all sum them in the
    // same order (lane l ranks l, l + 32, ..., then a shuffle tree).  Neither the
    // count nor the partials carry a fence: a partial that is not there yet is
    // known by its tag and looked at again.  One thread a CTA polls the count
    // because polling all partials from every CTA delays the stores they wait
    // for (an all-reduce of 148 CTAs: 1.2 us polling the count, 3.5 us and more
    // polling the partials while CTAs arrive apart, or with several partials a
    // line).  Two buffers suffice: a CTA publishes reduction e + 2 only once
    // every CTA has counted itself in for e + 1, and so has read e.  The waits
    // are bounded; false (in every thread) on error.
    template <class D, int NV>
    __device__ void publish(typename D::T (&v)[NV])
    {
        typedef typename D::T T;
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
        double* w = &sh->wsum[0][0][0];
        ++epoch;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const T a = warp_sum<D>(v[k]);
            if (lane == 0) *reinterpret_cast<T*>(w + k * kResMaxWarps + warp) = a;
        }
        __syncthreads();
        if (mute) return;
        if (threadIdx.x == 0)
            asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(&bar->arrived) : "memory");
        if (threadIdx.x < (uint32_t)NV) {
            // the warps in order, as the cooperative CG (grid_cg.cu) adds them
            const double* mine = w + threadIdx.x * kResMaxWarps;
            T a = *reinterpret_cast<const T*>(mine);
            for (uint32_t q = 1; q < nw; ++q) a = D::combine(a, *reinterpret_cast<const T*>(mine + q));
            put(part + (((epoch & 1u) * 2u + lane) * kResMaxGrid + rank) * kResLine, pack8(a), base + epoch);
        }
    }
    __device__ bool out_of_time(uint32_t spins) const
    {
        if (spins <= limit && ((spins & 63u) != 63u || !failed())) return false;
        fail();
        return true;
    }
    // For the waits that a block barrier follows before anyone reads `lost`.
    __device__ bool give_up(uint32_t spins) const
    {
        if (!out_of_time(spins)) return false;
        sh->lost = 1;
        return true;
    }
    template <class D, int NV>
    __device__ bool collect(typename D::T (&v)[NV])
    {
        typedef typename D::T T;
        const uint32_t lane = threadIdx.x & 31u;
        double* w = &sh->wsum[0][0][0] + 2 * kResMaxWarps;  // [value][rank]
        if (row_lost) sh->lost = 1;
        if (threadIdx.x == 0) {
            const uint32_t target = arrivals + epoch * size;
            for (uint32_t spins = 0;; ++spins) {
                uint32_t a;
                asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(a) : "l"(&bar->arrived) : "memory");
                if ((int32_t)(a - target) >= 0 || give_up(spins)) break;
            }
        }
        __syncthreads();
        if (threadIdx.x < size) {
            const uint32_t r = threadIdx.x;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const ulonglong2* from = part + (((epoch & 1u) * 2u + k) * kResMaxGrid + r) * kResLine;
                unsigned long long u, t;
                for (uint32_t spins = 0;; ++spins) {
                    get(from, u, t);
                    if (t == base + epoch || give_up(spins)) break;
                }
                *reinterpret_cast<T*>(w + k * kResMaxGrid + r) = unpack8<T>(u);
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            T a = D::zero();
#pragma unroll
            for (uint32_t m = 0; m < (uint32_t)kResMaxGrid / 32u; ++m)
                if (lane + 32u * m < size) a = D::combine(a, *reinterpret_cast<const T*>(w + k * kResMaxGrid + lane + 32u * m));
            v[k] = unpack8<T>(__shfl_sync(0xffffffffu, pack8(warp_sum<D>(a)), 0));
        }
        return sh->lost == 0;
    }
};

// ---- the solve --------------------------------------------------------------

// cg_stop (cg_common.cuh) with its bound computed once.
struct StopBound {
    double bound = 0.0;
    bool single = false;
    __device__ StopBound() {}
    __device__ StopBound(const StepScalars* sc, double b_delta, int dot)
    {
        const double tol = (double)sc->tol;
        single = sc->stop_rule == 0 && dot != 2;
        bound = sc->stop_rule != 0 ? tol * tol * b_delta
                : single           ? (double)(kEps * kEps * (float)b_delta)
                                   : (double)(kEps * kEps) * b_delta;
    }
    __device__ bool met(double delta) const { return (single ? (double)(float)delta : delta) <= bound; }
};

// One row: its blocks' first word (in the resident blocks or in ClothDev::vals),
// its slice's width, and the window indices of its columns, two a word.
template <int SLOTS>
struct ResRow {
    static constexpr int kSlots = SLOTS;
    uint32_t off, width;
    uint32_t col[SLOTS / 2];
};

template <int I>
struct ResInt {
    static constexpr int value = I;
};

// Word `q` cs of slot K: in shared memory at byte address a (+ 128 K), or in global memory.
template <int K>
__device__ __forceinline__ float res_word(uint32_t a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(128 * K));
    return v;
}
template <int K>
__device__ __forceinline__ float res_word(const float* a)
{
    return a[32 * K];
}

// p of window row j: three words a row, so that a warp's rows fall on
// different banks and one address serves the three.
__device__ __forceinline__ f3 ldp(const float* P, uint32_t j) { return f3{P[3 * j], P[3 * j + 1], P[3 * j + 2]}; }
__device__ __forceinline__ void stp(float* P, uint32_t j, f3 v)
{
    P[3 * j] = v.x;
    P[3 * j + 1] = v.y;
    P[3 * j + 2] = v.z;
}

// The blocks and directions of slots K .. K + G - 1, then their products in
// slot order, acc = acc + A_k p_k (b3Mat33 * b3Vec3, include/bounce/common/
// math/mat33.h:129-132): the loads of the G slots are in flight together.
template <int K, int G, class R, class A>
__device__ __forceinline__ f3 res_slots(f3 acc, const R& r, const A (&a)[9], const float* P)
{
    m3 m[G];
    f3 p[G];
    auto load = [&](auto g) {
        constexpr int k = K + decltype(g)::value;
        p[k - K] = ldp(P, (k & 1) ? r.col[k >> 1] >> 16 : r.col[k >> 1] & 0xffffu);
        m[k - K] = m3{f3{res_word<k>(a[0]), res_word<k>(a[1]), res_word<k>(a[2])},
                      f3{res_word<k>(a[3]), res_word<k>(a[4]), res_word<k>(a[5])},
                      f3{res_word<k>(a[6]), res_word<k>(a[7]), res_word<k>(a[8])}};
    };
    load(ResInt<0>());
    if constexpr (G > 1) load(ResInt<1>());
    if constexpr (G > 2) load(ResInt<2>()), load(ResInt<3>());
#pragma unroll
    for (int g = 0; g < G; ++g) acc = acc + m[g] * p[g];
    return acc;
}

// s_i = sum_k A_k p_k of one row.  The warp walks its slice's width (a row's
// padding holds zero blocks on the diagonal's column): fours where one row a
// thread leaves the registers for them (spills would go to L2: shared memory
// takes nearly all of L1), then a pair and a single slot.
template <int G, int K, class R, class A>
__device__ __forceinline__ f3 res_walk(f3 acc, const R& r, const A (&a)[9], const float* P)
{
    if constexpr (K < R::kSlots) {
        if (K + (uint32_t)G <= r.width) {
            acc = res_slots<K, G>(acc, r, a, P);
            return res_walk<G, K + G>(acc, r, a, P);
        }
        if constexpr (G > 2) {
            if (K + 2u <= r.width) {
                acc = res_slots<K, 2>(acc, r, a, P);
                if (K + 3u == r.width) acc = res_slots<K + 2, 1>(acc, r, a, P);
                return acc;
            }
        }
        if (K + 1u == r.width) acc = res_slots<K, 1>(acc, r, a, P);
    }
    return acc;
}
template <int G, class R>
__device__ __forceinline__ f3 res_row_times(const R& r, uint32_t blocks, const float* P)
{
    uint32_t a[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) a[q] = blocks + 4u * (r.off + q * 32u * r.width);
    return res_walk<G, 0>(zero3(), r, a, P);
}
template <int G, class R>
__device__ __forceinline__ f3 res_row_times(const R& r, const float* blocks, uint32_t plane, const float* P)
{
    const float* a[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) a[q] = blocks + r.off + (size_t)q * plane;
    return res_walk<G, 0>(zero3(), r, a, P);
}

// The whole solve by a team.  `smem`: kResHeader bytes (the scope's
// ResShared), then P (3 floats a row of the window), zs (3 chunk floats, clusters only), then
// the blocks from a_off on, up to smem_bytes.  `listed`: the CTA keeps p of the rows its rows touch
// (c.halo of them at most) instead of the band's.  `phase`: the copy barrier's
// phase, kept over the solves of a persistent launch; the barrier is
// initialised by the caller.  Returns false when a bounded wait gave up.
template <int DOT, int RPT, int SLOTS, class S>
__device__ bool resident_solve(const ClothDev& c, S& team, char* smem, uint32_t chunk, uint32_t listed,
                               uint32_t smem_bytes, uint32_t& phase)
{
    typedef DotT<DOT> D;
    typedef typename D::T T;
    constexpr bool kLean = RPT > 2;
    constexpr int G = RPT > 1 ? 2 : 4;
    const uint32_t n = c.n, B = blockDim.x, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nw = B >> 5;
    const StepScalars* sc = c.sc;
    const uint32_t r0 = min(n, team.rank * chunk), r1 = min(n, r0 + chunk);
    const bool empty = r0 == r1;  // a CTA past the last row still joins the reductions
    const uint32_t w0 = empty ? r0 : r0 > c.band ? r0 - c.band : 0u, w1 = empty ? r0 : min(n, r1 + c.band);
    // Local numbering of p: by band, the window from w0 on; listed (most of the
    // band is not needed), the CTA's rows and then the halo rows they touch.
    float* P = reinterpret_cast<float*>(smem + kResHeader);
    const bool zin = !S::kGrid && (kLean || team.size > 1);
    const uint32_t a_off = res_block_offset(res_rows(n, chunk, c.band, listed), zin ? 12u * chunk : 0u);
    float* As = reinterpret_cast<float*>(smem + a_off);
    const uint32_t q0 = r0 >> 5, q1 = empty ? q0 : (r1 + 31u) >> 5;
    if constexpr (!S::kGrid) {
        // one row a thread: a word a slice, summed in the order of the
        // per-iteration kernels (their FP32 sums come out the same)
        team.word = RPT > 1 ? team.rank * nw + warp : q0 + warp < q1 ? q0 + warp : (uint32_t)kResMaxWords;
        team.words = RPT > 1 ? team.size * nw : (n + 31u) >> 5;
    }
    const uint32_t room = (smem_bytes - a_off) / 36u;  // blocks
    // The resident slices: the widest that fit, since a slice left in L2 costs
    // its row's loads in turn.  (A CTA has at most kResMaxSlices slices.)
    __syncthreads();  // earlier reads of the buffer and of these are done
    const uint32_t nq = q1 - q0;
    if (tid < nq) team.sh->len[tid] = c.slice_off[q0 + tid + 1u] - c.slice_off[q0 + tid];
    if (tid == 0) team.sh->copied = 0u;
    __syncthreads();
    if (tid < nq) {
        const uint32_t len = team.sh->len[tid];
        uint32_t before = 0u;
        for (uint32_t j = 0; j < nq; ++j) {
            const uint32_t o = team.sh->len[j];
            if (o > len || (o == len && j < tid)) before += o;
        }
        const bool fits = before + len <= room;
        team.sh->at[tid] = fits ? before : ~0u;
        if (fits) atomicAdd(&team.sh->copied, len);
    }
    __syncthreads();

    ResRow<SLOTS> row[RPT];
    f3 r[RPT], s[RPT];
    f3 x[kLean ? 1 : RPT], z[kLean ? 1 : RPT], p[kLean ? 1 : RPT], pv[kLean ? 1 : RPT];
    uint32_t flags = 0u;  // per row: bit i active, bit 8 + i dynamic, bit 16 + i resident
    const uint32_t below = listed ? 0u : r0 - w0;  // local index of the CTA's first row
    uint32_t halo = r0 - w0 + (w1 - r1);
    uint32_t* bits = reinterpret_cast<uint32_t*>(As);  // scratch until the blocks are copied: a bit a row,
    uint32_t* rank_of = bits + (n + 31u) / 32u;        // the bits before each word,
    uint32_t* rows_of = rank_of + (n + 31u) / 32u;     // and the listed rows
    if (listed) {
        const uint32_t words = (n + 31u) / 32u;
        for (uint32_t i = tid; i < words; i += B) bits[i] = 0u;
        __syncthreads();
        for (uint32_t q = q0 + warp; q < q1; q += nw)
            for (uint32_t o = c.slice_off[q] + lane; o < c.slice_off[q + 1]; o += 32u) {
                const uint32_t col = c.cols[o];
                if (col < r0 || col >= r1) atomicOr(bits + (col >> 5), 1u << (col & 31u));
            }
        __syncthreads();
        // thread t numbers the rows of its run of words
        const uint32_t run = (words + B - 1u) / B, i0 = min(words, tid * run), i1 = min(words, i0 + run);
        uint32_t mine = 0u;
        for (uint32_t i = i0; i < i1; ++i) mine += __popc(bits[i]);
        uint32_t upto = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, upto, off);
            if (lane >= (uint32_t)off) upto += o;
        }
        uint32_t* warp_total = reinterpret_cast<uint32_t*>(&team.sh->wsum[0][0][0]);
        if (lane == 31u) warp_total[warp] = upto;
        __syncthreads();
        uint32_t at = upto - mine;
        halo = 0u;
        for (uint32_t q = 0; q < nw; ++q) {
            if (q < warp) at += warp_total[q];
            halo += warp_total[q];
        }
        for (uint32_t i = i0; i < i1; ++i) {
            rank_of[i] = at;
            for (uint32_t m = bits[i]; m; m &= m - 1u) rows_of[at++] = 32u * i + (uint32_t)__ffs(m) - 1u;
        }
        __syncthreads();
    }
    uint32_t hrow[kResHalo];  // the thread's halo rows
#pragma unroll
    for (int u = 0; u < kResHalo; ++u) {
        const uint32_t h = tid + u * B;
        hrow[u] = h >= halo ? ~0u : listed ? rows_of[h] : h < below ? w0 + h : r1 + (h - below);
    }
    auto halo_at = [&](int u) -> uint32_t { return listed ? chunk + tid + u * B : hrow[u] - w0; };
    auto local = [&](uint32_t col) -> uint32_t {
        if (!listed) return col - w0;
        if (col >= r0 && col < r1) return col - r0;
        return chunk + rank_of[col >> 5] + __popc(bits[col >> 5] & ((1u << (col & 31u)) - 1u));
    };
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const uint32_t q = q0 + warp + i * nw, g = 32u * q + lane;
        row[i].off = row[i].width = 0u;
        r[i] = s[i] = zero3();
        if constexpr (!kLean) x[i] = z[i] = p[i] = pv[i] = zero3();
#pragma unroll
        for (int k = 0; k < SLOTS / 2; ++k) row[i].col[k] = 0u;
        if (q < q1 && g < r1) {
            const uint32_t so = c.slice_off[q];
            const uint32_t at = team.sh->at[q - q0];
            const bool res = at != ~0u;
            const bool dyn = c.type[g] == 2;
            flags |= (1u << i) | (dyn ? 0x100u << i : 0u) | (res ? 0x10000u << i : 0u);
            const uint32_t len = c.slice_off[q + 1] - so;
            row[i].width = len >> 5;
            row[i].off = (res ? 9u * at : so) + lane;
#pragma unroll
            for (int k = 0; k < SLOTS; ++k)
                if ((uint32_t)k < row[i].width)
                    row[i].col[k >> 1] |= local(c.cols[so + lane + 32u * k]) << ((k & 1) * 16);
            if constexpr (!kLean) pv[i] = ld3(c.pinv, n, g);
        }
    }
    const bool copies = team.sh->copied != 0u;
    if (copies) {
        __syncthreads();  // the scratch is free
        if (tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&team.sh->mbar)),
                         "r"(team.sh->copied * 36u)
                         : "memory");
        }
        __syncthreads();
        for (uint32_t k = tid; k < 9u * nq; k += B) {
            const uint32_t q = k / 9u, comp = k % 9u;
            const uint32_t at = team.sh->at[q], len = team.sh->len[q];
            if (at != ~0u && len)
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        smem_addr(As + 9u * (size_t)at + (size_t)comp * len)),
                    "l"(c.vals + (size_t)comp * c.E + c.slice_off[q0 + q]), "r"(len * 4u), "r"(smem_addr(&team.sh->mbar))
                    : "memory");
        }
    }
    // x0 = S m_x over the CTA's rows and its halo (cg_soft: on every row)
    auto start_at = [&](uint32_t j) -> f3 { return (c.cg_soft || c.type[j] == 2) ? ld3(c.mx, n, j) : zero3(); };
    for (uint32_t j = r0 + tid; j < r1; j += B) stp(P, below + j - r0, start_at(j));
#pragma unroll
    for (int u = 0; u < kResHalo; ++u)
        if (hrow[u] != ~0u) stp(P, halo_at(u), start_at(hrow[u]));
    bool landed = true;
    if (copies) {
        const uint32_t mb = smem_addr(&team.sh->mbar);
        uint32_t done = 0u;
        for (uint32_t t = 0; !done && t < (1u << 20); ++t)
            asm volatile("{.reg .pred q; mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2; selp.u32 %0, 1, 0, q;}"
                         : "=r"(done)
                         : "r"(mb), "r"(phase)
                         : "memory");
        phase ^= 1u;
        landed = done != 0u;
    }
    __syncthreads();

    const uint32_t as_addr = smem_addr(As);
    f3 zh[kResHalo];  // z of the thread's halo rows
    uint32_t tag = 0u;
    // the sums of the phase that made z, and the halo's z
    auto sum_and_halo = [&](auto& v) -> bool {
        constexpr int NV = sizeof(v) / sizeof(v[0]);
        bool good;
        if constexpr (S::kGrid) {
            tag = team.z_tag();
            team.template publish<D, NV>(v);
            good = team.template collect<D, NV>(v);
        } else {
            good = team.template sum<D, NV>(v);
        }
#pragma unroll
        for (int u = 0; u < kResHalo; ++u)
            if (hrow[u] != ~0u) zh[u] = team.get_z(c, hrow[u], chunk, tag);
        return good;
    };
    const uint32_t max_iter = sc->max_iter;
    uint32_t it = 0, status = 0u;
    float beta = 0.0f;
    double b_delta = 0.0, delta = 0.0, delta0 = 0.0;
    StopBound stop;
    // The first pass multiplies A x0, every later one A p.
    for (bool start = true;; start = false) {
        if (!start) {
            // the window's p = z + beta p_old (cloth_force_solver.cpp:130)
            const bool first = it == 0;
#pragma unroll
            for (int u = 0; u < kResHalo; ++u)
                if (hrow[u] != ~0u) {
                    const uint32_t l = halo_at(u);
                    stp(P, l, first ? zh[u] : zh[u] + beta * ldp(P, l));
                }
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                if ((flags >> i) & 1u) {
                    const uint32_t l = below + 32u * (warp + i * nw) + lane;
                    if constexpr (kLean) {
                        const f3 zi = ld3(team.zs, chunk, l - below);
                        stp(P, l, first ? zi : zi + beta * ldp(P, l));
                    } else {
                        p[i] = first ? z[i] : z[i] + beta * p[i];
                        stp(P, l, p[i]);
                    }
                }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            s[i] = zero3();
            if ((flags >> (16 + i)) & 1u) s[i] = res_row_times<G>(row[i], as_addr, P);
            else if (row[i].width) s[i] = res_row_times<SLOTS == kResFewSlots ? 4 : G>(row[i], c.vals, c.E, P);
            if (!((flags >> (8 + i)) & 1u) && !start) s[i] = zero3();
        }
        if (start) {
            // r = S (b - A x0), z = S P^-1 r, b_delta, delta (cloth_force_solver.cpp:90-100;
            // softbody_force_solver.cpp:93-127 with cg_soft)
            T v2[2] = {D::zero(), D::zero()};
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                if ((flags >> i) & 1u) {
                    const uint32_t l = 32u * (warp + i * nw) + lane, g = r0 + l;
                    const bool dyn = (flags >> (8 + i)) & 1u;
                    const f3 bi = ld3(c.b, n, g);
                    const f3 x0 = ldp(P, below + l), pi = kLean ? ld3(c.pinv, n, g) : pv[kLean ? 0 : i];
                    if constexpr (kLean) st3(c.dv, n, g, x0);
                    else x[i] = x0;
                    r[i] = dyn ? bi - s[i] : zero3();
                    const f3 zi = dyn ? mk(r[i].x * pi.x, r[i].y * pi.y, r[i].z * pi.z) : zero3();
                    if constexpr (kLean) st3(team.zs, chunk, l, zi);
                    else z[i] = zi, team.put_z(c, g, l, chunk, zi);
                    const f3 bh = dyn ? bi : zero3();
                    const f3 w = c.cg_soft ? ld3(c.cg_diag, n, g) : pi;
                    v2[0] = D::add_term(v2[0], bh, mk(bh.x * w.x, bh.y * w.y, bh.z * w.z));
                    v2[1] = D::add_term(v2[1], r[i], zi);
                }
            }
            // a copy that never landed ends the whole team's solve as a breakdown
            if (!landed) v2[1] = D::add_term(v2[1], mk(NAN, NAN, NAN), mk(1.0f, 1.0f, 1.0f));
            __syncthreads();  // P is written again below
            if (!sum_and_halo(v2)) return false;
            b_delta = D::value(v2[0]), delta = D::value(v2[1]);
            if (DOT != 2) {
                b_delta = (double)(float)b_delta;
                delta = (double)(float)delta;
            }
            delta0 = delta;
            if (!isfinite(delta) || !isfinite(b_delta)) status = kStatusNumerical;
            stop = StopBound(sc, b_delta, DOT);
            if (status != 0u || max_iter == 0u || stop.met(delta)) break;
            continue;
        }
        // alpha = delta / p.s (cloth_force_solver.cpp:115-117)
        T v1[1] = {D::zero()};
#pragma unroll
        for (int i = 0; i < RPT; ++i)
            if ((flags >> i) & 1u)
                v1[0] = D::add_term(v1[0], kLean ? ldp(P, below + 32u * (warp + i * nw) + lane) : p[kLean ? 0 : i], s[i]);
        if constexpr (S::kGrid) {
            team.template publish<D, 1>(v1);
            if (!team.template collect<D, 1>(v1)) return false;
        } else {
            team.template sum<D, 1>(v1);
        }
        const double pAp = D::value(v1[0]);
        const float alpha = DOT == 2 ? (float)(delta / pAp) : (float)delta / (float)pAp;
        // the update (cloth_force_solver.cpp:119-128)
        T u1[1] = {D::zero()};
#pragma unroll
        for (int i = 0; i < RPT; ++i)
            if ((flags >> i) & 1u) {
                const uint32_t l = 32u * (warp + i * nw) + lane;
                const f3 pi = kLean ? ld3(c.pinv, n, r0 + l) : pv[kLean ? 0 : i];
                if constexpr (kLean) st3(c.dv, n, r0 + l, ld3(c.dv, n, r0 + l) + alpha * ldp(P, below + l));
                else x[i] = x[i] + alpha * p[i];
                r[i] = r[i] - alpha * s[i];
                const f3 h = mk(r[i].x * pi.x, r[i].y * pi.y, r[i].z * pi.z);
                const f3 zi = (flags >> (8 + i)) & 1u ? h : zero3();
                if constexpr (kLean) st3(team.zs, chunk, l, zi);
                else z[i] = zi, team.put_z(c, r0 + l, l, chunk, zi);
                u1[0] = D::add_term(u1[0], r[i], h);
            }
        if (!sum_and_halo(u1)) return false;
        double dn = D::value(u1[0]);
        if (DOT == 2) {
            beta = (float)(dn / delta);
        } else {
            dn = (double)(float)dn;
            beta = (float)dn / (float)delta;
        }
        delta = dn;
        ++it;
        if (!isfinite(dn) || !isfinite(alpha) || !isfinite(beta)) status = kStatusNumerical;
        if (status != 0u || it >= max_iter || stop.met(dn)) break;
    }
    if constexpr (!kLean) {
#pragma unroll
        for (int i = 0; i < RPT; ++i)
            if ((flags >> i) & 1u) st3(c.dv, n, r0 + 32u * (warp + i * nw) + lane, x[i]);
    }
    if (team.rank == 0 && tid == 0) {
        StepScalars* w = c.sc;
        w->b_delta = b_delta;
        w->delta0 = delta0;
        w->delta = delta;
        w->iter = it;
        w->status = status;
        w->cont = 0;
    }
    return true;
}

__device__ __forceinline__ void res_init_copy_barrier(ResShared* sh)
{
    if (threadIdx.x == 0) {
        sh->lost = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh->mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

}  // namespace
}  // namespace b3g
