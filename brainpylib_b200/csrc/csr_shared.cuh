// CSR products on whole matrices with the dense vector (or the sums) in shared memory, for matrices whose number of
// stored entries the caller knows and whose vector fits: what they have in common.  (The products are compiled apart, each as many
// kernels as there are lanes of a row, sizes of a block and types: csr_shared_gather.cu, csr_shared_scatter.cu,
// csr_shared_events_float.cu and _double.cu.  As one source they took 113 s of a build.)
//
// What bounds the plain kernels (csr_kernels.cu): a gather of x through L1 takes one clock per entry and SM whatever it
// hits (1e7 entries: 35 us, three times their memory time), a scattered reduction into L2 1.8 clocks (more on few
// columns: 1.9e7 entries into 2185 sums took 853 us, here 52).  A lookup in shared memory takes a tenth of a clock, an
// addition there 0.3.  So one block per SM holds the whole vector.
//
// Longer vectors are gathered through L1 (bands_kernel, csr_shared_gather.cu) or scattered into L2 (csr_kernels.cu).  What
// shared memory takes from the 256 KB of an SM is missing for the entries in flight, which pass through L1: 1e7 float entries, 80 MB,
// rows of 100, take 18.5 us with up to 131 KB of x, 19.3 with 132 (24 warps), 19.8 with 160 KB, 30 with 195 KB; rows of 1000 17.8 with
// 160 KB, 21.9 with 195 KB, 31.4 with 226 KB.  For that reason neither the first 160 KB of a longer vector here and the rest
// by the plain ways (100,000 columns: gather 44 us against 39, scatter 78 against 65), nor slices of it in several blocks
// that read the same rows side by side (58 us) paid; and reading a neighbour's slice out of its shared memory moves 0.33
// random words per clock and SM.
#ifndef BPL_CSRC_CSR_SHARED_CUH_
#define BPL_CSRC_CSR_SHARED_CUH_

#include <algorithm>
#include <type_traits>

#include "abi.h"
#include "common.cuh"
#include "csr_shared.h"
#include "row_scatter.cuh"

namespace bpl {
namespace {

// Warps of a block, one block per SM: as many as there may be beside a vector of up to 131 KB; with more of shared memory taken,
// the entries that so many have in flight no longer fit what is left of L1.  (24 and 32 warps: 1.57e7 double entries and
// events, 1 KB, 55.8 and 49.3 us; 1.2e7 floats, 80 KB of x, 23.7 and 22.1, transposed 36.4 and 34.9; 4.8e6 floats, 180 KB, 15.0
// and 16.4.)
constexpr uint32_t FEW_WARPS = 24, MANY_WARPS = 32, MANY_SMEM = 131u * 1024u;
constexpr uint32_t SHARED_SMEM = 226u * 1024u;       // the longest vector

// The rows of one block, in one walk that all three products share.
//
// A warp takes 32 / lpr rows at a time, lpr lanes each: a lane takes 4 consecutive entries per 128-bit load and U such
// loads per step.  Row groups are dealt out to the blocks in turn: neither a run of empty rows nor a run of long ones falls
// to one SM.  Two things held the first form at half the memory rate: a branch per entry (30 instructions each; the entries
// of a quad go through predicates now, and whether any lane's quad crosses the ends of its row is asked once per quad and
// warp), and a warp that waited for a step's entries before it asked for the next.  The entries of the next step, of this
// row or the next, are therefore requested before a step is worked on.
//
// The lanes of a row are chosen for the mean length.  A row that would keep them for 64 entries each, for more than twice a
// warp's share of all entries (per lane), and that is twice as long as the mean row, is cut there (`long_from`).  Behind its
// walk a warp takes its cut rows with all its lanes; those of more than BLOCK_ROW entries (LONG_ROWS of them at most) are left to
// all warps of the block.  (Lengths with a heavy tail: 100,000 rows of 20 on average, the longest 30,000, y = A^T x: 858 us by
// the lanes of each row.  A test of every row's length inside the walk, with a branch to a list, cost the event gather 1 to 5 us
// of 21.  Where there are fewer rows than the warps can hold, every row exceeds its warp's share, and sums of cut rows are taken
// again from the start: without the line at the mean, 2000 rows of 3000 entries took 19.8 us instead of 13.7, 4800 ragged rows of
// 2000 27.3 instead of 19.0.)
constexpr uint32_t LONG_ROWS = 128, BLOCK_ROW = 4096;

// Mean rows up to which 4, 8 and 16 lanes take a row.  More lanes mean fewer steps for a row, but each warp has fewer rows for
// what a row costs besides its entries: its pointers, the sum over the lanes, lanes that have nothing left.  8e6 ragged entries, float,
// by 4, 8, 16 and 32 lanes, us: events, rows of 40 (one weight) 18.5, 22.5, 28.8, 50.6; of 64 20.1, 18.5, 21.3, 26.1; of 150 18.6, 16.4,
// 17.6, 18.3; of 300 17.9, 17.3, 15.9, 17.7; products, rows of 64 20.0, 17.2, 20.5, 25.1; of 100 20.0, 17.4, 16.5, 19.0; of 300 17.0, 16.3,
// 15.9, 15.9; of 900 32.4, 26.5, 15.6, 14.0.  4e6 double: products, rows of 100 20.9, 17.9, 16.0, 16.5; transposed, rows of 64 31.7, 32.0,
// 30.8, 32.3, of 100 36.0, 31.7, 30.2, 28.7.  Transposed floats, 1.2e7 entries, by 16 and 32 lanes: rows of 300, 1700 columns 39.0, 36.9,
// 12,000 columns 34.9 both, 40,000 37.1, 38.9; of 396 40.8, 36.9; 34.9, 32.8; 37.1, 36.7.  (The lanes that finish a mean row in one step, which is what all of them had: events, rows
// of 150 by 32 lanes 20.6.)  The lanes are constants of the kernels: as numbers they cost 3 to 10 % (rows of 300, 16 lanes, 16.9 us
// and 15.9).  Products with outer values store what they read, and keep the lanes of one step.
// Where few rows leave most warps with one group, or with none, the longest chain counts: a warp's groups, times the steps of `step`
// entries per lane and one for the row.  (Products, 12,000 rows of 300, 12,000 columns: by 16 lanes 11.5 us, by 8, one group each,
// 10.2; 6000 rows of 433 transposed, 1700 columns: by 32 lanes 16.4, by 16 14.4.  With up to two groups per warp, rows of 900, the
// uneven lengths count for more: by 16 lanes 15.6, by 32 14.0.)
struct LaneRule { uint32_t four, eight, sixteen, step; };
template<typename T> constexpr LaneRule PRODUCT_LANES = sizeof(T) == 8 ? LaneRule{32, 80, 200, 4} : LaneRule{48, 80, 400, 8};
template<typename T> constexpr LaneRule SCATTER_LANES = sizeof(T) == 8 ? LaneRule{16, 40, 80, 4} : LaneRule{48, 80, 340, 8};
template<typename T> constexpr LaneRule EVENT_LANES = sizeof(T) == 8 ? LaneRule{80, 120, 400, 16} : LaneRule{48, 192, 400, 8};
template<int U> constexpr LaneRule STEP_LANES{16u * U, 32u * U, 64u * U, 4u * U};
inline uint32_t lanes_per_row(const uint32_t nse, const uint32_t n_row, const uint32_t warps, const LaneRule &rule) {
    const uint32_t mean = nse / n_row;
    const uint32_t lanes = mean <= rule.four ? 4u : mean <= rule.eight ? 8u : mean <= rule.sixteen ? 16u : 32u;
    if (static_cast<uint64_t>(n_row) * lanes >= 48u * warps) return lanes;
    auto chain = [&](const uint64_t l) { return (n_row * l + 32u * warps - 1u) / (32u * warps) * ((mean + l * rule.step - 1u) / (l * rule.step) + 1u); };
    uint32_t best = 32u;
    for (uint32_t l = 16u; l >= 4u; l /= 2u)
        if (chain(l) < chain(best)) best = l;
    return best;
}
template<uint32_t W, uint32_t LANES>
struct Deal {
    static constexpr uint32_t lpr = LANES, rows_per_warp = 32u / LANES;
    __device__ __forceinline__ uint32_t row(const uint32_t local_group, const uint32_t sub) const {
        return (local_group * gridDim.x + blockIdx.x) * rows_per_warp + sub;
    }
    // the i-th row that a warp walks (in an order of its groups)
    __device__ __forceinline__ uint32_t row_of_warp(const uint32_t warp, const uint32_t i) const {
        return row(warp + i / rows_per_warp * W, i % rows_per_warp);
    }
};

// Where a position lies from the first entry of a quad.  Positions have 32 bits; the host sends no matrix of 2^31 entries or
// more here, so that a row's ends lie less than that from any of its quads.
__host__ __device__ constexpr int from_quad(const uint32_t position, const uint32_t base) { return static_cast<int>(position - base); }
static_assert(from_quad(0x80000001u, 0x7ffffffcu) == 5 && from_quad(0x7ffffffdu, 0x80000000u) == -3, "");
constexpr uint32_t MOST_ENTRIES = 0x7fffffffu;

// Rows have 32 bits as well, and a walk asks for up to 256 rows per warp behind the last one: with at most so many rows, and 65536
// blocks, their numbers stay below 2^32, where one would wrap and the walk begin again.
constexpr uint32_t MOST_ROWS = 0x7fffffffu;
static_assert(MOST_ROWS + 256ull * MANY_WARPS * 65536u < 1ull << 32, "the rows that a walk asks for");

// `visit` has
//   fetch(row)                            what is needed of a row besides its entries (requested one row ahead)
//   quad<FULL>(base, c[4], w[4], lo, hi)  entries base .. base + 3, of which lo <= e < hi belong to the row (FULL: all)
//   entry(pos, c, w)                      one entry (the ragged end of the arrays)
//   begin(fetched)                        before a row
//   SUMS, Sum, total(lanes), put(row, s)  behind a row, where it has a result: the sum over aligned groups of lanes, and where
//                                         one lane leaves it
// (Behind the vector in dynamic shared memory: with static shared memory in the kernel the vector no longer lies at the address
// 0, and every look-up adds its base: 2 us of the event gather's 20.)
template<typename Sum, uint32_t W>
struct CutRows {
    uint32_t n, row[LONG_ROWS];
    bool block[W];          // a warp has rows of more than BLOCK_ROW
    Sum part[2][W];
};

inline __host__ __device__ uint32_t behind_vector(const size_t bytes) { return static_cast<uint32_t>((bytes + 15u) & ~static_cast<size_t>(15u)); }
template<typename Sum, uint32_t W>
__device__ __forceinline__ CutRows<Sum, W> &cut_rows_at(unsigned char *shared, const size_t bytes) {
    return *reinterpret_cast<CutRows<Sum, W> *>(shared + behind_vector(bytes));
}
template<typename Sum, uint32_t W>
uint32_t shared_bytes(const size_t vector_bytes) { return behind_vector(vector_bytes) + sizeof(CutRows<Sum, W>); }
constexpr uint32_t ALL_SMEM = 227u * 1024u;
static_assert(SHARED_SMEM + sizeof(CutRows<double, FEW_WARPS>) <= ALL_SMEM, "the longest vector and the list");

// The rows that the walk has cut; `mine`: this warp has some, `block`: some warps of the block have rows for all of it.
template<typename T, bool WEIGHTS, uint32_t W, uint32_t LANES, typename Visit>
__device__ __noinline__ void walk_cut_rows(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr,
                                           const T *__restrict__ data, const uint32_t n_row, const uint32_t nse,
                                           const uint32_t long_from, const Deal<W, LANES> deal, Visit visit, const bool mine, const bool block,
                                           CutRows<typename Visit::Sum, W> &cut_rows) {
    const uint32_t lane = threadIdx.x & 31, g_full = nse >> 2;
    auto span = [&](const uint32_t r, const uint32_t start, const uint32_t end, const uint32_t first, const uint32_t lanes) {
        constexpr int AHEAD = sizeof(T) == 8 ? 2 : 4;
        visit.begin(visit.fetch(r));
        const uint32_t g_stop = min((end + 3u) >> 2, g_full);
        for (uint32_t g0 = (start >> 2) + first; g0 < g_stop; g0 += AHEAD * lanes) {
            uint4 ix[AHEAD];
            Quad<T> w[WEIGHTS ? AHEAD : 1];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const uint32_t g = g0 + u * lanes;
                if (g >= g_stop) continue;
                ix[u] = ldg_stream_u4(indices + 4ull * g);
                if (WEIGHTS) load_quad(data + 4ull * g, w[u]);
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const uint32_t g = g0 + u * lanes, c[4] = {ix[u].x, ix[u].y, ix[u].z, ix[u].w};
                if (g < g_stop) visit.template quad<false>(4u * g, c, w[WEIGHTS ? u : 0].v, from_quad(start, 4u * g), from_quad(end, 4u * g));
            }
        }
        if (first == 0)
            for (uint32_t pos = max(4u * g_full, start); pos < end; ++pos) visit.entry(pos, indices[pos], WEIGHTS ? data[pos] : T(0));
    };
    const uint32_t warp = threadIdx.x >> 5, skip = Visit::SUMS ? 0u : long_from;     // (a sum is taken again as a whole)
    __syncwarp();                                          // (its results are replaced by other lanes)
    for (uint32_t i = 0; mine && deal.row_of_warp(warp, i) < n_row; i += 32u) {     // the warp's rows again, one per lane
        const uint32_t r = deal.row_of_warp(warp, i + lane);
        const uint32_t start = r < n_row ? indptr[r] : 0u, end = r < n_row ? indptr[r + 1] : 0u;
        for (uint32_t some = __ballot_sync(FULL_MASK, end - start > long_from); some; some &= some - 1u) {
            const int l = __ffs(some) - 1;
            const uint32_t r0 = __shfl_sync(FULL_MASK, r, l), s0 = __shfl_sync(FULL_MASK, start, l), e0 = __shfl_sync(FULL_MASK, end, l);
            uint32_t at = LONG_ROWS;
            if (e0 - s0 > BLOCK_ROW) {
                if (lane == 0) at = atomicAdd(&cut_rows.n, 1u);
                at = __shfl_sync(FULL_MASK, at, 0);
            }
            if (at < LONG_ROWS) {
                if (lane == 0) cut_rows.row[at] = r0;
                continue;
            }
            span(r0, s0 + skip, e0, lane, 32u);
            if (Visit::SUMS) {
                const typename Visit::Sum s = visit.total(32);
                if (lane == 0) visit.put(r0, s);
            }
        }
    }
    if (!block) return;
    __syncthreads();
    const uint32_t n = min(cut_rows.n, LONG_ROWS);
    uint32_t turn = 0;
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t r = cut_rows.row[i];
        span(r, indptr[r] + skip, indptr[r + 1], threadIdx.x, W * 32u);
        if (!Visit::SUMS) continue;
        // one barrier per row: the sums of the next go to the other half, and who reads these is through at the barrier after
        const typename Visit::Sum s = visit.total(32);
        if (lane == 0) cut_rows.part[turn & 1u][warp] = s;
        __syncthreads();
        if (warp == turn % W) {
            const typename Visit::Sum t = group_sum(lane < W ? cut_rows.part[turn & 1u][lane] : typename Visit::Sum(0), 32);
            if (lane == 0) visit.put(r, t);
        }
        ++turn;
    }
}

// `ready` runs before the first entry is visited, behind the first loads: it fills shared memory and ends with a barrier.
template<typename T, bool WEIGHTS, int U, uint32_t W, uint32_t LANES, typename Visit, typename Ready>
__device__ __forceinline__ void walk_rows(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr,
                                          const T *__restrict__ data, const uint32_t n_row, const uint32_t nse,
                                          const uint32_t long_from, const Deal<W, LANES> deal, Visit &visit,
                                          CutRows<typename Visit::Sum, W> &cut_rows, Ready ready) {
    const uint32_t lane = threadIdx.x & 31;
    constexpr uint32_t lpr = LANES;
    const uint32_t sub = lane / lpr, sl = lane % lpr;
    const uint32_t g_full = nse >> 2;
    using Fetched = decltype(visit.fetch(0u));
    struct Step {
        uint4 ix[U];
        Quad<T> w[WEIGHTS ? U : 1];
        uint32_t g0;                                       // the lane's first quad
    };
    struct Row {
        uint32_t start, end;
        Fetched fetched;
    };
    auto pointers = [&](const uint32_t group) {
        const uint32_t row = deal.row(group, sub);
        Row r{0u, 0u, visit.fetch(row)};
        if (row < n_row) { r.start = indptr[row]; r.end = indptr[row + 1]; }
        return r;
    };
    auto load = [&](Step &s, const Row &r) {
        const uint32_t g_stop = min((r.end + 3u) >> 2, g_full);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t g = s.g0 + u * lpr;
            if (g < g_stop) {
                s.ix[u] = ldg_stream_u4(indices + 4ull * g);
                if (WEIGHTS) load_quad(data + 4ull * g, s.w[u]);
            }
        }
    };
    auto cut = [&](Row &r) { r.end = min(r.end, r.start + long_from); };     // (where the pointers are needed, not where they are asked for)
    uint32_t group = threadIdx.x >> 5;
    Row row = pointers(group), next = pointers(group + W);
    cut(row);
    cut(next);
    if (threadIdx.x == 0) cut_rows.n = 0;
    // one step: request what comes after it (`after`), then work on it
    auto step = [&](Step &now, Step &after) {
        const uint32_t g_stop = min((row.end + 3u) >> 2, g_full);
        const bool more = __any_sync(FULL_MASK, now.g0 + U * lpr < g_stop);
        after.g0 = more ? now.g0 + U * lpr : (next.start >> 2) + sl;
        load(after, more ? row : next);
        Row later{0u, 0u, Fetched()};
        if (!more) later = pointers(group + 2 * W);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t base = 4u * (now.g0 + u * lpr);
            const bool here = now.g0 + u * lpr < g_stop;
            if (!__any_sync(FULL_MASK, here)) continue;
            const uint32_t c[4] = {now.ix[u].x, now.ix[u].y, now.ix[u].z, now.ix[u].w};
            const T *v = now.w[WEIGHTS ? u : 0].v;
            const int lo = from_quad(row.start, base), hi = from_quad(row.end, base);
            if (__all_sync(FULL_MASK, here && lo <= 0 && hi >= 4)) visit.template quad<true>(base, c, v, lo, hi);
            else visit.template quad<false>(base, c, v, lo, here ? hi : 0);
        }
        if (more) return;
        if (sl == 0)
            for (uint32_t pos = max(4u * g_full, row.start); pos < row.end; ++pos)
                visit.entry(pos, indices[pos], WEIGHTS ? data[pos] : T(0));
        if (Visit::SUMS) {
            const typename Visit::Sum s = visit.total(static_cast<int>(lpr));
            if (sl == 0 && deal.row(group, sub) < n_row) visit.put(deal.row(group, sub), s);
        }
        group += W;
        row = next;
        next = later;
        cut(next);
        visit.begin(row.fetched);
    };
    Step a, b;
#pragma unroll
    for (int u = 0; u < U; ++u) a.ix[u] = b.ix[u] = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < (WEIGHTS ? U : 1); ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) a.w[u].v[e] = b.w[u].v[e] = T(0);
    a.g0 = (row.start >> 2) + sl;
    load(a, row);
    // Has the warp rows that it will cut?  Asked here, where the answer comes with what the warp waits for anyway: behind the
    // walk it took 2 us of the event gather's 21.
    const uint32_t warp = threadIdx.x >> 5;
    bool some_cut = false, for_block = false;
    for (uint32_t i = 0; deal.row_of_warp(warp, i) < n_row; i += 128u) {
        uint32_t length[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t r = deal.row_of_warp(warp, i + 32u * k + lane);
            length[k] = r < n_row ? indptr[r + 1] - indptr[r] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            some_cut |= length[k] > long_from;
            for_block |= length[k] > max(long_from, BLOCK_ROW);
        }
    }
    some_cut = __any_sync(FULL_MASK, some_cut);
    for_block = __any_sync(FULL_MASK, for_block);
    if (lane == 0) cut_rows.block[warp] = for_block;
    ready();
    visit.begin(row.fetched);
    while (deal.row(group, 0) < n_row) {
        step(a, b);
        if (deal.row(group, 0) >= n_row) break;
        step(b, a);
    }
    for_block = __any_sync(FULL_MASK, lane < W && cut_rows.block[lane]);
    if (some_cut || for_block)
        walk_cut_rows<T, WEIGHTS>(indices, indptr, data, n_row, nse, long_from, deal, visit, some_cut, for_block, cut_rows);
}

// The first `count` elements of x into shared memory, by the whole block.
template<typename T>
__device__ __forceinline__ void fill_shared(T *shared, const T *__restrict__ p, const uint32_t count) {
    constexpr uint32_t PER = 16 / sizeof(T);
    const uint32_t n_vec = aligned16_device(p) ? count / PER : 0u;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n_vec; i += blockDim.x)
        reinterpret_cast<uint4 *>(shared)[i] = __ldg(reinterpret_cast<const uint4 *>(p) + i);
    for (uint32_t i = n_vec * PER + threadIdx.x; i < count; i += blockDim.x) shared[i] = __ldg(p + i);
}

// The same for words that the launch in front has written.
__device__ __forceinline__ void fill_words(uint32_t *shared, const uint32_t *p, const uint32_t count) {
    const uint32_t n_vec = aligned16_device(p) ? count / 4u : 0u;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n_vec; i += blockDim.x)
        reinterpret_cast<uint4 *>(shared)[i] = __ldcg(reinterpret_cast<const uint4 *>(p) + i);
    for (uint32_t i = n_vec * 4u + threadIdx.x; i < count; i += blockDim.x) shared[i] = __ldcg(p + i);
}

// ---- host side: the rules, in clocks of one SM (1.9 GHz) ----
template<typename T>
struct Plan {
    double per;                 // stored entries per SM
    double entry;               // clocks to stream an entry, by what is left for entries in flight (see above)
    double fill;                // clocks to start and to fill or clear the vector, 56 bytes per clock

    Plan(const CsrMatrix<T> &m, const bool values) {
        const double kb = static_cast<double>(m.n_col) * sizeof(T) / 1024.0;
        per = static_cast<double>(m.nse) / sm_count();
        entry = (4.0 + (values ? sizeof(T) : 0)) / (kb <= 131 ? 15.0 : kb <= 163 ? 14.0 : kb <= 195 ? 11.7 : 9.0);
        fill = 3000 + kb * 1024 / 56;
    }
};

template<typename T>
bool usable(const CsrMatrix<T> &m, const bool weights) {
    return m.n_row != 0 && m.n_row <= MOST_ROWS && m.n_col != 0 && m.nse != 0 && m.nse <= MOST_ENTRIES && m.n_col <= SHARED_SMEM / sizeof(T) && aligned16(m.indices) &&
           (!weights || aligned16(m.data));
}

// columns from which the bands are faster than x in shared memory (200 KB of floats; of doubles, 164 KB)
template<typename T> constexpr uint32_t BANDS_FROM = sizeof(T) == 4 ? 51200u : 21000u;

// Where a row is cut: see LONG_ROWS.  No farther than any row reaches, so that a row's start and this stay below 2^32.
constexpr uint32_t cut_from(const uint32_t nse, const uint32_t n_row, const uint32_t warps, const uint32_t lanes) {
    return std::min(std::max(std::max(64u, nse / warps / 16u) * lanes, 2u * (nse / n_row)), MOST_ENTRIES);
}
static_assert(MOST_ENTRIES + static_cast<uint64_t>(cut_from(MOST_ENTRIES, 1u, FEW_WARPS, 32u)) < 1ull << 32, "where the longest row is cut");

// go(warps of a block, lanes of a row, where rows are cut): the first two are constants
template<uint32_t W, typename Go>
void with_lanes(const uint32_t nse, const uint32_t n_row, const LaneRule &rule, Go go) {
    const uint32_t warps = static_cast<uint32_t>(sm_count()) * W, lanes = lanes_per_row(nse, n_row, warps, rule);
    const uint32_t long_from = cut_from(nse, n_row, warps, lanes);
    constexpr std::integral_constant<uint32_t, W> w;
    if (lanes == 4u) go(w, std::integral_constant<uint32_t, 4>(), long_from);
    else if (lanes == 8u) go(w, std::integral_constant<uint32_t, 8>(), long_from);
    else if (lanes == 16u) go(w, std::integral_constant<uint32_t, 16>(), long_from);
    else go(w, std::integral_constant<uint32_t, 32>(), long_from);
}
template<typename T, typename Go>
void with_block(const CsrMatrix<T> &m, const size_t vector_bytes, const LaneRule &rule, Go go) {
    if (vector_bytes <= MANY_SMEM) with_lanes<MANY_WARPS>(m.nse, m.n_row, rule, go);
    else with_lanes<FEW_WARPS>(m.nse, m.n_row, rule, go);
}

}  // namespace
}  // namespace bpl

#endif  // BPL_CSRC_CSR_SHARED_CUH_
