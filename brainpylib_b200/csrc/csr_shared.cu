// CSR products on whole matrices with the dense vector (or the sums) in shared memory, for matrices whose number of
// stored entries the caller knows and whose vector fits.
//
// What bounds the plain kernels (csr_kernels.cu): a gather of x through L1 takes one clock per entry and SM whatever it
// hits (1e7 entries: 35 us, three times their memory time), a scattered reduction into L2 1.8 clocks (more on few
// columns: 1.9e7 entries into 2185 sums took 853 us, here 46).  A lookup in shared memory takes a tenth of a clock, an
// addition there 0.3.  So one block per SM holds the whole vector.
//
// Longer vectors are gathered through L1 (bands_kernel) or scattered into L2 (csr_kernels.cu).  What shared memory takes from
// the 256 KB of an SM is missing for the entries in flight, which pass through L1: 1e7 float entries, 80 MB, take 18.6 us with up to 132 KB of x, 19.9 with
// 160 KB, 23 with 195 KB, 31 with 226 KB.  For that reason neither the first 160 KB of a longer vector here and the rest
// by the plain ways (100,000 columns: gather 44 us against 39, scatter 78 against 65), nor slices of it in several blocks
// that read the same rows side by side (58 us) paid; and reading a neighbour's slice out of its shared memory moves 0.33
// random words per clock and SM.
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
// 30.8, 32.3, of 100 36.0, 31.7, 30.2, 28.7.  (The lanes that finish a mean row in one step, which is what all of them had: events, rows
// of 150 by 32 lanes 20.6.)  The lanes are constants of the kernels: as numbers they cost 3 to 10 % (rows of 300, 16 lanes, 16.9 us
// and 15.9).  Products with outer values store what they read, and keep the lanes of one step.
// Where few rows leave most warps with one group, or with none, the longest chain counts: a warp's groups, times the steps of `step`
// entries per lane and one for the row.  (Products, 12,000 rows of 300, 12,000 columns: by 16 lanes 11.5 us, by 8, one group each,
// 10.2; 6000 rows of 433 transposed, 1700 columns: by 32 lanes 16.4, by 16 14.4.  With up to two groups per warp, rows of 900, the
// uneven lengths count for more: by 16 lanes 15.6, by 32 14.0.)
struct LaneRule { uint32_t four, eight, sixteen, step; };
template<typename T> constexpr LaneRule PRODUCT_LANES = sizeof(T) == 8 ? LaneRule{32, 80, 200, 4} : LaneRule{48, 80, 400, 8};
template<typename T> constexpr LaneRule SCATTER_LANES = sizeof(T) == 8 ? LaneRule{16, 40, 80, 4} : LaneRule{48, 80, 400, 8};
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

// y = A x
template<typename T, bool HOMO>
struct GatherVisit {
    const T *xs;
    T homo_w, *y;
    T acc;
    __device__ __forceinline__ int fetch(uint32_t) const { return 0; }
    __device__ __forceinline__ void begin(int) { acc = T(0); }
    template<bool FULL>
    __device__ __forceinline__ void quad(uint32_t, const uint32_t (&c)[4], const T *w, const int lo, const int hi) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (FULL || (e >= lo && e < hi)) acc += (HOMO ? homo_w : w[e]) * xs[c[e]];
    }
    __device__ __forceinline__ void entry(uint32_t, const uint32_t c, const T w) { acc += (HOMO ? homo_w : w) * xs[c]; }
    static constexpr bool SUMS = true;
    using Sum = T;
    __device__ __forceinline__ Sum total(const int lanes) const { return group_sum(acc, lanes); }
    __device__ __forceinline__ void put(const uint32_t row, const Sum s) const { y[row] = s; }
};

template<typename T, bool HOMO, int U, uint32_t W, uint32_t LANES>
__global__ void __launch_bounds__(W * 32, 1)
gather_shared_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr, const T *__restrict__ data,
                     const T *__restrict__ x, T *__restrict__ y, const uint32_t n_row, const uint32_t nse, const uint32_t n_col,
                     const uint32_t long_from) {
    extern __shared__ __align__(16) unsigned char shared_vector[];
    T *xs = reinterpret_cast<T *>(shared_vector);
    constexpr Deal<W, LANES> deal;
    auto &cut_rows = cut_rows_at<T, W>(shared_vector, n_col * sizeof(T));
    GatherVisit<T, HOMO> visit{xs, HOMO ? data[0] : T(0), y, T(0)};
    walk_rows<T, !HOMO, U>(indices, indptr, data, n_row, nse, long_from, deal, visit, cut_rows, [&]() {
        fill_shared(xs, x, n_col);
        __syncthreads();
    });
}

// y = A events: the events as one byte each in shared memory, or one bit where they are many.  The walk is bound by
// instruction issue, and a byte needs no shifts (1e8 entries, rows of 121, 3000 columns: 140 -> 109 us).  Homogeneous weights
// count hits and scale once (equal to the reference CPU kernel's float64 accumulation, brainpylib/_src/event_ops/event_csr_matvec.py:334-357).
template<typename T, bool HOMO, bool BYTES>
struct EventVisit {
    const uint32_t *mask;
    T homo_w, *y;
    T acc;
    uint32_t hits;
    __device__ __forceinline__ int fetch(uint32_t) const { return 0; }
    __device__ __forceinline__ void begin(int) {
        acc = T(0);
        hits = 0;
    }
    __device__ __forceinline__ uint32_t hit(const uint32_t c) const {
        return BYTES ? reinterpret_cast<const uint8_t *>(mask)[c] : (mask[c >> 5] >> (c & 31u)) & 1u;
    }
    template<bool FULL>
    __device__ __forceinline__ void quad(uint32_t, const uint32_t (&c)[4], const T *w, const int lo, const int hi) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (!FULL && !(e >= lo && e < hi)) continue;
            const uint32_t h = hit(c[e]);
            if (HOMO) hits += h;
            else if (h) acc += w[e];
        }
    }
    __device__ __forceinline__ void entry(uint32_t, const uint32_t c, const T w) {
        const uint32_t h = hit(c);
        if (HOMO) hits += h;
        else if (h) acc += w;
    }
    static constexpr bool SUMS = true;
    using Sum = std::conditional_t<HOMO, uint32_t, T>;
    __device__ __forceinline__ Sum total(const int lanes) const {
        if constexpr (HOMO) return group_sum(hits, lanes);
        else return group_sum(acc, lanes);
    }
    __device__ __forceinline__ void put(const uint32_t row, const Sum s) const {
        // no hit leaves +0 like an empty sum (the product with a negative weight would give -0)
        if constexpr (HOMO) y[row] = s ? static_cast<T>(static_cast<double>(s) * static_cast<double>(homo_w)) : T(0);
        else y[row] = s;
    }
};

// One byte per event, 0 or 1, 16 bytes of events per load where they are aligned, and their bytes in one store (single bytes
// meet in the banks).
template<typename E>
__device__ __forceinline__ void fill_bytes(uint8_t *bytes, const E *__restrict__ events, const uint32_t n) {
    constexpr uint32_t PER = 16 / sizeof(E);
    const uint32_t whole = aligned16_device(events) ? n / PER : 0u;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < whole; i += blockDim.x) {
        const uint4 raw = *reinterpret_cast<const uint4 *>(events + i * PER);
        const E *e = reinterpret_cast<const E *>(&raw);
        uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (uint32_t k = 0; k < PER; ++k) w[k / 4] |= (is_event(e[k]) ? 1u : 0u) << (8u * (k % 4));
        if (PER == 16) reinterpret_cast<uint4 *>(bytes)[i] = make_uint4(w[0], w[1], w[2], w[3]);
        else if (PER == 4) reinterpret_cast<uint32_t *>(bytes)[i] = w[0];
        else reinterpret_cast<uint16_t *>(bytes)[i] = static_cast<uint16_t>(w[0]);
    }
    for (uint32_t i = whole * PER + threadIdx.x; i < n; i += blockDim.x) bytes[i] = is_event(events[i]) ? 1 : 0;
}

template<typename T, typename E, bool HOMO, bool BYTES, int U, uint32_t W, uint32_t LANES>
__global__ void __launch_bounds__(W * 32, 1)
gather_events_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr, const T *__restrict__ data,
                     const E *__restrict__ events, const uint32_t *packed, T *__restrict__ y, const uint32_t n_row,
                     const uint32_t nse, const uint32_t n_col, const uint32_t long_from) {
    extern __shared__ __align__(16) unsigned char shared_vector[];
    uint32_t *mask = reinterpret_cast<uint32_t *>(shared_vector);
    constexpr Deal<W, LANES> deal;
    using Sum = typename EventVisit<T, HOMO, BYTES>::Sum;
    auto &cut_rows = cut_rows_at<Sum, W>(shared_vector, BYTES ? n_col : (n_col + 31u) / 32u * 4u);
    EventVisit<T, HOMO, BYTES> visit{mask, HOMO ? data[0] : T(0), y, T(0), 0u};
    walk_rows<T, !HOMO, U>(indices, indptr, data, n_row, nse, long_from, deal, visit, cut_rows, [&]() {
        if (BYTES) {
            fill_bytes(shared_vector, events, n_col);
        } else if (packed != nullptr) {
            pdl_wait();
            fill_words(mask, packed, (n_col + 31u) / 32u);
        } else {
            pack_event_mask(events, n_col, mask);
        }
        __syncthreads();
    });
}

// The bits of the events, once for all blocks.  (Every block packing them itself reads 148 times the events: a million
// float events take 60 us, their 125 KB of bits 1.)
template<typename E>
__global__ void __launch_bounds__(256) pack_events_kernel(const E *__restrict__ events, uint32_t *__restrict__ packed, const uint32_t n) {
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t w = (static_cast<uint64_t>(blockIdx.x) * 256u + threadIdx.x) >> 5; w * 32u < n; w += static_cast<uint64_t>(gridDim.x) * 8u) {
        const uint64_t i = w * 32u + lane;
        const uint32_t bits = __ballot_sync(FULL_MASK, i < n && is_event(events[i]));
        if (lane == 0) packed[w] = bits;
    }
}

// The two gathering products for a longer vector x, read through L1.  What bounds them there is the traffic from L2, 34
// bytes per clock and SM: every miss brings a sector of 32 bytes for one value, 2.7 times the matrix itself where most
// gathers miss (1e7 float entries, 100,000 columns: 39 us).  Stored rows are nearly always sorted by column.  So few
// lanes (one, where there are rows enough) walk a row together, 8 entries each at a time, and the rows of an SM, which
// start together, sweep over x together: at any time they read in a band of x that fits L1, and each of its sectors comes
// from L2 about once: 31 us, 80 % of the gathers hit.  More lanes per row, 1000 or 2000 per SM instead of 500: 37 and 45
// us.  (Unsorted rows are summed as correctly, with the misses of the plain kernel.)
// Rows that would keep their lanes far longer than an average one are put off and taken by whole warps, those of more than
// BAND_WARP_ROW entries by the block (100,000 rows, 2e7 entries, heavy tail up to 300,000: 15.6 ms by the lanes of each row).
//   SUM: y[row] = sum of weight * x[column];  OUTER: g[entry] = row_vector[row] * x[column];  SUM + OUTER: both, for one gather.
enum { BAND_SUM = 1, BAND_OUTER = 2 };
constexpr int BAND_THREADS = 128;
constexpr uint32_t BAND_WARP_ROW = 2048;

template<typename T, bool HOMO, int MODE>
__global__ void __launch_bounds__(BAND_THREADS)
bands_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr, const T *__restrict__ data,
             const T *__restrict__ row_vector, const T *__restrict__ x, T *__restrict__ y, T *__restrict__ out, const uint32_t n_row,
             const uint32_t nse, const uint32_t log_l) {
    constexpr bool SUM = (MODE & BAND_SUM) != 0, OUTER = (MODE & BAND_OUTER) != 0, WEIGHTS = SUM && !HOMO;
    __shared__ uint32_t n_long, long_row[BAND_THREADS];
    __shared__ T warp_part[2][BAND_THREADS / 32];
    struct Unit {
        uint32_t c[8];
        T w[WEIGHTS ? 8 : 1];
    };
    const uint32_t L = 1u << log_l, part = threadIdx.x & (L - 1u), lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t full = nse >> 3;                            // units that lie wholly inside the arrays
    const uint64_t rows_per_grid = (static_cast<uint64_t>(gridDim.x) * BAND_THREADS) >> log_l;
    const uint32_t long_from = max(128u, nse >> 15) << log_l;
    uint32_t start = 0, end = 0, u_end = 0;                    // the row that is walked
    T r = T(0), acc = T(0);
    const T homo_w = SUM && HOMO ? data[0] : T(0);
    auto enter = [&](const uint32_t row) {
        start = indptr[row];
        end = indptr[row + 1];
        if (OUTER) r = row_vector[row];
    };
    auto load = [&](Unit &v, const uint32_t at) {
        if (at < u_end && at < full) {
            ldg_stream_8(indices + 8ull * at, v.c);
            if (WEIGHTS) ldg_stream_8(data + 8ull * at, v.w);
        }
    };
    auto use = [&](const Unit &v, const uint32_t at) {
        const uint32_t pos = 8u * at;
        if (at >= full) {                                      // ragged end of the arrays
            for (uint32_t e = max(pos, start); e < end; ++e) {
                const T v = __ldg(x + indices[e]);
                if (OUTER) out[e] = r * v;
                if (SUM) acc += (WEIGHTS ? data[e] : homo_w) * v;
            }
            return;
        }
        T g[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            g[e] = T(0);
            if (pos + e >= start && pos + e < end) g[e] = __ldg(x + v.c[e]);
        }
        if (OUTER) {
            if (pos >= start && pos + 8u <= end) {
                store_quad(out + pos, r * g[0], r * g[1], r * g[2], r * g[3]);
                store_quad(out + pos + 4u, r * g[4], r * g[5], r * g[6], r * g[7]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (pos + e >= start && pos + e < end) out[pos + e] = r * g[e];
            }
        }
        if (SUM) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (pos + e >= start && pos + e < end) acc += (WEIGHTS ? v.w[WEIGHTS ? e : 0] : homo_w) * g[e];
        }
    };
    // the units of the row from its `first` on, every `lanes`-th
    auto walk = [&](const uint32_t first, const uint32_t lanes) {
        uint32_t u = (start >> 3) + first;
        u_end = start < end ? (end + 7u) >> 3 : 0u;
        acc = T(0);
        Unit a, b;
        load(a, u);
        while (u < u_end) {
            load(b, u + lanes);
            use(a, u);
            if (u + lanes < u_end) {
                load(a, u + 2u * lanes);
                use(b, u + lanes);
            }
            u += 2u * lanes;
        }
    };
    if (threadIdx.x == 0) n_long = 0;
    __syncthreads();
    for (uint64_t base = static_cast<uint64_t>(blockIdx.x) * (BAND_THREADS >> log_l); base < n_row; base += rows_per_grid) {
        const uint64_t row = base + (threadIdx.x >> log_l);
        start = end = 0;
        if (row < n_row) enter(static_cast<uint32_t>(row));
        bool later = end - start > long_from;
        if (__any_sync(FULL_MASK, later)) {                    // put off, as many as there is room for
            uint32_t at = BAND_THREADS;
            if (later && part == 0) at = atomicAdd(&n_long, 1u);
            later = __shfl_sync(FULL_MASK, at, lane - part) < BAND_THREADS;
            if (later) {
                if (part == 0) long_row[at] = static_cast<uint32_t>(row);
                start = end = 0;
            }
        }
        walk(part, L);
        if (SUM) {
            for (uint32_t o = L >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL_MASK, acc, o);
            if (part == 0 && row < n_row && !later) y[row] = acc;
        }
    }
    __syncthreads();
    const uint32_t n = min(n_long, static_cast<uint32_t>(BAND_THREADS));
    for (uint32_t i = warp; i < n; i += BAND_THREADS / 32) {
        enter(long_row[i]);
        if (end - start > BAND_WARP_ROW) continue;
        walk(lane, 32u);
        if (SUM) {
            acc = warp_sum(acc);
            if (lane == 0) y[long_row[i]] = acc;
        }
    }
    uint32_t turn = 0;
    for (uint32_t i = 0; i < n; ++i) {
        enter(long_row[i]);
        if (end - start <= BAND_WARP_ROW) continue;
        walk(threadIdx.x, BAND_THREADS);
        if (!SUM) continue;
        acc = warp_sum(acc);                                   // (a barrier per row: as in walk_cut_rows)
        if (lane == 0) warp_part[turn & 1u][warp] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            T sum = T(0);
            for (uint32_t k = 0; k < BAND_THREADS / 32; ++k) sum += warp_part[turn & 1u][k];
            y[long_row[i]] = sum;
        }
        ++turn;
    }
    if (OUTER) zero_outside_rows(out, indptr, n_row, nse);
}

// y += A^T x: sums in shared memory, added to the zero-filled y at the end
template<typename T, bool HOMO>
struct ScatterVisit {
    T *sums;
    uint32_t n_row;
    const T *x;
    T homo_w, scale;
    __device__ __forceinline__ T fetch(const uint32_t row) const { return row < n_row ? x[row] : T(0); }
    __device__ __forceinline__ void begin(const T s) { scale = s; }
    template<bool FULL>
    __device__ __forceinline__ void quad(uint32_t, const uint32_t (&c)[4], const T *w, const int lo, const int hi) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (FULL || (e >= lo && e < hi)) atomicAdd(sums + c[e], (HOMO ? homo_w : w[e]) * scale);
    }
    __device__ __forceinline__ void entry(uint32_t, const uint32_t c, const T w) { atomicAdd(sums + c, (HOMO ? homo_w : w) * scale); }
    static constexpr bool SUMS = false;
    using Sum = T;
    __device__ __forceinline__ Sum total(int) const { return T(0); }
    __device__ __forceinline__ void put(uint32_t, Sum) const {}
};

template<typename T, bool HOMO, int U, uint32_t W, uint32_t LANES>
__global__ void __launch_bounds__(W * 32, 1)
scatter_shared_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr, const T *__restrict__ data,
                      const T *__restrict__ x, T *__restrict__ y, const uint32_t n_row, const uint32_t nse,
                      const uint32_t n_col, const uint32_t long_from) {
    extern __shared__ __align__(16) unsigned char shared_vector[];
    T *sums = reinterpret_cast<T *>(shared_vector);
    constexpr Deal<W, LANES> deal;
    auto &cut_rows = cut_rows_at<T, W>(shared_vector, n_col * sizeof(T));
    ScatterVisit<T, HOMO> visit{sums, n_row, x, HOMO ? data[0] : T(0), T(0)};
    walk_rows<T, !HOMO, U>(indices, indptr, data, n_row, nse, long_from, deal, visit, cut_rows, [&]() {
        for (uint32_t i = threadIdx.x; i < n_col; i += W * 32u) sums[i] = T(0);
        __syncthreads();
    });
    __syncthreads();
    pdl_wait();                                            // y is zero
    add_sums(sums, y, n_col, blockIdx.x, gridDim.x);
}

// g[e] = row_vector[row] * col_vector[column]
template<typename T>
struct OuterVisit {
    const T *xs, *row_vector;
    T *g;
    uint32_t n_row;
    T r;
    __device__ __forceinline__ T fetch(const uint32_t row) const { return row < n_row ? row_vector[row] : T(0); }
    __device__ __forceinline__ void begin(const T v) { r = v; }
    template<bool FULL>
    __device__ __forceinline__ void quad(const uint32_t base, const uint32_t (&c)[4], const T *, const int lo, const int hi) {
        if (FULL) {
            store_quad(g + base, r * xs[c[0]], r * xs[c[1]], r * xs[c[2]], r * xs[c[3]]);
        } else if (lo <= 0 && hi >= 4) {
            store_quad(g + base, r * xs[c[0]], r * xs[c[1]], r * xs[c[2]], r * xs[c[3]]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (e >= lo && e < hi) g[base + e] = r * xs[c[e]];
        }
    }
    __device__ __forceinline__ void entry(const uint32_t pos, const uint32_t c, T) { g[pos] = r * xs[c]; }
    static constexpr bool SUMS = false;
    using Sum = T;
    __device__ __forceinline__ Sum total(int) const { return T(0); }
    __device__ __forceinline__ void put(uint32_t, Sum) const {}
};

// (`zero`: n_zero elements to clear for the launch behind this one, which may then start early.  Without it the launch behind may be
// any, also a dependent one that reads g as weights through the read-only path, and starts when this one has finished.)
template<typename T, int U, uint32_t W, uint32_t LANES>
__global__ void __launch_bounds__(W * 32, 1)
outer_shared_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr,
                    const T *__restrict__ row_vector, const T *__restrict__ col_vector, T *__restrict__ g, T *__restrict__ zero,
                    const uint32_t n_zero, const uint32_t n_row, const uint32_t nse, const uint32_t n_col, const uint32_t long_from) {
    extern __shared__ __align__(16) unsigned char shared_vector[];
    if (zero != nullptr) pdl_launch_dependents();
    for (uint32_t i = blockIdx.x * (W * 32u) + threadIdx.x; i < n_zero; i += gridDim.x * (W * 32u)) zero[i] = T(0);
    T *xs = reinterpret_cast<T *>(shared_vector);
    constexpr Deal<W, LANES> deal;
    auto &cut_rows = cut_rows_at<T, W>(shared_vector, n_col * sizeof(T));
    OuterVisit<T> visit{xs, row_vector, g, n_row, T(0)};
    walk_rows<T, false, U>(indices, indptr, nullptr, n_row, nse, long_from, deal, visit, cut_rows, [&]() {
        fill_shared(xs, col_vector, n_col);
        zero_outside_rows(g, indptr, n_row, nse);
        __syncthreads();
    });
}

// Both of one gather: y[row] = sum of weight * col_vector[column] and g[e] = row_vector[row] * col_vector[column], the two
// gradients of y = A^T x.  The indices are read once, and so is the vector (a row that is cut writes its g twice, the same).
template<typename T>
struct GatherOuterVisit {
    const T *xs, *row_vector;
    T *g, *y;
    uint32_t n_row;
    T r, acc;
    __device__ __forceinline__ T fetch(const uint32_t row) const { return row < n_row ? row_vector[row] : T(0); }
    __device__ __forceinline__ void begin(const T v) {
        r = v;
        acc = T(0);
    }
    template<bool FULL>
    __device__ __forceinline__ void quad(const uint32_t base, const uint32_t (&c)[4], const T *w, const int lo, const int hi) {
        if (FULL || (lo <= 0 && hi >= 4)) {
            const T v[4] = {xs[c[0]], xs[c[1]], xs[c[2]], xs[c[3]]};
            store_quad(g + base, r * v[0], r * v[1], r * v[2], r * v[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc += w[e] * v[e];
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (e >= lo && e < hi) entry(base + e, c[e], w[e]);
        }
    }
    __device__ __forceinline__ void entry(const uint32_t pos, const uint32_t c, const T w) {
        const T v = xs[c];
        g[pos] = r * v;
        acc += w * v;
    }
    static constexpr bool SUMS = true;
    using Sum = T;
    __device__ __forceinline__ Sum total(const int lanes) const { return group_sum(acc, lanes); }
    __device__ __forceinline__ void put(const uint32_t row, const Sum s) const { y[row] = s; }
};

template<typename T, int U, uint32_t W, uint32_t LANES>
__global__ void __launch_bounds__(W * 32, 1)
gather_outer_shared_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr, const T *__restrict__ data,
                           const T *__restrict__ row_vector, const T *__restrict__ col_vector, T *__restrict__ g,
                           T *__restrict__ y, const uint32_t n_row, const uint32_t nse, const uint32_t n_col,
                           const uint32_t long_from) {
    extern __shared__ __align__(16) unsigned char shared_vector[];
    T *xs = reinterpret_cast<T *>(shared_vector);
    constexpr Deal<W, LANES> deal;
    auto &cut_rows = cut_rows_at<T, W>(shared_vector, n_col * sizeof(T));
    GatherOuterVisit<T> visit{xs, row_vector, g, y, n_row, T(0), T(0)};
    walk_rows<T, true, U>(indices, indptr, data, n_row, nse, long_from, deal, visit, cut_rows, [&]() {
        fill_shared(xs, col_vector, n_col);
        zero_outside_rows(g, indptr, n_row, nse);
        __syncthreads();
    });
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

// The bands pay where the sectors of x are used again in an SM (as many entries as sectors: 2e6 entries, 100,000 columns
// 13.4 -> 11 us; two thirds, 400,000 columns: 26 -> 29), and where there are rows to sweep side by side (34 per SM: 26 ->
// 29 us, 135: 37 -> 28).  500 lanes per SM, 16 entries or more for each.
template<typename T, bool HOMO, int MODE>
bool bands(cudaStream_t stream, const CsrMatrix<T> &m, const T *row_vector, const T *x, T *y, T *out) {
    const uint32_t sms = static_cast<uint32_t>(sm_count());
    const auto aligned32 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; };
    if (m.n_row < 100u * sms || static_cast<double>(m.nse) / sms < m.n_col * (sizeof(T) / 32.0) || !aligned32(m.indices) ||
        ((MODE & BAND_SUM) && !HOMO && !aligned32(m.data)) || ((MODE & BAND_OUTER) && !aligned16(out)))
        return false;
    uint32_t log_l = 0;
    while (log_l < 5 && (static_cast<uint64_t>(m.n_row) << log_l) < 512u * sms && (m.nse / m.n_row >> log_l) >= 16u) ++log_l;
    const uint64_t blocks = ((static_cast<uint64_t>(m.n_row) << log_l) + BAND_THREADS - 1) / BAND_THREADS;
    bands_kernel<T, HOMO, MODE><<<static_cast<uint32_t>(std::min<uint64_t>(blocks, 64ull * sms)), BAND_THREADS, 0, stream>>>(
        m.indices, m.indptr, m.data, row_vector, x, y, out, m.n_row, m.nse, log_l);
    launch_ok();
    return true;
}
// columns from which the bands are faster than x in shared memory (200 KB of floats; of doubles, 164 KB)
template<typename T> constexpr uint32_t BANDS_FROM = sizeof(T) == 4 ? 51200u : 21000u;

// go(warps of a block, lanes of a row, where rows are cut): the first two are constants
template<uint32_t W, typename Go>
void with_lanes(const uint32_t nse, const uint32_t n_row, const LaneRule &rule, Go go) {
    const uint32_t warps = static_cast<uint32_t>(sm_count()) * W, lanes = lanes_per_row(nse, n_row, warps, rule);
    const uint32_t long_from = std::max(std::max(64u, nse / warps / 16u) * lanes, 2u * (nse / n_row));
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

template<typename T, bool HOMO>
bool gather_impl(cudaStream_t stream, const CsrMatrix<T> &m, const T *x, T *y) {
    constexpr int U = sizeof(T) == 8 ? 1 : 2;
    if (m.n_col > BANDS_FROM<T> && bands<T, HOMO, BAND_SUM>(stream, m, nullptr, x, y, nullptr)) return true;
    if (!usable(m, !HOMO)) return false;
    const Plan<T> p(m, !HOMO);
    if (p.fill + p.per * p.entry > 0.95 * (p.per * std::max(1.0, p.entry) + 1500)) return false;
    with_block(m, m.n_col * sizeof(T), PRODUCT_LANES<T>, [&](auto warps, auto lanes, const uint32_t long_from) {
        constexpr uint32_t W = decltype(warps)::value, L = decltype(lanes)::value;
        constexpr auto kernel = gather_shared_kernel<T, HOMO, U, W, L>;
        if (allow_shared<kernel>(ALL_SMEM))
            kernel<<<static_cast<uint32_t>(sm_count()), W * 32, shared_bytes<T, W>(m.n_col * sizeof(T)), stream>>>(
                m.indices, m.indptr, m.data, x, y, m.n_row, m.nse, m.n_col, long_from);
        launch_ok();
    });
    return true;
}

template<typename T, typename E, bool HOMO>
bool gather_events_impl(cudaStream_t stream, const CsrMatrix<T> &m, const E *events, uint32_t *workspace, T *y) {
    constexpr int U = sizeof(T) == 8 ? 1 : 2;
    using Sum = std::conditional_t<HOMO, uint32_t, T>;
    const uint32_t bytes = (m.n_col + 31u) / 32u * 4u;
    if (m.n_row == 0 || m.n_row > MOST_ROWS || m.n_col == 0 || m.nse == 0 || m.nse > MOST_ENTRIES || m.n_col > 8u * SHARED_SMEM || !aligned16(m.indices) ||
        (!HOMO && !aligned16(m.data)))
        return false;
    // The bits are packed by a launch of their own where the events are more than a block reads in its time (34 bytes per
    // clock).  The alternative gathers events through L1 and L2, 1.1 clocks each where they miss.
    const double per = static_cast<double>(m.nse) / sm_count(), gather = m.n_col * sizeof(E) > 200000u ? 1.0 : 0.6;
    const bool pack = m.n_col * sizeof(E) > 32768u;
    // Few events, which L1 serves by broadcast, and one weight: with the entries of doubles taken one quad at a time, this walk is
    // the slower one for rows of medium length (3001 columns, 1e8 entries, rows of 64, 121, 300, 512: plain kernel 113, 105, 119, 99
    // us, here 119, 129, 121, 116; rows of 700, here 114).  Floats take two quads, and are faster here throughout (plain 113,
    // 105, 121, 99; here 113, 86, 80, 79; with float events the same).  The lines lie where the plain kernel was measured to win.
    const double mean_row = static_cast<double>(m.nse) / m.n_row;
    if (HOMO && sizeof(T) == 8 && m.n_col * sizeof(E) <= 8192u && mean_row >= 64 && mean_row <= 512) return false;
    if (per * (gather - 0.25) < 2500 + (pack ? 2500 + bytes / 56.0 : m.n_col * sizeof(E) / 34.0)) return false;
    const uint32_t sms = static_cast<uint32_t>(sm_count());
    // Bytes take the vector's own length from L1, which streams the entries: 200 KB of them 157 us for 1e8 entries, bits 143.
    const bool as_bytes = m.n_col <= 131072u && m.n_col * sizeof(E) / 34.0 < (pack ? 2500 + bytes / 56.0 : m.n_col * sizeof(E) / 34.0) + 0.08 * per;
    if (as_bytes || !pack) {
        with_block(m, as_bytes ? m.n_col : bytes, EVENT_LANES<T>, [&](auto warps, auto lanes, const uint32_t long_from) {
            constexpr uint32_t W = decltype(warps)::value, L = decltype(lanes)::value;
            constexpr auto of_bytes = gather_events_kernel<T, E, HOMO, true, U, W, L>, of_bits = gather_events_kernel<T, E, HOMO, false, U, W, L>;
            if (as_bytes ? allow_shared<of_bytes>(ALL_SMEM) : allow_shared<of_bits>(ALL_SMEM))
                (as_bytes ? of_bytes : of_bits)<<<sms, W * 32, shared_bytes<Sum, W>(as_bytes ? m.n_col : bytes), stream>>>(
                    m.indices, m.indptr, m.data, events, nullptr, y, m.n_row, m.nse, m.n_col, long_from);
            launch_ok();
        });
        return true;
    }
    pack_events_kernel<E><<<std::min<uint32_t>((m.n_col + 255u) / 256u, 8u * sms), 256, 0, stream>>>(events, workspace, m.n_col);
    if (!launch_ok()) return true;
    with_block(m, bytes, EVENT_LANES<T>, [&](auto warps, auto lanes, const uint32_t long_from) {
        constexpr uint32_t W = decltype(warps)::value, L = decltype(lanes)::value;
        constexpr auto kernel = gather_events_kernel<T, E, HOMO, false, U, W, L>;
        if (!allow_shared<kernel>(ALL_SMEM)) {
            launch_ok();
            return;
        }
        const cudaError_t e = launch_dependent(kernel, dim3(sms), dim3(W * 32), shared_bytes<Sum, W>(bytes), stream, m.indices, m.indptr, m.data,
                                               events, workspace, y, m.n_row, m.nse, m.n_col,
                                               long_from);
        if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
    });
    return true;
}

template<typename T, bool HOMO>
bool scatter_pays(const CsrMatrix<T> &m) {
    if (!usable(m, !HOMO)) return false;
    const Plan<T> p(m, !HOMO);
    // a reduction into L2: slower the fewer columns share them (20,000 columns 3.1 clocks, 2000 columns 13), and in double
    const double words = sizeof(T) / 4, reduction = (1.85 + 25000.0 / m.n_col) * (sizeof(T) == 8 ? 1.25 : 1.0);
    return p.fill + 0.3 * words * m.n_col + p.per * (p.entry + 0.3 * words) <= 0.95 * (reduction * p.per + 1500);
}

// `behind_zero`: the launch in front clears y
template<typename T, bool HOMO>
bool scatter_impl(cudaStream_t stream, const CsrMatrix<T> &m, const T *x, T *y, const bool behind_zero = false) {
    constexpr int U = sizeof(T) == 8 ? 1 : 2;
    if (!scatter_pays<T, HOMO>(m)) return false;
    if (!behind_zero && cudaMemsetAsync(y, 0, sizeof(T) * static_cast<size_t>(m.n_col), stream) != cudaSuccess) return launch_ok(), true;
    with_block(m, m.n_col * sizeof(T), SCATTER_LANES<T>, [&](auto warps, auto lanes, const uint32_t long_from) {
        constexpr uint32_t W = decltype(warps)::value, L = decltype(lanes)::value;
        constexpr auto kernel = scatter_shared_kernel<T, HOMO, U, W, L>;
        const uint32_t smem = shared_bytes<T, W>(m.n_col * sizeof(T)), sms = static_cast<uint32_t>(sm_count());
        if (!allow_shared<kernel>(ALL_SMEM)) {
            launch_ok();
        } else if (behind_zero) {
            const cudaError_t e = launch_dependent(kernel, dim3(sms), dim3(W * 32), smem, stream, m.indices, m.indptr, m.data, x, y, m.n_row,
                                                   m.nse, m.n_col, long_from);
            if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
        } else {
            kernel<<<sms, W * 32, smem, stream>>>(m.indices, m.indptr, m.data, x, y, m.n_row, m.nse, m.n_col, long_from);
            launch_ok();
        }
    });
    return true;
}

// `zero`: elements to clear; false, and nothing cleared, where another kernel has to do the product
template<typename T>
bool outer_impl(cudaStream_t stream, const CsrMatrix<T> &m, const T *row_vector, const T *col_vector, T *g, T *zero = nullptr,
                const uint32_t n_zero = 0) {
    constexpr int U = 2;
    if (zero == nullptr && m.n_col > BANDS_FROM<T> && bands<T, true, BAND_OUTER>(stream, m, row_vector, col_vector, nullptr, g)) return true;
    if (!usable(m, false) || !aligned16(g)) return false;
    const Plan<T> p(m, true);                // one index in, one value out
    if (p.fill + p.per * p.entry > 0.95 * (p.per * std::max(1.0, p.entry) + 1500)) return false;
    with_block(m, m.n_col * sizeof(T), STEP_LANES<U>, [&](auto warps, auto lanes, const uint32_t long_from) {
        constexpr uint32_t W = decltype(warps)::value, L = decltype(lanes)::value;
        constexpr auto kernel = outer_shared_kernel<T, U, W, L>;
        if (allow_shared<kernel>(ALL_SMEM))
            kernel<<<static_cast<uint32_t>(sm_count()), W * 32, shared_bytes<T, W>(m.n_col * sizeof(T)), stream>>>(
                m.indices, m.indptr, row_vector, col_vector, g, zero, n_zero, m.n_row, m.nse, m.n_col, long_from);
        launch_ok();
    });
    return true;
}

// The gradients of a product, one launch (transposed product) or two without a memset between them.  A training step of a few
// million entries is bound by the host, and each launch costs it 2 to 3 us.
template<typename T>
bool gather_outer_impl(cudaStream_t stream, const CsrMatrix<T> &m, const T *row_vector, const T *col_vector, T *g, T *y) {
    constexpr int U = sizeof(T) == 8 ? 1 : 2;
    if (m.n_col > BANDS_FROM<T> && bands<T, false, BAND_SUM | BAND_OUTER>(stream, m, row_vector, col_vector, y, g)) return true;
    if (!usable(m, true) || !aligned16(g)) return false;
    const Plan<T> p(m, true);
    if (p.fill + p.per * p.entry > 0.95 * (p.per * std::max(1.0, p.entry) + 1500)) return false;
    constexpr uint32_t W = FEW_WARPS;        // (80 registers)
    with_lanes<W>(m.nse, m.n_row, STEP_LANES<U>, [&](auto, auto lanes, const uint32_t long_from) {
        constexpr auto kernel = gather_outer_shared_kernel<T, U, W, decltype(lanes)::value>;
        if (allow_shared<kernel>(ALL_SMEM))
            kernel<<<static_cast<uint32_t>(sm_count()), W * 32, shared_bytes<T, W>(m.n_col * sizeof(T)), stream>>>(
                m.indices, m.indptr, m.data, row_vector, col_vector, g, y, m.n_row, m.nse, m.n_col, long_from);
        launch_ok();
    });
    return true;
}

template<typename T>
bool outer_scatter_impl(cudaStream_t stream, const CsrMatrix<T> &m, const T *row_vector, const T *col_vector, T *g, T *y) {
    return m.n_col <= BANDS_FROM<T> && scatter_pays<T, false>(m) && outer_impl<T>(stream, m, row_vector, col_vector, g, y, m.n_col) &&
           scatter_impl<T, false>(stream, m, row_vector, y, true);
}

}  // namespace

bool gather_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *x, float *y) {
    return m.homo ? gather_impl<float, true>(stream, m, x, y) : gather_impl<float, false>(stream, m, x, y);
}
bool gather_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *x, double *y) {
    return m.homo ? gather_impl<double, true>(stream, m, x, y) : gather_impl<double, false>(stream, m, x, y);
}
template<typename T, typename E>
bool gather_events(cudaStream_t stream, const CsrMatrix<T> &m, const E *events, uint32_t *workspace, T *y) {
    return m.homo ? gather_events_impl<T, E, true>(stream, m, events, workspace, y)
                  : gather_events_impl<T, E, false>(stream, m, events, workspace, y);
}
template bool gather_events(cudaStream_t, const CsrMatrix<float> &, const uint8_t *, uint32_t *, float *);
template bool gather_events(cudaStream_t, const CsrMatrix<float> &, const float *, uint32_t *, float *);
template bool gather_events(cudaStream_t, const CsrMatrix<double> &, const uint8_t *, uint32_t *, double *);
template bool gather_events(cudaStream_t, const CsrMatrix<double> &, const double *, uint32_t *, double *);
bool scatter_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *x, float *y) {
    return m.homo ? scatter_impl<float, true>(stream, m, x, y) : scatter_impl<float, false>(stream, m, x, y);
}
bool scatter_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *x, double *y) {
    return m.homo ? scatter_impl<double, true>(stream, m, x, y) : scatter_impl<double, false>(stream, m, x, y);
}
bool outer_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *r, const float *c, float *g) {
    return outer_impl<float>(stream, m, r, c, g);
}
bool outer_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *r, const double *c, double *g) {
    return outer_impl<double>(stream, m, r, c, g);
}

bool gather_outer_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *r, const float *c, float *g, float *y) {
    return gather_outer_impl<float>(stream, m, r, c, g, y);
}
bool gather_outer_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *r, const double *c, double *g, double *y) {
    return gather_outer_impl<double>(stream, m, r, c, g, y);
}
bool outer_scatter_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *r, const float *c, float *g, float *y) {
    return outer_scatter_impl<float>(stream, m, r, c, g, y);
}
bool outer_scatter_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *r, const double *c, double *g, double *y) {
    return outer_scatter_impl<double>(stream, m, r, c, g, y);
}

}  // namespace bpl
