// Products that gather from a dense vector: y = A x, the gradient of the weights, and both gradients of a transposed product at once.
// With x in shared memory (csr_shared.cuh), or read through L1 in bands.
#include "csr_shared.cuh"

namespace bpl {
namespace {

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

// `zero`: elements to clear; false, and nothing cleared, where another kernel has to do the product
template<typename T>
bool outer_impl(cudaStream_t stream, const CsrMatrix<T> &m, const T *row_vector, const T *col_vector, T *g, T *zero,
                const uint32_t n_zero) {
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

}  // namespace

bool gather_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *x, float *y) {
    return m.homo ? gather_impl<float, true>(stream, m, x, y) : gather_impl<float, false>(stream, m, x, y);
}
bool gather_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *x, double *y) {
    return m.homo ? gather_impl<double, true>(stream, m, x, y) : gather_impl<double, false>(stream, m, x, y);
}
bool outer_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *r, const float *c, float *g, float *zero, uint32_t n_zero) {
    return outer_impl<float>(stream, m, r, c, g, zero, n_zero);
}
bool outer_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *r, const double *c, double *g, double *zero, uint32_t n_zero) {
    return outer_impl<double>(stream, m, r, c, g, zero, n_zero);
}
bool gather_outer_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *r, const float *c, float *g, float *y) {
    return gather_outer_impl<float>(stream, m, r, c, g, y);
}
bool gather_outer_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *r, const double *c, double *g, double *y) {
    return gather_outer_impl<double>(stream, m, r, c, g, y);
}

}  // namespace bpl
