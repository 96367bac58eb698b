// Products that scatter into sums in shared memory (csr_shared.cuh): y = A^T x, and both gradients of y = A x.
#include "csr_shared.cuh"

namespace bpl {
namespace {

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
    const auto launch = [&](auto warps, auto lanes, const uint32_t long_from) {
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
    };
    // Rows of 400 to 1000 floats: 24 warps beside any vector, 24 and 32 us: 6e6 entries, rows of 600, 2185 columns 22.6, 24.6, 8000
    // columns 20.5, 22.6; 1.2e7, of 500, 34.8, 36.8; 2e7, of 450, 51.3, 52.8; of 900 the same.  (Of 1500, 1.2e7, 34.8 and 32.8; doubles of
    // 1500 41.9 and 34.5, of 396, 1.5e6, 17.8 and 15.2.)
    const uint32_t mean = m.nse / m.n_row;
    LaneRule rule = SCATTER_LANES<T>;
    // Few columns: the 32 lanes sooner.  By 16 and 32, rows of 300: 1.2e7 entries, 1700 columns 39.0, 36.9, 8000 columns 35.7, 33.8,
    // 40,000 columns 35.9, 38.0; 2e7, 16,000 columns 47.5, 50.3, 40,000 columns 50.3, 52.3.
    if (sizeof(T) == 4 && m.n_col <= 8192u) rule.sixteen = 280u;
    if (sizeof(T) == 4 && mean > 400u && mean <= 1000u) with_lanes<FEW_WARPS>(m.nse, m.n_row, rule, launch);
    else with_block(m, m.n_col * sizeof(T), rule, launch);
    return true;
}

template<typename T>
bool outer_scatter_impl(cudaStream_t stream, const CsrMatrix<T> &m, const T *row_vector, const T *col_vector, T *g, T *y) {
    return m.n_col <= BANDS_FROM<T> && scatter_pays<T, false>(m) && outer_shared(stream, m, row_vector, col_vector, g, y, m.n_col) &&
           scatter_impl<T, false>(stream, m, row_vector, y, true);
}

}  // namespace

bool scatter_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *x, float *y) {
    return m.homo ? scatter_impl<float, true>(stream, m, x, y) : scatter_impl<float, false>(stream, m, x, y);
}
bool scatter_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *x, double *y) {
    return m.homo ? scatter_impl<double, true>(stream, m, x, y) : scatter_impl<double, false>(stream, m, x, y);
}
bool outer_scatter_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *r, const float *c, float *g, float *y) {
    return outer_scatter_impl<float>(stream, m, r, c, g, y);
}
bool outer_scatter_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *r, const double *c, double *g, double *y) {
    return outer_scatter_impl<double>(stream, m, r, c, g, y);
}

}  // namespace bpl
