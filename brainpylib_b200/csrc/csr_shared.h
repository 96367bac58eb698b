// Whole-matrix CSR products with a vector in shared memory (csr_shared.cuh).  Each function returns false, having done
// nothing, where the plain kernels are faster or the operands do not fit; nse is the number of stored entries.
#ifndef BPL_CSRC_CSR_SHARED_H_
#define BPL_CSRC_CSR_SHARED_H_

#include <cstdint>
#include <cuda_runtime_api.h>

namespace bpl {

template<typename T>
struct CsrMatrix {
    const uint32_t *indices, *indptr;
    const T *data;              // one weight (homo) or nse
    uint32_t n_row, n_col, nse;
    bool homo;
};

// y = A x
bool gather_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *x, float *y);
bool gather_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *x, double *y);
// y = A events (E: uint8_t, or T); workspace: n_col bits, in whole words
template<typename T, typename E>
bool gather_events(cudaStream_t stream, const CsrMatrix<T> &m, const E *events, uint32_t *workspace, T *y);
// y = A^T x; y need not be zero
bool scatter_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *x, float *y);
bool scatter_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *x, double *y);
// g[e] = row_vector[row of e] * col_vector[indices[e]]; m.data is not read.  `zero`: n_zero elements to clear for the launch behind
bool outer_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *row_vector, const float *col_vector, float *g,
                  float *zero = nullptr, uint32_t n_zero = 0);
bool outer_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *row_vector, const double *col_vector, double *g,
                  double *zero = nullptr, uint32_t n_zero = 0);
// g as above and y[row] = sum of data * col_vector[column] (the gradients of a transposed product), or y[column] = sum of
// data * row_vector[row] (of the other one); y need not be zero
bool gather_outer_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *row_vector, const float *col_vector, float *g, float *y);
bool gather_outer_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *row_vector, const double *col_vector, double *g, double *y);
bool outer_scatter_shared(cudaStream_t stream, const CsrMatrix<float> &m, const float *row_vector, const float *col_vector, float *g, float *y);
bool outer_scatter_shared(cudaStream_t stream, const CsrMatrix<double> &m, const double *row_vector, const double *col_vector, double *g, double *y);

}  // namespace bpl

#endif  // BPL_CSRC_CSR_SHARED_H_
