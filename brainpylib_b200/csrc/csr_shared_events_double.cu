#include "csr_shared_events.cuh"

namespace bpl {

template bool gather_events(cudaStream_t, const CsrMatrix<double> &, const uint8_t *, uint32_t *, double *);
template bool gather_events(cudaStream_t, const CsrMatrix<double> &, const double *, uint32_t *, double *);

}  // namespace bpl
