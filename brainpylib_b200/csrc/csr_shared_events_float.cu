#include "csr_shared_events.cuh"

namespace bpl {

template bool gather_events(cudaStream_t, const CsrMatrix<float> &, const uint8_t *, uint32_t *, float *);
template bool gather_events(cudaStream_t, const CsrMatrix<float> &, const float *, uint32_t *, float *);

}  // namespace bpl
