// Checks of what the just-in-time walks rest on (brainpylib_b200/csrc/jit_stream.cuh), on the device.  Test infrastructure.
#include "../brainpylib_b200/csrc/jit_stream.cuh"

namespace bpl {
namespace {

// The largest |L ln2 - log(u)| / (LOG_ABS + LOG_REL |L ln2|) of all 2^32 draws: at most 1 where the ends of a gap enclose the
// reference's quotient, for any probability.
__global__ void __launch_bounds__(256) log_error_kernel(unsigned long long *__restrict__ most) {
    double worst = 0.0;
    for (unsigned long long x = blockIdx.x * 256ull + threadIdx.x; x < 1ull << 32; x += gridDim.x * 256ull) {
        const float u = _curand_uniform(static_cast<uint32_t>(x));
        const double quick = lg2_approx(u) * 0.69314718055994530942, reference = log(u);
        worst = fmax(worst, fabs(quick - reference) / (LOG_ABS + LOG_REL * fabs(quick)));
    }
    for (int o = 16; o > 0; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if ((threadIdx.x & 31u) == 0) atomicMax(most, static_cast<unsigned long long>(__double_as_longlong(worst)));      // (not negative)
}

// Streams seed .. seed + n_streams - 1 in batches, and one connection at a time by the reference's expression: count[0] the
// connections inside the range, count[1] those whose position or raw draws differ.
template<int KIND, int COUNT, bool SUMS, bool LOW24>
__global__ void __launch_bounds__(256) batches_kernel(const GapParams g, const uint32_t seed, const uint32_t n_streams, const uint32_t n,
                                                      unsigned long long *__restrict__ count) {
    unsigned long long inside = 0, wrong = 0;
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n_streams; i += gridDim.x * 256u) {
        Xorwow s, t;
        s.seed(seed + i);
        t.seed(seed + i);
        Batch<KIND, true, COUNT, SUMS> b;
        uint32_t at = 0;
        double pos = 0.0;
        while (at < n) {
            b.template draw<LOW24>(s, at, n, g);
            uint32_t r0 = 0, r1 = 0;
            for (int j = 0; j < COUNT; ++j) {
                const double gap = ceil(log(_curand_uniform(t.next(g))) / g.log_p);
                if (KIND == W_UNIFORM) r0 = t.next(g);
                if (KIND == W_NORMAL && (j & 1) == 0) {
                    r0 = t.next(g);
                    r1 = t.next(g);
                }
                pos += gap;
                const uint32_t got = LOW24 ? b.pos[j] & 0xffffffu : b.pos[j];
                const uint32_t raw = KIND == W_NORMAL && (j & 1) ? r1 : r0;
                inside += pos < n;
                wrong += pos < n ? got != pos || (KIND != W_HOMO && b.raw[KIND == W_HOMO ? 0 : j] != raw) : got < n;
            }
            if (pos < n) wrong += at != pos; else wrong += at < n;
        }
    }
    atomicAdd(count, inside);
    atomicAdd(count + 1, wrong);
}

template<int KIND, int COUNT>
void batches(const bool sums, const bool low24, const GapParams &g, const uint32_t seed, const uint32_t n_streams, const uint32_t n,
             unsigned long long *count, cudaStream_t stream) {
    const unsigned blocks = (n_streams + 255u) / 256u;
    if (low24) batches_kernel<KIND, COUNT, true, true><<<blocks, 256, 0, stream>>>(g, seed, n_streams, n, count);
    else if (sums) batches_kernel<KIND, COUNT, true, false><<<blocks, 256, 0, stream>>>(g, seed, n_streams, n, count);
    else batches_kernel<KIND, COUNT, false, false><<<blocks, 256, 0, stream>>>(g, seed, n_streams, n, count);
}

}  // namespace
}  // namespace bpl

using namespace bpl;

extern "C" {

// All write to device memory that the caller has cleared, and return 0 or a CUDA error; -1 for a log_p outside the quick test's range.
int draws_log_error(double *most, cudaStream_t stream) {
    log_error_kernel<<<148 * 8, 256, 0, stream>>>(reinterpret_cast<unsigned long long *>(most));
    return cudaGetLastError();
}

// `kind` as in jit_stream.cuh; batches of 4, 6 or 8 connections
int draws_batch_mismatches(int kind, int per_batch, int sums, int low24, double log_p, uint32_t seed, uint32_t n_streams, uint32_t n,
                           unsigned long long *count, cudaStream_t stream) {
    const GapParams g = gap_params(log_p, n);
    if (!g.quick || kind < 0 || kind > 2 || (per_batch != 4 && per_batch != 6 && per_batch != 8)) return -1;
    using Call = void (*)(bool, bool, const GapParams &, uint32_t, uint32_t, uint32_t, unsigned long long *, cudaStream_t);
    static const Call calls[3][3] = {{batches<W_HOMO, 4>, batches<W_HOMO, 6>, batches<W_HOMO, 8>},
                                     {batches<W_UNIFORM, 4>, batches<W_UNIFORM, 6>, batches<W_UNIFORM, 8>},
                                     {batches<W_NORMAL, 4>, batches<W_NORMAL, 6>, batches<W_NORMAL, 8>}};
    calls[kind][per_batch / 2 - 2](sums != 0, low24 != 0, g, seed, n_streams, n, count, stream);
    return cudaGetLastError();
}

}  // extern "C"
