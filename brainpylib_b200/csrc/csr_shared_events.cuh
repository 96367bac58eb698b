// Products that gather from events (csr_shared.cuh); one source per type of the weights includes this.
#ifndef BPL_CSRC_CSR_SHARED_EVENTS_CUH_
#define BPL_CSRC_CSR_SHARED_EVENTS_CUH_

#include "csr_shared.cuh"

namespace bpl {
namespace {

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

constexpr uint32_t MOST_EVENT_BYTES = 131072u;

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
    const bool as_bytes = m.n_col <= MOST_EVENT_BYTES && m.n_col * sizeof(E) / 34.0 < (pack ? 2500 + bytes / 56.0 : m.n_col * sizeof(E) / 34.0) + 0.08 * per;
    if (as_bytes || !pack) {
        static_assert(MOST_EVENT_BYTES <= MANY_SMEM, "as many warps as there may be");
        with_lanes<MANY_WARPS>(m.nse, m.n_row, EVENT_LANES<T>, [&](auto warps, auto lanes, const uint32_t long_from) {
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

}  // namespace

template<typename T, typename E>
bool gather_events(cudaStream_t stream, const CsrMatrix<T> &m, const E *events, uint32_t *workspace, T *y) {
    return m.homo ? gather_events_impl<T, E, true>(stream, m, events, workspace, y)
                  : gather_events_impl<T, E, false>(stream, m, events, workspace, y);
}

}  // namespace bpl

#endif  // BPL_CSRC_CSR_SHARED_EVENTS_CUH_
