// Stored-matrix (CSR) synaptic propagation for sm_100a:
//   event_csr_matvec  (replaces lib/gpu_event_csr_matvec.cu of the reference)
//   csr_matvec        (replaces lib/gpu_csr_matvec.cu) and its transposed form
//   gpu_csr_event_sum (replaces the CSR half of lib/gpu_event_sum.cu)
//
// Scatter direction (y = A^T x, "transpose"): the spike vector is first compacted into a
// list of active rows (scan_events_kernel, which also zero-fills y), then only those rows
// are streamed with 128-bit loads and scattered with one `red.global.add` per synapse
// (row_scatter_kernel).  Homogeneous weights use the same float reductions: k additions
// of one value give the same float in any order, so the result equals the reference's
// sequential sum bit for bit.
//
// Gather direction (y = A x): a sub-warp per row streams the whole matrix with 128-bit
// loads and reduces with shuffles (row_gather_kernel).
#include "abi.h"
#include "common.cuh"
#include "spike_scan.cuh"
#include "row_scatter.cuh"
#include "csr_shared.h"

namespace bpl {
namespace {

// ------------------------------------------------------------------------------------------
// Gather direction: y[r] = sum_j w_j * f(x[col_j]) with a group of `lpr` lanes per row
// ------------------------------------------------------------------------------------------
// EVENT = true : f = truthiness of the event; homogeneous weights count hits and scale once
//                (equal to the reference CPU kernel's float64 accumulation,
//                brainpylib/_src/event_ops/event_csr_matvec.py:334-357).
// EVENT = false: f = x, products accumulated with fused multiply-adds as the reference
//                `sum += data[e] * x[col]` compiles to (lib/gpu_csr_matvec.cu:163).
//
// MASK = true (events only): the block first packs the event vector into a bitmask in shared memory
// (one ballot per 32 events) and tests bits instead of gathering event bytes through L1/L2; the
// whole-matrix stream then runs at HBM speed.  Blocks of 1024 threads, mask of n_col / 8 bytes.
constexpr int GATHER_MASK_THREADS = 1024;
constexpr uint32_t GATHER_MASK_MAX_BITS = 200u * 1024u * 8u;

template<typename T, typename X, bool HOMO, bool EVENT, bool VEC, bool MASK = false>
__global__ void __launch_bounds__(MASK ? GATHER_MASK_THREADS : ROW_THREADS)
row_gather_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr,
                  const T *__restrict__ data, const X *__restrict__ x, const uint32_t n_row,
                  T *__restrict__ y, const uint32_t n_col = 0) {
    extern __shared__ uint32_t event_mask[];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps_per_block = blockDim.x >> 5;
    if (MASK) {
        pack_event_mask(x, n_col, event_mask);
        __syncthreads();
    }
    auto hit = [&](uint32_t col) -> bool {
        if (MASK) return (event_mask[col >> 5] >> (col & 31u)) & 1u;
        return is_event(x[col]);
    };
    const uint32_t nse = indptr[n_row];
    const uint32_t mean = n_row ? nse / n_row : 0;
    // Lanes per row: a lane takes 4 consecutive entries per 128-bit load and up to GATHER_UNROLL such
    // loads per step, so mean / 16 lanes cover an average row in one step.  Few lanes per row means
    // several rows per warp in flight, which is what hides the pointer -> entries -> gather latency
    // chain when rows are short.
    const uint32_t want = (mean + 15u) / 16u;
    const uint32_t lpr = want <= 4u ? 4u : (want <= 8u ? 8u : (want <= 16u ? 16u : 32u));
    const uint32_t rows_per_warp = 32u / lpr;
    const uint32_t sub = lane / lpr, sl = lane % lpr;
    const T homo_w = HOMO ? data[0] : T(0);
    const uint64_t n_warps = static_cast<uint64_t>(gridDim.x) * warps_per_block;
    const uint64_t n_groups = (static_cast<uint64_t>(n_row) + rows_per_warp - 1) / rows_per_warp;
    const uint32_t g_full = nse >> 2;
    constexpr int GATHER_UNROLL = 4;

    for (uint64_t wg = static_cast<uint64_t>(blockIdx.x) * warps_per_block + (threadIdx.x >> 5); wg < n_groups;
         wg += n_warps) {
        const uint64_t row64 = wg * rows_per_warp + sub;
        const bool live = row64 < n_row;
        const uint32_t row = live ? static_cast<uint32_t>(row64) : 0u;
        const uint32_t start = live ? indptr[row] : 0u, end = live ? indptr[row + 1] : 0u;
        T acc = T(0);
        uint32_t hits = 0;
        if (VEC) {
            const uint32_t g_begin = start >> 2, g_end = (end + 3u) >> 2;
            for (uint32_t g0 = g_begin + sl; g0 < g_end; g0 += lpr * GATHER_UNROLL) {
                uint4 ix[GATHER_UNROLL];
                Quad<T> wq[GATHER_UNROLL];
#pragma unroll
                for (int u = 0; u < GATHER_UNROLL; ++u) {
                    const uint32_t g = g0 + u * lpr;
                    if (g < g_end && g < g_full) {
                        ix[u] = ldg_stream_u4(indices + 4ull * g);
                        if (!HOMO) load_quad(data + 4ull * g, wq[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < GATHER_UNROLL; ++u) {
                    const uint32_t g = g0 + u * lpr;
                    if (g >= g_end) continue;
                    if (g < g_full) {
                        const uint32_t c[4] = {ix[u].x, ix[u].y, ix[u].z, ix[u].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t pos = 4u * g + e;
                            if (pos >= start && pos < end) {
                                if (EVENT) {
                                    if (hit(c[e])) { if (HOMO) ++hits; else acc += wq[u].v[e]; }
                                } else {
                                    acc += (HOMO ? homo_w : wq[u].v[e]) * static_cast<T>(x[c[e]]);
                                }
                            }
                        }
                    } else {   // ragged tail of the arrays: element-wise
                        for (uint32_t pos = max(4u * g, start); pos < end; ++pos) {
                            const uint32_t col = indices[pos];
                            if (EVENT) {
                                if (hit(col)) { if (HOMO) ++hits; else acc += data[pos]; }
                            } else {
                                acc += (HOMO ? homo_w : data[pos]) * static_cast<T>(x[col]);
                            }
                        }
                    }
                }
            }
        } else {
            for (uint32_t pos = start + sl; pos < end; pos += lpr) {
                const uint32_t col = indices[pos];
                if (EVENT) {
                    if (hit(col)) { if (HOMO) ++hits; else acc += data[pos]; }
                } else {
                    acc += (HOMO ? homo_w : data[pos]) * static_cast<T>(x[col]);
                }
            }
        }
        if (EVENT && HOMO) {
            hits = group_sum(hits, static_cast<int>(lpr));
            // no hit leaves +0 like an empty sum (the product with a negative weight would give -0)
            acc = hits ? static_cast<T>(static_cast<double>(hits) * static_cast<double>(homo_w)) : T(0);
        } else {
            acc = group_sum(acc, static_cast<int>(lpr));
        }
        if (live && sl == 0) y[row] = acc;
    }
}

// ------------------------------------------------------------------------------------------
// g[e] = row_vector[row(e)] * col_vector[indices[e]]: gradient of a product with respect to the weights
// ------------------------------------------------------------------------------------------
// One pass instead of the array operations it replaces (row id of every entry, both ids widened to 64 bits, two gathered
// copies, a product: about 60 B per entry and a host synchronisation); here 4 B in and one value out per entry.
template<typename T, bool VEC>
__global__ void __launch_bounds__(ROW_THREADS)
csr_outer_kernel(const T *__restrict__ row_vector, const T *__restrict__ col_vector, const uint32_t *__restrict__ indices,
                 const uint32_t *__restrict__ indptr, T *__restrict__ g, const uint32_t n_row, const uint32_t nse) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t mean = n_row ? nse / n_row : 0;
    const uint32_t want = (mean + 15u) / 16u;
    const uint32_t lpr = want <= 4u ? 4u : (want <= 8u ? 8u : (want <= 16u ? 16u : 32u));
    const uint32_t rows_per_warp = 32u / lpr;
    const uint32_t sub = lane / lpr, sl = lane % lpr;
    const uint64_t n_warps = static_cast<uint64_t>(gridDim.x) * ROW_WARPS;
    const uint64_t n_groups = (static_cast<uint64_t>(n_row) + rows_per_warp - 1) / rows_per_warp;
    // A row that would keep its lanes for more than 8 steps, and for more than twice a warp's share of all, is put off and
    // taken by the whole block (20,000 rows, 2e6 entries, 300,000 of them in one row: 4.8 ms by the lanes of each row).
    constexpr uint32_t LONG_ROWS = 256;
    __shared__ uint32_t n_long, long_row[LONG_ROWS];
    const uint32_t long_from = max(128u, nse / (gridDim.x * ROW_WARPS) / 16u) * lpr;
    const uint32_t g_full = nse >> 2;
    constexpr int UNROLL = 4;
    // entries [start, end) by every `lanes`-th of some threads, the `first` this one
    auto span = [&](const uint32_t start, const uint32_t end, const T r, const uint32_t first, const uint32_t lanes) {
        if (VEC) {
            const uint32_t g_end = (end + 3u) >> 2;
            for (uint32_t g0 = (start >> 2) + first; g0 < g_end; g0 += lanes * UNROLL) {
                uint4 ix[UNROLL];
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    const uint32_t q = g0 + u * lanes;
                    if (q < g_end && q < g_full) ix[u] = ldg_stream_u4(indices + 4ull * q);
                }
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    const uint32_t q = g0 + u * lanes;
                    if (q >= g_end) continue;
                    if (q < g_full) {
                        const uint32_t c[4] = {ix[u].x, ix[u].y, ix[u].z, ix[u].w};
                        if (4u * q >= start && 4u * q + 4u <= end) {
                            store_quad(g + 4ull * q, r * col_vector[c[0]], r * col_vector[c[1]], r * col_vector[c[2]],
                                       r * col_vector[c[3]]);
                        } else {   // a quad shared with the neighbouring rows
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const uint32_t pos = 4u * q + e;
                                if (pos >= start && pos < end) g[pos] = r * col_vector[c[e]];
                            }
                        }
                    } else {       // ragged tail of the arrays
                        for (uint32_t pos = max(4u * q, start); pos < end; ++pos) g[pos] = r * col_vector[indices[pos]];
                    }
                }
            }
        } else {
            for (uint32_t pos = start + first; pos < end; pos += lanes) g[pos] = r * col_vector[indices[pos]];
        }
    };
    if (threadIdx.x == 0) n_long = 0;
    __syncthreads();
    for (uint64_t wg = static_cast<uint64_t>(blockIdx.x) * ROW_WARPS + (threadIdx.x >> 5); wg < n_groups; wg += n_warps) {
        const uint64_t row = wg * rows_per_warp + sub;
        if (row >= n_row) continue;
        const uint32_t start = indptr[row], end = indptr[row + 1];
        if (end - start > long_from) {
            uint32_t at = 0;
            if (sl == 0) at = atomicAdd(&n_long, 1u);
            at = __shfl_sync((FULL_MASK >> (32u - lpr)) << (sub * lpr), at, sub * lpr);      // (all lanes of the row are here)
            if (at < LONG_ROWS) {
                if (sl == 0) long_row[at] = static_cast<uint32_t>(row);
                continue;
            }
        }
        span(start, end, row_vector[row], sl, lpr);
    }
    __syncthreads();
    const uint32_t n = min(n_long, LONG_ROWS);
    for (uint32_t i = 0; i < n; ++i) span(indptr[long_row[i]], indptr[long_row[i] + 1], row_vector[long_row[i]], threadIdx.x, ROW_THREADS);
    zero_outside_rows(g, indptr, n_row, nse);
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
inline int persistent_blocks(int blocks_per_sm, uint64_t work_warps) {
    const uint64_t cap = static_cast<uint64_t>(sm_count()) * blocks_per_sm;
    const uint64_t need = (work_warps + ROW_WARPS - 1) / ROW_WARPS;
    return static_cast<int>(need < 1 ? 1 : (need < cap ? need : cap));
}

// y = A events, the events gathered through L1
template<typename T, typename E, bool HOMO>
void event_gather(cudaStream_t stream, const uint32_t *indices, const uint32_t *indptr, const T *data, const E *events, T *y,
                  const uint32_t n_row) {
    const int grid = persistent_blocks(8, n_row);
    if (aligned16(indices) && (HOMO || aligned16(data)))
        row_gather_kernel<T, E, HOMO, true, true><<<grid, ROW_THREADS, 0, stream>>>(indices, indptr, data, events, n_row, y);
    else
        row_gather_kernel<T, E, HOMO, true, false><<<grid, ROW_THREADS, 0, stream>>>(indices, indptr, data, events, n_row, y);
    launch_ok();
}

inline uint32_t direct_warps() { return 8u * static_cast<uint32_t>(sm_count()) * ROW_WARPS; }    // resident, one group each
inline bool direct_rows(const uint32_t n_row) { return n_row <= DIRECT_ROWS && n_row <= 32u * direct_warps(); }

// y = A^T events without a list; false where there are too many rows.  `pieces` of a row, or MOST_PIECES where the number of
// entries is not known here: a warp for each piece of each group (256 rows of 78,125 entries, 300,000 columns: 62 us, with a
// warp for four pieces 113).
template<typename T, typename E, bool HOMO>
bool event_scatter_direct(cudaStream_t stream, const uint32_t *indices, const uint32_t *indptr, const T *data, const E *events, T *y,
                          const uint32_t n_row, const uint32_t n_col, const uint32_t pieces) {
    if (!direct_rows(n_row)) return false;
    if (n_col == 0) return true;
    const uint32_t sms = static_cast<uint32_t>(sm_count()), warps = direct_warps();
    const uint32_t zero_grid = static_cast<uint32_t>(
        min((static_cast<uint64_t>(n_col) + 4 * ROW_THREADS - 1) / (4 * ROW_THREADS), static_cast<uint64_t>(8 * sms)));
    zero_kernel<T><<<zero_grid, ROW_THREADS, 0, stream>>>(y, n_col);
    if (!launch_ok() || n_row == 0) return true;
    const uint32_t per_group = (n_row + warps - 1) / warps, n_groups = (n_row + per_group - 1) / per_group;
    const dim3 grid((min(n_groups * pieces, warps) + ROW_WARPS - 1) / ROW_WARPS);
    if (profile_before()) cudaEventRecord(profile_before(), stream);
    const bool vec = aligned16(indices) && (HOMO || aligned16(data));
    const cudaError_t e = launch_dependent(vec ? event_scatter_kernel<T, E, HOMO, true> : event_scatter_kernel<T, E, HOMO, false>,
                                           grid, dim3(ROW_THREADS), 0, stream, indices, indptr, data, events, n_row, n_groups, y);
    if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
    if (profile_after()) cudaEventRecord(profile_after(), stream);
    return true;
}

template<typename T, typename E, bool HOMO>
void event_csr_matvec_impl(cudaStream_t stream, void **buffers, const char *opaque, size_t opaque_len) {
    const TwoUintOneBoolDescriptor *d = unpack<TwoUintOneBoolDescriptor>(opaque, opaque_len);
    if (!d) return;
    const uint32_t n_row = d->uint_x, n_col = d->uint_y;
    const T *data = static_cast<const T *>(buffers[0]);
    const uint32_t *indices = static_cast<const uint32_t *>(buffers[1]);
    const uint32_t *indptr = static_cast<const uint32_t *>(buffers[2]);
    const E *events = static_cast<const E *>(buffers[3]);
    T *y = static_cast<T *>(buffers[4]);
    const bool vec = aligned16(indices) && (HOMO || aligned16(data));

    if (d->bool_x) {
        if (n_col == 0) return;
        uint32_t *ws = static_cast<uint32_t *>(buffers[5]);
        if (ws == nullptr) {
            set_status(BPL_ERR_ARGUMENT, "event_csr_matvec(transpose=True) needs a workspace buffer");
            return;
        }
        if (event_scatter_direct<T, E, HOMO>(stream, indices, indptr, data, events, y, n_row, n_col, MOST_PIECES)) return;
        uint32_t *counts = ws, *ids = ws + MAX_CHUNKS;
        const ScanPlan p = plan_scan(n_row);
        const uint64_t zero_blocks = (static_cast<uint64_t>(n_col) + SCAN_TILE - 1) / SCAN_TILE;
        const uint64_t zero_cap = static_cast<uint64_t>(sm_count()) * 8;
        const uint32_t scan_grid = static_cast<uint32_t>(
            max(static_cast<uint64_t>(p.n_chunks), min(zero_blocks, zero_cap)));
        scan_events_kernel<T, E><<<scan_grid, SCAN_THREADS, 0, stream>>>(
            events, n_row, p.chunk, p.n_chunks, y, n_col, counts, ids);
        if (!launch_ok()) return;
        if (n_row == 0) return;
        // one warp per work item; the grid is sized for the worst case (every row active) but capped
        // four blocks per SM are resident; for large matrices four times as many are launched: with more blocks than
        // the SMs hold the L2 reductions spread better (1e7 synapses per call: 70.3 us with 4 per SM, 64.3 with 16,
        // 66.8 with 32).  Small matrices keep one wave: every block prefix-sums the chunk counts first, which a
        // launch-bound call (4000 rows: 6.6 us) would pay several times over (9.1 us).
        const int grid = persistent_blocks(n_row >= 262144u ? 16 : 4, static_cast<uint64_t>(n_row) * 16);
        if (profile_before()) cudaEventRecord(profile_before(), stream);
        // a dependent launch behind the scan: the blocks are resident and wait only where they first read the list
        const cudaError_t e =
            vec ? launch_dependent(row_scatter_kernel<T, HOMO, true, true>, dim3(grid), dim3(ROW_THREADS), 0, stream, indices,
                                   indptr, data, static_cast<const T *>(nullptr), n_row, p.chunk, p.n_chunks, counts, ids, y)
                : launch_dependent(row_scatter_kernel<T, HOMO, true, false>, dim3(grid), dim3(ROW_THREADS), 0, stream,
                                   indices, indptr, data, static_cast<const T *>(nullptr), n_row, p.chunk, p.n_chunks, counts,
                                   ids, y);
        if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
        if (profile_after()) cudaEventRecord(profile_after(), stream);
        launch_ok();
    } else {
        if (n_row == 0) return;
        if (vec && n_col >= 8192u && n_col <= GATHER_MASK_MAX_BITS && n_row >= 4096u) {
            const size_t smem = static_cast<size_t>((n_col + 31u) >> 5) * 4;
            static thread_local int configured_device = -1;
            int dev = 0;
            cudaGetDevice(&dev);
            if (configured_device != dev) {
                if (cudaFuncSetAttribute(row_gather_kernel<T, E, HOMO, true, true, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(GATHER_MASK_MAX_BITS / 8)) != cudaSuccess) {
                    launch_ok();
                    return;
                }
                configured_device = dev;
            }
            const int per_sm = smem <= 100u * 1024u ? 2 : 1;
            const uint64_t need = (static_cast<uint64_t>(n_row) + GATHER_MASK_THREADS / 32 - 1) / (GATHER_MASK_THREADS / 32);
            const uint64_t cap = static_cast<uint64_t>(sm_count()) * per_sm;
            const int grid = static_cast<int>(need < cap ? need : cap);
            row_gather_kernel<T, E, HOMO, true, true, true><<<grid, GATHER_MASK_THREADS, smem, stream>>>(
                indices, indptr, data, events, n_row, y, n_col);
            launch_ok();
            return;
        }
        event_gather<T, E, HOMO>(stream, indices, indptr, data, events, y, n_row);
    }
}

template<typename T, bool HOMO>
void csr_matvec_call(cudaStream_t stream, const T *data, const uint32_t *indices, const uint32_t *indptr, const T *x, T *y,
                     const uint32_t n_row, const uint32_t n_col, const bool transpose) {
    const bool vec = aligned16(indices) && (HOMO || aligned16(data));

    if (transpose) {
        if (n_col == 0) return;
        if (cudaMemsetAsync(y, 0, sizeof(T) * static_cast<size_t>(n_col), stream) != cudaSuccess) {
            launch_ok();
            return;
        }
        if (n_row == 0) return;
        // more blocks than the SMs hold: the L2 reductions spread better (1e7 entries: 74.9 us with 4 blocks per SM,
        // 66.5 with 16, 64.9 with 32: the reduction floor)
        const int grid = persistent_blocks(32, static_cast<uint64_t>(n_row) * 16);
        if (vec)
            row_scatter_kernel<T, HOMO, false, true><<<grid, ROW_THREADS, 0, stream>>>(
                indices, indptr, data, x, n_row, 0, 0, nullptr, nullptr, y);
        else
            row_scatter_kernel<T, HOMO, false, false><<<grid, ROW_THREADS, 0, stream>>>(
                indices, indptr, data, x, n_row, 0, 0, nullptr, nullptr, y);
    } else {
        if (n_row == 0) return;
        const int grid = persistent_blocks(8, n_row);
        if (vec)
            row_gather_kernel<T, T, HOMO, false, true><<<grid, ROW_THREADS, 0, stream>>>(
                indices, indptr, data, x, n_row, y);
        else
            row_gather_kernel<T, T, HOMO, false, false><<<grid, ROW_THREADS, 0, stream>>>(
                indices, indptr, data, x, n_row, y);
    }
    launch_ok();
}

template<typename T, bool HOMO>
void csr_matvec_impl(cudaStream_t stream, void **buffers, const char *opaque, size_t opaque_len,
                     bool transpose, int vector_slot) {
    const DoubleSizeDescriptor *d = unpack<DoubleSizeDescriptor>(opaque, opaque_len);
    if (!d) return;
    csr_matvec_call<T, HOMO>(stream, static_cast<const T *>(buffers[0]), static_cast<const uint32_t *>(buffers[1]),
                             static_cast<const uint32_t *>(buffers[2]), static_cast<const T *>(buffers[vector_slot]),
                             static_cast<T *>(buffers[vector_slot + 1]), d->size_x, d->size_y, transpose);
}

// Scatter from the spike list with the sums of all columns in shared memory, for few columns: reductions of many rows
// into the same lines of L2 queue up (1.5e6 synapses into 2716 sums: 65 us, 44 G per second), shared memory adds at the
// rate of the entries: 12 us.  (Not for one weight for all, whose sums equal the reference's bit for bit: partial sums
// of one value round differently from adding it k times.)
constexpr uint32_t LIST_SHARED_THREADS = 1024;
constexpr uint32_t LIST_SHARED_SMEM = 200u * 1024u;

template<typename T, bool VEC>
__global__ void __launch_bounds__(LIST_SHARED_THREADS, 1)
list_scatter_shared_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr, const T *__restrict__ data,
                           const uint32_t n_row, const uint32_t n_col, const uint32_t chunk, const uint32_t n_chunks,
                           const uint32_t *__restrict__ counts, const uint32_t *__restrict__ ids, T *__restrict__ y) {
    extern __shared__ __align__(16) unsigned char shared_sums[];
    __shared__ uint32_t prefix[MAX_CHUNKS + 1];
    __shared__ uint32_t warp_total[LIST_SHARED_THREADS / 32];
    T *sums = reinterpret_cast<T *>(shared_sums);
    for (uint32_t i = threadIdx.x; i < n_col; i += LIST_SHARED_THREADS) sums[i] = T(0);
    pdl_wait();                                            // the list is there and y is zero
    const uint32_t n_list = chunk_prefix(counts, n_chunks, prefix, warp_total);
    const uint32_t lane = threadIdx.x & 31, nse = indptr[n_row], S = pieces_per_row(nse, n_row);
    const uint64_t n_items = static_cast<uint64_t>(n_list) * S;
    for (uint64_t item = static_cast<uint64_t>(threadIdx.x >> 5) * gridDim.x + blockIdx.x; item < n_items;
         item += static_cast<uint64_t>(gridDim.x) * (LIST_SHARED_THREADS / 32)) {
        const uint32_t li = static_cast<uint32_t>(item / S), h = static_cast<uint32_t>(item % S);
        const uint32_t row = list_row(prefix, n_chunks, chunk, ids, li), start = indptr[row], end = indptr[row + 1];
        const uint32_t a = piece_cut(start, end, h, S), b = piece_cut(start, end, h + 1, S);
        if (a < b) scatter_span<T, false, false, VEC, false>(indices, data, T(0), T(1), a, b, nse, sums, lane);
    }
    __syncthreads();
    if (n_list != 0) add_sums(sums, y, n_col, blockIdx.x, gridDim.x);
}

// How many rows are active is not known here; the rule supposes 1 % (a convention, not a measurement).  In clocks of one SM: a reduction takes
// 1.85, and more the fewer columns share them; the sums take 0.4 each to clear and to add up, and 3000 in all.
inline bool list_shared_pays(uint32_t n_row, uint32_t n_col, uint32_t nse, bool homo, size_t elem) {
    const double active = 0.01 * nse / sm_count();
    return !homo && n_row != 0 && n_col != 0 && n_col <= LIST_SHARED_SMEM / elem &&
           active * (1.5 + 25000.0 / n_col) >= 3000 + 0.4 * (elem / 4) * n_col;
}

template<typename T, typename E>
bool list_scatter_shared(cudaStream_t stream, const CsrMatrix<T> &m, const E *events, uint32_t *ws, T *y) {
    if (!list_shared_pays(m.n_row, m.n_col, m.nse, m.homo, sizeof(T))) return false;
    const bool vec = aligned16(m.indices) && aligned16(m.data);
    constexpr auto wide = list_scatter_shared_kernel<T, true>, narrow = list_scatter_shared_kernel<T, false>;
    if (!(vec ? allow_shared<wide>(LIST_SHARED_SMEM) : allow_shared<narrow>(LIST_SHARED_SMEM))) return launch_ok(), true;
    uint32_t *counts = ws, *ids = ws + MAX_CHUNKS;
    const ScanPlan p = plan_scan(m.n_row);
    scan_events_kernel<T, E><<<max(p.n_chunks, (m.n_col + SCAN_TILE - 1) / SCAN_TILE), SCAN_THREADS, 0, stream>>>(
        events, m.n_row, p.chunk, p.n_chunks, y, m.n_col, counts, ids);
    if (!launch_ok()) return true;
    if (profile_before()) cudaEventRecord(profile_before(), stream);
    const cudaError_t e = launch_dependent(vec ? wide : narrow, dim3(sm_count()), dim3(LIST_SHARED_THREADS), m.n_col * sizeof(T), stream,
                                           m.indices, m.indptr, m.data, m.n_row, m.n_col, p.chunk, p.n_chunks, counts, ids, y);
    if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
    if (profile_after()) cudaEventRecord(profile_after(), stream);
    return true;
}

// y = A^T events in ONE launch, for small matrices.  A launch costs the host 2.7 us, half of such a call.  Every block owns
// a range of the columns, finds the active rows itself, reads ALL their entries (from L2, where the blocks read them side by
// side) and adds those of its range in shared memory; y is written once and needs no zero-fill, and a column's sum is formed
// in one place (equal weights add up to the reference's bits).  Teams of lpr lanes take a row each, a row of more than `piece`
// entries (four steps of a team) in pieces: how long single rows are is not known when the team is chosen, and every block
// would wait for the longest (4096 rows, 150,000 entries, half of them in one row: 808 us by one team, 18 in pieces).
constexpr uint32_t OWN_THREADS = 1024;
constexpr uint32_t OWN_ROWS = 8192;

template<typename T, typename E, bool HOMO, bool VEC>
__global__ void __launch_bounds__(OWN_THREADS)
event_columns_kernel(const uint32_t *__restrict__ indices, const uint32_t *__restrict__ indptr, const T *__restrict__ data,
                     const E *__restrict__ events, const uint32_t n_row, const uint32_t n_col, const uint32_t nse,
                     const uint32_t width, const uint32_t log_lpr, const uint32_t piece, T *__restrict__ y) {
    extern __shared__ __align__(16) unsigned char own_smem[];
    __shared__ uint32_t n_active;
    T *sums = reinterpret_cast<T *>(own_smem);
    uint2 *list = reinterpret_cast<uint2 *>(own_smem + static_cast<size_t>(width) * sizeof(T));    // where pieces of active rows lie
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t first = blockIdx.x * width, count = min(width, n_col - first);
    if (threadIdx.x == 0) n_active = 0;
    for (uint32_t i = threadIdx.x; i < count; i += OWN_THREADS) sums[i] = T(0);
    pdl_launch_dependents();
    pdl_wait();                                            // whatever wrote the operands, or still reads y
    __syncthreads();
    constexpr int PER = 4;
    for (uint32_t base = 0; base < n_row; base += PER * OWN_THREADS) {
        bool act[PER];
        uint32_t at[PER], start[PER], end[PER];            // (all loads of the four before a branch on any: 0.6 us)
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const uint32_t i = base + k * OWN_THREADS + threadIdx.x;
            act[k] = i < n_row && is_event(__ldcg(events + i));
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            start[k] = end[k] = 0;
            const uint32_t bits = __ballot_sync(FULL_MASK, act[k]);
            if (bits == 0) continue;
            uint32_t first = 0;
            if (lane == 0) first = atomicAdd(&n_active, static_cast<uint32_t>(__popc(bits)));
            at[k] = __shfl_sync(FULL_MASK, first, 0) + __popc(bits & ((1u << lane) - 1u));
            if (act[k]) {
                const uint32_t row = base + k * OWN_THREADS + threadIdx.x;
                start[k] = indptr[row];
                end[k] = indptr[row + 1];
            }
        }
        bool pieces = false;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (act[k]) list[at[k]] = make_uint2(start[k], min(end[k], start[k] + piece));
            pieces |= end[k] - start[k] > piece;
        }
        if (pieces) {
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                if (end[k] - start[k] <= piece) continue;
                const uint32_t more = (end[k] - start[k] - 1u) / piece, from = atomicAdd(&n_active, more);
                for (uint32_t j = 0; j < more; ++j)
                    list[from + j] = make_uint2(start[k] + (j + 1u) * piece, min(end[k], start[k] + (j + 2u) * piece));
            }
        }
    }
    __syncthreads();
    const uint32_t n = n_active, lpr = 1u << log_lpr, sl = threadIdx.x & (lpr - 1u), teams = OWN_THREADS >> log_lpr;
    const uint32_t g_full = nse >> 2;
    const T homo_w = HOMO ? data[0] : T(0);
    auto add = [&](const uint32_t c, const T w) {
        const uint32_t i = c - first;
        if (i < count) atomicAdd(sums + i, w);
    };
    if (VEC) {
        // steps of lpr * U quads along the team's rows, the next one's entries requested before a step is added
        constexpr int U = HOMO ? 4 : sizeof(T) == 8 ? 1 : 2;   // two steps in 64 registers
        struct Step {
            uint32_t i, g0, start, end;                     // row of the list, first quad of the lane; i >= n: no step
            uint4 ix[U];
            Quad<T> w[HOMO ? 1 : U];
        };
        auto load = [&](Step &s) {
            const uint32_t g_stop = min((s.end + 3u) >> 2, g_full);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t g = s.g0 + u * lpr;
                if (g < g_stop) {
                    s.ix[u] = __ldg(reinterpret_cast<const uint4 *>(indices + 4ull * g));
                    if (!HOMO) load_quad(data + 4ull * g, s.w[u]);
                }
            }
        };
        auto row = [&](Step &s, const uint32_t i) {
            s.i = i;
            s.start = s.end = s.g0 = 0;
            if (i < n) {
                const uint2 r = list[i];
                s.start = r.x;
                s.end = r.y;
                s.g0 = (r.x >> 2) + sl;
                load(s);
            }
        };
        auto next = [&](const Step &now, Step &s) {
            const uint32_t g0 = now.g0 + lpr * U;
            if (g0 - sl < min((now.end + 3u) >> 2, g_full)) {   // the row goes on (for the whole team)
                s.i = now.i;
                s.start = now.start;
                s.end = now.end;
                s.g0 = g0;
                load(s);
            } else {
                row(s, now.i + teams);
            }
        };
        auto use = [&](const Step &s) {
            const uint32_t stop = min(s.end, 4u * g_full);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t pos = 4u * (s.g0 + u * lpr), c[4] = {s.ix[u].x, s.ix[u].y, s.ix[u].z, s.ix[u].w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (pos + e >= s.start && pos + e < stop) add(c[e], HOMO ? homo_w : s.w[HOMO ? 0 : u].v[e]);
            }
        };
        Step a, b;
        row(a, threadIdx.x >> log_lpr);
        while (a.i < n) {
            next(a, b);
            use(a);
            if (b.i >= n) break;
            next(b, a);
            use(b);
        }
        // the last entries of the arrays, behind their last whole quad
        for (uint32_t i = threadIdx.x; i < n; i += OWN_THREADS)
            for (uint32_t pos = max(4u * g_full, list[i].x); pos < list[i].y; ++pos) add(indices[pos], HOMO ? homo_w : data[pos]);
    } else {
        for (uint32_t i = threadIdx.x >> log_lpr; i < n; i += teams)
            for (uint32_t pos = list[i].x + sl; pos < list[i].y; pos += lpr) add(indices[pos], HOMO ? homo_w : data[pos]);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < count; i += OWN_THREADS) y[first + i] = sums[i];
}

// Every block reads what the others read: the events, and the entries of the active rows, at 34 bytes per clock.  With the
// 10 % of a lively network active, OWN_BYTES of matrix take the 2 us that the second launch would (4000 x 4000, 320,000
// synapses, 5 %: 5.3 us per call, 6.9 with two launches; with 10 % 7.4 and 7.0: at that size and activity the line is late).
constexpr double OWN_BYTES = 1.3e6;

inline bool columns_pay(uint32_t n_row, uint32_t n_col, uint32_t nse, size_t per_entry, size_t event) {
    return n_row != 0 && n_row <= OWN_ROWS && n_col != 0 && n_col <= 500000u && static_cast<double>(nse) * per_entry <= OWN_BYTES &&
           n_row * event <= 32768u;
}

template<typename T, typename E, bool HOMO>
bool event_scatter_columns(cudaStream_t stream, const CsrMatrix<T> &m, const E *events, T *y) {
    if (!columns_pay(m.n_row, m.n_col, m.nse, 4 + (HOMO ? 0 : sizeof(T)), sizeof(E))) return false;
    const uint32_t sms = static_cast<uint32_t>(sm_count());
    const uint32_t width = max(128u, ((m.n_col + sms - 1) / sms + 31u) & ~31u), blocks = (m.n_col + width - 1) / width;
    const uint32_t mean = m.nse / m.n_row;
    const uint32_t per = HOMO ? 16u : sizeof(T) == 8 ? 4u : 8u;                // entries of a lane and step
    const uint32_t log_lpr = mean <= 4u * per ? 2u : mean <= 8u * per ? 3u : mean <= 16u * per ? 4u : 5u;
    const bool vec = aligned16(m.indices) && (HOMO || aligned16(m.data));
    constexpr auto wide = event_columns_kernel<T, E, HOMO, true>, narrow = event_columns_kernel<T, E, HOMO, false>;
    const uint32_t piece = (4u * per) << log_lpr;
    const size_t items = static_cast<size_t>(m.n_row) + m.nse / piece;         // of the list, at most
    constexpr unsigned most = 110u * 1024u;                                    // (8192 rows, 108,333 doubles, 500,000 columns: 104 KB)
    const size_t smem = width * sizeof(T) + sizeof(uint2) * items;
    if (smem > most) return false;
    if (!(vec ? allow_shared<wide>(most) : allow_shared<narrow>(most))) return launch_ok(), true;
    if (profile_before()) cudaEventRecord(profile_before(), stream);
    const cudaError_t e = launch_dependent(vec ? wide : narrow, dim3(blocks), dim3(OWN_THREADS),
                                           smem, stream, m.indices, m.indptr, m.data, events, m.n_row, m.n_col, m.nse, width, log_lpr, piece, y);
    if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
    if (profile_after()) cudaEventRecord(profile_after(), stream);
    return true;
}

template<typename T, typename E, bool HOMO>
void event_csr_known(cudaStream_t stream, void **buffers, uint32_t n_row, uint32_t n_col, uint32_t nse, bool transpose) {
    const CsrMatrix<T> m{static_cast<const uint32_t *>(buffers[1]), static_cast<const uint32_t *>(buffers[2]),
                         static_cast<const T *>(buffers[0]), n_row, n_col, nse, HOMO};
    if (!transpose) {
        const E *events = static_cast<const E *>(buffers[3]);
        T *y = static_cast<T *>(buffers[4]);
        if (n_row != 0 && !gather_events(stream, m, events, static_cast<uint32_t *>(buffers[5]), y))
            event_gather<T, E, HOMO>(stream, m.indices, m.indptr, m.data, events, y, n_row);
        return;
    }
    if (event_scatter_columns<T, E, HOMO>(stream, m, static_cast<const E *>(buffers[3]), static_cast<T *>(buffers[4])) ||
        list_scatter_shared<T, E>(stream, m, static_cast<const E *>(buffers[3]), static_cast<uint32_t *>(buffers[5]),
                                        static_cast<T *>(buffers[4])) ||
        event_scatter_direct<T, E, HOMO>(stream, m.indices, m.indptr, m.data, static_cast<const E *>(buffers[3]),
                                         static_cast<T *>(buffers[4]), n_row, n_col, pieces_per_row(nse, n_row)))
        return;
    TwoUintOneBoolDescriptor d;
    __builtin_memset(&d, 0, sizeof(d));
    d.uint_x = n_row;
    d.uint_y = n_col;
    d.bool_x = transpose;
    event_csr_matvec_impl<T, E, HOMO>(stream, buffers, reinterpret_cast<const char *>(&d), sizeof(d));
}

// With the number of stored entries known: the kernels that hold the vector in shared memory where they are faster.
template<typename T>
void csr_matvec_known(cudaStream_t stream, const void *data, const uint32_t *indices, const uint32_t *indptr, const void *x,
                      void *y, uint32_t n_row, uint32_t n_col, uint32_t nse, bool homo, bool transpose) {
    const T *d = static_cast<const T *>(data), *v = static_cast<const T *>(x);
    T *out = static_cast<T *>(y);
    const CsrMatrix<T> m{indices, indptr, d, n_row, n_col, nse, homo};
    if (transpose ? scatter_shared(stream, m, v, out) : gather_shared(stream, m, v, out)) return;
    if (homo) csr_matvec_call<T, true>(stream, d, indices, indptr, v, out, n_row, n_col, transpose);
    else csr_matvec_call<T, false>(stream, d, indices, indptr, v, out, n_row, n_col, transpose);
}

template<typename T>
void csr_outer_impl(cudaStream_t stream, const void *row_vector, const void *col_vector, const uint32_t *indices,
                    const uint32_t *indptr, void *out, uint32_t n_row, uint32_t n_col, uint32_t nse) {
    if (nse == 0) return;
    if (n_row == 0) {
        if (cudaMemsetAsync(out, 0, sizeof(T) * static_cast<size_t>(nse), stream) != cudaSuccess) launch_ok();
        return;
    }
    const int grid = persistent_blocks(8, n_row);
    const T *r = static_cast<const T *>(row_vector), *c = static_cast<const T *>(col_vector);
    T *g = static_cast<T *>(out);
    if (outer_shared(stream, CsrMatrix<T>{indices, indptr, nullptr, n_row, n_col, nse, false}, r, c, g)) return;
    if (aligned16(indices) && aligned16(out))
        csr_outer_kernel<T, true><<<grid, ROW_THREADS, 0, stream>>>(r, c, indices, indptr, g, n_row, nse);
    else
        csr_outer_kernel<T, false><<<grid, ROW_THREADS, 0, stream>>>(r, c, indices, indptr, g, n_row, nse);
    launch_ok();
}

// Both gradients of a product of per-entry weights.
template<typename T>
void csr_gradients_impl(cudaStream_t stream, const void *data, const uint32_t *indices, const uint32_t *indptr, const void *x,
                        const void *ct, void *g_data, void *g_x, uint32_t n_row, uint32_t n_col, uint32_t nse, bool transpose) {
    const CsrMatrix<T> m{indices, indptr, static_cast<const T *>(data), n_row, n_col, nse, false};
    const T *row_vector = static_cast<const T *>(transpose ? x : ct), *col_vector = static_cast<const T *>(transpose ? ct : x);
    T *g = static_cast<T *>(g_data), *y = static_cast<T *>(g_x);
    if (transpose ? gather_outer_shared(stream, m, row_vector, col_vector, g, y) : outer_scatter_shared(stream, m, row_vector, col_vector, g, y))
        return;
    csr_outer_impl<T>(stream, row_vector, col_vector, indices, indptr, g_data, n_row, n_col, nse);
    csr_matvec_known<T>(stream, data, indices, indptr, ct, g_x, n_row, n_col, nse, false, !transpose);
}

}  // namespace
}  // namespace bpl

using namespace bpl;

extern "C" {

void bpl_csr_gradients(bpl_stream_t stream, const void *data, const void *indices, const void *indptr, const void *vector,
                       const void *cotangent, void *data_gradient, void *vector_gradient, uint32_t n_row, uint32_t n_col,
                       uint32_t nse, int is_double, int transpose) {
    const uint32_t *ix = static_cast<const uint32_t *>(indices), *ip = static_cast<const uint32_t *>(indptr);
    (is_double ? csr_gradients_impl<double> : csr_gradients_impl<float>)(stream, data, ix, ip, vector, cotangent, data_gradient,
                                                                        vector_gradient, n_row, n_col, nse, transpose != 0);
}

void bpl_csr_outer(bpl_stream_t stream, const void *row_vector, const void *col_vector, const void *indices,
                   const void *indptr, void *out, uint32_t n_row, uint32_t n_col, uint32_t nse, int is_double) {
    const uint32_t *ix = static_cast<const uint32_t *>(indices), *ip = static_cast<const uint32_t *>(indptr);
    if (is_double) csr_outer_impl<double>(stream, row_vector, col_vector, ix, ip, out, n_row, n_col, nse);
    else csr_outer_impl<float>(stream, row_vector, col_vector, ix, ip, out, n_row, n_col, nse);
}

void bpl_csr_matvec(bpl_stream_t stream, const void *data, const void *indices, const void *indptr, const void *vector,
                    void *out, uint32_t n_row, uint32_t n_col, uint32_t nse, int homo, int is_double, int transpose) {
    const uint32_t *ix = static_cast<const uint32_t *>(indices), *ip = static_cast<const uint32_t *>(indptr);
    (is_double ? csr_matvec_known<double> : csr_matvec_known<float>)(stream, data, ix, ip, vector, out, n_row, n_col, nse,
                                                                    homo != 0, transpose != 0);
}

size_t bpl_event_csr_matvec_workspace(uint32_t n_row, uint32_t n_col, uint32_t nse, int homo, int is_double, int transpose) {
    if (!transpose) return (static_cast<size_t>(n_col) + 31) / 32 * 4;
    const bool list = list_shared_pays(n_row, n_col, nse, homo != 0, is_double ? 8 : 4) || !direct_rows(n_row);
    return list ? scatter_workspace_bytes(n_row) : 0;
}
void bpl_event_csr_matvec(bpl_stream_t stream, void **buffers, uint32_t n_row, uint32_t n_col, uint32_t nse, int homo,
                          int is_double, int bool_events, int transpose) {
    using Call = void (*)(cudaStream_t, void **, uint32_t, uint32_t, uint32_t, bool);
    static const Call calls[2][2][2] = {   // [double][bool events][homo]
        {{event_csr_known<float, float, false>, event_csr_known<float, float, true>},
         {event_csr_known<float, uint8_t, false>, event_csr_known<float, uint8_t, true>}},
        {{event_csr_known<double, double, false>, event_csr_known<double, double, true>},
         {event_csr_known<double, uint8_t, false>, event_csr_known<double, uint8_t, true>}}};
    calls[is_double != 0][bool_events != 0][homo != 0](stream, buffers, n_row, n_col, nse, transpose != 0);
}

size_t bpl_event_csr_workspace_bytes(uint32_t n_row, int transpose) {
    return transpose ? scatter_workspace_bytes(n_row) : 0;
}

#define EVENT_CSR_TARGET(name, T, E, HOMO) \
    void name(bpl_stream_t s, void **b, const char *o, size_t n) { event_csr_matvec_impl<T, E, HOMO>(s, b, o, n); }

EVENT_CSR_TARGET(event_csr_matvec_homo_float_bool, float, uint8_t, true)
EVENT_CSR_TARGET(event_csr_matvec_homo_float_float, float, float, true)
EVENT_CSR_TARGET(event_csr_matvec_homo_double_bool, double, uint8_t, true)
EVENT_CSR_TARGET(event_csr_matvec_homo_double_double, double, double, true)
EVENT_CSR_TARGET(event_csr_matvec_heter_float_bool, float, uint8_t, false)
EVENT_CSR_TARGET(event_csr_matvec_heter_float_float, float, float, false)
EVENT_CSR_TARGET(event_csr_matvec_heter_double_bool, double, uint8_t, false)
EVENT_CSR_TARGET(event_csr_matvec_heter_double_double, double, double, false)

// The reference's scalar / vector / adaptive methods (lib/gpu_csr_matvec.cu) differ only in
// how rows are mapped to threads; here all three names run the same kernel.  'adaptive'
// carries its row_blocks operand at slot 3, which is ignored.
#define CSR_TARGET(name, T, HOMO, TRANSPOSE, SLOT) \
    void name(bpl_stream_t s, void **b, const char *o, size_t n) { csr_matvec_impl<T, HOMO>(s, b, o, n, TRANSPOSE, SLOT); }

CSR_TARGET(csr_matvec_homo_scalar_float, float, true, false, 3)
CSR_TARGET(csr_matvec_homo_scalar_double, double, true, false, 3)
CSR_TARGET(csr_matvec_homo_vector_float, float, true, false, 3)
CSR_TARGET(csr_matvec_homo_vector_double, double, true, false, 3)
CSR_TARGET(csr_matvec_homo_adaptive_float, float, true, false, 4)
CSR_TARGET(csr_matvec_homo_adaptive_double, double, true, false, 4)
CSR_TARGET(csr_matvec_heter_scalar_float, float, false, false, 3)
CSR_TARGET(csr_matvec_heter_scalar_double, double, false, false, 3)
CSR_TARGET(csr_matvec_heter_vector_float, float, false, false, 3)
CSR_TARGET(csr_matvec_heter_vector_double, double, false, false, 3)
CSR_TARGET(csr_matvec_heter_adaptive_float, float, false, false, 4)
CSR_TARGET(csr_matvec_heter_adaptive_double, double, false, false, 4)
CSR_TARGET(csr_matvec_transpose_homo_float, float, true, true, 3)
CSR_TARGET(csr_matvec_transpose_homo_double, double, true, true, 3)
CSR_TARGET(csr_matvec_transpose_heter_float, float, false, true, 3)
CSR_TARGET(csr_matvec_transpose_heter_double, double, false, true, 3)

}  // extern "C"

// ------------------------------------------------------------------------------------------
// Transposed event product that allocates nothing and takes no workspace buffer
// ------------------------------------------------------------------------------------------
// Who needs it: a caller that runs as an XLA custom call (or inside any framework's stream
// capture) receives exactly the buffers the framework planned for it and must not call
// cudaMalloc itself: allocation is illegal while a stream is being captured, synchronises
// the device, and takes memory behind the back of the framework's own allocator.  The
// regular targets solve this by asking for one extra workspace buffer; a caller that cannot
// even declare that extra buffer (it must keep the reference's exact five-buffer list) can
// use this entry point instead.  Its scratch (the compacted spike list) lives in a
// file-scope device array of fixed size, so the number of matrix rows is limited.
//
// Cost and rules of the fixed array:
//  * every GPU that loads this library holds BPL_NOALLOC_MAX_ROWS * 4 + 4096 bytes (about
//    8.4 MB) from the first use of the library on that GPU until the process exits;
//  * all calls on one GPU share it.  Nothing in it has to start at zero (every word that is
//    read was written earlier in the same call), so stale contents of an earlier call are
//    harmless, but two calls that overlap on the GPU (different streams, no ordering between
//    them) race on it and give wrong results: keep such calls on one stream or order them;
//  * the first call on a device looks the array's device address up (cudaGetSymbolAddress,
//    with that device current).  That one call should be made before any stream capture
//    begins; later calls only launch kernels.
constexpr uint32_t NOALLOC_MAX_ROWS = 1u << 21;   // 2,097,152 rows
static __device__ __align__(256) uint32_t g_noalloc_scratch[MAX_CHUNKS + NOALLOC_MAX_ROWS];

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
uint32_t *g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {nullptr};

// Device address of the scratch array on the current device.  In host code the array's name
// is only a handle for the runtime, not a pointer a kernel could use.
uint32_t *noalloc_scratch_address() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        set_status(BPL_ERR_CUDA, "no-allocation entry point: cannot identify the current device");
        return nullptr;
    }
    uint32_t *p = __atomic_load_n(&g_noalloc_ptr[dev], __ATOMIC_ACQUIRE);
    if (p != nullptr) return p;
    void *addr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
    if (e != cudaSuccess || addr == nullptr) {
        set_status(BPL_ERR_CUDA, e != cudaSuccess ? cudaGetErrorString(e) : "cudaGetSymbolAddress returned null");
        return nullptr;
    }
    // a racing first call on another host thread stores the same address
    __atomic_store_n(&g_noalloc_ptr[dev], static_cast<uint32_t *>(addr), __ATOMIC_RELEASE);
    return static_cast<uint32_t *>(addr);
}
}  // namespace

extern "C" {

uint32_t bpl_noalloc_max_rows(void) { return NOALLOC_MAX_ROWS; }

// y = A^T events for heterogeneous float32 weights and float32 events, transpose only.
// buffers: [data f32(nse), indices u32(nse), indptr u32(n_row+1), events f32(n_row), y f32(n_col)]
// opaque : TwoUintOneBoolDescriptor{n_row, n_col, transpose = true}
void event_csr_matvec_heter_float_float_noalloc(bpl_stream_t stream, void **buffers, const char *opaque,
                                                size_t opaque_len) {
    const TwoUintOneBoolDescriptor *d = unpack<TwoUintOneBoolDescriptor>(opaque, opaque_len);
    if (!d) return;
    if (!d->bool_x) {
        set_status(BPL_ERR_ARGUMENT, "the no-allocation entry point computes transpose=True only");
        return;
    }
    const uint32_t n_row = d->uint_x, n_col = d->uint_y;
    if (n_row > NOALLOC_MAX_ROWS) {
        set_status(BPL_ERR_TOO_LARGE,
                   "event_csr_matvec_heter_float_float_noalloc: more than 2097152 matrix rows; "
                   "use event_csr_matvec_heter_float_float with a workspace buffer");
        return;
    }
    if (n_col == 0) return;
    uint32_t *scratch = noalloc_scratch_address();
    if (scratch == nullptr) return;
    const float *data = static_cast<const float *>(buffers[0]);
    const uint32_t *indices = static_cast<const uint32_t *>(buffers[1]);
    const uint32_t *indptr = static_cast<const uint32_t *>(buffers[2]);
    const float *events = static_cast<const float *>(buffers[3]);
    float *y = static_cast<float *>(buffers[4]);
    uint32_t *counts = scratch, *ids = scratch + MAX_CHUNKS;

    const ScanPlan p = plan_scan(n_row);
    const uint64_t zero_blocks = (static_cast<uint64_t>(n_col) + SCAN_TILE - 1) / SCAN_TILE;
    const uint64_t zero_cap = static_cast<uint64_t>(sm_count()) * 8;
    const uint32_t scan_grid = static_cast<uint32_t>(
        max(static_cast<uint64_t>(p.n_chunks), min(zero_blocks, zero_cap)));
    scan_events_kernel<float, float><<<scan_grid, SCAN_THREADS, 0, stream>>>(
        events, n_row, p.chunk, p.n_chunks, y, n_col, counts, ids);
    if (!launch_ok() || n_row == 0) return;
    const int grid = persistent_blocks(4, static_cast<uint64_t>(n_row) * 16);
    if (aligned16(indices) && aligned16(data))
        row_scatter_kernel<float, false, true, true><<<grid, ROW_THREADS, 0, stream>>>(
            indices, indptr, data, nullptr, n_row, p.chunk, p.n_chunks, counts, ids, y);
    else
        row_scatter_kernel<float, false, true, false><<<grid, ROW_THREADS, 0, stream>>>(
            indices, indptr, data, nullptr, n_row, p.chunk, p.n_chunks, counts, ids, y);
    launch_ok();
}

}  // extern "C"

// ------------------------------------------------------------------------------------------
// Transposed event product driven by a ready-made spike list (no counterpart in the reference)
// ------------------------------------------------------------------------------------------
// The scatter half of event_csr_matvec_heter_float_* on its own, for callers that already hold the
// compacted spike list in the layout of the workspace (counts[1024], then row ids in 4096-entry chunk
// segments): the multi-GPU exchange assembles exactly that on every rank.  y must be zero-filled by
// the caller (the exchange's wait does it).
//   buffers [data f32(nse), indices u32(nse), indptr u32(n_row + 1), list u32, y f32(n_col)]
//   opaque  TripleSizeDescriptor{n_row, n_col, n_chunks}
extern "C" void event_csr_matvec_list_heter_float(bpl_stream_t stream, void **buffers, const char *opaque,
                                                  size_t opaque_len) {
    struct Triple { unsigned int n_row, n_col, n_chunks; };
    const Triple *d = unpack<Triple>(opaque, opaque_len);
    if (!d) return;
    if (d->n_chunks > static_cast<unsigned int>(MAX_CHUNKS)) {
        set_status(BPL_ERR_ARGUMENT, "spike list: more than 1024 chunks");
        return;
    }
    if (d->n_row == 0 || d->n_col == 0 || d->n_chunks == 0) return;
    const float *data = static_cast<const float *>(buffers[0]);
    const uint32_t *indices = static_cast<const uint32_t *>(buffers[1]);
    const uint32_t *indptr = static_cast<const uint32_t *>(buffers[2]);
    const uint32_t *list = static_cast<const uint32_t *>(buffers[3]);
    float *y = static_cast<float *>(buffers[4]);
    const int grid = persistent_blocks(4, static_cast<uint64_t>(d->n_row) * 16);
    if (profile_before()) cudaEventRecord(profile_before(), stream);
    // behind lif_exp_step or another of these a dependent launch: its blocks are there when the list is (they wait for it)
    const cudaError_t e = launch_dependent(
        aligned16(indices) && aligned16(data) ? row_scatter_kernel<float, false, true, true, true>
                                              : row_scatter_kernel<float, false, true, false, true>,
        dim3(grid), dim3(ROW_THREADS), 0, stream, indices, indptr, data, static_cast<const float *>(nullptr), d->n_row,
        static_cast<uint32_t>(SCAN_TILE), d->n_chunks, list, list + MAX_CHUNKS, y);
    if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
    if (profile_after()) cudaEventRecord(profile_after(), stream);
    launch_ok();
}
