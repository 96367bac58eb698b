// Just-in-time connectivity products for sm_100a: the matrix is never stored, every row
// (or column) regenerates its synapses from the stream `seed + index`.
//   gpu_matvec{,_atomic}_prob_*_v2        replaces lib/gpu_jitconn_matvec{,_atomic}.cu
//   gpu_event_matvec{,_atomic}_prob_*_v2  replaces lib/gpu_jitconn_event_matvec{,_atomic}.cu
//   gpu_matmat_prob_prob_*_v1             replaces lib/gpu_jitconn_matmat.cu
//
// The generator scheme and the walk along a stream: jit_stream.cuh.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "abi.h"
#include "common.cuh"
#include "jit_stream.cuh"

namespace bpl {
namespace {

constexpr int JIT_THREADS = 256;

// Version 'v1' of the dense-vector product: a Bernoulli test per (row, column) instead of the
// geometric skip, `conn_prob` being the raw probability (lib/gpu_jitconn_matvec.cu:10-54, :141-187,
// :284-331).  One `curand_uniform` per column, the weight drawn only on a connection; a different
// random matrix from 'v2'.  The input vector is staged through shared memory tile by tile as in the
// reference (plus the barrier the reference omits before a tile is overwritten).
template<typename T, int KIND>
__global__ void __launch_bounds__(JIT_THREADS)
jit_rows_dense_v1_kernel(const T *__restrict__ vector, const unsigned int seed, const double conn_prob,
                         const double w1, const double w2, const unsigned int num_row,
                         const unsigned int num_col, T *__restrict__ out) {
    __shared__ T tile[JIT_THREADS];
    const unsigned int idx = threadIdx.x;
    const unsigned int row_i = blockIdx.x * blockDim.x + idx;
    curandState state;
    curand_init(seed + row_i, 0, 0, &state);
    T sum = 0;
    for (unsigned int c0 = 0, n_tile; c0 < num_col; c0 += n_tile) {
        n_tile = min(static_cast<unsigned int>(JIT_THREADS), num_col - c0);
        if (idx < n_tile) tile[idx] = vector[c0 + idx];
        __syncthreads();
        for (unsigned int sh_i = 0; sh_i < n_tile; ++sh_i) {
            if (curand_uniform(&state) < conn_prob) {
                if (KIND == W_HOMO) sum += tile[sh_i];
                else if (KIND == W_UNIFORM) sum += tile[sh_i] * (curand_uniform(&state) * w2 + w1);
                else sum += tile[sh_i] * (curand_normal(&state) * w2 + w1);
            }
        }
        __syncthreads();
    }
    if (row_i < num_row) out[row_i] = sum;
}

// ------------------------------------------------------------------------------------------
// Row-parallel (outdim_parallel = True): one thread walks the stream of one output row.
// ------------------------------------------------------------------------------------------
// Dense input: `sum += vector[pos] (* weight)`, lib/gpu_jitconn_matvec.cu:84-112, :220-251, :363-394.  Event input:
// lib/gpu_jitconn_event_matvec.cu:81-108 (homogeneous: adds the event VALUE), :217-248, :365-396 (the weight is added
// when the event is truthy; it is drawn always, its value computed on a hit only).
//
// Where the input is read decides the rate once the walk itself is cheap (1e6 x 1e6, 1e9 connections, all rows):
//   FROM_GLOBAL  a gather through L1: one 128-byte line per clock and SM whatever is used of it, 3.2 ms
//   FROM_MASK    events as one bit each in shared memory (1e6 inputs = 125 KB): truthiness is all that is needed.  A hit
//                leaves its raw draws in a queue of its thread (shared memory); the weights are computed when a queue is
//                full, by all threads of the warp together, instead of by one thread at a time where it hits
//   FROM_MASK_SHORT   the same with fewer connections per batch, which need shorter queues: beside long masks
//   FROM_BYTES   the same with one byte per event where they fit beside the queues: three instructions fewer per connection
//   FROM_TILES   the vector in shared memory, in as few tiles as fit (58,000 floats each).  Positions ascend along a
//                stream, so all streams of a block cross one tile together; a batch that straddles the end of a tile is
//                simply looked at again in the next one, where the other positions fall into range.
// A hit (the top bit of `hit`) leaves its draws at `next`, which moves on.  One comparison for both, no branch.
__device__ __forceinline__ void push_if(const uint32_t hit, uint32_t &next, const uint32_t x, const uint32_t step) {
    asm volatile("{ .reg .pred q; setp.lt.s32 q, %1, 0; @q st.shared.u32 [%0], %2; @q add.u32 %0, %0, %3; }"
                 : "+r"(next) : "r"(hit), "r"(x), "r"(step) : "memory");
}
// (`seconds`: one bit per hit, the last one lowest)
__device__ __forceinline__ void push_pair_if(const bool second, const uint32_t hit, uint32_t &next, const uint32_t x, const uint32_t y,
                                             const uint32_t step, uint32_t &seconds) {
    if (second)
        asm volatile("{ .reg .pred q; setp.lt.s32 q, %2, 0; @q st.shared.v2.u32 [%0], {%3, %4}; @q add.u32 %0, %0, %5; @q mad.lo.u32 %1, %1, 2, 1; }"
                     : "+r"(next), "+r"(seconds) : "r"(hit), "r"(x), "r"(y), "r"(step) : "memory");
    else
        asm volatile("{ .reg .pred q; setp.lt.s32 q, %2, 0; @q st.shared.v2.u32 [%0], {%3, %4}; @q add.u32 %0, %0, %5; @q add.u32 %1, %1, %1; }"
                     : "+r"(next), "+r"(seconds) : "r"(hit), "r"(x), "r"(y), "r"(step) : "memory");
}

enum { FROM_GLOBAL = 0, FROM_MASK = 1, FROM_TILES = 2, FROM_BYTES = 3, FROM_MASK_SHORT = 4 };

constexpr int WALK_THREADS = 1024;                          // per block with shared memory, one block per SM
constexpr int GATHER_THREADS = 256;                         // at most, per block without
constexpr unsigned int WALK_SMEM = 227u * 1024u;            // all that a block can have
constexpr unsigned int MASK_MAX_BITS = 200u * 1024u * 8u;   // the rest of it: the queues of hits

// Connections that a walk over truths takes at a time.  (Uniform weights, 1e9 connections: 1517 us with 5, 1392 with 8, 1420
// with 10, where the registers of 1024 threads run out; normal 1669 with 4, 1530 with 8.)
// A queue has one slot more than a batch at least.  Pairs of draws (normal) are 8 bytes, and from 1.26e6 events on the mask leaves
// room for fewer than 1024 threads with nine slots: batches of 4 with six.  (Normal weights, p = 0.0005, 2 % of the events, batches of
// 8 and of 4: 300,000 rows, 1.28e6 events 458, 375 us; 1.47e6 592, 480; 1.64e6 761, 600; 1e6 rows, 1.35e6 events 1283, 1222; 1.64e6
// 2138, 1816.  With five slots instead of six: 1e6 rows, 1.54e6 events, 1545 and 1461.)
constexpr int TRUTH_BATCH = 8, TRUTH_BATCH_SHORT = 4, SLOTS_SHORT = 6;
// and a walk over tiles (homogeneous weights, 100,000 streams of 400: 155 us with 5, 149 with 8; uniform and normal: 2 % and 1 %
// faster with 6 than with 5 and 4)
template<int KIND> constexpr int TILE_BATCH = KIND == W_HOMO ? 8 : 6;
__host__ __device__ constexpr unsigned int queue_slot_bytes(int kind) { return kind == W_NORMAL ? 8u : 4u; }
// shared memory of the events, as bits or bytes
__host__ __device__ constexpr unsigned int truth_bytes(unsigned int n, bool bytes) { return ((bytes ? n : (n + 7u) >> 3) + 7u) & ~7u; }

// The rows (columns) of a block: equal shares, so that no SM is left with a last wave of its own.  They are counted from the
// first: their numbers go up to 2^32 - 1, where a step of a block's threads would wrap.
struct Share {
    unsigned int begin, count;
    __device__ __forceinline__ explicit Share(unsigned int n) {
        begin = static_cast<unsigned int>(static_cast<unsigned long long>(n) * blockIdx.x / gridDim.x);
        count = static_cast<unsigned int>(static_cast<unsigned long long>(n) * (blockIdx.x + 1ull) / gridDim.x) - begin;
    }
};

// Elements [first, first + count) of `src` into shared memory, by the whole block.
template<typename T>
__device__ __forceinline__ void load_tile(T *tile, const T *__restrict__ src, const unsigned int first, const unsigned int count) {
    constexpr unsigned int PER = 16 / sizeof(T);
    const T *p = src + first;
    const unsigned int n_vec = (reinterpret_cast<uintptr_t>(p) & 15u) == 0 ? count / PER : 0u;
#pragma unroll 4
    for (unsigned int i = threadIdx.x; i < n_vec; i += blockDim.x)
        reinterpret_cast<uint4 *>(tile)[i] = reinterpret_cast<const uint4 *>(p)[i];
    for (unsigned int i = n_vec * PER + threadIdx.x; i < count; i += blockDim.x) tile[i] = p[i];
}

// One byte per event, 0 or -1, by the whole block.
template<typename E>
__device__ __forceinline__ void event_bytes(const E *__restrict__ in, const unsigned int n, unsigned char *bytes) {
    constexpr unsigned int PER = 16 / sizeof(E);
    const unsigned int whole = aligned16_device(in) ? n / PER : 0u;
#pragma unroll 4
    for (unsigned int i = threadIdx.x; i < whole; i += blockDim.x) {
        const uint4 raw = *reinterpret_cast<const uint4 *>(in + i * PER);
        const E *e = reinterpret_cast<const E *>(&raw);
        uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (unsigned int k = 0; k < PER; ++k) w[k / 4] |= (is_event(e[k]) ? 0xffu : 0u) << (8u * (k % 4));
        if (PER == 16) reinterpret_cast<uint4 *>(bytes)[i] = make_uint4(w[0], w[1], w[2], w[3]);
        else if (PER == 4) reinterpret_cast<uint32_t *>(bytes)[i] = w[0];
        else reinterpret_cast<uint16_t *>(bytes)[i] = static_cast<uint16_t>(w[0]);
    }
    for (unsigned int i = whole * PER + threadIdx.x; i < n; i += blockDim.x) bytes[i] = is_event(in[i]) ? 0xff : 0;
}

template<typename T, typename E, int KIND, bool EVENT, int FROM, bool QUICK>
__global__ void __launch_bounds__(FROM == FROM_GLOBAL ? GATHER_THREADS : WALK_THREADS)
jit_rows_kernel(const E *__restrict__ in, const unsigned int seed, const GapParams gp, const double w1, const double w2,
                const unsigned int num_row, const unsigned int num_col, const unsigned int tile_len, const unsigned int slots,
                const T scale, T *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char walk_smem[];
    uint32_t *mask = reinterpret_cast<uint32_t *>(walk_smem);
    constexpr bool BYTES = FROM == FROM_BYTES, BITS = FROM == FROM_MASK || FROM == FROM_MASK_SHORT, TRUTH = BITS || BYTES;
    // the queue of hits of this thread behind the events: slots of 4 (normal: 8) bytes, `queue_step` apart
    constexpr uint32_t SLOT = queue_slot_bytes(KIND);
    const uint32_t queue_step = SLOT * blockDim.x;
    const uint32_t queue = static_cast<uint32_t>(__cvta_generic_to_shared(walk_smem)) + truth_bytes(num_col, BYTES) + SLOT * threadIdx.x;
    E *tile = reinterpret_cast<E *>(walk_smem);
    constexpr bool SUMS = TRUTH || FROM == FROM_TILES;
    constexpr int N = FROM == FROM_MASK_SHORT ? TRUTH_BATCH_SHORT : TRUTH ? TRUTH_BATCH : FROM == FROM_TILES ? TILE_BATCH<KIND> : Batch<KIND, QUICK>::N;
    const Share share(num_row);
    const bool one_tile = tile_len >= num_col;

    if (BITS) {
        pack_event_mask(in, num_col, mask);
        __syncthreads();
        // the first event of a word in its top bit: one shift by the position brings an event into the sign bit
        for (unsigned int i = threadIdx.x; i < ((num_col + 31u) >> 5); i += blockDim.x) mask[i] = __brev(mask[i]);
        __syncthreads();
    } else if (BYTES) {
        event_bytes(in, num_col, walk_smem);
        __syncthreads();
    } else if (FROM == FROM_TILES && one_tile) {
        load_tile(tile, in, 0, num_col);
        __syncthreads();
    }
    for (unsigned int from = 0; from < share.count; from += blockDim.x) {
        const unsigned int row = share.begin + from + threadIdx.x;
        const bool live = from + threadIdx.x < share.count;
        if (FROM == FROM_GLOBAL && !live) break;
        if (TRUTH && !__any_sync(FULL_MASK, live)) break;
        Xorwow s;
        s.seed(seed + row);
        Batch<KIND, QUICK, N, SUMS> b;
        unsigned int at = 0;
        T sum = 0;
        if (FROM == FROM_TILES) {
            if (live) b.draw(s, at, num_col, gp);
            for (unsigned int t0 = 0; t0 < num_col; t0 += tile_len) {
                const unsigned int len = min(tile_len, num_col - t0);
                if (!one_tile) {
                    __syncthreads();                       // everyone is done with the tile before
                    load_tile(tile, in, t0, len);
                    __syncthreads();
                }
                while (live) {
                    T w[N];
                    b.weights(w, w1, w2);
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        const unsigned int i = b.pos[j] - t0;
                        if (i < len) {
                            if (KIND == W_HOMO) sum += static_cast<T>(tile[i]);
                            else sum += (static_cast<T>(tile[i]) * w[j]);
                        }
                    }
                    if (at - t0 >= len) break;             // the batch ends behind this tile
                    b.draw(s, at, num_col, gp);
                }
            }
        } else if (TRUTH) {
            // all lanes of the warp stay in the loop until the last is done: what a lane draws behind its end is no hit
            unsigned int hits = 0;                         // homogeneous: the float sum of 0/1 events is the exact count
            uint32_t next = queue, seconds = 0;            // where the next hit goes; which hits are the second of their pair
            const uint32_t full = queue + (slots - min(slots, static_cast<unsigned int>(N) - 1u)) * queue_step;
            if (!live) at = num_col;                       // draws behind the end from the start
            auto drain = [&]() {
                uint32_t last = KIND == W_NORMAL ? (next - queue) / queue_step : 0u;
                for (uint32_t from = queue; __any_sync(FULL_MASK, from < next); from += queue_step) {
                    if (from >= next) continue;
                    if (KIND == W_UNIFORM) {
                        uint32_t x;
                        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(from) : "memory");
                        sum += uniform_weight<T>(x, w1, w2);
                    }
                    if (KIND == W_NORMAL) {
                        uint32_t x, y;
                        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(from) : "memory");
                        sum += normal_weight<T>(x, y, (seconds >> --last) & 1u, w1, w2);
                    }
                }
                next = queue;
            };
            // checked: positions may lie behind the end
            auto look = [&](auto checked) {
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    uint32_t hit = 0;                      // its top bit
                    if (BYTES) {
                        if (!checked.value || b.pos[j] < num_col) hit = static_cast<int>(reinterpret_cast<const signed char *>(walk_smem)[b.pos[j]]);
                        if (KIND == W_HOMO) hits -= hit;
                    } else {
                        uint32_t word = 0;                 // 24 bits of the position hold it: the mask has at most 2^21
                        if (!checked.value || (b.pos[j] & 0xffffffu) < num_col)
                            word = *reinterpret_cast<const uint32_t *>(walk_smem + ((b.pos[j] >> 3) & 0x1ffffcu));
                        hit = __funnelshift_l(0u, word, b.pos[j]);
                        if (KIND == W_HOMO) hits += hit >> 31;
                    }
                    if (KIND == W_UNIFORM) push_if(hit, next, b.raw[j], queue_step);
                    if (KIND == W_NORMAL) push_pair_if(j & 1, hit, next, b.raw[j & ~1], b.raw[j | 1], queue_step, seconds);
                }
                if (KIND != W_HOMO && __any_sync(FULL_MASK, next >= full)) drain();
            };
            auto draw = [&]() {
                b.template draw<BITS>(s, at, num_col, gp);
                if (BYTES) at = min(at, num_col);
            };
            draw();
            while (__all_sync(FULL_MASK, at < num_col)) {
                look(std::false_type());
                draw();
            }
            look(std::true_type());
            while (__any_sync(FULL_MASK, at < num_col)) {
                draw();
                look(std::true_type());
            }
            if (KIND == W_HOMO) sum = static_cast<T>(hits);
            else drain();
        } else {
            do {
                b.draw(s, at, num_col, gp);
                E v[N];
#pragma unroll
                for (int j = 0; j < N; ++j) v[j] = b.pos[j] < num_col ? in[b.pos[j]] : E(0);
                T w[N];
                if (!EVENT) b.weights(w, w1, w2);
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    if (b.pos[j] >= num_col) continue;
                    if (KIND == W_HOMO) sum += static_cast<T>(v[j]);
                    else if (!EVENT) sum += (static_cast<T>(v[j]) * w[j]);
                    else if (is_event(v[j])) {
                        if (KIND == W_UNIFORM) sum += uniform_weight<T>(b.raw[j], w1, w2);
                        if (KIND == W_NORMAL) sum += normal_weight<T>(b.raw[j & ~1], b.raw[j | 1], j & 1, w1, w2);
                    }
                }
            } while (at < num_col);
        }
        if (live) out[row] = KIND == W_HOMO ? sum * scale : sum;
    }
}

// Few rows (jit_stream.cuh, GroupStep): eight lanes per row, the input gathered from global memory while the next step is
// drawn.  The sum takes the connections in stream order, as one lane would.  3000 rows of 200000 columns, p = 0.002, 3 %
// of the events set: uniform 49 -> 35 us, normal 55 -> 41; dense, 1500 rows of 20000, p = 0.01: 19 -> 10.5, 21 -> 14.5,
// 27 -> 18 (homogeneous, uniform, normal).
constexpr int GROUP_THREADS = 128;

template<typename T, typename E, int KIND, bool EVENT>
__global__ void __launch_bounds__(GROUP_THREADS)
jit_rows_group_kernel(const E *__restrict__ in, const unsigned int seed, const GapParams gp, const double w1, const double w2,
                      const unsigned int num_row, const unsigned int num_col, const T scale, T *__restrict__ out) {
    const unsigned int lane = threadIdx.x & 31u, sub = lane & (GROUP - 1u);
    const unsigned int row = blockIdx.x * (GROUP_THREADS / GROUP) + threadIdx.x / GROUP;
    const bool live = row < num_row;
    if (!__any_sync(FULL_MASK, live)) return;
    Xorwow s;
    s.seed(seed + row);
    GroupStep<KIND> now, next;
    unsigned int at = live ? 0u : num_col;                 // (a group without a row is at the end from the start)
    T sum = 0;
    now.draw(s, at, num_col, sub, gp);
    bool more = true;
    while (more) {
        E v = E(0);
        const bool inside = live && now.pos < num_col;
        if (inside) v = in[now.pos];
        more = __any_sync(FULL_MASK, at < num_col);
        if (more) next.draw(s, at, num_col, sub, gp);
        // (rounded as by one lane: a product and its sum in one operation)
        const bool has = inside && (!EVENT || is_event(v));
        const T x = has && !EVENT ? static_cast<T>(v) : T(0);
        const T w = has && KIND != W_HOMO ? now.template weight<T>(sub, w1, w2) : T(1);
        unsigned int mine = (__ballot_sync(FULL_MASK, has) >> (lane & ~(GROUP - 1u))) & ((1u << GROUP) - 1u);
        if (EVENT) {
            while (__any_sync(FULL_MASK, mine != 0u)) {
                const T t = __shfl_sync(FULL_MASK, w, mine ? __ffs(mine) - 1 : 0, GROUP);
                if (mine) sum += t;
                mine &= mine - 1u;
            }
        } else {
#pragma unroll
            for (int j = 0; j < GROUP; ++j) {
                const T t = __shfl_sync(FULL_MASK, x, j, GROUP);
                const T u = KIND == W_HOMO ? T(1) : __shfl_sync(FULL_MASK, w, j, GROUP);
                if ((mine >> j) & 1u) sum += t * u;
            }
        }
        now = next;
    }
    if (live && sub == 0) out[row] = KIND == W_HOMO ? sum * scale : sum;
}

// ------------------------------------------------------------------------------------------
// Column-parallel (outdim_parallel = False): one thread walks the stream of one input column and scatters.
// ------------------------------------------------------------------------------------------
// Dense input: lib/gpu_jitconn_matvec_atomic.cu:27-52, :82-110, :143-171.  The L2 of a B200 retires about 155 G scattered
// reductions per second (0.55 per clock and SM); an addition in shared memory runs six times faster.  TILES: a tile of the
// output lives in shared memory while all columns of the block cross it (positions ascend along a stream), and is then
// added to the zero-filled output with 16-byte reductions.
template<typename T, int KIND, bool TILES, bool QUICK>
__global__ void __launch_bounds__(TILES ? WALK_THREADS : GATHER_THREADS)
jit_cols_kernel(const T *__restrict__ vector, const unsigned int seed, const GapParams gp, const double w1, const double w2,
                const unsigned int num_row, const unsigned int num_col, const unsigned int tile_len, const T scale,
                T *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char walk_smem[];
    T *tile = reinterpret_cast<T *>(walk_smem);
    constexpr int N = TILES ? TILE_BATCH<KIND> : Batch<KIND, QUICK>::N;
    const Share share(num_col);
    for (unsigned int from = 0; from < share.count; from += blockDim.x) {
        const unsigned int col = share.begin + from + threadIdx.x;
        const bool live = from + threadIdx.x < share.count;
        if (!TILES && !live) break;
        Xorwow s;
        s.seed(seed + col);
        Batch<KIND, QUICK, N, TILES> b;
        unsigned int at = 0;
        T v = live ? vector[col] : T(0);
        if (KIND == W_HOMO) v = v * scale;
        if (live) b.draw(s, at, num_row, gp);
        for (unsigned int t0 = 0; t0 < num_row; t0 += tile_len) {
            const unsigned int len = min(tile_len, num_row - t0);
            if (TILES) {
                for (unsigned int i = threadIdx.x; i < len; i += blockDim.x) tile[i] = T(0);
                __syncthreads();
            }
            while (live) {
                T w[N];
                b.weights(w, w1, w2);
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const unsigned int i = b.pos[j] - t0;
                    if (i < len) {
                        const T add = KIND == W_HOMO ? v : v * w[j];
                        if (TILES) atomicAdd(tile + i, add);
                        else red_add(out + i, add);
                    }
                }
                if (at - t0 >= len) break;
                b.draw(s, at, num_row, gp);
            }
            if (TILES) {
                __syncthreads();
                add_sums(tile, out + t0, len, blockIdx.x, gridDim.x);
                __syncthreads();
            }
        }
    }
}

// Few columns: eight lanes each.  30000 rows, 3000 columns, p = 0.01: uniform 32 -> 24 us, normal 46 -> 26.
template<typename T, int KIND>
__device__ __forceinline__ void scatter_group(const unsigned int stream_seed, const bool live, const T v,
                                              const unsigned int num_row, const GapParams &gp, const double w1,
                                              const double w2, T *__restrict__ out) {
    const unsigned int sub = threadIdx.x & (GROUP - 1u);
    Xorwow s;
    s.seed(stream_seed);
    GroupStep<KIND> step;
    unsigned int at = live ? 0u : num_row;
    do {
        step.draw(s, at, num_row, sub, gp);
        if (live && step.pos < num_row) red_add(out + step.pos, KIND == W_HOMO ? v : v * step.template weight<T>(sub, w1, w2));
    } while (__any_sync(FULL_MASK, at < num_row));
}

template<typename T, int KIND>
__global__ void __launch_bounds__(GROUP_THREADS)
jit_cols_group_kernel(const T *__restrict__ vector, const unsigned int seed, const GapParams gp, const double w1, const double w2,
                      const unsigned int num_row, const unsigned int num_col, const T scale, T *__restrict__ out) {
    const unsigned int col = blockIdx.x * (GROUP_THREADS / GROUP) + threadIdx.x / GROUP;
    const bool live = col < num_col;
    T v = live ? vector[col] : T(0);
    if (KIND == W_HOMO) v = v * scale;
    scatter_group<T, KIND>(seed + col, live, v, num_row, gp, w1, w2, out);
}

// Event input: lib/gpu_jitconn_event_matvec_atomic.cu:30-58, :88-117, :150-178.  There every column walks its stream and
// only the atomicAdd is conditional; a silent column contributes nothing and its stream is private, so it is skipped
// here.  Each block compacts the firing columns of its chunk into shared memory and gives one thread to each of them, or eight
// lanes where there are at most `few`.  One block per SM: where four of them shared one, some ten firing columns each, give or
// take three, single blocks went the other way than their neighbours and held them up (1e6 x 1e6, p = 0.001, normal weights,
// 0.5 % firing: 125 us, now 77; 300,000 columns, 100,000 rows, p = 0.005, 0.5 %: 64, now 37).  The list has room for every
// column of the chunk, up to all of shared memory; more columns take several equal waves.  (With lists of 8192 and a second wave
// behind them, 1,250,000 columns, 2 % firing: 250 us, now 169.)
constexpr unsigned int COL_CHUNK = WALK_SMEM / sizeof(unsigned int) / 1024u * 1024u;

template<typename T>
__global__ void __launch_bounds__(256) jit_clear_kernel(T *__restrict__ out, const unsigned int n) {
    pdl_launch_dependents();
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull) out[i] = T(0);
}

template<typename T, typename E, int KIND, bool QUICK>
__global__ void __launch_bounds__(WALK_THREADS)
jit_cols_event_kernel(const E *__restrict__ events, const unsigned int seed, const GapParams gp, const double w1,
                      const double w2, const unsigned int num_row, const unsigned int num_col, const unsigned int chunk,
                      const unsigned int few, T *__restrict__ out) {
    extern __shared__ unsigned int active[];               // [chunk]
    __shared__ unsigned int n_active;
    constexpr int N = Batch<KIND, QUICK>::N;
    constexpr unsigned int PER = 16 / sizeof(E);           // events per load; chunk is a multiple of 16
    if (threadIdx.x == 0) n_active = 0;
    __syncthreads();
    // (counted from the first column of the chunk: numbers of columns go up to 2^32 - 1)
    const unsigned int base = blockIdx.x * chunk, count = min(chunk, num_col - base);
    const E *mine = events + base;
    const unsigned int whole = aligned16_device(events) ? count / PER * PER : 0u;
    for (unsigned int i = threadIdx.x * PER; i < whole; i += blockDim.x * PER) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4 *>(mine + i));
        const E *e = reinterpret_cast<const E *>(&raw);
        if ((raw.x | raw.y | raw.z | raw.w) == 0u) continue;
#pragma unroll
        for (unsigned int k = 0; k < PER; ++k)
            if (is_event(e[k])) active[atomicAdd(&n_active, 1u)] = base + i + k;
    }
    for (unsigned int i = whole + threadIdx.x; i < count; i += blockDim.x)
        if (is_event(mine[i])) active[atomicAdd(&n_active, 1u)] = base + i;
    __syncthreads();
    pdl_wait();                                            // the output is zero
    const unsigned int n = n_active, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    if (QUICK && n <= few) {
        // (One round, unless the output is short.  Inside the loop its walk is the slower one: 89,033 rows, 52 columns firing, p = 0.08,
        // homogeneous 211 us and 199, uniform 275 and 264, normal 363 and 356.)
        constexpr unsigned int PER_WARP = 32 / GROUP;
        unsigned int i = threadIdx.x / GROUP;
        if (n <= warps * PER_WARP) {
            if (warp * PER_WARP < n) scatter_group<T, KIND>(seed + (i < n ? active[i] : 0u), i < n, T(1), num_row, gp, w1, w2, out);
            return;
        }
        for (unsigned int i0 = warp * PER_WARP; i0 < n; i0 += warps * PER_WARP, i += warps * PER_WARP)
            scatter_group<T, KIND>(seed + (i < n ? active[i] : 0u), i < n, T(1), num_row, gp, w1, w2, out);
        return;
    }
    // As few warps as hold the columns, as many for each scheduler: a walk issues for all lanes of its warp.
    const unsigned int per_warp = (n + 4u * ((n + 127u) / 128u) - 1u) / max(4u * ((n + 127u) / 128u), 1u), lane = threadIdx.x & 31u;
    if (lane >= per_warp) return;
    for (unsigned int i = warp * per_warp + lane; i < n; i += warps * per_warp) {
        Xorwow s;
        s.seed(seed + active[i]);
        Batch<KIND, QUICK> b;
        unsigned int at = 0;
        do {
            b.draw(s, at, num_row, gp);
            T w[N];
            b.weights(w, w1, w2);
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (b.pos[j] < num_row) red_add(out + b.pos[j], KIND == W_HOMO ? T(1) : w[j]);
        } while (at < num_row);
    }
}

// ------------------------------------------------------------------------------------------
// Y = X @ M, M just-in-time with one stream per output column
// (lib/gpu_jitconn_matmat.cu:236-276 normal, :321-361 uniform).
// ------------------------------------------------------------------------------------------
// A thread owns one output column and 32 rows of X, as in the reference, and accumulates
// `sum += X[row][pos] * w` in synapse order (same bits).  What changes is where X comes from: the
// reference reads X[(m_i + i) * k + pos] from global memory, one 32-byte sector per float; here a
// K-tile of the 32 rows is staged TRANSPOSED in shared memory ([k][row]), so a synapse reads 32
// consecutive floats with 128-bit shared loads.  The lanes of a warp read different tile rows
// (their synapses sit at unrelated positions), which would put them on the same banks; instead
// lane l reads the 16-byte chunks of its row in the rotated order (c + l) mod CHUNKS, so the
// eight lanes served together always touch eight different chunks.  The accumulator register
// (c, i) of lane l therefore belongs to row ((c + l) mod CHUNKS) * PER_CHUNK + i; the rotation is
// undone when Y is written.
constexpr int MM_THREADS = 512;
constexpr int MM_ROWS = 32;

template<typename T> struct MMTile;
template<> struct MMTile<float> { static constexpr int KT = 512; static constexpr int CHUNKS = 8; };    // 64 KB
template<> struct MMTile<double> { static constexpr int KT = 256; static constexpr int CHUNKS = 16; };  // 64 KB

// Stages X[m_i .. m_i+31][k0 .. k0+KT) transposed into `tile` ([KT][MM_ROWS]): lane = row of X, so the 32 stores of
// a warp go to 32 consecutive words (no bank conflict); each lane reads VEC consecutive k from its own row (the
// other half of a touched sector is picked up from L1 by the next iteration).  Rows and columns past the matrix read
// as zero.
template<typename T, int KT>
__device__ __forceinline__ void mm_stage_tile(T *tile, const T *__restrict__ X, const unsigned int m_i,
                                              const unsigned int m, const unsigned int k, const unsigned int k0,
                                              const bool vec_ok, const unsigned int lane, const unsigned int warp) {
    constexpr int VEC = 16 / sizeof(T);
    const unsigned int r = lane;
    const bool row_ok = m_i + r < m;
    const T *src = X + static_cast<size_t>(m_i + r) * k + k0;
    for (unsigned int kk = warp * VEC; kk < KT; kk += (MM_THREADS / 32) * VEC) {
        T v[VEC];
        if (vec_ok && row_ok && k0 + kk + VEC <= k) {
            const uint4 u = *reinterpret_cast<const uint4 *>(src + kk);
            *reinterpret_cast<uint4 *>(v) = u;
        } else {
#pragma unroll
            for (int q = 0; q < VEC; ++q) v[q] = (row_ok && k0 + kk + q < k) ? src[kk + q] : T(0);
        }
#pragma unroll
        for (int q = 0; q < VEC; ++q) tile[(kk + q) * MM_ROWS + r] = v[q];
    }
}

template<typename T, int KIND>
__global__ void __launch_bounds__(MM_THREADS, (sizeof(T) == 8 ? 1 : 2))     // 32 double sums: more than 64 registers
jit_matmat_kernel(const T *__restrict__ X, const unsigned int seed, const GapParams gp, const double w1,
                  const double w2, const unsigned int m, const unsigned int k, const unsigned int n,
                  T *__restrict__ Y) {
    constexpr int KT = MMTile<T>::KT, CHUNKS = MMTile<T>::CHUNKS, PER_CHUNK = 16 / sizeof(T);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *tile = reinterpret_cast<T *>(smem_raw);   // [KT][MM_ROWS]

    const unsigned long long n_i64 = static_cast<unsigned long long>(blockIdx.x) * MM_THREADS + threadIdx.x;
    const bool live = n_i64 < n;
    const unsigned int n_i = static_cast<unsigned int>(n_i64);
    const unsigned int m_i = blockIdx.y * MM_ROWS;
    const unsigned int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool vec_ok = (k % (16 / sizeof(T)) == 0) && ((reinterpret_cast<uintptr_t>(X) & 15u) == 0);

    curandState st;
    curand_init(seed + n_i, 0, 0, &st);
    unsigned int pos = live ? next_position(0u, curand(&st), gp) : 0xffffffffu;
    T sum[MM_ROWS];
#pragma unroll
    for (int i = 0; i < MM_ROWS; ++i) sum[i] = 0;

    for (unsigned int k0 = 0; k0 < k; k0 += KT) {
        mm_stage_tile<T, KT>(tile, X, m_i, m, k, k0, vec_ok, lane, warp);
        __syncthreads();
        const unsigned int k_end = min(k0 + KT, k);
        while (pos < k_end) {
            T rand;
            if (KIND == W_NORMAL) rand = (T) (curand_normal(&st) * w2 + w1);
            else rand = (T) (curand_uniform(&st) * w2 + w1);
            const unsigned int kk = pos - k0;
            const T *row = tile + kk * MM_ROWS;
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                const unsigned int chunk = (c + lane) & (CHUNKS - 1);
                if (sizeof(T) == 4) {
                    const float4 x = *reinterpret_cast<const float4 *>(row + chunk * PER_CHUNK);
                    sum[c * 4 + 0] += (x.x * rand);
                    sum[c * 4 + 1] += (x.y * rand);
                    sum[c * 4 + 2] += (x.z * rand);
                    sum[c * 4 + 3] += (x.w * rand);
                } else {
                    const double2 x = *reinterpret_cast<const double2 *>(row + chunk * PER_CHUNK);
                    sum[c * 2 + 0] += (x.x * rand);
                    sum[c * 2 + 1] += (x.y * rand);
                }
            }
            pos = next_position(pos, curand(&st), gp);
        }
        __syncthreads();
    }
    if (live) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const unsigned int chunk = (c + lane) & (CHUNKS - 1);
#pragma unroll
            for (int i = 0; i < PER_CHUNK; ++i) {
                const unsigned int row = m_i + chunk * PER_CHUNK + i;
                if (row < m) Y[static_cast<size_t>(row) * n + n_i] = sum[c * PER_CHUNK + i];
            }
        }
    }
}

// Tests: how many of all 2^32 draws have another gap than the reference's expression gives.
__global__ void __launch_bounds__(256) jit_gap_mismatches_kernel(const GapParams g, unsigned long long *__restrict__ count) {
    unsigned long long wrong = 0;
    for (unsigned long long x = blockIdx.x * 256ull + threadIdx.x; x < 1ull << 32; x += gridDim.x * 256ull) {
        const float u = _curand_uniform(static_cast<uint32_t>(x));
        wrong += gap_of(static_cast<uint32_t>(x), g) != static_cast<int>(ceil(log(u) / g.log_p));
    }
    for (int o = 16; o > 0; o >>= 1) wrong += __shfl_xor_sync(FULL_MASK, wrong, o);
    if ((threadIdx.x & 31u) == 0 && wrong != 0) atomicAdd(count, wrong);
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
struct JitArgs {
    unsigned int n_row, n_col, seed;
    double log_p, w1, w2;
};

template<int KIND>
inline bool unpack_jit(const char *opaque, size_t opaque_len, JitArgs &a) {
    if (KIND == W_HOMO) {
        const JITConnProbHomoDescriptor *d = unpack<JITConnProbHomoDescriptor>(opaque, opaque_len);
        if (!d) return false;
        a = JitArgs{d->n_row, d->n_col, d->seed, d->prob, 0.0, 0.0};
    } else {
        const JITConnProbWeightedDescriptor *d = unpack<JITConnProbWeightedDescriptor>(opaque, opaque_len);
        if (!d) return false;
        a = JitArgs{d->n_row, d->n_col, d->seed, d->prob, d->w1, d->w2};
    }
    return true;
}

inline unsigned int blocks_for(unsigned int n, unsigned int per_block) {
    return static_cast<unsigned int>((static_cast<unsigned long long>(n) + per_block - 1) / per_block);
}

template<typename T, typename E>
struct JitCall {
    cudaStream_t stream;
    const E *in;
    T *out;
    JitArgs a;
    T scale;       // homogeneous weights: factor of the sums (rows) or of the input (columns)
};

// One block per SM (fewer when there is not a warp of streams for each) and the threads that split its streams into
// equal waves.
struct WalkGrid {
    unsigned int blocks, waves, threads;
    WalkGrid(unsigned int n, unsigned int at_least) {
        blocks = std::min(static_cast<unsigned int>(sm_count()), blocks_for(n, 32));
        const unsigned int per_block = blocks_for(n, blocks);
        waves = blocks_for(per_block, WALK_THREADS);
        threads = std::max(blocks_for(blocks_for(per_block, waves), 32) * 32u, at_least);
    }
    // no more threads than `most` (a multiple of 32)
    void at_most(unsigned int n, unsigned int most) {
        if (threads <= most) return;
        const unsigned int per_block = blocks_for(n, blocks);
        waves = blocks_for(per_block, most);
        threads = std::min(most, std::max(512u, blocks_for(blocks_for(per_block, waves), 32) * 32u));
    }
};

// Tiles of equal length, a multiple of 32 elements, as few as fit.
inline unsigned int tile_length(unsigned int n, size_t elem) {
    const unsigned int tiles = std::max(1u, blocks_for(n, static_cast<unsigned int>(WALK_SMEM / elem) & ~31u));
    return blocks_for(blocks_for(n, tiles), 32) * 32u;
}

// Streams per SM up to which eight lanes walk one: beyond, the extra instructions no longer fit the idle issue slots.  One
// lane per row takes dense homogeneous and uniform connections fast enough that the line lies lower (3000 rows, 100000
// columns, p = 0.1, uniform: 441 us by one lane, 497 by eight; normal: 922 and 652), and an event bit of a homogeneous one
// always (2300 rows, 20000 columns, p = 0.2: 133 and 172).
template<int KIND, bool EVENT>
constexpr int GROUP_ROWS = EVENT ? (KIND == W_HOMO ? 0 : 60) : KIND == W_NORMAL ? 40 : 16;
// Columns: reductions into a short output meet at the same addresses, where sums in shared memory are the better ones sooner
// (9000 columns, p = 0.1, uniform: 3000 rows 65 us by one lane and 110 by eight, 30000 rows 468 and 357).
constexpr unsigned int GROUP_LONG = 16384;
constexpr int GROUP_COLS = 32, GROUP_COLS_LONG = 60;
// Firing columns: at 30, 47 and 68 per SM of 1000 connections each, by eight lanes 77, 100 and 123 us, by one 113, 114 and 115 (normal);
// 61, 84 and 95 against 66, 68 and 80 (uniform); 47, 60 and 80 against 55, 58 and 78 (homogeneous).  A little above where both
// take the same: single blocks have more than others, and the slower of two kinds counts.
template<int KIND>
constexpr unsigned int GROUP_EVENTS = KIND == W_NORMAL ? 72 : KIND == W_UNIFORM ? 42 : 60;

// Rules in clocks of one SM.  A gather through L1 takes one clock per connection.  Filling shared memory reads the whole
// input per block, at about 56 bytes per clock, after a start of some 2000 clocks; a vector in several tiles is read
// again for every wave of streams.
template<typename T, typename E, int KIND, bool EVENT>
void jit_rows(const JitCall<T, E> &c) {
    const JitArgs &a = c.a;
    const GapParams gp = gap_params(a.log_p, a.n_col);
    const double gathers = static_cast<double>(a.n_row) * a.n_col * -std::expm1(a.log_p) / sm_count();
    constexpr bool TRUTH_ONLY = EVENT && (KIND != W_HOMO || sizeof(E) == 1);
    if constexpr (GROUP_ROWS<KIND, EVENT> > 0) {
        if (gp.quick && a.n_row <= static_cast<unsigned int>(GROUP_ROWS<KIND, EVENT> * sm_count())) {
            jit_rows_group_kernel<T, E, KIND, EVENT><<<blocks_for(a.n_row, GROUP_THREADS / GROUP), GROUP_THREADS, 0, c.stream>>>(
                c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, c.scale, c.out);
            launch_ok();
            return;
        }
    }
    WalkGrid g(a.n_row, 512);
    if constexpr (TRUTH_ONLY) {
        // Bytes where they leave room for queues of 12 (normal: 10) hits of 1024 threads; then bits, whose walk keeps positions
        // in 24 bits (a batch runs TRUTH_BATCH gaps, each below 23 mean ones, behind the end).  Matrices beyond are gathered from global
        // memory, which is faster for them (normal, 1e6 rows, 1.6e6 events, p = 1.2e-5, as bits in batches of 4: 236 us; gathered: 107).
        const unsigned int room = KIND == W_HOMO ? 0u : (KIND == W_UNIFORM ? 48u : 80u) * 1024u;
        const bool bytes = truth_bytes(a.n_col, true) <= WALK_SMEM - room && a.n_col <= WALK_SMEM;
        const bool bits = a.n_col <= MASK_MAX_BITS && a.n_col - TRUTH_BATCH * 23.0 / a.log_p < 16777216.0;
        if (gp.quick && (bytes || bits) && gathers > static_cast<double>(a.n_col) * sizeof(E) / 56 + 2000) {
            constexpr auto byte_kernel = jit_rows_kernel<T, E, KIND, EVENT, FROM_BYTES, true>;
            constexpr auto bit_kernel = jit_rows_kernel<T, E, KIND, EVENT, FROM_MASK, true>;
            constexpr auto short_kernel = jit_rows_kernel<T, E, KIND, EVENT, KIND == W_NORMAL ? FROM_MASK_SHORT : FROM_MASK, true>;
            // what the events leave holds the queues of hits, up to 16 slots per thread (`seconds` has 32 bits); where they do not
            // fit for all threads, for fewer, in equal waves again
            const unsigned int taken = truth_bytes(a.n_col, bytes), left = WALK_SMEM - taken, slot_bytes = queue_slot_bytes(KIND);
            unsigned int slots = 0;
            bool in_short = false;
            if (KIND != W_HOMO) {
                in_short = KIND == W_NORMAL && left < slot_bytes * (TRUTH_BATCH + 1) * g.threads;
                g.at_most(a.n_row, left / (slot_bytes * (in_short ? SLOTS_SHORT : TRUTH_BATCH + 1)) & ~31u);
                slots = std::min(16u, left / (slot_bytes * g.threads));
            }
            if (!(bytes ? allow_shared<byte_kernel>(WALK_SMEM) : in_short ? allow_shared<short_kernel>(WALK_SMEM) : allow_shared<bit_kernel>(WALK_SMEM))) {
                launch_ok();
                return;
            }
            (bytes ? byte_kernel : in_short ? short_kernel : bit_kernel)<<<g.blocks, g.threads, static_cast<size_t>(taken) + slots * slot_bytes * g.threads, c.stream>>>(
                c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, 0, slots, c.scale, c.out);
            launch_ok();
            return;
        }
    }
    if (gp.quick && !TRUTH_ONLY && (KIND == W_HOMO || !EVENT)) {
        const unsigned int len = tile_length(a.n_col, sizeof(E));
        const double loads = static_cast<double>(a.n_col) * sizeof(E) / 56 * (len >= a.n_col ? 1 : g.waves);
        if (0.75 * gathers > loads + 2000) {
            constexpr auto kernel = jit_rows_kernel<T, E, KIND, EVENT, TRUTH_ONLY ? FROM_GLOBAL : FROM_TILES, true>;
            if (!allow_shared<kernel>(WALK_SMEM)) {
                launch_ok();
                return;
            }
            kernel<<<g.blocks, g.threads, static_cast<size_t>(len) * sizeof(E), c.stream>>>(
                c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, len, 0, c.scale, c.out);
            launch_ok();
            return;
        }
    }
    // blocks small enough that every SM gets one
    const unsigned int threads = std::min(static_cast<unsigned int>(GATHER_THREADS), blocks_for(blocks_for(a.n_row, sm_count()), 32) * 32u);
    const unsigned int blocks = blocks_for(a.n_row, threads);
    if (gp.quick)
        jit_rows_kernel<T, E, KIND, EVENT, FROM_GLOBAL, true><<<blocks, threads, 0, c.stream>>>(
            c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, a.n_col, 0, c.scale, c.out);
    else
        jit_rows_kernel<T, E, KIND, EVENT, FROM_GLOBAL, false><<<blocks, threads, 0, c.stream>>>(
            c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, a.n_col, 0, c.scale, c.out);
    launch_ok();
}

// In clocks of one SM: a scattered reduction into L2 takes 1.8, an addition in shared memory 0.3; a tile costs about 0.8
// per element to clear and to flush, and to wait for its few last columns, once per wave of columns (738,704 outputs from
// 29,731 columns, 113 connections each per tile: 433 us in tiles, 282 with reductions).
template<typename T, int KIND>
void jit_cols(const JitCall<T, T> &c) {
    const JitArgs &a = c.a;
    if (cudaMemsetAsync(c.out, 0, sizeof(T) * static_cast<size_t>(a.n_row), c.stream) != cudaSuccess) {
        launch_ok();
        return;
    }
    if (a.n_col == 0) return;
    const GapParams gp = gap_params(a.log_p, a.n_row);
    const double additions = static_cast<double>(a.n_row) * a.n_col * -std::expm1(a.log_p) / sm_count();
    if (gp.quick && a.n_col <= static_cast<unsigned int>((a.n_row < GROUP_LONG ? GROUP_COLS : GROUP_COLS_LONG) * sm_count())) {
        jit_cols_group_kernel<T, KIND><<<blocks_for(a.n_col, GROUP_THREADS / GROUP), GROUP_THREADS, 0, c.stream>>>(
            c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, c.scale, c.out);
        launch_ok();
        return;
    }
    const WalkGrid g(a.n_col, 512);
    if (gp.quick && 1.8 * additions > 0.3 * (sizeof(T) / 4) * additions + 0.8 * (sizeof(T) / 4) * a.n_row * g.waves + 5000) {
        const unsigned int len = tile_length(a.n_row, sizeof(T));
        constexpr auto kernel = jit_cols_kernel<T, KIND, true, true>;
        if (!allow_shared<kernel>(WALK_SMEM)) {
                launch_ok();
                return;
            }
        kernel<<<g.blocks, g.threads, static_cast<size_t>(len) * sizeof(T), c.stream>>>(
            c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, len, c.scale, c.out);
        launch_ok();
        return;
    }
    const unsigned int threads = std::min(static_cast<unsigned int>(GATHER_THREADS), blocks_for(blocks_for(a.n_col, sm_count()), 32) * 32u);
    const unsigned int blocks = blocks_for(a.n_col, threads);
    (gp.quick ? jit_cols_kernel<T, KIND, false, true> : jit_cols_kernel<T, KIND, false, false>)<<<blocks, threads, 0, c.stream>>>(
        c.in, a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, a.n_row, c.scale, c.out);
    launch_ok();
}

template<typename T, typename E, int KIND>
void jit_cols_event(const JitCall<T, E> &c) {
    const JitArgs &a = c.a;
    if (a.n_col == 0) {                                    // (the clearing kernel lets the launch behind it start early: only with one of its own there)
        if (cudaMemsetAsync(c.out, 0, sizeof(T) * static_cast<size_t>(a.n_row), c.stream) != cudaSuccess) launch_ok();
        return;
    }
    const unsigned int sms = static_cast<unsigned int>(sm_count());
    const GapParams gp = gap_params(a.log_p, a.n_row);
    const unsigned int waves = blocks_for(a.n_col, sms * COL_CHUNK);
    const unsigned int chunk = blocks_for(blocks_for(a.n_col, sms * waves), 16) * 16u, blocks = blocks_for(a.n_col, chunk);
    const unsigned int threads = std::max(128u, std::min(static_cast<unsigned int>(WALK_THREADS), blocks_for(chunk, 4) * 32u));
    // In a short output the lanes of a warp that each walk a stream of their own meet at the same addresses; eight lanes of one
    // stream do not, but seed it and draw for it eight times, which streams of a few connections do not pay back.  3000 rows, 1e6
    // columns, 10 % firing, by eight lanes and by one, us (normal): 0.15 connections per stream 12.5, 8.2; 5 20.9, 24.6; 10 35.8, 51.3; 40 137,
    // 265; half of them firing, 3 connections 53.6, 50.4.  300,000 columns, 5 %: 5 connections 8.2, 8.2; 80 53.3, 59.5.  8000 rows, 101
    // firing columns per SM: 43.4, 37.7.
    const bool meet = a.n_row < 4096u && a.n_row * -std::expm1(a.log_p) >= 4.0;
    const unsigned int few = meet ? chunk : GROUP_EVENTS<KIND>;
    constexpr auto quick = jit_cols_event_kernel<T, E, KIND, true>, any = jit_cols_event_kernel<T, E, KIND, false>;
    if (!(gp.quick ? allow_shared<quick>(COL_CHUNK * sizeof(unsigned int)) : allow_shared<any>(COL_CHUNK * sizeof(unsigned int)))) {
        launch_ok();
        return;
    }
    // One block per SM, by its shared memory: started beside the clearing kernel, small blocks go to the SMs that it leaves first,
    // several to one.  (530,212 rows, 2 columns firing per SM, p = 0.019: homogeneous 303 us without, 274; uniform 429 and 369; normal 543
    // and 498.)
    const unsigned int smem = std::max(chunk * static_cast<unsigned int>(sizeof(unsigned int)), blocks <= sms ? WALK_SMEM / 2u : 0u);
    jit_clear_kernel<T><<<std::min(blocks_for(a.n_row, 1024), 8 * sms), 256, 0, c.stream>>>(c.out, a.n_row);
    if (!launch_ok()) return;
    const cudaError_t e = launch_dependent(gp.quick ? quick : any, dim3(blocks), dim3(threads), smem, c.stream, c.in,
                                           a.seed, gp, a.w1, a.w2, a.n_row, a.n_col, chunk, few, c.out);
    if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
}

template<typename T, int KIND, bool ROWS>
void jit_matvec_impl(cudaStream_t stream, void **buffers, const char *opaque, size_t opaque_len) {
    JitCall<T, T> c{stream, static_cast<const T *>(buffers[0]), static_cast<T *>(buffers[1]), {}, T(1)};
    if (!unpack_jit<KIND>(opaque, opaque_len, c.a) || c.a.n_row == 0) return;
    if (ROWS) jit_rows<T, T, KIND, false>(c);
    else jit_cols<T, KIND>(c);
}

// The same without a descriptor, for the operator layer.
template<typename T, int KIND>
void jit_dense_call(cudaStream_t stream, const void *in, void *out, const JitArgs &a, bool rows, double scale) {
    const JitCall<T, T> c{stream, static_cast<const T *>(in), static_cast<T *>(out), a, static_cast<T>(scale)};
    if (rows) jit_rows<T, T, KIND, false>(c);
    else jit_cols<T, KIND>(c);
}
template<typename T, typename E, int KIND>
void jit_event_call(cudaStream_t stream, const void *in, void *out, const JitArgs &a, bool rows, double scale) {
    const JitCall<T, E> c{stream, static_cast<const E *>(in), static_cast<T *>(out), a, static_cast<T>(scale)};
    if (rows) jit_rows<T, E, KIND, true>(c);
    else jit_cols_event<T, E, KIND>(c);
}

template<typename T, int KIND>
void jit_matvec_v1_impl(cudaStream_t stream, void **buffers, const char *opaque, size_t opaque_len) {
    JitArgs a;
    if (!unpack_jit<KIND>(opaque, opaque_len, a)) return;   // a.log_p holds the raw probability here
    if (a.n_row == 0) return;
    jit_rows_dense_v1_kernel<T, KIND><<<blocks_for(a.n_row, JIT_THREADS), JIT_THREADS, 0, stream>>>(
        static_cast<const T *>(buffers[0]), a.seed, a.log_p, a.w1, a.w2, a.n_row, a.n_col,
        static_cast<T *>(buffers[1]));
    launch_ok();
}

template<typename T, typename E, int KIND, bool ROWS>
void jit_event_matvec_impl(cudaStream_t stream, void **buffers, const char *opaque, size_t opaque_len) {
    JitCall<T, E> c{stream, static_cast<const E *>(buffers[0]), static_cast<T *>(buffers[1]), {}, T(1)};
    if (!unpack_jit<KIND>(opaque, opaque_len, c.a) || c.a.n_row == 0) return;
    if (ROWS) jit_rows<T, E, KIND, true>(c);
    else jit_cols_event<T, E, KIND>(c);
}

template<typename T, int KIND>
void jit_matmat_impl(cudaStream_t stream, void **buffers, const char *opaque, size_t opaque_len) {
    const MatMatJITProbDescriptor1 *d = unpack<MatMatJITProbDescriptor1>(opaque, opaque_len);
    if (!d) return;
    const T *X = static_cast<const T *>(buffers[0]);
    T *Y = static_cast<T *>(buffers[1]);
    if (d->m == 0 || d->n == 0) return;
    const unsigned int gy = blocks_for(d->m, MM_ROWS);
    if (gy > 65535u) {
        set_status(BPL_ERR_ARGUMENT, "matmat: more than 65535 * 32 rows in the dense operand");
        return;
    }
    constexpr size_t smem = static_cast<size_t>(MMTile<T>::KT) * MM_ROWS * sizeof(T);
    static thread_local int configured_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_device != dev) {
        if (cudaFuncSetAttribute(jit_matmat_kernel<T, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)) != cudaSuccess) {
            launch_ok();
            return;
        }
        configured_device = dev;
    }
    const dim3 grid(blocks_for(d->n, MM_THREADS), gy);
    jit_matmat_kernel<T, KIND><<<grid, MM_THREADS, smem, stream>>>(
        X, d->seed, gap_params(d->log_p, d->k), d->w1, d->w2, d->m, d->k, d->n, Y);
    launch_ok();
}

}  // namespace

}  // namespace bpl

using namespace bpl;

extern "C" {

void bpl_jit_matvec(bpl_stream_t stream, const void *in, void *out, int in_type, int events, int kind, int rows,
                    uint32_t n_row, uint32_t n_col, uint32_t seed, float log_p, float w1, float w2, double scale) {
    using Call = void (*)(cudaStream_t, const void *, void *, const JitArgs &, bool, double);
    static const Call dense[2][3] = {{jit_dense_call<float, W_HOMO>, jit_dense_call<float, W_UNIFORM>, jit_dense_call<float, W_NORMAL>},
                                     {jit_dense_call<double, W_HOMO>, jit_dense_call<double, W_UNIFORM>, jit_dense_call<double, W_NORMAL>}};
    static const Call event[3][3] = {
        {jit_event_call<float, bool, W_HOMO>, jit_event_call<float, bool, W_UNIFORM>, jit_event_call<float, bool, W_NORMAL>},
        {jit_event_call<float, float, W_HOMO>, jit_event_call<float, float, W_UNIFORM>, jit_event_call<float, float, W_NORMAL>},
        {jit_event_call<double, double, W_HOMO>, jit_event_call<double, double, W_UNIFORM>, jit_event_call<double, double, W_NORMAL>}};
    if (in_type < 0 || in_type > 2 || kind < 0 || kind > 2 || (!events && in_type == 0)) {
        set_status(BPL_ERR_ARGUMENT, "bpl_jit_matvec: unknown type or kind");
        return;
    }
    if (n_row == 0) return;
    const JitArgs a{n_row, n_col, seed, log_p, kind == W_HOMO ? 0.0 : static_cast<double>(w1),
                    kind == W_HOMO ? 0.0 : static_cast<double>(w2)};
    (events ? event[in_type] : dense[in_type - 1])[kind](stream, in, out, a, rows != 0, scale);
}

// Tests only: adds to *count (device memory) the draws whose gap the quick test gets wrong; 0 where log_p is outside its range.
int bpl_jit_gap_mismatches(bpl_stream_t stream, double log_p, unsigned long long *count) {
    const GapParams g = gap_params(log_p, 1u);
    if (!g.quick) return 0;
    jit_gap_mismatches_kernel<<<16 * sm_count(), 256, 0, stream>>>(g, count);
    return launch_ok() ? 1 : 0;
}

#define JIT_MATVEC(name, T, KIND, ROWS) \
    void name(bpl_stream_t s, void **b, const char *o, size_t n) { jit_matvec_impl<T, KIND, ROWS>(s, b, o, n); }
#define JIT_MATVEC_ALL(kind, KIND)                                           \
    JIT_MATVEC(gpu_matvec_prob_##kind##_v2_float, float, KIND, true)          \
    JIT_MATVEC(gpu_matvec_prob_##kind##_v2_double, double, KIND, true)        \
    JIT_MATVEC(gpu_matvec_atomic_prob_##kind##_v2_float, float, KIND, false)  \
    JIT_MATVEC(gpu_matvec_atomic_prob_##kind##_v2_double, double, KIND, false)
JIT_MATVEC_ALL(homo, W_HOMO)
JIT_MATVEC_ALL(uniform, W_UNIFORM)
JIT_MATVEC_ALL(normal, W_NORMAL)

#define JIT_MATVEC_V1(name, T, KIND) \
    void name(bpl_stream_t s, void **b, const char *o, size_t n) { jit_matvec_v1_impl<T, KIND>(s, b, o, n); }
JIT_MATVEC_V1(gpu_matvec_prob_homo_v1_float, float, W_HOMO)
JIT_MATVEC_V1(gpu_matvec_prob_homo_v1_double, double, W_HOMO)
JIT_MATVEC_V1(gpu_matvec_prob_uniform_v1_float, float, W_UNIFORM)
JIT_MATVEC_V1(gpu_matvec_prob_uniform_v1_double, double, W_UNIFORM)
JIT_MATVEC_V1(gpu_matvec_prob_normal_v1_float, float, W_NORMAL)
JIT_MATVEC_V1(gpu_matvec_prob_normal_v1_double, double, W_NORMAL)

#define JIT_EVENT(name, T, E, KIND, ROWS) \
    void name(bpl_stream_t s, void **b, const char *o, size_t n) { jit_event_matvec_impl<T, E, KIND, ROWS>(s, b, o, n); }
#define JIT_EVENT_ALL(kind, KIND)                                                               \
    JIT_EVENT(gpu_event_matvec_prob_##kind##_v2_float_bool, float, bool, KIND, true)             \
    JIT_EVENT(gpu_event_matvec_prob_##kind##_v2_float_float, float, float, KIND, true)           \
    JIT_EVENT(gpu_event_matvec_prob_##kind##_v2_double_bool, double, bool, KIND, true)           \
    JIT_EVENT(gpu_event_matvec_prob_##kind##_v2_double_double, double, double, KIND, true)       \
    JIT_EVENT(gpu_event_matvec_atomic_prob_##kind##_v2_float_bool, float, bool, KIND, false)     \
    JIT_EVENT(gpu_event_matvec_atomic_prob_##kind##_v2_float_float, float, float, KIND, false)   \
    JIT_EVENT(gpu_event_matvec_atomic_prob_##kind##_v2_double_bool, double, bool, KIND, false)   \
    JIT_EVENT(gpu_event_matvec_atomic_prob_##kind##_v2_double_double, double, double, KIND, false)
JIT_EVENT_ALL(homo, W_HOMO)
JIT_EVENT_ALL(uniform, W_UNIFORM)
JIT_EVENT_ALL(normal, W_NORMAL)

#define JIT_MATMAT(name, T, KIND) \
    void name(bpl_stream_t s, void **b, const char *o, size_t n) { jit_matmat_impl<T, KIND>(s, b, o, n); }
JIT_MATMAT(gpu_matmat_prob_prob_normal_float_v1, float, W_NORMAL)
JIT_MATMAT(gpu_matmat_prob_prob_normal_double_v1, double, W_NORMAL)
JIT_MATMAT(gpu_matmat_prob_prob_uniform_float_v1, float, W_UNIFORM)
JIT_MATMAT(gpu_matmat_prob_prob_uniform_double_v1, double, W_UNIFORM)

}  // extern "C"
