// Y = X @ M for a just-in-time M with one stream per output column, every stream generated ONCE (targets *_v1_ws).
//
// The inline kernel (jit_matmat_kernel, jitconn_kernels.cu) regenerates the stream of a column for every group of 32 rows
// of X, as the reference does (lib/gpu_jitconn_matmat.cu:236-276, :321-361).  Here one launch walks every stream once and
// writes its connections, position and weight (the same draws, the same conversions), into a list per column, while other
// blocks of it transpose X; a second launch multiplies from the lists.  Every (row, column) sum receives its products in
// stream order: the bits of the inline kernel.
//
// Workspace of one chunk of C columns (the host walks the columns chunk by chunk):
//   cnt u32[C] | Xt T[m_pad / 32][k][32] (X transposed in groups of 32 rows) | entries MMEntry<T>[C * stride]
// Entry j of column c sits at c * cap + j, position and weight side by side (8 bytes for float, 16 for double); a list
// ends with an entry whose position is k or more.  cap = expected connections per column + 10 standard deviations + 16, a
// multiple of 4.  A column with more (never seen; the bound is not a proof) reads as empty and is walked again, stream and
// all, by the warp or thread that owns it.
#include <algorithm>
#include <cmath>

#include <math_constants.h>

#include "abi.h"
#include "common.cuh"
#include "jit_stream.cuh"

namespace bpl {
namespace {

template<typename T> struct MMEntry;
template<> struct __align__(8) MMEntry<float> { unsigned int pos; float w; };
template<> struct __align__(16) MMEntry<double> { unsigned int pos, pad; double w; };
template<typename T> struct __align__(16) MMEntryPair { MMEntry<T> a, b; };
constexpr unsigned int LIST_END = 0xffffffffu;
// four entries, written as whole sectors
template<typename T> struct __align__(32) MMEntryQuad { MMEntry<T> e[4]; };
template<typename T>
__device__ __forceinline__ void store_entries(MMEntry<T> *to, const MMEntryQuad<T> &q) {
    const uint32_t *v = reinterpret_cast<const uint32_t *>(&q);
#pragma unroll
    for (unsigned int i = 0; i < sizeof(q) / 4; i += 8)
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                     :: "l"(reinterpret_cast<uint32_t *>(to) + i), "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]),
                        "r"(v[i + 4]), "r"(v[i + 5]), "r"(v[i + 6]), "r"(v[i + 7]) : "memory");
}

inline unsigned int blocks_for(unsigned long long n, unsigned int per_block) {
    return static_cast<unsigned int>((n + per_block - 1) / per_block);
}

template<typename T, int R> struct Values;
template<> struct Values<float, 1> { float v[1]; };
template<> struct __align__(8) Values<float, 2> { float v[2]; };
template<> struct __align__(16) Values<float, 4> { float v[4]; };
template<> struct Values<double, 1> { double v[1]; };
template<> struct __align__(16) Values<double, 2> { double v[2]; };

// ---- lists and transposition, in one launch ----
constexpr int FILL_THREADS = 128;
constexpr unsigned int MM_ROWS = 32;      // rows of X are padded to whole groups

// One thread per column: bound by the latency of its chain (65,536 columns: 14 warps per SM), hence the batches of
// jit_stream.cuh and small blocks, which spread over the SMs; and by the writes, 32 lists per warp: a batch is four entries
// and goes out as one sector (two for double), the last one with entries behind the end, which end the list.
template<typename T, int KIND, bool QUICK>
__device__ __forceinline__ void fill_list(const unsigned int seed, const GapParams &gp, const double w1, const double w2,
                                          const unsigned int k, const unsigned int cap, unsigned int *cnt, MMEntry<T> *mine) {
    Xorwow s;
    s.seed(seed);
    Batch<KIND, QUICK, 4> b;
    unsigned int count = 0, at = 0;
    do {
        b.draw(s, at, k, gp);
        T w[4];
        b.weights(w, w1, w2);
        MMEntryQuad<T> q;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            q.e[j].pos = b.pos[j];
            q.e[j].w = w[j];
        }
        if (count + 4u <= cap) store_entries(mine + count, q);
        count += 4u;
    } while (at < k);
    // of the last batch, the entries before the end
#pragma unroll
    for (int j = 0; j < 4; ++j) count -= b.pos[j] >= k;
    if (((count + 4u) & ~3u) > cap) {     // the batch with the end did not fit: reads as empty
        count = cap + 1u;
        mine[0].pos = LIST_END;
    }
    *cnt = count;
}

// 32 x 32 tiles of X through shared memory into Xt; rows past m are zero
template<typename T>
__device__ __forceinline__ void transpose_tile(const T *__restrict__ X, const unsigned int m, const unsigned int k,
                                               T *__restrict__ Xt, const unsigned int k0, const unsigned int m0, T (*t)[33]) {
    const unsigned int x = threadIdx.x & 31u, y = threadIdx.x >> 5;
    T v[32 / (FILL_THREADS / 32)];
#pragma unroll
    for (unsigned int i = 0; i < 32 / (FILL_THREADS / 32); ++i) {
        const unsigned int r = m0 + i * (FILL_THREADS / 32) + y, c = k0 + x;
        v[i] = (r < m && c < k) ? X[static_cast<size_t>(r) * k + c] : T(0);
    }
#pragma unroll
    for (unsigned int i = 0; i < 32 / (FILL_THREADS / 32); ++i) t[i * (FILL_THREADS / 32) + y][x] = v[i];
    __syncthreads();
#pragma unroll
    for (unsigned int i = 0; i < 32 / (FILL_THREADS / 32); ++i) {
        const unsigned int c = k0 + i * (FILL_THREADS / 32) + y;
        if (c < k) Xt[(static_cast<size_t>(m0 / MM_ROWS) * k + c) * MM_ROWS + x] = t[x][i * (FILL_THREADS / 32) + y];
    }
    __syncthreads();
}

// blocks [0, fill_blocks): columns; the others: tiles of X (none when Xt is already there)
template<typename T, int KIND, bool QUICK>
__global__ void __launch_bounds__(FILL_THREADS)
jit_matmat_prepare_kernel(const unsigned int seed, const GapParams gp, const double w1, const double w2, const unsigned int k,
                          const unsigned int cols, const unsigned int cap, unsigned int *__restrict__ cnt,
                          MMEntry<T> *__restrict__ entries, const unsigned int fill_blocks, const T *__restrict__ X,
                          const unsigned int m, const unsigned int m_pad, T *__restrict__ Xt) {
    __shared__ T tile[32][33];
    pdl_launch_dependents();                   // the multiply's blocks come up while the last lists are written
    if (blockIdx.x < fill_blocks) {
        const unsigned int c = blockIdx.x * FILL_THREADS + threadIdx.x;
        if (c < cols)
            fill_list<T, KIND, QUICK>(seed + c, gp, w1, w2, k, cap, cnt + c, entries + static_cast<size_t>(c) * cap);
        return;
    }
    const unsigned int tiles_k = (k + 31u) / 32u, n_tiles = tiles_k * (m_pad / 32u);
    for (unsigned int i = blockIdx.x - fill_blocks; i < n_tiles; i += gridDim.x - fill_blocks)
        transpose_tile(X, m, k, Xt, i % tiles_k * 32u, i / tiles_k * 32u, tile);
}

// ---- a column whose list overflowed, from its stream ----
// Every lane walks the same stream; `add(pos, w)` for every connection in order.
template<typename T, int KIND, typename Add>
__device__ __noinline__ void walk_column(const unsigned int seed, const GapParams &gp, const double w1, const double w2,
                                         const unsigned int k, Add add) {
    curandState st;
    curand_init(seed, 0, 0, &st);
    unsigned int pos = next_position(0u, curand(&st), gp);
    while (pos < k) {
        T w;
        if (KIND == W_NORMAL) w = (T) (curand_normal(&st) * w2 + w1);
        else w = (T) (curand_uniform(&st) * w2 + w1);
        add(pos, w);
        pos = next_position(pos, curand(&st), gp);
    }
}

// ---- the multiply, X staged in shared memory ----
// A thread owns one column and 32 rows of X and walks its own list; Xt is staged tile by tile into a ring of buffers, one
// block of up to 896 threads per SM.  A connection is 32 products against 8 reads of 16 bytes per lane: the lanes of a warp
// read different tile rows (their positions are unrelated), which would put them on the same banks, so lane l reads the
// 16-byte chunks of its row in the order c ^ (l mod CHUNKS): the eight lanes served together touch eight different chunks.
// The register (c, i) of lane l belongs to row (c ^ (l mod CHUNKS)) * PER_CHUNK + i.
//
// What bounds it is the shared-memory pipe, how many lanes of a warp have work in the tiles that are resident (the number of
// connections per column and tile is Poisson), and what a warp does once per tile.  It moves on when all its lanes are through
// with its oldest tile, while a lane that is through runs on into the next ones that have landed; and no warp waits for
// another: each waits for the arrival of a tile only (an mbarrier per buffer), and the last warp to leave a tile starts the
// copy (one bulk copy) that takes its place.  With eight tiles of 192 positions a warp spent 140 instructions per tile on that,
// twice what a connection takes: four tiles of 384 hold the same positions (192 KB: with more, L1 no longer holds the other
// half of the sectors that the lists come in), and it waits for the tile after its own before it goes on, so that lanes have
// somewhere to run on to.
// 256 x 65536 @ 65536^2, 1 %: 3.09 ms with one tile at a time and block barriers, 2.39 ms with the ring (without the lists),
// 2.25 now; 100 x 30000 @ 30000 x 40000, 0.5 %: whole call 321 -> 271 us.
//
// Measured alternatives: lanes as rows (a warp owns 30 columns x 64 rows, entries broadcast from a staging buffer, every
// lane works on every connection) 5.3 ms: 14 instructions per entry and 64 rows against 50 per 32 entries and 32 rows here;
// the same without staging 7.7-10 ms.  Lists read four entries at a time: 3 to 25 % slower.  Steps while some number of lanes
// have work, tiles given back behind the last lane of all: 5 to 60 % slower.  Packed multiply-adds: no change.
constexpr unsigned int RING = 4;                            // buffers of 48 KB
constexpr unsigned int AHEAD = 2;                           // tiles that have landed before a warp works on the first of them
template<typename T> struct ApplyShape;
template<> struct ApplyShape<float> { static constexpr int MAX_THREADS = 896, KT = 384, CHUNKS = 8; };
template<> struct ApplyShape<double> { static constexpr int MAX_THREADS = 512, KT = 192, CHUNKS = 16; };   // 32 double sums
constexpr unsigned int TILE_BYTES = 48u * 1024u;
constexpr unsigned int APPLY_SMEM = RING * TILE_BYTES;

__device__ __forceinline__ uint32_t shared_address(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void barrier_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(shared_address(bar)) : "memory");
}
// the one arrival of a phase, and the bytes that complete it
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, const uint32_t bytes, uint64_t *bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(shared_address(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(shared_address(dst)), "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(shared_address(bar)) : "memory");
}
__device__ __forceinline__ bool barrier_done(uint64_t *bar, const uint32_t parity) {
    uint32_t done;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(done) : "r"(shared_address(bar)), "r"(parity) : "memory");
    return done != 0;
}
// Waits for a phase; false when it has not come within a second or so.
__device__ __forceinline__ bool barrier_wait(uint64_t *bar, const uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(shared_address(bar)), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// sum[0 ..] += w * the 16 bytes at `at`
__device__ __forceinline__ void add_chunk(float *sum, const uint32_t at, const float w) {
    float x[4];
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(at) : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += (x[i] * w);
}
__device__ __forceinline__ void add_chunk(double *sum, const uint32_t at, const double w) {
    double x[2];
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x[0]), "=d"(x[1]) : "r"(at) : "memory");
#pragma unroll
    for (int i = 0; i < 2; ++i) sum[i] += (x[i] * w);
}

// grid = (row groups of 32, column blocks of blockDim.x columns): the blocks that walk the same columns' lists are
// launched side by side, so the lists come from DRAM once and from L2 for the other row groups.
template<typename T, int KIND>
__global__ void __launch_bounds__(ApplyShape<T>::MAX_THREADS, 1)
jit_matmat_apply_kernel(const T *Xt, const unsigned int m, const unsigned int k, const unsigned int n,
                        const unsigned int col0, const unsigned int cols, const unsigned int cap,
                        const unsigned int *cnt, const MMEntry<T> *entries,
                        const unsigned int seed, const GapParams gp, const double w1, const double w2, T *__restrict__ Y) {
    constexpr int KT = ApplyShape<T>::KT, CHUNKS = ApplyShape<T>::CHUNKS, PER_CHUNK = 16 / sizeof(T);
    static_assert(KT * MM_ROWS * sizeof(T) == TILE_BYTES, "a tile");
    extern __shared__ __align__(256) unsigned char mm_smem[];           // T [RING][KT][MM_ROWS]; a row of it (128 or 256 bytes) aligned to itself
    __shared__ __align__(8) uint64_t landed_bar[RING];
    __shared__ unsigned int left[RING];                                  // warps that are through with the tile of a buffer
    pdl_wait();

    const unsigned int c = blockIdx.y * blockDim.x + threadIdx.x;       // column within the chunk
    const bool live = c < cols;
    const unsigned int lane = threadIdx.x & 31u;
    const T *group = Xt + static_cast<size_t>(blockIdx.x) * k * MM_ROWS;
    const bool overflow = live && cnt[c] > cap;                         // its list reads as empty
    // The list is read two entries at a time (every lane reads its own list, so a warp's load touches 32 different lines).
    // `pos` and `weight` are the entry to come, `second` is the other one of its pair (while `odd`), and `next` the pair behind
    // it, requested when its predecessor is entered.  Positions ascend: a pair whose second is inside has a successor.
    const MMEntryPair<T> *pairs = reinterpret_cast<const MMEntryPair<T> *>(entries + static_cast<size_t>(c) * cap);
    MMEntry<T> second;
    MMEntryPair<T> next;
    unsigned int pos = LIST_END;
    T weight = T(0);
    bool odd = true;
    second.pos = next.a.pos = next.b.pos = LIST_END;
    second.w = next.a.w = next.b.w = T(0);
    if (live) {
        next = *pairs++;
        pos = next.a.pos;
        weight = next.a.w;
        second = next.b;
        if (max(pos, second.pos) < k) next = *pairs;
    }
    T sum[MM_ROWS];
#pragma unroll
    for (int i = 0; i < static_cast<int>(MM_ROWS); ++i) sum[i] = T(0);

    const unsigned int n_tiles = (k + KT - 1) / KT, n_warps = blockDim.x >> 5;
    auto issue = [&](const unsigned int t) {                             // tile t into buffer t mod RING
        const unsigned int rows = min(static_cast<unsigned int>(KT), k - t * KT);
        bulk_copy(mm_smem + (t % RING) * TILE_BYTES, group + static_cast<size_t>(t) * KT * MM_ROWS,
                  rows * static_cast<unsigned int>(MM_ROWS * sizeof(T)), &landed_bar[t % RING]);
    };
    if (threadIdx.x == 0) {
        for (unsigned int i = 0; i < RING; ++i) {
            barrier_init(&landed_bar[i]);
            left[i] = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (unsigned int t = 0; t < min(RING, n_tiles); ++t) issue(t);
    }
    __syncthreads();
    unsigned int landed = 0;                                             // tiles that this warp knows to be there
    const uint32_t home = shared_address(mm_smem) + (lane & (CHUNKS - 1)) * 16u;
    bool lost = false;
    for (unsigned int t = 0; t < n_tiles; ++t) {
        while (landed < min(t + AHEAD, n_tiles)) {                       // (below t + RING: started, at the latest when the last warp leaves tile t - 1)
            lost = __any_sync(FULL_MASK, !barrier_wait(&landed_bar[landed % RING], (landed / RING) & 1u));
            if (lost) break;
            ++landed;
        }
        if (lost) break;
        // further ones: below t + RING, whose buffer is the one of tile t
        while (landed < min(t + RING, n_tiles) && __all_sync(FULL_MASK, barrier_done(&landed_bar[landed % RING], (landed / RING) & 1u)))
            ++landed;
        const unsigned int first = t * KT, done = min(first + KT, k), open = min(landed * KT, k);
        const unsigned int slot0 = (t % RING) * KT;
        while (__any_sync(FULL_MASK, pos < done)) {
            if (pos < open) {
                unsigned int slot = slot0 + (pos - first);
                if (slot >= RING * KT) slot -= RING * KT;
                const uint32_t row = home + slot * static_cast<uint32_t>(MM_ROWS * sizeof(T));
                const T w = weight;
                if (odd) {
                    pos = second.pos;
                    weight = second.w;
                } else {
                    pos = next.a.pos;
                    weight = next.a.w;
                    second = next.b;
                    ++pairs;
                    if (second.pos < k) next = *pairs;
                }
                odd = !odd;
#pragma unroll
                for (int cc = 0; cc < CHUNKS; ++cc) add_chunk(&sum[cc * PER_CHUNK], row ^ (cc * 16u), w);
            }
        }
        __syncwarp();
        if (lane == 0 && t + RING < n_tiles) {
            __threadfence_block();                                       // the reads of this warp are over
            if (atomicAdd(&left[t % RING], 1u) == n_warps - 1u) {
                __threadfence_block();                                   // and those of the others
                left[t % RING] = 0;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue(t + RING);
            }
        }
    }
    if (lost) {                                                          // never seen: no result rather than a wrong one
        // the copies that may be in flight, each by the phase of its own tile (one that was never started runs the wait out)
        for (unsigned int i = 0; i < RING; ++i) barrier_wait(&landed_bar[i], ((landed + (i - landed) % RING) / RING) & 1u);
#pragma unroll
        for (int i = 0; i < static_cast<int>(MM_ROWS); ++i) sum[i] = T(CUDART_NAN_F);
    }
    const unsigned int row0 = blockIdx.x * MM_ROWS;
    if (live && !overflow) {
#pragma unroll
        for (int cc = 0; cc < CHUNKS; ++cc) {
            const unsigned int chunk = cc ^ (lane & (CHUNKS - 1));
#pragma unroll
            for (int i = 0; i < PER_CHUNK; ++i) {
                const unsigned int row = row0 + chunk * PER_CHUNK + i;
                if (row < m) Y[static_cast<size_t>(row) * n + col0 + c] = sum[cc * PER_CHUNK + i];
            }
        }
    }
    if (overflow) {
        T over[MM_ROWS];
        for (unsigned int r = 0; r < MM_ROWS; ++r) over[r] = T(0);
        walk_column<T, KIND>(seed + c, gp, w1, w2, k, [&](const unsigned int at, const T w) {
            for (unsigned int r = 0; r < MM_ROWS; ++r) over[r] += (group[static_cast<size_t>(at) * MM_ROWS + r] * w);
        });
        for (unsigned int r = 0; r < MM_ROWS; ++r)
            if (row0 + r < m) Y[static_cast<size_t>(row0 + r) * n + col0 + c] = over[r];
    }
}

// ---- the multiply, X read from L2 ----
// Staging pays when a staged position is used by several of a block's columns.  Where it is not (few columns, or a small
// probability: 5500 columns at 0.24 % use one position in four), a warp takes one column and 32 * V rows and reads the X
// values of its connections where they lie, 128 to 512 contiguous bytes each.  A block is 8 neighbouring columns, so that
// 32-byte pieces of Y are written at once.
constexpr int GATHER_COLS = 8;

template<typename T, int KIND, int V>
__global__ void __launch_bounds__(GATHER_COLS * 32)
jit_matmat_gather_kernel(const T *Xt, const unsigned int m, const unsigned int m_pad, const unsigned int k,
                         const unsigned int n, const unsigned int col0, const unsigned int cols, const unsigned int cap,
                         const unsigned int *cnt, const MMEntry<T> *entries,
                         const unsigned int seed, const GapParams gp, const double w1, const double w2, T *__restrict__ Y) {
    __shared__ T block[GATHER_COLS][32 * V + 1];
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    pdl_wait();
    const unsigned int c = blockIdx.x * GATHER_COLS + warp, row0 = blockIdx.y * 32u * V, row = row0 + lane * V;
    T sum[V];
#pragma unroll
    for (int v = 0; v < V; ++v) sum[v] = T(0);
    if (c < cols) {
        const bool inside = row < m_pad;                                 // (m_pad is a multiple of 32)
        const T *x = Xt + static_cast<size_t>(row / MM_ROWS) * k * MM_ROWS + row % MM_ROWS;
        const unsigned int count = cnt[c];
        auto add = [&](const unsigned int at, const T w) {
            if (!inside) return;
            const Values<T, V> q = *reinterpret_cast<const Values<T, V> *>(x + static_cast<size_t>(at) * MM_ROWS);
#pragma unroll
            for (int v = 0; v < V; ++v) sum[v] += (q.v[v] * w);
        };
        if (count <= cap) {
            const MMEntry<T> *list = entries + static_cast<size_t>(c) * cap;
            MMEntry<T> e;
            e.pos = 0;
            e.w = T(0);
            if (lane < count) e = list[lane];
            for (unsigned int base = 0; base < count; base += 32u) {
                const MMEntry<T> now = e;
                if (base + 32u + lane < count) e = list[base + 32u + lane];
                const unsigned int here = min(32u, count - base);
                unsigned int i = 0;
                for (; i + 8u <= here; i += 8u) {                        // eight reads in flight
                    Values<T, V> q[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const unsigned int at = __shfl_sync(FULL_MASK, now.pos, i + u);
                        if (inside) q[u] = *reinterpret_cast<const Values<T, V> *>(x + static_cast<size_t>(at) * MM_ROWS);
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const T w = __shfl_sync(FULL_MASK, now.w, i + u);
                        if (inside) {
#pragma unroll
                            for (int v = 0; v < V; ++v) sum[v] += (q[u].v[v] * w);
                        }
                    }
                }
                for (; i < here; ++i) add(__shfl_sync(FULL_MASK, now.pos, i), __shfl_sync(FULL_MASK, now.w, i));
            }
        } else {
            T over[V];                                                   // (its address is taken: not `sum`)
#pragma unroll
            for (int v = 0; v < V; ++v) over[v] = T(0);
            walk_column<T, KIND>(seed + c, gp, w1, w2, k, [&](const unsigned int at, const T w) {
                if (!inside) return;
                for (int v = 0; v < V; ++v) over[v] += (x[static_cast<size_t>(at) * MM_ROWS + v] * w);
            });
#pragma unroll
            for (int v = 0; v < V; ++v) sum[v] = over[v];
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) block[warp][lane * V + v] = sum[v];
    __syncthreads();
    for (unsigned int i = threadIdx.x; i < 32u * V * GATHER_COLS; i += GATHER_COLS * 32u) {
        const unsigned int r = i / GATHER_COLS, column = blockIdx.x * GATHER_COLS + i % GATHER_COLS;
        if (row0 + r < m && column < cols) Y[static_cast<size_t>(row0 + r) * n + col0 + column] = block[i % GATHER_COLS][r];
    }
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
constexpr size_t LIST_BUDGET = 768ull << 20;        // bytes of lists one chunk of columns may take
constexpr unsigned int CHUNK_UNIT = 512;            // columns
// tests: force a small capacity (columns overflow) or a small budget (several chunks of columns)
unsigned int g_list_cap_override = 0;
size_t g_list_budget_override = 0;

struct ListPlan {
    unsigned int cap;        // list slots per column
    unsigned int chunk;      // columns per chunk
    unsigned int m_pad;      // rows of X rounded up to whole groups
    double prob;
    size_t xt_off, entries_off, bytes;
};

ListPlan list_plan(unsigned int m, unsigned int k, unsigned int n, double log_p, size_t elem) {
    ListPlan p;
    p.prob = -std::expm1(log_p);                              // log_p = log(1 - conn_prob)
    const double mean = static_cast<double>(k) * p.prob;
    const double cap_d = std::ceil(mean + 10.0 * std::sqrt(mean * (1.0 - p.prob) + 1.0)) + 16.0;
    p.cap = static_cast<unsigned int>(std::min(cap_d, static_cast<double>(k) + 16.0));   // (k, and a batch that ends it)
    if (g_list_cap_override != 0) p.cap = g_list_cap_override;
    p.cap = (p.cap + 3u) & ~3u;
    const size_t entry = elem == 8 ? 16 : 8;        // sizeof(MMEntry<T>)
    const size_t per_col = static_cast<size_t>(p.cap) * entry + 4;
    const size_t n_round = (static_cast<size_t>(n) + CHUNK_UNIT - 1) / CHUNK_UNIT * CHUNK_UNIT;
    const size_t budget = g_list_budget_override != 0 ? g_list_budget_override : LIST_BUDGET;
    const size_t chunk = std::min(std::max<size_t>(budget / per_col / CHUNK_UNIT * CHUNK_UNIT, CHUNK_UNIT), n_round);
    p.chunk = static_cast<unsigned int>(chunk);
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    p.m_pad = (m + MM_ROWS - 1) / MM_ROWS * MM_ROWS;
    p.xt_off = up(4 * chunk);
    p.entries_off = up(p.xt_off + elem * static_cast<size_t>(k) * p.m_pad);
    p.bytes = up(p.entries_off + entry * chunk * static_cast<size_t>(p.cap));
    return p;
}

// Threads (= columns) per block of the staged form: the number whose last wave of blocks, one per SM, wastes least.
struct StagedChoice {
    unsigned int threads = 128;
    double clocks = 1e300;       // of one SM
};
template<typename T>
StagedChoice choose_staged(const ListPlan &p, unsigned int k, unsigned int cols) {
    const double sms = sm_count(), groups = p.m_pad / MM_ROWS, row_bytes = MM_ROWS * sizeof(T);
    StagedChoice best;
    for (unsigned int th = 128; th <= static_cast<unsigned int>(ApplyShape<T>::MAX_THREADS); th += 32) {
        const double waves = std::ceil(blocks_for(cols, th) * groups / sms);
        // per position: its copy into shared memory (16 bytes per clock: a tile is in flight while one is worked on), or the
        // connections that use it (2.5 clocks for 32 float rows; 2.0 to 3.7 measured, the more the fewer share a tile: where
        // the choice against the other kernel is close, both take the same to 6 %)
        const double clocks = waves * k * std::max(row_bytes / 16, th * p.prob * 2.5 * row_bytes / 128);
        if (clocks <= best.clocks) best = {th, clocks};
    }
    return best;
}

template<typename T, int KIND, int V>
void launch_gather(cudaStream_t stream, const ListPlan &p, const MatMatJITProbDescriptor1 *d, unsigned int col0, unsigned int cols,
                   const unsigned int *cnt, const MMEntry<T> *entries, const GapParams &gp, const T *Xt, T *Y) {
    const cudaError_t e = launch_dependent(
        jit_matmat_gather_kernel<T, KIND, V>, dim3(blocks_for(cols, GATHER_COLS), blocks_for(p.m_pad, 32 * V)),
        dim3(GATHER_COLS * 32), 0, stream, Xt, d->m, p.m_pad, d->k, d->n, col0, cols, p.cap, cnt, entries, d->seed + col0, gp,
        d->w1, d->w2, Y);
    if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
}

template<typename T, int KIND>
void jit_matmat_list_impl(cudaStream_t stream, void **buffers, const char *opaque, size_t opaque_len) {
    const MatMatJITProbDescriptor1 *d = unpack<MatMatJITProbDescriptor1>(opaque, opaque_len);
    if (!d) return;
    const T *X = static_cast<const T *>(buffers[0]);
    T *Y = static_cast<T *>(buffers[1]);
    unsigned char *ws = static_cast<unsigned char *>(buffers[2]);
    if (d->m == 0 || d->n == 0) return;
    if (d->m > 65535u * MM_ROWS) {
        set_status(BPL_ERR_ARGUMENT, "matmat: more than 65535 * 32 rows in the dense operand");
        return;
    }
    if (ws == nullptr || (reinterpret_cast<uintptr_t>(ws) & 255u) != 0) {
        set_status(BPL_ERR_ARGUMENT, "matmat: the workspace is missing or not aligned to 256 bytes");
        return;
    }
    if (d->k == 0) {
        if (cudaMemsetAsync(Y, 0, sizeof(T) * static_cast<size_t>(d->m) * d->n, stream) != cudaSuccess) launch_ok();
        return;
    }
    const ListPlan p = list_plan(d->m, d->k, d->n, d->log_p, sizeof(T));
    const GapParams gp = gap_params(d->log_p, d->k);
    unsigned int *cnt = reinterpret_cast<unsigned int *>(ws);
    T *Xt = reinterpret_cast<T *>(ws + p.xt_off);
    MMEntry<T> *entries = reinterpret_cast<MMEntry<T> *>(ws + p.entries_off);
    const double sms = sm_count();
    for (unsigned long long at = 0; at < d->n; at += p.chunk) {
        const unsigned int col0 = static_cast<unsigned int>(at);
        const unsigned int cols = static_cast<unsigned int>(std::min<unsigned long long>(d->n - at, p.chunk));
        const unsigned int fill = blocks_for(cols, FILL_THREADS);
        const unsigned long long x_tiles = static_cast<unsigned long long>(blocks_for(d->k, 32)) * (p.m_pad / 32);
        const unsigned int more = at == 0 ? static_cast<unsigned int>(std::min<unsigned long long>(x_tiles, 16ull * sm_count())) : 0u;
        (gp.quick ? jit_matmat_prepare_kernel<T, KIND, true> : jit_matmat_prepare_kernel<T, KIND, false>)<<<
            fill + more, FILL_THREADS, 0, stream>>>(d->seed + col0, gp, d->w1, d->w2, d->k, cols, p.cap, cnt, entries, fill, X, d->m,
                                                    p.m_pad, Xt);
        const StagedChoice staged = choose_staged<T>(p, d->k, cols);
        // read from L2: 28 bytes per clock and SM, 4 clocks or more per connection and warp
        const unsigned int v = sizeof(T) == 8 ? (d->m > 32 ? 2 : 1) : d->m > 64 ? 4 : d->m > 32 ? 2 : 1;
        const double visits = static_cast<double>(cols) * d->k * p.prob * blocks_for(p.m_pad, 32 * v) / sms;
        if (staged.clocks < visits * std::max(std::min(32.0 * v, 1.0 * p.m_pad) * sizeof(T) / 28, 4.0)) {
            constexpr auto kernel = jit_matmat_apply_kernel<T, KIND>;
            if (!allow_shared<kernel>(APPLY_SMEM)) break;
            const cudaError_t e = launch_dependent(
                kernel, dim3(p.m_pad / MM_ROWS, blocks_for(cols, staged.threads)), dim3(staged.threads), APPLY_SMEM, stream, Xt,
                d->m, d->k, d->n, col0, cols, p.cap, cnt, entries, d->seed + col0, gp, d->w1, d->w2, Y);
            if (e != cudaSuccess) set_status(BPL_ERR_CUDA, cudaGetErrorString(e));
        } else if (v == 1) {
            launch_gather<T, KIND, 1>(stream, p, d, col0, cols, cnt, entries, gp, Xt, Y);
        } else if (v == 2) {
            launch_gather<T, KIND, 2>(stream, p, d, col0, cols, cnt, entries, gp, Xt, Y);
        } else {
            if constexpr (sizeof(T) == 4) launch_gather<T, KIND, 4>(stream, p, d, col0, cols, cnt, entries, gp, Xt, Y);
        }
    }
    launch_ok();
}

}  // namespace

size_t matmat_list_workspace_bytes(const char *opaque, size_t opaque_len, size_t elem) {
    if (opaque == nullptr || opaque_len != sizeof(MatMatJITProbDescriptor1)) return 0;
    const MatMatJITProbDescriptor1 *d = reinterpret_cast<const MatMatJITProbDescriptor1 *>(opaque);
    if (d->n == 0) return 256;
    return list_plan(d->m, d->k, d->n, d->log_p, elem).bytes;
}

}  // namespace bpl

using namespace bpl;

extern "C" {

#define JIT_MATMAT_LIST(name, T, KIND) \
    void name(bpl_stream_t s, void **b, const char *o, size_t n) { jit_matmat_list_impl<T, KIND>(s, b, o, n); }
JIT_MATMAT_LIST(gpu_matmat_prob_prob_normal_float_v1_ws, float, W_NORMAL)
JIT_MATMAT_LIST(gpu_matmat_prob_prob_normal_double_v1_ws, double, W_NORMAL)
JIT_MATMAT_LIST(gpu_matmat_prob_prob_uniform_float_v1_ws, float, W_UNIFORM)
JIT_MATMAT_LIST(gpu_matmat_prob_prob_uniform_double_v1_ws, double, W_UNIFORM)

// Tests only: non-zero values replace the computed list capacity per column and the byte budget of one chunk of
// columns (0 restores them), so that a small matrix overflows its lists or is walked in several chunks.
void bpl_matmat_list_limits_for_tests(uint32_t cap, size_t budget_bytes) {
    g_list_cap_override = cap;
    g_list_budget_override = budget_bytes;
}

}  // extern "C"
