// Device helpers shared by the kernels: streaming 128-bit loads, warp reductions.
#ifndef BPL_CSRC_COMMON_CUH_
#define BPL_CSRC_COMMON_CUH_

#include <cstdint>
#include <cuda_runtime.h>

namespace bpl {

constexpr unsigned FULL_MASK = 0xffffffffu;

// 128-bit read-only load that bypasses L1 allocation: matrix entries are touched once per call.
__device__ __forceinline__ uint4 ldg_stream_u4(const void *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// A whole sector (8 words; doubles: two) with one load each, from a 32-byte aligned address.
__device__ __forceinline__ void ldg_stream_8(const uint32_t *p, uint32_t (&v)[8]) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "l"(p));
}
__device__ __forceinline__ void ldg_stream_8(const float *p, float (&v)[8]) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}
__device__ __forceinline__ void ldg_stream_8(const double *p, double (&v)[8]) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
    asm volatile("ld.global.nc.L1::no_allocate.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v[4]), "=d"(v[5]), "=d"(v[6]), "=d"(v[7]) : "l"(p + 4));
}
// (one weight for all: nothing to load)
template<typename T>
__device__ __forceinline__ void ldg_stream_8(const T *, T (&)[1]) {}

__device__ __forceinline__ uint32_t ldg_stream_u32(const void *p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ uint2 ldg_stream_u2(const void *p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// Programmatic dependent launch (scan -> scatter pairs): the scan lets its dependents start as soon as it runs, the
// scatter does everything that needs no input from the scan (clearing its shared memory) and then waits here until
// the scan has completed and its writes are visible.  In a kernel that was launched the ordinary way the wait returns
// at once.
// What the launch in front writes must not be read through the read-only path (`ld.global.nc`, which the compiler also takes
// for a `const __restrict__` kernel argument): it is specified for data that stays constant while the kernel runs, and the
// reading kernel runs already.  Such reads are written as __ldcg or __ldca, or their pointers carry no __restrict__.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch of a kernel that may start before the kernel in front of it on the stream has finished (it must call
// pdl_wait() before it touches anything that kernel writes).
template<typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}


// Lets KERNEL take `bytes` of dynamic shared memory on the current device (set once per device and host thread).
template<auto KERNEL>
inline bool allow_shared(unsigned bytes) {
    static thread_local int configured_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_device != dev) {
        if (cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) != cudaSuccess)
            return false;
        configured_device = dev;
    }
    return true;
}

// Reduction without a return value (one L2 operation, nothing travels back), spelled out so that no
// call site can turn into the value-returning form.
__device__ __forceinline__ void red_add(float *p, float v) {
    asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" :: "l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void red_add(double *p, double v) {
    asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" :: "l"(p), "d"(v) : "memory");
}

__device__ __forceinline__ void red_add_v4(float *p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                 :: "l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

__device__ __forceinline__ bool aligned16_device(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Adds `count` sums of shared memory to `out`, by the whole block: 16-byte reductions where the addresses allow it, zeros
// left out.  Block `turn` of `turns` that add to the same output starts at its own place (58,000 floats from 148 blocks:
// 8 us, 10 us from one place).
template<typename T>
__device__ __forceinline__ void add_sums(const T *sums, T *__restrict__ out, const uint32_t count, const uint32_t turn,
                                         const uint32_t turns) {
    const uint32_t n4 = sizeof(T) == 4 && aligned16_device(out) ? count / 4 : 0u;
    const uint32_t from = static_cast<uint32_t>(static_cast<uint64_t>(n4) * turn / turns);
    for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x) {
        const uint32_t j = i + from < n4 ? i + from : i + from - n4;
        const float4 v = reinterpret_cast<const float4 *>(sums)[j];
        if (v.x != 0.0f || v.y != 0.0f || v.z != 0.0f || v.w != 0.0f)
            red_add_v4(reinterpret_cast<float *>(out) + 4u * j, v.x, v.y, v.z, v.w);
    }
    const uint32_t rest = count - 4u * n4, start = static_cast<uint32_t>(static_cast<uint64_t>(rest) * turn / turns);
    for (uint32_t i = threadIdx.x; i < rest; i += blockDim.x) {
        const uint32_t j = 4u * n4 + (i + start < rest ? i + start : i + start - rest);
        if (sums[j] != T(0)) red_add(out + j, sums[j]);
    }
}

// Per-entry results of entries that no row owns (arrays longer than the matrix): zero, by the whole grid.
template<typename T>
__device__ __forceinline__ void zero_outside_rows(T *__restrict__ g, const uint32_t *__restrict__ indptr, const uint32_t n_row,
                                                  const uint32_t nse) {
    const uint64_t first = indptr[0], from = indptr[n_row], step = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint64_t me = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    for (uint64_t i = me; i < first; i += step) g[i] = T(0);
    for (uint64_t i = from + me; i < nse; i += step) g[i] = T(0);
}

// 4 consecutive values to a 16-byte aligned address
__device__ __forceinline__ void store_quad(float *p, float a, float b, float c, float d) {
    *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void store_quad(double *p, double a, double b, double c, double d) {
    *reinterpret_cast<double2 *>(p) = make_double2(a, b);
    *reinterpret_cast<double2 *>(p + 2) = make_double2(c, d);
}

template<typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

// Sum inside aligned groups of `width` lanes (width a power of two <= 32, uniform in the warp).
template<typename T>
__device__ __forceinline__ T group_sum(T v, int width) {
    for (int o = width >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

// Truthiness of one event element, as `if (x[i])` in the reference kernels
// (lib/gpu_event_csr_matvec.cu:65,88): bool as is, floating point != 0 (NaN is truthy).
__device__ __forceinline__ bool is_event(bool e) { return e; }
__device__ __forceinline__ bool is_event(uint8_t e) { return e != 0; }
__device__ __forceinline__ bool is_event(float e) { return e != 0.0f; }
__device__ __forceinline__ bool is_event(double e) { return e != 0.0; }

// Packs the truthiness of n events into a bitmask (bit i of word i / 32 = event i) held in shared
// memory, cooperatively by the whole block.  Where the event array is 16-byte aligned each lane reads
// 16 bytes at a time (16 bools, 4 floats or 2 doubles), so a block needs one or two rounds of loads
// even for a million events; the unaligned case and the ragged end use one ballot per 32 events.
template<typename E>
__device__ __forceinline__ void pack_event_mask(const E *__restrict__ x, const uint32_t n, uint32_t *mask) {
    constexpr uint32_t PER_LANE = 16 / sizeof(E);          // events per 128-bit load
    constexpr uint32_t SPAN = 32 * PER_LANE;               // events per warp-wide load
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    const bool vec_ok = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    const uint32_t n_vec = vec_ok ? (n / SPAN) * SPAN : 0u;
    for (uint32_t base = warp * SPAN; base < n_vec; base += n_warps * SPAN) {
        const uint4 raw = *reinterpret_cast<const uint4 *>(x + base + lane * PER_LANE);
        const E *e = reinterpret_cast<const E *>(&raw);
        uint32_t bits = 0;
#pragma unroll
        for (uint32_t k = 0; k < PER_LANE; ++k) bits |= (is_event(e[k]) ? 1u : 0u) << k;
        // PER_LANE bits per lane -> 32 / PER_LANE lanes make one word
        constexpr uint32_t LANES_PER_WORD = 32 / PER_LANE;
        uint32_t word = bits << (PER_LANE * (lane % LANES_PER_WORD));
#pragma unroll
        for (uint32_t o = 1; o < LANES_PER_WORD; o <<= 1) word |= __shfl_xor_sync(FULL_MASK, word, o);
        if (lane % LANES_PER_WORD == 0) mask[base / 32 + lane / LANES_PER_WORD] = word;
    }
    const uint32_t n_words = (n + 31u) >> 5;
    for (uint32_t w = n_vec / 32 + warp; w < n_words; w += n_warps) {
        const uint32_t i = w * 32u + lane;
        const uint32_t bits = __ballot_sync(FULL_MASK, (i < n) && is_event(x[i]));
        if (lane == 0) mask[w] = bits;
    }
}

}  // namespace bpl

#endif  // BPL_CSRC_COMMON_CUH_
