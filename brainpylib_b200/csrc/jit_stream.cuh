// The random stream of one row (or column) of a just-in-time matrix, several connections at a time.
//
// Scheme (must stay bit-identical to the reference, whose sampled connectivity is the contract): cuRAND XORWOW,
// `curand_init(seed + i, 0, 0)`; the next connection lies `(int) ceil(log(curand_uniform(&st)) / log_p)` positions on
// (float logarithm, division in double, lib/gpu_jitconn_matvec.cu:99-106), and its weight is drawn after its position:
// uniform `(T)(u * w_range + w_min)` (one draw), normal `(T)(n * w_sigma + w_mu)` with cuRAND's Box-Muller pairs (two
// draws on every other connection), evaluated in double (lib/gpu_jitconn_matvec.cu:243,386).
//
// What bounds the walk: instruction issue when all SMs are full of streams, the latency of one connection (state ->
// draw -> logarithm -> position -> test) when they are not.  A walk therefore takes a batch of connections per iteration.
// The draws of a batch depend on the generator's state alone, so their conversions, logarithms and gathers overlap; the
// five state words go round inside the batch without register moves; and one loop test serves the batch.  Connections
// drawn behind the end of a stream are dropped: nobody else reads it.
#ifndef BPL_CSRC_JIT_STREAM_CUH_
#define BPL_CSRC_JIT_STREAM_CUH_

#include <curand_kernel.h>

#include <cmath>
#include <cstdint>

namespace bpl {
namespace {

enum { W_HOMO = 0, W_UNIFORM = 1, W_NORMAL = 2 };

// Constants of the gap computation, made on the host once per call.
struct GapParams {
    double log_p;
    float inv_log_p;           // float(1 / log_p)
    float lo_scale, hi_scale;  // ln 2 / log_p, less and more the relative error
    float margin;              // the absolute error
    bool quick;                // the two-sided test below is in its range
    // 1, 2 and 16: shifts and additions as multiplications by a value that the compiler does not know run in the
    // multiply pipe, beside the logic pipe, which a walk fills first (half an instruction per clock)
    uint32_t one, two, sixteen;
};

// The gap is (int) ceil(log(u) / log_p): float logarithm, double division.  With L = lg2.approx(u), over all 2^32 draws (on the
// hardware: a test takes the largest share of it, 0.78)
//     |L ln2 - log(u)| <= LOG_ABS + LOG_REL |L ln2|,
// the error of the float logarithm included, so that the reference's quotient lies between the two ends
//     L ln2 / log_p (1 -+ LOG_REL) -+ LOG_ABS / |log_p|,
// whose roundings go outwards.  Adding 2^23 with rounding up leaves 2^23 + ceil() in the mantissa; where both ends agree that is
// the reference's gap.  Else (1 draw in 1400 at a mean gap of 1000) the reference's own logarithm decides, and where that lies
// too close to an integer, the reference's own expression.  (With the errors that the PTX ISA and CUDA bound, 1 draw in 700, and a
// walk over 1e9 events of uniform weights 1393 us instead of 1353.  Settling a lane's open draws in a loop with one place where
// the logarithm is taken: 1446 us.)
// `n`: length of a stream's range; a batch may run at most 8 gaps behind it (below 2^25 positions).
constexpr double LOG_ABS = 1.8 / 16777216.0, LOG_REL = 4.2 / 16777216.0;
inline GapParams gap_params(double log_p, uint32_t n) {
    GapParams g;
    g.one = 1u;
    g.two = 2u;
    g.sixteen = 16u;
    g.log_p = log_p;
    g.inv_log_p = static_cast<float>(1.0 / log_p);
    const double scale = 0.69314718055994530942 / log_p;
    const auto rounded = [](const double v, const float towards, const bool inwards) {     // to float, away from or towards 0
        const float f = static_cast<float>(v);
        return (std::fabs(static_cast<double>(f)) > std::fabs(v)) == inwards ? std::nextafterf(f, towards) : f;
    };
    g.lo_scale = rounded(scale * (1.0 - LOG_REL), 0.0f, true);
    g.hi_scale = rounded(scale * (1.0 + LOG_REL), -INFINITY, false);
    g.margin = rounded(-LOG_ABS / log_p, INFINITY, false);
    // |log(u)| < 23: q stays below 2^22, where the sums are exact in their integer part
    g.quick = log_p < 0.0 && -1.0 / log_p < 180000.0 && n < 0xfe000000u;
    return g;
}

__device__ __forceinline__ float lg2_approx(float u) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(u));
    return r;
}

__device__ __noinline__ int gap_exact(const float u, const double log_p, const float inv_log_p) {
    const float lg = log(u);
    // off from the reference's quotient by two float roundings (2^-23 q); rint by adding 1.5 * 2^23
    const float q = lg * inv_log_p;
    const float t = q + 12582912.0f;
    const float frac = q - (t - 12582912.0f);
    if (q < 4194304.0f && fabsf(frac) > q * 1.5e-7f) return (__float_as_int(t) - 0x4B400000) + (frac > 0.0f ? 1 : 0);
    return (int) ceil(lg / log_p);
}

// Both ends of a draw's gap, for `quick` parameters: 2^23 + the gap where they are equal.
__device__ __forceinline__ float gap_low(const float L, const GapParams &g) {
    return __fadd_ru(__fmaf_rd(L, g.lo_scale, -g.margin), 8388608.0f);
}
__device__ __forceinline__ float gap_high(const float L, const GapParams &g) {
    return __fadd_ru(__fmaf_ru(L, g.hi_scale, g.margin), 8388608.0f);
}
constexpr int GAP_ZERO = 0x4B000000;    // the bits of 2^23

__device__ __forceinline__ int gap_of(const uint32_t x, const GapParams &g) {
    const float u = _curand_uniform(x), L = lg2_approx(u), lo = gap_low(L, g);
    if (lo == gap_high(L, g)) return __float_as_int(lo) - GAP_ZERO;
    return gap_exact(u, g.log_p, g.inv_log_p);
}

// The next position of a stream of any parameters, for walks that take one connection at a time; the end is sticky.
__device__ __forceinline__ uint32_t next_position(const uint32_t pos, const uint32_t x, const GapParams &g) {
    if (g.quick) return pos + static_cast<uint32_t>(gap_of(x, g));
    const double q = ceil(log(_curand_uniform(x)) / g.log_p);
    return q >= 0.0 && q < 4294967295.0 - pos ? pos + static_cast<uint32_t>(q) : 0xffffffffu;
}

// XORWOW (G. Marsaglia, "Xorshift RNGs", J. Stat. Software 8(14), 2003: the generator of section 3.1 with the Weyl
// sequence), on a state that cuRAND has seeded.
struct Xorwow {
    uint32_t v0, v1, v2, v3, v4, d;
    __device__ __forceinline__ void seed(const uint32_t s) {
        curandState st;
        curand_init(s, 0, 0, &st);
        v0 = st.v[0]; v1 = st.v[1]; v2 = st.v[2]; v3 = st.v[3]; v4 = st.v[4];
        d = st.d;
    }
    __device__ __forceinline__ uint32_t next(const GapParams &g) {
        const uint32_t t = v0 ^ (v0 >> 2);
        v0 = v1; v1 = v2; v2 = v3; v3 = v4;
        v4 = (v4 ^ (v4 * g.sixteen)) ^ (t ^ (t * g.two));
        d += 362437u;
        return v4 + d;
    }
};

// Weights from raw draws, by cuRAND's own conversions; `second`: the other value of a pair.
template<typename T>
__device__ __forceinline__ T uniform_weight(const uint32_t x, const double w1, const double w2) {
    return (T) (_curand_uniform(x) * w2 + w1);
}
template<typename T>
__device__ __forceinline__ T normal_weight(const uint32_t x, const uint32_t y, const bool second, const double w1,
                                           const double w2) {
    const float2 v = _curand_box_muller(x, y);
    return (T) ((second ? v.y : v.x) * w2 + w1);
}

// One batch of connections: positions and the raw draws of their weights.  QUICK = false: parameters outside gap_of's
// range or streams too long for sums of gaps to stay below 2^32; the reference's expression for every draw, and a
// position behind the end (`n`) stays there.
// COUNT is even for normal weights, so that a batch starts with a new pair.
// SUMS: for walks that are bound by instruction issue, how the open draws are found (below).
template<int KIND, bool QUICK, int COUNT = KIND == W_NORMAL ? 4 : 5, bool SUMS = false>
struct Batch {
    static constexpr int N = COUNT;
    uint32_t pos[N];
    uint32_t raw[KIND == W_HOMO ? 1 : N];

    // LOW24: positions below 2^24, whose upper 8 bits are left undefined in pos[]; a stream that is through stays at n, so
    // that a batch reaches n + COUNT gaps at most
    template<bool LOW24 = false>
    __device__ __forceinline__ void draw(Xorwow &s, uint32_t &at, const uint32_t n, const GapParams &g) {
        uint32_t x[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            x[j] = s.next(g);
            if (KIND == W_UNIFORM) raw[j] = s.next(g);
            if (KIND == W_NORMAL && (j & 1) == 0) {
                raw[j] = s.next(g);
                raw[j + 1] = s.next(g);
            }
        }
        if (QUICK) {
            // One branch for the batch: the draws that gap_low and gap_high leave open are settled behind it.  SUMS: an upper end
            // is never below its lower one, so the sums of both are equal where all are, and additions, written as multiplications,
            // keep the logic pipe free of a comparison per draw: homogeneous event rows 1049 -> 985 us.  They stand in the chain
            // of positions, though: columns of events, which wait for their chains and for L2, 141 -> 143 us.
            float lo[N], hi[N];
            const uint32_t from = at;
            uint32_t upper = LOW24 ? from : from - static_cast<uint32_t>(N) * static_cast<uint32_t>(GAP_ZERO);
            bool open = false;
            auto advance = [&](const int j) {
                if (LOW24) at = static_cast<uint32_t>(__float_as_int(lo[j])) * g.one + at;
                else at += static_cast<uint32_t>(__float_as_int(lo[j]) - GAP_ZERO);
                pos[j] = at;
            };
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const float L = lg2_approx(_curand_uniform(x[j]));
                lo[j] = gap_low(L, g);
                hi[j] = gap_high(L, g);
                if (SUMS) {
                    advance(j);
                    upper = static_cast<uint32_t>(__float_as_int(hi[j])) * g.one + upper;
                } else {
                    open |= lo[j] != hi[j];
                }
            }
            if (SUMS ? at != upper : open) {
                at = from;
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    if (lo[j] != hi[j])
                        lo[j] = __int_as_float(gap_exact(_curand_uniform(x[j]), g.log_p, g.inv_log_p) + GAP_ZERO);
                    if (SUMS) advance(j);
                }
            }
            if (!SUMS) {
#pragma unroll
                for (int j = 0; j < N; ++j) advance(j);
            }
            if (LOW24) at = min(at & 0xffffffu, n);
        } else {
#pragma unroll
            for (int j = 0; j < N; ++j) {
                if (j == 0 || at < n) at = next_position(at, x[j], g);
                pos[j] = at;
            }
        }
    }
    // the weights of all connections (homogeneous: none)
    template<typename T>
    __device__ __forceinline__ void weights(T (&w)[N], const double w1, const double w2) const {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (KIND == W_UNIFORM) w[j] = uniform_weight<T>(raw[j], w1, w2);
            if (KIND == W_NORMAL && (j & 1) == 0) {
                const float2 v = _curand_box_muller(raw[j], raw[j + 1]);
                w[j] = (T) (v.x * w2 + w1);
                w[j + 1] = (T) (v.y * w2 + w1);
            }
        }
    }
};

// One stream walked by GROUP lanes together, GROUP connections per step, one each: where there are too few streams to fill
// the SMs, the walk of one is a chain of some 1000 clocks per four connections (draws, logarithms, weights, all by one
// lane).  Here every lane of the group runs the generator (the same instructions), and each converts its own connection;
// the positions are a prefix sum over the group.  Four times the instructions per connection, a third of the time per
// stream while issue slots are idle.  For `quick` parameters; all 32 lanes of the warp must call draw together.
constexpr int GROUP = 8;

template<int KIND>
struct GroupStep {
    uint32_t pos;              // of this lane's connection
    uint32_t r0, r1;           // raw draws of its weight (normal: of its pair)

    __device__ __forceinline__ void draw(Xorwow &s, uint32_t &at, const uint32_t n, const uint32_t sub, const GapParams &g) {
        uint32_t x = 0;
        r0 = r1 = 0;
#pragma unroll
        for (int j = 0; j < GROUP; ++j) {
            const uint32_t d = s.next(g);
            if (sub == j) x = d;
            if (KIND == W_UNIFORM) {
                const uint32_t r = s.next(g);
                if (sub == j) r0 = r;
            }
            if (KIND == W_NORMAL && (j & 1) == 0) {
                const uint32_t a = s.next(g), b = s.next(g);
                if ((sub & ~1u) == j) {
                    r0 = a;
                    r1 = b;
                }
            }
        }
        uint32_t sum = static_cast<uint32_t>(gap_of(x, g));
#pragma unroll
        for (int o = 1; o < GROUP; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, sum, o, GROUP);
            if (sub >= static_cast<uint32_t>(o)) sum += t;
        }
        pos = at + sum;
        at = min(__shfl_sync(0xffffffffu, pos, GROUP - 1, GROUP), n);     // (a stream that is through stays at its end)
    }
    template<typename T>
    __device__ __forceinline__ T weight(const uint32_t sub, const double w1, const double w2) const {
        if (KIND == W_UNIFORM) return uniform_weight<T>(r0, w1, w2);
        if (KIND == W_NORMAL) return normal_weight<T>(r0, r1, sub & 1u, w1, w2);
        return T(1);
    }
};

}  // namespace
}  // namespace bpl

#endif  // BPL_CSRC_JIT_STREAM_CUH_
