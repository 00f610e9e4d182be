// Prior samples drawn on the device, straight into a prior cache -- the
// producer of the reference's prior cache (JokerPrior.sample,
// thejoker/prior.py:297-407, with UniformLog / Kipping13Global of
// thejoker/distributions.py:19-28, 171-176) without the host draw, the
// HDF5 round trip and the upload.
//
// Random numbers: Philox4x32-10 (J. K. Salmon, M. A. Moraes, R. O. Dror and
// D. E. Shaw, "Parallel random numbers: as easy as 1, 2, 3", SC11, 2011), a
// counter-based generator: sample g's draws come from counters
// (g_lo, g_hi, block, STREAM_TAG) under key (seed_lo, seed_hi), so every
// sample is reproducible from (seed, g) whatever the launch shape.  Each
// block yields two 64-bit halves, each one uniform: a double
// u = (x >> 11) 2^-53 for P and the angles, a float with 24 significant bits
// for the rest.  Per sample, in order: u_P, u_omega, u_M0, [one Box-Muller
// pair for ln s], then the two gamma variates of the beta draw.
//   P     = P_min (P_max / P_min)^u_P                          (62-bit fixed
//           point, rounded to FP64; FP64 where P leaves the normal numbers)
//   omega = 2 pi u_omega,  M0 = 2 pi u_M0                      (FP64)
//   e     = X / (X + Y),  X ~ Gamma(alpha), Y ~ Gamma(beta)   (Marsaglia and
//           Tsang, ACM TOMS 26, 2000; shape < 1 through
//           Gamma(a) = Gamma(a + 1) U^(1/a))                   (FP32)
//   s     = s_value, or exp(s_mu + s_sigma z)                  (FP32)
// The beta and log-normal draws run in FP32: they are random draws whose
// distribution FP32 rounding does not change measurably, and FP64 (1/74 of
// the FP32 rate here) made them the bound of the kernel.  So did exp in FP64:
// 2^24 samples with the packed copy took 1314 us, with the period in fixed
// point, the tries in step and quick acceptance tests 929 us.
#include "joker_internal.cuh"
#include "joker_math.cuh"
#include "joker_fixed.cuh"
#include <cmath>

namespace joker {

namespace {
constexpr uint32_t PH_M0 = 0xD2511F53u, PH_M1 = 0xCD9E8D57u;
constexpr uint32_t PH_W0 = 0x9E3779B9u, PH_W1 = 0xBB67AE85u;
constexpr uint32_t STREAM_TAG = 0x4A6F6B72u;
constexpr int GAMMA_MAX_TRIES = 64;
}  // namespace

__host__ __device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)PH_M0 * c[0], p1 = (uint64_t)PH_M1 * c[2];
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k0, n1 = (uint32_t)p1;
        const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k1, n3 = (uint32_t)p0;
        c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
        k0 += PH_W0;
        k1 += PH_W1;
    }
}

// The constants of a gamma variate's rejection loop, made once per launch.
struct GammaShape {
    float d, c, ia;
    bool boost;

    explicit GammaShape(float a) {
        boost = a < 1.0f;
        const float k = boost ? a + 1.0f : a;
        d = k - 1.0f / 3.0f;
        c = 1.0f / sqrtf(9.0f * d);
        ia = 1.0f / a;
    }
    // log u < x^2 / 2 + d (1 - v + log v).  The hardware logarithms (2^-21 of
    // log u at most and of log v away from 1, 2^-21.4 there) decide where the
    // sides differ by more than they can be off, and by the roundings.
    __device__ __forceinline__ bool accept(float u, float x2, float v) const {
        const float lu = __logf(u), lv = __logf(v);
        const float right = 0.5f * x2 + d * (1.0f - v + lv);
        const float gap = lu - right;
        if (fabsf(gap) > 4e-6f * (1.0f - lu + x2 + d * (1.0f + v + fabsf(lv)))) return gap < 0.0f;
        return logf(u) < 0.5f * x2 + d * (1.0f - v + logf(v));
    }
};

// Sequential uniforms of one sample.
struct SampleRng {
    uint32_t g_lo, g_hi, k0, k1, block;
    uint64_t spare;
    bool have_spare;

    __device__ void init(uint64_t seed, uint64_t g) {
        g_lo = (uint32_t)g; g_hi = (uint32_t)(g >> 32);
        k0 = (uint32_t)seed; k1 = (uint32_t)(seed >> 32);
        block = 0;
        have_spare = false;
    }
    // the next 64-bit half of the sample's Philox stream
    __device__ uint64_t bits() {
        if (have_spare) { have_spare = false; return spare; }
        uint32_t c[4] = {g_lo, g_hi, block++, STREAM_TAG};
        philox4x32_10(c, k0, k1);
        spare = ((uint64_t)c[3] << 32) | c[2];
        have_spare = true;
        return ((uint64_t)c[1] << 32) | c[0];
    }
    // 53 bits m of the uniform m 2^-53
    __device__ uint64_t uniform53() { return bits() >> 11; }
    // 2 pi times it (the scale's power of two is exact)
    __device__ double angle() { return (double)uniform53() * (TWO_PI_D * 0x1.0p-53); }
    // A uniform float in (0, 1): the 24 bits of x / 2^64 below its leading
    // one, so the resolution follows the magnitude (down to 2^-64) and
    // log u reaches -44 (a Box-Muller normal is not cut off at 5.8 sigma).
    // Integer operations only.
    __device__ float uniform_f() {
        const uint64_t x = bits();
        if (x == 0) return 0x1.0p-65f;
        const int lz = __clzll(x);
        const uint32_t m = (uint32_t)((x << lz) >> 40);
        return __uint_as_float(((uint32_t)(126 - lz) << 23) | (m & 0x7fffffu));
    }
    // standard normal (Box-Muller in FP32; the second variate of the pair is dropped)
    __device__ float normal_f() {
        const float u1 = uniform_f();
        const float u2 = uniform_f();
        float s, c;
        sincospif(2.0f * u2, &s, &c);
        return sqrtf(-2.0f * logf(u1)) * c;
    }
    // Gamma(a, 1) in FP32, a > 0, from at most `tries` of the rejection loop;
    // *ok = false if it ran out of them
    __device__ float gamma_f(const GammaShape &a, int tries, bool *ok) {
        float v = 0.0f;
        bool got = false;
        for (int t = 0; t < tries && !got; ++t) {
            const float x = normal_f();
            const float w = fmaf(a.c, x, 1.0f);
            if (tries > 1 && w <= 0.0f) continue;
            v = w * w * w;
            const float u = uniform_f();
            const float x2 = x * x;
            got = w > 0.0f && ((u < 1.0f - 0.0331f * x2 * x2) || a.accept(u, x2, v));
        }
        if (!got) *ok = false;
        float g = a.d * v;
        if (a.boost) g *= powf(uniform_f(), a.ia);
        return g;
    }
};

// The period's range as powers of two: P = 2^(n0 + f0 + u (ns + fs)), f0 in
// Q62, fs in Q64; fixed: every P of the range is a normal number.
struct PeriodScale {
    int64_t f0;
    uint64_t fs;
    int32_t n0, ns, fixed;
};

static PeriodScale period_scale(double P_min, double P_max) {
    const long double y0 = log2l((long double)P_min), y1 = log2l((long double)P_max);
    PeriodScale r;
    r.fixed = y0 > -1020.0L && y1 < 1020.0L;
    const long double n0 = floorl(y0), ns = floorl(y1 - y0);
    r.n0 = (int32_t)n0;
    r.ns = (int32_t)ns;
    r.f0 = (int64_t)((y0 - n0) * 0x1p62L);
    r.fs = (uint64_t)((y1 - y0 - ns) * 0x1p63L) << 1;
    return r;
}

__device__ __forceinline__ double draw_period(const PeriodScale &s, uint64_t m) {
    const uint64_t a = m * (uint32_t)s.ns;                            // Q53
    const uint64_t f = (uint64_t)s.f0 + ((a << 9) & (uint64_t)(fx::ONE62 - 1)) +
                       (fx::hi64(m << 11, s.fs) >> 2);                // Q62, below 3
    return fx::exp2_fixed(s.n0 + (int)(a >> 53) + (int)(f >> 62),
                          (int64_t)(f & (uint64_t)(fx::ONE62 - 1)));
}

// A float as a double, without the FP64 pipe (zero and normal numbers).
__device__ __forceinline__ double widen(float x) {
    const uint32_t b = __float_as_uint(x);
    if ((b & 0x7f800000u) == 0u || (b & 0x7f800000u) == 0x7f800000u) return (double)x;
    return __longlong_as_double((long long)(((uint64_t)(b & 0x80000000u) << 32) |
                                            (((uint64_t)(b & 0x7fffffffu) << 29) +
                                             (896ull << 52))));
}

struct PriorOut {
    double *P, *E, *OM, *M0, *S;
    float4 *mx_a, *mx_b;
    float *mx_s2;
    double *packed;
    int *bad;
};

// Sample first_index + i into row row0 + i.  With one try a sample whose gamma
// variates were rejected is left (false): its draws beyond that try are not
// those of the stream.
template <int TRIES>
__device__ __forceinline__ bool draw_sample(const joker_prior_spec &spec, const PeriodScale &scale,
                                            const GammaShape &ga, const GammaShape &gb,
                                            double lpmin, double lspan, uint64_t seed,
                                            int64_t first_index, int64_t row0, int64_t i,
                                            const PriorOut &o) {
    SampleRng rng;
    rng.init(seed, (uint64_t)(first_index + i));
    const uint64_t mp = rng.uniform53();
    const double om = rng.angle();
    const double m0 = rng.angle();
    double s = spec.s_value;
    if (spec.s_kind == JOKER_S_LOGNORMAL)
        s = widen(expf(fmaf((float)spec.s_sigma, rng.normal_f(), (float)spec.s_mu)));
    bool ok = true;
    const float x = rng.gamma_f(ga, TRIES, &ok);
    const float y = rng.gamma_f(gb, TRIES, &ok);
    if (TRIES == 1 && !ok) return false;
    const double p = scale.fixed ? draw_period(scale, mp)
                                 : exp(fma((double)mp * 0x1.0p-53, lspan, lpmin));
    const float ef = x / (x + y);
    double e = widen(ef);
    if (!ok || !(ef >= 0.0f && ef < 1.0f)) {
        atomicAdd(o.bad, 1);
        e = e >= 1.0 ? 0x1.fffffffffffffp-1 : (e >= 0.0 ? e : 0.0);
    }
    const int64_t r = row0 + i;
    o.P[r] = p; o.E[r] = e; o.OM[r] = om; o.M0[r] = m0; o.S[r] = s;
    float4 pa, pb;
    float s2;
    prepare_sample(p, e, om, m0, s, pa, pb, s2);
    o.mx_a[r] = pa;
    o.mx_b[r] = pb;
    o.mx_s2[r] = s2;
    if (o.packed) {
        double *q = o.packed + i * 5;
        q[0] = p; q[1] = e; q[2] = om; q[3] = m0; q[4] = s;
    }
    return true;
}

constexpr int PRIOR_BLOCK = 256;

// Every sample takes one try of each gamma variate, in step: all lanes then use
// the same halves of their Philox blocks.  The few (about one in twenty) that a
// try rejects are listed and drawn again from their first counter, whole
// blocks of them at a time.  With the rejection loop inside, nearly every warp
// ran it two or three times for one or two lanes, and lanes whose tries
// differed computed each Philox block apart.
__global__ void __launch_bounds__(PRIOR_BLOCK)
prior_sample_kernel(joker_prior_spec spec, PeriodScale scale, GammaShape ga, GammaShape gb,
                    uint64_t seed, int64_t first_index, int64_t n, int64_t row0, PriorOut o) {
    __shared__ int64_t again[2 * PRIOR_BLOCK];
    __shared__ int n_again;
    const double lpmin = scale.fixed ? 0.0 : log(spec.P_min);
    const double lspan = scale.fixed ? 0.0 : log(spec.P_max) - lpmin;
    if (threadIdx.x == 0) n_again = 0;
    __syncthreads();
    for (int64_t base = blockIdx.x * (int64_t)PRIOR_BLOCK; base < n;
         base += (int64_t)gridDim.x * PRIOR_BLOCK) {
        const int64_t i = base + threadIdx.x;
        if (i < n && !draw_sample<1>(spec, scale, ga, gb, lpmin, lspan, seed, first_index,
                                                row0, i, o))
            again[atomicAdd(&n_again, 1)] = i;                // at most 2 PRIOR_BLOCK - 1
        __syncthreads();
        const int have = n_again;
        const bool last = base + (int64_t)gridDim.x * PRIOR_BLOCK >= n;
        if (have >= PRIOR_BLOCK || last) {
            const int first = have >= PRIOR_BLOCK ? have - PRIOR_BLOCK : 0;
            for (int k = first + threadIdx.x; k < have; k += PRIOR_BLOCK)
                draw_sample<GAMMA_MAX_TRIES>(spec, scale, ga, gb, lpmin, lspan, seed, first_index,
                                             row0, again[k], o);
            if (last && first > (int)threadIdx.x)
                draw_sample<GAMMA_MAX_TRIES>(spec, scale, ga, gb, lpmin, lspan, seed, first_index,
                                             row0, again[threadIdx.x], o);
            __syncthreads();
            if (threadIdx.x == 0) n_again = first;
        }
        __syncthreads();
    }
}

cudaError_t launch_prior_sample(const joker_prior_spec &spec, uint64_t seed, int64_t first_index,
                                int64_t n, int64_t row0, double *P, double *E, double *OM,
                                double *M0, double *S, float4 *mx_a, float4 *mx_b, float *mx_s2,
                                double *packed, int *bad, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int64_t blocks = (n + PRIOR_BLOCK - 1) / PRIOR_BLOCK;
    if (blocks > 152 * 16) blocks = 152 * 16;
    const PriorOut o = {P, E, OM, M0, S, mx_a, mx_b, mx_s2, packed, bad};
    prior_sample_kernel<<<(int)blocks, PRIOR_BLOCK, 0, st>>>(
        spec, period_scale(spec.P_min, spec.P_max), GammaShape((float)spec.e_alpha),
        GammaShape((float)spec.e_beta), seed, first_index, n, row0, o);
    count_launch();
    return cudaGetLastError();
}

}  // namespace joker
