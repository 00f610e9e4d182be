// FP64 per-sample marginal likelihood, shared by the FP64 kernel and the
// refinement step of the acceptance pass (both must give identical numbers).
#pragma once
#include "joker_internal.cuh"
#include "joker_math.cuh"
#include "joker_fixed.cuh"

namespace joker {

// Natural log of a positive double for the FP64-tail variant of the mixed
// path: exact binary exponent, FP32 logf of the mantissa in [1, 2).
__device__ __forceinline__ double log_mixed(double x) {
    const int hi = __double2hiint(x);
    const int ex = ((hi >> 20) & 0x7ff) - 1023;
    const double m = __hiloint2double((hi & 0x800fffff) | 0x3ff00000, __double2loint(x));
    if (ex == -1023 || ex == 1024) return log(x);   // zero, subnormal, inf, NaN
    return (double)ex * 0.69314718055994530942 + (double)logf((float)m);
}

// One Keplerian orbit in FP64: the unit-K radial velocity
//   m(dt) = cos(omega + f) + e cos(omega),  M = 2 pi dt / P - M0,
// in terms of the eccentric anomaly, m = (A cos E + B sin E - D)/(1 - e cos E) + D
// with A = cos omega, B = -sin omega sqrt(1 - e^2), D = e cos omega (the model
// twobody's c_rv_from_elements evaluates for thejoker/src/fast_likelihood.pyx
// :453-455).
struct OrbitF64 {
    double e, Ac, Bc, Dc, k2p, M0;
    float ef, omef, a1f;                 // the Kepler solver's FP32 constants

    __device__ __forceinline__ void init(double P, double e_, double om, double M0_) {
        e = e_;
        M0 = M0_;
        k2p = TWO_PI_D / P;                  // correctly rounded: it scales every phase
        double sw, cw;
        sincos_f64_table(om, sw, cw);
        Ac = cw;
        Bc = -sw * sqrt((1.0 - e) * (1.0 + e));
        Dc = e * cw;
        kepler_consts_f32(e, ef, omef, a1f);
    }

    __device__ __forceinline__ double rv_unit(double dt) const {
        double M = fma(dt, k2p, -M0);
        const double nrev = rint(M * INV_TWO_PI_D);
        M = fma(-nrev, TWO_PI_HI_D, M);
        M = fma(-nrev, TWO_PI_LO_D, M);
        double sE, cE;
        kepler_sincos_f64(M, e, ef, omef, a1f, sE, cE);
        return fma(fma(Ac, cE, fma(Bc, sE, -Dc)), rcp_newton(fma(-e, cE, 1.0)), Dc);
    }
};

// Per-sample FP64 state: the epoch sums and the sample's constants.
template <int L, bool JIT>
struct Acc64 {
    OrbitF64 orb;
    double s2, mu0;
    double A00, b0, A0[MAXL];            // no jitter
    double G[L][L], q[L], rWr;           // jitter: full system
    // jitter: prod_j (1 + s^2 ivar_j) = pj 2^ej (pj in [1, 2) after each
    // epoch) plus slog, the logs already summed (warp_sum); sum log w_j is
    // sum log ivar_j - log of the product.
    double pj, slog;
    int ej;

    __device__ __forceinline__ void init(const StarRec &st, double P, double e_, double om,
                                         double M0_, double s_) {
        orb.init(P, e_, om, M0_);
        s2 = s_ * s_;
        mu0 = st.mu0;
        A00 = 0.0;
        b0 = 0.0;
#pragma unroll
        for (int k = 0; k < MAXL; ++k) A0[k] = 0.0;
        rWr = 0.0;
        pj = 1.0;
        slog = 0.0;
        ej = 0;
        if (JIT) {
#pragma unroll
            for (int i = 0; i < L; ++i) {
                q[i] = 0.0;
#pragma unroll
                for (int k = 0; k < L; ++k) G[i][k] = 0.0;
            }
        }
    }

    // one epoch: dt = t - t_ref, y' = y - sum_{j>=1} mu_j T_j, ivar, T_1..T_{L-1}
    __device__ __forceinline__ void add(double dt, double yp, double iv, const double *T) {
        const double m = orb.rv_unit(dt);
        if (!JIT) {
            const double wm = iv * m;
            A00 = fma(wm, m, A00);
            b0 = fma(wm, yp, b0);
#pragma unroll
            for (int k = 1; k < L; ++k) A0[k] = fma(wm, T[k - 1], A0[k]);
        } else {
            const double dj = fma(s2, iv, 1.0);
            const double wj = iv * rcp_newton(dj);
            // pj *= dj, then the binary exponent moves to ej (integer ops);
            // dj >= 1 keeps pj >= 1, a positive normal number
            pj *= dj;
            const int hi = __double2hiint(pj);
            ej += (hi >> 20) - 1023;
            pj = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(pj));
            double x[L];
            x[0] = m;
#pragma unroll
            for (int k = 1; k < L; ++k) x[k] = T[k - 1];
            const double r = fma(-mu0, m, yp);
            rWr = fma(wj * r, r, rWr);
#pragma unroll
            for (int ii = 0; ii < L; ++ii) {
                const double wx = wj * x[ii];
                q[ii] = fma(wx, r, q[ii]);
#pragma unroll
                for (int k = 0; k <= ii; ++k) G[ii][k] = fma(wx, x[k], G[ii][k]);
            }
        }
    }

    // Sum the epoch sums of the 32 lanes of a warp (every lane gets the total).
    __device__ __forceinline__ void warp_sum() {
        if (!JIT) {
            A00 = wsum(A00);
            b0 = wsum(b0);
#pragma unroll
            for (int k = 1; k < L; ++k) A0[k] = wsum(A0[k]);
        } else {
            rWr = wsum(rWr);
            slog = wsum(log_prod());
            pj = 1.0;
            ej = 0;
#pragma unroll
            for (int ii = 0; ii < L; ++ii) {
                q[ii] = wsum(q[ii]);
#pragma unroll
                for (int k = 0; k <= ii; ++k) G[ii][k] = wsum(G[ii][k]);
            }
        }
    }

    // sum_j log(1 + s^2 ivar_j) over the epochs this accumulator has seen
    __device__ __forceinline__ double log_prod() const {
        return fma((double)ej, 0.69314718055994530942, slog + log(pj));
    }

    // sum_j log w_j, w_j = ivar_j / (1 + s^2 ivar_j)
    __device__ __forceinline__ double sum_log_w(const StarRec &st) const {
        return st.sum_log_ivar - log_prod();
    }

    static __device__ __forceinline__ double wsum(double x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    }

    __device__ __forceinline__ double finish(const StarRec &st, double P) const;
};

// Schur-complement tail (no jitter), FP64.
template <int L, bool MIXED_LOG>
__device__ __forceinline__ double tail_schur_d(const StarRec &st, double A00, const double *A0,
                                               double b0, double lam0, double log_lam0) {
    double gv = 0.0, gcC = 0.0;
#pragma unroll
    for (int j = 1; j < L; ++j) {
        double vj = 0.0;
#pragma unroll
        for (int k = 1; k < L; ++k) vj = fma(st.Cinv[j * MAXL + k], A0[k], vj);
        gv = fma(A0[j], vj, gv);
        gcC = fma(A0[j], st.cC[j], gcC);
    }
    const double a_minus = A00 - gv;           // s - 1/Lambda0
    const double u = b0 - gcC;
    const double mu0 = st.mu0;
    const double t = fma(-mu0, a_minus, u);
    double chi2 = st.chi2_0;
    if (mu0 != 0.0) chi2 = fma(mu0 * mu0, a_minus, fma(-2.0 * mu0, u, chi2));
    if constexpr (MIXED_LOG) {
        const double s = a_minus + 1.0 / lam0;
        chi2 -= t * t / s;
        return -0.5 * (chi2 + st.logdet_const + log_lam0 + log_mixed(s));
    } else {
        // Lambda0 s = Lambda0 (s - 1/Lambda0) + 1: t^2 / s and log Lambda0 + log s
        // from one reciprocal and one log
        const double ls = fma(lam0, a_minus, 1.0);
        chi2 = fma(-t * t * lam0, rcp_newton(ls), chi2);
        return -0.5 * (chi2 + st.logdet_const + log(ls));
    }
}

// Full tail (jitter applied), FP64: LDL^T of G, quadratic form, log det.
// logdet_const + log(scale * det G) is the log-determinant term.
template <int L, bool MIXED_LOG>
__device__ __forceinline__ double tail_full_d(const double (&G)[L][L], const double (&q)[L],
                                              double rWr, double logdet_const,
                                              double scale = 1.0) {
    double D[L], rD[L], Lw[L][L];
    double quad = 0.0, detp = 1.0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        double dk = G[k][k];
#pragma unroll
        for (int m = 0; m < k; ++m) dk = fma(-Lw[k][m] * Lw[k][m], D[m], dk);
        D[k] = dk;
        const double rdk = rcp_newton(dk);
        rD[k] = rdk;
#pragma unroll
        for (int i = k + 1; i < L; ++i) {
            double v = G[i][k];
#pragma unroll
            for (int m = 0; m < k; ++m) v = fma(-Lw[i][m] * Lw[k][m], D[m], v);
            Lw[i][k] = v * rdk;
        }
        detp *= dk;
    }
    double z[L];
#pragma unroll
    for (int k = 0; k < L; ++k) {
        double v = q[k];
#pragma unroll
        for (int m = 0; m < k; ++m) v = fma(-Lw[k][m], z[m], v);
        z[k] = v;
        quad = fma(v * v, rD[k], quad);
    }
    const double logdet = logdet_const + (MIXED_LOG ? log_mixed(detp) : log(scale * detp));
    return -0.5 * (rWr - quad + logdet);
}

// K prior variance per sample (fast_likelihood.pyx:461-464; clip: at max_K^2)
__device__ __forceinline__ double k_prior_variance(const StarRec &st, double P, double e,
                                                   bool clip = true) {
    if (!st.k_scaled) return st.lam0;
    const double y = rcbrt_newton(P * st.iP0);                  // (P / P0)^(-1/3)
    const double v = st.sigK0sq * (y * y) * rcp_newton(1.0 - e * e);
    return clip ? fmin(st.maxK2, v) : v;
}

template <int L, bool JIT>
__device__ __forceinline__ double Acc64<L, JIT>::finish(const StarRec &st, double P) const {
    const double lam0 = k_prior_variance(st, P, orb.e);
    if constexpr (!JIT) {
        return tail_schur_d<L, false>(st, A00, A0, b0, lam0, 0.0);
    } else {
        double Gs[L][L];
        const double ilam0 = st.k_scaled ? rcp_newton(lam0) : st.ilam[0];
#pragma unroll
        for (int ii = 0; ii < L; ++ii) {
#pragma unroll
            for (int k = 0; k <= ii; ++k) { Gs[ii][k] = G[ii][k]; Gs[k][ii] = G[ii][k]; }
            Gs[ii][ii] += ii == 0 ? ilam0 : st.ilam[ii];
        }
        // log det term: log_norm_rest + log Lambda0 - sum log w + log det G, with
        // -sum log w = -sum log ivar + slog + ej ln 2 + log pj
        return tail_full_d<L, false>(
            Gs, q, rWr,
            fma((double)ej, 0.69314718055994530942, st.log_norm_rest - st.sum_log_ivar + slog),
            lam0 * pj);
    }
}

// A product of numbers in (0, 1], m 2^(e - 62) with m in [2^61, 2^62).  Each
// factor truncates it, so its last bits depend on the factors' order.
struct FxProd {
    int64_t m;
    int32_t e;
    __device__ __forceinline__ void one() { m = fx::ONE62 - 1; e = 0; }
    __device__ __forceinline__ void times(int64_t m2, int32_t e2 = 0) {
        m = fx::mul(fx::split(m), fx::split(m2));
        const int z = fx::clz64((uint64_t)m) - 2;
        m <<= z;
        e += e2 - z;
    }
};

// Per-sample state of the fixed-point form: the integer epoch sums, and the
// same finish as Acc64's from their doubles.  Sums of integers do not depend
// on the order; the jitter's product is kept as four, of epochs i with the same
// i mod 4 in their order, that meet in that of i mod 4.  So every split of the
// epochs over threads gives the same ln L.
//
// With the jitter the weights are w_j = 2^ew g wn_j, g = 1 / (1 + a),
// a = s^2 2^ew, wn_j = v_j / d_j, v_j = ivar_j 2^-ew and
// d_j = v_j + g (1 - v_j) in [v_j, 1], and
// sum log(1 + s^2 ivar_j) = sum log d_j + n log(1 + a).
template <int L, bool JIT>
struct AccFx {
    fx::Orbit orb;
    fx::Sum96 A00, b0, A0[MAXL];             // no jitter; jitter: G00, q0, G0k
    fx::Sum96 G[L][L], q[L], rWr;            // jitter: the rest
    fx::limbs g62;
    double g, a;
    FxProd prod;                             // of the d_j, set before finish

    // False: the sample (or star) needs the FP64 form.
    __device__ __forceinline__ bool init(const StarRec &st, double P, double e, double om,
                                         double M0, double s) {
        orb.clear();                             // sliced_epochs stores bad() of every sample
        A00.zero();
        b0.zero();
#pragma unroll
        for (int k = 0; k < MAXL; ++k) A0[k].zero();
        if (JIT) {
#pragma unroll
            for (int i = 0; i < L; ++i) {
                q[i].zero();
#pragma unroll
                for (int k = 0; k < L; ++k) G[i][k].zero();
            }
            rWr.zero();
            a = s * s * st.fx_w;
            if (!(st.mu0 == 0.0 && a <= 0x1p40)) return false;
            g = rcp_newton(1.0 + a);
            g62 = fx::split(fx::fixed62(g));
        }
        return st.fx_ok && fx::as_exact(st.fx_tsh, P, e) &&
               orb.init(st.fx_tsh, st.fx_t0, P, e, om, M0);
    }

    // One epoch; with the jitter, its d_j (Q62).
    __device__ __forceinline__ int64_t add(const fx::EpochFx &r) {
        const int64_t mq = orb.column(r.t);                            // Q61
        const fx::limbs m = fx::split(mq);
        if (!JIT) {
            const int64_t wmq = fx::mul(r.w, m);                       // Q61
            const fx::limbs wm = fx::split(wmq);
            A00.add(fx::mul(wm, m));                                   // Q60
            b0.add(fx::mul(wm, r.y));                                  // Q61
            if (L > 1) A0[1].add(wmq);                                 // Q61; T_1 = 1
#pragma unroll
            for (int k = 2; k < L; ++k) A0[k].add(fx::mul(wm, r.T[k - 2]));
            return 0;
        } else {
            const int64_t v = fx::join(r.w);
            const int64_t d = fx::clamp62(v + fx::mul(g62, fx::split(fx::ONE62 - v)));
            const int64_t wq = fx::twice(fx::div61(v >> 1, d >> 1));   // Q62
            const fx::limbs w = fx::split(wq);
            const int64_t wmq = fx::mul(w, m), wyq = fx::mul(w, r.y);
            const fx::limbs wm = fx::split(wmq), wy = fx::split(wyq);
            A00.add(fx::mul(wm, m));                                   // Q60
            b0.add(fx::mul(wm, r.y));                                  // Q61
            rWr.add(fx::mul(wy, r.y));                                 // Q62
            if (L > 1) {
                A0[1].add(wmq);                                        // Q61
                G[1][1].add(wq);                                       // Q62
                q[1].add(wyq);                                         // Q62
            }
#pragma unroll
            for (int i = 2; i < L; ++i) {
                const int64_t wTq = fx::mul(w, r.T[i - 2]);
                const fx::limbs wT = fx::split(wTq);
                A0[i].add(fx::mul(wm, r.T[i - 2]));                    // Q61
                G[i][1].add(wTq);                                      // Q62
                q[i].add(fx::mul(wy, r.T[i - 2]));                     // Q62
#pragma unroll
                for (int k = 2; k <= i; ++k) G[i][k].add(fx::mul(wT, r.T[k - 2]));
            }
            return d;
        }
    }

    // f on every sum
    template <class F> __device__ __forceinline__ void each(F f) {
        f(A00);
        f(b0);
#pragma unroll
        for (int k = 1; k < L; ++k) f(A0[k]);
        if (JIT) {
            f(rWr);
#pragma unroll
            for (int i = 1; i < L; ++i) {
                f(q[i]);
#pragma unroll
                for (int k = 1; k <= i; ++k) f(G[i][k]);
            }
        }
    }
    static constexpr int SUMS = 1 + L + (JIT ? L + L * (L - 1) / 2 : 0);
    static constexpr int WORDS = 3 * SUMS + 1 + (JIT ? 1 : 0);           // of a stored state

    // The sums over the 32 lanes of a warp (every lane gets the totals).
    __device__ __forceinline__ void warp_sum() {
        each([](fx::Sum96 &v) { v.warp_sum(); });
    }

    // The sums (and prod's e) as WORDS words, 32 apart, and the sum with such a state.
    __device__ __forceinline__ void store(uint32_t *w) {
        int k = 0;
        auto put = [&](uint32_t v) { w[32 * k++] = v; };
        each([&](fx::Sum96 &v) {
            put((uint32_t)v.lo);
            put((uint32_t)(v.lo >> 32));
            put((uint32_t)v.hi);
        });
        put(orb.bad());
        if (JIT) put((uint32_t)prod.e);
    }
    __device__ __forceinline__ void merge(const uint32_t *w) {
        int k = 0;
        auto get = [&]() { return w[32 * k++]; };
        auto get64 = [&]() {
            const uint32_t l = get();
            return ((uint64_t)get() << 32) | l;
        };
        each([&](fx::Sum96 &v) {
            const int64_t l = (int64_t)get64();
            v.add(l, (int32_t)get());
        });
        if (get()) orb.far_r = fx::RI_MAX + 1;
        if (JIT) prod.e += (int32_t)get();
    }

    // The jitter form's sums as doubles: the lower triangle of M W M^T, M W y
    // and y W y.
    __device__ __forceinline__ void system(const StarRec &st, double (&Gd)[L][L], double (&qd)[L],
                                           double &yy) const {
        const double c = st.fx_w * g;
        Gd[0][0] = A00.value() * (c * 0x1p-60);
        qd[0] = b0.value() * (c * st.fx_y * 0x1p-61);
        yy = rWr.value() * (c * st.fx_y * st.fx_y * 0x1p-62);
#pragma unroll
        for (int i = 1; i < L; ++i) {
            const double ti = i == 1 ? c : c * st.fx_T[i];
            Gd[i][0] = A0[i].value() * (ti * 0x1p-61);
            qd[i] = q[i].value() * (ti * st.fx_y * 0x1p-62);
#pragma unroll
            for (int k = 1; k <= i; ++k)
                Gd[i][k] = G[i][k].value() * ((k == 1 ? ti : ti * st.fx_T[k]) * 0x1p-62);
        }
    }

    // No jitter: the K row A00, A0k of M W M^T and K's entry b0 of M W y.
    __device__ __forceinline__ void k_row(const StarRec &st, double &a00, double &b,
                                          double *a0) const {
        a00 = A00.value() * (st.fx_w * 0x1p-60);
        b = b0.value() * (st.fx_w * st.fx_y * 0x1p-61);
#pragma unroll
        for (int k = 1; k < L; ++k)
            a0[k] = A0[k].value() * ((k == 1 ? st.fx_w : st.fx_w * st.fx_T[k]) * 0x1p-61);
    }

    // sum log(1 + s^2 ivar_j) less log of the returned factor in [1/2, 1)
    __device__ __forceinline__ double log_rest(const StarRec &st, double &factor) const {
        factor = (double)prod.m * 0x1p-62;
        return fma((double)prod.e, 0.69314718055994530942, (double)st.n_epochs * log1p(a));
    }

    __device__ __forceinline__ double finish(const StarRec &st, double P, double e) const {
        const double lam0 = k_prior_variance(st, P, e);
        if constexpr (!JIT) {
            double a00, b, a0[MAXL];
            k_row(st, a00, b, a0);
            return tail_schur_d<L, false>(st, a00, a0, b, lam0, 0.0);
        } else {
            double Gd[L][L], qd[L], yy, f;
            system(st, Gd, qd, yy);
            const double ilam0 = st.k_scaled ? rcp_newton(lam0) : st.ilam[0];
#pragma unroll
            for (int i = 0; i < L; ++i) Gd[i][i] += i == 0 ? ilam0 : st.ilam[i];
            const double lr = log_rest(st, f);
            return tail_full_d<L, false>(Gd, qd, yy, st.log_norm_rest - st.sum_log_ivar + lr,
                                         lam0 * f);
        }
    }
};

// An epoch's fixed-point record, from global memory.
__device__ __forceinline__ fx::EpochFx load_epoch_fx(const double *rec) {
    fx::EpochFx r;
    const int4 *src = reinterpret_cast<const int4 *>(rec + FX64);
    int4 *dst = reinterpret_cast<int4 *>(&r);
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[k] = __ldg(src + k);
    return r;
}

// The fixed-point halves of n FP64 epoch records, into shared memory.
__device__ __forceinline__ void stage_epochs_fx(fx::EpochFx *sm, const double *src, int n) {
    const int4 *s4 = reinterpret_cast<const int4 *>(src + FX64);
    int4 *d4 = reinterpret_cast<int4 *>(sm);
    for (int i = threadIdx.x; i < n * 4; i += blockDim.x)
        d4[i] = __ldg(s4 + (i >> 2) * (REC64 / 2) + (i & 3));
}

// A block of 128 threads works on 128 / S samples, S = 1, 2 or 4: warp w takes
// every S-th epoch, from w % S on, of the 32 samples of group w / S, and the
// states meet in the group's first warp.  S > 1 is for calls whose samples
// alone leave SMs idle or the last wave short.
constexpr int SLICED_BLOCK = 128;

// Blocks per SM the registers are held to: six (80 registers, a few spills
// outside the epoch loop) against four gave 334 -> 318 us for 2^20 samples x
// 16 epochs and 105 -> 91 us for 100003 posterior rows; the large systems of
// the jitter form would spill their sums.
constexpr int fx_blocks(int L, bool jit) { return jit && L > 3 ? 3 : 6; }

// Shared memory of such a block: a tile of epochs, then the stored states; with
// the jitter, behind them, the four products of each sample.
template <int L, bool JIT> __host__ __device__ constexpr int sliced_states(int S) {
    const int tile = TILE * (int)sizeof(fx::EpochFx);
    const int states = (4 / S) * (S - 1) * AccFx<L, JIT>::WORDS * 128;
    return tile > states ? tile : states;
}
template <int L, bool JIT> constexpr int sliced_smem(int S) {
    return sliced_states<L, JIT>(S) + (JIT ? 4 * (SLICED_BLOCK / S) * 8 : 0);
}

// All epochs of a star into the samples' states; afterwards the first warp of
// each group holds the totals (true there).  `go`: this thread's sample takes
// the fixed-point form.  Called by the whole block.
template <int L, bool JIT>
__device__ __forceinline__ bool sliced_epochs(AccFx<L, JIT> &acc, bool go, const StarRec &st,
                                              const double *ep64, void *smem, int S) {
    fx::EpochFx *sm = static_cast<fx::EpochFx *>(smem);
    const int warp = threadIdx.x >> 5, slice = warp & (S - 1), N = st.n_epochs;
    // m of product c of this thread's sample at c * samples (their e's add up)
    const int samples = SLICED_BLOCK / S;
    int64_t *pm = reinterpret_cast<int64_t *>(static_cast<char *>(smem) +
                                              sliced_states<L, JIT>(S)) +
                  warp / S * 32 + (threadIdx.x & 31);
    if (JIT) {
        if (S > 1) __syncthreads();              // an earlier call's products are read
        acc.prod.one();
        for (int c = slice; c < 4; c += S) pm[c * samples] = acc.prod.m;
    }
    for (int t0 = 0; t0 < N; t0 += TILE) {
        const int nt = min(TILE, N - t0);
        __syncthreads();
        stage_epochs_fx(sm, ep64 + ((size_t)st.epoch_off + t0) * REC64, nt);
        __syncthreads();
        if (go)
            for (int i = (slice - t0) & (S - 1); i < nt; i += S) {
                const int64_t d = acc.add(sm[i]);
                if (JIT) {
                    int64_t *m = pm + (i & 3) * samples;         // TILE is a multiple of 4
                    acc.prod.m = *m;
                    acc.prod.times(d);
                    *m = acc.prod.m;
                }
            }
    }
    if (S > 1) {
        __syncthreads();
        uint32_t *w = static_cast<uint32_t *>(smem) +
                      ((warp / S) * (S - 1) * AccFx<L, JIT>::WORDS) * 32 + (threadIdx.x & 31);
        if (slice > 0) acc.store(w + (slice - 1) * AccFx<L, JIT>::WORDS * 32);
        __syncthreads();
        if (slice > 0) return false;
        for (int k = 0; k < S - 1; ++k) acc.merge(w + k * AccFx<L, JIT>::WORDS * 32);
    }
    if (JIT) {
        acc.prod.m = pm[0];
        for (int c = 1; c < 4; ++c) acc.prod.times(pm[c * samples]);
    }
    return true;
}

// S for n samples of N epochs (over several stars their mean, and the longest's)
// on a GPU that holds `wave` blocks at a time.  Four warps share a sample's
// epochs out but each makes the orbit's constants, worth some 4 epochs; they
// gain while the samples alone leave SMs idle or a last wave short.  Times of
// S = 4 over S = 1 (two linear parameters, six blocks an SM: 116736 samples a
// wave):
//   epochs   20000   60000   117000   160000   234000   311000 rows
//     16      0.66    1.00     1.08     1.16     1.19     1.28
//     40      0.58    0.91     0.95     1.00     1.03     1.10
//    300      0.53    0.76     0.85     0.89
// and likewise by waves with three blocks an SM: the line is N/32 waves, at most
// four.  Beside shorter stars the longest one's chain is what S = 4 cuts, as long
// as it outlasts the rest: seven stars of 3 epochs and one of 300, 50000 rows
// each, 441 -> 326 us, eight of 3 to 250 449 -> 478 (left at S = 1).
inline int slices_for(int64_t n, int N, int longest, int wave) {
    const int64_t w = (int64_t)wave * SLICED_BLOCK;
    const bool few = N >= 4 && 32 * n < N * w && n < 4 * w;
    const bool chain = longest >= 4 && 5 * n * (N + 14) < 4 * longest * w;
    return few || chain ? 4 : 1;
}

// FP64 ln L of one sample with the star's epochs read from global memory, in
// doubles: the form for what the fixed-point one does not take.
template <int L, bool JIT>
__device__ __noinline__ double fp64_lnl_doubles(const StarRec &st, const double *ep64, double P,
                                               double e, double om, double M0, double s) {
    Acc64<L, JIT> acc;
    acc.init(st, P, e, om, M0, s);
    const double *rec = ep64 + (size_t)st.epoch_off * REC64;
    for (int i = 0; i < st.n_epochs; ++i, rec += REC64) {
        double T[MAXL];
#pragma unroll
        for (int k = 1; k < L; ++k) T[k - 1] = __ldg(rec + 2 + k);
        acc.add(__ldg(rec), __ldg(rec + 1), __ldg(rec + 2), T);
    }
    return acc.finish(st, P);
}

// FP64 ln L of one sample with the star's epochs read from global memory.
template <int L, bool JIT>
__device__ __noinline__ double fp64_lnl_global(const StarRec &st, const double *ep64, double P,
                                               double e, double om, double M0, double s) {
    AccFx<L, JIT> acc;
    if (acc.init(st, P, e, om, M0, s)) {
        const double *rec = ep64 + (size_t)st.epoch_off * REC64;
        FxProd p[4];
        for (int c = 0; c < 4; ++c) p[c].one();
        for (int i = 0; i < st.n_epochs; ++i, rec += REC64) {
            const int64_t d = acc.add(load_epoch_fx(rec));
            if (JIT) p[i & 3].times(d);
        }
        acc.prod = p[0];
        if (JIT)
            for (int c = 1; c < 4; ++c) acc.prod.times(p[c].m, p[c].e);
        if (!acc.orb.bad()) return acc.finish(st, P, e);
    }
    return fp64_lnl_doubles<L, JIT>(st, ep64, P, e, om, M0, s);
}

// FP64 ln L of one sample evaluated by a whole warp: lane l takes epochs l,
// l + 32, ...; the sums are combined across the warp.  All 32 lanes must call
// it with the same sample; all return the value.  The fixed-point form gives
// fp64_lnl_global's number; the FP64 form sums in a different order (agreement
// to FP64 rounding of the sums).
template <int L, bool JIT>
__device__ __noinline__ double fp64_lnl_warp_t(const StarRec &st, const double *ep64, double P,
                                               double e, double om, double M0, double s) {
    const double *rec0 = ep64 + (size_t)st.epoch_off * REC64;
    AccFx<L, JIT> fxa;
    if (fxa.init(st, P, e, om, M0, s)) {
        const int lane = threadIdx.x & 31;
        FxProd p;                                // that of epochs i = lane mod 4
        p.one();
        for (int base = 0; base < st.n_epochs; base += 32) {
            int64_t d = 0;
            if (base + lane < st.n_epochs)
                d = fxa.add(load_epoch_fx(rec0 + (size_t)(base + lane) * REC64));
            if (JIT)
                for (int k = lane & 3, n = 0; n < 8; k += 4, ++n) {
                    const int64_t dk =
                        (int64_t)__shfl_sync(0xffffffffu, (unsigned long long)d, k);
                    if (base + k < st.n_epochs) p.times(dk);
                }
        }
        fxa.warp_sum();
        if (JIT) {
            fxa.prod.m = (int64_t)__shfl_sync(0xffffffffu, (unsigned long long)p.m, 0);
            fxa.prod.e = __shfl_sync(0xffffffffu, p.e, 0);
            for (int c = 1; c < 4; ++c)
                fxa.prod.times((int64_t)__shfl_sync(0xffffffffu, (unsigned long long)p.m, c),
                               __shfl_sync(0xffffffffu, p.e, c));
        }
        if (!__any_sync(0xffffffffu, fxa.orb.bad())) return fxa.finish(st, P, e);
    }
    Acc64<L, JIT> acc;
    acc.init(st, P, e, om, M0, s);
    for (int i = threadIdx.x & 31; i < st.n_epochs; i += 32) {
        const double *rec = rec0 + (size_t)i * REC64;
        double T[MAXL];
#pragma unroll
        for (int k = 1; k < L; ++k) T[k - 1] = __ldg(rec + 2 + k);
        acc.add(__ldg(rec), __ldg(rec + 1), __ldg(rec + 2), T);
    }
    acc.warp_sum();
    return acc.finish(st, P);
}

__device__ __forceinline__ double fp64_lnl_warp(int L, bool jit, const StarRec &st,
                                                const double *ep64, double P, double e,
                                                double om, double M0, double s) {
    switch (L) {
        case 1: return jit ? fp64_lnl_warp_t<1, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_warp_t<1, false>(st, ep64, P, e, om, M0, s);
        case 2: return jit ? fp64_lnl_warp_t<2, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_warp_t<2, false>(st, ep64, P, e, om, M0, s);
        case 3: return jit ? fp64_lnl_warp_t<3, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_warp_t<3, false>(st, ep64, P, e, om, M0, s);
        case 4: return jit ? fp64_lnl_warp_t<4, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_warp_t<4, false>(st, ep64, P, e, om, M0, s);
        case 5: return jit ? fp64_lnl_warp_t<5, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_warp_t<5, false>(st, ep64, P, e, om, M0, s);
        default: return jit ? fp64_lnl_warp_t<6, true>(st, ep64, P, e, om, M0, s)
                            : fp64_lnl_warp_t<6, false>(st, ep64, P, e, om, M0, s);
    }
}

__device__ __forceinline__ double fp64_lnl_sample(int L, bool jit, const StarRec &st,
                                                  const double *ep64, double P, double e,
                                                  double om, double M0, double s) {
    switch (L) {
        case 1: return jit ? fp64_lnl_global<1, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_global<1, false>(st, ep64, P, e, om, M0, s);
        case 2: return jit ? fp64_lnl_global<2, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_global<2, false>(st, ep64, P, e, om, M0, s);
        case 3: return jit ? fp64_lnl_global<3, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_global<3, false>(st, ep64, P, e, om, M0, s);
        case 4: return jit ? fp64_lnl_global<4, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_global<4, false>(st, ep64, P, e, om, M0, s);
        case 5: return jit ? fp64_lnl_global<5, true>(st, ep64, P, e, om, M0, s)
                           : fp64_lnl_global<5, false>(st, ep64, P, e, om, M0, s);
        default: return jit ? fp64_lnl_global<6, true>(st, ep64, P, e, om, M0, s)
                            : fp64_lnl_global<6, false>(st, ep64, P, e, om, M0, s);
    }
}

}  // namespace joker
