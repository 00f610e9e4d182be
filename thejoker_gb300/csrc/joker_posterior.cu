// Per-sample FP64 work after the acceptance pass:
//
// * the Gaussian posterior of the linear parameters of accepted samples --
//   the a and Ainv that CJokerHelper.likelihood_worker(1) builds
//   (thejoker/src/fast_likelihood.pyx:394-423, make_AAinv :255-297) and that
//   batch_get_posterior_samples (:471-545) hands to rng.multivariate_normal;
// * the unmarginalized ln-likelihood of full samples,
//   JokerSamples.ln_unmarginalized_likelihood (thejoker/samples.py:611-632):
//   the sum over epochs of ln N(y | K m(t) + trend(t), sigma^2 + s^2).
#include <cstdio>
#include "joker_fp64.cuh"

namespace joker {

// log of a product of positive doubles: exponents as integers, mantissas
// multiplied, one logarithm for all; what has no normal exponent (zero,
// subnormal, inf, NaN, negative) through log by itself.
struct LogProd {
    double m = 1.0, rest = 0.0;
    int e = 0;
    __device__ __forceinline__ void times(double x) {
        const int hi = __double2hiint(x), ex = hi >> 20;
        if (ex <= 0 || ex >= 2047) { rest += log(x); return; }
        e += ex - 1023;
        m *= __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(x));
    }
    __device__ __forceinline__ double value() const {
        return rest + fma((double)e, 0.69314718055994530942, log(m));
    }
};

// Posterior of the linear parameters of one sample from G0 = M W M^T (lower
// triangle), q = M W (y - M^T mu) and rWr: with G = Lambda^-1 + G0,
// a = mu + G^-1 q, A = G^-1 (G = Lw D Lw^T, A = Lw^-T D^-1 Lw^-1), and ln L
// from the same factorisation.  lp holds the factors of the log determinant
// that are known beforehand, logdet0 the rest of it.
template <int L>
__device__ __forceinline__ void posterior_tail(const StarRec &st, double (&G)[L][L],
                                               const double (&q)[L], double rWr, double logdet0,
                                               LogProd lp, double lam0, double *a_out,
                                               double *A_out, double *lnl_out) {
    double ilam0 = st.ilam[0];
    if (st.k_scaled) ilam0 = lam0 < 1e300 ? rcp_newton(lam0) : 1.0 / lam0;
    lp.times(lam0);
    double rD[L], Lw[L][L];
    bool ok = true;
    {
        double D[L];
#pragma unroll
        for (int k = 0; k < L; ++k) {
            double dk = G[k][k] + (k == 0 ? ilam0 : st.ilam[k]);
#pragma unroll
            for (int m = 0; m < k; ++m) dk -= Lw[k][m] * Lw[k][m] * D[m];
            D[k] = dk;
            ok = ok && dk > 0.0;
            lp.times(dk);
            rD[k] = dk < 1e300 ? rcp_newton(dk) : 1.0 / dk;
#pragma unroll
            for (int i = k + 1; i < L; ++i) {
                double v = G[i][k];
#pragma unroll
                for (int m = 0; m < k; ++m) v -= Lw[i][m] * Lw[k][m] * D[m];
                Lw[i][k] = v * rD[k];
            }
        }
    }
    // z = Lw^-1 q, quad = z^T D^-1 z, x = Lw^-T D^-1 z
    double x[L], quad = 0.0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        double v = q[k];
#pragma unroll
        for (int m = 0; m < k; ++m) v -= Lw[k][m] * x[m];
        x[k] = v;
        quad = fma(v * v, rD[k], quad);
    }
#pragma unroll
    for (int k = L - 1; k >= 0; --k) {
        double v = x[k] * rD[k];
#pragma unroll
        for (int m = k + 1; m < L; ++m) v -= Lw[m][k] * x[m];
        x[k] = v;
    }
#pragma unroll
    for (int k = 0; k < L; ++k) a_out[k] = ok ? st.mu[k] + x[k] : NAN;
    // Lw <- Lw^-1 (unit lower triangle), column by column
#pragma unroll
    for (int c = 0; c < L; ++c)
#pragma unroll
        for (int i = c + 1; i < L; ++i) {
            double v = Lw[i][c];
#pragma unroll
            for (int m = c + 1; m < i; ++m) v = fma(Lw[i][m], Lw[m][c], v);
            Lw[i][c] = -v;
        }
#pragma unroll
    for (int i = 0; i < L; ++i)
#pragma unroll
        for (int c = 0; c <= i; ++c) {
            double v = i == c ? rD[i] : rD[i] * Lw[i][c];
#pragma unroll
            for (int k = i + 1; k < L; ++k) v = fma(Lw[k][i] * rD[k], Lw[k][c], v);
            A_out[i * L + c] = A_out[c * L + i] = ok ? v : NAN;
        }
    if (lnl_out) *lnl_out = ok ? -0.5 * (rWr - quad + logdet0 + lp.value()) : INFINITY;
}

// The same without jitter, where only K's row A00, A0, b0 of the system depends
// on the sample: with the star's own C^-1 and beta = C^-1 c (trend block),
// v = C^-1 A0 and the Schur complement s = A00 + 1/Lambda0 - A0 v,
//   K = (b0 - A0 beta) / s,  trend = mu + beta - v K,
//   A = [1/s, -v^T/s; -v/s, C^-1 + v v^T / s]
// (mu0 = 0).  Eliminating the full system per sample instead would lose what
// the trend explains of y' (ln L: 1e-9 .. 1e-11 relative with a trend).
template <int L>
__device__ __forceinline__ void posterior_schur(const StarRec &st, double A00, const double *A0,
                                                double b0, double lam0, double *a_out,
                                                double *A_out, double *lnl_out) {
    double v[MAXL], gv = 0.0, u = b0;
#pragma unroll
    for (int j = 1; j < L; ++j) {
        v[j] = 0.0;
#pragma unroll
        for (int k = 1; k < L; ++k) v[j] = fma(st.Cinv[j * MAXL + k], A0[k], v[j]);
        gv = fma(A0[j], v[j], gv);
        u = fma(-A0[j], st.cC[j], u);
    }
    const double sm = A00 - gv, ls = fma(lam0, sm, 1.0);      // Lambda0 s
    const bool ok = ls > 0.0;
    // (Lambda0 s beyond a double's range, or Lambda0 infinite: 1/s by itself)
    const bool big = !(ls < 1e300);
    const double is = big ? 1.0 / (sm + 1.0 / lam0) : lam0 * rcp_newton(ls);
    const double K = u * is;
    a_out[0] = ok ? K : NAN;
    A_out[0] = ok ? is : NAN;
#pragma unroll
    for (int j = 1; j < L; ++j) {
        const double w = v[j] * is;
        a_out[j] = ok ? st.mu[j] + fma(-v[j], K, st.cC[j]) : NAN;
        A_out[j] = A_out[j * L] = ok ? -w : NAN;
#pragma unroll
        for (int k = 1; k <= j; ++k)
            A_out[j * L + k] = A_out[k * L + j] = ok ? fma(w, v[k], st.Cinv[j * MAXL + k]) : NAN;
    }
    if (lnl_out)
        *lnl_out = ok ? -0.5 * (fma(-u, K, st.chi2_0) + st.logdet_const +
                                (big ? log(lam0) - log(is) : log(ls))) : INFINITY;
}

// In doubles, one thread: the form for what the fixed-point one does not take.
template <int L>
__device__ __noinline__ void posterior_doubles(const StarRec &st, const double *ep64, double P,
                                               double e, double om, double M0, double s, int k_clip,
                                               double *a_out, double *A_out, double *lnl_out) {
    Acc64<L, true> acc;
    acc.init(st, P, e, om, M0, s);
    const double *rec = ep64 + (size_t)st.epoch_off * REC64;
    for (int i = 0; i < st.n_epochs; ++i, rec += REC64) {
        double T[MAXL];
#pragma unroll
        for (int k = 1; k < L; ++k) T[k - 1] = __ldg(rec + 2 + k);
        acc.add(__ldg(rec), __ldg(rec + 1), __ldg(rec + 2), T);
    }
    double lam0 = k_prior_variance(st, P, e, k_clip != 0);
    if (st.k_scaled && e * e == 1.0) {                        // no reciprocal of zero
        lam0 = st.sigK0sq / (1.0 - e * e) * pow(P / st.P0, -2.0 / 3.0);
        if (k_clip) lam0 = fmin(st.maxK2, lam0);
    }
    posterior_tail<L>(st, acc.G, acc.q, acc.rWr, st.log_norm_rest - acc.sum_log_w(st), LogProd(),
                      lam0, a_out, A_out, lnl_out);
}

// One sample per thread, epochs shared out over S warps (sliced_epochs).
// A warp per sample in doubles spent its time
// on idle lanes -- 40 epochs on 64 lanes, ten FP64 shuffles a sum, the tail on
// one lane: 100003 rows x 40 epochs, three linear parameters took
// 4326 us, now 91.
template <int L, bool JIT>
__global__ void __launch_bounds__(SLICED_BLOCK, fx_blocks(L, JIT))
posterior_kernel(const StarRec *stars, const double *ep64, int star, const double *P,
                 const double *E, const double *OM, const double *M0, const double *S,
                 int64_t stride, const int64_t *rows, int64_t n, int k_clip, double *a, double *A,
                 double *lnl, int slices) {
    extern __shared__ __align__(16) unsigned char smem[];
    const StarRec &st = stars[star];
    const int64_t i = blockIdx.x * (int64_t)(SLICED_BLOCK / slices) +
                      (threadIdx.x >> 5) / slices * 32 + (threadIdx.x & 31);
    const bool active = i < n;
    const int64_t r = rows[active ? i : n - 1] * stride;
    const double p = P[r], e = E[r], om = OM[r], m0 = M0[r], s = JIT ? S[r] : 0.0;
    AccFx<L, JIT> acc;
    // mu0 as the device has it: a launch captured for one star of a slot may be
    // replayed for another
    bool ok = st.mu0 == 0.0 && acc.init(st, p, e, om, m0, s);
    if (!sliced_epochs(acc, active && ok, st, ep64, smem, slices) || !active) return;
    double *a_out = a + i * L, *A_out = A + i * L * L, *l_out = lnl ? lnl + i : nullptr;
    if (!ok || acc.orb.bad()) {
        posterior_doubles<L>(st, ep64, p, e, om, m0, s, k_clip, a_out, A_out, l_out);
        return;
    }
    const double lam0 = k_prior_variance(st, p, e, k_clip != 0);
    if constexpr (JIT) {
        double G[L][L], q[L], rWr, f;
        LogProd lp;
        acc.system(st, G, q, rWr);
        const double lr = acc.log_rest(st, f);
        lp.times(f);
        posterior_tail<L>(st, G, q, rWr, st.log_norm_rest - st.sum_log_ivar + lr, lp, lam0, a_out,
                          A_out, l_out);
    } else {
        double A00, b0, A0[MAXL];
        acc.k_row(st, A00, b0, A0);
        posterior_schur<L>(st, A00, A0, b0, lam0, a_out, A_out, l_out);
    }
}

// For a star without a fixed-point form, one warp per sample, lanes over
// epochs.  Posterior of the linear parameters of one sample.  With W = diag(w),
// G = Lambda^-1 + M W M^T and q = M W (y - M^T mu) (Acc64 with the jitter
// form), a = mu + G^-1 q, A = G^-1, and ln L from the same factorisation.
template <int L>
__device__ __noinline__ void posterior_one(const StarRec &st, const double *ep64, double P,
                                           double e, double om, double M0, double s, int k_clip,
                                           double *a_out, double *A_out, double *lnl_out) {
    Acc64<L, true> acc;
    acc.init(st, P, e, om, M0, s);
    const double *rec0 = ep64 + (size_t)st.epoch_off * REC64;
    for (int i = threadIdx.x & 31; i < st.n_epochs; i += 32) {
        const double *rec = rec0 + (size_t)i * REC64;
        double T[MAXL];
#pragma unroll
        for (int k = 1; k < L; ++k) T[k - 1] = __ldg(rec + 2 + k);
        acc.add(__ldg(rec), __ldg(rec + 1), __ldg(rec + 2), T);
    }
    acc.warp_sum();
    if ((threadIdx.x & 31) != 0) return;
    double lam0 = st.lam0;
    if (st.k_scaled) {
        lam0 = st.sigK0sq / (1.0 - e * e) * pow(P / st.P0, -2.0 / 3.0);
        if (k_clip) lam0 = fmin(st.maxK2, lam0);
    }
    // G (full symmetric) and its LDL^T factorisation
    double G[L][L], D[L], Lw[L][L];
#pragma unroll
    for (int i = 0; i < L; ++i) {
#pragma unroll
        for (int k = 0; k <= i; ++k) { G[i][k] = acc.G[i][k]; G[k][i] = acc.G[i][k]; }
        G[i][i] += 1.0 / (i == 0 ? lam0 : st.lam[i]);
    }
    double logdetG = 0.0;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        double dk = G[k][k];
#pragma unroll
        for (int m = 0; m < k; ++m) dk -= Lw[k][m] * Lw[k][m] * D[m];
        D[k] = dk;
        ok = ok && dk > 0.0;
        logdetG += log(dk);
#pragma unroll
        for (int i = k + 1; i < L; ++i) {
            double v = G[i][k];
#pragma unroll
            for (int m = 0; m < k; ++m) v -= Lw[i][m] * Lw[k][m] * D[m];
            Lw[i][k] = v / dk;
        }
    }
    // solve G x = b for b = q and for the unit vectors
    auto solve = [&](const double *b, double *x) {
        double z[L];
#pragma unroll
        for (int k = 0; k < L; ++k) {
            double v = b[k];
#pragma unroll
            for (int m = 0; m < k; ++m) v -= Lw[k][m] * z[m];
            z[k] = v;
        }
#pragma unroll
        for (int k = L - 1; k >= 0; --k) {
            double v = z[k] / D[k];
#pragma unroll
            for (int m = k + 1; m < L; ++m) v -= Lw[m][k] * x[m];
            x[k] = v;
        }
    };
    double x[L], quad = 0.0;
    solve(acc.q, x);
#pragma unroll
    for (int k = 0; k < L; ++k) {
        a_out[k] = ok ? st.mu[k] + x[k] : NAN;
        quad += acc.q[k] * x[k];
    }
#pragma unroll
    for (int c = 0; c < L; ++c) {
        double ec[L], col[L];
#pragma unroll
        for (int k = 0; k < L; ++k) ec[k] = k == c ? 1.0 : 0.0;
        solve(ec, col);
#pragma unroll
        for (int k = 0; k < L; ++k) A_out[k * L + c] = ok ? col[k] : NAN;
    }
    if (lnl_out)
        *lnl_out = ok ? -0.5 * (acc.rWr - quad + st.log_norm_rest + log(lam0) - acc.sum_log_w(st) + logdetG)
                      : INFINITY;
}

template <int L>
__global__ void __launch_bounds__(256) posterior_warp_kernel(const StarRec *stars, const double *ep64,
                                                        int star, const double *P, const double *E,
                                                        const double *OM, const double *M0,
                                                        const double *S, int64_t stride,
                                                        const int64_t *rows, int64_t n, int jit,
                                                        int k_clip, double *a, double *A,
                                                        double *lnl) {
    const StarRec &st = stars[star];
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
         i += nw) {
        const int64_t r = rows[i] * stride;
        posterior_one<L>(st, ep64, P[r], E[r], OM[r], M0[r], jit ? S[r] : 0.0, k_clip,
                         a + i * L, A + i * L * L, lnl ? lnl + i : nullptr);
    }
}

// ln of the unmarginalized likelihood: pars row = P, e, omega, M0, s, K, v_0..v_{nt-1}.
__global__ void __launch_bounds__(256) unmarginalized_kernel(const StarRec *stars,
                                                             const double *ep64, int star, int L,
                                                             const double *pars, int64_t n,
                                                             int nt, double dt_shift,
                                                             double *out) {
    const StarRec &st = stars[star];
    const int lane = threadIdx.x & 31;
    const int np = 6 + nt;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
         i += nw) {
        const double *p = pars + i * np;
        const double P = p[0], e = p[1], om = p[2], M0 = p[3], s2 = p[4] * p[4], K = p[5];
        OrbitF64 orb;
        orb.init(P, e, om, M0);
        double acc = 0.0;
        const double *rec0 = ep64 + (size_t)st.epoch_off * REC64;
        for (int j = lane; j < st.n_epochs; j += 32) {
            const double *rec = rec0 + (size_t)j * REC64;
            const double dt = __ldg(rec) - dt_shift;
            // data velocity: y = y' + sum_{k>=1} mu_k T_k
            double y = __ldg(rec + 1);
            for (int k = 1; k < L; ++k) y += st.mu[k] * __ldg(rec + 2 + k);
            const double var = 1.0 / __ldg(rec + 2) + s2;
            const double m = orb.rv_unit(dt);
            // trend polynomial in (t - t_ref of the samples), Horner
            double tr = 0.0;
            for (int k = nt - 1; k >= 0; --k) tr = fma(tr, dt, p[6 + k]);
            const double d = fma(K, m, tr) - y;
            acc += -0.5 * (log(TWO_PI_D * var) + d * d / var);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) out[i] = acc;
    }
}

// rv[i * n_t + j] = K_i m_i(t_j - t0) for element rows (P, K, e, omega, M0).
// W lanes take up to 8 W times of one orbit, so that the orbit's constants are
// made once a lane for them; the times become integers on the scale of the
// largest.  One thread per (orbit, time) pair made them for each pair, and in
// doubles: 4096 orbits x 1001 times took 785 us, now 82 (W = 32).
constexpr int RV_LANE = 8;

template <int W>
__global__ void __launch_bounds__(128, 6)
rv_elements_kernel(const double *t, int n_t, const double *el, int64_t n, int per_row, double t0,
                   double *rv) {
    const int lane = threadIdx.x & (W - 1);
    // the group's lanes; groups of a warp go their own ways
    const unsigned group = W == 32 ? 0xffffffffu
                                   : ((1u << W % 32) - 1u) << (threadIdx.x & 31 & ~(W - 1));
    const int64_t step = (int64_t)gridDim.x * (blockDim.x / W);
    for (int64_t g = blockIdx.x * (int64_t)(blockDim.x / W) + threadIdx.x / W; g < n * per_row;
         g += step) {
        const int64_t i = g / per_row;
        const int j0 = (int)(g - i * per_row) * (W * RV_LANE);
        const int nt = min(n_t - j0, W * RV_LANE);
        const double *p = el + i * 5;
        const double K = p[1];
        double *out = rv + i * n_t + j0;
        // the exponent of the largest |dt|: 2^(ex - 1023) <= |dt| < twice that
        unsigned ex = 0;
        for (int j = lane; j < nt; j += W)
            ex = max(ex, (unsigned)(__double2hiint(t[j0 + j] - t0) >> 20) & 0x7ff);
        if (W > 1) ex = __reduce_max_sync(group, ex);
        const int tsh = 62 - ((int)ex - 1022);            // |dt| 2^tsh < 2^62
        fx::Orbit orb;
        bool ok = ex > 723 && ex < 1323 &&                // within 2^300 of one day
                  fx::as_exact(tsh, p[0], p[2]) &&
                  orb.init(tsh, -fx::ONE62, p[0], p[2], p[3], p[4]);
        if (ok) {
            for (int j = lane; j < nt; j += W) {
                const int64_t q = fx::fixed_signed(t[j0 + j] - t0, tsh);
                const double m = (double)orb.column((uint64_t)(q + fx::ONE62));
                out[j] = K * (m * 0x1p-61);
            }
            ok = W > 1 ? !__any_sync(group, orb.bad()) : !orb.bad();
        }
        if (!ok) {
            OrbitF64 o;
            o.init(p[0], p[2], p[3], p[4]);
            for (int j = lane; j < nt; j += W) out[j] = K * o.rv_unit(t[j0 + j] - t0);
        }
    }
}

template <int W>
static cudaError_t launch_rv(const double *t, int n_t, const double *el, int64_t n, double t0,
                             double *rv, cudaStream_t st) {
    const int per_row = (n_t + W * RV_LANE - 1) / (W * RV_LANE), groups = 128 / W;
    const int64_t blocks = (n * per_row + groups - 1) / groups;
    const unsigned grid = (unsigned)(blocks < 152 * 64 ? blocks : 152 * 64);
    rv_elements_kernel<W><<<grid, 128, 0, st>>>(t, n_t, el, n, per_row, t0, rv);
    count_launch();
    return cudaGetLastError();
}

// Lanes per orbit: a lane without a time still makes the orbit's constants (450
// instructions against a column's 250), so curves of a few times take fewer.
// 10^6 orbits x 1 time: a thread per pair in doubles 196 us, 32 lanes 1085, one
// 40; x 7 times: 1340, 1084, eight lanes 291; x 9: 1717, 1096 (32 lanes).
cudaError_t launch_rv_elements(const double *t, int n_t, const double *el, int64_t n, double t0,
                               double *rv, cudaStream_t st) {
    if (n_t == 1) return launch_rv<1>(t, n_t, el, n, t0, rv, st);
    if (n_t <= 8) return launch_rv<8>(t, n_t, el, n, t0, rv, st);
    return launch_rv<32>(t, n_t, el, n, t0, rv, st);
}

template <int L, bool JIT>
static cudaError_t launch_posterior_LJ(const StarRec *stars, const double *ep64, int star,
                                       int epochs, const double *P, const double *E,
                                       const double *OM, const double *M0, const double *S,
                                       int64_t stride, const int64_t *rows, int64_t n, int k_clip,
                                       double *a, double *A, double *lnl, cudaStream_t st) {
    int wave = 0;
    const cudaError_t e = persistent_grid(
        reinterpret_cast<const void *>(posterior_kernel<L, JIT>), SLICED_BLOCK, &wave);
    if (e != cudaSuccess) return e;
    const int sl = slices_for(n, epochs, epochs, wave), per = SLICED_BLOCK / sl;
    const int64_t blocks = (n + per - 1) / per;
    if (blocks > INT32_MAX) return cudaErrorInvalidValue;
    posterior_kernel<L, JIT><<<(unsigned)blocks, SLICED_BLOCK, sliced_smem<L, JIT>(sl), st>>>(
        stars, ep64, star, P, E, OM, M0, S, stride, rows, n, k_clip, a, A, lnl, sl);
    count_launch();
    return cudaGetLastError();
}

// fixed: the star has a fixed-point form (stars_fixed).
template <int L>
static cudaError_t launch_posterior_L(const StarRec *stars, const double *ep64, int star,
                                      bool fixed, int epochs, const double *P,
                                      const double *E, const double *OM, const double *M0,
                                      const double *S, int64_t stride, const int64_t *rows,
                                      int64_t n, int jit, int k_clip, double *a, double *A,
                                      double *lnl, cudaStream_t st) {
    if (fixed && jit)
        return launch_posterior_LJ<L, true>(stars, ep64, star, epochs, P, E, OM, M0, S, stride,
                                            rows, n, k_clip, a, A, lnl, st);
    if (fixed)
        return launch_posterior_LJ<L, false>(stars, ep64, star, epochs, P, E, OM, M0, S, stride,
                                             rows, n, k_clip, a, A, lnl, st);
    const int64_t warps = n < 152 * 8 * 4 ? n : 152 * 8 * 4;
    const unsigned grid = (unsigned)((warps + 7) / 8);
    posterior_warp_kernel<L><<<grid, 256, 0, st>>>(stars, ep64, star, P, E, OM, M0, S, stride, rows,
                                                   n, jit, k_clip, a, A, lnl);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_posterior(int L, const StarRec *stars, const double *ep64, int star,
                             bool fixed, int epochs, const double *P, const double *E, const double *OM,
                             const double *M0, const double *S, int64_t stride,
                             const int64_t *rows, int64_t n, int jit, int k_clip, double *a,
                             double *A, double *lnl, cudaStream_t st) {
    switch (L) {
#define JOKER_POST_CASE(LL) \
        case LL: return launch_posterior_L<LL>(stars, ep64, star, fixed, epochs, P, E, OM, M0, S, \
                                               stride, rows, n, jit, k_clip, a, A, lnl, st);
        JOKER_POST_CASE(1) JOKER_POST_CASE(2) JOKER_POST_CASE(3)
        JOKER_POST_CASE(4) JOKER_POST_CASE(5) JOKER_POST_CASE(6)
#undef JOKER_POST_CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_unmarginalized(const StarRec *stars, const double *ep64, int star, int L,
                                  const double *pars, int64_t n, int nt, double dt_shift,
                                  double *out, cudaStream_t st) {
    const int64_t warps = n < 152 * 8 * 4 ? n : 152 * 8 * 4;
    const unsigned grid = (unsigned)((warps + 7) / 8);
    unmarginalized_kernel<<<grid, 256, 0, st>>>(stars, ep64, star, L, pars, n, nt, dt_shift, out);
    count_launch();
    return cudaGetLastError();
}

}  // namespace joker

// ------------------------------------------------------------------ C ABI
namespace joker {
void set_last_error(const char *msg);
void stars_internals(const joker_stars *s, const StarRec **recs, const double **ep64,
                     const float **ep32, int *n_stars, int *L, int *jit, int **queue);
int stars_epochs(const joker_stars *s, int star);
bool stars_fixed(const joker_stars *s, int star);
void cache_internals(const joker_cache *c, int64_t *cap, const double **P, const double **E,
                     const double **OM, const double **M0, const double **S, int64_t *stride,
                     const float4 **mx_a, const float4 **mx_b, const float **mx_s2);
}  // namespace joker

using namespace joker;

static int post_fail(int code, const char *msg) {
    set_last_error(msg);
    return code;
}

extern "C" int joker_linear_posterior(const joker_stars *stars, const joker_cache *cache,
                                      int star, const int64_t *d_rows, int64_t n, int k_clip,
                                      double *d_a, double *d_A, double *d_lnl, void *stream) {
    if (!stars || !cache) return post_fail(JOKER_EINVAL, "joker_linear_posterior: NULL handle");
    if (n < 0) return post_fail(JOKER_EINVAL, "joker_linear_posterior: n < 0");
    if (n == 0) return JOKER_OK;
    if (!d_rows || !d_a || !d_A)
        return post_fail(JOKER_EINVAL, "joker_linear_posterior: NULL device pointer");
    const StarRec *recs; const double *ep64; const float *ep32; int n_stars, L, jit; int *q;
    stars_internals(stars, &recs, &ep64, &ep32, &n_stars, &L, &jit, &q);
    if (star < 0 || star >= n_stars)
        return post_fail(JOKER_EINVAL, "joker_linear_posterior: star out of range");
    int64_t cap, stride; const double *P, *E, *OM, *M0, *S; const float4 *ma, *mb; const float *ms;
    cache_internals(cache, &cap, &P, &E, &OM, &M0, &S, &stride, &ma, &mb, &ms);
    const cudaError_t e = launch_posterior(L, recs, ep64, star, stars_fixed(stars, star),
                                           stars_epochs(stars, star), P, E, OM, M0, S, stride, d_rows,
                                           n, jit, k_clip, d_a, d_A, d_lnl, (cudaStream_t)stream);
    if (e != cudaSuccess) return post_fail(JOKER_ECUDA, cudaGetErrorString(e));
    return JOKER_OK;
}

extern "C" int joker_unmarginalized_lnl(const joker_stars *stars, int star, const double *d_pars,
                                        int64_t n, int n_trend, double dt_shift, double *d_out,
                                        void *stream) {
    if (!stars) return post_fail(JOKER_EINVAL, "joker_unmarginalized_lnl: NULL handle");
    if (n < 0 || n_trend < 1 || n_trend > JOKER_MAX_LINEAR - 1)
        return post_fail(JOKER_EINVAL, "joker_unmarginalized_lnl: bad n or n_trend");
    if (n == 0) return JOKER_OK;
    if (!d_pars || !d_out)
        return post_fail(JOKER_EINVAL, "joker_unmarginalized_lnl: NULL device pointer");
    const StarRec *recs; const double *ep64; const float *ep32; int n_stars, L, jit; int *q;
    stars_internals(stars, &recs, &ep64, &ep32, &n_stars, &L, &jit, &q);
    if (star < 0 || star >= n_stars)
        return post_fail(JOKER_EINVAL, "joker_unmarginalized_lnl: star out of range");
    const cudaError_t e = launch_unmarginalized(recs, ep64, star, L, d_pars, n, n_trend, dt_shift,
                                                d_out, (cudaStream_t)stream);
    if (e != cudaSuccess) return post_fail(JOKER_ECUDA, cudaGetErrorString(e));
    return JOKER_OK;
}

extern "C" int joker_rv_from_elements(const double *d_t, int n_t, const double *d_elems,
                                      int64_t n, double t0, double *d_rv, void *stream) {
    if (n < 0 || n_t < 0) return post_fail(JOKER_EINVAL, "joker_rv_from_elements: n < 0 or n_t < 0");
    if (n == 0 || n_t == 0) return JOKER_OK;
    if (!d_t || !d_elems || !d_rv)
        return post_fail(JOKER_EINVAL, "joker_rv_from_elements: NULL device pointer");
    const cudaError_t e = launch_rv_elements(d_t, n_t, d_elems, n, t0, d_rv, (cudaStream_t)stream);
    if (e != cudaSuccess) return post_fail(JOKER_ECUDA, cudaGetErrorString(e));
    return JOKER_OK;
}
