// Marginal-likelihood kernels of libjoker_gb300 (sm_103a).
//
// For one star and one prior sample (P, e, omega, M0, s) the kernels evaluate
// the ln-likelihood with the linear parameters (K, v0, offsets, trend)
// integrated out under their Gaussian prior -- the quantity the reference
// computes in CJokerHelper.likelihood_worker (thejoker/src/fast_likelihood.pyx
// :359-425) through an N x N LU factorisation.  Here the same number comes
// from the matrix determinant lemma and the Woodbury identity in O(N L^2):
//
//   G = Lambda^-1 + M W M^T (L x L),  q = M W r,  r = y - M^T mu
//   chi2   = r^T W r - q^T G^-1 q
//   logdet = N log(2 pi) - sum log w + sum log Lambda_i + log det G
//   ln L   = -(chi2 + logdet) / 2
//
// Row 0 of M is the unit-K Kepler velocity, rows 1.. the trend/offset
// columns (row 1 is the constant v0 term).  Without jitter everything that
// does not depend on the sample -- the trend block C of G, its inverse, the
// trend-only chi2_0 -- is folded per star on the host, so per sample only the
// Schur complement of the K column remains:
//   s = A00 + 1/Lambda0 - g^T C^-1 g,   u = b0 - g^T C^-1 c,
//   t = u - mu0 (s - 1/Lambda0),
//   chi2 = chi2_0 - 2 mu0 u + mu0^2 (s - 1/Lambda0) - t^2 / s,
//   log det G = log det C + log s.
// With the jitter applied the weights change per sample and the full L x L
// system is factorised per sample (LDL^T, K last).
//
// One thread owns one sample (the FP64 kernel: up to four warps share the
// epochs of 32 samples) and walks the star's epochs, which the CTA stages in
// shared memory.  The mixed kernels' CTAs pull (star, sample-range) work items
// from a global counter (a persistent launch sized to the SM count); the FP64
// kernel takes one item per CTA.
#include "joker_mixed.cuh"

namespace joker {

// ------------------------------------------------------------- K1: FP64 path
// The fixed-point form (AccFx), epochs staged in shared memory; a sample that
// it does not take runs in doubles (fp64_lnl_doubles).  In doubles the FP64
// pipe bounded it (70-90 FP64 instructions per epoch, 16 cycles of an SM
// each); in fixed point the integer pipes do.  2^20 samples x 16 epochs:
// 2267 us in doubles, 318 us; 1.5e6 x 40 with the jitter: 9041, 1403 us.
// What bounds it now is the pipe of the wide integer multiplies (73 % busy).
template <int L, bool JIT>
__global__ void __launch_bounds__(SLICED_BLOCK, fx_blocks(L, JIT))
lnl_fp64_kernel(LnlArgs a, int S) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int per = SLICED_BLOCK / S;                     // samples per pass
    const int mine = (threadIdx.x >> 5) / S * 32 + (threadIdx.x & 31);
    const int n_items = item_count(a);
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const WorkItem w = get_item(a, it);
        const StarRec &st = a.stars[w.star];
        unsigned long long *mk = a.max_key ? a.max_key + w.max_slot : nullptr;
        for (int base = 0; base < w.count; base += per) {
            const int j = base + mine;
            const bool active = j < w.count;
            const int64_t row = (w.row0 + (active ? j : 0)) * a.stride;
            const double P = a.P[row], e = a.e[row], om = a.om[row], M0 = a.M0[row];
            const double s = JIT ? a.s[row] : 0.0;
            AccFx<L, JIT> acc;
            bool ok = acc.init(st, P, e, om, M0, s);
            if (!sliced_epochs(acc, active && ok, st, a.ep64, smem, S)) continue;
            double lnl = 0.0;
            if (active) {
                ok = ok && !acc.orb.bad();
                lnl = ok ? acc.finish(st, P, e)
                         : fp64_lnl_doubles<L, JIT>(st, a.ep64, P, e, om, M0, s);
                a.lnl[w.out_off + j] = lnl;
            }
            if (mk) warp_max_update(mk, active ? double_to_key(lnl) : 0ull);
        }
    }
}

// The same for calls none of whose stars has the fixed-point form (weights more
// than 2^8 apart, or with the jitter a K prior mean), one sample per thread in
// doubles: FP64 pipe, 70-90 instructions an epoch.  Through the kernel above
// such calls carried its state beside theirs, and under S = 4 one warp of four
// worked: 2^20 samples x 16 epochs 2308 us, here 2179, with the jitter 2731 and
// 2586; 60013 x 40 341 and 323.
template <int L, bool JIT>
__global__ void __launch_bounds__(SLICED_BLOCK) lnl_fp64_doubles_kernel(LnlArgs a) {
    __shared__ __align__(16) double sm[TILE * FX64];
    const int n_items = item_count(a);
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const WorkItem w = get_item(a, it);
        const StarRec &st = a.stars[w.star];
        const int N = st.n_epochs;
        unsigned long long *mk = a.max_key ? a.max_key + w.max_slot : nullptr;
        for (int base = 0; base < w.count; base += blockDim.x) {
            const int j = base + threadIdx.x;
            const bool active = j < w.count;
            const int64_t row = (w.row0 + (active ? j : 0)) * a.stride;
            const double P = a.P[row];
            Acc64<L, JIT> acc;
            acc.init(st, P, a.e[row], a.om[row], a.M0[row], JIT ? a.s[row] : 0.0);
            for (int t0 = 0; t0 < N; t0 += TILE) {
                const int nt = min(TILE, N - t0);
                const double2 *src = reinterpret_cast<const double2 *>(
                    a.ep64 + ((size_t)st.epoch_off + t0) * REC64);
                __syncthreads();
                for (int i = threadIdx.x; i < nt * (FX64 / 2); i += blockDim.x)
                    reinterpret_cast<double2 *>(sm)[i] =
                        __ldg(src + i / (FX64 / 2) * (REC64 / 2) + i % (FX64 / 2));
                __syncthreads();
                if (active)
                    for (int i = 0; i < nt; ++i) {
                        const double *rec = sm + i * FX64;
                        acc.add(rec[0], rec[1], rec[2], rec + 3);
                    }
            }
            double lnl = 0.0;
            if (active) {
                lnl = acc.finish(st, P);
                a.lnl[w.out_off + j] = lnl;
            }
            if (mk) warp_max_update(mk, active ? double_to_key(lnl) : 0ull);
        }
    }
}

// --------------------------------------------------------- cache preparation
// From the reference's packed chunk (n x 5 row-major FP64: P, e, omega, M0, s)
// to FP64 columns and the prepared mixed form.
__global__ void prepare_cache_kernel(const double *__restrict__ chunk, int64_t n, int64_t row0,
                                     double *P, double *E, double *OM, double *M0, double *S,
                                     float4 *mx_a, float4 *mx_b, float *mx_s2) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double p = chunk[i * 5 + 0], e = chunk[i * 5 + 1], om = chunk[i * 5 + 2];
        const double m0 = chunk[i * 5 + 3], s = chunk[i * 5 + 4];
        const int64_t r = row0 + i;
        P[r] = p; E[r] = e; OM[r] = om; M0[r] = m0; S[r] = s;
        float4 pa, pb;
        float s2;
        prepare_sample(p, e, om, m0, s, pa, pb, s2);
        mx_a[r] = pa;
        mx_b[r] = pb;
        mx_s2[r] = s2;
    }
}

// ------------------------------------------------------------------ launchers
cudaError_t launch_lnl_packed(int precision, int L, bool jit, const LnlArgs &a, int block,
                              cudaStream_t st);

// One block per work item (blocks start in order as others end, which spreads
// uneven items as a work counter would, without the launch that zeroes one);
// a count in device memory is shared out over a grid of one wave.
template <int L, bool JIT>
static cudaError_t launch_fp64_LJ(LnlArgs a, cudaStream_t st) {
    int grid = a.n_items, S = 1, block = SLICED_BLOCK;
    if (a.n_items_dev) {
        const cudaError_t e = persistent_grid(
            reinterpret_cast<const void *>(lnl_fp64_kernel<L, JIT>), SLICED_BLOCK, &grid);
        if (e != cudaSuccess) return e;
    } else if (!a.items) {
        // doubles: blocks of a warp while blocks of four would leave the SMs'
        // shares uneven (60013 x 40: 383 -> 323 us; 200000 x 40: 1046 -> 1017;
        // 310000 x 16: 652 -> 663)
        if (a.doubles)
            block = a.count * a.n_sel < 12 * 152 * SLICED_BLOCK ? 32 : SLICED_BLOCK;
        else {
            int wave = 0;
            const cudaError_t e = persistent_grid(
                reinterpret_cast<const void *>(lnl_fp64_kernel<L, JIT>), SLICED_BLOCK, &wave);
            if (e != cudaSuccess) return e;
            S = slices_for(a.count * a.n_sel, a.epochs, a.longest, wave);
        }
        const int64_t chunk = block / S, ips = (a.count + chunk - 1) / chunk;
        if (ips * a.n_sel <= INT32_MAX) {
            a.chunk = (int)chunk;
            a.ips = ips;
            grid = a.n_items = (int)(ips * a.n_sel);
        }
    }
    if (grid < 1) return cudaSuccess;
    if (a.doubles)
        lnl_fp64_doubles_kernel<L, JIT><<<grid, block, 0, st>>>(a);
    else
        lnl_fp64_kernel<L, JIT><<<grid, SLICED_BLOCK, sliced_smem<L, JIT>(S), st>>>(a, S);
    count_launch();
    return cudaGetLastError();
}

template <int L>
static cudaError_t launch_fp64_L(bool jit, const LnlArgs &a, cudaStream_t st) {
    return jit ? launch_fp64_LJ<L, true>(a, st) : launch_fp64_LJ<L, false>(a, st);
}

template <int L, int VAR>
static cudaError_t launch_mixed_LV(bool jit, const LnlArgs &a, int block, cudaStream_t st) {
    if (mixed_paired(L, jit)) {
        if constexpr (L <= 3) {
            if (jit) return launch_persistent(lnl_mixed2_kernel<L, true, VAR, false>, a, block, st);
        }
        return launch_persistent(lnl_mixed2_kernel<L, false, VAR, false>, a, block, st);
    }
    if (jit) return launch_persistent(lnl_mixed_kernel<L, true, VAR, false>, a, block, st);
    return launch_persistent(lnl_mixed_kernel<L, false, VAR, false>, a, block, st);
}

template <int L>
static cudaError_t launch_mixed_L(bool jit, int var, const LnlArgs &a, int block,
                                  cudaStream_t st) {
    if (var == 1) return launch_mixed_LV<L, 1>(jit, a, block, st);
    if (var == 2) return launch_mixed_LV<L, 2>(jit, a, block, st);
    return launch_mixed_LV<L, 0>(jit, a, block, st);
}

cudaError_t launch_lnl_fast(int L, bool jit, const LnlArgs &a, int block, cudaStream_t st);

cudaError_t launch_lnl(int precision, int L, bool jit, const LnlArgs &a, int block,
                       cudaStream_t st) {
    // The FP32-sum kernel covers any number of linear parameters without the
    // jitter and at most three with it; larger jittered systems run the
    // float-float kernel, whose outputs are of the same kind (tighter bound).
    if (precision == JOKER_MIXED_FAST) {
        if (!jit || L <= 3) return launch_lnl_fast(L, jit, a, block, st);
        precision = JOKER_MIXED;
    }
    if (precision == JOKER_FP64) {
        switch (L) {
            case 1: return launch_fp64_L<1>(jit, a, st);
            case 2: return launch_fp64_L<2>(jit, a, st);
            case 3: return launch_fp64_L<3>(jit, a, st);
            case 4: return launch_fp64_L<4>(jit, a, st);
            case 5: return launch_fp64_L<5>(jit, a, st);
            case 6: return launch_fp64_L<6>(jit, a, st);
        }
    } else if (a.mx_a == nullptr) {
        return launch_lnl_packed(precision, L, jit, a, block, st);
    } else {
        const int var = precision == JOKER_MIXED_ACCURATE ? 1
                      : precision == JOKER_MIXED_FP64_TAIL ? 2 : 0;
        switch (L) {
            case 1: return launch_mixed_L<1>(jit, var, a, block, st);
            case 2: return launch_mixed_L<2>(jit, var, a, block, st);
            case 3: return launch_mixed_L<3>(jit, var, a, block, st);
            case 4: return launch_mixed_L<4>(jit, var, a, block, st);
            case 5: return launch_mixed_L<5>(jit, var, a, block, st);
            case 6: return launch_mixed_L<6>(jit, var, a, block, st);
        }
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_prepare(const double *chunk, int64_t n, int64_t row0, double *P, double *E,
                           double *OM, double *M0, double *S, float4 *mx_a, float4 *mx_b,
                           float *mx_s2, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    prepare_cache_kernel<<<(int)blocks, 256, 0, st>>>(chunk, n, row0, P, E, OM, M0, S, mx_a, mx_b,
                                                      mx_s2);
    count_launch();
    return cudaGetLastError();
}

}  // namespace joker
