/*
 * Pieces of the FP64 FIRE step shared by the on-chip kernels (fire_res64.cu,
 * fire_dsm64.cu): the canonical reductions and the scalar update arranged for
 * the fewest FP64 instructions and the shortest chain.  On GB300 a warp's FP64
 * instruction takes the SM's FP64 pipe for 19 clocks and its scheduler's for
 * 64, so a lone warp pays 64 clocks for each, dependent or not.
 * Same operations on the same values as fire_common.cuh: the same bits.
 */
#ifndef NR_FP64_STEP_CUH
#define NR_FP64_STEP_CUH

#include "fire_common.cuh"

namespace nr {

/* Butterfly of three values at once: lane 0 gets sum(P), lane 16 sum(V),
 * lane 8 sum(F), each with the bits of warp_sum (an xor butterfly's lanes all
 * hold the same commutative sums, so half of them may work for another
 * value). */
__device__ __forceinline__ double warp_sum3(double P, double V, double F, int lane) {
    const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0;
    double a = b4 ? V : P;
    a = a + __shfl_xor_sync(kFull, b4 ? P : V, 16);
    F = F + __shfl_xor_sync(kFull, F, 16);
    double c = b3 ? F : a;
    c = c + __shfl_xor_sync(kFull, b3 ? a : F, 8);
    c = c + __shfl_xor_sync(kFull, c, 4);
    c = c + __shfl_xor_sync(kFull, c, 2);
    return c + __shfl_xor_sync(kFull, c, 1);
}

/* Largest of the lanes' non-negative doubles, compared as integers (a NaN
 * counts as 0, as fmax drops it). */
__device__ __forceinline__ unsigned long long max_bits(double v) {
    const unsigned long long u = ii_bits(v);
    return u > 0x7ff0000000000000ULL ? 0ULL : u;
}
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long u) {
    const unsigned hi = (unsigned)(u >> 32), mh = __reduce_max_sync(kFull, hi);
    const unsigned ml = __reduce_max_sync(kFull, hi == mh ? (unsigned)u : 0u);
    return ((unsigned long long)mh << 32) | ml;
}

/* Tree of the eight lane-group sums w[0..8), of which the first `ng` can be
 * nonzero (x + 0 = x). */
__device__ __forceinline__ double tree8_n(const double *w, int ng) {
    if (ng <= 1) return w[0];
    if (ng <= 2) return w[0] + w[1];
    if (ng <= 4) return (w[0] + w[1]) + (w[2] + w[3]);
    return tree8(w);
}

static __device__ __noinline__ double res_fmin(double a, double b) { return fmin(a, b); }
static __device__ __noinline__ double res_half_slow(double v) { return .5 * v; }
/* v / 2 by the exponent. */
__device__ __forceinline__ double res_half(double v) {
    const unsigned e = (unsigned)(ii_bits(v) >> 52) & 0x7ffu;
    return e - 2u < 2045u ? ii_double(ii_bits(v) - 0x0010000000000000ULL) : res_half_slow(v);
}
/* a < b for a >= 0 or NaN. */
__device__ __forceinline__ bool res_less(double a, double b) {
    return ii_positive(b) && ii_bits(b) <= 0x7ff0000000000000ULL && ii_abs_bits(a) < ii_bits(b);
}

/* scal_init / scal_step (fire_common.cuh) by one warp: the lanes of one
 * instruction stream take the three trees, the three roots and the four
 * quotients side by side, so the serial chain is a third of one thread's.
 * tot: [P, V2, F2] x 8 group sums; m2: bits of max|F|^2. */
__device__ __forceinline__ void scal_warp(Scal &s, const FireParamsDev &p, const double *tot, int ng,
                                          unsigned long long m2, double sqrt_dof, bool init) {
    const int lane = threadIdx.x & 31;
    double t = ii_double(m2);
    if (lane < 3) t = tree8_n(tot + 8 * lane, ng);
    const double root = sqrt_ieee(lane == 0 ? 1.0 : t);
    const double P = __shfl_sync(kFull, t, 0);
    const double vmag = __shfl_sync(kFull, root, 1), fmag = __shfl_sync(kFull, root, 2),
                 maxf = __shfl_sync(kFull, root, 3);
    const double dt_old = s.dt, alpha_old = s.alpha;
    int since = s.since;
    /* P > 0: neither sign bit nor zero nor NaN */
    const unsigned long long pb = ii_bits(P);
    const bool up = pb != 0ULL && pb <= 0x7ff0000000000000ULL;
    /* dt finc | dt fdec | alpha falpha on lanes 0 | 1 | 2 */
    const double pr = (lane == 2 ? alpha_old : dt_old) * (lane == 0 ? p.finc : lane == 1 ? p.fdec : p.falpha);
    const double grown = __shfl_sync(kFull, pr, 0), shrunk = __shfl_sync(kFull, pr, 1),
                 cooled = __shfl_sync(kFull, pr, 2);
    double dt = p.dt_max, alpha = p.alpha0;
    int zero_v = 0;
    if (init) {
        since = 0;
    } else if (up) {
        dt = dt_old;
        alpha = alpha_old;
        if (++since > p.nmin) {
            /* fmin of two non-negative numbers by their bits */
            const unsigned long long gb = ii_bits(grown);
            dt = gb <= 0x7ff0000000000000ULL ? (gb < ii_bits(p.dt_max) ? grown : p.dt_max) : res_fmin(grown, p.dt_max);
            alpha = cooled;
        }
    } else {
        since = 0;
        dt = shrunk;
        zero_v = 1;
    }
    /* alpha |v| on lane 0, dt / 2 on lane 1, dt^2 / 2 on lane 2 (halving is
     * exact, so the order of the reference's factors does not matter) */
    const double hdt = res_half(dt);
    double num = (lane == 0 ? alpha_old : lane == 1 ? 1.0 : hdt) * (lane == 0 ? vmag : lane == 1 ? hdt : dt);
    double den = p.mass;
    if (lane == 0) den = init ? 1.0 : fmag;
    if (lane == 3) {
        num = fmag;
        den = sqrt_dof;
    }
    const double q = div_ieee(num, den);
    const double dtm = __shfl_sync(kFull, q, 1), dtsq = __shfl_sync(kFull, q, 2), rms = __shfl_sync(kFull, q, 3);
    const bool finite = (ii_bits(fmag) & 0x7ff0000000000000ULL) != 0x7ff0000000000000ULL;
    __syncwarp();
    if (lane == 0) {
        s.dt = dt;
        s.dtm = dtm;
        s.dtsq = dtsq;
        s.alpha = alpha;
        s.since = since;
        s.fmag = fmag;
        s.maxf = maxf;
        s.zero_v = zero_v;
        s.converged = res_less(p.criterion == 1 ? maxf : rms, p.fcut);
        if (init) {
            s.mix_na = 0.0;
            s.mix_a = 0.0;
            s.power = 0.0;
            s.vmag = 0.0;
            s.mix_pending = 0;
            s.step = 0;
            s.status = finite ? 0 : NR_ERR_NONFINITE;
            s.done = p.max_steps <= 0 || s.status != 0;
        } else {
            s.step++;
            s.power = P;
            s.vmag = vmag;
            s.mix_a = q;
            s.mix_na = -alpha_old;
            s.mix_pending = 1;
            if (!finite || (pb & 0x7ff0000000000000ULL) == 0x7ff0000000000000ULL) s.status = NR_ERR_NONFINITE;
            s.done = s.converged || s.step >= p.max_steps || s.status != 0;
        }
    }
}

/* Pass A of one node (pass_a_node's operations, fire_fp64.cu). */
__device__ __forceinline__ void res_mix(const Scal &s, double2 &v, const double2 f) {
    if (s.mix_pending) {
        v.x = fma(s.mix_na, v.x, v.x);
        v.y = fma(s.mix_na, v.y, v.y);
        v.x = fma(s.mix_a, f.x, v.x);
        v.y = fma(s.mix_a, f.y, v.y);
        if (s.zero_v) v = make_double2(0.0, 0.0);
    }
}
__device__ __forceinline__ void res_drift(const Scal &s, double2 &x, const double2 v, const double2 f) {
    x.x = fma(s.dt, v.x, x.x);
    x.y = fma(s.dt, v.y, x.y);
    x.x = fma(s.dtsq, f.x, x.x);
    x.y = fma(s.dtsq, f.y, x.y);
}

}  // namespace nr

#endif
