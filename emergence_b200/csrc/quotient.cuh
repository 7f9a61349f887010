// Correctly rounded quotients and square roots of the plain FP64 form, and the
// Euler maps, HLLC flux and WENO5-Z interpolation built on them (device only).
#pragma once
#include "physics.cuh"

namespace emg {

// ------------------------------------------------------------------ correctly rounded quotients without branches
// The plain FP64 form's quotients and square roots round exactly as IEEE
// operations, but come from straight-line fused multiply-adds, so that the
// compiler can interleave the independent ones of a midpoint; its own
// division ends each with a branch to the special cases, which serialises them.
//
// Method: P. Markstein's theorem (IBM J. Res. Dev. 34, 1990; also Muller et
// al., Handbook of Floating-Point Arithmetic, division with an FMA): if
// y = RN(1/b) and q is a faithful rounding of a/b, then r = a − b·q is exact and
// RN(q + r·y) = RN(a/b). With a and b scaled to [1, 2) and q = RN(a·y):
//   a ≥ b: |a·y − a/b| ≤ a·2^-54 < ½ ulp, so q is faithful;
//   a < b: the error can reach (a/2) ulp < 1 ulp and q can miss the two
//   neighbours of a/b, but q + r·y is still within 2^-52 ulp of a/b, so the
//   result could only be wrong for an a/b that close to a midpoint, and to miss
//   there takes an error of 1 − 2^-52 ulp, that is a > 2 − 2^-51: no b is above.
// Operands must stay where nothing over- or underflows and every remainder is
// exact: denominators in [2^-100, 2^100) (densities and pressures of any
// unit system), numerators zero or in ±[2^-900, 2^900): velocities decay through
// every magnitude ahead of a front. (With numerators from 2^-760 and stencils from
// 2^-460 the 3-D shock-bubble's pre-front regions took the slow path: 163–197 ms
// for 12 steps, now 145–183.) Violations are collected in `bad`, and the caller
// then evaluates the whole expression again with the compiler's operations. Tested
// against those bit for bit over both ranges.
struct RecipRn {
    double b, y;  // b > 0
};
// y = RN(1/b): the PTX estimate r (2^-20), the series step r·(1 + h + h²)
// (2^-60 before its rounding, so a faithful reciprocal), and Markstein's
// correction, which rounds every reciprocal correctly but that of an all-ones
// significand, 2^-k·(1 + 2^-53 + …), which it rounds down to 2^-k: one ulp is
// added there (such a ρ = 1 − 2^-53 is common next to a uniform state of 1).
__device__ __forceinline__ RecipRn recip_rn(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    const double h = fma(-b, r, 1.0);
    r = fma(r, fma(h, h, h), r);
    r = fma(r, fma(-b, r, 1.0), r);
    const bool ones = ((hi_bits(b) | 0xfff00000u) & (unsigned)__double2loint(b)) == 0xffffffffu;
    return RecipRn{b, __hiloint2double(__double2hiint(r), __double2loint(r) + (ones ? 1 : 0))};
}
// One operation less, for sums of squares: two Newton steps, so y is within (½ + ε)
// ulp of 1/b, not always RN(1/b). quot_rn of it is RN(a/b) all the same, by its error
// for b < 2 − 4ε (scaled to [1, 2)): for an a/b next to a midpoint q is half an ulp
// away, so q + r·y is off by at most b·(1 + 2ε)·2^-55 ulp(q), while a/b keeps 2^-53/b
// ulp(q) from the midpoint, and b²(1 + 2ε) < 4; and for a q = RN(a·y) more than an ulp
// off there, a·(½ + ε) ≥ 1 − 2^-52, so b > a > 2 − 4ε. The estimate is good to 2^-19.9,
// which makes ε = 2^-26. For b = 2 − δ, δ ≤ 2^-20, the estimate is exactly ½ and
// ε = 2^48·δ⁴ + δ²/2 + 2^-52, so only δ = k·2^-52, k ≤ 4, is left, and there y = RN(1/b):
// the first step gives ½ + k·2^-54, for an odd k halfway between two values and
// rounded up, so that the second step sees 1/b's next term (rounded to nearest, k = 1
// stays at ½ in both steps and 2/b comes out as 1).
__device__ __forceinline__ RecipRn recip_sq(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    r = __fma_ru(r, fma(-b, r, 1.0), r);
    return RecipRn{b, fma(r, fma(-b, r, 1.0), r)};
}
// a/b without checks; the remainder's sign keeps the sign of a zero numerator
__device__ __forceinline__ double quot_rn(double a, const RecipRn& d) {
    const double q = a * d.y;
    return fma(-fma(d.b, q, -a), d.y, q);
}
// range tests on the high words (sign, exponent, 20 mantissa bits)
__device__ __forceinline__ bool den_out(double b) {  // not in [2^-100, 2^100)
    constexpr unsigned LO = (1023u - 100u) << 20, HI = (1023u + 100u) << 20;
    return hi_bits(b) - LO >= HI - LO;
}
__device__ __forceinline__ bool num_out(double a) {  // neither zero nor in ±[2^-900, 2^900)
    constexpr unsigned LO = (1023u - 900u) << 20, HI = (1023u + 900u) << 20;
    const unsigned h = hi_bits(a) & 0x7fffffffu;
    return h - LO >= HI - LO && (h | (unsigned)__double2loint(a)) != 0u;
}
__device__ __forceinline__ RecipRn den_rn(double b, bool& bad) {
    bad = bad || den_out(b);
    return recip_rn(b);
}
__device__ __forceinline__ double div_rn(double a, const RecipRn& d, bool& bad) {
    bad = bad || num_out(a);
    return quot_rn(a, d);
}
// a/b with b of either sign: both signs are flipped for b < 0
__device__ __forceinline__ double div_signed_rn(double a, double b, bool& bad) {
    const int sgn = __double2hiint(b) & 0x80000000;
    return div_rn(__hiloint2double(__double2hiint(a) ^ sgn, __double2loint(a)), den_rn(fabs(b), bad), bad);
}
// Square root: y ≈ 1/√x from the PTX estimate and the series of rsqrt_f, one
// Markstein correction g ← g + (x − g²)·y/2, then the exact remainder d = x −
// g² proves the rounding: g = RN(√x) when |d| < g·ulp(g), tested on the high
// words with a margin of 2^-18 (anything closer is redone by the caller).
__device__ __forceinline__ double sqrt_rn(double x, bool& bad) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double h = fma(-(x * r), r, 1.0);
    const double y = fma(r * h, fma(0.375, h, 0.5), r);
    double g = x * y;
    g = fma(fma(-g, g, x), 0.5 * y, g);
    const double d = fma(-g, g, x);
    // g·ulp(g) = m·2^(2e−52) for g = m·2^e: compare exponent and mantissa words
    const unsigned hg = hi_bits(g), e = hg & 0x7ff00000u;
    bad = bad || den_out(x) || (hi_bits(d) & 0x7fffffffu) + 8u >= hg + e - ((1023u + 52u) << 20);
    return g;
}

// Euler maps of the plain form with these quotients: the operations and their
// order are those of to_prim, to_cons, sound_speed and hllc above, with the
// quotients by one ρ sharing its reciprocal. `rg` is γ − 1 with its correctly
// rounded reciprocal.
__device__ __forceinline__ void to_prim_rn(const Eos<double>& e, const double* u, double* w, bool& bad) {
    const double rho = u[0];
    const RecipRn r = den_rn(rho, bad);
    const double vx = div_rn(u[1], r, bad), vy = div_rn(u[2], r, bad), vz = div_rn(u[3], r, bad);
    const double ein = div_rn(u[4], r, bad) - 0.5 * (vx * vx + vy * vy + vz * vz);
    const double v = r.y;  // RN(1/ρ)
    w[0] = rho;
    w[1] = vx;
    w[2] = vy;
    w[3] = vz;
    w[4] = div_rn((e.gamma - 1.0) * (ein - e.q), den_rn(v - e.b, bad), bad) - e.gamma * e.p_inf;
}
// v = RN(1/ρ)
__device__ __forceinline__ void to_cons_rn(const Eos<double>& e, const RecipRn& rg, const double* w, double v, double* u,
                                           bool& bad) {
    const double rho = w[0];
    const double ke = 0.5 * rho * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]);
    u[0] = rho;
    u[1] = rho * w[1];
    u[2] = rho * w[2];
    u[3] = rho * w[3];
    u[4] = rho * (div_rn((w[4] + e.gamma * e.p_inf) * (v - e.b), rg, bad) + e.q) + ke;
}
__device__ __forceinline__ double sound_speed_rn(const Eos<double>& e, double p, double v, bool& bad) {
    // no max(c², 0): sqrt_rn refuses what is not a positive number
    return sqrt_rn(div_rn(e.gamma * (p + e.p_inf) * v * v, den_rn(v - e.b, bad), bad), bad);
}
// vl, vr: RN(1/ρ)
__device__ __forceinline__ void hllc_rn(const Eos<double>& e, const RecipRn& rg, const double* wl, const double* wr,
                                        double vl, double vr, int un, double* f, bool& bad) {
    const double cl = sound_speed_rn(e, wl[4], vl, bad), cr = sound_speed_rn(e, wr[4], vr, bad);
    const double ul = wl[un], ur = wr[un];
    const double sl = fmin(ul - cl, ur - cr);
    const double sr = fmax(ul + cl, ur + cr);
    double ql[5], qr[5];
    to_cons_rn(e, rg, wl, vl, ql, bad);
    to_cons_rn(e, rg, wr, vr, qr, bad);
    if (sl >= 0.0) {
        flux_wq(wl, ql, un, f);
        return;
    }
    if (sr <= 0.0) {
        flux_wq(wr, qr, un, f);
        return;
    }
    const double rl = wl[0], rr = wr[0], pl = wl[4], pr = wr[4];
    const double ss =
        div_signed_rn(pr - pl + rl * ul * (sl - ul) - rr * ur * (sr - ur), rl * (sl - ul) - rr * (sr - ur), bad);
    const bool left = ss >= 0.0;
    double w[5], q[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        w[k] = left ? wl[k] : wr[k];
        q[k] = left ? ql[k] : qr[k];
    }
    const RecipRn ri{w[0], left ? vl : vr};
    const double s = left ? sl : sr;
    double fx[5];
    flux_wq(w, q, un, fx);
    const double rho = w[0], u = w[un];
    const double fac = div_signed_rn(rho * (s - u), s - ss, bad);
    double qs[5];
    qs[0] = fac;
    qs[1] = fac * w[1];
    qs[2] = fac * w[2];
    qs[3] = fac * w[3];
    qs[un] = fac * ss;
    qs[4] = fac * (div_rn(q[4], ri, bad) + (ss - u) * (ss + div_signed_rn(w[4], rho * (s - u), bad)));
#pragma unroll
    for (int k = 0; k < 5; k++) f[k] = fx[k] + s * (qs[k] - q[k]);
}

// Both WENO5-Z interpolations of a six-value stencil (v0..v4 towards the
// midpoint and its mirror image), each value rounded exactly as weno5z_interp
// rounds it. Powers of two are moved out of products (exact scalings), which
// saves multiplies and lets an exact product join its sum in one fused
// multiply-add: the weights carry a factor 16, the candidates a factor 8.
// `bad` is raised when an operand leaves the ranges of the branch-free
// quotients; the caller then evaluates with weno5z_interp.
//
// What it buys (each interpolation has four quotients; a midpoint of the Euler
// sweep has ten interpolations and some twenty more quotients and roots): 256³
// explosion step, plain form, 23.6 → 18.5 ms; 4096 batched lines, 20 steps of
// the longest, 67.7 → 49.4 ms; five-equation 96³ step 6.4 → 4.3 ms; 48² single
// step 0.31 → 0.20 ms. FP64 pipe instructions per cell and sweep 1724 → 1338;
// what bounds the sweep now is that pipe (53–63 % active at 24 warps per SM)
// and the latency of the chains that feed it.
// one side; t2 = RN(3·v2), t3 = RN(3·v3)
__device__ __forceinline__ double weno5z_rn(double v0, double v1, double v2, double v3, double v4, double t2, double t3,
                                            bool& bad) {
    // 8·q_k: 6x = 2·RN(3x) exactly
    const double Q0 = (3.0 * v0 - 10.0 * v1) + 15.0 * v2;
    const double Q1 = fma(2.0, t2, -v1) + t3;
    const double Q2 = fma(2.0, t3, t2) - v4;
    // 2x, 4x and the factor 1/4 are exact, so the fused forms round as the separate ones
    const double D0 = fma(-2.0, v1, v0) + v2, B0 = fma(-4.0, v1, v0) + t2;
    const double D1 = fma(-2.0, v2, v1) + v3, B1 = v1 - v3;
    const double D2 = fma(-2.0, v3, v2) + v4, B2 = fma(-4.0, v3, t2) + v4;
    const double b0 = fma(0.25, sq(B0), (13.0 / 12.0) * sq(D0));
    const double b1 = fma(0.25, sq(B1), (13.0 / 12.0) * sq(D1));
    const double b2 = fma(0.25, sq(B2), (13.0 / 12.0) * sq(D2));
    const double tau = fabs(b0 - b2);
    const double x0 = b0 + WENO_EPS, x1 = b1 + WENO_EPS, x2 = b2 + WENO_EPS;
    const double a0 = 1.0 + sq(quot_rn(tau, recip_sq(x0)));
    const double a1 = 10.0 * (1.0 + sq(quot_rn(tau, recip_sq(x1))));
    const double a2 = 5.0 * (1.0 + sq(quot_rn(tau, recip_sq(x2))));
    const double n = (a0 * Q0 + a1 * Q1) + a2 * Q2;
    const double s = (a0 + a1) + a2;
    // x < 2^500 (x ≥ 1e-40 by construction; a τ so small that its remainder is
    // not exact gives a ratio whose square vanishes beside 1), 16 ≤ s < 2^500
    // (overflowed ratios and NaN fail this), |n| ≥ 2^-460, or 2^-900 for s < 2^60
    // (the weights of values that small are the linear ones, s = 16), or a zero
    // stencil
    const unsigned hx = max(hi_bits(x0), max(hi_bits(x1), hi_bits(x2)));
    const unsigned hn = hi_bits(n) & 0x7fffffffu;
    const unsigned nlo = hi_bits(s) < ((1023u + 60u) << 20) ? (1023u - 900u) << 20 : 0x23300000u;
    const bool zero = (((hi_bits(Q0) | hi_bits(Q1) | hi_bits(Q2)) << 1) |
                       (unsigned)(__double2loint(Q0) | __double2loint(Q1) | __double2loint(Q2))) == 0u;
    bad = bad || hx >= 0x5f300000u || hi_bits(s) >= 0x5f300000u || !(hn - nlo < 0x60000000u - nlo || zero);
    return quot_rn(n, recip_sq(8.0 * s));
}
__device__ __forceinline__ void weno5z_pair_rn(const double* v, double& left, double& right, bool& bad) {
    const double t2 = 3.0 * v[2], t3 = 3.0 * v[3];
    left = weno5z_rn(v[0], v[1], v[2], v[3], v[4], t2, t3, bad);
    right = weno5z_rn(v[5], v[4], v[3], v[2], v[1], t3, t2, bad);
}

}  // namespace emg
