// Per-pair, per-side, per-link and per-particle arithmetic of the default HiDEM
// functors, written for the device. Every expression keeps the reference's operand
// order and association (HiDEM/Common/HiDEMDefaultFunctions.h) and the translation
// units are compiled with -fmad=false and IEEE division / square root, so results
// are bit-identical to the reference's IEEE CPU build for the same inputs.
#pragma once
#include "internal.h"

namespace hidem {

__device__ __forceinline__ float lsqrt(float v) { return sqrtf(v); }
__device__ __forceinline__ double lsqrt(double v) { return sqrt(v); }
__device__ __forceinline__ float labs_(float v) { return fabsf(v); }
__device__ __forceinline__ double labs_(double v) { return fabs(v); }

// ---- six-component values: (x, u), (y, v), (z, w) as pairs in single precision ----
//
// The mixed build's functors are bound by instruction issue (the force pass issues about 500
// instructions per contact and link end with scalar arithmetic), and sm_100's packed
// instructions do two IEEE single-precision operations per issue slot (same rounding per
// component; the FP32 pipe's rate is unchanged: 0.48 packed against 0.95 scalar instructions
// per clock and scheduler measured): 1.44 ms per step on the 5.7M slab against 1.54 ms with
// scalar operations. A translational component and its rotational partner
// take the same operations with the same transformation entries, so they form the pairs.
struct Pair {
    unsigned long long v;
};
__device__ __forceinline__ Pair pair_of(float lo, float hi) {
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ Pair pair_at(const float *two) {  // 8-byte aligned
    Pair r;
    r.v = *reinterpret_cast<const unsigned long long *>(two);
    return r;
}
__device__ __forceinline__ Pair pair_of(float both) { return pair_of(both, both); }
__device__ __forceinline__ void unpair(Pair p, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p.v));
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b) {
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pair operator+(Pair a, Pair b) {
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pair operator-(Pair a, Pair b) {
    Pair r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pair pair_fma(Pair a, Pair b, Pair c) {
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// A packed product that feeds a packed sum is a fused multiply-add onto -0 (the same rounding,
// signed zeros included) whose -0 the compiler cannot see through: ptxas 12.9 contracts a
// packed product and a packed sum into one fused operation even under -fmad=false and with
// .rn on both (measured: 45 % of random a b + c d differ). The value comes out of a shuffle,
// so it also stays in a register pair instead of being loaded again at each use.
template <class LP>
struct Rounding;
template <>
struct Rounding<float> {
    Pair minusZero;
    __device__ __forceinline__ static Rounding make() {
        Rounding r;
        r.minusZero.v = __shfl_sync(0xffffffffu, 0x8000000080000000ull, 0);
        return r;
    }
    __device__ __forceinline__ Pair product(Pair a, Pair b) const { return pair_fma(a, b, minusZero); }
};
template <>
struct Rounding<double> {
    __device__ __forceinline__ static Rounding make() { return Rounding(); }
};

template <class LP>
struct Six;
template <>
struct Six<float> {
    Pair p[3];  // components (0, 3), (1, 4), (2, 5)
    __device__ __forceinline__ static Six zero() {
        Six r;
#pragma unroll
        for (int q = 0; q < 3; ++q) r.p[q].v = 0ull;
        return r;
    }
    __device__ __forceinline__ static Six of(const float *f) {
        Six r;
#pragma unroll
        for (int q = 0; q < 3; ++q) r.p[q] = pair_of(f[q], f[q + 3]);
        return r;
    }
    __device__ __forceinline__ void get(float *f) const {
#pragma unroll
        for (int q = 0; q < 3; ++q) unpair(p[q], f[q], f[q + 3]);
    }
    __device__ __forceinline__ Six operator+(const Six &o) const {
        Six r;
#pragma unroll
        for (int q = 0; q < 3; ++q) r.p[q] = p[q] + o.p[q];
        return r;
    }
    __device__ __forceinline__ Six operator-(const Six &o) const {
        Six r;
#pragma unroll
        for (int q = 0; q < 3; ++q) r.p[q] = p[q] - o.p[q];
        return r;
    }
    __device__ __forceinline__ Six times(Pair k) const {
        Six r;
#pragma unroll
        for (int q = 0; q < 3; ++q) r.p[q] = p[q] * k;
        return r;
    }
    __device__ __forceinline__ Six times(const Rounding<float> &R, Pair k) const {
        Six r;
#pragma unroll
        for (int q = 0; q < 3; ++q) r.p[q] = R.product(p[q], k);
        return r;
    }
};
template <>
struct Six<double> {
    double f[6];
    __device__ __forceinline__ static Six zero() {
        Six r;
#pragma unroll
        for (int q = 0; q < 6; ++q) r.f[q] = 0.0;
        return r;
    }
    __device__ __forceinline__ static Six of(const double *v) {
        Six r;
#pragma unroll
        for (int q = 0; q < 6; ++q) r.f[q] = v[q];
        return r;
    }
    __device__ __forceinline__ void get(double *v) const {
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = f[q];
    }
    __device__ __forceinline__ Six operator+(const Six &o) const {
        Six r;
#pragma unroll
        for (int q = 0; q < 6; ++q) r.f[q] = f[q] + o.f[q];
        return r;
    }
    __device__ __forceinline__ Six operator-(const Six &o) const {
        Six r;
#pragma unroll
        for (int q = 0; q < 6; ++q) r.f[q] = f[q] - o.f[q];
        return r;
    }
};

// ---- correctly rounded square root, reciprocal and quotient from one approximate 1/sqrt ----
//
// The functors take square roots, their reciprocals and quotients by powers of them. Each is
// IEEE-rounded in the reference; here they share one approximate reciprocal square root r and
// are brought to the correctly rounded value by fused multiply-add residuals (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34 (1990) 111-119), valid for arguments in [2^-90, 2^90] (roots) whose intermediate
// powers stay clear of the denormals; callers take the plain IEEE operations outside.
//   root:        g = v r, s = g + (v - g^2) (r / 2). Equal to the IEEE root for every
//                significand and exponent parity (checked exhaustively, tests/test_gpu_rounding.py).
//   reciprocal:  y1 = y0 + y0 (1 - b y0), y = y1 + y1 (1 - b y1). Equal to the IEEE reciprocal
//                for every significand but the all-ones one, whose iteration ends in a tie:
//                squared lengths with such a root (tie_root) take the IEEE operations.
//   quotient:    q1 = q0 + y (a - b q0), q = q1 + y (a - b q1) with y the rounded 1/b: the
//                IEEE quotient for every divisor but one of all ones (all_ones).
__device__ __forceinline__ float rsqrt_start(float v) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float root_from(float v, float r) {
    const float g = v * r;
    return __fmaf_rn(__fmaf_rn(-g, g, v), 0.5f * r, g);
}
__device__ __forceinline__ float recip_from(float b, float y0) {
    const float y1 = __fmaf_rn(y0, __fmaf_rn(-b, y0, 1.0f), y0);
    return __fmaf_rn(y1, __fmaf_rn(-b, y1, 1.0f), y1);
}
// (the quotient's three steps from the rounded reciprocal y of b)
__device__ __forceinline__ float quotient_from(float a, float b, float y) {
    const float q0 = a * y;
    const float q1 = __fmaf_rn(__fmaf_rn(-b, q0, a), y, q0);
    return __fmaf_rn(__fmaf_rn(-b, q1, a), y, q1);
}
// the two largest values below an even power of two: their roots round to all ones
__device__ __forceinline__ bool tie_root(float v) { return ((__float_as_uint(v) ^ 0x007ffffeu) & 0x00fffffeu) == 0u; }
__device__ __forceinline__ bool all_ones(float v) { return (~__float_as_uint(v) & 0x007fffffu) == 0u; }
constexpr float kFastLo = 9.094947017729282e-13f;  // 2^-40
constexpr float kFastHi = 1.099511627776e12f;      // 2^40
constexpr float kRootLo = 8.077935669463161e-28f;  // 2^-90
constexpr float kRootHi = 1.2379400392853803e27f;  // 2^90

// Contact / damping between two particles: HiDEMDefNeighForceFunc::operator()
// (HiDEMDefaultFunctions.h:21-87). s = self (xDiff..wDiff), sr its radius, o / orr the
// other. Adds the six values the functor adds to the forces, in component order.
//
// A pair beyond the active distance gets mask 0, and every term the functor adds is then
// 0 times a finite value (the distance is positive there): adding those signed zeros
// leaves each force component's value unchanged (a zero component at most changes its
// sign, which no later operation can observe), so such pairs skip the arithmetic. A NaN
// distance fails the comparison and takes the full path, as in the functor, whose mask
// of 1 multiplies nothing here. contact_terms writes the values for an in-range pair (the
// item kernel's zeros for a skipped one) and returns whether there are any.
__device__ __forceinline__ bool contact_terms(const Consts<float> &c, const Rounding<float> &R, float xDist, float yDist, float zDist,
                                              const Six<float> &s, float sr, const Six<float> &o, float orr,
                                              Six<float> &t) {
    const float d2 = xDist * xDist + yDist * yDist + zDist * zDist;
    const float radSum = sr + orr;
    if (d2 >= (radSum + c.attractDistance) * (radSum + c.attractDistance)) return false;
    float dist, inv;
    if (d2 >= kFastLo && d2 < kFastHi && !tie_root(d2)) {
        const float r = rsqrt_start(d2);
        dist = root_from(d2, r);
        inv = recip_from(dist, r);
    } else {
        dist = sqrtf(d2);
        inv = 1.0f / dist;
    }
    const float dim = radSum - dist;
    float Cnst = 0.f;
    if (dist < radSum) {
        const float d3 = dim * dim * dim;
        Cnst = (d3 >= kRootLo && d3 < kRootHi) ? root_from(d3, rsqrt_start(d3)) : sqrtf(d3);
    }
    if (dist >= radSum && dist < radSum + c.attractDistance) Cnst = c.attractScaleForce * dim;
    Cnst = Cnst * c.scaleE;
    t = (s - o).times(pair_at(c.neighPair)).times(R, pair_at(c.neighPair + 2));
    const float comp[3] = {Cnst * (xDist * inv), Cnst * (yDist * inv), Cnst * (zDist * inv)};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        float a, b;
        unpair(t.p[q], a, b);
        t.p[q] = pair_of(a + comp[q], b);
    }
    return true;
}
__device__ __forceinline__ bool contact_terms(const Consts<double> &c, const Rounding<double> &, double xDist, double yDist, double zDist,
                                              const Six<double> &s, double sr, const Six<double> &o, double orr,
                                              Six<double> &t) {
    const double d2 = xDist * xDist + yDist * yDist + zDist * zDist;
    const double radSum = sr + orr;
    if (d2 >= (radSum + c.attractDistance) * (radSum + c.attractDistance)) return false;
    const double dist = sqrt(d2);
    const double inv = 1.0 / dist;
    const double dim = radSum - dist;
    double Cnst = 0.0;
    Cnst = (dist < radSum) ? sqrt(dim * dim * dim) : Cnst;
    Cnst = (dist >= radSum && dist < radSum + c.attractDistance) ? c.attractScaleForce * dim : Cnst;
    Cnst = Cnst * c.scaleE;
    const double comp[3] = {xDist * inv, yDist * inv, zDist * inv};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        t.f[q] = (-c.damping) * ((s.f[q] - o.f[q]) * c.invDt) + Cnst * comp[q];
        t.f[q + 3] = (-c.dampingRotation) * ((s.f[q + 3] - o.f[q + 3]) * c.invDt);
    }
    return true;
}

template <class LP>
__device__ __forceinline__ void contact_pair(const Consts<LP> &c, const Rounding<LP> &R, LP xDist, LP yDist, LP zDist,
                                             const Six<LP> &s, LP sr, const Six<LP> &o, LP orr, Six<LP> &F) {
    Six<LP> t;
    if (contact_terms(c, R, xDist, yDist, zDist, s, sr, o, orr, t)) F = F + t;
}

// The beam functor's values of one link end's geometry: 1 / length, 1 / length in the xy
// plane, the two squared lengths, and the stiffnesses E W4 / L^3 and E W4 / (2 L^2).
template <class LP>
struct BeamGeometry {
    LP invLI, invLP, D, xy, K1, K5;
};
template <class LP>
__device__ __forceinline__ BeamGeometry<LP> beam_geometry_ieee(const Consts<LP> &c, LP xDist, LP yDist, LP zDist) {
    BeamGeometry<LP> g;
    LP xDist2 = xDist * xDist;
    LP yDist2 = yDist * yDist;
    if (xDist == LP(0) && yDist == LP(0)) {
        xDist2 = LP(1e-10);
        yDist2 = LP(1e-10);
    }
    g.xy = xDist2 + yDist2;
    g.D = g.xy + zDist * zDist;
    g.invLI = LP(1) / lsqrt(g.D);
    g.invLP = LP(1) / lsqrt(g.xy);
    const LP LI = g.invLI * g.D;
    const LP L2 = LI * LI;
    const LP L3 = LI * LI * LI;
    g.K1 = c.EW4 / L3;
    g.K5 = c.EW4 / (LP(2) * L2);
    return g;
}
// Two approximate reciprocal square roots (of the squared length and its xy part) start
// everything: the two roots, their reciprocals, and, from the powers of 1 / length, the two
// quotients; c.beamFastLo admits the arguments for which no intermediate value leaves
// the normal numbers (it is infinite when E W4 itself is out of range).
__device__ __forceinline__ BeamGeometry<float> beam_geometry(const Consts<float> &c, float xDist, float yDist,
                                                             float zDist) {
    const float xy = xDist * xDist + yDist * yDist;
    const float D = xy + zDist * zDist;
    if (!(xy >= c.beamFastLo && D < kFastHi) || tie_root(xy) || tie_root(D)) return beam_geometry_ieee<float>(c, xDist, yDist, zDist);
    BeamGeometry<float> g;
    g.xy = xy;
    g.D = D;
    const float rD = rsqrt_start(D), rxy = rsqrt_start(xy);
    g.invLI = recip_from(root_from(D, rD), rD);
    g.invLP = recip_from(root_from(xy, rxy), rxy);
    const float LI = g.invLI * D;
    const float L2 = LI * LI, L3 = L2 * LI;
    const float i2 = g.invLI * g.invLI;
    g.K1 = quotient_from(c.EW4, L3, recip_from(L3, i2 * g.invLI));
    g.K5 = quotient_from(c.EW4, 2.0f * L2, recip_from(2.0f * L2, 0.5f * i2));
    if (all_ones(L3) || all_ones(L2)) {
        g.K1 = c.EW4 / L3;
        g.K5 = c.EW4 / (2.0f * L2);
    }
    return g;
}
__device__ __forceinline__ BeamGeometry<double> beam_geometry(const Consts<double> &c, double xDist, double yDist,
                                                              double zDist) {
    return beam_geometry_ieee<double>(c, xDist, yDist, zDist);
}

// Bonded beam on one link end: HiDEMDefLinkForceFunc::operator()
// (HiDEMDefaultFunctions.h:90-204). CT is this side's history state (in/out). The
// functor adds two values to each force component, first the damping term (dp), later
// minus the turned CT term (ct here): beam_side applies them in that order. The functor's
// mask multiplies both: by 1 for a whole link, which changes nothing and is left out, and
// by 0 for a broken one (whose products are zeros, or NaN where a term is not finite).
__device__ __forceinline__ void beam_terms(const Consts<float> &c, const Rounding<float> &R, bool whole, float xDist, float yDist, float zDist,
                                           const Six<float> &s, const Six<float> &o, float *CT, Six<float> &dp,
                                           Six<float> &ct) {
    dp = (s - o).times(pair_at(c.linkPair)).times(R, pair_at(c.linkPair + 2));
    const BeamGeometry<float> g = beam_geometry(c, xDist, yDist, zDist);
    const float invLILP = g.invLI * g.invLP;
    const Pair T00 = pair_of(xDist * g.invLI), T01 = pair_of(yDist * g.invLI), T02 = pair_of(zDist * g.invLI);
    const Pair T10 = pair_of(-yDist * g.invLP), T11 = pair_of(xDist * g.invLP);
    const Pair T20 = pair_of(-(zDist * xDist) * invLILP);
    const Pair T21 = pair_of(-(zDist * yDist) * invLILP);
    const Pair T22 = pair_of(g.xy * invLILP);

    const Pair s03 = R.product(T00, s.p[0]) + R.product(T01, s.p[1]) + R.product(T02, s.p[2]);  // (B0, B3)
    const Pair s14 = R.product(T10, s.p[0]) + R.product(T11, s.p[1]);                            // (B1, B4)
    const Pair s25 = R.product(T20, s.p[0]) + R.product(T21, s.p[1]) + R.product(T22, s.p[2]);  // (B2, B5)
    const Pair o03 = R.product(T00, o.p[0]) + R.product(T01, o.p[1]) + R.product(T02, o.p[2]);  // (B6, B9)
    const Pair o14 = R.product(T10, o.p[0]) + R.product(T11, o.p[1]);                            // (B7, B10)
    const Pair o25 = R.product(T20, o.p[0]) + R.product(T21, o.p[1]) + R.product(T22, o.p[2]);  // (B8, B11)
    float B1, B4, B2, B5, B7, B10, B8, B11;
    unpair(s14, B1, B4);
    unpair(s25, B2, B5);
    unpair(o14, B7, B10);
    unpair(o25, B8, B11);

    const float K1 = g.K1, K5 = g.K5;
    const float LIDiv6 = (1.0f / 6.0f) * g.invLI;
    const float K4 = c.EW4 * LIDiv6;
    const float K3 = K4 * 2.0f;
    const Pair K02 = pair_of(c.EW2 * g.invLI, c.GW4 * LIDiv6);
    const Pair c03 = pair_of(CT[0], CT[3]) + (R.product(K02, s03) - R.product(K02, o03));
    // CT1 with CT5, CT2 with CT4: their four terms take the same B values
    const Pair c15 = pair_of(CT[1], CT[5]) +
                     (pair_of(K1 * B1, K5 * B1) + pair_of(K5 * B5, K3 * B5) - pair_of(K1 * B7, K5 * B7) +
                      pair_of(K5 * B11, K4 * B11));
    const Pair c24 = pair_of(CT[2], CT[4]) +
                     (pair_of(K1 * B2, -K5 * B2) + pair_of(-K5 * B4, K3 * B4) - pair_of(K1 * B8, -K5 * B8) +
                      pair_of(-K5 * B10, K4 * B10));
    unpair(c03, CT[0], CT[3]);
    unpair(c15, CT[1], CT[5]);
    unpair(c24, CT[2], CT[4]);
    const Pair c14 = pair_of(CT[1], CT[4]), c25 = pair_of(CT[2], CT[5]);
    ct.p[0] = R.product(T00, c03) + R.product(T10, c14) + R.product(T20, c25);
    ct.p[1] = R.product(T01, c03) + R.product(T11, c14) + R.product(T21, c25);
    ct.p[2] = R.product(T02, c03) + R.product(T22, c25);
    if (!whole) {
        dp = dp.times(R, pair_of(0.f));
        ct = ct.times(R, pair_of(0.f));
    }
}
__device__ __forceinline__ void beam_terms(const Consts<double> &c, const Rounding<double> &, bool whole, double xDist, double yDist,
                                           double zDist, const Six<double> &s, const Six<double> &o, double *CT,
                                           Six<double> &dp, Six<double> &ct) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        dp.f[q] = -c.linkDamping * ((s.f[q] - o.f[q]) * c.linkInvDt);
        dp.f[q + 3] = -c.linkDampingRotation * ((s.f[q + 3] - o.f[q + 3]) * c.linkInvDt);
    }
    const BeamGeometry<double> g = beam_geometry(c, xDist, yDist, zDist);
    const double invLI = g.invLI, invLP = g.invLP, invLILP = invLI * invLP;
    const double T00 = xDist * invLI, T01 = yDist * invLI, T02 = zDist * invLI;
    const double T10 = -yDist * invLP, T11 = xDist * invLP;
    const double T20 = -(zDist * xDist) * invLILP;
    const double T21 = -(zDist * yDist) * invLILP;
    const double T22 = g.xy * invLILP;

    const double B0 = T00 * s.f[0] + T01 * s.f[1] + T02 * s.f[2];
    const double B1 = T10 * s.f[0] + T11 * s.f[1];
    const double B2 = T20 * s.f[0] + T21 * s.f[1] + T22 * s.f[2];
    const double B4 = T10 * s.f[3] + T11 * s.f[4];
    const double B5 = T20 * s.f[3] + T21 * s.f[4] + T22 * s.f[5];
    const double B6 = T00 * o.f[0] + T01 * o.f[1] + T02 * o.f[2];
    const double B7 = T10 * o.f[0] + T11 * o.f[1];
    const double B8 = T20 * o.f[0] + T21 * o.f[1] + T22 * o.f[2];
    const double B10 = T10 * o.f[3] + T11 * o.f[4];
    const double B11 = T20 * o.f[3] + T21 * o.f[4] + T22 * o.f[5];

    const double LIDiv6 = (1.0 / 6.0) * invLI;
    const double K0 = c.EW2 * invLI;
    const double K1 = g.K1, K5 = g.K5;
    CT[0] = CT[0] + (K0 * B0 + (-K0) * B6);
    CT[1] = CT[1] + (K1 * B1 + K5 * B5 + (-K1) * B7 + K5 * B11);
    CT[2] = CT[2] + (K1 * B2 + (-K5) * B4 + (-K1) * B8 + (-K5) * B10);
    ct.f[0] = T00 * CT[0] + T10 * CT[1] + T20 * CT[2];
    ct.f[1] = T01 * CT[0] + T11 * CT[1] + T21 * CT[2];
    ct.f[2] = T02 * CT[0] + T22 * CT[2];

    const double K2 = c.GW4 * LIDiv6;
    const double K3 = c.EW4 * LIDiv6 * 2.0;
    const double K4 = c.EW4 * LIDiv6;
    const double B3 = T00 * s.f[3] + T01 * s.f[4] + T02 * s.f[5];
    const double B9 = T00 * o.f[3] + T01 * o.f[4] + T02 * o.f[5];
    CT[3] = CT[3] + (K2 * B3 + (-K2) * B9);
    CT[4] = CT[4] + ((-K5) * B2 + K3 * B4 + K5 * B8 + K4 * B10);
    CT[5] = CT[5] + (K5 * B1 + K3 * B5 + (-K5) * B7 + K4 * B11);
    ct.f[3] = T00 * CT[3] + T10 * CT[4] + T20 * CT[5];
    ct.f[4] = T01 * CT[3] + T11 * CT[4] + T21 * CT[5];
    ct.f[5] = T02 * CT[3] + T22 * CT[5];
    if (!whole) {
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            dp.f[q] = dp.f[q] * 0.0;
            ct.f[q] = ct.f[q] * 0.0;
        }
    }
}

template <class LP>
__device__ __forceinline__ void beam_side(const Consts<LP> &c, const Rounding<LP> &R, bool whole, LP xDist, LP yDist, LP zDist,
                                          const Six<LP> &s, const Six<LP> &o, LP *CT, Six<LP> &F) {
    Six<LP> dp, ct;
    beam_terms(c, R, whole, xDist, yDist, zDist, s, o, CT, dp, ct);
    F = (F + dp) - ct;
}

// Link break test: HiDEMDefLinkBreakFunc::operator() (HiDEMDefaultFunctions.h:207-242)
// with end A as particle 1 and end B as particle 2 and the functor's two thresholds.
// Returns the new state.
// (P: anything with x, y, z and th[3])
template <class LP, class P>
__device__ __forceinline__ uint8_t break_link(const LP bendBreak, const LP maxLoad, const P &a, const P &b,
                                              uint8_t state, LP initialLen) {
    if (state == 0) return 0;
    LP xDist = (LP)(a.x - b.x);
    LP yDist = (LP)(a.y - b.y);
    LP zDist = (LP)(a.z - b.z);
    LP stretchLength = lsqrt((xDist * xDist) + (yDist * yDist) + (zDist * zDist));
    LP ax = labs_(a.th[0] - b.th[0]);
    LP ay = labs_(a.th[1] - b.th[1]);
    LP az = labs_(a.th[2] - b.th[2]);
    LP myz = (ay < az) ? az : ay;  // std::max(ay, az)
    LP maxBend = (ax < myz) ? myz : ax;
    LP load = (stretchLength - initialLen) / initialLen + bendBreak * maxBend;
    return (load >= maxLoad) ? uint8_t(0) : state;
}
template <class LP>
__device__ __forceinline__ uint8_t break_link(const Consts<LP> &c, const PRec<LP> &a,
                                              const PRec<LP> &b, uint8_t state, LP initialLen) {
    return break_link<LP>(c.bendBreak, c.maxLoad, a, b, state, initialLen);
}

// Map2d::interp (PLiB/Geometry/Map2d.h:93-152, indices from getIndexes 93-111):
// bilinear interpolation on the map's grid in float arithmetic, the cell corner found by
// floor and clamped to the grid, the edge cases of a degenerate cell handled as there.
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
template <class LP>
__device__ __forceinline__ LP map_interp(const Map2dView &m, float x, float y) {
    const LP *d = static_cast<const LP *>(m.data);
    // (the float value is clamped before the integer conversion, which leaves every
    // in-range index as it is)
    float fx = floorf(((x - m.xMin) * m.invXMaxMin) * (float)(m.xPoints - 1));
    float fy = floorf(((y - m.yMin) * m.invYMaxMin) * (float)(m.yPoints - 1));
    fx = fminf(fmaxf(fx, -1.0f), (float)m.xPoints);
    fy = fminf(fmaxf(fy, -1.0f), (float)m.yPoints);
    const int xp = (int)fx, yp = (int)fy;
    const int xl = clampi(xp, 0, m.xPoints - 1), yl = clampi(yp, 0, m.yPoints - 1);
    const int xh = clampi(xp + 1, 0, m.xPoints - 1), yh = clampi(yp + 1, 0, m.yPoints - 1);
    if (xl == xh && yl == yh) return d[xl + yl * m.xPoints];
    const float v00 = (float)d[xl + yl * m.xPoints];
    const float v01 = (float)d[xl + yh * m.xPoints];
    const float v10 = (float)d[xh + yl * m.xPoints];
    const float v11 = (float)d[xh + yh * m.xPoints];
    const float x0 = x - m.xMin, y0 = y - m.yMin;
    const float x1 = (float)xl * m.xRes, x2 = (float)xh * m.xRes;
    const float y1 = (float)yl * m.yRes, y2 = (float)yh * m.yRes;
    const float invX21 = 1.0f / (x2 - x1);
    const float c1 = (x2 - x0) * invX21, c2 = (x0 - x1) * invX21;
    float fxy1 = (c1 * v00) + (c2 * v10);
    float fxy2 = (c1 * v01) + (c2 * v11);
    if (xl == xh) {
        fxy1 = v00;
        fxy2 = v01;
    } else if (yl == yh) {
        return (LP)fxy1;
    }
    const float invY21 = 1.0f / (y2 - y1);
    return (LP)((((y2 - y0) * invY21) * fxy1) + (((y0 - y1) * invY21) * fxy2));
}

// ------------------------------------------------------------------ collision mesh
// Real3f of the reference (PLiB/Util/Real3.h:142-258): float components; dot sums
// left to right, cross by components, no fused multiply-adds.
struct V3f {
    float x, y, z;
};
__device__ __forceinline__ V3f v3_sub(V3f a, V3f b) { return V3f{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3f v3_mul(V3f a, V3f b) { return V3f{a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ float v3_dot(V3f a, V3f b) { return (a.x * b.x) + (a.y * b.y) + (a.z * b.z); }
__device__ __forceinline__ V3f v3_cross(V3f a, V3f b) {
    return V3f{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float sign_f(float x) { return x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f); }

// squared distance of point p from an edge e = b - a with q = p - a: the edge term of
// MeshAccel::triSDF2, the projection parameter clamped to [0, 1] in lp (clamp3)
template <class LP>
__device__ __forceinline__ float tri_edge2(V3f e, V3f q) {
    const float t = v3_dot(e, q) / v3_dot(e, e);
    LP tl = (LP)t;
    tl = tl < LP(0) ? LP(0) : (tl > LP(1) ? LP(1) : tl);
    const float tc = (float)tl;
    const V3f d = v3_sub(v3_mul(e, V3f{tc, tc, tc}), q);
    return v3_dot(d, d);
}

// MeshAccel::triSDF2 (PLiB/Geometry/MeshAccel.h:329-372): squared distance of p from the
// triangle abc — the nearest edge when p projects outside it, else the plane distance.
template <class LP>
__device__ __forceinline__ LP tri_sdf2(V3f p, V3f a, V3f b, V3f c) {
    const V3f ba = v3_sub(b, a), pa = v3_sub(p, a);
    const V3f cb = v3_sub(c, b), pb = v3_sub(p, b);
    const V3f ac = v3_sub(a, c), pc = v3_sub(p, c);
    const V3f nor = v3_cross(ba, ac);
    const float s = sign_f(v3_dot(v3_cross(ba, nor), pa)) + sign_f(v3_dot(v3_cross(cb, nor), pb)) +
                    sign_f(v3_dot(v3_cross(ac, nor), pc));
    if (s < 2.0f) {
        const float e1 = tri_edge2<LP>(ba, pa), e2 = tri_edge2<LP>(cb, pb), e3 = tri_edge2<LP>(ac, pc);
        const float m12 = (e2 < e1) ? e2 : e1;  // std::min(e1, e2)
        return (LP)((e3 < m12) ? e3 : m12);
    }
    const float dn = v3_dot(nor, pa);
    return (LP)(dn * dn / v3_dot(nor, nor));
}

template <class LP>
__device__ __forceinline__ V3f mesh_vertex(const MeshView<LP> &m, int i) {
    return V3f{(float)m.vx[i], (float)m.vy[i], (float)m.vz[i]};
}

// MeshAccel::getCell of a point given as lp (getCellCord, MeshAccel.h:295-316): the
// point as Real3f, minus the lower corner, times the inverse cell size, truncated.
// -1 where the cell lies outside the grid (which the reference's bounding-box test
// admits only through rounding at the upper faces, and then reads past its arrays).
template <class LP>
__device__ __forceinline__ int mesh_cell(const MeshView<LP> &m, LP x, LP y, LP z) {
    const float cx = (float)((LP)(float)x - m.xLower);
    const float cy = (float)((LP)(float)y - m.yLower);
    const float cz = (float)((LP)(float)z - m.zLower);
    const int xc = (int)((LP)cx * m.xInv), yc = (int)((LP)cy * m.yInv), zc = (int)((LP)cz * m.zInv);
    if (xc < 0 || yc < 0 || zc < 0 || xc >= m.xCount || yc >= m.yCount || zc >= m.zCount) return -1;
    return (xc * m.yCount * m.zCount) + (yc * m.zCount) + zc;
}

// MeshAccel::getClosestTriAccel (MeshAccel.h:375-412): the closest triangle of the
// point's cell within interactDist (the first of equals), or -1; *dist2 its squared
// distance. The cell's list is the reference's with the triangles removed that lie
// farther from every point of the cell than any particle's interaction distance
// (k_mesh_prune): those never pass the distance test, so the closest triangle and its
// distance are the same, found with fewer distance evaluations.
template <class LP>
__device__ __forceinline__ int mesh_closest(const MeshView<LP> &m, LP x, LP y, LP z, LP interactDist,
                                            LP *dist2) {
    if (x > m.xUpper || y > m.yUpper || z > m.zUpper || x < m.xLower || y < m.yLower || z < m.zLower)
        return -1;
    const int cell = mesh_cell(m, x, y, z);
    if (cell < 0) return -1;
    const int start = m.qStarts[cell], size = m.qSizes[cell];
    if (size == 0) return -1;
    const V3f p{(float)x, (float)y, (float)z};
    const LP id2 = interactDist * interactDist;
    LP minDist = sizeof(LP) == 4 ? (LP)3.40282347e+38f : (LP)1.7976931348623157e+308;
    int closest = -1;
    for (int i = start; i < start + size; ++i) {
        const int tri = m.qValues[i];
        const LP cur = tri_sdf2<LP>(p, mesh_vertex(m, 3 * tri), mesh_vertex(m, 3 * tri + 1),
                                    mesh_vertex(m, 3 * tri + 2));
        if (id2 > cur && cur < minDist) {
            minDist = cur;
            closest = tri;
        }
    }
    *dist2 = minDist;
    return closest;
}

// The sample integrate step on one particle (HiDEM/MeshBlock/MainMeshBlock.cpp:182-261:
// gravity / buoyancy, air / water drag, HiDEMDefTimeIntegration
// HiDEMDefaultFunctions.h:318-370) plus the optional GlacierDem bed terms
// (HiDEM/GlacierDem/MainDem.cpp:176-207), HiDEMDefVelocityLimit (245-290),
// HiDEMDefBoundaryCondition (293-315) and the fixed-layer / front-pressure extensions.
// `p` is updated in place; F is the particle's accumulated force.
template <class LP>
__device__ __forceinline__ void integrate_particle(const Consts<LP> &c, PRec<LP> &p, uint8_t type,
                                                   LP *F) {
    if (c.useFixed && (type & HIDEM_TYPE_FIXED)) {
        for (int k = 0; k < 6; ++k) p.d[k] = LP(0);
        return;
    }
    double xCord = p.x, yCord = p.y, zCord = p.z;
    const LP xDiff = p.d[0], yDiff = p.d[1], zDiff = p.d[2];
    const LP uDiff = p.d[3], vDiff = p.d[4], wDiff = p.d[5];
    LP xTheta = p.th[0], yTheta = p.th[1], zTheta = p.th[2];
    const LP radius = p.r;
    const LP diameter = radius * LP(2);

    // bed height and friction under the particle: the GlacierDem maps
    // (InputBed::getHeight / getFric, PLiB/Geometry/InputGeometry.h:58-68) or constants
    LP bedHeight = c.bedHeight, bedFriction = c.bedFriction;
    if (c.useBed && c.useBedMap) bedHeight = map_interp<LP>(c.bedMap, (float)xCord, (float)yCord);
    LP dragCoeff;
    if (c.useBed && ((zCord + (double)radius) - (double)bedHeight < (double)c.bedInteract)) {
        if (c.useFricMap) bedFriction = map_interp<LP>(c.fricMap, (float)xCord, (float)yCord);
        LP a = c.bedDrag * bedFriction;
        LP b = LP(1e+5) * c.scale * c.scale;
        dragCoeff = (b < a) ? b : a;  // std::min(a, b)
    } else if (zCord > (double)c.waterLevel) {
        dragCoeff = c.airDrag;
    } else {
        dragCoeff = c.waterDrag;
    }
    LP xForce = F[0], yForce = F[1], zForce = F[2];
    LP uForce = F[3], vForce = F[4], wForce = F[5];
    const LP particleMass = c.rhoIce * diameter * diameter * diameter;
    const LP particleMomentInertia = particleMass * diameter * diameter / LP(6);

    if (zCord > (double)c.waterLevel) zForce = zForce + -c.g * particleMass;
    if (zCord <= (double)c.waterLevel) zForce = zForce + c.lift * particleMass;
    if (c.useBed && zCord + (double)radius < (double)bedHeight)
        zForce = (LP)((double)zForce +
                      (double)c.bedStiffness * ((double)bedHeight - (zCord + (double)radius)));
    // collision mesh (HiDEM/MeshConstrainedDem/MainMeshDem.cpp:220-235)
    if (c.useMesh) {
        LP dist2;
        const int tri = mesh_closest(c.mesh, (LP)xCord, (LP)yCord, (LP)zCord, c.bedInteract + radius, &dist2);
        if (tri >= 0) {
            const float maxDist = (float)(c.bedInteract + radius);
            const LP dist = lsqrt(dist2);
            dragCoeff = c.mesh.drag * ((LP)maxDist - dist);
            const LP fx = -c.mesh.nx[tri] * ((LP)maxDist - dist) * c.mesh.force;
            const LP fy = -c.mesh.ny[tri] * ((LP)maxDist - dist) * c.mesh.force;
            const LP fz = -c.mesh.nz[tri] * ((LP)maxDist - dist) * c.mesh.force;
            atomicAdd(&c.mesh.fx[tri], fx);
            atomicAdd(&c.mesh.fy[tri], fy);
            atomicAdd(&c.mesh.fz[tri], fz);
            xForce = xForce + fx;
            yForce = yForce + fy;
            zForce = zForce + fz;
        }
    }
    // external force maps (ExternalForces, PLiB/ExternalForces.h; MainDem.cpp:211-216)
    if (c.useExtMaps) {
        const float fx = (float)xCord, fy = (float)yCord;
        xForce = xForce + map_interp<LP>(c.extMap[0], fx, fy);
        yForce = yForce + map_interp<LP>(c.extMap[1], fx, fy);
        zForce = zForce + map_interp<LP>(c.extMap[2], fx, fy);
        uForce = uForce + map_interp<LP>(c.extMap[3], fx, fy);
        vForce = vForce + map_interp<LP>(c.extMap[4], fx, fy);
        wForce = wForce + map_interp<LP>(c.extMap[5], fx, fy);
    }
    if (c.useFront && (type & HIDEM_TYPE_FRONT) && zCord < (double)c.waterLevel) {
        LP depth = (LP)((double)c.waterLevel - zCord);
        xForce = xForce - c.rhoWater * c.g * depth * diameter * diameter;
    }

    const LP dragInvDt2 = dragCoeff * c.invDt2;
    const LP massDtSqr = particleMass * c.invDtSqr;
    const LP pMassDtSqr = particleMass / c.dtSqr;
    const LP pMemDtSqr = particleMomentInertia / c.dtSqr;
    const LP invC1 = LP(1) / (pMassDtSqr + dragCoeff * c.invDt2);
    const LP invC2 = LP(1) / (pMemDtSqr + dragCoeff * c.invDt2);
    const LP interDtSqr = particleMomentInertia * c.invDtSqr;
    const LP xDN = (xForce + massDtSqr * xDiff + dragInvDt2 * -xDiff) * invC1;
    const LP yDN = (yForce + massDtSqr * yDiff + dragInvDt2 * -yDiff) * invC1;
    const LP zDN = (zForce + massDtSqr * zDiff + dragInvDt2 * -zDiff) * invC1;
    const LP uDN = (uForce + interDtSqr * uDiff + dragInvDt2 * -uDiff) * invC2;
    const LP vDN = (vForce + interDtSqr * vDiff + dragInvDt2 * -vDiff) * invC2;
    const LP wDN = (wForce + interDtSqr * wDiff + dragInvDt2 * -wDiff) * invC2;

    const double xPrev = xCord, yPrev = yCord, zPrev = zCord;
    const LP xThPrev = xTheta, yThPrev = yTheta, zThPrev = zTheta;
    xCord = xCord + (double)xDN;
    yCord = yCord + (double)yDN;
    zCord = zCord + (double)zDN;
    xTheta = xTheta + uDN;
    yTheta = yTheta + vDN;
    zTheta = zTheta + wDN;

    if (c.useVel) {
        const LP xVel = xDN * c.mainInvDt, yVel = yDN * c.mainInvDt, zVel = zDN * c.mainInvDt;
        const LP xTV = (xTheta - xThPrev) * c.mainInvDt;
        const LP yTV = (yTheta - yThPrev) * c.mainInvDt;
        const LP zTV = (zTheta - zThPrev) * c.mainInvDt;
        if (xVel > c.maxVel) xCord = (double)(c.dt * c.maxVel) + xPrev;
        if (yVel > c.maxVel) yCord = (double)(c.dt * c.maxVel) + yPrev;
        if (zVel > c.maxVel) zCord = (double)(c.dt * c.maxVel) + zPrev;
        if (xTV > c.maxRot) xTheta = c.dt * c.maxRot + xThPrev;
        if (yTV > c.maxRot) yTheta = c.dt * c.maxRot + yThPrev;
        if (zTV > c.maxRot) zTheta = c.dt * c.maxRot + zThPrev;
        if (xVel < -c.maxVel) xCord = (double)(c.dt * -c.maxVel) + xPrev;
        if (yVel < -c.maxVel) yCord = (double)(c.dt * -c.maxVel) + yPrev;
        if (zVel < -c.maxVel) zCord = (double)(c.dt * -c.maxVel) + zPrev;
        if (xTV < -c.maxRot) xTheta = c.dt * -c.maxRot + xThPrev;
        if (yTV < -c.maxRot) yTheta = c.dt * -c.maxRot + yThPrev;
        if (zTV < -c.maxRot) zTheta = c.dt * -c.maxRot + zThPrev;
    }
    if (c.useBnd) {
        if (xCord + (double)radius < c.lower[0] && c.bmin[0]) xCord = xPrev;
        if (xCord - (double)radius > c.upper[0] && c.bmax[0]) xCord = xPrev;
        if (yCord + (double)radius < c.lower[1] && c.bmin[1]) yCord = yPrev;
        if (yCord - (double)radius > c.upper[1] && c.bmax[1]) yCord = yPrev;
        if (zCord + (double)radius < c.lower[2] && c.bmin[2]) zCord = zPrev;
        if (zCord - (double)radius > c.upper[2] && c.bmax[2]) zCord = zPrev;
    }
    p.x = xCord;
    p.y = yCord;
    p.z = zCord;
    p.th[0] = xTheta;
    p.th[1] = yTheta;
    p.th[2] = zTheta;
    p.d[0] = (LP)(xCord - xPrev);
    p.d[1] = (LP)(yCord - yPrev);
    p.d[2] = (LP)(zCord - zPrev);
    p.d[3] = xTheta - xThPrev;
    p.d[4] = yTheta - yThPrev;
    p.d[5] = zTheta - zThPrev;
}

}  // namespace hidem
