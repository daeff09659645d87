// sp_physics64.cuh — FP64 explicit steps of the two problems with angle charts.
//
// The Neel spherical and Brown+Neel Euler/spherical problems of sp_physics.cuh, in the same
// formulas, arranged for the FP64 pipe (8-cycle dependent operations, two issue cycles per
// warp instruction):
//  - the angles of a state are wrapped, and their sines and cosines taken, by straight-line
//    code with one rare branch for the lot, so that the five chains interleave;
//  - a particle near a pole stays in its rotated chart from step to step.  The reference
//    rotates the angles before each step and back after it; the two cancel, so only a step
//    on which the chart changes needs the conversion (two atan2 and an acos), where every
//    step of such a particle paid it twice and held up its warp;
//  - the formulas are evaluated in the chart's own frame and vectors moved between frames by
//    selects, one copy of the code instead of one per chart.
// Brown+Neel, FP64 (B200, one ensemble at a time): see step_min_blocks in sp_kernels.cuh.
#pragma once

#include <type_traits>

#include "sp_physics.cuh"

namespace sp {

// The angles of one state, all at once.  FP64: straight-line code for every angle and one
// rare branch for the lot, so that the angles' FP64 chains interleave (a branch per angle
// keeps the scheduler from moving code across it).
static __device__ __noinline__ double fmod_two_pi_any(double x) { return ::fmod(x, M<double>::two_pi); }
// high words of the largest magnitude (NaN and infinity compare above every bound)
template <int N>
__device__ __forceinline__ int max_high_word(const double* y) {
    int m = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) m = max(m, __double2hiint(y[i]) & 0x7fffffff);
    return m;
}
// fmod(x, 2pi) without the software remainder loop: for |x| < 4pi the single
// subtraction x -/+ 2pi is exact (Sterbenz), so the result equals fmod bit for bit;
// larger arguments, which one step never produces, fall back to fmod.
template <int N>
__device__ __forceinline__ void wrap_angles(double* y) {
    constexpr int kFourPiHigh = 0x402921fb;  // high word of 4 pi
    const bool large = max_high_word<N>(y) >= kFourPiHigh;
    double v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = y[i] - (::fabs(y[i]) >= M<double>::two_pi ? ::copysign(M<double>::two_pi, y[i]) : 0.0);
    if (large) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = fmod_two_pi_any(y[i]);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) y[i] = v[i];
}
// sines and cosines of N angles; WRAPPED: each within +-2 pi, or NaN
template <int N, bool WRAPPED>
__device__ __forceinline__ void sincos_angles(const double* y, double* s, double* c) {
    SinCosD r[N];
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = sincos_reduced(y[i]);
    if constexpr (!WRAPPED) {
        if (max_high_word<N>(y) >= kSincosRangeHigh) {
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = sincos_any(y[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) { s[i] = r[i].s; c[i] = r[i].c; }
}
// A rotated chart measures its angles from the world's -x axis: chart coordinates of a world
// vector and back (identity while the chart is not rotated).  Selects, not branches: a warp
// with one rotated lane would run both sides.
__device__ __forceinline__ V3<double> to_chart(bool rot, V3<double> v) { return {rot ? v.z : v.x, v.y, rot ? -v.x : v.z}; }
__device__ __forceinline__ V3<double> to_world(bool rot, V3<double> v) { return {rot ? -v.z : v.x, v.y, rot ? v.x : v.z}; }

// Thresholds of one chart: [0] unrotated, on the angle, [1] rotated, on the cosine of the world
// angle; outside [lo, hi] the next step uses the rotated chart.
struct ChartBounds {
    double lo[2], hi[2];
};
// angle < lo or > hi  <=>  cosine > cos lo or < cos hi, for angles in [0, pi]
__device__ __forceinline__ ChartBounds chart_bounds(bool enabled, double lo, double hi) {
    const double inf = __longlong_as_double(0x7ff0000000000000ll), pi = 3.14159265358979323846;
    ChartBounds b;
    b.lo[0] = enabled ? lo : -inf;
    b.hi[0] = enabled ? hi : inf;
    b.hi[1] = lo <= 0.0 ? 2.0 : (lo > pi ? -2.0 : ::cos(lo));
    b.lo[1] = hi < 0.0 ? 2.0 : (hi >= pi ? -2.0 : ::cos(hi));
    return b;
}
// whether the next step's chart is rotated: `angle` of the unrotated chart, `cosine` of the
// world angle
__device__ __forceinline__ bool wants_rotation(const ChartBounds& b, bool rot, double angle, double cosine) {
    const double v = rot ? cosine : angle;
    return v < b.lo[rot] || v > b.hi[rot];
}

// Chart conversions (NeelRelaxationSpherical.h:568-602,
// BrownAndNeelRelaxationEulerSpherical.h:859-899) from the sines and cosines at hand; `back`:
// the inverse.  Rare, so called.
struct SphAngles {
    double t, p;
};
static __device__ __noinline__ SphAngles sph_turn(bool back, double st, double ct, double sp, double cp) {
    return SphAngles{::acos(back ? cp * st : -cp * st), ::atan2(sp * st, back ? -ct : ct)};
}
struct EulerAngles {
    double a, b, c;
};
static __device__ __noinline__ EulerAngles euler_turn(bool back, double S0, double C0, double S1, double C1, double S2,
                                                      double C2) {
    EulerAngles r;
    const double u = C0 * C2 - C1 * S0 * S2, v = S0 * C2 + C1 * C0 * S2;
    r.a = back ? ::atan2(u, -v) : ::atan2(-u, v);
    r.b = ::acos(back ? S1 * S2 : -S1 * S2);
    r.c = ::atan2(back ? -C1 : C1, C2 * S1);
    return r;
}
static __device__ __noinline__ SinCosD sincos_reduced_called(double x) { return sincos_reduced(x); }
template <int N>
__device__ __forceinline__ void sincos_angles_called(const double* y, double* s, double* c) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const SinCosD r = sincos_reduced_called(y[i]);
        s[i] = r.s;
        c[i] = r.c;
    }
}

// ======================================================================= Neel (spherical)
template <int A>
struct NeelSphD : NeelSph<double, A> {
    using Base = NeelSph<double, A>;
    using Par = typename Base::Par;
    static constexpr bool kCarriedChart = true;
    struct Cache {
        bool rot;
        double odst, ct;
        V3<double> md, P0, P1;
    };
    // sines and cosines of the state's angles, which are those of chart `rot`
    struct Trig {
        double s[2], c[2];
        bool rot;
    };
    static __device__ __forceinline__ void trig(const double* y, Trig& t) {
        sincos_angles<2, false>(y, t.s, t.c);
        t.rot = false;
    }
    static __device__ __forceinline__ void prepare_t(const Par& q, const Rot<double>&, double*, Cache& c, const Trig& t) {
        c.rot = t.rot;
        cache_from(q, t.s[0], t.c[0], t.s[1], t.c[1], c);
    }
    static __device__ __forceinline__ void recompute(const Par& q, const double* y, Cache& c) {
        double s[2], co[2];
        sincos_angles<2, false>(y, s, co);
        cache_from(q, s[0], co[0], s[1], co[1], c);
    }
    static __device__ __forceinline__ void cache_from(const Par& q, double st, double ct, double sp, double cp, Cache& c) {
        c.ct = ct;
        c.odst = rcp_or_zero(st);
        const V3<double> eth = v3(ct * cp, ct * sp, -st), eph = v3(-sp, cp, 0.0);
        const V3<double> P0 = (-q.NF1) * eph + q.NF2 * eth;
        V3<double> P1 = c.odst * (q.NF1 * eth + q.NF2 * eph);
        P1.z = c.odst == 0.0 ? q.NF1 : P1.z;
        c.md = to_world(c.rot, v3(st * cp, st * sp, ct));
        c.P0 = to_world(c.rot, P0);
        c.P1 = to_world(c.rot, P1);
    }
    static __device__ __forceinline__ void finish(const Rot<double>&, double* y, const Cache&) { wrap_angles<2>(y); }
    static __device__ __forceinline__ void det(const Par& q, const double*, const Cache& c, const double* B, double* a) {
        const V3<double> H = Base::heff(q, c.md, B);
        a[0] = dot(c.P0, H);
        a[1] = dot(c.P1, H);
    }
    static __device__ __forceinline__ void drift(const Par& q, const double*, const Cache& c, double* d) {
        d[0] = -0.5 * q.Dp * c.ct * c.odst;
        d[1] = 0.0;
    }
    static __device__ __forceinline__ void bdw(const Par& q, const double*, const Cache& c, const double* w, double* r) {
        const V3<double> W = v3(w[0], w[1], w[2]);
        r[0] = q.DN * dot(c.P0, W);
        r[1] = q.DN * dot(c.P1, W);
    }
    static __device__ __forceinline__ int compensated(const Cache&) { return 0; }
    static __device__ __forceinline__ void out_t(const double* y, double* o, Trig& t) {
        sincos_angles<2, true>(y, t.s, t.c);  // every step ends wrapped
        const V3<double> m = to_world(t.rot, v3(t.s[0] * t.c[1], t.s[0] * t.s[1], t.c[0]));
        o[0] = m.x; o[1] = m.y; o[2] = m.z;
    }
    // the chart of the next step
    static __device__ __forceinline__ void rechart(const ChartBounds* b, double* y, Trig& t) {
        const bool want = wants_rotation(b[0], t.rot, y[0], t.s[0] * t.c[1]);
        if (want != t.rot) {
            const SphAngles n = sph_turn(t.rot, t.s[0], t.c[0], t.s[1], t.c[1]);
            y[0] = n.t; y[1] = n.p;
            sincos_angles_called<2>(y, t.s, t.c);
            t.rot = want;
        }
    }
    static __device__ __forceinline__ unsigned char chart_bits(const Trig& t) { return t.rot ? kChartNeel : 0; }
    static __device__ __forceinline__ void set_chart(unsigned char bits, Trig& t) { t.rot = bits & kChartNeel; }
};

// ======================================================================= Brown + Neel, Euler/spherical
// SHARED: the prefactors and the window sums live in shared memory, one column per lane, and
// are read where a formula uses them: 13 prefactors and 9 sums with their compensations are
// 62 of the 128 registers a thread has, and the compiler spilled 600-800 bytes of them and of
// the step's temporaries to local memory (now 100-200).  65536 particles, Millstein / Heun: 4.06 /
// 5.96 us per step in registers, 3.76 / 5.49 shared; 262144: 12.9 / - and 11.9 / -.  Not for
// the uniaxial+cubic anisotropy, whose 24 prefactors leave no room for a second CTA, nor where
// the increments are copied: those run few warps, unbound in registers.
struct SharedPar {
    uint32_t at;  // shared address of the lane's prefactor 0; prefactor i is 256 i bytes on
};
template <int A, bool SHARED = false>
struct BrownNeelEulerD : BrownNeelEuler<double, A> {
    using Base = BrownNeelEuler<double, A>;
    using Par = std::conditional_t<SHARED, SharedPar, typename Base::Par>;
    using Cache = typename Base::Cache;
    static constexpr bool kCarriedChart = true;
    static constexpr int kSharedPar = SHARED ? kParamsBrownNeelEuler : 0;
    // the prefactors in registers; unused ones are not read
    static __device__ __forceinline__ typename Base::Par params(const Par& q) {
        if constexpr (SHARED) {
            uint32_t at = q.at;
            asm volatile("" : "+r"(at));  // read again, not kept from an earlier use
            return Base::load_with([&](int i) {
                double v;
                asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at + 256u * static_cast<uint32_t>(i)));
                return v;
            });
        } else {
            return q;
        }
    }
    // sines and cosines of the state's angles, which are those of the charts br, nr
    struct Trig {
        double S[5], C[5];
        bool br, nr;
    };
    static __device__ __forceinline__ void trig(const double* y, Trig& t) {
        sincos_angles<5, false>(y, t.S, t.C);
        t.br = t.nr = false;
    }
    static __device__ __forceinline__ void prepare_t(const Par&, const Rot<double>&, double*, Cache& c, const Trig& t) {
        c.br = t.br;
        c.nr = t.nr;
#pragma unroll
        for (int i = 0; i < 5; ++i) { c.S[i] = t.S[i]; c.C[i] = t.C[i]; }
        cache_from(c);
    }
    static __device__ __forceinline__ void recompute(const Par&, const double* y, Cache& c) {
        sincos_angles<5, false>(y, c.S, c.C);
        cache_from(c);
    }
    static __device__ __forceinline__ void cache_from(Cache& c) {
        c.csc = rcp_or_zero(c.S[1]);
        c.odst = rcp_or_zero(c.S[3]);
        c.md = to_world(c.nr, v3(c.S[3] * c.C[4], c.S[3] * c.S[4], c.C[3]));
    }
    // body axes in world coordinates (columns of the Euler rotation matrix, :183-304)
    static __device__ __forceinline__ void axes(const double* S, const double* C, bool br, V3<double>& x, V3<double>& y,
                                                V3<double>& z) {
        const double cphicpsi = C[0] * C[2], sphicpsi = S[0] * C[2], cphispsi = C[0] * S[2], sphispsi = S[0] * S[2];
        x = to_world(br, v3(cphicpsi - C[1] * sphispsi, C[1] * sphicpsi + cphispsi, S[1] * S[0]));
        y = to_world(br, v3(-sphicpsi - C[1] * cphispsi, C[1] * cphicpsi - sphispsi, S[1] * C[0]));
        z = to_world(br, v3(S[1] * S[2], -S[1] * C[2], C[1]));
    }
    // E313^-1 applied to v (EulerProjectionMatrix, :228-237)
    static __device__ __forceinline__ V3<double> eproj(const Cache& c, V3<double> v) {
        const double ctheta = c.C[1], cpsi = c.C[2], spsi = c.S[2], csc = c.csc;
        const V3<double> u = to_chart(c.br, v);
        const double first = csc * (spsi * u.x - cpsi * u.y);
        return v3(first, cpsi * u.x + spsi * u.y, u.z - ctheta * first);
    }
    // spherical projection (:324-329), 2 rows applied to v
    static __device__ __forceinline__ void sproj(const Cache& c, V3<double> v, double* o) {
        const double ct = c.C[3], cp = c.C[4], sp = c.S[4], od = c.odst;
        const V3<double> u = to_chart(c.nr, v);
        o[0] = cp * u.y - sp * u.x;
        o[1] = u.z - od * (ct * (cp * u.x + sp * u.y));
    }
    static __device__ __forceinline__ void finish(const Rot<double>&, double* y, const Cache&) { wrap_angles<5>(y); }
    // :363-425
    static __device__ __forceinline__ void det(const Par& par, const double*, const Cache& c, const double* B, double* a) {
        const typename Base::Par q = params(par);
        V3<double> x, y, z;
        axes(c.S, c.C, c.br, x, y, z);
        const V3<double> H = Base::heff(q, c.md, x, y, z, B);
        const V3<double> cTe = Base::ctorque(q, c, c.md, x, y, z);
        const V3<double> mxH = cross(c.md, H);
        const V3<double> wb = eproj(c, cTe + q.d * mxH);
        a[0] = wb.x; a[1] = wb.y; a[2] = wb.z;
        sproj(c, (-q.a) * H + q.bpd * mxH + cTe, a + 3);
    }
    // :427-497 applied to w = (wA, wB)
    static __device__ __forceinline__ void bdw(const Par& par, const double*, const Cache& c, const double* w, double* r) {
        const typename Base::Par q = params(par);
        const V3<double> wA = v3(w[0], w[1], w[2]), wB = v3(w[3], w[4], w[5]);
        const V3<double> cwA = q.cF * wA;
        const V3<double> mxw = cross(c.md, wB);  // shared by both rows
        const V3<double> b = eproj(c, cwA + q.dDN * mxw);
        r[0] = b.x; r[1] = b.y; r[2] = b.z;
        sproj(c, cwA + q.bpdDN * mxw - q.aDN * wB, r + 3);
    }
    // :499-601: both charts alike by straight-line code, else (rare) replaced
    static __device__ __forceinline__ void drift(const Par& par, const double*, const Cache& c, double* r) {
        const typename Base::Par q = params(par);
        const double ctheta = c.C[1], cpsi = c.C[2], spsi = c.S[2];
        const double cos_t = c.C[3], cos_p = c.C[4], sin_t = c.S[3], sin_p = c.S[4];
        const double csc = c.csc;
        Base::drift_same(q, csc, ctheta, cpsi, spsi, cos_t, cos_p, sin_t, sin_p, r);
        if (c.br != c.nr) {
            const V3<double> m = be_drift_mixed_cold<double>(c.br, q.adDN2, q.d2fDN2, q.cF2h, csc, ctheta, cpsi, spsi,
                                                             cos_t, cos_p, sin_t, sin_p);
            r[0] = m.x; r[1] = m.y; r[2] = m.z;
        }
        r[3] = q.nd * c.odst * cos_t;  // :597
        r[4] = 0.0;
    }
    // :673-735: x-axis, y-axis, magnetisation
    static __device__ __forceinline__ void out_t(const double* y, double* o, Trig& t) {
        sincos_angles<5, true>(y, t.S, t.C);  // every step ends wrapped
        V3<double> ax, ay, az;
        axes(t.S, t.C, t.br, ax, ay, az);
        const V3<double> m = to_world(t.nr, v3(t.S[3] * t.C[4], t.S[3] * t.S[4], t.C[3]));
        o[0] = ax.x; o[1] = ax.y; o[2] = ax.z;
        o[3] = ay.x; o[4] = ay.y; o[5] = ay.z;
        o[6] = m.x; o[7] = m.y; o[8] = m.z;
    }
    // the charts of the next step
    static __device__ __forceinline__ void rechart(const ChartBounds* b, double* y, Trig& t) {
        const bool wb = wants_rotation(b[0], t.br, ::fabs(y[1]), t.S[1] * t.S[2]);
        const bool wn = wants_rotation(b[1], t.nr, ::fabs(y[3]), t.S[3] * t.C[4]);
        if (wb != t.br || wn != t.nr) {
            if (wb != t.br) {
                const EulerAngles n = euler_turn(t.br, t.S[0], t.C[0], t.S[1], t.C[1], t.S[2], t.C[2]);
                y[0] = n.a; y[1] = n.b; y[2] = n.c;
            }
            if (wn != t.nr) {
                const SphAngles n = sph_turn(t.nr, t.S[3], t.C[3], t.S[4], t.C[4]);
                y[3] = n.t; y[4] = n.p;
            }
            sincos_angles_called<5>(y, t.S, t.C);
            t.br = wb;
            t.nr = wn;
        }
    }
    static __device__ __forceinline__ unsigned char chart_bits(const Trig& t) {
        return static_cast<unsigned char>((t.br ? kChartBrown : 0) | (t.nr ? kChartNeel : 0));
    }
    static __device__ __forceinline__ void set_chart(unsigned char bits, Trig& t) {
        t.br = bits & kChartBrown;
        t.nr = bits & kChartNeel;
    }
};

}  // namespace sp
