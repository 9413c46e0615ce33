// FP64 per-pair code of the near-field kernels: the reference's expressions,
// shared by the FP64 twin and the FP32 kernel's re-evaluation of ambiguous
// pairs.
#pragma once
#include "kernels.h"
#include "table_row.cuh"

namespace agb {

constexpr double APPROX_ZERO_D = 1.0e-6;
constexpr double PI_D = 3.14159265358979323846;

template <class R>
struct PairQ {
    int ad4_in;   // inside 8 A and not a skipped disordered hydrogen
    int bin;      // (int)(r*A_DIV), unclamped
    int bin_e;    // LOOP 1 bin (nested hypot), unclamped
    int ih;       // disordered-hydrogen row bin, clamped to [0, NEINT-1]
    R r, inv_rmax, racc, rdon, Hramp;
};

// FP64, expression-for-expression restatement of main.cpp:3037-3272 for one
// (point, atom) pair.  Explicit _rn intrinsics keep nvcc from contracting.
// The distance part: LOOP 2's distance, cutoff and bins (main.cpp:3037-3046,
// :3309-3311) and LOOP 1's nested-hypot distance and 1/max(r, 0.5)
// (main.cpp:2951-2956).  Returns the pair vector and r.
template <class R>
__device__ __forceinline__ void dist_exact(const DevProblem &p, int ia, double cx, double cy, double cz, PairQ<R> &o,
                                           double &d0, double &d1, double &d2, double &r_out)
{
    d0 = __dsub_rn(p.x[ia], cx); d1 = __dsub_rn(p.y[ia], cy); d2 = __dsub_rn(p.z[ia], cz);
    double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2)));
    double re = hypot(d0, hypot(d1, d2));
    o.ad4_in = !(r > AG_NBC);
    if (p.disorder_h && p.disorder[ia] && p.type[ia] == p.hydrogen_type) o.ad4_in = 0;
    if (r < APPROX_ZERO_D) r = APPROX_ZERO_D;
    if (re < APPROX_ZERO_D) re = APPROX_ZERO_D;
    o.r = (R)r;
    o.inv_rmax = (R)__ddiv_rn(1.0, re > 0.5 ? re : 0.5);
    o.bin = __double2int_rz(__dmul_rn(r, (double)AG_A_DIV));
    o.bin_e = __double2int_rz(__dmul_rn(re, (double)AG_A_DIV));
    int ih = __double2int_rz(__dmul_rn(__dsub_rn(r, 1.10), (double)AG_A_DIV));
    ih = ih < 0 ? 0 : ih;
    o.ih = ih > AG_NEINT - 1 ? AG_NEINT - 1 : ih;
    r_out = r;
}

// Distance part only; the directional factors stay FP32.
static __device__ __noinline__ void dist_exact_f(const DevProblem &p, int ia, double cx, double cy, double cz,
                                          PairQ<float> &o)
{
    double d0, d1, d2, r;
    dist_exact(p, ia, cx, cy, cz, o, d0, d1, d2, r);
}

// Directional factors racc, rdon, Hramp of main.cpp:3075-3272 for the pair
// vector d (atom - point) of length r; ch: the point's closest DS/D1 atom.
static __device__ __noinline__ void angular_exact(const DevProblem &p, int ia, int ch, double d0, double d1, double d2,
                                                  double r, PairQ<double> &o)
{
    o.racc = 1.0; o.rdon = 1.0; o.Hramp = 1.0;
    const double inv_r = __ddiv_rn(1.0, r);
    const double dn0 = __dmul_rn(d0, inv_r), dn1 = __dmul_rn(d1, inv_r), dn2 = __dmul_rn(d2, inv_r);
    const int hb = p.hbond[ia];
    const double *rv = p.rv + 3 * (size_t)ia;
    const double PI_halved = PI_D / 2.;
    auto negdot = [&](const double *v) {
        double c = 0.;
        c = __dsub_rn(c, __dmul_rn(dn0, v[0]));
        c = __dsub_rn(c, __dmul_rn(dn1, v[1]));
        c = __dsub_rn(c, __dmul_rn(dn2, v[2]));
        return c;
    };
    if (hb == 2) {
        const double cos_theta = negdot(rv);
        if (cos_theta <= 0.) {
            o.racc = 0.;
        } else {
            const int e = p.rexp[ia];
            if (e == 2) o.racc = __dmul_rn(cos_theta, cos_theta);
            else if (e == 4) { const double t = __dmul_rn(cos_theta, cos_theta); o.racc = __dmul_rn(t, t); }
            else o.racc = cos_theta;
            if (ia == ch || ch < 0) {  // ch < 0: no DS/D1 candidate in reach, then no pair comes here
                o.Hramp = 1.;
            } else {
                const double *rh = p.rv + 3 * (size_t)ch;
                double ct = 0.;
                ct = __dadd_rn(ct, __dmul_rn(rh[0], rv[0]));
                ct = __dadd_rn(ct, __dmul_rn(rh[1], rv[1]));
                ct = __dadd_rn(ct, __dmul_rn(rh[2], rv[2]));
                ct = ct < 1.0 ? ct : 1.0;
                ct = ct > -1.0 ? ct : -1.0;
                const double theta = acos(ct);
                o.Hramp = __dsub_rn(0.5, __dmul_rn(0.5, cos(__ddiv_rn(__dmul_rn(theta, 120.), 90.))));
            }
        }
    } else if (hb == 4) {
        const double cos_theta = negdot(rv);
        o.rdon = (cos_theta <= 0.) ? 0. : __dmul_rn(cos_theta, cos_theta);
    } else if (hb == 5 && !p.disorder[ia]) {
        const double *rv2 = p.rv2 + 3 * (size_t)ia;
        const double cos_theta = negdot(rv);
        double t0 = 0.;
        t0 = __dadd_rn(t0, __dmul_rn(dn0, rv2[0]));
        t0 = __dadd_rn(t0, __dmul_rn(dn1, rv2[1]));
        t0 = __dadd_rn(t0, __dmul_rn(dn2, rv2[2]));
        if (t0 > 1.) t0 = 1.; else if (t0 < -1.) t0 = -1.;
        t0 = __dsub_rn(PI_halved, acos(t0));
        const double c0 = __dsub_rn(__dmul_rn(dn1, rv2[2]), __dmul_rn(dn2, rv2[1]));
        const double c1 = __dsub_rn(__dmul_rn(dn2, rv2[0]), __dmul_rn(dn0, rv2[2]));
        const double c2 = __dsub_rn(__dmul_rn(dn0, rv2[1]), __dmul_rn(dn1, rv2[0]));
        double rd2 = __dadd_rn(__dadd_rn(__dmul_rn(c0, c0), __dmul_rn(c1, c1)), __dmul_rn(c2, c2));
        if (rd2 < APPROX_ZERO_D) rd2 = APPROX_ZERO_D;
        const double inv_rd = __ddiv_rn(1.0, __dsqrt_rn(rd2));
        double ti = 0.;
        ti = __dadd_rn(ti, __dmul_rn(__dmul_rn(c0, inv_rd), rv[0]));
        ti = __dadd_rn(ti, __dmul_rn(__dmul_rn(c1, inv_rd), rv[1]));
        ti = __dadd_rn(ti, __dmul_rn(__dmul_rn(c2, inv_rd), rv[2]));
        o.rdon = 0.;
        if (cos_theta >= 0.) {
            if (ti > 1.) ti = 1.; else if (ti < -1.) ti = -1.;
            ti = __dsub_rn(acos(ti), PI_halved);
            if (ti < 0.) ti = -ti;
            o.rdon = __dmul_rn(__dadd_rn(0.9, __dmul_rn(0.1, sin(__dadd_rn(ti, ti)))), cos(t0));
        } else if (cos_theta >= -0.34202) {
            const double b = __dsub_rn(0.116978, __dmul_rn(cos_theta, cos_theta));
            o.rdon = __dmul_rn(__dmul_rn(562.25, pow(b, 3.)), cos(t0));
        }
    } else if (p.disorder[ia] && hb == 5) {
        double cos_theta = negdot(rv);
        if (cos_theta > 1.) cos_theta = 1.; else if (cos_theta < -1.) cos_theta = -1.;
        const double theta = acos(cos_theta);
        o.racc = 0.; o.rdon = 0.;
        if (theta <= 1.24791 + PI_halved) {
            o.rdon = pow(cos(__dsub_rn(theta, 1.24791)), 4.);
            o.racc = o.rdon;
        }
    }
}

// LOOP 2's distance of a pair (main.cpp:3037-3046), at least APPROX_ZERO.
__device__ __forceinline__ double loop2_dist(const DevProblem &p, int ia, double cx, double cy, double cz, double &d0,
                                             double &d1, double &d2)
{
    d0 = __dsub_rn(p.x[ia], cx); d1 = __dsub_rn(p.y[ia], cy); d2 = __dsub_rn(p.z[ia], cz);
    const double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2)));
    return r < APPROX_ZERO_D ? APPROX_ZERO_D : r;
}

// Per-atom metadata packed for shared memory (built by the host, capi.cu).
constexpr int META_TYPE_MASK = 31;          // bits 0-4   receptor type
constexpr int META_HB_SHIFT = 5;            // bits 5-7   hbond class
constexpr int META_REXP_SHIFT = 8;          // bits 8-10  rexp
constexpr int META_DIS = 1 << 11;           // disorder flag
constexpr int META_RVZERO = 1 << 12;        // bond vector exactly zero
constexpr int META_SKIP_AD4 = 1 << 13;      // disordered hydrogen skipped by LOOP 2 (main.cpp:3052)

// Exact distance of the reference's closest-H search (main.cpp:2994-3002).
__device__ __forceinline__ double h_dist(const DevProblem &p, int a, double cx, double cy, double cz)
{
    const double d0 = __dsub_rn(p.x[a], cx), d1 = __dsub_rn(p.y[a], cy), d2 = __dsub_rn(p.z[a], cz);
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2)));
}

}  // namespace agb
