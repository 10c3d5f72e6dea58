// lcb_roche.h — the eclipse search of one element behind a Roche-distorted star
// (crates/roche/src/eclipse.rs:123-373), compiled for the device (k_roche and
// its siblings, nvcc) and for the host (the tests' comparison of its two
// paths, g++) from this one source.
//
// Two paths give the same ingress and egress:
//   ingress_egress  the general one: the reference's phase scan, steps and
//                   blocks of steps proven to miss by second-order bounds of
//                   the potential, then its two bisections;
//   limb_*          for a convex star: the two limb contacts by Newton's
//                   method, which decide all but a few of the same scan steps
//                   and bisection steps without a line-of-sight search.
#pragma once

#include <math.h>

#include "lcb_internal.h"

#if defined(__CUDACC__)
#define LCB_HD __host__ __device__
#define LCB_ROCHE_CALL __host__ __device__ __noinline__
#else
#define LCB_HD
#define LCB_ROCHE_CALL inline
#endif

namespace lcb {
namespace roche {

constexpr double kPi = 3.14159265358979323846;
constexpr double kTwoPi = 2.0 * kPi;
#ifndef LCB_CERT_BUDGET
#define LCB_CERT_BUDGET 32
#endif
constexpr int kCertBudget = LCB_CERT_BUDGET;  // miss-proof nodes per line of sight before the full search
#ifndef LCB_TUBE_MAX
#define LCB_TUBE_MAX 8
#endif
constexpr int kTubeMax = LCB_TUBE_MAX;  // scan steps per phase-block miss proof (1: single steps only)
#ifndef LCB_TUBE_BUDGET
#define LCB_TUBE_BUDGET 24
#endif
constexpr int kTubeBudget = LCB_TUBE_BUDGET;  // nodes of one phase-block proof
constexpr int kTubeCool = 8;  // single steps after a failed two-step block before the next block
#ifndef LCB_CHOP_BUDGET
#define LCB_CHOP_BUDGET 0
#endif
constexpr int kChopBudget = LCB_CHOP_BUDGET;  // the same in the bisections (0: no proofs there)

LCB_HD inline double sq(double x) { return x * x; }
LCB_HD inline int imin(int a, int b) { return a < b ? a : b; }
LCB_HD inline int imax(int a, int b) { return a > b ? a : b; }
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ double inv_sqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float inv_sqrtf(float x) { return rsqrtf(x); }
#else
LCB_HD inline double inv_sqrt(double x) { return 1.0 / sqrt(x); }
LCB_HD inline float inv_sqrtf(float x) { return 1.0f / sqrtf(x); }
#endif

// Potential along a line of sight p + lam*e for the eclipse search
// (potential.rs:110-117).  1/r from rsqrt: decisions against pref differ
// from the divided form only within an ulp of the surface.
struct Los {
    double px, py, pz, ex, ey, ez;
};
LCB_HD inline double los_pot(const RocheEcl& s, const Los& L, double lam) {
    double x = fma(lam, L.ex, L.px), y = fma(lam, L.ey, L.py), z = fma(lam, L.ez, L.pz);
    double x2y2 = x * x + y * y;
    double r1sq = x2y2 + z * z;
    double r2sq = r1sq + 1.0 - 2.0 * x;
    double v = -s.comp * inv_sqrt(r1sq) - s.mu * inv_sqrt(r2sq);
    if (s.primary) return v - s.ssq * x2y2 * 0.5 + s.mu * x;
    return v - s.ssq * (0.5 + 0.5 * x2y2 - x) - s.comp * x;
}
LCB_HD inline double los_dpot(const RocheEcl& s, const Los& L, double lam) {  // potential.rs:120-127
    double x = fma(lam, L.ex, L.px), y = fma(lam, L.ey, L.py), z = fma(lam, L.ez, L.pz);
    double r1sq = x * x + y * y + z * z, r2sq = r1sq + 1.0 - 2.0 * x;
    double i1 = inv_sqrt(r1sq), i2 = inv_sqrt(r2sq);
    double comp = s.comp * (i1 * i1 * i1), mu1 = s.mu * (i2 * i2 * i2);
    double gx = comp * x + mu1 * (x - 1.0) - (s.primary ? s.ssq * x - s.mu : s.ssq * (x - 1.0) - s.mu + 1.0);
    double gy = comp * y + mu1 * y - s.ssq * y;
    double gz = comp * z + mu1 * z;
    return gx * L.ex + gy * L.ey + gz * L.ez;
}

// Work counters of the eclipse search (potential and gradient evaluations, fblink calls),
// and the bound on one line-of-sight search's potential evaluations (the reference has
// none; reaching it marks the model failed: kStatusIterCap).
struct EclCount {
    int pot = 0, dpot = 0, fbl = 0, cert = 0, skipped = 0;
    int cap = kFblinkEvalCap;
};

// dbrent with stop-fast (crates/subs/src/numerical/dbrent.rs:20-165).
// Returns 1 = bracketed minimum below fref, 0 = not below.
// `local` counts the search's evaluations so far; past cnt.cap the search stops
// and sets `capped` (the model then fails).
LCB_HD inline bool dbrent_below(const RocheEcl& s, const Los& L, double ax, double bx, double cx, double acc,
                             double fref, EclCount& cnt, int& local, bool& capped) {
    double a = fmin(ax, cx), b = fmax(ax, cx);
    double x = bx, w = bx, v = bx;
    if (local + 2 > cnt.cap) { capped = true; return false; }
    local += 2;
    double fx = los_pot(s, L, x), fw = fx, fv = fx;
    ++cnt.pot;
    if (fx < fref) return true;
    double dx = los_dpot(s, L, x), dw = dx, dv = dx;
    ++cnt.dpot;
    double e = 0.0, d = 0.0;
    for (int it = 0; it < 100; ++it) {
        double xm = 0.5 * (a + b);
        double tol1 = acc, tol2 = 2.0 * tol1;
        if (fabs(x - xm) <= tol2 - 0.5 * (b - a)) return fx < fref;
        if (fabs(e) > tol1) {
            double d1 = 2.0 * (b - a), d2 = d1;
            if (dw != dx) d1 = (w - x) * dx / (dx - dw);
            if (dv != dx) d2 = (v - x) * dx / (dx - dv);
            double u1 = x + d1, u2 = x + d2;
            bool ok1 = (a - u1) * (u1 - b) > 0.0 && dx * d1 <= 0.0;
            bool ok2 = (a - u2) * (u2 - b) > 0.0 && dx * d2 <= 0.0;
            double olde = e;
            e = d;
            if (ok1 || ok2) {
                d = (ok1 && ok2) ? (fabs(d1) < fabs(d2) ? d1 : d2) : (ok1 ? d1 : d2);
                if (fabs(d) <= fabs(0.5 * olde)) {
                    double u = x + d;
                    if (u - a < tol2 || b - u < tol2) d = (xm - x >= 0.0) ? fabs(tol1) : -fabs(tol1);
                } else {
                    e = dx >= 0.0 ? a - x : b - x;
                    d = 0.5 * e;
                }
            } else {
                e = dx >= 0.0 ? a - x : b - x;
                d = 0.5 * e;
            }
        } else {
            e = dx >= 0.0 ? a - x : b - x;
            d = 0.5 * e;
        }
        double u, fu;
        if (local + 2 > cnt.cap) { capped = true; return false; }
        local += 2;
        if (fabs(d) >= tol1) {
            u = x + d;
            fu = los_pot(s, L, u);
            ++cnt.pot;
            if (fu < fref) return true;
        } else {
            u = x + (d >= 0.0 ? fabs(tol1) : -fabs(tol1));
            fu = los_pot(s, L, u);
            ++cnt.pot;
            if (fu < fref) return true;
            if (fu > fx) return fx < fref;
        }
        double du = los_dpot(s, L, u);
        ++cnt.dpot;
        if (fu <= fx) {
            if (u >= x) a = x; else b = x;
            v = w; fv = fw; dv = dw;
            w = x; fw = fx; dw = dx;
            x = u; fx = fu; dx = du;
        } else {
            if (u < x) a = u; else b = u;
            if (fu <= fw || w == x) {
                v = w; fv = fw; dv = dw;
                w = u; fw = fu; dw = du;
            } else if (fu < fv || v == x || v == w) {
                v = u; fv = fu; dv = du;
            }
        }
    }
    return false;  // iteration cap: the reference maps its Err to "not eclipsed"
}

// Squared distances from the segment p + lam*e, lam in [a, b] (|e| = 1), to the
// two stars' centres (the primary at the origin, the secondary at (1, 0, 0)).
LCB_HD inline void closest_sq(const Los& L, double a, double b, double& d1, double& d2) {
    double t1 = fmin(fmax(-(L.px * L.ex + L.py * L.ey + L.pz * L.ez), a), b);
    double x1 = fma(t1, L.ex, L.px), y1 = fma(t1, L.ey, L.py), z1 = fma(t1, L.ez, L.pz);
    d1 = x1 * x1 + y1 * y1 + z1 * z1;
    double qx = L.px - 1.0;
    double t2 = fmin(fmax(-(qx * L.ex + L.py * L.ey + L.pz * L.ez), a), b);
    double x2 = fma(t2, L.ex, qx), y2 = fma(t2, L.ey, L.py), z2 = fma(t2, L.ez, L.pz);
    d2 = x2 * x2 + y2 * y2 + z2 * z2;
}

#ifndef LCB_PROOF_FAST_RSQRT
#define LCB_PROOF_FAST_RSQRT 1
#endif
// 1/sqrt(x) for the miss proofs' nodes: a single-precision hardware estimate
// (rsqrtf, within 2 ulp of FP32, i.e. relative error e0 < 2^-22) refined by one
// Newton-Raphson step for the inverse square root in FP64, y1 = y0 (3 - x y0^2) / 2,
// whose relative error is 3/2 e0^2 + O(e0^3) < 2e-13 plus a few FP64 roundings.
// The proofs' 1e-9 relative margin above the surface value covers that many
// times over; the reference-path evaluations (los_pot, los_dpot) keep rsqrt.
// The squared distances to the two centres along a line of sight (a few
// separations long, in units of the separation) lie far inside FP32's normal
// range; at x = 0 the result is NaN, so the node's bound fails and the line of
// sight is left to the full search.
LCB_HD inline double proof_rsqrt(double x) {
#if LCB_PROOF_FAST_RSQRT
    const double y = (double)inv_sqrtf((float)x);
    return y * fma(-0.5 * x, y * y, 1.5);
#else
    return inv_sqrt(x);
#endif
}

// The potential and its derivative along the line of sight at one point
// (los_pot and los_dpot sharing the two distances), and the gradient's norm
// when `grad` is not null.  For the miss proofs only (proof_rsqrt).
LCB_HD inline void los_pot_dpot(const RocheEcl& s, const Los& L, double lam, double& f, double& df,
                                             double* grad = nullptr) {
    double x = fma(lam, L.ex, L.px), y = fma(lam, L.ey, L.py), z = fma(lam, L.ez, L.pz);
    double x2y2 = x * x + y * y;
    double r1sq = x2y2 + z * z, r2sq = r1sq + 1.0 - 2.0 * x;
    double i1 = proof_rsqrt(r1sq), i2 = proof_rsqrt(r2sq);
    double v = -s.comp * i1 - s.mu * i2;
    f = s.primary ? v - s.ssq * x2y2 * 0.5 + s.mu * x : v - s.ssq * (0.5 + 0.5 * x2y2 - x) - s.comp * x;
    double comp = s.comp * (i1 * i1 * i1), mu1 = s.mu * (i2 * i2 * i2);
    double gx = comp * x + mu1 * (x - 1.0) - (s.primary ? s.ssq * x - s.mu : s.ssq * (x - 1.0) - s.mu + 1.0);
    double gy = comp * y + mu1 * y - s.ssq * y;
    double gz = comp * z + mu1 * z;
    df = gx * L.ex + gy * L.ey + gz * L.ez;
    if (grad) {  // |grad| = n2 / sqrt(n2), to the same 2e-13 (n2 = 0: NaN, the node fails)
        const double n2 = gx * gx + gy * gy + gz * gz;
        *grad = n2 * proof_rsqrt(n2);
    }
}

// True when the potential provably stays above the surface value on the whole
// line-of-sight segment [a, b]: an adaptive march over sub-segments, each
// certified by a second-order bound.  Along a line the Roche potential's
// second derivative is at least -M, M = 2 comp / r1^3 + 2 mu / r2^3 + ssq with
// r1, r2 the segment's closest approaches to the two centres (each gravity
// term -c / r has second derivative c (r^2 - 3 s^2) / r^5 >= -2 c / r^3, s the
// distance along the line from the closest point; the centrifugal term
// -ssq (x^2 + y^2) / 2 contributes -ssq (ex^2 + ey^2) >= -ssq; the rest is
// linear), so on a sub-segment of length h around m
//   phi >= phi(m) - |phi'(m)| h / 2 - M h^2 / 8.
// The bound must clear the surface value by 1e-9 relative (far above the
// rounding of any evaluation).  False means "not proven".
//
// With w > 0 the segment stands for a fan of lines through p whose unit
// directions lie within w of L's: every point of the fan at parameter t is
// within |t| w of L's point at t.  The Hessian of the potential has norm at
// most H = 2 comp / r1^3 + 2 mu / r2^3 + ssq with r1, r2 now the closest
// approaches of that tube, so a point x within r of the sub-segment's point y
// has phi(x) >= phi(y) - |grad phi(y)| r - H r^2 / 2, and
// |grad phi(y)| <= |grad phi(m)| + H h / 2: each node subtracts
// (|grad phi(m)| + H h / 2) r + H r^2 / 2, r = (|m| + h / 2) w.
template <bool kTube>
LCB_HD inline bool certify_miss(const RocheEcl& s, const Los& L, double a, double b, int budget,
                                             int& nodes, double w = 0.0) {
    const double thr = s.pref + 1e-9 * fmax(fabs(s.pref), 1.0);
    const double hmin = 1e-6 * (b - a);
    double d1, d2;
    closest_sq(L, a, b, d1, d2);
    const double i1 = inv_sqrt(d1), i2 = inv_sqrt(d2);
    const double curv = 2.0 * s.comp * (i1 * i1 * i1) + 2.0 * s.mu * (i2 * i2 * i2) + s.ssq;
    double hess = 0.0;
    if (kTube) {
        const double widen = fmax(fabs(a), fabs(b)) * w;
        const double r1 = sqrt(d1) - widen, r2 = sqrt(d2) - widen;
        if (!(r1 > 1e-3 && r2 > 1e-3)) return false;
        hess = 2.0 * s.comp / (r1 * r1 * r1) + 2.0 * s.mu / (r2 * r2 * r2) + s.ssq;
    }
    double t = a, h = b - a;
    for (int it = 0; it < budget; ++it) {
        if (t >= b) return true;
        double hh = fmin(h, b - t);
        ++nodes;
        const double m = t + 0.5 * hh;
        double f, df, g = 0.0;
        los_pot_dpot(s, L, m, f, df, kTube ? &g : nullptr);
        double bound = f - fabs(df) * (0.5 * hh) - curv * (0.125 * hh * hh);
        if (kTube) {
            const double r = (fabs(m) + 0.5 * hh) * w;
            bound -= (g + hess * (0.5 * hh)) * r + 0.5 * hess * r * r;
        }
        if (bound > thr) {
            t += hh;
            h = 2.0 * hh;
        } else {
            if (hh <= hmin) return false;
            h = 0.5 * hh;
        }
    }
    return t >= b;
}

// Is point p hidden from earth direction e by the Roche star? (eclipse.rs:123-197)
// With `prove` > 0 (a node budget), a line of sight whose first reference evaluation is not
// inside the star is first tested with the rigorous second-order bound: every point
// the reference search evaluates lies in [lam1 - acc, lam2 + acc] (dbrent.rs:116
// may step acc past an end), so a proven miss is exactly its "false".
// Not inlined: as a call, the search's working set does not add to the
// registers the surrounding scan/bisection loop keeps live, which lets the
// kernel run 5 blocks per SM (451 -> 350 ms on the 1024-model batch).
LCB_ROCHE_CALL bool fblink(const RocheEcl& s, double acc, const Los& L, EclCount& cnt, bool& capped, int prove) {
    ++cnt.fbl;
    double dx = L.px - s.cofmx, dy = L.py, dz = L.pz;
    double bq = L.ex * dx + L.ey * dy + L.ez * dz;  // sphere_eclipse_los, eclipse.rs:202-224
    if (bq >= 0.0) return false;
    double cq = (dx * dx + dy * dy + dz * dz) - sq(s.rref);
    double fac = sq(bq) - cq;
    if (fac <= 0.0) return false;
    fac = sqrt(fac);
    double lam2 = -bq + fac, lam1 = fmax(cq / lam2, 0.0);
    if (lam1 == 0.0) return true;
    const double pref = s.pref;
    double step = lam2 - lam1;
    if (!(step > acc)) return false;  // no evaluation: flam = 1 > f1 = f2 = 0
    // the reference's first evaluation, at the middle of the chord
    const double lam0 = lam1 + step / 2.0;
    double flam = los_pot(s, L, lam0);
    ++cnt.pot;
    if (flam <= pref) return true;
    if (prove > 0) {  // prove: the miss-proof node budget (0: no proof)
        const double pad = 1.001 * acc + 1e-12;
        if (certify_miss<false>(s, L, lam1 - pad, lam2 + pad, prove, cnt.cert)) { ++cnt.skipped; return false; }
    }
    int nstep = 1;
    double f1 = los_pot(s, L, lam1), f2 = los_pot(s, L, lam2), lam = lam0;
    int local = 2;
    bool br = flam < f1 && flam < f2;
    if (!br) {
        step /= 2.0;
        nstep = 2;
        while (step > acc) {
            lam = lam1 + step / 2.0;
            for (int n = 0; n < nstep; ++n) {
                flam = los_pot(s, L, lam + (double)n * step);
                ++local;
                if (flam <= pref) { cnt.pot += local; return true; }
                if (flam < f1 && flam < f2) { lam = lam + (double)n * step; br = true; break; }
            }
            if (br) break;
            if (local > cnt.cap) { capped = true; cnt.pot += local; return false; }
            step /= 2.0;
            nstep *= 2;
        }
    }
    cnt.pot += local;
    if (br) return dbrent_below(s, L, lam1, lam, lam2, acc, pref, cnt, local, capped);
    return false;
}

// Phase-block miss proof: L is the middle line of a block of consecutive scan
// steps whose unit directions lie within tube_w of L's (all lines pass through
// p).  True when every step of the block provably misses, i.e. each step's own
// fblink would return false (see certify_miss).  A separate call from fblink:
// the single-step search keeps its own, smaller register allocation.
LCB_ROCHE_CALL bool tube_miss(const RocheEcl& s, double acc, const Los& L, double tube_w, int budget,
                                       int& nodes) {
    const double dx = L.px - s.cofmx, dy = L.py, dz = L.pz;
    // every step's b = e.d lies within |d| tube_w of the middle line's; its chord of the
    // bounding sphere, where it has one, within [c / lam2max, lam2max] (lam2 = -b +
    // sqrt(b^2 - c) falls as b rises)
    const double dd = dx * dx + dy * dy + dz * dz;
    const double cq = dd - sq(s.rref);
    if (!(cq > 0.0)) return false;
    const double bmin = L.ex * dx + L.ey * dy + L.ez * dz - sqrt(dd) * tube_w;
    if (bmin >= 0.0) return true;  // every step: b >= 0, no chord
    const double fac = sq(bmin) - cq;
    if (fac <= 0.0) return true;   // every step misses the bounding sphere
    const double lam2 = -bmin + sqrt(fac), lam1 = cq / lam2;
    const double pad = 1.001 * acc + 1e-12;
    return certify_miss<true>(s, L, lam1 - pad, lam2 + pad, budget, nodes, tube_w);
}

LCB_HD inline void earth_at(double cosi, double sini, double phase, double& ex, double& ey, double& ez) {
    double sn, cs;  // misc.rs:42-45
    sincos(kTwoPi * phase, &sn, &cs);
    ex = sini * cs;
    ey = -sini * sn;
    ez = cosi;
}

// Analytic sphere eclipse (eclipse.rs:229-265).
LCB_HD inline bool sphere_phase(double cosi, double sini, double px, double py, double pz, double cx, double rs,
                             double& phi1, double& phi2, double& lam1, double& lam2) {
    double dx = px - cx, dy = py, dz = pz;
    double pdist = sqrt(sq(dx) + sq(dy));
    double bq = dz * cosi - pdist * sini;
    if (bq >= 0.0) return false;
    double cq = (dx * dx + dy * dy + dz * dz) - sq(rs);
    double fac = sq(bq) - cq;
    if (fac <= 0.0) return false;
    fac = sqrt(fac);
    lam2 = -bq + fac;
    lam1 = fmax(cq / lam2, 0.0);
    if (cq < 0.0) {
        phi1 = 0.0;
        phi2 = 1.0;
    } else {
        double delta = acos((cosi * dz + sqrt(cq)) / (sini * pdist));
        double phi = atan2(dy, -dx);
        double p1 = (phi - delta) / kTwoPi;
        p1 -= floor(p1);
        phi1 = p1;
        phi2 = p1 + 2.0 * delta / kTwoPi;
    }
    return true;
}

// Ingress/egress of point p behind a Roche-distorted star (eclipse.rs:270-373).
// The phase scan of pot_min_search (eclipse.rs:347-373) and the two bisections
// (eclipse.rs:301-332) run as one loop with a single line-of-sight search call
// site: lanes of a warp in different stages reconverge inside the search, and
// the search code exists once.  Misses are proven (fblink's `prove`) only in the
// scan, where nearly all lines of sight miss by a wide margin.
// The phase scan of pot_min_search (eclipse.rs:347-373): phases phi1 + i dphi,
// i = 0 .. nsteps, and the search tolerance acc (eclipse.rs:297).
struct Scan {
    double phi1, phi2, acc, dphi;
    int nsteps;
};
LCB_HD inline bool scan_setup(const RocheEcl& s, double cosi, double sini, double delta, double px,
                                           double py, double pz, Scan& sc) {
    double lam1, lam2;
    if (!sphere_phase(cosi, sini, px, py, pz, s.cofmx, s.rref, sc.phi1, sc.phi2, lam1, lam2)) return false;
    sc.acc = 2.0 * sqrt(2.0 * kTwoPi * (lam2 - lam1) * delta);
    double ns = ceil((sc.phi2 - sc.phi1) / (sc.acc / kTwoPi));
    sc.nsteps = (ns != ns || ns <= 10.0) ? 10 : (ns >= 1000.0 ? 1000 : (int)ns);
    sc.dphi = (sc.phi2 - sc.phi1) / (double)sc.nsteps;
    return true;
}

// Bound on |e(ph) - e(mid)| for phases within `half` of mid: the earth vector's
// xy part (length sini) turns by 2 pi (ph - mid), a chord of 2 sini sin(pi |ph - mid|).
LCB_HD inline double tube_width(double sini, double half) {
    return 2.0 * sini * sin(fmin(kPi * half, 0.5 * kPi)) * (1.0 + 1e-12) + 1e-15;
}

constexpr int kNoHit = 0x7f7f7f7f;  // first-hit sentinel (the byte pattern a memset of 0x7f writes)

// `known_hit` >= 0: the scan's first hit is already known (split scan): go
// straight to the bisections from that phase; kNoHit: the point is not eclipsed.
// `only` = 1 or 2 runs just the ingress or just the egress bisection (the two are
// independent: both start from the first hit), leaving `ing` resp. the unwrapped
// `eg` set; the caller then applies egress < ingress -> egress + 1 itself.
// kScan = false compiles the bisections alone (a known first hit is then required).
template <bool kScan>
LCB_HD inline bool ingress_egress(const RocheEcl& s, double cosi, double sini, double delta, double px, double py,
                               double pz, double& ing, double& eg, bool& capped, EclCount& evals, int known_hit = -1,
                               int only = 0) {
    Scan sc;
    if (!scan_setup(s, cosi, sini, delta, px, py, pz, sc)) return false;
    if (known_hit == kNoHit) return false;
    const double phi1 = sc.phi1, phi2 = sc.phi2, acc = sc.acc, dphi = sc.dphi;
    const int nsteps = sc.nsteps;
    Los L{px, py, pz, 0.0, 0.0, 0.0};
    enum { SCAN, CHOP_IN, CHOP_EG };
    // blk: scan steps the next phase-block proof covers; after a failed two-step block,
    // kTubeCool single steps before the next (wait)
    int mode = SCAN, i = 0, it = 0, blk = kTubeMax, wait = 0, last = 0;
    double phi = 0.0, pin = 0.0, pout = 0.0;
    if (known_hit >= 0) {  // as the scan below sets up its first hit
        phi = phi1 + (double)known_hit * dphi;
        if (only == 2) { mode = CHOP_EG; pin = phi; pout = phi2; }
        else { mode = CHOP_IN; pin = phi; pout = phi1; }
    }
    for (;;) {
        double ph, tube = 0.0;
        if (kScan && mode == SCAN) {
            if (i > nsteps) return false;  // no eclipsed phase found
            last = wait > 0 ? i : imin(i + blk - 1, nsteps);
            if (last > i) {  // steps i .. last at once: one phase-block proof
                ph = phi1 + 0.5 * (double)(i + last) * dphi;
                tube = tube_width(sini, 0.5 * (double)(last - i) * dphi);
            } else {
                ph = phi1 + (double)i * dphi;
            }
        } else {
            if (!(fabs(pin - pout) > delta) || it >= 200) {
                double r = (pin + pout) / 2.0;
                r -= floor(r);
                if (mode == CHOP_IN) {
                    ing = r;
                    if (only == 1) return true;
                    mode = CHOP_EG; pin = phi; pout = phi2; it = 0;
                    continue;
                }
                eg = r;
                if (only == 2) return true;
                if (eg < ing) eg += 1.0;
                return true;
            }
            ph = (pin + pout) / 2.0;
        }
        earth_at(cosi, sini, ph, L.ex, L.ey, L.ez);
        const bool hit = tube > 0.0 ? tube_miss(s, acc, L, tube, kTubeBudget, evals.cert)
                                    : fblink(s, acc, L, evals, capped, !(kScan && mode == SCAN) ? kChopBudget : kCertBudget);
        if (capped) return false;
        if (kScan && mode == SCAN) {
            if (tube > 0.0) {
                if (hit) {  // the block's steps are all misses: counted as the searches they stand for
                    evals.fbl += last - i + 1;
                    ++evals.skipped;  // one proof
                    i = last + 1;
                    blk = imin(2 * blk, kTubeMax);
                } else {
                    blk >>= 1;
                    if (blk < 2) wait = kTubeCool;
                }
            } else if (hit) { phi = ph; mode = CHOP_IN; pin = phi; pout = phi1; it = 0; }
            else {
                ++i;
                if (wait > 0) --wait;
                if (wait == 0) blk = imax(blk, imin(2, kTubeMax));
            }
        } else {
            if (hit) pin = ph; else pout = ph;
            ++it;
        }
    }
}


// ---------------------------------------------------------------------------
// the limb path
// ---------------------------------------------------------------------------
// For a convex star an element is hidden on one arc of phases, whose ends are
// where its line of sight touches the surface: phi(p + t e) = pref with
// grad phi . e = 0.  Newton's method in (t, phase) finds each of the two
// contacts in a few steps of one potential, gradient and Hessian-vector
// product.  Around a contact at phase c:
//   - the tangent plane there supports the star, so every line of sight on its
//     outer side misses: all phases from the start of the scan (or its end) up
//     to c; the reference search returns true only at a point it has evaluated
//     below the surface value, in the chord or within acc of it, and where the
//     plane has the companion's well behind it as well (well_behind; else the
//     element is left to the general path) none is, hence "false" there.
//     kLimbEps keeps clear of rounding.
//   - on the inner side the line dips below pref by |dphi_min/dphase| (phase -
//     c); dbrent ends within 2 acc of the minimum along the line, so it finds
//     a point below pref once that depth exceeds phi'' (2 acc)^2 / 2.  Twice
//     that depth is the contact's margin (an eighth of it would still give
//     the same decisions on random elements); lines between the margins hit.
// The steps of the scan and of the bisections that lie between a contact and
// its margin are decided by the reference's own search.  On the 1024-model
// batch that is ~6 searches an element instead of ~118 (of which ~80 were
// proven misses): 240 proof nodes and 370 evaluations became ~40 and ~60.
constexpr double kLimbEps = 1e-8;   // phase; Newton's contacts are within ~1e-13
constexpr int kLimbIters = 10;
enum { LIMB_NONE = 0, LIMB_ECLIPSED = 1, LIMB_OPEN = -1 };  // OPEN: left to the general path

struct Geom {  // an element and its scan
    double px, py, pz, cosi, sini;
    double cq, far;  // of the bounding sphere: |p - c|^2 - r^2, and the farthest point of any chord
    Scan sc;
};
struct Contact {
    double phi, margin;
    bool ok;
};

// The point at t along the line of sight at `phase`: potential f, gradient
// g, e, de/dphase and Hessian times e.
struct LosPoint {
    double x[3], e[3], de[2], f, g[3], he[3];
};
LCB_HD inline void los_point(const RocheEcl& s, const Geom& G, double phase, double t, LosPoint& P) {
    double sn, cs;
    sincos(kTwoPi * phase, &sn, &cs);
    P.e[0] = G.sini * cs; P.e[1] = -G.sini * sn; P.e[2] = G.cosi;
    P.de[0] = kTwoPi * P.e[1]; P.de[1] = -kTwoPi * P.e[0];
    const double x = fma(t, P.e[0], G.px), y = fma(t, P.e[1], G.py), z = fma(t, P.e[2], G.pz);
    P.x[0] = x; P.x[1] = y; P.x[2] = z;
    const double x2y2 = x * x + y * y, r1sq = x2y2 + z * z, r2sq = r1sq + 1.0 - 2.0 * x;
    const double i1 = inv_sqrt(r1sq), i2 = inv_sqrt(r2sq);
    const double v = -s.comp * i1 - s.mu * i2;
    P.f = s.primary ? v - s.ssq * x2y2 * 0.5 + s.mu * x : v - s.ssq * (0.5 + 0.5 * x2y2 - x) - s.comp * x;
    const double i1s = i1 * i1, i2s = i2 * i2, a = s.comp * (i1s * i1), b = s.mu * (i2s * i2), w = x - 1.0;
    P.g[0] = a * x + b * w - (s.primary ? s.ssq * x - s.mu : s.ssq * w - s.mu + 1.0);
    P.g[1] = (a + b - s.ssq) * y;
    P.g[2] = (a + b) * z;
    const double d1 = 3.0 * a * i1s * (x * P.e[0] + y * P.e[1] + z * P.e[2]);
    const double d2 = 3.0 * b * i2s * (w * P.e[0] + y * P.e[1] + z * P.e[2]);
    P.he[0] = (a + b - s.ssq) * P.e[0] - d1 * x - d2 * w;
    P.he[1] = (a + b - s.ssq) * P.e[1] - (d1 + d2) * y;
    P.he[2] = (a + b) * P.e[2] - (d1 + d2) * z;
}

LCB_HD inline bool geom_setup(const RocheEcl& s, double cosi, double sini, double delta, double px, double py, double pz,
                              Geom& G) {
    G.px = px; G.py = py; G.pz = pz; G.cosi = cosi; G.sini = sini;
    if (!scan_setup(s, cosi, sini, delta, px, py, pz, G.sc)) return false;
    const double dx = px - s.cofmx, b = pz * cosi - sqrt(dx * dx + py * py) * sini;
    G.cq = dx * dx + py * py + pz * pz - sq(s.rref);
    G.far = -b + sqrt(fmax(b * b - G.cq, 0.0)) + G.sc.acc;
    return true;
}

// Whether the limb path may be tried: a convex star, and the element clear of
// the bounding sphere (the search's chords then start well beyond acc).
LCB_HD inline bool limb_applies(const RocheEcl& s, const Geom& G) {
    return s.convex && G.cq > 4.0 * G.sc.acc * G.far;
}

// Whether the star's tangent plane through (x, y, z), outward normal n, has on its inner side all that
// a search may reach of the companion's well (roche_pad): then a line of sight on its outer side meets no
// potential below the surface value, in the chord or within acc of it.
LCB_ROCHE_CALL bool well_behind_rim(const RocheEcl& s, double along, double n1, double n2, double off) {
    const double aside = sqrt(n1 * n1 + n2 * n2);
    if (!(along > 0.0)) return off > along * s.pad_near + aside * s.pad_sin;
    return along * s.pad_sin <= aside * s.pad_cos && off > along * s.pad_cos + aside * s.pad_sin;
}
// First by a box about the well, which does for most; then by its rim, the farthest of it towards a plane
// whose normal is farther from the companion's direction than the rim.
LCB_HD inline bool well_behind(const RocheEcl& s, const double* n, double x, double y, double z) {
    const double along = s.primary ? n[0] : -n[0], aside = fabs(n[1]) + fabs(n[2]);  // at least the normal's part
    const double off = n[0] * (x - s.cofmx) + n[1] * y + n[2] * z;
    return off > along * (along > 0.0 ? s.pad_far : s.pad_near) + aside * s.pad_sin ||
           well_behind_rim(s, along, n[1], n[2], off);
}

// First guess of the contacts: those of the ellipsoid with the star's half
// widths ry (for x and y) and rz.  False: the ellipsoid is not touched.
LCB_HD inline bool limb_guess(const RocheEcl& s, const Geom& G, double& half) {
    const double k = s.ry / s.rz, dx = G.px - s.cofmx, dz = G.pz * k, ez = G.cosi * k;
    const double pd = sqrt(dx * dx + G.py * G.py);
    const double d2 = pd * pd + dz * dz - sq(s.ry);
    const double c = (ez * dz + sqrt((sq(G.sini) + ez * ez) * fmax(d2, 0.0))) / (G.sini * pd);
    half = c < 1.0 && d2 > 0.0 ? acos(fmax(c, -1.0)) / kTwoPi : 0.0;
    return half > 0.0;
}

// Newton's method for the ingress or egress contact from the guess `phi`.
LCB_HD inline Contact limb_contact(const RocheEcl& s, const Geom& G, bool egress, double phi, EclCount& cnt) {
    Contact c{phi, 0.0, false};
    double sn, cs;
    sincos(kTwoPi * phi, &sn, &cs);
    double t = -(G.sini * (cs * (G.px - s.cofmx) - sn * G.py) + G.cosi * G.pz);
    LosPoint P;
    double A = 0.0, B = 0.0;
    bool conv = false;
    for (int it = 0; it < kLimbIters && !conv; ++it) {
        los_point(s, G, phi, t, P);
        cnt.cert += 2;
        const double F1 = P.f - s.pref, F2 = P.g[0] * P.e[0] + P.g[1] * P.e[1] + P.g[2] * P.e[2];
        const double gde = P.g[0] * P.de[0] + P.g[1] * P.de[1];
        A = t * gde;                                                       // d f / d phase
        B = P.e[0] * P.he[0] + P.e[1] * P.he[1] + P.e[2] * P.he[2];        // d2 f / d t2
        const double C = t * (P.de[0] * P.he[0] + P.de[1] * P.he[1]) + gde;  // d2 f / d t d phase
        const double idet = 1.0 / (F2 * C - A * B);
        double dt = (A * F2 - C * F1) * idet, dphi = (B * F1 - F2 * F2) * idet;
        if (!(fabs(dphi) < 0.5 && fabs(dt) < 4.0)) return c;  // also NaN
        dphi = fmin(fmax(dphi, -0.02), 0.02);
        dt = fmin(fmax(dt, -0.2), 0.2);
        conv = fabs(dphi) < 1e-7 && fabs(dt) < 1e-6;  // quadratic: the step taken below leaves ~1e-13
        phi += dphi;
        t += dt;
    }
    if (!conv || !(B > 0.0) || !(t > 0.0) || !(phi >= G.sc.phi1 && phi <= G.sc.phi2)) return c;
    if (!(egress ? A > 1e-5 : A < -1e-5)) return c;
    // the tangent plane's outer side holds every line of sight from this end of the scan to the contact
    const double end = egress ? G.sc.phi2 : G.sc.phi1;
    sincos(kTwoPi * end, &sn, &cs);
    if (!(G.sini * (P.g[0] * cs - P.g[1] * sn) + G.cosi * P.g[2] > 0.0) || fabs(end - phi) > 0.45) return c;
    if (!well_behind(s, P.g, G.px, G.py, G.pz)) return c;  // the plane goes through the element
    c.phi = phi;
    c.margin = kLimbEps + 4.0 * B * sq(G.sc.acc) / fabs(A);
    c.ok = true;
    return c;
}

// Whether the star's tangent plane at (x, y, z), gradient n, has every line of
// sight of the element on its outer side: n . (p + t e - x) > 0 for every phase
// and every t that a chord of the bounding sphere reaches.
LCB_HD inline bool plane_clears(const Geom& G, const double* n, double x, double y, double z) {
    const double nxy = sqrt(n[0] * n[0] + n[1] * n[1]);
    const double low = fmin(n[2] * G.cosi - G.sini * nxy, 0.0);  // least n . e over every phase
    const double off = n[0] * (G.px - x) + n[1] * (G.py - y) + n[2] * (G.pz - z);
    return off + G.far * low > 1e-8 * sqrt(nxy * nxy + n[2] * n[2]);
}

// LIMB_NONE: provably never hidden, some tangent plane clears the element's
// lines of sight.  First the plane at the point of the surface that faces the
// middle line of sight on the ellipsoid of half widths ry and rz, which does
// for most; then the one below the lowest potential that any line reaches
// (Newton's method in t and phase), which does close to a graze.
// LIMB_ECLIPSED: that lowest point is inside the star; [lo, hi] the contacts'
// first guess from the minimum's curvature.  LIMB_OPEN: neither shown.
LCB_HD inline int limb_lowest(const RocheEcl& s, const Geom& G, double& lo, double& hi, EclCount& cnt) {
    double phi = 0.5 * (G.sc.phi1 + G.sc.phi2), sn, cs;
    sincos(kTwoPi * phi, &sn, &cs);
    LosPoint P;
    Geom at = G;
    {
        const double k = s.ry / s.rz, k2 = k * k, ex = G.sini * cs, ey = -G.sini * sn, dx = G.px - s.cofmx;
        const double t = -(ex * dx + ey * G.py + k2 * G.cosi * G.pz) / (G.sini * G.sini + k2 * G.cosi * G.cosi);
        double w[3] = {fma(t, ex, dx), fma(t, ey, G.py), fma(t, G.cosi, G.pz)};
        const double il = inv_sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
        for (int i = 0; i < 3; ++i) w[i] *= il;
        double r = s.ry * inv_sqrt(w[0] * w[0] + w[1] * w[1] + k2 * w[2] * w[2]), over = 1.0;
        for (int it = 0; it < kLimbIters; ++it) {
            at.px = fma(r, w[0], s.cofmx); at.py = r * w[1]; at.pz = r * w[2];
            los_point(s, at, phi, 0.0, P);
            ++cnt.cert;
            over = P.f - s.pref;
            if (fabs(over) < 1e-10) break;
            r = fmin(fmax(r - over / (P.g[0] * w[0] + P.g[1] * w[1] + P.g[2] * w[2]), 0.2 * s.rref), s.rref);
        }
        if (fabs(over) < 1e-10 && plane_clears(G, P.g, at.px, at.py, at.pz) && well_behind(s, P.g, at.px, at.py, at.pz))
            return LIMB_NONE;
    }
    double t = -(G.sini * (cs * (G.px - s.cofmx) - sn * G.py) + G.cosi * G.pz);
    double bend = 0.0;  // of the lowest potential in phase
    bool conv = false;
    for (int it = 0; it < kLimbIters && !conv; ++it) {
        los_point(s, G, phi, t, P);
        cnt.cert += 2;
        // the minimum of f(t, phase): grad . e = 0 and grad . de = 0
        const double F2 = P.g[0] * P.e[0] + P.g[1] * P.e[1] + P.g[2] * P.e[2];
        const double F3 = P.g[0] * P.de[0] + P.g[1] * P.de[1];
        const double x = P.x[0], y = P.x[1], z = P.x[2], w = x - 1.0;
        const double r1sq = x * x + y * y + z * z, r2sq = r1sq + 1.0 - 2.0 * x;
        const double i1 = inv_sqrt(r1sq), i2 = inv_sqrt(r2sq);
        const double a = s.comp * (i1 * i1 * i1), b = s.mu * (i2 * i2 * i2);
        const double q1 = x * P.de[0] + y * P.de[1], q2 = w * P.de[0] + y * P.de[1];
        const double de2 = P.de[0] * P.de[0] + P.de[1] * P.de[1];
        const double ehe = P.e[0] * P.he[0] + P.e[1] * P.he[1] + P.e[2] * P.he[2];
        const double dhe = P.de[0] * P.he[0] + P.de[1] * P.he[1];
        const double dhd = (a + b - s.ssq) * de2 - 3.0 * a * i1 * i1 * q1 * q1 - 3.0 * b * i2 * i2 * q2 * q2;
        const double J12 = t * dhe + F3, J22 = t * dhd - sq(kTwoPi) * (P.g[0] * P.e[0] + P.g[1] * P.e[1]);
        const double idet = 1.0 / (ehe * J22 - J12 * dhe);
        double dt = (J12 * F3 - J22 * F2) * idet, dphi = (dhe * F2 - ehe * F3) * idet;
        if (!(fabs(dphi) < 0.5 && fabs(dt) < 4.0)) return LIMB_OPEN;
        bend = t * J22 - J12 * J12 / ehe;
        dphi = fmin(fmax(dphi, -0.02), 0.02);
        dt = fmin(fmax(dt, -0.2), 0.2);
        conv = fabs(dphi) < 1e-5 && fabs(dt) < 1e-4;  // the plane's test holds for any point
        phi += dphi;
        t += dt;
    }
    if (!conv || !(t > 0.0)) return LIMB_OPEN;
    // down to the surface along the gradient
    double over = 0.0;
    at.px = fma(t, P.e[0], G.px); at.py = fma(t, P.e[1], G.py); at.pz = fma(t, P.e[2], G.pz);
    for (int k = 0; k < kLimbIters; ++k) {
        los_point(s, at, phi, 0.0, P);
        ++cnt.cert;
        over = P.f - s.pref;
        if (k == 0 && !(over > 1e-9)) {
            const double half = sqrt(fmax(-2.0 * over / bend, 0.0));
            lo = phi - half; hi = phi + half;
            return over < 0.0 && bend > 0.0 ? LIMB_ECLIPSED : LIMB_OPEN;
        }
        if (fabs(over) < 1e-10) break;
        const double m = over / (P.g[0] * P.g[0] + P.g[1] * P.g[1] + P.g[2] * P.g[2]);
        at.px -= m * P.g[0]; at.py -= m * P.g[1]; at.pz -= m * P.g[2];
    }
    return fabs(over) < 1e-10 && plane_clears(G, P.g, at.px, at.py, at.pz) && well_behind(s, P.g, at.px, at.py, at.pz)
               ? LIMB_NONE : LIMB_OPEN;
}

struct Limb {
    double in, out, in_far, out_far;  // the contacts, and where the margins end
};
LCB_HD inline bool limb_make(const Contact& a, const Contact& b, Limb& L) {
    if (!a.ok || !b.ok || !(b.phi > a.phi)) return false;
    // The margins take the depth to grow linearly from a contact; over a width w it falls short by a
    // share margin / w, within their factor of two if w is twice them.  A narrower eclipse has no
    // phase that hits for certain.
    const bool wide = b.phi - a.phi > 2.0 * (a.margin + b.margin);
    L.in = a.phi - kLimbEps; L.in_far = wide ? a.phi + a.margin : L.in + 4.0;
    L.out = b.phi + kLimbEps; L.out_far = b.phi - b.margin;
    return true;
}
// 1 hit, 0 miss, -1: the reference's own search decides
LCB_HD inline int limb_decide(const Limb& L, double ph) {
    return ph < L.in || ph > L.out ? 0 : ph > L.in_far && ph < L.out_far ? 1 : -1;
}

// The scan's first hit from the contacts (-1: none): steps before the ingress
// contact miss.  cnt.fbl counts the scan's searches as the reference makes them.
LCB_HD inline int limb_scan(const RocheEcl& s, const Geom& G, const Limb& L, bool& capped, EclCount& cnt) {
    const Scan& sc = G.sc;
    int i = imax(0, (int)fmin(floor((L.in - sc.phi1) / sc.dphi), 1e6));
    Los l{G.px, G.py, G.pz, 0.0, 0.0, 0.0};
    const int fbl = cnt.fbl;
    int hit = -1;
    for (; i <= sc.nsteps; ++i) {
        const double ph = sc.phi1 + (double)i * sc.dphi;
        int d = limb_decide(L, ph);
        if (d < 0) {
            earth_at(G.cosi, G.sini, ph, l.ex, l.ey, l.ez);
            d = fblink(s, sc.acc, l, cnt, capped, 0);
            if (capped) return -1;
        }
        if (d) { hit = i; break; }
        if (ph > L.out) break;
    }
    cnt.fbl = fbl + (hit >= 0 ? hit : sc.nsteps) + 1;
    cnt.skipped += 2;
    return hit;
}

// One of the two bisections from the scan's hit at phase `from`
// (eclipse.rs:301-332), each step decided as above; the phase in [0, 1).
LCB_HD inline double limb_chop(const RocheEcl& s, const Geom& G, const Limb& L, bool egress, double from, double delta,
                               bool& capped, EclCount& cnt) {
    double pin = from, pout = egress ? G.sc.phi2 : G.sc.phi1;
    Los l{G.px, G.py, G.pz, 0.0, 0.0, 0.0};
    int it = 0;
    for (;;) {
        double ph;
        int d = 0;
        for (;;) {  // the steps that need no search, then the lanes of a warp meet at one
            if (!(fabs(pin - pout) > delta) || it >= 200) {
                double r = (pin + pout) / 2.0;
                return r - floor(r);
            }
            ph = (pin + pout) / 2.0;
            ++it;
            d = limb_decide(L, ph);
            if (d < 0) break;
            ++cnt.fbl;
            if (d) pin = ph; else pout = ph;
        }
        earth_at(G.cosi, G.sini, ph, l.ex, l.ey, l.ez);
        if (fblink(s, G.sc.acc, l, cnt, capped, 0)) pin = ph; else pout = ph;
        if (capped) return 0.0;
    }
}

// The whole limb path of one element (the kernels run its parts, the two sides
// on two lanes).  LIMB_OPEN: use ingress_egress.
LCB_HD inline int limb_interval(const RocheEcl& s, double cosi, double sini, double delta, double px, double py, double pz,
                                double& ing, double& eg, bool& capped, EclCount& cnt) {
    Geom G;
    if (!geom_setup(s, cosi, sini, delta, px, py, pz, G)) return LIMB_NONE;
    if (!limb_applies(s, G)) return LIMB_OPEN;
    double half;
    const double mid = 0.5 * (G.sc.phi1 + G.sc.phi2);
    Limb L;
    bool found = limb_guess(s, G, half) &&
                 limb_make(limb_contact(s, G, false, mid - half, cnt), limb_contact(s, G, true, mid + half, cnt), L);
    if (!found) {
        double lo, hi;
        const int st = limb_lowest(s, G, lo, hi, cnt);
        if (st == LIMB_NONE) {
            cnt.fbl += G.sc.nsteps + 1;
            ++cnt.skipped;
            return LIMB_NONE;
        }
        found = st == LIMB_ECLIPSED && limb_make(limb_contact(s, G, false, lo, cnt), limb_contact(s, G, true, hi, cnt), L);
        if (!found) return LIMB_OPEN;
    }
    const int hit = limb_scan(s, G, L, capped, cnt);
    if (capped || hit < 0) return LIMB_NONE;
    const double from = G.sc.phi1 + (double)hit * G.sc.dphi;
    ing = limb_chop(s, G, L, false, from, delta, capped, cnt);
    eg = limb_chop(s, G, L, true, from, delta, capped, cnt);
    if (eg < ing) eg += 1.0;
    return LIMB_ECLIPSED;
}

}  // namespace roche
}  // namespace lcb
