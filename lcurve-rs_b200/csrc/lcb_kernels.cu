// lcb_kernels.cu — sm_100a kernels of the light-curve path, in launch order.
//
//   k_phase    : one thread per datum: ephemeris + Roemer phase and the
//                exposure sub-divisions (orchestration.rs:231-241,
//                flux.rs:379-387) with their earth vectors.
//   k_elements : one thread per grid element of every model in the batch.
//                Surface point (surface.rs:54-121) or sphere point, area,
//                gravity (grid.rs:201-322; disc/rim/spot grid.rs:336-553);
//                eclipse intervals by a spherical star (eclipse.rs:229-265)
//                and by an opaque disc (disc_eclipse.rs:84-330); continuum
//                flux (brightness.rs).  Elements eclipsed by a Roche-distorted
//                star keep that slot for k_roche.
//   k_roche    : two threads per element eclipsed by a Roche-distorted star:
//                the FP64 ray-march ingress_egress (eclipse.rs:270-373) decided
//                from the star's limb contacts (lcb_roche.h).  The elements that
//                path leaves open take the general one: k_roche_open (phase scan
//                with exact second-order miss proofs and bisections; for short
//                lists the scan alone, split over several threads, first hit by
//                atomicMin) and k_roche_chop2 (the bisections from that hit).
//   k_aux      : per star element, the per-model FP64 sums of ginterp,
//                wdwarf, log g and radii (flux.rs:115-206, 288-373).
//   k_flux     : persistent FP32 flux sum (flux.rs:7-111) over work units of
//                (element range x 512 sub-phases), a block's or a warp's each.
//                A first pass sorts the unit's elements into bit masks per
//                quarter of the tile's sub-phases: out of sight, plain, on the
//                limb, partly eclipsed; the sums then run over the masks, each
//                thread with 4 sub-phases in registers, in pairs on the packed
//                FP32x2 pipe, in FP32 blocks of 32 elements folded into a
//                two-sum pair.  Visibility is decided exactly in FP64 per
//                (element, tile) and per sub-phase only where an eclipse edge
//                falls inside the tile.
//   k_curve    : per datum, the slots' partial sums under the ginterp scale
//                factors, exposure smearing, slope/third (orchestration.rs:
//                243-310), in tiles of 32 data per block.
//   k_results  : per model, re_scale and chi-squared (361-401), log g, radii,
//                and with iscale = 1 the per-component fluxes and their
//                one-sided Jacobi SVD scale factors (405-436).
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "lcb_kernels.cuh"
#include "lcb_roche.h"
#include "lcb_stream.h"

namespace lcb {

namespace {

// LCURVE_DEBUG_BOUNDS build (make bounds): index checks that record
// kStatusBounds for the model and skip the access instead of reading or
// writing out of range; in the normal build they compile to nothing.
#ifdef LCURVE_DEBUG_BOUNDS
#define LCB_IN_BOUNDS(cond, status_word) ((cond) || (atomicOr((status_word), kStatusBounds), false))
#else
#define LCB_IN_BOUNDS(cond, status_word) true
#endif

using namespace roche;
constexpr double kFac1 = 2.0e27 * 6.6262e-34 * 2.99792458e8;      // planck.rs:5
constexpr double kFac2 = 1.0e9 * 6.6262e-34 * 2.99792458e8 / 1.3806e-23;  // planck.rs:8
constexpr double kFwhmEfac = 2.3548200450309493;                  // brightness.rs:8
constexpr double kEfac = 1.0000001;                               // grid.rs:396
#ifndef LCB_ROCHE_MIN_BLOCKS
#define LCB_ROCHE_MIN_BLOCKS 5
#endif
constexpr int kRocheMinBlocks = LCB_ROCHE_MIN_BLOCKS;  // k_roche blocks per SM (128 threads): register budget
#ifndef LCB_SCAN_MIN_BLOCKS
#define LCB_SCAN_MIN_BLOCKS LCB_ROCHE_MIN_BLOCKS
#endif
#ifndef LCB_CHOP_MIN_BLOCKS
#define LCB_CHOP_MIN_BLOCKS 4
#endif
constexpr int kScanMinBlocks = LCB_SCAN_MIN_BLOCKS;  // the same for the split scan (small batches)
constexpr int kChopMinBlocks = LCB_CHOP_MIN_BLOCKS;  // and for its bisection kernel
#ifndef LCB_FLUX_UNROLL
#define LCB_FLUX_UNROLL 2
#endif
#ifndef LCB_DISC_UNROLL
#define LCB_DISC_UNROLL 4
#endif
#ifndef LCB_LIMB_UNROLL
#define LCB_LIMB_UNROLL 2
#endif
#ifndef LCB_GENERIC_UNROLL
#define LCB_GENERIC_UNROLL 1
#endif
#ifndef LCB_FLUX_MIN_BLOCKS
#define LCB_FLUX_MIN_BLOCKS 4
#endif
constexpr int kFluxMinBlocks = LCB_FLUX_MIN_BLOCKS;  // k_flux blocks per SM (128 threads): register budget
__device__ __forceinline__ double rad2deg(double r) { return r * (180.0 / kPi); }

__device__ __forceinline__ double planck_d(double wave, double temp) {  // planck.rs:16-23
    double e = kFac2 / (wave * temp);
    if (e > 40.0) return kFac1 * exp(-e) / (wave * sq(wave));
    return kFac1 / (exp(e) - 1.0) / (wave * sq(wave));
}

// ---------------------------------------------------------------------------
// Roche potentials
// ---------------------------------------------------------------------------
// Exact-rounding potential (surface.rs:54-121 builds the stars from it).
__device__ __forceinline__ double pot_exact(bool primary, double q, double ssq, double x, double y, double z) {
    double mu = q / (1.0 + q), comp = 1.0 - mu;
    double x2y2 = sq(x) + sq(y);
    double r1sq = x2y2 + sq(z);
    double r1 = sqrt(r1sq), r2 = sqrt(r1sq + 1.0 - 2.0 * x);
    if (primary) return -comp / r1 - mu / r2 - ssq * x2y2 / 2.0 + mu * x;
    return -comp / r1 - mu / r2 - ssq * (0.5 + 0.5 * x2y2 - x) - comp * x;
}
__device__ __forceinline__ void dpot_exact(bool primary, double q, double ssq, double x, double y, double z,
                                           double& gx, double& gy, double& gz) {
    double r1sq = x * x + y * y + z * z, r2sq = r1sq + 1.0 - 2.0 * x;
    double r1 = sqrt(r1sq), r2 = sqrt(r2sq);
    double mu = q / (1.0 + q);
    double mu1 = mu / r2 / r2sq, comp = (1.0 - mu) / r1 / r1sq;
    gx = comp * x + mu1 * (x - 1.0) - (primary ? ssq * x - mu : ssq * (x - 1.0) - mu + 1.0);
    gy = comp * y + mu1 * y - ssq * y;
    gz = comp * z + mu1 * z;
}

// Disc occultation (disc_eclipse.rs:29-70, 84-330); returns the number of pairs (<= 2).
__device__ __forceinline__ double cut_phase(double rxy, double rcone, double radius) {
    double c = (sq(rxy) + sq(rcone) - sq(radius)) / (2.0 * rcone * rxy);
    return acos(fmin(fmax(c, -1.0), 1.0)) / kTwoPi;
}
enum { C_ABOVE, C_INSIDE, C_OUTSIDE, C_SEPARATE, C_CROSSING };
__device__ __forceinline__ int circle_ecl(double rxy, double z, double zc, double radius, double tani, double& ph) {
    ph = 0.0;
    if (z >= zc) return C_ABOVE;
    double rcone = tani * (zc - z);
    if (rcone >= rxy + radius) return C_OUTSIDE;
    if (rxy >= rcone + radius) return C_SEPARATE;
    if (rxy + rcone <= radius) return C_INSIDE;
    ph = cut_phase(rxy, rcone, radius);
    return C_CROSSING;
}
__device__ int disc_eclipse(const ModelDev& M, double rdisc1, double px, double py, double pz, double* ing,
                            double* eg) {
    const double rdisc2 = M.rdisc2, beta = M.beta, height = M.height;
    double hout = height * pow(rdisc2, beta);
    if (pz >= hout) return 0;
    double sini = M.sini_d, cosi = M.cosi_d;
    if (cosi == 0.0) {
        if (fabs(pz) < hout) {
            double rxy = sqrt(sq(px) + sq(py));
            if (rxy <= rdisc2) { ing[0] = 0.0; eg[0] = 1.0; return 1; }
            double subtend = asin(rdisc2 / rxy) / kTwoPi;
            double pc = atan2(py, -px) / kTwoPi;
            double i0 = pc - subtend;
            i0 -= floor(i0);
            ing[0] = i0; eg[0] = i0 + 2.0 * subtend;
            return 1;
        }
        return 0;
    }
    double rxy = sqrt(sq(px) + sq(py));
    if (rdisc1 < rxy && rxy < rdisc2 && fabs(pz) < height * pow(rxy, beta)) { ing[0] = 0.0; eg[0] = 1.1; return 1; }
    double tani = sini / cosi;
    if (rxy < rdisc2 && pz >= height * pow(fmax(rdisc1, rxy), beta)) {
        double ph;
        int r = circle_ecl(rxy, pz, hout, rdisc2, tani, ph);
        if (r == C_OUTSIDE) { ing[0] = 0.0; eg[0] = 1.1; return 1; }
        if (r == C_CROSSING) {
            double i0 = atan2(py, -px) / kTwoPi + ph;
            i0 -= floor(i0);
            ing[0] = i0; eg[0] = i0 + 1.0 - 2.0 * ph;
            return 1;
        }
        return 0;
    }
    double rlo = fmax(tani * (-hout - pz), 0.0);
    if (rlo >= rxy + rdisc2) return 0;
    double rhi = tani * (hout - pz);
    if (rxy >= rhi + rdisc2) return 0;
    double ecl;
    if (rxy + rlo <= rdisc2) ecl = 0.5;
    else if (rxy <= rdisc2) ecl = cut_phase(rxy, rlo, rdisc2);
    else if (sq(rhi) + sq(rdisc2) >= sq(rxy) && sq(rlo) + sq(rdisc2) <= sq(rxy)) ecl = asin(rdisc2 / rxy) / kTwoPi;
    else if (sq(rhi) + sq(rdisc2) < sq(rxy)) ecl = cut_phase(rxy, rhi, rdisc2);
    else ecl = cut_phase(rxy, rlo, rdisc2);
    double hin = height * pow(rdisc1, beta);
    double app = -1.0;
    auto first = [&](double zc, double rad) {
        double ph;
        int r = circle_ecl(rxy, pz, zc, rad, tani, ph);
        if (r == C_INSIDE) app = 0.5; else if (r == C_CROSSING) app = ph;
    };
    auto next = [&](double zc, double rad) {
        if (!(app > 0.0)) return;
        double ph;
        int r = circle_ecl(rxy, pz, zc, rad, tani, ph);
        if (r == C_CROSSING) app = fmin(app, ph); else if (r != C_INSIDE) app = -1.0;
    };
    if (pz < -hout) {
        first(-hout, rdisc2); next(-hin, rdisc1); next(hin, rdisc1); next(hout, rdisc2);
    } else if (rxy < rdisc1) {
        if (pz < -hin) { first(-hin, rdisc1); next(hin, rdisc1); next(hout, rdisc2); }
        else if (pz < hin) { first(hin, rdisc1); next(hout, rdisc2); }
    }
    double phi0 = atan2(py, -px) / kTwoPi;
    if (app <= 0.0) {
        double i0 = phi0 - ecl;
        i0 -= floor(i0);
        ing[0] = i0; eg[0] = i0 + 2.0 * ecl;
        return 1;
    }
    if (app < ecl) {
        double i0 = phi0 - ecl;
        i0 -= floor(i0);
        ing[0] = i0; eg[0] = i0 + (ecl - app);
        double i1 = phi0 + app;
        i1 -= floor(i1);
        ing[1] = i1; eg[1] = i1 + (ecl - app);
        return 2;
    }
    return 0;
}

// Where the ray from a Roche star's centre along (ux, uy, uz) meets its surface
// (potential = pref): Newton's method from the ellipsoid of half widths ry and
// rz.  The bisection of surface.rs:54-121 needs only the side of the surface a
// radius lies on; away from the root by more than `tol` (the rounding of its
// own potential evaluation, thousands of times over) the root tells, so the ~25
// evaluations of two square roots and divisions each become ~5 of two
// reciprocal square roots, and the steps decide alike: the radius is the same
// to the bit where they are taken one by one, to a unit or two in the last
// place where `bisected` computes their end.  Not converged, or too flat to
// trust (near L1): tol is infinite and every step evaluates.
struct FaceRoot {
    double r, tol;
};
__device__ __forceinline__ FaceRoot face_root(const RocheEcl& s, double ux, double uy, double uz) {
    double r = inv_sqrt((ux * ux + uy * uy) / (s.ry * s.ry) + uz * uz / (s.rz * s.rz)), dr = 1.0, slope = 0.0;
    for (int it = 0; it < 8 && fabs(dr) > 1e-9; ++it) {
        const double x = fma(r, ux, s.cofmx), y = r * uy, z = r * uz;
        const double x2y2 = x * x + y * y, r1sq = x2y2 + z * z, r2sq = r1sq + 1.0 - 2.0 * x;
        const double i1 = inv_sqrt(r1sq), i2 = inv_sqrt(r2sq);
        const double v = -s.comp * i1 - s.mu * i2;
        const double f = s.primary ? v - s.ssq * x2y2 * 0.5 + s.mu * x : v - s.ssq * (0.5 + 0.5 * x2y2 - x) - s.comp * x;
        const double a = s.comp * (i1 * i1 * i1), b = s.mu * (i2 * i2 * i2), w = x - 1.0;
        const double gx = a * x + b * w - (s.primary ? s.ssq * x - s.mu : s.ssq * w - s.mu + 1.0);
        slope = gx * ux + (a + b - s.ssq) * y * uy + (a + b) * z * uz;
        dr = (f - s.pref) / slope;
        r = fmin(fmax(r - dr, 0.2 * s.rref), s.rref);
    }
    // quadratic: a last step below 1e-9 leaves far less than tol; the potential's rounding is ~1e-15
    // of its size (1/r of either star), in radius that over the slope
    const bool ok = fabs(dr) <= 1e-9 && slope > 1e-2;
    return FaceRoot{r, ok ? 1e-12 + 1e-13 * fmax(1.0, fabs(s.pref)) / slope : (double)INFINITY};
}

// x^(1/4): two square roots, a fifth of pow's FP64 instructions.
__device__ __forceinline__ double fourth_root(double x) { return sqrt(sqrt(x)); }

// The interval that bisecting (r, 2 r] down to a width <= acc ends with when every step is decided by
// the root, as its middle; 0 where a step would come within `tol` of it, or the steps are too many to
// count by exponents.  Every mid-point is a multiple of the last width from r, and the two nearest to
// the root are that interval's ends.  In place of ~27 steps of a serial add, halve and compare: with the
// fourth roots, k_elements of 1024 models 16.1 -> 14.5 ms.
__device__ __forceinline__ double bisected(const FaceRoot& root, double r, double acc) {
    const double x = r / acc;  // the first width is r
    if (!(x > 1.0 && x < 1e12 && root.r > r && root.r < 2.0 * r)) return 0.0;
    const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
    const double up = __hiloint2double((1023 + e) << 20, 0), steps = up < x ? 2.0 * up : up;  // 2^n >= x
    const double h = r / steps, t = (root.r - r) / h, j = floor(t);
    return (t - j) * h > root.tol && (j + 1.0 - t) * h > root.tol ? fma(j + 0.5, h, r) : 0.0;
}

// Irradiated temperature (brightness.rs:150-174) -> temp, geom.
__device__ __forceinline__ double irradiate(double tbase, double gravity, double gdcbol, double absorb, double tirr,
                                            double mu, double r, double rirr, double& geom) {
    double tg = gravity == 1.0 ? tbase : tbase * pow(gravity, gdcbol);  // 1 on spheres
    double tg4 = sq(tg) * sq(tg), ti4 = sq(tirr) * sq(tirr);
    if (mu >= rirr) {
        geom = sq(rirr / r) * mu;
        return fourth_root(tg4 + absorb * ti4 * geom);
    }
    if (mu > -rirr) {
        double x0 = -mu / rirr;
        geom = sq(rirr / r) * rirr * (sqrt(1.0 - x0 * x0) * (2.0 + x0 * x0) / 3.0 - x0 * (kPi / 2.0 - asin(x0))) / kPi;
        return fourth_root(tg4 + absorb * ti4 * geom);
    }
    geom = 0.0;
    return tg;
}

__device__ __forceinline__ double ang_dist(double px, double py, double pz, const SpotDev& s, double len) {
    if (len <= 0.0) return 180.0;  // brightness.rs:177-183
    double c = fmin(fmax((px * s.dx + py * s.dy + pz * s.dz) / len, -1.0), 1.0);
    return rad2deg(acos(c));
}

// LDC::imu in FP64 (types.rs:101-119)
__device__ __forceinline__ double imu_d(const double* l, int ltype, double mu) {
    if (mu <= 0.0) return 0.0;
    mu = fmin(mu, 1.0);
    double om = 1.0 - mu, im = 1.0;
    if (ltype == 0) {
        im -= om * (l[0] + om * (l[1] + om * (l[2] + om * l[3])));
    } else {
        im -= l[0] + l[1] + l[2] + l[3];
        double ms = sqrt(mu);
        im += ms * (l[0] + ms * (l[1] + ms * (l[2] + ms * l[3])));
    }
    return im;
}

__device__ __forceinline__ double lens_mag_d(double sx, double sy, double sz, double ex, double ey, double ez,
                                             double rl) {  // flux.rs:390-406
    double d = -(sx * ex + sy * ey + sz * ez);
    if (d <= 0.0) return 1.0;
    double ax = sx + d * ex, ay = sy + d * ey, az = sz + d * ez;
    double p = sqrt(ax * ax + ay * ay + az * az), ph = p / 2.0, phsq = ph * ph, rd = rl * d;
    double pd = phsq > 25.0 * rd ? p + rd / p : ph + sqrt(phsq + rd);
    return pd * pd / (pd - ph) / ph / 4.0;
}

// ---------------------------------------------------------------------------
// k_elements: grid, continuum, analytic eclipses
// ---------------------------------------------------------------------------
// Eclipse pair slots per element: star elements use slot 0 for the eclipse by
// the other star and slots 1-2 for the opaque disc; disc, rim and spot
// elements use slots 0-1 for the disc, 2 for star 1 and 3 for star 2.  A
// Roche-distorted eclipser leaves its slot empty here for k_roche to fill.
__device__ __forceinline__ int roche_slot(int kind, int by) {
    return (kind == SEG_STAR1 || kind == SEG_STAR2) ? 0 : (by == 1 ? 2 : 3);
}

__global__ void __launch_bounds__(kElemThreads) k_elements(ElemArgs A) {
    const ElemBlock blk = A.blocks[blockIdx.x];
    const SegDesc sg = A.segs[blk.seg];
    const ModelDev& M = A.models[sg.model];
    const int64_t i = blk.offset + threadIdx.x;
    if (i >= sg.count) return;

    double px = 0, py = 0, pz = 0, dx = 0, dy = 0, dz = 1;
    float area = 0.f, grav = 1.f, flux = 0.f;
    double2 ecl[kMaxEcl];
    for (int k = 0; k < kMaxEcl; ++k) ecl[k] = make_double2(INFINITY, -INFINITY);

    // analytic eclipse by a spherical star (grid.rs:49-73); Roche stars go to k_roche
    auto sphere_ecl = [&](int by, int slot) {
        if (by == 1 ? M.roche1 : M.roche2) return;
        double a, b, l1, l2;
        if (sphere_phase(M.cosi_e, M.sini_e, px, py, pz, by == 1 ? 0.0 : 1.0, by == 1 ? M.r1 : M.r2, a, b, l1, l2))
            ecl[slot] = make_double2(a, b);
    };
    auto disc_ecl = [&](double rdisc1, int slot) {
        double a[2], b[2];
        int n = disc_eclipse(M, rdisc1, px, py, pz, a, b);
        for (int k = 0; k < n; ++k) ecl[slot + k] = make_double2(a[k], b[k]);
    };

    if (sg.kind == SEG_STAR1 || sg.kind == SEG_STAR2) {
        const bool primary = sg.kind == SEG_STAR1;
        // band of element i (grid.rs:227-262)
        int lo = 0, hi = sg.ntable - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (A.bands[sg.table + mid].first <= i) lo = mid; else hi = mid - 1;
        }
        if (!LCB_IN_BOUNDS(sg.table + lo < A.sz.nbands && sg.first + i < A.sz.nelem, A.status + sg.model)) return;
        const Band b = A.bands[sg.table + lo];
        const int64_t np = i - b.first;
        double phi = b.phi1 + (b.phi2 - b.phi1) * ((double)np + 0.5) / (double)b.nphi;
        double sinp, cosp;
        sincos(phi, &sinp, &cosp);
        double ux, uy, uz;
        if (M.npole) { ux = b.sint * cosp; uy = b.sint * sinp; uz = b.cost; }
        else { ux = b.cost; uy = b.sint * cosp; uz = b.sint * sinp; }
        const bool roche = primary ? M.roche1 : M.roche2;
        const double cofm = primary ? 0.0 : 1.0;
        double rad, g;
        if (roche) {  // face (surface.rs:54-121)
            const double ssq = primary ? sq(M.spin1) : sq(M.spin2);
            const double rref = primary ? M.rref1 : M.rref2, pref = primary ? M.pref1 : M.pref2;
            const FaceRoot root = face_root(primary ? M.ecl1 : M.ecl2, ux, uy, uz);
            // 1 below the surface, 0 on or above it (potential > pref), -1 equal
            auto side = [&](double r) {
                if (fabs(r - root.r) > root.tol) return r < root.r ? 1 : 0;
                const double t = pot_exact(primary, M.q, ssq, cofm + r * ux, r * uy, r * uz);
                return t < pref ? 1 : t > pref ? 0 : -1;
            };
            double rlo = rref / 2.0, rhi = rref;
            bool above = true;
            for (int k = 0; k < 30 && above; ++k) {
                rlo = rhi / 2.0;
                above = side(rlo) == 0;
                if (above) rhi = rlo;
            }
            rad = bisected(root, rlo, M.acc_face);
            if (rad == 0.0) {
                for (int k = 0; k < 100 && rhi - rlo > M.acc_face; ++k) {
                    double mid = (rlo + rhi) / 2.0;
                    if (side(mid) == 1) rlo = mid;
                    else rhi = mid;
                }
                rad = (rlo + rhi) / 2.0;
            }
            px = cofm + rad * ux; py = rad * uy; pz = rad * uz;
            double gx, gy, gz;
            dpot_exact(primary, M.q, ssq, px, py, pz, gx, gy, gz);
            double n2 = gx * gx + gy * gy + gz * gz;
            g = sqrt(n2);
            if (n2 > 0.0) { dx = gx / g; dy = gy / g; dz = gz / g; }
            else { dx = gx; dy = gy; dz = gz; }
        } else {
            rad = primary ? M.r1 : M.r2;
            px = cofm + rad * ux; py = rad * uy; pz = rad * uz;
            dx = ux; dy = uy; dz = uz;
            g = 1.0;
        }
        area = (float)(((b.aphi * rad) * b.sint) * (b.ath * rad) / (ux * dx + uy * dy + uz * dz));
        grav = (float)(g / (primary ? M.gref1 : M.gref2));
        if (primary ? M.eclipse1 : M.eclipse2) sphere_ecl(primary ? 2 : 1, 0);
        if (M.add_disc && M.opaque) disc_ecl(M.rdisc1_l, 1);  // orchestration.rs:145-157
        // continuum (brightness.rs:49-144)
        const double cx = primary ? 1.0 : 0.0;
        double vx = cx - px, vy = -py, vz = -pz;
        double r = sqrt(vx * vx + vy * vy + vz * vz);
        double mu = (dx * vx + dy * vy + dz * vz) / r;
        double geom, temp;
        if (primary) {
            double t1 = M.t1, plen = sqrt(px * px + py * py + pz * pz);
            for (int k = 0; k < 3; ++k) {
                const SpotDev& s = M.spot1[k];
                if (!s.on) continue;
                double dist = ang_dist(px, py, pz, s, plen);
                t1 += (s.tcen - M.t1) * exp(-sq(dist / (s.fwhm / kFwhmEfac)) / 2.0);
            }
            if (M.uesp_on) {
                double el = sqrt(px * px + py * py);
                if (el > 0.0) {
                    double clat = fmin(fmax((px * px + py * py) / el / plen, -1.0), 1.0);
                    double dlat = rad2deg(acos(clat));
                    double clong = fmin(fmax((M.uesp_dx * px + M.uesp_dy * py) / el, -1.0), 1.0);
                    double dlong = rad2deg(acos(clong));
                    double hw = M.uesp_lathw, lw = M.uesp_longhw, tp = M.uesp_taper, ut = M.uesp_temp;
                    if (dlat <= hw && dlong <= lw) t1 = ut;
                    else if (dlat <= hw) t1 += (ut - M.t1) * exp(-(dlong - lw) / tp);
                    else if (dlong <= lw) t1 += (ut - M.t1) * exp(-(dlat - hw) / tp);
                    else t1 += (ut - M.t1) * exp(-(dlat - hw) / tp) * exp(-(dlong - lw) / tp);
                }
            }
            temp = irradiate(t1, (double)grav, M.gdcbol1, M.absorb, M.t2, mu, r, M.r2c, geom);
            flux = (float)((double)area * planck_d(M.wavelength, temp));
            if (M.mirror) flux += (float)((double)area * geom * M.planck_t2abs);
        } else {
            double t2 = fabs(M.t2);
            for (int k = 0; k < 2; ++k) {
                const SpotDev& s = M.spot2[k];
                if (!s.on) continue;
                double ox = px - 1.0, oy = py, oz = pz;
                double dist = ang_dist(ox, oy, oz, s, sqrt(ox * ox + oy * oy + oz * oz));
                t2 += (s.tcen - t2) * exp(-sq(dist / (s.fwhm / kFwhmEfac)) / 2.0);
            }
            temp = irradiate(t2, (double)grav, M.gdcbol2, M.absorb, M.t1, mu, r, M.r1c, geom);
            flux = (float)((double)area * planck_d(M.wavelength, temp));
            if (M.mirror) flux += (float)((double)area * geom * M.planck_t1);
        }
    } else if (sg.kind == SEG_DISC) {  // grid.rs:356-390, brightness.rs:204-212
        int lo = 0, hi = sg.ntable - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (A.rings[sg.table + mid].first <= i) lo = mid; else hi = mid - 1;
        }
        if (!LCB_IN_BOUNDS(sg.table + lo < A.sz.nrings && sg.first + i < A.sz.nelem, A.status + sg.model)) return;
        const Ring g = A.rings[sg.table + lo];
        double th = kTwoPi * (double)(i - g.first) / (double)g.ntheta;
        double st, ct;
        sincos(th, &st, &ct);
        px = g.rad * ct; py = g.rad * st; pz = g.h;
        dx = -ct * g.sinp; dy = -st * g.sinp; dz = g.cosp;
        area = (float)g.area;
        if (M.opaque) disc_ecl(M.rdisc1_g, 0);
        if (M.eclipse1) sphere_ecl(1, 2);
        if (M.eclipse2) sphere_ecl(2, 3);
        double r = sqrt(px * px + py * py + pz * pz);
        flux = (float)(M.disc_bright * pow(r / M.rdisc2, M.texp_disc) * (double)area);
    } else if (sg.kind == SEG_EDGE) {  // grid.rs:411-478, brightness.rs:215-239
        const int64_t col = i / M.edge_nout, row = i - col * M.edge_nout;
        double th = kTwoPi * (double)col / (double)M.edge_ntheta;
        double st, ct;
        sincos(th, &st, &ct);
        const double rv = M.edge_rad, h = M.edge_h;
        if (row == 0) {
            px = kEfac * rv * ct; py = kEfac * rv * st; pz = kEfac * h;
            area = (float)(M.edge_area / 2.0);
        } else {
            pz = -h + 2.0 * h * (double)(row - 1) / (double)(M.edge_nout - 1);
            px = kEfac * rv * ct; py = kEfac * rv * st;
            area = (float)M.edge_area;
        }
        dx = ct; dy = st; dz = 0.0;
        if (M.opaque) disc_ecl(M.rdisc1_g, 0);
        if (M.eclipse1) sphere_ecl(1, 2);
        if (M.eclipse2) sphere_ecl(2, 3);
        double vx = 1.0 - px, vy = -py, vz = -pz;
        double r = sqrt(vx * vx + vy * vy + vz * vz);
        double mu = (dx * vx + dy * vy + dz * vz) / r;
        double temp, r2 = M.r2e, t4 = sq(M.tedge) * sq(M.tedge), i4 = sq(M.t2abs) * sq(M.t2abs);
        if (mu >= r2) {
            double geom = sq(r2 / r) * mu;
            temp = fourth_root(t4 + M.absorb_edge * i4 * geom);
        } else if (mu > -r2) {
            double x0 = -mu / r2;
            double geom = sq(r2 / r) * r2 * (sqrt(1.0 - x0 * x0) * (2.0 + x0 * x0) / 3.0 - x0 * (kPi / 2.0 - asin(x0))) / kPi;
            temp = fourth_root(t4 + M.absorb_edge * i4 * geom);
        } else {
            temp = M.tedge;
        }
        flux = (float)((double)area * planck_d(M.wavelength, temp));
    } else {  // SEG_SPOT: grid.rs:520-550
        const int64_t k = i >> 1;
        const bool tilted = (i & 1) == 0;
        double dist = M.sfac_spot * (double)k / (double)(M.nspot - 1);
        double f = M.length_spot * (dist - M.bmax);
        px = M.bspot[0] + f * M.bvec[0]; py = M.bspot[1] + f * M.bvec[1]; pz = M.bspot[2] + f * M.bvec[2];
        if (M.eclipse1) sphere_ecl(1, 2);
        if (M.eclipse2) sphere_ecl(2, 3);
        double bright = M.bright_ref * pow(dist / M.bmax, M.expon_spot) *
                        exp(M.expon_spot / M.epow_spot - pow(dist, M.epow_spot));
        area = (float)M.area_spot;
        if (tilted) { dx = M.tvec[0]; dy = M.tvec[1]; dz = M.tvec[2]; flux = (float)(bright * (1.0 - M.cfrac_spot) * M.area_spot); }
        else { dx = 0.0; dy = 0.0; dz = 1.0; flux = (float)(bright * M.cfrac_spot * M.area_spot); }
    }
    const int64_t e = sg.first + i;
    if (!LCB_IN_BOUNDS(e < A.sz.nelem, A.status + sg.model)) return;
    A.el_rec[e] = make_float4((float)dx, (float)dy, (float)dz, flux);
    A.el_pos[e] = make_float4((float)px, (float)py, (float)pz, 0.f);
    A.el_p64[e] = make_double4(px, py, pz, (double)area);
    A.el_d64[e] = make_double4(dx, dy, dz, (double)grav);
    unsigned used = 0;
    for (int k = 0; k < kMaxEcl; ++k) {
        A.el_ecl[k * A.sz.nelem + e] = ecl[k];
        if (ecl[k].x <= 2.0) used |= 1u << k;
    }
    if (used) atomicOr(A.ecl_grp + e / kEclGroup, used);
}

// ---------------------------------------------------------------------------
// k_roche: eclipses by a Roche star (eclipse.rs:270-373), two threads an element
// ---------------------------------------------------------------------------
__device__ __forceinline__ void roche_counters(const ElemArgs& A, const EclCount& cnt);

// ORs each lane's slot bits into its element group's used-slot word with one
// atomic per distinct word of the warp (lanes hold consecutive elements, so a
// warp spans one or two words).  All 32 lanes call it; g < 0 or bits == 0: none.
__device__ __forceinline__ void group_or_warp(unsigned* grp, int64_t g, unsigned bits) {
    const bool mine = bits != 0u && g >= 0;
    unsigned pending = __ballot_sync(0xffffffffu, mine);
    while (pending) {
        const int src = __ffs(pending) - 1;
        const int64_t gs = __shfl_sync(0xffffffffu, g, src);
        const bool same = mine && g == gs;
        const unsigned all = __reduce_or_sync(0xffffffffu, same ? bits : 0u);
        if ((int)(threadIdx.x & 31) == src) atomicOr(grp + gs, all);
        pending &= ~__ballot_sync(0xffffffffu, same);
    }
}

// Eclipses by Roche-distorted stars through their limb contacts (lcb_roche.h):
// two adjacent lanes per element, one for the ingress and one for the egress,
// each with its own Newton iteration and bisection; block b covers half of
// Roche block b / 2.  Elements the limb path leaves open (stars that are not
// convex, elements near the bounding sphere, grazes narrower than the margins)
// go to a list that k_roche_open and k_roche_chop2 take.  Bound by FP64 latency
// and issue: ~12 contact nodes and ~6 searches an element of ~10 evaluations.
// 43 million elements (1024 models): 200 -> 50.6 ms, 92 evaluations an element
// instead of ~850; one model of 5,000 elements: 0.267 -> 0.064 ms.
__global__ void __launch_bounds__(kRocheBlock, kRocheMinBlocks) k_roche(ElemArgs A) {
    const int64_t rb = blockIdx.x >> 1;
    const int slot = (int)(blockIdx.x & 1) * (kRocheBlock / 2) + (int)(threadIdx.x >> 1);
    const bool egress = threadIdx.x & 1;
    const ElemBlock blk = A.rblocks[rb];
    const SegDesc sg = A.segs[blk.seg];
    const int64_t i = blk.offset + slot, e = sg.first + i;
    EclCount cnt, scan;  // scan: what both lanes of a pair do alike, counted by the first
    cnt.cap = scan.cap = A.fblink_cap;
    bool capped = false, open = false, hidden = false;
    const bool valid = i < sg.count && LCB_IN_BOUNDS(e < A.sz.nelem, A.status + sg.model);
    const ModelDev& M = A.models[sg.model];
    const RocheEcl& R = blk.by == 1 ? M.ecl1 : M.ecl2;
    Geom G;
    Limb L;
    bool found = false, seek = false;  // both contacts known; guesses in c.phi to try
    Contact c{0.0, 0.0, false};
    bool crosses = false;  // the bounding sphere, at some phase
    if (!R.convex || (R.wide && sg.kind != SEG_STAR1 && sg.kind != SEG_STAR2)) {
        open = true;  // the whole block, so that the list keeps its order and alignment
    } else if (valid) {
        const double4 p = A.el_p64[e];
        crosses = geom_setup(R, M.cosi_e, M.sini_e, M.delta, p.x, p.y, p.z, G);
        open = crosses && !limb_applies(R, G);
        double half;
        if (crosses && !open) {
            seek = limb_guess(R, G, half);
            c.phi = 0.5 * (G.sc.phi1 + G.sc.phi2) + (egress ? half : -half);
        }
    }
    for (int attempt = 0; attempt < 2; ++attempt) {  // from the ellipsoid, then from the lowest potential
        c.ok = false;
        if (seek) c = limb_contact(R, G, egress, c.phi, cnt);
        Contact o;  // the pair's other contact
        o.phi = __shfl_xor_sync(0xffffffffu, c.phi, 1);
        o.margin = __shfl_xor_sync(0xffffffffu, c.margin, 1);
        o.ok = __shfl_xor_sync(0xffffffffu, (int)c.ok, 1) != 0;
        if (seek) found = limb_make(egress ? o : c, egress ? c : o, L);
        const bool lost = crosses && !open && !found;
        if (attempt) {
            if (seek && !found) open = true;
            break;
        }
        seek = false;
        if (lost) {
            double lo, hi;
            const int st = limb_lowest(R, G, lo, hi, scan);
            if (st == LIMB_NONE) {
                scan.fbl += G.sc.nsteps + 1;
                ++scan.skipped;
            }
            open = st == LIMB_OPEN;
            seek = st == LIMB_ECLIPSED;
            c.phi = egress ? hi : lo;
        }
        if (!__any_sync(0xffffffffu, seek)) break;
    }
    double r = 0.0;
    if (found) {
        const int hit = limb_scan(R, G, L, capped, scan);
        if (!capped && hit >= 0) {
            r = limb_chop(R, G, L, egress, G.sc.phi1 + (double)hit * G.sc.dphi, M.delta, capped, cnt);
            hidden = !capped;
        }
    }
    const double eg = __shfl_xor_sync(0xffffffffu, r, 1);
    const bool hidden2 = __shfl_xor_sync(0xffffffffu, (int)hidden, 1) != 0 && hidden;
    int64_t grp = -1;
    unsigned bits = 0u;
    if (capped) atomicOr(A.status + sg.model, kStatusIterCap);
    if (!egress && hidden2) {
        const int slot = roche_slot(sg.kind, blk.by);
        A.el_ecl[slot * A.sz.nelem + e] = make_double2(r, eg < r ? eg + 1.0 : eg);
        grp = e / kEclGroup;
        bits = 1u << slot;
    }
    group_or_warp(A.ecl_grp, grp, bits);
    // open elements to the list, a block's in their order (neighbours search alike: fragments of a warp's
    // 16 cost k_roche_open a fifth)
    const unsigned mine = __ballot_sync(0xffffffffu, open && !egress);
    if (__syncthreads_or(mine != 0u)) {
        __shared__ unsigned found_open[kRocheBlock / 32], list_at;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane == 0) found_open[warp] = (unsigned)__popc(mine);
        __syncthreads();
        unsigned before = 0, total = 0;
        for (int w = 0; w < kRocheBlock / 32; ++w) {
            if (w < warp) before += found_open[w];
            total += found_open[w];
        }
        if (threadIdx.x == 0) list_at = atomicAdd(A.nopen, total);
        __syncthreads();
        if ((mine >> lane) & 1u) {
            const unsigned k = list_at + before + __popc(mine & ((1u << lane) - 1u));
            A.open[k] = (unsigned)(rb * kRocheBlock + slot);
            if (k < A.nfirst) A.firsthit[k] = kNoHit;
        }
    }
    if (!egress) {
        cnt.pot += scan.pot; cnt.dpot += scan.dpot; cnt.fbl += scan.fbl; cnt.cert += scan.cert; cnt.skipped += scan.skipped;
    }
    roche_counters(A, cnt);
}

// Threads per open element in the split phase scan: a power of two up to 16,
// until about sixteen waves of scan threads fill the GPU (the choices an
// autotuning of 8..128-model batches made); 1: whole searches, one thread
// each, where the scan proves blocks of steps at once.
__device__ __forceinline__ int open_split(const ElemArgs& A, unsigned n) {
    if (A.split_fix > 0) return n <= A.nfirst ? A.split_fix : 1;
    const unsigned threads = (n + kRocheBlock - 1) / kRocheBlock * kRocheBlock;
    int split = 1;
    while (split < 16 && (int64_t)(2 * split) * threads <= A.split_target) split *= 2;
    return n <= A.nfirst ? split : 1;
}

struct OpenElem {
    const ModelDev* M;
    const RocheEcl* R;
    int64_t e;
    int model, slot;
    bool valid;
};
__device__ __forceinline__ OpenElem open_elem(const ElemArgs& A, unsigned item) {
    const ElemBlock blk = A.rblocks[item / kRocheBlock];
    const SegDesc sg = A.segs[blk.seg];
    OpenElem o;
    o.M = A.models + sg.model;
    o.R = blk.by == 1 ? &o.M->ecl1 : &o.M->ecl2;
    const int64_t i = blk.offset + item % kRocheBlock;
    o.e = sg.first + i;
    o.model = sg.model;
    o.slot = roche_slot(sg.kind, blk.by);
    o.valid = i < sg.count && LCB_IN_BOUNDS(o.e < A.sz.nelem, A.status + sg.model);
    return o;
}

// One chunk of a split phase scan: scan indices [c L, (c+1) L) of 0 .. nsteps,
// L = ceil((nsteps+1)/K); the first hit is merged into *first with atomicMin,
// and a chunk stops once an earlier chunk has hit.  The minimum over chunks is
// the single scan's first hit, so the decision is the reference's.
__device__ void scan_chunk(const RocheEcl& s, double cosi, double sini, double delta, double px, double py,
                           double pz, int chunk, int split, int* first, bool& capped, EclCount& evals) {
    Scan sc;
    if (!scan_setup(s, cosi, sini, delta, px, py, pz, sc)) return;
    const int total = sc.nsteps + 1, len = (total + split - 1) / split;
    const int lo = chunk * len, hi = min(total, lo + len);
    Los L{px, py, pz, 0.0, 0.0, 0.0};
    for (int i = lo; i < hi; ++i) {
        if (((i - lo) & 7) == 0 && *(volatile int*)first < lo) return;
        earth_at(cosi, sini, sc.phi1 + (double)i * sc.dphi, L.ex, L.ey, L.ez);
        const bool hit = fblink(s, sc.acc, L, evals, capped, kCertBudget);
        if (capped) return;
        if (hit) {
            atomicMin(first, i);
            return;
        }
    }
}

__device__ __forceinline__ void roche_counters(const ElemArgs& A, const EclCount& cnt) {
    if (!A.counters) return;  // eclipse-search work counters, one atomic per warp and counter
    unsigned long long v[5] = {(unsigned long long)cnt.pot, (unsigned long long)cnt.dpot, (unsigned long long)cnt.fbl,
                               (unsigned long long)cnt.cert, (unsigned long long)cnt.skipped};
    for (int k = 0; k < 5; ++k) {
        unsigned long long x = v[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(A.counters + k, x);
    }
}

// The warp's next group of open elements: searches differ in length many times
// over, so that warps take them as they come.  (Strides instead gave a block the
// same chunk of every scan it took, the grid being a multiple of `split`: 64
// models of stars that are not convex 4.1 instead of 1.4 ms, 512 9.7 instead of 8.2.)
__device__ __forceinline__ unsigned next_group(unsigned* counter) {
    unsigned w = 0;
    if ((threadIdx.x & 31) == 0) w = atomicAdd(counter, 1u);
    return __shfl_sync(0xffffffffu, w, 0);
}

// The general search of the open elements: persistent warps over the list.
// Unsplit, one thread runs an element's whole search (phase scan with block
// proofs, then both bisections).  Split, the scans' chunks are spread over
// `split` threads an element and k_roche_chop2 bisects from the first hit: the
// time of a short list is otherwise its longest single scan.  Every element's
// first chunk comes before any second one: like work lies together, and a chunk
// finds the hits of those before it (eight models: 0.24 -> 0.21 ms).  kSplit: the batch is
// small enough that its lists always split (the whole search is not compiled in).
template <bool kSplit>
__global__ void __launch_bounds__(kRocheBlock, kScanMinBlocks) k_roche_open(ElemArgs A) {
    const unsigned n = *A.nopen;
    if (n == 0) return;
    const int split = open_split(A, n);
    const unsigned lists = (n + 31) / 32, groups = lists * split;
    EclCount cnt;
    cnt.cap = A.fblink_cap;
    for (unsigned w; (w = next_group(A.nopen + 1)) < groups;) {
        const unsigned chunk = w / lists, k = (w - chunk * lists) * 32 + (threadIdx.x & 31);
        int64_t g = -1;
        unsigned bits = 0u;
        if (k < n) {
            const OpenElem o = open_elem(A, A.open[k]);
            bool capped = false;
            if (o.valid) {
                const double4 p = A.el_p64[o.e];
                if (!kSplit && split == 1) {
                    double a, b;
                    if (ingress_egress<true>(*o.R, o.M->cosi_e, o.M->sini_e, o.M->delta, p.x, p.y, p.z, a, b, capped, cnt)) {
                        A.el_ecl[o.slot * A.sz.nelem + o.e] = make_double2(a, b);
                        g = o.e / kEclGroup;
                        bits = 1u << o.slot;
                    }
                } else {
                    const int fbl = cnt.fbl;  // k_roche_chop2 counts the reference's scan searches
                    scan_chunk(*o.R, o.M->cosi_e, o.M->sini_e, o.M->delta, p.x, p.y, p.z, (int)chunk, split,
                               A.firsthit + k, capped, cnt);
                    cnt.fbl = fbl;
                }
                if (capped) atomicOr(A.status + o.model, kStatusIterCap);
            }
        }
        if (!kSplit && split == 1) group_or_warp(A.ecl_grp, g, bits);
    }
    roche_counters(A, cnt);
}

// Split scan, second kernel with two threads per element: adjacent lanes run
// the ingress and the egress bisection of one element at once (each from the
// first hit, eclipse.rs:301-332), halving the longest chain of line-of-sight
// searches; the ingress lane combines the pair.
__global__ void __launch_bounds__(kRocheBlock, kChopMinBlocks) k_roche_chop2(ElemArgs A) {
    const unsigned n = *A.nopen;
    if (n == 0 || open_split(A, n) == 1) return;
    const int part = threadIdx.x & 1;  // 0: ingress, 1: egress
    EclCount cnt;
    cnt.cap = A.fblink_cap;
    for (unsigned w; (w = next_group(A.nopen + 2)) < (n + 15) / 16;) {
        const unsigned k = w * 16 + ((threadIdx.x & 31) >> 1);
        bool capped = false, found = false;
        double a = 0.0, b = 0.0;
        OpenElem o;
        o.valid = false;
        if (k < n) {
            o = open_elem(A, A.open[k]);
            if (o.valid) {
                const double4 p = A.el_p64[o.e];
                const int first = A.firsthit[k];
                Scan sc;
                if (part == 0 && scan_setup(*o.R, o.M->cosi_e, o.M->sini_e, o.M->delta, p.x, p.y, p.z, sc))
                    cnt.fbl += first == kNoHit ? sc.nsteps + 1 : first + 1;  // the single scan's searches
                found = ingress_egress<false>(*o.R, o.M->cosi_e, o.M->sini_e, o.M->delta, p.x, p.y, p.z, a, b, capped, cnt,
                                              first, part + 1);
            }
        }
        const double egress = __shfl_xor_sync(0xffffffffu, b, 1);
        const bool found_eg = __shfl_xor_sync(0xffffffffu, (int)found, 1) != 0;
        const bool capped_eg = __shfl_xor_sync(0xffffffffu, (int)capped, 1) != 0;
        int64_t g = -1;
        unsigned bits = 0u;
        if (o.valid && part == 0) {
            if (found && found_eg) {
                A.el_ecl[o.slot * A.sz.nelem + o.e] = make_double2(a, egress < a ? egress + 1.0 : egress);
                g = o.e / kEclGroup;
                bits = 1u << o.slot;
            }
            if (capped || capped_eg) atomicOr(A.status + o.model, kStatusIterCap);
        }
        group_or_warp(A.ecl_grp, g, bits);
    }
    roche_counters(A, cnt);
}

// ---------------------------------------------------------------------------
// k_aux: per-model FP64 sums over the star grids -- comp_star1/2 at the ginterp
// and wdwarf phases (flux.rs:115-206), log g (flux.rs:288-322), radii (347-373)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kElemThreads) k_aux(ElemArgs A) {
    const ElemBlock blk = A.ablocks[blockIdx.x];
    const SegDesc sg = A.segs[blk.seg];
    const ModelDev& M = A.models[sg.model];
    const int64_t i = blk.offset + threadIdx.x;
    const bool valid = i < sg.count && LCB_IN_BOUNDS(sg.first + i < A.sz.nelem, A.status + sg.model);
    const int star = sg.kind == SEG_STAR1 ? 1 : 2;
    double px = 0, py = 0, pz = 0, dx = 0, dy = 0, dz = 0, area = 0, grav = 0, flux = 0;
    double2 ecl[kMaxEcl];
    if (valid) {
        const int64_t e = sg.first + i;
        double4 p = A.el_p64[e], d = A.el_d64[e];
        px = p.x; py = p.y; pz = p.z; area = p.w;
        dx = d.x; dy = d.y; dz = d.z; grav = d.w;
        flux = (double)A.el_rec[e].w;
        for (int k = 0; k < kMaxEcl; ++k) ecl[k] = A.el_ecl[k * A.sz.nelem + e];
    }
    double vals[16];
    int slot[16];
    int nv = 0;
    for (int s = 0; s < M.nspec; ++s) {
        const SpecPhase& sp = M.spec[s];
        if (sp.star != star) continue;
        bool match = sg.role == ROLE_BOTH || (sg.role == ROLE_FINE) == (sp.fine != 0);
        if (!match) continue;
        double c = 0.0;
        if (valid) {
            // the ginterp sums run before the opaque-disc pairs exist (orchestration.rs:93-157)
            const int ne = sp.star_ecl_only ? 1 : kMaxEcl;
            bool vis = true;
            for (int k = 0; k < ne; ++k)
                if ((sp.phi >= ecl[k].x && sp.phi <= ecl[k].y) || sp.phi <= ecl[k].y - 1.0) vis = false;
            double mu = sp.ex * dx + sp.ey * dy + sp.ez * dz;
            const double* ld = star == 1 ? M.ld1 : M.ld2;
            int lt = star == 1 ? M.ltype1 : M.ltype2;
            double beam = star == 1 ? M.beam1 : M.beam2;
            if (vis && mu > (star == 1 ? M.mucrit1 : M.mucrit2)) {
                double mag = (star == 2 && M.glens1) ? lens_mag_d(px, py, pz, sp.ex, sp.ey, sp.ez, M.rlens1) : 1.0;
                if (beam != 0.0) {
                    double vxx = -M.vfac * py, vyy = M.vfac * (px - M.xcofm);
                    double vr = -(sp.ex * vxx + sp.ey * vyy), vn = dx * vxx + dy * vyy;
                    double mud = mu - mu * vr - vn;
                    c = mu * mag * flux * (1.0 - beam * vr) * imu_d(ld, lt, mud);
                } else {
                    c = mu * mag * flux * imu_d(ld, lt, mu);
                }
            }
        }
        vals[nv] = c;
        slot[nv] = AUX_SPEC0 + s;
        ++nv;
    }
    if (sg.fine_star) {
        double sa = 0.0, vol = 0.0;
        if (valid) {
            double wx = px - (star == 1 ? 0.0 : 1.0), wy = py, wz = pz;
            double r = sqrt(wx * wx + wy * wy + wz * wz);
            double rc = dx * wx + dy * wy + dz * wz;
            sa = area * rc / ((r * r) * r);
            vol = area * rc;
        }
        vals[nv] = flux * grav; slot[nv++] = star == 1 ? AUX_FG1 : AUX_FG2;
        vals[nv] = flux; slot[nv++] = star == 1 ? AUX_F1 : AUX_F2;
        vals[nv] = sa; slot[nv++] = star == 1 ? AUX_SA1 : AUX_SA2;
        vals[nv] = vol; slot[nv++] = star == 1 ? AUX_VOL1 : AUX_VOL2;
    }
    if (nv == 0) return;
    __shared__ double red[16][kElemThreads / 32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < nv; ++k) {
        double v = vals[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[k][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < nv) {
        double t = 0.0;
        for (int w = 0; w < kElemThreads / 32; ++w) t += red[threadIdx.x][w];
        atomicAdd(A.aux + (int64_t)sg.model * kNumAux + slot[threadIdx.x], t);
    }
}

// ---------------------------------------------------------------------------
// k_phase
// ---------------------------------------------------------------------------
__global__ void k_phase(PhaseArgs A) {
    const ModelDev& M = A.models[blockIdx.x];
    if (M.status < 0) return;
    for (int64_t m = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; m < M.ndatum; m += (int64_t)gridDim.y * blockDim.x) {
        const int64_t d = M.datum_begin + m;
        const lcb_datum D = A.data[M.data_begin + m];
        double phase = (D.time - M.t0) / M.period;
        for (int k = 0; k < 4; ++k)
            phase -= (M.t0 + phase * (M.period + M.pdot * phase) - D.time) / (M.period + 2.0 * M.pdot * phase);
        phase += M.deltat / M.period / 2.0 * (cos(2.0 * kPi * phase) - 1.0);
        double expose = D.expose / M.period;
        double frac = (D.time - M.middle) / M.range;
        A.d_slfac[d] = 1.0 + frac * (M.slope + frac * (M.quad + frac * M.cube));
        int64_t j = first_sub(M, A.dsub0, m);
        for (int nd = 0; nd < D.ndiv; ++nd, ++j) {
            double phi = phase, w = 1.0;
            if (D.ndiv != 1) {
                phi = phase + expose * ((double)nd - (double)(D.ndiv - 1) / 2.0) / (double)(D.ndiv - 1);
                w = (nd == 0 || nd == D.ndiv - 1) ? 0.5 : 1.0;
            }
            double sn, cs;
            sincos(kTwoPi * phi, &sn, &cs);
            A.sp_e[j] = make_float4((float)(M.sini_l * cs), (float)(-M.sini_l * sn), (float)M.cosi_l, 0.f);
            double pn = phi - floor(phi);
            A.sp_phi[j] = pn;
            int t = (pn <= M.phase1 || pn >= 1.0 - M.phase1) ? 1
                    : (((pn > M.phase1 && pn < M.phase2) || (pn > 1.0 - M.phase2 && pn < 1.0 - M.phase1)) ? 2 : 3);
            A.sp_type[j] = (int8_t)t;
            A.sp_w[j] = w;
        }
    }
}

// ---------------------------------------------------------------------------
// k_wait_probe: a bounded wait that runs out (no kernel of a light curve waits;
// the surrogate's GEMMs have the same bounded waits of their own)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after `limit` SM clock cycles; on time-out the caller
// records an error status instead of hanging.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit) {
    if (mbar_test(bar, parity)) return true;
    long long t0 = clock64();
    while (!mbar_test(bar, parity)) {
        __nanosleep(64);
        if (clock64() - t0 > limit) return false;
    }
    return true;
}

// The bounded wait on an mbarrier that nothing completes (no copy, no arrival):
// it must give up after `limit` cycles and report kStatusTmaTimeout.
__global__ void k_wait_probe(long long limit, int* status, long long* waited) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const long long t0 = clock64();
    const bool ok = mbar_wait(&bar, 0u, limit);
    const long long t1 = clock64();
    if (threadIdx.x == 0) {
        *status = ok ? 0 : kStatusTmaTimeout;
        *waited = t1 - t0;
    }
}

enum { CLS_VIS = 0, CLS_MIX = 1, CLS_HID = 2 };
constexpr int kFluxWarps = kFluxThreads / 32;
// used-slot words a flux unit spans (units hold at most 16 chunks of elements)
constexpr int kUnitGroups = 16 * kFluxChunk / kEclGroup + 2;

// Range classification of one eclipse pair against [lo, hi] (exact in FP64).
__device__ __forceinline__ int pair_cls(double ing, double eg, double lo, double hi) {
    if ((ing <= lo && hi <= eg) || hi <= eg - 1.0) return CLS_HID;
    if ((hi < ing || lo > eg) && lo > eg - 1.0) return CLS_VIS;
    return CLS_MIX;
}

// The phases of some sub-phases: their range in each half of [0, 1).
struct PhaseRange {
    double lo[2], hi[2];
    __device__ __forceinline__ void clear() {
        lo[0] = lo[1] = 2.0;
        hi[0] = hi[1] = -1.0;
    }
    // class of an element from its pairs' classes in the two halves (an empty half says nothing)
    __device__ __forceinline__ int join(const int* cls) const {
        const bool a = lo[0] <= hi[0], b = lo[1] <= hi[1];
        if (a && b) return cls[0] == cls[1] ? cls[0] : CLS_MIX;
        return a ? cls[0] : b ? cls[1] : CLS_HID;
    }
    __device__ __forceinline__ void add(int* cls, double2 p) const {
        for (int h = 0; h < 2; ++h) cls[h] = max(cls[h], pair_cls(p.x, p.y, lo[h], hi[h]));
    }
    __device__ __forceinline__ void put(double p) {
        const int h = p >= 0.5 ? 1 : 0;
        lo[h] = fmin(lo[h], p);
        hi[h] = fmax(hi[h], p);
    }
    __device__ __forceinline__ void join_range(const PhaseRange& r) {
        for (int h = 0; h < 2; ++h) {
            lo[h] = fmin(lo[h], r.lo[h]);
            hi[h] = fmax(hi[h], r.hi[h]);
        }
    }
    // over the warp: doubles >= 0 are ordered as their bits, reduced a word at a time
    __device__ __forceinline__ void warp_all() {
        for (int h = 0; h < 2; ++h) {
            const unsigned lh = __double2hiint(lo[h]), ll = __double2loint(lo[h]);
            const unsigned mh = __reduce_min_sync(0xffffffffu, lh);
            const unsigned ml = __reduce_min_sync(0xffffffffu, lh == mh ? ll : ~0u);
            const bool none = hi[h] < 0.0;
            const unsigned hh = none ? 0u : (unsigned)__double2hiint(hi[h]), hl = none ? 0u : (unsigned)__double2loint(hi[h]);
            const unsigned xh = __reduce_max_sync(0xffffffffu, hh);
            const unsigned xl = __reduce_max_sync(0xffffffffu, hh == xh ? hl : 0u);
            lo[h] = __hiloint2double((int)mh, (int)ml);
            hi[h] = lo[h] > 1.0 ? -1.0 : __hiloint2double((int)xh, (int)xl);
        }
    }
};

constexpr int kUnitLists = 16 * kFluxChunk / 32;  // groups of 32 elements of a unit
constexpr int kQuarters = kFluxThreads / 32;      // a tile's sub-phases, a warp's worth each

struct FluxWarpSmem {
    float4 rec[32];               // the warp's current 32 elements
    double2 pair[kMaxEcl][32];    // and the pairs of the mixed ones
    double ph[32 * kFluxR];       // the phases of its current quarter
};
struct FluxUnitSmem {             // a unit, sorted (flux_sort)
    PhaseRange own[kQuarters];    // of each quarter's sub-phases
    float2 trig[4 + 2 * kQuarters];  // (sin, cos) of the ends of the tile's and the quarters' arcs
    unsigned gw[kUnitGroups];     // the unit's words of used-slot masks (ecl_grp)
    unsigned list[kUnitLists];    // per 32 elements: those on the tile's list
    unsigned used[kUnitLists][kQuarters], plain[kUnitLists][kQuarters], mixed[kUnitLists][kQuarters];
    int unit;
};
static_assert(kFluxChunk % 32 == 0, "a chunk is whole groups of 32 elements");


// The earth vector of phase theta/2pi is (sini cos t, -sini sin t, cosi), so an
// element's mu over a phase arc is A cos t + B sin t + C.  The tile's active
// sub-phases lie on (at most) two arcs shorter than pi, one per half of [0, 1).
struct Arcs {
    float ca[2], sa[2], cb[2], sb[2];
    bool on[2];
};
// An element's mu over phases: A cos t + B sin t + C, amplitude R (a few ulp are
// far inside the margins).
struct MuCurve {
    float A, B, C, R;
    __device__ __forceinline__ MuCurve(float si, float ci, const float4& d) : A(si * d.x), B(-si * d.y), C(ci * d.z) {
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(R) : "f"(A * A + B * B));
    }
};
// Largest mu over the arcs (FP32; the caller keeps a margin).
__device__ __forceinline__ float max_mu(const Arcs& a, const MuCurve& u) {
    float m = -2.f;
    for (int h = 0; h < 2; ++h) {
        if (!a.on[h]) continue;
        float in1 = a.ca[h] * u.B - a.sa[h] * u.A, in2 = u.A * a.sb[h] - u.B * a.cb[h];
        float v = (in1 >= 0.f && in2 >= 0.f) ? u.R : fmaxf(u.A * a.ca[h] + u.B * a.sa[h], u.A * a.cb[h] + u.B * a.sb[h]);
        m = fmaxf(m, v + u.C);
    }
    return m;
}
constexpr float kFacingMargin = 2e-5f;  // far above the FP32 rounding of mu

// The single arc (shorter than pi) that a quarter's sub-phases lie on, and an
// element's extreme mu over it.
struct WarpArc {
    float ca, sa, cb, sb;
    // from the ranges in the two halves of [0, 1): the arc's ends; false: none such
    static __device__ __forceinline__ bool ends(const PhaseRange& r, double& from, double& to) {
        const bool a = r.lo[0] <= r.hi[0], b = r.lo[1] <= r.hi[1];
        from = a ? r.lo[0] : r.lo[1];
        to = b ? r.hi[1] : r.hi[0];
        if (a && b && to - from > 0.5) {  // through 0 instead of 0.5
            from = r.lo[1];
            to = r.hi[0] + 1.0;
        }
        return (a || b) && to - from < 0.49;
    }
    __device__ __forceinline__ void range(const MuCurve& u, float& mn, float& mx) const {
        const float va = u.A * ca + u.B * sa, vb = u.A * cb + u.B * sb;
        const float up = u.B * ca - u.A * sa, down = u.A * sb - u.B * cb;  // slope at the start, fall at the end
        mx = (up >= 0.f && down >= 0.f ? u.R : fmaxf(va, vb)) + u.C;
        mn = (up <= 0.f && down <= 0.f ? -u.R : fminf(va, vb)) + u.C;
    }
};

// The thread's sub-phases (bit k: phase ph[32 k]) at which element e is behind
// one of its npair >= 1 pairs.
__device__ __forceinline__ unsigned hidden_mask(const double2 (*ecl)[32], int npair, int e, const double* ph) {
    unsigned h = 0u;
    auto test = [&](double2 p) {
#pragma unroll
        for (int k = 0; k < kFluxR; ++k) {
            const double x = ph[32 * k];
            h |= (((x >= p.x && x <= p.y) || x <= p.y - 1.0) ? 1u : 0u) << k;
        }
    };
    test(ecl[0][e]);
#pragma unroll 1
    for (int j = 1; j < npair; ++j) test(ecl[j][e]);
    return h;
}

// 1/sqrt(x) of a normal positive x, by the hardware estimate that rsqrtf rounds to as well.
__device__ __forceinline__ float rsqrt_normal(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The mu above which an element of a unit's kind is seen.
__device__ __forceinline__ float mu_threshold(const ModelDev& M, int kind, int star) {
    if (kind == UK_DISC || kind == UK_DISC_LIN || kind == UK_SPOT) return 0.f;
    const float mc = star == 1 ? M.mucrit1f : M.mucrit2f;
    return kind == UK_STAR_GENERIC ? mc : fmaxf(mc, 0.f);  // see(mu) alone for the generic one
}

// Per-kind contribution of one element at one sub-phase (FP32).
template <int KIND>
struct Contrib {
    float a0, a1, a2, a3, thr, sumc, minus0;  // LD coefficients, mu threshold, sum of Claret coefficients
    __device__ void setup(const ModelDev& M, int star) {
        minus0 = __int_as_float(M.nslots >= 0 ? (int)0x80000000 : 0);
        const float* l = star == 1 ? M.ld1f : M.ld2f;
        a0 = l[0]; a1 = l[1]; a2 = l[2]; a3 = l[3];
        thr = mu_threshold(M, KIND, star);
        sumc = a0 + a1 + a2 + a3;
        if (KIND == UK_DISC || KIND == UK_DISC_LIN) { a0 = M.lin_ldf; a1 = M.quad_ldf; }
    }
    // Two sub-phases at once with the packed FP32x2 pipe (sm_100): each lane
    // rounded as a scalar operation is.
    // kInside: mu < 1 is known, so the clamp to 1 is left out (same bits), and
    // the product is an FMA with -0 (the same rounding; a value the compiler does
    // not know): it would fuse a plain packed product with the packed sum after it.
    template <bool kInside>
    __device__ __forceinline__ float2 pair(float2 mu, float fl) const {
        const float2 one = make_float2(1.f, 1.f), f2 = make_float2(fl, fl);
        const float2 nz = make_float2(minus0, minus0);
        auto product = [&](float2 x, float2 y) { return kInside ? __ffma2_rn(x, y, nz) : __fmul2_rn(x, y); };
        if (KIND == UK_SPOT) return product(mu, f2);
        const float2 mf = __fmul2_rn(mu, f2);
        if (KIND == UK_DISC || KIND == UK_DISC_LIN) {  // linear law: a1 om + a0 is a0
            const float2 om = __fadd2_rn(one, make_float2(-mu.x, -mu.y)), c0 = make_float2(a0, a0);
            const float2 q = KIND == UK_DISC ? __ffma2_rn(make_float2(a1, a1), om, c0) : c0;
            return product(mf, __ffma2_rn(make_float2(-om.x, -om.y), q, one));
        }
        const float2 m = kInside ? mu : make_float2(fminf(mu.x, 1.f), fminf(mu.y, 1.f));
        if (KIND == UK_STAR_CLARET) {
            const float2 ms = __fmul2_rn(m, kInside ? make_float2(rsqrt_normal(m.x), rsqrt_normal(m.y))
                                                               : make_float2(rsqrtf(m.x), rsqrtf(m.y)));
            float2 h = __ffma2_rn(ms, make_float2(a3, a3), make_float2(a2, a2));
            h = __ffma2_rn(ms, h, make_float2(a1, a1));
            h = __ffma2_rn(ms, h, make_float2(a0, a0));
            const float2 im = __ffma2_rn(ms, h, make_float2(1.f - sumc, 1.f - sumc));
            return product(mf, im);
        }
        const float2 om = __fadd2_rn(one, make_float2(-m.x, -m.y));
        float2 p;
        if (KIND == UK_STAR_POLY1) p = make_float2(a0, a0);
        else if (KIND == UK_STAR_POLY2) p = __ffma2_rn(om, make_float2(a1, a1), make_float2(a0, a0));
        else if (KIND == UK_STAR_POLY3) {
            p = __ffma2_rn(om, make_float2(a2, a2), make_float2(a1, a1));
            p = __ffma2_rn(om, p, make_float2(a0, a0));
        } else {
            p = __ffma2_rn(om, make_float2(a3, a3), make_float2(a2, a2));
            p = __ffma2_rn(om, p, make_float2(a1, a1));
            p = __ffma2_rn(om, p, make_float2(a0, a0));
        }
        return product(mf, __ffma2_rn(make_float2(-om.x, -om.y), p, one));
    }
};

// 1/x of a normal x by the hardware estimate.
__device__ __forceinline__ float rcp_normal(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Quotients and square roots, two at a time, of arguments far from the ends of
// the range: a hardware estimate and one Newton correction from its exact FMA
// residual (Markstein 1990), which rounds as / and sqrtf round but for a quotient
// within the estimate's error squared (~2^-44) of a tie.
// The general ones test each argument for the ends; the generic stars' terms are
// bound by issue slots, and by the special-function unit where they are lensed,
// so a square root's estimate serves the divisions by it as well.  Beaming alone,
// 73 and 151 latitudes at 3711 sub-phases (k_flux): 0.336 -> 0.197 ms; the lensed star's
// share of 5 million elements at 110,000 sub-phases: 351 -> 312 ms in all.
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
// a b + c d (+ e f), rounded as the compiler rounds the scalar expression.
__device__ __forceinline__ float2 dot_pair(float2 a, float2 b, float2 c, float2 d) {
    return __ffma2_rn(a, b, __fmul2_rn(c, d));
}
__device__ __forceinline__ float2 dot_pair(float2 a, float2 b, float2 c, float2 d, float2 e, float2 f) {
    return __ffma2_rn(e, f, dot_pair(a, b, c, d));
}
__device__ __forceinline__ float2 div_pair(float2 a, float2 b, float2 r) {  // r: an estimate of 1 / b
    const float2 q = __fmul2_rn(a, r);
    return __ffma2_rn(__ffma2_rn(neg2(b), q, a), r, q);
}
__device__ __forceinline__ float2 sqrt_pair(float2 x, float2 y) {  // y: an estimate of 1 / sqrt(x)
    const float2 s = __fmul2_rn(x, y);
    return __ffma2_rn(__ffma2_rn(neg2(s), s, x), __fmul2_rn(y, make_float2(0.5f, 0.5f)), s);
}

// Lensing magnification (flux.rs:390-406) at impact parameter sqrt(p2), Einstein
// radius squared rd.  Arguments near the ends of the range (a line of sight
// through the lens, say) take the scalar form, a lane at a time: a call instead
// of the loop cost beaming stars, which share this code, 40%.
__device__ __forceinline__ float2 lens_mag_pair(float2 p2, float2 rd) {
    const float lo = 1e-20f, hi = 1e20f;
    if (!(fminf(p2.x, p2.y) > lo && fmaxf(p2.x, p2.y) < hi && fmaxf(rd.x, rd.y) < hi)) {  // a NaN stays one either way
        float2 mag = p2;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            const float e = c ? rd.y : rd.x, pp = sqrtf(c ? p2.y : p2.x), phh = pp * 0.5f, phsq = phh * phh;
            const float pd = phsq > 25.f * e ? pp + e / pp : phh + sqrtf(fmaf(phh, phh, e));
            const float m = pd * pd / (pd - phh) / phh * 0.25f;
            if (c) mag.y = m;
            else mag.x = m;
        }
        return mag;
    }
    const float2 half = make_float2(0.5f, 0.5f), y = make_float2(rsqrt_normal(p2.x), rsqrt_normal(p2.y));
    const float2 pp = sqrt_pair(p2, y), phh = __fmul2_rn(pp, half), phsq = __fmul2_rn(phh, phh);
    float2 pd = __fadd2_rn(pp, div_pair(rd, pp, y));
    const bool nx = !(phsq.x > 25.f * rd.x), ny = !(phsq.y > 25.f * rd.y);
    if (nx || ny) {  // seldom: the line of sight passes within ten Einstein radii
        const float2 in = __ffma2_rn(phh, phh, rd);
        const float2 near = __fadd2_rn(phh, sqrt_pair(in, make_float2(rsqrt_normal(in.x), rsqrt_normal(in.y))));
        if (nx) pd.x = near.x;
        if (ny) pd.y = near.y;
    }
    const float2 b = __fadd2_rn(pd, neg2(phh));
    const float2 q = div_pair(__fmul2_rn(pd, pd), b, make_float2(rcp_normal(b.x), rcp_normal(b.y)));
    const float2 mag = div_pair(q, phh, __fadd2_rn(y, y));
    return __fmul2_rn(mag, make_float2(0.25f, 0.25f));
}

// LDC::imu of two sub-phases (types.rs:101-119).
__device__ __forceinline__ float2 imu_pair(const float (&l)[4], float sumc, int lt, float2 mu) {
    const float2 one = make_float2(1.f, 1.f), m = make_float2(fminf(mu.x, 1.f), fminf(mu.y, 1.f));
    const float2 l0 = make_float2(l[0], l[0]), l1 = make_float2(l[1], l[1]), l2 = make_float2(l[2], l[2]);
    const float2 l3 = make_float2(l[3], l[3]);
    const float2 x = lt == 0 ? __fadd2_rn(one, neg2(m)) : __fmul2_rn(m, make_float2(rsqrtf(m.x), rsqrtf(m.y)));
    const float2 h = __ffma2_rn(x, __ffma2_rn(x, __ffma2_rn(x, l3, l2), l1), l0);
    const float2 c = lt == 0 ? one : make_float2(1.f - sumc, 1.f - sumc);
    const float2 im = __ffma2_rn(lt == 0 ? neg2(x) : x, h, c);
    return make_float2(mu.x <= 0.f ? 0.f : im.x, mu.y <= 0.f ? 0.f : im.y);
}

// A unit's sub-phases are worked on in quarters of 32 n consecutive ones, n =
// ceil(tile / 128) to a thread, so that a quarter's lines of sight span a
// quarter of the tile's arc.  kBlock: the block's four warps share a unit, one
// quarter each, and sort its elements together; else each warp has a unit of its
// own and no barrier is met anywhere.
// flux_sort fills the unit's element masks; not a template over the kinds, so
// that all of them share its code.  Returns the quarters that have sub-phases
// (bit 2 q).
__device__ __forceinline__ bool sub_active(const FluxUnit& U, int t) {
    if (U.star == 1) return U.role == ROLE_BOTH || ((U.role == ROLE_FINE) == (t == 1));
    if (U.star == 2) return U.role == ROLE_BOTH || ((U.role == ROLE_FINE) == (t == 3));
    return true;
}

template <bool kBlock>
__device__ __noinline__ unsigned flux_sort(const FluxArgs& A, const FluxUnit& U, FluxUnitSmem& S) {
    const ModelDev& M = A.models[U.model];
    const int lane = threadIdx.x & 31;
    const int64_t sbase = M.sub_begin + U.t0;
    const int nslot = min(kFluxR, (U.nt + kFluxThreads - 1) / kFluxThreads);
    // ---- phase ranges of the quarters and of the tile, which decides the list of elements
    const int first = kBlock ? threadIdx.x >> 5 : 0, step = kBlock ? kFluxWarps : 1;
    auto sync = [] {
        if (kBlock) __syncthreads();
        else __syncwarp();
    };
    for (int q = first; q < kQuarters; q += step) {
        PhaseRange own;
        own.clear();
#pragma unroll
        for (int k = 0; k < kFluxR; ++k) {
            const int j = (q * nslot + k) * 32 + lane;
            if (k < nslot && j < U.nt && sub_active(U, A.sp_type[sbase + j])) own.put(A.sp_phi[sbase + j]);
        }
        own.warp_all();
        if (lane == 0) S.own[q] = own;
    }
    // the unit's used-slot words
    const int64_t g0 = U.e0 / kEclGroup;
    const int ngw = (int)((U.e0 + U.ne - 1) / kEclGroup - g0 + 1);
    for (int t = first * 32 + lane; t < ngw && t < kUnitGroups; t += 32 * step) S.gw[t] = A.ecl_grp[g0 + t];
    sync();
    PhaseRange tile = S.own[0];
    for (int q = 1; q < kQuarters; ++q) tile.join_range(S.own[q]);
    const bool any = tile.lo[0] <= tile.hi[0] || tile.lo[1] <= tile.hi[1];
    unsigned arc_on = 0u, arc_one = 0u;  // quarters with sub-phases; with all of them on one arc
    if (lane < 4 + 2 * kQuarters) {  // an angle per lane
        float x = 0.f;
        if (lane < 4) {
            const int h = lane >> 1;
            if (tile.lo[h] <= tile.hi[h]) x = (float)((lane & 1) ? tile.hi[h] : tile.lo[h]);
        } else {
            double from, to;
            const PhaseRange& r = S.own[(lane - 4) >> 1];
            if (WarpArc::ends(r, from, to)) arc_one = 1u;
            if (r.lo[0] <= r.hi[0] || r.lo[1] <= r.hi[1]) arc_on = 1u;
            x = (float)((lane & 1) ? to : from);
        }
        float sn, cs;
        sincospif(2.f * x, &sn, &cs);
        S.trig[lane] = make_float2(sn, cs);
    }
    arc_on = __ballot_sync(0xffffffffu, arc_on != 0u);
    arc_one = __ballot_sync(0xffffffffu, arc_one != 0u);
    __syncwarp();
    const float sif = (float)M.sini_l, cif = (float)M.cosi_l;
    const bool generic = U.kind == UK_STAR_GENERIC;
    const float thr = mu_threshold(M, U.kind, U.star), face_thr = thr - kFacingMargin;
    const int ngroups = any ? (U.ne + 31) / 32 : 0;
    const float4* recs = A.el_rec + U.e0 + lane;

    // ---- sort the elements, 32 at a time, a lane each.  The tile's list: those
    // that face the observer somewhere on the tile and are not hidden on all of it;
    // every 32 listed elements of a chunk the FP32 sums are folded into a two-sum
    // pair.  A quarter's arc then sorts the listed ones: those that never face it
    // or are hidden on all of it add nothing and are left out (leaving out zeros
    // changes neither blocks nor sums); plain ones face it throughout, unhidden and
    // with mu < 1, and need no test per sub-phase; limb ones need the test of mu;
    // mixed ones that of their pairs too.
    {
        Arcs arcs;
        for (int h = 0; h < 2; ++h) {
            arcs.on[h] = tile.lo[h] <= tile.hi[h];
            arcs.sa[h] = S.trig[2 * h].x; arcs.ca[h] = S.trig[2 * h].y;
            arcs.sb[h] = S.trig[2 * h + 1].x; arcs.cb[h] = S.trig[2 * h + 1].y;
        }
        float4 next = make_float4(0.f, 0.f, 0.f, 0.f);
        if (first * 32 + lane < U.ne) next = __ldg(recs + first * 32);
        for (int g = first; g < ngroups; g += step) {
            const MuCurve curve(sif, cif, next);
            const bool in = g * 32 + lane < U.ne;
            if ((g + step) * 32 + lane < U.ne) next = __ldg(recs + (g + step) * 32);
            bool list = in && !(max_mu(arcs, curve) <= face_thr);
            unsigned cls = 0u;  // per quarter two bits
            if (list) {
                const int64_t e = U.e0 + g * 32 + lane;
                const unsigned cm = S.gw[e / kEclGroup - g0];
                if (cm) {
                    int ct[2] = {CLS_VIS, CLS_VIS};
                    for (unsigned m = cm; m; m &= m - 1u)  // an unused slot, (inf, -inf), is neutral
                        tile.add(ct, __ldg(A.el_ecl + (__ffs(m) - 1) * A.sz.nelem + e));
                    const int t = tile.join(ct);
                    list = t != CLS_HID;
                    if (t == CLS_MIX)
                        for (int q = 0; q < kQuarters; ++q) {
                            int cq[2] = {CLS_VIS, CLS_VIS};
                            for (unsigned m = cm; m; m &= m - 1u)
                                S.own[q].add(cq, __ldg(A.el_ecl + (__ffs(m) - 1) * A.sz.nelem + e));
                            cls |= (unsigned)S.own[q].join(cq) << (2 * q);
                        }
                }
            }
            const unsigned listed = __ballot_sync(0xffffffffu, list);
            if (lane == 0) S.list[g] = listed;
            if (!listed) continue;
            for (int q = 0; q < kQuarters; ++q) {
                const unsigned c = (cls >> (2 * q)) & 3u;
                bool use = list && c != CLS_HID, plain = false;
                if ((arc_one >> (4 + 2 * q)) & 1u) {
                    const float2 a = S.trig[4 + 2 * q], b = S.trig[5 + 2 * q];
                    float mn, mx;
                    WarpArc{a.y, a.x, b.y, b.x}.range(curve, mn, mx);
                    use = use && mx > face_thr;
                    plain = !generic && c == CLS_VIS && mn > thr + kFacingMargin && mx < 1.f - kFacingMargin;
                }
                const unsigned us = __ballot_sync(0xffffffffu, use), pl = __ballot_sync(0xffffffffu, use && plain);
                const unsigned mi = __ballot_sync(0xffffffffu, use && c == CLS_MIX);
                if (lane == 0) {
                    S.used[g][q] = us;
                    S.plain[g][q] = pl;
                    S.mixed[g][q] = mi;
                }
            }
        }
    }
    sync();
    return any ? arc_on >> 4 & 0x55u : 0u;
}

// Quarters [q0, q1) of a sorted unit, by one warp.
template <int KIND>
__device__ __forceinline__ void flux_unit(const FluxArgs& A, const FluxUnit& U, int q0, int q1, unsigned arc_on,
                                          const FluxUnitSmem& T, FluxWarpSmem& S) {
    const ModelDev& M = A.models[U.model];
    const int lane = threadIdx.x & 31;
    const int64_t sbase = M.sub_begin + U.t0;
    const int nslot = min(kFluxR, (U.nt + kFluxThreads - 1) / kFluxThreads);
    q1 = min(q1, (U.nt + 32 * nslot - 1) / (32 * nslot));
    const int64_t g0 = U.e0 / kEclGroup;
    const int ngroups = (U.ne + 31) / 32;
    const float4* recs = A.el_rec + U.e0 + lane;
    Contrib<KIND> C;
    C.setup(M, U.star);
    // elements per unrolled step: more hides latency in long runs (a disc's), more code costs
    // instruction fetches where stars of two laws share an SM
    constexpr int kPlainUnroll = KIND == UK_DISC || KIND == UK_DISC_LIN ? LCB_DISC_UNROLL : LCB_FLUX_UNROLL;
    constexpr int kTestUnroll = KIND == UK_STAR_GENERIC ? LCB_GENERIC_UNROLL : LCB_LIMB_UNROLL;
    // generic-path constants
    const float ldc[4] = {C.a0, C.a1, C.a2, C.a3};
    const float vfac = M.vfacf, xcofm = M.xcofmf, rlens = M.rlens1f;
    const int ltg = U.star == 1 ? M.ltype1 : M.ltype2;
    const float beam = U.star == 1 ? M.beam1f : M.beam2f;
    const float spin = U.star == 1 ? M.spin1f : M.spin2f;
    const bool lens = U.star == 2 && M.glens1;
    double* out = A.partial + M.pbase + (int64_t)U.slot * M.nsub + U.t0;
    static_assert(kFluxR % 2 == 0, "sub-phases are processed in pairs");

    // ---- the sums, a quarter at a time
    for (int quarter = q0; quarter < q1; ++quarter) {
        const int j0 = quarter * 32 * nslot + lane;  // the thread's sub-phases: j0 + 32 k, k < nslot
        float ex[kFluxR], ey[kFluxR], ez[kFluxR];
        float2 ex2[kFluxR / 2], ey2[kFluxR / 2], ez2[kFluxR / 2], part[kFluxR / 2];
        float acc_hi[kFluxR], acc_lo[kFluxR];
        unsigned act = 0u;
#pragma unroll
        for (int k = 0; k < kFluxR; ++k) {
            const int j = j0 + 32 * k;
            float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
            double ph = -1.0;
            if (k < nslot && j < U.nt && sub_active(U, A.sp_type[sbase + j])) {
                e = A.sp_e[sbase + j];
                ph = A.sp_phi[sbase + j];
                act |= 1u << k;
            }
            S.ph[32 * k + lane] = ph;
            ex[k] = e.x; ey[k] = e.y; ez[k] = e.z;
            acc_hi[k] = acc_lo[k] = 0.f;
        }
#pragma unroll
        for (int k = 0; k < kFluxR; k += 2) {
            ex2[k / 2] = make_float2(ex[k], ex[k + 1]);
            ey2[k / 2] = make_float2(ey[k], ey[k + 1]);
            ez2[k / 2] = make_float2(ez[k], ez[k + 1]);
            part[k / 2] = make_float2(0.f, 0.f);
        }
        auto fold = [&] {
#pragma unroll
            for (int k = 0; k < kFluxR; ++k) {
                float& x = (k & 1) ? part[k / 2].y : part[k / 2].x;
                const float s = acc_hi[k] + x;
                const float bb = s - acc_hi[k];
                const float err = (acc_hi[k] - (s - bb)) + (x - bb);
                acc_hi[k] = s;
                acc_lo[k] += err;
                x = 0.f;
            }
        };
        auto mu_pair = [&](int k, const float4& r) {
            const float2 rx = make_float2(r.x, r.x), ry = make_float2(r.y, r.y), rz = make_float2(r.z, r.z);
            return __ffma2_rn(ez2[k], rz, __ffma2_rn(ey2[k], ry, __fmul2_rn(ex2[k], rx)));
        };
        const int ng = (arc_on >> (2 * quarter)) & 1u ? ngroups : 0;
        float4 next = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ng > 0 && lane < U.ne) next = __ldg(recs);
        int pos = 0;  // listed elements of the chunk so far
        for (int g = 0; g < ng; ++g) {
            const float4 mine = next;
            if ((g + 1) * 32 + lane < U.ne) next = __ldg(recs + (g + 1) * 32);
            const unsigned listed = T.list[g];
            if (listed) {
                const unsigned used = T.used[g][quarter], plains = T.plain[g][quarter], mixed = T.mixed[g][quarter];
                const int total = __popc(listed), room = 32 - (pos & 31);  // to the end of the FP32 block
                int npair = 0;
                if (used) {
                    S.rec[lane] = mine;
                    if ((mixed >> lane) & 1u) {
                        const int64_t e = U.e0 + g * 32 + lane;
                        for (unsigned m = T.gw[e / kEclGroup - g0]; m; m &= m - 1u) {
                            const double2 p = __ldg(A.el_ecl + (__ffs(m) - 1) * A.sz.nelem + e);
                            if (p.x <= 2.0) S.pair[npair++][lane] = p;
                        }
                    }
                    __syncwarp();
                }
                bool more = total >= room;  // the block ends in this group
                unsigned low = ~0u;
                if (more) low = __ballot_sync(0xffffffffu, __popc(listed & ((1u << lane) - 1u)) < room);
                unsigned m = used & low;
                for (;;) {
                    while (m) {
                        const int i = __ffs(m) - 1;
                        const float4* q = S.rec + i;
                        // a run of elements of one kind: plain, limb or mixed
                        const bool pl = (plains >> i) & 1u, mi = (mixed >> i) & 1u;
                        const unsigned rest = ~((m & (pl ? plains : mi ? mixed : ~(plains | mixed))) >> i);
                        const int len = rest ? __ffs(rest) - 1 : 32;
                        m &= ~((len < 32 ? (1u << len) - 1u : ~0u) << i);
                        if (KIND != UK_STAR_GENERIC && pl) {
#pragma unroll kPlainUnroll
                            for (int n = 0; n < len; ++n) {
                                const float4 r = q[n];
#pragma unroll
                                for (int k = 0; k < kFluxR / 2; ++k)
                                    part[k] = __fadd2_rn(part[k], C.template pair<true>(mu_pair(k, r), r.w));
                            }
                        } else if (KIND != UK_STAR_GENERIC && !mi) {
#pragma unroll kTestUnroll
                            for (int n = 0; n < len; ++n) {
                                const float4 r = q[n];
#pragma unroll
                                for (int k = 0; k < kFluxR / 2; ++k) {
                                    const float2 mu = mu_pair(k, r), c = C.template pair<false>(mu, r.w);
                                    if (mu.x > C.thr) part[k].x += c.x;
                                    if (mu.y > C.thr) part[k].y += c.y;
                                }
                            }
                        } else
#pragma unroll kTestUnroll
                        for (int n = 0; n < len; ++n) {
                        const float4 r = q[n];
                        // sub-phases behind one of the pairs (bit k: sub-phase k)
                        const int np = __shfl_sync(0xffffffffu, npair, i + n);
                        const unsigned hid = mi ? hidden_mask(S.pair, np, i + n, S.ph + lane) : 0u;
                        if (KIND == UK_STAR_GENERIC) {
                            const float4 p = __ldg(A.el_pos + U.e0 + g * 32 + i + n);
                            float vx, vy;
                            if (U.star == 1) { vx = -vfac * spin * p.y; vy = vfac * (spin * p.x - xcofm); }
                            else { vx = -vfac * spin * p.y; vy = vfac * (spin * (p.x - 1.f) + 1.f - xcofm); }
                            const float vn = r.x * vx + r.y * vy;
                            const float2 rx = make_float2(r.x, r.x), ry = make_float2(r.y, r.y), rz = make_float2(r.z, r.z);
                            const float2 px = make_float2(p.x, p.x), py = make_float2(p.y, p.y), pz = make_float2(p.z, p.z);
#pragma unroll
                            for (int k = 0; k < kFluxR / 2; ++k) {
                                const float2 mu = dot_pair(ex2[k], rx, ey2[k], ry, ez2[k], rz);
                                const bool sx = mu.x > C.thr && !((hid >> (2 * k)) & 1u);
                                const bool sy = mu.y > C.thr && !((hid >> (2 * k + 1)) & 1u);
                                if (!(sx || sy)) continue;
                                float2 t = mu, im = mu;
                                if (lens) {
                                    const float2 d = neg2(dot_pair(px, ex2[k], py, ey2[k], pz, ez2[k]));
                                    const float2 ax = __ffma2_rn(d, ex2[k], px), ay = __ffma2_rn(d, ey2[k], py), az = __ffma2_rn(d, ez2[k], pz);
                                    const float2 p2 = dot_pair(ax, ax, ay, ay, az, az);
                                    float2 mag = lens_mag_pair(p2, __fmul2_rn(make_float2(rlens, rlens), d));
                                    if (!(d.x > 0.f)) mag.x = 1.f;
                                    if (!(d.y > 0.f)) mag.y = 1.f;
                                    t = __fmul2_rn(mu, mag);
                                }
                                t = __fmul2_rn(t, make_float2(r.w, r.w));
                                if (beam != 0.f) {
                                    const float2 vr = neg2(dot_pair(ex2[k], make_float2(vx, vx), ey2[k], make_float2(vy, vy)));
                                    im = __fadd2_rn(__ffma2_rn(neg2(mu), vr, mu), make_float2(-vn, -vn));
                                    t = __fmul2_rn(t, __ffma2_rn(make_float2(-beam, -beam), vr, make_float2(1.f, 1.f)));
                                }
                                const float2 sum = __ffma2_rn(t, imu_pair(ldc, C.sumc, ltg, im), part[k]);
                                if (sx) part[k].x = sum.x;
                                if (sy) part[k].y = sum.y;
                            }
                        } else {
#pragma unroll
                            for (int k = 0; k < kFluxR; k += 2) {
                                const float2 mu = mu_pair(k / 2, r), c = C.template pair<false>(mu, r.w);
                                if (mu.x > C.thr && !((hid >> k) & 1u)) part[k / 2].x += c.x;
                                if (mu.y > C.thr && !((hid >> (k + 1)) & 1u)) part[k / 2].y += c.y;
                            }
                        }
                        }
                    }
                    if (!more) break;
                    fold();
                    more = false;
                    m = used & ~low;
                }
                pos += total;
                __syncwarp();  // the next group rewrites rec and pair
            }
            if (((g + 1) & (kFluxChunk / 32 - 1)) == 0 || g + 1 == ng) {  // the chunk's last block
                fold();
                pos = 0;
            }
        }
#pragma unroll
        for (int k = 0; k < kFluxR; ++k) {
            const int j = j0 + 32 * k;
            if (k < nslot && j < U.nt) out[j] = (act >> k) & 1u ? (double)acc_hi[k] + (double)acc_lo[k] : 0.0;
        }
        __syncwarp();  // the next quarter rewrites ph
    }
}

template <bool kBlock>
__global__ void __launch_bounds__(kFluxThreads, kFluxMinBlocks) k_flux(FluxArgs A) {
    __shared__ FluxUnitSmem units[kBlock ? 1 : kFluxWarps];
    __shared__ FluxWarpSmem warps[kFluxWarps];
    const int warp = threadIdx.x >> 5;
    FluxUnitSmem& T = units[kBlock ? 0 : warp];
    FluxWarpSmem& S = warps[warp];
    const int q0 = kBlock ? warp : 0, q1 = kBlock ? warp + 1 : kQuarters;
    for (;;) {
        if (kBlock) {
            __syncthreads();  // the last unit's masks are read
            if (threadIdx.x == 0) T.unit = atomicAdd(A.counter, 1);
            __syncthreads();
        } else {
            __syncwarp();
            if ((threadIdx.x & 31) == 0) T.unit = atomicAdd(A.counter, 1);
            __syncwarp();
        }
        const int64_t u = T.unit;
        if (u >= A.nunits) break;
        const FluxUnit U = A.units[u];
        if (!LCB_IN_BOUNDS(U.e0 + U.ne <= A.sz.nelem &&
                               A.models[U.model].sub_begin + U.t0 + U.nt <= A.sz.nsub &&
                               A.models[U.model].pbase + (int64_t)(U.slot + 1) * A.models[U.model].nsub <=
                                   A.sz.npartial,
                           A.status + U.model))
            continue;  // the unit is skipped by all who share it
        const unsigned on = flux_sort<kBlock>(A, U, T);
        switch (U.kind) {
            case UK_STAR_POLY1: flux_unit<UK_STAR_POLY1>(A, U, q0, q1, on, T, S); break;
            case UK_STAR_POLY2: flux_unit<UK_STAR_POLY2>(A, U, q0, q1, on, T, S); break;
            case UK_STAR_POLY3: flux_unit<UK_STAR_POLY3>(A, U, q0, q1, on, T, S); break;
            case UK_STAR_POLY4: flux_unit<UK_STAR_POLY4>(A, U, q0, q1, on, T, S); break;
            case UK_STAR_CLARET: flux_unit<UK_STAR_CLARET>(A, U, q0, q1, on, T, S); break;
            case UK_STAR_GENERIC: flux_unit<UK_STAR_GENERIC>(A, U, q0, q1, on, T, S); break;
            case UK_DISC: flux_unit<UK_DISC>(A, U, q0, q1, on, T, S); break;
            case UK_DISC_LIN: flux_unit<UK_DISC_LIN>(A, U, q0, q1, on, T, S); break;
            default: flux_unit<UK_SPOT>(A, U, q0, q1, on, T, S); break;
        }
    }
}

// ---------------------------------------------------------------------------
// k_curve, k_results
// ---------------------------------------------------------------------------
struct Gint {  // types.rs:130-202
    double p1, p2, s11, s12, s21, s22;
    __device__ double scale1(double phase) const {
        double pn = phase - floor(phase);
        if (pn <= p1 || pn >= 1.0 - p1) return 1.0;
        return (s11 * (1.0 - p1 - pn) + s12 * (pn - p1)) / (1.0 - 2.0 * p1);
    }
    __device__ double scale2(double phase) const {
        double pn = phase - floor(phase);
        if (pn >= p2 && pn <= 1.0 - p2) return 1.0;
        if (pn < 0.5) return (s22 * (p2 - pn) + s21 * (pn + p2)) / (2.0 * p2);
        return (s21 * (1.0 + p2 - pn) + s22 * (pn - 1.0 + p2)) / (2.0 * p2);
    }
};

constexpr int kEpiThreads = 256;

__device__ double block_sum(double v, double* red) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < kEpiThreads / 32; ++w) s += red[w];
    return s;
}

// Several block sums at once (one pair of barriers).
template <int N>
__device__ void block_sums(double (&v)[N], double (*red)[kEpiThreads / 32]) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; ++k) red[k][warp] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) {
        double s = 0.0;
        for (int w = 0; w < kEpiThreads / 32; ++w) s += red[k][w];
        v[k] = s;
    }
}

// iscale = 1 (orchestration.rs:185-227, 264-283, 405-436): the star-1, disc,
// rim, bright-spot and star-2 fluxes of each datum, and with scale the
// weighted least-squares scale factor of each, by one-sided Jacobi SVD of
// the design matrix (singular values at or below 1e-12 dropped), as the
// oracle restates nalgebra's solve.  No `third` term in this path.
// comp_star1/2 take the ginterp factor at the exposure's centre phase.
__device__ void epilogue_iscale(const EpiArgs& A, const ModelDev& M, const Gint& g, double s_wd, const double* aux,
                                double* res) {
    __shared__ double red[3][kEpiThreads / 32];
    const int ncol = M.t2 > 0.0 ? 5 : 4;
    const double* P = A.partial + M.pbase;
    double* F = A.fcomp + M.datum_begin * 5;
    double* X = A.svda + M.datum_begin * 5;
    for (int64_t d = threadIdx.x; d < M.ndatum; d += blockDim.x) {
        const int64_t gd = M.datum_begin + d;
        const lcb_datum D = A.data[M.data_begin + d];
        int64_t j = first_sub(M, A.dsub0, d) - M.sub_begin;
        const double centre = (D.ndiv > 0 ? A.sp_phi[M.sub_begin + j] : 0.0) +
                              (D.ndiv > 1 ? 0.5 * D.expose / M.period : 0.0);
        double f[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        for (int nd = 0; nd < D.ndiv; ++nd, ++j) {
            const double w = A.sp_w[M.sub_begin + j];
            double c[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
            for (int s = 0; s < M.g1_end; ++s) c[0] += P[(int64_t)s * M.nsub + j];
            for (int s = M.g2_end; s < M.gd_end; ++s) c[1] += P[(int64_t)s * M.nsub + j];
            for (int s = M.gd_end; s < M.ge_end; ++s) c[2] += P[(int64_t)s * M.nsub + j];
            for (int s = M.ge_end; s < M.nslots; ++s) c[3] += P[(int64_t)s * M.nsub + j];
            for (int s = M.g1_end; s < M.g2_end; ++s) c[4] += P[(int64_t)s * M.nsub + j];
            f[0] += w * g.scale1(centre) * c[0];
            f[1] += w * c[1];
            f[2] += w * c[2];
            f[3] += w * c[3];
            f[4] += w * g.scale2(centre) * c[4];
        }
        const double den = (double)max(1, D.ndiv - 1), slf = A.d_slfac[gd];
        for (int k = 0; k < 5; ++k) F[d * 5 + k] = k < ncol ? slf * (f[k] / den) : 0.0;
    }
    double sf[5] = {1.0, 1.0, 1.0, 1.0, 1.0}, wdf = 1.0;
    if (A.scale) {
        // rows with weight > 0, scaled by sqrt(weight)/ferr; other rows are zero and add nothing
        double nok[1] = {0.0};
        for (int64_t d = threadIdx.x; d < M.ndatum; d += blockDim.x) {
            const lcb_datum D = A.data[M.data_begin + d];
            const double w = D.weight > 0.0 ? sqrt(D.weight) / D.ferr : 0.0;
            if (D.weight > 0.0) nok[0] += 1.0;
            for (int k = 0; k < 5; ++k) X[d * 5 + k] = F[d * 5 + k] * w;
        }
        block_sums(nok, red);
        double x[5] = {1.0, 1.0, 1.0, 1.0, 1.0};
        if (nok[0] >= ncol && nok[0] > 0.0) {
            double V[5][5];
            for (int a = 0; a < 5; ++a)
                for (int b = 0; b < 5; ++b) V[a][b] = a == b ? 1.0 : 0.0;
            for (int sweep = 0; sweep < 60; ++sweep) {
                double off = 0.0;
                for (int p = 0; p < ncol; ++p)
                    for (int q = p + 1; q < ncol; ++q) {
                        double abg[3] = {0.0, 0.0, 0.0};
                        for (int64_t d = threadIdx.x; d < M.ndatum; d += blockDim.x) {
                            const double ap = X[d * 5 + p], aq = X[d * 5 + q];
                            abg[0] += ap * ap; abg[1] += aq * aq; abg[2] += ap * aq;
                        }
                        block_sums(abg, red);
                        const double alpha = abg[0], beta = abg[1], gamma = abg[2];
                        if (gamma == 0.0) continue;
                        off = fmax(off, fabs(gamma) / sqrt(alpha * beta));
                        const double zeta = (beta - alpha) / (2.0 * gamma);
                        const double t = (zeta >= 0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
                        const double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
                        for (int64_t d = threadIdx.x; d < M.ndatum; d += blockDim.x) {
                            const double ap = X[d * 5 + p], aq = X[d * 5 + q];
                            X[d * 5 + p] = c * ap - s * aq;
                            X[d * 5 + q] = s * ap + c * aq;
                        }
                        for (int i = 0; i < ncol; ++i) {  // every thread keeps the same V
                            const double vp = V[i][p], vq = V[i][q];
                            V[i][p] = c * vp - s * vq;
                            V[i][q] = s * vp + c * vq;
                        }
                    }
                if (off < 1e-15) break;
            }
            double sol[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
            for (int jc = 0; jc < ncol; ++jc) {
                double su[2] = {0.0, 0.0};
                for (int64_t d = threadIdx.x; d < M.ndatum; d += blockDim.x) {
                    const lcb_datum D = A.data[M.data_begin + d];
                    const double b = D.weight > 0.0 ? D.flux * sqrt(D.weight) / D.ferr : 0.0;
                    su[0] += X[d * 5 + jc] * X[d * 5 + jc];
                    su[1] += X[d * 5 + jc] * b;
                }
                block_sums(su, red);
                const double sj = sqrt(su[0]);
                if (!(sj > 1e-12)) continue;
                const double ub = su[1] / sj;
                for (int k = 0; k < ncol; ++k) sol[k] += V[k][jc] * ub / sj;
            }
            bool finite = true;
            for (int k = 0; k < ncol; ++k) finite = finite && isfinite(sol[k]);
            if (finite)
                for (int k = 0; k < ncol; ++k) x[k] = sol[k];
        }
        for (int k = 0; k < 5; ++k) sf[k] = k < ncol ? x[k] : 0.0;
        wdf = x[0];
    }
    double cw[2] = {0.0, 0.0};  // chi-squared, wnok
    for (int64_t d = threadIdx.x; d < M.ndatum; d += blockDim.x) {
        const int64_t gd = M.datum_begin + d;
        const lcb_datum D = A.data[M.data_begin + d];
        double c = sf[0] * F[d * 5 + 0] + sf[1] * F[d * 5 + 1] + sf[2] * F[d * 5 + 2] + sf[3] * F[d * 5 + 3];
        if (ncol == 5) c += sf[4] * F[d * 5 + 4];
        A.calc[gd] = c;
        if ((A.scale || A.rdata) && D.weight > 0.0) {
            cw[1] += D.weight;
            cw[0] += D.weight * sq((D.flux - c) / D.ferr);
        }
    }
    block_sums(cw, red);
    if (threadIdx.x == 0) {
        res[0] = s_wd * wdf;
        res[1] = cw[0];
        res[2] = cw[1];
        double fg1 = aux[AUX_FG1], f1 = aux[AUX_F1], fg2 = aux[AUX_FG2], f2 = aux[AUX_F2];
        res[3] = (M.glogg1 > 0.0 && fg1 > 0.0 && f1 > 0.0) ? log10(M.glogg1 * fg1 / f1) : 0.0;
        res[4] = (M.glogg2 > 0.0 && fg2 > 0.0 && f2 > 0.0) ? log10(M.glogg2 * fg2 / f2) : 0.0;
        res[5] = pow(aux[AUX_VOL1] / aux[AUX_SA1], 1.0 / 3.0);
        res[6] = pow(aux[AUX_VOL2] / aux[AUX_SA2], 1.0 / 3.0);
        for (int k = 0; k < 5; ++k) res[7 + k] = sf[k];
    }
}

// The ginterp scale factors of a model (orchestration.rs:86-131, with the live
// Ginterp) and its white-dwarf flux.
__device__ Gint model_gint(const ModelDev& M, const double* aux, double& s_wd) {
    Gint g{M.phase1, M.phase2, 1.0, 1.0, 1.0, 1.0};
    auto c1 = [&](int s) { return g.scale1(M.spec[s].phase) * aux[AUX_SPEC0 + s]; };
    auto c2 = [&](int s) { return g.scale2(M.spec[s].phase) * aux[AUX_SPEC0 + s]; };
    if (!M.copy1) {
        g.s11 = c1(M.spec_g11[0]) / c1(M.spec_g11[1]);
        g.s12 = c1(M.spec_g12[0]) / c1(M.spec_g12[1]);
    }
    if (!M.copy2) {
        g.s21 = c2(M.spec_g21[0]) / c2(M.spec_g21[1]);
        g.s22 = c2(M.spec_g22[0]) / c2(M.spec_g22[1]);
    }
    s_wd = g.scale1(0.5) * aux[AUX_SPEC0 + M.spec_wd];
    return g;
}

// Fluxes: per datum, the sum of its slots' partial sums under the ginterp
// factors, trapezoid over the exposure (orchestration.rs:243-310); and per
// block the sums that re_scale and the chi-squared need.  A tile is 32 data, a
// warp's lanes.  Bound by reading the partial sums (8 B a slot and sub-phase).
// kShare = 1: each warp takes tiles of its own.  kShare = 8 (few tiles: one
// long light curve): the block's eight warps share a tile's slots, which makes
// eight times the warps; one block per model took 48.7 ms for 1,240 slots x
// 110,000 sub-phases (1.74 ms here) and 1.26 ms for 110 x 50,000 (0.05 ms),
// almost all of it latency of one SM.
constexpr int kCurveTile = 32;

template <int kShare>
__global__ void __launch_bounds__(kEpiThreads) k_curve(EpiArgs A) {
    constexpr int kWarps = kEpiThreads / 32, kTiles = kWarps / kShare;  // tiles a block works on at once
    static_assert(kShare == 1 || kShare == kWarps, "a block's barriers are inside the tile loop");
    const int64_t m = blockIdx.x;
    const ModelDev& M = A.models[m];
    const bool in_range = LCB_IN_BOUNDS(M.pbase + (int64_t)M.nslots * M.nsub <= A.sz.npartial &&
                                            M.datum_begin + M.ndatum <= A.sz.ndatum && M.data_begin + M.ndatum <= A.sz.ndata &&
                                            M.sub_begin + M.nsub <= A.sz.nsub,
                                        A.bad + m);
    if (M.status < 0 || A.status[m] != 0 || !in_range) {
        for (int64_t d = (int64_t)blockIdx.y * kEpiThreads + threadIdx.x; d < M.ndatum; d += (int64_t)gridDim.y * kEpiThreads)
            A.calc[M.datum_begin + d] = NAN;
        return;
    }
    if (M.iscale) return;  // k_results: its fluxes are per component
    __shared__ double part[2][kShare][3][32];
    __shared__ double red[4][kWarps];
    __shared__ Gint G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int share = kShare > 1 ? warp : 0;           // the warp's part of a tile's slots
    const bool lead = share == 0;
    if (threadIdx.x == 0) {
        double wd;
        G = model_gint(M, A.aux + m * kNumAux, wd);
    }
    __syncthreads();
    const Gint g = G;
    const double* P = A.partial + M.pbase;
    double v[4] = {0.0, 0.0, 0.0, 0.0};  // chi, wnok, sdy, syy
    int buf = 0;
    const int64_t step = (int64_t)gridDim.y * kTiles * kCurveTile;
    for (int64_t d0 = ((int64_t)blockIdx.y * kTiles + (kShare > 1 ? 0 : warp)) * kCurveTile; d0 < M.ndatum; d0 += step) {
        const int64_t d = d0 + lane, gd = M.datum_begin + d;
        const bool on = d < M.ndatum;
        const int ndiv = on ? A.data[M.data_begin + d].ndiv : 0;
        const int64_t j0 = on ? first_sub(M, A.dsub0, d) - M.sub_begin : 0;
        const int most = __reduce_max_sync(0xffffffffu, ndiv);  // the same in every warp that shares the tile
        double sum = 0.0;
        for (int nd = 0; nd < most; ++nd, buf ^= 1) {
            const bool act = nd < ndiv;
            double t[3] = {0.0, 0.0, 0.0};
            if (act) {
                const double* q = P + j0 + nd;
                int s = share;
#pragma unroll 4
                for (; s < M.g1_end; s += kShare) t[0] += q[(int64_t)s * M.nsub];
#pragma unroll 4
                for (; s < M.g2_end; s += kShare) t[1] += q[(int64_t)s * M.nsub];
#pragma unroll 8
                for (; s < M.nslots; s += kShare) t[2] += q[(int64_t)s * M.nsub];
            }
            if (kShare > 1) {
                for (int k = 0; k < 3; ++k) part[buf][share][k][lane] = t[k];
                __syncthreads();  // the other buffer is free: the lead warp read it before it came here
                if (lead)
                    for (int k = 0; k < 3; ++k) {
                        t[k] = 0.0;
                        for (int w = 0; w < kShare; ++w) t[k] += part[buf][w][k][lane];
                    }
            }
            if (lead && act) {
                const double pn = A.sp_phi[M.sub_begin + j0 + nd];
                double ss = t[0] * g.scale1(pn);
                ss += g.scale2(pn) * t[1];
                ss += t[2];
                sum += A.sp_w[M.sub_begin + j0 + nd] * ss;
            }
        }
        if (lead && on) {
            const lcb_datum D = A.data[M.data_begin + d];
            const double c = A.d_slfac[gd] * (sum / (double)max(1, D.ndiv - 1)) + M.third;
            A.calc[gd] = c;
            if (D.weight > 0.0) {
                if (A.scale) {
                    const double w = D.weight / sq(D.ferr);
                    v[2] += w * D.flux * c;
                    v[3] += w * c * c;
                    v[1] += D.weight;
                } else if (A.rdata) {
                    v[1] += D.weight;
                    v[0] += D.weight * sq((D.flux - c) / D.ferr);
                }
            }
        }
    }
    block_sums(v, red);
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) A.episum[(m * gridDim.y + blockIdx.y) * 4 + k] = v[k];
}

// Per model: the scale factor and the chi-squared (orchestration.rs:361-401)
// from k_curve's sums, log g and radii.  gridDim.y > 1 (a light curve of many
// data, scaled) splits the rescaled pass over blocks; the last one to finish
// adds their chi-squared parts in block order.
__global__ void __launch_bounds__(kEpiThreads) k_results(EpiArgs A) {
    const int64_t m = blockIdx.x;
    const ModelDev& M = A.models[m];
    double* res = A.results + m * 12;
    __shared__ double red[kEpiThreads / 32], red4[4][kEpiThreads / 32];
    const bool in_range = M.pbase + (int64_t)M.nslots * M.nsub <= A.sz.npartial &&
                          M.datum_begin + M.ndatum <= A.sz.ndatum && M.data_begin + M.ndatum <= A.sz.ndata &&
                                            M.sub_begin + M.nsub <= A.sz.nsub;
    if (M.status < 0 || A.status[m] != 0 || !in_range) {
        if (blockIdx.y == 0 && threadIdx.x < 12) res[threadIdx.x] = NAN;
        return;
    }
    double* aux = A.aux + m * kNumAux;
    if (M.iscale) {
        if (blockIdx.y > 0) return;
        __shared__ Gint G;
        __shared__ double s_wd;
        if (threadIdx.x == 0) G = model_gint(M, aux, s_wd);
        __syncthreads();
        const Gint g = G;
        epilogue_iscale(A, M, g, s_wd, aux, res);
        return;
    }
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t k = threadIdx.x; k < A.curve_blocks; k += kEpiThreads)
        for (int i = 0; i < 4; ++i) v[i] += A.episum[(m * A.curve_blocks + k) * 4 + i];
    block_sums(v, red4);
    double chi = v[0], wnok = v[1], sfac = 1.0;
    const double sdy = v[2], syy = v[3];
    bool last = blockIdx.y == 0;
    if (A.scale) {  // re_scale (orchestration.rs:361-388)
        chi = 0.0;
        if (wnok > 0.0 && syy > 0.0) {
            sfac = sdy / syy;
            for (int64_t d = (int64_t)blockIdx.y * kEpiThreads + threadIdx.x; d < M.ndatum;
                 d += (int64_t)gridDim.y * kEpiThreads) {
                const int64_t gd = M.datum_begin + d;
                const lcb_datum D = A.data[M.data_begin + d];
                const double c = A.calc[gd] * sfac;
                A.calc[gd] = c;
                if (D.weight > 0.0) chi += D.weight * sq((D.flux - c) / D.ferr);
            }
            chi = block_sum(chi, red);
            if (gridDim.y > 1) {
                __shared__ bool s_last;
                if (threadIdx.x == 0) {
                    A.chipart[m * gridDim.y + blockIdx.y] = chi;
                    __threadfence();
                    s_last = atomicAdd(reinterpret_cast<unsigned*>(aux + AUX_DONE), 1u) == gridDim.y - 1;
                }
                __syncthreads();
                last = s_last;
                if (last) {
                    __threadfence();
                    chi = 0.0;
                    for (int64_t k = threadIdx.x; k < gridDim.y; k += kEpiThreads)
                        chi += *(volatile double*)(A.chipart + m * gridDim.y + k);
                    chi = block_sum(chi, red);
                }
            }
        } else {
            wnok = 0.0;
        }
    }
    if (!last) return;
    // a warp each for the values that need a logarithm or a power
    const double fg1 = aux[AUX_FG1], f1 = aux[AUX_F1], fg2 = aux[AUX_FG2], f2 = aux[AUX_F2];
    switch (threadIdx.x) {
        case 0: {
            double s_wd;
            model_gint(M, aux, s_wd);
            res[0] = s_wd * sfac;
            res[1] = chi;
            res[2] = wnok;
            for (int k = 0; k < 5; ++k) res[7 + k] = sfac;
            break;
        }
        case 32: res[3] = (M.glogg1 > 0.0 && fg1 > 0.0 && f1 > 0.0) ? log10(M.glogg1 * fg1 / f1) : 0.0; break;
        case 64: res[4] = (M.glogg2 > 0.0 && fg2 > 0.0 && f2 > 0.0) ? log10(M.glogg2 * fg2 / f2) : 0.0; break;
        case 96: res[5] = pow(aux[AUX_VOL1] / aux[AUX_SA1], 1.0 / 3.0); break;
        case 128: res[6] = pow(aux[AUX_VOL2] / aux[AUX_SA2], 1.0 / 3.0); break;
        default: break;
    }
}

// FMA throughput microbenchmark: 8 independent FMA chains per thread.
template <class T>
__global__ void __launch_bounds__(256) k_fma_peak(T* out, int iters, T seed) {
    T a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = seed + (T)(threadIdx.x + k);
    const T b = (T)0.999999, c = (T)1e-7;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = a[k] * b + c;
    }
    T s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += a[k];
    if (s == (T)-12345.0) out[0] = s;  // keeps the chains live
}

}  // namespace

cudaError_t measure_fma_peak(int fp64, int num_sms, cudaStream_t s, double* tflops) {
    void* out = nullptr;
    cudaError_t e = cudaMalloc(&out, 16);
    if (e != cudaSuccess) return e;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const int blocks = num_sms * 8, threads = 256, iters = fp64 ? 4096 : 8192;
    double best = 0.0;
    for (int rep = 0; rep < 4; ++rep) {
        cudaEventRecord(a, s);
        if (fp64) k_fma_peak<double><<<blocks, threads, 0, s>>>((double*)out, iters, 1.0);
        else k_fma_peak<float><<<blocks, threads, 0, s>>>((float*)out, iters, 1.0f);
        cudaEventRecord(b, s);
        e = cudaEventSynchronize(b);
        if (e != cudaSuccess) break;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, a, b);
        double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
        if (rep > 0) best = std::max(best, flops / (ms * 1e-3) / 1e12);
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(out);
    *tflops = best;
    return e != cudaSuccess ? e : cudaGetLastError();
}

__global__ void k_ecl_export(const double2* __restrict__ ecl, int64_t nelem, int64_t first, int64_t count,
                             double2* __restrict__ out) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // (element, slot), slot fastest
    if (j >= count * kMaxEcl) return;
    const int64_t i = j / kMaxEcl;
    const int k = (int)(j - i * kMaxEcl);
    out[j] = ecl[k * nelem + first + i];
}

__global__ void k_ecl_import(const double2* __restrict__ in, int64_t nelem, double2* __restrict__ ecl,
                             unsigned* __restrict__ grp) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nelem * kMaxEcl) return;
    const int64_t e = j / kMaxEcl;
    const int k = (int)(j - e * kMaxEcl);
    const double2 p = in[j];
    ecl[k * nelem + e] = p;
    if (p.x <= 2.0) atomicOr(grp + e / kEclGroup, 1u << k);
}

cudaError_t launch_ecl_export(const double2* ecl, int64_t nelem, int64_t first, int64_t count, double2* out,
                              cudaStream_t s) {
    const int64_t n = count * kMaxEcl;
    if (n > 0) k_ecl_export<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(ecl, nelem, first, count, out);
    return cudaGetLastError();
}

cudaError_t launch_ecl_import(const double2* in, int64_t nelem, double2* ecl, unsigned* ecl_grp, cudaStream_t s) {
    const int64_t n = nelem * kMaxEcl;
    if (n > 0) k_ecl_import<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, nelem, ecl, ecl_grp);
    return cudaGetLastError();
}

// The bright spot's gas-stream end point for pair i (lcb_stream.h, the planner's
// host code compiled for the device): one thread per pair, each in a block of its
// own, since every integration is one long serial chain of FP64 operations and
// the pairs' step sequences differ (lanes of one warp would diverge).
__global__ void __launch_bounds__(1) k_stream(const double* __restrict__ in, int n, double* __restrict__ out,
                                              int* __restrict__ status) {
    const int i = blockIdx.x;
    if (i >= n) return;
    double o[3] = {0.0, 0.0, 0.0};
    status[i] = stream::stream_to_radius_core(in[3 * i], in[3 * i + 1], in[3 * i + 2], o);
    out[3 * i] = o[0]; out[3 * i + 1] = o[1]; out[3 * i + 2] = o[2];
}

cudaError_t launch_stream(const double* in, int n, double* out, int* status, cudaStream_t s) {
    if (n > 0) k_stream<<<(unsigned)n, 1, 0, s>>>(in, n, out, status);
    return cudaGetLastError();
}

cudaError_t launch_wait_probe(long long limit, int* status, long long* waited, cudaStream_t s) {
    k_wait_probe<<<1, 32, 0, s>>>(limit, status, waited);
    return cudaGetLastError();
}

int flux_blocks_per_sm() {
    int n = 0, m = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_flux<false>, kFluxThreads, 0) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_flux<true>, kFluxThreads, 0) != cudaSuccess) return 0;
    return std::min(n, m);
}

cudaError_t launch_phase(const PhaseArgs& a, cudaStream_t s) {
    if (a.nmodels <= 0 || a.most <= 0) return cudaSuccess;
    const int64_t blocks = std::min<int64_t>((a.most + 127) / 128, 65535);
    k_phase<<<dim3((unsigned)a.nmodels, (unsigned)blocks), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_elements(const ElemArgs& a, cudaStream_t s) {
    if (a.nblocks > 0) {
        k_elements<<<(unsigned)a.nblocks, kElemThreads, 0, s>>>(a);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_roche(const ElemArgs& a, cudaStream_t s) {
    if (a.nrblocks <= 0) return cudaSuccess;
    k_roche<<<(unsigned)(2 * a.nrblocks), kRocheBlock, 0, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const unsigned grid = (unsigned)std::min<int64_t>(a.open_grid, 16 * a.nrblocks);
    if (a.split_all) k_roche_open<true><<<grid, kRocheBlock, 0, s>>>(a);
    else k_roche_open<false><<<grid, kRocheBlock, 0, s>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_roche_chop2<<<grid, kRocheBlock, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_aux(const ElemArgs& a, cudaStream_t s) {
    if (a.nablocks <= 0) return cudaSuccess;
    k_aux<<<(unsigned)a.nablocks, kElemThreads, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_flux(const FluxArgs& a, int grid, cudaStream_t s) {
    if (a.nunits <= 0) return cudaSuccess;
    if (a.share) k_flux<true><<<grid, kFluxThreads, 0, s>>>(a);
    else k_flux<false><<<grid, kFluxThreads, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_epilogue(const EpiArgs& a, cudaStream_t s) {
    if (a.nmodels <= 0) return cudaSuccess;
    const dim3 grid((unsigned)a.nmodels, (unsigned)a.curve_blocks);
    if (a.curve_share) k_curve<kEpiThreads / 32><<<grid, kEpiThreads, 0, s>>>(a);
    else k_curve<1><<<grid, kEpiThreads, 0, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_results<<<dim3((unsigned)a.nmodels, (unsigned)(a.scale ? a.result_blocks : 1)), kEpiThreads, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace lcb
