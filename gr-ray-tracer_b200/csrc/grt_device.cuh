// Device-side pieces of the per-photon hot path shared by the trace kernels:
// counter-based RNG, nonuniform-grid cell lookup, fluid sampling + tetrad,
// radiative transfer, scattering, packet generators and the camera test.
//
// Each function names the reference function it replaces (file:line within the
// reference project).  Floating-point expressions keep the reference's
// association so the FP64 parity kernel (built with -fmad=false) rounds like
// the reference; differences can come only from libdevice vs glibc in log,
// acos, atan2, exp and pow, which are called, never re-implemented.
#pragma once

#include <stdint.h>

#include "grt_kparams.h"
#include "grt_metric.cuh"
#include "grt_sincos.h"
#include "grt_user_physics.h"

namespace grt {
namespace dev {

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon, Moraes, Dror & Shaw, SC'11), key = 64-bit seed,
// counter = {id_lo, id_hi, domain, block}.  Each block gives four words = two
// doubles in [0,1) with 53 random bits.  One stream per (photon id, host step),
// which replaces the reference's Kokkos::Random_XorShift64_Pool
// (src/radiative_transfer/scattering.hpp:16-17) with a reproducible generator.
// ---------------------------------------------------------------------------
struct Philox {
    uint32_t k0, k1, c0, c1, c2, c3;
    uint32_t w[4];
    int used;

    GRT_DEV Philox(uint64_t seed, uint64_t id, uint32_t domain)
        : k0(static_cast<uint32_t>(seed)), k1(static_cast<uint32_t>(seed >> 32)),
          c0(static_cast<uint32_t>(id)), c1(static_cast<uint32_t>(id >> 32)), c2(domain), c3(0),
          used(4) {}

    static GRT_DEV void block(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t key0,
                              uint32_t key1, uint32_t out[4]) {
#pragma unroll 1
        for (int round = 0; round < 10; ++round) {
            const uint32_t hi0 = __umulhi(0xD2511F53u, x0), lo0 = 0xD2511F53u * x0;
            const uint32_t hi1 = __umulhi(0xCD9E8D57u, x2), lo1 = 0xCD9E8D57u * x2;
            x0 = hi1 ^ x1 ^ key0;
            x1 = lo1;
            x2 = hi0 ^ x3 ^ key1;
            x3 = lo0;
            key0 += 0x9E3779B9u;
            key1 += 0xBB67AE85u;
        }
        out[0] = x0; out[1] = x1; out[2] = x2; out[3] = x3;
    }

    GRT_DEV double drand() {
        if (used >= 4) {
            block(c0, c1, c2, c3, k0, k1, w);
            ++c3;
            used = 0;
        }
        const uint64_t hi = used == 0 ? w[0] : w[2];
        const uint64_t lo = used == 0 ? w[1] : w[3];
        used += 2;
        return static_cast<double>((hi << 21) | (lo >> 11)) * (1.0 / 9007199254740992.0);
    }
};
constexpr uint32_t kInitDomain = 0xFFFFFFFFu;    // disk-mode emission draws
constexpr uint32_t kScreenDomain = 0xFFFFFFFEu;  // image-mode random screen (u, v)

// ---------------------------------------------------------------------------
// Nonuniform (r, theta, phi) grid lookup (scattering.hpp:41-180)
// ---------------------------------------------------------------------------

// scattering.hpp:41-45
GRT_DEV double periodic_angle_distance(double lhs, double rhs) {
    const double d = fmod(fabs(lhs - rhs), 2.0 * kPi);
    return fmin(d, 2.0 * kPi - d);
}

// Separable sorted axes: the reference's linear argmin with strict '<'
// (first index wins ties, scattering.hpp:55-63,73-79,89-95) computed from the
// bracketing pair found by binary search.  Valid because the distance to a
// sorted axis is monotone on each side of the query (division and log are
// monotone); the host only enables this path when every axis is strictly
// increasing with neighbouring values separated by more than 1e-12 relative,
// which rules out equal distances at non-adjacent indices.
GRT_DEV int bracket(const double* axis, int n, double q) {
    int lo = -1, hi = n;  // axis[lo] <= q < axis[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (axis[mid] <= q) lo = mid; else hi = mid;
    }
    return lo;
}

GRT_DEV int nearest_polar_sorted(const double* th, int n, double polar) {
    const int lo = bracket(th, n, polar);
    if (lo < 0) return 0;
    if (lo + 1 >= n) return lo;
    const double dlo = fabs(polar - th[lo]);
    const double dhi = fabs(polar - th[lo + 1]);
    return dhi < dlo ? lo + 1 : lo;
}

// periodic_angle_distance for |lhs - rhs| <= 4 pi: fmod(v, 2 pi) is v, or
// exactly v - 2 pi (Sterbenz) for v in [2 pi, 4 pi).  The separable path has
// azimuth queries in [0, 2 pi] and axis values in [0, 2 pi).
GRT_DEV double periodic_angle_distance_near(double lhs, double rhs) {
    const double v = fabs(lhs - rhs);
    const double d = v >= 2.0 * kPi ? v - 2.0 * kPi : v;
    return fmin(d, 2.0 * kPi - d);
}

GRT_DEV int nearest_azimuth_sorted(const double* ph, int n, double az) {
    if (n == 1) return 0;
    const int lo = bracket(ph, n, az);
    const int c1 = lo < 0 ? n - 1 : lo;
    const int c2 = lo + 1 < n ? lo + 1 : 0;
    const double d1 = periodic_angle_distance_near(az, ph[c1]);
    const double d2 = periodic_angle_distance_near(az, ph[c2]);
    if (d1 < d2) return c1;
    if (d2 < d1) return c2;
    return c1 < c2 ? c1 : c2;
}

// The nearest radial cell and whether it accepts the radius (scattering.hpp:
// 99-117 with the neighbour half-span precomputed per axis value, see
// KGrid::r_half): the log distance of the chosen cell is the one the
// nearest-cell test computed, so it is evaluated once per candidate (one or
// two), through one site.  Ties go to the lower index.
GRT_DEV bool locate_radial_sorted(const double* r, const double* half, int n, double radius, int& i) {
    const int lo = bracket(r, n, radius);
    const int c0 = lo < 0 ? 0 : lo;
    const int ncand = (lo >= 0 && lo + 1 < n) ? 2 : 1;
    double best = 0.0;
    int bi = c0;
#pragma unroll 1
    for (int k = 0; k < ncand; ++k) {
        const double d = fabs(log(radius / r[c0 + k]));
        if (k == 0 || d < best) {
            best = d;
            bi = c0 + k;
        }
    }
    i = bi;
    return best <= half[bi];
}
GRT_DEV bool within_polar_sorted(const double* th, const double* half, int j, double polar) {
    return fabs(polar - th[j]) <= half[j];
}
GRT_DEV bool within_azimuth_sorted(const double* ph, const double* half, int k, double az) {
    return periodic_angle_distance_near(az, ph[k]) <= half[k];
}

// General (non-separable) coordinates: the reference's three coordinate-descent
// passes of linear scans over the full 3-D coordinate arrays
// (scattering.hpp:151-180), used when the grid is not separable.
struct Grid3 {
    const double* r;
    const double* th;
    const double* ph;
    int nr, nth, nph;
    GRT_DEV size_t at(int i, int j, int k) const {
        return (static_cast<size_t>(i) * nth + j) * nph + k;
    }
};

static __device__ __noinline__ bool locate_general(const Grid3& g, double radius, double polar, double az, int& i, int& j,
                            int& k) {
    j = g.nth / 2;
    k = g.nph / 2;
    i = g.nr / 2;
    for (int it = 0; it < 3; ++it) {
        {  // nearest_radial_index
            const double first = g.r[g.at(0, j, k)];
            if (!(first > 0.0)) return false;
            int best_i = 0;
            double best = fabs(log(radius / first));
            for (int q = 1; q < g.nr; ++q) {
                const double c = g.r[g.at(q, j, k)];
                if (!(c > 0.0)) continue;
                const double d = fabs(log(radius / c));
                if (d < best) { best_i = q; best = d; }
            }
            i = best_i;
        }
        {  // nearest_polar_index
            int best_j = 0;
            double best = fabs(polar - g.th[g.at(i, 0, k)]);
            for (int q = 1; q < g.nth; ++q) {
                const double d = fabs(polar - g.th[g.at(i, q, k)]);
                if (d < best) { best_j = q; best = d; }
            }
            j = best_j;
        }
        {  // nearest_azimuth_index
            int best_k = 0;
            double best = periodic_angle_distance(az, g.ph[g.at(i, j, 0)]);
            for (int q = 1; q < g.nph; ++q) {
                const double d = periodic_angle_distance(az, g.ph[g.at(i, j, q)]);
                if (d < best) { best_k = q; best = d; }
            }
            k = best_k;
        }
    }
    {  // within_radial_cell
        const double center = g.r[g.at(i, j, k)];
        if (!(center > 0.0)) return false;
        const double cd = fabs(log(radius / center));
        if (g.nr == 1) {
            if (!(cd <= 1.0e-10)) return false;
        } else {
            double span = 0.0;
            if (i > 0 && g.r[g.at(i - 1, j, k)] > 0.0)
                span = fmax(span, fabs(log(center / g.r[g.at(i - 1, j, k)])));
            if (i + 1 < g.nr && g.r[g.at(i + 1, j, k)] > 0.0)
                span = fmax(span, fabs(log(center / g.r[g.at(i + 1, j, k)])));
            if (!(cd <= 0.500001 * span)) return false;
        }
    }
    {  // within_polar_cell
        const double center = g.th[g.at(i, j, k)];
        const double cd = fabs(polar - center);
        if (g.nth == 1) {
            if (!(cd <= 1.0e-10)) return false;
        } else {
            double span = 0.0;
            if (j > 0) span = fmax(span, fabs(center - g.th[g.at(i, j - 1, k)]));
            if (j + 1 < g.nth) span = fmax(span, fabs(center - g.th[g.at(i, j + 1, k)]));
            if (!(cd <= 0.500001 * span)) return false;
        }
    }
    {  // within_azimuth_cell
        const double center = g.ph[g.at(i, j, k)];
        const double cd = periodic_angle_distance(az, center);
        if (g.nph == 1) {
            if (!(cd <= 1.0e-10)) return false;
        } else {
            double span = 0.0;
            if (k > 0) span = fmax(span, periodic_angle_distance(center, g.ph[g.at(i, j, k - 1)]));
            if (k + 1 < g.nph) span = fmax(span, periodic_angle_distance(center, g.ph[g.at(i, j, k + 1)]));
            if (!(cd <= 0.500001 * span)) return false;
        }
    }
    return true;
}

// ---------------------------------------------------------------------------
// Fluid sample + tetrad (scattering.hpp:185-251, fluid_frame.hpp:51-80)
// ---------------------------------------------------------------------------
struct FluidSample {
    FluidCellCGS fluid;
    double e[4][4];  // tetrad, e[0] = fluid four-velocity
    int cell;
};

// fluid_frame.hpp:51-80 with the metric already evaluated at the photon.
// UNROLL: as straight-line code, which disappears where its result is unused.
template <bool UNROLL = false>
GRT_DEV bool build_tetrad(const double g[4][4], const double u[4], double e[4][4]) {
    const double vn = metric_dot(g, u, u);
    if (!(vn < 0.0) || !isfinite(vn)) return false;
    const double inv = 1.0 / sqrt(-vn);
    const double ts = u[0] >= 0.0 ? 1.0 : -1.0;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) e[0][mu] = ts * u[mu] * inv;
    // Rolled over the spatial axes (one square-root and one division site).
#pragma unroll(UNROLL ? 3 : 1)
    for (int axis = 0; axis < 3; ++axis) {
        double cand[4];
        const double tp = metric_dot_unit(g, e[0], axis + 1);
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) cand[mu] = (mu == axis + 1 ? 1.0 : 0.0) + tp * e[0][mu];
#pragma unroll(UNROLL ? 3 : 1)
        for (int prev = 0; prev < axis; ++prev) {
            const double proj = metric_dot(g, e[prev + 1], cand);
#pragma unroll
            for (int mu = 0; mu < 4; ++mu) cand[mu] -= proj * e[prev + 1][mu];
        }
        const double n = metric_dot(g, cand, cand);
        if (!(n > 1.0e-20) || !isfinite(n)) return false;
        const double is = 1.0 / sqrt(n);
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) e[axis + 1][mu] = cand[mu] * is;
    }
    return true;
}

// sample_scattering_fluid (scattering.hpp:185-251) in parts, so that a step
// evaluates only what it uses:
//   locate_fluid   the cell a position samples;
//   fluid_cell     what the extension points receive, read from the cell;
//   fluid_valid    whether the fluid tetrad exists there;
//   full_sample    the cell with its tetrad and fluid-frame field (emission,
//                  scattering: once per event).
// Before, every in-grid step built the whole sample out of line -- the lookup
// with its logarithms, the tetrad's four square roots and 25 metric products --
// and passed it through local memory, though the default absorption and
// emission read the density and temperature alone; a lone packet's call spent
// about half of its 23,000 cycles on it.  In parts, with the FP32 lookup below,
// on one B200: 64 images (4.76e6 rays) 40.2 to 35.5 ms, 65,536 rays 1.17 to 1.06,
// the checkpointed forward of 16,384 rays 2.73 to 1.92, 1.1e5 disk packets 9.3
// to 6.9 and, with trace_body's deferred scattering, 2.07e6 packets 62.4 to 47.2.
// `radius` is compute_r(x, y, z, spin) of the state, which the caller has already.

// fluid_frame.hpp:28-48 on the device, times the [units] scale (raw layout only).
GRT_DEV void spherical_to_cartesian_scaled(double r, double th, double ph, double spin, const double* sv,
                                          double scale, double c[4]) {
    double st, ct, sp, cp;
    sincos(th, &st, &ct);
    sincos(ph, &sp, &cp);
    const double radial_x = cp * st, radial_y = sp * st, radial_z = ct;
    const double theta_x = (r * cp - spin * sp) * ct;
    const double theta_y = (r * sp + spin * cp) * ct;
    const double theta_z = -r * st;
    const double phi_x = (-r * sp - spin * cp) * st;
    const double phi_y = (r * cp - spin * sp) * st;
    c[0] = sv[0] * scale;
    c[1] = (radial_x * sv[1] + theta_x * sv[2] + phi_x * sv[3]) * scale;
    c[2] = (radial_y * sv[1] + theta_y * sv[2] + phi_y * sv[3]) * scale;
    c[3] = (radial_z * sv[1] + theta_z * sv[2]) * scale;
}

// Separable axes and their half-spans staged in shared memory.
struct Axes {
    const double* r;
    const double* th;
    const double* ph;
    const double* rh;
    const double* thh;
    const double* phh;
};

// The reference's lookup (scattering.hpp:41-180) with its own arithmetic: the
// cell index, or -1 outside every cell.
static __device__ __noinline__ int locate_exact(const KParams& kp, const Axes ax, double x, double y, double z,
                                                double radius) {
    const KGrid& G = kp.grid;
    int i, j, k;
    if (G.separable) {
        if (!locate_radial_sorted(ax.r, ax.rh, G.nr, radius, i)) return -1;
    }
    const double ct = fmax(-1.0, fmin(1.0, z / radius));
    const double polar = acos(ct);
    double az = atan2(radius * y - kp.a * x, radius * x + kp.a * y);
    if (az < 0.0) az += 2.0 * kPi;
    if (G.separable) {
        j = nearest_polar_sorted(ax.th, G.nth, polar);
        k = nearest_azimuth_sorted(ax.ph, G.nph, az);
        if (!within_polar_sorted(ax.th, ax.thh, j, polar) || !within_azimuth_sorted(ax.ph, ax.phh, k, az)) return -1;
    } else {
        const Grid3 g3{G.r3, G.th3, G.ph3, G.nr, G.nth, G.nph};
        if (!locate_general(g3, radius, polar, az, i, j, k)) return -1;
    }
    return (i * G.nth + j) * G.nph + k;
}

// The interval of a strictly increasing axis that holds q (axis[lo] <= q <
// axis[lo + 1]) for axis[0] <= q < axis[n - 1]: `guess`, the interval on an
// evenly spaced axis, when it does, else by search.
GRT_DEV int bracket_from(const double* axis, int n, double q, int guess) {
    guess = max(0, min(guess, n - 2));
    if (axis[guess] <= q && q < axis[guess + 1]) return guess;
    return bracket(axis, n, q);
}

// FP32 polar angle and azimuth of a position in Kerr-Schild coordinates:
// tan(theta) = sin / cos with sin^2 = (x^2 + y^2) / (r^2 + a^2), cos = z / r.
// For radii whose squares FP32 holds.
constexpr double kFp32RadiusMax = 1.0e12;
// False so close to the axis that the azimuth's arguments have no FP32 digits.
GRT_DEV bool angles_fp32(double a, double x, double y, double z, double r, float& th, float& az) {
    const float rf = static_cast<float>(r), af = static_cast<float>(a);
    th = atan2f(sqrtf(static_cast<float>(x * x + y * y)) * rf, static_cast<float>(z) * sqrtf(rf * rf + af * af));
    const float s = static_cast<float>(r * y - a * x), c = static_cast<float>(r * x + a * y);
    az = atan2f(s, c);
    return fmaxf(fabsf(s), fabsf(c)) > 1.0e-30f;
}

// locate_exact's cell on a separable grid without its logarithms and inverse
// trigonometric functions in double precision, or kUndecided: for axes of any
// spacing.  The angles and
// the logarithm are taken in FP32 (a few 1e-7 off, see kAngleMargin) and the
// radius is compared through squares; a position within the margin of a
// decision -- a midpoint between two cells, the end of a cell's acceptance --
// is left to locate_exact, about one in a thousand on a 128 x 64 x 64 grid.
// A position nearer to its cell's centre than the midpoint, by the margin, is
// inside the cell's half-width: that is 0.500001 times the larger neighbour
// gap.  Beyond the outermost centres the half-width itself decides.
constexpr int kUndecided = -2;
// Bound on the error of the FP32 angles: the arguments carry one rounding and
// the square root, quotient and atan2f a few ulp each, together below 2e-6 at
// 2 pi; five times that.  The FP32 logarithm of a ratio near 1 is far closer.
constexpr double kAngleMargin = 1.0e-5;

static __device__ __noinline__ int locate_stretched(const KGrid& G, const Axes ax, double a, double x, double y,
                                                    double z, double r) {
    if (!(r > G.r_fp32 && r < kFp32RadiusMax) || G.nr < 2 || G.nth < 2) return kUndecided;
    // radius: nearest in the logarithm.  The logarithms' rounding is far
    // inside the margins while the gap is above 1e-6.
    int i;
    if (r < ax.r[0] || r >= ax.r[G.nr - 1]) {
        i = r < ax.r[0] ? 0 : G.nr - 1;
        const double d = fabsf(logf(static_cast<float>(r / ax.r[i])));
        if (!(fabs(d - ax.rh[i]) > kAngleMargin)) return kUndecided;
        if (d > ax.rh[i]) return -1;
    } else {
        i = bracket_from(ax.r, G.nr, r, __float2int_rd((logf(static_cast<float>(r)) - G.origin[0]) * G.per[0]));
        const double rlo = ax.r[i], rhi = ax.r[i + 1];
        const double rr = r * r, mid = rlo * rhi;
        if (!(rhi - rlo > 1.0e-6 * rlo) || !(fabs(rr - mid) > 0x1p-40 * mid)) return kUndecided;
        if (rr > mid) ++i;
    }
    float thf, azf;
    if (!angles_fp32(a, x, y, z, r, thf, azf)) return kUndecided;
    const double th = thf;
    int j;
    if (th < ax.th[0] || th >= ax.th[G.nth - 1]) {
        j = th < ax.th[0] ? 0 : G.nth - 1;
        const double d = fabs(th - ax.th[j]);
        if (!(fabs(d - ax.thh[j]) > kAngleMargin)) return kUndecided;
        if (d > ax.thh[j]) return -1;
    } else {
        j = bracket_from(ax.th, G.nth, th, __float2int_rd(static_cast<float>(th - ax.th[0]) * G.per[1]));
        const double dth = (th - ax.th[j]) - (ax.th[j + 1] - th);
        if (!(fabs(dth) > 2.0 * kAngleMargin)) return kUndecided;
        if (dth > 0.0) ++j;
    }
    // azimuth: the neighbours on the circle
    const double az = azf < 0.0f ? static_cast<double>(azf) + 2.0 * kPi : static_cast<double>(azf);
    const int n = G.nph;
    const double p0 = ax.ph[0], p1 = ax.ph[n - 1];
    int k = n - 1, k2 = 0;
    double d, d2;  // distances to the centres on either side
    if (az < p0 || az >= p1) {
        d = az - p1 + (az < p0 ? 2.0 * kPi : 0.0);
        d2 = p0 - az + (az < p0 ? 0.0 : 2.0 * kPi);
        // a gap in azimuth: beyond the reach of the cells on both sides
        if (fmin(d, 2.0 * kPi - d) > ax.phh[k] + kAngleMargin && fmin(d2, 2.0 * kPi - d2) > ax.phh[k2] + kAngleMargin)
            return -1;
    } else {
        k = bracket_from(ax.ph, n, az, __float2int_rd(static_cast<float>(az - p0) * G.per[2]));
        k2 = k + 1;
        d = az - ax.ph[k];
        d2 = ax.ph[k2] - az;
    }
    // gaps of half the circle or more would make the other way round the shorter
    if (!(d + d2 < 3.0) || !(fabs(d - d2) > 2.0 * kAngleMargin)) return kUndecided;
    if (d2 < d) {
        k = k2;
        d = d2;
    }
    const double half = ax.phh[k];
    if (!(fabs(d - half) > kAngleMargin)) return kUndecided;
    if (d > half) return -1;
    return (i * G.nth + j) * G.nph + k;
}

// The same on a grid that is even in log r, theta and phi, with phi all the
// way round (KGrid::even; what the torus generators write): the cell is the
// nearest integer to the position in units of the spacing, no axis is read
// and no lane branches.  A position within KGrid::margin of a cell's edge --
// the error of the FP32 angle or logarithm in that unit, and the evenness the
// host asks of the axis -- is left to locate_exact; an edge cell ends within
// 0.500001 of the spacing, so beyond the margin a position outside is outside.
GRT_DEV int locate_even(const KGrid& G, double a, double x, double y, double z, double r) {
    if (!(r > G.r_fp32 && r < kFp32RadiusMax)) return kUndecided;
    float th, az;
    const bool known = angles_fp32(a, x, y, z, r, th, az);
    if (az < 0.0f) az += 6.2831853f;
    const float fi = (logf(static_cast<float>(r)) - G.origin[0]) * G.per[0];
    const float fj = (th - G.origin[1]) * G.per[1], fk = (az - G.origin[2]) * G.per[2];
    const float i = rintf(fi), j = rintf(fj), k = rintf(fk);
    if (!(known && fabsf(fi - i) < G.margin[0] && fabsf(fj - j) < G.margin[1] && fabsf(fk - k) < G.margin[2])) return kUndecided;
    if (i < 0.0f || i > static_cast<float>(G.nr - 1) || j < 0.0f || j > static_cast<float>(G.nth - 1)) return -1;
    int kk = static_cast<int>(k);
    kk += kk < 0 ? G.nph : kk >= G.nph ? -G.nph : 0;
    return (static_cast<int>(i) * G.nth + static_cast<int>(j)) * G.nph + kk;
}

// The cell that samples a position, or -1: the cheap rejections first.
GRT_DEV int locate_fluid(const KParams& kp, const Axes& ax, double x, double y, double z, double radius) {
    const KGrid& G = kp.grid;
    if (!G.available) return -1;
    if (!(radius > 0.0) || !isfinite(radius)) return -1;
    if (radius < G.r_reject_lo || radius > G.r_reject_hi) return -1;
    int cell = kUndecided;
    if (G.even) cell = locate_even(G, kp.a, x, y, z, radius);
    else if (G.separable) cell = locate_stretched(G, ax, kp.a, x, y, z, radius);
    if (cell == kUndecided) cell = locate_exact(kp, ax, x, y, z, radius);
    return cell;
}

// The cell's CGS record at a position, but for the fluid-frame field.  Parts
// that nothing reads are not loaded.
// RAW selects the grid layout: false -- packed (rho, T) pairs and Cartesian
// four-vectors precomputed on the host; true -- the reference's raw arrays,
// with the spherical-to-Cartesian conversion done per sample.
template <bool RAW>
GRT_DEV void fluid_cell(const KParams& kp, int cell, const double s[4], FluidCellCGS& f) {
    const KGrid& G = kp.grid;
    f.position_cm[0] = s[1] * kp.length_scale;
    f.position_cm[1] = s[2] * kp.length_scale;
    f.position_cm[2] = s[3] * kp.length_scale;
    f.coordinate_time_s = s[0] * kp.time_scale;
    if (RAW) {
        f.density_g_cm3 = G.rho_raw[cell] * kp.density_scale;
        f.temperature_k = G.T_raw[cell] * kp.temperature_scale;
        spherical_to_cartesian_scaled(G.r3[cell], G.th3[cell], G.ph3[cell], kp.a, G.vel_raw + 4 * cell,
                                      G.vel_scale, f.coordinate_four_velocity_cm_s);
    } else {
        const double2 rt = G.rho_t[cell];
        f.density_g_cm3 = rt.x * kp.density_scale;
        f.temperature_k = rt.y * kp.temperature_scale;
        const double2 u01 = G.vel[2 * cell], u23 = G.vel[2 * cell + 1];
        f.coordinate_four_velocity_cm_s[0] = u01.x;
        f.coordinate_four_velocity_cm_s[1] = u01.y;
        f.coordinate_four_velocity_cm_s[2] = u23.x;
        f.coordinate_four_velocity_cm_s[3] = u23.y;
    }
}

GRT_DEV bool fluid_finite(const FluidCellCGS& f) {
    return f.density_g_cm3 > 0.0 && isfinite(f.density_g_cm3) && isfinite(f.temperature_k);
}

// The tetrad at a position in `cell` (f from fluid_cell) and the fluid-frame
// field in it; false where there is no tetrad.
template <bool RAW, bool UNROLL = false>
GRT_DEV bool fluid_frame(const KParams& kp, int cell, double x, double y, double z, double radius, FluidCellCGS& f,
                         double e[4][4]) {
    const KGrid& G = kp.grid;
    double cm[4];
    if (RAW) {
        spherical_to_cartesian_scaled(G.r3[cell], G.th3[cell], G.ph3[cell], kp.a, G.mag_raw + 4 * cell,
                                      G.mag_scale, cm);
    } else {
        const double2 b01 = G.mag[2 * cell], b23 = G.mag[2 * cell + 1];
        cm[0] = b01.x; cm[1] = b01.y; cm[2] = b23.x; cm[3] = b23.y;
    }
    MetricAt m;
    ks_metric_from_r(x, y, z, radius, kp.a, kp.M, m);
    if (!build_tetrad<UNROLL>(m.g, f.coordinate_four_velocity_cm_s, e)) return false;
    f.magnetic_gauss[0] = -metric_dot(m.g, e[0], cm);
#pragma unroll
    for (int axis = 1; axis < 4; ++axis) f.magnetic_gauss[axis] = metric_dot(m.g, e[axis], cm);
    return true;
}

// The whole sample of `cell` at a position; false where the density, the
// temperature or the tetrad is not valid.
template <bool RAW>
static __device__ __noinline__ bool full_sample(const KParams& kp, int cell, double t, double x, double y, double z,
                                                double radius, FluidSample* out) {
    const double s[4] = {t, x, y, z};
    out->cell = cell;
    fluid_cell<RAW>(kp, cell, s, out->fluid);
    return fluid_finite(out->fluid) && fluid_frame<RAW>(kp, cell, x, y, z, radius, out->fluid, out->e);
}

// full_sample's verdict alone.
template <bool RAW>
static __device__ __noinline__ bool full_sample_valid(const KParams& kp, int cell, double t, double x, double y,
                                                      double z, double radius) {
    FluidSample fs;
    return full_sample<RAW>(kp, cell, t, x, y, z, radius, &fs);
}

// Whether the tetrad of four-velocity u exists at a position (build_tetrad's
// verdict).  u.u = -u0^2 + |u|^2 + 2H (l.u)^2 here carries a few roundings of
// its terms, so one that is negative by a thousandth of their sum is negative
// in build_tetrad's arithmetic too; the normalised e0 then stays below 32, and
// the norms that build_tetrad tests -- Schur complements of
// delta_ij + 2H l_i l_j + e0_i e0_j, at least 1 -- keep nine digits.  Anything
// closer to the light cone is left to build_tetrad itself.
GRT_DEV bool tetrad_certain(double x, double y, double z, double r, double a, double M, const double u[4]) {
    const double ar = a * a + r * r, az = a * z, r2 = r * r;
    const double lu = u[0] + ((r * x + a * y) * u[1] + (r * y - a * x) * u[2]) * rcp_rn_box(ar) + z * u[3] * rcp_rn_box(r);
    const double h = 2.0 * M * r2 * r * rcp_rn_box(r2 * r2 + az * az) * (lu * lu);
    const double t2 = u[0] * u[0], s2 = u[1] * u[1] + u[2] * u[2] + u[3] * u[3] + h;
    return s2 - t2 < -1.0e-3 * (s2 + t2) && t2 < 1.0e300 && r > 1.0e-6 && r < 1.0e30 && fabs(a) < 1.0e30;
}

// The fluid at a position, as the extension points and the scattering draw
// receive it: the cell, or -1 when nothing is sampled (scattering.hpp:185-251's
// false).  The fluid-frame field costs the whole tetrad; it is straight-line
// code that the compiler drops while no extension point reads magnetic_gauss.
template <bool RAW>
GRT_DEV int sample_fluid(const KParams& kp, const Axes& ax, const double s[8], double radius, FluidCellCGS& f) {
    const int cell = locate_fluid(kp, ax, s[1], s[2], s[3], radius);
    if (cell < 0) return -1;
    fluid_cell<RAW>(kp, cell, s, f);
    if (!fluid_finite(f)) return -1;
    if (!(radius > kp.grid.r_certain) &&
        !tetrad_certain(s[1], s[2], s[3], radius, kp.a, kp.M, f.coordinate_four_velocity_cm_s) &&
        !full_sample_valid<RAW>(kp, cell, s[0], s[1], s[2], s[3], radius))
        return -1;
    double e[4][4];
    fluid_frame<RAW, true>(kp, cell, s[1], s[2], s[3], radius, f, e);
    return cell;
}

// ---------------------------------------------------------------------------
// Scattering and packet generation
// ---------------------------------------------------------------------------
constexpr double kProtonMassCgs = 1.67262192369e-24;   // scattering.hpp:256
constexpr double kSigmaThomsonCgs = 6.6524587158e-25;  // scattering.hpp:257

// State a scattering event may change, passed by copy to the out-of-line
// scatter_packet so the caller's state never has its address taken (which
// would keep it in local memory for the whole trace loop).
struct ScatterState {
    double s[8];
    double I[4];
};

// maybe_scatter_photon (scattering.hpp:259-313) in two parts.  scatter_drawn is the
// part every sampled step takes, inline: the Thomson optical depth over the
// proposed step and the first draw; it says whether the packet scatters.
GRT_DEV bool scatter_drawn(double dl, double length_scale, const FluidCellCGS& fluid, Philox& rng) {
    const double path_cm = dl * length_scale;
    const double ne = fluid.density_g_cm3 / kProtonMassCgs;
    const double tau = kSigmaThomsonCgs * ne * path_cm;
    const double prob = 1.0 - exp(-tau);
    return !(rng.drand() >= prob);  // the reference's rejection test, NaN included
}

// The rest, out of line and only for a packet that scatters: the tetrad of its
// cell (which exists: the step sampled it), the isotropic
// fluid-frame direction (two more draws), the new covariant momentum and the
// albedo weights; false leaves the state as it was.  The stream of (photon,
// step) is opened again and scatter_drawn's draw passed over, so that no
// generator state waits with the packet.  The tetrad in its rolled form: the
// straight-line one, run by one warp iteration in five, drove the step loop
// out of the instruction cache (2.07e6 packets 42.4 ms against 38.9; with
// Philox's rounds rolled too 38.7).
template <bool RAW>
static __device__ __noinline__ bool scatter_packet(const KParams& kp, ScatterState* st, int cell, double radius,
                                                   uint64_t id, int64_t step) {
    Philox rng(kp.seed, id, static_cast<uint32_t>(step));
    rng.drand();
    double* s = st->s;
    double* I = st->I;
    const double albedo = kp.albedo;
    FluidCellCGS f;
    fluid_cell<RAW>(kp, cell, s, f);
    MetricAt m;
    ks_metric_from_r(s[1], s[2], s[3], radius, kp.a, kp.M, m);
    double e[4][4];
    build_tetrad(m.g, f.coordinate_four_velocity_cm_s, e);
    double E = 0.0;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) E -= s[4 + mu] * e[0][mu];
    if (!(E > 0.0) || !isfinite(E)) return false;
    const double mu_c = 2.0 * rng.drand() - 1.0;
    const double dphi = 2.0 * kPi * rng.drand();
    const double tr = sqrt(fmax(0.0, 1.0 - mu_c * mu_c));
    double sn, cs;
    det_sincos(dphi, &sn, &cs);  // the oracle's sin/cos bit for bit (grt_sincos.h)
    const double dx = tr * cs, dy = tr * sn, dz = mu_c;
    double w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = e[0][q] + dx * e[1][q] + dy * e[2][q] + dz * e[3][q];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double pq = 0.0;
#pragma unroll
        for (int nu = 0; nu < 4; ++nu) pq += m.g[q][nu] * w[nu];
        s[4 + q] = E * pq;
    }
    I[0] *= albedo;
    I[1] *= 0.5 * albedo;
    I[2] *= 0.5 * albedo;
    I[3] *= 0.25 * albedo;
    return true;
}

// GenerateBlackbody (photon_generation.hpp:99-124): Planck spectrum as a
// mixture of Gamma(4, n) with weights 1/n^4; the four product draws are taken
// in order.
static __device__ __noinline__ bool generate_blackbody(const FluidCellCGS& cell, Philox& rng, int packets, double energy,
                                double& nu, double& E) {
    if (!(cell.temperature_k > 0.0)) return false;
    const double inverse_zeta4 = 0.9239384029215902;
    const double choose = rng.drand();
    double cumulative = 0.0;
    int m = 1;
    for (; m < 64; ++m) {
        const double n = static_cast<double>(m);
        cumulative += inverse_zeta4 / (n * n * n * n);
        if (choose <= cumulative) break;
    }
    const double d1 = rng.drand(), d2 = rng.drand(), d3 = rng.drand(), d4 = rng.drand();
    const double product = fmax(1.0e-300, d1 * d2 * d3 * d4);
    const double x = -log(product) / static_cast<double>(m);
    nu = x * 2.0836619123327576e10 * cell.temperature_k;
    E = energy / static_cast<double>(packets);
    return isfinite(nu) && nu > 0.0;
}

// GeneratePowerLaw (photon_generation.hpp:126-143)
static __device__ __noinline__ bool generate_power_law(Philox& rng, int packets, double slope, double nu_min, double nu_max,
                                double energy, double& nu, double& E) {
    const double draw = rng.drand();
    if (fabs(slope - 1.0) < 1.0e-12) {
        nu = nu_min * pow(nu_max / nu_min, draw);
    } else {
        const double ex = 1.0 - slope;
        const double lo = pow(nu_min, ex);
        const double hi = pow(nu_max, ex);
        nu = pow(lo + draw * (hi - lo), 1.0 / ex);
    }
    E = energy / static_cast<double>(packets);
    return isfinite(nu) && nu > 0.0;
}

// ---------------------------------------------------------------------------
// Camera (integrate_cart_ks.hpp:96-130); the plane basis is precomputed on the host.
// ---------------------------------------------------------------------------
GRT_DEV int camera_crossing(const KImage& im, const double s[8], double& u, double& v) {
    const double pc = s[1] * im.cam_n[0] + s[2] * im.cam_n[1] + s[3] * im.cam_n[2];
    if (pc < im.cam_D) return 0;
    const double rel0 = s[1] - im.cam_D * im.cam_n[0];
    const double rel1 = s[2] - im.cam_D * im.cam_n[1];
    const double rel2 = s[3] - im.cam_D * im.cam_n[2];
    u = rel0 * im.cam_th[0] + rel1 * im.cam_th[1] + rel2 * im.cam_th[2];
    v = rel0 * im.cam_ph[0] + rel1 * im.cam_ph[1] + rel2 * im.cam_ph[2];
    const bool inside = fabs(u) <= 0.5 * im.cam_W && fabs(v) <= 0.5 * im.cam_H;
    return inside ? 1 : -1;
}

static __device__ __noinline__ double camera_observer_energy_at(double a, double M, double x, double y, double z,
                                                                double pt) {
    MetricAt m;
    ks_metric(x, y, z, a, M, m);
    if (!(m.g[0][0] < 0.0)) return 0.0;
    const double u0 = 1.0 / sqrt(-m.g[0][0]);
    return -pt * u0;
}

GRT_DEV double camera_observer_energy(const KParams& kp, const double s[8]) {
    return camera_observer_energy_at(kp.a, kp.M, s[1], s[2], s[3], s[4]);
}

}  // namespace dev
}  // namespace grt
