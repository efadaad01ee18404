// Host-side launch interface between the C ABI (grt_api.cu) and the kernel
// translation units.  Internal to the library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#include "grt_kparams.h"

namespace grt {

struct InitImageArgs {
    KPhotons ph;
    unsigned long long offset;     // first photon slot written
    unsigned long long nx, ny;
    unsigned long long row0, nrows;  // pixel rows [row0, row0 + nrows) of the ny-row screen
    unsigned long long id_offset;
    double W, H;
    double cx, cy, cz;
    double th_hat[3], ph_hat[3];
    double a, M;
    double dlambda0;               // initial_step * camera_distance (forward: * back distance)
    // line-of-sight forward rays: start on the plane -back * n, aimed along +n,
    // ImageForward, I = 0, frequency nu0, emission_frame_energy = -p_t
    int forward;
    double bx, by, bz;             // -back * n
    double nu0;
    // the reference's random screen instead of pixel centres: (u, v) from
    // Philox keyed by (seed, photon id), see kScreenDomain
    int random_screen;
    unsigned long long seed;
};

// initialize_photons_disk (initialize_photons.hpp:173-327): one photon per
// packet; the packet's cell comes from the prefix sum of per-cell counts.
struct DiskInitArgs {
    KPhotons ph;
    unsigned long long n;                // packets = offsets[ncell]
    const unsigned long long* offsets;   // [ncell + 1]
    unsigned long long ncell;
    const double* pos;                   // [ncell][3] Cartesian KS cell positions (host libm)
    const double2* rho_t;                // [ncell] (rho, T) code units
    const double2* vel;                  // [2 * ncell] Cartesian u^mu * velocity scale
    const double2* mag;                  // [2 * ncell] Cartesian b^mu * magnetic scale
    double density_scale, temperature_scale, length_scale, time_scale;
    double a, M;
    int generator;
    int pad;
    double energy, pl_slope, nu_min, nu_max, nu_custom;
    uint64_t seed;                       // scattering seed + rank (Philox key)
    unsigned long long id_offset;
    double dlambda0;                     // initial_step (disk mode: unscaled)
};

// One image of a products launch: its photon slots, screen and output buffers.
struct ProductsImage {
    unsigned long long offset, n;  // photon slots [offset, offset + n)
    unsigned long long nx, ny;
    double W, H;
    double* image;                 // [4][ny][nx] (I, Q, U, V), zeroed before the launch
    double* spectrum;              // [bins], zeroed
    unsigned long long* arrived;   // [1], zeroed
    unsigned block0;               // first block of this image in the launch
    unsigned pad;
};

// build_observation_products over up to kProductsMaxImages images in one
// launch; each block belongs to one image.
constexpr int kProductsMaxImages = 32;
constexpr unsigned long long kProductsSharedBins = 4096;  // spectrum privatised in shared memory up to this
struct ProductsSet {
    KPhotons ph;
    unsigned long long bins;
    double spec_min, spec_max, log_min, log_max;
    int nimages;
    unsigned blocks;
    ProductsImage img[kProductsMaxImages];
};

// Queue order of n rays at screen positions (u, v) in a W x H window: by cells
// of a 2^log_side x 2^log_side screen grid (log_side <= 8).
struct ScreenOrderArgs {
    const double *u, *v;           // [n]
    double W, H;
    unsigned long long n;          // < 2^32
    int log_side;
    int pad;
    unsigned *cell, *rank, *order; // [n]
    unsigned* count;               // [4^log_side + 1]
};

// Strided gather of an output step's photon fields (write_output_step):
// elements src[k][j * stride], j < count, of field k packed at dst + dst_off[k].
constexpr int kGatherMaxFields = 40;  // a selection's fields, "all" after 20 names included
struct GatherArgs {
    const void* src[kGatherMaxFields];
    unsigned long long dst_off[kGatherMaxFields];
    int item[kGatherMaxFields];  // element bytes: 8 or 1
    int nfields;
    int pad;
    unsigned long long count, stride;
    unsigned char* dst;
};

// Buffers of the adjoint pass (grt_adjoint.cu).
struct AdjointArgs {
    double* ckpt;              // [n][cap][16] ray state after emission and every K calls
    int cap;                   // checkpoints per ray
    int K;                     // calls between checkpoints
    int* nckpt;                // [n] checkpoints written
    long long* call0;          // [n] calls taken when checkpoint 0 was written (-1: never emitted)
    int* overflow;             // checkpoint/tape capacity errors
    const double* dL_dI;       // [ny][nx] dL/d(image_I)
    unsigned long long nx, ny;
    double W, H;
    double* g_abs;             // [ncell] dL/dm_abs (accumulated)
    double* g_emis;            // [ncell] dL/dm_emis
    double* tape;              // [threads][K][6] of a recomputed segment
    // the forward pass's own record of each ray's transfer updates: field f of
    // entry e of queue position q at full[(e * 6 + f) * n + q]
    double* full;
    int full_cap;              // entries a ray can keep (0: no record)
    int* nfull;                // [n] entries kept, -1 when the ray had more
    int* over;                 // rays with nfull -1
};

// Camera plane basis of integrate_cart_ks.hpp:97-107 with host libm, plus the
// image's coefficients.
inline KImage make_kimage(double theta, double phi, double distance, double width, double height, double nu_custom,
                          double kappa, double jcoef) {
    KImage im{};
    im.cam_D = distance;
    im.cam_W = width;
    im.cam_H = height;
    im.cam_n[0] = std::sin(theta) * std::cos(phi);
    im.cam_n[1] = std::sin(theta) * std::sin(phi);
    im.cam_n[2] = std::cos(theta);
    im.cam_th[0] = std::cos(theta) * std::cos(phi);
    im.cam_th[1] = std::cos(theta) * std::sin(phi);
    im.cam_th[2] = -std::sin(theta);
    im.cam_ph[0] = -std::sin(phi);
    im.cam_ph[1] = std::cos(phi);
    im.cam_ph[2] = 0.0;
    im.nu_custom = nu_custom;
    im.kappa = kappa;
    im.jcoef = jcoef;
    return im;
}

// Idle lanes before a warp takes new photons, when the caller set no launch
// shape.  Image rays of one tile need nearly the same calls: a warp that waits
// for its whole tile (32) keeps its lanes on one path, a warp refilled early
// mixes rays on their first and last calls.  Trace ms at 8 / 32: 64 images
// (4.76e6 rays) 50.3 / 40.0, 509 x 283 random screen 2.61 / 2.20, 256 x 256
// (all rays resident) 1.20 / 1.18.  Disk packets live from a few calls to
// hundreds, and waiting for the longest leaves the warp empty: at 1 / 4 / 8,
// 2.07e6 packets 38.2 / 38.0 / 39.4 (and more than twice that at 32).
inline int default_refill(int image_mode) { return image_mode ? 32 : 4; }

// Whether the spin a and mass M admit the reciprocal-quotient right-hand side
// (KParams::rcp_ok): |a| = 0 or in [2^-20, 2], M in [2^-20, 2^20].
inline int rcp_params_ok(double a, double M) {
    const double fa = std::fabs(a);
    const bool a_ok = fa == 0.0 || (fa >= std::ldexp(1.0, -20) && fa <= 2.0);
    const bool m_ok = M >= std::ldexp(1.0, -20) && M <= std::ldexp(1.0, 20);
    return a_ok && m_ok ? 1 : 0;
}

// The FP32 lookup's constants from the host's copy of separable axes.  Even:
// every value within 1e-6 of its place in units of the spacing, phi all the
// way round.  The FP32 error (4e-6 bounds angle, logarithm and its rounding
// in [0, 2 pi]; the logarithm's grows with its size) must stay below a
// hundredth of the spacing, and is taken five times over.
inline void set_axis_lookup(KGrid& g, const double* ra, const double* ta, const double* pa) {
    const double* axes[3] = {ra, ta, pa};
    const int n[3] = {g.nr, g.nth, g.nph};
    bool even = true;
    for (int q = 0; q < 3; ++q) {
        auto at = [&](int i) { return q == 0 ? std::log(axes[q][i]) : axes[q][i]; };
        const double lo = at(0), hi = at(n[q] - 1);
        const double per = n[q] > 1 && hi > lo ? (n[q] - 1) / (hi - lo) : 0.0;
        double err = 4.0e-6 * per;
        if (q == 0) err = (1.0e-6 + 3.0e-7 * std::fmax(std::fabs(lo), std::fabs(hi))) * per;
        g.origin[q] = static_cast<float>(lo);
        g.per[q] = static_cast<float>(per);
        // the float product is itself rounded: an index of n carries n 2^-23
        err = 5.0 * (err + 2.0e-6 + n[q] * 2.4e-7);
        g.margin[q] = static_cast<float>(0.5 - err);
        even = even && per > 0.0 && err < 0.05;
        if (q == 2) even = even && std::fabs(n[q] - per * 6.283185307179586) < 1.0e-6;
        for (int i = 0; i < n[q] && even; ++i) even = std::fabs((at(i) - lo) * per - i) < 1.0e-6;
    }
    g.even = even ? 1 : 0;
}

// Radius below which the FP32 lookups leave a position to the reference's
// arithmetic.  The Kerr-Schild radius carries a relative error of about
// 2^-53 (a / r)^2 and the reference's polar angle acos(z / r) near the axis the
// root of twice that: at r = a / 100 2e-6, a fifth of the lookups' margins (at a / 2e5
// ten times them).  Also where FP32 holds the squares.
inline double fp32_lookup_radius(double a) { return std::fmax(1.0e-12, 0.01 * std::fabs(a)); }

// Stage slots of an RK45 block: the disk mode's rolled error norm keeps the
// state in a sixth (rk45_attempt).
__host__ __device__ constexpr int stage_slots(bool disk) { return disk ? 6 : 5; }

// Dynamic shared memory of a trace launch: the stage slots for RK45 (7 doubles
// per thread and slot) plus the separable axes and their half-spans
// (2*(nr+nth+nph)).
inline size_t dev_trace_smem_bytes(int integrator, int threads, bool separable, int nr, int nth, int nph,
                                   bool disk = false) {
    size_t n = integrator == 1 ? static_cast<size_t>(stage_slots(disk) * 7) * threads : 0;
    if (separable) n += 2 * static_cast<size_t>(nr + nth + nph);
    return n * sizeof(double);
}

// Adjoint pass: checkpointed forward trace, the sweep of the rays it recorded and
// the reverse pass of the others, 128-thread blocks.
cudaError_t launch_adjoint_forward(const KParams& kp, const AdjointArgs& aa, int blocks, size_t smem,
                                   cudaStream_t stream);
cudaError_t launch_adjoint_sweep(const KParams& kp, const AdjointArgs& aa, cudaStream_t stream);
cudaError_t launch_adjoint_reverse(const KParams& kp, const AdjointArgs& aa, int blocks, size_t smem,
                                   cudaStream_t stream);

// Persistent trace launches (grt_trace_inst.cu): `blocks` blocks of 128
// threads; blocks_per_sm in {2, 3, 4} picks the register cap (255 / 170 /
// 128); leg 0 traces whole rays, legs 1 and 2 the backward leg and the rest
// of image-mode rays, leg 3 whole disk-mode rays (trace_body).
cudaError_t launch_trace_fp64_leg0(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                   cudaStream_t stream);
cudaError_t launch_trace_fp64_leg1(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                   cudaStream_t stream);
cudaError_t launch_trace_fp64_leg2(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                   cudaStream_t stream);
cudaError_t launch_trace_mixed_leg0(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                    cudaStream_t stream);
cudaError_t launch_trace_mixed_leg1(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                    cudaStream_t stream);
cudaError_t launch_trace_mixed_leg2(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                    cudaStream_t stream);
cudaError_t launch_trace_fp64_leg3(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                   cudaStream_t stream);
cudaError_t launch_trace_mixed_leg3(const KParams& kp, int integrator, int blocks_per_sm, int blocks, size_t smem,
                                    cudaStream_t stream);
// Packet generation between the backward-leg and forward-leg launches
// (photons with calls_carry < 0), one thread per queue index; smem holds the
// staged axes (dev_trace_smem_bytes with integrator 0).
cudaError_t launch_generate_pending(const KParams& kp, int sm_count, size_t smem, cudaStream_t stream);
// sm_count * launched blocks of the form's (FP64 or mixed) kernel for `leg`
// compiled for blocks_per_sm (launched <= blocks_per_sm).
cudaError_t launch_trace(const KParams& kp, bool mixed, int leg, int integrator, int sm_count, int blocks_per_sm,
                         int launched, size_t smem, cudaStream_t stream);
cudaError_t launch_init_image(const InitImageArgs& args, cudaStream_t stream);
cudaError_t launch_screen_order(const ScreenOrderArgs& a, cudaStream_t stream);
cudaError_t launch_init_disk(const DiskInitArgs& a, cudaStream_t stream);
// Fills block0 / blocks of `set` and launches it.
cudaError_t launch_image_products(ProductsSet& set, cudaStream_t stream);
cudaError_t launch_gather_fields(const GatherArgs& a, int sm_count, cudaStream_t stream);
cudaError_t launch_count_terminated(const uint8_t* term, unsigned long long n, unsigned long long* out,
                                    int sm_count, cudaStream_t stream);

}  // namespace grt
