// Parameters, outputs and records of the photon propagation kernels
// (mpf_exact.cuh: the reference's float64 order; mpf_fast.cuh: FP32 gathers):
// RK4 null-geodesic integration with CIC/TSC interpolation
// (src/integrator.h:409-445 dphotondl, :648-824 integrate with a stop
// criterion), the infinitesimal lensing Jacobian fused into the step
// (src/lensing.h:399-472) and the per-surface reduction of the map driver
// (src/hmaps.h:612-676).
//
// Fusing the Jacobian: the reference sums, over trajectory points i,
//     a(d) += (d - chi_i) chi_i / d * H_i * dr_i
// after the ray is finished, for each surface distance d.  Here the two
// d-independent sums S1 = sum chi H dr and S2 = sum chi^2 H dr accumulate
// during the step, and a(d) = S1 - S2 / d is read at the crossing of each
// surface, at the last point with chi <= d (the reference's upper_bound).
// The result equals the reference's up to float64 rounding of the
// re-association.
#pragma once
#include "mpf_device.cuh"

namespace mpf {

constexpr int kMaxPlanes = 16;
constexpr int kPhotonFields = 28;
constexpr int kPlaneFields = 20;
// Source mode (catalogue root-finder): one record per ray at its own stop
// radius: the 20 surface fields, then dtdl dxdl dydl dzdl interpolated at the
// radius (20-23) and the launch point's a, phi, dxdl, dydl, dzdl (24-28).
constexpr int kSourceFields = 32;
// Wide surface records (bundle Jacobian): the 20 surface fields, dtdl dxdl
// dydl dzdl interpolated at the surface (20-23) and whether the kept
// trajectory reached the surface at all (24).
constexpr int kWideFields = 32;

enum StopKind { STOP_REDSHIFT = 0, STOP_R = 1, STOP_LAMBDA = 2, STOP_T = 3, STOP_A = 4, STOP_PLANE = 5, STOP_S = 6 };

struct DevCosmo {
    const double* t;
    const double* a;
    const double* dadt;
    int n;
    // fast-mode search accelerator: lut[k] = upper_bound(t, t0 + k / lut_scale),
    // and per-interval slopes of a and da/dt
    const int* lut;
    int nlut;
    double t0, lut_scale;
    const double* slope_a;
    const double* slope_dadt;
    // per interval k (t[k], t[k+1]): slope of da/dt and width t[k+1] - t[k], in
    // FP32 (the RK4 stages' increments of da/dt from the step's start)
    const float2* seg;
};

struct PropParams {
    double length;
    double stop_ref;
    double ki[3];
    double planes[kMaxPlanes];
    long long max_steps;
    unsigned nsteps;
    int order;
    int stop_kind;
    int nplanes;
    int jacobian;
    // source mode: per-ray stop radius; the launch record is the start point
    // and a unit direction (Integrator::launch, (phi, theta) form)
    const double* ray_stop;
    // per-ray surface values (n x nplanes; the last one is the stop value), or null
    const double* ray_planes;
    // surface records of kWideFields doubles instead of kPlaneFields
    int wide;
    // launch records give the start point and the direction itself (the
    // bundle photons of Integrator::launch(photon, count, angle, rotation),
    // whose direction is not renormalised before integrate)
    int direct;
    // Order = -1 of the reference: every gather gives the homogeneous field
    // (a = 1, the rest 0).  1: the FLRW reference ray of the rays driver,
    // integrated on a uniform octree of level hom_level (every cell is of
    // that level); 2: the Born ray of hmaps / catalogues (hmaps.h:706-712,
    // catalogues.h:670-673), on the octree itself (its levels set the steps,
    // its field the Jacobian), with the Jacobian at each surface's value (a
    // radius) and, for a surface the ray never reaches, at its last point.
    // Mode 1: exact kernel only; mode 2: both kernels (the fast kernel's
    // Born instantiations).
    int homogeneous;
    int hom_level;
    // per-ray plane normals for the stop criterion "plane" with per-ray
    // surfaces (n x nplanes x 3; the last one is the stop plane's), or null
    const double* ray_ki;
    // observer velocity (parameters v0x v0y v0z, hmaps.h:80-84), read when the
    // octree carries a velocity field (integrator.h:537-538, 707-708)
    double vobs[3];
};

struct PropOut {
    long long* steps;      // n
    double* final_rec;     // n x 28, or null
    double* plane_rec;     // n x nplanes x 20, or null
    unsigned* status;      // bit 0: a ray hit max_steps
    double* traj;          // n x traj_cap x 28: every trajectory point, or null
    long long traj_cap;    // points kept per ray (status bit 3 when a ray has more)
};

// Utility::interpolate (src/utility.h:441-449)
__device__ __forceinline__ double interpolate(double x0, const double* __restrict__ x, const double* __restrict__ y, int n)
{
    int first = 0, count = n;
    while (count > 0) {
        const int step = count >> 1, it = first + step;
        if (!(x0 < __ldg(x + it))) { first = it + 1; count -= step + 1; }
        else count = step;
    }
    int i = first;
    i += (n > 1) * ((i <= 0) - (i >= n));
    if (n > 1) {
        const double xi = __ldg(x + i), xm = __ldg(x + i - 1), yi = __ldg(y + i), ym = __ldg(y + i - 1);
        return ym + ((yi - ym) * (x0 - xm) / (xi - xm));
    }
    return (n > 0) ? __ldg(y) : 0.0;
}

// Trajectory record, named as the reference's Photon<double, 3>.
struct Rec {
    double a, t, x, y, z, k0, k1, k2, k3;
    double level, ah, rho, phi, dx, dy, dz, dt, dphidl, lap, red, ds2, err, isw, iswold, chi, lambda, s, index;
};

__device__ __forceinline__ void write_rec(double* o, const Rec& r)
{
    const double v[kPhotonFields] = {r.a, r.t, r.x, r.y, r.z, r.k0, r.k1, r.k2, r.k3, r.level, r.ah, r.rho, r.phi, r.dx,
                                     r.dy, r.dz, r.dt, r.dphidl, r.lap, r.red, r.ds2, r.err, r.isw, r.iswold, r.chi,
                                     r.lambda, r.s, r.index};
#pragma unroll
    for (int k = 0; k < kPhotonFields; ++k) o[k] = v[k];
}

constexpr double kC = 299792458.0;

// The lanes of a warp that trace one ray together when it has `rays` of them
// and a Jacobian, whose six gathers they share out.
__host__ __device__ __forceinline__ int rays_to_lanes(int rays) { return (rays <= 5) ? 6 : (rays <= 10) ? 3 : (rays <= 16) ? 2 : 1; }

}  // namespace mpf
