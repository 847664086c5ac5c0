// Throughput mode of the propagation kernel.
//
// Same algorithm as propagate_one (mpf_exact.cuh: src/integrator.h:648-824 with the
// fused src/lensing.h:399-472 Jacobian), reorganised for the GB300's
// arithmetic balance:
//
//  * Stencil records.  Every cell carries, in HBM, its 27 same-level
//    neighbours resolved with the reference's lookup semantics, a mask of the
//    ones at exactly its level, its level / children flags and the cell whose
//    stencil a TSC gather ends at after the restarts at coarser neighbours
//    (simplehyperoctree.h:1532-1537; built on the GPU at upload,
//    mpf_octree.cu).  A TSC or CIC gather is then one or two 128-byte record
//    loads plus the payload loads.
//    The deepest cell of a point near a known cell is read from that cell's
//    record, so the RK stages, the post-step gather and the six Jacobian
//    gathers of a step do no octree walks in the common case.
//  * FP64 is kept for the RK4 state, the RHS, the affine parameter, redshift
//    and distances.  Cell coordinates use exact power-of-two scalings (no
//    divisions), TSC weights and field accumulation are FP32, the cosmology
//    search uses a uniform index table.
#pragma once
#include "mpf_fp64.cuh"
#include "mpf_propagate.cuh"

namespace mpf {

constexpr unsigned kFullMask = (1u << 27) - 1u;

// Launch shape of the persistent kernel: threads per block and the minimum
// resident blocks per SM promised to the register allocator.  128 x 2 (up to
// 255 registers, 8 warps per SM) measured fastest on the AMR and medium
// octrees, ahead of 128 x 3 (168 registers, spills) and 128 x 4.
// Overridable at build time for tuning sweeps.
#ifndef MPF_FAST_THREADS
#define MPF_FAST_THREADS 128
#endif
#ifndef MPF_FAST_MINB
#define MPF_FAST_MINB 2
#endif
constexpr int kFastThreads = MPF_FAST_THREADS;

// Utility::interpolate with the uniform index table (same bracketing interval
// as the reference's upper_bound; slope precomputed per interval).
__device__ __forceinline__ double interp_fast(const DevCosmo& C, double x0, const double* __restrict__ y,
                                              const double* __restrict__ slope)
{
    int i;
    if (x0 < C.t0) {
        i = 0;
    } else {
        const double kk = (x0 - C.t0) * C.lut_scale;
        const int k = (kk < (double)C.nlut) ? (int)kk : C.nlut;
        i = __ldg(C.lut + k);
        while (i < C.n && !(x0 < __ldg(C.t + i))) ++i;
    }
    const int n = C.n;
    i += (n > 1) * ((i <= 0) - (i >= n));
    if (n <= 1) return (n > 0) ? __ldg(y) : 0.0;
    return __ldg(y + i - 1) + __ldg(slope + i - 1) * (x0 - __ldg(C.t + i - 1));
}

// Upper-bound position of x0 in the cosmology table (the bracket
// Utility::interpolate uses), from the uniform index table.
__device__ __forceinline__ int bracket_lut(const DevCosmo& C, double x0)
{
    if (x0 < C.t0) return 0;
    const double kk = (x0 - C.t0) * C.lut_scale;
    const int k = (kk < (double)C.nlut) ? (int)kk : C.nlut;
    int i = __ldg(C.lut + k);
    while (i < C.n && !(x0 < __ldg(C.t + i))) ++i;
    return i;
}

// Utility::interpolate with the bracket carried from the previous call: a
// ray's conformal time moves by much less than a table interval between two
// calls, so `first` (the upper bound of x0) is re-checked, not searched.
__device__ __forceinline__ double interp_cached(const DevCosmo& C, double x0, const double* __restrict__ y,
                                                const double* __restrict__ slope, int& first)
{
    const int n = C.n;
    while (first < n && !(x0 < __ldg(C.t + first))) ++first;
    while (first > 0 && x0 < __ldg(C.t + first - 1)) --first;
    int i = first;
    i += (n > 1) * ((i <= 0) - (i >= n));
    if (n <= 1) return (n > 0) ? __ldg(y) : 0.0;
    return __ldg(y + i - 1) + __ldg(slope + i - 1) * (x0 - __ldg(C.t + i - 1));
}

__device__ __forceinline__ void tsc_w3(float f, float* w)
{
    const float m = 0.5f - f, p = 0.5f + f;
    w[0] = 0.5f * m * m;
    w[1] = 0.75f - f * f;
    w[2] = 0.5f * p * p;
}

// integer coordinates at level L and the offset of the point from its cell
// centre in cell units (exact scaling by 2^L / EXTENT)
__device__ __forceinline__ void point_cell(int L, double x, double y, double z, uint32_t* c, float* fd)
{
    const double s = pow2(L - kLevelShift);   // 2^L / EXTENT, exact
    const double u[3] = {(x + 2.0) * s, (y + 2.0) * s, (z + 2.0) * s};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double f = floor(u[d]);
        c[d] = (f > 0.0) ? (uint32_t)(uint64_t)f : 0u;
        fd[d] = (float)(u[d] - f) - 0.5f;
    }
}

// level | has_children << 8 of a cell
__device__ __forceinline__ int rec_flags(const DevTree& T, int cell) { return __ldg(&T.stencil[8 * (size_t)cell + 7].y) & 511; }
__device__ __forceinline__ int rec_entry(const DevTree& T, int cell, int j)
{
    return __ldg(reinterpret_cast<const int*>(T.stencil + 8 * (size_t)cell) + j);
}

// Build-time diagnostics (-DMPF_DIAG=1): counts of the rare paths, read by
// the launcher when MPF_STATS is set.  [0] gather restarts at a coarser
// cell, [1] full walks from the top grid.
#if MPF_DIAG
__device__ unsigned long long g_diag[4];
#define MPF_DIAG_COUNT(k) atomicAdd(&g_diag[k], 1ull)
#else
#define MPF_DIAG_COUNT(k) ((void)0)
#endif

// Out-of-line slow paths (reference semantics with full walks), single copies
// so that the hot loop stays small in the instruction cache.
static __device__ __noinline__ Field7 tsc_slow(const DevTree& T, double x, double y, double z, int need_all)
{
    return tsc(T, x, y, z, need_all != 0);
}
static __device__ __noinline__ Field7 cic_slow(const DevTree& T, double x, double y, double z, int need_all)
{
    return cic(T, x, y, z, need_all != 0);
}
static __device__ __noinline__ Found locate_slow(const DevTree& T, double x, double y, double z) { return locate(T, x, y, z); }
// the 7 fields and the velocity, full walk (velocity-field octrees)
static __device__ __noinline__ Field7 vel_slow(const DevTree& T, int order, double x, double y, double z, float* v)
{
    return gather_vel(T, order, x, y, z, v);
}

// A point given by its float64 coordinates.
struct PosAt {
    double x, y, z;
    __device__ __forceinline__ double px() const { return x; }
    __device__ __forceinline__ double py() const { return y; }
    __device__ __forceinline__ double pz() const { return z; }
};

// A located point: its deepest cell, that cell's level and integer
// coordinates, and the point's offset from the cell's centre in cell units.
struct Spot {
    int cell;
    int level;
    uint32_t c[3];
    float f[3];
};
// with the cell's centre
struct Loc : Spot {
    double cen[3];
    __device__ __forceinline__ void centre()
    {
#pragma unroll
        for (int d = 0; d < 3; ++d) cen[d] = coord_center(level, c[d]);
    }
};

__device__ __forceinline__ float cells_per_unit(int L) { return __int_as_float((127 + L - kLevelShift) << 23); }

// full location by a walk from the top grid (float64 coordinates)
static __device__ __noinline__ Loc locate_full(const DevTree& T, double x, double y, double z)
{
    MPF_DIAG_COUNT(1);
    Loc r;
    const Found f = locate(T, x, y, z);
    r.cell = f.cell;
    r.level = f.level;
    if (f.cell >= 0) {
        point_cell(f.level, x, y, z, r.c, r.f);
        r.centre();
    }
    return r;
}

// A point in the neighbour e (record entry (ox, oy, oz) of the located cell
// h) when e is not a leaf of h's level: a refined cell of h's level (the
// point's deepest cell is found by following e's children along the point's
// octants) or a coarser leaf (the point lies in it).  fx, fy, fz: the point's
// offset from the neighbour's centre in units of h's cells.  The tree is
// navigated through the node array and the offsets carried in FP32, instead
// of a float64 walk from the top grid; r.cell = -2 when neither case applies
// (a wrapped key, a partly refined node) and the caller walks.
static __device__ __noinline__ Spot neighbour_other(const DevTree& T, const Spot& h, int e, int fl, int ox, int oy, int oz,
                                             float fx, float fy, float fz)
{
    Spot r;
    r.cell = -2;
    const int L = h.level;
    const int le = fl & 255;
    const uint32_t lim = (uint32_t)((1ull << L) - 1ull);
    const uint32_t nc[3] = {h.c[0] + (uint32_t)ox, h.c[1] + (uint32_t)oy, h.c[2] + (uint32_t)oz};
    if (nc[0] > lim || nc[1] > lim || nc[2] > lim) return r;
    if (le == L && (fl & 256)) {
        uint32_t c[3] = {nc[0], nc[1], nc[2]};
        float f[3] = {fx, fy, fz};
        int cell = e, lev = L;
        int nd = __ldg(&T.stencil[8 * (size_t)e + 6].w);
        for (int guard = 0; guard < kMaxLevel; ++guard) {
            const int2 node = __ldg(T.node + nd);
            if (node.x < 0) break;   // e's descendant containing the point is a leaf
            const int b[3] = {f[0] >= 0.f ? 1 : 0, f[1] >= 0.f ? 1 : 0, f[2] >= 0.f ? 1 : 0};
            const int nd2 = node.x + (b[0] | (b[1] << 1) | (b[2] << 2));
            const int2 child = __ldg(T.node + nd2);
            if (child.y < 0) return r;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                c[d] = 2u * c[d] + (uint32_t)b[d];
                f[d] = 2.f * f[d] + 0.5f - (float)b[d];
            }
            cell = child.y;
            nd = nd2;
            ++lev;
        }
        r.cell = cell;
        r.level = lev;
#pragma unroll
        for (int d = 0; d < 3; ++d) { r.c[d] = c[d]; r.f[d] = f[d]; }
        return r;
    }
    if (le < L && !(fl & 256)) {
        const int k = L - le;
        const float sk = __int_as_float((127 - k) << 23);   // 2^-k
        const float fn[3] = {fx, fy, fz};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            r.c[d] = nc[d] >> k;
            const uint32_t low = nc[d] - (r.c[d] << k);
            r.f[d] = ((float)low + 0.5f + fn[d]) * sk - 0.5f;
        }
        r.cell = e;
        r.level = le;
        return r;
    }
    return r;
}

// Ancestor of a located cell at the coarser level lc, through the parents
// stored in the records; c and fd follow (fd' = (fd + bit - 1/2) / 2 per
// level).  -1 when a parent is missing.
__device__ __forceinline__ int ancestor_up(const DevTree& T, int cell, int L, int lc, uint32_t* c, float* fd)
{
    for (int guard = 0; guard < kMaxLevel && L > lc; ++guard) {
        const int p = __ldg(&T.stencil[8 * (size_t)cell + 7].z);
        if (p < 0) return -1;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            fd[d] = (fd[d] + (float)(c[d] & 1u) - 0.5f) * 0.5f;
            c[d] >>= 1;
        }
        cell = p;
        --L;
    }
    return (L == lc) ? cell : -1;
}

// Deepest cell of point (x, y, z) given a nearby located cell `h`: the offset
// from h's centre is formed in float64 (one subtraction per axis) and the rest
// in FP32; the cell is h or one of its 26 neighbours read from h's record when
// that neighbour is a leaf of h's level; otherwise a full walk.
template <class P>
__device__ __forceinline__ Loc locate_rel(const DevTree& T, const Loc& h, float rx, float ry, float rz, const P& pos)
{
    if (h.cell >= 0) {
        const int ox = (int)floorf(rx + 0.5f), oy = (int)floorf(ry + 0.5f), oz = (int)floorf(rz + 0.5f);
        if (ox == 0 && oy == 0 && oz == 0) {
            Loc r = h;
            r.f[0] = rx; r.f[1] = ry; r.f[2] = rz;
            return r;
        }
        if (within_one_cell(ox, oy, oz)) {
            const int e = rec_entry(T, h.cell, (ox + 1) * 9 + (oy + 1) * 3 + (oz + 1));
            if (e >= 0) {
                const int fl = rec_flags(T, e);
                if (!(fl & 256) && (fl & 255) == h.level) {
                    Loc r;
                    r.cell = e;
                    r.level = h.level;
                    const double w = cell_extent(h.level);
                    r.c[0] = h.c[0] + ox; r.c[1] = h.c[1] + oy; r.c[2] = h.c[2] + oz;
                    // +-w or 0 per axis (selects, no int-to-double conversion)
                    r.cen[0] = h.cen[0] + (ox > 0 ? w : (ox < 0 ? -w : 0.0));
                    r.cen[1] = h.cen[1] + (oy > 0 ? w : (oy < 0 ? -w : 0.0));
                    r.cen[2] = h.cen[2] + (oz > 0 ? w : (oz < 0 ? -w : 0.0));
                    r.f[0] = rx - (float)ox; r.f[1] = ry - (float)oy; r.f[2] = rz - (float)oz;
                    return r;
                }
                Loc r;
                static_cast<Spot&>(r) = neighbour_other(T, h, e, fl, ox, oy, oz, rx - (float)ox, ry - (float)oy, rz - (float)oz);
                if (r.cell != -2) {
                    r.centre();
                    return r;
                }
            }
        }
    }
    return locate_full(T, pos.px(), pos.py(), pos.pz());
}

// Deepest cell of a point given by float64 coordinates near a located cell:
// the offset from the cell's centre is formed in float64 (one subtraction per
// axis) and rounded to FP32 cell units.
__device__ __forceinline__ Loc locate_near(const DevTree& T, const Loc& h, double x, double y, double z)
{
    float rx = 0.f, ry = 0.f, rz = 0.f;
    if (h.cell >= 0) {
        const float sc = cells_per_unit(h.level);
        rx = (float)(x - h.cen[0]) * sc; ry = (float)(y - h.cen[1]) * sc; rz = (float)(z - h.cen[2]) * sc;
    }
    return locate_rel(T, h, rx, ry, rz, PosAt{x, y, z});
}

// TSC at a point whose deepest cell is `cell` (simplehyperoctree.h:1479-1541
// through the stencil records).  Returns false when a restart centre is not
// itself a cell (left to the slow path).
// VEL: also the velocity slots into vv[3] (with need_all).
template <bool VEL, class P>
__device__ __forceinline__ bool tsc_rec(const DevTree& T, const Spot& d, const P& pos, bool need_all, Field7& res, float* vv)
{
    int cell = d.cell, L = d.level;
    float fd[3] = {d.f[0], d.f[1], d.f[2]};
    uint32_t c[3] = {d.c[0], d.c[1], d.c[2]};
    for (int guard = 0; guard <= kMaxLevel; ++guard) {
        const int4* rp = T.stencil + 8 * (size_t)cell;
        const int4 r7 = __ldg(rp + 7);
        const unsigned exact = (unsigned)r7.x;
        if (exact == kFullMask) {
            float wx[3], wy[3], wz[3];
            tsc_w3(fd[0], wx);
            tsc_w3(fd[1], wy);
            tsc_w3(fd[2], wz);
            float gx = 0.f, gy = 0.f, gz = 0.f, gt = 0.f, rho = 0.f, phi = 0.f, a = 0.f;
            float ux = 0.f, uy = 0.f, uz = 0.f;
            int e[28];
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const int4 v = __ldg(rp + q);
                e[4 * q] = v.x; e[4 * q + 1] = v.y; e[4 * q + 2] = v.z; e[4 * q + 3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < 27; ++j) {
                // wy * wz is shared by the three x-slabs: 9 products, then one per cell
                const float wt = wx[j / 9] * (wy[(j / 3) % 3] * wz[j % 3]);
                const float4 g = __ldg(T.grad + e[j]);
                gx = fmaf(g.x, wt, gx); gy = fmaf(g.y, wt, gy); gz = fmaf(g.z, wt, gz); gt = fmaf(g.w, wt, gt);
                if (need_all) {
                    const float4 s = __ldg(T.scal + e[j]);
                    rho = fmaf(s.x, wt, rho); phi = fmaf(s.y, wt, phi); a = fmaf(s.z, wt, a);
                    if (VEL) {
                        const float4 u = __ldg(T.vel + e[j]);
                        ux = fmaf(u.x, wt, ux); uy = fmaf(u.y, wt, uy); uz = fmaf(u.z, wt, uz);
                    }
                }
            }
            res = Field7{rho, phi, gx, gy, gz, a, gt};
            if (VEL) { vv[0] = ux; vv[1] = uy; vv[2] = uz; }
            return true;
        }
        // first entry (x-major) not at this level: missing -> empty, coarser -> restart there
        const int j = __ffs(~exact & kFullMask) - 1;
        const int e = __ldg(reinterpret_cast<const int*>(rp) + j);
        if (e < 0) {
            clear(res);
            if (VEL) vv[0] = vv[1] = vv[2] = 0.f;
            return true;
        }
        const int lc = rec_flags(T, e) & 255;
        MPF_DIAG_COUNT(0);
        // the restart cell is the point's ancestor at level lc
        const int up = ancestor_up(T, cell, L, lc, c, fd);
        if (up >= 0) {
            cell = up;
            L = lc;
            continue;
        }
        const double x = pos.px(), y = pos.py(), z = pos.pz();
        const Found f = find_cell(T, lc, axis_coord(lc, x), axis_coord(lc, y), axis_coord(lc, z));
        if (f.cell < 0 || f.level != lc) return false;
        cell = f.cell;
        L = lc;
        point_cell(L, x, y, z, c, fd);
    }
    return false;
}

// CIC at a point whose deepest cell is `cell` (simplehyperoctree.h:1410-1469).
template <bool VEL, class P>
__device__ __forceinline__ bool cic_rec(const DevTree& T, const Spot& d, const P& pos, bool need_all, Field7& res, float* vv)
{
    int cell = d.cell, L = d.level;
    float fd[3] = {d.f[0], d.f[1], d.f[2]};
    uint32_t c[3] = {d.c[0], d.c[1], d.c[2]};
    for (int guard = 0; guard <= kMaxLevel; ++guard) {
        const int sx = (fd[0] >= 0.f) ? 1 : -1, sy = (fd[1] >= 0.f) ? 1 : -1, sz = (fd[2] >= 0.f) ? 1 : -1;
        const float ax = fabsf(fd[0]), ay = fabsf(fd[1]), az = fabsf(fd[2]);
        int lvl = L;
        bool missing = false;
        float gx = 0.f, gy = 0.f, gz = 0.f, gt = 0.f, rho = 0.f, phi = 0.f, a = 0.f;
        float ux = 0.f, uy = 0.f, uz = 0.f;
        for (int v = 0; v < 8; ++v) {
            const int ox = (v & 1) ? ((sx > 0) ? 1 : 0) : ((sx > 0) ? 0 : -1);
            const int oy = (v & 2) ? ((sy > 0) ? 1 : 0) : ((sy > 0) ? 0 : -1);
            const int oz = (v & 4) ? ((sz > 0) ? 1 : 0) : ((sz > 0) ? 0 : -1);
            const int e = rec_entry(T, cell, (ox + 1) * 9 + (oy + 1) * 3 + (oz + 1));
            if (e < 0) { missing = true; break; }
            const int le = rec_flags(T, e) & 255;
            lvl = min(lvl, le);
            // the neighbour cell gets |fd|, the centre cell 1 - |fd| (per axis)
            const float wt = (ox ? ax : 1.f - ax) * (oy ? ay : 1.f - ay) * (oz ? az : 1.f - az);
            const float4 g = __ldg(T.grad + e);
            gx = fmaf(g.x, wt, gx); gy = fmaf(g.y, wt, gy); gz = fmaf(g.z, wt, gz); gt = fmaf(g.w, wt, gt);
            if (need_all) {
                const float4 s = __ldg(T.scal + e);
                rho = fmaf(s.x, wt, rho); phi = fmaf(s.y, wt, phi); a = fmaf(s.z, wt, a);
                if (VEL) {
                    const float4 u = __ldg(T.vel + e);
                    ux = fmaf(u.x, wt, ux); uy = fmaf(u.y, wt, uy); uz = fmaf(u.z, wt, uz);
                }
            }
        }
        if (lvl == L) {
            if (missing) clear(res);
            else res = Field7{rho, phi, gx, gy, gz, a, gt};
            if (VEL) {
                vv[0] = missing ? 0.f : ux; vv[1] = missing ? 0.f : uy; vv[2] = missing ? 0.f : uz;
            }
            return true;
        }
        MPF_DIAG_COUNT(0);
        const int up = ancestor_up(T, cell, L, lvl, c, fd);
        if (up >= 0) {
            cell = up;
            L = lvl;
            continue;
        }
        const double x = pos.px(), y = pos.py(), z = pos.pz();
        const Found f = find_cell(T, lvl, axis_coord(lvl, x), axis_coord(lvl, y), axis_coord(lvl, z));
        if (f.cell < 0 || f.level != lvl) return false;
        cell = f.cell;
        L = lvl;
        point_cell(L, x, y, z, c, fd);
    }
    return false;
}

// maybe_origin: the point can be the exact origin (first step of a ray),
// where the reference's TSC falls back to CIC (simplehyperoctree.h:1570-1571)
// VEL (with need_all): the velocity slots into vv[3] as well.
template <int ORDER, bool VEL = false, class P>
__device__ __forceinline__ Field7 gather_at(const DevTree& T, const Spot& d, const P& pos, bool need_all,
                                            bool maybe_origin, float* vv = nullptr)
{
    constexpr int order = ORDER;
    Field7 r;
    if (d.cell < 0) {
        clear(r);
        if (VEL) vv[0] = vv[1] = vv[2] = 0.f;
        return r;
    }
    if (!(maybe_origin && pos.px() == 0.0 && pos.py() == 0.0 && pos.pz() == 0.0)) {
        const bool ok = (order == 1) ? cic_rec<VEL>(T, d, pos, need_all, r, vv) : tsc_rec<VEL>(T, d, pos, need_all, r, vv);
        if (ok) return r;
    }
    if (VEL && need_all) return vel_slow(T, order, pos.px(), pos.py(), pos.pz(), vv);
    return (order == 1) ? cic_slow(T, pos.px(), pos.py(), pos.pz(), need_all)
                        : tsc_slow(T, pos.px(), pos.py(), pos.pz(), need_all);
}

struct FastRec {
    double a, t, x, y, z, k0, k1, k2, k3;
    double phi, red, chi, lambda, s, isw, iswold;
    float rho, dx, dy, dz, dt, ah;   // dt: the photon's (forward) dphidt
    int level;
};

// 1/a: FP32 seed refined by two Newton steps (full float64 accuracy)
__device__ __forceinline__ double recip(double a)
{
    double r = (double)(1.0f / (float)a);
    r = fma(r, fma(-a, r, 1.0), r);
    r = fma(r, fma(-a, r, 1.0), r);
    return r;
}


// geodesic RHS (integrator.h:409-445) from the field at the point.
// in = (a, t, x, y, z, k0, k1, k2, k3).  The FP64 pipe of this GPU retires 2
// operations per cycle per SM (1/64 of FP32), so the RHS keeps in FP64 only
// what the trajectory's accuracy needs:
//  * dphi/dlambda and the terms built from it are FP32: they only enter as
//    (2/c^2) dphi/dlambda, a rate that multiplies k (its error changes |k| by
//    a relative 1e-7 of that term's increment, not the direction);
//  * the lensing source 2 dphi/dx^i k0^2 is an FP32 product (the field is FP32);
//  * the Hubble drag and the k^i multiplications stay FP64, so the direction
//    of k and the positions keep float64 accuracy;
//  * dx/dlambda is returned as k itself: the caller folds 1/scale into the
//    RK coefficient (one multiplication per stage instead of three).
// inv_a = 1 / in[0]; tb = the cosmology bracket carried along the ray.
// kf: k^1..k^3 rounded to FP32 (the next stage's point offset in cell units).
__device__ __forceinline__ void rhs_math(const DevCosmo& C, const Field7& g, const double* in, double inv_a, int& tb,
                                         double* out, float* kf)
{
    const double c2 = kC * kC;
    const float k0f = (float)in[5], k1f = (float)in[6], k2f = (float)in[7], k3f = (float)in[8];
    kf[0] = k1f; kf[1] = k2f; kf[2] = k3f;
    const float dphidl = g.dt * k0f + (g.dx * k1f + g.dy * k2f + g.dz * k3f);
    const double dadt = interp_cached(C, in[1], C.dadt, C.slope_dadt, tb);
    out[0] = in[5] * dadt;
    out[1] = in[5];
    out[2] = in[6];
    out[3] = in[7];
    out[4] = in[8];
    const double hub = 2.0 * out[0] * inv_a;
    const float two_c2 = (float)(2.0 / c2);
    const float k02 = 2.0f * k0f * k0f;
    out[5] = -(hub * in[5]) - (double)((two_c2 * k0f) * (dphidl - g.dt * k0f));
    const double coef = (double)(two_c2 * dphidl) - hub;
    out[6] = fma(coef, in[6], -(double)(g.dx * k02));
    out[7] = fma(coef, in[7], -(double)(g.dy * k02));
    out[8] = fma(coef, in[8], -(double)(g.dz * k02));
}

// The photon record (Photon<double,3> fields) of a fast-mode trajectory point;
// data_dt: the field's dphidt there, dphi_over_dl: the laplacian column
// ((phi - previous phi) / dl), k: the point's index.
__device__ __forceinline__ Rec fast_record(const FastRec& b, float data_dt, double dphi_over_dl, long long k)
{
    const double c2 = kC * kC;
    Rec r;
    r.a = b.a; r.t = b.t; r.x = b.x; r.y = b.y; r.z = b.z; r.k0 = b.k0; r.k1 = b.k1; r.k2 = b.k2; r.k3 = b.k3;
    r.level = b.level; r.ah = b.ah; r.rho = b.rho; r.phi = b.phi;
    r.dx = b.dx; r.dy = b.dy; r.dz = b.dz; r.dt = b.dt;
    r.dphidl = (k > 0) ? ((double)data_dt * b.k0 + ((double)b.dx * b.k1 + (double)b.dy * b.k2 + (double)b.dz * b.k3)) : 0.0;
    r.lap = (k > 0) ? dphi_over_dl : 0.0;
    const double kk = b.k1 * b.k1 + b.k2 * b.k2 + b.k3 * b.k3;
    r.ds2 = (b.a * b.a) * (-(c2 * (1.0 + 2.0 * (b.phi / c2)) * b.k0 * b.k0) + ((1.0 - 2.0 * (b.phi / c2)) * kk));
    r.err = 1.0 - ((1.0 - 2.0 * (b.phi / c2)) * kk) / (c2 * (1.0 + 2.0 * (b.phi / c2)) * b.k0 * b.k0);
    r.red = b.red; r.isw = b.isw; r.iswold = b.iswold; r.chi = b.chi; r.lambda = b.lambda; r.s = b.s;
    r.index = (double)k;
    return r;
}

// ---------------------------------------------------------------------------
// Gathers of the propagation kernel.
//
// A gather runs in three phases that all lanes of a warp pass through
// together: the point's cell is found, the stencil that the reference's
// restarts end at is looked up (the record's int 31, resolved at upload), and
// the 27 (8) cells are summed.  With the sum inside the restart loop, as the
// point gathers above have it, a warp whose rays sit in cells of two or three
// levels issues the sum once per level: 18.7 of 32 lanes were active per
// instruction on a refined cone, and an RK step took 277 warp instructions
// per photon-step.
//
// What bounds them is the latency of one warp's instruction stream (the 8
// warps of an SM hide little of it), so the sums use the packed FP32 FMA
// (fma.rn.f32x2): two fields per instruction, each rounded as fmaf rounds it.
// Measured on refined cones (TSC, Jacobian, 60 000 rays): 282 ms -> 205 ms to
// z = 2, 197 ms -> 141 ms for the maps of 60 000 pixels to z = 1.
// ---------------------------------------------------------------------------
typedef unsigned long long pair32;   // two floats in a 64-bit register

__device__ __forceinline__ pair32 pack2(float a, float b)
{
    pair32 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(pair32 v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ pair32 mul2(pair32 a, pair32 b)
{
    pair32 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair32 fma2(pair32 a, pair32 b, pair32 c)
{
    pair32 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// An RK stage point, b + c k, and a Jacobian point: their float64 coordinates
// are formed only where a rare path needs them.
struct PosStage {
    double bx, by, bz, dlL;
    float cfr, kx, ky, kz;
    __device__ __forceinline__ double c() const { return (double)cfr * dlL; }
    __device__ __forceinline__ double px() const { return fma(c(), (double)kx, bx); }
    __device__ __forceinline__ double py() const { return fma(c(), (double)ky, by); }
    __device__ __forceinline__ double pz() const { return fma(c(), (double)kz, bz); }
};
struct PosShift {
    double x, y, z;
    int level, axis, sgn;
    __device__ __forceinline__ double at(double v, int a) const
    {
        const double h = pow2(kLevelShift - level);
        return (axis == a) ? v + (sgn > 0 ? h : -h) : v;
    }
    __device__ __forceinline__ double px() const { return at(x, 0); }
    __device__ __forceinline__ double py() const { return at(y, 1); }
    __device__ __forceinline__ double pz() const { return at(z, 2); }
};

enum { kSpotSame = 0, kSpotLeaf = 1, kSpotOther = 2 };

// The deepest cell of a point whose offset from the located cell h is
// (ox, oy, oz) cells plus f (from that neighbour's centre).  r7: the last
// quarter of the cell's record.  Returns how it was reached.
template <class P>
__device__ __forceinline__ int find_spot(const DevTree& T, const Spot& h, int ox, int oy, int oz, float fx, float fy, float fz,
                                         const P& pos, Spot& d, int4& r7)
{
    d = h;
    d.f[0] = fx; d.f[1] = fy; d.f[2] = fz;
    const bool same = h.cell >= 0 && (ox | oy | oz) == 0;
    int q = same ? h.cell : -1, kind = same ? kSpotSame : kSpotLeaf;
    if (!same && h.cell >= 0 && within_one_cell(ox, oy, oz))
        q = rec_entry(T, h.cell, (ox + 1) * 9 + (oy + 1) * 3 + (oz + 1));
    if (q >= 0) {
        r7 = __ldg(T.stencil + 8 * (size_t)q + 7);
        if (!same) {
            const int fl = r7.y & 511;
            if (fl == h.level) {   // a leaf of h's level
                d.cell = q;
                d.c[0] += (uint32_t)ox; d.c[1] += (uint32_t)oy; d.c[2] += (uint32_t)oz;
            } else {
                const Spot r = neighbour_other(T, h, q, fl, ox, oy, oz, fx, fy, fz);
                kind = kSpotOther;
                q = r.cell;
                if (q >= 0) {
                    d = r;
                    r7 = __ldg(T.stencil + 8 * (size_t)q + 7);
                }
            }
        }
    }
    if (q < 0) {
        const Loc l = locate_full(T, pos.px(), pos.py(), pos.pz());
        kind = kSpotOther;
        d.cell = l.cell;
        d.level = l.level;
        if (l.cell >= 0) {
#pragma unroll
            for (int q2 = 0; q2 < 3; ++q2) { d.c[q2] = l.c[q2]; d.f[q2] = l.f[q2]; }
            r7 = __ldg(T.stencil + 8 * (size_t)l.cell + 7);
        }
    }
    return kind;
}

// The point gather through the chain of restarts, out of line: at a ray's
// start, and for the cells whose restart the upload could not resolve.
template <int ORDER, bool VEL>
static __device__ __noinline__ Field7 gather_chain(const DevTree& T, const Spot& s, double x, double y, double z, int need_all,
                                                   int maybe_origin, float* vv)
{
    return gather_at<ORDER, VEL>(T, s, PosAt{x, y, z}, need_all != 0, maybe_origin != 0, vv);
}

// Sum over the N cells e of a stencil with weights w(j): the gradient and
// dphidt, with need_all the other fields, with VEL the velocity.  One chain
// per field in the order of the cells.
template <int N, bool VEL, class W>
__device__ __forceinline__ void sum_cells(const DevTree& T, const int* e, const W& w, bool need_all, Field7& r, float* vv)
{
    pair32 gxy = 0, gzt = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const pair32 wt = w(j);
        const ulonglong2 g = __ldg(reinterpret_cast<const ulonglong2*>(T.grad) + e[j]);
        gxy = fma2(g.x, wt, gxy);
        gzt = fma2(g.y, wt, gzt);
    }
    unpack2(gxy, r.dx, r.dy);
    unpack2(gzt, r.dz, r.dt);
    if (need_all) {
        pair32 rp = 0, al = 0;   // (rho, phi), (a, the level's bits: not used)
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const pair32 wt = w(j);
            const ulonglong2 s = __ldg(reinterpret_cast<const ulonglong2*>(T.scal) + e[j]);
            rp = fma2(s.x, wt, rp);
            al = fma2(s.y, wt, al);
        }
        float level;
        unpack2(rp, r.rho, r.phi);
        unpack2(al, r.a, level);
        if (VEL) {
            pair32 uxy = 0, uz = 0;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const pair32 wt = w(j);
                const ulonglong2 u = __ldg(reinterpret_cast<const ulonglong2*>(T.vel) + e[j]);
                uxy = fma2(u.x, wt, uxy);
                uz = fma2(u.y, wt, uz);
            }
            float none;
            unpack2(uxy, vv[0], vv[1]);
            unpack2(uz, vv[2], none);
        }
    }
}

// TSC (ORDER 2, simplehyperoctree.h:1479-1541) or CIC (ORDER 1, :1410-1469) at
// a located point; r7: the last quarter of its cell's record.
template <int ORDER, bool VEL, class P>
__device__ __forceinline__ Field7 gather_spot(const DevTree& T, const Spot& d, const int4& r7, const P& pos, bool need_all,
                                              float* vv)
{
    Field7 r;
    clear(r);
    if (VEL) vv[0] = vv[1] = vv[2] = 0.f;
    int cell = d.cell, state = (cell >= 0) ? 0 : -1;   // 0: sum, -1: empty, -2: through the chain of restarts
    float fd[3] = {d.f[0], d.f[1], d.f[2]};
    if (ORDER == 2) {
        if (cell >= 0) {
            const int t = r7.w;
            int k = r7.y >> 16;
            if (t >= 0) {
                cell = t;
                uint32_t c[3] = {d.c[0], d.c[1], d.c[2]};
                for (; k > 0; --k) {   // the point's offset in its ancestor, one level at a time
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        fd[q] = (fd[q] + (float)(c[q] & 1u) - 0.5f) * 0.5f;
                        c[q] >>= 1;
                    }
                }
            } else {
                state = t;
            }
        }
        if (state == 0) {
            const int4* rp = T.stencil + 8 * (size_t)cell;
            int e[28];
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const int4 v = __ldg(rp + q);
                e[4 * q] = v.x; e[4 * q + 1] = v.y; e[4 * q + 2] = v.z; e[4 * q + 3] = v.w;
            }
            float wx[3], wy[3], wz[3];
            tsc_w3(fd[0], wx);
            tsc_w3(fd[1], wy);
            tsc_w3(fd[2], wz);
            pair32 w2[9], wx2[3];   // wy * wz is shared by the three x-slabs
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                const float v = wy[q / 3] * wz[q % 3];
                w2[q] = pack2(v, v);
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) wx2[q] = pack2(wx[q], wx[q]);
            sum_cells<27, VEL>(T, e, [&](int j) { return mul2(wx2[j / 9], w2[j % 9]); }, need_all, r, vv);
        }
    } else {
        // the eight cells of the point's octant: entries s0 + {0, 1} x 9 + {0, 1} x 3 + {0, 1}
        constexpr unsigned kOct = 0x1u | 0x2u | 0x8u | 0x10u | 0x200u | 0x400u | 0x1000u | 0x2000u;
        int s0 = 0;
        if (cell >= 0) {
            int L = d.level;
            unsigned exact = (unsigned)r7.x;
            uint32_t c[3] = {d.c[0], d.c[1], d.c[2]};
            for (int guard = 0;; ++guard) {
                s0 = ((fd[0] >= 0.f) ? 9 : 0) + ((fd[1] >= 0.f) ? 3 : 0) + ((fd[2] >= 0.f) ? 1 : 0);
                if (((exact >> s0) & kOct) == kOct) break;
                // a coarser or a missing one: again on the ancestor at the coarsest of the eight's levels
                int lvl = L;
                for (int v = 0; v < 8; ++v) {
                    const int e = rec_entry(T, cell, s0 + 9 * (v & 1) + 3 * ((v >> 1) & 1) + (v >> 2));
                    if (e < 0) break;
                    lvl = min(lvl, rec_flags(T, e) & 255);
                }
                if (lvl == L) { state = -1; break; }
                cell = ancestor_up(T, cell, L, lvl, c, fd);
                if (cell < 0 || guard >= kMaxLevel) { state = -2; break; }
                L = lvl;
                exact = (unsigned)__ldg(&T.stencil[8 * (size_t)cell + 7].x);
            }
        }
        if (state == 0) {
            int e[8];
#pragma unroll
            for (int v = 0; v < 8; ++v) e[v] = rec_entry(T, cell, s0 + 9 * (v & 1) + 3 * ((v >> 1) & 1) + (v >> 2));
            // the neighbour on the point's side gets |fd|, the centre cell 1 - |fd| (per axis)
            float w0[3], w1[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float a = fabsf(fd[q]);
                w0[q] = (fd[q] >= 0.f) ? 1.f - a : a;
                w1[q] = (fd[q] >= 0.f) ? a : 1.f - a;
            }
            sum_cells<8, VEL>(T, e, [&](int v) {
                const float w = ((v & 1) ? w1[0] : w0[0]) * ((v & 2) ? w1[1] : w0[1]) * ((v & 4) ? w1[2] : w0[2]);
                return pack2(w, w);
            }, need_all, r, vv);
        }
    }
    if (state == -2) r = gather_chain<ORDER, VEL>(T, d, pos.px(), pos.py(), pos.pz(), need_all, 0, vv);
    return r;
}

// Per-thread values that a step touches once, kept in shared memory so that
// they do not occupy registers through the gathers; one block of slots per
// warp (dynamic shared memory, kSlotBytes a thread).  S: the Jacobian's FP64 running sums; ck, ckm1: the last point's
// contribution to them and the one before it (FP32 products of the point's
// FP32 Hessian terms); cen: the centre of the point's cell; the running
// integrals of the ray; the comoving distances of the last two points before
// the current one; the last step's length and change of phi.
constexpr int kSlotDoubles = 16;
constexpr int kSlotFloats = 14;
constexpr int kSlotBytes = kSlotDoubles * 8 + kSlotFloats * 4;
// with several lanes a ray, also the field gradients of the six Jacobian points
constexpr int kSharedRaySlotBytes = kSlotBytes + 18 * 4;
struct RaySlots {
    double* d;
    float* f;
    __device__ __forceinline__ RaySlots(double* shared, int slot_bytes)
    {
        double* const warp = shared + (threadIdx.x >> 5) * (32 * slot_bytes / 8);
        d = warp + (threadIdx.x & 31);
        f = reinterpret_cast<float*>(warp + 32 * kSlotDoubles) + (threadIdx.x & 31);
    }
    // value q of the ray's Jacobian points: one copy for the ray's lanes
    __device__ __forceinline__ float& point(int sub, int q) const { return f[(kSlotFloats + q) * 32 - sub]; }
    __device__ __forceinline__ double& S(int q) const { return d[q * 32]; }
    __device__ __forceinline__ double& cen(int q) const { return d[(6 + q) * 32]; }
    __device__ __forceinline__ double& lambda() const { return d[9 * 32]; }
    __device__ __forceinline__ double& s() const { return d[10 * 32]; }
    __device__ __forceinline__ double& isw() const { return d[11 * 32]; }
    __device__ __forceinline__ double& iswold() const { return d[12 * 32]; }
    __device__ __forceinline__ double& chim1() const { return d[13 * 32]; }
    __device__ __forceinline__ double& chim2() const { return d[14 * 32]; }
    __device__ __forceinline__ double& last_dl() const { return d[15 * 32]; }
    __device__ __forceinline__ float& ck(int q) const { return f[q * 32]; }
    __device__ __forceinline__ float& ckm1(int q) const { return f[(6 + q) * 32]; }
    __device__ __forceinline__ float& last_dphi() const { return f[12 * 32]; }
    __device__ __forceinline__ float& rmax() const { return f[13 * 32]; }
};

// The lanes that trace one ray: a full warp has one ray a lane; a warp with
// few rays gives each of them 2, 3 or 6 lanes, which take the same steps with
// the same values (and write the same outputs) and share out the six gathers
// of the Jacobian, the larger part of a step (rays_to_lanes).
struct RayLanes {
    int per_ray;     // 1, 2, 3 or 6
    int sub;         // this lane's place among them
    unsigned mask;   // the lanes of the ray
    __device__ __forceinline__ RayLanes(int lanes_per_ray, int lane)
        : per_ray(lanes_per_ray), sub(lane % lanes_per_ray), mask(((1u << lanes_per_ray) - 1u) << (lane - lane % lanes_per_ray)) {}
};

// Jacobian terms (d1d1, d1d2, d2d2 of lensing.h:430-447) at a trajectory
// point located at `here`: six TSC gathers at +-1 cell of the point's level,
// the same in-cell offset in the neighbouring cell of the record.  With
// several lanes tracing the ray together each gathers its share of the six.
__device__ __forceinline__ void jac_fast(const DevTree& T, const Spot& here, double x, double y, double z, float* out3,
                                         const RaySlots& J, const RayLanes& R)
{
    // differences of the plus and minus points, before 1 / dl
    float dxx = 0.f, dxy = 0.f, dxz = 0.f, dyy = 0.f, dyz = 0.f, dzz = 0.f;
    float mx = 0.f, my = 0.f, mz = 0.f;
#pragma unroll 1
    for (int q = R.sub; q < 6; q += R.per_ray) {
        const int axis = q >> 1, sgn = (q & 1) ? 1 : -1;
        const int ox = axis == 0 ? sgn : 0, oy = axis == 1 ? sgn : 0, oz = axis == 2 ? sgn : 0;
        const PosShift pos{x, y, z, here.level, axis, sgn};
        Spot d;
        int4 r7;
        find_spot(T, here, ox, oy, oz, here.f[0], here.f[1], here.f[2], pos, d, r7);
        const Field7 f = gather_spot<2, false>(T, d, r7, pos, false, nullptr);
        if (R.per_ray > 1) {
            J.point(R.sub, 3 * q) = f.dx; J.point(R.sub, 3 * q + 1) = f.dy; J.point(R.sub, 3 * q + 2) = f.dz;
        } else if (sgn < 0) {
            mx = f.dx; my = f.dy; mz = f.dz;
        } else if (axis == 0) {
            dxx = f.dx - mx;
        } else if (axis == 1) {
            dxy = f.dx - mx; dyy = f.dy - my;
        } else {
            dxz = f.dx - mx; dyz = f.dy - my; dzz = f.dz - mz;
        }
    }
    if (R.per_ray > 1) {
        __syncwarp(R.mask);
        dxx = J.point(R.sub, 3) - J.point(R.sub, 0);
        dxy = J.point(R.sub, 9) - J.point(R.sub, 6); dyy = J.point(R.sub, 10) - J.point(R.sub, 7);
        dxz = J.point(R.sub, 15) - J.point(R.sub, 12); dyz = J.point(R.sub, 16) - J.point(R.sub, 13);
        dzz = J.point(R.sub, 17) - J.point(R.sub, 14);
        __syncwarp(R.mask);
    }
    // dl = 2^-(level - 1 - log2 EXTENT) (lensing.h:430), twice the shift
    const float idl = __int_as_float((127 + here.level - kLevelShift - 1) << 23);   // 1 / dl, exact
    dxx *= idl; dxy *= idl; dxz *= idl; dyy *= idl; dyz *= idl; dzz *= idl;
    const float fx = (float)x, fy = (float)y, fz = (float)z;
    const float rho = sqrtf(fx * fx + fy * fy);
    const float r = sqrtf(fx * fx + fy * fy + fz * fz);
    const float cp = (rho > 0.f) ? fx / rho : 1.f, sp = (rho > 0.f) ? fy / rho : 0.f;
    const float ct = fz / r, snt = rho / r;
    const float s2p = 2.f * sp * cp, s2t = 2.f * snt * ct;
    out3[0] = sp * sp * dxx + cp * cp * dyy - s2p * dxy;
    out3[1] = ct * cp * sp * (dyy - dxx) + (cp * cp - sp * sp) * ct * dxy + sp * snt * dxz - cp * snt * dyz;
    out3[2] = cp * cp * ct * ct * dxx + sp * sp * ct * ct * dyy + snt * snt * dzz + s2p * ct * ct * dxy - sp * s2t * dyz -
              cp * s2t * dxz;
}

// The surface record between two trajectory points (hmaps.h:612-676), the
// Jacobian aside: out of line, a step crosses a surface once in a ray.
struct SurfaceEnd {
    double x, y, z, t, a, red, chi, lambda, s, isw, rho, phi, k0, k1, k2, k3;
};
__device__ __forceinline__ void surface_record(double* o, bool wide_record, double first, double f, const SurfaceEnd& b,
                                               const SurfaceEnd& p, double rmax)
{
    const double px = b.x * f + p.x * (1 - f), py = b.y * f + p.y * (1 - f), pz = b.z * f + p.z * (1 - f);
    o[0] = first; o[1] = f; o[2] = px; o[3] = py; o[4] = pz; o[5] = sqrt(px * px + py * py + pz * pz);
    o[6] = o[7] = o[8] = 0.0;
    o[9] = b.t * f + p.t * (1 - f);
    o[10] = b.a * f + p.a * (1 - f);
    o[11] = b.red * f + p.red * (1 - f);
    o[12] = b.chi * f + p.chi * (1 - f);
    o[13] = b.lambda * f + p.lambda * (1 - f);
    o[14] = b.s * f + p.s * (1 - f);
    o[15] = b.isw * f + p.isw * (1 - f);
    o[16] = b.rho * f + p.rho * (1 - f);
    o[17] = b.phi * f + p.phi * (1 - f);
    o[18] = rmax;
    o[19] = 1.0;
    if (wide_record) {
        o[20] = b.k0 * f + p.k0 * (1 - f);
        o[21] = b.k1 * f + p.k1 * (1 - f);
        o[22] = b.k2 * f + p.k2 * (1 - f);
        o[23] = b.k3 * f + p.k3 * (1 - f);
    }
}

static __device__ __noinline__ void write_surface(double* o, bool wide_record, double first, double f, SurfaceEnd b, SurfaceEnd p,
                                                  double rmax)
{
    surface_record(o, wide_record, first, f, b, p, rmax);
}

// v.k / (c k0), the Doppler term of a point
static __device__ __noinline__ double doppler_of(float v0, float v1, float v2, double k0, double k1, double k2, double k3)
{
    return ((double)v0 * k1 + (double)v1 * k2 + (double)v2 * k3) / (kC * k0);
}

static __device__ __noinline__ double distance_of(double x, double y, double z) { return sqrt(x * x + y * y + z * z); }

// a trajectory point's state and the field there
struct RayPoint {
    double a, t, x, y, z, k0, k1, k2, k3, chi;
    Field7 g;
};

// SRC: source mode (one surface at the ray's own radius); WIDE: per-ray
// surfaces and wide surface records (bundle rays).  The plain instantiation,
// the map and benchmark path, carries neither.  VEL: a velocity-field octree
// (the reference's -DVELOCITYFIELD build): the post-step gathers also read
// the velocity slots, an all-zero record with a velocity is not empty, and
// the redshift takes the ISW, Doppler and observer terms
// (integrator.h:707-708, 765-767); plain instantiations only.
template <int ORDER, bool SRC, bool WIDE, bool BORN = false, bool VEL = false>
__device__ void propagate_fast(const DevTree& T, const DevCosmo& C, const PropParams& P, const double* L, long long i,
                               const PropOut& O, const RaySlots& J, const RayLanes& R)
{
    const double c2 = kC * kC;
    const double mn = -(double)kExtent / 2.0, mx = (double)kExtent / 2.0;
    const double scale = P.length;
    const double inv_scale = 1.0 / scale;
    const int np = SRC ? 1 : P.nplanes;
    const int skind = SRC ? (int)STOP_R : P.stop_kind;
    const double* rpl = (WIDE && P.ray_planes) ? P.ray_planes + i * np : P.planes;   // this ray's surfaces
    const double stop_ref = SRC ? P.ray_stop[i] : ((WIDE && P.ray_planes) ? rpl[np - 1] : P.stop_ref);
    const int rec_fields = SRC ? kSourceFields : (WIDE ? kWideFields : kPlaneFields);
    // Born ray (Order = -1 on the octree itself: hmaps.h:706-712,
    // catalogues.h:670-673), an instantiation of its own: the homogeneous
    // field in the stages and after each step, the octree's levels for the
    // step length, its field for the Jacobian
    constexpr bool born = BORN;
    // Where the FP64 pipe is the larger part of a step, FP64 operations are
    // traded for FP32 and integer ones below (a screen of the redshift tests,
    // the Doppler term formed where it is read, the ISW sum by points, compares
    // on integer bits): 4 096 CIC rays 3.28 -> 3.09 ms, 8 009 rays with a
    // velocity field 3.53 -> 3.35.  A plain TSC step with the Jacobian's six
    // gathers (2 200 instructions) waits for instructions as much as for that
    // pipe, and the added code made it slower (60 000 map rays 119 -> 126 ms).
    // The order decides, not the Jacobian, which no instantiation knows: CIC
    // with it still gains (20 011 rays on a uniform cone 6.40 -> 6.16 ms,
    // 3 001 and 60 000 on a refined one 30.7 -> 29.6 and 111 -> 109), and TSC
    // without it hardly (bundle maps of 9 001 pixels 35.6 -> 35.2 ms, 20 011
    // plain rays 35.1 in both forms).
    constexpr bool kLean = ORDER == 1 || VEL;
    // Stage 1 written out, the table slope kept for the step and the surface
    // record out of line pay everywhere but in the TSC source instantiation,
    // which the catalogue's persistent kernel inlines: there they cost 5 to 8 %
    // (16 384 sources on an AMR octree 236 -> 225 ms without them, 2 054 on a
    // uniform one 20.1 -> 18.7).
    constexpr bool kPlain = SRC && ORDER == 2;
    Field7 hom;
    clear(hom);
    hom.a = 1.f;
    RayPoint b;
    b.a = 1.0; b.t = 0.0; b.x = L[0]; b.y = L[1]; b.z = L[2]; b.k0 = 1.0;
    if (SRC || (WIDE && P.direct)) {
        // (phi, theta) launch form or a bundle photon: the direction is given
        b.k1 = L[3]; b.k2 = L[4]; b.k3 = L[5];
    } else {
        const double A = L[3] - L[0], B = L[4] - L[1], D = L[5] - L[2];
        const double norm = sqrt(A * A + B * B + D * D);
        b.k1 = A / norm; b.k2 = B / norm; b.k3 = D / norm;
    }
    Spot here;
    float vv[3] = {0.f, 0.f, 0.f};   // VEL: the velocity of the last post-step gather
    {
        const Loc l = locate_full(T, b.x, b.y, b.z);
        here = l;
#pragma unroll
        for (int a = 0; a < 3; ++a) J.cen(a) = l.cen[a];
        b.g = born ? hom : gather_chain<ORDER, VEL>(T, l, b.x, b.y, b.z, 1, 1, vv);
    }
    {
        const double ph = (double)b.g.phi / c2;
        const double norm = sqrt((c2 * (1.0 + 2.0 * ph) * b.k0 * b.k0) / ((1.0 - 2.0 * ph) * (b.k1 * b.k1 + b.k2 * b.k2 + b.k3 * b.k3)));
        b.k1 *= norm; b.k2 *= norm; b.k3 *= norm;
    }
    const double v0n = VEL ? (P.vobs[0] * b.k1 + P.vobs[1] * b.k2 + P.vobs[2] * b.k3) / (kC * b.k0) : 0.0;
    float bv0 = 0.f, bv1 = 0.f, bv2 = 0.f;   // VEL: the velocity at b
    // data != empty (integrator.h:715): with VEL the velocity slots count too
    auto empty = [&](const Field7& f) -> bool { return is_empty(f) && (!VEL || (vv[0] == 0.f && vv[1] == 0.f && vv[2] == 0.f)); };
    b.a = interp_fast(C, b.t, C.a, C.slope_a);
    float bdt = b.g.dt;   // the photon's (forward) dphidt
    float bah = 0.f;
    b.chi = 0.0;
    const double ratio_k = (scale / kC) / P.nsteps;
    double dl = (here.cell >= 0 ? cell_extent(here.level) : 0.0) * (b.a * b.a * ratio_k);
    const double a0 = b.a;
    int tb = bracket_lut(C, b.t);       // cosmology-table bracket of the ray's conformal time
    const double phi0c2 = (double)b.g.phi / c2;
    for (int q = 0; q < 6; ++q) { J.S(q) = 0.0; J.ck(q) = 0.f; J.ckm1(q) = 0.f; }
    J.chim1() = J.chim2() = 0.0;
    J.isw() = J.iswold() = J.lambda() = J.s() = 0.0;
    J.last_dl() = 1.0;
    J.last_dphi() = 0.f;
    J.rmax() = 0.f;
    long long k = 0;
    unsigned status = 0;
    // A point's redshift (integrator.h:769) is formed only where it is read:
    // surface records, the end of the ray, trajectory records.  The stop and
    // crossing tests compare a0 (1 + phi0/c^2 - phi/c^2) with (1 + z) a
    // instead, which needs no division.  The starting point's redshift is 0.
    const double opc = 1.0 + phi0c2;
    const double inv_c2 = 1.0 / c2;
    const float inv_c2f = (float)inv_c2;
    const float opcf = (float)(VEL ? opc - v0n : opc);
    double x_before = 0.0, y_before = 0.0, z_before = 0.0;
    float phi_start = 0.f;
    if (kLean) {
        phi_start = b.g.phi;
        x_before = b.x; y_before = b.y; z_before = b.z;
    }
    // VEL: a0 / a (1 + phi0/c^2 - phi/c^2 + isw + v.k / (c k0) - v0n) - 1
    auto zbracket = [&](float phi, double isw, double dop) -> double {
        if (VEL) return opc - (double)phi * inv_c2 + isw + dop - v0n;
        return opc - (double)phi * inv_c2;
    };
    auto red_of = [&](double a, float phi, double isw, double dop) -> double { return a0 * recip(a) * zbracket(phi, isw, dop) - 1.0; };
    auto red_above = [&](double a, float phi, double isw, double dop, double zref) -> bool {
        return a0 * zbracket(phi, isw, dop) > (1.0 + zref) * a;
    };
    // the comoving distance is carried where each step reads it (the Jacobian,
    // the stop at a radius, trajectories), else formed where a record does: its
    // square root is a tenth of the FP64 operations of a CIC step
    const bool want_chi = P.jacobian || skind == STOP_R || (WIDE && O.traj);
    // the running ISW column: read by photon records only, the final one's and
    // a trajectory's
    const bool want_iswold = O.final_rec || (WIDE && O.traj);
    // FP32 screen of red_above: true only where the point is surely not above.
    // z1: (1 + zref) / a0 in FP32; the rounding of all terms is below 1e-6 of
    // the sum of their magnitudes, a tenth of the margin, and a NaN or an
    // overflow falls through to the float64 test.  A step changes (1 + z) a by
    // 1e-4 and more, so nearly every step's tests end here: 6 to 12 operations
    // of the FP64 pipe a test, and with a velocity field the Doppler term's 17.
    auto red_below = [&](float af, float phi, float iswf, float dopf, float dopm, float z1) -> bool {
        const float ph = phi * inv_c2f, o = opcf, r = z1 * af;
        float l = o - ph, m = fabsf(o) + fabsf(ph) + fabsf(r);
        if (VEL) {
            l += iswf + dopf;
            m += fabsf(iswf) + dopm;
        }
        return fmaf(1e-5f, m, l) < r;
    };
    auto z1_of = [&](double zref) -> float { return (a0 > 0.0) ? (float)((1.0 + zref) / a0) : __int_as_float(0x7fffffff); };
    auto b_dop = [&]() -> double { return (VEL && k) ? doppler_of(bv0, bv1, bv2, b.k0, b.k1, b.k2, b.k3) : 0.0; };
    // the point b as the reference's photon record
    auto full_point = [&]() -> FastRec {
        FastRec r;
        r.a = b.a; r.t = b.t; r.x = b.x; r.y = b.y; r.z = b.z; r.k0 = b.k0; r.k1 = b.k1; r.k2 = b.k2; r.k3 = b.k3;
        r.phi = b.g.phi; r.chi = (want_chi || k == 0) ? b.chi : distance_of(b.x, b.y, b.z); r.lambda = J.lambda(); r.s = J.s(); r.isw = J.isw();
        r.iswold = J.iswold();
        if (kLean && want_iswold)
            r.iswold = (J.iswold() + (double)b.g.dx * (b.x - x_before) + (double)b.g.dy * (b.y - y_before) +
                        (double)b.g.dz * (b.z - z_before)) * (scale * inv_c2) -
                       ((double)b.g.phi - (double)phi_start) * (2.0 * inv_c2);
        r.red = (k == 0) ? 0.0 : red_of(b.a, b.g.phi, r.isw, b_dop());
        r.rho = b.g.rho; r.dx = b.g.dx; r.dy = b.g.dy; r.dz = b.g.dz; r.dt = bdt; r.ah = bah;
        r.level = (here.cell >= 0) ? here.level : 0;
        return r;
    };

    // every trajectory point (bundle rays), wide instantiation only
    double* const traj = (WIDE && O.traj) ? O.traj + i * O.traj_cap * kPhotonFields : nullptr;
    if (WIDE && traj && O.traj_cap > 0) write_rec(traj, fast_record(full_point(), 0.f, 0.0, 0));
    int next_plane = 0;
    long long cross_k[kMaxPlanes];
    for (int j = 0; j < np; ++j) cross_k[j] = -1;
    double* prow = O.plane_rec ? O.plane_rec + (long long)i * np * rec_fields : nullptr;
    if (SRC && prow) {
        prow[24] = b.a; prow[25] = b.g.phi; prow[26] = b.k1; prow[27] = b.k2; prow[28] = b.k3;
        prow[29] = prow[30] = prow[31] = 0.0;
    }
    // this ray's plane normals (stop criterion "plane" with per-ray surfaces; wide instantiation)
    const double* rki = (WIDE && P.ray_ki) ? P.ray_ki + i * np * 3 : nullptr;
    auto start_q = [&](int jn) -> double {
        if (rki && skind == STOP_PLANE) return b.x * rki[3 * jn] + b.y * rki[3 * jn + 1] + b.z * rki[3 * jn + 2];
        return (skind == STOP_T) ? b.t : 0.0;   // chi, lambda, s and the redshift start at 0
    };
    while (next_plane < np && ((skind == STOP_A) ? (b.a < (SRC ? stop_ref : rpl[next_plane]))
                                                  : (start_q(next_plane) > (SRC ? stop_ref : rpl[next_plane])))) {
        cross_k[next_plane] = 0;
        ++next_plane;
    }
    const float two_c2 = (float)(2.0 / c2);
    bool go = !empty(b.g);
    const float z_stop = (kLean && skind == STOP_REDSHIFT) ? z1_of(stop_ref) : 0.f;
    float z_next = (kLean && skind == STOP_REDSHIFT && next_plane < np) ? z1_of(SRC ? stop_ref : rpl[next_plane]) : 0.f;
    while (go) {
        if (k >= P.max_steps) { status |= 1u; break; }
        // ---- RK4 step (integrator.h:718-734).  The state stays FP64 and is
        // accumulated in FP64; the four stages are evaluated in FP32 as
        // increments from the step's start b (c = 0, 1/2, 1/2, 1; weights
        // w = 1, 2, 2, 1):
        //   k_s = k_b + q_s,  q_s = c_s dl k'_{s-1},
        //   k^i' = coef k^i - 2 dphi/dx^i k0^2,   k0' = coef0 k0,
        //   coef = (2/c^2) dphi/dlambda - h,  coef0 = -h - (2/c^2) grad(phi).k,
        // with h = 2 (a'/a) k0 the Hubble drag (integrator.h:437-441).  The
        // drag sets |k| and the redshift, so it is formed once per step in FP64
        // at b, h_b, and each stage contributes its relative change
        // h_s = h_b (1 + eps_s) (eps ~ dl/L, FP32).  Then
        //   k^i_new = k^i_b + dl/6 (k^i_b sum w coef_s + sum w (coef_s q^i_s - 2 dphi/dx^i k0_s^2))
        //   x^i_new = x^i_b + dl/L k^i_b + dl/(6 L) sum w q^i_s
        //   t_new   = t_b + dl k0_b + dl/6 sum w q0_s
        //   a_new   = a_b + dl k0_b a'_b (1 + sum w ((1 + u_s)(1 + q0_s / k0_b) - 1) / 6)
        // with u_s the stage's relative change of a'.  The terms that set the
        // direction of k, |k| and the positions (k_b times the FP64 rates,
        // dl k_b) are FP64 products; the FP32 parts are corrections of
        // relative size dl/L (1e-4 to 1e-3 of the state).
        // da/dt at b (FP64, from the bracket carried along the ray) and the
        // distance to the bracket's upper node; the stages' da/dt follow the
        // table's linear pieces in FP32 from there.
        int ib;
        double adb;
        float tnext;
        {
            const int n = C.n;
            auto before = [](double a, double c) -> bool { return kLean ? less64(a, c) : a < c; };
            while (tb < n && !before(b.t, __ldg(C.t + tb))) ++tb;
            while (tb > 0 && before(b.t, __ldg(C.t + tb - 1))) --tb;
            ib = tb + (n > 1) * ((tb <= 0) - (tb >= n));
            if (n > 1) {
                adb = __ldg(C.dadt + ib - 1) + __ldg(C.slope_dadt + ib - 1) * (b.t - __ldg(C.t + ib - 1));
                tnext = (ib < n - 1) ? (float)(__ldg(C.t + ib) - b.t) : __int_as_float(0x7f800000);
            } else {
                adb = (n > 0) ? __ldg(C.dadt) : 0.0;
                tnext = __int_as_float(0x7f800000);
            }
        }
        const float seg0 = (!kPlain && C.n > 1) ? __ldg(&C.seg[ib - 1].x) : 0.f;
        // da/dt(b.t + dt) - da/dt(b.t) along the table's pieces (dt >= 0; the
        // last piece extends past the table's end, as in Utility::interpolate)
        auto dadot = [&](float dt) -> float {
            if (C.n <= 1) return 0.f;
            if (!kPlain && !(dt > tnext)) return seg0 * dt;
            float tn = tnext, rem = dt, r = 0.f;
            float sl = kPlain ? __ldg(&C.seg[ib - 1].x) : seg0;
            int j = ib;
            for (int guard = 0; rem > tn && guard < 64; ++guard) {
                r = fmaf(sl, tn, r);
                rem -= tn;
                const float2 sj = __ldg(C.seg + j);
                sl = sj.x;
                tn = (j + 2 < C.n) ? sj.y : __int_as_float(0x7f800000);
                ++j;
            }
            return fmaf(sl, rem, r);
        };
        const double dlL = dl * inv_scale;
        const double hubb = 2.0 * adb * recip(b.a) * b.k0;
        const float dlf = (float)dl, dlLf = (float)dlL, hubbf = (float)hubb;
        const float kb0 = (float)b.k0, kb1 = (float)b.k1, kb2 = (float)b.k2, kb3 = (float)b.k3;
        const float abf = (float)b.a, adbf = (float)adb;
        const float inv_kb0 = 1.f / kb0, inv_adbf = (adbf != 0.f) ? 1.f / adbf : 0.f;
        const float cpu = cells_per_unit(here.level);
        // previous stage: its k' (d0..d3), a' (dA) and k (pk0..pk3)
        float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f, dA = 0.f;
        float pk0 = kb0, pk1 = kb1, pk2 = kb2, pk3 = kb3;
        // weighted sums over the stages: the gravitational parts of coef and
        // coef0 (Gd, Gk), the drag's relative changes (Se), the second-order
        // terms of k (E), the stage increments (S) and the a' terms (SA)
        float Gd = 0.f, Gk = 0.f, Se = 0.f, E0 = 0.f, E1 = 0.f, E2 = 0.f, E3 = 0.f;
        float S0 = 0.f, S1 = 0.f, S2 = 0.f, S3 = 0.f, SA = 0.f;
        float dtf = 0.f, ds = 0.f;   // the step's conformal-time increment and path length
        RayPoint p;
        Spot q;
        int kind = kSpotSame;
        Field7 g = b.g;
        // stages 1-4, then the post-step point: stage 1 is at b, where the
        // previous step's post-step gather read the field, and has no
        // increments (written out: 3 to 7 % of a step of 2200 instructions);
        // stages 2-4 are located from their FP32 offset to b's cell, the
        // post-step point from its float64 offset
        if (!kPlain) {
            // stage 1, at b: no increments, the drag of b itself
            const float gk = fmaf(g.dx, kb1, fmaf(g.dz, kb3, __fmul_rn(g.dy, kb2)));
            const float dphidl = fmaf(g.dt, kb0, gk);
            const float tg = __fmul_rn(two_c2, dphidl), tk = __fmul_rn(two_c2, gk);
            const float coef = tg - hubbf;
            const float coef0 = -tk - hubbf;
            const float k02 = 2.f * kb0 * kb0;
            const float G1 = g.dx * k02, G2 = g.dy * k02, G3 = g.dz * k02;
            Gd = tg;
            Gk = tk;
            E1 = -G1; E2 = -G2; E3 = -G3;
            d0 = coef0 * kb0;
            d1 = fmaf(coef, kb1, -G1); d2 = fmaf(coef, kb2, -G2); d3 = fmaf(coef, kb3, -G3);
            dA = kb0 * adbf;
        }
        // stages 2-4 (rolled: 1-4)
#pragma unroll 1
        for (int sg = kPlain ? 0 : 1; sg < 5; ++sg) {
            const float cfr = (kPlain && sg == 0) ? 0.f : (sg < 3) ? 0.5f : 1.f;
            if (sg == 4) {
                const double dl6 = dl * (1.0 / 6.0), dlL6 = dlL * (1.0 / 6.0);
                const float dl6f = (float)dl6, dlL6f = (float)dlL6;
                const double h6 = hubb * (6.0 + (double)Se);
                const double cd = dl6 * ((double)Gd - h6);
                p.k0 = fma(b.k0, dl6 * (-h6 - (double)Gk), b.k0 + (double)(dl6f * E0));
                p.k1 = fma(b.k1, cd, b.k1 + (double)(dl6f * E1));
                p.k2 = fma(b.k2, cd, b.k2 + (double)(dl6f * E2));
                p.k3 = fma(b.k3, cd, b.k3 + (double)(dl6f * E3));
                p.x = fma(dlL, b.k1, b.x + (double)(dlL6f * S1));
                p.y = fma(dlL, b.k2, b.y + (double)(dlL6f * S2));
                p.z = fma(dlL, b.k3, b.z + (double)(dlL6f * S3));
                p.t = fma(dl, b.k0, b.t + (double)(dl6f * S0));
                const double da = __dmul_rn(dl * b.k0, adb);
                p.a = fma(da, (double)(SA * (1.f / 6.f)), __dadd_rn(b.a, da));
                // the step's displacement and conformal-time increment in FP32
                // (path length s and the ISW integral)
                const float ex = fmaf(dlLf, kb1, dlL6f * S1), ey = fmaf(dlLf, kb2, dlL6f * S2), ez = fmaf(dlLf, kb3, dlL6f * S3);
                ds = sqrtf(ex * ex + ey * ey + ez * ez);
                dtf = fmaf(dlf, kb0, dl6f * S0);
            }
            if ((!kPlain || sg > 0) && (!born || sg == 4)) {
                float rx, ry, rz;
                if (sg == 4) {
                    rx = (float)(p.x - J.cen(0)) * cpu; ry = (float)(p.y - J.cen(1)) * cpu; rz = (float)(p.z - J.cen(2)) * cpu;
                } else {
                    const float cc = cfr * dlLf * cpu;
                    rx = fmaf(cc, pk1, here.f[0]); ry = fmaf(cc, pk2, here.f[1]); rz = fmaf(cc, pk3, here.f[2]);
                }
                // the post-step point's own coordinates stand in for the stage form (c = 0)
                const PosStage ps = (sg == 4) ? PosStage{p.x, p.y, p.z, 0.0, 0.f, 0.f, 0.f, 0.f}
                                              : PosStage{b.x, b.y, b.z, dlL, cfr, pk1, pk2, pk3};
                const int ox = (int)floorf(rx + 0.5f), oy = (int)floorf(ry + 0.5f), oz = (int)floorf(rz + 0.5f);
                int4 r7;
                kind = find_spot(T, here, ox, oy, oz, rx - (float)ox, ry - (float)oy, rz - (float)oz, ps, q, r7);
                if (!born) g = gather_spot<ORDER, VEL>(T, q, r7, ps, sg == 4, vv);
            }
            if (sg < 4) {
                if (born && (!kPlain || sg > 0)) g = hom;
                const float cdl = cfr * dlf;
                const float q0 = __fmul_rn(cdl, d0), q1 = __fmul_rn(cdl, d1), q2 = __fmul_rn(cdl, d2), q3 = __fmul_rn(cdl, d3);
                const float w = ((kPlain && sg == 0) || sg == 3) ? 1.f : 2.f;
                const float k0 = kb0 + q0, k1 = kb1 + q1, k2 = kb2 + q2, k3 = kb3 + q3;
                const float as = fmaf(cdl, dA, abf);
                const float dad = dadot(cdl * pk0);
                // (the products that are contracted are written out here and below:
                // every instantiation then rounds a step alike)
                const float gk = fmaf(g.dx, k1, fmaf(g.dz, k3, __fmul_rn(g.dy, k2)));
                const float dphidl = fmaf(g.dt, k0, gk);
                // the drag at the stage relative to b: a' (1 + u), a / (1 - v'), k0 (1 + wk)
                const float u = dad * inv_adbf, v = -(cdl * dA) / as, wk = q0 * inv_kb0;
                const float uv = __fmul_rn(u, v);
                const float eps = fmaf(uv, wk, (u + v + wk) + fmaf(v, wk, fmaf(u, wk, uv)));
                // 2 / c^2 times a sum, less the drag hubb (1 + eps)
                const float tg = __fmul_rn(two_c2, dphidl), tk = __fmul_rn(two_c2, gk);
                const float coef = fmaf(-hubbf, 1.f + eps, tg);
                const float coef0 = fmaf(-hubbf, 1.f + eps, -tk);
                const float k02 = 2.f * k0 * k0;
                const float G1 = g.dx * k02, G2 = g.dy * k02, G3 = g.dz * k02;
                Gd = fmaf(w, tg, Gd);
                Gk = fmaf(w, tk, Gk);
                Se = fmaf(w, eps, Se);
                E0 = fmaf(w, coef0 * q0, E0);
                E1 = fmaf(w, fmaf(coef, q1, -G1), E1);
                E2 = fmaf(w, fmaf(coef, q2, -G2), E2);
                E3 = fmaf(w, fmaf(coef, q3, -G3), E3);
                S0 = fmaf(w, q0, S0); S1 = fmaf(w, q1, S1); S2 = fmaf(w, q2, S2); S3 = fmaf(w, q3, S3);
                SA = fmaf(w, fmaf(u, wk, u + wk), SA);
                d0 = coef0 * k0;
                d1 = fmaf(coef, k1, -G1); d2 = fmaf(coef, k2, -G2); d3 = fmaf(coef, k3, -G3);
                dA = k0 * (adbf + dad);
                pk0 = k0; pk1 = k1; pk2 = k2; pk3 = k3;
            }
        }
        p.g = born ? hom : g;
        {
            // the extent test (integrator.h:757): a point in a located cell away from
            // the domain faces is inside; only cells on a face (or wrapped keys)
            // need the float64 comparison
            const uint32_t last = (q.cell >= 0) ? (uint32_t)((1ull << q.level) - 1ull) : 0u;
            const bool face = (q.cell < 0) || q.c[0] == 0u || q.c[1] == 0u || q.c[2] == 0u ||
                              q.c[0] >= last || q.c[1] >= last || q.c[2] >= last;
            if ((kLean ? negative(p.a) : p.a < 0.0) ||
                (face && !((p.x > mn) && (p.x < mx) && (p.y > mn) && (p.y < mx) && (p.z > mn) && (p.z < mx)))) {
                clear(p.g);
                if (VEL) vv[0] = vv[1] = vv[2] = 0.f;
            }
        }
        if (empty(p.g)) break;   // the new point is not appended: the ray ends at b
        // formed where a redshift is
        auto p_dop = [&]() -> double { return VEL ? doppler_of(vv[0], vv[1], vv[2], p.k0, p.k1, p.k2, p.k3) : 0.0; };
        const float pdt = -p.g.dt;
        const double b_isw = J.isw(), b_s = J.s(), b_lambda = J.lambda();
        const double p_isw = b_isw + (double)((bdt + pdt) * dtf * inv_c2f);
        const double p_s = b_s + (double)ds;
        const double p_lambda = b_lambda + dl;
        J.isw() = p_isw;
        J.s() = p_s;
        J.lambda() = p_lambda;
        if (want_iswold) {
            // the sum of (g_b + g_p).(x_p - x_b) over the steps, gathered by
            // point: g_k.(x_k+1 - x_k-1), the last point's part where it is read
            if (kLean) {
                J.iswold() += (double)b.g.dx * (p.x - x_before) + (double)b.g.dy * (p.y - y_before) + (double)b.g.dz * (p.z - z_before);
                x_before = b.x; y_before = b.y; z_before = b.z;
            } else {
                J.iswold() -= ((double)p.g.phi - (double)b.g.phi) * (2.0 * inv_c2) -
                              (((double)b.g.dx + (double)p.g.dx) * (p.x - b.x) + ((double)b.g.dy + (double)p.g.dy) * (p.y - b.y) +
                               ((double)b.g.dz + (double)p.g.dz) * (p.z - b.z)) * (scale * inv_c2);
            }
            J.last_dphi() = p.g.phi - b.g.phi;   // laplacian of the record, divided there
            J.last_dl() = dl;
        }
        if (want_chi) p.chi = sqrt(p.x * p.x + p.y * p.y + p.z * p.z);
        dl = (q.cell >= 0 ? cell_extent(q.level) : 0.0) * (p.a * p.a * ratio_k);
        ++k;
        const float paf = kLean ? (float)p.a : 0.f;
        float iswf = 0.f, dopf = 0.f, dopm = 0.f;   // dopm: the sum of its terms' magnitudes
        if (VEL && skind == STOP_REDSHIFT) {
            iswf = (float)p_isw;
            const float w = 1.f / ((float)kC * (float)p.k0);
            const float d1v = vv[0] * (float)p.k1 * w, d2v = vv[1] * (float)p.k2 * w, d3v = vv[2] * (float)p.k3 * w;
            dopf = d1v + d2v + d3v;
            dopm = fabsf(d1v) + fabsf(d2v) + fabsf(d3v);
        }
        // the surfaces the step crossed: everything but the Jacobian, from b and p
        const int first_crossed = next_plane;
        bool p_red_known = false;   // the stop test below reads p's redshift where a surface formed it
        double p_red = 0.0;
        while (next_plane < np) {
            const double* kj = (WIDE && rki && skind == STOP_PLANE) ? rki + 3 * next_plane : nullptr;
            const double ref = SRC ? stop_ref : rpl[next_plane];
            bool crossed;
            double q1 = 0.0;
            if (!kj && skind == STOP_REDSHIFT) {
                crossed = !(kLean && red_below(paf, p.g.phi, iswf, dopf, dopm, z_next)) && red_above(p.a, p.g.phi, p_isw, p_dop(), ref);
            } else {
                if (!kj && skind == STOP_PLANE && !p_red_known) { p_red = red_of(p.a, p.g.phi, p_isw, p_dop()); p_red_known = true; }
                q1 = kj ? (p.x * kj[0] + p.y * kj[1] + p.z * kj[2])
                   : (skind == STOP_R) ? p.chi : (skind == STOP_LAMBDA) ? p_lambda : (skind == STOP_T) ? p.t
                   : (skind == STOP_A) ? p.a : (skind == STOP_S) ? p_s : p_red;
                crossed = (skind == STOP_A) ? (q1 < ref) : (q1 > ref);
            }
            if (!crossed) break;
            const int j = next_plane++;
            if (kLean && !SRC && skind == STOP_REDSHIFT && next_plane < np) z_next = z1_of(rpl[next_plane]);
            cross_k[j] = k;
            if (prow) {
                if (!p_red_known) { p_red = red_of(p.a, p.g.phi, p_isw, p_dop()); p_red_known = true; }
                const double b_red = (k == 1) ? 0.0 : red_of(b.a, b.g.phi, b_isw, b_dop());
                const double b_chi = want_chi ? b.chi : (k == 1) ? 0.0 : distance_of(b.x, b.y, b.z);
                const double p_chi = want_chi ? p.chi : distance_of(p.x, p.y, p.z);
                double* o = prow + j * rec_fields;
                if (!kj && skind == STOP_REDSHIFT) q1 = p_red;
                const double q0 = kj ? (b.x * kj[0] + b.y * kj[1] + b.z * kj[2])
                                : (skind == STOP_R) ? b.chi : (skind == STOP_LAMBDA) ? b_lambda : (skind == STOP_T) ? b.t
                                : (skind == STOP_A) ? b.a : (skind == STOP_S) ? b_s : b_red;
                const SurfaceEnd e0{b.x, b.y, b.z, b.t, b.a, b_red, b_chi, b_lambda, b_s, b_isw, (double)b.g.rho, (double)b.g.phi,
                                    b.k0, b.k1, b.k2, b.k3};
                const SurfaceEnd e1{p.x, p.y, p.z, p.t, p.a, p_red, p_chi, p_lambda, p_s, p_isw, (double)p.g.rho, (double)p.g.phi,
                                    p.k0, p.k1, p.k2, p.k3};
                if (kPlain) surface_record(o, SRC || WIDE, (double)(k - 1), (q1 - ref) / (q1 - q0), e0, e1, (k >= 2) ? (double)J.rmax() : 0.0);
                else write_surface(o, SRC || WIDE, (double)(k - 1), (q1 - ref) / (q1 - q0), e0, e1, (k >= 2) ? (double)J.rmax() : 0.0);
            }
        }
        // the largest density of the points before the new one
        if (k == 1 || J.rmax() < b.g.rho) J.rmax() = b.g.rho;
        // p becomes the ray's last point
        const float dr = (float)(p.chi - b.chi);
        const double chi_b = b.chi;
        b = p;
        bdt = pdt;
        bah = p.g.a;
        if (VEL) { bv0 = vv[0]; bv1 = vv[1]; bv2 = vv[2]; }
        if (kind != kSpotSame) {
            if (kind == kSpotLeaf) {
                // +-w or 0 per axis (selects, no int-to-double conversion)
                const double w = cell_extent(q.level);
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int o = (int)(q.c[a] - here.c[a]);
                    if (o != 0) J.cen(a) += (o > 0) ? w : -w;
                }
            } else if (q.cell >= 0) {
#pragma unroll
                for (int a = 0; a < 3; ++a) J.cen(a) = coord_center(q.level, q.c[a]);
            }
        }
        here = q;
        if (P.jacobian) {
            float h3[3];
            jac_fast(T, here, b.x, b.y, b.z, h3, J, R);
            const float chif = (float)b.chi;
            J.chim2() = J.chim1();
            J.chim1() = chi_b;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                J.ckm1(a) = J.ck(a); J.ckm1(3 + a) = J.ck(3 + a);
                const float c1 = chif * (h3[a] * dr), c2v = chif * c1;
                J.ck(a) = c1;
                J.ck(3 + a) = c2v;
                J.S(a) += (double)c1;
                J.S(3 + a) += (double)c2v;
            }
            for (int j = first_crossed; prow && j < next_plane; ++j) {
                // at the surface's distance, or at the source radius in source
                // mode, or at the surface radius itself for a Born ray
                double* o = prow + j * rec_fields;
                const double jd = (SRC || born) ? (SRC ? stop_ref : rpl[j]) : o[5];
                double s1[3], s2[3];
                bool ok = true;
                if (b.chi <= jd) {
                    for (int a = 0; a < 3; ++a) { s1[a] = J.S(a); s2[a] = J.S(3 + a); }
                } else if (chi_b <= jd) {
                    for (int a = 0; a < 3; ++a) { s1[a] = J.S(a) - (double)J.ck(a); s2[a] = J.S(3 + a) - (double)J.ck(3 + a); }
                } else if (k >= 2 && J.chim2() <= jd) {
                    for (int a = 0; a < 3; ++a) {
                        s1[a] = J.S(a) - (double)J.ck(a) - (double)J.ckm1(a);
                        s2[a] = J.S(3 + a) - (double)J.ck(3 + a) - (double)J.ckm1(3 + a);
                    }
                } else {
                    ok = false;
                    status |= 2u;
                }
                if (ok) {
                    const double idist = 1.0 / jd;
                    o[6] = 1.0 - 2.0 * (s1[0] - s2[0] * idist) / c2 * P.length;
                    o[7] = -2.0 * (s1[1] - s2[1] * idist) / c2 * P.length;
                    o[8] = 1.0 - 2.0 * (s1[2] - s2[2] * idist) / c2 * P.length;
                } else {
                    o[6] = 1.0; o[7] = 0.0; o[8] = 1.0;
                }
            }
        }
        if (WIDE && traj) {
            const FastRec r = full_point();
            p_red = r.red;
            p_red_known = true;
            if (k < O.traj_cap) write_rec(traj + k * kPhotonFields, fast_record(r, -bdt, (double)J.last_dphi() / J.last_dl(), k));
            else status |= 8u;
        }
        bool stop;
        switch (skind) {
        case STOP_R: stop = b.chi > stop_ref; break;
        case STOP_LAMBDA: stop = J.lambda() > stop_ref; break;
        case STOP_REDSHIFT:
            stop = p_red_known ? (p_red > stop_ref)
                               : !(kLean && red_below(paf, b.g.phi, iswf, dopf, dopm, z_stop)) &&
                                     red_above(b.a, b.g.phi, J.isw(), b_dop(), stop_ref);
            break;
        case STOP_T: stop = b.t > stop_ref; break;
        case STOP_A: stop = b.a < stop_ref; break;
        case STOP_PLANE: {
            const double* kk = (WIDE && rki) ? rki + 3 * (np - 1) : P.ki;
            stop = (b.x * kk[0] + b.y * kk[1] + b.z * kk[2]) > stop_ref;
            break;
        }
        case STOP_S: stop = J.s() > stop_ref; break;
        default: stop = true;
        }
        go = !stop;
    }
    const FastRec r = full_point();
    long long size = k + 1;
    if (signbit(r.red) || signbit(r.a)) size -= 1;
    O.steps[i] = size;
    if (O.final_rec) {
        double* o = O.final_rec + i * kPhotonFields;
        if (size == k + 1) {
            write_rec(o, fast_record(r, -bdt, (double)J.last_dphi() / J.last_dl(), k));
        } else {
            for (int a = 0; a < kPhotonFields; ++a) o[a] = 0.0;
            status |= 4u;
        }
    }
    if (SRC && prow) {
        const long long ck = cross_k[0];
        const bool ok = (ck >= 1) && (ck < size);
        if (!ok) {
            for (int q = 0; q < 24; ++q) prow[q] = 0.0;
            const long long marked = size - 1;
            prow[0] = (double)(marked - (marked > 0));
            if (born && P.jacobian && ck < 0) {
                // a Born ray that ends short of the radius: the Jacobian at its last point
                const double idist = 1.0 / stop_ref;
                prow[6] = 1.0 - 2.0 * (J.S(0) - J.S(3) * idist) / c2 * P.length;
                prow[7] = -2.0 * (J.S(1) - J.S(4) * idist) / c2 * P.length;
                prow[8] = 1.0 - 2.0 * (J.S(2) - J.S(5) * idist) / c2 * P.length;
            }
        }
        prow[19] = ok ? 1.0 : 0.0;
    } else if (prow) {
        for (int j = 0; j < np; ++j) {
            double* o = prow + j * rec_fields;
            const long long ck = cross_k[j];
            const bool found = (ck >= 1) && (ck < size);
            const bool valid = found && !((ck - 1) == size - 1 || (ck - 1) == 0);
            if (ck < 0 || ck == 0 || ck >= size) {
                for (int q = 0; q < (WIDE ? 24 : kPlaneFields); ++q) o[q] = 0.0;
                o[0] = (ck == 0) ? 0.0 : (double)(size - 1);
            }
            o[19] = valid ? 1.0 : 0.0;
            if (WIDE) o[24] = found ? 1.0 : 0.0;
            if (born) {
                // Born ray (hmaps.h:712, 719): the Jacobian at the surface radius,
                // from the last point when the ray never got there; only a ray
                // that could not take a step is unusable
                if (P.jacobian && ck < 0) {
                    const double idist = 1.0 / rpl[j];
                    o[6] = 1.0 - 2.0 * (J.S(0) - J.S(3) * idist) / c2 * P.length;
                    o[7] = -2.0 * (J.S(1) - J.S(4) * idist) / c2 * P.length;
                    o[8] = 1.0 - 2.0 * (J.S(2) - J.S(5) * idist) / c2 * P.length;
                }
                o[19] = (size > 1) ? 1.0 : 0.0;
            }
        }
    }
    if (status) atomicOr(O.status, status);
}

// Persistent launch: each warp takes the next rays x depth rays of [lo, n)
// from a global counter until the range is exhausted, so uneven path lengths
// do not leave tail waves; it traces `rays` of them at a time with per_ray
// lanes each (rays x per_ray <= 32).  `queue` is zeroed before the launch.
// The launch shape and the order (perm: the ray at each position, or null) are
// the launcher's (mpf_prop_fast.cu); the rays' results do not depend on them.
#if defined(MPF_FAST_MAXNREG)
#define MPF_FAST_BOUNDS __maxnreg__(MPF_FAST_MAXNREG)
#else
#define MPF_FAST_BOUNDS __launch_bounds__(kFastThreads, MPF_FAST_MINB)
#endif
template <int ORDER, bool SRC, bool WIDE, bool BORN = false, bool VEL = false>
__global__ void MPF_FAST_BOUNDS k_propagate_fast(DevTree T, DevCosmo C, PropParams P,
                                                                    const double* __restrict__ launch, long long n, PropOut O,
                                                                    unsigned long long* queue, int rays, int per_ray, int depth,
                                                                    long long lo, const int* __restrict__ perm)
{
    extern __shared__ double slots[];
    const RaySlots J(slots, per_ray > 1 ? kSharedRaySlotBytes : kSlotBytes);
    const int lane = threadIdx.x & 31;
    const RayLanes R(per_ray, lane);
    const int ray = lane / per_ray;
    const unsigned long long per = (unsigned long long)rays * (unsigned long long)depth;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(queue, per);
        base = __shfl_sync(0xffffffffu, base, 0) + (unsigned long long)lo;
        if (base >= (unsigned long long)n) break;
        for (int d = 0; d < depth; ++d) {
            long long i = (long long)base + (long long)rays * d + ray;
            if (ray < rays && i < n) {
                if (perm) i = perm[i];
                propagate_fast<ORDER, SRC, WIDE, BORN, VEL>(T, C, P, launch + 6 * i, i, O, J, R);
            }
            __syncwarp();
        }
    }
}

// Fast-mode gathers through the stencil records (tests / mpf_interpolate).
static __global__ void k_gather_rec(DevTree T, int kind, const double* __restrict__ xyz, long long n, void* out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    const Loc d = locate_full(T, x, y, z);
    if (kind == 0) {
        ((long long*)out)[i] = d.cell;
        return;
    }
    const Field7 f = (kind == 1) ? gather_at<1>(T, d, PosAt{x, y, z}, true, true)
                                 : gather_at<2>(T, d, PosAt{x, y, z}, true, true);
    float* o = (float*)out + 7 * i;
    o[0] = f.rho; o[1] = f.phi; o[2] = f.dx; o[3] = f.dy; o[4] = f.dz; o[5] = f.a; o[6] = f.dt;
}

}  // namespace mpf
