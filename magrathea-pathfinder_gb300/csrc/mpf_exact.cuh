// The float64 kernel: gathers, geodesic steps and the lensing Jacobian in the
// reference's operation order and rounding (built with -fmad=false).  One ray
// per lane, or per 2, 3 or 6 lanes of a warp with few rays, which then share
// out the Jacobian's gathers.
//
// What bounds it is the FP64 pipe, which takes 64 cycles of an SM
// sub-partition for a warp's add, multiply, fused multiply-add, compare or
// conversion alike, however many of its lanes are active.  A
// field's multiply-accumulate is (float)((double)acc + (double)v * w): two
// operations and three conversions.  The conversions, products with powers of
// two, coordinates and table lookups are done on the integer bits here,
// weights and vertex coordinates once per axis instead of once per cell, the
// divisions by the box length by its reciprocal and two residuals, the record
// fields that only a photon record reports at the ray's end; the field at a
// step's start is the one already read after the step before it, and a point's
// cell is looked for around the last one's.  4099 rays of 277 steps on a
// refined cone (TSC, Jacobian): 202 ms -> 46 ms, the FP64 pipe busy 63 % of the
// time.
#pragma once
#include "mpf_fp64.cuh"
#include "mpf_propagate.cuh"

namespace mpf {

// acc += v * w with the reference's rounding, the accumulator a float held in
// a double: (float)((double)acc + (double)v * w)
__device__ __forceinline__ double mac64(double acc, float v, double w)
{
    return round32(__dadd_rn(acc, __dmul_rn(wide(v), w)));
}

// Fields of a gather: dphidx..z (Jacobian), with dphidt (RK stages), all
enum { kGradient3 = 0, kGradient4 = 1, kAllFields = 2 };

// Accumulator of the walks; V: also the velocity slots of the velocity-field
// octree (gravity2.h:45), which the reference's multiply-accumulate treats
// like the other fields (simplehyperoctree.h:1887-1910).
template <int F, bool V>
struct ExactAcc {
    double dx, dy, dz, dt, rho, phi, a, v[3];
    __device__ __forceinline__ void reset()
    {
        dx = dy = dz = dt = rho = phi = a = 0.0;
        if (V) v[0] = v[1] = v[2] = 0.0;
    }
    __device__ __forceinline__ void add(const DevTree& T, int cell, double w)
    {
        const float4 g = __ldg(T.grad + cell);
        dx = mac64(dx, g.x, w);
        dy = mac64(dy, g.y, w);
        dz = mac64(dz, g.z, w);
        if (F >= kGradient4) dt = mac64(dt, g.w, w);
        if (F == kAllFields) {
            const float4 s = __ldg(T.scal + cell);
            rho = mac64(rho, s.x, w);
            phi = mac64(phi, s.y, w);
            a = mac64(a, s.z, w);
        }
        if (V) {
            const float4 u = __ldg(T.vel + cell);
            v[0] = mac64(v[0], u.x, w);
            v[1] = mac64(v[1], u.y, w);
            v[2] = mac64(v[2], u.z, w);
        }
    }
    __device__ __forceinline__ Field7 field(float* vv) const
    {
        if (V)
            for (int q = 0; q < 3; ++q) vv[q] = (float)v[q];
        return Field7{(float)rho, (float)phi, (float)dx, (float)dy, (float)dz, (float)a, (float)dt};
    }
};

// A cell near the next point looked for, and its integer coordinates.
struct Hint {
    int cell;
    int level;
    uint32_t c[3];
};

// locate(): the deepest cell holding the point with level-32 coordinates c32.
// When it is the hint's cell or one of its 26 neighbours, a leaf of the
// hint's level, the record names it (find_cell's result for the key); else
// the walk from the top grid.  The hint moves to the cell found.
__device__ __forceinline__ Found locate_near32(const DevTree& T, const uint64_t* c32, Hint& h)
{
    if (h.cell >= 0) {
        int o[3];
        bool near = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            o[d] = (int)((uint32_t)(c32[d] >> (kMaxLevel - h.level)) - h.c[d]);
            near = near && o[d] >= -1 && o[d] <= 1;
        }
        if (near) {
            const int e = (o[0] | o[1] | o[2]) == 0
                              ? h.cell
                              : __ldg(reinterpret_cast<const int*>(T.stencil + 8 * (size_t)h.cell) + (o[0] + 1) * 9 + (o[1] + 1) * 3 + (o[2] + 1));
            if (e >= 0 && (__ldg(&T.stencil[8 * (size_t)e + 7].y) & 511) == h.level) {
                h.cell = e;
#pragma unroll
                for (int d = 0; d < 3; ++d) h.c[d] += (uint32_t)o[d];
                return Found{e, h.level};
            }
        }
    }
    const Found f = find_cell(T, kMaxLevel, c32[0], c32[1], c32[2]);
    h.cell = f.cell;
    h.level = f.level;
#pragma unroll
    for (int d = 0; d < 3; ++d) h.c[d] = (uint32_t)(c32[d] >> (kMaxLevel - f.level));
    return f;
}

// find_cell(T, L, k) for the integer coordinates k of a level-L key, read
// from the stencil record of the level-L cell `centre` (coordinates cc) when
// k is one of its 27 neighbours (the record holds find_cell's result for each
// of them), else found by the walk.  centre < 0: no record to read.
__device__ __forceinline__ Found find_near(const DevTree& T, int centre, int L, const uint64_t* cc, const uint64_t* k)
{
    if (centre >= 0 && L >= 2) {
        const uint64_t mask = (1ull << L) - 1ull;
        int o[3];
        bool ok = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const uint64_t dm = (k[d] - cc[d]) & mask;
            o[d] = (dm == 0) ? 0 : (dm == 1) ? 1 : (dm == mask) ? -1 : 2;
            ok = ok && o[d] != 2;
        }
        if (ok) {
            const int e = __ldg(reinterpret_cast<const int*>(T.stencil + 8 * (size_t)centre) + (o[0] + 1) * 9 +
                                (o[1] + 1) * 3 + (o[2] + 1));
            if (e < 0) return Found{-1, 0};
            return Found{e, __float_as_int(__ldg(&T.scal[e].w))};
        }
    }
    return find_cell(T, L, k[0], k[1], k[2]);
}

// the level-`to` ancestor of the level-`from` cell `cell` through the records'
// parent links, or -1
__device__ __forceinline__ int ancestor_cell(const DevTree& T, int cell, int from, int to)
{
    for (int l = from; l > to && cell >= 0; --l)
        cell = __ldg(reinterpret_cast<const int*>(T.stencil + 8 * (size_t)cell) + 30);
    return cell;
}

// Cloud-in-cell (simplehyperoctree.h:1410-1469): trilinear over the 8 cells
// of the located cell's level; restarts one level up when a neighbour is
// coarser; empty when a neighbour is missing.
template <int F, bool V>
__device__ Field7 cic_exact(const DevTree& T, double x, double y, double z, Hint& hint, float* vv)
{
    ExactAcc<F, V> res;
    res.reset();
    const uint64_t c32[3] = {axis_coord_bits(kMaxLevel, x), axis_coord_bits(kMaxLevel, y), axis_coord_bits(kMaxLevel, z)};
    const Found f0 = locate_near32(T, c32, hint);
    if (f0.cell < 0) return res.field(vv);
    int ilvl = f0.level, lvl = ilvl;
    int centre = f0.cell;   // the record of the centre cell at level ilvl
    const double pt[3] = {x, y, z};
    do {
        if (lvl < ilvl) centre = ancestor_cell(T, centre, ilvl, lvl);
        ilvl = lvl;
        const double half = half_cell(ilvl);
        const uint64_t m = (1ull << ilvl) - 1ull;
        uint64_t cc[3], k[3][2];
        double w[3][2];   // by the vertex's bit
        int site = 0;
        bool near = centre >= 0 && ilvl >= 2;
        int base[3];   // neighbour offset of the vertices with bit 0
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            cc[d] = c32[d] >> (kMaxLevel - ilvl);
            const int s = (ilvl < kMaxLevel) ? (int)((c32[d] >> (kMaxLevel - ilvl - 1)) & 1ull) : 0;
            site |= s << d;
            // over the cell size, a power of two
            const double dist = fabs(times_pow2(__dsub_rn(coord_center_bits(ilvl, cc[d]), pt[d]), ilvl - kLevelShift));
            // the neighbour on the point's side weighs dist, the centre cell 1 - dist
            const double rest = __dsub_rn(1.0, dist);
            w[d][0] = s ? rest : dist;
            w[d][1] = s ? dist : rest;
            k[d][0] = axis_coord_bits(ilvl, __dsub_rn(pt[d], half));
            k[d][1] = axis_coord_bits(ilvl, __dadd_rn(pt[d], half));
            base[d] = s - 1;
            near = near && k[d][0] == ((cc[d] + (uint64_t)(int64_t)(s - 1)) & m) && k[d][1] == ((cc[d] + (uint64_t)s) & m);
        }
        bool missing = false;
        const int* const rec = reinterpret_cast<const int*>(T.stencil + 8 * (size_t)(near ? centre : 0));
        const unsigned exact = near ? (unsigned)__ldg(rec + 28) : 0u;
        for (int v = 0; v < 8 && !missing; ++v) {
            const int b0 = v & 1, b1 = (v >> 1) & 1, b2 = v >> 2;
            const double wt = __dmul_rn(__dmul_rn(b0 ? w[0][1] : w[0][0], b1 ? w[1][1] : w[1][0]), b2 ? w[2][1] : w[2][0]);
            Found fi;
            if (near) {
                const int j = (base[0] + b0 + 1) * 9 + (base[1] + b1 + 1) * 3 + (base[2] + b2 + 1);
                fi.cell = __ldg(rec + j);
                fi.level = ((exact >> j) & 1u) ? ilvl : (fi.cell >= 0) ? __float_as_int(__ldg(&T.scal[fi.cell].w)) : 0;
            } else {
                const uint64_t kk[3] = {b0 ? k[0][1] : k[0][0], b1 ? k[1][1] : k[1][0], b2 ? k[2][1] : k[2][0]};
                fi = find_near(T, centre, ilvl, cc, kk);
            }
            if (fi.cell >= 0) {
                lvl = min(lvl, fi.level);
                res.add(T, fi.cell, wt);
            } else {
                missing = true;
            }
        }
        if (missing || lvl < ilvl) res.reset();
    } while (lvl < ilvl);
    return res.field(vv);
}

// the reference's a * 0.5 * (1.5 - d) * (1.5 - d) + (1 - a) * (0.75 - d * d),
// left to right, for a = 0 or 1: the other term is an exact zero
__device__ __forceinline__ double tsc_w1(int a, double d)
{
    if (a) {
        const double e = __dsub_rn(1.5, d);
        return __dmul_rn(times_pow2(e, -1), e);
    }
    return __dsub_rn(0.75, __dmul_rn(d, d));
}

// tsc_exact at a point with a level-32 coordinate of all ones: it may have
// saturated (from 2^34 on) where a coarser level's still wraps, so every
// vertex's coordinates are formed at its own level.  Out of line: rays do not
// get there.
template <int F, bool V>
static __device__ __noinline__ Field7 tsc_saturated(const DevTree& T, double x, double y, double z, Hint& hint, float* vv)
{
    ExactAcc<F, V> res;
    res.reset();
    const uint64_t c32[3] = {axis_coord(kMaxLevel, x), axis_coord(kMaxLevel, y), axis_coord(kMaxLevel, z)};
    const Found f0 = locate_near32(T, c32, hint);
    if (f0.cell < 0) return res.field(vv);
    int ilvl = f0.level, lvl = ilvl;
    const double pt[3] = {x, y, z};
    do {
        ilvl = lvl;
        const double tw = cell_extent(ilvl);
        bool stop = false;
#pragma unroll 1
        for (int v = 0; v < 27 && !stop; ++v) {
            double w = 1.0;
            uint64_t k[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int o = (d == 0 ? v / 9 : d == 1 ? (v / 3) % 3 : v % 3) - 1;
                k[d] = axis_coord(ilvl, __dadd_rn(pt[d], o == 0 ? 0.0 : o > 0 ? tw : -tw));
                w = __dmul_rn(w, tsc_w1(o != 0, fabs(times_pow2(__dsub_rn(coord_center(ilvl, k[d]), pt[d]), ilvl - kLevelShift))));
            }
            const Found fi = find_cell(T, ilvl, k[0], k[1], k[2]);
            if (fi.cell >= 0) lvl = min(lvl, fi.level);
            stop = fi.cell < 0 || lvl < ilvl;
            if (!stop) res.add(T, fi.cell, w);
        }
        if (stop) res.reset();
    } while (lvl < ilvl);
    return res.field(vv);
}

// Triangular-shaped cloud (simplehyperoctree.h:1479-1644): quadratic weights
// over the 27 cells of the located cell's level, x-major (ix, iy, iz) order;
// restarts at the level of the first coarser neighbour; empty when one is
// missing; CIC at the exact origin.
template <int F, bool V>
__device__ Field7 tsc_exact(const DevTree& T, double x, double y, double z, Hint& hint, float* vv)
{
    if (x == 0.0 && y == 0.0 && z == 0.0) return cic_exact<F, V>(T, 0., 0., 0., hint, vv);
    ExactAcc<F, V> res;
    res.reset();
    const uint64_t c32[3] = {axis_coord_bits(kMaxLevel, x), axis_coord_bits(kMaxLevel, y), axis_coord_bits(kMaxLevel, z)};
    // (the stages and the Jacobian's points of a ray lie within a step and a cell
    // of the domain, those of other rays are not kept)
    const uint64_t ones = 0xffffffffull;
    if (F == kAllFields && (c32[0] == ones || c32[1] == ones || c32[2] == ones)) return tsc_saturated<F, V>(T, x, y, z, hint, vv);
    const Found f0 = locate_near32(T, c32, hint);
    if (f0.cell < 0) return res.field(vv);
    int ilvl = f0.level, lvl = ilvl;
    int centre = f0.cell;   // the record of the centre cell at level ilvl
    const double pt[3] = {x, y, z};
    do {
        if (lvl < ilvl) centre = ancestor_cell(T, centre, ilvl, lvl);
        ilvl = lvl;
        const double tw = cell_extent(ilvl);
        const uint64_t m = (1ull << ilvl) - 1ull;
        uint64_t cc[3], k[3][3];
        double w[3][3];
        bool near = centre >= 0 && ilvl >= 2;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            cc[d] = c32[d] >> (kMaxLevel - ilvl);
            k[d][0] = axis_coord_bits(ilvl, __dsub_rn(pt[d], tw));
            k[d][1] = cc[d];
            k[d][2] = axis_coord_bits(ilvl, __dadd_rn(pt[d], tw));
            const bool next = k[d][0] == ((cc[d] - 1ull) & m) && k[d][2] == ((cc[d] + 1ull) & m);
            near = near && next;
            // the vertices' cell centres, one cell apart in the usual case (exact)
            const double c1 = coord_center_bits(ilvl, cc[d]);
            const bool inside = next && cc[d] > 0ull && cc[d] < m;
            const double c0 = inside ? __dsub_rn(c1, tw) : coord_center(ilvl, k[d][0]);
            const double c2 = inside ? __dadd_rn(c1, tw) : coord_center(ilvl, k[d][2]);
            // over the cell size, a power of two
            w[d][0] = tsc_w1(1, fabs(times_pow2(__dsub_rn(c0, pt[d]), ilvl - kLevelShift)));
            w[d][1] = tsc_w1(0, fabs(times_pow2(__dsub_rn(c1, pt[d]), ilvl - kLevelShift)));
            w[d][2] = tsc_w1(1, fabs(times_pow2(__dsub_rn(c2, pt[d]), ilvl - kLevelShift)));
        }
        if (near) {
            // the vertices are the record's 27 cells in order
            const int4* const rp = T.stencil + 8 * (size_t)centre;
            const int4 r7 = __ldg(rp + 7);
            const unsigned exact = (unsigned)r7.x, full = (1u << 27) - 1u;
            if (exact != full) {
                const int e = __ldg(reinterpret_cast<const int*>(rp) + (__ffs(~exact & full) - 1));
                if (e >= 0) lvl = __float_as_int(__ldg(&T.scal[e].w));
                continue;   // at the coarser level, or empty
            }
            int e[28];
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const int4 v = __ldg(rp + q);
                e[4 * q] = v.x; e[4 * q + 1] = v.y; e[4 * q + 2] = v.z; e[4 * q + 3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < 27; ++j) res.add(T, e[j], __dmul_rn(__dmul_rn(w[0][j / 9], w[1][(j / 3) % 3]), w[2][j % 3]));
            break;
        }
        bool stop = false;
        for (int ix = 0; ix < 3 && !stop; ++ix)
            for (int iy = 0; iy < 3 && !stop; ++iy)
                for (int iz = 0; iz < 3 && !stop; ++iz) {
                    const uint64_t kk[3] = {ix == 0 ? k[0][0] : ix == 1 ? k[0][1] : k[0][2], iy == 0 ? k[1][0] : iy == 1 ? k[1][1] : k[1][2],
                                            iz == 0 ? k[2][0] : iz == 1 ? k[2][1] : k[2][2]};
                    const double wt = __dmul_rn(__dmul_rn(ix == 0 ? w[0][0] : ix == 1 ? w[0][1] : w[0][2],
                                                          iy == 0 ? w[1][0] : iy == 1 ? w[1][1] : w[1][2]),
                                                iz == 0 ? w[2][0] : iz == 1 ? w[2][1] : w[2][2]);
                    const Found fi = find_near(T, centre, ilvl, cc, kk);
                    lvl = (fi.cell >= 0) ? min(lvl, fi.level) : lvl;
                    if (fi.cell >= 0 && lvl == ilvl) res.add(T, fi.cell, wt);
                    else {
                        res.reset();
                        stop = true;
                    }
                }
    } while (lvl < ilvl);
    return res.field(vv);
}

// the homogeneous field of the FLRW reference and the Born rays
__device__ __forceinline__ Field7 homogeneous_field()
{
    Field7 h;
    clear(h);
    h.a = 1.f;
    return h;
}

// the field at a point: the octree's NGP / CIC / TSC, or the homogeneous field
template <int F>
__device__ __forceinline__ Field7 field_at(const DevTree& T, const PropParams& P, double x, double y, double z, Hint& hint)
{
    if (P.homogeneous) return homogeneous_field();
    if (P.order == 0) return ngp(T, x, y, z);
    return (P.order == 1) ? cic_exact<F, false>(T, x, y, z, hint, nullptr) : tsc_exact<F, false>(T, x, y, z, hint, nullptr);
}

// the field and the velocity at a point of a velocity-field octree (the
// homogeneous field has no velocity: integrator.h:663-664)
__device__ __forceinline__ Field7 field_vel_at(const DevTree& T, const PropParams& P, double x, double y, double z, Hint& hint,
                                               float* v)
{
    v[0] = v[1] = v[2] = 0.f;
    if (P.homogeneous) return homogeneous_field();
    if (P.order == 0) {
        const Found c = locate(T, x, y, z);
        const float4 u = (c.cell >= 0) ? __ldg(T.vel + c.cell) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = u.x; v[1] = u.y; v[2] = u.z;
        return ngp(T, x, y, z);
    }
    return (P.order == 1) ? cic_exact<kAllFields, true>(T, x, y, z, hint, v) : tsc_exact<kAllFields, true>(T, x, y, z, hint, v);
}

// the cell of a trajectory point; the hint moves there
__device__ __forceinline__ Found locate_at(const DevTree& T, const PropParams& P, double x, double y, double z, Hint& hint)
{
    if (P.homogeneous == 1) return Found{0, P.hom_level};
    const uint64_t c32[3] = {axis_coord_bits(kMaxLevel, x), axis_coord_bits(kMaxLevel, y), axis_coord_bits(kMaxLevel, z)};
    return locate_near32(T, c32, hint);
}

// The lanes that trace one ray, and their shared Jacobian points (18 floats).
struct RaySet {
    int per_ray, sub;
    unsigned mask;
    float* points;
};

__device__ __forceinline__ bool vel_zero(const float* v) { return v[0] == 0.f && v[1] == 0.f && v[2] == 0.f; }

// Utility::interpolate with the upper bound carried from call to call: a ray's
// conformal time moves by less than a table interval between two calls
__device__ __forceinline__ double interpolate_near(double x0, const double* __restrict__ x, const double* __restrict__ y, int n, int& first)
{
    while (first < n && !less64(x0, __ldg(x + first))) ++first;
    while (first > 0 && less64(x0, __ldg(x + first - 1))) --first;
    int i = first;
    i += (n > 1) * ((i <= 0) - (i >= n));
    if (n > 1) {
        const double xi = __ldg(x + i), xm = __ldg(x + i - 1), yi = __ldg(y + i), ym = __ldg(y + i - 1);
        return ym + ((yi - ym) * (x0 - xm) / (xi - xm));
    }
    return (n > 0) ? __ldg(y) : 0.0;
}

// geodesic RHS (integrator.h:409-445) from the field at the point; y = 1 /
// scale rounded, first = the upper bound of the conformal time
__device__ __forceinline__ void rhs(const DevCosmo& C, double scale, double y, const Field7& f, const double* in, int& first, double* out)
{
    const double two = 2.0;
    const double c2 = kC * kC;
    const double dt = wide(f.dt), dx = wide(f.dx), dy = wide(f.dy), dz = wide(f.dz);
    const double dphidl = dt * in[5] + (dx * in[6] + dy * in[7] + dz * in[8]);
    const double dadt = interpolate_near(in[1], C.t, C.dadt, C.n, first);
    out[0] = in[5] * dadt;
    out[1] = in[5];
    out[2] = divide_by(in[6], scale, y);
    out[3] = divide_by(in[7], scale, y);
    out[4] = divide_by(in[8], scale, y);
    const double hub = two * dadt / in[0] * in[5];
    out[5] = -(hub * in[5]) - (two / c2 * in[5]) * (dphidl - dt * in[5]);
    const double g = two / c2 * dphidl;
    out[6] = -(hub * in[6]) + (g * in[6]) - (two * dx * in[5] * in[5]);
    out[7] = -(hub * in[7]) + (g * in[7]) - (two * dy * in[5] * in[5]);
    out[8] = -(hub * in[8]) + (g * in[8]) - (two * dz * in[5] * in[5]);
}

__device__ __forceinline__ double plane_q(int kind, const Rec& r, const double* ki = nullptr)
{
    if (kind == STOP_PLANE && ki) return r.x * ki[0] + r.y * ki[1] + r.z * ki[2];
    switch (kind) {
    case STOP_R: return r.chi;
    case STOP_LAMBDA: return r.lambda;
    case STOP_T: return r.t;
    case STOP_A: return r.a;
    case STOP_S: return r.s;
    default: return r.red;
    }
}

__device__ __forceinline__ bool plane_crossed(int kind, const Rec& r, double ref, const double* ki = nullptr)
{
    return (kind == STOP_A) ? (r.a < ref) : (plane_q(kind, r, ki) > ref);
}

// Jacobian running sums at one trajectory point (S1: chi H dr, S2: chi^2 H dr).
struct JSum {
    double s1[3], s2[3];
};

// a11 a12 a22 of the infinitesimal Jacobian at distance d from the sums at
// the last point with chi <= d (lensing.h:459-469)
__device__ __forceinline__ void jac_from_sums(const JSum& J, double d, double length, double* A)
{
    const double c2 = 299792458.0 * 299792458.0;
    const double a11 = J.s1[0] - J.s2[0] / d;
    const double a12 = J.s1[1] - J.s2[1] / d;
    const double a22 = J.s1[2] - J.s2[2] / d;
    A[0] = 1 - 2 * a11 / c2 * length;
    A[1] = -2 * a12 / c2 * length;
    A[2] = 1 - 2 * a22 / c2 * length;
}

// Hessian terms of the Jacobian at a trajectory point (lensing.h:430-447): six
// TSC gathers at +-1 cell, shared out to the ray's lanes.
__device__ void jac_point(const DevTree& T, const Rec& p, const Hint& at, double dr, double* H, const RaySet& R)
{
    const double x = p.x, y = p.y, z = p.z, r = p.chi;
    const double dl = ldexp(1.0, (int)(kLevelShift + 1 - (int)p.level));
    const double h = 0.5 * dl;
    // the plus and minus points of an axis: the components read there
    float g[6][3];
    for (int q = R.sub; q < 6; q += R.per_ray) {
        const int axis = q >> 1;
        const double qx = (axis == 0) ? ((q & 1) ? x + h : x - h) : x;
        const double qy = (axis == 1) ? ((q & 1) ? y + h : y - h) : y;
        const double qz = (axis == 2) ? ((q & 1) ? z + h : z - h) : z;
        Hint hint = at;
        const Field7 f = tsc_exact<kGradient3, false>(T, qx, qy, qz, hint, nullptr);
        float* const o = R.points + 3 * q;
        o[0] = f.dx; o[1] = f.dy; o[2] = f.dz;
    }
    __syncwarp(R.mask);
    for (int q = 0; q < 6; ++q)
        for (int c = 0; c < 3; ++c) g[q][c] = R.points[3 * q + c];
    __syncwarp(R.mask);
    // the direction's sines and cosines from its coordinates; 1 / dl is a power
    // of two
    const double rho = sqrt(x * x + y * y);
    const double cp = (rho > 0.0) ? x / rho : 1.0, sp = (rho > 0.0) ? y / rho : 0.0, ct = z / r, st = rho / r;
    const double s2p = 2.0 * sp * cp, s2t = 2.0 * st * ct;
    const int e = (int)p.level - kLevelShift - 1;
    const double dxxp = times_pow2(wide(g[1][0] - g[0][0]), e);
    const double dxyp = times_pow2(wide(g[3][0] - g[2][0]), e);
    const double dxzp = times_pow2(wide(g[5][0] - g[4][0]), e);
    const double dyyp = times_pow2(wide(g[3][1] - g[2][1]), e);
    const double dyzp = times_pow2(wide(g[5][1] - g[4][1]), e);
    const double dzzp = times_pow2(wide(g[5][2] - g[4][2]), e);
    const double d1d1p = sp * sp * dxxp + cp * cp * dyyp - s2p * dxyp;
    const double d2d2p = cp * cp * ct * ct * dxxp + sp * sp * ct * ct * dyyp + st * st * dzzp + s2p * ct * ct * dxyp -
                         sp * s2t * dyzp - cp * s2t * dxzp;
    const double d1d2p = ct * cp * sp * (dyyp - dxxp) + (cp * cp - sp * sp) * ct * dxyp + sp * st * dxzp - cp * st * dyzp;
    H[0] = d1d1p * dr;
    H[1] = d1d2p * dr;
    H[2] = d2d2p * dr;
}

template <bool SRC>
__device__ void propagate_one(const DevTree& T, const DevCosmo& C, const PropParams& P, const double* L, long long i,
                              const PropOut& O, const RaySet& R)
{
    const double zero = 0.0, one = 1.0, two = 2.0, six = 6.0;
    const double c2 = kC * kC;
    const double mn = 0.0 - (double)kExtent / two, mx = 0.0 + (double)kExtent / two;
    const double scale = P.length;
    const int np = SRC ? 1 : P.nplanes;
    const int kind = SRC ? (int)STOP_R : P.stop_kind;
    const double* rpl = (!SRC && P.ray_planes) ? P.ray_planes + i * np : P.planes;   // this ray's surfaces
    const double stop_ref = SRC ? P.ray_stop[i] : (P.ray_planes ? rpl[np - 1] : P.stop_ref);
    const int rec_fields = SRC ? kSourceFields : (P.wide ? kWideFields : kPlaneFields);
    Rec b;
    if (SRC || P.direct) {
        // launch, (phi, theta) form (src/integrator.h:305-329), or a bundle
        // photon (integrator.h:346-380): direction given
        b.a = one; b.t = zero; b.x = L[0]; b.y = L[1]; b.z = L[2]; b.k0 = one;
        b.k1 = L[3]; b.k2 = L[4]; b.k3 = L[5];
        b.index = 0.0;
    } else {
        // launch (src/integrator.h:283-309, 6-argument form)
        const double norm = sqrt((L[3] - L[0]) * (L[3] - L[0]) + (L[4] - L[1]) * (L[4] - L[1]) + (L[5] - L[2]) * (L[5] - L[2]));
        b.a = one; b.t = zero; b.x = L[0]; b.y = L[1]; b.z = L[2]; b.k0 = one;
        b.k1 = (L[3] - L[0]) / norm; b.k2 = (L[4] - L[1]) / norm; b.k3 = (L[5] - L[2]) / norm;
        b.index = 0.0;
    }
    // Velocity-field octree (the reference built with -DVELOCITYFIELD): the
    // record's velocity slots are gathered with the other fields, count in its
    // emptiness test (data != empty compares every member), and the redshift
    // takes the ISW, Doppler and observer terms (integrator.h:765-767).
    const bool velf = T.vel != nullptr;
    float vel[3] = {0.f, 0.f, 0.f};
    Hint hint{-1, 0, {0u, 0u, 0u}};   // the cell of the last trajectory point
    Found loc = locate_at(T, P, b.x, b.y, b.z, hint);
    Field7 data = velf ? field_vel_at(T, P, b.x, b.y, b.z, hint, vel) : field_at<kAllFields>(T, P, b.x, b.y, b.z, hint);
    {
        const double ph = (double)data.phi / c2;
        const double norm = sqrt((c2 * (one + two * ph) * b.k0 * b.k0) / ((one - two * ph) * (b.k1 * b.k1 + b.k2 * b.k2 + b.k3 * b.k3)));
        b.k1 *= norm; b.k2 *= norm; b.k3 *= norm;
    }
    // v0n: the observer velocity along the launch direction (integrator.h:707-708)
    const double v0n = velf ? (P.vobs[0] * b.k1 + P.vobs[1] * b.k2 + P.vobs[2] * b.k3) / (kC * b.k0) : 0.0;
    b.a = interpolate(b.t, C.t, C.a, C.n);
    b.level = (loc.cell >= 0) ? (double)loc.level : 0.0;
    b.ah = zero;
    b.rho = data.rho; b.phi = data.phi; b.dx = data.dx; b.dy = data.dy; b.dz = data.dz; b.dt = data.dt;
    b.dphidl = zero; b.lap = zero; b.red = zero;
    {
        const double kk = b.k1 * b.k1 + b.k2 * b.k2 + b.k3 * b.k3;
        b.ds2 = (b.a * b.a) * (-(c2 * (one + two * (b.phi / c2)) * b.k0 * b.k0) + ((one - two * (b.phi / c2)) * kk));
        b.err = one - ((one - two * (b.phi / c2)) * kk) / (c2 * (one + two * (b.phi / c2)) * b.k0 * b.k0);
    }
    b.isw = zero; b.chi = zero; b.iswold = zero; b.lambda = zero; b.s = zero;
    double ratio = b.a * b.a * (scale / kC) / P.nsteps;
    double dl = (loc.cell >= 0 ? cell_extent(loc.level) : 0.0) * ratio;
    const double a0 = b.a;
    const double phi0c2 = b.phi / c2;
    double* const traj = O.traj ? O.traj + i * O.traj_cap * kPhotonFields : nullptr;
    if (traj && O.traj_cap > 0) write_rec(traj, b);

    // surfaces
    int next_plane = 0;
    long long cross_k[kMaxPlanes];
    for (int j = 0; j < np; ++j) cross_k[j] = -1;
    double* prow = O.plane_rec ? O.plane_rec + (long long)i * np * rec_fields : nullptr;
    if (SRC && prow) {
        // trajectory[0] as the redshift decomposition reads it (catalogues.h:691-693)
        prow[24] = b.a; prow[25] = b.phi; prow[26] = b.k1; prow[27] = b.k2; prow[28] = b.k3;
        prow[29] = prow[30] = prow[31] = 0.0;
    }
    // a surface crossed by the first point lies at firstid 0: invalid in the map driver
    // this ray's plane normals (stop criterion "plane" with per-ray surfaces)
    const double* rki = (!SRC && P.ray_ki) ? P.ray_ki + (long long)i * np * 3 : nullptr;
    while (next_plane < np && plane_crossed(kind, b, SRC ? stop_ref : rpl[next_plane], rki ? rki + 3 * next_plane : nullptr)) {
        cross_k[next_plane] = 0;
        ++next_plane;
    }
    double rmax_before_b = 0.0;   // max rho over the points before b (std::max_element order)
    bool have_rmax = false;
    // Jacobian sums, at the current point and the two before it
    JSum S{{0, 0, 0}, {0, 0, 0}}, Sm1 = S, Sm2 = S;
    double chim1 = 0.0, chim2 = 0.0;
    long long k = 0;   // index of b
    unsigned status = 0;

    Rec p = b;
    p.isw = zero; p.iswold = zero; p.lambda = zero; p.s = zero;
    double core[9], dc0[9], dc1[9], dc2[9], dc3[9];
    const double inv_scale = __drcp_rn(scale);
    int first = 0;   // upper bound of the ray's conformal time in the table
    // the photon record's fields that no later step reads: formed for every
    // point of a trajectory, else for the last one
    double last_phi = b.phi, last_dl = one;
    float last_dt = data.dt;
    auto record_fields = [&](Rec& r) {
        if (r.index == zero) return;
        r.dphidl = (double)last_dt * r.k0 + (r.dx * r.k1 + r.dy * r.k2 + r.dz * r.k3);
        r.lap = (r.phi - last_phi) / last_dl;
        const double kk = r.k1 * r.k1 + r.k2 * r.k2 + r.k3 * r.k3;
        r.ds2 = (r.a * r.a) * ((-c2 * (one + two * (r.phi / c2)) * r.k0 * r.k0) + ((one - two * (r.phi / c2)) * kk));
        r.err = one - ((one - two * (r.phi / c2)) * kk) / (c2 * (one + two * (r.phi / c2)) * r.k0 * r.k0);
    };
    while (!(is_empty(data) && vel_zero(vel))) {
        if (k >= P.max_steps) { status |= 1u; break; }
        const double bcore[9] = {b.a, b.t, b.x, b.y, b.z, b.k0, b.k1, b.k2, b.k3};
        p.index = b.index + one;
        // the field at b is the one read after the previous step
        rhs(C, scale, inv_scale, data, bcore, first, dc0);
#pragma unroll
        for (int q = 0; q < 9; ++q) core[q] = bcore[q] + dl / two * dc0[q];
        {
            Hint h = hint;
            rhs(C, scale, inv_scale, field_at<kGradient4>(T, P, core[2], core[3], core[4], h), core, first, dc1);
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) core[q] = bcore[q] + dl / two * dc1[q];
        {
            Hint h = hint;
            rhs(C, scale, inv_scale, field_at<kGradient4>(T, P, core[2], core[3], core[4], h), core, first, dc2);
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) core[q] = bcore[q] + dl * dc2[q];
        {
            Hint h = hint;
            rhs(C, scale, inv_scale, field_at<kGradient4>(T, P, core[2], core[3], core[4], h), core, first, dc3);
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) core[q] = bcore[q] + (dl / six) * (dc0[q] + two * dc1[q] + two * dc2[q] + dc3[q]);
        p.a = core[0]; p.t = core[1]; p.x = core[2]; p.y = core[3]; p.z = core[4];
        p.k0 = core[5]; p.k1 = core[6]; p.k2 = core[7]; p.k3 = core[8];
        loc = locate_at(T, P, p.x, p.y, p.z, hint);
        data = velf ? field_vel_at(T, P, p.x, p.y, p.z, hint, vel) : field_at<kAllFields>(T, P, p.x, p.y, p.z, hint);
        if (!(!(p.a < zero) && ((p.x > mn) && (p.x < mx) && (p.y > mn) && (p.y < mx) && (p.z > mn) && (p.z < mx)))) {
            clear(data);
            vel[0] = vel[1] = vel[2] = 0.f;
        }
        p.level = (loc.cell >= 0) ? (double)loc.level : 0.0;
        p.ah = wide(data.a);
        p.rho = wide(data.rho); p.phi = wide(data.phi); p.dx = wide(data.dx); p.dy = wide(data.dy); p.dz = wide(data.dz);
        p.dt = -wide(data.dt);
        p.isw += (b.dt + p.dt) * (p.t - b.t) / c2;
        if (O.final_rec || traj)   // photon records only
            p.iswold -= 2 * (p.phi - b.phi) / c2 -
                    ((b.dx + p.dx) * (p.x - b.x) * scale + (b.dy + p.dy) * (p.y - b.y) * scale + (b.dz + p.dz) * (p.z - b.z) * scale) / c2;
        p.chi = sqrt(p.x * p.x + p.y * p.y + p.z * p.z);
        p.lambda += dl;
        p.s += sqrt((p.x - b.x) * (p.x - b.x) + (p.y - b.y) * (p.y - b.y) + (p.z - b.z) * (p.z - b.z));
        if (velf) {
            const double dop = ((double)vel[0] * p.k1 + (double)vel[1] * p.k2 + (double)vel[2] * p.k3) / (kC * p.k0);
            p.red = a0 / p.a * (one + phi0c2 - p.phi / c2 + p.isw + dop - v0n) - one;
        } else {
            p.red = a0 / p.a * (one + phi0c2 - p.phi / c2) - one;
        }
        bool appended = false;
        double step = dl;
        if (!(is_empty(data) && vel_zero(vel))) {
            step = dl;
            ratio = p.a * p.a * (scale / kC) / P.nsteps;
            dl = (loc.cell >= 0 ? cell_extent(loc.level) : 0.0) * ratio;
            appended = true;
        }
        if (appended) {
            // the new point p becomes trajectory[k+1]; b is trajectory[k]
            ++k;
            last_phi = b.phi;
            last_dl = step;
            last_dt = data.dt;
            if (P.jacobian) {
                double H[3];
                jac_point(T, p, hint, p.chi - b.chi, H, R);
                Sm2 = Sm1; Sm1 = S;
                chim2 = chim1; chim1 = b.chi;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    S.s1[q] += p.chi * H[q];
                    S.s2[q] += p.chi * p.chi * H[q];
                }
            }
            while (next_plane < np && plane_crossed(kind, p, SRC ? stop_ref : rpl[next_plane], rki ? rki + 3 * next_plane : nullptr)) {
                const int j = next_plane++;
                cross_k[j] = k;
                if (prow) {
                    double* o = prow + j * rec_fields;
                    const double ref = SRC ? stop_ref : rpl[j];
                    const double* kj = rki ? rki + 3 * j : nullptr;
                    const double q1 = plane_q(kind, p, kj), q0 = plane_q(kind, b, kj);
                    const double f = (q1 - ref) / (q1 - q0);
                    const double px = b.x * f + p.x * (1 - f), py = b.y * f + p.y * (1 - f), pz = b.z * f + p.z * (1 - f);
                    const double dist = sqrt(px * px + py * py + pz * pz);
                    o[0] = (double)(k - 1); o[1] = f; o[2] = px; o[3] = py; o[4] = pz; o[5] = dist;
                    o[9] = b.t * f + p.t * (1 - f);
                    o[10] = b.a * f + p.a * (1 - f);
                    o[11] = b.red * f + p.red * (1 - f);
                    o[12] = b.chi * f + p.chi * (1 - f);
                    o[13] = b.lambda * f + p.lambda * (1 - f);
                    o[14] = b.s * f + p.s * (1 - f);
                    o[15] = b.isw * f + p.isw * (1 - f);
                    o[16] = b.rho * f + p.rho * (1 - f);
                    o[17] = b.phi * f + p.phi * (1 - f);
                    // max rho over points [0, firstid) = [0, k-1): all points before b
                    o[18] = have_rmax ? rmax_before_b : 0.0;
                    o[19] = 1.0;
                    if (SRC || P.wide) {
                        o[20] = b.k0 * f + p.k0 * (1 - f);
                        o[21] = b.k1 * f + p.k1 * (1 - f);
                        o[22] = b.k2 * f + p.k2 * (1 - f);
                        o[23] = b.k3 * f + p.k3 * (1 - f);
                    }
                    if (P.jacobian) {
                        // the Jacobian at the surface's distance (hmaps.h:653-656),
                        // or at the source radius or Born surface radius itself
                        // (catalogues.h:517, hmaps.h:712)
                        const double jd = (SRC || P.homogeneous == 2) ? ref : dist;
                        // last point with chi <= jd among k, k-1, k-2
                        const JSum* J = nullptr;
                        if (p.chi <= jd) J = &S;
                        else if (chim1 <= jd) J = &Sm1;
                        else if (k >= 2 && chim2 <= jd) J = &Sm2;
                        double A[3] = {1.0, 0.0, 1.0};
                        if (J) {
                            jac_from_sums(*J, jd, P.length, A);
                        } else {
                            status |= 2u;
                        }
                        o[6] = A[0]; o[7] = A[1]; o[8] = A[2];
                    } else {
                        o[6] = o[7] = o[8] = 0.0;
                    }
                }
            }
            // b moves behind the new point: fold it into the running maximum
            if (!have_rmax || rmax_before_b < b.rho) rmax_before_b = b.rho;
            have_rmax = true;
            b = p;
            if (traj) {
                record_fields(b);
                if (k < O.traj_cap) write_rec(traj + k * kPhotonFields, b);
                else status |= 8u;
            }
        }
        // stop test on trajectory.back()
        bool stop = false;
        switch (kind) {
        case STOP_R: stop = b.chi > stop_ref; break;
        case STOP_LAMBDA: stop = b.lambda > stop_ref; break;
        case STOP_REDSHIFT: stop = b.red > stop_ref; break;
        case STOP_T: stop = b.t > stop_ref; break;
        case STOP_A: stop = b.a < stop_ref; break;
        case STOP_PLANE: {
            const double* kk = rki ? rki + 3 * (np - 1) : P.ki;
            stop = (p.x * kk[0] + p.y * kk[1] + p.z * kk[2]) > stop_ref;
            break;
        }
        case STOP_S: stop = b.s > stop_ref; break;
        default: stop = true;
        }
        if (stop) break;
    }
    // drop the last point when its redshift or scale factor is negative
    long long size = k + 1;
    if (signbit(b.red) || signbit(b.a)) size -= 1;
    O.steps[i] = size;
    if (O.final_rec) {
        double* o = O.final_rec + i * kPhotonFields;
        if (size == k + 1) {
            record_fields(b);
            write_rec(o, b);
        }
        else {
            // the popped point is not reported; the record before it is not kept,
            // so report zeros with the step count (only rays ending at z<0 or a<0)
            for (int q = 0; q < kPhotonFields; ++q) o[q] = 0.0;
            status |= 4u;
        }
    }
    if (SRC && prow) {
        // the source is reached when the last kept point is the crossing
        // (catalogues.h:433-442: marked > 0 and chi(marked) >= radius)
        const long long ck = cross_k[0];
        const bool ok = (ck >= 1) && (ck < size);
        if (!ok) {
            for (int q = 0; q < 24; ++q) prow[q] = 0.0;
            const long long marked = size - 1;
            prow[0] = (double)(marked - (marked > 0));
            // a Born ray that ends short of the radius: the Jacobian at its last point
            if (P.homogeneous == 2 && P.jacobian && ck < 0) jac_from_sums(S, stop_ref, P.length, prow + 6);
        }
        prow[19] = ok ? 1.0 : 0.0;
    } else if (prow) {
        for (int j = 0; j < np; ++j) {
            double* o = prow + j * rec_fields;
            const long long ck = cross_k[j];
            const bool found = (ck >= 1) && (ck < size);
            // map driver: firstid == size-1 or firstid == 0 -> invalid
            const bool valid = found && !((ck - 1) == size - 1 || (ck - 1) == 0);
            if (ck < 0 || ck == 0 || ck >= size) {
                for (int q = 0; q < (P.wide ? 24 : kPlaneFields); ++q) o[q] = 0.0;
                o[0] = (ck == 0) ? 0.0 : (double)(size - 1);
            }
            o[19] = valid ? 1.0 : 0.0;
            if (P.wide) o[24] = found ? 1.0 : 0.0;
            if (P.homogeneous == 2) {
                // Born ray (hmaps.h:712, 719): the Jacobian at the surface radius
                // (from the last point when the ray never got there); only a
                // ray that could not take a step is unusable
                if (P.jacobian && ck < 0) jac_from_sums(S, rpl[j], P.length, o + 6);
                o[19] = (size > 1) ? 1.0 : 0.0;
            }
        }
    }
    if (status) atomicOr(O.status, status);
}

// Each block is `warps` warps of `rays` rays with per_ray lanes each
// (rays x per_ray <= 32); the rays' results do not depend on the shape.
template <bool SRC>
__global__ void __launch_bounds__(128) k_propagate(DevTree T, DevCosmo C, PropParams P, const double* __restrict__ launch,
                                                   long long n, PropOut O, int rays, int per_ray)
{
    __shared__ float points[18 * 128];
    const int lane = threadIdx.x & 31, ray = lane / per_ray;
    const long long i = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * rays + ray;
    if (ray >= rays || i >= n) return;
    RaySet R;
    R.per_ray = per_ray;
    R.sub = lane % per_ray;
    R.mask = ((1u << per_ray) - 1u) << (lane - R.sub);
    R.points = points + 18 * (threadIdx.x - R.sub);
    propagate_one<SRC>(T, C, P, launch + 6 * i, i, O, R);
}

}  // namespace mpf
