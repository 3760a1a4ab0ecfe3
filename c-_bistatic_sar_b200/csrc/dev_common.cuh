// dev_common.cuh -- device-side DEM view and the reference's DEM / Fermat arithmetic.
//
// Everything in the FP64 section keeps the reference's operation order (sqrt and division
// are IEEE correctly rounded in CUDA, as on the host).  The units whose results reproduce the
// reference's bit for bit are compiled with --fmad=false (k_plain.cu, k_pulse.cu, k_synth.cu);
// k_mixed.cu, k_newton.cu and k_crossings.cu use the DEM lookup, the flat start and the facets
// with contraction on, within their tolerances.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "dev_view.hpp"

namespace bsar {

// std::min / std::max as libstdc++ defines them (their NaN order is part of the result).
__device__ __forceinline__ double std_min(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double std_max(double a, double b) { return (a < b) ? b : a; }

// First i with v[i] <= x <= v[i+1] (the reference's linear scan,
// src/raw_data_processing.cpp:625-640); -1 when none.  For non-decreasing axes the
// first match is found by a lower bound over v[1..n-1]; otherwise by the scan itself.
__device__ __forceinline__ int axis_interval(const double* __restrict__ v, int n, double x, int asc)
{
    if (n < 2) return -1;
    if (asc) {
        int lo = 1, hi = n;
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (__ldg(v + mid) < x) lo = mid + 1; else hi = mid;
        }
        if (lo >= n) return -1;
        int i = lo - 1;
        return (x >= __ldg(v + i) && x <= __ldg(v + i + 1)) ? i : -1;
    }
    for (int i = 0; i + 1 < n; i++)
        if (x >= __ldg(v + i) && x <= __ldg(v + i + 1)) return i;
    return -1;
}

// One axis of interpolateDEMElevation: indices (i0, i1) and the clamped weight,
// src/raw_data_processing.cpp:621-671.  An unmatched axis keeps (0, 0), its span is
// replaced by 1.0 and the weight is clamp(x - v[0], 0, 1).
struct AxisLookup {
    int i0, i1;
    double w;
};

__device__ __forceinline__ AxisLookup axis_lookup(const double* __restrict__ v, int n, double x, int asc)
{
    AxisLookup r;
    int i = axis_interval(v, n, x, asc);
    r.i0 = i < 0 ? 0 : i;
    r.i1 = i < 0 ? 0 : i + 1;
    double d = __ldg(v + r.i1) - __ldg(v + r.i0);
    if (d == 0) d = 1.0;
    double w = (x - __ldg(v + r.i0)) / d;
    r.w = std_max(0.0, std_min(1.0, w));
    return r;
}

// The same on a strictly ascending, equally spaced axis (v0, inv: its first node and
// 1 / spacing): the interval is a guess away, moved to the first match by the scan's own
// comparisons.
__device__ __forceinline__ AxisLookup axis_lookup_even(const double* __restrict__ v, int n, double x, double v0, double inv)
{
    AxisLookup r;
    r.i0 = r.i1 = 0;
    if (x >= v0 && x <= __ldg(v + n - 1)) {
        int i = min(max((int)((x - v0) * inv), 0), n - 2);
        while (i > 0 && x <= __ldg(v + i)) i--;
        while (i < n - 2 && x > __ldg(v + i + 1)) i++;
        r.i0 = i;
        r.i1 = i + 1;
    }
    double d = __ldg(v + r.i1) - __ldg(v + r.i0);
    if (d == 0) d = 1.0;
    double w = (x - __ldg(v + r.i0)) / d;
    r.w = std_max(0.0, std_min(1.0, w));
    return r;
}

// The height combination of interpolateDEMElevation, :649-677.
__device__ __forceinline__ double dem_combine(const DemView& d, const AxisLookup& ax, const AxisLookup& ay)
{
    const double* __restrict__ Z = d.z;
    double z00 = __ldg(Z + (int64_t)ay.i0 * d.nx + ax.i0);
    if (ax.i0 == ax.i1 && ay.i0 == ay.i1) return z00;
    double z01 = __ldg(Z + (int64_t)ay.i0 * d.nx + ax.i1);
    double z10 = __ldg(Z + (int64_t)ay.i1 * d.nx + ax.i0);
    double z11 = __ldg(Z + (int64_t)ay.i1 * d.nx + ax.i1);
    double wx = ax.w, wy = ay.w;
    return z00 * (1 - wx) * (1 - wy) + z01 * wx * (1 - wy) + z10 * (1 - wx) * wy + z11 * wx * wy;
}

// interpolateDEMElevation, src/raw_data_processing.cpp:615-680.
__device__ __forceinline__ double dem_elevation(const DemView& d, double x, double y)
{
    if (d.empty) return 0.0;
    AxisLookup ax = axis_lookup(d.xv, d.nx, x, d.asc_x);
    AxisLookup ay = axis_lookup(d.yv, d.ny, y, d.asc_y);
    return dem_combine(d, ax, ay);
}

// Optical path n1*|X-P1| + n2*|P2-X| as the grid search writes it (:532-534).
__device__ __forceinline__ double grid_optical(double px, double py, double pz, double x1, double y1,
                                               double z1, double x2, double y2, double z2,
                                               double n1, double n2)
{
    double d1 = sqrt((px - x1) * (px - x1) + (py - y1) * (py - y1) + (pz - z1) * (pz - z1));
    double d2 = sqrt((x2 - px) * (x2 - px) + (y2 - py) * (y2 - py) + (z2 - pz) * (z2 - pz));
    return n1 * d1 + n2 * d2;
}

// One level of the reference's grid search (:509-551) with a G x G grid.  The y-axis
// lookups of the G columns do not depend on the row, so they are made once per level.
// Column tables of one search level in shared memory, [column][thread] (consecutive
// lanes, consecutive words): the G column positions and y-axis lookups stay out of the
// registers.  TPB is the largest block the calling kernel launches with.
template <int TPB> struct GridCols {
    double py[15][TPB];
    double w[15][TPB];
    int2 ii[15][TPB];
};

template <int G, int TPB>
__device__ __forceinline__ void grid_level(const DemView& d, double x1, double y1, double z1,
                                           double x2, double y2, double z2, double n1, double n2,
                                           double R, double& bestX, double& bestY, double& minOP,
                                           GridCols<TPB>* cols)
{
    const double minX = bestX - R, maxX = bestX + R;
    const double minY = bestY - R, maxY = bestY + R;
    const int t = threadIdx.x;
#pragma unroll
    for (int j = 0; j < G; j++) {
        const double py = minY + j * (maxY - minY) / (G - 1);
        cols->py[j][t] = py;
        if (!d.empty) {
            const AxisLookup a = axis_lookup(d.yv, d.ny, py, d.asc_y);
            cols->w[j][t] = a.w;
            cols->ii[j][t] = make_int2(a.i0, a.i1);
        }
    }
    for (int i = 0; i < G; i++) {
        double px = minX + i * (maxX - minX) / (G - 1);
        AxisLookup ax;
        if (!d.empty) ax = axis_lookup(d.xv, d.nx, px, d.asc_x);
#pragma unroll
        for (int j = 0; j < G; j++) {
            const double py = cols->py[j][t];
            double pz = 0.0;
            if (!d.empty) {
                const int2 ii = cols->ii[j][t];
                const AxisLookup ay{ii.x, ii.y, cols->w[j][t]};
                pz = dem_combine(d, ax, ay);
            }
            double op = grid_optical(px, py, pz, x1, y1, z1, x2, y2, z2, n1, n2);
            if (op < minOP) {
                minOP = op;
                bestX = px;
                bestY = py;
            }
        }
    }
}

// One point of a search level, exactly as grid_level evaluates it: position, height, path.
struct GridPoint {
    double x, y, op;
};

template <int G>
__device__ __forceinline__ GridPoint grid_point(const DemView& d, double x1, double y1, double z1, double x2, double y2,
                                                double z2, double n1, double n2, double minX, double maxX, double minY,
                                                double maxY, double invx, double invy, int i, int j)
{
    GridPoint p;
    p.x = minX + i * (maxX - minX) / (G - 1);
    p.y = minY + j * (maxY - minY) / (G - 1);
    double pz = 0.0;
    if (!d.empty) {
        const AxisLookup ax = d.uniform && d.nx > 1 ? axis_lookup_even(d.xv, d.nx, p.x, d.x0, invx)
                                                    : axis_lookup(d.xv, d.nx, p.x, d.asc_x);
        const AxisLookup ay = d.uniform && d.ny > 1 ? axis_lookup_even(d.yv, d.ny, p.y, d.y0, invy)
                                                    : axis_lookup(d.yv, d.ny, p.y, d.asc_y);
        pz = dem_combine(d, ax, ay);
    }
    p.op = grid_optical(p.x, p.y, pz, x1, y1, z1, x2, y2, z2, n1, n2);
    return p;
}

// One search level by a whole warp: lanes take the points in turn, the warp keeps the
// smallest path and, among equal ones, the first point -- the scan's strict <.
template <int G>
__device__ __forceinline__ void grid_level_warp(const DemView& d, double x1, double y1, double z1, double x2, double y2,
                                                double z2, double n1, double n2, double invx, double invy, double R,
                                                double& bestX, double& bestY, double& minOP)
{
    const unsigned full = 0xffffffffu;
    const double minX = bestX - R, maxX = bestX + R;
    const double minY = bestY - R, maxY = bestY + R;
    double op = INFINITY, px = 0.0, py = 0.0;
    int at = 0x7fffffff;
#pragma unroll 1
    for (int k = threadIdx.x & 31; k < G * G; k += 32) {
        const GridPoint p = grid_point<G>(d, x1, y1, z1, x2, y2, z2, n1, n2, minX, maxX, minY, maxY, invx, invy, k / G,
                                          k % G);
        if (p.op < op) {
            op = p.op;
            px = p.x;
            py = p.y;
            at = k;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double q = __shfl_xor_sync(full, op, o), qx = __shfl_xor_sync(full, px, o), qy = __shfl_xor_sync(full, py, o);
        const int qa = __shfl_xor_sync(full, at, o);
        if (q < op || (q == op && qa < at)) {
            op = q;
            px = qx;
            py = qy;
            at = qa;
        }
    }
    if (op < minOP) {
        minOP = op;
        bestX = px;
        bestY = py;
    }
}

// calculateRefractionPoint by a whole warp (all 32 lanes call with one pair); the same
// point, bit for bit, as one thread's scan.
__device__ __forceinline__ void refraction_grid_warp(const DemView& d, double x1, double y1, double z1, double x2,
                                                     double y2, double z2, double n1, double n2, double out[3])
{
    double bestX = (x1 + x2) / 2.0;
    double bestY = (y1 + y2) / 2.0;
    double dd = sqrt((x2 - x1) * (x2 - x1) + (y2 - y1) * (y2 - y1));
    double R = std_max(dd, 500.0);
    double minOP = 1e9;
    const double invx = 1.0 / d.stepx, invy = 1.0 / d.stepy;
    grid_level_warp<15>(d, x1, y1, z1, x2, y2, z2, n1, n2, invx, invy, R, bestX, bestY, minOP);
    R /= 5.0;
#pragma unroll 1
    for (int level = 1; level < 5; level++) {
        grid_level_warp<11>(d, x1, y1, z1, x2, y2, z2, n1, n2, invx, invy, R, bestX, bestY, minOP);
        R /= 3.0;
    }
    out[0] = bestX;
    out[1] = bestY;
    out[2] = dem_elevation(d, bestX, bestY);
}

// ------------------------- search levels behind an FP32 filter -----------------------
// For the back-projection, where a warp's lanes search for 32 pulses of one voxel: a level's
// points are first valued in FP32 against the DEM's FP32 heights, and only points whose
// value, less its error bound, does not exceed an upper bound of the level's minimum are
// evaluated in FP64, in the scan's order with its strict <.  Every other point is larger than
// the minimum, so the result is the scan's, bit for bit.
//   upper bound   the path at the level's centre point, which is one of its points (level 0)
//                 or the point the search already holds (later levels); then the smallest
//                 FP32 value plus its error bound
//   error bound   2e-6 of the FP32 path plus (n1 + n2) times 4e-7 of the endpoints' heights and
//                 2.5e-6 of the largest of the cell's corners (rows and columns: of the DEM):
//                 FP32 rounding of offsets, heights and square roots is below 5e-7 of them, and
//                 an interpolated height is off by the weights' 3.6e-7 times the span of the
//                 corners, per axis.  The DEM's largest height for every point would be 3 %
//                 faster, and 2.7 times slower beside no-data values
//   rows, columns a row's path is at least n1 sqrt(dx1^2 + h1^2) + n2 sqrt(dx2^2 + h2^2), h1
//                 and h2 the endpoints' distances from the DEM's range of heights; rows and
//                 columns above the bound for every lane are skipped
//   outside       an axis value within 1e-9 of the DEM's edge (relative) may fall on either
//                 side of it, where the lookup jumps: always evaluated
// Where it holds: grid_filter_ok (kernels.hpp).  All 32 lanes call.  TPB: the block size.
// What bounds it: FP32 issue and the FP64 evaluations left (one to three points a level).
// 41 x 41 x 21 voxels x 256 pulses, mean legs, with upload and upsampling: 107 -> 24.2 ms on
// one B200 against every point in FP64 (grid_level).  That is at six CTAs per SM (80 registers);
// four, which the compiler takes by itself, 25.4 ms; five 32 ms (spills in the point loop).
template <int TPB> struct FilterCols {
    float4 c[15][TPB];     // (y - y1)^2, (y - y2)^2, weight, row offset (int; < 0: at the edge)
};

struct FilterAxis {
    float w;
    int i;        // cell, or 0 with weight 0 outside
    bool edge;
};

__device__ __forceinline__ FilterAxis filter_axis(const double* __restrict__ v, int n, double x, double v0, double inv)
{
    FilterAxis r{0.0f, 0, false};
    const double vn = __ldg(v + n - 1), eps = 1e-9 * (fabs(v0) + fabs(vn) + 1.0);
    r.edge = fabs(x - v0) < eps || fabs(x - vn) < eps;
    if (x >= v0 && x <= vn) {
        int i = min(max((int)((x - v0) * inv), 0), n - 2);
        double a = __ldg(v + i), b = __ldg(v + i + 1);
        if (x < a && i > 0) {
            i--;
            b = a;
            a = __ldg(v + i);
        } else if (x > b && i < n - 2) {
            i++;
            a = b;
            b = __ldg(v + i + 1);
        }
        r.i = i;
        r.w = fminf(fmaxf(__fdividef((float)(x - a), (float)(b - a)), 0.0f), 1.0f);
    }
    return r;
}

template <int G, int TPB>
__device__ __forceinline__ void grid_level_filter(const DemView& d, int pitch, float zlo, float zhi, double x1, double y1,
                                                  double z1, double x2, double y2, double z2, double n1, double n2,
                                                  double invx, double invy, double R, double& bestX, double& bestY,
                                                  double& minOP, FilterCols<TPB>* cols)
{
    const unsigned full = 0xffffffffu;
    const double minX = bestX - R, maxX = bestX + R;
    const double minY = bestY - R, maxY = bestY + R;
    auto point = [&](int i, int j) {
        return grid_point<G>(d, x1, y1, z1, x2, y2, z2, n1, n2, minX, maxX, minY, maxY, invx, invy, i, j);
    };
    const int t = threadIdx.x;
    const float n1f = (float)n1, n2f = (float)n2;
    const float z1f = (float)(z1 - d.z0), z2f = (float)(z2 - d.z0);
    const float base_err = 4e-7f * (n1f + n2f) * (fabsf(z1f) + fabsf(z2f));
    const float zerr = 2.5e-6f * (n1f + n2f), z_err = fmaf(zerr, fmaxf(fabsf(zlo), fabsf(zhi)), base_err);
    double top = minOP;
    if (G == 15) top = fmin(top, point((G - 1) / 2, (G - 1) / 2).op);
    // bound of the level's minimum, rounded up
    float thr = (float)top * (1.0f + 1e-6f) + base_err;
    const double sx = (maxX - minX) / (G - 1), sy = (maxY - minY) / (G - 1);
    auto clear = [&](float z) { return fmaxf(fmaxf(zlo - z, z - zhi), 0.0f) * (1.0f - 1e-6f); };
    const float h1 = clear(z1f) * clear(z1f), h2 = clear(z2f) * clear(z2f);
    auto far = [&](float a2, float b2) {      // a row or column none of whose points can win
        const float qa = a2 + h1, qb = b2 + h2;
        const float L = n1f * (qa * rsqrtf(fmaxf(qa, 1e-30f))) + n2f * (qb * rsqrtf(fmaxf(qb, 1e-30f)));
        return L - 2e-6f * L - z_err > thr;
    };
    unsigned keep = 0;                        // columns to visit (of the warp)
#pragma unroll 1
    for (int j = 0; j < G; j++) {
        const double py = minY + j * sy;
        const float a = (float)(py - y1), b = (float)(py - y2);
        if (!__any_sync(full, !far(a * a, b * b))) continue;
        keep |= 1u << j;
        const FilterAxis f = filter_axis(d.yv, d.ny, py, d.y0, invy);
        cols->c[j][t] = make_float4(a * a, b * b, f.w, __int_as_float(f.edge ? -1 : f.i * pitch));
    }
    // the (up to) three lowest points of this lane, and the value of the fourth
    float v0 = INFINITY, v1 = INFINITY, v2 = INFINITY, v3 = INFINITY;
    int k0 = -1, k1 = -1, k2 = -1;
#pragma unroll 1
    for (int i = 0; i < G; i++) {
        const double px = minX + i * sx;
        const float a = (float)(px - x1), b = (float)(px - x2);
        const float a2 = a * a, b2 = b * b;
        if (!__any_sync(full, !far(a2, b2))) continue;
        const FilterAxis fx = filter_axis(d.xv, d.nx, px, d.x0, invx);
        const float* __restrict__ zc = d.z32 + fx.i;
#pragma unroll 1
        for (unsigned rest = keep; rest; rest &= rest - 1) {
            const int j = __ffs(rest) - 1;
            const float4 c = cols->c[j][t];
            const int off = __float_as_int(c.w);
            const float* r0 = zc + max(off, 0);
            const float* r1 = r0 + pitch;
            const float z00 = __ldg(r0), z01 = __ldg(r0 + 1), z10 = __ldg(r1), z11 = __ldg(r1 + 1);
            const float za = fmaf(fx.w, z01 - z00, z00), zb = fmaf(fx.w, z11 - z10, z10);
            const float z = fmaf(c.z, zb - za, za);
            const float dz1 = z - z1f, dz2 = z - z2f;
            const float q1 = fmaf(dz1, dz1, a2 + c.x), q2 = fmaf(dz2, dz2, b2 + c.y);
            const float L = n1f * (q1 * rsqrtf(fmaxf(q1, 1e-30f))) + n2f * (q2 * rsqrtf(fmaxf(q2, 1e-30f)));
            const float zmax = fmaxf(fmaxf(fabsf(z00), fabsf(z01)), fmaxf(fabsf(z10), fabsf(z11)));
            const float err = fmaf(2e-6f, L, fmaf(zerr, zmax, base_err));
            const bool edge = off < 0 || fx.edge;
            const float low = edge ? -INFINITY : L - err;
            thr = edge ? thr : fminf(thr, L + err);
            if (low < v3 && low <= thr) {
                const int k = i * G + j;
                const bool p0 = low < v0, p1 = low < v1, p2 = low < v2;
                v3 = p2 ? v2 : low;
                v2 = p2 ? (p1 ? v1 : low) : v2;
                k2 = p2 ? (p1 ? k1 : k) : k2;
                v1 = p1 ? (p0 ? v0 : low) : v1;
                k1 = p1 ? (p0 ? k0 : k) : k1;
                v0 = p0 ? low : v0;
                k0 = p0 ? k : k0;
            }
        }
    }
    if (v3 <= thr) {
        // more than three near the minimum: this lane scans the level
#pragma unroll 1
        for (int k = 0; k < G * G; k++) {
            const GridPoint p = point(k / G, k % G);
            if (p.op < minOP) {
                minOP = p.op;
                bestX = p.x;
                bestY = p.y;
            }
        }
        return;
    }
    // those within the final bound, in the scan's order
    if (!(v0 <= thr)) k0 = -1;
    if (!(v1 <= thr)) k1 = -1;
    if (!(v2 <= thr)) k2 = -1;
    const int lo = min(k0, min(k1, k2)), hi = max(k0, max(k1, k2));
    const int mid = k0 + k1 + k2 - lo - hi;
    double nx = bestX, ny = bestY;
#pragma unroll 1
    for (int s = 0; s < 3; s++) {
        const int k = s == 0 ? lo : (s == 1 ? mid : hi);
        if (k < 0) continue;
        const GridPoint p = point(k / G, k % G);
        if (p.op < minOP) {
            minOP = p.op;
            nx = p.x;
            ny = p.y;
        }
    }
    bestX = nx;
    bestY = ny;
}

template <int TPB>
__device__ __forceinline__ void refraction_grid_filter(const DemView& d, int pitch, float zlo, float zhi, double x1,
                                                       double y1, double z1, double x2, double y2, double z2, double n1,
                                                       double n2, FilterCols<TPB>* cols, double out[3])
{
    double bestX = (x1 + x2) / 2.0;
    double bestY = (y1 + y2) / 2.0;
    double dd = sqrt((x2 - x1) * (x2 - x1) + (y2 - y1) * (y2 - y1));
    double R = std_max(dd, 500.0);
    double minOP = 1e9;
    const double invx = 1.0 / d.stepx, invy = 1.0 / d.stepy;
    grid_level_filter<15, TPB>(d, pitch, zlo, zhi, x1, y1, z1, x2, y2, z2, n1, n2, invx, invy, R, bestX, bestY, minOP,
                               cols);
    R /= 5.0;
#pragma unroll 1
    for (int level = 1; level < 5; level++) {
        grid_level_filter<11, TPB>(d, pitch, zlo, zhi, x1, y1, z1, x2, y2, z2, n1, n2, invx, invy, R, bestX, bestY,
                                   minOP, cols);
        R /= 3.0;
    }
    const AxisLookup ax = axis_lookup_even(d.xv, d.nx, bestX, d.x0, invx);
    const AxisLookup ay = axis_lookup_even(d.yv, d.ny, bestY, d.y0, invy);
    out[0] = bestX;
    out[1] = bestY;
    out[2] = dem_combine(d, ax, ay);
}

// calculateRefractionPoint, src/raw_data_processing.cpp:455-572.
template <int TPB>
__device__ __forceinline__ void refraction_grid(const DemView& d, double x1, double y1, double z1,
                                                double x2, double y2, double z2, double n1,
                                                double n2, GridCols<TPB>* cols, double out[3])
{
    double bestX = (x1 + x2) / 2.0;
    double bestY = (y1 + y2) / 2.0;
    double dd = sqrt((x2 - x1) * (x2 - x1) + (y2 - y1) * (y2 - y1));
    double R = std_max(dd, 500.0);
    double minOP = 1e9;
    grid_level<15, TPB>(d, x1, y1, z1, x2, y2, z2, n1, n2, R, bestX, bestY, minOP, cols);
    R /= 5.0;
#pragma unroll 1
    for (int level = 1; level < 5; level++) {
        grid_level<11, TPB>(d, x1, y1, z1, x2, y2, z2, n1, n2, R, bestX, bestY, minOP, cols);
        R /= 3.0;
    }
    out[0] = bestX;
    out[1] = bestY;
    out[2] = dem_elevation(d, bestX, bestY);
}

// ---------------------------------------------------------------------------------
// Newton Fermat solver, FP64.  Steps: flat-interface Snell start; node scan of
// +-W DEM nodes around it; active-set projected Newton on the facets sharing the best
// node; one final step on the winning facet.  (No reference counterpart; the oracle's
// bo_refraction_newton restates it.)
// ---------------------------------------------------------------------------------
constexpr int kFlatIters = 4;
constexpr int kPolishIters = 3;

struct Facet64 {
    double x0, y0, dx, dy, z00, b, c, e;
};

__device__ __forceinline__ void facet_load(const DemView& d, int fi, int fj, Facet64& F)
{
    const double* __restrict__ Z = d.z;
    int64_t nx = d.nx;
    F.x0 = __ldg(d.xv + fi);
    F.y0 = __ldg(d.yv + fj);
    F.dx = __ldg(d.xv + fi + 1) - F.x0;
    F.dy = __ldg(d.yv + fj + 1) - F.y0;
    double z00 = __ldg(Z + fj * nx + fi), z01 = __ldg(Z + fj * nx + fi + 1);
    double z10 = __ldg(Z + (fj + 1) * nx + fi), z11 = __ldg(Z + (fj + 1) * nx + fi + 1);
    F.z00 = z00;
    F.b = z01 - z00;
    F.c = z10 - z00;
    F.e = z11 - z01 - z10 + z00;
}

__device__ __forceinline__ double clamp01(double t) { return t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t); }

__device__ __forceinline__ bool facet_step(const Facet64& F, const double A[3], const double B[3],
                                           double na, double nb, double& u, double& v)
{
    double x = F.x0 + u * F.dx, y = F.y0 + v * F.dy;
    double h = F.z00 + F.b * u + F.c * v + F.e * u * v;
    double zx = (F.b + F.e * v) / F.dx;
    double zy = (F.c + F.e * u) / F.dy;
    double zxy = F.e / (F.dx * F.dy);
    double r1x = x - A[0], r1y = y - A[1], r1z = h - A[2];
    double r2x = x - B[0], r2y = y - B[1], r2z = h - B[2];
    double q1 = r1x * r1x + r1y * r1y + r1z * r1z;
    double q2 = r2x * r2x + r2y * r2y + r2z * r2z;
    double g1 = na / sqrt(q1), g2 = nb / sqrt(q2);
    double a1x = r1x + r1z * zx, a1y = r1y + r1z * zy;
    double a2x = r2x + r2z * zx, a2y = r2y + r2z * zy;
    double gx = g1 * a1x + g2 * a2x;
    double gy = g1 * a1y + g2 * a2y;
    double txx = 1.0 + zx * zx, tyy = 1.0 + zy * zy, txy = zx * zy;
    double hxx = g1 * (txx - a1x * a1x / q1) + g2 * (txx - a2x * a2x / q2);
    double hyy = g1 * (tyy - a1y * a1y / q1) + g2 * (tyy - a2y * a2y / q2);
    double hxy = g1 * (txy - a1x * a1y / q1) + g2 * (txy - a2x * a2y / q2) + (g1 * r1z + g2 * r2z) * zxy;
    bool au = (u <= 0.0 && gx > 0.0) || (u >= 1.0 && gx < 0.0);
    bool av = (v <= 0.0 && gy > 0.0) || (v >= 1.0 && gy < 0.0);
    double gs = g1 + g2;
    double su, sv;
    if (au && av) return false;
    if (au) {
        su = 0.0;
        sv = (hyy > 0.0) ? -gy / hyy : -gy / gs;
    } else if (av) {
        sv = 0.0;
        su = (hxx > 0.0) ? -gx / hxx : -gx / gs;
    } else {
        double det = hxx * hyy - hxy * hxy;
        if (det > 0.0 && hxx > 0.0) {
            su = -(hyy * gx - hxy * gy) / det;
            sv = -(hxx * gy - hxy * gx) / det;
        } else {
            su = -gx / gs;
            sv = -gy / gs;
        }
    }
    u = clamp01(u + su / F.dx);
    v = clamp01(v + sv / F.dy);
    return true;
}

__device__ __forceinline__ double facet_eval(const Facet64& F, const double A[3], const double B[3],
                                             double na, double nb, double u, double v, double X[3])
{
    X[0] = F.x0 + u * F.dx;
    X[1] = F.y0 + v * F.dy;
    X[2] = F.z00 + F.b * u + F.c * v + F.e * u * v;
    double r1x = X[0] - A[0], r1y = X[1] - A[1], r1z = X[2] - A[2];
    double r2x = X[0] - B[0], r2y = X[1] - B[1], r2z = X[2] - B[2];
    return na * sqrt(r1x * r1x + r1y * r1y + r1z * r1z) + nb * sqrt(r2x * r2x + r2y * r2y + r2z * r2z);
}

__device__ __forceinline__ void flat_start(const double U[3], const double L[3], double nu, double nl,
                                           double h0, int iters, double& sx, double& sy)
{
    double hx = L[0] - U[0], hy = L[1] - U[1];
    double D = sqrt(hx * hx + hy * hy);
    if (!(D >= 1e-9)) {
        sx = L[0];
        sy = L[1];
        return;
    }
    double ha = fabs(U[2] - h0), hb = fabs(L[2] - h0);
    double s = D * ha / (ha + hb + 1e-30);
    if (!(s >= 0.0)) s = 0.0;
    if (s > D) s = D;
    for (int it = 0; it < iters; it++) {
        double q1 = sqrt(s * s + ha * ha);
        double r = D - s;
        double q2 = sqrt(r * r + hb * hb);
        double g = nu * s / q1 - nl * r / q2;
        double gp = nu * ha * ha / (q1 * q1 * q1) + nl * hb * hb / (q2 * q2 * q2);
        if (!(gp > 0.0)) break;
        s = s - g / gp;
        if (s < 0.0) s = 0.0;
        if (s > D) s = D;
    }
    sx = U[0] + hx * (s / D);
    sy = U[1] + hy * (s / D);
}

__device__ __forceinline__ int nearest_node(double v0, double step, int n, double s)
{
    double t = floor((s - v0) / step + 0.5);
    if (!(t >= 0.0)) return 0;
    if (t > (double)(n - 1)) return n - 1;
    return (int)t;
}

// Crossing point of the path A (index na) -> B (index nb), FP64.
__device__ __forceinline__ void refraction_newton(const DemView& d, const double A[3], const double B[3],
                                                  double na, double nb, int W, double out[3])
{
    const bool lower_b = nb >= na;
    const double* Lp = lower_b ? B : A;
    const double* Up = lower_b ? A : B;
    double nl = lower_b ? nb : na, nu = lower_b ? na : nb;
    double h0 = dem_elevation(d, Lp[0], Lp[1]);
    double sx, sy;
    if (d.empty || d.nx < 2 || d.ny < 2) {
        flat_start(Up, Lp, nu, nl, h0, 4 * kFlatIters, sx, sy);
        out[0] = sx;
        out[1] = sy;
        out[2] = dem_elevation(d, sx, sy);
        return;
    }
    flat_start(Up, Lp, nu, nl, h0, kFlatIters, sx, sy);
    int is = nearest_node(d.x0, d.stepx, d.nx, sx), js = nearest_node(d.y0, d.stepy, d.ny, sy);
    int ia = max(is - W, 0), ib = min(is + W, d.nx - 1);
    int ja = max(js - W, 0), jb = min(js + W, d.ny - 1);
    double bestL = INFINITY;
    int bi = is, bj = js;
    const double* __restrict__ Z = d.z;
    for (int i = ia; i <= ib; i++) {
        double xi = __ldg(d.xv + i);
        double r1x = xi - A[0], r2x = xi - B[0];
        for (int j = ja; j <= jb; j++) {
            double yj = __ldg(d.yv + j);
            double zij = __ldg(Z + (int64_t)j * d.nx + i);
            double r1y = yj - A[1], r1z = zij - A[2];
            double r2y = yj - B[1], r2z = zij - B[2];
            double L = na * sqrt(r1x * r1x + r1y * r1y + r1z * r1z) + nb * sqrt(r2x * r2x + r2y * r2y + r2z * r2z);
            if (L < bestL) {
                bestL = L;
                bi = i;
                bj = j;
            }
        }
    }
    // fallback facet (kept only when no facet path compares below +inf, e.g. NaN input)
    int bfi = min(bi, d.nx - 2), bfj = min(bj, d.ny - 2);
    double bestF = INFINITY, bu = (double)(bi - bfi), bv = (double)(bj - bfj);
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
        int fi = bi - 1 + (k >> 1), fj = bj - 1 + (k & 1);
        if (fi < 0 || fj < 0 || fi > d.nx - 2 || fj > d.ny - 2) continue;
        Facet64 F;
        facet_load(d, fi, fj, F);
        double u = (double)(bi - fi), v = (double)(bj - fj);
#pragma unroll 1
        for (int it = 0; it < kPolishIters; it++)
            if (!facet_step(F, A, B, na, nb, u, v)) break;
        double X[3];
        double L = facet_eval(F, A, B, na, nb, u, v, X);
        if (L < bestF) {
            bestF = L;
            bu = u;
            bv = v;
            bfi = fi;
            bfj = fj;
        }
    }
    Facet64 F;
    facet_load(d, bfi, bfj, F);
    facet_step(F, A, B, na, nb, bu, bv);
    facet_eval(F, A, B, na, nb, bu, bv, out);
}

// The Newton crossing by a whole warp (all 32 lanes call with one pair): lanes share the node
// scan, lanes 0-3 polish one facet each.  The same crossing, bit for bit, as one thread's
// solve: the smallest node value with the lowest scan index, the first smallest facet path.
__device__ __forceinline__ void refraction_newton_warp(const DemView& d, const double A[3], const double B[3], double na,
                                                       double nb, int W, double out[3])
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool lower_b = nb >= na;
    const double* Lp = lower_b ? B : A;
    const double* Up = lower_b ? A : B;
    const double nl = lower_b ? nb : na, nu = lower_b ? na : nb;
    const double h0 = dem_elevation(d, Lp[0], Lp[1]);
    double sx, sy;
    if (d.empty || d.nx < 2 || d.ny < 2) {
        flat_start(Up, Lp, nu, nl, h0, 4 * kFlatIters, sx, sy);
        out[0] = sx;
        out[1] = sy;
        out[2] = dem_elevation(d, sx, sy);
        return;
    }
    flat_start(Up, Lp, nu, nl, h0, kFlatIters, sx, sy);
    const int is = nearest_node(d.x0, d.stepx, d.nx, sx), js = nearest_node(d.y0, d.stepy, d.ny, sy);
    const int ia = max(is - W, 0), ib = min(is + W, d.nx - 1);
    const int ja = max(js - W, 0), jb = min(js + W, d.ny - 1);
    const int nj = jb - ja + 1, n = (ib - ia + 1) * nj;
    double best = INFINITY;
    int at = 0x7fffffff;
#pragma unroll 1
    for (int k = lane; k < n; k += 32) {
        const int i = ia + k / nj, j = ja + k % nj;
        const double xi = __ldg(d.xv + i), yj = __ldg(d.yv + j), zij = __ldg(d.z + (int64_t)j * d.nx + i);
        const double r1x = xi - A[0], r2x = xi - B[0];
        const double r1y = yj - A[1], r1z = zij - A[2];
        const double r2y = yj - B[1], r2z = zij - B[2];
        const double L = na * sqrt(r1x * r1x + r1y * r1y + r1z * r1z) + nb * sqrt(r2x * r2x + r2y * r2y + r2z * r2z);
        if (L < best) {
            best = L;
            at = k;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double q = __shfl_xor_sync(full, best, o);
        const int qa = __shfl_xor_sync(full, at, o);
        if (q < best || (q == best && qa < at)) {
            best = q;
            at = qa;
        }
    }
    const int bi = at < n ? ia + at / nj : is, bj = at < n ? ja + at % nj : js;
    // one facet per lane
    const int k = lane & 3;
    const int fi = bi - 1 + (k >> 1), fj = bj - 1 + (k & 1);
    double Lf = INFINITY, u = (double)(bi - fi), v = (double)(bj - fj);
    if (lane < 4 && fi >= 0 && fj >= 0 && fi <= d.nx - 2 && fj <= d.ny - 2) {
        Facet64 F;
        facet_load(d, fi, fj, F);
#pragma unroll 1
        for (int it = 0; it < kPolishIters; it++)
            if (!facet_step(F, A, B, na, nb, u, v)) break;
        double X[3];
        Lf = facet_eval(F, A, B, na, nb, u, v, X);
    }
    // fallback facet (kept only when no facet path compares below +inf, e.g. NaN input)
    int bfi = min(bi, d.nx - 2), bfj = min(bj, d.ny - 2);
    double bestF = INFINITY, bu = (double)(bi - bfi), bv = (double)(bj - bfj);
#pragma unroll 1
    for (int q = 0; q < 4; q++) {
        const double L = __shfl_sync(full, Lf, q), uq = __shfl_sync(full, u, q), vq = __shfl_sync(full, v, q);
        if (L < bestF) {
            bestF = L;
            bu = uq;
            bv = vq;
            bfi = bi - 1 + (q >> 1);
            bfj = bj - 1 + (q & 1);
        }
    }
    Facet64 F;
    facet_load(d, bfi, bfj, F);
    facet_step(F, A, B, na, nb, bu, bv);
    facet_eval(F, A, B, na, nb, bu, bv, out);
}

// A crossing by a whole warp, solver 0 = grid, 1 = Newton.
template <int SOLVER>
__device__ __forceinline__ void refraction_point_warp(const DemView& d, const double A[3], const double B[3], double na,
                                                      double nb, int W, double out[3])
{
    if constexpr (SOLVER == 0)
        refraction_grid_warp(d, A[0], A[1], A[2], B[0], B[1], B[2], na, nb, out);
    else
        refraction_newton_warp(d, A, B, na, nb, W, out);
}

// Column tables of a thread's grid search (none for the Newton solver).
template <int SOLVER, int TPB> struct SolverShared { GridCols<TPB> cols; };
template <int TPB> struct SolverShared<1, TPB> {};

// A crossing by one thread, solver 0 = grid, 1 = Newton.
// TPB: the largest block size the calling kernel launches with (the grid search keeps
// one column of shared-memory tables per thread).
template <int SOLVER, int TPB>
__device__ __forceinline__ void refraction_point(const DemView& d, const double A[3], const double B[3],
                                                 double na, double nb, int W, SolverShared<SOLVER, TPB>* sh, double out[3])
{
    if constexpr (SOLVER == 0)
        refraction_grid<TPB>(d, A[0], A[1], A[2], B[0], B[1], B[2], na, nb, &sh->cols, out);
    else
        refraction_newton(d, A, B, na, nb, W, out);
}

}  // namespace bsar
