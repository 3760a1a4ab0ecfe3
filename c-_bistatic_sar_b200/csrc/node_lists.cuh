// node_lists.cuh -- candidate lists of a node scan, shared by a warp's (antenna, voxel)
// pairs, for the mixed (k_mixed.cu) and the FP64 Newton (k_newton.cu) back-projection.  FP32
// arithmetic with explicit FMA where a value must not depend on the unit's --fmad setting.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "dev_common.cuh"
#include "kernels.hpp"

namespace bsar {

// FP32 node-scan ranking ambiguity threshold, metres of optical path.  The largest FP32
// error of a node's ranking value measured against FP64 over 6e9 medium-scene solves was
// 4.8e-6 m (in units of L / ng), so two nodes are mis-ordered only within ~1e-5 m.
constexpr float kTieM = 5.0e-5f;
// Longer paths round coarser: 1.6e-7 of the value each, as measured, and the coordinates of a
// DEM that is kilometres wide.  Below 50 m of value on DEMs up to 100 m it is the band above.
constexpr float kTieRel = 4.0e-7f, kTieExtent = 1.0e-7f;
// A FP32 flat start closer than this to a node-cell boundary is redone in FP64: metres
// of start-position error (the largest measured FP32 start error was 3.1e-5 node units,
// 7.6e-6 m) plus the FP32 quantisation of the node coordinate (ulps of the largest index).
constexpr float kStartBandM = 2.5e-5f;
constexpr float kStartBandUlps = 8.0f;

// The DEM as the lists see it: sizes, FP32 spacing (and its reciprocal); the FP32 frame's
// origin is the first node and, in z, DemView::z0.
struct ListGrid {
    int nx, ny;
    float stepx, stepy;             // uniform node spacing
    float istepx, istepy;           // 1 / spacing
    float start_band;               // node units: FP32 starts this close to a cell boundary go FP64
    float extent;                   // largest coordinate of the FP32 frame
};

// Tie band of ranking values around v (L / ng).
__device__ __forceinline__ float tie_band(const ListGrid& m, float ng, float v)
{
    return fmaxf(kTieM / ng, fmaf(kTieRel, v, kTieExtent * m.extent));
}

// Start band of a DEM (node units), see kStartBandM.
inline __host__ __device__ float list_start_band(const DemView& d)
{
    const double step = d.stepx < d.stepy ? d.stepx : d.stepy;
    const double nmax = (double)(d.nx > d.ny ? d.nx : d.ny);
    return (float)((double)kStartBandM / step + (double)kStartBandUlps * nmax * 0x1.0p-23);
}

__device__ __forceinline__ float warp_max(float v)   // v >= 0
{
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}

// FP64 distance of (x, y, z) from a leg's endpoint, and a path from its two legs, with the
// FP64 solver's operations (no contraction): a node's path has the same bits wherever it is
// formed (a pulse block's tables, the FP64 re-rank, the final step), and ranks as there.
__device__ __forceinline__ double leg_len64(double x, double y, double z, const double E[3])
{
    const double dx = __dsub_rn(x, E[0]), dy = __dsub_rn(y, E[1]), dz = __dsub_rn(z, E[2]);
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
}

__device__ __forceinline__ double path64(double lenE, double lenG, double nE, double nG)
{
    return __dadd_rn(__dmul_rn(nE, lenE), __dmul_rn(nG, lenG));
}

// Node optical path in FP64.
__device__ __forceinline__ double node_l64(const DemView& d, int i, int j, const double E[3], const double G[3],
                                           double nE, double nG)
{
    const double x = __ldg(d.xv + i), y = __ldg(d.yv + j), z = __ldg(d.z + (int64_t)j * d.nx + i);
    return path64(leg_len64(x, y, z, E), leg_len64(x, y, z, G), nE, nG);
}

// One active-set projected Newton step in FP64 on a facet from (u, v), false at a corner that
// is the facet's minimum; idx_, idy: 1 / the facet's extents.
// Also the path, its gradient and its Hessian at the given (u, v) (at such a corner: only the
// path and the gradient).
__device__ __forceinline__ bool facet_newton64(const Facet64& F, const double A[3], const double B[3], double na,
                                               double nb, double idx_, double idy, double& u, double& v, double& L,
                                               double& gx, double& gy, double& hxx, double& hyy, double& hxy)
{
    double x = F.x0 + u * F.dx, y = F.y0 + v * F.dy;
    double h = F.z00 + F.b * u + F.c * v + F.e * u * v;
    double zx = (F.b + F.e * v) * idx_;
    double zy = (F.c + F.e * u) * idy;
    double zxy = F.e * idx_ * idy;
    double r1x = x - A[0], r1y = y - A[1], r1z = h - A[2];
    double r2x = x - B[0], r2y = y - B[1], r2z = h - B[2];
    double q1 = r1x * r1x + r1y * r1y + r1z * r1z;
    double q2 = r2x * r2x + r2y * r2y + r2z * r2z;
    double s1 = rsqrt(q1), s2 = rsqrt(q2);
    double g1 = na * s1, g2 = nb * s2;
    double iq1 = s1 * s1, iq2 = s2 * s2;
    double a1x = r1x + r1z * zx, a1y = r1y + r1z * zy;
    double a2x = r2x + r2z * zx, a2y = r2y + r2z * zy;
    L = g1 * q1 + g2 * q2;
    gx = g1 * a1x + g2 * a2x;
    gy = g1 * a1y + g2 * a2y;
    const bool au = (u <= 0.0 && gx > 0.0) || (u >= 1.0 && gx < 0.0);
    const bool av = (v <= 0.0 && gy > 0.0) || (v >= 1.0 && gy < 0.0);
    if (au && av) return false;
    double txx = 1.0 + zx * zx, tyy = 1.0 + zy * zy, txy = zx * zy;
    hxx = g1 * (txx - a1x * a1x * iq1) + g2 * (txx - a2x * a2x * iq2);
    hyy = g1 * (tyy - a1y * a1y * iq1) + g2 * (tyy - a2y * a2y * iq2);
    hxy = g1 * (txy - a1x * a1y * iq1) + g2 * (txy - a2x * a2y * iq2) + (g1 * r1z + g2 * r2z) * zxy;
    // one division: the reciprocal of the pivot the taken branch needs
    double det = hxx * hyy - hxy * hxy;
    const bool newton = !au && !av && det > 0.0 && hxx > 0.0;
    const bool axis = (au && hyy > 0.0) || (av && !au && hxx > 0.0);
    const double piv = newton ? det : (axis ? (au ? hyy : hxx) : g1 + g2);
    const double ip = 1.0 / piv;
    double su, sv;
    if (newton) {
        su = -(hyy * gx - hxy * gy) * ip;
        sv = -(hxx * gy - hxy * gx) * ip;
    } else if (au) {
        su = 0.0;
        sv = -gy * ip;
    } else if (av) {
        sv = 0.0;
        su = -gx * ip;
    } else {
        su = -gx * ip;
        sv = -gy * ip;
    }
    u = clamp01(u + su * idx_);
    v = clamp01(v + sv * idy);
    return true;
}

__device__ __forceinline__ bool facet_newton64(const Facet64& F, const double A[3], const double B[3], double na,
                                               double nb, double idx_, double idy, double& u, double& v)
{
    double L, gx, gy, hxx, hyy, hxy;
    return facet_newton64(F, A, B, na, nb, idx_, idy, u, v, L, gx, gy, hxx, hyy, hxy);
}

// ----------------------------- the facets around a node ------------------------------
// A node's four facets, k = 2 (on the +x side) + (on the +y side).  The path is a sum of
// norms, so it is convex along straight lines in space, and a bilinear facet is straight
// along both of its axes.
struct NodePatch {
    float z[3][3];          // heights of the 3 x 3 nodes less the node's (index 1 + offset; clamped at the DEM's border)
    float rE[3], rG[3];     // the node less the antenna, less the voxel
    float Fx, Fy, Fz;       // the path's gradient at the node
    float gxb, gxf, gyb, gyf;   // its one-sided derivatives along the four edges (backward, forward)
};

__device__ __forceinline__ void patch_gradient(NodePatch& p, const ListGrid& m, float nE, float nG)
{
    const float qe = p.rE[0] * p.rE[0] + p.rE[1] * p.rE[1] + p.rE[2] * p.rE[2];
    const float qg = p.rG[0] * p.rG[0] + p.rG[1] * p.rG[1] + p.rG[2] * p.rG[2];
    const float se = rsqrtf(qe), sg = rsqrtf(qg);
    const float ge = nE * se, gg = nG * sg;
    p.Fx = ge * p.rE[0] + gg * p.rG[0];
    p.Fy = ge * p.rE[1] + gg * p.rG[1];
    p.Fz = ge * p.rE[2] + gg * p.rG[2];
    p.gxb = fmaf(p.Fz, -p.z[0][1] * m.istepx, p.Fx);
    p.gxf = fmaf(p.Fz, p.z[2][1] * m.istepx, p.Fx);
    p.gyb = fmaf(p.Fz, -p.z[1][0] * m.istepy, p.Fy);
    p.gyf = fmaf(p.Fz, p.z[1][2] * m.istepy, p.Fy);
}

// Facets to polish: those whose corner at the node is not their minimum because the path
// falls from it along at least one of the facet's two edges.
__device__ __forceinline__ unsigned patch_todo(const NodePatch& p, bool xm, bool xp, bool ym, bool yp)
{
    const bool ixm = !(p.gxb < 0.0f), ixp = !(p.gxf > 0.0f), iym = !(p.gyb < 0.0f), iyp = !(p.gyf > 0.0f);
    return (unsigned)(xm && ym && (ixm || iym)) | (unsigned)(xm && yp && (ixm || iyp)) << 1 |
           (unsigned)(xp && ym && (ixp || iym)) << 2 | (unsigned)(xp && yp && (ixp || iyp)) << 3;
}

// The path at (u, v) on facet (fi, fj); on a node, that node's path.  Out of line: the final
// step rarely needs it.
static __device__ __noinline__ double facet_path64(const DemView d, int fi, int fj, double Ex, double Ey, double Ez, double Gx,
                                            double Gy, double Gz, double nE, double nG, double u, double v)
{
    const double E[3] = {Ex, Ey, Ez}, G[3] = {Gx, Gy, Gz};
    Facet64 F;
    facet_load(d, fi, fj, F);
    double x = F.x0 + u * F.dx, y = F.y0 + v * F.dy, z = F.z00 + F.b * u + F.c * v + F.e * u * v;
    if ((u == 0.0 || u == 1.0) && (v == 0.0 || v == 1.0)) {
        const int i = fi + (int)u, j = fj + (int)v;
        x = __ldg(d.xv + i);
        y = __ldg(d.yv + j);
        z = __ldg(d.z + (int64_t)j * d.nx + i);
    }
    return path64(leg_len64(x, y, z, E), leg_len64(x, y, z, G), nE, nG);
}

// The path after the FP64 final step from (u, v) on facet (fi, fj), idx_, idy: 1 / the
// facet's extents.  A step below half a millimetre moves the path by its second-order
// expansion (the third order is below 1e-11 m); a result on a node is that node's path.
__device__ __forceinline__ double final_path64(const DemView& d, int fi, int fj, const double E[3], const double G[3],
                                               double nE, double nG, double idx_, double idy, double u, double v)
{
    Facet64 F;
    facet_load(d, fi, fj, F);
    double L, gx, gy, hxx, hyy, hxy;
    const double u0 = u, v0 = v;
    facet_newton64(F, E, G, nE, nG, idx_, idy, u, v, L, gx, gy, hxx, hyy, hxy);
    const double du = (u - u0) * F.dx, dv = (v - v0) * F.dy;
    const bool node = (u == 0.0 || u == 1.0) && (v == 0.0 || v == 1.0);
    if (!node && fabs(du) + fabs(dv) < 5e-4)
        return L + (gx * du + gy * dv + 0.5 * (hxx * du * du + hyy * dv * dv) + hxy * du * dv);
    return facet_path64(d, fi, fj, E[0], E[1], E[2], G[0], G[1], G[2], nE, nG, u, v);
}

// Flat-interface start (FP32) of the path Up (index nu) -> Lp (index nl) over the height h0:
// (sx, sy), the horizontal distance D of the endpoints and the length of the last step.
struct FlatStart {
    float sx, sy, D, last;
};

__device__ __forceinline__ FlatStart flat_start32(const float Up[3], const float Lp[3], float nu, float nl, float h0)
{
    FlatStart f;
    const float hx = Lp[0] - Up[0], hy = Lp[1] - Up[1];
    const float D2 = hx * hx + hy * hy;
    const float D = D2 * rsqrtf(D2);
    f.sx = Lp[0];
    f.sy = Lp[1];
    f.D = 0.0f;
    f.last = 0.0f;
    if (D >= 1e-6f) {
        float ha = fabsf(Up[2] - h0), hb = fabsf(Lp[2] - h0);
        float s = fminf(fmaxf(__fdividef(D * ha, ha + hb + 1e-30f), 0.f), D);
        float before = s;
#pragma unroll 1
        for (int it = 0; it < kFlatIters; it++) {
            float q1 = s * s + ha * ha, r = D - s, q2 = r * r + hb * hb;
            float i1 = rsqrtf(q1), i2 = rsqrtf(q2);
            float g = nu * s * i1 - nl * r * i2;
            float gp = nu * ha * ha * i1 * i1 * i1 + nl * hb * hb * i2 * i2 * i2;
            before = s;
            if (gp > 0.f) s = fminf(fmaxf(s - __fdividef(g, gp), 0.f), D);
        }
        const float t = __fdividef(s, D);
        f.sx = Up[0] + hx * t;
        f.sy = Up[1] + hy * t;
        f.D = D;
        f.last = fabsf(s - before);
    }
    return f;
}

__device__ __forceinline__ bool lower_is_voxel(float nE, float nG, bool to_voxel)
{
    return to_voxel ? nG >= nE : nG > nE;
}

// ------------------------------- candidate lists -------------------------------------
// The node scan, shared by a warp's 32 voxels and a block of consecutive pulses.  A scan
// keeps the node with the smallest ranking value L'(N) = re |N - E| + |N - G| in a window
// around its flat start.  Neighbouring voxels G and consecutive antenna positions E rank
// the same few nodes best, so the warp ranks the nodes once per block for the block's
// centre antenna Ec and the warp's centre voxel Gc and lists those that can win for any of
// its (voxel, pulse) pairs; each solve then ranks the list, with the scan's own
// arithmetic, instead of the window.
//
// With S a node that every window holds, gap(N) = L'(N) - L'(S) moves with E by at most
// re |u_N - u_S| per metre, u the unit vectors from the nodes to E, and |u_N - u_S| <=
// 2 |N - S| / (|N - E| + |S - E|); likewise with G.  So a node with
//     gap(N) at (Ec, Gc) > slack(N) + tie,
//     slack(N) = 2 |N - S| (re rE / (|N-Ec| + |S-Ec| - 2 rE) + rG / (|N-Gc| + |S-Gc| - 2 rG)),
// rE and rG the largest distances of the block's antennas and the warp's voxels from the
// centres, is worse than S by more than the tie band for every pair: it is neither the
// best node nor within the tie band of it, and the scan's result (best node, tie decision)
// needs only the others.  A margin far above the FP32 rounding of the gaps is added.
//
// Windows.  A start moves with E by at most kappa = nE hG / (nE hG + nG hE) per metre
// horizontally (hE, hG: the endpoints' heights over the start height; Snell's law gives
// 0 <= d(dist)/dD <= dist / D <= kappa for nE <= nG), and by at most kappa D / hE per metre
// of antenna height.  From the lanes' own starts at Ec this bounds every window centre of
// the block: the warp ranks the union of the windows and requires S in their
// intersection.  When all listed nodes lie in the intersection the starts themselves are
// not needed; otherwise each solve makes its start and drops the nodes outside its window.
//
// No lists at all for indices that are not positive (lists_hold, kernels.hpp).  No list for a
// block (m = -1): antenna on the side of the larger index, start not converged, intersection
// empty, or more nodes than the list holds; those blocks scan every window node (scan_warp),
// as the exhaustive flag does.
constexpr int kListCap = 128;
constexpr int kBlockPulses = 32;    // longest pulse block

constexpr int kCore = 1, kTables = 2;
// Lists of at most kTabled nodes carry their FP64 legs (node_tables).
constexpr int kTabled = 4;

struct LegList {
    int m;               // listed nodes (i-major order), -1: no list
    int mode;            // kCore: every listed node lies in every window of the block
    int i0, j0;          // origin of the entries' packed offsets
    int si, sj;          // the last block's S (in: a first guess)
    int pinned;          // kTables: bit k set when node k is its own crossing for the whole block
    int pad;
    int2 node[kTabled];  // kTables: the listed nodes
};

// Entry: x, y, z of the node in the FP32 frame, (i - i0) << 16 | (j - j0).
__device__ __forceinline__ float4 list_entry(float x, float y, float z, int i, int j)
{
    return make_float4(x, y, z, __int_as_float((i << 16) | j));
}

__device__ __forceinline__ unsigned ordered_bits(float f)   // unsigned order = float order
{
    const unsigned u = __float_as_uint(f);
    return u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u);
}

// A block's centres and S: the gap of a node and its test against the slack.
struct GapRef {
    float E[3], G[3];     // block and warp centres
    float S[3], eS, gS;   // S and its distances |S - Ec|, |S - Gc|
    float re, cE, cG, rE2, rG2;
};

__device__ __forceinline__ void gap_set(GapRef& g, float x, float y, float z)
{
    g.S[0] = x;
    g.S[1] = y;
    g.S[2] = z;
    float dx = x - g.E[0], dy = y - g.E[1], dz = z - g.E[2];
    float q = fmaf(dz, dz, fmaf(dx, dx, dy * dy));
    g.eS = q * rsqrtf(q);
    dx = x - g.G[0], dy = y - g.G[1], dz = z - g.G[2];
    q = fmaf(dz, dz, fmaf(dx, dx, dy * dy));
    g.gS = q * rsqrtf(q);
}

// Whether the node may win somewhere in the block, gap <= thr + slack, and its gap.  With
// slack = |N - S| (cE / dE + cG / dG) the test is squared and multiplied out: the node ranking
// is bound by the special-function unit, which here takes the two distances' square roots
// only.
__device__ __forceinline__ bool gap_keep(const GapRef& g, float x, float y, float z, float thr, float& gap)
{
    float dx = x - g.E[0], dy = y - g.E[1], dz = z - g.E[2];
    float q = fmaf(dz, dz, fmaf(dx, dx, dy * dy));
    const float e = q * rsqrtf(q);
    dx = x - g.G[0], dy = y - g.G[1], dz = z - g.G[2];
    q = fmaf(dz, dz, fmaf(dx, dx, dy * dy));
    const float v = q * rsqrtf(q);
    dx = x - g.S[0], dy = y - g.S[1], dz = z - g.S[2];
    const float s2 = fmaf(dz, dz, fmaf(dx, dx, dy * dy));
    gap = fmaf(g.re, e - g.eS, v - g.gS);
    // at or below zero (a voxel or antenna among the nodes): the node is kept
    const float dE = fmaxf(e + g.eS - g.rE2, 1e-6f), dG = fmaxf(v + g.gS - g.rG2, 1e-6f);
    const float t = gap - thr, a = t * (dE * dG), b = fmaf(g.cE, dG, g.cG * dE);
    return t <= 0.0f || a * a <= s2 * (b * b) * 1.00001f;
}

// The tie band and a margin for the FP32 rounding of a gap: of its two distances, and of the
// coordinates of S and of the nodes that can win, which lie within the distances of S.
__device__ __forceinline__ float gap_margin(const ListGrid& m, const GapRef& g, float nG)
{
    return tie_band(m, nG, g.eS + g.gS) + 1e-4f + 2e-6f * (g.eS + g.gS) + 5e-7f * (m.extent + fabsf(g.S[2]));
}

// (float)i for 0 <= i < 2^23 without the conversion unit.
__device__ __forceinline__ float small_float(int i) { return __int_as_float(0x4b000000 | i) - 8388608.0f; }

// Builds one leg's list for the block (all 32 lanes call).  E: the block's centre antenna,
// rEh / rEz / rE the antennas' largest horizontal, vertical and 3-D distance from it, dh0
// the spread of the start height over the block when it lies under the antenna (else 0);
// G this lane's voxel, Gc / rG the warp's centre and radius; nE <= nG the indices.
template <typename Z>
__device__ __forceinline__ void build_list(const ListGrid& m, Z zat, float4* list, LegList* H, int W,
                                           const float E[3], float rEh, float rEz, float rE, const float G[3],
                                           float h0, float dh0, bool lp_is_g, const float Gc[3], float rG, float nE,
                                           float nG)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int si = H->si, sj = H->sj;
    __syncwarp();                                  // readers of the previous list are done
    // window centres of the block
    float up[3], lo[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        up[c] = lp_is_g ? E[c] : G[c];
        lo[c] = lp_is_g ? G[c] : E[c];
    }
    const FlatStart f = flat_start32(up, lo, lp_is_g ? nE : nG, lp_is_g ? nG : nE, h0);
    const float hE = fabsf(E[2] - h0), hG = fabsf(G[2] - h0), hEm = hE - rEz - dh0;
    const float kappa = __fdividef(nE * hG, nE * hG + nG * hEm);
    const float D = f.D + rEh;
    const float move = kappa * (rEh + __fdividef(D * rEz, hEm)) + __fdividef(2.0f * D * dh0, hE + hG);
    const bool ok = nE <= nG && hEm > 0.75f * hE && f.last <= 0.02f * fminf(m.stepx, m.stepy);
    const float mx = fmaf(move, m.istepx, 0.06f + m.start_band), my = fmaf(move, m.istepy, 0.06f + m.start_band);
    const float fx = f.sx * m.istepx, fy = f.sy * m.istepy;
    const int ilo = __reduce_min_sync(full, min(max(__float2int_rn(fx - mx), 0), m.nx - 1));
    const int ihi = __reduce_max_sync(full, min(max(__float2int_rn(fx + mx), 0), m.nx - 1));
    const int jlo = __reduce_min_sync(full, min(max(__float2int_rn(fy - my), 0), m.ny - 1));
    const int jhi = __reduce_max_sync(full, min(max(__float2int_rn(fy + my), 0), m.ny - 1));
    const int ca = max(ihi - W, 0), cb = min(ilo + W, m.nx - 1);      // intersection of the windows
    const int da = max(jhi - W, 0), db = min(jlo + W, m.ny - 1);
    const int ua = max(ilo - W, 0), ub = min(ihi + W, m.nx - 1);      // union
    const int va = max(jlo - W, 0), vb = min(jhi + W, m.ny - 1);
    if (!__all_sync(full, ok) || ca > cb || da > db || ub - ua > 32000 || vb - va > 32000) {
        if (lane == 0) H->m = -1;
        __syncwarp();
        return;
    }
    const int nj = vb - va + 1, n = (ub - ua + 1) * nj;
    zat.cover(ua, ub, va, vb);
    if (!(si >= ca && si <= cb && sj >= da && sj <= db)) {
        si = (ca + cb) >> 1;
        sj = (da + db) >> 1;
    }
    GapRef g;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        g.E[c] = E[c];
        g.G[c] = Gc[c];
    }
    g.re = __fdividef(nE, nG);
    g.cE = 2.0f * g.re * rE;
    g.cG = 2.0f * rG;
    g.rE2 = 2.0f * rE;
    g.rG2 = 2.0f * rG;
    gap_set(g, (float)si * m.stepx, (float)sj * m.stepy, zat(si, sj));
    const unsigned below = (1u << lane) - 1u;
    // lane / nj and 32 / nj (small integers: exact in FP32)
    const float inj = __fdividef(1.0f, (float)nj);
    const int li = (int)((small_float(lane) + 0.5f) * inj), di = (int)(32.5f * inj), dj = 32 - di * nj;
    int cnt = 0;
    bool outside = false;
#pragma unroll 1
    for (int attempt = 0; attempt < 2; attempt++) {
        const float thr = gap_margin(m, g, nG);
        float best = INFINITY;
        int bij = 0;
        int i = ua + li, j = va + lane - li * nj;
        cnt = 0;
        outside = false;
#pragma unroll 1
        for (int base = 0; base < n; base += 32) {
            const bool in = base + lane < n;
            bool keep = false;
            float x = 0.f, y = 0.f, z = 0.f;
            if (in) {
                x = small_float(i) * m.stepx;
                y = small_float(j) * m.stepy;
                z = zat(i, j);
                float gap;
                keep = gap_keep(g, x, y, z, thr, gap);
                const bool core = i >= ca && i <= cb && j >= da && j <= db;
                outside |= keep && !core;
                if (core && gap < best) {
                    best = gap;
                    bij = ((i - ua) << 16) | (j - va);
                }
            }
            const unsigned bal = __ballot_sync(full, keep);
            const int pos = cnt + __popc(bal & below);
            if (keep && pos < kListCap) list[pos] = list_entry(x, y, z, i - ua, j - va);
            cnt += __popc(bal);
            i += di;
            j += dj;
            if (j > vb) {
                j -= nj;
                i++;
            }
        }
        __syncwarp();
        // the best node inside every window becomes S: the tightest list, and the next
        // block's first guess
        const unsigned key = ordered_bits(best), kmin = __reduce_min_sync(full, key);
        const int w = __shfl_sync(full, bij, __ffs(__ballot_sync(full, key == kmin)) - 1);
        const int ni = ua + (w >> 16), nj2 = va + (w & 0xffff);
        const bool same = ni == si && nj2 == sj;
        si = ni;
        sj = nj2;
        if (same || cnt <= 1) break;
        gap_set(g, small_float(si) * m.stepx, small_float(sj) * m.stepy, zat(si, sj));
        if (cnt <= kListCap) {
            // list against the better S, in place and in order
            const float thr2 = gap_margin(m, g, nG);
            const int c0 = cnt;
            cnt = 0;
            outside = false;
#pragma unroll 1
            for (int base = 0; base < c0; base += 32) {
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                bool keep = false;
                if (base + lane < c0) {
                    q = list[base + lane];
                    float gap;
                    keep = gap_keep(g, q.x, q.y, q.z, thr2, gap);
                    const int pk = __float_as_int(q.w);
                    const int i2 = ua + (pk >> 16), j2 = va + (pk & 0xffff);
                    outside |= keep && !(i2 >= ca && i2 <= cb && j2 >= da && j2 <= db);
                }
                const unsigned bal = __ballot_sync(full, keep);
                if (keep) list[cnt + __popc(bal & below)] = q;
                cnt += __popc(bal);
            }
            break;
        }
    }
    const bool any_out = __any_sync(full, outside);
    if (lane == 0) {
        H->m = (cnt >= 1 && cnt <= kListCap) ? cnt : -1;
        H->mode = any_out ? 0 : kCore;
        H->i0 = ua;
        H->j0 = va;
        H->si = si;
        H->sj = sj;
    }
    __syncwarp();
}

// Whether the listed node (i, j) is the crossing itself for every (antenna, voxel) of the
// block: the path's one-sided derivatives along the four edges at the node, which point
// uphill at (Ec, Gc) by more than they can turn over the block.  With t the edge's tangent
// the derivative is nE u_E.t + nG u_G.t (u: unit vectors from the endpoints), and u turns by
// at most 2 r / (2 |N - Ec| - r) over a distance r.  Then each of the four facets has its
// minimum at the node (the corner test of finish_leg), with a margin far above the FP32
// rounding of the derivatives: of the coordinates (as if the antenna and the voxel moved by
// it) and of the slopes, two heights' rounding over the spacing (a neighbour's height is the
// node's and a rise, whose rounding is far below the margin).  Nodes on the DEM's border have
// missing facets: never.
template <typename Z>
__device__ __forceinline__ bool node_pinned(const ListGrid& m, const Z& zat, int i, int j, const float E[3], const float G[3], float rE,
                                            float rG, float nE, float nG)
{
    if (i < 1 || j < 1 || i > m.nx - 2 || j > m.ny - 2) return false;
    const float z = zat(i, j);
    const float sxb = (z - zat(i - 1, j)) * m.istepx, sxf = (zat(i + 1, j) - z) * m.istepx;
    const float syb = (z - zat(i, j - 1)) * m.istepy, syf = (zat(i, j + 1) - z) * m.istepy;
    const float coord = 2.5e-7f * (m.extent + fabsf(z));
    const float slope = 1.3e-7f * (nE + nG) * fabsf(z) * fmaxf(m.istepx, m.istepy);
    rE += coord;
    rG += coord;
    const float x = (float)i * m.stepx, y = (float)j * m.stepy;
    const float ex = x - E[0], ey = y - E[1], ez = z - E[2];
    const float gx = x - G[0], gy = y - G[1], gz = z - G[2];
    const float qe = ex * ex + ey * ey + ez * ez, qg = gx * gx + gy * gy + gz * gz;
    const float se = nE * rsqrtf(qe), sg = nG * rsqrtf(qg);
    const float Fx = se * ex + sg * gx, Fy = se * ey + sg * gy, Fz = se * ez + sg * gz;
    const float dE = 2.0f * qe * rsqrtf(qe) - rE, dG = 2.0f * qg * rsqrtf(qg) - rG;
    if (!(dE > rE && dG > rG)) return false;
    const float turn = 2.0f * (nE * __fdividef(rE, dE) + nG * __fdividef(rG, dG)) + 1e-5f * (nE + nG);
    auto tangent = [](float sl) { return sqrtf(1.0f + sl * sl); };
    return fmaf(Fz, sxf, Fx) > turn * tangent(sxf) + slope && -fmaf(Fz, sxb, Fx) > turn * tangent(sxb) + slope &&
           fmaf(Fz, syf, Fy) > turn * tangent(syf) + slope && -fmaf(Fz, syb, Fy) > turn * tangent(syb) + slope;
}

// Short lists (kTables): nE |N - E| of every listed node and pulse of the block and
// nG |N - G| of every node and lane, in FP64.  A solve adds two of them per node and keeps
// the smallest sum, which is the FP64 solver's ranking value, bit for bit; where that node
// is pinned the sum is the leg's path and the solve is done.
struct NodeTables {
    double E[kTabled][kBlockPulses], G[kTabled][32];
};

// Smallest sum of pulse q (of the block) and this lane over m listed nodes, and its node.
__device__ __forceinline__ double table_min(const NodeTables& t, int m, int q, int lane, int& c)
{
    double v = __dadd_rn(t.E[0][q], t.G[0][lane]);
    c = 0;
#pragma unroll 1
    for (int k = 1; k < m; k++) {
        const double u = __dadd_rn(t.E[k][q], t.G[k][lane]);
        if (u < v) {
            v = u;
            c = k;
        }
    }
    return v;
}


// The lists of one block's legs, or the tables of a leg's short list.
struct BlockLists {
    union {
        float4 list[2][kListCap];
        NodeTables tab[2];
    };
};
static_assert(sizeof(NodeTables) == sizeof(float4) * kListCap, "one leg's tables take its list's place");

// Centre and radius of a warp's voxels.
struct WarpVoxels {
    float c[3], r;
};

__device__ __forceinline__ WarpVoxels warp_voxels(const float P[3])
{
    WarpVoxels w;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        float lo = P[c], hi = P[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        w.c[c] = 0.5f * (lo + hi);
    }
    const float dx = P[0] - w.c[0], dy = P[1] - w.c[1], dz = P[2] - w.c[2];
    w.r = warp_max(sqrtf(dx * dx + dy * dy + dz * dz)) * 1.0001f + 1e-5f;
    return w;
}

// Takes the next pulse block, from pulse i (< np): as many pulses as keep both antennas close
// together, and both legs' lists for it (all 32 lanes call; P, P32, h0: the lane's voxel in
// FP64 and in the FP32 frame and the height under it there).  `slope` bounds the antennas' movement
// from the block's first pulse: re * distance / |E - G| stays below twice it, which sets the
// lists' slack and with it their length.  Returns the number of pulses, at most kBlockPulses.  Both
// legs have a list or neither (m = -1), as when `lists` is false.
template <typename Z>
__device__ __forceinline__ int pulse_block(const ListGrid& m, Z zat, const DemView& d, BlockLists& bl, LegList* heads,
                                           const double* __restrict__ tx, const double* __restrict__ rx, int i, int np,
                                           double ox, double oy, const double P[3], const float P32[3], float h0v,
                                           const WarpVoxels& wv, double n1, double n2, int W, float slope,
                                           bool lists)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const float n1f = (float)n1, n2f = (float)n2;
    const int pl = min(i + lane, np - 1);
    float e[2][3], far = 0.f;
#pragma unroll
    for (int leg = 0; leg < 2; leg++) {
        const double* tr = (leg ? rx : tx) + 3 * pl;
        e[leg][0] = (float)(__ldg(tr) - ox);
        e[leg][1] = (float)(__ldg(tr + 1) - oy);
        e[leg][2] = (float)(__ldg(tr + 2) - d.z0);
        const float dx = e[leg][0] - __shfl_sync(full, e[leg][0], 0);
        const float dy = e[leg][1] - __shfl_sync(full, e[leg][1], 0);
        const float dz = e[leg][2] - __shfl_sync(full, e[leg][2], 0);
        const float gx = e[leg][0] - wv.c[0], gy = e[leg][1] - wv.c[1], gz = e[leg][2] - wv.c[2];
        // movement against the antenna's distance from the voxels
        far = fmaxf(far, __fdividef(dx * dx + dy * dy + dz * dz, gx * gx + gy * gy + gz * gz));
    }
    const float re = fminf(__fdividef(n1f, n2f), 1.0f);
    const unsigned stop = __ballot_sync(full, !(far * re * re <= 4.0f * slope * slope) && lane > 0);
    const int n = min(min(stop ? __ffs(stop) - 1 : 32, kBlockPulses), np - i);
    if (!lists) {
        if (lane < 2) heads[lane].m = -1;
        __syncwarp();
        return n;
    }
#pragma unroll 1
    for (int leg = 0; leg < 2; leg++) {
        const float x = leg ? e[1][0] : e[0][0], y = leg ? e[1][1] : e[0][1], z = leg ? e[1][2] : e[0][2];
        const int mid = (n - 1) >> 1;
        const float E[3] = {__shfl_sync(full, x, mid), __shfl_sync(full, y, mid), __shfl_sync(full, z, mid)};
        const float dx = x - E[0], dy = y - E[1], dz = fabsf(z - E[2]);
        const bool in = lane < n;
        const float h2 = dx * dx + dy * dy;
        const float rEh = warp_max(in ? sqrtf(h2) : 0.f) * 1.0001f + 1e-5f;
        const float rEz = warp_max(in ? dz : 0.f) * 1.0001f + 1e-5f;
        const float rE = warp_max(in ? sqrtf(h2 + dz * dz) : 0.f) * 1.0001f + 1e-5f;
        // start height: under the voxel, or under the antenna where the antenna is the path's
        // lower endpoint (equal indices, second leg)
        const bool lp_is_g = lower_is_voxel(n1f, n2f, leg == 0);
        float h0 = h0v, dh0 = 0.f;
        if (!lp_is_g) {
            const float h = zat.ground(x, y);
            h0 = __shfl_sync(full, h, mid);
            dh0 = warp_max(in ? fabsf(h - h0) : 0.f) * 1.0001f + 1e-5f;
        }
        LegList* H = heads + leg;
        build_list(m, zat, bl.list[leg], H, W, E, rEh, rEz, rE, P32, h0, dh0, lp_is_g, wv.c, wv.r, n1f, n2f);
        const int cnt = H->m;
        if (cnt > 0 && cnt <= kTabled) {
            const int pk = __float_as_int(bl.list[leg][min(lane, cnt - 1)].w);     // lane k: node k
            const int ni = H->i0 + (pk >> 16), nj = H->j0 + (pk & 0xffff);
            const bool pin = node_pinned(m, zat, ni, nj, E, wv.c, rE, wv.r, n1f, n2f);
            const unsigned pinned = __ballot_sync(full, pin && lane < cnt);
            if (lane < cnt) H->node[lane] = make_int2(ni, nj);
            if (lane == 0) {
                H->mode |= kTables;
                H->pinned = (int)pinned;
            }
            const double* tr = (leg ? rx : tx) + 3 * pl;
            const double El[3] = {__ldg(tr), __ldg(tr + 1), __ldg(tr + 2)};
            __syncwarp();                    // the entries are read: their place is free
#pragma unroll 1
            for (int k = 0; k < cnt; k++) {
                const int2 nd = H->node[k];
                const double nx = __ldg(d.xv + nd.x), ny = __ldg(d.yv + nd.y);
                const double nz = __ldg(d.z + (int64_t)nd.y * d.nx + nd.x);
                const double le = __dmul_rn(n1, leg_len64(nx, ny, nz, El));
                bl.tab[leg].E[k][lane] = le;
                bl.tab[leg].G[k][lane] = __dmul_rn(n2, leg_len64(nx, ny, nz, P));
            }
        }
    }
    __syncwarp();
    const bool none = heads[0].m < 0 || heads[1].m < 0;
    __syncwarp();
    if (none && lane < 2) heads[lane].m = -1;
    __syncwarp();
    return n;
}

// Whether a leg's paths come from its tables alone: every listed node lies in every window
// and is pinned.
__device__ __forceinline__ bool all_pinned(const LegList& H)
{
    return H.m > 0 && H.mode == (kCore | kTables) && H.pinned == (1 << H.m) - 1;
}

// The voxel at index k of a request's range: ranges of whole z-planes in the compact order
// (compact_voxel), others in the reference's flat order (z -> x -> y).
__device__ __forceinline__ int3 voxel_at(const BpArgs& a, int compact, int64_t k)
{
    int x, y, z;
    if (compact) {
        const int64_t plane = (int64_t)a.nx * a.ny;
        compact_voxel(a.nx, a.ny, (int)(a.v_count / plane), k, x, y, z);
        z += (int)(a.v_begin / plane);
    } else {
        const int64_t v = a.v_begin + k;
        x = (int)((v / a.ny) % a.nx);
        y = (int)(v % a.ny);
        z = (int)(v / ((int64_t)a.nx * a.ny));
    }
    return make_int3(x, y, z);
}

}  // namespace bsar
