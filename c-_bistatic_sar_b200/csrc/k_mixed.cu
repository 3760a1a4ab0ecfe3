// k_mixed.cu -- the mixed-precision back-projection kernel.
//
// One thread per voxel; the 32 voxels of a warp are a compact block of the grid
// (compact_voxel) and walk the pulses in order, in blocks of up to 32 consecutive pulses
// whose antennas lie close together.
//
// Per pulse block and leg (Tx -> voxel, voxel -> Rx), by the warp together:
//   candidate list: the DEM nodes that can win the node scan of any (voxel, pulse) pair of
//           the block, found by one bounded ranking for the block's centre antenna and the
//           warp's centre voxel (build_list); lists of up to four nodes carry the nodes' FP64
//           path legs per pulse and per voxel, and whether each node is itself the crossing
//           for the whole block (node_pinned)
// Per (voxel, pulse) and leg:
//   node    the list's best node: the smallest sum of two tabled FP64 legs, or FP32 values
//           with near ties re-ranked in FP64 -- the node the FP64 solver's scan picks
//   path    a pinned node's sum is the path; otherwise FP32 active-set Newton polish of the
//           four facets around the node and one FP64 final Newton step
//   delay / phase: dL = L - L_ref(pulse) rounded to FP32; the fast-time bin and carrier
//           phase are FP32 offsets from per-pulse FP64 anchors (integer bin + fraction,
//           phase reduced to [-pi, pi) in FP64)
//   gather: two complex64 (or FP16 complex x pulse scale) samples, linear interpolation
//           (proc_test_script.cpp:589-636), times exp(j phi), Kahan-compensated FP32 sum.
// A block's legs are solved leg by leg over its pulses, then all its delays, gathers and
// sums run in one short loop: the warps of an SM stay in small pieces of code.
//
// What bounds it: instruction latency and fetch at 12 warps an SM, an issue in 44 % of the
// cycles.  On the medium scene the rough DEM leaves a quarter of the leg solves to polish, so
// a warp goes through list building, polish, final step and gathers, some 100 KB of code;
// unrolling the gather loop or inlining rare branches made every scene slower, and
// three CTAs per SM (168 registers) run faster than four (98.7 against 109.4 ms on 161 x 161
// x 81 voxels x 1024 pulses) or two.  Rare work is out of line.  Against the scan of every
// lane's own window with per-lane lower bounds, with pulse compression, one B200: the medium
// scene 487 ms before, 66 ms; 256 x 256 x 8 x 2048 on a 0.125 m DEM 614, 40 ms; 97 x 83 x 11
// x 701 on 0.2 m (no compile-time scan width) 72, 5 ms.
//
// DEM tile: for wide scans (25 x 25 and generic widths) every CTA stages a TI x TJ FP32
// tile of the DEM around its voxels (shifted by the scene's mean crossing offset) into
// shared memory with one TMA 2-D tiled load (cp.async.bulk.tensor, no multicast) completing
// on an mbarrier; rankings whose nodes lie inside the tile read it from there, others read
// the FP32 DEM in global memory.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "dev_common.cuh"
#include "kernels.hpp"
#include "mixed_solve.cuh"
#include "node_lists.cuh"

namespace bsar {

namespace {

constexpr int TI = kMixedTileI;    // tile columns (x); 176 B rows, a multiple of 16 B
constexpr int TJ = kMixedTileJ;    // tile rows (y)
constexpr long kWaitSpins = 1L << 24;

// Start heights under a voxel (the lower endpoint of both of its paths when the ground
// index exceeds the air index): FP32 bilinear for the FP32 start, the FP64 DEM lookup for
// the FP64 start.  Computed once per voxel instead of once per solve.
struct VoxelStart {
    float h32;
    double h64;
};

// A DEM tile in shared memory: node (i, j) at s[(j - j0) * TI + (i - i0)].
struct Tile {
    const float* s;
    int i0, j0;
    bool ok;
};

// Heights for the candidate lists: from the tile when it covers the nodes to rank.
struct TileHeights {
    const MixedCtx& m;
    const Tile& T;
    bool in_tile;
    __device__ __forceinline__ TileHeights(const MixedCtx& m_, const Tile& T_) : m(m_), T(T_), in_tile(false) {}
    __device__ __forceinline__ void cover(int ia, int ib, int ja, int jb)
    {
        in_tile = T.ok && ia >= T.i0 && ib < T.i0 + TI && ja >= T.j0 && jb < T.j0 + TJ;
    }
    __device__ __forceinline__ float ground(float x, float y) const;     // height under a point
    __device__ __forceinline__ float operator()(int i, int j) const
    {
        return in_tile ? T.s[(j - T.j0) * TI + (i - T.i0)] : zf(m, i, j);
    }
};

__device__ __forceinline__ float TileHeights::ground(float x, float y) const { return height32(m, x, y); }

__device__ __forceinline__ bool facet_step32(const Facet32& F, const float A[3], const float B[3], float na,
                                             float nb, float& u, float& v)
{
    float x = fmaf(u, F.dx, F.x0), y = fmaf(v, F.dy, F.y0);
    float h = F.z00 + F.b * u + F.c * v + F.e * u * v;
    const float idx_ = F.idx, idy = F.idy;
    float zx = (F.b + F.e * v) * idx_;
    float zy = (F.c + F.e * u) * idy;
    float r1x = x - A[0], r1y = y - A[1], r1z = h - A[2];
    float r2x = x - B[0], r2y = y - B[1], r2z = h - B[2];
    float q1 = r1x * r1x + r1y * r1y + r1z * r1z;
    float q2 = r2x * r2x + r2y * r2y + r2z * r2z;
    float s1 = rsqrtf(q1), s2 = rsqrtf(q2);
    float g1 = na * s1, g2 = nb * s2;
    float a1x = r1x + r1z * zx, a1y = r1y + r1z * zy;
    float a2x = r2x + r2z * zx, a2y = r2y + r2z * zy;
    float gx = g1 * a1x + g2 * a2x;
    float gy = g1 * a1y + g2 * a2y;
    // active set first: a corner the gradient pushes outward of on both axes is this
    // facet's minimum, and the Hessian is not needed
    bool au = (u <= 0.0f && gx > 0.0f) || (u >= 1.0f && gx < 0.0f);
    bool av = (v <= 0.0f && gy > 0.0f) || (v >= 1.0f && gy < 0.0f);
    if (au && av) return false;
    float zxy = F.e * idx_ * idy;
    float iq1 = s1 * s1, iq2 = s2 * s2;
    float txx = 1.0f + zx * zx, tyy = 1.0f + zy * zy, txy = zx * zy;
    float hxx = g1 * (txx - a1x * a1x * iq1) + g2 * (txx - a2x * a2x * iq2);
    float hyy = g1 * (tyy - a1y * a1y * iq1) + g2 * (tyy - a2y * a2y * iq2);
    float hxy = g1 * (txy - a1x * a1y * iq1) + g2 * (txy - a2x * a2y * iq2) + (g1 * r1z + g2 * r2z) * zxy;
    // approximate reciprocals (2 ulp): they set a Newton step's length, which the FP64
    // final step corrects, so a correctly rounded one buys nothing
    float igs = __fdividef(1.0f, g1 + g2);
    float su, sv;
    if (au) {
        su = 0.0f;
        sv = (hyy > 0.0f) ? -gy * __fdividef(1.0f, hyy) : -gy * igs;
    } else if (av) {
        sv = 0.0f;
        su = (hxx > 0.0f) ? -gx * __fdividef(1.0f, hxx) : -gx * igs;
    } else {
        float det = hxx * hyy - hxy * hxy;
        if (det > 0.0f && hxx > 0.0f) {
            float idet = __fdividef(1.0f, det);
            su = -(hyy * gx - hxy * gy) * idet;
            sv = -(hxx * gy - hxy * gx) * idet;
        } else {
            su = -gx * igs;
            sv = -gy * igs;
        }
    }
    u = __saturatef(u + su * idx_);
    v = __saturatef(v + sv * idy);
    return true;
}

__device__ __forceinline__ float facet_eval32(const Facet32& F, const float A[3], const float B[3], float na,
                                              float nb, float u, float v)
{
    float x = fmaf(u, F.dx, F.x0), y = fmaf(v, F.dy, F.y0);
    float h = F.z00 + F.b * u + F.c * v + F.e * u * v;
    float r1x = x - A[0], r1y = y - A[1], r1z = h - A[2];
    float r2x = x - B[0], r2y = y - B[1], r2z = h - B[2];
    float q1 = r1x * r1x + r1y * r1y + r1z * r1z;
    float q2 = r2x * r2x + r2y * r2y + r2z * r2z;
    return na * (q1 * rsqrtf(q1)) + nb * (q2 * rsqrtf(q2));
}

// Generic node scan over [ia, ib] x [ja, jb]: both legs per node, z from the tile when
// `in_tile`, else from global memory.
__device__ __noinline__ Rank scan_generic(const MixedCtx m, const float* ts, int ti0, int tj0, bool in_tile, int ia,
                                          int ib, int ja, int jb, float ex, float ey, float ez, float gx, float gy,
                                          float gz, float re, Rank r)
{
    for (int i = ia; i <= ib; i++) {
        float xi = (float)i * m.stepx;
        float dxe = xi - ex, dxg = xi - gx;
        float sxe = dxe * dxe, sxg = dxg * dxg;
        for (int j = ja; j <= jb; j++) {
            float yj = (float)j * m.stepy;
            float dye = yj - ey, dyg = yj - gy;
            float z = in_tile ? ts[(j - tj0) * TI + (i - ti0)] : zf(m, i, j);
            float dze = z - ez, dzg = z - gz;
            float qe = fmaf(dze, dze, fmaf(dye, dye, sxe));
            float qg = fmaf(dzg, dzg, fmaf(dyg, dyg, sxg));
            rank(fmaf(re, qe * rsqrtf(qe), qg * rsqrtf(qg)), i, j, r.v1, r.v2, r.bi, r.bj);
        }
    }
    return r;
}

// Per-warp table over the union of the 32 lanes' windows: (z, re |N-E|) per node, the
// height next to the E-leg term (all lanes solve the same pulse, so this leg does not
// depend on the voxel), so the scan reads both with one 8-byte load.  Lane l fills column
// j0 + l.  Warp-uniform; `ok` is false when the union does not fit.
constexpr int TBJ = 32;
// table rows for a compile-time node-scan half width: the window plus slack for the
// spread of the 32 lanes' window centres
template <int WT> struct TableRows { static constexpr int v = WT > 0 ? 2 * WT + 1 + (WT >= 12 ? 1 : 7) : 1; };

struct AirTable {
    float2* t;
    int i0, j0;
    bool ok;
};

template <int TBI>
__device__ __forceinline__ AirTable build_air_table(const MixedCtx& m, const Tile& T, float2* buf, int is, int js, int W,
                                                    float ex, float ey, float ez, float re)
{
    const unsigned full = 0xffffffffu;
    int i0 = max(__reduce_min_sync(full, is) - W, 0), i1 = min(__reduce_max_sync(full, is) + W, m.nx - 1);
    int j0 = max(__reduce_min_sync(full, js) - W, 0), j1 = min(__reduce_max_sync(full, js) + W, m.ny - 1);
    AirTable A{buf, i0, j0, false};
    __syncwarp();                       // readers of the previous table are done
    if (i1 - i0 + 1 > TBI || j1 - j0 + 1 > TBJ) return A;
    const int lane = threadIdx.x & 31;
    const int j = j0 + lane;
    const bool in_tile = T.ok && i0 >= T.i0 && i1 < T.i0 + TI && j0 >= T.j0 && j1 < T.j0 + TJ;
    if (j <= j1) {
        float dy = (float)j * m.stepy - ey;
        float sy = dy * dy;
        for (int i = i0; i <= i1; i++) {
            float z = in_tile ? T.s[(j - T.j0) * TI + (i - T.i0)] : zf(m, i, j);
            float dx = (float)i * m.stepx - ex, dz = z - ez;
            float q = fmaf(dz, dz, fmaf(dx, dx, sy));
            buf[(i - i0) * TBJ + lane] = make_float2(z, re * (q * rsqrtf(q)));
        }
    }
    __syncwarp();
    A.ok = true;
    return A;
}

// Full (2W+1)^2 window inside the DEM and the warp table: height and E leg from the
// table (one 8-byte load per node), the G leg per node, columns unrolled with
// compile-time offsets.  The best node's row is updated once per row.
template <int W>
__device__ __forceinline__ void scan_table(const MixedCtx& m, const AirTable& AT, int is, int js, float gx, float gy,
                                           float gz, float& v1, float& v2, int& bi, int& bj)
{
    constexpr int NJ = 2 * W + 1;
    float syg[NJ];
#pragma unroll
    for (int c = 0; c < NJ; c++) {
        float dy = (float)(js - W + c) * m.stepy - gy;
        syg[c] = dy * dy;
    }
    const float2* row0 = AT.t + (is - W - AT.i0) * TBJ + (js - W - AT.j0);
    int bc = bj - (js - W);
#pragma unroll 1
    for (int r = 0; r < NJ; r++) {
        const int i = is - W + r;
        const float dx = (float)i * m.stepx - gx;
        const float sxg = dx * dx;
        const float2* row = row0 + r * TBJ;
        const float v1_row = v1;
#pragma unroll
        for (int c = 0; c < NJ; c++) {
            const float2 e = row[c];
            const float dz = e.x - gz;
            const float q = fmaf(dz, dz, sxg + syg[c]);
            const float L = fmaf(q, rsqrtf(q), e.y);
            v2 = fminf(v2, fmaxf(v1, L));
            const bool p = L < v1;
            v1 = p ? L : v1;
            bc = p ? c : bc;
        }
        bi = (v1 < v1_row) ? i : bi;
    }
    bj = js - W + bc;
}

// FP64 re-ranking of the nodes within the FP32 ambiguity band: each lane whose FP32
// runner-up lies within it (`need`) has its window re-ranked by the whole warp, 32 nodes at a
// time; the smallest FP64 value with the lowest i-major index wins, which is the node the
// FP64 scan's strict < keeps.  All 32 lanes call it.
__device__ __noinline__ int2 rerank64_warp(const DemView d, const MixedCtx m, const float* ts, int ti0, int tj0,
                                           bool tok, bool need, int is, int js, int Wr, float ex, float ey, float ez,
                                           float gx, float gy, float gz, float re, float limit, double Ax, double Ay,
                                           double Az, double Bx, double By, double Bz, double na, double nb,
                                           int2 best_ij)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned pending = __ballot_sync(full, need);
    int2 result = best_ij;
    while (pending) {
        const int l = __ffs(pending) - 1;
        pending &= pending - 1;
        const int lis = __shfl_sync(full, is, l), ljs = __shfl_sync(full, js, l);
        const float lex = __shfl_sync(full, ex, l), ley = __shfl_sync(full, ey, l), lez = __shfl_sync(full, ez, l);
        const float lgx = __shfl_sync(full, gx, l), lgy = __shfl_sync(full, gy, l), lgz = __shfl_sync(full, gz, l);
        const float llim = __shfl_sync(full, limit, l);
        const double A[3] = {__shfl_sync(full, Ax, l), __shfl_sync(full, Ay, l), __shfl_sync(full, Az, l)};
        const double B[3] = {__shfl_sync(full, Bx, l), __shfl_sync(full, By, l), __shfl_sync(full, Bz, l)};
        const int ia = max(lis - Wr, 0), ib = min(lis + Wr, m.nx - 1);
        const int ja = max(ljs - Wr, 0), jb = min(ljs + Wr, m.ny - 1);
        const bool in_tile = tok && ia >= ti0 && ib < ti0 + TI && ja >= tj0 && jb < tj0 + TJ;
        const int nj = jb - ja + 1, n = (ib - ia + 1) * nj;
        double best = INFINITY;
        int bidx = 0x7fffffff;
        for (int k = lane; k < n; k += 32) {
            const int i = ia + k / nj, j = ja + k % nj;
            float xi = (float)i * m.stepx, yj = (float)j * m.stepy;
            float dxe = xi - lex, dxg = xi - lgx;
            float dye = yj - ley, dyg = yj - lgy;
            float z = in_tile ? ts[(j - tj0) * TI + (i - ti0)] : zf(m, i, j);
            float dze = z - lez, dzg = z - lgz;
            float qe = dxe * dxe + dye * dye + dze * dze;
            float qg = dxg * dxg + dyg * dyg + dzg * dzg;
            if (re * sqrtf(qe) + sqrtf(qg) <= llim) {
                double L = node_l64(d, i, j, A, B, na, nb);
                if (L < best) {
                    best = L;
                    bidx = k;
                }
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(full, best, o);
            const int oi = __shfl_xor_sync(full, bidx, o);
            if (ob < best || (ob == best && oi < bidx)) {
                best = ob;
                bidx = oi;
            }
        }
        if (lane == l && bidx != 0x7fffffff) result = make_int2(ia + bidx / nj, ja + bidx % nj);
    }
    return result;
}

// FP64 flat-interface start and its nearest node, exactly as the FP64 solver makes them
// (used when the FP32 start lies within rounding distance of a node-cell boundary).
__device__ __noinline__ int2 start_node64(const DemView d, double Ex, double Ey, double Ez, double Gx, double Gy,
                                          double Gz, double nE, double nG, bool g_lower, double h0_known)
{
    const double E[3] = {Ex, Ey, Ez}, G[3] = {Gx, Gy, Gz};
    const double* Lp = g_lower ? G : E;
    const double* Up = g_lower ? E : G;
    double nl = g_lower ? nG : nE, nu = g_lower ? nE : nG;
    const double h0 = isnan(h0_known) ? dem_elevation(d, Lp[0], Lp[1]) : h0_known;
    double sx, sy;
    flat_start(Up, Lp, nu, nl, h0, kFlatIters, sx, sy);
    return make_int2(nearest_node(d.x0, d.stepx, d.nx, sx), nearest_node(d.y0, d.stepy, d.ny, sy));
}

// One leg of one (voxel, pulse): the antenna E (index nE) and the voxel G (index nG), in
// FP64 and in the FP32 frame.  The path is the same in both directions; only the flat start
// asks which endpoint is the lower one (the one of the larger index, the leg's second
// endpoint when they are equal).
struct Leg {
    double E[3], G[3];
    float E32[3], G32[3];
    float nE, nG;
    double nE64, nG64;
    bool g_lower, to_voxel;
};

// Window centre of a leg's node scan: the node nearest the flat start.  A start within
// rounding distance of a cell boundary is redone in FP64 so both forms scan the same
// window.
__device__ __noinline__ int2 start_node(const DemView d, const MixedCtx m, const Leg l, const VoxelStart vs)
{
    const float* Lp = l.g_lower ? l.G32 : l.E32;      // the lower endpoint is normally the voxel itself
    const float* Up = l.g_lower ? l.E32 : l.G32;
    const float h0 = l.g_lower ? vs.h32 : height32(m, Lp[0], Lp[1]);
    const FlatStart f = flat_start32(Up, Lp, l.g_lower ? l.nE : l.nG, l.g_lower ? l.nG : l.nE, h0);
    const float fx = f.sx * m.istepx, fy = f.sy * m.istepy;
    int2 c = make_int2(min(max(__float2int_rn(fx), 0), m.nx - 1), min(max(__float2int_rn(fy), 0), m.ny - 1));
    if (fabsf(fabsf(fx - rintf(fx)) - 0.5f) < m.start_band || fabsf(fabsf(fy - rintf(fy)) - 0.5f) < m.start_band)
        c = start_node64(d, l.E[0], l.E[1], l.E[2], l.G[0], l.G[1], l.G[2], l.nE64, l.nG64, l.g_lower,
                         l.g_lower ? vs.h64 : (double)NAN);
    return c;
}

// Best node of every lane's own window, every node ranked (all 32 lanes call): windows of the
// common widths from the warp's table, near ties re-ranked in FP64 by the warp together.  Runs for the exhaustive
// flag and where no candidate list holds, so it stays out of the pulse loop's
// instruction stream.
template <int WT>
__device__ __noinline__ int2 scan_warp(const DemView d, const MixedCtx m, const Tile T, float2* table_buf, const Leg& l,
                                       const VoxelStart vs, int W)
{
    const int2 c = start_node(d, m, l, vs);
    const float* E = l.E32;
    const float* G = l.G32;
    const float re = __fdividef(l.nE, l.nG);
    const int ia = max(c.x - W, 0), ib = min(c.x + W, m.nx - 1);
    const int ja = max(c.y - W, 0), jb = min(c.y + W, m.ny - 1);
    Rank r{INFINITY, INFINITY, c.x, c.y};
    bool done = false;
    if constexpr (WT > 0) {
        const AirTable AT = build_air_table<TableRows<WT>::v>(m, T, table_buf, c.x, c.y, W, E[0], E[1], E[2], re);
        if (AT.ok && W == WT && ia == c.x - WT && ib == c.x + WT && ja == c.y - WT && jb == c.y + WT) {
            scan_table<WT>(m, AT, c.x, c.y, G[0], G[1], G[2], r.v1, r.v2, r.bi, r.bj);
            done = true;
        }
    }
    if (!done) {
        const bool in_tile = T.ok && ia >= T.i0 && ib < T.i0 + TI && ja >= T.j0 && jb < T.j0 + TJ;
        r = scan_generic(m, T.s, T.i0, T.j0, in_tile, ia, ib, ja, jb, E[0], E[1], E[2], G[0], G[1], G[2], re, r);
    }
    int2 best = make_int2(r.bi, r.bj);
    const float tie = tie_band(m, l.nG, r.v1);
    const bool need = !(r.v2 - r.v1 >= tie);
    if (__any_sync(0xffffffffu, need))
        best = rerank64_warp(d, m, T.s, T.i0, T.j0, T.ok, need, c.x, c.y, W, E[0], E[1], E[2], G[0], G[1], G[2], re,
                             r.v1 + tie, l.E[0], l.E[1], l.E[2], l.G[0], l.G[1], l.G[2], l.nE64, l.nG64,
                             best);
    return best;
}

// A solve's ranking of a longer list: the best entry.  Near ties are re-ranked in FP64 with the
// FP64 solver's arithmetic and order (the list is i-major).
__device__ __noinline__ int rerank_list(const DemView d, const float4* list, int n, int core, int i0, int j0, int is,
                                        int js, int W, float ex, float ey, float ez, float gx, float gy, float gz,
                                        float re, float limit, double Ax, double Ay, double Az, double Bx, double By,
                                        double Bz, double na, double nb, int best_k)
{
    const double A[3] = {Ax, Ay, Az}, B[3] = {Bx, By, Bz};
    double best = INFINITY;
    for (int k = 0; k < n; k++) {
        const float4 q = list[k];
        const int pk = __float_as_int(q.w), i = i0 + (pk >> 16), j = j0 + (pk & 0xffff);
        if (!core && (abs(i - is) > W || abs(j - js) > W)) continue;
        const float dxe = q.x - ex, dye = q.y - ey, dze = q.z - ez;
        const float dxg = q.x - gx, dyg = q.y - gy, dzg = q.z - gz;
        const float qe = dxe * dxe + dye * dye + dze * dze;
        const float qg = dxg * dxg + dyg * dyg + dzg * dzg;
        if (re * sqrtf(qe) + sqrtf(qg) <= limit) {
            const double L = node_l64(d, i, j, A, B, na, nb);
            if (L < best) {
                best = L;
                best_k = k;
            }
        }
    }
    return best_k;
}

__device__ __forceinline__ int2 rank_list(const DemView& d, const MixedCtx& m, const float4* list, const LegList& H,
                                          const Leg& l, const VoxelStart& vs, int W)
{
    int c = 0;
    if (H.m > 1) {
        int2 st = make_int2(0, 0);
        if (!(H.mode & kCore)) st = start_node(d, m, l, vs);
        const float* E = l.E32;
        const float* G = l.G32;
        const float re = __fdividef(l.nE, l.nG);
        float v1 = INFINITY, v2 = INFINITY;
#pragma unroll 1
        for (int k = 0; k < H.m; k++) {
            const float4 q = list[k];
            const float dye = q.y - E[1], dxe = q.x - E[0], dze = q.z - E[2];
            const float qe = fmaf(dze, dze, fmaf(dxe, dxe, dye * dye));
            const float dxg = q.x - G[0], dyg = q.y - G[1], dzg = q.z - G[2];
            const float qg = fmaf(dzg, dzg, fmaf(dxg, dxg, dyg * dyg));
            float L = fmaf(qg, rsqrtf(qg), re * (qe * rsqrtf(qe)));
            if (!(H.mode & kCore)) {
                const int pk = __float_as_int(q.w);
                if (abs(H.i0 + (pk >> 16) - st.x) > W || abs(H.j0 + (pk & 0xffff) - st.y) > W) L = INFINITY;
            }
            v2 = fminf(v2, fmaxf(v1, L));
            const bool p = L < v1;
            v1 = p ? L : v1;
            c = p ? k : c;
        }
        const float tie = tie_band(m, l.nG, v1);
        if (!(v2 - v1 >= tie))
            c = rerank_list(d, list, H.m, H.mode & kCore, H.i0, H.j0, st.x, st.y, W, E[0], E[1], E[2], G[0], G[1], G[2], re,
                            v1 + tie, l.E[0], l.E[1], l.E[2], l.G[0], l.G[1], l.G[2], l.nE64, l.nG64, c);
    }
    const int pk = __float_as_int(list[c].w);
    return make_int2(H.i0 + (pk >> 16), H.j0 + (pk & 0xffff));
}

// The facet that holds the crossing around the best node (bi, bj), by FP32 polish, and the
// crossing's (u, v) on it.  False: the node itself is the crossing.  Heights from the DEM tile when the node's 3 x 3 neighbourhood lies in it.
// The nine heights are loaded once (indices clamped to the DEM; a facet that would need a
// clamped one is not polished), and the path's gradient at the node is formed once: with
// G = na (N - A)/|N - A| + nb (N - B)/|N - B|, a facet with the node at its corner (u0, v0)
// has the gradient (Gx + Gz zx, Gy + Gz zy), zx and zy the facet's slopes along the edges
// through the node (one-sided differences: backward where u0 = 1, forward where u0 = 0).
// When it points out of the facet on both axes, the corner is that facet's minimum and the
// facet keeps the node's path; the others take the Newton steps.  A facet whose steps end back
// on the node ties with those that keep it, and the first in order wins, as in the FP64 solver:
// one more step would leave the node (voxels at the surface).  Each lane takes its own
// facets one after the other, so lanes whose crossings lie on different sides of a node step
// together.
__device__ __forceinline__ bool polish_leg(const MixedCtx& m, const Tile& T, const Leg& l, int bi, int bj, int& bfi,
                                           int& bfj, float& bu, float& bv)
{
    // the path's direction, which sets the order of its sums
    float A32[3], B32[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        A32[c] = l.to_voxel ? l.E32[c] : l.G32[c];
        B32[c] = l.to_voxel ? l.G32[c] : l.E32[c];
    }
    const float na = l.to_voxel ? l.nE : l.nG, nb = l.to_voxel ? l.nG : l.nE;
    const bool xm = bi > 0, xp = bi < m.nx - 1, ym = bj > 0, yp = bj < m.ny - 1;
    const bool nt = T.ok && bi - 1 >= T.i0 && bi + 1 < T.i0 + TI && bj - 1 >= T.j0 && bj + 1 < T.j0 + TJ;
    float zmm, zm0, zmp, z0m, z00n, z0p, zpm, zp0, zpp;
    {
        const float* r0 = nt ? T.s + (bj - T.j0) * TI + (bi - T.i0) : m.z32 + (int64_t)bj * m.pitch + bi;
        const int row = nt ? TI : m.pitch;
        const float *rm = r0 - (ym ? row : 0), *rp = r0 + (yp ? row : 0);
        const int om = xm ? -1 : 0, op = xp ? 1 : 0;
        zmm = rm[om], z0m = rm[0], zpm = rm[op];
        zm0 = r0[om], z00n = r0[0], zp0 = r0[op];
        zmp = rp[om], z0p = rp[0], zpp = rp[op];
    }
    float Lnode, gxb, gxf, gyb, gyf;
    {
        float xn = (float)bi * m.stepx, yn = (float)bj * m.stepy;
        float r1x = xn - A32[0], r1y = yn - A32[1], r1z = z00n - A32[2];
        float r2x = xn - B32[0], r2y = yn - B32[1], r2z = z00n - B32[2];
        float q1 = r1x * r1x + r1y * r1y + r1z * r1z, q2 = r2x * r2x + r2y * r2y + r2z * r2z;
        const float s1 = rsqrtf(q1), s2 = rsqrtf(q2);
        Lnode = na * (q1 * s1) + nb * (q2 * s2);
        const float g1 = na * s1, g2 = nb * s2;
        const float Gx = g1 * r1x + g2 * r2x, Gy = g1 * r1y + g2 * r2y, Gz = g1 * r1z + g2 * r2z;
        gxb = fmaf(Gz, (z00n - zm0) * m.istepx, Gx);
        gxf = fmaf(Gz, (zp0 - z00n) * m.istepx, Gx);
        gyb = fmaf(Gz, (z00n - z0m) * m.istepy, Gy);
        gyf = fmaf(Gz, (z0p - z00n) * m.istepy, Gy);
    }
    const bool ixm = !(gxb < 0.0f), ixp = !(gxf > 0.0f), iym = !(gyb < 0.0f), iyp = !(gyf > 0.0f);
    const unsigned facets = (unsigned)(xm && ym) | (unsigned)(xm && yp) << 1 | (unsigned)(xp && ym) << 2 |
                            (unsigned)(xp && yp) << 3;
    unsigned todo = facets & ((unsigned)(ixm || iym) | (unsigned)(ixm || iyp) << 1 | (unsigned)(ixp || iym) << 2 |
                              (unsigned)(ixp || iyp) << 3);
    bool moved = false;
    // a facet whose minimum is the node gives its path; the first of them
    const int first = todo == facets ? 4 : __ffs(facets & ~todo) - 1;
    float best = todo == facets ? INFINITY : Lnode;
#pragma unroll 1
    while (todo) {
        const int k = __ffs(todo) - 1;
        todo &= todo - 1;
        const bool kx = k >> 1, ky = k & 1;       // facet on the +x / +y side of the node
        const int fi = bi - 1 + kx, fj = bj - 1 + ky;
        Facet32 F;
        F.x0 = (float)fi * m.stepx;
        F.y0 = (float)fj * m.stepy;
        F.dx = m.stepx;
        F.dy = m.stepy;
        F.idx = m.istepx;
        F.idy = m.istepy;
        // corners (fi, fj), (fi + 1, fj), (fi, fj + 1), (fi + 1, fj + 1) of the 3 x 3 block
        const float z00 = kx ? (ky ? z00n : z0m) : (ky ? zm0 : zmm);
        const float z01 = kx ? (ky ? zp0 : zpm) : (ky ? z00n : z0m);
        const float z10 = kx ? (ky ? z0p : z00n) : (ky ? zmp : zm0);
        const float z11 = kx ? (ky ? zpp : zp0) : (ky ? z0p : z00n);
        F.z00 = z00;
        F.b = z01 - z00;
        F.c = z10 - z00;
        F.e = z11 - z01 - z10 + z00;
        float u = kx ? 0.0f : 1.0f, v = ky ? 0.0f : 1.0f;
        bool m1 = false;
#pragma unroll 1
        for (int it = 0; it < kPolishIters; it++) {
            if (!facet_step32(F, A32, B32, na, nb, u, v)) break;
            m1 = true;
        }
        if (k > first && u == (kx ? 0.0f : 1.0f) && v == (ky ? 0.0f : 1.0f)) continue;
        const float L = m1 ? facet_eval32(F, A32, B32, na, nb, u, v) : Lnode;
        if (L < best || (L == best && !moved)) {
            best = L;
            moved = m1;
            bu = u;
            bv = v;
            bfi = fi;
            bfj = fj;
        }
    }
    return moved;
}

// From the best node (bi, bj) to the leg's FP64 path: FP32 polish, FP64 final step.
// `known`: the node's own path is node_path.
__device__ __forceinline__ double finish_leg(const DemView& d, const MixedCtx& m, const Tile& T, const Leg& l, int bi,
                                             int bj, bool known, double node_path)
{
    int fi, fj;
    float u, v;
    if (polish_leg(m, T, l, bi, bj, fi, fj, u, v))
        return final_path64(d, fi, fj, l.E, l.G, l.nE64, l.nG64, m.idx64, m.idy64, (double)u, (double)v);
    return known ? node_path : node_l64(d, bi, bj, l.E, l.G, l.nE64, l.nG64);
}

// ------------------------------- TMA tile staging -----------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t mbar_try_wait_parity(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done;
}

// A copy that missed its deadline may still be in flight: wait for it (bounded) before
// the CTA's shared memory is released.
__device__ void drain_tile(uint64_t* mbar, uint32_t parity)
{
    const uint32_t bar = smem_u32(mbar);
    uint32_t done = 0;
    for (long s = 0; s < kWaitSpins && !done; s++) done = mbar_try_wait_parity(bar, parity);
}

// Arms `mbar` and has one elected thread load the tile with a TMA 2-D tiled copy that
// completes on it; every thread then waits for the barrier's phase `parity`, at most
// `polls` polls (the draining wait before exit has its own fixed limit, kWaitSpins).
// Returns false (and raises *status) if the copy did not complete in time.  The caller
// has initialised the barrier and synchronised the CTA after the previous tile's readers.
__device__ bool stage_tile(const void* tmap, float* tile, uint64_t* mbar, int i0, int j0, uint32_t parity, long long polls,
                           int* status)
{
    const uint32_t bar = smem_u32(mbar);
    if (threadIdx.x == 0) {
        const uint32_t bytes = TI * TJ * sizeof(float);
        // the tensor map sits in global memory written by host copies (a request slot is
        // reused by later requests): acquire it for the tensormap proxy before the copy
        asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(tmap))
                     : "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
                "r"(smem_u32(tile)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(i0), "r"(j0), "r"(bar)
            : "memory");
    }
    uint32_t done = 0;
    for (long long s = 0; s < polls && !done; s++) done = mbar_try_wait_parity(bar, parity);
    if (!done && status) atomicExch(status, 1);
    return done != 0;
}

__device__ __forceinline__ MixedCtx req_ctx(const MixedReq& r)
{
    MixedCtx m;
    m.z32 = r.z32;
    m.pitch = r.pitch;
    m.nx = r.a.dem.nx;
    m.ny = r.a.dem.ny;
    m.stepx = r.stepx;
    m.stepy = r.stepy;
    m.istepx = r.istepx;
    m.istepy = r.istepy;
    m.ox = r.ox;
    m.oy = r.oy;
    m.oz = r.a.dem.z0;
    m.idx64 = r.idx64;
    m.idy64 = r.idy64;
    m.start_band = r.start_band;
    m.lists = !r.exhaustive;
    m.extent = fmaxf((float)m.nx * m.stepx, (float)m.ny * m.stepy);
    return m;
}

// Shared memory of one warp.  A pulse block has lists for both legs or none: the lists (or
// their tables) share their place with the table of the scans that rank every node.
constexpr int kPathPulses = 8;               // pulses whose legs are solved before they are summed
// Length of the pulse blocks (pulse_block): 0.011 / 0.013 / 0.016: 37.3 / 36.0 / 34.8 ms on a
// served burst, 3.55 / 3.58 / 3.47 ms on the small scene, 2.57 / 2.55 / 2.59 ms on an FP16
// slice; the medium and large scenes stay within 1 %.
constexpr float kBlockSlope = 0.016f;

template <int WT> struct WarpShared {
    union {
        BlockLists l;
        float2 table[TableRows<WT>::v * TBJ];
    } u;
    double path[kPathPulses][32];            // per pulse and lane: the paths of the legs solved one by one
    double ref_L[kBlockPulses];              // the block's anchors
    float4 anchor[kBlockPulses];             // fast-time bin fraction, reduced phase, FP16 scale, bin (int)
    LegList h[2];
};

// One voxel of a request over pulses [p0, p1) (k: index in the request's voxel range;
// k >= v_count repeats the last voxel without storing it, so whole warps stay active).
// The sum goes to dst at the voxel's image index; add: MixedBatch::add.
template <int WT, bool CH>
__device__ __forceinline__ void voxel_mixed(const BpArgs& a, const MixedCtx& m, const Tile& T,
                                            WarpShared<WT>* ws, bool fp16, int compact, int64_t kk, int p0, int p1,
                                            double2* __restrict__ dst, int add)
{
    const int lane = threadIdx.x & 31;
    const int np = CH ? p1 : a.np;
    const float k_bin = (float)(a.fs_eff / a.c);
    const float k_phase = (float)(2.0 * 3.14159265358979323846 / a.lambda);
    const float n1f = (float)a.n1, n2f = (float)a.n2;
    const int64_t nr = a.nr;
    const int3 vx = voxel_at(a, compact, kk < a.v_count ? kk : a.v_count - 1);
    const double P[3] = {__ldg(a.gx + vx.x), __ldg(a.gy + vx.y), __ldg(a.gz + vx.z)};
    const float P32[3] = {(float)(P[0] - m.ox), (float)(P[1] - m.oy), (float)(P[2] - m.oz)};
    const VoxelStart vs{height32(m, P32[0], P32[1]), dem_elevation(a.dem, P[0], P[1])};
    const WarpVoxels wv = warp_voxels(P32);
    if (lane < 2) ws->h[lane].si = ws->h[lane].sj = -1;
    __syncwarp();
    float accr = 0.f, acci = 0.f, cmpr = 0.f, cmpi = 0.f;
    int block_end;
    for (int i = CH ? p0 : 0; i < np; i = block_end) {
        const int n = pulse_block(m, TileHeights(m, T), a.dem, ws->u.l, ws->h, a.tx, a.rx, i, np, m.ox, m.oy, P, P32,
                                  vs.h32, wv, a.n1, a.n2, a.W, kBlockSlope, m.lists != 0);
        block_end = i + n;
        if (lane < n) {
            ws->ref_L[lane] = __ldg(a.ref_L + i + lane);
            ws->anchor[lane] = make_float4(__ldg(a.ref_bin_f + i + lane), __ldg(a.ref_phase + i + lane),
                                           fp16 ? __ldg(a.scale16 + i + lane) : 1.0f,
                                           __int_as_float(__ldg(a.ref_bin_i + i + lane)));
        }
        __syncwarp();
        const int hm0 = ws->h[0].m, hm1 = ws->h[1].m;
        // legs whose listed nodes are all pinned: the paths come from the tables alone
        const int m0 = all_pinned(ws->h[0]) ? hm0 : 0, m1 = all_pinned(ws->h[1]) ? hm1 : 0;
        double* path = ws->path[0];
        for (int b = i; b < block_end; b += kPathPulses) {
            const int step = min(kPathPulses, block_end - b);
            // per-pulse legs: n1*r1Tx + n2*r2Tx (Tx -> voxel) + n2*r2Rx + n1*r1Rx (voxel -> Rx);
            // the legs to solve, one after the other over the block's pulses
#pragma unroll 1
            for (int leg = m0 ? 1 : 0; leg < (m1 ? 1 : 2); leg++) {
                const LegList* H = &ws->h[leg];
                const int hm = H->m, mode = H->mode;
                Leg l;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    l.G[c] = P[c];
                    l.G32[c] = P32[c];
                }
                l.nE = n1f;
                l.nG = n2f;
                l.nE64 = a.n1;
                l.nG64 = a.n2;
                l.g_lower = lower_is_voxel(n1f, n2f, leg == 0);
                l.to_voxel = leg == 0;
#pragma unroll 1
                for (int p = b; p < b + step; p++) {
                    double L = 0.0;
                    int2 node = make_int2(0, 0);
                    bool solved = false, known = false;
                    if (hm > 0 && mode == (kCore | kTables)) {
                        int c;
                        known = true;
                        L = table_min(ws->u.l.tab[leg], hm, p - i, lane, c);
                        solved = (H->pinned >> c) & 1;
                        node = H->node[c];
                    }
                    if (!solved) {
                        const double* tr = (leg ? a.rx : a.tx) + 3 * p;
#pragma unroll
                        for (int c = 0; c < 3; c++) l.E[c] = __ldg(tr + c);
                        l.E32[0] = (float)(l.E[0] - m.ox);
                        l.E32[1] = (float)(l.E[1] - m.oy);
                        l.E32[2] = (float)(l.E[2] - m.oz);
                        if (hm < 0) {
                            const Leg lc = l;
                            node = scan_warp<WT>(a.dem, m, T, ws->u.table, lc, vs, a.W);
                        } else if (!(mode & kTables)) {
                            node = rank_list(a.dem, m, ws->u.l.list[leg], *H, l, vs, a.W);
                        } else if (!(mode & kCore)) {
                            // a listed node may lie outside this solve's window
                            const int2 st = start_node(a.dem, m, l, vs);
                            const NodeTables* t = &ws->u.l.tab[leg];
                            double v = INFINITY;
                            int c = 0;
#pragma unroll 1
                            for (int k = 0; k < hm; k++) {
                                const int2 nd = H->node[k];
                                const double u = __dadd_rn(t->E[k][p - i], t->G[k][lane]);
                                if (u < v && abs(nd.x - st.x) <= a.W && abs(nd.y - st.y) <= a.W) {
                                    v = u;
                                    c = k;
                                }
                            }
                            node = H->node[c];
                        }
                        L = finish_leg(a.dem, m, T, l, node.x, node.y, known, L);
                    }
                    double* d = path + (p - b) * 32 + lane;
                    *d = (leg && !m0) ? __dadd_rn(*d, L) : L;
                }
            }
            // delays, gathers and sums of the block's pulses
#pragma unroll 1
            for (int p = b; p < b + step; p++) {
                const int q0 = p - i;
                double L = (m0 && m1) ? 0.0 : path[(p - b) * 32 + lane];
                int c;
                if (m0) L = __dadd_rn(L, table_min(ws->u.l.tab[0], m0, q0, lane, c));
                if (m1) L = __dadd_rn(L, table_min(ws->u.l.tab[1], m1, q0, lane, c));
                const float dL = (float)(L - ws->ref_L[q0]);
                const float4 an = ws->anchor[q0];
                // fast-time bin: integer anchor + FP32 offset
                const float t = an.x + dL * k_bin;
                const float fl = floorf(t);
                const int64_t lo = (int64_t)__float_as_int(an.w) + (int)fl;
                const float q = t - fl;
                const bool exact = (q == 0.0f);
                // |fl| < 2^31 also drops a path that is not a number
                if (fabsf(fl) < 2.0e9f && lo >= 0 && (lo < nr - 1 || (lo == nr - 1 && exact))) {
                    float s0r, s0i, s1r = 0.f, s1i = 0.f;
                    const int64_t base = (int64_t)p * nr + lo;
                    if (fp16) {
                        float2 f0 = __half22float2(a.rc16[base]);
                        s0r = f0.x * an.z;
                        s0i = f0.y * an.z;
                        if (!exact) {
                            float2 f1 = __half22float2(a.rc16[base + 1]);
                            s1r = f1.x * an.z;
                            s1i = f1.y * an.z;
                        }
                    } else {
                        float2 f0 = __ldg(a.rc32 + base);
                        s0r = f0.x;
                        s0i = f0.y;
                        if (!exact) {
                            float2 f1 = __ldg(a.rc32 + base + 1);
                            s1r = f1.x;
                            s1i = f1.y;
                        }
                    }
                    const float w0 = 1.0f - q;
                    const float vr = exact ? s0r : fmaf(w0, s0r, q * s1r);
                    const float vi = exact ? s0i : fmaf(w0, s0i, q * s1i);
                    // carrier phase: FP64-reduced anchor + FP32 offset, reduced again to [-pi, pi]
                    float ph = an.y + dL * k_phase;
                    const float kr = rintf(ph * 0.15915494309189535f);
                    ph = fmaf(-kr, 6.28318548202514648f, ph);
                    ph = fmaf(-kr, -1.7484555e-7f, ph);
                    float sn, cs;
                    __sincosf(ph, &sn, &cs);
                    const float cr = vr * cs - vi * sn;
                    const float ci = vr * sn + vi * cs;
                    // Kahan-compensated sums
                    float y = cr - cmpr;
                    float tt = accr + y;
                    cmpr = (tt - accr) - y;
                    accr = tt;
                    y = ci - cmpi;
                    tt = acci + y;
                    cmpi = (tt - acci) - y;
                    acci = tt;
                }
            }
        }
    }
    if (kk < a.v_count) {
        double2* o = (CH ? dst : a.out) + ((int64_t)vx.x * a.ny + vx.y) * a.nz + vx.z;
        double2 s = make_double2((double)accr - (double)cmpr, (double)acci - (double)cmpi);
        if (CH && add) {
            const double2 q = add == 2 ? *o : make_double2(0.0, 0.0);
            s = make_double2(q.x + s.x, q.y + s.y);
        }
        *o = s;
    }
}

// The last of a tile's pulse chunks to finish adds the chunks' sums, in chunk order, into
// the image (partial sums of the other CTAs are read from L2).
__device__ __forceinline__ void reduce_chunks(const BpArgs& a, const double2* __restrict__ partial, int compact, int K,
                                              int64_t kk)
{
    if (kk >= a.v_count) return;
    const int3 vx = voxel_at(a, compact, kk);
    const int64_t idx = ((int64_t)vx.x * a.ny + vx.y) * a.nz + vx.z;
    const int64_t nvox = (int64_t)a.nx * a.ny * a.nz;
    double sr = 0.0, si = 0.0;
    for (int c = 0; c < K; c++) {
        const double2 q = __ldcg(partial + c * nvox + idx);
        sr += q.x;
        si += q.y;
    }
    a.out[idx] = make_double2(sr, si);
}

}  // namespace

// Persistent mixed back-projection.  Every CTA takes work items -- one request and 128
// consecutive voxels of it -- from the batch's list through an atomic counter until the
// list is exhausted, so tiles of several requests share one launch.  The 128 voxels of a
// work item are the same 128 a one-request launch gives a CTA, so a voxel's arithmetic
// (warp tables, DEM tile, sums) does not depend on what else is in the batch.
// CH: the instantiation for batches holding small-grid requests whose tiles run in pulse
// chunks (MixedChunks); the last chunk of a tile to finish adds the chunks' sums in chunk
// order.  Batches without chunks run the other instantiation, which never reads them.
// The DEM tile is staged only for wide node scans (WT = 12, and the generic width), whose
// exhaustive form builds 30-row warp tables every pulse and reads them from the tile faster
// than through L1.  For 7 x 7 and 13 x 13 scans the tile's bookkeeping costs registers and
// its 7 KB per CTA shrinks L1: heights come from global memory, the same FP32 values, so the
// same image.  (Measured with the scans that rank every node, which the exhaustive flag
// still runs.)
template <int WT> struct StagesTile { static constexpr bool v = WT == 0 || WT >= 12; };

template <int WT, bool CH>
__global__ void __launch_bounds__(128, 3) k_bp_mixed(MixedBatch b)
{
    constexpr bool kTile = StagesTile<WT>::v;
    __shared__ alignas(128) float tile_s[kTile ? TI * TJ : 32];
    __shared__ alignas(16) WarpShared<WT> warp_s[4];
    __shared__ alignas(8) uint64_t mbar;
    __shared__ int2 work;
    __shared__ int last_chunk;
    WarpShared<WT>* ws = &warp_s[threadIdx.x >> 5];
    const int ntiles = b.ntiles_dev ? *b.ntiles_dev : b.ntiles;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    uint32_t parity = 0;
    bool copy_pending = false;     // a tile copy that timed out may still land
    for (;;) {
        __syncthreads();           // previous work item done (tile, table, `work`)
        if (threadIdx.x == 0) {
            const int t = atomicAdd(b.counter, 1);
            work = (t < ntiles) ? (b.tiles ? b.tiles[t] : make_int2(0, t)) : make_int2(-1, -1);
        }
        __syncthreads();
        const int2 w = work;
        if (w.x < 0) break;
        const MixedReq& R = b.reqs[w.x];
        const BpArgs& a = R.a;
        const MixedCtx m = req_ctx(R);
        // work item -> (128-voxel tile, pulse chunk); the unchunked kernel has one chunk
        const int K = CH && b.chunks ? max(b.chunks[w.x].nchunk, 1) : 1;
        const int tile = CH ? w.y / K : w.y;
        const int chunk = CH ? w.y - tile * K : 0;
        Tile T{tile_s, 0, 0, false};
        if (kTile && R.use_tile && !copy_pending) {
            // DEM tile centred on this work item's voxels plus the mean crossing offset
            const int64_t k0 = (int64_t)tile * 128;
            const int3 vm = voxel_at(a, R.compact, (k0 + min(k0 + 128, a.v_count) - 1) / 2);
            const double cx = __ldg(a.gx + vm.x) + R.off_x;
            const double cy = __ldg(a.gy + vm.y) + R.off_y;
            const int ci = (int)floor((cx - m.ox) / m.stepx), cj = (int)floor((cy - m.oy) / m.stepy);
            T.i0 = ((ci - TI / 2) >> 2) << 2;      // TMA: x offset a multiple of 4 floats (16 B)
            T.j0 = cj - TJ / 2;
            const bool seen = stage_tile(R.tmap, tile_s, &mbar, T.i0, T.j0, parity, b.wait_polls, b.status);
            parity ^= 1u;
            // one view for the whole CTA: the tile is used only if every thread saw it land,
            // and a copy is still in flight only if the thread that issued it did not
            T.ok = __syncthreads_and(seen);
            copy_pending = __syncthreads_or(threadIdx.x == 0 && !seen);
        }
        if constexpr (!CH) {
            voxel_mixed<WT, false>(a, m, T, ws, R.fp16 != 0, R.compact, (int64_t)w.y * 128 + threadIdx.x, 0,
                                   0, nullptr, 0);
        } else {
            const int p0 = (int)((int64_t)chunk * a.np / K), p1 = (int)((int64_t)(chunk + 1) * a.np / K);
            double2* dst = K == 1 ? a.out : b.chunks[w.x].partial + chunk * ((int64_t)a.nx * a.ny * a.nz);
            voxel_mixed<WT, true>(a, m, T, ws, R.fp16 != 0, R.compact, (int64_t)tile * 128 + threadIdx.x,
                                  p0, p1, dst, b.add);
            // the work item again from shared memory, so none of it stays live over the pulses
            const volatile int* wv = reinterpret_cast<volatile int*>(&work);
            const int2 w2 = make_int2(wv[0], wv[1]);
            const MixedChunks C = b.chunks ? b.chunks[w2.x] : MixedChunks{1, 0, nullptr, nullptr};
            if (C.nchunk > 1) {
                const int tile2 = w2.y / C.nchunk;
                __threadfence();   // this chunk's sums before the count that publishes them
                __syncthreads();
                if (threadIdx.x == 0) last_chunk = atomicAdd(C.tile_done + tile2, 1) == C.nchunk - 1;
                __syncthreads();
                if (last_chunk) {
                    __threadfence();
                    reduce_chunks(b.reqs[w2.x].a, C.partial, b.reqs[w2.x].compact, C.nchunk,
                                  (int64_t)tile2 * 128 + threadIdx.x);
                }
            }
        }
    }
    if (copy_pending) drain_tile(&mbar, parity ^ 1u);
}

float mixed_start_band(const DemView& d) { return list_start_band(d); }

// Shared-memory carve-out for 3 resident CTAs per SM (DEM tile + 4 warps' lists each),
// set once per device; the rest of the unified L1 stays cache for the sample gathers.
template <int WT, bool CH> static void set_carveout()
{
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, k_bp_mixed<WT, CH>) != cudaSuccess) return;
    const double need = 3.0 * (double)(fa.sharedSizeBytes + 1024);
    int pct = (int)(100.0 * need / (228.0 * 1024.0)) + 1;
    pct = pct > 100 ? 100 : pct;
    cudaFuncSetAttribute(k_bp_mixed<WT, CH>, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
}

static void mixed_setup_device()
{
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load() & bit) return;
    set_carveout<0, false>();
    set_carveout<3, false>();
    set_carveout<6, false>();
    set_carveout<12, false>();
    set_carveout<0, true>();
    set_carveout<3, true>();
    set_carveout<6, true>();
    set_carveout<12, true>();
    done.fetch_or(bit);
}

int mixed_chunks(int64_t voxels, int pulses)
{
    constexpr int kMinChunkPulses = 32;    // below this a chunk's fixed cost (start heights, first block) shows
    constexpr int64_t kItemsPerCta = 4;    // work items per resident CTA that even out their unequal costs
    const int64_t tiles = (voxels + 127) / 128;
    const int64_t want = std::min<int64_t>(kItemsPerCta * mixed_grid_ctas(), kMaxChunkedTiles);
    if (tiles <= 0 || tiles >= want) return 1;
    const int64_t k = std::min<int64_t>({(want + tiles - 1) / tiles, kMaxChunks, pulses / kMinChunkPulses});
    return k < 1 ? 1 : (int)k;
}

// Resident CTAs of the current device, looked up once per device: the pulse-chunk count
// (and with it a small grid's summation order) follows the device the call runs on, so
// GPUs of different kinds in one process each get their own.
int mixed_grid_ctas()
{
    mixed_setup_device();
    constexpr int kDevs = 64;
    static std::atomic<int> ctas[kDevs];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int>* slot = (dev >= 0 && dev < kDevs) ? &ctas[dev] : nullptr;
    int n = slot ? slot->load() : 0;
    if (!n) {
        int sms = 148, per = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_bp_mixed<6, false>, 128, 0);
        n = sms * (per > 0 ? per : 1);
        if (slot) slot->store(n);
    }
    return n;
}

template <bool CH> static void launch_w(const MixedBatch& b, int W, int grid, cudaStream_t st)
{
    switch (W) {
    case 3: k_bp_mixed<3, CH><<<grid, 128, 0, st>>>(b); break;
    case 6: k_bp_mixed<6, CH><<<grid, 128, 0, st>>>(b); break;
    case 12: k_bp_mixed<12, CH><<<grid, 128, 0, st>>>(b); break;
    default: k_bp_mixed<0, CH><<<grid, 128, 0, st>>>(b); break;
    }
}

cudaError_t launch_bp_mixed(const MixedBatch& b, int W, int grid, cudaStream_t st, bool chunked)
{
    mixed_setup_device();
    if (chunked)
        launch_w<true>(b, W, grid, st);
    else
        launch_w<false>(b, W, grid, st);
    return cudaGetLastError();
}

}  // namespace bsar
