// k_newton.cu -- FP64 back-projection with the Newton solver and per-pulse legs.
//
// The layout of the mixed kernel (k_mixed.cu): one thread per voxel, a warp's 32 voxels a
// compact block of the grid, pulses in blocks of up to 32 whose antennas lie close together,
// and per block and leg one candidate list of the DEM nodes that can win the node scan of
// any of its (voxel, pulse) pairs (node_lists.cuh; the lists' bounds are FP32 with margins,
// every path, ranking, Newton step, delay, phase and sum here is FP64).  Lists of up to four
// nodes carry the nodes' path legs; where every listed node is itself the crossing for the
// whole block, a solve is two table reads per node.  The other solves rank the list and polish
// the facets around the best node (active-set Newton, one final step on the winning facet).
//
// A CTA's warps share 32 voxels and take the pulses in consecutive parts of 16 (8 to 32
// parts), handed out as warps get free: parts differ in work (solves that a list's tables
// answer against solves that are polished), and with one part a warp the others waited for the
// slowest for a third of their time.  The parts' sums are added in pulse order.  The split is a
// function of the pulses alone, so a voxel's value does not depend on the grid it is computed
// in.  81 x 77 voxels x planes x pulses at two warps per 32 voxels, parts of 16 / 20 / 24 / 32
// pulses: 13 x 512 5.36 / 5.36 / 5.36 / 5.39 ms, 1 x 512 0.81 / 0.89 / 0.95 / 1.09, 60 x 512 21.1 /
// 20.7 / 20.7 / 20.4, 13 x 128 2.36 / 2.48 / 2.61 / 2.59.  At four and eight warps (launch_bp_newton)
// 13 x 512 4.85, 1 x 512 0.82, 60 x 512 19.6; a split that followed the grid's size took 5.71, 0.96
// and 20.0.
//
// What bounds it: instruction latency and fetch at 12 to 16 warps an SM (an issue in 44 % of the
// cycles; the FP64 unit is 20 % busy).  The same scene took 82 ms with one warp per voxel and
// every pulse's own scan of (2W+1)^2 nodes, two FP64 square roots each.
#include <cuda_runtime.h>

#include <cstdint>

#include "dev_common.cuh"
#include "kernels.hpp"
#include "node_lists.cuh"

namespace bsar {

namespace {

// Heights for the candidate lists from the FP64 DEM.
struct Heights64 {
    const DemView& d;
    __device__ __forceinline__ explicit Heights64(const DemView& d_) : d(d_) {}
    __device__ __forceinline__ void cover(int, int, int, int) {}
    __device__ __forceinline__ float operator()(int i, int j) const { return (float)(__ldg(d.z + (int64_t)j * d.nx + i) - d.z0); }
    __device__ __forceinline__ float ground(float x, float y) const
    {
        return (float)(dem_elevation(d, (double)x + d.x0, (double)y + d.y0) - d.z0);
    }
};

struct Leg64 {
    double E[3], G[3], nE, nG;
    bool g_lower;
};

// Window centre of a leg's node scan; h64: the height under the voxel.
__device__ __noinline__ int2 start_node64(const DemView d, const Leg64 l, double h64)
{
    const double* Lp = l.g_lower ? l.G : l.E;
    const double* Up = l.g_lower ? l.E : l.G;
    const double h0 = l.g_lower ? h64 : dem_elevation(d, Lp[0], Lp[1]);
    double sx, sy;
    flat_start(Up, Lp, l.g_lower ? l.nE : l.nG, l.g_lower ? l.nG : l.nE, h0, kFlatIters, sx, sy);
    return make_int2(nearest_node(d.x0, d.stepx, d.nx, sx), nearest_node(d.y0, d.stepy, d.ny, sy));
}

// Every node of one lane's window, in the solver's order (no list for the block).  Wide windows of
// voxels several nodes apart are the one place where a lane per voxel loses to a warp per voxel
// (k_bp_plain), whose lanes share a window: 81 x 77 x 13 voxels 0.5 m apart, 128 pulses, 51 x 51
// nodes 310 ms against 178, 151 x 151 nodes 2.7 s against 2.0; with 13 x 13 nodes 17 against 32.
__device__ __noinline__ int2 scan_all64(const DemView d, const Leg64 l, double h64, int W)
{
    int2 best = start_node64(d, l, h64);
    const int ia = max(best.x - W, 0), ib = min(best.x + W, d.nx - 1);
    const int ja = max(best.y - W, 0), jb = min(best.y + W, d.ny - 1);
    // node_l64 with a column's terms formed once and the endpoints in registers
    const double ex = l.E[0], ey = l.E[1], ez = l.E[2], gx = l.G[0], gy = l.G[1], gz = l.G[2], nE = l.nE, nG = l.nG;
    double v = INFINITY;
#pragma unroll 1
    for (int i = ia; i <= ib; i++) {
        const double x = __ldg(d.xv + i), dxe = __dsub_rn(x, ex), dxg = __dsub_rn(x, gx);
        const double sxe = __dmul_rn(dxe, dxe), sxg = __dmul_rn(dxg, dxg);
        const double* zr = d.z + (int64_t)ja * d.nx + i;
#pragma unroll 4
        for (int j = ja; j <= jb; j++, zr += d.nx) {
            const double y = __ldg(d.yv + j), z = __ldg(zr);
            const double dye = __dsub_rn(y, ey), dze = __dsub_rn(z, ez), dyg = __dsub_rn(y, gy), dzg = __dsub_rn(z, gz);
            const double qe = __dadd_rn(__dadd_rn(sxe, __dmul_rn(dye, dye)), __dmul_rn(dze, dze));
            const double qg = __dadd_rn(__dadd_rn(sxg, __dmul_rn(dyg, dyg)), __dmul_rn(dzg, dzg));
            const double u = path64(__dsqrt_rn(qe), __dsqrt_rn(qg), nE, nG);
            if (u < v) {
                v = u;
                best = make_int2(i, j);
            }
        }
    }
    return best;
}

// A longer list, ranked in FP64 (it is in the solver's order).
__device__ __forceinline__ int2 rank_list64(const DemView& d, const float4* list, const LegList& H, const Leg64& l,
                                            double h64, int W)
{
    int2 st = make_int2(0, 0), best = make_int2(H.si, H.sj);
    const bool core = H.mode & kCore;
    if (!core) st = start_node64(d, l, h64);
    double v = INFINITY;
#pragma unroll 1
    for (int k = 0; k < H.m; k++) {
        const int pk = __float_as_int(list[k].w), i = H.i0 + (pk >> 16), j = H.j0 + (pk & 0xffff);
        if (!core && (abs(i - st.x) > W || abs(j - st.y) > W)) continue;
        const double u = node_l64(d, i, j, l.E, l.G, l.nE, l.nG);
        if (u < v) {
            v = u;
            best = make_int2(i, j);
        }
    }
    return best;
}

__device__ __forceinline__ double facet_path(const Facet64& F, const Leg64& l, double u, double v)
{
    const double x = F.x0 + u * F.dx, y = F.y0 + v * F.dy, z = F.z00 + F.b * u + F.c * v + F.e * u * v;
    return path64(leg_len64(x, y, z, l.E), leg_len64(x, y, z, l.G), l.nE, l.nG);
}

// polish64 where a facet whose steps ended at the node ties with facets that keep the node:
// every facet in the solver's order, with its own rounding of the node's path.  The first
// smallest wins, and its one more step may leave the node (voxels at the surface, whose undamped
// steps cycle between corners).
__device__ __noinline__ double polish_tied64(const DemView d, const Leg64 l, int bi, int bj)
{
    double best = INFINITY, bu = 0.0, bv = 0.0;
    Facet64 F;
    int bk = 0;
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
        const int fi = bi - 1 + (k >> 1), fj = bj - 1 + (k & 1);
        if (fi < 0 || fj < 0 || fi > d.nx - 2 || fj > d.ny - 2) continue;
        facet_load(d, fi, fj, F);
        const double idx = 1.0 / F.dx, idy = 1.0 / F.dy;
        double u = (double)(bi - fi), v = (double)(bj - fj);
#pragma unroll 1
        for (int it = 0; it < kPolishIters; it++)
            if (!facet_newton64(F, l.E, l.G, l.nE, l.nG, idx, idy, u, v)) break;
        const double L = facet_path(F, l, u, v);
        if (L < best) {
            best = L;
            bu = u;
            bv = v;
            bk = k;
        }
    }
    facet_load(d, bi - 1 + (bk >> 1), bj - 1 + (bk & 1), F);
    facet_newton64(F, l.E, l.G, l.nE, l.nG, 1.0 / F.dx, 1.0 / F.dy, bu, bv);
    return facet_path(F, l, bu, bv);
}

// From the best node (bi, bj) to the path, as the FP64 solver (refraction_newton) forms it: each
// of the four facets that have the node as a corner is polished, unless that corner is its
// minimum (the path's one-sided derivatives at the node; such a facet has the node's path); one
// more step on the best facet.  Where no facet has its minimum at the node, the node's path is
// not a candidate, even if three steps end above it (voxels at the surface).  Leaving out facets whose minimum lies on an
// edge of another polished one saved nothing (13 planes of 6237 voxels 5.97 ms, without 5.84;
// 60 planes 20.0 and 19.6; one plane 1.15 and 1.21), and where three steps had not reached that
// edge's minimum from the other side, single paths came out 1e-7 m long.
__device__ __forceinline__ double polish64(const DemView& d, const ListGrid& m, const Leg64& l, int bi, int bj)
{
    const double x = __ldg(d.xv + bi), y = __ldg(d.yv + bj);
    const bool xm = bi > 0, xp = bi < d.nx - 1, ym = bj > 0, yp = bj < d.ny - 1;
    const double* zr = d.z + (int64_t)bj * d.nx + bi;
    const double z = __ldg(zr);
    const double node = path64(leg_len64(x, y, z, l.E), leg_len64(x, y, z, l.G), l.nE, l.nG);
    // which facets to polish: FP32 derivatives; a corner within their rounding is polished, and
    // its Newton step then finds it in FP64
    NodePatch p;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const double* r = zr + (j == 0 ? (ym ? -d.nx : 0) : (j == 2 ? (yp ? d.nx : 0) : 0));
        p.z[0][j] = (float)(__ldg(r + (xm ? -1 : 0)) - z);
        p.z[1][j] = (float)(__ldg(r) - z);
        p.z[2][j] = (float)(__ldg(r + (xp ? 1 : 0)) - z);
    }
    p.rE[0] = (float)(x - l.E[0]), p.rE[1] = (float)(y - l.E[1]), p.rE[2] = (float)(z - l.E[2]);
    p.rG[0] = (float)(x - l.G[0]), p.rG[1] = (float)(y - l.G[1]), p.rG[2] = (float)(z - l.G[2]);
    const float nE = (float)l.nE, nG = (float)l.nG;
    patch_gradient(p, m, nE, nG);
    const float noise = 2e-5f * (nE + nG);
    p.gxb += noise * (1.0f + fabsf(p.z[0][1]) * m.istepx);
    p.gxf -= noise * (1.0f + fabsf(p.z[2][1]) * m.istepx);
    p.gyb += noise * (1.0f + fabsf(p.z[1][0]) * m.istepy);
    p.gyf -= noise * (1.0f + fabsf(p.z[1][2]) * m.istepy);
    unsigned todo = patch_todo(p, xm, xp, ym, yp);
    const unsigned facets = (unsigned)(xm && ym) | (unsigned)(xm && yp) << 1 | (unsigned)(xp && ym) << 2 |
                            (unsigned)(xp && yp) << 3;
    const bool keeps = todo != facets;     // some facet's minimum is the node
    bool step = !keeps;
    double best = keeps ? node : (double)INFINITY;
    int bfi = min(bi, d.nx - 2), bfj = min(bj, d.ny - 2);     // kept only when no path compares below infinity
    double bu = (double)(bi - bfi), bv = (double)(bj - bfj);
#pragma unroll 1
    while (todo) {
        const int k = __ffs(todo) - 1;
        todo &= todo - 1;
        const bool kx = k >> 1, ky = k & 1;
        const int fi = bi - 1 + kx, fj = bj - 1 + ky;
        Facet64 F;
        facet_load(d, fi, fj, F);
        const double idx = 1.0 / F.dx, idy = 1.0 / F.dy;
        double u = kx ? 0.0 : 1.0, v = ky ? 0.0 : 1.0;
        bool m1 = false;
#pragma unroll 1
        for (int it = 0; it < kPolishIters; it++) {
            if (!facet_newton64(F, l.E, l.G, l.nE, l.nG, idx, idy, u, v)) break;
            m1 = true;
        }
        const double L = m1 ? facet_path(F, l, u, v) : node;
        if (m1 && keeps && u == (kx ? 0.0 : 1.0) && v == (ky ? 0.0 : 1.0)) return polish_tied64(d, l, bi, bj);
        if (L < best) {
            best = L;
            step = true;
            bu = u;
            bv = v;
            bfi = fi;
            bfj = fj;
        }
    }
    if (step) {
        Facet64 F;
        facet_load(d, bfi, bfj, F);
        facet_newton64(F, l.E, l.G, l.nE, l.nG, 1.0 / F.dx, 1.0 / F.dy, bu, bv);
        best = facet_path(F, l, bu, bv);
    }
    return best;
}

constexpr int kPathPulses = 16;         // pulses whose legs are solved before they are summed
constexpr float kBlockSlope = 0.013f;   // length of the pulse blocks (pulse_block); 0.016: 4 % slower

struct NewtonWarp {
    BlockLists l;
    double path[kPathPulses][32];       // the paths of the legs solved one by one
    LegList h[2];
};

}  // namespace

// The parts a CTA's warps take: a function of the pulses alone, so that a voxel's sum has the
// same order, and its value the same bits, in every grid.
constexpr int kMaxParts = 32, kPartPulses = 16;
static int pulse_parts(int np)
{
    const int least = np < 8 ? np : 8, n = np / kPartPulses;
    return n < least ? least : (n > kMaxParts ? kMaxParts : n);
}

template <int WPC>
__global__ void __launch_bounds__(32 * WPC, WPC < 8 ? 12 / WPC : 16 / WPC)
    k_bp_newton(BpArgs a, float start_band, int compact, int nparts)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    NewtonWarp* ws = reinterpret_cast<NewtonWarp*>(smem_raw) + (threadIdx.x >> 5);
    double2 (*part)[32] = reinterpret_cast<double2(*)[32]>(reinterpret_cast<NewtonWarp*>(smem_raw) + WPC);
    __shared__ int next;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const DemView& d = a.dem;
    ListGrid m;
    m.nx = d.nx;
    m.ny = d.ny;
    m.stepx = (float)d.stepx;
    m.stepy = (float)d.stepy;
    m.istepx = (float)(1.0 / d.stepx);
    m.istepy = (float)(1.0 / d.stepy);
    m.start_band = start_band;
    m.extent = fmaxf((float)d.nx * m.stepx, (float)d.ny * m.stepy);
    const int64_t kk = (int64_t)blockIdx.x * 32 + lane;
    const int3 vx = voxel_at(a, compact, kk < a.v_count ? kk : a.v_count - 1);
    const double P[3] = {__ldg(a.gx + vx.x), __ldg(a.gy + vx.y), __ldg(a.gz + vx.z)};
    const float P32[3] = {(float)(P[0] - d.x0), (float)(P[1] - d.y0), (float)(P[2] - d.z0)};
    const double h64 = dem_elevation(d, P[0], P[1]);
    const WarpVoxels wv = warp_voxels(P32);
    if (threadIdx.x == 0) next = WPC;   // the parts after the first WPC go to the warps that are done
    __syncthreads();
    const double inv_c = 1.0 / a.c, inv_lambda = 1.0 / a.lambda;
    const Heights64 zat(d);
    // a first guess for each list, from part to part (the list does not depend on it)
    if (lane < 2) ws->h[lane].si = ws->h[lane].sj = -1;
    __syncwarp();
    for (int k = w; k < nparts;) {
        const int p0 = (int)((int64_t)k * a.np / nparts), p1 = (int)((int64_t)(k + 1) * a.np / nparts);
        double accr = 0.0, acci = 0.0;
        int n;
        for (int i = p0; i < p1; i += n) {
            n = pulse_block(m, zat, d, ws->l, ws->h, a.tx, a.rx, i, p1, d.x0, d.y0, P, P32, (float)(h64 - d.z0), wv, a.n1, a.n2, a.W,
                            kBlockSlope, !a.exhaustive);
            const int m0 = all_pinned(ws->h[0]) ? ws->h[0].m : 0, m1 = all_pinned(ws->h[1]) ? ws->h[1].m : 0;
            for (int b = 0; b < n; b += kPathPulses) {
                const int step = min(kPathPulses, n - b);
                // the legs to solve, one after the other over the block's pulses
#pragma unroll 1
                for (int leg = m0 ? 1 : 0; leg < (m1 ? 1 : 2); leg++) {
                    const LegList* H = &ws->h[leg];
                    const int hm = H->m, mode = H->mode;
                    Leg64 l;
#pragma unroll
                    for (int c = 0; c < 3; c++) l.G[c] = P[c];
                    l.nE = a.n1;
                    l.nG = a.n2;
                    l.g_lower = lower_is_voxel((float)a.n1, (float)a.n2, leg == 0);
#pragma unroll 1
                    for (int q = b; q < b + step; q++) {
                        double L = 0.0;
                        int2 node = make_int2(0, 0);
                        bool solved = false;
                        if (hm > 0 && mode == (kCore | kTables)) {
                            int c;
                            L = table_min(ws->l.tab[leg], hm, q, lane, c);
                            solved = (H->pinned >> c) & 1;
                            node = H->node[c];
                        }
                        if (!solved) {
                            const double* tr = (leg ? a.rx : a.tx) + 3 * (i + q);
#pragma unroll
                            for (int c = 0; c < 3; c++) l.E[c] = __ldg(tr + c);
                            if (hm < 0) {
                                node = scan_all64(d, l, h64, a.W);
                            } else if (!(mode & kTables)) {
                                node = rank_list64(d, ws->l.list[leg], *H, l, h64, a.W);
                            } else if (!(mode & kCore)) {
                                // a listed node may lie outside this solve's window
                                const int2 st = start_node64(d, l, h64);
                                const NodeTables* t = &ws->l.tab[leg];
                                double v = INFINITY;
                                int c = 0;
#pragma unroll 1
                                for (int k = 0; k < hm; k++) {
                                    const int2 nd = H->node[k];
                                    const double u = __dadd_rn(t->E[k][q], t->G[k][lane]);
                                    if (u < v && abs(nd.x - st.x) <= a.W && abs(nd.y - st.y) <= a.W) {
                                        v = u;
                                        c = k;
                                    }
                                }
                                node = H->node[c];
                            }
                            L = polish64(d, m, l, node.x, node.y);
                        }
                        double* path = &ws->path[q - b][lane];
                        *path = (leg && !m0) ? *path + L : L;
                    }
                }
                // delays, gathers and sums of the block's pulses
#pragma unroll 1
                for (int q = b; q < b + step; q++) {
                    double L = (m0 && m1) ? 0.0 : ws->path[q - b][lane];
                    int c;
                    if (m0) L += table_min(ws->l.tab[0], m0, q, lane, c);
                    if (m1) L += table_min(ws->l.tab[1], m1, q, lane, c);
                    const double t_val = inv_c * L;                          // proc_test_script.cpp:565
                    const double bin = (1.0 + t_val * a.fs_eff) - 1.0;         // :569, :593
                    // (int)floor(bin) >= 0 && (int)ceil(bin) < nr  <=>  0 <= bin <= nr - 1 (NaN fails both)
                    if (bin >= 0.0 && bin <= (double)(a.nr - 1)) {
                        const double lo_d = floor(bin);
                        const int lo = (int)lo_d;                            // nr <= 2^30
                        const double qf = bin - lo_d;
                        const double2* row = a.rc64 + (int64_t)(i + q) * a.nr + lo;
                        const double2 s0 = __ldg(row);
                        double vr = s0.x, vi = s0.y;
                        if (qf != 0.0) {
                            const double2 s1 = __ldg(row + 1);
                            vr = (1.0 - qf) * s0.x + qf * s1.x;              // :635
                            vi = (1.0 - qf) * s0.y + qf * s1.y;
                        }
                        // carrier phase (:573, :638) in turns, reduced before the sine
                        const double turns = rint(L * inv_lambda);
                        double sn, cs;
                        sincospi(2.0 * (fma(-turns, a.lambda, L) * inv_lambda), &sn, &cs);
                        accr += vr * cs - vi * sn;
                        acci += vr * sn + vi * cs;
                    }
                }
            }
        }
        part[k][lane] = make_double2(accr, acci);
        if (lane == 0) k = atomicAdd(&next, 1);
        k = __shfl_sync(0xffffffffu, k, 0);
    }
    __syncthreads();
    if (w == 0 && kk < a.v_count) {
        double accr = 0.0, acci = 0.0;
        for (int q = 0; q < nparts; q++) {
            accr += part[q][lane].x;
            acci += part[q][lane].y;
        }
        a.out[((int64_t)vx.x * a.ny + vx.y) * a.nz + vx.z] = make_double2(accr, acci);
    }
}

template <int WPC> static cudaError_t launch_wpc(const BpArgs& a, float band, int compact, cudaStream_t st)
{
    const int nparts = pulse_parts(a.np);
    const size_t sm = sizeof(NewtonWarp) * WPC + sizeof(double2) * 32 * nparts;
    cudaError_t e = cudaFuncSetAttribute(k_bp_newton<WPC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_bp_newton<WPC><<<(unsigned)((a.v_count + 31) / 32), 32 * WPC, sm, st>>>(a, band, compact, nparts);
    return cudaGetLastError();
}

cudaError_t launch_bp_newton(const BpArgs& a, cudaStream_t st)
{
    const int64_t plane = (int64_t)a.nx * a.ny;
    const int compact = a.v_begin % plane == 0 && a.v_count % plane == 0;
    const float band = list_start_band(a.dem);
    // warps per 32 voxels: enough for about three waves of 16 warps per SM; more than four only
    // with at least two pulse blocks each, eight from 512 pulses on (16 parts of a warp's own
    // keep them busy): 81 x 77 x 13 voxels x 512 pulses 4.85 ms, with four 5.27; 60 planes 19.6 and
    // 19.8; 161 x 161 x 81 x 1024 141.6 and 143.4, x 100 43.4 and 39.1.  Two are slower on every
    // grid (60 planes 20.7)
    constexpr int64_t kWarps = 148 * 48;
    const int64_t tiles = (plane * a.nz + 31) / 32;
    int wpc = a.np >= 512 ? 8 : 4;
    while (wpc < 16 && tiles * wpc < kWarps && a.np >= 2 * wpc * kBlockPulses) wpc *= 2;
    if (wpc == 16) return launch_wpc<16>(a, band, compact, st);
    if (wpc == 8) return launch_wpc<8>(a, band, compact, st);
    return launch_wpc<4>(a, band, compact, st);
}

}  // namespace bsar
