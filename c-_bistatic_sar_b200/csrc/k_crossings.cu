// k_crossings.cu -- crossing points of the mixed solver (FP32 node scan and polish, FP64 final
// step) for a batch of (start, end) pairs: the data behind the mixed form's crossing error.
//
// One thread per pair, which ranks every node of its own window.  The nodes and the FP64 final
// step are those of the mixed back-projection; a crossing also depends on the facet it lies
// on, so the choice among facets whose FP32 paths tie is pinned here (crossing_point).
#include <cuda_runtime.h>

#include <cstdint>

#include "dev_common.cuh"
#include "kernels.hpp"
#include "mixed_solve.cuh"
#include "node_lists.cuh"

namespace bsar {

namespace {

// One pair: A (index na) and B (index nb), in FP64 and in the FP32 frame.
struct Pair {
    double A[3], B[3];
    float A32[3], B32[3];
    float na, nb;
};

// FP64 flat-interface start and its nearest node, as the FP64 solver makes them.
__device__ __noinline__ int2 pair_start64(const DemView d, const Pair p, double h_b)
{
    const bool lower_b = p.nb >= p.na;
    const double* Lp = lower_b ? p.B : p.A;
    const double* Up = lower_b ? p.A : p.B;
    const double h0 = lower_b ? h_b : dem_elevation(d, Lp[0], Lp[1]);
    double sx, sy;
    flat_start(Up, Lp, lower_b ? p.na : p.nb, lower_b ? p.nb : p.na, h0, kFlatIters, sx, sy);
    return make_int2(nearest_node(d.x0, d.stepx, d.nx, sx), nearest_node(d.y0, d.stepy, d.ny, sy));
}

// FP64 re-ranking of the nodes within the FP32 ambiguity band, with the FP64 solver's
// arithmetic and order (i-major, j-minor, strict <).
__device__ __noinline__ int2 pair_rerank64(const DemView d, const MixedCtx m, const Pair p, int ia, int ib, int ja, int jb,
                                           float re, float limit, int2 best_ij)
{
    double best = INFINITY;
    for (int i = ia; i <= ib; i++) {
        float xi = (float)i * m.stepx;
        float dxe = xi - p.A32[0], dxg = xi - p.B32[0];
        for (int j = ja; j <= jb; j++) {
            float yj = (float)j * m.stepy;
            float dye = yj - p.A32[1], dyg = yj - p.B32[1];
            float z = zf(m, i, j);
            float dze = z - p.A32[2], dzg = z - p.B32[2];
            float qe = dxe * dxe + dye * dye + dze * dze;
            float qg = dxg * dxg + dyg * dyg + dzg * dzg;
            if (re * sqrtf(qe) + sqrtf(qg) <= limit) {
                double L = node_l64(d, i, j, p.A, p.B, (double)p.na, (double)p.nb);
                if (L < best) {
                    best = L;
                    best_ij = make_int2(i, j);
                }
            }
        }
    }
    return best_ij;
}

// Best node of the pair's window (FP32, near ties in FP64).  A start within rounding distance
// of a node-cell boundary is redone in FP64, so both forms scan the same window.
__device__ __forceinline__ int2 pair_node(const DemView& d, const MixedCtx& m, const Pair& p, int W)
{
    const float* A = p.A32;
    const float* B = p.B32;
    const bool lower_b = p.nb >= p.na;
    const float h0 = lower_b ? height32(m, B[0], B[1]) : height32(m, A[0], A[1]);
    const FlatStart f = flat_start32(lower_b ? A : B, lower_b ? B : A, lower_b ? p.na : p.nb, lower_b ? p.nb : p.na, h0);
    const float fx = f.sx * m.istepx, fy = f.sy * m.istepy;
    int2 c = make_int2(min(max(__float2int_rn(fx), 0), m.nx - 1), min(max(__float2int_rn(fy), 0), m.ny - 1));
    if (fabsf(fabsf(fx - rintf(fx)) - 0.5f) < m.start_band || fabsf(fabsf(fy - rintf(fy)) - 0.5f) < m.start_band)
        c = pair_start64(d, p, dem_elevation(d, p.B[0], p.B[1]));
    const int ia = max(c.x - W, 0), ib = min(c.x + W, m.nx - 1);
    const int ja = max(c.y - W, 0), jb = min(c.y + W, m.ny - 1);
    const float re = __fdividef(p.na, p.nb), tie = kTieM / p.nb;
    Rank r{INFINITY, INFINITY, c.x, c.y};
    for (int i = ia; i <= ib; i++) {
        float xi = (float)i * m.stepx;
        float dxe = xi - A[0], dxg = xi - B[0];
        float sxe = dxe * dxe, sxg = dxg * dxg;
        for (int j = ja; j <= jb; j++) {
            float yj = (float)j * m.stepy;
            float dye = yj - A[1], dyg = yj - B[1];
            float z = zf(m, i, j);
            float dze = z - A[2], dzg = z - B[2];
            float qe = fmaf(dze, dze, fmaf(dye, dye, sxe));
            float qg = fmaf(dzg, dzg, fmaf(dyg, dyg, sxg));
            rank(fmaf(re, qe * rsqrtf(qe), qg * rsqrtf(qg)), i, j, r.v1, r.v2, r.bi, r.bj);
        }
    }
    if (r.v2 - r.v1 >= tie) return make_int2(r.bi, r.bj);
    return pair_rerank64(d, m, p, ia, ib, ja, jb, re, r.v1 + tie, make_int2(r.bi, r.bj));
}

// a b + c d, the first product in the FMA.
__device__ __forceinline__ float sum2(float a, float b, float c, float d) { return fmaf(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ float diff2(float a, float b, float c, float d) { return fmaf(a, b, -__fmul_rn(c, d)); }
__device__ __forceinline__ float norm2(float x, float y, float z) { return fmaf(z, z, fmaf(y, y, __fmul_rn(x, x))); }

__device__ __forceinline__ float facet_height(const Facet32& F, float u, float v)
{
    return fmaf(__fmul_rn(F.e, u), v, fmaf(F.c, v, fmaf(F.b, u, F.z00)));
}

// One active-set projected Newton step (the step of the back-projection's polish) and the
// path, in explicit FMAs: their last bits choose among tied facets.
__device__ __forceinline__ bool pinned_step(const Facet32& F, const float A[3], const float B[3], float na, float nb, float& u,
                                            float& v)
{
    const float x = fmaf(u, F.dx, F.x0), y = fmaf(v, F.dy, F.y0), h = facet_height(F, u, v);
    const float zx = __fmul_rn(fmaf(F.e, v, F.b), F.idx), zy = __fmul_rn(__fadd_rn(F.c, __fmul_rn(F.e, u)), F.idy);
    const float r1x = x - A[0], r1y = y - A[1], r1z = h - A[2];
    const float r2x = x - B[0], r2y = y - B[1], r2z = h - B[2];
    const float s1 = rsqrtf(norm2(r1x, r1y, r1z)), s2 = rsqrtf(norm2(r2x, r2y, r2z));
    const float g1 = __fmul_rn(na, s1), g2 = __fmul_rn(nb, s2);
    const float a1x = fmaf(r1z, zx, r1x), a1y = fmaf(r1z, zy, r1y);
    const float a2x = fmaf(r2z, zx, r2x), a2y = fmaf(r2z, zy, r2y);
    const float gx = sum2(g1, a1x, g2, a2x), gy = sum2(g1, a1y, g2, a2y);
    const bool au = (u <= 0.0f && gx > 0.0f) || (u >= 1.0f && gx < 0.0f);
    const bool av = (v <= 0.0f && gy > 0.0f) || (v >= 1.0f && gy < 0.0f);
    if (au && av) return false;
    const float zxy = __fmul_rn(__fmul_rn(F.e, F.idx), F.idy);
    const float iq1 = __fmul_rn(s1, s1), iq2 = __fmul_rn(s2, s2);
    const float txx = fmaf(zx, zx, 1.0f), tyy = fmaf(zy, zy, 1.0f), txy = __fmul_rn(zx, zy);
    const float hxx = sum2(g1, fmaf(-__fmul_rn(a1x, a1x), iq1, txx), g2, fmaf(-__fmul_rn(a2x, a2x), iq2, txx));
    const float hyy = sum2(g1, fmaf(-__fmul_rn(a1y, a1y), iq1, tyy), g2, fmaf(-__fmul_rn(a2y, a2y), iq2, tyy));
    const float hxy = fmaf(sum2(g1, r1z, g2, r2z), zxy,
                           sum2(g1, fmaf(-__fmul_rn(a1x, a1y), iq1, txy), g2, fmaf(-__fmul_rn(a2x, a2y), iq2, txy)));
    const float igs = __fdividef(1.0f, __fadd_rn(g1, g2));
    float su, sv;
    if (au) {
        su = 0.0f;
        sv = __fmul_rn(-gy, (hyy > 0.0f) ? __fdividef(1.0f, hyy) : igs);
    } else if (av) {
        sv = 0.0f;
        su = __fmul_rn(-gx, (hxx > 0.0f) ? __fdividef(1.0f, hxx) : igs);
    } else {
        const float det = diff2(hxx, hyy, hxy, hxy);
        if (det > 0.0f && hxx > 0.0f) {
            const float idet = __fdividef(1.0f, det);
            su = __fmul_rn(-diff2(hyy, gx, hxy, gy), idet);
            sv = __fmul_rn(-diff2(hxx, gy, hxy, gx), idet);
        } else {
            su = __fmul_rn(-gx, igs);
            sv = __fmul_rn(-gy, igs);
        }
    }
    u = __saturatef(fmaf(su, F.idx, u));
    v = __saturatef(fmaf(sv, F.idy, v));
    return true;
}

__device__ __forceinline__ float pinned_path(float r1x, float r1y, float r1z, float r2x, float r2y, float r2z, float na,
                                             float nb)
{
    const float q1 = norm2(r1x, r1y, r1z), q2 = norm2(r2x, r2y, r2z);
    return sum2(na, __fmul_rn(q1, rsqrtf(q1)), nb, __fmul_rn(q2, rsqrtf(q2)));
}

// The crossing around the best node (bi, bj): FP32 polish of the node's four facets and one
// FP64 final step on the best one.  FP32 paths of 50 m tie within 4e-6 m, and tied facets may
// cross millimetres apart, so the choice is part of the result: of the facets in order
// (-x -y, -x +y, +x -y, +x +y) the first with the smallest path, where a facet whose minimum is
// its corner at the node has the node's path.
__device__ __forceinline__ void crossing_point(const DemView& d, const MixedCtx& m, const Pair& p, int bi, int bj, double X[3])
{
    const float *A32 = p.A32, *B32 = p.B32;
    const float na = p.na, nb = p.nb;
    // the nine heights (indices clamped to the DEM; a facet that would need a clamped one is
    // not polished), and the path and its one-sided derivatives at the node
    const int im = max(bi - 1, 0), ip = min(bi + 1, m.nx - 1);
    const int jm = max(bj - 1, 0), jp = min(bj + 1, m.ny - 1);
    const float zmm = zf(m, im, jm), zm0 = zf(m, im, bj), zmp = zf(m, im, jp);
    const float z0m = zf(m, bi, jm), z00n = zf(m, bi, bj), z0p = zf(m, bi, jp);
    const float zpm = zf(m, ip, jm), zp0 = zf(m, ip, bj), zpp = zf(m, ip, jp);
    float Lnode, gxb, gxf, gyb, gyf;
    {
        const float fi = (float)bi, fj = (float)bj;
        const float r1x = fmaf(fi, m.stepx, -A32[0]), r1y = fmaf(fj, m.stepy, -A32[1]), r1z = z00n - A32[2];
        const float r2x = fmaf(fi, m.stepx, -B32[0]), r2y = fmaf(fj, m.stepy, -B32[1]), r2z = z00n - B32[2];
        Lnode = pinned_path(r1x, r1y, r1z, r2x, r2y, r2z, na, nb);
        const float g1 = __fmul_rn(na, rsqrtf(norm2(r1x, r1y, r1z))), g2 = __fmul_rn(nb, rsqrtf(norm2(r2x, r2y, r2z)));
        const float Gx = sum2(g1, r1x, g2, r2x), Gy = sum2(g1, r1y, g2, r2y), Gz = sum2(g1, r1z, g2, r2z);
        gxb = fmaf(Gz, __fmul_rn(z00n - zm0, m.istepx), Gx);
        gxf = fmaf(Gz, __fmul_rn(zp0 - z00n, m.istepx), Gx);
        gyb = fmaf(Gz, __fmul_rn(z00n - z0m, m.istepy), Gy);
        gyf = fmaf(Gz, __fmul_rn(z0p - z00n, m.istepy), Gy);
    }
    int bfi = min(bi, m.nx - 2), bfj = min(bj, m.ny - 2);     // kept only when no path compares below infinity
    float bestF = INFINITY, bu = (float)(bi - bfi), bv = (float)(bj - bfj);
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
        const bool kx = k >> 1, ky = k & 1;       // facet on the +x / +y side of the node
        int fi = bi - 1 + kx, fj = bj - 1 + ky;
        if (fi < 0 || fj < 0 || fi > m.nx - 2 || fj > m.ny - 2) continue;
        float u = (float)(bi - fi), v = (float)(bj - fj);
        float L = Lnode;
        const bool corner = (kx ? gxf > 0.0f : gxb < 0.0f) && (ky ? gyf > 0.0f : gyb < 0.0f);
        if (!corner) {
            Facet32 F;
            F.x0 = __fmul_rn((float)fi, m.stepx);
            F.y0 = __fmul_rn((float)fj, m.stepy);
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
            bool moved = false;
#pragma unroll 1
            for (int it = 0; it < kPolishIters; it++) {
                if (!pinned_step(F, A32, B32, na, nb, u, v)) break;
                moved = true;
            }
            if (moved) {
                const float x = fmaf(u, F.dx, F.x0), y = fmaf(v, F.dy, F.y0), h = facet_height(F, u, v);
                L = pinned_path(x - A32[0], y - A32[1], h - A32[2], x - B32[0], y - B32[1], h - B32[2], na, nb);
            }
        }
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
    double u = bu, v = bv;
    facet_newton64(F, p.A, p.B, (double)na, (double)nb, m.idx64, m.idy64, u, v);
    X[0] = F.x0 + u * F.dx;
    X[1] = F.y0 + v * F.dy;
    X[2] = F.z00 + F.b * u + F.c * v + F.e * u * v;
}

}  // namespace

__global__ void k_refraction_mixed(DemView d, MixedCtx m, const double* __restrict__ p1, const double* __restrict__ p2,
                                   int64_t n, float na, float nb, int W, double* __restrict__ out)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        Pair p;
        for (int c = 0; c < 3; c++) {
            const double o = c == 0 ? m.ox : (c == 1 ? m.oy : m.oz);
            p.A[c] = p1[3 * k + c];
            p.B[c] = p2[3 * k + c];
            p.A32[c] = (float)(p.A[c] - o);
            p.B32[c] = (float)(p.B[c] - o);
        }
        p.na = na;
        p.nb = nb;
        const int2 node = pair_node(d, m, p, W);
        double X[3];
        crossing_point(d, m, p, node.x, node.y, X);
        out[3 * k] = X[0];
        out[3 * k + 1] = X[1];
        out[3 * k + 2] = X[2];
    }
}

cudaError_t launch_refraction_mixed(const DemView& d, int pitch, const double* p1, const double* p2, int64_t n,
                                    double n1, double n2, int W, double* out, cudaStream_t st)
{
    MixedCtx m;
    m.z32 = d.z32;
    m.pitch = pitch;
    m.nx = d.nx;
    m.ny = d.ny;
    m.stepx = (float)d.stepx;
    m.stepy = (float)d.stepy;
    m.istepx = (float)(1.0 / d.stepx);
    m.istepy = (float)(1.0 / d.stepy);
    m.ox = d.x0;
    m.oy = d.y0;
    m.oz = d.z0;
    m.idx64 = 1.0 / d.stepx;
    m.idy64 = 1.0 / d.stepy;
    m.start_band = list_start_band(d);
    m.lists = 0;
    m.extent = 0.0f;
    const int64_t b = (n + 127) / 128;
    const int blocks = (int)(b < 1 ? 1 : (b > 148 * 64 ? 148 * 64 : b));
    k_refraction_mixed<<<blocks, 128, 0, st>>>(d, m, p1, p2, n, (float)n1, (float)n2, W, out);
    return cudaGetLastError();
}

}  // namespace bsar
