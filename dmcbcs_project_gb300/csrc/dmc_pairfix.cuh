// Pair terms of the FP64 walker path.
//
// GB300 issues one FP64 warp instruction per 64 cycles and sub-partition
// (DFMA, DADD and every conversion to or from double alike), a 64 x 64 -> 128
// high product (__mul64hi) takes 28 cycles there and a 64-bit add 2.  So
// whatever is bounded is computed in 64-bit fixed point on the integer pipe
// (at least 58 fractional bits where a double has 52), and FP64 keeps what
// needs a floating exponent: distances, tables, the pair sums.
#pragma once

#include <cuda_runtime.h>

#include "dmc_device.cuh"

namespace dmc {
namespace walker {

// ---- fixed point: 2^62 stands for 1 ----------------------------------------

constexpr long long kFixOne = 1ll << 62;
constexpr double kFixScale = 4611686018427387904.0;   // 2^62

// wrapping two's-complement arithmetic (a sum may leave the range on the way
// to a result inside it)
__device__ __forceinline__ long long fadd(long long a, long long b)
{
    return (long long)((unsigned long long)a + (unsigned long long)b);
}
__device__ __forceinline__ long long fsub(long long a, long long b)
{
    return (long long)((unsigned long long)a - (unsigned long long)b);
}
__device__ __forceinline__ long long fshl(long long a, int n) { return (long long)((unsigned long long)a << n); }
// a b / 4 of two fixed-point values (shift left by 2 for the product)
__device__ __forceinline__ long long fmh(long long a, long long b) { return __mul64hi(a, b); }
__device__ __forceinline__ long long fmul(long long a, long long b) { return fshl(__mul64hi(a, b), 2); }

// cos and sin of the pair's axis angles 2 pi (x_i - x_j) / L from the
// particles' tables tr[6][P] (cos, sin per axis)
__device__ __forceinline__ void pair_axes(const long long* tr, int P, int i, int j, long long (&c)[3], long long (&s)[3],
                                          bool want_sin)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const long long ci = tr[(2 * a) * P + i], si = tr[(2 * a + 1) * P + i];
        const long long cj = tr[(2 * a) * P + j], sj = tr[(2 * a + 1) * P + j];
        c[a] = fshl(fadd(fmh(ci, cj), fmh(si, sj)), 2);
        if (want_sin) s[a] = fshl(fsub(fmh(si, cj), fmh(ci, sj)), 2);
    }
}

// The pair function's value, gradient with respect to x_i (without its
// factor -2 pi / L) and Laplacian (without -(2 pi / L)^2), in PhiFix units.
struct PhiPair {
    long long f, g[3], l;
};

// Symmetric form for |n|^2 <= 6.  With c, d the cosines of one and two axis
// angles, u_x = c_y c_z, y_x = (d_y c_z + c_y d_z) / 2, t_x = (c_y + c_z) / 2,
// w_x = (d_y + d_z) / 2 and cyclic, a_m = vorb of the shell |n|^2 = m:
//   phi = a0 + 2 a1 sum c + 4 a2 sum u + 8 a3 c_x u_x + 2 a4 sum d + 8 a5 sum y
//         + 8 a6 sum d u,
//   d phi / d c_x = 2 a1 + 8 a2 t_x + 8 a3 u_x + 8 a5 w_x + 16 a6 y_x
//                   + 4 c_x (2 a4 + 8 a5 t_x + 8 a6 u_x),
// 64 high products for value, gradient and Laplacian, where the plane-wave
// sums take 3 x 80 multiply-adds at seven shells.
__device__ __forceinline__ void phi_sym(const PhiFix* F, const long long* tr, int P, int i, int j, bool all, PhiPair& o)
{
    long long c[3], s[3], d[3], u[3], y[3];
    pair_axes(tr, P, i, j, c, s, all);
#pragma unroll
    for (int a = 0; a < 3; ++a) d[a] = fsub(fshl(fmh(c[a], c[a]), 3), kFixOne);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, e = (a + 2) % 3;
        u[a] = fmul(c[b], c[e]);
        y[a] = fshl(fadd(fmh(d[b], c[e]), fmh(c[b], d[e])), 1);
    }
    // sums in quarters (each at most 3)
    const long long e1 = (c[0] >> 2) + (c[1] >> 2) + (c[2] >> 2);
    const long long e2 = (u[0] >> 2) + (u[1] >> 2) + (u[2] >> 2);
    const long long e3 = fmul(c[0], u[0]);
    const long long e4 = (d[0] >> 2) + (d[1] >> 2) + (d[2] >> 2);
    const long long e5 = (y[0] >> 2) + (y[1] >> 2) + (y[2] >> 2);
    const long long e6 = fmh(d[0], u[0]) + fmh(d[1], u[1]) + fmh(d[2], u[2]);
    const long long* f = F->f;
    o.f = fadd(f[0], fshl(fadd(fadd(fadd(fmh(f[1], e1), fmh(f[2], e2)), fadd(fmh(f[3], e3), fmh(f[4], e4))),
                               fadd(fmh(f[5], e5), fmh(f[6], e6))), 2));
    if (!all) return;
    o.l = fshl(fadd(fadd(fadd(fmh(f[7], e1), fmh(f[8], e2)), fadd(fmh(f[9], e3), fmh(f[10], e4))),
                    fadd(fmh(f[11], e5), fmh(f[12], e6))), 2);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, e = (a + 2) % 3;
        const long long t = (c[b] >> 1) + (c[e] >> 1), w = (d[b] >> 1) + (d[e] >> 1);
        // the brackets are at most 1; their sum in quarters
        const long long p1 = fadd(f[13] >> 2, fadd(fadd(fmh(f[14], t), fmh(f[15], u[a])), fadd(fmh(f[16], w), fmh(f[17], y[a]))));
        const long long p2 = fadd(f[18], fshl(fadd(fmh(f[19], t), fmh(f[20], u[a])), 2));
        o.g[a] = fmul(s[a], fadd(p1, fmul(c[a], p2)));
    }
}

// Octant form for any shells: c_m, s_m by the recurrence x_{m+1} = 2 c_1 x_m
// - x_{m-1}, the z sum innermost.
static __device__ __noinline__ void phi_octant(const PhiFix* F, const long long* oct, const long long* tr, int P, int i, int j,
                                        PhiPair& o)
{
    long long c[3], s[3];
    pair_axes(tr, P, i, j, c, s, true);
    const int M1 = F->M + 1, kM = F->kM, n3 = M1 * M1 * M1;
    long long f = 0, gx = 0, gy = 0, gz = 0, l = 0;
    long long cx = kFixOne, sx = 0, px = c[0], qx = -s[0];     // c_m, s_m and their predecessors
    for (int nx = 0; nx < M1; ++nx) {
        long long cy = kFixOne, sy = 0, py = c[1], qy = -s[1];
        long long f1 = 0, g1 = 0, z1 = 0, l1 = 0;
        for (int ny = 0; ny < M1; ++ny) {
            long long cz = kFixOne, sz = 0, pz = c[2], qz = -s[2];
            long long f2 = 0, z2 = 0, l2 = 0;
            const long long* A = oct + (nx * M1 + ny) * M1;
            for (int nz = 0; nz < M1; ++nz) {
                const long long a = __ldg(A + nz), b = __ldg(A + n3 + nz);
                f2 = fadd(f2, fmul(a, cz));
                z2 = fadd(z2, fmul((a >> kM) * nz, sz));
                l2 = fadd(l2, fmul(b, cz));
                const long long cn = fsub(fshl(fmh(c[2], cz), 3), pz), sn = fsub(fshl(fmh(c[2], sz), 3), qz);
                pz = cz;
                qz = sz;
                cz = cn;
                sz = sn;
            }
            f1 = fadd(f1, fmul(f2, cy));
            g1 = fadd(g1, fmul((f2 >> kM) * ny, sy));
            z1 = fadd(z1, fmul(z2, cy));
            l1 = fadd(l1, fmul(l2, cy));
            const long long cn = fsub(fshl(fmh(c[1], cy), 3), py), sn = fsub(fshl(fmh(c[1], sy), 3), qy);
            py = cy;
            qy = sy;
            cy = cn;
            sy = sn;
        }
        f = fadd(f, fmul(f1, cx));
        gx = fadd(gx, fmul((f1 >> kM) * nx, sx));
        gy = fadd(gy, fmul(g1, cx));
        gz = fadd(gz, fmul(z1, cx));
        l = fadd(l, fmul(l1, cx));
        const long long cn = fsub(fshl(fmh(c[0], cx), 3), px), sn = fsub(fshl(fmh(c[0], sx), 3), qx);
        px = cx;
        qx = sx;
        cx = cn;
        sx = sn;
    }
    o.f = f;
    o.g[0] = gx;
    o.g[1] = gy;
    o.g[2] = gz;
    o.l = l;
}

// ---- FP64 ------------------------------------------------------------------

// r = sqrt(r2) and 1/r for r2 in [1, 2^128): a single-precision reciprocal
// square root (converted by shifting exponents, on the integer pipe) refined
// by one step of Householder's third-order iteration, y <- y (1 + e/2 + 3 e^2/8)
// with e = 1 - r2 y^2, then one Newton correction of r = r2 y.  Eight FP64
// instructions where sqrt and a division take fourteen.
__device__ __forceinline__ void inv_dist(double r2, double& r, double& ri)
{
    const unsigned hi = (unsigned)__double2hiint(r2), lo = (unsigned)__double2loint(r2);
    const float x = __uint_as_float(((hi - 0x38000000u) << 3) | (lo >> 29));
    const unsigned yb = __float_as_uint(rsqrtf(x));
    const double y = __hiloint2double((int)((yb >> 3) + 0x38000000u), (int)(yb << 29));
    const double e = fma(-(r2 * y), y, 1.0);
    ri = fma(y * e, fma(e, 0.375, 0.5), y);
    const double h = __hiloint2double(__double2hiint(ri) - 0x00100000, __double2loint(ri));   // ri / 2
    const double q = r2 * ri;
    r = fma(fma(-q, q, r2), h, q);
}

// grid interval of position g >= 0 (index clamp of coshpot.f90:174) and the
// offset t from it: the integer part by masking the significand, one FP64
// subtraction
__device__ __forceinline__ int grid_split(double g, int ntab, double& t)
{
    const int hi = __double2hiint(g), e = (hi >> 20) - 1023;
    int idx;
    double base;
    if (e >= 0 && e <= 20) {
        idx = ((hi & 0xfffff) | 0x100000) >> (20 - e);
        base = __hiloint2double(hi & ~((1 << (20 - e)) - 1), 0);
    } else {
        idx = (int)g;
        base = (double)idx;
    }
    const int ic = max(1, min(idx, ntab - 2));
    t = g - (ic == idx ? base : (double)ic);
    return ic;
}

__device__ __forceinline__ double poly3(const double* c, double t)
{
    const double2 a = *reinterpret_cast<const double2*>(c), b = *reinterpret_cast<const double2*>(c + 2);
    return fma(fma(fma(b.y, t, b.x), t, a.y), t, a.x);
}

}  // namespace walker
}  // namespace dmc
