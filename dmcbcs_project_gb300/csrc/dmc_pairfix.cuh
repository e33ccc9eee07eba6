// Pair terms of the FP64 walker path.
//
// GB300 issues one FP64 warp instruction per 64 cycles and sub-partition
// (DFMA, DADD and every conversion to or from double alike), a 64 x 64 -> 128
// high product (__mul64hi) takes 28 cycles there and a 64-bit add 2.  So
// whatever is bounded is computed in 64-bit fixed point on the integer pipe
// (good to 2^-57 or better, where a double's values near 1 are spaced 2^-53), and FP64 keeps what
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

// cos and sin of the turn fraction t (2^64 is one turn): the nearest quarter
// turn off, then the Taylor series in y^2, y = theta / (pi/4), with
// coefficients (pi/4)^n / n! (the first one left out is below 2^-63).
// Nineteen high products, where sincospi takes some thirty FP64 instructions.
__device__ __forceinline__ void fix_sincos(long long t, long long& c, long long& s)
{
    // (-1)^k (pi/4)^(2k) / (2k)! and (-1)^k (pi/4)^(2k+1) / (2k+1)!
    constexpr long long kc[10] = {
        4611686018427387904ll, -1422359894497287770ll, 73115257680538683ll, -1503372227063806ll, 16559920924893ll,
        -113499908640ll, 530397347ll, -1797669ll, 4620ll, -9ll};
    constexpr long long ks[9] = {
        3622009729038561421ll, -372372949609452720ll, 11484917819725252ll, -168677969434092ll, 1445125720046ll,
        -8103874527ll, 32044085ll, -94126ll, 213ll};
    const unsigned q = (unsigned)((unsigned long long)fadd(t, 1ll << 61) >> 62);
    const long long y = fshl(fsub(t, (long long)((unsigned long long)q << 62)), 1);
    const long long w = fmul(y, y);
    long long a = kc[9], b = ks[8];
#pragma unroll
    for (int k = 8; k >= 0; --k) a = fadd(kc[k], fmul(a, w));
#pragma unroll
    for (int k = 7; k >= 0; --k) b = fadd(ks[k], fmul(b, w));
    b = fmul(b, y);
    const long long cc = (q & 1u) ? b : a, ss = (q & 1u) ? a : b;
    c = (q == 1u || q == 2u) ? -cc : cc;
    s = q >= 2u ? -ss : ss;
}

// x / L as a turn fraction: h + l, l the division's remainder, so that the
// fraction is exact to 2^-64 whatever the coordinate
__device__ __forceinline__ long long box_fraction(double x, double el, double eli)
{
    const double two64 = 18446744073709551616.0;
    const double h = x * eli, l = fma(-h, el, x) * eli;
    return fadd(__double2ll_rn((h - rint(h)) * two64), __double2ll_rn(l * two64));
}

// cos and sin of the axis angles between a point (ci, si) and particle j of
// the table tr[6][P] (cos, sin per axis)
__device__ __forceinline__ void rel_axes(const long long (&ci)[3], const long long (&si)[3], const long long* tr, int P,
                                         int j, long long (&c)[3], long long (&s)[3], bool want_sin)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const long long cj = tr[(2 * a) * P + j], sj = tr[(2 * a + 1) * P + j];
        c[a] = fshl(fadd(fmh(ci[a], cj), fmh(si[a], sj)), 2);
        if (want_sin) s[a] = fshl(fsub(fmh(si[a], cj), fmh(ci[a], sj)), 2);
    }
}
__device__ __forceinline__ void pair_axes(const long long* tr, int P, int i, int j, long long (&c)[3], long long (&s)[3],
                                          bool want_sin)
{
    const long long ci[3] = {tr[i], tr[2 * P + i], tr[4 * P + i]}, si[3] = {tr[P + i], tr[3 * P + i], tr[5 * P + i]};
    rel_axes(ci, si, tr, P, j, c, s, want_sin);
}

// The pair function's value, gradient with respect to x_i (without its
// factor -2 pi / L) and Laplacian (without -(2 pi / L)^2), each in its PhiFix
// units.
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
// sums take 3 x 80 multiply-adds at seven shells.  SymTerms holds d, u, y and
// the sums e1..e6 (sum c, sum u, sum d, sum y and sum d u in quarters, c_x u_x
// whole).
struct SymTerms {
    long long d[3], u[3], y[3], e[6];
};
__device__ __forceinline__ void sym_terms(const long long (&c)[3], SymTerms& t)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) t.d[a] = fsub(fshl(fmh(c[a], c[a]), 3), kFixOne);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, e = (a + 2) % 3;
        t.u[a] = fmul(c[b], c[e]);
        t.y[a] = fshl(fadd(fmh(t.d[b], c[e]), fmh(c[b], t.d[e])), 1);
    }
    t.e[0] = (c[0] >> 2) + (c[1] >> 2) + (c[2] >> 2);
    t.e[1] = (t.u[0] >> 2) + (t.u[1] >> 2) + (t.u[2] >> 2);
    t.e[2] = fmul(c[0], t.u[0]);
    t.e[3] = (t.d[0] >> 2) + (t.d[1] >> 2) + (t.d[2] >> 2);
    t.e[4] = (t.y[0] >> 2) + (t.y[1] >> 2) + (t.y[2] >> 2);
    t.e[5] = fmh(t.d[0], t.u[0]) + fmh(t.d[1], t.u[1]) + fmh(t.d[2], t.u[2]);
}
// sum of six coefficients times e1..e6
__device__ __forceinline__ long long sym_dot(const long long* f, const long long (&e)[6])
{
    return fshl(fadd(fadd(fadd(fmh(f[0], e[0]), fmh(f[1], e[1])), fadd(fmh(f[2], e[2]), fmh(f[3], e[3]))),
                     fadd(fmh(f[4], e[4]), fmh(f[5], e[5]))), 2);
}
__device__ __forceinline__ void phi_sym(const PhiFix* F, const long long* tr, int P, int i, int j, PhiPair& o)
{
    long long c[3], s[3];
    SymTerms q;
    pair_axes(tr, P, i, j, c, s, true);
    sym_terms(c, q);
    const long long* f = F->f;
    o.f = fadd(f[0], sym_dot(f + 1, q.e));
    o.l = sym_dot(f + 7, q.e);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, e = (a + 2) % 3;
        const long long t = (c[b] >> 1) + (c[e] >> 1), w = (q.d[b] >> 1) + (q.d[e] >> 1);
        // the brackets are at most 1; their sum in quarters
        const long long p1 = fadd(f[13] >> 2, fadd(fadd(fmh(f[14], t), fmh(f[15], q.u[a])),
                                                   fadd(fmh(f[16], w), fmh(f[17], q.y[a]))));
        const long long p2 = fadd(f[18], fshl(fadd(fmh(f[19], t), fmh(f[20], q.u[a])), 2));
        o.g[a] = fmul(s[a], fadd(p1, fmul(c[a], p2)));
    }
}

// Octant form for any shells: c_m, s_m by the recurrence x_{m+1} = 2 c_1 x_m
// - x_{m-1}, the z sum innermost.  o.f is left without n = 0 and in the gradient's
// units: phi_value (here it would hold F's registers through the loops, which
// cost the walker kernel 1 %).
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

__device__ __forceinline__ long long phi_value(const PhiFix* F, long long f) { return fadd(F->f[0], f >> F->kphi); }

// ---- FP64 ------------------------------------------------------------------

// r = sqrt(r2) and 1/r for r2 in [2^-126, 2^128), FP32's normal numbers: a
// single-precision reciprocal square root (converted by shifting exponents, on the integer pipe) refined
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
