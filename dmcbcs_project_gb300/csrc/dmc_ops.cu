// Operators of the reference's block loop (operators.f90:90-124) on the GPU:
//  - g(r) of up-down, up-up and down-down pairs and the density profile
//    along x, y, z of each species (gofr.f90:53-92),
//  - S(q) of the up, down and up-down densities (sofq.f90:43-64),
//  - n(k) from single-particle moves (momentum3d.f90:89-124).
// Per walker, one CTA fills integer pair/density histograms and the S(q)
// values; for n(k), one CTA per walker runs the N x nsamp moves over its
// warps (ratios from the walker's inverse, random displacements from the
// walker's own stream by jump-ahead).  A last pass adds every walker's
// contributions with its weight, one thread per output, walkers in pop order,
// so the sums are deterministic.
#include <cuda_runtime.h>
#include <math.h>

#include "dmc_device.cuh"
#include "dmc_kernels.h"
#include "dmc_single.cuh"
#include "dmc_smem.cuh"
#include "dmc_walker.cuh"

namespace dmc {

namespace {

// r in units of L 2^-64 from a difference of positions as box fractions
__device__ __forceinline__ double fix_dist(long long e0, long long e1, long long e2)
{
    if (((e0 | e1) | e2) == 0) return 0.0;
    const double d0 = (double)e0, d1 = (double)e1, d2 = (double)e2;
    double r, ri;
    walker::inv_dist(fma(d0, d0, fma(d1, d1, d2 * d2)), r, ri);
    return r;
}

// The distance that decides a bin near an edge: r, or within 2^-46 of the range
// (and with `wide` anywhere) the minimum-image distance in FP64 from the
// positions themselves.
__device__ __noinline__ double edge_dist(double r, double pos, const double* xi, const double* xj, double el, int ntabg, bool wide)
{
    if (!wide && fabs(pos - rint(pos)) > 1.4210854715202004e-14 * ntabg) return r;
    double r2 = 0.0;
    for (int c = 0; c < 3; ++c) {
        double dx = xi[c] - xj[c];
        dx = dx - el * single::fnint(dx / el);
        r2 += dx * dx;
    }
    return sqrt(r2);
}

// One CTA per walker.  Distances and plane waves come from positions as
// 64-bit fractions of the box (dmc_pairfix.cuh): a pair's difference wraps to
// the minimum image, q.x is an integer combination of a particle's fractions,
// and rho_q is summed in fixed point (2^54 = 1) by a few threads per q vector.
// A bin is the direct distance's: the two agree to 2^-47 of the range with both
// particles within eight boxes, so within 2^-46 of a bin's edge (lattice sites
// meet the edges exactly), or with a particle farther out, the direct form
// decides.
// The FP64 pipe bounds the direct form (three divisions and a root per pair, a
// sincos per q and particle).
__global__ void __launch_bounds__(kThreads) ops_walker_kernel(const __grid_constant__ DevParams p,
                                                             const __grid_constant__ OpsDev o,
                                                             const double* __restrict__ x, int n,
                                                             int* __restrict__ hg, int* __restrict__ hd,
                                                             double* __restrict__ sv)
{
    extern __shared__ __align__(16) double osm[];
    const int P = p.npart, nup = p.nup;
    const int ng = o.ntabg > 0 ? 3 * (o.ntabg + 1) : 0, ndh = o.ntabg > 0 ? 6 * (2 * o.ntabg + 1) : 0;
    long long* xf = reinterpret_cast<long long*>(osm);
    int* g = reinterpret_cast<int*>(xf + 3 * P);
    int* d = g + ng;
    const double unit = o.el * 5.421010862427522e-20;   // L 2^-64
    for (int w = blockIdx.x; w < n; w += gridDim.x) {
        const double* xw = x + (size_t)w * 3 * P;
        unsigned long long* rho = reinterpret_cast<unsigned long long*>(sv + (size_t)w * o.nqtot * 4);
        int nan = 0;   // bit 0, 1: an up, a down coordinate that is not finite; 2: one beyond eight boxes
        for (int t = threadIdx.x; t < 3 * P; t += kThreads) {
            const double xv = xw[t];
            xf[t] = walker::box_fraction(xv, p.el, p.eli);
            if (!isfinite(xv)) nan |= t < 3 * nup ? 1 : 2;
            if (!(fabs(xv) <= 8.0 * o.el)) nan |= 4;
        }
        for (int t = threadIdx.x; t < 4 * o.nqtot; t += kThreads) rho[t] = 0ull;
        if (o.ntabg > 0)
            for (int t = threadIdx.x; t < ng + ndh; t += kThreads) g[t] = 0;
        bool nan_up = false, nan_dn = false, wide = false;
        if (__syncthreads_or(nan)) {
            nan_up = __syncthreads_or(nan & 1) != 0;
            nan_dn = __syncthreads_or(nan & 2) != 0;
            wide = __syncthreads_or(nan & 4) != 0;
        }
        if (o.ntabg > 0) {
            // every pair once (gofr.f90:57-73): particle i with i + 1 .. i + P / 2 around the ring
            const int half = P / 2;
            for (int t = threadIdx.x; t < P * half; t += kThreads) {
                const int i0 = t / half, st = t - i0 * half + 1;
                if (2 * st == P && i0 >= half) continue;
                const int j0 = i0 + st < P ? i0 + st : i0 + st - P;
                const int i = min(i0, j0), j = max(i0, j0);
                const int itab = (i < nup && j < nup) ? 1 : ((i >= nup && j >= nup) ? 2 : 0);
                double r = unit * fix_dist(walker::fsub(xf[3 * i], xf[3 * j]), walker::fsub(xf[3 * i + 1], xf[3 * j + 1]),
                                           walker::fsub(xf[3 * i + 2], xf[3 * j + 2]));
                double pos = o.scaleg * r;
                // FP32 looks first, 2^-22 of the range, at pos cut to 24 bits by shifting (an FP64
                // conversion was 3 % of g(r); below 2^-126 the value is none, but the bin is 0 in either form)
                const unsigned hi = (unsigned)__double2hiint(pos), lo = (unsigned)__double2loint(pos);
                const float at = __uint_as_float(((hi - 0x38000000u) << 3) | (lo >> 29));
                if (wide || fabsf(at - rintf(at)) <= 2.3841858e-7f * o.ntabg) {
                    r = edge_dist(r, pos, xw + 3 * i, xw + 3 * j, o.el, o.ntabg, wide);
                    pos = o.scaleg * r;
                }
                const int index = r < 0.5 * o.el ? (int)pos : o.ntabg;   // NaN counts as far
                atomicAdd(&g[itab * (o.ntabg + 1) + index], 1);
            }
            // density profile about the origin (gofr.f90:75-90)
            for (int t = threadIdx.x; t < 3 * P; t += kThreads) {
                const int i = t / 3, is = t % 3;
                double dx = xw[t];
                dx = dx - o.el * single::fnint(dx / o.el);
                const int itab = i < nup ? is : is + 3;
                const int index = (int)(o.scaleg * dx);
                atomicAdd(&d[itab * (2 * o.ntabg + 1) + index + o.ntabg], 1);
            }
        }
        // S(q): rho_k of each species, k = ak(:,1..nqtot) (k = 0 first);
        // slices of the particles, integer sums (the same in any order)
        if (o.nqtot > 0) {
            const int nsl = max(1, kThreads / o.nqtot);
            const double kap = 0.15915494309189535 * o.el;   // k -> integer components
            for (int t = threadIdx.x; t < o.nqtot * nsl; t += kThreads) {
                const int iq = t % o.nqtot, sl = t / o.nqtot;
                const double* a = o.akq + 3 * iq;
                const long long n0 = (long long)rint(a[0] * kap), n1 = (long long)rint(a[1] * kap);
                const long long n2 = (long long)rint(a[2] * kap);
                long long ur = 0, ui = 0, dr = 0, di = 0;
                for (int i = sl; i < P; i += nsl) {
                    const unsigned long long th = (unsigned long long)n0 * (unsigned long long)xf[3 * i] +
                                                  (unsigned long long)n1 * (unsigned long long)xf[3 * i + 1] +
                                                  (unsigned long long)n2 * (unsigned long long)xf[3 * i + 2];
                    long long c, s;
                    walker::fix_sincos((long long)th, c, s);
                    if (i < nup) {
                        ur += c >> 8;
                        ui -= s >> 8;
                    } else {
                        dr += c >> 8;
                        di -= s >> 8;
                    }
                }
                atomicAdd(&rho[4 * iq], (unsigned long long)ur);
                atomicAdd(&rho[4 * iq + 1], (unsigned long long)ui);
                atomicAdd(&rho[4 * iq + 2], (unsigned long long)dr);
                atomicAdd(&rho[4 * iq + 3], (unsigned long long)di);
            }
        }
        __syncthreads();
        for (int iq = threadIdx.x; iq < o.nqtot; iq += kThreads) {
            const double sc = 5.551115123125783e-17;   // 2^-54
            const double bad = __longlong_as_double(0x7ff8000000000000ll);
            const double ur = nan_up ? bad : (double)(long long)__ldcg(rho + 4 * iq) * sc;
            const double ui = nan_up ? bad : (double)(long long)__ldcg(rho + 4 * iq + 1) * sc;
            const double dr = nan_dn ? bad : (double)(long long)__ldcg(rho + 4 * iq + 2) * sc;
            const double di = nan_dn ? bad : (double)(long long)__ldcg(rho + 4 * iq + 3) * sc;
            double* out = sv + ((size_t)w * o.nqtot + iq) * 4;
            out[0] = ur * ur + ui * ui;
            out[1] = dr * dr + di * di;
            out[2] = ur * dr + ui * di;   // rhokup * conjg(rhokdn)
            out[3] = ui * dr - ur * di;
        }
        if (o.ntabg > 0) {
            for (int t = threadIdx.x; t < ng; t += kThreads) hg[(size_t)w * ng + t] = g[t];
            for (int t = threadIdx.x; t < ndh; t += kThreads) hd[(size_t)w * ndh + t] = d[t];
        }
        __syncthreads();
    }
}

// ---- n(k) with the pair function in fixed point (momentum3d.f90:89-124) -----
//
// One walker per CTA, one move per thread: move m = i nsamp + ii displaces
// particle i by L (u - 1/2) per axis (draws 3m+1..3m+3 of the walker's
// stream), and its thread runs over the opposite-spin partners j once for
// both ratios, the pair function's new entry times the inverse and the
// Jastrow sum, from one distance.  The displacement is an exact turn fraction,
// so the moved particle's axis cosines are one rotation of its own.  The
// moves' ratios times the cosine products then go to the k vectors in tiles
// of kEnkTile moves.  Bound: about 26 FP64 instructions per move and partner
// (the warp-per-move form ran a second, nearly empty round for the 33rd
// partner and took sums over k: 13.5 ms for 512 walkers at N = 66).
constexpr int kEnkTile = 32;

struct EnkLayout {
    int xf, tr, nf, Si, uold, rat, cd, A, B, C, acc, total, nsl;   // offsets in doubles
};
__host__ __device__ inline EnkLayout enk_layout(const DevParams& p, const OpsDev& o)
{
    EnkLayout L;
    const int P = p.npart, nct = o.nnk + 1;
    int off = (int)(sizeof(PhiFix) / 8) + 3 * P;   // coefficients, positions
    auto take = [&](int nd) { int q = off; off += nd; return q; };
    L.xf = take(3 * P);
    L.tr = take(6 * P);
    L.nf = take(P);
    L.Si = take(p.nd * p.nd);
    L.uold = take(P);
    L.rat = take(kThreads);
    L.cd = take(3 * kThreads);
    L.A = take(nct * kEnkTile);
    L.B = take(nct * nct * (kEnkTile + 1));
    L.C = take(nct * (kEnkTile + 1));
    L.nsl = o.nkv > 0 && o.nkv < kThreads ? kThreads / o.nkv : 1;
    L.acc = take(L.nsl * o.nkv);
    L.total = off;
    return L;
}

__global__ void __launch_bounds__(kThreads, 2) ops_enk_sym_kernel(const __grid_constant__ DevParams p,
                                                                 const __grid_constant__ OpsDev o, EnkLayout L,
                                                                 const PhiFix* __restrict__ phi,
                                                                 const TabPoly* __restrict__ tpoly,
                                                                 const TabUD* __restrict__ tud,
                                                                 const TabSS* __restrict__ tss,
                                                                 const double* __restrict__ x,
                                                                 const unsigned long long* __restrict__ irn,
                                                                 const double* __restrict__ sinv, int n,
                                                                 double* __restrict__ tk)
{
    using namespace walker;
    extern __shared__ __align__(16) double osm[];
    const int P = p.npart, nd = p.nd, nup = p.nup, ndn = p.ndn, nct = o.nnk + 1;
    const PhiFix* F = reinterpret_cast<const PhiFix*>(osm);
    double* xs = osm + sizeof(PhiFix) / 8;
    long long* xf = reinterpret_cast<long long*>(osm + L.xf);
    long long* tr = reinterpret_cast<long long*>(osm + L.tr);
    int* nf = reinterpret_cast<int*>(osm + L.nf);
    double *Si = osm + L.Si, *uold = osm + L.uold, *rat = osm + L.rat, *A = osm + L.A, *B = osm + L.B, *C = osm + L.C;
    double* acc = osm + L.acc;
    long long* cd = reinterpret_cast<long long*>(osm + L.cd);
    for (int t = threadIdx.x; t < (int)(sizeof(PhiFix) / 8); t += kThreads)
        osm[t] = reinterpret_cast<const double*>(phi)[t];
    const double unit = p.el * 5.421010862427522e-20;                  // L 2^-64
    const double tscale = (double)p.ntab * 1.0842021724855044e-19;     // grid points per unit
    const double r_min = 1.0e-14 / unit;
    const long long half = 0x43E0000000000000ll;                       // 2^63, L/2
    const double bad = __longlong_as_double(0x7ff8000000000000ll);
    // Jastrow u of an opposite-spin pair at r (units) with its grid interval,
    // zero beyond the healing distance and beyond L/2
    auto jas = [&](double r, const TabPoly* T, double t) {
        if (!(__double_as_longlong(r) < half)) return 0.0;
        if (r < r_min) T = tpoly + grid_split(r_min * tscale, p.ntab, t);
        return (int)(T - tpoly) - 1 <= p.ntab0 ? poly3(T->c[4], t) : 0.0;
    };
    const int nmove = P * o.nsamp;
    for (int w = blockIdx.x; w < n; w += gridDim.x) {
        __syncthreads();
        for (int t = threadIdx.x; t < 3 * P; t += kThreads) {
            const int pt = t / 3, a = t - 3 * pt;
            const double* xw = x + (size_t)w * 3 * P + 3 * pt;
            xs[t] = xw[a];
            const long long f = box_fraction(xw[a], p.el, p.eli);
            xf[t] = f;
            fix_sincos(f, tr[(2 * a) * P + pt], tr[(2 * a + 1) * P + pt]);
            if (a == 0) nf[pt] = !(isfinite(xw[0]) && isfinite(xw[1]) && isfinite(xw[2]));
        }
        for (int t = threadIdx.x; t < nd * nd; t += kThreads) Si[t] = sinv[(size_t)w * nd * nd + t];
        for (int t = threadIdx.x; t < L.nsl * o.nkv; t += kThreads) acc[t] = 0.0;
        __syncthreads();
        // Jastrow sums at the current positions, four lanes per particle
        for (int t0 = 0; t0 < 4 * P; t0 += kThreads) {
            const int i = (t0 + (int)threadIdx.x) >> 2, sl = threadIdx.x & 3;
            double u = 0.0;
            if (i < P) {
                const bool up = i < nup;
                const int j0 = up ? nup : 0, nj = up ? ndn : nup;
                for (int q = sl; q < nj; q += 4) {
                    const int j = j0 + q;
                    const double r = (nf[i] | nf[j]) ? bad
                                                     : fix_dist(fsub(xf[3 * i], xf[3 * j]), fsub(xf[3 * i + 1], xf[3 * j + 1]),
                                                                fsub(xf[3 * i + 2], xf[3 * j + 2]));
                    double g;
                    const TabPoly* T = tpoly + grid_split(r * tscale, p.ntab, g);
                    u += jas(r, T, g);
                }
                if (p.ieq)
                    for (int j = (up ? 0 : nup) + sl; j < (up ? nup : P); j += 4)
                        if (j != i) {
                            const double r = (nf[i] | nf[j]) ? bad
                                                             : unit * fix_dist(fsub(xf[3 * i], xf[3 * j]),
                                                                               fsub(xf[3 * i + 1], xf[3 * j + 1]),
                                                                               fsub(xf[3 * i + 2], xf[3 * j + 2]));
                            u += single::jastrow_u(p, tud, tss, false, r < 1.0e-14 ? 1.0e-14 : r);
                        }
            }
            u += __shfl_xor_sync(0xffffffffu, u, 1);
            u += __shfl_xor_sync(0xffffffffu, u, 2);
            if (i < P && sl == 0) uold[i] = u;
        }
        __syncthreads();
        const unsigned long long s0 = irn[w];
        for (int m0 = 0; m0 < nmove; m0 += kThreads) {
            const int m = m0 + (int)threadIdx.x;
            if (m < nmove) {
                const int i = m / o.nsamp;
                const bool up = i < nup;
                long long xi[3], ci[3], si[3];
                double ri[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const unsigned long long st = lcg_jump(s0, o.jA, o.jC, 3 * m + c + 1) | 1ull;
                    const long long dl = (long long)((st << 16) ^ 0x8000000000000000ull);   // u - 1/2
                    xi[c] = fadd(xf[3 * i + c], dl);
                    ri[c] = xs[3 * i + c] + ((double)st * kTwoM48 - 0.5) * p.el;
                    long long cc, ss;
                    fix_sincos(dl, cc, ss);
                    cd[3 * threadIdx.x + c] = cc;
                    const long long c0 = tr[(2 * c) * P + i], t0 = tr[(2 * c + 1) * P + i];
                    ci[c] = fshl(fsub(fmh(c0, cc), fmh(t0, ss)), 2);
                    si[c] = fshl(fadd(fmh(t0, cc), fmh(c0, ss)), 2);
                }
                double a = 0.0, u = 0.0;
                const int j0 = up ? nup : 0, nj = up ? ndn : nup;
                const double* col = up ? Si + (size_t)i * nd : Si + (i - nup);
                const int cs = up ? 1 : nd;
                for (int q = 0; q < nj; ++q) {
                    const int j = j0 + q;
                    long long c[3], sn[3];
                    SymTerms T;
                    rel_axes(ci, si, tr, P, j, c, sn, false);
                    sym_terms(c, T);
                    const long long f = fadd(F->f[0], sym_dot(F->f + 1, T.e));
                    const bool nan = (nf[i] | nf[j]) != 0;
                    const double r = nan ? bad
                                         : fix_dist(fsub(xi[0], xf[3 * j]), fsub(xi[1], xf[3 * j + 1]),
                                                    fsub(xi[2], xf[3 * j + 2]));
                    double g;
                    const TabPoly* tp = tpoly + grid_split(r * tscale, p.ntab, g);
                    const double b = !p.nobeta && (__double_as_longlong(r) <= half || nan) ? poly3(tp->c[0], g) : 0.0;
                    a = fma(col[q * cs], nan ? bad : fma((double)f, F->sphi, b), a);
                    u += jas(r, tp, g);
                }
                // unpaired plane waves of the moved particle (psislaterbcs.f90:352-365)
                for (int q = 0; q < (up ? p.nexup : p.nexdn); ++q) {
                    const double* k = up ? p.akup[q] : p.akdn[q];
                    const double arg = k[0] * ri[0] + k[1] * ri[1] + k[2] * ri[2];
                    a = fma(col[(nj + q) * cs], (up ? p.sinup[q] : p.sindn[q]) ? sin(arg) : cos(arg), a);
                }
                if (p.ieq)
                    for (int j = up ? 0 : nup; j < (up ? nup : P); ++j)
                        if (j != i) {
                            const double r = (nf[i] | nf[j]) ? bad
                                                             : unit * fix_dist(fsub(xi[0], xf[3 * j]), fsub(xi[1], xf[3 * j + 1]),
                                                                               fsub(xi[2], xf[3 * j + 2]));
                            u += single::jastrow_u(p, tud, tss, false, r < 1.0e-14 ? 1.0e-14 : r);
                        }
                rat[threadIdx.x] = exp(u - uold[i]) * a;
            } else {
                rat[threadIdx.x] = 0.0;
                cd[3 * threadIdx.x] = cd[3 * threadIdx.x + 1] = cd[3 * threadIdx.x + 2] = kFixOne;
            }
            __syncthreads();
            // psirat cos(2 pi ix dx) cos(2 pi iy dy) cos(2 pi iz dz) onto the k vectors
            const int nm = min(kThreads, nmove - m0);
            for (int b0 = 0; b0 < nm; b0 += kEnkTile) {
                const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mt = b0 + lane;
                if (warp < 3) {
                    // axis `warp`: cosines of the multiples by recurrence
                    const long long c1 = cd[3 * mt + warp];
                    long long c = kFixOne, pc = c1;
                    for (int k = 0; k < nct; ++k) {
                        const double v = (double)c * (1.0 / kFixScale);
                        if (warp == 0)
                            A[k * kEnkTile + lane] = v * rat[mt];
                        else if (warp == 1)
                            B[(k * nct) * (kEnkTile + 1) + lane] = v;   // row (k, 0), multiplied below
                        else
                            C[k * (kEnkTile + 1) + lane] = v;
                        const long long nc = fsub(fshl(fmh(c1, c), 3), pc);
                        pc = c;
                        c = nc;
                    }
                }
                __syncthreads();
                // B[iy][ix] = A[ix] cos(iy): rows by warps, ix = 0 last
                for (int k = warp; k < nct; k += kWarps) {
                    double* row = B + (size_t)k * nct * (kEnkTile + 1) + lane;
                    const double v = row[0];
                    for (int ix = nct - 1; ix >= 0; --ix) row[ix * (kEnkTile + 1)] = A[ix * kEnkTile + lane] * v;
                }
                __syncthreads();
                for (int t = threadIdx.x; t < L.nsl * o.nkv; t += kThreads) {
                    const int v = t % o.nkv, sl = t / o.nkv;
                    const int* ikv = o.ik + 3 * v;
                    const double* b = B + (size_t)(ikv[1] * nct + ikv[0]) * (kEnkTile + 1);
                    const double* c = C + (size_t)ikv[2] * (kEnkTile + 1);
                    double s = acc[t];
                    for (int k = sl; k < kEnkTile; k += L.nsl) s = fma(b[k], c[k], s);
                    acc[t] = s;
                }
                __syncthreads();
            }
        }
        // per shell, slices then vectors in order
        for (int k = threadIdx.x; k <= o.ntabk; k += kThreads) {
            double s = 0.0;
            for (int sl = 0; sl < L.nsl; ++sl)
                for (int j = 0; j < o.nkk[k]; ++j) s += acc[sl * o.nkv + o.indk[k] + j];
            tk[(size_t)w * (o.ntabk + 1) + k] = s;
        }
    }
}

// The same with the plane waves as sums over k, for shells beyond the symmetric
// form: n(k) of one walker per CTA; warp m % kWarps runs
// move m = i * nsamp + ii, whose three uniforms are draws 3m+1..3m+3 of the
// walker's stream
__global__ void __launch_bounds__(kThreads) ops_enk_kernel(const __grid_constant__ DevParams p,
                                                          const __grid_constant__ OpsDev o,
                                                          const KVecDev* __restrict__ kv,
                                                          const TabUD* __restrict__ tud,
                                                          const TabSS* __restrict__ tss,
                                                          const double* __restrict__ x,
                                                          const unsigned long long* __restrict__ irn,
                                                          const double* __restrict__ sinv, int n,
                                                          double* __restrict__ tk, int tab)
{
    extern __shared__ __align__(16) double osm[];
    const int P = p.npart, nd = p.nd, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nct = o.nnk + 1, nq = p.nk - 1;
    double* xs = osm;
    double* accv = xs + 3 * P;   // [kWarps][nkv]
    // with tab: (cos, sin) of every k vector at every particle, [nq][P], and
    // at each warp's moved particle, [kWarps][nq]
    // (16-byte aligned: the offset from the aligned start is rounded up to an even count)
    double2* cs = reinterpret_cast<double2*>(osm + ((3 * P + kWarps * o.nkv + 1) & ~1));
    double2* csn = cs + (size_t)nq * P + (size_t)warp * nq;
    // with tab: each particle's Jastrow sum at its current position, [P]
    double* uold = reinterpret_cast<double*>(cs + (size_t)nq * P + (size_t)kWarps * nq);
    for (int w = blockIdx.x; w < n; w += gridDim.x) {
        for (int t = threadIdx.x; t < 3 * P; t += kThreads) xs[t] = x[(size_t)w * 3 * P + t];
        for (int t = threadIdx.x; t < kWarps * o.nkv; t += kThreads) accv[t] = 0.0;
        __syncthreads();
        if (tab)
            for (int t = threadIdx.x; t < nq * P; t += kThreads) {
                const int k = t / P + 1, j = t - (k - 1) * P;
                double sn, c;
                sincos(kv[k].k[0] * xs[3 * j] + kv[k].k[1] * xs[3 * j + 1] + kv[k].k[2] * xs[3 * j + 2], &sn, &c);
                cs[t] = make_double2(c, sn);
            }
        if (tab)
            for (int i = warp; i < P; i += kWarps) {
                const double r[3] = {xs[3 * i], xs[3 * i + 1], xs[3 * i + 2]};
                const double u = single::warp_jastrow_sum(p, tud, tss, xs, i, r);
                if (lane == 0) uold[i] = u;
            }
        __syncthreads();
        const unsigned long long s0 = irn[w];
        const double* S = sinv + (size_t)w * nd * nd;
        double* mine = accv + warp * o.nkv;
        for (int m = warp; m < P * o.nsamp; m += kWarps) {
            const int i = m / o.nsamp;
            double dx[3], drr[3], xi[3];
            for (int c = 0; c < 3; ++c) {
                const unsigned long long st = walker::lcg_jump(s0, o.jA, o.jC, 3 * m + c + 1);
                dx[c] = (walker::lcg_uniform(st) - 0.5) * p.el;
                drr[c] = -dx[c];
                xi[c] = xs[3 * i + c] + dx[c];
            }
            double rat1, rat2;
            if (tab) {
                // getphione as exp(U(x_i') - U(x_i)) with U(x_i) computed once per walker
                rat1 = exp(single::warp_jastrow_sum(p, tud, tss, xs, i, xi) - uold[i]);
                for (int k = lane; k < nq; k += 32) {
                    double sn, c;
                    sincos(kv[k + 1].k[0] * xi[0] + kv[k + 1].k[1] * xi[1] + kv[k + 1].k[2] * xi[2], &sn, &c);
                    const double v = kv[k + 1].v;   // the shell amplitude 2 vorb, applied once per move
                    csn[k] = make_double2(v * c, v * sn);
                }
                __syncwarp();
                rat2 = single::warp_bcsone_tab(p, kv, tud, xs, S, i, xi, cs, csn);
                __syncwarp();
            } else {
                rat1 = single::warp_getphione(p, tud, tss, xs, i, drr);
                rat2 = i < p.nup ? single::warp_bcsone(p, kv, tud, xs, S + (size_t)i * p.nd, 1, i, xi)
                                : single::warp_bcsone(p, kv, tud, xs, S + (i - p.nup), p.nd, i, xi);
            }
            const double psirat = rat1 * rat2;
            // cos(dk m dx_c) for m = 0..nnk, c = 0..2, one per lane
            double ct = 1.0;
            if (lane < 3 * nct) {
                const int c = lane / nct, mm = lane % nct;
                ct = cos(o.dk * mm * dx[c]);
            }
            for (int v0 = 0; v0 < o.nkv; v0 += 32) {
                const int v = v0 + lane;
                const int* ikv = o.ik + 3 * (v < o.nkv ? v : 0);
                const double c0 = __shfl_sync(0xffffffffu, ct, ikv[0]);
                const double c1 = __shfl_sync(0xffffffffu, ct, nct + ikv[1]);
                const double c2 = __shfl_sync(0xffffffffu, ct, 2 * nct + ikv[2]);
                if (v < o.nkv) mine[v] += psirat * c0 * c1 * c2;
            }
        }
        __syncthreads();
        // per shell, warps then vectors in order
        for (int k = threadIdx.x; k <= o.ntabk; k += kThreads) {
            double s = 0.0;
            for (int ww = 0; ww < kWarps; ++ww)
                for (int j = 0; j < o.nkk[k]; ++j) s += accv[ww * o.nkv + o.indk[k] + j];
            tk[(size_t)w * (o.ntabk + 1) + k] = s;
        }
        __syncthreads();
    }
}

// Weight of each walker for the operator sums: weight * exp(psil - psigl) *
// is * wt0 (operators.f90:103), once per walker.
__global__ void ops_weight_kernel(DevStack s, int n, double* __restrict__ wt)
{
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += gridDim.x * blockDim.x)
        wt[w] = s.weight[w] * exp(s.psil[w] - s.psigl[w]) * s.is[w] * (double)s.wt0[w];
}

// The weighted sums (addgofr/addsofq/addenk accumulation), walkers in pop
// order (index n-1 first), one thread per running sum, with the walker
// weights of ops_weight_kernel.  Each sum is a serial chain over the walkers;
// small CTAs spread the chains over the SMs and eight walkers' loads are in
// flight at a time (one CTA for all sums took 4.2 ms for 512 walkers).
constexpr int kReduceThreads = 64;

template <class Term>
__device__ __forceinline__ double pop_order_sum(double acc, int n, Term term)
{
    int w = n - 1;
    for (; w >= 7; w -= 8) {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = term(w - k);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc += v[k];
    }
    for (; w >= 0; --w) acc += term(w);
    return acc;
}

__global__ void __launch_bounds__(kReduceThreads) ops_reduce_kernel(const __grid_constant__ OpsDev o, int n,
                                                                   const double* __restrict__ wts,
                                                                   const int* __restrict__ hg,
                                                                   const int* __restrict__ hd,
                                                                   const double* __restrict__ sv,
                                                                   const double* __restrict__ tk,
                                                                   double* __restrict__ sums)
{
    const int ng = o.ntabg > 0 ? 3 * (o.ntabg + 1) : 0, ndh = o.ntabg > 0 ? 6 * (2 * o.ntabg + 1) : 0;
    const int nq = 3 * o.nqtot, nk = o.nkv > 0 ? o.ntabk + 1 : 0;
    const int total = 2 * (ng + ndh + nq + nk) + 3;
    const int u = blockIdx.x * kReduceThreads + threadIdx.x;
    if (u >= total) return;
    double acc = sums[u];
    if (u < 2 * ng) {
        const int b = u % ng;
        const double f = u < ng ? 2.0 : 4.0;
        acc = pop_order_sum(acc, n, [&](int w) { return f * wts[w] * (double)hg[(size_t)w * ng + b]; });
    } else if (u < 2 * (ng + ndh)) {
        const int v = u - 2 * ng, b = v % ndh;
        const bool center = (b % (2 * o.ntabg + 1)) == o.ntabg;
        const double f = v < ndh ? (center ? 0.5 : 1.0) : (center ? 0.25 : 1.0);
        acc = pop_order_sum(acc, n, [&](int w) { return f * wts[w] * (double)hd[(size_t)w * ndh + b]; });
    } else if (u < 2 * (ng + ndh + nq)) {
        const int v = u - 2 * (ng + ndh), b = v % nq, itab = b / o.nqtot, iq = b % o.nqtot;
        acc = pop_order_sum(acc, n, [&](int w) {
            const double* e = sv + ((size_t)w * o.nqtot + iq) * 4;
            const double val = e[itab];
            const double sq = itab < 2 ? val * val : e[2] * e[2] - e[3] * e[3];
            return (v < nq ? val : sq) * wts[w];
        });
    } else if (u < total - 3) {
        const int v = u - 2 * (ng + ndh + nq), k = v % nk;
        const double nkk = o.nkk[k];
        acc = pop_order_sum(acc, n, [&](int w) {
            const double e = tk[(size_t)w * nk + k] / nkk;
            return (v < nk ? e : e * e) * wts[w];
        });
    } else {   // wsg = wsq, wsk
        const double f = u == total - 1 ? o.nsamp : 1.0;
        acc = pop_order_sum(acc, n, [&](int w) { return wts[w] * f; });
    }
    sums[u] = acc;
}

}  // namespace

static AttrCache g_attr;
enum : int { kAttrWalker = 0, kAttrEnkSym, kAttrEnk };

size_t ops_walker_smem(const DevParams& p, const OpsDev& o)
{
    return sizeof(double) * 3 * p.npart + sizeof(int) * (size_t)(3 * (o.ntabg + 1) + 6 * (2 * o.ntabg + 1)) + 16;
}

cudaError_t launch_ops_walker(const DevParams& p, const OpsDev& o, const double* x, int n, int* hg, int* hd,
                              double* sv, int grid, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const size_t smem = ops_walker_smem(p, o);
    cudaError_t e = allow_smem(g_attr, kAttrWalker, ops_walker_kernel, smem);
    if (e != cudaSuccess) return e;
    ops_walker_kernel<<<grid < n ? grid : n, kThreads, smem, st>>>(p, o, x, n, hg, hd, sv);
    return cudaGetLastError();
}

cudaError_t launch_ops_enk(const DevParams& p, const OpsDev& o, const KVecDev* kv, const TabUD* tud,
                           const TabSS* tss, const PhiFix* phi, const TabPoly* tpoly, bool sym, const double* x,
                           const unsigned long long* irn, const double* sinv, int n, double* tk, int nsm,
                           cudaStream_t st)
{
    if (n <= 0 || o.nkv <= 0) return cudaSuccess;
    // the symmetric form wherever the shells allow it and its arrays (the
    // inverse above all) fit on chip: 13.5 -> 0.6 ms for 512 walkers at N = 66
    const EnkLayout L = enk_layout(p, o);
    int dev0 = 0, optin0 = 0;
    cudaGetDevice(&dev0);
    cudaDeviceGetAttribute(&optin0, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev0);
    if (sym && (size_t)L.total * 8 <= (size_t)optin0) {
        const size_t smem = (size_t)L.total * 8;
        cudaError_t e = allow_smem(g_attr, kAttrEnkSym, ops_enk_sym_kernel, smem);
        int per_sm = 1;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ops_enk_sym_kernel, kThreads, smem);
        if (e != cudaSuccess) return e;
        const int g = nsm * (per_sm > 0 ? per_sm : 1);
        ops_enk_sym_kernel<<<g < n ? g : n, kThreads, smem, st>>>(p, o, L, phi, tpoly, tud, tss, x, irn, sinv, n, tk);
        return cudaGetLastError();
    }
    const size_t base = sizeof(double) * ((3 * (size_t)p.npart + (size_t)kWarps * o.nkv + 1) & ~(size_t)1);
    const size_t nq = p.nk > 1 ? p.nk - 1 : 1;
    const size_t with_tab = base + sizeof(double2) * nq * ((size_t)p.npart + kWarps) + sizeof(double) * p.npart;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const int tab = with_tab <= (size_t)optin ? 1 : 0;   // plane-wave tables on chip when they fit
    const size_t smem = tab ? with_tab : base;
    cudaError_t e = allow_smem(g_attr, kAttrEnk, ops_enk_kernel, smem);
    if (e != cudaSuccess) return e;
    ops_enk_kernel<<<2 * nsm < n ? 2 * nsm : n, kThreads, smem, st>>>(p, o, kv, tud, tss, x, irn, sinv, n, tk, tab);
    return cudaGetLastError();
}

cudaError_t launch_ops_reduce(const OpsDev& o, int n, const DevStack& s, const int* hg, const int* hd,
                              const double* sv, const double* tk, double* sums, double* wts, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    ops_weight_kernel<<<(n + 255) / 256, 256, 0, st>>>(s, n, wts);
    const int ng = o.ntabg > 0 ? 3 * (o.ntabg + 1) : 0, ndh = o.ntabg > 0 ? 6 * (2 * o.ntabg + 1) : 0;
    const int nk = o.nkv > 0 ? o.ntabk + 1 : 0, total = 2 * (ng + ndh + 3 * o.nqtot + nk) + 3;
    ops_reduce_kernel<<<(total + kReduceThreads - 1) / kReduceThreads, kReduceThreads, 0, st>>>(o, n, wts, hg, hd, sv, tk,
                                                                                              sums);
    return cudaGetLastError();
}

}  // namespace dmc
