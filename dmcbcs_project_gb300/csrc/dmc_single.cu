// Single-particle moves and parameter derivatives of the DMCBS walker path
// (sm_103a):
//  - bcsone   (psislaterbcs.f90:296-376): determinant ratio for one particle
//    moved, from the stored inverse of the pair matrix;
//  - getphione (coshpot.f90:207-264): Jastrow ratio exp(U' - U) for the same
//    move; move1 (wavefunction.f90:393-404) is their product;
//  - getderbcs (psislaterbcs.f90:449-524, optsw on, optbeta off):
//    d log|det| / d vorb(shell) = tr(S^-1 dS/dvorb);
//  - the sums that calder (optimizer.f90:90-116) accumulates over a walker
//    population for the stochastic-reconfiguration step;
//  - the adjoint parameter gradients d log Psi / d theta and d E_L / d theta
//    for theta = (vorb(1..norb), bfact, b, d) of the pair function
//    (psislaterbcs.f90:249-293, betafun.f90:12-125) and the 16 knots of the
//    opt-in Jastrow spline.
// Two warps per walker for the ratios (a few hundred flops each); one CTA per
// walker for the derivatives, which contract the whole inverse.
#include <cuda_runtime.h>
#include <math.h>

#include "dmc_device.cuh"
#include "dmc_kernels.h"
#include "dmc_walker.cuh"
#include "dmc_single.cuh"
#include "dmc_smem.cuh"
#include "dmc_spline.h"

namespace dmc {


namespace {

// Single-particle ratios: kMoveThreads threads per walker (33 partners at
// N = 66 in one round; a call is often a few dozen walkers, so latency counts).
constexpr int kMoveThreads = 64;

__device__ __forceinline__ double move_sum(double v)
{
    __shared__ double red[kMoveThreads / 32];
    v = walker::warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = red[0];
#pragma unroll
    for (int k = 1; k < kMoveThreads / 32; ++k) t += red[k];
    return t;
}

// bcsone (psislaterbcs.f90:296-376) with the shells in the symmetric form: an
// entry is one polynomial of the displacement's axis cosines in fixed point
// instead of a cosine per k vector (64 walkers at N = 66: 144 -> 10 us).  inv:
// the moved particle's column (up) or row (down) of the inverse, [nw][nd].
__global__ void __launch_bounds__(kMoveThreads) bcsone_sym_kernel(const __grid_constant__ DevParams p,
                                                                 const PhiFix* __restrict__ F,
                                                                 const TabPoly* __restrict__ tpoly,
                                                                 const double* __restrict__ x,
                                                                 const double* __restrict__ inv,
                                                                 const int* __restrict__ ipart,
                                                                 const double* __restrict__ dr,
                                                                 double* __restrict__ ratio)
{
    const int w = blockIdx.x, P = p.npart, nd = p.nd;
    const double* xw = x + (size_t)w * 3 * P;
    const int i = ipart[w] - 1;   // checked on the host
    const bool up = i < p.nup;
    const double xi[3] = {xw[3 * i] - dr[3 * w], xw[3 * i + 1] - dr[3 * w + 1], xw[3 * i + 2] - dr[3 * w + 2]};
    const int nloop = up ? p.ndn : p.nup, j0 = up ? p.nup : 0;
    double acc = 0.0;
    for (int q = threadIdx.x; q < nd; q += kMoveThreads) {
        double ph;
        if (q < nloop) {
            double d[3];
            for (int c = 0; c < 3; ++c) d[c] = xi[c] - xw[3 * (j0 + q) + c];
            ph = single::phi_beta_sym(p, F, tpoly, d);
        } else {
            // unpaired plane wave of the moved particle (psislaterbcs.f90:352-365)
            const int u = q - nloop;
            const double* k = up ? p.akup[u] : p.akdn[u];
            const double arg = k[0] * xi[0] + k[1] * xi[1] + k[2] * xi[2];
            ph = (up ? p.sinup[u] : p.sindn[u]) ? sin(arg) : cos(arg);
        }
        // up: row i of S replaced, ratio = sum_q Sinv(q,i) phi_q; down: column
        acc = fma(inv[(size_t)w * nd + q], ph, acc);
    }
    const double r = move_sum(acc);
    if (threadIdx.x == 0) ratio[w] = r;
}

__global__ void bcsone_kernel(const __grid_constant__ DevParams p, const KVecDev* __restrict__ kv,
                              const TabUD* __restrict__ tud, const double* __restrict__ x,
                              const double* __restrict__ inv, const int* __restrict__ ipart,
                              const double* __restrict__ dr, double* __restrict__ ratio, int nw)
{
    const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= nw) return;
    const int P = p.npart, nd = p.nd;
    const double* xw = x + (size_t)w * 3 * P;
    const int i = ipart[w] - 1;   // checked on the host
    const double xi[3] = {xw[3 * i] - dr[3 * w], xw[3 * i + 1] - dr[3 * w + 1], xw[3 * i + 2] - dr[3 * w + 2]};
    const double r = single::warp_bcsone(p, kv, tud, xw, inv + (size_t)w * nd, 1, i, xi);
    if (lane == 0) ratio[w] = r;
}

__global__ void __launch_bounds__(kMoveThreads) getphione_kernel(const __grid_constant__ DevParams p,
                                                                const TabPoly* __restrict__ tpoly,
                                                                const TabUD* __restrict__ tud,
                                                                const TabSS* __restrict__ tss,
                                                                const double* __restrict__ x,
                                                                const int* __restrict__ ipart,
                                                                const double* __restrict__ drr,
                                                                double* __restrict__ ratio)
{
    const int w = blockIdx.x, P = p.npart;
    const double* xw = x + (size_t)w * 3 * P;
    const int i = ipart[w] - 1;
    const bool up = i < p.nup;
    // opposite-spin partners first, then (equal-spin Jastrow on) the others
    const int no = up ? p.ndn : p.nup, o0 = up ? p.nup : 0, s0 = up ? 0 : p.nup;
    const int cnt = p.ieq ? P : no;
    double u = 0.0;
    for (int q = threadIdx.x; q < cnt; q += kMoveThreads) {
        const bool opp = q < no;
        const int j = opp ? o0 + q : s0 + q - no;
        if (j == i) continue;
        double a[3], b[3];
        for (int c = 0; c < 3; ++c) {
            const double d = xw[3 * i + c] - xw[3 * j + c], e = d - drr[3 * w + c];
            a[c] = d - p.el * single::fnint(d * p.eli);
            b[c] = e - p.el * single::fnint(e * p.eli);
        }
        const double ro = single::length(a), rn = single::length(b);
        u += opp ? single::jastrow_ud(p, tpoly, rn) - single::jastrow_ud(p, tpoly, ro)
                 : single::jastrow_u(p, tud, tss, false, fmax(rn, 1.0e-14)) -
                       single::jastrow_u(p, tud, tss, false, fmax(ro, 1.0e-14));
    }
    const double t = move_sum(u);
    if (threadIdx.x == 0) ratio[w] = exp(t);
}

// d log|det| / d vorb(shell) with the shells in the symmetric form (at most
// seven, |n|^2 = shell - 1): tr(S^-1 dS/dvorb) is the inverse's up-down block
// against each pair's shell sums e1..e6, which come from one set of axis
// cosines.  One walker per CTA; 13 FP64 instructions a pair.
__global__ void __launch_bounds__(kThreads) derbcs_sym_kernel(const __grid_constant__ DevParams p,
                                                             const double* __restrict__ x,
                                                             const double* __restrict__ smati,
                                                             double* __restrict__ dpsi, int nw, int stride, int off)
{
    using namespace walker;
    __shared__ long long tr[6 * DMC_MAX_PART];
    __shared__ int nf[DMC_MAX_PART];
    __shared__ double red[kWarps][8];
    const int nd = p.nd, nup = p.nup, ndn = p.ndn, P = p.npart;
    // e1..e6 in their units: 2 sum c, 4 sum u, 8 c_x u_x, 2 sum d, 8 sum y, 8 sum d u
    const double unit[6] = {8.0, 16.0, 8.0, 8.0, 32.0, 32.0};
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        const double* xw = x + (size_t)w * 3 * P;
        const double* Si = smati + (size_t)w * nd * nd;
        for (int t = threadIdx.x; t < 3 * P; t += kThreads) {
            const int pt = t / 3, a = t - 3 * pt;
            fix_sincos(box_fraction(xw[t], p.el, p.eli), tr[(2 * a) * P + pt], tr[(2 * a + 1) * P + pt]);
            if (a == 0) nf[pt] = !(isfinite(xw[t]) && isfinite(xw[t + 1]) && isfinite(xw[t + 2]));
        }
        __syncthreads();
        double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const UDiv dv(ndn > 0 ? ndn : 1);
        for (int t = threadIdx.x; t < nup * ndn; t += kThreads) {
            const int i = dv.quo(t), j = t - i * ndn;
            double a = Si[j + (size_t)i * nd];
            long long c[3], s[3];
            SymTerms q;
            pair_axes(tr, P, i, nup + j, c, s, false);
            sym_terms(c, q);
            acc[0] += a;
            if (nf[i] | nf[nup + j]) a = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (k + 1 < p.norb) acc[k + 1] = fma(a, (double)q.e[k], acc[k + 1]);
        }
        const double v = warp_sum8(acc);
        const int lane = threadIdx.x & 31;
        if ((lane & 3) == 0) red[threadIdx.x >> 5][lane >> 2] = v;
        __syncthreads();
        if ((int)threadIdx.x < p.norb) {
            double t = 0.0;
            for (int k = 0; k < kWarps; ++k) t += red[k][threadIdx.x];
            if (threadIdx.x > 0) t *= unit[threadIdx.x - 1] * (1.0 / kFixScale);
            dpsi[(size_t)w * stride + off + threadIdx.x] = t;
        }
        __syncthreads();
    }
}

// The same for any shells:
// d log|det| / d vorb(shell) for one walker per CTA.  smati is the inverse in
// the reference's column-major layout: smati[j + i*nd] = inv(S)[j][i].
//  shell 1: sum over the up-down block of inv(S)[j][i];
//  shell s >= 2: sum_{k in s} 2 sum_i [cos(k.r_i) sum_j inv(S)[j][i] cos(k.r_j)
//                                     + sin(k.r_i) sum_j inv(S)[j][i] sin(k.r_j)]
// (cos(k.(r_i - r_j)) split into the two products).  k vectors are taken in
// chunks of kChunk with the down particles' cos/sin tabulated on chip; the
// per-(k, i) terms are summed per shell in a fixed order.
constexpr int kChunk = 8;

__global__ void __launch_bounds__(kThreads) derbcs_kernel(const __grid_constant__ DevParams p,
                                                         const KVecDev* __restrict__ kv,
                                                         const double* __restrict__ x,
                                                         const double* __restrict__ smati,
                                                         double* __restrict__ dpsi, int nw, int stride, int off)
{
    extern __shared__ __align__(16) double sm[];
    const int nd = p.nd, nup = p.nup, ndn = p.ndn, P = p.npart, norb = p.norb;
    double* Si = sm;                                  // nd*nd, column-major as smati
    double* xs = Si + nd * nd;                        // 3P
    double* cs = xs + 3 * P;                          // [kChunk][ndn][2]
    double* term = cs + kChunk * ndn * 2;             // [kChunk][nup]
    double* dsh = term + kChunk * nup;                // norb
    double* red = dsh + norb;                         // kThreads
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        for (int t = threadIdx.x; t < nd * nd; t += kThreads) Si[t] = smati[(size_t)w * nd * nd + t];
        for (int t = threadIdx.x; t < 3 * P; t += kThreads) xs[t] = x[(size_t)w * 3 * P + t];
        for (int t = threadIdx.x; t < norb; t += kThreads) dsh[t] = 0.0;
        __syncthreads();
        // shell 1: block sum of the inverse over up rows i < nup, down cols j < ndn
        {
            double s = 0.0;
            for (int t = threadIdx.x; t < nup * ndn; t += kThreads) {
                const int i = t / ndn, j = t % ndn;
                s += Si[j + i * nd];
            }
            red[threadIdx.x] = s;
            __syncthreads();
            if (threadIdx.x == 0) {
                double tot = 0.0;
                for (int t = 0; t < kThreads; ++t) tot += red[t];
                dsh[0] = tot;
            }
            __syncthreads();
        }
        for (int q0 = 1; q0 < p.nk; q0 += kChunk) {
            const int nq = min(kChunk, p.nk - q0);
            for (int t = threadIdx.x; t < nq * ndn; t += kThreads) {
                const int ql = t / ndn, j = t % ndn;
                const KVecDev& K = kv[q0 + ql];
                const double* xj = xs + 3 * (nup + j);
                double s, c;
                sincos(K.k[0] * xj[0] + K.k[1] * xj[1] + K.k[2] * xj[2], &s, &c);
                cs[2 * (ql * ndn + j)] = c;
                cs[2 * (ql * ndn + j) + 1] = s;
            }
            __syncthreads();
            for (int t = threadIdx.x; t < nq * nup; t += kThreads) {
                const int ql = t / nup, i = t % nup;
                const KVecDev& K = kv[q0 + ql];
                const double* xi = xs + 3 * i;
                double si, ci;
                sincos(K.k[0] * xi[0] + K.k[1] * xi[1] + K.k[2] * xi[2], &si, &ci);
                double gc = 0.0, gs = 0.0;
                const double* col = Si + (size_t)i * nd;
                const double* cq = cs + 2 * ql * ndn;
                for (int j = 0; j < ndn; ++j) {
                    gc = fma(col[j], cq[2 * j], gc);
                    gs = fma(col[j], cq[2 * j + 1], gs);
                }
                term[ql * nup + i] = 2.0 * (ci * gc + si * gs);
            }
            __syncthreads();
            if (threadIdx.x == 0)
                for (int ql = 0; ql < nq; ++ql) {
                    double s = 0.0;
                    for (int i = 0; i < nup; ++i) s += term[ql * nup + i];
                    dsh[kv[q0 + ql].shell - 1] += s;
                }
            __syncthreads();
        }
        for (int t = threadIdx.x; t < norb; t += kThreads) dpsi[(size_t)w * stride + off + t] = dsh[t];
        __syncthreads();
    }
}

// N sums over the CTA (N a multiple of 8) in a fixed order: transposed warp
// sums, then the warps in order.  red holds at least kWarps * N doubles; the
// first n of the sums k < N/2 go to outa[k], those of the rest to
// outb[k - N/2].
template <int N>
__device__ void block_sum_n(double (&v)[N], double* red, double* outa, double* outb, int n)
{
    static_assert(N % 8 == 0 && N * kWarps <= kThreads, "sums of eight, in the reduction buffer");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int g = 0; g < N / 8; ++g) {
        double u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] = v[8 * g + k];
        const double a = walker::warp_sum8(u);
        if ((lane & 3) == 0) red[warp * N + 8 * g + (lane >> 2)] = a;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        const bool second = threadIdx.x >= N / 2;
        const int k = second ? (int)threadIdx.x - N / 2 : (int)threadIdx.x;
        double t = 0.0;
        for (int q = 0; q < kWarps; ++q) t += red[q * N + threadIdx.x];
        if (k < n) (second ? outb : outa)[k] = t;
    }
    __syncthreads();
}

// Adjoint parameter gradients, one walker per CTA (FP64).
//
// The determinant's share of the kinetic term of E_L = -hbar d2psi + v is
//   Q = sum_p (1/m_p) [ lap_p Phi / Phi + 2 grad_p log Phi . grad_p J ]
//     = tr(S^-1 M),   M_ij = sum over the particles p that entry (i,j) of the
//                     pair matrix depends on of (1/m_p) lap_p S_ij
//                     + 2 grad_p S_ij . w_p,   w_p = grad_p J / m_p,
// because S is linear in each particle's row or column (psislaterbcs.f90:
// 209-223).  J (Jastrow, one-body and long-range terms) and v do not depend
// on theta, so with S' = dS/dtheta and M' = dM/dtheta
//   d log Psi / d theta = tr(S^-1 S')
//   d Q / d theta       = tr(S^-1 M') - tr(T S'),   T = S^-1 M S^-1
// and d E_L / d theta = -hbar dQ/dtheta: one extra pair of nd^3 products per
// walker gives every parameter.  Only the up-down block depends on the pair
// function's parameters: phi = vorb(1) + sum_k 2 vorb(shell k) cos(k.r) +
// beta(r), beta linear in bfact and given with its b and d derivatives as
// tables on the beta grid (the derivatives of the image-summed, shifted,
// bfact-scaled table that Psi uses).
//
// Per up-down pair (i, j) and shell s >= 2 (all k of a shell have the same
// k^2 and amplitude v_s = 2 vorb(s)), with C_s = sum_{k in s} cos(k.r_ij) and
// H_s = sum_{k in s} k sin(k.r_ij):
//   S_ij  = ... + v_s C_s                      S'_s,ij = 2 C_s
//   M_ij  = ... - v_s (k_s^2 C_s (1/m_i + 1/m_j) + 2 H_s . (w_i - w_j))
//   M'_s,ij = -2 k_s^2 C_s (1/m_i + 1/m_j) - 4 H_s . (w_i - w_j)
// and M is the sum of vorb(s) M'_s and of beta's share.  SYM (shells in the
// symmetric form, |n|^2 = s - 1 <= 6): with kappa = 2 pi / L, S'_s is a
// polynomial U_s of the pair's axis cosines c_a, and
//   M'_s,ij = -kappa^2 (s - 1) (1/m_i + 1/m_j) S'_s
//             - 2 kappa sum_a sin_a dU_s/dc_a (w_i - w_j)_a,
// 34 integer high products and 65 FP64 instructions a pair for six shells,
// where the 40 k vectors took about 400.  The pass that forms M keeps
// (S', M') of every pair and pair-function parameter, so that the sums after
// T cost three multiply-adds a pair and parameter, and it takes the distance
// and the grid interval once for beta, its derivatives and the knots, each a
// cubic per interval.
//
// The 16 knots t_k of the opt-in up-down Jastrow spline are Jastrow
// parameters: J = ... + sum_pairs sum_k t_k phi_k(r), so
//   d log Psi / d t_k = sum_pairs phi_k(r)
//   d E_L / d t_k     = -hbar sum_pairs [ (1/m_i + 1/m_j)(phi_k'' + 2 phi_k'/r)
//                        + 2 phi_k'/r d.(g_i - g_j) ],  g_p = grad_p log Psi / m_p,
// with phi_k, phi_k', phi_k'' interpolated from their values on the Jastrow
// table's grid (the values the table itself was built from) with the pair's
// 4-point interpolation, as the pair loop interpolates the Jastrow table they
// are added to.
// Inputs per walker: x, the inverse (column-major as smati), the total and
// determinant drifts (grad / sqrt m) whose difference is grad J.  Outputs
// dlog[w*np + t], deloc[w*np + t] for t = vorb(1..norb), then bfact, b, d
// (nbeta = 3 with the beta function on), then the knots (nknot = 16 with the
// spline on).
// Memory: the CTA's core (inverse, M, product buffer, per-particle vectors,
// reductions) in shared memory (in core_g when it does not fit); the per-pair
// parameter derivatives and, without SYM, the axis powers e^{i 2 pi m x_a / L}
// and the plane waves of every k at every particle in the CTA's slice of
// slice_g (L2).
// Bound: the FP64 pipe (89 % busy); 66 of its instructions a pair are the two
// products, about 190 the pass that forms M.  2048 walkers at N = 66 with 26
// parameters: 1.37 ms, the whole call 5.12 -> 2.33 ms (sums over k vectors,
// Lagrange weights and a distance per parameter group before).
template <bool SYM>
__global__ void __launch_bounds__(kThreads, 2) pgrad_kernel(const __grid_constant__ DevParams p,
                                                            const KVecDev* __restrict__ kv,
                                                            const TabPoly* __restrict__ tpoly,
                                                            const double* __restrict__ x,
                                                            const double* __restrict__ sinv,
                                                            const double* __restrict__ dpsi,
                                                            const double* __restrict__ dphi, double* __restrict__ dlog,
                                                            double* __restrict__ deloc, int nw, int np, double bfact,
                                                            const PgPoly* __restrict__ btd,
                                                            const PgPoly* __restrict__ ktd, int nbeta, int nknot,
                                                            double* core_g, size_t core_per, double* slice_g,
                                                            size_t slice_per)
{
    using namespace walker;
    extern __shared__ __align__(16) double smp[];
    double* base = core_g ? core_g + (size_t)blockIdx.x * core_per : smp;
    const int nd = p.nd, nup = p.nup, ndn = p.ndn, P = p.npart, nq = p.nk - 1, norb = p.norb;
    const size_t nd2 = (size_t)nd * nd;
    double* Si = base;                 // (S^-1)_{rc} = Si[r + c nd]
    double* M = Si + nd2;              // M, later T
    double* B = M + nd2;               // M S^-1
    double* xs = B + nd2;              // [P][3]
    double* w = xs + 3 * P;            // [P][3]: grad J / m
    double* gt = w + 3 * P;            // [P][3]: grad log Psi / m
    double* red = gt + 3 * P;
    double* res = red + kThreads;      // [2][kPgradMax]: d log Psi, then d Q
    double* va = res + 2 * kPgradMax;  // vorb of the shells s >= 2
    int* sh0 = reinterpret_cast<int*>(va + norb);             // first k of each shell s >= 2, then the end
    int* nf = sh0 + norb + 1;                                 // [P]: a coordinate that is not finite
    long long* xf = reinterpret_cast<long long*>(va + norb + (norb + 2 + P) / 2);   // [P][3]: fractions of the box
    long long* tr = xf + 3 * P;                               // [6][P]: cos, sin of the axis angles
    const int np1 = p.nmax + 1, nsh = norb - 1, npairs = nup * ndn;
    const int nsp = nsh + nbeta;       // parameters with an entry in dsm
    double2* dsm = reinterpret_cast<double2*>(slice_g + (size_t)blockIdx.x * slice_per);   // [nsp][npairs]
    double2* E = dsm + (size_t)nsp * npairs;                                               // [P][3][np1]
    double2* cs = E + (size_t)3 * P * np1;                                                 // [nq][P]
    const int npb = norb + nbeta;      // parameters of the pair function
    const double imu = p.imass[0], imd = p.imass[1], ims = imu + imd;
    // distances in units of L 2^-64 (L/2 = 2^63), as in the walker kernel
    const double unit = p.el * 5.421010862427522e-20, iu = 1.0 / unit;
    const double tscale = (double)p.ntab * 1.0842021724855044e-19, r_min = 1.0e-14 * iu;
    const long long half = 0x43E0000000000000ll;
    const double two62 = 4.611686018427387904e18, i62 = 1.0 / two62;
    const double kap = 6.283185307179586 * p.eli;
    const UDiv dv(ndn > 0 ? ndn : 1);
    if (threadIdx.x == 0) {
        // k vectors are sorted by shell; shell 1 is k = 0
        int q = 1;
        for (int sh = 2; sh <= norb; ++sh) {
            sh0[sh - 2] = q;
            va[sh - 2] = q < p.nk && kv[q].shell == sh ? 0.5 * kv[q].v : 0.0;
            while (q < p.nk && kv[q].shell == sh) ++q;
        }
        sh0[norb - 1] = q;
    }
    for (int wk = blockIdx.x; wk < nw; wk += gridDim.x) {
        for (size_t t = threadIdx.x; t < nd2; t += kThreads) Si[t] = sinv[(size_t)wk * nd2 + t];
        for (int t = threadIdx.x; t < 3 * P; t += kThreads) {
            const size_t g = (size_t)wk * 3 * P + t;
            const int pt = t / 3, a = t - 3 * pt;
            const double xv = x[g];
            xs[t] = xv;
            const int sp = pt < nup ? 0 : 1;
            w[t] = (dpsi[g] - dphi[g]) * p.isqm[sp];
            gt[t] = dpsi[g] * p.isqm[sp];
            xf[t] = box_fraction(xv, p.el, p.eli);
            if (a == 0) nf[pt] = !(isfinite(xv) && isfinite(x[g + 1]) && isfinite(x[g + 2]));
            if constexpr (SYM) {
                fix_sincos(xf[t], tr[(2 * a) * P + pt], tr[(2 * a + 1) * P + pt]);
            } else {
                // powers of e^{i 2 pi x_a / L}, m = 0..nmax
                double s1, c1;
                sincospi(2.0 * xv * p.eli, &s1, &c1);
                double2* e = E + (size_t)t * np1;
                e[0] = make_double2(1.0, 0.0);
                double cr = c1, ci = s1;
                if (np1 > 1) e[1] = make_double2(c1, s1);
                for (int m = 2; m < np1; ++m) {
                    const double nr = cr * c1 - ci * s1, ni = cr * s1 + ci * c1;
                    cr = nr;
                    ci = ni;
                    e[m] = make_double2(cr, ci);
                }
            }
        }
        __syncthreads();
        if constexpr (!SYM) {
            // e^{i k_q . x_p} as the product of the three axis powers
            for (int t = threadIdx.x; t < nq * P; t += kThreads) {
                const int q = t / P + 1, pp = t - (q - 1) * P;
                const KVecDev& K = kv[q];
                const double2* eb = E + (size_t)pp * 3 * np1;
                const int n0 = K.n[0];
                const double2 e0 = eb[n0 < 0 ? -n0 : n0];
                double zr = e0.x, zi = n0 < 0 ? -e0.y : e0.y;
#pragma unroll
                for (int a = 1; a < 3; ++a) {
                    const int n = K.n[a];
                    const double2 e = eb[a * np1 + (n < 0 ? -n : n)];
                    const double er = e.x, ei = n < 0 ? -e.y : e.y;
                    const double nr = zr * er - zi * ei, ni = zr * ei + zi * er;
                    zr = nr;
                    zi = ni;
                }
                cs[t] = make_double2(zr, zi);
            }
            __syncthreads();
        }
        // the up-down block of M (psislaterbcs.f90:249-293 for the entries and
        // their derivatives), every pair's parameter derivatives on the side,
        // and the knots' sums, which need no more than the pair
        double kacc[2 * kJastrowKnots];
#pragma unroll
        for (int k = 0; k < 2 * kJastrowKnots; ++k) kacc[k] = 0.0;
        for (int t = threadIdx.x; t < npairs; t += kThreads) {
            const int i = dv.quo(t), j = t - i * ndn, pj = nup + j;
            const double wd[3] = {w[3 * i] - w[3 * pj], w[3 * i + 1] - w[3 * pj + 1], w[3 * i + 2] - w[3 * pj + 2]};
            const bool nan = (nf[i] | nf[pj]) != 0;
            const double not_num = __longlong_as_double(0x7ff8000000000000ll);
            double2* dp = dsm + t;
            double m = 0.0;
            if constexpr (SYM) {
                // S' in units of 2^-62 {8, 16, 8, 8, 32, 32}, M' likewise
                long long c[3], s[3];
                SymTerms q;
                pair_axes(tr, P, i, pj, c, s, true);
                sym_terms(c, q);
                double g[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int b = (a + 1) % 3, e = (a + 2) % 3;
                    const long long tm = (c[b] >> 1) + (c[e] >> 1), hw = (q.d[b] >> 3) + (q.d[e] >> 3);
                    const double f = wd[a] * (double)s[a];
                    g[0] += f;
                    g[1] = fma(f, (double)tm, g[1]);
                    g[2] = fma(f, (double)q.u[a], g[2]);
                    g[3] = fma(f, (double)c[a], g[3]);
                    g[4] = fma(f, (double)fadd(hw, fmul(c[a], tm)), g[4]);
                    g[5] = fma(f, (double)fadd(q.y[a] >> 1, fmul(c[a], q.u[a])), g[5]);
                }
                constexpr double ratio[6] = {0.25, 0.5, 1.0, 1.0, 1.0, 1.0}, un[6] = {8.0, 16.0, 8.0, 8.0, 32.0, 32.0};
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    if (k < nsh) {
                        const double ds = nan ? not_num : (double)q.e[k];
                        const double dm = fma(g[k], -2.0 * ratio[k] * kap * (k == 0 ? 1.0 : i62),
                                              ds * (-kap * kap * (k + 1) * ims));
                        m = fma(va[k] * (un[k] * i62), dm, m);
                        dp[(size_t)k * npairs] = make_double2(ds, dm);
                    }
            } else {
                double l = 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0;
                for (int s = 0; s < nsh; ++s) {
                    const int q0 = sh0[s], q1 = sh0[s + 1];
                    double cc = 0.0, h0 = 0.0, h1 = 0.0, h2 = 0.0;
                    for (int q = q0; q < q1; ++q) {
                        const KVecDev& K = kv[q];
                        const double2 ci = cs[(size_t)(q - 1) * P + i];
                        const double2 cj = cs[(size_t)(q - 1) * P + pj];
                        const double co = fma(ci.x, cj.x, ci.y * cj.y);
                        const double si = fma(ci.y, cj.x, -ci.x * cj.y);
                        cc += co;
                        h0 = fma(si, K.k[0], h0);
                        h1 = fma(si, K.k[1], h1);
                        h2 = fma(si, K.k[2], h2);
                    }
                    double ds = 0.0, dm = 0.0;
                    if (q1 > q0) {
                        const double v = kv[q0].v, k2c = kv[q0].k2 * cc;
                        const double hw = h0 * wd[0] + h1 * wd[1] + h2 * wd[2];
                        l -= v * k2c;
                        g0 -= v * h0;
                        g1 -= v * h1;
                        g2 -= v * h2;
                        ds = 2.0 * cc;
                        dm = -2.0 * k2c * ims - 4.0 * hw;
                    }
                    dp[(size_t)s * npairs] = make_double2(ds, dm);
                }
                m = l * ims + 2.0 * (g0 * wd[0] + g1 * wd[1] + g2 * wd[2]);
            }
            if (nbeta > 0 || nknot > 0) {
                const long long e0 = fsub(xf[3 * i], xf[3 * pj]), e1 = fsub(xf[3 * i + 1], xf[3 * pj + 1]);
                const long long e2 = fsub(xf[3 * i + 2], xf[3 * pj + 2]);
                double d0 = (double)e0, d1 = (double)e1, d2 = (double)e2, r, ri;
                if (nan) d0 = not_num;
                if (((e0 | e1) | e2) != 0 || nan) {
                    inv_dist(fma(d0, d0, fma(d1, d1, d2 * d2)), r, ri);
                } else {   // closer than a unit, or coincident
                    d0 = min_image(xs[3 * i] - xs[3 * pj], p) * iu;
                    d1 = min_image(xs[3 * i + 1] - xs[3 * pj + 1], p) * iu;
                    d2 = min_image(xs[3 * i + 2] - xs[3 * pj + 2], p) * iu;
                    r = sqrt(norm2(d0, d1, d2));
                    ri = r > 0.0 ? 1.0 / r : 0.0;
                }
                double tt;
                int o = grid_split(r * tscale, p.ntab, tt);
                if (nbeta > 0) {
                    // bfact (beta itself, over bfact at the end), b and d
                    double f[3] = {0.0, 0.0, 0.0}, dm[3] = {0.0, 0.0, 0.0};
                    if (__double_as_longlong(r) <= half || nan) {
                        const double gw = 2.0 * (ri * fma(d0, wd[0], fma(d1, wd[1], d2 * wd[2])));
                        const TabPoly* T = tpoly + o;
                        f[0] = poly3(T->c[0], tt);
                        dm[0] = fma(poly3(T->c[2], tt), ims, poly3(T->c[1], tt) * gw);
#pragma unroll
                        for (int q = 1; q < 3; ++q) {
                            const PgPoly* G = btd + 2 * o + (q - 1);
                            f[q] = poly3(G->c[0], tt);
                            dm[q] = fma(poly3(G->c[2], tt), ims, poly3(G->c[1], tt) * gw);
                        }
                    }
                    m += dm[0];
#pragma unroll
                    for (int q = 0; q < 3; ++q) dp[(size_t)(nsh + q) * npairs] = make_double2(f[q], dm[q]);
                }
                if (nknot > 0) {
                    if (!(r >= r_min)) {   // the reference's clamp, coshpot.f90:170
                        r = r_min;
                        ri = 1.0 / r_min;
                        o = grid_split(r * tscale, p.ntab, tt);
                    }
                    if (__double_as_longlong(r) < half) {
                        const double gd = fma(d0, gt[3 * i] - gt[3 * pj],
                                              fma(d1, gt[3 * i + 1] - gt[3 * pj + 1], d2 * (gt[3 * i + 2] - gt[3 * pj + 2])));
                        const double cp = 2.0 * ri * fma(ims, iu, gd);   // weight of phi' (phi'' has ims)
                        // grid rows o - 1 .. o + 2 in units of the knot spacing
                        // (t = r / h): the knots whose support (k - 2, k + 2)
                        // (and the mirror image of k = 1 below one spacing)
                        // reaches them, with a margin over FP32's rounding
                        const float ts = 0.5f * (float)kJastrowCells / (float)p.ntab;
                        const int klo = max(0, (int)((o - 1) * ts - 1.0e-4f) - 1);
                        const int khi = min(kJastrowKnots - 1, (int)((o + 2) * ts + 1.0e-4f) + 2);
                        const PgPoly* T = ktd + (size_t)o * kJastrowKnots;
#pragma unroll 1
                        for (int k = klo; k <= khi; ++k) {
                            const double fp = poly3(T[k].c[1], tt), fpp = poly3(T[k].c[2], tt);
                            kacc[k] += poly3(T[k].c[0], tt);
                            kacc[kJastrowKnots + k] = fma(ims, fpp, fma(cp, fp, kacc[kJastrowKnots + k]));
                        }
                    }
                }
            }
            M[i + (size_t)j * nd] = m;
        }
        // unpaired plane waves (psislaterbcs.f90:171-206): up ones in columns
        // j >= ndn (each depends on up particle i), down ones in rows i >= nup
        // (on down particle j), and the zero corner
        const int nun = (nd - ndn) * nd, nrow = (nd - nup) * ndn;
        for (int t = threadIdx.x; t < nun + nrow; t += kThreads) {
            int i, j;
            if (t < nun) {
                i = t % nd;
                j = ndn + t / nd;
            } else {
                i = nup + (t - nun) / ndn;
                j = (t - nun) % ndn;
            }
            double m = 0.0;
            if (i < nup) {
                const int u = j - ndn;
                const double* k = p.akup[u];
                double sn, c;
                sincos(k[0] * xs[3 * i] + k[1] * xs[3 * i + 1] + k[2] * xs[3 * i + 2], &sn, &c);
                const double a = p.sinup[u] ? c : -sn;        // d/d(k.x) of the entry
                const double e = p.sinup[u] ? sn : c;
                m = -p.ak2up[u] * e * imu + 2.0 * a * (k[0] * w[3 * i] + k[1] * w[3 * i + 1] + k[2] * w[3 * i + 2]);
            } else if (j < ndn) {
                const int u = i - nup, pj = nup + j;
                const double* k = p.akdn[u];
                double sn, c;
                sincos(k[0] * xs[3 * pj] + k[1] * xs[3 * pj + 1] + k[2] * xs[3 * pj + 2], &sn, &c);
                const double a = p.sindn[u] ? c : -sn;
                const double e = p.sindn[u] ? sn : c;
                m = -p.ak2dn[u] * e * imd + 2.0 * a * (k[0] * w[3 * pj] + k[1] * w[3 * pj + 1] + k[2] * w[3 * pj + 2]);
            }
            M[i + (size_t)j * nd] = m;
        }
        __syncthreads();
        if (nknot > 0) block_sum_n<2 * kJastrowKnots>(kacc, red, res + npb, res + kPgradMax + npb, nknot);
        // B = M S^-1, then T = S^-1 B (into M)
        for (size_t t = threadIdx.x; t < nd2; t += kThreads) {
            const int i = (int)(t % nd), j = (int)(t / nd);
            double s = 0.0;
            for (int k = 0; k < nd; ++k) s = fma(M[i + (size_t)k * nd], Si[k + (size_t)j * nd], s);
            B[t] = s;
        }
        __syncthreads();
        for (size_t t = threadIdx.x; t < nd2; t += kThreads) {
            const int i = (int)(t % nd), j = (int)(t / nd);
            double s = 0.0;
            for (int k = 0; k < nd; ++k) s = fma(Si[i + (size_t)k * nd], B[k + (size_t)j * nd], s);
            M[t] = s;
        }
        __syncthreads();
        // per pair-function parameter (twelve at a time): sums over the up-down
        // pairs of S^-1_ji S'_ij and S^-1_ji M'_ij - T_ji S'_ij
        for (int th0 = 0; th0 < npb; th0 += 12) {
            double acc[24];
#pragma unroll
            for (int k = 0; k < 24; ++k) acc[k] = 0.0;
            for (int t = threadIdx.x; t < npairs; t += kThreads) {
                const int i = dv.quo(t), j = t - i * ndn;
                const double a = Si[j + (size_t)i * nd], tt = M[j + (size_t)i * nd];
#pragma unroll
                for (int u = 0; u < 12; ++u) {
                    const int th = th0 + u;
                    if (th < npb) {
                        if (th == 0) {   // vorb(1): S' = 1, M' = 0
                            acc[u] += a;
                            acc[12 + u] -= tt;
                        } else {
                            const double2 v = dsm[(size_t)(th - 1) * npairs + t];
                            acc[u] = fma(a, v.x, acc[u]);
                            acc[12 + u] = fma(-tt, v.x, fma(a, v.y, acc[12 + u]));
                        }
                    }
                }
            }
            block_sum_n<24>(acc, red, res + th0, res + kPgradMax + th0, npb - th0);
        }
        for (int th = threadIdx.x; th < np; th += kThreads) {
            double f = 1.0;   // of the shells' units, and of beta / bfact
            if (SYM && th > 0 && th < norb) f = (th == 2 ? 16.0 : th >= 5 ? 32.0 : 8.0) * i62;
            if (nbeta > 0 && th == norb) f = 1.0 / bfact;
            dlog[(size_t)wk * np + th] = res[th] * f;
            deloc[(size_t)wk * np + th] = -p.hbar * (res[kPgradMax + th] * f);
        }
        __syncthreads();
    }
}

// getjasder (jastrowlongrange.f90:63-78) for one walker per CTA: the
// long-range Jastrow at beta + dp, (beta + dp) - 2 dp and back, from the
// densities rho_q; d/d beta by central differences as the reference takes
// them, d/d gamma = U / gamma.  Writes dpsi[w*stride + 0..1].
__global__ void __launch_bounds__(kThreads) jasder_kernel(const __grid_constant__ DevParams p,
                                                         const double* __restrict__ jq,
                                                         const double* __restrict__ x,
                                                         double* __restrict__ dpsi, int nw, int stride)
{
    extern __shared__ __align__(16) double sm[];
    const int P = p.npart;
    double* r2 = sm;   // |rho_q|^2 - N per q
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        const double* xw = x + (size_t)w * 3 * P;
        for (int q = threadIdx.x; q < p.nql; q += kThreads) {
            const double* Q = jq + 8 * q;
            double re = 0.0, im = 0.0;
            for (int i = 0; i < P; ++i) {
                double sn, cs;
                sincos(Q[0] * xw[3 * i] + Q[1] * xw[3 * i + 1] + Q[2] * xw[3 * i + 2], &sn, &cs);
                re += cs;
                im += sn;
            }
            r2[q] = re * re + im * im - (double)P;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const double dp = 0.0001;
            const double b1 = p.jbeta + dp, b2 = b1 - 2.0 * dp, b3 = b2 + dp;
            double u1 = 0.0, u2 = 0.0, u3 = 0.0;
            for (int q = 0; q < p.nql; ++q) {
                const double qmod = sqrt(jq[8 * q + 3]);
                u1 += p.jgamma * exp(-b1 * qmod) / qmod * r2[q];
                u2 += p.jgamma * exp(-b2 * qmod) / qmod * r2[q];
                u3 += p.jgamma * exp(-b3 * qmod) / qmod * r2[q];
            }
            dpsi[(size_t)w * stride] = (u1 - u2) / (2.0 * dp);
            dpsi[(size_t)w * stride + 1] = u3 / p.jgamma;
        }
        __syncthreads();
    }
}

// calder sums (optimizer.f90:105-115) over a population, in pop order (the
// top of the stack, index n-1, first): ovec += d, ovecw += d*e, pmat += d d^T,
// esum += e, esum2 += e^2 with e = E_L / eunit / npart.  One thread per
// output, so every sum runs over the walkers in the same order as the
// reference's loop; products are rounded before the add (no contraction).
// ene = (-hbar*d2psi + v)/eunit/npart (dmcbcs.f90:497), once per walker
__global__ void sr_energy_kernel(const double* __restrict__ d2psi, const double* __restrict__ v, int n,
                                 double hbar, double eunit, double npart, double* __restrict__ ene)
{
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += gridDim.x * blockDim.x)
        ene[w] = __ddiv_rn(__ddiv_rn(__dadd_rn(__dmul_rn(-hbar, d2psi[w]), v[w]), eunit), npart);
}

// Bound: the serial chain of one addition per walker (65 cycles each).  One
// warp per CTA adds 32 outputs' chains; the other three make the next tile's
// products meanwhile, so nothing but the addition is on the chain (loads and
// products on it too, in one CTA: 0.95 ms for 2048 walkers and 65 sums).
constexpr int kSrTile = 64, kSrOut = 32;

__global__ void __launch_bounds__(128) sr_sums_kernel(const double* __restrict__ der, const double* __restrict__ ene,
                                                      int n, int np, double* __restrict__ sums)
{
    __shared__ double term[2][kSrTile][kSrOut + 1];
    const int nout = np * np + 2 * np + 2, o0 = blockIdx.x * kSrOut;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = o0 + lane;
    const int ntile = (n + kSrTile - 1) / kSrTile;
    // the terms of tile k (walkers n-1 - k kSrTile downwards), every third row by each of three warps
    auto fill = [&](int k) {
        if (t >= nout) return;
        for (int r = warp - 1; r < kSrTile; r += 3) {
            const int w = n - 1 - k * kSrTile - r;
            if (w < 0) break;
            const double e = ene[w];
            const double* d = der + (size_t)w * np;
            double v;
            if (t < np)
                v = d[t];
            else if (t < 2 * np)
                v = __dmul_rn(d[t - np], e);
            else if (t < 2 * np + np * np) {
                const int q = t - 2 * np, i = q % np, j = q / np;   // column-major pmat(i,j)
                v = __dmul_rn(d[i], d[j]);
            } else
                v = t == nout - 2 ? e : __dmul_rn(e, e);
            term[k & 1][r][lane] = v;
        }
    };
    double s = warp == 0 && t < nout ? sums[t] : 0.0;
    if (warp > 0) fill(0);
    __syncthreads();
    for (int k = 0; k < ntile; ++k) {
        if (warp == 0) {
            if (t < nout) {
                const int m = min(kSrTile, n - k * kSrTile);
                for (int r = 0; r < m; ++r) s = __dadd_rn(s, term[k & 1][r][lane]);
            }
        } else if (k + 1 < ntile) {
            fill(k + 1);
        }
        __syncthreads();
    }
    if (warp == 0 && t < nout) sums[t] = s;
}

}  // namespace

// The cubic through four grid points in t = position - 1, from differences (an
// interval's own points give no cancellation).
__device__ __forceinline__ void interval_cubic(double t0, double t1, double t2, double t3, double* c)
{
    const double d1 = t2 - t1;
    const double a3 = fma(-3.0, d1, t3 - t0) / 6.0, a2 = ((t0 - t1) + d1) * 0.5;
    c[0] = t1;
    c[1] = (d1 - a2) - a3;
    c[2] = a2;
    c[3] = a3;
}

// One thread per cubic.  Made on the host and copied, they cost set_beta 0.18 ms
// (716 -> 480 us with one copy of the tables) and the gradient after it as much.
__global__ void tab_poly_kernel(const TabUD* __restrict__ tud, TabPoly* __restrict__ out, int nt)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / 7, k = t - 7 * i;
    if (i >= nt) return;
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    if (i >= 1 && i + 2 < nt) {
        constexpr int field[7] = {4, 5, 6, 0, 1, 2, 3};   // beta, beta', lap beta, v, u, u', u'' in a TabUD
        const double* T = reinterpret_cast<const double*>(tud + i - 1) + field[k];
        constexpr int ld = sizeof(TabUD) / 8;
        interval_cubic(T[0], T[ld], T[2 * ld], T[3 * ld], c);
    }
    for (int m = 0; m < 4; ++m) out[i].c[k][m] = c[m];
}
__global__ void pg_poly_kernel(const double* __restrict__ raw, PgPoly* __restrict__ out, int n, int nt)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / (3 * n), f = (t - 3 * n * i) / 3, m = t % 3;
    if (i >= nt) return;
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    const double* T = raw + ((size_t)m * n + f) * nt + i - 1;
    if (i >= 1 && i + 2 < nt) interval_cubic(T[0], T[1], T[2], T[3], c);
    for (int q = 0; q < 4; ++q) out[(size_t)i * n + f].c[m][q] = c[q];
}

cudaError_t launch_tab_poly(const TabUD* tud, TabPoly* out, int nt, cudaStream_t st)
{
    static_assert(sizeof(TabUD) == 64, "fields by number");
    tab_poly_kernel<<<(7 * nt + 255) / 256, 256, 0, st>>>(tud, out, nt);
    return cudaGetLastError();
}
cudaError_t launch_pg_poly(const double* raw, PgPoly* out, int n, int nt, cudaStream_t st)
{
    pg_poly_kernel<<<(3 * n * nt + 255) / 256, 256, 0, st>>>(raw, out, n, nt);
    return cudaGetLastError();
}

cudaError_t launch_bcsone(const DevParams& p, const KVecDev* kv, const TabUD* tud, const PhiFix* phi,
                          const TabPoly* tpoly, bool sym, const double* x, const double* inv, const int* ipart,
                          const double* dr, double* ratio, int nw, cudaStream_t st)
{
    if (nw <= 0) return cudaSuccess;
    if (sym) {
        bcsone_sym_kernel<<<nw, kMoveThreads, 0, st>>>(p, phi, tpoly, x, inv, ipart, dr, ratio);
        return cudaGetLastError();
    }
    const int warps = 8;
    bcsone_kernel<<<(nw + warps - 1) / warps, 32 * warps, 0, st>>>(p, kv, tud, x, inv, ipart, dr, ratio, nw);
    return cudaGetLastError();
}

cudaError_t launch_getphione(const DevParams& p, const TabPoly* tpoly, const TabUD* tud, const TabSS* tss,
                             const double* x, const int* ipart, const double* drr, double* ratio, int nw,
                             cudaStream_t st)
{
    if (nw <= 0) return cudaSuccess;
    getphione_kernel<<<nw, kMoveThreads, 0, st>>>(p, tpoly, tud, tss, x, ipart, drr, ratio);
    return cudaGetLastError();
}

static AttrCache g_attr;
enum : int { kAttrDerbcs = 0, kAttrPgrad = 1 };   // pgrad: + 1 in the symmetric form

size_t derbcs_smem_bytes(const DevParams& p)
{
    return sizeof(double) * ((size_t)p.nd * p.nd + 3 * p.npart + 2 * kChunk * p.ndn + (size_t)kChunk * p.nup +
                             p.norb + kThreads);
}

cudaError_t launch_derbcs(const DevParams& p, const KVecDev* kv, const double* x, const double* smati, double* dpsi,
                          int nw, int grid, cudaStream_t st, int stride, int off, bool sym)
{
    if (nw <= 0) return cudaSuccess;
    if (sym) {
        // 1.19 -> 0.07 ms for 2048 walkers at N = 66
        derbcs_sym_kernel<<<nw, kThreads, 0, st>>>(p, x, smati, dpsi, nw, stride < 0 ? p.norb : stride, off);
        return cudaGetLastError();
    }
    const size_t smem = derbcs_smem_bytes(p);
    cudaError_t e = allow_smem(g_attr, kAttrDerbcs, derbcs_kernel, smem);
    if (e != cudaSuccess) return e;
    derbcs_kernel<<<grid < nw ? grid : nw, kThreads, smem, st>>>(p, kv, x, smati, dpsi, nw, stride < 0 ? p.norb : stride,
                                                                 off);
    return cudaGetLastError();
}

// Layout of one pgrad CTA's core, in doubles: inverse, M, product buffer
// (nd^2 each), positions, grad J / m and grad log Psi / m (3 npart each),
// reduction buffer, results, amplitudes and first k of each shell, flags,
// box fractions and axis cos/sin.
size_t pgrad_doubles(const DevParams& p)
{
    const size_t nd2 = (size_t)p.nd * p.nd;
    return 3 * nd2 + 18 * (size_t)p.npart + kThreads + 2 * (size_t)kPgradMax + (size_t)p.norb +
           (size_t)(p.norb + 2 + p.npart) / 2;
}

// The CTA's global slice, in doubles (even): (S', M') of every up-down pair
// for the shells and beta's three parameters; without the symmetric form also
// axis powers (3 npart (nmax+1) complex) and plane waves (npart (nk-1) complex).
size_t pgrad_slice_doubles(const DevParams& p, bool sym)
{
    const size_t nq = p.nk > 1 ? (size_t)p.nk - 1 : 1, nsp = (size_t)p.norb - 1 + (p.nobeta ? 0 : 3);
    const size_t waves = sym ? 0 : 3 * (size_t)p.npart * (p.nmax + 1) + (size_t)p.npart * nq;
    return 2 * (nsp * p.nup * p.ndn + waves + 1);
}

// CTAs of one pgrad launch: as many as are resident on the device's SMs
// together, at most one per walker.
int pgrad_grid(const DevParams& p, int nw, int nsm, int smem_limit, bool sym)
{
    const auto kern = sym ? pgrad_kernel<true> : pgrad_kernel<false>;
    const size_t need = pgrad_doubles(p) * 8;
    const int smem = need <= (size_t)smem_limit ? (int)need : 0;
    int per_sm = 1;
    if (smem > 0 && allow_smem(g_attr, kAttrPgrad + (sym ? 1 : 0), kern, smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem) != cudaSuccess) return 0;
    const long long g = (long long)(per_sm > 0 ? per_sm : 1) * nsm;
    return (int)(g < nw ? g : (nw > 0 ? nw : 1));
}

cudaError_t launch_pgrad(const DevParams& p, const KVecDev* kv, const TabPoly* tpoly, const double* x,
                         const double* sinv, const double* dpsi, const double* dphi, double* dlog, double* deloc, int nw,
                         int np, double bfact, const PgPoly* btd, const PgPoly* ktd, int nbeta, int nknot, bool sym,
                         int grid, double* gscr, double* slices, int smem_limit, cudaStream_t st)
{
    if (np > kPgradMax || nknot > kJastrowKnots || np != p.norb + nbeta + nknot || (nbeta > 1 && !btd) ||
        (nknot > 0 && !ktd) || !slices || grid < 1)
        return cudaErrorInvalidValue;
    if (nw <= 0) return cudaSuccess;
    const auto kern = sym ? pgrad_kernel<true> : pgrad_kernel<false>;
    const size_t need = pgrad_doubles(p);
    const bool on_chip = need * 8 <= (size_t)smem_limit;
    const size_t smem = on_chip ? need * 8 : 0;
    if (on_chip) {
        cudaError_t e = allow_smem(g_attr, kAttrPgrad + (sym ? 1 : 0), kern, smem);
        if (e != cudaSuccess) return e;
    } else if (!gscr) {
        return cudaErrorInvalidValue;
    }
    kern<<<grid < nw ? grid : nw, kThreads, smem, st>>>(p, kv, tpoly, x, sinv, dpsi, dphi, dlog, deloc, nw, np, bfact,
                                                        btd, ktd, nbeta, nknot, on_chip ? nullptr : gscr, need, slices,
                                                        pgrad_slice_doubles(p, sym));
    return cudaGetLastError();
}

cudaError_t launch_jasder(const DevParams& p, const double* jq, const double* x, double* dpsi, int nw, int grid,
                          cudaStream_t st, int stride)
{
    if (nw <= 0) return cudaSuccess;
    const size_t smem = sizeof(double) * (size_t)(p.nql > 0 ? p.nql : 1);
    jasder_kernel<<<grid < nw ? grid : nw, kThreads, smem, st>>>(p, jq, x, dpsi, nw, stride);
    return cudaGetLastError();
}

cudaError_t launch_sr_sums(const double* der, const double* d2psi, const double* v, int n, int np, double hbar,
                           double eunit, int npart, double* sums, double* ene, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    sr_energy_kernel<<<(n + 255) / 256, 256, 0, st>>>(d2psi, v, n, hbar, eunit, (double)npart, ene);
    const int nout = np * np + 2 * np + 2;
    sr_sums_kernel<<<(nout + kSrOut - 1) / kSrOut, 128, 0, st>>>(der, ene, n, np, sums);
    return cudaGetLastError();
}

}  // namespace dmc
