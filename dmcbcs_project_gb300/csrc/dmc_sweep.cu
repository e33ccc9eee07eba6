// Particle-by-particle Metropolis sweeps with Sherman-Morrison updates of the
// inverse pair matrix, in FP32 (sm_103a).
//
// No counterpart in the reference's walker loop, whose moves are
// all-particle (step.f90:43-285); the single-particle ratio it builds on is
// bcsone / getphione / move1 (psislaterbcs.f90:296-376, coshpot.f90:207-264,
// wavefunction.f90:393-404), which the reference uses only for n(k).
//
// Four warps, two or one per walker (launch_sweeps).  Per move of particle i (in
// order 0..npart-1, every sweep):
//   - five draws of the walker's ran1 stream (ran.f90:8-27): three Gaussian
//     deviates (gaussian(3), ran.f90:74-104) and one uniform, and the
//     proposal x_i' = x_i + sigma_i g (sigma of setstep, step.f90:29-30)
//     wrapped into the box, all in FP64 for the whole sweep ahead of its
//     moves, one move per thread (particle i has not moved before its own move
//     of the sweep);
//   - distances in FP32;
//   - the new row (up particle) or column (down particle) s' of the pair
//     matrix: phi(r_i' - r_j) = v_0 + sum_q 2 vorb(shell q) cos(k_q.(r_i'-r_j))
//     + beta(|r_i' - r_j|), and the unpaired plane waves at r_i', from a
//     cos/sin table of every k vector at every particle;
//   - determinant ratio R = s'.X(:,i) (row) or X(c,:).s' (column) and the
//     Jastrow ratio exp(U' - U) from the pair tables;
//   - accept when u < R^2 exp(2 (U' - U)); on acceptance the inverse X is
//     updated by Sherman-Morrison (rank one, FP32) and the table column of
//     particle i is replaced.
// The inverse X enters in FP64 (a fresh inverse of the pair matrix from the
// FP64 walker kernel: the periodic full recompute) or as the FP32 inverse
// carried from the previous call; it leaves in FP32.
#include <cuda_runtime.h>
#include <math.h>

#include "dmc_device.cuh"
#include "dmc_kernels.h"
#include "dmc_smem.cuh"
#include "dmc_walker.cuh"

namespace dmc {
namespace {

// Threads per walker.  Bound: the latency of a move's chain of stages, one move
// after another.  A warp per walker took 24k cycles a move at N = 66: every
// loop over 33 entries or 40 k vectors had a second, nearly empty round and the
// table's loads were exposed.  Here an entry has two threads (the chains over
// the even and over the odd k vectors, two of its four partial sums), the last
// warp takes the Jastrow beside them and the rank-one update all of them; every
// sum keeps its order and rounding.  One sweep of 1024 walkers at N = 66:
// 822 -> 274 us.

// floats of a walker's shared memory: FP32 positions for the distances (3
// npart), X (nd x ldx), the new entries s' and the v / w vector (nd each),
// the moved particle's orbitals (v-scaled and plain, 2 (nk-1) float2), the
// Jastrow difference (two slots).  The FP64 positions stay in the walker stack
// and the sweep's proposals in a global slice per walker.
__host__ __device__ inline int sweep_floats(const DevParams& p)
{
    const int ldx = p.nd | 1;
    const int nq = p.nk > 1 ? p.nk - 1 : 1;
    return 3 * p.npart + 2 + p.nd * ldx + 2 * p.nd + 8 * nq + 8;
}
// the same in whole float2, with the cos/sin table where it is on chip
__host__ __device__ inline int walker_floats(const DevParams& p, bool onchip)
{
    return (sweep_floats(p) + 1) / 2 * 2 + (onchip ? 2 * (p.nk > 1 ? p.nk - 1 : 1) * p.npart : 0);
}

// FP32 4-point Lagrange grid position (index clamp of coshpot.f90:174)
__device__ __forceinline__ walker::Lagrange<float> lag_f(float r, float scale, int ntab)
{
    const float t = r * scale;
    int idx = (int)t;
    idx = max(1, min(idx, ntab - 2));
    return walker::lagrange_f(t - (float)idx, idx);
}

// u(r) of an up-down (or, with ss, a same-spin) pair, FP32; zero beyond L/2
__device__ __forceinline__ float jas_u(const DevParams& p, const TabUDmp* tud, const TabSSmp* tss, bool opposite,
                                       float r)
{
    if (!(r < (float)p.range)) return 0.0f;
    const walker::Lagrange<float> W = lag_f(r, (float)p.scale, p.ntab);
    if (opposite) {
        const TabUDmp* T = tud + (W.idx - 1);
        return W.c1 * T[0].u.hi + W.c2 * T[1].u.hi + W.c3 * T[2].u.hi + W.c4 * T[3].u.hi;
    }
    const TabSSmp* T = tss + (W.idx - 1);
    return W.c1 * T[0].u + W.c2 * T[1].u + W.c3 * T[2].u + W.c4 * T[3].u;
}

// beta(r) (radialfun, betafun.f90:173-194), FP32
__device__ __forceinline__ float beta_f(const DevParams& p, const TabUDmp* tud, float r)
{
    if (p.nobeta || r > (float)p.rangeb) return 0.0f;
    const walker::Lagrange<float> W = lag_f(r, (float)p.scaleb, p.ntab);
    const TabUDmp* T = tud + (W.idx - 1);
    return W.c1 * T[0].b.hi + W.c2 * T[1].b.hi + W.c3 * T[2].b.hi + W.c4 * T[3].b.hi;
}

__device__ __forceinline__ float warp_sum_f(float v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double ran1_step(unsigned long long& s)
{
    s = (44485709377909ull * s + 96309754297ull) & walker::kMask48;
    return walker::lcg_uniform(s);
}

// FP32 minimum image
__device__ __forceinline__ float min_image_f(float d, float el, float eli) { return d - el * rintf(d * eli); }

// barrier of the threads that form the new entries
template <int W>
__device__ __forceinline__ void row_sync()
{
    if constexpr (W == 2)
        __syncwarp();
    else
        asm volatile("bar.sync 1, %0;" ::"n"(32 * (W - 1)) : "memory");
}

// A CTA of W warps per walker.  ONCHIP: the cos/sin table in shared memory,
// otherwise in tab.  (Registers for 128 threads: with those for 64, two warps
// took 5 % longer.)
template <int W, bool ONCHIP>
__global__ void __launch_bounds__(128) sweep_kernel(const __grid_constant__ DevParams p, DevStack st,
                                                              int nsweep, const double* __restrict__ inv64,
                                                              float* __restrict__ inv32, float2* __restrict__ tab,
                                                              const KVecMP* __restrict__ kv,
                                                              const TabUDmp* __restrict__ tud,
                                                              const TabSSmp* __restrict__ tss,
                                                              const unsigned long long* __restrict__ jA,
                                                              const unsigned long long* __restrict__ jC,
                                                              unsigned long long* __restrict__ accepted,
                                                              double* __restrict__ prop)
{
    extern __shared__ __align__(16) float smw[];
    constexpr int NT = 32 * W, NR = NT - 32;   // all threads; those for the new entries
    const int tid = threadIdx.x, lane = tid & 31;
    const int P = p.npart, nd = p.nd, ldx = nd | 1, nq = p.nk - 1, nup = p.nup;
    float* xsf = smw;
    float* X = xsf + 3 * P + (P & 1);                  // X(r, c) = X[r + c ldx]: column-major as smati
    float* snew = X + nd * ldx;
    float* vw = snew + nd;
    float2* onew = reinterpret_cast<float2*>(vw + nd + (((nd * ldx + 2 * nd) & 1) ? 1 : 0));   // v-scaled
    float2* oraw = onew + (nq > 0 ? nq : 1);                                                 // plain
    float* s_du = reinterpret_cast<float*>(oraw + (nq > 0 ? nq : 1));                        // by the move's parity
    const float v0 = kv[0].v.hi;
    const float elf = (float)p.el, elif = (float)p.eli;
    const int w = blockIdx.x;
    double* xs = st.x + (size_t)w * 3 * P;     // FP64 positions, wrapped in place
    double* drw = prop + (size_t)w * 4 * P;    // [P][4]: the proposal x_i + sigma g and u of move i
    // ---- load the walker: positions (wrapped), inverse, cos/sin table ----
    for (int e = tid; e < 3 * P; e += NT) {
        const double xv = walker::min_image(xs[e], p);
        xs[e] = xv;
        xsf[e] = (float)xv;
    }
    for (int e = tid; e < nd * nd; e += NT) {
        const int r = e % nd, c = e / nd;
        X[r + c * ldx] = inv64 ? (float)inv64[(size_t)w * nd * nd + e] : inv32[(size_t)w * nd * nd + e];
    }
    // T[q P + j] = (cos, sin)(k_{q+1} . x_j)
    float2* T = ONCHIP ? reinterpret_cast<float2*>(xsf + walker_floats(p, false)) : tab + (size_t)w * nq * P;
    __syncthreads();
    for (int e = tid; e < nq * P; e += NT) {
        const int q = e / P, j = e % P;
        const KVecMP& K = kv[q + 1];
        float sn, cs;
        sincosf(K.k[0].hi * (float)xs[3 * j] + K.k[1].hi * (float)xs[3 * j + 1] + K.k[2].hi * (float)xs[3 * j + 2],
                &sn, &cs);
        T[e] = make_float2(cs, sn);
    }
    unsigned long long s = st.irn[w] & walker::kMask48;
    unsigned long long nacc = 0;
    const walker::UDiv dv(nd);
    for (int sw = 0; sw < nsweep; ++sw) {
        // the sweep's draws, one move per thread: move i takes ran1 draws
        // 5i+1 .. 5i+5 of the stream -- gaussian(3) from four uniforms, then
        // the acceptance uniform -- reached by jump-ahead.  Particle i moves
        // only at its own move, so its proposal x_i + sigma g is fixed by the
        // sweep's start and is made here too: the moves themselves do no FP64
        // arithmetic
        for (int i = tid; i < P; i += NT) {
            unsigned long long t = (jA[5 * i] * s + jC[5 * i]) & walker::kMask48;
            const double u1 = ran1_step(t), u2 = ran1_step(t), u3 = ran1_step(t), u4 = ran1_step(t);
            const double rn = ran1_step(t);
            double sn, cs;
            sincospi(2.0 * u1, &sn, &cs);
            const double r12 = sqrt(-2.0 * log(u2));
            const double g[3] = {sn * r12, cs * r12, cospi(2.0 * u3) * sqrt(-2.0 * log(u4))};
            const double sig = p.sigma[i < nup ? 0 : 1];
            for (int c = 0; c < 3; ++c) drw[4 * i + c] = walker::min_image(xs[3 * i + c] + sig * g[c], p);
            drw[4 * i + 3] = rn;
        }
        s = (jA[5 * P] * s + jC[5 * P]) & walker::kMask48;
        __syncthreads();
        // lanes 0-3 of each warp hold move i's proposal and uniform, read one move ahead
        double pv = lane < 4 ? drw[lane] : 0.0;
        for (int i = 0; i < P; ++i) {
            const bool up = i < nup;
            const double xn[3] = {__shfl_sync(0xffffffffu, pv, 0), __shfl_sync(0xffffffffu, pv, 1),
                                  __shfl_sync(0xffffffffu, pv, 2)};   // the proposal, FP64
            const double rn = __shfl_sync(0xffffffffu, pv, 3);
            const double pcur = pv;
            if (lane < 4 && i + 1 < P) pv = drw[4 * (i + 1) + lane];
            const float xf[3] = {(float)xn[0], (float)xn[1], (float)xn[2]};
            if (tid < NR) {
                // the moved particle's plane waves
                for (int q = tid; q < nq; q += NR) {
                    const KVecMP& K = kv[q + 1];
                    float sn, cs;
                    sincosf(K.k[0].hi * xf[0] + K.k[1].hi * xf[1] + K.k[2].hi * xf[2], &sn, &cs);
                    oraw[q] = make_float2(cs, sn);
                    const float vq = K.v.hi;
                    onew[q] = make_float2(vq * cs, vq * sn);
                }
                row_sync<W>();
                // the new row (up) or column (down) of the pair matrix: two
                // threads per entry, the chain over the even and the one over
                // the odd k vectors
                const int nloop = up ? p.npair + p.nexdn : p.npair + p.nexup;
                for (int t0 = 0; t0 < 2 * nd; t0 += NR) {
                    const int e = (t0 + tid) >> 1, h = tid & 1;
                    float acc = h == 0 ? v0 : 0.0f, rest = 0.0f;
                    if (e < nloop && e < nd) {
                        const int jj = up ? e + p.npair + p.nexup : e;
                        float d2 = 0.0f;
                        for (int c = 0; c < 3; ++c) {
                            const float d = min_image_f(xf[c] - xsf[3 * jj + c], elf, elif);
                            d2 = fmaf(d, d, d2);
                        }
                        rest = beta_f(p, tud, sqrtf(d2));
#pragma unroll 10
                        for (int q = h; q < nq; q += 2) {
                            const float2 a = onew[q], b = T[q * P + jj];
                            acc = fmaf(a.x, b.x, fmaf(a.y, b.y, acc));
                        }
                    } else if (e < nd) {
                        const int u = e - nloop;
                        const double* a = up ? p.akup[u] : p.akdn[u];
                        const int sn = up ? p.sinup[u] : p.sindn[u];
                        const float arg = (float)a[0] * xf[0] + (float)a[1] * xf[1] + (float)a[2] * xf[2];
                        rest = sn ? sinf(arg) : cosf(arg);
                    }
                    const float odd = __shfl_xor_sync(0xffffffffu, acc, 1);
                    if (h == 0 && e < nd) snew[e] = e < nloop ? (acc + odd) + rest : rest;
                }
            } else {
                // Jastrow: U(r_i') - U(r_i) over the pairs getphione counts.  A
                // lane takes its partners j = lane + 32 u kJasLanes at a time, all
                // their table lookups in flight before any is used; the
                // differences are added in partner order (skipped pairs add 0).
                constexpr int kJasLanes = 3;
                float du = 0.0f;
                for (int j0 = lane; j0 < P; j0 += 32 * kJasLanes) {
                    float dj[kJasLanes];
#pragma unroll
                    for (int u = 0; u < kJasLanes; ++u) {
                        const int j = j0 + 32 * u;
                        dj[u] = 0.0f;
                        const bool opp = up != (j < nup);
                        if (j < P && j != i && (opp || p.ieq)) {
                            float dn = 0.0f, dold = 0.0f;
                            for (int c = 0; c < 3; ++c) {
                                const float a = min_image_f(xf[c] - xsf[3 * j + c], elf, elif);
                                const float b = min_image_f(xsf[3 * i + c] - xsf[3 * j + c], elf, elif);
                                dn = fmaf(a, a, dn);
                                dold = fmaf(b, b, dold);
                            }
                            dj[u] = jas_u(p, tud, tss, opp, fmaxf(sqrtf(dn), 1.0e-14f)) -
                                    jas_u(p, tud, tss, opp, fmaxf(sqrtf(dold), 1.0e-14f));
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kJasLanes; ++u)
                        if (j0 + 32 * u < P) du += dj[u];
                }
                du = warp_sum_f(du);
                if (lane == 0) s_du[i & 1] = du;
            }
            __syncthreads();
            // v_k = sum_q s'_q X(q, k) (row i replaced) or w_k = sum_q X(k, q) s'_q
            // (column c replaced); the ratio is v_i or w_c.  Four partial sums
            // an entry, two on each of its two threads.
            const int cix = up ? i : i - nup;
            const int rs = up ? 1 : ldx, cs = up ? ldx : 1;   // X(q, k) or X(k, q)
            for (int t0 = 0; t0 < 2 * nd; t0 += NT) {
                const int k = (t0 + tid) >> 1, h = tid & 1;
                float a = 0.0f, b = 0.0f;
                if (k < nd) {
                    const float* xb = X + k * cs;
                    int q = 2 * h;
#pragma unroll 4
                    for (; q - 2 * h + 3 < nd; q += 4) {
                        a = fmaf(snew[q], xb[q * rs], a);
                        b = fmaf(snew[q + 1], xb[(q + 1) * rs], b);
                    }
                    if (h == 0)
                        for (; q < nd; ++q) a = fmaf(snew[q], xb[q * rs], a);
                }
                a += b;
                const float other = __shfl_xor_sync(0xffffffffu, a, 1);
                if (h == 0 && k < nd) vw[k] = a + other;
            }
            __syncthreads();
            const float R = vw[cix];
            const float prob = R * R * expf(2.0f * s_du[i & 1]);
            const bool acc = rn < (double)prob;   // R = 0 or NaN: rejected
            if (acc) {
                const float iR = 1.0f / R;
                // Sherman-Morrison (rank one): every column (row) but cix first
                for (int e = tid; e < nd * nd; e += NT) {
                    const int c = dv.quo(e), r = e - c * nd;
                    const int k = up ? c : r;
                    if (k == cix) continue;
                    const float f = vw[k] * iR;
                    float* x = X + r + c * ldx;
                    *x = fmaf(-(up ? X[r + cix * ldx] : X[cix + c * ldx]), f, *x);
                }
                __syncthreads();
                for (int q = tid; q < nd; q += NT) X[up ? q + cix * ldx : cix + q * ldx] *= iR;
                for (int q = tid; q < nq; q += NT) T[q * P + i] = oraw[q];
                if (tid < 3) {
                    xs[3 * i + tid] = pcur;
                    xsf[3 * i + tid] = (float)pcur;
                }
                ++nacc;
                __syncthreads();
            }
        }
    }
    // ---- write back (the positions are already in the stack) ----
    __syncthreads();
    for (int e = tid; e < nd * nd; e += NT) {
        const int r = e % nd, c = e / nd;
        inv32[(size_t)w * nd * nd + e] = X[r + c * ldx];
    }
    if (tid == 0) {
        st.irn[w] = s;
        accepted[w] += nacc;
    }
}

// One warp per walker, four walkers a CTA (fewer where they do not fit), the
// table in global memory: the same sums in the same order.  A move takes it two
// to three times as long as four warps, but 36 walkers are on an SM at once; it is
// the faster where the other form would go round several times (launch_sweeps).
__global__ void __launch_bounds__(128) sweep_warp_kernel(const __grid_constant__ DevParams p, DevStack st, int n,
                                                         int nsweep, const double* __restrict__ inv64,
                                                         float* __restrict__ inv32, float2* __restrict__ tab,
                                                         const KVecMP* __restrict__ kv,
                                                         const TabUDmp* __restrict__ tud,
                                                         const TabSSmp* __restrict__ tss,
                                                         const unsigned long long* __restrict__ jA,
                                                         const unsigned long long* __restrict__ jC,
                                                         unsigned long long* __restrict__ accepted,
                                                         double* __restrict__ prop)
{
    extern __shared__ __align__(16) float smw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int P = p.npart, nd = p.nd, ldx = nd | 1, nq = p.nk - 1, nup = p.nup;
    float* xsf = smw + wib * walker_floats(p, false);
    float* X = xsf + 3 * P + (P & 1);                  // X(r, c) = X[r + c ldx]: column-major as smati
    float* snew = X + nd * ldx;
    float* vw = snew + nd;
    float2* onew = reinterpret_cast<float2*>(vw + nd + (((nd * ldx + 2 * nd) & 1) ? 1 : 0));   // v-scaled
    float2* oraw = onew + (nq > 0 ? nq : 1);                                                 // plain
    const float v0 = kv[0].v.hi;
    const float elf = (float)p.el, elif = (float)p.eli;
    const int w = blockIdx.x * (blockDim.x >> 5) + wib;
    if (w >= n) return;   // whole warps only: the warp is the unit below
    double* xs = st.x + (size_t)w * 3 * P;     // FP64 positions, wrapped in place
    double* drw = prop + (size_t)w * 4 * P;    // [P][4]: the proposal x_i + sigma g and u of move i
    // ---- load the walker: positions (wrapped), inverse, cos/sin table ----
    for (int e = lane; e < 3 * P; e += 32) {
        const double xv = walker::min_image(xs[e], p);
        xs[e] = xv;
        xsf[e] = (float)xv;
    }
    if (inv64) {
        for (int e = lane; e < nd * nd; e += 32) {
            const int r = e % nd, c = e / nd;
            X[r + c * ldx] = (float)inv64[(size_t)w * nd * nd + e];
        }
    } else {
        for (int e = lane; e < nd * nd; e += 32) {
            const int r = e % nd, c = e / nd;
            X[r + c * ldx] = inv32[(size_t)w * nd * nd + e];
        }
    }
    float2* T = tab + (size_t)w * nq * P;   // T[q P + j] = (cos, sin)(k_{q+1} . x_j)
    __syncwarp();
    for (int e = lane; e < nq * P; e += 32) {
        const int q = e / P, j = e % P;
        const KVecMP& K = kv[q + 1];
        float sn, cs;
        sincosf(K.k[0].hi * (float)xs[3 * j] + K.k[1].hi * (float)xs[3 * j + 1] + K.k[2].hi * (float)xs[3 * j + 2],
                &sn, &cs);
        T[e] = make_float2(cs, sn);
    }
    unsigned long long s = st.irn[w] & walker::kMask48;
    unsigned long long nacc = 0;
    __syncwarp();
    for (int sw = 0; sw < nsweep; ++sw) {
        // the sweep's draws, one move per lane
        for (int i = lane; i < P; i += 32) {
            unsigned long long t = (jA[5 * i] * s + jC[5 * i]) & walker::kMask48;
            const double u1 = ran1_step(t), u2 = ran1_step(t), u3 = ran1_step(t), u4 = ran1_step(t);
            const double rn = ran1_step(t);
            double sn, cs;
            sincospi(2.0 * u1, &sn, &cs);
            const double r12 = sqrt(-2.0 * log(u2));
            const double g[3] = {sn * r12, cs * r12, cospi(2.0 * u3) * sqrt(-2.0 * log(u4))};
            const double sig = p.sigma[i < nup ? 0 : 1];
            for (int c = 0; c < 3; ++c) drw[4 * i + c] = walker::min_image(xs[3 * i + c] + sig * g[c], p);
            drw[4 * i + 3] = rn;
        }
        s = (jA[5 * P] * s + jC[5 * P]) & walker::kMask48;
        __syncwarp();
        // lanes 0-3 hold move i's proposal and uniform, read one move ahead
        double pv = lane < 4 ? drw[lane] : 0.0;
        for (int i = 0; i < P; ++i) {
            const bool up = i < nup;
            const double xn[3] = {__shfl_sync(0xffffffffu, pv, 0), __shfl_sync(0xffffffffu, pv, 1),
                                  __shfl_sync(0xffffffffu, pv, 2)};   // the proposal, FP64
            const double rn = __shfl_sync(0xffffffffu, pv, 3);
            const double pcur = pv;
            if (lane < 4 && i + 1 < P) pv = drw[4 * (i + 1) + lane];
            const float xf[3] = {(float)xn[0], (float)xn[1], (float)xn[2]};
            // the moved particle's plane waves
            for (int q = lane; q < nq; q += 32) {
                const KVecMP& K = kv[q + 1];
                float sn, cs;
                sincosf(K.k[0].hi * xf[0] + K.k[1].hi * xf[1] + K.k[2].hi * xf[2], &sn, &cs);
                oraw[q] = make_float2(cs, sn);
                const float vq = K.v.hi;
                onew[q] = make_float2(vq * cs, vq * sn);
            }
            __syncwarp();
            // the new row (up) or column (down) of the pair matrix
            const int nloop = up ? p.npair + p.nexdn : p.npair + p.nexup;
            for (int e = lane; e < nd; e += 32) {
                float ph;
                if (e < nloop) {
                    const int jj = up ? e + p.npair + p.nexup : e;
                    // two chains, loads unrolled ahead of the multiply-adds
                    float acc = v0, acc2 = 0.0f;
                    int q = 0;
#pragma unroll 4
                    for (; q + 1 < nq; q += 2) {
                        const float2 a = onew[q], b = T[q * P + jj];
                        const float2 a2 = onew[q + 1], b2 = T[(q + 1) * P + jj];
                        acc = fmaf(a.x, b.x, fmaf(a.y, b.y, acc));
                        acc2 = fmaf(a2.x, b2.x, fmaf(a2.y, b2.y, acc2));
                    }
                    if (q < nq) {
                        const float2 a = onew[q], b = T[q * P + jj];
                        acc = fmaf(a.x, b.x, fmaf(a.y, b.y, acc));
                    }
                    acc += acc2;
                    float d2 = 0.0f;
                    for (int c = 0; c < 3; ++c) {
                        const float d = min_image_f(xf[c] - xsf[3 * jj + c], elf, elif);
                        d2 = fmaf(d, d, d2);
                    }
                    ph = acc + beta_f(p, tud, sqrtf(d2));
                } else {
                    const int u = e - nloop;
                    const double* a = up ? p.akup[u] : p.akdn[u];
                    const int sn = up ? p.sinup[u] : p.sindn[u];
                    const float arg = (float)a[0] * xf[0] + (float)a[1] * xf[1] + (float)a[2] * xf[2];
                    ph = sn ? sinf(arg) : cosf(arg);
                }
                snew[e] = ph;
            }
            __syncwarp();
            // v_k = sum_q s'_q X(q, k) (row i replaced) or w_k = sum_q X(k, q) s'_q
            // (column c replaced); the ratio is v_i or w_c
            const int cix = up ? i : i - nup;
            for (int k = lane; k < nd; k += 32) {
                // four partial sums: the chain is shared-memory latency bound
                float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                const int rs = up ? 1 : ldx, cs = up ? ldx : 1;   // X(q, k) or X(k, q)
                const float* xb = X + k * cs;
                int q = 0;
                for (; q + 3 < nd; q += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) a[u] = fmaf(snew[q + u], xb[(q + u) * rs], a[u]);
                }
                for (; q < nd; ++q) a[0] = fmaf(snew[q], xb[q * rs], a[0]);
                vw[k] = (a[0] + a[1]) + (a[2] + a[3]);
            }
            // Jastrow
            constexpr int kJasLanes = 3;
            float du = 0.0f;
            for (int j0 = lane; j0 < P; j0 += 32 * kJasLanes) {
                float dj[kJasLanes];
#pragma unroll
                for (int u = 0; u < kJasLanes; ++u) {
                    const int j = j0 + 32 * u;
                    dj[u] = 0.0f;
                    const bool opp = up != (j < nup);
                    if (j < P && j != i && (opp || p.ieq)) {
                        float dn = 0.0f, dold = 0.0f;
                        for (int c = 0; c < 3; ++c) {
                            const float a = min_image_f(xf[c] - xsf[3 * j + c], elf, elif);
                            const float b = min_image_f(xsf[3 * i + c] - xsf[3 * j + c], elf, elif);
                            dn = fmaf(a, a, dn);
                            dold = fmaf(b, b, dold);
                        }
                        dj[u] = jas_u(p, tud, tss, opp, fmaxf(sqrtf(dn), 1.0e-14f)) -
                                jas_u(p, tud, tss, opp, fmaxf(sqrtf(dold), 1.0e-14f));
                    }
                }
#pragma unroll
                for (int u = 0; u < kJasLanes; ++u)
                    if (j0 + 32 * u < P) du += dj[u];
            }
            du = warp_sum_f(du);
            __syncwarp();
            const float R = vw[cix];
            const float prob = R * R * expf(2.0f * du);
            const bool acc = rn < (double)prob;   // R = 0 or NaN: rejected
            if (acc) {
                const float iR = 1.0f / R;
                // Sherman-Morrison (rank one): every column (row) but cix first
                if (up) {
                    for (int k = lane; k < nd; k += 32) {
                        if (k == cix) continue;
                        const float f = vw[k] * iR;
                        for (int q = 0; q < nd; ++q) X[q + k * ldx] = fmaf(-X[q + cix * ldx], f, X[q + k * ldx]);
                    }
                    __syncwarp();
                    for (int q = lane; q < nd; q += 32) X[q + cix * ldx] *= iR;
                } else {
                    for (int k = lane; k < nd; k += 32) {
                        if (k == cix) continue;
                        const float f = vw[k] * iR;
                        for (int q = 0; q < nd; ++q) X[k + q * ldx] = fmaf(-X[cix + q * ldx], f, X[k + q * ldx]);
                    }
                    __syncwarp();
                    for (int q = lane; q < nd; q += 32) X[cix + q * ldx] *= iR;
                }
                for (int q = lane; q < nq; q += 32) T[q * P + i] = oraw[q];
                if (lane < 3) {
                    xs[3 * i + lane] = pcur;
                    xsf[3 * i + lane] = (float)pcur;
                }
                ++nacc;
            }
            __syncwarp();
        }
    }
    // ---- write back (the positions are already in the stack) ----
    for (int e = lane; e < nd * nd; e += 32) {
        const int r = e % nd, c = e / nd;
        inv32[(size_t)w * nd * nd + e] = X[r + c * ldx];
    }
    if (lane == 0) {
        st.irn[w] = s;
        accepted[w] += nacc;
    }
}

AttrCache g_attr;   // shared-memory limit and carveout of each variant

}  // namespace

cudaError_t launch_sweeps(const DevParams& p, const DevStack& st, int n, int nsweep, const double* inv64,
                          float* inv32, float2* tab, const KVecMP* kv, const TabUDmp* tud, const TabSSmp* tss,
                          const unsigned long long* jA, const unsigned long long* jC, unsigned long long* accepted,
                          double* prop, cudaStream_t stream)
{
    if (n <= 0 || nsweep <= 0) return cudaSuccess;
    if (!prop) return cudaErrorInvalidValue;
    int dev = 0, optin = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // Four warps with the table on chip are the fastest while every walker is
    // resident.  Beyond that the rounds count: two warps (1.0 to 1.7 of the
    // time of a round) let twice as many small walkers in, the table in global
    // memory (1.25 to 1.6, more with more k vectors) more of the large ones, and
    // one warp a walker four times as many.  Its round is the longer the more k
    // vectors its one thread per entry sums, and the shorter against the others'
    // the better the entries fill its lanes; beyond 32 of them it takes two turns
    // and does not pay, nor where its walkers' tables do not stay in L2 (19/19 at
    // twelve shells, 4096 walkers, 111 MB: 837, four warps 555).  us per sweep,
    // four on chip / two on chip / four with a global table / one warp:
    //   5/5   2700:  89 / 62 / 82 / 58         4096: 120 / 71 / 123 / 66
    //   19/19 1024: 124 / 153 / 174 / 323      4096: 458 / 374 / 537 / 372
    //   26/26 2000: 355 / 449 / 490 / 452      4096: 693 / 711 / 786 / 564
    //   33/33 1024: 275 / 395 / 337 / 826      4096: 1019 / 1505 / 1117 / 1068
    //   66/66  256: 798 / 1322 / 1027 / 2607   1024: 2481 / 3981 / 1350 / 2685
    const int nq = p.nk > 1 ? p.nk - 1 : 1;
    struct Variant {
        decltype(&sweep_kernel<4, true>) kern;
        int warps;
        bool onchip;
        double round;
    };
    const Variant variants[3] = {{sweep_kernel<4, true>, 4, true, 1.0},
                                 {sweep_kernel<2, true>, 2, true, 1.3},
                                 {sweep_kernel<4, false>, 4, false, 1.35 + 0.02 * (nq > 40 ? nq - 40 : 0)}};
    const Variant* best = nullptr;
    double least = 0.0;
    int per_sm = 0;
    for (const Variant& v : variants) {
        const size_t smem = (size_t)walker_floats(p, v.onchip) * 4;
        if (smem > (size_t)optin) continue;
        const int kind = 2 * (int)(&v - variants);
        e = allow_smem(g_attr, kind, v.kern, smem);
        if (e == cudaSuccess) e = max_carveout(g_attr, kind + 1, v.kern);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, v.kern, 32 * v.warps, smem);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) continue;
        const long long room = (long long)nsm * per_sm;
        const double cost = (double)((n + room - 1) / room) * v.round;
        if (!best || cost < least) {
            best = &v;
            least = cost;
        }
    }
    if (!best) return cudaErrorInvalidValue;
    if (p.nd <= 32) {
        int wpc = 4, l2 = 0;
        const size_t one = (size_t)walker_floats(p, false) * 4;
        while (wpc > 1 && wpc * one > (size_t)optin) wpc /= 2;
        e = cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
        if (e == cudaSuccess) e = allow_smem(g_attr, 6, sweep_warp_kernel, wpc * one);
        if (e == cudaSuccess) e = max_carveout(g_attr, 7, sweep_warp_kernel);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sweep_warp_kernel, 32 * wpc, wpc * one);
        if (e != cudaSuccess) return e;
        const long long room = (long long)nsm * per_sm * wpc;
        const double round = 2.2 + 0.025 * nq - 0.04 * (p.nd > 16 ? p.nd - 16 : 0);
        const double tables = 8.0 * nq * p.npart * (double)(n < room ? n : room);
        if (room > 0 && (double)((n + room - 1) / room) * round < least && tables < 0.8 * l2) {
            sweep_warp_kernel<<<(n + wpc - 1) / wpc, 32 * wpc, wpc * one, stream>>>(p, st, n, nsweep, inv64, inv32, tab, kv, tud, tss,
                                                                                   jA, jC, accepted, prop);
            return cudaGetLastError();
        }
    }
    best->kern<<<n, 32 * best->warps, (size_t)walker_floats(p, best->onchip) * 4, stream>>>(
        p, st, nsweep, inv64, inv32, tab, kv, tud, tss, jA, jC, accepted, prop);
    return cudaGetLastError();
}

}  // namespace dmc
