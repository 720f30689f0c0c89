// Multi-shift tridiagonal route of the pole solves (sm_103a).
//
// All M/2 poles of a window share its standard-form matrix A = L^-1 H_W L^-T (real
// symmetric): the shifted systems differ only by z_k I.  The route therefore reduces A
// once per Hamiltonian to tridiagonal form T = Q^T A Q (Householder), carries the
// owned-point rows through the same reflectors, Y = F^ Q, and then every pole costs a
// complex-symmetric LDL^T of the tridiagonal z_k I - T (O(n)) and one forward sweep per
// row (O(n)):
//
//     d_k(r) = f^_r (z_k I - A)^-1 f^_r^T = y_r (z_k I - T)^-1 y_r^T = sum_i u_i^2 / D_i,
//     D_0 = z - t_0,   D_i = (z - t_i) - e_{i-1}^2 / D_{i-1},
//     u_0 = y_0,       u_i = y_i + (e_{i-1} / D_{i-1}) u_{i-1}.
//
// For Im z > 0, Im D_i >= Im z > 0, so no pivot vanishes and no pivoting is needed.  This
// is the multi-shift reduction used for transfer functions at many frequencies (A. J.
// Laub, "Efficient multivariable frequency response computations", IEEE Trans. Autom.
// Control 26 (1981) 407-408: one Hessenberg reduction, then each shift in O(n^2); for a
// symmetric matrix the Hessenberg form is tridiagonal and each shift is O(n)).  The
// quantities are the same as those of the LDL^T route (window_ldl.cu): the density, the
// electron count and the band energy of every window at every pole, and the pole sums
// are fused into the pass kernel.
//
// Kernels (R = float for the mixed path, double for the FP64 path):
//   tri_reduce_kernel  one CTA per window (work queue, largest first): blocked Householder
//                      tridiagonalisation of the full symmetric window matrix held in an
//                      L2-resident working copy; the rank-2 updates of each panel of nb
//                      columns are delayed (the panel's v and w vectors in shared memory)
//                      and applied once per panel; three barriers per column (the norm, the
//                      dots and A x taken over the unscaled column in one phase).
//                      Algorithmic work (4/3) n^3 flops.
//   tri_reduce_reg_kernel  (FP32, tridiag_reg.cu) the reduction with the window held on its SM.
//   tri_apply_res_kernel  (FP32) one CTA per (window, block of up to 128 rows) with the
//                      rows resident in shared memory through all panels: Y = F^ Q by
//                      panels in compact WY form, Y <- Y - ((Y V) T_p) V^T, 4 x 4 register
//                      tiles.  Algorithmic work 2 m n^2 flops per window.
//   tri_gram_kernel / tri_tfactor_kernel   per (window, panel): V^T V (one CTA), then the
//                      T_p of the compact WY form (one warp), once per Hamiltonian for all
//                      row sets.
//   tri_apply_kernel   one CTA per (window, block of up to 256 rows), one thread per row,
//                      the rows re-read from global memory per panel (FP32, the
//                      configurations without resident rows).
//   tri_pass_kernel    one CTA per (window, batch of rows) from a work queue: thread =
//                      (pole, rows); the pivot recurrence of its pole is shared by its rows,
//                      the row values staged in shared memory by asynchronous copies; the
//                      quadratic forms are reduced over the poles into n(r) and e(r) in
//                      FP64 in a fixed order.  Algorithmic work ~11 real flops per (pole,
//                      row, step) plus the pivot recurrence.
//   tri_sturm_kernel / tri_mineig_kernel   Sturm counts of T - sigma (FP64 arithmetic): the
//                      Sylvester inertia of sigma S_W - H_W, and the smallest eigenvalue of
//                      every window by bisection.
#include "common.cuh"
#include "launch.cuh"
#include "lres_internal.h"

#include <algorithm>
#include <cmath>

namespace lres {
namespace {

template <class R> struct Cplx;
template <> struct Cplx<float> { using T = float2; };
template <> struct Cplx<double> { using T = double2; };

template <class R>
__device__ __forceinline__ R warp_sum(R x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Sum over the CTA; every thread gets the same value, bit for bit (the butterfly gives all
// lanes one result and the warp totals are added in one fixed order).  red: NT/32 slots.
template <int NT, class R>
__device__ __forceinline__ R block_sum(R x, R* red) {
    x = warp_sum(x);
    __syncthreads();                          // red may still be read by a previous call
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    R s = red[0];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) s += red[w];
    return s;
}

template <class R>
__device__ __forceinline__ void cp_async4(R* dst, const R* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(R) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

constexpr int kAppRows = 256;                 // rows of one item of the apply kernel

// ---------------------------------------------------------------------------
// Householder tridiagonalisation
// ---------------------------------------------------------------------------

// Four consecutive rows of a column (16-byte aligned for float, two 16-byte loads for double).
__device__ __forceinline__ void ld4(const float* p, float (&x)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&x)[4]) {
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}
__device__ __forceinline__ void st4(float* p, const float (&x)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
__device__ __forceinline__ void st4(double* p, const double (&x)[4]) {
    *reinterpret_cast<double2*>(p) = make_double2(x[0], x[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(x[2], x[3]);
}

template <class R>
struct TriReduceParams {
    int nwin;
    const int* order;        // windows, largest first
    int* counter;            // work-queue head (zeroed before launch)
    const int* n_w;
    const long long* offC;   // standard-form blocks (n x n, column-major)
    const long long* offA;   // working blocks (ld x n, ld = n rounded up to 4)
    const long long* offN;   // window vectors (n)
    const R* H;              // standard-form matrices (lower triangle read)
    R* A;                    // working copies; on return the reflectors below the subdiagonal
    R* d;                    // diagonal of T
    R* e;                    // subdiagonal of T (e[i] couples i and i+1)
    R* tau;                  // reflector scalars
    int* status;
    int nb;                  // panel width (<= 32)
    int ldv;                 // length of the shared vectors (multiple of 32, >= every n)
    int keep;                // > 0: stop before the last `keep` columns (tridiag_reg.cu takes over)
};

// Shared memory of the reduction, in elements of R.
inline size_t reduce_smem_elems(int nb, int ldv, int nt, int cl = 1) {
    const size_t big = std::max((size_t)2 * nb * ldv, (size_t)(nt / 32) * 32 * 33);
    return big + (4 + cl) * (size_t)ldv + 4 * (size_t)nt + 64 + nt / 32;
}

// CTAs per SM that the reduction is compiled for (registers: 65536 / (NT * that)).
constexpr int reduce_min_ctas(int nt, int elem) { return elem != 4 ? 512 / nt : 1024 / nt; }

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Barrier of the cluster; what its CTAs wrote before (global and shared memory) is visible after.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// x to the same shared variable of CTA `rank` of the cluster
__device__ __forceinline__ void st_cluster(double* dst, unsigned rank, double x) {
    unsigned a = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}

// In FP64 every warp instruction holds its quarter of the SM for 80 clocks, so nothing is computed twice that
// one warp can publish: the root and divisions of the reflector run in the last warp beside the others' A x,
// the sum of p^T v in the warps that own rows only (in every warp, the same bits: a third of the FP64
// instructions; 54 windows 7.6 -> 5.55 ms, one of 96 functions 1.64 -> 1.03 ms; with panels of 8 5.17 and 0.92).
//
// CL = 2: a cluster of two CTAs per window, for fewer windows than half the SMs.  Both form the columns, reflectors
// and vectors (the same bits); the row quads of q = A x and the blocks of the trailing update, which hold the
// FP64 pipe, are dealt to them, q exchanged through distributed shared memory (two buffers by column parity:
// the other CTA may be a phase ahead).  One and two CTAs, 1 to 54 windows (the same time): 48 functions 0.50 and
// 0.65 ms, 96 0.91 and 1.11, where the barriers outweigh the work, 160 1.86 and 1.93, 192 2.58 and 2.43, 240
// 4.08 and 3.45, 300 6.87 and 5.17, 384 12.7 and 8.5, 510 27.3 and 16.7.
template <class R, int NT, int CL = 1>
__global__ void __launch_bounds__(NT, reduce_min_ctas(NT, sizeof(R))) tri_reduce_kernel(TriReduceParams<R> p) {
    constexpr int NW = NT / 32;
    constexpr bool FP64 = sizeof(R) == 8;
    constexpr int NA = FP64 ? NT - 32 : NT;              // threads of q = A x (FP64: the last warp forms the reflector)
    const int rank = CL > 1 ? (int)cluster_rank() : 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ldv = p.ldv, nb = p.nb;
    R* const big = reinterpret_cast<R*>(smem_raw);
    R* const Vs = big;                                   // [nb][ldv]: v_l[i] at Vs[l*ldv + i]
    R* const Ws = big + (size_t)nb * ldv;                // [nb][ldv]
    R* const cv = big + std::max((size_t)2 * nb * ldv, (size_t)NW * 32 * 33);   // [ldv] current column
    R* const pv = cv + ldv;                              // [ldv] p = tau (A v)
    R* const qx0 = pv + ldv;                             // [CL][ldv] q = A x (unsplit)
    R* const acol = qx0 + CL * ldv;                      // [2][ldv] panel-start columns j, j+1
    R* const psum = acol + 2 * ldv;                      // [4 NT] split sums of A x
    R* const dots = psum + 4 * NT;                       // [64] W^T x, V^T x, x^T x
    R* const red = dots + 64;                            // [NW]
    __shared__ int item_sh;
    __shared__ R refl[3];                                // beta, tau, 1 / (alpha - beta) of the column
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (;;) {
        int it;
        if constexpr (CL > 1) {                           // one window per cluster
            it = blockIdx.x / CL;
        } else {
            if (tid == 0) item_sh = atomicAdd(p.counter, 1);
            __syncthreads();
            it = item_sh;
        }
        if (it >= p.nwin) return;
        const int w = p.order[it];
        const int n = p.n_w[w];
        if (n > ldv || n < 1) {
            if (tid == 0) atomicOr(p.status, ST_BAD_SHAPE);
            if constexpr (CL > 1) return;
            __syncthreads();
            continue;
        }
        if (n <= p.keep) {
            if constexpr (CL > 1) return;
            __syncthreads();                      // item_sh is read before the next fetch
            continue;
        }
        const int ld = (n + 3) & ~3;
        const R* H = p.H + p.offC[w];
        R* A = p.A + p.offA[w];
        R* dw = p.d + p.offN[w];
        R* ew = p.e + p.offN[w];
        R* tw = p.tau + p.offN[w];

        // ---- A = the full symmetric matrix from the lower triangle of H, by 32 x 32 blocks
        //      (each warp owns a padded tile: both the block and its transpose are written
        //      with coalesced stores)
        {
            R* tile = big + (size_t)warp * 32 * 33;
            const int nt = (n + 31) / 32;
            for (int t = warp + rank * NW; t < nt * (nt + 1) / 2; t += NW * CL) {
                int bi = 0, bk = t;                      // t-th block of the lower block triangle
                while (bk > bi) {
                    bk -= bi + 1;
                    ++bi;
                }
                const int i0 = bi * 32, k0 = bk * 32;
                for (int c = 0; c < 32; ++c) {
                    const int i = i0 + lane, k = k0 + c;
                    tile[c * 33 + lane] = (i < n && k < n) ? H[i + (long long)k * n] : R(0);
                }
                __syncwarp();
                for (int c = 0; c < 32; ++c) {
                    const int i = i0 + lane, k = k0 + c;
                    if (i < n && k < n)
                        A[i + (long long)k * ld] = (bi != bk || lane >= c) ? tile[c * 33 + lane] : tile[lane * 33 + c];
                }
                if (bi != bk)
                    for (int c = 0; c < 32; ++c) {
                        const int k = k0 + lane, i = i0 + c;
                        if (i < n && k < n) A[k + (long long)i * ld] = tile[lane * 33 + c];
                    }
                __syncwarp();
            }
        }
        if constexpr (CL > 1) cluster_sync();
        else __syncthreads();

        // Each column takes three barriers.  Rows are owned by threads (row i by thread i mod NT)
        // for the column, the reflector and w; the norm, the dots W^T x, V^T x and q = A x are
        // taken over the unscaled column x (rows >= j+2) in one phase, and the reflector's scale
        // is applied afterwards: A v = A e_{j+1} + scal A x, X^T v = X_{j+1} + scal X^T x.  The
        // panel-start column j+1 of the owned rows is fetched by cp.async during column j: it
        // is A e_{j+1} of column j and the start of column j+1.
        R Kprev = R(0);
        for (int j0 = 0; j0 < n - 2 && n - j0 > p.keep; j0 += nb) {
            const int nbp = min(nb, n - 2 - j0);
            for (int jj = 0; jj < nbp; ++jj) {
                const int j = j0 + jj;
                R* const anext = acol + ((j + 1) & 1) * ldv;
                const R* const acur = acol + (j & 1) * ldv;
                for (int i = tid; i < n; i += NT)
                    if (i > j) cp_async4(anext + i, A + i + (long long)(j + 1) * ld);
                cp_commit();
                // (a) column j of the current matrix (panel-start values minus the pending rank-2
                //     updates of this panel) on the owned rows >= j.  w_{jj-1} at row j is
                //     p_j - K (v_{jj-1} is 1 there); every thread forms it from the published p.
                {
                    for (int i = tid; i < n; i += NT) {
                        if (i < j) continue;
                        const R wlast = jj > 0 ? pv[j] - Kprev : R(0);
                        R c = jj > 0 ? acur[i] : A[i + (long long)j * ld];
                        for (int l = 0; l < jj; ++l) {
                            const R wlj = l == jj - 1 ? wlast : Ws[l * ldv + j];
                            if constexpr (FP64) c = fma(-Ws[l * ldv + i], Vs[l * ldv + j], fma(-Vs[l * ldv + i], wlj, c));
                            else c -= Vs[l * ldv + i] * wlj + Ws[l * ldv + i] * Vs[l * ldv + j];
                        }
                        cv[i] = c;
                    }
                }
                __syncthreads();
                // (b) q = A x on rows >= j+1 by quads of rows (16-byte loads) from the aligned row
                //     i0 <= j+1; when the quads are few, the columns are split across thread groups
                //     and the partial sums added in a fixed order.  Sums are blocked: each run of
                //     32 terms from zero.
                const int i0 = (j + 1) & ~3;
                const int nq = (ld - i0) >> 2;
                const int nqo = (nq + CL - 1) / CL;             // this CTA's quads: rank, rank + CL, ...
                const int nsplit = nqo >= NA ? 1 : NA / nqo;
                R* const qx = qx0 + (j & (CL - 1)) * ldv;
                auto publish = [&](int i, R x) {
                    qx[i] = x;
                    if constexpr (CL > 1) st_cluster(qx + i, rank ^ 1, x);
                };
                {
                    const int qstep = nqo >= NA ? NA : nqo;
                    if (tid < qstep * nsplit) {
                        const int sp = tid / qstep;
                        for (int u = tid % qstep; u < nqo; u += qstep) {
                            const int q = u * CL + rank;
                            if (q >= nq) break;
                            const R* Aq = A + i0 + 4 * q;
                            R a[4] = {R(0), R(0), R(0), R(0)};
                            for (int kb = j + 2 + sp; kb < n; kb += 32 * nsplit) {
                                const int ke = min(n, kb + 32 * nsplit);
                                R c[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll 8
                                for (int k = kb; k < ke; k += nsplit) {
                                    R x[4];
                                    ld4(Aq + (long long)k * ld, x);
                                    const R xk = cv[k];
#pragma unroll
                                    for (int r = 0; r < 4; ++r) c[r] = fma(x[r], xk, c[r]);
                                }
#pragma unroll
                                for (int r = 0; r < 4; ++r) a[r] = kb == j + 2 + sp ? c[r] : a[r] + c[r];
                            }
                            if (nsplit > 1) {
                                st4(psum + (sp * nqo + u) * 4, a);   // 16-byte stores: no bank conflicts
                            } else {
#pragma unroll
                                for (int r = 0; r < 4; ++r) {
                                    const int i = i0 + 4 * q + r;
                                    if (i > j && i < n) publish(i, a[r]);
                                }
                            }
                        }
                    }
                }
                //     dots[l] = W_l^T x, dots[jj + l] = V_l^T x over rows >= j+2, a warp each; the last warp:
                //     x^T x and from it the reflector H_j = I - tau v v^T with v_{j+1} = 1 mapping rows j+1..
                //     of the column onto beta e_{j+1}
                auto dot = [&](const R* X) {
                    R acc = R(0);
                    for (int i = j + 2 + lane; i < n; i += 32) acc += X[i] * cv[i];
                    return warp_sum(acc);
                };
                if (warp == NW - 1) {
                    const R s2 = dot(cv);
                    const R alpha = cv[j + 1];
                    R beta = alpha, tau = R(0), scal = R(0);
                    if (s2 > R(0)) {
                        const R nrm = sqrt(alpha * alpha + s2);
                        beta = alpha >= R(0) ? -nrm : nrm;
                        tau = (beta - alpha) / beta;
                        scal = R(1) / (alpha - beta);
                    }
                    if (lane == 0) {
                        refl[0] = beta;
                        refl[1] = tau;
                        refl[2] = scal;
                    }
                } else {
                    for (int q = NW - 2 - warp; q < 2 * jj; q += NW - 1) {
                        const R acc = dot(q < jj ? Ws + (size_t)q * ldv : Vs + (size_t)(q - jj) * ldv);
                        if (lane == 0) dots[q] = acc;
                    }
                }
                if constexpr (CL > 1) {
                    if (nsplit > 1) {
                        __syncthreads();
                        for (int idx = tid; idx < 4 * nqo; idx += NT) {
                            const int u = idx >> 2, r = idx & 3, i = i0 + 4 * (u * CL + rank) + r;
                            if (i <= j || i >= n) continue;
                            R qi = R(0);
                            for (int sp = 0; sp < nsplit; ++sp) qi += psum[(sp * nqo + u) * 4 + r];
                            publish(i, qi);
                        }
                    }
                    cluster_sync();
                } else {
                    __syncthreads();
                }
                // (c) p = tau (A v - V (W^T v) - W (V^T v)) on the owned rows, partial sums of p^T v
                const R beta = refl[0], tau = refl[1], scal = refl[2];
                const bool owner = n > NT || (32 * warp + 31 > j && 32 * warp < n);     // rows > j in this warp
                if (tid == 0 && rank == 0) {
                    dw[j] = cv[j];
                    ew[j] = beta;
                    tw[j] = tau;
                    if (!isfinite((double)beta) || !isfinite((double)cv[j])) atomicOr(p.status, ST_ZERO_PIVOT);
                }
                cp_wait<0>();
                R partK = R(0);
                for (int i = tid; i < ldv; i += NT) {
                    R vi = R(0);
                    if (i == j + 1) vi = R(1);
                    else if (i > j + 1 && i < n) vi = cv[i] * scal;
                    Vs[jj * ldv + i] = vi;
                    if (i > j && i < n) {
                        if (i > j + 1 && rank == 0) A[i + (long long)j * ld] = vi;      // kept for Y = F^ Q
                        R qi;
                        if (CL == 1 && nsplit > 1) {
                            const int q = (i - i0) >> 2, r = (i - i0) & 3;
                            qi = R(0);
                            for (int sp = 0; sp < nsplit; ++sp) qi += psum[(sp * nq + q) * 4 + r];
                        } else {
                            qi = qx[i];
                        }
                        R pi = anext[i] + scal * qi;
                        for (int l = 0; l < jj; ++l) {
                            const R dW = Ws[l * ldv + j + 1] + scal * dots[l];
                            const R dV = Vs[l * ldv + j + 1] + scal * dots[jj + l];
                            if constexpr (FP64) pi = fma(-Ws[l * ldv + i], dV, fma(-Vs[l * ldv + i], dW, pi));
                            else pi -= Vs[l * ldv + i] * dW + Ws[l * ldv + i] * dV;
                        }
                        pi *= tau;
                        pv[i] = pi;
                        partK += pi * vi;
                    }
                }
                if (owner) partK = warp_sum(partK);
                if (lane == 0) red[warp] = partK;
                __syncthreads();
                // (d) K = tau/2 p^T v, w = p - K v on the owned rows
                R K = R(0);
                if (owner) K = R(0.5) * tau * warp_sum(lane < NW ? red[lane] : R(0));
                Kprev = K;
                for (int i = tid; i < ldv; i += NT)
                    Ws[jj * ldv + i] = (i > j && i < n) ? pv[i] - K * Vs[jj * ldv + i] : R(0);
            }
            __syncthreads();
            // ---- trailing update A -= V W^T + W V^T on rows, columns >= t0: the blocks on and below
            //      the diagonal, each written to its mirror image as well (half the multiply-adds, which
            //      bound the FP64 kernel: 54 windows 11.2 -> 9.2 ms, 432 windows 31.9 -> 26.5 ms).  One quad of rows x one aligned quad of columns per thread,
            //      consecutive threads down a column quad: the v, w values of both quads come from
            //      shared memory as 16-byte vectors; rows and columns below t0 are left unchanged.
            const int t0 = j0 + nbp;
            if (t0 < n) {
                const int q0 = t0 & ~3;
                const int nq = (ld - q0) >> 2;
                for (int tile = tid + rank * NT; tile < nq * (nq + 1) / 2; tile += NT * CL) {
                    // column quads from the last: quad nq-1-u has u + 1 blocks
                    int u = (int)((sqrtf(8.0f * tile + 1.0f) - 1.0f) * 0.5f);
                    while ((u + 1) * (u + 2) / 2 <= tile) ++u;
                    while (u * (u + 1) / 2 > tile) --u;
                    const int cb = nq - 1 - u, q = cb + tile - u * (u + 1) / 2;
                    const int i = q0 + 4 * q, c0 = q0 + 4 * cb;
                    R acc[4][4];
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int r = 0; r < 4; ++r) acc[c][r] = R(0);
                    for (int l = 0; l < nbp; ++l) {
                        R vi[4], wi[4], vk[4], wk[4];
                        ld4(Vs + (size_t)l * ldv + i, vi);
                        ld4(Ws + (size_t)l * ldv + i, wi);
                        ld4(Vs + (size_t)l * ldv + c0, vk);
                        ld4(Ws + (size_t)l * ldv + c0, wk);
#pragma unroll
                        for (int c = 0; c < 4; ++c)
#pragma unroll
                            for (int r = 0; r < 4; ++r) acc[c][r] = fma(vi[r], wk[c], fma(wi[r], vk[c], acc[c][r]));
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int col = c0 + c;
                        if (col < t0 || col >= n) continue;
                        R x[4];
                        R* dst = A + i + (long long)col * ld;
                        ld4(dst, x);
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            if (i + r >= t0) x[r] -= acc[c][r];
                            acc[c][r] = x[r];
                        }
                        st4(dst, x);
                    }
                    if (q == cb) continue;                           // (both halves of a diagonal block)
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (i + r >= n) continue;                    // (i > c0, so i + r >= t0)
                        R* dst = A + c0 + (long long)(i + r) * ld;
                        if (c0 >= t0) {
                            const R x[4] = {acc[0][r], acc[1][r], acc[2][r], acc[3][r]};
                            st4(dst, x);
                        } else {
#pragma unroll
                            for (int c = 0; c < 4; ++c)
                                if (c0 + c >= t0) dst[c] = acc[c][r];
                        }
                    }
                }
            }
            if constexpr (CL > 1) cluster_sync();
            else __syncthreads();
        }
        // ---- the last (at most 2 x 2) block, fully updated
        if (tid == 0 && rank == 0 && !p.keep) {
            if (n >= 2) {
                dw[n - 2] = A[(n - 2) + (long long)(n - 2) * ld];
                ew[n - 2] = A[(n - 1) + (long long)(n - 2) * ld];
                dw[n - 1] = A[(n - 1) + (long long)(n - 1) * ld];
                tw[n - 2] = R(0);
                tw[n - 1] = R(0);
                ew[n - 1] = R(0);
            } else {
                dw[0] = A[0];
                tw[0] = R(0);
                ew[0] = R(0);
            }
        }
        if constexpr (CL > 1) return;                     // (the last cluster barrier is behind every exchange)
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Y = F^ Q: the rows through the reflectors, compact WY per panel
// ---------------------------------------------------------------------------

template <class R>
struct TriApplyParams {
    int nitems;
    const int4* items;       // (window, first row, rows <= 256, -)
    const int* n_w;
    const int* m_w;          // rows of each window
    const long long* offA;   // reflectors (working blocks, leading dimension n rounded up to 4)
    const long long* offN;
    const long long* offF;   // row blocks, F[r + a*m]
    const R* A;              // reflectors below the subdiagonal (tri_reduce_kernel)
    const R* tau;
    const R* F;              // standard-form rows
    R* Y;                    // F^ Q, same layout
    int ldv;
};

// Index of v_l[k] in the staged panel: rows of NB values, 16-byte groups of each row permuted
// by XOR with the row index, so that the staging stores (consecutive k, one l) spread over the
// banks while each row is still read as aligned 16-byte vectors.
template <class R, int NB>
__device__ __forceinline__ int panel_index(int k, int l) {
    constexpr int GW = 16 / (int)sizeof(R) < NB ? 16 / (int)sizeof(R) : NB;   // elements per group
    constexpr int NG = NB / GW;                                                 // groups per row
    return k * NB + (((l / GW) ^ (k % NG)) * GW) + (l % GW);
}

// One 16-byte group of a staged row (4 floats or 2 doubles; a narrower panel row whole).
template <class R, int GW>
__device__ __forceinline__ void ld_group(const R* src, R (&x)[GW]) {
    if constexpr (sizeof(R) == 4 && GW == 4) {
        const float4 v = *reinterpret_cast<const float4*>(src);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else if constexpr (sizeof(R) == 8 && GW == 2) {
        const double2 v = *reinterpret_cast<const double2*>(src);
        x[0] = v.x; x[1] = v.y;
    } else {
#pragma unroll
        for (int e = 0; e < GW; ++e) x[e] = src[e];
    }
}

// NT threads handle the item's rows (at most NT * RPT), RPT rows each (rows tid + u NT), so
// that every staged reflector value feeds RPT multiply-adds.
template <class R, int NT, int NB, int RPT>
__global__ void __launch_bounds__(NT, RPT == 1 && NB <= 16 ? 3 : 1) tri_apply_kernel(TriApplyParams<R> p) {
    constexpr int GW = 16 / (int)sizeof(R) < NB ? 16 / (int)sizeof(R) : NB;
    constexpr int NG = NB / GW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* const Vs = reinterpret_cast<R*>(smem_raw);         // [ldv][NB], panel_index layout
    R* const Tm = Vs + (size_t)p.ldv * NB;                 // [NB][NB] upper triangular factor
    R* const Gm = Tm + NB * NB;                            // [NB][NB] V^T V (above the diagonal)
    const int4 item = p.items[blockIdx.x];
    const int w = item.x, r0 = item.y, nr = item.z;
    const int n = p.n_w[w], m = p.m_w[w];
    if (n > p.ldv) return;                                 // the reduction flagged this window
    const long long ld = (n + 3) & ~3;
    const R* Aw = p.A + p.offA[w];
    const R* tw = p.tau + p.offN[w];
    const R* Fw = p.F + p.offF[w];
    R* Yw = p.Y + p.offF[w];
    const int tid = threadIdx.x;
    bool act[RPT];
    long long rr[RPT];
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int t = tid + u * NT;
        act[u] = t < nr && r0 + t < m;
        rr[u] = act[u] ? r0 + t : 0;
    }
#pragma unroll
    for (int u = 0; u < RPT; ++u)
        if (act[u]) {
#pragma unroll 8
            for (int k = 0; k < n; ++k) Yw[rr[u] + (long long)k * m] = Fw[rr[u] + (long long)k * m];
        }

    for (int j0 = 0; j0 < n - 2; j0 += NB) {
        const int nbp = min(NB, n - 2 - j0);
        const int nk = n - j0 - 1;                         // rows j0+1 .. n-1
        __syncthreads();                                   // the previous panel is consumed
        // v_l (l < nbp) lives on rows j0+l+1 .. n-1 (v_l[j0+l+1] = 1); reads run down the
        // columns of the reflector storage (coalesced)
        for (int idx = tid; idx < nk * NB; idx += NT) {
            const int l = idx / nk, k = j0 + 1 + idx % nk;
            R v = R(0);
            if (l < nbp) {
                const int j = j0 + l;
                if (k == j + 1) v = R(1);
                else if (k > j + 1) v = Aw[k + j * ld];
            }
            Vs[panel_index<R, NB>(k, l)] = v;
        }
        __syncthreads();
        // G = V^T V by 2 x 2 blocks per thread (entries above the diagonal are used)
        for (int q = tid; q < NB * NB / 4; q += NT) {
            const int a0 = 2 * (q / (NB / 2)), b0 = 2 * (q % (NB / 2));
            R g00 = R(0), g01 = R(0), g10 = R(0), g11 = R(0);
            if (b0 + 1 > a0) {
                for (int k = j0 + 1; k < n; ++k) {
                    const R va0 = Vs[panel_index<R, NB>(k, a0)], va1 = Vs[panel_index<R, NB>(k, a0 + 1)];
                    const R vb0 = Vs[panel_index<R, NB>(k, b0)], vb1 = Vs[panel_index<R, NB>(k, b0 + 1)];
                    g00 = fma(va0, vb0, g00);
                    g01 = fma(va0, vb1, g01);
                    g10 = fma(va1, vb0, g10);
                    g11 = fma(va1, vb1, g11);
                }
            }
            Gm[a0 * NB + b0] = g00;
            Gm[a0 * NB + b0 + 1] = g01;
            Gm[(a0 + 1) * NB + b0] = g10;
            Gm[(a0 + 1) * NB + b0 + 1] = g11;
        }
        __syncthreads();
        // T (forward, columnwise): T_ll = tau_l, T[0:l, l] = -tau_l T[0:l, 0:l] (V^T V)[0:l, l]
        if (tid < 32) {
            for (int l = 0; l < NB; ++l) {
                const R tl = l < nbp ? tw[j0 + l] : R(0);
                for (int a = tid; a < NB; a += 32) {
                    R val = R(0);
                    if (a < l) {
                        R sacc = R(0);
                        for (int b = a; b < l; ++b) sacc = fma(Tm[a * NB + b], Gm[b * NB + l], sacc);
                        val = -tl * sacc;
                    } else if (a == l) {
                        val = tl;
                    }
                    Tm[a * NB + l] = val;
                }
                __syncwarp();
            }
        }
        __syncthreads();
        R sv[RPT][NB];
#pragma unroll
        for (int u = 0; u < RPT; ++u)
#pragma unroll
            for (int l = 0; l < NB; ++l) sv[u][l] = R(0);
#pragma unroll 4
        for (int k = j0 + 1; k < n; ++k) {
            R y[RPT];
#pragma unroll
            for (int u = 0; u < RPT; ++u) y[u] = act[u] ? Yw[rr[u] + (long long)k * m] : R(0);
            const R* row = Vs + (size_t)k * NB;
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                R x[GW];
                ld_group<R, GW>(row + ((g ^ (k % NG)) * GW), x);
#pragma unroll
                for (int u = 0; u < RPT; ++u)
#pragma unroll
                    for (int e = 0; e < GW; ++e) sv[u][g * GW + e] = fma(y[u], x[e], sv[u][g * GW + e]);
            }
        }
        // s <- s T in place (T upper triangular: column b needs s_0..s_b, so b descends)
#pragma unroll
        for (int b = NB - 1; b >= 0; --b) {
            R acc[RPT];
#pragma unroll
            for (int u = 0; u < RPT; ++u) acc[u] = R(0);
#pragma unroll
            for (int a = 0; a <= b; ++a) {
                const R t = Tm[a * NB + b];
#pragma unroll
                for (int u = 0; u < RPT; ++u) acc[u] = fma(sv[u][a], t, acc[u]);
            }
#pragma unroll
            for (int u = 0; u < RPT; ++u) sv[u][b] = acc[u];
        }
#pragma unroll 4
        for (int k = j0 + 1; k < n; ++k) {
            const R* row = Vs + (size_t)k * NB;
            R acc[RPT];
#pragma unroll
            for (int u = 0; u < RPT; ++u) acc[u] = R(0);
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                R x[GW];
                ld_group<R, GW>(row + ((g ^ (k % NG)) * GW), x);
#pragma unroll
                for (int u = 0; u < RPT; ++u)
#pragma unroll
                    for (int e = 0; e < GW; ++e) acc[u] = fma(sv[u][g * GW + e], x[e], acc[u]);
            }
#pragma unroll
            for (int u = 0; u < RPT; ++u)
                if (act[u]) Yw[rr[u] + (long long)k * m] -= acc[u];
        }
    }
}

// ---------------------------------------------------------------------------
// Y = F^ Q with the item's rows resident in shared memory (FP32)
// ---------------------------------------------------------------------------
//
// The rows of one item (at most kResRows) stay in shared memory through all panels, so Y
// crosses to global memory once per launch instead of once per panel.  Per panel of NB
// reflectors: S = Y V (a thread = 4 rows x 4 reflectors; a warp = 8 row quads x 4 reflector
// quads, so that every 16-byte shared load serves a broadcast or one conflict-free
// wavefront), S <- S T (same tiles), Y <- Y - S V^T (a thread = 4 rows x 4 columns; a warp =
// 8 row quads x 4 column quads).  The T factor of every (window, panel) is formed once per
// Hamiltonian by tri_gram_kernel and tri_tfactor_kernel.

constexpr int kResRows = 128;                 // rows of an item of the resident application
constexpr int kResNT = 512;

// Staged panel: rows of NB values v_l[k]; the 16-byte groups of row kk permuted by XOR with
// kk / 4, so that rows 4 apart (one per column quad of a warp) hit different banks.
template <int NB>
__device__ __forceinline__ int res_index(int kk, int l) {
    constexpr int NG = NB / 4;
    return kk * NB + ((((l >> 2) ^ (kk >> 2)) & (NG - 1)) << 2) + (l & 3);
}

// v_l (l < nbp) on the panel rows kk = 0..nk-1 (window row j0+1+kk), v_l = 1 on row j0+l+1,
// zero above; reads run down the reflector columns (coalesced).
// The reflector values go by asynchronous copies (all of a thread's copies in flight at
// once), the zeros and ones by plain stores; the caller waits (cp_wait) before the barrier.
template <int NT, int NB>
__device__ __forceinline__ void res_stage(float* Vs, const float* Aw, long long ld, int j0, int nbp, int nk) {
    // warp per reflector column, lanes down its rows (no division by nk)
    const int lane = threadIdx.x & 31;
    for (int l = threadIdx.x >> 5; l < NB; l += NT / 32) {
        const int j = j0 + l;
        const float* src = Aw + (long long)j * ld;
        for (int kk = lane; kk < nk; kk += 32) {
            const int k = j0 + 1 + kk;
            float* dst = Vs + res_index<NB>(kk, l);
            if (l < nbp && k > j + 1) cp_async4(dst, src + k);
            else *dst = (l < nbp && k == j + 1) ? 1.0f : 0.0f;
        }
    }
    cp_commit();
}

constexpr int kTfSplit = 4;                   // row ranges of V^T V in the T-factor kernel

// scratch of the partial blocks of V^T V, in floats (aliases T and what follows it)
__host__ __device__ inline int tf_part_elems(int nb) { return kTfSplit * (nb / 4) * (nb / 4 + 1) / 2 * 16; }

struct TriTParams {
    int nwin;
    int maxp;                // panels per window at most
    const int* n_w;
    const long long* offA;
    const long long* offN;
    const float* A;
    const float* tau;
    float* T;                // [window][panel][NB][NB], upper triangular
    long long tstride;       // per window
    int ldv;
};

// T of the compact WY form of one panel, Q_p = I - V T V^T: T_ll = tau_l,
// T[0:l, l] = -tau_l T[0:l, 0:l] (V^T V)[0:l, l].  One CTA per (window, panel).
template <int NB>
__global__ void __launch_bounds__(128) tri_gram_kernel(TriTParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* const Vs = reinterpret_cast<float*>(smem_raw);      // [ldv][NB]
    float* const Gm = Vs + (size_t)p.ldv * NB;                  // [NB][NB]
    float* const Tm = Gm + NB * NB;                              // [NB][NB]; the partial blocks of G first
    const int w = blockIdx.x / p.maxp, panel = blockIdx.x % p.maxp;
    const int n = p.n_w[w];
    const int j0 = panel * NB;
    if (n > p.ldv || j0 >= n - 2) return;
    const int tid = threadIdx.x;
    const int nbp = min(NB, n - 2 - j0), nk = n - j0 - 1;
    const long long ld = (n + 3) & ~3;
    res_stage<128, NB>(Vs, p.A + p.offA[w], ld, j0, nbp, nk);
    cp_wait<0>();
    __syncthreads();
    // G = V^T V by 4 x 4 blocks on or above the diagonal (16-byte reads of the staged rows),
    // the rows split into kTfSplit ranges whose partial blocks are added in range order
    {
        constexpr int NQ = NB / 4, NTILE = NQ * (NQ + 1) / 2;
        float* const part = Tm;                                  // [kTfSplit][NTILE][16] scratch
        for (int item = tid; item < NTILE * kTfSplit; item += 128) {
            const int tile = item % NTILE, sp = item / NTILE;
            int qa = 0, rem = tile;                              // tile-th (qa <= qb) pair
            while (rem >= NQ - qa) {
                rem -= NQ - qa;
                ++qa;
            }
            const int qb = qa + rem;
            const int k0 = nk * sp / kTfSplit, k1 = nk * (sp + 1) / kTfSplit;
            float g[4][4] = {};
            for (int kk = k0; kk < k1; ++kk) {
                const float4 x = *reinterpret_cast<const float4*>(Vs + kk * NB + (((qa ^ (kk >> 2)) & (NQ - 1)) << 2));
                const float4 y = *reinterpret_cast<const float4*>(Vs + kk * NB + (((qb ^ (kk >> 2)) & (NQ - 1)) << 2));
                const float xa[4] = {x.x, x.y, x.z, x.w}, yb[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) g[r][c] = fmaf(xa[r], yb[c], g[r][c]);
            }
            float* dst = part + ((size_t)sp * NTILE + tile) * 16;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) dst[r * 4 + c] = g[r][c];
        }
        __syncthreads();
        for (int item = tid; item < NTILE * 16; item += 128) {
            const int tile = item / 16, e = item % 16;
            int qa = 0, rem = tile;
            while (rem >= NQ - qa) {
                rem -= NQ - qa;
                ++qa;
            }
            const int qb = qa + rem;
            float s = 0.0f;
            for (int sp = 0; sp < kTfSplit; ++sp) s += part[((size_t)sp * NTILE + tile) * 16 + e];
            Gm[(4 * qa + e / 4) * NB + 4 * qb + e % 4] = s;
        }
        __syncthreads();
    }
    // G (the blocks on and above the diagonal) into the panel's T slot; tri_tfactor_kernel
    // turns it into T in place
    float* Gw = p.T + (long long)w * p.tstride + (long long)panel * NB * NB;
    for (int i = tid; i < NB * NB; i += 128) Gw[i] = Gm[i];
}

// T of the compact WY form of one panel from its G = V^T V (in the T slot), one warp per
// (window, panel): T_ll = tau_l, T[0:l, l] = -tau_l T[0:l, 0:l] G[0:l, l].  The recurrence is
// sequential in l; a warp per panel keeps many panels in flight on each SM.
template <int NB>
__global__ void __launch_bounds__(32) tri_tfactor_kernel(TriTParams p) {
    static_assert(NB <= 32, "one lane per reflector of the panel");
    __shared__ float Gm[NB * NB], Tm[NB * NB];
    const int w = blockIdx.x / p.maxp, panel = blockIdx.x % p.maxp;
    const int n = p.n_w[w];
    const int j0 = panel * NB;
    if (n > p.ldv || j0 >= n - 2) return;
    const int tid = threadIdx.x;
    const int nbp = min(NB, n - 2 - j0);
    float* Tw = p.T + (long long)w * p.tstride + (long long)panel * NB * NB;
    for (int i = tid; i < NB * NB; i += 32) Gm[i] = Tw[i];
    // the panel's tau, one per lane (NB <= 32), broadcast in the recurrence (no global load on
    // its sequential path)
    const float* tw = p.tau + p.offN[w];
    const float my_tau = tid < nbp ? tw[j0 + tid] : 0.0f;
    __syncwarp();
    for (int l = 0; l < NB; ++l) {
        const float tl = __shfl_sync(0xffffffffu, my_tau, l);
        for (int a = tid; a < NB; a += 32) {
            float val = 0.0f;
            if (a < l) {
                // four independent partial sums (b mod 4), added in a fixed order
                float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                int b = a;
                for (; b + 3 < l; b += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) s[u] = fmaf(Tm[a * NB + b + u], Gm[(b + u) * NB + l], s[u]);
                }
                for (; b < l; ++b) s[0] = fmaf(Tm[a * NB + b], Gm[b * NB + l], s[0]);
                val = -tl * ((s[0] + s[1]) + (s[2] + s[3]));
            } else if (a == l) {
                val = tl;
            }
            Tm[a * NB + l] = val;
        }
        __syncwarp();
    }
    for (int i = tid; i < NB * NB; i += 32) Tw[i] = Tm[i];
}

inline size_t res_smem_bytes(int nb, int ldv, int rows) {
    return sizeof(float) * ((size_t)ldv * rows + (size_t)ldv * nb + (size_t)nb * rows + (size_t)nb * nb);
}

// Bound by issue and by the shared-memory reads of the 4 x 4 tiles; the rows go in pairs (FFMA2: the same FMAs
// and bits in half the issue slots): with V^T V and T, 1024 windows 2.44 -> 2.34 ms, 512 cell windows of 1000
// points and their trace rows 8.14 -> 7.82 ms.
template <int NB>
__global__ void __launch_bounds__(kResNT, 1) tri_apply_res_kernel(TriApplyParams<float> p, const float* Tg,
                                                                  long long tstride, int rows) {
    constexpr int NG = NB / 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ldv = p.ldv;
    float* const Ys = reinterpret_cast<float*>(smem_raw);       // [ldv][rows]: Y[r][k] at Ys[k * rows + r]
    float* const Vs = Ys + (size_t)ldv * rows;                   // [ldv][NB], res_index layout
    float* const Ss = Vs + (size_t)ldv * NB;                     // [NB][rows]: S[r][l] at Ss[l * rows + r]
    float* const Tm = Ss + (size_t)NB * rows;                    // [NB][NB]
    const int4 item = p.items[blockIdx.x];
    const int w = item.x, r0 = item.y, nr = item.z;
    const int n = p.n_w[w], m = p.m_w[w];
    if (n > ldv || nr > rows) return;                           // flagged by the reduction / never built
    const long long ld = (n + 3) & ~3;
    const float* Aw = p.A + p.offA[w];
    const float* Fw = p.F + p.offF[w] + r0;
    float* Yw = p.Y + p.offF[w] + r0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rq = (nr + 31) / 32;                               // groups of 8 row quads
    for (int k = warp; k < n; k += kResNT / 32)                  // warp per column, lanes down the rows
        for (int r = lane; r < rq * 32; r += 32) {
            if (r < nr) cp_async4(Ys + (size_t)k * rows + r, Fw + r + (long long)k * m);
            else Ys[(size_t)k * rows + r] = 0.0f;
        }
    cp_commit();
    const int rt_l = lane & 7, ct_l = lane >> 3;                 // lane: row quad, reflector / column quad
    for (int j0 = 0; j0 < n - 2; j0 += NB) {
        const int nbp = min(NB, n - 2 - j0);
        const int nk = n - j0 - 1;
        const float* Tp = Tg + (long long)w * tstride + (long long)(j0 / NB) * NB * NB;
        __syncthreads();                                         // the previous panel is consumed
        res_stage<kResNT, NB>(Vs, Aw, ld, j0, nbp, nk);
        for (int i = tid; i < NB * NB; i += kResNT) cp_async4(Tm + i, Tp + i);
        cp_commit();
        cp_wait<0>();                                            // Y (first panel), V, T
        __syncthreads();
        const int nw1 = rq * (NB / 16);                          // 8 x 4 quad tiles of S (phase 2)
        // S = Y V over the panel rows: a warp = 4 row quads x 4 reflector quads x 2 halves of
        // the panel rows, the halves added by a shuffle
        {
            const int kh = lane >> 4, sub = lane & 15;
            const int rt_h = sub & 3, lt_h = sub >> 2;
            const int nwh = 2 * rq * (NB / 16);                  // warp tiles of S
            const int kmid = (nk + 1) >> 1;
            const int ka = kh ? kmid : 0, kz = kh ? nk : kmid;
            for (int wt = warp; wt < nwh; wt += kResNT / 32) {
                const int rt = (wt % (2 * rq)) * 4 + rt_h, lt = (wt / (2 * rq)) * 4 + lt_h;
                float2 acc[2][4];                                // rows 2i, 2i + 1
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
                const float* yp = Ys + (size_t)(j0 + 1) * rows + 4 * rt;
#pragma unroll 4
                for (int kk = ka; kk < kz; ++kk) {
                    const float4 y = *reinterpret_cast<const float4*>(yp + (size_t)kk * rows);
                    const float4 v = *reinterpret_cast<const float4*>(Vs + kk * NB + ((lt ^ (kk >> 2)) & (NG - 1)) * 4);
                    const float2 yy[2] = {make_float2(y.x, y.y), make_float2(y.z, y.w)};
                    const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            acc[i][j] = __ffma2_rn(yy[i], make_float2(vv[j], vv[j]), acc[i][j]);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        acc[i][j].x += __shfl_xor_sync(0xffffffffu, acc[i][j].x, 16);
                        acc[i][j].y += __shfl_xor_sync(0xffffffffu, acc[i][j].y, 16);
                    }
                if (kh == 0) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<float4*>(Ss + (size_t)(4 * lt + j) * rows + 4 * rt) =
                            make_float4(acc[0][j].x, acc[0][j].y, acc[1][j].x, acc[1][j].y);
                }
            }
        }
        __syncthreads();
        // S <- S T (T upper triangular)
        float st[4][4] = {};
        int st_rt = -1, st_bt = 0;
        if (warp < nw1) {                                        // nw1 <= 8: one tile per warp
            st_rt = (warp % rq) * 8 + rt_l;
            st_bt = (warp / rq) * 4 + ct_l;
            const int amax = min(NB, 4 * st_bt + 4);
            for (int a = 0; a < amax; ++a) {
                const float4 s = *reinterpret_cast<const float4*>(Ss + (size_t)a * rows + 4 * st_rt);
                const float4 tt = *reinterpret_cast<const float4*>(Tm + a * NB + 4 * st_bt);
                const float ss[4] = {s.x, s.y, s.z, s.w}, t4[4] = {tt.x, tt.y, tt.z, tt.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) st[i][j] = fmaf(ss[i], t4[j], st[i][j]);
            }
        }
        __syncthreads();
        if (st_rt >= 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(Ss + (size_t)(4 * st_bt + j) * rows + 4 * st_rt) =
                    make_float4(st[0][j], st[1][j], st[2][j], st[3][j]);
        }
        __syncthreads();
        // Y <- Y - S V^T on the panel rows
        const int nw3 = rq * ((nk + 15) / 16);
        for (int wt = warp; wt < nw3; wt += kResNT / 32) {
            const int rt = (wt % rq) * 8 + rt_l, kt = (wt / rq) * 4 + ct_l;
            float2 acc[2][4];                                    // [rows 2i, 2i + 1][column]
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = make_float2(0.f, 0.f);
#pragma unroll
            for (int lc = 0; lc < NG; ++lc) {
                float2 s[4][2];                                  // s[l][rows]
                float v[4][4];                                   // v[column][l]
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const float4 x = *reinterpret_cast<const float4*>(Ss + (size_t)(4 * lc + jj) * rows + 4 * rt);
                    s[jj][0] = make_float2(x.x, x.y);
                    s[jj][1] = make_float2(x.z, x.w);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int kk = 4 * kt + q;
                    const float4 x = *reinterpret_cast<const float4*>(Vs + kk * NB + ((lc ^ kt) & (NG - 1)) * 4);
                    v[q][0] = x.x; v[q][1] = x.y; v[q][2] = x.z; v[q][3] = x.w;
                }
#pragma unroll
                for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            acc[i][q] = __ffma2_rn(s[jj][i], make_float2(v[q][jj], v[q][jj]), acc[i][q]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int kk = 4 * kt + q;
                if (kk < nk) {
                    float4* yp = reinterpret_cast<float4*>(Ys + (size_t)(j0 + 1 + kk) * rows + 4 * rt);
                    float4 y = *yp;
                    y.x -= acc[0][q].x;
                    y.y -= acc[0][q].y;
                    y.z -= acc[1][q].x;
                    y.w -= acc[1][q].y;
                    *yp = y;
                }
            }
        }
    }
    cp_wait<0>();                                                // (no panel: the rows as loaded)
    __syncthreads();
    for (int k = warp; k < n; k += kResNT / 32)
        for (int r = lane; r < nr; r += 32) Yw[r + (long long)k * m] = Ys[(size_t)k * rows + r];
}

// ---------------------------------------------------------------------------
// shifted tridiagonal solves at all poles, fused with the pole sums
// ---------------------------------------------------------------------------

template <class R>
struct TriPassParams {
    int nitems;
    const int4* items;       // (window, first row, rows <= rows per batch, -)
    int* counter;
    const int* n_w;
    const int* m_w;
    const long long* offN;
    const long long* offF;   // rows Y[r + i*m]
    const long long* offQ;   // first point of each window in Oflat
    const long long* Oflat;  // grid index of every owned point (nullable: no density)
    const R* Y;
    const R* d;
    const R* e;
    int P;                   // poles (upper half plane)
    const typename Cplx<R>::T* shifts;
    const double2* wq;       // w_k
    const double2* wzq;      // w_k z_k
    double* dens;            // nullable
    double* part;            // [2 * nitems]: sum over the item's rows of n(r), e(r)
    int* status;
    int ldv;
};

constexpr int kPassNT = 256;
constexpr int kPassIC = 32;                   // steps per staged chunk
constexpr int kPassMaxRows = 256;             // rows per pass item at most

// Row groups of the pass kernel: thread = (pole, group), each group RR rows.
__host__ __device__ inline int pass_groups(int P, int RR) {
    const int g = kPassNT / P, cap = kPassMaxRows / RR;
    return g < cap ? g : cap;
}

inline size_t pass_smem_bytes(int elem, int P, int RR, int ldv) {
    const int RB = pass_groups(P, RR) * RR;
    return sizeof(double2) * (size_t)RB * P + (size_t)elem * (2 * (size_t)ldv + 2 * (size_t)kPassIC * RB);
}

// Unevaluated pairs of floats (hi + lo): the row sums of the FP32 pass and its pole
// weighting, with the rounding errors kept (Knuth's TwoSum, FMA-exact products), so that no
// FP64 arithmetic runs per item (GB300's FP64 rate is 1/64 of FP32).
__device__ __forceinline__ void df_add(float& hi, float& lo, float x) {
    const float s = hi + x;
    const float bp = s - hi;
    lo += (hi - (s - bp)) + (x - bp);
    hi = s;
}
__device__ __forceinline__ void df_mul(float ah, float al, float bh, float bl, float& ph, float& pl) {
    ph = ah * bh;
    pl = fmaf(ah, bh, -ph);
    pl = fmaf(ah, bl, pl);
    pl = fmaf(al, bh, pl);
}
// Re((ar + i ai)(qr + i qi)) as a pair
__device__ __forceinline__ void df_cre(const float4& a, float qrh, float qrl, float qih, float qil, float& h,
                                       float& l) {
    float p1h, p1l, p2h, p2l;
    df_mul(a.x, a.y, qrh, qrl, p1h, p1l);
    df_mul(a.z, a.w, qih, qil, p2h, p2l);
    h = p1h;
    l = p1l;
    df_add(h, l, -p2h);
    l -= p2l;
}
__device__ __forceinline__ float4 df_split(double2 a) {
    const float rh = (float)a.x, ih = (float)a.y;
    return make_float4(rh, (float)(a.x - (double)rh), ih, (float)(a.y - (double)ih));
}

// 1 / x correctly rounded (the value of R(1) / x)
__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }

template <class R, int NT, int RR>
__global__ void __launch_bounds__(NT) tri_pass_kernel(TriPassParams<R> p) {
    using C = typename Cplx<R>::T;
    constexpr int IC = kPassIC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int P = p.P;
    const int G = pass_groups(P, RR);              // row groups
    const int RB = G * RR;                         // rows per item
    constexpr bool kDF = sizeof(R) == 4;           // FP32 path: float pairs for the sums
    // [RB][P] weighted quadratic forms: (n, e) as double2, or (n_hi, n_lo, e_hi, e_lo)
    double2* const red = reinterpret_cast<double2*>(smem_raw);
    float4* const redf = reinterpret_cast<float4*>(smem_raw);
    R* const ds = reinterpret_cast<R*>(red + (size_t)RB * P);         // [ldv]
    R* const es = ds + p.ldv;                                         // [ldv]
    R* const yb = es + p.ldv;                                         // [2][IC][RB]
    __shared__ double sred[NT / 32];
    __shared__ int item_sh;
    const int tid = threadIdx.x;
    const int k = tid % P, g = tid / P;
    const bool on = g < G;
    float4 wsp = make_float4(0.f, 0.f, 0.f, 0.f), wzsp = wsp;      // w_k, w_k z_k split (FP32 path)
    if (kDF && on) {
        wsp = df_split(p.wq[k]);
        wzsp = df_split(p.wzq[k]);
    }

    for (;;) {
        if (tid == 0) item_sh = atomicAdd(p.counter, 1);
        __syncthreads();
        const int it = item_sh;
        if (it >= p.nitems) return;
        const int4 item = p.items[it];
        const int w = item.x, r0 = item.y, nr = item.z;
        const int n = p.n_w[w], m = p.m_w[w];
        if (n > p.ldv || nr > RB) {
            if (tid == 0) atomicOr(p.status, ST_BAD_SHAPE);
            __syncthreads();
            continue;
        }
        const R* Yw = p.Y + p.offF[w] + r0;
        for (int i = tid; i < n; i += NT) {
            ds[i] = p.d[p.offN[w] + i];
            es[i] = i < n - 1 ? p.e[p.offN[w] + i] : R(0);
        }
        // rows [r0, r0 + nr) of the window; steps i staged by chunks of IC
        auto stage = [&](int c, int buf) {
            R* dst = yb + (size_t)buf * IC * RB;
            for (int idx = tid; idx < IC * RB; idx += NT) {
                const int ic = idx / RB, row = idx % RB;
                const int i = c * IC + ic;
                if (row < nr && i < n) cp_async4(dst + idx, Yw + row + (long long)i * m);
                else dst[idx] = R(0);
            }
            cp_commit();
        };
        const int nch = (n + IC - 1) / IC;
        stage(0, 0);

        const C z = p.shifts[k < P ? k : 0];
        C gp = C{R(0), R(0)};                       // 1 / D_{i-1}
        C uc[RR], pr[RR];                           // FP64 path
        float2 ucr[RR / 2], uci[RR / 2], prr[RR / 2], pri[RR / 2];      // FP32 path: rows in pairs
#pragma unroll
        for (int u = 0; u < RR / 2; ++u) ucr[u] = uci[u] = prr[u] = pri[u] = make_float2(0.f, 0.f);
        double2 acc[RR];                            // FP64 path: row sums
        float4 accf[RR];                            // FP32 path: (re_hi, re_lo, im_hi, im_lo)
#pragma unroll
        for (int u = 0; u < RR; ++u) {
            uc[u] = C{R(0), R(0)};
            pr[u] = C{R(0), R(0)};
            acc[u] = make_double2(0.0, 0.0);
            accf[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int c = 0; c < nch; ++c) {
            if (c + 1 < nch) {
                stage(c + 1, (c + 1) & 1);
                cp_wait<1>();
            } else {
                cp_wait<0>();
            }
            __syncthreads();                          // chunk c (and d, e) visible
            const R* yc = yb + (size_t)(c & 1) * IC * RB + g * RR;
            const int i0 = c * IC, i1 = min(n, i0 + IC);
            if (on) {
                for (int i = i0; i < i1; ++i) {
                    const R di = ds[i];
                    C t, D;
                    if (i == 0) {
                        t = C{R(0), R(0)};
                        D = C{z.x - di, z.y};
                    } else {
                        const R ei = es[i - 1];
                        t = C{ei * gp.x, ei * gp.y};
                        D = C{z.x - di - ei * t.x, z.y - ei * t.y};
                    }
                    const R inv = rcp_rn(D.x * D.x + D.y * D.y);
                    gp = C{D.x * inv, -D.y * inv};
                    // u^2 / D = (ur^2 - ui^2 + 2i ur ui) gp: the factor 2 (exact in binary) is
                    // carried by the pole's g2 = 2 gp, so each row takes one product ur ui
                    const C g2 = C{R(2) * gp.x, R(2) * gp.y};
                    const R* yi = yc + (size_t)(i - i0) * RB;
                    // the group's RR staged values of step i as 16-byte vectors (the chunk, the
                    // group offset g RR and the step stride RB are multiples of 16 bytes)
                    R yv[RR];
                    if constexpr (sizeof(R) == 4 && RR % 4 == 0) {
#pragma unroll
                        for (int q4 = 0; q4 < RR / 4; ++q4) {
                            const float4 v = reinterpret_cast<const float4*>(yi)[q4];
                            yv[4 * q4] = v.x;
                            yv[4 * q4 + 1] = v.y;
                            yv[4 * q4 + 2] = v.z;
                            yv[4 * q4 + 3] = v.w;
                        }
                    } else if constexpr (sizeof(R) == 8 && RR % 2 == 0) {
#pragma unroll
                        for (int q2 = 0; q2 < RR / 2; ++q2) {
                            const double2 v = reinterpret_cast<const double2*>(yi)[q2];
                            yv[2 * q2] = v.x;
                            yv[2 * q2 + 1] = v.y;
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < RR; ++u) yv[u] = yi[u];
                    }
                    if constexpr (kDF) {
                        // rows in pairs (FFMA2: the kernel is bound by issue, 69 % of the slots against 53 %
                        // of the FMA pipe); the same operations, bit for bit.  1024 windows 1.85 -> 1.59 ms
                        const float2 tx = make_float2(t.x, t.x), ty = make_float2(t.y, t.y), nty = make_float2(-t.y, -t.y);
                        const float2 gx = make_float2(gp.x, gp.x), gy = make_float2(gp.y, gp.y);
                        const float2 hx = make_float2(g2.x, g2.x), nhy = make_float2(-g2.y, -g2.y);
#pragma unroll
                        for (int u = 0; u < RR / 2; ++u) {
                            const float2 y = make_float2(yv[2 * u], yv[2 * u + 1]);
                            const float2 ur = __ffma2_rn(tx, ucr[u], __ffma2_rn(nty, uci[u], y));
                            const float2 ui = __ffma2_rn(tx, uci[u], __fmul2_rn(ty, ucr[u]));
                            ucr[u] = ur;
                            uci[u] = ui;
                            const float2 nui = make_float2(-ui.x, -ui.y);
                            const float2 sr = __ffma2_rn(ur, ur, __fmul2_rn(nui, ui));
                            const float2 q = __fmul2_rn(ur, ui);
                            prr[u] = __ffma2_rn(sr, gx, __ffma2_rn(q, nhy, prr[u]));
                            pri[u] = __ffma2_rn(sr, gy, __ffma2_rn(q, hx, pri[u]));
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < RR; ++u) {
                            const R y = yv[u];
                            const R ur = fma(t.x, uc[u].x, fma(-t.y, uc[u].y, y));
                            const R ui = fma(t.x, uc[u].y, t.y * uc[u].x);
                            uc[u] = C{ur, ui};
                            const R sr = fma(ur, ur, -ui * ui);
                            const R q = ur * ui;
                            pr[u].x = fma(sr, gp.x, fma(-q, g2.y, pr[u].x));
                            pr[u].y = fma(sr, gp.y, fma(q, g2.x, pr[u].y));
                        }
                    }
                }
                // each chunk's sum is formed from zero and added to the row sums
#pragma unroll
                for (int u = 0; u < RR; ++u) {
                    if constexpr (kDF) {
                        df_add(accf[u].x, accf[u].y, u & 1 ? prr[u / 2].y : prr[u / 2].x);
                        df_add(accf[u].z, accf[u].w, u & 1 ? pri[u / 2].y : pri[u / 2].x);
                    } else {
                        acc[u].x += (double)pr[u].x;
                        acc[u].y += (double)pr[u].y;
                    }
                    pr[u] = C{R(0), R(0)};
                }
#pragma unroll
                for (int u = 0; u < RR / 2; ++u) prr[u] = pri[u] = make_float2(0.f, 0.f);
            }
            __syncthreads();                          // buffer c & 1 is free for chunk c + 2
        }
        // pole sums: n(r) = 4 Re sum_k w_k d_k(r), e(r) = 4 Re sum_k w_k z_k d_k(r)
        if (on) {
            if constexpr (kDF) {
#pragma unroll
                for (int u = 0; u < RR; ++u) {
                    float nh, nl, eh, el;
                    df_cre(wsp, accf[u].x, accf[u].y, accf[u].z, accf[u].w, nh, nl);
                    df_cre(wzsp, accf[u].x, accf[u].y, accf[u].z, accf[u].w, eh, el);
                    redf[(size_t)(g * RR + u) * P + k] = make_float4(nh, nl, eh, el);
                }
            } else {
                const double2 a = p.wq[k], b = p.wzq[k];
#pragma unroll
                for (int u = 0; u < RR; ++u) {
                    const double qx = acc[u].x, qy = acc[u].y;
                    red[(size_t)(g * RR + u) * P + k] = make_double2(a.x * qx - a.y * qy, b.x * qx - b.y * qy);
                }
            }
        }
        __syncthreads();
        double tn = 0.0, te = 0.0;
        for (int row = tid; row < nr; row += NT) {
            double sn = 0.0, se = 0.0;
            if constexpr (kDF) {
                float nh = 0.f, nl = 0.f, eh = 0.f, el = 0.f;
                for (int kk = 0; kk < P; ++kk) {
                    const float4 v = redf[(size_t)row * P + kk];
                    df_add(nh, nl, v.x);
                    nl += v.y;
                    df_add(eh, el, v.z);
                    el += v.w;
                }
                sn = (double)nh + (double)nl;
                se = (double)eh + (double)el;
            } else {
                for (int kk = 0; kk < P; ++kk) {
                    const double2 v = red[(size_t)row * P + kk];
                    sn += v.x;
                    se += v.y;
                }
            }
            const double nrow = 4.0 * sn, erow = 4.0 * se;
            if (!isfinite(nrow) || !isfinite(erow)) atomicOr(p.status, ST_ZERO_PIVOT);
            if (p.dens) p.dens[p.Oflat[p.offQ[w] + r0 + row]] = nrow;
            tn += nrow;
            te += erow;
        }
        tn = block_sum<NT>(tn, sred);
        te = block_sum<NT>(te, sred);
        if (tid == 0) {
            p.part[2 * (size_t)it] = tn;
            p.part[2 * (size_t)it + 1] = te;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// electron count and band energy without rows (FP64): tr((z_k - T)^-1 K), K = Y^T Y
// ---------------------------------------------------------------------------
//
// A trial of the chemical potential needs N and E_band only, and those depend on the rows through
// K (n x n, formed once per Hamiltonian).  The upper triangle of G = (z - T)^-1 is
// G_ij = G_jj t_{i+1} ... t_j (t_i = e_{i-1} / D_{i-1}), so
//
//     tr(G K) = sum_j G_jj (K_jj + 2 h_j),  h_j = sum_{i<j} K_ij t_{i+1} ... t_j.
//
// By blocks of 32 rows: with L_i = t_{i+1} ... t_e, e the end of i's block, h_j grows by sum_i K_ij L_i
// per block (2 FP64 multiply-adds per pole, i and j) and takes the factor of the whole block (L of its first
// row) from one to the next; Horner in i (5) is left for the diagonal blocks.  1.2 n^2 FP64 instructions a
// pole against the 11 m n of the rows.  The FP64 pipe bounds it: 54 windows of 276-300 functions (256
// rows) 4.7 -> 0.61 ms per trial (0.95 ms by Horner alone).

// 1 / x: from the FP32 reciprocal by one third-order step (y (1 + e + e^2), e = 1 - x y), by the
// division outside its range.
__device__ __forceinline__ double recip_f64(double x) {
    if (x > 1e-30 && x < 1e30) {
        const double y = (double)(1.0f / (float)x);
        const double e = fma(-x, y, 1.0);
        return fma(y * e, 1.0 + e, y);
    }
    return 1.0 / x;
}

constexpr int kSemi = 32;                      // rows of a block of G

// The products L_i behind the (t, G) pairs.
__device__ __forceinline__ const double2* semi_products(const double4* coef, int nitems, int ld) {
    return reinterpret_cast<const double2*>(coef + (size_t)nitems * ld);
}

// Per (window, pole): coef[item * ld + i] = (t_i, G_ii), G_ii = 1 / D_i + t_{i+1}^2 G_{i+1,i+1}, and the
// products L_i = t_{i+1} ... t_e to the end e of i's block.  Two serial chains of n steps, bound by their
// latency and the issue of FP64 instructions (27 a step, 80 clocks each on a quarter of an SM: a form with one reciprocal
// per two steps, 32 instructions for 28, measured 8 % slower); the second reads what the first stored four
// steps ahead.
__global__ void tri_diag_kernel(int nwin, int P, const int* n_w, const long long* offN, const double* __restrict__ d,
                                const double* __restrict__ e, const double2* z, int ld, double4* coef) {
    const int it = blockIdx.x * blockDim.x + threadIdx.x;
    if (it >= nwin * P) return;
    const int w = it / P;
    const double2 zk = z[it - w * P];
    const int n = n_w[w];
    const double *dw = d + offN[w], *ew = e + offN[w];
    double4* out = coef + (size_t)it * ld;
    double2 t = make_double2(0.0, 0.0), g = t;
    double el = 0.0;                                                 // e_{i-1}
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
        t = make_double2(el * g.x, el * g.y);
        const double2 D = make_double2(fma(-el, t.x, zk.x - dw[i]), fma(-el, t.y, zk.y));
        const double inv = recip_f64(D.x * D.x + D.y * D.y);
        g = make_double2(D.x * inv, -D.y * inv);
        out[i] = make_double4(t.x, t.y, g.x, g.y);
        el = ew[i];
    }
    double2* const Lo = reinterpret_cast<double2*>(coef + (size_t)nwin * P * ld) + (size_t)it * ld;
    double2 G = make_double2(0.0, 0.0), L = G;
    double2 tn = make_double2(0.0, 0.0);                             // t_{i+1}
    for (int i1 = n - 1; i1 >= 0; i1 -= 4) {
        double4 c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = out[max(i1 - u, 0)];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (i1 - u < 0) break;
            const double2 t2 = make_double2(tn.x * tn.x - tn.y * tn.y, 2.0 * tn.x * tn.y);
            G = make_double2(fma(t2.x, G.x, fma(-t2.y, G.y, c[u].z)), fma(t2.x, G.y, fma(t2.y, G.x, c[u].w)));
            const bool last = (i1 - u) % kSemi == kSemi - 1;
            L = last ? tn : make_double2(fma(tn.x, L.x, -tn.y * L.y), fma(tn.x, L.y, tn.y * L.x));
            Lo[i1 - u] = L;
            tn = make_double2(c[u].x, c[u].y);
            reinterpret_cast<double2*>(out + i1 - u)[1] = G;
        }
    }
}

constexpr int kCountNT = 320;

// One CTA per (window, kCountPoles poles), thread = column j; the lanes of a warp run over the same i, so that
// K is read along its rows and t or L is one broadcast.  A warp's columns lie in one block.
template <int kCountPoles>
__global__ void __launch_bounds__(kCountNT) tri_count_kernel(int P, int groups, const int* n_w, const long long* offC,
                                                             const double* K, const double4* coef, int ld,
                                                             double2* trace) {
    static_assert(kSemi == 32 && kCountNT % 32 == 0, "a warp's columns lie in one block");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* const ts = reinterpret_cast<double2*>(smem_raw);       // [n][kCountPoles]
    __shared__ double red[kCountNT / 32];
    const int w = blockIdx.x / groups, k0 = (blockIdx.x % groups) * kCountPoles;
    const int n = n_w[w], tid = threadIdx.x;
    const double* const Kw = K + offC[w];
    const double4* const cf = coef + ((size_t)w * P + k0) * ld;
    const int np = min(kCountPoles, P - k0);
    for (int idx = tid; idx < n * kCountPoles; idx += kCountNT) {
        const int q = idx / n, i = idx - q * n;
        const double4 c = q < np ? cf[(size_t)q * ld + i] : make_double4(0.0, 0.0, 0.0, 0.0);
        ts[i * kCountPoles + q] = make_double2(c.x, c.y);
    }
    __syncthreads();
    const double2* Lq[kCountPoles];
    const int nitems = (int)(gridDim.x / groups) * P;
    double2 acc[kCountPoles];
#pragma unroll
    for (int q = 0; q < kCountPoles; ++q) {
        Lq[q] = semi_products(coef, nitems, ld) + ((size_t)w * P + min(k0 + q, P - 1)) * ld;
        acc[q] = make_double2(0.0, 0.0);
    }
    for (int j = tid; j < n; j += kCountNT) {
        double2 h[kCountPoles];
#pragma unroll
        for (int q = 0; q < kCountPoles; ++q) h[q] = make_double2(0.0, 0.0);
        const int jb = j / kSemi * kSemi;
        for (int i0 = 0; i0 < jb; i0 += kSemi) {
            if (i0) {
#pragma unroll
                for (int q = 0; q < kCountPoles; ++q) {
                    const double2 f = Lq[q][i0];
                    h[q] = make_double2(fma(f.x, h[q].x, -f.y * h[q].y), fma(f.x, h[q].y, f.y * h[q].x));
                }
            }
#pragma unroll 4
            for (int i = i0; i < i0 + kSemi; ++i) {
                const double x = Kw[j + (long long)i * n];
#pragma unroll
                for (int q = 0; q < kCountPoles; ++q) {
                    const double2 f = Lq[q][i];
                    h[q] = make_double2(fma(x, f.x, h[q].x), fma(x, f.y, h[q].y));
                }
            }
        }
#pragma unroll 4
        for (int i = jb; i < j; ++i) {
            const double x = Kw[j + (long long)i * n];
#pragma unroll
            for (int q = 0; q < kCountPoles; ++q) {
                const double2 t = ts[(i + 1) * kCountPoles + q];
                const double u = h[q].x + x;
                h[q] = make_double2(fma(t.x, u, -t.y * h[q].y), fma(t.y, u, t.x * h[q].y));
            }
        }
        const double kjj = Kw[j + (long long)j * n];
#pragma unroll
        for (int q = 0; q < kCountPoles; ++q) {
            if (q >= np) break;
            const double4 c = cf[(size_t)q * ld + j];
            const double u = fma(2.0, h[q].x, kjj), v = 2.0 * h[q].y;
            acc[q].x += c.z * u - c.w * v;
            acc[q].y += c.z * v + c.w * u;
        }
    }
#pragma unroll
    for (int q = 0; q < kCountPoles; ++q) {
        const double x = block_sum<kCountNT>(acc[q].x, red), y = block_sum<kCountNT>(acc[q].y, red);
        if (tid == 0 && q < np) trace[(size_t)w * P + k0 + q] = make_double2(x, y);
    }
}

// tr(G_k K G_k) = -d/dz tr(G_k K) of every (window, pole): the sums above with their derivatives in z, from
// t', G' (dcoef) and L' behind them.  FP64, for the derivatives of N and E_band in the chemical potential, which
// are small differences of large sums: from the FP32 sweeps of the mixed adjoint they carry an error of 1e-6 of
// N, whatever their size.
constexpr int kSlopePoles = 2;

// (t'_i, G'_ii) and L'_i from (t_i, G_ii) and L_i: D' = 1 - e t', (1 / D)' = -D' / D^2.
__global__ void tri_slope_diag_kernel(int nwin, int P, const int* n_w, const long long* offN, const double* __restrict__ d,
                                      const double* __restrict__ e, const double2* z, int ld, const double4* coef,
                                      double4* dcoef) {
    const int it = blockIdx.x * blockDim.x + threadIdx.x;
    if (it >= nwin * P) return;
    const int w = it / P, n = n_w[w];
    const double2 zk = z[it - w * P];
    const double *dw = d + offN[w], *ew = e + offN[w];
    const double4* const in = coef + (size_t)it * ld;
    const double2* const L = semi_products(coef, nwin * P, ld) + (size_t)it * ld;
    double4* const out = dcoef + (size_t)it * ld;
    double2* const Ld = reinterpret_cast<double2*>(dcoef + (size_t)nwin * P * ld) + (size_t)it * ld;
    auto mul = [](double2 a, double2 b) { return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x)); };
    double2 td = make_double2(0.0, 0.0), gd = td;
    double el = 0.0;                                                 // e_{i-1}
    for (int i = 0; i < n; ++i) {
        const double2 t = make_double2(in[i].x, in[i].y);
        td = make_double2(el * gd.x, el * gd.y);
        const double2 D = make_double2(fma(-el, t.x, zk.x - dw[i]), fma(-el, t.y, zk.y));
        const double inv = recip_f64(D.x * D.x + D.y * D.y);
        const double2 g = make_double2(D.x * inv, -D.y * inv);
        const double2 g2 = mul(g, g), Dd = make_double2(fma(-el, td.x, 1.0), -el * td.y);
        gd = mul(make_double2(-g2.x, -g2.y), Dd);
        out[i] = make_double4(td.x, td.y, gd.x, gd.y);
        el = ew[i];
    }
    double2 G = make_double2(0.0, 0.0), Gd = G, tn = G, tnd = G, Lp = G, Lc = G;     // of i + 1; L', L
    for (int i = n - 1; i >= 0; --i) {
        const double4 c = in[i], o = out[i];
        const double2 t2 = mul(tn, tn), x = mul(mul(make_double2(2.0 * tn.x, 2.0 * tn.y), tnd), G), y = mul(t2, Gd);
        Gd = make_double2(o.z + x.x + y.x, o.w + x.y + y.y);
        G = make_double2(c.z, c.w);
        if (i % kSemi == kSemi - 1) {
            Lp = tnd;
        } else {
            const double2 a = mul(tn, Lp), b = mul(tnd, Lc);
            Lp = make_double2(a.x + b.x, a.y + b.y);
        }
        Lc = L[i];
        Ld[i] = Lp;
        tn = make_double2(c.x, c.y);
        tnd = make_double2(o.x, o.y);
        out[i] = make_double4(o.x, o.y, Gd.x, Gd.y);
    }
}

__global__ void __launch_bounds__(kCountNT) tri_slope_kernel(int P, int groups, const int* n_w, const long long* offC,
                                                             const double* K, const double4* coef, const double4* dcoef,
                                                             int ld, double2* slope) {
    __shared__ double red[kCountNT / 32];
    const int w = blockIdx.x / groups, k0 = (blockIdx.x % groups) * kSlopePoles;
    const int n = n_w[w], tid = threadIdx.x, nitems = (int)(gridDim.x / groups) * P;
    const double* const Kw = K + offC[w];
    auto mul = [](double2 a, double2 b) { return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x)); };
    for (int q = 0; q < kSlopePoles && k0 + q < P; ++q) {
        const size_t it = ((size_t)w * P + k0 + q) * ld;
        const double4 *cf = coef + it, *cd = dcoef + it;
        const double2 *L = semi_products(coef, nitems, ld) + it, *Ld = semi_products(dcoef, nitems, ld) + it;
        double2 acc = make_double2(0.0, 0.0);
        for (int j = tid; j < n; j += kCountNT) {
            double2 h = make_double2(0.0, 0.0), hd = h;
            const int jb = j / kSemi * kSemi;
            for (int i0 = 0; i0 < jb; i0 += kSemi) {
                if (i0) {
                    const double2 f = L[i0], fd = Ld[i0], a = mul(hd, f), b = mul(h, fd);
                    hd = make_double2(a.x + b.x, a.y + b.y);
                    h = mul(h, f);
                }
#pragma unroll 8
                for (int i = i0; i < i0 + kSemi; ++i) {
                    const double x = Kw[j + (long long)i * n];
                    const double2 f = L[i], fd = Ld[i];
                    h = make_double2(fma(x, f.x, h.x), fma(x, f.y, h.y));
                    hd = make_double2(fma(x, fd.x, hd.x), fma(x, fd.y, hd.y));
                }
            }
#pragma unroll 4
            for (int i = jb; i < j; ++i) {
                const double4 t4 = cf[i + 1], d4 = cd[i + 1];
                const double2 t = make_double2(t4.x, t4.y), td = make_double2(d4.x, d4.y);
                const double2 u = make_double2(h.x + Kw[j + (long long)i * n], h.y), a = mul(hd, t), b = mul(u, td);
                hd = make_double2(a.x + b.x, a.y + b.y);
                h = mul(u, t);
            }
            const double2 u = make_double2(fma(2.0, h.x, Kw[j + (long long)j * n]), 2.0 * h.y);
            const double2 a = mul(make_double2(cd[j].z, cd[j].w), u);
            const double2 b = mul(make_double2(cf[j].z, cf[j].w), make_double2(2.0 * hd.x, 2.0 * hd.y));
            acc = make_double2(acc.x + a.x + b.x, acc.y + a.y + b.y);
        }
        const double x = block_sum<kCountNT>(acc.x, red), y = block_sum<kCountNT>(acc.y, red);
        if (tid == 0) slope[(size_t)w * P + k0 + q] = make_double2(-x, -y);
    }
}

// u[c * nwin + w] = Re sum_k c_k tr(G_k K G_k), poles in order
__global__ void tri_slope_sums_kernel(int nwin, int P, const double2* slope, const double2* cw, double* u) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nwin) return;
    for (int c = 0; c < 3; ++c) {
        double s = 0.0;
        for (int k = 0; k < P; ++k) {
            const double2 x = slope[(size_t)w * P + k], a = cw[c * P + k];
            s += a.x * x.x - a.y * x.y;
        }
        u[(size_t)c * nwin + w] = s;
    }
}

// per-window N and E_band from the traces, poles in order
__global__ void tri_count_sums_kernel(int nwin, int P, const double2* trace, const double2* wq, const double2* wzq,
                                      double dV, double* nw, double* ew, int* status) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nwin) return;
    double sn = 0.0, se = 0.0;
    for (int k = 0; k < P; ++k) {
        const double2 x = trace[(size_t)w * P + k], a = wq[k], b = wzq[k];
        sn += a.x * x.x - a.y * x.y;
        se += b.x * x.x - b.y * x.y;
    }
    if (!isfinite(sn) || !isfinite(se)) atomicOr(status, ST_ZERO_PIVOT);
    nw[w] = 4.0 * sn * dV;
    ew[w] = 4.0 * se * dV;
}

// ---------------------------------------------------------------------------
// density pass through the pole-weighted matrix (FP64)
// ---------------------------------------------------------------------------
//
// n(r) = 4 y_r P y_r^T and, since Re sum_k w_k = 0, e(r) = 4 y_r T P y_r^T with P = Re sum_k w_k G_k (n x n,
// real).  P costs 1.2 n^2 FP64 instructions a pole instead of the rows' 11 m n, and V = Y P is a
// dense product for the tensor cores (oz_gemm.cu); what is left per row is two inner products.
// Measured: 54 windows of 276-300 functions and 256 rows 4.7 -> 1.6 ms, 432 windows 29.4 ->
// 8.0 ms.

constexpr int kPmatWarps = 4, kPmatPoles = 8;

// One CTA per (window, 32 columns), lane = column j, the poles dealt to the warps.  In the diagonal block row
// by row up, G_ij = G_{i+1,j} t_{i+1} (5 FP64 instructions per pole, row and column); above it
// G_ij = L_i s_j with s_j = t_{e+1} ... t_j G_jj carried from block to block (2; with 5 throughout: 54 windows
// 2.39 ms, 432 windows 11.1 ms a pass).  The warps' sums of 32 rows are joined in shared memory and
// written with their mirror image.
__global__ void __launch_bounds__(32 * kPmatWarps) tri_pmat_kernel(int P, const int* n_w, const long long* offC,
                                                                   const double4* coef, int ld, const double2* wq,
                                                                   double* Pm) {
    __shared__ double part[kPmatWarps][32][33];
    const int w = blockIdx.y, n = n_w[w];
    const int b = blockIdx.x;
    if (32 * b >= n) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = 32 * b + lane;
    double* const Pw = Pm + offC[w];
    static_assert(kSemi == 32, "a CTA's columns are a block");
    const double4* const cw = coef + (size_t)w * P * ld;
    const double2* const lw = semi_products(coef, (int)gridDim.y * P, ld) + (size_t)w * P * ld;
    for (int k0 = 0; k0 < P; k0 += kPmatWarps * kPmatPoles) {
        const double4* cf[kPmatPoles];                              // this warp's poles
        const double2* lf[kPmatPoles];
        double2 s[kPmatPoles], init[kPmatPoles];
#pragma unroll
        for (int q = 0; q < kPmatPoles; ++q) {
            const int k = k0 + warp + q * kPmatWarps;
            cf[q] = cw + (size_t)min(k, P - 1) * ld;
            lf[q] = lw + (size_t)min(k, P - 1) * ld;
            init[q] = s[q] = make_double2(0.0, 0.0);
            if (k < P && j < n) {
                const double4 g = cf[q][j];
                const double2 wk = wq[k];
                init[q] = make_double2(wk.x * g.z - wk.y * g.w, wk.x * g.w + wk.y * g.z);
            }
        }
        for (int ib = b; ib >= 0; --ib) {
            if (ib < b) {
#pragma unroll 4
                for (int r = 0; r < 32; ++r) {
                    double s0 = 0.0, s1 = 0.0;
#pragma unroll
                    for (int q = 0; q < kPmatPoles; ++q) {
                        const double2 f = lf[q][32 * ib + r];
                        s0 = fma(f.x, s[q].x, s0);
                        s1 = fma(f.y, s[q].y, s1);
                    }
                    part[warp][r][lane] = s0 - s1;
                }
#pragma unroll
                for (int q = 0; q < kPmatPoles; ++q) {
                    const double2 f = lf[q][32 * ib];
                    s[q] = make_double2(fma(f.x, s[q].x, -f.y * s[q].y), fma(f.x, s[q].y, f.y * s[q].x));
                }
            } else {
#pragma unroll 2
                for (int r = 31; r >= 0; --r) {
                    const int i = 32 * ib + r;
                    if (i >= n) continue;                           // (the same for every lane)
                    double sum = 0.0;
#pragma unroll
                    for (int q = 0; q < kPmatPoles; ++q) {
                        if (i == j) s[q] = init[q];
                        sum += s[q].x;
                        if (r == 0) continue;                       // (s stays G_ij of the block's first row)
                        const double2 t = *reinterpret_cast<const double2*>(cf[q] + i);
                        s[q] = make_double2(fma(t.x, s[q].x, -t.y * s[q].y), fma(t.x, s[q].y, t.y * s[q].x));
                    }
                    part[warp][r][lane] = sum;                      // (zero below the diagonal: s is zero there)
                }
            }
            __syncthreads();
            for (int r = warp; r < 32; r += kPmatWarps) {
                const int i = 32 * ib + r;
                if (i < n && j < n && i <= j) {
                    double x = part[0][r][lane];
#pragma unroll
                    for (int q = 1; q < kPmatWarps; ++q) x += part[q][r][lane];
                    if (k0) x += Pw[j + (long long)i * n];
                    Pw[j + (long long)i * n] = x;
                    part[0][r][lane] = x;
                }
            }
            __syncthreads();
            for (int c = warp; c < 32; c += kPmatWarps) {           // column 32 b + c, rows along the lanes
                const int i = 32 * ib + lane, jc = 32 * b + c;
                if (jc < n && i < jc) Pw[i + (long long)jc * n] = part[0][lane][c];
            }
            __syncthreads();
        }
    }
}

// n(r) and e(r) of an item's rows from V = Y P, sums of the item; rows along the lanes, the columns
// split over the warps.
__global__ void __launch_bounds__(128) tri_rowdot_kernel(int w0, const int4* items, const int* first, const int* count,
                                                         const int* n_w, const int* m_w, const long long* offN,
                                                         const long long* offF, const long long* offV,
                                                         const long long* offQ, const long long* Oflat, const double* Y,
                                                         const double* V, const double* d, const double* e, double* dens,
                                                         double* part, int* status) {
    __shared__ double sn[4][32], se[4][32];
    if ((int)blockIdx.x >= count[w0 + blockIdx.y]) return;
    const int it = first[w0 + blockIdx.y] + blockIdx.x;
    const int4 item = items[it];
    const int w = item.x, r0 = item.y, nr = item.z;
    const int n = n_w[w], m = m_w[w];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double *dw = d + offN[w], *ew = e + offN[w];
    double tn = 0.0, te = 0.0;                                      // (warp 0: sums of the item)
    for (int rb = 0; rb < nr; rb += 32) {
        double an = 0.0, ae = 0.0;
        if (rb + lane < nr) {
            const double* const y = Y + offF[w] + r0 + rb + lane;
            const double* const v = V + offV[w] + r0 + rb + lane;
            const int j0 = n * warp / 4, j1 = n * (warp + 1) / 4;
            double yp = j0 > 0 ? y[(long long)(j0 - 1) * m] : 0.0, yc = j0 < n ? y[(long long)j0 * m] : 0.0;
            for (int j = j0; j < j1; ++j) {
                const double yn = j + 1 < n ? y[(long long)(j + 1) * m] : 0.0;
                const double x = v[(long long)j * m];
                const double ty = fma(dw[j], yc, fma(j > 0 ? ew[j - 1] : 0.0, yp, (j + 1 < n ? ew[j] : 0.0) * yn));
                an = fma(x, yc, an);
                ae = fma(x, ty, ae);
                yp = yc;
                yc = yn;
            }
        }
        __syncthreads();
        sn[warp][lane] = an;
        se[warp][lane] = ae;
        __syncthreads();
        if (warp == 0) {
            const double nrow = 4.0 * ((sn[0][lane] + sn[1][lane]) + (sn[2][lane] + sn[3][lane]));
            const double erow = 4.0 * ((se[0][lane] + se[1][lane]) + (se[2][lane] + se[3][lane]));
            if (rb + lane < nr) {
                if (!isfinite(nrow) || !isfinite(erow)) atomicOr(status, ST_ZERO_PIVOT);
                if (dens) dens[Oflat[offQ[w] + r0 + rb + lane]] = nrow;
            }
            tn += warp_sum(nrow);
            te += warp_sum(erow);
        }
    }
    if (threadIdx.x == 0) {
        part[2 * (size_t)it] = tn;
        part[2 * (size_t)it + 1] = te;
    }
}

// per-window totals from the items of each window (contiguous, fixed order)
__global__ void tri_window_sums_kernel(int nwin, const int* first, const int* count, const double* part, double dV,
                                       double* nw, double* ew) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nwin) return;
    double sn = 0.0, se = 0.0;
    for (int i = first[w]; i < first[w] + count[w]; ++i) {
        sn += part[2 * (size_t)i];
        se += part[2 * (size_t)i + 1];
    }
    nw[w] = sn * dV;
    ew[w] = se * dV;
}

// ---------------------------------------------------------------------------
// Sturm counts on T (FP64 arithmetic)
// ---------------------------------------------------------------------------

// Eigenvalues of the tridiagonal (d, e) below sigma = negative pivots of T - sigma I.
template <class R>
__device__ int sturm_count(int n, const R* d, const R* e, double sigma) {
    constexpr double pivmin = 1e-290;
    int cnt = 0;
    double q = (double)d[0] - sigma;
    if (fabs(q) < pivmin) q = -pivmin;
    if (q < 0.0) ++cnt;
    for (int i = 1; i < n; ++i) {
        const double ee = (double)e[i - 1];
        q = ((double)d[i] - sigma) - ee * ee / q;
        if (fabs(q) < pivmin) q = -pivmin;
        if (q < 0.0) ++cnt;
    }
    return cnt;
}

template <class R>
__global__ void tri_sturm_kernel(int nwin, const int* n_w, const long long* offN, const R* d, const R* e,
                                 double sigma, int* below) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nwin) return;
    below[w] = sturm_count(n_w[w], d + offN[w], e + offN[w], sigma);
}

// Smallest eigenvalue of every window: bisection on the Sturm count from the Gershgorin
// interval down to width tol; lam[w] = midpoint of the last bracket.
template <class R>
__global__ void tri_mineig_kernel(int nwin, const int* n_w, const long long* offN, const R* d, const R* e,
                                  double tol, double* lam) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nwin) return;
    const int n = n_w[w];
    const R* dw = d + offN[w];
    const R* ew = e + offN[w];
    double lo = 1e300, hi = -1e300;
    for (int i = 0; i < n; ++i) {
        const double r = (i > 0 ? fabs((double)ew[i - 1]) : 0.0) + (i < n - 1 ? fabs((double)ew[i]) : 0.0);
        lo = fmin(lo, (double)dw[i] - r);
        hi = fmax(hi, (double)dw[i] + r);
    }
    const double pad = 1e-12 * fmax(1.0, fmax(fabs(lo), fabs(hi)));
    double a = lo - pad, b = hi + pad;
    for (int iter = 0; iter < 200 && b - a > tol; ++iter) {
        const double mid = 0.5 * (a + b);
        if (sturm_count(n, dw, ew, mid) >= 1) b = mid;
        else a = mid;
    }
    lam[w] = 0.5 * (a + b);
}

}  // namespace

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------

// Tile configurations of the tridiagonal route: reduction panel width and threads, row
// application panel width, rows per thread of the row-per-thread application and whether
// the rows stay resident in shared memory (res; FP32 only).  Panel widths are capped by
// what fits the shared memory at windows of nmax.
struct TriCfg {
    int nb, nba, rpt, res, reg;          // reg: the reduction with the window on its SM (tridiag_reg.cu)
    int rows;                            // resident application: rows per item at most
};
// Measured at 1024 electrons (mixed): reduction 3.5 ms with the window on its SM, 6.7 ms with the
// L2-resident working copy (nb 16, 512 threads, two CTAs per SM; nb 8 6.75 ms, nb 32 7.35 ms; 256
// threads at four CTAs per SM and 384 at three 7.8 ms); row application 2.0 ms with resident rows
// (NB 32), 6.3 ms one row per thread.
static const TriCfg kTriCfg[6] = {{16, 32, 1, 1, 1, 128}, {16, 32, 1, 1, 0, 128}, {16, 32, 1, 0, 0, 0},
                                  {16, 16, 1, 1, 0, 64},  {16, 32, 1, 1, 1, 32},  {8, 32, 1, 1, 0, 128}};
constexpr int kReduceNT = 512;           // threads of the reduction (256 where FP64 CTAs go in pairs)

int tri_pick(bool fp32, int nmax, int P, size_t smem_budget, int cfg, TriPick* out) {
    if (tri_rows_per_item(fp32, P) < 1) {
        lres_set_error("the tridiagonal route takes at most %d poles (got %d)", kPassNT, P);
        return LRES_EINVAL;
    }
    const int el = fp32 ? 4 : 8;
    TriPick r;
    r.ldv = (std::max(nmax, 1) + 31) / 32 * 32;
    if (cfg < 0 || cfg >= 6) cfg = 0;
    const TriCfg& t = kTriCfg[cfg];
    r.reg = t.reg && fp32;
    // FP64: panels of 8, the pending updates cost instructions of its pipe and the L2 traffic of more frequent
    // updates does not bound it (54 windows: panels of 4, 8, 16 take 5.23, 5.19, 5.58 ms; 432 windows 20.9,
    // 20.9, 22.5 ms; one window of 96 functions 0.88, 0.91, 1.03 ms)
    const int nbmax = fp32 ? t.nb : std::min(t.nb, 8);
    for (int b : {32, 16, 8, 4})
        if (b <= nbmax && !r.nb && reduce_smem_elems(b, r.ldv, kReduceNT) * el <= smem_budget) r.nb = b;
    if (t.res && fp32)
        for (int b : {32, 16})
            for (int rows = std::min(kResRows, t.rows); rows >= 32 && !r.nb_apply; rows -= 32)
                if (b <= t.nba && res_smem_bytes(b, r.ldv, rows) <= smem_budget) {
                    r.nb_apply = b;
                    r.arows = rows;
                    r.rpt = 0;
                }
    if (!r.nb_apply) {
        for (int b : {32, 16, 8, 4})
            if (b <= t.nba && !r.nb_apply && (size_t)el * ((size_t)r.ldv * b + 2 * b * b) <= smem_budget) r.nb_apply = b;
        r.rpt = r.nb_apply >= 16 ? t.rpt : 1;
        r.arows = kAppRows;
    }
    if (!r.nb || !r.nb_apply) {
        lres_set_error("windows of %d functions exceed the shared memory of the tridiagonal reduction", nmax);
        return LRES_EINVAL;
    }
    // T factors of the resident application: panels of nb_apply, per window
    r.tstride = r.rpt == 0 ? (long long)(r.ldv / r.nb_apply + 1) * r.nb_apply * r.nb_apply : 0;
    *out = r;
    return LRES_OK;
}

template <class R, int NT>
static int launch_reduce(const TriReduceParams<R>& p, size_t smem_budget, cudaStream_t s) {
    const size_t smem = reduce_smem_elems(p.nb, p.ldv, NT) * sizeof(R);
    if (smem > smem_budget) {
        lres_set_error("tridiagonal reduction needs %zu B of shared memory", smem);
        return LRES_EINVAL;
    }
    int per_sm = 0;
    if (int rc = prepare_kernel<tri_reduce_kernel<R, NT>>(NT, smem, &per_sm)) return rc;
    const int grid = std::min(p.nwin, std::max(1, per_sm) * device_sms());
    tri_reduce_kernel<R, NT><<<grid, NT, smem, s>>>(p);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

// Two CTAs per window.
static int launch_reduce_cluster(const TriReduceParams<double>& p, cudaStream_t s) {
    constexpr int NT = kReduceNT;
    const size_t smem = reduce_smem_elems(p.nb, p.ldv, NT, 2) * sizeof(double);
    int per_sm = 0;
    if (int rc = prepare_kernel<tri_reduce_kernel<double, NT, 2>>(NT, smem, &per_sm)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)p.nwin);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    LRES_CUDA_TRY(cudaLaunchKernelEx(&cfg, tri_reduce_kernel<double, NT, 2>, p));
    return LRES_OK;
}

int tri_reduce(bool fp32, int nwin, const int* order, int* counter, const int* n_w, const long long* offC,
               const long long* offA, const long long* offN, const void* H, void* A, void* d, void* e, void* tau,
               int* status, const TriPick& pk, int nmax, size_t smem_budget, cudaStream_t s) {
    if (!nwin) return LRES_OK;
    const int nb = pk.nb, ldv = pk.ldv;
    LRES_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(int), s));
    if (fp32) {
        TriReduceParams<float> p{nwin, order, counter, n_w, offC, offA, offN, (const float*)H, (float*)A,
                                 (float*)d, (float*)e, (float*)tau, status, nb, ldv, 0};
        if (pk.reg) {
            // windows beyond the resident size: their first columns from the L2-resident copy
            if (nmax > kTriRegMax) {
                p.keep = kTriRegMax;
                if (int rc = launch_reduce<float, kReduceNT>(p, smem_budget, s)) return rc;
            }
            return tri_reduce_reg(nwin, order, counter, n_w, offC, offA, offN, (const float*)H, (float*)A, (float*)d,
                                  (float*)e, (float*)tau, status, nb, nmax, smem_budget, s);
        }
        return launch_reduce<float, kReduceNT>(p, smem_budget, s);
    }
    TriReduceParams<double> p{nwin, order, counter, n_w, offC, offA, offN, (const double*)H, (double*)A,
                              (double*)d, (double*)e, (double*)tau, status, nb, ldv, 0};
    // two CTAs per window while they find an SM each and the windows are large enough to share (the line lies
    // between 160 and 192 functions, see the kernel); else one CTA of 512 threads, or two of 256 per SM (TriPick)
    if (2 * nwin <= device_sms() && nmax >= 192 &&
        reduce_smem_elems(nb, ldv, kReduceNT, 2) * sizeof(double) <= smem_budget)
        return launch_reduce_cluster(p, s);
    if (pk.pairs && 2 * (reduce_smem_elems(nb, ldv, 256) * sizeof(double) + 1024) <= smem_budget + 1024)
        return launch_reduce<double, 256>(p, smem_budget, s);
    return launch_reduce<double, kReduceNT>(p, smem_budget, s);
}

template <class R, int NB, int RPT>
static int launch_apply(const TriApplyParams<R>& p, cudaStream_t s) {
    constexpr int NT = kAppRows / RPT;
    const size_t smem = sizeof(R) * ((size_t)p.ldv * NB + 2 * NB * NB);
    int per_sm = 0;
    if (int rc = prepare_kernel<tri_apply_kernel<R, NT, NB, RPT>>(NT, smem, &per_sm)) return rc;
    tri_apply_kernel<R, NT, NB, RPT><<<p.nitems, NT, smem, s>>>(p);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

template <class R>
static int dispatch_apply(const TriApplyParams<R>& p, int nb, int rpt, cudaStream_t s) {
    if (nb == 32 && rpt == 2) return launch_apply<R, 32, 2>(p, s);
    if (nb == 16 && rpt == 4) return launch_apply<R, 16, 4>(p, s);
    if (nb == 16 && rpt == 2) return launch_apply<R, 16, 2>(p, s);
    switch (nb) {
        case 32: return launch_apply<R, 32, 1>(p, s);
        case 16: return launch_apply<R, 16, 1>(p, s);
        case 8: return launch_apply<R, 8, 1>(p, s);
        case 4: return launch_apply<R, 4, 1>(p, s);
        default:
            lres_set_error("tridiagonal panel width %d not compiled", nb);
            return LRES_EINVAL;
    }
}

template <int NB>
static int launch_apply_res(const TriApplyParams<float>& p, const TriTParams& tp, int rows, size_t smem_budget,
                            cudaStream_t s) {
    const size_t smem_t = sizeof(float) * ((size_t)p.ldv * NB + NB * NB + std::max(NB * NB, tf_part_elems(NB)));
    const size_t smem = res_smem_bytes(NB, p.ldv, rows);
    if (smem > smem_budget || rows > kResRows || rows % 32) {
        lres_set_error("resident row application needs %zu B of shared memory", smem);
        return LRES_EINVAL;
    }
    int per_sm = 0;
    if (tp.maxp > 0 && tp.nwin > 0) {
        if (int rc = prepare_kernel<tri_gram_kernel<NB>>(128, smem_t, &per_sm)) return rc;
        tri_gram_kernel<NB><<<(unsigned)tp.nwin * tp.maxp, 128, smem_t, s>>>(tp);
        LRES_CUDA_TRY(cudaGetLastError());
        tri_tfactor_kernel<NB><<<(unsigned)tp.nwin * tp.maxp, 32, 0, s>>>(tp);
        LRES_CUDA_TRY(cudaGetLastError());
    }
    if (int rc = prepare_kernel<tri_apply_res_kernel<NB>>(kResNT, smem, &per_sm)) return rc;
    tri_apply_res_kernel<NB><<<p.nitems, kResNT, smem, s>>>(p, tp.T, tp.tstride, rows);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_apply(int nitems, const int4* items, const int* n_w, const int* m_w, const long long* offA,
              const long long* offN, const long long* offF, const float* A, const float* tau, const float* F, float* Y,
              const TriPick& pk, int nwin, bool tfactors, float* T, size_t smem_budget, cudaStream_t s) {
    if (!nitems) return LRES_OK;
    TriApplyParams<float> p{nitems, items, n_w, m_w, offA, offN, offF, A, tau, F, Y, pk.ldv};
    if (pk.rpt) return dispatch_apply(p, pk.nb_apply, pk.rpt, s);
    if (!T) {
        lres_set_error("resident row application without a T-factor buffer");
        return LRES_ESTATE;
    }
    const int maxp = tfactors ? (pk.ldv + pk.nb_apply - 1) / pk.nb_apply : 0;
    TriTParams tp{nwin, maxp, n_w, offA, offN, A, tau, T, pk.tstride, pk.ldv};
    if (pk.nb_apply == 32) return launch_apply_res<32>(p, tp, pk.arows, smem_budget, s);
    if (pk.nb_apply == 16) return launch_apply_res<16>(p, tp, pk.arows, smem_budget, s);
    lres_set_error("resident row application: panel width %d not compiled", pk.nb_apply);
    return LRES_EINVAL;
}

int tri_rows_per_item(bool fp32, int P) {
    const int RR = fp32 ? 8 : 4;
    return pass_groups(std::max(P, 1), RR) * RR;
}

template <class R, int RR>
static int launch_pass(const TriPassParams<R>& p, size_t smem_budget, cudaStream_t s) {
    const size_t smem = pass_smem_bytes(sizeof(R), p.P, RR, p.ldv);
    if (smem > smem_budget) {
        lres_set_error("pole pass needs %zu B of shared memory (P = %d, windows up to %d)", smem, p.P, p.ldv);
        return LRES_EINVAL;
    }
    int per_sm = 0;
    if (int rc = prepare_kernel<tri_pass_kernel<R, kPassNT, RR>>(kPassNT, smem, &per_sm)) return rc;
    const int grid = std::min(p.nitems, std::max(1, per_sm) * device_sms());
    tri_pass_kernel<R, kPassNT, RR><<<grid, kPassNT, smem, s>>>(p);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_pass(bool fp32, int nitems, const int4* items, int* counter, const int* n_w, const int* m_w,
             const long long* offN, const long long* offF, const long long* offQ, const long long* Oflat,
             const void* Y, const void* d, const void* e, int P, const void* shifts, const double2* wq,
             const double2* wzq, double* dens, double* part, int* status, int ldv, size_t smem_budget,
             cudaStream_t s) {
    if (!nitems) return LRES_OK;
    if (P < 1 || P > kPassNT) {
        lres_set_error("pole pass supports 1..%d poles per half plane (got %d)", kPassNT, P);
        return LRES_EINVAL;
    }
    LRES_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(int), s));
    if (fp32) {
        TriPassParams<float> p{nitems, items, counter, n_w, m_w, offN, offF, offQ, Oflat, (const float*)Y,
                               (const float*)d, (const float*)e, P, (const float2*)shifts, wq, wzq, dens, part,
                               status, ldv};
        return launch_pass<float, 8>(p, smem_budget, s);
    }
    TriPassParams<double> p{nitems, items, counter, n_w, m_w, offN, offF, offQ, Oflat, (const double*)Y,
                            (const double*)d, (const double*)e, P, (const double2*)shifts, wq, wzq, dens, part,
                            status, ldv};
    return launch_pass<double, 4>(p, smem_budget, s);
}

int tri_count(int nwin, int P, int nmax, const int* n_w, const long long* offN, const long long* offC, const double* d,
              const double* e, const double* K, const double2* shifts, const double2* wq, const double2* wzq,
              double dV, double4* coef, double2* trace, double* nw, double* ew, int* status, size_t smem_budget,
              cudaStream_t s) {
    if (!nwin) return LRES_OK;
    // four poles a CTA share the reads of K and the broadcasts; one where that leaves SMs without a CTA (one
    // window of 96 functions, 32 poles: 85 -> 35 us)
    const int np = (long long)nwin * ((P + 3) / 4) < device_sms() ? 1 : 4;
    const size_t smem = sizeof(double2) * np * (size_t)nmax;
    if (smem > smem_budget) {
        lres_set_error("count pass needs %zu B of shared memory", smem);
        return LRES_EINVAL;
    }
    tri_diag_kernel<<<(unsigned)(((long long)nwin * P + 31) / 32), 32, 0, s>>>(nwin, P, n_w, offN, d, e, shifts, nmax,
                                                                              coef);
    LRES_CUDA_TRY(cudaGetLastError());
    int per_sm = 0;
    const int groups = (P + np - 1) / np;
    if (np == 1) {
        if (int rc = prepare_kernel<tri_count_kernel<1>>(kCountNT, smem, &per_sm)) return rc;
        tri_count_kernel<1><<<(unsigned)nwin * groups, kCountNT, smem, s>>>(P, groups, n_w, offC, K, coef, nmax, trace);
    } else {
        if (int rc = prepare_kernel<tri_count_kernel<4>>(kCountNT, smem, &per_sm)) return rc;
        tri_count_kernel<4><<<(unsigned)nwin * groups, kCountNT, smem, s>>>(P, groups, n_w, offC, K, coef, nmax, trace);
    }
    LRES_CUDA_TRY(cudaGetLastError());
    tri_count_sums_kernel<<<(nwin + 63) / 64, 64, 0, s>>>(nwin, P, trace, wq, wzq, dV, nw, ew, status);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_slopes(int nwin, int P, int nmax, const int* n_w, const long long* offN, const long long* offC, const double* d,
               const double* e, const double* K, const double2* shifts, const double2* cw, const double4* coef,
               double4* dcoef, double2* slope, double* u, cudaStream_t s) {
    if (!nwin) return LRES_OK;
    tri_slope_diag_kernel<<<(unsigned)(((long long)nwin * P + 31) / 32), 32, 0, s>>>(nwin, P, n_w, offN, d, e, shifts,
                                                                                    nmax, coef, dcoef);
    LRES_CUDA_TRY(cudaGetLastError());
    const int groups = (P + kSlopePoles - 1) / kSlopePoles;
    tri_slope_kernel<<<(unsigned)nwin * groups, kCountNT, 0, s>>>(P, groups, n_w, offC, K, coef, dcoef, nmax, slope);
    LRES_CUDA_TRY(cudaGetLastError());
    tri_slope_sums_kernel<<<(nwin + 63) / 64, 64, 0, s>>>(nwin, P, slope, cw, u);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_pmat(int nwin, int P, int nmax, const int* n_w, const long long* offN, const long long* offC, const double* d,
             const double* e, const double2* shifts, const double2* wq, double4* coef, double* Pm, cudaStream_t s) {
    if (!nwin) return LRES_OK;
    tri_diag_kernel<<<(unsigned)(((long long)nwin * P + 31) / 32), 32, 0, s>>>(nwin, P, n_w, offN, d, e, shifts, nmax,
                                                                              coef);
    LRES_CUDA_TRY(cudaGetLastError());
    tri_pmat_kernel<<<dim3((nmax + 31) / 32, nwin), 32 * kPmatWarps, 0, s>>>(P, n_w, offC, coef, nmax, wq, Pm);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_rowdot(int w0, int nwin, int maxitems, const int4* items, const int* first, const int* count, const int* n_w,
               const int* m_w, const long long* offN, const long long* offF, const long long* offV,
               const long long* offQ, const long long* Oflat, const double* Y, const double* V, const double* d,
               const double* e, double* dens, double* part, int* status, cudaStream_t s) {
    if (!nwin || !maxitems) return LRES_OK;
    tri_rowdot_kernel<<<dim3(maxitems, nwin), 128, 0, s>>>(w0, items, first, count, n_w, m_w, offN, offF, offV, offQ,
                                                           Oflat, Y, V, d, e, dens, part, status);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_window_sums(int nwin, const int* first, const int* count, const double* part, double dV, double* nw,
                    double* ew, cudaStream_t s) {
    if (!nwin) return LRES_OK;
    tri_window_sums_kernel<<<(nwin + 127) / 128, 128, 0, s>>>(nwin, first, count, part, dV, nw, ew);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_sturm(bool fp32, int nwin, const int* n_w, const long long* offN, const void* d, const void* e,
              double sigma, int* below, cudaStream_t s) {
    if (!nwin) return LRES_OK;
    const int grid = (nwin + 63) / 64;
    if (fp32) tri_sturm_kernel<float><<<grid, 64, 0, s>>>(nwin, n_w, offN, (const float*)d, (const float*)e, sigma, below);
    else tri_sturm_kernel<double><<<grid, 64, 0, s>>>(nwin, n_w, offN, (const double*)d, (const double*)e, sigma, below);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int tri_min_eig(bool fp32, int nwin, const int* n_w, const long long* offN, const void* d, const void* e,
                double tol, double* lam, cudaStream_t s) {
    if (!nwin) return LRES_OK;
    const int grid = (nwin + 31) / 32;
    if (fp32) tri_mineig_kernel<float><<<grid, 32, 0, s>>>(nwin, n_w, offN, (const float*)d, (const float*)e, tol, lam);
    else tri_mineig_kernel<double><<<grid, 32, 0, s>>>(nwin, n_w, offN, (const double*)d, (const double*)e, tol, lam);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

}  // namespace lres
