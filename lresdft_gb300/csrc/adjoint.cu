// Adjoint of the window solve: gradient of the band energy at fixed electron number with
// respect to the window matrices H_W, S_W and the grid potential v.
//
// For window B and upper-half-plane pole z_k the forward kernel (keep mode) leaves the
// complete factor of the augmented matrix [[A, F^T], [F, 0]], A = z_k S_W - H_W (or
// z_k I - H^_W in the standard form of the mixed path), A = G G^T, in one workspace slot:
// rows [0, np) hold G, rows [np, np + m) hold G21 = F G^-T.  Then
//
//   Z_k = A^-1 F^T = G^-T G21^T                       (adj_backsolve_kernel, in place)
//   A_c = Re sum_k c_k Z_k Z_k^T,  c in {w, w z, w z^2} (adj_accum_kernel)
//
// and with U_c = 4 dV <S_W, A_c> summed over windows (identity S in the standard form),
// N and E_band from the same pass, the fixed-N derivatives are
//
//   dN/dmu = N/(2R) - U_{w z'},  dE/dmu = E/R + N/2 - c N/(2R) - U_{w z z'},
//   z' = (1 + zeta)/2 written as real combinations of 1 and z,  kappa = dE/dmu / dN/dmu,
//   dE/dH_W = 4 dV (A_wz - kappa A_w),  dE/dS_W = -4 dV (A_wz2 - kappa A_wz).
//
// The mixed path maps these back with L^-T ( . ) L^-1.  dE/dv(r) = dV x_r^T (sum_B dE/dH_W) x_r
// over the atom pairs that share the point r (the adjoint of the H(v) assembly).
#include "common.cuh"
#include "launch.cuh"
#include "lres_internal.h"

#include <algorithm>

namespace lres {

// ---------------------------------------------------------------------------
// back-substitution  y G = g21  for every owned-point row (thread = row), blocks of NB
// columns from the last: the row's finished y entries stream from the slot, the G rows
// of the finished entries are staged in shared memory in chunks of KC, and every chunk's
// sum is formed from zero before it is subtracted (the forward kernel's rounding pattern).
// ---------------------------------------------------------------------------
template <class T, int NB, int NT, int KC>
__global__ void __launch_bounds__(NT) adj_backsolve_kernel(const int2* items, int nitems, const int* n_w,
                                                            const int* m_w, T* ws, long long ws_stride,
                                                            int* status) {
    using E = El<T>;
    __shared__ T Bs[KC * NB];               // Bs[kk*NB + c] = G[i0 + kk, j0 + c]
    __shared__ T Dblk[NB * (NB + 1)];       // Dblk[c*(NB+1) + c2] = G[j0 + c, j0 + c2], c2 <= c
    __shared__ T Dinv[NB];
    const int it = blockIdx.x;
    if (it >= nitems) return;
    const int w = items[it].x;
    const int n = n_w[w], m = m_w[w];
    const int np = (n + NB - 1) / NB * NB;
    const long long ld = np + m;
    T* G = ws + (size_t)it * ws_stride;
    const int tid = threadIdx.x;
    for (int b0 = 0; b0 < m; b0 += NT) {
        const int r = b0 + tid;
        const bool active = r < m;
        T* yrow = G + np + r;                // y_i of this row at yrow[i*ld] (in place of g21)
        for (int j0 = np - NB; j0 >= 0; j0 -= NB) {
            T acc[NB];
#pragma unroll
            for (int c = 0; c < NB; ++c) acc[c] = active ? yrow[(long long)(j0 + c) * ld] : E::zero();
            for (int i0 = j0 + NB; i0 < np; i0 += KC) {
                const int kc = min(KC, np - i0);
                __syncthreads();
                for (int idx = tid; idx < kc * NB; idx += NT) {
                    const int c = idx / kc, kk = idx % kc;   // column segments are contiguous
                    Bs[kk * NB + c] = G[(i0 + kk) + (long long)(j0 + c) * ld];
                }
                __syncthreads();
                if (active) {
                    T tmp[NB];
#pragma unroll
                    for (int c = 0; c < NB; ++c) tmp[c] = E::zero();
                    for (int kk = 0; kk < kc; ++kk) {
                        const T y = yrow[(long long)(i0 + kk) * ld];
#pragma unroll
                        for (int c = 0; c < NB; ++c) tmp[c] = E::fma(y, Bs[kk * NB + c], tmp[c]);
                    }
#pragma unroll
                    for (int c = 0; c < NB; ++c) acc[c] = E::sub(acc[c], tmp[c]);
                }
            }
            __syncthreads();
            for (int idx = tid; idx < NB * NB; idx += NT) {
                const int c2 = idx / NB, c = idx % NB;       // column c2, row c
                if (c2 <= c) Dblk[c * (NB + 1) + c2] = G[(j0 + c) + (long long)(j0 + c2) * ld];
            }
            __syncthreads();
            if (tid < NB) {
                const T d = Dblk[tid * (NB + 1) + tid];
                const double m2 = (double)E::mag2(d);
                if (!(m2 > 0.0) || !isfinite(m2)) atomicOr(status, ST_ZERO_PIVOT);
                Dinv[tid] = E::inv(d);
            }
            __syncthreads();
            if (active) {
#pragma unroll
                for (int c = NB - 1; c >= 0; --c) {
                    const T y = E::mul(acc[c], Dinv[c]);
                    acc[c] = y;
#pragma unroll
                    for (int c2 = 0; c2 < c; ++c2) acc[c2] = E::fms(y, Dblk[c * (NB + 1) + c2], acc[c2]);
                }
#pragma unroll
                for (int c = 0; c < NB; ++c) yrow[(long long)(j0 + c) * ld] = acc[c];
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// A_c[a, b] = Re sum_k c_k sum_r Z_k[a, r] Z_k[b, r]  for one 32 x 32 tile (a-block I >=
// b-block J) of one window; 16 x 16 threads with 2 x 2 outputs each.  Per pole the r sum is
// taken in chunks of 32 in the working precision, each chunk added in FP64.
// ---------------------------------------------------------------------------
template <class T, int NBF>
__global__ void __launch_bounds__(256) adj_accum_kernel(const int* wins, int P, const int* n_w, const int* m_w,
                                                         const long long* offC, const T* ws, long long ws_stride,
                                                         const double2* cw, double* A0, double* A1, double* A2) {
    using E = El<T>;
    __shared__ T Ya[32][33];
    __shared__ T Yb[32][33];
    const int bw = blockIdx.y;
    const int w = wins[bw];
    const int n = n_w[w], m = m_w[w];
    const int t = blockIdx.x;
    int I = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while ((I + 1) * (I + 2) / 2 <= t) ++I;
    while (I * (I + 1) / 2 > t) --I;
    const int J = t - I * (I + 1) / 2;
    if (I * 32 >= n) return;
    const int np = (n + NBF - 1) / NBF * NBF;
    const long long ld = np + m;
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    double acc[3][2][2] = {};
    for (int k = 0; k < P; ++k) {
        const T* Y = ws + (size_t)(bw * P + k) * ws_stride + np;    // Z_k[a, r] at Y[r + a*ld]
        double ud[2][2][2] = {};
        for (int r0 = 0; r0 < m; r0 += 32) {
            const int rc = min(32, m - r0);
            __syncthreads();
            for (int idx = tid; idx < 32 * 32; idx += 256) {
                const int ii = idx / 32, rr = idx % 32;
                const int a = I * 32 + ii, b = J * 32 + ii;
                Ya[rr][ii] = (rr < rc && a < n) ? Y[(r0 + rr) + (long long)a * ld] : E::zero();
                Yb[rr][ii] = (rr < rc && b < n) ? Y[(r0 + rr) + (long long)b * ld] : E::zero();
            }
            __syncthreads();
            T tmp[2][2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int v = 0; v < 2; ++v) tmp[u][v] = E::zero();
            for (int rr = 0; rr < rc; ++rr) {
                const T a0 = Ya[rr][tx], a1 = Ya[rr][tx + 16];
                const T b0 = Yb[rr][ty], b1 = Yb[rr][ty + 16];
                tmp[0][0] = E::fma(a0, b0, tmp[0][0]);
                tmp[0][1] = E::fma(a0, b1, tmp[0][1]);
                tmp[1][0] = E::fma(a1, b0, tmp[1][0]);
                tmp[1][1] = E::fma(a1, b1, tmp[1][1]);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    ud[u][v][0] += (double)tmp[u][v].x;
                    ud[u][v][1] += (double)tmp[u][v].y;
                }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double2 cc = cw[c * P + k];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int v = 0; v < 2; ++v) acc[c][u][v] += cc.x * ud[u][v][0] - cc.y * ud[u][v][1];
        }
    }
    double* outs[3] = {A0, A1, A2};
    const long long o = offC[w];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int a = I * 32 + tx + 16 * u, b = J * 32 + ty + 16 * v;
            if (a >= n || b >= n) continue;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                outs[c][o + a + (long long)b * n] = acc[c][u][v];
                if (I != J) outs[c][o + b + (long long)a * n] = acc[c][u][v];
            }
        }
}

// ---------------------------------------------------------------------------
// The same accumulations from the tridiagonal form (FP64 path on the tridiagonal route).
//
// With A^ = L^-1 H_W L^-T = Q T Q^T, Y = F^ Q and K = Y^T Y,
//
//     A_c = W X_c W^T,  W = L^-T Q,  X_c = Re sum_k c_k G_k K G_k,  G_k = (z_k - T)^-1,
//
// so a pole costs two tridiagonal solves with n right-hand sides instead of a dense
// factorisation and m back-substitutions: ~23 n^2 FP64 multiply-adds against
// 4 (n^3 / 3 + 3 m n^2).  The FP64 pipe bounds it (54 windows x 32 poles: 6.6 ms at 1.6
// multiply-adds per clock and SM; measured 7.9 ms, 9.2 without the loads ahead of the chain; in FP32, 128
// windows, 6.9 ms, 14.8 without).
// ---------------------------------------------------------------------------

// Per (window, pole): the multipliers t_i = e_{i-1} / D_{i-1} and 1 / D_i of the LDL^T of z_k - T
// (D_i = z - d_i - e_{i-1} t_i; Im D_i >= Im z), coef[item * ld + i] = (t, 1 / D).
__global__ void adj_pivot_kernel(int nwin, int P, const int* n_w, const long long* offN, const double* d,
                                 const double* e, const double2* z, int ld, double4* coef) {
    const int it = blockIdx.x * blockDim.x + threadIdx.x;
    if (it >= nwin * P) return;
    const int w = it / P;
    const double2 zk = z[it - w * P];
    const int n = n_w[w];
    const double *dw = d + offN[w], *ew = e + offN[w];
    double4* out = coef + (size_t)it * ld;
    double2 t = make_double2(0.0, 0.0), g = t;
    for (int i = 0; i < n; ++i) {
        double2 D = make_double2(zk.x - dw[i], zk.y);
        if (i) {
            const double el = ew[i - 1];
            t = make_double2(el * g.x, el * g.y);
            D.x = fma(-el, t.x, D.x);
            D.y = fma(-el, t.y, D.y);
        }
        const double inv = 1.0 / (D.x * D.x + D.y * D.y);
        g = make_double2(D.x * inv, -D.y * inv);
        out[i] = make_double4(t.x, t.y, g.x, g.y);
    }
}

constexpr int kSweepNT = 320;

template <class R> struct Sweep;
template <> struct Sweep<double> { using C2 = double2; using C4 = double4; };
template <> struct Sweep<float> { using C2 = float2; using C4 = float4; };

// One CTA per (window, group of poles): X_c += Re c_k G_k K G_k over its poles, the upper triangle of
// group g at Xc[g * sizeC + offC + i + j n], i <= j.  Thread = column of K for G_k K, then row of it for
// the second solve (whose back substitution stops at the diagonal); every access but the reads of the
// second forward sweep runs along the threads, and CH steps are loaded ahead of the chain.  R = float (mixed precision): the sweeps in FP32 from the
// FP64 pivots, the poles still summed in FP64.
template <class R>
__global__ void __launch_bounds__(kSweepNT) adj_sweep_kernel(const int* wins, int P, int groups, const int* n_w,
                                                             const long long* offC, long long sizeC, const R* K,
                                                             const double4* coef, int ld, const double2* cw,
                                                             typename Sweep<R>::C2* ws, long long ws_stride, double* Xa,
                                                             double* Xb, double* Xc) {
    using C2 = typename Sweep<R>::C2;
    using C4 = typename Sweep<R>::C4;
    constexpr int CH = 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C4* const cf = reinterpret_cast<C4*>(smem_raw);                 // [n + 1]
    const int w = wins[blockIdx.x / groups], grp = blockIdx.x % groups;
    const int n = n_w[w], tid = threadIdx.x;
    const int k0 = P * grp / groups, k1 = P * (grp + 1) / groups;
    const R* const Kw = K + offC[w];
    C2* const B = ws + (size_t)blockIdx.x * ws_stride;              // (G K)^T: B[j + i n] = (G K)_ij
    C2* const U = B + (size_t)n * n;                                // U[i + j n]
    for (int k = k0; k < k1; ++k) {
        __syncthreads();
        const double4* const src = coef + (size_t)(w * P + k) * ld;
        for (int i = tid; i < n; i += kSweepNT) cf[i] = C4{(R)src[i].x, (R)src[i].y, (R)src[i].z, (R)src[i].w};
        if (tid == 0) cf[n] = C4{R(0), R(0), R(0), R(0)};
        __syncthreads();
        for (int j = tid; j < n; j += kSweepNT) {
            C2 u = C2{R(0), R(0)};
            for (int i0 = 0; i0 < n; i0 += CH) {
                R kv[CH];
#pragma unroll
                for (int q = 0; q < CH; ++q) kv[q] = Kw[j + (long long)min(i0 + q, n - 1) * n];
#pragma unroll
                for (int q = 0; q < CH; ++q) {
                    if (i0 + q >= n) break;
                    const C4 c = cf[i0 + q];
                    u = C2{fma(c.x, u.x, fma(-c.y, u.y, kv[q])), fma(c.x, u.y, c.y * u.x)};
                    B[j + (long long)(i0 + q) * n] = u;
                }
            }
            C2 x = C2{R(0), R(0)};
            for (int i1 = n - 1; i1 >= 0; i1 -= CH) {
                C2 v[CH];
#pragma unroll
                for (int q = 0; q < CH; ++q) v[q] = B[j + (long long)max(i1 - q, 0) * n];
#pragma unroll
                for (int q = 0; q < CH; ++q) {
                    if (i1 - q < 0) break;
                    const C4 c = cf[i1 - q], cn = cf[i1 - q + 1];
                    x = C2{fma(v[q].x, c.z, fma(-v[q].y, c.w, fma(cn.x, x.x, -cn.y * x.y))),
                           fma(v[q].x, c.w, fma(v[q].y, c.z, fma(cn.x, x.y, cn.y * x.x)))};
                    B[j + (long long)(i1 - q) * n] = x;
                }
            }
        }
        __syncthreads();
        const C2 c0 = C2{(R)cw[k].x, (R)cw[k].y}, c1 = C2{(R)cw[P + k].x, (R)cw[P + k].y},
                 c2 = C2{(R)cw[2 * P + k].x, (R)cw[2 * P + k].y};
        double* const X0 = Xa + (size_t)grp * sizeC + offC[w];
        double* const X1 = Xb + (size_t)grp * sizeC + offC[w];
        double* const X2 = Xc + (size_t)grp * sizeC + offC[w];
        for (int i = tid; i < n; i += kSweepNT) {
            C2 u = C2{R(0), R(0)};
            for (int j0 = 0; j0 < n; j0 += CH) {
                C2 bv[CH];
#pragma unroll
                for (int q = 0; q < CH; ++q) bv[q] = B[min(j0 + q, n - 1) + (long long)i * n];
#pragma unroll
                for (int q = 0; q < CH; ++q) {
                    const int j = j0 + q;
                    if (j >= n) break;
                    const C4 c = cf[j];
                    u = C2{fma(c.x, u.x, fma(-c.y, u.y, bv[q].x)), fma(c.x, u.y, fma(c.y, u.x, bv[q].y))};
                    if (j >= i) U[i + (long long)j * n] = u;
                }
            }
            C2 x = C2{R(0), R(0)};
            constexpr int CX = 4;
            for (int j1 = n - 1; j1 >= i; j1 -= CX) {
                C2 v[CX];
                double y[CX][3];
#pragma unroll
                for (int q = 0; q < CX; ++q) {
                    const long long at = i + (long long)max(j1 - q, i) * n;
                    v[q] = U[at];
                    y[q][0] = y[q][1] = y[q][2] = 0.0;
                    if (k != k0) {
                        y[q][0] = X0[at];
                        y[q][1] = X1[at];
                        y[q][2] = X2[at];
                    }
                }
#pragma unroll
                for (int q = 0; q < CX; ++q) {
                    const int j = j1 - q;
                    if (j < i) break;
                    const C4 c = cf[j], cn = cf[j + 1];
                    const long long at = i + (long long)j * n;
                    x = C2{fma(v[q].x, c.z, fma(-v[q].y, c.w, fma(cn.x, x.x, -cn.y * x.y))),
                           fma(v[q].x, c.w, fma(v[q].y, c.z, fma(cn.x, x.y, cn.y * x.x)))};
                    if constexpr (sizeof(R) == 8) {
                        X0[at] = fma(c0.x, x.x, fma(-c0.y, x.y, y[q][0]));
                        X1[at] = fma(c1.x, x.x, fma(-c1.y, x.y, y[q][1]));
                        X2[at] = fma(c2.x, x.x, fma(-c2.y, x.y, y[q][2]));
                    } else {
                        X0[at] = y[q][0] + (double)fma(c0.x, x.x, -c0.y * x.y);
                        X1[at] = y[q][1] + (double)fma(c1.x, x.x, -c1.y * x.y);
                        X2[at] = y[q][2] + (double)fma(c2.x, x.x, -c2.y * x.y);
                    }
                }
            }
        }
    }
}

// A_c = the sum of the groups' upper triangles in order, both triangles written (32 x 32 tiles; one
// group may be in place).
__global__ void __launch_bounds__(256) adj_groups_kernel(int groups, const int* n_w, const long long* offC,
                                                         long long sizeC, const double* Xa, const double* Xb,
                                                         const double* Xc, double* A0, double* A1, double* A2) {
    __shared__ double tile[32][33];
    const int w = blockIdx.z, n = n_w[w];
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
    if (i0 > j0 || j0 >= n) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const double* const ins[3] = {Xa, Xb, Xc};
    double* const outs[3] = {A0, A1, A2};
    for (int c = 0; c < 3; ++c) {
        const double* const src = ins[c] + offC[w];
        double* const dst = outs[c] + offC[w];
        __syncthreads();
        for (int q = ty; q < 32; q += 8) {
            const int i = i0 + tx, j = j0 + q;
            if (i <= j && j < n) {
                double s = 0.0;
                for (int g = 0; g < groups; ++g) s += src[(size_t)g * sizeC + i + (long long)j * n];
                dst[i + (long long)j * n] = s;
                tile[q][tx] = s;
            }
        }
        __syncthreads();
        for (int q = ty; q < 32; q += 8) {
            const int i = i0 + q, j = j0 + tx;
            if (i < j && j < n) dst[j + (long long)i * n] = tile[tx][q];
        }
    }
}

// Pole weights of the three accumulations: c_0 = w_k, c_1 = w_k z_k, c_2 = w_k z_k^2,
// nodes as the forward pass computes them (lrft/core.py:130-139).
__global__ void adj_weights_kernel(int P, int M, double mu, double e_lo, double2* cw) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= P) return;
    const double cc = 0.5 * (mu + e_lo), R = 0.5 * (mu - e_lo);
    double sn, cs;
    sincospi((double)(2 * k + 1) / (double)M, &sn, &cs);
    const double zr = cc + R * cs, zi = R * sn;
    const double wr = R * cs / M, wi = R * sn / M;
    const double w1r = wr * zr - wi * zi, w1i = wr * zi + wi * zr;
    cw[k] = make_double2(wr, wi);
    cw[P + k] = make_double2(w1r, w1i);
    cw[2 * P + k] = make_double2(w1r * zr - w1i * zi, w1r * zi + w1i * zr);
}

// u[c*nwin + w] = <S_W, A_c> (S given) or tr(A_c) (S null), fixed-order reduction.
__global__ void __launch_bounds__(256) adj_inner_kernel(int nwin, const int* n_w, const long long* offC,
                                                         const double* S, const double* A0, const double* A1,
                                                         const double* A2, double* u) {
    const int w = blockIdx.x;
    if (w >= nwin) return;
    const int n = n_w[w];
    const long long o = offC[w];
    const long long cnt = S ? (long long)n * n : n;
    double s[3] = {0.0, 0.0, 0.0};
    for (long long i = threadIdx.x; i < cnt; i += 256) {
        const long long e = S ? o + i : o + i + i * n;
        const double f = S ? S[e] : 1.0;
        s[0] = fma(f, A0[e], s[0]);
        s[1] = fma(f, A1[e], s[1]);
        s[2] = fma(f, A2[e], s[2]);
    }
    __shared__ double red[3][256];
    for (int c = 0; c < 3; ++c) red[c][threadIdx.x] = s[c];
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h)
            for (int c = 0; c < 3; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x < 3) u[threadIdx.x * nwin + w] = red[threadIdx.x][0];
}

// X = a (A1 - kappa A0), Y = b (A2 - kappa A1), elementwise.
__global__ void adj_combine_kernel(long long nval, const double* A0, const double* A1, const double* A2,
                                   double kappa, double a, double b, double* X, double* Y) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= nval) return;
    const double x = a * (A1[i] - kappa * A0[i]);
    const double y = b * (A2[i] - kappa * A1[i]);
    X[i] = x;
    Y[i] = y;
}

// Global gradient blocks: gH[block (g,h)] = sum over the windows holding g and h of their
// dE/dH_W block, windows in ascending order (one warp per block).
__global__ void __launch_bounds__(256) adj_block_gather_kernel(int nblk, const int* brow, const int* bcol,
                                                                const int* gptr, const long long* boff,
                                                                const long long* eoff, const int4* ent,
                                                                const int* n_w, const long long* offC,
                                                                const double* dHW, double* gH) {
    const int b = blockIdx.x * 8 + threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (b >= nblk) return;
    const int g = brow[b], h = bcol[b];
    const int nfg = gptr[g + 1] - gptr[g], nfh = gptr[h + 1] - gptr[h];
    const int nv = nfg * nfh;
    for (int vi = lane; vi < nv; vi += 32) {
        const int a = vi / nfh, c = vi % nfh;
        double s = 0.0;
        for (long long e = eoff[b]; e < eoff[b + 1]; ++e) {
            const int4 t = ent[e];             // (window, local offset of g, local offset of h)
            s += dHW[offC[t.x] + (t.y + a) + (long long)(t.z + c) * n_w[t.x]];
        }
        gH[boff[b] + vi] = s;
    }
}

// dE/dv(r) = dV sum_{g,h covering r} x_g(r)^T gH_gh x_h(r) (thread = grid point).
__global__ void __launch_bounds__(256) adj_point_kernel(long long ng, const long long* poff, const int2* pent,
                                                         const double* sval, const int* gptr, const int* bptr,
                                                         const int* bcol, const long long* boff,
                                                         const double* gH, double dV, double* dv) {
    const long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (r >= ng) return;
    const long long e0 = poff[r], e1 = poff[r + 1];
    double s = 0.0;
    for (long long e = e0; e < e1; ++e) {
        const int2 gs = pent[e];
        const int g = gs.x;
        const int nfg = gptr[g + 1] - gptr[g];
        const double* xg = sval + (size_t)gs.y * 8;
        const int b0 = bptr[g], b1 = bptr[g + 1];
        for (long long f = e; f < e1; ++f) {                         // (gH is symmetric: pairs once)
            const double twice = f == e ? 1.0 : 2.0;
            const int2 hs = pent[f];
            const int h = hs.x;
            int lo = b0, hi = b1;              // block (g, h) in the sorted block row g
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (bcol[mid] < h) lo = mid + 1;
                else hi = mid;
            }
            if (lo >= b1 || bcol[lo] != h) continue;
            const int nfh = gptr[h + 1] - gptr[h];
            const double* xh = sval + (size_t)hs.y * 8;
            const double* blk = gH + boff[lo];
            for (int a = 0; a < nfg; ++a) {
                double t = 0.0;
                for (int c = 0; c < nfh; ++c) t = fma(blk[a * nfh + c], xh[c], t);
                s = fma(twice * xg[a], t, s);
            }
        }
    }
    dv[r] = dV * s;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
int adj_backsolve(bool fp32, const int2* items, int nitems, const int* n_w, const int* m_w, void* ws,
                  long long ws_stride, int* status, cudaStream_t s) {
    if (!nitems) return LRES_OK;
    if (fp32)
        adj_backsolve_kernel<float2, kKeepNB64, 128, 32><<<nitems, 128, 0, s>>>(items, nitems, n_w, m_w,
                                                                                (float2*)ws, ws_stride, status);
    else
        adj_backsolve_kernel<double2, kKeepNB128, 128, 32><<<nitems, 128, 0, s>>>(items, nitems, n_w, m_w,
                                                                                  (double2*)ws, ws_stride, status);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int adj_accumulate(bool fp32, const int* wins, int nwin_batch, int P, int nmax, const int* n_w, const int* m_w,
                   const long long* offC, const void* ws, long long ws_stride, const double2* cw, double* A0,
                   double* A1, double* A2, cudaStream_t s) {
    if (!nwin_batch) return LRES_OK;
    const int T = (nmax + 31) / 32;
    dim3 grid(T * (T + 1) / 2, nwin_batch);
    if (fp32)
        adj_accum_kernel<float2, kKeepNB64><<<grid, 256, 0, s>>>(wins, P, n_w, m_w, offC, (const float2*)ws,
                                                                 ws_stride, cw, A0, A1, A2);
    else
        adj_accum_kernel<double2, kKeepNB128><<<grid, 256, 0, s>>>(wins, P, n_w, m_w, offC, (const double2*)ws,
                                                                   ws_stride, cw, A0, A1, A2);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

// pole groups of a window in the sweeps: two CTAs per SM in all
int adj_sweep_groups(int nwin, int P) {
    return std::max(1, std::min(P, 2 * device_sms() / std::max(nwin, 1)));
}

template <class R>
static int launch_sweeps(int nwin, int P, int groups, int batch, int nmax, const int* wins, const int* n_w,
                         const long long* offC, long long sizeC, const R* K, const double4* coef, const double2* cw,
                         void* ws, double* Xa, double* Xb, double* Xc, size_t smem_budget, cudaStream_t s) {
    const size_t smem = sizeof(typename Sweep<R>::C4) * ((size_t)nmax + 1);
    if (smem > smem_budget) {
        lres_set_error("adjoint sweeps need %zu B of shared memory", smem);
        return LRES_EINVAL;
    }
    int per_sm = 0;
    if (int rc = prepare_kernel<adj_sweep_kernel<R>>(kSweepNT, smem, &per_sm)) return rc;
    for (int w0 = 0; w0 < nwin; w0 += batch) {
        adj_sweep_kernel<R><<<(unsigned)std::min(batch, nwin - w0) * groups, kSweepNT, smem, s>>>(
            wins + w0, P, groups, n_w, offC, sizeC, K, coef, nmax, cw, static_cast<typename Sweep<R>::C2*>(ws),
            2LL * nmax * nmax, Xa, Xb, Xc);
        LRES_CUDA_TRY(cudaGetLastError());
    }
    return LRES_OK;
}

int adj_tri(int nwin, int P, int groups, int batch, int nmax, const int* wins, const int* n_w, const long long* offN,
            const long long* offC, long long sizeC, const double* d, const double* e, const double2* shifts,
            const double2* cw, const double* K, const float* K32, double4* coef, void* ws, double* X, double* A0,
            double* A1, double* A2, size_t smem_budget, cudaStream_t s) {
    if (!nwin) return LRES_OK;
    if (nwin > 65535) {
        lres_set_error("adjoint supports at most 65535 windows (got %d)", nwin);
        return LRES_EINVAL;
    }
    adj_pivot_kernel<<<(unsigned)(((long long)nwin * P + 31) / 32), 32, 0, s>>>(nwin, P, n_w, offN, d, e, shifts, nmax,
                                                                               coef);
    LRES_CUDA_TRY(cudaGetLastError());
    // one group accumulates in place
    double* const Xa = groups > 1 ? X : A0;
    double* const Xb = groups > 1 ? Xa + (size_t)groups * sizeC : A1;
    double* const Xc = groups > 1 ? Xb + (size_t)groups * sizeC : A2;
    if (int rc = K32 ? launch_sweeps<float>(nwin, P, groups, batch, nmax, wins, n_w, offC, sizeC, K32, coef, cw, ws, Xa,
                                            Xb, Xc, smem_budget, s)
                     : launch_sweeps<double>(nwin, P, groups, batch, nmax, wins, n_w, offC, sizeC, K, coef, cw, ws, Xa,
                                             Xb, Xc, smem_budget, s))
        return rc;
    const int T = (nmax + 31) / 32;
    adj_groups_kernel<<<dim3(T, T, nwin), 256, 0, s>>>(groups, n_w, offC, sizeC, Xa, Xb, Xc, A0, A1, A2);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int adj_weights(int P, int M, double mu, double e_lo, double2* cw, cudaStream_t s) {
    adj_weights_kernel<<<(P + 63) / 64, 64, 0, s>>>(P, M, mu, e_lo, cw);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int adj_inner(int nwin, const int* n_w, const long long* offC, const double* S, const double* A0, const double* A1,
              const double* A2, double* u, cudaStream_t s) {
    adj_inner_kernel<<<nwin, 256, 0, s>>>(nwin, n_w, offC, S, A0, A1, A2, u);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int adj_combine(long long nval, const double* A0, const double* A1, const double* A2, double kappa, double a,
                double b, double* X, double* Y, cudaStream_t s) {
    adj_combine_kernel<<<(unsigned)((nval + 255) / 256), 256, 0, s>>>(nval, A0, A1, A2, kappa, a, b, X, Y);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int adj_block_gather(const BlockPattern& bp, const long long* eoff, const int4* ent, const int* n_w,
                     const long long* offC, const double* dHW, double* gH, cudaStream_t s) {
    adj_block_gather_kernel<<<(bp.nblk + 7) / 8, 256, 0, s>>>(bp.nblk, bp.brow, bp.bcol, bp.gptr, bp.boff, eoff,
                                                              ent, n_w, offC, dHW, gH);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int adj_point(long long ng, const long long* poff, const int2* pent, const Supports& sp, const BlockPattern& bp,
              const double* gH, double dV, double* dv, cudaStream_t s) {
    adj_point_kernel<<<(unsigned)((ng + 255) / 256), 256, 0, s>>>(ng, poff, pent, sp.sval, bp.gptr, bp.bptr,
                                                                   bp.bcol, bp.boff, gH, dV, dv);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

}  // namespace lres
