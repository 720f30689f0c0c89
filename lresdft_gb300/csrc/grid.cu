// Grid kernels of the SCF step: a hand-written mixed-radix FFT of real grids (3-D, FP64), FFT
// Hartree, LDA exchange-correlation, the ion potential and Voronoi ownership.
//
// FFT: what bounds it is the FP64 pipe (1/64 of the FP32 rate: 1 TFLOP/s), not memory: a 108^3
// Hartree step moves 0.12 GB through L2 and issues ~0.1 G FP64 instructions.  So no FP64 work
// that a table can replace (the twiddles are read, not evaluated), and only half of the
// spectrum is computed: two real lines make one complex line along the contiguous axis, and the
// other two axes run over n3/2+1 wave numbers.  The x axis is transformed, divided by G^2 and
// transformed back in one kernel: five passes per Hartree step.  Each CTA holds 8 lines in shared
// memory ([element][line], rows of 9 so that neither direction conflicts) and runs a Stockham
// autosort over the factors of the length (4, 2, 3, 5 in registers, any other prime by a direct
// DFT): 8 lines per CTA give 2 or more CTAs per SM from 64^3 on.
// Measured (LDA + Hartree): 64^3 0.48 -> 0.24 ms, 108^3 9.3 -> 0.84 ms (evaluated twiddles and
// radix-3 and -5 factors by sincospi, six complex passes, before); 0.114 and 0.38 ms with the LDA
// kernel's roots below.
#include "common.cuh"
#include "lres_internal.h"

#include <cmath>
#include <vector>

namespace lres {

constexpr int kFftNT = 128;
constexpr int kFftLines = 8, kFftRow = kFftLines + 1;
constexpr int kFftFac = 14;

// One axis: its length, factors and twiddle table exp(-2 pi i k / L), k < L.
struct FftAxis {
    int L = 0, nf = 0;
    int fac[kFftFac] = {};
    const double2* tw = nullptr;
    const double* k = nullptr;        // wave numbers
};

struct FFT3 {
    FftAxis ax[3];
    double2* d_tw = nullptr;
    double* d_k = nullptr;
    double2* d_ion = nullptr;         // scratch of the ion potential
    size_t ion_size = 0;
};

static std::vector<int> factorise(int n) {
    std::vector<int> f;
    while (n % 4 == 0) { f.push_back(4); n /= 4; }
    while (n % 2 == 0) { f.push_back(2); n /= 2; }
    for (int p = 3; p * p <= n; p += 2)
        while (n % p == 0) { f.push_back(p); n /= p; }
    if (n > 1) f.push_back(n);
    return f;
}

int fft3_create(FFT3** out, const int64_t shape[3], const double cell[3]) {
    size_t total = 0;
    for (int a = 0; a < 3; ++a) {
        if (shape[a] < 1 || shape[a] > 4096 || factorise((int)shape[a]).size() > kFftFac) {
            lres_set_error("grid axis of length %lld not supported by the FFT", (long long)shape[a]);
            return LRES_EINVAL;
        }
        total += shape[a];
    }
    std::vector<double2> tw(total);
    std::vector<double> kv(total);
    FFT3* f = new FFT3();
    size_t off = 0;
    for (int a = 0; a < 3; ++a) {
        const int L = (int)shape[a];
        const std::vector<int> fac = factorise(L);
        f->ax[a].L = L;
        f->ax[a].nf = (int)fac.size();
        for (size_t i = 0; i < fac.size(); ++i) f->ax[a].fac[i] = fac[i];
        // wave numbers as numpy: 2 pi (f (1 / (m (L / m)))) with f the fftfreq index
        const double val = 1.0 / ((double)L * (cell[a] / (double)L));
        for (int i = 0; i < L; ++i) {
            const long double ph = 2.0L * acosl(-1.0L) * i / L;
            tw[off + i] = make_double2((double)cosl(ph), (double)-sinl(ph));
            kv[off + i] = 2.0 * M_PI * ((double)(i < (L + 1) / 2 ? i : i - L) * val);
        }
        off += L;
    }
    if (cudaMalloc(&f->d_tw, sizeof(double2) * total) != cudaSuccess ||
        cudaMalloc(&f->d_k, sizeof(double) * total) != cudaSuccess ||
        cudaMemcpy(f->d_tw, tw.data(), sizeof(double2) * total, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(f->d_k, kv.data(), sizeof(double) * total, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        fft3_destroy(f);
        lres_set_error("FFT plan allocation failed");
        return LRES_ENOMEM;
    }
    off = 0;
    for (FftAxis& x : f->ax) {
        x.tw = f->d_tw + off;
        x.k = f->d_k + off;
        off += x.L;
    }
    *out = f;
    return LRES_OK;
}

void fft3_destroy(FFT3* f) {
    if (!f) return;
    cudaFree(f->d_tw);
    cudaFree(f->d_k);
    cudaFree(f->d_ion);
    delete f;
}

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a + s i b (s = -1 forward, +1 inverse)
template <bool INV>
__device__ __forceinline__ double2 add_i(double2 a, double2 b) {
    return INV ? make_double2(a.x - b.y, a.y + b.x) : make_double2(a.x + b.y, a.y - b.x);
}
template <bool INV>
__device__ __forceinline__ double2 twiddle(const double2* tw, int k) {
    double2 w = tw[k];
    if (INV) w.y = -w.y;
    return w;
}

// a[t] <- sum_j a[j] exp(-+ 2 pi i j t / R)
template <int R, bool INV>
__device__ __forceinline__ void dft(double2 (&a)[R]) {
    if constexpr (R == 2) {
        const double2 t = a[0];
        a[0] = cadd(t, a[1]);
        a[1] = csub(t, a[1]);
    } else if constexpr (R == 3) {
        const double c = 0.86602540378443864676;                     // sin(2 pi / 3)
        const double2 t = cadd(a[1], a[2]), d = make_double2(c * (a[1].x - a[2].x), c * (a[1].y - a[2].y));
        const double2 m = make_double2(fma(-0.5, t.x, a[0].x), fma(-0.5, t.y, a[0].y));
        a[0] = cadd(a[0], t);
        a[1] = add_i<INV>(m, d);
        a[2] = add_i<!INV>(m, d);
    } else if constexpr (R == 4) {
        const double2 t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]), t2 = cadd(a[1], a[3]), t3 = csub(a[1], a[3]);
        a[0] = cadd(t0, t2);
        a[1] = add_i<INV>(t1, t3);
        a[2] = csub(t0, t2);
        a[3] = add_i<!INV>(t1, t3);
    } else {
        static_assert(R == 5, "radix");
        const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;   // cos(2 pi / 5), cos(4 pi / 5)
        const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
        const double2 t1 = cadd(a[1], a[4]), t2 = cadd(a[2], a[3]), t3 = csub(a[1], a[4]), t4 = csub(a[2], a[3]);
        const double2 m1 = make_double2(fma(c1, t1.x, fma(c2, t2.x, a[0].x)), fma(c1, t1.y, fma(c2, t2.y, a[0].y)));
        const double2 m2 = make_double2(fma(c2, t1.x, fma(c1, t2.x, a[0].x)), fma(c2, t1.y, fma(c1, t2.y, a[0].y)));
        const double2 n1 = make_double2(fma(s1, t3.x, s2 * t4.x), fma(s1, t3.y, s2 * t4.y));
        const double2 n2 = make_double2(fma(s2, t3.x, -s1 * t4.x), fma(s2, t3.y, -s1 * t4.y));
        a[0] = cadd(a[0], cadd(t1, t2));
        a[1] = add_i<INV>(m1, n1);
        a[2] = add_i<INV>(m2, n2);
        a[3] = add_i<!INV>(m2, n2);
        a[4] = add_i<!INV>(m1, n1);
    }
}

// One Stockham stage of radix R: sub-transforms of length m R, stride s (m R s = L).
template <int R, bool INV>
__device__ __forceinline__ void fft_stage(const double2* x, double2* y, int m, int s, const double2* tw) {
    for (int idx = threadIdx.x; idx < m * s * kFftLines; idx += kFftNT) {
        const int b = idx & (kFftLines - 1), pq = idx / kFftLines;
        const int p = pq / s, q = pq - p * s;
        double2 a[R];
#pragma unroll
        for (int j = 0; j < R; ++j) a[j] = x[(q + s * (p + j * m)) * kFftRow + b];
        dft<R, INV>(a);
#pragma unroll
        for (int t = 0; t < R; ++t) {
            if (t && p) a[t] = cmulc(a[t], twiddle<INV>(tw, p * t * s));
            y[(q + s * (R * p + t)) * kFftRow + b] = a[t];
        }
    }
}

// The same for any radix r, one output per thread.
template <bool INV>
__device__ __forceinline__ void fft_stage_any(const double2* x, double2* y, int r, int m, int s, const double2* tw) {
    const int step = m * s;                                          // L / r
    for (int idx = threadIdx.x; idx < r * m * s * kFftLines; idx += kFftNT) {
        const int b = idx & (kFftLines - 1), k = idx / kFftLines;
        const int q = k % s, pt = k / s, t = pt % r, p = pt / r;
        double2 acc = make_double2(0.0, 0.0);
        for (int j = 0, e = 0; j < r; ++j) {
            acc = cadd(acc, cmulc(x[(q + s * (p + j * m)) * kFftRow + b], twiddle<INV>(tw, e * step)));
            e += t;
            if (e >= r) e -= r;
        }
        if (p && t) acc = cmulc(acc, twiddle<INV>(tw, p * t * s));
        y[k * kFftRow + b] = acc;
    }
}

// The 8 lines in x transformed in place of x or y (the buffer that holds the result is returned).
template <bool INV>
__device__ double2* fft_lines(double2* x, double2* y, const FftAxis& ax, const double2* tw) {
    int n = ax.L, s = 1;
    for (int i = 0; i < ax.nf; ++i) {
        const int r = ax.fac[i], m = n / r;
        if (r == 4) fft_stage<4, INV>(x, y, m, s, tw);
        else if (r == 2) fft_stage<2, INV>(x, y, m, s, tw);
        else if (r == 3) fft_stage<3, INV>(x, y, m, s, tw);
        else if (r == 5) fft_stage<5, INV>(x, y, m, s, tw);
        else fft_stage_any<INV>(x, y, r, m, s, tw);
        __syncthreads();
        double2* const t = x;
        x = y;
        y = t;
        n = m;
        s *= r;
    }
    return x;
}

inline size_t fft_smem(int L) { return sizeof(double2) * ((size_t)2 * L * kFftRow + L); }

// Real lines of the contiguous axis: lines 2l and 2l+1 as the real and imaginary part of one.
// Forward: the half spectra w[line * h + k], k < h; inverse: the lines scaled by `scale`.
template <bool INV>
__global__ void __launch_bounds__(kFftNT) fft_real_kernel(FftAxis ax, long long nlines, double* r, double2* w,
                                                          double scale) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int L = ax.L, h = L / 2 + 1;
    double2* const tw = reinterpret_cast<double2*>(smraw);
    double2* x = tw + L;
    double2* y = x + (size_t)L * kFftRow;
    const long long l0 = 2 * (long long)blockIdx.x * kFftLines;      // first line
    for (int i = threadIdx.x; i < L; i += kFftNT) tw[i] = ax.tw[i];
    if (!INV) {
        for (int idx = threadIdx.x; idx < L * kFftLines; idx += kFftNT) {
            const int b = idx / L, t = idx - b * L;
            const long long a = l0 + 2 * b;
            x[t * kFftRow + b] = make_double2(a < nlines ? r[a * L + t] : 0.0, a + 1 < nlines ? r[(a + 1) * L + t] : 0.0);
        }
    } else {
        for (int idx = threadIdx.x; idx < h * kFftLines; idx += kFftNT) {
            const int b = idx / h, k = idx - b * h;
            const long long a = l0 + 2 * b;
            double2 u = a < nlines ? w[a * h + k] : make_double2(0.0, 0.0);
            double2 v = a + 1 < nlines ? w[(a + 1) * h + k] : make_double2(0.0, 0.0);
            if (k == 0 || 2 * k == L) u.y = v.y = 0.0;              // (the real part of the line is wanted)
            x[k * kFftRow + b] = make_double2(u.x - v.y, u.y + v.x);                    // u + i v
            if (k && 2 * k < L) x[(L - k) * kFftRow + b] = make_double2(u.x + v.y, v.x - u.y);
        }
    }
    __syncthreads();
    const double2* z = fft_lines<INV>(x, y, ax, tw);
    if (!INV) {
        for (int idx = threadIdx.x; idx < h * kFftLines; idx += kFftNT) {
            const int b = idx / h, k = idx - b * h;
            const long long a = l0 + 2 * b;
            const double2 p = z[k * kFftRow + b], q = z[(k ? L - k : 0) * kFftRow + b];
            if (a < nlines) w[a * h + k] = make_double2(0.5 * (p.x + q.x), 0.5 * (p.y - q.y));
            if (a + 1 < nlines) w[(a + 1) * h + k] = make_double2(0.5 * (p.y + q.y), 0.5 * (q.x - p.x));
        }
    } else {
        for (int idx = threadIdx.x; idx < L * kFftLines; idx += kFftNT) {
            const int b = idx / L, t = idx - b * L;
            const long long a = l0 + 2 * b;
            const double2 p = z[t * kFftRow + b];
            if (a < nlines) r[a * L + t] = p.x * scale;
            if (a + 1 < nlines) r[(a + 1) * L + t] = p.y * scale;
        }
    }
}

// Lines of another axis over the half spectrum, 8 neighbouring wave numbers k of the contiguous
// axis per CTA: element t of line (o, k) at w[o * ostride + t * tstride + k].  POISSON: forward,
// times 4 pi scale / G^2 (0 at G = 0), back (the x axis; o is then the index of the y axis).
template <bool INV, bool POISSON>
__global__ void __launch_bounds__(kFftNT) fft_axis_kernel(FftAxis ax, int h, long long ostride, long long tstride,
                                                          double2* w, const double* ky, const double* kz,
                                                          double scale) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int L = ax.L;
    double2* const tw = reinterpret_cast<double2*>(smraw);
    double2* x = tw + L;
    double2* y = x + (size_t)L * kFftRow;
    const int groups = (h + kFftLines - 1) / kFftLines;
    const int o = blockIdx.x / groups, k0 = (blockIdx.x - o * groups) * kFftLines;
    double2* const base = w + o * ostride + k0;
    for (int i = threadIdx.x; i < L; i += kFftNT) tw[i] = ax.tw[i];
    for (int idx = threadIdx.x; idx < L * kFftLines; idx += kFftNT) {
        const int b = idx & (kFftLines - 1), t = idx / kFftLines;
        x[t * kFftRow + b] = k0 + b < h ? base[t * tstride + b] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    double2* z = fft_lines<INV>(x, y, ax, tw);
    if (POISSON) {
        for (int idx = threadIdx.x; idx < L * kFftLines; idx += kFftNT) {
            const int b = idx & (kFftLines - 1), t = idx / kFftLines;
            const double kx = ax.k[t], gy = ky[o], gz = kz[min(k0 + b, h - 1)];
            const double g2 = kx * kx + gy * gy + gz * gz;
            const double f = g2 > 0.0 ? 4.0 * M_PI * scale / g2 : 0.0;
            double2& v = z[t * kFftRow + b];
            v = make_double2(f * v.x, f * v.y);
        }
        __syncthreads();
        z = fft_lines<true>(z, z == x ? y : x, ax, tw);
    }
    for (int idx = threadIdx.x; idx < L * kFftLines; idx += kFftNT) {
        const int b = idx & (kFftLines - 1), t = idx / kFftLines;
        if (k0 + b < h) base[t * tstride + b] = z[t * kFftRow + b];
    }
}

template <bool INV>
static int fft_real(const FFT3* f, double* r, double2* w, double scale, cudaStream_t s) {
    const long long nlines = (long long)f->ax[0].L * f->ax[1].L;
    const size_t smem = fft_smem(f->ax[2].L);
    LRES_CUDA_TRY(cudaFuncSetAttribute(fft_real_kernel<INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long blocks = (nlines + 2 * kFftLines - 1) / (2 * kFftLines);
    fft_real_kernel<INV><<<(unsigned)blocks, kFftNT, smem, s>>>(f->ax[2], nlines, r, w, scale);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

// axis 0 (x) or 1 (y) of the half spectrum
template <bool INV, bool POISSON>
static int fft_axis(const FFT3* f, int axis, double2* w, double scale, cudaStream_t s) {
    const int h = f->ax[2].L / 2 + 1;
    const long long row = h, plane = (long long)f->ax[1].L * h;
    const size_t smem = fft_smem(f->ax[axis].L);
    LRES_CUDA_TRY(cudaFuncSetAttribute(fft_axis_kernel<INV, POISSON>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
    const unsigned blocks = (unsigned)(f->ax[1 - axis].L * ((h + kFftLines - 1) / kFftLines));
    fft_axis_kernel<INV, POISSON><<<blocks, kFftNT, smem, s>>>(f->ax[axis], h, axis ? plane : row, axis ? row : plane, w,
                                                               f->ax[1].k, f->ax[2].k, scale);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

int hartree_apply(FFT3* f, const double* dens, double* vh, double2* work, cudaStream_t s) {
    const double scale = 1.0 / ((double)f->ax[0].L * f->ax[1].L * f->ax[2].L);
    int rc = fft_real<false>(f, const_cast<double*>(dens), work, 1.0, s);
    if (!rc) rc = fft_axis<false, false>(f, 1, work, 1.0, s);
    if (!rc) rc = fft_axis<false, true>(f, 0, work, scale, s);
    if (!rc) rc = fft_axis<true, false>(f, 1, work, 1.0, s);
    if (!rc) rc = fft_real<true>(f, vh, work, 1.0, s);
    return rc;
}

// ---------------------------------------------------------------------------
// LDA: Slater exchange + Perdew-Zunger 1981 correlation (lrft/three_d.py:132-148)
//
// Bound by the FP64 pipe: two pow, a square root, a division and, inside the core, a logarithm
// cost ~350 FP64 instructions a point (0.59 ms at 108^3).  The roots and the reciprocal start
// from the FP32 functions (relative error below 1e-6) and take one step of Householder's
// iteration of order three in FP64, whose error is the cube of that: ~45 FP64 instructions,
// 0.14 ms at 108^3.
// ---------------------------------------------------------------------------

// n^(-1/3): y <- y (1 + e/3 + 2 e^2 / 9), e = 1 - n y^3
__device__ __forceinline__ double rcbrt_f64(double n) {
    const double y = (double)rcbrtf((float)n);
    const double e = fma(-n, y * y * y, 1.0);
    return fma(y * e, fma(e, 2.0 / 9.0, 1.0 / 3.0), y);
}
// a^(1/2) = a y, y = a^(-1/2): y <- y (1 + e/2 + 3 e^2 / 8), e = 1 - a y^2
__device__ __forceinline__ double sqrt_f64(double a) {
    const double y = (double)rsqrtf((float)a);
    const double e = fma(-a, y * y, 1.0);
    return a * fma(y * e, fma(e, 0.375, 0.5), y);
}
// 1/a: y <- y (1 + e + e^2), e = 1 - a y
__device__ __forceinline__ double recip_f64(double a) {
    const double y = (double)(1.0f / (float)a);
    const double e = fma(-a, y, 1.0);
    return fma(y * e, 1.0 + e, y);
}

__global__ void __launch_bounds__(256) lda_kernel(const double* dens, double* exc, double* vxc, long long n) {
    const double cx = -0.73855876638202240588;                       // -3/4 (3 / pi)^(1/3)
    const double cr = 0.62035049089940001667;                        // (3 / (4 pi))^(1/3)
    const double g = -0.1423, b1 = 1.0529, b2 = 0.3334;
    const double A = 0.0311, Bc = -0.048, C = 0.0020, D = -0.0116;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double nn = fmax(dens[i], 1e-14);
    double y, third;                                                  // n^(-1/3), n^(1/3)
    if (nn < 1e30) {
        y = rcbrt_f64(nn);
        third = nn * (y * y);
    } else {                                                          // (beyond the FP32 functions' range)
        third = cbrt(nn);
        y = 1.0 / third;
    }
    const double rs = cr * y;
    const double ex = cx * third;
    const double vx = 4.0 / 3.0 * ex;
    double ec, vc;
    if (rs >= 1.0) {
        const double sr = sqrt_f64(rs);
        const double den = 1.0 + b1 * sr + b2 * rs;
        const double inv = recip_f64(den);
        ec = g * inv;
        vc = ec * (1.0 + 7.0 / 6.0 * b1 * sr + 4.0 / 3.0 * b2 * rs) * inv;
    } else {
        const double lr = log(rs);
        ec = A * lr + Bc + C * rs * lr + D * rs;
        vc = A * lr + (Bc - A / 3.0) + 2.0 / 3.0 * C * rs * lr + (2.0 * D - C) / 3.0 * rs;
    }
    exc[i] = ex + ec;
    vxc[i] = vx + vc;
}

int lda_apply(long long n, const double* dens, double* exc, double* vxc, cudaStream_t s) {
    lda_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dens, exc, vxc, n);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

// ---------------------------------------------------------------------------
// ion potential: v(G) = -4 pi / G^2 * sum_a Z_a exp(-i G.R_a - G^2 rc_a^2 / 4) / vol,
// G = 0 removed, then v(r) = IFFT(v(G)) * ng (lrft/three_d.py:102-112,119)
//
// The exponential is a product over the axes, E_x E_y E_z with E = exp(-i k R - k^2 rc^2 / 4), so
// sincos and exp run per (atom, axis, wave number) instead of per (atom, G), and what is left is
// a contraction over the atoms on the FP64 pipe.  With Q = Z E_x E_z and E_y = c - i s, the sums
// U = sum Q c and V = sum Q s give the structure factor at both +k_y (U - iV) and -k_y (U + iV):
// two FP64 multiply-adds per (atom, G) plus the product Q, shared by the lanes' columns.
// Measured (1024 atoms, 64^3): 24.7 ms one sincos and exp per (atom, G) of the full grid, 15.7 ms
// of the half spectrum, 1.25 ms this way.
// ---------------------------------------------------------------------------

// E[a * ld + i], i <= L / 2, times Z_a on the x axis: the non-negative wave numbers of x and y; of z as
// numpy's (the highest of an even axis is negative: on that plane its sign goes with those of x and y).
__global__ void ion_axis_kernel(int natoms, int axis, int ld, const double* k, const double* pos, const double* Z,
                                const double* rc, double2* E) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= natoms * ld) return;
    const int a = idx / ld, i = idx - a * ld;
    const double q = axis == 2 ? k[i] : fabs(k[i]);
    double sn, cs;
    sincos(q * pos[3 * a + axis], &sn, &cs);
    const double amp = (axis == 0 ? Z[a] : 1.0) * exp(-q * q * rc[a] * rc[a] / 4.0);
    E[idx] = make_double2(amp * cs, -amp * sn);
}

constexpr int kIonCols = 4;                   // wave numbers k_y of a thread
constexpr int kIonWarps = 3;                  // groups of columns of a CTA

// Structure factor on the extended half grid T[(i * (2 l2) + j) * h + k]: i over 2 l1 - 1 signed wave
// numbers of the x axis (0 .. l1-1, then -1 .. -(l1-1)), j over +0 .. +(l2-1), -0 .. -(l2-1).
// Lane = (i, k), k fastest; a warp takes kIonCols columns.
__global__ void __launch_bounds__(32 * kIonWarps) ion_sum_kernel(int natoms, int l1, int l2, int h, const double2* Ex,
                                                                 const double2* Ey, const double2* Ez, double2* T) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows = (2 * l1 - 1) * h;
    const int row = min(blockIdx.x * 32 + lane, rows - 1);
    const int i = row / h, k = row - i * h;
    const int ia = i < l1 ? i : i - l1 + 1;
    const double sx = i < l1 ? 1.0 : -1.0;
    const int j0 = (blockIdx.y * kIonWarps + warp) * kIonCols;
    if (j0 >= l2) return;
    int jj[kIonCols];
    double2 U[kIonCols], V[kIonCols];
#pragma unroll
    for (int c = 0; c < kIonCols; ++c) {
        jj[c] = min(j0 + c, l2 - 1);
        U[c] = V[c] = make_double2(0.0, 0.0);
    }
#pragma unroll 2
    for (int a = 0; a < natoms; ++a) {
        double2 x = Ex[(long long)a * l1 + ia];
        x.y *= sx;
        const double2 z = Ez[(long long)a * h + k];
        const double2 q = cmulc(x, z);
#pragma unroll
        for (int c = 0; c < kIonCols; ++c) {
            const double2 y = Ey[(long long)a * l2 + jj[c]];       // (c, -s)
            U[c].x = fma(q.x, y.x, U[c].x);
            U[c].y = fma(q.y, y.x, U[c].y);
            V[c].x = fma(q.x, y.y, V[c].x);
            V[c].y = fma(q.y, y.y, V[c].y);
        }
    }
    if (blockIdx.x * 32 + lane >= rows) return;
    double2* const out = T + (long long)i * 2 * l2 * h + k;
#pragma unroll
    for (int c = 0; c < kIonCols; ++c) {
        if (j0 + c >= l2) break;
        out[(long long)(j0 + c) * h] = make_double2(U[c].x - V[c].y, U[c].y + V[c].x);        // U + i (-sum Q s)
        out[(long long)(l2 + j0 + c) * h] = make_double2(U[c].x + V[c].y, U[c].y - V[c].x);
    }
}

// v(G) on the half spectrum.  At the highest wave number of an even axis, where +k and -k are one,
// the mean of both signs (the real part of the full transform is wanted; on the planes k = 0 and
// n3 / 2 the real lines take it).
__global__ void ion_potential_kernel(int n1, int n2, int n3, const double* k1, const double* k2, const double* k3,
                                     double vol, const double2* T, double2* w) {
    const int h = n3 / 2 + 1, l1 = n1 / 2 + 1, l2 = n2 / 2 + 1;
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= (long long)n1 * n2 * h) return;
    const int k = (int)(idx % h), j = (int)((idx / h) % n2), i = (int)(idx / ((long long)n2 * h));
    const double kx = k1[i], ky = k2[j], kz = k3[k];
    const double G2 = kx * kx + ky * ky + kz * kz;
    // rows of the signed wave numbers: the highest one of an even axis is negative, as numpy's
    const int pi = kx >= 0.0 ? i : l1 - 1 + (n1 - i), pj = ky >= 0.0 ? j : l2 + (n2 - j);
    double2 v = T[((long long)pi * 2 * l2 + pj) * h + k];
    const bool inner = k > 0 && 2 * k != n3, ny1 = inner && 2 * i == n1, ny2 = inner && 2 * j == n2;
    if (ny1 || ny2) {
        const int qi = ny1 ? i : pi, qj = ny2 ? j : pj;            // the positive sign
        const double2 u = T[((long long)qi * 2 * l2 + qj) * h + k];
        v = make_double2(0.5 * (v.x + u.x), 0.5 * (v.y + u.y));
    }
    const double f = idx == 0 ? 0.0 : -4.0 * M_PI / G2 / vol;
    w[idx] = make_double2(f * v.x, f * v.y);
}

int ion_apply(FFT3* f, const double cell[3], int natoms, const double* pos, const double* Z, const double* rc,
              double* vion, double2* work, cudaStream_t s) {
    const FftAxis* ax = f->ax;
    const int l[3] = {ax[0].L / 2 + 1, ax[1].L / 2 + 1, ax[2].L / 2 + 1}, h = l[2];
    // the axis factors and the extended structure factor
    const size_t nE = (size_t)natoms * (l[0] + l[1] + l[2]), nT = (size_t)(2 * l[0] - 1) * 2 * l[1] * h;
    if (f->ion_size < nE + nT) {                   // kept with the plan, grown on demand
        if (f->d_ion) cudaFree(f->d_ion);
        f->d_ion = nullptr;
        f->ion_size = 0;
        if (cudaMalloc(&f->d_ion, sizeof(double2) * (nE + nT)) != cudaSuccess) {
            cudaGetLastError();
            lres_set_error("ion potential: allocation of %zu bytes failed", sizeof(double2) * (nE + nT));
            return LRES_ENOMEM;
        }
        f->ion_size = nE + nT;
    }
    double2* E[3] = {f->d_ion, nullptr, nullptr};
    E[1] = E[0] + (size_t)natoms * l[0];
    E[2] = E[1] + (size_t)natoms * l[1];
    double2* const T = E[0] + nE;
    for (int a = 0; a < 3; ++a)
        ion_axis_kernel<<<(natoms * l[a] + 127) / 128, 128, 0, s>>>(natoms, a, l[a], ax[a].k, pos, Z, rc, E[a]);
    const dim3 grid(((2 * l[0] - 1) * h + 31) / 32, (l[1] + kIonWarps * kIonCols - 1) / (kIonWarps * kIonCols));
    ion_sum_kernel<<<grid, 32 * kIonWarps, 0, s>>>(natoms, l[0], l[1], h, E[0], E[1], E[2], T);
    const long long n = (long long)ax[0].L * ax[1].L * h;
    ion_potential_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(ax[0].L, ax[1].L, ax[2].L, ax[0].k, ax[1].k,
                                                                     ax[2].k, cell[0] * cell[1] * cell[2], T, work);
    int r = LRES_OK;
    if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) {
        lres_set_error("ion potential: %s", cudaGetErrorString(e));
        r = LRES_ECUDA;
    }
    // (the inverse transform's 1/ng and the reference's factor ng cancel)
    if (!r) r = fft_axis<true, false>(f, 0, work, 1.0, s);
    if (!r) r = fft_axis<true, false>(f, 1, work, 1.0, s);
    if (!r) r = fft_real<true>(f, vion, work, 1.0, s);
    return r;
}

// ---------------------------------------------------------------------------
// Voronoi ownership with the reference's operation order (lrft/lcao3d.py:141-150):
// r = index * dx; dd = (r - c) - L * rint((r - c) / L); d2 = (dd0^2 + dd2^2) + dd1^2
// (numpy's einsum order for 3-vectors); strict '<' keeps the lowest centre index.
// Intrinsics with explicit rounding keep the compiler from fusing multiply-adds.
// ---------------------------------------------------------------------------
__global__ void voronoi_kernel(int n1, int n2, int n3, double dx, double L0, double L1, double L2, int ncent,
                               const double* cen, int* owner) {
    __shared__ double cs[3 * 256];
    const long long n = (long long)n1 * n2 * n3;
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int k = (int)(idx % n3), j = (int)((idx / n3) % n2), i = (int)(idx / ((long long)n2 * n3));
    const double r0 = __dmul_rn((double)i, dx), r1 = __dmul_rn((double)j, dx), r2 = __dmul_rn((double)k, dx);
    double best = INFINITY;
    int who = 0;
    for (int c0 = 0; c0 < ncent; c0 += 256) {
        __syncthreads();
        for (int t = threadIdx.x; t < 3 * 256 && 3 * c0 + t < 3 * ncent; t += blockDim.x) cs[t] = cen[3 * c0 + t];
        __syncthreads();
        const int cend = min(256, ncent - c0);
        if (idx < n) {
            for (int c = 0; c < cend; ++c) {
                double d0 = __dsub_rn(r0, cs[3 * c]), d1 = __dsub_rn(r1, cs[3 * c + 1]), d2 = __dsub_rn(r2, cs[3 * c + 2]);
                d0 = __dsub_rn(d0, __dmul_rn(L0, rint(__ddiv_rn(d0, L0))));
                d1 = __dsub_rn(d1, __dmul_rn(L1, rint(__ddiv_rn(d1, L1))));
                d2 = __dsub_rn(d2, __dmul_rn(L2, rint(__ddiv_rn(d2, L2))));
                const double q = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d2, d2)), __dmul_rn(d1, d1));
                if (q < best) {
                    best = q;
                    who = c0 + c;
                }
            }
        }
    }
    if (idx < n) owner[idx] = who;
}

int voronoi_apply(const int64_t shape[3], const double cell[3], int ncent, const double* centres, int* owner,
                  cudaStream_t s) {
    const long long n = shape[0] * shape[1] * shape[2];
    const double dx = cell[0] / (double)shape[0];
    const int blocks = (int)((n + 255) / 256);
    voronoi_kernel<<<blocks, 256, 0, s>>>((int)shape[0], (int)shape[1], (int)shape[2], dx, cell[0], cell[1], cell[2],
                                          ncent, centres, owner);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

}  // namespace lres
