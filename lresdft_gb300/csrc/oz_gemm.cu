// Batched FP64 matrix products on the tensor cores (sm_103a): C_w = op(A_w) op(B_w).
//
// GB300 issues 1.6 FP64 multiply-adds per clock and SM, its bf16 tensor cores ~1000 (mma.sync).  Every
// operand row (column of B) is scaled by a power of two to 63-bit fixed point and cut into 9 signed
// digits of 7 bits, exact in bf16 (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59 (2012) 95-118).  Products of digits sum exactly in the FP32 accumulators: 64 x 64 x
// 9 pairs x 448 terms < 2^24 (longer sums are taken in runs of 448).  The 45 digit pairs s + t <= 8
// are kept, summed by s + t in 9 accumulators and joined with two roundings.
//
// Error: per term at most 2^-58, as a rule 2^-62, of the product of the row's and the column's largest element
// (the eight pairs s + t = 9 that are dropped first, 64 x 64 each at most, in units of 2^-73), where the
// FP64 pipe errs by 2^-53 of the term itself: more accurate where the terms are of one size, less where a term
// lies more than 2^-5 to 2^-9 below that product and matters all the same.  What makes them so in the sums over
// basis functions, functions of different size, is taken out first (oz_balance_kernel).
// (8 digits: 2^-51 and 2^-55, a fifth less time, and the density of 54 windows 2.1e-14 off 64 bits against
// 1.6e-14, both with the asymmetry of H_W in them, which alone is most of the 1.6e-14.)
//
// Kernels: oz_slice_kernel writes the digits of an operand ([digit][row][k], k contiguous), each
// element once; oz_gemm_kernel, one CTA per 64 x 64 tile, stages 32 terms of all digits of both
// operands by cp.async (three stages of 72 KB) and issues 45 m16n8k16 products per warp tile and 16
// terms, 8 warps of 32 x 16.  The digit pairs bound it: 45 x 4096 flops per 2048 multiply-adds at
// ~600 TFLOP/s is 21 FP64 multiply-adds per clock and SM.  The windows go in batches, so that the
// digits take at most ~1 GB whatever the context's size.
//
// Measured (432 windows of 270-306 functions): the standard form's two products 23.5 -> 5.9 ms (54
// windows 3.7 -> 0.81), with the balance.
#include "common.cuh"
#include "launch.cuh"
#include "lres_internal.h"

#include <algorithm>

namespace lres {
namespace {

constexpr int kDig = 9;                       // digits of an operand
constexpr int kBits = 7;                      // bits of a digit
constexpr int kTop = kBits * (kDig - 1) + 5 - 52;    // bits below FP64's last of a row's largest value
constexpr unsigned long long bias_of(int digits) { return digits ? 64ull << (7 * (digits - 1)) | bias_of(digits - 1) : 0; }
constexpr unsigned long long kBias = bias_of(kDig);
constexpr int kOzT = 64;                      // tile edge
constexpr int kOzK = 32;                      // terms of a stage
constexpr int kOzStages = 3;
constexpr int kOzNT = 256;
constexpr int kOzRun = 448;                   // terms that sum exactly: kDig 64 64 kOzRun <= 2^24
constexpr int kOzBad = 1 << 20;               // exponent of a row with a non-finite value
constexpr int kOzNone = -(1 << 13);           // that of a row of zeros
constexpr int kStageBytes = 2 * kDig * kOzT * kOzK * 2;
constexpr int kOzSmem = kOzStages * kStageBytes;

// One operand of a batch: window w's matrix at X[off[w]], element (r, k) at r + k ld (k_contig = 0) or
// k + r ld (k_contig = 1), ld = rows or cols unless given.  Reflectors (OzForm::refl): the stored entry
// (row i, reflector l) counts below the diagonal, is 1 on it and 0 above.
struct Operand {
    const double* X;
    const long long* off;
    const int* rows;
    const int* cols;
    OzForm f;
};

__device__ __forceinline__ int ilogb_bits(double x) {
    const int e = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    return e == 0 ? -1022 : e - 1023;
}

// A digit's place is fixed by the largest element of its row, so an operand whose elements grow along k against a
// partner that falls (H_W and L^-T of basis functions of different size) would keep few bits of the terms
// that matter.  Term k is therefore taken as (a 2^s) (b 2^-s), s the exponent of its largest b: what is dropped
// then lies below the largest term of the product's row, and scaling the basis functions by powers of two
// changes no digit.  Non-finite elements are left out (their columns are given up anyway).  One read of B (the
// standard form's two products of 54 windows of 290 functions 0.76 -> 0.81 ms, of 432 5.6 -> 5.9 ms).
__global__ void __launch_bounds__(256) oz_balance_kernel(int w0, Operand b, int Kp, int* sk) {
    __shared__ int top[32];
    const int slot = blockIdx.y, w = w0 + slot, k0 = blockIdx.x * 32;
    const int R = b.rows[w], K = b.cols[w];
    if (k0 >= K) return;
    const double* const X = b.X + b.off[w];
    const long long ld = b.f.ld ? (b.f.ld[w] + 3) & ~3 : b.f.k_contig ? K : R;
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    auto exponent = [](double x) {
        const int e = ilogb_bits(x);
        return x != 0.0 && e < 1024 ? e : kOzNone;
    };
    if (tid < 32) top[tx] = kOzNone;
    __syncthreads();
    if (b.f.k_contig) {
        int e = kOzNone;
        if (k0 + tx < K) {
#pragma unroll 8
            for (int r = ty; r < R; r += 8) e = max(e, exponent(X[k0 + tx + r * ld]));
        }
        atomicMax(&top[tx], e);
    } else {
        for (int k = ty; k < 32; k += 8) {
            int e = kOzNone;
            if (k0 + k < K)
                for (int r = tx; r < R; r += 32) e = max(e, exponent(X[r + (k0 + k) * ld]));
            e = __reduce_max_sync(0xffffffffu, e);
            if (tx == 0) top[k] = e;
        }
    }
    __syncthreads();
    if (tid < 32) sk[(size_t)slot * Kp + k0 + tx] = max(top[tx], -2400);   // (b zero throughout: a is put out of the way)
}

// Digits of 32 rows of one window: dig[((slot * kDig + s) * Rp + r) * Kp + k], ex[slot * Rp + r]; element (r, k)
// times 2^(sign sk[slot Kp + k]), sign 0, 1 or -1.
template <int SIGN>
__global__ void __launch_bounds__(256) oz_slice_kernel(int w0, Operand o, int Rp, int Kp, const int* sk,
                                                       unsigned short* dig, int* ex) {
    __shared__ double tile[32][33];
    __shared__ int emax[32];
    const int slot = blockIdx.y, w = w0 + slot, r0 = blockIdx.x * 32;
    const int R = o.rows[w], K = o.cols[w];
    if (r0 >= (R + kOzT - 1) / kOzT * kOzT) return;                 // (tiles beyond are never read)
    const double* const X = o.X + o.off[w];
    const long long ld = o.f.ld ? (o.f.ld[w] + 3) & ~3 : o.f.k_contig ? K : R;
    auto at = [&](int r, int k) -> double {
        const int i = o.f.k_contig ? k : r, l = o.f.k_contig ? r : k;
        if (o.f.refl && i <= l) return i == l ? 1.0 : 0.0;
        return X[i + l * ld];
    };
    const int* const sw = SIGN ? sk + (size_t)slot * Kp : nullptr;
    auto exponent = [&](double x, int k) {
        const int e = ilogb_bits(x);
        return x == 0.0 ? kOzNone : e == 1024 ? kOzBad : SIGN ? e + SIGN * sw[k] : e;
    };
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    if (tid < 32) emax[tid] = kOzNone;
    __syncthreads();
    // the largest exponent of every row
    if (o.f.k_contig) {
        for (int r = ty; r < 32; r += 8) {
            int e = kOzNone;
            if (r0 + r < R)
                for (int k = tx; k < K; k += 32) e = max(e, exponent(at(r0 + r, k), k));
            e = __reduce_max_sync(0xffffffffu, e);
            if (tx == 0) emax[r] = e;
        }
    } else {
        int e = kOzNone;
        if (r0 + tx < R)
            for (int k = ty; k < K; k += 8) e = max(e, exponent(at(r0 + tx, k), k));
        atomicMax(&emax[tx], e);
    }
    __syncthreads();
    if (tid < 32) ex[(size_t)slot * Rp + r0 + tid] = emax[tid];
    const int r = tid >> 3, kq = (tid & 7) * 4;                     // this thread: row r, 4 terms
    const int E = emax[r];
    for (int k0 = 0; k0 < Kp; k0 += 32) {
        if (k0 >= (K + kOzK - 1) / kOzK * kOzK) break;
        __syncthreads();
        for (int q = ty; q < 32; q += 8) {
            double x = 0.0;
            if (o.f.k_contig) {
                if (r0 + q < R && k0 + tx < K) x = at(r0 + q, k0 + tx);
                tile[q][tx] = x;
            } else {
                if (r0 + tx < R && k0 + q < K) x = at(r0 + tx, k0 + q);
                tile[tx][q] = x;
            }
        }
        __syncthreads();
        unsigned d[kDig][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long b = __double_as_longlong(tile[r][kq + u]);
            const int ef = (int)((b >> 52) & 0x7ff);
            long long m = b & 0xfffffffffffffLL;
            if (ef) m |= 1LL << 52;
            const int s2 = SIGN && k0 + kq + u < K ? SIGN * sw[k0 + kq + u] : 0;
            const int sh = (ef ? ef - 1023 : -1022) + s2 - E + kTop;   // q = x 2^(52 + kTop + s2 - E) < 2^62
            long long q = 0;
            if (m == 0) q = 0;
            else if (sh >= 0) q = m << sh;                           // (sh <= kTop)
            else if (sh > -60) q = (m + (1LL << (-sh - 1))) >> -sh;
            if (b < 0) q = -q;
            // all digits at once: with 64 added at every place they are the 7-bit fields (the first may
            // be 128); to float by the exponent of 2^23, exact in bf16
            const unsigned long long z = (unsigned long long)q + kBias;
#pragma unroll
            for (int s = 0; s < kDig; ++s) {
                const unsigned t = (unsigned)(z >> (kBits * (kDig - 1 - s))) & (s ? 127u : 255u);
                d[s][u] = __float_as_uint(__uint_as_float(0x4B000000u | t) - 8388672.0f);   // 2^23 + 64
            }
        }
#pragma unroll
        for (int s = 0; s < kDig; ++s) {
            const uint2 v = make_uint2(__byte_perm(d[s][0], d[s][1], 0x7632), __byte_perm(d[s][2], d[s][3], 0x7632));
            *reinterpret_cast<uint2*>(dig + (((size_t)slot * kDig + s) * Rp + r0 + r) * Kp + k0 + kq) = v;
        }
    }
}

__device__ __forceinline__ void cp16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void ldm4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// sum_d acc_d 2^(-7 d) in units of 2^-14: groups of three exact in integers, joined with two roundings
__device__ __forceinline__ double oz_join(const float (&a)[kDig]) {
    static_assert(kDig == 9, "three groups of three");
    double g[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        long long v = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) v = (v << kBits) + __float2int_rn(a[3 * q + d]);
        // |v| < 2^39: to double by the exponent of 1.5 2^52
        g[q] = __longlong_as_double(0x4338000000000000LL + v) - 6755399441055744.0;
    }
    const double u = 4.76837158203125e-07;                          // 2^-21
    return fma(fma(g[2], u, g[1]), u, g[0]);
}

// KLIM: 1, B upper triangular (k <= column); 2, A lower triangular (k <= row) and the
// lower triangle of C only.  LONG: sums of more than kOzRun terms.
template <int KLIM, bool LONG>
__global__ void __launch_bounds__(kOzNT, 1) oz_gemm_kernel(int w0, const int* m_w, const int* n_w, const int* k_w,
                                                           int Rp, int Cp, int Kp, const unsigned short* da,
                                                           const unsigned short* db, const int* ea, const int* eb,
                                                           const long long* offC, double* C, int subtract) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int slot = blockIdx.z, w = w0 + slot;
    const int M = m_w[w], N = n_w[w], K = k_w[w];
    const int m0 = blockIdx.x * kOzT, n0 = blockIdx.y * kOzT;
    if (m0 >= M || n0 >= N) return;
    if (KLIM == 2 && m0 + kOzT - 1 < n0) return;
    const int kend = KLIM == 1 ? min(K, n0 + kOzT) : KLIM == 2 ? min(K, m0 + kOzT) : K;
    const int nk = (kend + kOzK - 1) / kOzK;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned short* const A = da + ((size_t)slot * kDig * Rp + m0) * Kp;
    const unsigned short* const B = db + ((size_t)slot * kDig * Cp + n0) * Kp;
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem);
    // stage: [operand][digit][row][4 chunks of 16 bytes], chunk c of row r at c ^ (r >> 1 & 3)
    auto load = [&](int kt, int buf) {
        const unsigned dst = sbase + buf * kStageBytes;
#pragma unroll
        for (int q = 0; q < 2 * kDig; ++q) {                        // (a digit of an operand: 256 chunks)
            const int c = tid & 3, r = tid >> 2, s = q % kDig, op = q / kDig;
            const unsigned short* src = op ? B + ((size_t)s * Cp + r) * Kp : A + ((size_t)s * Rp + r) * Kp;
            cp16(dst + (((op * kDig + s) * kOzT + r) * 4 + (c ^ (r >> 1 & 3))) * 16, src + kt * kOzK + c * 8);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 16;
    const int ar = (lane & 7) + ((lane >> 3) & 1) * 8, ac = lane >> 4;       // ldmatrix rows and chunks
    const int br = (lane & 7) + (lane >> 4) * 8, bc = (lane >> 3) & 1;
    float acc[kDig][2][2][4];
    double sum[2][2][4];
    auto clear = [&]() {
#pragma unroll
        for (int d = 0; d < kDig; ++d)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[d][i][j][e] = 0.0f;
    };
    auto flush = [&]() {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float a[kDig];
#pragma unroll
                    for (int d = 0; d < kDig; ++d) a[d] = acc[d][i][j][e];
                    const double x = oz_join(a);
                    if constexpr (LONG) sum[i][j][e] += x;
                    else sum[i][j][e] = x;
                }
    };
    if constexpr (LONG) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[i][j][e] = 0.0;
    }
    clear();
#pragma unroll
    for (int q = 0; q < kOzStages - 1; ++q) {
        if (q < nk) load(q, q);
        else asm volatile("cp.async.commit_group;\n" ::);
    }
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kOzStages - 2) : "memory");
        __syncthreads();                                            // stage kt here; stage kt - 1 consumed
        if (kt + kOzStages - 1 < nk) load(kt + kOzStages - 1, (kt + kOzStages - 1) % kOzStages);
        else asm volatile("cp.async.commit_group;\n" ::);
        const unsigned st = sbase + (kt % kOzStages) * kStageBytes;
#pragma unroll
        for (int h = 0; h < kOzK / 16; ++h) {
            unsigned bf[kDig][4];
#pragma unroll
            for (int t = 0; t < kDig; ++t) {
                const int r = wn + br;
                ldm4(bf[t], st + (((kDig + t) * kOzT + r) * 4 + ((2 * h + bc) ^ (r >> 1 & 3))) * 16);
            }
#pragma unroll
            for (int s = 0; s < kDig; ++s) {
                unsigned af[2][4];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int r = wm + 16 * i + ar;
                    ldm4(af[i], st + ((s * kOzT + r) * 4 + ((2 * h + ac) ^ (r >> 1 & 3))) * 16);
                }
#pragma unroll
                for (int t = 0; t < kDig - s; ++t)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int j = 0; j < 2; ++j) mma(acc[s + t][i][j], af[i], bf[t][2 * j], bf[t][2 * j + 1]);
            }
        }
        if constexpr (LONG) {
            if ((kt + 1) % (kOzRun / kOzK) == 0 && kt + 1 < nk) {
                flush();
                clear();
            }
        }
    }
    flush();
    double* const Cw = C + offC[w];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int gi = m0 + wm + 16 * i + (lane >> 2) + 8 * (e >> 1), gj = n0 + wn + 8 * j + 2 * (lane & 3) + (e & 1);
                if (gi >= M || gj >= N) continue;
                const int xa = ea[(size_t)slot * Rp + gi], xb = eb[(size_t)slot * Cp + gj];
                const int p = xa + xb - 24;                          // the join is in units of 2^(Ea + Eb - 10 - 14)
                double x = sum[i][j][e];
                if (xa >= kOzBad || xb >= kOzBad) x = __longlong_as_double(0x7ff8000000000000LL);
                else if (p > -960 && p < 960) x *= __longlong_as_double((long long)(p + 1023) << 52);
                else x = ldexp(x, p);
                double* const dst = Cw + gi + (long long)gj * M;
                *dst = subtract ? *dst - x : x;
            }
}

}  // namespace

void OzWork::release() {
    if (buf) cudaFree(buf);
    *this = OzWork{};
}

// Padded sizes and windows per batch: about 1 GB of digits at most (one window at least).
struct OzPlan {
    int Rp, Cp, Kp, batch;
    size_t perw;
};
static OzPlan oz_plan(int nwin, int mmax, int nmax, int kmax) {
    OzPlan p;
    p.Rp = (mmax + kOzT - 1) / kOzT * kOzT;
    p.Cp = (nmax + kOzT - 1) / kOzT * kOzT;
    p.Kp = (std::max(kmax, 1) + kOzK - 1) / kOzK * kOzK;
    p.perw = sizeof(unsigned short) * kDig * (size_t)(p.Rp + p.Cp) * p.Kp + sizeof(int) * (size_t)(p.Rp + p.Cp + p.Kp);
    p.batch = (int)std::min<size_t>({(size_t)nwin, std::max<size_t>(((size_t)1 << 30) / p.perw, 1), (size_t)65535});
    return p;
}

static int oz_alloc(OzWork& wk, size_t bytes) {
    wk.release();
    if (cudaMalloc(&wk.buf, bytes) != cudaSuccess) {
        cudaGetLastError();
        wk.buf = nullptr;
        lres_set_error("tensor-core FP64 product: allocation of %zu bytes failed", bytes);
        return LRES_ENOMEM;
    }
    wk.bytes = bytes;
    return LRES_OK;
}

// `bytes`, or as much of it as the device has, in halves.
static int oz_grow(OzWork& wk, size_t bytes, size_t least) {
    while (oz_alloc(wk, bytes) != LRES_OK) {
        if (bytes == least) return LRES_ENOMEM;
        bytes = std::max(bytes / 2, least);
    }
    return LRES_OK;
}

int oz_reserve(OzWork& wk, int nwin, int mmax, int nmax) {
    const OzPlan a = oz_plan(nwin, mmax, nmax, nmax), b = oz_plan(nwin, nmax, nmax, mmax);
    const size_t bytes = std::max(a.perw * a.batch, b.perw * b.batch);
    return wk.bytes >= bytes ? LRES_OK : oz_grow(wk, bytes, std::max(a.perw, b.perw));
}

int oz_gemm(OzWork& wk, int nwin, int mmax, int nmax, int kmax, const int* m_w, const int* n_w, const int* k_w,
            const double* A, const long long* offA, OzForm fa, const double* B, const long long* offB, OzForm fb,
            double* C, const long long* offC, int klim, bool subtract, bool balance, size_t smem_budget, cudaStream_t s) {
    if (nwin < 1 || mmax < 1 || nmax < 1) return LRES_OK;
    if ((size_t)kOzSmem > smem_budget) {
        lres_set_error("tensor-core FP64 product needs %d B of shared memory", kOzSmem);
        return LRES_EINVAL;
    }
    // within the workspace that is there (a captured graph keeps its address): it grows only where one
    // window does not fit
    const OzPlan p = oz_plan(nwin, mmax, nmax, kmax);
    if (wk.bytes < p.perw)
        if (int rc = oz_grow(wk, p.perw * p.batch, p.perw)) return rc;
    const int Rp = p.Rp, Cp = p.Cp, Kp = p.Kp, batch = (int)std::min<size_t>(p.batch, wk.bytes / p.perw);
    unsigned short* const da = static_cast<unsigned short*>(wk.buf);
    // (a Gram product has one operand)
    const bool same = A == B && offA == offB && m_w == n_w && fa.k_contig == fb.k_contig && fa.ld == fb.ld &&
                      fa.refl == fb.refl && Rp == Cp;
    unsigned short* const db = same ? da : da + (size_t)batch * kDig * Rp * Kp;
    int* const ea = reinterpret_cast<int*>(da + (size_t)batch * kDig * (Rp + Cp) * Kp);
    int* const eb = same ? ea : ea + (size_t)batch * Rp;
    int* const sk = balance && !same ? ea + (size_t)batch * (Rp + Cp) : nullptr;
    const bool lng = kmax > kOzRun;
    int per_sm = 0;
    auto launch = [&](auto kern, int w0, int nb) {
        const dim3 grid((mmax + kOzT - 1) / kOzT, (nmax + kOzT - 1) / kOzT, nb);
        kern<<<grid, kOzNT, kOzSmem, s>>>(w0, m_w, n_w, k_w, Rp, Cp, Kp, da, db, ea, eb, offC, C, subtract ? 1 : 0);
    };
    for (int w0 = 0; w0 < nwin; w0 += batch) {
        const int nb = std::min(batch, nwin - w0);
        const Operand oa{A, offA, m_w, k_w, fa}, ob{B, offB, n_w, k_w, fb};
        if (sk) oz_balance_kernel<<<dim3(Kp / 32, nb), 256, 0, s>>>(w0, ob, Kp, sk);
        (sk ? oz_slice_kernel<1> : oz_slice_kernel<0>)<<<dim3(Rp / 32, nb), 256, 0, s>>>(w0, oa, Rp, Kp, sk, da, ea);
        if (!same)
            (sk ? oz_slice_kernel<-1> : oz_slice_kernel<0>)<<<dim3(Cp / 32, nb), 256, 0, s>>>(w0, ob, Cp, Kp, sk, db, eb);
        LRES_CUDA_TRY(cudaGetLastError());
#define OZ_RUN(KL, LG)                                                                  \
    do {                                                                                \
        if (int rc = prepare_kernel<oz_gemm_kernel<KL, LG>>(kOzNT, kOzSmem, &per_sm)) return rc; \
        launch(oz_gemm_kernel<KL, LG>, w0, nb);                                         \
    } while (0)
        if (klim == 1) {
            if (lng) OZ_RUN(1, true);
            else OZ_RUN(1, false);
        } else if (klim == 2) {
            if (lng) OZ_RUN(2, true);
            else OZ_RUN(2, false);
        } else {
            if (lng) OZ_RUN(0, true);
            else OZ_RUN(0, false);
        }
#undef OZ_RUN
        LRES_CUDA_TRY(cudaGetLastError());
    }
    return LRES_OK;
}

// ---------------------------------------------------------------------------
// rows through the Householder reflectors, compact WY panels of 128 (FP64)
// ---------------------------------------------------------------------------
//
// Y <- Y - ((Y V) T) V^T per panel, three products on the tensor cores; V^T V (for T) a fourth, once per
// Hamiltonian for all row sets.  Panels of 128 rather than the 32 of tri_apply_kernel: a product over
// 32 terms would spend more on the digits and the joining than on its terms.  The FP64 pipe does the
// T recurrence only.  Measured (with T): 54 windows of 256 rows 7.5 -> 1.86 ms, 432 windows 32.5 ->
// 11.4 ms.

namespace {

constexpr int kTNT = 4 * kOzPanel;             // four threads a row
constexpr int kTLd = kOzPanel + 8;            // (four columns of eight rows in 16 banks each)

// T of every (window, panel) from G = V^T V in its slot: T_ll = tau_l, T[0:l, l] = -tau_l T[0:l, 0:l] G[0:l, l],
// T in place of G (column-major, zero below the diagonal).  T by columns and G's upper triangle packed by
// columns in shared memory.  Bound by the FP64 pipe (q^3 / 6 multiply-adds, 80 clocks a warp's on a quarter of
// the SM): a row's sum is dealt to four threads of a warp, so that the rows of a warp have nearly the same
// length and sixteen warps share the pipe (a thread per row, the first warp's the longest: 432 windows of 290
// functions 2.54 -> 1.17 ms, 54 windows 0.43 -> 0.20 ms).
__global__ void __launch_bounds__(kTNT) oz_tfactor_kernel(int nwin, const int* q_w, const long long* offT,
                                                          const long long* offN, const double* tau, int qmax, double* T) {
    extern __shared__ __align__(128) unsigned char smem[];
    double* const Ts = reinterpret_cast<double*>(smem);             // [qmax][kTLd]
    double* const Gs = Ts + (size_t)qmax * kTLd;                    // (a, b), a <= b at b (b + 1) / 2 + a
    const int w = blockIdx.x % nwin, p = blockIdx.x / nwin, a = threadIdx.x >> 2, part = threadIdx.x & 3;
    const int q = q_w[blockIdx.x];
    if (q < 1) return;
    double* const Tw = T + offT[blockIdx.x];
    for (int b = threadIdx.x >> 7; b < q; b += kTNT / kOzPanel) {
        const int r = threadIdx.x & (kOzPanel - 1);
        if (r <= b) Gs[b * (b + 1) / 2 + r] = Tw[r + (long long)b * q];
    }
    __syncthreads();
    const double* const tw = tau + offN[w] + p * kOzPanel;
    const int first = a & ~7;                                       // the warp's first row
    for (int l = 0; l < q; ++l) {
        const double tl = tw[l];
        double val = a == l ? tl : 0.0;
        if (first < l) {                                            // (the same for the warp)
            const double* const g = Gs + l * (l + 1) / 2;
            double s = 0.0;
            for (int b = a + part; b < l; b += 4) s = fma(Ts[b * kTLd + a], g[b], s);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (a < l) val = -tl * s;
        }
        if (part == 0) Ts[l * kTLd + a] = val;
        __syncwarp();
    }
    __syncthreads();
    for (int b = threadIdx.x >> 7; b < q; b += kTNT / kOzPanel) {
        const int r = threadIdx.x & (kOzPanel - 1);
        if (r < q) Tw[r + (long long)b * q] = Ts[b * kTLd + r];
    }
}

}  // namespace

void OzRows::release() {
    for (void* p : {(void*)q, (void*)r, (void*)offV, (void*)offT, (void*)T})
        if (p) cudaFree(p);
    *this = OzRows{};
}
void OzRowSet::release() {
    for (void* p : {(void*)offS, (void*)offY, (void*)S, (void*)S2})
        if (p) cudaFree(p);
    *this = OzRowSet{};
}

int oz_tfactors(OzWork& wk, const OzRows& o, int nwin, int nmax, const int* n_w, const double* A, const double* tau,
                const long long* offN, size_t smem_budget, cudaStream_t s) {
    for (int p = 0; p < o.panels; ++p) {
        const int j0 = p * kOzPanel, qm = std::min(kOzPanel, nmax - 2 - j0), rm = nmax - 1 - j0;
        const int *q = o.q + (size_t)p * nwin, *r = o.r + (size_t)p * nwin;
        const long long *offV = o.offV + (size_t)p * nwin, *offT = o.offT + (size_t)p * nwin;
        const OzForm v(true, n_w, true);
        if (int rc = oz_gemm(wk, nwin, qm, qm, rm, q, q, r, A, offV, v, A, offV, v, o.T, offT, 0, false, false, smem_budget, s))
            return rc;
    }
    if (o.panels) {
        const int qm = std::min(kOzPanel, nmax - 2);
        const size_t smem = sizeof(double) * ((size_t)qm * kTLd + (size_t)qm * (qm + 1) / 2);
        int per_sm = 0;
        if (int rc = prepare_kernel<oz_tfactor_kernel>(kTNT, smem, &per_sm)) return rc;
        oz_tfactor_kernel<<<(unsigned)nwin * o.panels, kTNT, smem, s>>>(nwin, o.q, o.offT, offN, tau, qm, o.T);
        LRES_CUDA_TRY(cudaGetLastError());
    }
    return LRES_OK;
}

int oz_rows(OzWork& wk, const OzRows& o, const OzRowSet& rs, int nwin, int nmax, const int* n_w, const int* m_w,
            const double* A, double* Y, size_t smem_budget, cudaStream_t s) {
    for (int p = 0; p < o.panels; ++p) {
        const int j0 = p * kOzPanel, qm = std::min(kOzPanel, nmax - 2 - j0), rm = nmax - 1 - j0;
        const int *q = o.q + (size_t)p * nwin, *r = o.r + (size_t)p * nwin;
        const long long *offV = o.offV + (size_t)p * nwin, *offT = o.offT + (size_t)p * nwin;
        const long long* offY = rs.offY + (size_t)p * nwin;
        if (int rc = oz_gemm(wk, nwin, rs.mmax, qm, rm, m_w, q, r, Y, offY, OzForm(false), A, offV,
                             OzForm(true, n_w, true), rs.S, rs.offS, 0, false, false, smem_budget, s))
            return rc;
        if (int rc = oz_gemm(wk, nwin, rs.mmax, qm, qm, m_w, q, q, rs.S, rs.offS, OzForm(false), o.T, offT,
                             OzForm(true), rs.S2, rs.offS, 1, false, false, smem_budget, s))
            return rc;
        if (int rc = oz_gemm(wk, nwin, rs.mmax, rm, qm, m_w, r, q, rs.S2, rs.offS, OzForm(false), A, offV,
                             OzForm(false, n_w, true), Y, offY, 0, true, false, smem_budget, s))
            return rc;
    }
    return LRES_OK;
}

}  // namespace lres
