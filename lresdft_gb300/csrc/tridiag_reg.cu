// Householder tridiagonalisation with the window held on the SM (FP32, sm_103a).
//
// What bounds it: the chain of n columns, each of which needs the whole trailing matrix once
// (q = A x) before the next can start.  tri_reduce_kernel (tridiag.cu) reads that matrix from
// an L2-resident copy for every column: 5 us a column for a window alone on its SM.  Here the
// lower triangle stays on the SM for all columns, and a column costs shared-memory latency and
// FP32 issue only.
//
// Layout: 8 warps; warp p, lane q hold the elements (row 8a + p, column 32b + q), a >= 4b: the
// lower triangle in 32 x 32 blocks, the diagonal blocks whole.  The cyclic rows and columns
// keep every thread busy while the trailing matrix shrinks.  The window is padded at the front
// to N = 32 NB rows.  The last 8 column blocks (256 columns) live in registers (144 of a
// thread's 255), the blocks before them in shared memory, each thread's elements in its own
// slots ([element][thread]: no bank conflicts): NB <= 12, windows of up to 384 functions in one
// CTA.  Larger windows reduce their first columns with tri_reduce_kernel.  When the reduction
// reaches a register block, that block moves to the slots that the first block has left, so
// that any thread can read the current column.  An off-diagonal element a_ij serves the row
// product (a_ij x_j, summed over the lanes by a butterfly that halves the rows at each step)
// and the column product (a_ij x_i, summed over the warps through shared memory); the diagonal
// blocks serve rows only.
//
// Rank-2 updates wait for the panel of 4 columns and are subtracted as one sum: applied one by
// one they round every element twice a column and double the error of the density (7.3e-7
// against 3.1e-7 in an emulation of the arithmetic; panels of 4: 3.0e-7).
//
// Per column c, two barriers:
//   S  (panel start: A -= sum of v w^T + w v^T over the panel); q = A x over the unscaled column
//      x on the rows >= c+2, x^T A x, |x|^2 (by every warp: beta, tau, scal are formed beside
//      the products), w_l^T x and v_l^T x of the panel (a warp per pair)
//   C  y = A v = A e_{c+1} + scal q - V (W^T v) - W (V^T v);
//      v^T y = a_{c+1,c+1} + 2 scal q_{c+1} + scal^2 x^T A x - 2 (V^T v)(W^T v) (q_{c+1} = x^T A e_{c+1});
//      w = tau y - tau^2/2 (v^T y) v; column c+1 of the current matrix
// Sums: at most 12 products in a thread, then trees.
//
// Measured: 54 windows of 276-300 functions 1.46 -> 0.53 ms, 1024 windows of 264-312 6.7 -> 3.5 ms,
// 1024 of 198-366 6.9 -> 4.0 ms, 512 of 396 (12 columns by tri_reduce_kernel first) 9.6 -> 5.2 ms.
// A column takes 3200 clocks, about 700 of them the panel's update, 700 step C; the code is
// written out for every live block count, without which branches and index arithmetic were 60 %
// of the instructions (0.89 ms).
#include "common.cuh"
#include "launch.cuh"
#include "lres_internal.h"

#include <algorithm>
#include <type_traits>

namespace lres {
namespace {

constexpr int kRegNT = 256, kRegNW = kRegNT / 32;
constexpr int kRegBlk = 8;                    // column blocks in registers
constexpr int kRegSlots = 2 * kRegBlk * (kRegBlk + 1);
constexpr int kRegMaxNB = 12;                 // column blocks in all
static_assert(32 * kRegMaxNB == kTriRegMax, "windows of the resident reduction");

template <int I, int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}

// Register slot of row slot a, column block b (both relative to the register part).
constexpr int reg_slot(int a, int b) { return 4 * b * kRegBlk - 2 * b * (b - 1) + a - 4 * b; }

// Shared slots before column block b of a window of NB blocks.
__host__ __device__ constexpr int sh_slot(int b, int NB) { return 4 * b * NB - 2 * b * (b - 1); }

// Slots of the shared part; one register block at a time needs 4 kRegBlk of them.
__host__ __device__ constexpr int sh_slots(int NB) {
    return sh_slot(NB - kRegBlk, NB) > 4 * kRegBlk ? sh_slot(NB - kRegBlk, NB) : 4 * kRegBlk;
}
// Row-ordered copy of x: row 8a + p at p * row_ld(NB) + a (16-byte groups of a warp's rows).
__host__ __device__ constexpr int row_ld(int NB) { return 4 * NB + 4; }

// Shared memory of windows of NB column blocks, in floats.
inline size_t reg_smem_floats(int NB) {
    const int N = 32 * NB;
    return (size_t)(8 + 1 + 1 + kRegNW) * N + kRegNW * row_ld(NB) + 64 + kRegNT + (size_t)kRegNT * sh_slots(NB);
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Sums of NR values (rows) over the lanes: halves the rows held at each step, then sums the
// groups of lanes that hold the same row.  Lane group g (of NR) ends with row rowof(lane).
template <int NR>
__device__ __forceinline__ float rows_sum(float* r, int lane) {
    int o = 16;
#pragma unroll
    for (int half = NR / 2; half; half >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float send = up ? r[i] : r[i + half];
            const float keep = up ? r[i + half] : r[i];
            r[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float x = r[0];
#pragma unroll
    for (; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

struct TriRegParams {
    int nwin;
    const int* order;        // windows, largest first
    int* counter;            // work-queue head (zeroed before launch)
    const int* n_w;
    const long long* offC;   // standard-form blocks (n x n, column-major)
    const long long* offA;   // working blocks (ld x n, ld = n rounded up to 4)
    const long long* offN;
    const float* H;          // standard-form matrices (lower triangle read)
    float* A;                // on return the reflectors below the subdiagonal; for windows beyond
                             // kTriRegMax on entry the matrix reduced up to column first
    float *d, *e, *tau;
    int* status;
    int nb;                  // panel width of the reduction that came before (large windows)
    int NBmax;               // column blocks that the launch's shared memory holds
};

__global__ void __launch_bounds__(kRegNT, 1) tri_reduce_reg_kernel(TriRegParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int item_sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (;;) {
        if (tid == 0) item_sh = atomicAdd(p.counter, 1);
        __syncthreads();
        const int it = item_sh;
        if (it >= p.nwin) return;
        const int w = p.order[it];
        const int n = p.n_w[w];
        // columns before `first` are done (windows beyond the resident size)
        const int first = n > kTriRegMax ? (n - kTriRegMax + p.nb - 1) / p.nb * p.nb : 0;
        const int nt = n - first;
        const int NB = max(kRegBlk, (nt + 31) >> 5);
        if (n < 1 || NB > p.NBmax) {
            if (tid == 0) atomicOr(p.status, ST_BAD_SHAPE);
            __syncthreads();
            continue;
        }
        const int N = 32 * NB, pad = N - nt, B0 = NB - kRegBlk;
        float* const VW = reinterpret_cast<float*>(smem_raw);       // [2][N][4] (v, w) of the panel's columns
        float* const xs = VW + 8 * N;                               // [N] x, zero on rows < c+2
        float* const xr = xs + N;                                   // [8][row_ld] x by rows of a warp
        float* const rowp = xr + kRegNW * row_ld(NB);               // [N] row products of q
        float* const colp = rowp + N;                               // [8][N] column products of q
        float* const xq = colp + kRegNW * N;                        // [256] x^T A x by thread
        float* const dots = xq + kRegNT;                            // [8] (v_l^T x, w_l^T x)
        float* const pub = dots + 8;                                // alpha = x_{c+1}, tau, scal
        float* const S = dots + 64 + tid;                           // [slot][256]: this thread's
        const int ld = (n + 3) & ~3;
        float* const Aw = p.A + p.offA[w];
        const float* const src = first ? Aw : p.H + p.offC[w];
        const long long lds = first ? ld : n;
        const int goff = first - pad;                               // window index of local index 0
        float* const dw = p.d + p.offN[w];
        float* const ew = p.e + p.offN[w];
        float* const tw = p.tau + p.offN[w];

        // The lower triangle by tiles of 32 columns x 128 rows through shared memory (columns are read
        // coalesced; an element above the diagonal of a diagonal block is the mirrored one).
        float* const tile = VW;                                     // [32][129] over the vectors below S
        auto load_tile = [&](int b, int i0) {                       // rows i0.. of column block b
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 32 / kRegNW; ++k) {
                const int j = warp + k * kRegNW, gj = 32 * b + j - pad;
#pragma unroll
                for (int r = 0; r < 128; r += 32) {
                    const int i = i0 + r + lane;
                    tile[j * 129 + r + lane] =
                        i < N && gj >= 0 && i >= 32 * b + j ? src[(goff + i) + (long long)(first + gj) * lds] : 0.0f;
                }
            }
            __syncthreads();
        };
        auto element = [&](int i, int j) {                          // (i, j) within the tile, diagonal block at its top
            return i >= j || i >= 32 ? tile[j * 129 + i] : tile[i * 129 + j];
        };
        float A[kRegSlots];
        static_for<0, kRegBlk>([&](auto bc) {
            constexpr int b = decltype(bc)::value;
            static_for<0, (kRegBlk - b + 3) / 4>([&](auto tc) {
                constexpr int t = decltype(tc)::value;
                load_tile(B0 + b, 32 * (B0 + b) + 128 * t);
                static_for<0, 16>([&](auto rc) {
                    constexpr int r = decltype(rc)::value, a = 4 * b + 16 * t + r;
                    if constexpr (a < 4 * kRegBlk) {
                        if constexpr (t == 0 && r < 4) A[reg_slot(a, b)] = element(8 * r + warp, lane);
                        else A[reg_slot(a, b)] = tile[lane * 129 + 8 * r + warp];
                    }
                });
            });
        });
        for (int b = 0; b < B0; ++b)
            for (int a0 = 4 * b; a0 < 4 * NB; a0 += 16) {
                load_tile(b, 8 * a0);
                for (int r = 0; r < min(16, 4 * NB - a0); ++r)
                    S[(sh_slot(b, NB) + a0 + r - 4 * b) * kRegNT] =
                        a0 == 4 * b ? element(8 * r + warp, lane) : tile[lane * 129 + 8 * r + warp];
            }
        __syncthreads();

        // column c on the elements N-1-tid and N-257-tid (the second die first)
        float x[2];
        auto publish = [&](int i, int c, float xi) {                // x_i of column c
            if (i == c) {
                dw[goff + c] = xi;
                if (!isfinite(xi)) atomicOr(p.status, ST_ZERO_PIVOT);
            }
            if (i == c + 1) pub[0] = xi;
            const float xm = i >= c + 2 ? xi : 0.0f;
            xs[i] = xm;
            xr[(i & 7) * row_ld(NB) + (i >> 3)] = xm;
        };
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = N - 1 - tid - u * kRegNT;
            x[u] = i >= pad ? src[(goff + i) + (long long)first * lds] : 0.0f;
            if (i >= 0) publish(i, pad, x[u]);
        }
        __syncthreads();

        // One column.  SB: the register block that column c+1 lies in (it is then in shared memory
        // and the blocks before it are done), -1 while column c+1 lies in the shared part: the code
        // of each value is straight.
        auto column_step = [&](auto sbc, int c) {
            constexpr int SB = decltype(sbc)::value;
            // ---- S: rows and columns >= c+1
            const int jj = (c - pad) & 3;                           // pairs (v_l, w_l), l < jj, pending
            const int bs = SB >= 0 ? B0 + SB : (c + 1) >> 5;        // first live column block
            // slots of block b, row slot a (absolute)
            auto slot = [&](int a, int b) {
                return SB >= 0 ? (a - 4 * (B0 + SB)) * kRegNT : (sh_slot(b, NB) + a - 4 * b) * kRegNT;
            };
            const int bl = SB >= 0 ? bs : B0 - 1;                   // last live block in shared memory

            if (jj == 0 && c > pad) {
                // A -= sum_l v_l w_l^T + w_l v_l^T, rows in fours
                float rvw[4][8];
                auto rows4 = [&](int i0) {
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float4 f = *reinterpret_cast<const float4*>(VW + 4 * (i0 + 8 * r));
                        const float4 h = *reinterpret_cast<const float4*>(VW + 4 * (N + i0 + 8 * r));
                        rvw[r][0] = f.x; rvw[r][1] = f.y; rvw[r][2] = f.z; rvw[r][3] = f.w;
                        rvw[r][4] = h.x; rvw[r][5] = h.y; rvw[r][6] = h.z; rvw[r][7] = h.w;
                    }
                };
                auto upd = [&](float e, int r, const float4& f, const float4& h) {
                    float t = rvw[r][0] * f.y;
                    t = fmaf(rvw[r][1], f.x, t);
                    t = fmaf(rvw[r][2], f.w, t);
                    t = fmaf(rvw[r][3], f.z, t);
                    t = fmaf(rvw[r][4], h.y, t);
                    t = fmaf(rvw[r][5], h.x, t);
                    t = fmaf(rvw[r][6], h.w, t);
                    t = fmaf(rvw[r][7], h.z, t);
                    return e - t;
                };
                auto shared_blocks = [&](int a0, int blast) {       // rows 8 a0 + p .. of blocks bs..blast
                    for (int b = bs; b <= blast; ++b) {
                        const float4 f = *reinterpret_cast<const float4*>(VW + 4 * (32 * b + lane));
                        const float4 h = *reinterpret_cast<const float4*>(VW + 4 * (N + 32 * b + lane));
                        float* const sl = S + slot(a0, b);
#pragma unroll
                        for (int r = 0; r < 4; ++r) sl[r * kRegNT] = upd(sl[r * kRegNT], r, f, h);
                    }
                };
                if constexpr (SB < 0) {
                    for (int g = bs; g < B0; ++g) {
                        rows4(32 * g + warp);
                        shared_blocks(4 * g, g);
                    }
                }
                static_for<(SB > 0 ? SB : 0), kRegBlk>([&](auto gc) {
                    constexpr int g = decltype(gc)::value;
                    rows4(32 * (B0 + g) + warp);
                    shared_blocks(4 * (B0 + g), bl);
                    static_for<SB + 1, g + 1>([&](auto bc) {
                        constexpr int b = decltype(bc)::value;
                        const float4 f = *reinterpret_cast<const float4*>(VW + 4 * (32 * (B0 + b) + lane));
                        const float4 h = *reinterpret_cast<const float4*>(VW + 4 * (N + 32 * (B0 + b) + lane));
                        static_for<0, 4>([&](auto rc) {
                            constexpr int r = decltype(rc)::value;
                            float& e = A[reg_slot(4 * g + r, b)];
                            e = upd(e, r, f, h);
                        });
                    });
                });
            }

            // x on this lane's columns
            float xc[kRegBlk];
            static_for<(SB > 0 ? SB : 0), kRegBlk>([&](auto bc) {
                constexpr int b = decltype(bc)::value;
                xc[b] = xs[32 * (B0 + b) + lane];
            });
            // one sum over the rows for each warp: the panel's v_l^T x (warp 2l) and w_l^T x (2l + 1),
            // |x|^2 and the reflector's scalars (the last warp)
            if (warp < 2 * jj || warp == kRegNW - 1) {
                const float* const vec = VW + (warp >> 2) * 4 * N + (warp & 3);
                const bool norm = warp == kRegNW - 1;
                float sum = 0.0f;
                static_for<(SB > 0 ? SB : 0), kRegBlk>([&](auto bc) {
                    constexpr int b = decltype(bc)::value;
                    sum = fmaf(norm ? xc[b] : vec[4 * (32 * (B0 + b) + lane)], xc[b], sum);
                });
                if constexpr (SB < 0) {
                    for (int i = 32 * bs + lane; i < 32 * B0; i += 32) sum = fmaf(norm ? xs[i] : vec[4 * i], xs[i], sum);
                }
                sum = warp_sum(sum);
                if (!norm) {
                    if (lane == 0) dots[warp] = sum;
                } else {
                    const float alpha = pub[0];
                    float beta = alpha, tau = 0.0f, scal = 0.0f;
                    if (sum > 0.0f) {
                        const float nrm = sqrtf(alpha * alpha + sum);
                        beta = alpha >= 0.0f ? -nrm : nrm;
                        tau = (beta - alpha) / beta;
                        scal = 1.0f / (alpha - beta);
                    }
                    if (lane == 0) {
                        pub[1] = tau;
                        pub[2] = scal;
                        ew[goff + c] = beta;
                        tw[goff + c] = tau;
                        if (!isfinite(beta)) atomicOr(p.status, ST_ZERO_PIVOT);
                    }
                }
            }

            float qx = 0.0f;                                        // x^T A x of this thread's elements
            // rows of the shared part, 32 at a time
            if constexpr (SB < 0) {
              for (int g = bs; g < B0; ++g) {
                const float4 x4 = *reinterpret_cast<const float4*>(xr + warp * row_ld(NB) + 4 * g);
                const float rx[4] = {x4.x, x4.y, x4.z, x4.w};
                float rp[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                for (int b = bs; b <= g; ++b) {
                    const float xb = xs[32 * b + lane];
                    const float* const sl = S + slot(4 * g, b);
                    float cp = 0.0f;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float e = sl[r * kRegNT];
                        rp[r] = fmaf(e, xb, rp[r]);
                        cp = fmaf(e, rx[r], cp);
                    }
                    float* const dst = colp + warp * N + 32 * b + lane;
                    if (b == g) {
                        *dst = 0.0f;                                // the block's first rows: its diagonal
                    } else {
                        *dst += cp;
                        qx = fmaf(cp, xb, qx);
                    }
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) qx = fmaf(rp[r], rx[r], qx);
                const float sum = rows_sum<4>(rp, lane);
                if ((lane & 7) == 0) rowp[32 * g + 8 * (lane >> 3) + warp] = sum;
              }
            }
            // rows of the register part, 64 at a time
            float cpr[kRegBlk];
#pragma unroll
            for (int b = 0; b < kRegBlk; ++b) cpr[b] = 0.0f;
            constexpr int NR = SB >= 0 ? 8 * (kRegBlk / 2 - SB / 2) : 8;
            float rows[NR];
            static_for<(SB > 0 ? SB / 2 : 0), kRegBlk / 2>([&](auto gc) {
                constexpr int g = decltype(gc)::value;
                const float* const xw = xr + warp * row_ld(NB) + 4 * B0 + 8 * g;
                const float4 x4 = *reinterpret_cast<const float4*>(xw), x5 = *reinterpret_cast<const float4*>(xw + 4);
                const float rx[8] = {x4.x, x4.y, x4.z, x4.w, x5.x, x5.y, x5.z, x5.w};
                constexpr int R0 = SB >= 0 ? 8 * (g - SB / 2) : 0;
                float* const rp = rows + R0;
#pragma unroll
                for (int r = 0; r < 8; ++r) rp[r] = 0.0f;
                if constexpr (SB >= 0) {
                    // the block in shared memory: its first rows are its diagonal (rows only)
                    static_for<0, 8>([&](auto rc) {
                        constexpr int r = decltype(rc)::value, a = 8 * g + r;
                        if constexpr (a >= 4 * SB) {
                            const float e = S[(a - 4 * SB) * kRegNT];
                            rp[r] = fmaf(e, xc[SB], rp[r]);
                            if constexpr (a / 4 != SB) cpr[SB] = fmaf(e, rx[r], cpr[SB]);
                        }
                    });
                } else {
                    for (int b = bs; b < B0; ++b) {
                        const float xb = xs[32 * b + lane];
                        const float* const sl = S + slot(4 * B0 + 8 * g, b);
                        float cp = 0.0f;
#pragma unroll
                        for (int r = 0; r < 8; ++r) {
                            const float e = sl[r * kRegNT];
                            rp[r] = fmaf(e, xb, rp[r]);
                            cp = fmaf(e, rx[r], cp);
                        }
                        colp[warp * N + 32 * b + lane] += cp;
                        qx = fmaf(cp, xb, qx);
                    }
                }
                static_for<SB + 1, 2 * g + 2>([&](auto bc) {
                    constexpr int b = decltype(bc)::value;
                    static_for<0, 8>([&](auto rc) {
                        constexpr int r = decltype(rc)::value, a = 8 * g + r;
                        if constexpr (a >= 4 * b) {
                            const float e = A[reg_slot(a, b)];
                            rp[r] = fmaf(e, xc[b], rp[r]);
                            if constexpr (a / 4 != b) cpr[b] = fmaf(e, rx[r], cpr[b]);
                        }
                    });
                });
#pragma unroll
                for (int r = 0; r < 8; ++r) qx = fmaf(rp[r], rx[r], qx);
                if constexpr (SB < 0) {
                    const float sum = rows_sum<8>(rows, lane);
                    if ((lane & 3) == 0) rowp[32 * B0 + 64 * g + warp + 8 * (lane >> 2)] = sum;
                }
            });
            if constexpr (SB >= 0) {
                // all rows in one butterfly (its five exchanges are waited for once)
                float* const dst = rowp + 32 * B0 + 64 * (SB / 2) + warp;
                if constexpr (NR >= 32) {
                    dst[8 * lane] = rows_sum<32>(rows, lane);
                } else if constexpr (NR >= 16) {
                    const float sum = rows_sum<16>(rows, lane);
                    if ((lane & 1) == 0) dst[8 * (lane >> 1)] = sum;
                }
                if constexpr (NR == 8 || NR == 24) {
                    const float sum = rows_sum<8>(rows + NR - 8, lane);
                    if ((lane & 3) == 0) dst[8 * (NR - 8) + 8 * (lane >> 2)] = sum;
                }
            }
            static_for<(SB > 0 ? SB : 0), kRegBlk>([&](auto bc) {
                constexpr int b = decltype(bc)::value;
                colp[warp * N + 32 * (B0 + b) + lane] = cpr[b];
                qx = fmaf(cpr[b], xc[b], qx);
            });
            xq[tid] = qx;
            __syncthreads();

            // ---- C
            // x^T A x: every warp sums the threads' parts (beside the loads below)
            const float4 xa = *reinterpret_cast<const float4*>(xq + 4 * lane);
            const float4 xb4 = *reinterpret_cast<const float4*>(xq + 128 + 4 * lane);
            const float xax = warp_sum(((xa.x + xa.y) + (xa.z + xa.w)) + ((xb4.x + xb4.y) + (xb4.z + xb4.w)));
            const int c1 = c + 1;
            // column c1 at row i: lane c1 % 32 of warp i % 8
            const float* const col = S - tid + (c1 & 31);
            auto column = [&](int i) { return col[slot(i >> 3, bs) + (i & 7) * 32]; };
            auto product = [&](int i) {
                float q[kRegNW];
#pragma unroll
                for (int k = 0; k < kRegNW; ++k) q[k] = colp[k * N + i];
                return ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7])) + rowp[i];
            };
            // this thread's elements (the second: rows of the shared part only)
            constexpr int NU = SB >= 0 ? 1 : 2;
            float q[NU], rw[NU], t[NU][6];
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                const int i = max(N - 1 - tid - u * kRegNT, c1);    // (dead rows: any value)
                q[u] = product(i);
                rw[u] = column(i);
                const float4 f = *reinterpret_cast<const float4*>(VW + 4 * i);
                const float2 h = *reinterpret_cast<const float2*>(VW + 4 * (N + i));
                t[u][0] = f.x; t[u][1] = f.y; t[u][2] = f.z; t[u][3] = f.w; t[u][4] = h.x; t[u][5] = h.y;
            }
            // row c1 (every thread, the same bits): v^T y, K, w_{c1}
            const float tau = pub[1], scal = pub[2];
            const float q1 = product(c1), a1 = column(c1);
            const float4 f1 = *reinterpret_cast<const float4*>(VW + 4 * c1);
            const float2 h1 = *reinterpret_cast<const float2*>(VW + 4 * (N + c1));
            float p1[6] = {f1.x, f1.y, f1.z, f1.w, h1.x, h1.y};     // (v_l, w_l) of row c1
            float y1 = fmaf(scal, q1, a1);
            float s = a1 + scal * (2.0f * q1 + scal * xax);
            float DV[3], DW[3];                                     // V^T v, W^T v
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const float2 d2 = *reinterpret_cast<const float2*>(dots + 2 * l);
                DV[l] = l < jj ? fmaf(scal, d2.x, p1[2 * l]) : 0.0f;
                DW[l] = l < jj ? fmaf(scal, d2.y, p1[2 * l + 1]) : 0.0f;
                if (l >= jj) p1[2 * l] = p1[2 * l + 1] = 0.0f;
                y1 -= p1[2 * l] * DW[l] + p1[2 * l + 1] * DV[l];
                s -= 2.0f * DV[l] * DW[l];
            }
            const float K = 0.5f * tau * (tau * s);
            const float w1 = tau * y1 - K;                          // w_{c1} (v_{c1} = 1)
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                const int i = N - 1 - tid - u * kRegNT;
                if (i < 0) continue;
                float y = fmaf(scal, q[u], rw[u]);
                float pend = 0.0f;                                  // the pending pairs at column c1
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    if (l >= jj) continue;
                    y -= t[u][2 * l] * DW[l] + t[u][2 * l + 1] * DV[l];
                    pend += t[u][2 * l] * p1[2 * l + 1] + t[u][2 * l + 1] * p1[2 * l];
                }
                const bool live = i >= c1;
                const float vi = i == c1 ? 1.0f : live ? x[u] * scal : 0.0f;
                const float wi = live ? tau * y - K * vi : 0.0f;
                x[u] = live ? rw[u] - (pend + (vi * w1 + wi)) : 0.0f;
                *reinterpret_cast<float2*>(VW + 4 * ((jj >> 1) * N + i) + 2 * (jj & 1)) = make_float2(vi, wi);
                publish(i, c1, x[u]);
                if (i > c1) Aw[(goff + i) + (long long)(goff + c) * ld] = vi;   // kept for Y = F^ Q
            }
            __syncthreads();
        };
        for (int c = pad; c < 32 * B0 - 1; ++c) column_step(std::integral_constant<int, -1>{}, c);
        static_for<0, kRegBlk>([&](auto sbc) {
            constexpr int b = decltype(sbc)::value;
            const int lo = max(pad, 32 * (B0 + b) - 1), hi = min(N - 1, 32 * (B0 + b) + 31);
            if (lo >= hi) return;
            // (the slots that receive the block are read no more: the blocks before it are done)
            static_for<4 * b, 4 * kRegBlk>([&](auto ac) {
                constexpr int a = decltype(ac)::value;
                S[(a - 4 * b) * kRegNT] = A[reg_slot(a, b)];
            });
            for (int c = lo; c < hi; ++c) column_step(sbc, c);
        });
        if (tid == 0) {
            ew[n - 1] = 0.0f;
            tw[n - 1] = 0.0f;
        }
        __syncthreads();
    }
}

}  // namespace

int tri_reduce_reg(int nwin, const int* order, int* counter, const int* n_w, const long long* offC,
                   const long long* offA, const long long* offN, const float* H, float* A, float* d, float* e,
                   float* tau, int* status, int nb, int nmax, size_t smem_budget, cudaStream_t s) {
    const int NB = std::max(kRegBlk, (std::min(nmax, kTriRegMax) + 31) / 32);
    const size_t smem = reg_smem_floats(NB) * sizeof(float);
    if (smem > smem_budget) {
        lres_set_error("resident tridiagonal reduction needs %zu B of shared memory", smem);
        return LRES_EINVAL;
    }
    LRES_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(int), s));
    int per_sm = 0;
    if (int rc = prepare_kernel<tri_reduce_reg_kernel>(kRegNT, smem, &per_sm)) return rc;
    const int grid = std::min(nwin, std::max(1, per_sm) * device_sms());
    TriRegParams p{nwin, order, counter, n_w, offC, offA, offN, H, A, d, e, tau, status, nb, NB};
    tri_reduce_reg_kernel<<<grid, kRegNT, smem, s>>>(p);
    LRES_CUDA_TRY(cudaGetLastError());
    return LRES_OK;
}

}  // namespace lres
