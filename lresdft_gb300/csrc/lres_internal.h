// Internal declarations shared by the translation units of liblres_gb300.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>
#include "../../include/lres_gb300.h"

namespace lres {

// One launch of the fused window LDL^T kernel (window_ldl.cu).
struct LdlJob {
    enum Kind { C128, C64, R64 } kind;
    int nitems = 0;
    const int2* items = nullptr;
    int* counter = nullptr;
    const int* n_w = nullptr;
    const int* m_w = nullptr;
    const long long* offC = nullptr;
    const long long* offF = nullptr;
    const long long* offQ = nullptr;
    const void* C = nullptr;
    const void* B = nullptr;
    const void* F = nullptr;
    const void* shifts = nullptr;
    void* q = nullptr;
    long long qstride = 0;
    double* mult = nullptr;
    int* npos = nullptr;
    int* status = nullptr;
    void* ws = nullptr;
    long long ws_stride = 0;
    int ldp = 0, nmax = 0, mmax = 0;
    int grid = 0;
    size_t smem_budget = 0;
    int config = 0;                 // complex kernels: tile configuration (see lres_tune)
    int keep = 0;                   // complex kernels: keep every item's factor (slot = item index)
    const int* c0 = nullptr;        // per window: the F rows are zero in the columns before c0[w]
};

// Panel width of the factor kept for the adjoint (the window is padded to a multiple).
constexpr int kKeepNB64 = 32, kKeepNB128 = 16;

// Tile configurations of the complex pole kernel, index = LdlJob::config:
//   0: NB 32 (c64) / 16 (c128), 256 threads, k-chunk 32     1: 128 threads
//   2: k-chunk 16                                           3: NB 16 (c64) / 8 (c128)
//   4: c64: chunk products on the tensor cores (tcgen05, 3xTF32); c128: NB 8, 128 threads
//   5: operands of every chunk brought in by bulk asynchronous copies, 128 threads
constexpr int kLeftConfigs = 6;

int run_ldl(const LdlJob& j, cudaStream_t s);
size_t ldl_smem_bytes(int elem_bytes, int nb, int ldp, int mmax);

// Block-sparse (atom-pair) storage of the nb x nb matrices S, T, H.
struct BlockPattern {
    int ngroups = 0;
    int nblk = 0;                     // stored blocks (both triangles)
    int npair = 0;                    // blocks with g <= h (assembled by the H(v) kernel)
    int nfmax = 0;                    // largest group (functions per atom)
    // device arrays
    int* gptr = nullptr;              // [ngroups+1] first function of each group
    int* bptr = nullptr;              // [ngroups+1] blocks of block-row g: [bptr[g], bptr[g+1])
    int* bcol = nullptr;              // [nblk] column group
    int* brow = nullptr;              // [nblk] row group
    long long* boff = nullptr;        // [nblk] value offset (nf_g * nf_h values, row-major)
    int* btrans = nullptr;            // [nblk] index of the transposed block
    int* pair_blk = nullptr;          // [npair] block index of pair p (g <= h)
    long long nval = 0;
};

// Group supports on the grid and common-point lists of overlapping pairs.
struct Supports {
    long long nslot = 0;
    long long* soff = nullptr;        // [ngroups+1] slot range of each group
    int* sgrid = nullptr;             // [nslot] grid index of each slot
    double* sval = nullptr;           // [nslot * 8] basis values, 8 per slot (zero padded)
    float* sval32 = nullptr;          // the same in FP32 (mixed precision only)
    float* vslot = nullptr;           // [nslot] FP32 potential at each slot (mixed H(v) scratch)
    long long ncommon = 0;
    long long* coff = nullptr;        // [npair+1] common-point range of each pair
    int2* cslot = nullptr;            // [ncommon] (slot in g, slot in h)
};

// Kernel launchers implemented in hamiltonian.cu / grid.cu / dense.cu
int pair_common_points(const BlockPattern& bp, Supports& sp, int ngroups, const std::vector<int>& pair_g,
                       const std::vector<int>& pair_h, cudaStream_t s);
int assemble_h(const BlockPattern& bp, const Supports& sp, const double* Tblk, const double* v, double dV,
               double* Hblk, cudaStream_t s);
bool assemble_h32_supported(const BlockPattern& bp);
int assemble_h32(const BlockPattern& bp, const Supports& sp, const double* Tblk, const double* v, double dV,
                 double* Hblk, long long ng, double* vcopy, cudaStream_t s);   // vcopy (nullable): ng values of v
// Dense window blocks (column-major, every element written) from the atom-pair blocks; with
// blk32 and dense32, also the FP32 windows from the FP32 copy of the blocks.
int gather_windows(int nwin, int nmax, const int* fn, const long long* fnoff, const int* btab, const long long* btoff,
                   const int* nlg, const long long* offC, const int* n_w, const double* blk, double* dense,
                   const float* blk32, float* dense32, cudaStream_t s);
// B_w = (A_w + A_w^T) / 2 (n_w x n_w)
int symmetrise_windows(int nwin, int nmax, const int* n_w, const long long* offC, const double* A, double* B, cudaStream_t s);
int build_F(int nwin, const long long* Xp, const int* Xi, const double* Xv, const int* group_of_fn,
            const int* gptr, const int* gloc, int ngroups, const long long* Ooff, const long long* Oflat,
            const long long* offF, const int* m_w, int mmax, double* F, cudaStream_t s);
// FP64 products on the tensor cores (oz_gemm.cu): C_w = op(A_w) op(B_w) (or C_w -= it), C_w m_w x n_w
// column-major at offC, K = k_w terms.  klim 1: op(B) upper triangular, 2: op(A) lower triangular and
// the lower triangle of C only.  balance: the terms' factors are brought to one size first (operands whose
// elements vary along k; plain storage).  The workspace grows on demand.
struct OzForm {                       // how an operand is stored
    bool k_contig;                    // op(A)(i, k) at A[k + i ld] (op(B)(k, j) at B[k + j ld]), else at A[i + k ld] (B[j + k ld])
    const int* ld = nullptr;          // leading dimension ld[w] rounded up to 4; none: that of a dense block
    bool refl = false;                // Householder vectors (row i, reflector l): 1 on the diagonal, 0 above
    OzForm(bool kc, const int* l = nullptr, bool r = false) : k_contig(kc), ld(l), refl(r) {}
};
struct OzWork {
    void* buf = nullptr;
    size_t bytes = 0;
    void release();
};
// Workspace for products of up to mmax (>= nmax) rows, nmax columns and nmax terms, or nmax rows and columns
// and mmax terms: for all windows (up to 1 GB), or for as many at a time as the device has room for.  A
// product whose windows fit one by one allocates nothing.
int oz_reserve(OzWork& wk, int nwin, int mmax, int nmax);
int oz_gemm(OzWork& wk, int nwin, int mmax, int nmax, int kmax, const int* m_w, const int* n_w, const int* k_w,
            const double* A, const long long* offA, OzForm fa, const double* B, const long long* offB, OzForm fb,
            double* C, const long long* offC, int klim, bool subtract, bool balance, size_t smem_budget,
            cudaStream_t s);
int batched_gram(int nwin, const int* n_w, const int* m_w, const long long* offF, const long long* offK, int nmax,
                 const double* F, double* K, cudaStream_t s);
int batched_gemm_rect_upper(int nwin, const int* n_w, const int* m_w, const long long* offA, const long long* offU,
                            int nmax, int mmax, const double* A, const double* U, double* C, cudaStream_t s);
int convert_f64_f32(const double* a, float* b, long long n, cudaStream_t s);
int split_f64(const double* a, float2* b, long long n, cudaStream_t s);
int batched_gemm_df64(int nwin, const int* n_w, const long long* off, int nmax, bool transA, int klim,
                      const float2* A, const float2* B, float2* C, float* C32, cudaStream_t s);
// C = A B for every window block: A column-major (FP64 or FP32), B k-major (Bt[j + k n] =
// B[k][j]), C column-major or row-major (c_rowmajor); klim as oz_gemm.
int batched_gemm_f32(int nwin, const int* n_w, const long long* off, int nmax, int klim, const void* A, bool a_f64,
                     const float* Bt, float* C, bool c_rowmajor, cudaStream_t s);
// batched_gemm_f32's products on the tensor cores (tcgen05, 3xTF32, 32-term chunks); a timed-out
// completion wait sets ST_TIMEOUT in *status (device)
int batched_gemm_tc(int nwin, const int* n_w, const long long* off, int nmax, int klim, const void* A, bool a_f64,
                    const float* Bt, float* C, bool c_rowmajor, int* status, cudaStream_t s);
int batched_transpose_f32(int nwin, const int* n_w, const long long* off, int nmax, const float* A, float* B,
                          cudaStream_t s);
int pole_sums(int nwin, const long long* offQ, const int* m_w, const long long* Oflat, bool fp32,
              const void* q, long long qstride, int npoles, const double2* wq, const double2* wzq, double dV,
              double* dens, double* n_w, double* e_w, cudaStream_t s);

// Multi-shift tridiagonal route (tridiag.cu): R = float (fp32) or double.
// Tile configuration of the tridiagonal route for windows of at most nmax functions and P poles; LRES_EINVAL
// where they are too large or too many for its kernels.
struct TriPick {
    int nb = 0;                // reduction panel width
    bool pairs = false;        // FP64: reductions two to an SM, beyond an SM for each
    int reg = 0;               // 1: the reduction holds each window on its SM (FP32, tridiag_reg.cu)
    int nb_apply = 0;          // row application panel width
    int rpt = 1;               // rows per thread of the row-per-thread application; 0: resident rows
    int arows = 0;             // rows per application item
    int ldv = 0;               // shared vector length (multiple of 32, >= nmax)
    long long tstride = 0;     // T-factor elements per window (resident application)
};
int tri_pick(bool fp32, int nmax, int P, size_t smem_budget, int cfg, TriPick* out);
int tri_reduce(bool fp32, int nwin, const int* order, int* counter, const int* n_w, const long long* offC,
               const long long* offA, const long long* offN, const void* H, void* A, void* d, void* e, void* tau,
               int* status, const TriPick& pk, int nmax, size_t smem_budget, cudaStream_t s);
// The reduction with the window on the SM, for the last kTriRegMax columns of each window; larger
// windows come with the columns before those reduced in panels of nb.
constexpr int kTriRegMax = 384;
int tri_reduce_reg(int nwin, const int* order, int* counter, const int* n_w, const long long* offC,
                   const long long* offA, const long long* offN, const float* H, float* A, float* d, float* e,
                   float* tau, int* status, int nb, int nmax, size_t smem_budget, cudaStream_t s);
// tfactors: form the T factors of every (window, panel) first (once per Hamiltonian)
int tri_apply(int nitems, const int4* items, const int* n_w, const int* m_w, const long long* offA,
              const long long* offN, const long long* offF, const float* A, const float* tau, const float* F, float* Y,
              const TriPick& pk, int nwin, bool tfactors, float* T, size_t smem_budget, cudaStream_t s);
// Rows of a set through the reflectors on the tensor cores (FP64): panels of kOzPanel reflectors.
constexpr int kOzPanel = 128;
struct OzRows {                       // per panel and window, panel-major: reflectors, rows below, offsets of
    int panels = 0;                   // the panel's reflectors, its T (kOzPanel^2 apart)
    int *q = nullptr, *r = nullptr;
    long long *offV = nullptr, *offT = nullptr;
    double* T = nullptr;
    void release();
};
struct OzRowSet {                     // one row set: S scratch and, per panel and window, offsets of Y's block
    long long *offS = nullptr, *offY = nullptr;
    double *S = nullptr, *S2 = nullptr;
    int mmax = 0;
    void release();
};
int oz_tfactors(OzWork& wk, const OzRows& o, int nwin, int nmax, const int* n_w, const double* A, const double* tau,
                const long long* offN, size_t smem_budget, cudaStream_t s);
int oz_rows(OzWork& wk, const OzRows& o, const OzRowSet& rs, int nwin, int nmax, const int* n_w, const int* m_w,
            const double* A, double* Y, size_t smem_budget, cudaStream_t s);
int tri_rows_per_item(bool fp32, int P);
int tri_pass(bool fp32, int nitems, const int4* items, int* counter, const int* n_w, const int* m_w,
             const long long* offN, const long long* offF, const long long* offQ, const long long* Oflat,
             const void* Y, const void* d, const void* e, int P, const void* shifts, const double2* wq,
             const double2* wzq, double* dens, double* part, int* status, int ldv, size_t smem_budget,
             cudaStream_t s);
// Elements of the coefficients of G_k: (t_i, G_ii) of nwin * P * nmax, then the products of t within blocks.
inline size_t tri_coef_elems(int nwin, int P, int nmax) { return ((size_t)nwin * P * nmax * 3 + 1) / 2; }
// N and E_band of every window from K = Y^T Y (FP64): coef tri_coef_elems, trace nwin * P elements
int tri_count(int nwin, int P, int nmax, const int* n_w, const long long* offN, const long long* offC, const double* d,
              const double* e, const double* K, const double2* shifts, const double2* wq, const double2* wzq,
              double dV, double4* coef, double2* trace, double* nw, double* ew, int* status, size_t smem_budget,
              cudaStream_t s);
// u[c * nwin + w] = Re sum_k cw[c P + k] tr(G_k K G_k), c = 0, 1, 2, after tri_count: its coef, dcoef as coef,
// slope nwin * P elements.
int tri_slopes(int nwin, int P, int nmax, const int* n_w, const long long* offN, const long long* offC, const double* d,
               const double* e, const double* K, const double2* shifts, const double2* cw, const double4* coef,
               double4* dcoef, double2* slope, double* u, cudaStream_t s);
// P = Re sum_k w_k (z_k - T)^-1 of every window (FP64); the rows' n, e from V = Y P for windows w0 ..
// w0 + nwin - 1 (V of window w at offV[w], maxitems pass items of a window at most).
int tri_pmat(int nwin, int P, int nmax, const int* n_w, const long long* offN, const long long* offC, const double* d,
             const double* e, const double2* shifts, const double2* wq, double4* coef, double* Pm, cudaStream_t s);
int tri_rowdot(int w0, int nwin, int maxitems, const int4* items, const int* first, const int* count, const int* n_w,
               const int* m_w, const long long* offN, const long long* offF, const long long* offV,
               const long long* offQ, const long long* Oflat, const double* Y, const double* V, const double* d,
               const double* e, double* dens, double* part, int* status, cudaStream_t s);
int tri_window_sums(int nwin, const int* first, const int* count, const double* part, double dV, double* nw,
                    double* ew, cudaStream_t s);
int tri_sturm(bool fp32, int nwin, const int* n_w, const long long* offN, const void* d, const void* e,
              double sigma, int* below, cudaStream_t s);
int tri_min_eig(bool fp32, int nwin, const int* n_w, const long long* offN, const void* d, const void* e,
                double tol, double* lam, cudaStream_t s);

// Adjoint of the window solve (adjoint.cu)
int adj_backsolve(bool fp32, const int2* items, int nitems, const int* n_w, const int* m_w, void* ws,
                  long long ws_stride, int* status, cudaStream_t s);
int adj_accumulate(bool fp32, const int* wins, int nwin_batch, int P, int nmax, const int* n_w, const int* m_w,
                   const long long* offC, const void* ws, long long ws_stride, const double2* cw, double* A0,
                   double* A1, double* A2, cudaStream_t s);
// A_c in the tridiagonal basis, X_c = Re sum_k c_k G_k K G_k, in batches of windows: coef nwin * P * nmax,
// ws batch * groups * 2 nmax^2 complex values, X 3 * groups * sizeC elements (unused with one group); with
// K32 the sweeps run in FP32
int adj_sweep_groups(int nwin, int P);
int adj_tri(int nwin, int P, int groups, int batch, int nmax, const int* wins, const int* n_w, const long long* offN,
            const long long* offC, long long sizeC, const double* d, const double* e, const double2* shifts,
            const double2* cw, const double* K, const float* K32, double4* coef, void* ws, double* X, double* A0,
            double* A1, double* A2, size_t smem_budget, cudaStream_t s);
int adj_weights(int P, int M, double mu, double e_lo, double2* cw, cudaStream_t s);
int adj_inner(int nwin, const int* n_w, const long long* offC, const double* S, const double* A0, const double* A1,
              const double* A2, double* u, cudaStream_t s);
int adj_combine(long long nval, const double* A0, const double* A1, const double* A2, double kappa, double a,
                double b, double* X, double* Y, cudaStream_t s);
int adj_block_gather(const BlockPattern& bp, const long long* eoff, const int4* ent, const int* n_w,
                     const long long* offC, const double* dHW, double* gH, cudaStream_t s);
int adj_point(long long ng, const long long* poff, const int2* pent, const Supports& sp, const BlockPattern& bp,
              const double* gH, double dV, double* dv, cudaStream_t s);

struct FFT3;
int fft3_create(FFT3** out, const int64_t shape[3], const double cell[3]);
void fft3_destroy(FFT3* f);
// work: n1 n2 (n3 / 2 + 1) complex values
int hartree_apply(FFT3* f, const double* dens, double* vh, double2* work, cudaStream_t s);
int lda_apply(long long n, const double* dens, double* exc, double* vxc, cudaStream_t s);
int ion_apply(FFT3* f, const double cell[3], int natoms, const double* pos, const double* Z, const double* rc,
              double* vion, double2* work, cudaStream_t s);
int voronoi_apply(const int64_t shape[3], const double cell[3], int ncent, const double* centres, int* owner,
                  cudaStream_t s);

}  // namespace lres
