// Device-resident BiCGSTAB scalars and launcher declarations.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.hpp"

namespace cfdg {

enum : int { KS_RUNNING = 0, KS_CONVERGED = 1, KS_DIVERGED = 2, KS_MAXIT = 3 };

// Scalars of BiCGSTAB::solve (src/linalg/bicgstab.cpp:42-201) kept on the
// device so that an iteration needs no host round trip.  `state` is the
// first member: kernels early-exit when it is not KS_RUNNING.
struct KrylovScalars {
    int state;
    int it;
    int max_it;
    int guess;  // in: 1 when x holds an initial guess that may be rejected; out: 2 when rejected
    int body_runs;  // device loop: iterations the graph body has run (bounds the loop by max_it)
    double rel_tol, abs_tol;
    double bnorm, scale, tol, initial, rnorm;
    double rho, rho_old, rho_new, alpha, omega, omega_new, beta;
    // Solves reduced to the rows outside the first colour
    // (kernels_reduced.cu): the caller's vectors, the arrival counter of the
    // grid sums, the updates x has had, |rho_0|^2 and the colour-0
    // multiples of rho_0 in r, p and s (cp_new: p after the update).
    double* x;
    const double* b;
    unsigned arrived;
    int updates;
    double q0, cr, cp, cp_new, cs;
};

// A multicolour system for the reduced BiCGSTAB: colour 0 at positions
// [0, n0), colour 1 at [n0, n1).  Position = row (rows null) when the rows are
// in colour order, else rows[position] with two colours.  mid[row]: first
// block outside the colour-0 columns (rows in colour order only).
struct RedView {
    int32_t n, n0, n1, bs;
    const int32_t *row_ptr, *cols, *diag, *mid, *rows;
};
enum : int { RED_BACK0, RED_BACK, RED_FWD, RED_ETA, RED_WSUM, RED_XRED };
int red_partials();  // doubles of the reduction buffer
// *flag = 1 when a diagonal block would cost the reduced product accuracy
void launch_red_check(const RedView& A, const double* vals, const double* dinv, int* flag, cudaStream_t st);
// r0 = b - A x (v = A x; null: x = 0), r and p on the rest rows, the scalars
void launch_red_init(const RedView& A, KrylovScalars* ks, const double* v, double* r, double* r0, double* p,
                     double* partials, bool guess, cudaStream_t st);
// One sweep pass over the positions [pos0, pos1); second: the s vector's
// sweep (cs), else the p vector's (cp)
void launch_red_sweep(const RedView& A, const double* vals, const double* dinv, int kind, int32_t pos0, int32_t pos1,
                      const double* src, const double* w, double* z, double* e, const KrylovScalars* ks, bool second,
                      cudaStream_t st);
void launch_red_product(const RedView& A, const double* vals, const double* src, const double* e, double* out,
                        const double* r0, KrylovScalars* ks, double* partials, bool first, cudaStream_t st);
void launch_red_s(const RedView& A, const double* dinv, const double* r, const double* v, const double* w, double* s,
                  double* z, const KrylovScalars* ks, cudaStream_t st);
void launch_red_update(const RedView& A, const double* dinv, const double* zs, const double* s, const double* t,
                       const double* v, const double* w, double* r, double* p, double* zp, KrylovScalars* ks,
                       double* partials, cudaGraphConditionalHandle cond, bool use_cond, cudaStream_t st);
void launch_red_enter(const KrylovScalars* ks, cudaGraphConditionalHandle cond, cudaStream_t st);

// Up to five (a, b) vector pairs; a null pointer stands for the SpMV output.
struct DotSpec {
    const double* a[5];
    const double* b[5];
    int n;
};

// Jacobian-free product y = (alpha - V diag) x + (R(U + eps x) + b) / eps
// from the perturbed residual `resp` (SoA, cell order), with the dots `ds`;
// returns the partial count.
int launch_jf_combine(const DevMesh& m, int nv, const double* alpha, double diag, const double* x, const double* b,
                      const double* resp, const double* scal, double* y, const DotSpec& ds, double* partials,
                      const int* active, cudaStream_t s);

// y = alpha A x + beta y on rows [row_begin, n), optional fused dots
template <typename MT>
void launch_spmv_ex(const BsrView& A, const MT* vals, const double* x, double* y, double alpha, double beta,
                    const DotSpec& ds, double* partials, const int* active, cudaStream_t s, int32_t row_begin = 0);
// Last backward pass of the split multicolour sweep (colour 0 = rows
// [0, n_rows), `dinv` the inverse diagonal blocks) fused with y = A z and the
// dots on those rows; partials: sgs_last_spmv_blocks(n_rows, bs) * ds.n.
template <typename MT>
void launch_sgs_last_spmv(const BsrView& A, const MT* vals, const MT* dinv, int32_t n_rows, double* z, double* y,
                          const DotSpec& ds, double* partials, const int* active, cudaStream_t s);
int sgs_last_spmv_blocks(int32_t n_rows, int32_t bs);
// rows: the pass's row list, or null for the contiguous rows row0 ..
// inverse: `lu` holds D^-1 (launch_lu_setup with inverse)
template <typename MT>
void launch_sgs_rows_ex(const BsrView& A, const MT* vals, const MT* lu, const int8_t* piv, const int32_t* rows,
                        int32_t row0, int32_t n_rows, const double* r, double* z, int mode, bool inverse,
                        const int* active, cudaStream_t s);
// The whole level-scheduled symmetric sweep (forward levels, then backward
// levels; z zeroed by the caller) as one cooperative launch with a grid
// barrier per level; rows as (row, row_ptr[row], row_ptr[row+1], diag[row])
// records in level order.  False when the device or block size has no
// cooperative launch (the caller then launches level by level).
template <typename MT>
bool launch_sgs_level_coop(const BsrView& A, const MT* vals, const MT* lu, const int8_t* piv, const int4* fwd_rows,
                           const int32_t* fwd_off, int n_fwd, const int4* bwd_rows, const int32_t* bwd_off,
                           int n_bwd, const double* r, double* z, const int* active, cudaStream_t s);
// The same sweep for a system whose z fits in the shared memory of one
// cluster: sgs_level_cluster gives the cluster's CTAs and their shared-memory
// bytes (0: it does not fit, its levels are too wide for one cluster, or block
// sizes other than 5 and 6; offsets on the host).  from_zero: z starts from zero
// (else from the array); z is written once at the end.  False: not launched.
int sgs_level_cluster(int32_t n, int bs, bool mixed, const int32_t* fwd_off, int n_fwd, const int32_t* bwd_off,
                      int n_bwd, int* smem);
template <typename MT>
bool launch_sgs_level_cluster(const BsrView& A, const MT* vals, const MT* lu, const int8_t* piv, const int4* fwd_rows,
                              const int32_t* fwd_off, int n_fwd, const int4* bwd_rows, const int32_t* bwd_off,
                              int n_bwd, const double* r, double* z, bool from_zero, int C, int smem,
                              const int* active, cudaStream_t s);
// A colour-ordered system in slices of 32 rows (kernels_sell.cu).  Slot
// (slice, lane) holds row[slot] (-1: none) with len[slot] blocks below and above
// the diagonal; column c of the values is 32 blocks, entry e of lane l at
// (c * bs^2 + e) * 32 + l, cols[c * 32 + l] the block's column.  desc[slice]:
// first lower column, their count, first upper column, their count; its diagonal
// blocks are column diag0 + slice, its D^-1 column `slice` of their array.
struct SellView {
    int32_t bs, diag0;
    const int32_t *row, *cols;
    const int2* len;
    const int4* desc;
};
// Passes (z the vector the neighbour blocks multiply):
//   DIAG  z = D^-1 r            LOW  z = D^-1 (r - L z)   FULL  z = D^-1 (r - L z - U z)
//   UP    z += D^-1 (-U z)      UPY  as UP, and y = U z + D z (the row's product when L is empty)
//   MUL   y = A z
enum : int { SELL_DIAG, SELL_LOW, SELL_UP, SELL_UPY, SELL_FULL, SELL_MUL };
// Whether the device can run the passes (asked once, outside a capture).
bool sell_ready(int bs, bool mixed);
template <typename MT>
void launch_sell_copy(int bs, int64_t columns, const int32_t* src, const MT* from, MT* to, cudaStream_t s);
template <typename MT>
void launch_sell_rows(const SellView& A, const MT* vals, const MT* dinv, int kind, int32_t s0, int32_t s1,
                      const double* r, double* z, double* y, const int* active, cudaStream_t s);
// Inner products of y = A z as k_sgs_last_spmv (rows [0, n0), n0 = 0: none) and
// k_spmv (the rest) sum them; returns the partial rows.
int launch_dots(int32_t n0, int32_t n, int bs, const double* y, const DotSpec& ds, double* partials, const int* active,
                cudaStream_t s);
void launch_krylov_init(int64_t len, const double* b, const double* v, double* r, double* r0, double* p,
                        double* partials, KrylovScalars* ks, cudaStream_t s);
// After launch_krylov_init: a rejected initial guess (||b - A x0|| >=
// ||b||) restarts from x = 0 (r = r0 = p = b).
void launch_krylov_guess_reset(int64_t len, const KrylovScalars* ks, const double* b, double* x, double* r, double* r0,
                               double* p, cudaStream_t s);
void launch_krylov_begin(KrylovScalars* ks, cudaStream_t s);
void launch_krylov_gamma(KrylovScalars* ks, const double* partials, int nblocks, cudaStream_t s);
void launch_krylov_s(int64_t len, const KrylovScalars* ks, const double* r, const double* v, double* sv,
                     cudaStream_t s);
void launch_krylov_omega(KrylovScalars* ks, const double* partials, int nblocks, cudaStream_t s);
void launch_krylov_update(int64_t len, const KrylovScalars* ks, double* x, const double* phat, const double* shat,
                          const double* sv, const double* tv, double* r, double* p, const double* v,
                          double* partials, cudaStream_t s);
void launch_krylov_post(KrylovScalars* ks, const double* partials, int nblocks, cudaStream_t s);
// Last node of the device loop's body: counts the body run and sets the
// while-condition to (state == running and runs < max_it).
void launch_krylov_cond(KrylovScalars* ks, cudaGraphConditionalHandle h, cudaStream_t s);

}  // namespace cfdg
