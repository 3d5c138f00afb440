// BiCGSTAB with the multicolour SGS preconditioner, reduced to the rows
// outside the first colour.
//
// With the rows in colour order, A = L + D + U and M = (D+L) D^-1 (D+U), the
// sweep z = M^-1 p leaves y = (D+L)^-1 p (forward) and e = y - z = D^-1 U z
// (backward), and the product needs no second pass over the matrix:
//     A z = (D+U) z + L z = D y + L z = p - L e.
// Rows of the first colour have no L, so there (A z)_0 = p_0: v_0 = p_0 and
// t_0 = s_0, and the colour-0 parts of r, p, s, v, t stay multiples
// (cr, cp, cs, ...) of the initial residual's, rho_0, which the device
// scalars carry.  The forward sweep's colour-0 contribution is linear in p_0
// too: w = A_{R0} D_0^-1 rho_0 is formed once per solve.  An application then
// reads every off-diagonal block outside the colour-0 columns of the forward
// sweep, the upper blocks and the lower blocks once (two colours: each
// off-diagonal block once, against one and a half times for the sweep plus
// product, and no diagonal block), the vectors are touched on the rest rows
// only, and x_0 follows at the end from its own rows,
//     x_0 = D_0^-1 (b_0 - cr rho_0 - U x_R).
// The iterates are those of BiCGSTAB::solve (src/linalg/bicgstab.cpp:42-201)
// on the full system up to rounding, as far as D D^-1 = I holds: the product
// does not multiply by D, so its error is that of D (D^-1 p) where the full
// product's is that of A z.  k_red_check measures the difference for each
// diagonal block, and the solve runs in the full form when one exceeds
// kGrowthLimit.  FP64 matrices only: the FP32 inverse of a mixed-precision system
// holds D D^-1 = I to 1e-7.
//
// All passes are bound by the matrix and vector traffic; the reductions end in
// the last block of the kernel that forms them (one counter, fixed order),
// so an iteration of two colours is six launches and no single-block kernel.
#include "krylov.hpp"

namespace cfdg {
namespace {

constexpr int kThreads = 256;
constexpr int64_t kGridCap = 148 * 8;  // resident 256-thread blocks; bounds the partials a last block reads

// BS consecutive entries at p (matrix block row or vector block); 6 and 4
// entries start on pair boundaries and load as pairs.
template <int BS>
__device__ __forceinline__ void load_row(const double* p, double (&out)[BS]) {
    if constexpr (BS == 6 || BS == 4) {
        const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
        for (int h = 0; h < BS / 2; ++h) {
            const double2 v = __ldg(q + h);
            out[2 * h] = v.x;
            out[2 * h + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < BS; ++j) out[j] = __ldg(p + j);
    }
}

// sum over blocks [k0, k1) (skipping block `skip`) of A_k[ii][:] . x_col(k);
// PAIRS: x is 16-byte aligned (the system's own vectors; a caller's may not be)
template <int BS, bool PAIRS = true>
__device__ __forceinline__ double row_sum(const RedView& A, const double* __restrict__ vals, const double* x, int ii,
                                          int32_t k0, int32_t k1, int32_t skip) {
    double acc = 0.0;
    for (int32_t k = k0; k < k1; ++k) {
        if (k == skip) continue;
        double a[BS], xb[BS];
        load_row<BS>(vals + int64_t(k) * (BS * BS) + ii * BS, a);
        const double* xk = x + int64_t(__ldg(A.cols + k)) * BS;
        if constexpr (PAIRS) {
            load_row<BS>(xk, xb);
        } else {
#pragma unroll
            for (int j = 0; j < BS; ++j) xb[j] = xk[j];
        }
        double t = 0.0;
#pragma unroll
        for (int jj = 0; jj < BS; ++jj) t += a[jj] * xb[jj];
        acc += t;
    }
    return acc;
}

// Row ii of D^-1 (row i) times the row's vector, whose entry ii this lane
// holds; every lane of the warp takes part in the exchange.
template <int BS>
__device__ __forceinline__ double apply_dinv(const double* __restrict__ dinv, int32_t i, int ii, int base, bool act,
                                             double s) {
    double b[BS];
#pragma unroll
    for (int j = 0; j < BS; ++j) b[j] = __shfl_sync(0xffffffffu, s, base + j);
    double out = 0.0;
    if (act) {
        double d[BS];
        load_row<BS>(dinv + int64_t(i) * (BS * BS) + ii * BS, d);
#pragma unroll
        for (int j = 0; j < BS; ++j) out += d[j] * b[j];
    }
    return out;
}

// Lane layout of every kernel here: a warp takes 32 / BS consecutive
// positions, lane ii of a group holds component ii of its row.
template <int BS>
struct Lanes {
    static constexpr int GPW = 32 / BS;
    int grp, ii, base;
    __device__ Lanes() {
        const int lane = threadIdx.x & 31;
        grp = lane / BS;
        ii = lane - grp * BS;
        base = (grp < GPW ? grp : 0) * BS;
    }
};

__device__ __forceinline__ int64_t warp_id() { return (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; }

// Sums over the grid of ND values per thread; true in the last block to
// arrive, whose threads then all hold the totals.  Blocks add in a fixed
// order, so the totals do not depend on the arrival order.
template <int ND>
__device__ bool grid_sums(double (&pr)[ND], double* partials, unsigned* counter, double (&tot)[ND]) {
    __shared__ bool last;
    __shared__ double sh[ND][kThreads / 32], total[ND];
    block_reduce_store<ND, kThreads>(pr, partials + size_t(blockIdx.x) * ND);
    if (threadIdx.x == 0) {  // the thread that stored the block's partials
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s[ND];
#pragma unroll
    for (int k = 0; k < ND; ++k) s[k] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kThreads)
#pragma unroll
        for (int k = 0; k < ND; ++k) s[k] += __ldcg(partials + size_t(b) * ND + k);
#pragma unroll
    for (int k = 0; k < ND; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_down_sync(0xffffffffu, s[k], o);
        if (lane == 0) sh[k][warp] = s[k];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < ND; ++k) {
            double x = lane < kThreads / 32 ? sh[k][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) total[k] = x;
        }
        if (lane == 0) *counter = 0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ND; ++k) tot[k] = total[k];
    return true;
}

// r = b - A x on every row (v = A x; null: x starts from zero and is cleared
// here); r0 = r everywhere, p = r on the rest rows.  The last block forms
// ||b||, ||r|| and the state.
template <int BS>
__global__ void __launch_bounds__(kThreads) k_red_init(RedView A, KrylovScalars* ks, const double* __restrict__ v,
                                                       double* __restrict__ r, double* __restrict__ r0,
                                                       double* __restrict__ p, double* __restrict__ partials) {
    const Lanes<BS> L;
    const double* b = ks->b;
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    double pr[4] = {0.0, 0.0, 0.0, 0.0};  // rest b.b, r.r; colour 0 b.b, r.r
    for (int64_t w = warp_id(); w * L.GPW < A.n; w += warps) {
        const int64_t pos = w * L.GPW + L.grp;
        if (L.grp >= L.GPW || pos >= A.n) continue;
        const int64_t t = int64_t(A.rows ? A.rows[pos] : static_cast<int32_t>(pos)) * BS + L.ii;
        const double bt = b[t];
        const double rt = v ? bt - v[t] : bt;
        if (!v) ks->x[t] = 0.0;
        r0[t] = rt;
        if (pos < A.n0) {
            pr[2] += bt * bt;
            pr[3] += rt * rt;
        } else {
            r[t] = rt;
            p[t] = rt;
            pr[0] += bt * bt;
            pr[1] += rt * rt;
        }
    }
    double tot[4];
    if (!grid_sums<4>(pr, partials, &ks->arrived, tot) || threadIdx.x != 0) return;
    const double bnorm = sqrt(tot[0] + tot[2]);
    double rnorm = sqrt(tot[1] + tot[3]);
    const double scale = (bnorm > 0.0) ? bnorm : 1.0;
    ks->bnorm = bnorm;
    ks->scale = scale;
    ks->tol = fmax(ks->abs_tol, ks->rel_tol * scale);
    ks->q0 = tot[3];
    if (ks->guess == 1 && !(rnorm < bnorm)) {  // the guess does not beat x = 0
        ks->guess = 2;
        rnorm = bnorm;
        ks->q0 = tot[2];
    }
    ks->initial = rnorm;
    ks->rnorm = rnorm;
    ks->it = 0;
    ks->state = !isfinite(rnorm) ? KS_DIVERGED : (rnorm <= ks->tol ? KS_CONVERGED : KS_RUNNING);
    ks->rho = rnorm * rnorm;
    ks->alpha = 1.0;
    ks->omega = 1.0;
    ks->beta = 0.0;
    ks->cr = ks->cp = ks->cs = 1.0;
}

// A rejected guess restarts from x = 0.
template <int BS>
__global__ void __launch_bounds__(kThreads) k_red_guess_reset(RedView A, const KrylovScalars* __restrict__ ks,
                                                              double* __restrict__ r, double* __restrict__ r0,
                                                              double* __restrict__ p) {
    if (ks->guess != 2) return;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x, len = int64_t(A.n) * BS;
    const double* b = ks->b;
    double* x = ks->x;
    for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < len; t += stride) {
        const double bt = b[t];
        x[t] = 0.0;
        r[t] = bt;
        r0[t] = bt;
        p[t] = bt;
    }
}

// Sweep passes over the positions [pos0, pos1) (one colour).
//   BACK0  colour 0, backward:    e_i = D_i^-1 sum_upper A z
//   BACK   a middle colour:       e_i likewise, z_i -= e_i
//   FWD    forward:               z_i = D_i^-1 (src_i - c w_i - sum_mid A z),
//          mid: the lower blocks outside the colour-0 columns
//   ETA    colour 0, once:        e_i = D_i^-1 r0_i
//   W      rest rows, once:       w_i = sum_{colour-0 columns} A e
//   XRED   colour 0, at the end:  x_i = D_i^-1 (b_i - cr r0_i - sum_upper A x)
// Bound by the blocks read; a lane's block row and the neighbour's vector
// block are independent loads, and a row's blocks follow one another.
enum { BACK0, BACK, FWD, ETA, WSUM, XRED };

template <int BS, bool LIST, int KIND>
__global__ void __launch_bounds__(kThreads, BS <= 5 ? 8 : 6)
    k_red_sweep(RedView A, const double* __restrict__ vals, const double* __restrict__ dinv, int32_t pos0, int32_t pos1,
                const double* src, const double* w, double* z, double* e, const KrylovScalars* __restrict__ ks,
                int second) {
    if (KIND == XRED ? ks->updates == 0 : ks->state != KS_RUNNING) return;
    const Lanes<BS> L;
    const int64_t pos = pos0 + warp_id() * L.GPW + L.grp;
    const bool act = L.grp < L.GPW && pos < pos1;
    int32_t i = 0;
    double s = 0.0;
    if (act) {
        i = LIST ? A.rows[pos] : static_cast<int32_t>(pos);
        const int64_t t = int64_t(i) * BS + L.ii;
        const int32_t d = A.diag[i];
        if (KIND == BACK0 || KIND == BACK) {
            s = row_sum<BS>(A, vals, z, L.ii, LIST ? A.row_ptr[i] : d + 1, A.row_ptr[i + 1], d);
        } else if (KIND == FWD) {
            const double c = second ? ks->cs : ks->cp;
            s = src[t] - c * w[t];
            if (!LIST) s -= row_sum<BS>(A, vals, z, L.ii, A.mid[i], d, d);  // a list has two colours: no mid
        } else if (KIND == ETA) {
            s = src[t];
        } else if (KIND == WSUM) {
            s = LIST ? row_sum<BS>(A, vals, e, L.ii, A.row_ptr[i], A.row_ptr[i + 1], d)
                     : row_sum<BS>(A, vals, e, L.ii, A.row_ptr[i], A.mid[i], d);
        } else {
            const double* x = ks->x;
            s = ks->b[t] - ks->cr * src[t];
            s -= row_sum<BS, false>(A, vals, x, L.ii, LIST ? A.row_ptr[i] : d + 1, A.row_ptr[i + 1], d);
        }
    }
    if constexpr (KIND == WSUM) {
        if (act) z[int64_t(i) * BS + L.ii] = s;
    } else {
        const double o = apply_dinv<BS>(dinv, i, L.ii, L.base, act, s);
        if (act) {
            const int64_t t = int64_t(i) * BS + L.ii;
            if (KIND == BACK0 || KIND == ETA) e[t] = o;
            if (KIND == BACK) {
                e[t] = o;
                z[t] -= o;
            }
            if (KIND == FWD) z[t] = o;
            if (KIND == XRED) ks->x[t] = o;
        }
    }
}

// out = src - L e on the rest rows with the inner products of the iteration:
// FIRST (v = A M^-1 p): gamma = r0.v -> alpha, and s_0 = cs rho_0;
// else (t = A M^-1 s): the five products -> omega, |r|, rho and beta
// (bicgstab.cpp:112-158) with the colour-0 parts from the scalars.
template <int BS, bool LIST, bool FIRST>
__global__ void __launch_bounds__(kThreads, BS <= 5 ? 6 : 5)
    k_red_product(RedView A, const double* __restrict__ vals, const double* __restrict__ src, const double* __restrict__ e,
                  double* __restrict__ out, const double* __restrict__ r0, KrylovScalars* ks,
                  double* __restrict__ partials) {
    if (ks->state != KS_RUNNING) return;
    constexpr int ND = FIRST ? 1 : 5;
    const Lanes<BS> L;
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    double pr[ND];
#pragma unroll
    for (int k = 0; k < ND; ++k) pr[k] = 0.0;
    for (int64_t wq = warp_id(); A.n0 + wq * L.GPW < A.n; wq += warps) {
        const int64_t pos = A.n0 + wq * L.GPW + L.grp;
        if (L.grp >= L.GPW || pos >= A.n) continue;
        const int32_t i = LIST ? A.rows[pos] : static_cast<int32_t>(pos);
        const int64_t t = int64_t(i) * BS + L.ii;
        const int32_t d = A.diag[i];
        const double sv = src[t];
        const double o = sv - row_sum<BS>(A, vals, e, L.ii, A.row_ptr[i], LIST ? A.row_ptr[i + 1] : d, d);
        out[t] = o;
        const double q = r0[t];
        if constexpr (FIRST) {
            pr[0] += q * o;
        } else {
            pr[0] += o * o;
            pr[1] += o * sv;
            pr[2] += q * o;
            pr[3] += q * sv;
            pr[4] += sv * sv;
        }
    }
    double tot[ND];
    if (!grid_sums<ND>(pr, partials, &ks->arrived, tot) || threadIdx.x != 0) return;
    const double q0 = ks->q0;
    if constexpr (FIRST) {
        ks->it += 1;
        if (ks->it > 1 && !isfinite(ks->beta)) {
            ks->state = KS_DIVERGED;
            return;
        }
        const double gamma = tot[0] + ks->cp * q0;
        if (!isfinite(gamma) || gamma == 0.0) {
            ks->state = KS_DIVERGED;
            return;
        }
        ks->alpha = ks->rho / gamma;
        ks->cs = ks->cr - ks->alpha * ks->cp;
    } else {
        const double cs = ks->cs, c2 = cs * cs * q0;
        const double tt = tot[0] + c2, ts = tot[1] + c2, r0t = tot[2] + cs * q0, r0s = tot[3] + cs * q0,
                     ss = tot[4] + c2;
        if (!isfinite(ts) || !isfinite(tt) || tt == 0.0) {
            ks->state = KS_DIVERGED;
            return;
        }
        const double omega_new = ts / tt;
        const double rn2 = ss - 2.0 * omega_new * ts + omega_new * omega_new * tt;
        ks->omega_new = omega_new;
        ks->rnorm = sqrt(fmax(rn2, 0.0));
        ks->rho_new = r0s - omega_new * r0t;
        ks->beta = (ks->rho_new / ks->rho) * (ks->alpha / omega_new);
        // the colour-0 parts after this iteration's update
        const double cr = cs - omega_new * cs;
        ks->cr = cr;
        ks->cp_new = cr + ks->beta * (ks->cp - omega_new * ks->cp);
        ks->updates += 1;
    }
}

// s = r - alpha v on the rest rows and, on colour 1, the first step of its
// sweep z = D^-1 (s - cs w) (later colours follow in k_red_sweep).
template <int BS>
__global__ void __launch_bounds__(kThreads) k_red_s(RedView A, const double* __restrict__ dinv,
                                                    const double* __restrict__ r, const double* __restrict__ v,
                                                    const double* __restrict__ w, double* __restrict__ s,
                                                    double* __restrict__ z, const KrylovScalars* __restrict__ ks) {
    if (ks->state != KS_RUNNING) return;
    const Lanes<BS> L;
    const double alpha = ks->alpha, cs = ks->cs;
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t wq = warp_id(); A.n0 + wq * L.GPW < A.n; wq += warps) {
        const int64_t pos = A.n0 + wq * L.GPW + L.grp;
        const bool act = L.grp < L.GPW && pos < A.n;
        int32_t i = 0;
        double y = 0.0;
        if (act) {
            i = A.rows ? A.rows[pos] : static_cast<int32_t>(pos);
            const int64_t t = int64_t(i) * BS + L.ii;
            const double st = r[t] + (-alpha) * v[t];
            s[t] = st;
            if (pos < A.n1) y = st - cs * w[t];
        }
        if (A.n0 + wq * L.GPW >= A.n1) continue;  // warp-uniform: past colour 1
        const bool c1 = act && pos < A.n1;
        const double o = apply_dinv<BS>(dinv, i, L.ii, L.base, c1, y);
        if (c1) z[int64_t(i) * BS + L.ii] = o;
    }
}

// x += alpha z_p + omega z_s; r = s - omega t; p = r + beta (p - omega v) on
// the rest rows and, on colour 1, the first step of the next sweep into z_p.
// The last block runs the post-update checks (bicgstab.cpp:149-176) and sets
// the loop condition.
template <int BS>
__global__ void __launch_bounds__(kThreads) k_red_update(RedView A, const double* __restrict__ dinv,
                                                         const double* __restrict__ zs, const double* __restrict__ s,
                                                         const double* __restrict__ tv, const double* __restrict__ v,
                                                         const double* __restrict__ w, double* __restrict__ r,
                                                         double* __restrict__ p, double* __restrict__ zp,
                                                         KrylovScalars* ks, double* __restrict__ partials,
                                                         cudaGraphConditionalHandle cond, int use_cond) {
    const bool run = ks->state == KS_RUNNING;  // the same for every block
    double pr[1] = {0.0};
    if (run) {
        const Lanes<BS> L;
        double* x = ks->x;
        const double alpha = ks->alpha, omega = ks->omega_new, beta = ks->beta, cp = ks->cp_new;
        const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
        for (int64_t wq = warp_id(); A.n0 + wq * L.GPW < A.n; wq += warps) {
            const int64_t pos = A.n0 + wq * L.GPW + L.grp;
            const bool act = L.grp < L.GPW && pos < A.n;
            int32_t i = 0;
            double y = 0.0;
            if (act) {
                i = A.rows ? A.rows[pos] : static_cast<int32_t>(pos);
                const int64_t t = int64_t(i) * BS + L.ii;
                double xv = x[t] + alpha * zp[t];
                xv = xv + omega * zs[t];
                x[t] = xv;
                const double rv = s[t] + (-omega) * tv[t];
                r[t] = rv;
                double pv = beta * p[t];
                pv = pv + (-beta * omega) * v[t];
                pv = pv + 1.0 * rv;
                p[t] = pv;
                pr[0] += rv * rv;
                if (pos < A.n1) y = pv - cp * w[t];
            }
            if (A.n0 + wq * L.GPW >= A.n1) continue;  // warp-uniform: past colour 1
            const bool c1 = act && pos < A.n1;
            const double o = apply_dinv<BS>(dinv, i, L.ii, L.base, c1, y);
            if (c1) zp[int64_t(i) * BS + L.ii] = o;
        }
    }
    double tot[1];
    if (!grid_sums<1>(pr, partials, &ks->arrived, tot) || threadIdx.x != 0) return;
    if (run) {
        const double omega_new = ks->omega_new;
        double rnorm = ks->rnorm;
        if (!isfinite(rnorm) || !isfinite(omega_new) || omega_new == 0.0) {
            ks->state = KS_DIVERGED;
        } else {
            if (ks->it % 32 == 0) {
                rnorm = sqrt(tot[0] + ks->cr * ks->cr * ks->q0);
                ks->rnorm = rnorm;
            }
            if (rnorm <= ks->tol) {
                ks->state = KS_CONVERGED;
            } else if (!isfinite(ks->rho_new) || ks->rho_new == 0.0) {
                ks->state = KS_DIVERGED;
            } else {
                ks->rho = ks->rho_new;
                ks->omega = omega_new;
                ks->cp = ks->cp_new;
            }
        }
    }
    // the loop ends after at most max_it runs of its body whatever the state
    ks->body_runs += 1;
    if (use_cond) cudaGraphSetConditional(cond, ks->state == KS_RUNNING && ks->body_runs < ks->max_it ? 1u : 0u);
}

// The while-condition before the first body run.
__global__ void k_red_enter(const KrylovScalars* ks, cudaGraphConditionalHandle cond) {
    if (threadIdx.x == 0) cudaGraphSetConditional(cond, ks->state == KS_RUNNING && ks->max_it > 0 ? 1u : 0u);
}

// Sets *flag when a diagonal block amplifies the rounding of the reduced
// product.  With s = D v, the full product is wrong by about eps |D||v| and the
// reduced one by eps |D||D^-1||s|, so in a norm that follows the scales of the
// block's rows the loss is at most the norm of G = |D||D^-1|.  Scaled by a
// positive x that norm is max_i (G x)_i / x_i, and three steps x <- G x bring it
// close to its least value, the spectral radius: equations or variables in
// other units change nothing (a transport Jacobian has 1.0 to 1.3 in SI units,
// where cond(D) is 1e8), coupled stiff terms do.  Limit 8: on matrices whose blocks
// have 4 to 8, both forms end at the same true residual, 2.6e-16 |b| (the worst
// 1.25 times the other's); at 16 to 23 the reduced form ends at 1.7 times the
// full one's, at 90 to 128 at 6 times, at 1e8 at 1e7 times.  Bound by L1 wavefronts
// and shuffles (a lane holds a row of both factors): set-up of 480k rows of 5x5
// 94 -> 143 us, of 48k 31 -> 33, where an iteration of the solve saves 300 and 30; a
// thread per block, staged through shared memory, spilled and took 170.
constexpr double kGrowthLimit = 8.0;

template <int BS>
__global__ void __launch_bounds__(kThreads) k_red_check(RedView A, const double* vals, const double* dinv, int* flag) {
    pdl_enter();
    const Lanes<BS> L;
    const int64_t i = warp_id() * L.GPW + L.grp;
    const bool act = L.grp < L.GPW && i < A.n;
    double d[BS], v[BS];
    const double* dp = vals + (act ? int64_t(A.diag[i]) : 0) * (BS * BS) + L.ii * BS;
    const double* vp = dinv + (act ? i : 0) * (BS * BS) + L.ii * BS;
#pragma unroll
    for (int j = 0; j < BS; ++j) {
        d[j] = act ? fabs(dp[j]) : 0.0;
        v[j] = act ? fabs(vp[j]) : 0.0;
    }
    auto times = [&](const double (&m)[BS], double x) {
        double y = 0.0;
#pragma unroll
        for (int j = 0; j < BS; ++j) y += m[j] * __shfl_sync(0xffffffffu, x, L.base + j);
        return y;
    };
    double x = 1.0, y = 1.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        x = y;
        y = times(d, times(v, x));
    }
    if (act && !(y <= kGrowthLimit * x)) *flag = 1;  // not finite: over the limit too
}

template <int BS>
unsigned capped_grid(int64_t rows, int64_t cap) {
    const int64_t warps = (rows + (32 / BS) - 1) / (32 / BS);
    const int64_t g = (warps + kThreads / 32 - 1) / (kThreads / 32);
    return static_cast<unsigned>(g < 1 ? 1 : (g < cap ? g : cap));
}

template <typename F>
void by_block_size(int bs, F&& f) {
    switch (bs) {
        case 1: f(std::integral_constant<int, 1>{}); break;
        case 3: f(std::integral_constant<int, 3>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        default: break;
    }
}

}  // namespace

int red_partials() { return static_cast<int>(kGridCap) * 5; }

void launch_red_init(const RedView& A, KrylovScalars* ks, const double* v, double* r, double* r0, double* p,
                     double* partials, bool guess, cudaStream_t st) {
    by_block_size(A.bs, [&](auto c) {
        constexpr int BS = decltype(c)::value;
        const unsigned g = capped_grid<BS>(A.n, kGridCap);
        k_red_init<BS><<<g, kThreads, 0, st>>>(A, ks, v, r, r0, p, partials);
        if (guess) k_red_guess_reset<BS><<<g, kThreads, 0, st>>>(A, ks, r, r0, p);
    });
}

void launch_red_sweep(const RedView& A, const double* vals, const double* dinv, int kind, int32_t pos0, int32_t pos1,
                      const double* src, const double* w, double* z, double* e, const KrylovScalars* ks, bool second,
                      cudaStream_t st) {
    if (pos1 <= pos0) return;
    by_block_size(A.bs, [&](auto c) {
        constexpr int BS = decltype(c)::value;
        const unsigned g = capped_grid<BS>(pos1 - pos0, int64_t(1) << 31);
        auto go = [&](auto list, auto k) {
            k_red_sweep<BS, decltype(list)::value, decltype(k)::value>
                <<<g, kThreads, 0, st>>>(A, vals, dinv, pos0, pos1, src, w, z, e, ks, second ? 1 : 0);
        };
        auto by_list = [&](auto k) {
            if (A.rows) go(std::true_type{}, k);
            else go(std::false_type{}, k);
        };
        switch (kind) {
            case RED_BACK0: by_list(std::integral_constant<int, BACK0>{}); break;
            case RED_BACK: go(std::false_type{}, std::integral_constant<int, BACK>{}); break;  // three colours up
            case RED_FWD: by_list(std::integral_constant<int, FWD>{}); break;
            case RED_ETA: by_list(std::integral_constant<int, ETA>{}); break;
            case RED_WSUM: by_list(std::integral_constant<int, WSUM>{}); break;
            default: by_list(std::integral_constant<int, XRED>{}); break;
        }
    });
}

void launch_red_product(const RedView& A, const double* vals, const double* src, const double* e, double* out,
                        const double* r0, KrylovScalars* ks, double* partials, bool first, cudaStream_t st) {
    by_block_size(A.bs, [&](auto c) {
        constexpr int BS = decltype(c)::value;
        // exactly the resident blocks of the launch bounds
        const unsigned g = capped_grid<BS>(A.n - A.n0, 148 * (BS <= 5 ? 6 : 5));
        auto go = [&](auto list, auto f) {
            k_red_product<BS, decltype(list)::value, decltype(f)::value>
                <<<g, kThreads, 0, st>>>(A, vals, src, e, out, r0, ks, partials);
        };
        if (A.rows) first ? go(std::true_type{}, std::true_type{}) : go(std::true_type{}, std::false_type{});
        else first ? go(std::false_type{}, std::true_type{}) : go(std::false_type{}, std::false_type{});
    });
}

void launch_red_s(const RedView& A, const double* dinv, const double* r, const double* v, const double* w, double* s,
                  double* z, const KrylovScalars* ks, cudaStream_t st) {
    by_block_size(A.bs, [&](auto c) {
        constexpr int BS = decltype(c)::value;
        k_red_s<BS><<<capped_grid<BS>(A.n - A.n0, kGridCap), kThreads, 0, st>>>(A, dinv, r, v, w, s, z, ks);
    });
}

void launch_red_update(const RedView& A, const double* dinv, const double* zs, const double* s, const double* t,
                       const double* v, const double* w, double* r, double* p, double* zp, KrylovScalars* ks,
                       double* partials, cudaGraphConditionalHandle cond, bool use_cond, cudaStream_t st) {
    by_block_size(A.bs, [&](auto c) {
        constexpr int BS = decltype(c)::value;
        k_red_update<BS><<<capped_grid<BS>(A.n - A.n0, kGridCap), kThreads, 0, st>>>(
            A, dinv, zs, s, t, v, w, r, p, zp, ks, partials, cond, use_cond ? 1 : 0);
    });
}

void launch_red_check(const RedView& A, const double* vals, const double* dinv, int* flag, cudaStream_t st) {
    by_block_size(A.bs, [&](auto c) {
        constexpr int BS = decltype(c)::value;
        launch_after(k_red_check<BS>, capped_grid<BS>(A.n, int64_t(1) << 31), kThreads, 0, st, A, vals, dinv, flag);
    });
}

void launch_red_enter(const KrylovScalars* ks, cudaGraphConditionalHandle cond, cudaStream_t st) {
    k_red_enter<<<1, 32, 0, st>>>(ks, cond);
}

}  // namespace cfdg
