// Restarted GMRES building blocks (right-preconditioned, classical
// Gram-Schmidt with one reorthogonalisation pass).  The Krylov basis is one
// array of (restart + 1) vectors of `len` doubles; the projections go
// through fused multi-dot products (up to gm_chunk(len) basis vectors against w
// per launch, w read once per launch) and one fused update
// w -= sum_k h_k V_k.  Reductions are per block in a fixed order, then a
// finaliser per coefficient over the blocks in block order: the grid depends
// only on the length, so the coefficients repeat run to run.
#include "kernels.hpp"

namespace cfdg {

namespace {

constexpr int kGmThreads = 256;
constexpr int64_t kGmGridCap = 148 * 8;
constexpr int kGmChunk = 24, kGmLongChunk = 8;

inline unsigned gm_grid(int64_t len) {
    const int64_t g = grid_for(len, kGmThreads);
    return static_cast<unsigned>(g < kGmGridCap ? g : kGmGridCap);
}

// partials[b * C + k] = sum over block b's entries of V_{k0+k} . w, k < kn
// (kn <= C).  V = w with kn = 1 gives |w|^2.  While a thread has one entry (up to
// 303,104), a launch is latency: all C basis entries load at once, and C follows
// the number of vectors (8, 16 or 24) so that a basis of 24 is one launch instead
// of three.  Longer vectors are bound by memory, where the fewer blocks that 24
// sums leave room for cost more than reading w again: they go by eight.  The 60
// launches' products of a 30-vector cycle, us, 24 / 8 a launch: 725 / 902 at 80k
// entries, 1,423 / 1,479 at 240k, 2,413 / 2,152 at 655k, 9,391 / 7,173 at 4.1M.  With
// the update's norm in the same pass and the host reading a column while the next
// product runs, a Jacobian-free step of the 131k-cell plate takes 7.08 ms instead
// of 7.20.
template <int C>
__global__ void __launch_bounds__(kGmThreads) k_gm_dots(int64_t len, const double* V, int64_t ld, int k0,
                                                        int kn, const double* w,
                                                        double* partials) {
    pdl_enter();
    double s[C];
#pragma unroll
    for (int k = 0; k < C; ++k) s[k] = 0.0;
    for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < len; t += int64_t(gridDim.x) * blockDim.x) {
        const double wt = w[t];
#pragma unroll
        for (int k = 0; k < C; ++k)
            if (k < kn) s[k] += V[int64_t(k0 + k) * ld + t] * wt;
    }
    block_reduce_store<C, kGmThreads>(s, partials + size_t(blockIdx.x) * C);
}

// h[k0 + k] = sum over blocks of partials[b * stride + k], one warp per
// coefficient: lane-strided sums in block order, then a fixed shuffle tree.
__global__ void k_gm_dots_fin(int nblocks, int stride, int k0, int kn, const double* partials,
                              double* h) {
    pdl_enter();
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= kn) return;
    double s = 0.0;
#pragma unroll 8
    for (int b = lane; b < nblocks; b += 32) s += partials[size_t(b) * stride + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) h[k0 + k] = s;
}

// w -= sum_{k < kn} h_k V_k  (SUBTRACT), or w = sum_{k < kn} h_k V_k (the
// combination of the basis with the least-squares solution).  NORM: partials of
// the new |w|^2 as k_gm_dots forms them.  Eight basis entries load at once; the
// sum stays in order.
template <bool SUBTRACT, bool NORM>
__global__ void __launch_bounds__(kGmThreads) k_gm_update(int64_t len, const double* V, int64_t ld, int kn,
                                                          const double* h, double* w,
                                                          double* partials) {
    pdl_enter();
    constexpr int U = 8;
    double s[1] = {0.0};
    for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < len; t += int64_t(gridDim.x) * blockDim.x) {
        double acc = SUBTRACT ? w[t] : 0.0;
        for (int k = 0; k < kn; k += U) {
            double v[U], c[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int q = k + u < kn ? k + u : kn - 1;
                c[u] = h[q];
                v[u] = V[int64_t(q) * ld + t];
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k + u < kn) acc = SUBTRACT ? acc - c[u] * v[u] : acc + c[u] * v[u];
        }
        w[t] = acc;
        if (NORM) s[0] += acc * acc;
    }
    if (NORM) block_reduce_store<1, kGmThreads>(s, partials + blockIdx.x);
}

// w /= sqrt(*norm2): the basis vector of a Gram-Schmidt residual
__global__ void __launch_bounds__(kGmThreads) k_gm_normalise(int64_t len, const double* norm2,
                                                             double* w) {
    pdl_enter();
    const double a = 1.0 / sqrt(fmax(*norm2, 0.0));
    for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < len; t += int64_t(gridDim.x) * blockDim.x)
        w[t] = a * w[t];
}

// y = a x (+ y when accumulate)
__global__ void __launch_bounds__(kGmThreads) k_gm_axpy(int64_t len, double a, const double* x,
                                                        double* y, int accumulate) {
    pdl_enter();
    for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < len; t += int64_t(gridDim.x) * blockDim.x)
        y[t] = accumulate ? y[t] + a * x[t] : a * x[t];
}

}  // namespace

int gm_partial_blocks(int64_t len) { return static_cast<int>(gm_grid(len)); }
int gm_chunk(int64_t len) { return len <= kGmGridCap * kGmThreads ? kGmChunk : kGmLongChunk; }

void launch_gm_dots(int64_t len, const double* V, int64_t ld, int k0, int kn, const double* w, double* partials,
                    double* h, cudaStream_t s) {
    const unsigned gr = gm_grid(len);
    const int chunk = gm_chunk(len);
    for (int c = 0; c < kn; c += chunk) {
        const int m = kn - c < chunk ? kn - c : chunk;
        const int stride = m == 1 ? 1 : m <= 8 ? 8 : m <= 16 ? 16 : 24;
        if (m == 1) launch_after(k_gm_dots<1>, gr, kGmThreads, 0, s, len, V, ld, k0 + c, m, w, partials);
        else if (m <= 8) launch_after(k_gm_dots<8>, gr, kGmThreads, 0, s, len, V, ld, k0 + c, m, w, partials);
        else if (m <= 16) launch_after(k_gm_dots<16>, gr, kGmThreads, 0, s, len, V, ld, k0 + c, m, w, partials);
        else launch_after(k_gm_dots<24>, gr, kGmThreads, 0, s, len, V, ld, k0 + c, m, w, partials);
        launch_after(k_gm_dots_fin, 1, 32 * m, 0, s, static_cast<int>(gr), stride, k0 + c, m, partials, h);
    }
}

void launch_gm_update(int64_t len, const double* V, int64_t ld, int kn, const double* h, double* w, bool subtract,
                      cudaStream_t s) {
    if (subtract) launch_after(k_gm_update<true, false>, gm_grid(len), kGmThreads, 0, s, len, V, ld, kn, h, w, nullptr);
    else launch_after(k_gm_update<false, false>, gm_grid(len), kGmThreads, 0, s, len, V, ld, kn, h, w, nullptr);
}

void launch_gm_update_norm(int64_t len, const double* V, int64_t ld, int kn, const double* h, double* w,
                           double* partials, double* norm2, cudaStream_t s) {
    const unsigned gr = gm_grid(len);
    launch_after(k_gm_update<true, true>, gr, kGmThreads, 0, s, len, V, ld, kn, h, w, partials);
    launch_after(k_gm_dots_fin, 1, 32, 0, s, static_cast<int>(gr), 1, 0, 1, partials, norm2);
}

void launch_gm_normalise(int64_t len, const double* norm2, double* w, cudaStream_t s) {
    launch_after(k_gm_normalise, gm_grid(len), kGmThreads, 0, s, len, norm2, w);
}

void launch_gm_axpy(int64_t len, double a, const double* x, double* y, bool accumulate, cudaStream_t s) {
    launch_after(k_gm_axpy, gm_grid(len), kGmThreads, 0, s, len, a, x, y, accumulate ? 1 : 0);
}

}  // namespace cfdg
