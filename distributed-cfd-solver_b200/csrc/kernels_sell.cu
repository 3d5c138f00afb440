// The multicolour sweep and its product on a sliced copy of a colour-ordered
// matrix that does not stay in L2.
//
// Reading a 5x5 or 6x6 block with one component a lane costs an L1 wavefront
// for every block row, since each load touches all of them; that, not DRAM, held
// the row-by-row passes to 3.1 TB/s (5x5 FP32), 4.0 (6x6 FP32) and 5.0 (5x5
// FP64).  Here a lane has a whole row: the k-th blocks of 32 rows are one column
// of 32 * BS^2 consecutive values, entry e of lane l at e * 32 + l.  Rows of one
// colour are ordered by their block counts within windows of 256, so that the
// 32 rows of a slice end together (tetrahedra: up to four blocks on a side).
//
// FP32 (k_sell_ring): with 4-byte entries a lane has too few bytes in flight
// from registers alone.  A column is contiguous (3.2 or 4.6 KB) and a warp's
// columns are known ahead, so each warp streams its own through a ring of
// kStages in shared memory (cp.async, no barrier but the warp's), across slice
// boundaries, and gathers the neighbours' vector entries one column ahead.  516k
// 6x6 rows: 5.2 TB/s, 4.0 row by row; 768k tetrahedra: 3.8, 3.2.  All passes of a
// sweep as one cooperative launch were slower (12.0 ms against 10.6), gathers
// then having to go through L2.
// FP64 5x5 (k_sell_rows): one slice a warp, straight from memory, which
// measured faster there (sweeps of 1M hex cells 17.5 ms against 18.7, 21.6 row
// by row); 6x6 FP64 blocks run at 0.94 of the copy bandwidth row by row.
//
// A row's arithmetic is that of k_sgs_rows / k_spmv / k_sgs_last_spmv: blocks in
// ascending column order, each block's partial sum formed first, D^-1 as a
// block-row product; k_dots forms the inner products in their order, so the
// iterates are the same to the bit.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "krylov.hpp"

namespace cfdg {
namespace {

constexpr int kCopyThreads = 128;
constexpr int kSellThreads = 128;
constexpr int kStages = 4;  // one being read, its successor complete, two in flight

// Copies the blocks of each slice column (32 blocks, one per row) from the
// row-by-row array: a warp reads them one by one, coalesced, and writes the
// entries transposed.  src[column * 32 + lane]: block index, -1 where the row
// has none.
template <typename MT, int BS>
__global__ void __launch_bounds__(kCopyThreads) k_sell_copy(int64_t columns, const int32_t* __restrict__ src,
                                                            const MT* __restrict__ from, MT* __restrict__ to) {
    constexpr int B2 = BS * BS, SP = B2 % 2 == 0 ? B2 + 1 : B2;  // odd stride: distinct banks
    __shared__ MT sm[kCopyThreads / 32][32 * SP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t col = int64_t(blockIdx.x) * (kCopyThreads / 32) + warp;
    if (col >= columns) return;  // whole warps
    const int32_t mine = __ldg(src + col * 32 + lane);
    MT* s = sm[warp];
#pragma unroll 8
    for (int q = 0; q < 32; ++q) {
        const int32_t b = __shfl_sync(0xffffffffu, mine, q);
        if (b < 0) continue;
        const MT* g = from + int64_t(b) * B2;
        if (lane < B2) s[q * SP + lane] = __ldg(g + lane);
        if (B2 > 32 && lane < B2 - 32) s[q * SP + 32 + lane] = __ldg(g + 32 + lane);
    }
    __syncwarp();
    if (mine < 0) return;
    MT* o = to + col * (B2 * 32) + lane;
#pragma unroll
    for (int e = 0; e < B2; ++e) o[e * 32] = s[lane * SP + e];
}

template <int BS>
__device__ __forceinline__ void load_vec(const double* __restrict__ x, double (&out)[BS]) {
    if constexpr (BS == 6) {  // a row of a 6-variable vector is 48 bytes
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            const double2 v = __ldg(reinterpret_cast<const double2*>(x) + h);
            out[2 * h] = v.x;
            out[2 * h + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < BS; ++j) out[j] = __ldg(x + j);
    }
}
template <int BS>
__device__ __forceinline__ void store_vec(double* x, const double (&v)[BS]) {
    if constexpr (BS == 6) {
#pragma unroll
        for (int h = 0; h < 3; ++h) reinterpret_cast<double2*>(x)[h] = make_double2(v[2 * h], v[2 * h + 1]);
    } else {
#pragma unroll
        for (int j = 0; j < BS; ++j) x[j] = v[j];
    }
}

// acc (+|-)= the lane's block of a column times x, one row's sum at a time
template <typename MT, int BS, bool SUB>
__device__ __forceinline__ void block_times(const MT* a, const double (&x)[BS], double (&acc)[BS]) {
#pragma unroll
    for (int i = 0; i < BS; ++i) {
        double t = 0.0;
#pragma unroll
        for (int j = 0; j < BS; ++j) t += static_cast<double>(a[(i * BS + j) * 32]) * x[j];
        acc[i] = SUB ? acc[i] - t : acc[i] + t;
    }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// The blocks are read once a pass: leaving them first in L2 keeps the vectors
// there (516k 6x6 rows: sweeps 7.45 -> 6.97 ms, products 3.10 -> 2.85).
__device__ __forceinline__ uint64_t streaming() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

template <int KIND>
struct Pass {
    static constexpr bool low = KIND == SELL_LOW || KIND == SELL_FULL || KIND == SELL_MUL;
    static constexpr bool up = KIND == SELL_UP || KIND == SELL_UPY || KIND == SELL_FULL || KIND == SELL_MUL;
    // d = {first lower column, their count, first upper column, their count}
    static __device__ __forceinline__ int neighbours(int4 d) { return (low ? d.y : 0) + (up ? d.w : 0); }
    // columns a slice takes: the neighbours' and D^-1 (MUL: the diagonal blocks
    // between lower and upper; UPY: and the diagonal blocks)
    static __device__ __forceinline__ int count(int4 d) { return neighbours(d) + (KIND == SELL_UPY ? 2 : 1); }
    // columns multiplied by gathered vector entries
    static __device__ __forceinline__ int gathers(int4 d) { return neighbours(d) + (KIND == SELL_MUL ? 1 : 0); }
    // column e of the values, -1: the slice's column of D^-1
    static __device__ __forceinline__ int column(int4 d, int diag, int e) {
        if (KIND == SELL_MUL) return e < d.y ? d.x + e : e == d.y ? diag : d.z + e - d.y - 1;
        if (low && e < d.y) return d.x + e;
        if (up && e - (low ? d.y : 0) < d.w) return d.z + e - (low ? d.y : 0);
        return KIND == SELL_UPY && e > d.w ? diag : -1;
    }
    // whether the lane's row, len blocks below and above, has a block there
    static __device__ __forceinline__ bool has(int4 d, int2 len, int e) {
        if (KIND == SELL_MUL) return e < d.y ? e < len.x : e == d.y || e - d.y - 1 < len.y;
        if (low && e < d.y) return e < len.x;
        return up && e - (low ? d.y : 0) < len.y;
    }
};

// A column and the block columns of its 32 blocks.
template <typename MT, int BS>
constexpr int kStageBytes = 32 * BS * BS * int(sizeof(MT)) + 128;

// Slices [s0, s1) of one pass (SELL_* in krylov.hpp), the resident warps
// striding over them.  Bound by the blocks read from DRAM.
template <typename MT, int BS, int KIND>
__global__ void __launch_bounds__(kSellThreads) k_sell_ring(SellView A, const MT* __restrict__ vals,
                                                            const MT* __restrict__ dinv, int32_t s0, int32_t s1,
                                                            const double* __restrict__ r, double* z,
                                                            double* __restrict__ y, const int* __restrict__ active) {
    if (active && *active != 0) return;
    using P = Pass<KIND>;
    constexpr int B2 = BS * BS, COL = 32 * B2 * int(sizeof(MT)), STAGE = kStageBytes<MT, BS>;
    constexpr bool RHS = KIND == SELL_DIAG || KIND == SELL_LOW || KIND == SELL_FULL;
    constexpr bool OLD = KIND == SELL_UP || KIND == SELL_UPY;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = gridDim.x * (kSellThreads / 32);
    const int first = s0 + blockIdx.x * (kSellThreads / 32) + warp;
    if (first >= s1) return;
    const uint64_t policy = streaming();
    unsigned char* ring = smem + warp * (kStages * STAGE);
    const uint32_t ring_addr = smem_addr(ring);
    auto desc = [&](int s) { return s < s1 ? __ldg(A.desc + s) : make_int4(0, 0, 0, 0); };

    // the next column to fetch
    int ps = first, pe = 0, slot_in = 0;
    int4 pd = desc(ps), pn = desc(ps + nw);
    auto fetch = [&]() {
        if (ps < s1) {
            const int c = P::column(pd, A.diag0 + ps, pe);
            const uint32_t dst = ring_addr + slot_in * STAGE;
            const char* src = c >= 0 ? reinterpret_cast<const char*>(vals) + int64_t(c) * COL
                                     : reinterpret_cast<const char*>(dinv) + int64_t(ps) * COL;
#pragma unroll
            for (int q = 0; q < COL / 16; q += 32)
                if (q + 32 <= COL / 16 || q + lane < COL / 16)
                    copy16(dst + (q + lane) * 16, src + (q + lane) * 16, policy);
            if (c >= 0) copy4(dst + COL + lane * 4, A.cols + int64_t(c) * 32 + lane);
            if (++pe == P::count(pd)) {
                pe = 0;
                ps += nw;
                pd = pn;
                pn = desc(ps + nw);
            }
        }
        slot_in = slot_in + 1 == kStages ? 0 : slot_in + 1;
        copies_commit();
    };
    static_assert(kStages == 4);
    fetch();
    fetch();
    fetch();

    auto row_of = [&](int s) { return s < s1 ? __ldg(A.row + int64_t(s) * 32 + lane) : -1; };
    auto own_of = [&](int32_t i, double (&v)[BS]) {
#pragma unroll
        for (int j = 0; j < BS; ++j) v[j] = 0.0;
        if (i < 0) return;
        if (RHS) load_vec<BS>(r + int64_t(i) * BS, v);
        if (OLD) {  // written below, by this lane
#pragma unroll
            for (int j = 0; j < BS; ++j) v[j] = z[int64_t(i) * BS + j];
        }
    };
    int slot = 0;
    double x[BS], own_next[BS];
    auto gather = [&](int at, double (&v)[BS]) {
        const int32_t c = reinterpret_cast<const int32_t*>(ring + at * STAGE + COL)[lane];
        load_vec<BS>(z + int64_t(c) * BS, v);
    };
    int4 d = desc(first), dn = desc(first + nw);
    int32_t i = row_of(first), i_next = row_of(first + nw);
    own_of(i, own_next);
    copies_wait<2>();
    __syncwarp();
    if (P::gathers(d) > 0) gather(0, x);
    for (int s = first; s < s1; s += nw) {
        double own[BS], acc[BS], out[BS];
#pragma unroll
        for (int j = 0; j < BS; ++j) {
            own[j] = own_next[j];
            acc[j] = RHS ? own[j] : 0.0;
            out[j] = 0.0;
        }
        const int2 len = __ldg(A.len + int64_t(s) * 32 + lane);
        const int64_t t = int64_t(i) * BS;
        own_of(i_next, own_next);
        const int32_t i_after = row_of(s + 2 * nw);
        const int n = P::count(d), ng = P::gathers(d);
        for (int e = 0; e < n; ++e) {
            copies_wait<1>();  // this column and the next
            __syncwarp();
            fetch();  // over the column read last
            const int next = slot + 1 == kStages ? 0 : slot + 1;
            double xn[BS];
            if (e + 1 < n ? e + 1 < ng : s + nw < s1 && P::gathers(dn) > 0) {
                gather(next, xn);
            } else {
#pragma unroll
                for (int j = 0; j < BS; ++j) xn[j] = 0.0;
            }
            const MT* a = reinterpret_cast<const MT*>(ring + slot * STAGE) + lane;
            if (e < ng) {
                if (P::has(d, len, e)) block_times<MT, BS, KIND != SELL_MUL>(a, x, acc);
            } else if (KIND == SELL_UPY && e == n - 1) {  // (A z)_i = sum_upper A z + A_ii z_i
                double p[BS];
#pragma unroll
                for (int j = 0; j < BS; ++j) p[j] = 0.0;
                block_times<MT, BS, false>(a, out, p);
#pragma unroll
                for (int j = 0; j < BS; ++j) p[j] = p[j] - acc[j];
                if (i >= 0) store_vec<BS>(y + t, p);
            } else {
                block_times<MT, BS, false>(a, acc, out);
                if (OLD) {
#pragma unroll
                    for (int j = 0; j < BS; ++j) out[j] = own[j] + out[j];
                }
                if (i >= 0) store_vec<BS>(z + t, out);
            }
#pragma unroll
            for (int j = 0; j < BS; ++j) x[j] = xn[j];
            slot = next;
        }
        if (KIND == SELL_MUL && i >= 0) store_vec<BS>(y + t, acc);
        d = dn;
        dn = desc(s + 2 * nw);
        i = i_next;
        i_next = i_after;
    }
    copies_wait<0>();
}

// The same pass, a slice a warp, the blocks straight from memory: a lane's 25
// entries of a block are independent loads.
template <typename MT, int BS, int KIND>
__global__ void __launch_bounds__(kSellThreads) k_sell_rows(SellView A, const MT* __restrict__ vals,
                                                            const MT* __restrict__ dinv, int32_t s0, int32_t s1,
                                                            const double* __restrict__ r, double* z,
                                                            double* __restrict__ y, const int* __restrict__ active) {
    if (active && *active != 0) return;
    constexpr int B2 = BS * BS;
    constexpr bool LOWER = KIND == SELL_LOW || KIND == SELL_FULL || KIND == SELL_MUL;
    constexpr bool UPPER = KIND == SELL_UP || KIND == SELL_UPY || KIND == SELL_FULL || KIND == SELL_MUL;
    constexpr bool SUB = KIND != SELL_MUL;
    const int lane = threadIdx.x & 31;
    const int32_t sl = s0 + static_cast<int32_t>((int64_t(blockIdx.x) * kSellThreads + threadIdx.x) >> 5);
    if (sl >= s1) return;
    const int32_t i = __ldg(A.row + int64_t(sl) * 32 + lane);
    if (i < 0) return;
    const int64_t t = int64_t(i) * BS;
    double acc[BS];
    if constexpr (KIND == SELL_DIAG || KIND == SELL_LOW || KIND == SELL_FULL) {
        load_vec<BS>(r + t, acc);
    } else {
#pragma unroll
        for (int j = 0; j < BS; ++j) acc[j] = 0.0;
    }
    // a row's blocks fill the first columns of its slice
    auto side = [&](int64_t c0, int len) {
        if (len == 0) return;
        int32_t col = __ldg(A.cols + c0 * 32 + lane);
        for (int k = 0; k < len; ++k) {
            const int64_t c = c0 + k;
            const int32_t next = k + 1 < len ? __ldg(A.cols + (c + 1) * 32 + lane) : col;
            double x[BS];
            load_vec<BS>(z + int64_t(col) * BS, x);
            block_times<MT, BS, SUB>(vals + c * (B2 * 32) + lane, x, acc);
            col = next;
        }
    };
    const int4 d = __ldg(A.desc + sl);
    const int2 len = __ldg(A.len + int64_t(sl) * 32 + lane);
    if (LOWER) side(d.x, len.x);
    if constexpr (KIND == SELL_MUL) {
        double x[BS];
        load_vec<BS>(z + t, x);
        block_times<MT, BS, false>(vals + int64_t(A.diag0 + sl) * (B2 * 32) + lane, x, acc);
    }
    if (UPPER) side(d.z, len.y);
    if constexpr (KIND == SELL_MUL) {
        store_vec<BS>(y + t, acc);
    } else {
        double out[BS];
#pragma unroll
        for (int j = 0; j < BS; ++j) out[j] = 0.0;
        block_times<MT, BS, false>(dinv + int64_t(sl) * (B2 * 32) + lane, acc, out);
        if constexpr (KIND == SELL_UP || KIND == SELL_UPY) {
#pragma unroll
            for (int j = 0; j < BS; ++j) out[j] = z[t + j] + out[j];
        }
        store_vec<BS>(z + t, out);
        if constexpr (KIND == SELL_UPY) {  // (A z)_i = sum_upper A z + A_ii z_i
            double d[BS];
#pragma unroll
            for (int j = 0; j < BS; ++j) d[j] = 0.0;
            block_times<MT, BS, false>(vals + int64_t(A.diag0 + sl) * (B2 * 32) + lane, out, d);
#pragma unroll
            for (int j = 0; j < BS; ++j) d[j] = d[j] - acc[j];
            store_vec<BS>(y + t, d);
        }
    }
}

// Blocks that share an SM (0: the ring does not fit), cached per device.
template <typename MT, int BS, int KIND>
int sell_grid() {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cache[kMaxDevices];  // 0: unknown, -1: unavailable
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        return 0;
    }
    int grid = cache[dev].load();
    if (grid == 0) {
        constexpr int bytes = kSellThreads / 32 * kStages * kStageBytes<MT, BS>;
        auto* fn = k_sell_ring<MT, BS, KIND>;
        int sms = 0, per_sm = 0;
        grid = -1;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSellThreads, bytes) == cudaSuccess &&
            per_sm > 0)
            grid = sms * per_sm;
        cudaGetLastError();
        cache[dev].store(grid);
    }
    return grid > 0 ? grid : 0;
}

template <typename F>
auto by_kind(int kind, F&& f) {
    switch (kind) {
        case SELL_DIAG: return f(std::integral_constant<int, SELL_DIAG>{});
        case SELL_LOW: return f(std::integral_constant<int, SELL_LOW>{});
        case SELL_UP: return f(std::integral_constant<int, SELL_UP>{});
        case SELL_UPY: return f(std::integral_constant<int, SELL_UPY>{});
        case SELL_FULL: return f(std::integral_constant<int, SELL_FULL>{});
        default: return f(std::integral_constant<int, SELL_MUL>{});
    }
}

template <typename MT, int BS>
void rows(const SellView& A, const MT* vals, const MT* dinv, int kind, int32_t s0, int32_t s1, const double* r,
          double* z, double* y, const int* active, cudaStream_t st) {
    by_kind(kind, [&](auto kc) {
        constexpr int KIND = decltype(kc)::value, W = kSellThreads / 32;
        if constexpr (sizeof(MT) == 4) {
            const int grid = std::min(sell_grid<MT, BS, KIND>(), (s1 - s0 + W - 1) / W);
            k_sell_ring<MT, BS, KIND><<<grid, kSellThreads, W * kStages * kStageBytes<MT, BS>, st>>>(
                A, vals, dinv, s0, s1, r, z, y, active);
        } else {
            k_sell_rows<MT, BS, KIND><<<(s1 - s0 + W - 1) / W, kSellThreads, 0, st>>>(A, vals, dinv, s0, s1, r, z, y,
                                                                                   active);
        }
    });
}

}  // namespace

// Block sizes and types with slices: 5x5, and 6x6 in FP32.
bool sell_ready(int bs, bool mixed) {
    if (!mixed) return bs == 5;
    for (int kind : {SELL_DIAG, SELL_LOW, SELL_UP, SELL_UPY, SELL_FULL, SELL_MUL})
        if (by_kind(kind, [&](auto kc) {
                constexpr int KIND = decltype(kc)::value;
                return bs == 6 ? sell_grid<float, 6, KIND>() : bs == 5 ? sell_grid<float, 5, KIND>() : 0;
            }) <= 0)
            return false;
    return true;
}

template <typename MT>
void launch_sell_copy(int bs, int64_t columns, const int32_t* src, const MT* from, MT* to, cudaStream_t s) {
    if (columns <= 0) return;
    const unsigned g = grid_for(columns * 32, kCopyThreads);
    if constexpr (sizeof(MT) == 4)
        if (bs == 6) return k_sell_copy<MT, 6><<<g, kCopyThreads, 0, s>>>(columns, src, from, to);
    k_sell_copy<MT, 5><<<g, kCopyThreads, 0, s>>>(columns, src, from, to);
}

template <typename MT>
void launch_sell_rows(const SellView& A, const MT* vals, const MT* dinv, int kind, int32_t s0, int32_t s1,
                      const double* r, double* z, double* y, const int* active, cudaStream_t s) {
    if (s1 <= s0) return;
    if constexpr (sizeof(MT) == 4)
        if (A.bs == 6) return rows<MT, 6>(A, vals, dinv, kind, s0, s1, r, z, y, active, s);
    rows<MT, 5>(A, vals, dinv, kind, s0, s1, r, z, y, active, s);
}

template void launch_sell_copy<double>(int, int64_t, const int32_t*, const double*, double*, cudaStream_t);
template void launch_sell_copy<float>(int, int64_t, const int32_t*, const float*, float*, cudaStream_t);
template void launch_sell_rows<double>(const SellView&, const double*, const double*, int, int32_t, int32_t,
                                       const double*, double*, double*, const int*, cudaStream_t);
template void launch_sell_rows<float>(const SellView&, const float*, const float*, int, int32_t, int32_t,
                                      const double*, double*, double*, const int*, cudaStream_t);

}  // namespace cfdg
