// fp32 products on the CUDA cores: D[i][j] = sum_k P(i, k) * Q(j, k) with exact fp32 FMAs in k order, for CB_MATH_FP32
// and for operands the TMA-fed kernels cannot address (rows TMA cannot start at, convolution geometries outside conv_sm100.cu),
// where a product is too small for split_core.cuh or belongs to a model's pass. One kernel body serves the GEMM forms and the three
// convolution passes; an operand source (below) says where element (i, k) lies.
//
// What bounds it: the fp32 pipe (128 FMA per SM and clock) as long as the extents are large, so everything is laid out to
// leave the issue slots to FMAs: 8 x 8 (or 8 x 4) outputs per thread, packed two-wide FMAs (fma.rn.f32x2, each half an
// ordinary IEEE fused multiply-add), 16-byte shared-memory reads, and operands that arrive by 4-byte cp.async in a
// kStages-deep ring (no register staging; padding and ragged edges are zero-filled by the copy itself). 4-byte copies
// because nothing is known about alignment here: per k-slice they are 2 % of the instructions of a 128 x 128 tile.
//
// Shared memory holds a slice as [16 k][extent + 4 pad]: a copy whose 32 lanes are 32 consecutive i of one k, a copy whose
// lanes are 8 consecutive k of four i (operands with k contiguous in memory: 32-byte sectors; the pad puts the 8 rows 4
// banks apart) and the 16-byte reads of the inner loop are all free of bank conflicts.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cb_internal.h"

namespace cb {
namespace simt {

constexpr int kBK = 16;
constexpr int kStages = 4;

__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src, bool ok) {
    const int n = ok ? 4 : 0;  // 0: nothing is read, the word is zero-filled
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void lds16(uint32_t addr, uint64_t& a, uint64_t& b) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}

// Byte offset of element (k, e) of a slice with `EXT` columns.
template <int EXT>
__device__ __forceinline__ constexpr uint32_t slot(int k, int e) {
    return (uint32_t)(k * (EXT + 4) + e) * 4u;
}
template <int EXT>
constexpr uint32_t kOperandBytes = (uint32_t)(kBK * (EXT + 4) * 4);

// Which elements of a slice a thread copies. MN lanes: the 32 lanes of a warp are 32 consecutive i of one k, and a
// thread's i is the same in every copy. K lanes: 8 consecutive k of 4 consecutive i, and a thread's k is the same.
template <int EXT, int NW>
struct MnLanes {
    static constexpr int kCopies = EXT / 32 * kBK / NW;
    static_assert(NW % (EXT / 32) == 0, "a warp keeps its columns");
    static constexpr int kStep = NW / (EXT / 32);  // k between consecutive copies
    static __device__ __forceinline__ int e(int warp, int lane) { return (warp % (EXT / 32)) * 32 + lane; }
    static __device__ __forceinline__ int k(int warp, int r) { return warp / (EXT / 32) + r * kStep; }
};
template <int EXT, int NW>
struct KLanes {
    static constexpr int kCopies = EXT / 4 * 2 / NW;
    static constexpr int kStep = NW / 2 * 4;  // e between consecutive copies
    static __device__ __forceinline__ int k(int warp, int lane) { return (warp & 1) * 8 + (lane & 7); }
    static __device__ __forceinline__ int e(int warp, int lane, int r) { return (warp >> 1) * 4 + (lane >> 3) + r * kStep; }
};

// Shapes of a CTA tile: BM x BN outputs, warps of 8 x 4 threads, 8 x TN outputs per thread (64 x 4*TN per warp).
template <int BM_, int BN_, int TN_>
struct Tile {
    static constexpr int BM = BM_, BN = BN_, TN = TN_;
    static constexpr int WM = BM / 64, WN = BN / (4 * TN), NW = WM * WN, NT = 32 * NW;
    static constexpr int kMinCtas = TN == 8 ? 512 / (NT + (NT == 128 ? 42 : 0)) : 4;  // registers: 128 a thread, 168 for the 4-warp 8 x 8 tile
    static constexpr int kStageBytes = kOperandBytes<BM> + kOperandBytes<BN>;
    static constexpr int kSmem = kStages * kStageBytes;
};

// This thread's first row and column of the tile; it owns rows +0..3 and +32..35, columns +0..3 (and +16..19 with TN == 8).
// Neighbouring lanes (lane ^ 1) read the same rows and lanes two apart the same columns: a 16-byte shared-memory read in
// which such pairs share their address takes two wavefronts instead of four.
template <class T>
__device__ __forceinline__ int own_row() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    return (warp % T::WM) * 64 + ((lane >> 1) & 7) * 4;
}
template <class T>
__device__ __forceinline__ int own_col() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    return (warp / T::WM) * (4 * T::TN) + ((lane & 1) | ((lane >> 3) & 2)) * 4;
}

// Accumulators: for row pair x and column pair y, acc[y][x][0] holds (r0 c0, r1 c1) and acc[y][x][1] holds (r0 c1, r1 c0):
// the packed FMA then needs one swapped copy of each column pair where broadcasting the columns would need two.
template <class T>
using Acc = uint64_t[T::TN / 2][4][2];

// The main loop over `slices` k-slices of a CTA. `op.begin(t)` is called by every thread before the copies of slice t
// (a barrier lies between begin(t) and load(t)); op.load(t, base) issues this thread's copies of the slice.
template <class T, class Op>
__device__ __forceinline__ void main_loop(Op& op, int slices, uint32_t smem, Acc<T>& acc) {
    const uint32_t pi = slot<T::BM>(0, own_row<T>()), qi = kOperandBytes<T::BM> + slot<T::BN>(0, own_col<T>());
#pragma unroll
    for (int y = 0; y < T::TN / 2; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][x][0] = acc[y][x][1] = 0ull;
    op.begin(0);
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kStages - 1; ++t) {
        if (t < slices) op.load(t, smem + t * T::kStageBytes);
        cp_async_commit();
        op.begin(t + 1);
        __syncthreads();
    }
    for (int t = 0; t < slices; ++t) {
        cp_async_wait<kStages - 2>();
        __syncthreads();  // slice t is complete for every thread, and everybody is done with slice t - 1
        const int nt = t + kStages - 1;
        if (nt < slices) op.load(nt, smem + (nt % kStages) * T::kStageBytes);
        cp_async_commit();
        op.begin(nt + 1);
        const uint32_t stage = smem + (t % kStages) * T::kStageBytes;
        const uint32_t sp = stage + pi, sq = stage + qi;
#pragma unroll
        for (int k = 0; k < kBK; ++k) {
            uint64_t a[4], q[T::TN / 2];
            lds16(sp + slot<T::BM>(k, 0), a[0], a[1]);
            lds16(sp + slot<T::BM>(k, 32), a[2], a[3]);
            lds16(sq + slot<T::BN>(k, 0), q[0], q[1]);
            if (T::TN == 8) lds16(sq + slot<T::BN>(k, 16), q[T::TN / 2 - 2], q[T::TN / 2 - 1]);
#pragma unroll
            for (int y = 0; y < T::TN / 2; ++y) {
                float lo, hi;
                unpack2(q[y], lo, hi);
                const uint64_t swapped = pack2(hi, lo);
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    fma2(acc[y][x][0], a[x], q[y]);
                    fma2(acc[y][x][1], a[x], swapped);
                }
            }
        }
    }
    cp_async_wait<0>();
}

// Calls store(j, i, v) for this thread's 4-row pieces: v[x] is the value at row i + x of column j.
template <class T, class Store>
__device__ __forceinline__ void for_outputs(Acc<T>& acc, int i0, int j0, Store store) {
    const int ei = own_row<T>(), ej = own_col<T>();
#pragma unroll
    for (int y = 0; y < T::TN / 2; ++y)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float u[4], v[4];  // columns 2y and 2y + 1
            unpack2(acc[y][2 * h][0], u[0], v[1]);
            unpack2(acc[y][2 * h][1], v[0], u[1]);
            unpack2(acc[y][2 * h + 1][0], u[2], v[3]);
            unpack2(acc[y][2 * h + 1][1], v[2], u[3]);
            const int j = j0 + ej + (2 * y & 3) + (y >> 1) * 16;
            store(j, i0 + ei + 32 * h, u);
            store(j + 1, i0 + ei + 32 * h, v);
        }
}

// How many CTAs a product gets: extents, contraction length in slices, independent copies (batch matrices, phases), and
// whether the contraction may be split over CTAs (their sums then meet in memory through atomic adds).
struct Choice {
    int tile;    // index into the tile list of with_tile
    int splits;
    int per_split;  // slices of a split
};
// Tile list: 0: 128 x 128, 1: 128 x 64, 2: 128 x 32, 3: 64 x 64, 4: 64 x 32.
template <class F>
auto with_tile(int tile, F f) {
    switch (tile) {
        case 0: return f(Tile<128, 128, 8>{});
        case 1: return f(Tile<128, 64, 8>{});
        case 2: return f(Tile<128, 32, 4>{});
        case 3: return f(Tile<64, 64, 4>{});
        default: return f(Tile<64, 32, 4>{});
    }
}
// The cheapest pair of tile and split by a model in SM clocks. What a sweep of all pairs over 19 products and convolution
// passes showed: the 64 x 64 tile is best or within 2 % nearly everywhere, because four of its CTAs fit an SM and 16 warps
// hide the shared-memory and barrier latencies that 8 warps of the 128 x 128 tile do not; tiles with 32 columns pay for
// outputs that narrow; splitting pays down to about four slices a CTA as long as the atomic adds (three a clock and SM)
// stay small.
inline Choice search_tile(int sm_count, long long I, long long J, long long slices, long long copies, bool may_split) {
    static const int bm[5] = {128, 128, 128, 64, 64}, bn[5] = {128, 64, 32, 64, 32}, nw[5] = {8, 4, 4, 4, 2};
    static const int resident[5] = {2, 3, 4, 4, 8};                   // CTAs of the tile an SM holds
    static const double eff[5] = {1.0, 0.97, 0.85, 0.95, 0.75};       // rate of the inner loop with many warps
    static const int pieces[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512};
    Choice best{3, 1, (int)slices};
    double best_cost = 1e300;
    for (int c = 0; c < 5; ++c) {
        const long long tiles = (I + bm[c] - 1) / bm[c] * ((J + bn[c] - 1) / bn[c]) * copies;
        for (int want : pieces) {
            if (want > 1 && (!may_split || slices < 4LL * want || tiles * want > 64LL * sm_count)) break;
            const long long per = (slices + want - 1) / want;
            const long long splits = per > 0 ? (slices + per - 1) / per : 1;
            const long long q = (tiles * splits + sm_count - 1) / sm_count;
            const double warps = (double)(q < resident[c] ? q : resident[c]) * nw[c];
            double cost = (double)q * bm[c] * bn[c] * (double)per / 8.0 / (eff[c] * warps / (warps + 6.0));
            cost += (double)((q + resident[c] - 1) / resident[c]) * 2000.0;
            if (splits > 1) cost += (double)q * bm[c] * bn[c] / 3.0 + 2000.0;
            if (cost < best_cost) {
                best_cost = cost;
                best = Choice{c, (int)(splits < 1 ? 1 : splits), (int)per};
            }
        }
    }
    return best;
}

// The search costs microseconds, a visible share of a small call, and depends on these numbers only: a thread keeps the
// answers of the last shapes it saw.
inline Choice choose_tile(int sm_count, long long I, long long J, long long slices, long long copies, bool may_split) {
    struct Entry {
        long long I, J, slices, copies;
        int sm_count, may_split;
        Choice choice;
    };
    static thread_local Entry table[64];
    const unsigned long long h = (unsigned long long)I * 0x9E3779B97F4A7C15ull ^ (unsigned long long)J * 0xC2B2AE3D27D4EB4Full ^
                                 (unsigned long long)slices * 0x165667B19E3779F9ull ^ (unsigned long long)copies;
    Entry& e = table[(h >> 32) & 63];
    if (e.sm_count != sm_count || e.I != I || e.J != J || e.slices != slices || e.copies != copies || e.may_split != (int)may_split)
        e = Entry{I, J, slices, copies, sm_count, may_split ? 1 : 0, search_tile(sm_count, I, J, slices, copies, may_split)};
    return e.choice;
}

}  // namespace simt
}  // namespace cb
