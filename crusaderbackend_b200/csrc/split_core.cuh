// fp32 products on the tensor cores: D[i][j] = sum_k P(i, k) * Q(j, k) at the accuracy of fp32 FMAs, for CB_MATH_FP32 and for
// operands the TMA-fed kernels cannot address, where the product is large enough to pay for it. One kernel body serves the GEMM
// forms and the three convolution passes; an operand source (below) says where element (i, k) lies.
//
// Every fp32 value from 2^-110 on is the sum of three bf16 values: x = x1 + x2 + x3 with x1 = x cut off, x2 = x - x1 rounded, x3 the
// rest, all of it exact (8 + 8 + 8 significant bits; below, the third runs into bf16's least subnormal, 2^-133: see kLow). Six of the
// nine products of two such sums leave out up to 2^-22 of the product (x2 y3 + x3 y2, of either sign: x2 is rounded for that; 2^-26 on
// average): x2 y2, x1 y3, x3 y1, x1 y2, x2 y1, x1 y1, issued smallest first. (The splitting is that of G. Henry, P. T. P. Tang and A.
// Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", 2019.) What the tensor core
// does not give is fp32's rounding of sums (TMEM truncates every addition), so no chain of additions there is longer than two k-blocks
// of 32: their sum is read back and added to the running total in a register, by ordinary fp32 additions.
//
// What bounds it: shared-memory bandwidth, were both operands read from there (a 128 x 128 x 16 UMMA reads 8 KB in its 64 clocks;
// with the loaders' own accesses a k-block of 32 took 1800 clocks, 12 UMMAs 768). So the pieces of P go to TMEM, straight from the
// registers they are formed in, and only those of Q to shared memory. fp32 FMAs would need 4096 clocks.
//
// Roles: loader warps (global memory -> registers, a block ahead -> pieces: P's in TMEM, 48 columns a stage, Q's as three bf16 tiles
// of K-major rows of 64 bytes under the 64-byte swizzle) and summing warps, which own the output and of which the first issues
// the UMMAs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cb_internal.h"
#include "cb_ptx.cuh"

namespace cb {
namespace split {

constexpr int kBK = 32;             // k of a block
constexpr uint32_t kPieceRow = 64;  // bytes: 32 bf16
constexpr int kAcc = 2;             // accumulators in TMEM
constexpr int kStages = 4;
constexpr int kChunk = 2;           // k-blocks a sum in TMEM runs over
constexpr float kFinite = 3.402823466e38f, kWhole = 0x1p-110f, kLow = 0x1p-70f;  // see where the sums are checked
constexpr uint32_t kPCols = 48;     // TMEM columns of a stage of P: three pieces of 32 k, two a column

// What a loader does is a chain of latencies (fetch, three dependent steps of a split, store, fences): with eight loader warps an SM a
// block of 128 x 128 took 1780 clocks, 1550 of them the loaders'. With sixteen the CTA's registers no longer divide evenly, so the
// summing warps take some of theirs (setmaxnreg; the shares add up to what the CTA is launched with).
template <int BN_>
struct Shape {
    static constexpr int BM = 128, BN = BN_;
    static constexpr int kLoaders = BN == 32 ? 256 : 512;  // loader threads
    static constexpr int kSumWarps = BN == 32 ? 4 : 8;
    static constexpr int kCols = BN / (kSumWarps / 4);     // columns a summing thread holds
    static constexpr int NT = 32 * kSumWarps + kLoaders;
    static constexpr int kCtas = BN == 32 ? 2 : 1;         // an SM
    static constexpr int kSumRegs = 112, kLoaderRegs = 64; // of 80 at launch, where there are 768 threads
    static_assert(NT != 768 || 32 * kSumWarps * kSumRegs + kLoaders * kLoaderRegs <= 80 * NT, "setmaxnreg would wait for ever");
    static constexpr uint32_t kPieceQ = BN * kPieceRow, kStageBytes = 3 * kPieceQ;
    static constexpr uint32_t kTmemCols = BN == 32 ? 256 : 512;
    static constexpr int kSmem = kStages * (int)kStageBytes + 1024;
    static_assert(kAcc * BN + kStages * kPCols <= kTmemCols && kStages * (int)kStageBytes >= BN * 512, "");
};

// How the loader threads share an operand's block of 32 k. P: warp w takes kValues k (part w / 4) of the 32 rows of TMEM lane quarter
// w % 4, and must end up with one row a lane: at once where rows are contiguous in memory (MN), by way of a patch of shared memory
// of its own where k is (K: a load is these k of a few rows). Q: MN: 8 k of one row; K: two neighbouring k of several rows; KV (k on
// 16 bytes): 8 k of a row in two 16-byte loads.
enum Kind { MN, K, KV };
template <class S, Kind KIND>
struct ShareP {
    static_assert(KIND != KV, "");
    static constexpr int kValues = S::BM * kBK / S::kLoaders;
    static constexpr int kPatch = 32 * kValues;                      // words of a warp
    static constexpr int kPatches = KIND == K ? S::kLoaders / 32 * kPatch : 1;
    // row and k of value x
    static __device__ __forceinline__ int row(int tid, int x) {
        return 32 * ((tid >> 5) & 3) + (KIND == MN ? (tid & 31) : (tid & 31) / kValues + 32 / kValues * x);
    }
    static __device__ __forceinline__ int k(int tid, int x) { return kValues * (tid >> 7) + (KIND == MN ? x : tid % kValues); }
};
template <class S, Kind KIND>
struct ShareQ {
    static constexpr int ROWS = S::BN, kLoaders = S::kLoaders;
    static constexpr int kUnit = KIND == K ? 2 : 8;
    static constexpr int kUnits = KIND == K ? ROWS * 16 / kLoaders : (ROWS * 4 >= kLoaders ? ROWS * 4 / kLoaders : 1);  // a thread's
    static constexpr int kValues = kUnits * kUnit;
    static __device__ __forceinline__ bool active(int tid) { return KIND == K || ROWS * 4 >= kLoaders || tid < ROWS * 4; }
    static __device__ __forceinline__ int row(int tid, int u) {
        if (KIND == MN) return tid % ROWS;
        if (KIND == KV) return (tid >> 2) + kLoaders / 4 * u;
        return (tid >> 4) + kLoaders / 16 * u;
    }
    static __device__ __forceinline__ int k(int tid, int u) {  // first of the unit's k
        if (KIND == MN) return 8 * (tid / ROWS + u * (kLoaders / ROWS));
        if (KIND == KV) return 8 * (tid & 3);
        return 2 * (tid & 15);
    }
};

// Pairs of fp32 in one instruction each: the loaders and the summing warps are bound by issue slots.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {  // a - b, exact where it is used
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// (x0, x1) as three pairs of bf16, x0 in the low halves
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    const uint32_t a0 = __float_as_uint(x0), a1 = __float_as_uint(x1);
    const uint64_t r = sub2(pack2(x0, x1), pack2(__uint_as_float(a0 & 0xffff0000u), __uint_as_float(a1 & 0xffff0000u)));
    float r0, r1, c0, c1;
    unpack2(r, r0, r1);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(r1), "f"(r0));
    unpack2(sub2(r, pack2(__uint_as_float(p2 << 16), __uint_as_float(p2 & 0xffff0000u))), c0, c1);
    p1 = __byte_perm(a0, a1, 0x7632);
    p3 = __byte_perm(__float_as_uint(c0), __float_as_uint(c1), 0x7632);
}
// Address of 16-byte chunk q of a row of a piece: the 64-byte swizzle exchanges chunks by bits 1 and 2 of the row.
__device__ __forceinline__ uint32_t piece_chunk(uint32_t piece, int row, int q) {
    return piece + (uint32_t)row * kPieceRow + (uint32_t)((q ^ (row >> 1)) & 3) * 16u;
}
// Splits a thread's values of Q's block and stores the pieces. Free of bank conflicts in all three kinds: eight lanes with
// neighbouring rows and one chunk, or two rows and four chunks, cover 128 bytes.
template <class Sh, Kind KIND>
__device__ __forceinline__ void put_q(const float (&v)[ShareQ<Sh, KIND>::kValues], uint32_t pieces, int tid) {
    typedef ShareQ<Sh, KIND> S;
    constexpr uint32_t kPiece = Sh::kPieceQ;
    if (!S::active(tid)) return;
#pragma unroll
    for (int u = 0; u < S::kUnits; ++u) {
        const int row = S::row(tid, u), k = S::k(tid, u);
        const uint32_t dst = piece_chunk(pieces, row, k >> 3) + (uint32_t)(k & 7) * 2u;
        uint32_t p[3][4];
#pragma unroll
        for (int x = 0; x < S::kUnit; x += 2) split2(v[u * S::kUnit + x], v[u * S::kUnit + x + 1], p[0][x / 2], p[1][x / 2], p[2][x / 2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (KIND == K) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + i * kPiece), "r"(p[i][0]) : "memory");
            else asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + i * kPiece), "r"(p[i][0]), "r"(p[i][1]), "r"(p[i][2]), "r"(p[i][3]) : "memory");
        }
    }
}
// The same for P, into the TMEM columns of a stage (`at`: this warp's lanes and part).
template <class Sh, Kind KIND>
__device__ __forceinline__ void put_p(float (&v)[ShareP<Sh, KIND>::kValues], uint32_t at, uint32_t patch, int lane) {
    typedef ShareP<Sh, KIND> S;
    constexpr int V = S::kValues;
    if (KIND == K) {
        // [32 rows][V k], 16-byte chunks exchanged by row * V / 32: a store is 32 words in a row, eight lanes read eight chunks of
        // different banks (rows of V + 1 words read word by word: two conflicts a store, four times the loads)
        constexpr int kChunks = V / 4;
#pragma unroll
        for (int x = 0; x < V; ++x)  // row lane / V + 32 / V * x, k lane % V
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(patch + (uint32_t)(32 * x + (lane ^ (x % kChunks * 4))) * 4u), "f"(v[x]) : "memory");
        __syncwarp();
#pragma unroll
        for (int c = 0; c < kChunks; ++c)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[4 * c]), "=f"(v[4 * c + 1]), "=f"(v[4 * c + 2]), "=f"(v[4 * c + 3])
                         : "r"(patch + (uint32_t)(lane * V + 4 * (c ^ (lane * V / 32 % kChunks))) * 4u) : "memory");
        __syncwarp();
    }
    uint32_t p[3][V / 2];
#pragma unroll
    for (int x = 0; x < V; x += 2) split2(v[x], v[x + 1], p[0][x / 2], p[1][x / 2], p[2][x / 2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) tmem_st(at + 16u * i, p[i]);
    tmem_st_wait();
}

// base + n * stride in one instruction
__device__ __forceinline__ const float* step(const float* base, uint32_t stride_bytes, uint32_t n) {
    const float* r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(stride_bytes), "r"(n), "l"(base));
    return r;
}

// *src, or 0: one predicated load (a branch around each load cost more than the loads). Volatile: the compiler must not move it ahead of
// griddep_wait_then_launch, up to which the kernel before may still write what it reads.
__device__ __forceinline__ float load_if(const float* src, bool ok) {
    float v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}" : "=f"(v) : "l"(src), "r"((int)ok));
    return v;
}

// The loader threads alone (named barrier 1); all threads, from within their roles (2).
template <class S>
__device__ __forceinline__ void loader_sync() { asm volatile("bar.sync 1, %0;" ::"n"(S::kLoaders) : "memory"); }
template <class S>
__device__ __forceinline__ void all_sync() { asm volatile("bar.sync 2, %0;" ::"n"(S::NT) : "memory"); }

struct __align__(8) Barriers {
    uint64_t full[kStages], empty[kStages], tfull[kAcc], tempty[kAcc], drain;
    uint32_t tmem_base;
    int abort_flag;
    int again;    // the tile has outputs that fp32 FMAs have to form
    int cut;      // found on the way: factors below 2^-110; the largest factor's magnitude, as bits
    unsigned largest;
};

__device__ __forceinline__ float word(uint32_t at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
// Value of column c (of a summing thread's own) where it left its sums.
__device__ __forceinline__ float staged(uint32_t mine, int c) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(mine + (uint32_t)c * 512u));
    return v;
}

// *dst += y among other CTAs. The atomic add of memory takes subnormals, its own result too, for 0; LOW: an addition that keeps them, for
// outputs of the second pass.
template <bool LOW>
__device__ __forceinline__ void add_to(float* dst, float y) {
    if (!LOW) {
        atomicAdd(dst, y);
        return;
    }
    unsigned* word = reinterpret_cast<unsigned*>(dst);
    for (unsigned old = 0u, seen;; old = seen) {
        seen = atomicCAS(word, old, __float_as_uint(__uint_as_float(old) + y));
        if (seen == old) return;
    }
}

// The second pass over the contraction, by fp32 FMAs in k order, for the outputs of a tile that the pieces do not give. The loaders
// fetch the blocks once more and leave them as they are in shared memory, kSliceK at a time behind the sums: [k][128 rows],
// [k][BN columns]; the summing threads multiply. An infinity or a NaN in one operand makes whole rows of outputs need this, so it is a
// product like any other: 64 FMAs a thread and k at BN = 128, 4096 clocks a block as on the CUDA cores. us, finite values / a NaN in
// every output / the latter with one thread an output, whose every step waits for its loads: 256 x 256 x 8192 in one share
// 190 / 750 / 10190, 1000 x 777 x 1501 36 / 187 / 2330, weight gradient 16 -> 64 of 8 maps of 28 x 28 in one share 180 / 770 / 60300.
template <class S>
struct Again {
    static constexpr int kSliceK = S::BN / 4;
    static_assert(kBK % kSliceK == 0 && S::BN * 512 + kSliceK * (S::BM + S::BN) * 4 <= kStages * (int)S::kStageBytes, "");
    template <Kind KP, Kind KQ>
    static __device__ __forceinline__ void put(const float (&vp)[ShareP<S, KP>::kValues], const float (&vq)[ShareQ<S, KQ>::kValues], int first, uint32_t slice, int tid) {
        typedef ShareP<S, KP> P;
        typedef ShareQ<S, KQ> Q;
#pragma unroll
        for (int x = 0; x < P::kValues; ++x) {
            const int k = P::k(tid, x) - first;
            if ((unsigned)k < (unsigned)kSliceK)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(slice + (uint32_t)(k * S::BM + P::row(tid, x)) * 4u), "f"(vp[x]) : "memory");
        }
        if (!Q::active(tid)) return;
#pragma unroll
        for (int x = 0; x < Q::kValues; ++x) {
            const int k = Q::k(tid, x / Q::kUnit) + x % Q::kUnit - first;
            if ((unsigned)k < (unsigned)kSliceK)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(slice + (uint32_t)((kSliceK * S::BM + k * S::BN) + Q::row(tid, x / Q::kUnit)) * 4u), "f"(vq[x]) : "memory");
        }
    }
    // The summing threads': (row, first ...) are a thread's outputs, staged from `mine` on; wanted: whether its warp has some to form.
    static __device__ __noinline__ void sum(Barriers& b, int blocks, uint32_t slice, uint32_t mine, int row, int first, bool wanted) {
        float plain[S::kCols];
#pragma unroll
        for (int c = 0; c < S::kCols; ++c) plain[c] = 0.f;
        for (int s = 0; s < blocks * (kBK / kSliceK); ++s) {
            all_sync<S>();
            all_sync<S>();
            // whether the slice holds factors below kWhole, and its largest finite factor (what an infinity touches is not finite)
            unsigned largest = 0;
#pragma unroll 1
            for (int i = threadIdx.x; i < kSliceK * (S::BM + S::BN); i += 32 * S::kSumWarps) {
                const float v = fabsf(word(slice + (uint32_t)i * 4u));
                if (v > 0.f && v < kWhole) b.cut = 1;
                if (v <= kFinite) largest = max(largest, __float_as_uint(v));
            }
            largest = __reduce_max_sync(0xffffffffu, largest);
            if ((threadIdx.x & 31) == 0) atomicMax(&b.largest, largest);
            if (!wanted) continue;
            for (int k = 0; k < kSliceK; ++k) {
                const float p = word(slice + (uint32_t)(k * S::BM + row) * 4u);
#pragma unroll
                for (int c = 0; c < S::kCols; c += 4) {
                    float q0, q1, q2, q3;
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q0), "=f"(q1), "=f"(q2), "=f"(q3)
                                 : "r"(slice + (uint32_t)(kSliceK * S::BM + k * S::BN + first + c) * 4u) : "memory");
                    plain[c] = fmaf(p, q0, plain[c]);
                    plain[c + 1] = fmaf(p, q1, plain[c + 1]);
                    plain[c + 2] = fmaf(p, q2, plain[c + 2]);
                    plain[c + 3] = fmaf(p, q3, plain[c + 3]);
                }
            }
        }
        asm volatile("bar.sync 3, %0;" ::"n"(32 * S::kSumWarps) : "memory");  // the loaders are through with theirs
        if (!wanted) return;
        // magnitude from which on what was lost is less than 2^-24 of an output
        const float least = b.cut ? __uint_as_float(b.largest) * 0x1p-60f * (float)(blocks * kBK) * 0x1p-49f : 0.f;
#pragma unroll
        for (int c = 0; c < S::kCols; ++c) {
            const float v = fabsf(staged(mine, c));
            if (!(v <= kFinite) || v < least) asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + c * 512u), "f"(plain[c]) : "memory");
        }
    }
};

// The whole kernel behind its index arithmetic: `blocks` k-blocks of the tile through `src`.
// Source: kP, kQ (Kind); prepare(t, tid), when kTable: entry tid of the table that load() of block t and the kLoaders / 32 - 1 after it
// may read;
// load(t, tid, p, q): this thread's values of block t, asked for in ascending order from 0 on, at most twice over;
// store<LOW>(row, first, n, mine): outputs (row, first .. first + n - 1) of the tile, to be read by staged(), added by add_to<LOW>.
// patches: ShareP::kPatches floats of shared memory.
template <class S, class Src>
__device__ __forceinline__ void run(Src& src, int blocks, uint8_t* smem_raw, Barriers& b, float* patches, int* status) {
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t st_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    volatile int* abort_flag = &b.abort_flag;
    if (threadIdx.x == 0) {
        b.abort_flag = 0;
        b.again = b.cut = 0;
        b.largest = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&b.full[s]), S::kLoaders / 32);
            mbar_init(smem_u32(&b.empty[s]), 1);
        }
        for (int a = 0; a < kAcc; ++a) {
            mbar_init(smem_u32(&b.tfull[a]), 1);
            mbar_init(smem_u32(&b.tempty[a]), S::kSumWarps);
        }
        mbar_init(smem_u32(&b.drain), 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&b.tmem_base), S::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_wait_then_launch();
    const uint32_t tmem_base = b.tmem_base;
    const uint32_t slice = st_base + S::BN * 512u;  // of a second pass, behind the sums

    if (warp >= S::kSumWarps) {
        if (S::NT == 768) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::kLoaderRegs));
        const int tid = (int)threadIdx.x - 32 * S::kSumWarps;
        uint32_t s = 0, ph = 0;
        typedef ShareP<S, Src::kP> SP;
        typedef ShareQ<S, Src::kQ> SQ;
        const uint32_t lw = (uint32_t)(warp - S::kSumWarps);
        const uint32_t p_at = tmem_base + kAcc * S::BN + SP::kValues / 2u * (lw >> 2) + ((32u * (lw & 3u)) << 16);
        const uint32_t patch = smem_u32(patches) + lw * (SP::kPatch * 4u);
        auto store_block = [&](float (&vp)[SP::kValues], const float (&vq)[SQ::kValues]) {
            if (!mbar_wait_uniform(smem_u32(&b.empty[s]), ph ^ 1u, abort_flag, status, CBK_TIMEOUT_EMPTY)) return false;
            tc_fence_after();
            put_q<S, Src::kQ>(vq, st_base + s * S::kStageBytes, tid);
            put_p<S, Src::kP>(vp, p_at + s * kPCols, patch, lane);
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&b.full[s]));
            if (++s == kStages) { s = 0; ph ^= 1u; }
            return true;
        };
        // A table of the source serves kLoaders / 32 blocks, an entry a loader: its divisions would take longer than a block. A loader
        // that gave up keeps to the barriers, so that none of the others waits there for it.
        bool ok = true;
        auto fetch = [&](int t, float (&vp)[SP::kValues], float (&vq)[SQ::kValues]) {
            if (t >= blocks) return;
            if (Src::kTable && t % (S::kLoaders / kBK) == 0) {
                if (t) loader_sync<S>();
                src.prepare(t, tid);
                loader_sync<S>();
            }
            src.load(t, tid, vp, vq);
        };
        float p[2][SP::kValues], q[2][SQ::kValues];
        fetch(0, p[0], q[0]);
        for (int t = 0; t < blocks; t += 2) {
            fetch(t + 1, p[1], q[1]);
            ok = ok && store_block(p[0], q[0]);
            fetch(t + 2, p[0], q[0]);
            if (t + 1 < blocks) ok = ok && store_block(p[1], q[1]);
        }
        all_sync<S>();
        if (b.again && !b.abort_flag) {
            for (int t = 0; t < blocks; ++t) {
                fetch(t, p[0], q[0]);
                for (int k = 0; k < kBK; k += Again<S>::kSliceK) {
                    all_sync<S>();  // the slice before this one has been read
                    Again<S>::template put<Src::kP, Src::kQ>(p[0], q[0], k, slice, tid);
                    all_sync<S>();
                }
            }
        }
    } else {
        if (S::NT == 768) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::kSumRegs));
        const int quarter = warp & 3, first = (warp >> 2) * S::kCols;
        uint64_t sum[S::kCols / 2];
#pragma unroll
        for (int c = 0; c < S::kCols / 2; ++c) sum[c] = 0ull;
        // Warp 0 issues too: chunk c + 1 before it adds chunk c, whose successor's UMMAs then run behind its additions.
        uint32_t s = 0, ph = 0;
        const int chunks = (blocks + kChunk - 1) / kChunk;
        auto issue = [&](int c) {
            const uint32_t a = (uint32_t)c % kAcc;
            if (!mbar_wait_uniform(smem_u32(&b.tempty[a]), (((uint32_t)c / kAcc) & 1u) ^ 1u, abort_flag, status, CBK_TIMEOUT_TMEM_EMPTY)) return false;
            const uint32_t d = tmem_base + a * S::BN, idesc = umma_idesc_bf16(128, (uint32_t)S::BN);
            const int n = min(kChunk, blocks - c * kChunk);
            for (int leading = 0; leading < 2; ++leading) {  // x1 y1 of the whole chunk comes last
                uint32_t at = s;
                for (int t = 0; t < n; ++t) {
                    if (!leading && !mbar_wait_uniform(smem_u32(&b.full[at]), ph ^ (at < s ? 1u : 0u), abort_flag, status, CBK_TIMEOUT_FULL)) return false;
                    tc_fence_after();
                    const uint64_t dq = umma_smem_desc(st_base + at * S::kStageBytes, 16u, 512u, UMMA_SW_64B);
                    const uint32_t dp = tmem_base + kAcc * S::BN + at * kPCols;
                    // 16 k each: 8 columns, 32 bytes apart
                    if (leading) {
                        umma_bf16_ts_elect(d, dp, dq, idesc, 1u);
                        umma_bf16_ts_elect(d, dp + 8u, dq + 2u, idesc, 1u);
                        tc_commit_elect(smem_u32(&b.empty[at]));
                    } else {
                        constexpr int pp[5] = {1, 0, 2, 0, 1}, qq[5] = {1, 2, 0, 1, 0};
#pragma unroll
                        for (int x = 0; x < 5; ++x)
#pragma unroll
                            for (uint32_t ks = 0; ks < 2; ++ks)
                                umma_bf16_ts_elect(d, dp + 16u * pp[x] + 8u * ks, dq + (uint64_t)((qq[x] * S::kPieceQ >> 4) + 2 * ks), idesc, t + x + ks ? 1u : 0u);
                    }
                    if (++at == kStages) at = 0;
                }
                if (leading) {
                    if (at < s) ph ^= 1u;
                    s = at;
                }
            }
            tc_commit_elect(smem_u32(&b.tfull[a]));
            return true;
        };
        bool ok = warp != 0 || issue(0);
        for (int c = 0; c < chunks && ok; ++c) {
            if (warp == 0 && c + 1 < chunks && !issue(c + 1)) { ok = false; break; }
            const uint32_t a = (uint32_t)c % kAcc;
            ok = mbar_wait_uniform(smem_u32(&b.tfull[a]), ((uint32_t)c / kAcc) & 1u, abort_flag, status, CBK_TIMEOUT_TMEM_FULL);
            if (!ok) break;
            tc_fence_after();
            const uint32_t at = tmem_base + a * S::BN + (uint32_t)first + ((uint32_t)(32 * quarter) << 16);
#pragma unroll
            for (int col = 0; col < S::kCols; col += 32) {
                uint32_t v[32];
                tmem_ld32(at + (uint32_t)col, v);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; e += 2)
                    sum[(col + e) / 2] = add2(sum[(col + e) / 2], pack2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&b.tempty[a]));
        }
        // Every UMMA has read its operands: the stages take the sums, so that what follows is a loop (unrolled over registers, its
        // branches took longer to fetch than a small product to compute).
        // Outputs that are formed again. A value that has no pieces (an infinity, a NaN) or a sum that left the range on the way shows as a
        // result that is not finite. A factor below kWhole loses up to 2^-133, what lies under bf16's least subnormal, so outputs are off by
        // up to K 2^-133 times the largest factor. Asking every factor cost the loaders 1 to 4 % of a launch; so an output below kLow
        // (but not 0) brings the second pass, which looks at the factors. Outputs above it may be off by more than 2^-24 of
        // themselves only where K times the largest factor exceeds 2^39.
        const int row = 32 * quarter + lane;
        const uint32_t mine = st_base + (uint32_t)(first * 128 + row) * 4u;
        uint64_t zeros = 0;
        unsigned smallest = 0xffffffffu;
        if (ok) {
#pragma unroll
            for (int c = 0; c < S::kCols; c += 2) {
                float lo, hi;
                unpack2(sum[c / 2], lo, hi);
                // a product with 0 is a NaN for what is not finite; the bits without their sign, less one, put 0 above everything
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(zeros) : "l"(sum[c / 2]), "l"(0ull));
                smallest = min(smallest, min(2u * __float_as_uint(lo) - 1u, 2u * __float_as_uint(hi) - 1u));
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + c * 512u), "f"(lo) : "memory");
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + c * 512u + 512u), "f"(hi) : "memory");
            }
        }
        const bool wanted = __any_sync(0xffffffffu, (zeros & 0x7fffffff7fffffffull) != 0 || smallest < 2u * __float_as_uint(kLow) - 1u);
        if (wanted) b.again = 1;
        else if (ok) src.template store<false>(row, first, S::kCols, mine);
        all_sync<S>();
        if (b.again && !b.abort_flag) {
            Again<S>::sum(b, blocks, slice, mine, row, first, wanted);
            if (wanted) src.template store<true>(row, first, S::kCols, mine);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (b.abort_flag) {  // issued UMMAs may still run: a bounded chance to finish before TMEM and shared memory go
            tc_commit_elect(smem_u32(&b.drain));
            if (lane == 0) mbar_drain(smem_u32(&b.drain), 0, status);
            __syncwarp();
        }
        tc_fence_after();
        tmem_dealloc(tmem_base, S::kTmemCols);
    }
}

// A summing thread's n outputs into memory `step` floats apart. plain: stored, or (add) added to what is there, one atomic add being
// a read, an addition and a write without the wait for the read. Otherwise value(c, y, old place) is what is stored, or added.
template <bool LOW, class F>
__device__ __forceinline__ void store_columns(float* dst, long long step, int n, uint32_t mine, bool plain, bool add, F value) {
    if (plain) {  // without a branch in the loop: reads of several columns are in flight together
        if (add)
#pragma unroll 8
            for (int c = 0; c < n; ++c, dst += step) add_to<LOW>(dst, staged(mine, c));
        else
#pragma unroll 8
            for (int c = 0; c < n; ++c, dst += step) *dst = staged(mine, c);
        return;
    }
#pragma unroll 4
    for (int c = 0; c < n; ++c, dst += step) {
        const float y = value(c, staged(mine, c), dst);
        if (add) add_to<LOW>(dst, y);
        else *dst = y;
    }
}

// Whether a product comes here rather than to the CUDA cores. Contractions of less than 16: the rounding of a few fp32 FMAs is less
// than what the six products leave out (2-norm error at K = 2: 1.8e-8 .. 3.4e-8 against 2.1e-8 .. 5.7e-8; at K = 16 7.5e-8 against
// 5.4e-8, at 1501 3.5e-7 against 1.1e-7). Small products: bound by their launch on either path. Whether the contraction may be shared
// does not matter: with one share on each side (deterministic contexts, a ReLU, models) this kernel takes less in all of 57
// products from 64 x 64 x 4096 (90 us against 151) to 20000 x 32 x 64 (11.1 and 12.2) and in 43 convolution passes (1.75 to 2.9 times).
inline bool worth_it(long long I, long long J, long long K, long long copies, long long least_fmas) {
    return K >= 16 && (double)I * (double)J * (double)K * (double)copies >= (double)least_fmas;
}

// What a tile costs, in SM clocks of a model: a round of CTAs; a block of 128, 64 and 32 columns; how much longer two CTAs of 32 columns
// on an SM take; values an SM adds into memory a clock; the launch that clears the output before. Fitted to sweeps of all tiles and shares.
struct Costs {
    double round, block[3], pair, flush, clear;
};
// 515 products (17 to 4600 rows and columns, K 64 to 5500, all forms): what it takes is 0.8 % from the best on average, 13 % at most. A fit
// to 25 larger ones gave outputs of few columns too few shares: 6 % on average, 59 % at most, 16 products slower than on the CUDA cores,
// where now none is. 2048 x 32 x 512: 10.9 us, 8.9 on the CUDA cores, 8.5 now; 4096 x 20 x 512 16.6, 13.3, 10.6.
constexpr Costs kMatrix{2880.0, {710.0, 665.0, 610.0}, 1.29, 11.8, 1120.0};
// 48 convolution passes; over 178 others the gathers are 1.6 % from the best on average, 24 % at most, the weight gradient 0.7 and 14 %.
constexpr Costs kGather{2300.0, {690.0 * 1.9, 630.0 * 1.9, 440.0 * 1.9}, 1.77, 3.94, 1030.0}, kWgrad{2300.0, {690.0 * 2.5, 630.0 * 2.5, 440.0 * 2.5}, 1.77, 3.94, 1030.0};

// Columns of the CTA tile and how many CTAs share the contraction (their sums then meet in memory through atomic adds): the cheapest.
struct Choice {
    int bn, splits, per_split;
};
inline Choice choose_shape(int sm_count, long long I, long long J, long long blocks, long long copies, bool may_split, const Costs& costs) {
    static const int bns[3] = {128, 64, 32};
    static const int pieces[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128};
    Choice best{64, 1, (int)blocks};
    double best_cost = 1e300;
    for (int b = 0; b < 3; ++b) {
        const int bn = bns[b];
        const long long tiles = (I + 127) / 128 * ((J + bn - 1) / bn) * copies;
        for (int want : pieces) {
            if (want > 1 && (!may_split || blocks < 2LL * want || tiles * want > 16LL * sm_count)) break;
            const long long per = (blocks + want - 1) / want, splits = (blocks + per - 1) / per, ctas = tiles * splits;
            const bool pairs = bn == 32 && ctas > sm_count;
            const long long slots = pairs ? 2LL * sm_count : sm_count;
            const double load = pairs ? costs.pair : 1.0, rounds = (double)((ctas + slots - 1) / slots);
            double cost = rounds * (costs.round + (double)per * costs.block[b] * load);
            if (splits > 1) cost += rounds * 128.0 * bn / costs.flush * load + costs.clear;
            if (cost < best_cost) {
                best_cost = cost;
                best = Choice{bn, (int)splits, (int)per};
            }
        }
    }
    return best;
}

}  // namespace split
}  // namespace cb
