// CUDA-core fp32 GEMM: CB_MATH_FP32 and operand pairs TMA cannot address, as far as gemm_split.cu does not take them, on the shared
// main loop of simt_core.cuh; kernels for thin products and short contractions.
#include <utility>

#include "cb_ptx.cuh"
#include "simt_core.cuh"

namespace cb {
namespace {

using simt::kBK;

struct SimtParams {
    int I, J, K, batch;
    const float* P; long long ldp, strideP;
    const float* Q; long long ldq, strideQ;
    int p_mn, q_mn;
    float* C; long long ldc, strideC; int out_mode, accumulate, atomic_out;
    const float* bias_i; const float* bias_j; int relu;
    int splits, k_per_split;  // k_per_split counts k-slices of 16 (simt_gemm_kernel) or k (thin_gemm_*)
    int slices;               // k-slices of the whole contraction
    int per_fold;             // k-slices of one operand pair (batch folded into the contraction), else = slices
    float* thin_sum;          // thin_gemm_mn_kernel: += sum over k of the thin operand, I values (null = none)
};

// Copies of one operand: element (e, k) at base + e * ld + k (K-major) or base + k * ld + e (MN-major). A slice that lies
// inside the matrix (`inside`, the same for the whole CTA) needs no tests: pointer and one constant step.
template <bool MN, int EXT, int NW>
__device__ __forceinline__ void load_operand(uint32_t dst, const float* base, long long ld, int e0, int E, int k0, int K) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    typedef simt::MnLanes<EXT, NW> M;
    typedef simt::KLanes<EXT, NW> L;
    constexpr int kCopies = MN ? M::kCopies : L::kCopies;
    const int e = MN ? M::e(warp, lane) : L::e(warp, lane, 0), k = MN ? M::k(warp, 0) : L::k(warp, lane);
    constexpr int kStepE = MN ? 0 : L::kStep, kStepK = MN ? M::kStep : 0;  // between a thread's consecutive copies
    const float* src = base + (MN ? (long long)(k0 + k) * ld + e0 + e : (long long)(e0 + e) * ld + k0 + k);
    const long long step = (long long)(MN ? kStepK : kStepE) * ld;
    dst += simt::slot<EXT>(k, e);
    if (e0 + EXT <= E && k0 + kBK <= K) {
#pragma unroll
        for (int r = 0; r < kCopies; ++r, src += step) simt::cp_async4(dst + simt::slot<EXT>(r * kStepK, r * kStepE), src, true);
    } else {
#pragma unroll
        for (int r = 0; r < kCopies; ++r, src += step) {
            const bool ok = e0 + e + r * kStepE < E && k0 + k + r * kStepK < K;
            simt::cp_async4(dst + simt::slot<EXT>(r * kStepK, r * kStepE), ok ? src : base, ok);
        }
    }
}

template <class T, bool P_MN, bool Q_MN>
struct GemmSource {
    const SimtParams& p;
    int b, i0, j0, slice0;
    __device__ __forceinline__ void begin(int) {}
    __device__ __forceinline__ void load(int t, uint32_t dst) {
        int s = slice0 + t, pair = b;
        if (p.per_fold != p.slices) {
            pair = s / p.per_fold;
            s -= pair * p.per_fold;
        }
        load_operand<P_MN, T::BM, T::NW>(dst, p.P + pair * p.strideP, p.ldp, i0, p.I, s * kBK, p.K);
        load_operand<Q_MN, T::BN, T::NW>(dst + simt::kOperandBytes<T::BM>, p.Q + pair * p.strideQ, p.ldq, j0, p.J, s * kBK, p.K);
    }
};

// 1000 x 777 x 1501 NN: 267 us with the 64 x 64 tile of scalar loads and 4 x 4 outputs this replaces (8.7 TFLOP/s).
template <class T, bool P_MN, bool Q_MN>
__global__ void __launch_bounds__(T::NT, T::kMinCtas) simt_gemm_kernel(const SimtParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    griddep_wait_then_launch();
    const int b = blockIdx.z / p.splits, split = blockIdx.z - b * p.splits;
    const int i0 = blockIdx.x * T::BM, j0 = blockIdx.y * T::BN;
    GemmSource<T, P_MN, Q_MN> src{p, b, i0, j0, split * p.k_per_split};
    simt::Acc<T> acc;
    simt::main_loop<T>(src, min(p.k_per_split, p.slices - src.slice0), (uint32_t)__cvta_generic_to_shared(smem), acc);
    float* Cb = p.C + (long long)b * p.strideC;
    simt::for_outputs<T>(acc, i0, j0, [&](int j, int i, float (&v)[4]) {
        if (j >= p.J) return;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (i + x >= p.I) return;
            float y = v[x];
            if (split == 0) {
                if (p.bias_i) y += p.bias_i[i + x];
                if (p.bias_j) y += p.bias_j[j];
            }
            float* dst = p.out_mode == 0 ? Cb + (long long)j * p.ldc + i + x : Cb + (long long)(i + x) * p.ldc + j;
            if (p.atomic_out) {
                atomicAdd(dst, y);
            } else {
                if (p.accumulate) y += *dst;
                if (p.relu) y = fmaxf(y, 0.f);
                *dst = y;
            }
        }
    });
}

// Thin products (I <= 16, classifier layers and single samples): bound by reading the wide operand once, so the thin one
// is staged in shared memory, the contraction is split over enough CTAs to have the whole GPU loading, and the partial
// sums meet in C through atomics (or stay in one CTA on deterministic contexts). IT: I rounded up to 4, 8 or 16.
constexpr int kThinK = 256;  // k of a staged piece

template <int IT>
__device__ __forceinline__ void stage_thin(float (&sP)[IT][kThinK], const SimtParams& p, int k0, int k1) {
    for (int e = threadIdx.x; e < IT * kThinK; e += 256) {
        // consecutive threads along whichever index is contiguous in memory
        const int i = p.p_mn ? e % IT : e / kThinK, kk = p.p_mn ? e / IT : e % kThinK;
        const int k = k0 + kk;
        sP[i][kk] = (i < p.I && k < k1) ? (p.p_mn ? p.P[(long long)k * p.ldp + i] : p.P[(long long)i * p.ldp + k]) : 0.f;
    }
}
// A pointer for loads that must stay behind griddep_wait_then_launch: made behind that call, it depends on an assembly statement that the
// compiler keeps there. (Volatile loads, in an order of their own: a dense layer's three launches 13.54 -> 13.65 us.)
struct BehindWait {
    const float* p;
    explicit __device__ __forceinline__ BehindWait(const float* q) : p(q) { asm volatile("" : "+l"(p)); }
};
// src.p[at], or 0: one predicated load.
__device__ __forceinline__ float load_or_zero(BehindWait src, long long at, bool ok) {
    float v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}" : "=f"(v) : "l"(src.p + at), "r"((int)ok));
    return v;
}
__device__ __forceinline__ float* place_thin(const SimtParams& p, int i, int j) {
    return p.out_mode == 0 ? p.C + (long long)j * p.ldc + i : p.C + (long long)i * p.ldc + j;
}
__device__ __forceinline__ void store_thin(const SimtParams& p, int i, int j, float v, bool first, float old) {
    if (i >= p.I || j >= p.J) return;
    if (first) {
        if (p.bias_i) v += p.bias_i[i];
        if (p.bias_j) v += p.bias_j[j];
    }
    float* dst = place_thin(p, i, j);
    if (p.atomic_out) {
        atomicAdd(dst, v);
    } else {
        if (p.accumulate) v += old;
        if (p.relu) v = fmaxf(v, 0.f);
        *dst = v;
    }
}
__device__ __forceinline__ void store_thin(const SimtParams& p, int i, int j, float v, bool first) {
    store_thin(p, i, j, v, first, p.accumulate && !p.atomic_out && i < p.I && j < p.J ? *place_thin(p, i, j) : 0.f);
}

// Sums of NV values over a warp's lanes by one butterfly: after the step with offset o a lane keeps the half of its values that its bit o
// selects. Returns which it is left with, in acc[0 ..].
template <int NV>
__device__ __forceinline__ int butterfly(float (&acc)[NV], int lane) {
    int base = 0, n = NV;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int v = 0; v < NV / 2; ++v)
                if (v < n) {
                    const float give = up ? acc[v] : acc[v + n], keep = up ? acc[v + n] : acc[v];
                    acc[v] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            base += up ? n : 0;
        } else {
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
        }
    }
    return base;
}

// Wide operand with k contiguous: lanes walk k, a warp holds 4 rows of it against all IT thin ones, and one butterfly
// that halves the accumulators at every step replaces a full reduction of each.
template <int IT>
__global__ void __launch_bounds__(256) thin_gemm_k_kernel(const SimtParams p) {
    __shared__ float sP[IT][kThinK];
    constexpr int NV = 4 * IT;
    griddep_wait_then_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j0 = blockIdx.x * 32 + warp * 4;
    const int k_begin = blockIdx.y * p.k_per_split, k_end = min(p.K, k_begin + p.k_per_split);
    float acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.f;
    const float* row[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) row[r] = p.Q + (long long)min(j0 + r, p.J - 1) * p.ldq;
    for (int k0 = k_begin; k0 < k_end; k0 += kThinK) {
        stage_thin<IT>(sP, p, k0, k_end);
        __syncthreads();
#pragma unroll 2
        for (int kk = lane; kk < kThinK; kk += 32) {
            float q[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) q[r] = k0 + kk < k_end ? row[r][k0 + kk] : 0.f;
#pragma unroll
            for (int i = 0; i < IT; ++i) {
                const float a = sP[i][kk];
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[i * 4 + r] = fmaf(a, q[r], acc[i * 4 + r]);
            }
        }
        __syncthreads();
    }
    const int base = butterfly<NV>(acc, lane);
    constexpr int kLeft = NV > 32 ? NV / 32 : 1;   // values a lane is left with
    if (NV < 32 && (lane & (32 / NV - 1)) != 0) return;  // the last steps left equal values in several lanes
#pragma unroll
    for (int v = 0; v < kLeft; ++v) store_thin(p, (base + v) >> 2, j0 + ((base + v) & 3), acc[v], blockIdx.y == 0);
}

// Both operands with k contiguous, few enough rows j that the launch is a chain of latencies (a classifier's forward pass): a block holds
// kThinRows rows against all IT thin ones and a share of k, every warp 128 k of it at a time, all of a step's loads in flight together, the
// thin operand's straight from the cache. The shares of a contraction are the blocks of a cluster, which add up through their shared memory: no
// cleared output, no atomics, reproducible. 128 x 10 x 4096, bias: 6.7 us as shares added by atomics on the tensor cores (TF32,
// clear launch included), 5.4 here.
constexpr int kThinRows = 4, kThinStep = 8 * 128;  // k a block's warps take at a time
template <int IT, bool V>
__global__ void __launch_bounds__(256) thin_rows_kernel(const SimtParams p) {
    constexpr int NV = kThinRows * IT, kLeft = NV > 32 ? NV / 32 : 1;  // values; those a lane is left with
    __shared__ float part[8][NV];
    __shared__ __align__(16) float whole[NV];
    griddep_wait_then_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = blockIdx.x % p.splits, j0 = (int)(blockIdx.x / p.splits) * kThinRows;
    const int k_begin = rank * p.k_per_split, k_end = min(p.K, k_begin + p.k_per_split);
    float acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.f;
    const float* row[kThinRows];
#pragma unroll
    for (int r = 0; r < kThinRows; ++r) row[r] = p.Q + (long long)min(j0 + r, p.J - 1) * p.ldq;
    for (int k0 = k_begin + warp * 128; k0 < k_end; k0 += kThinStep) {
        float q[kThinRows][4];
        if (V) {
            const int k = k0 + 4 * lane;
            const bool in = k < k_end;  // shares and K are whole float4s
#pragma unroll
            for (int r = 0; r < kThinRows; ++r)
                *reinterpret_cast<float4*>(q[r]) = in ? __ldg(reinterpret_cast<const float4*>(row[r] + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
            float4 a[IT];  // all of them before the first is used (with a test between one row and the next a launch took 0.16 us a row)
#pragma unroll
            for (int i = 0; i < IT; ++i)
                a[i] = in && i < p.I ? __ldg(reinterpret_cast<const float4*>(p.P + (long long)i * p.ldp + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < IT; ++i)
#pragma unroll
                for (int r = 0; r < kThinRows; ++r)
                    acc[i * kThinRows + r] = fmaf(a[i].w, q[r][3], fmaf(a[i].z, q[r][2], fmaf(a[i].y, q[r][1], fmaf(a[i].x, q[r][0], acc[i * kThinRows + r]))));
        } else {
#pragma unroll
            for (int r = 0; r < kThinRows; ++r)
#pragma unroll
                for (int e = 0; e < 4; ++e) q[r][e] = k0 + lane + 32 * e < k_end ? __ldg(row[r] + k0 + lane + 32 * e) : 0.f;
            float a[IT][4];
#pragma unroll
            for (int i = 0; i < IT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) a[i][e] = i < p.I && k0 + lane + 32 * e < k_end ? __ldg(p.P + (long long)i * p.ldp + k0 + lane + 32 * e) : 0.f;
#pragma unroll
            for (int i = 0; i < IT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int r = 0; r < kThinRows; ++r) acc[i * kThinRows + r] = fmaf(a[i][e], q[r][e], acc[i * kThinRows + r]);
        }
    }
    const int base = butterfly<NV>(acc, lane);
    if (NV >= 32 || (lane & (32 / NV - 1)) == 0)
#pragma unroll
        for (int v = 0; v < kLeft; ++v) part[warp][base + v] = acc[v];
    __syncthreads();
    float sum = 0.f;
    if (threadIdx.x < NV) {
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += part[w][threadIdx.x];
        whole[threadIdx.x] = sum;
    }
    if (p.splits > 1) {
        cluster_sync();
        if (rank == 0 && threadIdx.x < p.I) {
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(whole + 4 * threadIdx.x);
            float4 t = ld_cluster_f4(at, 0);
            for (int r = 1; r < p.splits; ++r) {
                const float4 u = ld_cluster_f4(at, (uint32_t)r);
                t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
            }
            const float y[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int r = 0; r < kThinRows; ++r) store_thin(p, (int)threadIdx.x, j0 + r, y[r], true);
        }
        cluster_sync();  // nobody's shared memory goes away while it is read
        return;
    }
    if (threadIdx.x < NV) store_thin(p, (int)threadIdx.x / kThinRows, j0 + (int)threadIdx.x % kThinRows, sum, true);
}

// Wide operand with j contiguous: lanes are 32 consecutive j, the eight warps take every eighth k of the piece, and the
// thin values are shared-memory broadcasts, four a load. Latency bound where a piece is all there is (parameter gradients of a classifier): a
// warp's first sixteen loads, the thin operand's and what is added to are on their way together. The sum of the thin operand over k (the
// bias gradient of that layer) comes from what the first block has staged; as a kernel of its own it took 7 us, of one block that waits
// for this one. 4096 -> 10, batch 128, weights and bias: 15.6 -> 5.7 us with that; 3.6 with four values a load, the old outputs read ahead
// and the sum shared by all threads without bank conflicts.
template <int IT>
__global__ void __launch_bounds__(256) thin_gemm_mn_kernel(const SimtParams p) {
    constexpr int kOuts = (IT + 7) / 8;  // thin rows a warp stores
    __shared__ __align__(16) float sP[kThinK][IT];
    __shared__ float part[IT][8][32];
    __shared__ float sums[8][IT];
    griddep_wait_then_launch();
    const BehindWait thin(p.P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane;
    const int k_begin = blockIdx.y * p.k_per_split, k_end = min(p.K, k_begin + p.k_per_split);
    float acc[IT], old[kOuts], sum = 0.f;  // old: what this thread's outputs are added to; sum: of a thin row's share
#pragma unroll
    for (int i = 0; i < IT; ++i) acc[i] = 0.f;
#pragma unroll
    for (int r = 0; r < kOuts; ++r) {
        const int i = warp + 8 * r;
        old[r] = p.accumulate && !p.atomic_out && i < p.I && j < p.J ? *place_thin(p, i, j) : 0.f;
    }
    const float* col = p.Q + min(j, p.J - 1);
    const bool summing = p.thin_sum != nullptr && blockIdx.x == 0;
    auto add = [&](int kk, float q) {
#pragma unroll
        for (int i = 0; i < IT; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(&sP[kk][i]);
            acc[i] = fmaf(a.x, q, acc[i]);
            acc[i + 1] = fmaf(a.y, q, acc[i + 1]);
            acc[i + 2] = fmaf(a.z, q, acc[i + 2]);
            acc[i + 3] = fmaf(a.w, q, acc[i + 3]);
        }
    };
    for (int k0 = k_begin; k0 < k_end; k0 += kThinK) {
        constexpr int kAhead = 16;
        const int n = min(kThinK, k_end - k0);
        float q[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) q[u] = warp + 8 * u < n ? col[(long long)(k0 + warp + 8 * u) * p.ldq] : 0.f;
        // consecutive threads along whichever index is contiguous in memory; values past the end are 0
        if (p.p_mn) {
            const int i = threadIdx.x % IT;
#pragma unroll
            for (int kk = threadIdx.x / IT, u = 0; u < IT; ++u, kk += 256 / IT) sP[kk][i] = load_or_zero(thin, (long long)(k0 + kk) * p.ldp + i, i < p.I && kk < n);
        } else {
#pragma unroll
            for (int i = 0; i < IT; ++i) sP[threadIdx.x][i] = load_or_zero(thin, (long long)i * p.ldp + k0 + threadIdx.x, i < p.I && (int)threadIdx.x < n);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (warp + 8 * u < n) add(warp + 8 * u, q[u]);
#pragma unroll 8
        for (int kk = warp + 8 * kAhead; kk < n; kk += 8) add(kk, col[(long long)(k0 + kk) * p.ldq]);
        if (summing)
            for (int kk = threadIdx.x / IT; kk < n; kk += 256 / IT) sum += sP[kk][threadIdx.x % IT];
        __syncthreads();
    }
    if (summing) {
#pragma unroll
        for (int o = 16; o >= IT; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane < IT) sums[warp][lane] = sum;
    }
#pragma unroll
    for (int i = 0; i < IT; ++i) part[i][warp][lane] = acc[i];
    __syncthreads();
    if (summing && threadIdx.x < p.I) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += sums[w][threadIdx.x];
        atomicAdd(p.thin_sum + threadIdx.x, v);  // one share, or one of each split
    }
#pragma unroll
    for (int r = 0; r < kOuts; ++r) {
        const int i = warp + 8 * r;
        if (i >= IT) break;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += part[i][w][lane];
        store_thin(p, i, j, v, blockIdx.y == 0, old[r]);
    }
}

// Short contractions (K <= KT, the input gradient of a classifier layer): bound by writing the output. A thread keeps the K values of
// four columns of P in registers and forms kShortRows rows of the output, whose Q values are shared-memory broadcasts; products are
// added in k order by FMAs, as everywhere here. us, 64 x 64 tiles (one slice of 16 k) / here: 128 x 4096 x 10 6.8 / 2.9, x 15 6.8 / 3.9.
constexpr int kShortRows = 2, kShortGroups = 8;  // rows a thread, rows of threads
// Whether it reads and writes 16 bytes at a time.
template <class T>
bool short_vec(const T& p) {
    return ((p.I | p.ldp | p.strideP | p.ldc | p.strideC) & 3) == 0 && ((reinterpret_cast<uintptr_t>(p.P) | reinterpret_cast<uintptr_t>(p.C)) & 15u) == 0;
}
// Which products it takes: every sixteen rows read P's columns again, so where there are many the tiles are faster. us, tiles / here: K
// = 10 on 16 bytes 2000 x 4096 28.1 / 14.8, off them 1000 x 4095 16.9 / 16.9, 8000 x 4095 97 / 114 (K = 3 97 / 57, 7 97 / 98); K = 11
// to 15 256 x 4095 7.4 / 8.0 to 9.0, 8000 x 4095 97 / 173 to 190, 2000 x 4096 28.2 / 32.4 to 34.7 (60 x 40000 13.9 / 11.8 to 12.5).
bool short_pays(const GemmCall& g) {
    const double outputs = (double)g.I * g.J * g.batch;
    if (g.K > 10) return outputs <= (double)(1 << 19) || (g.J <= 64 && short_vec(g));
    return g.K <= 4 || short_vec(g) || outputs <= (double)(1 << 22);
}
template <int KT, bool V>
__global__ void __launch_bounds__(32 * kShortGroups) short_gemm_kernel(const SimtParams p) {
    __shared__ float sQ[kShortRows * kShortGroups][KT];
    griddep_wait_then_launch();
    const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
    const int i = (blockIdx.x * 32 + lane) * 4, j0 = blockIdx.y * kShortRows * kShortGroups, b = blockIdx.z;
    const float* P = p.P + (long long)b * p.strideP;
    const float* Q = p.Q + (long long)b * p.strideQ;
    float a[KT][4];
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        if (V) {
            *reinterpret_cast<float4*>(a[k]) = k < p.K && i < p.I ? *reinterpret_cast<const float4*>(P + (long long)k * p.ldp + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
#pragma unroll
            for (int x = 0; x < 4; ++x) a[k][x] = k < p.K && i + x < p.I ? P[(long long)k * p.ldp + i + x] : 0.f;
        }
    }
    for (int e = threadIdx.x; e < kShortRows * kShortGroups * KT; e += 32 * kShortGroups) {
        const int r = e / KT, k = e % KT, j = j0 + r;
        sQ[r][k] = j < p.J && k < p.K ? Q[p.q_mn ? (long long)k * p.ldq + j : (long long)j * p.ldq + k] : 0.f;
    }
    __syncthreads();
    if (i >= p.I) return;
#pragma unroll
    for (int r = 0; r < kShortRows; ++r) {
        const int row = r * kShortGroups + group, j = j0 + row;
        if (j >= p.J) return;
        float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int x = 0; x < 4; ++x)
                if (k < p.K) y[x] = fmaf(a[k][x], sQ[row][k], y[x]);
        float* dst = p.C + (long long)b * p.strideC + (long long)j * p.ldc + i;
        if (V && !p.accumulate && !p.bias_i && !p.bias_j && !p.relu) {
            *reinterpret_cast<float4*>(dst) = make_float4(y[0], y[1], y[2], y[3]);
            continue;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (i + x >= p.I) break;
            float v = y[x];
            if (p.bias_i) v += p.bias_i[i + x];
            if (p.bias_j) v += p.bias_j[j];
            if (p.accumulate) v += dst[x];
            dst[x] = p.relu ? fmaxf(v, 0.f) : v;
        }
    }
}
cudaError_t launch_short(cb_ctx* ctx, const SimtParams& p) {
    const bool vec = short_vec(p);
    typedef void (*Kernel)(const SimtParams);
    static const Kernel kernels[2][3] = {{short_gemm_kernel<4, false>, short_gemm_kernel<10, false>, short_gemm_kernel<16, false>},
                                         {short_gemm_kernel<4, true>, short_gemm_kernel<10, true>, short_gemm_kernel<16, true>}};
    const dim3 grid((unsigned)((p.I + 127) / 128), (unsigned)((p.J + kShortRows * kShortGroups - 1) / (kShortRows * kShortGroups)), (unsigned)p.batch);
    cudaError_t e = launch_dep(ctx, kernels[vec ? 1 : 0][p.K <= 4 ? 0 : (p.K <= 10 ? 1 : 2)], grid, dim3(32 * kShortGroups), 0, p);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

cudaError_t launch_rows(cb_ctx* ctx, const SimtParams& sp) {
    typedef void (*Kernel)(const SimtParams);
    static const Kernel kernels[2][3] = {{thin_rows_kernel<4, false>, thin_rows_kernel<8, false>, thin_rows_kernel<16, false>},
                                         {thin_rows_kernel<4, true>, thin_rows_kernel<8, true>, thin_rows_kernel<16, true>}};
    const bool vec = ((sp.ldp | sp.ldq | sp.K) & 3) == 0 && ((reinterpret_cast<uintptr_t>(sp.P) | reinterpret_cast<uintptr_t>(sp.Q)) & 15u) == 0;
    const dim3 grid((unsigned)((sp.J + kThinRows - 1) / kThinRows * sp.splits));
    cudaError_t e = launch_dep_on(ctx->stream, ctx->pdl != 0, kernels[vec ? 1 : 0][sp.I <= 4 ? 0 : (sp.I <= 8 ? 1 : 2)], grid, dim3(256), 0, sp.splits, sp);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

cudaError_t launch_thin(cb_ctx* ctx, const SimtParams& sp, dim3 grid) {
    typedef void (*Kernel)(const SimtParams);
    static const Kernel kernels[2][3] = {{thin_gemm_k_kernel<4>, thin_gemm_k_kernel<8>, thin_gemm_k_kernel<16>},
                                         {thin_gemm_mn_kernel<4>, thin_gemm_mn_kernel<8>, thin_gemm_mn_kernel<16>}};
    cudaError_t e = launch_dep(ctx, kernels[sp.q_mn ? 1 : 0][sp.I <= 4 ? 0 : (sp.I <= 8 ? 1 : 2)], grid, dim3(256), 0, sp);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

template <class T>
cudaError_t launch_tile(cb_ctx* ctx, const SimtParams& sp, dim3 grid) {
    typedef void (*Kernel)(const SimtParams);
    static const Kernel forms[4] = {simt_gemm_kernel<T, false, false>, simt_gemm_kernel<T, false, true>,
                                    simt_gemm_kernel<T, true, false>, simt_gemm_kernel<T, true, true>};
    const Kernel k = forms[(sp.p_mn ? 2 : 0) + (sp.q_mn ? 1 : 0)];
    cudaError_t e = raise_dynamic_smem_once(k, ctx->device, ctx->max_smem_optin, nullptr);
    if (e != cudaSuccess) return e;
    e = launch_dep(ctx, k, grid, dim3(T::NT), T::kSmem, sp);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

// V: one run of quads. Otherwise `items` floats as rows of `width`, ld apart, in matrices of `rows`, stride apart.
template <bool V>
__global__ void __launch_bounds__(256) clear_kernel(float* __restrict__ p, const FastDiv width, const FastDiv rows, long long ld,
                                                    long long stride, uint32_t items) {
    griddep_wait_then_launch();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < items; i += gridDim.x * blockDim.x) {
        if (V) {
            reinterpret_cast<float4*>(p)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            uint32_t c, r;
            const uint32_t b = rows.split(width.split(i, c), r);
            p[b * stride + r * ld + c] = 0.f;
        }
    }
}

}  // namespace

// Clears the output of a product whose contraction is split over atomic adds. One launch that chains to the kernels around it: a
// cudaMemset2DAsync per matrix of a batch took longer than the product (8 x 129 x 131 x 133: 24.7 us). Split outputs are small, so
// 32-bit indexes do: at most 32 tiles of 128 x 128 an SM on the CUDA cores, half a tile of 128 x 256 an SM on the tensor cores.
int clear_output(cb_ctx* ctx, float* p, long long width, long long ld, long long rows, long long stride, long long batch, const char* who) {
    if (ld == width) {
        width *= rows;
        rows = 1;
        ld = width;
    }
    if (rows == 1 && (stride == width || batch == 1)) {
        width *= batch;
        batch = 1;
    }
    const long long n = width * rows * batch;
    const bool vec = rows * batch == 1 && (n & 3) == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
    const uint32_t items = (uint32_t)(vec ? n / 4 : n);
    long long grid = ((long long)items + 1023) / 1024;
    if (grid > ctx->sm_count * 8) grid = ctx->sm_count * 8;
    cudaError_t e = launch_dep(ctx, vec ? clear_kernel<true> : clear_kernel<false>, dim3((unsigned)grid), dim3(256), 0, p, FastDiv(width),
                               FastDiv(rows), ld, stride, items);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, who);
    ctx->launches += 1;
    return CB_OK;
}

static int gemm_zero_output(cb_ctx* ctx, const GemmCall& g) {
    // rows of the output as laid out in memory: out_mode 0 -> J rows of I floats, 1 -> I rows of J floats
    return clear_output(ctx, g.C, g.out_mode == 0 ? g.I : g.J, g.ldc, g.out_mode == 0 ? g.J : g.I, g.strideC, g.batch, "clear of a split product");
}

// Puts the thin extent on the I side: D'[j][i] with the operands' roles swapped.
static void swap_sides(GemmCall& g) {
    std::swap(g.I, g.J);
    std::swap(g.P, g.Q); std::swap(g.ldp, g.ldq); std::swap(g.strideP, g.strideQ); std::swap(g.p_mn, g.q_mn);
    std::swap(g.ep.bias_i, g.ep.bias_j);
    g.out_mode ^= 1;
}
static void set_operands(SimtParams& sp, const GemmCall& g) {
    sp.I = g.I; sp.J = g.J; sp.K = g.K; sp.batch = g.batch;
    sp.P = g.P; sp.ldp = g.ldp; sp.strideP = g.strideP; sp.p_mn = g.p_mn;
    sp.Q = g.Q; sp.ldq = g.ldq; sp.strideQ = g.strideQ; sp.q_mn = g.q_mn;
    sp.C = g.C; sp.ldc = g.ldc; sp.strideC = g.strideC; sp.out_mode = g.out_mode; sp.accumulate = g.accumulate;
    sp.bias_i = g.ep.bias_i; sp.bias_j = g.ep.bias_j; sp.relu = g.ep.relu;
}

int launch_thin_rows(cb_ctx* ctx, const GemmCall& g_in) {
    GemmCall g = g_in;
    if (ctx->model_pass || g.batch != 1 || g.kfold > 1 || g.p_mn || g.q_mn || g.K < 64) return CB_EUNSUPPORTED;
    if (g.J <= 16 && g.I > 16) swap_sides(g);
    const bool fp32 = ctx->math == CB_MATH_FP32;
    // Every block reads the whole thin operand and blocks of up to 16 thin rows are one to an SM (8: two), so larger products are the tensor
    // cores' (or, fp32, thin_gemm_k_kernel's). us, TF32 there / here, I x J x K: 10 x 128 x 64 4.3 / 3.1, x 1024 7.2 / 3.4, x 4096 6.7 / 5.4; 10 x
    // 1024 x 64 4.6 / 5.3, x 1024 8.7 / 6.1, 10 x 1024 x 4096 10.7 / 13.9; 2 x 4096 x 4096 23.8 / 9.6. Over 272 products of 33 to 4000 rows, K 67 to
    // 8000, 1 to 16 columns, both modes: 1.30 times as fast, none slower by more than 3 %.
    const int blocks = (g.J + kThinRows - 1) / kThinRows, room = g.I > 8 ? ctx->sm_count : 2 * ctx->sm_count;
    if (g.I > 16 || g.J < 32 || (double)g.J * g.K > (double)(g.I <= 4 ? 1 << 24 : fp32 ? 1 << 18 : g.I <= 8 ? 1 << 21 : 1 << 20) || (fp32 && g.I > 4 && g.K > 2048) || (blocks > room && g.K < 512))
        return CB_EUNSUPPORTED;
    SimtParams sp{};
    set_operands(sp, g);
    sp.splits = 1;
    // As many clusters as are resident at a time: those of 4 and 8 don't fill every group of SMs (one block an SM: 33 and 15 of them, two: 71
    // and 33). One cluster more cost a second round: 133 x 10 x 4096 6.9 us on the tensor cores, 8.3 here in 34 clusters of 4.
    auto fits = [&](int splits) { return blocks * splits <= (splits < 4 ? room : splits == 4 ? room * 7 / 8 : room * 3 / 4); };
    while (sp.splits < 8 && fits(sp.splits * 2) && g.K > sp.splits * kThinStep) sp.splits *= 2;
    sp.k_per_split = ((g.K + sp.splits - 1) / sp.splits + 127) / 128 * 128;
    cudaError_t e = launch_rows(ctx, sp);
    if (e != cudaSuccess) return check_cuda(ctx, e, "thin_rows_kernel launch");
    ctx->launches += 1;
    ctx->last_kernel = "simt_fp32";
    return CB_OK;
}

static int launch_simt_gemm(cb_ctx* ctx, const GemmCall& g_in, bool* summed) {
    GemmCall g = g_in;
    const int fold = g.kfold > 1 ? g.kfold : 1;
    const bool short_k = g.K <= 16 && g.p_mn && g.out_mode == 0 && fold == 1 && g.I >= 128 && g.J <= 65535 * kShortRows * kShortGroups && g.batch <= 65535 &&
                         short_pays(g);
    const bool swapped = !short_k && g.J <= 16 && g.I > 16;
    if (swapped) swap_sides(g);
    // no atomic sums in a model's passes: one rounding in an activation moves the gradients of a deep model by percents
    const bool may_split = !ctx->deterministic && !ctx->model_pass && g.ep.relu == 0;
    SimtParams sp{};
    set_operands(sp, g);
    if (short_k) {
        cudaError_t e = launch_short(ctx, sp);
        if (e != cudaSuccess) return check_cuda(ctx, e, "short_gemm_kernel launch");
        ctx->launches += 1;
        ctx->last_kernel = "simt_fp32";
        return CB_OK;
    }
    // A tile of 32 or more rows would be mostly padding; below 64 k the tiled kernel's one or two slices cost no more.
    if (g.I <= 16 && g.batch == 1 && fold == 1 && g.J >= 32 && g.K >= 64) {
        const int jblocks = (g.J + 31) / 32;
        int splits = 1;
        if (may_split) {
            splits = 2 * ctx->sm_count / jblocks;
            if (splits > g.K / 128) splits = g.K / 128;
            if (splits < 1) splits = 1;
        }
        int kps = (g.K + splits - 1) / splits;
        kps = ((kps + 31) / 32) * 32;
        splits = (g.K + kps - 1) / kps;
        sp.splits = splits; sp.k_per_split = kps;
        sp.atomic_out = splits > 1 ? 1 : 0;
        if (sp.atomic_out && !g.accumulate) {
            int rc = gemm_zero_output(ctx, g);
            if (rc != CB_OK) return rc;
        }
        if (splits > 65535) return fail(ctx, CB_EUNSUPPORTED, "thin gemm: contraction too long");
        if (g_in.q_sum && swapped && sp.q_mn) {
            sp.thin_sum = g_in.q_sum;
            if (summed) *summed = true;
        }
        cudaError_t e = launch_thin(ctx, sp, dim3((unsigned)jblocks, (unsigned)splits));
        if (e != cudaSuccess) return check_cuda(ctx, e, "thin_gemm_kernel launch");
        ctx->launches += 1;
        ctx->last_kernel = "simt_fp32";
        return CB_OK;
    }
    sp.per_fold = (g.K + kBK - 1) / kBK;
    if ((long long)sp.per_fold * fold > (1LL << 30)) return fail(ctx, CB_EUNSUPPORTED, "simt gemm: contraction longer than 2^34");
    sp.slices = sp.per_fold * fold;
    const simt::Choice c = simt::choose_tile(ctx->sm_count, g.I, g.J, sp.slices, g.batch, may_split);
    sp.splits = c.splits; sp.k_per_split = c.per_split;
    sp.atomic_out = c.splits > 1 ? 1 : 0;
    if ((long long)g.batch * c.splits > 65535) return fail(ctx, CB_EUNSUPPORTED, "simt gemm: batch*splits > 65535");
    if (sp.atomic_out && !g.accumulate) {
        int rc = gemm_zero_output(ctx, g);
        if (rc != CB_OK) return rc;
    }
    cudaError_t e = cudaSuccess;
    const int rc_grid = simt::with_tile(c.tile, [&](auto tile) {
        typedef decltype(tile) T;
        const long long gy = ((long long)g.J + T::BN - 1) / T::BN;
        if (gy > 65535) return fail(ctx, CB_EUNSUPPORTED, "simt gemm: more than 65535 column tiles");
        e = launch_tile<T>(ctx, sp, dim3((unsigned)((g.I + T::BM - 1) / T::BM), (unsigned)gy, (unsigned)(g.batch * c.splits)));
        return (int)CB_OK;
    });
    if (rc_grid != CB_OK) return rc_grid;
    if (e != cudaSuccess) return check_cuda(ctx, e, "simt_gemm_kernel launch");
    ctx->launches += 1;
    ctx->last_kernel = "simt_fp32";
    return CB_OK;
}

// Products of CB_MATH_FP32 and those TMA cannot address. In the passes of a model they stay on the CUDA cores, where they take two to three
// times as long: their sums are then those that models have always had. (One rounding in an activation moves the gradients of a deep
// model by percents, whatever code computed it; neither path is the better one in that.)
int launch_fp32_gemm(cb_ctx* ctx, const GemmCall& g, bool* summed) {
    if (!ctx->model_pass) {
        int rc = launch_split_gemm(ctx, g);
        if (rc == CB_EUNSUPPORTED) rc = launch_thin_rows(ctx, g);
        if (rc != CB_EUNSUPPORTED) return rc;
    }
    return launch_simt_gemm(ctx, g, summed);
}

}  // namespace cb
