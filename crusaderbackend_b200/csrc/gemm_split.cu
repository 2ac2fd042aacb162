// GEMM forms on the bf16-split tensor-core body of split_core.cuh: CB_MATH_FP32 and every operand pair TMA cannot address, where
// the product is large enough (gemm_simt.cu serves the others).
#include <cstdlib>

#include "split_core.cuh"

namespace cb {
namespace {

using split::kBK;
using split::Kind;

struct SplitParams {
    int I, J, K, batch;
    const float* P; long long ldp, strideP;
    const float* Q; long long ldq, strideQ;
    float* C; long long ldc, strideC; int out_mode, accumulate, atomic_out;
    const float* bias_i; const float* bias_j; int relu;
    int splits, per_split;  // k-blocks of a split
    int blocks, per_fold;   // k-blocks of the whole contraction, of one operand pair (batch folded into it, else = blocks)
    int* status;
};

// Element (e, k) of an operand: base + e * ld + k, or base + k * ld + e where MN. Rows past the end repeat the last one: their
// outputs are not stored.
template <Kind KIND>
__device__ __forceinline__ const float* element(const float* base, long long ld, int e, int k) {
    return base + (KIND == split::MN ? (long long)k * ld + e : (long long)e * ld + k);
}
template <class Sh, Kind KIND>
__device__ __forceinline__ void load_p(float (&v)[split::ShareP<Sh, KIND>::kValues], const float* base, long long ld, int e0, int E, int k0, int K, int tid) {
    typedef split::ShareP<Sh, KIND> S;
    const int k = k0 + S::k(tid, 0);
    if (k0 + kBK <= K) {  // the same for the whole CTA
        const float* src = element<KIND>(base, ld, KIND == split::MN ? min(e0 + S::row(tid, 0), E - 1) : 0, k);
#pragma unroll
        for (int x = 0; x < S::kValues; ++x)
            v[x] = __ldg(split::step(src, (uint32_t)ld * 4u, KIND == split::MN ? x : min(e0 + S::row(tid, x), E - 1)));
    } else {
#pragma unroll
        for (int x = 0; x < S::kValues; ++x) {
            const int kx = k0 + S::k(tid, x);
            v[x] = split::load_if(element<KIND>(base, ld, min(e0 + S::row(tid, x), E - 1), kx), kx < K);
        }
    }
}
template <class Sh, Kind KIND>
__device__ __forceinline__ void load_q(float (&v)[split::ShareQ<Sh, KIND>::kValues], const float* base, long long ld, int e0, int E,
                                       int k0, int K, int tid) {
    typedef split::ShareQ<Sh, KIND> S;
    if (!S::active(tid)) return;
    if (k0 + kBK <= K) {
#pragma unroll
        for (int u = 0; u < S::kUnits; ++u) {
            const float* src = element<KIND>(base, ld, min(e0 + S::row(tid, u), E - 1), k0 + S::k(tid, u));
            if (KIND == split::KV) {
                *reinterpret_cast<float4*>(&v[u * 8]) = __ldg(reinterpret_cast<const float4*>(src));
                *reinterpret_cast<float4*>(&v[u * 8 + 4]) = __ldg(reinterpret_cast<const float4*>(src) + 1);
            } else {
#pragma unroll
                for (int x = 0; x < S::kUnit; ++x) v[u * S::kUnit + x] = __ldg(KIND == split::MN ? split::step(src, (uint32_t)ld * 4u, x) : src + x);
            }
        }
    } else {
#pragma unroll
        for (int u = 0; u < S::kUnits; ++u)
#pragma unroll
            for (int x = 0; x < S::kUnit; ++x) {
                const int k = k0 + S::k(tid, u) + x;
                v[u * S::kUnit + x] = split::load_if(element<KIND>(base, ld, min(e0 + S::row(tid, u), E - 1), k), k < K);
            }
    }
}

template <class S, Kind P_, Kind Q_>
struct GemmSource {
    static constexpr Kind kP = P_, kQ = Q_;
    static constexpr bool kTable = false;
    const SplitParams& p;
    int b, part, i0, j0, block0;
    // operand pair and first k of a k-block of the contraction
    __device__ __forceinline__ void where(int t, int& pair, int& k) const {
        pair = b;
        k = t;
        if (p.per_fold != p.blocks) {
            pair = k / p.per_fold;
            k -= pair * p.per_fold;
        }
        k *= kBK;
    }
    __device__ __forceinline__ void prepare(int, int) {}
    __device__ __forceinline__ void load(int t, int tid, float (&vp)[split::ShareP<S, kP>::kValues], float (&vq)[split::ShareQ<S, kQ>::kValues]) {
        int pair, k;
        where(block0 + t, pair, k);
        load_p<S, kP>(vp, p.P + pair * p.strideP, p.ldp, i0, p.I, k, p.K, tid);
        load_q<S, kQ>(vq, p.Q + pair * p.strideQ, p.ldq, j0, p.J, k, p.K, tid);
    }
    template <bool LOW>
    __device__ __forceinline__ void store(int row, int first, int n, uint32_t mine) const {
        const int i = i0 + row;
        n = min(n, p.J - j0 - first);
        if (i >= p.I) return;
        const bool biased = part == 0 && p.bias_i != nullptr;
        const float bias = biased ? p.bias_i[i] : 0.f;
        const float* bias_j = part == 0 && p.bias_j ? p.bias_j + j0 + first : nullptr;
        float* dst = p.C + (long long)b * p.strideC + (p.out_mode == 0 ? (long long)(j0 + first) * p.ldc + i : (long long)i * p.ldc + j0 + first);
        const long long step = p.out_mode == 0 ? p.ldc : 1;
        if (!biased && !bias_j && !p.relu) {
            // the plain forms without a branch in the loop: reads of several columns are in flight together. One atomic add to an
            // output is what a read, an addition and a write are, without waiting for the read.
            if (p.atomic_out || p.accumulate)
#pragma unroll 8
                for (int c = 0; c < n; ++c, dst += step) split::add_to<LOW>(dst, split::staged(mine, c));
            else
#pragma unroll 8
                for (int c = 0; c < n; ++c, dst += step) *dst = split::staged(mine, c);
            return;
        }
#pragma unroll 4
        for (int c = 0; c < n; ++c, dst += step) {
            float y = split::staged(mine, c);
            if (biased) y += bias;
            if (bias_j) y += bias_j[c];
            if (p.atomic_out) {
                split::add_to<LOW>(dst, y);
            } else {
                if (p.accumulate) y += *dst;
                if (p.relu) y = fmaxf(y, 0.f);
                *dst = y;
            }
        }
    }
};

template <class S, Kind KP, Kind KQ>
__global__ void __launch_bounds__(S::NT, S::kCtas) split_gemm_kernel(const __grid_constant__ SplitParams p) {
    extern __shared__ uint8_t smem[];
    __shared__ split::Barriers bars;
    __shared__ __align__(16) float patches[split::ShareP<S, KP>::kPatches];
    const int b = blockIdx.z / p.splits, part = blockIdx.z - b * p.splits;
    GemmSource<S, KP, KQ> src{p, b, part, (int)blockIdx.x * S::BM, (int)blockIdx.y * S::BN, part * p.per_split};
    split::run<S>(src, min(p.per_split, p.blocks - src.block0), smem, bars, patches, p.status);
}

template <class S, Kind KP, Kind KQ>
cudaError_t launch_kernel(cb_ctx* ctx, const SplitParams& sp, dim3 grid) {
    auto kernel = split_gemm_kernel<S, KP, KQ>;
    cudaError_t e = raise_dynamic_smem_once(kernel, ctx->device, ctx->max_smem_optin, nullptr);
    if (e != cudaSuccess) return e;
    e = launch_dep(ctx, kernel, grid, dim3(S::NT), (size_t)S::kSmem, sp);
    return e == cudaSuccess ? cudaGetLastError() : e;
}
template <class S, Kind KP>
cudaError_t launch_q(cb_ctx* ctx, const SplitParams& sp, dim3 grid, Kind q) {
    switch (q) {
        case split::MN: return launch_kernel<S, KP, split::MN>(ctx, sp, grid);
        case split::K: return launch_kernel<S, KP, split::K>(ctx, sp, grid);
        default: return launch_kernel<S, KP, split::KV>(ctx, sp, grid);
    }
}
template <class S>
cudaError_t launch_shape(cb_ctx* ctx, const SplitParams& sp, dim3 grid, Kind p, Kind q) {
    return p == split::MN ? launch_q<S, split::MN>(ctx, sp, grid, q) : launch_q<S, split::K>(ctx, sp, grid, q);
}

Kind kind_of(const float* base, long long ld, long long stride, int mn) {
    if (mn) return split::MN;
    return ((reinterpret_cast<uintptr_t>(base) & 15u) == 0 && ((ld | stride) & 3) == 0) ? split::KV : split::K;
}

}  // namespace

// Thin products stay on the kernels that stream the long operand once, contractions of one or two blocks on the CUDA cores. The least
// multiplications: where a launch of gemm_simt.cu and one of these take the same time (257^3: 9.4 us against 8.6 to 10.2, 513 x 65 x
// 257: 10.2 against 9.7; 515^3 17.8 against 10.6, 2047^3 421 against 123).
constexpr long long kLeastGemm = 1LL << 24;

int launch_split_gemm(cb_ctx* ctx, const GemmCall& g) {
    const int fold = g.kfold > 1 ? g.kfold : 1;
    if (g.I <= 16 || g.J <= 16 || g.K < 64 || !split::worth_it(g.I, g.J, g.K, (long long)g.batch * fold, kLeastGemm)) return CB_EUNSUPPORTED;
    const bool may_split = !ctx->deterministic && !ctx->model_pass && g.ep.relu == 0;
    SplitParams sp{};
    sp.I = g.I; sp.J = g.J; sp.K = g.K; sp.batch = g.batch;
    sp.P = g.P; sp.ldp = g.ldp; sp.strideP = g.strideP;
    sp.Q = g.Q; sp.ldq = g.ldq; sp.strideQ = g.strideQ;
    sp.C = g.C; sp.ldc = g.ldc; sp.strideC = g.strideC; sp.out_mode = g.out_mode; sp.accumulate = g.accumulate;
    sp.bias_i = g.ep.bias_i; sp.bias_j = g.ep.bias_j; sp.relu = g.ep.relu;
    sp.status = ctx->d_status;
    sp.per_fold = (g.K + kBK - 1) / kBK;
    if ((long long)sp.per_fold * fold > (1LL << 30) || g.ldp >= (1LL << 30) || g.ldq >= (1LL << 30)) return CB_EUNSUPPORTED;
    sp.blocks = sp.per_fold * fold;
    const split::Choice c = split::choose_shape(ctx->sm_count, g.I, g.J, sp.blocks, g.batch, may_split, split::kMatrix);
    sp.splits = c.splits; sp.per_split = c.per_split;
    sp.atomic_out = c.splits > 1 ? 1 : 0;
    const long long gy = ((long long)g.J + c.bn - 1) / c.bn, gz = (long long)g.batch * c.splits;
    if (gy > 65535 || gz > 65535) return CB_EUNSUPPORTED;
    if (sp.atomic_out && !g.accumulate) {
        const int rc = clear_output(ctx, g.C, g.out_mode == 0 ? g.I : g.J, g.ldc, g.out_mode == 0 ? g.J : g.I, g.strideC, g.batch, "clear of a split product");
        if (rc != CB_OK) return rc;
    }
    const dim3 grid((unsigned)((g.I + 127) / 128), (unsigned)gy, (unsigned)gz);
    const Kind kp = g.p_mn ? split::MN : split::K, kq = kind_of(g.Q, g.ldq, g.strideQ, g.q_mn);
    cudaError_t e = c.bn == 128 ? launch_shape<split::Shape<128>>(ctx, sp, grid, kp, kq)
                  : c.bn == 64 ? launch_shape<split::Shape<64>>(ctx, sp, grid, kp, kq)
                               : launch_shape<split::Shape<32>>(ctx, sp, grid, kp, kq);
    if (e != cudaSuccess) return check_cuda(ctx, e, "split_gemm_kernel launch");
    ctx->launches += 1;
    ctx->last_kernel = "umma_fp32";
    return CB_OK;
}

}  // namespace cb
