// CUDA-core fp32 convolution kernels (any filter size, stride and padding) and the cb_conv_* dispatchers.
// These serve CB_MATH_FP32 and every geometry the tensor-core implicit-GEMM kernels do not cover; they compute
// exact fp32 FMAs. Index maps follow seblas/operations/cuConv.cu:105-115 (forward) and the adjoint of it for the
// two gradients (the reference's weight-gradient map at :570-571 is wrong for stride > 1 and is not reproduced).
#include <cstdlib>
#include <cstring>

#include "cb_ptx.cuh"
#include "conv_gather.cuh"
#include "conv_patch.h"
#include "simt_core.cuh"
#include "split_core.cuh"

namespace cb {

using namespace gather;

// conv_split.cu
cudaError_t launch_split_gather(cb_ctx* ctx, const GatherParams& p, const split::Choice& c, bool mask, long long pixels, int sets);
cudaError_t launch_split_wgrad(cb_ctx* ctx, const WgradParams& p, const split::Choice& c, bool mask);

namespace {

// ---- forward and data gradient
template <class T, bool MASK>
struct GatherSource {
    const GatherParams& p;
    const PixelSet& s;
    TapK* table;             // [2][kBK]
    const float* img;        // this thread's pixel: its image, its taps, offset of the first tap
    Position at;
    int base;
    int j0, slice0;
    __device__ __forceinline__ void begin(int t) {
        if (threadIdx.x < simt::kBK) table[(t & 1) * simt::kBK + threadIdx.x] = tap_of<MASK>(p, s, (slice0 + t) * simt::kBK + threadIdx.x);
    }
    __device__ __forceinline__ void load(int t, uint32_t dst) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const TapK* tab = table + (t & 1) * simt::kBK;
        typedef simt::MnLanes<T::BM, T::NW> L;
        const uint32_t dp = dst + simt::slot<T::BM>(L::k(warp, 0), L::e(warp, lane));
#pragma unroll
        for (int r = 0; r < L::kCopies; ++r) {
            const TapK q = tab[L::k(warp, r)];
            const bool ok = tap_inside<MASK>(at, q.bits, p.H, p.W) && (MASK || q.woff >= 0);
            simt::cp_async4(dp + simt::slot<T::BM>(r * L::kStep, 0), img + (ok ? base + q.off : 0), ok);
        }
        typedef simt::KLanes<T::BN, T::NW> R;
        const int k = R::k(warp, lane), j = j0 + R::e(warp, lane, 0);
        const int woff = tab[k].woff;
        const float* src = p.Wt + (long long)j * p.w_out + woff;
        const long long step = (long long)R::kStep * p.w_out;
        const uint32_t dq = dst + simt::kOperandBytes<T::BM> + simt::slot<T::BN>(k, R::e(warp, lane, 0));
#pragma unroll
        for (int r = 0; r < R::kCopies; ++r, src += step) {
            const bool ok = woff >= 0 && j + r * R::kStep < p.OUTC;
            simt::cp_async4(dq + simt::slot<T::BN>(0, r * R::kStep), ok ? src : p.Wt, ok);
        }
    }
};

// 32 -> 32 channels, 28 x 28 maps, batch 32, 3 x 3: 141 us (forward) and 140 us (data gradient) with the kernels this
// replaces, one thread per pixel and 8 channels, 1.6 TFLOP/s: two loads per eight FMAs.
template <class T, bool MASK>
__global__ void __launch_bounds__(T::NT, T::kMinCtas) conv_gather_simt(const __grid_constant__ GatherParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ TapK table[2 * simt::kBK];
    griddep_wait_then_launch();
    const int set = blockIdx.z / p.splits, split = blockIdx.z - set * p.splits;
    const PixelSet& s = p.sets[set];
    const long long pixels = (long long)p.N * s.UH * s.UW;
    const long long i0 = (long long)blockIdx.x * T::BM;
    if (i0 >= pixels) return;  // the grid is sized for the largest set
    GatherSource<T, MASK> src{p, s, table, p.In, Position{-(1 << 29), 0, 0u}, 0, (int)blockIdx.y * T::BN, split * p.per_split};
    {
        const long long i = i0 + simt::MnLanes<T::BM, T::NW>::e(threadIdx.x >> 5, threadIdx.x & 31);
        if (i < pixels) {
            src.at = input_of<MASK>(p, s, i, src.img);
            src.base = src.at.h0 * p.W + src.at.w0;
        }
    }
    const int slices = (s.K + simt::kBK - 1) / simt::kBK;
    simt::Acc<T> acc;
    simt::main_loop<T>(src, max(0, min(p.per_split, slices - src.slice0)), (uint32_t)__cvta_generic_to_shared(smem), acc);

    const int plane = p.OHH * p.OWW;
    int at[2][4];            // position of this thread's pixels in an output plane, -1: past the end
    float* out[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const long long i = i0 + simt::own_row<T>() + 32 * h + x;
            at[h][x] = -1;
            out[h][x] = p.Out;
            if (i < pixels) at[h][x] = output_of(p, s, i, out[h][x]);
        }
    simt::for_outputs<T>(acc, 0, src.j0, [&](int j, int i, float (&v)[4]) {
        if (j >= p.OUTC) return;
        const int h = (i >> 5) & 1;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (at[h][x] < 0) return;
            const long long idx = (long long)j * plane;
            float* dst = out[h][x] + idx;
            if (p.atomic_out) {
                float y = v[x];
                if (split == 0 && p.ep.bias) y += p.ep.bias[j];
                atomicAdd(dst, y);
            } else {
                *dst = apply_epilogue(p.ep, v[x], j, idx + at[h][x], p.ep.accumulate ? *dst : 0.f);
            }
        }
    });
}

// ---- weight gradient
template <class T, bool MASK>
struct WgradSource {
    const WgradParams& p;
    PixelK* table;           // [2][kBK]
    const TapI* rows;        // [BM]
    int j0, slice0, opix;
    __device__ __forceinline__ void begin(int t) {
        if (threadIdx.x < simt::kBK) table[(t & 1) * simt::kBK + threadIdx.x] = pixel_of<MASK>(p, (slice0 + t) * simt::kBK + threadIdx.x);
    }
    __device__ __forceinline__ void load(int t, uint32_t dst) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        typedef simt::KLanes<T::BM, T::NW> L;
        const int k = L::k(warp, lane);
        const PixelK q = table[(t & 1) * simt::kBK + k];
        const float* first = p.X + q.x;
        const TapI* row = rows + L::e(warp, lane, 0);
        const uint32_t dp = dst + simt::slot<T::BM>(k, L::e(warp, lane, 0));
#pragma unroll
        for (int r = 0; r < L::kCopies; ++r) {
            const TapI w = row[r * L::kStep];
            const bool ok = tap_inside<MASK>(q.at, w.bits, p.g.IH, p.g.IW) && (MASK || w.off >= 0);
            simt::cp_async4(dp + simt::slot<T::BM>(0, r * L::kStep), ok ? first + w.off : p.X, ok);
        }
        typedef simt::KLanes<T::BN, T::NW> R;
        const int j = j0 + R::e(warp, lane, 0);
        const float* src = p.dY + q.y + (long long)j * opix;
        const long long step = (long long)R::kStep * opix;
        const uint32_t dq = dst + simt::kOperandBytes<T::BM> + simt::slot<T::BN>(k, R::e(warp, lane, 0));
#pragma unroll
        for (int r = 0; r < R::kCopies; ++r, src += step) {
            const bool ok = q.y >= 0 && j + r * R::kStep < p.g.OC;
            simt::cp_async4(dq + simt::slot<T::BN>(0, r * R::kStep), ok ? src : p.dY, ok);
        }
    }
};

// 32 -> 32 channels, 28 x 28 maps, batch 32, 3 x 3: 534 us with the kernel this replaces (one block per channel pair,
// every pixel of X and dY re-read by 32 of them).
template <class T, bool MASK>
__global__ void __launch_bounds__(T::NT, T::kMinCtas) conv_wgrad_simt(const WgradParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ PixelK table[2 * simt::kBK];
    __shared__ TapI rows[T::BM];
    griddep_wait_then_launch();
    const int i0 = blockIdx.x * T::BM;
    for (int e = threadIdx.x; e < T::BM; e += T::NT) rows[e] = row_of<MASK>(p, i0 + e);
    WgradSource<T, MASK> src{p, table, rows, (int)blockIdx.y * T::BN, (int)blockIdx.z * p.per_split, p.g.OH * p.g.OW};
    const int slices = (p.pixels + simt::kBK - 1) / simt::kBK;
    simt::Acc<T> acc;
    simt::main_loop<T>(src, min(p.per_split, slices - src.slice0), (uint32_t)__cvta_generic_to_shared(smem), acc);
    simt::for_outputs<T>(acc, i0, src.j0, [&](int j, int i, float (&v)[4]) {
        if (j >= p.g.OC) return;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (i + x >= p.I) return;
            float* dst = p.dW + (long long)j * p.I + i + x;
            if (p.mode == 2) atomicAdd(dst, v[x]);
            else if (p.mode == 1) *dst += v[x];
            else *dst = v[x];
        }
    });
}

// Multiplications from which a pass runs at fp32 accuracy on the tensor cores (conv_split.cu).
constexpr long long kLeastConv = 1LL << 22;

// us a launch of conv_gather_split takes, by a model fitted to 555 passes (7.5 % off on average). conv_patch.cu is taken where its own model
// is 12 % below: 6400 passes of drawn layers that go there are 1.43 times as fast as without it, 3 % of them slower by more than 4 %, by 12 % on
// average and 1.41 to 1.56 times at most (5x5 filters, grids of just under two CTAs an SM). us without / with: forward 32 -> 32 at 28 x 28, batch
// 32 14.6 / 10.9, its data gradient 17.6 / 10.9; 32 -> 64 at 32 x 32, stride 2, batch 128 21.1 / 18.2; 16 -> 32 5x5 at 46 x 46, batch 23 29.0 /
// 19.0 and 61.2 / 26.0; few channels at stride 2 stay: 5 -> 38 at 32 x 32, batch 18 4.8 / 6.8.
double gather_us(int sm_count, long long I, int OUTC, long long blocks, bool may_split, const GatherParams& p, const PixelSet* sets) {
    const split::Choice c = split::choose_shape(sm_count, I, OUTC, blocks, 1, may_split, split::kGather);
    const long long ctas = (I + 127) / 128 * ((OUTC + c.bn - 1) / c.bn) * c.splits;
    const bool pairs = c.bn == 32 && ctas > sm_count, dgrad = p.sgn < 0, strided = dgrad && sets[0].ohs == 2;
    const double block = (c.bn == 128 ? 1.303 : c.bn == 64 ? 0.756 : 0.621) * (dgrad ? 1.263 : 1.0) * (strided ? 0.833 : 1.0), load = pairs ? 1.6 : 1.0;
    const double rounds = (double)((ctas + (pairs ? 2 : 1) * sm_count - 1) / ((pairs ? 2 : 1) * sm_count));
    const double us = 1.0 + rounds * (2.76 + c.per_split * block * load) + (c.splits > 1 ? rounds * 128.0 * c.bn * 0.00017 * load + 0.98 : 0.0);
    return us;
}

// One launch for up to four pixel sets. In the passes of a model the two that later layers read stay on the CUDA cores (see
// launch_fp32_gemm), except the 3xTF32 ones that never ran there. The contraction is split over CTAs where the output alone
// does not fill the GPU and the epilogue is a plain sum (the output is then cleared first), except in the passes of a model: atomic
// sums come in any order, and one rounding more or less in an activation moves the gradients of a deep model by percents from one run
// to the next.
enum class Route { Any, TensorCores, PatchesOnly };  // by the rules below; on the tensor cores in models too; conv_patch.cu or CB_EUNSUPPORTED
int launch_gather(cb_ctx* ctx, GatherParams p, const PixelSet* sets, int nsets, Route route, const char* who) {
    const long long out_elems = (long long)p.OUTC * p.OHH * p.OWW;
    if ((long long)p.C * p.H * p.W >= (1LL << 29) || out_elems >= (1LL << 31) || (long long)p.C * p.w_ch >= (1LL << 31))
        return fail(ctx, CB_EUNSUPPORTED, std::string(who) + ": an image or filter of more than 2^29 values");
    bool may_split = !ctx->deterministic && !ctx->model_pass && !p.ep.scale && !p.ep.relu;
    int most = 0;
    for (int i = 0; i < nsets; ++i) most = sets[i].K > most ? sets[i].K : most;
    const long long I = (long long)p.N * sets[0].UH * sets[0].UW * nsets;
    const bool on_tensor_cores = (!ctx->model_pass || route == Route::TensorCores) && split::worth_it(I, p.OUTC, most, 1, kLeastConv);
    if (on_tensor_cores && !ctx->model_pass && nsets <= kMaxSets) {
        std::memcpy(p.sets, sets, nsets * sizeof(PixelSet));
        PatchPlan plan{};
        void* pieces = nullptr;
        if (plan_patch(ctx, p, nsets, may_split, plan) && plan.us < 0.88 * gather_us(ctx->sm_count, I, p.OUTC, (most + split::kBK - 1) / split::kBK, may_split, p, sets)) {
            // In place of the one-pass form pieces lie in the workspace, where that would pack its filter: on every stream, and in a capture whose
            // call was made before. (Elsewhere than on the context's own stream it would go to that form, whose blocks no call has grown.) The
            // gathers need no scratch, so what could go there must not depend on the workspace.
            if (route != Route::PatchesOnly) pieces = filter_pieces(ctx, plan.filter_bytes);
            else if (plan.filter_bytes <= kFilterPieces && ensure_workspace(ctx, plan.filter_bytes) == CB_OK) pieces = ctx->workspace;
        }
        if (pieces) {
            const cudaError_t e = launch_patch(ctx, plan, pieces);
            if (e != cudaSuccess) return check_cuda(ctx, e, who);
            ctx->launches += 2;
            ctx->last_kernel = "umma_fp32";
            return CB_OK;
        }
    }
    if (route == Route::PatchesOnly) return CB_EUNSUPPORTED;
    simt::Choice c{};
    split::Choice sc{};
    if (on_tensor_cores) sc = split::choose_shape(ctx->sm_count, I, p.OUTC, (most + split::kBK - 1) / split::kBK, 1, may_split, split::kGather);
    else c = simt::choose_tile(ctx->sm_count, I, p.OUTC, (most + simt::kBK - 1) / simt::kBK, 1, may_split);
    p.splits = on_tensor_cores ? sc.splits : c.splits;
    p.per_split = on_tensor_cores ? sc.per_split : c.per_split;
    p.atomic_out = p.splits > 1 ? 1 : 0;
    if (p.atomic_out && !p.ep.accumulate) {
        const int rc = clear_output(ctx, p.Out, out_elems, p.out_batch, p.N, 0, 1, who);
        if (rc != CB_OK) return rc;
    }
    bool mask = true;
    for (int i = 0; i < nsets; ++i) mask = mask && sets[i].TH <= kMaskTaps && sets[i].TW <= kMaskTaps;
    for (int first = 0; first < nsets; first += kMaxSets) {
        const int count = nsets - first < kMaxSets ? nsets - first : kMaxSets;
        long long pixels = 0;
        for (int i = 0; i < count; ++i) {
            p.sets[i] = sets[first + i];
            const long long n = (long long)p.N * p.sets[i].UH * p.sets[i].UW;
            pixels = n > pixels ? n : pixels;
        }
        if (pixels == 0) continue;
        cudaError_t e = on_tensor_cores ? launch_split_gather(ctx, p, sc, mask, pixels, count) : simt::with_tile(c.tile, [&](auto tile) {
            typedef decltype(tile) T;
            auto kernel = mask ? conv_gather_simt<T, true> : conv_gather_simt<T, false>;
            cudaError_t er = raise_dynamic_smem_once(kernel, ctx->device, ctx->max_smem_optin, nullptr);
            if (er != cudaSuccess) return er;
            const long long gx = (pixels + T::BM - 1) / T::BM, gy = (p.OUTC + T::BN - 1) / T::BN, gz = (long long)count * c.splits;
            if (gx > 0x7fffffffLL || gy > 65535 || gz > 65535) return cudaErrorInvalidConfiguration;
            er = launch_dep(ctx, kernel, dim3((unsigned)gx, (unsigned)gy, (unsigned)gz), dim3(T::NT), T::kSmem, p);
            return er == cudaSuccess ? cudaGetLastError() : er;
        });
        if (e != cudaSuccess) return check_cuda(ctx, e, who);
        ctx->launches += 1;
    }
    ctx->last_kernel = on_tensor_cores ? "umma_fp32" : "simt_fp32";
    return CB_OK;
}

int fp32_conv_fwd(cb_ctx* ctx, const float* W, const float* X, float* Y, const ConvGeo& g, const ConvEpilogue& ep, Route route, const char* who) {
    GatherParams p{};
    p.In = X; p.in_batch = g.x_batch; p.C = g.IC; p.H = g.IH; p.W = g.IW;
    p.Wt = W; p.w_ch = g.FH * g.FW; p.w_out = g.IC * g.FH * g.FW; p.FW = g.FW;
    p.Out = Y; p.out_batch = g.y_batch; p.OUTC = g.OC; p.OHH = g.OH; p.OWW = g.OW;
    p.N = g.N; p.sgn = 1; p.ep = ep;
    const PixelSet s{g.OH, g.OW, g.sH, -g.pH, g.sW, -g.pW, 0, 1, 0, 1, g.FH, g.FW, 0, 1, 0, 1, g.IC * g.FH * g.FW};
    return launch_gather(ctx, p, &s, 1, route, who);
}

int fp32_conv_dgrad(cb_ctx* ctx, const float* W, const float* dY, float* dX, const ConvGeo& g, int accumulate, Route route, const char* who) {
    GatherParams p{};
    p.In = dY; p.in_batch = g.y_batch; p.C = g.OC; p.H = g.OH; p.W = g.OW;
    p.Wt = W; p.w_ch = g.IC * g.FH * g.FW; p.w_out = g.FH * g.FW; p.FW = g.FW;
    p.Out = dX; p.out_batch = g.x_batch; p.OUTC = g.IC; p.OHH = g.IH; p.OWW = g.IW;
    p.N = g.N; p.sgn = -1; p.ep.accumulate = accumulate; p.tap_major = 1;
    std::vector<PixelSet> sets;
    for (int a = 0; a < g.sH; ++a)
        for (int b = 0; b < g.sW; ++b) {
            // pixels ih = a + sH*u: tap fh reaches them from row (ih + pH - fh) / sH when sH divides it
            PixelSet s{};
            if (a >= g.IH || b >= g.IW) continue;
            s.UH = (g.IH - a + g.sH - 1) / g.sH; s.UW = (g.IW - b + g.sW - 1) / g.sW;
            const int f0 = (a + g.pH) % g.sH, e0 = (b + g.pW) % g.sW;
            s.TH = f0 < g.FH ? (g.FH - 1 - f0) / g.sH + 1 : 0;
            s.TW = e0 < g.FW ? (g.FW - 1 - e0) / g.sW + 1 : 0;
            s.hs = 1; s.hb = (a + g.pH - f0) / g.sH; s.ws = 1; s.wb = (b + g.pW - e0) / g.sW;
            s.oh0 = a; s.ohs = g.sH; s.ow0 = b; s.ows = g.sW;
            s.wt0 = f0; s.wts = g.sH; s.wu0 = e0; s.wus = g.sW;
            s.K = g.OC * s.TH * s.TW;
            sets.push_back(s);
        }
    return launch_gather(ctx, p, sets.data(), (int)sets.size(), route, who);
}

int fp32_conv_wgrad(cb_ctx* ctx, const float* dY, const float* X, float* dW, const ConvGeo& g, int accumulate, const char* who) {
    WgradParams p{};
    p.X = X; p.dY = dY; p.dW = dW; p.g = g;
    const long long I = (long long)g.IC * g.FH * g.FW, pixels = (long long)g.N * g.OH * g.OW;
    if (I >= (1LL << 31) || pixels >= (1LL << 31) - 64 || (long long)g.IC * g.IH * g.IW >= (1LL << 29))
        return fail(ctx, CB_EUNSUPPORTED, std::string(who) + ": more than 2^31 pixels or filter values");
    const bool mask = g.FH <= kMaskTaps && g.FW <= kMaskTaps;
    p.I = (int)I; p.pixels = (int)pixels;
    // Not in a model's backward pass, on whichever stream (cbt_set_wgrad_streams moves launches, it does not choose kernels): a CTA of
    // conv_wgrad_split holds an SM, which the stream beside it would miss (ResNet-50 on 16 x 16 images, batch 78: 2300 us a step
    // against 2263)
    const bool on_tensor_cores = !ctx->model_pass && split::worth_it(I, g.OC, pixels, 1, kLeastConv);
    simt::Choice c{};
    split::Choice sc{};
    if (on_tensor_cores) sc = split::choose_shape(ctx->sm_count, I, g.OC, (pixels + split::kBK - 1) / split::kBK, 1, !ctx->deterministic, split::kWgrad);
    else c = simt::choose_tile(ctx->sm_count, I, g.OC, (pixels + simt::kBK - 1) / simt::kBK, 1, !ctx->deterministic);
    p.splits = on_tensor_cores ? sc.splits : c.splits;
    p.per_split = on_tensor_cores ? sc.per_split : c.per_split;
    p.mode = p.splits > 1 ? 2 : (accumulate ? 1 : 0);
    if (p.mode == 2 && !accumulate) {
        const int rc = clear_output(ctx, dW, I * g.OC, I * g.OC, 1, 0, 1, who);
        if (rc != CB_OK) return rc;
    }
    cudaError_t e = on_tensor_cores ? launch_split_wgrad(ctx, p, sc, mask) : simt::with_tile(c.tile, [&](auto tile) {
        typedef decltype(tile) T;
        auto kernel = mask ? conv_wgrad_simt<T, true> : conv_wgrad_simt<T, false>;
        cudaError_t er = raise_dynamic_smem_once(kernel, ctx->device, ctx->max_smem_optin, nullptr);
        if (er != cudaSuccess) return er;
        const long long gx = (I + T::BM - 1) / T::BM, gy = (g.OC + T::BN - 1) / T::BN;
        if (gy > 65535 || c.splits > 65535) return cudaErrorInvalidConfiguration;
        er = launch_dep(ctx, kernel, dim3((unsigned)gx, (unsigned)gy, (unsigned)c.splits), dim3(T::NT), T::kSmem, p);
        return er == cudaSuccess ? cudaGetLastError() : er;
    });
    if (e != cudaSuccess) return check_cuda(ctx, e, who);
    ctx->launches += 1;
    ctx->last_kernel = on_tensor_cores ? "umma_fp32" : "simt_fp32";
    return CB_OK;
}

int make_geo(cb_ctx* ctx, ConvGeo& g, int N, int IC, int IH, int IW, int OC, int FH, int FW, int sH, int sW, int pH,
             int pW, long long x_batch, long long y_batch, const char* who) {
    if (N < 0 || IC < 0 || OC < 0 || IH < 0 || IW < 0) return fail(ctx, CB_EINVAL, std::string(who) + ": negative extent");
    if (FH < 1 || FW < 1 || sH < 1 || sW < 1 || pH < 0 || pW < 0)
        return fail(ctx, CB_EINVAL, std::string(who) + ": filter, stride must be >= 1 and padding >= 0");
    if (IH + 2 * pH < FH || IW + 2 * pW < FW) return fail(ctx, CB_EINVAL, std::string(who) + ": filter larger than the padded input");
    g = ConvGeo{N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, (IH - FH + 2 * pH) / sH + 1, (IW - FW + 2 * pW) / sW + 1, 0, 0};
    const long long x_dense = (long long)IC * IH * IW, y_dense = (long long)OC * g.OH * g.OW;
    if ((x_batch && x_batch < x_dense) || (y_batch && y_batch < y_dense))
        return fail(ctx, CB_EINVAL, std::string(who) + ": batch stride smaller than one image");
    g.x_batch = x_batch ? x_batch : x_dense;
    g.y_batch = y_batch ? y_batch : y_dense;
    return CB_OK;
}

}  // namespace

}  // namespace cb

using namespace cb;

// Whether the TF32 kernels take the maps' width. Filters their one-pass 3xTF32 form does not take run at fp32 accuracy on the tensor
// cores, in models too: three TF32 passes into temporaries took 137 us where that takes 14 (64 -> 128, stride 2, 64 maps of 16 x 16),
// 41 against 11 (96 -> 96, 9 of 16 x 16).
static bool tf32_width(const ConvGeo& g) {
    const int w = g.sW == 2 ? g.IW / 2 : g.IW;
    return g.FH <= 3 && g.FW <= 3 && (w == 8 || w == 16 || w == 32);
}
// Stride-2 3x3 layers of 3xTF32 whose passes run at fp32 accuracy: the one-pass form pays for a phase split and lo parts through memory. us,
// one pass / fp32: 32 -> 64 at 32 x 32, batch 128: forward 37 / 18, data gradient 30.2 / 25.8, weight gradient 34 / 26. Over 53 layers of 3 to 128
// channels, 16 x 16 to 64 x 64, 1.38, 1.76 and 1.46 times as fast with every layer of 2^22 multiplications on there; below 2^26 both are a few
// launches. What stays in the one-pass form: few input channels on many pixels forward, where each of the gather's outputs has little to
// sum (16 channels, more than 2^15 pixels: 0.81 to 0.97, or 1.1 to 1.6 for the 17 to 32 outputs that fill its narrowest tile); data
// gradients of up to 16 channels (0.81 to 1.22), from many pixels (2^15 on: 0.45 to 1.09; 2^14 on from up to 16 channels to more than 32:
// 0.98), and those that conv_patch.cu does not take.
enum class Pass { Forward, DataGradient, WeightGradient };
static bool x3_at_fp32(const ConvGeo& g, Pass pass) {
    if ((double)g.N * g.OH * g.OW >= (double)(1LL << 30) || (double)g.IC * g.IH * g.IW >= (double)(1LL << 28) || (double)g.OC * g.OH * g.OW >= (double)(1LL << 28))
        return false;  // 32-bit indexes
    const long long pixels = (long long)g.N * g.OH * g.OW;
    if (pass == Pass::Forward && g.IC <= 16 && pixels > (1 << 15) && (g.OC <= 16 || g.OC > 32)) return false;
    if (pass == Pass::DataGradient && (g.IC <= 16 || pixels > (1 << 15) || (pixels > (1 << 14) && g.IC > 32 && g.OC <= 16))) return false;
    return g.sH == 2 && g.sW == 2 && g.FH == 3 && g.FW == 3 && (double)pixels * g.OC * g.IC * 9.0 >= (double)(1LL << 26);
}

static int conv_fwd_impl(cb_ctx* ctx, const float* W, const float* X, float* Y, int N, int IC, int IH, int IW, int OC, int FH,
                         int FW, int sH, int sW, int pH, int pW, const cb_epilogue* cep, const char* who) {
    if (int rc_enter = enter(ctx)) return rc_enter;
    ConvEpilogue ep{};
    long long xb = 0, yb = 0;
    if (cep) {
        ep.bias = cep->bias; ep.scale = cep->scale; ep.shift = cep->shift;
        ep.per_position = cep->per_position ? 1 : 0; ep.relu = cep->relu ? 1 : 0; ep.accumulate = cep->accumulate ? 1 : 0;
        xb = cep->x_batch_stride; yb = cep->y_batch_stride;
        if ((ep.scale == nullptr) != (ep.shift == nullptr)) return fail(ctx, CB_EINVAL, std::string(who) + ": scale and shift go together");
    }
    ConvGeo g;
    int rc = make_geo(ctx, g, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, xb, yb, who);
    if (rc != CB_OK) return rc;
    const long long npix = (long long)N * g.OH * g.OW;
    if (npix == 0 || OC == 0) return CB_OK;
    if (!W || !X || !Y) return fail(ctx, CB_EINVAL, std::string(who) + ": null operand");
    const bool x3 = ctx->math == CB_MATH_3XTF32;
    if (ctx->math != CB_MATH_FP32 && !(x3 && !ctx->model_pass && x3_at_fp32(g, Pass::Forward))) {
        rc = umma_conv_fwd(ctx, W, X, Y, ep, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, false, xb, yb, x3);
        if (rc != CB_EUNSUPPORTED) return rc == CB_OK ? finish(ctx, who) : rc;
    }
    rc = fp32_conv_fwd(ctx, W, X, Y, g, ep, x3 && tf32_width(g) ? Route::TensorCores : Route::Any, who);
    return rc == CB_OK ? finish(ctx, who) : rc;
}

static int conv_dgrad_impl(cb_ctx* ctx, const float* W, const float* dY, float* dX, int N, int IC, int IH, int IW, int OC,
                           int FH, int FW, int sH, int sW, int pH, int pW, int accumulate, long long dy_batch, long long dx_batch,
                           const char* who) {
    if (int rc_enter = enter(ctx)) return rc_enter;
    ConvGeo g;
    int rc = make_geo(ctx, g, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, dx_batch, dy_batch, who);
    if (rc != CB_OK) return rc;
    const long long npix = (long long)N * IH * IW;
    if (npix == 0 || IC == 0) return CB_OK;
    if (!W || !dY || !dX) return fail(ctx, CB_EINVAL, std::string(who) + ": null operand");
    ConvEpilogue ep{};
    ep.accumulate = accumulate ? 1 : 0;
    const bool x3 = ctx->math == CB_MATH_3XTF32;
    if (x3 && !ctx->model_pass && x3_at_fp32(g, Pass::DataGradient)) {
        rc = fp32_conv_dgrad(ctx, W, dY, dX, g, accumulate ? 1 : 0, Route::PatchesOnly, who);
        if (rc != CB_EUNSUPPORTED) return rc == CB_OK ? finish(ctx, who) : rc;
    }
    if (ctx->math != CB_MATH_FP32) {
        rc = umma_conv_fwd(ctx, W, dY, dX, ep, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, true, dy_batch, dx_batch, x3);
        if (rc != CB_EUNSUPPORTED) return rc == CB_OK ? finish(ctx, who) : rc;
    }
    rc = fp32_conv_dgrad(ctx, W, dY, dX, g, accumulate ? 1 : 0, x3 && tf32_width(g) ? Route::TensorCores : Route::Any, who);
    return rc == CB_OK ? finish(ctx, who) : rc;
}

extern "C" {

int cb_conv_fwd(cb_ctx* ctx, const float* W, const float* X, float* Y, const float* bias, int N, int IC, int IH,
                int IW, int OC, int FH, int FW, int sH, int sW, int pH, int pW, int relu) {
    cb_epilogue ep{};
    ep.bias = bias;
    ep.relu = relu;
    return conv_fwd_impl(ctx, W, X, Y, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, &ep, "cb_conv_fwd");
}

int cb_conv_fwd_ex(cb_ctx* ctx, const float* W, const float* X, float* Y, int N, int IC, int IH, int IW, int OC, int FH,
                   int FW, int sH, int sW, int pH, int pW, const cb_epilogue* ep) {
    return conv_fwd_impl(ctx, W, X, Y, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, ep, "cb_conv_fwd_ex");
}

int cb_conv_dgrad(cb_ctx* ctx, const float* W, const float* dY, float* dX, int N, int IC, int IH, int IW, int OC,
                  int FH, int FW, int sH, int sW, int pH, int pW) {
    return conv_dgrad_impl(ctx, W, dY, dX, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, 0, 0, 0, "cb_conv_dgrad");
}

int cb_conv_dgrad_ex(cb_ctx* ctx, const float* W, const float* dY, float* dX, int N, int IC, int IH, int IW, int OC,
                     int FH, int FW, int sH, int sW, int pH, int pW, int accumulate, long long dy_batch_stride,
                     long long dx_batch_stride) {
    return conv_dgrad_impl(ctx, W, dY, dX, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, accumulate, dy_batch_stride,
                           dx_batch_stride, "cb_conv_dgrad_ex");
}

int cb_conv_cache_filters(cb_ctx* ctx, int on) {
    if (!ctx) return CB_EINVAL;
    ctx->filter_cache_on = on ? 1 : 0;
    ctx->filter_version += 1;
    return CB_OK;
}

int cb_filters_changed(cb_ctx* ctx) {
    if (int rc_enter = enter(ctx)) return rc_enter;
    const int rc = filter_cache_repack_all(ctx);
    return rc == CB_OK ? finish(ctx, "cb_filters_changed") : rc;
}

}  // extern "C"

// Weight gradients that the TF32 kernel would cut into several launches (filters beyond its accumulator) run in one at fp32 accuracy
// where that takes less: 6 us + 45 us for 10^9 multiplications against 6.5 us a launch (TF32) or 8 us and 9 for the lo parts (3xTF32).
// 128 -> 128 3x3, 4 maps of 16 x 16: 25.9 us TF32, 32.5 3xTF32, 7.9 here; 330 -> 48 1x1, 64 of 8 x 8: 14.6 TF32, 7.9 here;
// 288 -> 48 1x1, 64 of 16 x 16: 14.1 TF32, 18.0 here. Of 140 other layers of either mode one is slower for it (16 -> 176 1x1, 15 of 32 x 32:
// 11.3 TF32, 12.9 here).
static bool wgrad_at_fp32(const ConvGeo& g, bool x3) {
    const int launches = umma_wgrad_launches(g.IC, g.OC, g.FH, g.FW);
    const double fmas = (double)g.N * g.OH * g.OW * g.OC * g.IC * g.FH * g.FW;
    return g.sH == 1 && g.sW == 1 && launches > 1 && fmas >= (double)kLeastConv && 6.0 + 45e-9 * fmas < (x3 ? 9.0 + 8.0 * launches : 6.5 * launches);
}

static int conv_wgrad_impl(cb_ctx* ctx, const float* dY, const float* X, float* dW, int N, int IC, int IH, int IW, int OC,
                           int FH, int FW, int sH, int sW, int pH, int pW, int accumulate, long long dy_batch, long long x_batch,
                           const char* who) {
    if (int rc_enter = enter(ctx)) return rc_enter;
    ConvGeo g;
    int rc = make_geo(ctx, g, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, x_batch, dy_batch, who);
    if (rc != CB_OK) return rc;
    if (OC == 0 || IC == 0) return CB_OK;
    if (!dW) return fail(ctx, CB_EINVAL, std::string(who) + ": null operand");
    const size_t wbytes = (size_t)OC * IC * FH * FW * sizeof(float);
    if ((long long)N * g.OH * g.OW == 0) {
        if (!accumulate) {
            cudaError_t e = cudaMemsetAsync(dW, 0, wbytes, ctx->stream);
            if (e != cudaSuccess) return check_cuda(ctx, e, "convolution weight gradient: clear");
        }
        return finish(ctx, who);
    }
    if (!dY || !X) return fail(ctx, CB_EINVAL, std::string(who) + ": null operand");
    // 3xTF32: the products dY_hi X_hi, dY_hi X_lo, dY_lo X_hi in one launch that walks the pixels three times
    const bool x3 = ctx->math == CB_MATH_3XTF32;
    // (models keep the kernel that leaves half the SMs to the stream beside it: a DenseNet-100 step took 3571 us with its widest layers
    // here, 3561 without; without such streams too, or a gradient's accuracy would depend on their number)
    if (ctx->math != CB_MATH_FP32 && (ctx->deterministic || ctx->model_pass || !((x3 && x3_at_fp32(g, Pass::WeightGradient)) || wgrad_at_fp32(g, x3)))) {
        rc = umma_conv_wgrad(ctx, dY, X, dW, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, accumulate, dy_batch, x_batch, x3);
        if (rc == CB_OK && x3) ctx->last_kernel = "umma_3xtf32";
        if (rc != CB_EUNSUPPORTED) return rc == CB_OK ? finish(ctx, who) : rc;
    }
    rc = fp32_conv_wgrad(ctx, dY, X, dW, g, accumulate ? 1 : 0, who);
    return rc == CB_OK ? finish(ctx, who) : rc;
}

extern "C" {

int cb_conv_wgrad(cb_ctx* ctx, const float* dY, const float* X, float* dW, int N, int IC, int IH, int IW, int OC,
                  int FH, int FW, int sH, int sW, int pH, int pW, int accumulate) {
    return conv_wgrad_impl(ctx, dY, X, dW, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, accumulate, 0, 0, "cb_conv_wgrad");
}

int cb_conv_wgrad_ex(cb_ctx* ctx, const float* dY, const float* X, float* dW, int N, int IC, int IH, int IW, int OC,
                     int FH, int FW, int sH, int sW, int pH, int pW, int accumulate, long long dy_batch_stride,
                     long long x_batch_stride) {
    return conv_wgrad_impl(ctx, dY, X, dW, N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, accumulate, dy_batch_stride,
                           x_batch_stride, "cb_conv_wgrad_ex");
}

}  // extern "C"
