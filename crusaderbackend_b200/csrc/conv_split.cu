// The three convolution passes at fp32 accuracy on the tensor cores: the gathers of conv_simt.cu (any filter size, stride and padding)
// feeding the body of split_core.cuh. conv_simt.cu decides which launches come here.
#include "conv_gather.cuh"
#include "split_core.cuh"

namespace cb {

using namespace gather;

namespace {

using split::kBK;

// Forward and data gradient: rows are pixels, columns output channels.
template <class S, bool MASK>
struct SplitGather {
    static constexpr split::Kind kP = split::MN, kQ = split::K;
    static constexpr bool kTable = true;
    typedef split::ShareP<S, kP> SP;
    typedef split::ShareQ<S, kQ> SQ;
    const GatherParams& p;
    const PixelSet& s;
    TapK* table;             // [kLoaders]
    int* woffs;              // [kLoaders]: TapK::woff, two neighbours in one load without bank conflicts
    const float* img;        // a loader thread's pixel: its image, its taps, offset of the first tap
    Position at;
    int base;
    long long i0, pixels;
    int j0, block0, part;
    __device__ __forceinline__ void prepare(int t, int tid) {
        const TapK e = tap_of<MASK>(p, s, (block0 + t) * kBK + tid);
        table[tid] = e;
        woffs[tid] = e.woff;
    }
    __device__ __forceinline__ void load(int t, int tid, float (&vp)[SP::kValues], float (&vq)[SQ::kValues]) {
        const TapK* tab = table + t % (S::kLoaders / kBK) * kBK;
#pragma unroll
        for (int x = 0; x < SP::kValues; ++x) {
            const TapK q = tab[SP::k(tid, x)];
            const bool ok = tap_inside<MASK>(at, q.bits, p.H, p.W) && (MASK || q.woff >= 0);
            vp[x] = split::load_if(img + (base + q.off), ok);
        }
        const int2 w = *reinterpret_cast<const int2*>(woffs + t % (S::kLoaders / kBK) * kBK + SQ::k(tid, 0));
        const int w0 = w.x, w1 = w.y;
#pragma unroll
        for (int u = 0; u < SQ::kUnits; ++u) {
            const float* row = p.Wt + (long long)min(j0 + SQ::row(tid, u), p.OUTC - 1) * p.w_out;
            vq[2 * u] = split::load_if(row + w0, w0 >= 0);
            vq[2 * u + 1] = split::load_if(row + w1, w1 >= 0);
        }
    }
    template <bool LOW>
    __device__ __forceinline__ void store(int row, int first, int n, uint32_t mine) const {
        if (i0 + row >= pixels) return;
        float* out;
        const int place = output_of(p, s, i0 + row, out), plane = p.OHH * p.OWW, j = j0 + first;
        const bool bias = p.ep.bias && part == 0;
        split::store_columns<LOW>(out + (long long)j * plane, plane, min(n, p.OUTC - j), mine,
                      p.atomic_out ? !bias : !p.ep.scale && !p.ep.bias && !p.ep.relu, p.atomic_out || (p.ep.accumulate && !p.ep.relu && !p.ep.scale && !p.ep.bias),
                      [&](int c, float y, const float* dst) {
                          if (p.atomic_out) return y + p.ep.bias[j + c];
                          return apply_epilogue(p.ep, y, j + c, (long long)(j + c) * plane + place, p.ep.accumulate ? *dst : 0.f);
                      });
    }
};

template <class S, bool MASK>
__global__ void __launch_bounds__(S::NT, S::kCtas) conv_gather_split(const __grid_constant__ GatherParams p, int* status) {
    extern __shared__ uint8_t smem[];
    __shared__ split::Barriers bars;
    __shared__ TapK table[S::kLoaders];
    __shared__ __align__(8) int woffs[S::kLoaders];
    const int set = blockIdx.z / p.splits, part = blockIdx.z - set * p.splits;
    const PixelSet& s = p.sets[set];
    SplitGather<S, MASK> src{p, s, table, woffs, p.In, Position{-(1 << 29), 0, 0u}, 0, (long long)blockIdx.x * S::BM, (long long)p.N * s.UH * s.UW,
                             (int)blockIdx.y * S::BN, part * p.per_split, part};
    const int blocks = min(p.per_split, (s.K + kBK - 1) / kBK - src.block0);
    // the grid is sized for the largest set; a share without a block has nothing to add, but a set without any product is still stored
    if (src.i0 >= src.pixels || (blocks <= 0 && part > 0)) return;
    const int tid = (int)threadIdx.x - 32 * S::kSumWarps;
    if (tid >= 0) {
        const long long i = src.i0 + split::ShareP<S, split::MN>::row(tid, 0);
        if (i < src.pixels) {
            src.at = input_of<MASK>(p, s, i, src.img);
            src.base = src.at.h0 * p.W + src.at.w0;
        }
    }
    split::run<S>(src, max(blocks, 1), smem, bars, nullptr, status);
}

// Weight gradient: rows are filter positions (ic, fh, fw), columns output channels, the contraction runs over the pixels.
template <class S, bool MASK>
struct SplitWgrad {
    static constexpr split::Kind kP = split::K, kQ = split::K;
    static constexpr bool kTable = true;
    typedef split::ShareP<S, kP> SP;
    typedef split::ShareQ<S, kQ> SQ;
    const WgradParams& p;
    // PixelK of kLoaders pixels, field by field: lanes read neighbouring pixels, entries of 32 bytes were 2- to 8-way bank conflicts
    // (shared memory was busy 1440 clocks of a block's 2640). 32 -> 64 channels, 32 x 32, stride 2, batch 128: 29.3 -> 24.0 us, with the
    // patches of put_p; 64 -> 64, 32 x 32, batch 128: 230 -> 208.
    longlong2* ys;           // [kLoaders / 2]
    long long* xs;           // [kLoaders]
    Position* at;            // [kLoaders]; MASK: only the masks, as words
    const TapI* rows;        // [BM]
    int i0, j0, block0, opix;
    __device__ __forceinline__ void prepare(int t, int tid) {
        const PixelK e = pixel_of<MASK>(p, (block0 + t) * kBK + tid);
        xs[tid] = e.x;
        reinterpret_cast<long long*>(ys)[tid] = e.y;
        if (MASK) reinterpret_cast<uint32_t*>(at)[tid] = e.at.mask;
        else at[tid] = e.at;
    }
    __device__ __forceinline__ void load(int t, int tid, float (&vp)[SP::kValues], float (&vq)[SQ::kValues]) {
        const int tab = t % (S::kLoaders / kBK) * kBK, k = tab + SP::k(tid, 0);
        const float* first = p.X + xs[k];
        Position here{0, 0, 0u};
        if (MASK) here.mask = reinterpret_cast<const uint32_t*>(at)[k];
        else here = at[k];
#pragma unroll
        for (int x = 0; x < SP::kValues; ++x) {
            const TapI w = rows[SP::row(tid, x)];
            const bool ok = tap_inside<MASK>(here, w.bits, p.g.IH, p.g.IW) && (MASK || w.off >= 0);
            vp[x] = split::load_if(first + w.off, ok);
        }
        const longlong2 y = ys[(tab + SQ::k(tid, 0)) / 2];
        const long long y0 = y.x, y1 = y.y;
#pragma unroll
        for (int u = 0; u < SQ::kUnits; ++u) {
            const float* row = p.dY + (long long)min(j0 + SQ::row(tid, u), p.g.OC - 1) * opix;
            vq[2 * u] = split::load_if(row + y0, y0 >= 0);
            vq[2 * u + 1] = split::load_if(row + y1, y1 >= 0);
        }
    }
    template <bool LOW>
    __device__ __forceinline__ void store(int row, int first, int n, uint32_t mine) const {
        const int i = i0 + row, j = j0 + first;
        if (i >= p.I) return;
        split::store_columns<LOW>(p.dW + (long long)j * p.I + i, p.I, min(n, p.g.OC - j), mine, true, p.mode != 0, [](int, float y, const float*) { return y; });
    }
};

template <class S, bool MASK>
__global__ void __launch_bounds__(S::NT, S::kCtas) conv_wgrad_split(const __grid_constant__ WgradParams p, int* status) {
    extern __shared__ uint8_t smem[];
    __shared__ split::Barriers bars;
    __shared__ __align__(16) float patches[split::ShareP<S, split::K>::kPatches];
    __shared__ longlong2 ys[S::kLoaders / 2];
    __shared__ long long xs[S::kLoaders];
    __shared__ Position at[MASK ? (S::kLoaders + 2) / 3 : S::kLoaders];
    __shared__ TapI rows[S::BM];
    const int i0 = blockIdx.x * S::BM;
    for (int e = threadIdx.x; e < S::BM; e += S::NT) rows[e] = row_of<MASK>(p, i0 + e);  // read behind the barrier of run()
    SplitWgrad<S, MASK> src{p, ys, xs, at, rows, i0, (int)blockIdx.y * S::BN, (int)blockIdx.z * p.per_split, p.g.OH * p.g.OW};
    split::run<S>(src, min(p.per_split, (p.pixels + kBK - 1) / kBK - src.block0), smem, bars, patches, status);
}

template <class F>
cudaError_t with_shape(int bn, F f) {
    return bn == 128 ? f(split::Shape<128>{}) : bn == 64 ? f(split::Shape<64>{}) : f(split::Shape<32>{});
}

}  // namespace

cudaError_t launch_split_gather(cb_ctx* ctx, const GatherParams& p, const split::Choice& c, bool mask, long long pixels, int sets) {
    return with_shape(c.bn, [&](auto shape) {
        typedef decltype(shape) S;
        auto kernel = mask ? conv_gather_split<S, true> : conv_gather_split<S, false>;
        cudaError_t e = raise_dynamic_smem_once(kernel, ctx->device, ctx->max_smem_optin, nullptr);
        if (e != cudaSuccess) return e;
        const long long gx = (pixels + S::BM - 1) / S::BM, gy = (p.OUTC + S::BN - 1) / S::BN, gz = (long long)sets * c.splits;
        if (gx > 0x7fffffffLL || gy > 65535 || gz > 65535) return cudaErrorInvalidConfiguration;
        e = launch_dep(ctx, kernel, dim3((unsigned)gx, (unsigned)gy, (unsigned)gz), dim3(S::NT), (size_t)S::kSmem, p, ctx->d_status);
        return e == cudaSuccess ? cudaGetLastError() : e;
    });
}

cudaError_t launch_split_wgrad(cb_ctx* ctx, const WgradParams& p, const split::Choice& c, bool mask) {
    return with_shape(c.bn, [&](auto shape) {
        typedef decltype(shape) S;
        auto kernel = mask ? conv_wgrad_split<S, true> : conv_wgrad_split<S, false>;
        cudaError_t e = raise_dynamic_smem_once(kernel, ctx->device, ctx->max_smem_optin, nullptr);
        if (e != cudaSuccess) return e;
        const long long gx = (p.I + S::BM - 1) / S::BM, gy = (p.g.OC + S::BN - 1) / S::BN;
        if (gy > 65535 || c.splits > 65535) return cudaErrorInvalidConfiguration;
        e = launch_dep(ctx, kernel, dim3((unsigned)gx, (unsigned)gy, (unsigned)c.splits), dim3(S::NT), (size_t)S::kSmem, p, ctx->d_status);
        return e == cudaSuccess ? cudaGetLastError() : e;
    });
}

}  // namespace cb
