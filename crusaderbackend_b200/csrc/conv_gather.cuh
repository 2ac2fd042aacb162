// Index arithmetic of a convolution whose operands are gathered element by element, shared by the fp32 kernels on the CUDA cores
// (conv_simt.cu) and on the tensor cores (conv_split.cu).
#pragma once
#include "cb_internal.h"

namespace cb {
namespace gather {

struct ConvGeo {
    int N, IC, IH, IW, OC, FH, FW, sH, sW, pH, pW, OH, OW;
    long long x_batch, y_batch;  // elements between consecutive images of the input-side / output-side tensor
};

__device__ __forceinline__ float apply_epilogue(const ConvEpilogue& ep, float v, int oc, long long pos_idx, float old) {
    if (ep.scale) {
        const long long si = ep.per_position ? pos_idx : (long long)oc;
        v = fmaf(v, ep.scale[si], ep.shift[si]);
    }
    if (ep.bias) v += ep.bias[oc];
    if (ep.accumulate) v += old;
    if (ep.relu) v = fmaxf(v, 0.f);
    return v;
}

// ---- forward and data gradient as D[pixel][channel] = sum_k In(pixel, k) * W(channel, k), k = (input channel, tap)
//
// A launch covers a set of output pixels on a regular grid: pixel (u, v) of an image reads In at row hs*u + hb + sgn*th
// and column ws*v + wb + sgn*tw for its taps (th, tw), and is written at row oh0 + ohs*u, column ow0 + ows*v. The forward
// pass is one such set (sgn = +1). The data gradient of a strided convolution is sH x sW sets, one for each phase of the
// input row and column: only every sH-th tap reaches a pixel of a phase, so a set's contraction holds just those taps
// (sgn = -1) and no products with structural zeros are formed.
struct PixelSet {
    int UH, UW;              // pixels of an image in the set
    int hs, hb, ws, wb;      // first tap's input row / column
    int oh0, ohs, ow0, ows;  // output row / column
    int TH, TW;              // taps
    int wt0, wts, wu0, wus;  // filter row of tap th: wt0 + wts*th; filter column: wu0 + wus*tw
    int K;                   // channels * TH * TW
};
constexpr int kMaxSets = 4;  // pixel sets of one launch: the four phases of a stride-2 data gradient
struct GatherParams {
    const float* In; long long in_batch; int C, H, W;       // the tensor the taps read
    const float* Wt; int w_ch, w_out, FW;                    // filter strides: contraction channel, output channel; width
    float* Out; long long out_batch; int OUTC, OHH, OWW;     // output channels, rows, columns
    int N, sgn;
    int splits, per_split, atomic_out, tap_major;
    ConvEpilogue ep;
    PixelSet sets[kMaxSets]; // blockIdx.z = set * splits + split
};

// Which taps of a pixel lie inside the tensor. Filters of up to 15 x 15 taps keep it as one word, tap rows in the low half
// and tap columns in the high half, and a tap's test is (mask & bits) == bits; larger ones compare coordinates.
constexpr int kMaskTaps = 15;
__device__ __forceinline__ uint32_t range_mask(int first, int sgn, int count, int extent) {
    // taps t in [0, count) with 0 <= first + sgn * t < extent
    int lo = sgn > 0 ? -first : first - extent + 1, hi = sgn > 0 ? extent - first : first + 1;
    lo = min(max(lo, 0), count);
    hi = min(max(hi, 0), count);
    return hi > lo ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
}
struct Position {
    int h0, w0;      // coordinates of the first tap
    uint32_t mask;
};
template <bool MASK>
__device__ __forceinline__ bool tap_inside(const Position& at, uint32_t bits, int H, int W) {
    if (MASK) return (at.mask & bits) == bits;
    return (unsigned)(at.h0 + ((int)bits >> 16)) < (unsigned)H && (unsigned)(at.w0 + (short)bits) < (unsigned)W;
}
template <bool MASK>
__device__ __forceinline__ uint32_t tap_bits(int th, int tw, int sgn) {
    if (MASK) return (1u << th) | (1u << (16 + tw));
    return ((uint32_t)(sgn * th) << 16) | ((uint32_t)(sgn * tw) & 0xffffu);
}

// What the copies of one k need: offset from a pixel's first tap, tap test, offset in the filter (-1: past the end).
struct TapK {
    int off;
    uint32_t bits;
    int woff, pad;
};
template <bool MASK>
__device__ __forceinline__ TapK tap_of(const GatherParams& p, const PixelSet& s, int k) {
    TapK e{0, 0xffffffffu, -1, 0};
    if (k < s.K) {
        const int taps = s.TH * s.TW;
        // the order in which a pixel's products are added: channel by channel, or (data gradient) tap by tap
        const int c = p.tap_major ? k % p.C : k / taps, r = p.tap_major ? k / p.C : k - c * taps;
        const int th = r / s.TW, tw = r - th * s.TW;
        e.off = (c * p.H + p.sgn * th) * p.W + p.sgn * tw;
        e.bits = tap_bits<MASK>(th, tw, p.sgn);
        e.woff = c * p.w_ch + (s.wt0 + s.wts * th) * p.FW + s.wu0 + s.wus * tw;
    }
    return e;
}
// Pixel i of a set: its image in the input and where its first tap lies; its place in an output plane and in the output.
template <bool MASK>
__device__ __forceinline__ Position input_of(const GatherParams& p, const PixelSet& s, long long i, const float*& img) {
    const int per = s.UH * s.UW;
    const int n = (int)(i / per), r = (int)(i - (long long)n * per);
    const int u = r / s.UW, v = r - u * s.UW;
    img = p.In + (long long)n * p.in_batch;
    Position at{s.hs * u + s.hb, s.ws * v + s.wb, 0u};
    if (MASK) at.mask = range_mask(at.h0, p.sgn, s.TH, p.H) | (range_mask(at.w0, p.sgn, s.TW, p.W) << 16);
    return at;
}
__device__ __forceinline__ int output_of(const GatherParams& p, const PixelSet& s, long long i, float*& out) {
    const int per = s.UH * s.UW;
    const int n = (int)(i / per), r = (int)(i - (long long)n * per);
    const int u = r / s.UW, v = r - u * s.UW;
    const int at = (s.oh0 + s.ohs * u) * p.OWW + s.ow0 + s.ows * v;
    out = p.Out + (long long)n * p.out_batch + at;
    return at;
}

// ---- weight gradient as D[(ic, fh, fw)][oc] = sum over pixels of X(pixel + tap) * dY(pixel)
struct WgradParams {
    const float* X; const float* dY; float* dW;
    ConvGeo g;
    int I;                   // IC * FH * FW
    int pixels;              // N * OH * OW
    int splits, per_split;
    int mode;                // 0 store, 1 add, 2 atomic add
};
struct PixelK {
    long long x, y;          // offsets of the pixel's first tap in X and of the pixel in dY (-1: past the end)
    Position at;
    int pad;
};
struct TapI {
    int off;
    uint32_t bits;
};
template <bool MASK>
__device__ __forceinline__ PixelK pixel_of(const WgradParams& p, int k) {
    const ConvGeo& g = p.g;
    PixelK e{0, -1, Position{-(1 << 29), 0, 0u}, 0};
    if (k < p.pixels) {
        const int opix = g.OH * g.OW, n = k / opix, r = k - n * opix;
        const int oh = r / g.OW, ow = r - oh * g.OW;
        e.at.h0 = oh * g.sH - g.pH;
        e.at.w0 = ow * g.sW - g.pW;
        if (MASK) e.at.mask = range_mask(e.at.h0, 1, g.FH, g.IH) | (range_mask(e.at.w0, 1, g.FW, g.IW) << 16);
        e.x = (long long)n * g.x_batch + e.at.h0 * g.IW + e.at.w0;
        e.y = (long long)n * g.y_batch + r;
    }
    return e;
}
template <bool MASK>
__device__ __forceinline__ TapI row_of(const WgradParams& p, int i) {
    TapI w{-1, 0xffffffffu};  // past the end: the tap test fails
    if (i < p.I) {
        const int taps = p.g.FH * p.g.FW, ic = i / taps, r = i - ic * taps;
        const int fh = r / p.g.FW, fw = r - fh * p.g.FW;
        w.off = (ic * p.g.IH + fh) * p.g.IW + fw;
        w.bits = tap_bits<MASK>(fh, fw, 1);
    }
    return w;
}

}  // namespace gather
}  // namespace cb
