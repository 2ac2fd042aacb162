// Launch parameters of conv_patch.cu, shared with the dispatch in conv_simt.cu.
#pragma once
#include "conv_gather.cuh"

namespace cb {

constexpr int kPatchTaps = 32;  // taps of a filter at most

// A chunk of channels as every role of the kernel walks it: steps (16 channels, one tap each; taps fastest) in blocks of at most kChain.
struct ChunkSteps {
    int channels16, steps, blocks, per_block;
    __device__ __forceinline__ int in_block(int b) const { return min(per_block, steps - b * per_block); }
};
struct PatchSet {
    int planes;          // input planes the taps read: 1, or up to four of even / odd rows and columns
    int ph[4], pw[4];    // row and column phase of each
    // fold: the set holds the even and odd output columns of a stride-2 data gradient; column 2c + b of the product is phase b of channel c.
    // Tap tw of the set, distance wb - tw, is filter column f0[b] + 2 (phase_wb[b] - wb + tw) of phase b, where the filter has that.
    int f0[2], phase_wb[2], phase_UW[2];
    int distance[kPatchTaps];  // of each tap in a patch, planes one behind the other: where its first row of A lies
    int taps, steps;     // of the set; steps of its whole contraction
    int pairs;           // planes 2k and 2k + 1 are even and odd columns of the same rows and are read together
    ChunkSteps full, last;  // a whole chunk; the last one
    int first;           // the taps' least distance on the line
    FastDiv segs = FastDiv(1);  // by the 32-position runs of a group of channels
    long long filter_at; // bytes to the set's filter blocks
};
struct PatchParams {
    gather::GatherParams p;              // splits: shares of the contraction, of per_split chunks of channels
    PatchSet sets[gather::kMaxSets];
    int GH, GW;                          // rows of an image and columns of a row on the line of positions
    uint32_t items;                      // tiles x column tiles x shares x sets
    FastDiv tiles = FastDiv(1), columns = FastDiv(1), splits = FastDiv(1);
    int chunks;                          // of cw channels
    int fold, cols;                      // every set's; columns of the product: output channels, twice as many with fold
    FastDiv image_out = FastDiv(1);      // by the values of an output image (pack_patch_filter clears it)
    FastDiv run = FastDiv(1);            // by a run of the filter's values (pack_patch_filter)
    FastDiv image = FastDiv(1), row = FastDiv(1);  // by GH * GW, by GW
    int px;                              // positions of a plane of a patch
    int cw;                              // channels of a chunk
    int filter_plane, run_out;           // values of a filter plane; run_out: an output channel's planes follow one another (else a channel's)
    int pslots, fslots;                  // ring slots of patches and of filter blocks
    uint32_t pslot_bytes, fslot_bytes;
    const uint8_t* filter;               // packed (pack_patch_filter)
    // Offset in a filter plane of tap (th, tw) for column j of the product, -1 where that phase has no such tap.
    template <bool FOLD>
    __device__ __forceinline__ int filter_of(int set, int th, int tw, int j) const {
        const gather::PixelSet& s = p.sets[set];
        const PatchSet& ps = sets[set];
        const int row = (s.wt0 + s.wts * th) * p.FW;
        if (!FOLD) return row + s.wu0 + s.wus * tw;
        const int fw = ps.f0[j & 1] + 2 * (ps.phase_wb[j & 1] - s.wb + tw);
        return fw >= 0 && fw < p.FW ? row + fw : -1;
    }
    // Pixel at a position of the line: its image and place; false where there is none.
    __device__ __forceinline__ bool pixel_of(const gather::PixelSet& s, int N, int at, int& n, int& u, int& v) const {
        uint32_t in, col;
        n = (int)image.split((uint32_t)at, in);
        u = (int)row.split(in, col);
        v = (int)col;
        return n < N && u < s.UH && v < s.UW;
    }
};
struct PatchPlan {
    PatchParams q;
    int bn, nsets, ctas_sm;
    double us;           // what the launches take, by a model
    size_t smem, filter_bytes;
};
bool plan_patch(const cb_ctx* ctx, const gather::GatherParams& p, int nsets, bool may_split, PatchPlan& best);
cudaError_t launch_patch(cb_ctx* ctx, PatchPlan& plan, void* scratch);  // scratch: filter_bytes on 128 bytes

}  // namespace cb
