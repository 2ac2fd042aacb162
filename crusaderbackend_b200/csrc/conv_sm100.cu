// Tensor-core implicit-GEMM convolution for sm_100a (TF32 mode), NCHW fp32, no materialised im2col.
//
// Forward and data-gradient run the same kernel: D[pixel][oc] = sum over (tap, c) of In[n, c, oh+fh-pH, ow+fw-pW]
// * Wp[tap][oc][c]. The 128 TMEM lanes of an accumulator are 128 output pixels (UMMA M), the columns are the output
// channels (UMMA N), K walks 8 input channels of one filter tap per tcgen05.mma.
//
//  * Pixels are grouped in "lines" of 32 consecutive floats of one channel plane (32/W image rows of a W-wide map,
//    W in {8,16,32}); a CTA tile is 4 lines. For each filter row fh and line, one TMA box (32 pixels of the
//    flattened H*W plane, 8*KS channels) of the NCHW input lands as [channels][128 bytes] — exactly the MN-major
//    operand layout the tensor core reads (128-byte swizzle with 32-byte atoms). Rows above / below the image are out
//    of bounds for the tensor map and arrive as zeros, which is the vertical padding.
//  * A TMA box may not start at an odd column (its innermost coordinate must be 16-byte aligned), so the
//    horizontal taps cannot be fetched as shifted boxes. They are not shifted on the input side at all: the three
//    horizontal taps of a filter row are folded into the UMMA N dimension (accumulator column fw*OCs + oc holds the
//    partial sum of tap fw evaluated at the UNSHIFTED pixel), and the epilogue adds D0[x-1] + D1[x] + D2[x+1] with
//    two warp shuffles per value; lanes at a row edge take zero instead, which is the horizontal padding.
//  * The filter reaches the kernel already packed as [fh][32-channel group][fw][oc][32 channels] (K-major rows of
//    128 bytes, zero padded) in global memory and is fetched once per CTA by TMA into 128-byte-swizzled shared
//    memory, where it stays for the whole persistent CTA. The packing is a separate small kernel
//    (pack_filter_kernel); with the context's filter cache on it runs once per weight update instead of once per call
//    (cb_conv_cache_filters / cb_filters_changed). For the data gradient the pack transposes the channel roles and
//    rotates the filter by 180 degrees (seblas/operations/cuConv.cu:321-326 does the same rotation on the fly).
//  * When a layer has fewer pixel tiles than the GPU has CTA slots, the output channels are split over 2 or 4 CTAs
//    per tile (each fetches only its slice of the packed filter and runs a narrower UMMA), so that small feature maps
//    still occupy the whole GPU.
//  * Epilogue (two warps per TMEM lane quarter where two CTAs share an SM, else four): tcgen05.ld, tap combine, then
//    optional per-channel or per-position scale / shift, bias, ReLU, and 1 KB of staging a warp that leaves by TMA store, or
//    by TMA reduce-add where it adds onto the output; outputs TMA cannot address are written directly, 128 bytes a warp.
//
// Covered geometry: stride 1, filter 1x1 (pad 0) or 3x3 (pad 1) per axis, W in {8,16,32}, (32/W) | H,
// FW * OC(rounded to 16) <= 256 per CTA, packed filter slice <= ~150 KB; stride 2 through the phase split below.
// Everything else is served by the gathers of conv_simt.cu (CUDA cores) and conv_split.cu (tensor cores at fp32 accuracy).
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "conv_common.cuh"

namespace cb {
namespace {

struct ConvParams {
    int N, Cin, H, W, Cout;   // "input" and "output" of this pass (forward: X -> Y, dgrad: dY -> dX)
    int FH, FW, pH, pW;       // taps and padding: tap (fh, fw) reads the input at offset (fh - pH, fw - pW), each in [-1, 1]
    int OCs;                  // output channels one CTA computes (a multiple of 16)
    int nsplit;               // CTAs sharing a pixel tile, CTA b taking channels [(b % nsplit) * OCs, +OCs)
    int NQ;                   // UMMA N = FW * OCs
    int CG;                   // 32-channel groups of the packed filter
    int KS;                   // UMMA K steps (8 channels each) per pipeline stage
    int NCB;                  // ceil(Cin / (8 * KS)) pipeline stages per tile
    int L;                    // image rows per line (32 / W)
    int LPI;                  // lines per image (H / L)
    int shared_rows;          // 1: the FH taps of a tile share FH + 3 row blocks (W == 32); 0: FH * 4 blocks
    int nblocks;              // row blocks per stage
    long long total_lines;    // N * LPI
    int tiles;                // ceil(total_lines / 4)
    int stages;
    int tmem_cols;
    uint32_t w_bytes;         // resident slice of the packed filter
    uint32_t block_bytes;     // one line of a stage: 8 * KS channels x 128 B
    uint32_t stage_bytes;     // nblocks * block_bytes
    int epi_sets;             // sets of epilogue warps that take the tiles in turn
    int tma_out;              // 1: results leave through TMA stores (2: TMA reduce-adds) staged in shared memory
    float* Out;
    long long out_batch;      // elements between consecutive images of the output
    ConvEpilogue ep;
    int f_wrap;         // > 0: K steps (8 channels) from f_wrap on take the packed filter's rows f_wrap steps earlier (3xTF32)
    int c_wrap;         // > 0: input channels from c_wrap on are read again from channel (c - c_wrap) (3xTF32 form), and of the
                        // channels before it the second half comes first
    int* status;
    long long* trace;
    int dbg;       // development probes of the trace build
};

struct __align__(8) ConvSmem {
    uint64_t full[kConvMaxStages];
    uint64_t empty[kConvMaxStages];
    uint64_t tfull[2];
    uint64_t tempty[2];
    uint64_t wbar;
    uint64_t drain;
    uint32_t tmem_base;
    int abort_flag;
};

enum { PACK_FWD = 0, PACK_DGRAD = 1, PACK_S2_FWD = 2, PACK_S2_DGRAD = 3 };
constexpr int kMaxTileUmmas = 256;  // most UMMAs of one tile (filter rows x 8-channel steps) a plan may need

// Horizontal tap sets the kernel is instantiated for: the taps' column offsets fw - pW.
enum { TAPS_1 = 0 /* {0} */, TAPS_3 = 1 /* {-1, 0, +1} */, TAPS_2L = 2 /* {-1, 0} */, TAPS_2R = 3 /* {0, +1} */ };

// One chunk of 8 output channels of a tile's epilogue: the horizontal taps were accumulated at the unshifted pixel in
// column blocks fw*OCs + c; the tap with column offset d holds its partial sum d lanes away, and lanes that would read
// across a row edge take zero instead (the horizontal padding). The epilogue is bound by latency and instruction issue (an SM
// runs up to 16 epilogue warps of two CTAs), so the tap set is a template parameter and the plain forms take a branch-free path.
// The 8 x 32 results leave either through one TMA store of the [8 channels][32 pixels] block, staged in this warp's
// shared-memory slot `stage` (eight direct stores per thread land in eight different 4 KB-apart lines and were the
// slowest part of the kernel), or, for the epilogue forms TMA cannot express (accumulate followed by ReLU), directly.
template <int TAPS>
__device__ __forceinline__ void conv_epilogue_chunk(const ConvParams& p, const CUtensorMap* tmOut, uint32_t t_row, int c,
                                                    int oc0, float* img, long long plane, int pix, int n, bool valid,
                                                    bool has_left, bool has_right, uint32_t stage, int lane, bool traced) {
    uint32_t r0[8], r1[8], r2[8];
    tmem_ld8(t_row + (uint32_t)c, r0);
    if (TAPS != TAPS_1) tmem_ld8(t_row + (uint32_t)(p.OCs + c), r1);
    if (TAPS == TAPS_3) tmem_ld8(t_row + (uint32_t)(2 * p.OCs + c), r2);
    tmem_ld_wait();
    if (traced) CB_TRACE_EVENT(p.trace, 13);
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        if (TAPS == TAPS_1) {
            v[e] = __uint_as_float(r0[e]);
        } else if (TAPS == TAPS_3) {
            const float up = __shfl_up_sync(0xffffffffu, __uint_as_float(r0[e]), 1);
            const float dn = __shfl_down_sync(0xffffffffu, __uint_as_float(r2[e]), 1);
            v[e] = ((has_left ? up : 0.f) + __uint_as_float(r1[e])) + (has_right ? dn : 0.f);
        } else if (TAPS == TAPS_2L) {
            const float up = __shfl_up_sync(0xffffffffu, __uint_as_float(r0[e]), 1);
            v[e] = (has_left ? up : 0.f) + __uint_as_float(r1[e]);
        } else {
            const float dn = __shfl_down_sync(0xffffffffu, __uint_as_float(r1[e]), 1);
            v[e] = __uint_as_float(r0[e]) + (has_right ? dn : 0.f);
        }
    }
    if (traced) CB_TRACE_EVENT(p.trace, 14);
    const bool plain = p.ep.scale == nullptr && p.ep.bias == nullptr;
    if (p.tma_out) {
        // the store issued from this slot before must have finished reading it
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
        const uint32_t mine = stage + (uint32_t)(lane * 4);
        if (plain) {
            const bool relu = p.ep.relu != 0;
#pragma unroll
            for (int e = 0; e < 8; ++e)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + (uint32_t)(e * 128)), "f"(relu ? fmaxf(v[e], 0.f) : v[e])
                             : "memory");
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int oc = oc0 + c + e;
                float y = v[e];
                if (oc < p.Cout) {
                    if (p.ep.scale) {
                        const long long si = p.ep.per_position ? (long long)oc * plane + pix : (long long)oc;
                        y = fmaf(y, __ldg(p.ep.scale + si), __ldg(p.ep.shift + si));
                    }
                    if (p.ep.bias) y += __ldg(p.ep.bias + oc);
                    if (p.ep.relu) y = fmaxf(y, 0.f);
                }
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + (uint32_t)(e * 128)), "f"(y) : "memory");
            }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && valid) {
            if (p.tma_out == 2) tma_reduce_add_3d(tmOut, stage, pix, oc0 + c, n);
            else tma_store_3d(tmOut, stage, pix, oc0 + c, n);
            tma_store_commit();
        }
    } else if (valid) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int oc = oc0 + c + e;
            if (oc < p.Cout) {
                float y = v[e];
                const long long idx = (long long)oc * plane + pix;
                if (p.ep.scale) {
                    const long long si = p.ep.per_position ? idx : (long long)oc;
                    y = fmaf(y, __ldg(p.ep.scale + si), __ldg(p.ep.shift + si));
                }
                if (p.ep.bias) y += __ldg(p.ep.bias + oc);
                if (p.ep.accumulate) y += img[idx];
                if (p.ep.relu) y = fmaxf(y, 0.f);
                img[idx] = y;
            }
        }
    }
    if (traced) CB_TRACE_EVENT(p.trace, 15);
}

// Epilogue warps: eight (two per TMEM lane quarter) where two CTAs share an SM (outputs of at most 32 channels per CTA with a
// small filter: their UMMA chains overlap), else sixteen. A warp's chunk of 8 channels is a chain of latencies (TMEM load,
// shuffles, staging, proxy fence, TMA store: ~1100 clocks), so the chunks of a tile go to different warps, and where a tile
// has fewer chunks than warps they form sets that take the tiles in turn. 64 -> 64 at 32 x 32 with eight warps was bound by
// this; 16 -> 16 pays more for the start of 1152 threads an SM than the second eight warps of each CTA gain.
template <int kEpiWarps, int TAPS>
__global__ void __launch_bounds__(64 + 32 * kEpiWarps, kEpiWarps == 8 ? 2 : 1)
    umma_conv_kernel(const __grid_constant__ CUtensorMap tmIn, const __grid_constant__ CUtensorMap tmW,
                     const __grid_constant__ CUtensorMap tmOut, const ConvParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ ConvSmem cs;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // uniform for the compiler too
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &cs.abort_flag;

    const uint32_t w_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t st_base = w_base + p.w_bytes;
    const uint32_t out_base = st_base + (uint32_t)p.stages * p.stage_bytes;  // epilogue staging: 1 KB per epilogue warp
    // this CTA's slice of the output channels and its walk over the pixel tiles
    const int split = (int)blockIdx.x % p.nsplit;
    const int tile0 = (int)blockIdx.x / p.nsplit;
    const int tile_step = (int)gridDim.x / p.nsplit;
    const int oc0 = split * p.OCs;

    if (threadIdx.x == 0) {
        CB_TRACE_WALL(p.trace, 0);
        CB_TRACE_EVENT(p.trace, 1);
        cs.abort_flag = 0;
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&cs.full[s]), 1);
            mbar_init(smem_u32(&cs.empty[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&cs.tfull[a]), 1);
            mbar_init(smem_u32(&cs.tempty[a]), (uint32_t)(kEpiWarps / p.epi_sets));
        }
        mbar_init(smem_u32(&cs.wbar), 1);
        mbar_init(smem_u32(&cs.drain), 1);
        mbar_fence_init();
        tma_prefetch_desc(&tmIn);
        tma_prefetch_desc(&tmW);
        if (p.tma_out) tma_prefetch_desc(&tmOut);
    }
    __syncthreads();
    if (warp == 1) {
        tmem_alloc(smem_u32(&cs.tmem_base), (uint32_t)p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Up to here nothing has touched global memory (barriers, descriptor prefetch of kernel parameters, TMEM): the
    // kernel before this one may still be running. From here on its results are complete, and the kernel after this
    // one may begin its own preamble.
    griddep_wait_then_launch();
    const uint32_t tmem_base = cs.tmem_base;
    const uint32_t acc_stride = (uint32_t)p.tmem_cols >> 1;
    uint32_t fills = 0;  // producer: stages filled so far
    if (threadIdx.x == 0) CB_TRACE_EVENT(p.trace, 2);

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        uint32_t s = 0, ph = 0, ahead = 0;
        bool ok = true;
        for (int tile = tile0; tile < p.tiles && ok; tile += tile_step) {
            // the tile's four lines; lines past the end use an image index >= N: their boxes are zero-filled
            int n[4], h0[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int g = 4 * tile + j;  // 32-bit: a 64-bit division costs ~100 cycles on this path
                n[j] = g / p.LPI;
                h0[j] = (g - n[j] * p.LPI) * p.L;
            }
            for (int cb = 0; cb < p.NCB; ++cb) {
                if (!__all_sync(0xffffffffu, ahead)) {
                    ok = mbar_wait_uniform(smem_u32(&cs.empty[s]), ph ^ 1u, abort_flag, p.status, CBK_TIMEOUT_EMPTY);
                    if (!ok) break;
                }
                const uint32_t s1 = s + 1 == (uint32_t)p.stages ? 0u : s + 1, ph1 = s1 ? ph : ph ^ 1u;
                ahead = mbar_test(smem_u32(&cs.empty[s1]), ph1 ^ 1u);
                const uint32_t full = smem_u32(&cs.full[s]);
                const uint32_t dst0 = st_base + s * p.stage_bytes;
                mbar_expect_tx_elect(full, p.stage_bytes);
                int c0 = cb * p.KS * kCB;
                if (p.c_wrap)  // 3xTF32: [x ; x_lo] in memory is read as x_lo, x, x
                    c0 = c0 >= p.c_wrap ? c0 - p.c_wrap : (2 * c0 >= p.c_wrap ? c0 - p.c_wrap / 2 : c0 + p.c_wrap / 2);
                if (p.shared_rows) {
                    // W == 32: the tile is 4 consecutive rows of one image; ONE box (32 px, 8*KS channels, FH+3
                    // rows) lands as [row][channel][128 B]; rows above / below the image are zero-filled
                    tma_load_4d_elect(dst0, &tmIn, full, 0, c0, h0[0] - p.pH, n[0]);
                } else {
                    for (int fh = 0; fh < p.FH; ++fh) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            tma_load_3d_elect(dst0 + (uint32_t)(fh * 4 + j) * p.block_bytes, &tmIn, full,
                                              (h0[j] + fh - p.pH) * p.W, c0, n[j]);
                    }
                }
                ++fills;
                s = s1;
                ph = ph1;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ UMMA issuer
        // One thread feeds the tensor core, and what it spends per tcgen05.mma bounds the kernel (a 128 x 48 x 8 UMMA is
        // ~50 cycles of tensor pipe). The operand descriptors are advanced by plain integer arithmetic on values that
        // come from kernel parameters and loop counters only: a descriptor offset fetched from a shared-memory table
        // costs ~113 cycles per UMMA whatever its size (measured with the UMMA-only loop of peak_sm100.cu: 52 -> 113
        // cycles at N = 64, 103 -> 124 at N = 192), one computed with divisions ~150 instructions.
        const uint32_t idesc = umma_idesc_tf32(128, (uint32_t)p.NQ, 1u, 0u);
        // P: 4 lines x [8 channels][128 B], MN-major: block_bytes between lines (LBO), 512 B per 4 channel rows (SBO)
        const uint64_t descP0 = umma_smem_desc(0, p.block_bytes, 512u, UMMA_SW_128B_BASE32B);
        // Q: packed filter rows [(fw, oc)][32 channels], K-major 128-byte rows
        const uint64_t descQ0 = umma_smem_desc(w_base, 16u, 1024u, UMMA_SW_128B);
        const uint32_t blk_units = p.block_bytes >> 4;                     // descriptor address units (16 B) per line block
        const uint32_t fh_units = (p.shared_rows ? 1u : 4u) * blk_units;  // between consecutive filter rows of P
        const uint32_t q_group_units = (uint32_t)p.NQ * (kRowBytes >> 4);  // one (filter row, 32-channel group) of Q
        const uint32_t q_fh_units = (uint32_t)p.CG * q_group_units;        // between consecutive filter rows of Q
        // The whole warp runs the loop with the same values (waits go through votes) and one elected lane issues, so that
        // the descriptors stay in uniform registers; the next stage's barrier is tested while this one's UMMAs are issued.
        uint32_t s = 0, ph = 0, lt = 0, ahead = 0;
        {
            // this warp fetches the resident filter slice, while the producer is already at the first stage: one box
            // [FW taps][OCs rows][32 channels] per (filter row, channel group)
            const uint32_t wbar = smem_u32(&cs.wbar);
            mbar_expect_tx_elect(wbar, p.w_bytes);
            const int boxes = p.FH * p.CG;
            for (int b = 0; b < boxes; ++b)
                tma_load_3d_elect(w_base + (uint32_t)b * p.NQ * kRowBytes, &tmW, wbar, 0, oc0, b * p.FW);
        }
        bool ok = mbar_wait_uniform(smem_u32(&cs.wbar), 0, abort_flag, p.status, CBK_TIMEOUT_FULL);
        if (lane == 0) CB_TRACE_EVENT(p.trace, 4);
        for (int tile = tile0; tile < p.tiles && ok; tile += tile_step, ++lt) {
            const uint32_t a = lt & 1u;
            ok = mbar_wait_uniform(smem_u32(&cs.tempty[a]), ((lt >> 1) & 1u) ^ 1u, abort_flag, p.status, CBK_TIMEOUT_TMEM_EMPTY);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + a * acc_stride;
            uint32_t acc = 0u;
            for (int cb = 0; cb < p.NCB; ++cb) {
                if (!__all_sync(0xffffffffu, ahead)) {
                    ok = mbar_wait_uniform(smem_u32(&cs.full[s]), ph, abort_flag, p.status, CBK_TIMEOUT_FULL);
                    if (!ok) break;
                }
                const uint32_t s1 = s + 1 == (uint32_t)p.stages ? 0u : s + 1, ph1 = s1 ? ph : ph ^ 1u;
                ahead = mbar_test(smem_u32(&cs.full[s1]), ph1);
                tc_fence_after();
                if (lane == 0 && lt == 0 && cb == 0) CB_TRACE_EVENT(p.trace, 5);
                if (lane == 0 && lt == 1 && cb == 0) CB_TRACE_EVENT(p.trace, 3);
                const uint64_t pbase = descP0 + (uint64_t)(((st_base + s * p.stage_bytes) >> 4) & 0x3FFFu);
                // a stage holds 1, 2 or 4 K steps of 8 channels, never across a 32-channel group of the packed filter
                const uint32_t ks0 = (uint32_t)(cb * p.KS);
                // 3xTF32: the groups [x_lo ; x ; x] meet the packed groups [w ; w_lo] as w, w_lo, w
                const uint32_t fs0 = p.f_wrap && ks0 >= (uint32_t)p.f_wrap ? ks0 - (uint32_t)p.f_wrap : ks0;
                const uint64_t q0 = descQ0 + (uint64_t)((fs0 >> 2) * q_group_units + (fs0 & 3u) * 2u);
                for (int fh = 0; fh < p.FH; ++fh) {
                    const uint64_t dp = pbase + (uint64_t)((uint32_t)fh * fh_units);
                    const uint64_t dq = q0 + (uint64_t)((uint32_t)fh * q_fh_units);
                    umma_tf32_elect(d_tmem, dp, dq, idesc, acc);
                    acc = 1u;
                    if (p.KS >= 2) umma_tf32_elect(d_tmem, dp + 64u, dq + 2u, idesc, 1u);
                    if (p.KS == 4) {
                        umma_tf32_elect(d_tmem, dp + 128u, dq + 4u, idesc, 1u);
                        umma_tf32_elect(d_tmem, dp + 192u, dq + 6u, idesc, 1u);
                    }
                }
                tc_commit_elect(smem_u32(&cs.empty[s]));
                if (cb == p.NCB - 1) tc_commit_elect(smem_u32(&cs.tfull[a]));
                if (lane == 0 && lt == 0 && cb == p.NCB - 1) CB_TRACE_EVENT(p.trace, 6);
                s = s1;
                ph = ph1;
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2 ..)
        const int quarter = warp & 3;
        const int per_set = kEpiWarps / 4 / p.epi_sets;           // warps of a set on this lane quarter
        const int set = ((warp - 2) >> 2) / per_set, slot = ((warp - 2) >> 2) - set * per_set;
        const uint32_t my_stage = out_base + (uint32_t)(warp - 2) * 1024u;
        uint32_t lt = 0;
        bool ok = true;
        const long long plane = (long long)p.H * p.W;
        const int col = lane & (p.W - 1);
        const bool has_left = col > 0, has_right = col < p.W - 1;
        lt = (uint32_t)set;
        for (int tile = tile0 + set * tile_step; tile < p.tiles && ok; tile += p.epi_sets * tile_step, lt += (uint32_t)p.epi_sets) {
            const uint32_t a = lt & 1u;
            const int g = 4 * tile + quarter;
            const bool valid = g < (int)p.total_lines;
            const int n = g / p.LPI;
            const int h0 = (g - n * p.LPI) * p.L;
            // lane x of the line is pixel (h0 + x / W, x % W): 32 consecutive floats of the output plane
            float* img = p.Out + (long long)n * p.out_batch;
            const int pix = h0 * p.W + lane;
            ok = mbar_wait_uniform(smem_u32(&cs.tfull[a]), (lt >> 1) & 1u, abort_flag, p.status, CBK_TIMEOUT_TMEM_FULL);
            if (!ok) break;
            tc_fence_after();
            if (threadIdx.x == 64 && lt == 0) CB_TRACE_EVENT(p.trace, 7);
            if (threadIdx.x == 64 && lt == 1) CB_TRACE_EVENT(p.trace, 9);
            const uint32_t t_row = tmem_base + a * acc_stride + ((uint32_t)(32 * quarter) << 16);
#ifdef CB_TRACE
            if (p.dbg & 1) {  // development probe: leave the accumulator unread (how fast is the MMA phase alone?)
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&cs.tempty[a]));
                continue;
            }
#endif
            for (int c = slot * 8; c < p.OCs; c += 8 * per_set)
                conv_epilogue_chunk<TAPS>(p, &tmOut, t_row, c, oc0, img, plane, pix, n, valid, has_left, has_right,
                                    my_stage, lane, threadIdx.x == 64 && lt == 0 && c == 0);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&cs.tempty[a]));
            if (threadIdx.x == 64 && lt == 0) CB_TRACE_EVENT(p.trace, 8);
            if (threadIdx.x == 64) CB_TRACE_EVENT(p.trace, 10);
        }
        // this warp's stores must have read their staging memory before it is released with the CTA (the writes themselves
        // are complete when the grid is)
        if (p.tma_out && lane == 0) tma_store_wait_read<0>();
    }

    tc_fence_before();
    __syncthreads();
    if (cs.abort_flag) {
        // A bounded wait gave up somewhere in this CTA. Copies armed before that may still be in flight towards this
        // CTA's shared memory and issued MMAs may still be running on its accumulators: give both a bounded chance to
        // finish before the shared memory and TMEM are released.
        if (warp == 1 && lane == 0) mbar_drain(smem_u32(&cs.wbar), 0, p.status);
        if (warp == 0 && lane == 0) {
            const uint32_t n = (uint32_t)p.stages;  // stage st was last filled as number st + n * round: parity of the round
            for (uint32_t st = 0; st < n && st < fills; ++st) mbar_drain(smem_u32(&cs.full[st]), ((fills - 1 - st) / n) & 1u, p.status);
        }
        if (warp == 1) {  // the commit comes from the lane that issued the MMAs
            tc_commit_elect(smem_u32(&cs.drain));
            if (lane == 0) mbar_drain(smem_u32(&cs.drain), 0, p.status);
        }
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
    if (threadIdx.x == 0) {
        CB_TRACE_EVENT(p.trace, 11);
        CB_TRACE_WALL(p.trace, 12);
    }
}

// What one packed filter is made from: W is the caller's OC x IC x FHs x FWs filter, (FHc, FWc) the taps of the
// convolution the kernel runs. Row index = ((fh * CG + cg) * FWc + fw) * OCp + o, 32 floats per row.
//   PACK_FWD:      row[c] = W[o][cg*32 + c][fh][fw]
//   PACK_DGRAD:    row[c] = W[cg*32 + c][o][FH-1-fh][FW-1-fw]          (o = input channel of the convolution)
//   PACK_S2_FWD:   the stride-2 3x3 convolution as a 2x2 convolution over the 4 input phases stacked as channels
//                  c' = phase*IC + c: row[c'] = W[o][c][s2_tap(ph, fh)][s2_tap(pw, fw)] (zero where no tap lands)
//   PACK_S2_DGRAD: its adjoint: input channels are the OC planes of dY, output o' = out_first + o indexes (phase, c),
//                  taps flipped: row[oc] = W[oc][c][s2_tap(ph, 1-fh)][s2_tap(pw, 1-fw)]
// x3 > 0 (a multiple of 8, at least the pass's input channels): the packed channels are two groups of x3, the filter and its
// lo part (3xTF32: lo = rna_tf32(w - hi) with hi the 19 bits the tensor core reads).
struct PackJob {
    const float* W;
    float* Wp;
    int OC, IC, FHs, FWs, FHc, FWc, OCp, CG, mode, out_first, out_count, x3;
    unsigned total;   // floats of the packed filter (of at most a few hundred kilobytes)
};

// Value of the packed filter at channel ch of row (fh, fw, o), zero outside the filter.
__device__ __forceinline__ float pack_source(const PackJob& j, int ch, int fh, int fw, int o) {
    const float* W = j.W;
    const int OC = j.OC, IC = j.IC, FHs = j.FHs, FWs = j.FWs;
    if (j.mode == PACK_FWD) {
        if (o < OC && ch < IC) return W[((o * IC + ch) * FHs + fh) * FWs + fw];
    } else if (j.mode == PACK_DGRAD) {
        if (o < IC && ch < OC) return W[((ch * IC + o) * FHs + (FHs - 1 - fh)) * FWs + (FWs - 1 - fw)];
    } else if (j.mode == PACK_S2_FWD) {
        if (o < OC && ch < 4 * IC) {
            const int phase = ch / IC, cc = ch - phase * IC;
            const int sh = s2_tap(phase >> 1, fh), sw = s2_tap(phase & 1, fw);
            if (sh >= 0 && sw >= 0) return W[(((long long)o * IC + cc) * FHs + sh) * FWs + sw];
        }
    } else {
        if (o < j.out_count && ch < OC) {
            const int og = j.out_first + o;
            const int phase = og / IC, cc = og - phase * IC;
            const int sh = s2_tap(phase >> 1, 1 - fh), sw = s2_tap(phase & 1, 1 - fw);
            if (sh >= 0 && sw >= 0) return W[(((long long)ch * IC + cc) * FHs + sh) * FWs + sw];
        }
    }
    return 0.f;
}
__device__ __forceinline__ float tf32_lo(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u)));
    return __uint_as_float(r);
}
__device__ __forceinline__ float pack_value(const PackJob& j, unsigned i) {
    const int c = (int)(i & 31);
    unsigned r = i >> 5;
    const int o = (int)(r % (unsigned)j.OCp);
    r /= (unsigned)j.OCp;
    const int fw = (int)(r % (unsigned)j.FWc);
    r /= (unsigned)j.FWc;
    const int cg = (int)(r % (unsigned)j.CG);
    const int fh = (int)(r / (unsigned)j.CG);
    const int ch = cg * 32 + c;
    if (j.x3 == 0 || ch < j.x3) return pack_source(j, ch, fh, fw, o);
    return ch < 2 * j.x3 ? tf32_lo(pack_source(j, ch - j.x3, fh, fw, o)) : 0.f;
}

__global__ void pack_filter_kernel(const PackJob j) {
    griddep_wait_then_launch();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < j.total; i += gridDim.x * blockDim.x) j.Wp[i] = pack_value(j, i);
}
// Every cached filter of a context in one launch: blockIdx.y indexes a device table of jobs.
__global__ void pack_filter_table_kernel(const PackJob* __restrict__ jobs) {
    griddep_wait_then_launch();
    const PackJob j = jobs[blockIdx.y];
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < j.total; i += gridDim.x * blockDim.x) j.Wp[i] = pack_value(j, i);
}

// ---- re-layout kernels of the stride-2 path (memory-bound, one element per thread, coalesced on the write side)
// Xs[n][phase*C + c][i][j] = X[n][c][2i + (phase >> 1)][2j + (phase & 1)]
__global__ void space_to_depth2_kernel(const float* __restrict__ X, float* __restrict__ Xs, int C, int H, int W,
                                       long long total) {
    griddep_wait_then_launch();
    const int H2 = H / 2, W2 = W / 2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(i % W2);
        long long r = i / W2;
        const int ii = (int)(r % H2);
        r /= H2;
        const int cp = (int)(r % (4 * C));
        const long long n = r / (4 * C);
        const int phase = cp / C, c = cp - phase * C;
        Xs[i] = X[((n * C + c) * H + 2 * ii + (phase >> 1)) * W + 2 * j + (phase & 1)];
    }
}
// dX[n][c][y][x] (+)= dXs[group][n][o][y/2][x/2] with phase*C + c = group*per_group + o
__global__ void depth_to_space2_kernel(const float* __restrict__ dXs, float* __restrict__ dX, int N, int C, int H, int W,
                                       int per_group, long long total, int accumulate) {
    griddep_wait_then_launch();
    const int H2 = H / 2, W2 = W / 2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % W);
        long long r = i / W;
        const int y = (int)(r % H);
        r /= H;
        const int c = (int)(r % C);
        const long long n = r / C;
        const int og = ((y & 1) * 2 + (x & 1)) * C + c;
        const int g = og / per_group, o = og - g * per_group;
        const float v = dXs[((((long long)g * N + n) * per_group + o) * H2 + (y >> 1)) * W2 + (x >> 1)];
        dX[i] = accumulate ? dX[i] + v : v;
    }
}
// Xsub[nc][i][j] = X[nc][2i][2j]
__global__ void subsample2_kernel(const float* __restrict__ X, float* __restrict__ Xsub, long long NC, int H, int W,
                                  long long total) {
    griddep_wait_then_launch();
    const int H2 = H / 2, W2 = W / 2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(i % W2);
        const long long r = i / W2;
        const int ii = (int)(r % H2);
        const long long nc = r / H2;
        Xsub[i] = X[(nc * H + 2 * ii) * W + 2 * j];
    }
}
// dX[nc][y][x] (+)= (y, x both even) ? dXsub[nc][y/2][x/2] : 0
__global__ void upsample2_zero_kernel(const float* __restrict__ dXsub, float* __restrict__ dX, int H, int W,
                                      long long total, int accumulate) {
    griddep_wait_then_launch();
    const int H2 = H / 2, W2 = W / 2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % W);
        const long long r = i / W;
        const int y = (int)(r % H);
        const long long nc = r / H;
        const float v = ((x | y) & 1) ? 0.f : dXsub[(nc * H2 + (y >> 1)) * W2 + (x >> 1)];
        if (accumulate) {
            if (!((x | y) & 1)) dX[i] += v;
        } else {
            dX[i] = v;
        }
    }
}

// Vector forms of the four re-layout kernels for 16-byte aligned tensors with W % 4 == 0: one item is four consecutive pixels
// of an input row (a 16-byte access on the full-resolution side, two 8-byte accesses on the half-resolution side), so every
// access is coalesced. kRelayoutItems items a thread are loaded before the first is stored.
struct PlaneIndex {      // item -> (plane n * C + c, row y, quad q)
    FastDiv wq, h, c;
};
constexpr int kRelayoutItems = 4;
__global__ void __launch_bounds__(256) space_to_depth2_vec_kernel(const float* __restrict__ X, float* __restrict__ Xs, const PlaneIndex ix,
                                                                  int W2, long long plane2, uint32_t items) {
    griddep_wait_then_launch();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < items; i0 += kRelayoutItems * stride) {
        float4 v[kRelayoutItems];
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u)
            if (i0 + u * stride < items) v[u] = reinterpret_cast<const float4*>(X)[i0 + u * stride];
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u) {
            if (i0 + u * stride >= items) break;
            uint32_t q, y, c;
            const uint32_t n = ix.c.split(ix.h.split(ix.wq.split(i0 + u * stride, q), y), c);
            float* d0 = Xs + ((long long)(n * 4 + 2 * (y & 1)) * ix.c.d + c) * plane2 + (y >> 1) * W2 + 2 * q;  // phase (row, 0)
            *reinterpret_cast<float2*>(d0) = make_float2(v[u].x, v[u].z);
            *reinterpret_cast<float2*>(d0 + ix.c.d * plane2) = make_float2(v[u].y, v[u].w);                     // phase (row, 1)
        }
    }
}
__global__ void __launch_bounds__(256) depth_to_space2_vec_kernel(const float* __restrict__ dXs, float* __restrict__ dX, const PlaneIndex ix,
                                                                  int N, int W2, long long plane2, const FastDiv group, uint32_t items,
                                                                  int accumulate) {
    griddep_wait_then_launch();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < items; i0 += kRelayoutItems * stride) {
        float4 v[kRelayoutItems];
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u) {
            if (i0 + u * stride >= items) break;
            uint32_t q, y, c;
            const uint32_t n = ix.c.split(ix.h.split(ix.wq.split(i0 + u * stride, q), y), c);
            float2 ph[2];
#pragma unroll
            for (uint32_t col = 0; col < 2; ++col) {
                uint32_t o;
                const uint32_t g = group.split(((y & 1) * 2 + col) * ix.c.d + c, o);
                ph[col] = *reinterpret_cast<const float2*>(dXs + (((long long)g * N + n) * group.d + o) * plane2 + (y >> 1) * W2 + 2 * q);
            }
            v[u] = make_float4(ph[0].x, ph[1].x, ph[0].y, ph[1].y);
            if (accumulate) {
                const float4 old = reinterpret_cast<const float4*>(dX)[i0 + u * stride];
                v[u] = make_float4(old.x + v[u].x, old.y + v[u].y, old.z + v[u].z, old.w + v[u].w);
            }
        }
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u)
            if (i0 + u * stride < items) reinterpret_cast<float4*>(dX)[i0 + u * stride] = v[u];
    }
}
// item: four pixels of an even row
__global__ void __launch_bounds__(256) subsample2_vec_kernel(const float* __restrict__ X, float* __restrict__ Xsub, const FastDiv wq, int W,
                                                             uint32_t items) {
    griddep_wait_then_launch();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < items; i += gridDim.x * blockDim.x) {
        uint32_t q;
        const uint32_t row = wq.split(i, q);  // plane * H/2 + output row: H is even, so input row 2 * row of the stack of planes
        const float4 v = *reinterpret_cast<const float4*>(X + 2LL * row * W + 4 * q);
        reinterpret_cast<float2*>(Xsub)[i] = make_float2(v.x, v.z);
    }
}
__global__ void __launch_bounds__(256) upsample2_zero_vec_kernel(const float* __restrict__ dXsub, float* __restrict__ dX, const FastDiv wq,
                                                                 uint32_t items, int accumulate) {
    griddep_wait_then_launch();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < items; i += gridDim.x * blockDim.x) {
        uint32_t q;
        const uint32_t row = wq.split(i, q);  // row of the stack of planes
        float4* dst = reinterpret_cast<float4*>(dX) + i;
        if (row & 1) {
            if (!accumulate) *dst = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const float2 a = reinterpret_cast<const float2*>(dXsub)[(row >> 1) * wq.d + q];
        if (accumulate) {
            const float4 old = *dst;
            *dst = make_float4(old.x + a.x, old.y, old.z + a.y, old.w);
        } else {
            *dst = make_float4(a.x, 0.f, a.y, 0.f);
        }
    }
}
// the vector kernels index items, and step past the end by up to kRelayoutItems grids, in 32 bits
constexpr long long kMostItems = 1LL << 30;
static bool vec_ok(const void* a, const void* b, int W) {
    return (W & 3) == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15u) == 0;
}

// 3xTF32 in one pass: X2[n][c] = X[n][c] and X2[n][Cp + c] = lo part of X[n][c] (x = hi + lo with hi the 19 bits the
// tensor core reads, lo = rna_tf32(x - hi)), four pixels per thread; planes C .. Cp of both halves are zeroed (Cp: C rounded up
// to the 8 channels of a K step). X may be batch-strided, X2 is dense.
__device__ __forceinline__ float4 lo4(float4 v) { return make_float4(tf32_lo(v.x), tf32_lo(v.y), tf32_lo(v.z), tf32_lo(v.w)); }
__global__ void __launch_bounds__(256) tf32_split2_kernel(const float* __restrict__ X, float* __restrict__ X2, long long per4,
                                                          const FastDiv perp4, long long x_batch, uint32_t items) {
    griddep_wait_then_launch();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < items; i0 += kRelayoutItems * stride) {
        float4 v[kRelayoutItems];
        uint32_t n[kRelayoutItems], r[kRelayoutItems];
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u) {
            n[u] = perp4.split(i0 + u * stride, r[u]);
            v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i0 + u * stride < items && r[u] < per4) v[u] = *reinterpret_cast<const float4*>(X + n[u] * x_batch + 4LL * r[u]);
        }
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u) {
            if (i0 + u * stride >= items) break;
            float4* dst = reinterpret_cast<float4*>(X2) + 2LL * n[u] * perp4.d + r[u];
            dst[0] = v[u];
            dst[perp4.d] = lo4(v[u]);
        }
    }
}
// The same together with the phase split of a stride-2 convolution: X2 holds 2 * Cp planes of H/2 x W/2, the 4 C phase planes
// of X and, Cp planes later, their lo parts (Cp: 4 C rounded up to a multiple of 8, the planes between zeroed).
__global__ void __launch_bounds__(256) space_to_depth2_split_kernel(const float* __restrict__ X, float* __restrict__ X2, const PlaneIndex ix,
                                                                    int Cp, int W2, long long plane2, uint32_t items) {
    griddep_wait_then_launch();
    const uint32_t stride = gridDim.x * blockDim.x, C = ix.c.d;
    const long long half = Cp * plane2, pad = (Cp - 4LL * C) * plane2;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < items; i0 += kRelayoutItems * stride) {
        float4 v[kRelayoutItems];
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u)
            if (i0 + u * stride < items) v[u] = reinterpret_cast<const float4*>(X)[i0 + u * stride];
#pragma unroll
        for (int u = 0; u < kRelayoutItems; ++u) {
            if (i0 + u * stride >= items) break;
            uint32_t q, y, c;
            const uint32_t n = ix.c.split(ix.h.split(ix.wq.split(i0 + u * stride, q), y), c);
            const float4 l = lo4(v[u]);
            float* image = X2 + n * 2 * half;
            float* d0 = image + (2LL * (y & 1) * C + c) * plane2 + (y >> 1) * W2 + 2 * q;  // phase (row, 0)
            float* d1 = d0 + C * plane2;                                                   // phase (row, 1)
            *reinterpret_cast<float2*>(d0) = make_float2(v[u].x, v[u].z);
            *reinterpret_cast<float2*>(d1) = make_float2(v[u].y, v[u].w);
            *reinterpret_cast<float2*>(d0 + half) = make_float2(l.x, l.z);
            *reinterpret_cast<float2*>(d1 + half) = make_float2(l.y, l.w);
            // the padding planes of an image are spread over its items
            const uint32_t per_image = C * ix.h.d * ix.wq.d;
            for (long long z = i0 + u * stride - n * per_image; z < pad; z += per_image)
                image[half - pad + z] = image[2 * half - pad + z] = 0.f;
        }
    }
}

int relayout_grid(const cb_ctx* ctx, long long n, int per_thread = 1) {
    long long g = (n + 256LL * per_thread - 1) / (256LL * per_thread);
    const long long cap = (long long)ctx->sm_count * 16;
    return (int)(g > cap ? cap : (g < 1 ? 1 : g));
}

// Where a launch takes its stream, scratch and status word from: a cb_ctx or the static arrays of the allocation-free
// entry point.
struct ConvEnv {
    cudaStream_t stream;
    int sm_count, smem_optin;
    int* status;
};

// Geometry the tensor-core forward / data-gradient kernel covers; fills the derived sizes.
struct ConvPlan {
    int Cin, Cout, OCp, OCs, nsplit, NQ, CG, L, KS, shared_rows, nblocks, stages;
    int x3 = 0;      // set by the caller before planning: channels of a group of the 3xTF32 form (0: plain)
    int ks_max = 4;  // set by the caller before planning: most K steps a stage may carry
    int ew;      // epilogue warps of the kernel instantiation: 8 or 16
    int per_sm;  // CTAs the plan expects to share an SM (2 for narrow outputs with a small filter, else 1)
    size_t w_bytes;       // one CTA's slice of the packed filter
    size_t w_total_bytes; // the whole packed filter
    uint32_t block_bytes, stage_bytes;
};

// Development override of the output-channel split (1, 2 or 4); 0 = choose from the tile count.
int forced_nsplit() {
    static const int v = [] {
        const char* e = std::getenv("CB_CONV_NSPLIT");
        return e ? std::atoi(e) : 0;
    }();
    return v;
}

int plan_conv(ConvPlan& q, int smem_optin, int sm_count, const float* X, int N, int Cin, int Cout, int IH, int IW, int FH,
              int FW, int pH, int pW) {
    // every tap must read within one pixel of the output position: offsets fh - pH and fw - pW in [-1, 1]
    if (FH < 1 || FH > 3 || FW < 1 || FW > 3 || pH < 0 || pH > 1 || pW < 0 || pW > 1) return CB_EUNSUPPORTED;
    if (FH - 1 - pH > 1 || FW - 1 - pW > 1) return CB_EUNSUPPORTED;
    if (FW == 1 && pW != 0) return CB_EUNSUPPORTED;  // the kernel's one-tap form reads the output's own column
    if (IW != 8 && IW != 16 && IW != 32) return CB_EUNSUPPORTED;
    q.L = 32 / IW;
    if (IH % q.L) return CB_EUNSUPPORTED;
    q.Cin = Cin;
    q.Cout = Cout;
    q.OCp = (q.Cout + 15) / 16 * 16;
    if (q.Cin < 1) return CB_EUNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(X) & 15u) != 0) return CB_EUNSUPPORTED;
    q.CG = (q.Cin - q.x3 + 31) / 32;  // the 3xTF32 form packs two groups for three
    q.w_total_bytes = (size_t)FH * q.CG * FW * q.OCp * kRowBytes;
    q.shared_rows = (q.L == 1 && IH % 4 == 0) ? 1 : 0;
    q.nblocks = q.shared_rows ? FH + 3 : FH * 4;
    const long long tiles = ((long long)N * (IH / q.L) + 3) / 4;
    const int cin8 = (q.Cin + 7) / 8;
    // Candidate splits of the output channels over 1, 2 or 4 CTAs per pixel tile: the widest split that still fits the
    // resident CTA slots in one wave wins (small feature maps then fill the GPU); each candidate must be launchable.
    int best = 0;
    ConvPlan bestq{};
    bool forced_hit = false;
    for (int ns = 1; ns <= 4 && !forced_hit; ns <<= 1) {
        // a four-way split only when forced or when nothing narrower fits the 256 accumulator columns (very wide outputs)
        if (ns == 4 && forced_nsplit() != 4 && best != 0) break;
        // a split that needs extra padding channels only when no narrower split fits at all
        if (q.OCp % (16 * ns) != 0 && best != 0) break;
        ConvPlan c = q;
        c.nsplit = ns;
        // the packed filter is padded to a whole number of 16-channel groups per CTA; channels past Cout are zero rows
        // and their outputs are dropped by the store
        c.OCp = (q.Cout + 16 * ns - 1) / (16 * ns) * (16 * ns);
        c.w_total_bytes = (size_t)FH * q.CG * FW * c.OCp * kRowBytes;
        c.OCs = c.OCp / ns;
        c.NQ = FW * c.OCs;
        if (c.NQ > 256) continue;
        c.w_bytes = (size_t)FH * c.CG * c.NQ * kRowBytes;
        // narrow outputs with a small filter are sized so that two CTAs fit one SM (shared memory and TMEM halves)
        const bool two_per_sm = c.OCs <= 32 && c.w_bytes <= 40 * 1024;
        c.ew = two_per_sm ? 8 : 16;
        const long long avail = two_per_sm ? (long long)(smem_optin < 113 * 1024 ? smem_optin : 113 * 1024) : (long long)smem_optin;
        const long long cap = avail - 4096 - (long long)c.w_bytes - 1024LL * c.ew;  // static shared memory, alignment slack; store staging
        // as many K steps per stage as leaves at least 2 stages: fewer, larger TMA boxes measured faster than a deeper
        // pipeline of small ones. The steps of a stage are also the order in which a pixel's products are added, so they
        // are chosen as if every plan staged for sixteen epilogue warps: no result depends on how many a plan has.
        c.KS = 0;
        for (int ks = 4; ks >= 1; ks >>= 1) {
            if (ks > cin8 && ks > 1) continue;
            if (ks > q.ks_max) continue;
            const long long bytes = (long long)c.nblocks * ks * kCB * kRowBytes, st = cap / bytes;
            if ((cap - 1024LL * (16 - c.ew)) / bytes >= 2) {
                c.KS = ks;
                c.stages = (int)(st > kConvMaxStages ? kConvMaxStages : st);
                break;
            }
        }
        if (c.KS == 0) continue;
        if ((cin8 + c.KS - 1) / c.KS * c.KS * FH > kMaxTileUmmas) continue;
        c.block_bytes = (uint32_t)c.KS * kCB * kRowBytes;
        c.stage_bytes = (uint32_t)c.nblocks * c.block_bytes;
        c.per_sm = two_per_sm ? 2 : 1;
        const long long slots = (long long)sm_count * c.per_sm;
        forced_hit = forced_nsplit() == ns;
        if (best == 0 || tiles * ns <= slots || forced_hit) {
            best = ns;
            bestq = c;
        }
    }
    if (best == 0) return CB_EUNSUPPORTED;
    q = bestq;
    return CB_OK;
}

// How the caller's filter becomes the packed filter of the convolution the kernel runs.
struct PackSpec {
    int mode, OC, IC, FHs, FWs, out_first, out_count;  // mode and geometry of pack_source
};

PackJob make_job(const PackSpec& ps, const ConvPlan& q, const float* W, float* dst, int FH, int FW) {
    PackJob j{};
    j.W = W; j.Wp = dst;
    j.OC = ps.OC; j.IC = ps.IC; j.FHs = ps.FHs; j.FWs = ps.FWs; j.FHc = FH; j.FWc = FW;
    j.OCp = q.OCp; j.CG = q.CG; j.x3 = q.x3; j.mode = ps.mode; j.out_first = ps.out_first; j.out_count = ps.out_count;
    j.total = (unsigned)(q.w_total_bytes / 4);
    return j;
}

int launch_pack(cb_ctx* err_ctx, const ConvEnv& env, const PackJob& j) {
    int grid = (int)((j.total + 255) / 256);
    if (grid > env.sm_count * 8) grid = env.sm_count * 8;
    cudaError_t e = launch_dep_on(env.stream, err_ctx && err_ctx->pdl, pack_filter_kernel, dim3((unsigned)grid), dim3(256), 0, 1, j);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(err_ctx, e, "pack_filter_kernel launch");
    return CB_OK;
}

// Launches the kernel on an already packed filter: Y (N x q.Cout x IH x IW) = taps (FH, FW, pH, pW) over
// X (N x q.Cin x IH x IW). in_batch / out_batch: elements between consecutive images (0 = densely packed).
int launch_conv(cb_ctx* err_ctx, const ConvEnv& env, const ConvPlan& q, const float* packed, const float* X, float* Y,
                const ConvEpilogue& ep, int N, int IH, int IW, int FH, int FW, int pH, int pW, long long in_batch,
                long long out_batch) {
    ConvParams p{};
    p.N = N; p.Cin = q.Cin; p.H = IH; p.W = IW; p.Cout = q.Cout;
    p.FH = FH; p.FW = FW; p.pH = pH; p.pW = pW;
    p.OCs = q.OCs; p.nsplit = q.nsplit; p.NQ = q.NQ; p.CG = q.CG; p.KS = q.KS;
    p.c_wrap = 2 * q.x3;
    p.f_wrap = p.c_wrap / kCB;
    p.NCB = (q.Cin + q.KS * kCB - 1) / (q.KS * kCB);
    p.L = q.L; p.LPI = IH / q.L;
    p.shared_rows = q.shared_rows; p.nblocks = q.nblocks;
    p.total_lines = (long long)N * p.LPI;
    if (p.total_lines > (1LL << 29)) return fail(err_ctx, CB_EUNSUPPORTED, "convolution: more than 2^29 lines of 32 pixels");
    p.tiles = (int)((p.total_lines + 3) / 4);
    p.stages = q.stages;
    p.epi_sets = q.OCs / 8 <= q.ew / 8 ? 2 : 1;
    int cols = 32;
    while (cols < 2 * q.NQ) cols <<= 1;
    p.tmem_cols = cols;
    p.w_bytes = (uint32_t)q.w_bytes;
    p.block_bytes = q.block_bytes;
    p.stage_bytes = q.stage_bytes;
    const uint64_t plane = (uint64_t)IH * IW;
    p.Out = Y;
    p.out_batch = out_batch ? out_batch : (long long)q.Cout * (long long)plane;
    p.ep = ep;
    p.status = env.status;
    p.trace = err_ctx ? err_ctx->trace : nullptr;
#ifdef CB_TRACE
    {
        const char* e = std::getenv("CB_DBG");
        p.dbg = e ? std::atoi(e) : 0;
    }
#endif
    const uint64_t in_stride = (uint64_t)(in_batch ? in_batch : (long long)q.Cin * (long long)plane) * 4;
    if (in_stride & 15u) return fail(err_ctx, CB_EUNSUPPORTED, "convolution: the input batch stride must be a multiple of 4 floats");

    CUtensorMap tmIn, tmW;
    int rc;
    if (q.shared_rows) {
        // 32-wide maps: (w, channel, row, image) so that one box of FH+3 rows lands as [row][channel][128 B]
        uint64_t dims[4] = {32, (uint64_t)q.Cin, (uint64_t)IH, (uint64_t)N};
        uint64_t str[3] = {plane * 4, 128, in_stride};
        uint32_t box[4] = {32u, (uint32_t)(q.KS * kCB), (uint32_t)q.nblocks, 1u};
        rc = encode_tmap(err_ctx, &tmIn, X, 4, dims, str, box, nullptr, 129);
    } else {
        // planes flattened to (H*W, C, N): a box is 32 consecutive floats of 8*KS channel planes, starting at pixel
        // (row * W) — a multiple of 4 floats, as TMA requires of the innermost coordinate. Pixels before the plane's
        // first row or after its last one, and channels >= C, are out of bounds and read as zero. (A box whose inner
        // extent is below the 128-byte swizzle span would be padded to 128 bytes per inner row in shared memory, so
        // the (W, H) plane is never used as two tensor-map dimensions when W < 32.)
        uint64_t dims[3] = {plane, (uint64_t)q.Cin, (uint64_t)N};
        uint64_t str[2] = {plane * 4, in_stride};
        uint32_t box[3] = {32u, (uint32_t)(q.KS * kCB), 1u};
        rc = encode_tmap(err_ctx, &tmIn, X, 3, dims, str, box, nullptr, 129);
    }
    if (rc != CB_OK) return rc;
    {
        // packed filter as (32 channels, OCp rows, (fh, channel group, fw) planes): a box is FW planes of OCs rows
        const uint64_t planes = (uint64_t)FH * q.CG * FW;
        uint64_t dims[3] = {32, (uint64_t)q.OCp, planes};
        uint64_t str[2] = {128, (uint64_t)q.OCp * 128};
        uint32_t box[3] = {32, (uint32_t)q.OCs, (uint32_t)FW};
        rc = encode_tmap(err_ctx, &tmW, packed, 3, dims, str, box, nullptr, 128);
        if (rc != CB_OK) return rc;
    }
    // Results leave through TMA unless the epilogue needs the old output before a ReLU, or the output is not 16-byte
    // aligned in every plane and image (TMA's base and stride rules).
    const long long out_stride_b = p.out_batch * 4;
    p.tma_out = (ep.accumulate && ep.relu) ? 0 : (ep.accumulate ? 2 : 1);
    if ((reinterpret_cast<uintptr_t>(Y) & 15u) || (out_stride_b & 15)) p.tma_out = 0;
    CUtensorMap tmOut = tmIn;  // placeholder when unused
    if (p.tma_out) {
        uint64_t dims[3] = {plane, (uint64_t)q.Cout, (uint64_t)N};
        uint64_t str[2] = {plane * 4, (uint64_t)out_stride_b};
        uint32_t box[3] = {32u, 8u, 1u};
        rc = encode_tmap(err_ctx, &tmOut, Y, 3, dims, str, box, nullptr, 0);
        if (rc != CB_OK) return rc;
    }
    const size_t smem = q.w_bytes + (size_t)p.stages * q.stage_bytes + 1024u * (size_t)q.ew + 1024;
    // per device: the opt-in shared-memory size is raised to the maximum once (several host threads may race here)
    static std::once_flag attr_once[64];
    static cudaError_t attr_error[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    typedef void (*KernelFn)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const ConvParams);
    static const KernelFn kernels[2][4] = {
        {umma_conv_kernel<8, TAPS_1>, umma_conv_kernel<8, TAPS_3>, umma_conv_kernel<8, TAPS_2L>, umma_conv_kernel<8, TAPS_2R>},
        {umma_conv_kernel<16, TAPS_1>, umma_conv_kernel<16, TAPS_3>, umma_conv_kernel<16, TAPS_2L>, umma_conv_kernel<16, TAPS_2R>}};
    auto raise_limits = [&]() -> cudaError_t {
        for (const auto& row : kernels)
            for (KernelFn k : row) {
                cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, env.smem_optin - 3072);
                if (e != cudaSuccess) return e;
            }
        return cudaSuccess;
    };
    cudaError_t attr_e;
    if (dev >= 0 && dev < 64) {
        std::call_once(attr_once[dev], [&] { attr_error[dev] = raise_limits(); });
        attr_e = attr_error[dev];
    } else {
        attr_e = raise_limits();
    }
    if (attr_e != cudaSuccess) return check_cuda(err_ctx, attr_e, "umma_conv_kernel attribute");
    const int slots = env.sm_count * q.per_sm;  // resident CTAs
    int per_split = slots / q.nsplit;
    if (per_split < 1) per_split = 1;
    if (per_split > p.tiles) per_split = p.tiles;
    const int grid = per_split * q.nsplit;
    const int taps = FW == 1 ? TAPS_1 : (FW == 3 ? TAPS_3 : (pW == 1 ? TAPS_2L : TAPS_2R));
    cudaError_t e = launch_dep_on(env.stream, err_ctx && err_ctx->pdl, kernels[q.ew == 8 ? 0 : 1][taps], dim3((unsigned)grid),
                                  dim3((unsigned)(64 + 32 * q.ew)), smem, 1, tmIn, tmW, tmOut, p);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(err_ctx, e, "umma_conv_kernel launch");
    return CB_OK;
}

}  // namespace

int launch_space_to_depth2(cb_ctx* ctx, const float* X, float* Xs, int N, int C, int H, int W) {
    const long long n_el = (long long)N * C * H * W;
    cudaError_t e = vec_ok(X, Xs, W) && n_el / 4 <= kMostItems
                        ? launch_dep(ctx, space_to_depth2_vec_kernel, dim3((unsigned)relayout_grid(ctx, n_el / 4, kRelayoutItems)), dim3(256), 0, X, Xs,
                                     PlaneIndex{FastDiv(W / 4), FastDiv(H), FastDiv(C)}, W / 2, (long long)(H / 2) * (W / 2), (uint32_t)(n_el / 4))
                        : launch_dep(ctx, space_to_depth2_kernel, dim3((unsigned)relayout_grid(ctx, n_el)), dim3(256), 0, X, Xs, C, H, W, n_el);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "space_to_depth2_kernel launch");
    ctx->launches += 1;
    return CB_OK;
}
int launch_subsample2(cb_ctx* ctx, const float* X, float* Xsub, long long NC, int H, int W) {
    const long long n_sub = NC * (H / 2) * (W / 2);
    const long long n_items = NC * (H / 2) * (W / 4);
    cudaError_t e = vec_ok(X, Xsub, W) && n_items <= kMostItems
                        ? launch_dep(ctx, subsample2_vec_kernel, dim3((unsigned)relayout_grid(ctx, n_items)), dim3(256), 0, X, Xsub, FastDiv(W / 4), W,
                                     (uint32_t)n_items)
                        : launch_dep(ctx, subsample2_kernel, dim3((unsigned)relayout_grid(ctx, n_sub)), dim3(256), 0, X, Xsub, NC, H, W, n_sub);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "subsample2_kernel launch");
    ctx->launches += 1;
    return CB_OK;
}

// ------------------------------------------------------------------------------------------ packed-filter cache
// With the cache on (cb_conv_cache_filters), a context keeps one packed copy per (filter pointer, geometry, pass) it
// has seen and re-packs it only after the caller announced a weight update: cb_filters_changed re-packs every cached
// filter in ONE launch, so a training step pays one pack launch instead of two per convolution. Filters the context's
// own update calls may have touched (cb_momentum*, cb_tensor_op) are re-packed lazily by the next convolution that
// uses them.
struct FilterCacheEntry {
    PackJob job;
    long long version;  // value of cb_ctx::filter_version when the packed copy was last written
};
// The jobs of one launch of pack_filter_table_kernel. A table whose launch was captured belongs to the caller's graph as well: it
// stays until the context goes.
struct FilterTable {
    std::vector<PackJob> jobs;
    PackJob* dev;
    bool captured;
};
struct FilterCache {
    std::vector<FilterCacheEntry> entries;
    std::vector<FilterTable> tables;  // the last one holds every entry (and forgotten ones), unless `changed`
    bool changed = true;
    long long biggest = 0;
    std::vector<std::pair<size_t, float*>> spare;  // packed copies of forgotten filters, by size, for the next filters
};

static bool same_job(const PackJob& a, const PackJob& b) {
    return a.W == b.W && a.OC == b.OC && a.IC == b.IC && a.FHs == b.FHs && a.FWs == b.FWs && a.FHc == b.FHc &&
           a.FWc == b.FWc && a.OCp == b.OCp && a.CG == b.CG && a.mode == b.mode && a.x3 == b.x3 && a.out_first == b.out_first &&
           a.out_count == b.out_count;
}

void filter_cache_destroy(cb_ctx* ctx) {
    FilterCache* fc = static_cast<FilterCache*>(ctx->filter_cache);
    if (!fc) return;
    for (FilterCacheEntry& e : fc->entries) cudaFree(e.job.Wp);
    for (FilterTable& t : fc->tables) cudaFree(t.dev);
    for (auto& s : fc->spare) cudaFree(s.second);
    delete fc;
    ctx->filter_cache = nullptr;
}

// Packed filter for this call: from the cache (packing it now if it is new or stale) or, with the cache off, packed
// into the context workspace.
static int packed_filter(cb_ctx* ctx, const ConvEnv& env, const ConvPlan& q, const PackSpec& ps, const float* W, int FH,
                         int FW, const float** out) {
    if (!ctx->filter_cache_on) {
        int rc = ensure_workspace(ctx, q.w_total_bytes);
        if (rc != CB_OK) return rc;
        const PackJob j = make_job(ps, q, W, static_cast<float*>(ctx->workspace), FH, FW);
        rc = launch_pack(ctx, env, j);
        if (rc != CB_OK) return rc;
        ctx->launches += 1;
        *out = j.Wp;
        return CB_OK;
    }
    if (!ctx->filter_cache) ctx->filter_cache = new FilterCache();
    FilterCache* fc = static_cast<FilterCache*>(ctx->filter_cache);
    PackJob want = make_job(ps, q, W, nullptr, FH, FW);
    FilterCacheEntry* hit = nullptr;
    for (FilterCacheEntry& e : fc->entries)
        if (same_job(e.job, want)) { hit = &e; break; }
    if (!hit) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(ctx->stream, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone)
            return fail(ctx, CB_ENOMEM, "a convolution filter was seen for the first time while the stream is being captured: "
                                        "run the same calls once before the capture so that its packed copy exists");
        for (size_t i = 0; i < fc->spare.size() && !want.Wp; ++i)
            if (fc->spare[i].first == q.w_total_bytes) {
                want.Wp = fc->spare[i].second;
                fc->spare.erase(fc->spare.begin() + (long)i);
            }
        if (!want.Wp) {
            void* d = nullptr;
            cudaError_t e = cudaMalloc(&d, q.w_total_bytes);
            if (e != cudaSuccess) {
                check_cuda(ctx, e, "packed filter cudaMalloc");
                return CB_ENOMEM;
            }
            want.Wp = static_cast<float*>(d);
        }
        fc->entries.push_back(FilterCacheEntry{want, -1});
        fc->changed = true;
        hit = &fc->entries.back();
    }
    if (hit->version != ctx->filter_version) {
        int rc = launch_pack(ctx, env, hit->job);
        if (rc != CB_OK) return rc;
        ctx->launches += 1;
        hit->version = ctx->filter_version;
    }
    *out = hit->job.Wp;
    return CB_OK;
}

bool filter_cache_fresh(const cb_ctx* ctx) {
    const FilterCache* fc = static_cast<const FilterCache*>(ctx->filter_cache);
    if (!ctx->filter_cache_on) return false;
    if (!fc) return true;  // nothing was ever packed: fp32 mode, or no map the tensor cores take
    for (const FilterCacheEntry& e : fc->entries)
        if (e.version != ctx->filter_version) return false;
    return true;
}

int filter_cache_size(const cb_ctx* ctx) {
    const FilterCache* fc = static_cast<const FilterCache*>(ctx->filter_cache);
    return fc ? (int)fc->entries.size() : 0;
}

// Re-packs every cached filter in one launch and marks them current.
int filter_cache_repack_all(cb_ctx* ctx) {
    ctx->filter_version += 1;
    FilterCache* fc = static_cast<FilterCache*>(ctx->filter_cache);
    if (!ctx->filter_cache_on || !fc || fc->entries.empty()) return CB_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool capturing = cudaStreamIsCapturing(ctx->stream, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone;
    if (fc->changed) {
        if (capturing) return CB_OK;  // filters first seen after the last table build: they re-pack lazily at their next use
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return check_cuda(ctx, e, "filter table rebuild");
        if (!fc->tables.empty() && !fc->tables.back().captured) {
            cudaFree(fc->tables.back().dev);
            fc->tables.pop_back();
        }
        FilterTable t{{}, nullptr, false};
        fc->biggest = 0;
        for (const FilterCacheEntry& en : fc->entries) {
            t.jobs.push_back(en.job);
            if (en.job.total > fc->biggest) fc->biggest = en.job.total;
        }
        void* d = nullptr;
        e = cudaMalloc(&d, sizeof(PackJob) * t.jobs.size());
        if (e == cudaSuccess) e = cudaMemcpy(d, t.jobs.data(), sizeof(PackJob) * t.jobs.size(), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            if (d) cudaFree(d);
            return check_cuda(ctx, e, "filter table upload");
        }
        t.dev = static_cast<PackJob*>(d);
        fc->tables.push_back(std::move(t));
        fc->changed = false;
    }
    FilterTable& table = fc->tables.back();
    table.captured = table.captured || capturing;
    int gx = (int)((fc->biggest + 255) / 256);
    if (gx > 64) gx = 64;
    if (gx < 1) gx = 1;
    cudaError_t e = launch_dep(ctx, pack_filter_table_kernel, dim3((unsigned)gx, (unsigned)table.jobs.size()), dim3(256), 0,
                               (const PackJob*)table.dev);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "pack_filter_table_kernel launch");
    ctx->launches += 1;
    for (FilterCacheEntry& en : fc->entries) en.version = ctx->filter_version;
    return CB_OK;
}

// Forgets the filters in [first, last): the memory may be released, and no later launch reads it, nor does a graph that captured
// one of the tables (its job does nothing from here on).
void filter_cache_forget(cb_ctx* ctx, const float* first, const float* last) {
    FilterCache* fc = static_cast<FilterCache*>(ctx->filter_cache);
    if (!fc) return;
    auto inside = [&](const PackJob& j) { return j.W >= first && j.W < last; };
    bool any = false;
    for (const FilterCacheEntry& e : fc->entries) any = any || inside(e.job);
    for (const FilterTable& t : fc->tables)
        for (const PackJob& j : t.jobs) any = any || inside(j);
    if (!any) return;
    cudaDeviceSynchronize();  // re-packs in flight, also those of graphs on other streams
    for (size_t i = fc->entries.size(); i-- > 0;)
        if (inside(fc->entries[i].job)) {
            fc->spare.emplace_back((size_t)fc->entries[i].job.total * sizeof(float), fc->entries[i].job.Wp);
            fc->entries.erase(fc->entries.begin() + (long)i);
        }
    for (FilterTable& t : fc->tables) {
        bool dirty = false;
        for (PackJob& j : t.jobs)
            if (inside(j)) {
                j.total = 0;
                j.W = nullptr;
                dirty = true;
            }
        if (dirty) cudaMemcpy(t.dev, t.jobs.data(), sizeof(PackJob) * t.jobs.size(), cudaMemcpyHostToDevice);
    }
}

static int conv_on_packed(cb_ctx* ctx, const ConvEnv& env, const ConvPlan& q, const PackSpec& ps, const float* W,
                          const float* X, float* Y, const ConvEpilogue& ep, int N, int IH, int IW, int FH, int FW, int pH,
                          int pW, long long in_batch, long long out_batch) {
    const float* packed = nullptr;
    int rc = packed_filter(ctx, env, q, ps, W, FH, FW, &packed);
    if (rc != CB_OK) return rc;
    rc = launch_conv(ctx, env, q, packed, X, Y, ep, N, IH, IW, FH, FW, pH, pW, in_batch, out_batch);
    if (rc != CB_OK) return rc;
    ctx->launches += 1;
    return CB_OK;
}

// Plan of one convolution of the path below: cin input channels of IH x IW, cout outputs. With x3 the contraction runs over
// three groups of channels (see umma_conv_fwd).
static int plan_pass(const cb_ctx* ctx, ConvPlan& q, bool x3, const float* X, int N, int cin, int cout, int IH, int IW, int FH, int FW,
                     int pH, int pW) {
    q = ConvPlan{};
    if (!x3) return plan_conv(q, ctx->max_smem_optin, ctx->sm_count, X, N, cin, cout, IH, IW, FH, FW, pH, pW);
    if (((long long)IH * IW) % 4 || (reinterpret_cast<uintptr_t>(X) & 15u)) return CB_EUNSUPPORTED;
    q.x3 = (cin + 7) / 8 * 8;
    q.ks_max = q.x3 % 32 == 0 ? 4 : (q.x3 % 16 == 0 ? 2 : 1);  // a stage's channels stay inside one group
    const int rc = plan_conv(q, ctx->max_smem_optin, ctx->sm_count, nullptr /* the scratch copy is aligned */, N, 3 * q.x3, cout, IH,
                             IW, FH, FW, pH, pW);
    if (rc != CB_OK) return rc;
    // A filter that only fits when the output channels are split four ways makes every CTA re-read the input for a quarter
    // of them, which pays on small maps and not on large ones (64 -> 64: 21 us against 36 composed at 8 x 8).
    if (q.nsplit > 2 && ((long long)N * (IH / q.L) + 3) / 4 > ctx->sm_count) return CB_EUNSUPPORTED;
    return CB_OK;
}

// 3xTF32 scratch of one pass over `channels` input channels and their lo parts; of a layer, when the block has to grow:
// `layer` is the most channels that either of its tensors has.
static int ensure_split_scratch(cb_ctx* ctx, int N, int channels, int layer, long long plane) {
    auto bytes = [&](int c) { return (size_t)N * 2 * ((c + 7) / 8 * 8) * plane * sizeof(float); };
    return ensure_workspace3(ctx, bytes(channels), bytes(layer));
}

// One planned convolution on `X` (N images of `cin` planes, in_batch floats apart or dense). With q.x3 the input is first
// written as [x ; x_lo] to scratch; `layer`: see ensure_split_scratch.
static int run_pass(cb_ctx* ctx, const ConvEnv& env, const ConvPlan& q, const PackSpec& ps, const float* W, const float* X, int cin,
                    int layer, float* Y, const ConvEpilogue& ep, int N, int IH, int IW, int FH, int FW, int pH, int pW, long long in_batch,
                    long long out_batch) {
    if (q.x3) {
        const long long plane = (long long)IH * IW, per = cin * plane, perp = q.x3 * plane;
        if (in_batch & 3) return CB_EUNSUPPORTED;
        int rc = ensure_split_scratch(ctx, N, q.x3, layer, plane);
        if (rc != CB_OK) return rc;
        float* X2 = static_cast<float*>(ctx->workspace3);
        const long long items = (long long)N * (perp / 4);
        if (items > kMostItems) return CB_EUNSUPPORTED;
        cudaError_t e = launch_dep(ctx, tf32_split2_kernel, dim3((unsigned)relayout_grid(ctx, items, kRelayoutItems)), dim3(256), 0, X, X2,
                                   per / 4, FastDiv(perp / 4), in_batch ? in_batch : per, (uint32_t)items);
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e != cudaSuccess) return check_cuda(ctx, e, "tf32_split2_kernel launch");
        ctx->launches += 1;
        X = X2;
        in_batch = 2 * perp;
    }
    return conv_on_packed(ctx, env, q, ps, W, X, Y, ep, N, IH, IW, FH, FW, pH, pW, in_batch, out_batch);
}

int launch_space_to_depth2_split(cb_ctx* ctx, const float* X, float* X2, int N, int C, int Cp, int H, int W) {
    const long long items = (long long)N * C * H * (W / 4);
    if (items > kMostItems) return CB_EUNSUPPORTED;
    cudaError_t e = launch_dep(ctx, space_to_depth2_split_kernel, dim3((unsigned)relayout_grid(ctx, items, kRelayoutItems)), dim3(256), 0, X,
                               X2, PlaneIndex{FastDiv(W / 4), FastDiv(H), FastDiv(C)}, Cp, W / 2, (long long)(H / 2) * (W / 2), (uint32_t)items);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "space_to_depth2_split_kernel launch");
    ctx->launches += 1;
    return CB_OK;
}

// Forward (dgrad_of = false: Y = conv(W, X), full epilogue) or data gradient (dgrad_of = true: X is dY, Y is dX; of the
// epilogue only `accumulate` applies). Returns CB_EUNSUPPORTED, before any work is queued, for geometries outside the
// tensor-core kernel.
//
// x3: 3xTF32 in ONE pass of the kernel. With x = x_hi + x_lo and w = w_hi + w_lo, y = x_hi w_hi + x_lo w_hi + x_hi w_lo is a
// single convolution over three groups of input channels, [x_lo ; x ; x] against [w ; w_lo ; w], because the tensor core itself
// takes the hi part of what it reads. The two corrections come first: TMEM truncates every addition at the accumulator's
// magnitude, which they leave small (against double, 64 -> 64 channels, 3x3: 5.3e-7, and 2.3e-6 with x w first). A small kernel
// writes [x ; x_lo] (dense scratch; for stride 2 in the phase-split layout), the packed filter holds [w ; w_lo] (cached like any
// other), the kernel reads x a second time and w twice. Everything accumulates in one TMEM accumulator and leaves through the
// ordinary epilogue. (Three passes into temporaries, their lo parts and a sum took 229 us for the three passes of the layer 32 -> 64,
// stride 2 at 32 x 32, batch 128.)
int umma_conv_fwd(cb_ctx* ctx, const float* W, const float* X, float* Y, const ConvEpilogue& ep, int N, int IC, int IH,
                  int IW, int OC, int FH, int FW, int sH, int sW, int pH, int pW, bool dgrad_of, long long in_batch,
                  long long out_batch, bool x3) {
    ConvEnv env{ctx->stream, ctx->sm_count, ctx->max_smem_optin, ctx->d_status};
    ConvPlan q{};
    int rc;
    const char* name = x3 ? "umma_3xtf32" : "umma_tf32";
    if (sH == 1 && sW == 1) {
        // ---- stride 1: 1x1 (pad 0) or 3x3 (pad 1) per axis
        if (!((FH == 1 && pH == 0) || (FH == 3 && pH == 1))) return CB_EUNSUPPORTED;
        if (!((FW == 1 && pW == 0) || (FW == 3 && pW == 1))) return CB_EUNSUPPORTED;
        const int cin = dgrad_of ? OC : IC, cout = dgrad_of ? IC : OC;
        rc = plan_pass(ctx, q, x3, X, N, cin, cout, IH, IW, FH, FW, pH, pW);
        if (rc != CB_OK) return rc;
        const PackSpec ps{dgrad_of ? PACK_DGRAD : PACK_FWD, OC, IC, FH, FW, 0, 0};
        rc = run_pass(ctx, env, q, ps, W, X, cin, IC > OC ? IC : OC, Y, ep, N, IH, IW, FH, FW, pH, pW, in_batch, out_batch);
        if (rc == CB_OK) ctx->last_kernel = name;
        return rc;
    }
    // ---- stride 2 (square): 3x3 pad 1 through the 4 input phases, 1x1 pad 0 through phase (0,0); dense tensors only
    if (sH != 2 || sW != 2 || FH != FW || pH != pW || (IH & 1) || (IW & 1)) return CB_EUNSUPPORTED;
    if (!((FH == 3 && pH == 1) || (FH == 1 && pH == 0))) return CB_EUNSUPPORTED;
    if (in_batch || out_batch) return CB_EUNSUPPORTED;
    const int H2 = IH / 2, W2 = IW / 2;
    const long long plane2 = (long long)H2 * W2;
    const ConvEpilogue plain{};
    if (FH == 1) {
        // Y = W * X[:, :, ::2, ::2]  /  dX[:, :, ::2, ::2] = W^T dY, zero elsewhere
        const int cin = dgrad_of ? OC : IC;
        rc = plan_pass(ctx, q, x3, dgrad_of ? X : nullptr /* the sub-sampled copy is aligned */, N, cin, dgrad_of ? IC : OC, H2, W2, 1, 1,
                       0, 0);
        if (rc != CB_OK) return rc;
        const size_t sub_bytes = (size_t)N * IC * plane2 * sizeof(float);
        rc = ensure_workspace2(ctx, sub_bytes);
        if (rc != CB_OK) return rc;
        float* sub = static_cast<float*>(ctx->workspace2);
        const PackSpec ps{dgrad_of ? PACK_DGRAD : PACK_FWD, OC, IC, 1, 1, 0, 0};
        if (!dgrad_of) {
            rc = launch_subsample2(ctx, X, sub, (long long)N * IC, IH, IW);
            if (rc == CB_OK) rc = run_pass(ctx, env, q, ps, W, sub, cin, IC > OC ? IC : OC, Y, ep, N, H2, W2, 1, 1, 0, 0, 0, 0);
        } else {
            rc = run_pass(ctx, env, q, ps, W, X /* = dY */, cin, IC > OC ? IC : OC, sub, plain, N, H2, W2, 1, 1, 0, 0, 0, 0);
            const long long n_full = (long long)N * IC * IH * IW;
            if (rc == CB_OK) {
                if (vec_ok(sub, Y, IW) && n_full / 4 <= kMostItems)
                    launch_dep(ctx, upsample2_zero_vec_kernel, dim3((unsigned)relayout_grid(ctx, n_full / 4)), dim3(256), 0,
                               (const float*)sub, Y /* = dX */, FastDiv(IW / 4), (uint32_t)(n_full / 4), ep.accumulate ? 1 : 0);
                else
                    launch_dep(ctx, upsample2_zero_kernel, dim3((unsigned)relayout_grid(ctx, n_full)), dim3(256), 0, (const float*)sub,
                               Y /* = dX */, IH, IW, n_full, ep.accumulate ? 1 : 0);
                ctx->launches += 1;
            }
        }
        if (rc != CB_OK) return rc;
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return check_cuda(ctx, e, "stride-2 1x1 convolution");
        ctx->last_kernel = name;
        return CB_OK;
    }
    const int C4 = 4 * IC;
    const size_t s2d_bytes = (size_t)N * C4 * plane2 * sizeof(float);
    if (!dgrad_of) {
        // Xs[n][phase*IC + c] = X[n][c][phase rows / cols]; Y = 2x2 convolution (taps at -1, 0) over the 4*IC planes
        const PackSpec ps{PACK_S2_FWD, OC, IC, 3, 3, 0, 0};
        rc = plan_pass(ctx, q, x3, nullptr /* the re-laid-out copy is aligned */, N, C4, OC, H2, W2, 2, 2, 1, 1);
        if (rc != CB_OK) return rc;
        if (x3) {
            if (!vec_ok(X, nullptr, IW)) return CB_EUNSUPPORTED;
            const long long perp = 2LL * q.x3 * plane2;
            rc = ensure_split_scratch(ctx, N, q.x3, C4 > OC ? C4 : OC, plane2);
            if (rc != CB_OK) return rc;
            float* X2 = static_cast<float*>(ctx->workspace3);
            rc = launch_space_to_depth2_split(ctx, X, X2, N, IC, q.x3, IH, IW);
            if (rc == CB_OK) rc = conv_on_packed(ctx, env, q, ps, W, X2, Y, ep, N, H2, W2, 2, 2, 1, 1, perp, 0);
        } else {
            rc = ensure_workspace2(ctx, s2d_bytes);
            if (rc != CB_OK) return rc;
            float* Xs = static_cast<float*>(ctx->workspace2);
            rc = launch_space_to_depth2(ctx, X, Xs, N, IC, IH, IW);
            if (rc == CB_OK) rc = conv_on_packed(ctx, env, q, ps, W, Xs, Y, ep, N, H2, W2, 2, 2, 1, 1, 0, 0);
        }
        if (rc == CB_OK) ctx->last_kernel = name;
        return rc;
    }
    // data gradient: dXs (4*IC phase planes) = adjoint 2x2 convolution (taps at 0, +1) over dY, in channel groups small
    // enough for the accumulator (FW * roundup16(channels) <= 256), then interleaved back into dX
    int groups = 1;
    while (groups <= 4 && 2 * ((C4 / groups + 15) / 16 * 16) > 256) groups *= 2;
    if (groups > 4) return CB_EUNSUPPORTED;
    const int per_group = C4 / groups;
    rc = plan_pass(ctx, q, x3, X /* = dY */, N, OC, per_group, H2, W2, 2, 2, 0, 0);
    if (rc == CB_OK) rc = ensure_workspace2(ctx, s2d_bytes, x3 ? 2 * s2d_bytes : 0);  // 3xTF32: the weight gradient has lo parts too
    if (rc != CB_OK) return rc;
    float* dXs = static_cast<float*>(ctx->workspace2);
    for (int g = 0; g < groups; ++g) {
        const PackSpec ps{PACK_S2_DGRAD, OC, IC, 3, 3, g * per_group, per_group};
        rc = run_pass(ctx, env, q, ps, W, X /* = dY */, OC, C4 > OC ? C4 : OC, dXs + (size_t)g * N * per_group * plane2, plain, N, H2, W2, 2, 2, 0, 0, 0,
                      0);
        if (rc != CB_OK) return rc;
    }
    const long long n_full = (long long)N * IC * IH * IW;
    cudaError_t e = vec_ok(dXs, Y, IW) && n_full / 4 <= kMostItems
                        ? launch_dep(ctx, depth_to_space2_vec_kernel, dim3((unsigned)relayout_grid(ctx, n_full / 4, kRelayoutItems)), dim3(256), 0,
                                     (const float*)dXs, Y /* = dX */, PlaneIndex{FastDiv(IW / 4), FastDiv(IH), FastDiv(IC)}, N, W2, plane2,
                                     FastDiv(per_group), (uint32_t)(n_full / 4), ep.accumulate ? 1 : 0)
                        : launch_dep(ctx, depth_to_space2_kernel, dim3((unsigned)relayout_grid(ctx, n_full)), dim3(256), 0,
                                     (const float*)dXs, Y /* = dX */, N, IC, IH, IW, per_group, n_full, ep.accumulate ? 1 : 0);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "depth_to_space2_kernel launch");
    ctx->launches += 1;
    ctx->last_kernel = name;
    return CB_OK;
}

// ------------------------------------------------------------------------------------------ allocation-free forward
// cb_conv_fwd_noalloc: the tensor-core forward convolution for callers that must not allocate device memory —
// code running under a memory manager that has already claimed the whole GPU (so cudaMalloc would fail), code
// on a latency-critical path where cudaMalloc's implicit device synchronisation is unacceptable, and code that
// runs while a stream is being captured (allocation calls are not allowed there). The ordinary entry point keeps
// its packed filter in a context workspace that grows with cudaMalloc; this one keeps it in the fixed array below,
// which every GPU that loads the library holds from load to exit (160 KiB + one status word).
namespace {

constexpr int kNoAllocPackFloats = 40960;  // 160 KiB: enough for a 64 -> 64 channel 3x3 filter (147 456 bytes)
static __device__ __align__(256) float g_noalloc_pack[kNoAllocPackFloats];
static __device__ __align__(16) int g_noalloc_status;

struct NoAllocDevice {
    std::once_flag once;
    cudaError_t init_error = cudaSuccess;
    int major = 0;
    float* pack = nullptr;  // device address of g_noalloc_pack on this GPU (the symbol itself is a host stand-in)
    int* status = nullptr;
    int sm_count = 0;
    int smem_optin = 0;
};
constexpr int kNoAllocMaxDevices = 64;
NoAllocDevice g_noalloc_dev[kNoAllocMaxDevices];

int noalloc_fail(char* err, int err_len, int code, const char* msg) {
    if (err && err_len > 0) snprintf(err, (size_t)err_len, "%s", msg);
    return code;
}

// Makes `device` current for the duration of a call and puts the caller's device back on every return path.
struct DeviceScope {
    int prev = -1;
    cudaError_t error;
    explicit DeviceScope(int device) {
        error = cudaGetDevice(&prev);
        if (error == cudaSuccess && prev != device) error = cudaSetDevice(device);
    }
    ~DeviceScope() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

// Once per device, with that device current: resolves the device addresses of the static arrays and reads the
// attributes the launch needs. Safe when several host threads make their first call at the same time.
NoAllocDevice* noalloc_device(int device, char* err, int err_len, int* rc) {
    NoAllocDevice& d = g_noalloc_dev[device];
    std::call_once(d.once, [&] {
        cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&d.pack), g_noalloc_pack);
        if (e == cudaSuccess) e = cudaGetSymbolAddress(reinterpret_cast<void**>(&d.status), g_noalloc_status);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&d.major, cudaDevAttrComputeCapabilityMajor, device);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, device);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
        d.init_error = e;
    });
    if (d.init_error != cudaSuccess) {
        *rc = noalloc_fail(err, err_len, CB_ECUDA, cudaGetErrorString(d.init_error));
        return nullptr;
    }
    if (d.major != 10) {
        *rc = noalloc_fail(err, err_len, CB_EUNSUPPORTED, "this library only carries sm_100a code");
        return nullptr;
    }
    return &d;
}

}  // namespace
}  // namespace cb

extern "C" int cb_conv_fwd_noalloc(int device, void* cuda_stream, const float* W, const float* X, float* Y,
                                   const float* bias, int N, int IC, int IH, int IW, int OC, int FH, int FW, int sH,
                                   int sW, int pH, int pW, int relu, char* err, int err_len) {
    using namespace cb;
    if (err && err_len > 0) err[0] = 0;
    if (device < 0 || device >= kNoAllocMaxDevices) return noalloc_fail(err, err_len, CB_EINVAL, "device index out of range");
    if (N < 0 || IC < 1 || OC < 1 || IH < 1 || IW < 1) return noalloc_fail(err, err_len, CB_EINVAL, "bad extent");
    if (!W || !X || !Y) return noalloc_fail(err, err_len, CB_EINVAL, "null operand");
    if (sH != 1 || sW != 1 || !((FH == 1 && pH == 0) || (FH == 3 && pH == 1)) ||
        !((FW == 1 && pW == 0) || (FW == 3 && pW == 1)) || (IW != 8 && IW != 16 && IW != 32) || (IH % (32 / IW)) ||
        (reinterpret_cast<uintptr_t>(X) & 15u))
        return noalloc_fail(err, err_len, CB_EUNSUPPORTED,
                            "cb_conv_fwd_noalloc covers stride 1, 1x1 (pad 0) / 3x3 (pad 1) filters, map width 8, 16 or 32 "
                            "and a 16-byte aligned input");
    const size_t w_need = (size_t)FH * ((IC + 31) / 32) * FW * ((OC + 15) / 16 * 16) * kRowBytes;
    if (FW * ((OC + 15) / 16 * 16) > 256) return noalloc_fail(err, err_len, CB_EUNSUPPORTED, "FW * OC (rounded up to 16) exceeds 256");
    if (w_need > sizeof(float) * (size_t)kNoAllocPackFloats) {
        char msg[200];
        snprintf(msg, sizeof(msg), "packed filter needs %zu bytes; the static scratch of cb_conv_fwd_noalloc holds %zu",
                 w_need, sizeof(float) * (size_t)kNoAllocPackFloats);
        return noalloc_fail(err, err_len, CB_EINVAL, msg);
    }
    if (N == 0) return CB_OK;

    DeviceScope scope(device);
    if (scope.error != cudaSuccess) return noalloc_fail(err, err_len, CB_ECUDA, cudaGetErrorString(scope.error));
    int rc = CB_OK;
    NoAllocDevice* d = noalloc_device(device, err, err_len, &rc);
    if (!d) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);

    ConvPlan q{};
    if (plan_conv(q, d->smem_optin, d->sm_count, X, N, IC, OC, IH, IW, FH, FW, pH, pW) != CB_OK)
        return noalloc_fail(err, err_len, CB_EUNSUPPORTED, "geometry outside the tensor-core convolution kernel");
    // The scratch keeps the previous call's contents: the pack kernel rewrites all w_bytes (padding included). The
    // status word is NOT cleared here, so that a device-side timeout of an earlier call stays visible until
    // cb_conv_fwd_noalloc_status reads (and clears) it.
    ConvEnv env{stream, d->sm_count, d->smem_optin, d->status};
    const PackSpec ps{PACK_FWD, OC, IC, FH, FW, 0, 0};
    cb_ctx messages;  // host-side only: collects the text of a CUDA / tensor-map error; owns no device memory
    messages.device = device;
    ConvEpilogue ep{};
    ep.bias = bias;
    ep.relu = relu ? 1 : 0;
    rc = launch_pack(&messages, env, make_job(ps, q, W, d->pack, FH, FW));
    if (rc == CB_OK) rc = launch_conv(&messages, env, q, d->pack, X, Y, ep, N, IH, IW, FH, FW, pH, pW, 0, 0);
    if (rc != CB_OK)
        return noalloc_fail(err, err_len, rc, messages.last_error.empty() ? "kernel launch or tensor map encoding failed"
                                                                          : messages.last_error.c_str());
    return CB_OK;
}

extern "C" int cb_conv_fwd_noalloc_status(int device, void* cuda_stream, char* err, int err_len) {
    using namespace cb;
    if (err && err_len > 0) err[0] = 0;
    if (device < 0 || device >= kNoAllocMaxDevices) return noalloc_fail(err, err_len, CB_EINVAL, "device index out of range");
    DeviceScope scope(device);
    if (scope.error != cudaSuccess) return noalloc_fail(err, err_len, CB_ECUDA, cudaGetErrorString(scope.error));
    int rc = CB_OK;
    NoAllocDevice* d = noalloc_device(device, err, err_len, &rc);
    if (!d) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    cudaError_t e = cudaStreamSynchronize(stream);
    int st = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&st, d->status, sizeof(int), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return noalloc_fail(err, err_len, CB_ECUDA, cudaGetErrorString(e));
    if (st != 0) {
        e = cudaMemsetAsync(d->status, 0, sizeof(int), stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        char msg[160];
        snprintf(msg, sizeof(msg), "a bounded device-side wait of cb_conv_fwd_noalloc expired: device status %d (%s)", st,
                 status_name(st));
        return noalloc_fail(err, err_len, CB_ETIMEOUT, msg);
    }
    return CB_OK;
}
