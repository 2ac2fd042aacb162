// Convolution forward and data gradient at fp32 accuracy on the tensor cores, for filters of a few taps at stride 1 and 2: the arithmetic of
// split_core.cuh (three bf16 pieces a value, six products, short sums in TMEM), but a value is fetched and split
// once for all the taps that read it. conv_split.cu's gather does that for every tap, nine times for a 3x3 filter, and is bound by it.
//
// Layout: all output pixels of the batch lie on one line, rows of GW and images of GH rows, with as many unused columns and rows as the taps
// reach beyond the tensor; those read 0. A tap is then one constant distance on that line. Shared memory holds, per piece and group of
// 8 channels, 16 bytes (8 bf16) a position: K-major core matrices without swizzle whose 8 rows are 8 neighbouring positions, so a UMMA's
// A operand for a tap is the same memory from another first position on. A stride of 2 splits the input into the four planes of even and odd
// rows and columns, each a line of its own; the data gradient of stride 2 is two sets of pixels, of even and odd rows, with the even and odd
// columns side by side in the product (plan_patch).
//
// A UMMA of few columns is bound by reading its 128 rows of A, so the pieces of the filter are stacked in N: x1 meets [y1 y2 y3], x2
// [y1 y2] and x3 [y1], in three groups of accumulator columns for products of the orders 1, 2^-8 and 2^-16: 3 UMMAs a step instead of 6
// (N = 32: 144 clocks instead of 240). The groups are added smallest first, then to the sums in registers.
//
// Roles: patch warps (global memory -> registers -> pieces), one or two issuing warps, one that copies the filter's pieces, which
// pack_patch_filter has made before, and summing warps, which help with the first patch.
//
// us, conv_split.cu's gather / here: 32 -> 32 3x3, 28 x 28, batch 32, forward 14.6 / 10.9, data gradient 17.6 / 10.9; 32 -> 64 3x3 stride 2, 32 x
// 32, batch 128 21.1 / 18.2, its data gradient 37.2 / 25.7; 128 -> 128 3x3, 4 maps of 56 x 56 37.7 / 32.4 and 65.6 / 32.6; 16 -> 32 5x5, 46 x 46,
// batch 23 29.0 / 19.0 and 61.2 / 26.0. What bounds it now: in the first of these 3.2 us are pack_patch_filter's, 2.6 a CTA's start until its first patch is there; then
// UMMAs, 60 clocks each whatever their width, and between blocks of them the hand-over of accumulators (a second issuing warp, a
// second CTA on the SM). One CTA an SM that walks over tiles, fetching ahead, took 12.7 us there: what a patch warp executes for a run of
// 32 positions x 8 channels, ~150 instructions a chain of 1500 clocks, was then the bound. Error against fp64 at K = 288, 576,
// 1152, in one share: 0.90, 0.98, 1.02e-7 of the norm; the gathers' 0.94, 1.02, 1.16e-7 (1.03e-7 in two shares).
#include "conv_gather.cuh"
#include "conv_patch.h"
#include "split_core.cuh"

namespace cb {

using namespace gather;

namespace {

constexpr int kMaxRing = 4;   // slots of the patch and the filter ring at most
constexpr int kChain = 5;     // steps of 16 k whose sum stays in TMEM
constexpr int kGroup = 8;     // blocks whose sums are added one after another
constexpr int kPackCols = 8;  // columns of a block of pack_patch_filter

// Two CTAs an SM, so that one computes while the other starts, adds or stores. Each has 256 columns of TMEM: two accumulators of 3 x 32
// columns, each with an issuing warp of its own, or one of 3 x 64. Twice 512 threads leave 64 registers a thread: 4 to 60 bytes of
// spill stores (ptxas), the price of the second CTA.
template <int BN_>
struct PatchShape {
    static constexpr int BM = 128, BN = BN_, NT = 512, kCtas = 2;
    static constexpr int kSumWarps = 8, kCols = BN / 2;
    static constexpr int kAcc = BN == 32 ? 2 : 1, kIssuer = 16 - 1 - kAcc, kCopier = 15, kPatchWarps = kIssuer - kSumWarps;
    static constexpr uint32_t kTmemCols = 256;
    static constexpr uint32_t kRowsB = 3u * BN * 16u;            // a group of 8 k of a step of the filter: the three pieces' rows
    static constexpr uint32_t kStepB = 2u * kRowsB;
    static constexpr int kSlice = 16;                            // k of a piece of the second pass
    static constexpr uint32_t kStaging = BN * 512u + kSlice * (BM + BN) * 4u;  // the tile's sums; a slice of the second pass
};

struct __align__(8) PatchBarriers {
    uint64_t pfull[kMaxRing], pempty[kMaxRing], ffull[kMaxRing], fempty[kMaxRing], tfull[2], tempty[2], drain;
    uint32_t tmem_base;
    int abort_flag;
    int cut;           // of the second pass: factors below split::kWhole; the largest factor's magnitude, as bits
    unsigned largest;
};

// The parameters arrive 64 bytes a miss: every warp asks for a part, or the misses come one after the other as the code gets to them.
__device__ __forceinline__ void fetch_parameters(const PatchParams& q, int warp, int warps) {
    for (int at = warp * 16; at < (int)(sizeof(PatchParams) / 4); at += warps * 16) asm volatile("" ::"r"(reinterpret_cast<const int*>(&q)[at]));
}

// What a CTA does at a time: a tile of pixels of a set, a column tile, a share of the contraction.
struct PatchItem {
    int set, part, line0, j0;
    int chunk0, chunk1, chunks_all;
    __device__ __forceinline__ PatchItem(const PatchParams& q, uint32_t item, int bn) {
        uint32_t tile, rest, column;
        rest = q.tiles.split(item, tile);
        rest = q.columns.split(rest, column);
        set = (int)q.splits.split(rest, rest);
        part = (int)rest;
        line0 = (int)tile * 128;
        j0 = (int)column * bn;
        chunks_all = q.sets[set].full.steps ? q.chunks : 0;
        chunk0 = part * q.p.per_split;
        chunk1 = min(chunks_all, chunk0 + q.p.per_split);
    }
    __device__ __forceinline__ const ChunkSteps& steps(const PatchParams& q, int chunk) const {
        return chunk + 1 < chunks_all ? q.sets[set].full : q.sets[set].last;
    }
};

// Two runs of 32 positions x 8 channels of a patch on their way from memory to a warp's pieces of it: of one plane each, or (pairs, even
// and odd columns of a stride of 2) the same positions of two planes by 8-byte loads.
struct PatchLoads {
    float v[2][8];
    uint32_t dst[2];  // in a slot; ~0: nothing
    uint32_t piece;
};
__device__ __forceinline__ int patch_runs(const PatchParams& q, const PatchItem& it, int chunk) {
    return (int)q.sets[it.set].segs.d * 2 * it.steps(q, chunk).channels16;
}
// Runs i and i + of of a chunk; pairs: i.
__device__ __forceinline__ void load_patch(const PatchParams& q, const PatchItem& it, int chunk, int runs, int i, int of, PatchLoads& l) {
    const GatherParams& p = q.p;
    const PixelSet& s = p.sets[it.set];
    const PatchSet& ps = q.sets[it.set];
    const int lane = threadIdx.x & 31, pairs = ps.pairs, cells = (ps.planes * q.px) >> pairs, plane_in = p.H * p.W;
    const uint32_t row_bytes = (uint32_t)(ps.planes * q.px) * 16u;
    l.piece = (uint32_t)(q.cw >> 3) * row_bytes;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        if (pairs && u == 1) break;
        uint32_t seg;
        const uint32_t run = i + u * of, g = ps.segs.split(run, seg), cell = seg * 32 + lane;
        const bool here = run < (uint32_t)runs && cell < (uint32_t)cells;
        // where the position lies in the input, if anywhere (0 is read elsewhere)
        const int plane = (((int)cell >= q.px) + ((int)cell >= 2 * q.px) + ((int)cell >= 3 * q.px)), at = it.line0 + ps.first + (int)cell - plane * q.px;
        uint32_t in, col;
        const uint32_t n = q.image.split((uint32_t)max(at, 0), in), row = q.row.split(in, col);
        const int h = (int)row * s.hs + ps.ph[plane << pairs], w = (int)col * s.ws + ps.pw[plane << pairs], c = chunk * q.cw + 8 * (int)g;
        const bool ok = here && at >= 0 && (int)n < p.N && h < p.H && w < p.W;
        const float* src = p.In + (long long)n * p.in_batch + (long long)c * plane_in + h * p.W + w;
        const int channels = ok ? p.C - c : 0;
        l.dst[u] = here ? g * row_bytes + (cell + (pairs ? plane * q.px : 0)) * 16u : ~0u;
        if (pairs) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t@q ld.global.nc.v2.f32 {%0, %1}, [%2];\n\t}"
                    : "=f"(l.v[0][e]), "=f"(l.v[1][e]) : "l"(split::step(src, (uint32_t)plane_in * 4u, e)), "r"((int)(e < channels)));
            l.dst[1] = here ? l.dst[0] + (uint32_t)q.px * 16u : ~0u;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) l.v[u][e] = split::load_if(split::step(src, (uint32_t)plane_in * 4u, e), e < channels);
        }
    }
}
__device__ __forceinline__ void store_patch(const PatchLoads& l, uint32_t slot) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        if (l.dst[u] == ~0u) continue;
        uint32_t x[3][4];
#pragma unroll
        for (int e = 0; e < 8; e += 2) split::split2(l.v[u][e], l.v[u][e + 1], x[0][e / 2], x[1][e / 2], x[2][e / 2]);
#pragma unroll
        for (int t = 0; t < 3; ++t)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(slot + l.dst[u] + t * l.piece), "r"(x[t][0]), "r"(x[t][1]), "r"(x[t][2]), "r"(x[t][3]) : "memory");
    }
}

// Share `mine` of `of` warps of a chunk's patch.
__device__ __forceinline__ void fetch_patch(const PatchParams& q, const PatchItem& it, uint32_t slot, int chunk, int mine, int of) {
    const int runs = patch_runs(q, it, chunk);
    for (int i = mine; i < runs; i += q.sets[it.set].pairs ? of : 2 * of) {
        PatchLoads l;
        load_patch(q, it, chunk, runs, i, of, l);
        store_patch(l, slot);
    }
    fence_proxy_async_smem();
    __syncwarp();
}

// The second pass of split::Again, by the summing warps alone: the share's products once more by fp32 FMAs in the CUDA cores' order, for the
// outputs of warps that want it; (row, first ...) are a thread's.
template <class S, bool FOLD>
__device__ __noinline__ void sum_again(const PatchParams& q, const PatchItem& it, PatchBarriers& b, uint32_t slice, uint32_t mine, int row, int first, bool wanted) {
    const GatherParams& p = q.p;
    const PixelSet& s = p.sets[it.set];
    const int taps = s.TH * s.TW, channels = max(min(it.chunk1 * q.cw, p.C) - it.chunk0 * q.cw, 0), K = channels * taps, plane_in = p.H * p.W;
    constexpr int kThreads = 32 * S::kSumWarps;
    const int tid = threadIdx.x, r = tid & (S::BM - 1);
    int n, u, v;
    const bool live = q.pixel_of(s, p.N, it.line0 + r, n, u, v);
    const float* img = p.In + (live ? (long long)n * p.in_batch : 0);
    float plain[S::kCols];
#pragma unroll
    for (int c = 0; c < S::kCols; ++c) plain[c] = 0.f;
    if (tid == 0) {
        b.cut = 0;
        b.largest = 0;
    }
    for (int k0 = 0; k0 < K; k0 += S::kSlice) {
        asm volatile("bar.sync 3, %0;" ::"n"(kThreads) : "memory");
        unsigned largest = 0;
        auto put = [&](int word, float x) {
            const float m = fabsf(x);
            if (m > 0.f && m < split::kWhole) b.cut = 1;
            if (m <= split::kFinite) largest = max(largest, __float_as_uint(m));
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(slice + (uint32_t)word * 4u), "f"(x) : "memory");
        };
        auto place = [&](int k, int& tap, int& c) {
            tap = p.tap_major ? k / channels : k % taps;
            c = it.chunk0 * q.cw + (p.tap_major ? k - tap * channels : k / taps);
        };
        for (int k = tid / S::BM; k < S::kSlice; k += kThreads / S::BM) {
            float x = 0.f;
            if (live && k0 + k < K) {
                int tap, c;
                place(k0 + k, tap, c);
                const int th = tap / s.TW, tw = tap - th * s.TW, h = s.hs * u + s.hb + p.sgn * th, w = s.ws * v + s.wb + p.sgn * tw;
                if ((unsigned)h < (unsigned)p.H && (unsigned)w < (unsigned)p.W) x = __ldg(img + (long long)c * plane_in + h * p.W + w);
            }
            put(k * S::BM + r, x);
        }
        for (int i = tid; i < S::kSlice * S::BN; i += kThreads) {
            const int k = i / S::BN, j = it.j0 + i % S::BN;
            float y = 0.f;
            if (k0 + k < K && j < q.cols) {
                int tap, c;
                place(k0 + k, tap, c);
                const int th = tap / s.TW, at = q.filter_of<FOLD>(it.set, th, tap - th * s.TW, j);
                if (at >= 0) y = __ldg(p.Wt + (long long)(FOLD ? j >> 1 : j) * p.w_out + (long long)c * p.w_ch + at);
            }
            put(S::kSlice * S::BM + i, y);
        }
        largest = __reduce_max_sync(0xffffffffu, largest);
        if ((tid & 31) == 0) atomicMax(&b.largest, largest);
        asm volatile("bar.sync 3, %0;" ::"n"(kThreads) : "memory");
        if (!wanted) continue;
        // Bit 2k + b: phase b of the output has the tap of k. 0 in place of one that it does not have would make a NaN of an infinity, and
        // any other value may be the filter's own.
        uint32_t has = ~0u;
        if (FOLD) {
            int tap = 0, c;
            const int k = k0 + ((tid & 31) >> 1);
            if (k < K) place(k, tap, c);
            const int th = tap / s.TW;
            has = __ballot_sync(0xffffffffu, k < K && q.filter_of<FOLD>(it.set, th, tap - th * s.TW, tid & 1) >= 0);
        }
        for (int k = 0; k < S::kSlice; ++k) {
            const bool even = (has >> (2 * k)) & 1u, odd = (has >> (2 * k + 1)) & 1u;
            const float x = split::word(slice + (uint32_t)(k * S::BM + row) * 4u);
#pragma unroll
            for (int c = 0; c < S::kCols; c += 4) {
                float y0, y1, y2, y3;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(y0), "=f"(y1), "=f"(y2), "=f"(y3)
                             : "r"(slice + (uint32_t)(S::kSlice * S::BM + k * S::BN + first + c) * 4u) : "memory");
                if (!FOLD || even) {
                    plain[c] = fmaf(x, y0, plain[c]);
                    plain[c + 2] = fmaf(x, y2, plain[c + 2]);
                }
                if (!FOLD || odd) {
                    plain[c + 1] = fmaf(x, y1, plain[c + 1]);
                    plain[c + 3] = fmaf(x, y3, plain[c + 3]);
                }
            }
        }
    }
    asm volatile("bar.sync 3, %0;" ::"n"(kThreads) : "memory");
    if (wanted) {
        // magnitude from which on what was lost is less than 2^-24 of an output
        const float least = b.cut ? __uint_as_float(b.largest) * 0x1p-60f * (float)K * 0x1p-49f : 0.f;
#pragma unroll
        for (int c = 0; c < S::kCols; ++c) {
            const float x = fabsf(split::staged(mine, c));
            if (!(x <= split::kFinite) || x < least) asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + c * 512u), "f"(plain[c]) : "memory");
        }
    }
    asm volatile("bar.sync 3, %0;" ::"n"(kThreads) : "memory");  // b.cut is the next tile's
}

template <class S, bool FOLD>
__global__ void __launch_bounds__(S::NT, S::kCtas) conv_patch_kernel(const __grid_constant__ PatchParams q, int* status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ PatchBarriers b;
    const GatherParams& p = q.p;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;
    const uint32_t fbase = base + q.pslots * q.pslot_bytes, staging = base;  // what the sums are staged in has been read by then
    fetch_parameters(q, warp, S::NT / 32);
    volatile int* abort_flag = &b.abort_flag;
    const PatchItem it(q, blockIdx.x, S::BN);
    const PatchSet& ps = q.sets[it.set];
    if (it.part > 0 && it.chunk0 >= it.chunk1) return;  // a share of nothing; a set without taps is still stored

    if (threadIdx.x == 0) {
        b.abort_flag = 0;
        for (int i = 0; i < kMaxRing; ++i) {
            mbar_init(smem_u32(&b.pfull[i]), S::kPatchWarps + S::kSumWarps);
            mbar_init(smem_u32(&b.pempty[i]), S::kAcc);
            mbar_init(smem_u32(&b.ffull[i]), 1);
            mbar_init(smem_u32(&b.fempty[i]), 1);
        }
        for (int a = 0; a < S::kAcc; ++a) {
            mbar_init(smem_u32(&b.tfull[a]), 1);
            mbar_init(smem_u32(&b.tempty[a]), S::kSumWarps);
        }
        mbar_init(smem_u32(&b.drain), S::kAcc);
        mbar_fence_init();
    }
    // Ahead of every griddep_wait_then_launch: a kernel that may start after that call could take the columns that another stream's kernel
    // gives back on this SM, and wait for this kernel's end while this kernel waits for them.
    if (warp == S::kIssuer) {
        tmem_alloc(smem_u32(&b.tmem_base), S::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = b.tmem_base;
    uint32_t fills = 0;  // filter blocks asked for

    if (warp == S::kCopier) {
        // ------------------------------------------------------------ filter blocks, as pack_patch_filter left them
        griddep_wait_then_launch();
        uint32_t slot = 0, ph = 0;
        bool ok = true;
        const uint8_t* src = q.filter + ps.filter_at + ((long long)(it.j0 / S::BN) * ps.steps + (long long)it.chunk0 * ps.full.steps) * S::kStepB;
        for (int chunk = it.chunk0; chunk < it.chunk1 && ok; ++chunk) {
            const ChunkSteps& cs = it.steps(q, chunk);
            for (int blk = 0; blk < cs.blocks; ++blk) {
                ok = mbar_wait_uniform(smem_u32(&b.fempty[slot]), ph ^ 1u, abort_flag, status, CBK_TIMEOUT_EMPTY);
                if (!ok) break;
                const uint32_t bytes = (uint32_t)cs.in_block(blk) * S::kStepB;
                if (lane == 0) {
                    mbar_expect_tx(smem_u32(&b.ffull[slot]), bytes);
                    bulk_load(fbase + slot * q.fslot_bytes, src, bytes, smem_u32(&b.ffull[slot]));
                }
                __syncwarp();
                src += bytes;
                ++fills;
                if (++slot == (uint32_t)q.fslots) { slot = 0; ph ^= 1u; }
            }
        }
    } else if (warp >= S::kIssuer) {
        // ------------------------------------------------------------ UMMAs: two warps take the blocks in turn, each with an accumulator of
        // its own. What one does between two blocks (barriers, commits, addresses: 500 to 1000 clocks) is then behind the other's
        // UMMAs. Descriptors come from parameters alone: one that comes from memory is not in uniform registers, at ~110 clocks a UMMA.
        const uint32_t a = (uint32_t)(warp - S::kIssuer);
        griddep_wait_then_launch();
        bool ok = true;
        const uint32_t d = tmem_base + a * (3u * S::BN);
        uint32_t p_slot = 0, p_ph = 0, f_slot = 0, f_ph = 0, a_ph = 0, turn = 0;
        const uint32_t row_bytes = (uint32_t)(ps.planes * q.px) * 16u, piece = (uint32_t)(q.cw >> 3) * row_bytes;
        for (int chunk = it.chunk0; chunk < it.chunk1 && ok; ++chunk) {
            const ChunkSteps& cs = it.steps(q, chunk);
            ok = mbar_wait_uniform(smem_u32(&b.pfull[p_slot]), p_ph, abort_flag, status, CBK_TIMEOUT_FULL);
            if (!ok) break;
            uint64_t da_group = umma_smem_desc(base + p_slot * q.pslot_bytes, row_bytes, 128u, UMMA_SW_NONE);  // 16 channels
            int tap = 0, left = cs.steps;
            for (int blk = 0; blk < cs.blocks; ++blk, turn = turn + 1 == S::kAcc ? 0u : turn + 1) {
                const int n = min(cs.per_block, left);
                left -= n;
                if (turn == a) {
                    // In this order: a ring of three slots gives a slot's fills to the two warps in turn, and a barrier that is still in the
                    // phase of the fill before this block's (block i - 3, the other warp's) passes a test for this one's parity. With the
                    // accumulator free, block i - 2 has been added up, and i - 3 before it: that fill has landed, the phase is right.
                    ok = mbar_wait_uniform(smem_u32(&b.tempty[a]), a_ph ^ 1u, abort_flag, status, CBK_TIMEOUT_TMEM_EMPTY) &&
                         mbar_wait_uniform(smem_u32(&b.ffull[f_slot]), f_ph, abort_flag, status, CBK_TIMEOUT_FULL);
                    if (!ok) break;
                    tc_fence_after();
                    a_ph ^= 1u;
                    uint64_t db = umma_smem_desc(fbase + f_slot * q.fslot_bytes, S::kRowsB, 128u, UMMA_SW_NONE);
                    for (int t = 0; t < n; ++t) {
                        const uint64_t da = da_group + (uint64_t)(uint32_t)ps.distance[tap];
                        umma_bf16_elect(d, da, db, umma_idesc_bf16(128, 3 * S::BN), t ? 1u : 0u);
                        umma_bf16_elect(d + S::BN, da + (uint64_t)(piece >> 4), db, umma_idesc_bf16(128, 2 * S::BN), 1u);
                        umma_bf16_elect(d + 2 * S::BN, da + (uint64_t)(2u * piece >> 4), db, umma_idesc_bf16(128, S::BN), 1u);
                        db += (uint64_t)(S::kStepB >> 4);
                        if (++tap == ps.taps) {
                            tap = 0;
                            da_group += (uint64_t)(2u * row_bytes >> 4);
                        }
                    }
                    tc_commit_elect(smem_u32(&b.tfull[a]));
                    tc_commit_elect(smem_u32(&b.fempty[f_slot]));
                } else {
                    for (tap += n; tap >= ps.taps; tap -= ps.taps) da_group += (uint64_t)(2u * row_bytes >> 4);
                }
                if (++f_slot == (uint32_t)q.fslots) { f_slot = 0; f_ph ^= 1u; }
            }
            if (!ok) break;
            tc_commit_elect(smem_u32(&b.pempty[p_slot]));  // at once where this warp had no block of the chunk
            if (++p_slot == (uint32_t)q.pslots) { p_slot = 0; p_ph ^= 1u; }
        }
    } else if (warp >= S::kSumWarps) {
        // ------------------------------------------------------------ patches. The kernel just before this one is pack_patch_filter, which
        // writes nothing that is read here: no wait (griddep_wait_then_launch has the rule). The summing warps help with the first.
        const int mine = warp - S::kSumWarps;
        uint32_t slot = 0, ph = 0;
        for (int chunk = it.chunk0; chunk < it.chunk1; ++chunk) {
            if (!mbar_wait_uniform(smem_u32(&b.pempty[slot]), ph ^ 1u, abort_flag, status, CBK_TIMEOUT_EMPTY)) break;
            const bool first = chunk == it.chunk0;
            fetch_patch(q, it, base + slot * q.pslot_bytes, chunk, mine, first ? S::kPatchWarps + S::kSumWarps : S::kPatchWarps);
            if (lane == 0) mbar_arrive_n(smem_u32(&b.pfull[slot]), !first && mine == 0 ? 1 + S::kSumWarps : 1);
            if (++slot == (uint32_t)q.pslots) { slot = 0; ph ^= 1u; }
        }
        griddep_wait_then_launch();
    } else {
        // ------------------------------------------------------------ sums and outputs
        if (it.chunk0 < it.chunk1) {
            fetch_patch(q, it, base, it.chunk0, S::kPatchWarps + warp, S::kPatchWarps + S::kSumWarps);
            if (lane == 0) mbar_arrive(smem_u32(&b.pfull[0]));
        }
        griddep_wait_then_launch();
        bool ok = true;
        const int quarter = warp & 3, first = (warp >> 2) * S::kCols, row = 32 * quarter + lane;
        const uint32_t mine = staging + (uint32_t)(first * 128 + row) * 4u, slice = staging + S::BN * 512u;
        uint32_t a = 0, a_ph = 0;
        const PixelSet& s = p.sets[it.set];
        uint64_t sum[S::kCols / 2];
#pragma unroll
        for (int c = 0; c < S::kCols / 2; ++c) sum[c] = 0ull;
        // Sums of more than kGroup blocks are sums of groups, which wait in the 64 columns of TMEM that no accumulator has: one addition after
        // another rounds at the magnitude of the whole (error at K = 1152: 1.11e-7 of the norm without, 1.02e-7 with groups).
        const uint32_t parked = tmem_base + 6u * 32u + (uint32_t)first + ((uint32_t)(32 * quarter) << 16);
        int added = 0;
        auto with_parked = [&](bool keep) {
#pragma unroll
            for (int col = 0; col < S::kCols; col += 8) {
                uint32_t v[8];
                tmem_ld8(parked + (uint32_t)col, v);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    uint64_t& t = sum[(col + e) / 2];
                    if (added > kGroup) t = split::add2(t, split::pack2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])));
                    float lo, hi;
                    split::unpack2(t, lo, hi);
                    v[e] = __float_as_uint(lo);
                    v[e + 1] = __float_as_uint(hi);
                    if (keep) t = 0ull;
                }
                if (keep) tmem_st(parked + (uint32_t)col, v);
            }
            if (keep) tmem_st_wait();
        };
        for (int chunk = it.chunk0; chunk < it.chunk1 && ok; ++chunk)
            for (int left = it.steps(q, chunk).blocks; left > 0; --left) {
                ok = mbar_wait_uniform(smem_u32(&b.tfull[a]), a_ph, abort_flag, status, CBK_TIMEOUT_TMEM_FULL);
                if (!ok) break;
                tc_fence_after();
                const uint32_t at = tmem_base + a * (3u * S::BN) + (uint32_t)first + ((uint32_t)(32 * quarter) << 16);
#pragma unroll
                for (int col = 0; col < S::kCols; col += 8) {
                    uint32_t v0[8], v1[8], v2[8];
                    tmem_ld8(at + (uint32_t)col, v0);
                    tmem_ld8(at + (uint32_t)(S::BN + col), v1);
                    tmem_ld8(at + (uint32_t)(2 * S::BN + col), v2);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const uint64_t low = split::add2(split::pack2(__uint_as_float(v2[e]), __uint_as_float(v2[e + 1])), split::pack2(__uint_as_float(v1[e]), __uint_as_float(v1[e + 1])));
                        sum[(col + e) / 2] = split::add2(sum[(col + e) / 2], split::add2(low, split::pack2(__uint_as_float(v0[e]), __uint_as_float(v0[e + 1]))));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&b.tempty[a]));
                if (++a == S::kAcc) { a = 0; a_ph ^= 1u; }
                if (++added % kGroup == 0 && !(left == 1 && chunk + 1 == it.chunk1)) with_parked(true);
            }
        if (added > kGroup) with_parked(false);
        // Outputs that need the second pass: as in split::run
        int n, u, v;
        const bool live = q.pixel_of(s, p.N, it.line0 + row, n, u, v);
        uint64_t zeros = 0;
        unsigned smallest = 0xffffffffu;
#pragma unroll
        for (int c = 0; c < S::kCols; c += 2) {
            float lo, hi;
            split::unpack2(sum[c / 2], lo, hi);
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(zeros) : "l"(sum[c / 2]), "l"(0ull));
            smallest = min(smallest, min(2u * __float_as_uint(lo) - 1u, 2u * __float_as_uint(hi) - 1u));
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + c * 512u), "f"(lo) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + c * 512u + 512u), "f"(hi) : "memory");
        }
        const bool wanted = __any_sync(0xffffffffu, live && ok && ((zeros & 0x7fffffff7fffffffull) != 0 || smallest < 2u * __float_as_uint(split::kLow) - 1u));
        uint32_t again;  // any warp's
        asm volatile("{\n\t.reg .pred w, r;\n\tsetp.ne.b32 w, %1, 0;\n\tbarrier.cta.red.or.pred r, 3, %2, w;\n\tselp.b32 %0, 1, 0, r;\n\t}" : "=r"(again) : "r"((int)wanted), "n"(32 * S::kSumWarps) : "memory");
        if (again) sum_again<S, FOLD>(q, it, b, slice, mine, row, first, wanted);
        if (live && ok) {
            const int plane = p.OHH * p.OWW, place = (s.oh0 + s.ohs * u) * p.OWW + s.ow0 + s.ows * v, j = it.j0 + first;
            float* out = p.Out + (long long)n * p.out_batch + place + (long long)(FOLD ? j >> 1 : j) * plane;
            const bool bias = p.ep.bias && it.part == 0, plain = p.atomic_out ? !bias : !p.ep.scale && !p.ep.bias && !p.ep.relu;
            const bool add = p.atomic_out || (p.ep.accumulate && !p.ep.relu && !p.ep.scale && !p.ep.bias);
            auto value = [&](int c, float y, const float* dst) {
                if (p.atomic_out) return y + p.ep.bias[j + c];
                return apply_epilogue(p.ep, y, j + c, (long long)(j + c) * plane + place, p.ep.accumulate ? *dst : 0.f);
            };
            if (FOLD) {  // two neighbouring columns of a channel; a data gradient has no epilogue but the addition
                const int count = min(S::kCols, q.cols - j) / 2;
                const bool both = v < ps.phase_UW[1];
                const bool pairs = both && !add && ((plane | p.OWW) & 1) == 0 && (p.out_batch & 1) == 0 && (reinterpret_cast<uintptr_t>(p.Out) & 7u) == 0;
#pragma unroll 4
                for (int c = 0; c < count; ++c, out += plane) {
                    const float y0 = split::staged(mine, 2 * c), y1 = split::staged(mine, 2 * c + 1);
                    if (pairs) {
                        *reinterpret_cast<float2*>(out) = make_float2(y0, y1);
                    } else if (add) {
                        if (wanted) {
                            split::add_to<true>(out, y0);
                            if (both) split::add_to<true>(out + 1, y1);
                        } else {
                            atomicAdd(out, y0);
                            if (both) atomicAdd(out + 1, y1);
                        }
                    } else {
                        out[0] = y0;
                        if (both) out[1] = y1;
                    }
                }
            } else if (wanted) split::store_columns<true>(out, plane, min(S::kCols, p.OUTC - j), mine, plain, add, value);
            else split::store_columns<false>(out, plane, min(S::kCols, p.OUTC - j), mine, plain, add, value);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (b.abort_flag) {  // issued UMMAs and copies may still run: a bounded chance to finish before TMEM and shared memory go
        if (warp >= S::kIssuer && warp < S::kCopier) {
            tc_commit_elect(smem_u32(&b.drain));
            if (lane == 0) mbar_drain(smem_u32(&b.drain), 0, status);
        }
        if (warp == S::kCopier && lane == 0)
            for (uint32_t i = 0; i < (uint32_t)q.fslots && i < fills; ++i) mbar_drain(smem_u32(&b.ffull[i]), ((fills - 1 - i) / q.fslots) & 1u, status);
        __syncthreads();
    }
    if (warp == S::kIssuer) {
        tc_fence_after();
        tmem_dealloc(tmem_base, S::kTmemCols);
    }
}

// The filter's pieces in the order in which conv_patch_kernel reads them, for every set of pixels and column tile: [step][group of 8 k]
// [piece][BN columns][8 bf16], steps as in ChunkSteps (16 channels, the taps of those, ...). A block takes the 16 channels of 8
// columns, all taps: its values are runs of consecutive floats, of a column or of a channel. Splitting the filter in every CTA took
// four times as long as the patches (128 -> 128, 4 maps of 56 x 56: 88 us).
template <bool FOLD>
__global__ void __launch_bounds__(128, 8) pack_patch_filter(const __grid_constant__ PatchParams q, uint8_t* out, int bn, int packing, uint32_t clear) {
    extern __shared__ float raw[];
    griddep_wait_then_launch();
    const GatherParams& p = q.p;
    if ((int)blockIdx.x >= packing) {  // the output that shares of the contraction are to be added into
        for (uint32_t i = (blockIdx.x - packing) * 128u + threadIdx.x; i < clear; i += (gridDim.x - packing) * 128u) {
            uint32_t r;
            const uint32_t n = q.image_out.split(i, r);
            p.Out[(long long)n * p.out_batch + r] = 0.f;
        }
        return;
    }
    const int groups = (p.C + 15) >> 4, columns = (int)(q.columns.d * (uint32_t)bn) / kPackCols;
    const int c16 = (int)blockIdx.x % groups, column = (int)blockIdx.x / groups % columns, set = (int)blockIdx.x / groups / columns;
    const PixelSet& s = p.sets[set];
    const int F = q.filter_plane, c0 = c16 * 16, j0 = column * kPackCols, taps = s.TH * s.TW;
    const int runs = q.run_out ? kPackCols >> (FOLD ? 1 : 0) : 16, len = (q.run_out ? 16 : kPackCols >> (FOLD ? 1 : 0)) * F, pitch = len | 1;
    const int channels = min(16, p.C - c0), here = max(0, min(kPackCols >> (FOLD ? 1 : 0), p.OUTC - (j0 >> (FOLD ? 1 : 0))));
    const int real_runs = q.run_out ? here : channels, real_len = (q.run_out ? channels : here) * F;
    const float* src = p.Wt + (long long)c0 * p.w_ch + (long long)(j0 >> (FOLD ? 1 : 0)) * p.w_out;
    const long long step = q.run_out ? p.w_out : p.w_ch;
    for (int i0 = threadIdx.x; i0 < runs * len; i0 += 9 * 128) {  // a 3x3 filter's loads all at once
        float v[9];
        int at[9];
#pragma unroll
        for (int u = 0; u < 9; ++u) {
            const int i = i0 + 128 * u, r = (int)q.run.div((uint32_t)i), o = i - r * len;
            at[u] = i < runs * len ? r * pitch + o : -1;
            v[u] = split::load_if(src + r * step + o, at[u] >= 0 && r < real_runs && o < real_len);
        }
#pragma unroll
        for (int u = 0; u < 9; ++u)
            if (at[u] >= 0) raw[at[u]] = v[u];
    }
    __syncthreads();
    const int tile = j0 / bn, n0 = j0 - tile * bn, steps = groups * taps;
    const uint32_t group = 3u * (uint32_t)bn * 16u;
    uint8_t* dst = out + q.sets[set].filter_at + ((long long)tile * steps + (long long)c16 * taps) * (2u * group);
    for (int i = threadIdx.x; i < taps * 2 * kPackCols; i += 128) {
        const int n = i % kPackCols, g = i / kPackCols % 2, t = i / (2 * kPackCols), th = t / s.TW, tw = t - th * s.TW;
        const int at = q.filter_of<FOLD>(set, th, tw, n), col = n >> (FOLD ? 1 : 0);
        uint32_t y[3][4];
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
            float v[2];
            for (int x = 0; x < 2; ++x) v[x] = at < 0 ? 0.f : raw[q.run_out ? col * pitch + (8 * g + e + x) * F + at : (8 * g + e + x) * pitch + col * F + at];
            split::split2(v[0], v[1], y[0][e / 2], y[1][e / 2], y[2][e / 2]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
            *reinterpret_cast<uint4*>(dst + (uint32_t)(t * 2 + g) * group + (uint32_t)(k * bn + n0 + n) * 16u) = make_uint4(y[k][0], y[k][1], y[k][2], y[k][3]);
    }
}

template <int BN>
bool fit(const cb_ctx* ctx, const GatherParams& p, int nsets, PatchPlan& plan) {
    typedef PatchShape<BN> S;
    PatchParams& q = plan.q;
    int most = 0, planes = 1;
    for (int i = 0; i < nsets; ++i) {
        most = q.p.sets[i].TH * q.p.sets[i].TW > most ? q.p.sets[i].TH * q.p.sets[i].TW : most;
        planes = q.sets[i].planes > planes ? q.sets[i].planes : planes;
    }
    const int channels = (p.C + 15) / 16 * 16;
    // channels of a chunk: enough for a few steps a chunk of the set with the fewest taps
    int cw = 16;
    for (int i = 0; i < nsets; ++i) {
        const int taps = p.sets[i].TH * p.sets[i].TW;
        while (taps > 0 && cw < 64 && cw < channels && taps * cw < 48) cw *= 2;
    }
    const long long whole = (long long)ctx->max_smem_optin - 2048, half = 112 * 1024;
    for (; cw >= 16; cw /= 2) {
        const int chunks = (p.C + cw - 1) / cw;
        q.pslot_bytes = (uint32_t)(((long long)planes * q.px * (cw / 8) * 48 + 127) & ~127LL);
        const int steps = most * (cw / 16);
        // two CTAs an SM where the rings can be cut down to it
        for (int ctas = S::kCtas; ctas >= 1; --ctas)
            for (int pslots = chunks > 1 ? 2 : 1; pslots >= 1; --pslots)
                for (int chain = kChain; chain >= 3; --chain) {
                    const int first = (steps + chain - 1) / chain, block = first ? (steps + first - 1) / first : 1;
                    q.fslot_bytes = (uint32_t)block * S::kStepB;
                    for (int fslots = kMaxRing; fslots >= 2; --fslots) {
                        long long bytes = (long long)pslots * q.pslot_bytes + (long long)fslots * q.fslot_bytes;
                        if (bytes < (long long)S::kStaging) bytes = S::kStaging;
                        bytes += 128;
                        if (bytes > (ctas == 2 ? half : whole)) continue;
                        q.cw = cw; q.pslots = pslots; q.fslots = fslots; q.chunks = chunks;
                        plan.smem = (size_t)bytes;
                        plan.ctas_sm = ctas;
                        for (int i = 0; i < nsets; ++i) {
                            q.sets[i].taps = p.sets[i].TH * p.sets[i].TW;
                            q.sets[i].steps = (p.C + 15) / 16 * q.sets[i].taps;
                            for (int end = 0; end < 2; ++end) {
                                ChunkSteps& cs = end ? q.sets[i].last : q.sets[i].full;
                                cs.channels16 = end ? (p.C - (chunks - 1) * cw + 15) / 16 : cw / 16;
                                cs.steps = cs.channels16 * q.sets[i].taps;
                                cs.blocks = (cs.steps + block - 1) / block;
                                cs.per_block = cs.blocks ? (cs.steps + cs.blocks - 1) / cs.blocks : 0;
                                if (cs.per_block) cs.blocks = (cs.steps + cs.per_block - 1) / cs.per_block;
                            }
                        }
                        return true;
                    }
                }
    }
    return false;
}

}  // namespace

// Whether the launch can come here, and how. Shares of the contraction are whole chunks of channels.
bool plan_patch(const cb_ctx* ctx, const GatherParams& given, int nsets, bool may_split, PatchPlan& best) {
    if (nsets < 1 || nsets > kMaxSets || given.N < 1) return false;
    PatchPlan plan{};
    PatchParams& q = plan.q;
    q.p = given;
    GatherParams& p = q.p;
    // The four sets of a stride-2 data gradient as two, of even and odd rows, whose column phases lie side by side in the product: the patch of
    // a distance serves both, and pairs of columns leave together. 32 -> 64 at 32 x 32, batch 128: 34.5 us as
    // four sets, 25.7.
    q.fold = nsets == 4 && p.sgn < 0 && p.sets[0].ohs == 2 && p.sets[0].ows == 2 ? 1 : 0;
    if (q.fold) {
        for (int a = 0; a < 2; ++a) {
            const PixelSet even = p.sets[2 * a], odd = p.sets[2 * a + 1];
            PixelSet s = even;
            PatchSet& ps = q.sets[a];
            int lo = 1 << 20, hi = -(1 << 20);  // columns the taps of either phase reach
            const PixelSet* phases[2] = {&even, &odd};
            for (int b = 0; b < 2; ++b) {
                ps.f0[b] = phases[b]->wu0; ps.phase_wb[b] = phases[b]->wb; ps.phase_UW[b] = phases[b]->UW;
                if (phases[b]->TW == 0) continue;
                hi = phases[b]->wb > hi ? phases[b]->wb : hi;
                lo = phases[b]->wb - phases[b]->TW + 1 < lo ? phases[b]->wb - phases[b]->TW + 1 : lo;
            }
            s.wb = hi >= lo ? hi : 0;
            s.TW = hi >= lo ? hi - lo + 1 : 0;
            s.UW = even.UW > odd.UW ? even.UW : odd.UW;
            p.sets[a] = s;
        }
        nsets = 2;
    }
    q.cols = p.OUTC << q.fold;
    int GH = 1, GW = 1, px = 128;
    long long useful = 0;
    struct Reach {
        int lo_h, hi_h, lo_w, hi_w;
    } reach[kMaxSets];
    int tap_h[kMaxSets][kPatchTaps], tap_w[kMaxSets][kPatchTaps];
    for (int i = 0; i < nsets; ++i) {
        const PixelSet& s = p.sets[i];
        if (s.TH * s.TW > kPatchTaps || s.hs < 1 || s.hs > 2 || s.ws < 1 || s.ws > 2) return false;
        useful += (long long)s.UH * s.UW;
        PatchSet& ps = q.sets[i];
        int plane[4] = {};
        ps.planes = 0;
        int lo_h = 0, hi_h = 0, lo_w = 0, hi_w = 0;
        bool rows_used[2] = {false, false}, cols_used[2] = {false, false};
        for (int t = 0; t < s.TH; ++t) {
            const int e = s.hb + p.sgn * t, d = s.hs == 2 ? e >> 1 : e;
            rows_used[s.hs == 2 ? e & 1 : 0] = true;
            lo_h = d < lo_h ? d : lo_h; hi_h = d > hi_h ? d : hi_h;
        }
        for (int t = 0; t < s.TW; ++t) {
            const int e = s.wb + p.sgn * t, d = s.ws == 2 ? e >> 1 : e;
            cols_used[s.ws == 2 ? e & 1 : 0] = true;
            lo_w = d < lo_w ? d : lo_w; hi_w = d > hi_w ? d : hi_w;
        }
        for (int a = 0; a < 2; ++a)
            for (int c = 0; c < 2; ++c)
                if (rows_used[a] && cols_used[c]) {
                    ps.ph[ps.planes] = a;
                    ps.pw[ps.planes] = c;
                    plane[a * 2 + c] = ps.planes++;
                }
        if (ps.planes == 0) ps.planes = 1;
        for (int t = 0; t < s.TH * s.TW; ++t) {  // row and column of the distance, until GW is known
            const int e = s.hb + p.sgn * (t / s.TW), f = s.wb + p.sgn * (t % s.TW);
            tap_h[i][t] = s.hs == 2 ? e >> 1 : e;
            tap_w[i][t] = s.ws == 2 ? f >> 1 : f;
            ps.distance[t] = plane[(s.hs == 2 ? (e & 1) : 0) * 2 + (s.ws == 2 ? (f & 1) : 0)];
        }
        reach[i] = Reach{lo_h, hi_h, lo_w, hi_w};
        const int rows = (p.H + s.hs - 1) / s.hs, cols = (p.W + s.ws - 1) / s.ws;
        auto up = [](int& m, int v) { m = v > m ? v : m; };
        up(GH, rows - lo_h); up(GH, s.UH + hi_h); up(GH, s.UH);
        up(GW, cols - lo_w); up(GW, s.UW + hi_w); up(GW, s.UW);
    }
    for (int i = 0; i < nsets; ++i) {
        const Reach& r = reach[i];
        q.sets[i].first = r.lo_h * GW + r.lo_w;
        const long long span = 128LL + (long long)(r.hi_h - r.lo_h) * GW + r.hi_w - r.lo_w;
        if (span > 2048) return false;
        px = span > px ? (int)span : px;
    }
    q.GH = GH; q.GW = GW; q.px = px;
    for (int i = 0; i < nsets; ++i)
        for (int t = 0; t < p.sets[i].TH * p.sets[i].TW; ++t)
            q.sets[i].distance[t] = q.sets[i].distance[t] * px + tap_h[i][t] * GW + tap_w[i][t] - q.sets[i].first;
    const long long image = (long long)GH * GW, lines = image * p.N, tiles = (lines + 127) / 128;
    // 32-bit distances on the line and from a patch's first image; half of the line at least is pixels
    if (lines + image + 8LL * px >= (1LL << 31)) return false;
    if (useful * 2 < image * nsets) return false;
    q.image = FastDiv(image);
    q.row = FastDiv(GW);
    q.filter_plane = p.w_ch < p.w_out ? p.w_ch : p.w_out;
    if (q.filter_plane > kPatchTaps) return false;
    for (int i = 0; i < nsets; ++i) {
        // even and odd columns in one load: both are there for every row phase, and 8 bytes are aligned
        PatchSet& ps = q.sets[i];
        ps.pairs = p.sets[i].ws == 2 && (ps.planes == 2 || ps.planes == 4) && ps.pw[0] == 0 && ps.pw[1] == 1 && ps.ph[0] == ps.ph[1] &&
                   ((p.W | p.in_batch) & 1) == 0 && (reinterpret_cast<uintptr_t>(p.In) & 7u) == 0;
        ps.segs = FastDiv(((ps.planes * px >> ps.pairs) + 31) / 32);
    }
    q.run_out = p.w_ch < p.w_out || (p.w_ch == p.w_out && p.C == 1) ? 1 : 0;
    q.run = FastDiv((q.run_out ? 16 : kPackCols >> q.fold) * q.filter_plane);
    double best_cost = 1e300;
    for (int bn = 64; bn >= 32; bn /= 2) {
        PatchPlan c = plan;
        c.bn = bn;
        if (!(bn == 64 ? fit<64>(ctx, c.q.p, nsets, c) : fit<32>(ctx, c.q.p, nsets, c))) continue;
        const long long groups = (long long)((q.cols + bn - 1) / bn) * nsets;
        double steps = 0, runs = 0;  // of a set: steps, and runs of 32 positions x 8 channels of a chunk's patch
        for (int i = 0; i < nsets; ++i) {
            steps += (double)c.q.sets[i].steps / nsets;
            runs += (double)((c.q.sets[i].planes * px + 31) / 32) * (c.q.cw / 8) / nsets;
        }
        const int chunks = c.q.chunks;
        for (int want = 1; want <= chunks; ++want) {
            if (want > 1 && (!may_split || (double)p.N * p.OUTC * p.OHH * p.OWW >= (double)(1 << 30) || tiles * groups * want > 4LL * ctx->sm_count)) break;
            const int per = (chunks + want - 1) / want, splits = (chunks + per - 1) / per;
            if (splits != want) continue;
            const long long items = tiles * groups * splits;
            if (items >= (1LL << 31)) return false;
            // us: launches; a round of CTAs: start and end, UMMAs, fetching; what two CTAs an SM cost each other; adding up shares. Fitted to
            // 2051 launches of 279 layers (3 to 128 channels, 1x1 to 5x5, stride 1 and 2, 8 x 8 to 56 x 56), 8.6 % off on average.
            const long long slots = (long long)ctx->sm_count * (items > ctx->sm_count ? c.ctas_sm : 1);
            const double rounds = (double)((items + slots - 1) / slots), load = c.ctas_sm == 1 ? 3.57 : slots > ctx->sm_count ? 1.61 : 1.0;
            const double fetches = runs * per / (bn == 64 ? 12.0 : 10.0);
            double cost = 3.10 + rounds * (2.68 + load * (steps * per / chunks * (bn == 64 ? 0.1755 : 0.0944) + 0.445 * fetches));
            if (splits > 1) cost += rounds * 128.0 * bn * 2e-5;
            cost = cost < 6.7 ? 6.7 : cost;
            if (cost < best_cost) {
                best_cost = cost;
                best = c;
                best.us = cost;
                best.q.p.splits = splits;
                best.q.p.per_split = per;
                best.q.items = (uint32_t)items;
                best.q.tiles = FastDiv(tiles);
                best.q.columns = FastDiv((q.cols + bn - 1) / bn);
                best.q.splits = FastDiv(splits);
                best.q.image_out = FastDiv((long long)p.OUTC * p.OHH * p.OWW);
            }
        }
    }
    if (best_cost == 1e300) return false;
    best.nsets = nsets;
    best.q.p.atomic_out = best.q.p.splits > 1 ? 1 : 0;
    long long bytes = 0;
    const long long columns = (q.cols + best.bn - 1) / best.bn;
    for (int i = 0; i < nsets; ++i) {
        best.q.sets[i].filter_at = bytes;
        bytes += columns * ((p.C + 15) / 16) * p.sets[i].TH * p.sets[i].TW * 96LL * best.bn;
    }
    best.filter_bytes = (size_t)bytes;
    return true;
}

cudaError_t launch_patch(cb_ctx* ctx, PatchPlan& plan, void* scratch) {
    plan.q.filter = static_cast<const uint8_t*>(scratch);
    const int cols = (plan.q.cols + plan.bn - 1) / plan.bn * plan.bn;
    const int F = plan.q.filter_plane, raw = (plan.q.run_out ? kPackCols * (16 * F | 1) : 16 * (kPackCols * F | 1)) * 4;  // (half of it with fold)
    // further blocks clear the output where shares of the contraction are added up in it
    const uint32_t clear = plan.q.p.atomic_out && !plan.q.p.ep.accumulate ? plan.q.image_out.d * (uint32_t)plan.q.p.N : 0u;
    const long long packing = (plan.q.p.C + 15LL) / 16 * (cols / kPackCols) * plan.nsets;
    const long long clearing = ((long long)clear + 1023) / 1024 < 8LL * ctx->sm_count ? ((long long)clear + 1023) / 1024 : 8LL * ctx->sm_count;
    cudaError_t ep = launch_dep(ctx, plan.q.fold ? pack_patch_filter<true> : pack_patch_filter<false>, dim3((unsigned)(packing + clearing)), dim3(128), (size_t)raw, plan.q, static_cast<uint8_t*>(scratch), plan.bn,
                                (int)packing, clear);
    if (ep == cudaSuccess) ep = cudaGetLastError();
    if (ep != cudaSuccess) return ep;
    // Of a grid of about as many CTAs as SMs some would share an SM while others had none: more than half of the shared memory keeps them
    // apart, as the cost model has it (112 to 140 CTAs of 64 columns 1.08 to 1.19 times as fast over 550 layers, of 32 columns 1.01 to 1.1).
    // The last SMs are busy with the clearing of the output for a while where shares are added up (146 CTAs: 7 % slower so). Up to half as
    // many CTAs as SMs find one of their own, and start sooner beside pack_patch_filter without.
    const int items = (int)plan.q.items, most = ctx->sm_count - (plan.q.p.splits > 1 ? 8 : 0);
    const size_t alone = 116 * 1024, smem = items > ctx->sm_count / 2 && items <= most && plan.smem < alone ? alone : plan.smem;
    auto go = [&](auto shape) {
        typedef decltype(shape) S;
        auto kernel = plan.q.fold ? conv_patch_kernel<S, true> : conv_patch_kernel<S, false>;
        cudaError_t e = raise_dynamic_smem_once(kernel, ctx->device, ctx->max_smem_optin, nullptr);
        if (e != cudaSuccess) return e;
        e = launch_dep(ctx, kernel, dim3(plan.q.items), dim3(S::NT), smem, plan.q, ctx->d_status);
        return e == cudaSuccess ? cudaGetLastError() : e;
    };
    return plan.bn == 64 ? go(PatchShape<64>{}) : go(PatchShape<32>{});
}

}  // namespace cb
