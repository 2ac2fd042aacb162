// Tensor-core weight gradient of the convolution for sm_100a (TF32 mode), NCHW fp32.
#include <cstdlib>

#include "conv_common.cuh"

namespace cb {
namespace {

// ------------------------------------------------------------------------------------------ weight gradient
// dW[oc][c][fh][fw] = sum over output pixels of dY[oc][pix] * X[c][pix shifted by (fh-pH, fw-pW)]: a contraction
// over pixels, so both operands are K-major (32 pixels of one channel plane = one 128-byte row, standard 128-byte
// swizzle). Per line of 32 output pixels a stage holds
//   A: FH blocks [Cp channel rows][32 px] of X, fetched at the vertically shifted pixel offsets (UMMA M side,
//      rows stacked as (fh, c); 128 rows per M tile) — on 32-pixel-wide maps as one box [Cp][FH image rows][32 px],
//      rows stacked as (c, fh) — and
//   B: the dY line [OCp rows][32 px] three times, as (fw, oc) rows of the UMMA N side: the centre copy comes from
//      TMA, the copies for fw = 0 / fw = 2 are the same rows rotated by one pixel (zeros entering at the image row
//      edges), written by eight shift warps — shifting dY by -d is the same sum as shifting X by +d.
// A pipeline stage carries `lps` such lines (1, 2 or 4: as many as leave at least three stages), so that the per-stage
// hand-offs between the producer, the shift warps and the MMA issuer are paid once per 32*lps pixels. Every CTA walks
// its share of the line groups accumulating D[(fh,c)][(fw,oc)] in TMEM (the whole K split across CTAs). Its tile then
// leaves in one of two ways: laid out in filter order in the (by then idle) pipeline stages and added into dW by bulk
// copies that add on arrival, or by scalar atomics where dW's runs are not whole 16-byte words (`direct`, the default: one
// launch), or written to the workspace as a partial, column
// by column (the 32 lanes of a warp hold 32 consecutive rows: full 128-byte lines), for a second kernel that adds the
// partials in a fixed order (deterministic contexts).
struct WgradParams {
    int N, Cin, H, W, OC;
    int FH, FW, pH, pW;
    int Cp, OCp, NQ, mtiles, rowsA;  // rowsA = FH * Cp valid accumulator rows
    int L, LPI;
    long long total_lines;
    int nsplit;                      // CTAs that share a line group, each taking OCp of the output channels (below)
    int lps;                         // lines per pipeline stage
    int groups;                      // ceil(total_lines / lps)
    // 3xTF32 in one launch: the line groups are walked three times, as (lo part of X, dY), (X, lo part of dY) and
    // (X, dY) — the tensor core reads the hi part of whatever it is given — and all of it lands in one accumulator
    int vgroups;                     // groups, or 3 * groups
    int stages, tmem_cols;
    // In a stage: from a line's A rows to the next line's, to the first line's B rows, from a line's B rows to the next line's; what the
    // copies of a stage bring of X
    uint32_t stage_bytes, a_step, b_at, b_step, x_bytes;
    float* partial;                  // [gridDim.x][NQ][mtiles * 128]; with `atomic`: ONE such tile that every CTA adds into
    int atomic;
    // direct != 0: no second kernel. The CTA lays its tile out in the idle pipeline stages in the order of the filter
    // block it belongs to (`OC` runs of `run` floats) and adds the runs into dW (vec4 != 0: by bulk copies):
    // dW[base_off + oc * oc_stride + j] += tile[oc * run + j]. dW must already hold what the sums are added to.
    int direct, vec4, run, s2, IC_src;
    // rows_cf != 0 (32-pixel-wide maps): a line is one image row, so the FH vertically shifted X blocks of a line are
    // FH consecutive image rows and arrive as ONE 4-D box [channel][fh][32 px]: the accumulator rows are then ordered
    // (c, fh) instead of (fh, c), and a line costs two TMA boxes instead of FH + 1.
    int rows_cf;
    // rows_shared != 0 (the same maps, several lines a stage): the FH blocks of one line are those of the next moved by one, so a stage
    // holds lps + FH - 1 image rows, [row][channel][32 px], as ONE box, and a line's A rows, ordered (fh, c), start one row further on. X
    // comes 1.5 times (lps 4) or twice (2) in place of FH times, and a stage takes less room: 48 -> 12, batch 64 10.5 -> 9.7 us, 24 -> 40, batch 33
    // 9.8 -> 9.4, 16 -> 16, batch 128 10.7 -> 10.6 (bound by the shift warps then).
    int rows_shared;
    long long oc_stride, base_off;
    float* dW;
    int* status;
    long long* trace;
};

struct __align__(8) WgradSmem {
    uint64_t full[kConvMaxStages];
    uint64_t empty[kConvMaxStages];
    uint64_t xf[kConvMaxStages];
    uint64_t tfull;
    uint64_t drain;
    uint32_t tmem_base;
    int abort_flag;
};

constexpr int kShiftWarps = 8;  // one scheduler cannot hide the shared-memory latencies of a single warp

// One 16-byte chunk (pixels 4q .. 4q+3, eight neighbouring lanes a row) of a dY row and of its horizontally shifted copies: tap offset -1 pairs
// X[px] with dY[px + 1], tap offset +1 with dY[px - 1]. Image rows are whole chunks, so zeros enter in a chunk's last or first pixel alone.
struct ShiftChunk {
    float4 v;
    __device__ __forceinline__ void load(uint32_t at) {
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
    }
    // m1, p1: bytes from the row to its copies, 0: there is no such tap; whole warp
    __device__ __forceinline__ void store(uint32_t at, uint32_t m1, uint32_t p1, bool row_begins, bool row_ends, bool ok) const {
        const float right = __shfl_down_sync(0xffffffffu, v.x, 1, 8), left = __shfl_up_sync(0xffffffffu, v.w, 1, 8);
        if (ok && m1) asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + m1), "f"(v.y), "f"(v.z), "f"(v.w), "f"(row_ends ? 0.f : right) : "memory");
        if (ok && p1) asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + p1), "f"(row_begins ? 0.f : left), "f"(v.x), "f"(v.y), "f"(v.z) : "memory");
    }
};

// The four K steps (8 pixels each) of one line on one M tile; b_units: from the A tile to the line's B rows.
__device__ __forceinline__ void issue_line(uint32_t d_tmem, uint64_t dA, uint32_t b_units, uint32_t idesc, uint32_t accumulate) {
    const uint64_t dB = dA + (uint64_t)b_units;
    umma_tf32_elect(d_tmem, dA, dB, idesc, accumulate);
    umma_tf32_elect(d_tmem, dA + 2, dB + 2, idesc, 1u);
    umma_tf32_elect(d_tmem, dA + 4, dB + 4, idesc, 1u);
    umma_tf32_elect(d_tmem, dA + 6, dB + 6, idesc, 1u);
}

__global__ void __launch_bounds__(192 + 32 * kShiftWarps, 1)
    umma_wgrad_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmdY,
                      const __grid_constant__ CUtensorMap tmXlo, const __grid_constant__ CUtensorMap tmdYlo,
                      const WgradParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ WgradSmem ws;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // uniform for the compiler too
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &ws.abort_flag;
    const uint32_t st_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t set_bytes = (uint32_t)p.OCp * kRowBytes;
    // this CTA's output channels and its walk over the line groups
    const int oc_first = ((int)blockIdx.x % p.nsplit) * p.OCp, oc_here = min(p.OCp, p.OC - oc_first);
    const int cta = (int)blockIdx.x / p.nsplit, ctas = (int)gridDim.x / p.nsplit;
    const int centre = p.pW;  // (fw, oc) rows of the N side: the unshifted copy is the tap with fw - pW == 0

    if (threadIdx.x == 0) {
        CB_TRACE_WALL(p.trace, 0);
        CB_TRACE_EVENT(p.trace, 1);
        ws.abort_flag = 0;
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&ws.full[s]), 1);
            mbar_init(smem_u32(&ws.empty[s]), 1);
            mbar_init(smem_u32(&ws.xf[s]), kShiftWarps);
        }
        mbar_init(smem_u32(&ws.tfull), 1);
        mbar_init(smem_u32(&ws.drain), 1);
        mbar_fence_init();
        tma_prefetch_desc(&tmX);
        tma_prefetch_desc(&tmdY);
        if (p.vgroups > p.groups) {
            tma_prefetch_desc(&tmXlo);
            tma_prefetch_desc(&tmdYlo);
        }
    }
    __syncthreads();
    if (warp == 1) {
        tmem_alloc(smem_u32(&ws.tmem_base), (uint32_t)p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // nothing above touches global memory: the kernel before this one may still be running until here
    griddep_wait_then_launch();
    const uint32_t tmem_base = ws.tmem_base;
    if (threadIdx.x == 0) CB_TRACE_EVENT(p.trace, 2);

    uint32_t fills = 0;  // producer: stages filled so far
    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        uint32_t s = 0, ph = 0, ahead = 0;
        const bool x3 = p.vgroups > p.groups;
        for (int g = cta; g < p.vgroups; g += ctas) {
            if (!__all_sync(0xffffffffu, ahead) &&
                !mbar_wait_uniform(smem_u32(&ws.empty[s]), ph ^ 1u, abort_flag, p.status, CBK_TIMEOUT_EMPTY))
                break;
            const uint32_t s1 = s + 1 == (uint32_t)p.stages ? 0u : s + 1, ph1 = s1 ? ph : ph ^ 1u;
            ahead = mbar_test(smem_u32(&ws.empty[s1]), ph1 ^ 1u);
            const uint32_t full = smem_u32(&ws.full[s]);
            mbar_expect_tx_elect(full, p.x_bytes + (uint32_t)p.lps * set_bytes);
            // 3xTF32 form: the two small cross terms first, while the accumulator is small (the tensor core's
            // fp32 accumulation error is relative to what the accumulator holds), the hi x hi products last
            const int pass = x3 ? g / p.groups : 0, gg = g - pass * p.groups;
            const CUtensorMap* mx = (x3 && pass == 0) ? &tmXlo : &tmX;
            const CUtensorMap* my = (x3 && pass == 1) ? &tmdYlo : &tmdY;
            // lines past the end use an image index >= N: their boxes are zero-filled and add nothing
            const int g0 = gg * p.lps;  // total_lines < 2^29 (checked on the host)
            int n = g0 / p.LPI, line = g0 - n * p.LPI;
            const uint32_t stage = st_base + s * p.stage_bytes;
            if (p.rows_shared) tma_load_4d_elect(stage, mx, full, 0, 0, line - p.pH, n);
            for (int l = 0; l < p.lps; ++l) {
                const uint32_t stg = stage + (uint32_t)l * p.a_step;
                const int h0 = line * p.L;
                if (p.rows_shared) {
                } else if (p.rows_cf) {
                    tma_load_4d_elect(stg, mx, full, 0, h0 - p.pH, 0, n);
                } else {
                    for (int fh = 0; fh < p.FH; ++fh)
                        tma_load_3d_elect(stg + (uint32_t)fh * p.Cp * kRowBytes, mx, full, (h0 + fh - p.pH) * p.W, 0, n);
                }
                tma_load_3d_elect(stage + p.b_at + (uint32_t)l * p.b_step + (uint32_t)centre * set_bytes, my, full, h0 * p.W, oc_first, n);
                if (++line == p.LPI) {
                    line = 0;
                    ++n;
                }
            }
            ++fills;
            s = s1;
            ph = ph1;
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ UMMA issuer
        const uint32_t idesc = umma_idesc_tf32(128, (uint32_t)p.NQ, 0u, 0u);
        const uint64_t desc0 = umma_smem_desc(0, 16u, 1024u, UMMA_SW_128B);  // K-major 128-byte rows; address added per stage
        // The whole warp runs the loop with the same values (waits go through votes) and one elected lane issues: the
        // descriptors stay in uniform registers (see umma_tf32_elect).
        const bool shifted = p.FW > 1;
        const uint32_t a_units = p.a_step >> 4, b_units = p.b_at >> 4, ba_units = (p.b_step >> 4) - (p.a_step >> 4);  // descriptor address units
        uint32_t s = 0, ph = 0, ahead = 0;
        bool first_line = true;
        for (int g = cta; g < p.vgroups; g += ctas) {
            // with shifted copies the shift warps' arrival implies that the copies' source has landed; the rest of the
            // stage is part of the same transaction count
            if (!__all_sync(0xffffffffu, ahead) &&
                !mbar_wait_uniform(smem_u32(shifted ? &ws.xf[s] : &ws.full[s]), ph, abort_flag, p.status,
                                   shifted ? CBK_TIMEOUT_XFORM : CBK_TIMEOUT_FULL))
                break;
            const uint32_t s1 = s + 1 == (uint32_t)p.stages ? 0u : s + 1, ph1 = s1 ? ph : ph ^ 1u;
            ahead = mbar_test(smem_u32(shifted ? &ws.xf[s1] : &ws.full[s1]), ph1);
            tc_fence_after();
            if (lane == 0 && first_line) CB_TRACE_EVENT(p.trace, 5);
            const uint64_t stg = desc0 + (uint64_t)(((st_base + s * p.stage_bytes) >> 4) & 0x3FFFu);
            if (p.lps == 4 && p.mtiles == 1) {  // the narrow layers: 16 small UMMAs, whose loop would cost as much as they do
#pragma unroll
                for (uint32_t l = 0; l < 4; ++l)
                    issue_line(tmem_base, stg + (uint64_t)(l * a_units), b_units + l * ba_units, idesc, first_line && l == 0 ? 0u : 1u);
            } else {
                for (uint32_t l = 0; l < (uint32_t)p.lps; ++l)
                    for (uint32_t m = 0; m < (uint32_t)p.mtiles; ++m) {
                        const uint32_t shift = m * (16384u >> 4);
                        issue_line(tmem_base + m * (uint32_t)p.NQ, stg + (uint64_t)(l * a_units + shift), b_units + l * ba_units - shift, idesc,
                                   first_line && l == 0 ? 0u : 1u);
                    }
            }
            tc_commit_elect(smem_u32(&ws.empty[s]));
            if (g + ctas >= p.vgroups) tc_commit_elect(smem_u32(&ws.tfull));
            if (lane == 0 && first_line) CB_TRACE_EVENT(p.trace, 6);
            if (lane == 0 && g + ctas >= p.vgroups) CB_TRACE_EVENT(p.trace, 7);
            first_line = false;
            s = s1;
            ph = ph1;
        }
    } else {
        // ------------------------------------------------------------ shift warps (6..): fw = 0 and fw = 2 copies of dY
        if (warp >= 6 && p.FW > 1) {
            // A thread takes one chunk of every 32nd row (a multiple of the swizzle's eight, so its place in the row is the same in all of them);
            // where those lie in a stage is worked out once, and a stage's reads are all under way before the first is used. Reading the
            // neighbours' pixels from shared memory too, four-way bank conflicts, one row after the other, these warps were the bound of
            // most launches: 16 -> 16 at 32 x 32, batch 128 10.6 -> 8.6 us, 64 -> 64 30.9 -> 25.7.
            constexpr int kRows = 4;  // of a thread at a time
            const int t = threadIdx.x - 192, rows = p.lps * p.OCp, q = t & 7, row0 = t >> 3;
            const uint32_t chunk = (uint32_t)(q ^ (row0 & 7)) << 4;
            auto place = [&](int row) {
                uint32_t at = chunk;
                for (; row >= p.OCp; row -= p.OCp) at += p.b_step;
                return at + (uint32_t)row * kRowBytes;
            };
            uint32_t at[kRows];
#pragma unroll
            for (int u = 0; u < kRows; ++u) at[u] = place(min(row0 + 32 * u, rows - 1));
            const uint32_t m1 = centre >= 1 ? 0u - set_bytes : 0u, p1 = centre + 1 < p.FW ? set_bytes : 0u;  // taps fw = pW - 1, pW + 1
            const bool row_begins = ((4 * q) & (p.W - 1)) == 0, row_ends = ((4 * q + 4) & (p.W - 1)) == 0;
            uint32_t s = 0, ph = 0;
            for (int g = cta; g < p.vgroups; g += ctas) {
                if (!mbar_wait_uniform(smem_u32(&ws.full[s]), ph, abort_flag, p.status, CBK_TIMEOUT_XFORM_FULL)) break;
                const uint32_t base = st_base + s * p.stage_bytes + p.b_at + (uint32_t)centre * set_bytes;
                ShiftChunk c[kRows];
#pragma unroll
                for (int u = 0; u < kRows; ++u)
                    if (32 * u < rows) c[u].load(base + at[u]);
#pragma unroll
                for (int u = 0; u < kRows; ++u)
                    if (32 * u < rows) c[u].store(base + at[u], m1, p1, row_begins, row_ends, row0 + 32 * u < rows);
                for (int r = 32 * kRows; r < rows; r += 32) {
                    const uint32_t more = base + place(min(row0 + r, rows - 1));
                    c[0].load(more);
                    c[0].store(more, m1, p1, row_begins, row_ends, row0 + r < rows);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ws.xf[s]));
                if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
            }
        }

        // ------------------------------------------------------------ epilogue: twelve warps, three per TMEM lane quarter
        // (four warps alone spent 4000 clocks on the tile of a 64-channel layer)
        const int quarter = warp & 3, slot = (warp - 2) >> 2;
        constexpr int kEpiSlots = (4 + kShiftWarps) / 4;
        const bool ok = mbar_wait_warp(smem_u32(&ws.tfull), 0, lane, abort_flag, p.status, CBK_TIMEOUT_TMEM_FULL, 128);
        if (threadIdx.x == 64) CB_TRACE_EVENT(p.trace, 8);
        if (ok) {
            tc_fence_after();
            const int rows_tot = p.mtiles * 128;
            for (int m = 0; m < p.mtiles && p.direct; ++m) {
                const int r = m * 128 + 32 * quarter + lane;
                if (m * 128 + 32 * quarter >= p.rowsA) continue;  // warp-uniform: no valid row in this quarter
                // Every UMMA of this CTA has completed (tfull), so nothing reads or writes the pipeline stages any more:
                // they take the tile in filter order. Consecutive lanes are consecutive channels, FH*FW words apart
                // (9 for a 3x3 filter): odd strides spread over the banks.
                const int fh = p.rows_cf ? r % p.FH : r / p.Cp;
                const int c = p.rows_cf ? r / p.FH : r - fh * p.Cp;
                bool row_ok = r < p.rowsA && c < p.Cin;
                int roff, pw = 0;
                if (!p.s2) {
                    roff = (c * p.FH + fh) * p.FW;
                } else {
                    const int phase = c / p.IC_src, cc = c - phase * p.IC_src;
                    const int sh = s2_tap(phase >> 1, fh);
                    row_ok = row_ok && sh >= 0;
                    roff = (cc * 3 + sh) * 3;
                    pw = phase & 1;
                }
                const uint32_t t_row = tmem_base + (uint32_t)m * p.NQ + ((uint32_t)(32 * quarter) << 16);
                for (int c0 = slot * 16; c0 < p.NQ; c0 += 16 * kEpiSlots) {
                    uint32_t v[16];
                    tmem_ld16(t_row + (uint32_t)c0, v);
                    tmem_ld_wait();
                    const int fw = c0 / p.OCp, oc0 = c0 - fw * p.OCp;  // OCp is a multiple of 16: one fw per chunk
                    const int sw = p.s2 ? s2_tap(pw, fw) : fw;
                    if (row_ok && sw >= 0) {
                        const uint32_t dst = st_base + 4u * (uint32_t)(oc0 * p.run + roff + sw);
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            if (oc0 + e < oc_here)
                                asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + 4u * (uint32_t)(e * p.run)), "f"(__uint_as_float(v[e])) : "memory");
                    }
                    __syncwarp();  // the next tcgen05.ld is warp-wide
                }
            }
            if (p.direct) fence_proxy_async_smem();  // the tile leaves through bulk copies
            for (int m = 0; m < p.mtiles && !p.direct; ++m) {
                const int r = m * 128 + 32 * quarter + lane;
                if (m * 128 + 32 * quarter >= p.rowsA) continue;  // warp-uniform: no valid row in this quarter
                // partial[cta][col][row]: for one column the warp's 32 rows are 128 contiguous bytes
                float* dst = p.partial + (p.atomic ? 0LL : (long long)blockIdx.x * p.NQ * rows_tot) + r;
                const uint32_t t_row = tmem_base + (uint32_t)m * p.NQ + ((uint32_t)(32 * quarter) << 16);
                for (int c = slot * 16; c < p.NQ; c += 16 * kEpiSlots) {
                    uint32_t v[16];
                    tmem_ld16(t_row + (uint32_t)c, v);
                    tmem_ld_wait();
                    if (r < p.rowsA) {
                        if (p.atomic) {
#pragma unroll
                            for (int e = 0; e < 16; ++e) atomicAdd(dst + (long long)(c + e) * rows_tot, __uint_as_float(v[e]));
                        } else {
#pragma unroll
                            for (int e = 0; e < 16; ++e) dst[(long long)(c + e) * rows_tot] = __uint_as_float(v[e]);
                        }
                    }
                }
            }
        }
    }

    if (threadIdx.x == 64) CB_TRACE_EVENT(p.trace, 10);
    tc_fence_before();
    __syncthreads();
    if (ws.abort_flag) {
        // A bounded wait gave up somewhere in this CTA: copies armed before that may still be in flight towards its
        // shared memory and issued MMAs may still run on its accumulator; both get a bounded chance to finish before
        // the shared memory and TMEM are released.
        if (warp == 0 && lane == 0) {
            const uint32_t n = (uint32_t)p.stages;  // stage st was last filled as number st + n * round: parity of the round
            for (uint32_t st = 0; st < n && st < fills; ++st) mbar_drain(smem_u32(&ws.full[st]), ((fills - 1 - st) / n) & 1u, p.status);
        }
        if (warp == 1) {  // the commit comes from the lane that issued the MMAs
            tc_commit_elect(smem_u32(&ws.drain));
            if (lane == 0) mbar_drain(smem_u32(&ws.drain), 0, p.status);
        }
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
    if (p.direct && !ws.abort_flag) {
        // The staged tile is added into dW, every CTA starting at another place of it: in step they would all add into the
        // same few lines at once.
        float* out = p.dW + p.base_off + (long long)oc_first * p.oc_stride;
        if (p.vec4) {
            // runs start on 16-byte boundaries and are whole float4s: bulk copies that add on arrival, of a run each or,
            // where the runs are contiguous, of 4 KB (the same through vector atomics of 448 threads took 10,000 clocks for
            // a 64-channel layer, most of the kernel)
            const bool whole = p.oc_stride == p.run;
            const int total = oc_here * p.run, piece = whole ? 1024 : p.run;  // floats
            const int pieces = (total + piece - 1) / piece;
            const int rotation = (int)((long long)cta * pieces / ctas);
            for (int k = threadIdx.x; k < pieces; k += blockDim.x) {
                const int i = k + rotation < pieces ? k + rotation : k + rotation - pieces;
                const int n = min(piece, total - i * piece);
                bulk_reduce_add_f32(out + (long long)i * (whole ? piece : p.oc_stride), st_base + 4u * (uint32_t)(i * piece), 4u * (uint32_t)n);
            }
            tma_store_commit();
            tma_store_wait_read<0>();
        } else {
            const int total = oc_here * p.run, chunk = (int)blockDim.x, padded = (total + chunk - 1) / chunk * chunk;
            const int rotation = (int)((long long)cta * (padded / chunk) / ctas);
            for (int k = threadIdx.x; k < padded; k += chunk) {
                int i = k + rotation * chunk;
                if (i >= padded) i -= padded;
                if (i >= total) continue;
                const int oc = i / p.run, j = i - oc * p.run;
                float v;
                asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(st_base + 4u * (uint32_t)i));
                atomicAdd(out + (long long)oc * p.oc_stride + j, v);
            }
        }
    }
    if (threadIdx.x == 0) {
        CB_TRACE_EVENT(p.trace, 11);
        CB_TRACE_WALL(p.trace, 12);
    }
}

// dW[oc][c][fh][fw] (+)= sum over CTAs of partial[cta][fw*OCp + oc][fh*Cp + c], summed in CTA order.
// s2 != 0: the rows are (tap of the 2x2 phase convolution, phase*IC + c) and map back to the 3x3 stride-2 filter.
template <int kReduceGroups>
__global__ void __launch_bounds__(32 * kReduceGroups) wgrad_reduce_kernel(float* __restrict__ partial, float* __restrict__ dW,
                                                           int nparts, int rows_tot, int rowsA, int NQ, int Cp, int Cin,
                                                           int OC, int OCp, int FH, int FW, int accumulate, int s2,
                                                           int IC_src, int clear, int IC_total, int c_off, int oc_off,
                                                           int rows_cf) {
    // Per-CTA partials (clear == 0): block = 32 consecutive valid accumulator rows of one column x kReduceGroups groups
    // of partials; each thread sums its group's partials in order, the group sums are added in order in shared memory:
    // a fixed summation order (deterministic). One shared accumulator tile (clear != 0): every thread row of the block
    // takes its own 32 rows, reads the sum and leaves zero behind for the next call.
    __shared__ float red[kReduceGroups][33];
    griddep_wait_then_launch();
    const long long total = (long long)rows_tot * NQ;
    const int row_blocks = (rowsA + 31) / 32;
    const int grp = threadIdx.y;
    const int unit = clear ? (int)blockIdx.x * kReduceGroups + grp : (int)blockIdx.x;
    const int col = unit / row_blocks;
    const int r = (unit - col * row_blocks) * 32 + (int)threadIdx.x;
    const bool live = col < NQ && r < rowsA;
    float sum = 0.f;
    if (clear) {
        if (!live) return;
        float* src = partial + (long long)col * rows_tot + r;  // element of the [col][row] tile layout
        sum = *src;
        *src = 0.f;
    } else {
        float s = 0.f;
        if (live) {
            const float* src = partial + (long long)col * rows_tot + r;
#pragma unroll 4
            for (int q = grp; q < nparts; q += kReduceGroups) s += __ldg(src + q * total);
        }
        red[grp][threadIdx.x] = s;
        __syncthreads();
        if (grp != 0 || !live) return;
#pragma unroll
        for (int g = 0; g < kReduceGroups; ++g) sum += red[g][threadIdx.x];
    }
    const int fh = rows_cf ? r % FH : r / Cp;  // accumulator rows are (c, fh) or (fh, c): see WgradParams::rows_cf
    const int c = rows_cf ? r / FH : r - fh * Cp;
    const int fw = col / OCp, oc = col - fw * OCp;
    if (c >= Cin || oc >= OC) return;
    float* dst;
    if (!s2) {
        // this launch may cover a block (oc_off.., c_off..) of a wider filter with IC_total input channels
        dst = dW + (((long long)(oc_off + oc) * IC_total + c_off + c) * FH + fh) * FW + fw;
    } else {
        const int phase = c / IC_src, cc = c - phase * IC_src;
        const int sh = s2_tap(phase >> 1, fh), sw = s2_tap(phase & 1, fw);
        if (sh < 0 || sw < 0) return;
        dst = dW + (((long long)oc * IC_src + cc) * 3 + sh) * 3 + sw;
    }
    *dst = accumulate ? *dst + sum : sum;
}

// lo[n][i] = rna_tf32(x - hi(x)) of x[n * x_batch + i], hi = the 19 bits the tensor core reads; four elements per
// thread, lo dense with `per4` float4 per image.
__global__ void __launch_bounds__(256) tf32_lo4_kernel(const float* __restrict__ x, float* __restrict__ lo, const FastDiv per4,
                                                       long long x_batch, uint32_t items) {
    griddep_wait_then_launch();
    constexpr int U = 4;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < items; i0 += U * stride) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            uint32_t r;
            const uint32_t n = per4.split(i0 + u * stride, r);
            if (i0 + u * stride < items) v[u] = *reinterpret_cast<const float4*>(x + n * x_batch + 4LL * r);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u * stride >= items) break;
            const float in[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
            float out[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                uint32_t q;
                asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(q) : "f"(in[e] - __uint_as_float(__float_as_uint(in[e]) & 0xFFFFE000u)));
                out[e] = __uint_as_float(q);
            }
            reinterpret_cast<float4*>(lo)[i0 + u * stride] = make_float4(out[0], out[1], out[2], out[3]);
        }
    }
}

int launch_lo(cb_ctx* ctx, const float* x, float* lo, long long images, long long per, long long x_batch) {
    const long long items = images * (per / 4);
    if (items > (1LL << 30)) return CB_EUNSUPPORTED;  // 32-bit item indexes
    long long g = (items + 1023) / 1024;
    const long long cap = (long long)ctx->sm_count * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    cudaError_t e = launch_dep(ctx, tf32_lo4_kernel, dim3((unsigned)g), dim3(256), 0, x, lo, FastDiv(per / 4), x_batch ? x_batch : per, (uint32_t)items);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "tf32_lo4_kernel launch");
    ctx->launches += 1;
    return CB_OK;
}

// lo parts of X and dY for the one-launch 3xTF32 form (dense scratch; batch strides 0 = dense)
struct LoParts {
    const float* x = nullptr;
    const float* dy = nullptr;
    long long x_batch = 0, dy_batch = 0;
};

}  // namespace

// dW (+)= contraction over the pixels of N x Cin x IH x IW planes `X` and N x OC x IH x IW planes `dY` with taps
// (FH, FW, pH, pW) in the same-size convention of the forward kernel. s2 / IC_src: see wgrad_reduce_kernel.
static int wgrad_core(cb_ctx* ctx, const float* dY, const float* X, float* dW, int N, int Cin, int IH, int IW, int OC, int FH,
                      int FW, int pH, int pW, int accumulate, int s2, int IC_src, long long dy_batch, long long x_batch,
                      int IC_total = 0, int c_off = 0, int oc_off = 0, const LoParts& lo = LoParts()) {
    if (IC_total == 0) IC_total = Cin;
    if (FH < 1 || FH > 3 || FW < 1 || FW > 3 || pH < 0 || pH > 1 || pW < 0 || pW > 1) return CB_EUNSUPPORTED;
    if (FH - 1 - pH > 1 || FW - 1 - pW > 1) return CB_EUNSUPPORTED;
    if (IW != 8 && IW != 16 && IW != 32) return CB_EUNSUPPORTED;
    const int L = 32 / IW;
    if (IH % L) return CB_EUNSUPPORTED;
    const int Cp = (Cin + 7) / 8 * 8;
    const int rowsA = FH * Cp;
    const int mtiles = (rowsA + 127) / 128;
    if (Cp > 256 || (OC + 15) / 16 * 16 > 128) return CB_EUNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(X) & 15u) || (reinterpret_cast<uintptr_t>(dY) & 15u)) return CB_EUNSUPPORTED;
    const long long smem_cap = (long long)ctx->max_smem_optin - 2048;
    const int max_ctas = ctx->wgrad_grid_cap > 0 && ctx->wgrad_grid_cap < ctx->sm_count ? ctx->wgrad_grid_cap : ctx->sm_count;
    const long long total_lines = (long long)N * (IH / L), passes = lo.x ? 3 : 1;
    if (total_lines > (1LL << 29)) return CB_EUNSUPPORTED;
    const int run = s2 ? IC_src * 9 : Cin * FH * FW;
    // The output channels of a line group go to one CTA or are shared by two or four. An SM adds into global memory at about
    // 14 bytes a clock whatever the form of the atomics, so a 64-channel layer's 147 KB tile takes 10,000 clocks to leave a
    // CTA; sharing divides that (and the UMMAs of a line) while X is fetched once more for each share. Small maps gain
    // (64 -> 64 at 8 x 8), large ones, bound by fetching, do not. Clocks of a launch by candidate:
    struct Shape {
        int nsplit, OCp, NQ, lps, grid;
        uint32_t line_bytes;
        long long stages;
    } sh{};
    double best_cost = 1e300;
    for (int ns = 1; ns <= 4; ns <<= 1) {
        Shape c{};
        c.nsplit = ns;
        c.OCp = ((OC + ns - 1) / ns + 15) / 16 * 16;
        if (ns > 1 && (ctx->deterministic || c.OCp * (ns - 1) >= OC)) break;
        c.NQ = FW * c.OCp;
        if (c.NQ > 256 || mtiles * c.NQ > 512) continue;
        int rows_stage = rowsA + c.NQ;
        if (rows_stage < mtiles * 128) rows_stage = mtiles * 128;
        c.line_bytes = ((uint32_t)rows_stage * kRowBytes + 1023u) & ~1023u;
        if (smem_cap / c.line_bytes < 2) continue;
        // as many lines per stage as leave three stages: the hand-offs between the roles are paid per stage
        c.lps = 1;
        for (int cand = 4; cand >= 2; cand >>= 1)
            if (smem_cap / ((long long)cand * c.line_bytes) >= 3) { c.lps = cand; break; }
        c.stages = smem_cap / ((long long)c.lps * c.line_bytes);
        if (c.stages > kConvMaxStages) c.stages = kConvMaxStages;
        const long long tile_bytes = 4LL * c.OCp * run;
        if (ns > 1 && tile_bytes > c.stages * c.lps * (long long)c.line_bytes) continue;  // only the staged flush knows shares
        const long long groups = (total_lines + c.lps - 1) / c.lps * passes;
        long long per_share = max_ctas / ns;
        if (per_share < 1) break;
        if (per_share > groups) per_share = groups;
        c.grid = (int)per_share * ns;
        const double umma = c.NQ <= 96 ? 58.0 : 0.52 * c.NQ, fetch = (rowsA + c.OCp) * kRowBytes / 27.0;
        const double issue = 4.0 * mtiles * umma + 60.0;
        const double line = issue > fetch ? issue : fetch;
        const double cost = (double)((groups + per_share - 1) / per_share) * c.lps * line + (double)tile_bytes / 14.0 +
                            12.0 * mtiles * c.NQ;
        if (cost < best_cost) {
            best_cost = cost;
            sh = c;
        }
    }
    if (sh.nsplit == 0) return CB_EUNSUPPORTED;
    const int OCp = sh.OCp, NQ = sh.NQ, lps = sh.lps, grid = sh.grid;
    // The choice above, by lines of their own, stays: which lines a CTA sums is part of a gradient's last bits.
    long long stages = sh.stages;
    uint32_t a_step = sh.line_bytes, b_at = (uint32_t)rowsA * kRowBytes, b_step = sh.line_bytes, stage_bytes = (uint32_t)lps * sh.line_bytes;
    uint32_t x_bytes = (uint32_t)lps * (uint32_t)rowsA * kRowBytes;
    bool rows_shared = false;
    if (IW == 32 && FH == 3 && !s2 && lps > 1 && IH % lps == 0) {
        const uint32_t row = (uint32_t)Cp * kRowBytes, rows = (uint32_t)(lps + FH - 1) * row, set = (uint32_t)NQ * kRowBytes;
        // an M tile's 128 rows may begin in the last line's few and must end in the stage
        const uint32_t reach = (uint32_t)(lps - 1) * row + (uint32_t)mtiles * 128u * kRowBytes, bytes = rows + (uint32_t)lps * set;
        const uint32_t whole = ((bytes < reach ? reach : bytes) + 1023u) & ~1023u;
        const long long fit = smem_cap / whole < kConvMaxStages ? smem_cap / whole : kConvMaxStages, tile = 4LL * OCp * run;
        rows_shared = tile <= fit * whole || tile > stages * (long long)stage_bytes;  // the tile leaves as it would have
        if (rows_shared) {
            a_step = row; b_at = x_bytes = rows; b_step = set; stage_bytes = whole;
            stages = fit;
        }
    }

    WgradParams p{};
    p.N = N; p.Cin = Cin; p.H = IH; p.W = IW; p.OC = OC;
    p.FH = FH; p.FW = FW; p.pH = pH; p.pW = pW;
    p.Cp = Cp; p.OCp = OCp; p.NQ = NQ; p.mtiles = mtiles; p.rowsA = rowsA;
    p.L = L; p.LPI = IH / L;
    p.total_lines = total_lines;
    p.nsplit = sh.nsplit;
    p.stages = (int)stages;
    int cols = 32;
    while (cols < mtiles * NQ) cols <<= 1;
    p.tmem_cols = cols;
    p.stage_bytes = stage_bytes;
    p.a_step = a_step; p.b_at = b_at; p.b_step = b_step; p.x_bytes = x_bytes;
    p.lps = lps;
    p.groups = (int)((p.total_lines + lps - 1) / lps);
    p.vgroups = lo.x ? 3 * p.groups : p.groups;
    p.status = ctx->d_status;
    p.trace = ctx->trace;
    // Partial sums: one tile per CTA added in a fixed order by the second kernel (deterministic contexts), or one
    // zero-filled tile that every CTA adds into with atomics and the second kernel moves into dW and clears again.
    p.atomic = ctx->deterministic ? 0 : 1;
    p.s2 = s2; p.IC_src = IC_src;
    p.rows_shared = rows_shared ? 1 : 0;
    p.rows_cf = (IW == 32 && FH > 1 && !s2 && !rows_shared) ? 1 : 0;
    p.run = run;
    p.oc_stride = s2 ? (long long)IC_src * 9 : (long long)IC_total * FH * FW;
    p.base_off = s2 ? 0 : ((long long)oc_off * IC_total + c_off) * FH * FW;
    p.dW = dW;
    p.direct = (p.atomic && 4LL * OCp * p.run <= stages * (long long)stage_bytes) ? 1 : 0;
    p.vec4 = ((p.run & 3) == 0 && (p.oc_stride & 3) == 0 && (p.base_off & 3) == 0 &&
              (reinterpret_cast<uintptr_t>(dW) & 15u) == 0) ? 1 : 0;
    int rc;
    if (p.direct) {
        if (!accumulate) {
            cudaError_t em = cudaMemset2DAsync(dW + p.base_off, (size_t)p.oc_stride * 4, 0, (size_t)p.run * 4, (size_t)OC, ctx->stream);
            if (em != cudaSuccess) return check_cuda(ctx, em, "cudaMemset2DAsync(weight gradient)");
        }
    } else if (p.atomic) {
        rc = ensure_wgrad_acc(ctx, (size_t)mtiles * 128 * NQ * sizeof(float));
        if (rc != CB_OK) return rc;
        p.partial = static_cast<float*>(ctx->wgrad_acc);
    } else {
        rc = ensure_workspace(ctx, (size_t)grid * mtiles * 128 * NQ * sizeof(float));
        if (rc != CB_OK) return rc;
        p.partial = static_cast<float*>(ctx->workspace);
    }

    CUtensorMap tmX, tmdY;
    // X as (32 px, image row, channel, image) with a box of FH rows, or as (pixel, channel, image) with a box per tap
    auto encode_x = [&](CUtensorMap* tm, const float* base, long long batch) -> int {
        const uint64_t bstride = (uint64_t)(batch ? batch : (long long)Cin * IH * IW) * 4;
        if (bstride & 15u) return CB_EUNSUPPORTED;
        if (rows_shared) {
            uint64_t dims[4] = {32u, (uint64_t)Cin, (uint64_t)IH, (uint64_t)N};
            uint64_t str[3] = {(uint64_t)IH * IW * 4, 128u, bstride};
            uint32_t box[4] = {32u, (uint32_t)Cp, (uint32_t)(lps + FH - 1), 1u};
            return encode_tmap(ctx, tm, base, 4, dims, str, box, nullptr, 128);
        }
        if (p.rows_cf) {
            uint64_t dims[4] = {32u, (uint64_t)IH, (uint64_t)Cin, (uint64_t)N};
            uint64_t str[3] = {128u, (uint64_t)IH * IW * 4, bstride};
            uint32_t box[4] = {32u, (uint32_t)FH, (uint32_t)Cp, 1u};
            return encode_tmap(ctx, tm, base, 4, dims, str, box, nullptr, 128);
        }
        uint64_t dims[3] = {(uint64_t)IH * IW, (uint64_t)Cin, (uint64_t)N};
        uint64_t str[2] = {(uint64_t)IH * IW * 4, bstride};
        uint32_t box[3] = {32u, (uint32_t)Cp, 1u};
        return encode_tmap(ctx, tm, base, 3, dims, str, box, nullptr, 128);
    };
    rc = encode_x(&tmX, X, x_batch);
    if (rc != CB_OK) return rc;
    {
        uint64_t dims[3] = {(uint64_t)IH * IW, (uint64_t)OC, (uint64_t)N};
        uint64_t str[2] = {(uint64_t)IH * IW * 4, (uint64_t)(dy_batch ? dy_batch : (long long)OC * IH * IW) * 4};
        if (str[1] & 15u) return CB_EUNSUPPORTED;
        uint32_t box[3] = {32u, (uint32_t)OCp, 1u};
        rc = encode_tmap(ctx, &tmdY, dY, 3, dims, str, box, nullptr, 128);
        if (rc != CB_OK) return rc;
    }
    CUtensorMap tmXlo = tmX, tmdYlo = tmdY;
    if (lo.x) {
        rc = encode_x(&tmXlo, lo.x, lo.x_batch);
        if (rc != CB_OK) return rc;
        uint64_t dimsy[3] = {(uint64_t)IH * IW, (uint64_t)OC, (uint64_t)N};
        uint64_t stry[2] = {(uint64_t)IH * IW * 4, (uint64_t)(lo.dy_batch ? lo.dy_batch : (long long)OC * IH * IW) * 4};
        uint32_t boxy[3] = {32u, (uint32_t)OCp, 1u};
        rc = encode_tmap(ctx, &tmdYlo, lo.dy, 3, dimsy, stry, boxy, nullptr, 128);
        if (rc != CB_OK) return rc;
    }
    const size_t smem = (size_t)p.stages * stage_bytes + 1024;
    int smem_bound = 0;
    cudaError_t e = raise_dynamic_smem_once(umma_wgrad_kernel, ctx->device, ctx->max_smem_optin, &smem_bound);
    if (e != cudaSuccess) return check_cuda(ctx, e, "umma_wgrad_kernel attribute");
    if ((int)smem > smem_bound) return CB_EUNSUPPORTED;
    e = launch_dep(ctx, umma_wgrad_kernel, dim3((unsigned)grid), dim3(192 + 32 * kShiftWarps), smem, tmX, tmdY, tmXlo, tmdYlo, p);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "umma_wgrad_kernel launch");
    if (p.direct) {
        ctx->launches += 1;
        ctx->last_kernel = "umma_tf32";
        return CB_OK;
    }
    const int rgrid = NQ * ((rowsA + 31) / 32);
    static const int groups = [] {
        const char* env = std::getenv("CB_WGRAD_REDUCE_GROUPS");  // development override: 2, 4 or 8
        const int v = env ? std::atoi(env) : 8;
        return v == 2 || v == 4 ? v : 8;
    }();
    auto* reduce = groups == 2 ? wgrad_reduce_kernel<2> : (groups == 4 ? wgrad_reduce_kernel<4> : wgrad_reduce_kernel<8>);
    if (p.atomic)
        e = launch_dep(ctx, wgrad_reduce_kernel<8>, dim3((unsigned)((rgrid + 7) / 8)), dim3(32, 8), 0, p.partial, dW, 1, mtiles * 128,
                       rowsA, NQ, Cp, Cin, OC, OCp, FH, FW, accumulate ? 1 : 0, s2, IC_src, 1, IC_total, c_off, oc_off, p.rows_cf);
    else
        e = launch_dep(ctx, reduce, dim3((unsigned)rgrid), dim3(32, (unsigned)groups), 0, p.partial, dW, grid, mtiles * 128,
                       rowsA, NQ, Cp, Cin, OC, OCp, FH, FW, accumulate ? 1 : 0, s2, IC_src, 0, IC_total, c_off, oc_off, p.rows_cf);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return check_cuda(ctx, e, "wgrad_reduce_kernel launch");
    ctx->launches += 2;
    ctx->last_kernel = "umma_tf32";
    return CB_OK;
}

// How the filter of a stride-1 layer is cut into blocks of input x output channels, a launch each (c_blocks 0: not at all).
struct WgradBlocks {
    int oc_blocks, oc_step, c_blocks, c_step;
};
static WgradBlocks wgrad_blocks(int IC, int OC, int FH, int FW) {
    const int OCp_all = (OC + 15) / 16 * 16;
    int oc_max = (256 / FW) & ~15;
    if (oc_max > 128) oc_max = 128;
    WgradBlocks b{};
    if (oc_max < 16) return b;
    b.oc_blocks = (OCp_all + oc_max - 1) / oc_max;
    b.oc_step = ((OC + b.oc_blocks - 1) / b.oc_blocks + 15) & ~15;
    const int nq = FW * (b.oc_blocks > 1 ? b.oc_step : OCp_all);
    int c_max = ((512 / nq) * 128 / FH) & ~7;
    if (c_max > 256) c_max = 256;
    if (c_max < 8) return b;
    b.c_blocks = (IC + c_max - 1) / c_max;
    b.c_step = ((IC + b.c_blocks - 1) / b.c_blocks + 7) & ~7;
    return b;
}
int umma_wgrad_launches(int IC, int OC, int FH, int FW) {
    if (FH > 3 || FW > 3) return 0;
    const WgradBlocks b = wgrad_blocks(IC, OC, FH, FW);
    return b.oc_blocks * b.c_blocks;
}

int umma_conv_wgrad(cb_ctx* ctx, const float* dY, const float* X, float* dW, int N, int IC, int IH, int IW, int OC,
                    int FH, int FW, int sH, int sW, int pH, int pW, int accumulate, long long dy_batch, long long x_batch,
                    bool x3) {
    // 3xTF32: lo parts of the two operands (as the kernel will read them: after the stride-2 re-layout) in scratch
    auto make_lo = [&](const float* Xsrc, long long x_per, long long xb, const float* dYsrc, long long dy_per, long long yb,
                       LoParts& lo) -> int {
        auto up = [](long long n) { return (n + 63) & ~63LL; };
        const long long xe = (long long)N * x_per, ye = (long long)N * dy_per;
        int rc = ensure_workspace3(ctx, (size_t)(up(xe) + up(ye)) * sizeof(float));
        if (rc != CB_OK) return rc;
        float* xl = static_cast<float*>(ctx->workspace3);
        float* yl = xl + up(xe);
        rc = launch_lo(ctx, Xsrc, xl, N, x_per, xb);
        if (rc == CB_OK) rc = launch_lo(ctx, dYsrc, yl, N, dy_per, yb);
        lo.x = xl; lo.dy = yl; lo.x_batch = x_per; lo.dy_batch = dy_per;
        return rc;
    };
    if (N < 1 || ((long long)IH * IW & 3)) return CB_EUNSUPPORTED;
    if (((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(dY)) & 15u) || (x3 && ((x_batch | dy_batch) & 3))) return CB_EUNSUPPORTED;
    if (sH == 1 && sW == 1) {
        if (!((FH == 1 && pH == 0) || (FH == 3 && pH == 1))) return CB_EUNSUPPORTED;
        if (!((FW == 1 && pW == 0) || (FW == 3 && pW == 1))) return CB_EUNSUPPORTED;
        // Filters wider than one launch covers (256 input channels, 128 output channels, 512 accumulator columns) are
        // cut into blocks of input x output channels: each block is its own launch pair on channel slices of X and dY
        // (same batch strides) that writes its block of dW.
        const WgradBlocks bl = wgrad_blocks(IC, OC, FH, FW);
        if (bl.c_blocks == 0) return CB_EUNSUPPORTED;
        const int oc_blocks = bl.oc_blocks, oc_step = bl.oc_step, c_blocks = bl.c_blocks, c_step = bl.c_step;
        if (IW != 8 && IW != 16 && IW != 32) return CB_EUNSUPPORTED;  // before the lo parts are queued
        const long long plane = (long long)IH * IW;
        LoParts lo;
        if (x3) {
            const int rc = make_lo(X, (long long)IC * plane, x_batch, dY, (long long)OC * plane, dy_batch, lo);
            if (rc != CB_OK) return rc;
        }
        if (oc_blocks == 1 && c_blocks == 1)
            return wgrad_core(ctx, dY, X, dW, N, IC, IH, IW, OC, FH, FW, pH, pW, accumulate, 0, IC, dy_batch, x_batch, 0, 0, 0, lo);
        const long long xb = x_batch ? x_batch : (long long)IC * plane, yb = dy_batch ? dy_batch : (long long)OC * plane;
        for (int o0 = 0; o0 < OC; o0 += oc_step) {
            const int on = OC - o0 < oc_step ? OC - o0 : oc_step;
            for (int c0 = 0; c0 < IC; c0 += c_step) {
                const int cn = IC - c0 < c_step ? IC - c0 : c_step;
                LoParts lc = lo;
                if (x3) { lc.x = lo.x + c0 * plane; lc.dy = lo.dy + o0 * plane; }
                const int rc = wgrad_core(ctx, dY + o0 * plane, X + c0 * plane, dW, N, cn, IH, IW, on, FH, FW, pH, pW, accumulate, 0, cn,
                                          yb, xb, IC, c0, o0, lc);
                if (rc != CB_OK) return rc;
            }
        }
        return CB_OK;
    }
    if (sH != 2 || sW != 2 || FH != FW || pH != pW || (IH & 1) || (IW & 1)) return CB_EUNSUPPORTED;
    if (!((FH == 3 && pH == 1) || (FH == 1 && pH == 0))) return CB_EUNSUPPORTED;
    if (dy_batch || x_batch) return CB_EUNSUPPORTED;  // the stride-2 path re-lays dense tensors out
    const int H2 = IH / 2, W2 = IW / 2;
    if (W2 != 8 && W2 != 16 && W2 != 32) return CB_EUNSUPPORTED;
    const long long plane2 = (long long)H2 * W2;
    if (FH == 1) {
        const long long n_sub = (long long)N * IC * plane2;
        int rc = ensure_workspace2(ctx, (size_t)n_sub * sizeof(float));
        if (rc != CB_OK) return rc;
        float* sub = static_cast<float*>(ctx->workspace2);
        rc = launch_subsample2(ctx, X, sub, (long long)N * IC, IH, IW);
        if (rc != CB_OK) return rc;
        LoParts lo;
        if (x3) {
            rc = make_lo(sub, (long long)IC * plane2, 0, dY, (long long)OC * plane2, 0, lo);
            if (rc != CB_OK) return rc;
        }
        return wgrad_core(ctx, dY, sub, dW, N, IC, H2, W2, OC, 1, 1, 0, 0, accumulate, 0, IC, 0, 0, 0, 0, 0, lo);
    }
    if (4 * IC > 256) return CB_EUNSUPPORTED;
    if (x3) {
        // phase planes and their lo parts in one pass
        const long long half = 4LL * IC * plane2, dy_per = (long long)OC * plane2;
        int rc = ensure_workspace2(ctx, (size_t)N * 2 * half * sizeof(float));
        if (rc == CB_OK) rc = ensure_workspace3(ctx, (size_t)N * dy_per * sizeof(float));
        if (rc != CB_OK) return rc;
        float* X2 = static_cast<float*>(ctx->workspace2);
        float* yl = static_cast<float*>(ctx->workspace3);
        rc = launch_space_to_depth2_split(ctx, X, X2, N, IC, 4 * IC, IH, IW);
        if (rc == CB_OK) rc = launch_lo(ctx, dY, yl, N, dy_per, 0);
        if (rc != CB_OK) return rc;
        LoParts lo;
        lo.x = X2 + half; lo.x_batch = 2 * half; lo.dy = yl; lo.dy_batch = dy_per;
        return wgrad_core(ctx, dY, X2, dW, N, 4 * IC, H2, W2, OC, 2, 2, 1, 1, accumulate, 1, IC, 0, 2 * half, 0, 0, 0, lo);
    }
    const long long n_el = (long long)N * 4 * IC * plane2;
    int rc = ensure_workspace2(ctx, (size_t)n_el * sizeof(float));
    if (rc != CB_OK) return rc;
    float* Xs = static_cast<float*>(ctx->workspace2);
    rc = launch_space_to_depth2(ctx, X, Xs, N, IC, IH, IW);
    if (rc != CB_OK) return rc;
    return wgrad_core(ctx, dY, Xs, dW, N, 4 * IC, H2, W2, OC, 2, 2, 1, 1, accumulate, 1, IC, 0, 0);
}

}  // namespace cb
