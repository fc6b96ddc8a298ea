// tkd_api.cu: the extern "C" entry points of libtkd (include/tkd.h): argument checks, the launch plan, the launches.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <atomic>

#include "../../include/tkd.h"
#include "tkd_internal.h"
#include "tkd_layout.h"

static_assert(TKD_FMT_BFP8 == TKD_BFP8 && TKD_FMT_BFP4 == TKD_BFP4 && TKD_FMT_BF16 == TKD_BF16 && TKD_FMT_INT4 == TKD_INT4,
              "format codes");

namespace {

constexpr int kMaxSmem = 227 * 1024;  // dynamic shared memory a CTA may take on sm_100
constexpr int kMaxPanels = 48 * 1024;  // panel counters at the start of the workspace (6 M columns a call)
constexpr int kMaxUnits = 16 * 1024;   // then the top-k unit counters; 256 KB together
constexpr int kMaxMisc = 64;           // then the call's finished-CTA counter (exchange between GPUs)
constexpr int64_t kCounterBytes = (int64_t)(kMaxPanels + kMaxUnits + kMaxMisc) * 4;

inline int cuda_err(cudaError_t e) { return e == cudaSuccess ? TKD_OK : TKD_ERR_CUDA + (int)e; }
inline int launch_err(int e) { return e == 0 ? TKD_OK : TKD_ERR_CUDA + e; }
inline bool fmt_ok(int fmt) { return fmt == TKD_BFP8 || fmt == TKD_BFP4 || fmt == TKD_BF16 || fmt == TKD_INT4; }
// (formats whose stream carries biased exponents against a side array of per-group maxima)
inline bool has_emax(int fmt) { return fmt == TKD_BFP8 || fmt == TKD_BFP4; }
inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        cached[dev] = n;
    }
    return cached[dev];
}

// Clusters of four CTAs that the tensor-memory kernel of a format can run at a time on the current device: asked once.
int tc_cluster_count(int fmt, size_t smem) {
    static std::atomic<int> cached[64][4];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int n = cached[dev][fmt].load(std::memory_order_relaxed);
    if (!n) {
        n = 1 + (fmt == TKD_BFP8 ? tkd_tc_clusters_bfp8(smem) : fmt == TKD_BFP4 ? tkd_tc_clusters_bfp4(smem) : tkd_tc_clusters_bf16(smem));
        cached[dev][fmt].store(n, std::memory_order_relaxed);
    }
    return n - 1;
}

// 9 to 32 rows: tkd_rows_kernel's chunks of a stage, with its shared-memory map in p; 0: the tensor-memory kernel. A rule on K, the
// format and the number of rows only, because the two kernels' sums are different ones and a column's must not depend on more; it
// goes for records and exchanged calls as well. Measured, launches in a graph over weights larger than L2, us with tkd_rows_kernel /
// the tensor-memory kernel, 900 shapes of 9 to 32 rows, K 544 to 4096, N 1024 to 14336:
// 9 to 16 rows, wherever x leaves 80 KB of the 227 to the ring: bfloat8_b [1280, 4096] 4.5 / 6.4, [2048, 14336] 10.5 / 11.7, [3584, 14336]
// with 16 rows, the worst, 17.9 / 15.0 ([3584, 4096] 7.4 / 9.1); bfloat4_b [2816, 4096] 5.4 / 7.7; bf16, 16 rows, [2048, 4096] 5.6 / 7.7,
// [3072, 4096] 7.1 / 8.7, but [3072, 2048] 6.4 / 4.9 and [3072, 14336] 19.2 / 17.3 (over all N, 16 rows of K 3072 1.06 of the other's time,
// of K 2048 0.91, 9 rows of K 4096 1.04). Less of a ring: bfloat8_b, 16 rows, [4096, 14336] 20.0 / 16.3, [4096, 4096] 8.0 / 9.2.
// 17 to 24 rows, three MMAs a fragment: of four slices, where the other runs in clusters, up to K 1536 (bfloat8_b [1056, 4096] 5.3 / 7.2;
// of K 2048, 24 rows, N 2048 6.1 / 5.3, N 4096 6.5 / 7.3, N 14336 13.6 / 12.7, though 17 rows of K 2048 would take 0.9 of the other's time
// over all N; bf16 of K 1536, N 2048 5.3 / 4.4, over all N 0.99); of other numbers of slices always (bfloat4_b [2816, 4096] 6.3 / 8.2).
// 25 to 32 rows of other numbers of slices: bf16 with four MMAs a fragment ([1056, 14336] 11.6 / 11.9, [1056, 4096] 5.9 / 6.8); block-float
// decodes beside four MMAs took longer than the tensor memory's way ([1056, 14336] 19.5 / 16.2, before either kernel's last speed-up), and
// so run as two tiles of sixteen rows, a team of CTAs each ([1056, 14336] 12.4 / 14.0; bfloat4_b [1056, 4096] 5.9 / 7.3), as do 17 and
// more rows whose x does not fit, up to K 2816 (bfloat4_b [2816, 4096] 8.0 / 8.7, [2816, 14336] 18.4 / 17.4; of K 3072, N 2048 5.8 / 8.2, N
// 8192 12.3 / 14.4, N 14336 18.9 / 17.0).
// N may not enter, and the gain of 17 and more rows of a block-float weight ends at some 12000 to 20000 columns: 24 rows of bfloat4_b,
// [1056, 14336] 9.8 / 11.8, 32 rows of bfloat8_b [1536, 4096] 6.5 / 7.4, [1536, 14336] 14.1 / 13.7, of bfloat4_b [2560, 14336] 17.6 / 16.6.
int rows_layout(TkdParams& p, int sab) {
    const int ck = tkd_chunk_k(p.fmt), nch = (p.K + ck - 1) / ck;
    if (p.M > 16 && p.nslices == 4 && (p.M > 24 || p.K > 1536)) return 0;
    if (p.M > 24 && p.fmt != TKD_BF16 && p.K > 2816) return 0;  // (no tiles, and no instance of four MMAs a block-float fragment)
    for (int rows = p.M > 24 && p.fmt != TKD_BF16 ? 16 : p.M;; rows = 16) {
        const int mt = (rows + 7) / 8;
        const int64_t x_row = (int64_t)nch * ck * 2 + 64, tbuf = TKD_SMEM_HEAD + 8 * 8 * mt * TKD_ROWS_PITCH * 4;
        const int64_t xt = tbuf + 1024, ring = align_up(xt + rows * x_row, 128);  // (1 KB: the lists of top-k records)
        for (int chunks = 4; chunks >= (p.fmt == TKD_BF16 ? 4 : 2); chunks -= 2) {
            const int stage = (nch < chunks ? nch : chunks) * 2 * tkd_subsa(p.fmt) * sab;
            const int64_t stages = (kMaxSmem - ring) / stage;
            if (stages < 3 || kMaxSmem - ring < 80 * 1024) continue;
            p.off_pbuf = TKD_SMEM_HEAD, p.off_tbuf = (int)tbuf, p.off_xt = (int)xt, p.off_ring = (int)ring;
            p.x_stride = (int)x_row, p.stage_bytes = stage, p.nstages = (int)(stages < TKD_MAX_STAGES ? stages : TKD_MAX_STAGES);
            p.rows_tile = rows < p.M ? rows : 0;
            return chunks;
        }
        if (rows <= 16 || p.K > 2816 || p.fmt == TKD_BF16) return 0;  // (bf16: the rows of such a K fit)
    }
}

struct Layout {
    TkdParams p;
    int grid;
    size_t smem;
    int64_t weight_bytes;
    // workspace map
    int64_t off_counters, off_units, off_misc, off_scratch, off_ytmp, ws_bytes;
};

// Everything a launch needs except the device pointers into the workspace. sms 0: ask the device.
// counted: the kernel with the counters and slice sums of the workspace, even where tkd_narrow_kernel could run. tile: a is a tile of the
// rows of a call of more than 32.
int make_layout(const TkdMatmul* a, Layout* L, int sms, bool counted = false, bool tile = false) {
    if (!a || !fmt_ok(a->fmt)) return TKD_ERR_BAD_ARG;
    if (a->m < 1 || a->m > 32 || a->k < 32 || a->k % 32 || a->k > (1 << 24)) return TKD_ERR_BAD_ARG;
    // (the int4 weight with group scales is the reference's one-token op; more rows go through its dequantised
    // bfloat8_b form, as there: int4/w4a16.py dequantize)
    if (a->fmt == TKD_INT4 && a->m > 8) return TKD_ERR_UNSUPPORTED;
    if (a->nblocks < 1 || a->nblocks > 4) return TKD_ERR_BAD_ARG;
    if (a->epilogue < TKD_EPI_PLAIN || a->epilogue > TKD_EPI_SILU) return TKD_ERR_BAD_ARG;
    const bool glu = a->epilogue == TKD_EPI_GLU_IL || a->epilogue == TKD_EPI_GLU2;
    if (a->nblocks > 1 && !(a->epilogue == TKD_EPI_PLAIN || a->epilogue == TKD_EPI_GLU2)) return TKD_ERR_BAD_ARG;
    if (a->nblocks > 1 && (a->scale_dtype != TKD_DT_NONE || (a->topk_k && a->epilogue != TKD_EPI_PLAIN))) return TKD_ERR_BAD_ARG;
    if (a->topk_k && (glu || a->epilogue >= TKD_EPI_RESIDUAL)) return TKD_ERR_BAD_ARG;
    if (a->epilogue == TKD_EPI_SILU && a->nranks > 1) return TKD_ERR_BAD_ARG;
    if ((a->epilogue == TKD_EPI_OUT32) != (a->out_dtype == TKD_DT_F32)) return TKD_ERR_BAD_ARG;
    if (a->out_dtype != TKD_DT_F32 && a->out_dtype != TKD_DT_BF16) return TKD_ERR_BAD_ARG;
    if (a->nranks < 0 || a->nranks > TKD_MAX_RANKS || (a->nranks > 1 && (a->rank < 0 || a->rank >= a->nranks)))
        return TKD_ERR_BAD_ARG;

    const int repeats = a->repeats > 1 ? a->repeats : 1;
    if (a->repeats < 0 || (repeats > 1 && (!a->topk_k || a->topk_write_y || a->nblocks > 1 || a->epilogue != TKD_EPI_PLAIN ||
                                           a->scale_dtype != TKD_DT_NONE || repeats > (1 << 16))))
        return TKD_ERR_BAD_ARG;

    TkdParams& p = L->p;
    memset(&p, 0, sizeof(p));
    p.fmt = a->fmt;
    p.M = a->m;
    p.K = (int)a->k;
    p.nseg = a->nblocks;
    p.epi = a->epilogue;
    p.act = a->epilogue == TKD_EPI_SILU ? 0 : a->act;  // (silu is no GLU's choice)
    p.mul16 = 16, p.mul128 = 128;
    const int mt = a->m <= 8 ? 1 : (a->m <= 16 ? 2 : 4);
    const int sab = tkd_sab(a->fmt);
    const int chunk_k = tkd_chunk_k(a->fmt);
    // k per slice: a function of K and the format only (a column's sum must not depend on anything else). 1024 (less
    // for a short K) divides the items well among the CTAs; but every slice a panel is cut into is another M x 128 sums
    // through the scratch buffer for the CTA that adds the panel up, and another hand-over: a long K is cut into four
    // slices, at most 4096 each (config 3, K 14336, one row: 18.8 us with 1024, 16.4 with 1792, 15.6 with 3584).
    int ks_k = a->k >= 4096 ? 1024 : (a->k >= 2048 ? 512 : 256);
    {
        int part = (int)((a->k / 4 + chunk_k - 1) / chunk_k) * chunk_k;
        if (part > 4096) part = 4096;
        if (part > ks_k) ks_k = part;
    }
    p.ks = a->ks ? a->ks : (ks_k < chunk_k ? chunk_k : ks_k);
    if (p.ks < chunk_k || p.ks % chunk_k || p.ks > 4096) return TKD_ERR_BAD_ARG;
    p.nslices = (p.K + p.ks - 1) / p.ks;
    p.panel_bytes = tkd_panel_bytes(a->fmt, a->k);

    int panels = 0;
    L->weight_bytes = 0;
    for (int s = 0; s < a->nblocks; ++s) {
        const TkdBlock& b = a->block[s];
        if (b.n < 1 || b.out_col0 < 0 || b.n > (1 << 28)) return TKD_ERR_BAD_ARG;
        if (glu && a->epilogue == TKD_EPI_GLU_IL && b.n % 64) return TKD_ERR_BAD_ARG;
        const int64_t npad = tkd_padded_cols(b.n) * repeats;
        if (npad > (1 << 28)) return TKD_ERR_BAD_ARG;
        if (repeats > 1) p.rep_panels = (int)(npad / repeats / TKD_PANEL_COLS);
        TkdSegDev& d = p.seg[s];
        d.w = static_cast<const uint8_t*>(b.w);
        d.w2 = static_cast<const uint8_t*>(b.w_up);
        d.emax = b.emax;
        d.emax2 = b.emax_up;
        d.n_valid = (int)b.n;
        d.out_col0 = (int)b.out_col0;
        d.panel0 = panels;
        const bool two = a->epilogue == TKD_EPI_GLU2;
        panels += (int)(two ? npad / 64 : npad / TKD_PANEL_COLS);  // a (gate, up) panel: 64 columns of each weight
        L->weight_bytes += (two ? 2 : 1) * tkd_stream_bytes(a->fmt, a->k, npad);
    }
    p.total_panels = panels;
    p.total_items = (int64_t)panels * p.nslices;
    const bool on_device = sms <= 0;
    if (sms <= 0) sms = sm_count();
    if (sms <= 0) sms = 148;
    if (a->max_ctas > 0 && a->max_ctas < sms) sms = a->max_ctas;

    // shared-memory map: barriers, the hand-over buffers of the streaming warps, the GLU exchange buffer, the ring
    const int xslots = a->fmt == TKD_BF16 ? TKD_TC_XSLOTS : TKD_TC_SLOTS;
    const int mp = mt == 1 ? 8 : (mt == 2 ? 24 : 40);
    p.stage_bytes = 8 * tkd_subsa(a->fmt) * sab;
    p.off_pbuf = TKD_SMEM_HEAD;
    if (a->m > 8) {
        // 9 to 32 rows, the tensor-memory kernel: the running sums [128][40] floats, then (from the next 1024-byte
        // boundary of the window, hence the slack) `xslots` slots of two x tiles (4 KB each), then the ring. (The kernel
        // addresses x by 32-bit element offsets.)
        if (a->ldx > (1 << 26)) return TKD_ERR_BAD_ARG;
        p.tc = 1;
        p.off_tbuf = TKD_SMEM_HEAD;
        p.off_xt = p.off_tbuf + TKD_PANEL_COLS * 40 * 4;
        p.off_ring = (int)align_up(p.off_xt + 1024 + xslots * 2 * 4096, 128);
    } else {
        // (one to eight rows: two hand-over buffers; all of x in shared memory, K rounded up to a chunk, if that leaves
        // the ring at least four stages; rows 64 bytes further apart than their length, so that the eight rows a warp
        // reads together fall on different banks)
        p.off_tbuf = p.off_pbuf + 2 * 2 * TKD_PANEL_COLS * mp * 4;
        p.off_xt = (int)align_up(p.off_tbuf + TKD_PANEL_COLS * mp * 4, 128);
        int64_t xt_bytes = 0;
        const int64_t x_row = (a->k + chunk_k - 1) / chunk_k * chunk_k * 2 + (a->m > 1 ? 64 : 0);
        if (p.off_xt + a->m * x_row + 4 * (int64_t)p.stage_bytes + 256 <= kMaxSmem) {
            p.x_smem = 1;
            p.x_stride = (int)x_row;
            xt_bytes = a->m * x_row;
        }
        // Items of 32 columns over all of K (tkd_narrow.cuh) where the call is a plain one of one to four slices, and two stages of
        // the ring fit beside x (a stage has a chunk of every slice, 35 KB at four; bf16, whose loads need the most in flight, three).
        // A streaming warp stays with one slice, so those of a short last slice wait, and with fewer slices some have none; still
        // that is the faster form, since no sums go through L2, but for a K of one slice, whose sums need not: there only up to an item
        // for every other CTA; and of two or three slices at one row, or of bf16, only up to six items a CTA. Measured, launches in a
        // graph over weights larger than L2, us with this kernel / the counting one. One slice: bfloat8_b one row, [256, 2048] 1.8 / 2.3,
        // [256, 4096] 2.4 / 2.3, [256, 20480] 4.7 / 4.6; bfloat4_b [512, 2048] 1.9 / 2.7, [512, 4096] 2.6 / 2.7, eight rows 3.1 / 3.3; bf16
        // [128, 2048] 1.8 / 2.1, [128, 4096] 2.4 / 2.1, [256, 20480] 6.0 / 4.4. Two and three: with w_up bfloat8_b [1536, 10240] 9.0 / 9.8,
        // [1536, 20480] 14.4 / 13.5, bf16 [384, 10240] 6.9 / 7.3, [384, 20480] 10.4 / 8.8 (one row of bfloat8_b [768, 28672] would take 7.1
        // where the other takes 8.7); bfloat8_b [1280, 4096] 2.95 / 4.6, eight rows 3.5 / 5.9; bfloat4_b, eight rows, [5120, 4096] 5.4 / 10.4, [2560,
        // 28672] 13.3 / 12.7. Four: bfloat8_b [2080, 4096] (a third of the last) 3.7 / 5.6; two stages of the ring, eight rows: bfloat8_b [8192,
        // 11008] 25.0 / 25.8, bfloat4_b 16.6 / 22.0. Two stages of bf16, eight rows: [8192, 1024] 12.6 / 11.5 (before this kernel's last speed-up).
        const int64_t narrow_xt = p.off_pbuf + 2 * 8 * 32 * (a->m > 1 ? 8 : 1) * 4;
        const int narrow_stage = p.nslices * 2 * tkd_subsa(a->fmt) * sab;
        const int64_t items = 4 * (int64_t)panels;
        const bool faster = p.nslices == 1   ? 2 * items <= sms
                            : p.nslices < 4 ? items <= 6 * (int64_t)sms || (a->m > 1 && a->fmt != TKD_BF16)
                                            : p.nslices == 4;
        if (!counted && faster && !a->topk_k && a->nranks <= 1 &&
            narrow_xt + a->m * x_row + (a->fmt == TKD_BF16 ? 3 : 2) * (int64_t)narrow_stage + 128 <= kMaxSmem) {
            p.stage_bytes = narrow_stage;
            p.narrow = p.x_smem = 1;
            p.off_xt = (int)narrow_xt;
            p.x_stride = (int)x_row;
            xt_bytes = a->m * x_row;
        }
        p.off_ring = (int)align_up(p.off_xt + xt_bytes, 128);
    }
    p.nstages = (kMaxSmem - p.off_ring) / p.stage_bytes;
    if (p.nstages > TKD_MAX_STAGES) p.nstages = TKD_MAX_STAGES;
    if (p.nstages < 2) return TKD_ERR_UNSUPPORTED;
    L->smem = (size_t)p.off_ring + (size_t)p.nstages * p.stage_bytes;

    // (a K of one slice: the tensor-memory kernel, a panel an item, no sums through L2. Us with tkd_rows_kernel / with that: bfloat4_b
    // [512, 11008] 24 rows 7.1 / 5.0; bfloat8_b [256, 11008] 32 rows 7.6 / 4.4, [256, 5392] 9 rows 4.7 / 3.3, with w_up [256, 2048] 4.0 / 4.1)
    if (p.tc && !a->ks && (p.nslices > 1 || tile)) p.rows_chunks = rows_layout(p, sab);
    if (p.rows_chunks) p.tc = 0, L->smem = (size_t)p.off_ring + (size_t)p.nstages * p.stage_bytes;
    const int64_t items = p.narrow || p.rows_chunks ? 4 * (int64_t)panels : p.total_items;
    // (tiles of rows: a team of CTAs each; where max_ctas leaves fewer than the tiles, one for several)
    const int tiles = p.rows_tile ? (p.M + p.rows_tile - 1) / p.rows_tile : 1, teams = sms < tiles ? sms : tiles, team = sms / teams;
    L->grid = teams * (int)(items < team ? items : team);
    if (p.rows_tile) p.rows_team = L->grid / teams;
    p.rows_turns = teams < tiles;
    // 9 to 32 rows: clusters of four CTAs, one to a slice (tkd_stream_tc.cuh), for a plain call of four slices. They take whole
    // panels and leave some SMs idle (a GPC's number of SMs is not a multiple of four: 132 of 148 CTAs on a B200), so they are
    // taken where no CTA gets more items for it; from four items on the other form's SMs that have one less leave theirs to the rest.
    // 32 rows, us in clusters / without: one item, bfloat8_b [4096, 2048] 6.9 / 9.0, [4096, 4224] 9.6 / 10.0, bf16 10.2 / 10.1; two, [4096,
    // 6144] 12.9 / 14.6, bf16 13.8 / 15.1, where it is one without, [4096, 4736] 13.1 / 10.7; three, [4096, 12672] 17.3 / 17.8, bf16, whose
    // bytes want every SM, 21.9 / 20.8 (K 8192 34.3 / 36.1); four, [4096, 14336] 21.0 / 17.3, [4096, 16896] 21.3 / 21.0, [8192, 16896] 30.7 /
    // 33.1, seven, [4096, 28672] 34.1 / 27.9.
    if (p.tc && !counted && on_device && p.nslices == 4 && !a->topk_k && a->nranks <= 1) {
        const int off_xt = p.off_tbuf + 2 * 4 * 8 * 32 * 16, off_ring = (int)align_up(off_xt + 1024 + xslots * 2 * 4096, 128);
        const int stages = (int)((kMaxSmem - off_ring) / p.stage_bytes < TKD_MAX_STAGES ? (kMaxSmem - off_ring) / p.stage_bytes : TKD_MAX_STAGES);
        const size_t smem = (size_t)off_ring + (size_t)stages * p.stage_bytes;
        int clusters = tc_cluster_count(a->fmt, smem);
        if (clusters > sms / 4) clusters = sms / 4;
        if (clusters > panels) clusters = panels;
        if (clusters > 0) {
            const int items = (panels + clusters - 1) / clusters;  // of a CTA, at most
            if (items <= 3 && items <= (4 * panels + sms - 1) / sms) {
                p.tc_cluster = 1;
                p.off_xt = off_xt, p.off_ring = off_ring, p.nstages = stages;
                L->smem = smem;
                L->grid = 4 * clusters;
            }
        }
    }
    p.small = (p.total_items + 1) * (int64_t)(L->grid + 1) < (1ll << 32);

    // top-k
    p.topk_k = a->topk_k;
    int units = 0;
    if (a->topk_k) {
        if (a->topk_rows < 1 || a->topk_rows > 16 || a->topk_k < 1 || a->topk_rows * a->topk_k > 64) return TKD_ERR_BAD_ARG;
        if (a->topk_rows > a->m) return TKD_ERR_BAD_ARG;
        if (a->topk_unit < TKD_PANEL_COLS || a->topk_unit % TKD_PANEL_COLS || a->topk_unit > 2048) return TKD_ERR_BAD_ARG;
        p.topk_rows = a->topk_rows;
        p.topk_unit = a->topk_unit;
        p.topk_slot0 = a->topk_slot0;
        p.write_y = a->topk_write_y;
        p.topk_base = a->topk_base;
        p.topk_n = a->topk_n;
        for (int s = 1; s < a->nblocks; ++s)
            if (a->block[s].n != a->block[0].n) return TKD_ERR_BAD_ARG;
        units = a->nblocks * repeats * ((panels / (a->nblocks * repeats) * TKD_PANEL_COLS + a->topk_unit - 1) / a->topk_unit);
    }
    // workspace map. The counters live in a fixed region at the start, the same for every call: they must stay zero
    // between calls, so no call's slice sums or outputs may ever be laid over another call's counters.
    if (panels > kMaxPanels || units > kMaxUnits) return TKD_ERR_UNSUPPORTED;
    L->off_counters = 0;
    L->off_units = (int64_t)kMaxPanels * 4;
    L->off_misc = (int64_t)(kMaxPanels + kMaxUnits) * 4;
    L->off_scratch = kCounterBytes;
    // (the kernel for up to eight rows reads eight rows of every slice)
    const int64_t scratch = p.nslices > 1 ? ((int64_t)panels * p.nslices * 2 * p.M + (p.M > 1 && p.M < 8 ? 8 : 0)) * TKD_PANEL_COLS * 4 : 0;
    L->off_ytmp = align_up(L->off_scratch + scratch, 256);
    p.ld_ytmp = (int64_t)panels * TKD_PANEL_COLS;
    const int64_t ytmp = a->topk_k && !a->topk_write_y ? (int64_t)a->topk_rows * p.ld_ytmp * 2 : 0;
    L->ws_bytes = align_up(L->off_ytmp + ytmp, 256);
    return TKD_OK;
}

}  // namespace

extern "C" {

int tkd_version(void) { return 3; }

int tkd_layout_version(void) { return TKD_LAYOUT_VERSION; }

int tkd_struct_bytes(int which) {
    return which == 0 ? (int)sizeof(TkdMatmul) : which == 1 ? (int)sizeof(TkdPlan) : which == 2 ? (int)sizeof(TkdBlock) : which == 3 ? (int)sizeof(TkdMoe) : 0;
}

const char* tkd_error_string(int code) {
    switch (code) {
        case TKD_OK: return "ok";
        case TKD_ERR_BAD_ARG: return "bad argument";
        case TKD_ERR_UNSUPPORTED: return "unsupported";
        case TKD_ERR_TIMEOUT: return "a kernel's bounded wait gave up";
        case TKD_ERR_WORKSPACE: return "workspace missing or too small";
        case TKD_ERR_WIDE: return "exponent spread inside a column group too wide for the stream";
        case TKD_ERR_FIXED_SCRATCH: return "the call needs more scratch than tkd_matmul_noalloc's built-in array holds";
        default: return code > TKD_ERR_CUDA ? cudaGetErrorString((cudaError_t)(code - TKD_ERR_CUDA)) : "unknown";
    }
}

int64_t tkd_padded_cols(int64_t n) { return (n + 127) / 128 * 128; }

int64_t tkd_packed_bytes(int fmt, int64_t k, int64_t n) {
    return fmt_ok(fmt) ? tkd_stream_bytes(fmt, k, tkd_padded_cols(n)) : -1;
}

int tkd_quantise(int fmt, const float* src, int orient, int64_t k, int64_t n, const float* col_div, uint8_t* exps,
                 void* codes, void* stream) {
    if (!fmt_ok(fmt) || fmt == TKD_INT4 || !src || !codes || k < 1 || n < 1 || (fmt != TKD_BF16 && !exps) ||
        (orient != 0 && orient != 1))
        return TKD_ERR_BAD_ARG;
    return launch_err(tkd_launch_quantise(fmt, src, orient, k, n, tkd_padded_cols(n), col_div, exps, codes,
                                          static_cast<cudaStream_t>(stream)));
}

int tkd_pack(int fmt, int64_t k, int64_t n, const uint8_t* exps, const void* codes, void* packed, uint8_t* emax,
             int32_t* info, void* stream) {
    if (!fmt_ok(fmt) || !codes || !packed || k < 1 || n < 1) return TKD_ERR_BAD_ARG;
    if (has_emax(fmt) && (!exps || !emax || !info)) return TKD_ERR_BAD_ARG;
    if (fmt == TKD_INT4 && !exps) return TKD_ERR_BAD_ARG;  // (the group scales)
    return launch_err(tkd_launch_permute(fmt, k, tkd_padded_cols(n), exps, codes, emax, info, packed,
                                         static_cast<cudaStream_t>(stream)));
}

static int pack_weight(int fmt, const float* src, int orient, int64_t ld, int64_t k, int64_t n, const float* col_div, void* col_scale, bool unit,
                       void* packed, uint8_t* emax, int32_t* info, void* stream) {
    if (!fmt_ok(fmt) || fmt == TKD_INT4 || !src || !packed || k < 32 || k % 32 || n < 1 || (orient != 0 && orient != 1) ||
        ld < (orient ? n : k) || (col_div && col_scale) || (has_emax(fmt) && (!emax || !info)))
        return TKD_ERR_BAD_ARG;
    if (orient == 0 && (ld % 4 || reinterpret_cast<uintptr_t>(src) & 15)) return TKD_ERR_BAD_ARG;
    if (reinterpret_cast<uintptr_t>(packed) & 15) return TKD_ERR_BAD_ARG;
    if (k > 100 * 1024) return TKD_ERR_UNSUPPORTED;  // (two bytes a k in shared memory)
    return launch_err(tkd_launch_pack_weight(fmt, src, orient, ld, k, n, tkd_padded_cols(n), col_div, static_cast<uint16_t*>(col_scale), unit,
                                             packed, emax, info, static_cast<cudaStream_t>(stream)));
}

int tkd_pack_weight(int fmt, const float* src, int orient, int64_t ld, int64_t k, int64_t n, const float* col_div, void* col_scale,
                    void* packed, uint8_t* emax, int32_t* info, void* stream) {
    return pack_weight(fmt, src, orient, ld, k, n, col_div, col_scale, false, packed, emax, info, stream);
}

int tkd_pack_weight_unit(int fmt, const float* src, int orient, int64_t ld, int64_t k, int64_t n, void* ones, void* packed, uint8_t* emax,
                         int32_t* info, void* stream) {
    return ones ? pack_weight(fmt, src, orient, ld, k, n, nullptr, ones, true, packed, emax, info, stream) : TKD_ERR_BAD_ARG;
}

int tkd_dequantise_bf16(int fmt, int64_t k, int64_t n, const uint8_t* exps, const void* codes, void* out_bf16, void* stream) {
    if ((fmt != TKD_BFP8 && fmt != TKD_BFP4) || !exps || !codes || !out_bf16 || k < 1 || n < 1) return TKD_ERR_BAD_ARG;
    return launch_err(tkd_launch_dequantise_bf16(fmt, k, tkd_padded_cols(n), exps, codes, out_bf16,
                                                 static_cast<cudaStream_t>(stream)));
}

int tkd_unpack(int fmt, int64_t k, int64_t n, const void* packed, const uint8_t* emax, float* out, void* stream) {
    if (!fmt_ok(fmt) || !packed || !out || k < 1 || n < 1 || (has_emax(fmt) && !emax)) return TKD_ERR_BAD_ARG;
    return launch_err(
        tkd_launch_unpack(fmt, k, tkd_padded_cols(n), packed, emax, out, static_cast<cudaStream_t>(stream)));
}

int tkd_matmul_plan(const TkdMatmul* a, TkdPlan* plan) {
    Layout L;
    if (!plan) return TKD_ERR_BAD_ARG;
    // (no device needed: without one the plan is made for 148 SMs)
    int sms = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        sms = 148;
    }
    const int rc = make_layout(a, &L, sms);
    if (rc) return rc;
    plan->ks = L.p.ks;
    plan->nslices = L.p.nslices;
    plan->panels = L.p.total_panels;
    plan->grid = L.grid;
    plan->stages = L.p.nstages;
    plan->stream_warps = TKD_STREAM_WARPS;
    plan->chunk_k = tkd_chunk_k(L.p.fmt);
    plan->smem_bytes = (int32_t)L.smem;
    plan->items = L.p.total_items;
    plan->weight_bytes = L.weight_bytes;
    return TKD_OK;
}

int tkd_matmul_workspace(const TkdMatmul* a, uint64_t* bytes) {
    Layout L;
    if (!bytes) return TKD_ERR_BAD_ARG;
    int sms = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        sms = 148;
    }
    const int rc = make_layout(a, &L, sms);
    if (rc) return rc;
    *bytes = (uint64_t)L.ws_bytes;
    return TKD_OK;
}

// A call's tensors and options against one another.
static int check_pointers(const TkdMatmul* a) {
    if (!a->x || !a->out || a->ldx < a->k || a->ldx % 8 || (reinterpret_cast<uintptr_t>(a->x) & 15)) return TKD_ERR_BAD_ARG;
    for (int s = 0; s < a->nblocks; ++s) {
        const TkdBlock& b = a->block[s];
        if (!b.w || (reinterpret_cast<uintptr_t>(b.w) & 15)) return TKD_ERR_BAD_ARG;
        if (has_emax(a->fmt) && !b.emax) return TKD_ERR_BAD_ARG;
        if (a->epilogue == TKD_EPI_GLU2) {
            if (!b.w_up || (reinterpret_cast<uintptr_t>(b.w_up) & 15) || (has_emax(a->fmt) && !b.emax_up))
                return TKD_ERR_BAD_ARG;
        }
        const int64_t width = a->epilogue == TKD_EPI_GLU_IL ? b.n / 2 : b.n;
        if (b.out_col0 + width > a->ldo) return TKD_ERR_BAD_ARG;
    }
    if (a->scale_dtype != TKD_DT_NONE) {
        if (!a->scale || (a->epilogue == TKD_EPI_GLU2 && !a->scale_up)) return TKD_ERR_BAD_ARG;
        if (a->scale_dtype != TKD_DT_BF16 && a->scale_dtype != TKD_DT_F32) return TKD_ERR_BAD_ARG;
    }
    if (a->epilogue == TKD_EPI_RESIDUAL && (!a->residual || a->residual_dtype != TKD_DT_BF16)) return TKD_ERR_BAD_ARG;
    if (a->epilogue == TKD_EPI_OUT32 && a->residual && a->residual_dtype != TKD_DT_F32) return TKD_ERR_BAD_ARG;
    if (a->epilogue != TKD_EPI_RESIDUAL && a->epilogue != TKD_EPI_OUT32 && a->residual) return TKD_ERR_BAD_ARG;
    return TKD_OK;
}

// ---- more than 32 rows -----------------------------------------------------------------------------------------------

// The launch of such a call, without the pointers into the workspace. sms 0: ask the device.
static int make_wide(const TkdMatmul* a, TkdWide* w, size_t* smem, uint64_t* ws_bytes, int sms, double* us_out = nullptr) {
    if (!a || !fmt_ok(a->fmt) || a->m < 33 || a->m > TKD_ROWS_MAX || a->k < 32 || a->k % 32 || a->k > (1 << 24)) return TKD_ERR_BAD_ARG;
    if (a->epilogue < TKD_EPI_PLAIN || a->epilogue > TKD_EPI_SILU || a->nblocks != 1 || a->topk_k) return TKD_ERR_BAD_ARG;
    if ((a->epilogue == TKD_EPI_OUT32) != (a->out_dtype == TKD_DT_F32)) return TKD_ERR_BAD_ARG;
    if (a->fmt == TKD_INT4 || a->hadamard || a->nranks > 1) return TKD_ERR_UNSUPPORTED;
    const TkdBlock& b = a->block[0];
    if (b.n < 1 || b.out_col0 < 0 || b.n > (1 << 28) || (a->epilogue == TKD_EPI_GLU_IL && b.n % 64)) return TKD_ERR_BAD_ARG;
    memset(w, 0, sizeof(*w));
    TkdWide& p = *w;
    p.M = a->m, p.K = (int)a->k;
    p.nkb = (p.K + 127) / 128 * 2;
    const int64_t npad = tkd_padded_cols(b.n);
    const int64_t panels = a->epilogue == TKD_EPI_GLU2 ? npad / 64 : npad / TKD_PANEL_COLS;
    const int chunk_k = tkd_chunk_k(a->fmt);
    p.chunks = (p.K + chunk_k - 1) / chunk_k;
    if (a->ks < 0 || a->ks % chunk_k) return TKD_ERR_BAD_ARG;
    if (sms <= 0) sms = sm_count();
    if (sms <= 0) sms = 148;
    if (a->max_ctas > 0 && a->max_ctas < sms) sms = a->max_ctas;
    // The rows of a tile and the blocks it is cut into, by what the kernel measured (B200, us; a fit to 350 launches in a graph of 40 to
    // 512 rows, K 1024 to 4096, N 2048 to 14336, three formats, 7 % on average): besides 2.6 + K / 3000 a launch, a unit of 128 k takes
    // 0.4 + nt / 2250 (the decode, then the MMAs; bf16, whose weights are twice the traffic, nt / 750), a tile's output nt / 37, a cut
    // tile 2.2 and nt / 31 for each part that its last CTA adds up.
    const double per_row = a->fmt == TKD_BF16 ? 1 / 750. : 1 / 2250.;
    double best = 0;
    for (int nrt = (p.M + 255) / 256, nrt1 = (p.M + 31) / 32; nrt <= nrt1; ++nrt) {
        const int nt = ((p.M + nrt - 1) / nrt + 15) / 16 * 16;
        if (panels * nrt > kMaxPanels) break;
        for (int cut = 1; cut <= 8; ++cut) {
            const int q = a->ks ? a->ks / chunk_k < p.chunks ? a->ks / chunk_k : p.chunks : (p.chunks + cut - 1) / cut;
            const int blocks = (p.chunks + q - 1) / q;
            const int64_t total = panels * nrt * blocks, grid = total < sms ? total : sms;
            const int64_t run = (total + grid - 1) / grid;
            const double units = (double)(run * q * chunk_k) / 128;
            // parts of a tile: one whenever runs are whole tiles
            const int parts = total % grid == 0 && run % blocks == 0 ? 1 : (int)((blocks + run - 2) / run) + 1;
            const double us = units * (0.4 + nt * per_row) + (double)((run + blocks - 1) / blocks) * nt / 37. +
                              (parts > 1 ? 2.2 + (parts - 1) * nt / 31. : 0);
            if (best == 0 || us < best) {
                best = us;
                p.nrt = nrt, p.nt = nt, p.q = q, p.blocks = blocks, p.total = (int)total, p.grid = (int)grid;
            }
            if (a->ks) break;
        }
    }
    if (best == 0) return TKD_ERR_UNSUPPORTED;
    if (us_out) *us_out = best;
    // (an MMA of up to 128 rows is shorter than its issue: two warps, an accumulator each)
    p.nmma = p.nt <= 128 ? 2 : 1;
    p.nset = p.nmma * p.nt * 2 <= 256 ? 2 : 1;
    p.nx = p.nt <= 128 ? 8 : 4;  // (a multiple of two tiles for each MMA warp: a warp's slots wrap with one subtraction, tkd_wide.cuh)
    p.panel_bytes = tkd_panel_bytes(a->fmt, a->k);
    p.stage_bytes = 8 * tkd_subsa(a->fmt) * tkd_sab(a->fmt);
    p.off_stage = TKD_SMEM_HEAD;
    p.off_x = p.off_stage + (p.nset == 1 ? 5 : 1) * 16 * 64 * 4;  // (GLU: a staging buffer for each worker of the output)
    p.off_ring = (int)align_up(p.off_x + 1023 + p.nx * p.nt * 128, 128);
    p.nstages = (kMaxSmem - p.off_ring) / p.stage_bytes;
    if (p.nstages > TKD_MAX_STAGES) p.nstages = TKD_MAX_STAGES;
    if (p.nstages < 2) return TKD_ERR_UNSUPPORTED;
    *smem = (size_t)p.off_ring + (size_t)p.nstages * p.stage_bytes;
    p.epi = a->epilogue, p.act = a->act, p.mul16 = 16, p.mul128 = 128;
    // workspace: the counters every call shares, the cut tiles' partial sums, the x tiles
    const int64_t scratch = (int64_t)p.grid * 2 * p.nt * 512;
    *ws_bytes = (uint64_t)(kCounterBytes + scratch + (int64_t)p.nrt * p.nkb * p.nt * 128);
    return TKD_OK;
}

int tkd_matmul_rows_workspace(const TkdMatmul* a, uint64_t* bytes) {
    if (!bytes) return TKD_ERR_BAD_ARG;
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        sms = 148;
    }
    TkdWide w;
    size_t smem;
    return make_wide(a, &w, &smem, bytes, sms);
}

// Whether a call of more than 32 rows runs tkd_rows_kernel in tiles of rows (of sixteen, less where x is too long for that), its
// launch in L without the tensors. wide_us: what make_wide's model expects of tkd_wide_kernel's units and outputs.
// Fitted to launches in a graph (B200, us): 1870 shapes of 33 to 512 rows, K 32 to 3136, N 16 to 8192, three formats, every kind of
// output, each with both kernels, by those whose two times lie within a factor of 1.5. A launch of this kernel goes by K in whole chunks
// and the items of its longest CTA (5 % off on average, 18 % at most); one of tkd_wide_kernel, with the one that lays x out, by make_wide's
// model, x and the kind of output (6 %, 24 %). The rule's time is 1.001 of the better of the two (K below 256 1.003), at worst 1.12; on 260
// other shapes, and on 360 of K 2688 to 5440, 1.001 and 1.09. This kernel / the other: bfloat8_b, 40 rows [1056, 4096] 7.1 / 7.3, 128 rows
// [2048, 2048] 10.2 / 11.3, 64 rows of gate and up [2944, 1728] 14.1 / 17.6, 48 rows [576, 4096] 6.3 / 5.4; bfloat4_b, 64 rows [576, 4096]
// 7.4 / 5.4, 128 rows [2048, 2048] 9.2 / 11.2; bf16, 40 rows [1056, 4096] 6.9 / 7.2, 256 rows of K 2048, N 1024 10.5 / 11.4, N 4096 31.6 /
// 12.4. A weight is taken apart anew for every tile here: with N or rows the other is the faster one.
static bool rows_tiles(const TkdMatmul* a, Layout* L, double wide_us) {
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    if (a->max_ctas > 0 && a->max_ctas < sms) sms = a->max_ctas;
    if (a->ks || a->m > 16 * sms) return false;
    TkdMatmul one = *a;
    TkdParams& p = L->p;
    for (one.m = 16; one.m >= 12; one.m -= 4) {
        if (make_layout(&one, L, sms, false, true)) return false;
        if (p.rows_chunks) break;
    }
    if (!p.rows_chunks) return false;
    const int tiles = (a->m + one.m - 1) / one.m, items = 4 * p.total_panels;
    if (tiles > sms) return false;
    p.rows_team = sms / tiles < items ? sms / tiles : items;
    p.rows_tile = one.m, p.M = a->m;
    L->grid = tiles * p.rows_team;
    struct Fit { double launch, launch_k, item, item_k, wide, wide_k, wide_us; };
    const Fit f = p.fmt == TKD_BFP8   ? Fit{2.9, 0.3, 0.56, 0.557, 2.44, 0.56, 0.88}
                  : p.fmt == TKD_BFP4 ? Fit{2.53, 0.58, 0.69, 0.373, 2.86, 2.03, 0.365}
                                      : Fit{2.92, 0.165, 0.45, 0.716, 2.92, 0.9, 0.663};
    const bool glu = p.epi == TKD_EPI_GLU2 || p.epi == TKD_EPI_GLU_IL, silu = p.epi == TKD_EPI_SILU, res = a->residual != nullptr;
    const int ck = tkd_chunk_k(p.fmt);
    const double k = p.K / 1000., kc = (p.K + ck - 1) / ck * ck / 1000., most = (items + p.rows_team - 1) / p.rows_team;
    // (bfloat8_b in stages of two chunks, K 3360 to 3840 and from 4384 on: 1.28 times as long an item, 372 rows [4640, 448] 21.5 us where
    // the other kernel takes 16.2; bfloat4_b 1.06)
    const double item = (f.item + f.item_k * kc + (glu || silu ? 0.145 : res ? 0.11 : 0)) * (p.fmt == TKD_BFP8 && p.rows_chunks == 2 ? 1.28 : 1);
    const double mine = f.launch + f.launch_k * kc + most * item;
    return mine < f.wide + f.wide_k * k + f.wide_us * wide_us + 0.002 * a->m * k + (glu ? 4.7 : silu ? 1.85 : res ? 1.2 : 0);
}

// Whether a call's output shares memory with x. (More than 32 rows may: tkd_wide_kernel reads a copy of x.)
static bool out_meets_x(const TkdMatmul* a) {
    const TkdBlock& b = a->block[0];
    const int64_t width = a->epilogue == TKD_EPI_GLU_IL ? b.n / 2 : b.n, esz = a->out_dtype == TKD_DT_F32 ? 4 : 2;
    const uintptr_t x0 = reinterpret_cast<uintptr_t>(a->x), x1 = x0 + ((a->m - 1) * a->ldx + a->k) * 2;
    const uintptr_t y0 = reinterpret_cast<uintptr_t>(a->out) + b.out_col0 * esz, y1 = y0 + ((a->m - 1) * a->ldo + width) * esz;
    return x0 < y1 && y0 < x1;
}

// A call's tensors in the parameters of its launch (but for the workspace).
static void bind(const TkdMatmul* a, TkdParams* p) {
    p->x = static_cast<const uint16_t*>(a->x);
    p->ldx = a->ldx;
    p->scale = a->scale;
    p->scale2 = a->scale_up;
    p->scale_dt = a->scale_dtype;
    p->res = a->residual;
    p->res_dt = a->residual ? a->residual_dtype : TKD_DT_NONE;
    p->ldr = a->ldr;
    p->out = a->out;
    p->out_dt = a->out_dtype;
    p->ldo = a->ldo;
    p->status = a->status;
    p->no_pdl = a->weights_fresh != 0;
}

int tkd_matmul_rows(const TkdMatmul* a, void* stream) {
    TkdWide p;
    size_t smem;
    uint64_t need;
    double us;
    const int rc = make_wide(a, &p, &smem, &need, 0, &us);
    if (rc) return rc;
    const int ra = check_pointers(a);
    if (ra) return ra;
    if (!a->workspace || a->workspace_bytes < need) return TKD_ERR_WORKSPACE;
    if (reinterpret_cast<uintptr_t>(a->workspace) & 255) return TKD_ERR_BAD_ARG;
    Layout L;
    if (!out_meets_x(a) && rows_tiles(a, &L, us)) {  // (that kernel reads x while other CTAs write their outputs)
        bind(a, &L.p);
        return launch_err(tkd_launch_stream(L.p, L.grid, L.smem, static_cast<cudaStream_t>(stream)));
    }
    const TkdBlock& b = a->block[0];
    p.w = static_cast<const uint8_t*>(b.w), p.w2 = static_cast<const uint8_t*>(b.w_up), p.emax = b.emax, p.emax2 = b.emax_up;
    p.n_valid = (int)b.n, p.out_col0 = (int)b.out_col0;
    p.x = static_cast<const uint16_t*>(a->x), p.ldx = a->ldx;
    p.scale = a->scale, p.scale2 = a->scale_up, p.scale_dt = a->scale_dtype;
    p.res = a->residual, p.ldr = a->ldr, p.out = a->out, p.ldo = a->ldo;
    uint8_t* ws = static_cast<uint8_t*>(a->workspace);
    p.counters = reinterpret_cast<int*>(ws);
    p.scratch = reinterpret_cast<float*>(ws + kCounterBytes);
    p.xt = ws + kCounterBytes + (int64_t)p.grid * 2 * p.nt * 512;
    p.status = a->status;
    p.no_pdl = a->weights_fresh != 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return launch_err(a->fmt == TKD_BFP8 ? tkd_launch_wide_bfp8(p, smem, st)
                                         : a->fmt == TKD_BFP4 ? tkd_launch_wide_bfp4(p, smem, st) : tkd_launch_wide_bf16(p, smem, st));
}

static int run_matmul(const TkdMatmul* a, void* workspace, uint64_t workspace_bytes, void* stream, bool counted = false) {
    Layout L;
    const int rc = make_layout(a, &L, 0, counted);
    if (rc) return rc;
    TkdParams& p = L.p;
    const int ra = check_pointers(a);
    if (ra) return ra;
    if (a->topk_k && !a->records) return TKD_ERR_BAD_ARG;
    if (!workspace || workspace_bytes < (uint64_t)L.ws_bytes) return TKD_ERR_WORKSPACE;
    if (workspace && (reinterpret_cast<uintptr_t>(workspace) & 255)) return TKD_ERR_BAD_ARG;

    bind(a, &p);
    p.records = static_cast<uint32_t*>(a->records);
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    p.counters = reinterpret_cast<int*>(ws + L.off_counters);
    p.unit_counters = reinterpret_cast<int*>(ws + L.off_units);
    p.scratch = reinterpret_cast<float*>(ws + L.off_scratch);
    p.ytmp = reinterpret_cast<uint16_t*>(ws + L.off_ytmp);
    if (a->hadamard) {
        if (a->fmt != TKD_INT4 || a->k % 1024 || !p.x_smem) return TKD_ERR_UNSUPPORTED;
        if (reinterpret_cast<uintptr_t>(a->hadamard) & 15) return TKD_ERR_BAD_ARG;
        p.had = a->hadamard;
    }
    if (a->nranks > 1) {
        if (!a->flags) return TKD_ERR_BAD_ARG;
        p.npeers = a->nranks - 1;
        p.rank = a->rank;
        for (int q = 0; q < p.npeers; ++q) {
            if (!a->peer_flags[q]) return TKD_ERR_BAD_ARG;
            p.peer_out[q] = a->peer_out[q];
            p.peer_records[q] = static_cast<uint32_t*>(a->peer_records[q]);
            p.peer_flags[q] = a->peer_flags[q];
        }
        p.flags = a->flags;
        p.grid_counter = reinterpret_cast<int*>(ws + L.off_misc);
        p.exchange_wait = a->exchange_wait;
    }
    return launch_err(tkd_launch_stream(p, L.grid, L.smem, static_cast<cudaStream_t>(stream)));
}

int tkd_matmul(const TkdMatmul* a, void* stream) {
    if (!a) return TKD_ERR_BAD_ARG;
    return run_matmul(a, a->workspace, a->workspace_bytes, stream);
}

int tkd_matmul_host(const TkdMatmul* a, const void* x_host, void* out_host, void* stream) {
    if (!a || !x_host || !out_host || !a->x || !a->out) return TKD_ERR_BAD_ARG;
    if (a->ldx != a->k) return TKD_ERR_BAD_ARG;  // the staging copy of x is one contiguous block
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemcpyAsync(const_cast<void*>(a->x), x_host, (size_t)a->m * a->k * 2, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return cuda_err(e);
    const int rc = run_matmul(a, a->workspace, a->workspace_bytes, stream);
    if (rc) return rc;
    const size_t esz = a->out_dtype == TKD_DT_F32 ? 4 : 2;
    e = cudaMemcpyAsync(out_host, a->out, (size_t)a->m * a->ldo * esz, cudaMemcpyDeviceToHost, st);
    return cuda_err(e);
}

// ---- tkd_matmul for callers that must not allocate ----------------------------------------------------------------
// The same launch as tkd_matmul, with the kernel's workspace (its panel and unit counters, the slice sums of panels
// spread over several CTAs, the bf16 outputs of a top-k call that writes no y) taken from an array that is part of
// the library's device image instead of from the caller. Every GPU that loads libtkd holds these
// TKD_NOALLOC_SCRATCH_BYTES until the process exits.
//
// tkd_noalloc_scratch below is the HOST-side handle of that array: passing it to a kernel would hand the GPU a host
// address. The array's address on a device comes from cudaGetSymbolAddress, asked once per device with that device
// current, and that address is what the kernel gets.
static __device__ __align__(256) unsigned char tkd_noalloc_scratch[TKD_NOALLOC_SCRATCH_BYTES];

// The array's address on the current device, resolved on first use (a thread that loses the race to publish it has
// resolved the same address). first: set when this call was the one that resolved it.
static int noalloc_address(void** out, bool* first) {
    static std::atomic<void*> dev_ptr[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_err(e);
    if (dev < 0 || dev >= 64) return TKD_ERR_UNSUPPORTED;
    void* ptr = dev_ptr[dev].load(std::memory_order_acquire);
    if (first) *first = false;
    if (!ptr) {
        e = cudaGetSymbolAddress(&ptr, tkd_noalloc_scratch);
        if (e != cudaSuccess) return cuda_err(e);
        void* expected = nullptr;
        if (dev_ptr[dev].compare_exchange_strong(expected, ptr, std::memory_order_acq_rel) && first) *first = true;
    }
    *out = ptr;
    return TKD_OK;
}

int tkd_matmul_noalloc(const TkdMatmul* a, void* stream) {
    Layout L;
    const int rc = make_layout(a, &L, 0, true);
    if (rc) return rc;
    if ((uint64_t)L.ws_bytes > (uint64_t)TKD_NOALLOC_SCRATCH_BYTES) return TKD_ERR_FIXED_SCRATCH;
    void* ptr = nullptr;
    bool first = false;
    const int ra = noalloc_address(&ptr, &first);
    if (ra) return ra;
    if (first) {
        // first call on this device: the array's counters start from zero
        const cudaError_t e = cudaMemsetAsync(ptr, 0, (size_t)kCounterBytes, static_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return cuda_err(e);
    }
    // (its counters and their reset are part of this entry point: it stays with the kernel that uses them)
    return run_matmul(a, ptr, TKD_NOALLOC_SCRATCH_BYTES, stream, true);
}

int tkd_matmul_noalloc_reset(void* stream) {
    void* ptr = nullptr;
    const int ra = noalloc_address(&ptr, nullptr);
    if (ra) return ra;
    return cuda_err(cudaMemsetAsync(ptr, 0, (size_t)kCounterBytes, static_cast<cudaStream_t>(stream)));
}

int tkd_noalloc_scratch_address(void** ptr) {
    if (!ptr) return TKD_ERR_BAD_ARG;
    return noalloc_address(ptr, nullptr);
}

int tkd_hadamard(const void* x, int64_t ldx, const uint32_t* signs, int rows, int k, void* out, int64_t ldo, void* stream) {
    if (!x || !signs || !out || rows < 1 || rows > 65535 || k < 1024 || k % 1024 || ldx < k || ldo < k || (ldx | ldo) % 4)
        return TKD_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(signs)) & 7)
        return TKD_ERR_BAD_ARG;
    return launch_err(tkd_launch_hadamard(x, ldx, signs, rows, k, out, ldo, static_cast<cudaStream_t>(stream)));
}

int tkd_topk_merge(const uint32_t* records, int nrecords, int rows, int k, int top, uint32_t* out, void* stream) {
    if (!records || !out || nrecords < 1 || rows < 1 || rows > 16 || k < 1 || rows * k > 64 || top < 1 || top > 1024)
        return TKD_ERR_BAD_ARG;
    if ((int64_t)nrecords * k > (1 << 24)) return TKD_ERR_BAD_ARG;
    return launch_err(tkd_launch_topk_merge(records, nrecords, rows, k, top, out, static_cast<cudaStream_t>(stream)));
}

int tkd_head_pick(const uint32_t* records, int nrecords, int rows, int k, int top, uint32_t vocab, const void* x,
                  int64_t ldx, int dim, const void* head_rows, int64_t ld_head, int round_bf16, uint32_t* out,
                  uint32_t* ids_out, void* stream) {
    if (!records || !out || !x || !head_rows || nrecords < 1 || rows < 1 || rows > 32 || k < 1 || top < 1 || top > 32)
        return TKD_ERR_BAD_ARG;
    if (dim < 8 || dim % 8 || ldx < dim || ldx % 8 || ld_head < dim || ld_head % 8 || vocab < 1) return TKD_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(head_rows)) & 15) return TKD_ERR_BAD_ARG;
    if ((int64_t)nrecords * k > (1 << 24)) return TKD_ERR_BAD_ARG;
    return launch_err(tkd_launch_head_pick(records, nrecords, rows, k, top, vocab, static_cast<const uint16_t*>(x), ldx, dim,
                                           static_cast<const uint16_t*>(head_rows), ld_head, round_bf16, out, ids_out,
                                           static_cast<cudaStream_t>(stream)));
}

int tkd_head_pick_records(const uint32_t* records, int nrecords, int rows, int k, uint32_t vocab, const uint32_t* token_map,
                          uint32_t* out, uint32_t* ids_out, void* stream) {
    if (!records || !out || nrecords < 1 || rows < 1 || rows > 32 || k < 1 || vocab < 1) return TKD_ERR_BAD_ARG;
    if ((int64_t)nrecords * k > (1 << 24)) return TKD_ERR_BAD_ARG;
    return launch_err(tkd_launch_head_pick_records(records, nrecords, rows, k, vocab, token_map, out, ids_out,
                                                   static_cast<cudaStream_t>(stream)));
}

// ---- exchange between GPUs -------------------------------------------------------------------------------------------

int tkd_exchange_wait(uint32_t* flags, int nranks, int32_t* status, void* stream) {
    if (!flags || nranks < 1 || nranks > TKD_MAX_RANKS) return TKD_ERR_BAD_ARG;
    return launch_err(tkd_launch_exchange_wait(flags, nranks, status, static_cast<cudaStream_t>(stream)));
}

int tkd_exchange_publish(uint32_t* flags, uint32_t* const* peer_flags, int nranks, int rank, int lag_wait, int32_t* status,
                         void* stream) {
    if (!flags || !peer_flags || nranks < 2 || nranks > TKD_MAX_RANKS || rank < 0 || rank >= nranks) return TKD_ERR_BAD_ARG;
    TkdPeerFlags pf = {};
    for (int q = 0; q < nranks - 1; ++q) {
        if (!peer_flags[q]) return TKD_ERR_BAD_ARG;
        pf.p[q] = peer_flags[q];
    }
    return launch_err(tkd_launch_exchange_publish(flags, pf, nranks, rank, lag_wait, status, static_cast<cudaStream_t>(stream)));
}

int tkd_peer_alloc(uint64_t bytes, void** ptr, void* handle) {
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the handle is 64 bytes");
    if (!bytes || !ptr || !handle) return TKD_ERR_BAD_ARG;
    void* d = nullptr;
    cudaError_t e = cudaMalloc(&d, (size_t)bytes);
    if (e != cudaSuccess) return cuda_err(e);
    e = cudaMemset(d, 0, (size_t)bytes);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaIpcMemHandle_t h;
    if (e == cudaSuccess) e = cudaIpcGetMemHandle(&h, d);
    if (e != cudaSuccess) {
        (void)cudaFree(d);
        return cuda_err(e);
    }
    memcpy(handle, &h, sizeof(h));
    *ptr = d;
    return TKD_OK;
}

int tkd_peer_free(void* ptr) { return ptr ? cuda_err(cudaFree(ptr)) : TKD_ERR_BAD_ARG; }

int tkd_peer_open(const void* handle, void** ptr) {
    if (!handle || !ptr) return TKD_ERR_BAD_ARG;
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, sizeof(h));
    return cuda_err(cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess));
}

int tkd_peer_close(void* ptr) { return ptr ? cuda_err(cudaIpcCloseMemHandle(ptr)) : TKD_ERR_BAD_ARG; }

}  // extern "C"
