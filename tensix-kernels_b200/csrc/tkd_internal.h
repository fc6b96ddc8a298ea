// tkd_internal.h: what the translation units of libtkd share (not part of the C-ABI).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tkd.h"

// --- packer (tkd_pack.cu) ---
int tkd_launch_quantise(int fmt, const float* src, int orient, int64_t K, int64_t N, int64_t npad,
                        const float* col_div, uint8_t* exps, void* codes, cudaStream_t st);
int tkd_launch_permute(int fmt, int64_t K, int64_t npad, const uint8_t* exps, const void* codes, uint8_t* emax,
                       int* info, void* stream, cudaStream_t st);
int tkd_launch_pack_weight(int fmt, const float* src, int orient, int64_t ld, int64_t K, int64_t N, int64_t npad, const float* col_div,
                           uint16_t* scale_out, bool unit, void* packed, uint8_t* emax, int* info, cudaStream_t st);  // unit: scales of one
int tkd_launch_dequantise_bf16(int fmt, int64_t K, int64_t npad, const uint8_t* exps, const void* codes, void* out,
                               cudaStream_t st);
int tkd_launch_unpack(int fmt, int64_t K, int64_t npad, const void* stream, const uint8_t* emax, float* out,
                      cudaStream_t st);

// --- streaming matmul (tkd_stream.cu) ---
// (the TKD_EPI_* and TKD_DT_* codes are those of include/tkd.h)

#define TKD_STREAM_WARPS 16    // streaming warps: 8 groups of 16 columns x 2 halves of each chunk's super-atoms
#ifndef TKD_STREAM_WARPS_16ROWS
#define TKD_STREAM_WARPS_16ROWS 8  // ... of the kernel for 9 to 16 rows (as for 32: measured faster than 16)
#endif
#ifndef TKD_STREAM_WARPS_32ROWS
#define TKD_STREAM_WARPS_32ROWS 8
#endif
//  // ... of the kernel for 17 to 32 rows: a warp per column group, both halves
#define TKD_THREADS ((1 + TKD_STREAM_WARPS + 4) * 32)  // + 1 producer warp + 4 output warps
#define TKD_PANEL_COLS 128     // columns one work item covers
#define TKD_MAX_STAGES 16
#define TKD_SMEM_HEAD 1024     // barriers, the stage headers, flags
#define TKD_ROWS_PITCH 36      // tkd_rows_kernel: floats from a row of an item's sums to the next (36: no bank conflicts either way)
#define TKD_TC_SLOTS 6         // tensor-memory kernel: slots of weights in tensor memory (a unit of two 64-k tiles: 64 columns)
#define TKD_TC_XSLOTS 8        // ... of activations in shared memory (8 KB a unit), bf16; block float: as many as of weights

struct TkdSegDev {
    const uint8_t* w;     // packed stream (the gate's with a separate up weight)
    const uint8_t* w2;    // the up weight's stream, or null
    const uint8_t* emax;  // per group of 16 columns (null for bf16)
    const uint8_t* emax2;
    int n_valid;          // real columns of w
    int out_col0;         // first output column of the segment in out (elements)
    int panel0;           // first panel of the segment in the call's panel list
    int pad_;
};

struct TkdParams {
    TkdSegDev seg[4];
    int nseg;
    int fmt, M, K;
    const uint16_t* x;  // bf16 bits, row-major, ldx elements a row
    int64_t ldx;
    int ks;             // k per slice (a multiple of the chunk depth)
    int nslices;        // ceil(K / ks)
    int nstages;
    int64_t panel_bytes;  // bytes of one 128-column panel of the stream
    int total_panels;
    int64_t total_items;
    int small;          // item counts times the grid fit 32 bits: the kernel divides in 32-bit arithmetic
    int epi, act;
    uint32_t mul16, mul128;  // 16 and 128: shifts done as multiplies (see shl_fma)
    const void* scale;   // per output column of w (bf16 or f32), or null
    const void* scale2;  // the up weight's, GLU two-weight form
    int scale_dt;
    const void* res;     // residual, bf16 (reference form) or f32 (with a float32 output)
    int res_dt;
    int64_t ldr;
    void* out;
    int out_dt;
    int64_t ldo;
    // top-k records (output warps)
    uint32_t* records;
    int topk_k, topk_rows, topk_unit, topk_slot0, write_y;
    uint32_t topk_base;
    int rep_panels;      // the call's weight is several of this many panels each, back to back (0: one)
    int64_t topk_n;
    uint16_t* ytmp;      // bf16 outputs of a call that does not write y: [rows][ld_ytmp]
    int64_t ld_ytmp;
    int* unit_counters;
    // slice sums of panels whose slices are spread over several CTAs: [panel][slice][half][row][128] floats
    float* scratch;
    int* counters;
    int* status;
    // exchange with the other GPUs of a column-sharded weight: the output stage repeats its stores of y and of the
    // records into the other ranks' buffers; npeers == 0: none
    int npeers, rank;
    void* peer_out[7];
    uint32_t* peer_records[7];
    uint32_t* peer_flags[7];
    uint32_t* flags;     // this rank's flag words
    int* grid_counter;   // CTAs of this call that have finished their output (returns to zero)
    int exchange_wait;
    int tc;              // 9 to 32 rows: the tensor-memory kernel (tkd_stream_tc.cuh); off_xt is where its operand tiles go
    int tc_cluster;      // ... in clusters of four CTAs, a slice each
    int rows_chunks;     // 9 and more rows: chunks of a stage of tkd_rows_kernel (tkd_rows.cuh); 0: another kernel
    int rows_tile, rows_team;  // ... in tiles of rows (17 and more): rows of a tile, CTAs of each tile (0: all rows, all CTAs)
    int rows_turns;            // ... and the CTAs are fewer than the tiles, which they take in turn
    int x_smem;          // 1 to 8 rows, and all of x (K rounded up to a chunk) fits in shared memory at off_xt
    int narrow;          // ... and the call runs tkd_narrow_kernel (tkd_narrow.cuh)
    int x_stride;        // ... bytes from one row of it to the next
    int no_pdl;          // launch without programmatic dependent launch (the weights may still be being written)
    const uint32_t* had;  // TKD_INT4: sign words of the block Hadamard applied to x in shared memory first (or null)
    // shared-memory map (bytes from the start of dynamic shared memory)
    int off_pbuf, off_tbuf, off_xt, off_ring;
    int stage_bytes;
};

// --- more than 32 rows (tkd_wide.cuh) ---
#define TKD_WIDE_XT 8  // x tiles in shared memory, at most
struct TkdWide {
    const uint8_t *w, *w2;  // the packed stream (the gate's), the up weight's or null
    const uint8_t *emax, *emax2;
    int n_valid, out_col0;
    int M, K;
    int nt, nrt;        // rows of a tile (a multiple of 16, at most 256), row tiles
    int chunks;         // chunks of K a tile
    int q, blocks, total;  // chunks a block; blocks a tile, of all tiles
    int grid;
    int64_t panel_bytes;
    const uint16_t* x;
    int64_t ldx;
    uint8_t* xt;        // x in tiles of [nt][64 k], tile (row tile, k block)
    int nkb;            // 64-k blocks of a row tile (K padded to 128)
    int nmma, nset;     // MMA warps (and accumulators of a set), sets of accumulators
    int nx, nstages, stage_bytes;
    int off_stage, off_x, off_ring;  // shared-memory map
    int epi, act;
    const void *scale, *scale2;
    int scale_dt;
    const void* res;
    int64_t ldr;
    void* out;
    int64_t ldo;
    float* scratch;     // partial sums of cut tiles: two a CTA, [nt / 4][128 columns][4] floats
    int* counters;      // per tile: parts delivered
    int* status;
    int no_pdl;
    uint32_t mul16, mul128;
};

int tkd_launch_wide_bfp8(const TkdWide& p, size_t smem, cudaStream_t st);
int tkd_launch_wide_bfp4(const TkdWide& p, size_t smem, cudaStream_t st);
int tkd_launch_wide_bf16(const TkdWide& p, size_t smem, cudaStream_t st);
int tkd_launch_stream(const TkdParams& p, int grid, size_t smem, cudaStream_t st);
int tkd_tc_clusters_bfp8(size_t smem);  // clusters of four CTAs of the tensor-memory kernel that run at a time (0: cannot tell)
int tkd_tc_clusters_bfp4(size_t smem);
int tkd_tc_clusters_bf16(size_t smem);
int tkd_launch_hadamard(const void* x, int64_t ldx, const uint32_t* signs, int rows, int K, void* out, int64_t ldo,
                        cudaStream_t st);
int tkd_launch_topk_merge(const uint32_t* records, int nrec, int rows, int k, int top, uint32_t* out, cudaStream_t st);
int tkd_launch_head_pick(const uint32_t* records, int nrec, int rows, int k, int top, uint32_t vocab, const uint16_t* x,
                         int64_t ldx, int dim, const uint16_t* head, int64_t ld_head, int round, uint32_t* out,
                         uint32_t* ids_out, cudaStream_t st);
int tkd_launch_head_pick_records(const uint32_t* records, int nrec, int rows, int k, uint32_t vocab, const uint32_t* tmap,
                                 uint32_t* out, uint32_t* ids_out, cudaStream_t st);
int tkd_launch_exchange_wait(uint32_t* flags, int nranks, int* status, cudaStream_t st);
struct TkdPeerFlags {
    uint32_t* p[7];
};
int tkd_launch_exchange_publish(uint32_t* flags, const TkdPeerFlags& peers, int nranks, int rank, int lag_wait, int* status,
                                cudaStream_t st);
