// tkd_stream_bf16.cu: the stream kernel's instantiations for one weight format (a translation unit per format, so that
// they compile side by side).
#include "tkd_rows.cuh"
#include "tkd_stream_tc.cuh"

int tkd_launch_stream_bf16(const TkdParams& p, int grid, size_t smem, cudaStream_t st) {
    if (p.rows_chunks) return launch_rows_kernel<TKD_BF16>(p, grid, smem, st);
    if (p.narrow) return launch_narrow<TKD_BF16>(p, grid, smem, st);
    return launch_fmt_all<TKD_BF16>(p, grid, smem, st);
}
int tkd_tc_clusters_bf16(size_t smem) { return tc_clusters<TKD_BF16>(smem); }
