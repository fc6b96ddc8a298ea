// tkd_wide_bfp8.cu: the kernel for more than 32 rows, for one weight format.
#include "tkd_wide.cuh"

int tkd_launch_wide_bfp8(const TkdWide& p, size_t smem, cudaStream_t st) { return launch_wide_fmt<TKD_BFP8>(p, smem, st); }
