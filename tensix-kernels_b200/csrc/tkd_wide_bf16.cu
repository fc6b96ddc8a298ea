// tkd_wide_bf16.cu: the kernel for more than 32 rows, for one weight format.
#include "tkd_wide.cuh"

int tkd_launch_wide_bf16(const TkdWide& p, size_t smem, cudaStream_t st) { return launch_wide_fmt<TKD_BF16>(p, smem, st); }
