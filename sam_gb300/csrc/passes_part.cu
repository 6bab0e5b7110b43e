// One unit of a pass's kernels: the lengths of part SAMGPU_PART of SAMGPU_PARTS
// of pass SAMGPU_PASS (zinv, yinv, x, yfwd, zfwd) in precision SAMGPU_T.
// build.py compiles this file once for each.
#include "passes_impl.cuh"

namespace samgpu {

#define SAMGPU_ARGS_zinv ZInvArgs
#define SAMGPU_ARGS_yinv YInvArgs
#define SAMGPU_ARGS_x XPassArgs
#define SAMGPU_ARGS_yfwd YFwdArgs
#define SAMGPU_ARGS_zfwd ZFwdArgs
#define SAMGPU_LAUNCH_zinv launch_z_inv_part
#define SAMGPU_LAUNCH_yinv launch_y_inv_part
#define SAMGPU_LAUNCH_x launch_x_pass_part
#define SAMGPU_LAUNCH_yfwd launch_y_fwd_part
#define SAMGPU_LAUNCH_zfwd launch_z_fwd_part
#define SAMGPU_SMEM_zinv smem_zinv_part
#define SAMGPU_SMEM_yinv smem_yinv_part
#define SAMGPU_SMEM_x smem_x_part
#define SAMGPU_SMEM_yfwd smem_yfwd_part
#define SAMGPU_SMEM_zfwd smem_zfwd_part
#define SAMGPU_CAT2(a, b) a##b
#define SAMGPU_CAT(a, b) SAMGPU_CAT2(a, b)

template void SAMGPU_CAT(SAMGPU_LAUNCH_, SAMGPU_PASS)<SAMGPU_T, SAMGPU_PART, SAMGPU_PARTS>(
    const SAMGPU_CAT(SAMGPU_ARGS_, SAMGPU_PASS)<SAMGPU_T>&, const FftPlan*, size_t, cudaStream_t);
template void SAMGPU_CAT(SAMGPU_SMEM_, SAMGPU_PASS)<SAMGPU_T, SAMGPU_PART, SAMGPU_PARTS>(int, int);

}  // namespace samgpu
