// The passes' launchers: each hands a length to the unit that compiled its
// kernels (passes_part.cu).  The numbers of units are build.py's.
#include "passes.cuh"

namespace samgpu {

#define SAMGPU_DECLARE(LAUNCH, ARGS, PASS)                                                      \
  template <typename T, int PART, int PARTS>                                                    \
  void LAUNCH##_part(const ARGS<T>& a, const FftPlan* pl, size_t smem, cudaStream_t s);          \
  template <typename T, int PART, int PARTS> void smem_##PASS##_part(int n, int optin);
SAMGPU_DECLARE(launch_z_inv, ZInvArgs, zinv)
SAMGPU_DECLARE(launch_y_inv, YInvArgs, yinv)
SAMGPU_DECLARE(launch_x_pass, XPassArgs, x)
SAMGPU_DECLARE(launch_y_fwd, YFwdArgs, yfwd)
SAMGPU_DECLARE(launch_z_fwd, ZFwdArgs, zfwd)

#define SAMGPU_CASE(CALL, T, I, PARTS) \
  case I:                              \
    CALL(T, I, PARTS);                 \
    break;
#define SAMGPU_SWITCH_2(CALL, T, P) SAMGPU_CASE(CALL, T, 0, P) SAMGPU_CASE(CALL, T, 1, P)
#define SAMGPU_SWITCH_3(CALL, T, P) SAMGPU_SWITCH_2(CALL, T, P) SAMGPU_CASE(CALL, T, 2, P)
#define SAMGPU_SWITCH_4(CALL, T, P) SAMGPU_SWITCH_3(CALL, T, P) SAMGPU_CASE(CALL, T, 3, P)
#define SAMGPU_SWITCH_6(CALL, T, P) SAMGPU_SWITCH_4(CALL, T, P) SAMGPU_CASE(CALL, T, 4, P) SAMGPU_CASE(CALL, T, 5, P)

#define SAMGPU_PASS(LAUNCH, ARGS, PASS, N, PREP, T, PARTS)                                                        \
  template <> void LAUNCH<T>(const ARGS<T>& a0, const FftPlan* pl, size_t smem, cudaStream_t s) {                \
    const ARGS<T> a = PREP(a0);                                                                                  \
    switch (path_part(a.g.N, PARTS)) { SAMGPU_SWITCH_##PARTS(SAMGPU_RUN_##PASS, T, PARTS) }                       \
  }                                                                                                               \
  static void smem_##PASS(T*, int n, int optin) {                                                                 \
    switch (path_part(n, PARTS)) { SAMGPU_SWITCH_##PARTS(SAMGPU_OPT_##PASS, T, PARTS) }                           \
  }
#define SAMGPU_RUN_zinv(T, I, P) launch_z_inv_part<T, I, P>(a, pl, smem, s)
#define SAMGPU_RUN_yinv(T, I, P) launch_y_inv_part<T, I, P>(a, pl, smem, s)
#define SAMGPU_RUN_x(T, I, P) launch_x_pass_part<T, I, P>(a, pl, smem, s)
#define SAMGPU_RUN_yfwd(T, I, P) launch_y_fwd_part<T, I, P>(a, pl, smem, s)
#define SAMGPU_RUN_zfwd(T, I, P) launch_z_fwd_part<T, I, P>(a, pl, smem, s)
#define SAMGPU_OPT_zinv(T, I, P) smem_zinv_part<T, I, P>(n, optin)
#define SAMGPU_OPT_yinv(T, I, P) smem_yinv_part<T, I, P>(n, optin)
#define SAMGPU_OPT_x(T, I, P) smem_x_part<T, I, P>(n, optin)
#define SAMGPU_OPT_yfwd(T, I, P) smem_yfwd_part<T, I, P>(n, optin)
#define SAMGPU_OPT_zfwd(T, I, P) smem_zfwd_part<T, I, P>(n, optin)

SAMGPU_PASS(launch_z_inv, ZInvArgs, zinv, nz, , double, 3)
SAMGPU_PASS(launch_y_inv, YInvArgs, yinv, ny, , double, 3)
SAMGPU_PASS(launch_x_pass, XPassArgs, x, nx, prep_x_pass, double, 6)
SAMGPU_PASS(launch_y_fwd, YFwdArgs, yfwd, ny, , double, 3)
SAMGPU_PASS(launch_z_fwd, ZFwdArgs, zfwd, nz, prep_z_fwd, double, 4)
SAMGPU_PASS(launch_z_inv, ZInvArgs, zinv, nz, , float, 2)
SAMGPU_PASS(launch_y_inv, YInvArgs, yinv, ny, , float, 2)
SAMGPU_PASS(launch_x_pass, XPassArgs, x, nx, prep_x_pass, float, 3)
SAMGPU_PASS(launch_y_fwd, YFwdArgs, yfwd, ny, , float, 2)
SAMGPU_PASS(launch_z_fwd, ZFwdArgs, zfwd, nz, prep_z_fwd, float, 2)

template <typename T> static void smem_all(int nx, int ny, int nz) {
  const int optin = smem_optin();
  T* t = nullptr;
  smem_zinv(t, nz, optin);
  smem_yinv(t, ny, optin);
  smem_x(t, nx, optin);
  smem_yfwd(t, ny, optin);
  smem_zfwd(t, nz, optin);
}
template <> void set_smem_limits<double>(int nx, int ny, int nz) { smem_all<double>(nx, ny, nz); }
template <> void set_smem_limits<float>(int nx, int ny, int nz) { smem_all<float>(nx, ny, nz); }

}  // namespace samgpu
