// Argument blocks and launchers of the transform passes (passes_impl.cuh,
// instantiated in passes_part.cu and passes_ens.cu).
// Strides are in complex (or real, for physical arrays) elements.
#pragma once
#include "common.cuh"

namespace samgpu {

// The gradient fields of a subgrid closure behind the Lu factors: the strain
// S11 S12 S22 S13 S23 S33, with buoyancy the three parts of grad T, and for
// the learned closure's invariants the three of the vorticity.  k_z enters
// S13, S23, S33, dT/dz and the first two parts of the vorticity.
__host__ __device__ inline bool derive_in_y(int n, int lu, int lr) {
  const int m = n - lu;
  return m >= 0 && (m < 3 || (m >= 6 && m < lr && m < 8) || m == lr + 2);
}
// field of the j-th line the z pass takes, and the number of lines for nvar fields
__host__ __device__ inline int derive_z_field(int j, int lu, int lr) {
  const int t = lr > 6 ? 1 : 0, m = j - lu;
  return m < 0 ? j : lu + (m < 3 ? 3 + m : (m < 3 + t ? 8 : lr + m - 3 - t));
}
inline int derive_z_lines(int nvar, int lu, int lr) {
  int k = 0;
  for (int n = 0; n < nvar; ++n) k += !derive_in_y(n, lu, lr);
  return k;
}

template <typename T>
struct ZInvArgs {
  Grid g;
  // FFT schedule of length-256 lines: 0 the 16 x 16 register path, 1 the
  // compile-time Stockham stages (radix 8, 8, 4); chosen by the autotuner
  int sched;
  const cx_t<T>* in;   // rows of Nz_min modes
  cx_t<T>* out;        // A(n, z, kx, ky)
  const tw_t<T>* tw;   // twiddles of the Nz plan
  int nvar, ty, ld;
  // derive = 1: fields n >= Lu are gradient fields formed from the velocity
  // (and T) rows while loading; the launch has those that k_z enters
  // (derive_z_field), the y pass forms the others
  int derive;
  long long in_ky, in_kx, in_n;
  long long out_kx, out_z, out_n;
};

template <typename T>
struct YInvArgs {
  Grid g;
  // FFT schedule of length-256 lines: 0 the 16 x 16 register path, 1 the
  // compile-time Stockham stages (radix 8, 8, 4); chosen by the autotuner
  int sched;
  const cx_t<T>* in;  // rows (one per kx) of Ny_min modes or Ny values
  cx_t<T>* out;       // B(n, z, y, kx)
  const tw_t<T>* tw;
  int nvar, tx, ld, in_full;
  int derive;  // 1: gradient fields without k_z (derive_in_y) are formed while loading
  long long in_kx, in_z, in_n;
  long long out_y, out_z, out_n;
};

// Threads of an x pass CTA.  In the FP32 16 x 16 register path (n = 256) a
// team of 16 threads transforms one line, and an 8-row tile holds 4 x 4
// input and 9 x 4 product lines: 18 teams do them in one and two full rounds
// (16 teams would need a third round a quarter full).  Other forms keep
// kThreads.
__host__ __device__ constexpr int x_threads(int bytes, bool reg16) { return bytes == 4 && reg16 ? 288 : kThreads; }

template <typename T>
struct XPassArgs {
  Grid g;
  // FFT schedule of length-256 lines: 0 the 16 x 16 register path, 1 the
  // compile-time Stockham stages (radix 8, 8, 4); chosen by the autotuner
  int sched;
  const cx_t<T>* in;   // in_mode 0: B(n, z, y, kx)
  const T* in_phys;    // in_mode 1: P(n, z, y, x)
  cx_t<T>* out;        // out_mode 1/2: C(m, z, kx, y)
  T* out_phys;         // out_mode 0: P(n, z, y, x)
  double* partials;    // vel_max partials (nblocks, lu, 4) or null
  const tw_t<T>* tw;
  // group: product lines transformed per round of out_mode 2 (a multiple of
  // the CTA's teams where it exceeds them), any split of the Lr * Y/2 lines
  int in_mode, out_mode, nin, yt, group, ld;
  int prod_lines;  // lines of room behind the input lines (products, vel_max's scratch)
  // vel_max partials: max_only = 1 leaves the sums to k_parseval (FP32 form)
  int max_only;
  int* vmax;  // max_only: per-field max |u| (float bit patterns) and the NaN flag, atomically
  T fn;  // 1/(2 Nx Ny): xy_trans_f.f:20's scale and the 1/2 of the pair split (launcher)
  // subgrid stress (les = 1): input fields Lu .. Lu+Lr-1 are the gradient
  // fields of the products; nu_t = C delta^2 |S| with C delta^2 read from
  // les_cds, kappa_t = nu_t * les_prt_inv
  // les = 2: per-point coefficients les_coef[(z Ny + y) Nx + x] =
  // (C_nu, C_kappa) of the learned closure, nu_t = C_nu les_dsq |S|,
  // kappa_t = C_kappa les_dsq |S|
  int les;
  const double* les_cds;
  double les_prt_inv;
  const float2* les_coef;
  double les_dsq;
  // out_mode 4: the closure's 12 invariants of point (z Ny + y) Nx + x as
  // BF16 [16] (columns 12..14 = 1.0, the network's bias inputs; 15 = 0)
  // from the input fields S (6), dT/dx (3, when Lr = 9) and w (3);
  // f_bz = buoy_fac_z, f_n2 = N^2, f_dsq = delta^2, f_nu = viscosity
  void* feat;
  double f_bz, f_n2, f_dsq, f_nu;
  long long in_y, in_z, in_n;
  long long out_kx, out_z, out_n;
  long long out_py, out_pz, out_pn;
  FastDiv fd_mx, fd_yp, fd_nx, fd_y;  // filled by the launcher
};

// The fused x passes of 256-point lines (k_x_pass_f256, k_x_pass_fx256): the
// resident step's form of the pass, with or without a subgrid closure.
constexpr int kXf256Threads = 288;                  // 18 teams of 16 (two rounds of 9 x 4 product lines)
constexpr int kXf256Teams = kXf256Threads / 16;
constexpr int kXf256Ld = 271;                       // line_stride(256)
static_assert(kXf256Ld == ((256 + (255 >> 4)) | 1), "line stride of a 256-point line");
__host__ __device__ constexpr size_t x_f256_smem(int lines, bool les) {
  return sizeof(float2) * (256 + (size_t)(lines + (les ? 0 : kXf256Teams)) * kXf256Ld);
}
// 16 or, with a closure, 18 teams (the 18 product lines of a 4-row tile)
__host__ __device__ constexpr int x_fx256_threads(bool les) { return les ? 288 : 256; }
__host__ __device__ constexpr size_t x_fx256_smem(int lines, bool les) {
  return (size_t)lines * (sizeof(fxc) * kXf256Ld + sizeof(FxLine)) +
         (les ? 0 : sizeof(fxw) * 256 + (size_t)(x_fx256_threads(false) / 16) * kXf256Ld * sizeof(long long));
}
template <typename T> inline size_t x_fused_smem(const XPassArgs<T>& a) {
  const int lines = a.nin * (a.yt / 2);
  return sizeof(T) == 4 ? x_f256_smem(lines, a.les != 0) : x_fx256_smem(lines, a.les != 0);
}
// whether a fused kernel runs this launch (else the general kernel)
template <typename T> inline bool x_fused(const XPassArgs<T>& a) {
  return a.g.nx == 256 && a.sched == 0 && a.in_mode == 0 && a.out_mode == 2 &&
         a.nin == a.g.lu + (a.les ? a.g.lr : 0) && (a.g.lr == 6 || a.g.lr == 9) && (!a.partials || a.max_only) &&
         a.yt >= 2 && a.yt % 2 == 0 && x_fused_smem(a) + 2048 <= (size_t)smem_optin();
}
// rows of a fused tile with a closure: 26 lines, three (FP32) or two CTAs per SM
constexpr int kXFusedLesRows = 4;

// The tables of a stage's integrating factors (FP64 resident step): 5 Mz
// doubles per kz, then, aligned, four per row (kx, ky).
__host__ __device__ inline size_t z_row_off(const Grid& g) { return (5 * (size_t)g.mz + 3) / 4 * 4; }
struct __align__(16) RowFactors {
  double ef[2], et[2];  // exp(-nu k^2 dt_fac) less one and itself, and with nu / Pr
};
template <typename D> __host__ __device__ inline auto z_row_tab(D* kz_tab, const Grid& g) {
  using V = typename std::conditional<std::is_const<D>::value, const RowFactors, RowFactors>::type;
  return reinterpret_cast<V*>(kz_tab + z_row_off(g));
}

template <typename T>
struct YFwdArgs {
  Grid g;
  // FFT schedule of length-256 lines: 0 the 16 x 16 register path, 1 the
  // compile-time Stockham stages (radix 8, 8, 4); chosen by the autotuner
  int sched;
  const cx_t<T>* in;  // C(m, z, kx, y)
  cx_t<T>* out;       // D(m, kx, ky, z)
  const tw_t<T>* tw;
  int nvar, tz, ld;
  long long in_kx, in_z, in_n;
  long long out_ky, out_kx, out_n;
  // FP64 form, resident stage: Mx more CTAs write the z-forward pass's tables of
  // this stage (ZFwdArgs::kz_tab, RowFactors), dt read on the device
  double* kz_tab;
  const DevState* kz_state;
  double kz_gamma, kz_zeta, kz_vis, kz_pr_inv;
};

// What a ky row of a z-forward tile contributes to its modes' wave numbers
// and (FP64 form) integrating factors exp(-nu k^2 dt_fac) = e(kx, ky) e(kz), each
// factor less one and itself, for the velocity and for T.
template <typename W> struct EpiRow {
  W rky, k_sq, ef[2], et[2];
};
// (these records follow the 16-byte elements of the lines)
static_assert(sizeof(FxScale) == 16 && sizeof(FxLine) == 16, "records keep the alignment of what follows them");
// Shared memory behind the lines of a z-forward tile of ty rows and nf
// fields (modes 1, 2): the scale of each fixed-point line, the rows' constants.
template <typename T> constexpr size_t z_fwd_extra(int mode, int nf, int ty) {
  if (mode == 0) return 0;
  return (sizeof(T) == 8 ? sizeof(FxScale) * nf * ty : 0) + sizeof(EpiRow<T>) * ty;
}

template <typename T>
struct ZFwdArgs {
  Grid g;
  // FFT schedule of length-256 lines: 0 the 16 x 16 register path, 1 the
  // compile-time Stockham stages (radix 8, 8, 4); chosen by the autotuner
  int sched;
  cx_t<T>* in;  // D(m, kx, ky, z); mode 0 writes the result back here
  const tw_t<T>* tw;
  int mode, nf, ty, ld;
  long long in_ky, in_kx, in_n;
  // mode 1 (rhs): r out and u_sav in
  cx_t<T>* r;
  long long r_ky, r_kx, r_n;
  const cx_t<T>* usav;
  long long sav_ky, sav_kx, sav_n;
  // mode 2 (stage): u, r (same layout), p, device state
  cx_t<T>* u;
  cx_t<T>* p;
  long long u_ky, u_kx, u_n;
  DevState* state;
  StageConsts sc;
  // FP64 form, mode 2: rkz(k), then the integrating factors' kz part less one
  // and itself for the velocity, then for T, written by the stage's y-forward pass (null: formed
  // per mode)
  const double* kz_tab;
  T nz_inv;                  // filled by the launcher: 1/Nz
  FastDiv fd_t, fd_m;  // filled by the launcher: ty, Nz_min
};

// A pass's kernels of one precision are compiled in `parts` units (passes_part.cu):
// length i of the compile-time lengths in unit i % parts, the run-time path in
// unit 0.
__host__ __device__ constexpr int path_part(int n, int parts) {
  if (!ct_length(n)) return 0;
  int i = 0;
  for (int m = 8; m < n; ++m) i += ct_length(m);
  return i % parts;
}
template <typename T>
inline int x_pass_blocks(const XPassArgs<T>& a) {
  return a.g.nz * ((a.g.ny + a.yt - 1) / a.yt);
}
// the launch-time fields of the x pass's and the z-forward pass's argument
// blocks (fast divisors, scales), shared by the launchers and the ensemble
// stage recorder
template <typename T>
XPassArgs<T> prep_x_pass(const XPassArgs<T>& a0) {
  XPassArgs<T> a = a0;
  a.fd_mx = make_fastdiv(a.g.mx);
  a.fd_yp = make_fastdiv(a.yt / 2);
  a.fd_nx = make_fastdiv(a.g.nx);
  a.fd_y = make_fastdiv(a.yt);
  a.fn = (T)(0.5 / ((double)a.g.nx * (double)a.g.ny));
  return a;
}
template <typename T>
ZFwdArgs<T> prep_z_fwd(const ZFwdArgs<T>& a0) {
  ZFwdArgs<T> a = a0;
  a.fd_t = make_fastdiv(a.ty);
  a.fd_m = make_fastdiv(a.g.mz);
  a.nz_inv = (T)(1.0 / (double)a.g.nz);
  return a;
}

template <typename T> void launch_z_inv(const ZInvArgs<T>& a, const FftPlan* pl, size_t smem, cudaStream_t s);
template <typename T> void launch_y_inv(const YInvArgs<T>& a, const FftPlan* pl, size_t smem, cudaStream_t s);
template <typename T> void launch_x_pass(const XPassArgs<T>& a, const FftPlan* pl, size_t smem, cudaStream_t s);
template <typename T> void launch_y_fwd(const YFwdArgs<T>& a, const FftPlan* pl, size_t smem, cudaStream_t s);
template <typename T> void launch_z_fwd(const ZFwdArgs<T>& a, const FftPlan* pl, size_t smem, cudaStream_t s);
// loads the pass kernels of precision T for a grid and opts them into the
// device's largest dynamic shared memory (before anything is captured)
template <typename T> void set_smem_limits(int nx, int ny, int nz);
// Shared memory of an FP64 x pass with products behind its lines: scale and
// norm of each of `in` input lines, scale of each of `prod` product lines.
template <typename T> constexpr size_t x_extra(int out_mode, int in, int prod) {
  return std::is_same<T, double>::value && out_mode == 2 ? sizeof(FxLine) * in + sizeof(FxScale) * prod : 0;
}
// vmax (max_only forms): ints 0..7 hold the per-field maxima (FP32 form: the
// float bit patterns in ints 0..3; FP64 form: bit patterns of doubles in ints
// 0..7, vkind = 1), int 8 the non-finite flag
void launch_vel_max_finish(const double* partials, int nblk, const Grid& g, DevState* st, int i_cfl, double cfl0,
                           double adv_cfl_limit, cudaStream_t s, const double* pv = nullptr, int npv = 0,
                           int* vmax = nullptr, int vkind = 0);
constexpr int kVmaxInts = 16;  // the vmax block at the end of pv
// vel_max's sums from wave space (Parseval), FP64 arithmetic on the state U
// (Lu fields (kx, ky, kz)): pv[b * Lu + f] = block b's share of
// sum w |u|^2 (w = 1 for kx = 0, 2 otherwise), pv[npv * Lu + f] = u(0,0,0).
constexpr int kParsevalBlocks = 152 * 6;  // at most
// four modes a thread at least (a 32^3 run has 4851)
inline int parseval_blocks(const Grid& g) {
  const long long b = ((long long)g.mx * g.my * g.mz + 4 * kThreads - 1) / (4 * kThreads);
  return (int)(b < kParsevalBlocks ? b : kParsevalBlocks);
}
template <typename T> void launch_parseval(const cx_t<T>* u, const Grid& g, double* pv, cudaStream_t s);
void launch_x2z(const double2* in, double2* out, const Grid& g, int nvar, int nx2, cudaStream_t s);

}  // namespace samgpu
