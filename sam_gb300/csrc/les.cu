// Subgrid-model routines of the reference (filter.f, sm.f, dm.f) and the
// mean-profile routine get_mean.f, in FP64 on haloed (Nx+2, Ny+2, Nz+2) grids.
//
// filter.f, sm.f and dm.f include a header the reference does not ship
// (speciso.h).  Its symbols are defined from their use:
//   Lx = Nx+2, Ly = Ny+2, Lz = Nz+2: planes 1 and N+2 are periodic halos
//     (periodicity.f:7-32);
//   ifact = (1,1,1,2,2,2) over the symmetric tensor (S11,S22,S33,S12,S23,S13);
//   ip = (1,2,3,1,2,1), jp = (1,2,3,2,3,3): index pairs of that tensor;
//   alpha_sq = 4: (test/grid filter width)^2 for the 1-4-1 test filter;
//   delta_sq = (dx dy dz)^(2/3) (init.f:28).
// The plane-by-plane sweeps of sm.f and dm.f become stencils over the whole
// volume: with periodic halos in the input every plane slot they read is the
// periodic neighbour of the plane being processed, so each point can be
// computed independently.
#include <cuda_runtime.h>
#include <math.h>

#include "common.cuh"
#include "fx64.cuh"
#include "les.cuh"

namespace samgpu {

struct Halo {
  int nx, ny, nz;
  __device__ __forceinline__ long long at(int i, int j, int k) const {
    return (long long)i + (long long)(nx + 2) * ((long long)j + (long long)(ny + 2) * k);
  }
  __device__ __forceinline__ long long vol() const { return (long long)(nx + 2) * (ny + 2) * (nz + 2); }
  // interior (periodic) index 0..n-1 of a wrapped coordinate; the stencils
  // reach one point past either side, so a conditional add or subtract
  // replaces the integer remainder (valid for -n <= i < 2n)
  __device__ __forceinline__ static int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
  __device__ __forceinline__ int wx(int i) const { return wrap(i, nx); }
  __device__ __forceinline__ int wy(int j) const { return wrap(j, ny); }
  __device__ __forceinline__ int wz(int k) const { return wrap(k, nz); }
  __device__ __forceinline__ long long in(int i, int j, int k) const {
    return (long long)wx(i) + (long long)nx * ((long long)wy(j) + (long long)ny * wz(k));
  }
  __device__ __forceinline__ long long ninterior() const { return (long long)nx * ny * nz; }
};

// index pairs of the tensor's six components, ifact = (1,1,1,2,2,2)
__device__ constexpr int kIp[6] = {0, 1, 2, 0, 1, 0};
__device__ constexpr int kJp[6] = {0, 1, 2, 1, 2, 2};

// ---- filter.f:7-42 on one 2-D plane set: 1-4-1 across the three planes of
// f_bar(Lx,Ly,n_var,3) (halos included), 1-4-1 along y using those halo rows,
// then along x with periodic wrap, normalised by 1/6^3; halos periodic.
__global__ void k_filter(const double* __restrict__ f_bar, double* __restrict__ f_hat, int nx, int ny, int n_var) {
  const int lx = nx + 2, ly = ny + 2;
  const long long pl = (long long)lx * ly;
  const long long tot = (long long)lx * ly * n_var;
  const double w_inv = 1.0 / (6.0 * 6.0 * 6.0);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % lx), j = (int)((e / lx) % ly), n = (int)(e / pl);
    // the value at halo points is the periodic image of the interior result
    const int ii = i == 0 ? nx : (i == nx + 1 ? 1 : i);
    const int jj = j == 0 ? ny : (j == ny + 1 ? 1 : j);
    auto h = [&](int a, int b) {
      const long long o = (long long)a + (long long)lx * b + pl * n;
      return f_bar[o] + 4 * f_bar[o + pl * n_var] + f_bar[o + 2 * pl * n_var];
    };
    auto g = [&](int a) { return h(a, jj - 1) + 4 * h(a, jj) + h(a, jj + 1); };
    const int am = ii - 1 == 0 ? nx : ii - 1;  // periodic wrap of the y-filtered rows
    const int ap = ii + 1 == nx + 1 ? 1 : ii + 1;
    f_hat[e] = w_inv * (g(am) + 4 * g(ii) + g(ap));
  }
}

// ---- staggered-to-centre velocity u_bar on the interior (sm.f:47-49)
__global__ void k_ubar(const double* __restrict__ u, double* __restrict__ ub, Halo H) {
  const long long n = H.ninterior(), vol = H.vol();
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % H.nx) + 1, j = (int)((e / H.nx) % H.ny) + 1, k = (int)(e / ((long long)H.nx * H.ny)) + 1;
    ub[e] = 0.5 * (u[H.at(i, j, k)] + u[H.at(i - 1, j, k)]);
    ub[n + e] = 0.5 * (u[vol + H.at(i, j, k)] + u[vol + H.at(i, j - 1, k)]);
    ub[2 * n + e] = 0.5 * (u[2 * vol + H.at(i, j, k)] + u[2 * vol + H.at(i, j, k - 1)]);
  }
}

// strain (sm.f:57-75) at interior point (x, y, z) from periodic u_bar
__device__ __forceinline__ void strain(const double* __restrict__ ub, const Halo& H, int x, int y, int z, double dxi,
                                       double dyi, double dzi, double* s) {
  const long long n = H.ninterior();
  auto U = [&](int c, int a, int b, int d) { return ub[c * n + H.in(a, b, d)]; };
  s[0] = 0.5 * (U(0, x + 1, y, z) - U(0, x - 1, y, z)) * dxi;
  s[1] = 0.5 * (U(1, x, y + 1, z) - U(1, x, y - 1, z)) * dyi;
  s[2] = 0.5 * (U(2, x, y, z + 1) - U(2, x, y, z - 1)) * dzi;
  s[3] = .25 * ((U(0, x, y + 1, z) - U(0, x, y - 1, z)) * dyi + (U(1, x + 1, y, z) - U(1, x - 1, y, z)) * dxi);
  s[4] = .25 * ((U(1, x, y, z + 1) - U(1, x, y, z - 1)) * dzi + (U(2, x, y + 1, z) - U(2, x, y - 1, z)) * dyi);
  s[5] = .25 * ((U(2, x + 1, y, z) - U(2, x - 1, y, z)) * dxi + (U(0, x, y, z + 1) - U(0, x, y, z - 1)) * dzi);
}

__device__ __forceinline__ double smag(const double* s) {
  const double d = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
  const double o = s[3] * s[3] + s[4] * s[4] + s[5] * s[5];
  return sqrt(2.0 * (d + 2.0 * o));
}

// sm.f:77-86: vt = c_smag delta^2 |S| on the interior of the haloed output
__global__ void k_sm(const double* __restrict__ ub, double* __restrict__ vt, Halo H, double c_delta_sq, double dxi,
                     double dyi, double dzi) {
  const long long n = H.ninterior();
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(e % H.nx), y = (int)((e / H.nx) % H.ny), z = (int)(e / ((long long)H.nx * H.ny));
    double s[6];
    strain(ub, H, x, y, z, dxi, dyi, dzi, s);
    vt[H.at(x + 1, y + 1, z + 1)] = c_delta_sq * smag(s);
  }
}

// periodicity.f:7-32 on a haloed volume (every halo point from its image)
__global__ void k_periodic3(double* __restrict__ f, Halo H) {
  const long long tot = H.vol();
  const int lx = H.nx + 2, ly = H.ny + 2;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % lx), j = (int)((e / lx) % ly), k = (int)(e / ((long long)lx * ly));
    const bool halo = i == 0 || i == H.nx + 1 || j == 0 || j == H.ny + 1 || k == 0 || k == H.nz + 1;
    if (!halo) continue;
    const int ii = i == 0 ? H.nx : (i == H.nx + 1 ? 1 : i);
    const int jj = j == 0 ? H.ny : (j == H.ny + 1 ? 1 : j);
    const int kk = k == 0 ? H.nz : (k == H.nz + 1 ? 1 : k);
    f[e] = f[H.at(ii, jj, kk)];
  }
}

// dm.f:99-116: |S|, |S| S_ij and u_bar_i u_bar_j on the interior
//   q[0..5] = S, q[6..11] = |S| S, q[12..17] = ub_i ub_j, q[18] = |S| (with vt)
__global__ void k_dm_fields(const double* __restrict__ ub, double* __restrict__ q, Halo H, double dxi, double dyi,
                            double dzi, int with_smag) {
  const long long n = H.ninterior();
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(e % H.nx), y = (int)((e / H.nx) % H.ny), z = (int)(e / ((long long)H.nx * H.ny));
    double s[6];
    strain(ub, H, x, y, z, dxi, dyi, dzi, s);
    const double sm = smag(s);
    const double u[3] = {ub[e], ub[n + e], ub[2 * n + e]};
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      q[c * n + e] = s[c];
      q[(6 + c) * n + e] = sm * s[c];
      q[(12 + c) * n + e] = u[kIp[c]] * u[kJp[c]];
    }
    if (with_smag) q[18 * n + e] = sm;
  }
}

// dm.f:122-150: L_ij, M_ij at each interior point, per-CTA sums of
// ifact L M and ifact M M (fixed order, deterministic).  The 1-4-1 test filter
// is taken one direction at a time (across planes, along y, along x: filter.f's
// order): a CTA does a 32 x 8 x 2 tile, each of the 21 fields in turn.  In FP64
// that is 7 operations a point and field on the pipe that bounds the kernel
// (66 cycles each), so the filter runs on integers, as the transforms do: a
// tile's values of one field under its own power of two (55 bits below its
// largest value, cut off there: a quarter of an FP64 rounding of it), exact
// sums, one conversion back.  A tile that holds infinities, NaN, nothing but
// zeros or numbers near the smallest takes the sums in FP64.  The filtered
// values stay scaled by 216/256 (a power of two costs the integers nothing, and
// below one nothing that was finite overflows); the factors are taken out of
// the sums.
// Loads of the next field are in flight while this one is filtered.
// 256^3: 3.2 ms with integers (FP64 pipe 43 %, ALU 48 %), 6.9 in FP64 one
// direction at a time, 22 with the 27-point stencil.  64 registers (four CTAs
// per SM, a few spills) against 80 and 128: 3.2, 3.5 and 4.7 ms.
constexpr int kDmTx = 32, kDmTy = 8, kDmTz = 2;
static_assert(kDmTx * kDmTy == kThreads, "one column of points per thread");
static long long dm_tiles(int nx, int ny, int nz) {
  return (long long)((nx + kDmTx - 1) / kDmTx) * ((ny + kDmTy - 1) / kDmTy) * ((nz + kDmTz - 1) / kDmTz);
}
// 1-4-1 sums
__device__ __forceinline__ double sum141(double a, double b, double c) { return a + 4 * b + c; }
__device__ __forceinline__ long long sum141(long long a, long long b, long long c) { return a + (b << 2) + c; }

__global__ void __launch_bounds__(kThreads, 4)
    k_dm_lm(const double* __restrict__ ub, const double* __restrict__ q, Halo H, double alpha_sq,
            double* __restrict__ part) {
  constexpr int HX = kDmTx + 2, HY = kDmTy + 2, PZ = kDmTz + 2, NW = kThreads / 32;
  constexpr int kPts = HY * HX, kRows = kDmTy * HX;
  __shared__ long long s_h[kDmTz][kPts], s_g[kDmTz][kRows];
  __shared__ uint32_t s_max[2][NW];
  __shared__ double red[2][kThreads];
  const long long n = H.ninterior(), pl = (long long)H.nx * H.ny;
  const int tid = threadIdx.x, tx = tid & (kDmTx - 1), ty = tid / kDmTx;
  const int ntx = (H.nx + kDmTx - 1) / kDmTx, nty = (H.ny + kDmTy - 1) / kDmTy;
  const long long tiles = (long long)ntx * nty * ((H.nz + kDmTz - 1) / kDmTz);
  const double wm = 256.0 * (alpha_sq / 216.0);
  double num = 0.0, den = 0.0;
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int z0 = (int)(t / (ntx * nty)) * kDmTz, r = (int)(t % (ntx * nty));
    const int x0 = (r % ntx) * kDmTx, y0 = (r / ntx) * kDmTy;
    // this thread's points of the tile with halo (at most two), the planes' offsets
    long long off[2], zo[PZ];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = min(tid + i * kThreads, kPts - 1);
      const int xx = (x0 + e % HX - 1 + H.nx) % H.nx, yy = (y0 + e / HX - 1 + H.ny) % H.ny;
      off[i] = (long long)yy * H.nx + xx;
    }
#pragma unroll
    for (int p = 0; p < PZ; ++p) zo[p] = (long long)((z0 + p - 1 + H.nz) % H.nz) * pl;

    double v[2][PZ] = {};  // the current field at this thread's points
    const auto load = [&](const double* __restrict__ f) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (tid + i * kThreads < kPts)
#pragma unroll
          for (int p = 0; p < PZ; ++p) v[i][p] = f[zo[p] + off[i]];
    };
    const auto largest = [&](int buf) {  // of the loaded field, per warp
      uint32_t hm = 0;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (tid + i * kThreads < kPts)
#pragma unroll
          for (int p = 0; p < PZ; ++p) hm = max(hm, (uint32_t)__double2hiint(v[i][p]) & 0x7fffffffu);
      hm = __reduce_max_sync(0xffffffffu, hm);
      if ((tid & 31) == 0) s_max[buf][tid >> 5] = hm;
    };
    int buf = 0;
    __syncthreads();  // (the last tile's reads are done)
    load(ub);
    largest(buf);
    __syncthreads();
    // 216/256 of the loaded field, filtered, at this thread's points; loads the next field
    const auto filt = [&](const double* __restrict__ next, double* out) {
      uint32_t hm = s_max[buf][0];
#pragma unroll
      for (int w = 1; w < NW; ++w) hm = max(hm, s_max[buf][w]);
      const int E = (int)(hm >> 20);
      buf ^= 1;
      const bool fx = E >= 64 && E < 0x7ff;  // |v| < 2^(E - 1022)
      const auto planes = [&](auto conv) {
        using V = decltype(conv(0.0));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int e = tid + i * kThreads;
          if (e >= kPts) break;
          V c[PZ];
#pragma unroll
          for (int p = 0; p < PZ; ++p) c[p] = conv(v[i][p]);
#pragma unroll
          for (int p = 0; p < kDmTz; ++p) reinterpret_cast<V*>(s_h[p])[e] = sum141(c[p], c[p + 1], c[p + 2]);
        }
        __syncthreads();
        if (next) load(next);
#pragma unroll
        for (int p = 0; p < kDmTz; ++p)
          for (int e = tid; e < kRows; e += kThreads) {
            const V* h = reinterpret_cast<const V*>(s_h[p]) + e;
            reinterpret_cast<V*>(s_g[p])[e] = sum141(h[0], h[HX], h[2 * HX]);
          }
        if (next) largest(buf);
        __syncthreads();
      };
      if (fx) {
        planes([&](double d) { return fx_from(d, E + 8); });  // integers below 2^55, their sums below 2^63
#pragma unroll
        for (int p = 0; p < kDmTz; ++p) {
          const long long* g = s_g[p] + ty * HX + tx;
          out[p] = fx_to_alu(sum141(g[0], g[1], g[2]), E - 1085);
        }
      } else {
        planes([](double d) { return d; });
#pragma unroll
        for (int p = 0; p < kDmTz; ++p) {
          const double* g = reinterpret_cast<const double*>(s_g[p]) + ty * HX + tx;
          out[p] = 0x1p-8 * sum141(g[0], g[1], g[2]);
        }
      }
    };
    double uh[3][kDmTz], sh[6][kDmTz], w[kDmTz];
#pragma unroll
    for (int c = 0; c < 3; ++c) filt(c < 2 ? ub + (c + 1) * n : q, uh[c]);
#pragma unroll
    for (int c = 0; c < 6; ++c) filt(q + (c < 5 ? c + 1 : 6) * n, sh[c]);
#pragma unroll
    for (int p = 0; p < kDmTz; ++p) {
      double m[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) m[c] = sh[c][p];
      w[p] = wm * smag(m);
    }
    double n2[2][kDmTz] = {}, d2[2][kDmTz] = {};
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      double a[kDmTz], b[kDmTz];
      filt(q + (12 + c) * n, a);                    // |S| S_c
      filt(c < 5 ? q + (7 + c) * n : nullptr, b);   // u_i u_j
#pragma unroll
      for (int p = 0; p < kDmTz; ++p) {
        const double M = w[p] * sh[c][p] - a[p];                                    // 216/256 M
        const double L = 216.0 / 256.0 * b[p] - uh[kIp[c]][p] * uh[kJp[c]][p];      // (216/256)^2 L
        n2[c / 3][p] += L * M;
        d2[c / 3][p] += M * M;
      }
    }
    if (x0 + tx < H.nx && y0 + ty < H.ny)
#pragma unroll
      for (int p = 0; p < kDmTz; ++p)
        if (z0 + p < H.nz) {
          num += n2[0][p] + 2 * n2[1][p];
          den += d2[0][p] + 2 * d2[1][p];
        }
  }
  num *= 0x1p24 * (1.0 / (216.0 * 216.0 * 216.0));
  den *= 0x1p16 * (1.0 / (216.0 * 216.0));
  red[0][threadIdx.x] = num;
  red[1][threadIdx.x] = den;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) {
      red[0][threadIdx.x] += red[0][threadIdx.x + h];
      red[1][threadIdx.x] += red[1][threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = red[0][0];
    part[2 * blockIdx.x + 1] = red[1][0];
  }
}

// dm.f:176 and 183-189: c_delta_sq = -num / (2 den); vt = c_delta_sq |S|.
// clip: the coefficient the coupled closure uses, dm.f's value, or 0 where it
// is negative (backscatter would make the eddy viscosity negative) or
// undefined (no strain: 0/0)
__global__ void k_dm_finish(const double* __restrict__ part, int nblk, double* __restrict__ cds, int clip) {
  __shared__ double red[2][kThreads];
  double num = 0.0, den = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    num += part[2 * b];
    den += part[2 * b + 1];
  }
  red[0][threadIdx.x] = num;
  red[1][threadIdx.x] = den;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) {
      red[0][threadIdx.x] += red[0][threadIdx.x + h];
      red[1][threadIdx.x] += red[1][threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double v = -0.5 * red[0][0] / red[1][0];
    cds[0] = clip && !(v > 0.0) ? 0.0 : v;
  }
}

__global__ void k_dm_vt(const double* __restrict__ q, const double* __restrict__ cds, double* __restrict__ vt, Halo H) {
  const long long n = H.ninterior();
  const double c = cds[0];
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(e % H.nx), y = (int)((e / H.nx) % H.ny), z = (int)(e / ((long long)H.nx * H.ny));
    vt[H.at(x + 1, y + 1, z + 1)] = c * q[18 * n + e];
  }
}

// ---- get_mean.f:8-56 (i_symm = 0) on the kx = ky = 0 column.  One CTA;
// line 0 of the shared tile holds the synthesis, line 1 the linear profile.
__global__ void k_get_mean(double2* __restrict__ col, int mz, int kz, int nz, int i_remove,
                           const FftPlan* __restrict__ gpl, const fxw* __restrict__ gtw,
                           double* __restrict__ u_mean, double* __restrict__ jump_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FftPlan pl;
  __shared__ double s_jump;
  load_plan(&pl, gpl);
  __syncthreads();
  const int ld = line_stride(nz);
  fxw* s_tw = reinterpret_cast<fxw*>(smem_raw);
  double2* ln = reinterpret_cast<double2*>(s_tw + pl.tw_total);
  for (int e = threadIdx.x; e < pl.tw_total; e += blockDim.x) s_tw[e] = gtw[e];
  const double nz_inv = 1.0 / nz;
  for (int pass = 0; pass < 2; ++pass) {
    // rfftb of the packed profile: u_mean(1) = Re u(1), (2k-2, 2k-1) = u(k),
    // k = 2..kz_max+1; as a complex synthesis with the Hermitian extension
    for (int p = threadIdx.x; p < nz; p += blockDim.x) {
      double2 v = make_double2(0.0, 0.0);
      if (p == 0) v = make_double2(col[0].x, 0.0);
      else if (p <= kz) v = col[p];
      else if (p >= nz - kz) v = make_double2(col[nz - p].x, -col[nz - p].y);
      ln[sidx(p)] = v;
    }
    __syncthreads();
    fft_lines<+1>(ln, ld, 1, s_tw, pl);
    __syncthreads();
    if (threadIdx.x == 0) {
      const double m0 = ln[sidx(0)].x, m1 = ln[sidx(1 % nz)].x, m2 = ln[sidx(2 % nz)].x;
      const double l0 = ln[sidx(nz - 1)].x, l1 = ln[sidx((nz - 2 + nz) % nz)].x, l2 = ln[sidx((nz - 3 + nz) % nz)].x;
      const double u_n = 3.0 * m0 - 3.0 * m1 + m2;
      const double u_1 = 3.0 * l0 - 3.0 * l1 + l2;
      const double jmp = 0.5 * ((l0 - u_n) + (u_1 - m0));
      if (pass == 0) s_jump = jmp;
      else s_jump = s_jump - jmp;
    }
    for (int p = threadIdx.x; p < nz; p += blockDim.x) u_mean[p] = ln[sidx(p)].x;
    __syncthreads();
    if (pass == 1 || i_remove != 1) break;
    // the linear profile jump (k/Nz - 1/2), rfftf, and its first kz_max+1
    // packed entries scaled by 1/Nz (get_mean.f:24-32)
    const double jump = s_jump;
    __syncthreads();
    for (int p = threadIdx.x; p < nz; p += blockDim.x) ln[sidx(p)] = make_double2(jump * ((double)p * nz_inv - 0.5), 0.0);
    __syncthreads();
    fft_lines<-1>(ln, ld, 1, s_tw, pl);
    __syncthreads();
    if (threadIdx.x == 0) {
      // packed r(0) = X0, r(2k-1) = Re Xk, r(2k) = Im Xk (0-based)
      auto packed = [&](int idx) {
        if (idx == 0) return ln[sidx(0)].x;
        const int k = (idx + 1) / 2;
        return (idx % 2 == 1) ? ln[sidx(k)].x : ln[sidx(k)].y;
      };
      auto scaled = [&](int idx) { return idx <= kz ? packed(idx) * nz_inv : packed(idx); };
      col[0].x -= scaled(0);
      for (int k = 1; k <= kz; ++k) {
        const double wr = scaled(2 * k - 1), wi = scaled(2 * k);
        const int k2 = mz - k;
        col[k].x -= wr;
        col[k].y -= wi;
        col[k2].x -= wr;
        col[k2].y += wi;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) jump_out[0] = s_jump;
}

static int grid_of(long long n) {
  long long g = (n + kThreads - 1) / kThreads;
  if (g > sm_count() * 16) g = sm_count() * 16;
  return (int)(g < 1 ? 1 : g);
}

void les_filter(const double* f_bar, double* f_hat, int nx, int ny, int n_var, cudaStream_t s) {
  k_filter<<<grid_of((long long)(nx + 2) * (ny + 2) * n_var), kThreads, 0, s>>>(f_bar, f_hat, nx, ny, n_var);
}

static Halo halo(int nx, int ny, int nz) {
  Halo H;
  H.nx = nx; H.ny = ny; H.nz = nz;
  return H;
}

void les_sm(const double* u, double* ub, double* vt, int nx, int ny, int nz, double c_delta_sq, double dxi, double dyi,
            double dzi, cudaStream_t s) {
  const Halo H = halo(nx, ny, nz);
  const long long n = (long long)nx * ny * nz;
  k_ubar<<<grid_of(n), kThreads, 0, s>>>(u, ub, H);
  k_sm<<<grid_of(n), kThreads, 0, s>>>(ub, vt, H, c_delta_sq, dxi, dyi, dzi);
  k_periodic3<<<grid_of((long long)(nx + 2) * (ny + 2) * (nz + 2)), kThreads, 0, s>>>(vt, H);
}

int les_dm_blocks(int nx, int ny, int nz) {
  const long long t = dm_tiles(nx, ny, nz);
  return (int)(t < sm_count() * 12 ? t : sm_count() * 12);
}

void les_dm(const double* u, double* ub, double* q, double* part, double* cds, double* vt, int nx, int ny, int nz,
            double alpha_sq, double dxi, double dyi, double dzi, cudaStream_t s) {
  const Halo H = halo(nx, ny, nz);
  const long long n = (long long)nx * ny * nz;
  const int nb = grid_of(n), nt = les_dm_blocks(nx, ny, nz);
  k_ubar<<<nb, kThreads, 0, s>>>(u, ub, H);
  k_dm_fields<<<nb, kThreads, 0, s>>>(ub, q, H, dxi, dyi, dzi, 1);
  k_dm_lm<<<nt, kThreads, 0, s>>>(ub, q, H, alpha_sq, part);
  k_dm_finish<<<1, kThreads, 0, s>>>(part, nt, cds, 0);
  k_dm_vt<<<nb, kThreads, 0, s>>>(q, cds, vt, H);
  k_periodic3<<<grid_of((long long)(nx + 2) * (ny + 2) * (nz + 2)), kThreads, 0, s>>>(vt, H);
}

// ---- coupled dynamic closure: u_bar (sm.f:47-49) straight from the physical
// velocity P(n, z, y, x) of the x pass (working precision), periodic
template <typename T>
__global__ void k_ubar_phys(const T* __restrict__ u, double* __restrict__ ub, Halo H) {
  const long long n = H.ninterior();
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(e % H.nx), y = (int)((e / H.nx) % H.ny), z = (int)(e / ((long long)H.nx * H.ny));
    ub[e] = 0.5 * ((double)u[e] + (double)u[H.in(x - 1, y, z)]);
    ub[n + e] = 0.5 * ((double)u[n + e] + (double)u[n + H.in(x, y - 1, z)]);
    ub[2 * n + e] = 0.5 * ((double)u[2 * n + e] + (double)u[2 * n + H.in(x, y, z - 1)]);
  }
}

// u_bar (3), the 18 fields of k_dm_fields, partial sums
size_t les_dynamic_work(int nx, int ny, int nz) {
  const size_t n = (size_t)nx * ny * nz;
  return 21 * n + 2 * (size_t)les_dm_blocks(nx, ny, nz);
}

template <typename T>
void les_dynamic(const T* phys, double* work, double* cds, int nx, int ny, int nz, double dxi, double dyi,
                 double dzi, cudaStream_t s) {
  const Halo H = halo(nx, ny, nz);
  const size_t n = (size_t)nx * ny * nz;
  double* ub = work;
  double* q = ub + 3 * n;
  double* part = q + 18 * n;
  const int nb = grid_of((long long)n), nt = les_dm_blocks(nx, ny, nz);
  k_ubar_phys<T><<<nb, kThreads, 0, s>>>(phys, ub, H);
  k_dm_fields<<<nb, kThreads, 0, s>>>(ub, q, H, dxi, dyi, dzi, 0);
  k_dm_lm<<<nt, kThreads, 0, s>>>(ub, q, H, 4.0, part);
  k_dm_finish<<<1, kThreads, 0, s>>>(part, nt, cds, 1);
}
template void les_dynamic<double>(const double*, double*, double*, int, int, int, double, double, double,
                                  cudaStream_t);
template void les_dynamic<float>(const float*, double*, double*, int, int, int, double, double, double,
                                 cudaStream_t);

// ---- training data of the learned closure: box filter and downsample by f
// of the physical fields P(n, z, y, x) (Lu fields): block means of u_a,
// T, the velocity products u_a u_b (rhs.f's order) and u_a T, written as
// out(X, Y, Z, m) with X = Nx/f fastest, m = 0..Lu+Lr-1.
template <typename T>
__global__ void k_box_filter(const T* __restrict__ ph, int lu, int nx, int ny, int nz, int f, double* __restrict__ out) {
  const int cx = nx / f, cy = ny / f, cz = nz / f;
  const long long nc = (long long)cx * cy * cz, np = (long long)nx * ny * nz;
  const int lr = lu == 4 ? 9 : 6;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nc; e += (long long)gridDim.x * blockDim.x) {
    const int X = (int)(e % cx), Y = (int)((e / cx) % cy), Z = (int)(e / ((long long)cx * cy));
    double acc[13];
#pragma unroll
    for (int m = 0; m < 13; ++m) acc[m] = 0.0;
    for (int k = 0; k < f; ++k)
      for (int j = 0; j < f; ++j)
        for (int i = 0; i < f; ++i) {
          const long long p = ((long long)(Z * f + k) * ny + (Y * f + j)) * nx + (X * f + i);
          const double u = ph[p], v = ph[np + p], w = ph[2 * np + p];
          const double t = lu == 4 ? (double)ph[3 * np + p] : 0.0;
          acc[0] += u; acc[1] += v; acc[2] += w; acc[3] += t;
          acc[4] += u * u; acc[5] += u * v; acc[6] += v * v; acc[7] += u * w; acc[8] += v * w; acc[9] += w * w;
          acc[10] += u * t; acc[11] += v * t; acc[12] += w * t;
        }
    const double inv = 1.0 / ((double)f * f * f);
    int m = 0;
    for (int q = 0; q < lu; ++q) out[(long long)(m++) * nc + e] = acc[q] * inv;
    for (int q = 0; q < lr; ++q) out[(long long)(m++) * nc + e] = acc[4 + q] * inv;
  }
}

template <typename T>
__global__ void k_to_double(const T* __restrict__ a, double* __restrict__ b, long long n) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    b[e] = (double)a[e];
}

template <typename T>
void les_box_filter(const T* ph, int lu, int nx, int ny, int nz, int f, double* out, cudaStream_t s) {
  const long long nc = (long long)(nx / f) * (ny / f) * (nz / f);
  k_box_filter<T><<<grid_of(nc), kThreads, 0, s>>>(ph, lu, nx, ny, nz, f, out);
}
template <typename T>
void les_to_double(const T* a, double* b, long long n, cudaStream_t s) {
  k_to_double<T><<<grid_of(n), kThreads, 0, s>>>(a, b, n);
}
template void les_box_filter<double>(const double*, int, int, int, int, int, double*, cudaStream_t);
template void les_box_filter<float>(const float*, int, int, int, int, int, double*, cudaStream_t);
template void les_to_double<double>(const double*, double*, long long, cudaStream_t);
template void les_to_double<float>(const float*, double*, long long, cudaStream_t);

void les_get_mean(double2* col, int mz, int kz, int nz, int i_remove, const FftPlan* dplan, const fxw* tw,
                  const FftPlan& hplan, double* u_mean, double* jump, cudaStream_t s) {
  const int ld = line_stride(nz);
  const size_t sm = sizeof(double2) * ((size_t)hplan.tw_total + (size_t)ld) + 16;
  k_get_mean<<<1, kThreads, sm, s>>>(col, mz, kz, nz, i_remove, dplan, tw, u_mean, jump);
}

}  // namespace samgpu
