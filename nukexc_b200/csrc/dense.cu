// Dense-matrix entry points with the shapes of the reference's dense
// algorithm (fill_collocation, compute_density_and_sigma, compute_gga ...,
// sto_potential_collocation_scaled, compute_half_inverse).  They operate on
// caller-owned device buffers.  The batched, screened Fock build of plan.cu
// is the hot path; these exist so the reference's dense call sequence can be
// replaced one function at a time.
#include <cublas_v2.h>
#include <cusolverDn.h>

#include <algorithm>
#include <functional>
#include <mutex>
#include <vector>

#include "dmma.cuh"
#include "functionals.cuh"
#include "host_setup.hpp"

namespace nkx {

nkx_status run_guarded(const char *where, const std::function<void()> &fn);

// Workspaces of the dense entry points come from a memory pool of the
// library's own, one per device, allocated and freed in stream order: a call
// allocates and frees up to a few hundred megabytes, which took cudaMalloc /
// cudaFree 1 to 3 ms (and a device-wide synchronisation) against 0.1 to 0.5 ms
// of kernels.  The pool keeps at most kPoolKeep bytes between calls: workspaces
// are freed before a call's last synchronisation, which is when the pool gives
// back what exceeds that.  What it keeps is not lost to the process: the driver
// takes it back for a cudaMalloc that would fail otherwise.  A call that needs more
// in all takes it by cudaMalloc: a pool that has to grow for every call is slower
// (core Hamiltonian of three waters, 1.1 GB: 11.6 ms by the pool, 7.8 by cudaMalloc).
constexpr uint64_t kPoolKeep = (uint64_t)256 << 20;
static cudaMemPool_t workspace_pool(int dev, bool create) {
  static std::mutex mu;
  static cudaMemPool_t pools[128] = {};
  NKX_REQUIRE(dev >= 0 && dev < 128, NKX_ERR_ARG, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(mu);
  if (!pools[dev] && create) {
    cudaMemPoolProps p{};
    p.allocType = cudaMemAllocationTypePinned;
    p.location.type = cudaMemLocationTypeDevice;
    p.location.id = dev;
    cudaMemPool_t pool = nullptr;
    NKX_CUDA(cudaMemPoolCreate(&pool, &p));
    uint64_t keep = kPoolKeep;
    NKX_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    pools[dev] = pool;
  }
  return pools[dev];
}
cudaError_t device_free_bytes(size_t *bytes) {
  size_t tot = 0;
  uint64_t held = 0, used = 0;
  int dev = 0;
  cudaMemPool_t pool = nullptr;
  const cudaError_t e = cudaMemGetInfo(bytes, &tot);
  if (e == cudaSuccess && cudaGetDevice(&dev) == cudaSuccess && (pool = workspace_pool(dev, false)) &&
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess && held > used)
    *bytes += held - used;
  return e;
}

// where a call's workspaces come from, by the bytes of all of them
struct Source {
  cudaStream_t s;
  bool pooled;
  Source(cudaStream_t stream, size_t bytes = 0) : s(stream), pooled(bytes <= kPoolKeep) {}
};

template <class T>
struct DevBuf {
  T *p = nullptr;
  Source from;
  DevBuf(size_t n, Source source) : from(source) {
    if (!n) return;
    int dev = 0;
    NKX_CUDA(cudaGetDevice(&dev));
    if (from.pooled)
      NKX_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void **>(&p), n * sizeof(T), workspace_pool(dev, true), from.s));
    else
      NKX_CUDA(cudaMalloc(&p, n * sizeof(T)));
  }
  ~DevBuf() {
    if (p && from.pooled) cudaFreeAsync(p, from.s);
    if (p && !from.pooled) cudaFree(p);
  }
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
};

// fn's work on s, then the wait for it, with fn's workspaces freed in between
template <class F>
static void run_and_wait(cudaStream_t s, F &&fn) {
  fn();
  NKX_CUDA(cudaStreamSynchronize(s));
}

// fill_collocation / fill_grad_collocation, a thread per element (one water,
// 68k points: 50 us with gradients; a thread per point and run of functions
// sharing the radial factor, through a shared tile, took 64)
__global__ void colloc_dense_kernel(const StoFunc *__restrict__ f, int nbf, const double *__restrict__ pts,
                                    long npts, double *phi, double *gx, double *gy, double *gz) {
  const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= (long)nbf * npts) return;
  const int mu = (int)(idx % nbf);
  const long g = idx / nbf;
  const double px = pts[3 * g], py = pts[3 * g + 1], pz = pts[3 * g + 2];
  if (gx) {
    double v, a, b, c;
    sto_value_grad(f[mu], px, py, pz, v, a, b, c);
    phi[idx] = v;
    gx[idx] = a;
    gy[idx] = b;
    gz[idx] = c;
  } else {
    phi[idx] = sto_value(f[mu], px, py, pz);
  }
}

// T_i = sum_mu C(mu,i) phi(mu,g); rho = sum occ_i T_i^2, grad rho =
// 2 sum occ_i T_i grad T_i, sigma = |grad rho|^2 (density.hpp:188-255).  One
// CTA per 64 points with gradients or 256 without: its 256 (component, point)
// rows go 32 to a warp as four 8-row DMMA tiles against 8 NN orbitals, 16
// functions a step through a ring of shared stages (rows padded by four
// doubles: conflict-free fragments); orbital tiles follow one another and the
// sums stay in registers.  VEC: every row starts on a 16-byte boundary (even
// nbf, aligned matrices) and is copied 16 bytes at a time, else 8.
// Bound: the collocation's HBM reads up to about 16 orbitals, then FP64 (one
// water with gradients, 5 orbitals: 103 us with a warp per point, 36 now).
constexpr int kDdK = 16, kDdLd = kDdK + 4, kDdStages = 3;
template <int NN>
constexpr int kDdSmem = kDdStages * (256 + 8 * NN) * kDdLd * 8;
template <bool GRAD, int NN, bool VEC>
__global__ void __launch_bounds__(256)
    density_dense_kernel(int nbf, long npts, const double *__restrict__ phi, const double *__restrict__ gx,
                         const double *__restrict__ gy, const double *__restrict__ gz, int nocc,
                         const double *__restrict__ C, const double *__restrict__ occ, double *__restrict__ rho,
                         double *__restrict__ grad, double *__restrict__ sigma) {
  constexpr int NT = 8 * NN, kStage = (256 + NT) * kDdLd, PTS = GRAD ? 64 : 256;
  constexpr int W = VEC ? 2 : 1, PARTS = kDdK / W;  // doubles a copy, copies a row
  extern __shared__ __align__(16) double dsm[];
  const long g0 = blockIdx.x * (long)PTS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fk = lane & 3;
  const int ksteps = (nbf + kDdK - 1) / kDdK, total = ksteps * ((nocc + NT - 1) / NT);
  auto copy = [&](double *dst, const double *src, bool in) {
    if constexpr (VEC)
      cp_async16_fill(dst, src, in);
    else
      cp_async8_fill(dst, src, in);
  };
  auto issue = [&](int t, int st) {
    if (t < total) {
      const int f0 = (t % ksteps) * kDdK, i0 = (t / ksteps) * NT;
      double *Ps = dsm + st * kStage, *Cs = Ps + 256 * kDdLd;
#pragma unroll
      for (int e = threadIdx.x; e < 256 * PARTS; e += 256) {
        const int row = e / PARTS, part = W * (e % PARTS);
        // GRAD: row = 32 (point / 8) + 8 comp + point % 8
        const int c = GRAD ? (row / 8) % 4 : 0;
        const long g = g0 + (GRAD ? 8 * (row / 32) + row % 8 : row);
        const double *src = c == 0 ? phi : c == 1 ? gx : c == 2 ? gy : gz;
        const bool in = g < npts && f0 + part < nbf;
        copy(Ps + row * kDdLd + part, in ? src + (size_t)g * nbf + f0 + part : src, in);
      }
      for (int e = threadIdx.x; e < NT * PARTS; e += 256) {
        const int row = e / PARTS, part = W * (e % PARTS);
        const bool in = i0 + row < nocc && f0 + part < nbf;
        copy(Cs + row * kDdLd + part, in ? C + (size_t)(i0 + row) * nbf + f0 + part : C, in);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int st = 0; st < kDdStages - 1; ++st) issue(st, st);
  double sm[4] = {0.0, 0.0, 0.0, 0.0}, acc[4][NN][2];
  for (int t = 0; t < total; ++t) {
    if (t % ksteps == 0) {
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < NN; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
    }
    cp_async_wait<kDdStages - 2>();
    __syncthreads();  // step t is visible; the stage refilled below was read in step t - 1
    issue(t + kDdStages - 1, (t + kDdStages - 1) % kDdStages);
    const double *Ps = dsm + (t % kDdStages) * kStage, *Cs = Ps + 256 * kDdLd;
#pragma unroll
    for (int k = 0; k < kDdK; k += 4) {
      double av[4], bv[NN];
#pragma unroll
      for (int m = 0; m < 4; ++m) av[m] = Ps[(32 * warp + 8 * m + fr) * kDdLd + k + fk];
#pragma unroll
      for (int n = 0; n < NN; ++n) bv[n] = Cs[(8 * n + fr) * kDdLd + k + fk];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < NN; ++n) dmma884(acc[m][n], av[m], bv[n]);
    }
    if (t % ksteps == ksteps - 1) {
#pragma unroll
      for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = (t / ksteps) * NT + 8 * n + 2 * fk + h;
          if (i >= nocc) continue;  // a zero column, but 0 x Inf is NaN
          const double o = occ[i];
#pragma unroll
          for (int m = 0; m < 4; ++m) sm[m] += o * acc[GRAD ? 0 : m][n][h] * acc[m][n][h];
        }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    sm[m] += __shfl_xor_sync(0xffffffffu, sm[m], 1);
    sm[m] += __shfl_xor_sync(0xffffffffu, sm[m], 2);
  }
  if (fk != 0) return;
  if constexpr (GRAD) {
    const long g = g0 + 8 * warp + fr;
    if (g >= npts) return;
    rho[g] = sm[0];
    if (grad) {
      grad[g] = 2 * sm[1];
      grad[npts + g] = 2 * sm[2];
      grad[2 * npts + g] = 2 * sm[3];
    }
    if (sigma) sigma[g] = 4.0 * (sm[1] * sm[1] + sm[2] * sm[2] + sm[3] * sm[3]);
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const long g = g0 + 32 * warp + 8 * m + fr;
      if (g < npts) rho[g] = sm[m];
    }
  }
}

template <bool GRAD, int NN, bool VEC>
static void launch_density_dense_nn(int nbf, long npts, const double *phi, const double *gx, const double *gy,
                                    const double *gz, int nocc, const double *C, const double *occ, double *rho,
                                    double *grad, double *sigma, cudaStream_t s) {
  NKX_CUDA(cudaFuncSetAttribute(density_dense_kernel<GRAD, NN, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kDdSmem<NN>));
  const int pts = GRAD ? 64 : 256;
  density_dense_kernel<GRAD, NN, VEC><<<(unsigned)((npts + pts - 1) / pts), 256, kDdSmem<NN>, s>>>(
      nbf, npts, phi, gx, gy, gz, nocc, C, occ, rho, grad, sigma);
}

// rho (and, with gx given, grad / sigma where not null) of one spin
static void launch_density_dense(int nbf, long npts, const double *phi, const double *gx, const double *gy,
                                 const double *gz, int nocc, const double *C, const double *occ, double *rho,
                                 double *grad, double *sigma, cudaStream_t s) {
  bool vec = nbf % 2 == 0;
  for (const double *q : {phi, gx, gy, gz, C}) vec = vec && ((uintptr_t)q & 15) == 0;
  auto go = [&](auto g, auto v) {
    constexpr bool G = decltype(g)::value, V = decltype(v)::value;
    auto f = nocc <= 8    ? launch_density_dense_nn<G, 1, V>
             : nocc <= 16 ? launch_density_dense_nn<G, 2, V>
             : nocc <= 32 ? launch_density_dense_nn<G, 4, V>
                          : launch_density_dense_nn<G, 8, V>;
    f(nbf, npts, phi, gx, gy, gz, nocc, C, occ, rho, grad, sigma, s);
  };
  if (gx)
    vec ? go(std::true_type{}, std::true_type{}) : go(std::true_type{}, std::false_type{});
  else
    vec ? go(std::false_type{}, std::true_type{}) : go(std::false_type{}, std::false_type{});
  NKX_LAUNCH_CHECK();
}

// libxc-layout functional evaluation (thread per point)
__global__ void xc_eval_kernel(XcSpec s, int nspin, long n, const double *rho, const double *sigma, double *exc,
                               double *vrho, double *vsigma) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= n) return;
  if (nspin == 1) {
    double f, vr, vs;
    const double r = rho[g];
    xc_unpol(s, r, sigma ? sigma[g] : 0.0, f, vr, vs);
    exc[g] = (r > 0 && f != 0.0) ? f / r : 0.0;
    vrho[g] = vr;
    if (vsigma) vsigma[g] = vs;
  } else {
    double f, d[5];
    const double ra = rho[2 * g], rb = rho[2 * g + 1];
    xc_pol(s, ra, rb, sigma ? sigma[3 * g] : 0.0, sigma ? sigma[3 * g + 1] : 0.0, sigma ? sigma[3 * g + 2] : 0.0,
           f, d);
    exc[g] = (ra + rb > 0 && f != 0.0) ? f / (ra + rb) : 0.0;
    vrho[2 * g] = d[0];
    vrho[2 * g + 1] = d[1];
    if (vsigma) {
      vsigma[3 * g] = d[2];
      vsigma[3 * g + 1] = d[3];
      vsigma[3 * g + 2] = d[4];
    }
  }
}

// Per point: functional of the (spin) densities, energy, and the coefficients
// of Z(mu, g) = w (1/2 phi vrho + vec . grad phi) (xc_integrals.hpp:486-515,
// :655-697), which take the place of rho (w vrho / 2) and grad rho (w vec).
__global__ void __launch_bounds__(128) xc_coef_dense_kernel(XcSpec s, bool gga, long npts, int nspin,
                                                            const double *__restrict__ w, double *rho, double *grad,
                                                            double *Eacc) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  double e = 0.0;
  if (g < npts) {
    double vr[2] = {0, 0}, vec[2][3] = {{0, 0, 0}, {0, 0, 0}};
    double gr[2][3] = {{0, 0, 0}, {0, 0, 0}};
    for (int sp = 0; sp < nspin; ++sp)
      if (gga)
        for (int k = 0; k < 3; ++k) gr[sp][k] = grad[(size_t)sp * 3 * npts + k * npts + g];
    if (nspin == 1) {
      const double r = rho[g];
      const double sg = gr[0][0] * gr[0][0] + gr[0][1] * gr[0][1] + gr[0][2] * gr[0][2];
      double f, vrho, vs;
      xc_unpol(s, r, sg, f, vrho, vs);
      e = w[g] * f;
      vr[0] = vrho;
      for (int k = 0; k < 3; ++k) vec[0][k] = 2.0 * vs * gr[0][k];
    } else {
      const double ra = rho[g], rb = rho[npts + g];
      const double saa = gr[0][0] * gr[0][0] + gr[0][1] * gr[0][1] + gr[0][2] * gr[0][2];
      const double sab = gr[0][0] * gr[1][0] + gr[0][1] * gr[1][1] + gr[0][2] * gr[1][2];
      const double sbb = gr[1][0] * gr[1][0] + gr[1][1] * gr[1][1] + gr[1][2] * gr[1][2];
      double f, d[5];
      xc_pol(s, ra, rb, saa, sab, sbb, f, d);
      e = w[g] * f;
      vr[0] = d[0];
      vr[1] = d[1];
      for (int k = 0; k < 3; ++k) {
        vec[0][k] = 2.0 * d[2] * gr[0][k] + d[3] * gr[1][k];
        vec[1][k] = 2.0 * d[4] * gr[1][k] + d[3] * gr[0][k];
      }
    }
    for (int sp = 0; sp < nspin; ++sp) {
      rho[(size_t)sp * npts + g] = 0.5 * w[g] * vr[sp];
      if (gga)
        for (int k = 0; k < 3; ++k) grad[(size_t)sp * 3 * npts + k * npts + g] = w[g] * vec[sp][k];
    }
  }
  for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(Eacc, e);
}

// Z holds nspin blocks of nbf x npts: block (x, spin) walks the rows of
// kZPts points with the functions contiguous.  Bound: HBM (one water: 164 us
// with a thread per point walking its row, 13 + 27 now).
constexpr int kZPts = 64;
template <bool GGA>
__global__ void __launch_bounds__(256) xc_z_dense_kernel(int nbf, long npts, const double *__restrict__ phi,
                                                         const double *__restrict__ gx, const double *__restrict__ gy,
                                                         const double *__restrict__ gz, const double *__restrict__ c0,
                                                         const double *__restrict__ ck, double *__restrict__ Z) {
  __shared__ double cf[GGA ? 4 : 1][kZPts];
  const long g0 = blockIdx.x * (long)kZPts;
  const int sp = blockIdx.y, np = (int)min((long)kZPts, npts - g0);
  for (int e = threadIdx.x; e < (GGA ? 4 : 1) * kZPts; e += 256) {
    const int k = e / kZPts, p = e % kZPts;
    if (p < np)
      cf[k][p] = k == 0 ? c0[(size_t)sp * npts + g0 + p] : ck[((size_t)sp * 3 + k - 1) * npts + g0 + p];
  }
  __syncthreads();
  const int n = np * nbf;
  const size_t base = (size_t)g0 * nbf;
  double *Zs = Z + (size_t)sp * nbf * npts;
#pragma unroll 4
  for (int t = threadIdx.x; t < n; t += 256) {
    const int p = t / nbf;
    double r = cf[0][p] * phi[base + t];
    if (GGA) r += cf[GGA ? 1 : 0][p] * gx[base + t] + cf[GGA ? 2 : 0][p] * gy[base + t] + cf[GGA ? 3 : 0][p] * gz[base + t];
    Zs[base + t] = r;
  }
}

// the functional and Z of the dense build, from rho and grad in place
static void launch_xc_z_dense(const XcSpec &sp, bool gga, int nbf, long npts, int nspin, const double *phi,
                              const double *gx, const double *gy, const double *gz, const double *w, double *rho,
                              double *grad, double *Z, double *E, cudaStream_t s) {
  xc_coef_dense_kernel<<<(unsigned)((npts + 127) / 128), 128, 0, s>>>(sp, gga, npts, nspin, w, rho, grad, E);
  auto *kernel = gga ? xc_z_dense_kernel<true> : xc_z_dense_kernel<false>;
  kernel<<<dim3((unsigned)((npts + kZPts - 1) / kZPts), nspin), 256, 0, s>>>(nbf, npts, phi, gx, gy, gz, rho, grad, Z);
  NKX_LAUNCH_CHECK();
}

// V += Vbar + Vbar^T with Vbar(i,j) = sum_g A(i,g) B(j,g); A, B column-major
// n x npts (xc_integrals.hpp:148-153 forms Vbar by DGEMM and then adds its
// transpose).  n is small (the basis) and npts large, so the point range is
// split over blockIdx.z: each block forms a 64 x 64 tile over its slice of
// points, eight warps of 32 x 16 on DMMA tiles, 32 points a step through a
// ring of shared stages (rows padded by four doubles), and adds it to V(i,j)
// and V(j,i) atomically.  V must be zero on entry.  VEC as in
// density_dense_kernel (one water: 50 us on CUDA-core tiles, 31 now).  With v, B(j,g) is taken times v(g) / 2 (J = Phi
// diag(v) Phi^T, whose Vbar is symmetric).
constexpr int kGemmTile = 64, kGemmK = 32, kGemmLd = kGemmTile + 4, kGemmStages = 3;
constexpr int kGemmStage = 2 * kGemmK * kGemmLd, kGemmSmem = kGemmStages * kGemmStage * 8;
template <bool VEC, bool SCALE>
__global__ void __launch_bounds__(256, 2) nt_gemm_sym_kernel(int n, long npts, long kslice, const double *__restrict__ A,
                                                             const double *__restrict__ B,
                                                             const double *__restrict__ v, double *V) {
  extern __shared__ __align__(16) double gsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fk = lane & 3;
  const int i0 = blockIdx.y * kGemmTile, j0 = blockIdx.x * kGemmTile;
  const long g_lo = blockIdx.z * kslice, g_hi = min(npts, g_lo + kslice);
  const int total = (int)((g_hi - g_lo + kGemmK - 1) / kGemmK);
  constexpr int W = VEC ? 2 : 1, PARTS = kGemmTile / W;
  auto issue = [&](int t, int st) {
    if (t < total) {
      double *As = gsm + st * kGemmStage, *Bs = As + kGemmK * kGemmLd;
#pragma unroll
      for (int r = 0; r < kGemmK * PARTS / 256; ++r) {
        const int e = threadIdx.x + 256 * r, k = e / PARTS, part = W * (e % PARTS);
        const long g = g_lo + (long)t * kGemmK + k;
        const bool ia = g < g_hi && i0 + part < n, ib = g < g_hi && j0 + part < n;
        const double *a = ia ? A + (size_t)g * n + i0 + part : A, *b = ib ? B + (size_t)g * n + j0 + part : B;
        if constexpr (VEC) {
          cp_async16_fill(As + k * kGemmLd + part, a, ia);
          cp_async16_fill(Bs + k * kGemmLd + part, b, ib);
        } else {
          cp_async8_fill(As + k * kGemmLd + part, a, ia);
          cp_async8_fill(Bs + k * kGemmLd + part, b, ib);
        }
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int st = 0; st < kGemmStages - 1; ++st) issue(st, st);
  double acc[4][2][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  const int r0 = 32 * (warp & 1) + fr, c0 = 16 * (warp >> 1) + fr;
  for (int t = 0; t < total; ++t) {
    cp_async_wait<kGemmStages - 2>();
    __syncthreads();  // step t is visible; the stage refilled below was read in step t - 1
    issue(t + kGemmStages - 1, (t + kGemmStages - 1) % kGemmStages);
    const double *As = gsm + (t % kGemmStages) * kGemmStage, *Bs = As + kGemmK * kGemmLd;
#pragma unroll
    for (int k = 0; k < kGemmK; k += 4) {
      double av[4], bv[2];
#pragma unroll
      for (int a = 0; a < 4; ++a) av[a] = As[(k + fk) * kGemmLd + r0 + 8 * a];
#pragma unroll
      for (int b = 0; b < 2; ++b) bv[b] = Bs[(k + fk) * kGemmLd + c0 + 8 * b];
      if constexpr (SCALE) {
        const double h = 0.5 * v[min(g_lo + (long)t * kGemmK + k + fk, npts - 1)];  // rows past g_hi are zero
#pragma unroll
        for (int b = 0; b < 2; ++b) bv[b] *= h;
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) dmma884(acc[a][b], av[a], bv[b]);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + r0 + 8 * a, j = j0 + 16 * (warp >> 1) + 8 * b + 2 * fk + h;
        if (i < n && j < n) {
          atomicAdd(&V[(size_t)i + (size_t)j * n], acc[a][b][h]);
          atomicAdd(&V[(size_t)j + (size_t)i * n], acc[a][b][h]);
        }
      }
}

// Launch of nt_gemm_sym_kernel for one n x n output (zeroed here): enough
// point slices to give every SM a couple of blocks.
static void launch_nt_gemm_sym(int n, long npts, const double *A, const double *B, double *V, cudaStream_t s,
                               const double *v = nullptr) {
  NKX_CUDA(cudaMemsetAsync(V, 0, sizeof(double) * n * n, s));
  const int nt = (n + kGemmTile - 1) / kGemmTile;
  const long want = std::max<long>(1, (2L * 148 + (long)nt * nt - 1) / ((long)nt * nt));
  const long nsl = std::max<long>(1, std::min<long>(want, (npts + 255) / 256));
  const long kslice = ((npts + nsl - 1) / nsl + kGemmK - 1) / kGemmK * kGemmK;
  const long nz = (npts + kslice - 1) / kslice;
  const bool vec = n % 2 == 0 && (((uintptr_t)A | (uintptr_t)B) & 15) == 0;
  auto *kernel = v ? (vec ? nt_gemm_sym_kernel<true, true> : nt_gemm_sym_kernel<false, true>)
                   : (vec ? nt_gemm_sym_kernel<true, false> : nt_gemm_sym_kernel<false, false>);
  NKX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
  kernel<<<dim3(nt, nt, (unsigned)nz), 256, kGemmSmem, s>>>(n, npts, kslice, A, B, v, V);
}

// The dense table Vw(a, g), functions a contiguous, one CTA per 128
// points and chunk of at most kDenseF functions.  A thread owns a point and
// walks every kDenseG-th run of the chunk's functions, so the basis data, the harmonic's branch and
// the loop bounds are the same for the whole warp, and the functions of a run
// (one centre, exponent, n and l) share the radial factor; the chunk leaves
// through a shared tile with the functions contiguous.
constexpr int kDenseP = 128, kDenseF = 16, kDenseG = 4, kDenseT = kDenseP * kDenseG;
struct DenseRun {
  int first, nm;  // functions [first, first + nm)
};
struct DenseChunk {
  int run0, run1, f0, nf;
};

// Runs of consecutive functions for which same(i, i + 1) holds (at most 15
// long), and chunks of whole runs
template <class Same>
static void dense_runs(int n, Same &&same, std::vector<DenseRun> &runs, std::vector<DenseChunk> &chunks) {
  for (int i = 0; i < n;) {
    int e = i + 1;
    while (e < n && e - i < 15 && same(e - 1, e)) ++e;
    if (chunks.empty() || chunks.back().nf + (e - i) > kDenseF)
      chunks.push_back(DenseChunk{(int)runs.size(), (int)runs.size(), i, 0});
    DenseChunk &c = chunks.back();
    runs.push_back(DenseRun{i, e - i});
    c.run1 = (int)runs.size();
    c.nf += e - i;
    i = e;
  }
}

// the chunk's runs and functions into shared memory
template <class F>
__device__ __forceinline__ void dense_load(const F *__restrict__ fn, const DenseRun *__restrict__ runs,
                                           const DenseChunk &ch, F *sfn, DenseRun *srun) {
  for (int e = threadIdx.x; e < ch.nf; e += kDenseT) sfn[e] = fn[ch.f0 + e];
  for (int e = threadIdx.x; e < ch.run1 - ch.run0; e += kDenseT) srun[e] = runs[ch.run0 + e];
  __syncthreads();
}

// one chunk's tile [f][point] to its place in the output
__device__ __forceinline__ void dense_store(const double *tile, int nf, int f0, int nfun, long g0, int np,
                                            double *__restrict__ out) {
  for (int e = threadIdx.x; e < np * nf; e += kDenseT) {
    const int pt = e / nf, f = e - pt * nf;
    out[(size_t)(g0 + pt) * nfun + f0 + f] = tile[f * (kDenseP + 1) + pt];
  }
}

// Vw(a, g) = V_a(r_g) w_g.  Bound: FP64 issue of the incomplete gamma functions,
// evaluated once per run and point (one water, 143 functions, 68k points:
// 311 us with a thread per element, 111 us now).
__global__ void __launch_bounds__(kDenseT) potential_dense_kernel(const AuxFunc *__restrict__ fn,
                                                                  const DenseRun *__restrict__ runs,
                                                                  const DenseChunk *__restrict__ chunks, int naux,
                                                                  const double *__restrict__ pts,
                                                                  const double *__restrict__ w, long npts,
                                                                  double *__restrict__ Vw) {
  extern __shared__ double dtile[];  // [kDenseF][kDenseP + 1]
  __shared__ AuxFunc sfn[kDenseF];
  __shared__ DenseRun srun[kDenseF];
  const DenseChunk ch = chunks[blockIdx.y];
  const long g0 = blockIdx.x * (long)kDenseP, g = min(g0 + threadIdx.x % kDenseP, npts - 1);
  const int np = (int)min((long)kDenseP, npts - g0);
  const double px = pts[3 * g], py = pts[3 * g + 1], pz = pts[3 * g + 2], wg = w[g];
  dense_load(fn, runs, ch, sfn, srun);
  for (int r = threadIdx.x / kDenseP; r < ch.run1 - ch.run0; r += kDenseG) {
    const int k0 = srun[r].first - ch.f0, nm = srun[r].nm;
    const AuxFunc &f = sfn[k0];
    const double dx = px - f.cx, dy = py - f.cy, dz = pz - f.cz;
    const double R = aux_radial(f, sqrt(dx * dx + dy * dy + dz * dz));
#pragma unroll 1
    for (int k = k0; k < k0 + nm; ++k) {
      double x = dx, y = dy, z = dz;
      opaque(x, y, z);
      dtile[k * (kDenseP + 1) + threadIdx.x % kDenseP] = f.C * solid_harmonic(f.l, sfn[k].m, x, y, z) * R * wg;
    }
  }
  __syncthreads();
  dense_store(dtile, ch.nf, ch.f0, naux, g0, np, Vw);
}

__global__ void precondition_kernel(int N, const double *S, double *A, double *D) {
  const int i = blockIdx.y * blockDim.y + threadIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N && j < N) A[(size_t)i + (size_t)j * N] = S[(size_t)i + (size_t)j * N] /
                                                      sqrt(S[(size_t)i + (size_t)i * N] * S[(size_t)j + (size_t)j * N]);
  if (j == 0 && i < N) D[i] = sqrt(S[(size_t)i + (size_t)i * N]);
}

XcSpec make_spec(const nkx_plan_options *o) {
  XcSpec s;
  NKX_REQUIRE(o && o->nfunc >= 1 && o->nfunc <= 4, NKX_ERR_ARG, "opts.nfunc must be 1..4");
  s.nfunc = o->nfunc;
  for (int i = 0; i < 4; ++i) s.ids[i] = i < o->nfunc ? o->func_ids[i] : 0;
  for (int i = 0; i < o->nfunc; ++i)
    NKX_REQUIRE(func_supported(o->func_ids[i]), NKX_ERR_UNSUPPORTED, "unsupported functional id");
  s.thr = o->dens_threshold > 0 ? o->dens_threshold : 1e-15;
  return s;
}

bool spec_is_gga(const XcSpec &s) {
  for (int i = 0; i < s.nfunc; ++i)
    if (func_is_gga(s.ids[i])) return true;
  return false;
}

}  // namespace nkx

using namespace nkx;

static unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

// the runs and chunks of an aux function table, on the device
struct DenseTable {
  std::vector<DenseChunk> hchunks;  // filled while hruns is made
  std::vector<DenseRun> hruns;
  int nchunk;
  DevBuf<DenseRun> runs;
  DevBuf<DenseChunk> chunks;
  static std::vector<DenseRun> split(const std::vector<AuxFunc> &t, std::vector<DenseChunk> &c) {
    std::vector<DenseRun> r;
    dense_runs((int)t.size(), [&](int i, int j) {
      const AuxFunc &x = t[i], &y = t[j];
      return x.cx == y.cx && x.cy == y.cy && x.cz == y.cz && x.zeta == y.zeta && x.l == y.l && x.a == y.a;
    }, r, c);
    return r;
  }
  DenseTable(const std::vector<AuxFunc> &t, cudaStream_t s)
      : hruns(split(t, hchunks)), nchunk((int)hchunks.size()), runs(hruns.size(), s), chunks(hchunks.size(), s) {
    NKX_CUDA(cudaMemcpyAsync(runs.p, hruns.data(), sizeof(DenseRun) * hruns.size(), cudaMemcpyHostToDevice, s));
    NKX_CUDA(cudaMemcpyAsync(chunks.p, hchunks.data(), sizeof(DenseChunk) * hchunks.size(), cudaMemcpyHostToDevice, s));
  }
};

extern "C" nkx_status nkx_fill_collocation(const nkx_basis *basis, const double *d_points, long npts, double *d_phi,
                                           double *d_gx, double *d_gy, double *d_gz, void *stream) {
  return run_guarded("nkx_fill_collocation", [&] {
    NKX_REQUIRE(basis && basis->nbf > 0 && npts >= 0 && d_points && d_phi, NKX_ERR_ARG, "invalid arguments");
    NKX_REQUIRE(!d_gx || (d_gy && d_gz), NKX_ERR_ARG, "gradient buffers must be given together");
    for (int i = 0; i < basis->nbf; ++i)
      NKX_REQUIRE(basis->l[i] >= 0 && basis->l[i] <= 7 && basis->n[i] > basis->l[i] &&
                      abs(basis->m[i]) <= basis->l[i] && basis->zeta[i] > 0,
                  NKX_ERR_UNSUPPORTED, "basis function outside n > l, |m| <= l <= 7, zeta > 0");
    auto tab = make_sto_table(*basis);
    cudaStream_t s = (cudaStream_t)stream;
    DevBuf<StoFunc> df(tab.size(), s);
    NKX_CUDA(cudaMemcpyAsync(df.p, tab.data(), tab.size() * sizeof(StoFunc), cudaMemcpyHostToDevice, s));
    const long tot = (long)basis->nbf * npts;
    if (tot > 0) colloc_dense_kernel<<<nblk(tot, 128), 128, 0, s>>>(df.p, basis->nbf, d_points, npts, d_phi, d_gx, d_gy, d_gz);
    NKX_LAUNCH_CHECK();
    NKX_CUDA(cudaStreamSynchronize(s));
  });
}

extern "C" nkx_status nkx_density_dense(int nbf, long npts, const double *d_phi, const double *d_gx,
                                        const double *d_gy, const double *d_gz, int nocc, const double *d_C,
                                        const double *d_occ, double *d_rho, double *d_grad, double *d_sigma,
                                        void *stream) {
  return run_guarded("nkx_density_dense", [&] {
    NKX_REQUIRE(nbf > 0 && npts >= 0 && nocc > 0 && d_phi && d_C && d_occ && d_rho, NKX_ERR_ARG,
                "invalid arguments");
    NKX_REQUIRE(!(d_grad || d_sigma) || (d_gx && d_gy && d_gz), NKX_ERR_ARG, "gradient output needs grad inputs");
    cudaStream_t s = (cudaStream_t)stream;
    if (npts > 0)
      launch_density_dense(nbf, npts, d_phi, (d_grad || d_sigma) ? d_gx : nullptr, d_gy, d_gz, nocc, d_C, d_occ, d_rho,
                           d_grad, d_sigma, s);
    NKX_CUDA(cudaStreamSynchronize(s));
  });
}

extern "C" nkx_status nkx_xc_eval(int func_id, int nspin, long n, const double *d_rho, const double *d_sigma,
                                  double dens_threshold, double *d_exc, double *d_vrho, double *d_vsigma,
                                  void *stream) {
  return run_guarded("nkx_xc_eval", [&] {
    NKX_REQUIRE((nspin == 1 || nspin == 2) && n >= 0 && d_rho && d_exc && d_vrho, NKX_ERR_ARG, "invalid arguments");
    NKX_REQUIRE(func_supported(func_id), NKX_ERR_UNSUPPORTED, "unsupported functional id");
    NKX_REQUIRE(!func_is_gga(func_id) || (d_sigma && d_vsigma), NKX_ERR_ARG, "GGA needs sigma and vsigma");
    XcSpec sp;
    sp.nfunc = 1;
    sp.ids[0] = func_id;
    sp.ids[1] = sp.ids[2] = sp.ids[3] = 0;
    sp.thr = dens_threshold > 0 ? dens_threshold : 1e-15;
    cudaStream_t s = (cudaStream_t)stream;
    if (n > 0) xc_eval_kernel<<<nblk(n, 128), 128, 0, s>>>(sp, nspin, n, d_rho, d_sigma, d_exc, d_vrho, d_vsigma);
    NKX_LAUNCH_CHECK();
    NKX_CUDA(cudaStreamSynchronize(s));
  });
}

extern "C" nkx_status nkx_xc_dense(int nbf, long npts, const double *d_phi, const double *d_gx, const double *d_gy,
                                   const double *d_gz, const double *d_w, int nspin, int nocc, const double *d_C,
                                   const double *d_occ, const nkx_plan_options *opts, double *E, double *d_V,
                                   void *stream) {
  return run_guarded("nkx_xc_dense", [&] {
    NKX_REQUIRE(nbf > 0 && npts > 0 && (nspin == 1 || nspin == 2) && nocc > 0 && d_phi && d_w && d_C && d_occ &&
                    E && d_V,
                NKX_ERR_ARG, "invalid arguments");
    const XcSpec sp = make_spec(opts);
    const bool gga = spec_is_gga(sp);
    NKX_REQUIRE(!gga || (d_gx && d_gy && d_gz), NKX_ERR_ARG, "GGA needs collocation gradients");
    cudaStream_t s = (cudaStream_t)stream;
    run_and_wait(s, [&] {
      const Source ws(s, sizeof(double) * nspin * npts * (nbf + (size_t)4));
      DevBuf<double> rho((size_t)nspin * npts, ws), grad((size_t)nspin * 3 * npts, ws),
          Z((size_t)nspin * nbf * npts, ws), Ed(1, ws);
      for (int sp_i = 0; sp_i < nspin; ++sp_i)
        launch_density_dense(nbf, npts, d_phi, gga ? d_gx : nullptr, d_gy, d_gz, nocc, d_C + (size_t)sp_i * nbf * nocc,
                             d_occ + (size_t)sp_i * nocc, rho.p + (size_t)sp_i * npts,
                             gga ? grad.p + (size_t)sp_i * 3 * npts : nullptr, nullptr, s);
      NKX_CUDA(cudaMemsetAsync(Ed.p, 0, sizeof(double), s));
      launch_xc_z_dense(sp, gga, nbf, npts, nspin, d_phi, d_gx, d_gy, d_gz, d_w, rho.p, grad.p, Z.p, Ed.p, s);
      for (int sp_i = 0; sp_i < nspin; ++sp_i)
        launch_nt_gemm_sym(nbf, npts, d_phi, Z.p + (size_t)sp_i * nbf * npts, d_V + (size_t)sp_i * nbf * nbf, s);
      NKX_LAUNCH_CHECK();
      NKX_CUDA(cudaMemcpyAsync(E, Ed.p, sizeof(double), cudaMemcpyDeviceToHost, s));
    });
  });
}

extern "C" nkx_status nkx_potential_collocation(const nkx_basis *aux, const double *d_points, const double *d_w,
                                                long npts, double *d_Vw, void *stream) {
  return run_guarded("nkx_potential_collocation", [&] {
    NKX_REQUIRE(aux && aux->nbf > 0 && npts >= 0 && d_points && d_w && d_Vw, NKX_ERR_ARG, "invalid arguments");
    auto tab = make_aux_table(*aux);
    cudaStream_t s = (cudaStream_t)stream;
    DevBuf<AuxFunc> df(tab.size(), s);
    NKX_CUDA(cudaMemcpyAsync(df.p, tab.data(), tab.size() * sizeof(AuxFunc), cudaMemcpyHostToDevice, s));
    const DenseTable dt(tab, s);
    if (npts > 0)
      potential_dense_kernel<<<dim3(nblk(npts, kDenseP), dt.nchunk), kDenseT, kDenseF * (kDenseP + 1) * 8, s>>>(
          df.p, dt.runs.p, dt.chunks.p, aux->nbf, d_points, d_w, npts, d_Vw);
    NKX_LAUNCH_CHECK();
    NKX_CUDA(cudaStreamSynchronize(s));
  });
}

// S(f, g) = Phi(f, g) v(g)
__global__ void scale_columns_kernel(int nbf, long npts, const double *__restrict__ phi, const double *__restrict__ v,
                                     double *__restrict__ S) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e < (long)nbf * npts) S[e] = phi[e] * v[e / nbf];
}

// part[slice][a] = sum over a slice of points of Vw(a, g) rho(g): warp w of a
// block takes points w, w + 8, .. of the slice, lane l function a0 + l
// (coulomb.hpp:84-85).  Bound: Vw from HBM (78 MB in 20 us).
__global__ void __launch_bounds__(256) vw_rho_kernel(int naux, long npts, long slice, const double *__restrict__ Vw,
                                                     const double *__restrict__ rho, double *__restrict__ part) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, a = blockIdx.x * 32 + lane;
  const long g1 = min(npts, (blockIdx.y + 1) * slice);
  double s = 0.0;
  if (a < naux) {
#pragma unroll 8
    for (long g = blockIdx.y * slice + warp; g < g1; g += 8) s += Vw[(size_t)g * naux + a] * rho[g];
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && a < naux) {
#pragma unroll
    for (int w = 1; w < 8; ++w) s += red[w][lane];
    part[(size_t)blockIdx.y * naux + a] = s;
  }
}
// out(a) = sum_k M(a, k) x(k) over the n columns of M (m x n, column-major;
// x == nullptr: ones), a warp per row: y from its slices' shares, c = X t
__global__ void __launch_bounds__(256) rows_dot_kernel(int m, int n, const double *__restrict__ M,
                                                       const double *__restrict__ x, double *__restrict__ out) {
  const int a = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (a >= m) return;
  double s = 0.0;
#pragma unroll 4
  for (int k = lane; k < n; k += 32) s += M[(size_t)k * m + a] * (x ? x[k] : 1.0);
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[a] = s;
}
// out(j) = sum_a M(a, j) x(a) for the n columns of M (m x n, column-major),
// a warp per column: t = X^T y, and v = Vw^T c with one column per point
// (coulomb.hpp:86-95)
__global__ void __launch_bounds__(256) columns_dot_kernel(int m, long n, const double *__restrict__ M,
                                                          const double *__restrict__ x, double *__restrict__ out) {
  const long j = (blockIdx.x * 256L + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= n) return;
  double s = 0.0;
#pragma unroll 4
  for (int a = lane; a < m; a += 32) s += M[(size_t)j * m + a] * x[a];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[j] = s;
}

extern "C" nkx_status nkx_coulomb_dense(int nbf, int naux, long npts, const double *d_phi, const double *d_Vw,
                                        const double *d_X, int K, int nocc, const double *d_C, const double *d_occ,
                                        double *d_J, void *stream) {
  return run_guarded("nkx_coulomb_dense", [&] {
    NKX_REQUIRE(nbf > 0 && naux > 0 && npts > 0 && K > 0 && K <= naux && nocc > 0 && d_phi && d_Vw && d_X && d_C &&
                    d_occ && d_J,
                NKX_ERR_ARG, "invalid arguments");
    cudaStream_t s = (cudaStream_t)stream;
    // about eight blocks an SM over (32-function tiles) x (slices of 128 points and more)
    const long na = (naux + 31) / 32, nsl = std::max<long>(1, std::min<long>((8 * 148 + na - 1) / na, npts / 128));
    const long slice = (npts + nsl - 1) / nsl;
    run_and_wait(s, [&] {
      const Source ws(s, sizeof(double) * (2 * (size_t)npts + (size_t)nsl * naux));
      DevBuf<double> rho(npts, ws), y(naux, ws), t(K, ws), c(naux, ws), v(npts, ws), part((size_t)nsl * naux, ws);
      launch_density_dense(nbf, npts, d_phi, nullptr, nullptr, nullptr, nocc, d_C, d_occ, rho.p, nullptr, nullptr, s);
      vw_rho_kernel<<<dim3((unsigned)na, (unsigned)nsl), 256, 0, s>>>(naux, npts, slice, d_Vw, rho.p, part.p);
      rows_dot_kernel<<<nblk(naux * 32L, 256), 256, 0, s>>>(naux, (int)nsl, part.p, nullptr, y.p);
      columns_dot_kernel<<<nblk(K * 32L, 256), 256, 0, s>>>(naux, K, d_X, y.p, t.p);
      rows_dot_kernel<<<nblk(naux * 32L, 256), 256, 0, s>>>(naux, K, d_X, t.p, c.p);
      columns_dot_kernel<<<nblk(npts * 32, 256), 256, 0, s>>>(naux, npts, d_Vw, c.p, v.p);
      NKX_LAUNCH_CHECK();
      launch_nt_gemm_sym(nbf, npts, d_phi, d_phi, d_J, s, v.p);
      NKX_LAUNCH_CHECK();
    });
  });
}

// compute_exact_exchange (nukexc/exact_exchange.hpp:57-119), the reference's
// dense grid RI-K: T = Phi^T C (npts x nocc), then per orbital i
//   B = Phi o T_i (columns scaled), (P|mu i) = Vw B^T (naux x nbf),
//   Y = (P|mu i)^T X (nbf x K),  K += occ_i Y Y^T,
// FP64 cuBLAS GEMMs.  The work is nocc * naux * nbf * npts: small systems.
extern "C" nkx_status nkx_exchange_dense(int nbf, int naux, long npts, const double *d_phi, const double *d_Vw,
                                         const double *d_X, int K, int nocc, const double *d_C, const double *d_occ,
                                         double *d_K, void *stream) {
  return run_guarded("nkx_exchange_dense", [&] {
    NKX_REQUIRE(nbf > 0 && naux > 0 && npts > 0 && K > 0 && K <= naux && nocc > 0 && d_phi && d_Vw && d_X && d_C &&
                    d_occ && d_K,
                NKX_ERR_ARG, "invalid arguments");
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<double> occ(nocc);
    NKX_CUDA(cudaMemcpyAsync(occ.data(), d_occ, sizeof(double) * nocc, cudaMemcpyDeviceToHost, s));
    NKX_CUDA(cudaStreamSynchronize(s));
    cublasHandle_t h = nullptr;
    bool ok = true;
    run_and_wait(s, [&] {
      const Source ws(s, sizeof(double) * ((size_t)npts * (nocc + nbf) + (size_t)nbf * (naux + K)));
      DevBuf<double> T((size_t)npts * nocc, ws), B((size_t)nbf * npts, ws), P3((size_t)naux * nbf, ws),
          Y((size_t)nbf * K, ws);
      NKX_REQUIRE(cublasCreate(&h) == CUBLAS_STATUS_SUCCESS, NKX_ERR_CUDA, "cublasCreate failed");
      cublasSetStream(h, s);
      const double one = 1.0, zero = 0.0;
      ok = cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, (int)npts, nocc, nbf, &one, d_phi, nbf, d_C, nbf, &zero, T.p,
                       (int)npts) == CUBLAS_STATUS_SUCCESS;
      ok = ok && cudaMemsetAsync(d_K, 0, sizeof(double) * nbf * nbf, s) == cudaSuccess;
      for (int i = 0; i < nocc && ok; ++i) {
        scale_columns_kernel<<<nblk((long)nbf * npts, 256), 256, 0, s>>>(nbf, npts, d_phi, T.p + (size_t)i * npts,
                                                                          B.p);
        ok = cudaGetLastError() == cudaSuccess;
        ok = ok && cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, naux, nbf, (int)npts, &one, d_Vw, naux, B.p, nbf, &zero,
                               P3.p, naux) == CUBLAS_STATUS_SUCCESS;
        ok = ok && cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, nbf, K, naux, &one, P3.p, naux, d_X, naux, &zero, Y.p,
                               nbf) == CUBLAS_STATUS_SUCCESS;
        const double oi = occ[i];
        ok = ok && cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, nbf, nbf, K, &oi, Y.p, nbf, Y.p, nbf, &one, d_K, nbf) ==
                       CUBLAS_STATUS_SUCCESS;
      }
    });
    cublasDestroy(h);
    NKX_REQUIRE(ok, NKX_ERR_CUDA, "cuBLAS call in nkx_exchange_dense failed");
  });
}

// per chunk point g: ws[g] = w_g, wv[g] = w_g sum_A Z_A / (|r_g - R_A| + 1e-30)
// (core_hamiltonian.hpp:226-236)
__global__ void core_weights_kernel(const double *__restrict__ pts, const double *__restrict__ w, long n,
                                    const double *__restrict__ centers, const double *__restrict__ Zc, int natoms,
                                    double *__restrict__ wv) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= n) return;
  double v = 0.0;
  for (int a = 0; a < natoms; ++a) {
    const double dx = pts[3 * g] - centers[3 * a], dy = pts[3 * g + 1] - centers[3 * a + 1],
                 dz = pts[3 * g + 2] - centers[3 * a + 2];
    v += Zc[a] / (sqrt(dx * dx + dy * dy + dz * dz) + 1e-30);
  }
  wv[g] = w[g] * v;
}
// out(mu, g) = in(mu, g) * s[g]
__global__ void scale_cols_kernel(int nbf, long n, const double *__restrict__ in, const double *__restrict__ s,
                                  double *__restrict__ out) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e < (long)nbf * n) out[e] = in[e] * s[e / nbf];
}

extern "C" nkx_status nkx_core_hamiltonian_dense(const nkx_basis *basis, const nkx_molecule *mol,
                                                 const double *d_points, const double *d_w, long npts, double *d_S,
                                                 double *d_T, double *d_V, void *stream) {
  return run_guarded("nkx_core_hamiltonian_dense", [&] {
    NKX_REQUIRE(basis && basis->nbf > 0 && mol && mol->natoms > 0 && d_points && d_w && npts > 0 && d_S && d_T && d_V,
                NKX_ERR_ARG, "invalid arguments");
    cudaStream_t s = (cudaStream_t)stream;
    const int nbf = basis->nbf;
    auto tab = make_sto_table(*basis);
    std::vector<double> zc(mol->natoms);
    for (int a = 0; a < mol->natoms; ++a) zc[a] = mol->Z[a];
    cublasHandle_t h = nullptr;
    bool ok = true;
    run_and_wait(s, [&] {
      DevBuf<StoFunc> df(tab.size(), s);
      NKX_CUDA(cudaMemcpyAsync(df.p, tab.data(), sizeof(StoFunc) * tab.size(), cudaMemcpyHostToDevice, s));
      DevBuf<double> dc(3 * (size_t)mol->natoms, s), dz(mol->natoms, s);
      NKX_CUDA(cudaMemcpyAsync(dc.p, mol->xyz, sizeof(double) * 3 * mol->natoms, cudaMemcpyHostToDevice, s));
      NKX_CUDA(cudaMemcpyAsync(dz.p, zc.data(), sizeof(double) * mol->natoms, cudaMemcpyHostToDevice, s));
      // points in chunks holding 6 nbf x chunk matrices in about 1 GiB
      const long chunk = std::max<long>(256, std::min<long>(npts, ((long)1 << 27) / (6L * nbf)));
      const Source ws(s, sizeof(double) * (5 * (size_t)nbf * chunk + chunk));
      DevBuf<double> phi((size_t)nbf * chunk, ws), gx((size_t)nbf * chunk, ws), gy((size_t)nbf * chunk, ws),
          gz((size_t)nbf * chunk, ws), sc((size_t)nbf * chunk, ws), wv(chunk, ws);
      NKX_CUDA(cudaMemsetAsync(d_S, 0, sizeof(double) * nbf * nbf, s));
      NKX_CUDA(cudaMemsetAsync(d_T, 0, sizeof(double) * nbf * nbf, s));
      NKX_CUDA(cudaMemsetAsync(d_V, 0, sizeof(double) * nbf * nbf, s));
      NKX_REQUIRE(cublasCreate(&h) == CUBLAS_STATUS_SUCCESS, NKX_ERR_CUDA, "cublasCreate failed");
      cublasSetStream(h, s);
      const double one = 1.0, half = 0.5, mone = -1.0;
      for (long g0 = 0; g0 < npts && ok; g0 += chunk) {
        const long n = std::min(chunk, npts - g0);
        const long tot = (long)nbf * n;
        colloc_dense_kernel<<<nblk(tot, 128), 128, 0, s>>>(df.p, nbf, d_points + 3 * g0, n, phi.p, gx.p, gy.p, gz.p);
        core_weights_kernel<<<nblk(n, 128), 128, 0, s>>>(d_points + 3 * g0, d_w + g0, n, dc.p, dz.p, mol->natoms, wv.p);
        // S += phi (w phi)^T
        scale_cols_kernel<<<nblk(tot, 256), 256, 0, s>>>(nbf, n, phi.p, d_w + g0, sc.p);
        ok = ok && cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, nbf, nbf, (int)n, &one, phi.p, nbf, sc.p, nbf, &one, d_S,
                               nbf) == CUBLAS_STATUS_SUCCESS;
        // V -= phi (w v phi)^T
        scale_cols_kernel<<<nblk(tot, 256), 256, 0, s>>>(nbf, n, phi.p, wv.p, sc.p);
        ok = ok && cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, nbf, nbf, (int)n, &mone, phi.p, nbf, sc.p, nbf, &one, d_V,
                               nbf) == CUBLAS_STATUS_SUCCESS;
        // T += 1/2 sum_k g_k (w g_k)^T
        for (double *gk : {gx.p, gy.p, gz.p}) {
          scale_cols_kernel<<<nblk(tot, 256), 256, 0, s>>>(nbf, n, gk, d_w + g0, sc.p);
          ok = ok && cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, nbf, nbf, (int)n, &half, gk, nbf, sc.p, nbf, &one, d_T,
                                 nbf) == CUBLAS_STATUS_SUCCESS;
        }
        ok = ok && cudaGetLastError() == cudaSuccess;
      }
    });
    cublasDestroy(h);
    NKX_REQUIRE(ok, NKX_ERR_CUDA, "kernel or cuBLAS failure in nkx_core_hamiltonian_dense");
  });
}

extern "C" nkx_status nkx_half_inverse(int N, const double *d_S, double thr, double *d_X, int *K, void *stream) {
  return run_guarded("nkx_half_inverse", [&] {
    NKX_REQUIRE(N > 0 && d_S && d_X && K, NKX_ERR_ARG, "invalid arguments");
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<double> hl(N), hU((size_t)N * N), hD(N);
    run_and_wait(s, [&] {
      const Source ws(s, sizeof(double) * 4 * (size_t)N * N);  // the solver's own is about 2 N^2
      DevBuf<double> A((size_t)N * N, ws), D(N, ws), lam(N, ws);
      DevBuf<int> info(1, s);
      dim3 tb(16, 16), gb(nblk(N, 16), nblk(N, 16));
      precondition_kernel<<<gb, tb, 0, s>>>(N, d_S, A.p, D.p);
      NKX_LAUNCH_CHECK();
      cusolverDnHandle_t h;
      NKX_REQUIRE(cusolverDnCreate(&h) == CUSOLVER_STATUS_SUCCESS, NKX_ERR_CUDA, "cusolverDnCreate failed");
      cusolverDnSetStream(h, s);
      int lwork = 0;
      cusolverDnDsyevd_bufferSize(h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, N, A.p, N, lam.p, &lwork);
      DevBuf<double> work(lwork > 0 ? lwork : 1, ws);
      const cusolverStatus_t st = cusolverDnDsyevd(h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, N, A.p, N,
                                                   lam.p, work.p, lwork, info.p);
      cusolverDnDestroy(h);
      NKX_REQUIRE(st == CUSOLVER_STATUS_SUCCESS, NKX_ERR_CUDA, "cusolverDnDsyevd failed");
      NKX_CUDA(cudaMemcpyAsync(hl.data(), lam.p, sizeof(double) * N, cudaMemcpyDeviceToHost, s));
      NKX_CUDA(cudaMemcpyAsync(hU.data(), A.p, sizeof(double) * N * N, cudaMemcpyDeviceToHost, s));
      NKX_CUDA(cudaMemcpyAsync(hD.data(), D.p, sizeof(double) * N, cudaMemcpyDeviceToHost, s));
    });
    // singular values of a symmetric matrix are |eigenvalues|; keep s > thr,
    // largest first (the reference's SVD ordering)
    std::vector<int> order(N);
    for (int i = 0; i < N; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return fabs(hl[a]) > fabs(hl[b]); });
    std::vector<double> hX((size_t)N * N, 0.0);
    int k = 0;
    for (int oi = 0; oi < N; ++oi) {
      const int e = order[oi];
      const double sv = fabs(hl[e]);
      if (!(sv > thr)) continue;
      for (int i = 0; i < N; ++i) hX[(size_t)i + (size_t)k * N] = hU[(size_t)i + (size_t)e * N] / sqrt(sv) / hD[i];
      ++k;
    }
    NKX_CUDA(cudaMemcpyAsync(d_X, hX.data(), sizeof(double) * N * N, cudaMemcpyHostToDevice, s));
    NKX_CUDA(cudaStreamSynchronize(s));
    *K = k;
  });
}

// ---------------------------------------------------------------------------
// nkx_xc_dense_noalloc: the dense XC build of nkx_xc_dense for callers that
// must not allocate device memory.  Some host programs hand (almost) all of
// the GPU's memory to their own pool allocator when they start, so a
// cudaMalloc from a library would fail or fragment that pool; others run the
// Fock build inside a latency-critical loop where cudaMalloc / cudaFree,
// which synchronise the whole device, are not acceptable.  This entry point
// keeps its scratch (energy accumulator, per-point density and gradient, the
// Z matrix) in one file-scope __device__ array of kNoAllocScratchDoubles
// doubles (32 MiB), which every GPU that loads the library holds until the
// process exits, and it calls no cudaMalloc, cudaFree or allocating library
// routine.
//
// In host code the array's name is only a host-side stand-in, never a device
// address, so the first call made on a device (with that device current)
// looks the address up with cudaGetSymbolAddress and remembers it for that
// device; that first call should come before any stream capture.  The
// remembered address belongs to the device's current context: the library
// must not be used across a cudaDeviceReset.  Every call shares the array and
// finds the previous call's contents there, so everything that must start at
// zero is cleared by the call itself; calls whose work overlaps on the GPU
// (other streams, other host threads) race on the array and must be
// serialised by the caller.  Problems that need more scratch than the array
// holds are rejected with NKX_ERR_ARG before anything is launched.
// ---------------------------------------------------------------------------
#include <mutex>

namespace nkx {

constexpr size_t kNoAllocScratchDoubles = (size_t)4 << 20;
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

static double *noalloc_scratch_address() {
  static std::mutex mu;
  static double *addr[128] = {nullptr};
  int dev = 0;
  NKX_CUDA(cudaGetDevice(&dev));
  NKX_REQUIRE(dev >= 0 && dev < 128, NKX_ERR_ARG, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void *p = nullptr;
    NKX_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    addr[dev] = static_cast<double *>(p);
  }
  return addr[dev];
}

}  // namespace nkx

extern "C" nkx_status nkx_xc_dense_noalloc(int nbf, long npts, const double *d_phi, const double *d_gx,
                                           const double *d_gy, const double *d_gz, const double *d_w, int nspin,
                                           int nocc, const double *d_C, const double *d_occ,
                                           const nkx_plan_options *opts, double *E, double *d_V, void *stream) {
  return run_guarded("nkx_xc_dense_noalloc", [&] {
    NKX_REQUIRE(nbf > 0 && npts > 0 && (nspin == 1 || nspin == 2) && nocc > 0 && d_phi && d_w && d_C && d_occ &&
                    E && d_V,
                NKX_ERR_ARG, "invalid arguments");
    const XcSpec sp = make_spec(opts);
    const bool gga = spec_is_gga(sp);
    NKX_REQUIRE(!gga || (d_gx && d_gy && d_gz), NKX_ERR_ARG, "GGA needs collocation gradients");
    // layout in doubles, each piece 256-byte aligned: E | rho | grad | Z.
    // npts is bounded first, so the products below cannot wrap around.
    const size_t per_point = (size_t)nspin * ((size_t)nbf + 4);
    const std::string too_large =
        "problem too large for the fixed 32 MiB scratch: needs about nspin*npts*(nbf+4) doubles <= 4194304";
    NKX_REQUIRE((size_t)npts <= kNoAllocScratchDoubles / per_point, NKX_ERR_ARG,
                too_large + " (nspin " + std::to_string(nspin) + ", npts " + std::to_string(npts) + ", nbf " +
                    std::to_string(nbf) + ")");
    auto up = [](size_t n) { return (n + 31) & ~(size_t)31; };
    const size_t nE = 32, nrho = up((size_t)nspin * npts), ngrad = up((size_t)nspin * 3 * npts);
    const size_t nZ = up((size_t)nspin * nbf * npts);
    const size_t need = nE + nrho + ngrad + nZ;
    NKX_REQUIRE(need <= kNoAllocScratchDoubles, NKX_ERR_ARG, too_large + " (" + std::to_string(need) + " requested)");
    double *base = noalloc_scratch_address();
    double *Ed = base, *rho = base + nE, *grad = rho + nrho, *Z = grad + ngrad;
    cudaStream_t s = (cudaStream_t)stream;
    for (int sp_i = 0; sp_i < nspin; ++sp_i)
      launch_density_dense(nbf, npts, d_phi, gga ? d_gx : nullptr, d_gy, d_gz, nocc, d_C + (size_t)sp_i * nbf * nocc,
                           d_occ + (size_t)sp_i * nocc, rho + (size_t)sp_i * npts,
                           gga ? grad + (size_t)sp_i * 3 * npts : nullptr, nullptr, s);
    NKX_CUDA(cudaMemsetAsync(Ed, 0, sizeof(double), s));  // the array keeps the previous call's sum
    launch_xc_z_dense(sp, gga, nbf, npts, nspin, d_phi, d_gx, d_gy, d_gz, d_w, rho, grad, Z, Ed, s);
    for (int sp_i = 0; sp_i < nspin; ++sp_i)
      launch_nt_gemm_sym(nbf, npts, d_phi, Z + (size_t)sp_i * nbf * npts, d_V + (size_t)sp_i * nbf * nbf, s);
    NKX_LAUNCH_CHECK();
    NKX_CUDA(cudaMemcpyAsync(E, Ed, sizeof(double), cudaMemcpyDeviceToHost, s));
    NKX_CUDA(cudaStreamSynchronize(s));
  });
}
