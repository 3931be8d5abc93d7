// XC nuclear gradient at fixed orbitals (FP64).  No counterpart in the
// reference; it differentiates exactly what nkx_fock_build integrates:
//
//   E_xc(R) = sum_g w_g(R) f(rho(r_g), grad rho(r_g)),
//   r_g = R_owner(g) + fixed offset,   w_g = a_g P_owner(r_g) / sum_i P_i(r_g)
//
// (grid points move with their owner atom; a_g, the radial x angular weight,
// does not depend on the geometry; P_i are Becke cell functions with the
// Laqua clamp R_ij = min(|R_i - R_j|, clamp), partitioning.hpp:126-213).
//
// dE/dR_A = sum_g w_g sum_s sum_mu t_(s,mu,g) (delta_(owner(g),A) - delta_(atom(mu),A))
//         + sum_g f_g a_g dQ_g/dR_A,
//
// with X^s_mu(g) = sum_nu P^s_mu,nu phi_nu(g) = sum_i C^s_mu,i occ_i T^s_i(g)
// (T = C^T Phi, the orbital values) and, per spin,
//   t_j = 4 c0 d_j phi X + 2 sum_k c_k (d_j d_k phi X + d_j phi d_k X),
// c0 = w v_rho / 2 and c_k = w df/d(d_k rho_s) being the Z coefficients of the
// Fock build (xc_integrals.hpp:506-514, :655-664).  The first sum holds the
// basis-centre and the point-motion terms, the second the Becke-weight term.
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "dmma.cuh"
#include "nkx.h"
#include "plan.cuh"
#include "sto.cuh"

namespace nkx {

nkx_status run_guarded(const char *where, const std::function<void()> &fn);

static inline unsigned gblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

// (C occ)[spin][i][f], the B operand of x_fp64_kernel
__global__ void scale_orbitals_kernel(const double *__restrict__ Ct, const double *__restrict__ occ, int nbf_pad,
                                      long n, double *__restrict__ out) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e < n) out[e] = Ct[e] * occ[e / nbf_pad];
}

// X_c(g, mu) = sum_i T_c(g, i) occ_i C(mu, i) in FP64, one 128-point x
// 128-function tile of one (pair, spin, component) per CTA: eight warps of
// 64 x 32 on DMMA tiles, the i rows of T (256 points) and of C occ (128
// functions) streamed by 16-byte cp.async, 16 orbitals a step (rows past
// nocc filled with zeros).  Bound: FP64 pipe.
constexpr int kXKs = 16, kXStages = 3, kXLd = kBlockF + 4;
constexpr int kXSmem = kXStages * 2 * kXKs * kXLd * 8;
__global__ void __launch_bounds__(256, 1)
    x_fp64_kernel(const double *__restrict__ T, const double *__restrict__ Cocc, int nocc, int nocc_pad, int nbf_pad,
                  int nspin, int nc, const int *__restrict__ pair_batch, const int *__restrict__ pair_blk, long pstart,
                  long sb0, double *__restrict__ X) {
  extern __shared__ __align__(16) double xsm[];  // [stage][A | B][kXKs][kXLd]
  const long q = blockIdx.x / 2;
  const int half = blockIdx.x % 2, sc = blockIdx.y, s = sc / nc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double *A = T + ((size_t)(pair_batch[pstart + q] - sb0) * nspin * nc + sc) * nocc_pad * kBatch + 128 * half;
  const double *Bp = Cocc + (size_t)s * nocc * nbf_pad + (size_t)pair_blk[pstart + q] * kBlockF;
  const int total = (nocc + kXKs - 1) / kXKs;
  auto issue = [&](int t, int st) {
    if (t < total) {
      double *dA = xsm + st * 2 * kXKs * kXLd, *dB = dA + kXKs * kXLd;
#pragma unroll
      for (int r = 0; r < (kXKs * kBlockF / 2) / 256; ++r) {
        const int e = threadIdx.x + 256 * r, k = e / 64, part = 2 * (e % 64), i = t * kXKs + k;
        const bool in = i < nocc;
        cp_async16_fill(dA + k * kXLd + part, A + (size_t)(in ? i : 0) * kBatch + part, in);
        cp_async16_fill(dB + k * kXLd + part, Bp + (size_t)(in ? i : 0) * nbf_pad + part, in);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int st = 0; st < kXStages - 1; ++st) issue(st, st);
  double acc[8][4][2];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int fr = lane >> 2, fk = lane & 3, r0 = 64 * (warp & 1) + fr, c0 = 32 * (warp >> 1) + fr;
  for (int t = 0; t < total; ++t) {
    cp_async_wait<kXStages - 2>();
    __syncthreads();  // step t is visible; the stage refilled below was read in step t - 1
    issue(t + kXStages - 1, (t + kXStages - 1) % kXStages);
    const double *As = xsm + (t % kXStages) * 2 * kXKs * kXLd, *Bs = As + kXKs * kXLd;
#pragma unroll
    for (int k = 0; k < kXKs; k += 4) {
      double av[8], bv[4];
#pragma unroll
      for (int i = 0; i < 8; ++i) av[i] = As[(k + fk) * kXLd + r0 + 8 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = Bs[(k + fk) * kXLd + c0 + 8 * j];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma884(acc[i][j], av[i], bv[j]);
    }
  }
  cp_async_wait<0>();
  double *o = X + ((size_t)q * nspin * nc + sc) * kBatch * kBlockF + (size_t)(128 * half + r0) * kBlockF +
              32 * (warp >> 1) + 2 * fk;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<double2 *>(o + (size_t)8 * i * kBlockF + 8 * j) = make_double2(acc[i][j][0], acc[i][j][1]);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Basis-centre and point-motion terms of one (batch, block) pair and spin,
// from X[pair][spin][comp][g][mu].  Lane l of a warp takes functions 4l .. 4l + 3,
// whose slots share a solid harmonic over the warp (the plan order), and a
// warp 32 of the batch's points, in the order of their owner atoms: the
// point-motion sum of a run of points with one owner stays in registers and
// is reduced over the warp when the owner changes.  Per point the warp forms
// each shell's radial factor R, R'/(r R) = C and D = ((R'' / R) - C) / r^2
// once; with S the harmonic, A = 4 c0 X + 2 c . grad X and B = 2 X,
//   t = R [(C S A + B (D S d.c + C c.grad S)) d + (A + B C d.c) grad S
//          + B C S c + B (hess S) c],   d = r - centre,
// which needs no second derivative of phi itself.  FAST (the mixed-precision
// gradient) takes e^x from exp_neg.
//
// Bound: FP64 issue.  (H2O)_8 PBE: 17.4 ms per gradient with each thread
// evaluating its functions' radial factors and all six second derivatives,
// 2.63 ms now (X alone is 6.2 GB of HBM reads, 1 ms).
template <bool GRAD, bool FAST>
__global__ void __launch_bounds__(256, 2) grad_pair_kernel(
    const StoFunc *__restrict__ sto, const int *__restrict__ fshell, const StoShell *__restrict__ bshell,
    const int *__restrict__ bnshell, const int *__restrict__ fatom, const double *__restrict__ px,
    const double *__restrict__ py, const double *__restrict__ pz, const int *__restrict__ owner,
    const int *__restrict__ pair_batch, const int *__restrict__ pair_blk, long pstart, int nspin,
    int spin, const double *__restrict__ coef, long npad, const double *__restrict__ Xin, double *__restrict__ F) {
  constexpr int NC = GRAD ? 4 : 1;
  __shared__ BlockFuncs B;
  __shared__ double rad[8][3][128];  // R, C, D per warp; at the end the warps' function sums
  __shared__ int s_owner[kBatch], s_fatom[kBlockF], rep_f[kBlockF];
  __shared__ short order[kBatch];
  __shared__ double tfs[kBlockF][3];
  const long p = pstart + blockIdx.x;
  const int b = pair_batch[p], I = pair_blk[p];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  load_block_funcs(B, sto, fshell, bshell, bnshell, I, tid, 256);
  s_owner[tid] = owner[(long)b * kBatch + tid];
  if (tid < kBlockF) s_fatom[tid] = fatom[I * kBlockF + tid];
  __syncthreads();
  {
    const int own = s_owner[tid];
    int rank = 0;
    for (int h = 0; h < kBatch; ++h) rank += s_owner[h] < own || (s_owner[h] == own && h < tid);
    order[rank] = (short)tid;
    if (tid < kBlockF) {
      int rf = 0;
      while (s_fatom[rf] != s_fatom[tid]) ++rf;
      rep_f[tid] = rf;
      tfs[tid][0] = tfs[tid][1] = tfs[tid][2] = 0.0;
    }
  }
  __syncthreads();
  double *wR = rad[warp][0], *wC = rad[warp][1], *wD = rad[warp][2];
  double tf[4][3], tq[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int c = 0; c < 4; ++c) tf[c][0] = tf[c][1] = tf[c][2] = 0.0;
  int cur = s_owner[order[32 * warp]];
  auto flush = [&]() {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double v = warp_sum(tq[j]);
      if (lane == 0 && v != 0.0) atomicAdd(&F[3 * cur + j], v);
      tq[j] = 0.0;
    }
  };
  for (int k = 0; k < 32; ++k) {
    const int g = order[32 * warp + k];
    if (s_owner[g] != cur) {
      flush();
      cur = s_owner[g];
    }
    const long gg = (long)b * kBatch + g;
    const double x = px[gg], y = py[gg], z = pz[gg];
    double X[4][NC], cf[4] = {0.0, 0.0, 0.0, 0.0};
    const double *Xs = Xin + (((size_t)blockIdx.x * nspin + spin) * NC * kBatch + g) * kBlockF + 4 * lane;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double2 *xp = reinterpret_cast<const double2 *>(Xs + (size_t)c * kBatch * kBlockF);
      const double2 u = xp[0], v = xp[1];
      X[0][c] = u.x;
      X[1][c] = u.y;
      X[2][c] = v.x;
      X[3][c] = v.y;
      cf[c] = coef[((size_t)spin * 4 + c) * npad + gg];
    }
    __syncwarp();
    for (int s = lane; s < B.nshell; s += 32) {
      const double dx = x - B.scx[s], dy = y - B.scy[s], dz = z - B.scz[s];
      const double r2 = dx * dx + dy * dy + dz * dz, r = sqrt(r2), zeta = B.szeta[s];
      const int kk = B.sk[s];
      wR[s] = ipow(r, kk) * (FAST ? exp_neg(-zeta * r) : exp(-zeta * r));
      double C = 0.0, D = 0.0;
      if (r > 0.0) {
        const double ir = 1.0 / r, a = kk * ir - zeta;
        C = a * ir;
        D = ((a * a - kk * ir * ir) - C) * (ir * ir);
      }
      wC[s] = C;
      wD[s] = D;
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int sh = B.sh[c][lane], l = B.l[c][lane], m = B.m[c][lane];
      const double d[3] = {x - B.scx[sh], y - B.scy[sh], z - B.scz[sh]};
      const double R = B.norm[c][lane] * wR[sh], C = wC[sh];
      double S, gS[3];
      solid_harmonic_grad(l, m, d[0], d[1], d[2], S, gS[0], gS[1], gS[2]);
      double t[3];
      if constexpr (GRAD) {
        const double Bx = 2.0 * X[c][0];
        const double A = 4.0 * cf[0] * X[c][0] + 2.0 * (cf[1] * X[c][1] + cf[2] * X[c][2] + cf[3] * X[c][3]);
        const double dc = d[0] * cf[1] + d[1] * cf[2] + d[2] * cf[3];
        const double gc = gS[0] * cf[1] + gS[1] * cf[2] + gS[2] * cf[3];
        const double CS = C * S;
        const double pd = CS * A + Bx * (wD[sh] * S * dc + C * gc), pg = A + Bx * C * dc, pc = Bx * CS;
#pragma unroll
        for (int j = 0; j < 3; ++j) t[j] = pd * d[j] + pg * gS[j] + pc * cf[1 + j];
        if (l >= 2) {
          double h[6];
          solid_harmonic_hess(l, m, d[0], d[1], d[2], h[0], h[1], h[2], h[3], h[4], h[5]);
          t[0] += Bx * (h[0] * cf[1] + h[1] * cf[2] + h[2] * cf[3]);
          t[1] += Bx * (h[1] * cf[1] + h[3] * cf[2] + h[4] * cf[3]);
          t[2] += Bx * (h[2] * cf[1] + h[4] * cf[2] + h[5] * cf[3]);
        }
      } else {
        const double A = 4.0 * cf[0] * X[c][0];
#pragma unroll
        for (int j = 0; j < 3; ++j) t[j] = A * (gS[j] + C * S * d[j]);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        tf[c][j] = fma(R, t[j], tf[c][j]);
        tq[j] = fma(R, t[j], tq[j]);
      }
    }
  }
  flush();
  __syncthreads();  // every warp is past its radial factors
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int j = 0; j < 3; ++j) rad[warp][j][4 * lane + c] = tf[c][j];
  __syncthreads();
  for (int e = tid; e < 3 * kBlockF; e += 256) {
    const int j = e / kBlockF, f = e % kBlockF;
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += rad[w][j][f];
    atomicAdd(&tfs[rep_f[f]][j], v);
  }
  __syncthreads();
  if (tid < kBlockF && rep_f[tid] == tid)
    for (int j = 0; j < 3; ++j)
      if (tfs[tid][j] != 0.0) atomicAdd(&F[3 * s_fatom[tid] + j], -tfs[tid][j]);
}

// Becke-weight term: for point g with owner o, Q = P_o / Z, Z = sum_i P_i,
// dQ = sum_i kappa_i sum_(j != i) s'(mu_ij)/s(mu_ij) dmu_ij with
// kappa_i = Q (delta_io - P_i / Z), and
// dmu_ij/dR_A = [u_i (d_oA - d_iA) - u_j (d_oA - d_jA)] / R_ij
//             - mu_ij (e_ij (d_iA - d_jA)) / R_ij   (last term only where
// R_ij = |R_i - R_j| is below the clamp), u_i = (r - R_i)/|r - R_i|,
// e_ij = (R_i - R_j)/|R_i - R_j|.  One thread per point; the gradient is
// accumulated in shared memory (3 natoms doubles) when it fits, else in
// global memory directly.
__device__ __forceinline__ void becke_s_ds(double mu, double &s, double &ds) {
  const double p1 = 1.5 * mu - 0.5 * mu * mu * mu;
  const double p2 = 1.5 * p1 - 0.5 * p1 * p1 * p1;
  const double p3 = 1.5 * p2 - 0.5 * p2 * p2 * p2;
  s = 0.5 * (1.0 - p3);
  ds = -0.5 * (1.5 - 1.5 * p2 * p2) * (1.5 - 1.5 * p1 * p1) * (1.5 - 1.5 * mu * mu);
}

// Atoms that can contribute at a point: with the Laqua clamp Rc, a cell i
// with r_i >= r_min + Rc has P_i = 0 exactly (the nearest atom gives
// mu >= 1), and a factor j with r_j >= r_i + Rc is exactly 1 with s' = 0
// (mu <= -1), so every non-trivial cell, factor and derivative term involves
// only atoms with r < r_min + 2 Rc -- the same exact screening as
// becke_kernel.  Without the clamp, or when more than kGradList atoms are that
// close, the loops run over all atoms.
constexpr int kGradList = 192;

// The Becke-weight term of one point over its candidate list (n <= kGradList
// atoms): the distances to the listed atoms once, every cell function once,
// then the pair terms.  Of the three atoms a pair term (i, j) moves, the
// owner's and i's shares are summed in registers and added once per point
// and per i; only j's share goes to shared memory per pair.
__device__ void becke_grad_listed(const double *__restrict__ C, const double r[3], int o, const int *list, int n,
                                  double rmin, double clamp, double wg, double eg, double *Fa) {
  double rd[kGradList], Pl[kGradList];
  for (int k = 0; k < n; ++k) {
    const int a = list[k];
    const double dx = r[0] - C[3 * a], dy = r[1] - C[3 * a + 1], dz = r[2] - C[3 * a + 2];
    rd[k] = sqrt(dx * dx + dy * dy + dz * dz);
  }
  double Z = 0.0, Po = 0.0;
  for (int k = 0; k < n; ++k) {
    const int i = list[k];
    double P = 0.0;
    if (rd[k] < rmin + clamp) {  // else P_i = 0 exactly (Laqua clamp)
      P = 1.0;
      for (int c = 0; c < n && P != 0.0; ++c) {
        if (c == k) continue;
        const int j = list[c];
        const double dx = C[3 * i] - C[3 * j], dy = C[3 * i + 1] - C[3 * j + 1], dz = C[3 * i + 2] - C[3 * j + 2];
        const double Rij = fmin(sqrt(dx * dx + dy * dy + dz * dz), clamp);
        double mu = (rd[k] - rd[c]) / Rij;
        mu = mu > 1.0 ? 1.0 : (mu < -1.0 ? -1.0 : mu);
        double sv, dsv;
        becke_s_ds(mu, sv, dsv);
        P *= sv;
      }
    }
    Pl[k] = P;
    Z += P;
    if (i == o) Po = P;
  }
  if (!(Po > 0.0 && Z > 0.0)) return;
  const double Q = Po / Z, fa = eg * (wg / Q);
  double Fo[3] = {0.0, 0.0, 0.0};
  for (int ci = 0; ci < n; ++ci) {
    const int i = list[ci];
    const double kappa = Q * ((i == o ? 1.0 : 0.0) - Pl[ci] / Z);
    if (kappa == 0.0 || !(rd[ci] > 0.0)) continue;
    const double ri = rd[ci];
    const double ui[3] = {(r[0] - C[3 * i]) / ri, (r[1] - C[3 * i + 1]) / ri, (r[2] - C[3 * i + 2]) / ri};
    double Fi[3] = {0.0, 0.0, 0.0};
    for (int cj = 0; cj < n; ++cj) {
      if (cj == ci) continue;
      const int j = list[cj];
      const double rj = rd[cj];
      if (!(rj > 0.0)) continue;
      const double e[3] = {C[3 * i] - C[3 * j], C[3 * i + 1] - C[3 * j + 1], C[3 * i + 2] - C[3 * j + 2]};
      const double dij = sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
      const bool clamped = dij >= clamp;
      const double Rij = clamped ? clamp : dij;
      const double mu = (ri - rj) / Rij;
      if (!(mu > -1.0 && mu < 1.0)) continue;  // clamped: s' = 0
      double sv, ds;
      becke_s_ds(mu, sv, ds);
      if (!(sv > 0.0)) continue;
      const double lam = fa * kappa * ds / sv / Rij;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double uj = (r[k] - C[3 * j + k]) / rj;
        const double ek = clamped ? 0.0 : mu * e[k] / dij;
        Fo[k] += lam * (ui[k] - uj);
        Fi[k] -= lam * (ui[k] + ek);
        atomicAdd(&Fa[3 * j + k], lam * (uj + ek));
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (Fi[k] != 0.0) atomicAdd(&Fa[3 * i + k], Fi[k]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (Fo[k] != 0.0) atomicAdd(&Fa[3 * o + k], Fo[k]);
}

__global__ void becke_grad_kernel(const double *__restrict__ C, int natoms, const double *__restrict__ px,
                                  const double *__restrict__ py, const double *__restrict__ pz,
                                  const double *__restrict__ w, const int *__restrict__ owner,
                                  const double *__restrict__ edens, long npad, double clamp, bool smem,
                                  double *__restrict__ F) {
  extern __shared__ double Fs[];
  double *Fa = smem ? Fs : F;
  if (smem) {
    for (int e = threadIdx.x; e < 3 * natoms; e += blockDim.x) Fs[e] = 0.0;
    __syncthreads();
  }
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g < npad && w[g] != 0.0 && edens[g] != 0.0) {
    const double r[3] = {px[g], py[g], pz[g]};
    const int o = owner[g];
    auto dist = [&](int a) {
      const double dx = r[0] - C[3 * a], dy = r[1] - C[3 * a + 1], dz = r[2] - C[3 * a + 2];
      return sqrt(dx * dx + dy * dy + dz * dz);
    };
    int list[kGradList];
    int nl = 0;
    bool full = !(clamp > 0.0);
    double rmin = 1e300;
    if (!full) {
      for (int a = 0; a < natoms; ++a) rmin = fmin(rmin, dist(a));
      for (int a = 0; a < natoms; ++a)
        if (dist(a) < rmin + 2.0 * clamp) {
          if (nl == kGradList) {
            full = true;
            break;
          }
          list[nl++] = a;
        }
    }
    if (!full) {
      becke_grad_listed(C, r, o, list, nl, rmin, clamp, w[g], edens[g], Fa);
    } else {
      // without the clamp, or with more than kGradList candidates: every atom
      const int n = natoms;
      auto atom = [&](int k) { return k; };
      // P_i over the candidate set (factors of the other atoms are exactly 1)
      auto cellP = [&](int i) {
        const double ri = dist(i);
        if (!full && ri >= rmin + clamp) return 0.0;
        double P = 1.0;
        for (int c = 0; c < n && P != 0.0; ++c) {
          const int j = atom(c);
          if (j == i) continue;
          const double dx = C[3 * i] - C[3 * j], dy = C[3 * i + 1] - C[3 * j + 1], dz = C[3 * i + 2] - C[3 * j + 2];
          double Rij = sqrt(dx * dx + dy * dy + dz * dz);
          if (clamp > 0.0) Rij = fmin(Rij, clamp);
          double mu = (ri - dist(j)) / Rij;
          mu = mu > 1.0 ? 1.0 : (mu < -1.0 ? -1.0 : mu);
          double sv, dsv;
          becke_s_ds(mu, sv, dsv);
          P *= sv;
        }
        return P;
      };
      double Z = 0.0, Po = 0.0;
      for (int c = 0; c < n; ++c) {
        const int i = atom(c);
        const double P = cellP(i);
        Z += P;
        if (i == o) Po = P;
      }
      if (Po > 0.0 && Z > 0.0) {
        const double Q = Po / Z, a = w[g] / Q, fa = edens[g] * a;
        for (int ci = 0; ci < n; ++ci) {
          const int i = atom(ci);
          const double Pi = (i == o) ? Po : cellP(i);
          const double kappa = Q * ((i == o ? 1.0 : 0.0) - Pi / Z);
          if (kappa == 0.0) continue;
          double ui[3] = {r[0] - C[3 * i], r[1] - C[3 * i + 1], r[2] - C[3 * i + 2]};
          const double ri = sqrt(ui[0] * ui[0] + ui[1] * ui[1] + ui[2] * ui[2]);
          if (!(ri > 0.0)) continue;
          for (int k = 0; k < 3; ++k) ui[k] /= ri;
          for (int cj = 0; cj < n; ++cj) {
            const int j = atom(cj);
            if (j == i) continue;
            double e[3] = {C[3 * i] - C[3 * j], C[3 * i + 1] - C[3 * j + 1], C[3 * i + 2] - C[3 * j + 2]};
            const double dij = sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
            const bool clamped = clamp > 0.0 && dij >= clamp;
            const double Rij = clamped ? clamp : dij;
            double uj[3] = {r[0] - C[3 * j], r[1] - C[3 * j + 1], r[2] - C[3 * j + 2]};
            const double rj = sqrt(uj[0] * uj[0] + uj[1] * uj[1] + uj[2] * uj[2]);
            if (!(rj > 0.0)) continue;
            const double mu = (ri - rj) / Rij;
            if (!(mu > -1.0 && mu < 1.0)) continue;  // clamped: s' = 0
            double sv, ds;
            becke_s_ds(mu, sv, ds);
            if (!(sv > 0.0)) continue;
            const double lam = fa * kappa * ds / sv / Rij;
            for (int k = 0; k < 3; ++k) {
              uj[k] /= rj;
              const double ek = clamped ? 0.0 : mu * e[k] / dij;
              atomicAdd(&Fa[3 * o + k], lam * (ui[k] - uj[k]));
              atomicAdd(&Fa[3 * i + k], -lam * (ui[k] + ek));
              atomicAdd(&Fa[3 * j + k], lam * (uj[k] + ek));
            }
          }
        }
      }
    }  // every atom
  }
  if (smem) {
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * natoms; e += blockDim.x)
      if (Fs[e] != 0.0) atomicAdd(&F[e], Fs[e]);
  }
}

// The Becke-weight term of molecules of up to kGradCap atoms, a block of
// W warps per 32 points (a point per lane, the same in every warp),
// with the screening of becke_grad_kernel: atoms with r < r_min + 2 Rc of any
// of the points are candidates.  Warp w lists those among the atoms w,
// w + W, ...; shared memory holds per candidate and point the
// distance, the cell function P and the weight D.  With
// a_ij = f a kappa_i s'(mu_ij) / (s(mu_ij) R_ij) the terms of all pairs collapse to
//   F_k += -D_k u_k,  F_o += sum_k D_k u_k,   D_k = sum_j a_kj - sum_i a_ik,
//   F_i -= G_ij e_ij, F_j += G_ij e_ij,       G_ij = sum_points a_ij mu_ij
// (e_ij terms only where |R_i - R_j| is below the clamp), so a pair costs one
// scalar per point, and one warp reduction when it is not clamped; vectors
// appear once per atom.  A warp takes the cells i of its own list for P and the
// atoms j of its own list for D, so only the sums over j (Ss) meet between
// warps.  Each block strides over the points and adds its sums to F once.
//
// Bound: FP64 issue; the candidates' arrays in shared memory set how many
// points an SM has in flight, which is why several warps share them.  By W, in ms
// (a thread per point with vector atomics in shared memory per pair: 0):
//   atoms  points    W = 0   W = 1   W = 4   W = 8   W = 16
//     24   0.22 M     3.97    1.21    0.67    0.79    1.21
//     48   0.43 M    15.3     5.84    2.60    2.57    3.05
//     96   0.85 M    67.0             13.5    8.8     13.9
//    192   1.68 M     250             68.6    42.9    38.3
// so four up to 48 atoms and eight beyond, up to what shared memory holds.
constexpr int kGradCap = 192, kGradNarrow = 48;  // kGradCap a multiple of every W
constexpr size_t kGradAtomBytes = 4 * 32 * sizeof(double) + 3 * sizeof(double) + sizeof(int);
template <int W>
__global__ void __launch_bounds__(32 * W)
    becke_grad_warp_kernel(const double *__restrict__ C, int natoms, const double *__restrict__ px,
                           const double *__restrict__ py, const double *__restrict__ pz, const double *__restrict__ w,
                           const int *__restrict__ owner, const double *__restrict__ edens, long npad, double clamp,
                           double *__restrict__ F) {
  extern __shared__ double gsm[];  // r, P, D, S [slots][32], F [3 natoms], list [slots]
  __shared__ double red[2][W][32], redP[W][32], redZ[W][32];
  __shared__ int nw[W];
  const int seg = (natoms + W - 1) / W, slots = seg * W;
  double *rs = gsm, *Ps = rs + slots * 32, *Ds = Ps + slots * 32, *Ss = Ds + slots * 32, *Fa = Ss + slots * 32;
  int *list = reinterpret_cast<int *>(Fa + 3 * natoms);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, s0 = warp * seg;
  for (int e = threadIdx.x; e < 3 * natoms; e += blockDim.x) Fa[e] = 0.0;
  const double Rc = clamp > 0.0 ? clamp : 1e300;
  int turn = 0;
  for (long g0 = blockIdx.x * 32L; g0 < npad; g0 += gridDim.x * 32L, turn ^= 1) {  // npad is a multiple of 256
    const long g = g0 + lane;
    const double r[3] = {px[g], py[g], pz[g]};
    const double wg = w[g], eg = edens[g];
    const int o = owner[g];
    auto dist2 = [&](int a) {
      const double dx = r[0] - C[3 * a], dy = r[1] - C[3 * a + 1], dz = r[2] - C[3 * a + 2];
      return dx * dx + dy * dy + dz * dz;
    };
    double r2min = 1e300;
    for (int a = warp; a < natoms; a += W) r2min = fmin(r2min, dist2(a));
    red[turn][warp][lane] = r2min;
    __syncthreads();
#pragma unroll
    for (int v = 0; v < W; ++v) r2min = fmin(r2min, red[turn][v][lane]);
    const double rmin = sqrt(r2min), lim = rmin + 2.0 * Rc;
    const bool live = wg != 0.0 && eg != 0.0 && sqrt(dist2(o)) < rmin + Rc;  // else no term, or P_o == 0
    if (!__any_sync(0xffffffffu, live)) continue;  // alike in every warp
    int nl = 0;
    for (int a = warp; a < natoms; a += W) {
      const double ra = sqrt(dist2(a));
      if (!__any_sync(0xffffffffu, live && ra < lim)) continue;
      rs[(s0 + nl) * 32 + lane] = ra;
      Ds[(s0 + nl) * 32 + lane] = Ss[(s0 + nl) * 32 + lane] = 0.0;
      if (lane == 0) list[s0 + nl] = a;
      ++nl;
    }
    if (lane == 0) nw[warp] = nl;
    __syncthreads();
    // |R_i - R_j| of atom i and the candidate in slot c (inverse of the clamped one)
    auto inverse = [&](int i, int c, bool in, double &dij) {
      dij = 0.0;
      if (!in || list[c] == i) return 0.0;
      const int j = list[c];
      const double dx = C[3 * i] - C[3 * j], dy = C[3 * i + 1] - C[3 * j + 1], dz = C[3 * i + 2] - C[3 * j + 2];
      dij = sqrt(dx * dx + dy * dy + dz * dz);
      return 1.0 / fmin(dij, Rc);
    };
    double Z = 0.0, Po = 0.0;
    for (int a = s0; a < s0 + nl; ++a) {
      const double ri = rs[a * 32 + lane];
      const bool cell = live && ri < rmin + Rc;  // else P_i = 0 exactly
      double P = cell ? 1.0 : 0.0;
      const int i = list[a];
      if (__any_sync(0xffffffffu, cell)) {
        const double reach = cell ? ri + Rc : -1.0;
        for (int v = 0; v < W; ++v)
          for (int c0 = 0; c0 < nw[v]; c0 += 32) {
            double dij;
            const int n = min(32, nw[v] - c0), cb = v * seg + c0;
            const double iR = inverse(i, cb + lane, lane < n, dij);
            for (int t = 0; t < n; ++t) {
              const double rj = rs[(cb + t) * 32 + lane];
              if (!__any_sync(0xffffffffu, rj < reach) || cb + t == a) continue;
              double mu = (ri - rj) * __shfl_sync(0xffffffffu, iR, t), sv, dsv;
              mu = mu > 1.0 ? 1.0 : (mu < -1.0 ? -1.0 : mu);
              becke_s_ds(mu, sv, dsv);
              P *= sv;
            }
          }
      }
      Ps[a * 32 + lane] = P;
      Z += P;
      if (i == o) Po = P;
    }
    redZ[warp][lane] = Z;
    redP[warp][lane] = Po;
    __syncthreads();
    Z = Po = 0.0;
#pragma unroll
    for (int v = 0; v < W; ++v) {
      Z += redZ[v][lane];
      Po += redP[v][lane];  // one of them, the others are zero
    }
    const bool on = live && Po > 0.0 && Z > 0.0;
    const double Q = on ? Po / Z : 0.0, fa = on ? eg * (wg / Q) : 0.0, iZ = on ? 1.0 / Z : 0.0;
    for (int v = 0; v < W; ++v)
      for (int a = v * seg; a < v * seg + nw[v]; ++a) {
        const double ri = rs[a * 32 + lane];
        const int i = list[a];
        const double kappa = Q * ((i == o ? 1.0 : 0.0) - Ps[a * 32 + lane] * iZ);
        const bool cell = on && kappa != 0.0 && ri > 0.0;
        if (!__any_sync(0xffffffffu, cell)) continue;
        const double reach = cell ? ri + Rc : -1.0, fk = cell ? fa * kappa : 0.0;
        double S = 0.0;
        for (int c0 = 0; c0 < nl; c0 += 32) {
          double dij;
          const int n = min(32, nl - c0), cb = s0 + c0;
          const double iR = inverse(i, cb + lane, lane < n, dij);
          for (int t = 0; t < n; ++t) {
            const double rj = rs[(cb + t) * 32 + lane];
            if (!__any_sync(0xffffffffu, rj < reach) || cb + t == a) continue;
            const double iRt = __shfl_sync(0xffffffffu, iR, t), dt = __shfl_sync(0xffffffffu, dij, t);
            const double mu = (ri - rj) * iRt;
            double sv, ds, lam = 0.0;
            becke_s_ds(mu, sv, ds);
            if (rj > 0.0 && mu > -1.0 && mu < 1.0 && sv > 0.0) lam = fk * ds / sv * iRt;
            S += lam;
            Ds[(cb + t) * 32 + lane] -= lam;
            if (dt < Rc) {
              const double G = warp_sum(lam * mu);
              if (lane < 3 && G != 0.0) {
                const int j = list[cb + t];
                const double e = G * (C[3 * i + lane] - C[3 * j + lane]) / dt;
                atomicAdd(&Fa[3 * i + lane], -e);
                atomicAdd(&Fa[3 * j + lane], e);
              }
            }
          }
        }
        if (S != 0.0) atomicAdd(&Ss[a * 32 + lane], S);
      }
    __syncthreads();
    // the u terms: per atom over the points, and per point to its owner
    double Fo[3] = {0.0, 0.0, 0.0};
    for (int a = s0; a < s0 + nl; ++a) {
      const double ra = rs[a * 32 + lane], D = Ds[a * 32 + lane] + Ss[a * 32 + lane];
      const double h = ra > 0.0 ? D / ra : 0.0;
      if (!__any_sync(0xffffffffu, h != 0.0)) continue;
      const int i = list[a];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double v = h * (r[k] - C[3 * i + k]);
        Fo[k] += v;
        const double t = warp_sum(v);
        if (lane == 0 && t != 0.0) atomicAdd(&Fa[3 * i + k], -t);
      }
    }
    // lanes of one owner together (most warps have a single one)
    unsigned todo = __ballot_sync(0xffffffffu, on);
    while (todo) {
      const int own = __shfl_sync(0xffffffffu, o, __ffs(todo) - 1);
      const bool mine = on && o == own;
      todo &= ~__ballot_sync(0xffffffffu, mine);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double t = warp_sum(mine ? Fo[k] : 0.0);
        if (lane == 0 && t != 0.0) atomicAdd(&Fa[3 * own + k], t);
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 3 * natoms; e += blockDim.x)
    if (Fa[e] != 0.0) atomicAdd(&F[e], Fa[e]);
}

static void launch_becke_grad(Plan &P, const double *edens, double clamp, double *F, cudaStream_t s) {
  if (P.natoms <= kGradCap) {
    auto go = [&](auto warps) {
      constexpr int W = decltype(warps)::value;
      const size_t smem = (size_t)((P.natoms + W - 1) / W * W) * kGradAtomBytes;
      // the limit is the same for every call, so that threads cannot lower it for one another
      NKX_CUDA(cudaFuncSetAttribute(becke_grad_warp_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(kGradCap * kGradAtomBytes)));
      int per_sm = 1;
      NKX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, becke_grad_warp_kernel<W>, 32 * W, smem));
      const unsigned grid = (unsigned)std::min<long>(P.npad / 32, (long)std::max(1, per_sm) * P.nsm);
      becke_grad_warp_kernel<W><<<grid, 32 * W, smem, s>>>(P.d_centers, P.natoms, P.d_px, P.d_py, P.d_pz, P.d_w,
                                                          P.d_owner, edens, P.npad, clamp, F);
    };
    P.natoms <= kGradNarrow ? go(std::integral_constant<int, 4>{}) : go(std::integral_constant<int, 8>{});
  } else {
    const size_t fs_bytes = sizeof(double) * 3 * (size_t)P.natoms;
    const bool smem = fs_bytes <= 48 * 1024;
    becke_grad_kernel<<<gblk(P.npad, 128), 128, smem ? fs_bytes : 0, s>>>(P.d_centers, P.natoms, P.d_px, P.d_py,
                                                                         P.d_pz, P.d_w, P.d_owner, edens, P.npad,
                                                                         clamp, smem, F);
  }
  NKX_LAUNCH_CHECK();
}

struct GradState {
  double *T = nullptr, *X = nullptr, *Cocc = nullptr, *edens = nullptr, *F = nullptr;
  size_t T_cap = 0, X_cap = 0, C_cap = 0;
  ~GradState() {
    for (double *p : {T, X, Cocc, edens, F}) cudaFree(p);
  }
  static double *alloc(size_t n) {
    double *p = nullptr;
    if (cudaMalloc(&p, std::max<size_t>(1, n) * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      throw Error{NKX_ERR_ALLOC, "gradient workspace allocation of " + std::to_string(n * 8) + " bytes failed"};
    }
    return p;
  }
  static void give_back(double *&p, size_t &cap) {
    cudaFree(p);
    p = nullptr;
    cap = 0;
  }
  static void ensure(double *&p, size_t &cap, size_t n) {
    if (n <= cap) return;
    give_back(p, cap);
    p = alloc(n);
    cap = n;
  }
};

void destroy_grad_state(void *p) { delete static_cast<GradState *>(p); }

static GradState &grad_state(Plan &P) {
  if (!P.grad_state) {
    GradState *G = new GradState();
    P.grad_state = G;
    G->edens = GradState::alloc(P.npad);
    G->F = GradState::alloc(3 * (size_t)P.natoms);
  }
  return *static_cast<GradState *>(P.grad_state);
}

template <bool FAST>
static void launch_grad_pairs(Plan &P, long q0, long q1, int nspin, const double *X, double *F, cudaStream_t s) {
  auto *kernel = P.gga ? grad_pair_kernel<true, FAST> : grad_pair_kernel<false, FAST>;
  for (int spin = 0; spin < nspin; ++spin) {
    kernel<<<(unsigned)(q1 - q0), 256, 0, s>>>(P.d_sto, P.d_fshell, P.d_bshell, P.d_bnshell, P.d_fatom, P.d_px, P.d_py,
                                               P.d_pz, P.d_owner, P.d_pair_batch, P.d_pair_blk, q0, nspin, spin,
                                               P.d_coef, P.npad, X, F);
    NKX_LAUNCH_CHECK();
    ++P.launches;
  }
}

// T and X of the FP64 gradient go through buffers of at most this many bytes, and
// through smaller ones on a card that has no room for these
constexpr size_t kGradTBytes = (size_t)512 << 20, kGradXBytes = (size_t)1536 << 20;

// FP64 part of the gradient: per chunk the FP64 collocation, then per range
// of its batches the orbital values T with the density, the functional,
// X = (C occ) T of the range's pairs, and the pair terms.
static void fp64_gradient_chunks(Plan &P, GradState &G, int nspin, int nocc, cudaStream_t s) {
  const int NC = P.gga ? 4 : 1;
  int nn = 0;
  const int nocc_pad = fp64_orbital_pad(nocc, &nn);
  const size_t t1 = (size_t)nspin * NC * nocc_pad * kBatch, x1 = (size_t)nspin * NC * kBatch * kBlockF;
  fp64_density_begin(P, nspin, nocc, s);
  G.ensure(G.Cocc, G.C_cap, (size_t)nspin * nocc * P.nbf_pad);
  const long nC = (long)nspin * nocc * P.nbf_pad;
  scale_orbitals_kernel<<<gblk(nC, 256), 256, 0, s>>>(P.d_Ct, P.d_occ, P.nbf_pad, nC, G.Cocc);
  NKX_LAUNCH_CHECK();
  ++P.launches;
  long cap_b = std::max<long>(1, (long)(kGradTBytes / 8 / t1));
  long cap_q = std::max<long>(P.nblk, (long)(kGradXBytes / 8 / x1));
  // end of the range of chunk c's batches that starts at b0
  auto range_end = [&](const Chunk &c, long b0) {
    long b1 = b0 + 1;
    while (b1 < c.b1 && b1 - b0 < cap_b && P.h_pair_off[b1 + 1] - P.h_pair_off[b0] <= cap_q) ++b1;
    return b1;
  };
  for (;; cap_b = std::max(1L, cap_b / 2), cap_q = std::max<long>(P.nblk, cap_q / 2)) {
    long nb = 0, nq = 0;
    for (const Chunk &c : P.chunks)
      for (long b0 = c.b0, b1; b0 < c.b1; b0 = b1) {
        b1 = range_end(c, b0);
        nb = std::max(nb, b1 - b0);
        nq = std::max<long>(nq, P.h_pair_off[b1] - P.h_pair_off[b0]);
      }
    try {
      G.ensure(G.T, G.T_cap, (size_t)nb * t1);
      G.ensure(G.X, G.X_cap, (size_t)nq * x1);
      break;
    } catch (const Error &e) {
      if (e.code != NKX_ERR_ALLOC || (cap_b == 1 && cap_q == P.nblk)) throw;
      G.give_back(G.T, G.T_cap);
    }
  }
  NKX_CUDA(cudaFuncSetAttribute(x_fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kXSmem));
  for (const Chunk &c : P.chunks) {
    launch_colloc(P, c, s);
    for (long b0 = c.b0, b1; b0 < c.b1; b0 = b1) {
      b1 = range_end(c, b0);
      const long q0 = P.h_pair_off[b0], q1 = P.h_pair_off[b1];
      fp64_density_range(P, b0, b1, c.p0, nspin, nocc, G.T, s);
      const long g0 = b0 * kBatch, n = (b1 - b0) * kBatch;
      functional_kernel<<<gblk(n, 256), 256, 0, s>>>(P.xc, P.gga, nspin, P.npad, n, P.d_w + g0, P.d_rho + g0,
                                                     P.d_grad + g0, nullptr, P.d_coef + g0, P.d_E, G.edens + g0);
      NKX_LAUNCH_CHECK();
      ++P.launches;
      if (q1 <= q0) continue;
      x_fp64_kernel<<<dim3((unsigned)(2 * (q1 - q0)), nspin * NC), 256, kXSmem, s>>>(
          G.T, G.Cocc, nocc, nocc_pad, P.nbf_pad, nspin, NC, P.d_pair_batch, P.d_pair_blk, q0, b0, G.X);
      NKX_LAUNCH_CHECK();
      ++P.launches;
      launch_grad_pairs<false>(P, q0, q1, nspin, G.X, G.F, s);
    }
  }
}

static void xc_gradient(Plan &P, int precision, int nspin, int nocc, const double *C, const double *occ, int mem,
                        double clamp, double *grad, cudaStream_t s) {
  NKX_REQUIRE(precision == NKX_PREC_FP64 || precision == NKX_PREC_MIXED, NKX_ERR_ARG,
              "precision must be NKX_PREC_FP64 or NKX_PREC_MIXED");
  NKX_REQUIRE(precision == NKX_PREC_FP64 || mixed_available(P), NKX_ERR_UNSUPPORTED,
              "the mixed-precision gradient needs an sm_100 device");
  NKX_REQUIRE(nspin == 1 || nspin == 2, NKX_ERR_ARG, "nspin must be 1 or 2");
  NKX_REQUIRE(nocc > 0 && C && occ && grad, NKX_ERR_ARG, "invalid arguments");
  NKX_REQUIRE(mem == NKX_MEM_DEVICE || mem == NKX_MEM_HOST, NKX_ERR_ARG, "mem must be NKX_MEM_DEVICE or NKX_MEM_HOST");
  NKX_REQUIRE(P.natoms > 0 && P.d_owner, NKX_ERR_ARG, "the gradient needs a plan created with atoms and point owners");
  NKX_REQUIRE(P.all_funcs_on_atoms, NKX_ERR_ARG, "the gradient needs every basis function centred on an atom");
  P.launches = 0;
  NKX_CUDA(cudaMemsetAsync(P.d_status, 0, sizeof(int) * 2, s));
  upload_orbitals(P, nspin, nocc, C, occ, mem, s);
  const bool mixed = precision == NKX_PREC_MIXED;
  GradState &G = grad_state(P);
  NKX_CUDA(cudaMemsetAsync(P.d_E, 0, sizeof(double), s));
  NKX_CUDA(cudaMemsetAsync(G.F, 0, sizeof(double) * 3 * P.natoms, s));
  if (mixed) {
    // Mixed precision: per chunk, the orbital values T_c come from the int8
    // digit contraction on the tensor cores, which also gives rho, grad rho
    // and the functional of the chunk's points, and so do X = C (occ T) and
    // its gradient; the pair terms and the Becke term are FP64.
    mixed_gradient_begin(P, nspin, nocc, s);
    for (const Chunk &c : P.chunks) {
      const double *X = mixed_gradient_chunk(P, c, nspin, nocc, G.edens, s);
      if (c.p1 > c.p0) launch_grad_pairs<true>(P, c.p0, c.p1, nspin, X, G.F, s);
    }
  } else {
    fp64_gradient_chunks(P, G, nspin, nocc, s);
  }
  const size_t fs_bytes = sizeof(double) * 3 * (size_t)P.natoms;
  launch_becke_grad(P, G.edens, clamp, G.F, s);
  ++P.launches;
  NKX_CUDA(cudaMemcpyAsync(grad, G.F, fs_bytes, cudaMemcpyDeviceToHost, s));
  int status[2] = {0, 0};
  NKX_CUDA(cudaMemcpyAsync(status, P.d_status, sizeof(status), cudaMemcpyDeviceToHost, s));
  NKX_CUDA(cudaStreamSynchronize(s));
  NKX_REQUIRE(status[0] == 0, NKX_ERR_TIMEOUT, "a tensor-core kernel wait gave up; the gradient is invalid");
  NKX_REQUIRE(status[1] == 0, NKX_ERR_NUMERIC, "non-finite value in the orbitals or occupations");
}

}  // namespace nkx

extern "C" NKX_API nkx_status nkx_xc_gradient(nkx_plan *plan, int precision, int nspin, int nocc, const double *C,
                                               const double *occ, int mem, double becke_clamp, double *grad,
                                               void *stream) {
  return nkx::run_guarded("nkx_xc_gradient", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    nkx::Plan &P = *reinterpret_cast<nkx::Plan *>(plan);
    nkx::xc_gradient(P, precision, nspin, nocc, C, occ, mem, becke_clamp, grad,
                     stream ? (cudaStream_t)stream : P.stream);
  });
}
