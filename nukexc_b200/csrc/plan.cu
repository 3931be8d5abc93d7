// The batched, screened grid-integration Fock build (the hot path).
//
// Once per geometry (nkx_plan_create): the grid is sorted into Morton order
// and cut into 256-point batches (create_bounding_boxes,
// nukexc/octree.hpp:70-141); basis functions are grouped into blocks of 128
// (by reach where that pays, then by centre in Morton order) and a block is significant for a batch when the cutoff
// sphere of any of its functions meets the batch's bounding box
// (build_neighbor_list, nukexc/octree.hpp:317-390); the aux Coulomb metric is
// integrated on the grid and Cholesky-factorised in FP64.
//
// Per SCF iteration (nkx_fock_build), streamed over chunks of batches that
// fit the workspace:
//   pass A  collocation  PhiT[pair][g][f] (value + gradient)       colloc_*
//           density      T = PhiT C, rho = sum occ T^2, grad rho    density_*
//   J       y = (Vw rho), c = (A|B)^-1 y, v_g = sum c_a V_a(g) w_g  aux_*
//   XC      functional on every point, E_xc, Z coefficients         functional_kernel
//   pass B  Z^T[pair][g][f] = a_g phi + b_g . grad phi              zbuild_*
//           Vbar(I,J) += sum_b PhiT_bI^T Z_bJ  per function-block tile
//   end     V = Vbar + Vbar^T, unpadded to nbf x nbf
// (compute_gga / compute_gga_lsda, nukexc/xc_integrals.hpp:424-726, and
// compute_coulomb, nukexc/coulomb.hpp:56-115, reorganised into batches).
#include <cublas_v2.h>
#include <cusolverDn.h>

#include <algorithm>
#include <parallel/algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <numeric>
#include <vector>

#include "dmma.cuh"
#include "functionals.cuh"
#include "host_setup.hpp"
#include "plan.cuh"

namespace nkx {

// ------------------------------------------------------------- errors ----
static thread_local std::string g_last_error;
void set_error(const std::string &msg) { g_last_error = msg; }

nkx_status run_guarded(const char *where, const std::function<void()> &fn) {
  try {
    fn();
    return NKX_OK;
  } catch (const Error &e) {
    set_error(std::string(where) + ": " + e.msg);
    return e.code;
  } catch (const std::bad_alloc &) {
    set_error(std::string(where) + ": host allocation failed");
    return NKX_ERR_ALLOC;
  } catch (const std::exception &e) {
    set_error(std::string(where) + ": " + e.what());
    return NKX_ERR_ARG;
  }
}

XcSpec make_spec(const nkx_plan_options *o);
bool spec_is_gga(const XcSpec &s);

template <class T>
static T *dalloc(size_t n) {
  T *p = nullptr;
  if (n == 0) return nullptr;
  const cudaError_t e = cudaMalloc(&p, n * sizeof(T));
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error{NKX_ERR_ALLOC, "cudaMalloc of " + std::to_string(n * sizeof(T)) + " bytes failed"};
  }
  return p;
}

static unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

// ========================================================== kernels ======

// Collocation of one (batch, function block) pair per CTA.  Lane l of a warp
// owns the four consecutive functions f = 4l .. 4l+3 of the block; warp w owns
// points g = w + 8j.  Per point the warp first evaluates the radial factor of
// each of the block's shells once (block_radials), since the plan order gives
// a lane four functions of different shells.  Output PhiT[pair][comp][g][f],
// comp 0 = value, 1..3 = gradient (GRAD only); each warp store covers 32 x 4
// consecutive f.
template <bool GRAD>
__global__ void __launch_bounds__(256) colloc_fp64_kernel(const StoFunc *__restrict__ sto, const int *__restrict__ fshell,
                                                          const StoShell *__restrict__ bshell,
                                                          const int *__restrict__ bnshell, const double *__restrict__ px,
                                                          const double *__restrict__ py, const double *__restrict__ pz,
                                                          const int *__restrict__ pair_batch,
                                                          const int *__restrict__ pair_blk, long p0,
                                                          double *__restrict__ out) {
  const long p = p0 + blockIdx.x;
  const int b = pair_batch[p], I = pair_blk[p];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ double sx[kBatch], sy[kBatch], sz[kBatch];
  __shared__ BlockFuncs B;
  __shared__ double wR[8][128], wC[8][128];
  for (int g = threadIdx.x; g < kBatch; g += blockDim.x) {
    sx[g] = px[(long)b * kBatch + g];
    sy[g] = py[(long)b * kBatch + g];
    sz[g] = pz[(long)b * kBatch + g];
  }
  load_block_funcs(B, sto, fshell, bshell, bnshell, I, threadIdx.x, blockDim.x);
  __syncthreads();
  const size_t tile = (size_t)kBatch * kBlockF;
  double *o = out + (size_t)blockIdx.x * (GRAD ? 4 : 1) * tile;
  const int npt = kBatch / gridDim.y, g0 = blockIdx.y * npt;  // this CTA's points
  for (int g = g0 + warp; g < g0 + npt; g += 8) {
    const double x = sx[g], y = sy[g], z = sz[g];
    double v[4][4];
    __syncwarp();
    block_radials<GRAD, false>(B, lane, x, y, z, wR[warp], wC[warp]);
    __syncwarp();
    block_funcs_eval4<GRAD>(B, lane, x, y, z, wR[warp], wC[warp], v[0], v[1], v[2], v[3]);
    const size_t idx = (size_t)g * kBlockF + 4 * lane;
#pragma unroll
    for (int k = 0; k < (GRAD ? 4 : 1); ++k) {
      double2 *dst = reinterpret_cast<double2 *>(o + k * tile + idx);
      dst[0] = make_double2(v[k][0], v[k][1]);
      dst[1] = make_double2(v[k][2], v[k][3]);
    }
  }
}

// Density of one slab of one batch for one spin, FP64: T(g, i) = sum_f
// PhiT(g, f) C(f, i) over the batch's significant blocks (and the three
// gradient components), then rho = sum_i occ_i T^2 and grad rho =
// 2 sum_i occ_i T grad T (density.hpp:188-255).  A CTA takes 64 points with
// gradients or all 256 without, and NT = 8 NN orbitals.  Its 256 (component,
// point) rows go 32 to a warp as four 8-row DMMA tiles -- the four components
// of eight points, so a thread holds T and grad T of the same point and
// orbitals.  A K step is 16 functions of one block: the rows of PhiT and of
// the function-major orbitals Cf stream into shared memory by 16-byte
// cp.async through a ring of STAGES; rows are padded by four doubles, which
// makes both fragment reads free of bank conflicts.  The orbital tile is the
// fastest grid index, so the CTAs of one slab run together and read its PhiT
// rows from L2; each adds its share of rho and grad rho atomically (zeroed by
// the caller).  With T (the gradient) the orbital values are also written,
// T[(b - b0, spin, comp)][i][g].
//
// Bound: FP64 pipe from about 16 orbitals on, PhiT from HBM below.  The
// orbital tile is ceil(nocc / ntile / 8) * 8 wide instead of a fixed 64, so 5
// to 40 occupied orbitals do not pay for 64 columns; up to 32 columns the
// accumulators leave room for two CTAs an SM.
constexpr int kDKs = 16;
template <int NN>
struct DShape {
  static constexpr int NT = 8 * NN, LDP = kDKs + 4, LDC = NT + 4;
  static constexpr int STAGES = NN <= 4 ? 2 : 3, CTAS = NN <= 4 ? 2 : 1;
  static constexpr int kStage = 256 * LDP + kDKs * LDC;  // doubles
  static constexpr int kSmem = STAGES * kStage * 8;
};

template <bool GRAD, int NN>
__global__ void __launch_bounds__(256, DShape<NN>::CTAS)
    density_fp64_kernel(const double *__restrict__ phiT, const double *__restrict__ Cf, const double *__restrict__ occ,
                        int nocc, int nocc_pad, int nbf_pad, const int *__restrict__ pair_off,
                        const int *__restrict__ pair_blk, long b0, long p0, double *__restrict__ rho,
                        double *__restrict__ grad, long npad, double *__restrict__ T) {
  using Sh = DShape<NN>;
  constexpr int NC = GRAD ? 4 : 1, NT = Sh::NT, LDP = Sh::LDP, LDC = Sh::LDC, ST = Sh::STAGES;
  constexpr int SLABS = GRAD ? 4 : 1;  // slabs of a batch
  extern __shared__ __align__(16) double dsm[];  // [stage][Ps: 256 rows x LDP | Cs: 16 x LDC]
  const int spin = blockIdx.y;
  const int ntile = nocc_pad / NT;
  const int i0 = (blockIdx.x % ntile) * NT;
  const long bq = blockIdx.x / ntile;
  const long b = b0 + bq / SLABS;
  const int g0 = (int)(bq % SLABS) * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double *C = Cf + (size_t)spin * nbf_pad * nocc_pad;
  const double *oc = occ + (size_t)spin * nocc;
  const int q0 = pair_off[b], q1 = pair_off[b + 1];
  const size_t tile = (size_t)kBatch * kBlockF;
  const int total = (q1 - q0) * (kBlockF / kDKs);  // K steps of the orbital tile
  if (total == 0) return;  // no significant function: nothing to add (and no pair that reads T)
  auto issue = [&](int t, int st) {
    if (t < total) {
      const int q = q0 + t / (kBlockF / kDKs), f0 = (t % (kBlockF / kDKs)) * kDKs;
      const double *P = phiT + (size_t)(q - p0) * NC * tile + (size_t)g0 * kBlockF + f0;
      double *Ps = dsm + st * Sh::kStage, *Cs = Ps + 256 * LDP;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int e = threadIdx.x + 256 * r, row = e / (kDKs / 2), part = e % (kDKs / 2);
        // GRAD: row = 32 (point / 8) + 8 comp + point % 8
        const int c = GRAD ? (row / 8) % 4 : 0, pt = GRAD ? 8 * (row / 32) + row % 8 : row;
        cp_async16(Ps + row * LDP + 2 * part, P + c * tile + (size_t)pt * kBlockF + 2 * part);
      }
      const double *Cr = C + (size_t)(pair_blk[q] * kBlockF + f0) * nocc_pad + i0;
      for (int e = threadIdx.x; e < kDKs * NT / 2; e += 256) {
        const int k = e / (NT / 2), part = e % (NT / 2);
        cp_async16(Cs + k * LDC + 2 * part, Cr + (size_t)k * nocc_pad + 2 * part);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int st = 0; st < ST - 1; ++st) issue(st, st);
  double acc[4][NN][2];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < NN; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
  const int fr = lane >> 2, fk = lane & 3;
  for (int t = 0; t < total; ++t) {
    cp_async_wait<ST - 2>();
    __syncthreads();  // step t is visible; the stage refilled below was read in step t - 1
    issue(t + ST - 1, (t + ST - 1) % ST);
    const double *Ps = dsm + (t % ST) * Sh::kStage, *Cs = Ps + 256 * LDP;
#pragma unroll
    for (int k = 0; k < kDKs; k += 4) {
      double av[4], bv[NN];
#pragma unroll
      for (int m = 0; m < 4; ++m) av[m] = Ps[(32 * warp + 8 * m + fr) * LDP + k + fk];
#pragma unroll
      for (int n = 0; n < NN; ++n) bv[n] = Cs[(k + fk) * LDC + 8 * n + fr];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < NN; ++n) dmma884(acc[m][n], av[m], bv[n]);
    }
  }
  cp_async_wait<0>();
  if (T) {
    double *Tb = T + ((size_t)(b - b0) * gridDim.y + spin) * NC * nocc_pad * kBatch;
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          Tb[((size_t)(GRAD ? m : 0) * nocc_pad + i0 + 8 * n + 2 * fk + h) * kBatch +
             (GRAD ? g0 + 8 * warp + fr : 32 * warp + 8 * m + fr)] = acc[m][n][h];
  }
  // contract over this orbital tile: the four lanes of a row hold its columns
  double sm[4] = {0, 0, 0, 0};
#pragma unroll
  for (int n = 0; n < NN; ++n)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = i0 + 8 * n + 2 * fk + h;
      const double o = i < nocc ? oc[i] : 0.0;
#pragma unroll
      for (int m = 0; m < 4; ++m) sm[m] += o * acc[GRAD ? 0 : m][n][h] * acc[m][n][h];
    }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    sm[m] += __shfl_xor_sync(0xffffffffu, sm[m], 1);
    sm[m] += __shfl_xor_sync(0xffffffffu, sm[m], 2);
  }
  if (fk == 0) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (GRAD) {
        const long g = b * kBatch + g0 + 8 * warp + fr;
        if (m == 0)
          atomicAdd(&rho[(size_t)spin * npad + g], sm[0]);
        else
          atomicAdd(&grad[((size_t)spin * 3 + m - 1) * npad + g], 2.0 * sm[m]);
      } else {
        atomicAdd(&rho[(size_t)spin * npad + b * kBatch + 32 * warp + 8 * m + fr], sm[m]);
      }
    }
  }
}

// Orbitals in function-major order for density_fp64_kernel:
// Cf[spin][f][i] = Ct[spin][i][f], orbitals padded to nocc_pad with zeros.
__global__ void transpose_orbitals_kernel(const double *__restrict__ Ct, int nocc, int nocc_pad, int nbf_pad,
                                          double *__restrict__ Cf) {
  __shared__ double t[32][33];
  const int spin = blockIdx.z;
  const int f0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r;
    t[r][threadIdx.x] = i < nocc ? Ct[((size_t)spin * nocc + i) * nbf_pad + f0 + threadIdx.x] : 0.0;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y)
    if (i0 + threadIdx.x < nocc_pad) Cf[((size_t)spin * nbf_pad + f0 + r) * nocc_pad + i0 + threadIdx.x] = t[threadIdx.x][r];
}

// Functional on points [0, n) of the arrays given (plane stride npad; callers
// offset the pointers to work on a range): E_xc, and the Z coefficients
// coef[spin][0][g] = w (1/2 vrho + 1/2 vJ), coef[spin][1..3][g] = w vec
// (xc_integrals.hpp:506-514 closed shell, :655-664 open shell).  vj (may be
// null) is the weighted fitted Coulomb potential folded into both spins.
__global__ void functional_kernel(XcSpec s, bool gga, int nspin, long npad, long n, const double *__restrict__ w,
                                  const double *__restrict__ rho, const double *__restrict__ grad,
                                  const double *__restrict__ vj, double *__restrict__ coef, double *Eacc,
                                  double *__restrict__ edens) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  double e = 0.0, fdens = 0.0;
  if (g < n) {
    const double wg = w[g];
    double vr[2] = {0, 0}, vec[2][3] = {{0, 0, 0}, {0, 0, 0}}, gr[2][3] = {{0, 0, 0}, {0, 0, 0}};
    if (gga)
      for (int sp = 0; sp < nspin; ++sp)
        for (int k = 0; k < 3; ++k) gr[sp][k] = grad[((size_t)sp * 3 + k) * npad + g];
    if (wg != 0.0) {
      if (nspin == 1) {
        const double sg = gr[0][0] * gr[0][0] + gr[0][1] * gr[0][1] + gr[0][2] * gr[0][2];
        double f, vrho, vs;
        xc_unpol(s, rho[g], sg, f, vrho, vs);
        fdens = f;
        e = wg * f;
        vr[0] = vrho;
        for (int k = 0; k < 3; ++k) vec[0][k] = 2.0 * vs * gr[0][k];
      } else {
        const double saa = gr[0][0] * gr[0][0] + gr[0][1] * gr[0][1] + gr[0][2] * gr[0][2];
        const double sab = gr[0][0] * gr[1][0] + gr[0][1] * gr[1][1] + gr[0][2] * gr[1][2];
        const double sbb = gr[1][0] * gr[1][0] + gr[1][1] * gr[1][1] + gr[1][2] * gr[1][2];
        double f, d[5];
        xc_pol(s, rho[g], rho[npad + g], saa, sab, sbb, f, d);
        fdens = f;
        e = wg * f;
        vr[0] = d[0];
        vr[1] = d[1];
        for (int k = 0; k < 3; ++k) {
          vec[0][k] = 2.0 * d[2] * gr[0][k] + d[3] * gr[1][k];
          vec[1][k] = 2.0 * d[4] * gr[1][k] + d[3] * gr[0][k];
        }
      }
    }
    if (edens) edens[g] = fdens;
    const double vjg = vj ? vj[g] : 0.0;
    for (int sp = 0; sp < nspin; ++sp) {
      coef[((size_t)sp * 4 + 0) * npad + g] = wg * 0.5 * vr[sp] + 0.5 * vjg;
      coef[((size_t)sp * 4 + 1) * npad + g] = wg * vec[sp][0];
      coef[((size_t)sp * 4 + 2) * npad + g] = wg * vec[sp][1];
      coef[((size_t)sp * 4 + 3) * npad + g] = wg * vec[sp][2];
    }
  }
  __shared__ double red[32];
  for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x < 32) {
    e = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (threadIdx.x == 0) atomicAdd(Eacc, e);
  }
}

// Z^T[pair][spin][g][f] = coef0 phi + coef1 dphi/dx + coef2 dphi/dy + coef3 dphi/dz.
// Spin index nspin (when jonly) builds Z_J = 1/2 vJ phi for a separate J.
// SPLIT: a pair's points are dealt to gridDim.y CTAs (else a constant count, with
// which LDA planes of many pairs take a tenth less)
template <bool GRAD, bool SPLIT>
__global__ void zbuild_fp64_kernel(const double *__restrict__ phiT, const double *__restrict__ coef,
                                   const double *__restrict__ vj, const int *__restrict__ pair_batch, long p0,
                                   int nz, int nspin, long npad, double *__restrict__ zT) {
  constexpr int NC = GRAD ? 4 : 1;
  const long q = blockIdx.x;
  const int b = pair_batch[p0 + q];
  const size_t tile = (size_t)kBatch * kBlockF;
  const double *P = phiT + q * NC * tile;
  const int ne = kBatch * kBlockF / (SPLIT ? gridDim.y : 1), e0 = SPLIT ? blockIdx.y * ne : 0;  // this CTA's elements
  for (int e = e0 + threadIdx.x; e < e0 + ne; e += blockDim.x) {
    const int g = e / kBlockF;
    const long gg = (long)b * kBatch + g;
    const double v = P[e];
    double dx = 0, dy = 0, dz = 0;
    if (GRAD) {
      dx = P[tile + e];
      dy = P[2 * tile + e];
      dz = P[3 * tile + e];
    }
    for (int s = 0; s < nz; ++s) {
      double z;
      if (s < nspin) {
        const double *c = coef + (size_t)s * 4 * npad;
        z = c[gg] * v;
        if (GRAD) z += c[npad + gg] * dx + c[2 * npad + gg] * dy + c[3 * npad + gg] * dz;
      } else {
        z = 0.5 * vj[gg] * v;
      }
      zT[(q * nz + s) * tile + e] = z;
    }
  }
}

__device__ __forceinline__ int block_pos(const uint32_t *m, int I) {
  int pos = 0;
  for (int w = 0; w < (I >> 5); ++w) pos += __popc(m[w]);
  return pos + __popc(m[I >> 5] & ((1u << (I & 31)) - 1u));
}
__device__ __forceinline__ bool block_has(const uint32_t *m, int I) { return (m[I >> 5] >> (I & 31)) & 1u; }

// V contraction of the FP64 build: Vbar(I, J) += sum_b PhiT_b,I^T Z_b,J over
// the chunk's batches b where blocks I and J are both significant
// (xc_integrals.hpp:677-706), one 128 x 128 output tile per CTA: eight warps
// of 64 x 32, DMMA tiles of 8 x 8 x 4.  The operand rows of a pair, PhiT[g][f]
// and Z^T[g][f], are 1 KB rows of 128 functions per point, so each 16-point K
// step of both operands (32 KB) streams into shared memory with 16-byte
// cp.async copies through a ring of kVStages stages while the previous steps
// are multiplied; rows are padded by four doubles (conflict-free fragments).
//
// Split over batches: a basis of one to a few blocks has only nz nblk^2
// output tiles, far fewer than SMs.  With nsplit > 1 the batches of a tile
// are dealt to nsplit CTAs, each of which writes its partial tile to part[]
// (thread-major, coalesced); vpart_reduce_kernel adds the parts in order, so
// the result does not depend on scheduling.
//
// Bound: FP64 tensor pipe (80 % active at (H2O)_16).  V alone, before
// (CUDA-core tiles, one CTA per output tile) and after: one water 13.4 ms (on
// two SMs) -> 78 us, (H2O)_5 open-shell PBE 64.3 ms (on eight) -> 3.15 ms,
// (H2O)_64 now 2.43 s (25.6 TFLOP/s, 72 % of a cuBLAS DGEMM).
constexpr int kVKs = 16, kVStages = 4, kVLd = kBlockF + 4;
constexpr int kVStageDoubles = 2 * kVKs * kVLd;
constexpr int kVSmemBytes = kVStages * kVStageDoubles * 8;

// next K step of a V unit: step k of batch b, batches without both blocks
// skipped; b walks with stride db
__device__ __forceinline__ void vstep_next(const uint32_t *__restrict__ mask, int mask_words, long b1, int db, int I,
                                           int J, long &b, int &k) {
  if (++k < kBatch / kVKs) return;
  k = 0;
  for (b += db; b < b1; b += db) {
    const uint32_t *m = mask + b * mask_words;
    if (block_has(m, I) && block_has(m, J)) return;
  }
}

// Output tiles: SL slots of each lane of both blocks (positions 4 lane + c,
// c < SL), 32 SL rows and columns.  A block of at most 64 functions has them all
// in two slots, so a basis of one such block multiplies a quarter of the tile
// (SL = 2; one water, 48 functions, FP64 V of two planes: 176 us with SL = 4,
// 78 us).  Row or column r of the tile is position vtile_pos<SL>(r) of its block.
template <int SL>
__device__ __forceinline__ int vtile_pos(int r) {
  return SL == 4 ? r : 4 * (r / SL) + r % SL;
}
// element e of thread t of a tile: rows and columns of warp (t / 32)'s
// 16 SL x 8 SL part
template <int SL>
__device__ __forceinline__ void vtile_element(int t, int e, int &r, int &c) {
  const int lane = t & 31, warp = t >> 5;
  r = vtile_pos<SL>(16 * SL * (warp & 1) + 8 * (e / (2 * SL)) + (lane >> 2));
  c = vtile_pos<SL>(8 * SL * (warp >> 1) + 8 * ((e >> 1) % SL) + 2 * (lane & 3) + (e & 1));
}

template <int SL>
__global__ void __launch_bounds__(256, 1)
    vgemm_fp64_kernel(const double *__restrict__ phiT, const double *__restrict__ zT, int phi_stride_tiles,
                      int z_stride, const int *__restrict__ pair_off, const uint32_t *__restrict__ mask,
                      int mask_words, long b0, long b1, long p0, int nsplit, int nbf_pad, double *__restrict__ V,
                      double *__restrict__ part) {
  extern __shared__ __align__(16) double vsm[];  // [stage][A | B][kVKs][kVLd]
  const int J = blockIdx.x, I = blockIdx.y, zi = blockIdx.z / nsplit, sp = blockIdx.z % nsplit;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t tile = (size_t)kBatch * kBlockF;
  // first step: the split's first batch with both blocks significant
  long lb = b0 + sp - nsplit;
  int lk = kBatch / kVKs - 1;
  vstep_next(mask, mask_words, b1, nsplit, I, J, lb, lk);
  if (lb >= b1 && nsplit == 1) return;
  long cb = lb;
  int ck = lk;
  auto issue = [&](int st) {
    if (lb < b1) {
      const uint32_t *m = mask + lb * mask_words;
      const long qb = pair_off[lb] - p0;
      const double *A = phiT + (size_t)(qb + block_pos(m, I)) * phi_stride_tiles * tile + (size_t)lk * kVKs * kBlockF;
      const double *B = zT + ((size_t)(qb + block_pos(m, J)) * z_stride + zi) * tile + (size_t)lk * kVKs * kBlockF;
      double *dA = vsm + st * kVStageDoubles, *dB = dA + kVKs * kVLd;
#pragma unroll
      for (int r = 0; r < (kVKs * kBlockF / 2) / 256; ++r) {
        const int e = 2 * (threadIdx.x + 256 * r), d = (e / kBlockF) * kVLd + e % kBlockF;
        cp_async16(dA + d, A + e);
        cp_async16(dB + d, B + e);
      }
      vstep_next(mask, mask_words, b1, nsplit, I, J, lb, lk);
    }
    cp_async_commit();  // an empty group past the end keeps the group count uniform
  };
#pragma unroll
  for (int st = 0; st < kVStages - 1; ++st) issue(st);
  constexpr int NI = 2 * SL, NJ = SL;
  double acc[NI][NJ][2];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  // fragment rows 8 i + fr of the warp's part; eight rows are 32 / SL positions
  const int fr = lane >> 2, fk = lane & 3, r0 = vtile_pos<SL>(16 * SL * (warp & 1) + fr),
            c0 = vtile_pos<SL>(8 * SL * (warp >> 1) + fr);
  constexpr int kStep = SL == 4 ? 8 : 32 / SL;
  for (int it = 0; cb < b1; ++it) {
    cp_async_wait<kVStages - 2>();
    __syncthreads();  // step it is visible; the stage refilled below was read in step it - 1
    issue((it + kVStages - 1) % kVStages);
    const double *As = vsm + (it % kVStages) * kVStageDoubles, *Bs = As + kVKs * kVLd;
#pragma unroll
    for (int k = 0; k < kVKs; k += 4) {
      double a[NI], bb[NJ];
#pragma unroll
      for (int i = 0; i < NI; ++i) a[i] = As[(k + fk) * kVLd + r0 + kStep * i];
#pragma unroll
      for (int j = 0; j < NJ; ++j) bb[j] = Bs[(k + fk) * kVLd + c0 + kStep * j];
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma884(acc[i][j], a[i], bb[j]);
    }
    vstep_next(mask, mask_words, b1, nsplit, I, J, cb, ck);
  }
  cp_async_wait<0>();
  if (nsplit > 1) {
    double *o = part + ((((size_t)zi * gridDim.y + I) * gridDim.x + J) * nsplit + sp) * 4 * SL * SL * 256 + threadIdx.x;
#pragma unroll
    for (int e = 0; e < 4 * SL * SL; ++e) o[e * 256] = acc[e / (2 * SL)][(e >> 1) % SL][e & 1];
    return;
  }
  double *Vz = V + (size_t)zi * nbf_pad * nbf_pad;
#pragma unroll
  for (int e = 0; e < 4 * SL * SL; ++e) {
    int r, c;
    vtile_element<SL>(threadIdx.x, e, r, c);
    Vz[(size_t)I * 128 + r + ((size_t)J * 128 + c) * nbf_pad] += acc[e / (2 * SL)][(e >> 1) % SL][e & 1];
  }
}

// Vbar += the parts of a split vgemm_fp64_kernel, in split order: block
// (tile, element e of every thread), one output element per thread
template <int SL>
__global__ void __launch_bounds__(256) vpart_reduce_kernel(const double *__restrict__ part, int nsplit, int nblk,
                                                           int nbf_pad, double *__restrict__ V) {
  const int t = blockIdx.x, J = t % nblk, I = (t / nblk) % nblk, zi = t / (nblk * nblk);
  const double *p = part + (size_t)t * nsplit * 4 * SL * SL * 256 + threadIdx.x;
  double *Vz = V + (size_t)zi * nbf_pad * nbf_pad;
  const int e = blockIdx.y;
  double s = 0.0;
#pragma unroll 8
  for (int k = 0; k < nsplit; ++k) s += p[((size_t)k * 4 * SL * SL + e) * 256];
  int r, c;
  vtile_element<SL>(threadIdx.x, e, r, c);
  Vz[(size_t)I * 128 + r + ((size_t)J * 128 + c) * nbf_pad] += s;
}

// out(i, j) = Vp(pi, pj) + Vp(pj, pi), p = finv[.] the plan position of
// caller function i (symmetrise, unpad and undo the plan order)
// Plan-order density of one spin (blockIdx.y) -> caller order: rho and the
// gradient are written, or added to the output with accumulate (the
// "accumulated into" contract of compute_density_and_sigma_sparse,
// nukexc/density.hpp:257-260); sigma = |grad rho|^2 of the resulting
// gradient.  Output planes are npts long: rho[s], grad[3 s + d], sigma[s].
__global__ void density_out_kernel(long npts, long npad, const long *__restrict__ perm, const double *__restrict__ rho,
                                   const double *__restrict__ grad, int accumulate, double *__restrict__ orho,
                                   double *__restrict__ ograd, double *__restrict__ osigma) {
  const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int s = blockIdx.y;
  if (p >= npts) return;
  const long g = perm[p];
  if (orho) {
    const double v = rho[(size_t)s * npad + p];
    orho[(size_t)s * npts + g] = accumulate ? orho[(size_t)s * npts + g] + v : v;
  }
  if (ograd || osigma) {
    double sg = 0.0;
    for (int d = 0; d < 3; ++d) {
      double v = grad[((size_t)s * 3 + d) * npad + p];
      if (ograd) {
        const size_t o = ((size_t)s * 3 + d) * npts + g;
        if (accumulate) v += ograd[o];
        ograd[o] = v;
      }
      sg += v * v;
    }
    if (osigma) osigma[(size_t)s * npts + g] = sg;
  }
}

__global__ void symmetrize_unpad_kernel(int n, int npad, const int *__restrict__ finv, const double *__restrict__ Vp,
                                        double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i < n && j < n) {
    const size_t pi = finv[i], pj = finv[j];
    out[(size_t)i + (size_t)j * n] = Vp[pi + pj * npad] + Vp[pj + pi * npad];
  }
}

// C (nbf x nocc column-major, per spin) -> Ct[spin][i][p] = C(fperm[p], i)
// in plan order, zero at padding positions (fperm < 0)
// Orbitals into plan order; a non-finite coefficient or occupation raises
// nonfinite[0] (the build then returns NKX_ERR_NUMERIC).
__global__ void pack_orbitals_kernel(const double *__restrict__ C, const double *__restrict__ occ,
                                     const int *__restrict__ fperm, int nbf, int nocc, int nspin, int nbf_pad,
                                     double *__restrict__ Ct, int *nonfinite) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const long tot = (long)nspin * nocc * nbf_pad;
  if (e >= tot) return;
  const int f = fperm[e % nbf_pad];
  const long si = e / nbf_pad;
  const double c = f >= 0 ? C[si * nbf + f] : 0.0;
  Ct[e] = c;
  bool bad = !isfinite(c);
  if (e < (long)nspin * nocc) bad = bad || !isfinite(occ[e]);
  if (bad) atomicOr(nonfinite, 1);
}

// y[slice][a] = sum over a slice of points of w_g rho_g V_a(g) for the functions of
// one aux shell: the radial factor once per point, then C S_lm per m
// (coulomb.hpp:84-85).  Every thread of a block works on the same shell, so
// the solid-harmonic branch is uniform.
__global__ void aux_y_shell_kernel(const AuxShell *__restrict__ shells, const int *__restrict__ list,
                                   const double *__restrict__ px, const double *__restrict__ py,
                                   const double *__restrict__ pz, const double *__restrict__ w,
                                   const double *__restrict__ rho, int nspin, long npad, long slice,
                                   const float *__restrict__ rtab, int naux, double *__restrict__ y) {
  const int shell = list[blockIdx.x];
  const AuxShell sh = shells[shell];
  const AuxFunc &f = sh.f;
  const long g0 = blockIdx.y * slice, g1 = min(npad, g0 + slice);
  double acc[15];
#pragma unroll
  for (int k = 0; k < 15; ++k) acc[k] = 0.0;
  for (long g = g0 + threadIdx.x; g < g1; g += blockDim.x) {
    double r = rho[g];
    if (nspin == 2) r += rho[npad + g];
    const double wr = w[g] * r;
    if (wr == 0.0) continue;
    const double dx = px[g] - f.cx, dy = py[g] - f.cy, dz = pz[g] - f.cz;
    const double wI =
        wr * (rtab ? (double)rtab[(size_t)shell * npad + g] : f.C * aux_radial(f, sqrt(dx * dx + dy * dy + dz * dz)));
#pragma unroll
    for (int k = 0; k < 15; ++k)
      if (k < sh.nm) acc[k] += wI * solid_harmonic(f.l, f.m + k, dx, dy, dz);
  }
  __shared__ double red[32];
  for (int k = 0; k < sh.nm; ++k) {
    double s = acc[0];
#pragma unroll
    for (int q = 1; q < 15; ++q)
      if (q == k) s = acc[q];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
      s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (threadIdx.x == 0) y[(size_t)blockIdx.y * naux + sh.first + k] = s;
    }
  }
}

// y over the functions of one (centre, l) group of complete shells: per
// point one distance, one set of 2L+1 solid harmonics, then the radial factor
// of each shell (coulomb.hpp:84-85).
// FP32 table of the aux shells' scaled radial factors C R(shell, g), with
// R = I(|r_g - A|) the factor aux_radial evaluates (V_a = C S_lm R), one row
// of npad points per shell.  It depends on the geometry only, so the mixed-precision build
// computes it once per plan and both J passes read it instead of
// re-evaluating the incomplete gamma functions: the grid RI-J's 3-index
// contractions in mixed precision (FP32 operands, FP64 accumulation).
__global__ void aux_rtab_kernel(const AuxShell *__restrict__ shells, int nshell, const double *__restrict__ px,
                                const double *__restrict__ py, const double *__restrict__ pz, long npad,
                                float *__restrict__ rtab) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int sh = blockIdx.y;
  if (g >= npad || sh >= nshell) return;
  const AuxFunc &f = shells[sh].f;
  const double dx = px[g] - f.cx, dy = py[g] - f.cy, dz = pz[g] - f.cz;
  rtab[(size_t)sh * npad + g] = (float)(f.C * aux_radial(f, sqrt(dx * dx + dy * dy + dz * dz)));
}

// TAB: C R from the mixed build's table (no distance powers or radial
// factors evaluated here); QM: the most shells the group may have
template <int L, int QM, bool TAB>
__device__ __forceinline__ void aux_y_group(const AuxGroup &G, const AuxShell *__restrict__ shells,
                                   const double *__restrict__ px, const double *__restrict__ py,
                                   const double *__restrict__ pz, const double *__restrict__ w,
                                   const double *__restrict__ rho, int nspin, long npad, long slice,
                                   const float *__restrict__ rtab, int naux, int sl, double *__restrict__ y,
                                   double (*red)[36]) {
  constexpr int NM = 2 * L + 1;
  const long g0 = sl * slice, g1 = min(npad, g0 + slice);
  double acc[QM][NM];
#pragma unroll
  for (int q = 0; q < QM; ++q)
#pragma unroll
    for (int m = 0; m < NM; ++m) acc[q][m] = 0.0;
  if constexpr (TAB) {
    // two points per thread and iteration, every table load of both issued
    // before use (fixed-count shell loop, loads predicated on the group's
    // size): the loop is load-latency bound otherwise
    const float *tab = rtab + (size_t)G.first * npad;
    for (long ga = g0 + threadIdx.x; ga < g1; ga += 2 * blockDim.x) {
      const long gb = ga + blockDim.x;
      const bool hb = gb < g1;
      double wr[2], S[2][NM];
      float t[2][QM];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const long g = k ? (hb ? gb : ga) : ga;
        double r = rho[g];
        if (nspin == 2) r += rho[npad + g];
        wr[k] = (k == 0 || hb) ? w[g] * r : 0.0;
#pragma unroll
        for (int q = 0; q < QM; ++q) t[k][q] = q < G.n ? tab[(size_t)q * npad + g] : 0.0f;
        solid_harmonics_all<L>(px[g] - G.cx, py[g] - G.cy, pz[g] - G.cz, S[k]);
      }
#pragma unroll
      for (int q = 0; q < QM; ++q) {
        const double wa = wr[0] * (double)t[0][q], wb = wr[1] * (double)t[1][q];
#pragma unroll
        for (int m = 0; m < NM; ++m) acc[q][m] = fma(wb, S[1][m], fma(wa, S[0][m], acc[q][m]));
      }
    }
  } else {
  for (long g = g0 + threadIdx.x; g < g1; g += blockDim.x) {
    double r = rho[g];
    if (nspin == 2) r += rho[npad + g];
    const double wr = w[g] * r;
    if (wr == 0.0) continue;
    const double dx = px[g] - G.cx, dy = py[g] - G.cy, dz = pz[g] - G.cz;
    double S[NM];
    solid_harmonics_all<L>(dx, dy, dz, S);
    {
      const double rr = sqrt(dx * dx + dy * dy + dz * dz);
      const double r2l1inv = rr < 1e-12 ? 0.0 : ipow_c<2 * L + 1>(1.0 / rr);
#pragma unroll
      for (int q = 0; q < QM; ++q) {
        if (q >= G.n) break;
        const AuxFunc &f = shells[G.first + q].f;
        const double wI = wr * (f.C * aux_radial_r(f, rr, r2l1inv));
#pragma unroll
        for (int m = 0; m < NM; ++m) acc[q][m] = fma(wI, S[m], acc[q][m]);
      }
    }
  }
  }
  // every sum over its warp first, then all of them over the warps behind
  // one barrier (two barriers a sum took most of a short slice's time)
#pragma unroll
  for (int q = 0; q < QM; ++q) {
    if (q >= G.n) break;
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      double s = acc[q][m];
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q * NM + m] = s;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < G.n * NM; e += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w][e];
    y[(size_t)sl * naux + shells[G.first + e / NM].first + e % NM] = s;
  }
}

// every group of every l in one launch (a block per group and slice): with few centres
// the launches of single l leave most SMs idle (one water, FP64: 149 us in
// four launches; (H2O)_8, tables: 790 and 707, 324 with the harmonics chosen at
// compile time).  Block order: l, slice, group, so that the blocks on the chip read
// the same points and run the same code.  With the tables the fixed-count shell loops
// come in quarters of the l's largest group, so that a group of 6 s shells does not
// pay for 16; without, a loop ends with its group, and one loop an l is all that the
// instruction caches hold beside the incomplete gamma functions (J of an FP64
// build, ms, with quarters and the groups fastest; with the order only; now):
//   143 functions, one water    0.30   0.27   0.26
//   1144, (H2O)_8               7.8    5.3    4.7
//   4576, (H2O)_32              98     62     53
template <bool TAB>
__global__ void __launch_bounds__(256, TAB ? 2 : 1)
    aux_y_groups_kernel(const AuxGroup *__restrict__ groups, int4 goff, const AuxShell *__restrict__ shells,
                        const double *__restrict__ px, const double *__restrict__ py, const double *__restrict__ pz,
                        const double *__restrict__ w, const double *__restrict__ rho, int nspin, long npad, long slice,
                        const float *__restrict__ rtab, int naux, int nsl, double *__restrict__ y) {
  __shared__ double red[8][36];
  // block -> l (groups [o0, o1)), then slice, then group
  const int b = blockIdx.x / nsl, o0 = b < goff.x ? 0 : b < goff.y ? goff.x : b < goff.z ? goff.y : goff.z,
            o1 = b < goff.x ? goff.x : b < goff.y ? goff.y : b < goff.z ? goff.z : goff.w,
            r = blockIdx.x - o0 * nsl, sl = r / (o1 - o0);
  const AuxGroup G = groups[o0 + r % (o1 - o0)];
  auto go = [&](auto l) {
    constexpr int L = decltype(l)::value, QM = aux_group_max(L);
    if constexpr (TAB) {
      const int quarter = (4 * G.n + QM - 1) / QM;
      if (quarter <= 1)
        aux_y_group<L, (QM + 3) / 4, TAB>(G, shells, px, py, pz, w, rho, nspin, npad, slice, rtab, naux, sl, y, red);
      else if (quarter == 2)
        aux_y_group<L, (2 * QM + 3) / 4, TAB>(G, shells, px, py, pz, w, rho, nspin, npad, slice, rtab, naux, sl, y, red);
      else if (quarter == 3)
        aux_y_group<L, (3 * QM + 3) / 4, TAB>(G, shells, px, py, pz, w, rho, nspin, npad, slice, rtab, naux, sl, y, red);
      else
        aux_y_group<L, QM, TAB>(G, shells, px, py, pz, w, rho, nspin, npad, slice, rtab, naux, sl, y, red);
    } else {
      aux_y_group<L, QM, TAB>(G, shells, px, py, pz, w, rho, nspin, npad, slice, rtab, naux, sl, y, red);
    }
  };
  switch (G.l) {
    case 0: return go(std::integral_constant<int, 0>{});
    case 1: return go(std::integral_constant<int, 1>{});
    case 2: return go(std::integral_constant<int, 2>{});
    default: return go(std::integral_constant<int, 3>{});
  }
}

template <int L>
__device__ __forceinline__ double aux_group_v(const AuxGroup &G, const AuxShell *__restrict__ shells,
                                              const double *__restrict__ c, double x, double y, double z) {
  constexpr int NM = 2 * L + 1;
  const double dx = x - G.cx, dy = y - G.cy, dz = z - G.cz;
  double S[NM];
  solid_harmonics_all<L>(dx, dy, dz, S);
  double s = 0.0;
  const double rr = sqrt(dx * dx + dy * dy + dz * dz);
  const double r2l1inv = rr < 1e-12 ? 0.0 : ipow_c<2 * L + 1>(1.0 / rr);
  for (int q = 0; q < G.n; ++q) {
    const AuxShell &sh = shells[G.first + q];
    double a = 0.0;
#pragma unroll
    for (int m = 0; m < NM; ++m) a += c[sh.first + m] * (sh.f.C * S[m]);
    if (a != 0.0) s += a * aux_radial_r(sh.f, rr, r2l1inv);
  }
  return s;
}

// y_a = the sum of its slices' shares, in a fixed order (the fit amplifies
// rounding differences of y, so the sum must not depend on scheduling)
__global__ void __launch_bounds__(256) aux_y_reduce_kernel(const double *__restrict__ part, int nsl, int naux,
                                                           double *__restrict__ y) {
  const int a = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;  // a warp per function
  if (a >= naux) return;
  double s = 0.0;
  for (int k = lane; k < nsl; k += 32) s += part[(size_t)k * naux + a];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) y[a] = s;
}

// v_g = w_g sum_a c_a V_a(g) over the groups; aux_v_loose_kernel adds the loose
// shells (coulomb.hpp:90-95)
// v of two points (ga, gb) from one group with the C R table: the group's
// data and the fit coefficients are loaded once for both
template <int L>
__device__ __forceinline__ void aux_group_v2_tab(const AuxGroup &G, const AuxShell *__restrict__ shells,
                                                 const double *__restrict__ c, const double (&x)[2],
                                                 const double (&y)[2], const double (&z)[2],
                                                 const float *__restrict__ rtab, long npad, long ga, long gb,
                                                 double (&s)[2]) {
  constexpr int NM = 2 * L + 1;
  double S[2][NM];
  solid_harmonics_all<L>(x[0] - G.cx, y[0] - G.cy, z[0] - G.cz, S[0]);
  solid_harmonics_all<L>(x[1] - G.cx, y[1] - G.cy, z[1] - G.cz, S[1]);
#pragma unroll 2
  for (int q = 0; q < G.n; ++q) {
    const int f0 = shells[G.first + q].first;
    const float *row = rtab + (size_t)(G.first + q) * npad;
    const double ra = (double)row[ga], rb = (double)row[gb];
    double a0 = 0.0, a1 = 0.0;
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      const double cm = c[f0 + m];
      a0 = fma(cm, S[0][m], a0);
      a1 = fma(cm, S[1][m], a1);
    }
    s[0] = fma(a0, ra, s[0]);
    s[1] = fma(a1, rb, s[1]);
  }
}

// the table form of aux_v_group_kernel: two points per thread.  ((H2O)_8, 1144
// functions: 672 us with the harmonics' switch in the loops, 500 now)
__global__ void __launch_bounds__(256, 3)
    aux_v_group_tab_kernel(const AuxGroup *__restrict__ groups, int4 goff,
                           const AuxShell *__restrict__ shells,
                           const double *__restrict__ c, const double *__restrict__ px,
                           const double *__restrict__ py, const double *__restrict__ pz,
                           const double *__restrict__ w, long npad, const float *__restrict__ rtab,
                           double *__restrict__ v) {
  const long ga = blockIdx.x * 2L * blockDim.x + threadIdx.x;
  if (ga >= npad) return;
  const long gb = min(ga + (long)blockDim.x, npad - 1);  // a duplicate of the last point when past the end
  const double x[2] = {px[ga], px[gb]}, y[2] = {py[ga], py[gb]}, z[2] = {pz[ga], pz[gb]};
  double s[2] = {0.0, 0.0};
#pragma unroll 1
  for (int k = 0; k < goff.x; ++k) aux_group_v2_tab<0>(groups[k], shells, c, x, y, z, rtab, npad, ga, gb, s);
#pragma unroll 1
  for (int k = goff.x; k < goff.y; ++k) aux_group_v2_tab<1>(groups[k], shells, c, x, y, z, rtab, npad, ga, gb, s);
#pragma unroll 1
  for (int k = goff.y; k < goff.z; ++k) aux_group_v2_tab<2>(groups[k], shells, c, x, y, z, rtab, npad, ga, gb, s);
#pragma unroll 1
  for (int k = goff.z; k < goff.w; ++k) aux_group_v2_tab<3>(groups[k], shells, c, x, y, z, rtab, npad, ga, gb, s);
  v[ga] = s[0] * w[ga];
  if (ga + (long)blockDim.x < npad) v[gb] = s[1] * w[gb];
}

__global__ void __launch_bounds__(128, 6)
    aux_v_group_kernel(const AuxGroup *__restrict__ groups, int4 goff,
                       const AuxShell *__restrict__ shells,
                       const double *__restrict__ c, const double *__restrict__ px,
                       const double *__restrict__ py, const double *__restrict__ pz,
                       const double *__restrict__ w, long npad, double *__restrict__ v) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= npad) return;
  if (w[g] == 0.0) {
    v[g] = 0.0;
    return;
  }
  const double x = px[g], y = py[g], z = pz[g];
  double s = 0.0;
  // groups sorted by l: [0, goff.x) l = 0, [goff.x, goff.y) l = 1, ...
#pragma unroll 1
  for (int k = 0; k < goff.x; ++k) s += aux_group_v<0>(groups[k], shells, c, x, y, z);
#pragma unroll 1
  for (int k = goff.x; k < goff.y; ++k) s += aux_group_v<1>(groups[k], shells, c, x, y, z);
#pragma unroll 1
  for (int k = goff.y; k < goff.z; ++k) s += aux_group_v<2>(groups[k], shells, c, x, y, z);
#pragma unroll 1
  for (int k = goff.z; k < goff.w; ++k) s += aux_group_v<3>(groups[k], shells, c, x, y, z);
  v[g] = s * w[g];
}

// The loose shells (l > 3, parts of a shell) are added to v by a kernel of their own,
// so that the switch over all harmonics takes no registers from the groups' loops;
// opaque coordinates keep it from forming the products of all harmonics for each
// shell ((H2O)_4, 1296 functions in random order: 21.5 ms in FP64 and 17.6 with the
// table where it does, 4.9 and 2.7 now).  rtab: C R from the mixed build's table.
template <bool TAB>
__global__ void aux_v_loose_kernel(const AuxShell *__restrict__ shells, const int *__restrict__ loose, int nloose,
                                   const double *__restrict__ c, const double *__restrict__ px,
                                   const double *__restrict__ py, const double *__restrict__ pz,
                                   const double *__restrict__ w, long npad, const float *__restrict__ rtab,
                                   double *__restrict__ v) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= npad || w[g] == 0.0) return;
  const double x = px[g], y = py[g], z = pz[g];
  double s = 0.0;
  for (int k = 0; k < nloose; ++k) {
    const AuxShell &sh = shells[loose[k]];
    const AuxFunc &f = sh.f;
    const double dx = x - f.cx, dy = y - f.cy, dz = z - f.cz;
    double a = 0.0;
#pragma unroll 1
    for (int m = 0; m < sh.nm; ++m) {
      double hx = dx, hy = dy, hz = dz;
      opaque(hx, hy, hz);
      a += c[sh.first + m] * solid_harmonic(f.l, f.m + m, hx, hy, hz);
    }
    if (a != 0.0)
      s += a * (TAB ? (double)rtab[(size_t)loose[k] * npad + g] : f.C * aux_radial(f, sqrt(dx * dx + dy * dy + dz * dz)));
  }
  v[g] += s * w[g];
}

// Aux collocation phi_A(g) and weighted potential Vw_B(g) of a slice of
// points, column-major naux x np (metric (A|B) set-up, standalone.cxx:443-461)
__global__ void aux_tables_kernel(const StoFunc *__restrict__ sto, const AuxFunc *__restrict__ aux, int naux,
                                  const double *__restrict__ px, const double *__restrict__ py,
                                  const double *__restrict__ pz, const double *__restrict__ w, long g0, long np,
                                  double *__restrict__ phi, double *__restrict__ vw) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= (long)naux * np) return;
  const int a = (int)(e % naux);
  const long g = g0 + e / naux;
  phi[e] = sto_value(sto[a], px[g], py[g], pz[g]);
  vw[e] = aux_potential(aux[a], px[g], py[g], pz[g]) * w[g];
}

// interleaved points xyz[3n] -> planes x[n], y[n], z[n]
__global__ void split_points_kernel(long n, const double *__restrict__ xyz, double *__restrict__ soa) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= n) return;
  for (int d = 0; d < 3; ++d) soa[(size_t)d * n + g] = xyz[3 * g + d];
}

__global__ void gather_kernel(int K, const int *__restrict__ piv, const double *__restrict__ y, double *__restrict__ t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < K) t[i] = y[piv[i]];
}
__global__ void scatter_kernel(int K, const int *__restrict__ piv, const double *__restrict__ t, double *__restrict__ c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < K) c[piv[i]] = t[i];
}

__global__ void sym_half_kernel(int n, double *S) {
  const int i = blockIdx.y * blockDim.y + threadIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && j < n && i < j) {
    const double v = 0.5 * (S[(size_t)i + (size_t)j * n] + S[(size_t)j + (size_t)i * n]);
    S[(size_t)i + (size_t)j * n] = v;
    S[(size_t)j + (size_t)i * n] = v;
  }
}

// (A|B) = (M + M^T) / 2 with M_AB = sum_g phi_A(g) w_g V_B(g): the grid
// Coulomb metric of coulomb_overlap_integral(_sparse/_tiled)
// (nukexc/coulomb.hpp:691-813, :827-958), FP64 GEMMs over point slices of at
// most 256 MB of tables; S is naux x naux, column-major, on the device.
static void grid_metric(const StoFunc *d_asto, const AuxFunc *d_aux, int naux, const double *px, const double *py,
                        const double *pz, const double *w, long n, cublasHandle_t hb, cudaStream_t s, double *S) {
  const size_t NA = naux;
  const long slice = std::max<long>(kBatch, std::min<long>(n, (long)((size_t)1 << 28) / (16 * NA)));
  double *sphi = dalloc<double>(NA * slice), *svw = dalloc<double>(NA * slice);
  NKX_CUDA(cudaMemsetAsync(S, 0, sizeof(double) * NA * NA, s));
  for (long g0 = 0; g0 < n; g0 += slice) {
    const long np = std::min(slice, n - g0);
    aux_tables_kernel<<<nblk(NA * np, 128), 128, 0, s>>>(d_asto, d_aux, naux, px, py, pz, w, g0, np, sphi, svw);
    NKX_LAUNCH_CHECK();
    const double one = 1.0;
    NKX_REQUIRE(cublasDgemm(hb, CUBLAS_OP_N, CUBLAS_OP_T, naux, naux, (int)np, &one, sphi, naux, svw, naux, &one, S,
                            naux) == CUBLAS_STATUS_SUCCESS,
                NKX_ERR_CUDA, "cublasDgemm failed");
  }
  dim3 tb(16, 16), gb(nblk(naux, 16), nblk(naux, 16));
  sym_half_kernel<<<gb, tb, 0, s>>>(naux, S);
  NKX_LAUNCH_CHECK();
  NKX_CUDA(cudaStreamSynchronize(s));
  cudaFree(sphi);
  cudaFree(svw);
}

// ========================================================= plan set-up ==

static uint64_t spread3(uint64_t v) {
  v &= 0x1fffff;
  v = (v | v << 32) & 0x1f00000000ffffULL;
  v = (v | v << 16) & 0x1f0000ff0000ffULL;
  v = (v | v << 8) & 0x100f00f00f00f00fULL;
  v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
  v = (v | v << 2) & 0x1249249249249249ULL;
  return v;
}

// Morton (Z-order) permutation of n points xyz[3n]: 21-bit codes per axis
// over the points' bounding box, ties kept in input order.  perm[k] is the
// input index of the k-th point in the order (the space-filling-curve
// permutation of create_bounding_boxes, nukexc/octree.hpp:85-104).
static void morton_order(long n, const double *xyz, std::vector<long> &perm) {
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (long g = 0; g < n; ++g)
    for (int d = 0; d < 3; ++d) {
      lo[d] = std::min(lo[d], xyz[3 * g + d]);
      hi[d] = std::max(hi[d], xyz[3 * g + d]);
    }
  // (code, index) pairs sorted lexicographically: the stable Morton order
  std::vector<std::pair<uint64_t, long>> key(n);
#pragma omp parallel for schedule(static)
  for (long g = 0; g < n; ++g) {
    uint64_t c = 0;
    for (int d = 0; d < 3; ++d) {
      const double span = hi[d] > lo[d] ? hi[d] - lo[d] : 1.0;
      const double u = (xyz[3 * g + d] - lo[d]) / span;
      c |= spread3((uint64_t)std::min(2097151.0, std::max(0.0, u * 2097151.0))) << d;
    }
    key[g] = {c, g};
  }
  __gnu_parallel::sort(key.begin(), key.end());
  perm.resize(n);
  for (long g = 0; g < n; ++g) perm[g] = key[g].second;
}

void destroy_mixed_state(void *p);

// A plan's place for a build's result in page-locked memory.  One block of 1 KB
// serves the first 64 plans alive at a time (to page-lock memory takes 1.2 to 3
// ms, an eighth of a small plan's creation; a copy to pageable memory costs
// each build 7 us); it stays until the process ends.  take: a free place, or
// nullptr; else `r` is given back.
static Plan::Result *result_slot(bool take, Plan::Result *r) {
  static std::mutex mu;
  static Plan::Result *block = nullptr;
  static uint64_t used = 0;
  std::lock_guard<std::mutex> lock(mu);
  if (!take) {
    if (block && r >= block && r < block + 64) used &= ~(1ull << (r - block));
    return nullptr;
  }
  if (!block && cudaHostAlloc(&block, 64 * sizeof(Plan::Result), cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    block = nullptr;
  }
  if (!block || used == ~0ull) return nullptr;
  const int k = __builtin_ctzll(~used);
  used |= 1ull << k;
  return block + k;
}

Plan::~Plan() {
  for (BuildGraph &g : graphs)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  if (mx_state) destroy_mixed_state(mx_state);
  if (grad_state) destroy_grad_state(grad_state);
  for (void *p : allocs) cudaFree(p);
  if (cublas) cublasDestroy((cublasHandle_t)cublas);
  if (cusolver) cusolverDnDestroy((cusolverDnHandle_t)cusolver);
  for (auto &e : ev) cudaEventDestroy(e);
  for (auto &e : ev_pool) cudaEventDestroy(e);
  result_slot(false, h_result);
  if (stream) cudaStreamDestroy(stream);
}

template <class T>
T *Plan::alloc(size_t n) {
  T *p = dalloc<T>(n);
  if (p) allocs.push_back(p);
  return p;
}

// Factor of the Coulomb metric held in P.h_metric (naux x naux, column-major,
// symmetrised): the reference's preconditioned half inverse when the plan
// was created with metric_svd_thr > 0, else a pivoted Cholesky of the
// Jacobi-preconditioned metric.  Used at plan creation and by
// nkx_plan_set_metric (the full-grid metric of a grid sharded over ranks).
static void factor_metric(Plan &P) {
  const size_t NA = P.naux;
  NKX_CUDA(cudaMemcpy(P.d_L, P.h_metric.data(), sizeof(double) * NA * NA, cudaMemcpyHostToDevice));
  if (P.svd_mode) {
    // the reference's preconditioned half inverse: c = X X^T y
    int K = 0;
    NKX_REQUIRE(nkx_half_inverse(P.naux, P.d_L, P.metric_svd_thr, P.d_X, &K, P.stream) == NKX_OK,
                NKX_ERR_NUMERIC, "half inverse of the metric failed");
    P.K = K;
    P.metric_min_diag = 0.0;
  } else {
    // Pivoted Cholesky of the Jacobi-preconditioned metric A = D^-1 S D^-1:
    // the grid-integrated (A|B) of an even-tempered aux set is indefinite
    // at the 1e-4 level (diffuse functions reach past the grid), so aux
    // functions whose remaining diagonal falls below kMetricTol are
    // dropped (their fit coefficient is 0) and the kept block is factorised.
    const double kMetricTol = 1e-5;
    std::vector<double> D(NA), A(NA * NA);
    for (size_t i = 0; i < NA; ++i) D[i] = std::sqrt(P.h_metric[i + i * NA]);
    for (size_t j = 0; j < NA; ++j)
      for (size_t i = 0; i < NA; ++i) A[i * NA + j] = P.h_metric[i + j * NA] / (D[i] * D[j]);
    std::vector<double> Lr(NA * NA, 0.0), d(NA);  // row-major rows of L
    std::vector<char> used(NA, 0);
    for (size_t i = 0; i < NA; ++i) d[i] = A[i * NA + i];
    std::vector<int> piv;
    for (size_t k = 0; k < NA; ++k) {
      long p = -1;
      double best = kMetricTol;
      for (size_t i = 0; i < NA; ++i)
        if (!used[i] && d[i] >= best) {
          best = d[i];
          p = (long)i;
        }
      if (p < 0) break;
      used[p] = 1;
      piv.push_back((int)p);
      const double sq = std::sqrt(d[p]);
      const double *lp = &Lr[(size_t)p * NA];
#pragma omp parallel for schedule(static)
      for (long i = 0; i < (long)NA; ++i) {
        if (used[i] && i != p) continue;
        const double *li = &Lr[(size_t)i * NA];
        double acc = A[(size_t)i * NA + p];
        for (size_t c = 0; c < k; ++c) acc -= li[c] * lp[c];
        const double v = acc / sq;
        Lr[(size_t)i * NA + k] = v;
        if (i != p) d[i] -= v * v;
      }
    }
    const int K = (int)piv.size();
    NKX_REQUIRE(K > 0, NKX_ERR_NUMERIC, "aux metric (A|B) has no positive pivot");
    // F = D_sel L_sel, lower triangular K x K in pivot order, column-major
    std::vector<double> F((size_t)K * K, 0.0);
    double mn = 1e300;
    for (int a = 0; a < K; ++a)
      for (int c = 0; c <= a; ++c) F[a + (size_t)c * K] = D[piv[a]] * Lr[(size_t)piv[a] * NA + c];
    for (int a = 0; a < K; ++a) mn = std::min(mn, F[a + (size_t)a * K] / D[piv[a]]);
    P.K = K;
    P.h_piv = piv;
    NKX_CUDA(cudaMemcpy(P.d_L, F.data(), sizeof(double) * K * K, cudaMemcpyHostToDevice));
    NKX_CUDA(cudaMemcpy(P.d_piv, piv.data(), sizeof(int) * K, cudaMemcpyHostToDevice));
    P.metric_min_diag = mn;
  }
}

void Plan::release(void *p) {
  if (!p) return;
  cudaFree(p);
  allocs.erase(std::remove(allocs.begin(), allocs.end(), p), allocs.end());
}

// Device bytes a chunk needs per (batch, block) pair: the FP64 staging of
// four 256 x 128 planes (1 MB) plus the mixed build's int8 digits (1 MB), or
// the FP64 build's three Z planes (0.75 MB).  The default workspace is
// kDefaultWorkspace or a third of the free memory, whichever is smaller.
constexpr size_t kPairBytes = (size_t)2 << 20;
constexpr size_t kDefaultWorkspace = (size_t)24 << 30;

// Chunks of consecutive batches holding at most maxp (batch, block) pairs,
// and the chunk-sized staging: the FP64 planes now; the FP64 build's Z
// planes and the mixed build's digits when a build first needs them.
void plan_chunks(Plan &P, long maxp) {
  P.drop_graphs();
  P.chunks.clear();
  P.max_chunk_pairs = 0;
  long b = 0;
  while (b < P.nbatch) {
    Chunk c;
    c.b0 = b;
    c.p0 = P.h_pair_off[b];
    while (b < P.nbatch && (P.h_pair_off[b + 1] - c.p0 <= maxp || b == c.b0)) ++b;
    c.b1 = b;
    c.p1 = P.h_pair_off[b];
    P.max_chunk_pairs = std::max(P.max_chunk_pairs, c.p1 - c.p0);
    P.chunks.push_back(c);
  }
  P.chunk_pair_limit = maxp;
  // V output tiles of each chunk.  A unit of the V contraction is one
  // (I, J) tile walking the chunk's batches where both blocks are
  // significant; tiles with no such batch get no unit, and the rest are
  // ordered heaviest first (round-robin over the SMs then spreads the heavy
  // tiles evenly).  Ties keep a square-patch order (row blocks in super-rows
  // of about sqrt(SMs)), so that the units running at once share their phi
  // and Z tiles in L2; on a dense problem every tile costs the same and the
  // whole order is the patch order.
  {
    int nsm = 148;
    NKX_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, P.device));
    const int nb = P.nblk, vrow = std::max(1, std::min(nb, (int)std::lround(std::sqrt((double)nsm))));
    NKX_REQUIRE(nb < (1 << 15), NKX_ERR_UNSUPPORTED, "more than 32767 function blocks");
    std::vector<int> patch;
    patch.reserve((size_t)nb * nb);
    for (int r0 = 0; r0 < nb; r0 += vrow)
      for (int J = 0; J < nb; ++J)
        for (int I = r0; I < std::min(nb, r0 + vrow); ++I) patch.push_back(I * nb + J);
    // pair tiles (R, J) of the CTA-pair V contraction: row blocks 2R and
    // 2R + 1 together, costed by the batches where J and either row block
    // are significant, in the same patch order over about sqrt(SMs / 2) row
    // pairs
    const int nr = (nb + 1) / 2, vrow2 = std::max(1, std::min(nr, (int)std::lround(std::sqrt(nsm / 2.0))));
    std::vector<int> patch2;
    patch2.reserve((size_t)nr * nb);
    for (int r0 = 0; r0 < nr; r0 += vrow2)
      for (int J = 0; J < nb; ++J)
        for (int R = r0; R < std::min(nr, r0 + vrow2); ++R) patch2.push_back(R * nb + J);
    std::vector<int> cnt((size_t)nb * nb), cnt2((size_t)nr * nb), blk, rows, tiles, all, all2;
    for (Chunk &c : P.chunks) {
      std::fill(cnt.begin(), cnt.end(), 0);
      std::fill(cnt2.begin(), cnt2.end(), 0);
      for (long b = c.b0; b < c.b1; ++b) {
        blk.clear();
        rows.clear();
        for (int w = 0; w < P.mask_words; ++w)
          for (uint32_t m = P.h_mask[b * P.mask_words + w]; m; m &= m - 1) blk.push_back(32 * w + __builtin_ctz(m));
        for (int I : blk)
          if (rows.empty() || rows.back() != I / 2) rows.push_back(I / 2);  // blk is ascending
        for (int I : blk)
          for (int J : blk) ++cnt[(size_t)I * nb + J];
        for (int R : rows)
          for (int J : blk) ++cnt2[(size_t)R * nb + J];
      }
      tiles.clear();
      for (int t : patch)
        if (cnt[t]) tiles.push_back(t);
      std::stable_sort(tiles.begin(), tiles.end(), [&](int x, int y) { return cnt[x] > cnt[y]; });
      c.t0 = (long)all.size();
      for (int t : tiles) all.push_back(((t / nb) << 16) | (t % nb));
      c.t1 = (long)all.size();
      tiles.clear();
      for (int t : patch2)
        if (cnt2[t]) tiles.push_back(t);
      std::stable_sort(tiles.begin(), tiles.end(), [&](int x, int y) { return cnt2[x] > cnt2[y]; });
      c.u0 = (long)all2.size();
      for (int t : tiles) all2.push_back(((t / nb) << 16) | (t % nb));
      c.u1 = (long)all2.size();
    }
    P.release(P.d_vtiles);
    P.d_vtiles = P.alloc<int>(std::max<size_t>(1, all.size()));
    if (!all.empty())
      NKX_CUDA(cudaMemcpy(P.d_vtiles, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice));
    P.release(P.d_vtiles2);
    P.d_vtiles2 = P.alloc<int>(std::max<size_t>(1, all2.size()));
    if (!all2.empty())
      NKX_CUDA(cudaMemcpy(P.d_vtiles2, all2.data(), sizeof(int) * all2.size(), cudaMemcpyHostToDevice));
  }
  const size_t tile = (size_t)kBatch * kBlockF;
  P.release(P.ws_phi);
  P.release(P.ws_z);
  P.ws_z = nullptr;
  if (P.mx_state) {
    destroy_mixed_state(P.mx_state);
    P.mx_state = nullptr;
  }
  P.ws_phi = P.alloc<double>(std::max<long>(1, P.max_chunk_pairs) * 4 * tile);
}

static double box_distance2(const double *c, const double *lo, const double *hi) {
  double d2 = 0.0;
  for (int d = 0; d < 3; ++d) {
    const double e = c[d] < lo[d] ? lo[d] - c[d] : (c[d] > hi[d] ? c[d] - hi[d] : 0.0);
    d2 += e * e;
  }
  return d2;
}

// Functions of one atom reach very differently far (zeta 0.5 to 26: 46 to 1
// bohr at 1e-10), and a 128-function block is significant where any of its
// functions is, so blocks cut along the Morton order of the centres are
// significant almost everywhere.  This splits the order at a cutoff radius --
// the far-reaching functions first, then the others, each in the given
// order -- or sorts it by radius, if the blocks significant in a sample of
// batches then cost less: V takes n^2 tile products of a batch with n blocks,
// the other passes about kLinear times n ((H2O)_64 PBE: 37 ns a product, 0.87
// us a pair).  Blocks of like reach are screened with radii of a tolerance
// 1e-6 times the caller's, so that no term above FP64 rounding is dropped that
// the mixed blocks would have kept; the gain of three per cent asked for
// counts that.  On a change `order` and the radii `cut` are replaced.
// ((H2O)_64: 24 -> 22.2 blocks a batch, 576 -> 493 products; 624 -> 567 ms per
// build.)
static void group_by_reach(const nkx_basis &prim, double tol, long nbatch, const std::vector<double> &blo,
                           const std::vector<double> &bhi, std::vector<int> &order, std::vector<double> &cut) {
  if (tol < 1e-280) return;
  constexpr double kLinear = 23.0;
  const int nbf = prim.nbf, nblk = (nbf + kBlockF - 1) / kBlockF;
  const auto far = make_cutoffs(prim, 1e-6 * tol);
  const long ns = std::min<long>(nbatch, 256);
  std::vector<char> sig((size_t)ns * nbf), sig0((size_t)ns * nbf);
#pragma omp parallel for schedule(static)
  for (long k = 0; k < ns; ++k) {
    const long b = ns > 1 ? k * (nbatch - 1) / (ns - 1) : 0;
    for (int f = 0; f < nbf; ++f) {
      const double d2 = box_distance2(&prim.center[3 * f], &blo[3 * b], &bhi[3 * b]);
      sig[k * nbf + f] = d2 <= far[f] * far[f];
      sig0[k * nbf + f] = d2 <= cut[f] * cut[f];
    }
  }
  auto cost = [&](const std::vector<int> &o, const std::vector<char> &s) {
    double c = 0.0;
    for (long k = 0; k < ns; ++k) {
      long n = 0;
      for (int I = 0; I < nblk; ++I) {
        bool any = false;
        for (int p = I * kBlockF; p < std::min(nbf, (I + 1) * kBlockF) && !any; ++p) any = s[k * nbf + o[p]];
        n += any;
      }
      c += (double)n * n + kLinear * n;
    }
    return c;
  };
  // the radii that occur, at most 24 of them
  std::vector<double> radii(far);
  std::sort(radii.begin(), radii.end());
  radii.erase(std::unique(radii.begin(), radii.end(), [](double x, double y) { return y - x < 1e-9 * y; }),
              radii.end());
  const long nr = (long)radii.size(), nc = std::min<long>(nr - 1, 24);
  std::vector<std::vector<int>> cand(nc + 1, order);
  for (long i = 0; i < nc; ++i) {
    const double r = radii[i * (nr - 1) / nc] * (1.0 + 1e-8);
    std::stable_partition(cand[i].begin(), cand[i].end(), [&](int f) { return far[f] > r; });
  }
  std::stable_sort(cand[nc].begin(), cand[nc].end(), [&](int x, int y) { return far[x] > far[y]; });
  std::vector<double> costs(nc + 1);
#pragma omp parallel for schedule(dynamic)
  for (long i = 0; i <= nc; ++i) costs[i] = cost(cand[i], sig);
  const long best = std::min_element(costs.begin(), costs.end()) - costs.begin();
  if (costs[best] < 0.97 * cost(order, sig0)) {
    order = cand[best];
    cut = far;
  }
}

static void build_plan(Plan &P, const nkx_molecule *mol, const nkx_basis *prim, const nkx_basis *aux, long npoints,
                       const double *xyz, const double *w, const int *owner, const nkx_plan_options *opts) {
  NKX_REQUIRE(prim && prim->nbf > 0 && npoints > 0 && xyz && w && opts, NKX_ERR_ARG, "invalid arguments");
  NKX_REQUIRE(opts->batch_points == 0 || opts->batch_points == kBatch, NKX_ERR_UNSUPPORTED,
              "batch_points must be 256");
  for (int i = 0; i < prim->nbf; ++i)
    NKX_REQUIRE(prim->l[i] >= 0 && prim->l[i] <= 7 && prim->n[i] > prim->l[i] && abs(prim->m[i]) <= prim->l[i] &&
                    prim->zeta[i] > 0,
                NKX_ERR_UNSUPPORTED, "basis function outside n > l, |m| <= l <= 7, zeta > 0");
  P.xc = make_spec(opts);
  P.gga = spec_is_gga(P.xc);
  NKX_CUDA(cudaGetDevice(&P.device));
  NKX_CUDA(cudaDeviceGetAttribute(&P.nsm, cudaDevAttrMultiProcessorCount, P.device));
  NKX_CUDA(cudaStreamCreateWithFlags(&P.stream, cudaStreamNonBlocking));
  for (auto &e : P.ev) NKX_CUDA(cudaEventCreate(&e));
  P.nbf = prim->nbf;
  P.nblk = (P.nbf + kBlockF - 1) / kBlockF;
  P.nbf_pad = P.nblk * kBlockF;
  P.mask_words = (P.nblk + 31) / 32;
  P.npts = npoints;
  P.nbatch = (npoints + kBatch - 1) / kBatch;
  P.npad = P.nbatch * kBatch;

  // --- Morton order of the points (create_bounding_boxes, octree.hpp:70-110)
  morton_order(npoints, xyz, P.perm);
  std::vector<double> hx(P.npad), hy(P.npad), hz(P.npad), hw(P.npad, 0.0);
  for (long p = 0; p < P.npad; ++p) {
    const long g = P.perm[std::min(p, npoints - 1)];
    hx[p] = xyz[3 * g];
    hy[p] = xyz[3 * g + 1];
    hz[p] = xyz[3 * g + 2];
    if (p < npoints) hw[p] = w[g];
  }

  // --- basis table in plan order (padded positions have norm 0).  Within
  // each 128-function block, position p = 4 lane + c holds the block's
  // function of rank 32 c + lane, ranks sorted by (l, m): the collocation
  // kernels give lane l of a warp positions 4l .. 4l+3, so the 32 lanes
  // evaluating slot c take the same solid-harmonic branch.  Blocks keep
  // their function sets.
  auto tab0 = make_sto_table(*prim);
  // Before that, the functions are grouped by centre (runs of one centre in
  // the caller's order) and the centres put in Morton order of position, so
  // the 128-function blocks are compact in space and screening keeps few
  // blocks per batch even when the caller lists atoms in random order.
  std::vector<int> order(P.nbf);
  {
    struct Run {
      int first, n;
      uint64_t code;
    };
    std::vector<Run> runs;
    auto same_centre = [&](int f, int g) {
      return prim->center[3 * f] == prim->center[3 * g] && prim->center[3 * f + 1] == prim->center[3 * g + 1] &&
             prim->center[3 * f + 2] == prim->center[3 * g + 2];
    };
    for (int f = 0; f < P.nbf; ++f) {
      if (!runs.empty() && same_centre(runs.back().first, f)) {
        ++runs.back().n;
        continue;
      }
      runs.push_back(Run{f, 1, 0});
    }
    double clo[3] = {1e300, 1e300, 1e300}, chi[3] = {-1e300, -1e300, -1e300};
    for (const Run &r : runs)
      for (int d = 0; d < 3; ++d) {
        clo[d] = std::min(clo[d], prim->center[3 * r.first + d]);
        chi[d] = std::max(chi[d], prim->center[3 * r.first + d]);
      }
    for (Run &r : runs) {
      uint64_t c = 0;
      for (int d = 0; d < 3; ++d) {
        const double span = chi[d] > clo[d] ? chi[d] - clo[d] : 1.0;
        const double u = (prim->center[3 * r.first + d] - clo[d]) / span;
        c |= spread3((uint64_t)std::min(2097151.0, std::max(0.0, u * 2097151.0))) << d;
      }
      r.code = c;
    }
    std::stable_sort(runs.begin(), runs.end(), [](const Run &a, const Run &b) { return a.code < b.code; });
    int k = 0;
    for (const Run &r : runs)
      for (int i = 0; i < r.n; ++i) order[k++] = r.first + i;
  }
  const double tol = opts->screen_tol > 0 ? opts->screen_tol : 1e-10;
  auto cut = make_cutoffs(*prim, tol);
  // bounding boxes of the batches
  std::vector<double> blo(3 * (size_t)P.nbatch), bhi(3 * (size_t)P.nbatch);
#pragma omp parallel for schedule(static)
  for (long b = 0; b < P.nbatch; ++b)
    for (int d = 0; d < 3; ++d) {
      const std::vector<double> &h = d == 0 ? hx : d == 1 ? hy : hz;
      // a NaN compares false and stays out of the box, so that its batch is
      // not screened away and the point shows in the build
      double lo = 1e300, hi = -1e300;
      for (long p = b * kBatch; p < (b + 1) * kBatch; ++p) {
        lo = std::min(lo, h[p]);
        hi = std::max(hi, h[p]);
      }
      blo[3 * b + d] = lo;
      bhi[3 * b + d] = hi;
    }
  if (P.nblk > 1) group_by_reach(*prim, tol, P.nbatch, blo, bhi, order, cut);
  std::vector<StoFunc> tab(P.nbf_pad);
  P.h_fperm.assign(P.nbf_pad, -1);
  std::vector<int> finv(std::max(1, P.nbf), 0);
  for (int I = 0; I < P.nblk; ++I) {
    std::vector<int> fs;
    for (int q = I * kBlockF; q < std::min(P.nbf, (I + 1) * kBlockF); ++q) fs.push_back(order[q]);
    std::stable_sort(fs.begin(), fs.end(), [&](int x, int y) {
      return tab0[x].l != tab0[y].l ? tab0[x].l < tab0[y].l : tab0[x].m < tab0[y].m;
    });
    for (int k = 0; k < (int)fs.size(); ++k) {
      const int pos = I * kBlockF + 4 * (k % 32) + k / 32;
      P.h_fperm[pos] = fs[k];
      finv[fs[k]] = pos;
    }
  }
  for (int p = 0; p < P.nbf_pad; ++p) {
    if (P.h_fperm[p] >= 0) {
      tab[p] = tab0[P.h_fperm[p]];
    } else {
      tab[p] = tab0[0];
      tab[p].norm = 0.0;
    }
  }
  // --- atoms, point owners (plan order) and the atom of every function, for
  // the nuclear gradient; functions whose centre is on no atom get -1
  if (mol && mol->natoms > 0 && mol->xyz) {
    P.natoms = mol->natoms;
    P.h_centers.assign(mol->xyz, mol->xyz + 3 * (size_t)mol->natoms);
    P.d_centers = P.alloc<double>(3 * (size_t)P.natoms);
    NKX_CUDA(cudaMemcpy(P.d_centers, P.h_centers.data(), sizeof(double) * 3 * P.natoms, cudaMemcpyHostToDevice));

    std::vector<int> fatom(P.nbf_pad, 0);
    P.all_funcs_on_atoms = true;
    for (int q = 0; q < P.nbf_pad; ++q) {
      const int f = P.h_fperm[q];
      if (f < 0) continue;
      int best = -1;
      for (int a = 0; a < P.natoms; ++a) {
        double d2 = 0.0;
        for (int d = 0; d < 3; ++d) {
          const double e = prim->center[3 * f + d] - mol->xyz[3 * a + d];
          d2 += e * e;
        }
        if (d2 < 1e-20) best = a;
      }
      if (best < 0) P.all_funcs_on_atoms = false;
      fatom[q] = std::max(best, 0);
    }
    P.d_fatom = P.alloc<int>(P.nbf_pad);
    NKX_CUDA(cudaMemcpy(P.d_fatom, fatom.data(), sizeof(int) * P.nbf_pad, cudaMemcpyHostToDevice));
    if (owner) {
      std::vector<int> ho(P.npad, 0);
      for (long p = 0; p < npoints; ++p) {
        const int o = owner[P.perm[p]];
        NKX_REQUIRE(o >= 0 && o < P.natoms, NKX_ERR_ARG, "point owner outside [0, natoms)");
        ho[p] = o;
      }
      P.d_owner = P.alloc<int>(P.npad);
      NKX_CUDA(cudaMemcpy(P.d_owner, ho.data(), sizeof(int) * P.npad, cudaMemcpyHostToDevice));
    }
  }
  // radial shells of every block (functions sharing centre, zeta and
  // n - l - 1), for the collocation kernels' shared radial factors; padding
  // positions (norm 0) point at shell 0
  {
    std::vector<StoShell> hsh((size_t)P.nblk * kBlockF);
    std::vector<int> hns(P.nblk, 0), hfs(P.nbf_pad, 0);
    for (int I = 0; I < P.nblk; ++I) {
      int n = 0;
      StoShell *S = hsh.data() + (size_t)I * kBlockF;
      for (int q = I * kBlockF; q < (I + 1) * kBlockF; ++q) {
        if (P.h_fperm[q] < 0) continue;
        const StoFunc &f = tab[q];
        int s = 0;
        while (s < n && !(S[s].cx == f.cx && S[s].cy == f.cy && S[s].cz == f.cz && S[s].zeta == f.zeta &&
                          S[s].k == f.k))
          ++s;
        if (s == n) S[n++] = StoShell{f.cx, f.cy, f.cz, f.zeta, f.k, 0};
        hfs[q] = s;
      }
      if (n == 0) S[n++] = StoShell{tab[I * kBlockF].cx, tab[I * kBlockF].cy, tab[I * kBlockF].cz, 1.0, 0, 0};
      hns[I] = n;
    }
    P.d_bshell = P.alloc<StoShell>(hsh.size());
    NKX_CUDA(cudaMemcpy(P.d_bshell, hsh.data(), sizeof(StoShell) * hsh.size(), cudaMemcpyHostToDevice));
    P.d_bnshell = P.alloc<int>(P.nblk);
    NKX_CUDA(cudaMemcpy(P.d_bnshell, hns.data(), sizeof(int) * P.nblk, cudaMemcpyHostToDevice));
    P.d_fshell = P.alloc<int>(P.nbf_pad);
    NKX_CUDA(cudaMemcpy(P.d_fshell, hfs.data(), sizeof(int) * P.nbf_pad, cudaMemcpyHostToDevice));
  }
  P.d_fperm = P.alloc<int>(P.nbf_pad);
  NKX_CUDA(cudaMemcpy(P.d_fperm, P.h_fperm.data(), sizeof(int) * P.nbf_pad, cudaMemcpyHostToDevice));
  P.d_finv = P.alloc<int>(finv.size());
  NKX_CUDA(cudaMemcpy(P.d_finv, finv.data(), sizeof(int) * finv.size(), cudaMemcpyHostToDevice));

  // --- screening: block I is significant for batch b if any function's
  // cutoff sphere meets the batch bounding box (octree.hpp:331-366)
  P.h_mask.assign((size_t)P.nbatch * P.mask_words, 0u);
  P.h_pair_off.assign(P.nbatch + 1, 0);
  // per block, the box holding every function's cutoff sphere: a block whose
  // box misses the batch box has no significant function there
  std::vector<double> flo(3 * (size_t)P.nblk, 1e300), fhi(3 * (size_t)P.nblk, -1e300);
  for (int q = 0; q < P.nbf_pad; ++q) {
    const int f = P.h_fperm[q], I = q / kBlockF;
    if (f < 0) continue;
    for (int d = 0; d < 3; ++d) {
      flo[3 * I + d] = std::min(flo[3 * I + d], prim->center[3 * f + d] - cut[f]);
      fhi[3 * I + d] = std::max(fhi[3 * I + d], prim->center[3 * f + d] + cut[f]);
    }
  }
#pragma omp parallel for schedule(dynamic, 64)
  for (long b = 0; b < P.nbatch; ++b) {
    const double *bl = &blo[3 * b], *bh = &bhi[3 * b];
    for (int I = 0; I < P.nblk; ++I) {
      bool near = true;
      for (int d = 0; d < 3; ++d) near = near && flo[3 * I + d] <= bh[d] && fhi[3 * I + d] >= bl[d];
      if (!near) continue;
      bool sig = false;
      for (int q = I * kBlockF; q < (I + 1) * kBlockF && !sig; ++q) {
        const int f = P.h_fperm[q];
        if (f < 0) continue;
        sig = box_distance2(&prim->center[3 * f], bl, bh) <= cut[f] * cut[f];
      }
      if (sig) P.h_mask[b * P.mask_words + I / 32] |= 1u << (I % 32);
    }
  }
  std::vector<int> pblk, pbatch;
  for (long b = 0; b < P.nbatch; ++b) {
    for (int I = 0; I < P.nblk; ++I)
      if ((P.h_mask[b * P.mask_words + I / 32] >> (I % 32)) & 1u) {
        pblk.push_back(I);
        pbatch.push_back((int)b);
      }
    P.h_pair_off[b + 1] = (int)pblk.size();
  }
  P.npairs = (long)pblk.size();

  // --- device copies
  P.d_px = P.alloc<double>(P.npad);
  P.d_py = P.alloc<double>(P.npad);
  P.d_pz = P.alloc<double>(P.npad);
  P.d_w = P.alloc<double>(P.npad);
  NKX_CUDA(cudaMemcpy(P.d_px, hx.data(), sizeof(double) * P.npad, cudaMemcpyHostToDevice));
  NKX_CUDA(cudaMemcpy(P.d_py, hy.data(), sizeof(double) * P.npad, cudaMemcpyHostToDevice));
  NKX_CUDA(cudaMemcpy(P.d_pz, hz.data(), sizeof(double) * P.npad, cudaMemcpyHostToDevice));
  NKX_CUDA(cudaMemcpy(P.d_w, hw.data(), sizeof(double) * P.npad, cudaMemcpyHostToDevice));
  P.d_sto = P.alloc<StoFunc>(P.nbf_pad);
  NKX_CUDA(cudaMemcpy(P.d_sto, tab.data(), sizeof(StoFunc) * P.nbf_pad, cudaMemcpyHostToDevice));
  P.d_mask = P.alloc<uint32_t>(P.h_mask.size());
  NKX_CUDA(cudaMemcpy(P.d_mask, P.h_mask.data(), sizeof(uint32_t) * P.h_mask.size(), cudaMemcpyHostToDevice));
  P.d_pair_off = P.alloc<int>(P.nbatch + 1);
  NKX_CUDA(cudaMemcpy(P.d_pair_off, P.h_pair_off.data(), sizeof(int) * (P.nbatch + 1), cudaMemcpyHostToDevice));
  P.d_pair_blk = P.alloc<int>(std::max<long>(1, P.npairs));
  P.d_pair_batch = P.alloc<int>(std::max<long>(1, P.npairs));
  if (P.npairs) {
    NKX_CUDA(cudaMemcpy(P.d_pair_blk, pblk.data(), sizeof(int) * P.npairs, cudaMemcpyHostToDevice));
    NKX_CUDA(cudaMemcpy(P.d_pair_batch, pbatch.data(), sizeof(int) * P.npairs, cudaMemcpyHostToDevice));
  }

  // --- chunks of batches sized by the workspace
  size_t ws = opts->workspace_bytes;
  if (ws == 0) {
    size_t fr = 0;
    NKX_CUDA(device_free_bytes(&fr));
    ws = std::min<size_t>(kDefaultWorkspace, fr / 3);
  }
  plan_chunks(P, std::max<long>(1, (long)(ws / kPairBytes)));

  // per-point arrays (two spins)
  P.d_rho = P.alloc<double>(2 * P.npad);
  P.d_grad = P.alloc<double>(6 * P.npad);
  P.d_coef = P.alloc<double>(8 * P.npad);
  P.d_vj = P.alloc<double>(P.npad);
  P.d_V = P.alloc<double>(3 * (size_t)P.nbf_pad * P.nbf_pad);
  P.d_E = P.alloc<double>(2);
  P.d_status = reinterpret_cast<int *>(P.d_E + 1);
  if (Plan::Result *r = result_slot(true, nullptr)) P.h_result = r;
  NKX_CUDA(cudaMemset(P.d_status, 0, sizeof(int) * 2));
  NKX_CUDA(cudaMemset(P.d_rho, 0, sizeof(double) * 2 * P.npad));
  NKX_CUDA(cudaMemset(P.d_grad, 0, sizeof(double) * 6 * P.npad));

  // --- aux metric and its factor
  if (aux && aux->nbf > 0) {
    for (int i = 0; i < aux->nbf; ++i)
      NKX_REQUIRE(aux->l[i] >= 0 && aux->l[i] <= 7 && aux->n[i] > aux->l[i] && abs(aux->m[i]) <= aux->l[i] &&
                      aux->zeta[i] > 0,
                  NKX_ERR_UNSUPPORTED, "aux function outside n > l, |m| <= l <= 7, zeta > 0");
    P.naux = aux->nbf;
    auto atab = make_aux_table(*aux);
    auto astab = make_sto_table(*aux);
    P.d_aux = P.alloc<AuxFunc>(P.naux);
    NKX_CUDA(cudaMemcpy(P.d_aux, atab.data(), sizeof(AuxFunc) * P.naux, cudaMemcpyHostToDevice));
    const auto ash = make_aux_shells(atab);
    P.nashell = (int)ash.size();
    P.d_ashell = P.alloc<AuxShell>(ash.size());
    NKX_CUDA(cudaMemcpy(P.d_ashell, ash.data(), sizeof(AuxShell) * ash.size(), cudaMemcpyHostToDevice));
    std::vector<int> loose;
    const auto grp = make_aux_groups(ash, loose);
    P.nagroup = (int)grp.size();
    P.nloose = (int)loose.size();
    P.h_group_off.assign(5, 0);
    for (const AuxGroup &G : grp) ++P.h_group_off[G.l + 1];
    for (int L = 0; L < 4; ++L) P.h_group_off[L + 1] += P.h_group_off[L];
    P.d_agroup = P.alloc<AuxGroup>(std::max<size_t>(1, grp.size()));
    if (!grp.empty())
      NKX_CUDA(cudaMemcpy(P.d_agroup, grp.data(), sizeof(AuxGroup) * grp.size(), cudaMemcpyHostToDevice));
    P.d_loose = P.alloc<int>(std::max<size_t>(1, loose.size()));
    if (!loose.empty())
      NKX_CUDA(cudaMemcpy(P.d_loose, loose.data(), sizeof(int) * loose.size(), cudaMemcpyHostToDevice));
    StoFunc *d_asto = dalloc<StoFunc>(P.naux);
    NKX_CUDA(cudaMemcpy(d_asto, astab.data(), sizeof(StoFunc) * P.naux, cudaMemcpyHostToDevice));
    const size_t NA = P.naux;
    P.d_L = P.alloc<double>(NA * NA);
    P.d_y = P.alloc<double>(NA);
    P.d_c = P.alloc<double>(NA);
    P.d_info = P.alloc<int>(1);
    cublasHandle_t hb;
    NKX_REQUIRE(cublasCreate(&hb) == CUBLAS_STATUS_SUCCESS, NKX_ERR_CUDA, "cublasCreate failed");
    P.cublas = hb;
    cublasSetStream(hb, P.stream);
    grid_metric(d_asto, P.d_aux, P.naux, P.d_px, P.d_py, P.d_pz, P.d_w, P.npad, hb, P.stream, P.d_L);
    cudaFree(d_asto);
    P.h_metric.resize(NA * NA);
    NKX_CUDA(cudaMemcpy(P.h_metric.data(), P.d_L, sizeof(double) * NA * NA, cudaMemcpyDeviceToHost));
    cusolverDnHandle_t hs;
    NKX_REQUIRE(cusolverDnCreate(&hs) == CUSOLVER_STATUS_SUCCESS, NKX_ERR_CUDA, "cusolverDnCreate failed");
    P.cusolver = hs;
    cusolverDnSetStream(hs, P.stream);
    P.svd_mode = opts->metric_svd_thr > 0;
    P.metric_svd_thr = opts->metric_svd_thr;
    P.d_X = P.svd_mode ? P.alloc<double>(NA * NA) : nullptr;
    P.d_t = P.alloc<double>(NA);
    P.d_piv = P.alloc<int>(NA);
    factor_metric(P);
  }
  NKX_CUDA(cudaStreamSynchronize(P.stream));
}

// ------------------------------------------------- core Hamiltonian ----
// w_g v_n(g) = w_g sum_A Z_A / (|r_g - R_A| + 1e-30), the nuclear attraction
// weight of core_hamiltonian.hpp:133-289 (V_n = -sum_g w v_n phi phi^T)
__global__ void core_vne_kernel(const double *__restrict__ px, const double *__restrict__ py,
                                const double *__restrict__ pz, const double *__restrict__ w, long npad,
                                const double *__restrict__ centers, const double *__restrict__ charges, int natoms,
                                double *__restrict__ wv) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= npad) return;
  double v = 0.0;
  if (w[g] != 0.0)
    for (int a = 0; a < natoms; ++a) {
      const double dx = px[g] - centers[3 * a], dy = py[g] - centers[3 * a + 1], dz = pz[g] - centers[3 * a + 2];
      v += charges[a] / (sqrt(dx * dx + dy * dy + dz * dz) + 1e-30);
    }
  wv[g] = w[g] * v;
}

// Z planes of the core Hamiltonian for the pairs of one chunk, Z^T[pair][3][g][f]
// from PhiT[pair][4][g][f]: pass 0: plane 0 = 1/2 w phi (S), plane 1 =
// -1/2 w v_n phi (V_n); pass 1: plane k = 1/4 w d_k phi (T, k = x, y, z), so
// that Vbar + Vbar^T of each contraction is the matrix itself.
__global__ void core_z_kernel(const double *__restrict__ phiT, const double *__restrict__ w,
                              const double *__restrict__ wv, const int *__restrict__ pair_batch, long p0, int pass,
                              double *__restrict__ zT) {
  const size_t tile = (size_t)kBatch * kBlockF;
  const long q = blockIdx.x;
  const long b = pair_batch[p0 + q];
  const double *P = phiT + (size_t)q * 4 * tile;
  double *Z = zT + (size_t)q * 3 * tile;
  for (int e = threadIdx.x; e < (int)tile; e += blockDim.x) {
    const long g = b * kBatch + e / kBlockF;
    if (pass == 0) {
      Z[e] = 0.5 * w[g] * P[e];
      Z[tile + e] = -0.5 * wv[g] * P[e];
    } else {
      const double h = 0.25 * w[g];
      Z[e] = h * P[tile + e];
      Z[2 * tile + e] = h * P[3 * tile + e];
      Z[tile + e] = h * P[2 * tile + e];
    }
  }
}

// ========================================================= Fock build ===

void launch_colloc(Plan &P, const Chunk &c, cudaStream_t s) {
  const long np = c.p1 - c.p0;
  if (np <= 0) return;
  auto *kernel = P.gga ? colloc_fp64_kernel<true> : colloc_fp64_kernel<false>;
  kernel<<<dim3((unsigned)np, point_split(np, P.nsm)), 256, 0, s>>>(P.d_sto, P.d_fshell, P.d_bshell, P.d_bnshell,
                                                                    P.d_px, P.d_py, P.d_pz, P.d_pair_batch,
                                                                    P.d_pair_blk, c.p0, P.ws_phi);
  NKX_LAUNCH_CHECK();
  ++P.launches;
}

// The grid RI-J fit (coulomb.hpp:84-95) in two steps, so that a grid
// sharded over ranks can sum y between them: coulomb_y forms this plan's
// y = Vw rho_total over its points; coulomb_solve solves c = (A|B)^-1 y
// (pivoted Cholesky or half inverse) and forms v_g = w_g sum_a c_a V_a(g).
// The FP64 build evaluates the potentials' radial factors; the mixed build
// reads them from the plan's FP32 table when it fits (coulomb_table).
// The FP32 radial-factor table of the mixed build (aux_rtab_kernel), made on
// first use when it fits in a quarter of the free device memory (and
// kRtabMaxBytes); otherwise the J passes evaluate the factors as FP64 does.
constexpr size_t kRtabMaxBytes = (size_t)32 << 30;
static const float *coulomb_table(Plan &P, bool mixed, cudaStream_t s) {
  if (!mixed || P.rtab_failed) return nullptr;
  if (!P.d_rtab) {
    const size_t bytes = (size_t)P.nashell * P.npad * sizeof(float);
    size_t fr = 0;
    NKX_CUDA(device_free_bytes(&fr));
    if (bytes > kRtabMaxBytes || bytes > fr / 4 || cudaMalloc(&P.d_rtab, bytes) != cudaSuccess) {
      cudaGetLastError();
      P.d_rtab = nullptr;
      P.rtab_failed = true;
      return nullptr;
    }
    P.allocs.push_back(P.d_rtab);
    aux_rtab_kernel<<<dim3(nblk(P.npad, 256), (unsigned)P.nashell), 256, 0, s>>>(P.d_ashell, P.nashell, P.d_px, P.d_py,
                                                                                P.d_pz, P.npad, P.d_rtab);
    NKX_LAUNCH_CHECK();
    ++P.launches;
  }
  return P.d_rtab;
}

// groups of l = 0 are [0, .x), of l = 1 [.x, .y), ...
static int4 group_ends(const Plan &P) {
  return make_int4(P.h_group_off[1], P.h_group_off[2], P.h_group_off[3], P.h_group_off[4]);
}

void coulomb_y(Plan &P, int nspin, cudaStream_t s, bool mixed) {
    const float *rtab = coulomb_table(P, mixed, s);
    // point slices: 64 or one per 4096 points, and more (down to 1024 points
    // each) where there are few groups, so that four blocks an SM are in flight
    long nsl = std::max<long>(1, std::min<long>(64, (P.npad + 4095) / 4096));
    auto more_slices = [&](int groups) {
      if (groups > 0) nsl = std::max(nsl, std::min((4L * P.nsm + groups - 1) / groups, P.npad / 1024));
    };
    more_slices(P.nagroup);
    more_slices(P.nloose);
    const long slice = (P.npad + nsl - 1) / nsl;
    if (!P.d_ypart) P.d_ypart = P.alloc<double>((size_t)nsl * P.naux);
    if (P.nagroup > 0) {
      auto *kernel = rtab ? aux_y_groups_kernel<true> : aux_y_groups_kernel<false>;
      kernel<<<(unsigned)(P.nagroup * nsl), 256, 0, s>>>(P.d_agroup, group_ends(P), P.d_ashell, P.d_px, P.d_py, P.d_pz,
                                                        P.d_w, P.d_rho, nspin, P.npad, slice, rtab, P.naux, (int)nsl,
                                                        P.d_ypart);
      NKX_LAUNCH_CHECK();
      ++P.launches;
    }
    if (P.nloose > 0) {
      aux_y_shell_kernel<<<dim3(P.nloose, (unsigned)nsl), 256, 0, s>>>(P.d_ashell, P.d_loose, P.d_px, P.d_py, P.d_pz,
                                                                      P.d_w, P.d_rho, nspin, P.npad, slice, rtab,
                                                                      P.naux, P.d_ypart);
      NKX_LAUNCH_CHECK();
      ++P.launches;
    }
    aux_y_reduce_kernel<<<nblk(P.naux * 32L, 256), 256, 0, s>>>(P.d_ypart, (int)nsl, P.naux, P.d_y);
    NKX_LAUNCH_CHECK();
    ++P.launches;
}

void coulomb_solve(Plan &P, cudaStream_t s, bool mixed) {
    const float *rtab = coulomb_table(P, mixed, s);
    if (P.svd_mode) {
      const double one = 1.0, zero = 0.0;
      cublasHandle_t hb = (cublasHandle_t)P.cublas;
      cublasSetStream(hb, s);
      NKX_REQUIRE(cublasDgemv(hb, CUBLAS_OP_T, P.naux, P.K, &one, P.d_X, P.naux, P.d_y, 1, &zero, P.d_t, 1) ==
                          CUBLAS_STATUS_SUCCESS &&
                      cublasDgemv(hb, CUBLAS_OP_N, P.naux, P.K, &one, P.d_X, P.naux, P.d_t, 1, &zero, P.d_c, 1) ==
                          CUBLAS_STATUS_SUCCESS,
                  NKX_ERR_CUDA, "cublasDgemv failed");
    } else {
      gather_kernel<<<nblk(P.K, 128), 128, 0, s>>>(P.K, P.d_piv, P.d_y, P.d_t);
      cusolverDnHandle_t hs = (cusolverDnHandle_t)P.cusolver;
      cusolverDnSetStream(hs, s);
      NKX_REQUIRE(cusolverDnDpotrs(hs, CUBLAS_FILL_MODE_LOWER, P.K, 1, P.d_L, P.K, P.d_t, P.K, P.d_info) ==
                      CUSOLVER_STATUS_SUCCESS,
                  NKX_ERR_CUDA, "cusolverDnDpotrs failed");
      NKX_CUDA(cudaMemsetAsync(P.d_c, 0, sizeof(double) * P.naux, s));
      scatter_kernel<<<nblk(P.K, 128), 128, 0, s>>>(P.K, P.d_piv, P.d_t, P.d_c);
      NKX_LAUNCH_CHECK();
      P.launches += 2;
    }
    const int4 goff = group_ends(P);
    if (rtab)
      aux_v_group_tab_kernel<<<nblk(P.npad, 256), 128, 0, s>>>(P.d_agroup, goff, P.d_ashell, P.d_c, P.d_px, P.d_py,
                                                               P.d_pz, P.d_w, P.npad, rtab, P.d_vj);
    else
      aux_v_group_kernel<<<nblk(P.npad, 128), 128, 0, s>>>(P.d_agroup, goff, P.d_ashell, P.d_c, P.d_px, P.d_py, P.d_pz,
                                                           P.d_w, P.npad, P.d_vj);
    NKX_LAUNCH_CHECK();
    ++P.launches;
    if (P.nloose > 0) {
      auto *kernel = rtab ? aux_v_loose_kernel<true> : aux_v_loose_kernel<false>;
      kernel<<<nblk(P.npad, 128), 128, 0, s>>>(P.d_ashell, P.d_loose, P.nloose, P.d_c, P.d_px, P.d_py, P.d_pz, P.d_w,
                                               P.npad, rtab, P.d_vj);
      NKX_LAUNCH_CHECK();
      ++P.launches;
    }
}

template <bool GRAD, int NN>
static void launch_density_fp64(Plan &P, long b0, long b1, long p0, int nspin, int nocc, int nocc_pad, double *T,
                                cudaStream_t s) {
  NKX_CUDA(cudaFuncSetAttribute(density_fp64_kernel<GRAD, NN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                DShape<NN>::kSmem));
  const dim3 grid((unsigned)((b1 - b0) * (GRAD ? 4 : 1) * (nocc_pad / (8 * NN))), nspin);
  density_fp64_kernel<GRAD, NN><<<grid, 256, DShape<NN>::kSmem, s>>>(P.ws_phi, P.d_Cf, P.d_occ, nocc, nocc_pad,
                                                                    P.nbf_pad, P.d_pair_off, P.d_pair_blk, b0, p0,
                                                                    P.d_rho, P.d_grad, P.npad, T);
}

// orbital tiles of at most 64, equally wide, in multiples of 8: *nn eighths
// of a tile; returns the padded orbital count
int fp64_orbital_pad(int nocc, int *nn) {
  const int ntile = (nocc + 63) / 64;
  *nn = ((nocc + ntile - 1) / ntile + 7) / 8;
  return ntile * 8 * *nn;
}

// The FP64 density of batches [b0, b1) of a chunk whose collocation is in
// ws_phi (first pair p0), after fp64_density_begin
void fp64_density_range(Plan &P, long b0, long b1, long p0, int nspin, int nocc, double *T, cudaStream_t s) {
  int nn = 0;
  const int np = fp64_orbital_pad(nocc, &nn);
  auto go = [&](auto grad) {
    constexpr bool G = decltype(grad)::value;
    switch (nn) {
      case 1: return launch_density_fp64<G, 1>(P, b0, b1, p0, nspin, nocc, np, T, s);
      case 2: return launch_density_fp64<G, 2>(P, b0, b1, p0, nspin, nocc, np, T, s);
      case 3: return launch_density_fp64<G, 3>(P, b0, b1, p0, nspin, nocc, np, T, s);
      case 4: return launch_density_fp64<G, 4>(P, b0, b1, p0, nspin, nocc, np, T, s);
      case 5: return launch_density_fp64<G, 5>(P, b0, b1, p0, nspin, nocc, np, T, s);
      case 6: return launch_density_fp64<G, 6>(P, b0, b1, p0, nspin, nocc, np, T, s);
      case 7: return launch_density_fp64<G, 7>(P, b0, b1, p0, nspin, nocc, np, T, s);
      default: return launch_density_fp64<G, 8>(P, b0, b1, p0, nspin, nocc, np, T, s);
    }
  };
  P.gga ? go(std::true_type{}) : go(std::false_type{});
  NKX_LAUNCH_CHECK();
  ++P.launches;
}

// The FP64 V contraction of one chunk: nz planes of zT (stride z_stride
// tiles) against PhiT into V.
static void launch_vgemm_fp64(Plan &P, const Chunk &c, const double *phiT, const double *zT, int phi_stride,
                              int z_stride, int nz, double *V, cudaStream_t s) {
  const long parts = (long)nz * P.nblk * P.nblk;
  const int nsplit = batch_split(parts, c.b1 - c.b0, P.nsm);
  if (nsplit > 1 && !P.d_vpart) P.d_vpart = P.alloc<double>((size_t)4 * P.nsm * kBlockF * kBlockF);
  auto go = [&](auto slots) {
    constexpr int SL = decltype(slots)::value;
    NKX_CUDA(cudaFuncSetAttribute(vgemm_fp64_kernel<SL>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVSmemBytes));
    vgemm_fp64_kernel<SL><<<dim3(P.nblk, P.nblk, nz * nsplit), 256, kVSmemBytes, s>>>(
        phiT, zT, phi_stride, z_stride, P.d_pair_off, P.d_mask, P.mask_words, c.b0, c.b1, c.p0, nsplit, P.nbf_pad, V,
        P.d_vpart);
    ++P.launches;
    if (nsplit > 1) {
      vpart_reduce_kernel<SL><<<dim3((unsigned)parts, 4 * SL * SL), 256, 0, s>>>(P.d_vpart, nsplit, P.nblk, P.nbf_pad,
                                                                               V);
      ++P.launches;
    }
  };
  // a block's functions fill slot after slot (build_plan)
  P.nbf <= 64 ? go(std::integral_constant<int, 2>{}) : go(std::integral_constant<int, 4>{});
  NKX_LAUNCH_CHECK();
}

// function-major orbitals, and rho / grad rho cleared for the kernels' shares
void fp64_density_begin(Plan &P, int nspin, int nocc, cudaStream_t s) {
  int nn = 0;
  const int nocc_pad = fp64_orbital_pad(nocc, &nn);
  if ((size_t)nocc_pad * P.nbf_pad * 2 > P.cf_cap) {
    P.cf_cap = (size_t)nocc_pad * P.nbf_pad * 2;
    P.d_Cf = P.alloc<double>(P.cf_cap);
  }
  transpose_orbitals_kernel<<<dim3(P.nbf_pad / 32, (nocc_pad + 31) / 32, nspin), dim3(32, 8), 0, s>>>(
      P.d_Ct, nocc, nocc_pad, P.nbf_pad, P.d_Cf);
  NKX_LAUNCH_CHECK();
  ++P.launches;
  NKX_CUDA(cudaMemsetAsync(P.d_rho, 0, sizeof(double) * nspin * P.npad, s));
  if (P.gga) NKX_CUDA(cudaMemsetAsync(P.d_grad, 0, sizeof(double) * 3 * nspin * P.npad, s));
}

// FP64 pass A: collocation + density of every chunk into d_rho / d_grad
void fp64_density_pass(Plan &P, int nspin, int nocc, cudaStream_t s, StageTimer &T) {
  fp64_density_begin(P, nspin, nocc, s);
  for (const Chunk &c : P.chunks) {
    if (c.p1 - c.p0 > 0) {
      T.begin(ST_COLLOC, s);
      launch_colloc(P, c, s);
      T.end(s);
    }
    T.begin(ST_DENSITY, s);
    fp64_density_range(P, c.b0, c.b1, c.p0, nspin, nocc, nullptr, s);
    T.end(s);
  }
}

void fock_build_fp64(Plan &P, int nspin, int nocc, bool needJ, bool fuse, bool separateJ, cudaStream_t s,
                     StageTimer &T, int phase) {
  const bool multi = P.chunks.size() > 1;
  const int nzs = nspin + (separateJ ? 1 : 0);
  if (!P.ws_z) P.ws_z = P.alloc<double>(std::max<long>(1, P.max_chunk_pairs) * 3 * (size_t)kBatch * kBlockF);
  if (phase != 2) {
    // ---- pass A: collocation + density, and this plan's share of the J fit vector
    fp64_density_pass(P, nspin, nocc, s, T);
    if (needJ) {
      T.begin(ST_COULOMB, s);
      coulomb_y(P, nspin, s, false);
      T.end(s);
    }
    if (phase == 1) return;
  }
  // ---- J: fit coefficients and fitted potential
  if (needJ) {
    T.begin(ST_COULOMB, s);
    coulomb_solve(P, s, false);
    T.end(s);
  }
  // ---- functional
  T.begin(ST_FUNC, s);
  NKX_CUDA(cudaMemsetAsync(P.d_E, 0, sizeof(double), s));
  functional_kernel<<<nblk(P.npad, 256), 256, 0, s>>>(P.xc, P.gga, nspin, P.npad, P.npad, P.d_w, P.d_rho, P.d_grad,
                                                      (needJ && fuse) ? P.d_vj : nullptr, P.d_coef, P.d_E,
                                                      nullptr);
  NKX_LAUNCH_CHECK();
  ++P.launches;
  T.end(s);
  // ---- pass B: Z and the V contraction
  const size_t tile = (size_t)kBatch * kBlockF;
  NKX_CUDA(cudaMemsetAsync(P.d_V, 0, sizeof(double) * nzs * P.nbf_pad * P.nbf_pad, s));
  for (const Chunk &c : P.chunks) {
    const long np = c.p1 - c.p0;
    if (np <= 0) continue;
    if (multi) {
      T.begin(ST_COLLOC, s);
      launch_colloc(P, c, s);
      T.end(s);
    }
    T.begin(ST_ZBUILD, s);
    const dim3 zgrid((unsigned)np, point_split(np, P.nsm));
    auto *zbuild = zgrid.y > 1 ? (P.gga ? zbuild_fp64_kernel<true, true> : zbuild_fp64_kernel<false, true>)
                               : (P.gga ? zbuild_fp64_kernel<true, false> : zbuild_fp64_kernel<false, false>);
    zbuild<<<zgrid, 256, 0, s>>>(P.ws_phi, P.d_coef, P.d_vj, P.d_pair_batch, c.p0, nzs, nspin, P.npad, P.ws_z);
    NKX_LAUNCH_CHECK();
    ++P.launches;
    T.end(s);
    T.begin(ST_VGEMM, s);
    launch_vgemm_fp64(P, c, P.ws_phi, P.ws_z, P.gga ? 4 : 1, nzs, nzs, P.d_V, s);
    T.end(s);
  }
  (void)tile;
}

// orbitals -> Ct[spin][i][p] in plan order (host or device C / occ)
void upload_orbitals(Plan &P, int nspin, int nocc, const double *C, const double *occ, int mem, cudaStream_t s) {
  if (nocc > P.nocc_cap) {
    P.nocc_cap = nocc;
    P.d_Ct = P.alloc<double>((size_t)2 * nocc * P.nbf_pad);
    P.d_occ = P.alloc<double>((size_t)2 * nocc);
    P.d_Cin = P.alloc<double>((size_t)2 * nocc * P.nbf);
  }
  const double *Cd = C;
  if (mem == NKX_MEM_HOST) {
    NKX_CUDA(cudaMemcpyAsync(P.d_Cin, C, sizeof(double) * nspin * nocc * P.nbf, cudaMemcpyHostToDevice, s));
    NKX_CUDA(cudaMemcpyAsync(P.d_occ, occ, sizeof(double) * nspin * nocc, cudaMemcpyHostToDevice, s));
    Cd = P.d_Cin;
  } else {
    NKX_CUDA(cudaMemcpyAsync(P.d_occ, occ, sizeof(double) * nspin * nocc, cudaMemcpyDeviceToDevice, s));
  }
  pack_orbitals_kernel<<<nblk((long)nspin * nocc * P.nbf_pad, 256), 256, 0, s>>>(
      Cd, P.d_occ, P.d_fperm, P.nbf, nocc, nspin, P.nbf_pad, P.d_Ct, P.d_status + 1);
  NKX_LAUNCH_CHECK();
  ++P.launches;
}

// One Fock build (phase 0), or one half of a build whose grid is sharded
// over ranks: phase 1 uploads the orbitals, runs the density pass and writes
// this plan's share of the J fit vector y to `y` (naux doubles, host or
// device by `mem`); the caller sums y over the ranks; phase 2 takes the
// summed y (same memory kind) and finishes the build (fit, functional, V and
// J on this plan's points).  Phase 2 needs a phase 1 of the same
// precision, spin count and orbitals on this plan immediately before it.
// One build on the stream.  capture_only (device buffers, phase 0): only the
// device work is issued -- no events, host copies, synchronisation or status
// check -- so that it can be recorded into a CUDA graph.
static void fock_build_once(Plan &P, int precision, int nspin, int nocc, const double *C, const double *occ, int mem,
                            int fuse_j, double *E, double *V, double *J, cudaStream_t user, int phase, double *y,
                            bool capture_only) {
  if (phase == 2) {
    NKX_REQUIRE(P.phase1_done, NKX_ERR_ARG, "phase 2 of a sharded build needs phase 1 on this plan first");
    precision = P.phase1_precision;
    nspin = P.phase1_nspin;
    nocc = P.phase1_nocc;
  }
  NKX_REQUIRE(nspin == 1 || nspin == 2, NKX_ERR_ARG, "nspin must be 1 or 2");
  NKX_REQUIRE(phase == 2 || (nocc > 0 && C && occ), NKX_ERR_ARG, "invalid orbitals");
  NKX_REQUIRE(phase == 1 || (E && (V || J)), NKX_ERR_ARG, "invalid outputs");
  NKX_REQUIRE(phase == 0 || (y && P.naux > 0), NKX_ERR_ARG, "a sharded build needs y and a plan with an aux basis");
  NKX_REQUIRE(mem == NKX_MEM_DEVICE || mem == NKX_MEM_HOST, NKX_ERR_ARG, "mem must be NKX_MEM_DEVICE or NKX_MEM_HOST");
  NKX_REQUIRE(precision == NKX_PREC_FP64 || precision == NKX_PREC_MIXED, NKX_ERR_ARG, "unknown precision");
  const bool needJ = P.naux > 0 && (J != nullptr || fuse_j || phase != 0);
  NKX_REQUIRE(!(fuse_j && P.naux == 0), NKX_ERR_ARG, "fuse_j needs a plan with an aux basis");
  // V may be NULL only when J alone is asked for (the exchange-correlation
  // terms are then formed and dropped)
  NKX_REQUIRE(phase == 1 || V != nullptr || (J != nullptr && !fuse_j && P.naux > 0), NKX_ERR_ARG,
              "V must be given unless J alone is requested from a plan with an aux basis");
  const bool separateJ = needJ && !fuse_j && J;
  cudaStream_t s = user ? user : P.stream;
  P.launches = 0;
  StageTimer T(P);
  T.on = !capture_only;
  if (!capture_only) NKX_CUDA(cudaEventRecord(P.ev[0], s));
  P.phase1_done = false;
  if (phase == 2) {
    NKX_CUDA(cudaMemcpyAsync(P.d_y, y, sizeof(double) * P.naux,
                             mem == NKX_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, s));
  } else {
    NKX_CUDA(cudaMemsetAsync(P.d_status, 0, sizeof(int) * 2, s));
    upload_orbitals(P, nspin, nocc, C, occ, mem, s);
  }

  const bool mixed = precision == NKX_PREC_MIXED && mixed_available(P);
  NKX_REQUIRE(mixed || precision == NKX_PREC_FP64, NKX_ERR_UNSUPPORTED, "mixed precision path unavailable");
  if (mixed)
    fock_build_mixed(P, nspin, nocc, needJ, fuse_j != 0, separateJ, s, T, phase);
  else
    fock_build_fp64(P, nspin, nocc, needJ, fuse_j != 0, separateJ, s, T, phase);

  if (phase == 1) {
    NKX_CUDA(cudaMemcpyAsync(y, P.d_y, sizeof(double) * P.naux,
                             mem == NKX_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, s));
    NKX_CUDA(cudaMemcpyAsync(P.h_result, P.d_E, sizeof(Plan::Result), cudaMemcpyDeviceToHost, s));
    NKX_CUDA(cudaStreamSynchronize(s));
    const int *status = P.h_result->status;
    NKX_REQUIRE(status[0] == 0, NKX_ERR_TIMEOUT, "a tensor-core kernel wait gave up in phase 1");
    NKX_REQUIRE(status[1] == 0, NKX_ERR_NUMERIC, "non-finite value in the orbitals, occupations or an operand");
    P.phase1_done = true;
    P.phase1_precision = precision;
    P.phase1_nspin = nspin;
    P.phase1_nocc = nocc;
    return;
  }

  // symmetrise + unpad into the output (device) or a staging buffer (host)
  const size_t nn = (size_t)P.nbf * P.nbf;
  const int nout = nspin + (separateJ ? 1 : 0);
  double *dst = nullptr;
  if (mem == NKX_MEM_DEVICE) {
    dst = V;
  } else {
    if (!P.d_out) P.d_out = P.alloc<double>(3 * nn);
    dst = P.d_out;
  }
  dim3 tb(16, 16), gb(nblk(P.nbf, 16), nblk(P.nbf, 16));
  for (int z = 0; z < nout; ++z) {
    if (z < nspin && !V) continue;
    double *o = (z < nspin) ? dst + z * nn : (mem == NKX_MEM_DEVICE ? J : dst + nspin * nn);
    symmetrize_unpad_kernel<<<gb, tb, 0, s>>>(P.nbf, P.nbf_pad, P.d_finv, P.d_V + (size_t)z * P.nbf_pad * P.nbf_pad,
                                              o);
    ++P.launches;
  }
  NKX_LAUNCH_CHECK();
  if (capture_only) return;
  if (mem == NKX_MEM_HOST) {
    if (V) NKX_CUDA(cudaMemcpyAsync(V, dst, sizeof(double) * nspin * nn, cudaMemcpyDeviceToHost, s));
    if (separateJ) NKX_CUDA(cudaMemcpyAsync(J, dst + nspin * nn, sizeof(double) * nn, cudaMemcpyDeviceToHost, s));
  }
  NKX_CUDA(cudaMemcpyAsync(P.h_result, P.d_E, sizeof(Plan::Result), cudaMemcpyDeviceToHost, s));
  NKX_CUDA(cudaEventRecord(P.ev[1], s));
  NKX_CUDA(cudaStreamSynchronize(s));
  *E = P.h_result->E;
  const int *status = P.h_result->status;
  float st[6];
  T.collect(st);
  P.last.colloc_ms = st[ST_COLLOC];
  P.last.density_ms = st[ST_DENSITY];
  P.last.functional_ms = st[ST_FUNC];
  P.last.coulomb_ms = st[ST_COULOMB];
  P.last.zbuild_ms = st[ST_ZBUILD];
  P.last.vgemm_ms = st[ST_VGEMM];
  cudaEventElapsedTime(&P.last.total_ms, P.ev[0], P.ev[1]);
  P.last.launches = P.launches;
  P.last_nspin = nspin;
  NKX_REQUIRE(status[0] == 0, NKX_ERR_TIMEOUT,
              "a tensor-core kernel wait gave up (wait code " + std::to_string(status[0]) + "); outputs are invalid");
  NKX_REQUIRE(status[1] == 0 && std::isfinite(*E), NKX_ERR_NUMERIC,
              "non-finite value in the orbitals, occupations, grid or an operand of the build; outputs are invalid");
}

void Plan::drop_graphs() {
  for (BuildGraph &g : graphs) {
    if (g.exec) cudaGraphExecDestroy(g.exec);
    release(g.C);
    release(g.occ);
    release(g.V);
    release(g.J);
  }
  graphs.clear();
}

// A build replayed from a CUDA graph (graph mode, device buffers, phase 0).
// The second build of a kind (precision, spins, orbitals, outputs) records the
// device work of a build that reads the orbitals from, and writes V and J to,
// buffers of the graph's own; every build of that kind then copies the
// caller's orbitals in, launches the graph and copies the results out.  A
// build of another kind, or any change of the plan, drops the graphs first
// (their launch arguments and buffers are baked in).  If recording fails the
// kind keeps running ordinary builds.
static void fock_build_graph(Plan &P, int precision, int nspin, int nocc, const double *C, const double *occ,
                             int fuse_j, double *E, double *V, double *J, cudaStream_t user) {
  BuildGraph *g = nullptr;
  for (BuildGraph &x : P.graphs)
    if (x.precision == precision && x.nspin == nspin && x.nocc == nocc && x.fuse == fuse_j && x.hasV == (V != nullptr) &&
        x.hasJ == (J != nullptr))
      g = &x;
  if (!g || g->failed || !g->exec) {
    const bool record = g && !g->failed;
    if (!record) {
      // first build of this kind: an ordinary build (it may grow buffers the
      // recorded builds of other kinds use), then remember the kind
      P.drop_graphs();
      fock_build_once(P, precision, nspin, nocc, C, occ, NKX_MEM_DEVICE, fuse_j, E, V, J, user, 0, nullptr, false);
      BuildGraph n;
      n.precision = precision;
      n.nspin = nspin;
      n.nocc = nocc;
      n.fuse = fuse_j;
      n.hasV = V != nullptr;
      n.hasJ = J != nullptr;
      if (!g) P.graphs.push_back(n);
      return;
    }
    // second build of this kind: record it
    const size_t nn = (size_t)P.nbf * P.nbf;
    g->C = P.alloc<double>((size_t)nspin * nocc * P.nbf);
    g->occ = P.alloc<double>((size_t)nspin * nocc);
    g->V = V ? P.alloc<double>(nspin * nn) : nullptr;
    g->J = J ? P.alloc<double>(nn) : nullptr;
    cudaStream_t s = user ? user : P.stream;
    cudaGraph_t graph = nullptr;
    double e_unused = 0.0;
    NKX_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    try {
      fock_build_once(P, precision, nspin, nocc, g->C, g->occ, NKX_MEM_DEVICE, fuse_j, &e_unused, g->V, g->J, s, 0,
                      nullptr, true);
    } catch (...) {
      cudaStreamEndCapture(s, &graph);
      if (graph) cudaGraphDestroy(graph);
      cudaGetLastError();
      g->failed = true;
      fock_build_once(P, precision, nspin, nocc, C, occ, NKX_MEM_DEVICE, fuse_j, E, V, J, user, 0, nullptr, false);
      return;
    }
    NKX_CUDA(cudaStreamEndCapture(s, &graph));
    const cudaError_t ie = cudaGraphInstantiate(&g->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) {
      cudaGetLastError();
      g->exec = nullptr;
      g->failed = true;
      fock_build_once(P, precision, nspin, nocc, C, occ, NKX_MEM_DEVICE, fuse_j, E, V, J, user, 0, nullptr, false);
      return;
    }
    g->launches = P.launches;
  }
  // replay
  cudaStream_t s = user ? user : P.stream;
  const size_t nn = (size_t)P.nbf * P.nbf;
  NKX_CUDA(cudaEventRecord(P.ev[0], s));
  NKX_CUDA(cudaMemcpyAsync(g->C, C, sizeof(double) * nspin * nocc * P.nbf, cudaMemcpyDeviceToDevice, s));
  NKX_CUDA(cudaMemcpyAsync(g->occ, occ, sizeof(double) * nspin * nocc, cudaMemcpyDeviceToDevice, s));
  NKX_CUDA(cudaGraphLaunch(g->exec, s));
  if (V) NKX_CUDA(cudaMemcpyAsync(V, g->V, sizeof(double) * nspin * nn, cudaMemcpyDeviceToDevice, s));
  if (J) NKX_CUDA(cudaMemcpyAsync(J, g->J, sizeof(double) * nn, cudaMemcpyDeviceToDevice, s));
  NKX_CUDA(cudaMemcpyAsync(P.h_result, P.d_E, sizeof(Plan::Result), cudaMemcpyDeviceToHost, s));
  NKX_CUDA(cudaEventRecord(P.ev[1], s));
  NKX_CUDA(cudaStreamSynchronize(s));
  *E = P.h_result->E;
  const int *status = P.h_result->status;
  P.last = nkx_build_timing{};
  cudaEventElapsedTime(&P.last.total_ms, P.ev[0], P.ev[1]);
  P.last.launches = g->launches;
  P.last_nspin = nspin;
  ++P.graph_replays;
  NKX_REQUIRE(status[0] == 0, NKX_ERR_TIMEOUT, "a tensor-core kernel wait gave up; outputs are invalid");
  NKX_REQUIRE(status[1] == 0 && std::isfinite(*E), NKX_ERR_NUMERIC,
              "non-finite value in the orbitals, occupations, grid or an operand of the build; outputs are invalid");
}

void fock_build(Plan &P, int precision, int nspin, int nocc, const double *C, const double *occ, int mem, int fuse_j,
                double *E, double *V, double *J, cudaStream_t user, int phase, double *y) {
  if (P.graph_mode && phase == 0 && mem == NKX_MEM_DEVICE) {
    NKX_REQUIRE(nspin == 1 || nspin == 2, NKX_ERR_ARG, "nspin must be 1 or 2");
    NKX_REQUIRE(nocc > 0 && C && occ && E && (V || J), NKX_ERR_ARG, "invalid arguments");
    fock_build_graph(P, precision, nspin, nocc, C, occ, fuse_j, E, V, J, user);
    return;
  }
  if (!P.graphs.empty()) P.drop_graphs();  // an ordinary build may grow buffers a graph uses
  fock_build_once(P, precision, nspin, nocc, C, occ, mem, fuse_j, E, V, J, user, phase, y, false);
}

}  // namespace nkx

using namespace nkx;

extern "C" {

NKX_API const char *nkx_last_error(void) { return g_last_error.c_str(); }

NKX_API nkx_status nkx_plan_create(const nkx_molecule *mol, const nkx_basis *prim, const nkx_basis *aux, long npoints,
                                   const double *xyz, const double *w, const int *owner, const nkx_plan_options *opts,
                                   nkx_plan **plan) {
  return run_guarded("nkx_plan_create", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan pointer is NULL");
    *plan = nullptr;
    auto P = std::make_unique<Plan>();
    build_plan(*P, mol, prim, aux, npoints, xyz, w, owner, opts);
    *plan = reinterpret_cast<nkx_plan *>(P.release());
  });
}

NKX_API nkx_status nkx_plan_get_info(const nkx_plan *plan, nkx_plan_info *info) {
  return run_guarded("nkx_plan_get_info", [&] {
    NKX_REQUIRE(plan && info, NKX_ERR_ARG, "invalid arguments");
    const Plan &P = *reinterpret_cast<const Plan *>(plan);
    info->npoints = P.npts;
    info->nbatches = P.nbatch;
    info->nbf = P.nbf;
    info->naux = P.naux;
    info->nblocks = P.nblk;
    info->npairs = P.npairs;
    info->nchunks = (int)P.chunks.size();
    info->metric_min_diag = P.metric_min_diag;
    info->graph_replays = P.graph_replays;
  });
}

NKX_API nkx_status nkx_fock_build(nkx_plan *plan, int precision, int nspin, int nocc, const double *C,
                                  const double *occ, int mem, int fuse_j, double *E, double *V, double *J,
                                  void *stream) {
  return run_guarded("nkx_fock_build", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    fock_build(P, precision, nspin, nocc, C, occ, mem, fuse_j, E, V, J, (cudaStream_t)stream);
  });
}

NKX_API nkx_status nkx_fock_build_phase1(nkx_plan *plan, int precision, int nspin, int nocc, const double *C,
                                         const double *occ, int mem, double *y, void *stream) {
  return run_guarded("nkx_fock_build_phase1", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    fock_build(P, precision, nspin, nocc, C, occ, mem, 0, nullptr, nullptr, nullptr, (cudaStream_t)stream, 1, y);
  });
}

NKX_API nkx_status nkx_fock_build_phase2(nkx_plan *plan, const double *y, int mem, int fuse_j, double *E, double *V,
                                         double *J, void *stream) {
  return run_guarded("nkx_fock_build_phase2", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    fock_build(P, 0, 0, 0, nullptr, nullptr, mem, fuse_j, E, V, J, (cudaStream_t)stream, 2, const_cast<double *>(y));
  });
}

NKX_API nkx_status nkx_plan_set_metric(nkx_plan *plan, const double *S, int mem) {
  return run_guarded("nkx_plan_set_metric", [&] {
    NKX_REQUIRE(plan && S, NKX_ERR_ARG, "invalid arguments");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    P.drop_graphs();
    NKX_REQUIRE(P.naux > 0, NKX_ERR_ARG, "the plan has no aux basis");
    NKX_REQUIRE(mem == NKX_MEM_DEVICE || mem == NKX_MEM_HOST, NKX_ERR_ARG, "mem must be NKX_MEM_DEVICE or NKX_MEM_HOST");
    const size_t NA = P.naux;
    P.h_metric.resize(NA * NA);
    NKX_CUDA(cudaMemcpy(P.h_metric.data(), S, sizeof(double) * NA * NA,
                        mem == NKX_MEM_HOST ? cudaMemcpyHostToHost : cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < NA; ++i)
      NKX_REQUIRE(std::isfinite(P.h_metric[i + i * NA]) && P.h_metric[i + i * NA] > 0, NKX_ERR_NUMERIC,
                  "metric diagonal must be positive and finite");
    // the mode chosen at plan creation (a caller's half inverse is replaced)
    P.svd_mode = P.metric_svd_thr > 0;
    if (P.svd_mode && !P.d_X) P.d_X = P.alloc<double>(NA * NA);
    factor_metric(P);
    NKX_CUDA(cudaStreamSynchronize(P.stream));
  });
}

NKX_API nkx_status nkx_get_last_timing(const nkx_plan *plan, nkx_build_timing *t) {
  return run_guarded("nkx_get_last_timing", [&] {
    NKX_REQUIRE(plan && t, NKX_ERR_ARG, "invalid arguments");
    *t = reinterpret_cast<const Plan *>(plan)->last;
  });
}

NKX_API nkx_status nkx_plan_last_density(const nkx_plan *plan, double *rho, long *perm) {
  return run_guarded("nkx_plan_last_density", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    const Plan &P = *reinterpret_cast<const Plan *>(plan);
    if (rho) {
      std::vector<double> h(2 * P.npad);
      NKX_CUDA(cudaMemcpy(h.data(), P.d_rho, sizeof(double) * 2 * P.npad, cudaMemcpyDeviceToHost));
      const int ns = std::max(1, P.last_nspin);
      for (long p = 0; p < P.npts; ++p)
        for (int s = 0; s < ns; ++s) rho[p * ns + s] = h[(size_t)s * P.npad + p];
    }
    if (perm)
      for (long p = 0; p < P.npts; ++p) perm[p] = P.perm[p];
  });
}

NKX_API nkx_status nkx_plan_batch_blocks(const nkx_plan *plan, int *counts) {
  return run_guarded("nkx_plan_batch_blocks", [&] {
    NKX_REQUIRE(plan && counts, NKX_ERR_ARG, "invalid arguments");
    const Plan &P = *reinterpret_cast<const Plan *>(plan);
    for (long b = 0; b < P.nbatch; ++b) counts[b] = P.h_pair_off[b + 1] - P.h_pair_off[b];
  });
}

NKX_API nkx_status nkx_plan_set_functional(nkx_plan *plan, int nfunc, const int *func_ids, double dens_threshold) {
  return run_guarded("nkx_plan_set_functional", [&] {
    NKX_REQUIRE(plan && func_ids, NKX_ERR_ARG, "invalid arguments");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    P.drop_graphs();
    nkx_plan_options o{};
    o.nfunc = nfunc;
    for (int i = 0; i < 4 && i < nfunc; ++i) o.func_ids[i] = func_ids[i];
    o.dens_threshold = dens_threshold;
    const XcSpec x = make_spec(&o);  // validates nfunc and the ids
    P.xc = x;
    P.gga = spec_is_gga(x);
  });
}

NKX_API nkx_status nkx_plan_set_half_inverse(nkx_plan *plan, int K, const double *X, int mem) {
  return run_guarded("nkx_plan_set_half_inverse", [&] {
    NKX_REQUIRE(plan && X, NKX_ERR_ARG, "invalid arguments");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    P.drop_graphs();
    NKX_REQUIRE(P.naux > 0, NKX_ERR_ARG, "the plan has no aux basis");
    NKX_REQUIRE(K >= 1 && K <= P.naux, NKX_ERR_ARG, "K must be in [1, naux]");
    NKX_REQUIRE(mem == NKX_MEM_DEVICE || mem == NKX_MEM_HOST, NKX_ERR_ARG, "mem must be NKX_MEM_DEVICE or NKX_MEM_HOST");
    const size_t NA = P.naux;
    if (!P.d_X) P.d_X = P.alloc<double>(NA * NA);
    if (!P.d_t) P.d_t = P.alloc<double>(NA);
    NKX_CUDA(cudaMemcpy(P.d_X, X, sizeof(double) * NA * K,
                        mem == NKX_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice));
    P.K = K;
    P.svd_mode = true;
  });
}

NKX_API nkx_status nkx_plan_set_wait_limit(nkx_plan *plan, unsigned long long ns, int stall) {
  return run_guarded("nkx_plan_set_wait_limit", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    P.drop_graphs();
    P.wait_ns = ns ? ns : 2000000000ull;
    P.stall_test = stall != 0;
  });
}

NKX_API nkx_status nkx_plan_set_graph(nkx_plan *plan, int enable) {
  return run_guarded("nkx_plan_set_graph", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    P.drop_graphs();
    P.graph_mode = enable != 0;
  });
}

NKX_API nkx_status nkx_plan_aux_metric(const nkx_plan *plan, double *S, int mem) {
  return run_guarded("nkx_plan_aux_metric", [&] {
    NKX_REQUIRE(plan && S, NKX_ERR_ARG, "invalid arguments");
    const Plan &P = *reinterpret_cast<const Plan *>(plan);
    NKX_REQUIRE(P.naux > 0, NKX_ERR_ARG, "the plan has no aux basis");
    NKX_REQUIRE(mem == NKX_MEM_DEVICE || mem == NKX_MEM_HOST, NKX_ERR_ARG, "mem must be NKX_MEM_DEVICE or NKX_MEM_HOST");
    const size_t bytes = sizeof(double) * P.naux * P.naux;
    if (mem == NKX_MEM_HOST)
      std::memcpy(S, P.h_metric.data(), bytes);
    else
      NKX_CUDA(cudaMemcpy(S, P.h_metric.data(), bytes, cudaMemcpyHostToDevice));
  });
}

NKX_API nkx_status nkx_plan_density(nkx_plan *plan, int nspin, int nocc, const double *C, const double *occ, int mem,
                                    int accumulate, double *rho, double *grad, double *sigma, void *stream) {
  return run_guarded("nkx_plan_density", [&] {
    NKX_REQUIRE(plan, NKX_ERR_ARG, "plan is NULL");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    NKX_REQUIRE(nspin == 1 || nspin == 2, NKX_ERR_ARG, "nspin must be 1 or 2");
    NKX_REQUIRE(nocc > 0 && C && occ && (rho || grad || sigma), NKX_ERR_ARG, "invalid arguments");
    NKX_REQUIRE(mem == NKX_MEM_DEVICE || mem == NKX_MEM_HOST, NKX_ERR_ARG, "mem must be NKX_MEM_DEVICE or NKX_MEM_HOST");
    cudaStream_t s = stream ? (cudaStream_t)stream : P.stream;
    const size_t n = (size_t)P.npts;
    if (!P.d_perm) {
      P.d_perm = P.alloc<long>(n);
      NKX_CUDA(cudaMemcpy(P.d_perm, P.perm.data(), sizeof(long) * n, cudaMemcpyHostToDevice));
    }
    NKX_CUDA(cudaMemsetAsync(P.d_status, 0, sizeof(int) * 2, s));
    upload_orbitals(P, nspin, nocc, C, occ, mem, s);
    // the gradient needs the gradient collocation whatever the functional
    const bool gga = P.gga;
    P.gga = grad || sigma;
    StageTimer T(P);
    try {
      fp64_density_pass(P, nspin, nocc, s, T);
    } catch (...) {
      P.gga = gga;
      throw;
    }
    P.gga = gga;
    // outputs: the caller's device buffers, or device staging for host ones
    double *orho = rho, *ograd = grad, *osig = sigma;
    if (mem == NKX_MEM_HOST) {
      if (!P.d_dens_out) P.d_dens_out = P.alloc<double>(2 * 5 * n);
      orho = rho ? P.d_dens_out : nullptr;
      ograd = grad ? P.d_dens_out + 2 * n : nullptr;
      osig = sigma ? P.d_dens_out + 8 * n : nullptr;
      if (accumulate && rho)
        NKX_CUDA(cudaMemcpyAsync(orho, rho, sizeof(double) * nspin * n, cudaMemcpyHostToDevice, s));
      if (accumulate && grad)
        NKX_CUDA(cudaMemcpyAsync(ograd, grad, sizeof(double) * 3 * nspin * n, cudaMemcpyHostToDevice, s));
    }
    density_out_kernel<<<dim3(nblk((long)n, 256), nspin), 256, 0, s>>>((long)n, P.npad, P.d_perm, P.d_rho, P.d_grad,
                                                                        accumulate != 0, orho, ograd, osig);
    NKX_LAUNCH_CHECK();
    if (mem == NKX_MEM_HOST) {
      if (rho) NKX_CUDA(cudaMemcpyAsync(rho, orho, sizeof(double) * nspin * n, cudaMemcpyDeviceToHost, s));
      if (grad) NKX_CUDA(cudaMemcpyAsync(grad, ograd, sizeof(double) * 3 * nspin * n, cudaMemcpyDeviceToHost, s));
      if (sigma) NKX_CUDA(cudaMemcpyAsync(sigma, osig, sizeof(double) * nspin * n, cudaMemcpyDeviceToHost, s));
    }
    int status[2] = {0, 0};
    NKX_CUDA(cudaMemcpyAsync(status, P.d_status, sizeof(status), cudaMemcpyDeviceToHost, s));
    NKX_CUDA(cudaStreamSynchronize(s));
    P.last_nspin = nspin;
    NKX_REQUIRE(status[1] == 0, NKX_ERR_NUMERIC, "non-finite value in the orbitals or occupations");
  });
}

NKX_API nkx_status nkx_plan_core_hamiltonian(nkx_plan *plan, const nkx_molecule *mol, double *S, double *T,
                                             double *V, int mem, void *stream) {
  return run_guarded("nkx_plan_core_hamiltonian", [&] {
    NKX_REQUIRE(plan && mol && mol->natoms > 0 && mol->xyz && mol->Z && S && T && V, NKX_ERR_ARG,
                "invalid arguments");
    NKX_REQUIRE(mem == NKX_MEM_DEVICE || mem == NKX_MEM_HOST, NKX_ERR_ARG, "mem must be NKX_MEM_DEVICE or NKX_MEM_HOST");
    Plan &P = *reinterpret_cast<Plan *>(plan);
    cudaStream_t s = stream ? (cudaStream_t)stream : P.stream;
    const size_t tile = (size_t)kBatch * kBlockF, nn = (size_t)P.nbf_pad * P.nbf_pad;
    std::vector<double> zc(mol->natoms);
    for (int a = 0; a < mol->natoms; ++a) zc[a] = mol->Z[a];
    double *dc = P.alloc<double>(3 * (size_t)mol->natoms), *dz = P.alloc<double>(mol->natoms);
    NKX_CUDA(cudaMemcpyAsync(dc, mol->xyz, sizeof(double) * 3 * mol->natoms, cudaMemcpyHostToDevice, s));
    NKX_CUDA(cudaMemcpyAsync(dz, zc.data(), sizeof(double) * mol->natoms, cudaMemcpyHostToDevice, s));
    if (!P.ws_z) P.ws_z = P.alloc<double>(std::max<long>(1, P.max_chunk_pairs) * 3 * tile);
    core_vne_kernel<<<nblk(P.npad, 256), 256, 0, s>>>(P.d_px, P.d_py, P.d_pz, P.d_w, P.npad, dc, dz, mol->natoms,
                                                     P.d_vj);
    NKX_LAUNCH_CHECK();
    NKX_CUDA(cudaMemsetAsync(P.d_V, 0, sizeof(double) * 3 * nn, s));
    // the collocation with gradients whatever the plan's functional
    const bool gga = P.gga;
    P.gga = true;
    try {
      for (const Chunk &c : P.chunks) {
        const long np = c.p1 - c.p0;
        if (np <= 0) continue;
        launch_colloc(P, c, s);
        // S (plane 0) and V_n (plane 1)
        core_z_kernel<<<(unsigned)np, 256, 0, s>>>(P.ws_phi, P.d_w, P.d_vj, P.d_pair_batch, c.p0, 0, P.ws_z);
        launch_vgemm_fp64(P, c, P.ws_phi, P.ws_z, 4, 3, 2, P.d_V, s);
        // T (plane 2): the three gradient components into one output
        core_z_kernel<<<(unsigned)np, 256, 0, s>>>(P.ws_phi, P.d_w, P.d_vj, P.d_pair_batch, c.p0, 1, P.ws_z);
        for (int k = 0; k < 3; ++k)
          launch_vgemm_fp64(P, c, P.ws_phi + (size_t)(k + 1) * tile, P.ws_z + (size_t)k * tile, 4, 3, 1,
                            P.d_V + 2 * nn, s);
        NKX_LAUNCH_CHECK();
      }
    } catch (...) {
      P.gga = gga;
      throw;
    }
    P.gga = gga;
    const size_t nb = (size_t)P.nbf * P.nbf;
    double *out = nullptr;
    if (mem == NKX_MEM_HOST) {
      if (!P.d_out) P.d_out = P.alloc<double>(3 * nb);
      out = P.d_out;
    }
    double *dst[3] = {mem == NKX_MEM_HOST ? out : S, mem == NKX_MEM_HOST ? out + nb : V,
                      mem == NKX_MEM_HOST ? out + 2 * nb : T};
    dim3 tb(16, 16), gb(nblk(P.nbf, 16), nblk(P.nbf, 16));
    for (int z = 0; z < 3; ++z)
      symmetrize_unpad_kernel<<<gb, tb, 0, s>>>(P.nbf, P.nbf_pad, P.d_finv, P.d_V + z * nn, dst[z]);
    NKX_LAUNCH_CHECK();
    if (mem == NKX_MEM_HOST) {
      NKX_CUDA(cudaMemcpyAsync(S, dst[0], sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
      NKX_CUDA(cudaMemcpyAsync(V, dst[1], sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
      NKX_CUDA(cudaMemcpyAsync(T, dst[2], sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
    }
    NKX_CUDA(cudaStreamSynchronize(s));
    P.release(dc);
    P.release(dz);
  });
}

NKX_API nkx_status nkx_morton_order(long npoints, const double *xyz, long *perm) {
  return run_guarded("nkx_morton_order", [&] {
    NKX_REQUIRE(npoints > 0 && xyz && perm, NKX_ERR_ARG, "invalid arguments");
    std::vector<long> p;
    morton_order(npoints, xyz, p);
    std::copy(p.begin(), p.end(), perm);
  });
}

NKX_API nkx_status nkx_aux_metric(const nkx_basis *aux, long npoints, const double *d_xyz, const double *d_w,
                                  double *d_S, void *stream) {
  return run_guarded("nkx_aux_metric", [&] {
    NKX_REQUIRE(aux && aux->nbf > 0 && npoints > 0 && d_xyz && d_w && d_S, NKX_ERR_ARG, "invalid arguments");
    for (int i = 0; i < aux->nbf; ++i)
      NKX_REQUIRE(aux->l[i] >= 0 && aux->l[i] <= 7 && aux->n[i] > aux->l[i] && abs(aux->m[i]) <= aux->l[i] &&
                      aux->zeta[i] > 0,
                  NKX_ERR_UNSUPPORTED, "aux function outside n > l, |m| <= l <= 7, zeta > 0");
    cudaStream_t s = (cudaStream_t)stream;
    const auto atab = make_aux_table(*aux);
    const auto astab = make_sto_table(*aux);
    auto del = [](void *q) { cudaFree(q); };
    std::unique_ptr<void, decltype(del)> a1(dalloc<AuxFunc>(aux->nbf), del), a2(dalloc<StoFunc>(aux->nbf), del),
        a3(dalloc<double>(3 * (size_t)npoints), del);
    AuxFunc *d_aux = static_cast<AuxFunc *>(a1.get());
    StoFunc *d_asto = static_cast<StoFunc *>(a2.get());
    double *soa = static_cast<double *>(a3.get());
    NKX_CUDA(cudaMemcpy(d_aux, atab.data(), sizeof(AuxFunc) * aux->nbf, cudaMemcpyHostToDevice));
    NKX_CUDA(cudaMemcpy(d_asto, astab.data(), sizeof(StoFunc) * aux->nbf, cudaMemcpyHostToDevice));
    split_points_kernel<<<nblk(npoints, 256), 256, 0, s>>>(npoints, d_xyz, soa);
    NKX_LAUNCH_CHECK();
    cublasHandle_t hb;
    NKX_REQUIRE(cublasCreate(&hb) == CUBLAS_STATUS_SUCCESS, NKX_ERR_CUDA, "cublasCreate failed");
    std::unique_ptr<cublasContext, decltype(&cublasDestroy)> hguard(hb, &cublasDestroy);
    cublasSetStream(hb, s);
    grid_metric(d_asto, d_aux, aux->nbf, soa, soa + npoints, soa + 2 * npoints, d_w, npoints, hb, s, d_S);
  });
}

NKX_API nkx_status nkx_plan_destroy(nkx_plan *plan) {
  return run_guarded("nkx_plan_destroy", [&] { delete reinterpret_cast<Plan *>(plan); });
}

}  // extern "C"
