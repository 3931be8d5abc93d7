// The plan object behind nkx_plan (internal).
#pragma once

#include <cstdint>
#include <vector>

#include "functionals.cuh"
#include "potential.cuh"

namespace nkx {

struct Chunk {
  long b0 = 0, b1 = 0;  // batch range
  long p0 = 0, p1 = 0;  // (batch, block) pair range
  long t0 = 0, t1 = 0;  // range of the chunk's V output tiles in d_vtiles
  long u0 = 0, u1 = 0;  // range of its V pair tiles (row blocks 2R, 2R + 1) in d_vtiles2
};

// Choices of the mixed-precision build that the autotuner (nkx_plan_autotune)
// measures; the defaults are what it found best on (H2O)_64.
struct Tuning {
  int v_n = 128;   // tcgen05 MMA width N of the V contraction (128 or 64)
  int dens_n = 0;  // MMA width of the density contraction (64, 128, or 0: by orbital count, density_width)
  int ypath = -1;  // GGA density gradient through Y = T0 (C occ)^T: -1 from 256 orbitals, 0 off, 1 on
  int v_warps = 16; // epilogue warps of the N = 128 V contraction (16 of 32 columns, or 8 of 64)
  // V on CTA pairs (M = 256 x N = 64, double-buffered TMEM, v_warps
  // epilogue warps a CTA) instead of one CTA per tile
  int v_pair = 0;
};

// A Fock build recorded into a CUDA graph (graph mode) with the buffers it
// reads its orbitals from and writes its results to.
struct BuildGraph {
  int precision = 0, nspin = 0, nocc = 0, fuse = 0;
  bool hasV = false, hasJ = false, failed = false;
  cudaGraphExec_t exec = nullptr;
  double *C = nullptr, *occ = nullptr, *V = nullptr, *J = nullptr;
  int launches = 0;
};

struct Plan {
  int device = 0, nsm = 148;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  std::vector<cudaEvent_t> ev_pool;  // stage events, made on first use and kept
  size_t ev_used = 0;
  std::vector<void *> allocs;
  void *cublas = nullptr, *cusolver = nullptr;

  XcSpec xc{};
  bool gga = false;

  int nbf = 0, nbf_pad = 0, nblk = 0, mask_words = 0, naux = 0;
  long npts = 0, nbatch = 0, npad = 0, npairs = 0;
  std::vector<long> perm;  // plan point p <- caller point perm[p]

  // grid (Morton order, padded to nbatch * 256; padded points have w = 0)
  double *d_px = nullptr, *d_py = nullptr, *d_pz = nullptr, *d_w = nullptr;
  StoFunc *d_sto = nullptr;  // basis in plan order (see build_plan)
  std::vector<int> h_fperm;  // plan position -> caller function (-1: padding)
  int *d_fperm = nullptr, *d_finv = nullptr;
  StoShell *d_bshell = nullptr;  // radial shells per block [nblk][128]
  int *d_bnshell = nullptr, *d_fshell = nullptr;
  // atoms (for the nuclear gradient)
  int natoms = 0;
  std::vector<double> h_centers;
  double *d_centers = nullptr;
  int *d_fatom = nullptr;  // atom of each function, plan order
  int *d_owner = nullptr;  // owner atom of each point, plan order (null if not given)
  bool all_funcs_on_atoms = false;
  void *grad_state = nullptr;
  AuxFunc *d_aux = nullptr;
  AuxShell *d_ashell = nullptr;
  int nashell = 0;
  AuxGroup *d_agroup = nullptr;  // (centre, l) groups, sorted by l
  int nagroup = 0, nloose = 0;
  std::vector<int> h_group_off;  // groups of l = L at [off[L], off[L+1])
  int *d_loose = nullptr;        // shells outside the groups
  float *d_rtab = nullptr;       // FP32 radial factors [shell][point] of the mixed build's J
  bool rtab_failed = false;      // the table did not fit: the mixed J evaluates the factors

  // screening: pairs of (batch, significant function block), CSR by batch
  std::vector<int> h_pair_off;
  std::vector<uint32_t> h_mask;
  int *d_pair_off = nullptr, *d_pair_blk = nullptr, *d_pair_batch = nullptr;
  uint32_t *d_mask = nullptr;

  std::vector<Chunk> chunks;
  long max_chunk_pairs = 0, chunk_pair_limit = 0;
  // V output tiles (I << 16 | J) of each chunk that have at least one batch
  // with both blocks significant, heaviest first (plan_chunks)
  int *d_vtiles = nullptr;
  int *d_vtiles2 = nullptr;  // V pair tiles (R << 16 | J), by chunk
  Tuning tune;
  double *ws_phi = nullptr;  // PhiT tiles of a chunk: [pair][comp][g][f]
  double *ws_z = nullptr;    // Z^T tiles of a chunk:  [pair][z][g][f]

  // per point (two spins)
  double *d_rho = nullptr, *d_grad = nullptr, *d_coef = nullptr, *d_vj = nullptr;
  // orbitals
  int nocc_cap = 0;
  double *d_Ct = nullptr, *d_occ = nullptr, *d_Cin = nullptr;
  double *d_Cf = nullptr;  // function-major orbitals of the FP64 density pass
  size_t cf_cap = 0;
  // accumulators / outputs
  double *d_V = nullptr, *d_E = nullptr, *d_out = nullptr;
  double *d_vpart = nullptr;  // partial tiles of a split FP64 V contraction (4 nsm tiles)
  // caller-order density outputs (nkx_plan_density)
  long *d_perm = nullptr;
  double *d_dens_out = nullptr;

  // Coulomb metric
  bool svd_mode = false;
  double metric_svd_thr = 0.0;
  int K = 0, lwork = 0;
  double *d_L = nullptr, *d_X = nullptr, *d_t = nullptr, *d_y = nullptr, *d_c = nullptr, *d_work = nullptr;
  double *d_ypart = nullptr;  // per-slice shares of y
  int *d_info = nullptr, *d_piv = nullptr;
  std::vector<int> h_piv;
  double metric_min_diag = 0.0;
  std::vector<double> h_metric;

  // mixed-precision workspaces (tensor-core path)
  float *mx_phi = nullptr, *mx_a = nullptr, *mx_b = nullptr, *mx_c = nullptr;
  void *mx_state = nullptr;

  // build status words, zeroed by every build: [0] code of the first
  // tensor-core wait that gave up, [1] non-finite input or operand seen
  int *d_status = nullptr;
  // E_xc and the status words lie together on the device and come back in one
  // copy to page-locked memory (result_slot), or to own_result if there is none
  struct Result {
    double E;
    int status[2];
  } own_result{}, *h_result = &own_result;
  // limit of the device waits that may be abandoned (nkx_plan_set_wait_limit)
  unsigned long long wait_ns = 2000000000ull;
  int stall_test = 0;  // tests of the error path: tensor-core kernels wait on a barrier nothing completes
  // state kept between the two phases of a sharded build
  bool phase1_done = false;
  int phase1_precision = 0, phase1_nspin = 1, phase1_nocc = 0;

  // CUDA-graph replay of builds with device buffers (nkx_plan_set_graph)
  bool graph_mode = false;
  std::vector<BuildGraph> graphs;
  long graph_replays = 0;
  void drop_graphs();

  nkx_build_timing last{};
  int launches = 0;
  int last_nspin = 1;

  ~Plan();
  template <class T>
  T *alloc(size_t n);
  void release(void *p);  // frees one allocation made with alloc
};

void plan_chunks(Plan &P, long max_pairs);
// one Fock build, or phase 1 / 2 of a build on a sharded grid (plan.cu)
void fock_build(Plan &P, int precision, int nspin, int nocc, const double *C, const double *occ, int mem, int fuse_j,
                double *E, double *V, double *J, cudaStream_t user, int phase = 0, double *y = nullptr);
void destroy_mixed_state(void *p);

// Accumulates CUDA-event time per build stage, with the plan's events.
struct StageTimer {
  Plan &P;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> marks;
  cudaEvent_t begin_ev = nullptr;
  int cur = -1;
  bool on = true;  // off while a build is recorded into a CUDA graph
  explicit StageTimer(Plan &plan) : P(plan) { P.ev_used = 0; }
  cudaEvent_t next() {
    if (P.ev_used == P.ev_pool.size()) {
      cudaEvent_t e;
      NKX_CUDA(cudaEventCreate(&e));
      P.ev_pool.push_back(e);
    }
    return P.ev_pool[P.ev_used++];
  }
  void begin(int stage, cudaStream_t s) {
    if (!on) return;
    begin_ev = next();
    NKX_CUDA(cudaEventRecord(begin_ev, s));
    cur = stage;
  }
  void end(cudaStream_t s) {
    if (!on) return;
    const cudaEvent_t e = next();
    NKX_CUDA(cudaEventRecord(e, s));
    marks.push_back({cur, {begin_ev, e}});
  }
  void collect(float out[6]) {
    for (int i = 0; i < 6; ++i) out[i] = 0.f;
    for (auto &m : marks) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, m.second.first, m.second.second);
      out[m.first] += ms;
    }
  }
};

enum { ST_COLLOC = 0, ST_DENSITY = 1, ST_FUNC = 2, ST_COULOMB = 3, ST_ZBUILD = 4, ST_VGEMM = 5 };

bool mixed_available(const Plan &P);
void upload_orbitals(Plan &P, int nspin, int nocc, const double *C, const double *occ, int mem, cudaStream_t s);
void fp64_density_pass(Plan &P, int nspin, int nocc, cudaStream_t s, StageTimer &T);
int fp64_orbital_pad(int nocc, int *nn);
void fp64_density_begin(Plan &P, int nspin, int nocc, cudaStream_t s);
void fp64_density_range(Plan &P, long b0, long b1, long p0, int nspin, int nocc, double *T, cudaStream_t s);
void launch_colloc(Plan &P, const Chunk &c, cudaStream_t s);
void destroy_grad_state(void *p);
__global__ void functional_kernel(XcSpec s, bool gga, int nspin, long npad, long n, const double *__restrict__ w,
                                  const double *__restrict__ rho, const double *__restrict__ grad,
                                  const double *__restrict__ vj, double *__restrict__ coef, double *Eacc,
                                  double *__restrict__ edens);
// MMA width of the density contraction: the tuning's, or by default 128 from
// 1024 (padded) orbitals on -- half as many orbital tiles re-read each
// Phi tile (1500-atom aggregate, 2850 orbitals: 11.0 vs 12.0 s) -- else 64
// (two TMEM buffers; ahead for short orbital ranges)
inline int density_width(const Plan &P, int nocc) {
  if (P.tune.dens_n) return P.tune.dens_n;
  return ((nocc + 127) / 128) * 128 >= 1024 ? 128 : 64;
}
// CTAs a pair's points are split over (1 to 8) in the kernels that take a CTA
// of eight warps per (batch, block) pair: while there are fewer than eight an
// SM, the pairs alone leave SMs with a few warps whose latencies show (one
// water, 261 pairs: FP64 collocation 59 -> 42 us, Z operands 95 -> 42, pass A
// 67 -> 45)
inline unsigned point_split(long pairs, int nsm) {
  unsigned k = 1;
  while (k < 8 && pairs * k < 8L * nsm) k *= 2;
  return k;
}
// Units a V output tile's batches are dealt to: the fewest that fill nine
// tenths of the last wave of `nsm` CTAs, up to four waves (else the best
// found).  `parts` tiles alone leave SMs idle where a basis has few blocks
// (one water: 1 tile) or spill into a nearly empty wave ((H2O)_8 with a J
// plane: 18 tiles in 9 shares each took two waves for 162 units, 8 take one).
inline int batch_split(long parts, long nbatch, int nsm) {
  int nsplit = 1;
  double best = 0.0;
  for (long k = 1; parts > 0 && (k == 1 || (k <= nbatch && parts * k <= 4L * nsm)); ++k) {
    const double fill = (double)(parts * k) / (double)((parts * k + nsm - 1) / nsm * nsm);
    if (fill > best + 1e-9) {
      best = fill;
      nsplit = (int)k;
    }
    if (best >= 0.9) break;
  }
  return nsplit;
}
void mixed_gradient_begin(Plan &P, int nspin, int nocc, cudaStream_t s);
const double *mixed_gradient_chunk(Plan &P, const Chunk &c, int nspin, int nocc, double *edens, cudaStream_t s);
void fock_build_mixed(Plan &P, int nspin, int nocc, bool needJ, bool fuse, bool separateJ, cudaStream_t s,
                      StageTimer &T, int phase);
// mixed: read the aux radial factors from the plan's FP32 table (made on first use)
void coulomb_y(Plan &P, int nspin, cudaStream_t s, bool mixed);
void coulomb_solve(Plan &P, cudaStream_t s, bool mixed);

}  // namespace nkx
