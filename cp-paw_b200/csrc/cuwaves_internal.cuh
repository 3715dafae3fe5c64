// Internal state and device helpers of the cuwaves engine (sm_100a).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/cuwaves.h"

namespace cuw {

// ---------------------------------------------------------------------------
// error handling: every CUDA call is checked and turned into a status code
// ---------------------------------------------------------------------------
struct Status {
  int code = CUW_OK;
  std::string msg;
};

#define CUW_TRY(expr)                                              \
  do {                                                             \
    cudaError_t e__ = (expr);                                      \
    if (e__ != cudaSuccess) {                                      \
      cudaGetLastError(); /* not the next launch's error */        \
      return h->fail(CUW_ERR_CUDA, std::string(#expr) + ": " +     \
                                       cudaGetErrorString(e__));   \
    }                                                              \
  } while (0)

#define CUW_LAUNCH_CHECK(name)                                      \
  do {                                                              \
    ++h->launches;                                                  \
    cudaError_t e__ = cudaGetLastError();                           \
    if (e__ != cudaSuccess)                                         \
      return h->fail(CUW_ERR_CUDA, std::string(name) + ": " +       \
                                       cudaGetErrorString(e__));    \
  } while (0)

#define CUW_RET(expr)            \
  do {                           \
    int r__ = (expr);            \
    if (r__ != CUW_OK) return r__; \
  } while (0)

// Projector descriptor: IPRO -> (atom, bare projector column, LM, L)
struct ProDesc {
  int iat;
  int ibare;
  int lm;
  int l;
};

// FFT plan of one grid axis: radix sequence of a Stockham transform
struct AxisPlan {
  int n = 0;
  int nstage = 0;
  int radix[8] = {0};
};

// Device arrays of one wave-function set.
struct Device {
  // wave functions (ld = ldg complex numbers per band)
  double2 *psi0 = nullptr, *psim = nullptr, *hpsi = nullptr, *opsi = nullptr;
  double2 *proj = nullptr;       // (NBH, NPRO)
  double2 *oproj = nullptr;      // (NBH, NPRO) scratch
  double2 *hproj = nullptr;      // (NBH, NPRO) scratch
  double2 *pbuf = nullptr;       // (NBH, NPRO) scratch
  double2 *rlam0 = nullptr;      // (NB, NB) complex, Fortran layout
  double2 *rlamm = nullptr;
  // g-set
  int *igvec = nullptr;          // (3, NGL)
  int *minusg = nullptr;         // (NGL) 0-based
  double *gx = nullptr, *gy = nullptr, *gz = nullptr, *g2 = nullptr;
  double *pro = nullptr;         // (NGL, NBAREPRO)
  double *ylm = nullptr;         // (NGL, LMX)
  double *mpsi = nullptr;        // (NGL)
  double *rmpsi = nullptr;       // (NGL) 1 / MPSI
  double *bucket = nullptr;      // (NGL) or null
  ProDesc *pdesc = nullptr;      // (NPRO)
  // FFT
  int *plane_iz = nullptr;       // (nzp) occupied z planes
  int2 *plane_rows = nullptr;    // (nzp) first row and row count of the plane's G vectors
  int *plane_off = nullptr;      // (nzp+1) CSR offsets of the G lists
  int *plane_g = nullptr;        // (NGL) G index, grouped by plane
  int *plane_pos = nullptr;      // (NGL) ix + NR1*iy of that G
  int *zslot = nullptr;          // (NR3) compact plane index or -1
  double *v = nullptr;           // (NR1*NR2*NR3) local potential
  void *grid = nullptr;          // (batch, nzp, NR2, NR1) work grid, double2 or float2 (mixed)
  double* rho = nullptr;         // (NR) pseudo density of cuwaves_density (allocated on first use)
  double2 *tw1 = nullptr, *tw2 = nullptr, *tw3 = nullptr;  // twiddles exp(+2 pi i k/n)
  // atoms and one-centre data
  double *r0 = nullptr, *rp = nullptr, *rm = nullptr;  // (3, NAT)
  double *force = nullptr;       // (3, NAT)
  double *mass = nullptr;        // (NAT)
  double2 *eigr = nullptr;       // (NGL, NAT) structure factors of the last position set (G sets without parity)
  // folded arrays of the FP64 products (fold.cu): the +-G pairs of the sphere,
  // P(r,p) of the last position set (LDU, NPRO) and two slots of U(r,n) (LDU, NB)
  int2 *half = nullptr;
  double *prox = nullptr;
  double *uf = nullptr;
  // mixed path: the two slots of U in fp32, and the operands split into tf32 B
  // tiles: the two slots of U, and the small matrix of the product under way.
  // P(r,p) in fp32 lies in prox, and the split slots in uf: a product takes the
  // FP64 or the split form, and each is formed anew for the products that read it
  float *pf() const { return reinterpret_cast<float*>(prox); }
  float *bpre() const { return reinterpret_cast<float*>(uf); }
  float *u32 = nullptr;
  float *bsmall = nullptr;
  double *diag = nullptr;        // FP64 diagonals of the two slots' overlaps (mixed path)
  double *jac_a = nullptr;                   // packed matrix of the eigensolver when NB is too large for shared memory
  double2 *dh = nullptr;         // (LMNXX, LMNXX, NAT)
  double *dover = nullptr;       // (LNXX, LNXX, NSP)
  double *occ = nullptr;         // (NB)
  // orthogonalisation (real NB x NB)
  double *mat = nullptr, *omat = nullptr, *oomat = nullptr;
  double *lam = nullptr, *lam2 = nullptr, *lam0 = nullptr;  // lam0: start of a solve that may be redone
  double *u = nullptr, *u2 = nullptr, *eig = nullptr;
  double *haux = nullptr, *gamn = nullptr, *work = nullptr, *wk2 = nullptr;
  double *smat = nullptr, *emat = nullptr, *gt = nullptr, *xb = nullptr, *tb = nullptr;
  double *maxpart = nullptr;
  int *ostatus = nullptr;        // [0] status, [1] iterations
  int *smap = nullptr;           // (NB) state order of WAVES_ORTHO_Y_C (SAFEORTHO = F, SWAPSTATES = T)
  // (NGL) ANNEEVEC, 1 / (1 + ANNEEVEC) and GSET%DBUCKET of the cell friction
  double *anv = nullptr, *aninv = nullptr, *dbucket = nullptr;
  // scratch for split-K partial sums and band reductions
  double2 *part = nullptr;
  size_t part_bytes = 0;
  double *red = nullptr;         // reductions
  double *scal = nullptr;        // small scalar results
  // potential (POTENTIAL$VOFRHO): the density G set (one G of each +-G pair),
  // its tables and work arrays
  int *r_plus = nullptr, *r_minus = nullptr;   // (NGLH) grid offsets of +G and -G
  double *r_gx = nullptr, *r_gy = nullptr, *r_gz = nullptr, *r_g2 = nullptr;  // (NGLH)
  double *r_ylm = nullptr;                     // (LMRXX, NGLH) Y_lm(G) |G|^l
  double *r_g0 = nullptr, *r_v0 = nullptr, *r_pscore = nullptr, *r_vbar = nullptr;  // (NGLH, NSP)
  int *r_lmrx = nullptr;                       // (NSP)
  double *qlm = nullptr;                       // (LMRXX, NAT)
  double2 *r_rhog = nullptr, *r_vg = nullptr, *r_pot = nullptr, *r_vtot = nullptr;  // (NGLH)
  double2 *r_grid = nullptr;                   // (NR1*NR2*NR3) full complex grid
  double *r_part = nullptr;                    // block partial sums
  double *fpot = nullptr;                      // (3, NAT) Hartree and pseudo-core forces
  double *vqlm = nullptr;                      // (LMRXX, NAT)
  double *r_out = nullptr;                     // [0] EHARTREE [1] EXC [2] RHOB of the last cuwaves_vofrho
  // projector-map tables: first IPRO and #LMN per atom, species per atom,
  // (LN, M) of each IPRO, first LMN of each (species, LN), LOX (-1 = none)
  int *t_ipro0 = nullptr, *t_nlmn = nullptr, *t_isp = nullptr, *t_lnofp = nullptr, *t_mofp = nullptr,
      *t_lmn0ln = nullptr, *t_lox = nullptr;
};

struct Handle {
  cuw_dims d{};
  std::vector<int> isp;          // 0-based
  std::vector<int> lmnx, ibpro, ipro0;
  std::vector<ProDesc> pdesc;
  int npro = 0, nbarepro = 0, lmnxx = 0, lnxx = 0;
  int ldg = 0;                   // leading dimension of wave-function arrays
  int nh = 0, ldu = 0;           // +-G pairs of the sphere, leading dimension of folded arrays (>= 2 nh)
  bool sym = false;              // the G set's tables have the parity of real-valued projectors
  double gweight = 0.0;
  double gbas[9] = {0};
  std::vector<int> igvec_h;      // IGVEC(3,NGL) of the G set (restart records)
  double delt = 0.0, annee = 0.0;
  bool have_gset = false, have_v = false, have_dh = false, have_do = false;
  bool have_hpsi = false, have_rlamm = false, have_opsi = false, have_u = false;
  bool tbucket = false;
  bool async = false;
  // page-locked host block of cuwaves_cp_step's results (8 sums, the 16 status
  // words, the forces): one copy each and one wait per step
  double* res_h = nullptr;
  int band_bps[3] = {0, 0, 0};  // resident blocks per SM of the band-sum kernels (0: not yet queried)
  int nzp = 0;                   // occupied z planes
  int batch = 0;                 // bands per FFT batch
  int grid_bands = 0;            // bands the FFT work grid has room for
  // split-K factors of the projections and Gram products, as multiples of the
  // default (about two waves of CTAs); set by cuwaves_autotune
  double split_proj = 1.0, split_gram = 1.0;
  AxisPlan ax[3];
  int (*fft_run)(Handle*, const double2*, double2*, bool) = nullptr;  // chosen by fft_setup
  int (*fft_rho)(Handle*, const double2*, double*) = nullptr;          // density, chosen by fft_setup
  int fft_variant = 0;        // plan variant of the compiled FFT kernels (autotuner)
  int stream_prio = 0;        // 1: the stream has the device's highest priority
  bool fft_compiled = false;  // the grid has kernels compiled for its lengths
  size_t nr = 0;
  std::vector<double> occ_h;
  double waveekin1 = 0.0, waveekin2 = 0.0;
  cudaStream_t stream = nullptr;
  // nsm: SMs the launch shapes assume (the device's nsm_dev, or the share of a
  // set that runs beside others, CUW_OPT_SM_SHARE)
  int device = 0, nsm = 148, nsm_dev = 148;
  // CUDA graphs of cuwaves_cp_step.  A step's launches depend on host-side
  // state only through the PSI0/PSIM swap, the buffer EIGR was built from,
  // the Lagrange history flag and the arguments; one graph is kept per such
  // state (two in a run of steps).  `epoch` changes with every call that
  // could change what a step enqueues otherwise (inputs by value, scratch
  // reallocation, set-up routines), which retires the graphs.
  struct StepGraph {
    const void* key[6];
    int tabs = 0;
    int move = 0, max_iter = 0, rlamm = 0;
    double eps = 0.0;
    long long epoch = -1;
    const double* eigr_after = nullptr;  // the projector tables' source buffer after the step
    int tabs_after = 0;
    long long launches = 0;              // kernels in the graph
    cudaGraphExec_t exec = nullptr;
  };
  std::vector<StepGraph> graphs;
  long long epoch = 0;
  bool use_graphs = true;
  bool capturing = false;
  long long graph_replays = 0;
  void touch() { ++epoch; }
  void drop_graphs() {
    for (StepGraph& sg : graphs)
      if (sg.exec) cudaGraphExecDestroy(sg.exec);
    graphs.clear();
  }
  // measurement: kernel launches, and per-phase device time of cuwaves_cp_step
  long long launches = 0;
  bool timing = false;
  static constexpr int kPhases = 11;
  double phase_ms[kPhases] = {0};
  long long phase_calls = 0;
  std::vector<cudaEvent_t> ev;
  std::vector<int> ev_phase;
  int nev = 0;
  bool mixed() const { return d.precision == CUW_PREC_MIXED; }
  bool fp64_only = false;  // contractions in FP64 even on the mixed path (start-up orthonormalisation)
  // mixed path: the contractions on FP64 DMMA tiles (64 x 64, m8n8k4) instead
  // of the split-tf32 tcgen05 tiles (128 x 128 x 8); set by the autotuner or
  // CUW_OPT_CONTRACTION_TILES
  bool dmma_tiles = false;
  bool tc_on() const { return mixed() && !fp64_only && !dmma_tiles && sym; }
  // relative accuracy to which each ORTHO_X iteration solves its Lyapunov
  // equation (0: to rounding).  Measured on Si64 over 40 CP steps against the
  // solve to rounding: 1e-6 moves the FP64 total energy by 3e-12 Ha and the
  // forces by 1e-13 Ha/bohr with 40% of the sweeps; 1e-2 moves it by 6e-7 Ha
  // (1e-8 Ha/atom) and the forces by 1e-8 Ha/bohr with 16% of the sweeps, far
  // inside the mixed path's own error.
  double lyap_tol = 0.0;
  // WAVES$ORTHOGONALIZE branch (src/paw_waves1.f90:221-222): SAFEORTHO = T runs
  // WAVES_ORTHO_X, F runs WAVES_ORTHO_Y_C, in the order of the RLAM0 diagonal
  // when SWAPSTATES = T
  bool safeortho = true, swapstates = false;
  // cell friction of WAVES$PROPAGATE (cuwaves_set_cell_friction)
  bool fric_on = false, have_dbucket = false;
  double fricmat[9] = {0};
  double emass = 0.0, emasscg2 = 0.0;
  int lyap_max_sweeps = 64;  // sweeps per Lyapunov solve before the fixed point counts as failed
  bool ortho_panel = true;   // ORTHO_X by the panel-staged cluster kernel where it applies (64 < NB <= 128)
  // position buffer (r0, rp or rm) that the projector tables were built from,
  // and which of them (TAB_*, 0: none) is current for it
  const double* eigr_src = nullptr;
  int tabs = 0;
  // potential: density G set size, LMRXX, index of G = 0 (-1: none), and
  // whether cuwaves_cp_step forms V(r) from the density first
  int nglh = 0, lmrxx = 0, ngamma = -1;
  bool have_rhoset = false, have_qlm = false, scf = false;
  Device g;
  std::string err;

  int fail(int code, const std::string& m) {
    err = m;
    return code;
  }
  int sync() {
    if (async) return CUW_OK;
    cudaError_t e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return fail(CUW_ERR_CUDA, std::string("stream: ") + cudaGetErrorString(e));
    return tc_status();
  }
  // error flag of the tensor-core pipelines (a bounded wait that ran out)
  int tc_status() {
    if (!mixed()) return CUW_OK;
    int f = 0;
    cudaError_t e = cudaMemcpy(&f, g.ostatus + 12, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(CUW_ERR_CUDA, std::string("status: ") + cudaGetErrorString(e));
    return tc_flag(f);
  }
  int tc_flag(int f) {
    if (mixed() && f) return fail(CUW_ERR_CUDA, "tensor-core pipeline: a bounded wait ran out");
    return CUW_OK;
  }
  // Copy of n bytes of caller input to the device, ordered on the handle's
  // stream after the work enqueued before it.  Synchronous mode waits for it;
  // asynchronous mode only enqueues (the runtime stages a pageable buffer
  // before the call returns; a page-locked one is read when the stream gets
  // there, so the caller keeps it unchanged until cuwaves_synchronize).
  cudaError_t h2d(void* dst, const void* src, size_t n, bool wait = true) {
    cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess && wait && !async) e = cudaStreamSynchronize(stream);
    return e;
  }
  // the wait of synchronous mode after copies enqueued with h2d(..., false)
  cudaError_t h2d_done() { return async ? cudaSuccess : cudaStreamSynchronize(stream); }
  // set-up calls (new G set, new buffers) wait for the work in flight first
  cudaError_t settle() { return async ? cudaStreamSynchronize(stream) : cudaSuccess; }
};

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
// the same for float2 (FP32 transforms of the mixed-precision path)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// Sum over split-K partials for output i: scaled(sum of part[z][i], z < nz) + oc[z][i]
// (z < kc), every array n wide; scaled acts on each thread's share.  A block of 32 x kSumZ threads has kSumZ threads
// on each of 32 outputs, each with every kSumZ-th split (the outputs of small
// sets are too few to hide the latency of 140 splits one after another: the
// overlaps of 32 bands took 27 us and take 12); the result is valid in the threads with threadIdx.y == 0.
constexpr int kSumZ = 8;
__device__ __forceinline__ double2 split_get(const double2* p) { return *p; }
__device__ __forceinline__ double2 split_get(const float2* p) { return make_double2((double)p->x, (double)p->y); }
template <class P, class F>
__device__ __forceinline__ double2 split_sum(const P* __restrict__ part, int nz, size_t n, size_t i, F scaled,
                                             const double2* __restrict__ oc, int kc) {
  __shared__ double2 sh[kSumZ][32];
  double2 s = make_double2(0.0, 0.0);
  if (i < n) {
#pragma unroll 4
    for (int z = threadIdx.y; z < nz; z += kSumZ) s = cadd(s, split_get(part + (size_t)z * n + i));
    s = scaled(s);
#pragma unroll 4
    for (int z = threadIdx.y; z < kc; z += kSumZ) s = cadd(s, oc[(size_t)z * n + i]);
  }
  sh[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0) {
#pragma unroll
    for (int y = 1; y < kSumZ; ++y) s = cadd(s, sh[y][threadIdx.x]);
  }
  return s;
}
struct Scaled {
  double f;
  __device__ __forceinline__ double2 operator()(double2 s) const { return cscale(s, f); }
};

// (-i)^l
__device__ __forceinline__ double2 mipow(int l) {
  switch (l & 3) {
    case 0: return make_double2(1.0, 0.0);
    case 1: return make_double2(0.0, -1.0);
    case 2: return make_double2(-1.0, 0.0);
    default: return make_double2(0.0, 1.0);
  }
}

// PRO(g,p) = Y_lm(g) P_ln(|g|) (-i)^l EIGR(g,a) generated from the tables
// (WAVES_EXPANDPRO, src/paw_waves1.f90:6070-6109)
__device__ __forceinline__ double2 pro_value(int g, int ngl, const ProDesc& d, const double* __restrict__ ylm,
                                             const double* __restrict__ pro, const double2* __restrict__ eigr) {
  double s = ylm[(size_t)g + (size_t)ngl * d.lm] * pro[(size_t)g + (size_t)ngl * d.ibare];
  double2 e = cmul(mipow(d.l), eigr[(size_t)g + (size_t)ngl * d.iat]);
  return make_double2(s * e.x, s * e.y);
}

// coefficients of the fused ADDPRO epilogues (see k_addpro)
struct StepCoef {
  double a1, a2, a3, oscale;
  // 1 / (1 + ANNEEVEC(G)) of the G-dependent friction of a moving cell
  // (src/paw_waves1.f90:6536-6540) or null; with it the propagation coefficients
  // are formed per G from fr[g] and dt2 = DELT^2 instead of a1, a2, a3
  const double* fr = nullptr;
  double dt2 = 0.0;
};

// FP64 tensor-core MMA, m8n8k4, A row-major / B column-major fragments:
//   a = A[lane>>2][lane&3], b = B[lane&3][lane>>2],
//   c[0..1] = C[lane>>2][2*(lane&3)+0..1]
// The instruction needs the whole warp, converged.  `volatile` keeps the compiler
// from sinking it into code that only some lanes run (its result is often used
// there alone), and every block of products starts with a __syncwarp, because
// lanes that took different ways through the loads before need not have met again.
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}
// Elements i and i + 1 of a row at p (16-byte aligned, at least two elements), or
// zeros where !in: the load is unconditional, from the row's start if need be, so
// that no branch depends on the lane.
__device__ __forceinline__ double2 row2(const double* p, int i, bool in) {
  const double2 v = *reinterpret_cast<const double2*>(p + (in ? i : 0));
  return make_double2(in ? v.x : 0.0, in ? v.y : 0.0);
}
// A warp's 8 x 16 block of A B^T over n values of k (n even), straight from global
// memory (L2): c0 and c1 are its two 8 x 8 halves; a, b0, b1 the lane's rows
// (lane / 4) of the operands, k contiguous, and whether they are within them.  Lane
// k of a fragment takes two neighbouring values of k with one 16-byte load, which
// fills the fragments of two MMAs.  The sums are short, so what counts is loads in
// flight: those of the next 64 values are issued before the MMAs of the present
// ones (the __syncwarp, which no load may pass, would else put them behind the
// MMAs: 128 bands by 512 projectors take 10.7 us from cold caches, and took 12.4 so).
__device__ __forceinline__ void rows_8x16(const double* __restrict__ a, bool ain, const double* __restrict__ b0,
                                          bool in0, const double* __restrict__ b1, bool in1, int n, double (&c0)[2],
                                          double (&c1)[2]) {
  constexpr int U = 8, K = 8 * U;
  const int fk = threadIdx.x & 3;
  double2 av[2][U], v0[2][U], v1[2][U];
  auto load = [&](int s, int k0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + 8 * u + 2 * fk;
      av[s][u] = row2(a, k, ain && k < n);
      v0[s][u] = row2(b0, k, in0 && k < n);
      v1[s][u] = row2(b1, k, in1 && k < n);
    }
  };
  auto products = [&](int s) {
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      dmma(c0, av[s][u].x, v0[s][u].x);
      dmma(c1, av[s][u].x, v1[s][u].x);
      dmma(c0, av[s][u].y, v0[s][u].y);
      dmma(c1, av[s][u].y, v1[s][u].y);
    }
  };
  load(0, 0);
  for (int k0 = 0; k0 < n; k0 += 2 * K) {  // n is the same for the whole warp
    const bool second = k0 + K < n;
    if (second) load(1, k0 + K);
    products(0);
    if (k0 + 2 * K < n) load(0, k0 + 2 * K);
    if (second) products(1);
  }
}

// frees device buffers; what is not allocated again at once stays null
template <class... T>
inline void drop(T*&... p) {
  ((p ? (void)cudaFree(p) : (void)0, p = nullptr), ...);
}

// host helpers implemented in the .cu files
int fft_setup(Handle* h, const int* igvec_host);
int fft_vpsi(Handle* h, const double2* psi, double2* out, bool add_kinetic);
int fft_density(Handle* h, const double2* psi, double* rho);
int grid_fft(Handle* h, double2* grid, int dir);  // full-grid FP64 transform, unscaled
int fft_set_variant(Handle* h, int v);  // FFT plan variant of the compiled kernels
int fft_variants(const Handle* h);
int vofrho_run(Handle* h, const double* rho_dev);  // POTENTIAL$VOFRHO on the device
int denmat_run(Handle* h, int lmnxx, double2* denmat, double2* edenmat);
int eigr_compute(Handle* h, const double* r_dev);
int proj_compute(Handle* h, const double2* psiA, double2* projA, const double2* psiB, double2* projB,
                 bool folded = false);
int addpro_run(Handle* h, int mode, const double2* hpc, const double2* opc);
int hproj_compute(Handle* h, const double2* proj, double2* out);
int oproj_compute(Handle* h, const double2* proj, double2* out, const double2* proj2 = nullptr,
                  double2* out2 = nullptr);
int hoproj_compute(Handle* h, const double2* proj, double2* hout, double2* oout);
int ortho_solve(Handle* h, int max_iter, double eps);
int ortho_result(Handle* h, const int* st, int* iters);
int addoproj_run(Handle* h, double2* proj, const double2* oproj, const double* lam);
int band_reduce(Handle* h, int what, double* out_host, double* eig_host);
int force_run(Handle* h, double* force_host);
int force_gemm(Handle* h, const double2* ded, double* force_dev);
int small_tables_setup(Handle* h);
int gemm_setup(Handle* h);
// folded FP64 products (fold.cu); slots 0 and 1 hold folded wave-function arrays
struct FoldPair {
  int x, y;                // slots
  const double2 *px, *py;  // projections of x and DO * projections of y
};
int fold_setup(Handle* h, const std::vector<int>& minusg);
int fold_kernels_setup(Handle* h);
struct TcRooms {
  size_t split, u32, small, diag;  // bytes
};
struct FoldRooms {
  size_t uf, prox, eigr;  // prox for tables with parity, else eigr
  TcRooms tc;             // mixed path
};
size_t fold_bytes(Handle* h);
int fold_rooms(Handle* h);
int fold_table(Handle* h, const double* r_dev);
int fold_psi(Handle* h, const double2* psi, int slot);
int fold_proj(Handle* h, double2* proj0, double2* proj1);
// <x|O|y> of up to three pairs as real NB x NB matrices
int fold_gram(Handle* h, const FoldPair* pairs, int npair, double* o0, double* o1, double* o2);
// ADDPRO_FUSED leaves folded PSIM in slot 0 and OPSI in slot 1
int fold_addpro(Handle* h, int mode, const double2* hpc, const double2* opc, const StepCoef& sc);
int fold_addx(Handle* h, int slot, const double* lam, double2* out);
// the one-centre part of fold_gram alone: kc FP64 partial matrices per pair
int fold_oc_splits(const Handle* h, int npair);
int fold_oc(Handle* h, const FoldPair* pairs, int npair, int kc, double* oc);
int fold_force(Handle* h, const double2* ded, double* fpart, int* nt);
size_t part_bytes(const Handle* h);
size_t fold_part_bytes(const Handle* h);
size_t tc_part_bytes(const Handle* h);
int ensure_part(Handle* h, size_t bytes);  // split-K scratch h->g.part of at least `bytes`
// Raises (never lowers) the dynamic shared-memory limit of kernel fn on the
// current device.  The limit belongs to the function, so it is shared by all
// handles of the process: a handle of a smaller system must not lower the
// limit that a larger one launches with.
cudaError_t smem_allow(const void* fn, int bytes);
// split-precision (tf32 x3) tensor-core versions, used when tc_on(); tc_fold
// puts a wave-function array into a slot of U in fp32, tc_split forms the split
// B operands of slots 0 .. nset-1
int tc_setup(Handle* h);
TcRooms tc_room_sizes(const Handle* h);
int tc_clear_padding(Handle* h);
int tc_pro_table(Handle* h, const double* r_dev);
int tc_fold(Handle* h, const double2* psi, int slot);
int tc_split(Handle* h, int nset);
int tc_proj(Handle* h, double2* proj0, double2* proj1);
int tc_addpro(Handle* h, int mode, const double2* hpc, const double2* opc, const StepCoef& sc);
int tc_gram(Handle* h, const FoldPair* pairs, int npair, double* o0, double* o1, double* o2);
int tc_addx(Handle* h, int slot, const double* lam, double2* out);
int tc_force(Handle* h, const double2* ded, double* fpart, int* ntile);
int propagate_run(Handle* h);
int opsi_scale(Handle* h, double oscale);
int switch_lambda_run(Handle* h);
int gramschmidt_run(Handle* h, double2* psi, const double* r_dev);
int atoms_verlet_run(Handle* h, const double* mass_dev);

enum { TAB_EIGR = 1, TAB_F32 = 2, TAB_F64 = 4 };
enum { ADDPRO_HPSI = 0, ADDPRO_OPSI = 1, ADDPRO_FUSED = 2 };
enum { RED_EKIN = 0, RED_WAVEKIN = 1, RED_EXPECT = 2 };

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

}  // namespace cuw
