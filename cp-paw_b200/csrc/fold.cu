// FP64 contractions of the Gamma-point path as real matrix products on the
// FP64 tensor cores (mma.sync m8n8k4 f64).
//
// A super wave function psi = phi1 + i phi2 holds two bands that are real in
// r (PLANEWAVE, src/paw_fft.f90:35-55), and every projector is real in r, so
// over a pair (G, -G) of the sphere
//   phi(-G) = conj phi(G),   p(-G) = conj p(G)
// and all contractions of the path are real products over half the sphere:
// with the folded array
//   U(2h,   2b..2b+1) = Re, Im of u = psi(G) + psi(-G)         (2 Re phi)
//   U(2h+1, 2b..2b+1) = Re, Im of w = -i (psi(G) - psi(-G))    (2 Im phi)
// for pair h, and the table P(2h, p) = Re p(G), P(2h+1, p) = Im p(G),
//   <p|psi>        = Omega   sum_r P(r,p) U(r,n)      (WAVES_PROJECTIONS)
//   <phi_m|phi_n>  = Omega/2 sum_r U(r,m) U(r,n)      (WAVES_OVERLAP)
//   sum_p p(G) c_p = s + i t, at -G: s - i t, with (s,t)(h) = sum_p P(r,p) c_p
//   phi' = phi + sum_m phi_m Lambda(m,n) likewise on U (WAVES_ADDOPSI)
// A G that is its own partner (G = 0) keeps U = psi in both rows: p is real
// there, and the two rows carry its half weight in the overlaps.
//
// This takes 2 real products per G, projector and super wave function where
// the complex form takes 4 (3 in the three-multiplication form), and half the
// table: on B200, Si64 (NGL 23847, 64 super wave functions, 512 projectors)
// the FP64 tensor pipe bounds both forms.
//
// The projectors satisfy p(-G) = conj p(G) whenever the tables of the G set do
// (Y_lm(-G) = (-1)^l Y_lm(G), P(|G|) even, G(-G) = -G(G)); fold_setup checks
// that to the last few bits and, where a caller's tables do not, leaves the
// projector contractions to the complex kernels of gemm.cu.  The overlaps and the
// rotation by Lambda need only MINUSG and are folded always.
//
// One CTA of 128 threads (2 x 2 warps) forms a tile of 16 MI x 16 NI outputs,
// K slices of 16 by 16-byte cp.async three deep, two CTAs per SM so that the
// prologue and epilogue of one run under the products of the other.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "cuwaves_internal.cuh"

namespace cuw {

namespace {

constexpr int RT = 128;   // threads of a CTA
constexpr int RK = 16;    // K values of a slice
constexpr int RS = 3;     // slices in flight
constexpr int RLD = 20;   // row stride of [row][k] tiles: fragment reads hit distinct banks

// Operand of a product: element (row, k) at p[row*ld + k] (K contiguous, KF)
// or p[row + k*ld].  Extents along the contiguous index are even and rows
// start on 16 bytes, so that elements travel in pairs.
struct Op {
  const double* p;
  long long ld;
  int n;  // rows
};

// doubles of a staged tile of ROWS rows (either layout fits)
template <int ROWS>
constexpr int tile_sz = ROWS * RLD > RK * (ROWS + 4) ? ROWS * RLD : RK * (ROWS + 4);
template <int MI, int NI>
constexpr size_t rsmem() {
  return sizeof(double) * RS * (size_t)(tile_sz<16 * MI> + tile_sz<16 * NI>);
}

__device__ const double2 g_zero[1] = {{0.0, 0.0}};

// 16 bytes to shared memory; zeros when src is null
__device__ __forceinline__ void cpa(double* dst, const double* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d),
               "l"(src ? src : reinterpret_cast<const double*>(g_zero)), "r"(src ? 16 : 0)
               : "memory");
}

// Copies of one thread for slices of ROWS rows of an operand from row0: element
// pairs at fixed distances from one pointer, so that a copy costs an add and a
// select (with an address formed from row and k for each, the main loop spent
// four integer instructions per MMA).  No branch depends on the lane: the warp
// stays converged for the MMAs.  K contiguous: rows tid/8 + 16 i, k = 2 (tid%8).
// Row contiguous: k = tid/8, rows 2 (tid%8) + 16 i.
template <bool KF, int ROWS>
struct Loader {
  const double* src;  // the thread's first pair of slice 0
  long long ld;
  int nrow;           // rows of the operand from the thread's first on
  __device__ __forceinline__ Loader(const double* p, long long ld_, int n, int row0, int kbeg) : ld(ld_) {
    const int q = threadIdx.x >> 3, e = 2 * (threadIdx.x & 7);
    const int row = row0 + (KF ? q : e), k = kbeg + (KF ? e : q);
    src = KF ? p + (long long)row * ld + k : p + row + (long long)k * ld;
    nrow = n - row;
  }
  // slice sl, whose K range holds kleft more values
  __device__ __forceinline__ void operator()(double* dst, int sl, int kleft) const {
    const int q = threadIdx.x >> 3, e = 2 * (threadIdx.x & 7);
    double* d = dst + (KF ? q * RLD + e : q * (ROWS + 4) + e);
    const double* s = src + (KF ? (long long)(sl * RK) : sl * (RK * ld));
    const int nr = (KF ? e : q) < kleft ? nrow : 0;
#pragma unroll
    for (int i = 0; i < ROWS / 16; ++i)
      cpa(d + i * (KF ? 16 * RLD : 16), 16 * i < nr ? s + (KF ? i * 16 * ld : (long long)(16 * i)) : nullptr);
  }
};
// the same for two row-contiguous sources of one shape side by side (H and O
// coefficients): the first half of the tile's rows from p, the second from p2
template <int ROWS>
struct Loader2 {
  Loader<false, ROWS / 2> a;
  const double* src2;
  __device__ __forceinline__ Loader2(const double* p, const double* p2, long long ld, int n, int row0)
      : a(p, ld, n, row0, 0), src2(p2 + (a.src - p)) {}
  __device__ __forceinline__ void operator()(double* dst, int sl, int kleft) const {
    const int q = threadIdx.x >> 3, e = 2 * (threadIdx.x & 7);
    double* d = dst + q * (ROWS + 4) + e;
    const double *s = a.src + sl * (RK * a.ld), *s2 = src2 + sl * (RK * a.ld);
    const int nr = q < kleft ? a.nrow : 0;
#pragma unroll
    for (int i = 0; i < ROWS / 32; ++i) {
      cpa(d + 16 * i, 16 * i < nr ? s + 16 * i : nullptr);
      cpa(d + ROWS / 2 + 16 * i, 16 * i < nr ? s2 + 16 * i : nullptr);
    }
  }
};
template <bool KF, int ROWS>
__device__ __forceinline__ double frag(const double* t, int row, int k) {
  if constexpr (KF) return t[row * RLD + k];
  else return t[k * (ROWS + 4) + row];
}

// acc += A B^T over nk values of K.  Warp (wm, wn) owns the 8 MI x 8 NI block
// at (wm, wn); acc[mi][ni][e] is element (8 mi + lane/4, 8 ni + 2 (lane%4) + e)
// of it.
template <int MI, int NI, bool AKF, bool BKF, class LA, class LB>
__device__ __forceinline__ void rloop(double* sm, const LA& la, const LB& lb, int nk, double (&acc)[MI][NI][2]) {
  constexpr int AR = 16 * MI, BR = 16 * NI, TA = tile_sz<AR>, ST = TA + tile_sz<BR>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wm = warp >> 1, wn = warp & 1;
  const int r8 = lane >> 2, c4 = lane & 3;
  const int nsl = (nk + RK - 1) / RK;
  auto issue = [&](int sl) {
    double* s = sm + (size_t)(sl % RS) * ST;
    la(s, sl, nk - sl * RK);
    lb(s + TA, sl, nk - sl * RK);
  };
#pragma unroll
  for (int sl = 0; sl < RS - 1; ++sl) {
    if (sl < nsl) issue(sl);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int sl = 0; sl < nsl; ++sl) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(RS - 2) : "memory");
    __syncthreads();
    if (sl + RS - 1 < nsl) issue(sl + RS - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    __syncwarp();
    const double* ta = sm + (size_t)(sl % RS) * ST;
    const double* tb = ta + TA;
#pragma unroll
    for (int ks = 0; ks < RK / 4; ++ks) {
      double av[MI], bv[NI];
#pragma unroll
      for (int i = 0; i < MI; ++i) av[i] = frag<AKF, AR>(ta, wm * 8 * MI + 8 * i + r8, 4 * ks + c4);
#pragma unroll
      for (int i = 0; i < NI; ++i) bv[i] = frag<BKF, BR>(tb, wn * 8 * NI + 8 * i + r8, 4 * ks + c4);
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) dmma(acc[i][j], av[i], bv[j]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
}

template <int MI, int NI, bool AKF, bool BKF>
__device__ __forceinline__ void rmain(double* sm, const Op& a, int m0, const Op& b, int n0, int kbeg, int kend,
                                      double (&acc)[MI][NI][2]) {
  const Loader<AKF, 16 * MI> la(a.p, a.ld, a.n, m0, kbeg);
  const Loader<BKF, 16 * NI> lb(b.p, b.ld, b.n, n0, kbeg);
  rloop<MI, NI, AKF, BKF>(sm, la, lb, kend - kbeg, acc);
}

// Tile of block blockIdx.x of a product over the sphere's rows: the column tiles of
// one row tile are neighbours (they share its rows of the table in L2).  One grid
// dimension for both, because only x takes more than 65535 row tiles (2.1 million
// plane waves in tiles of 32 rows).
__device__ __forceinline__ void tile_of_block(int ncol, int& row, int& col) {
  row = blockIdx.x / ncol;
  col = blockIdx.x - row * ncol;
}

template <int MI, int NI>
__device__ __forceinline__ void azero(double (&acc)[MI][NI][2]) {
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
}

// ---------------------------------------------------------------------------
// tables: symmetry of the G set, folded wave functions, folded projectors
// ---------------------------------------------------------------------------
// Parity to within kParityUlp units in the last place (of |G|, of the radial
// value, and of 1 for the spherical harmonics, which cancel near their nodal
// planes): a host's vectorised or fused arithmetic need not give both signs of G
// the same bits.  The folded table then takes the values at one of the two, which
// changes the projectors by less than the phase exp(-iG.R) is rounded.  With bit
// equality asked for, one such value sent the whole set to the complex kernels (a
// CP step of Si64 takes 2.57 ms there against 1.59 in FP64, and 2.38 against 1.02
// on the mixed path).
constexpr double kParityUlp = 8 * 2.220446049250313e-16;
__device__ __forceinline__ bool near(double a, double b, double scale) { return fabs(a - b) <= kParityUlp * scale; }

__global__ void k_sym_check(int ngl, int nbare, int lmx, const int* __restrict__ minusg, const double* __restrict__ gx,
                            const double* __restrict__ gy, const double* __restrict__ gz,
                            const double* __restrict__ ylm, const double* __restrict__ pro, int* __restrict__ bad) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ngl) return;
  const int m = minusg[g];
  const double len = fabs(gx[g]) + fabs(gy[g]) + fabs(gz[g]);
  bool ok = near(gx[m], -gx[g], len) && near(gy[m], -gy[g], len) && near(gz[m], -gz[g], len);
  for (int i = 0; i < nbare; ++i) {
    const double p = pro[(size_t)g + (size_t)ngl * i];
    ok = ok && near(pro[(size_t)m + (size_t)ngl * i], p, fabs(p));
  }
  for (int l = 0; l * l < lmx; ++l)
    for (int i = l * l; i < min(lmx, (l + 1) * (l + 1)); ++i) {
      const double y = ylm[(size_t)g + (size_t)ngl * i];
      ok = ok && near(ylm[(size_t)m + (size_t)ngl * i], (l & 1) ? -y : y, 1.0);
    }
  if (!ok) *bad = 1;
}

// U(r, n) of a wave-function array, n-th row at u + n*ldu: bound by HBM (48 MB
// for Si64)
__global__ void k_fold(const double2* __restrict__ psi, const int2* __restrict__ half, int nh, int ldg, int ldu,
                       double* __restrict__ u) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (h >= nh) return;
  const int2 g = half[h];
  const double2* p = psi + (size_t)ldg * b;
  const double2 x = p[g.x], y = p[g.y];
  double2 re, im;  // (u, w) of the real and of the imaginary part
  if (g.x == g.y) {
    re = make_double2(x.x, x.x);
    im = make_double2(x.y, x.y);
  } else {
    re = make_double2(x.x + y.x, x.y - y.y);
    im = make_double2(x.y + y.y, y.x - x.x);
  }
  double* o = u + (size_t)ldu * (2 * b) + 2 * h;
  *reinterpret_cast<double2*>(o) = re;
  *reinterpret_cast<double2*>(o + ldu) = im;
}

__global__ void k_scale(double2* __restrict__ psi, const double* __restrict__ w, int ngl, int ldg, double f) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ngl) return;
  double2* p = psi + (size_t)ldg * blockIdx.y + g;
  *p = cscale(*p, w[g] * f);
}

// P(r, p) of every projector at the positions r (WAVES_EXPANDPRO,
// src/paw_waves1.f90:6070-6109), p-th row at tab + p*ldu: one thread per
// (pair, atom) forms exp(-iG.R) and writes the atom's projectors
__global__ void k_pro_fold(int nh, int ngl, int ldu, const int2* __restrict__ half, const double* __restrict__ gx,
                           const double* __restrict__ gy, const double* __restrict__ gz, const double* __restrict__ r,
                           const int* __restrict__ ipro0, const int* __restrict__ nlmn,
                           const ProDesc* __restrict__ pdesc, const double* __restrict__ ylm,
                           const double* __restrict__ pro, double* __restrict__ tab) {
  const int a = blockIdx.y, h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= nh) return;
  const int g = half[h].x, p0 = ipro0[a], np = nlmn[a];
  double sn, cs;
  sincos(gx[g] * r[3 * a] + gy[g] * r[3 * a + 1] + gz[g] * r[3 * a + 2], &sn, &cs);
  const double2 ei = make_double2(cs, -sn);
  for (int k = 0; k < np; ++k) {
    const ProDesc d = pdesc[p0 + k];
    const double sv = ylm[(size_t)g + (size_t)ngl * d.lm] * pro[(size_t)g + (size_t)ngl * d.ibare];
    const double2 e = cmul(mipow(d.l), ei);
    *reinterpret_cast<double2*>(tab + (size_t)ldu * (p0 + k) + 2 * h) = make_double2(sv * e.x, sv * e.y);
  }
}

// ---------------------------------------------------------------------------
// <p|psi>: part[z][p][n] = sum_{r in split z} P(r,p) U(r,n)
// ---------------------------------------------------------------------------
template <int MI, int NI>
__global__ void __launch_bounds__(RT, 2) k_rproj(Op p, Op u, int kchunk, int nr, double* __restrict__ part) {
  extern __shared__ __align__(16) double rsm[];
  const int n0 = blockIdx.x * 16 * NI, m0 = blockIdx.y * 16 * MI;
  const int kbeg = blockIdx.z * kchunk, kend = min(nr, kbeg + kchunk);
  double acc[MI][NI][2];
  azero(acc);
  rmain<MI, NI, true, true>(rsm, p, m0, u, n0, kbeg, kend, acc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int m = m0 + (warp >> 1) * 8 * MI + 8 * i + (lane >> 2);
    if (m >= p.n) continue;
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int n = n0 + (warp & 1) * 8 * NI + 8 * j + 2 * (lane & 3);
      if (n < u.n)
        *reinterpret_cast<double2*>(part + ((size_t)blockIdx.z * p.n + m) * u.n + n) =
            make_double2(acc[i][j][0], acc[i][j][1]);
    }
  }
}

// PROJ(b, p) of one or two wave-function arrays (nbh super wave functions each);
// the split sums are those of split_sum (cuwaves_internal.cuh)
__global__ void __launch_bounds__(32 * kSumZ)
    k_rproj_sum(const double2* __restrict__ part, int nz, int nbh, int nset, int npro, double scale,
                double2* __restrict__ out0, double2* __restrict__ out1) {
  const int nw = nset * nbh;
  const size_t n = (size_t)nw * npro, i = blockIdx.x * (size_t)32 + threadIdx.x;
  const double2 s = split_sum(part, nz, n, i, Scaled{scale}, (const double2*)nullptr, 0);
  if (threadIdx.y || i >= n) return;
  const int b = (int)(i % nw);
  const size_t p = i / nw;
  (b < nbh ? out0 : out1)[(b < nbh ? b : b - nbh) + (size_t)nbh * p] = s;
}

// ---------------------------------------------------------------------------
// Overlaps of up to three pairs: part[z][pair][i][j], z < ks: the plane-wave
// sum over split z of U(r,i) V(r,j); z >= ks: the one-centre sum over split z - ks
// of the projectors of P_x(i,p) (DO P_y)(j,p)  (WAVES_OVERLAP + WAVES_1COVERLAP,
// src/paw_waves2.f90:761-1022)
// ---------------------------------------------------------------------------
struct RGramArgs {
  const double* x[3];   // U rows of the pairs
  const double* y[3];
  const double* px[3];  // projections, real view (n + NB p)
  const double* py[3];
  int npair, nb, npro, nr, ldu, kchunk, ks, pchunk;
};
template <int MI, int NI>
__global__ void __launch_bounds__(RT, 2) k_rgram(RGramArgs a, double* __restrict__ part) {
  extern __shared__ __align__(16) double rsm[];
  const int pair = blockIdx.z % a.npair, z = blockIdx.z / a.npair;
  const int n0 = blockIdx.x * 16 * NI, m0 = blockIdx.y * 16 * MI;
  auto of = [pair](const double* const(&v)[3]) { return pair == 0 ? v[0] : (pair == 1 ? v[1] : v[2]); };
  double acc[MI][NI][2];
  azero(acc);
  if (z < a.ks) {
    const Op x{of(a.x), a.ldu, a.nb}, y{of(a.y), a.ldu, a.nb};
    rmain<MI, NI, true, true>(rsm, x, m0, y, n0, z * a.kchunk, min(a.nr, (z + 1) * a.kchunk), acc);
  } else {
    const Op x{of(a.px), a.nb, a.nb}, y{of(a.py), a.nb, a.nb};
    const int k0 = (z - a.ks) * a.pchunk;
    rmain<MI, NI, false, false>(rsm, x, m0, y, n0, k0, min(a.npro, k0 + a.pchunk), acc);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int m = m0 + (warp >> 1) * 8 * MI + 8 * i + (lane >> 2);
    if (m >= a.nb) continue;
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int n = n0 + (warp & 1) * 8 * NI + 8 * j + 2 * (lane & 3);
      if (n < a.nb)
        *reinterpret_cast<double2*>(part + ((size_t)blockIdx.z * a.nb + m) * a.nb + n) =
            make_double2(acc[i][j][0], acc[i][j][1]);
    }
  }
}

// out_pair(i + NB j) = scale * the ks plane-wave parts + the kc one-centre parts
__global__ void __launch_bounds__(32 * kSumZ)
    k_rgram_sum(const double2* __restrict__ part, int ks, int kc, int nb, int npair, double scale,
                double* __restrict__ o0, double* __restrict__ o1, double* __restrict__ o2) {
  const size_t per = (size_t)nb * nb / 2, n = per * npair, t = blockIdx.x * (size_t)32 + threadIdx.x;
  const double2 s = split_sum(part, ks, n, t, Scaled{scale}, part + (size_t)ks * n, kc);
  if (threadIdx.y || t >= n) return;
  const int pair = (int)(t / per);
  const size_t e = 2 * (t % per);
  const int i = (int)(e / nb), j = (int)(e % nb);
  double* o = pair == 0 ? o0 : (pair == 1 ? o1 : o2);
  o[i + (size_t)nb * j] = s.x;
  o[i + (size_t)nb * (j + 1)] = s.y;
}

// The complex value at this lane's G from the row values v = (Re, Im) of a
// pair: even rows hold s and take G (s + i t), odd rows hold t and take -G
// (s - i t); the rows of a pair are four lanes apart.
__device__ __forceinline__ double2 unfold(double2 v, bool odd) {
  double2 o;
  o.x = __shfl_xor_sync(0xffffffffu, v.x, 4);
  o.y = __shfl_xor_sync(0xffffffffu, v.y, 4);
  return odd ? make_double2(o.x + v.y, o.y - v.x) : make_double2(v.x - o.y, v.y + o.x);
}
// the row value of U (u of even rows, w of odd rows) from this lane's psi
__device__ __forceinline__ double2 refold(double2 v, bool odd, bool self) {
  double2 o;
  o.x = __shfl_xor_sync(0xffffffffu, v.x, 4);
  o.y = __shfl_xor_sync(0xffffffffu, v.y, 4);
  if (self) return odd ? o : v;
  return odd ? make_double2(o.y - v.y, v.x - o.x) : make_double2(v.x + o.x, v.y + o.y);
}

// ---------------------------------------------------------------------------
// ADDPRO with the step epilogues (WAVES_ADDPRO, src/paw_waves1.f90:5908-6067;
// WAVES$HPSI :4793-4916, WAVES_OPSI :5043-5096, the mass scaling of
// src/paw_waves2.f90:140-162 and WAVES$PROPAGATE :6575-6583).
//   k_raddpro      : out = base + P C (H|psi>: base = out = V psi; O|psi>: base =
//                    psi0, scaled by the mass afterwards)
//   k_raddpro_step : both with C1 and C2 of the same bands in one tile, then
//                    psim = a1 psi0 + a2 psim + a3/m_G hpsi.  The folded psim
//                    and opsi that the projections and overlaps at R(+) need
//                    are written on the way (um, uo).
// ---------------------------------------------------------------------------
template <int MI, int NI>
__global__ void __launch_bounds__(RT, 2) k_raddpro(Op p, Op c, int npro, const double2* base, double2* out,
                                                   const int2* __restrict__ half, int nh, int ldg, int nbh) {
  extern __shared__ __align__(16) double rsm[];
  int tm, tn;
  tile_of_block((c.n + 16 * NI - 1) / (16 * NI), tm, tn);
  const int m0 = tm * 16 * MI, n0 = tn * 16 * NI;
  double acc[MI][NI][2];
  azero(acc);
  rmain<MI, NI, false, false>(rsm, p, m0, c, n0, 0, npro, acc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = n0 + (warp & 1) * 8 * NI;
  const bool odd = (lane >> 2) & 1;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = m0 + (warp >> 1) * 8 * MI + 8 * i + (lane >> 2);
    const bool rok = r < 2 * nh;
    const int2 gp = rok ? half[r >> 1] : make_int2(0, 0);
    const bool mine = rok && !(odd && gp.x == gp.y);
    const int g = odd ? gp.y : gp.x;
    double2 x[NI];
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int b = (nw + 8 * j) / 2 + (lane & 3);
      x[j] = base[mine && b < nbh ? (size_t)g + (size_t)ldg * b : 0];
    }
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int b = (nw + 8 * j) / 2 + (lane & 3);
      const double2 v = unfold(make_double2(acc[i][j][0], acc[i][j][1]), odd);
      if (mine && b < nbh) out[(size_t)g + (size_t)ldg * b] = cadd(x[j], v);
    }
  }
}

struct RStepArgs {
  double2 *hpsi, *opsi, *psim;
  const double2* psi0;
  const double* rmpsi;
  const int2* half;
  double *um, *uo;
  int ldg, ldu, nh, nbh;
  StepCoef sc;
};
template <int MI, int NI>
__global__ void __launch_bounds__(RT, 2) k_raddpro_step(RStepArgs a, Op p, Op c1, Op c2, int npro) {
  extern __shared__ __align__(16) double rsm[];
  int tm, tn;
  tile_of_block((c1.n + 8 * NI - 1) / (8 * NI), tm, tn);
  const int m0 = tm * 16 * MI, n0 = tn * 8 * NI;
  double acc[MI][NI][2];
  azero(acc);
  const Loader<false, 16 * MI> la(p.p, p.ld, p.n, m0, 0);
  const Loader2<16 * NI> lb(c1.p, c2.p, c1.ld, c1.n, n0);
  rloop<MI, NI, false, false>(rsm, la, lb, npro, acc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool hcol = (warp & 1) == 0;  // the left warps hold the H products, the right ones the O products
  const bool odd = (lane >> 2) & 1;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = m0 + (warp >> 1) * 8 * MI + 8 * i + (lane >> 2);
    const bool rok = r < 2 * a.nh;
    const int2 gp = rok ? a.half[r >> 1] : make_int2(0, 0);
    const bool self = gp.x == gp.y, mine = rok && !(odd && self);
    const int g = odd ? gp.y : gp.x;
    const double rm = a.rmpsi[g];
    double a1 = a.sc.a1, a2 = a.sc.a2, a3 = a.sc.a3 * rm;
    if (a.sc.fr) {  // cell friction ANNEEVEC(G) (src/paw_waves1.f90:6536-6540)
      const double ai = a.sc.fr[g];
      a1 = 2.0 * ai;
      a2 = 1.0 - a1;
      a3 = -a.sc.dt2 * ai * rm;
    }
    const double os = a.sc.oscale * rm;
    constexpr int KB = NI < 4 ? NI : 4;  // columns whose loads are in flight together
#pragma unroll
    for (int j0 = 0; j0 < NI; j0 += KB) {
      double2 x0[KB], x1[KB], x2[KB];
#pragma unroll
      for (int q = 0; q < KB; ++q) {
        const int b = (n0 + 8 * (j0 + q)) / 2 + (lane & 3);
        const size_t k = mine && b < a.nbh ? (size_t)g + (size_t)a.ldg * b : 0;
        x1[q] = a.psi0[k];
        x0[q] = hcol ? a.hpsi[k] : make_double2(0.0, 0.0);
        x2[q] = hcol ? a.psim[k] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int q = 0; q < KB; ++q) {
        const int b = (n0 + 8 * (j0 + q)) / 2 + (lane & 3);
        const bool bok = b < a.nbh, ok = mine && bok;
        const size_t k = (size_t)g + (size_t)a.ldg * b;
        const double2 v = unfold(make_double2(acc[i][j0 + q][0], acc[i][j0 + q][1]), odd);
        double2 res;  // psi(+) or O psi at this lane's G
        if (hcol) {
          const double2 hv = cadd(x0[q], v);
          res = make_double2(a1 * x1[q].x + a2 * x2[q].x + a3 * hv.x, a1 * x1[q].y + a2 * x2[q].y + a3 * hv.y);
          if (ok) {
            a.hpsi[k] = hv;
            a.psim[k] = res;
          }
        } else {
          res = make_double2((x1[q].x + v.x) * os, (x1[q].y + v.y) * os);
          if (ok) a.opsi[k] = res;
        }
        const double2 f = refold(res, odd, self);
        if (rok && bok) {
          double* u = (hcol ? a.um : a.uo) + (size_t)a.ldu * (2 * b) + r;
          u[0] = f.x;
          u[a.ldu] = f.y;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// psi(+) += O|psi0> Lambda (WAVES_ADDOPSI, src/paw_waves2.f90:547-615; the PSI
// update of WAVES_GRAMSCHMIDT :2131-2136): U of the operand times the real
// Lambda (m + NB n), unfolded into out
// ---------------------------------------------------------------------------
template <int MI, int NI>
__global__ void __launch_bounds__(RT, 2) k_raddx(Op u, Op lam, double2* __restrict__ out,
                                                 const int2* __restrict__ half, int nh, int ldg, int nbh) {
  extern __shared__ __align__(16) double rsm[];
  int tm, tn;
  tile_of_block((lam.n + 16 * NI - 1) / (16 * NI), tm, tn);
  const int m0 = tm * 16 * MI, n0 = tn * 16 * NI;
  double acc[MI][NI][2];
  azero(acc);
  rmain<MI, NI, false, true>(rsm, u, m0, lam, n0, 0, 2 * nbh, acc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = n0 + (warp & 1) * 8 * NI;
  const bool odd = (lane >> 2) & 1;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = m0 + (warp >> 1) * 8 * MI + 8 * i + (lane >> 2);
    const bool rok = r < 2 * nh;
    const int2 gp = rok ? half[r >> 1] : make_int2(0, 0);
    const bool self = gp.x == gp.y, mine = rok && !(odd && self);
    const int g = odd ? gp.y : gp.x;
    double2 old[NI];
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int b = (nw + 8 * j) / 2 + (lane & 3);
      old[j] = out[mine && b < nbh ? (size_t)g + (size_t)ldg * b : 0];
    }
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int b = (nw + 8 * j) / 2 + (lane & 3);
      const double2 w = make_double2(acc[i][j][0], acc[i][j][1]), v = unfold(w, odd);
      if (mine && b < nbh)
        out[(size_t)g + (size_t)ldg * b] = self ? cadd(old[j], w) : make_double2(old[j].x + 0.5 * v.x, old[j].y + 0.5 * v.y);
    }
  }
}

// ---------------------------------------------------------------------------
// Forces (WAVES_DEDPRO + WAVES_PROFORCE, src/paw_waves1.f90:5694-5743,
// 6112-6234): D(r,p) = sum_n U(r,n) E(n,p), and with it
//   f_p = sum_h G_h (Re p Im D - Im p Re D) = sum_r +-P(r^1,p) D(r,p) G
// (the factor 2 of U stands for the pair).  A CTA walks every gridDim.x-th
// row tile of its projector tile; fpart(blockIdx.x, p, c).
// ---------------------------------------------------------------------------
template <int MI, int NI>
__global__ void __launch_bounds__(RT, 2) k_rforce(Op u, Op ded, const double* __restrict__ tab,
                                                  const int2* __restrict__ half, int nh, int ldu,
                                                  const double* __restrict__ gx, const double* __restrict__ gy,
                                                  const double* __restrict__ gz, int nb, double* __restrict__ fpart) {
  extern __shared__ __align__(16) double rsm[];
  __shared__ double fsum[2][16 * NI][3];  // of the two warp rows
  const int n0 = blockIdx.y * 16 * NI, npro = ded.n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wm = warp >> 1, wn = warp & 1;
  const int r8 = lane >> 2, c4 = lane & 3;
  // sums over G in batches of JB column blocks: NV values of a lane (2 JB
  // projectors by three components, padded to a multiple of eight)
  constexpr int JB = NI < 4 ? NI : 4, NV = (6 * JB + 7) / 8 * 8;
  double sum[NI / JB][NV / 8];
#pragma unroll
  for (int i = 0; i < NI / JB * (NV / 8); ++i) (&sum[0][0])[i] = 0.0;
  const int nt = (2 * nh + 16 * MI - 1) / (16 * MI);
  for (int t = blockIdx.x; t < nt; t += gridDim.x) {
    const int m0 = t * 16 * MI + wm * 8 * MI + r8;
    // the table values of the tile, loaded before the products so that their
    // latency lies under the MMAs (after them, one dependent load per pair of
    // columns, they took as long as the products)
    double pv[MI][NI][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = m0 + 8 * i, p = n0 + wn * 8 * NI + 8 * j + 2 * c4 + e;
          pv[i][j][e] = (p < npro && r < 2 * nh) ? tab[(size_t)ldu * p + (r ^ 1)] : 0.0;
        }
    double acc[MI][NI][2];
    azero(acc);
    rmain<MI, NI, false, true>(rsm, u, t * 16 * MI, ded, n0, 0, nb, acc);
    double gv[MI][3];
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int r = m0 + 8 * i;
      const int g = r < 2 * nh ? half[r >> 1].x : 0;
      const double sg = (r & 1) ? 1.0 : -1.0;  // (rows past the sphere have zero table values)
      gv[i][0] = sg * gx[g];
      gv[i][1] = sg * gy[g];
      gv[i][2] = sg * gz[g];
    }
#pragma unroll
    for (int jb = 0; jb < NI / JB; ++jb) {
      double v[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) v[i] = 0.0;
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < JB; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const double sv = pv[i][jb * JB + j][e] * acc[i][jb * JB + j][e];
#pragma unroll
            for (int c = 0; c < 3; ++c) v[3 * (2 * j + e) + c] += sv * gv[i][c];
          }
      // sums over the eight rows of a column (lanes four apart): every exchange
      // halves the values a lane keeps
#pragma unroll
      for (int w = NV / 2, d = 16; d >= 4; d >>= 1, w >>= 1) {
        const bool up = lane & d;
#pragma unroll
        for (int i = 0; i < NV / 2; ++i)
          if (i < w) {
            const double give = up ? v[i] : v[i + w];
            const double keep = up ? v[i + w] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, d);
          }
      }
#pragma unroll
      for (int i = 0; i < NV / 8; ++i) sum[jb][i] += v[i];
    }
  }
  // index of the lane's first value: the bits of its row from the first exchange down
  const int v0 = ((lane >> 4) & 1) * (NV / 2) + ((lane >> 3) & 1) * (NV / 4) + ((lane >> 2) & 1) * (NV / 8);
#pragma unroll
  for (int jb = 0; jb < NI / JB; ++jb)
#pragma unroll
    for (int i = 0; i < NV / 8; ++i) {
      const int k = v0 + i, je = k / 3;
      if (k < 6 * JB) fsum[wm][wn * 8 * NI + 8 * (jb * JB + (je >> 1)) + 2 * c4 + (je & 1)][k % 3] = sum[jb][i];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * NI * 3; i += RT) {
    const int pl = i / 3, c = i % 3, p = n0 + pl;
    if (p < npro) fpart[((size_t)blockIdx.x * npro + p) * 3 + c] = fsum[0][pl][c] + fsum[1][pl][c];
  }
}

// PROJ(n, p) += sum_m O(m, p) Lambda(m, n) on the real views (n + NB p) of the
// projection arrays (WAVES_ADDOPROJ, src/paw_waves2.f90:687-758), 8 n x 16 p a
// warp: 128 bands and 512 projectors take 10.7 us (19.5 through shared memory, 32
// values of m at a time).
__global__ void __launch_bounds__(128) k_raddoproj(double* __restrict__ out, const double* __restrict__ x,
                                                   const double* __restrict__ lam, int npro, int nb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fk = lane & 3;
  const int n0 = (blockIdx.y * 4 + warp) * 8, p0 = blockIdx.x * 16;
  if (n0 >= nb) return;  // the whole warp
  const bool an = n0 + fr < nb, b0 = p0 + fr < npro, b1 = p0 + 8 + fr < npro;
  const double* la = lam + (size_t)nb * (an ? n0 + fr : 0);
  const double* x0 = x + (size_t)nb * (b0 ? p0 + fr : 0);
  const double* x1 = x + (size_t)nb * (b1 ? p0 + 8 + fr : 0);
  double old[4], c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
  const int n = n0 + fr;
  auto col = [&](int k) { return p0 + 8 * (k >> 1) + 2 * fk + (k & 1); };
#pragma unroll
  for (int k = 0; k < 4; ++k) old[k] = an && col(k) < npro ? out[n + (size_t)nb * col(k)] : 0.0;  // under the products
  rows_8x16(la, an, x0, b0, x1, b1, nb, c0, c1);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (an && col(k) < npro) out[n + (size_t)nb * col(k)] = old[k] + (k < 2 ? c0[k] : c1[k - 2]);
}

}  // namespace

// Tile families (MI, NI): 64 or 48 rows of the sphere by 128 columns, and 32 by
// 64 or 32 for few bands, whose columns a wide tile would leave empty.
// Tile for `cols` real columns and `rows` rows of the long dimension on nsm
// SMs: the columns fix NI; of the row tiles, the one whose busiest SM has the
// fewest rows (a product of 374 tiles of 64 rows on 148 SMs keeps some SMs at
// three tiles and the average at 2.5).
struct RTile {
  int mi, ni;
};
static RTile pick_tile(const Handle* h, int rows, int cols) {
  if (cols <= 32) return {2, 2};
  if (cols <= 64) return {2, 4};
  const int ct = ceil_div(cols, 128);
  auto load = [&](int mi) { return ceil_div(ceil_div(rows, 16 * mi) * ct, h->nsm) * 16 * mi; };
  return {load(3) < load(4) ? 3 : 4, 8};
}
// products whose K splits even out the waves use the 64-row tile only
#define RTILE_SWITCH_K(T, LAUNCH)                  \
  do {                                             \
    if ((T).ni == 2) { LAUNCH(2, 2); }             \
    else if ((T).ni == 4) { LAUNCH(2, 4); }        \
    else { LAUNCH(4, 8); }                         \
  } while (0)
#define RTILE_SWITCH_F(T, LAUNCH)                  \
  do {                                             \
    if ((T).ni == 2) { LAUNCH(2, 2); }             \
    else if ((T).ni == 4) { LAUNCH(2, 4); }        \
    else { LAUNCH(3, 8); }                         \
  } while (0)
#define RTILE_SWITCH(T, LAUNCH)                    \
  do {                                             \
    if ((T).ni == 2) { LAUNCH(2, 2); }             \
    else if ((T).ni == 4) { LAUNCH(2, 4); }        \
    else if ((T).mi == 3) { LAUNCH(3, 8); }        \
    else { LAUNCH(4, 8); }                         \
  } while (0)

// K splits of a product of `tiles` output tiles: at most two CTAs per SM and
// wave (rounded down: a CTA past a whole wave would cost a wave of its own)
static int rsplit(const Handle* h, int tiles, int nk, double mul) {
  const int want = std::max(1, (int)std::floor(2.0 * h->nsm * mul / std::max(1, tiles)));
  return std::min(want, std::max(1, ceil_div(nk, 128)));
}

int fold_setup(Handle* h, const std::vector<int>& mg) {
  Device& g = h->g;
  const int ngl = h->d.ngl;
  std::vector<int2> half;
  half.reserve(ngl / 2 + 1);
  for (int i = 0; i < ngl; ++i)
    if (i <= mg[i]) half.push_back(make_int2(i, mg[i]));
  const int nh = (int)half.size(), ldu = ceil_div(2 * nh, 32) * 32;
  if (nh != h->nh) {
    drop(g.half, g.uf, g.prox, g.u32, g.bsmall, g.diag);
    h->nh = 0;  // an allocation that fails is made again by the next set-up
    CUW_TRY(cudaMalloc(&g.half, sizeof(int2) * nh));
    h->nh = nh;
    h->ldu = ldu;
  }
  CUW_TRY(cudaMemcpy(g.half, half.data(), sizeof(int2) * nh, cudaMemcpyHostToDevice));
  int bad = 0;
  int* flag = g.ostatus + 13;
  CUW_TRY(cudaMemsetAsync(flag, 0, sizeof(int), h->stream));
  k_sym_check<<<ceil_div(ngl, 256), 256, 0, h->stream>>>(ngl, h->nbarepro, h->d.lmx, g.minusg, g.gx, g.gy, g.gz, g.ylm,
                                                         g.pro, flag);
  CUW_LAUNCH_CHECK("k_sym_check");
  CUW_TRY(cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  CUW_TRY(cudaStreamSynchronize(h->stream));
  h->sym = bad == 0;
  CUW_RET(fold_rooms(h));
  return ensure_part(h, part_bytes(h));
}

// Buffers whose sizes follow from the folded sphere: two folded wave-function
// arrays (rows of slot 1 follow slot 0's; on the mixed path the split forms lie in
// the same buffer), the projector table (FP64 or fp32) or, for tables without
// parity, EIGR, and what else the tensor-core products need.  No later call
// allocates them, so that no step captured into a graph does.
static FoldRooms room_sizes(const Handle* h) {
  FoldRooms r{};
  r.uf = sizeof(double) * (size_t)h->ldu * h->d.nb * 2;
  r.prox = sizeof(double) * (size_t)h->ldu * h->npro;
  r.eigr = sizeof(double2) * (size_t)h->d.ngl * std::max(1, h->d.nat);
  if (h->mixed()) {
    r.tc = tc_room_sizes(h);
    r.uf = std::max(r.uf, r.tc.split);  // whatever the parity: a later G set of the same size keeps the buffer
  }
  return r;
}

// bytes of all of them and of the split-sum scratch, whatever the tables' parity;
// of the handle only the sizes are read
size_t fold_bytes(Handle* h) {
  const FoldRooms r = room_sizes(h);
  const bool sym = h->sym;
  size_t n = 0;
  for (bool s : {false, true}) {
    h->sym = s;
    n = std::max(n, part_bytes(h) + (s ? r.prox + r.tc.u32 + r.tc.small + r.tc.diag : r.eigr));
  }
  h->sym = sym;
  return sizeof(int2) * h->nh + r.uf + n;
}

int fold_rooms(Handle* h) {
  auto room = [&](auto*& p, size_t bytes, const char* what) -> int {
    if (p || bytes == 0) return CUW_OK;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
      return h->fail(CUW_ERR_NOMEM, std::string("cudaMalloc of the ") + what + " failed");
    }
    return CUW_OK;
  };
  Device& g = h->g;
  const FoldRooms r = room_sizes(h);
  CUW_RET(room(g.uf, r.uf, "folded wave functions"));
  if (!h->sym) return room(g.eigr, r.eigr, "structure factors");
  CUW_RET(room(g.prox, r.prox, "projector table"));
  if (!h->mixed()) return CUW_OK;
  const bool fresh = !g.u32;
  CUW_RET(room(g.u32, r.tc.u32, "fp32 folded wave functions"));
  CUW_RET(room(g.bsmall, r.tc.small, "split matrices"));
  CUW_RET(room(g.diag, r.tc.diag, "overlap diagonals"));
  return fresh ? tc_clear_padding(h) : CUW_OK;
}

static double* slot_ptr(const Handle* h, int slot) { return h->g.uf + (size_t)slot * h->d.nb * h->ldu; }

int fold_psi(Handle* h, const double2* psi, int slot) {
  k_fold<<<dim3(ceil_div(h->nh, 256), h->d.nbh), 256, 0, h->stream>>>(psi, h->g.half, h->nh, h->ldg, h->ldu,
                                                                      slot_ptr(h, slot));
  CUW_LAUNCH_CHECK("k_fold");
  return CUW_OK;
}

int fold_table(Handle* h, const double* r_dev) {
  const Device& g = h->g;
  k_pro_fold<<<dim3(ceil_div(h->nh, 256), h->d.nat), 256, 0, h->stream>>>(h->nh, h->d.ngl, h->ldu, g.half, g.gx, g.gy,
                                                                          g.gz, r_dev, g.t_ipro0, g.t_nlmn, g.pdesc,
                                                                          g.ylm, g.pro, g.prox);
  CUW_LAUNCH_CHECK("k_pro_fold");
  return CUW_OK;
}

// tile and K splits of the projections of nset arrays, and the bytes of their sums
struct ProjSplit {
  RTile t;
  int ks, kchunk;
  size_t bytes;
};
static ProjSplit proj_split(const Handle* h, int nset) {
  const int nt = h->d.nb * nset, npro = h->npro, nr = 2 * h->nh;
  ProjSplit s;
  s.t = pick_tile(h, npro, nt);
  s.t.mi = s.t.ni == 8 ? 4 : 2;
  const int tiles = ceil_div(nt, 16 * s.t.ni) * ceil_div(npro, 16 * s.t.mi);
  s.kchunk = ceil_div(ceil_div(nr, rsplit(h, tiles, nr, h->split_proj)), RK) * RK;
  s.ks = ceil_div(nr, s.kchunk);
  s.bytes = sizeof(double) * (size_t)s.ks * nt * npro;
  return s;
}

// PROJ of slot 0 (and slot 1 when proj1 is given)
int fold_proj(Handle* h, double2* proj0, double2* proj1) {
  const int nset = proj1 ? 2 : 1, nt = h->d.nb * nset, npro = h->npro, nr = 2 * h->nh;
  if (npro == 0) return CUW_OK;
  const ProjSplit s = proj_split(h, nset);
  const RTile t = s.t;
  const int ks = s.ks, kchunk = s.kchunk;
  CUW_RET(ensure_part(h, s.bytes));
  double* part = reinterpret_cast<double*>(h->g.part);
  const Op p{h->g.prox, h->ldu, npro}, u{h->g.uf, h->ldu, nt};
  const dim3 grid(ceil_div(nt, 16 * t.ni), ceil_div(npro, 16 * t.mi), ks);
#define L(MI, NI) k_rproj<MI, NI><<<grid, RT, rsmem<MI, NI>(), h->stream>>>(p, u, kchunk, nr, part)
  RTILE_SWITCH_K(t, L);
#undef L
  CUW_LAUNCH_CHECK("k_rproj");
  const size_t n = (size_t)nt / 2 * npro;
  k_rproj_sum<<<(unsigned)((n + 31) / 32), dim3(32, kSumZ), 0, h->stream>>>(
      h->g.part, ks, h->d.nbh, nset, npro, h->gweight, proj0, proj1);
  CUW_LAUNCH_CHECK("k_rproj_sum");
  return CUW_OK;
}

static int gram_args(Handle* h, const FoldPair* pairs, int npair, RGramArgs* a) {
  if (npair < 1 || npair > 3) return h->fail(CUW_ERR_ARG, "overlaps: one to three pairs");
  *a = RGramArgs{};
  for (int i = 0; i < npair; ++i) {
    a->x[i] = slot_ptr(h, pairs[i].x);
    a->y[i] = slot_ptr(h, pairs[i].y);
    a->px[i] = reinterpret_cast<const double*>(pairs[i].px);
    a->py[i] = reinterpret_cast<const double*>(pairs[i].py);
  }
  a->npair = npair;
  a->nb = h->d.nb;
  a->npro = h->npro;
  a->nr = 2 * h->nh;
  a->ldu = h->ldu;
  return CUW_OK;
}
static RTile gram_tile(const Handle* h) {
  RTile t = pick_tile(h, h->d.nb, h->d.nb);
  t.mi = t.ni == 8 ? 4 : 2;
  return t;
}
static int gram_launch(Handle* h, const RGramArgs& a, RTile t, int nz, double* part) {
  const dim3 grid(ceil_div(a.nb, 16 * t.ni), ceil_div(a.nb, 16 * t.mi), nz * a.npair);
#define L(MI, NI) k_rgram<MI, NI><<<grid, RT, rsmem<MI, NI>(), h->stream>>>(a, part)
  RTILE_SWITCH_K(t, L);
#undef L
  CUW_LAUNCH_CHECK("k_rgram");
  return CUW_OK;
}

// splits of the overlaps of npair pairs, and the bytes of their sums
struct GramSplit {
  int ks, kchunk, kc, pchunk;
  size_t bytes;
};
static GramSplit gram_split(const Handle* h, int npair) {
  const RTile t = gram_tile(h);
  const int nb = h->d.nb, npro = h->npro, nr = 2 * h->nh;
  const int tiles = ceil_div(nb, 16 * t.ni) * ceil_div(nb, 16 * t.mi) * npair;
  // the one-centre sums take splits of about the same length
  const int ks0 = rsplit(h, tiles, nr, h->split_gram);
  GramSplit s;
  s.pchunk = std::max(RK, ceil_div(std::min(npro, ceil_div(nr, ks0)), RK) * RK);
  s.kc = ceil_div(npro, s.pchunk);
  s.kchunk = ceil_div(ceil_div(nr, std::max(1, ks0 - s.kc)), RK) * RK;
  s.ks = ceil_div(nr, s.kchunk);
  s.bytes = sizeof(double) * (size_t)(s.ks + s.kc) * npair * nb * nb;
  return s;
}

int fold_gram(Handle* h, const FoldPair* pairs, int npair, double* o0, double* o1, double* o2) {
  RGramArgs a;
  CUW_RET(gram_args(h, pairs, npair, &a));
  const RTile t = gram_tile(h);
  const GramSplit s = gram_split(h, npair);
  a.pchunk = s.pchunk;
  a.kchunk = s.kchunk;
  a.ks = s.ks;
  const int ks = s.ks, kc = s.kc, nb = a.nb;
  CUW_RET(ensure_part(h, s.bytes));
  CUW_RET(gram_launch(h, a, t, ks + kc, reinterpret_cast<double*>(h->g.part)));
  const size_t n = (size_t)nb * nb / 2 * npair;
  k_rgram_sum<<<(unsigned)((n + 31) / 32), dim3(32, kSumZ), 0, h->stream>>>(h->g.part, ks, kc, nb, npair,
                                                                            0.5 * h->gweight, o0, o1, o2);
  CUW_LAUNCH_CHECK("k_rgram_sum");
  return CUW_OK;
}

// one wave of CTAs, at least 32 projectors each
int fold_oc_splits(const Handle* h, int npair) {
  const RTile t = gram_tile(h);
  const int nb = h->d.nb, tiles = ceil_div(nb, 16 * t.ni) * ceil_div(nb, 16 * t.mi) * npair;
  const int want = std::max(1, std::min(2 * h->nsm / std::max(1, tiles), ceil_div(h->npro, 32)));
  return ceil_div(h->npro, std::max(RK, ceil_div(ceil_div(h->npro, want), RK) * RK));
}
int fold_oc(Handle* h, const FoldPair* pairs, int npair, int kc, double* oc) {
  if (kc == 0) return CUW_OK;
  RGramArgs a;
  CUW_RET(gram_args(h, pairs, npair, &a));
  a.pchunk = ceil_div(ceil_div(a.npro, kc), RK) * RK;
  return gram_launch(h, a, gram_tile(h), kc, oc);
}

// opsi *= oscale / m_G (src/paw_waves2.f90:140-162)
int opsi_scale(Handle* h, double oscale) {
  k_scale<<<dim3(ceil_div(h->d.ngl, 256), h->d.nbh), 256, 0, h->stream>>>(h->g.opsi, h->g.rmpsi, h->d.ngl, h->ldg,
                                                                         oscale);
  CUW_LAUNCH_CHECK("k_scale");
  return CUW_OK;
}

int fold_addpro(Handle* h, int mode, const double2* hpc, const double2* opc, const StepCoef& sc) {
  Device& g = h->g;
  const int nb = h->d.nb, npro = h->npro;
  const Op p{g.prox, h->ldu, 2 * h->nh};
  if (mode == ADDPRO_FUSED) {
      const RStepArgs a{g.hpsi, g.opsi, g.psim, g.psi0, g.rmpsi, g.half, slot_ptr(h, 0), slot_ptr(h, 1),
                      h->ldg, h->ldu, h->nh, h->d.nbh, sc};
    const Op c1{reinterpret_cast<const double*>(hpc), nb, nb}, c2{reinterpret_cast<const double*>(opc), nb, nb};
    const RTile t = pick_tile(h, 2 * h->nh, 2 * nb);
    const int grid = ceil_div(2 * nb, 16 * t.ni) * ceil_div(2 * h->nh, 16 * t.mi);
#define L(MI, NI) k_raddpro_step<MI, NI><<<grid, RT, rsmem<MI, NI>(), h->stream>>>(a, p, c1, c2, npro)
    RTILE_SWITCH(t, L);
#undef L
    CUW_LAUNCH_CHECK("k_raddpro_step");
    return CUW_OK;
  }
  const bool o = mode == ADDPRO_OPSI;
  const Op c{reinterpret_cast<const double*>(o ? opc : hpc), nb, nb};
  const RTile t = pick_tile(h, 2 * h->nh, nb);
  const int grid = ceil_div(nb, 16 * t.ni) * ceil_div(2 * h->nh, 16 * t.mi);
#define L(MI, NI)                                                                                              \
  k_raddpro<MI, NI><<<grid, RT, rsmem<MI, NI>(), h->stream>>>(p, c, npro, o ? g.psi0 : g.hpsi, o ? g.opsi : g.hpsi, \
                                                              g.half, h->nh, h->ldg, h->d.nbh)
  RTILE_SWITCH(t, L);
#undef L
  CUW_LAUNCH_CHECK("k_raddpro");
  return o ? opsi_scale(h, sc.oscale) : CUW_OK;
}

int fold_addx(Handle* h, int slot, const double* lam, double2* out) {
  const int nb = h->d.nb;
  const Op u{slot_ptr(h, slot), h->ldu, 2 * h->nh}, l{lam, nb, nb};
  const RTile t = pick_tile(h, 2 * h->nh, nb);
  const int grid = ceil_div(nb, 16 * t.ni) * ceil_div(2 * h->nh, 16 * t.mi);
#define L(MI, NI)                                                                                             \
  k_raddx<MI, NI><<<grid, RT, rsmem<MI, NI>(), h->stream>>>(u, l, out, h->g.half, h->nh, h->ldg, h->d.nbh)
  RTILE_SWITCH(t, L);
#undef L
  CUW_LAUNCH_CHECK("k_raddx");
  return CUW_OK;
}

int addoproj_run(Handle* h, double2* proj, const double2* oproj, const double* lam) {
  if (h->npro == 0) return CUW_OK;
  k_raddoproj<<<dim3(ceil_div(h->npro, 16), ceil_div(h->d.nb, 32)), 128, 0, h->stream>>>(
      reinterpret_cast<double*>(proj), reinterpret_cast<const double*>(oproj), lam, h->npro, h->d.nb);
  CUW_LAUNCH_CHECK("k_raddoproj");
  return CUW_OK;
}

// force partial sums of slot 0 with E = ded; *nt row groups
int fold_force(Handle* h, const double2* ded, double* fpart, int* nt) {
  const int nb = h->d.nb, npro = h->npro;
  const Op u{slot_ptr(h, 0), h->ldu, 2 * h->nh}, d{reinterpret_cast<const double*>(ded), nb, npro};
  RTile t = pick_tile(h, 2 * h->nh, npro);
  if (t.ni == 8) t.mi = 3;  // the table values of 64 rows do not fit the registers
  const int rows = ceil_div(2 * h->nh, 16 * t.mi), cols = ceil_div(npro, 16 * t.ni);
  // each CTA takes the same number of row tiles, two CTAs per SM
  const int per = ceil_div(rows * cols, 2 * h->nsm), gx = ceil_div(rows, per);
  const dim3 grid(gx, cols);
#define L(MI, NI)                                                                                             \
  k_rforce<MI, NI><<<grid, RT, rsmem<MI, NI>(), h->stream>>>(u, d, h->g.prox, h->g.half, h->nh, h->ldu, h->g.gx, \
                                                             h->g.gy, h->g.gz, nb, fpart)
  RTILE_SWITCH_F(t, L);
#undef L
  CUW_LAUNCH_CHECK("k_rforce");
  *nt = gx;
  return CUW_OK;
}

// bytes of the split sums that the folded products of this set need at most
size_t fold_part_bytes(const Handle* h) {
  size_t n = std::max(gram_split(h, 1).bytes, gram_split(h, 3).bytes);
  if (h->sym && h->npro) n = std::max({n, proj_split(h, 1).bytes, proj_split(h, 2).bytes});
  return n;
}

int fold_kernels_setup(Handle* h) {
#define ALLOW(K, MI, NI) CUW_TRY(smem_allow((const void*)K, (int)rsmem<MI, NI>()))
#define ALLOW_K(MI, NI)             \
  ALLOW((k_rproj<MI, NI>), MI, NI); \
  ALLOW((k_rgram<MI, NI>), MI, NI)
#define ALLOW_ALL(MI, NI)                          \
  ALLOW((k_raddpro<MI, NI>), MI, NI);              \
  ALLOW((k_raddpro_step<MI, NI>), MI, NI);         \
  ALLOW((k_raddx<MI, NI>), MI, NI)
  ALLOW_ALL(2, 2);
  ALLOW_ALL(2, 4);
  ALLOW_ALL(3, 8);
  ALLOW_ALL(4, 8);
  ALLOW_K(2, 2);
  ALLOW_K(2, 4);
  ALLOW_K(4, 8);
  ALLOW((k_rforce<2, 2>), 2, 2);
  ALLOW((k_rforce<2, 4>), 2, 4);
  ALLOW((k_rforce<3, 8>), 3, 8);
#undef ALLOW_K
#undef ALLOW_ALL
#undef ALLOW
  return CUW_OK;
}

}  // namespace cuw
