// Mixed-precision contractions on the 5th-generation tensor cores (tcgen05).
//
// Every product is a real GEMM C = A * B^T whose operands are split into tf32
// pairs (hi + lo) and multiplied as lo*hi + hi*lo + hi*hi with fp32
// accumulation in tensor memory (three-term split precision), drained after
// every K = 8 step into register sums (tc_pipe.cuh).  The A operands are the
// folded fp32 arrays (projector table, wave functions), fetched by TMA several
// chunks ahead and split by the converter warps on their way into tensor memory;
// the B operands (folded wave functions, small FP64 matrices) are split by
// k_bsplit beforehand and arrive by bulk copies.  Every wait is bounded; a wait
// that runs out sets an error flag and the kernel leaves through its cleanup path
// (TMEM released) instead of hanging.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>

#include "cuwaves_internal.cuh"
#include "tc_pipe.cuh"

namespace cuw {
namespace {

// Real K values per chunk: 16 (two MMA steps of K = 8).
// The accumulation run stays one MMA step: the tensor core's truncating fp32
// accumulation was measured on B200 at a signed mean error of -3.7e-8 /
// -8.7e-8 / -1.8e-7 of |C| for runs of 8 / 16 / 32 real K, and one step keeps
// the energy bias below 1e-6 Ha/atom.
constexpr int kCK = 16, kNSplit = 8;

// Every contraction is a real product over the folded half sphere (fold.cu):
// A rows are projectors, bands or sphere rows r, and a raw A slot is one TMA box
// of 16 K values of 128 rows in fp32: either K contiguous (64-byte rows, 64-byte
// swizzle, so that eight consecutive rows read down a column hit distinct banks)
// or row contiguous (16 rows of 512 bytes).  The B operands arrive already split
// (k_bsplit) as one bulk copy per chunk.
constexpr int kRawFold = 8192;
constexpr int kRawGemm = 36864;   // A, B 128 rows x 16 doubles (144-byte rows, element copies)
// Chunks travel in pairs through the copy and conversion hand-overs (the last
// template argument): each hand-over costs several hundred cycles whatever it
// carries, and pairs took 10-20 % off these kernels on B200 (Si64 and Si128
// projections, back-projection, Gram; more raw slots than listed here gained
// nothing).  Stage and slot counts below count pairs.
using ProjPipe = tc::Pipe<4, 4, kRawFold, true, 2, 2, 2>;
using AddproPipe = tc::Pipe<4, 4, kRawFold, true, 2, 2, 2>;
using GramPipe = tc::Pipe<4, 4, kRawFold, true, 2, 2, 2>;
using AddxPipe = tc::Pipe<4, 4, kRawFold, true, 2, 2, 2>;
using ForcePipe = tc::Pipe<4, 4, kRawFold, true, 2, 2, 2>;
using GemmPipe = tc::Pipe<kNSplit, 2, kRawGemm, false>;
constexpr int kThreads = ProjPipe::kThreads;
constexpr int kBTile = 4096;              // floats of one split B chunk (hi and lo tiles)
static_assert(ProjPipe::kSmem <= 232448 && GramPipe::kSmem <= 232448 && AddxPipe::kSmem <= 232448 &&
                  GemmPipe::kSmem <= 232448 && ForcePipe::kSmem <= 232448 && AddproPipe::kSmem <= 232448,
              "shared memory");
// rows of the force kernels' FP64 tiles are padded to an odd number of doubles
// so that the column stores of a warp (one row per lane) spread over the banks
constexpr int kSvLd = 65, kSvLd1 = 129;
static_assert(ForcePipe::kSplitBytes + ForcePipe::kNRaw * ForcePipe::kG * kRawFold >=
                  sizeof(double) * (128 * kSvLd1 + 4 * 128 + 4 * 384),
              "stage area too small");

// offset of 16-byte piece e of row r in a box with 64-byte rows under the TMA
// 64-byte swizzle: address bits 4-5 are XORed with bits 7-8
__device__ __forceinline__ int sw64(int r, int e) { return r * 64 + ((e ^ ((r >> 1) & 3)) << 4); }

template <class T>
__device__ __forceinline__ T at(const unsigned char* raw, int byte) {
  return *reinterpret_cast<const T*>(raw + byte);
}
__device__ __forceinline__ double2 dz() { return make_double2(0.0, 0.0); }

// B functors of the pipelines that do not use them
struct NoLoadB {
  __device__ void operator()(int, int, tc::Copier&) const {}
};
struct NoConvertB {
  __device__ void operator()(int, const unsigned char*, int, float*, float*) const {}
};
// bulk copy of the pre-split B chunk (tile, chunk) of a k_bsplit array
__device__ __forceinline__ void load_bsplit(tc::Copier& cp, int lane, const float* bs, int nchk, int tile, int chunk) {
  if (lane == 0) cp.bulk(0, bs + ((size_t)tile * nchk + chunk) * kBTile, 4 * kBTile);
}

// the eight K values 8 kh.. of A row r in a K-contiguous / row-contiguous box
__device__ __forceinline__ void a_kfast(const unsigned char* raw, int r, int kh, float (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 x = at<float4>(raw, sw64(r, 2 * kh + i));
    v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
  }
}
__device__ __forceinline__ void a_mfast(const unsigned char* raw, int r, int kh, float (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = at<float>(raw, (8 * kh + i) * 512 + 4 * r);
}

// ---------------------------------------------------------------------------
// Plain real GEMM C(M,N) = A(M,K) * B(N,K)^T, FP64 in and out, row-major with
// K contiguous: the reference product of the split-precision machinery.
// One CTA computes a 128 x 128 tile over the whole K range.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 1)
    k_tf32x3_gemm(int M, int N, int K, const double* __restrict__ A, const double* __restrict__ B,
                  double* __restrict__ C, int* __restrict__ err) {
  const int m0 = blockIdx.x * 128, n0 = blockIdx.y * 128;
  constexpr int RS = 144;  // raw row stride (16 doubles + 16 bytes)
  auto load = [&](int c, int lane, tc::Copier& cp) {
    const int k0 = c * 16;
    for (int it = lane; it < 2 * 128 * 16; it += 32) {
      const int op = it / (128 * 16), r = (it / 16) % 128, kk = it % 16;
      const int row = (op == 0 ? m0 : n0) + r, lim = op == 0 ? M : N;
      if (row < lim && k0 + kk < K) cp.el8(op * 128 * RS + r * RS + kk * 8, (op == 0 ? A : B) + (size_t)row * K + k0 + kk);
    }
  };
  auto a_row = [&](int c, const unsigned char* raw, int row, int kh, float (&v)[8]) {
    const bool rok = m0 + row < M;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = c * 16 + 8 * kh + i;
      v[i] = (rok && k < K) ? (float)at<double>(raw, row * RS + (8 * kh + i) * 8) : 0.f;
    }
  };
  auto convert_b = [&](int c, const unsigned char* raw, int ct, float* bhi, float* blo) {
    for (int it = ct; it < 128 * 4; it += GemmPipe::kGroup) {
      const int r = it % 128, g = it / 128;
      double x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = c * 16 + 4 * g + i;
        x[i] = (n0 + r < N && k < K) ? at<double>(raw, 128 * RS + r * RS + (4 * g + i) * 8) : 0.0;
      }
      tc::store_split4(bhi, blo, tc::tile_f4(r, g), x[0], x[1], x[2], x[3]);
    }
  };
  auto finish = [&](const float (&acc)[GemmPipe::kCols], int row, int col0) {
    if (m0 + row >= M) return;
    double* out = C + (size_t)(m0 + row) * N + n0 + col0;
    const int nc = min(GemmPipe::kCols, N - n0 - col0);
#pragma unroll
    for (int j = 0; j < GemmPipe::kCols; ++j)
      if (j < nc) out[j] = (double)acc[j];
  };
  NoLoadB no_b;
  tc::pipe_run<GemmPipe>((K + 15) / 16, load, no_b, a_row, convert_b, finish, err);
}

// PROJ(b, p) of one or two arrays from part[z][p][set][b]
__global__ void __launch_bounds__(32 * kSumZ)
    k_tc_proj_sum(const float2* __restrict__ part, int nz, int nbh, int nset, int npro, double scale,
                  double2* __restrict__ out0, double2* __restrict__ out1) {
  const int nw = nset * nbh;
  const size_t n = (size_t)nw * npro, i = blockIdx.x * (size_t)32 + threadIdx.x;
  const double2 s = split_sum(part, nz, n, i, Scaled{scale}, (const double2*)nullptr, 0);
  if (threadIdx.y || i >= n) return;
  const int b = (int)(i % nw);
  const size_t p = i / nw;
  (b < nbh ? out0 : out1)[(b < nbh ? b : b - nbh) + (size_t)nbh * p] = s;
}

// out_pair(i + NB j) = scale * sum_z part[z][pair][i][j] + one-centre sum
// oc[z][pair][i][j] (FP64, kc splits); on the diagonal the plane-wave sum is that
// of the nd ranges of dg (diag_sums; which[pair]: 0, 1 or 2 there)
__global__ void __launch_bounds__(32 * kSumZ)
    k_tc_gram_sum(const float2* __restrict__ part, int nz, const double2* __restrict__ oc, int kc,
                  const double* __restrict__ dg, int nd, int3 which, int nb, int npair, double scale,
                  double* __restrict__ o0, double* __restrict__ o1, double* __restrict__ o2) {
  // one row of one pair and 32 pairs of columns a block (index divisions in front of
  // the loads took 3 us of 10)
  const int pair = blockIdx.z, i = blockIdx.y, c = blockIdx.x * 32 + threadIdx.x, j = 2 * c, w = nb / 2;
  const size_t n = (size_t)npair * nb * w, t = c < w ? ((size_t)pair * nb + i) * w + c : n;
  const int q = pair == 0 ? which.x : (pair == 1 ? which.y : which.z);
  auto scaled = [&](double2 v) {
    v = cscale(v, scale);
    if (c == i >> 1) {
      double d = 0.0;
#pragma unroll 4
      for (int z = threadIdx.y; z < nd; z += kSumZ) d += dg[((size_t)z * 3 + q) * nb + i];
      (i & 1 ? v.y : v.x) = scale * d;
    }
    return v;
  };
  const double2 s = split_sum(part, nz, n, t, scaled, oc, kc);
  if (threadIdx.y || t >= n) return;
  double* o = pair == 0 ? o0 : (pair == 1 ? o1 : o2);
  o[i + (size_t)nb * j] = s.x;
  o[i + (size_t)nb * (j + 1)] = s.y;
}

// Folded projector table of the mixed path: P(r, p) in fp32 (k_pro_fold of
// fold.cu evaluates the same in FP64).  The single rounding to fp32 is the one
// the split into tf32 pairs starts from.
__global__ void k_pro_f32(int nh, int ngl, int ldu, const int2* __restrict__ half, const double* __restrict__ gx,
                          const double* __restrict__ gy, const double* __restrict__ gz, const double* __restrict__ r,
                          const int* __restrict__ ipro0, const int* __restrict__ nlmn,
                          const ProDesc* __restrict__ pdesc, const double* __restrict__ ylm,
                          const double* __restrict__ pro, float* __restrict__ pf) {
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
    *reinterpret_cast<float2*>(pf + (size_t)ldu * (p0 + k) + 2 * h) = make_float2((float)(sv * e.x), (float)(sv * e.y));
  }
}

// U(r, n) of a wave-function array in fp32 (k_fold of fold.cu; the sums and
// differences are formed in FP64)
__global__ void k_fold_f32(const double2* __restrict__ psi, const int2* __restrict__ half, int nh, int ldg, int ldu,
                           float* __restrict__ u) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (h >= nh) return;
  const int2 g = half[h];
  const double2* p = psi + (size_t)ldg * b;
  const double2 x = p[g.x], y = p[g.y];
  const bool self = g.x == g.y;
  float* o = u + (size_t)ldu * (2 * b) + 2 * h;
  *reinterpret_cast<float2*>(o) = make_float2((float)(self ? x.x : x.x + y.x), (float)(self ? x.x : x.y - y.y));
  *reinterpret_cast<float2*>(o + ldu) = make_float2((float)(self ? x.y : x.y + y.y), (float)(self ? x.y : y.x - x.x));
}

// ---------------------------------------------------------------------------
// Products with K along the half sphere: part[z][i][n] = sum_{r in split z}
// A(r,i) B(r,n), fp32.
//   projections (WAVES_PROJECTIONS, src/paw_waves1.f90:5746-5905): A = P, B = U
//     of one or two arrays (column tiles of the second follow the first's)
//   overlaps (PLANEWAVE$SCALARPRODUCT, src/paw_fft.f90:2344-2422): A = U of x,
//     B = U of y for up to three pairs (blockIdx.z = split*npair + pair)
// Rows tile blockIdx.x, column tile blockIdx.y.
// ---------------------------------------------------------------------------
struct TcTnArgs {
  int npair, nk, kchunk, nchk;
  int nrow, ncol;       // rows of A, columns of one array
  int tps, ldp;         // column tiles of one array, row length of part
  const float* bs[3];   // split B of each pair
};
struct TcTnMaps {
  CUtensorMap a[3];
};
template <class P>
__global__ void __launch_bounds__(kThreads, 1)
    k_tc_tn(TcTnArgs a, const __grid_constant__ TcTnMaps tm, float* __restrict__ part, int* __restrict__ err) {
  const int pair = blockIdx.z % a.npair, split = blockIdx.z / a.npair;
  const int m0 = blockIdx.x * 128;
  const int kbeg = split * a.kchunk, kend = min(a.nk, kbeg + a.kchunk);
  const float* bs = a.bs[pair];
  // zeros past NK and the rows; chunks never straddle a split boundary (kchunk
  // is a multiple of 16)
  auto load = [&](int c, int lane, tc::Copier& cp) {
    if (lane == 0) cp.tensor(0, &tm.a[pair], kbeg + c * kCK, m0, kRawFold);
  };
  auto load_b = [&](int c, int lane, tc::Copier& cp) { load_bsplit(cp, lane, bs, a.nchk, blockIdx.y, kbeg / kCK + c); };
  auto a_row = [&](int c, const unsigned char* raw, int r, int kh, float (&v)[8]) { a_kfast(raw, r, kh, v); };
  auto finish = [&](const float (&acc)[P::kCols], int row, int col0) {
    const int i = m0 + row;
    if (i >= a.nrow) return;
    const int set = blockIdx.y / a.tps, n0 = 128 * (blockIdx.y - set * a.tps) + col0;
    float* out = part + ((size_t)blockIdx.z * a.nrow + i) * a.ldp + (size_t)set * a.ncol + n0;
#pragma unroll
    for (int j = 0; j < P::kCols; j += 2)
      if (n0 + j < a.ncol) *reinterpret_cast<float2*>(out + j) = make_float2(acc[j], acc[j + 1]);
  };
  NoConvertB no_cb;
  const int nchunk = kend > kbeg ? (kend - kbeg + kCK - 1) / kCK : 0;
  tc::pipe_run<P>(nchunk, load, load_b, a_row, no_cb, finish, err);
}

// the value at this lane's G from the row values of a pair (adjacent lanes):
// even rows hold s and take G (s + i t), odd rows hold t and take -G (s - i t)
__device__ __forceinline__ double2 unfold(double2 v, bool odd) {
  double2 o;
  o.x = __shfl_xor_sync(0xffffffffu, v.x, 1);
  o.y = __shfl_xor_sync(0xffffffffu, v.y, 1);
  return odd ? make_double2(o.x + v.y, o.y - v.x) : make_double2(v.x - o.y, v.y + o.x);
}
// the row value of U (u of even rows, w of odd rows) from this lane's psi
__device__ __forceinline__ double2 refold(double2 v, bool odd, bool self) {
  double2 o;
  o.x = __shfl_xor_sync(0xffffffffu, v.x, 1);
  o.y = __shfl_xor_sync(0xffffffffu, v.y, 1);
  if (self) return odd ? o : v;
  return odd ? make_double2(o.y - v.y, v.x - o.x) : make_double2(v.x + o.x, v.y + o.y);
}

// ---------------------------------------------------------------------------
// ADDPRO with the step epilogues (WAVES_ADDPRO, src/paw_waves1.f90:5908-6067,
// and the epilogues of the FP64 form): 128 sphere rows (64 pairs) x 32 super
// wave functions per CTA (column tile blockIdx.x, row tile blockIdx.y), the tile
// columns hold C1 (hproj) products, then C2 (oproj) products.  FUSED leaves the
// folded psim and opsi in um and uo.
// ---------------------------------------------------------------------------
struct TcAddproArgs {
  double2 *hpsi, *opsi, *psim;
  const double2* psi0;
  const double* rmpsi;
  const int2* half;
  float *um, *uo;
  int ldg, ldu, nh, nbh, npro, nchk;
  const float* bc;
  StepCoef sc;
};
template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
    k_tc_addpro(TcAddproArgs a, const __grid_constant__ CUtensorMap tm_pf, int* __restrict__ err) {
  constexpr bool USE_H = (MODE != ADDPRO_OPSI);
  constexpr bool USE_O = (MODE != ADDPRO_HPSI);
  // the column tiles of one row tile are consecutive blocks (blockIdx.x), so the
  // second read of the row tile's projectors comes from L2
  const int m0 = blockIdx.y * 128, b0 = blockIdx.x * 32;
  auto load = [&](int c, int lane, tc::Copier& cp) {
    if (lane == 0) cp.tensor(0, &tm_pf, m0, c * kCK, kRawFold);
  };
  auto load_b = [&](int c, int lane, tc::Copier& cp) { load_bsplit(cp, lane, a.bc, a.nchk, blockIdx.x, c); };
  auto a_row = [&](int c, const unsigned char* raw, int r, int kh, float (&v)[8]) { a_mfast(raw, r, kh, v); };
  auto finish = [&](const float (&acc)[AddproPipe::kCols], int row, int col0) {
    const int r = m0 + row;
    const bool rok = r < 2 * a.nh, odd = row & 1;
    const int2 gp = rok ? a.half[r >> 1] : make_int2(0, 0);
    const bool self = gp.x == gp.y, mine = rok && !(odd && self);
    const int g = odd ? gp.y : gp.x;
    const double rm = a.rmpsi[g];
    const bool hcol = col0 < 64;  // columns 0..63: C1 (H) products, 64..127: C2 (O); uniform in a warp
    const int bl0 = b0 + (col0 & 63) / 2;
    if (hcol ? !USE_H : !USE_O) return;
    double a1 = a.sc.a1, a2 = a.sc.a2, a3 = a.sc.a3 * rm;
    if (MODE == ADDPRO_FUSED && a.sc.fr) {  // cell friction ANNEEVEC(G) (src/paw_waves1.f90:6536-6540)
      const double ai = a.sc.fr[g];
      a1 = 2.0 * ai;
      a2 = 1.0 - a1;
      a3 = -a.sc.dt2 * ai * rm;
    }
    // columns in groups of kB whose loads are all issued before any store of
    // the group (the arrays may alias as far as the compiler knows, so a load
    // after a store would wait for it: one memory round trip per group, not
    // two per column)
    constexpr int kB = 2;
#pragma unroll
    for (int j0 = 0; j0 < AddproPipe::kCols / 2; j0 += kB) {
      double2 hv[kB], p0v[kB], pm[kB];
#pragma unroll
      for (int q = 0; q < kB; ++q) {
        const int b = bl0 + j0 + q;
        const size_t k = mine && b < a.nbh ? (size_t)g + (size_t)a.ldg * b : 0;
        if (hcol) {
          hv[q] = a.hpsi[k];
          if (MODE == ADDPRO_FUSED) {
            p0v[q] = a.psi0[k];
            pm[q] = a.psim[k];
          }
        } else {
          p0v[q] = a.psi0[k];
        }
      }
#pragma unroll
      for (int q = 0; q < kB; ++q) {
        const int b = bl0 + j0 + q, j = j0 + q;
        const bool bok = b < a.nbh, ok = mine && bok;
        const size_t k = (size_t)g + (size_t)a.ldg * b;
        const double2 v = unfold(make_double2((double)acc[2 * j], (double)acc[2 * j + 1]), odd);
        double2 res = dz();  // psi(+) or O psi at this lane's G
        if (hcol) {
          const double2 h2 = cadd(hv[q], v);
          if (ok) a.hpsi[k] = h2;
          if (MODE == ADDPRO_FUSED) {
            res = make_double2(a1 * p0v[q].x + a2 * pm[q].x + a3 * h2.x, a1 * p0v[q].y + a2 * pm[q].y + a3 * h2.y);
            if (ok) a.psim[k] = res;
          }
        } else {
          const double s = a.sc.oscale * rm;
          res = make_double2((p0v[q].x + v.x) * s, (p0v[q].y + v.y) * s);
          if (ok) a.opsi[k] = res;
        }
        if (MODE == ADDPRO_FUSED) {
          const double2 f = refold(res, odd, self);
          if (rok && bok) {
            float* u = (hcol ? a.um : a.uo) + (size_t)a.ldu * (2 * b) + r;
            u[0] = (float)f.x;
            u[a.ldu] = (float)f.y;
          }
        }
      }
    }
  };
  NoConvertB no_cb;
  tc::pipe_run<AddproPipe>(a.nchk, load, load_b, a_row, no_cb, finish, err);
}

// ---------------------------------------------------------------------------
// psi(+) += O|psi0> Lambda (WAVES_ADDOPSI, src/paw_waves2.f90:547-615): U of the
// operand times the real Lambda, unfolded into out
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 1)
    k_tc_addx(double2* __restrict__ out, const int2* __restrict__ half, int nh, int ldg, int nbh, int nchk,
              const float* __restrict__ ls, const __grid_constant__ CUtensorMap tm_u, int* __restrict__ err) {
  const int m0 = blockIdx.x * 128;
  auto load = [&](int c, int lane, tc::Copier& cp) {
    if (lane == 0) cp.tensor(0, &tm_u, m0, c * kCK, kRawFold);
  };
  auto load_b = [&](int c, int lane, tc::Copier& cp) { load_bsplit(cp, lane, ls, nchk, blockIdx.y, c); };
  auto a_row = [&](int c, const unsigned char* raw, int r, int kh, float (&v)[8]) { a_mfast(raw, r, kh, v); };
  auto finish = [&](const float (&acc)[AddxPipe::kCols], int row, int col0) {
    const int r = m0 + row;
    const bool rok = r < 2 * nh, odd = row & 1;
    const int2 gp = rok ? half[r >> 1] : make_int2(0, 0);
    const bool self = gp.x == gp.y, mine = rok && !(odd && self);
    const int g = odd ? gp.y : gp.x, b0 = (blockIdx.y * 128 + col0) / 2;
    // four columns' loads before their stores (one memory round trip per group)
#pragma unroll
    for (int j0 = 0; j0 < AddxPipe::kCols / 2; j0 += 4) {
      double2 o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int b = b0 + j0 + q;
        o[q] = out[mine && b < nbh ? (size_t)g + (size_t)ldg * b : 0];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int b = b0 + j0 + q, j = j0 + q;
        const double2 w = make_double2((double)acc[2 * j], (double)acc[2 * j + 1]), v = unfold(w, odd);
        if (mine && b < nbh)
          out[(size_t)g + (size_t)ldg * b] =
              self ? cadd(o[q], w) : make_double2(o[q].x + 0.5 * v.x, o[q].y + 0.5 * v.y);
      }
    }
  };
  NoConvertB no_cb;
  tc::pipe_run<AddxPipe>(nchk, load, load_b, a_row, no_cb, finish, err);
}

// ---------------------------------------------------------------------------
// Forces (WAVES_DEDPRO + WAVES_PROFORCE, src/paw_waves1.f90:5694-5743,
// 6112-6234): D(r,p) = sum_n U(r,n) E(n,p) on the tensor cores for 128 sphere
// rows x 128 projectors, then sv(r,p) = +-P(r^1,p) D(r,p) in the drain warps
// (into the freed stage buffers) and fpart[tile][p][c] = sum_r sv(r,p) G_c by
// the whole CTA.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 1)
    k_tc_force(const __grid_constant__ CUtensorMap tm_u, const float* __restrict__ be, int nchk, int nh, int npro,
               int ldu, const float* __restrict__ pf, const int2* __restrict__ half, const double* __restrict__ gx,
               const double* __restrict__ gy, const double* __restrict__ gz, double* __restrict__ fpart,
               int* __restrict__ err) {
  const int m0 = blockIdx.x * 128, p0 = blockIdx.y * 128;
  auto load = [&](int c, int lane, tc::Copier& cp) {
    if (lane == 0) cp.tensor(0, &tm_u, m0, c * kCK, kRawFold);
  };
  auto load_b = [&](int c, int lane, tc::Copier& cp) { load_bsplit(cp, lane, be, nchk, blockIdx.y, c); };
  auto a_row = [&](int c, const unsigned char* raw, int r, int kh, float (&v)[8]) { a_mfast(raw, r, kh, v); };
  // [128][kSvLd1], over the stage and raw buffers: when a drain thread finishes,
  // every chunk has been converted and multiplied and no copy is in flight
  double* sv = reinterpret_cast<double*>(tc::pipe_stage_base());
  auto finish = [&](const float (&acc)[ForcePipe::kCols], int row, int col0) {
    const int r = m0 + row;
    const double sg = (row & 1) ? 1.0 : -1.0;
#pragma unroll
    for (int j = 0; j < ForcePipe::kCols; ++j) {
      const int p = p0 + col0 + j;
      sv[row * kSvLd1 + col0 + j] =
          (r < 2 * nh && p < npro) ? sg * (double)__ldg(&pf[(size_t)ldu * p + (r ^ 1)]) * (double)acc[j] : 0.0;
    }
  };
  NoConvertB no_cb;
  tc::pipe_run<ForcePipe>(nchk, load, load_b, a_row, no_cb, finish, err);
  // pipe_run ended with a CTA barrier: sv is complete (if a wait ran out the
  // error flag is set and the caller discards the result).  G components of the
  // rows, then fpart = sum_r sv(r,p) G_c in four row quarters combined in a
  // fixed order
  double* gsh = sv + 128 * kSvLd1;  // [128][4]
  double* qsum = gsh + 4 * 128;     // [4][384]
  for (int i = threadIdx.x; i < 3 * 128; i += blockDim.x) {
    const int c = i / 128, row = i % 128, r = m0 + row;
    gsh[4 * row + c] = r < 2 * nh ? (c == 0 ? gx : (c == 1 ? gy : gz))[half[r >> 1].x] : 0.0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * 384; i += blockDim.x) {
    const int qr = i / 384, k = i % 384, pl = k / 3, c = k % 3;
    double s = 0.0;
#pragma unroll 8
    for (int r = 32 * qr; r < 32 * qr + 32; ++r) s += sv[r * kSvLd1 + pl] * gsh[4 * r + c];
    qsum[i] = s;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 384; k += blockDim.x) {
    const int pl = k / 3, c = k % 3, p = p0 + pl;
    if (p < npro) fpart[((size_t)blockIdx.x * npro + p) * 3 + c] = ((qsum[k] + qsum[384 + k]) + qsum[768 + k]) + qsum[1152 + k];
  }
}

// ---------------------------------------------------------------------------
// Forces, persistent form for NBH <= 64 (an even number of K chunks, at most
// eight): the same D(r,p) = sum_n U(r,n) E(n,p) and force sums as k_tc_force,
// but one CTA per SM walks a contiguous run of (row tile, projector tile) items.
// The split U rows of a row tile (all of K: 8 chunks x 32 TMEM columns) stay in
// tensor memory for every projector tile of that row tile, so only the pre-split
// E chunks stream.  Each item accumulates in one of two TMEM regions (two chunks
// at a time: cross terms, then hi*hi); the drain warps copy the region to
// registers and release it at once, so the MMAs of the next items run while the
// drains form sv(r,p) = +-P(r^1,p) D(r,p) from the fp32 projector table and the
// G-weighted column sums of this item, 64 projectors at a time.
//   warp 0   TMEM allocation, MMA issue (one thread)
//   warp 1   TMA copies of raw U chunks (two raw slots, one per converter group)
//   warp 2   bulk copies of the split E chunks into kFNS stages
//   3..10    converters (two groups of four warps, alternate chunks of a row tile)
//   11..26   drains and the per-item force epilogue
// Barriers: rawfull/rawempty (raw U slots), afull[c] (A chunk c of the
// current row tile in TMEM), afree (MMAs of the last item of a row tile done),
// sfull/sfree (B stages), bfull/bempty (accumulation regions, one item each).
// Every wait is bounded; the drain group decides to leave by one vote per item
// (a reduction barrier all 16 drain warps reach), so none of them is left at a
// barrier.  The hand-over protocol is model-checked on the CPU
// (tests/test_pipe_protocol.py).
// ---------------------------------------------------------------------------
constexpr int kFNS = 6;        // B stages (16 KB each)
constexpr int kFMaxChunks = 8; // K chunks of a resident A tile (TMEM columns 256..511)
constexpr size_t kForcePSmem = (size_t)kFNS * 16384 + 2 * kRawFold +
                               sizeof(double) * (128 * kSvLd + 4 * 128 + 4 * 192) + 1024 + 512;
static_assert(kForcePSmem <= 232448, "shared memory");

__global__ void __launch_bounds__(kThreads, 1)
    k_tc_force_p(const __grid_constant__ CUtensorMap tm_u, const float* __restrict__ be, int nchk, int nh, int npro,
                 int ldu, int tn, int nitems, const float* __restrict__ pf, const int2* __restrict__ half,
                 const double* __restrict__ gx, const double* __restrict__ gy, const double* __restrict__ gz,
                 double* __restrict__ fpart, int* __restrict__ err) {
  using namespace tc;
  float* st = pipe_stage_base();
  unsigned char* raw0 = reinterpret_cast<unsigned char*>(st) + (size_t)kFNS * 16384;
  double* sv = reinterpret_cast<double*>(raw0 + 2 * kRawFold);  // [128][kSvLd]
  double* gsh = sv + 128 * kSvLd;                            // [128][4]
  double* qsum = gsh + 4 * 128;                              // [4][192]
  uint64_t* rawfull = reinterpret_cast<uint64_t*>(qsum + 4 * 192);
  uint64_t* rawempty = rawfull + 2;
  uint64_t* sfull = rawempty + 2;
  uint64_t* sfree = sfull + kFNS;
  uint64_t* bfull = sfree + kFNS;
  uint64_t* bempty = bfull + 2;
  uint64_t* afull = bempty + 2;
  uint64_t* afree = afull + kFMaxChunks;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(afree + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long G = gridDim.x;
  const int w0 = (int)((long long)blockIdx.x * nitems / G), w1 = (int)((long long)(blockIdx.x + 1) * nitems / G);
  const int m_first = w0 / tn;
  const int nm = w1 > w0 ? (w1 - 1) / tn - m_first + 1 : 0;  // row tiles of this CTA
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&rawfull[i], 1);
      mbar_init(&rawempty[i], 128);
      mbar_init(&bfull[i], 1);
      mbar_init(&bempty[i], 512);
    }
    for (int i = 0; i < kFNS; ++i) {
      mbar_init(&sfull[i], 1);
      mbar_init(&sfree[i], 1);
    }
    for (int c = 0; c < kFMaxChunks; ++c) mbar_init(&afull[c], 128);
    mbar_init(afree, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(tslot, 512);
    tmem_relinquish();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tslot;
  auto raise = [&]() {
    *abort_flag = 1;
    atomicExch(err, 1);
  };
  if (warp == 0) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_tf32(128, 128);
      constexpr uint32_t lbo = 128 * 16;
      const uint64_t dsc0 = sdesc(0, lbo, 128);
      const uint32_t st0 = smem_u32(st) >> 4;
      constexpr uint32_t kStageU = 16384u >> 4, kLoU = 8192u >> 4, kOffU = (2 * lbo) >> 4;
      int it = 0, j = 0;
      bool ok = true, pending = false;  // pending: MMAs issued since the last bfull commit
      for (int w = w0; w < w1 && ok && !*abort_flag; ++w, ++it) {
        const int im = w / tn - m_first, r = it & 1;
        const bool first_of_m = (w == w0) || (w % tn == 0), last_of_m = (w == w1 - 1) || ((w + 1) % tn == 0);
        if (it >= 2) ok = mbar_wait(&bempty[r], ((it >> 1) - 1) & 1, kWaitCycles);
        const uint32_t d = tmem + (uint32_t)(r * 128);
        for (int rr = 0; rr < nchk / 2 && ok; ++rr, j += 2) {
          for (int i = 0; i < 2 && ok; ++i) {
            if (first_of_m) ok = mbar_wait(&afull[2 * rr + i], im & 1, kWaitCycles);
            if (ok) ok = mbar_wait(&sfull[(j + i) % kFNS], ((j + i) / kFNS) & 1, kWaitCycles);
          }
          if (!ok) break;
          fence_after_sync();
#pragma unroll
          for (int pass = 0; pass < 2; ++pass)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int c = 2 * rr + i, s = (j + i) % kFNS;
              const uint32_t bu = st0 + (uint32_t)s * kStageU;
              const uint32_t ta = tmem + (uint32_t)(256 + 32 * c);
#pragma unroll
              for (int ks = 0; ks < 2; ++ks) {
                const uint64_t bhi = dsc0 | (uint64_t)(bu + ks * kOffU), blo = dsc0 | (uint64_t)(bu + kLoU + ks * kOffU);
                const uint32_t ahi = ta + 8 * ks, alo = ahi + 16;
                if (pass == 0) {
                  mma_tf32_ta(d, alo, bhi, idesc, (rr | i | ks) ? 1u : 0u);
                  mma_tf32_ta(d, ahi, blo, idesc, 1u);
                } else {
                  mma_tf32_ta(d, ahi, bhi, idesc, 1u);
                }
              }
            }
          mma_commit(&sfree[j % kFNS]);
          mma_commit(&sfree[(j + 1) % kFNS]);
          pending = true;
        }
        if (!ok) break;
        mma_commit(&bfull[r]);
        pending = false;
        if (last_of_m) mma_commit(afree);
      }
      if (!ok) raise();
      // the MMAs in flight finish before TMEM is released (after an abort in
      // the middle of an item, through one more commit on its region)
      if (pending) {
        mma_commit(&bfull[it & 1]);
        mbar_wait(&bfull[it & 1], (it >> 1) & 1, kWaitCycles);
      } else if (it > 0) {
        mbar_wait(&bfull[(it - 1) & 1], ((it - 1) >> 1) & 1, kWaitCycles);
      }
    }
  } else if (warp == 1) {
    // raw U chunks: chunk c of the im-th row tile goes to slot c % 2 (the slot
    // of converter group c % 2)
    int issued = 0;
    const int total = nm * nchk;
    for (int q = 0; q < total; ++q) {
      const int slot = q & 1, m = m_first + q / nchk, c = q % nchk;
      bool ok = true;
      if (lane == 0) {
        if (q >= 2) ok = mbar_wait(&rawempty[slot], ((q >> 1) - 1) & 1, kWaitCycles);
        ok = ok && !*abort_flag;
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) raise();
        break;
      }
      if (lane == 0) {
        tma_load_2d(raw0 + slot * kRawFold, &tm_u, 128 * m, c * kCK, &rawfull[slot]);
        mbar_arrive_expect_tx(&rawfull[slot], kRawFold);
      }
      issued = q + 1;
    }
    if (*abort_flag && lane == 0)
      for (int q = max(0, issued - 2); q < issued; ++q) mbar_wait(&rawfull[q & 1], (q >> 1) & 1, kWaitCycles);
  } else if (warp == 2) {
    int issued = 0;
    int j = 0;
    for (int w = w0; w < w1; ++w) {
      const int n = w % tn;
      bool ok = true;
      for (int c = 0; c < nchk; ++c, ++j) {
        const int s = j % kFNS;
        if (lane == 0) {
          if (j >= kFNS) ok = mbar_wait(&sfree[s], ((j / kFNS) - 1) & 1, kWaitCycles);
          ok = ok && !*abort_flag;
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        if (lane == 0) {
          bulk_g2s(st + (size_t)s * 4096, be + ((size_t)n * nchk + c) * kBTile, 16384, &sfull[s]);
          mbar_arrive_expect_tx(&sfull[s], 16384);
        }
        issued = j + 1;
      }
      if (!ok) {
        if (lane == 0) raise();
        break;
      }
    }
    if (*abort_flag && lane == 0)
      for (int q = max(0, issued - kFNS); q < issued; ++q) mbar_wait(&sfull[q % kFNS], (q / kFNS) & 1, kWaitCycles);
  } else if (warp < 11) {
    // converters: group grp owns chunks grp, grp + 2, ... of every row tile
    const int grp = (warp - 3) >> 2;
    const int arow = 32 * (warp & 3) + lane;
    const uint32_t tlane = (uint32_t)(32 * (warp & 3)) << 16;
    bool ok = true;
    for (int im = 0; im < nm && ok; ++im) {
      for (int c = grp; c < nchk; c += 2) {
        const int q = im * nchk + c, slot = q & 1;
        bool got = mbar_wait(&rawfull[slot], (q >> 1) & 1, kWaitCycles);
        if (got && c == grp && im >= 1) got = mbar_wait(afree, (im - 1) & 1, kWaitCycles);
        ok = __all_sync(0xffffffffu, got && !*abort_flag);
        if (!ok) {
          if (lane == 0) raise();
          break;
        }
        const unsigned char* raw = raw0 + slot * kRawFold;
#pragma unroll
        for (int kh = 0; kh < 2; ++kh) {
          float v[8];
          a_mfast(raw, arow, kh, v);
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float h0, l0;
            split_tf32f(v[i], h0, l0);
            hi[i] = __float_as_uint(h0), lo[i] = __float_as_uint(l0);
          }
          const uint32_t ta = tmem + tlane + (uint32_t)(256 + 32 * c + 8 * kh);
          tmem_st8(ta, hi);
          tmem_st8(ta + 16, lo);
        }
        tmem_wait_st();
        fence_before_sync();
        mbar_arrive(&afull[c]);
        mbar_arrive(&rawempty[slot]);
      }
    }
  } else {
    const int q = warp & 3, dw = warp - 11, col0 = 32 * (dw / 4), dt = tid - 11 * 32;
    const uint32_t lane_base = ((uint32_t)(32 * q) << 16) + (uint32_t)col0;
    const int row = 32 * q + lane;
    const double sg = (row & 1) ? 1.0 : -1.0;
    // expected truncation loss: a quarter unit in the last place per K=8 step
    const float half_ulps = kLossPerStep * (float)(2 * nchk);
    int it = 0;
    for (int w = w0; w < w1; ++w, ++it) {
      const int m = w / tn, n = w % tn, rr = m * 128 + row, r = it & 1;
      bool got = mbar_wait(&bfull[r], (it >> 1) & 1, kWaitCycles);
      got = __all_sync(0xffffffffu, got && !*abort_flag);
      float acc[32];
      if (got) {
        fence_after_sync();
        uint32_t v[2][16];
        tmem_ld16(tmem + lane_base + (uint32_t)(r * 128), v[0]);
        tmem_ld16(tmem + lane_base + (uint32_t)(r * 128 + 16), v[1]);
        tmem_wait_ld();
        fence_before_sync();
        mbar_arrive(&bempty[r]);  // the region is free for the item after next
#pragma unroll
        for (int k = 0; k < 32; ++k) acc[k] = untruncate(__uint_as_float(v[k >> 4][k & 15]), half_ulps);
      }
      // one decision for the whole drain group, reached by all 16 warps
      if (bar_or(1, 512, !got)) {
        if (dt == 0) raise();
        break;
      }
      // G components of the item's row tile ([row][4]: the three components of
      // a row in different banks)
      if (dt < 128) {
        const int r1 = m * 128 + dt;
        const int g = r1 < 2 * nh ? half[r1 >> 1].x : -1;
        gsh[4 * dt] = g >= 0 ? gx[g] : 0.0;
        gsh[4 * dt + 1] = g >= 0 ? gy[g] : 0.0;
        gsh[4 * dt + 2] = g >= 0 ? gz[g] : 0.0;
      }
#pragma unroll 1
      for (int hb = 0; hb < 2; ++hb) {  // projectors 64 hb .. 64 hb + 63 of the item
        if ((col0 >> 6) == hb) {
          // thirty-two table loads of a thread, sixteen in flight together
#pragma unroll
          for (int jb = 0; jb < 32; jb += 16) {
            float pfv[16];
#pragma unroll
            for (int jx = 0; jx < 16; ++jx) {
              const int p = n * 128 + col0 + jb + jx;
              pfv[jx] = (rr < 2 * nh && p < npro) ? __ldg(&pf[(size_t)p * ldu + (rr ^ 1)]) : 0.f;
            }
#pragma unroll
            for (int jx = 0; jx < 16; ++jx)
              sv[row * kSvLd + (col0 & 63) + jb + jx] = sg * (double)pfv[jx] * (double)acc[jb + jx];
          }
        }
        bar_sync(1, 512);
        // fpart[m][p][c] = sum_r sv(r,p) G_c: four row quarters, fixed order
        for (int t = dt; t < 4 * 192; t += 512) {
          const int qr = t / 192, k = t % 192, pl = k / 3, c = k % 3;
          double sum = 0.0;
#pragma unroll 8
          for (int rw = 32 * qr; rw < 32 * qr + 32; ++rw) sum += sv[rw * kSvLd + pl] * gsh[4 * rw + c];
          qsum[t] = sum;
        }
        bar_sync(1, 512);
        if (dt < 192) {
          const int pl = dt / 3, c = dt % 3, p = n * 128 + 64 * hb + pl;
          if (p < npro)
            fpart[((size_t)m * npro + p) * 3 + c] = ((qsum[dt] + qsum[192 + dt]) + qsum[384 + dt]) + qsum[576 + dt];
        }
      }
      bar_sync(1, 512);
    }
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

// Source of a split B operand: value(row, k)
//   kind 0: xf[k + ld*row]  (fp32)   kind 1: x[k + ld*row]
//   kind 2: tile of 64 rows of x then 64 rows of x2, each x[row + ld*k] (null: zero)
struct BSplitSrc {
  int kind;
  const double* x;
  const double* x2;
  const float* xf;
  long long ld;
  int nrow, nk;
  int tps;              // tiles of one array (kind 0); the next array's tiles
  long long set_stride; // follow, its values set_stride further
};

// dg[z][q][n] = sum_{r in range z} of U_0 U_0, U_1 U_0, U_1 U_1 (q = 0, 1, 2) at
// (r,n) in FP64, one warp per (range, n): the diagonals of the plane-wave
// overlaps.  What the tensor-core product leaves in an overlap is the rounding
// of its fp32 running sums (one addition per K = 8), which scales with the sum
// itself: about 1e-7 of the diagonals, the norms of 192 bands of 50000 plane
// waves, and next to nothing of the other overlaps, which are small.  A step's
// norm error enters the next step's wave-function velocities, and the forces of
// Si96 at 36 Ry were 8e-6 off after four steps; with these sums they are 2e-6 off.
// The sums ride in the launch that splits the operands (a launch of their own
// cost a step of Si8 13 us of 190).
constexpr int kDiagK = 1024;
struct DiagSums {
  const float *u0, *u1;
  int nk, ldu, nb, nd;  // nd ranges; 0: none
  double* dg;
};
__device__ __forceinline__ void diag_sums(const DiagSums& a, int item) {
  const int z = item % a.nd, b = item / a.nd * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= a.nb) return;  // the whole warp
  const float *x = a.u0 + (size_t)a.ldu * b, *y = a.u1 + (size_t)a.ldu * b;
  const int k1 = min(a.nk, (z + 1) * kDiagK);  // rows are padded with zeros to 32 values
  double q[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int k = z * kDiagK + 4 * lane; k < k1; k += 128) {
    const float4 u = *reinterpret_cast<const float4*>(x + k), v = *reinterpret_cast<const float4*>(y + k);
    const float uv[4] = {u.x, u.y, u.z, u.w}, vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double ud = uv[e], vd = vv[e];
      q[0] = fma(ud, ud, q[0]);
      q[1] = fma(ud, vd, q[1]);
      q[2] = fma(vd, vd, q[2]);
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q[i] += __shfl_xor_sync(0xffffffffu, q[i], o);
  if (lane < 3) a.dg[((size_t)z * 3 + lane) * a.nb + b] = lane == 0 ? q[0] : (lane == 1 ? q[1] : q[2]);
}

// B operand split into tf32 hi/lo tiles in the shared-memory layout of the
// pipeline (tc_pipe.cuh): block (tile, chunk) of 4096 floats = hi then lo,
// element (row, k) of 128 rows x 16 K at (k/4)*512 + row*4 + k%4.  Zero outside
// the source.  The first ndiag columns of blocks take the items of diag_sums.
__global__ void __launch_bounds__(256) k_bsplit(BSplitSrc b, int nchk, float* __restrict__ out, DiagSums d, int ndiag) {
  if ((int)blockIdx.x < ndiag) {
    diag_sums(d, blockIdx.x * gridDim.y + blockIdx.y);
    return;
  }
  const int tile = blockIdx.y, c = blockIdx.x - ndiag;
  float* o = out + ((size_t)tile * nchk + c) * kBTile;
  for (int it = threadIdx.x; it < 512; it += blockDim.x) {
    const int R = it & 127, kg = it >> 7, k0 = c * kCK + 4 * kg;
    float w[4] = {0.f, 0.f, 0.f, 0.f};
    if (b.kind == 0) {
      const int set = tile / b.tps, row = 128 * (tile - set * b.tps) + R;
      // (rows are padded to 32 values, zero past NK)
      if (row < b.nrow && k0 < b.nk) {
        const float4 x = *reinterpret_cast<const float4*>(b.xf + set * b.set_stride + k0 + b.ld * row);
        w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
      }
    } else {
      const int row = b.kind == 1 ? 128 * tile + R : 64 * tile + (R & 63);
      const double* src = b.kind == 1 || R < 64 ? b.x : b.x2;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = k0 + e;
        if (src && row < b.nrow && k < b.nk) w[e] = (float)(b.kind == 1 ? src[k + b.ld * row] : src[row + b.ld * k]);
      }
    }
    float4 h, l;
    tc::split_tf32f(w[0], h.x, l.x);
    tc::split_tf32f(w[1], h.y, l.y);
    tc::split_tf32f(w[2], h.z, l.z);
    tc::split_tf32f(w[3], h.w, l.w);
    reinterpret_cast<float4*>(o)[kg * 128 + R] = h;
    reinterpret_cast<float4*>(o + 2048)[kg * 128 + R] = l;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// host side of the split-precision contractions
// ---------------------------------------------------------------------------
static int* tc_err(Handle* h) { return h->g.ostatus + 12; }

// number of K splits so that tiles * splits fills the GPU once (one CTA per SM)
static int tc_splits(const Handle* h, int tiles, int nk, double mul) {
  // at most mul waves of one CTA per SM (rounded down: a CTA past a whole
  // wave would cost a wave of its own)
  const int want = std::max(1, (int)std::floor(h->nsm * mul / std::max(1, tiles)));
  return std::max(1, std::min(want, ceil_div(nk, 4 * kCK)));
}

static int tiles_per_array(const Handle* h) { return ceil_div(h->d.nb, 128); }
// K splits of the projections of nset arrays and of the overlaps of npair pairs,
// and the bytes of their sums
struct TcSplit {
  int ks, kchunk, kc;  // kc: splits of the one-centre sums
  size_t oc, bytes;    // oc: offset of the one-centre sums
};
static TcSplit tc_split_k(const Handle* h, int tiles, double mul) {
  const int nk = 2 * h->nh;
  TcSplit s{};
  s.kchunk = ceil_div(ceil_div(nk, tc_splits(h, tiles, nk, mul)), kCK) * kCK;
  s.ks = ceil_div(nk, s.kchunk);
  return s;
}
static TcSplit tc_proj_split(const Handle* h, int nset) {
  TcSplit s = tc_split_k(h, ceil_div(h->npro, 128) * nset * tiles_per_array(h), h->split_proj);
  s.bytes = sizeof(float2) * (size_t)nset * h->d.nbh * h->npro * s.ks;
  return s;
}
static TcSplit tc_gram_split(const Handle* h, int npair) {
  TcSplit s = tc_split_k(h, tiles_per_array(h) * tiles_per_array(h) * npair, h->split_gram);
  // the one-centre sums stay in FP64, behind the fp32 partials
  const size_t n = (size_t)h->d.nb * h->d.nb * npair;
  s.kc = fold_oc_splits(h, npair);
  s.oc = (sizeof(float) * n * s.ks + 255) / 256 * 256;
  s.bytes = s.oc + sizeof(double) * n * s.kc;
  return s;
}
// bytes of the split sums that the tensor-core products of this set need at most
size_t tc_part_bytes(const Handle* h) {
  return std::max({tc_proj_split(h, 1).bytes, tc_proj_split(h, 2).bytes, tc_gram_split(h, 3).bytes});
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (the
// library links the runtime only)
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiled encode_tiled() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
    cudaGetLastError();
  });
  return fn;
}

// 2-D map of `rows` rows of `inner` fp32 values, rows `ld` values apart, box bx
// x by; elements outside read as zero
static int make_map(Handle* h, CUtensorMap* m, const float* base, long long inner, long long rows, long long ld, int bx,
                    int by, CUtensorMapSwizzle sw) {
  const EncodeTiled fn = encode_tiled();
  if (!fn) return h->fail(CUW_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[2] = {(cuuint64_t)std::max(1ll, inner), (cuuint64_t)std::max(1ll, rows)};
  const cuuint64_t strides[1] = {(cuuint64_t)(ld * 4)};
  const cuuint32_t box[2] = {(cuuint32_t)bx, (cuuint32_t)by};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return h->fail(CUW_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return CUW_OK;
}
// a folded array (rows of 2 nh sphere values) as K-contiguous or row-contiguous
// A operand
static int map_kfast(Handle* h, CUtensorMap* m, const float* base, int rows) {
  return make_map(h, m, base, 2 * h->nh, rows, h->ldu, 16, 128, CU_TENSOR_MAP_SWIZZLE_64B);
}
static int map_mfast(Handle* h, CUtensorMap* m, const float* base, int rows) {
  return make_map(h, m, base, 2 * h->nh, rows, h->ldu, 128, 16, CU_TENSOR_MAP_SWIZZLE_NONE);
}
static float* u32_slot(const Handle* h, int slot) { return h->g.u32 + (size_t)slot * h->d.nb * h->ldu; }
// ranges of diag_sums
static int diag_ranges(const Handle* h) { return ceil_div(2 * h->nh, kDiagK); }

int tc_setup(Handle* h) {
  CUW_TRY(smem_allow((const void*)k_tc_tn<ProjPipe>, (int)ProjPipe::kSmem));
  CUW_TRY(smem_allow((const void*)k_tc_tn<GramPipe>, (int)GramPipe::kSmem));
  CUW_TRY(smem_allow((const void*)k_tc_addpro<ADDPRO_HPSI>, (int)AddproPipe::kSmem));
  CUW_TRY(smem_allow((const void*)k_tc_addpro<ADDPRO_OPSI>, (int)AddproPipe::kSmem));
  CUW_TRY(smem_allow((const void*)k_tc_addpro<ADDPRO_FUSED>, (int)AddproPipe::kSmem));
  CUW_TRY(smem_allow((const void*)k_tc_addx, (int)AddxPipe::kSmem));
  CUW_TRY(smem_allow((const void*)k_tc_force, (int)ForcePipe::kSmem));
  CUW_TRY(smem_allow((const void*)k_tc_force_p, (int)kForcePSmem));
  if (!encode_tiled()) return h->fail(CUW_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  return CUW_OK;
}

// bytes of the buffers of the tensor-core products
TcRooms tc_room_sizes(const Handle* h) {
  const int np = std::max(1, h->npro), nb = h->d.nb;
  // largest small-matrix operand: [C1 | C2] of ADDPRO, DEDPRO or Lambda
  size_t slot = (size_t)ceil_div(nb, 64) * ceil_div(np, kCK);
  slot = std::max(slot, (size_t)ceil_div(np, 128) * ceil_div(nb, kCK));
  slot = std::max(slot, (size_t)ceil_div(nb, 128) * ceil_div(nb, kCK));
  TcRooms r;
  r.split = sizeof(float) * kBTile * 2 * (size_t)tiles_per_array(h) * ceil_div(2 * h->nh, kCK);
  r.u32 = sizeof(float) * (size_t)h->ldu * nb * 2;
  r.small = sizeof(float) * slot * kBTile;
  r.diag = sizeof(double) * 3 * (size_t)diag_ranges(h) * nb;
  return r;
}
// the padding of the rows of U is read as K values past the sphere (k_bsplit)
int tc_clear_padding(Handle* h) {
  if (h->ldu > 2 * h->nh)
    CUW_TRY(cudaMemset2DAsync(h->g.u32 + 2 * h->nh, sizeof(float) * h->ldu, 0, sizeof(float) * (h->ldu - 2 * h->nh),
                              (size_t)2 * h->d.nb, h->stream));
  return CUW_OK;
}

int tc_pro_table(Handle* h, const double* r_dev) {
  if (h->npro == 0) return CUW_OK;
  const Device& g = h->g;
  k_pro_f32<<<dim3(ceil_div(h->nh, 256), h->d.nat), 256, 0, h->stream>>>(h->nh, h->d.ngl, h->ldu, g.half, g.gx, g.gy,
                                                                         g.gz, r_dev, g.t_ipro0, g.t_nlmn, g.pdesc,
                                                                         g.ylm, g.pro, g.pf());
  CUW_LAUNCH_CHECK("k_pro_f32");
  return CUW_OK;
}

int tc_fold(Handle* h, const double2* psi, int slot) {
  k_fold_f32<<<dim3(ceil_div(h->nh, 256), h->d.nbh), 256, 0, h->stream>>>(psi, h->g.half, h->nh, h->ldg, h->ldu,
                                                                          u32_slot(h, slot));
  CUW_LAUNCH_CHECK("k_fold_f32");
  return CUW_OK;
}

static int tc_bsplit(Handle* h, const BSplitSrc& b, int ntile, int nchk, float* out, const DiagSums& d = {}) {
  const int ndiag = ceil_div(d.nd * ceil_div(d.nb, 8), ntile);
  k_bsplit<<<dim3(ndiag + nchk, ntile), 256, 0, h->stream>>>(b, nchk, out, d, ndiag);
  CUW_LAUNCH_CHECK("k_bsplit");
  return CUW_OK;
}

// split forms of folded slots 0 .. nset-1 (B operands of tc_proj and tc_gram);
// of both, the diagonals of their overlaps too
int tc_split(Handle* h, int nset) {
  BSplitSrc b{};
  b.xf = h->g.u32;
  b.ld = h->ldu;
  b.nrow = h->d.nb;
  b.nk = 2 * h->nh;
  b.tps = tiles_per_array(h);
  b.set_stride = (long long)h->d.nb * h->ldu;
  DiagSums d{};
  if (nset == 2) d = {u32_slot(h, 0), u32_slot(h, 1), b.nk, h->ldu, b.nrow, diag_ranges(h), h->g.diag};
  return tc_bsplit(h, b, nset * b.tps, ceil_div(2 * h->nh, kCK), h->g.bpre(), d);
}

// PROJ of slot 0 (and slot 1 when proj1 is given), from the split forms
int tc_proj(Handle* h, double2* proj0, double2* proj1) {
  const int nb = h->d.nb, npro = h->npro, nset = proj1 ? 2 : 1;
  TcTnArgs a{};
  a.npair = 1;
  a.nk = 2 * h->nh;
  a.nrow = npro;
  a.ncol = nb;
  a.tps = tiles_per_array(h);
  a.ldp = nset * nb;
  a.nchk = ceil_div(a.nk, kCK);
  a.bs[0] = h->g.bpre();
  TcTnMaps tm;
  CUW_RET(map_kfast(h, &tm.a[0], h->g.pf(), npro));
  tm.a[1] = tm.a[2] = tm.a[0];
  const int tn = ceil_div(npro, 128), tb = nset * a.tps;
  const TcSplit s = tc_proj_split(h, nset);
  const int ks = s.ks;
  a.kchunk = s.kchunk;
  const size_t n = (size_t)nset * h->d.nbh * npro;
  CUW_RET(ensure_part(h, s.bytes));
  k_tc_tn<ProjPipe><<<dim3(tn, tb, ks), kThreads, ProjPipe::kSmem, h->stream>>>(a, tm, reinterpret_cast<float*>(h->g.part),
                                                                      tc_err(h));
  CUW_LAUNCH_CHECK("k_tc_tn");
  k_tc_proj_sum<<<(unsigned)((n + 31) / 32), dim3(32, kSumZ), 0, h->stream>>>(
      reinterpret_cast<const float2*>(h->g.part), ks, h->d.nbh, nset, npro, h->gweight, proj0, proj1);
  CUW_LAUNCH_CHECK("k_tc_proj_sum");
  return CUW_OK;
}

int tc_addpro(Handle* h, int mode, const double2* hpc, const double2* opc, const StepCoef& sc) {
  Device& g = h->g;
  const int nb = h->d.nb, npro = h->npro;
  CUtensorMap tpf;
  CUW_RET(map_mfast(h, &tpf, g.pf(), npro));
  const int nchk = ceil_div(npro, kCK);
  BSplitSrc b{};
  b.kind = 2;
  b.x = mode == ADDPRO_OPSI ? nullptr : reinterpret_cast<const double*>(hpc);
  b.x2 = mode == ADDPRO_HPSI ? nullptr : reinterpret_cast<const double*>(opc);
  b.ld = nb;
  b.nrow = nb;
  b.nk = npro;
  CUW_RET(tc_bsplit(h, b, ceil_div(nb, 64), nchk, g.bsmall));
  const TcAddproArgs a{g.hpsi, g.opsi, g.psim, g.psi0, g.rmpsi, g.half, u32_slot(h, 0), u32_slot(h, 1),
                       h->ldg, h->ldu, h->nh, h->d.nbh, npro, nchk, g.bsmall, sc};
  const dim3 grid(ceil_div(nb, 64), ceil_div(2 * h->nh, 128));
  if (mode == ADDPRO_HPSI) k_tc_addpro<ADDPRO_HPSI><<<grid, kThreads, AddproPipe::kSmem, h->stream>>>(a, tpf, tc_err(h));
  else if (mode == ADDPRO_OPSI) k_tc_addpro<ADDPRO_OPSI><<<grid, kThreads, AddproPipe::kSmem, h->stream>>>(a, tpf, tc_err(h));
  else k_tc_addpro<ADDPRO_FUSED><<<grid, kThreads, AddproPipe::kSmem, h->stream>>>(a, tpf, tc_err(h));
  CUW_LAUNCH_CHECK("k_tc_addpro");
  return CUW_OK;
}

// overlaps of the slots that tc_split(h, 2) has split
int tc_gram(Handle* h, const FoldPair* pairs, int npair, double* o0, double* o1, double* o2) {
  if (npair < 1 || npair > 3) return h->fail(CUW_ERR_ARG, "overlaps: one to three pairs");
  const int nb = h->d.nb, tps = tiles_per_array(h);
  TcTnArgs a{};
  a.npair = npair;
  a.nk = 2 * h->nh;
  a.nrow = a.ncol = a.ldp = nb;
  a.tps = tps;
  a.nchk = ceil_div(a.nk, kCK);
  TcTnMaps tm;
  for (int i = 0; i < 3; ++i) {
    const FoldPair& q = pairs[std::min(i, npair - 1)];
    CUW_RET(map_kfast(h, &tm.a[i], u32_slot(h, q.x), nb));
    a.bs[i] = h->g.bpre() + (size_t)q.y * tps * a.nchk * kBTile;
  }
  const TcSplit s = tc_gram_split(h, npair);
  const int ks = s.ks, kc = s.kc;
  a.kchunk = s.kchunk;
  const size_t n = (size_t)nb * nb * npair;
  CUW_RET(ensure_part(h, s.bytes));
  double* oc = reinterpret_cast<double*>(reinterpret_cast<char*>(h->g.part) + s.oc);
  CUW_RET(fold_oc(h, pairs, npair, kc, oc));
  k_tc_tn<GramPipe><<<dim3(tps, tps, ks * npair), kThreads, GramPipe::kSmem, h->stream>>>(
      a, tm, reinterpret_cast<float*>(h->g.part), tc_err(h));
  CUW_LAUNCH_CHECK("k_tc_tn");
  auto which = [&](int i) { return i < npair ? pairs[i].x + pairs[i].y : 0; };
  k_tc_gram_sum<<<dim3(ceil_div(nb / 2, 32), nb, npair), dim3(32, kSumZ), 0, h->stream>>>(
      reinterpret_cast<const float2*>(h->g.part), ks, reinterpret_cast<const double2*>(oc), kc, h->g.diag,
      diag_ranges(h), make_int3(which(0), which(1), which(2)), nb, npair, 0.5 * h->gweight, o0, o1, o2);
  CUW_LAUNCH_CHECK("k_tc_gram_sum");
  return CUW_OK;
}

int tc_addx(Handle* h, int slot, const double* lam, double2* out) {
  const int nb = h->d.nb, nchk = ceil_div(nb, kCK);
  CUtensorMap tu;
  CUW_RET(map_mfast(h, &tu, u32_slot(h, slot), nb));
  BSplitSrc b{};
  b.kind = 1;
  b.x = lam;
  b.ld = nb;
  b.nrow = nb;
  b.nk = nb;
  CUW_RET(tc_bsplit(h, b, ceil_div(nb, 128), nchk, h->g.bsmall));
  const dim3 grid(ceil_div(2 * h->nh, 128), ceil_div(nb, 128));
  k_tc_addx<<<grid, kThreads, AddxPipe::kSmem, h->stream>>>(out, h->g.half, h->nh, h->ldg, h->d.nbh, nchk, h->g.bsmall,
                                                            tu, tc_err(h));
  CUW_LAUNCH_CHECK("k_tc_addx");
  return CUW_OK;
}

// force partial sums of slot 0 with E = ded; *ntile row tiles
int tc_force(Handle* h, const double2* ded, double* fpart, int* ntile) {
  const Device& g = h->g;
  const int nb = h->d.nb, npro = h->npro;
  const int tm = ceil_div(2 * h->nh, 128), tn = ceil_div(npro, 128);
  CUtensorMap tu;
  CUW_RET(map_mfast(h, &tu, u32_slot(h, 0), nb));
  const int nchk = ceil_div(nb, kCK);
  BSplitSrc b{};
  b.kind = 1;
  b.x = reinterpret_cast<const double*>(ded);
  b.ld = nb;
  b.nrow = npro;
  b.nk = nb;
  CUW_RET(tc_bsplit(h, b, tn, nchk, g.bsmall));
  *ntile = tm;
  if (nchk % 2 == 0 && nchk <= kFMaxChunks) {
    // persistent form: the U tile stays in tensor memory across projector tiles
    const int nitems = tm * tn;
    k_tc_force_p<<<std::min(nitems, h->nsm), kThreads, kForcePSmem, h->stream>>>(
        tu, g.bsmall, nchk, h->nh, npro, h->ldu, tn, nitems, g.pf(), g.half, g.gx, g.gy, g.gz, fpart, tc_err(h));
    CUW_LAUNCH_CHECK("k_tc_force_p");
    return CUW_OK;
  }
  k_tc_force<<<dim3(tm, tn), kThreads, ForcePipe::kSmem, h->stream>>>(tu, g.bsmall, nchk, h->nh, npro, h->ldu, g.pf(),
                                                                     g.half, g.gx, g.gy, g.gz, fpart, tc_err(h));
  CUW_LAUNCH_CHECK("k_tc_force");
  return CUW_OK;
}

}  // namespace cuw

// Check of the split-precision tensor-core path (no reference counterpart):
// C(M,N) = A(M,K) B(N,K)^T on device buffers, FP64 row-major with K
// contiguous, computed as three tf32 products with fp32 accumulation.
// err (device int) is set to 1 if a bounded wait ran out.
extern "C" int cuwaves_tc_gemm_check(int M, int N, int K, const double* A, const double* B, double* C, int* err,
                                     void* stream) {
  using namespace cuw;
  if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C || !err) return CUW_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t smem = GemmPipe::kSmem;
  if (smem_allow((const void*)k_tf32x3_gemm, (int)smem) != cudaSuccess) return CUW_ERR_CUDA;
  dim3 grid((M + 127) / 128, (N + 127) / 128);
  k_tf32x3_gemm<<<grid, kThreads, smem, st>>>(M, N, K, A, B, C, err);
  if (cudaGetLastError() != cudaSuccess) return CUW_ERR_CUDA;
  return CUW_OK;
}
