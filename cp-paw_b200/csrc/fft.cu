// Band-batched 3-D FFT with the local potential fused in (WAVES_VPSI).
//
// Reference: WAVES_VPSI (src/paw_waves1.f90:5099-5194) runs, per band, the
// three 1-D passes of PLANEWAVE_FFTGTOR (src/paw_fft.f90:2012-2177), multiplies
// by V(r), and runs the three passes of PLANEWAVE_FFTRTOG (:2180-2341).
// Conventions (src/paw_library.f90:2635-2728): G->r is exp(+iGr) and unscaled;
// r->G is exp(-iGr) with 1/N.  Like the reference, only the z-planes that hold
// G vectors are transformed in x and y (its NR3END1/NR3END2 pruning).
//
// B200 layout: three kernels per band batch.
//   gtor_plane : sphere -> xy-plane in shared memory, x then y transforms,
//                plane written to the work grid (only occupied planes).
//   zcol       : z columns: inverse z transform, V(r) and the 1/N scale, forward
//                z transform, between registers and one shared-memory tile.
//   rtog_plane : forward y then x transforms of a plane, gathered back onto
//                the sphere with 1/2|G|^2 (+bucket) psi added.
// A 1-D transform of a common length is two butterflies in registers with one
// exchange through shared memory (N = R1 R2, factors up to 12 or 16); any other
// length with prime factors up to 11 takes the Stockham stages (radix
// 2,3,4,5,7,8,11), which read all of their inputs into registers before a
// barrier and write after it, and so work in place.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "cuwaves_internal.cuh"

namespace cuw {

namespace {

constexpr int kMaxV = 8;   // complex values per thread per stage
// Grids (NR1, NR2, NR3) with kernels compiled for their lengths: the cubic
// grids of the benchmark systems, the grids the reference's rule picks for
// Si8 and Si64 at 60 Ry (28^3, 56^3), and the bulk-Si, water and small-system
// grids of the serving and batched workloads.
#define CUW_FFT_GRIDS                                                                              \
  CUW_FFT_GRID(18, 18, 18) CUW_FFT_GRID(18, 18, 36) CUW_FFT_GRID(24, 24, 24) CUW_FFT_GRID(28, 28, 28) \
  CUW_FFT_GRID(28, 28, 56) CUW_FFT_GRID(28, 56, 56) CUW_FFT_GRID(32, 32, 32) CUW_FFT_GRID(36, 36, 36) \
  CUW_FFT_GRID(48, 48, 48) CUW_FFT_GRID(56, 56, 56) CUW_FFT_GRID(56, 56, 110) CUW_FFT_GRID(64, 64, 64) \
  CUW_FFT_GRID(72, 72, 72) CUW_FFT_GRID(80, 80, 80) CUW_FFT_GRID(96, 96, 96)
constexpr int kPlaneThreads = 256;

// The transforms are written once for double2 (FP64 path) and float2 (the FP32
// FFT of the mixed-precision path).
template <class C>
struct CT;
template <>
struct CT<double2> {
  using R = double;
  __device__ __forceinline__ static double2 mk(double x, double y) { return make_double2(x, y); }
};
template <>
struct CT<float2> {
  using R = float;
  __device__ __forceinline__ static float2 mk(float x, float y) { return make_float2(x, y); }
};

// --- radix butterflies: v <- DFT_R(v) with exp(sign*2*pi*i*q*s/R) -----------
template <class C>
__device__ __forceinline__ C mul_i(C a, typename CT<C>::R sgn) {  // a * (sgn*i)
  return CT<C>::mk(-sgn * a.y, sgn * a.x);
}

template <int R>
struct Bfly;

template <>
struct Bfly<2> {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[2], typename CT<C>::R, const C*, int) {
    C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

template <>
struct Bfly<3> {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[3], typename CT<C>::R sgn, const C*, int) {
    using T = typename CT<C>::R;
    const T h = (T)0.86602540378443864676;  // sqrt(3)/2
    C a = v[0], t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    C u = mul_i(cscale(d, h), sgn);
    C m = CT<C>::mk(a.x - (T)0.5 * t.x, a.y - (T)0.5 * t.y);
    v[0] = cadd(a, t);
    v[1] = cadd(m, u);
    v[2] = csub(m, u);
  }
};

template <>
struct Bfly<4> {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[4], typename CT<C>::R sgn, const C*, int) {
    C t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    C t2 = cadd(v[1], v[3]), t3 = mul_i(csub(v[1], v[3]), sgn);
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3);
    v[3] = csub(t1, t3);
  }
};

template <>
struct Bfly<5> {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[5], typename CT<C>::R sgn, const C*, int) {
    using T = typename CT<C>::R;
    const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
    const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
    C a = v[0];
    C p1 = cadd(v[1], v[4]), m1 = csub(v[1], v[4]);
    C p2 = cadd(v[2], v[3]), m2 = csub(v[2], v[3]);
    C r1 = CT<C>::mk(a.x + c1 * p1.x + c2 * p2.x, a.y + c1 * p1.y + c2 * p2.y);
    C r2 = CT<C>::mk(a.x + c2 * p1.x + c1 * p2.x, a.y + c2 * p1.y + c1 * p2.y);
    C i1 = mul_i(CT<C>::mk(s1 * m1.x + s2 * m2.x, s1 * m1.y + s2 * m2.y), sgn);
    C i2 = mul_i(CT<C>::mk(s2 * m1.x - s1 * m2.x, s2 * m1.y - s1 * m2.y), sgn);
    v[0] = CT<C>::mk(a.x + p1.x + p2.x, a.y + p1.y + p2.y);
    v[1] = cadd(r1, i1);
    v[4] = csub(r1, i1);
    v[2] = cadd(r2, i2);
    v[3] = csub(r2, i2);
  }
};

template <>
struct Bfly<8> {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[8], typename CT<C>::R sgn, const C*, int) {
    using T = typename CT<C>::R;
    const T q = (T)0.70710678118654752440;
    C e[4] = {v[0], v[2], v[4], v[6]};
    C o[4] = {v[1], v[3], v[5], v[7]};
    Bfly<4>::run(e, sgn, (const C*)nullptr, 0);
    Bfly<4>::run(o, sgn, (const C*)nullptr, 0);
    // twiddles W8^k = exp(sgn*i*pi*k/4)
    C w1 = CT<C>::mk(q, sgn * q), w3 = CT<C>::mk(-q, sgn * q);
    C o1 = cmul(o[1], w1), o2 = mul_i(o[2], sgn), o3 = cmul(o[3], w3);
    v[0] = cadd(e[0], o[0]);
    v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], o1);
    v[5] = csub(e[1], o1);
    v[2] = cadd(e[2], o2);
    v[6] = csub(e[2], o2);
    v[3] = cadd(e[3], o3);
    v[7] = csub(e[3], o3);
  }
};

// cos and sin of 2 pi k / R, k = 0 .. R/2, of the butterflies whose twiddles
// are not handled above
template <int R>
__host__ __device__ constexpr double root_c(int k) {
  constexpr double c7[4] = {1.0, 0.623489801858733530525, -0.222520933956314404288, -0.900968867902419126236};
  constexpr double c9[5] = {1.0, 0.766044443118978035202, 0.173648177666930348851, -0.5, -0.939692620785908384054};
  constexpr double c11[6] = {1.0, 0.841253532831181168861, 0.415415013001886425529, -0.142314838273285140443,
                             -0.654860733945285064056, -0.959492973614497389890};
  constexpr double c16[9] = {1.0, 0.923879532511286756128, 0.707106781186547524400, 0.382683432365089771728, 0.0,
                             -0.382683432365089771728, -0.707106781186547524400, -0.923879532511286756128, -1.0};
  return R == 7 ? c7[k] : (R == 9 ? c9[k] : (R == 11 ? c11[k] : c16[k]));
}
template <int R>
__host__ __device__ constexpr double root_s(int k) {
  constexpr double s7[4] = {0.0, 0.781831482468029808708, 0.974927912181823607018, 0.433883739117558120476};
  constexpr double s9[5] = {0.0, 0.642787609686539326323, 0.984807753012208059367, 0.866025403784438646764,
                            0.342020143325668733044};
  constexpr double s11[6] = {0.0, 0.540640817455597582108, 0.909631995354518371412, 0.989821441880932732377,
                             0.755749574354258283774, 0.281732556841429697711};
  constexpr double s16[9] = {0.0, 0.382683432365089771728, 0.707106781186547524400, 0.923879532511286756128, 1.0,
                             0.923879532511286756128, 0.707106781186547524400, 0.382683432365089771728, 0.0};
  return R == 7 ? s7[k] : (R == 9 ? s9[k] : (R == 11 ? s11[k] : s16[k]));
}

// odd prime radix: the symmetric and antisymmetric sums of v[q], v[R-q] with
// real constants
template <int R>
struct BflyPrime {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[R], typename CT<C>::R sgn, const C*, int) {
    using T = typename CT<C>::R;
    constexpr int H = R / 2;
    C p[H], m[H];
    const C a = v[0];
    C t = a;
#pragma unroll
    for (int q = 0; q < H; ++q) {
      p[q] = cadd(v[q + 1], v[R - 1 - q]);
      m[q] = csub(v[q + 1], v[R - 1 - q]);
      t = cadd(t, p[q]);
    }
    v[0] = t;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      C r = a, i = CT<C>::mk(0, 0);
#pragma unroll
      for (int q = 1; q <= H; ++q) {
        const int e = (q * k) % R, f = e <= H ? e : R - e;
        const T c = (T)root_c<R>(f), d = (T)(e <= H ? root_s<R>(f) : -root_s<R>(f));
        r.x += c * p[q - 1].x;
        r.y += c * p[q - 1].y;
        i.x += d * m[q - 1].x;
        i.y += d * m[q - 1].y;
      }
      i = mul_i(i, sgn);
      v[k] = cadd(r, i);
      v[R - k] = csub(r, i);
    }
  }
};
template <>
struct Bfly<7> : BflyPrime<7> {};
template <>
struct Bfly<11> : BflyPrime<11> {};

// radix A*B with coprime A and B, without twiddles: element (B a + A b) mod R
// of the input and element k = (ka mod A, kb mod B) of the output
template <int A, int B>
__host__ __device__ constexpr int crt(int ka, int kb) {
  for (int k = 0; k < A * B; ++k)
    if (k % A == ka && k % B == kb) return k;
  return 0;
}
template <int A, int B>
struct BflyCoprime {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[A * B], typename CT<C>::R sgn, const C*, int) {
    constexpr int R = A * B;
    C y[B][A];
#pragma unroll
    for (int b = 0; b < B; ++b) {
#pragma unroll
      for (int a = 0; a < A; ++a) y[b][a] = v[(B * a + A * b) % R];
      Bfly<A>::run(y[b], sgn, (const C*)nullptr, 0);
    }
#pragma unroll
    for (int a = 0; a < A; ++a) {
      C z[B];
#pragma unroll
      for (int b = 0; b < B; ++b) z[b] = y[b][a];
      Bfly<B>::run(z, sgn, (const C*)nullptr, 0);
#pragma unroll
      for (int b = 0; b < B; ++b) v[crt<A, B>(a, b)] = z[b];
    }
  }
};
template <>
struct Bfly<6> : BflyCoprime<2, 3> {};
template <>
struct Bfly<10> : BflyCoprime<2, 5> {};
template <>
struct Bfly<12> : BflyCoprime<4, 3> {};

// radix Q*Q with constant twiddles
template <int Q>
struct BflySquare {
  template <class C>
  __device__ __forceinline__ static void run(C (&v)[Q * Q], typename CT<C>::R sgn, const C*, int) {
    using T = typename CT<C>::R;
    constexpr int R = Q * Q;
    C y[Q][Q];
#pragma unroll
    for (int b = 0; b < Q; ++b) {
#pragma unroll
      for (int a = 0; a < Q; ++a) y[b][a] = v[b + Q * a];
      Bfly<Q>::run(y[b], sgn, (const C*)nullptr, 0);
#pragma unroll
      for (int a = 1; a < Q; ++a) {
        if (b == 0) continue;
        const int e = a * b, f = e <= R / 2 ? e : R - e;
        const T c = (T)root_c<R>(f), d = (T)(e <= R / 2 ? root_s<R>(f) : -root_s<R>(f));
        y[b][a] = cmul(y[b][a], CT<C>::mk(c, sgn * d));
      }
    }
#pragma unroll
    for (int a = 0; a < Q; ++a) {
      C z[Q];
#pragma unroll
      for (int b = 0; b < Q; ++b) z[b] = y[b][a];
      Bfly<Q>::run(z, sgn, (const C*)nullptr, 0);
#pragma unroll
      for (int b = 0; b < Q; ++b) v[a + Q * b] = z[b];
    }
  }
};
template <>
struct Bfly<9> : BflySquare<3> {};
template <>
struct Bfly<16> : BflySquare<4> {};

// N = r1 * r2 (r1 <= r2) with the two factors as even as the butterflies allow
// (both at most 12, or 8 x 16); {0, 0} when N has no such split
struct Split2 {
  int r1, r2;
};
__host__ __device__ constexpr bool has_bfly(int r) { return (r >= 2 && r <= 12) || r == 16; }
__host__ __device__ constexpr Split2 split2(int N) {
  for (int a = 12; a >= 2; --a)
    if (N % a == 0 && a <= N / a && has_bfly(N / a)) return Split2{a, N / a};
  return Split2{0, 0};
}

// One Stockham stage on lines [line0, line0+nl) of length n held in shared
// memory: element e of line L lives at buf[L*ls + e*es].  tw[k] = exp(sgn*2 pi i k/n).
// Consecutive threads take consecutive lines.
// The caller guarantees nl*n/R <= blockDim.x * BPT.
template <int R, class C>
__device__ __noinline__ void stage(C* buf, int n, int ns, int line0, int nl, int ls, int es,
                                      const C* tw, typename CT<C>::R sgn) {
  constexpr int BPT = (kMaxV / R) > 0 ? (kMaxV / R) : 1;
  const int nq = n / R;
  const int total = nl * nq;
  C v[BPT][R];
  int line_[BPT], j_[BPT];
#pragma unroll
  for (int t = 0; t < BPT; ++t) {
    int bf = threadIdx.x + t * blockDim.x;
    line_[t] = -1;
    if (bf < total) {
      const int j = bf / nl, line = line0 + bf % nl;
      line_[t] = line;
      j_[t] = j;
      const int k = j % ns;
      const int tstep = n / (ns * R);
      C* base = buf + (size_t)line * ls;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        C x = base[(size_t)(j + r * nq) * es];
        if (r && k) x = cmul(x, tw[(r * k * tstep) % n]);
        v[t][r] = x;
      }
      Bfly<R>::run(v[t], sgn, tw, n);
    }
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < BPT; ++t) {
    if (line_[t] >= 0) {
      const int j = j_[t], k = j % ns;
      const int idxd = (j / ns) * ns * R + k;
      C* base = buf + (size_t)line_[t] * ls;
#pragma unroll
      for (int r = 0; r < R; ++r) base[(size_t)(idxd + r * ns) * es] = v[t][r];
    }
  }
  __syncthreads();
}

__host__ __device__ constexpr int bpt_of(int r) { return (kMaxV / r) > 0 ? (kMaxV / r) : 1; }

struct AxisArg {
  int n;
  int nstage;
  int radix[8];
};

// ---------------------------------------------------------------------------
// Compile-time specialisation of the Stockham stages: every divisor of
// the index arithmetic is a constant, the stages are inlined and the block
// size is fixed (kPlaneThreads), so the lines per chunk are constant too.
// ---------------------------------------------------------------------------
struct RadixList {
  int n;
  int r[8];
};
__host__ __device__ constexpr RadixList radices_of(int N) {
  RadixList L{0, {0, 0, 0, 0, 0, 0, 0, 0}};
  int m = N;
  const int order[7] = {8, 4, 2, 3, 5, 7, 11};
  for (int i = 0; i < 7; ++i)
    while (m % order[i] == 0 && L.n < 8) {
      L.r[L.n++] = order[i];
      m /= order[i];
    }
  return L;
}
__host__ __device__ constexpr int chunk_lines(int N) {
  RadixList L = radices_of(N);
  int lc = 1 << 30;
  for (int s = 0; s < L.n; ++s) {
    int cap = (kPlaneThreads * bpt_of(L.r[s]) * L.r[s]) / N;
    if (cap < 1) cap = 1;
    lc = lc < cap ? lc : cap;
  }
  return lc;
}

template <int N, int R, int NS, int LC, class C>
__device__ __forceinline__ void stage_fixed(C* buf, int line0, int nl, int ls, int es, const C* tw,
                                            typename CT<C>::R sgn) {
  constexpr int BPT = bpt_of(R);
  constexpr int NQ = N / R;
  constexpr int TSTEP = N / (NS * R);
  // the full chunk LC*NQ decoded modulo LC, with the lines beyond nl masked
  C v[BPT][R];
  int off_[BPT];
  bool act[BPT];
#pragma unroll
  for (int t = 0; t < BPT; ++t) {
    const int bf = threadIdx.x + t * kPlaneThreads;
    const int line = bf % LC, j = bf / LC;
    act[t] = line < nl && j < NQ;
    const int k = j % NS;
    off_[t] = line * N + ((j / NS) * NS * R + k);  // (line, destination index) packed
    if (act[t]) {
      C* base = buf + (size_t)(line0 + line) * ls;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        C x = base[(size_t)(j + r * NQ) * es];
        if (r && k) x = cmul(x, tw[(r * k * TSTEP) % N]);
        v[t][r] = x;
      }
      Bfly<R>::run(v[t], sgn, tw, N);
    }
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < BPT; ++t) {
    if (act[t]) {
      const int line = off_[t] / N, idxd = off_[t] % N;
      C* base = buf + (size_t)(line0 + line) * ls;
#pragma unroll
      for (int r = 0; r < R; ++r) base[(size_t)(idxd + r * NS) * es] = v[t][r];
    }
  }
  __syncthreads();
}

template <int N, int S, int NS, int LC, class C>
__device__ __forceinline__ void stages_fixed(C* buf, int line0, int nl, int ls, int es, const C* tw,
                                             typename CT<C>::R sgn) {
  constexpr RadixList L = radices_of(N);
  if constexpr (S < L.n) {
    constexpr int R = L.r[S];
    stage_fixed<N, R, NS, LC>(buf, line0, nl, ls, es, tw, sgn);
    stages_fixed<N, S + 1, NS * R, LC>(buf, line0, nl, ls, es, tw, sgn);
  }
}

template <int N, class C>
__device__ void transform_fixed(C* buf, int nlines, int ls, int es, const C* tw, typename CT<C>::R sgn) {
  constexpr int LC = chunk_lines(N);
  for (int l0 = 0; l0 < nlines; l0 += LC) {
    const int nl = min(LC, nlines - l0);
    stages_fixed<N, 0, 1, LC>(buf, l0, nl, ls, es, tw, sgn);
  }
}

// lines per chunk so that every stage fits one pass of the block
__device__ __forceinline__ int lines_per_chunk(const AxisArg& ax, int nlines) {
  int lc = nlines;
  for (int s = 0; s < ax.nstage; ++s) {
    int r = ax.radix[s];
    int cap = (int)(((long)blockDim.x * bpt_of(r) * r) / ax.n);
    if (cap < 1) cap = 1;
    lc = min(lc, cap);
  }
  return lc;
}

template <class C>
__device__ void transform(C* buf, const AxisArg& ax, int nlines, int ls, int es, const C* tw,
                          typename CT<C>::R sgn) {
  switch (ax.n) {
    case 16: transform_fixed<16>(buf, nlines, ls, es, tw, sgn); return;
    case 20: transform_fixed<20>(buf, nlines, ls, es, tw, sgn); return;
    case 24: transform_fixed<24>(buf, nlines, ls, es, tw, sgn); return;
    case 28: transform_fixed<28>(buf, nlines, ls, es, tw, sgn); return;
    case 32: transform_fixed<32>(buf, nlines, ls, es, tw, sgn); return;
    case 36: transform_fixed<36>(buf, nlines, ls, es, tw, sgn); return;
    case 40: transform_fixed<40>(buf, nlines, ls, es, tw, sgn); return;
    case 48: transform_fixed<48>(buf, nlines, ls, es, tw, sgn); return;
    case 56: transform_fixed<56>(buf, nlines, ls, es, tw, sgn); return;
    case 64: transform_fixed<64>(buf, nlines, ls, es, tw, sgn); return;
    case 72: transform_fixed<72>(buf, nlines, ls, es, tw, sgn); return;
    case 80: transform_fixed<80>(buf, nlines, ls, es, tw, sgn); return;
    case 96: transform_fixed<96>(buf, nlines, ls, es, tw, sgn); return;
    default: break;
  }
  const int lc = lines_per_chunk(ax, nlines);
  for (int l0 = 0; l0 < nlines; l0 += lc) {
    const int nl = min(lc, nlines - l0);
    int ns = 1;
    for (int s = 0; s < ax.nstage; ++s) {
      switch (ax.radix[s]) {
        case 2: stage<2>(buf, ax.n, ns, l0, nl, ls, es, tw, sgn); break;
        case 3: stage<3>(buf, ax.n, ns, l0, nl, ls, es, tw, sgn); break;
        case 4: stage<4>(buf, ax.n, ns, l0, nl, ls, es, tw, sgn); break;
        case 5: stage<5>(buf, ax.n, ns, l0, nl, ls, es, tw, sgn); break;
        case 7: stage<7>(buf, ax.n, ns, l0, nl, ls, es, tw, sgn); break;
        case 8: stage<8>(buf, ax.n, ns, l0, nl, ls, es, tw, sgn); break;
        case 11: stage<11>(buf, ax.n, ns, l0, nl, ls, es, tw, sgn); break;
      }
      ns *= ax.radix[s];
    }
  }
}

// load twiddles exp(sgn*2 pi i k/n) from the FP64 table exp(+2 pi i k/n)
template <class C>
__device__ void load_tw(C* dst, const double2* src, int n, double sgn) {
  using T = typename CT<C>::R;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    double2 w = src[k];
    dst[k] = CT<C>::mk((T)w.x, (T)(sgn * w.y));
  }
}

template <class C>
__device__ __forceinline__ C from_d2(double2 a) {
  using T = typename CT<C>::R;
  return CT<C>::mk((T)a.x, (T)a.y);
}
__device__ __forceinline__ double2 to_d2(double2 a) { return a; }
__device__ __forceinline__ double2 to_d2(float2 a) { return make_double2((double)a.x, (double)a.y); }

// Shared-memory layout of an xy plane: rows of NR1 elements at a stride of
// NR1+1, and the x lines transformed with consecutive threads on consecutive
// rows.  With the odd stride, the eight (FP64) or sixteen (FP32) threads that
// share a shared-memory wavefront touch eight/sixteen different 16/8-byte bank
// groups in every Stockham stage; with the dense stride NR1 = 2^k, the
// scattered writes of the first radix-8 stage of the x lines (stride 8
// elements) hit one bank group eight times.
__host__ __device__ constexpr int plane_stride(int nr1) { return nr1 + 1; }
// ---------------------------------------------------------------------------
// The kernels take the work-grid type C (double2 or float2); the sphere
// coefficients psi/out stay FP64 and are converted at the gather/scatter.
template <class C>
__global__ void __launch_bounds__(kPlaneThreads, 2)
    k_gtor_any(const double2* __restrict__ psi, int ldg, int b0, const int* __restrict__ plane_off,
                 const int* __restrict__ plane_g, const int* __restrict__ plane_pos,
                 C* __restrict__ grid, int nzp, AxisArg a1, AxisArg a2, const double2* __restrict__ tw1g,
                 const double2* __restrict__ tw2g) {
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  const int nr1 = a1.n, nr2 = a2.n, npl = nr1 * nr2, ps = plane_stride(nr1);
  C* plane = sm;  // [nr2][ps]
  C* tw1 = sm + nr2 * ps;
  C* tw2 = tw1 + nr1;
  const int p = blockIdx.x, bl = blockIdx.y, b = b0 + bl;
  for (int i = threadIdx.x; i < nr2 * ps; i += blockDim.x) plane[i] = CT<C>::mk(0, 0);
  load_tw(tw1, tw1g, nr1, +1.0);
  load_tw(tw2, tw2g, nr2, +1.0);
  __syncthreads();
  const double2* src = psi + (size_t)ldg * b;
  for (int k = plane_off[p] + threadIdx.x; k < plane_off[p + 1]; k += blockDim.x)
    plane[plane_pos[k]] = from_d2<C>(src[plane_g[k]]);
  __syncthreads();
  transform(plane, a1, nr2, ps, 1, tw1, (typename CT<C>::R)1);   // x lines
  transform(plane, a2, nr1, 1, ps, tw2, (typename CT<C>::R)1);   // y lines
  C* dst = grid + ((size_t)bl * nzp + p) * npl;
  for (int i = threadIdx.x; i < npl; i += blockDim.x) dst[i] = plane[i + i / nr1];
}

// z columns of any length: Stockham stages on a tile of kTX columns of a y row
constexpr int kTX = 16;
template <class C>
__global__ void __launch_bounds__(kPlaneThreads, 2)
    k_zcol_v(C* __restrict__ grid, const double* __restrict__ v, const int* __restrict__ zslot, int nzp, int nr1,
             int nr2, AxisArg a3, const double2* __restrict__ tw3g, double scale) {
  using T = typename CT<C>::R;
  constexpr int TX = kTX;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  const int nr3 = a3.n;
  C* tile = sm;             // [nr3][TX]
  C* tw = sm + nr3 * TX;
  const int nxb = (nr1 + TX - 1) / TX;
  const int iy = blockIdx.x / nxb, x0 = (blockIdx.x % nxb) * TX;
  const int bl = blockIdx.y;
  const size_t npl = (size_t)nr1 * nr2;
  C* gb = grid + (size_t)bl * nzp * npl;
  load_tw(tw, tw3g, nr3, +1.0);
  for (int i = threadIdx.x; i < nr3 * TX; i += blockDim.x) {
    int iz = i / TX, x = i % TX;
    int s = zslot[iz];
    C val = CT<C>::mk(0, 0);
    if (s >= 0 && x0 + x < nr1) val = gb[(size_t)s * npl + (size_t)iy * nr1 + x0 + x];
    tile[i] = val;
  }
  __syncthreads();
  transform(tile, a3, TX, 1, TX, tw, (T)1);
  for (int i = threadIdx.x; i < nr3 * TX; i += blockDim.x) {
    int iz = i / TX, x = i % TX;
    double vv = 0.0;
    if (x0 + x < nr1) vv = v[(size_t)x0 + x + (size_t)nr1 * (iy + (size_t)nr2 * iz)] * scale;
    tile[i] = cscale(tile[i], (T)vv);
  }
  __syncthreads();
  // forward transform: conjugated twiddles
  for (int k = threadIdx.x; k < nr3; k += blockDim.x) tw[k].y = -tw[k].y;
  __syncthreads();
  transform(tile, a3, TX, 1, TX, tw, (T)-1);
  for (int i = threadIdx.x; i < nr3 * TX; i += blockDim.x) {
    int iz = i / TX, x = i % TX;
    int s = zslot[iz];
    if (s >= 0 && x0 + x < nr1) gb[(size_t)s * npl + (size_t)iy * nr1 + x0 + x] = tile[i];
  }
}

// z transforms of lengths N = R1 R2 with both factors in one butterfly: kZX
// consecutive columns of the xy plane per block (whatever rows they lie in),
// one column per lane, and R2 warps.  Warp t takes x[t + R2 r] from the work
// grid into registers, a radix-R1 butterfly and the twiddles, and leaves
// element (k1, t) in shared memory; warp k1 reads its row (k1, .), and after a
// radix-R2 butterfly holds X[k1 + R1 k2] = psi(z).  V(r) is applied there in
// registers, and the R->G transform runs the same two steps backwards: radix R2
// over k2, twiddles, the same row of slots, and warp m1's radix-R1 butterfly
// gives x[m1 + R2 m2], which goes straight to the work grid.  Shared memory is
// crossed twice and there are two barriers a band; every slot is written by the
// thread that read it last, so the next band needs no barrier of its own.
// V of the block's columns stays in registers over the `nbb` bands of a block.
//
// What bounds it: the work grid's bytes from L2 (the batch is sized for it)
// and the barriers' latency, hidden by 2 to 4 blocks an SM.  The Stockham
// stages that it replaces crossed shared memory once more for every radix and
// for the copies in and out, with two block barriers each: 32 bands of 72^3 in
// FP32 took 384 us and take 42, 43 bands of 64^3 69 (by a kernel of their own)
// and 36; a whole CP step of Si128 (56 x 56 x 110, FP64) 12.6 ms and 11.0 ms.
constexpr int kZX = 32;
template <int N>
constexpr int kZThreads = kZX * split2(N).r2;
// blocks an SM that the register limit leaves room for: about 64 registers a
// thread in FP32 and 128 in FP64
template <class C, int N>
constexpr int kZBlocks = ((sizeof(C) == 8 ? 1024 : 512) + kZThreads<N> / 4) / kZThreads<N>;

// shared memory of a z kernel with TX columns: tile, twiddles, plane offsets
template <class C>
constexpr int z_smem(int n, int tx) { return (int)((n * tx + n) * sizeof(C) + n * sizeof(int)); }

template <class C, int N>
__global__ void __launch_bounds__(kZThreads<N>, kZBlocks<C, N>)
    k_zcol(C* __restrict__ grid, const double* __restrict__ v, const int* __restrict__ zslot, int nzp, int npl,
           const double2* __restrict__ tw3g, double scale, int nb, int nbb) {
  using T = typename CT<C>::R;
  constexpr int R1 = split2(N).r1, R2 = split2(N).r2;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = reinterpret_cast<C*>(smraw);  // [R1][R2][kZX]
  C* tw = buf + N * kZX;
  int* zs = reinterpret_cast<int*>(tw + N);
  const int x = threadIdx.x % kZX, j = threadIdx.x / kZX;
  const int c = blockIdx.x * kZX + x;
  const bool in = c < npl;
  load_tw(tw, tw3g, N, +1.0);
  for (int i = threadIdx.x; i < N; i += blockDim.x) zs[i] = zslot[i];
  T vr[R2];
  if (j < R1) {
#pragma unroll
    for (int k = 0; k < R2; ++k) vr[k] = in ? (T)(v[(size_t)(j + R1 * k) * npl + c] * scale) : (T)0;
  }
  __syncthreads();
  const int b1 = min(nb, ((int)blockIdx.y + 1) * nbb);
  for (int bl = blockIdx.y * nbb; bl < b1; ++bl) {
    C* gb = grid + (size_t)bl * nzp * npl + c;
    C a[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      const int s = zs[j + R2 * r];
      a[r] = in && s >= 0 ? gb[(size_t)s * npl] : CT<C>::mk(0, 0);
    }
    Bfly<R1>::run(a, (T)1, (const C*)nullptr, 0);
    C* slot = buf + j * kZX + x;
    slot[0] = a[0];
#pragma unroll
    for (int k = 1; k < R1; ++k) slot[k * R2 * kZX] = cmul(a[k], tw[k * j]);
    __syncthreads();
    if (j < R1) {
      C b[R2];
      C* row = buf + j * R2 * kZX + x;
#pragma unroll
      for (int t = 0; t < R2; ++t) b[t] = row[t * kZX];
      Bfly<R2>::run(b, (T)1, (const C*)nullptr, 0);
#pragma unroll
      for (int k = 0; k < R2; ++k) b[k] = cscale(b[k], vr[k]);
      Bfly<R2>::run(b, (T)-1, (const C*)nullptr, 0);
      row[0] = b[0];
#pragma unroll
      for (int m = 1; m < R2; ++m) row[m * kZX] = cmulc(b[m], tw[m * j]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < R1; ++k) a[k] = slot[k * R2 * kZX];
    Bfly<R1>::run(a, (T)-1, (const C*)nullptr, 0);
#pragma unroll
    for (int m = 0; m < R1; ++m) {
      const int s = zs[j + R2 * m];
      if (in && s >= 0) gb[(size_t)s * npl] = a[m];
    }
  }
}

// Pseudo density of WAVES_DENSITY (src/paw_waves1.f90:5377-5500) for super
// wave functions at the Gamma point: after the x/y passes of k_gtor_plane, the
// G->R z transform of the block's x columns of every band of the batch in turn,
// and rho(r) += f1 Re(psi)^2 + f2 Im(psi)^2 (= Re[psi (s1 conj psi + s2 psi)]
// with s1,2 = (f1 +- f2)/2, :5474-5496) in FP64, bands in order, so that the
// sum is deterministic; `first` starts rho from zero, else the batch adds to it.
// Lengths N = R1 R2 take the first two steps of k_zcol, with rho(r) of the
// thread's points in registers and the next band's elements loaded before the
// current band's second step; kRhoX columns a block, because the bands are a
// serial chain and more blocks in flight hide its barriers.  The register limit
// leaves room for 480 threads an SM: at 72^3 in FP64 the 324 blocks then fit
// one wave (three an SM), 16 bands in 31.9 us; with two an SM they took 49.0.
constexpr int kRhoX = 16;
template <int N>
constexpr int kRhoThreads = (kRhoX * split2(N).r2 + 31) / 32 * 32;

template <class C, int N>
__global__ void __launch_bounds__(kRhoThreads<N>, 480 / kRhoThreads<N>)
    k_zrho(const C* __restrict__ grid, const int* __restrict__ zslot, int nzp, int npl,
           const double2* __restrict__ tw3g, const double* __restrict__ occ, int nb, int b0, int nbatch,
           double* __restrict__ rho, int first) {
  using T = typename CT<C>::R;
  constexpr int R1 = split2(N).r1, R2 = split2(N).r2;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = reinterpret_cast<C*>(smraw);  // [R1][R2][kRhoX]
  C* tw = buf + N * kRhoX;
  int* zs = reinterpret_cast<int*>(tw + N);
  const int x = threadIdx.x % kRhoX, j = threadIdx.x / kRhoX;
  const int c = blockIdx.x * kRhoX + x;
  const bool in = c < npl, one = j < R2, two = j < R1;  // the block is padded to whole warps
  load_tw(tw, tw3g, N, +1.0);
  for (int i = threadIdx.x; i < N; i += blockDim.x) zs[i] = zslot[i];
  double acc[R2];
#pragma unroll
  for (int k = 0; k < R2; ++k) acc[k] = !first && in && two ? rho[(size_t)(j + R1 * k) * npl + c] : 0.0;
  __syncthreads();
  C a[R1];
  auto load = [&](int bl) {
    const C* gb = grid + (size_t)bl * nzp * npl + c;
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      const int s = one ? zs[j + R2 * r] : -1;
      a[r] = in && s >= 0 ? gb[(size_t)s * npl] : CT<C>::mk(0, 0);
    }
  };
  load(0);
  for (int bl = 0; bl < nbatch; ++bl) {
    const int b = b0 + bl;
    const double f1 = occ[2 * b], f2 = 2 * b + 1 < nb ? occ[2 * b + 1] : 0.0;
    const bool live = f1 != 0.0 || f2 != 0.0;  // the same for the whole block
    if (live) {
      Bfly<R1>::run(a, (T)1, (const C*)nullptr, 0);
      if (one) {
        C* slot = buf + j * kRhoX + x;
        slot[0] = a[0];
#pragma unroll
        for (int k = 1; k < R1; ++k) slot[k * R2 * kRhoX] = cmul(a[k], tw[k * j]);
      }
    }
    if (bl + 1 < nbatch) load(bl + 1);
    if (!live) continue;
    __syncthreads();
    if (two) {
      C d[R2];
      const C* row = buf + j * R2 * kRhoX + x;
#pragma unroll
      for (int t = 0; t < R2; ++t) d[t] = row[t * kRhoX];
      Bfly<R2>::run(d, (T)1, (const C*)nullptr, 0);
#pragma unroll
      for (int k = 0; k < R2; ++k) {
        const double re = (double)d[k].x, im = (double)d[k].y;
        acc[k] += f1 * re * re + f2 * im * im;
      }
    }
    __syncthreads();  // the rows are read before the next band writes them
  }
#pragma unroll
  for (int k = 0; k < R2; ++k)
    if (in && two) rho[(size_t)(j + R1 * k) * npl + c] = acc[k];
}

// the same for any other length: Stockham stages on a tile of kRhoTX columns
constexpr int kRhoTX = 16;
template <class C>
__global__ void __launch_bounds__(kPlaneThreads, 2)
    k_zcol_rho(const C* __restrict__ grid, const int* __restrict__ zslot, int nzp, int nr1, int nr2, AxisArg a3,
               const double2* __restrict__ tw3g, const double* __restrict__ occ, int nb, int b0, int nbatch,
               double* __restrict__ rho, int first) {
  using T = typename CT<C>::R;
  constexpr int TX = kRhoTX;
  constexpr int EPT = 8;  // tile elements per thread (nr3 * TX <= EPT * blockDim)
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  const int nr3 = a3.n;
  C* tile = sm;  // [nr3][TX]
  C* tw = sm + nr3 * TX;
  const int nxb = (nr1 + TX - 1) / TX;
  const int iy = blockIdx.x / nxb, x0 = (blockIdx.x % nxb) * TX;
  const size_t npl = (size_t)nr1 * nr2;
  load_tw(tw, tw3g, nr3, +1.0);
  double acc[EPT];
#pragma unroll
  for (int e = 0; e < EPT; ++e) {
    const int i = threadIdx.x + e * blockDim.x, iz = i / TX, x = i % TX;
    const bool in = i < nr3 * TX && x0 + x < nr1;
    acc[e] = (!first && in) ? rho[(size_t)x0 + x + (size_t)nr1 * (iy + (size_t)nr2 * iz)] : 0.0;
  }
  for (int bl = 0; bl < nbatch; ++bl) {
    const int b = b0 + bl;
    const double f1 = occ[2 * b], f2 = 2 * b + 1 < nb ? occ[2 * b + 1] : 0.0;
    if (f1 == 0.0 && f2 == 0.0) continue;  // the same for the whole block
    const C* gb = grid + (size_t)bl * nzp * npl;
    __syncthreads();  // the previous band's reads of the tile are done
    for (int i = threadIdx.x; i < nr3 * TX; i += blockDim.x) {
      const int iz = i / TX, x = i % TX, s = zslot[iz];
      C val = CT<C>::mk(0, 0);
      if (s >= 0 && x0 + x < nr1) val = gb[(size_t)s * npl + (size_t)iy * nr1 + x0 + x];
      tile[i] = val;
    }
    __syncthreads();
    transform(tile, a3, TX, 1, TX, tw, (T)1);
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const int i = threadIdx.x + e * blockDim.x;
      if (i < nr3 * TX) {
        const double re = (double)tile[i].x, im = (double)tile[i].y;
        acc[e] += f1 * re * re + f2 * im * im;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < EPT; ++e) {
    const int i = threadIdx.x + e * blockDim.x, iz = i / TX, x = i % TX;
    if (i < nr3 * TX && x0 + x < nr1) rho[(size_t)x0 + x + (size_t)nr1 * (iy + (size_t)nr2 * iz)] = acc[e];
  }
}

// xy planes of compiled lengths, each axis N = R1 R2 in two register steps that
// work in place: a thread reads the R1 (then R2) elements of its butterfly from
// shared memory and writes its results to the same slots, so that a step needs
// one barrier and no staging.  The digit reversal this leaves is taken out
// where the values are permuted anyway: x line slot r + R1 t holds x = t + R2 r
// when the sphere is scattered (k_gtor_plane), and slot R2 k1 + k2 holds
// x = k1 + R1 k2 when it is gathered (k_rtog_plane).  The last y step of G->R
// writes the work grid itself, and the first one of R->G reads it, so the plane
// crosses shared memory three and a half times.  Only the rows that hold G
// vectors (y0 + l mod N2, l < ny; one range of signed y) are cleared, get x
// transforms, and are read by the first y step or written by the last.
//
// What bounds them: shared-memory passes and the barriers between them (a plane
// is 33 to 150 KB, so few blocks share an SM).  Before, every radix of a
// Stockham stage crossed shared memory with two barriers and the plane was
// copied in and out: 32 bands of 72^3 in FP32, G->R 63.3 -> 28.6 us and R->G
// 97.0 -> 33.8 us; 16 bands of 72^3 in FP64, G->R 44.7 -> 26.1 us.
//
// Plan variants V (chosen per handle by the autotuner; src/paw_library.f90
// LIB_FFTW3 leaves the same choice to FFTW's measured planning):
//   bit 0: 512 instead of 256 threads a plane;
//   bit 1: R1 and R2 exchanged.
// V = 0 is the default: H|psi> of 32 H2O on 72^3 takes 497, 552 and 498 us with
// V = 0, 1, 2 in FP64 and 307, 324 and 306 us in mixed precision; the tuner
// finds the handles where another order of the factors is ahead.
// Variants 0, 1 and 2 are V = 0, 1, 2; 64^3 grids also have variant 3, both.
constexpr int kFftVariants = 4;
__host__ __device__ constexpr int plane_threads(int V) { return (V & 1) ? 2 * kPlaneThreads : kPlaneThreads; }
template <int N, int V>
struct Axis2 {
  static constexpr int R1 = (V & 2) ? split2(N).r2 : split2(N).r1;
  static constexpr int R2 = (V & 2) ? split2(N).r1 : split2(N).r2;
};
// blocks an SM that registers are budgeted for: 64 registers a thread in FP32, 128 in FP64
template <class C, int V>
constexpr int kPlaneBlocks = (sizeof(C) == 8 ? 1024 : 512) / plane_threads(V);

// R elements at p, p + st, ..., through a butterfly; element k times exp(sgn 2 pi i k e / N)
template <int R, class C>
__device__ __forceinline__ void take(C (&a)[R], const C* p, int st) {
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = p[r * st];
}
template <int R, bool TW, class C>
__device__ __forceinline__ void put(const C (&a)[R], C* p, int st, const C* tw, int e) {
  p[0] = a[0];
#pragma unroll
  for (int k = 1; k < R; ++k) p[k * st] = TW ? cmul(a[k], tw[k * e]) : a[k];
}

template <class C, int N1, int N2, int V>
__global__ void __launch_bounds__(plane_threads(V), kPlaneBlocks<C, V>)
    k_gtor_plane(const double2* __restrict__ psi, int ldg, int b0, const int* __restrict__ plane_off,
                 const int* __restrict__ plane_g, const int* __restrict__ plane_pos, const int2* __restrict__ plane_rows,
                 C* __restrict__ grid, int nzp, const double2* __restrict__ tw1g, const double2* __restrict__ tw2g) {
  using T = typename CT<C>::R;
  constexpr int NT = plane_threads(V), PS = plane_stride(N1);
  constexpr int A1 = Axis2<N1, V>::R1, A2 = Axis2<N1, V>::R2, B1 = Axis2<N2, V>::R1, B2 = Axis2<N2, V>::R2;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* plane = reinterpret_cast<C*>(smraw);  // [N2][PS]
  C* tw1 = plane + N2 * PS;
  C* tw2 = tw1 + N1;
  const int p = blockIdx.x, bl = blockIdx.y, b = b0 + bl;
  const int2 rows = plane_rows[p];
  const int y0 = rows.x, ny = rows.y;
  for (int i = threadIdx.x; i < ny * N1; i += NT) {
    int y = y0 + i / N1;
    if (y >= N2) y -= N2;
    plane[y * PS + i % N1] = CT<C>::mk(0, 0);
  }
  load_tw(tw1, tw1g, N1, +1.0);
  load_tw(tw2, tw2g, N2, +1.0);
  __syncthreads();
  const double2* src = psi + (size_t)ldg * b;
  for (int k = plane_off[p] + threadIdx.x; k < plane_off[p + 1]; k += NT) {
    const int pos = plane_pos[k], x = pos % PS;
    plane[pos - x + x / A2 + A1 * (x % A2)] = from_d2<C>(src[plane_g[k]]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ny * A2; i += NT) {  // x, radix A1
    const int t = i / ny;
    int y = y0 + i - t * ny;
    if (y >= N2) y -= N2;
    C a[A1], *q = plane + y * PS + A1 * t;
    take(a, q, 1);
    Bfly<A1>::run(a, (T)1, (const C*)nullptr, 0);
    put<A1, true>(a, q, 1, tw1, t);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ny * A1; i += NT) {  // x, radix A2
    const int k1 = i / ny;
    int y = y0 + i - k1 * ny;
    if (y >= N2) y -= N2;
    C a[A2], *q = plane + y * PS + k1;
    take(a, q, A1);
    Bfly<A2>::run(a, (T)1, (const C*)nullptr, 0);
    put<A2, false>(a, q, A1, tw1, 0);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N1 * B2; i += NT) {  // y, radix B1
    const int t = i / N1, x = i % N1;
    C a[B1], *q = plane + t * PS + x;
#pragma unroll
    for (int r = 0; r < B1; ++r) {
      int l = t + B2 * r - y0;  // rows outside the range hold nothing
      if (l < 0) l += N2;
      a[r] = l < ny ? q[r * B2 * PS] : CT<C>::mk(0, 0);
    }
    Bfly<B1>::run(a, (T)1, (const C*)nullptr, 0);
    put<B1, true>(a, q, B2 * PS, tw2, t);
  }
  __syncthreads();
  C* dst = grid + ((size_t)bl * nzp + p) * (N1 * N2);
  for (int i = threadIdx.x; i < N1 * B1; i += NT) {  // y, radix B2
    const int k1 = i / N1, x = i % N1;
    C a[B2];
    take(a, plane + k1 * B2 * PS + x, PS);
    Bfly<B2>::run(a, (T)1, (const C*)nullptr, 0);
    put<B2, false>(a, dst + k1 * N1 + x, B1 * N1, tw2, 0);
  }
}

template <class C, int N1, int N2, int V>
__global__ void __launch_bounds__(plane_threads(V), kPlaneBlocks<C, V>)
    k_rtog_plane(const C* __restrict__ grid, int nzp, const int* __restrict__ plane_off,
                 const int* __restrict__ plane_g, const int* __restrict__ plane_pos, const int2* __restrict__ plane_rows,
                 double2* __restrict__ out, const double2* __restrict__ psi, int ldg, int b0,
                 const double* __restrict__ g2, const double* __restrict__ bucket, int add_kin,
                 const double2* __restrict__ tw1g, const double2* __restrict__ tw2g) {
  using T = typename CT<C>::R;
  constexpr int NT = plane_threads(V), PS = plane_stride(N1);
  constexpr int A1 = Axis2<N1, V>::R1, A2 = Axis2<N1, V>::R2, B1 = Axis2<N2, V>::R1, B2 = Axis2<N2, V>::R2;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* plane = reinterpret_cast<C*>(smraw);  // [N2][PS]
  C* tw1 = plane + N2 * PS;
  C* tw2 = tw1 + N1;
  const int p = blockIdx.x, bl = blockIdx.y, b = b0 + bl;
  const int2 rows = plane_rows[p];
  const int y0 = rows.x, ny = rows.y;
  load_tw(tw1, tw1g, N1, -1.0);
  load_tw(tw2, tw2g, N2, -1.0);
  __syncthreads();
  const C* srcp = grid + ((size_t)bl * nzp + p) * (N1 * N2);
  for (int i = threadIdx.x; i < N1 * B2; i += NT) {  // y, radix B1
    const int t = i / N1, x = i % N1;
    C a[B1];
    take(a, srcp + t * N1 + x, B2 * N1);
    Bfly<B1>::run(a, (T)-1, (const C*)nullptr, 0);
    put<B1, true>(a, plane + B1 * t * PS + x, PS, tw2, t);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N1 * B1; i += NT) {  // y, radix B2
    const int k1 = i / N1, x = i % N1;
    C a[B2], *q = plane + k1 * PS + x;
    take(a, q, B1 * PS);
    Bfly<B2>::run(a, (T)-1, (const C*)nullptr, 0);
#pragma unroll
    for (int k = 0; k < B2; ++k) {
      int l = k1 + B1 * k - y0;  // rows outside the range are not read
      if (l < 0) l += N2;
      if (l < ny) q[k * B1 * PS] = a[k];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ny * A2; i += NT) {  // x, radix A1
    const int t = i / ny;
    int y = y0 + i - t * ny;
    if (y >= N2) y -= N2;
    C a[A1], *q = plane + y * PS + t;
    take(a, q, A2);
    Bfly<A1>::run(a, (T)-1, (const C*)nullptr, 0);
    put<A1, true>(a, q, A2, tw1, t);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ny * A1; i += NT) {  // x, radix A2
    const int k1 = i / ny;
    int y = y0 + i - k1 * ny;
    if (y >= N2) y -= N2;
    C a[A2], *q = plane + y * PS + A2 * k1;
    take(a, q, 1);
    Bfly<A2>::run(a, (T)-1, (const C*)nullptr, 0);
    put<A2, false>(a, q, 1, tw1, 0);
  }
  __syncthreads();
  double2* dst = out + (size_t)ldg * b;
  const double2* ps = psi + (size_t)ldg * b;
  for (int k = plane_off[p] + threadIdx.x; k < plane_off[p + 1]; k += NT) {
    const int g = plane_g[k], pos = plane_pos[k], x = pos % PS;
    double2 val = to_d2(plane[pos - x + x / A1 + A2 * (x % A1)]);
    if (add_kin) {
      const double kin = 0.5 * g2[g] + (bucket ? bucket[g] : 0.0);
      const double2 c = ps[g];
      val.x += kin * c.x;
      val.y += kin * c.y;
    }
    dst[g] = val;
  }
}

// planes of any other lengths: Stockham stages on every line
template <class C>
__global__ void __launch_bounds__(kPlaneThreads, 2)
    k_rtog_any(const C* __restrict__ grid, int nzp, const int* __restrict__ plane_off,
                 const int* __restrict__ plane_g, const int* __restrict__ plane_pos,
                 double2* __restrict__ out,
                 const double2* __restrict__ psi, int ldg, int b0, const double* __restrict__ g2,
                 const double* __restrict__ bucket, int add_kin, AxisArg a1, AxisArg a2,
                 const double2* __restrict__ tw1g, const double2* __restrict__ tw2g) {
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  const int nr1 = a1.n, nr2 = a2.n, npl = nr1 * nr2, pst = plane_stride(nr1);
  C* plane = sm;  // [nr2][pst]
  C* tw1 = sm + nr2 * pst;
  C* tw2 = tw1 + nr1;
  const int p = blockIdx.x, bl = blockIdx.y, b = b0 + bl;
  const C* srcp = grid + ((size_t)bl * nzp + p) * npl;
  for (int i = threadIdx.x; i < npl; i += blockDim.x) plane[i + i / nr1] = srcp[i];
  load_tw(tw1, tw1g, nr1, -1.0);
  load_tw(tw2, tw2g, nr2, -1.0);
  __syncthreads();
  transform(plane, a2, nr1, 1, pst, tw2, (typename CT<C>::R)-1);  // y lines
  transform(plane, a1, nr2, pst, 1, tw1, (typename CT<C>::R)-1);  // x lines
  double2* dst = out + (size_t)ldg * b;
  const double2* ps = psi + (size_t)ldg * b;
  for (int k = plane_off[p] + threadIdx.x; k < plane_off[p + 1]; k += blockDim.x) {
    int g = plane_g[k];
    double2 val = to_d2(plane[plane_pos[k]]);
    if (add_kin) {
      double kin = 0.5 * g2[g] + (bucket ? bucket[g] : 0.0);
      double2 c = ps[g];
      val.x += kin * c.x;
      val.y += kin * c.y;
    }
    dst[g] = val;
  }
}

// One pass of a 3-D transform of a full FP64 complex grid (x fastest), for
// the single real functions of the potential (PLANEWAVE$SUPFFT of
// POTENTIAL$VOFRHO): every block transforms kGridTX lines of one axis in
// shared memory.  x lines are rows (tile [line][x] at a row stride n + 1);
// y and z lines are taken as kGridTX consecutive x columns of one z plane
// (axis 1) or one y row (axis 2), loaded and stored coalesced along x.
constexpr int kGridTX = 16;
__global__ void __launch_bounds__(kPlaneThreads)
    k_grid_lines(double2* __restrict__ grid, int nr1, int nr2, int nr3, int axis, AxisArg ax,
                 const double2* __restrict__ twg, double sgn) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* tile = reinterpret_cast<double2*>(smraw);
  const int n = ax.n;
  const int TX = kGridTX;
  double2* tw = tile + (size_t)TX * (n + 1);
  load_tw(tw, twg, n, sgn);
  if (axis == 0) {
    const int nrows = nr2 * nr3, row0 = blockIdx.x * TX, nl = min(TX, nrows - row0);
    for (int i = threadIdx.x; i < nl * n; i += blockDim.x) {
      const int r = i / n, x = i % n;
      tile[r * (n + 1) + x] = grid[(size_t)(row0 + r) * nr1 + x];
    }
    __syncthreads();
    transform(tile, ax, nl, n + 1, 1, tw, sgn);
    for (int i = threadIdx.x; i < nl * n; i += blockDim.x) {
      const int r = i / n, x = i % n;
      grid[(size_t)(row0 + r) * nr1 + x] = tile[r * (n + 1) + x];
    }
    return;
  }
  // axis 1: lines along y at fixed z; axis 2: lines along z at fixed y
  const int nxb = (nr1 + TX - 1) / TX;
  const int x0 = (blockIdx.x % nxb) * TX, other = blockIdx.x / nxb;
  const size_t es = axis == 1 ? (size_t)nr1 : (size_t)nr1 * nr2;
  const size_t base = axis == 1 ? (size_t)nr1 * nr2 * other : (size_t)nr1 * other;
  const int nl = min(TX, nr1 - x0);
  for (int i = threadIdx.x; i < n * TX; i += blockDim.x) {
    const int e = i / TX, x = i % TX;
    tile[i] = x < nl ? grid[base + (size_t)e * es + x0 + x] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  transform(tile, ax, TX, 1, TX, tw, sgn);
  for (int i = threadIdx.x; i < n * TX; i += blockDim.x) {
    const int e = i / TX, x = i % TX;
    if (x < nl) grid[base + (size_t)e * es + x0 + x] = tile[i];
  }
}

AxisArg make_axis(const AxisPlan& p) {
  AxisArg a;
  a.n = p.n;
  a.nstage = p.nstage;
  for (int i = 0; i < 8; ++i) a.radix[i] = p.radix[i];
  return a;
}

bool plan_axis(int n, AxisPlan& p) {
  p.n = n;
  p.nstage = 0;
  int m = n;
  const int order[] = {8, 4, 2, 3, 5, 7, 11};
  for (int r : order) {
    while (m % r == 0 && p.nstage < 8) {
      p.radix[p.nstage++] = r;
      m /= r;
    }
  }
  // prefer a radix-8 stage over 4*2
  return m == 1;
}

}  // namespace

// z lengths with two-step kernels: those of the grids above and the other
// lengths up to 128 that the grids of larger or finer cells take
#define CUW_Z_LENGTHS(F)                                                                                     \
  F(18) F(20) F(24) F(28) F(30) F(32) F(36) F(40) F(42) F(44) F(48) F(50) F(54) F(56) F(60) F(64) F(66) F(70) F(72) \
  F(80) F(84) F(88) F(90) F(96) F(100) F(108) F(110) F(120) F(128)

// shared-memory limits of the z kernels of this grid (outside any capture)
template <class C>
static int z_setup(Handle* h) {
  const int n = h->d.nr3;
  switch (n) {
#define CUW_Z(N)                                                                  \
  case N:                                                                         \
    CUW_TRY(smem_allow((const void*)k_zcol<C, N>, z_smem<C>(N, kZX)));              \
    return smem_allow((const void*)k_zrho<C, N>, z_smem<C>(N, kRhoX)) == cudaSuccess ? CUW_OK : CUW_ERR_CUDA;
    CUW_Z_LENGTHS(CUW_Z)
#undef CUW_Z
    default: break;
  }
  CUW_TRY(smem_allow((const void*)k_zcol_v<C>, (int)(((size_t)n * kTX + n) * sizeof(C))));
  CUW_TRY(smem_allow((const void*)k_zcol_rho<C>, (int)(((size_t)n * kRhoTX + n) * sizeof(C))));
  return CUW_OK;
}

// z transforms and V(r) of nb bands of the work grid
template <class C>
static int z_vpsi(Handle* h, int nb) {
  const int nr1 = h->d.nr1, nr2 = h->d.nr2, nr3 = h->d.nr3, npl = nr1 * nr2;
  const double scale = 1.0 / ((double)nr1 * nr2 * nr3);
  Device& g = h->g;
  C* grid = reinterpret_cast<C*>(g.grid);
  // bands per block: V is read once for all of them; up to 4 while the launch
  // still has eight blocks for every SM
  const int nx = ceil_div(npl, kZX);
  const int nbb = std::max(1, std::min(4, nx * nb / (8 * h->nsm)));
  const dim3 gr(nx, ceil_div(nb, nbb));
  switch (nr3) {
#define CUW_Z(N)                                                                                                 \
  case N:                                                                                                        \
    k_zcol<C, N><<<gr, kZThreads<N>, z_smem<C>(N, kZX), h->stream>>>(grid, g.v, g.zslot, h->nzp, npl, g.tw3, scale, \
                                                                     nb, nbb);                                   \
    break;
    CUW_Z_LENGTHS(CUW_Z)
#undef CUW_Z
    default:
      k_zcol_v<C><<<dim3(nr2 * ceil_div(nr1, kTX), nb), kPlaneThreads, ((size_t)nr3 * kTX + nr3) * sizeof(C),
                    h->stream>>>(grid, g.v, g.zslot, h->nzp, nr1, nr2, make_axis(h->ax[2]), g.tw3, scale);
  }
  CUW_LAUNCH_CHECK("k_zcol");
  return CUW_OK;
}

// z transforms and density of nb bands from band b0
template <class C>
static int z_rho(Handle* h, double* rho, int b0, int nb) {
  const int nr1 = h->d.nr1, nr2 = h->d.nr2, nr3 = h->d.nr3, npl = nr1 * nr2;
  Device& g = h->g;
  const C* grid = reinterpret_cast<const C*>(g.grid);
  switch (nr3) {
#define CUW_Z(N)                                                                                                     \
  case N:                                                                                                            \
    k_zrho<C, N><<<ceil_div(npl, kRhoX), kRhoThreads<N>, z_smem<C>(N, kRhoX), h->stream>>>(                            \
        grid, g.zslot, h->nzp, npl, g.tw3, g.occ, h->d.nb, b0, nb, rho, b0 == 0);                                      \
    break;
    CUW_Z_LENGTHS(CUW_Z)
#undef CUW_Z
    default:
      if (nr3 * kRhoTX > 8 * kPlaneThreads) return h->fail(CUW_ERR_UNSUPPORTED, "density: NR3 above 128");
      k_zcol_rho<C><<<nr2 * ceil_div(nr1, kRhoTX), kPlaneThreads, ((size_t)nr3 * kRhoTX + nr3) * sizeof(C), h->stream>>>(
          grid, g.zslot, h->nzp, nr1, nr2, make_axis(h->ax[2]), g.tw3, g.occ, h->d.nb, b0, nb, rho, b0 == 0);
  }
  CUW_LAUNCH_CHECK("k_zrho");
  return CUW_OK;
}

// x and y transforms of the planes of nb bands from band b0, and back
template <class C, int N1, int N2, int V>
static int planes_gtor(Handle* h, const double2* psi, int b0, int nb, int smem) {
  Device& g = h->g;
  C* grid = reinterpret_cast<C*>(g.grid);
  const dim3 gr(h->nzp, nb);
  if constexpr (N1 > 0)
    k_gtor_plane<C, N1, N2, V><<<gr, plane_threads(V), smem, h->stream>>>(
        psi, h->ldg, b0, g.plane_off, g.plane_g, g.plane_pos, g.plane_rows, grid, h->nzp, g.tw1, g.tw2);
  else
    k_gtor_any<C><<<gr, kPlaneThreads, smem, h->stream>>>(psi, h->ldg, b0, g.plane_off, g.plane_g, g.plane_pos, grid,
                                                          h->nzp, make_axis(h->ax[0]), make_axis(h->ax[1]), g.tw1,
                                                          g.tw2);
  CUW_LAUNCH_CHECK("k_gtor_plane");
  return CUW_OK;
}
template <class C, int N1, int N2, int V>
static int planes_rtog(Handle* h, const double2* psi, double2* out, int add_kinetic, int b0, int nb, int smem) {
  Device& g = h->g;
  const C* grid = reinterpret_cast<const C*>(g.grid);
  const dim3 gr(h->nzp, nb);
  if constexpr (N1 > 0)
    k_rtog_plane<C, N1, N2, V><<<gr, plane_threads(V), smem, h->stream>>>(
        grid, h->nzp, g.plane_off, g.plane_g, g.plane_pos, g.plane_rows, out, psi, h->ldg, b0, g.g2, g.bucket,
        add_kinetic, g.tw1, g.tw2);
  else
    k_rtog_any<C><<<gr, kPlaneThreads, smem, h->stream>>>(grid, h->nzp, g.plane_off, g.plane_g, g.plane_pos, out, psi,
                                                          h->ldg, b0, g.g2, g.bucket, add_kinetic,
                                                          make_axis(h->ax[0]), make_axis(h->ax[1]), g.tw1, g.tw2);
  CUW_LAUNCH_CHECK("k_rtog_plane");
  return CUW_OK;
}
template <class C>
static int plane_smem(const Handle* h) {
  return (int)(((size_t)h->d.nr2 * plane_stride(h->d.nr1) + h->d.nr1 + h->d.nr2) * sizeof(C));
}

// out = FFT_RTOG[ V * FFT_GTOR[psi] ] (+ 1/2 G^2 psi + bucket psi when add_kinetic)
template <class C, int N1, int N2, int V>
static int fft_vpsi_t(Handle* h, const double2* psi, double2* out, bool add_kinetic) {
  const int smem = plane_smem<C>(h);
  for (int b0 = 0; b0 < h->d.nbh; b0 += h->batch) {
    const int nb = std::min(h->batch, h->d.nbh - b0);
    CUW_RET((planes_gtor<C, N1, N2, V>(h, psi, b0, nb, smem)));
    CUW_RET(z_vpsi<C>(h, nb));
    CUW_RET((planes_rtog<C, N1, N2, V>(h, psi, out, add_kinetic ? 1 : 0, b0, nb, smem)));
  }
  return CUW_OK;
}

// rho = sum over the bands of this set of f |psi(r)|^2 terms (WAVES_DENSITY
// for TINV at Gamma), batch by batch through the work grid
template <class C, int N1, int N2, int V>
static int fft_density_t(Handle* h, const double2* psi, double* rho) {
  const int smem = plane_smem<C>(h);
  for (int b0 = 0; b0 < h->d.nbh; b0 += h->batch) {
    const int nb = std::min(h->batch, h->d.nbh - b0);
    CUW_RET((planes_gtor<C, N1, N2, V>(h, psi, b0, nb, smem)));
    CUW_RET(z_rho<C>(h, rho, b0, nb));
  }
  return CUW_OK;
}

// kernels of work-grid type C and xy lengths N1, N2 (0: any lengths):
// shared-memory limits and the launchers
template <class C, int N1, int N2, int V>
static int fft_select_v(Handle* h) {
  const int smem = plane_smem<C>(h);
  if constexpr (N1 > 0) {
    CUW_TRY(smem_allow((const void*)k_gtor_plane<C, N1, N2, V>, smem));
    CUW_TRY(smem_allow((const void*)k_rtog_plane<C, N1, N2, V>, smem));
  } else {
    CUW_TRY(smem_allow((const void*)k_gtor_any<C>, smem));
    CUW_TRY(smem_allow((const void*)k_rtog_any<C>, smem));
  }
  CUW_RET(z_setup<C>(h));
  h->fft_run = &fft_vpsi_t<C, N1, N2, V>;
  h->fft_rho = &fft_density_t<C, N1, N2, V>;
  return CUW_OK;
}
// the plan variant h->fft_variant of a grid with compiled lengths (variant 0
// for the kernels with run-time lengths)
template <class C, int N1, int N2>
static int fft_select(Handle* h) {
  if constexpr (N1 > 0) {
    switch (h->fft_variant) {
      case 1: return fft_select_v<C, N1, N2, 1>(h);
      case 2: return fft_select_v<C, N1, N2, 2>(h);
      case 3:
        if constexpr (N1 == 64 && N2 == 64) return fft_select_v<C, N1, N2, 3>(h);
        break;
      default: break;
    }
  }
  return fft_select_v<C, N1, N2, 0>(h);
}

// Kernels of the handle's grid and plan variant: grids of the table get xy planes
// compiled for their lengths (two register steps an axis); any other grid takes
// the Stockham stages of run-time lengths.  The z kernels go by NR3 alone.
static int fft_choose(Handle* h) {
  const int nr1 = h->d.nr1, nr2 = h->d.nr2, nr3 = h->d.nr3;
  int rc = CUW_OK;
  bool found = false;
#define CUW_FFT_GRID(A, B, Z)                                                                        \
  if (!found && nr1 == A && nr2 == B && nr3 == Z) {                                                  \
    found = true;                                                                                    \
    rc = h->mixed() ? fft_select<float2, A, B>(h) : fft_select<double2, A, B>(h); \
  }
  CUW_FFT_GRIDS
#undef CUW_FFT_GRID
  h->fft_compiled = found;
  if (!found) {
    h->fft_variant = 0;
    rc = h->mixed() ? fft_select<float2, 0, 0>(h) : fft_select<double2, 0, 0>(h);
  }
  return rc;
}

int fft_setup(Handle* h, const int* igvec) {
  const int nr1 = h->d.nr1, nr2 = h->d.nr2, nr3 = h->d.nr3, ngl = h->d.ngl;
  for (int a = 0; a < 3; ++a) {
    int n = a == 0 ? nr1 : (a == 1 ? nr2 : nr3);
    if (!plan_axis(n, h->ax[a]))
      return h->fail(CUW_ERR_UNSUPPORTED, "FFT length " + std::to_string(n) + " has a prime factor above 11");
  }
  const size_t npl = (size_t)nr1 * nr2;
  // work-grid element: FP64 complex, or FP32 complex on the mixed path
  const size_t es = h->mixed() ? sizeof(float2) : sizeof(double2);
  const size_t plane_elems = (size_t)nr2 * plane_stride(nr1) + nr1 + nr2;
  if (plane_elems * es > (size_t)(220 * 1024) || ((size_t)nr3 * kTX + nr3) * es > 14000 * sizeof(double2))
    return h->fail(CUW_ERR_UNSUPPORTED, "FFT plane too large for shared memory");
  // occupied planes and the per-plane G lists
  std::vector<int> cnt(nr3, 0);
  std::vector<int> iz_of(ngl), pos_of(ngl);
  for (int g = 0; g < ngl; ++g) {
    int i1 = ((igvec[3 * g] % nr1) + nr1) % nr1;
    int i2 = ((igvec[3 * g + 1] % nr2) + nr2) % nr2;
    int i3 = ((igvec[3 * g + 2] % nr3) + nr3) % nr3;
    iz_of[g] = i3;
    pos_of[g] = i1 + plane_stride(nr1) * i2;  // padded shared-memory plane
    cnt[i3]++;
  }
  std::vector<int> zslot(nr3, -1), plane_iz, off(1, 0);
  for (int z = 0; z < nr3; ++z)
    if (cnt[z]) {
      zslot[z] = (int)plane_iz.size();
      plane_iz.push_back(z);
      off.push_back(off.back() + cnt[z]);
    }
  const int nzp = (int)plane_iz.size();
  // signed row range of every occupied plane: rows (y0 + l) mod NR2, l < ny
  std::vector<int> ylo(nzp, 1 << 30), yhi(nzp, -(1 << 30));
  for (int gg = 0; gg < ngl; ++gg) {
    const int s = zslot[iz_of[gg]];
    int y = ((igvec[3 * gg + 1] % nr2) + nr2) % nr2;
    if (y > nr2 / 2) y -= nr2;
    ylo[s] = std::min(ylo[s], y);
    yhi[s] = std::max(yhi[s], y);
  }
  std::vector<int2> rows(nzp);
  for (int s = 0; s < nzp; ++s) {
    int ny = yhi[s] - ylo[s] + 1;
    int y0 = (ylo[s] + nr2) % nr2;
    if (ny > nr2) { ny = nr2; y0 = 0; }
    rows[s] = make_int2(y0, ny);
  }
  std::vector<int> fill(off.begin(), off.end() - 1), pg(ngl), pp(ngl);
  for (int g = 0; g < ngl; ++g) {
    int s = zslot[iz_of[g]];
    int k = fill[s]++;
    pg[k] = g;
    pp[k] = pos_of[g];
  }
  h->nzp = nzp;
  // band batch: keep the work grid near 48 MB so that it stays in L2
  const size_t per_band = (size_t)nzp * npl * es;
  int batch = (int)std::max<size_t>(1, (48u << 20) / per_band);
  batch = std::min(batch, h->d.nbh);
  h->batch = batch;
  Device& g = h->g;
  drop(g.plane_off, g.plane_g, g.plane_pos, g.zslot, g.plane_iz, g.plane_rows, g.grid, g.tw1, g.tw2, g.tw3);
  CUW_TRY(cudaMalloc(&g.plane_off, sizeof(int) * (nzp + 1)));
  CUW_TRY(cudaMalloc(&g.plane_g, sizeof(int) * ngl));
  CUW_TRY(cudaMalloc(&g.plane_pos, sizeof(int) * ngl));
  CUW_TRY(cudaMalloc(&g.zslot, sizeof(int) * nr3));
  CUW_TRY(cudaMalloc(&g.plane_iz, sizeof(int) * nzp));
  CUW_TRY(cudaMalloc(&g.plane_rows, sizeof(int2) * nzp));
  CUW_TRY(cudaMalloc(&g.grid, per_band * batch));
  h->grid_bands = batch;
  CUW_TRY(cudaMemcpy(g.plane_off, off.data(), sizeof(int) * (nzp + 1), cudaMemcpyHostToDevice));
  CUW_TRY(cudaMemcpy(g.plane_g, pg.data(), sizeof(int) * ngl, cudaMemcpyHostToDevice));
  CUW_TRY(cudaMemcpy(g.plane_pos, pp.data(), sizeof(int) * ngl, cudaMemcpyHostToDevice));
  CUW_TRY(cudaMemcpy(g.zslot, zslot.data(), sizeof(int) * nr3, cudaMemcpyHostToDevice));
  CUW_TRY(cudaMemcpy(g.plane_iz, plane_iz.data(), sizeof(int) * nzp, cudaMemcpyHostToDevice));
  CUW_TRY(cudaMemcpy(g.plane_rows, rows.data(), sizeof(int2) * nzp, cudaMemcpyHostToDevice));
  double2** tws[3] = {&g.tw1, &g.tw2, &g.tw3};
  for (int a = 0; a < 3; ++a) {
    int n = h->ax[a].n;
    std::vector<double2> t(n);
    for (int k = 0; k < n; ++k) {
      double ang = 2.0 * M_PI * (double)k / (double)n;
      t[k] = make_double2(std::cos(ang), std::sin(ang));
    }
    CUW_TRY(cudaMalloc(tws[a], sizeof(double2) * n));
    CUW_TRY(cudaMemcpy(*tws[a], t.data(), sizeof(double2) * n, cudaMemcpyHostToDevice));
  }
  return fft_choose(h);
}

// 3-D transform of a full FP64 complex grid (x fastest), in place and
// unscaled: dir = +1 is G->R (exp(+iGr)), dir = -1 is R->G (exp(-iGr)); the
// caller applies the 1/N of the reference's R->G transform.
int grid_fft(Handle* h, double2* grid, int dir) {
  const int n[3] = {h->d.nr1, h->d.nr2, h->d.nr3};
  const double2* tw[3] = {h->g.tw1, h->g.tw2, h->g.tw3};
  for (int a = 0; a < 3; ++a) {
    const AxisArg ax = make_axis(h->ax[a]);
    const int smem = (int)(((size_t)kGridTX * (n[a] + 1) + n[a]) * sizeof(double2));
    CUW_TRY(smem_allow((const void*)k_grid_lines, smem));
    const int nxb = (n[0] + kGridTX - 1) / kGridTX;
    const int blocks = a == 0 ? ceil_div(n[1] * n[2], kGridTX) : nxb * (a == 1 ? n[2] : n[1]);
    k_grid_lines<<<blocks, kPlaneThreads, smem, h->stream>>>(grid, n[0], n[1], n[2], a, ax, tw[a], (double)dir);
    CUW_LAUNCH_CHECK("k_grid_lines");
  }
  return CUW_OK;
}

// FP64 transforms, or FP32 transforms and V(r) product on the mixed path, with
// the kernels chosen by fft_setup for the grid
int fft_vpsi(Handle* h, const double2* psi, double2* out, bool add_kinetic) {
  if (!h->fft_run) return h->fail(CUW_ERR_STATE, "FFT not set up");
  return h->fft_run(h, psi, out, add_kinetic);
}

int fft_density(Handle* h, const double2* psi, double* rho) {
  if (!h->fft_rho) return h->fail(CUW_ERR_STATE, "FFT not set up");
  return h->fft_rho(h, psi, rho);
}

// plan variant v (0 .. fft_variants()-1) of the compiled kernels; grids with
// run-time lengths have variant 0 only
// variant 3 exists for 64^3 grids only
static bool z64_grid(const Handle* h) { return h->d.nr1 == 64 && h->d.nr2 == 64 && h->d.nr3 == 64; }
int fft_variants(const Handle* h) { return !h->fft_compiled ? 1 : (z64_grid(h) ? kFftVariants : kFftVariants - 1); }
int fft_set_variant(Handle* h, int v) {
  if (!h->fft_run) return h->fail(CUW_ERR_STATE, "FFT not set up");
  if (v < 0 || v >= fft_variants(h)) return CUW_ERR_UNSUPPORTED;
  h->fft_variant = v;
  h->touch();
  return fft_choose(h);
}

}  // namespace cuw
