// Sliced fixed-point products on the 8-bit integer tensor cores (tcgen05
// kind::i8, sm_100a).
//
// An operand row is scaled by a power of two to an integer of 8 S - 2 bits and
// cut into S balanced base-256 digits (signed bytes, most significant first):
//   x = scale * sum_i d_i 256^(S-1-i)
// A product of two rows is then a sum of exact integer products of digit rows,
//   sum_k a_k b_k = sa sb sum_q 256^(2S-2-q) acc_q,  acc_q = sum_(i+j=q) sum_k d_i e_j
// of which the S diagonals q < S are formed (the rest lies below the last digit
// kept).  The tensor core adds in 32-bit integers, exactly, so a whole K range
// accumulates in tensor memory and is read once; what remains are the rounding
// of the operands to 8 S - 2 bits of their row's largest element and the dropped
// diagonals, about 2^(2-8S) of the rows' maxima each.  |acc_q| < S K 2^14 must
// stay below 2^31.
//
// Digit tiles: rows R (128 of the A operand, NB of the B operand) by 32 K per
// chunk and digit, in the K-major core-matrix layout without swizzle: byte
//   (k / 16) * (R * 16) + row * 16 + k % 16
// digits of a chunk one after another, chunks of a tile one after another, so
// that a chunk arrives by one bulk copy per operand.
#pragma once

#include "tc_sm100.cuh"

namespace cuw {
namespace i8 {

using tc::smem_u32;

constexpr long long kWaitCycles = 1ll << 31;  // about one second at 2 GHz

// instruction descriptor of kind::i8: D 32-bit integer, A and B signed bytes, both K-major
__host__ __device__ constexpr uint32_t idesc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// D[tmem] (+)= A[smem] * B[smem]^T, K = 32, issued by one thread
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// S digits, 128 x NB tile, NST stages of one chunk (32 K)
template <int S, int NB, int NST>
struct Cfg {
  static_assert(S * NB <= 512, "TMEM columns");
  static_assert(NB % 16 == 0 && NB <= 256, "N of kind::i8");
  static constexpr int kS = S, kNB = NB, kNst = NST;
  static constexpr int kABytes = S * 128 * 32, kBBytes = S * NB * 32;
  static constexpr int kStage = kABytes + kBBytes;
  static constexpr size_t kSmem = (size_t)NST * kStage + 1024 + 256;
  static constexpr int kThreads = 192;  // MMA, copies, four epilogue warps
};

// One 128 x NB tile over nchunk chunks; a(c) / b(c): the digit tiles of chunk c.
// epi(row, j, v): the four epilogue warps receive, for tile row `row`, the
// values of columns 16 j .. 16 j + 15 in units of 256^(S-1) sa sb, in FP64.
// done() runs in every epilogue thread afterwards.  Every wait is bounded; one
// that runs out sets *err and every role leaves.
template <class C, class FA, class FB, class Epi>
__device__ __forceinline__ void run(int nchunk, FA a, FB b, Epi& epi, int* err) {
  extern __shared__ __align__(1024) unsigned char i8_smem[];
  unsigned char* st = i8_smem + ((1024u - (smem_u32(i8_smem) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(st + (size_t)C::kNst * C::kStage);
  uint64_t* empty = full + C::kNst;
  uint64_t* done = empty + C::kNst;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < C::kNst; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], 1);
    }
    tc::mbar_init(done, 1);
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  auto raise = [&]() {
    *abort_flag = 1;
    atomicExch(err, 1);
  };
  if (warp == 0) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_i8(128, C::kNB);
      const uint64_t da0 = tc::sdesc(0, 128 * 16, 128), db0 = tc::sdesc(0, C::kNB * 16, 128);
      const uint32_t s0 = smem_u32(st) >> 4;
      bool ok = true;
      for (int c = 0; c < nchunk; ++c) {
        const int s = c % C::kNst;
        ok = tc::mbar_wait(&full[s], (c / C::kNst) & 1, kWaitCycles) && !*abort_flag;
        if (!ok) {
          raise();
          break;
        }
        tc::fence_after_sync();
        const uint32_t ua = s0 + (uint32_t)(s * (C::kStage >> 4)), ub = ua + (uint32_t)(C::kABytes >> 4);
#pragma unroll
        for (int q = 0; q < C::kS; ++q)
#pragma unroll
          for (int i = 0; i <= q; ++i)
            mma_i8(tmem + (uint32_t)(q * C::kNB), da0 | (uint64_t)(ua + i * (128 * 32 >> 4)),
                   db0 | (uint64_t)(ub + (q - i) * (C::kNB * 32 >> 4)), idesc, (c | i) ? 1u : 0u);
        tc::mma_commit(&empty[s]);
      }
      // the MMAs issued have finished before tensor memory is read or released
      tc::mma_commit(done);
      tc::mbar_wait(done, 0, kWaitCycles);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int issued = 0;
      for (int c = 0; c < nchunk; ++c) {
        const int s = c % C::kNst;
        bool ok = c < C::kNst || tc::mbar_wait(&empty[s], ((c / C::kNst) - 1) & 1, kWaitCycles);
        ok = ok && !*abort_flag;
        if (!ok) {
          raise();
          break;
        }
        tc::mbar_arrive_expect_tx(&full[s], C::kStage);
        tc::bulk_g2s(st + (size_t)s * C::kStage, a(c), C::kABytes, &full[s]);
        tc::bulk_g2s(st + (size_t)s * C::kStage + C::kABytes, b(c), C::kBBytes, &full[s]);
        issued = c + 1;
      }
      if (*abort_flag)  // copies nobody consumed complete before the CTA ends
        for (int c = max(0, issued - C::kNst); c < issued; ++c)
          tc::mbar_wait(&full[c % C::kNst], (c / C::kNst) & 1, kWaitCycles);
    }
  } else {
    const int q = warp & 3, row = 32 * q + lane;
    bool ok = tc::mbar_wait(done, 0, kWaitCycles);
    ok = __all_sync(0xffffffffu, ok && !*abort_flag);
    if (ok) {
      tc::fence_after_sync();
      const uint32_t base = tmem + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
      for (int j = 0; j < C::kNB / 16; ++j) {
        double v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.0;
        // least significant diagonal first
#pragma unroll
        for (int d = C::kS - 1; d >= 0; --d) {
          uint32_t r[16];
          tc::tmem_ld16(base + (uint32_t)(d * C::kNB + 16 * j), r);
          tc::tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = fma(v[i], 1.0 / 256.0, (double)(int)r[i]);
        }
        epi(row, j, v);
      }
    } else if (lane == 0) {
      raise();
    }
    tc::fence_before_sync();
  }
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) {
    __syncwarp();
    tc::tmem_dealloc(tmem, 512);
  }
}

}  // namespace i8
}  // namespace cuw
