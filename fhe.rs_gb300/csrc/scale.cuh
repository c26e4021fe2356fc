// Pieces shared by the RNS scaling kernels (scale.cu, scale_hat.cu): exact
// multi-word sums, the tensor-core operand bytes and the forward stages the
// kernels apply to their outputs.
#pragma once

#include <cuda_fp16.h>

#include "lib.hpp"
#include "ntt.cuh"
#include "tc.cuh"

namespace fheg {
namespace {

__device__ __forceinline__ uint64_t join(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

// Low 128 bits of (w >> s) for an nw-word little-endian value (32-bit words).
__device__ __forceinline__ void shr_words(const uint32_t* w, int nw, uint32_t s, uint64_t* lo, uint64_t* hi) {
  uint32_t o[4];
  const uint32_t ws = s >> 5, bs = s & 31;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t idx = ws + k;
    uint32_t a = 0, b = 0;
#pragma unroll
    for (int m = 0; m < 8; m++) {
      if (m < nw && (uint32_t)m == idx) a = w[m];
      if (m < nw && (uint32_t)m == idx + 1) b = w[m];
    }
    o[k] = bs ? ((a >> bs) | (b << (32 - bs))) : a;
  }
  *lo = join(o[0], o[1]);
  *hi = join(o[2], o[3]);
}

// 256-bit a += b, a -= b (32-bit words).
__device__ __forceinline__ void add256w(uint32_t* a, const uint32_t* b) {
  asm("add.cc.u32 %0, %0, %8;\n\taddc.cc.u32 %1, %1, %9;\n\taddc.cc.u32 %2, %2, %10;\n\taddc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\taddc.cc.u32 %5, %5, %13;\n\taddc.cc.u32 %6, %6, %14;\n\taddc.u32 %7, %7, %15;"
      : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7])
      : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

__device__ __forceinline__ void sub256w(uint32_t* a, const uint32_t* b) {
  asm("sub.cc.u32 %0, %0, %8;\n\tsubc.cc.u32 %1, %1, %9;\n\tsubc.cc.u32 %2, %2, %10;\n\tsubc.cc.u32 %3, %3, %11;\n\t"
      "subc.cc.u32 %4, %4, %12;\n\tsubc.cc.u32 %5, %5, %13;\n\tsubc.cc.u32 %6, %6, %14;\n\tsubc.u32 %7, %7, %15;"
      : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7])
      : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

// Full 128 x 128 -> 256-bit product (32-bit words).
__device__ __forceinline__ void mul128x128w(uint32_t* r, uint64_t alo, uint64_t ahi, uint64_t blo, uint64_t bhi) {
#pragma unroll
  for (int k = 0; k < 8; k++) r[k] = 0;
  uint32_t t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  mac256(t, alo, blo, bhi);  // alo * b at word 0
  uint32_t hi6[6] = {0, 0, 0, 0, 0, 0};
  mac192(hi6, ahi, blo, bhi);  // ahi * b at word 2 (< 2^192)
  uint32_t u[8] = {0, 0, hi6[0], hi6[1], hi6[2], hi6[3], hi6[4], hi6[5]};
  add256w(t, u);
#pragma unroll
  for (int k = 0; k < 8; k++) r[k] = t[k];
}

// Forward stages of the kernel's epilogue (ForwardTop for one launch; primes
// null: none).
struct FwdEpilogue {
  const DevPrime* primes;
  uint32_t period, take;
  const DevPrime* digit_primes;
  uint32_t digit_limbs, digit_raw;
  PolyRef digits;
};

// Two bytes of w (prmt selector sel) as the half2 (b0, b1): 0x64bb is the
// FP16 value 1024 + b, less 1024.
__device__ __forceinline__ uint32_t tc_bytes_half2(uint32_t w, uint32_t sel) {
  uint32_t t;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(t) : "r"(w), "r"(0x64646464u), "r"(sel));
  __half2 h = *reinterpret_cast<__half2*>(&t);
  h = __hsub2(h, __halves2half2(__ushort_as_half(0x6400), __ushort_as_half(0x6400)));
  return *reinterpret_cast<uint32_t*>(&h);
}

// The dynamic shared memory of a TC launch: the stage buffer, overlaid by A
// (128 x KP FP16) once the residues are in registers, then B.
__device__ __forceinline__ uint8_t* tc_dyn_smem() {
  extern __shared__ __align__(128) uint8_t tc_dyn[];
  return tc_dyn;
}

constexpr uint32_t kTcWaitTries = 1u << 20;

// 228 KB of shared memory per SM over its 512 tensor-memory columns.
constexpr size_t kTcSmemPerColumn = 233472 / 512;

// The outputs of a CTA's 128 >> TOP groups (staged[(o * 2^TOP + t) * G + g])
// through the first TOP forward stages: over their own limbs (fwd_here), or, as
// digits, in every key modulus (FwdEpilogue).
template <int TOP, bool FOLD>
__device__ __forceinline__ void scale_epilogue(const uint64_t* staged, bool fwd_here, uint32_t out_len, uint32_t poly,
                                               uint32_t b0, uint32_t logb, const PolyRef& out, const FwdEpilogue& fe) {
  constexpr int G = 128 >> TOP;
  if (fwd_here) {
    for (uint32_t item = threadIdx.x; item < out_len * G; item += 128) {
      const uint32_t o = item / G, g2 = item % G;
      uint64_t x[1 << TOP];
#pragma unroll
      for (int u = 0; u < (1 << TOP); u++) x[u] = staged[(o * (1 << TOP) + u) * G + g2];
      fwd_top_stages<TOP, FOLD>(x, fe.primes[o]);
      uint64_t* row = out.at(poly, o) + b0 + g2;
#pragma unroll
      for (int u = 0; u < (1 << TOP); u++) row[(uint64_t)u << logb] = x[u];
    }
  } else {
    // Digit d (output limb d) in key limb j: key_switching_key.rs:227-235
    // with rq/mod.rs:518-540, the first forward stages of its transform. G
    // threads take every second digit of one key limb, whose constants and
    // twiddles they load once.
    const uint32_t pbase = (poly / fe.period) * out_len, g2 = threadIdx.x % G;
    for (uint32_t u = threadIdx.x / G; u < 2 * fe.digit_limbs; u += 128 / G) {
      const uint32_t j = u >> 1;
      const DevPrime kp = fe.digit_primes[j];
      for (uint32_t d = u & 1; d < out_len; d += 2) {
        uint64_t x[1 << TOP];
#pragma unroll
        for (int e = 0; e < (1 << TOP); e++) {
          const uint64_t v = staged[(d * (1 << TOP) + e) * G + g2];
          if constexpr (FOLD) x[e] = (uint64_t)fold_lift(v, kp);
          else x[e] = fe.digit_raw ? v : reduce64_lazy(v, kp);
        }
        fwd_top_stages<TOP, FOLD>(x, kp);
        uint64_t* row = fe.digits.at(pbase + d, j) + b0 + g2;
#pragma unroll
        for (int e = 0; e < (1 << TOP); e++) row[(uint64_t)e << logb] = x[e];
      }
    }
  }
}

}  // namespace
}  // namespace fheg
