// RNS scaling between primes just below a power of two (Context::fold), on the
// tensor cores.
//
// With m_k the source moduli, M their product and hat_k = M / m_k, the residues
// r_k enter as z_k = r_k hat_k^-1 mod m_k (where an inverse NTT ends in this
// kernel, as part of the constant it scales by), and
//   x = sum_k z_k hat_k - v M,   v = round(sum_k z_k / m_k),
// is the representative of the residues in [-M/2, M/2) that rns/scaler.rs
// works with (its v counts multiples of M in sum_k r_k garner_k, a number of 66
// bits that takes 192-bit sums; this one is at most F). With the factor num / den
//   hat_k num / den = Phi_k + phi_k,   M num / den = Gamma + gamma
// (integer and fraction), the scaled value is
//   round(x num / den) = sum_k z_k Phi_k - v (Gamma + 1) + w,
//   w = round(sum_k z_k phi_k + v (1 - gamma)) >= 0.
// phi_k is zero for the sources that divide out of den, so the t/Q scale-down of
// a multiplication sums only its L base moduli for w. Rounding is the reference's
// except where a fraction lies within its margin of 1/2: v is computed to about
// F 2^-31 (62-bit moduli) and w to 2^-47, and the rare coefficient that close to
// a boundary takes the reference's own sums (hat_exact).
//
// The sums over z_k Phi_k modulo each target are the byte products of scale.cu's
// tensor-core form: with the bytes a_kb of z_k and x_kbc of Phi_k 2^(8b) mod q_j,
// D_c = sum_(k,b) a_kb x_kbc, exact in FP32 (below 2^23 for up to 16 sources,
// below 2^24 for up to 32). One MMA pass of N = 8 columns an output, which runs
// while the threads form w. For up to 16 sources one more column of A and B
// adds 2^23 to every D_c, so that the FP32 bits are an integer plus a constant.
//
// Stage times, events, against the CUDA-core extension and the two- and
// four-pass tensor-core scale-down (scale.cu) in the same multiplication: 64
// pairs at N = 2^14, L = 6: extension 0.326 -> 0.216 ms, scale-down 0.490 -> 0.330;
// 16 pairs at N = 2^15, L = 12: 0.379 -> 0.283 and 0.764 -> 0.510 (both with the
// transforms' stages on either side in fold arithmetic as well). Bound by
// latency at 24-28 warps an SM beside the multiplier (59-61% busy, the tensor
// pipe 5-7%).

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "scale.cuh"

namespace fheg {

// Everything the reference's own sums need (device memory).
struct HatExact {
  uint32_t from_len, is_one, shift, tg_sign, to_sign;
  uint64_t tg_lo, tg_hi;
  const DevPrime* from;
  const DevPrime* to;
  const uint64_t *hat, *gar_lo, *gar_hi, *om_lo, *om_hi;  // [F]; hat_k mod m_k
  const uint64_t* omega;                                  // [T][F]
  const uint64_t *gneg, *gneg_hi;                         // [T]
};

namespace {

// Count of waits of this kernel that ran out (hat_wait_failures).
__device__ uint32_t g_hat_wait_failures;

// Constants of one launch, read from the parameter bank. The sources with a
// nonzero phi_k come first (k < frac <= MS).
template <int MAXF, int MAXT, int MS>
struct HatLaunch {
  uint32_t from_len, out_len, frac;
  uint32_t cols, b_offset, b_rows;
  uint32_t chunk_words;           // FP16 words from a chunk's matrix to the next one's
  uint32_t inv[MAXF], zsh[MAXF];  // 2^(k + 27) / m_k and k - 31 for m_k just below 2^k
  uint64_t v_margin, w_margin;
  uint32_t th1[MS], th2[MS], th3[MS], th4[MS];  // phi_k as 28-bit digits
  uint32_t g1, g2;                     // 1 - gamma, two of them
  uint64_t gneg[MAXT];                 // -(Gamma + 1) mod q_j
  uint64_t p[MAXT];
  uint32_t c[MAXT], sh[MAXT];
};

// The outputs start .. start + n of one coefficient by the reference's sums
// (rns/scaler.rs:249-352) from the z_k: any rounding.
__device__ __noinline__ void hat_exact(const HatExact* e, const uint64_t* z, uint32_t start, uint32_t n, uint64_t* y) {
  const uint32_t F = e->from_len;
  uint64_t r[32];
#pragma unroll 1
  for (uint32_t k = 0; k < F; k++) r[k] = mul_mod(z[k], e->hat[k], e->from[k]);
  uint32_t g[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
  for (uint32_t k = 0; k < F; k++) mac192(g, r[k], e->gar_lo[k], e->gar_hi[k]);
  uint64_t vlo, vhi;
  shr_words(g, 6, e->shift - 1, &vlo, &vhi);
  const uint64_t odd = vlo & 1;
  vlo = (vlo >> 1) | (vhi << 63);
  vhi >>= 1;
  vlo += odd;
  vhi += (vlo < odd);
  bool w_sign = false;
  uint64_t wlo = 0, whi = 0;
  if (!e->is_one) {
    uint32_t pos[8] = {0, 0, 0, 0, 0, 0, 0, 0}, neg[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
    for (uint32_t k = 0; k < F; k++) {
      if ((e->to_sign >> k) & 1) mac256(neg, r[k], e->om_lo[k], e->om_hi[k]);
      else mac256(pos, r[k], e->om_lo[k], e->om_hi[k]);
    }
    sub256w(pos, neg);
    uint32_t vt[8];
    mul128x128w(vt, vlo, vhi, e->tg_lo, e->tg_hi);
    if (e->tg_sign) add256w(pos, vt);
    else sub256w(pos, vt);
    w_sign = (pos[7] >> 31) != 0;
    if (w_sign) {
#pragma unroll
      for (int k = 0; k < 8; k++) pos[k] = ~pos[k];
    }
    shr_words(pos, 8, 126, &wlo, &whi);
    const uint64_t up = w_sign ? 1 : wlo & 1;
    if (w_sign) {
      wlo += 1;
      whi += (wlo == 0);
      wlo = (wlo >> 1) | (whi << 63);
      whi >>= 1;
    } else {
      wlo = (wlo >> 1) | (whi << 63);
      whi >>= 1;
      wlo += up;
      whi += (wlo < up);
    }
  }
  const uint64_t v_low = vlo & ((1ull << 62) - 1), v_top = (vlo >> 62) | (vhi << 2);
#pragma unroll 1
  for (uint32_t o = 0; o < n; o++) {
    const uint32_t j = start + o;
    const DevPrime pr = e->to[j];
    uint64_t lo = 0, hi = 0;
    if (!e->is_one) {
      const uint64_t wj = reduce128_lazy(whi, wlo, pr);
      lo = w_sign ? pr.p2 - wj : wj;
    }
    mac128(hi, lo, v_low, e->gneg[j]);
    mac128(hi, lo, v_top, e->gneg_hi[j]);
#pragma unroll 1
    for (uint32_t k = 0; k < F; k++) {
      mac128(hi, lo, r[k], e->omega[j * F + k]);
      if ((k % 14) == 13) {  // keep the exact sum below 2^128
        lo = reduce128(hi, lo, pr);
        hi = 0;
      }
    }
    y[o] = reduce128(hi, lo, pr);
  }
}

// A column sum as an integer: the FP32 bits less those of 2^23 (BIASED), or by
// conversion.
template <bool BIASED>
__device__ __forceinline__ uint32_t hat_int(uint32_t f) {
  if constexpr (BIASED) return f - 0x4B000000u;
  else return __float2uint_rz(__uint_as_float(f));
}

// sum_c 2^(8c) D_c of an output's eight columns, below 2^81.
template <bool BIASED>
__device__ __forceinline__ void hat_sum(const uint32_t* d, uint64_t* lo, uint32_t* hi) {
  uint64_t h[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    // D + D' 2^8 < 2^32. (The constant of a biased D' leaves by the shift.)
    uint32_t e0 = hat_int<BIASED>(d[4 * q]), e1 = hat_int<BIASED>(d[4 * q + 2]);
    e0 += (BIASED ? d[4 * q + 1] : hat_int<BIASED>(d[4 * q + 1])) << 8;
    e1 += (BIASED ? d[4 * q + 3] : hat_int<BIASED>(d[4 * q + 3])) << 8;
    h[q] = (uint64_t)e0 + ((uint64_t)e1 << 16);
  }
  *lo = h[0] + (h[1] << 32);
  *hi = (uint32_t)(h[1] >> 32) + (*lo < h[0] ? 1u : 0u);
}

// Operand shapes. Above 12 sources they go through A in two chunks, the second
// accumulating onto the first: half of A and B leaves shared memory for more
// CTAs (13 sources into 6 outputs: 7 on an SM by registers instead of 5, and 25
// into 12: 4 instead of 2).
template <int MAXF>
struct HatShape {
  static constexpr bool kBiased = MAXF <= 16;
  static constexpr int kChunks = MAXF > 12 ? 2 : 1;
  static constexpr int kPer = (MAXF + kChunks - 1) / kChunks;  // sources of a chunk
  static constexpr uint32_t kKp = (8 * (kPer + (kBiased ? 1 : 0)) + 15) / 16 * 16;
};

// Row threadIdx.x of A for chunk CH: the bytes of its z_k, one 16-byte
// core-matrix row each, and in chunk 0 the column of 2^11 (by 2^12 in B).
template <int MAXF, int CH>
__device__ __forceinline__ void hat_operand(uint8_t* sa, const uint64_t* z) {
  using K = HatShape<MAXF>;
#pragma unroll
  for (uint32_t l = 0; l < K::kKp / 8; l++) {
    uint4 v = make_uint4(0, 0, 0, 0);
    const int k = CH * K::kPer + (int)l;
    if ((int)l < K::kPer && k < MAXF) {
      const uint64_t x = z[k < MAXF ? k : 0];
      const uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32);
      v = make_uint4(tc_bytes_half2(lo, 0x4140), tc_bytes_half2(lo, 0x4342), tc_bytes_half2(hi, 0x4140),
                     tc_bytes_half2(hi, 0x4342));
    } else if (K::kBiased && CH == 0 && (int)l == K::kPer) {
      v.x = 0x6800;
    }
    *reinterpret_cast<uint4*>(sa + tc_core_off(threadIdx.x, 8 * l, K::kKp)) = v;
  }
}

// Thread 0: the MMAs of a chunk once phase `phase` of bar_b has its operand B.
// A copy that does not land in time is counted and the MMAs are skipped (the
// outputs are then not valid); no thread waits longer than its own bounded
// wait.
template <uint32_t KP>
__device__ __forceinline__ void hat_mma(uint32_t bar_b, uint32_t phase, uint32_t bar_mma, uint32_t tmem, uint32_t a_addr,
                                        uint32_t b_addr, uint32_t rows, uint32_t accumulate) {
  if (mbar_wait(bar_b, phase, kTcWaitTries)) {
    const uint32_t idesc = tc_idesc_f16_f32(128, rows);
#pragma unroll
    for (uint32_t kk = 0; kk < KP / 16; kk++)
      tc_mma_f16(tmem, tc_smem_desc(a_addr + kk * 256, 16 * KP), tc_smem_desc(b_addr + kk * 256, 16 * KP), idesc,
                 kk > 0 ? 1u : accumulate);
    tc_commit(bar_mma);
  } else {
    atomicAdd(&g_hat_wait_failures, 1u);
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_mma) : "memory");
    mbar_wait(bar_b, phase, kTcWaitTries);
  }
}

// One thread per coefficient, 128 per CTA. TOP > 0: as in scale.cu, `in` holds
// the block pass of a two-pass inverse NTT whose last TOP stages run here (a
// CTA owns 128 >> TOP groups), and the outputs may leave through the first
// TOP stages of a forward one. zc: per source the digits (fold_mul) of
// hat_k^-1, N^-1 hat_k^-1 and zetas_inv[N - 2] N^-1 hat_k^-1.
template <int MAXF, int MAXT, int MS, int TOP, bool ONE>
__global__ void __launch_bounds__(128) k_rns_hat(const __grid_constant__ HatLaunch<MAXF, MAXT, MS> s,
                                                 uint32_t logn, PolyRef in, PolyRef out, const DevPrime* src_primes,
                                                 const int4* zc, const uint16_t* mat, const HatExact* ex,
                                                 uint32_t start, const FwdEpilogue fe) {
  constexpr int G = 128 >> TOP;
  using K = HatShape<MAXF>;
  constexpr bool BIASED = K::kBiased;
  constexpr uint32_t KP = K::kKp;
  __shared__ __align__(8) uint64_t bars[3];
  __shared__ uint32_t slot;
  uint8_t* sa = tc_dyn_smem();
  const uint32_t bar_b = smem_u32(&bars[0]), bar_mma = smem_u32(&bars[1]);  // bar_mma + 8 ch: chunk ch's
  const uint32_t a_addr = smem_u32(sa), b_addr = a_addr + s.b_offset;
  const uint32_t F = s.from_len;
  // Operand B in flight and the tensor memory allocated while the kernel
  // before ends and the sources load.
  if (threadIdx.x == 0) {
    mbar_init(bar_b, 1);
    mbar_init(bar_mma, 1);
    mbar_init(bar_mma + 8, 1);
    fence_proxy_async_smem();
    mbar_expect_tx(bar_b, s.out_len * 16 * KP);
    bulk_g2s(b_addr, mat, s.out_len * 16 * KP, bar_b);
  }
  if ((threadIdx.x >> 5) == 1) tc_alloc(smem_u32(&slot), s.cols);
  pdl_wait();

  const uint32_t poly = blockIdx.x >> (logn - 7), part = blockIdx.x & ((1u << (logn - 7)) - 1);
  uint32_t i, b0 = 0, logb = logn, t = 0, gi = 0;
  bool fwd_here = false, dig_here = false;  // uniform across the CTA
  uint64_t z[MAXF];
  if constexpr (TOP == 0) {
    i = part * 128 + threadIdx.x;
    const uint64_t* src = in.at(poly, 0) + i;
#pragma unroll
    for (int k = 0; k < MAXF; k++) z[k] = k < (int)F ? src[(uint64_t)k << logn] : 0;
#pragma unroll
    for (int k = 0; k < MAXF; k++) {
      if (k < (int)F) {
        const DevPrime& pr = src_primes[k];
        z[k] = (uint64_t)fold_lift((uint64_t)fold_mul(fold_lift(z[k], pr), __ldg(zc + 3 * k), pr) + pr.f_bias, pr);
      }
    }
  } else {
    uint64_t* staged = reinterpret_cast<uint64_t*>(sa);
    b0 = part * G;
    logb = logn - TOP;
    constexpr int IT = (MAXF * G + 127) / 128;
    uint64_t x[IT][1 << TOP];
#pragma unroll
    for (int u = 0; u < IT; u++) {
      const uint32_t item = threadIdx.x + 128 * u;
      if (item < F * G) {
        const uint64_t* row = in.at(poly, item / G) + b0 + item % G;
#pragma unroll
        for (int e = 0; e < (1 << TOP); e++) x[u][e] = row[(uint64_t)e << logb];
      }
    }
#pragma unroll
    for (int u = 0; u < IT; u++) {
      const uint32_t item = threadIdx.x + 128 * u;
      if (item < F * G) {
        const uint32_t k = item / G, g2 = item % G;
        inv_top_fold<TOP, false>(x[u], src_primes[k], 1u << logn, __ldg(zc + 3 * k + 1), __ldg(zc + 3 * k + 2));
#pragma unroll
        for (int e = 0; e < (1 << TOP); e++) staged[(k * (1 << TOP) + e) * G + g2] = x[u][e];
      }
    }
    __syncthreads();
    t = threadIdx.x / G;
    gi = threadIdx.x % G;
    i = b0 + gi + (t << logb);
#pragma unroll
    for (int k = 0; k < MAXF; k++) z[k] = k < (int)F ? staged[(k * (1 << TOP) + t) * G + gi] : 0;
    if (fe.primes) {
      const uint32_t which = fe.period ? poly % fe.period : 0;
      fwd_here = which < fe.take;
      dig_here = !fwd_here && fe.digit_primes != nullptr;
    }
    __syncthreads();  // A overlays the buffer
  }

  hat_operand<MAXF, 0>(sa, z);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = slot;
  if (threadIdx.x == 0) hat_mma<KP>(bar_b, 0, bar_mma, tmem, a_addr, b_addr, s.b_rows, 0);

  // v = round(sum z_k / m_k) in units of 2^-58, and whether it is too close to
  // a boundary.
  uint64_t acc = 1ull << 57;
#pragma unroll
  for (int k = 0; k < MAXF; k++)
    if (k < (int)F) acc = fold_madu(__funnelshift_r((uint32_t)z[k], (uint32_t)(z[k] >> 32), s.zsh[k]), s.inv[k], acc);
  const uint32_t v = (uint32_t)(acc >> 58);
  bool near = (acc & ((1ull << 58) - 1)) - s.v_margin > (1ull << 58) - 2 * s.v_margin;
  // w = round(sum z_k phi_k + v (1 - gamma)): the digit products sum without
  // carries (16 terms of 2^60), then meet in units of 2^-56. Five of the seven
  // would give w to 2^-18, too little: at 49152 coefficients a multiplication
  // every third one then waited 18 us for a thread in hat_exact.
  uint64_t wlo = 0, whi = 0;
  if constexpr (!ONE) {
    uint64_t a1 = 0, a2 = 0, a3 = 0, b1 = 0, b2 = 0, b3 = 0, b4 = 0;
#pragma unroll
    for (int k = 0; k < MS; k++) {
      if (k < MAXF && k < (int)s.frac) {
        const uint32_t z0 = (uint32_t)z[k], z1 = (uint32_t)(z[k] >> 32);
        a1 = fold_madu(z0, s.th1[k], a1);
        b1 = fold_madu(z1, s.th1[k], b1);
        a2 = fold_madu(z0, s.th2[k], a2);
        b2 = fold_madu(z1, s.th2[k], b2);
        a3 = fold_madu(z0, s.th3[k], a3);
        b3 = fold_madu(z1, s.th3[k], b3);
        b4 = fold_madu(z1, s.th4[k], b4);
      }
    }
    a1 = fold_madu(v, s.g1, a1);
    a2 = fold_madu(v, s.g2, a2);
    unsigned __int128 sum = (unsigned __int128)a1 << 28;
    sum += (unsigned __int128)b1 << 60;
    sum += (unsigned __int128)b2 << 32;
    sum += (unsigned __int128)b3 << 4;
    sum += a2 + (unsigned __int128)((a3 >> 28) + (b4 >> 24));
    sum += 1ull << 55;
    const uint64_t frac = (uint64_t)sum & ((1ull << 56) - 1);
    near = near || frac - s.w_margin > (1ull << 56) - 2 * s.w_margin;
    sum >>= 56;
    wlo = (uint64_t)sum;
    whi = (uint64_t)(sum >> 64);
  }
  if constexpr (K::kChunks == 2) {
    // The second half of the sources over the first, once its MMAs are done.
    if (!mbar_wait(bar_mma, 0, kTcWaitTries)) atomicAdd(&g_hat_wait_failures, 1u);
    if (threadIdx.x == 0) {
      mbar_expect_tx(bar_b, s.out_len * 16 * KP);
      bulk_g2s(b_addr, mat + s.chunk_words, s.out_len * 16 * KP, bar_b);
    }
    hat_operand<MAXF, 1>(sa, z);
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) hat_mma<KP>(bar_b, 1, bar_mma + 8, tmem, a_addr, b_addr, s.b_rows, 1);
  }
  uint64_t ye[MAXT];
  if (near) {
    uint64_t zl[MAXF];
#pragma unroll
    for (int k = 0; k < MAXF; k++) zl[k] = z[k];
    hat_exact(ex, zl, start, s.out_len, ye);
  }
  __syncwarp();

  if (!mbar_wait(bar_mma + 8 * (K::kChunks - 1), 0, kTcWaitTries)) atomicAdd(&g_hat_wait_failures, 1u);
  tc_fence_after();
  const uint32_t lane = tmem + (((threadIdx.x >> 5) * 32u) << 16);
  uint64_t* dst = out.at(poly, 0) + i;
#pragma unroll
  for (int q = 0; q < MAXT; q += 4) {
    if (q >= (int)s.out_len) continue;
    uint32_t d[32];
    tc_ld32(lane + 8 * q, d);  // the columns beyond the outputs are allocated too
#pragma unroll
    for (int o = q; o < q + 4; o++) {
      if (o >= (int)s.out_len) continue;
      uint32_t hi;
      uint64_t lo;
      hat_sum<BIASED>(d + 8 * (o - q), &lo, &hi);
      // T = sum + v gneg + w, below 2^(k + 32), folded once at 2^k.
      const uint64_t p0 = fold_madu(v, (uint32_t)s.gneg[o], 0);
      const uint64_t p1 = fold_madu(v, (uint32_t)(s.gneg[o] >> 32), p0 >> 32);
      unsigned __int128 T = ((unsigned __int128)hi << 64) + lo;
      T += ((unsigned __int128)(p1 >> 32) << 64) + pack64((uint32_t)p0, (uint32_t)p1);
      if constexpr (!ONE) T += ((unsigned __int128)whi << 64) + wlo;
      const uint64_t tlo = (uint64_t)T;
      const uint32_t th = (uint32_t)(tlo >> 32), top = (uint32_t)(uint64_t)(T >> 64);
      uint64_t y = fold_madu(__funnelshift_r(th, top, s.sh[o]), s.c[o], pack64((uint32_t)tlo, th & ((1u << s.sh[o]) - 1)));
      y = csub(y, s.p[o]);
      if (near) y = ye[o];
      if (TOP > 0 && (fwd_here || dig_here))
        reinterpret_cast<uint64_t*>(sa)[(o * (1 << TOP) + t) * G + gi] = y;
      else dst[(uint64_t)o << logn] = y;
    }
  }
  // Every lane's reads are done (tc_ld32 waits for them): free the columns.
  tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 1) tc_dealloc(tmem, s.cols);
  pdl_trigger();
  if constexpr (TOP > 0) {
    if (fwd_here || dig_here)
      scale_epilogue<TOP, true>(reinterpret_cast<uint64_t*>(sa), fwd_here, s.out_len, poly, b0, logb, out, fe);
  }
}

// Sources, outputs and sources with a fraction of the kernels. A scaler takes
// the first one that holds all three. Scale-downs of multiplications have a
// fraction at up to F / 2 + 1 sources, decryption's at every one: up to 16 sources
// the kernels come with both (one with them all is 0.5% slower for the former,
// whose unrolled sums it skips one by one; the next larger class was 20-45% slower
// for the latter: 13 sources to 1 output 27.4 -> 18.7 us, 12 to 12 with
// six fractions 43.2 on k_rns_scale's tensor cores -> 35.1).
struct HatClass {
  uint32_t maxf, maxt, maxs;
};
constexpr HatClass kHatOne[] = {{3, 8, 1}, {6, 8, 1}, {8, 16, 1}, {12, 16, 1}, {16, 16, 1}};
constexpr HatClass kHatDown[] = {{7, 8, 4},   {7, 8, 7},    {13, 8, 7},   {13, 8, 13},
                                 {16, 16, 9}, {16, 16, 16}, {25, 16, 13}, {32, 16, 16}};

// HatShape at run time.
constexpr uint32_t hat_chunks(uint32_t maxf) { return maxf > 12 ? 2 : 1; }
constexpr uint32_t hat_per(uint32_t maxf) { return (maxf + hat_chunks(maxf) - 1) / hat_chunks(maxf); }
constexpr uint32_t hat_kp(uint32_t maxf) { return (8 * (hat_per(maxf) + (maxf <= 16 ? 1 : 0)) + 15) / 16 * 16; }

// FP16 bit pattern of an integer 0..255 (exact).
uint16_t byte_half(uint32_t v) {
  if (v == 0) return 0;
  const int e = 31 - __builtin_clz(v);
  return (uint16_t)(((e + 15) << 10) | ((v << (10 - e)) & 0x3FF));
}

// Once per kernel and device: raises the dynamic shared memory limit; returns
// the kernel's static shared memory.
size_t hat_prepare(const void* kern, size_t most) {
  struct Entry {
    const void* kern;
    int dev;
    size_t stat;
  };
  static std::mutex mu;
  static std::vector<Entry> done;
  int dev = 0;
  check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> lock(mu);
  for (const Entry& e : done)
    if (e.kern == kern && e.dev == dev) return e.stat;
  cudaFuncAttributes a{};
  check_cuda(cudaFuncGetAttributes(&a, kern), "cudaFuncGetAttributes");
  check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most),
             "cudaFuncSetAttribute");
  done.push_back(Entry{kern, dev, a.sharedSizeBytes});
  return a.sharedSizeBytes;
}

template <int MAXF, int MAXT, int MS, int TOP, bool ONE>
void launch_hat_top(const RnsScalerD& sc, uint32_t logn, PolyRef in, PolyRef out, uint32_t start, uint32_t out_len,
                    uint64_t total, cudaStream_t st, const FwdEpilogue& fe) {
  constexpr uint32_t KP = HatShape<MAXF>::kKp;
  const RnsHatD& h = *sc.hat;
  if (h.kp != KP) throw Error(FHEG_ERR_INTERNAL, "tensor-core scaler matrix of another width");
  HatLaunch<MAXF, MAXT, MS> s;
  memset(&s, 0, sizeof(s));
  s.from_len = (uint32_t)sc.host.from_len;
  s.out_len = out_len;
  s.frac = h.frac;
  s.chunk_words = (uint32_t)sc.host.to_len * 8 * KP;
  for (uint32_t k = 0; k < s.from_len; k++) {
    s.inv[k] = h.inv[k];
    s.zsh[k] = h.zsh[k];
  }
  for (uint32_t k = 0; k < h.frac; k++) {
    s.th1[k] = h.th[4 * k];
    s.th2[k] = h.th[4 * k + 1];
    s.th3[k] = h.th[4 * k + 2];
    s.th4[k] = h.th[4 * k + 3];
  }
  s.g1 = h.g1;
  s.g2 = h.g2;
  s.v_margin = h.v_margin;
  s.w_margin = h.w_margin;
  for (uint32_t o = 0; o < out_len; o++) {
    const size_t j = start + o;
    s.gneg[o] = h.gneg[j];
    s.p[o] = sc.to_moduli[j];
    s.c[o] = h.c[j];
    s.sh[o] = h.sh[j];
  }
  s.b_rows = (8 * out_len + 15) / 16 * 16;
  s.cols = s.b_rows <= 32 ? 32 : s.b_rows <= 64 ? 64 : 128;
  auto kern = k_rns_hat<MAXF, MAXT, MS, TOP, ONE>;
  // The stage buffer (TOP > 0) overlaid by A, then B; at least 456 bytes per
  // tensor-memory column (with the 1 KB the SM reserves per CTA), so that the
  // CTAs an SM holds never ask for more than its 512 columns.
  constexpr size_t kStage = TOP > 0 ? (size_t)(MAXF > MAXT ? MAXF : MAXT) * 128 * 8 : 0;
  constexpr size_t kA = ((128 * KP * 2 > kStage ? 128 * KP * 2 : kStage) + 127) / 128 * 128;
  const size_t stat = hat_prepare(reinterpret_cast<const void*>(kern),
                                  std::max<size_t>(kA + 8 * MAXT * 2 * KP, 128 * kTcSmemPerColumn));
  s.b_offset = (uint32_t)kA;
  const size_t dyn = std::max<size_t>(kA + (size_t)s.b_rows * 2 * KP, s.cols * kTcSmemPerColumn - 1024 - stat);
  launch_dependent(kern, dim3((unsigned)(total / 128)), 128, dyn, st, s, logn, in, out, h.from_primes, h.zc,
                   h.mat + (size_t)start * 8 * KP, static_cast<const HatExact*>(h.exact), start, fe);
  after_launch("k_rns_hat");
}

template <int MAXF, int MAXT, int MS, bool ONE>
void launch_hat(const RnsScalerD& sc, uint32_t logn, PolyRef in, PolyRef out, uint32_t start, uint32_t out_len,
                uint64_t total, cudaStream_t st, uint32_t top, const FwdEpilogue& fe) {
  switch (top) {
    case 0: launch_hat_top<MAXF, MAXT, MS, 0, ONE>(sc, logn, in, out, start, out_len, total, st, fe); break;
    case 1: launch_hat_top<MAXF, MAXT, MS, 1, ONE>(sc, logn, in, out, start, out_len, total, st, fe); break;
    case 2: launch_hat_top<MAXF, MAXT, MS, 2, ONE>(sc, logn, in, out, start, out_len, total, st, fe); break;
    case 3: launch_hat_top<MAXF, MAXT, MS, 3, ONE>(sc, logn, in, out, start, out_len, total, st, fe); break;
    default: throw Error(FHEG_ERR_INTERNAL, "unsupported strided stage count");
  }
}

}  // namespace

uint64_t hat_wait_failures() {
  uint32_t v = 0;
  check_cuda(cudaMemcpyFromSymbol(&v, g_hat_wait_failures, sizeof(v)), "cudaMemcpyFromSymbol");
  return v;
}

void rns_scale_hat(const RnsScalerD& sc, uint32_t logn, PolyRef in, PolyRef out, uint32_t start, uint32_t out_len,
                   uint64_t polys, cudaStream_t st, const InverseTop* top, const ForwardTop* fwd) {
  FwdEpilogue fe{};
  if (fwd) fe = FwdEpilogue{fwd->primes, fwd->period, fwd->take, fwd->digit_primes, fwd->digit_limbs, fwd->digit_raw,
                            fwd->digits};
  const uint64_t total = polys << logn;
  const uint32_t s1 = top ? top->s1 : 0;
  const bool one = sc.host.is_one;
  const uint32_t cls = sc.hat->maxf, fr = sc.hat->maxs;
#define HAT(F_, T_, S_, ONE_) launch_hat<F_, T_, S_, ONE_>(sc, logn, in, out, start, out_len, total, st, s1, fe)
  if (one) {
    if (cls == 3) HAT(3, 8, 1, true);
    else if (cls == 6) HAT(6, 8, 1, true);
    else if (cls == 8) HAT(8, 16, 1, true);
    else if (cls == 12) HAT(12, 16, 1, true);
    else HAT(16, 16, 1, true);
  } else {
    if (cls == 7 && fr == 4) HAT(7, 8, 4, false);
    else if (cls == 7) HAT(7, 8, 7, false);
    else if (cls == 13 && fr == 7) HAT(13, 8, 7, false);
    else if (cls == 13) HAT(13, 8, 13, false);
    else if (cls == 16 && fr == 9) HAT(16, 16, 9, false);
    else if (cls == 16) HAT(16, 16, 16, false);
    else if (cls == 25) HAT(25, 16, 13, false);
    else HAT(32, 16, 16, false);
  }
#undef HAT
}

std::unique_ptr<RnsHatD> make_rns_hat(const Context& from, const Context& to, const RnsScalerHost& host,
                                      const std::vector<uint64_t>& gneg, const std::vector<uint64_t>& gneg_hi,
                                      const BigUint& num, const BigUint& den) {
  const size_t F = from.L(), T = to.L();
  if (!from.fold || !to.fold || F > 32) return nullptr;
  auto h = std::make_unique<RnsHatD>();
  const BigUint& M = from.rns->product;
  // Phi_k, phi_k (112 bits) and Gamma, gamma.
  std::vector<BigUint> phi_int(F);
  std::vector<u128> phi(F);
  h->frac = 0;
  std::vector<uint64_t> hat_mod(F), hat_inv(F);
  for (size_t k = 0; k < F; k++) {
    const uint64_t m = from.moduli[k];
    const BigUint hat = M / BigUint(m);
    hat_mod[k] = hat.mod_u64(m);
    hat_inv[k] = invmod(hat_mod[k], m);
    if (host.is_one) {
      phi_int[k] = hat;
      continue;
    }
    BigUint rem;
    BigUint::divmod(hat * num, den, &phi_int[k], &rem);
    if (rem.is_zero()) continue;
    phi[k] = ((rem << 112) / den).low_u128();
    h->frac = (uint32_t)k + 1;
  }
  BigUint gamma_int = M, gamma_rem;
  if (!host.is_one) BigUint::divmod(M * num, den, &gamma_int, &gamma_rem);
  // 1 - gamma with gamma rounded up; without a fraction, Gamma itself and 0.
  uint64_t one_minus = 0;
  if (!gamma_rem.is_zero()) {
    gamma_int = gamma_int + BigUint(1);
    one_minus = (uint64_t)((((den - gamma_rem) << 56) / den).low_u128());
  }
  h->g1 = (uint32_t)(one_minus >> 28);
  h->g2 = (uint32_t)(one_minus & ((1u << 28) - 1));
  // The kernel class, by the outputs a scaling writes (with factor one, without
  // the leading moduli both sides share); where none holds them all, for calls
  // that ask for fewer.
  size_t outs = T;
  if (host.is_one)
    for (size_t k = 0; k < F && k < T && from.moduli[k] == to.moduli[k]; k++) outs--;
  h->maxf = h->maxt = h->maxs = 0;
  auto pick = [&](const HatClass& c, size_t least) {
    if (!h->maxf && F <= c.maxf && h->frac <= c.maxs && least <= c.maxt) h->maxf = c.maxf, h->maxt = c.maxt, h->maxs = c.maxs;
  };
  for (const size_t least : {outs, (size_t)0}) {
    if (host.is_one)
      for (const HatClass& c : kHatOne) pick(c, least);
    else
      for (const HatClass& c : kHatDown) pick(c, least);
  }
  if (!h->maxf) return nullptr;
  h->kp = hat_kp(h->maxf);
  h->v_margin = 0;
  for (size_t k = 0; k < F; k++) {
    const DevPrime& d = from.primes[k]->dev;
    const uint32_t bits = (uint32_t)d.f_sh + 32;
    h->zsh.push_back(bits - 31);
    // Error of v, in units of 2^-58: 2^27 and a little for z_k to 31 bits, and
    // 2^31 times what the rounded inverse is off (for m_k close to 2^k, next to
    // nothing).
    const u128 full = (u128)1 << (bits + 27), r = (full + d.p / 2) / d.p;
    h->inv.push_back((uint32_t)r);
    const u128 off = r * d.p > full ? r * d.p - full : full - r * d.p;
    h->v_margin += (1ull << 27) + (1ull << 24) + (uint64_t)((off << 32) / d.p) + 1;
  }
  for (size_t k = 0; k < h->frac; k++)
    for (int q = 3; q >= 0; q--) h->th.push_back((uint32_t)(phi[k] >> (28 * q)) & ((1u << 28) - 1));
  // Error of w, in units of 2^-56: 2^6 a source for 112-bit phi and the dropped
  // digit product, a few more for the two shifts and v (1 - gamma).
  h->w_margin = (uint64_t)(h->frac + 1) << 7;
  // One fold must take T = sum + v gneg + w below 2 q_j: T is below
  // (2040 F + 2 F + 2) q_j + frac 2^62 + 2^8, and T >> k must fit 32 bits.
  unsigned zbits = 0;
  for (size_t k = 0; k < h->frac; k++) zbits = std::max<unsigned>(zbits, h->zsh[k] + 31);
  for (size_t j = 0; j < T; j++) {
    const DevPrime& d = to.primes[j]->dev;
    const unsigned bits = (unsigned)d.f_sh + 32;
    u128 most = (u128)(2042 * F + 2) * d.p + 256;
    if (h->frac) most += (u128)(2 * h->frac) << zbits;
    const u128 n = most >> bits;
    if (n >> 32) return nullptr;
    if (((u128)1 << bits) + n * (u128)d.f_c >= 2 * (u128)d.p) return nullptr;
    const uint64_t g = gamma_int.mod_u64(d.p);
    h->gneg.push_back(g ? d.p - g : 0);
    h->c.push_back((uint32_t)d.f_c);
    h->sh.push_back((uint32_t)d.f_sh);
  }
  // The byte matrix of each chunk: rows 8j + c hold byte c of Phi_k 2^(8b) mod
  // q_j at column 8 (k mod per) + b (core matrices of 8 rows by 16 bytes, tc.cuh).
  const uint32_t kp = h->kp, per = hat_per(h->maxf);
  std::vector<uint16_t> mat(hat_chunks(h->maxf) * T * 8 * kp, 0);
  auto at = [&](size_t row, size_t k, size_t b) -> uint16_t& {
    return mat[(k / per) * T * 8 * kp + ((row & 7) * 16 + b * 2 + (k % per) * 128 + (row >> 3) * 16 * kp) / 2];
  };
  for (size_t j = 0; j < T; j++) {
    const uint64_t q = to.moduli[j];
    for (size_t k = 0; k < F; k++) {
      uint64_t v = phi_int[k].mod_u64(q);
      for (uint32_t b = 0; b < 8; b++) {
        for (uint32_t c = 0; c < 8; c++) at(8 * j + c, k, b) = byte_half((uint32_t)(v >> (8 * c)) & 255);
        v = mulmod(v, 256, q);
      }
    }
    if (h->maxf <= 16)
      for (uint32_t c = 0; c < 8; c++) mat[(c * 16 + per * 128 + j * 16 * kp) / 2] = 0x6C00;
  }
  // hat_k^-1 alone and with the last constants of an inverse NTT.
  std::vector<int4> zc(3 * F);
  for (size_t k = 0; k < F; k++) {
    const DevPrime& d = from.primes[k]->dev;
    zc[3 * k] = fold_constant(hat_inv[k], d);
    zc[3 * k + 1] = fold_constant(mulmod(hat_inv[k], d.ninv, d.p), d);
    zc[3 * k + 2] = fold_constant(mulmod(hat_inv[k], d.zlast_ninv, d.p), d);
  }
  h->from_primes = from.primes_dev();
  // One device buffer and one copy: the matrix, the digits, the reference's
  // sums for hat_exact and their directory.
  std::vector<uint8_t> buf;
  auto put = [&](const void* v, size_t bytes) {
    const size_t o = (buf.size() + 127) / 128 * 128;
    buf.resize(o + bytes);
    memcpy(buf.data() + o, v, bytes);
    return o;
  };
  auto put64 = [&](const std::vector<uint64_t>& v) { return put(v.data(), v.size() * 8); };
  const size_t o_mat = put(mat.data(), mat.size() * 2), o_zc = put(zc.data(), zc.size() * sizeof(int4));
  const size_t o_hat = put64(hat_mod), o_gl = put64(host.theta_garner_lo), o_gh = put64(host.theta_garner_hi),
               o_ol = put64(host.theta_omega_lo), o_oh = put64(host.theta_omega_hi), o_om = put64(host.omega),
               o_g = put64(gneg), o_gg = put64(gneg_hi);
  const size_t o_ex = (buf.size() + 127) / 128 * 128;
  h->tables.alloc(o_ex + sizeof(HatExact));
  uint8_t* base = static_cast<uint8_t*>(h->tables.ptr);
  auto words = [&](size_t o) { return reinterpret_cast<const uint64_t*>(base + o); };
  HatExact e{};
  e.from_len = (uint32_t)F;
  e.is_one = host.is_one ? 1 : 0;
  e.shift = (uint32_t)host.theta_garner_shift;
  e.tg_sign = host.theta_gamma_sign ? 1 : 0;
  for (size_t k = 0; k < F; k++)
    if (host.theta_omega_sign[k]) e.to_sign |= 1u << k;
  e.tg_lo = host.theta_gamma_lo;
  e.tg_hi = host.theta_gamma_hi;
  e.from = from.primes_dev();
  e.to = to.primes_dev();
  e.hat = words(o_hat);
  e.gar_lo = words(o_gl);
  e.gar_hi = words(o_gh);
  e.om_lo = words(o_ol);
  e.om_hi = words(o_oh);
  e.omega = words(o_om);
  e.gneg = words(o_g);
  e.gneg_hi = words(o_gg);
  put(&e, sizeof(e));
  upload(base, buf.data(), buf.size());
  h->mat = reinterpret_cast<const uint16_t*>(base + o_mat);
  h->zc = reinterpret_cast<const int4*>(base + o_zc);
  h->exact = base + o_ex;
  return h;
}

}  // namespace fheg
