// Fused key-switching row kernel for N = 2^16.
//
// Between the two fused column passes of a key switch (modswitch.cu) every
// remaining step is row-local in the 16 x 4096 limb layout:
//   * the ModUp NTT row phase of every digit (src/core/NTT.cu NTTForModUp),
//   * the key inner product sum_i ModUp(d)_i (.) key_i (Context.cpp:609-647),
//   * the P * (d0, d1) term (Context.cpp:687-699) with the tensor product
//     d0 = b1 b2, d1 = b1 a2 + a1 b2 recomputed from the inputs
//     (ElementWise.cu:504-575), and the own-digit ModUp value d2 = a1 a2,
//   * and, for the primes that ModDown drops, the INTT row phase
//     (NTT.cu:973-1128, INTTForModDown).
// One CTA owns one row of one prime of the extended basis Q u P for one
// ciphertext (each ciphertext names the row tables of its own level, so
// ciphertexts at different levels share a launch); it reads each input row
// once and writes either the
// evaluation-domain accumulator (kept primes, consumed by the ModDown
// epilogue) or the INTT row-phase output (dropped primes, consumed by the
// ModDown column pass).
#include "arith.cuh"
#include "kernels.h"
#include "ntt_common.cuh"

namespace chd {
namespace {

// Inner-product accumulators are 64-bit sums kept below q 2^32: two products
// of canonical residues (2 q^2 < q 2^32) may be added before the high word,
// then below 2q, is brought back below q (one instruction; q 2^32 is a
// multiple of q).  One Montgomery reduction at the end replaces one per
// product.
__device__ __forceinline__ void acc_fold(uint64_t &s, uint32_t q) {
  const uint32_t hi = reduce2q(static_cast<uint32_t>(s >> 32), q);
  s = (static_cast<uint64_t>(hi) << 32) | static_cast<uint32_t>(s);
}
// s 2^-32 mod q, canonical, for s < 2 q 2^32: with m = lo(s) q^-1,
// (s - m q) / 2^32 = hi(s) - hi(m q)
__device__ __forceinline__ uint32_t acc_reduce(uint64_t s, uint32_t q, int32_t qi) {
  const uint32_t hi = reduce2q(static_cast<uint32_t>(s >> 32), q);
  const uint32_t r = hi - __umulhi(static_cast<uint32_t>(s) * static_cast<uint32_t>(qi), q);  // (-q, q)
  return min(r, r + q);
}

__global__ void __launch_bounds__(kRowThreads, 2) k_ks_rows(const __grid_constant__ KSRowsDesc d) {
  __shared__ __align__(16) uint32_t sm[2][kRowLen];
  // grid (count, 16, max_rows): the ciphertexts sharing one key row are
  // neighbours in launch order, so the key row comes from HBM once
  const int j = blockIdx.z;
  const KSRowsCt &c = d.ct[blockIdx.x];
  const KSRowsLevel &L = d.lv[c.lv];
  if (j >= L.rows) return;  // a ciphertext below the launch's largest level
  const int g = L.gidx[j];
  const uint32_t q = __ldg(d.primes + g);
  const int32_t qi = __ldg(d.qinvs + g);
  const uint2 *tw = d.tw + (static_cast<size_t>(g) << 16);
  const int t = threadIdx.x, r = blockIdx.y;
  const size_t row = static_cast<size_t>(j) * 65536 + r * kRowLen;
  const size_t off = row + chunk_off(t);  // input rows share the accumulator row index for q primes
  const size_t koff = static_cast<size_t>(L.key_row[j]) * 65536 + r * kRowLen + chunk_off(t);
  const bool is_q = j < L.nq;
  const int mode = d.mode;
  uint64_t sb[16], sa[16];
#pragma unroll
  for (int k = 0; k < 16; k++) sb[k] = sa[k] = 0;
  const int own = L.own_digit[j];
  int buf = 0;
  for (int i = 0; i < L.beta; i++) {
    uint32_t v[16];
    if (own == i) {
      // own primes of the digit: the ModUp value is the key-switched input
      ld_chunks((mode == 2 ? c.a2 : c.a1) + off, v);
      if (mode == 0) {
        uint32_t y[16];
        ld_chunks(c.a2 + off, y);
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = mont_mul(v[k], y[k], q, qi);
      }
    } else {
      const uint32_t *src = c.mu[i] + row;
#pragma unroll
      for (int k = 0; k < 16; k++) v[k] = src[t + 256 * k];
      row_fwd(v, sm[buf], tw, r, t, q);
      buf ^= 1;
#pragma unroll
      for (int k = 0; k < 16; k++) v[k] = reduce2q(v[k], q);
    }
    const uint32_t *kb = L.kb[i] + koff, *ka = L.ka[i] + koff;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const uint4 b4 = __ldg(reinterpret_cast<const uint4 *>(kb + 64 * e));
      const uint4 a4 = __ldg(reinterpret_cast<const uint4 *>(ka + 64 * e));
      const uint32_t kbv[4] = {b4.x, b4.y, b4.z, b4.w}, kav[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        sb[4 * e + k] += static_cast<uint64_t>(v[4 * e + k]) * kbv[k];
        sa[4 * e + k] += static_cast<uint64_t>(v[4 * e + k]) * kav[k];
      }
    }
    if (i & 1) {
#pragma unroll
      for (int k = 0; k < 16; k++) {
        acc_fold(sb[k], q);
        acc_fold(sa[k], q);
      }
    }
  }
  if (is_q && c.b1 != nullptr) {
    // P * (d0, d1): HMult d0 = b1 b2, d1 = b1 a2 + a1 b2; MultKey d0 = bx;
    // Relinearize d0 = bx, d1 = ax.  Without b1: the bare inner product.
    const uint64_t pp = L.p_prod[j];
    const uint32_t qneg = 0u - static_cast<uint32_t>(qi);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      auto ld4 = [&](const uint32_t *p, uint32_t *x) {
        const uint4 v4 = __ldg(reinterpret_cast<const uint4 *>(p + off + 64 * e));
        x[0] = v4.x; x[1] = v4.y; x[2] = v4.z; x[3] = v4.w;
      };
      uint32_t b1[4];
      ld4(c.b1, b1);
      if (mode == 0) {
        uint32_t b2[4], a1[4], a2[4];
        ld4(c.b2, b2);
        ld4(c.a1, a1);
        ld4(c.a2, a2);
#pragma unroll
        for (int k = 0; k < 4; k++) {
          sb[4 * e + k] += pp * mont_mul(b1[k], b2[k], q, qi);
          sa[4 * e + k] += pp * mont_mac2(b1[k], a2[k], a1[k], b2[k], q, qneg);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++) sb[4 * e + k] += pp * b1[k];
        if (mode == 2) {
          uint32_t a1[4];
          ld4(c.a1, a1);
#pragma unroll
          for (int k = 0; k < 4; k++) sa[4 * e + k] += pp * a1[k];
        }
      }
    }
  }
  uint32_t ob[16], oa[16];
#pragma unroll
  for (int k = 0; k < 16; k++) {
    ob[k] = acc_reduce(sb[k], q, qi);
    oa[k] = acc_reduce(sa[k], q, qi);
  }
  const int di = L.drop_idx[j];
  if (di < 0) {
    st_chunks(c.acc_b + off, ob);
    st_chunks(c.acc_a + off, oa);
    return;
  }
  // dropped prime: INTT row phase of both accumulators (ModDown's first step)
  const uint2 *itw = d.itw + (static_cast<size_t>(g) << 16);
  const size_t doff = static_cast<size_t>(di) * 65536 + r * kRowLen + t;
  row_inv(ob, sm[buf], itw, r, t, q);
#pragma unroll
  for (int k = 0; k < 16; k++) c.drop_b[doff + 256 * k] = ob[k];
  row_inv(oa, sm[buf ^ 1], itw, r, t, q);
#pragma unroll
  for (int k = 0; k < 16; k++) c.drop_a[doff + 256 * k] = oa[k];
}

}  // namespace

void launch_ks_rows(const KSRowsDesc &d, int log_n, cudaStream_t s) {
  if (d.count <= 0 || d.max_rows <= 0 || log_n != 16) return;
  k_ks_rows<<<dim3(d.count, kLimbRows, d.max_rows), kRowThreads, 0, s>>>(d);
}

}  // namespace chd
