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
#include "launch.cuh"
#include "ntt_common.cuh"

namespace chd {
namespace {

constexpr int kWholeDigits = 4;  // digits whose rows wait in shared memory together
constexpr int kGroupDigits = 2;  // digits of a group where there are more

// Inner-product accumulators are 64-bit sums kept below q 2^32: two products
// of canonical residues (2 q^2 < q 2^32) may be added before the high word,
// then below 2q, is brought back below q (one instruction; q 2^32 is a
// multiple of q).  One Montgomery reduction at the end (of a group of digits)
// replaces one per product.  The P term comes before the first two products:
// three of them, below 3 q^2 < 2 q 2^32.
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

// Inner product and P (d0, d1) of one row, four coefficients at a time, for
// the B digits from i0 on, whose canonical ModUp rows lie in the row buffers
// sm (B known at compile time, so that the key words of all digits can be in
// flight together and their pointers stay in registers).  GROUPED: the sums
// over the groups of digits, canonical between them, lie in the two row
// buffers `res`; otherwise there is one group, and res = sm.
template <int B, bool GROUPED>
__device__ __forceinline__ void inner_product(const KSRowsCt &c, const KSRowsLevel &L, const uint32_t *sm, uint32_t *res,
                                              int i0, int j, int mode, size_t off, size_t koff, uint32_t q, int32_t qi,
                                              int t) {
  const bool is_q = j < L.nq, first = !GROUPED || i0 == 0, last = !GROUPED || i0 + B == L.beta;
  const bool with_p = is_q && first && c.b1 != nullptr;
  const int own = L.own_digit[j] - i0, di = L.drop_idx[j];
  const uint32_t *kb[B], *ka[B];
#pragma unroll
  for (int i = 0; i < B; i++) {
    kb[i] = L.kb[i0 + i] + koff;
    ka[i] = L.ka[i0 + i] + koff;
  }
#pragma unroll 1
  for (int e = 0; e < 4; e++) {
    auto ld4 = [&](const uint32_t *p, uint32_t *x) {
      const uint4 v4 = *reinterpret_cast<const uint4 *>(p + 64 * e);
      x[0] = v4.x; x[1] = v4.y; x[2] = v4.z; x[3] = v4.w;
    };
    uint64_t sb[4] = {0, 0, 0, 0}, sa[4] = {0, 0, 0, 0};
    uint32_t vo[4] = {0, 0, 0, 0};
    if (is_q && (first || (own >= 0 && own < B))) {
      // the own digit's ModUp value is the key-switched input; P * (d0, d1):
      // HMult d0 = b1 b2, d1 = b1 a2 + a1 b2; MultKey d0 = bx; Relinearize
      // d0 = bx, d1 = ax.  Without b1: the bare inner product.
      const uint64_t pp = L.p_prod[j];
      uint32_t a1[4], a2[4], b1[4], b2[4];
      ld4(c.a1 + off, a1);
      if (mode != 1) ld4(c.a2 + off, a2);
      if (with_p) ld4(c.b1 + off, b1);
      if (mode == 0 && !first) {
#pragma unroll
        for (int k = 0; k < 4; k++) vo[k] = mont_mul(a1[k], a2[k], q, qi);
      } else if (mode == 0) {
        ld4(c.b2 + off, b2);
        const uint32_t qneg = 0u - static_cast<uint32_t>(qi);
#pragma unroll
        for (int k = 0; k < 4; k++) {
          vo[k] = mont_mul(a1[k], a2[k], q, qi);
          sb[k] = pp * mont_mul(b1[k], b2[k], q, qi);
          sa[k] = pp * mont_mac2(b1[k], a2[k], a1[k], b2[k], q, qneg);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          vo[k] = mode == 1 ? a1[k] : a2[k];
          if (with_p) sb[k] = pp * b1[k];
          if (with_p && mode == 2) sa[k] = pp * a1[k];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < B; i++) {
      uint32_t b4[4], a4[4];
      ld4(kb[i], b4);
      ld4(ka[i], a4);
      uint4 v4 = make_uint4(vo[0], vo[1], vo[2], vo[3]);
      if (own != i) v4 = chunk_ld4(sm + i * kRowBuf, t, e);
      const uint32_t v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        sb[k] += static_cast<uint64_t>(v[k]) * b4[k];
        sa[k] += static_cast<uint64_t>(v[k]) * a4[k];
      }
      if (i & 1) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          acc_fold(sb[k], q);
          acc_fold(sa[k], q);
        }
      }
    }
    uint32_t ob[4], oa[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      ob[k] = acc_reduce(sb[k], q, qi);
      oa[k] = acc_reduce(sa[k], q, qi);
    }
    if (!first) {
      const uint4 b4 = chunk_ld4(res, t, e), a4 = chunk_ld4(res + kRowBuf, t, e);
      const uint32_t pb[4] = {b4.x, b4.y, b4.z, b4.w}, pa[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        ob[k] = add_mod(ob[k], pb[k], q);
        oa[k] = add_mod(oa[k], pa[k], q);
      }
    }
    const uint4 b4 = make_uint4(ob[0], ob[1], ob[2], ob[3]), a4 = make_uint4(oa[0], oa[1], oa[2], oa[3]);
    if (last && di < 0) {
      *reinterpret_cast<uint4 *>(c.acc_b + off + 64 * e) = b4;
      *reinterpret_cast<uint4 *>(c.acc_a + off + 64 * e) = a4;
    } else {
      // this thread has read chunk e of every digit
      chunk_st4(res, t, e, b4);
      chunk_st4(res + kRowBuf, t, e, a4);
    }
  }
}

// What bounds it: integer issue (64 % of cycles, the multiplier 68 % busy) and
// the latency of its loads, so occupancy decides.  Each digit's transformed
// row waits in shared memory and the inner product runs over four
// coefficients at a time, so that 64 registers suffice and four CTAs share an
// SM.  8 multiplications at level 22, one stream: 186 us.  Beside a form of it
// that took 198: with 64-bit accumulators of the whole row in registers (128,
// two CTAs) 235, with 32-bit ones (80 and spilled, three CTAs) 224; the 128 x
// 512 form before it 218 with three stages fewer.  Two digits per transform
// (sharing twiddles, 80 registers, three CTAs) 227; L2 prefetch of the key
// rows no gain.
//
// More than four digits (GROUPED) go through two row buffers in groups of two,
// the sums between groups in two more: 64 KiB and three CTAs whatever the
// digits, where a buffer per digit leaves two CTAs from five digits on and
// one at eight.  8 multiplications over 24 primes, 5 / 6 / 7 / 8 digits (7: 21
// primes): 563 / 601 / 599 / 718 us, with a buffer per digit 650 / 709 / 704 /
// 1247; one multiplication of 8 digits 125 and 189.  Groups of one at four
// CTAs 584 / 634 / 632 / 763, of three or four at two CTAs 596-621 / 633-661 /
// 640-644 / 769-778.
template <bool GROUPED>
__global__ void __launch_bounds__(kRowThreads, GROUPED ? 3 : 4) k_ks_rows(const __grid_constant__ KSRowsDesc d) {
  // one row buffer per digit (of a group), at least two; GROUPED: two more for the sums
  extern __shared__ __align__(16) uint32_t sm[];
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
  const int own = L.own_digit[j], beta = L.beta;
  const size_t off = row + chunk_off(t);  // input rows share the accumulator row index for q primes
  const size_t koff = static_cast<size_t>(L.key_row[j]) * 65536 + r * kRowLen + chunk_off(t);
  const int di = L.drop_idx[j];
  uint32_t *const res = GROUPED ? sm + kGroupDigits * kRowBuf : sm;
  grid_wait();
  for (int i0 = 0; i0 < (GROUPED ? beta : 1); i0 += kGroupDigits) {
    const int digits = GROUPED ? min(kGroupDigits, beta - i0) : beta;
    if (i0) __syncthreads();  // every thread is done with the rows of the group before
    // ---- ModUp NTT rows: each digit's row stays in its buffer
    for (int i = 0; i < digits; i++) {
      if (own == i0 + i) continue;
      const uint32_t *src = c.mu[i0 + i] + row;
      uint32_t v[1][16];
      uint32_t *bufs[1] = {sm + i * kRowBuf};
#pragma unroll
      for (int k = 0; k < 16; k++) v[0][k] = src[t + 256 * k];
      row_fwd_group<1>(v, false, bufs, tw, r, t, q);
#pragma unroll
      for (int k = 0; k < 16; k++) v[0][k] = reduce2q(v[0][k], q);
      group_st(bufs[0], t, v[0]);
    }
    __syncwarp();  // chunks are read back within the half-warp that wrote them
    // ---- inner product and P (d0, d1)
    switch (digits) {
      case 1: inner_product<1, GROUPED>(c, L, sm, res, i0, j, d.mode, off, koff, q, qi, t); break;
      case 2: inner_product<2, GROUPED>(c, L, sm, res, i0, j, d.mode, off, koff, q, qi, t); break;
      case 3:
        if (!GROUPED) inner_product<3, GROUPED>(c, L, sm, res, i0, j, d.mode, off, koff, q, qi, t);
        break;
      default:
        if (!GROUPED) inner_product<kWholeDigits, GROUPED>(c, L, sm, res, i0, j, d.mode, off, koff, q, qi, t);
        break;
    }
  }
  if (di < 0) return;
  // dropped prime: INTT row phase of both accumulators (ModDown's first step)
  const uint2 *itw = d.itw + (static_cast<size_t>(g) << 16);
  const size_t doff = static_cast<size_t>(di) * 65536 + r * kRowLen + t;
#pragma unroll 1
  for (int p = 0; p < 2; p++) {
    uint32_t x[1][16];
    uint32_t *bufs[1] = {res + p * kRowBuf};
    uint32_t *dst = (p == 0 ? c.drop_b : c.drop_a) + doff;
    row_inv_stored<1>(x, false, bufs, itw, r, t, q);
#pragma unroll
    for (int k = 0; k < 16; k++) dst[256 * k] = x[0][k];
  }
}

}  // namespace

void launch_ks_rows(const KSRowsDesc &d, int log_n, cudaStream_t s) {
  if (d.count <= 0 || d.max_rows <= 0 || log_n != 16) return;
  int digits = 2;
  for (int i = 0; i < d.nlv; i++) digits = d.lv[i].beta > digits ? d.lv[i].beta : digits;
  const dim3 grid(d.count, kLimbRows, d.max_rows);
  auto go = [&](auto *kern, int bufs) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bufs * kRowBuf * 4);
    launch_dependent(kern, grid, kRowThreads, bufs * kRowBuf * 4, s, d);
  };
  if (digits <= kWholeDigits)
    go(k_ks_rows<false>, digits);
  else
    go(k_ks_rows<true>, kGroupDigits + 2);
}

}  // namespace chd
