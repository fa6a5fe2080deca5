// Negacyclic NTT / INTT kernels.
//
// Transform semantics (what every kernel here must reproduce exactly): the
// forward transform of a limb a (natural order) is
//     A[k] = sum_i a_i * psi^((2 brev(k) + 1) i)  mod q,
// stored bit-reversed, with psi the primitive 2N-th root derived from the
// smallest generator of Z_q^* and twiddles psi_rev[j] = psi^brev(j)
// (src/core/NTT.cu:1233-1299 and include/common/PrimeUtils.h:135-196 of the
// reference).  Stage m of the Cooley-Tukey network pairs index j with
// j + N/(2m) using twiddle psi_rev[m + floor(j m / N)]; the inverse runs the
// Gentleman-Sande network with psi^-1.  All arithmetic is exact mod q: values
// travel lazily in [0, 2q) between stages (Shoup products, arith.cuh) and are
// reduced to [0, q) on output, so every output word is the canonical residue.
//
// Layout for N = 2^16: the limb is a 16 x 4096 row-major matrix
// (ntt_common.cuh).  Stages m = 1..8 only pair elements of the same column
// (one thread per column, no exchange); stages m = 16..32768 stay inside one
// 4096-element row (one CTA per row, three radix-16 rounds exchanged through
// shared memory).  The inverse runs rows first, then columns, and fuses the
// per-limb output constant and the optional centring into the column phase.  For N <= 2^15 the whole limb
// fits in shared memory and one kernel runs every stage.
#include <atomic>
#include <type_traits>

#include "arith.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "ntt_common.cuh"

namespace chd {
namespace {

constexpr int kColThreads = 128;  // columns per CTA of the column phases

// ---------------------------------------------------------------- N = 2^16
// Column phase of the forward transform: stages m = 1 .. 8, one column of 16
// elements per thread.
template <class RB>
__global__ void __launch_bounds__(kColThreads) k_fwd_cols16(const __grid_constant__ RB rb) {
  const RowDesc &rd = rb.rows[blockIdx.y];
  const uint32_t q = rd.q;
  const int c = blockIdx.x * kColThreads + threadIdx.x;
  uint32_t x[16];
  uint2 w[16];
  tw_radix16(rd.tw, 1, w);
  grid_wait();
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = rd.src[k * kRowLen + c];
  if (rd.flags & kPreMult) {
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = shoup_lazy(x[k], rd.c0, rd.c0s, q);
  }
  radix16_fwd(x, w, q);
#pragma unroll
  for (int k = 0; k < 16; k++) rd.dst[k * kRowLen + c] = x[k];  // lazy [0, 2q)
}

// Row phase of the forward transform (input lazy from the column phase),
// canonical output, with the optional ModDown epilogue (src2 * c1 - x) * c2.
// A CTA takes one row of one or (P = 2) two limbs of a prime.
template <int P, int MINB, class RB>
__global__ void __launch_bounds__(kRowThreads, MINB) k_fwd_rows16(const __grid_constant__ RB rb) {
  __shared__ __align__(16) uint32_t sm[P][kRowBuf];
  const int first = P == 1 ? blockIdx.y : rb.first[blockIdx.y];
  const bool two = P > 1 && rb.first[blockIdx.y + 1] - first > 1;
  const uint32_t q = rb.rows[first].q;
  const int t = threadIdx.x, r = blockIdx.x;
  uint32_t x[P][16];
  uint32_t *bufs[P];
  grid_wait();
#pragma unroll
  for (int p = 0; p < P; p++) {
    bufs[p] = sm[p];
    if (p == 0 || two) {
      const uint32_t *src = rb.rows[first + p].dst + r * kRowLen;  // the column phase wrote dst
#pragma unroll
      for (int k = 0; k < 16; k++) x[p][k] = src[t + 256 * k];
    }
  }
  row_fwd_group<P>(x, two, bufs, rb.rows[first].tw, r, t, q);
#pragma unroll
  for (int p = 0; p < P; p++)
    if (p == 0 || two) {
#pragma unroll
      for (int k = 0; k < 16; k++) x[p][k] = reduce2q(x[p][k], q);
      group_st(bufs[p], t, x[p]);
    }
  __syncwarp();
  const unsigned base = r * kRowLen + chunk_off(t);
#pragma unroll
  for (int p = 0; p < P; p++)
    if (p == 0 || two) {
      const RowDesc &rd = rb.rows[first + p];
      uint32_t y[16];
      chunk_ld(bufs[p], t, y);
      if (rd.flags & kModDownEpi) {
        uint32_t v[16];
        if (rd.flags & kHasSrc2) {
          ld_chunks(rd.src2 + base, v);
          if (rd.flags & kPadSrc2) {
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = reduce2q(shoup_lazy(v[k], rd.c1, rd.c1s, q), q);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 16; k++) v[k] = 0;
        }
#pragma unroll
        for (int k = 0; k < 16; k++) y[k] = reduce2q(shoup_lazy(v[k] - y[k] + q, rd.c2, rd.c2s, q), q);
      }
      st_chunks(rd.dst + base, y);
    }
}

// Inverse, row phase: Gentleman-Sande stages m = 32768 .. 16 (lazy output).
template <int P, int MINB, class RB>
__global__ void __launch_bounds__(kRowThreads, MINB) k_inv_rows16(const __grid_constant__ RB rb) {
  __shared__ __align__(16) uint32_t sm[P][kRowBuf];
  const int first = P == 1 ? blockIdx.y : rb.first[blockIdx.y];
  const bool two = P > 1 && rb.first[blockIdx.y + 1] - first > 1;
  const uint32_t q = rb.rows[first].q;
  const int t = threadIdx.x, r = blockIdx.x;
  const unsigned base = r * kRowLen + chunk_off(t);
  uint32_t x[P][16];
  uint32_t *bufs[P];
  grid_wait();
#pragma unroll
  for (int p = 0; p < P; p++) {
    bufs[p] = sm[p];
    if (p == 0 || two) ld_chunks(rb.rows[first + p].src + base, x[p]);
  }
#pragma unroll
  for (int p = 0; p < P; p++)
    if (p == 0 || two) {
      const RowDesc &rd = rb.rows[first + p];
      if (rd.flags & kMulSrc2) {
        uint32_t y[16];
        ld_chunks(rd.src2 + base, y);
#pragma unroll
        for (int k = 0; k < 16; k++) x[p][k] = mont_mul(x[p][k], y[k], q, rd.qinv);
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
        chunk_st4(bufs[p], t, i, make_uint4(x[p][4 * i], x[p][4 * i + 1], x[p][4 * i + 2], x[p][4 * i + 3]));
    }
  row_inv_stored<P>(x, two, bufs, rb.rows[first].tw, r, t, q);
#pragma unroll
  for (int p = 0; p < P; p++)
    if (p == 0 || two) {
      uint32_t *dst = rb.rows[first + p].dst + r * kRowLen;
#pragma unroll
      for (int k = 0; k < 16; k++) dst[t + 256 * k] = x[p][k];
    }
}

// Inverse, column phase: stages m = 8 .. 1, then x * c0, canonical or centred.
template <class RB>
__global__ void __launch_bounds__(kColThreads) k_inv_cols16(const __grid_constant__ RB rb) {
  const RowDesc &rd = rb.rows[blockIdx.y];
  const uint32_t q = rd.q;
  const int c = blockIdx.x * kColThreads + threadIdx.x;
  uint32_t *p = rd.dst;  // the row phase wrote dst
  uint32_t x[16];
  uint2 w[16];
  tw_radix16(rd.tw, 1, w);
  grid_wait();
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = p[k * kRowLen + c];
  radix16_inv(x, w, q);
  const bool centre_out = (rd.flags & kCentre) != 0;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    uint32_t v = reduce2q(shoup_lazy(x[k], rd.c0, rd.c0s, q), q);
    if (centre_out) v = static_cast<uint32_t>(centre(v, q));
    p[k * kRowLen + c] = v;
  }
}

// ------------------------------------------------------------ N <= 2^15
// Whole limb in shared memory, one CTA per limb.
template <bool kFwd>
__global__ void __launch_bounds__(1024) k_small(const __grid_constant__ RowBatch rb, int log_n) {
  extern __shared__ uint32_t sa[];
  const RowDesc &rd = rb.rows[blockIdx.x];
  const uint32_t q = rd.q;
  const uint2 *tw = rd.tw;
  const int n = 1 << log_n, half = n >> 1;
  grid_wait();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    uint32_t v = rd.src[i];
    if (kFwd && (rd.flags & kPreMult)) v = shoup_lazy(v, rd.c0, rd.c0s, q);
    sa[i] = v;
  }
  __syncthreads();
  if (kFwd) {
    for (int m = 1, lt = log_n - 1; m < n; m <<= 1, lt--) {
      const int t = 1 << lt;
      for (int b = threadIdx.x; b < half; b += blockDim.x) {
        const int i = b >> lt, j = 2 * i * t + (b & (t - 1));
        ct_lazy(sa[j], sa[j + t], __ldg(tw + m + i), q);
      }
      __syncthreads();
    }
  } else {
    for (int m = half, lt = 0; m >= 1; m >>= 1, lt++) {
      const int t = 1 << lt;
      for (int b = threadIdx.x; b < half; b += blockDim.x) {
        const int i = b >> lt, j = 2 * i * t + (b & (t - 1));
        gs_lazy(sa[j], sa[j + t], __ldg(tw + m + i), q);
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    uint32_t x = reduce2q(sa[i], q);
    if (kFwd) {
      if (rd.flags & kModDownEpi) {
        uint32_t v = 0;
        if (rd.flags & kHasSrc2) {
          v = rd.src2[i];
          if (rd.flags & kPadSrc2) v = reduce2q(shoup_lazy(v, rd.c1, rd.c1s, q), q);
        }
        x = reduce2q(shoup_lazy(v - x + q, rd.c2, rd.c2s, q), q);
      }
    } else {
      x = reduce2q(shoup_lazy(x, rd.c0, rd.c0s, q), q);
      if (rd.flags & kCentre) x = static_cast<uint32_t>(centre(x, q));
    }
    rd.dst[i] = x;
  }
}

}  // namespace

namespace {
// go(batch), in a smaller batch when the rows are few (`first` stays unset:
// only launches of pairs, which are large, read it)
template <class F>
void with_rows(const RowBatch &rb, F &&go) {
  if (rb.count > kFewRows) {
    go(rb);
    return;
  }
  RowBatchOf<kFewRows> few;
  few.count = rb.count;
  for (int i = 0; i < rb.count; i++) few.rows[i] = rb.rows[i];
  go(few);
}
}  // namespace

void launch_ntt_fwd_cols(const RowBatch &rb, int log_n, cudaStream_t s) {
  if (rb.count <= 0) return;
  with_rows(rb, [&](const auto &b) {
    launch_dependent(k_fwd_cols16<std::decay_t<decltype(b)>>, dim3(kRowLen / kColThreads, b.count), kColThreads, 0, s, b);
  });
}

namespace {
int device_sms() {
  constexpr int kDevices = 64;
  static std::atomic<int> cached[kDevices];
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= kDevices) dev = 0;
  sms = cached[dev].load(std::memory_order_relaxed);
  if (sms == 0 && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) cached[dev] = sms;
  return sms;
}

// Neighbouring limbs of one prime share a CTA: rb.first receives the first
// limb of each group of one or two; returns the number of groups, or 0 where
// single rows are to be taken.  Pairs of rows run at 3 CTAs per SM (80
// registers), single rows at 4 (64): pairs read half the twiddles, but half
// as many CTAs leave SMs idle in small launches (one multiplication at level
// 22, 23 pairs: 102.8 us against 100.7; one launch of 48 pairs, 4 inverse
// transforms of 24 primes: 26.6 against 25.7), so pairs are taken where they
// fill two waves.  Two launches that alternate between streams fill them
// together (beside = 2): 55 and 48 pairs a launch, forward and inverse
// transforms of 32 and of 16 polynomials of 24 primes, 180 + 185 us in pairs
// and 196 + 193 in single rows, 90 + 88 and 96 + 95.
int pair_rows(RowBatch &rb, int beside) {
  int groups = 0;
  for (int i = 0; i < rb.count; groups++) {
    rb.first[groups] = static_cast<uint16_t>(i);
    i += i + 1 < rb.count && rb.rows[i + 1].tw == rb.rows[i].tw ? 2 : 1;
  }
  rb.first[groups] = static_cast<uint16_t>(rb.count);
  if (groups == rb.count) return 0;
  return groups * kLimbRows * beside < 2 * 3 * device_sms() ? 0 : groups;
}
}  // namespace

void launch_ntt_fwd_rows(RowBatch &rb, int log_n, cudaStream_t s, int beside) {
  if (rb.count <= 0) return;
  const int groups = pair_rows(rb, beside);
  if (!groups)
    with_rows(rb, [&](const auto &b) {
      launch_dependent(k_fwd_rows16<1, 4, std::decay_t<decltype(b)>>, dim3(kLimbRows, b.count), kRowThreads, 0, s, b);
    });
  else
    launch_dependent(k_fwd_rows16<2, 3, RowBatch>, dim3(kLimbRows, groups), kRowThreads, 0, s, rb);
}

void launch_ntt_fwd(RowBatch &rb, int log_n, cudaStream_t s, int beside) {
  if (rb.count <= 0) return;
  if (log_n == 16) {
    launch_ntt_fwd_cols(rb, log_n, s);
    launch_ntt_fwd_rows(rb, log_n, s, beside);
  } else {
    size_t smem = sizeof(uint32_t) << log_n;
    cudaFuncSetAttribute(k_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    launch_dependent(k_small<true>, rb.count, 1024, smem, s, rb, log_n);
  }
}

void launch_ntt_inv_rows(RowBatch &rb, int log_n, cudaStream_t s, int beside) {
  if (rb.count <= 0) return;
  const int groups = pair_rows(rb, beside);
  if (!groups)
    with_rows(rb, [&](const auto &b) {
      launch_dependent(k_inv_rows16<1, 4, std::decay_t<decltype(b)>>, dim3(kLimbRows, b.count), kRowThreads, 0, s, b);
    });
  else
    launch_dependent(k_inv_rows16<2, 3, RowBatch>, dim3(kLimbRows, groups), kRowThreads, 0, s, rb);
}

void launch_ntt_inv(RowBatch &rb, int log_n, cudaStream_t s, int beside) {
  if (rb.count <= 0) return;
  if (log_n == 16) {
    launch_ntt_inv_rows(rb, log_n, s, beside);
    with_rows(rb, [&](const auto &b) {
      launch_dependent(k_inv_cols16<std::decay_t<decltype(b)>>, dim3(kRowLen / kColThreads, b.count), kColThreads, 0, s,
                       b);
    });
  } else {
    size_t smem = sizeof(uint32_t) << log_n;
    cudaFuncSetAttribute(k_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    launch_dependent(k_small<false>, rb.count, 1024, smem, s, rb, log_n);
  }
}

}  // namespace chd
