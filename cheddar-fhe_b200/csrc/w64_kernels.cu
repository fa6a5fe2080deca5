// Kernels of the 64-bit word path (w64.h), N = 2^16: the NTT in two passes
// (16-element columns, 4096-element rows, the layout and twiddle semantics of
// the 32-bit path), exact base conversion with 128-bit totals, tensor
// product, key inner product and the automorphism.  Lazy Shoup butterflies keep values in [0, 2q) (q < 2^62);
// Montgomery products use R = 2^64 as the reference's
// __mult_montgomery_lazy<uint64_t> (include/common/Basic.cuh:128-137).
#include "launch.cuh"
#include "w64.h"

namespace chd {
namespace w64 {
namespace {

__device__ __forceinline__ u64 shoup(u64 b, u64 w, u64 ws, u64 q) { return b * w - __umul64hi(b, ws) * q; }
__device__ __forceinline__ u64 red2q(u64 x, u64 q) { return x >= q ? x - q : x; }
__device__ __forceinline__ u64 add_mod(u64 a, u64 b, u64 q) { return red2q(a + b, q); }
// Montgomery reduction of a signed 128-bit value (|a| < q 2^63): a 2^-64 mod q
__device__ __forceinline__ u64 redc(i128 a, u64 q, i64 qinv) {
  const i64 lo = static_cast<i64>(a), hi = static_cast<i64>(a >> 64);
  const i64 t = lo * qinv;
  i64 r = hi - __mul64hi(t, static_cast<i64>(q));
  if (r < 0) r += static_cast<i64>(q);
  return static_cast<u64>(r);
}
__device__ __forceinline__ u64 mont_mul(u64 a, u64 b, u64 q, i64 qinv) {
  return redc(static_cast<i128>(static_cast<u128>(a) * b), q, qinv);
}
__device__ __forceinline__ i64 centre(u64 a, u64 q) {
  return a > (q >> 1) ? static_cast<i64>(a) - static_cast<i64>(q) : static_cast<i64>(a);
}

// butterflies on lazy [0, 2q) values
__device__ __forceinline__ void ct(u64 &a, u64 &b, ulonglong2 w, u64 q) {
  const u64 x = red2q(a, q);
  const u64 t = red2q(shoup(b, w.x, w.y, q), q);
  a = x + t;
  b = x - t + q;
}
__device__ __forceinline__ void gs(u64 &a, u64 &b, ulonglong2 w, u64 q) {
  const u64 x = red2q(a, q), y = red2q(b, q);
  a = x + y;
  b = shoup(x - y + q, w.x, w.y, q);
}

// NARROW butterflies (every prime below 2^58): a 64-bit word holds 64 q, and a
// Shoup product takes any word, so that values may grow.  Forward, a stage
// adds at most 2q: sixteen stages from [0, 2q) stay below 34 q with no
// reduction at all.  Inverse, the sums double: from [0, 2q) the four stages of
// a round reach 32 q in element 0 and less where a product came later
// (element j: 2q 2^(4 - bits of j)), and a round ends by bringing them back.
// ModUp and ModDown at level 25: 328 us with the two conditional subtractions
// per butterfly, 296 without.
__device__ __forceinline__ void ct_narrow(u64 &a, u64 &b, ulonglong2 w, u64 q) {
  const u64 t = shoup(b, w.x, w.y, q);
  b = a - t + 2 * q;
  a = a + t;
}
// y < off, a multiple of q
__device__ __forceinline__ void gs_narrow(u64 &a, u64 &b, ulonglong2 w, u64 q, u64 off) {
  const u64 d = a - b + off;
  a = a + b;
  b = shoup(d, w.x, w.y, q);
}
// [0, q 2^n) -> [0, q)
template <int n>
__device__ __forceinline__ u64 shrink(u64 x, u64 q) {
#pragma unroll
  for (int i = n - 1; i >= 0; i--) x = red2q(x, q << i);
  return x;
}

// Radix-16 networks on x[0..15] at register distances 8, 4, 2, 1 (forward) or
// 1, 2, 4, 8 (inverse); w(s, g) gives the twiddle of group g < 2^s of stage s.
// LAST: the inverse leaves its values as they are (below 32 q).
template <bool NARROW, class W>
__device__ __forceinline__ void r16_fwd(u64 *x, u64 q, W &&w) {
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const int m = 1 << s, h = 8 >> s;
#pragma unroll
    for (int g = 0; g < m; g++) {
      const ulonglong2 v = w(s, g);
#pragma unroll
      for (int j = 0; j < h; j++) {
        if (NARROW)
          ct_narrow(x[g * 2 * h + j], x[g * 2 * h + j + h], v, q);
        else
          ct(x[g * 2 * h + j], x[g * 2 * h + j + h], v, q);
      }
    }
  }
}
template <bool NARROW, bool LAST, class W>
__device__ __forceinline__ void r16_inv(u64 *x, u64 q, W &&w) {
#pragma unroll
  for (int s = 3; s >= 0; s--) {
    const int m = 1 << s, h = 8 >> s;
#pragma unroll
    for (int g = 0; g < m; g++) {
      const ulonglong2 v = w(s, g);
#pragma unroll
      for (int j = 0; j < h; j++) {
        if (NARROW)
          gs_narrow(x[g * 2 * h + j], x[g * 2 * h + j + h], v, q, q << (4 - s));
        else
          gs(x[g * 2 * h + j], x[g * 2 * h + j + h], v, q);
      }
    }
  }
  if (NARROW && !LAST) {
    x[0] = shrink<4>(x[0], 2 * q);
    x[1] = shrink<3>(x[1], 2 * q);
    x[2] = shrink<2>(x[2], 2 * q);
    x[3] = shrink<2>(x[3], 2 * q);
#pragma unroll
    for (int j = 4; j < 8; j++) x[j] = shrink<1>(x[j], 2 * q);
  }
}

// Layout (that of the 32-bit path, ntt_common.cuh): a limb is a 16 x 4096
// row-major matrix.  Stages m = 1 .. 8 act on columns of 16, one per thread;
// stages m = 16 .. 32768 on one row per CTA of 256 threads, 16 elements each,
// in three radix-16 rounds: across the row (one CTA barrier), then inside
// blocks of 256 elements owned by a half-warp.  The 128 x 512 form before it
// (seven column stages through shared memory, rows in three radix-8 rounds of
// two barriers each, 64-byte strides between a thread's 8-byte accesses) took
// 0.46 + 0.68 us per limb forward at 64 limbs, this one 0.21 + 0.69 at 106.
// The row kernels are bound by the 64-bit products' integer instructions; 80
// or 64 registers (three or four CTAs per SM) were 2 and 4 % slower than 128.
constexpr int kRow = 4096, kColThreads = 128;

struct TwGroup {  // pairs (B << s) + g
  const ulonglong2 *tw;
  unsigned B;
  __device__ __forceinline__ ulonglong2 operator()(int s, int g) const { return __ldg(tw + (B << s) + g); }
};
struct TwLast {  // last round of row r, thread t: stored chunk-major (tw_position64)
  const ulonglong2 *tw;
  int r, t;
  __device__ __forceinline__ ulonglong2 operator()(int s, int g) const {
    return __ldg(tw + (4096 << s) + (r << (8 + s)) + 256 * g + t);
  }
};

// Row buffer: element 256 b + 16 k + u.  Free of bank conflicts for 8-byte
// accesses with u the lane (a half-warp covers 16 consecutive words) and for
// 16-byte accesses to chunks u / 2 with k the lane.
__device__ __forceinline__ int pos64(int b, int k, int u) {
  return 256 * b + 16 * k + ((((u >> 1) ^ (k & 7)) << 1) | (u & 1));
}
__device__ __forceinline__ void group64_st(u64 *sm, int t, const u64 *x) {
#pragma unroll
  for (int i = 0; i < 8; i++)
    *reinterpret_cast<ulonglong2 *>(sm + pos64(t >> 4, t & 15, 2 * i)) = make_ulonglong2(x[2 * i], x[2 * i + 1]);
}
__device__ __forceinline__ void group64_ld(const u64 *sm, int t, u64 *x) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(sm + pos64(t >> 4, t & 15, 2 * i));
    x[2 * i] = v.x;
    x[2 * i + 1] = v.y;
  }
}

// forward column phase
template <bool NARROW>
__global__ void __launch_bounds__(kColThreads) k64_fwd_cols(const __grid_constant__ RowBatch64 rb) {
  const Row64 &rd = rb.rows[blockIdx.y];
  const u64 q = rd.q;
  const int c = blockIdx.x * kColThreads + threadIdx.x;
  grid_wait();
  u64 x[16];
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = rd.src[k * kRow + c];
  if (rd.flags & kPreMult) {
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = shoup(x[k], rd.c0, rd.c0s, q);
  }
  r16_fwd<NARROW>(x, q, TwGroup{rd.tw, 1});
#pragma unroll
  for (int k = 0; k < 16; k++) rd.dst[k * kRow + c] = x[k];
}

// forward row phase, canonical output, optional ModDown epilogue
// (src2 c1 - x) c2; global accesses are 8 bytes (the raw entry points promise
// no more), 128 contiguous bytes per half-warp
template <bool NARROW>
__global__ void __launch_bounds__(256, 2) k64_fwd_rows(const __grid_constant__ RowBatch64 rb) {
  __shared__ __align__(16) u64 sm[kRow];
  const Row64 &rd = rb.rows[blockIdx.y];
  const u64 q = rd.q;
  const int t = threadIdx.x, r = blockIdx.x, b = t >> 4, u = t & 15;
  u64 *dst = rd.dst + r * kRow;  // the column phase wrote dst
  grid_wait();
  u64 x[16];
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = dst[t + 256 * k];
  r16_fwd<NARROW>(x, q, TwGroup{rd.tw, 16u + r});
#pragma unroll
  for (int k = 0; k < 16; k++) sm[pos64(k, b, u)] = x[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = sm[pos64(b, k, u)];
  r16_fwd<NARROW>(x, q, TwGroup{rd.tw, 256u + 16u * r + b});
#pragma unroll
  for (int k = 0; k < 16; k++) sm[pos64(b, k, u)] = x[k];
  __syncwarp();
  group64_ld(sm, t, x);
  r16_fwd<NARROW>(x, q, TwLast{rd.tw, r, t});
  group64_st(sm, t, x);
  __syncwarp();
  const int base = 256 * b + u;
  if (rd.flags & kModDownEpi) {
    if (rd.flags & kHasSrc2) {
#pragma unroll
      for (int k = 0; k < 16; k++) x[k] = rd.src2[r * kRow + base + 16 * k];
      if (rd.flags & kPadSrc2) {
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = red2q(shoup(x[k], rd.c1, rd.c1s, q), q);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 16; k++) x[k] = 0;
    }
    const u64 c2 = rd.c2, c2s = rd.c2s;
#pragma unroll
    for (int k = 0; k < 16; k++)
      dst[base + 16 * k] = red2q(NARROW ? shoup(x[k] - sm[pos64(b, k, u)] + 34 * q, c2, c2s, q)
                                       : shoup(x[k] - red2q(sm[pos64(b, k, u)], q) + q, c2, c2s, q), q);
  } else {
#pragma unroll
    for (int k = 0; k < 16; k++)
      dst[base + 16 * k] = NARROW ? shrink<6>(sm[pos64(b, k, u)], q) : red2q(sm[pos64(b, k, u)], q);
  }
}

// inverse row phase (lazy output)
template <bool NARROW>
__global__ void __launch_bounds__(256, 2) k64_inv_rows(const __grid_constant__ RowBatch64 rb) {
  __shared__ __align__(16) u64 sm[kRow];
  const Row64 &rd = rb.rows[blockIdx.y];
  const u64 q = rd.q;
  const int t = threadIdx.x, r = blockIdx.x, b = t >> 4, u = t & 15;
  const u64 *src = rd.src + r * kRow + 256 * b + u;
  grid_wait();
  u64 x[16];
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = src[16 * k];
#pragma unroll
  for (int k = 0; k < 16; k++) sm[pos64(b, k, u)] = x[k];
  __syncwarp();
  group64_ld(sm, t, x);
  r16_inv<NARROW, false>(x, q, TwLast{rd.tw, r, t});
  group64_st(sm, t, x);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = sm[pos64(b, k, u)];
  r16_inv<NARROW, false>(x, q, TwGroup{rd.tw, 256u + 16u * r + b});
#pragma unroll
  for (int k = 0; k < 16; k++) sm[pos64(b, k, u)] = x[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = sm[pos64(k, b, u)];
  r16_inv<NARROW, false>(x, q, TwGroup{rd.tw, 16u + r});
  u64 *dst = rd.dst + r * kRow;
#pragma unroll
  for (int k = 0; k < 16; k++) dst[t + 256 * k] = x[k];
}

// inverse column phase, then x c0, canonical or centred
template <bool NARROW>
__global__ void __launch_bounds__(kColThreads) k64_inv_cols(const __grid_constant__ RowBatch64 rb) {
  const Row64 &rd = rb.rows[blockIdx.y];
  const u64 q = rd.q;
  u64 *p = rd.dst + blockIdx.x * kColThreads + threadIdx.x;
  grid_wait();
  u64 x[16];
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = p[k * kRow];
  r16_inv<NARROW, true>(x, q, TwGroup{rd.tw, 1});
  const bool centre_out = (rd.flags & kCentre) != 0;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    u64 v = red2q(shoup(x[k], rd.c0, rd.c0s, q), q);
    if (centre_out) v = static_cast<u64>(centre(v, q));
    p[k * kRow] = v;
  }
}

// Base conversion: a thread loads its coefficient's K sources once and
// produces every target; the table and the targets' primes sit in shared
// memory.  KMAX >= K bounds the unrolled loops.
//
// NARROW (every prime of the context below 2^58): sources offset by 2^57 and
// table words taken plain are 58-bit numbers, split into 29-bit halves whose
// products need no carries: the sums of up to 16 low, crossed and high
// products stay below 2^62, 2^63 and 2^62, so that a term is four wide
// multiply-adds instead of a signed 128-bit product and its carry chain.  The
// total is below 16 2^58 p, inside the reduction's window p 2^63; the offset
// is taken back through corr = -2^57 sum_k T mod p.  104 + 50 outputs of 7
// and 8 sources (ModUp and ModDown at level 25): 72 + 48 us with 128-bit
// sums, 59 + 41 now; bound by the multiplier.
template <int KMAX, bool NARROW>
__global__ void __launch_bounds__(256) k64_bconv(const __grid_constant__ BConv64Batch b) {
  __shared__ u64 tab[64 * 16];  // NARROW: low half in the low word, high half in the high word
  __shared__ u64 sp[64], corr[64];
  __shared__ i64 sq[64];
  const BConv64Job &j = b.jobs[blockIdx.y];
  const int K = j.K, M = j.M;
  for (int t = threadIdx.x; t < M * K; t += blockDim.x) {
    u64 v = static_cast<u64>(j.table[t]);
    if (NARROW) {
      if (static_cast<i64>(v) < 0) v += b.primes[j.out_gidx[t / K]];
      v = (v & 0x1fffffffu) | ((v >> 29) << 32);
    }
    tab[t] = v;
  }
  for (int t = threadIdx.x; t < M; t += blockDim.x) {
    const u64 p = b.primes[j.out_gidx[t]];
    sp[t] = p;
    sq[t] = b.qinvs[j.out_gidx[t]];
    if (NARROW) {
      u64 c = 0;
      for (int k = 0; k < K; k++) {
        const i64 v = j.table[t * K + k];
        c = add_mod(c, v < 0 ? static_cast<u64>(v) + p : static_cast<u64>(v), p);
      }
      for (int k = 0; k < 57; k++) c = add_mod(c, c, p);
      corr[t] = c ? p - c : 0;
    }
  }
  grid_wait();
  __syncthreads();
  if (NARROW) {
    // two coefficients, i and i + 32768, share the table reads
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t x0[2][KMAX], x1[2][KMAX];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int k = 0; k < KMAX; k++) {
        const u64 v = k < K ? static_cast<u64>(j.xt[(static_cast<size_t>(k) << 16) + i + (h << 15)] + (1ll << 57)) : 0;
        x0[h][k] = static_cast<uint32_t>(v) & 0x1fffffffu;
        x1[h][k] = static_cast<uint32_t>(v >> 29);
      }
    for (int m = 0; m < M; m++) {
      const uint2 *tm = reinterpret_cast<const uint2 *>(tab + m * K);
      u64 s0[2] = {0, 0}, s1[2] = {0, 0}, s2[2] = {0, 0};
#pragma unroll
      for (int k = 0; k < KMAX; k++)
        if (k < K) {
          const uint2 c = tm[k];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            s0[h] += static_cast<u64>(x0[h][k]) * c.x;
            s1[h] += static_cast<u64>(x0[h][k]) * c.y;
            s1[h] += static_cast<u64>(x1[h][k]) * c.x;
            s2[h] += static_cast<u64>(x1[h][k]) * c.y;
          }
        }
      const u64 p = sp[m], cr = corr[m];
      const u64 pinv = static_cast<u64>(sq[m]);
      u64 *out = j.out + (static_cast<size_t>(j.out_row[m]) << 16) + i;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const u128 v = static_cast<u128>(s0[h]) + cr + (static_cast<u128>(s1[h]) << 29) + (static_cast<u128>(s2[h]) << 58);
        // v < p 2^62 and not negative: hi(v) - hi(m p) with m = lo(v) p^-1 is in (-p, p)
        const u64 r = static_cast<u64>(v >> 64) - __umul64hi(static_cast<u64>(v) * pinv, p);
        out[h << 15] = static_cast<i64>(r) < 0 ? r + p : r;
      }
    }
  } else {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    i64 x[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; k++) x[k] = k < K ? j.xt[(static_cast<size_t>(k) << 16) + i] : 0;
    for (int m = 0; m < M; m++) {
      const i64 *tm = reinterpret_cast<const i64 *>(tab) + m * K;
      i128 acc = 0;
#pragma unroll
      for (int k = 0; k < KMAX; k++)
        if (k < K) acc += static_cast<i128>(x[k]) * tm[k];
      j.out[(static_cast<size_t>(j.out_row[m]) << 16) + i] = redc(acc, sp[m], sq[m]);
    }
  }
}

__global__ void __launch_bounds__(256) k64_tensor(const __grid_constant__ Elem64Batch b) {
  const Elem64Row &e = b.rows[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  grid_wait();
  const u64 b1 = e.b1[i], a1 = e.a1[i], b2 = e.b2[i], a2 = e.a2[i];
  e.o0[i] = mont_mul(b1, b2, e.q, e.qinv);
  e.o1[i] = add_mod(mont_mul(b1, a2, e.q, e.qinv), mont_mul(a1, b2, e.q, e.qinv), e.q);
  e.o2[i] = mont_mul(a1, a2, e.q, e.qinv);
}

__global__ void __launch_bounds__(256) k64_add(const __grid_constant__ Elem64Batch b) {
  const Elem64Row &e = b.rows[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  grid_wait();
  e.o0[i] = add_mod(e.a1[i], e.b1[i], e.q);
}

template <Elem64Op OP>
__global__ void __launch_bounds__(256) k64_elem(const __grid_constant__ Elem64Batch b) {
  const Elem64Row &e = b.rows[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  grid_wait();
  const u64 q = e.q, x = e.a1[i];
  u64 o;
  switch (OP) {
    case Elem64Op::kAdd: o = add_mod(x, e.b1[i], q); break;
    case Elem64Op::kSub: o = red2q(x + q - e.b1[i], q); break;
    case Elem64Op::kNeg: o = x ? q - x : 0; break;
    case Elem64Op::kMult: o = mont_mul(x, e.b1[i], q, e.qinv); break;
    case Elem64Op::kMultConst: o = mont_mul(x, e.c, q, e.qinv); break;
    case Elem64Op::kAddConst: o = add_mod(x, e.c, q); break;
    case Elem64Op::kCopy: o = x; break;
    case Elem64Op::kMultImagUnit: o = mont_mul(x, (i & 32768) ? q - e.c : e.c, q, e.qinv); break;
  }
  e.o0[i] = o;
}

__device__ __forceinline__ uint32_t brev17(uint32_t x) { return __brev(x) >> 15; }

__global__ void __launch_bounds__(256) k64_permute(const __grid_constant__ Elem64Batch b, u64 galois) {
  const Elem64Row &e = b.rows[blockIdx.y];
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  grid_wait();
  const uint32_t ex = (brev17(k) + 1u) * static_cast<uint32_t>(galois) - 1u;
  const uint32_t src = brev17(ex & ((1u << 17) - 1u));
  e.o0[k] = e.a1[src];
}

__global__ void __launch_bounds__(256) k64_key_mac(const __grid_constant__ KeyMac64Batch b) {
  const KeyMac64Row &r = b.rows[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  grid_wait();
  const u64 q = r.q;
  u64 sb = 0, sa = 0;
  for (int d = 0; d < r.beta; d++) {
    const u64 v = r.mu[d][i];
    sb = add_mod(sb, mont_mul(v, r.kb[d][i], q, r.qinv), q);
    sa = add_mod(sa, mont_mul(v, r.ka[d][i], q, r.qinv), q);
  }
  if (r.d0) sb = add_mod(sb, mont_mul(r.d0[i], r.p, q, r.qinv), q);
  if (r.d1) sa = add_mod(sa, mont_mul(r.d1[i], r.p, q, r.qinv), q);
  r.acc_b[i] = sb;
  r.acc_a[i] = sa;
}

}  // namespace

namespace {
template <bool NARROW>
void ntt64(const RowBatch64 &rb, bool fwd, cudaStream_t s) {
  const dim3 cols(kRow / kColThreads, rb.count), rows(16, rb.count);
  if (fwd) {
    launch_dependent(k64_fwd_cols<NARROW>, cols, kColThreads, 0, s, rb);
    launch_dependent(k64_fwd_rows<NARROW>, rows, 256, 0, s, rb);
  } else {
    launch_dependent(k64_inv_rows<NARROW>, rows, 256, 0, s, rb);
    launch_dependent(k64_inv_cols<NARROW>, cols, kColThreads, 0, s, rb);
  }
}
void ntt64(const RowBatch64 &rb, bool fwd, cudaStream_t s) {
  if (rb.count <= 0) return;
  // the words' headroom decides, prime by prime of the launch
  bool narrow = true;
  for (int i = 0; i < rb.count; i++) narrow = narrow && rb.rows[i].q < (1ull << 58);
  if (narrow)
    ntt64<true>(rb, fwd, s);
  else
    ntt64<false>(rb, fwd, s);
}
}  // namespace

void launch_ntt64_fwd(const RowBatch64 &rb, cudaStream_t s) { ntt64(rb, true, s); }

void launch_ntt64_inv(const RowBatch64 &rb, cudaStream_t s) { ntt64(rb, false, s); }

void launch_bconv64(const BConv64Batch &b, cudaStream_t s) {
  if (b.count <= 0) return;
  int max_k = 0;
  for (int j = 0; j < b.count; j++) max_k = b.jobs[j].K > max_k ? b.jobs[j].K : max_k;
  if (!b.narrow)
    launch_dependent(k64_bconv<16, false>, dim3(65536 / 256, b.count), 256, 0, s, b);
  else if (max_k <= 8)
    launch_dependent(k64_bconv<8, true>, dim3(32768 / 128, b.count), 128, 0, s, b);
  else
    launch_dependent(k64_bconv<16, true>, dim3(32768 / 128, b.count), 128, 0, s, b);
}

void launch_tensor64(const Elem64Batch &b, cudaStream_t s) {
  if (b.count <= 0) return;
  launch_dependent(k64_tensor, dim3(65536 / 256, b.count), 256, 0, s, b);
}

void launch_add64(const Elem64Batch &b, cudaStream_t s) {
  if (b.count <= 0) return;
  launch_dependent(k64_add, dim3(65536 / 256, b.count), 256, 0, s, b);
}

void launch_elem64(Elem64Op op, const Elem64Batch &b, cudaStream_t s) {
  if (b.count <= 0) return;
  const dim3 grid(65536 / 256, b.count);
  switch (op) {
    case Elem64Op::kAdd: launch_dependent(k64_elem<Elem64Op::kAdd>, grid, 256, 0, s, b); break;
    case Elem64Op::kSub: launch_dependent(k64_elem<Elem64Op::kSub>, grid, 256, 0, s, b); break;
    case Elem64Op::kNeg: launch_dependent(k64_elem<Elem64Op::kNeg>, grid, 256, 0, s, b); break;
    case Elem64Op::kMult: launch_dependent(k64_elem<Elem64Op::kMult>, grid, 256, 0, s, b); break;
    case Elem64Op::kMultConst: launch_dependent(k64_elem<Elem64Op::kMultConst>, grid, 256, 0, s, b); break;
    case Elem64Op::kAddConst: launch_dependent(k64_elem<Elem64Op::kAddConst>, grid, 256, 0, s, b); break;
    case Elem64Op::kCopy: launch_dependent(k64_elem<Elem64Op::kCopy>, grid, 256, 0, s, b); break;
    case Elem64Op::kMultImagUnit: launch_dependent(k64_elem<Elem64Op::kMultImagUnit>, grid, 256, 0, s, b); break;
  }
}

void launch_permute64(const Elem64Batch &b, u64 galois, cudaStream_t s) {
  if (b.count <= 0) return;
  launch_dependent(k64_permute, dim3(65536 / 256, b.count), 256, 0, s, b, galois);
}

void launch_key_mac64(const KeyMac64Batch &b, cudaStream_t s) {
  if (b.count <= 0) return;
  launch_dependent(k64_key_mac, dim3(65536 / 256, b.count), 256, 0, s, b);
}

}  // namespace w64
}  // namespace chd
