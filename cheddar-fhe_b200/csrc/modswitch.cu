// Fused ModSwitch column kernel for N = 2^16.
//
// ModUp and ModDown (src/core/ModSwitch.cu:429-684 of the reference) are
//   INTT(sources) * (N q-hat_k)^-1 (centred)  ->  BConv  ->  NTT(targets).
// With the 16 x 4096 limb layout (ntt_common.cuh) the INTT's last four
// stages, the base conversion and the NTT's first four stages all act on the
// same column of 16 elements, so a thread takes a column through all three
// in registers.  The row phases before (INTT) and after (NTT, with the
// ModDown epilogue) stay in ntt.cu and keyswitch.cu.
//
// The base conversion
//   V[m][n] = sum_k x_k[n] T[m][k]   (x centred, T the centred table)
// runs as byte-limb MMAs (exact in int32):
//   * the sources are offset, x' = x + 2^30 in [0, 2^31), so that their four
//     bytes are plain unsigned digits (A operand, u8);
//   * B holds the bytes of c[m][k][j] = 2^(8j) T[m][k] mod p_m (u8): K byte
//     4k + j pairs with byte j of x'_k, column (m, i) is byte i of c;
//   * D[n][(m, i)] = sum_(k, j) byte_j(x'_k) byte_i(c[m][k][j]) + byte i of
//     corr_m < 2^23, and sum_i 2^(8i) D[n][(m, i)] (< 2^48) with
//     corr_m = -2^30 sum_k T[m][k] mod p_m is congruent to V[m][n].
// One Montgomery reduction then gives a residue of V 2^-32 mod p_m.
//
// The MMA is the warp-level m16n8k32 / m16n8k16: its A fragment gives lane
// (g, tq) of a warp (g = lane / 4, tq = lane % 4) the four bytes 4 tq .. of
// rows g and g + 8, which is exactly one source word per register, and its
// accumulator gives the lane columns 2 tq, 2 tq + 1 of those rows.  So a
// warp takes 8 columns of the limb; lane (g, tq) transforms sources
// tq, tq + 4, ... of column g, pairs of its 16 elements are the two rows of
// one MMA, and with the B columns ordered (bytes 0, 1 of four targets), then
// (bytes 2, 3), the lane ends up with all four byte sums of target tq for
// column g: the layout its forward transform needs.  No shared memory, no
// barrier and no exchange between the sources' loads and the targets'
// stores; warps are independent.
//
// Why not tcgen05 here: its operands go through shared memory and TMEM, and
// an M = 128 tile ties four warps together at every chunk of targets.  The
// contraction is 4 K <= 64 bytes deep, 2 % of the tensor pipe either way;
// the pass is bound by the integer multiplies of the butterflies (8 of the
// 9.2 cycles a warp needs per butterfly), and what it needs is warps that
// never wait for one another.
#include <type_traits>

#include "arith.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "ntt_common.cuh"

namespace chd {
namespace {

constexpr int32_t kOffset = 1 << 30;  // makes centred sources non-negative
constexpr int kColWarps = 4;          // warps per CTA
constexpr int kCtaCols = 8 * kColWarps;

__device__ __forceinline__ void mma_k32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_k16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

// byte sums -> a value in [0, 2p) congruent to (sum_i 2^(8i) d_i) 2^-32
__device__ __forceinline__ uint32_t join(int d0, int d1, int d2, int d3, uint32_t p, int32_t pinv) {
  const uint32_t lo = static_cast<uint32_t>(d0) + (static_cast<uint32_t>(d1) << 8);
  const uint32_t hi = static_cast<uint32_t>(d2) + (static_cast<uint32_t>(d3) << 8);
  const uint64_t val = (static_cast<uint64_t>(hi) << 16) + lo;
  return static_cast<uint32_t>(mont_reduce_lazy(static_cast<int64_t>(val), p, pinv)) + p;
}

// KR: source rounds (sources tq + 4 i, i < KR; K <= 4 KR).  MINB CTAs per SM
// (72, 80, 96 and 128 registers for KR = 1 .. 4, a few words spilled):
// left alone the compiler takes 134 to 188, and the batch of 8 below slows
// to 96 / 74 us; one step tighter spills and gives 94 / 76 us.
//
// Measured, 8 multiplications at level 22 on one stream: ModUp (24 jobs of
// 8 sources and 24 targets) 82 us, ModDown + Rescale (16 jobs of 9 and 23)
// 68 us; the 128 x 512 tcgen05 pass before it took 172 and 141 us.
template <int KR, int MINB, class B>
__global__ void __launch_bounds__(32 * kColWarps, MINB) k_modswitch_cols(const __grid_constant__ B b) {
  const MSColJob &jb = b.jobs[blockIdx.y];
  const int lane = threadIdx.x & 31, tq = lane & 3;
  const int col = (blockIdx.x * kColWarps + (threadIdx.x >> 5)) * 8 + (lane >> 2);
  const int K = jb.K, M = jb.M;
  const int steps = (K + 7) / 8;  // K steps of 8 sources in the fragment table
  const int groups = (M + 3) / 4;
  // Staged in shared memory, before the wait for the kernel in front: what
  // every warp of the CTA would otherwise fetch for itself, at four cache
  // lines per access (the lanes of a quad need four different primes) and in
  // chains of dependent loads.
  //   tws, tws_dst: the fifteen twiddles of every source and target prime (the
  //     column stages use the first sixteen table entries), [group of four
  //     primes][pair of entries][prime], 64 contiguous bytes per access;
  //   prm: prime, inverse and destination row of every target;
  //   frg: the B fragments.
  extern __shared__ uint4 tws[];
  uint4 *const tws_dst = tws + 32 * KR, *const prm = tws_dst + 32 * groups, *const frg = prm + 4 * groups;
  for (int i = threadIdx.x; i < 8 * (K + M); i += 32 * kColWarps) {
    const int k = i >> 3, c = i & 7;
    const bool src = k < K;
    const int g = src ? jb.src_gidx[k] : jb.dst_gidx[k - K], x = src ? k : k - K;
    const uint2 *tab = (src ? b.itw : b.tw) + (static_cast<size_t>(g) << 16);
    (src ? tws : tws_dst)[32 * (x >> 2) + 4 * c + (x & 3)] = __ldg(reinterpret_cast<const uint4 *>(tab) + c);
  }
  for (int m = threadIdx.x; m < M; m += 32 * kColWarps) {
    const int g = jb.dst_gidx[m];
    prm[m] = make_uint4(__ldg(b.primes + g), static_cast<uint32_t>(__ldg(b.qinvs + g)), jb.dst_row[m], 0);
  }
  for (int i = threadIdx.x; i < 32 * groups * (steps + 1); i += 32 * kColWarps) frg[i] = __ldg(jb.frag + i);
  grid_wait();
  auto twiddles = [&](const uint4 *p, uint2 *w) {
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const uint4 v = p[4 * c];
      w[2 * c] = make_uint2(v.x, v.y);
      w[2 * c + 1] = make_uint2(v.z, v.w);
    }
  };
  // ---- INTT column stages, output constant, centring, offset
  uint32_t xs[KR][16];
#pragma unroll
  for (int i = 0; i < KR; i++) {
    if (4 * i < K) {
      // lanes past the last source repeat it: its B bytes are zero there
      const int k = min(4 * i + tq, K - 1);
      const int g = jb.src_gidx[k];
      const uint32_t q = __ldg(b.primes + g);
      const uint32_t *src = jb.src + (static_cast<size_t>(jb.src_row[k]) << 16) + col;
      const uint32_t c0 = jb.c0[k], c0s = jb.c0s[k];
      uint2 w[16];
#pragma unroll
      for (int e = 0; e < 16; e++) xs[i][e] = src[e * kRowLen];
      if (i == 0) __syncthreads();  // the staged tables
      twiddles(tws + 32 * i + (k & 3), w);
      radix16_inv(xs[i], w, q);
#pragma unroll
      for (int e = 0; e < 16; e++)
        xs[i][e] = static_cast<uint32_t>(centre(reduce2q(shoup_lazy(xs[i][e], c0, c0s, q), q), q) + kOffset);
    } else {
#pragma unroll
      for (int e = 0; e < 16; e++) xs[i][e] = 0u;
    }
  }
  // ---- four targets at a time: MMAs, reduction, NTT column stages, store
  constexpr int kSteps = (KR + 1) / 2;
  for (int mg = 0; mg < groups; mg++) {
    const uint4 *frag = frg + mg * (steps + 1) * 32 + lane;
    const int m = min(4 * mg + tq, M - 1);
    const uint4 pr = prm[m];
    const uint32_t p = pr.x;
    const int32_t pinv = static_cast<int32_t>(pr.y);
    uint4 bw[kSteps];
#pragma unroll
    for (int s = 0; s < kSteps; s++) bw[s] = s < steps ? frag[32 * s] : make_uint4(0, 0, 0, 0);
    const uint4 cc = frag[32 * steps];
    uint32_t v[16];
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
      int lo[4] = {static_cast<int>(cc.x), static_cast<int>(cc.y), static_cast<int>(cc.x), static_cast<int>(cc.y)};
      int hi[4] = {static_cast<int>(cc.z), static_cast<int>(cc.w), static_cast<int>(cc.z), static_cast<int>(cc.w)};
#pragma unroll
      for (int s = 0; s < kSteps; s++) {
        if (2 * s + 1 < KR) {
          mma_k32(lo, xs[2 * s][e], xs[2 * s][e + 1], xs[2 * s + 1][e], xs[2 * s + 1][e + 1], bw[s].x, bw[s].y);
          mma_k32(hi, xs[2 * s][e], xs[2 * s][e + 1], xs[2 * s + 1][e], xs[2 * s + 1][e + 1], bw[s].z, bw[s].w);
        } else {
          mma_k16(lo, xs[2 * s][e], xs[2 * s][e + 1], bw[s].x);
          mma_k16(hi, xs[2 * s][e], xs[2 * s][e + 1], bw[s].z);
        }
      }
      v[e] = join(lo[0], lo[1], hi[0], hi[1], p, pinv);
      v[e + 1] = join(lo[2], lo[3], hi[2], hi[3], p, pinv);
    }
    uint2 w[16];
    twiddles(tws_dst + 32 * mg + (m & 3), w);
    radix16_fwd(v, w, p);
    if (4 * mg + tq < M) {
      uint32_t *dst = jb.dst + (static_cast<size_t>(pr.z) << 16) + col;
#pragma unroll
      for (int e = 0; e < 16; e++) dst[e * kRowLen] = v[e];
    }
  }
}

}  // namespace

void launch_modswitch_cols(const MSColBatch &b, int log_n, cudaStream_t s) {
  if (b.count <= 0 || log_n != 16) return;
  int max_k = 0, max_m = 0;
  for (int j = 0; j < b.count; j++) {
    max_k = b.jobs[j].K > max_k ? b.jobs[j].K : max_k;
    max_m = b.jobs[j].M > max_m ? b.jobs[j].M : max_m;
  }
  // the kernel's staged tables: 512 bytes of twiddles per group of four
  // primes, 64 of prime data and 512 per fragment step and group of targets
  const int groups = (max_m + 3) / 4, steps = (max_k + 7) / 8;
  const size_t smem = 512 * ((max_k + 3) / 4 + groups) + 64 * groups + 512 * static_cast<size_t>(groups) * (steps + 1);
  // one CTA per 32 columns of a job, each converting all of the job's targets:
  // sharing a job's targets out over 2 to 6 CTAs (each repeating the source
  // stages) was slower at every size, down to the two one-source jobs of a
  // rescale (plaintext product and rescale at level 5: 23.6 us in one part,
  // 25.6 us in two; a multiplication at level 22: 98.7, 103.5 and 107.7 us in
  // one, two and three parts)
  const dim3 grid(kRowLen / kCtaCols, b.count);
  // 35 KiB of shared memory at most (16 sources, 64 targets)
  auto go = [&](const auto &x) {
    using B = std::decay_t<decltype(x)>;
    if (max_k <= 4)
      launch_dependent(k_modswitch_cols<1, 7, B>, grid, 32 * kColWarps, smem, s, x);
    else if (max_k <= 8)
      launch_dependent(k_modswitch_cols<2, 6, B>, grid, 32 * kColWarps, smem, s, x);
    else if (max_k <= 12)
      launch_dependent(k_modswitch_cols<3, 5, B>, grid, 32 * kColWarps, smem, s, x);
    else
      launch_dependent(k_modswitch_cols<4, 4, B>, grid, 32 * kColWarps, smem, s, x);
  };
  if (b.count > kFewJobs) {
    go(b);
    return;
  }
  MSColBatchOf<kFewJobs> few;
  few.count = b.count;
  few.tw = b.tw;
  few.itw = b.itw;
  few.primes = b.primes;
  few.qinvs = b.qinvs;
  for (int i = 0; i < b.count; i++) few.jobs[i] = b.jobs[i];
  go(few);
}

}  // namespace chd
