// Building blocks shared by the NTT kernels (ntt.cu), the fused ModSwitch
// column pass (modswitch.cu) and the fused key-switch row pass
// (keyswitch.cu): radix-16 networks of lazy Shoup butterflies with
// vectorised twiddle loads, and the row phase with its shared-memory
// exchanges.
#pragma once

#include "arith.cuh"

namespace chd {

// ---- N = 2^16 geometry: a limb is a 16 x 4096 row-major matrix ----
// Stages m = 1 .. 8 pair elements of one column (a 16-point column transform
// held by one thread); stages m = 16 .. 32768 stay inside one 4096-element
// row, held by the 256 threads of a CTA with 16 elements each, in three
// radix-16 rounds.  Between the first two rounds the row crosses the CTA
// (one barrier); the last two work on blocks of 256 elements, each owned by
// one half-warp, which exchanges them under __syncwarp.  A radix-16 column
// needs no exchange, so the fused base-conversion column pass
// (modswitch.cu) keeps everything in registers; with the earlier 128 x 512
// split the same pass crossed shared memory and a CTA barrier per source
// and per target and took 313 us of a 642 us batch of 8 multiplications.
constexpr int kRowLen = 4096;      // elements per row
constexpr int kRowThreads = 256;   // threads per row
constexpr int kLimbRows = 16;      // rows per limb

// Twiddle loads: tables hold (w, companion) pairs; pairs at even (resp.
// multiple-of-4) indices are 16- (resp. 32-) byte aligned, so 2 and 4
// consecutive pairs are fetched with 128-bit loads.
__device__ __forceinline__ void tw_ld2(const uint2 *tw, uint2 *w) {
  const uint4 v = __ldg(reinterpret_cast<const uint4 *>(tw));
  w[0] = make_uint2(v.x, v.y);
  w[1] = make_uint2(v.z, v.w);
}

// The fifteen twiddles of a radix-16 network over group index B (16 / 2^s
// consecutive stages m' = 2^s B' share the numbering): stage s uses pairs
// (B << s) + g, g < 2^s.  w[2^s + g] receives them.
__device__ __forceinline__ void tw_radix16(const uint2 *tw, unsigned B, uint2 *w) {
  w[1] = __ldg(tw + B);
  tw_ld2(tw + 2u * B, w + 2);
#pragma unroll
  for (int c = 0; c < 2; c++) tw_ld2(tw + 4u * B + 2 * c, w + 4 + 2 * c);
#pragma unroll
  for (int c = 0; c < 4; c++) tw_ld2(tw + 8u * B + 2 * c, w + 8 + 2 * c);
}
// The same for the last round of row r (B = 4096 + 256 r + 16 b + u): the
// tables of N = 2^16 store the pairs of stages m = 16384 and 32768 of one
// row chunk-major (tw_position), so that a warp's 16-byte loads are
// contiguous.
__device__ __forceinline__ void tw_radix16_last(const uint2 *tw, int r, int t, uint2 *w) {
  const unsigned s = t;
  const uint2 *t1 = tw + 4096 + 256 * r, *t2 = tw + 8192 + 512 * r, *t4 = tw + 16384 + 1024 * r,
              *t8 = tw + 32768 + 2048 * r;
  w[1] = __ldg(t1 + s);
  tw_ld2(t2 + 2u * s, w + 2);
#pragma unroll
  for (int c = 0; c < 2; c++) tw_ld2(t4 + 2u * s + 512 * c, w + 4 + 2 * c);
#pragma unroll
  for (int c = 0; c < 4; c++) tw_ld2(t8 + 2u * s + 512 * c, w + 8 + 2 * c);
}

// Radix-16 forward network (CT stages at register distances 8, 4, 2, 1).
__device__ __forceinline__ void radix16_fwd(uint32_t *x, const uint2 *w, uint32_t q) {
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const int m = 1 << s, h = 8 >> s;
#pragma unroll
    for (int g = 0; g < m; g++)
#pragma unroll
      for (int j = 0; j < h; j++) ct_lazy(x[g * 2 * h + j], x[g * 2 * h + j + h], w[m + g], q);
  }
}
// Radix-16 inverse network (GS stages at distances 1, 2, 4, 8), its mirror.
__device__ __forceinline__ void radix16_inv(uint32_t *x, const uint2 *w, uint32_t q) {
#pragma unroll
  for (int s = 3; s >= 0; s--) {
    const int m = 1 << s, h = 8 >> s;
#pragma unroll
    for (int g = 0; g < m; g++)
#pragma unroll
      for (int j = 0; j < h; j++) gs_lazy(x[g * 2 * h + j], x[g * 2 * h + j + h], w[m + g], q);
  }
}

// Row buffer in shared memory: element 256 b + 16 k + u (b, k, u < 16) of a
// row lies at rpos(b, k, u), so that every access of the row phase is free of
// bank conflicts: 32-bit accesses with k the register, u the lane and b, b + 1
// the halves of a warp (bit 4 tells them apart), or with b the register and
// 16 k + u the thread; 128-bit accesses to chunks u / 4 with k the lane, or
// with (k, u / 4) counting through the lanes.  No padding: three buffers at
// four CTAs are 196 KiB, the last step before the shared memory takes all
// of an SM's cache but 28 KiB (a padded layout with fewer address
// instructions did: the key-switch row pass took 211 us instead of 203).
__host__ __device__ constexpr int rpos(int b, int k, int u) {
  return 256 * b + 16 * (k ^ (b & 1)) + (u ^ (((k >> 1) & 3) << 2));
}
constexpr int kRowBuf = 4096;  // words per row buffer

// Thread t's block (see above) and lane in it for the last two rounds
__device__ __forceinline__ int row_block(int t) { return t >> 4; }
__device__ __forceinline__ int row_lane(int t) { return t & 15; }

// "Row order" below: thread t holds x[k] = element t + 256 k.  "Chunk order":
// with b = row_block(t), u = row_lane(t), x[4 i + c] = element
// 256 b + 64 i + 4 u + c, so that a half-warp's 16-byte accesses to memory
// cover 256 contiguous bytes.
__device__ __forceinline__ unsigned chunk_off(int t) { return 256u * row_block(t) + 4u * row_lane(t); }  // + 64 i

// chunk order -> own group of 16 consecutive elements and back, inside the
// half-warp's block of the row buffer
__device__ __forceinline__ void group_st(uint32_t *sm, int t, const uint32_t *x) {
#pragma unroll
  for (int i = 0; i < 4; i++)
    *reinterpret_cast<uint4 *>(sm + rpos(row_block(t), row_lane(t), 4 * i)) =
        make_uint4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
}
__device__ __forceinline__ void group_ld(const uint32_t *sm, int t, uint32_t *x) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint4 v = *reinterpret_cast<const uint4 *>(sm + rpos(row_block(t), row_lane(t), 4 * i));
    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
  }
}
// chunk i: k = 4 i + u / 4, elements 4 (u % 4) ..
__device__ __forceinline__ int chunk_pos(int t, int i) {
  const int u = row_lane(t);
  return rpos(row_block(t), 4 * i + (u >> 2), 4 * (u & 3));
}
__device__ __forceinline__ void chunk_st4(uint32_t *sm, int t, int i, uint4 v) {
  *reinterpret_cast<uint4 *>(sm + chunk_pos(t, i)) = v;
}
__device__ __forceinline__ uint4 chunk_ld4(const uint32_t *sm, int t, int i) {
  return *reinterpret_cast<const uint4 *>(sm + chunk_pos(t, i));
}
__device__ __forceinline__ void chunk_ld(const uint32_t *sm, int t, uint32_t *x) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint4 v = chunk_ld4(sm, t, i);
    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
  }
}
// round-1 view of the buffer (x[k] = element t + 256 k) and round-2 view
// (x[k] = element 256 b + 16 k + u)
__device__ __forceinline__ void row1_st(uint32_t *sm, int t, const uint32_t *x) {
#pragma unroll
  for (int k = 0; k < 16; k++) sm[rpos(k, t >> 4, t & 15)] = x[k];
}
__device__ __forceinline__ void row1_ld(const uint32_t *sm, int t, uint32_t *x) {
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = sm[rpos(k, t >> 4, t & 15)];
}
__device__ __forceinline__ void row2_st(uint32_t *sm, int t, const uint32_t *x) {
#pragma unroll
  for (int k = 0; k < 16; k++) sm[rpos(row_block(t), k, row_lane(t))] = x[k];
}
__device__ __forceinline__ void row2_ld(const uint32_t *sm, int t, uint32_t *x) {
#pragma unroll
  for (int k = 0; k < 16; k++) x[k] = sm[rpos(row_block(t), k, row_lane(t))];
}

// The row phases below take one or two rows at once (`two`, uniform over the
// CTA; the second in x[P - 1], only for P = 2): rows of one prime share the
// twiddles in registers, the barrier, and the wait for every load.  sm[i] is
// row i's buffer.  One CTA barrier; a caller that runs another row transform
// of the CTA uses other buffers (a thread past the barrier of one transform
// knows that every thread is done with the buffers of the one before).

// The 12 row stages (m = 16 .. 32768) of the forward transform on row r of
// limbs of one prime: x in row order -> own group of 16, lazy [0, 2q).
template <int P>
__device__ __forceinline__ void row_fwd_group(uint32_t (&x)[P][16], bool two, uint32_t *const (&sm)[P], const uint2 *tw,
                                              int r, int t, uint32_t q) {
  {
    uint2 w[16];
    tw_radix16(tw, 16 + r, w);
#pragma unroll
    for (int p = 0; p < P; p++)
      if (p == 0 || two) {
        radix16_fwd(x[p], w, q);
        row1_st(sm[p], t, x[p]);
      }
  }
  __syncthreads();
  {
    uint2 w[16];
    tw_radix16(tw, 256 + 16 * r + row_block(t), w);
#pragma unroll
    for (int p = 0; p < P; p++)
      if (p == 0 || two) {
        row2_ld(sm[p], t, x[p]);
        radix16_fwd(x[p], w, q);
        row2_st(sm[p], t, x[p]);
      }
  }
  __syncwarp();
  {
    uint2 w[16];
    tw_radix16_last(tw, r, t, w);
#pragma unroll
    for (int p = 0; p < P; p++)
      if (p == 0 || two) {
        group_ld(sm[p], t, x[p]);
        radix16_fwd(x[p], w, q);
      }
  }
}

// The 12 row stages of the inverse transform: chunks stored to the buffers by
// their half-warps -> x in row order.
template <int P>
__device__ __forceinline__ void row_inv_stored(uint32_t (&x)[P][16], bool two, uint32_t *const (&sm)[P],
                                               const uint2 *tw, int r, int t, uint32_t q) {
  __syncwarp();
  {
    uint2 w[16];
    tw_radix16_last(tw, r, t, w);
#pragma unroll
    for (int p = 0; p < P; p++)
      if (p == 0 || two) {
        group_ld(sm[p], t, x[p]);
        radix16_inv(x[p], w, q);
        group_st(sm[p], t, x[p]);
      }
  }
  __syncwarp();
  {
    uint2 w[16];
    tw_radix16(tw, 256 + 16 * r + row_block(t), w);
#pragma unroll
    for (int p = 0; p < P; p++)
      if (p == 0 || two) {
        row2_ld(sm[p], t, x[p]);
        radix16_inv(x[p], w, q);
        row2_st(sm[p], t, x[p]);
      }
  }
  __syncthreads();
  {
    uint2 w[16];
    tw_radix16(tw, 16 + r, w);
#pragma unroll
    for (int p = 0; p < P; p++)
      if (p == 0 || two) {
        row1_ld(sm[p], t, x[p]);
        radix16_inv(x[p], w, q);
      }
  }
}

// 16 words of a row in chunk order; p = row start + chunk_off(t)
__device__ __forceinline__ void ld_chunks(const uint32_t *p, uint32_t *x) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint4 v = *reinterpret_cast<const uint4 *>(p + 64 * i);
    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
  }
}
__device__ __forceinline__ void st_chunks(uint32_t *p, const uint32_t *x) {
#pragma unroll
  for (int i = 0; i < 4; i++)
    *reinterpret_cast<uint4 *>(p + 64 * i) = make_uint4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
}

}  // namespace chd
