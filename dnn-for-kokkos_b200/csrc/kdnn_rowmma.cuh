// Batched GEMM of Q5_K, Q6_K and Q8_0 rows against several int8 activation rows on the tensor cores
// (mma.sync s8 x s8 -> s32): one matrix, Y[m, j] = sum_k W[j, k] * q(x[m, :])[k].
//
// These formats keep the integer path: sc * q of Q6_K (13 bits and a sign) does not fit fp16 exactly, so the split-fp16
// kernel of kdnn_split.cuh is not open to them. What the per-lane dp4a kernel (kdnn_grouped.cuh) lost was parallelism: a CTA
// owned 128 rows and all of K, 32 CTAs for a 4096-row matrix, each lane waiting on its own 2-byte loads.
//
// Split: a CTA owns 16 * MT weight rows and 8 * NT activation rows; its warps take the 256-element super-blocks of K
// in turn (warp w: w, w + warps, ...) and meet once at the end in shared memory, in warp order. Every warp is on its own
// until then: its ring of two stages (the packed bytes of its rows, unaligned formats from the 16-byte boundary below,
// and the matching activations) is filled by its own cp.async, no CTA barrier inside the loop.
//
// Fragments: lane (r = lane / 4, t = lane % 4) of an m16n8k16 product holds word t of a 16-element granule of rows r and
// r + 8, which is one aligned-or-funnelled word of the packed row per two or four granules, so a weight is unpacked once, in
// registers, in its place. The activation rows are written in that order too (rowmma_quantize_kernel): per 8 rows and
// 64 elements 512 bytes, 16 per lane (word t of its row's four granules), then one float4 of factors per row.
//
// The accumulator starts at the bit pattern of 12582912.0f, so the int32 sum is already a float; with an integer scale the
// offset leaves in the same fma, exactly (|sc * dot| < 2^24): two fma per product, the block's d once per 256 elements.
//
// Bound by unpack and fold issue, not by memory (7.4 us of packed bytes): a 4096 x 14336 Q6_K matrix against 16 rows takes 32.3 us
// with the quantizer launch, 1.5 TB/s; the dp4a kernel took 433 us.
#pragma once

#include "kdnn_mma.cuh"
#include "kdnn_tc.cuh"

namespace kdnn {

constexpr int kRmTileBytes = 640;                   // 8 activation rows x 64 elements: 512 of int8, 8 float4
constexpr int kRmBlockBytes = 4 * kRmTileBytes;     // the same rows x 256 elements
constexpr int kRmSmemMax = 227 * 1024;

template <uint32_t DT> struct RmFormat;             // bytes of 256 elements, 16-byte pieces that cover them, row pitch in a stage
template <> struct RmFormat<KDNN_GGML_Q5_K> { static constexpr int kBytes = 176, kPieces = 11, kPitch = 176; };
template <> struct RmFormat<KDNN_GGML_Q6_K> { static constexpr int kBytes = 210, kPieces = 14, kPitch = 240; };
template <> struct RmFormat<KDNN_GGML_Q8_0> { static constexpr int kBytes = 272, kPieces = 18, kPitch = 304; };
// The pitches are an odd number of 16-byte pieces: the eight rows of a fragment load fall on different banks.

struct RmParams {
  const uint8_t* w;          // 16-byte aligned
  size_t row_bytes, total;   // total: bytes of the matrix, nothing is read behind them
  int N, M, blocks;          // blocks = K / 256
  const uint8_t* x;          // activations, rowmma_quantize_kernel's layout
  void* y;
  size_t ldy;
  int y_bf16;
};

inline size_t rowmma_x_bytes(size_t M, size_t K) { return (M + 7) / 8 * (K / 64) * kRmTileBytes; }

template <uint32_t DT, class SRC>
__global__ void rowmma_quantize_kernel(const SRC* __restrict__ src, size_t ld, int K, uint8_t* __restrict__ dst) {
  pdl_launch_dependents();   // launched plainly: everything earlier in the stream is complete, so the product may read weights
  const int row = blockIdx.y, lane = threadIdx.x & 31, l8 = lane & 7;
  const int nblk = K / 32, nitems = K / 64;
  const SRC* x = src + static_cast<size_t>(row) * ld;
  const bool vec_ok = (reinterpret_cast<uintptr_t>(x) & (sizeof(SRC) * 4 - 1)) == 0;
  uint8_t* out = dst + static_cast<size_t>(row >> 3) * nitems * kRmTileBytes;
  const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int base = gwarp * 4; base < nblk; base += nwarp * 4) {
    const int b = base + (lane >> 3);
    const bool valid = b < nblk;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (valid) load4<SRC>(x, static_cast<size_t>(b) * 32 + l8 * 4, vec_ok, v);
    float d;
    int part, total;
    const uint32_t packed = quantize_block_lane(v, d, part, total);
    if (!valid) continue;
    int item, g;
    granule_map<DT>(b, l8 >> 2, item, g);
    uint8_t* tile = out + static_cast<size_t>(item) * kRmTileBytes;
    *reinterpret_cast<uint32_t*>(tile + ((row & 7) * 4 + (l8 & 3)) * 16 + g * 4) = packed;
    float* f = reinterpret_cast<float*>(tile + 512 + (row & 7) * 16);
    if (DT == KDNN_GGML_Q6_K) {
      if ((l8 & 3) == 0) f[g] = d;                       // the four granules lie in four different blocks
    } else if (l8 == 0) {
      f[g >> 1] = d;                                     // {d0, d1, d0 * sum0, d1 * sum1}
      f[2 + (g >> 1)] = d * static_cast<float>(total);
    }
  }
}

__device__ __forceinline__ void cp_async16_n(uint32_t dst, const void* src, int n) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
// Four bytes at an even address: the two words around it (the second one lies inside the row's pitch).
__device__ __forceinline__ uint32_t lds32_even(uint32_t a) {
  return __funnelshift_r(lds32(a & ~3u), lds32((a & ~3u) + 4u), (a & 3u) * 8u);
}
__device__ __forceinline__ void mma_s8_k16_magic(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a0), "r"(a1), "r"(b), "r"(kM2MagicI));
}
__device__ __forceinline__ void mma_s8_k32_magic(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                                 uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(kM2MagicI));
}
// Byte `i` of w as a signed number: the byte with its sign flipped is the low byte of a float around 2^23.
template <int I>
__device__ __forceinline__ float s8_float(uint32_t w_flipped) {
  return __uint_as_float(__byte_perm(w_flipped, 0x4B000000u, 0x7440 | I)) - 8388736.0f;
}
template <int I>
__device__ __forceinline__ float u8_float(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | I)) - 8388608.0f;
}

// One row's share of 64 elements in a lane: word t of the four granules and the factors of the fold.
//   Q6_K: s = sc of the granule (integer).  Q5_K: s[0..1] = sc, s[2..3] = mn.  Q8_0: s[0..1] = d of the two blocks.
template <uint32_t DT, int IT>
__device__ __forceinline__ void rm_unpack(uint32_t row, int t, uint32_t (&w)[4], float (&s)[4]) {
  if (DT == KDNN_GGML_Q6_K) {
    constexpr int chunk = IT >> 1, half = IT & 1;
    const uint32_t a = row + chunk * 64 + half * 16 + 4 * t;
    const uint32_t l0 = lds32_even(a), l1 = lds32_even(a + 32);
    const uint32_t h = lds32_even(row + 128 + chunk * 32 + half * 16 + 4 * t);
    const uint32_t q[4] = {(l0 & 0x0F0F0F0Fu) | ((h << 4) & 0x30303030u), (l1 & 0x0F0F0F0Fu) | ((h << 2) & 0x30303030u),
                           ((l0 >> 4) & 0x0F0F0F0Fu) | (h & 0x30303030u), ((l1 >> 4) & 0x0F0F0F0Fu) | ((h >> 2) & 0x30303030u)};
#pragma unroll
    for (int g = 0; g < 4; ++g) w[g] = (q[g] + 0x60606060u) ^ 0x80808080u;   // q - 32 in each byte, no carry between bytes
    const uint32_t c0 = lds32_even(row + 192 + chunk * 8) ^ 0x80808080u, c1 = lds32_even(row + 196 + chunk * 8) ^ 0x80808080u;
    s[0] = s8_float<half>(c0); s[1] = s8_float<2 + half>(c0);
    s[2] = s8_float<half>(c1); s[3] = s8_float<2 + half>(c1);
  } else if (DT == KDNN_GGML_Q5_K) {
    const uint32_t h0 = lds32(row + 16 + 4 * t) >> (2 * IT), h1 = lds32(row + 32 + 4 * t) >> (2 * IT);
    const uint32_t qa = lds32(row + 48 + IT * 32 + 4 * t), qb = lds32(row + 64 + IT * 32 + 4 * t);
    w[0] = (qa & 0x0F0F0F0Fu) | ((h0 & 0x01010101u) << 4);
    w[1] = (qb & 0x0F0F0F0Fu) | ((h1 & 0x01010101u) << 4);
    w[2] = ((qa >> 4) & 0x0F0F0F0Fu) | ((h0 & 0x02020202u) << 3);
    w[3] = ((qb >> 4) & 0x0F0F0F0Fu) | ((h1 & 0x02020202u) << 3);
    uint32_t scp, mnp;
    q4k_scale_pair(lds32(row + 4), lds32(row + 8), lds32(row + 12), IT, scp, mnp);
    s[0] = u8_float<0>(scp); s[1] = u8_float<1>(scp);
    s[2] = u8_float<0>(mnp); s[3] = u8_float<1>(mnp);
  } else {
    const uint32_t b = row + IT * 68;
    w[0] = lds32_even(b + 2 + 4 * t);  w[1] = lds32_even(b + 18 + 4 * t);
    w[2] = lds32_even(b + 36 + 4 * t); w[3] = lds32_even(b + 52 + 4 * t);
    s[0] = h2f(lds16(b)); s[1] = h2f(lds16(b + 34));
    s[2] = s[3] = 0.f;
  }
}

template <uint32_t DT, int MT, int NT, int IT>
__device__ __forceinline__ void rm_item(const uint32_t (&row)[MT][2], uint32_t xs, int lane, int live, float (&acc)[MT][NT][4],
                                        float (&acm)[MT][NT][4]) {
  const int t = lane & 3;
  uint32_t w[MT][2][4];
  float s[MT][2][4];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    rm_unpack<DT, IT>(row[m][0], t, w[m][0], s[m][0]);
    rm_unpack<DT, IT>(row[m][1], t, w[m][1], s[m][1]);
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    if (n < live) {
      const uint32_t tile = xs + n * kRmBlockBytes + IT * kRmTileBytes;
      const int4 q  = lds128_g(tile + lane * 16);
      const int4 f0 = lds128_g(tile + 512 + t * 32), f1 = lds128_g(tile + 528 + t * 32);
      const uint32_t b[4] = {(uint32_t)q.x, (uint32_t)q.y, (uint32_t)q.z, (uint32_t)q.w};
      const float x0[4] = {__int_as_float(f0.x), __int_as_float(f0.y), __int_as_float(f0.z), __int_as_float(f0.w)};
      const float x1[4] = {__int_as_float(f1.x), __int_as_float(f1.y), __int_as_float(f1.z), __int_as_float(f1.w)};
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        int c[4];
        if (DT == KDNN_GGML_Q6_K) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            mma_s8_k16_magic(c, w[m][0][g], w[m][1][g], b[g]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float sc = s[m][i >> 1][g];
              acc[m][n][i] = fmaf(fmaf(__int_as_float(c[i]), sc, -kM2MagicF * sc), (i & 1) ? x1[g] : x0[g], acc[m][n][i]);
            }
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            mma_s8_k32_magic(c, w[m][0][2 * h], w[m][1][2 * h], w[m][0][2 * h + 1], w[m][1][2 * h + 1], b[2 * h], b[2 * h + 1]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float sc = s[m][i >> 1][h], dx = (i & 1) ? x1[h] : x0[h];
              if (DT == KDNN_GGML_Q5_K) {
                acc[m][n][i] = fmaf(fmaf(__int_as_float(c[i]), sc, -kM2MagicF * sc), dx, acc[m][n][i]);
                acm[m][n][i] = fmaf(s[m][i >> 1][2 + h], (i & 1) ? x1[2 + h] : x0[2 + h], acm[m][n][i]);
              } else {
                acc[m][n][i] = fmaf((__int_as_float(c[i]) - kM2MagicF) * sc, dx, acc[m][n][i]);
              }
            }
          }
        }
      }
    }
  }
}

template <uint32_t DT, int MT, int NT>
__global__ void __launch_bounds__(256, 1) rowmma_kernel(const RmParams p) {
  using F = RmFormat<DT>;
  constexpr int kRows = 16 * MT, kW = kRows * F::kPitch, kStage = kW + NT * kRmBlockBytes;
  extern __shared__ __align__(16) uint8_t rm_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const uint32_t ring = smem_u32(rm_smem) + warp * 2 * kStage;
  const int row0 = blockIdx.x * kRows, tile0 = blockIdx.y * NT;
  const int live = min(NT, (p.M + 7) / 8 - tile0);
  pdl_launch_dependents();

  auto load_w = [&](int blk, int st) {
    for (int c = lane; c < kRows * F::kPieces; c += 32) {
      const int r = c / F::kPieces, i = c - r * F::kPieces;
      const size_t off = static_cast<size_t>(min(row0 + r, p.N - 1)) * p.row_bytes + static_cast<size_t>(blk) * F::kBytes;
      const size_t from = (off & ~size_t(15)) + 16 * i;
      if (from < off + F::kBytes)
        cp_async16_n(ring + st * kStage + r * F::kPitch + 16 * i, p.w + from, static_cast<int>(min(size_t(16), p.total - from)));
    }
  };
  auto load_x = [&](int blk, int st) {
    for (int n = 0; n < live; ++n) {
      const uint8_t* src = p.x + (static_cast<size_t>(tile0 + n) * p.blocks + blk) * kRmBlockBytes;
#pragma unroll
      for (int c = 0; c < kRmBlockBytes / 512; ++c)
        cp_async16_n(ring + st * kStage + kW + n * kRmBlockBytes + (c * 32 + lane) * 16, src + (c * 32 + lane) * 16, 16);
    }
  };

  float tot[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) tot[m][n][i] = 0.f;

  if (warp < p.blocks) load_w(warp, 0);
  pdl_wait();                          // the activations come from the kernel before this one
  if (warp < p.blocks) load_x(warp, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  int st = 0;
  for (int blk = warp; blk < p.blocks; blk += warps, st ^= 1) {
    if (blk + warps < p.blocks) {
      load_w(blk + warps, st ^ 1);
      load_x(blk + warps, st ^ 1);
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
    __syncwarp();                      // every lane's pieces of this stage have landed
    uint32_t row[MT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 16 * m + 8 * h + (lane >> 2);
        const size_t off = static_cast<size_t>(min(row0 + r, p.N - 1)) * p.row_bytes + static_cast<size_t>(blk) * F::kBytes;
        row[m][h] = ring + st * kStage + r * F::kPitch + static_cast<uint32_t>(off & 15);
      }
    const uint32_t xs = ring + st * kStage + kW;
    float acc[MT][NT][4], acm[MT][NT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][n][i] = acm[m][n][i] = 0.f;
    rm_item<DT, MT, NT, 0>(row, xs, lane, live, acc, acm);
    rm_item<DT, MT, NT, 1>(row, xs, lane, live, acc, acm);
    rm_item<DT, MT, NT, 2>(row, xs, lane, live, acc, acm);
    rm_item<DT, MT, NT, 3>(row, xs, lane, live, acc, acm);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float d  = DT == KDNN_GGML_Q8_0 ? 1.0f : h2f(lds16(row[m][h] + (DT == KDNN_GGML_Q6_K ? 208 : 0)));
        const float dm = DT == KDNN_GGML_Q5_K ? h2f(lds16(row[m][h] + 2)) : 0.f;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 2 * h; i < 2 * h + 2; ++i) {
            if (DT == KDNN_GGML_Q8_0) tot[m][n][i] += acc[m][n][i];
            else if (DT == KDNN_GGML_Q6_K) tot[m][n][i] = fmaf(d, acc[m][n][i], tot[m][n][i]);
            else tot[m][n][i] += d * acc[m][n][i] - dm * acm[m][n][i];
          }
      }
    __syncwarp();                      // this stage is read: the next round refills it
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float* part = reinterpret_cast<float*>(rm_smem);   // [warp][activation row][weight row], over the ring
  constexpr int kOut = kRows * 8 * NT;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        part[warp * kOut + (8 * n + 2 * (lane & 3) + (i & 1)) * kRows + 16 * m + 8 * (i >> 1) + (lane >> 2)] = tot[m][n][i];
  __syncthreads();
  for (int e = threadIdx.x; e < kOut; e += blockDim.x) {
    const int j = row0 + e % kRows, x = tile0 * 8 + e / kRows;
    if (j >= p.N || x >= p.M) continue;
    float v = 0.f;
    for (int k = 0; k < warps; ++k) v += part[k * kOut + e];
    const size_t o = static_cast<size_t>(x) * p.ldy + j;
    if (p.y_bf16) store_scalar(static_cast<__nv_bfloat16*>(p.y) + o, v);
    else store_scalar(static_cast<float*>(p.y) + o, v);
  }
}

template <uint32_t DT, int MT, int NT>
static cudaError_t launch_rowmma_tile(const RmParams& p, cudaStream_t st) {
  constexpr int kStage = 16 * MT * RmFormat<DT>::kPitch + NT * kRmBlockBytes;
  constexpr int kFit = kRmSmemMax / (2 * kStage), kWarps = kFit < 8 ? kFit : 8;   // K is split over as many warps as two stages each allow
  static_assert(2 * kStage >= 16 * MT * 8 * NT * 4, "the partial sums lie over the ring");
  auto kern = rowmma_kernel<DT, MT, NT>;
  static SmemAttrOnce once;
  const cudaError_t e = set_max_smem_once(once, kern, kWarps * 2 * kStage);
  if (e != cudaSuccess) return e;
  return launch_chained(kern, dim3((p.N + 16 * MT - 1) / (16 * MT), ((p.M + 7) / 8 + NT - 1) / NT), dim3(32 * kWarps), kWarps * 2 * kStage, st, p);
}

template <uint32_t DT, class SRC>
static cudaError_t launch_rowmma(const RmParams& p, const SRC* X, size_t ldx, uint8_t* x, cudaStream_t st) {
  const int K = p.blocks * 256;
  rowmma_quantize_kernel<DT, SRC><<<dim3(min(8, (K / 32 + 31) / 32), p.M), 256, 0, st>>>(X, ldx, K, x);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // 32 weight rows per CTA halve the activation traffic; 16 as long as they leave no SM a second CTA. Above 16 activation
  // rows a weight is unpacked once per 32 of them, and two stages of that fit with 16 weight rows.
  const bool two = (p.N + 15) / 16 > device_sm_count();
  if (p.M > 16) return launch_rowmma_tile<DT, 1, 4>(p, st);
  if (p.M > 8) return two ? launch_rowmma_tile<DT, 2, 2>(p, st) : launch_rowmma_tile<DT, 1, 2>(p, st);
  return two ? launch_rowmma_tile<DT, 2, 1>(p, st) : launch_rowmma_tile<DT, 1, 1>(p, st);
}

}  // namespace kdnn
