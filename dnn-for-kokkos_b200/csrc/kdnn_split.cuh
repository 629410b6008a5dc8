// Grouped tile GEMM for packed K-quant weights on the 5th-generation tensor cores in fp16 with SPLIT activations
// (tcgen05.mma kind::f16, both the unpacked weights and the accumulators in tensor memory): the kernel behind the
// MoE expert products and the batched GEMM.
//
//   dst[pos, j] = sum_k W_g[j, k] * x[row(pos), k],  x = the reference's per-32 int8 activations q * d
//
// Numerics. Inside a 256-element super-block the weight is d * (sc * q) - dmin * mn, 6-bit sc and 4-bit q. The tensor core
// accumulates in fp32 and TRUNCATES, so what it sums has to be exact or small beside the result:
//   * A = sc * q - t is an integer that fp16 holds exactly, t about 7 sc in the even and 8 sc in the odd sub-blocks (what one
//     fp16 fma can form): weights around zero, so that activations of one sign build no large sum that the min term takes
//     off again, and what is left of it (c below) has both signs;
//   * the rest of the weight is one number per 32 elements, c = d * t - dmin * mn, formed in fp32 and multiplied with the
//     block's activation sum in a product of its own: c relative to a power of two e as two fp16 parts, the sum as two;
//   * the activation row is written once (split_store_lane8) as two fp16 parts of  v = q * (256 * d / D),  D the largest d
//     of a G-element group (G = 256 or 128), so |v| <= 32512. hi is v rounded to a multiple of u: the products of A and hi are
//     multiples of u and their sum is exact below 2^24 u; u is the power of two that leaves two to three standard
//     deviations of the sum (230 |v|_2 and less), and the mean that A still has, below that. In a block far below the largest one hi
//     is rounded to eleven bits of that block instead (the products stay small beside the sum if the large block's weights
//     count, and exact if they do not). mid = fp16(v - hi) carries the next eleven bits.
// hi, mid and the block sums have accumulator columns of their own. The drain adds, in fp32 and once per group,
//   acc += D * (d / 256 * (P_hi + P_mid) + e / 16 * P_c)
// Error against float64 (relative 2-norm, 2048 x 4096, 24 rows; the integer tcgen05 kernel beside it): N(0, 1) 1.1e-7 (2.3e-7), its
// absolute values 2.0e-7 (4.5e-7), a block 1000 times larger whose weights are zero 1.4e-7 (2.2e-7), 1e6 times 1.9e-6 (2.2e-7). With
// A = sc * q, c left to the min term and one step u for the whole group: 2.2e-7, 2.5e-5, 2.4e-5, 3.1e-4; 14336 x 4096 against
// 8 / 32 / 500 rows 23.8 / 28.4 / 179 us then, 24.2 / 28.6 / 185 now.
//
// What bounds it: the per-32 rescale of the integer path (kdnn_mma.cuh, kdnn_tc.cuh) costs two to three instructions
// per (row, activation row, 32 elements); here the work per weight is the unpack, nine instructions per eight weights
// (four and-or, four fp16 fma, one shift), and it lands in tensor memory: no shared-memory round trip and no bank
// conflicts (a lane reads its own row: 144-byte rows put eight lanes' 16-byte pieces on distinct banks).
//
// One persistent CTA per SM, 28 warps. Warp-specialised, because what limits a warp here is its own dependent chain
// (about four clocks per instruction): unpack and drain need several warps per scheduler each.
//   NH = 1 (groups of up to 32 activation rows): 16 unpack warps, 8 drain warps; NH = 2 (up to 64): 8 and 16
//   unpack       lane = weight row; two (NH = 1: four) warpgroups, alternate tiles (128 rows x 256 elements; each half
//                of K one warpgroup when there are four), a TMEM buffer of 128 columns per tile parity
//   drain        lane = weight row, 32 activation rows per thread; tcgen05.ld, the fold above, the epilogue
//   MMA warp     issues the MMAs (M 128, N 16 per 8 activation rows, A from TMEM, B from shared memory). Its control
//                flow and operands are kept warp-uniform (votes, warp reductions, constant TMEM addresses), so that
//                descriptors live in uniform registers: issued from a divergent branch an MMA took 100 clocks
//   loaders      weights by tensor-map TMA, activation rows by cp.async into the 128-byte-swizzled layout
// Inner loops stay rolled and small: with every role unrolled the warps waited for instructions more than they ran.
// PAIR = 2: a unit of work is two row tiles that share each activation stage (MODE 1: gate and up); PAIR = 1: one
// row tile, the warpgroups alternate along K and their sums meet at the end.
//
// Every wait is bounded; a wait that gives up raises a CTA-wide abort flag, records KDNN_ERR_DEVICE_WAIT, waits
// (bounded) for the copies and MMAs in flight, and the CTA frees its TMEM and returns.
#pragma once

#include <algorithm>

#include "kdnn_tc.cuh"

namespace kdnn {

constexpr int kSpThreads = 28 * 32;
constexpr int kSpWarpMma = 24, kSpWarpW = 25, kSpWarpX = 26;
constexpr uint32_t kSpTmemA = 192, kSpTmemC = 448;    // D: 2 x 96 columns, A: 2 tile parities x 128, c: 2 x 16
constexpr int kSpExPitch = 132;                       // floats per activation row of the exchange tile (128 rows + pad)

// ---- split activation rows -------------------------------------------------------------------------
// Per super-block 1024 bytes: 256 fp16 hi, 256 fp16 mid (element order 0 2 1 3 inside every four, the order the
// nibble unpack produces); then per group of G elements 32 bytes: fp16 (block sum * 16 d / D) of the group's
// blocks in high and low parts, per two blocks {high, high, low, low}, twice over when the group has four blocks (the
// operand beside the high and the low parts of c); then D per group as float.
__host__ __device__ inline size_t split_sums_offset(size_t K) { return K * 4; }
__host__ __device__ inline size_t split_scale_offset(size_t K, int G) { return K * 4 + K / G * 32; }
inline size_t split_row_pitch(size_t K, int G) { return (split_scale_offset(K, G) + K / G * 4 + 255) & ~size_t(255); }

__device__ __forceinline__ uint32_t pack_half2(__half a, __half b) {
  return static_cast<uint32_t>(__half_as_ushort(a)) | (static_cast<uint32_t>(__half_as_ushort(b)) << 16);
}
// One warp, one super-block (four lanes per 32-block, eight elements per lane: quantize_block_lane8's mapping with
// the warp's first block a multiple of eight): writes the super-block's share of the split row. All lanes call it.
template <int G>
__device__ __forceinline__ void split_store_lane8(uint8_t* row, size_t K, int b, uint2 packed, float d, int total) {
  const int l4 = threadIdx.x & 3, blk = b & 7, sb = b >> 3;
  float dm = fmaxf(d, __shfl_xor_sync(0xffffffffu, d, 4));
  dm = fmaxf(dm, __shfl_xor_sync(0xffffffffu, dm, 8));
  if (G == 256) dm = fmaxf(dm, __shfl_xor_sync(0xffffffffu, dm, 16));
  const float r = dm > 0.0f ? 256.0f * __fdiv_rn(d, dm) : 0.0f;
  const float sum = __fmul_rn(static_cast<float>(total), 0.0625f * r);   // at most 65024 in size
  float v[8], n2 = 0.0f, s1 = fabsf(sum);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int q = static_cast<int8_t>(((i < 4 ? packed.x : packed.y) >> (8 * (i & 3))) & 0xFFu);
    v[i] = __fmul_rn(static_cast<float>(q), r);
    n2 += v[i] * v[i];
  }
#pragma unroll
  for (int o = 1; o < G / 8; o <<= 1) {
    n2 += __shfl_xor_sync(0xffffffffu, n2, o);                        // |v|^2 of the group
    if (o >= 4) s1 += __shfl_xor_sync(0xffffffffu, s1, o);            // its blocks' |sum|
  }
  // u: the power of two at or above max(600 |v|, 48 sum of |block sums of v|) / 2^24, from 2 to 32
  const float need = fminf(fmaxf(fmaxf(600.0f * sqrtf(n2), 768.0f * s1) * 0x1p-24f, 2.0f), 32.0f);
  const float u = __uint_as_float((__float_as_uint(need) + 0x7FFFFFu) & 0x7F800000u);
  // this block's own step: its largest |v|, 127 * r, is 1016 to 2032 of them (2^-24 is fp16's last bit)
  const float own = fmaxf(__uint_as_float(__float_as_uint(r) & 0x7F800000u) * 0.125f, 0x1p-24f);
  const float step = fminf(u, own), rstep = __uint_as_float(0x7F000000u - __float_as_uint(step));
  __half hi[8], mid[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    hi[i] = __float2half_rn(rintf(v[i] * rstep) * step);
    mid[i] = __float2half_rn(v[i] - __half2float(hi[i]));
  }
  uint8_t* o = row + static_cast<size_t>(sb) * 1024 + blk * 64 + l4 * 16;
  *reinterpret_cast<uint4*>(o) = make_uint4(pack_half2(hi[0], hi[2]), pack_half2(hi[1], hi[3]), pack_half2(hi[4], hi[6]), pack_half2(hi[5], hi[7]));
  *reinterpret_cast<uint4*>(o + 512) = make_uint4(pack_half2(mid[0], mid[2]), pack_half2(mid[1], mid[3]), pack_half2(mid[4], mid[6]), pack_half2(mid[5], mid[7]));
  const int grp = G == 256 ? sb : 2 * sb + (blk >> 2);
  __half* sums = reinterpret_cast<__half*>(row + split_sums_offset(K)) + static_cast<size_t>(grp) * 16;
  if (l4 < (G == 256 ? 1 : 2)) {
    __half* mine = sums + (G == 256 ? blk >> 1 : 2 * l4 + ((blk >> 1) & 1)) * 4 + (blk & 1);
    const __half h = __float2half_rn(sum);
    mine[0] = h;
    mine[2] = __float2half_rn(sum - __half2float(h));
  } else if (l4 == 2 && (blk & (G / 32 - 1)) == 0) {
    reinterpret_cast<float*>(row + split_scale_offset(K, G))[grp] = dm;
  }
}

// Batched activation rows in split form (G = 256), one warp per super-block; CTA (0, 0) also writes the group list of
// a single-matrix call: `cap` consecutive rows per group.
template <class SRC>
__global__ void split_rows_kernel(const SRC* src, size_t ld, int nrows, int K, uint8_t* dst, size_t pitch, int4* groups,
                                  int* n_groups, int cap) {
  pdl_chain_entry();
  if (blockIdx.x == 0 && blockIdx.y == 0) {
    const int ng = (nrows + cap - 1) / cap;
    for (int g = threadIdx.x; g < ng; g += blockDim.x) groups[g] = make_int4(0, g * cap, min(cap, nrows - g * cap), 0);
    if (threadIdx.x == 0) *n_groups = ng;
  }
  const int row = blockIdx.y, lane = threadIdx.x & 31, l4 = lane & 3;
  const SRC* x      = src + static_cast<size_t>(row) * ld;
  const bool vec_ok = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int sb = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; sb < K / 256; sb += warps) {
    const int b = sb * 8 + (lane >> 2);
    float v[8];
    load8<SRC>(x, static_cast<size_t>(b) * 32 + l4 * 8, vec_ok, v);
    float d;
    int part, total;
    const uint2 packed = quantize_block_lane8(v, d, part, total);
    split_store_lane8<256>(dst + static_cast<size_t>(row) * pitch, static_cast<size_t>(K), b, packed, d, total);
  }
}
template <class SRC>
static cudaError_t launch_split_rows(const SRC* src, size_t ld, int nrows, int K, uint8_t* dst, int4* groups, int* n_groups,
                                     int cap, cudaStream_t st) {
  const int bx = std::max(1, std::min(8, (K / 256 + 3) / 4));
  return launch_chained(split_rows_kernel<SRC>, dim3(bx, nrows), dim3(128), 0, st, src, ld, nrows, K, dst,
                        split_row_pitch(K, 256), groups, n_groups, cap);
}

// ---- parameters and shared-memory layout ----------------------------------------------------------------
struct alignas(64) SplitParams {
  CUtensorMap one;            // the matrix of a single-matrix call (maps0 == nullptr): boxes of box_rows x one super-block
  const CUtensorMap* maps0;   // per-expert tensor maps (gate / down), boxes of 32 rows
  const CUtensorMap* maps1;   // up (MODE 1)
  int N, K;                   // weight rows of each matrix, elements per row
  int tile_rows;              // weight rows per row tile (<= 128; MODE 1: 128)
  int box_rows, boxes;        // rows of one TMA box, boxes per row tile
  int row_units;              // units along the rows: ceil(N / (tile_rows * row tiles per unit))
  const int4* groups;         // {table index of the expert, first position, activation rows, 0}
  const int* n_groups;
  const int* list;            // slot id at each position (MODE 0 by slot, MODE 1)
  int S;                      // slots per token
  const uint8_t* xrows;       // split activation rows: MODE 0, 2 by position, MODE 1 by slot / S
  size_t x_pitch;
  void* dst;                  // MODE 0: float [npos, N]; MODE 2: YT [npos, ld_dst]
  size_t ld_dst;
  int round_bf16;             // MODE 1: Scalar = bf16
  uint8_t* qdst;              // MODE 1: split rows (G = 128) by position
  size_t q_pitch;
  int* status;
  PeerOut po;                 // MODE 0: po.out != null writes the rows into this rank's slot-indexed buffer
};

template <int MODE, int PAIR, int NH, int KH>
struct SpLayout {
  static constexpr bool kEx = MODE == 1 || PAIR == 1;       // the drain warpgroups exchange a tile
  static constexpr int kNT = 32 * NH;                       // activation rows per unit
  // Weight stages (one row tile x one super-block each): an EVEN number, so that a stage always belongs to the same
  // unpack warpgroup and its barrier's phases are all seen by the threads that wait on it.
  static constexpr int kW = NH == 1 && !kEx ? 6 : 4;
  static constexpr int kB = NH == 1 ? 3 : 2;                // activation stages (one super-block each)
  static constexpr uint32_t kWStage = 128 * 144;
  static constexpr uint32_t kBK = 2 * kNT * 128;            // 64 elements of K: hi and mid rows in groups of eight
  static constexpr uint32_t kBStage = 4 * kBK;
  static constexpr uint32_t scl = KH * kNT * 32;            // inside a stage's block sums and scales
  static constexpr uint32_t kSStage = scl + KH * kNT * 4;
  static constexpr uint32_t b = 0;
  static constexpr uint32_t w = b + kB * kBStage;
  static constexpr uint32_t sums = w + kW * kWStage;
  static constexpr uint32_t dd = sums + kB * kSStage;       // [4 tiles][128 rows] {d / 256, e / 16}
  static constexpr uint32_t ex = dd + 4 * 128 * 8;          // MODE 1: [NH][gate, up][kExRows][kSpExPitch] float; PAIR 1: [32][kSpExPitch]
  static constexpr int kExRows = 16 / NH;
  static constexpr uint32_t rowp = ex + (kEx ? 32 * kSpExPitch * 4 : 0);
  static constexpr uint32_t bar = rowp + kNT * 8;
  static constexpr uint32_t total = bar + 320 + 1024;       // + slack for the 1024-byte alignment of the base
};

// ---- PTX wrappers ---------------------------------------------------------------------------------------
// K-major operand, 128-byte swizzle: eight rows of 128 bytes per 1024-byte atom, next eight rows +1024
__device__ __forceinline__ uint64_t sp_desc_sw128(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) |
         (uint64_t(1) << 46) | (uint64_t(2) << 61);
}
// D = F32, A = B = F16, K-major, M = 128
__device__ __forceinline__ uint32_t sp_idesc(int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void sp_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0)
      : "memory");
}
__device__ __forceinline__ void sp_st32(uint32_t t, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
      "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
      "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
      "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
// two and four words, each twice
__device__ __forceinline__ void sp_st2x2(uint32_t t, uint32_t a, uint32_t b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%1,%2,%2};" ::"r"(t), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sp_st4x2(uint32_t t, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%2,%2,%3,%3,%4,%4};" ::"r"(t), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void sp_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- unpack ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
constexpr uint32_t kH2Magic = 0x64006400u;   // {1024, 1024}: the low four mantissa bits count units, the next four sixteens
// 64 elements (32 bytes: low nibbles = one sub-block, high nibbles = the next) -> 32 words of pairs sc * q - t, each in one
// exact fp16 fma: (1024 + q) * sc - fp16(1031 sc), an integer of at most 520, and (1024 + 16 q) * (sc / 16) - 72 sc.
__device__ __forceinline__ void sp_unpack64(const uint4& a, const uint4& b, uint32_t sc_pair4, int j, uint32_t (&o)[32]) {
  const uint32_t s0 = h2_sub(__byte_perm(sc_pair4, 0x64646464u, 0x4040u + 0x0101u * j), kH2Magic);
  const uint32_t s1 = h2_sub(__byte_perm(sc_pair4, 0x64646464u, 0x4040u + 0x0101u * (j + 1)), kH2Magic);
  const uint32_t c0 = h2_mul(s0, 0xE407E407u);      // -1031 * sc, rounded
  const uint32_t c1 = h2_mul(s1, 0xD480D480u);      // -72 * sc'
  const uint32_t s1d = h2_mul(s1, 0x2C002C00u);     // sc' / 16
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t u = w[i] >> 8;
    o[2 * i]          = h2_fma((w[i] & 0x000F000Fu) | kH2Magic, s0, c0);
    o[2 * i + 1]      = h2_fma((u & 0x000F000Fu) | kH2Magic, s0, c0);
    o[16 + 2 * i]     = h2_fma((w[i] & 0x00F000F0u) | kH2Magic, s1d, c1);
    o[16 + 2 * i + 1] = h2_fma((u & 0x00F000F0u) | kH2Magic, s1d, c1);
  }
}
__device__ __forceinline__ float2 h2_to_f2(uint32_t h) { return __half22float2(*reinterpret_cast<const __half2*>(&h)); }
__device__ __forceinline__ uint32_t f2_to_h2(float2 f) {
  const __half2 h = __float22half2_rn(f);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// c / e of the same two sub-blocks in two fp16 parts; nd = -d / e, ndm = -dmin / e. -t is what the fma above leaves for q = 0.
template <int J>
__device__ __forceinline__ void sp_offsets(uint32_t sc_pair4, uint32_t mn_pair4, float2 nd, float2 ndm, uint32_t& hi, uint32_t& lo) {
  const uint32_t sc = h2_sub(__byte_perm(sc_pair4, 0x64646464u, J == 0 ? 0x4140u : 0x4342u), kH2Magic);
  const uint32_t mn = h2_sub(__byte_perm(mn_pair4, 0x64646464u, J == 0 ? 0x4140u : 0x4342u), kH2Magic);
  const uint32_t nt = h2_fma(sc, 0x00006400u, h2_mul(sc, 0xC800E407u));   // {1024 sc - fp16(1031 sc), -8 sc'}
  const float2 c = ffma2(ndm, h2_to_f2(mn), fmul2(nd, h2_to_f2(nt)));
  hi = f2_to_h2(c);
  const float2 h = h2_to_f2(hi);
  lo = f2_to_h2(fadd2(c, make_float2(-h.x, -h.y)));
}

// Eight activation rows of one TMEM lane, one group of K: acc += D * (d * (hi + mid) + e * c).
__device__ __forceinline__ void sp_fold8(float* acc, const int (&p)[16], const int (&m)[8], const float* scale, float2 d2, float2 e2) {
  const float4 s0 = *reinterpret_cast<const float4*>(scale), s1 = *reinterpret_cast<const float4*>(scale + 4);
  const float2 s[4] = {make_float2(s0.x, s0.y), make_float2(s0.z, s0.w), make_float2(s1.x, s1.y), make_float2(s1.z, s1.w)};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = fadd2(make_float2(__int_as_float(p[2 * i]), __int_as_float(p[2 * i + 1])),
                     make_float2(__int_as_float(p[8 + 2 * i]), __int_as_float(p[9 + 2 * i])));
    t = ffma2(e2, make_float2(__int_as_float(m[2 * i]), __int_as_float(m[2 * i + 1])), fmul2(d2, t));
    const float2 r = ffma2(s[i], t, make_float2(acc[2 * i], acc[2 * i + 1]));
    acc[2 * i] = r.x;
    acc[2 * i + 1] = r.y;
  }
}

__device__ __forceinline__ bool sp_elect() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0;
}
// The products of one group of K (256 / KH elements of a tile) with 8 * n8 activation rows: the MMAs for hi and mid,
// then c: its high and low parts in turn, or (KH = 2) both for the group's four blocks. bk: the group's activation operand, ms: its block sums.
template <int KH, uint32_t BK>
__device__ __forceinline__ void sp_group(uint32_t td, uint32_t ta, uint32_t tc, uint32_t bk, uint32_t ms, int n8) {
  const uint64_t bd = sp_desc_sw128(bk);
  const uint32_t id = sp_idesc(16 * n8);
#pragma unroll
  for (int j = 0; j < 16 / KH; ++j) sp_mma(td, ta + 8 * j, bd + (((j >> 2) * BK + (j & 3) * 32) >> 4), id, j != 0);
  sp_mma(td + 64, tc, tc_desc(ms), sp_idesc((8 * n8 + 15) & ~15), 0u);
  if (KH == 1) sp_mma(td + 64, tc + 8, tc_desc(ms), sp_idesc((8 * n8 + 15) & ~15), 1u);
}

// MODE 0: dst[pos, j] = W0[j,:] . x[pos,:]                               (down projection)
// MODE 1: split row of Scalar(silu(W0 . x) * (W1 . x)) at qdst[pos]       (gate / up + SwiGLU + quantization)
// MODE 2: dst[pos, j] = YT(W0[j,:] . x[pos,:])                            (plain batched GEMM)
// KH: groups of K per super-block (G = 256 / KH); NH: 32-row halves of the activation rows of a unit.
template <int MODE, int PAIR, int NH, int KH, class YT>
__global__ void __launch_bounds__(kSpThreads, 1) grouped_split_q4k_kernel(const __grid_constant__ SplitParams p) {
  static_assert(MODE != 1 || PAIR == 2, "gate and up are the two row tiles of a unit");
  static_assert(PAIR == 2 || NH == 1, "one row tile: up to 32 activation rows");
  using L = SpLayout<MODE, PAIR, NH, KH>;
  constexpr int kW = L::kW, kB = L::kB, kNT = L::kNT, G = 256 / KH;
  constexpr int kU = 4 / NH;                   // unpack warpgroups; drain: 2 NH
  extern __shared__ __align__(1024) uint8_t sp_smem_raw[];
  const uint32_t base = (smem_u32(sp_smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = sp_smem_raw + (base - smem_u32(sp_smem_raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const uint32_t bars = base + L::bar;
  auto w_full  = [&](int s) { return bars + 8u * s; };
  auto w_empty = [&](int s) { return bars + 48u + 8u * s; };
  auto b_full  = [&](int s) { return bars + 96u + 8u * s; };
  auto b_empty = [&](int s) { return bars + 120u + 8u * s; };
  auto a_full  = [&](int par) { return bars + 144u + 8u * par; };
  auto a_empty = [&](int par) { return bars + 160u + 8u * par; };
  auto d_full  = [&](int par, int d) { return bars + 176u + 8u * (2 * par + d); };   // per tile parity: its drain warps see every phase
  auto d_empty = [&](int d) { return bars + 208u + 8u * d; };
  auto ex_full  = [&](int hh) { return bars + 224u + 8u * hh; };
  auto ex_empty = [&](int hh) { return bars + 240u + 8u * hh; };
  const uint32_t mma_end = bars + 256u;
  uint32_t* tmem_slot      = reinterpret_cast<uint32_t*>(smem + L::bar + 288);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::bar + 292);
  RingArmed* ring_end      = reinterpret_cast<RingArmed*>(smem + L::bar + 296);   // what the weight loader armed last

  if (warp == kSpWarpMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kW; ++s) { mbar_init(w_full(s), 1); mbar_init(w_empty(s), 2 * kU); }
    for (int s = 0; s < kB; ++s) { mbar_init(b_full(s), 32); mbar_init(b_empty(s), 1 + 4 * NH * PAIR); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(a_full(i), 2 * kU);
      mbar_init(a_empty(i), 1);
      mbar_init(d_full(0, i), 1);
      mbar_init(d_full(1, i), 1);
      mbar_init(d_empty(i), 4);
      mbar_init(ex_full(i), MODE == 1 ? 8 : 4);
      mbar_init(ex_empty(i), MODE == 1 ? 8 : 4);
    }
    mbar_init(mma_end, 1);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  tc_before();
  __syncthreads();
  tc_after();
  // all 512 columns are ours, so the allocation starts at column 0: a constant in every address below
  constexpr uint32_t tmem = 0;
  if (*tmem_slot != tmem) *abort_flag = 1;   // (cannot happen; every wait below then gives up)
  pdl_launch_dependents();
  pdl_wait();

  // Bounded wait of a whole warp; the vote makes the verdict, and the control flow behind it, uniform.
  auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
    for (uint32_t i = 0; i < (1u << 21); ++i) {
      if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
      if ((i & 31u) == 31u && __any_sync(0xffffffffu, *abort_flag != 0)) return false;
    }
    *abort_flag = 1;
    return false;
  };

  const int n_groups = __reduce_max_sync(0xffffffffu, ld_dep(p.n_groups));   // (a warp reduction: uniform to the compiler)
  const int units = n_groups * p.row_units;
  const int nsb = p.K / 256;
  const int tiles_u = nsb * PAIR;    // tiles (row tile x super-block) per unit
  const int my_units = static_cast<int>(blockIdx.x) < units ? (units - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1 : 0;
  auto group_of = [&](int i) {       // group record of this CTA's i-th unit
    const int u = blockIdx.x + i * gridDim.x;
    return i < my_units ? ld_dep(p.groups + u / p.row_units) : make_int4(0, 0, 0, 0);
  };
  bool ok = true;

  if (warp < 4 * kU) {
    // ------------------------------------------------------------------ unpack (lane = weight row of the tile)
    const int par = (warp >> 2) & 1, q = warp & 3, row = q * 32 + lane;
    const int g_lo = kU == 4 ? (warp >> 3) * 2 : 0, g_hi = kU == 4 ? g_lo + 2 : 4;   // 64-element groups of the super-block
    const bool live = q * 32 < p.tile_rows;     // warps past the tile's rows only keep the barriers moving
    const uint32_t ta = tmem + (static_cast<uint32_t>(q * 32) << 16) + kSpTmemA + par * 128;
    const uint32_t tc = tmem + (static_cast<uint32_t>(q * 32) << 16) + kSpTmemC + par * 16;
    const int total = my_units * tiles_u;
    int s = par;
    uint32_t ph = 0, k = 0;                      // weight stage and its phase; this parity's tile count
    for (int t = par; t < total; t += 2, ++k) {
      if (!wait(w_full(s), ph)) { ok = false; break; }
      const uint8_t* mine = smem + L::w + s * L::kWStage + row * 144;
      const uint4 hdr = *reinterpret_cast<const uint4*>(mine);
      uint4 qa = *reinterpret_cast<const uint4*>(mine + 16 + 32 * g_lo), qb = *reinterpret_cast<const uint4*>(mine + 32 + 32 * g_lo);
      // scales and mins of this warp's sub-blocks: four of the eight when there are four warpgroups
      const uint32_t sc_lo = hdr.y & 0x3F3F3F3Fu, sc_hi = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
#pragma unroll 1
      for (int g = g_lo; g < g_hi; ++g) {
        const uint4 ca = qa, cb = qb;
        if (g + 1 < g_hi) {
          qa = *reinterpret_cast<const uint4*>(mine + 48 + 32 * g);
          qb = *reinterpret_cast<const uint4*>(mine + 64 + 32 * g);
        }
        uint32_t o[32];
        if (live) sp_unpack64(ca, cb, g < 2 ? sc_lo : sc_hi, 2 * (g & 1), o);
        if (g == g_lo) {   // (the first group is formed while the previous tile's MMAs still read the buffer)
          if (!wait(a_empty(par), (k & 1u) ^ 1u)) { ok = false; break; }
          tc_after();
        }
        if (live) {
          sp_st32(ta + 32 * g, o);
        }
      }
      if (!ok) break;
      const uint32_t mn_lo = hdr.z & 0x3F3F3F3Fu, mn_hi = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
      // e: the power of two below the larger of 520 |d| and 63 |dmin|, so |c / e| < 4
      const float2 dw = h2_to_f2(hdr.x);
      const float em = fmaxf(fmaxf(520.0f * fabsf(dw.x), 63.0f * fabsf(dw.y)), 0x1p-40f);
      const float e = __uint_as_float(__float_as_uint(em) & 0x7F800000u), re = __uint_as_float(0x7F000000u - __float_as_uint(e));
      const float2 nd = make_float2(-dw.x * re, -dw.x * re), ndm = make_float2(-dw.y * re, -dw.y * re);
      if (live) {
        uint32_t ch[4], cl[4];
        sp_offsets<0>(g_lo == 0 ? sc_lo : sc_hi, g_lo == 0 ? mn_lo : mn_hi, nd, ndm, ch[0], cl[0]);
        sp_offsets<1>(g_lo == 0 ? sc_lo : sc_hi, g_lo == 0 ? mn_lo : mn_hi, nd, ndm, ch[1], cl[1]);
        if (kU == 2) {
          sp_offsets<0>(sc_hi, mn_hi, nd, ndm, ch[2], cl[2]);
          sp_offsets<1>(sc_hi, mn_hi, nd, ndm, ch[3], cl[3]);
        }
        if (kU == 4) {   // this warpgroup's two groups: blocks 0 to 3 or 4 to 7
          if (KH == 1) { sp_st2x2(tc + 2 * g_lo, ch[0], ch[1]); sp_st2x2(tc + 8 + 2 * g_lo, cl[0], cl[1]); }
          else sp_st4x2(tc + 4 * g_lo, ch[0], ch[1], cl[0], cl[1]);
        } else if (KH == 1) {
          sp_st4x2(tc, ch[0], ch[1], ch[2], ch[3]);
          sp_st4x2(tc + 8, cl[0], cl[1], cl[2], cl[3]);
        } else {
          sp_st4x2(tc, ch[0], ch[1], cl[0], cl[1]);
          sp_st4x2(tc + 8, ch[2], ch[3], cl[2], cl[3]);
        }
        if (g_lo == 0) reinterpret_cast<float2*>(smem + L::dd)[(t & 3) * 128 + row] = make_float2(dw.x * 0x1p-8f, e * 0.0625f);
      }
      sp_wait_st();
      tc_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(a_full(par));
        mbar_arrive(w_empty(s));
      }
      s += 2;
      if (s >= kW) { s -= kW; ph ^= 1u; }
    }
  } else if (warp < kSpWarpMma) {
    // ------------------------------------------------------------------ drain + epilogue
    const int dw = (warp >> 2) - kU, par = dw & 1, hh = dw >> 1, q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
    int4 gi_next = group_of(0);
    uint32_t round = 0, k = 0;                   // exchange rounds; this parity's tile count
    int bs = 0;
    for (int ui = 0; ui < my_units && ok; ++ui) {
      const int4 gi = gi_next;
      gi_next = group_of(ui + 1);
      const int u = blockIdx.x + ui * gridDim.x, ru = u % p.row_units;
      const int nh = min(32, max(0, gi.z - 32 * hh)), n8 = (nh + 7) >> 3;   // this thread's activation rows
      float acc[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) acc[c] = 0.f;
      for (int sb = 0; sb < nsb && ok; ++sb) {
        const int t = ui * tiles_u + (PAIR == 2 ? 2 * sb + par : sb);
        if (PAIR == 2 || (t & 1) == par) {
          const float* scl = reinterpret_cast<const float*>(smem + L::sums + bs * L::kSStage + L::scl) + hh * 32;
#pragma unroll 1
          for (int kh = 0; kh < KH; ++kh) {
            // columns: one buffer per half of the activation rows, else per group of K, else per tile parity; this
            // parity's uses of a buffer: one per tile, two when both halves and both groups exist
            const int buf = NH == 2 ? hh : KH == 2 ? kh : par;
            const uint32_t use = NH * KH == 4 ? k * 2 + kh : k;
            if (!wait(d_full(par, buf), use & 1u)) { ok = false; break; }
            tc_after();
            const float2 dd = reinterpret_cast<const float2*>(smem + L::dd)[(t & 3) * 128 + row];
            const float2 d2 = make_float2(dd.x, dd.x), e2 = make_float2(dd.y, dd.y);
            const uint32_t td = lane_base + buf * 96;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (c < n8) {
                int p0[16], m0[8];
                tc_ld16(td + 16 * c, p0);
                tc_ld8(td + 64 + 8 * c, m0);
                tc_wait_ld();
                sp_fold8(acc + 8 * c, p0, m0, scl + kh * kNT + 8 * c, d2, e2);
              }
            }
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty(buf));
          }
          if (!ok) break;
          if (lane == 0) mbar_arrive(b_empty(bs));   // done with this stage's scales
          ++k;
        }
        if (++bs == kB) bs = 0;
      }
      if (!ok) break;
      // ---- epilogue ----
      float* ex = reinterpret_cast<float*>(smem + L::ex);
      if (MODE == 1) {
        // kExRows activation rows at a time: gate and up sums meet in shared memory, then sixteen lanes per
        // activation row form the activation of 128 columns (one group of the down projection's rows), apply the
        // reference's per-32 quantizer and write the split row the down projection reads
        constexpr int R = L::kExRows;
        float* exh = ex + hh * (2 * R * kSpExPitch);
#pragma unroll
        for (int r = 0; r < 32 / R; ++r) {
          const int nr = nh - R * r;
          if (nr <= 0) continue;
          if (!wait(ex_empty(hh), (round & 1u) ^ 1u)) { ok = false; break; }
#pragma unroll
          for (int c = 0; c < R; ++c) exh[(par * R + c) * kSpExPitch + row] = acc[r * R + c];
          __syncwarp();
          if (lane == 0) mbar_arrive(ex_full(hh));
          if (!wait(ex_full(hh), round & 1u)) { ok = false; break; }
          const int tok0 = (par * 4 + q) * 2, tk = min(tok0 + (lane >> 4), nr - 1);   // a row past the end repeats the last one
          if (tok0 < min(nr, R)) {
            const float* eg = exh + tk * kSpExPitch + (lane & 15) * 8;
            const float* eu = eg + R * kSpExPitch;
            float g8[8], u8[8], v[8];
#pragma unroll
            for (int i = 0; i < 8; i += 4) {
              *reinterpret_cast<float4*>(g8 + i) = *reinterpret_cast<const float4*>(eg + i);
              *reinterpret_cast<float4*>(u8 + i) = *reinterpret_cast<const float4*>(eu + i);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              v[i] = (g8[i] / (1.0f + expf(-g8[i]))) * u8[i];
              if (p.round_bf16) v[i] = __bfloat162float(__float2bfloat16_rn(v[i]));
            }
            float d;
            int part, sum;
            const uint2 packed = quantize_block_lane8(v, d, part, sum);
            split_store_lane8<128>(p.qdst + static_cast<size_t>(gi.y + hh * 32 + r * R + tk) * p.q_pitch, static_cast<size_t>(p.N),
                                   ru * 4 + ((lane & 15) >> 2), packed, d, sum);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(ex_empty(hh));
          ++round;
        }
      } else {
        if (PAIR == 1) {   // the two parities' sums meet; parity 0 stores
          if (par == 1) {
            if (!wait(ex_empty(0), (round & 1u) ^ 1u)) { ok = false; break; }
#pragma unroll
            for (int c = 0; c < 32; ++c)
              if (c < nh) ex[c * kSpExPitch + row] = acc[c];
            __syncwarp();
            if (lane == 0) mbar_arrive(ex_full(0));
          } else {
            if (!wait(ex_full(0), round & 1u)) { ok = false; break; }
#pragma unroll
            for (int c = 0; c < 32; ++c)
              if (c < nh) acc[c] += ex[c * kSpExPitch + row];
            __syncwarp();
            if (lane == 0) mbar_arrive(ex_empty(0));
          }
          ++round;
        }
        const int j = (ru * PAIR + (PAIR == 2 ? par : 0)) * p.tile_rows + row;
        if ((PAIR == 2 || par == 0) && row < p.tile_rows && j < p.N) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if (c < nh) {
              const size_t ps = static_cast<size_t>(gi.y + hh * 32 + c);
              if (MODE == 2) store_scalar(static_cast<YT*>(p.dst) + ps * p.ld_dst + j, acc[c]);
              else if (p.po.out != nullptr) peer_out_row(p.po, ld_dep(p.list + ps), p.N)[j] = acc[c];
              else static_cast<float*>(p.dst)[ps * p.N + j] = acc[c];
            }
          }
        }
      }
    }
  } else if (warp == kSpWarpMma) {
    // ------------------------------------------------------------------ MMA issue
    const bool leader = sp_elect();
    int nt_next = group_of(0).z;
    int bs = 0;
    uint32_t bph = 0, t = 0;           // activation stage and its phase, tile number
    for (int ui = 0; ui < my_units && ok; ++ui) {
      const int nt = __reduce_max_sync(0xffffffffu, nt_next);
      nt_next = group_of(ui + 1).z;
      for (int sb = 0; sb < nsb && ok; ++sb) {
        const uint32_t bst = base + L::b + bs * L::kBStage, sst = base + L::sums + bs * L::kSStage;
        if (!wait(b_full(bs), bph)) { ok = false; break; }
        fence_proxy_async();           // the activation rows were written by cp.async (generic proxy)
#pragma unroll 1
        for (int m = 0; m < PAIR; ++m, ++t) {
          const uint32_t par = t & 1u;
          const uint32_t ta = kSpTmemA + par * 128, tc = kSpTmemC + par * 16;
          if (!wait(a_full(par), (t >> 1) & 1u)) { ok = false; break; }
#pragma unroll 1
          for (int sub = 0; sub < NH * KH; ++sub) {
            const int hh = NH == 2 ? sub & 1 : 0, kh = KH == 2 ? sub / NH : 0;
            const uint32_t s = t * (NH * KH) + sub, buf = s & 1u;   // the two buffers take turns
            if (!wait(d_empty(buf), ((s >> 1) & 1u) ^ 1u)) { ok = false; break; }
            tc_after();
            const int n8 = (min(32, max(0, nt - 32 * hh)) + 7) >> 3;
            if (leader) {
              const uint32_t bk = bst + hh * 8192 + kh * (2 * L::kBK), ms = sst + kh * (kNT * 32) + hh * 1024;
              if (n8 > 0) sp_group<KH, L::kBK>(buf * 96, ta + kh * 64, tc + kh * 8, bk, ms, n8);
              if (sub == NH * KH - 1) {
                tc_commit(a_empty(par));
                if (m == PAIR - 1) tc_commit(b_empty(bs));
              }
              tc_commit(d_full(par, buf));
            }
            __syncwarp();
          }
          if (!ok) break;
        }
        if (++bs == kB) { bs = 0; bph ^= 1u; }
      }
    }
  } else if (warp == kSpWarpW) {
    // ------------------------------------------------------------------ weights
    const bool leader = sp_elect();
    int e_next = group_of(0).x, s = 0;
    uint32_t ph = 1;
    RingArmed ring;
    for (int ui = 0; ui < my_units && ok; ++ui) {
      const int e = e_next;             // requested a unit ago
      e_next = group_of(ui + 1).x;
      const int u = blockIdx.x + ui * gridDim.x, ru = u % p.row_units;
      const CUtensorMap* m0 = p.maps0 ? p.maps0 + e : &p.one;
      const CUtensorMap* m1 = MODE == 1 ? p.maps1 + e : m0;
      if (leader && p.maps0) {
        tensormap_acquire(m0);
        if (MODE == 1) tensormap_acquire(m1);
      }
      for (int sb = 0; sb < nsb && ok; ++sb) {
#pragma unroll
        for (int m = 0; m < PAIR; ++m) {
          if (!wait(w_empty(s), ph)) { ok = false; break; }
          ring.arm(s, ph ^ 1u);
          if (leader) {
            const CUtensorMap* mp = MODE == 1 && m == 1 ? m1 : m0;
            const int r0 = (MODE == 1 ? ru : ru * PAIR + m) * p.tile_rows;
            const uint32_t dst = base + L::w + s * L::kWStage;
            mbar_expect_tx(w_full(s), static_cast<uint32_t>(p.boxes * p.box_rows) * 144u);
            for (int bx = 0; bx < p.boxes; ++bx)
              tma_load_2d(dst + bx * p.box_rows * 144, mp, sb * 144, r0 + bx * p.box_rows, w_full(s));
          }
          __syncwarp();
          if (++s == kW) { s = 0; ph ^= 1u; }
        }
      }
    }
    if (lane == 0) *ring_end = ring;
  } else if (warp == kSpWarpX) {
    // ------------------------------------------------------------------ activation rows
    unsigned long long* rowp = reinterpret_cast<unsigned long long*>(smem + L::rowp);
    // Metadata runs ahead so that no load waits for another on the way: the group record of unit i + 2 and the row
    // ids of unit i + 1 are requested when unit i is entered.
    int4 gi = group_of(0), gi1 = group_of(1);
    auto row_of = [&](const int4& g, int n) -> int {     // activation row of the group's n-th position (rows past the end: the last)
      const int ps = g.y + min(n, max(g.z - 1, 0));
      return MODE == 1 && g.z > 0 ? ld_dep(p.list + ps) / p.S : ps;
    };
    int rows[NH], rows1[NH];
#pragma unroll
    for (int hh = 0; hh < NH; ++hh) rows[hh] = row_of(gi, lane + 32 * hh);
    int bs = 0;
    uint32_t ph = 1;
    const int c = lane & 7, nl = lane >> 3;
    for (int ui = 0; ui < my_units && ok; ++ui) {
      const int4 gi2 = group_of(ui + 2);
#pragma unroll
      for (int hh = 0; hh < NH; ++hh) rows1[hh] = row_of(gi1, lane + 32 * hh);
      __syncwarp();
#pragma unroll
      for (int hh = 0; hh < NH; ++hh)
        rowp[lane + 32 * hh] = reinterpret_cast<unsigned long long>(p.xrows + static_cast<size_t>(rows[hh]) * p.x_pitch);
      __syncwarp();
      const int n8 = (__reduce_max_sync(0xffffffffu, gi.z) + 7) >> 3;
      for (int sb = 0; sb < nsb; ++sb) {
        if (!wait(b_empty(bs), ph)) { ok = false; break; }
        const uint32_t bst = base + L::b + bs * L::kBStage, sst = base + L::sums + bs * L::kSStage;
#pragma unroll 2
        for (int g = 0; g < n8; ++g) {            // eight activation rows: two steps of four rows x 128 bytes per (kb, part)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = 4 * i + nl;             // row inside its group of eight
            const uint8_t* src = reinterpret_cast<const uint8_t*>(rowp[8 * g + r]) + static_cast<size_t>(sb) * 1024 + c * 16;
            const uint32_t dst = bst + g * 2048 + r * 128 + ((c ^ r) << 4);
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
              cp_async16(dst + kb * L::kBK, src + kb * 128, true);
              cp_async16(dst + kb * L::kBK + 1024, src + 512 + kb * 128, true);
            }
          }
        }
        for (int i = lane; i < 8 * n8; i += 32) {   // one lane per activation row: its block sums and scales
          const uint8_t* row = reinterpret_cast<const uint8_t*>(rowp[i]);
          const uint8_t* sums = row + split_sums_offset(p.K) + static_cast<size_t>(sb) * (KH * 32);
          const uint8_t* scl = row + split_scale_offset(p.K, G) + static_cast<size_t>(sb) * (KH * 4);
#pragma unroll
          for (int h = 0; h < KH; ++h) {
            const uint32_t d = sst + h * (kNT * 32) + (i >> 3) * 256 + (i & 7) * 16;
            cp_async16(d, sums + h * 32, true);
            cp_async16(d + 128, sums + h * 32 + 16, true);
            cp_async4(sst + L::scl + (h * kNT + i) * 4, scl + h * 4, true);
          }
        }
        cp_async_arrive(b_full(bs));
        if (++bs == kB) { bs = 0; ph ^= 1u; }
      }
      gi = gi1;
      gi1 = gi2;
#pragma unroll
      for (int hh = 0; hh < NH; ++hh) rows[hh] = rows1[hh];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  if (!ok && lane == 0) atomicExch(p.status, KDNN_ERR_DEVICE_WAIT);
  if (MODE == 0) peer_out_finish(p.po, gridDim.x);
  tc_before();
  __syncthreads();
  if (*abort_flag) {
    // some role gave up: the copies and MMAs still in flight end (bounded) before the CTA gives its memory back
    if (warp == kSpWarpW && lane == 0)
      ring_drain(*ring_end, kW, 1u << 14, [&](int s, uint32_t parity) { return mbar_try_wait(w_full(s), parity); });
    if (warp == kSpWarpMma && sp_elect()) {
      tc_commit(mma_end);
      mbar_wait_bounded(mma_end, 0u, 1u << 16);
    }
    __syncthreads();
  }
  if (warp == kSpWarpMma)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "r"(512u) : "memory");
}

template <int MODE, int PAIR, int NH, int KH, class YT>
static cudaError_t launch_grouped_split(const SplitParams& p, int max_units, cudaStream_t st) {
  using L = SpLayout<MODE, PAIR, NH, KH>;
  static_assert(L::total <= 232448, "one CTA's shared memory");
  auto kern = grouped_split_q4k_kernel<MODE, PAIR, NH, KH, YT>;
  static SmemAttrOnce once;
  const cudaError_t e = set_max_smem_once(once, kern, (int)L::total);
  if (e != cudaSuccess) return e;
  return launch_chained(kern, dim3((unsigned)std::max(1, std::min(device_sm_count(), max_units))), dim3(kSpThreads), L::total, st, p);
}

}  // namespace kdnn
