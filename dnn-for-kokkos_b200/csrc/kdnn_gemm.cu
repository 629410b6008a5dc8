// Batched GEMV / skinny GEMM Y[M,N] = X[M,K] W[N,K]^T with packed W and per-row int8 activations; row m of Y is the
// decode GEMV applied to row m, up to the order of fp32 sums. Up to three rows run as GEMVs; Q4_K runs on kdnn_split.cuh (the
// integer kernels of kdnn_tc.cuh and kdnn_mma.cuh where that does not apply), the other formats on kdnn_rowmma.cuh, and what
// neither takes on the grouped kernel of kdnn_grouped.cuh with one group that holds all rows.
#include "kdnn_grouped.cuh"
#include "kdnn_mma.cuh"
#include "kdnn_rowmma.cuh"
#include "kdnn_split.cuh"
#include "kdnn_tc.cuh"

namespace kdnn {

int tile_kind();
cudaError_t moe_status_ptr(int** out);
cudaError_t gemv_launch(uint32_t dt, const void* w, size_t rows, size_t cols, const void* x, int xs,
                        void* y, int ys, void* scratch, const kdnn_b200_gemv_layout* layout, cudaStream_t stream);

// workspace: [offs: 2 ints, group count | pad to 256][wptr: 1 address | pad to 256][list: M ints][groups][items: M x K/64]
static size_t gemm_groups_offset(size_t M) { return 512 + ((M * sizeof(int) + 255) & ~size_t(255)); }
static size_t gemm_items_offset(size_t M) {
  return gemm_groups_offset(M) + (((M + kTcNT - 1) / kTcNT * sizeof(int4) + 255) & ~size_t(255));
}
// What every call needs: the integer kernels' rows. A workspace of this size is served by them alone.
size_t gemm_workspace_min_bytes(size_t M, size_t K) {
  const size_t a = M * (K / 64) * sizeof(ActItem), b = M * act_row_pitch(K);
  return gemm_items_offset(M) + (a > b ? a : b);
}
// What the faster kernels need as well: split rows (4.14 bytes an element; rowmma_x_bytes of four rows and more is less).
size_t gemm_workspace_bytes(size_t M, size_t K) {
  const size_t least = gemm_workspace_min_bytes(M, K), want = gemm_items_offset(M) + M * split_row_pitch(K, 256);
  return K % 256 == 0 && want > least ? want : least;
}

__global__ void gemm_setup_kernel(int M, uintptr_t w, int* offs, uintptr_t* wptr, int* list, int4* groups) {
  pdl_chain_entry();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    offs[0] = 0;
    offs[1] = M;
    offs[2] = (M + kTcNT - 1) / kTcNT;   // groups of the tensor-core tile kernel: 32 activation rows each
    wptr[0] = w;
  }
  if (i < M) list[i] = i;
  if (i * kTcNT < M) groups[i] = make_int4(0, i * kTcNT, min(kTcNT, M - i * kTcNT), 0);
}

// Weight rows per tile of the tcgen05 kernel for a single matrix: as close to 128 as gives every SM the
// same number of tiles (a 14336-row matrix on 148 SMs: 97 rows, one tile each).
static int gemm_tile_rows(size_t N, size_t groups) {
  const size_t sms = static_cast<size_t>(device_sm_count());
  for (size_t rounds = 1; rounds <= 64; ++rounds) {
    const size_t per = sms * rounds / groups;   // row tiles per group for `rounds` full waves, not one CTA more
    if (per == 0) continue;
    const size_t tr = (N + per - 1) / per;
    if (tr <= 128) return static_cast<int>(tr < 32 ? 32 : tr);
  }
  return 128;
}

// Q4_K rows against M activation rows on the split-fp16 tensor-core kernel: the row quantizer and one tile launch.
// `served` = false: no tensor map for this matrix, nothing was launched.
static cudaError_t gemm_split(const void* w, size_t N, size_t K, const void* X, size_t ldx, size_t M, int xs, void* Y,
                              size_t ldy, int ys, uint8_t* b, bool& served, cudaStream_t st) {
  int* n_groups = reinterpret_cast<int*>(b) + 2;
  int4* groups  = reinterpret_cast<int4*>(b + gemm_groups_offset(M));
  uint8_t* xrows = b + gemm_items_offset(M);
  SplitParams q{};
  cudaError_t err = moe_status_ptr(&q.status);
  if (err != cudaSuccess) return err;
  // Two row tiles per activation stage and 64-row groups once that fills the chip; below, one row tile per CTA, its
  // rows chosen so that every SM gets the same number of tiles, and 32-row groups.
  const size_t sms = static_cast<size_t>(device_sm_count());
  const bool wide = M > 32 && (N + 255) / 256 * ((M + 63) / 64) >= sms;
  const int cap = wide ? 64 : 32;
  const size_t ngroups = (M + cap - 1) / cap;
  q.tile_rows = wide ? 128 : gemm_tile_rows(N, ngroups);
  q.box_rows = q.tile_rows; q.boxes = 1;
  const size_t unit_rows = static_cast<size_t>(q.tile_rows) * (wide ? 2 : 1);
  q.row_units = (int)((N + unit_rows - 1) / unit_rows);
  served = tc_encode_matrix(&q.one, w, N, row_bytes_of(KDNN_GGML_Q4_K, K), q.box_rows) == cudaSuccess;
  if (!served) return cudaSuccess;
  err = xs == KDNN_F32
            ? launch_split_rows<float>(static_cast<const float*>(X), ldx, (int)M, (int)K, xrows, groups, n_groups, cap, st)
            : launch_split_rows<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(X), ldx, (int)M, (int)K, xrows, groups, n_groups, cap, st);
  if (err != cudaSuccess) return err;
  q.N = (int)N; q.K = (int)K; q.groups = groups; q.n_groups = n_groups; q.S = 1;
  q.xrows = xrows; q.x_pitch = split_row_pitch(K, 256); q.dst = Y; q.ld_dst = ldy;
  const int units = (int)(ngroups * q.row_units);
  if (wide) return ys == KDNN_F32 ? launch_grouped_split<2, 2, 2, 1, float>(q, units, st) : launch_grouped_split<2, 2, 2, 1, __nv_bfloat16>(q, units, st);
  return ys == KDNN_F32 ? launch_grouped_split<2, 1, 1, 1, float>(q, units, st) : launch_grouped_split<2, 1, 1, 1, __nv_bfloat16>(q, units, st);
}

// Whether the split kernel is the faster one for more than eight rows: with few super-blocks of K its fixed cost (tensor memory,
// ring fill, the quantizer's larger rows) is not earned back, except where the mma.sync kernel needs another pass of 32 rows or
// its 128-row CTAs leave most of the chip idle. mma.sync / split in us:
//   K = 512    14336 x: 16 rows 10.2 / 11.6, 64 rows 15.3 / 16.1, 160 rows 25.5 / 21.2;  4096 x: 96 rows 11.0 / 11.8, 160 rows 17.3 / 15.1
//   K = 1024   14336 x: 16 rows 13.0 / 14.7, 32 rows 15.9 / 16.0, 48 rows 18.3 / 21.2, 96 rows 30.0 / 29.3;  512 x: 16 rows 11.0 / 10.8
//   K = 1536   14336 x: 16 rows 15.8 / 16.1, 24 rows 17.6 / 16.9;  8192 x: 9 rows 14.9 / 15.7, 48 rows 19.3 / 17.6
//   K = 4096   14336 x: 16 rows 28.9 / 25.7, 32 rows 37.1 / 28.8, 64 rows 57 / 47
static bool gemm_split_pays(size_t M, size_t N, size_t K) {
  if (M <= 8) return true;
  if (K <= 512) return M > 96;
  if (N <= 2048) return true;
  if (K <= 1024) return (M > 24 && M <= 32) || M > 64;
  return K > 1536 || M > 16;
}

template <uint32_t DT>
static cudaError_t gemm_rowmma_dt(const RmParams& p, const void* X, size_t ldx, int xs, uint8_t* xrows, cudaStream_t st) {
  return xs == KDNN_F32 ? launch_rowmma<DT, float>(p, static_cast<const float*>(X), ldx, xrows, st)
                        : launch_rowmma<DT, __nv_bfloat16>(p, static_cast<const __nv_bfloat16*>(X), ldx, xrows, st);
}
static cudaError_t gemm_rowmma(uint32_t dt, const void* w, size_t N, size_t K, const void* X, size_t ldx, size_t M, int xs,
                               void* Y, size_t ldy, int ys, uint8_t* xrows, cudaStream_t st) {
  RmParams p{};
  p.w = static_cast<const uint8_t*>(w);
  p.row_bytes = row_bytes_of(dt, K); p.total = N * p.row_bytes;
  p.N = (int)N; p.M = (int)M; p.blocks = (int)(K / 256);
  p.x = xrows; p.y = Y; p.ldy = ldy; p.y_bf16 = ys == KDNN_BF16;
  if (dt == KDNN_GGML_Q5_K) return gemm_rowmma_dt<KDNN_GGML_Q5_K>(p, X, ldx, xs, xrows, st);
  if (dt == KDNN_GGML_Q6_K) return gemm_rowmma_dt<KDNN_GGML_Q6_K>(p, X, ldx, xs, xrows, st);
  return gemm_rowmma_dt<KDNN_GGML_Q8_0>(p, X, ldx, xs, xrows, st);
}

// `dots` (parity probe, tcgen05 kernel only): int32 [M][N][K/32] raw sub-block dots, or nullptr.
cudaError_t gemm_launch(uint32_t dt, const void* w, size_t N, size_t K, const void* X, size_t ldx,
                        size_t M, int xs, void* Y, size_t ldy, int ys, void* ws, size_t ws_bytes, int32_t* dots,
                        cudaStream_t st) {
  uint8_t* b      = static_cast<uint8_t*>(ws);
  const size_t room = ws_bytes - gemm_items_offset(M);   // bytes for quantized rows
  // Up to three rows one GEMV launch per row is the fastest (14336 x 4096 Q4_K: 6.9 us each, the tile kernels 23 us and up);
  // above, the split-fp16 kernel on Q4_K (8 / 32 rows: 24.5 / 28.7 us; integer tcgen05 27.4 / 42, mma.sync 30 / 37).
  int kind = tile_kind();
  if (kind >= 3 && dots == nullptr) {
    if (M <= 3 && kind == 3) {
      uint8_t* scratch = b + gemm_items_offset(M);   // room for one staged row: the workspace holds M of them
      const size_t xb = xs == KDNN_F32 ? 4 : 2, yb = ys == KDNN_F32 ? 4 : 2;
      for (size_t m = 0; m < M; ++m) {
        const cudaError_t e = gemv_launch(dt, w, N, K, static_cast<const uint8_t*>(X) + m * ldx * xb, xs,
                                          static_cast<uint8_t*>(Y) + m * ldy * yb, ys, scratch, nullptr, st);
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    }
    if (dt == KDNN_GGML_Q4_K && (reinterpret_cast<uintptr_t>(w) & 15u) == 0 && M * split_row_pitch(K, 256) <= room &&
        (kind == 4 || gemm_split_pays(M, N, K))) {
      bool served = false;
      const cudaError_t e = gemm_split(w, N, K, X, ldx, M, xs, Y, ldy, ys, b, served, st);
      if (e != cudaSuccess || served) return e;
    }
    // Every other format whose rows are whole 256-element groups (Q8_0 rows may not be) and start the matrix on 16 bytes
    // (its 16-byte copies step back to that boundary): 4096 x 14336 Q6_K, 16 rows 32.3 us, 433 on the dp4a kernel below.
    if (dt != KDNN_GGML_Q4_K && K % 256 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0 && rowmma_x_bytes(M, K) <= room)
      return gemm_rowmma(dt, w, N, K, X, ldx, M, xs, Y, ldy, ys, b + gemm_items_offset(M), st);
    kind = M <= 8 ? 2 : 1;   // the integer kernels' crossover: 27 against 30 us at 8 rows, 28 against 31 at 16
  } else if (kind >= 3) {
    kind = 2;
  }
  int* offs       = reinterpret_cast<int*>(b);
  uintptr_t* wptr = reinterpret_cast<uintptr_t*>(b + 256);
  int* list       = reinterpret_cast<int*>(b + 512);
  int4* groups    = reinterpret_cast<int4*>(b + gemm_groups_offset(M));
  cudaError_t err = launch_chained(gemm_setup_kernel, dim3((unsigned)((M + 255) / 256)), dim3(256), 0, st, (int)M,
                                   reinterpret_cast<uintptr_t>(w), offs, wptr, list, groups);
  if (err != cudaSuccess) return err;
  if (dt == KDNN_GGML_Q4_K && kind != 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0) {
    uint8_t* xrows = b + gemm_items_offset(M);
    int* status = nullptr;
    err = moe_status_ptr(&status);
    if (err != cudaSuccess) return err;
    err = xs == KDNN_F32
              ? launch_quantize_rows<float>(static_cast<const float*>(X), ldx, (int)M, (int)K, nullptr, xrows, act_row_pitch(K), st)
              : launch_quantize_rows<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(X), ldx, (int)M, (int)K, nullptr, xrows, act_row_pitch(K), st);
    if (err != cudaSuccess) return err;
    if (kind == 2) {
      TcParams t{};
      err = tc_encode_matrix(&t.one, w, N, row_bytes_of(dt, K));
      if (err == cudaSuccess) {
        const size_t ngroups = (M + kTcNT - 1) / kTcNT;
        t.N = (int)N; t.K = (int)K;
        t.tile_rows = gemm_tile_rows(N, ngroups);
        t.row_tiles = (int)((N + t.tile_rows - 1) / t.tile_rows);
        t.groups = groups; t.n_groups = offs + 2; t.list = list; t.S = 1;
        t.xrows = xrows; t.x_pitch = act_row_pitch(K); t.dst = Y; t.ld_dst = ldy; t.status = status;
        t.dots = dots;
        const int tiles = (int)(ngroups * t.row_tiles);
        return ys == KDNN_F32 ? launch_grouped_tc<2, float>(t, tiles, st) : launch_grouped_tc<2, __nv_bfloat16>(t, tiles, st);
      }
      // no tensor-map encoder in this driver: the mma.sync kernel serves the call
    }
    MmaParams q{};
    q.w0 = wptr; q.row_bytes = (int)row_bytes_of(dt, K);
    q.N = (int)N; q.K = (int)K; q.offs = offs; q.list = list; q.S = 1; q.g_first = 0;
    q.xrows = xrows; q.x_pitch = act_row_pitch(K); q.dst = Y; q.ld_dst = ldy; q.status = status;
    q.passes_z = static_cast<int>(M <= 32 ? 1 : (M + 31) / 32 > 4 ? 4 : (M + 31) / 32);
    q.early = M <= 8;   // the row quantizer in front of it is then a handful of CTAs
    return ys == KDNN_F32 ? launch_grouped_mma<2, float>(q, 1, st) : launch_grouped_mma<2, __nv_bfloat16>(q, 1, st);
  }
  ActItem* items = reinterpret_cast<ActItem*>(b + gemm_items_offset(M));
  err = xs == KDNN_F32
            ? launch_quantize_items<float>(dt, static_cast<const float*>(X), ldx, (int)M, (int)K, nullptr, items, st)
            : launch_quantize_items<__nv_bfloat16>(dt, static_cast<const __nv_bfloat16*>(X), ldx, (int)M, (int)K, nullptr, items, st);
  if (err != cudaSuccess) return err;
  GroupedParams p{};
  p.w0 = wptr;
  p.row_bytes0 = (int)row_bytes_of(dt, K);
  p.N = (int)N; p.K = (int)K;
  p.offs = offs; p.list = list; p.S = 1; p.g_first = 0;
  p.src = items; p.dst = Y; p.ld_dst = ldy;
  if (xs == KDNN_F32 && ys == KDNN_F32) return launch_grouped_dt<2, float, float>(dt, p, 1, st);
  if (xs == KDNN_BF16 && ys == KDNN_BF16) return launch_grouped_dt<2, __nv_bfloat16, __nv_bfloat16>(dt, p, 1, st);
  if (xs == KDNN_BF16 && ys == KDNN_F32) return launch_grouped_dt<2, __nv_bfloat16, float>(dt, p, 1, st);
  return launch_grouped_dt<2, float, __nv_bfloat16>(dt, p, 1, st);
}

}  // namespace kdnn
