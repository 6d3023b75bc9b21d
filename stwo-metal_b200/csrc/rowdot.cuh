// Row-wise M31 x QM31 dot products on the tensor cores (sm_100a).
//
// The composition, the FRI quotients and accumulate_numerators all combine
// ~100 column-major columns at every row, S[row] = sum_c W_c f_c[row] with
// QM31 weights: a contraction of depth n_cols with 4 outputs a row.  As an
// 8-bit product (umma.cuh) it is D[row][4 k + j] = sum_(c, b) byte_b(f_c[row])
// byte_j(W_(c,k) 2^(8b) mod P), k = 0..3, j = 0..3: N = 16, K = 4 n_cols, and
// the sums (at most 1024 columns: below 2^29) stay in tensor memory over the
// whole row.  On the integer pipes a cell took 4 wide multiply-adds and
// their folds; here it takes a quarter of a 16-byte load and of a 16-byte
// shared store.  What is left is the memory time of the columns, the latency of
// a chunk's loads (12 warps an SM) and the arithmetic of a tile's rows.
// Measured against the integer-pipe kernels on a shared-memory ring: composition
// of 100 columns of 2^21 points 283 -> 195 us (0.87 GB, 4.5 TB/s), quotients of
// 108 240 -> 190 us (0.94 GB, 4.9 TB/s), numerators of 107 terms at 2^20 168 ->
// 107 us.  Above 160 columns (the quotients, with their tables: 128) the weights
// leave room for two blocks an SM, quotients of 264 columns of 2^20 points 264 ->
// 191 us; above 768 (736) for one, 1024 columns of 2^18 points 265 -> 277 us.
//
// A block of 128 threads owns 512 consecutive rows, thread t rows 4t..4t+3:
// it loads 16 bytes of each of 16 columns, and row 4t + r of 4 of them is one
// 16-byte store into row t of operand r (four products of 128 rows each).
// Chunks of 16 columns alternate between the two halves of the operands'
// 128-byte rows, so a chunk is written while the previous one is multiplied
// and the loads of the next are in flight.
#pragma once
#include <algorithm>

#include "rowops.cuh"
#include "umma.cuh"

namespace stwo_b200 {

constexpr int kDotTileBits = 9, kDotRows = 1 << kDotTileBits;  // rows of a tile
constexpr int kDotThreads = kDotRows / 4;
constexpr int kDotChunk = 16;             // columns of a chunk: half an operand row
constexpr int kDotBlocks = 3;              // blocks of an SM (launch bounds)
constexpr uint32_t kDotMaxCols = 1024;
constexpr uint32_t kDotCols = 16;         // accumulator columns: 4 components x 4 byte planes
constexpr uint32_t kDotStage = 2048;      // bytes of the weights of 32 columns (16 rows x 128)
struct DotSync {
  uint64_t bar[2];
  uint64_t drain;  // completes after every product, when a wait has run out
  uint32_t tmem;
  uint32_t pad;
};
__host__ __device__ constexpr uint32_t dot_stages(uint32_t n_cols) { return (n_cols + 31) / 32; }
__host__ __device__ constexpr size_t dot_smem(uint32_t n_cols) {
  return 4 * (size_t)kUmmaOperand + dot_stages(n_cols) * (size_t)kDotStage + sizeof(DotSync);
}

// The walk of one block over its tiles (blockIdx.x, + gridDim.x, ...):
//   col(c)           column c's words (16-byte aligned),
//   weight(c)        its QM31 weight (canonical),
//   begin()          before a tile's first column,
//   word(r, x)       the operand word (any representative mod P) at row 4t + r
//                    of the column whose word is x; called in column order, and
//                    past the last column (whose weights are zero),
//   rows(tile, s)    the tile's sums of this thread's 4 rows.
// `sm8`: dot_smem(n_cols) bytes, 1024-byte aligned.  Every wait polls at most
// `spin` times; a thread whose wait ran out sets *err (if given), waits no more
// and has no more rows.  Returns the first of the block's tiles whose sums this
// thread did not get: n_tiles or above when it got them all.
template <typename ColFn, typename WeightFn, typename BeginFn, typename WordFn, typename RowsFn>
__device__ __forceinline__ uint32_t row_dot(uint8_t* sm8, uint32_t n_cols, uint32_t n_tiles, uint32_t spin,
                                            uint32_t* err, ColFn col, WeightFn weight, BeginFn begin, WordFn word,
                                            RowsFn rows) {
  uint8_t* opA = sm8;
  uint8_t* opB = sm8 + 4 * kUmmaOperand;
  DotSync* sy = reinterpret_cast<DotSync*>(opB + dot_stages(n_cols) * kDotStage);
  const uint32_t tid = threadIdx.x;
  const uint32_t n_chunks = (n_cols + kDotChunk - 1) / kDotChunk;
  uint4 cur[kDotChunk];
  auto load = [&](uint32_t tile, uint32_t chunk) {
    const uint64_t at = (uint64_t)tile * kDotRows + 4 * tid;
#pragma unroll
    for (int u = 0; u < kDotChunk; u++) {
      const uint32_t c = chunk * kDotChunk + u;
      if (c < n_cols) cur[u] = ldg4(col(c) + at);
    }
  };
  if (tid < 32) tmem_alloc<4 * kDotCols>(&sy->tmem);
  if (tid == 0) {
    mbar_init(&sy->bar[0], 1);
    mbar_init(&sy->bar[1], 1);
    mbar_init(&sy->drain, 1);
    mbar_fence_init();
  }
  load(blockIdx.x, 0);  // gridDim.x <= n_tiles
  for (uint32_t c = tid; c < dot_stages(n_cols) * 32; c += kDotThreads) {
    const qm31 w = c < n_cols ? weight(c) : qm31_zero();
    const uint32_t comp[4] = {w.a, w.b, w.c, w.d};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      uint32_t plane[4];
      umma_weight(comp[k], plane);
#pragma unroll
      for (int j = 0; j < 4; j++)
        *reinterpret_cast<uint32_t*>(opB + (c >> 5) * kDotStage + sw128(4 * k + j, 4 * (c & 31))) = plane[j];
    }
  }
  __syncthreads();
  const uint32_t tmem = sy->tmem;
  bool ok = true;
  uint32_t left = blockIdx.x;  // first tile without its sums
  uint32_t g = 0;  // chunks so far: chunk g uses half g & 1, its products complete phase g >> 1 of bar[g & 1]
  for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    begin();
    for (uint32_t k = 0; k < n_chunks; k++, g++) {
      const uint32_t half = g & 1;
      if (g >= 2) ok = ok && mbar_wait(&sy->bar[half], ((g >> 1) - 1) & 1, spin);
#pragma unroll
      for (int q = 0; q < kDotChunk / 4; q++) {
        uint32_t w[4][4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint4 x = cur[4 * q + u];
#pragma unroll
          for (int r = 0; r < 4; r++) w[r][u] = word(r, u4get(x, r));
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
          *reinterpret_cast<uint4*>(opA + r * kUmmaOperand + sw128(tid, 64 * half + 16 * q)) =
              make_uint4(w[r][0], w[r][1], w[r][2], w[r][3]);
      }
      if (k + 1 < n_chunks)
        load(tile, k + 1);
      else if (tile + gridDim.x < n_tiles)
        load(tile + gridDim.x, 0);
      umma_fence_operand();
      umma_fence_before();
      __syncthreads();
      if (tid == 0) {
        umma_fence_after();
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const uint64_t a = umma_desc(smem_addr(opA) + r * kUmmaOperand) + 4 * half;
          const uint64_t b = umma_desc(smem_addr(opB) + (k >> 1) * kDotStage) + 4 * (k & 1);
          umma_mma(tmem + kDotCols * r, a, b, umma_idesc(kDotCols), k != 0);
          if (n_cols - k * kDotChunk > kDotChunk / 2) umma_mma(tmem + kDotCols * r, a + 2, b + 2, umma_idesc(kDotCols), 1);
        }
        umma_commit(&sy->bar[half]);
      }
    }
    ok = ok && mbar_wait(&sy->bar[(g - 1) & 1], ((g - 1) >> 1) & 1, spin);
    umma_fence_after();
    qm31 s[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      uint32_t d[16];
      tmem_ld16(tmem + kDotCols * r + ((tid & 96) << 16), d);
      tmem_ld_wait(d);
      s[r] = {umma_value(d), umma_value(d + 4), umma_value(d + 8), umma_value(d + 12)};
    }
    if (ok) {
      rows(tile, s);
      left = tile + gridDim.x;
    }
  }
  if (!ok) {
    if (tid == 0) {
      umma_commit(&sy->drain);
      (void)mbar_wait(&sy->drain, 0);
    }
    if (err) *err = 1;
  }
  umma_fence_before();
  __syncthreads();
  if (tid < 32) tmem_free<4 * kDotCols>(tmem);
  return left;
}

// Persistent grid: as many blocks as are resident at once, never more blocks
// than tiles.  The register bound of the kernels holds three blocks on an SM;
// their shared memory (the operands take 64 KB) may hold fewer.
inline unsigned dot_grid(size_t smem, size_t static_smem, uint32_t n_tiles) {
  int dev = 0, sms = 148, sm_smem = 228 << 10;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  const size_t block = smem + static_smem + 1024;  // and what the system keeps of each block's
  const uint32_t per_sm = (uint32_t)std::max<size_t>(1, std::min<size_t>(kDotBlocks, (size_t)sm_smem / block));
  return std::max(1u, std::min(n_tiles, (uint32_t)std::max(1, sms) * per_sm));
}

}  // namespace stwo_b200
