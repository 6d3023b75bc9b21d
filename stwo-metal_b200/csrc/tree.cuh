// Merkle node levels of a tree in one launch (sm_100a).
//
// The upper levels of a tree are bound by latency: a level is one compression
// behind the level below it (about 1710 cycles for one to four warps of an SM,
// one per scheduler; 3290 for eight), however few hashes it has.  What can be
// saved is what stands between the levels: launches (2 to 3 us each with the
// gap before them) and first levels of more than one warp a scheduler.  So
// blocks of 128 threads (one warp a scheduler) take 2^8 hashes to one and the
// block that arrives last takes the blocks' hashes to the root: no block waits
// for another.  Against blocks of 256 threads, 8 levels a launch and a launch
// for the last levels: tree of 2^11 leaves 16 -> 15 us, of 2^18 (with the
// three-levels-a-thread kernel first) 44 -> 38 us with the gaps.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "blake2s.cuh"
#include "field.cuh"

namespace stwo_b200 {

constexpr int kTreeThreads = 128;
constexpr uint32_t kTreeBlockLog = 8;   // a block takes 2^8 hashes to one
constexpr uint32_t kTreeLastLog = 9;    // hashes that the last block can stage
// Input level of the largest tree that one launch takes to its root.
constexpr uint32_t kTreeMaxLog = kTreeBlockLog + kTreeLastLog;
struct TreeLevels {
  uint8_t* out[32];  // level k: 2^k hashes of 32 bytes, 16-byte aligned
};
struct TreeSmem {
  uint4 ping[2 << kTreeLastLog];
  uint4 pong[1 << kTreeLastLog];
  uint32_t last;
};

// Slot of the u-th 16 bytes of a level in shared memory: the 64 bytes of a
// pair stay together, and the same quarter of 8 neighbouring pairs lies in 8
// different bank groups.
__device__ __forceinline__ uint32_t tree_slot(uint32_t u) { return u ^ ((u >> 3) & 3); }

__device__ __forceinline__ void tree_put(uint4* level, uint32_t i, const uint32_t h[8]) {
  level[tree_slot(2 * i)] = make_uint4(h[0], h[1], h[2], h[3]);
  level[tree_slot(2 * i + 1)] = make_uint4(h[4], h[5], h[6], h[7]);
}

// n hashes of global memory, written by other blocks (of this launch or an
// earlier one), into shared memory.
__device__ __forceinline__ void tree_stage(uint4* level, const uint8_t* from, uint32_t n) {
  const uint4* g = reinterpret_cast<const uint4*>(from);
  for (uint32_t u = threadIdx.x; u < 2 * n; u += kTreeThreads) level[tree_slot(u)] = __ldcg(g + u);
}

// The levels below level `lg`, down to `stop`, of which this block has the
// w <= 2^kTreeBlockLog hashes from `base` on (w a power of two) in sm.ping;
// called by all threads, with those words visible to all.  With `arrivals` (one
// zero word, zero again when the launch ends) and stop == 0 the last block goes
// on to the root.  True in the block that has the root, in *root.
// begin() runs in the last block before the rest of its levels.
template <bool LAT, class BeginFn>
__device__ __forceinline__ bool tree_climb(TreeSmem& sm, const TreeLevels& t, uint32_t lg, uint64_t base, uint32_t w,
                                           uint32_t stop, uint32_t* arrivals, bool m31, BeginFn begin,
                                           const uint4** root) {
  uint4* src = sm.ping;
  uint4* dst = sm.pong;
  if (gridDim.x == 1) begin();
#pragma unroll 1
  while (lg > stop) {
    if (w == 1) {  // this block's subtree is done
      if (!arrivals) return false;
      if (threadIdx.x == 0) {  // the thread that wrote its hash
        __threadfence();
        const uint32_t before = atomicAdd(arrivals, 1u);
        sm.last = before == gridDim.x - 1;
        if (sm.last) {
          *arrivals = 0;
          __threadfence();
        }
      }
      __syncthreads();
      if (!sm.last) return false;
      begin();
      src = sm.ping;
      dst = sm.pong;
      tree_stage(src, t.out[lg], 1u << lg);
      __syncthreads();
      base = 0;
      w = 1u << lg;
      arrivals = nullptr;
    }
    w >>= 1;
    base >>= 1;
    lg--;
    for (uint32_t p = threadIdx.x; p < w; p += kTreeThreads) {
      uint32_t m[16], h[8];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint4 x = src[tree_slot(4 * p + q)];
        m[4 * q] = x.x;
        m[4 * q + 1] = x.y;
        m[4 * q + 2] = x.z;
        m[4 * q + 3] = x.w;
      }
      blake2s_init(h);
      if (LAT)
        blake2s_compress_lat(h, m, 64, true);
      else
        blake2s_compress(h, m, 64, true);
      if (m31) {
#pragma unroll
        for (int k = 0; k < 8; k++) h[k] = m31_reduce_u32(h[k]);
      }
      uint4* g = reinterpret_cast<uint4*>(t.out[lg] + (base + p) * 32);
      g[0] = make_uint4(h[0], h[1], h[2], h[3]);
      g[1] = make_uint4(h[4], h[5], h[6], h[7]);
      tree_put(dst, p, h);
    }
    __syncthreads();
    uint4* x = src;
    src = dst;
    dst = x;
  }
  *root = src;
  return lg == 0;
}

// Blocks of a launch whose first level in shared memory has 2^log hashes.
inline unsigned tree_blocks(uint32_t log, uint32_t block_log) { return log > block_log ? 1u << (log - block_log) : 1u; }

// Level at which one launch takes a tree of 2^L leaves over: above it a thread
// hashes three levels at a time (node_subtree3_kernel).
uint32_t node_levels_wide(uint32_t L);

// build_leaves_impl / build_node_layers_impl (merkle.cu).  `arrivals`: one zero
// word of device memory that no launch running beside this one uses (left zero);
// without one the root's own buffer serves, cleared first.
int build_leaves_impl(const uint32_t* const* d_cols, const uint32_t* log_sizes, uint32_t n_cols, uint32_t L, int m31,
                      uint8_t* d_leaves, uint8_t* const* layer_ws, cudaStream_t s, char* err, size_t err_len);
int build_node_layers_impl(const uint8_t* in, uint32_t in_log, uint32_t stop_log, int m31, uint8_t* const* outs_by_log,
                           uint32_t* arrivals, cudaStream_t s, char* err, size_t err_len);
int build_layers_impl(const uint32_t* const* d_cols, const uint32_t* log_sizes, uint32_t n_cols, uint32_t L, int m31,
                      uint8_t* const* d_layers, uint32_t* arrivals, cudaStream_t s, char* err, size_t err_len);

}  // namespace stwo_b200
