// Sort of a query's result when it is small (up to kSmallSortMax rows), the
// count known on the device only: two launches.
//   chunk  a block for 256 items: warps sort runs of 32 by exchanges, then runs
//          merge pairwise in shared memory, each item finding its place in the
//          other run by binary search;
//   rank   a block per SM takes all sorted keys into shared memory and, for its
//          share of the items, finds every chunk's number of smaller items by
//          binary search; their sum is the item's rank, and its value goes there.
//          Lanes search neighbouring chunks, so a chunk takes 257 places: with
//          256 they met in one bank (16 us instead of 10 for 11K items and 512 threads).
// Short chunks, because a block's searches serialise on its SM's shared memory
// (chunks of 2048 items: 20 us for 11K items on six SMs); searches through L1
// (8 to 18 us) are bound by one 128-byte line per cycle.
// Items compare by (64-bit key, 32-bit tie); pairs are unique, so the order is
// total whatever order the items came in.  A count above the limit sets
// *overflow and sorts nothing: the caller sorts another way.  Against one
// thread-block cluster's radix sort (cluster_sort_kernel), whose every 8-bit
// digit is a round of cluster barriers: 13 us against 32 for Q3's 11K rows, 10
// against 43 for Q18's 7K rows (whose two keys are two sorts there).
#pragma once

#include <algorithm>

#include "common.cuh"
#include "context.cuh"

namespace bo {

constexpr int kSsChunk = 256;
constexpr int kSsRow = kSsChunk + 1;      // places of a chunk in shared memory
constexpr int64_t kSmallSortMax = 24576;  // their keys: 193 KB of shared memory
constexpr int kSsChunks = (int)(kSmallSortMax / kSsChunk);
constexpr int kSsRankBlock = 768;  // 512: Q3 71 us instead of 68, Q18 75 instead of 70; 1024 the same
constexpr size_t kSsSmem = (size_t)kSsChunks * kSsRow * sizeof(unsigned long long);

// The sorted chunks: keys apart from {tie, value}, which are read once per item
// (and where two keys are equal).
struct SsItems {
  unsigned long long* key;  // kSmallSortMax
  uint2* rest;              // kSmallSortMax
};
constexpr size_t kSsItemBytes = kSmallSortMax * (sizeof(unsigned long long) + sizeof(uint2));

// An item: {tie, key low, key high, value}.
__device__ __forceinline__ uint4 ss_item(unsigned long long key, uint32_t tie, uint32_t val) {
  return make_uint4(tie, (uint32_t)key, (uint32_t)(key >> 32), val);
}

__device__ __forceinline__ bool ss_less(const uint4& a, const uint4& b) {
  const unsigned long long ka = ((unsigned long long)a.z << 32) | a.y, kb = ((unsigned long long)b.z << 32) | b.y;
  return ka < kb || (ka == kb && a.x < b.x);
}

// Block b makes items [256 b, 256 (b + 1)) with make(i) and stores them sorted.
template <class Make>
__global__ void __launch_bounds__(kSsChunk) ss_chunk_kernel(Make make, const unsigned long long* __restrict__ n_dev,
                                                            SsItems items, uint32_t* __restrict__ overflow) {
  __shared__ uint4 buf[2][kSsChunk];
  pdl_launch_dependents();
  pdl_wait();
  const unsigned long long n = ld_prior(n_dev);
  if (n > (unsigned long long)kSmallSortMax) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *overflow = 1u;
    return;
  }
  const uint32_t t = threadIdx.x, lo = blockIdx.x * kSsChunk, lane = t & 31;
  if (lo >= n) return;
  // Pads are larger than every item, and in their own order.
  uint4 v = lo + t < n ? make(lo + t) : make_uint4(0xffffff00u + t, ~0u, ~0u, 0u);
#pragma unroll
  for (uint32_t k = 2; k <= 32; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      uint4 o;
      o.x = __shfl_xor_sync(0xffffffffu, v.x, j);
      o.y = __shfl_xor_sync(0xffffffffu, v.y, j);
      o.z = __shfl_xor_sync(0xffffffffu, v.z, j);
      o.w = __shfl_xor_sync(0xffffffffu, v.w, j);
      const bool up = (lane & k) == 0, first = (lane & j) == 0;
      if (ss_less(o, v) == (up == first)) v = o;  // the smaller one where `up` wants it
    }
  }
  int src = 0;
  buf[0][t] = v;
  __syncthreads();
#pragma unroll
  for (uint32_t run = 32; run < (uint32_t)kSsChunk; run <<= 1) {
    const uint32_t mine = t & ~(run - 1u);
    const uint4* other = buf[src] + (mine ^ run);
    v = buf[src][t];
    uint32_t at = 0;
#pragma unroll
    for (uint32_t half = run / 2; half > 0; half >>= 1)
      if (ss_less(other[at + half - 1], v)) at += half;
    if (ss_less(other[at], v)) ++at;
    buf[src ^ 1][(mine & ~run) + (t - mine) + at] = v;
    __syncthreads();
    src ^= 1;
  }
  v = buf[src][t];
  items.key[lo + t] = ((unsigned long long)v.z << 32) | v.y;
  items.rest[lo + t] = make_uint2(v.x, v.w);
}

static __global__ void __launch_bounds__(kSsRankBlock) ss_rank_kernel(SsItems items,
                                                                      const unsigned long long* __restrict__ n_dev,
                                                                      uint32_t* __restrict__ out_vals) {
  extern __shared__ unsigned long long ss_keys[];
  __shared__ uint32_t rank[kSsRankBlock];
  pdl_launch_dependents();
  pdl_wait();
  const unsigned long long nd = ld_prior(n_dev);
  if (nd > (unsigned long long)kSmallSortMax) return;
  const uint32_t n = (uint32_t)nd, chunks = (n + kSsChunk - 1) / kSsChunk;
  const uint32_t share = (n + gridDim.x - 1) / gridDim.x;  // <= kSsRankBlock (the host's grid)
  const uint32_t e0 = blockIdx.x * share, mine = e0 >= n ? 0u : (n - e0 < share ? n - e0 : share);
  if (mine == 0) return;
  for (uint32_t i = threadIdx.x; i < chunks * kSsChunk; i += kSsRankBlock)
    ss_keys[i / kSsChunk * kSsRow + i % kSsChunk] = ld_prior(items.key + i);
  rank[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t w = threadIdx.x; w < mine * chunks; w += kSsRankBlock) {
    const uint32_t e = w / chunks, c = w - e * chunks, i = e0 + e;
    uint32_t at = 0;
    if (c == i / kSsChunk) {
      at = i % kSsChunk;
    } else {
      const unsigned long long key = ss_keys[i / kSsChunk * kSsRow + i % kSsChunk];
      const unsigned long long* run = ss_keys + c * kSsRow;
      auto before = [&](uint32_t j) {  // the chunk's item j before item i
        const unsigned long long k = run[j];
        return k < key || (k == key && ld_prior(&items.rest[c * kSsChunk + j].x) < ld_prior(&items.rest[i].x));
      };
#pragma unroll
      for (uint32_t half = kSsChunk / 2; half > 0; half >>= 1)
        if (before(at + half - 1)) at += half;
      if (before(at)) ++at;
    }
    atomicAdd(rank + e, at);
  }
  __syncthreads();
  if (threadIdx.x < mine) out_vals[rank[threadIdx.x]] = ld_prior(&items.rest[e0 + threadIdx.x].y);
}

// Sorts the *n_dev items make(0) .. make(n - 1) and writes their values in
// order to out_vals; `scratch` holds kSsItemBytes.
template <class Make>
int small_sort(bo_ctx* ctx, const Make& make, const unsigned long long* n_dev, void* scratch, uint32_t* out_vals,
               uint32_t* overflow) {
  auto* key = static_cast<unsigned long long*>(scratch);
  const SsItems items{key, reinterpret_cast<uint2*>(key + kSmallSortMax)};
  BO_CUDA(ctx, launch_dependent(&ss_chunk_kernel<Make>, kSsChunks, kSsChunk, 0, ctx->stream, make, n_dev, items,
                                overflow));
  int rc = after_launch(ctx, "ss_chunk_kernel");
  if (rc) return rc;
  static bool ready = false;
  if (!ready)
    BO_CUDA(ctx, cudaFuncSetAttribute(reinterpret_cast<const void*>(&ss_rank_kernel),
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSsSmem));
  ready = true;
  const int grid = std::max(ctx->num_sms, (int)((kSmallSortMax + kSsRankBlock - 1) / kSsRankBlock));
  BO_CUDA(ctx, launch_dependent(&ss_rank_kernel, grid, kSsRankBlock, kSsSmem, ctx->stream, items, n_dev, out_vals));
  return after_launch(ctx, "ss_rank_kernel");
}

// A query's last kernel leaves the result count, the overflow word and the
// error word in the context's pinned words (one thread, after all other
// kernels of the query), so that the host only waits for the stream.
struct HostWords {
  unsigned long long* words;  // pinned, two
  const unsigned long long* n_out;
  const uint32_t* overflow;
  const uint32_t* err;
  __device__ __forceinline__ void store() const {
    volatile unsigned long long* w = words;
    w[0] = *n_out;
    w[1] = (unsigned long long)*overflow | ((unsigned long long)__ldcg(err) << 32);
  }
};

// After a stream whose last kernel stored HostWords: waits, clears the error
// word if it was set, and reports count and overflow.
inline int read_host_words(bo_ctx* ctx, const char* op, int64_t n_max, int64_t* n, bool* overflow) {
  if (int rc = drain_host_work(ctx)) return rc;
  BO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const uint32_t bits = (uint32_t)(ctx->h_word[1] >> 32);
  if (bits) BO_CUDA(ctx, cudaMemsetAsync(ctx->d_err, 0, sizeof(uint32_t), ctx->stream));
  if (int rc = device_error_status(ctx, bits, op)) return rc;
  const unsigned long long nd = ctx->h_word[0], most = (unsigned long long)(n_max > 0 ? n_max : 0);
  *n = (int64_t)(nd < most ? nd : most);
  *overflow = (uint32_t)ctx->h_word[1] != 0u;
  return BO_OK;
}

}  // namespace bo
