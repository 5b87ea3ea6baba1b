// Skewed three-way join + high-cardinality group-by + ordered top-k (K4, with
// the K5 onesweep sort and K6 top-k of radix_sort.cu).
//
// Reference patterns this restates (no reference function computes the whole
// pipeline verbatim):
//   * dimension filters turned into dense masks and fact scans that count per
//     id with bounds checks: bespoke_ceb/query_q1a.cpp (mask builders before
//     :156, cast_info scan :503-601);
//   * group-by with a min aggregate: bespoke_ceb/query_q10a.cpp:843-856;
//   * order by count desc, id asc: bespoke_tpch/query_q10.cpp:318-372.
//
// Pipeline for  A(id)  B(a_id, c_id)  C(category, year; c_id = row index):
//   init     capacity (host exact count, or device-side from a predicted group
//            count), clear the group table, the Bloom filter and the A mask;
//   cfilter  C rows -> exact pass bitmap (one 32-row word per thread, no
//            atomics) and the passing ids into a 64 KB blocked Bloom filter;
//   amask    A ids -> bitmap over [0, a_id_max];
//   scan     B streamed 8 rows per lane (one 256-bit c_id load and one
//            256-bit a_id load, both L2 evict-first and prefetched a step
//            ahead, so no survivor waits on a scattered a_id read); the Bloom
//            filter (read through L1) rejects ~97% of rows without leaving
//            the SM; hits are compacted per warp with their a_id, checked
//            against the exact bitmap and the A mask, and only survivors load
//            the C year (late materialisation).  Survivors aggregate first
//            into a per-block shared-memory table (count, min year) so Zipf
//            heavy hitters cost one global update per block, then the block
//            flushes into a global open-addressing table (key << 32 | count
//            with 64-bit atomicCAS, min year by atomicMin).  The plain form's
//            exact pre-pass runs the same scan setting bits of a distinct
//            bitmap instead;
//   compact  occupied slots -> packed sort keys ((cmax - count) << wa | a_id)
//            with the min year as the value;
//   sort     onesweep LSD radix sort over the key bits actually used, key
//            count read from the device (no host round trip);
//   topk     first k sorted entries decoded into the result record.
#include <algorithm>

#include "common.cuh"
#include "rows.cuh"
#include "context.cuh"

namespace bo {

// The group table and the C-id Bloom filter use the join's slot and filter
// formats (rows.cuh).
constexpr unsigned long long kGbEmpty = kEmptySlot;
constexpr int kGbBloomLog2Words = kBloomLog2Words;
constexpr uint32_t kGbBloomWords = kBloomWords;
constexpr uint32_t kGbBloomBytes = kBloomBytes;
constexpr int kGbBlock = 256;
constexpr int kGbWarps = kGbBlock / 32;
constexpr int kGbRowsPerLane = 8;
constexpr int kGbRowsPerWarpStep = 32 * kGbRowsPerLane;
constexpr int kGbQueue = 384;        // per-warp candidate queue (entries)
constexpr int kGbFlushAt = 128;      // resolve once this many candidates are queued
constexpr int kGbResolveR = 4;       // independent candidates per lane per resolve round
// Per-block pre-aggregation table for Zipf heavy hitters: small (tail keys go
// straight to the global table, where they do not contend) and probed at most
// kGbLocalProbes times, so a full table costs a tail key two shared CAS.
constexpr int kGbLocalSlots = 256;
constexpr int kGbLocalProbes = 2;
constexpr int kGbMinCapLog2 = 10;
constexpr float kGbPresizeFactor = 2.5f;
constexpr int kMaxCats = 64;

struct GbMeta {
  int32_t cap_log2;
  uint32_t overflow;
  uint32_t done;
  uint32_t no_filter;                 // dense form: the Bloom filter was not filled
  unsigned long long joined;          // joined (surviving) B rows
  unsigned long long distinct;        // groups inserted into the global table
  unsigned long long n_out;           // compacted groups (sort key count)
  unsigned long long c_pass;          // qualifying C rows
  unsigned long long exact_distinct;  // plain pre-pass result
  unsigned long long inv_max;         // largest packed (cmax - count): the smallest count's
};

struct CatSet {
  uint16_t v[kMaxCats];
  int32_t n;
};

__device__ __forceinline__ int32_t gb_presize_log2(const float* pred, int32_t host_log2, int32_t max_log2) {
  if (!pred) return host_log2;
  float p = *pred;
  if (!(p >= 0.0f)) p = 0.0f;
  const double want = (double)p * kGbPresizeFactor;
  int32_t cl = kGbMinCapLog2;
  while (cl < max_log2 && (double)(1ull << cl) < want) ++cl;
  return cl;
}

// ------------------------------------------------------------------ init --
// clear_filters = 0 re-initialises only the group table (the plain form's
// second phase keeps the C bitmap, Bloom filter, A mask and filter counters).
__global__ void gb_init_kernel(unsigned long long* slots, int32_t* mins, uint32_t* bloom, uint32_t* amask,
                               uint32_t* dbits, int64_t mask_words, GbMeta* meta, const float* pred, int32_t host_log2,
                               int32_t max_log2, int clear_filters) {
  const int32_t cl = gb_presize_log2(pred, host_log2, max_log2);
  const uint64_t cap = 1ull << cl;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (uint64_t i = tid; i < cap; i += stride) {
    slots[i] = kGbEmpty;
    mins[i] = 0x7fffffff;
  }
  if (clear_filters) {
    for (uint64_t i = tid; i < kGbBloomWords; i += stride) bloom[i] = 0;
    for (uint64_t i = tid; i < (uint64_t)mask_words; i += stride) {
      amask[i] = 0;
      if (dbits) dbits[i] = 0;
    }
  }
  if (tid == 0) {
    meta->cap_log2 = cl;
    meta->overflow = 0;
    meta->done = 0;
    meta->joined = 0;
    meta->distinct = 0;
    meta->n_out = 0;
    meta->inv_max = 0;
    if (clear_filters) {
      meta->c_pass = 0;
      meta->exact_distinct = 0;
    }
  }
}

// --------------------------------------------------------------- cfilter --
// Thread w owns C rows [32w, 32w+32): one full bitmap word, written with a
// plain store.  The category set lives in a shared 65536-bit mask.
__global__ void __launch_bounds__(256) gb_cfilter_kernel(bo_gb_c_cols c, CatSet cats, int32_t year_lo,
                                                         int32_t year_hi, uint32_t* __restrict__ cbits,
                                                         uint32_t* __restrict__ bloom, GbMeta* meta) {
  __shared__ uint32_t catmask[2048];
  for (int i = threadIdx.x; i < 2048; i += blockDim.x) catmask[i] = 0;
  __syncthreads();
  if (threadIdx.x < cats.n) atomicOr(&catmask[cats.v[threadIdx.x] >> 5], 1u << (cats.v[threadIdx.x] & 31u));
  __syncthreads();
  const int64_t n = c.n_rows;
  const int64_t words = (n + 31) / 32;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  uint32_t passed = 0;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += stride) {
    const int64_t r0 = w * 32;
    uint32_t bits = 0;
    if (r0 + 32 <= n) {
      int8v cat[2];
      cat[0] = ld_stream_v8(c.category + r0);
      cat[1] = ld_stream_v8(c.category + r0 + 16);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int8v y = ld_stream_v8(c.year + r0 + 8 * q);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int row = 8 * q + k;
          const uint32_t word = (uint32_t)cat[row >> 4].v[(row & 15) >> 1];
          const uint32_t cv = (row & 1) ? (word >> 16) : (word & 0xffffu);
          const bool ok = ((catmask[cv >> 5] >> (cv & 31u)) & 1u) && y.v[k] >= year_lo && y.v[k] <= year_hi;
          bits |= (uint32_t)ok << row;
        }
      }
    } else {
      for (int k = 0; k < 32 && r0 + k < n; ++k) {
        const uint32_t cv = c.category[r0 + k];
        const int32_t y = c.year[r0 + k];
        const bool ok = ((catmask[cv >> 5] >> (cv & 31u)) & 1u) && y >= year_lo && y <= year_hi;
        bits |= (uint32_t)ok << k;
      }
    }
    cbits[w] = bits;
    passed += __popc(bits);
    uint32_t b = bits;
    while (b) {
      const int k = __ffs(b) - 1;
      b &= b - 1;
      uint32_t bw, bb;
      bloom_pos((uint32_t)(r0 + k), bw, bb);
      atomicOr(bloom + bw, bb);
    }
  }
  __shared__ uint32_t part[8];
  passed = warp_sum_u32(passed);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = passed;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += part[i];
    if (t) atomicAdd(&meta->c_pass, (unsigned long long)t);
  }
}

// ----------------------------------------------------------------- amask --
__global__ void gb_amask_kernel(bo_gb_a_cols a, int32_t a_id_max, uint32_t* __restrict__ amask, uint32_t* err) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  uint32_t bad = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n_rows; i += stride) {
    const int32_t id = a.id[i];
    if (id < 0) continue;  // the reference's id masks skip negative ids
    if (id > a_id_max) {
      bad = 1;
      continue;
    }
    atomicOr(amask + (id >> 5), 1u << (id & 31));
  }
  if (bad) raise_error(err, kErrValueRange);
}

// ------------------------------------------------------------------ scan --

// kMode 0: exact distinct pre-pass (bits of a distinct bitmap); 1: aggregate.
// Records of the radix-partitioned form: the scan appends (key, count, min
// year, partition) records to one array through a warp-aggregated cursor (so
// skewed keys cannot overflow a partition's share), and a counting scatter
// then groups them by partition; the partition of a key is the top bits of
// hash32(key) (shift = 32 - log2 partitions; 32 for one partition).
struct GbParts {
  uint4* records = nullptr;
  uint32_t* cursor = nullptr;
  uint32_t cap = 0;
  uint32_t shift = 32;
  __device__ __forceinline__ uint32_t of(uint32_t key) const { return shift >= 32 ? 0u : hash32(key) >> shift; }
  __device__ __forceinline__ bool put(uint32_t pos, uint32_t key, uint32_t cnt, int32_t mn) const {
    if (pos >= cap) return false;  // more records than the prediction allowed for: the call reruns exactly
    records[pos] = make_uint4(key, cnt, (uint32_t)mn, of(key));
    return true;
  }
};

template <int kMode>
__global__ void __launch_bounds__(kGbBlock) gb_scan_kernel(bo_gb_b_cols b, int64_t n_c, int32_t a_id_max,
                                                           const uint32_t* __restrict__ bloom_g,
                                                           const uint32_t* __restrict__ cbits,
                                                           const int32_t* __restrict__ c_year,
                                                           const uint32_t* __restrict__ amask,
                                                           unsigned long long* slots, int32_t* mins, uint32_t* dbits,
                                                           GbMeta* meta, uint64_t probe_limit, GbParts parts,
                                                           uint32_t* err) {
  __shared__ int32_t q_c[kGbWarps][kGbQueue];
  __shared__ uint32_t q_row[kGbWarps][kGbQueue];
  __shared__ uint32_t l_key[kGbLocalSlots];
  __shared__ uint32_t l_cnt[kGbLocalSlots];
  __shared__ int32_t l_min[kGbLocalSlots];
  __shared__ uint32_t red[3][kGbWarps];
  for (int i = threadIdx.x; i < kGbLocalSlots; i += blockDim.x) {
    l_key[i] = 0xffffffffu;
    l_cnt[i] = 0;
    l_min[i] = 0x7fffffff;
  }
  __syncthreads();
  uint32_t bad = 0;
  // The Bloom filter is read through L1 (64 KB, shared by the SM's CTAs) rather
  // than copied into every CTA's shared memory: registers then allow 3 CTAs
  // per SM instead of 2 (measured ~8% faster per query than the staged copy).
  const uint32_t* bl = bloom_g;
  const uint32_t wmask = kGbBloomWords - 1u;
  const int32_t cl = kMode ? __ldg(&meta->cap_log2) : 0;
  const uint64_t mask = (1ull << cl) - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t* qc = q_c[warp];
  uint32_t* qr = q_row[warp];
  uint32_t qn = 0;  // queued candidates (warp-uniform)
  uint32_t joined = 0, newkeys = 0, full = 0;
  const int64_t n = b.n_rows;
  const int64_t steps = (n + kGbRowsPerWarpStep - 1) / kGbRowsPerWarpStep;
  const int64_t nwarps = (int64_t)gridDim.x * kGbWarps;
  // One step of software prefetch: the next step's c_ids are in flight while
  // the current step is tested and resolved.
  auto load_step = [&](int64_t st, int32_t (&out)[kGbRowsPerLane], int32_t (&out_a)[kGbRowsPerLane], uint32_t& vmask) {
    const int64_t r0 = st * kGbRowsPerWarpStep + lane * kGbRowsPerLane;
    vmask = 0;
    if (st >= steps) return;
    if (r0 + kGbRowsPerLane <= n) {
      const int8v c0 = ld_first_v8(b.c_id + r0);
      const int8v a0 = ld_first_v8(b.a_id + r0);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        out[k] = c0.v[k];
        out_a[k] = a0.v[k];
      }
      vmask = 0xffu;
    } else {
#pragma unroll
      for (int k = 0; k < kGbRowsPerLane; ++k) {
        out[k] = -1;
        out_a[k] = -1;
        if (r0 + k < n) {
          out[k] = b.c_id[r0 + k];
          out_a[k] = b.a_id[r0 + k];
          vmask |= 1u << k;
        }
      }
    }
  };
  // Resolves the warp's queued candidates: lanes take up to kGbResolveR
  // entries each and every round issues its loads for all of them at once
  // (exact C bitmap; then the C year of the passing ones; then the A mask),
  // so a warp has many independent memory chains in flight.  The queue holds
  // each candidate's c_id and a_id.
  auto resolve = [&](uint32_t cnt) {
    __syncwarp();
    for (uint32_t i0 = 0; i0 < cnt; i0 += 32 * kGbResolveR) {
      int32_t c[kGbResolveR];
      uint32_t row[kGbResolveR], w[kGbResolveR];
      int32_t a[kGbResolveR], y[kGbResolveR];
#pragma unroll
      for (int r = 0; r < kGbResolveR; ++r) {
        const uint32_t i = i0 + r * 32 + lane;
        c[r] = i < cnt ? qc[i] : -1;
        row[r] = i < cnt ? qr[i] : 0u;  // the candidate's a_id
        const bool in = (uint32_t)c[r] < (uint32_t)n_c;  // negative or past C: no partner
        w[r] = in ? __ldg(cbits + (c[r] >> 5)) : 0u;
      }
#pragma unroll
      for (int r = 0; r < kGbResolveR; ++r) {
        const bool pass = (w[r] >> (c[r] & 31)) & 1u;
        a[r] = pass ? (int32_t)row[r] : -1;
        y[r] = (pass && kMode >= 1) ? __ldg(c_year + c[r]) : 0;
      }
      // Survivors: A-mask test, then the heavy-hitter table in shared memory;
      // the rest try their first global slot with one CAS each, all issued
      // before any result is used (collisions continue out of line).
      bool pend[kGbResolveR];
#pragma unroll
      for (int r = 0; r < kGbResolveR; ++r) {
        const bool in_a = a[r] >= 0 && a[r] <= a_id_max;
        const uint32_t m = in_a ? __ldg(amask + (a[r] >> 5)) : 0u;
        pend[r] = false;
        if (!in_a || !((m >> (a[r] & 31)) & 1u)) continue;
        ++joined;
        if (kMode == 0) {
          atomicOr(dbits + (a[r] >> 5), 1u << (a[r] & 31));
          continue;
        }
        const uint32_t h = hash32((uint32_t)a[r]);
        bool done = false;
#pragma unroll 1
        for (int p = 0; p < kGbLocalProbes && !done; ++p) {
          const int sl = (int)((h + p) & (kGbLocalSlots - 1));
          const uint32_t old = atomicCAS(&l_key[sl], 0xffffffffu, (uint32_t)a[r]);
          if (old == 0xffffffffu || old == (uint32_t)a[r]) {
            atomicAdd(&l_cnt[sl], 1u);
            atomicMin(&l_min[sl], y[r]);
            done = true;
          }
        }
        pend[r] = !done;
      }
      if (kMode == 2) {
        // Partitioned form: each survivor appends a (key, 1, year) record;
        // the warp reserves its records with one atomic per round.
#pragma unroll
        for (int r = 0; r < kGbResolveR; ++r) {
          const uint32_t pm = __ballot_sync(0xffffffffu, pend[r]);
          if (!pm) continue;  // warp-uniform
          const int leader = __ffs(pm) - 1;
          uint32_t first_pos = 0;
          if (lane == leader) first_pos = atomicAdd(parts.cursor, (uint32_t)__popc(pm));
          first_pos = __shfl_sync(0xffffffffu, first_pos, leader);
          if (pend[r] && !parts.put(first_pos + __popc(pm & ((1u << lane) - 1u)), (uint32_t)a[r], 1u, y[r]))
            full = 1;
        }
      }
      if (kMode == 1) {
        unsigned long long got[kGbResolveR];
        uint64_t first[kGbResolveR];
#pragma unroll
        for (int r = 0; r < kGbResolveR; ++r) {
          first[r] = pend[r] ? (hash32((uint32_t)a[r]) & mask) : 0;
          got[r] = pend[r] ? atomicCAS(slots + first[r], kGbEmpty, (unsigned long long)(uint32_t)a[r] << 32)
                           : 0ull;
        }
#pragma unroll
        for (int r = 0; r < kGbResolveR; ++r) {
          if (!pend[r]) continue;
          if (got[r] == kGbEmpty) ++newkeys;
          if (got[r] == kGbEmpty || (uint32_t)(got[r] >> 32) == (uint32_t)a[r]) {
            atomicAdd(slots + first[r], 1ull);
            atomicMin(mins + first[r], y[r]);
          } else if (!gb_global_insert(slots, mins, mask, (uint32_t)a[r], 1u, y[r], newkeys, (first[r] + 1) & mask,
                                              probe_limit)) {
            full = 1;
          }
        }
      }
    }
    __syncwarp();
  };
  int32_t nxt[kGbRowsPerLane], nxt_a[kGbRowsPerLane];
  uint32_t nxt_valid;
  int64_t st = (int64_t)blockIdx.x * kGbWarps + warp;
  load_step(st, nxt, nxt_a, nxt_valid);
  for (; st < steps; st += nwarps) {
    const int64_t base = st * kGbRowsPerWarpStep;
    int32_t cid[kGbRowsPerLane], aid[kGbRowsPerLane];
#pragma unroll
    for (int k = 0; k < kGbRowsPerLane; ++k) {
      cid[k] = nxt[k];
      aid[k] = nxt_a[k];
    }
    const uint32_t valid = nxt_valid;
    load_step(st + nwarps, nxt, nxt_a, nxt_valid);
    // Branch-free Bloom test of all 8 rows (every lookup is issued; without
    // the filter every word reads as all ones).
    // (The c_id range check happens in the rare resolve path below.)
    uint32_t hit = 0;
#pragma unroll
    for (int k = kGbRowsPerLane - 1; k >= 0; --k) {
      const uint32_t h = (uint32_t)cid[k] * 0x9E3779B1u;
      const uint32_t x = __ldg(bl + ((h >> (32 - kGbBloomLog2Words)) & wmask));
      hit = (hit << 1) | (__funnelshift_r(x, x, h) & __funnelshift_r(x, x, h >> 5) & 1u);
    }
    hit &= valid;
#pragma unroll
    for (int half = 0; half < 1; ++half) {
      const uint32_t hm = (hit >> (8 * half)) & 0xffu;
      uint32_t total;
      uint32_t pos = warp_exclusive_scan(__popc(hm), total);
      if (total == 0) continue;  // warp-uniform
      if (qn + total > kGbQueue) {  // keep room: resolve what is queued first
        resolve(qn);
        qn = 0;
      }
      pos += qn;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if ((hm >> k) & 1u) {
          qc[pos] = cid[8 * half + k];
          qr[pos] = (uint32_t)aid[8 * half + k];
          ++pos;
        }
      }
      qn += total;
      __syncwarp();
      if (qn >= kGbFlushAt) {
        resolve(qn);
        qn = 0;
      }
    }
  }
  if (qn) resolve(qn);
  __syncthreads();
  if (kMode == 1) {
    // Flush the block's pre-aggregated groups into the global table.
    for (int i = threadIdx.x; i < kGbLocalSlots; i += blockDim.x) {
      if (l_key[i] != 0xffffffffu)
        if (!gb_global_insert(slots, mins, mask, l_key[i], l_cnt[i], l_min[i], newkeys, ~0ull, probe_limit))
          full = 1;
    }
  } else if (kMode == 2) {
    // ... or as records, one per pre-aggregated group.
    for (int i = threadIdx.x; i < kGbLocalSlots; i += blockDim.x) {
      if (l_key[i] != 0xffffffffu)
        if (!parts.put(atomicAdd(parts.cursor, 1u), l_key[i], l_cnt[i], l_min[i])) full = 1;
    }
  }
  if (bad) raise_error(err, bad);
  const uint32_t wj = warp_sum_u32(joined), wn = warp_sum_u32(newkeys);
  const unsigned wf = __any_sync(0xffffffffu, full != 0);
  if (lane == 0) {
    red[0][warp] = wj;
    red[1][warp] = wn;
    red[2][warp] = wf;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tj = 0, tn = 0, tf = 0;
    for (int w = 0; w < kGbWarps; ++w) {
      tj += red[0][w];
      tn += red[1][w];
      tf |= red[2][w];
    }
    if (tj) atomicAdd(&meta->joined, (unsigned long long)tj);
    if (tn) {
      const unsigned long long before = atomicAdd(&meta->distinct, (unsigned long long)tn);
      if (kMode == 1 && before + tn > (mask + 1) - ((mask + 1) >> 3)) atomicOr(&meta->overflow, 1u);
    }
    if (tf) atomicOr(&meta->overflow, 1u);
  }
}

__global__ void gb_popcount_kernel(const uint32_t* __restrict__ dbits, int64_t words, GbMeta* meta) {
  uint32_t c = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) c += __popc(dbits[i]);
  c = warp_sum_u32(c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(&meta->exact_distinct, (unsigned long long)c);
}

// --------------------------------------------------------------- compact --
// Each block compacts a contiguous range of slots: warps count their occupied
// slots, one atomic per block reserves the block's output range (per-warp
// atomics on the single counter would serialise in L2).
constexpr int kCompactBlock = 256;
constexpr int kCompactPerThread = 8;

__global__ void __launch_bounds__(kCompactBlock) gb_compact_kernel(const unsigned long long* __restrict__ slots,
                                                                   const int32_t* __restrict__ mins, GbMeta* meta,
                                                                   int wa, unsigned long long cmax,
                                                                   unsigned long long* __restrict__ keys,
                                                                   uint32_t* __restrict__ vals) {
  __shared__ uint32_t warp_off[kCompactBlock / 32 + 1];
  __shared__ unsigned long long block_base;
  const int32_t cl = __ldg(&meta->cap_log2);
  const uint64_t cap = 1ull << cl;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t span = (uint64_t)kCompactBlock * kCompactPerThread;
  for (uint64_t b0 = (uint64_t)blockIdx.x * span; b0 < cap; b0 += (uint64_t)gridDim.x * span) {
    uint32_t occ = 0;
    unsigned long long v[kCompactPerThread];
#pragma unroll
    for (int j = 0; j < kCompactPerThread; ++j) {
      const uint64_t i = b0 + (uint64_t)j * kCompactBlock + threadIdx.x;
      v[j] = i < cap ? slots[i] : kGbEmpty;
      occ += v[j] != kGbEmpty;
    }
    uint32_t wtot;
    const uint32_t mine = warp_exclusive_scan(occ, wtot);
    if (lane == 0) warp_off[warp] = wtot;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t t = 0;
      for (int w = 0; w < kCompactBlock / 32; ++w) {
        const uint32_t c = warp_off[w];
        warp_off[w] = t;
        t += c;
      }
      block_base = t ? atomicAdd(&meta->n_out, (unsigned long long)t) : 0ull;
    }
    __syncthreads();
    unsigned long long pos = block_base + warp_off[warp] + mine;
    unsigned long long cmaxc = 0;  // largest count seen by this thread
#pragma unroll
    for (int j = 0; j < kCompactPerThread; ++j) {
      if (v[j] != kGbEmpty) {
        const uint64_t i = b0 + (uint64_t)j * kCompactBlock + threadIdx.x;
        const unsigned long long cnt = v[j] & 0xffffffffull;
        cmaxc = cnt > cmaxc ? cnt : cmaxc;
        keys[pos] = ((cmax - cnt) << wa) | (v[j] >> 32);
        vals[pos] = (uint32_t)mins[i];
        ++pos;
      }
    }
    // The select digit of the top-k must sit below the highest bit that
    // differs among the packed counts: track the largest count.
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, cmaxc, o);
      cmaxc = other > cmaxc ? other : cmaxc;
    }
    if (lane == 0 && cmaxc) atomicMax(&meta->inv_max, cmaxc);
    __syncthreads();
  }
}

// ------------------------------------------------- partitioned aggregate --
// Counting scatter of the records by partition (histogram, exclusive scan,
// scatter), then one block per partition (grid-stride over partitions): the
// partition's records aggregate in a shared-memory table (key, count, min
// year) and its groups are written as packed sort keys like
// gb_compact_kernel's.  A partition with more groups than the table holds
// sets the overflow flag (the caller reruns exactly).
constexpr int kPartBlock = 512;
constexpr int kPartSlots = 8192;  // slots of a partition's shared table
constexpr uint32_t kPartMaxGroups = kPartSlots / 8 * 7;  // fuller counts as overflow
constexpr int kPartProbes = 256;  // probe-chain bound: a longer chain counts as overflow
constexpr size_t kPartSmem = (size_t)kPartSlots * 12;
constexpr int kPartScanBlock = 1024;

__global__ void __launch_bounds__(kPartBlock) gb_part_hist_kernel(GbParts parts, uint32_t n_parts,
                                                                  uint32_t* __restrict__ counts) {
  extern __shared__ uint32_t hist[];
  for (uint32_t i = threadIdx.x; i < n_parts; i += kPartBlock) hist[i] = 0;
  __syncthreads();
  const uint32_t n = min(__ldcg(parts.cursor), parts.cap);
  for (uint32_t i = blockIdx.x * kPartBlock + threadIdx.x; i < n; i += gridDim.x * kPartBlock)
    atomicAdd(hist + parts.records[i].w, 1u);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n_parts; i += kPartBlock)
    if (hist[i]) atomicAdd(counts + i, hist[i]);
}

// offsets[p] = records before partition p (offsets[n_parts] = all); fill = offsets.
__global__ void __launch_bounds__(kPartScanBlock) gb_part_scan_kernel(const uint32_t* __restrict__ counts,
                                                                      uint32_t n_parts, uint32_t* __restrict__ offsets,
                                                                      uint32_t* __restrict__ fill) {
  __shared__ uint32_t warp_tot[kPartScanBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t per = (n_parts + kPartScanBlock - 1) / kPartScanBlock;
  const uint32_t lo = threadIdx.x * per, hi = min(lo + per, n_parts);
  uint32_t local = 0;
  for (uint32_t i = lo; i < hi; ++i) local += counts[i];
  uint32_t wt;
  const uint32_t wex = warp_exclusive_scan(local, wt);
  if (lane == 0) warp_tot[warp] = wt;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kPartScanBlock / 32; ++w) {
      const uint32_t x = warp_tot[w];
      warp_tot[w] = t;
      t += x;
    }
    offsets[n_parts] = t;
  }
  __syncthreads();
  uint32_t run = warp_tot[warp] + wex;
  for (uint32_t i = lo; i < hi; ++i) {
    offsets[i] = run;
    fill[i] = run;
    run += counts[i];
  }
}

// Records -> their partition's range; the lanes of one partition reserve
// their slots with one atomic (match_any groups them).
__global__ void __launch_bounds__(kPartBlock) gb_part_scatter_kernel(GbParts parts, uint32_t* __restrict__ fill,
                                                                     uint4* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const uint32_t n = min(__ldcg(parts.cursor), parts.cap);
  const uint32_t warps = gridDim.x * (kPartBlock / 32);
  for (uint32_t i0 = (blockIdx.x * kPartBlock + threadIdx.x) & ~31u; i0 < n; i0 += warps * 32) {
    const uint32_t i = i0 + lane;
    const bool valid = i < n;
    const uint4 r = valid ? parts.records[i] : make_uint4(0, 0, 0, 0xffffffffu);
    const uint32_t peers = __match_any_sync(0xffffffffu, r.w);
    const int leader = __ffs(peers) - 1;
    uint32_t first_pos = 0;
    if (valid && lane == leader) first_pos = atomicAdd(fill + r.w, (uint32_t)__popc(peers));
    first_pos = __shfl_sync(0xffffffffu, first_pos, leader);
    if (valid) out[first_pos + __popc(peers & ((1u << lane) - 1u))] = r;
  }
}

__global__ void __launch_bounds__(kPartBlock) gb_part_agg_kernel(const uint4* __restrict__ recs,
                                                                 const uint32_t* __restrict__ offsets, int n_parts,
                                                                 GbMeta* meta, int wa, unsigned long long cmax,
                                                                 unsigned long long* __restrict__ keys,
                                                                 uint32_t* __restrict__ vals) {
  extern __shared__ __align__(16) uint32_t part_smem[];
  uint32_t* t_key = part_smem;
  uint32_t* t_cnt = part_smem + kPartSlots;
  int32_t* t_min = reinterpret_cast<int32_t*>(part_smem + 2 * kPartSlots);
  __shared__ uint32_t warp_off[kPartBlock / 32];
  __shared__ unsigned long long base;
  __shared__ uint32_t full_s, used_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPer = kPartSlots / kPartBlock;
  unsigned long long cmaxc = 0;
  for (int p = blockIdx.x; p < n_parts; p += gridDim.x) {
    for (int i = threadIdx.x; i < kPartSlots; i += kPartBlock) {
      t_key[i] = 0xffffffffu;
      t_cnt[i] = 0;
      t_min[i] = 0x7fffffff;
    }
    if (threadIdx.x == 0) full_s = used_s = 0;
    __syncthreads();
    const uint32_t b0 = offsets[p], b1 = offsets[p + 1];
    for (uint32_t i = b0 + threadIdx.x; i < b1; i += kPartBlock) {
      if (*reinterpret_cast<volatile uint32_t*>(&full_s)) break;  // the call reruns: stop early
      const uint4 r = recs[i];
      uint32_t sl = hash32(r.x) & (kPartSlots - 1);
      bool done = false;
      for (int step = 0; step < kPartProbes && !done; ++step) {
        const uint32_t old = atomicCAS(t_key + sl, 0xffffffffu, r.x);
        if (old == 0xffffffffu || old == r.x) {
          if (old == 0xffffffffu && atomicAdd(&used_s, 1u) + 1u > kPartMaxGroups) full_s = 1;
          atomicAdd(t_cnt + sl, r.y);
          atomicMin(t_min + sl, (int32_t)r.z);
          done = true;
        }
        sl = (sl + 1) & (kPartSlots - 1);
      }
      if (!done) full_s = 1;
    }
    __syncthreads();
    // Emit the partition's groups: one reservation per block.
    uint32_t occ = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) occ += t_key[j * kPartBlock + threadIdx.x] != 0xffffffffu;
    uint32_t wtot;
    const uint32_t mine = warp_exclusive_scan(occ, wtot);
    if (lane == 0) warp_off[warp] = wtot;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t t = 0;
      for (int w = 0; w < kPartBlock / 32; ++w) {
        const uint32_t x = warp_off[w];
        warp_off[w] = t;
        t += x;
      }
      base = t ? atomicAdd(&meta->n_out, (unsigned long long)t) : 0ull;
      if (t) atomicAdd(&meta->distinct, (unsigned long long)t);
      if (full_s) atomicOr(&meta->overflow, 1u);
    }
    __syncthreads();
    unsigned long long pos = base + warp_off[warp] + mine;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = j * kPartBlock + threadIdx.x;
      if (t_key[i] != 0xffffffffu) {
        const unsigned long long cnt = t_cnt[i];
        cmaxc = cnt > cmaxc ? cnt : cmaxc;
        keys[pos] = ((cmax - cnt) << wa) | t_key[i];
        vals[pos] = (uint32_t)t_min[i];
        ++pos;
      }
    }
    __syncthreads();
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, cmaxc, o);
    cmaxc = other > cmaxc ? other : cmaxc;
  }
  if (lane == 0 && cmaxc) atomicMax(&meta->inv_max, cmaxc);
}

// ============================================================ dense form ==
// Aggregation by a_id itself instead of a hash table: one entry per id in [0,
// a_id_max], where those fit the memory of the group table (gb_dense_fits).  A
// survivor then costs L2 atomics without a returned value (the hash table: a
// CAS round trip, then an add and a min), A's mask is applied to ids instead of
// rows, and the top k comes out of one pass over the entries.
//   cfilter  C rows -> one code byte per row (0: fails; else 1 + year -
//            year_lo), and the 128 KB Bloom filter of the passing ids;
//   scan     few C rows pass (gd_scan_kernel, one block per SM): the filter sits
//            in shared memory (a random word costs about 3.4 bank cycles a warp
//            there, 32 tag lookups a warp through L1), its hits queue per warp,
//            and only rows whose code byte confirms them load their a_id.  Many
//            pass (gd_scan_all_kernel): no filter, every row reads its code byte
//            and streams its a_id; counts alone take a bit per row from
//            gd_planes_kernel.  The device decides, the other one returns;
//   collect  entries of A's ids: groups, joined rows, the k best of each block,
//            and in the last block the k best of all and the result record;
//   years    (counts alone) B once more for the smallest years of the k groups.
// Entries are {count, smallest year} pairs while those stay well inside L2, and
// counts alone beyond (kGdPairIds) and in the partitioned form, whose calls have
// many groups: half the memory, half the atomics, no code bytes.
// Measured (B200, device time): A 2.5M, B 36M, C 4M, 1% of C: 92 us (cfilter 12,
// scan 54, collect 21) against 137 us of the hash form; A 25M, B 60M, C 4M, half
// of C: 560 against 3300 us partitioned by hash (scan 1810, scatter 800, ...).
constexpr int kGdBlock = 1024;
constexpr int kGdWarps = kGdBlock / 32;
constexpr int kGdLog2Words = 15;  // Bloom filter: 2^15 words = 128 KB
constexpr uint32_t kGdWords = 1u << kGdLog2Words;
constexpr uint32_t kGdFilterBytes = kGdWords * 4;
constexpr int kGdFlushAt = 64;
constexpr int kGdQueue = 320;     // per-warp candidate queue: up to kGdFlushAt left over + one step of 256 rows
constexpr int kGdResolveR = 2;
constexpr int kGdLocalSlots = 512;
constexpr size_t kGdSmem = kGdFilterBytes + (size_t)kGdWarps * kGdQueue * 8;
// The filter is used while at most a quarter of its bits can be set.
constexpr unsigned long long kGdFilterKeys = (unsigned long long)kGdWords * 32 / 8;
// B rows below which copying the filter to every SM costs more than it saves.
constexpr int64_t kGdFilterRows = 1 << 20;
// Smallest years are kept as the largest (kGdYearTop - code), 0 where there is
// none, so that entries start as zero bytes.
constexpr uint32_t kGdYearTop = 255;
// Counts are added to in passes over ids that each have at most this many bytes
// of them, half of L2 (25M ids, 100 MB: the query in one pass 798 us, in two 575,
// in three 660; 12.5M ids, 50 MB: one 286, two 328).
constexpr int64_t kGdPassBytes = 64 << 20;
constexpr int64_t kGdPairIds = 8 << 20;  // 64 MB of pairs: half of L2

__device__ __forceinline__ void gd_bloom_pos(uint32_t key, uint32_t& word, uint32_t& bits) {
  const uint32_t h = key * 0x9E3779B1u;
  word = h >> (32 - kGdLog2Words);
  bits = (1u << (h & 31u)) | (1u << ((h >> 5) & 31u));
}

// Thread w owns C rows [32w, 32w + 32): 32 code bytes.
__global__ void __launch_bounds__(256) gd_cfilter_kernel(bo_gb_c_cols c, CatSet cats, int32_t year_lo, int32_t year_hi,
                                                         uint8_t* __restrict__ code, uint32_t* __restrict__ cbits,
                                                         uint32_t* __restrict__ bloom, uint4* __restrict__ entries,
                                                         int64_t entry_vecs, GbMeta* meta, const float* pred,
                                                         int32_t host_log2, int32_t max_log2) {
  __shared__ uint32_t catmask[2048];
  pdl_launch_dependents();
  for (int i = threadIdx.x; i < 2048; i += blockDim.x) catmask[i] = 0;
  __syncthreads();
  if (threadIdx.x < cats.n) atomicOr(&catmask[cats.v[threadIdx.x] >> 5], 1u << (cats.v[threadIdx.x] & 31u));
  __syncthreads();
  const int64_t n = c.n_rows;
  const int64_t words = (n + 31) / 32;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid == 0) meta->cap_log2 = gb_presize_log2(pred, host_log2, max_log2);
  // A table that would fill the filter many times over is not put into it: 256
  // rows spread over the table, the same for every block, tell (4M rows of
  // which half pass: 52 -> 24 us).
  if (bloom && n > 4 * (int64_t)kGdFilterKeys) {
    const int64_t r = (int64_t)(((uint64_t)hash32(threadIdx.x) * (uint64_t)n) >> 32);
    const uint32_t cv = c.category[r];
    const int32_t y = c.year[r];
    const int got = __syncthreads_count(((catmask[cv >> 5] >> (cv & 31u)) & 1u) && y >= year_lo && y <= year_hi);
    if ((int64_t)got * n > 256 * 4 * (int64_t)kGdFilterKeys) {
      bloom = nullptr;
      if (tid == 0) meta->no_filter = 1;
    }
  }
  for (int64_t i = tid; i < entry_vecs; i += stride) entries[i] = make_uint4(0, 0, 0, 0);
  uint32_t passed = 0;
  for (int64_t w = tid; w < words; w += stride) {
    const int64_t r0 = w * 32;
    uint32_t bits = 0;
    if (r0 + 32 <= n) {
      int8v cat[2];
      cat[0] = ld_stream_v8(c.category + r0);
      cat[1] = ld_stream_v8(c.category + r0 + 16);
      uint32_t cw[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int8v y = ld_stream_v8(c.year + r0 + 8 * q);
        cw[2 * q] = cw[2 * q + 1] = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int row = 8 * q + k;
          const uint32_t word = (uint32_t)cat[row >> 4].v[(row & 15) >> 1];
          const uint32_t cv = (row & 1) ? (word >> 16) : (word & 0xffffu);
          const bool ok = ((catmask[cv >> 5] >> (cv & 31u)) & 1u) && y.v[k] >= year_lo && y.v[k] <= year_hi;
          bits |= (uint32_t)ok << row;
          cw[row >> 2] |= ok ? (uint32_t)(y.v[k] - year_lo + 1) << (8 * (row & 3)) : 0u;
        }
      }
      uint4* dst = reinterpret_cast<uint4*>(code + r0);
      dst[0] = make_uint4(cw[0], cw[1], cw[2], cw[3]);
      dst[1] = make_uint4(cw[4], cw[5], cw[6], cw[7]);
    } else {
      for (int k = 0; k < 32 && r0 + k < n; ++k) {
        const uint32_t cv = c.category[r0 + k];
        const int32_t y = c.year[r0 + k];
        const bool ok = ((catmask[cv >> 5] >> (cv & 31u)) & 1u) && y >= year_lo && y <= year_hi;
        bits |= (uint32_t)ok << k;
        code[r0 + k] = ok ? (uint8_t)(y - year_lo + 1) : 0;
      }
    }
    cbits[w] = bits;
    passed += __popc(bits);
    if (!bloom) continue;
    while (bits) {
      const int k = __ffs(bits) - 1;
      bits &= bits - 1;
      uint32_t bw, bb;
      gd_bloom_pos((uint32_t)(r0 + k), bw, bb);
      if ((__ldcg(bloom + bw) & bb) != bb) atomicOr(bloom + bw, bb);  // a filling filter costs reads, not atomics
    }
  }
  __shared__ uint32_t part[8];
  passed = warp_sum_u32(passed);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = passed;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += part[i];
    if (t) atomicAdd(&meta->c_pass, (unsigned long long)t);
  }
}

// Whether the filtered scan runs.
__device__ __forceinline__ bool gd_filtered(const GbMeta* meta, bool has_filter) {
  return has_filter && !ld_prior(&meta->no_filter) && ld_prior(&meta->c_pass) <= kGdFilterKeys;
}

// A block's pre-aggregation of heavy hitters, as gb_scan_kernel's, which a warp
// leaves once it has seen that fewer than a quarter of its keys are there.
struct GdLocal {
  uint32_t key[kGdLocalSlots], cnt[kGdLocalSlots], year[kGdLocalSlots];
  __device__ __forceinline__ void clear() {
    for (int i = threadIdx.x; i < kGdLocalSlots; i += blockDim.x) {
      key[i] = 0xffffffffu;
      cnt[i] = 0;
      year[i] = 0;
    }
  }
};

struct GdTries {
  uint32_t tries = 0, hits = 0;
};

// True if the local table took the key.
template <bool kYear>
__device__ __forceinline__ bool gd_add_local(GdLocal& l, GdTries& t, uint32_t a, uint32_t year) {
  const uint32_t h = hash32(a);
  ++t.tries;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int sl = (int)((h + p) & (kGdLocalSlots - 1));
    const uint32_t old = atomicCAS(&l.key[sl], 0xffffffffu, a);
    if (old == 0xffffffffu || old == a) {
      t.hits += old == a;
      atomicAdd(&l.cnt[sl], 1u);
      if (kYear) atomicMax(&l.year[sl], year);
      return true;
    }
  }
  return false;
}

// Whether the warp keeps to the local table (asked by all lanes together).
__device__ __forceinline__ bool gd_keep_local(const GdTries& t) {
  const uint32_t tries = __reduce_add_sync(0xffffffffu, t.tries), hits = __reduce_add_sync(0xffffffffu, t.hits);
  return tries < 512u || hits * 4u >= tries;
}

// Eight consecutive ids of this lane in a warp's step of 256 rows; -1 past the
// end (no partner).
__device__ __forceinline__ void gd_load8(const int32_t* col, int64_t n, int64_t st, int32_t (&out)[8]) {
  const int64_t r0 = st * 256 + (threadIdx.x & 31) * 8;
  if (r0 + 8 <= n) {
    const int8v v = ld_first_v8(col + r0);
#pragma unroll
    for (int k = 0; k < 8; ++k) out[k] = v.v[k];
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) out[k] = r0 + k < n ? col[r0 + k] : -1;
  }
}

// One survivor into its entry: a pair's count and year, or a count alone.
template <bool kYear>
__device__ __forceinline__ void gd_add(uint32_t* entries, uint32_t a, uint32_t cnt, uint32_t year) {
  if (kYear) {
    atomicAdd(entries + 2 * (size_t)a, cnt);
    atomicMax(entries + 2 * (size_t)a + 1, year);
  } else {
    atomicAdd(entries + a, cnt);
  }
}

template <bool kYear>
__device__ __forceinline__ void gd_flush_local(const GdLocal& l, uint32_t* entries) {
  __syncthreads();
  for (int i = threadIdx.x; i < kGdLocalSlots; i += blockDim.x)
    if (l.key[i] != 0xffffffffu) gd_add<kYear>(entries, l.key[i], l.cnt[i], l.year[i]);
}

template <bool kYear>
__global__ void __launch_bounds__(kGdBlock, 1) gd_scan_kernel(bo_gb_b_cols b, int64_t n_c, int32_t a_id_max,
                                                              const uint8_t* __restrict__ code,
                                                              const uint32_t* __restrict__ bloom,
                                                              const GbMeta* __restrict__ meta,
                                                              uint32_t* __restrict__ entries, uint32_t* err) {
  pdl_launch_dependents();
  pdl_wait();
  if (!gd_filtered(meta, true)) return;
  extern __shared__ __align__(128) uint32_t gd_smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ GdLocal local;
  local.clear();
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_arrive_expect_tx(&bar, kGdFilterBytes);
    bulk_copy_g2s(gd_smem, bloom, kGdFilterBytes / 2, &bar);
    bulk_copy_g2s(gd_smem + kGdWords / 2, bloom + kGdWords / 2, kGdFilterBytes / 2, &bar);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = b.n_rows;
  const int64_t steps = (n + 255) / 256;
  const int64_t nwarps = (int64_t)gridDim.x * kGdWarps;
  const uint32_t nc = (uint32_t)n_c;  // n_c < 2^31; ids outside [0, n_c) have no partner
  int64_t st = (int64_t)blockIdx.x * kGdWarps + warp;
  int32_t n1[8], n2[8];  // the next two steps' ids, in flight
  if (st < steps) gd_load8(b.c_id, n, st, n1);
  if (st + nwarps < steps) gd_load8(b.c_id, n, st + nwarps, n2);
  __syncthreads();
  // Without the filter (a timed-out copy, never expected) every word is taken as all ones: same answer.
  const uint32_t pass = mbar_wait_bounded(&bar, 0, kWaitLimitNs) ? 0u : 0xffffffffu;
  if (pass) raise_error(err, kErrSpinTimeout);
  uint32_t* qc = gd_smem + kGdWords + warp * kGdQueue * 2;
  uint32_t* qr = qc + kGdQueue;
  uint32_t qn = 0;  // queued candidates (warp-uniform)
  GdTries tries;
  bool use_local = true;
  auto resolve = [&]() {
    __syncwarp();
    for (uint32_t i0 = 0; i0 < qn; i0 += 32 * kGdResolveR) {
      uint32_t c[kGdResolveR], row[kGdResolveR], y[kGdResolveR];
      int32_t a[kGdResolveR];
#pragma unroll
      for (int r = 0; r < kGdResolveR; ++r) {
        const uint32_t i = i0 + r * 32 + lane;
        c[r] = i < qn ? qc[i] : 0xffffffffu;
        row[r] = i < qn ? qr[i] : 0u;
        y[r] = c[r] < nc ? ld_prior(code + c[r]) : 0u;
      }
#pragma unroll
      for (int r = 0; r < kGdResolveR; ++r) a[r] = y[r] ? __ldg(b.a_id + row[r]) : -1;
#pragma unroll
      for (int r = 0; r < kGdResolveR; ++r) {
        if (a[r] < 0 || a[r] > a_id_max) continue;
        const uint32_t yr = kGdYearTop - y[r];
        if (use_local && gd_add_local<kYear>(local, tries, (uint32_t)a[r], yr)) continue;
        gd_add<kYear>(entries, (uint32_t)a[r], 1u, yr);
      }
    }
    qn = 0;
    if (use_local) use_local = gd_keep_local(tries);
    __syncwarp();
  };
  // One step's ids: tests, then its few hits into the queue, one per lane and
  // round (a lane rarely has two), and the ids of two steps on requested into
  // the same registers.
  auto step = [&](int32_t (&cid)[8]) {
    uint32_t hit = 0;
#pragma unroll
    for (int k = 7; k >= 0; --k) {
      const uint32_t h = (uint32_t)cid[k] * 0x9E3779B1u;
      const uint32_t x = gd_smem[h >> (32 - kGdLog2Words)] | pass;
      hit = (hit << 1) | (__funnelshift_r(x, x, h) & __funnelshift_r(x, x, h >> 5) & 1u);
    }
    const uint32_t r0 = (uint32_t)(st * 256) + lane * 8;
    for (uint32_t who = __ballot_sync(0xffffffffu, hit != 0); who; who = __ballot_sync(0xffffffffu, hit != 0)) {
      if (hit) {
        const int k = __ffs(hit) - 1;
        hit &= hit - 1;
        const int32_t c01 = k & 1 ? cid[1] : cid[0], c23 = k & 1 ? cid[3] : cid[2];
        const int32_t c45 = k & 1 ? cid[5] : cid[4], c67 = k & 1 ? cid[7] : cid[6];
        const int32_t c03 = k & 2 ? c23 : c01, c47 = k & 2 ? c67 : c45;
        const uint32_t pos = qn + __popc(who & ((1u << lane) - 1u));
        qc[pos] = (uint32_t)(k & 4 ? c47 : c03);
        qr[pos] = r0 + k;
      }
      qn += __popc(who);
    }
    if (st + 2 * nwarps < steps) gd_load8(b.c_id, n, st + 2 * nwarps, cid);
    if (qn >= kGdFlushAt) resolve();
    st += nwarps;
  };
  while (st < steps) {
    step(n1);
    if (st < steps) step(n2);
  }
  if (qn) resolve();
  gd_flush_local<kYear>(local, entries);
  if (pass) mbar_wait_bounded(&bar, 0, kWaitLimitNs);  // the copy may still be in flight
}

// Counts alone: the exact bit of every row's c_id, looked up in shared memory.  A
// block holds one of `ranges` parts of C's bitmap and tests all rows of its group
// of that many blocks, which read them at about the same time, so that DRAM
// delivers them once; its answers are one plane of a bit per row (a byte per lane
// and step).  60M rows, 4M C rows in three parts: 92 us for the planes, bound by
// the three lookups a row in shared memory, and 2 x 118 us for the passes of
// gd_scan_all_kernel over them; with lookups through L1 those took 633 us, of
// which the atomics were 65.  20M rows, 1.3M C rows: 356 -> 212 us the query, 10M:
// 221 -> 165.
constexpr int kGpBlock = 1024;
constexpr int64_t kGpRangeBits = 1600 * 1024;  // 200 KB of shared memory
constexpr int kGpMaxRanges = 4;

__global__ void __launch_bounds__(kGpBlock, 1)
    gd_planes_kernel(bo_gb_b_cols b, int64_t n_c, const uint32_t* __restrict__ cbits, uint32_t ranges, uint32_t range,
                     const GbMeta* __restrict__ meta, bool has_filter, uint8_t* __restrict__ planes,
                     int64_t plane_bytes) {
  extern __shared__ __align__(128) uint32_t gp_bits[];  // `range` bits, a multiple of 128, and a zero word
  pdl_launch_dependents();
  const uint32_t part = blockIdx.x % ranges, lo = part * range;
  const int64_t steps = (b.n_rows + 255) / 256;
  const int64_t nwarps = (int64_t)(gridDim.x / ranges) * (kGpBlock / 32);
  int64_t st = (int64_t)(blockIdx.x / ranges) * (kGpBlock / 32) + (threadIdx.x >> 5);
  int32_t n1[8], n2[8];
  if (st < steps) gd_load8(b.c_id, b.n_rows, st, n1);
  if (st + nwarps < steps) gd_load8(b.c_id, b.n_rows, st + nwarps, n2);
  pdl_wait();
  if (gd_filtered(meta, has_filter)) return;
  const int64_t words = (n_c + 31) / 32 - lo / 32;  // of the bitmap from lo on; none past its end
  for (int i = threadIdx.x; i < (int)(range / 128); i += kGpBlock) {
    uint4 v = make_uint4(0, 0, 0, 0);
    const uint32_t* src = cbits + lo / 32 + 4 * i;
    if (4 * i + 4 <= words) {
      v = ld_prior_v4(src);
    } else {
      if (4 * i < words) v.x = ld_prior(src);
      if (4 * i + 1 < words) v.y = ld_prior(src + 1);
      if (4 * i + 2 < words) v.z = ld_prior(src + 2);
    }
    reinterpret_cast<uint4*>(gp_bits)[i] = v;
  }
  if (threadIdx.x == 0) gp_bits[range / 32] = 0;
  __syncthreads();
  uint8_t* plane = planes + part * plane_bytes + (threadIdx.x & 31);
  auto step = [&](int32_t (&cid)[8]) {
    uint32_t hit = 0;
#pragma unroll
    for (int k = 7; k >= 0; --k) {
      const uint32_t off = min((uint32_t)cid[k] - lo, range);
      const uint32_t x = gp_bits[off >> 5];
      hit = (hit << 1) | (__funnelshift_r(x, x, off) & 1u);
    }
    plane[st * 32] = (uint8_t)hit;
    if (st + 2 * nwarps < steps) gd_load8(b.c_id, b.n_rows, st + 2 * nwarps, cid);
    st += nwarps;
  };
  while (st < steps) {
    step(n1);
    if (st < steps) step(n2);
  }
}

// Every row: its code byte (random, from L2), its a_id (streamed), its atomics.
// Counts alone need no year, so a bit of the exact bitmap does, an eighth of the
// bytes, or (kPlanes) the answers of gd_planes_kernel; then L2 bounds it (63 %
// busy with a quarter of the rows' atomics a pass; requesting a step ahead in
// more registers and fewer warps: 563 -> 598 us the query).
constexpr int kGaBlock = 256;

template <bool kYear, bool kPlanes>
__global__ void __launch_bounds__(kGaBlock, 8)
    gd_scan_all_kernel(bo_gb_b_cols b, int64_t n_c, int32_t id_lo, int32_t id_hi, const uint8_t* __restrict__ code,
                       const uint32_t* __restrict__ cbits, const uint8_t* __restrict__ planes, uint32_t ranges,
                       int64_t plane_bytes, const GbMeta* __restrict__ meta, bool has_filter,
                       uint32_t* __restrict__ entries) {
  pdl_launch_dependents();
  pdl_wait();
  if (gd_filtered(meta, has_filter)) return;
  __shared__ GdLocal local;
  local.clear();
  __syncthreads();
  const int64_t n = b.n_rows;
  const int64_t steps = (n + 255) / 256;
  const int64_t nwarps = (int64_t)gridDim.x * (kGaBlock / 32);
  const uint32_t nc = (uint32_t)n_c;
  GdTries tries;
  bool use_local = true;
  for (int64_t st = (int64_t)blockIdx.x * (kGaBlock / 32) + (threadIdx.x >> 5); st < steps; st += nwarps) {
    int32_t cid[8], aid[8];
    uint32_t hit = 0;
    gd_load8(b.a_id, n, st, aid);
    if constexpr (kPlanes) {
      uint32_t plane[kGpMaxRanges];  // requested together
#pragma unroll
      for (uint32_t r = 0; r < (uint32_t)kGpMaxRanges; ++r)
        plane[r] = r < ranges ? ld_prior(planes + r * plane_bytes + st * 32 + (threadIdx.x & 31)) : 0u;
#pragma unroll
      for (int r = 0; r < kGpMaxRanges; ++r) hit |= plane[r];
    } else {
      gd_load8(b.c_id, n, st, cid);
    }
    if (kPlanes && !use_local) {  // few instructions a row: the pass streams
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (((hit >> k) & 1u) && (uint32_t)(aid[k] - id_lo) <= (uint32_t)(id_hi - id_lo)) atomicAdd(entries + aid[k], 1u);
      continue;
    }
    uint32_t y[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in_a = aid[k] >= id_lo && aid[k] <= id_hi;
      if constexpr (kPlanes) {
        y[k] = in_a ? (hit >> k) & 1u : 0u;
        continue;
      }
      const bool in = in_a && (uint32_t)cid[k] < nc;
      if (kYear) y[k] = in ? ld_prior(code + cid[k]) : 0u;
      else y[k] = in ? (ld_prior(cbits + (cid[k] >> 5)) >> (cid[k] & 31)) & 1u : 0u;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (!y[k]) continue;
      if (use_local && gd_add_local<kYear>(local, tries, (uint32_t)aid[k], kGdYearTop - y[k])) continue;
      gd_add<kYear>(entries, (uint32_t)aid[k], 1u, kGdYearTop - y[k]);
    }
    if (use_local) use_local = gd_keep_local(tries);
  }
  gd_flush_local<kYear>(local, entries);
}

constexpr int kGcBlock = 256;
constexpr int kGcPer = 8;                  // consecutive ids per thread and step
constexpr int kGcTile = kGcBlock * kGcPer;
constexpr int kGcKeep = kGcTile;           // candidates kept between steps before they are cut to k
constexpr int kGcBuf = kGcKeep + kGcTile;

// Upper bound of the k-th smallest of the block's keys, k <= 64: the k-th
// smallest of the minima of 64 groups of four threads (k keys do not exceed
// it; ~0 if fewer groups have a key).  All threads of the block call it.
__device__ __forceinline__ unsigned long long gc_bound(unsigned long long mine, int k) {
  __shared__ unsigned long long gmin[64], bound;
  for (int o = 1; o < 4; o <<= 1) {
    const unsigned long long x = __shfl_xor_sync(0xffffffffu, mine, o);
    mine = x < mine ? x : mine;
  }
  if ((threadIdx.x & 3) == 0) gmin[threadIdx.x >> 2] = mine;
  if (threadIdx.x == 0) bound = ~0ull;
  __syncthreads();
  if (threadIdx.x < 64) {
    const unsigned long long v = gmin[threadIdx.x];
    int r = 0;
#pragma unroll 16
    for (int i = 0; i < 64; ++i) r += gmin[i] < v;
    if (r == k - 1) bound = v;  // unique unless ~0
  }
  __syncthreads();
  return bound;
}

// The k smallest of the m <= kGcBuf unique keys in buf, ascending, to its front.
// All threads of the block call it.  Few keys: each thread ranks one; more: cut
// down by the bound of gc_bound first (m keys leave at most k * ceil(m / 64)).
__device__ __forceinline__ uint32_t gc_cut(unsigned long long* buf, uint32_t m, int k) {
  __shared__ uint32_t left;
  while (m > (uint32_t)kGcBlock) {
    unsigned long long own[kGcBuf / kGcBlock], mine = ~0ull;
#pragma unroll
    for (int i = 0; i < kGcBuf / kGcBlock; ++i) {
      const uint32_t at = i * kGcBlock + threadIdx.x;
      own[i] = at < m ? buf[at] : ~0ull;
      mine = own[i] < mine ? own[i] : mine;
    }
    if (threadIdx.x == 0) left = 0;
    const unsigned long long bound = gc_bound(mine, k);  // also: all keys are in registers
#pragma unroll
    for (int i = 0; i < kGcBuf / kGcBlock; ++i)
      if (own[i] <= bound && own[i] != ~0ull) buf[atomicAdd(&left, 1u)] = own[i];
    __syncthreads();
    if (left == m) break;  // cannot shrink further (k near 64 of few hundred keys): ranked below
    m = left;
    __syncthreads();
  }
  unsigned long long v[kGcBuf / kGcBlock];
  uint32_t r[kGcBuf / kGcBlock];
  const int per = (int)((m + kGcBlock - 1) / kGcBlock);
  for (int i = 0; i < per; ++i) {
    const uint32_t at = i * kGcBlock + threadIdx.x;
    v[i] = at < m ? buf[at] : ~0ull;
    r[i] = 0;
    for (uint32_t j = 0; j < m; ++j) r[i] += buf[j] < v[i];
  }
  __syncthreads();
  for (int i = 0; i < per; ++i)
    if (v[i] != ~0ull && r[i] < (uint32_t)k) buf[r[i]] = v[i];
  __syncthreads();
  return m < (uint32_t)k ? m : (uint32_t)k;
}

// kParts: also counts groups per hash partition (the partitioned form's rule
// for too few partitions).  kPairs: entries are {count, year}.
template <bool kParts, bool kPairs>
__global__ void __launch_bounds__(kGcBlock, 3) gd_collect_kernel(const uint32_t* __restrict__ entries, int64_t n_ids,
                                                              const uint32_t* __restrict__ amask, GbMeta* meta,
                                                              int32_t year_lo, int k, int wa, unsigned long long cmax,
                                                              uint32_t* __restrict__ part_counts, uint32_t n_parts,
                                                              unsigned long long* __restrict__ cand,
                                                              bo_gb_result* __restrict__ out) {
  extern __shared__ uint32_t hist[];  // kParts: n_parts counters
  __shared__ unsigned long long buf[kGcBuf];
  __shared__ uint32_t count_s, over_s;
  __shared__ unsigned long long red[2][kGcBlock / 32];
  pdl_launch_dependents();
  if (threadIdx.x == 0) count_s = over_s = 0;
  if (kParts)
    for (uint32_t i = threadIdx.x; i < n_parts; i += kGcBlock) hist[i] = 0;
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long limit = k > 0 ? ~0ull : 0ull;  // only keys below it can be among the k best
  uint32_t groups = 0;
  unsigned long long joined = 0;
  // This thread's eight counts of tile t, zero where the id is not one of A's.
  auto load = [&](int64_t t, uint32_t (&c)[kGcPer]) {
    const int64_t id0 = t * kGcTile + threadIdx.x * kGcPer;
    if (id0 + kGcPer <= n_ids) {
      if (kPairs) {
        const int8v v0 = ld_prior_v8(entries + 2 * id0), v1 = ld_prior_v8(entries + 2 * id0 + 8);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          c[j] = (uint32_t)v0.v[2 * j];
          c[4 + j] = (uint32_t)v1.v[2 * j];
        }
      } else {
        const int8v v = ld_prior_v8(entries + id0);
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = (uint32_t)v.v[j];
      }
      const uint32_t am = __ldg(amask + (id0 >> 5)) >> (id0 & 31) & 0xffu;  // id0 is a multiple of eight
      if (am != 0xffu) {
#pragma unroll
        for (int j = 0; j < kGcPer; ++j)
          if (!((am >> j) & 1u)) c[j] = 0;
      }
    } else {
#pragma unroll
      for (int j = 0; j < kGcPer; ++j) {
        const int64_t id = id0 + j;
        c[j] = 0;
        if (id < n_ids && ((__ldg(amask + (id >> 5)) >> (id & 31)) & 1u)) c[j] = ld_prior(entries + (kPairs ? 2 * id : id));
      }
    }
  };
  // Appends this thread's keys below the limit to the candidates; the first
  // call of a phase takes the limit from the keys themselves.  (some: false
  // where the caller knows that no key of this thread is below it.)
  auto keep = [&](const unsigned long long (&key)[kGcPer], bool first, bool some) {
    if (first && k > 0) {
      unsigned long long mine = ~0ull;
#pragma unroll
      for (int j = 0; j < kGcPer; ++j) mine = key[j] < mine ? key[j] : mine;
      const unsigned long long b = gc_bound(mine, k);
      if (b != ~0ull) limit = b + 1;
    }
    uint32_t take = 0;
    if (some) {
#pragma unroll
      for (int j = 0; j < kGcPer; ++j) take |= (uint32_t)(key[j] < limit) << j;
    }
    if (!__syncthreads_or(take != 0)) return;  // uniform
    if (__any_sync(0xffffffffu, take != 0)) {
      uint32_t total, pos = 0;
      const uint32_t before = warp_exclusive_scan(__popc(take), total);
      if (lane == 0) pos = atomicAdd(&count_s, total);
      pos = __shfl_sync(0xffffffffu, pos, 0) + before;
#pragma unroll
      for (int j = 0; j < kGcPer; ++j)
        if ((take >> j) & 1u) buf[pos++] = key[j];
    }
    __syncthreads();
    const uint32_t m = count_s;
    if (m > (uint32_t)kGcKeep) {  // uniform
      const uint32_t left = gc_cut(buf, m, k);
      if (threadIdx.x == 0) count_s = left;
      limit = buf[k - 1];
    }
    __syncthreads();
  };
  const int64_t tiles = (n_ids + kGcTile - 1) / kGcTile;
  // Contiguous runs of tiles: a block meets ids in ascending order.
  const int64_t per = (tiles + gridDim.x - 1) / gridDim.x;
  const int64_t t0 = blockIdx.x * per, t1 = t0 + per < tiles ? t0 + per : tiles;
  uint32_t n1[kGcPer], n2[kGcPer];  // the next two tiles, in flight
  if (t0 < t1) load(t0, n1);
  if (t0 + 1 < t1) load(t0 + 1, n2);
  __syncthreads();
  auto step = [&](int64_t t, uint32_t (&c)[kGcPer]) {
    const uint32_t id0 = (uint32_t)(t * kGcTile) + threadIdx.x * kGcPer;
    // Counts below the limit's cannot be among the best: most threads stop here.
    const unsigned long long need = limit == ~0ull ? 1ull : cmax - (limit >> wa);
    uint32_t most = 0, sum = 0;
#pragma unroll
    for (int j = 0; j < kGcPer; ++j) {
      groups += min(c[j], 1u);
      sum += c[j];  // at most B's rows
      most = max(most, c[j]);
      if (kParts && c[j]) atomicAdd(hist + __umulhi(hash32(id0 + j), n_parts), 1u);  // n_parts: a power of two
    }
    joined += sum;
    const bool some = most >= need && most > 0;
    unsigned long long key[kGcPer];
    if (some) {
#pragma unroll
      for (int j = 0; j < kGcPer; ++j) key[j] = c[j] ? ((cmax - c[j]) << wa) | (id0 + j) : ~0ull;
    } else {
#pragma unroll
      for (int j = 0; j < kGcPer; ++j) key[j] = ~0ull;
    }
    if (t + 2 < t1) load(t + 2, c);
    keep(key, t == t0, some);
  };
  for (int64_t t = t0; t < t1; t += 2) {
    step(t, n1);
    if (t + 1 < t1) step(t + 1, n2);
  }
  uint32_t mine = k > 0 ? gc_cut(buf, count_s, k) : 0;
  if (threadIdx.x < (uint32_t)k)
    cand[(size_t)blockIdx.x * k + threadIdx.x] = threadIdx.x < mine ? buf[threadIdx.x] : ~0ull;
  if (kParts)
    for (uint32_t i = threadIdx.x; i < n_parts; i += kGcBlock)
      if (hist[i]) atomicAdd(part_counts + i, hist[i]);
  groups = warp_sum_u32(groups);
  joined = (unsigned long long)warp_sum_i64((int64_t)joined);
  if (lane == 0) {
    red[0][warp] = groups;
    red[1][warp] = joined;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long g = 0, jr = 0;
    for (int w = 0; w < kGcBlock / 32; ++w) {
      g += red[0][w];
      jr += red[1][w];
    }
    if (g) atomicAdd(&meta->n_out, g);
    if (jr) atomicAdd(&meta->joined, jr);
  }
  if (!last_block(&meta->done)) return;
  if (kParts)
    for (uint32_t i = threadIdx.x; i < n_parts; i += kGcBlock)
      if (__ldcg(part_counts + i) > kPartMaxGroups) over_s = 1;
  if (gridDim.x > 1 && k > 0) {
    if (threadIdx.x == 0) count_s = 0;
    limit = ~0ull;
    __syncthreads();
    const uint32_t all = gridDim.x * (uint32_t)k;
    for (uint32_t i0 = 0; i0 < all; i0 += kGcTile) {
      unsigned long long key[kGcPer];
#pragma unroll
      for (int j = 0; j < kGcPer; ++j) {
        const uint32_t i = i0 + j * kGcBlock + threadIdx.x;
        key[j] = i < all ? __ldcg(cand + i) : ~0ull;
      }
      keep(key, i0 == 0, true);
    }
    mine = gc_cut(buf, count_s, k);
  }
  __syncthreads();
  const unsigned long long n = __ldcg(&meta->n_out);
  if (threadIdx.x < mine) {
    const unsigned long long key = buf[threadIdx.x];
    const uint32_t id = (uint32_t)(key & ((1ull << wa) - 1ull));
    bo_gb_row r;
    r.a_id = (int32_t)id;
    r.min_year = kPairs ? year_lo + (int32_t)(kGdYearTop - ld_prior(entries + 2 * (size_t)id + 1)) - 1 : 0x7fffffff;
    r.count = (int64_t)(cmax - (key >> wa));
    out->rows[threadIdx.x] = r;
  }
  if (threadIdx.x == 0) {
    const int32_t cl = __ldcg(&meta->cap_log2);
    const unsigned long long cap = 1ull << cl;
    out->n_groups = (int64_t)n;
    out->joined_rows = (int64_t)__ldcg(&meta->joined);
    out->c_qualifying = (int64_t)__ldcg(&meta->c_pass);
    out->capacity_log2 = cl;
    // The table a prediction sized (or a partition's) would have been too full.
    out->overflowed = kParts ? (int32_t)over_s : (int32_t)(n > cap - (cap >> 3));
    out->reruns = 0;
    out->mode = kParts ? 2 : 1;
    out->n_rows_out = (int32_t)mine;
    out->exact_distinct = 0;
  }
}

// Counts alone: the smallest years of the result's groups.  Bound by streaming
// B's a_ids; a row of one of the at most 64 groups is rare.
__global__ void __launch_bounds__(256) gd_years_kernel(bo_gb_b_cols b, int64_t n_c, int32_t year_lo,
                                                       const uint8_t* __restrict__ code,
                                                       bo_gb_result* __restrict__ out) {
  pdl_wait();
  constexpr int kBits = 1 << 16;  // one hashed bit per group: at most one other row in a thousand gets past it
  __shared__ uint32_t bits[kBits / 32];
  __shared__ int32_t key[BO_GB_MAX_K];
  const int rows = out->n_rows_out;
  for (int i = threadIdx.x; i < kBits / 32; i += 256) bits[i] = 0;
  __syncthreads();
  if (threadIdx.x < rows) {
    const int32_t a = out->rows[threadIdx.x].a_id;
    key[threadIdx.x] = a;
    const uint32_t h = ((uint32_t)a * 0x9E3779B1u) >> 16;
    atomicOr(bits + (h >> 5), 1u << (h & 31u));
  }
  __syncthreads();
  const int64_t n = b.n_rows;
  const int64_t steps = (n + 255) / 256;
  for (int64_t st = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); st < steps; st += (int64_t)gridDim.x * 8) {
    int32_t a[8];
    gd_load8(b.a_id, n, st, a);
    uint32_t hit = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t h = ((uint32_t)a[j] * 0x9E3779B1u) >> 16;
      hit |= ((bits[h >> 5] >> (h & 31u)) & 1u) << j;
    }
    if (!hit) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (!((hit >> j) & 1u)) continue;
      const int64_t r = st * 256 + (threadIdx.x & 31) * 8 + j;
      if (r >= n) continue;
      for (int i = 0; i < rows; ++i) {
        if (key[i] != a[j]) continue;
        const int32_t c = b.c_id[r];
        const uint32_t y = (uint32_t)c < (uint32_t)n_c ? ld_prior(code + c) : 0u;
        if (y) atomicMin(&out->rows[i].min_year, year_lo + (int32_t)y - 1);
      }
    }
  }
}

// ------------------------------------------------------------------ topk --
__global__ void gb_topk_kernel(const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals,
                               GbMeta* meta, int k, int wa, unsigned long long cmax, int mode,
                               bo_gb_result* __restrict__ out) {
  const unsigned long long n = __ldcg(&meta->n_out);
  const int t = threadIdx.x;
  if (t < k && (unsigned long long)t < n) {
    const unsigned long long key = keys[t];
    bo_gb_row r;
    r.a_id = (int32_t)(key & ((1ull << wa) - 1ull));
    r.min_year = (int32_t)vals[t];
    r.count = (int64_t)(cmax - (key >> wa));
    out->rows[t] = r;
  }
  if (t == 0) {
    out->n_groups = (int64_t)n;
    out->joined_rows = (int64_t)__ldcg(&meta->joined);
    out->c_qualifying = (int64_t)__ldcg(&meta->c_pass);
    out->capacity_log2 = __ldcg(&meta->cap_log2);
    out->overflowed = (int32_t)__ldcg(&meta->overflow);
    out->reruns = 0;
    out->mode = mode;
    out->n_rows_out = (int32_t)(n < (unsigned long long)k ? n : (unsigned long long)k);
    out->exact_distinct = (int64_t)__ldcg(&meta->exact_distinct);
  }
}

// ------------------------------------------------------------------ host --
namespace {

int bit_length(uint64_t v) {
  int b = 0;
  while (v) {
    ++b;
    v >>= 1;
  }
  return b;
}

struct GbWs {
  unsigned long long* slots;
  int32_t* mins;
  uint32_t* bloom;
  uint32_t* cbits;
  uint32_t* amask;
  uint32_t* dbits;
  GbMeta* meta;
  float* pred;
  unsigned long long* keys;
  uint32_t* vals;
  unsigned long long* tkeys;
  uint32_t* tvals;
  int32_t max_log2;
  int64_t mask_words;
};

int gb_workspace(bo_ctx* ctx, const bo_gb_b_cols& b, const bo_gb_c_cols& c, int32_t a_id_max, GbWs* ws) {
  const uint64_t groups_max = std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)a_id_max + 1, (uint64_t)b.n_rows));
  const int32_t max_log2 = std::max(kGbMinCapLog2, bit_length(groups_max * 2 - 1));
  const uint64_t cap = 1ull << max_log2;
  const int64_t mask_words = ((int64_t)a_id_max + 1 + 31) / 32;
  const int64_t cwords = (c.n_rows + 31) / 32;
  size_t total = 0;
  auto add = [&](size_t bytes) { total += (bytes + 255) & ~size_t(255); };
  add(8 * cap);                       // slots
  add(4 * cap);                       // mins
  add(kGbBloomBytes);                 // bloom
  add(4 * (size_t)std::max<int64_t>(cwords, 1));
  add(4 * (size_t)mask_words);        // amask
  add(4 * (size_t)mask_words);        // dbits
  add(sizeof(GbMeta) + 64);
  add(8 * cap);                       // keys
  add(4 * cap);                       // vals
  add(8 * cap);                       // tmp keys
  add(4 * cap);                       // tmp vals
  void* base = nullptr;
  int rc = region(ctx, "gb_ws", total, &base);
  if (rc) return rc;
  char* p = static_cast<char*>(base);
  ws->slots = carve<unsigned long long>(p, cap);
  ws->mins = carve<int32_t>(p, cap);
  ws->bloom = carve<uint32_t>(p, kGbBloomWords);
  ws->cbits = carve<uint32_t>(p, (size_t)std::max<int64_t>(cwords, 1));
  ws->amask = carve<uint32_t>(p, (size_t)mask_words);
  ws->dbits = carve<uint32_t>(p, (size_t)mask_words);
  char* meta_p = p;
  p += (sizeof(GbMeta) + 64 + 255) & ~size_t(255);
  ws->meta = reinterpret_cast<GbMeta*>(meta_p);
  ws->pred = reinterpret_cast<float*>(meta_p + sizeof(GbMeta));
  ws->keys = carve<unsigned long long>(p, cap);
  ws->vals = carve<uint32_t>(p, cap);
  ws->tkeys = carve<unsigned long long>(p, cap);
  ws->tvals = carve<uint32_t>(p, cap);
  ws->max_log2 = max_log2;
  ws->mask_words = mask_words;
  return BO_OK;
}

int check_gb(bo_ctx* ctx, const bo_gb_a_cols* a, const bo_gb_b_cols* b, const bo_gb_c_cols* c,
             const bo_gb_params* prm) {
  if (!a || !b || !c || !prm) return set_error(ctx, BO_ERR_INVALID, "groupby: null argument");
  if (a->n_rows < 0 || b->n_rows < 0 || c->n_rows < 0) return set_error(ctx, BO_ERR_INVALID, "groupby: negative rows");
  if (c->n_rows > 0x7fffffffll || b->n_rows > 0xffffffffll)
    return set_error(ctx, BO_ERR_INVALID, "groupby: C above 2^31 rows or B above 2^32 rows");
  if (prm->a_id_max < 0) return set_error(ctx, BO_ERR_INVALID, "groupby: a_id_max must be >= 0");
  if (prm->k < 0 || prm->k > BO_GB_MAX_K) return set_error(ctx, BO_ERR_INVALID, "groupby: k outside [0, %d]", BO_GB_MAX_K);
  if (prm->n_categories < 0 || prm->n_categories > kMaxCats || (prm->n_categories > 0 && !prm->categories))
    return set_error(ctx, BO_ERR_INVALID, "groupby: at most %d categories", kMaxCats);
  if (b->n_rows > 0 && (!b->a_id || !b->c_id || !aligned32(b->a_id) || !aligned32(b->c_id)))
    return set_error(ctx, BO_ERR_INVALID, "groupby: B columns null or not 32-byte aligned");
  if (c->n_rows > 0 && (!c->category || !c->year || !aligned32(c->category) || !aligned32(c->year)))
    return set_error(ctx, BO_ERR_INVALID, "groupby: C columns null or not 32-byte aligned");
  if (a->n_rows > 0 && !a->id) return set_error(ctx, BO_ERR_INVALID, "groupby: A column null");
  return BO_OK;
}

int grid_res(bo_ctx* ctx, const void* k, int block, size_t smem, int64_t items) {
  const int64_t resident = (int64_t)ctx->num_sms * occupancy_blocks(k, block, smem);
  const int64_t need = (items + block - 1) / block;
  return (int)std::max<int64_t>(1, std::min(resident, need));
}

// Filters (init, C filter, A mask): common to both forms.
int gb_prepare(bo_ctx* ctx, const bo_gb_a_cols& a, const bo_gb_c_cols& c, const bo_gb_params& prm, const GbWs& ws,
               const float* pred, int32_t host_log2) {
  const void* ki = reinterpret_cast<const void*>(&gb_init_kernel);
  const int gi = grid_res(ctx, ki, 256, 0, std::max<int64_t>((int64_t)1 << std::min(ws.max_log2, 24), ws.mask_words));
  gb_init_kernel<<<gi, 256, 0, ctx->stream>>>(ws.slots, ws.mins, ws.bloom, ws.amask, ws.dbits, ws.mask_words, ws.meta,
                                              pred, host_log2, ws.max_log2, 1);
  int rc = after_launch(ctx, "gb_init_kernel");
  if (rc) return rc;
  CatSet cs{};
  cs.n = prm.n_categories;
  for (int i = 0; i < prm.n_categories; ++i) cs.v[i] = prm.categories[i];
  const int64_t cwords = (c.n_rows + 31) / 32;
  if (cwords > 0) {
    const void* kc = reinterpret_cast<const void*>(&gb_cfilter_kernel);
    const int gc = grid_res(ctx, kc, 256, 0, cwords);
    gb_cfilter_kernel<<<gc, 256, 0, ctx->stream>>>(c, cs, prm.year_lo, prm.year_hi, ws.cbits, ws.bloom, ws.meta);
    if ((rc = after_launch(ctx, "gb_cfilter_kernel"))) return rc;
  }
  if (a.n_rows > 0 && !prm.a_mask) {
    const void* ka = reinterpret_cast<const void*>(&gb_amask_kernel);
    const int ga = grid_res(ctx, ka, 256, 0, a.n_rows);
    gb_amask_kernel<<<ga, 256, 0, ctx->stream>>>(a, prm.a_id_max, ws.amask, ctx->d_err);
    if ((rc = after_launch(ctx, "gb_amask_kernel"))) return rc;
  }
  return BO_OK;
}

template <int kMode>
int gb_launch_scan(bo_ctx* ctx, const bo_gb_b_cols& b, const bo_gb_c_cols& c, const bo_gb_params& prm,
                   const GbWs& ws, uint64_t probe_limit = ~0ull, GbParts parts = GbParts{}) {
  const void* k = reinterpret_cast<const void*>(&gb_scan_kernel<kMode>);
  const int grid = grid_res(ctx, k, kGbBlock, 0, (b.n_rows + kGbRowsPerLane - 1) / kGbRowsPerLane);
  gb_scan_kernel<kMode><<<grid, kGbBlock, 0, ctx->stream>>>(
      b, c.n_rows, prm.a_id_max, ws.bloom, ws.cbits, c.year, prm.a_mask ? prm.a_mask : ws.amask, ws.slots, ws.mins,
      ws.dbits, ws.meta, probe_limit, parts, ctx->d_err);
  return after_launch(ctx, "gb_scan_kernel");
}

// Aggregate + compact + sort + top-k, asynchronous.
int gb_aggregate_order(bo_ctx* ctx, const bo_gb_b_cols& b, const bo_gb_c_cols& c, const bo_gb_params& prm,
                       const GbWs& ws, bo_gb_result* out, int32_t mode) {
  // Exact-size tables (mode 0) probe without a bound; presized ones fail fast.
  int rc = gb_launch_scan<1>(ctx, b, c, prm, ws, mode == 0 ? ~0ull : kPresizedProbeLimit);
  if (rc) return rc;
  const int wa = std::max(1, bit_length((uint64_t)prm.a_id_max));
  const int wc = std::max(1, bit_length((uint64_t)b.n_rows));
  const unsigned long long cmax = (wc >= 64) ? ~0ull : ((1ull << wc) - 1ull);
  const uint64_t cap_max = 1ull << ws.max_log2;
  const void* kc = reinterpret_cast<const void*>(&gb_compact_kernel);
  const int gc = grid_res(ctx, kc, kCompactBlock, 0, (int64_t)cap_max / kCompactPerThread);
  gb_compact_kernel<<<gc, kCompactBlock, 0, ctx->stream>>>(ws.slots, ws.mins, ws.meta, wa, cmax, ws.keys, ws.vals);
  if ((rc = after_launch(ctx, "gb_compact_kernel"))) return rc;
  // ORDER BY count desc, a_id asc LIMIT k: radix select of the k smallest
  // packed keys, then the onesweep / in-CTA LSD sort of the candidates.
  // The candidates go to the temporary buffers; the sort uses the key
  // buffers (no longer needed) as its scratch.
  // (cmax - count) for counts in [1, max_count] shares every bit above the
  // highest bit of max_count with cmax: the select digit goes just below it
  // (inv_max holds the largest count; topk_shift takes its bit length).
  if ((rc = radix_topk_pairs(ctx, ws.keys, ws.vals, (int64_t)cap_max, &ws.meta->n_out, wa + wc, prm.k, ws.tkeys,
                             ws.tvals, ws.keys, ws.vals, wa, &ws.meta->inv_max)))
    return rc;
  gb_topk_kernel<<<1, BO_GB_MAX_K, 0, ctx->stream>>>(ws.tkeys, ws.tvals, ws.meta, prm.k, wa, cmax, mode, out);
  return after_launch(ctx, "gb_topk_kernel");
}

// The dense form takes a call whose entries (8 B per id) fit the group table's
// slots and whose years fit a byte.  The presized form also wants at most one
// id per two B rows: the entries are cleared and read once whatever joins,
// which beyond that costs more than the small hash table of a selective query.
bool gb_dense_fits(const bo_gb_b_cols& b, const bo_gb_params& prm, const GbWs& ws, bool partitioned) {
  const int64_t ids = (int64_t)prm.a_id_max + 1;
  if ((int64_t)prm.year_hi - prm.year_lo > 253 || ids > ((int64_t)1 << ws.max_log2)) return false;
  return partitioned || ids <= std::max<int64_t>(b.n_rows / 2, 1 << 16);
}

// The dense form, asynchronous; n_parts == 0: presized from pred, else the
// partitioned form with n_parts partitions.  *took is false when its
// scratch cannot be had (the hash form then runs).
int gb_dense(bo_ctx* ctx, const bo_gb_a_cols& a, const bo_gb_b_cols& b, const bo_gb_c_cols& c, const bo_gb_params& prm,
             const GbWs& ws, const float* pred, uint32_t n_parts, uint32_t shift, bo_gb_result* out, bool* took) {
  const bool parts = n_parts > 0;
  const int64_t ids = (int64_t)prm.a_id_max + 1;
  auto al = [](size_t v) { return (v + 255) & ~size_t(255); };
  const int64_t tiles = (ids + kGcTile - 1) / kGcTile;
  const int gk = (int)std::min<int64_t>(tiles, (int64_t)ctx->num_sms * 3);  // all resident; few candidates to merge
  const size_t meta_bytes = al(sizeof(GbMeta)), cnt_bytes = al(4 * (size_t)n_parts);
  const size_t cand_bytes = al(8 * (size_t)BO_GB_MAX_K * gk), code_bytes = al((size_t)c.n_rows + 32);
  void* base = nullptr;
  *took = false;
  if (region(ctx, "gb_dense", meta_bytes + kGdFilterBytes + cnt_bytes + cand_bytes + code_bytes, &base) != BO_OK) {
    cudaGetLastError();
    return BO_OK;
  }
  *took = true;
  char* p = static_cast<char*>(base);
  GbMeta* meta = reinterpret_cast<GbMeta*>(p);
  uint32_t* bloom = reinterpret_cast<uint32_t*>(p + meta_bytes);
  uint32_t* part_counts = reinterpret_cast<uint32_t*>(p + meta_bytes + kGdFilterBytes);
  auto* cand = reinterpret_cast<unsigned long long*>(p + meta_bytes + kGdFilterBytes + cnt_bytes);
  uint8_t* code = reinterpret_cast<uint8_t*>(p + meta_bytes + kGdFilterBytes + cnt_bytes + cand_bytes);
  BO_CUDA(ctx, cudaMemsetAsync(p, 0, meta_bytes + kGdFilterBytes + cnt_bytes, ctx->stream));
  const uint32_t* amask = prm.a_mask ? prm.a_mask : ws.amask;
  int rc;
  if (!prm.a_mask) {
    BO_CUDA(ctx, cudaMemsetAsync(ws.amask, 0, 4 * (size_t)ws.mask_words, ctx->stream));
    if (a.n_rows > 0) {
      const void* ka = reinterpret_cast<const void*>(&gb_amask_kernel);
      gb_amask_kernel<<<grid_res(ctx, ka, 256, 0, a.n_rows), 256, 0, ctx->stream>>>(a, prm.a_id_max, ws.amask,
                                                                                    ctx->d_err);
      if ((rc = after_launch(ctx, "gb_amask_kernel"))) return rc;
    }
  }
  CatSet cs{};
  cs.n = prm.n_categories;
  for (int i = 0; i < prm.n_categories; ++i) cs.v[i] = prm.categories[i];
  const bool filter = b.n_rows >= kGdFilterRows, pairs = ids <= kGdPairIds && !parts;
  uint32_t* entries = reinterpret_cast<uint32_t*>(ws.slots);
  const int64_t vecs = (ids * (pairs ? 8 : 4) + 15) / 16;
  const void* kc = reinterpret_cast<const void*>(&gd_cfilter_kernel);
  gd_cfilter_kernel<<<grid_res(ctx, kc, 256, 0, std::max<int64_t>((c.n_rows + 31) / 32, vecs / 8)), 256, 0,
                      ctx->stream>>>(c, cs, prm.year_lo, prm.year_hi, code, ws.cbits, filter ? bloom : nullptr,
                                     reinterpret_cast<uint4*>(entries), vecs, meta, pred, kGbMinCapLog2, ws.max_log2);
  if ((rc = after_launch(ctx, "gd_cfilter_kernel"))) return rc;
  const int64_t steps = (b.n_rows + 255) / 256;
  const int64_t lanes = steps * 32;
  if (filter) {
    const auto ks = pairs ? &gd_scan_kernel<true> : &gd_scan_kernel<false>;
    static bool ready[2] = {false, false};
    if (!ready[pairs])
      BO_CUDA(ctx, cudaFuncSetAttribute(reinterpret_cast<const void*>(ks), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kGdSmem));
    ready[pairs] = true;
    const int gs = (int)std::min<int64_t>(ctx->num_sms, (steps + kGdWarps - 1) / kGdWarps);
    BO_CUDA(ctx, launch_dependent(ks, gs, kGdBlock, kGdSmem, ctx->stream, b, c.n_rows, prm.a_id_max,
                                  (const uint8_t*)code, (const uint32_t*)bloom, (const GbMeta*)meta, entries,
                                  ctx->d_err));
    if ((rc = after_launch(ctx, "gd_scan_kernel"))) return rc;
  }
  if (b.n_rows > 0) {
    const uint32_t ranges = (uint32_t)((c.n_rows + kGpRangeBits - 1) / kGpRangeBits);
    const int64_t plane_bytes = steps * 32;
    void* planes = nullptr;
    if (!pairs && filter && ranges >= 1 && ranges <= (uint32_t)kGpMaxRanges &&
        region(ctx, "gb_planes", (size_t)plane_bytes * ranges, &planes) != BO_OK) {
      cudaGetLastError();
      planes = nullptr;
    }
    if (planes) {
      const uint32_t range = (uint32_t)(((c.n_rows + ranges - 1) / ranges + 127) / 128 * 128);
      const size_t smem = range / 8 + 16;
      static bool planes_ready = false;
      if (!planes_ready)
        BO_CUDA(ctx, cudaFuncSetAttribute(reinterpret_cast<const void*>(&gd_planes_kernel),
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kGpRangeBits / 8 + 16)));
      planes_ready = true;
      BO_CUDA(ctx, launch_dependent(&gd_planes_kernel, ctx->num_sms / (int)ranges * (int)ranges, kGpBlock, smem,
                                    ctx->stream, b, c.n_rows, (const uint32_t*)ws.cbits, ranges, range,
                                    (const GbMeta*)meta, filter, static_cast<uint8_t*>(planes), plane_bytes));
      if ((rc = after_launch(ctx, "gd_planes_kernel"))) return rc;
    }
    const auto ka = pairs ? &gd_scan_all_kernel<true, false>
                          : planes ? &gd_scan_all_kernel<false, true> : &gd_scan_all_kernel<false, false>;
    const int ga = grid_res(ctx, reinterpret_cast<const void*>(ka), kGaBlock, 0, lanes);
    const int64_t passes = pairs ? 1 : (4 * ids + kGdPassBytes - 1) / kGdPassBytes, span = (ids + passes - 1) / passes;
    for (int64_t lo = 0; lo < ids; lo += span) {
      BO_CUDA(ctx, launch_dependent(ka, ga, kGaBlock, 0, ctx->stream, b, c.n_rows, (int32_t)lo,
                                    (int32_t)(std::min(lo + span, ids) - 1), (const uint8_t*)code,
                                    (const uint32_t*)ws.cbits, (const uint8_t*)planes, ranges, plane_bytes,
                                    (const GbMeta*)meta, filter, entries));
      if ((rc = after_launch(ctx, "gd_scan_all_kernel"))) return rc;
    }
  }
  const int wa = std::max(1, bit_length((uint64_t)prm.a_id_max));
  const int wc = std::max(1, bit_length((uint64_t)b.n_rows));
  const unsigned long long cmax = (wc >= 64) ? ~0ull : ((1ull << wc) - 1ull);
  const auto kk = parts ? (pairs ? &gd_collect_kernel<true, true> : &gd_collect_kernel<true, false>)
                        : (pairs ? &gd_collect_kernel<false, true> : &gd_collect_kernel<false, false>);
  static bool kk_ready[2] = {false, false};
  if (parts && !kk_ready[pairs])
    BO_CUDA(ctx, cudaFuncSetAttribute(reinterpret_cast<const void*>(kk), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(4u << BO_GB_MAX_LOG2_PARTITIONS)));
  if (parts) kk_ready[pairs] = true;
  BO_CUDA(ctx, launch_dependent(kk, gk, kGcBlock, 4 * (size_t)n_parts, ctx->stream, (const uint32_t*)entries, ids,
                                amask, meta, prm.year_lo, (int)prm.k, wa, cmax, part_counts, n_parts, cand, out));
  if ((rc = after_launch(ctx, "gd_collect_kernel"))) return rc;
  if (pairs || b.n_rows == 0 || prm.k == 0) return BO_OK;
  const void* ky = reinterpret_cast<const void*>(&gd_years_kernel);
  BO_CUDA(ctx, launch_dependent(&gd_years_kernel, grid_res(ctx, ky, 256, 0, lanes), 256, 0, ctx->stream, b, c.n_rows,
                                prm.year_lo, (const uint8_t*)code, out));
  return after_launch(ctx, "gd_years_kernel");
}

int gb_finish(bo_ctx* ctx, bo_gb_result* host, const bo_gb_result* dev) {
  return read_result(ctx, "groupby", host, dev, sizeof(bo_gb_result));
}

int gb_plain_impl(bo_ctx* ctx, const bo_gb_a_cols& a, const bo_gb_b_cols& b, const bo_gb_c_cols& c,
                  const bo_gb_params& prm, bo_gb_result* out_host, int32_t reruns) {
  GbWs ws;
  int rc = gb_workspace(ctx, b, c, prm.a_id_max, &ws);
  if (rc) return rc;
  if ((rc = gb_prepare(ctx, a, c, prm, ws, nullptr, kGbMinCapLog2))) return rc;
  // Exact pre-pass: distinct qualifying groups, then one host round trip.
  if ((rc = gb_launch_scan<0>(ctx, b, c, prm, ws))) return rc;
  const void* kp = reinterpret_cast<const void*>(&gb_popcount_kernel);
  const int gp = grid_res(ctx, kp, 256, 0, ws.mask_words);
  gb_popcount_kernel<<<gp, 256, 0, ctx->stream>>>(ws.dbits, ws.mask_words, ws.meta);
  if ((rc = after_launch(ctx, "gb_popcount_kernel"))) return rc;
  unsigned long long distinct = 0;
  BO_CUDA(ctx, cudaMemcpyAsync(&distinct, &ws.meta->exact_distinct, sizeof(distinct), cudaMemcpyDeviceToHost,
                               ctx->stream));
  BO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const int32_t cl = std::min(ws.max_log2, std::max(kGbMinCapLog2, bit_length(std::max<uint64_t>(distinct, 1) * 2 - 1)));
  // Re-initialise only the group table at the exact size; the filters stay.
  const void* ki = reinterpret_cast<const void*>(&gb_init_kernel);
  const int gi = grid_res(ctx, ki, 256, 0, (int64_t)1 << std::min(ws.max_log2, 24));
  gb_init_kernel<<<gi, 256, 0, ctx->stream>>>(ws.slots, ws.mins, ws.bloom, ws.amask, ws.dbits, ws.mask_words, ws.meta,
                                              nullptr, cl, ws.max_log2, 0);
  if ((rc = after_launch(ctx, "gb_init_kernel"))) return rc;
  void* dout = nullptr;
  if ((rc = region(ctx, "gb_out", sizeof(bo_gb_result), &dout))) return rc;
  bo_gb_result* d = static_cast<bo_gb_result*>(dout);
  if ((rc = gb_aggregate_order(ctx, b, c, prm, ws, d, 0))) return rc;
  if ((rc = gb_finish(ctx, out_host, d))) return rc;
  out_host->reruns = reruns;
  out_host->exact_distinct = (int64_t)distinct;
  if (out_host->overflowed) return set_error(ctx, BO_ERR_OVERFLOW, "groupby: exact-size table overflowed");
  return BO_OK;
}

}  // namespace
}  // namespace bo

using namespace bo;

extern "C" {

int bo_groupby_topk_plain(bo_ctx* ctx, const bo_gb_a_cols* a, const bo_gb_b_cols* b, const bo_gb_c_cols* c,
                          const bo_gb_params* prm, bo_gb_result* out_host) {
  BO_CHECK_CTX(ctx);
  int rc = check_gb(ctx, a, b, c, prm);
  if (rc) return rc;
  if (!out_host) return set_error(ctx, BO_ERR_INVALID, "groupby: null output");
  return gb_plain_impl(ctx, *a, *b, *c, *prm, out_host, 0);
}

int bo_groupby_topk_presized_device(bo_ctx* ctx, const bo_gb_a_cols* a, const bo_gb_b_cols* b,
                                    const bo_gb_c_cols* c, const bo_gb_params* prm, const float* pred_groups_device,
                                    bo_gb_result* out_device) {
  BO_CHECK_CTX(ctx);
  int rc = check_gb(ctx, a, b, c, prm);
  if (rc) return rc;
  if (!pred_groups_device || !out_device) return set_error(ctx, BO_ERR_INVALID, "groupby: null prediction/output");
  GbWs ws;
  if ((rc = gb_workspace(ctx, *b, *c, prm->a_id_max, &ws))) return rc;
  if (gb_dense_fits(*b, *prm, ws, false)) {
    bool took = false;
    rc = gb_dense(ctx, *a, *b, *c, *prm, ws, pred_groups_device, 0, 32, out_device, &took);
    if (rc || took) return rc;
  }
  if ((rc = gb_prepare(ctx, *a, *c, *prm, ws, pred_groups_device, 0))) return rc;
  return gb_aggregate_order(ctx, *b, *c, *prm, ws, out_device, 1);
}

int bo_groupby_topk_presized(bo_ctx* ctx, const bo_gb_a_cols* a, const bo_gb_b_cols* b, const bo_gb_c_cols* c,
                             const bo_gb_params* prm, const float* pred_groups_device, bo_gb_result* out_host) {
  BO_CHECK_CTX(ctx);
  if (!out_host) return set_error(ctx, BO_ERR_INVALID, "groupby: null output");
  void* dout = nullptr;
  int rc = region(ctx, "gb_out", sizeof(bo_gb_result), &dout);
  if (rc) return rc;
  bo_gb_result* d = static_cast<bo_gb_result*>(dout);
  if ((rc = bo_groupby_topk_presized_device(ctx, a, b, c, prm, pred_groups_device, d))) return rc;
  if ((rc = gb_finish(ctx, out_host, d))) return rc;
  if (out_host->overflowed) {
    if ((rc = gb_plain_impl(ctx, *a, *b, *c, *prm, out_host, 1))) return rc;
    out_host->mode = 1;
  }
  return BO_OK;
}

int bo_groupby_topk_partitioned_device(bo_ctx* ctx, const bo_gb_a_cols* a, const bo_gb_b_cols* b,
                                       const bo_gb_c_cols* c, const bo_gb_params* prm, int32_t log2_partitions,
                                       float predicted_joined_rows, bo_gb_result* out_device) {
  BO_CHECK_CTX(ctx);
  int rc = check_gb(ctx, a, b, c, prm);
  if (rc) return rc;
  if (!out_device) return set_error(ctx, BO_ERR_INVALID, "groupby: null output");
  if (log2_partitions < 0 || log2_partitions > BO_GB_MAX_LOG2_PARTITIONS)
    return set_error(ctx, BO_ERR_INVALID, "groupby: log2_partitions %d outside [0, %d]", log2_partitions,
                     BO_GB_MAX_LOG2_PARTITIONS);
  GbWs ws;
  if ((rc = gb_workspace(ctx, *b, *c, prm->a_id_max, &ws))) return rc;
  if (gb_dense_fits(*b, *prm, ws, true)) {
    bool took = false;
    rc = gb_dense(ctx, *a, *b, *c, *prm, ws, nullptr, 1u << log2_partitions,
                  log2_partitions == 0 ? 32u : (uint32_t)(32 - log2_partitions), out_device, &took);
    if (rc || took) return rc;
  }
  // The global group table is not used: initialise the smallest one.
  if ((rc = gb_prepare(ctx, *a, *c, *prm, ws, nullptr, kGbMinCapLog2))) return rc;
  const uint32_t n_parts = 1u << log2_partitions;
  // Records: at most one per joined row, so at most one per B row.  The
  // buffers take that bound while it stays within kRecordBoundBytes (HBM is
  // plentiful: 60M B rows need 1.9 GB for the two record arrays); beyond it
  // they are sized from the predicted joined rows with a margin and slack.
  constexpr double kRecordBoundBytes = 16.0 * (1ull << 30);
  const double bound = (double)b->n_rows + 65536.0;
  double want = bound;
  if (bound * 2 * sizeof(uint4) > kRecordBoundBytes)
    want = std::min(bound, std::max(0.0, (double)predicted_joined_rows) * 1.25 + 65536.0);
  if (want * 2 * sizeof(uint4) > (double)(64ull << 30))
    return set_error(ctx, BO_ERR_INVALID, "groupby: predicted partition records above 64 GiB");
  GbParts parts;
  parts.cap = (uint32_t)std::min(want, (double)0xfffffff0u);
  parts.shift = log2_partitions == 0 ? 32u : (uint32_t)(32 - log2_partitions);
  const size_t rec_bytes = ((size_t)parts.cap * sizeof(uint4) + 255) & ~size_t(255);
  const size_t ctr_bytes = 4 * (3 * (size_t)n_parts + 2) + 256;
  void* pbase = nullptr;
  if ((rc = region(ctx, "gb_parts", 2 * rec_bytes + ctr_bytes, &pbase))) return rc;
  char* pp = static_cast<char*>(pbase);
  parts.records = reinterpret_cast<uint4*>(pp);
  uint4* scattered = reinterpret_cast<uint4*>(pp + rec_bytes);
  uint32_t* ctr = reinterpret_cast<uint32_t*>(pp + 2 * rec_bytes);
  parts.cursor = ctr;                   // [0]
  uint32_t* counts = ctr + 1;           // [1, 1 + n_parts)
  uint32_t* offsets = counts + n_parts; // n_parts + 1
  uint32_t* fill = offsets + n_parts + 1;
  BO_CUDA(ctx, cudaMemsetAsync(ctr, 0, 4 * (1 + (size_t)n_parts), ctx->stream));
  if ((rc = gb_launch_scan<2>(ctx, *b, *c, *prm, ws, ~0ull, parts))) return rc;
  const int wa = std::max(1, bit_length((uint64_t)prm->a_id_max));
  const int wc = std::max(1, bit_length((uint64_t)b->n_rows));
  const unsigned long long cmax = (wc >= 64) ? ~0ull : ((1ull << wc) - 1ull);
  static bool ready = false;
  const void* kh = reinterpret_cast<const void*>(&gb_part_hist_kernel);
  const void* kp = reinterpret_cast<const void*>(&gb_part_agg_kernel);
  if (!ready) {
    BO_CUDA(ctx, cudaFuncSetAttribute(kh, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(4u << BO_GB_MAX_LOG2_PARTITIONS)));
    BO_CUDA(ctx, cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPartSmem));
    ready = true;
  }
  const size_t hsmem = 4 * (size_t)n_parts;
  gb_part_hist_kernel<<<ctx->num_sms * 2, kPartBlock, hsmem, ctx->stream>>>(parts, n_parts, counts);
  if ((rc = after_launch(ctx, "gb_part_hist_kernel"))) return rc;
  gb_part_scan_kernel<<<1, kPartScanBlock, 0, ctx->stream>>>(counts, n_parts, offsets, fill);
  if ((rc = after_launch(ctx, "gb_part_scan_kernel"))) return rc;
  gb_part_scatter_kernel<<<ctx->num_sms * 4, kPartBlock, 0, ctx->stream>>>(parts, fill, scattered);
  if ((rc = after_launch(ctx, "gb_part_scatter_kernel"))) return rc;
  const int gp = (int)std::min<int64_t>(n_parts, (int64_t)ctx->num_sms * occupancy_blocks(kp, kPartBlock, kPartSmem));
  gb_part_agg_kernel<<<std::max(gp, 1), kPartBlock, kPartSmem, ctx->stream>>>(scattered, offsets, (int)n_parts,
                                                                              ws.meta, wa, cmax, ws.keys, ws.vals);
  if ((rc = after_launch(ctx, "gb_part_agg_kernel"))) return rc;
  const uint64_t cap_max = 1ull << ws.max_log2;
  if ((rc = radix_topk_pairs(ctx, ws.keys, ws.vals, (int64_t)cap_max, &ws.meta->n_out, wa + wc, prm->k, ws.tkeys,
                             ws.tvals, ws.keys, ws.vals, wa, &ws.meta->inv_max)))
    return rc;
  gb_topk_kernel<<<1, BO_GB_MAX_K, 0, ctx->stream>>>(ws.tkeys, ws.tvals, ws.meta, prm->k, wa, cmax, 2, out_device);
  return after_launch(ctx, "gb_topk_kernel");
}

int bo_groupby_topk_partitioned(bo_ctx* ctx, const bo_gb_a_cols* a, const bo_gb_b_cols* b, const bo_gb_c_cols* c,
                                const bo_gb_params* prm, int32_t log2_partitions, float predicted_joined_rows,
                                bo_gb_result* out_host) {
  BO_CHECK_CTX(ctx);
  if (!out_host) return set_error(ctx, BO_ERR_INVALID, "groupby: null output");
  void* dout = nullptr;
  int rc = region(ctx, "gb_out", sizeof(bo_gb_result), &dout);
  if (rc) return rc;
  bo_gb_result* d = static_cast<bo_gb_result*>(dout);
  if ((rc = bo_groupby_topk_partitioned_device(ctx, a, b, c, prm, log2_partitions, predicted_joined_rows, d)))
    return rc;
  if ((rc = gb_finish(ctx, out_host, d))) return rc;
  if (out_host->overflowed) {
    if ((rc = gb_plain_impl(ctx, *a, *b, *c, *prm, out_host, 1))) return rc;
    out_host->mode = 2;
  }
  return BO_OK;
}

int bo_groupby_a_mask_device(bo_ctx* ctx, const bo_gb_a_cols* a, int32_t a_id_max, uint32_t* mask_device) {
  BO_CHECK_CTX(ctx);
  if (!a || !mask_device || a_id_max < 0 || a->n_rows < 0 || (a->n_rows > 0 && !a->id))
    return set_error(ctx, BO_ERR_INVALID, "groupby_a_mask: bad argument");
  const int64_t words = ((int64_t)a_id_max + 1 + 31) / 32;
  BO_CUDA(ctx, cudaMemsetAsync(mask_device, 0, sizeof(uint32_t) * (size_t)words, ctx->stream));
  if (a->n_rows == 0) return BO_OK;
  const void* ka = reinterpret_cast<const void*>(&gb_amask_kernel);
  gb_amask_kernel<<<grid_res(ctx, ka, 256, 0, a->n_rows), 256, 0, ctx->stream>>>(*a, a_id_max, mask_device,
                                                                                   ctx->d_err);
  return after_launch(ctx, "gb_amask_kernel");
}

int bo_groupby_distinct_device(bo_ctx* ctx, const bo_gb_a_cols* a, const bo_gb_b_cols* b, const bo_gb_c_cols* c,
                               const bo_gb_params* prm, int64_t* out_device) {
  BO_CHECK_CTX(ctx);
  int rc = check_gb(ctx, a, b, c, prm);
  if (rc) return rc;
  if (!out_device) return set_error(ctx, BO_ERR_INVALID, "groupby: null output");
  GbWs ws;
  if ((rc = gb_workspace(ctx, *b, *c, prm->a_id_max, &ws))) return rc;
  if ((rc = gb_prepare(ctx, *a, *c, *prm, ws, nullptr, kGbMinCapLog2))) return rc;
  if ((rc = gb_launch_scan<0>(ctx, *b, *c, *prm, ws))) return rc;
  const void* kp = reinterpret_cast<const void*>(&gb_popcount_kernel);
  gb_popcount_kernel<<<grid_res(ctx, kp, 256, 0, ws.mask_words), 256, 0, ctx->stream>>>(ws.dbits, ws.mask_words,
                                                                                          ws.meta);
  if ((rc = after_launch(ctx, "gb_popcount_kernel"))) return rc;
  // out[0] = exact distinct groups, out[1] = joined rows
  BO_CUDA(ctx, cudaMemcpyAsync(out_device, &ws.meta->exact_distinct, sizeof(int64_t), cudaMemcpyDeviceToDevice,
                               ctx->stream));
  BO_CUDA(ctx, cudaMemcpyAsync(out_device + 1, &ws.meta->joined, sizeof(int64_t), cudaMemcpyDeviceToDevice,
                               ctx->stream));
  return BO_OK;
}

}  // extern "C"
