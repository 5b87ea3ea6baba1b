// Shared filtered joins: up to 32 joins of the same build and probe tables
// that differ only in their predicate constants (date_lt, segment_eq), in one
// pass over each table -- the serving loop's answer to many concurrent join
// requests over the same device-resident tables, where every solo join would
// stream the same probe side again.  No reference counterpart (the reference
// runs one query per call, bespoke_tpch/query_impl.cpp:159-388); each query's
// result equals the solo filtered join (join.cu), which restates the filtered
// join of run_q3 (bespoke_tpch/query_q3.cpp:182-260).
//
// The queries are sorted by date_lt, so the queries a build row qualifies for
// are "its segment's queries" AND "the queries with date_lt > date" -- a
// suffix of its segment's queries, named by the first of them: with j = the
// number of date_lt <= date,
//   class(row) = first query k >= j of the row's segment (none: no query)
// and query k's rows are those of the classes <= k of its segment.  At most 32
// classes exist, so a key carries one byte and a matching probe row adds to one
// class; the queries' totals are sums over classes at the end.
//   range   the smallest and largest key of all build rows decide how keys are
//           stored:
//   dense   one byte per key value between the smallest and the largest key,
//           where that fits the table's memory (sixteen bytes per build row):
//           15M dense keys are 15 MB that stay in L2;
//   count   else one pass: rows per class and the range of their keys alone, for
//           which the dense form gets a second chance; or
//   hash    slots of key << 32 | class, sized by the union count (rows of any
//           class), behind a Bloom filter;
//   init    clears whichever it is;
//   build   one pass: rows with a class store it (and, dense, are counted, unless
//           they have been: each query's qualifying rows follow from the counts,
//           and the size of the table there would have been); a key already present
//           (two build rows with one key) cannot carry per-query multiplicities
//           in one byte, so it marks the whole call for an exact solo rerun of
//           every query;
//   probe   one pass: each matching row adds its count, T and rr to its class in
//           the warp's shared-memory accumulators; blocks add the classes' totals
//           into 128-bit totals and the last block writes every query's result.
// The kernels of the form that was not chosen return at once.  Measured (B200,
// build 15M, probe 60M, 16 queries, dense keys): 433 us a call (range 14, build
// 113, probe 306; with a counting pass over all columns, 62 us, instead of the
// range: 478) against 2934 us with a query mask per hashed slot and a warp
// reduction per query; keys over the whole 32-bit range (hash): 2703 against
// 2950 us, 25K x 100K rows: 41 and 64 against 77 us.  The line between the forms
// is the table's memory and no lower: just inside it (keys ten apart) dense
// takes 885 us for 2 queries, hash 1656 us just outside (twenty apart).
#include <algorithm>
#include <numeric>

#include "common.cuh"
#include "rows.cuh"
#include "context.cuh"

namespace bo {
namespace {

constexpr int kMq = BO_JOIN_MULTI_MAX;  // queries per call (one mask bit each)
constexpr int kMqBlock = 512;
constexpr int kMqBuildBlock = 256;
constexpr int kMqRowsPerLane = 8;       // probe rows per lane per warp step
constexpr int kMqBuildRows = 8;         // build rows per thread
constexpr int kMqWarps = kMqBlock / 32;
constexpr int kMqMinCapLog2 = 10;

// Predicate constants, queries in date_lt order (sorted index k).
struct MultiQ {
  int32_t n;
  int32_t n_seg;                 // distinct segments among the queries
  int32_t date_lt[kMq];          // ascending
  uint32_t seg_of[kMq];          // compact segment of sorted query k
  uint32_t segmask[kMq];         // queries of compact segment i
  int32_t perm[kMq];             // caller's index of sorted query k
  int16_t seg_idx[256];          // segment byte -> compact segment or -1
};

// Device state of one call ("join_multi_meta" region; cleared by the host
// before every call).  Class codes are 1 + the class's first query; 0 is none.
struct MqState {
  unsigned long long hist[kMq + 1];          // rows per class code
  unsigned long long count[kMq];             // qualifying rows per sorted query
  unsigned long long acc[kMq * 6];           // per class 128-bit match count, sum T, sum rr
  unsigned long long distinct;
  uint32_t key_max, key_nmin;                // largest key and largest ~key, in unsigned order
  uint32_t base, range;                      // dense: smallest key, key values from it to the largest
  uint32_t ticket_range, ticket_count, ticket_probe, dup, overflow;
  int32_t cap_log2, dense;
  int32_t counted, any;                      // by the counting pass; any row with a class
};

__device__ __forceinline__ void mq_load_queries(MultiQ& q, const MultiQ& qv) {
  static_assert(sizeof(MultiQ) % 4 == 0, "copied in words");
  const uint32_t* src = reinterpret_cast<const uint32_t*>(&qv);
  uint32_t* dst = reinterpret_cast<uint32_t*>(&q);
  for (int i = threadIdx.x; i < (int)(sizeof(MultiQ) / 4); i += blockDim.x) dst[i] = src[i];
}

__device__ __forceinline__ uint32_t mq_first_above(const int32_t* date_lt, int n, int32_t date) {
  uint32_t lo = 0, hi = (uint32_t)n;  // first sorted query with date_lt > date
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (date_lt[mid] > date) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

__device__ __forceinline__ uint32_t mq_suffix(uint32_t j) { return j >= 32u ? 0u : (~0u << j); }

// Class code of a build row (0: no query wants it).
__device__ __forceinline__ uint32_t mq_class(const MultiQ& q, int32_t date, uint32_t seg_byte) {
  const int idx = q.seg_idx[seg_byte & 0xffu];
  if (idx < 0) return 0u;
  return (uint32_t)__ffs((int)(q.segmask[idx] & mq_suffix(mq_first_above(q.date_lt, q.n, date))));
}

// Class codes and keys of the kRows build rows from r0 on (codes 0 past the end).
template <int kRows>
__device__ __forceinline__ void mq_build_rows(const bo_join_build_cols& b, const MultiQ& q, int64_t r0,
                                              uint32_t (&code)[kRows], uint32_t (&key)[kRows]) {
  static_assert(kRows == 8, "one 256-bit load of dates and of keys");
  if (r0 + kRows <= b.n_rows) {
    const uint2 sg = ld_stream_v2(b.segment + r0);
    const int8v d = ld_first_v8(b.date + r0), k = ld_first_v8(b.key + r0);
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      code[j] = mq_class(q, d.v[j], (j < 4 ? sg.x : sg.y) >> (8 * (j & 3)));
      key[j] = (uint32_t)k.v[j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      code[j] = 0;
      key[j] = 0;
      if (r0 + j < b.n_rows) {
        code[j] = mq_class(q, b.date[r0 + j], b.segment[r0 + j]);
        key[j] = (uint32_t)b.key[r0 + j];
      }
    }
  }
}

// --------------------------------------------------------------- range ---
constexpr uint32_t kSign = 0x80000000u;  // int32 order as uint32 order

// The block's smallest and largest key into the state's.
__device__ __forceinline__ void mq_take_range(MqState* st, uint32_t kmax, uint32_t nmin) {
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  nmin = __reduce_max_sync(0xffffffffu, nmin);
  if ((threadIdx.x & 31) == 0 && (kmax | nmin)) {
    atomicMax(&st->key_max, kmax);
    atomicMax(&st->key_nmin, nmin);
  }
}

__device__ __forceinline__ void mq_decide(MqState* st, bool rows, uint32_t dense_max) {
  const uint32_t lo = ~__ldcg(&st->key_nmin), hi = __ldcg(&st->key_max);
  const uint64_t range = rows ? (uint64_t)hi - lo + 1 : 0;
  st->dense = range <= dense_max;
  st->base = lo ^ kSign;
  st->range = (uint32_t)range;
}

__global__ void __launch_bounds__(kMqBuildBlock) mq_range_kernel(bo_join_build_cols b, MqState* st,
                                                                 uint32_t dense_max) {
  pdl_launch_dependents();
  const int64_t chunks = (b.n_rows + kMqBuildRows - 1) / kMqBuildRows;
  uint32_t kmax = 0, nmin = 0;
  auto take = [&](int32_t key) {
    const uint32_t k = (uint32_t)key ^ kSign;
    kmax = max(kmax, k);
    nmin = max(nmin, ~k);
  };
  for (int64_t c = (int64_t)blockIdx.x * kMqBuildBlock + threadIdx.x; c < chunks;
       c += (int64_t)gridDim.x * kMqBuildBlock) {
    const int64_t r0 = c * kMqBuildRows;
    if (r0 + kMqBuildRows <= b.n_rows) {
      const int8v k = ld_stream_v8(b.key + r0);
#pragma unroll
      for (int j = 0; j < kMqBuildRows; ++j) take(k.v[j]);
    } else {
      for (int64_t r = r0; r < b.n_rows; ++r) take(b.key[r]);
    }
  }
  // One pair of atomics per block: thousands of warps on two words serialise in L2.
  __shared__ uint32_t bmax, bnmin;
  if (threadIdx.x == 0) bmax = bnmin = 0;
  __syncthreads();
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  nmin = __reduce_max_sync(0xffffffffu, nmin);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&bmax, kmax);
    atomicMax(&bnmin, nmin);
  }
  __syncthreads();
  if (threadIdx.x == 0 && (bmax | bnmin)) {
    atomicMax(&st->key_max, bmax);
    atomicMax(&st->key_nmin, bnmin);
  }
  if (!last_block(&st->ticket_range) || threadIdx.x != 0) return;
  mq_decide(st, b.n_rows > 0, dense_max);
  if (!st->dense) st->key_max = st->key_nmin = 0;  // the counting pass tries the keys of rows with a class
}

// --------------------------------------------------------------- count ---
constexpr int kMqClassCopies = 8;  // of each class's counter: lanes of one class spread over them

// The block's class counters into the call's, and in the last block each
// query's qualifying rows, the union's, and the hash table's size.  True there.
__device__ __forceinline__ bool mq_count_finish(const uint32_t* h, const MultiQ& q, MqState* st, int32_t max_log2) {
  __shared__ unsigned long long tot[kMq + 1];
  __syncthreads();
  if (threadIdx.x <= kMq) {
    uint32_t t = 0;
    for (int i = 0; i < kMqClassCopies; ++i) t += h[threadIdx.x * kMqClassCopies + i];
    if (t) atomicAdd(st->hist + threadIdx.x, (unsigned long long)t);
  }
  if (!last_block(&st->ticket_count)) return false;
  if (threadIdx.x <= kMq) tot[threadIdx.x] = __ldcg(st->hist + threadIdx.x);
  __syncthreads();
  if (threadIdx.x < q.n) {
    const uint32_t k = threadIdx.x;
    unsigned long long c = 0;
    for (uint32_t j = 0; j <= k; ++j)
      if (q.seg_of[j] == q.seg_of[k]) c += tot[j + 1];
    st->count[k] = c;
  }
  if (threadIdx.x == 0) {
    unsigned long long u = 0;
    for (int k = 1; k <= kMq; ++k) u += tot[k];
    const double want = (double)(float)u * 2.0;  // exact count: load <= 0.5
    int32_t cl = kMqMinCapLog2;
    while (cl < max_log2 && (double)(1ull << cl) < want) ++cl;
    st->cap_log2 = cl;
    st->any = u != 0;
  }
  return true;
}

// Where the keys of all rows do not fit the dense form: rows per class before
// the build, and whether the keys of those rows alone fit it.
__global__ void __launch_bounds__(kMqBuildBlock) mq_count_kernel(bo_join_build_cols b, MultiQ qv, MqState* st,
                                                                 uint32_t dense_max, int32_t max_log2) {
  __shared__ MultiQ q;
  __shared__ uint32_t h[(kMq + 1) * kMqClassCopies];
  pdl_launch_dependents();
  pdl_wait();
  if (ld_prior(&st->dense)) return;
  mq_load_queries(q, qv);
  for (int i = threadIdx.x; i < (kMq + 1) * kMqClassCopies; i += kMqBuildBlock) h[i] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t chunks = (b.n_rows + kMqBuildRows - 1) / kMqBuildRows;
  uint32_t kmax = 0, nmin = 0;
  for (int64_t c = (int64_t)blockIdx.x * kMqBuildBlock + threadIdx.x; c < chunks;
       c += (int64_t)gridDim.x * kMqBuildBlock) {
    uint32_t code[kMqBuildRows], key[kMqBuildRows];
    mq_build_rows(b, q, c * kMqBuildRows, code, key);
#pragma unroll
    for (int j = 0; j < kMqBuildRows; ++j) {
      if (!code[j]) continue;
      atomicAdd(h + code[j] * kMqClassCopies + (lane & (kMqClassCopies - 1)), 1u);
      const uint32_t k = key[j] ^ kSign;
      kmax = max(kmax, k);
      nmin = max(nmin, ~k);
    }
  }
  mq_take_range(st, kmax, nmin);
  if (!mq_count_finish(h, q, st, max_log2)) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    st->counted = 1;
    mq_decide(st, st->any != 0, dense_max);
  }
}

// ---------------------------------------------------------------- init ---
__global__ void mq_init_kernel(unsigned long long* slots, uint32_t* bloom, MqState* st) {
  pdl_launch_dependents();
  pdl_wait();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ld_prior(&st->dense)) {
    uint4* v = reinterpret_cast<uint4*>(slots);
    for (uint64_t i = tid; i < ((uint64_t)ld_prior(&st->range) + 15) / 16; i += stride) v[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  const int32_t cl = ld_prior(&st->cap_log2);
  const uint64_t cap = 1ull << cl;
  ulonglong2* s2 = reinterpret_cast<ulonglong2*>(slots);
  for (uint64_t i = tid; i < cap / 2; i += stride) s2[i] = make_ulonglong2(kEmptySlot, kEmptySlot);
  uint4* b4 = reinterpret_cast<uint4*>(bloom);
  for (uint64_t i = tid; i < kBloomWords / 4; i += stride) b4[i] = make_uint4(0, 0, 0, 0);
}

// --------------------------------------------------------------- build ---
// Dense: the class byte is ORed into its word, the old byte tells a repeated
// key; a thread's atomics are all issued before any old value is used.
__global__ void __launch_bounds__(kMqBuildBlock) mq_build_dense_kernel(bo_join_build_cols b, MultiQ qv,
                                                                       uint32_t* __restrict__ bytes, MqState* st,
                                                                       int32_t max_log2) {
  __shared__ MultiQ q;
  __shared__ uint32_t h[(kMq + 1) * kMqClassCopies];
  pdl_launch_dependents();
  mq_load_queries(q, qv);
  for (int i = threadIdx.x; i < (kMq + 1) * kMqClassCopies; i += kMqBuildBlock) h[i] = 0;
  pdl_wait();
  if (!ld_prior(&st->dense)) return;
  __syncthreads();
  const uint32_t copy = threadIdx.x & (kMqClassCopies - 1);
  const uint32_t base = ld_prior(&st->base);
  const int64_t chunks = (b.n_rows + kMqBuildRows - 1) / kMqBuildRows;
  uint32_t dup = 0;
  for (int64_t c = (int64_t)blockIdx.x * kMqBuildBlock + threadIdx.x; c < chunks;
       c += (int64_t)gridDim.x * kMqBuildBlock) {
    uint32_t code[kMqBuildRows], key[kMqBuildRows], old[kMqBuildRows];
    mq_build_rows(b, q, c * kMqBuildRows, code, key);
#pragma unroll
    for (int j = 0; j < kMqBuildRows; ++j) {
      const uint32_t off = key[j] - base;
      old[j] = code[j] ? atomicOr(bytes + (off >> 2), code[j] << (8 * (off & 3u))) : 0u;
    }
#pragma unroll
    for (int j = 0; j < kMqBuildRows; ++j)
      if (code[j]) atomicAdd(h + code[j] * kMqClassCopies + copy, 1u);
#pragma unroll
    for (int j = 0; j < kMqBuildRows; ++j) dup |= (old[j] >> (8 * ((key[j] - base) & 3u))) & 0xffu;
  }
  if (__any_sync(0xffffffffu, dup != 0) && (threadIdx.x & 31) == 0) atomicOr(&st->dup, 1u);
  if (!ld_prior(&st->counted)) mq_count_finish(h, q, st, max_log2);
}

__device__ __forceinline__ void mq_insert(unsigned long long* slots, uint32_t* bloom, uint64_t mask, int32_t key,
                                          uint32_t code, uint32_t& newkeys, uint32_t& dup, uint32_t& full) {
  uint64_t idx = hash32((uint32_t)key) & mask;
  const unsigned long long mine = ((unsigned long long)(uint32_t)key << 32) | code;
  for (uint64_t step = 0; step <= mask; ++step) {
    const unsigned long long old = atomicCAS(slots + idx, kEmptySlot, mine);
    if (old == kEmptySlot) {
      ++newkeys;
      uint32_t w, bits;
      bloom_pos((uint32_t)key, w, bits);
      atomicOr(bloom + w, bits);
      return;
    }
    if ((uint32_t)(old >> 32) == (uint32_t)key) {
      dup = 1;
      return;
    }
    idx = (idx + 1) & mask;
  }
  full = 1;
}

__global__ void __launch_bounds__(kMqBuildBlock) mq_build_kernel(bo_join_build_cols b, MultiQ qv,
                                                                 unsigned long long* slots, uint32_t* bloom,
                                                                 MqState* st) {
  pdl_launch_dependents();
  pdl_wait();
  if (ld_prior(&st->dense)) return;
  __shared__ MultiQ q;
  __shared__ uint32_t queue[kMqBuildBlock / 32][2][32 * kMqBuildRows];
  mq_load_queries(q, qv);
  __syncthreads();
  const uint64_t mask = (1ull << ld_prior(&st->cap_log2)) - 1;
  const int lane = threadIdx.x & 31;
  uint32_t* qk = queue[threadIdx.x >> 5][0];
  uint32_t* qm = queue[threadIdx.x >> 5][1];
  uint32_t newkeys = 0, dup = 0, full = 0;
  const int64_t steps = (b.n_rows + kMqBuildRows - 1) / kMqBuildRows;
  const int64_t steps_w = (steps + 31) & ~int64_t(31);  // whole warps: the queue steps stay converged
  for (int64_t s = (int64_t)blockIdx.x * kMqBuildBlock + threadIdx.x; s < steps_w;
       s += (int64_t)gridDim.x * kMqBuildBlock) {
    uint32_t code[kMqBuildRows], key[kMqBuildRows];
    mq_build_rows(b, q, s * kMqBuildRows, code, key);
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < kMqBuildRows; ++k) any |= (uint32_t)(code[k] != 0u) << k;
    uint32_t total;
    uint32_t pos = warp_exclusive_scan(__popc(any), total);
    if (total == 0) continue;  // warp-uniform
#pragma unroll
    for (int k = 0; k < kMqBuildRows; ++k)
      if ((any >> k) & 1u) {
        qk[pos] = key[k];
        qm[pos] = code[k];
        ++pos;
      }
    __syncwarp();
    for (uint32_t i = lane; i < total; i += 32) mq_insert(slots, bloom, mask, (int32_t)qk[i], qm[i], newkeys, dup, full);
    __syncwarp();
  }
  const uint32_t wn = warp_sum_u32(newkeys);
  const unsigned wd = __any_sync(0xffffffffu, dup), wf = __any_sync(0xffffffffu, full);
  if (lane == 0) {
    if (wn) atomicAdd(&st->distinct, (unsigned long long)wn);
    if (wd) atomicOr(&st->dup, 1u);
    if (wf) atomicOr(&st->overflow, 1u);
  }
}

// --------------------------------------------------------------- probe ---
// Per-class sums of one warp in shared memory, 32-bit words added to by
// atomics; four copies of each class (by lane) keep lanes of one class from
// queueing on one word.  A matching row adds T in two 16-bit halves and
// 1 << 20 | rr (rr < 100): at most kMqFlush rows may be added before a flush.
constexpr int kMqCopies = 4;
constexpr int kMqAccWords = 3;
constexpr uint32_t kMqFlush = 4095;  // count < 2^12 above bit 20; sum rr < 2^19; halves < 2^28

struct MqWarpAcc {
  uint32_t w[kMqAccWords][kMq * kMqCopies];
};

// Lane k's 64-bit totals of class k, taken out of the warp's accumulators.
struct MqAcc {
  unsigned long long cnt = 0, t = 0, rr = 0;
  uint32_t bad = 0;
};

__device__ __forceinline__ void mq_flush(MqWarpAcc& wa, MqAcc& acc) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int c = 0; c < kMqCopies; ++c) {
    const int i = lane * kMqCopies + c;
    const uint32_t lo = wa.w[0][i], hi = wa.w[1][i], pk = wa.w[2][i];
    wa.w[0][i] = wa.w[1][i] = wa.w[2][i] = 0;
    acc.cnt += pk >> 20;
    acc.rr += pk & 0xfffffu;
    acc.t += lo + ((unsigned long long)hi << 16);
  }
  __syncwarp();
}

__device__ __forceinline__ void mq_add(MqWarpAcc& wa, uint32_t code, uint64_t p, uint64_t d, MqAcc& acc) {
  if (p >= 0x80000000ull || d > 100u) {
    acc.bad |= kErrValueRange;
    return;
  }
  const uint32_t m = 100u - (uint32_t)d, pq = (uint32_t)p / 100u, pr = (uint32_t)p - pq * 100u;
  const uint32_t rm = pr * m, rq = rm / 100u, T = pq * m + rq;
  const uint32_t i = (code - 1u) * kMqCopies + (threadIdx.x & (kMqCopies - 1));
  atomicAdd(&wa.w[0][i], T & 0xffffu);
  atomicAdd(&wa.w[1][i], T >> 16);
  atomicAdd(&wa.w[2][i], (1u << 20) | (rm - rq * 100u));
}

// The block's totals per class into the 128-bit totals; the last block writes
// every query's result (the sum of its segment's classes up to it).
__device__ __forceinline__ void mq_finish(MqWarpAcc* wa, int warps, MqAcc& acc, MqState* st, const MultiQ& qv,
                                          bo_join_result* out, uint32_t* err) {
  __shared__ __int128 cls[kMq][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  mq_flush(wa[warp], acc);
  if (acc.bad) raise_error(err, acc.bad);
  // The accumulators' memory now carries each warp's 64-bit totals.
  static_assert(sizeof(MqWarpAcc) >= sizeof(unsigned long long) * 3 * 32, "per-warp totals fit");
  unsigned long long* mine = reinterpret_cast<unsigned long long*>(wa + warp);
  mine[lane * 3] = acc.cnt;
  mine[lane * 3 + 1] = acc.t;
  mine[lane * 3 + 2] = acc.rr;
  __syncthreads();
  if (threadIdx.x < 32 * 3) {
    unsigned long long v = 0;  // per block: < 2^32 rows x < 2^31, fits 64 bits
    for (int w = 0; w < warps; ++w) v += reinterpret_cast<unsigned long long*>(wa + w)[threadIdx.x];
    if (v) atomic_add_i128(st->acc + 2 * threadIdx.x, (__int128)v);
  }
  if (!last_block(&st->ticket_probe)) return;
  if (threadIdx.x < 32 * 3) cls[threadIdx.x / 3][threadIdx.x % 3] = load_i128(st->acc + 2 * threadIdx.x);
  __syncthreads();
  if (threadIdx.x < qv.n) {
    const int k = threadIdx.x;
    uint32_t fbad = 0;
    __int128 m = 0, t = 0, rr = 0;
    for (int c = 0; c <= k; ++c)
      if (qv.seg_of[c] == qv.seg_of[k]) {
        m += cls[c][0];
        t += cls[c][1];
        rr += cls[c][2];
      }
    bo_join_result r;
    r.build_rows = (int64_t)__ldcg(&st->count[k]);
    r.distinct_keys = r.build_rows;  // no key repeats (else the call is marked for rerun)
    r.match_count = narrow_i64(m, fbad);
    r.sum_trunc = to_bo_i128(t);
    r.sum_exact = to_bo_i128(t * 100 + rr);
    r.capacity_log2 = __ldcg(&st->cap_log2);
    r.overflowed = (int32_t)(__ldcg(&st->dup) | __ldcg(&st->overflow));
    r.reruns = 0;
    r.mode = 0;
    out[qv.perm[k]] = r;
    if (fbad) raise_error(err, fbad);
  }
}

// Dense: a warp owns 256 consecutive rows per step, lane-strided (row base + 32 j
// + lane) so that the price / discount loads of one j coalesce.  Bound by the
// random byte loads: L1 79% and L2 71% busy, DRAM 48% (305 us for 60M rows).
constexpr int kMqDenseBlock = 256;

__global__ void __launch_bounds__(kMqDenseBlock) mq_probe_dense_kernel(bo_join_probe_cols p,
                                                                       const uint8_t* __restrict__ bytes, MqState* st,
                                                                       bo_join_result* out, MultiQ qv, uint32_t* err) {
  pdl_launch_dependents();
  pdl_wait();
  if (!ld_prior(&st->dense)) return;
  constexpr int kWarps = kMqDenseBlock / 32;
  __shared__ __align__(16) MqWarpAcc wa[kWarps];
  for (int i = threadIdx.x; i < (int)(sizeof(wa) / 4); i += kMqDenseBlock) reinterpret_cast<uint32_t*>(wa)[i] = 0;
  __syncthreads();
  const uint32_t base_key = ld_prior(&st->base), range = ld_prior(&st->range);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = p.n_rows;
  constexpr int kStep = 32 * kMqRowsPerLane;
  const int64_t steps = (n + kStep - 1) / kStep;
  MqAcc acc;
  uint32_t added = 0;
  for (int64_t s = (int64_t)blockIdx.x * kWarps + warp; s < steps; s += (int64_t)gridDim.x * kWarps) {
    const int64_t r0 = s * kStep + lane;
    uint32_t off[kMqRowsPerLane], code[kMqRowsPerLane];
#pragma unroll
    for (int j = 0; j < kMqRowsPerLane; ++j)
      off[j] = r0 + 32 * j < n ? (uint32_t)__ldcs(p.fk + r0 + 32 * j) - base_key : ~0u;
#pragma unroll
    for (int j = 0; j < kMqRowsPerLane; ++j) code[j] = off[j] < range ? ld_prior(bytes + off[j]) : 0u;
    uint64_t pr[kMqRowsPerLane], dc[kMqRowsPerLane];
#pragma unroll
    for (int j = 0; j < kMqRowsPerLane; ++j) {
      pr[j] = code[j] ? (uint64_t)__ldcs(p.price + r0 + 32 * j) : 0u;
      dc[j] = code[j] ? (uint64_t)__ldcs(p.discount + r0 + 32 * j) : 0u;
    }
    if (added + kStep > kMqFlush) {
      mq_flush(wa[warp], acc);
      added = 0;
    }
    added += kStep;
#pragma unroll
    for (int j = 0; j < kMqRowsPerLane; ++j)
      if (code[j]) mq_add(wa[warp], code[j], pr[j], dc[j], acc);
  }
  mq_finish(wa, kWarps, acc, st, qv, out, err);
}

// Resolves the warp's queued candidates (as probe_resolve in rows.cuh, R = 2
// per lane per round) and adds the matches to their classes.
__device__ __forceinline__ void mq_resolve(const int32_t* qf, const uint8_t* qo, uint32_t total, int64_t base,
                                           const unsigned long long* slots, uint64_t mask, const int64_t* price,
                                           const int64_t* disc, MqWarpAcc& wa, MqAcc& acc) {
  constexpr int R = 2;
  const int lane = threadIdx.x & 31;
  for (uint32_t i0 = 0; i0 < total; i0 += 32 * R) {
    int32_t key[R];
    int64_t row[R];
    uint64_t idx[R];
    unsigned long long v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t i = i0 + r * 32 + lane;
      const bool ok = i < total;
      key[r] = ok ? qf[i] : 0;
      row[r] = ok ? base + qo[i] : 0;
      idx[r] = hash32((uint32_t)key[r]) & mask;
      v[r] = ok ? ld_prior(slots + idx[r]) : kEmptySlot;
    }
    uint32_t code[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      code[r] = 0;
      if (v[r] != kEmptySlot) {
        if ((uint32_t)(v[r] >> 32) == (uint32_t)key[r])
          code[r] = (uint32_t)v[r];
        else
          code[r] = (uint32_t)probe_slow<false>(slots, mask, idx[r], (uint32_t)key[r], ~0ull);
      }
    }
    uint64_t pr[R], dc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      pr[r] = code[r] ? (uint64_t)__ldg(price + row[r]) : 0u;
      dc[r] = code[r] ? (uint64_t)__ldg(disc + row[r]) : 0u;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (code[r]) mq_add(wa, code[r], pr[r], dc[r], acc);
  }
}

__global__ void __launch_bounds__(kMqBlock, 2) mq_probe_kernel(bo_join_probe_cols p, const unsigned long long* slots,
                                                              const uint32_t* bloom_g, MqState* st,
                                                              bo_join_result* out, MultiQ qv, uint32_t* err) {
  pdl_launch_dependents();
  pdl_wait();
  if (ld_prior(&st->dense)) return;
  extern __shared__ __align__(128) uint32_t bloom_s[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int32_t q_fk[kMqWarps][32 * kMqRowsPerLane];
  __shared__ uint8_t q_off[kMqWarps][32 * kMqRowsPerLane];
  MqWarpAcc* wa = reinterpret_cast<MqWarpAcc*>(bloom_s + kBloomWords);
  for (int i = threadIdx.x; i < (int)(kMqWarps * sizeof(MqWarpAcc) / 4); i += kMqBlock)
    reinterpret_cast<uint32_t*>(wa)[i] = 0;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_arrive_expect_tx(&bar, kBloomBytes);
    bulk_copy_g2s(bloom_s, bloom_g, kBloomBytes, &bar);
  }
  __syncthreads();
  // Without the filter (a timed-out copy) every row probes the table: same answer.
  const bool use_bloom = mbar_wait_bounded(&bar, 0, kWaitLimitNs);
  __shared__ uint32_t all_ones;
  if (threadIdx.x == 0) all_ones = 0xffffffffu;
  __syncthreads();
  const uint32_t* bl = use_bloom ? bloom_s : &all_ones;
  const uint32_t wmask = use_bloom ? (kBloomWords - 1u) : 0u;
  MqAcc acc;
  if (!use_bloom) acc.bad |= kErrSpinTimeout;
  const uint64_t mask = (1ull << ld_prior(&st->cap_log2)) - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t* qf = q_fk[warp];
  uint8_t* qo = q_off[warp];
  const int64_t n = p.n_rows;
  constexpr int kStep = 32 * kMqRowsPerLane;
  const int64_t steps = (n + kStep - 1) / kStep;
  uint32_t added = 0;
  for (int64_t s = (int64_t)blockIdx.x * kMqWarps + warp; s < steps; s += (int64_t)gridDim.x * kMqWarps) {
    const int64_t base = s * kStep;
    const int64_t r0 = base + lane * kMqRowsPerLane;
    int32_t fk[kMqRowsPerLane];
    uint32_t valid = 0xffu;
    if (r0 + kMqRowsPerLane <= n) {
      const int8v f0 = ld_stream_v8(p.fk + r0);
#pragma unroll
      for (int k = 0; k < kMqRowsPerLane; ++k) fk[k] = f0.v[k];
    } else {
      valid = 0;
#pragma unroll
      for (int k = 0; k < kMqRowsPerLane; ++k) {
        fk[k] = 0;
        if (r0 + k < n) {
          fk[k] = p.fk[r0 + k];
          valid |= 1u << k;
        }
      }
    }
    uint32_t hit = 0;
#pragma unroll
    for (int k = kMqRowsPerLane - 1; k >= 0; --k) hit = (hit << 1) | bloom_test(bl, wmask, (uint32_t)fk[k]);
    hit &= valid;
    uint32_t total;
    uint32_t pos = warp_exclusive_scan(__popc(hit), total);
#pragma unroll
    for (int k = 0; k < kMqRowsPerLane; ++k)
      if ((hit >> k) & 1u) {
        qf[pos] = fk[k];
        qo[pos] = (uint8_t)(lane * kMqRowsPerLane + k);
        ++pos;
      }
    if (added + total > kMqFlush) {
      mq_flush(wa[warp], acc);
      added = 0;
    }
    added += total;
    __syncwarp();
    mq_resolve(qf, qo, total, base, slots, mask, p.price, p.discount, wa[warp], acc);
    __syncwarp();
  }
  if (!use_bloom) mbar_wait_bounded(&bar, 0, kWaitLimitNs);  // the copy may still be in flight
  mq_finish(wa, kMqWarps, acc, st, qv, out, err);
}

int ceil_log2_u64(uint64_t v) {
  int l = 0;
  while ((1ull << l) < v) ++l;
  return l;
}

int mq_grid(bo_ctx* ctx, const void* k, int block, size_t smem, int64_t items) {
  const int64_t resident = (int64_t)ctx->num_sms * occupancy_blocks(k, block, smem);
  return (int)std::max<int64_t>(1, std::min<int64_t>(resident, (items + block - 1) / block));
}

int mq_check(bo_ctx* ctx, const bo_join_build_cols* b, const bo_join_probe_cols* p, const bo_join_params* prm,
             int32_t n) {
  if (!b || !p || !prm) return set_error(ctx, BO_ERR_INVALID, "join_multi: null argument");
  if (n < 1 || n > kMq) return set_error(ctx, BO_ERR_INVALID, "join_multi: %d queries (1..%d)", n, kMq);
  if (b->n_rows < 0 || p->n_rows < 0 || b->n_rows > 0x7fffffffll)
    return set_error(ctx, BO_ERR_INVALID, "join_multi: row counts");
  if (b->n_rows > 0 && (!b->key || !b->date || !b->segment || !aligned32(b->key) || !aligned32(b->date) ||
                        !aligned32(b->segment)))
    return set_error(ctx, BO_ERR_INVALID, "join_multi: build column null or not 32-byte aligned");
  if (p->n_rows > 0 && (!p->fk || !p->price || !p->discount || !aligned32(p->fk) || !aligned32(p->price) ||
                        !aligned32(p->discount)))
    return set_error(ctx, BO_ERR_INVALID, "join_multi: probe column null or not 32-byte aligned");
  for (int i = 0; i < n; ++i)
    if (prm[i].segment_eq < 0 || prm[i].segment_eq > 255)
      return set_error(ctx, BO_ERR_INVALID, "join_multi: segment_eq %d outside uint8", prm[i].segment_eq);
  return BO_OK;
}

}  // namespace
}  // namespace bo

using namespace bo;

extern "C" int bo_join_multi_device(bo_ctx* ctx, const bo_join_build_cols* b, const bo_join_probe_cols* p,
                                    const bo_join_params* prm, int32_t n_queries, bo_join_result* out_device) {
  BO_CHECK_CTX(ctx);
  int rc = mq_check(ctx, b, p, prm, n_queries);
  if (rc) return rc;
  if (!out_device) return set_error(ctx, BO_ERR_INVALID, "join_multi: null output");
  // Sort the queries by date_lt (stable) and compact their segments.
  MultiQ q{};
  q.n = n_queries;
  std::vector<int> order(n_queries);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return prm[x].date_lt < prm[y].date_lt; });
  for (int i = 0; i < 256; ++i) q.seg_idx[i] = -1;
  for (int k = 0; k < n_queries; ++k) {
    const bo_join_params& x = prm[order[k]];
    q.date_lt[k] = x.date_lt;
    q.perm[k] = order[k];
    int16_t& si = q.seg_idx[x.segment_eq];
    if (si < 0) si = (int16_t)q.n_seg++;
    q.seg_of[k] = (uint32_t)si;
    q.segmask[si] |= 1u << k;
  }
  const int32_t max_log2 = std::max(kMqMinCapLog2, ceil_log2_u64((uint64_t)std::max<int64_t>(b->n_rows, 1) * 2));
  void* ptr = nullptr;
  if ((rc = region(ctx, "join_multi_slots", sizeof(unsigned long long) << max_log2, &ptr))) return rc;
  auto* slots = static_cast<unsigned long long*>(ptr);
  if ((rc = region(ctx, "join_multi_bloom", kBloomBytes, &ptr))) return rc;
  auto* bloom = static_cast<uint32_t*>(ptr);
  if ((rc = region(ctx, "join_multi_meta", sizeof(MqState), &ptr))) return rc;
  auto* st = static_cast<MqState*>(ptr);
  BO_CUDA(ctx, cudaMemsetAsync(st, 0, sizeof(MqState), ctx->stream));

  // Dense form while the key values from smallest to largest fit the table's memory.
  const uint32_t dense_max = (uint32_t)std::min<uint64_t>(sizeof(unsigned long long) << max_log2, 0xfffffff0ull);
  const int64_t chunks = (b->n_rows + kMqBuildRows - 1) / kMqBuildRows;
  const void* kr = reinterpret_cast<const void*>(&mq_range_kernel);
  mq_range_kernel<<<mq_grid(ctx, kr, kMqBuildBlock, 0, chunks), kMqBuildBlock, 0, ctx->stream>>>(*b, st, dense_max);
  if ((rc = after_launch(ctx, "mq_range_kernel"))) return rc;
  const void* kc = reinterpret_cast<const void*>(&mq_count_kernel);
  BO_CUDA(ctx, launch_dependent(&mq_count_kernel, mq_grid(ctx, kc, kMqBuildBlock, 0, chunks), kMqBuildBlock, 0,
                                ctx->stream, *b, q, st, dense_max, max_log2));
  if ((rc = after_launch(ctx, "mq_count_kernel"))) return rc;
  const void* ki = reinterpret_cast<const void*>(&mq_init_kernel);
  BO_CUDA(ctx, launch_dependent(&mq_init_kernel, mq_grid(ctx, ki, 256, 0, (int64_t)1 << std::min(max_log2, 24)), 256, 0,
                                ctx->stream, slots, bloom, st));
  if ((rc = after_launch(ctx, "mq_init_kernel"))) return rc;
  const void* kd = reinterpret_cast<const void*>(&mq_build_dense_kernel);
  BO_CUDA(ctx, launch_dependent(&mq_build_dense_kernel, mq_grid(ctx, kd, kMqBuildBlock, 0, chunks), kMqBuildBlock, 0,
                                ctx->stream, *b, q, reinterpret_cast<uint32_t*>(slots), st, max_log2));
  if ((rc = after_launch(ctx, "mq_build_dense_kernel"))) return rc;
  const void* kb = reinterpret_cast<const void*>(&mq_build_kernel);
  BO_CUDA(ctx, launch_dependent(&mq_build_kernel, mq_grid(ctx, kb, kMqBuildBlock, 0, chunks), kMqBuildBlock, 0,
                                ctx->stream, *b, q, slots, bloom, st));
  if ((rc = after_launch(ctx, "mq_build_kernel"))) return rc;
  const int64_t lanes = (p->n_rows + kMqRowsPerLane - 1) / kMqRowsPerLane;
  const void* kq = reinterpret_cast<const void*>(&mq_probe_dense_kernel);
  BO_CUDA(ctx, launch_dependent(&mq_probe_dense_kernel, mq_grid(ctx, kq, kMqDenseBlock, 0, lanes), kMqDenseBlock, 0,
                                ctx->stream, *p, reinterpret_cast<const uint8_t*>(slots), st, out_device, q,
                                ctx->d_err));
  if ((rc = after_launch(ctx, "mq_probe_dense_kernel"))) return rc;
  const void* kp = reinterpret_cast<const void*>(&mq_probe_kernel);
  constexpr size_t smem = kBloomBytes + kMqWarps * sizeof(MqWarpAcc);
  static bool ready = false;
  if (!ready) {
    BO_CUDA(ctx, cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ready = true;
  }
  BO_CUDA(ctx, launch_dependent(&mq_probe_kernel, mq_grid(ctx, kp, kMqBlock, smem, lanes), kMqBlock, smem, ctx->stream,
                                *p, (const unsigned long long*)slots, (const uint32_t*)bloom, st, out_device, q,
                                ctx->d_err));
  return after_launch(ctx, "mq_probe_kernel");
}

extern "C" int bo_join_multi_host(bo_ctx* ctx, const bo_join_build_cols* b, const bo_join_probe_cols* p,
                                  const bo_join_params* prm, int32_t n_queries, bo_join_result* out_host) {
  BO_CHECK_CTX(ctx);
  if (!out_host) return set_error(ctx, BO_ERR_INVALID, "join_multi: null output");
  void* dout = nullptr;
  int rc = region(ctx, "join_multi_out", sizeof(bo_join_result) * kMq, &dout);
  if (rc) return rc;
  if ((rc = bo_join_multi_device(ctx, b, p, prm, n_queries, static_cast<bo_join_result*>(dout)))) return rc;
  if ((rc = read_result(ctx, "join_multi", out_host, dout, sizeof(bo_join_result) * (size_t)n_queries))) return rc;
  if (out_host[0].overflowed) {  // repeated build keys: every query alone, exactly
    for (int i = 0; i < n_queries; ++i) {
      if ((rc = bo_join_plain(ctx, b, p, &prm[i], &out_host[i]))) return rc;
      out_host[i].reruns = 1;
    }
  }
  return BO_OK;
}
