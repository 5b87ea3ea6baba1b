// TPC-H Q3 over the storage-plan layout: run_q3 of bespoke_tpch/query_q3.cpp:153-365.
//
// The reference walks the orders sorted by date, takes the qualifying ones
// (orderdate < D, customer in the segment; :207-322) and sums each one's
// lineitems with shipdate > D through its CSR range (:219-260), then sorts all
// resulting orders by revenue desc, orderdate asc (:348-355).  On the GPU the
// same result comes from three data-parallel passes and a sort:
//   cust   segment membership as a bitmap over custkey (:182-204);
//   orders orderdate < D and the customer's bit (:311-322): a qualifying order
//          sets its orderkey's bit and clears its revenue;
//   lines  every lineitem with shipdate > D tests its orderkey's bit (neighbouring
//          lineitems share words of that bitmap, so the test stays in L1, where
//          the map from orderkey to row is 4 bytes per key), and only the ~2%
//          that pass look up the row and add their discounted price with 64-bit
//          atomics.  An order's first such lineitem (`has_lineitem`, :248) sets
//          its bit in a second bitmap and lists the order;
//   sort   the listed orders by (revenue desc, orderdate asc, orderkey): the
//          two-launch sort of small_sort.cuh, sized on the device; more orders
//          than it takes come out of the second bitmap in orderkey order and
//          are sorted after the count was read back;
//   rows   staged in shared memory and stored straight into the caller's
//          mapped pinned memory where it is that, so the query synchronises
//          once.  The reference's std::sort leaves rows equal in both keys in
//          unspecified order; here they keep orderkey order, a canonical form of
//          the same result.
// Measured (1.5M orders, 6M lineitems, 11K rows): 72 us a call (orders 6, lines 14,
// sort 15, rows 10) against 138 us with the map read for every lineitem (21 us),
// the result compacted from a bitmap in three launches, a cluster sort (32 us),
// five memsets and two copies back.
#include <algorithm>

#include "common.cuh"
#include "compact.cuh"
#include "context.cuh"
#include "small_sort.cuh"

namespace bo {
namespace {

constexpr int kQ3Block = 256;
constexpr unsigned long long kRevBits = 47;  // revenue < 2^47 (checked) so (rev, date) packs into 63 bits

__global__ void q3_cust_kernel(const int32_t* __restrict__ custkey, const uint16_t* __restrict__ seg, int64_t n,
                               int32_t segment_code, int32_t bound, uint32_t* __restrict__ mask) {
  pdl_launch_dependents();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if ((int32_t)seg[i] != segment_code) continue;
    const int32_t k = custkey[i];
    if (k >= 0 && k < bound) atomicOr(mask + (k >> 5), 1u << (k & 31));
  }
}

// Qualifying orders into the orderkey bitmap, if the map leads back to them.
__global__ void q3_orders_kernel(const int32_t* __restrict__ o_orderkey, const int32_t* __restrict__ o_custkey,
                                 const int16_t* __restrict__ o_orderdate, int64_t n, int16_t date_offset, int32_t bound,
                                 const uint32_t* __restrict__ mask, const int32_t* __restrict__ key_to_row,
                                 int64_t n_map, uint32_t* __restrict__ qual, unsigned long long* __restrict__ rev) {
  pdl_launch_dependents();
  pdl_wait();
  // Four rows at a time, each step's loads requested together.
  constexpr int kRows = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kRows * stride) {
    int32_t c[kRows], key[kRows];
    uint32_t take = 0;
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const int64_t i = i0 + j * stride;
      c[j] = i < n && o_orderdate[i] < date_offset ? o_custkey[i] : -1;
    }
#pragma unroll
    for (int j = 0; j < kRows; ++j)
      take |= (uint32_t)(c[j] >= 0 && c[j] < bound && ((ld_prior(mask + (c[j] >> 5)) >> (c[j] & 31)) & 1u)) << j;
    if (!take) continue;
#pragma unroll
    for (int j = 0; j < kRows; ++j) key[j] = (take >> j) & 1u ? o_orderkey[i0 + j * stride] : -1;
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const int64_t i = i0 + j * stride;
      if (key[j] < 0 || (int64_t)key[j] >= n_map || __ldg(key_to_row + key[j]) != (int32_t)i) continue;
      rev[i] = 0;
      atomicOr(qual + (key[j] >> 5), 1u << (key[j] & 31));
    }
  }
}

// What the lineitem pass does with a row past the date whose order qualifies.
// New orders are listed per block first, with one reservation at the end; past
// a full list (over a million result rows) each warp reserves for its lanes.
constexpr int kQ3List = 1024;

struct Q3Lines {
  const int32_t* key_to_row;
  const int32_t* dprice;
  unsigned long long* rev;
  uint32_t* kept;            // bit per orderkey: the order has been listed
  uint2* list;               // {orderkey, row}
  unsigned long long* n_out;
  __device__ __forceinline__ void add(int64_t i, int32_t key, uint2* mine, uint32_t* n_mine) const {
    const int32_t row = __ldg(key_to_row + key);
    atomicAdd(rev + row, (unsigned long long)(int64_t)__ldg(dprice + i));
    const uint32_t bit = 1u << (key & 31);
    if (atomicOr(kept + (key >> 5), bit) & bit) return;
    const uint32_t at = atomicAdd(n_mine, 1u);
    if (at < (uint32_t)kQ3List) {
      mine[at] = make_uint2((uint32_t)key, (uint32_t)row);
      return;
    }
    const uint32_t with = __activemask(), lane = threadIdx.x & 31, first = __ffs(with) - 1;
    unsigned long long pos = 0;
    if (lane == first) pos = atomicAdd(n_out, (unsigned long long)__popc(with));
    pos = __shfl_sync(with, pos, first) + __popc(with & ((1u << lane) - 1u));
    list[pos] = make_uint2((uint32_t)key, (uint32_t)row);
  }
  __device__ __forceinline__ void flush(const uint2* mine, const uint32_t* n_mine, unsigned long long* base) const {
    __syncthreads();
    const uint32_t n = *n_mine < (uint32_t)kQ3List ? *n_mine : (uint32_t)kQ3List;
    if (threadIdx.x == 0) *base = n ? atomicAdd(n_out, (unsigned long long)n) : 0ull;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) list[*base + i] = mine[i];
  }
};

__device__ __forceinline__ unsigned long long q3_sort_key(unsigned long long r, int16_t date, uint32_t* err) {
  if (r >> kRevBits) raise_error(err, kErrValueRange);
  const unsigned long long inv = ((1ull << kRevBits) - 1ull) - (r & ((1ull << kRevBits) - 1ull));
  return (inv << 16) | (unsigned long long)(uint16_t)(date + 32768);
}

// Listed order i as an item of the small sort.
struct Q3Item {
  const uint2* list;
  const unsigned long long* rev;
  const int16_t* o_orderdate;
  uint32_t* err;
  __device__ __forceinline__ uint4 operator()(uint32_t i) const {
    const uint2 e = list[i];
    return ss_item(q3_sort_key(rev[e.y], o_orderdate[e.y], err), e.x, e.y);
  }
};

// More orders than the small sort takes: sort keys of the kept orderkeys.
// vals[i] holds a kept orderkey on entry and its order row on return.
__global__ void q3_key2_kernel(uint32_t* __restrict__ vals, const int32_t* __restrict__ key_to_row,
                               const unsigned long long* __restrict__ rev, const int16_t* __restrict__ o_orderdate,
                               const unsigned long long* n_out, unsigned long long* __restrict__ keys, uint32_t* err) {
  const unsigned long long n = *n_out;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t row = (uint32_t)__ldg(key_to_row + vals[i]);  // valid: the lineitem pass marked it
    vals[i] = row;
    keys[i] = q3_sort_key(rev[row], o_orderdate[row], err);
  }
}

// The result rows (the first min(*n_out, limit)), one per thread, staged in
// shared memory and stored as consecutive 16-byte words: out may be mapped
// pinned host memory (the rows then cross PCIe as whole writes) or device
// memory.  out is 16-byte aligned.
constexpr int kQ3RowsBlock = 128;

__global__ void __launch_bounds__(kQ3RowsBlock) q3_gather_kernel(
    const uint32_t* __restrict__ vals, const unsigned long long* __restrict__ rev,
    const int32_t* __restrict__ o_orderkey, const int16_t* __restrict__ o_orderdate,
    const int32_t* __restrict__ o_shippriority, const unsigned long long* n_out, int64_t limit,
    bo_tpch_q3_row* __restrict__ out, HostWords words) {
  __shared__ bo_tpch_q3_row stage[kQ3RowsBlock];
  pdl_wait();
  if (words.words) {
    if (blockIdx.x == 0 && threadIdx.x == 0) words.store();
    if (*words.overflow) return;  // vals were not sorted
  }
  static_assert((sizeof(bo_tpch_q3_row) * kQ3RowsBlock) % 16 == 0, "a block's rows are whole 16-byte words");
  const unsigned long long nd = *n_out;
  const int64_t n = nd < (unsigned long long)limit ? (int64_t)nd : limit;
  for (int64_t base = (int64_t)blockIdx.x * kQ3RowsBlock; base < n; base += (int64_t)gridDim.x * kQ3RowsBlock) {
    const int64_t i = base + threadIdx.x;
    if (i < n) {
      const uint32_t row = ld_prior(vals + i);
      bo_tpch_q3_row r;
      r.revenue_raw = (int64_t)ld_prior(rev + row);
      r.orderkey = o_orderkey[row];
      r.shippriority = o_shippriority ? o_shippriority[row] : 0;
      r.orderdate_offset = o_orderdate[row];
      r.pad0 = 0;
      r.pad1 = 0;
      stage[threadIdx.x] = r;
    }
    __syncthreads();
    const int rows = (int)(n - base < kQ3RowsBlock ? n - base : kQ3RowsBlock);
    const int words = (int)((sizeof(bo_tpch_q3_row) * rows + 15) / 16);  // the tail word may carry pad bytes
    const uint4* src = reinterpret_cast<const uint4*>(stage);
    uint4* dst = reinterpret_cast<uint4*>(out + base);
    if (rows == kQ3RowsBlock || (sizeof(bo_tpch_q3_row) * rows) % 16 == 0) {
      for (int w = threadIdx.x; w < words; w += kQ3RowsBlock) dst[w] = src[w];
    } else {  // a ragged last block: 8-byte words, so nothing past row n - 1 is written
      const uint2* s2 = reinterpret_cast<const uint2*>(stage);
      uint2* d2 = reinterpret_cast<uint2*>(out + base);
      for (int w = threadIdx.x; w < (int)(sizeof(bo_tpch_q3_row) / 8) * rows; w += kQ3RowsBlock) d2[w] = s2[w];
    }
    __syncthreads();
  }
}

// The lineitem pass, 8 rows per thread per step: one 16-byte load of 8
// shipdates, and for a step with any row past the date one 32-byte pair of
// orderkey loads; the bits of the passing rows are all requested before any is
// used, and the few rows that qualify are put off to a second phase, so that
// the stream does not wait on their lookups (row, price, atomics) step by
// step.  Columns 16-byte aligned (kWide; else every row goes through the scalar
// loop); the last n % 8 rows go through the scalar loop.
constexpr int kQ3Later = 1024;  // rows put off per block; further ones are done at once

template <bool kWide>
__global__ void __launch_bounds__(kQ3Block) q3_lineitem_kernel(const int32_t* __restrict__ l_orderkey,
                                                               const int16_t* __restrict__ l_shipdate, int64_t n,
                                                               int16_t date_offset, int64_t n_map,
                                                               const uint32_t* __restrict__ qual, Q3Lines lines) {
  __shared__ uint2 mine[kQ3List];
  __shared__ int64_t later_row[kQ3Later];
  __shared__ int32_t later_key[kQ3Later];
  __shared__ uint32_t n_mine, n_later;
  __shared__ unsigned long long base;
  if (threadIdx.x == 0) n_mine = n_later = 0;
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait();
  const int64_t chunks = kWide ? n >> 3 : 0;
  auto qualifies = [&](int64_t row, int32_t key) {
    const uint32_t at = atomicAdd(&n_later, 1u);
    if (at < (uint32_t)kQ3Later) {
      later_row[at] = row;
      later_key[at] = key;
    } else {
      lines.add(row, key, mine, &n_mine);
    }
  };
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t c = tid; c < chunks; c += stride) {
    const int64_t r0 = c << 3;
    const int4 sd = ld_stream_v4(l_shipdate + r0);
    const int4 k0 = ld_stream_v4(l_orderkey + r0), k1 = ld_stream_v4(l_orderkey + r0 + 4);
    const uint32_t sw[4] = {(uint32_t)sd.x, (uint32_t)sd.y, (uint32_t)sd.z, (uint32_t)sd.w};
    const int32_t key[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
    uint32_t word[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int16_t d = (int16_t)((sw[k >> 1] >> (16 * (k & 1))) & 0xffffu);
      word[k] = d > date_offset && key[k] >= 0 && (int64_t)key[k] < n_map ? ld_prior(qual + (key[k] >> 5)) : 0u;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if ((word[k] >> (key[k] & 31)) & 1u) qualifies(r0 + k, key[k]);
  }
  for (int64_t i = (chunks << 3) + tid; i < n; i += stride) {
    if (l_shipdate[i] <= date_offset) continue;
    const int32_t key = l_orderkey[i];
    if (key < 0 || (int64_t)key >= n_map || !((ld_prior(qual + (key >> 5)) >> (key & 31)) & 1u)) continue;
    qualifies(i, key);
  }
  __syncthreads();
  const uint32_t todo = n_later < (uint32_t)kQ3Later ? n_later : (uint32_t)kQ3Later;
  for (uint32_t i = threadIdx.x; i < todo; i += kQ3Block) lines.add(later_row[i], later_key[i], mine, &n_mine);
  lines.flush(mine, &n_mine, &base);
}

int grid_of(bo_ctx* ctx, int64_t items) {
  const int64_t need = (items + kQ3Block - 1) / kQ3Block;
  return (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)ctx->num_sms * 8));
}

}  // namespace
}  // namespace bo

using namespace bo;

extern "C" int bo_tpch_q3(bo_ctx* ctx, const bo_tpch_q3_tables* t, int16_t date_offset, int32_t segment_code,
                          bo_tpch_q3_row* out_host, int64_t max_rows, int64_t* n_rows) {
  BO_CHECK_CTX(ctx);
  if (!t || !n_rows || max_rows < 0 || (max_rows > 0 && !out_host))
    return set_error(ctx, BO_ERR_INVALID, "q3: null argument");
  if (t->n_customer < 0 || t->n_orders < 0 || t->n_lineitem < 0 || t->n_orderkey_map < 0 || t->custkey_bound < 0)
    return set_error(ctx, BO_ERR_INVALID, "q3: negative size");
  if (t->n_orders > 0xffffffffll) return set_error(ctx, BO_ERR_INVALID, "q3: more than 2^32 orders");
  if ((t->n_customer > 0 && (!t->c_custkey || !t->c_mktsegment)) ||
      (t->n_orders > 0 && (!t->o_orderkey || !t->o_custkey || !t->o_orderdate)) ||
      (t->n_orderkey_map > 0 && !t->orderkey_to_row) ||
      (t->n_lineitem > 0 && (!t->l_orderkey || !t->l_shipdate || !t->l_discounted_price)))
    return set_error(ctx, BO_ERR_INVALID, "q3: null column");
  *n_rows = 0;
  const int64_t no = t->n_orders;
  if (no == 0 || segment_code < 0) return BO_OK;  // no order can qualify (unknown segment: none, :176-183)
  const int64_t mask_words = ((int64_t)t->custkey_bound + 31) / 32 + 1;
  const int64_t kept_words = t->n_orderkey_map / 32 + 1;
  const int64_t tiles = (kept_words + kBitmapTileWords - 1) / kBitmapTileWords;
  size_t total = 0;
  auto add = [&](size_t b) { total += (b + 255) & ~size_t(255); };
  add(64);
  add(4 * (size_t)mask_words);
  add(4 * (size_t)kept_words);  // orderkeys of qualifying orders
  add(4 * (size_t)kept_words);  // orderkeys with a counted lineitem
  add(8 * (size_t)no);          // revenue
  add(8 * (size_t)no);          // keys
  add(4 * (size_t)no);          // vals
  add(8 * (size_t)no);          // listed orders / tmp keys
  add(4 * (size_t)no);          // tmp vals
  add(sizeof(bo_tpch_q3_row) * (size_t)no);
  add(4 * (size_t)std::max<int64_t>(tiles, 1));  // bitmap compaction's tile counts
  add(kSsItemBytes);
  add(4 * (size_t)kSmallSortMax);
  void* base = nullptr;
  int rc = region(ctx, "q3_ws", total, &base);
  if (rc) return rc;
  char* p = static_cast<char*>(base);
  unsigned long long* n_out = carve<unsigned long long>(p, 8);
  uint32_t* mask = carve<uint32_t>(p, (size_t)mask_words);
  uint32_t* qual = carve<uint32_t>(p, (size_t)kept_words);
  uint32_t* kept = carve<uint32_t>(p, (size_t)kept_words);
  const size_t zeroed = (size_t)(p - static_cast<char*>(base));
  unsigned long long* rev = carve<unsigned long long>(p, (size_t)no);
  unsigned long long* keys = carve<unsigned long long>(p, (size_t)no);
  uint32_t* vals = carve<uint32_t>(p, (size_t)no);
  unsigned long long* tkeys = carve<unsigned long long>(p, (size_t)no);
  uint32_t* tvals = carve<uint32_t>(p, (size_t)no);
  bo_tpch_q3_row* rows = carve<bo_tpch_q3_row>(p, (size_t)no);
  uint32_t* tile_counts = carve<uint32_t>(p, (size_t)std::max<int64_t>(tiles, 1));
  char* items = carve<char>(p, kSsItemBytes);
  uint32_t* sorted = carve<uint32_t>(p, (size_t)kSmallSortMax);
  uint2* list = reinterpret_cast<uint2*>(tkeys);
  uint32_t* overflow = reinterpret_cast<uint32_t*>(n_out + 1);
  // The count, the overflow word and the bitmaps start at zero.
  BO_CUDA(ctx, cudaMemsetAsync(base, 0, zeroed, ctx->stream));
  q3_cust_kernel<<<grid_of(ctx, t->n_customer), kQ3Block, 0, ctx->stream>>>(
      t->c_custkey, t->c_mktsegment, t->n_customer, segment_code, t->custkey_bound, mask);
  if ((rc = after_launch(ctx, "q3_cust_kernel"))) return rc;
  BO_CUDA(ctx, launch_dependent(&q3_orders_kernel, grid_of(ctx, no), kQ3Block, 0, ctx->stream, t->o_orderkey,
                                t->o_custkey, t->o_orderdate, no, date_offset, t->custkey_bound,
                                (const uint32_t*)mask, t->orderkey_to_row, t->n_orderkey_map, qual, rev));
  if ((rc = after_launch(ctx, "q3_orders_kernel"))) return rc;
  const bool wide = aligned16(t->l_orderkey) && aligned16(t->l_shipdate);
  const Q3Lines lines{t->orderkey_to_row, t->l_discounted_price, rev, kept, list, n_out};
  BO_CUDA(ctx, launch_dependent(wide ? &q3_lineitem_kernel<true> : &q3_lineitem_kernel<false>,
                                grid_of(ctx, wide ? (t->n_lineitem + 7) / 8 : t->n_lineitem), kQ3Block, 0, ctx->stream,
                                t->l_orderkey, t->l_shipdate, t->n_lineitem, date_offset, t->n_orderkey_map,
                                (const uint32_t*)qual, lines));
  if ((rc = after_launch(ctx, "q3_lineitem_kernel"))) return rc;
  // The sort without the result's size on the host, and the rows straight into
  // out_host when it is mapped pinned memory: the query synchronises once.
  if ((rc = small_sort(ctx, Q3Item{list, rev, t->o_orderdate, ctx->d_err}, n_out, items, sorted, overflow))) return rc;
  bo_tpch_q3_row* direct = max_rows > 0 ? static_cast<bo_tpch_q3_row*>(mapped_device_ptr(out_host)) : nullptr;
  auto gather = [&](const uint32_t* order, HostWords words) -> int {
    const int64_t lim = direct ? std::min<int64_t>(max_rows, no) : no;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((lim + kQ3RowsBlock - 1) / kQ3RowsBlock,
                                                                 (int64_t)ctx->num_sms * 8));
    BO_CUDA(ctx, launch_dependent(&q3_gather_kernel, grid, kQ3RowsBlock, 0, ctx->stream, order,
                                  (const unsigned long long*)rev, t->o_orderkey, t->o_orderdate, t->o_shippriority,
                                  (const unsigned long long*)n_out, lim, direct ? direct : rows, words));
    return after_launch(ctx, "q3_gather_kernel");
  };
  if ((rc = gather(sorted, HostWords{ctx->h_word, n_out, overflow, ctx->d_err}))) return rc;
  int64_t ns = 0;
  bool over = false;
  if ((rc = read_host_words(ctx, "q3", no, &ns, &over))) return rc;
  if (over) {
    // Orders with a counted lineitem in ascending orderkey order (the order
    // query_q3.cpp:348-355 leaves ties in), then one stable sort.
    if ((rc = bitmap_compact(ctx, kept, kept_words, tile_counts, vals, n_out))) return rc;
    q3_key2_kernel<<<grid_of(ctx, ns), kQ3Block, 0, ctx->stream>>>(vals, t->orderkey_to_row, rev, t->o_orderdate,
                                                                   n_out, keys, ctx->d_err);
    if ((rc = after_launch(ctx, "q3_key2_kernel"))) return rc;
    if ((rc = radix_sort_pairs(ctx, keys, vals, tkeys, tvals, ns, 0, 64, nullptr))) return rc;
    if ((rc = gather(vals, HostWords{}))) return rc;
  }
  const int64_t m = std::min<int64_t>(ns, max_rows);
  if (!direct && m > 0)
    BO_CUDA(ctx, cudaMemcpyAsync(out_host, rows, sizeof(bo_tpch_q3_row) * (size_t)m, cudaMemcpyDeviceToHost,
                                 ctx->stream));
  if (over || (!direct && m > 0)) {
    uint32_t bits = 0;
    if ((rc = consume_device_errors(ctx, &bits))) return rc;
    if ((rc = device_error_status(ctx, bits, "q3"))) return rc;
  }
  *n_rows = ns;
  return BO_OK;
}
