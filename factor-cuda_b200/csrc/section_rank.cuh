// section_rank.cuh -- exact ranks of one section (a date's row of f32 keys) by
// buckets spread over the section's own values.
//
// A radix sort of a section moves every (key, column) pair through shared
// memory once per digit, and its match-based digit ranking is a serial chain
// per warp.  Ranks do not need the pairs in order: it is enough to know, for
// each cell, how many pairs are smaller.
//   1. The key range [kmin, kmax] is cut into K equal bins, and a histogram
//      says how many cells each bin holds.
//   2. A bin gets as many buckets as it has cells (plus one), spread evenly
//      over the bin: bucket(key) = start[bin] + floor(frac * width[bin]), with
//      bin and frac the high and low words of one 64-bit product.  Every step
//      is monotone in the key, so equal keys share a bucket and buckets are
//      ordered, whatever the histogram says; it only decides how even they are.
//   3. One counting pass over the buckets, one scan, one scatter of the
//      (key, column) words into bucket slots.
//   4. A cell's rank is its bucket's start plus the number of smaller words in
//      its bucket (two cells on average): the first four slots are compared
//      without a loop.
// A section whose buckets come out crowded (many equal values, or a cluster
// far narrower than a bin) is better sorted by radix: spread_place returns
// false and the caller takes its radix form.
#pragma once

#include "row_io.cuh"

namespace fcb {

// Threads of one SM the section kernels are compiled for: 64 registers each.
// Fewer registers (three 512-thread CTAs per SM) spill and take longer.
constexpr int kSmThreads = 1024;

// Largest bucket, and largest mean bucket seen by a cell (sum of squared
// sizes over cells), that the in-bucket counts take.  The largest bucket also
// bounds the 9-bit fields of the tie words.
constexpr uint32_t kSpreadMaxBucket = 500;
constexpr uint32_t kSpreadMeanBucket = 24;
// Equal neighbours (columns 2i, 2i + 1) above which a section goes to its
// radix form before any bucket is counted: twice their number estimates the
// mean number of cells that share a cell's value.
constexpr uint32_t kSpreadMaxEqualPairs = 8;
// A bucket above this size (a few equal values, as a rule) is ranked by warps,
// 32 of its words at a time against all of them, and not by its cells' own
// threads, whose warps would wait for the longest loop.
constexpr uint32_t kSpreadHeavy = 16;
// A section whose bins hold, by the mean over its cells, more than this
// fraction of it is a cluster far narrower than its range.  (Above 1024 cells:
// the few bins of a narrow block hold as much of an ordinary section, whose keys
// lie within a few exponents, and there the counting pass costs little.)
constexpr uint32_t kSpreadBinShare = 8;

// One block shape: NT threads with V vectors of four cells each.
template <int NT, int V>
struct SectionShape {
  static constexpr int kThreads = NT, kVectors = V, kCap = 4 * NT * V;
};

// Calls go(SectionShape<NT, V>{}) with the block shape for sections of N cells,
// many of them.  A section takes the same time however many of its block's
// cells it fills (rank + IC: 12 to 14 ps per cell of capacity, whatever the
// shape), so the shapes follow the width closely.  2 M cells x 8 factors as
// sections of 250, 500, 768, 1500 and 2500 cells: 0.72 ms -> 0.23, 0.38 -> 0.22,
// 0.26 -> 0.20, 0.24 -> 0.20, 0.24 -> 0.19, against shapes of 256 x 1, 256 x 2
// and 384 x 2 alone.  At 5000 cells 448 x 3 takes 47 us per 1218 dates of
// cs_rank, 512 x 3 51, 256 x 5 58 and 1024 x 2 78.
template <typename Go>
auto section_shape(int N, Go&& go) {
  if (N <= 256) return go(SectionShape<64, 1>{});
  if (N <= 512) return go(SectionShape<128, 1>{});
  if (N <= 768) return go(SectionShape<192, 1>{});
  if (N <= 1024) return go(SectionShape<256, 1>{});
  if (N <= 1536) return go(SectionShape<192, 2>{});
  if (N <= 2048) return go(SectionShape<256, 2>{});
  if (N <= 2560) return go(SectionShape<320, 2>{});
  if (N <= 3072) return go(SectionShape<256, 3>{});
  if (N <= 4096) return go(SectionShape<512, 2>{});
  if (N <= 5376) return go(SectionShape<448, 3>{});
  if (N <= 6144) return go(SectionShape<512, 3>{});
  if (N <= 8192) return go(SectionShape<512, 4>{});
  return go(SectionShape<1024, 4>{});
}

// Up to one section per SM the CTAs do not share SMs: wider CTAs shorten each
// (one date of 5000 takes 17 us a call, most of it on the host).
constexpr int kFewSections = 148;
template <typename Go>
auto section_shape_few(int N, Go&& go) {
  if (N <= 1024) return section_shape(N, go);
  if (N <= 4096) return go(SectionShape<1024, 1>{});
  if (N <= 8192) return go(SectionShape<1024, 2>{});
  return go(SectionShape<1024, 4>{});
}

template <int NT, int V>
struct SpreadLayout {
  static constexpr int K = 2 * NT;  // bins: two per thread
  static_assert(V <= 4, "the list of heavy buckets fits the bins");
  // counters one thread scans: they cover every bucket (a power of two where
  // that wastes little; 32 for V = 4 would spill)
  static constexpr int P = V == 1 ? 8 : V <= 3 ? 16 : 4 * V + 4;
  size_t red, tab, knots, bits, bits2, cnt, mem, total;
  int S;  // counter stride: bucket b is counter (b % P) * S + b / P
  __host__ __device__ explicit SpreadLayout(int n) {
    size_t o = 0;
    red = o; o += 1024;
    tab = o; o += size_t(K) * 4;
    knots = tab; o = tab + size_t(K > kCdfKnots ? K : kCdfKnots) * 4;  // k_ric_learned's table
    bits = o; o = al16(o + size_t(mark_words(n)) * 4);   // two bitmaps over positions
    bits2 = o; o = al16(o + size_t(mark_words(n)) * 4);  // for the kernels' own use
    S = ((n + K + P - 1) / P + 3) & ~3;  // at most n + K buckets
    cnt = o; o += size_t(P) * S * 4;
    mem = o; o = al16(o + size_t(n + 4) * 8);  // the four words after the last cell's are the pad
    total = o;
  }
  static_assert(4 * V * NT + K <= P * NT, "one scan step covers every bucket");
};

// One word per warp in shared memory -> block result, in every thread.
template <int NW>
FCB_DEV uint32_t warps_min(const uint32_t* r) {
  return __reduce_min_sync(kFull, lane_id() < NW ? r[lane_id()] : 0xFFFFFFFFu);
}
template <int NW>
FCB_DEV uint32_t warps_max(const uint32_t* r) {
  return __reduce_max_sync(kFull, lane_id() < NW ? r[lane_id()] : 0u);
}
template <int NW>
FCB_DEV uint32_t warps_sum(const uint32_t* r) {
  return __reduce_add_sync(kFull, lane_id() < NW ? r[lane_id()] : 0u);
}
// Sum of the words of the warps before this one.
template <int NW>
FCB_DEV uint32_t warps_before(const uint32_t* r) {
  return __reduce_add_sync(kFull, lane_id() < (threadIdx.x >> 5) ? r[lane_id()] : 0u);
}

// Shared-memory accesses under a predicate, without a branch around them.
FCB_DEV void smem_inc_if(bool p, uint32_t addr) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p red.shared.add.u32 [%1], 1;\n}\n" ::"r"(uint32_t(p)),
               "r"(addr)
               : "memory");
}
FCB_DEV uint32_t smem_fetch_inc_if(bool p, uint32_t addr) {
  uint32_t v = 0u;
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %1, 0;\n @p atom.shared.add.u32 %0, [%2], 1;\n}\n"
               : "+r"(v)
               : "r"(uint32_t(p)), "r"(addr)
               : "memory");
  return v;
}
FCB_DEV uint32_t smem_load_if(bool p, uint32_t addr) {
  uint32_t v = 0u;
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %1, 0;\n @p ld.shared.u32 %0, [%2];\n}\n"
               : "+r"(v)
               : "r"(uint32_t(p)), "r"(addr)
               : "memory");
  return v;
}
FCB_DEV void smem_store2_if(bool p, uint32_t addr, uint32_t lo, uint32_t hi) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p st.shared.v2.u32 [%1], {%2, %3};\n}\n" ::"r"(
                   uint32_t(p)),
               "r"(addr), "r"(lo), "r"(hi)
               : "memory");
}

struct SpreadTotals {
  int m;           // valid cells
  bool heavy;      // some bucket is above kSpreadHeavy
  uint32_t range;  // largest valid key less the smallest
  uint32_t largest;  // largest bucket: no value is shared by more cells
};

// Counters -> packed (start | size << 16) per bucket.  Thread t takes the P
// consecutive buckets from P * t on; their counters lie S words apart, so a
// warp's accesses are free of bank conflicts.  red: words [128, 160).  One
// barrier inside; ends without one.
template <int NW, int P>
FCB_DEV void bucket_scan(uint32_t* cnt, int S, uint32_t* red) {
  const int tid = static_cast<int>(threadIdx.x);
  uint32_t v[P], tot = 0u;
  if (tid < S) {
#pragma unroll
    for (int j = 0; j < P; ++j) v[j] = cnt[j * S + tid];
#pragma unroll
    for (int j = 0; j < P; ++j) tot += v[j];
  }
  const uint32_t inc = warp_inclusive_sum(tot);
  if (lane_id() == 31) red[128 + (tid >> 5)] = inc;
  __syncthreads();
  uint32_t run = warps_before<NW>(red + 128) + inc - tot;
  if (tid < S) {
#pragma unroll
    for (int j = 0; j < P; ++j) {
      cnt[j * S + tid] = run + (v[j] << 14);
      run += v[j];
    }
  }
}

// Column of cell c of this thread in the vector layout.
template <int NT>
FCB_DEV uint32_t cell_col(int c) { return 4u * ((c >> 2) * NT + threadIdx.x) + (c & 3); }

// Counts the cells (key[c] <= range) into their buckets: buckets(j, b) gives
// the buckets of the four cells of vector j (anything for the others).  The
// counters are zero before.  W[c] becomes the counter index | slot << 16, with
// slot the cell's arrival number in its bucket, so that the largest slot is
// the largest bucket's size less one and twice the slots' sum is the sum of
// squared sizes less m.  Ends with a barrier.  red: words [160, 224).
struct CountTotals {
  uint32_t largest, squares;  // largest bucket; sum of squared sizes less m
};
template <int NT, int V, typename Buckets>
FCB_DEV CountTotals count_cells(const uint32_t (&key)[4 * V], uint32_t range, const SpreadLayout<NT, V>& L, uint8_t* sm,
                                uint32_t (&W)[4 * V], Buckets buckets) {
  constexpr int NW = NT / 32, P = SpreadLayout<NT, V>::P;
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  const uint32_t cnt_s = smem_u32(sm + L.cnt);
  uint32_t sum = 0u, mx = 0u;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    uint32_t b[4];
    buckets(j, b);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      const uint32_t q = (b[k] % P) * L.S + b[k] / P;
      const uint32_t s = smem_fetch_inc_if(key[c] <= range, cnt_s + 4u * q);
      sum += s;
      mx = max(mx, s);
      W[c] = q | (s << 16);
    }
  }
  sum = __reduce_add_sync(kFull, sum);
  mx = __reduce_max_sync(kFull, mx);
  if (lane_id() == 0) {
    red[160 + (threadIdx.x >> 5)] = sum;
    red[192 + (threadIdx.x >> 5)] = mx;
  }
  __syncthreads();
  return CountTotals{warps_max<NW>(red + 192) + 1u, 2u * warps_sum<NW>(red + 160)};
}

// Scans the counters and scatters the cells into their bucket slots: W[c] of
// a counted cell becomes its bucket's start | size << 14, 0 for the others;
// mem holds the (key << 32 | column) words grouped by bucket, then four
// all-ones words.  Ends with a barrier.
template <int NT, int V>
FCB_DEV void scatter_cells(const uint32_t (&key)[4 * V], uint32_t range, int m, const SpreadLayout<NT, V>& L,
                           uint8_t* sm, uint32_t (&W)[4 * V]) {
  uint32_t* cnt = reinterpret_cast<uint32_t*>(sm + L.cnt);
  const uint32_t cnt_s = smem_u32(cnt), mem_s = smem_u32(sm + L.mem);
  bucket_scan<NT / 32, SpreadLayout<NT, V>::P>(cnt, L.S, reinterpret_cast<uint32_t*>(sm + L.red));
  if (threadIdx.x < 4) reinterpret_cast<unsigned long long*>(sm + L.mem)[m + threadIdx.x] = ~0ull;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < V; ++j) {  // four cells' loads in flight at a time
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = smem_load_if(key[4 * j + k] <= range, cnt_s + 4u * (W[4 * j + k] & 0xFFFFu));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      const uint32_t p = (w[k] & 0x3FFFu) + (W[c] >> 16);
      smem_store2_if(key[c] <= range, mem_s + 8u * p, cell_col<NT>(c), key[c]);
      W[c] = w[k];
    }
  }
  __syncthreads();
}

// Places the valid cells (key[c] != kInvalidKey32) in bucket slots.  key[c]
// becomes the distance from the smallest valid key, above T.range for the
// invalid cells.  On true, W[c] of a valid cell is its bucket's start | size
// << 14 and mem its words (scatter_cells).  On false (crowded buckets) shared memory holds nothing
// of use, and the valid cells are still those at or below T.range, in order.  Uniform across
// the block; every thread calls; ends with a barrier.  T.m == 0 returns true
// with nothing placed but the pad.
template <int NT, int V>
FCB_DEV bool spread_place(uint32_t (&key)[4 * V], const SpreadLayout<NT, V>& L, uint8_t* sm, uint32_t (&W)[4 * V],
                          SpreadTotals& T) {
  constexpr int C = 4 * V, NW = NT / 32, K = SpreadLayout<NT, V>::K, P = SpreadLayout<NT, V>::P;
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  uint32_t* tab = reinterpret_cast<uint32_t*>(sm + L.tab);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(sm + L.cnt);
  const uint32_t tab_s = smem_u32(tab);
  const int tid = static_cast<int>(threadIdx.x), wi = tid >> 5;
  // ---- key range; clear the bins and the bucket counters
  *reinterpret_cast<uint2*>(tab + 2 * tid) = make_uint2(0u, 0u);
  for (int k = tid; k < P / 4 * L.S; k += NT) reinterpret_cast<uint4*>(cnt)[k] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) red[224] = 0u;
  uint32_t lo = kInvalidKey32, hi = 0u, eq = 0u;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    lo = min(lo, key[c]);
    hi = max(hi, key[c] + 1u);  // 0 for an invalid cell
    if (c % 2 == 0) eq += key[c] == key[c + 1] && key[c] != kInvalidKey32 ? 1u : 0u;
  }
  lo = __reduce_min_sync(kFull, lo);
  hi = __reduce_max_sync(kFull, hi);
  eq = __reduce_add_sync(kFull, eq);
  if (lane_id() == 0) {
    red[wi] = lo;
    red[32 + wi] = hi;
    red[64 + wi] = eq;
  }
  __syncthreads();
  const uint32_t kmin = warps_min<NW>(red), range = warps_max<NW>(red + 32) - 1u - kmin;
  if (warps_sum<NW>(red + 64) > kSpreadMaxEqualPairs) {
    T.range = kInvalidKey32 - 1u;  // (the keys are as they were)
    __syncthreads();  // the caller reuses the shared memory
    return false;
  }
  if (kmin == kInvalidKey32) {  // no valid cell
    T.m = 0;
    T.heavy = false;
    T.range = T.largest = 0u;
#pragma unroll
    for (int c = 0; c < C; ++c) W[c] = 0u;
    if (tid < 4) reinterpret_cast<unsigned long long*>(sm + L.mem)[tid] = ~0ull;
    __syncthreads();  // (the caller also reuses red)
    return true;
  }
  T.range = range;
  // distance * scale < K * 2^32: the quotient is rounded below the exact one
  const uint32_t scale =
      static_cast<uint32_t>(fminf(static_cast<float>(K) * 4294967296.0f * (1.0f - 1.0f / 1048576.0f) /
                                      (static_cast<float>(range) + 1.0f),
                                  4294963200.0f));
#pragma unroll
  for (int c = 0; c < C; ++c) {
    key[c] -= kmin;  // an invalid cell stays above range
    smem_inc_if(key[c] <= range, tab_s + 4u * __umulhi(key[c], scale));
  }
  __syncthreads();
  // ---- bin -> (first bucket, buckets)
  {
    const uint2 v = *reinterpret_cast<const uint2*>(tab + 2 * tid);
    const uint32_t w0 = v.x + 1u, w1 = v.y + 1u;
    const uint32_t inc = warp_inclusive_sum(w0 + w1);
    const uint32_t sq = __reduce_add_sync(kFull, v.x * v.x + v.y * v.y);
    if (lane_id() == 31) {
      red[96 + wi] = inc;
      red[192 + wi] = sq;
    }
    __syncthreads();
    const uint32_t ex = warps_before<NW>(red + 96) + inc - w0 - w1;
    T.m = static_cast<int>(warps_sum<NW>(red + 96)) - K;
    const uint32_t m = static_cast<uint32_t>(T.m);
    if (m > 1024u && warps_sum<NW>(red + 192) > m * m / kSpreadBinShare) {
      __syncthreads();  // the caller reuses the shared memory
      return false;
    }
    *reinterpret_cast<uint2*>(tab + 2 * tid) = make_uint2(ex | (w0 << 16), (ex + w0) | (w1 << 16));
  }
  __syncthreads();
  // ---- counts, scan, scatter
  const CountTotals ct = count_cells<NT, V>(key, range, L, sm, W, [&](int j, uint32_t (&b)[4]) {
    uint32_t bw[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)  // four cells' loads in flight at a time
      bw[k] = smem_load_if(key[4 * j + k] <= range, tab_s + 4u * __umulhi(key[4 * j + k], scale));
#pragma unroll
    for (int k = 0; k < 4; ++k) b[k] = (bw[k] & 0xFFFFu) + __umulhi(key[4 * j + k] * scale, bw[k] >> 16);
  });
  if (ct.largest > kSpreadMaxBucket || ct.squares > (kSpreadMeanBucket - 1u) * static_cast<uint32_t>(T.m)) {
    __syncthreads();  // the caller reuses the shared memory
    return false;
  }
  T.heavy = ct.largest > kSpreadHeavy;
  T.largest = ct.largest;
  scatter_cells<NT, V>(key, range, T.m, L, sm, W);
  return true;
}

FCB_DEV unsigned long long smem_load64(uint32_t addr) {
  unsigned long long v;
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
  return v;
}

// What a cell's words count in its bucket, from slot k on.
struct InBucket {
  uint32_t before = 0u, less = 0u, le = 0u;  // smaller words; smaller keys; keys no larger
  template <bool TIES>
  FCB_DEV void add(unsigned long long o, unsigned long long mine) {
    before += o < mine ? 1u : 0u;
    if (TIES) {
      less += static_cast<uint32_t>(o >> 32) < static_cast<uint32_t>(mine >> 32) ? 1u : 0u;
      le += static_cast<uint32_t>(o >> 32) <= static_cast<uint32_t>(mine >> 32) ? 1u : 0u;
    }
  }
  // the bucket starts at s: the sorted position, or the tie word
  template <bool TIES>
  FCB_DEV uint32_t result(uint32_t s) const {
    return TIES ? (s + less) | ((before - less) << 14) | ((le - less) << 23) : s + before;
  }
};

// The scanned buckets above kSpreadHeavy, one item (start | part << 16, size)
// per 32 words; *items (0 before) counts them.
FCB_DEV void list_heavy(const uint32_t* cnt, int counters, uint2* list, uint32_t* items) {
  for (int i = static_cast<int>(threadIdx.x); i < counters; i += static_cast<int>(blockDim.x)) {
    const uint32_t w = cnt[i], n = w >> 14;
    if (n > kSpreadHeavy) {  // (an empty bucket at 2^14 reads n = 1)
      const uint32_t parts = (n + 31u) / 32u, at = atomicAdd(items, parts);
      for (uint32_t k = 0; k < parts; ++k) list[at + k] = make_uint2((w & 0x3FFFu) | (k << 16), n);
    }
  }
}

// Buckets above kSpreadHeavy: a word per column, over the bucket counters, with
// the cell's sorted position or (TIES) its tie word.  The buckets are listed
// where the bins were; each warp takes 32 words of one against all of its
// words (broadcast reads).  Call when some bucket is that large (uniform);
// ends with a barrier.
template <int NT, int V, bool TIES>
FCB_DEV void rank_heavy(const SpreadLayout<NT, V>& L, uint8_t* sm) {
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  uint2* list = reinterpret_cast<uint2*>(sm + L.tab);
  uint32_t* by_col = reinterpret_cast<uint32_t*>(sm + L.cnt);
  const uint32_t mem_s = smem_u32(sm + L.mem);
  list_heavy(by_col, SpreadLayout<NT, V>::P * L.S, list, &red[224]);
  __syncthreads();
  const int items = static_cast<int>(red[224]);
  for (int it = static_cast<int>(threadIdx.x >> 5); it < items; it += NT / 32) {
    const uint2 w = list[it];
    const uint32_t s = w.x & 0xFFFFu, n = w.y, i = (w.x >> 16) * 32u + lane_id();
    const unsigned long long mine = i < n ? smem_load64(mem_s + 8u * (s + i)) : 0ull;
    InBucket ib;
#pragma unroll 4
    for (uint32_t k = 0; k < n; ++k) ib.add<TIES>(smem_load64(mem_s + 8u * (s + k)), mine);
    if (i < n) by_col[static_cast<uint32_t>(mine)] = ib.result<TIES>(s);
  }
  __syncthreads();
}

// Sorted position of every cell, in place of its W (of no use for the cells
// with W = 0).  TIES: its tie word instead, less | t << 14 | q << 23 (q = 0 for
// the cells with W = 0): less = sorted position of its first equal key, t equal
// keys at smaller columns (position less + t), q equal keys in all.
// The first four slots of four cells at a time are compared in straight line,
// so that their loads overlap: slots past a bucket's end hold larger words,
// and lanes with nothing (more) to compare share the pad's all-ones words,
// which costs no bank conflict.  by_col: rank_heavy's results.
template <int NT, int V, bool TIES>
FCB_DEV void spread_positions(const SpreadLayout<NT, V>& L, uint8_t* sm, int m, bool heavy, const uint32_t (&key)[4 * V],
                              uint32_t (&W)[4 * V]) {
  const uint32_t* by_col = reinterpret_cast<const uint32_t*>(sm + L.cnt);
  const uint32_t mem_s = smem_u32(sm + L.mem), pad_s = mem_s + 8u * static_cast<uint32_t>(m);
  if (heavy) rank_heavy<NT, V, TIES>(L, sm);  // uniform
#pragma unroll
  for (int j = 0; j < V; ++j) {
    uint32_t r[4], most = 0u;
    InBucket ib[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      const uint32_t n = W[c] >> 14, s = W[c] & 0x3FFFu, a = mem_s + 8u * s;
      const uint32_t a01 = n > 1u ? a : pad_s;  // a bucket of one is the cell itself
      const uint32_t a23 = n > 2u ? a + 16u : pad_s;
      const unsigned long long mine = (static_cast<unsigned long long>(key[c]) << 32) | cell_col<NT>(c);
      ib[k].add<TIES>(smem_load64(a01), mine);
      ib[k].add<TIES>(smem_load64(a01 + 8u), mine);
      ib[k].add<TIES>(smem_load64(a23), mine);
      ib[k].add<TIES>(smem_load64(a23 + 8u), mine);
      r[k] = ib[k].result<TIES>(s);
      if (TIES && n <= 1u) r[k] = s | (n << 23);  // the pad does not hold the cell itself
      most = max(most, W[c]);
    }
    if (most >= (5u << 14)) {  // some bucket of more than four
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = 4 * j + k;
        const uint32_t n = W[c] >> 14, s = W[c] & 0x3FFFu;
        if (n > kSpreadHeavy) {
          r[k] = by_col[cell_col<NT>(c)];
        } else if (n > 4u) {
          const unsigned long long mine = (static_cast<unsigned long long>(key[c]) << 32) | cell_col<NT>(c);
          for (uint32_t i = 4u; i < n; ++i) ib[k].add<TIES>(smem_load64(mem_s + 8u * (s + i)), mine);
          r[k] = ib[k].result<TIES>(s);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) W[4 * j + k] = r[k];
  }
}

// Bitmap over sorted positions, 16 positions per word: bits 0-15 the marks,
// bits 16-31 (after mark_prefix) the marks before the word.
FCB_DEV void mark_set(uint32_t* bits, uint32_t p) { atomicOr(&bits[p >> 4], 1u << (p & 15u)); }
FCB_DEV void mark_prefix(uint32_t* bits, int nwords) {  // one warp
  uint32_t carry = 0;
  for (int base = 0; base < nwords; base += 32) {
    const int k = base + static_cast<int>(lane_id());
    const uint32_t v = k < nwords ? bits[k] : 0u;
    const uint32_t c = __popc(v);
    const uint32_t inc = warp_inclusive_sum(c);
    if (k < nwords) bits[k] = v | ((carry + inc - c) << 16);
    carry += __shfl_sync(kFull, inc, 31);
  }
}
FCB_DEV uint32_t marks_before(const uint32_t* bits, uint32_t p) {
  const uint32_t v = bits[p >> 4];
  uint32_t below;
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(below) : "r"(p & 15u));  // the bits below p's
  return (v >> 16) + __popc(v & below);
}

}  // namespace fcb
