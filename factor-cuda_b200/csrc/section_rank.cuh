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

// Largest bucket, and largest mean bucket seen by a cell (sum of squared
// sizes over cells), that the in-bucket counts take.  The largest bucket also
// bounds the 9-bit fields of W and of the tie words.
constexpr uint32_t kSpreadMaxBucket = 500;
constexpr uint32_t kSpreadMeanBucket = 24;
// Equal neighbours (columns 2i, 2i + 1) above which a section goes to its
// radix form before any bucket is counted: twice their number estimates the
// mean number of cells that share a cell's value.
constexpr uint32_t kSpreadMaxEqualPairs = 8;
// A bucket above this size is ranked by warps, 32 of its words at a time
// against all of them, and not by its cells' own threads, whose warps would
// wait for the longest loop.
constexpr uint32_t kSpreadHeavy = 16;
// A section whose bins hold, by the mean over its cells, more than this
// fraction of it is a cluster far narrower than its range.
constexpr uint32_t kSpreadBinShare = 8;

template <int NT, int V>
struct SpreadLayout {
  static constexpr int K = 2 * NT;  // bins: two per thread
  // counters one thread scans: they cover every bucket (a power of two where
  // that wastes little; 32 for V = 4 would spill)
  static constexpr int P = V == 1 ? 8 : V <= 3 ? 16 : 4 * V + 4;
  size_t red, tab, bits, cnt, mem, total;
  int S;  // counter stride: bucket b is counter (b % P) * S + b / P
  __host__ __device__ explicit SpreadLayout(int n) {
    size_t o = 0;
    red = o; o += 1024;
    tab = o; o += size_t(K) * 4;
    bits = o; o = al16(o + size_t(n / 16 + 2) * 4);
    S = ((n + K + P - 1) / P + 3) & ~3;  // at most n + K buckets
    cnt = o; o += size_t(P) * S * 4;
    mem = o; o = al16(o + size_t(n + 4) * 8);  // the four words after the last cell's are the pad
    total = o;
  }
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
  bool heavy;      // some bucket may be above kSpreadHeavy
  uint32_t range;  // largest valid key less the smallest
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

// The scanned buckets above kSpreadHeavy, one item (start | size << 14 | part
// << 23) per 32 words; *items (0 before) counts them.
FCB_DEV void list_heavy(const uint32_t* cnt, int counters, uint32_t* list, uint32_t* items) {
  for (int i = static_cast<int>(threadIdx.x); i < counters; i += static_cast<int>(blockDim.x)) {
    const uint32_t w = cnt[i], n = w >> 14;
    if (n > kSpreadHeavy && n <= kSpreadMaxBucket) {  // n of an empty bucket at 2^14 reads 1
      const uint32_t parts = (n + 31u) / 32u, at = atomicAdd(items, parts);
      for (uint32_t k = 0; k < parts; ++k) list[at + k] = w | (k << 23);
    }
  }
}

// Column of cell c of this thread in the vector layout.
template <int NT>
FCB_DEV uint32_t cell_col(int c) { return 4u * ((c >> 2) * NT + threadIdx.x) + (c & 3); }

// Places the valid cells (key[c] != kInvalidKey32) in bucket slots.  key[c]
// becomes the distance from the smallest valid key, above T.range for the
// invalid cells.  On true, W[c] of a valid cell is its bucket's start | size
// << 14 and its own slot in the bucket << 23, 0 for the others; mem holds the
// (distance << 32 | column) words of the valid cells grouped by bucket, then
// four all-ones words.  On false (crowded buckets) shared memory holds nothing
// of use.  Uniform across
// the block; every thread calls; ends with a barrier.  T.m == 0 returns true
// with nothing placed.
template <int NT, int V>
FCB_DEV bool spread_place(uint32_t (&key)[4 * V], const SpreadLayout<NT, V>& L, uint8_t* sm, uint32_t (&W)[4 * V],
                          SpreadTotals& T) {
  constexpr int C = 4 * V, NW = NT / 32, K = SpreadLayout<NT, V>::K, P = SpreadLayout<NT, V>::P;
  static_assert(4 * NT * V + K <= P * NT, "one scan step covers every bucket");
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  uint32_t* tab = reinterpret_cast<uint32_t*>(sm + L.tab);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(sm + L.cnt);
  const uint32_t tab_s = smem_u32(tab), cnt_s = smem_u32(cnt), mem_s = smem_u32(sm + L.mem);
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
    __syncthreads();  // the caller reuses the shared memory
    return false;
  }
  if (kmin == kInvalidKey32) {  // no valid cell
    T.m = 0;
    T.heavy = false;
    T.range = 0u;
#pragma unroll
    for (int c = 0; c < C; ++c) W[c] = 0u;
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
    if (m > 256u && warps_sum<NW>(red + 192) > m * m / kSpreadBinShare) {
      __syncthreads();  // the caller reuses the shared memory
      return false;
    }
    *reinterpret_cast<uint2*>(tab + 2 * tid) = make_uint2(ex | (w0 << 16), (ex + w0) | (w1 << 16));
  }
  __syncthreads();
  // ---- bucket of every cell, counted; the returned count is the cell's slot
  // in the bucket, so twice their sum is the sum of squared sizes less m
  uint32_t sum = 0u, any = 0u;
#pragma unroll
  for (int j = 0; j < V; ++j) {  // four cells' loads in flight at a time
    uint32_t bw[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      bw[k] = smem_load_if(key[4 * j + k] <= range, tab_s + 4u * __umulhi(key[4 * j + k], scale));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      const uint32_t b = (bw[k] & 0xFFFFu) + __umulhi(key[c] * scale, bw[k] >> 16);
      const uint32_t q = (b % P) * L.S + b / P;
      const uint32_t s = smem_fetch_inc_if(key[c] <= range, cnt_s + 4u * q);
      sum += s;
      any |= s;
      W[c] = q | (s << 16);
    }
  }
  sum = __reduce_add_sync(kFull, sum);
  if (lane_id() == 0) red[160 + wi] = sum;
  T.heavy = __syncthreads_or(any >= kSpreadHeavy);  // a slot above 15
  sum = 2u * warps_sum<NW>(red + 160) + static_cast<uint32_t>(T.m);
  if (sum > kSpreadMaxBucket * kSpreadMaxBucket || sum > kSpreadMeanBucket * static_cast<uint32_t>(T.m)) {
    __syncthreads();  // the caller reuses the shared memory
    return false;
  }
  bucket_scan<NW, P>(cnt, L.S, red);
  if (tid < 4) reinterpret_cast<unsigned long long*>(sm + L.mem)[T.m + tid] = ~0ull;
  __syncthreads();
  // ---- scatter
#pragma unroll
  for (int j = 0; j < V; ++j) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = smem_load_if(key[4 * j + k] <= range, cnt_s + 4u * (W[4 * j + k] & 0xFFFFu));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      smem_store2_if(key[c] <= range, mem_s + 8u * ((w[k] & 0x3FFFu) + (W[c] >> 16)), cell_col<NT>(c), key[c]);
      W[c] = w[k] + ((W[c] >> 16) << 23);
    }
  }
  __syncthreads();
  return true;
}

FCB_DEV unsigned long long smem_load64(uint32_t addr) {
  unsigned long long v;
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
  return v;
}

// Tie words of the buckets above kSpreadHeavy, one per slot, over the bucket
// counters: less | t << 14 | q << 23 (see spread_ties).  The buckets are listed
// where the bins were; each warp takes 32 words of one against all of its
// words (broadcast reads).  Call when T.heavy (uniform); ends with a barrier.
template <int NT, int V>
FCB_DEV void spread_heavy(const SpreadLayout<NT, V>& L, uint8_t* sm) {
  constexpr int P = SpreadLayout<NT, V>::P;
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  uint32_t* list = reinterpret_cast<uint32_t*>(sm + L.tab);
  uint32_t* tie = reinterpret_cast<uint32_t*>(sm + L.cnt);
  const uint32_t mem_s = smem_u32(sm + L.mem);
  list_heavy(tie, P * L.S, list, &red[224]);
  __syncthreads();
  const int items = static_cast<int>(red[224]);
  for (int it = static_cast<int>(threadIdx.x >> 5); it < items; it += NT / 32) {
    const uint32_t w = list[it], s = w & 0x3FFFu, n = (w >> 14) & 0x1FFu, i = (w >> 23) * 32u + lane_id();
    const unsigned long long mine = i < n ? smem_load64(mem_s + 8u * (s + i)) : 0ull;
    const uint32_t key = static_cast<uint32_t>(mine >> 32);
    uint32_t less = 0u, le = 0u, before = 0u;
#pragma unroll 4
    for (uint32_t k = 0; k < n; ++k) {
      const unsigned long long o = smem_load64(mem_s + 8u * (s + k));
      const uint32_t ok = static_cast<uint32_t>(o >> 32);
      less += ok < key ? 1u : 0u;
      le += ok <= key ? 1u : 0u;
      before += o < mine ? 1u : 0u;
    }
    if (i < n) tie[s + i] = (s + less) | ((before - less) << 14) | ((le - less) << 23);
  }
  __syncthreads();
}

// Sorted position of every cell, in place of its W: its bucket's start plus
// the smaller words in its bucket (0 for the cells with W = 0, which read
// nothing of use).  The first four slots of four cells at a time are compared
// in straight line, so that their loads overlap; slots past a bucket's end
// hold larger words, and lanes with nothing (more) to compare share the pad's
// all-ones words, which costs no bank conflict.  tie: spread_heavy's words.
template <int NT, int V>
FCB_DEV void spread_positions(uint32_t mem_s, uint32_t pad_s, const uint32_t* tie, const uint32_t (&key)[4 * V],
                              uint32_t (&W)[4 * V]) {
#pragma unroll
  for (int j = 0; j < V; ++j) {
    uint32_t r[4], most = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      const uint32_t n = (W[c] >> 14) & 0x1FFu, s = W[c] & 0x3FFFu, a = mem_s + 8u * s;
      const uint32_t a01 = n > 1u ? a : pad_s;  // a bucket of one is the cell itself
      const uint32_t a23 = n > 2u ? a + 16u : pad_s;
      const unsigned long long mine = (static_cast<unsigned long long>(key[c]) << 32) | cell_col<NT>(c);
      const unsigned long long o0 = smem_load64(a01), o1 = smem_load64(a01 + 8u);
      const unsigned long long o2 = smem_load64(a23), o3 = smem_load64(a23 + 8u);
      r[k] = s + (o0 < mine ? 1u : 0u) + (o1 < mine ? 1u : 0u) + (o2 < mine ? 1u : 0u) + (o3 < mine ? 1u : 0u);
      most = max(most, n);
    }
    if (most > 4u) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = 4 * j + k;
        const uint32_t n = (W[c] >> 14) & 0x1FFu, s = W[c] & 0x3FFFu;
        if (n > kSpreadHeavy) {
          const uint32_t v = tie[s + (W[c] >> 23)];
          r[k] = (v & 0x3FFFu) + ((v >> 14) & 0x1FFu);
        } else {
          const unsigned long long mine = (static_cast<unsigned long long>(key[c]) << 32) | cell_col<NT>(c);
          for (uint32_t i = 4u; i < n; ++i) r[k] += smem_load64(mem_s + 8u * (s + i)) < mine ? 1u : 0u;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) W[4 * j + k] = r[k];
  }
}

// One cell with its ties, less | t << 14 | q << 23 (0 for a cell with W = 0):
// less = sorted position of its first equal key, t equal keys at smaller
// columns (position less + t), q equal keys in all, itself included.
FCB_DEV uint32_t spread_ties(uint32_t mem_s, const uint32_t* tie, uint32_t w, uint32_t key, uint32_t i) {
  const uint32_t s = w & 0x3FFFu, n = (w >> 14) & 0x1FFu;
  if (n > kSpreadHeavy) return tie[s + (w >> 23)];
  uint32_t v = s | (n == 1u ? 1u << 23 : 0u);  // a bucket of one is the cell itself
  if (n > 1u)
    for (uint32_t k = 0; k < n; ++k) {
      const unsigned long long o = smem_load64(mem_s + 8u * (s + k));
      const uint32_t ok = static_cast<uint32_t>(o >> 32);
      v += ok < key ? 1u : 0u;
      if (ok == key) v += (1u << 23) + (static_cast<uint32_t>(o) < i ? 1u << 14 : 0u);
    }
  return v;
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
  return (v >> 16) + __popc(v & ((1u << (p & 15u)) - 1u));
}

}  // namespace fcb
