// rank_slices.cu -- cs_rank of rows too wide for one CTA's shared memory, by
// slices of their value range, for sm_100a.
//
// A row is ranked by R CTAs that do not wait for one another.  Each reads the
// whole row (from L2 but for the first), takes the cells of its own slice of
// the key range in column order, counts the valid cells below the slice, ranks
// its cells by value-spread buckets (section_rank.cuh) and writes their ranks
// by column.  The slices part at order statistics of 512 evenly spaced cells,
// which every CTA finds for itself: any parting gives the same ranks, it only
// decides how even the slices are.  A slice that holds more cells than a CTA
// takes (a much repeated value, a sample that does not show the row) is worked
// off in parts, cut at the median of the cells that it could hold.
//
// A row with few valid cells takes as many fewer slices.  Where a value repeats in
// the sample so that slices would begin at it in vain, those only write their
// share of the NaNs, and the last of them ranks the value's cells by column in a
// second pass over the row; a slice of one value needs no ranking (its list is in
// column order).
//
// Measured on a B200, against one CTA per row that sorts it in global memory:
// 4 x 16500 151 -> 26 us, 61 x 20000 182 -> 53, 64 x 40000 350 -> 142, 500 x
// 17000 633 -> 260; integers 0..6 64 x 40000 148 -> 116, 98 % of the cells
// invalid 41 -> 48, one value 62 -> 80 (three passes; the sort
// has nothing to do).  What bounds it is instruction issue: ranking the slice,
// and reading the row R times at about 12 instructions per cell and slice;
// cs_rank_by_slices says where the sort is taken instead.
//
// The CTAs of a row read all of it while others write its ranks: out must not
// overlap X.
//
// Semantics: cs_rank_gpu (src/cross_sectional_rank.cu:228-372).
#include <algorithm>

#include "section_rank.cuh"

namespace fcb {
namespace {

constexpr int kSlNT = 512, kSlV = 2, kSlWarps = kSlNT / 32;
constexpr int kSlCap = 4 * kSlNT * kSlV;  // cells a CTA ranks at a time
// Cells of a slice on average.  With s sampled cells a slice, its size varies by
// 1 / sqrt(s), 16 % at 32768 cells; one above the cap costs its CTA two more
// passes over the row.  (61 x 20000: 58 us at 2304, 50 at 2900, or 60 where one
// slice comes out above the cap, one call in ten; 64 x 40000 147 and 133-153;
// 30 x 65000 149 at 2304.)
constexpr int slice_mean(int N) { return N <= 32768 ? 2900 : 2304; }
constexpr int kSlTile = 4 * kSlNT;        // cells per step over the row
constexpr int kSlSample = 16;             // sampled cells per lane

struct SliceSmem {
  size_t sec, col, wt, total;
  __host__ __device__ SliceSmem() {
    const size_t a = SpreadLayout<kSlNT, kSlV>(kSlCap).total, b = SortedLayout<kSlNT>(kSlCap).total;
    sec = 0;
    col = al16(a > b ? a : b);
    wt = col + size_t(kSlCap) * 4;
    total = wt + 512;
  }
};

struct SliceRow {
  const float* x;
  const uint8_t* mask;
  int N;
  bool desc, vec;  // vec: 16-byte loads of cells and 4-byte loads of mask bytes
  FCB_DEV uint32_t key(float v, uint32_t m) const {
    return m != 0u && finite_f32(v) ? key_finite_f32(desc ? -v : v) : kInvalidKey32;
  }
  FCB_DEV uint32_t one(int i) const { return key(__ldg(x + i), mask != nullptr ? __ldg(mask + i) : 1u); }
  // Cells i0 .. i0 + 3 (kInvalidKey32 beyond the row).
  FCB_DEV void four(int i0, uint32_t (&k)[4]) const {
    if (vec && i0 + 3 < N) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(x + i0));
      const uint32_t m = mask != nullptr ? __ldg(reinterpret_cast<const uint32_t*>(mask + i0)) : 0x01010101u;
      k[0] = key(v.x, m & 0xFFu);
      k[1] = key(v.y, m & 0xFF00u);
      k[2] = key(v.z, m & 0xFF0000u);
      k[3] = key(v.w, m & 0xFF000000u);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) k[q] = i0 + q < N ? one(i0 + q) : kInvalidKey32;
    }
  }
};

// The key of 0-based rank `rank` among a warp's samples, `rank` being below
// their number: the largest v with no more than `rank` keys below it.
FCB_DEV uint32_t sample_rank(const uint32_t (&k)[kSlSample], uint32_t rank) {
  uint32_t v = 0u;
  for (uint32_t bit = 0x80000000u; bit != 0u; bit >>= 1) {
    uint32_t c = 0u;
#pragma unroll
    for (int q = 0; q < kSlSample; ++q) c += k[q] < (v | bit) ? 1u : 0u;
    if (__reduce_add_sync(kFull, c) <= rank) v |= bit;
  }
  return v;
}

enum class Take { kFirst, kHeavy, kList, kTies };

// NaN for the invalid cells of every R-th tile from r on.
FCB_DEV void slice_nans(const SliceRow& row, float* out, int r, int R) {
  for (int t0 = r * kSlTile; t0 < row.N; t0 += R * kSlTile) {
    const int i0 = t0 + 4 * static_cast<int>(threadIdx.x);
    uint32_t k[4];
    row.four(i0, k);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (k[q] == kInvalidKey32 && i0 + q < row.N) out[i0 + q] = __uint_as_float(kQuietNanBits);
  }
}

// The cells with a <= key < b in column order: their keys and columns into the
// lists as far as these reach or (kTies) their ranks from first + 1 on into out.
// Returns their number.  kFirst and kHeavy also count the valid cells below a
// into `below` (kHeavy: below a - 1, and those equal to a - 1 into `ties`) and
// write NaN for the invalid cells of every R-th tile from r on.  wt: 112 words
// without [96, 101); ends with a barrier.
template <Take TAKE>
FCB_DEV uint32_t slice_collect(const SliceRow& row, uint32_t a, uint32_t b, uint32_t* keys, uint32_t* cols,
                               uint32_t first, float* out, uint32_t* wt, int r, int R, uint32_t& below,
                               uint32_t& ties) {
  constexpr bool kWhole = TAKE == Take::kFirst || TAKE == Take::kHeavy;
  const int wi = static_cast<int>(threadIdx.x >> 5);
  uint32_t run = 0u, under = 0u, same = 0u;
  int buf = 0, tile = 0;
  uint32_t next[4];
  row.four(4 * static_cast<int>(threadIdx.x), next);
  for (int t0 = 0; t0 < row.N; t0 += kSlTile, buf ^= 32) {
    const int i0 = t0 + 4 * static_cast<int>(threadIdx.x);
    uint32_t k[4], h = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      k[q] = next[q];
      h += k[q] - a < b - a ? 1u : 0u;
      if (kWhole) under += k[q] < a ? 1u : 0u;
      if (TAKE == Take::kHeavy) same += k[q] == a - 1u ? 1u : 0u;
    }
    if (t0 + kSlTile < row.N) row.four(i0 + kSlTile, next);
    if (kWhole) {
      if (tile == r) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (k[q] == kInvalidKey32 && i0 + q < row.N) out[i0 + q] = __uint_as_float(kQuietNanBits);
      }
      tile = tile + 1 == R ? 0 : tile + 1;
    }
    const uint32_t inc = warp_inclusive_sum(h);
    if (lane_id() == 31) wt[buf + wi] = inc;
    __syncthreads();  // (the other half of wt is rewritten after the next one)
    uint32_t p = run + warps_before<kSlWarps>(wt + buf) + inc - h;
    run += warps_sum<kSlWarps>(wt + buf);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (k[q] - a < b - a) {
        if (TAKE == Take::kTies) {
          out[i0 + q] = static_cast<float>(first + p + 1u);
        } else if (p < kSlCap) {
          keys[p] = k[q];
          cols[p] = static_cast<uint32_t>(i0 + q);
        }
        ++p;
      }
  }
  if (kWhole) {
    under = __reduce_add_sync(kFull, under);
    same = __reduce_add_sync(kFull, same);
    if (lane_id() == 0) {
      wt[64 + wi] = under;
      wt[80 + wi] = same;
    }
  }
  __syncthreads();
  if (kWhole) {
    ties = warps_sum<kSlWarps>(wt + 80);
    below = warps_sum<kSlWarps>(wt + 64) - ties;
  }
  return run;
}

// Positions of n keys (key[c] at list index cell_col(c)) by radix sort, in W.
__device__ __noinline__ void slice_radix(const uint32_t* key, int n, uint8_t* sm, uint32_t* W) {
  const SortedLayout<kSlNT> L(kSlCap);
  uint32_t* k0 = reinterpret_cast<uint32_t*>(sm + L.k0);
  uint32_t* k1 = reinterpret_cast<uint32_t*>(sm + L.k1);
  uint16_t* i0 = reinterpret_cast<uint16_t*>(sm + L.i0);
  uint16_t* i1 = reinterpret_cast<uint16_t*>(sm + L.i1);
  for (int c = 0; c < 4 * kSlV; ++c) {
    const int i = static_cast<int>(cell_col<kSlNT>(c));
    if (i < n) {
      k0[i] = key[c];
      i0[i] = static_cast<uint16_t>(i);
    }
  }
  __syncthreads();
  uint32_t* ks;
  uint16_t* is;
  block_radix_sort<kSlNT, 4 * kSlV, uint32_t>(k0, i0, k1, i1, n, sm + L.scratch, &ks, &is);
  uint32_t* pos = ks == k0 ? k1 : k0;
  for (int p = static_cast<int>(threadIdx.x); p < n; p += kSlNT) pos[is[p]] = static_cast<uint32_t>(p);
  __syncthreads();
  for (int c = 0; c < 4 * kSlV; ++c) {
    const int i = static_cast<int>(cell_col<kSlNT>(c));
    W[c] = i < n ? pos[i] : 0u;
  }
  __syncthreads();
}

// One CTA per (date, slice).
__global__ void __launch_bounds__(kSlNT, kSmThreads / kSlNT)
    k_cs_slices(const float* __restrict__ X, const uint8_t* __restrict__ mask, int N, int desc, int R,
                float* __restrict__ out) {
  constexpr int C = 4 * kSlV;
  extern __shared__ __align__(16) uint8_t sm[];
  const SliceSmem S;
  const SpreadLayout<kSlNT, kSlV> L(kSlCap);
  uint32_t* cols = reinterpret_cast<uint32_t*>(sm + S.col);
  uint32_t* keys = reinterpret_cast<uint32_t*>(sm + L.mem);  // read out before the buckets are filled
  uint32_t* wt = reinterpret_cast<uint32_t*>(sm + S.wt);     // [0, 96) counts, [96, 101) the slice's ends, the slices and a cut
  const int t = static_cast<int>(blockIdx.x) / R, r = static_cast<int>(blockIdx.x) % R;
  const int tid = static_cast<int>(threadIdx.x), wi = tid >> 5, lane = tid & 31;
  const size_t at = static_cast<size_t>(t) * N;
  SliceRow row{X + at, mask != nullptr ? mask + at : nullptr, N, desc != 0, false};
  row.vec = (reinterpret_cast<uintptr_t>(row.x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(row.mask) & 3u) == 0;
  out += at;
  if (wi < 3) {  // warp w: the key at which slice r - 1 + w begins
    uint32_t k[kSlSample], ms = 0u;
#pragma unroll
    for (int q = 0; q < kSlSample; ++q) {
      k[q] = row.one(static_cast<int>(static_cast<long long>(q * 32 + lane) * N / (32 * kSlSample)));
      ms += k[q] != kInvalidKey32 ? 1u : 0u;
    }
    ms = __reduce_add_sync(kFull, ms);
    // a row with few valid cells, by its sample and two standard deviations, takes
    // as many fewer slices
    const uint32_t valid = min(512u, ms + 2u * static_cast<uint32_t>(sqrtf(static_cast<float>(ms))) + 2u);
    const int rows_slices = static_cast<int>((static_cast<uint32_t>(R) * valid + 511u) / 512u);
    const int begin = r - 1 + wi;
    uint32_t v = 0u;
    if (begin >= rows_slices)
      v = kInvalidKey32;
    else if (begin > 0)  // (no valid sample: the first slice takes all cells)
      v = sample_rank(k, ms * static_cast<uint32_t>(begin) / static_cast<uint32_t>(rows_slices));
    if (lane == 0) wt[96 + wi] = v;
    if (lane == 0 && wi == 0) wt[99] = static_cast<uint32_t>(rows_slices);
  }
  __syncthreads();
  R = static_cast<int>(wt[99]);
  if (r >= R) return;
  uint32_t a = wt[97], below = 0u;
  const uint32_t end = wt[98];
  uint32_t b = end;
  if (a == b) {  // between two equal sampled cells: the last slice that begins at them has theirs
    slice_nans(row, out, r, R);
    return;
  }
  uint32_t n, ties = 0u;
  if (r > 0 && wt[96] == a) {  // a value that fills a slice or more: by column, apart from the others
    ++a;
    n = slice_collect<Take::kHeavy>(row, a, b, keys, cols, 0u, out, wt, r, R, below, ties);
    below += slice_collect<Take::kTies>(row, a - 1u, a, nullptr, nullptr, below, out, wt, r, R, below, ties);
  } else {
    n = slice_collect<Take::kFirst>(row, a, b, keys, cols, 0u, out, wt, r, R, below, ties);
  }
  for (;;) {  // uniform: the slice, as a rule in one part
    if (n > kSlCap) {
      if (b - a == 1u) {  // one value: ranked by column
        below += slice_collect<Take::kTies>(row, a, b, nullptr, nullptr, below, out, wt, r, R, below, ties);
      } else {
        // up to the median of the full list; a value that fills half of it is
        // thereby taken alone
        if (wi == 0) {
          uint32_t k[kSlSample];
#pragma unroll
          for (int q = 0; q < kSlSample; ++q) k[q] = keys[(q * 32 + lane) * (kSlCap / (32 * kSlSample))];
          const uint32_t v = sample_rank(k, 16 * kSlSample);
          if (lane == 0) wt[100] = max(v, a + 1u);
        }
        __syncthreads();
        b = wt[100];
        n = slice_collect<Take::kList>(row, a, b, keys, cols, 0u, out, wt, r, R, below, ties);
        continue;
      }
    } else {
      uint32_t key[C], W[C];
      const uint32_t key0 = keys[0];
      bool differs = false;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const uint32_t i = cell_col<kSlNT>(c);
        key[c] = i < n ? keys[i] : kInvalidKey32;
        differs = differs || (i < n && key[c] != key0);
      }
      SpreadTotals T;
      if (!__syncthreads_or(differs)) {  // (the keys' place becomes the buckets')
#pragma unroll
        for (int c = 0; c < C; ++c) W[c] = cell_col<kSlNT>(c);  // one value: the list is in column order
      } else if (spread_place<kSlNT, kSlV>(key, L, sm, W, T)) {
        spread_positions<kSlNT, kSlV, false>(L, sm, T.m, T.heavy, key, W);
      } else {
        uint32_t kk[C], w[C];
#pragma unroll
        for (int c = 0; c < C; ++c) kk[c] = key[c];
        slice_radix(kk, static_cast<int>(n), sm, w);
#pragma unroll
        for (int c = 0; c < C; ++c) W[c] = w[c];
      }
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const uint32_t i = cell_col<kSlNT>(c);
        if (i < n) out[cols[i]] = static_cast<float>(below + W[c] + 1u);
      }
      below += n;
      __syncthreads();  // the lists are rewritten
    }
    if (b == end) break;
    a = b;
    b = end;
    n = slice_collect<Take::kList>(row, a, b, keys, cols, 0u, out, wt, r, R, below, ties);
  }
}
}  // namespace

cudaError_t launch_cs_rank_slices(const float* X, const uint8_t* mask, int T, int N, int desc, float* out,
                                  cudaStream_t st) {
  if (N < 1 || N > kSliceMaxN || T < 1) return cudaErrorInvalidValue;
  // two CTAs an SM; with few rows more and smaller slices, so that every SM has some
  const int R = std::max((N + slice_mean(N) - 1) / slice_mean(N), std::min(296 / T, N / 512));
  const size_t smem = SliceSmem().total;
  const long long grid = static_cast<long long>(T) * R;
  if (grid > 2147483647LL) return cudaErrorInvalidValue;
  const cudaError_t e =
      cudaFuncSetAttribute(k_cs_slices, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  k_cs_slices<<<static_cast<unsigned>(grid), kSlNT, smem, st>>>(X, mask, N, desc, R, out);
  return cudaGetLastError();
}

}  // namespace fcb
