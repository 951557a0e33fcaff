// rank_ic_pair.cu -- daily Spearman IC of one factor row against one returns
// row, one CTA per (date, factor), for sm_100a.
//
// Both rows are ranked in turn by value-spread buckets (section_rank.cuh).  A
// thread owns the same columns in both, so the returns positions stay in
// registers (two to a word) while the factor is ranked, and nothing but the
// rows, the masks and the results crosses memory.  A cell's joint rank is its
// position less the cells before it that are not joint (bitmaps over positions
// with per-word prefix counts); the IC follows from the exact integer sum of
// rank products.
//
// f64 rows use the same 32-bit keys: the value rounded to f32 keeps the order
// of all but nearly equal values, and those that share a key (one pair in a few
// thousand cells, as a rule) are put in order by their full values, read again.
// Rows that are all near ties, or beyond the f32 range, come out crowded and
// are radix-sorted on 64-bit keys.
//
// Crowded rows are radix-sorted in shared memory (pair_radix).
//
// Measured on a B200, against two radix sorts per date in 512-thread CTAs:
// 1218 x 5000 f32 391 -> 129 us, f64 1108 -> 176, 250 x 500 f64 45 -> 23 (the
// kernel 13.1); integers against returns rounded to 1e-4 252 -> 213, f64 587 ->
// 397.  What bounds it is instruction issue (64 k warp instructions per date of
// 5000 at 54 % of the slots).  Full keys of f64 ties read from global memory by
// every comparison took 1662 us on a plane with 3 % zeros, from shared memory 461
// (the radix form 1098).
//
// Semantics: rolling_ic_gpu (src/rolling_ic.cu:306-540) / np_rolling_ic
// (fc/_cpu_core.py:271-293); ties rank by column, a pair that is constant on
// either side over the joint set has no IC.
#include <algorithm>
#include <type_traits>

#include "section_rank.cuh"

namespace fcb {
namespace {

// One side of the pair: a row of f32 or f64 values.
struct PairRow {
  const void* p;
  bool f64;
  FCB_DEV double at(int i) const {
    return f64 ? __ldg(static_cast<const double*>(p) + i) : static_cast<double>(__ldg(static_cast<const float*>(p) + i));
  }
};

// Keys of the row's valid cells (finite, and a nonzero mask byte); the others
// are kInvalidKey32.  Returns the valid cells' bits.
template <int NT, int V, bool WIDE>
FCB_DEV uint32_t pair_keys(const PairRow row, const uint8_t* __restrict__ mask, int N, uint32_t (&key)[4 * V]) {
  constexpr int C = 4 * V;
  uint32_t valid = 0u, mk[C];
  load_mask4<NT, V>(mask, N, mk);
  if (!WIDE || !row.f64) {
    float x[C];
    load_row_f32<NT, V, true>(static_cast<const float*>(row.p), N, x);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const bool v = finite_f32(x[c]) && mk[c];
      key[c] = v ? key_finite_f32(x[c]) : kInvalidKey32;
      valid |= v ? 1u << c : 0u;
    }
  } else {
    const double* p = static_cast<const double*>(row.p);
    const bool al = (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int i0 = 4 * (j * NT + static_cast<int>(threadIdx.x));
      double x[4];
      if (al && i0 + 3 < N) {
        const double2 a = __ldcs(reinterpret_cast<const double2*>(p + i0));
        const double2 b = __ldcs(reinterpret_cast<const double2*>(p + i0 + 2));
        x[0] = a.x;
        x[1] = a.y;
        x[2] = b.x;
        x[3] = b.y;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = i0 + k < N ? p[i0 + k] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = 4 * j + k;
        const bool v = finite_f64(x[k]) && mk[c];  // (no mask byte beyond the row)
        key[c] = v ? key_finite_f32(static_cast<float>(x[k])) : kInvalidKey32;
        valid |= v ? 1u << c : 0u;
      }
    }
  }
  return valid;
}

// Sorted positions of the row's valid cells by radix sort of the full keys, in
// W.  Ends with a barrier.
template <int NT, int V, bool WIDE>
__device__ __noinline__ void pair_radix(const PairRow row, int N, uint32_t valid, uint8_t* sm, uint32_t* W) {
  using K = std::conditional_t<WIDE, unsigned long long, uint32_t>;
  constexpr int C = 4 * V;
  const SortedLayout<NT, sizeof(K)> L(N);
  K* k0 = reinterpret_cast<K*>(sm + L.k0);
  K* k1 = reinterpret_cast<K*>(sm + L.k1);
  uint16_t* i0 = reinterpret_cast<uint16_t*>(sm + L.i0);
  uint16_t* i1 = reinterpret_cast<uint16_t*>(sm + L.i1);
  int base[V];
  const int m = compact_bases<NT, V>(valid, base, reinterpret_cast<unsigned long long*>(sm + L.red));
#pragma unroll
  for (int j = 0; j < V; ++j) {
    int p = base[j];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      if ((valid >> c) & 1u) {
        const int i = static_cast<int>(cell_col<NT>(c));
        if constexpr (WIDE)
          k0[p] = KeyOf<double>::key(row.at(i));
        else
          k0[p] = KeyOf<float>::key(__ldg(static_cast<const float*>(row.p) + i));
        i0[p] = static_cast<uint16_t>(i);
        ++p;
      }
    }
  }
  __syncthreads();
  K* ks;
  uint16_t* is;
  block_radix_sort<NT, C, K>(k0, i0, k1, i1, m, sm + L.scratch, &ks, &is);
  uint16_t* pos = reinterpret_cast<uint16_t*>(ks == k0 ? k1 : k0);
  for (int p = static_cast<int>(threadIdx.x); p < m; p += NT) pos[is[p]] = static_cast<uint16_t>(p);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < C; ++c) W[c] = (valid >> c) & 1u ? pos[cell_col<NT>(c)] : 0u;
  __syncthreads();
}

// Sorted positions of the row's valid cells in W (key: pair_keys; changed).
// Returns a number of cells that no value's ties exceed.  Ends with a barrier.
template <int NT, int V, bool WIDE>
FCB_DEV uint32_t pair_positions(const PairRow row, int N, uint32_t (&key)[4 * V], uint32_t valid, uint8_t* sm,
                                uint32_t (&W)[4 * V]) {
  constexpr int C = 4 * V;
  const SpreadLayout<NT, V> L(N);
  SpreadTotals T;
  if (!spread_place<NT, V>(key, L, sm, W, T)) {
    uint32_t w[C];
    pair_radix<NT, V, WIDE>(row, N, valid, sm, w);
#pragma unroll
    for (int c = 0; c < C; ++c) W[c] = w[c];
    return 0xFFFFFFFFu;
  }
  spread_positions<NT, V, WIDE>(L, sm, T.m, T.heavy, key, W);
  if constexpr (!WIDE) {
    __syncthreads();
  } else {
    // W: smaller keys | equal keys at smaller columns << 14 | equal keys << 23
    bool tied = false;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (!((valid >> c) & 1u)) W[c] = 0u;
      tied = tied || W[c] >= (2u << 23);
    }
    if (__syncthreads_or(tied)) {
      // the full keys of the cells that share a key, at their sorted positions:
      // groups in column order, over the words of the buckets
      unsigned long long* full = reinterpret_cast<unsigned long long*>(sm + L.mem);
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (W[c] >= (2u << 23))
          full[(W[c] & 0x3FFFu) + ((W[c] >> 14) & 0x1FFu)] =
              KeyOf<double>::key(row.at(static_cast<int>(cell_col<NT>(c))));
      __syncthreads();
#pragma unroll 1
      for (int c = 0; c < C; ++c) {
        uint32_t w = 0u;
#pragma unroll
        for (int q = 0; q < C; ++q) w = q == c ? W[q] : w;
        if (w < (2u << 23)) continue;
        const uint32_t s = w & 0x3FFFu, mine = s + ((w >> 14) & 0x1FFu), e = s + (w >> 23);
        const unsigned long long k = full[mine];
        uint32_t r = s;
#pragma unroll 4
        for (uint32_t p = s; p < e; ++p) {
          const unsigned long long o = full[p];
          r += o < k || (o == k && p < mine) ? 1u : 0u;
        }
#pragma unroll
        for (int q = 0; q < C; ++q) W[q] = q == c ? r : W[q];
      }
      __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < C; ++c) W[c] &= 0x3FFFu;  // (a cell that shares no key has none at smaller columns)
  }
  return T.largest;
}

// Whether the row's cells in `joint` (some) all have the same value.  red: 128
// words.  Ends with a barrier.
template <int NT, int V>
__device__ __noinline__ bool pair_constant(const PairRow row, uint32_t joint, uint32_t* red) {
  unsigned long long lo = ~0ull, hi = 0ull;
  for (uint32_t b = joint; b != 0u; b &= b - 1u) {
    const unsigned long long k = KeyOf<double>::key(row.at(static_cast<int>(cell_col<NT>(__ffs(b) - 1))));
    lo = min(lo, k);
    hi = max(hi, k);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(kFull, lo, o));
    hi = max(hi, __shfl_xor_sync(kFull, hi, o));
  }
  unsigned long long* r = reinterpret_cast<unsigned long long*>(red);
  __syncthreads();
  if (lane_id() == 0) {
    r[threadIdx.x >> 5] = lo;
    r[32 + (threadIdx.x >> 5)] = hi;
  }
  __syncthreads();
  for (int w = 0; w < NT / 32; ++w) {
    lo = min(lo, r[w]);
    hi = max(hi, r[32 + w]);
  }
  __syncthreads();
  return lo == hi;
}

// Four consecutive f64 values of a row from column i0 on.
FCB_DEV void store_quad_f64(double* __restrict__ row, int N, int i0, const double (&v)[4]) {
  if ((reinterpret_cast<uintptr_t>(row) & 15u) == 0 && i0 + 3 < N) {
    __stcs(reinterpret_cast<double2*>(row + i0), make_double2(v[0], v[1]));
    __stcs(reinterpret_cast<double2*>(row + i0 + 2), make_double2(v[2], v[3]));
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i0 + k < N) row[i0 + k] = v[k];
  }
}

// The arguments without the rows' types.
struct PairArgs {
  const void *X, *R;
  const uint8_t *fmask, *rmask;
  int F, T, N, min_valid, ic_ld;
  bool x64, r64;
  float* ranks_out;
  double *ic_out, *rank_f_out, *rank_r_out;
};

// WIDE: some side is f64.
template <int NT, int V, bool WIDE>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_ic_pair(PairArgs a) {
  constexpr int C = 4 * V, NW = NT / 32;
  extern __shared__ __align__(16) uint8_t sm[];
  const int N = a.N, t = static_cast<int>(blockIdx.x) / a.F, f = static_cast<int>(blockIdx.x) % a.F;
  const int wi = static_cast<int>(threadIdx.x >> 5), nbw = mark_words(N);
  uint32_t* marks = reinterpret_cast<uint32_t*>(sm);  // factor positions without a valid return
  uint32_t* drop = marks + (nbw + 3) / 4 * 4;         // returns positions without a valid factor
  uint8_t* sec = sm + 2 * al16(static_cast<size_t>(nbw) * 4);
  uint32_t* red = reinterpret_cast<uint32_t*>(sec);
  const size_t row = static_cast<size_t>(t) * N, frow = (static_cast<size_t>(f) * a.T + t) * N;
  const PairRow rr{static_cast<const uint8_t*>(a.R) + row * (WIDE && a.r64 ? 8 : 4), WIDE && a.r64};
  const PairRow rf{static_cast<const uint8_t*>(a.X) + frow * (WIDE && a.x64 ? 8 : 4), WIDE && a.x64};
  // the factor's row and mask are on their way to L2 while the returns are ranked
  for (int b = 128 * static_cast<int>(threadIdx.x); b < N * (rf.f64 ? 8 : 4); b += 128 * NT)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint8_t*>(rf.p) + b));
  if (a.fmask != nullptr)
    for (int b = 128 * static_cast<int>(threadIdx.x); b < N; b += 128 * NT)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a.fmask + row + b));
  for (int k = static_cast<int>(threadIdx.x); k < nbw; k += NT) marks[k] = drop[k] = 0u;
  uint32_t key[C], W[C], pr[C / 2];
  const uint32_t rv = pair_keys<NT, V, WIDE>(rr, a.rmask != nullptr ? a.rmask + row : nullptr, N, key);
  const uint32_t rties = pair_positions<NT, V, WIDE>(rr, N, key, rv, sec, W);
#pragma unroll
  for (int c = 0; c < C; c += 2) pr[c / 2] = (W[c] & 0x3FFFu) | ((W[c + 1] & 0x3FFFu) << 16);
  auto ret_pos = [&](int c) { return (pr[c / 2] >> (16 * (c & 1))) & 0xFFFFu; };
  const uint32_t fv = pair_keys<NT, V, WIDE>(rf, a.fmask != nullptr ? a.fmask + row : nullptr, N, key);
  const uint32_t joint = fv & rv, lone = fv & ~rv, dropped = rv & ~fv;
#pragma unroll
  for (int c = 0; c < C; ++c)
    if ((dropped >> c) & 1u) mark_set(drop, ret_pos(c));
  const uint32_t fties = pair_positions<NT, V, WIDE>(rf, N, key, fv, sec, W);
#pragma unroll
  for (int c = 0; c < C; ++c)
    if ((lone >> c) & 1u) mark_set(marks, W[c]);
  const uint32_t nj = __reduce_add_sync(kFull, static_cast<uint32_t>(__popc(joint)));
  if (lane_id() == 0) red[128 + wi] = nj;
  const bool any_drop = __syncthreads_or(dropped != 0u), any_lone = __syncthreads_or(lone != 0u);
  if (wi == 0 && any_lone) mark_prefix(marks, nbw);
  if (wi == 1 && any_drop) mark_prefix(drop, nbw);
  const uint32_t m = warps_sum<NW>(red + 128);
  bool some = m >= 2u && static_cast<int>(m) >= a.min_valid;
  // a side can be constant on the joint set only when that is no larger than its
  // largest group of ties may be; the rows are read again for it, so before any
  // output (which may be written in their place)
  if (some && m <= fties) some = !pair_constant<NT, V>(rf, joint, red);
  if (some && m <= rties) some = !pair_constant<NT, V>(rr, joint, red);
  if (a.ranks_out != nullptr) {
    float v[C];
#pragma unroll
    for (int c = 0; c < C; ++c)
      v[c] = (fv >> c) & 1u ? static_cast<float>(W[c] + 1u) : __uint_as_float(kQuietNanBits);
    store_row_f32v<NT, V>(a.ranks_out + frow, N, v);
  }
  if (any_lone || any_drop) __syncthreads();
  // 32 bits hold a thread's sum: ranks are distinct and at most 4 * V * NT,
  // which is at most 2^14 with 16 cells a thread
  static_assert(C <= 16 && 4 * V * NT <= 16384, "32-bit partial sums");
  uint32_t sum32 = 0u;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    double df[4], dr[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      uint32_t x = 0u, y = 0u;
      if ((joint >> c) & 1u) {
        x = W[c] + 1u;
        y = ret_pos(c) + 1u;
        if (any_lone) x -= marks_before(marks, x - 1u);
        if (any_drop) y -= marks_before(drop, y - 1u);
      }
      sum32 += x * y;
      df[k] = static_cast<double>(x);
      dr[k] = static_cast<double>(y);
    }
    if (a.rank_f_out != nullptr) {
      store_quad_f64(a.rank_f_out + frow, N, static_cast<int>(cell_col<NT>(4 * j)), df);
      store_quad_f64(a.rank_r_out + frow, N, static_cast<int>(cell_col<NT>(4 * j)), dr);
    }
  }
  // a 64-bit sum in two pieces that cannot overflow 32 lanes
  auto warp_sum64 = [](unsigned long long v) {
    const uint32_t lo = __reduce_add_sync(kFull, static_cast<uint32_t>(v) & 0x3FFFFFFu);
    const uint32_t hi = __reduce_add_sync(kFull, static_cast<uint32_t>(v >> 26));
    return (static_cast<unsigned long long>(hi) << 26) + lo;
  };
  unsigned long long* red64 = reinterpret_cast<unsigned long long*>(red);
  const unsigned long long wsum = warp_sum64(sum32);
  if (lane_id() == 0) red64[wi] = wsum;
  __syncthreads();
  const unsigned long long sum = warp_sum64(lane_id() < NW ? red64[lane_id()] : 0ull);
  if (threadIdx.x == 0)
    a.ic_out[static_cast<size_t>(f) * (a.ic_ld > 0 ? a.ic_ld : a.T) + t] =
        some ? spearman_from_sum(static_cast<long long>(m), static_cast<long long>(sum))
             : __longlong_as_double(0x7ff8000000000000ll);
}

template <int NT, int V, bool WIDE>
size_t pair_smem(int N) {
  return 2 * al16(static_cast<size_t>(mark_words(N)) * 4) +
         std::max(SpreadLayout<NT, V>(N).total, SortedLayout<NT, WIDE ? 8 : 4>(N).total);
}

template <int NT, int V, bool WIDE>
cudaError_t pair_launch(const PairArgs& a, cudaStream_t st) {
  const size_t smem = pair_smem<NT, V, WIDE>(a.N);
  const long long grid = static_cast<long long>(a.T) * a.F;
  if (smem > kMaxSmemPerBlock || a.N > 4 * NT * V || grid > 2147483647LL) return cudaErrorInvalidValue;
  auto* k = k_ic_pair<NT, V, WIDE>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  k<<<static_cast<unsigned>(grid), NT, smem, st>>>(a);
  return cudaGetLastError();
}

// Wide keys' radix form takes 20 bytes a cell: from 5377 cells on one CTA fills
// an SM, which then should have 1024 threads.
template <bool WIDE>
cudaError_t pair_by_width(const PairArgs& a, cudaStream_t st) {
  auto go = [&](auto shape) {
    return pair_launch<decltype(shape)::kThreads, decltype(shape)::kVectors, WIDE>(a, st);
  };
  const bool few = static_cast<long long>(a.T) * a.F <= kFewSections || (WIDE && a.N > 5376);
  return few ? section_shape_few(a.N, go) : section_shape(a.N, go);
}
}  // namespace

template <typename TF, typename TR>
bool rank_ic_fits(int N) {
  constexpr bool kWide = sizeof(TF) == 8 || sizeof(TR) == 8;
  return N >= 1 && N <= kSmemRankCap && pair_smem<1024, 4, kWide>(N) <= kMaxSmemPerBlock;
}

template <typename TF, typename TR>
cudaError_t launch_rank_ic(const RankIcArgs<TF, TR>& a, cudaStream_t st) {
  if (a.N < 1 || a.N > kSmemRankCap) return cudaErrorInvalidValue;
  constexpr bool kX64 = sizeof(TF) == 8, kR64 = sizeof(TR) == 8;
  const PairArgs p{a.X,   a.R,  a.fmask, a.rmask,     a.F,      a.T,          a.N,         a.min_valid,
                   a.ic_ld, kX64, kR64,    a.ranks_out, a.ic_out, a.rank_f_out, a.rank_r_out};
  return pair_by_width<kX64 || kR64>(p, st);
}

template bool rank_ic_fits<float, float>(int);
template bool rank_ic_fits<float, double>(int);
template bool rank_ic_fits<double, float>(int);
template bool rank_ic_fits<double, double>(int);
template cudaError_t launch_rank_ic<float, float>(const RankIcArgs<float, float>&, cudaStream_t);
template cudaError_t launch_rank_ic<float, double>(const RankIcArgs<float, double>&, cudaStream_t);
template cudaError_t launch_rank_ic<double, float>(const RankIcArgs<double, float>&, cudaStream_t);
template cudaError_t launch_rank_ic<double, double>(const RankIcArgs<double, double>&, cudaStream_t);

}  // namespace fcb
