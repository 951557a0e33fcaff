// rank_ic_bucket.cu -- cs_rank + daily Spearman IC of F factor panels against
// one forward-return panel, one CTA per (date, factor), for sm_100a.
//
//  k_ric_prep     one CTA per date: ranks the date's valid forward returns
//                 once (section_rank.cuh) and writes one 32-bit word per
//                 stock: its position in their ascending order, the position
//                 where its tie group starts, and the returns-valid and
//                 factor-mask bits.  The rows stay in L2 while the F factor
//                 CTAs of the date read them.
//  k_ric_plain    ranks the factor's valid cells by value-spread buckets
//                 (section_rank.cuh).
//  k_ric_learned  learned splitters: the factor's tabulated CDF network maps
//                 each valid cell to a bucket; counting, scan, scatter and the
//                 in-bucket ranks are those of section_rank.cuh.  The map is
//                 monotone in the key whenever the table is non-decreasing,
//                 which each CTA checks as it stages the table; a bucket above
//                 the cap, an unusable scale or a rejected table hands the
//                 section to k_ric_plain through a device list.
//
// Sections whose value-spread buckets come out crowded are radix-sorted in
// shared memory instead (ric_prep_radix, ric_radix).
//
// All keep every cell's state in registers (each thread owns four consecutive
// columns per 128-bit vector, loaded and stored with coalesced vector
// accesses) and share one epilogue: the joint-set rank of a cell is its
// position minus the number of cells before it that are not joint, on the
// factor side and on the returns side (bitmaps over positions with per-word
// prefix counts), and the IC follows from the exact integer sum of rank
// products (see spearman_from_sum).
//
// Measured on a B200: 1218 x 5000 x 12 radix-sorted 2.06 ms, learned 1.28 ms
// (both with a radix-sorted returns pass); now k_ric_prep 0.068 (from 0.188),
// k_ric_plain 0.84 and k_ric_learned 1.12 ms; 250 x 8000 x 16 1.33 -> 0.43 ms.
// What bounds k_ric_plain is instruction issue and barrier latency: 35 k warp
// instructions per 5000-cell section (51 k before) at 55 % of the issue slots
// of two 448-thread CTAs per SM; HBM stands at 11 %.  Learned buckets are a
// little less even (2.2-2.5 cells per cell against 1.9), and their map costs
// about 30 instructions per cell against 25 with the histogram's.
//
// Semantics: cs_rank_gpu (src/cross_sectional_rank.cu:228-372) for the ranks,
// rolling_ic_gpu (src/rolling_ic.cu:306-540) / np_rolling_ic
// (fc/_cpu_core.py:271-293) for the IC; the reference sorts with CUB's global
// segmented radix sort instead.
#include "learned_sort.cuh"
#include "section_rank.cuh"

namespace fcb {
namespace {

constexpr uint32_t kPosBits = 0x3FFFu;      // prepared word: bits 0-13 returns position
constexpr int kGidShift = 14;               //                bits 14-27 tie-group start
constexpr uint32_t kRetValid = 1u << 28;    //                bit 28 returns valid
constexpr uint32_t kFacMask = 1u << 29;     //                bit 29 factor mask

// Block-uniform flags of a section, in red[225] (lone) and red[226] (drop).
constexpr int kAnyLone = 225, kAnyDrop = 226;

// Row t's cells of factor f as the rank kernels need them: keys of the valid
// cells (finite and mask; kInvalidKey32 for the others), joint (bit c: cell c
// is valid on both sides) and lone (valid, but no valid return).  Clears both
// bitmaps and marks the returns positions with no valid factor in `drop`; the
// marks and the flags are complete after the caller's next barrier.
template <int NT, int V, bool STREAM>
FCB_DEV void ric_cells(const RankIcArgs<float, float>& a, const RicPrep& rp, int t, int f, uint32_t* drop,
                       uint32_t* marks, uint32_t* red, uint32_t (&key)[4 * V], uint32_t& joint, uint32_t& lone) {
  constexpr int C = 4 * V;
  const int N = a.N;
  const uint32_t* words = rp.word + static_cast<size_t>(t) * rp.ld;
  uint32_t dropped = 0u;
  joint = 0u;
  lone = 0u;
  {
    float x[C];
    uint32_t w[C];
    load_row_f32<NT, V, STREAM>(a.X + (static_cast<size_t>(f) * a.T + t) * N, N, x);
    load_words<NT, V>(words, N, w);
    for (int k = static_cast<int>(threadIdx.x); k < mark_words(N); k += NT) {
      drop[k] = 0u;
      marks[k] = 0u;
    }
    if (threadIdx.x == 0) red[kAnyLone] = red[kAnyDrop] = 0u;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const bool v = finite_f32(x[c]) && (w[c] & kFacMask), r = (w[c] & kRetValid) != 0u;
      key[c] = v ? key_finite_f32(x[c]) : kInvalidKey32;
      joint |= v && r ? 1u << c : 0u;
      lone |= v && !r ? 1u << c : 0u;
      dropped |= r && !v ? 1u << c : 0u;
    }
  }
  __syncthreads();
  if (lone != 0u) red[kAnyLone] = 1u;
  if (dropped != 0u) red[kAnyDrop] = 1u;
  for (uint32_t d = dropped; d != 0u; d &= d - 1u)  // few: their words are read again
    mark_set(drop, __ldg(words + cell_col<NT>(__ffs(d) - 1)) & kPosBits);
}

// The shared epilogue, after the cells are placed (so that the marks and flags
// of ric_cells are complete): W[c] is the sorted position of a valid cell
// (key[c] <= range).  Writes the rank row and the IC.  A cell's joint rank
// leaves out the lone cells at smaller positions, its return's joint rank the
// dropped ones.  largest: no value is shared by more than that many valid
// cells, so that the factor can be constant on the joint set only when that
// set is no larger.  red: words [0, 225) idle.
template <int NT, int V>
FCB_DEV void ric_epilogue(const RankIcArgs<float, float>& a, const RicPrep& rp, int t, int f,
                          const uint32_t (&key)[4 * V], uint32_t range, const uint32_t (&W)[4 * V], uint32_t joint,
                          uint32_t lone, uint32_t largest, uint32_t* drop, uint32_t* marks, uint32_t* red) {
  constexpr int C = 4 * V, NW = NT / 32;
  const int N = a.N, wi = static_cast<int>(threadIdx.x >> 5);
  const bool any_lone = red[kAnyLone] != 0u, any_drop = red[kAnyDrop] != 0u;
  if (any_lone) {
#pragma unroll
    for (int c = 0; c < C; ++c)
      if ((lone >> c) & 1u) mark_set(marks, W[c]);
    __syncthreads();
    if (wi == 1) mark_prefix(marks, mark_words(N));
  }
  if (any_drop && wi == 0) mark_prefix(drop, mark_words(N));
  uint32_t w[C];
  load_words<NT, V>(rp.word + static_cast<size_t>(t) * rp.ld, N, w);
  if (a.ranks_out != nullptr) {
    float v[C];
    const float qnan = __uint_as_float(kQuietNanBits);
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = key[c] <= range ? static_cast<float>(W[c] + 1u) : qnan;
    store_row_f32v<NT, V>(a.ranks_out + (static_cast<size_t>(f) * a.T + t) * N, N, v);
  }
  if (any_lone || any_drop) __syncthreads();
  // 32 bits hold a thread's sum: ranks are distinct and at most 4 * V * NT,
  // which is at most 2^14 with 16 cells a thread
  static_assert(C <= 16 && 4 * V * NT <= 16384, "32-bit partial sums");
  uint32_t sum32 = 0u, gand = 0xFFFFFFFFu, gor = 0u;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    if ((joint >> c) & 1u) {
      uint32_t rf = W[c] + 1u, rr = (w[c] & kPosBits) + 1u;
      if (any_lone) rf -= marks_before(marks, W[c]);
      if (any_drop) rr -= marks_before(drop, w[c] & kPosBits);
      sum32 += rf * rr;
      gand &= w[c];
      gor |= w[c];
    }
  }
  // warp results: a 64-bit sum in two pieces that cannot overflow 32 lanes
  unsigned long long* red64 = reinterpret_cast<unsigned long long*>(red);
  auto warp_sum64 = [](unsigned long long v) {
    const uint32_t lo = __reduce_add_sync(kFull, static_cast<uint32_t>(v) & 0x3FFFFFFu);
    const uint32_t hi = __reduce_add_sync(kFull, static_cast<uint32_t>(v >> 26));
    return (static_cast<unsigned long long>(hi) << 26) + lo;
  };
  const unsigned long long wsum = warp_sum64(sum32);
  gand = __reduce_and_sync(kFull, gand);
  gor = __reduce_or_sync(kFull, gor);
  const uint32_t nj = __reduce_add_sync(kFull, static_cast<uint32_t>(__popc(joint)));
  if (lane_id() == 0) {
    red64[wi] = wsum;
    red[64 + wi] = gand;
    red[96 + wi] = gor;
    red[128 + wi] = nj;
  }
  __syncthreads();
  const uint32_t m = warps_sum<NW>(red + 128);
  bool fconst = false;
  if (m <= largest) {  // uniform: compare the joint keys
    uint32_t kmin = 0xFFFFFFFFu, kmax = 0u;
#pragma unroll
    for (int c = 0; c < C; ++c)
      if ((joint >> c) & 1u) {
        kmin = min(kmin, key[c]);
        kmax = max(kmax, key[c]);
      }
    kmin = __reduce_min_sync(kFull, kmin);
    kmax = __reduce_max_sync(kFull, kmax);
    if (lane_id() == 0) {
      red[160 + wi] = kmin;
      red[192 + wi] = kmax;
    }
    __syncthreads();
    fconst = warps_min<NW>(red + 160) == warps_max<NW>(red + 192);
  }
  if (wi == 0) {
    const unsigned long long sum = warp_sum64(lane_id() < NW ? red64[lane_id()] : 0ull);
    gand = __reduce_and_sync(kFull, lane_id() < NW ? red[64 + lane_id()] : 0xFFFFFFFFu);
    gor = __reduce_or_sync(kFull, lane_id() < NW ? red[96 + lane_id()] : 0u);
    const bool rconst = (((gand ^ gor) >> kGidShift) & kPosBits) == 0u;  // one tie group
    if (lane_id() == 0) {
      double ic = __longlong_as_double(0x7ff8000000000000ll);
      if (static_cast<int>(m) >= a.min_valid && m >= 2u && !fconst && !rconst)
        ic = spearman_from_sum(static_cast<long long>(m), static_cast<long long>(sum));
      a.ic_out[static_cast<size_t>(f) * (a.ic_ld > 0 ? a.ic_ld : a.T) + t] = ic;
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// per-date returns preparation
// ---------------------------------------------------------------------------
// Date t of returns R (T,N) and masks: the prepared words of row t into out,
// by radix sort.
template <int NT, int V>
__device__ __noinline__ void ric_prep_radix(const float* __restrict__ R, const uint8_t* __restrict__ rmask,
                                            const uint8_t* __restrict__ fmask, int N, int t,
                                            uint32_t* __restrict__ out, uint8_t* sm) {
  constexpr int C = 4 * V;
  const SortedLayout<NT> L(N);
  unsigned long long* scan64 = reinterpret_cast<unsigned long long*>(sm + L.red);
  const size_t row = static_cast<size_t>(t) * N;
  float r[C];
  load_row_f32<NT, V, true>(R + row, N, r);
  uint32_t fmb = 0u, rvb = 0u;  // per-cell bits: factor mask, returns valid
  {
    uint32_t rmk[C], fmk[C];
    load_mask4<NT, V>(rmask != nullptr ? rmask + row : nullptr, N, rmk);
    load_mask4<NT, V>(fmask != nullptr ? fmask + row : nullptr, N, fmk);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      rvb |= ((finite_f32(r[c]) && rmk[c]) ? 1u : 0u) << c;
      fmb |= (fmk[c] ? 1u : 0u) << c;
    }
  }
  int base[V];
  const int mr = compact_bases<NT, V>(rvb, base, scan64);
  uint32_t* k0 = reinterpret_cast<uint32_t*>(sm + L.k0);
  uint32_t* k1 = reinterpret_cast<uint32_t*>(sm + L.k1);
  uint16_t* i0 = reinterpret_cast<uint16_t*>(sm + L.i0);
  uint16_t* i1 = reinterpret_cast<uint16_t*>(sm + L.i1);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    int p = base[j];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      if ((rvb >> c) & 1u) {
        k0[p] = key_f32(r[c]);
        i0[p] = static_cast<uint16_t>(4 * (j * NT + static_cast<int>(threadIdx.x)) + k);
        ++p;
      }
    }
  }
  __syncthreads();
  uint32_t* ks;
  uint16_t* is;
  block_radix_sort<NT, C, uint32_t>(k0, i0, k1, i1, mr, sm + L.scratch, &ks, &is);
  // words of the valid returns, by column: position | tie-group start
  uint32_t* W = (ks == k0) ? k1 : k0;
  const int per = (mr + NT - 1) / NT;
  const int b0 = static_cast<int>(threadIdx.x) * per, b1 = min(mr, b0 + per);
  int last = -1;
  for (int p = b0; p < b1; ++p)
    if (p == 0 || ks[p] != ks[p - 1]) last = p;
  // exclusive max-scan of the chunk's last group start (identity -1)
  int inc = last;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(kFull, inc, o);
    if (lane_id() >= static_cast<unsigned>(o)) inc = max(inc, u);
  }
  int* sc = reinterpret_cast<int*>(scan64);
  const int wi = static_cast<int>(threadIdx.x >> 5);
  if (lane_id() == 31) sc[wi] = inc;
  __syncthreads();
  int carry = -1;
  for (int i = 0; i < wi; ++i) carry = max(carry, sc[i]);
  const int up = __shfl_up_sync(kFull, inc, 1);
  if (lane_id() > 0) carry = max(carry, up);
  for (int p = b0; p < b1; ++p) {
    if (p == 0 || ks[p] != ks[p - 1]) carry = p;
    W[is[p]] = static_cast<uint32_t>(p) | (static_cast<uint32_t>(carry) << kGidShift) | kRetValid;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i0c = 4 * (j * NT + static_cast<int>(threadIdx.x));
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      v[k] = (((rvb >> c) & 1u) ? W[i0c + k] : 0u) | (((fmb >> c) & 1u) ? kFacMask : 0u);
    }
    if (i0c + 3 < N) {
      *reinterpret_cast<uint4*>(out + i0c) = make_uint4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i0c + k < N) out[i0c + k] = v[k];
    }
  }
}

// The same by value-spread buckets.
template <int NT, int V>
FCB_DEV void ric_prep_body(const float* __restrict__ R, const uint8_t* __restrict__ rmask,
                           const uint8_t* __restrict__ fmask, int N, int t, uint32_t* __restrict__ out, uint8_t* sm) {
  constexpr int C = 4 * V;
  const SpreadLayout<NT, V> L(N);
  const size_t row = static_cast<size_t>(t) * N;
  uint32_t key[C], W[C], fmb = 0u;
  {
    float r[C];
    uint32_t mk[C];
    load_row_f32<NT, V, true>(R + row, N, r);
    load_mask4<NT, V>(rmask != nullptr ? rmask + row : nullptr, N, mk);
#pragma unroll
    for (int c = 0; c < C; ++c) key[c] = finite_f32(r[c]) && mk[c] ? key_finite_f32(r[c]) : kInvalidKey32;
    load_mask4<NT, V>(fmask != nullptr ? fmask + row : nullptr, N, mk);
#pragma unroll
    for (int c = 0; c < C; ++c) fmb |= (mk[c] ? 1u : 0u) << c;
  }
  SpreadTotals T;
  if (!spread_place<NT, V>(key, L, sm, W, T)) {
    ric_prep_radix<NT, V>(R, rmask, fmask, N, t, out, sm);
    return;
  }
  spread_positions<NT, V, true>(L, sm, T.m, T.heavy, key, W);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i0 = 4 * (j * NT + static_cast<int>(threadIdx.x));
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      const uint32_t less = W[c] & kPosBits, pos = less + ((W[c] >> 14) & 0x1FFu);
      v[k] = (W[c] >> 23 ? pos | (less << kGidShift) | kRetValid : 0u) | ((fmb >> c) & 1u ? kFacMask : 0u);
    }
    if (i0 + 3 < N) {
      *reinterpret_cast<uint4*>(out + i0) = make_uint4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i0 + k < N) out[i0 + k] = v[k];
    }
  }
}

template <int NT, int V>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_ric_prep(const float* __restrict__ R,
                                                                  const uint8_t* __restrict__ rmask,
                                                                  const uint8_t* __restrict__ fmask, int N, RicPrep rp) {
  extern __shared__ __align__(16) uint8_t sm[];
  if (blockIdx.x == 0 && threadIdx.x == 0) *rp.fb_count = 0;
  ric_prep_body<NT, V>(R, rmask, fmask, N, blockIdx.x, rp.word + static_cast<size_t>(blockIdx.x) * rp.ld, sm);
}

// ---------------------------------------------------------------------------
// learned splitters
// ---------------------------------------------------------------------------
// Section (t, f); item_id is what a fallback queues on fb.
template <int NT, int V>
FCB_DEV void ric_learned_body(const RankIcArgs<float, float>& a, const RicPrep& rp, const int t, const int f,
                              const int item_id, RicList fb, uint8_t* sm) {
  constexpr int C = 4 * V, NW = NT / 32;
  const int N = a.N;
  const SpreadLayout<NT, V> L(N);
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  uint32_t* tab = reinterpret_cast<uint32_t*>(sm + L.knots);
  uint32_t* drop = reinterpret_cast<uint32_t*>(sm + L.bits);
  uint32_t* marks = reinterpret_cast<uint32_t*>(sm + L.bits2);
  const int tid = static_cast<int>(threadIdx.x), wi = tid >> 5, lane = tid & 31;
  const size_t frow = (static_cast<size_t>(f) * a.T + t) * N;
  int* stats = a.learn_stats != nullptr ? a.learn_stats + (static_cast<size_t>(f) * a.T + t) * 4 : nullptr;

  // warp 0 issues the loads of the location / scale sample (used below) with
  // the row's, so that both wait out one memory latency, not two
  float xs[8];
  uint32_t vs = 0u;
  if (wi == 0) {
    const int S = min(N, 256);  // i = s*N/S: s*N/256 when N >= 256, else s
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int s = q * 32 + lane;
      xs[q] = 0.0f;
      if (s < S) {
        const int i = N >= 256 ? (s * N) >> 8 : s;
        const float v = a.X[frow + i];
        if (finite_f32(v) && (rp.word[static_cast<size_t>(t) * rp.ld + i] & kFacMask)) {
          xs[q] = v;
          vs |= 1u << q;
        }
      }
    }
  }
  // the table's knots, four per thread, checked to be non-decreasing within
  // [0, 1] (a NaN fails every comparison)
  constexpr int KT = (kCdfKnots / 4 + NT - 1) / NT;
  float kn[KT][5];
  int tab_bad = 0;
  {
    const float* tg = a.cdf_table + static_cast<size_t>(f) * kCdfKnots;
#pragma unroll
    for (int q = 0; q < KT; ++q) {
      const int k = tid + q * NT;
      if (k < kCdfKnots / 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(tg) + k);
        kn[q][0] = v.x;
        kn[q][1] = v.y;
        kn[q][2] = v.z;
        kn[q][3] = v.w;
        kn[q][4] = 4 * k + 4 < kCdfKnots ? __ldg(tg + 4 * k + 4) : 1.0f;
        tab_bad |= (0.0f <= v.x && v.x <= v.y && v.y <= v.z && v.z <= v.w && v.w <= kn[q][4] && kn[q][4] <= 1.0f) ? 0 : 1;
      }
    }
  }
  for (int k = tid; k < SpreadLayout<NT, V>::P / 4 * L.S; k += NT)
    reinterpret_cast<uint4*>(sm + L.cnt)[k] = make_uint4(0u, 0u, 0u, 0u);
  uint32_t key[C], W[C], joint, lone;
  ric_cells<NT, V, true>(a, rp, t, f, drop, marks, red, key, joint, lone);
  // ---- warp 0: location / scale from an evenly spaced sample of the row
  // (mean and mean absolute deviation of up to 256 valid cells; they only
  // shape the bucket map -- the order is exact whatever they are)
  if (wi == 0) {
    int ns = 0;
    float s1 = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if ((vs >> q) & 1u) {
        s1 += xs[q];
        ++ns;
      }
    const float n_s = static_cast<float>(warp_sum(ns));
    const float mean = warp_sum(s1) / n_s;
    float s2 = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if ((vs >> q) & 1u) s2 += fabsf(xs[q] - mean);
    const float mad = warp_sum(s2) / n_s;
    if (lane == 0) {
      red[96] = __float_as_uint(mean);
      red[97] = __float_as_uint(mad);
    }
  } else if (tid == 32) {
    const float lo = a.cdf_zrange[2 * f], hi = a.cdf_zrange[2 * f + 1];
    red[98] = __float_as_uint(lo);
    red[99] = __float_as_uint(static_cast<float>((kCdfKnots - 1) / static_cast<double>(hi - lo)));
    red[224] = 0u;
  }
  uint32_t nval = 0u;
#pragma unroll
  for (int c = 0; c < C; ++c) nval += key[c] != kInvalidKey32 ? 1u : 0u;
  nval = __reduce_add_sync(kFull, nval);
  if (lane == 0) red[wi] = nval;
  tab_bad = __syncthreads_or(tab_bad);
  const int m = static_cast<int>(warps_sum<NW>(red));
  const float loc = __uint_as_float(red[96]), mad = __uint_as_float(red[97]);
  const float inv_scale = mad > 0.0f ? 1.0f / mad : 0.0f;
  const float lo = __uint_as_float(red[98]), inv_dz = __uint_as_float(red[99]);
  const int B = m > 0 ? m : 1;
  const bool scale_ok = (mad > 0.0f) && isfinite(loc) && isfinite(inv_scale) && (inv_scale > 0.0f) &&
                        isfinite(inv_dz) && (inv_dz > 0.0f);
  if (tab_bad || (m >= 2 && !scale_ok)) {  // uniform across the block
    if (m >= 2) {
      if (tid == 0) {
        if (stats != nullptr) {
          stats[0] = tab_bad ? kLearnJudge : kLearnScale;
          stats[1] = 0;
          stats[2] = 0;
          stats[3] = m;
        }
        fb.items[atomicAdd(fb.count, 1)] = item_id;
      }
      return;
    }
  }
  // ---- the table as bucket ranges of this section: a knot's first bucket and
  // the buckets up to the next knot's, within [0, B) whatever the table holds
  {
    const float Bf = static_cast<float>(B);
    auto bucket = [&](float u) { return max(0, min(B - 1, static_cast<int>(Bf * u))); };
#pragma unroll
    for (int q = 0; q < KT; ++q) {
      const int k = tid + q * NT;
      if (k < kCdfKnots / 4) {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int b0 = bucket(kn[q][i]), b1 = bucket(kn[q][i + 1]);
          v[i] = static_cast<uint32_t>(b0) | (static_cast<uint32_t>(max(0, b1 - b0)) << 16);
        }
        reinterpret_cast<uint4*>(tab)[k] = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
  }
  __syncthreads();
  // ---- buckets: z = (x - loc) * inv_scale on the knot grid, then the fraction
  // of the way to the next knot
  constexpr uint32_t kAll = kInvalidKey32 - 1u;  // every valid key
  const CountTotals ct = count_cells<NT, V>(key, kAll, L, sm, W, [&](int j, uint32_t (&b)[4]) {
    uint32_t tw[4];
    float fr[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // four cells' loads in flight at a time
      const float z = (key_to_f32(key[4 * j + k]) - loc) * inv_scale;
      float u = (z - lo) * inv_dz;
      u = fminf(fmaxf(u, 0.0f), static_cast<float>(kCdfKnots - 1));
      const int kk = min(static_cast<int>(u), kCdfKnots - 2);
      fr[k] = fminf(u - static_cast<float>(kk), 0.99999994f);
      tw[k] = tab[kk];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      b[k] = (tw[k] & 0xFFFFu) + static_cast<uint32_t>(static_cast<float>(tw[k] >> 16) * fr[k]);
  });
  const int largest = m > 0 ? static_cast<int>(ct.largest) : 0;
  const bool fits = largest <= min(a.learn_cap, 0xFFF);
  if (tid == 0 && stats != nullptr) {
    stats[0] = fits ? kLearnOk : kLearnOverflow;
    stats[1] = largest;
    stats[2] = static_cast<int>(ct.squares) + m;
    stats[3] = m;
  }
  if (!fits) {  // uniform across the block
    if (tid == 0) fb.items[atomicAdd(fb.count, 1)] = item_id;
    return;
  }
  scatter_cells<NT, V>(key, kAll, m, L, sm, W);
  spread_positions<NT, V, false>(L, sm, m, ct.largest > kSpreadHeavy, key, W);
  // No order check is needed: the bucket map is non-decreasing in the key
  // (each step -- the exact key-to-value inverse, the affine standardisation
  // by a positive scale, the clamped knot position, the two knots' buckets
  // of a non-decreasing table and the fraction below one between them -- is
  // monotone under round-to-nearest, and a bucket ends at or below the next
  // knot's), so every bucket holds smaller keys than the next, and the table
  // was checked above.
  ric_epilogue<NT, V>(a, rp, t, f, key, kAll, W, joint, lone, ct.largest, drop, marks, red);
}

template <int NT, int V>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_ric_learned(RankIcArgs<float, float> a, RicPrep rp) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int item = static_cast<int>(blockIdx.x);
  ric_learned_body<NT, V>(a, rp, item / a.F, item % a.F, item, RicList{rp.fb_count, rp.fb_items}, sm);
}

// ---------------------------------------------------------------------------
// plain path (and the learned path's fallback)
// ---------------------------------------------------------------------------
// Section (t, f) by the radix sort.
template <int NT, int V>
__device__ __noinline__ void ric_radix(const RankIcArgs<float, float>& a, const RicPrep& rp, const int t, const int f,
                                       uint8_t* sm) {
  constexpr int C = 4 * V;
  const SortedLayout<NT> L(a.N);
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  unsigned long long* scan64 = reinterpret_cast<unsigned long long*>(sm + L.red);
  uint32_t* drop = reinterpret_cast<uint32_t*>(sm + L.dw);
  uint32_t* marks = reinterpret_cast<uint32_t*>(sm + L.dw2);
  uint32_t* k0 = reinterpret_cast<uint32_t*>(sm + L.k0);
  uint32_t* k1 = reinterpret_cast<uint32_t*>(sm + L.k1);
  uint16_t* i0 = reinterpret_cast<uint16_t*>(sm + L.i0);
  uint16_t* i1 = reinterpret_cast<uint16_t*>(sm + L.i1);
  uint32_t key[C], W[C], joint, lone;
  ric_cells<NT, V, false>(a, rp, t, f, drop, marks, red, key, joint, lone);
  const uint32_t valid = joint | lone;
  int base[V];
  const int m = compact_bases<NT, V>(valid, base, scan64);  // its barriers complete the marks
#pragma unroll
  for (int j = 0; j < V; ++j) {
    int p = base[j];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      if ((valid >> c) & 1u) {
        k0[p] = key[c];
        i0[p] = static_cast<uint16_t>(cell_col<NT>(c));
        ++p;
      }
    }
  }
  __syncthreads();
  uint32_t* ks;
  uint16_t* is;
  block_radix_sort<NT, C, uint32_t>(k0, i0, k1, i1, m, sm + L.scratch, &ks, &is);
  uint32_t* RK = (ks == k0) ? k1 : k0;  // sorted position by column
  for (int p = static_cast<int>(threadIdx.x); p < m; p += NT) RK[is[p]] = static_cast<uint32_t>(p);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < C; ++c) W[c] = ((valid >> c) & 1u) ? RK[cell_col<NT>(c)] : 0u;
  ric_epilogue<NT, V>(a, rp, t, f, key, kInvalidKey32 - 1u, W, joint, lone, static_cast<uint32_t>(m), drop, marks, red);
}

// Section (t, f) by value-spread buckets.
template <int NT, int V, bool STREAM>
FCB_DEV void ric_plain_body(const RankIcArgs<float, float>& a, const RicPrep& rp, const int t, const int f,
                            uint8_t* sm) {
  constexpr int C = 4 * V;
  const SpreadLayout<NT, V> L(a.N);
  uint32_t* red = reinterpret_cast<uint32_t*>(sm + L.red);
  uint32_t* drop = reinterpret_cast<uint32_t*>(sm + L.bits);
  uint32_t* marks = reinterpret_cast<uint32_t*>(sm + L.bits2);
  uint32_t key[C], W[C], joint, lone;
  ric_cells<NT, V, STREAM>(a, rp, t, f, drop, marks, red, key, joint, lone);
  SpreadTotals T;
  if (!spread_place<NT, V>(key, L, sm, W, T)) {
    ric_radix<NT, V>(a, rp, t, f, sm);
    return;
  }
  spread_positions<NT, V, false>(L, sm, T.m, T.heavy, key, W);
  ric_epilogue<NT, V>(a, rp, t, f, key, T.range, W, joint, lone, kSpreadMaxBucket, drop, marks, red);
}

// LIST: sections come from the learned kernel's fallback list (persistent
// CTAs stride over it); otherwise blockIdx.x = t * F + f.
template <int NT, int V, bool LIST>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_ric_plain(RankIcArgs<float, float> a, RicPrep rp) {
  extern __shared__ __align__(16) uint8_t sm[];
  if (!LIST) {
    ric_plain_body<NT, V, true>(a, rp, static_cast<int>(blockIdx.x) / a.F, static_cast<int>(blockIdx.x) % a.F, sm);
    return;
  }
  const int nitems = *static_cast<volatile int*>(rp.fb_count);
  for (int it = blockIdx.x; it < nitems; it += static_cast<int>(gridDim.x)) {
    const int item = rp.fb_items[it];
    ric_plain_body<NT, V, false>(a, rp, item / a.F, item % a.F, sm);
    __syncthreads();  // the next section reuses the shared memory
  }
}

// ---------------------------------------------------------------------------
// many panels per launch (the batch)
// ---------------------------------------------------------------------------
// The panels of one size variant share a launch: one CTA per item (a date of
// a panel for the returns pass, a (date, factor) section for the rank pass),
// the item's panel found by binary search over the exclusive prefix `off` of
// the panels' item counts.
FCB_DEV int panel_of(const int* __restrict__ off, int np, int item) {
  int lo = 0, hi = np - 1;  // the last panel whose first item is <= item
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(off + mid) <= item) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <int NT, int V>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_ric_prep_batch(const RicPanel* __restrict__ P,
                                                                        const int* __restrict__ off, int np) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int item = static_cast<int>(blockIdx.x);
  const int q = panel_of(off, np, item);
  const RankIcArgs<float, float> a = P[q].a;
  const RicPrep rp = P[q].rp;
  const int t = item - __ldg(off + q);
  ric_prep_body<NT, V>(a.R, a.rmask, a.fmask, a.N, t, rp.word + static_cast<size_t>(t) * rp.ld, sm);
}

template <int NT, int V>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_ric_items_batch(const RicPanel* __restrict__ P,
                                                                         const int* __restrict__ off, int np) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int item = static_cast<int>(blockIdx.x);
  const int q = panel_of(off, np, item);
  const RankIcArgs<float, float> a = P[q].a;
  const RicPrep rp = P[q].rp;
  const int l = item - __ldg(off + q);
  ric_plain_body<NT, V, true>(a, rp, l / a.F, l % a.F, sm);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {
// Shared memory of the kernels of one variant at width N: the spread layout
// or, for crowded sections, the radix forms' layout in the same memory.
template <int NT, int V>
size_t ric_smem(int N) {
  const size_t a = SpreadLayout<NT, V>(N).total, b = SortedLayout<NT>(N).total;
  return a > b ? a : b;
}
template <typename K>
cudaError_t set_smem(K* kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}
// One wave of CTAs of a kernel that strides over a device list.
template <typename K>
cudaError_t one_wave(K* kernel, int threads, size_t smem, long long* grid) {
  int occ = 0, dev = 0, sms = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem);
  if (e != cudaSuccess) return e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  *grid = static_cast<long long>(occ > 0 ? occ : 1) * (sms > 0 ? sms : 1);
  return cudaSuccess;
}

template <int NT, int V>
cudaError_t ric_launch(const RankIcArgs<float, float>& a, RicPrep rp, bool learned, cudaStream_t st) {
  const size_t smem = ric_smem<NT, V>(a.N);
  if (smem > kMaxSmemPerBlock || a.N > 4 * NT * V) return cudaErrorInvalidValue;
  cudaError_t e = set_smem(k_ric_prep<NT, V>, smem);
  if (e != cudaSuccess) return e;
  k_ric_prep<NT, V><<<a.T, NT, smem, st>>>(a.R, a.rmask, a.fmask, a.N, rp);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const long long grid = static_cast<long long>(a.T) * a.F;
  if (grid > 2147483647LL) return cudaErrorInvalidValue;
  if (!learned) {
    if ((e = set_smem(k_ric_plain<NT, V, false>, smem)) != cudaSuccess) return e;
    k_ric_plain<NT, V, false><<<static_cast<unsigned>(grid), NT, smem, st>>>(a, rp);
    return cudaGetLastError();
  }
  if ((e = set_smem(k_ric_learned<NT, V>, smem)) != cudaSuccess) return e;
  k_ric_learned<NT, V><<<static_cast<unsigned>(grid), NT, smem, st>>>(a, rp);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  // the plain kernel takes the sections the learned kernel handed back;
  // persistent CTAs (one wave) read the list length on the device and exit at
  // once when it is empty
  if ((e = set_smem(k_ric_plain<NT, V, true>, smem)) != cudaSuccess) return e;
  long long fb_grid = 0;
  if ((e = one_wave(k_ric_plain<NT, V, true>, NT, smem, &fb_grid)) != cudaSuccess) return e;
  k_ric_plain<NT, V, true><<<static_cast<unsigned>(fb_grid < grid ? fb_grid : grid), NT, smem, st>>>(a, rp);
  return cudaGetLastError();
}
}  // namespace

size_t ric_prep_bytes(int T, int N, int F) {
  const size_t ld = (static_cast<size_t>(N) + 3) / 4 * 4;
  return static_cast<size_t>(T) * ld * 4 + 256 + (static_cast<size_t>(T) * F + 64) * 4 + 256;
}

RicPrep ric_prep_carve(void* base, int T, int N, int F) {
  RicPrep rp{};
  rp.ld = (N + 3) / 4 * 4;
  uint8_t* p = static_cast<uint8_t*>(base);
  rp.word = reinterpret_cast<uint32_t*>(p);
  p += (static_cast<size_t>(T) * rp.ld * 4 + 255) & ~size_t(255);
  rp.fb_count = reinterpret_cast<int*>(p);
  p += 256;
  rp.fb_items = reinterpret_cast<int*>(p);
  (void)F;
  return rp;
}


namespace {
template <int NT, int V>
cudaError_t ric_batch_launch(const RicBatchVariant& v, bool prep, cudaStream_t st) {
  const size_t smem = ric_smem<NT, V>(v.maxN);
  if (smem > kMaxSmemPerBlock || v.maxN > 4 * NT * V) return cudaErrorInvalidValue;
  const cudaError_t e = prep ? set_smem(k_ric_prep_batch<NT, V>, smem) : set_smem(k_ric_items_batch<NT, V>, smem);
  if (e != cudaSuccess) return e;
  if (prep)
    k_ric_prep_batch<NT, V><<<v.dates, NT, smem, st>>>(v.panels, v.off_dates, v.np);
  else
    k_ric_items_batch<NT, V><<<v.items, NT, smem, st>>>(v.panels, v.off_items, v.np);
  return cudaGetLastError();
}

cudaError_t ric_batch(int variant, const RicBatchVariant& v, bool prep, cudaStream_t st) {
  if (v.np < 1 || v.items < 1 || v.maxN > ric_variant_cap(variant)) return cudaErrorInvalidValue;
  switch (variant) {
    case 0: return ric_batch_launch<128, 1>(v, prep, st);
    case 1: return ric_batch_launch<192, 1>(v, prep, st);
    case 2: return ric_batch_launch<256, 1>(v, prep, st);
    case 3: return ric_batch_launch<192, 2>(v, prep, st);
    case 4: return ric_batch_launch<256, 2>(v, prep, st);
    case 5: return ric_batch_launch<256, 3>(v, prep, st);
    case 6: return ric_batch_launch<448, 3>(v, prep, st);
    case 7: return ric_batch_launch<512, 4>(v, prep, st);
    default: return ric_batch_launch<1024, 4>(v, prep, st);
  }
}
}  // namespace

int ric_variant_cap(int variant) {
  static const int caps[kRicVariants] = {512, 768, 1024, 1536, 2048, 3072, 5120, 8192, 16384};
  return (variant >= 0 && variant < kRicVariants) ? caps[variant] : 0;
}

cudaError_t launch_rank_ic_prep_batch(int variant, const RicBatchVariant& v, cudaStream_t st) {
  return ric_batch(variant, v, true, st);
}
cudaError_t launch_rank_ic_items_batch(int variant, const RicBatchVariant& v, cudaStream_t st) {
  return ric_batch(variant, v, false, st);
}

bool ric_items_fit(int N) { return N >= 1 && N <= kSmemRankCap; }

cudaError_t launch_rank_ic_items(const RankIcArgs<float, float>& a, RicPrep rp, bool learned, cudaStream_t st) {
  if (!ric_items_fit(a.N) || a.rank_f_out != nullptr || a.rank_r_out != nullptr) return cudaErrorInvalidValue;
  if (learned && (a.cdf_table == nullptr || a.cdf_zrange == nullptr)) return cudaErrorInvalidValue;
  return section_shape(a.N, [&](auto shape) {
    return ric_launch<decltype(shape)::kThreads, decltype(shape)::kVectors>(a, rp, learned, st);
  });
}

}  // namespace fcb
