// stock_corr.cu -- FP64 pairwise-complete Pearson of every pair of columns of
// a (T,N) panel (the drop-in path), for sm_100a.
//
// A pair's six moment sums run over the dates on which both columns are
// valid.  Only one of them, sum x'y' of column-centred values (0 where
// invalid), is a matrix product; it runs on the FP64 tensor cores
// (k_sc_gram).  The other five are cheaper than products:
//   * n is a population count of the AND of two validity bitmasks;
//   * sum x' and sum x'^2 over the other column's valid dates are the column's
//     totals less the dates that the other column misses.  A column misses few
//     dates as a rule, so k_sc_pairsum adds up short lists: one CTA keeps the
//     centred values of 16 columns in shared memory ([date][16], and the sums
//     of every 32 dates) and walks every column's list of missing dates (of
//     valid dates where more than a sixth is missing); 32 dates that are
//     all on the list count as one entry.  Where what is taken away is more than a
//     quarter of the column's sum of squares (an outlier on a date that the other
//     column misses, as a rule), the pair's sums are formed over the joint dates
//     directly: the subtraction then rounds less than the sums do.
// Steps: column statistics (compensated mean, extrema; replaces
// stock_corr_gpu's col_stats_kernel, src/stock_corr.cu:73-116, and the
// demean_kernel's mean, :244-261), column-major copies and bitmasks, lists,
// pair sums, Gram pass with the finalize and its gates
// (src/stock_corr_impl.cuh:102-132), and the two-pass fallback of the flagged
// pairs (two_pass_centered, src/stock_corr_impl.cuh:150-201; _two_pass_corr,
// fc/_cpu_core.py:111-137).
// Measured on a B200, 1218 x 2000 f32 masked (7 % missing): 2.71 ms -> 0.44 ms a
// call; k_sc_gram 218 us (from 1905; FP64 tensor pipe, 150 us at its peak, and
// the finalize on the same pipe), k_sc_pairsum 120 (shared-memory bandwidth),
// k_sc_direct 10, statistics, copies and lists 38 (from 103).
// 64 x 32 tiles, four CTAs per SM: 64 x 64 tiles take 267-294 us, their last
// wave being nearly empty.  Against 80-bit sums the rms error of a correlation
// of 0.1 is 2.4e-17 (2.7e-17 with the six products): every long sum is a sum of
// short ones, single chains over all dates gave 1.1e-16.
// The domain check and the full-validity flag stay on the device: the later
// kernels return at once when the panel is out of the domain, and the host
// reads the summary once, at the end.
#include <algorithm>

#include "corr_common.cuh"
#include "fcb_kernels.h"

namespace fcb {
namespace {

constexpr int kScRows = 16;      // columns of one k_sc_pairsum CTA
constexpr int kScChunk = 1536;   // dates it holds at a time (192 KB, and 12 KB of sums)
constexpr int kScTile = 64, kScTileJ = 32;  // k_sc_gram tile: rows, columns
constexpr int kScK = 32;         // dates per stage
constexpr int kScBlock = 5120;   // columns whose pair sums are held at a time
constexpr int kScDirect = 1 << 18;  // pair sums that k_sc_direct takes of them

FCB_DEV bool out_of_domain(const ScSummary* s) {
  const double mx = __longlong_as_double(static_cast<long long>(s->max_abs));
  const double mn = __longlong_as_double(static_cast<long long>(~s->min_abs_inv));
  return mx > 1e150 || mn < 1e-150;  // (no valid nonzero cell: mn is a NaN)
}

// The mask byte of a cell (1 without a mask); valid = finite and nonzero byte.
FCB_DEV uint32_t sc_mask(const uint8_t* mask, size_t e) { return mask != nullptr ? __ldg(mask + e) : 1u; }

// ---------------------------------------------------------------------------
// column statistics
// ---------------------------------------------------------------------------
// 32 columns per CTA, lane = column (coalesced rows); warp w takes every 32nd
// date with its own compensated sum, and the 32 partials merge pairwise.  (One
// serial compensated sum per column costs four dependent FP64 adds, about 120
// clocks, per date: 80 us for 1218 dates.)  The mean is the shift of the
// centred values; the fallback forms its own means.
constexpr int kStWarps = 32;
template <typename TIN>
__global__ void __launch_bounds__(32 * kStWarps) k_sc_colstats(const TIN* __restrict__ X, const uint8_t* __restrict__ mask,
                                                               int T, int N, ColStat* __restrict__ st,
                                                               ScSummary* __restrict__ sum) {
  constexpr int kHalf = kStWarps / 2;
  __shared__ double ps[kHalf][32], pc[kHalf][32], pmn[kHalf][32], pmx[kHalf][32], pna[kHalf][32];
  __shared__ int pn[kHalf][32];
  const int lane = static_cast<int>(threadIdx.x & 31), w = static_cast<int>(threadIdx.x >> 5);
  const int i = blockIdx.x * 32 + lane;
  Kahan k;
  int cnt = 0;
  TIN lo = TIN(0), hi = TIN(0), near0 = TIN(0);  // extrema in the input type
  if (i < N) {
    constexpr int U = 8;  // dates loaded ahead of their use
    for (int t0 = w; t0 < T; t0 += U * kStWarps) {
      TIN x[U];
      uint32_t m[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * kStWarps;
        const size_t e = static_cast<size_t>(t) * N + i;
        x[u] = t < T ? __ldg(X + e) : TIN(0);
        m[u] = t < T ? sc_mask(mask, e) : 0u;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const TIN v = x[u];
        if (m[u] != 0u && finite_f64(static_cast<double>(v))) {
          k.add(static_cast<double>(v));
          lo = cnt > 0 ? (v < lo ? v : lo) : v;
          hi = cnt > 0 ? (v > hi ? v : hi) : v;
          ++cnt;
          const TIN av = v < TIN(0) ? -v : v;
          if (av != TIN(0) && (near0 == TIN(0) || av < near0)) near0 = av;
        }
      }
    }
  }
  double mn = cnt > 0 ? static_cast<double>(lo) : kBigPos, mx = cnt > 0 ? static_cast<double>(hi) : -kBigPos;
  double mna = near0 != TIN(0) ? static_cast<double>(near0) : kBigPos;
  // pairwise merge of the warps' partials
  for (int h = kStWarps / 2; h > 0; h >>= 1) {
    if (w >= h && w < 2 * h) {
      ps[w - h][lane] = k.s;
      pc[w - h][lane] = k.c;
      pn[w - h][lane] = cnt;
      pmn[w - h][lane] = mn;
      pmx[w - h][lane] = mx;
      pna[w - h][lane] = mna;
    }
    __syncthreads();
    if (w < h) {
      k.add(ps[w][lane]);
      k.add(-pc[w][lane]);
      cnt += pn[w][lane];
      mn = fmin(mn, pmn[w][lane]);
      mx = fmax(mx, pmx[w][lane]);
      mna = fmin(mna, pna[w][lane]);
    }
    __syncthreads();
  }
  if (w != 0) return;
  const double mxa = cnt > 0 ? fmax(fabs(mn), fabs(mx)) : 0.0;
  if (i < N) {
    ColStat c;
    c.count = static_cast<double>(cnt);
    c.mean = cnt > 0 ? k.s / static_cast<double>(cnt) : 0.0;
    c.min = mn;
    c.max = mx;
    c.min_abs = mna;
    c.max_abs = mxa;
    c.s2 = 0.0;
    c.s1 = 0.0;
    st[i] = c;
  }
  // non-negative doubles order like their bit patterns
  unsigned long long a = static_cast<unsigned long long>(__double_as_longlong(mxa));
  unsigned long long z = mna < kBigPos ? ~static_cast<unsigned long long>(__double_as_longlong(mna)) : 0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a2 = __shfl_xor_sync(kFull, a, o), z2 = __shfl_xor_sync(kFull, z, o);
    a = a2 > a ? a2 : a;
    z = z2 > z ? z2 : z;
  }
  const bool part = __any_sync(kFull, i < N && cnt < T);
  if (lane == 0) {
    atomicMax(&sum->max_abs, a);
    atomicMax(&sum->min_abs_inv, z);
    if (part) atomicExch(&sum->masked, 1);
  }
}

// (T,N) row-major -> column-major Xraw, Xc (N,Tp) (0 where invalid or past T)
// and validity bits (N, Tp/32).
template <typename TIN>
__global__ void k_sc_transpose(const TIN* __restrict__ X, const uint8_t* __restrict__ mask, int T, int N, int Tp,
                               const ColStat* __restrict__ st, double* __restrict__ Xraw, double* __restrict__ Xc,
                               uint32_t* __restrict__ bits) {
  __shared__ double tx[32][33];
  __shared__ uint8_t tm[32][33];
  const int t0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
  TIN x[4];
  uint32_t m[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {  // blockDim.y is 8
    const int t = t0 + q * 8 + threadIdx.y, i = i0 + threadIdx.x;
    const bool in = t < T && i < N;
    const size_t e = static_cast<size_t>(t) * N + i;
    x[q] = in ? __ldg(X + e) : TIN(0);
    m[q] = in ? sc_mask(mask, e) : 0u;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double v = static_cast<double>(x[q]);
    const bool ok = m[q] != 0u && finite_f64(v);
    tx[q * 8 + threadIdx.y][threadIdx.x] = ok ? v : 0.0;
    tm[q * 8 + threadIdx.y][threadIdx.x] = ok ? 1 : 0;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r;
    if (i >= N) continue;  // uniform across the warp
    const double v = tx[threadIdx.x][r];
    const bool ok = tm[threadIdx.x][r] != 0;
    const size_t e = static_cast<size_t>(i) * Tp + t0 + threadIdx.x;
    Xraw[e] = v;
    Xc[e] = ok ? v - st[i].mean : 0.0;
    const unsigned b = __ballot_sync(kFull, ok);
    if (threadIdx.x == 0) bits[static_cast<size_t>(i) * (Tp / 32) + blockIdx.x] = b;
  }
}

// One warp per column: sums of the centred values and their squares, and the
// column's list -- its missing dates when they are at most a sixth (invert =
// 1), its valid dates otherwise.  Per chunk of dates two runs of entries: the
// listed dates, then the aligned groups of 32 dates that are listed as a whole
// (date and group numbers within the chunk), each run padded to eight with the
// number of a row of zeros.  ptr[2c], ptr[2c + 1] are where chunk c's runs
// start.
__global__ void k_sc_lists(const double* __restrict__ Xc, const uint32_t* __restrict__ bits, int T, int N, int Tp,
                           int nchunk, int lcap, ColStat* __restrict__ st, uint16_t* __restrict__ list,
                           int* __restrict__ ptr, int* __restrict__ invert) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= N) return;
  TwoSum s2, s1;  // the lists' sums are taken away from these
#pragma unroll 4
  for (int t = lane; t < Tp; t += 32) {
    const double d = Xc[static_cast<size_t>(w) * Tp + t];
    s2.add(d * d);
    s1.add(d);
  }
  s2.warp_total();
  s1.warp_total();
  const int missing = T - static_cast<int>(st[w].count);
  const bool inv = 6ll * missing <= T;
  if (lane == 0) {
    st[w].s2 = s2.value();
    st[w].s1 = s1.value();
    invert[w] = inv ? 1 : 0;
  }
  uint16_t* out = list + static_cast<size_t>(w) * lcap;
  int* p = ptr + static_cast<size_t>(w) * (2 * nchunk + 1);
  const uint32_t* b = bits + static_cast<size_t>(w) * (Tp / 32);
  int pos = 0;
  auto pad_to = [&](int zero_row) {
    const int pad = (8 - (pos & 7)) & 7;
    if (lane < pad) out[pos + lane] = static_cast<uint16_t>(zero_row);
    pos += pad;
  };
  for (int c = 0; c < nchunk; ++c) {
    const int tn = min(T - c * kScChunk, kScChunk), nw = (tn + 31) / 32;
    // a lane keeps the words lane, lane + 32 of the chunk (at most 48)
    uint32_t word[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int k = q * 32 + lane;
      uint32_t m = k < nw ? b[c * (kScChunk / 32) + k] : 0u;
      if (inv) m = ~m;
      if (k == tn / 32) m &= (1u << (tn & 31)) - 1u;  // (the last, partial word)
      word[q] = k < nw ? m : 0u;
    }
    if (lane == 0) p[2 * c] = pos;
    for (int k = 0; k < nw; ++k) {
      const uint32_t m = __shfl_sync(kFull, k < 32 ? word[0] : word[1], k & 31);
      if (m == kFull) continue;
      if ((m >> lane) & 1u) out[pos + __popc(m & lanemask_lt())] = static_cast<uint16_t>(32 * k + lane);
      pos += __popc(m);
    }
    pad_to(tn);
    if (lane == 0) p[2 * c + 1] = pos;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const unsigned whole = __ballot_sync(kFull, word[q] == kFull);
      if (word[q] == kFull) out[pos + __popc(whole & lanemask_lt())] = static_cast<uint16_t>(q * 32 + lane);
      pos += __popc(whole);
    }
    pad_to(nw);
  }
  if (lane == 0) p[2 * nchunk] = pos;
}

// ---------------------------------------------------------------------------
// pair sums: AB[(j - ja) * ld + (i - ia)] = (sum x'_i, sum x'_i^2) over the
// valid dates of column j
// ---------------------------------------------------------------------------
// Sum and sum of squares of a column's centred values over the dates in `bits`,
// by W lanes of a warp (mask `lanes`): a lane every W-th date, eight loads ahead
// of their use.
template <int W>
FCB_DEV double2 joint_sums(const double* __restrict__ x, const uint32_t* __restrict__ bits, int T, int lane,
                           uint32_t lanes) {
  constexpr int U = 8;
  double a[4] = {}, q[4] = {};
  for (int t0 = lane; t0 < T; t0 += U * W) {
    double v[U];
    uint32_t b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + W * u;
      b[u] = t < T ? __ldg(bits + (t >> 5)) >> (t & 31) : 0u;
      v[u] = t < T ? __ldg(x + t) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double d = (b[u] & 1u) != 0u ? v[u] : 0.0;
      a[u & 3] += d;
      q[u & 3] = fma(d, d, q[u & 3]);
    }
  }
  double2 s = make_double2((a[0] + a[1]) + (a[2] + a[3]), (q[0] + q[1]) + (q[2] + q[3]));
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) {
    s.x += __shfl_xor_sync(lanes, s.x, o);
    s.y += __shfl_xor_sync(lanes, s.y, o);
  }
  return s;
}

// A half-warp takes one column j at a time: lane = column i.  A listed date
// costs one 128-byte shared-memory row and two FP64 instructions per lane, a
// listed group of 32 dates twice the row.  Shared-memory bandwidth bounds it.
// Chunk c of the dates; the sums of earlier chunks wait in AB.
// LONG: the list's short chains are added to twice the precision (see k_sc_gram).
template <typename TIN, bool LONG>
__global__ void __launch_bounds__(1024, 1)
    k_sc_pairsum(const TIN* __restrict__ X, const uint8_t* __restrict__ mask, const double* __restrict__ Xc,
                 const uint32_t* __restrict__ bits, const ColStat* __restrict__ st, const uint16_t* __restrict__ list,
                 const int* __restrict__ ptr, const int* __restrict__ invert, int T, int N, int Tp, int nchunk,
                 int lcap, int c, int ia, int ib, int ja, int jb, int ld, double2* __restrict__ AB,
                 int* __restrict__ direct_list, ScSummary* __restrict__ sum) {
  if (sum->masked == 0 || out_of_domain(sum)) return;  // a full panel needs no pair sums
  extern __shared__ __align__(16) double xs[];  // [tn + 1][kScRows] values, [nw + 1][kScRows] sums; last rows zero
  const int t0 = c * kScChunk, tn = min(T - t0, kScChunk), nw = (tn + 31) / 32;
  double2* gs = reinterpret_cast<double2*>(xs + static_cast<size_t>(tn + 1) * kScRows);
  const int i0 = ia + static_cast<int>(blockIdx.x) * kScRows;
  {
    const int li = static_cast<int>(threadIdx.x) % kScRows, i = i0 + li, step = static_cast<int>(blockDim.x) / kScRows;
    const double mean = i < ib ? st[i].mean : 0.0;
    constexpr int U = 8;  // dates loaded ahead of their use
    for (int t1 = static_cast<int>(threadIdx.x) / kScRows; t1 < tn; t1 += U * step) {
      TIN x[U];
      uint32_t m[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t1 + u * step;
        const bool in = t < tn && i < ib;
        const size_t at = static_cast<size_t>(t0 + t) * N + i;
        x[u] = in ? __ldg(X + at) : TIN(0);
        m[u] = in ? sc_mask(mask, at) : 0u;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t1 + u * step;
        const double v = static_cast<double>(x[u]);
        if (t < tn) xs[t * kScRows + li] = m[u] != 0u && finite_f64(v) ? v - mean : 0.0;
      }
    }
    if (threadIdx.x < kScRows) xs[tn * kScRows + li] = 0.0;
  }
  __syncthreads();
  for (int e = static_cast<int>(threadIdx.x); e < (nw + 1) * kScRows; e += static_cast<int>(blockDim.x)) {
    const int k = e / kScRows;
    double a = 0.0, q = 0.0;
    if (k < nw)
      for (int t = 32 * k; t < min(tn, 32 * k + 32); ++t) {
        const double x = xs[t * kScRows + e % kScRows];
        a += x;
        q = fma(x, x, q);
      }
    gs[e] = make_double2(a, q);
  }
  __syncthreads();
  const int lane = threadIdx.x & 15, i = i0 + lane;
  const uint32_t half = 0xFFFFu << (threadIdx.x & 16);
  const int hw = static_cast<int>(threadIdx.x >> 4), nhw = static_cast<int>(blockDim.x >> 4);
  const double* col = xs + lane;
  const double2* gcol = gs + lane;
  const double s1 = i < ib ? st[i].s1 : 0.0, s2 = i < ib ? st[i].s2 : 0.0;
  for (int j = ja + static_cast<int>(blockIdx.y) * nhw + hw; j < jb; j += nhw * static_cast<int>(gridDim.y)) {
    const int* p = ptr + static_cast<size_t>(j) * (2 * nchunk + 1) + 2 * c;
    const uint4* l = reinterpret_cast<const uint4*>(list + static_cast<size_t>(j) * lcap);
    const int k0 = p[0] >> 3, k1 = p[1] >> 3, k2 = p[2] >> 3;
    double a0 = 0.0, a1 = 0.0, q0 = 0.0, q1 = 0.0;
    TwoSum ta, tq;
    auto add_chains = [&](TwoSum& t, double x) {
      if (LONG)
        t.add(x);
      else
        t.s += x;
    };
    uint4 next = k0 < k2 ? __ldg(l + k0) : make_uint4(0u, 0u, 0u, 0u);
    for (int k = k0; k < k1; ++k) {
      const uint4 v = next;
      if (k + 1 < k2) next = __ldg(l + k + 1);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double x = col[(w[u] & 0xFFFFu) * kScRows];
        const double y = col[(w[u] >> 16) * kScRows];
        a0 += x;
        q0 = fma(x, x, q0);
        a1 += y;
        q1 = fma(y, y, q1);
      }
      if (((k - k0) & 3) == 3) {  // long lists: short chains round less
        add_chains(ta, a0 + a1);
        add_chains(tq, q0 + q1);
        a0 = a1 = q0 = q1 = 0.0;
      }
    }
    for (int k = k1; k < k2; ++k) {
      const uint4 v = next;
      if (k + 1 < k2) next = __ldg(l + k + 1);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double2 x = gcol[(w[u] & 0xFFFFu) * kScRows];
        const double2 y = gcol[(w[u] >> 16) * kScRows];
        a0 += x.x;
        q0 += x.y;
        a1 += y.x;
        q1 += y.y;
      }
      if (LONG && ((k - k1) & 3) == 3) {
        add_chains(ta, a0 + a1);
        add_chains(tq, q0 + q1);
        a0 = a1 = q0 = q1 = 0.0;
      }
    }
    add_chains(ta, a0 + a1);
    add_chains(tq, q0 + q1);
    double a = ta.value(), q = tq.value();
    double2* o = AB + static_cast<size_t>(j - ja) * ld + (i - ia);
    if (c > 0 && i < ib) {
      const double2 e = *o;
      a += e.x;
      q += e.y;
    }
    if (c == nchunk - 1 && invert[j] != 0) {
      // where a quarter of the squares or more would be taken away, the sums are
      // formed over the joint dates: by k_sc_direct, or here when its list is full
      bool here = false;
      if (i < ib && q > 0.25 * s2) {
        const int at = atomicAdd(&sum->direct, 1);
        here = at >= kScDirect;
        if (!here) direct_list[at] = (j - ja) * ld + (i - ia);
      }
      uint32_t direct = __ballot_sync(half, here) & half;
      a = s1 - a;
      q = s2 - q;
      for (; direct != 0u; direct &= direct - 1u) {  // uniform across the half-warp
        const int l = (__ffs(direct) - 1) & 15;
        const double2 d = joint_sums<16>(Xc + static_cast<size_t>(i0 + l) * Tp,
                                         bits + static_cast<size_t>(j) * (Tp / 32), T, lane, half);
        if (lane == l) {
          a = d.x;
          q = d.y;
        }
      }
    }
    if (i < ib) *o = make_double2(a, q);
  }
}

// The listed pair sums over the joint dates, one warp each.  (One column's
// outlier on a date that half of the others miss lists a thousand pairs of one
// k_sc_pairsum CTA, 8 us each there: 1218 x 2000 587 us a call, and 442 so.)
__global__ void __launch_bounds__(256) k_sc_direct(const double* __restrict__ Xc, const uint32_t* __restrict__ bits,
                                                   int T, int Tp, int ia, int ja, int ld, const int* __restrict__ list,
                                                   double2* __restrict__ AB, const ScSummary* __restrict__ sum) {
  const int cnt = min(sum->direct, kScDirect), nw = static_cast<int>(gridDim.x * blockDim.x) >> 5;
  for (int g = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < cnt; g += nw) {
    const int e = list[g], j = ja + e / ld, i = ia + e % ld, lane = static_cast<int>(threadIdx.x & 31);
    const double2 s = joint_sums<32>(Xc + static_cast<size_t>(i) * Tp, bits + static_cast<size_t>(j) * (Tp / 32), T,
                                     lane, kFull);
    if (lane == 0) AB[e] = s;
  }
}

// ---------------------------------------------------------------------------
// Gram pass
// ---------------------------------------------------------------------------
// Tile b of the row-major list of tiles on or above the diagonal: row block ib
// has the nj - 2 ib column blocks from 2 ib on (64-row blocks, 32-column
// blocks).
FCB_DEV void tri_tile(int b, int ni, int nj, int& ib, int& jb) {
  int lo = 0, hi = ni - 1;
  auto first = [&](int r) { return static_cast<long long>(r) * nj - static_cast<long long>(r) * (r - 1); };
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (first(mid) <= b) lo = mid; else hi = mid - 1;
  }
  ib = lo;
  jb = 2 * ib + static_cast<int>(b - first(ib));
}

FCB_DEV void cp_async16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// One stage: 32 dates of the tile's two sets of columns, and their bits.
struct ScStage {
  double a[kScTile][kScK], b[kScTileJ][kScK];
};
// Where date t of a staged row lies. Odd rows have their halves swapped, so
// that the 8 threads of a 16-byte load phase (2 rows x 8 dates) meet every bank
// once.
FCB_DEV int sc_at(int row, int t) { return t ^ ((row & 1) << 3); }
// The tile's products and counts, for the finalize, and the bits that are
// counted.
constexpr int kScWords = 48;
struct ScProducts {
  double xy[kScTile][kScTileJ + 1];
  uint32_t n[kScTile][kScTileJ + 1];
  uint32_t w[kScTile + kScTileJ][kScWords + 1];  // words of 32 dates each
};

// 64 x 32 tiles of columns [ia, ib) x [ja, jb) (the same range: the tiles on
// and above the diagonal); eight warps of 16 x 16, 2 x 2 FP64 matrix
// instructions per four dates and warp against four fragment loads.  The FP64 tensor
// pipe bounds it: one product instead of the six masked sums per pair and
// date (eight FP64 instructions) that it formed before.
// LONG (above kTwoPassKahanT dates, where the two-pass sums of pairs that fail the
// cancellation gate were compensated): the stages' sums are added to twice the
// precision, 3 CTAs per SM.  (2500 dates, correlations near 0.9, means of 50
// spreads: rms error 9e-17, 2.4e-16 with plain additions, 7.5e-17 by two passes;
// 3000 x 1000 308 -> 342 us a call, the two passes 24.9 ms.)
template <bool LONG>
__global__ void __launch_bounds__(256, LONG ? 3 : 4)
    k_sc_gram(const double* __restrict__ Xc, const uint32_t* __restrict__ bits, const ColStat* __restrict__ st, int T,
              int N, int Tp, int ia, int ib, int ja, int jb, const double2* __restrict__ ABij,
              const double2* __restrict__ ABji, double* __restrict__ out, int* __restrict__ fb_list,
              ScSummary* __restrict__ sum) {
  if (out_of_domain(sum)) return;
  extern __shared__ __align__(16) uint8_t smem[];
  ScStage* stage = reinterpret_cast<ScStage*>(smem);
  const bool full = sum->masked == 0;
  int bi, bj;
  if (ia == ja) {
    tri_tile(blockIdx.x, (ib - ia + kScTile - 1) / kScTile, (ib - ia + kScTileJ - 1) / kScTileJ, bi, bj);
  } else {
    const int nj = (jb - ja + kScTileJ - 1) / kScTileJ;
    bi = static_cast<int>(blockIdx.x) / nj;
    bj = static_cast<int>(blockIdx.x) % nj;
  }
  const int i0 = ia + bi * kScTile, j0 = ja + bj * kScTileJ;
  const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, wr = (tid >> 6) * 16, wc = ((tid >> 5) & 1) * 16;
  const int W = Tp / 32, r = lane >> 2, kq = lane & 3;
  // Six 16-byte pieces a thread and stage: rows 16 apart, the first four of the
  // tile's rows. Rows past the end are zero.
  const int lrow = tid >> 4, lt = (tid & 15) * 2;
  const double* src = Xc + lt;
  auto load = [&](int s) {
    const uint32_t dst = smem_u32(&stage[s].a[lrow][sc_at(lrow, lt)]);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int g = (q < 4 ? i0 : j0 - kScTile) + lrow + 16 * q;
      const int end = q < 4 ? ib : jb, any = q < 4 ? ia : ja;
      cp_async16(dst + q * 16 * kScK * sizeof(double), src + static_cast<size_t>(g < end ? g : any) * Tp, g < end);
    }
    src += kScK;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  TwoSum acc[2][2][2];
  load(0);
  for (int kc = 0; kc < W; ++kc) {
    if (kc + 1 < W) {
      load((kc + 1) & 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const ScStage& S = stage[kc & 1];
    // The stage's own sums, then one addition each: chains of 8 products round
    // less than chains of T / 4.
    double part[2][2][2] = {};
#pragma unroll
    for (int k = 0; k < kScK; k += 8) {
      double2 b[2];
#pragma unroll
      for (int c = 0; c < 2; ++c)
        b[c] = *reinterpret_cast<const double2*>(&S.b[wc + c * 8 + r][sc_at(r, k + 2 * kq)]);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const double2 a = *reinterpret_cast<const double2*>(&S.a[wr + m * 8 + r][sc_at(r, k + 2 * kq)]);
#pragma unroll
        for (int c = 0; c < 2; ++c) dmma_f64(part[m][c], a.x, b[c].x);
#pragma unroll
        for (int c = 0; c < 2; ++c) dmma_f64(part[m][c], a.y, b[c].y);
      }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (LONG)
            acc[m][c][e].add(part[m][c][e]);
          else
            acc[m][c][e].s += part[m][c][e];
        }
    __syncthreads();  // the stage is refilled two steps on
  }
  ScProducts& P = *reinterpret_cast<ScProducts*>(smem);
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int e = 0; e < 2; ++e) P.xy[wr + m * 8 + r][wc + c * 8 + 2 * kq + e] = acc[m][c][e].value();
  // The counts come after the products: both sets of sums do not fit the 64
  // registers that 4 CTAs per SM leave a thread. Rows 2 rp, 2 rp + 1 and
  // columns cp, cp + 8, cp + 16, cp + 24 are this thread's.
  const int rp = (tid >> 3) * 2, cp = tid & 7;
  uint32_t n[2][4] = {{0u, 0u, 0u, 0u}, {0u, 0u, 0u, 0u}};
  for (int w0 = 0; w0 < W && !full; w0 += kScWords) {
    const int nw = min(W - w0, kScWords);
    __syncthreads();
    for (int row = tid >> 3; row < kScTile + kScTileJ; row += 32) {
      const bool left = row < kScTile;
      const int g = left ? i0 + row : j0 + row - kScTile;
      const bool in = g < (left ? ib : jb);
      for (int w = cp; w < nw; w += 8) P.w[row][w] = in ? bits[static_cast<size_t>(g) * W + w0 + w] : 0u;
    }
    __syncthreads();
    for (int w = 0; w < nw; ++w) {
      const uint32_t x0 = P.w[rp][w], x1 = P.w[rp + 1][w];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t y = P.w[kScTile + cp + 8 * c][w];
        n[0][c] += __popc(x0 & y);
        n[1][c] += __popc(x1 & y);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int c = 0; c < 4; ++c) P.n[rp + m][cp + 8 * c] = full ? static_cast<uint32_t>(T) : n[m][c];
  __syncthreads();
  // a warp finishes 8 x 4 pairs at a time: whole sectors of both triangles
  const int ldi = ib - ia, ldj = jb - ja;
  int gated = 0;
#pragma unroll 1
  for (int q = tid >> 5; q < (kScTile / 8) * (kScTileJ / 4); q += 8) {
    const int li = (q >> 3) * 8 + (lane & 7), lj = (q & 7) * 4 + (lane >> 3);
    const int i = i0 + li, j = j0 + lj;
    if (i >= ib || j >= jb || i > j) continue;
    double v;
    const ColStat& si = st[i];
    if (i == j) {
      // diagonal: 1.0 iff the column's centred sum of squares is usable
      v = (si.count >= 2.0 && si.min != si.max && si.s2 > 0.0 && isfinite(si.s2)) ? 1.0 : dnan();
    } else {
      const ColStat& sj = st[j];
      const double2 x = full ? make_double2(si.s1, si.s2) : ABij[static_cast<size_t>(j - ja) * ldi + (i - ia)];
      const double2 y = full ? make_double2(sj.s1, sj.s2) : ABji[static_cast<size_t>(i - ia) * ldj + (j - ja)];
      const PairResult p =
          finalize_pair(static_cast<double>(P.n[li][lj]), x.x, y.x, P.xy[li][lj], x.y, y.y, si.mean, sj.mean);
      v = p.r;
      gated += p.gate ? 1 : 0;
      if (p.redo) fb_list[atomicAdd(&sum->flagged, 1)] = i * N + j;  // N*N <= INT32_MAX
    }
    out[static_cast<size_t>(i) * N + j] = v;
    out[static_cast<size_t>(j) * N + i] = v;
  }
  gated = __reduce_add_sync(kFull, gated);
  if (lane == 0 && gated != 0) atomicAdd(&sum->gated, gated);
}

// ---------------------------------------------------------------------------
// two-pass fallback of the flagged pairs
// ---------------------------------------------------------------------------
// One warp per pair, a lane every 32nd date: means from sums carried to twice
// the precision (the mean two-pass reference's compensated sums, without
// their serial chain: four dependent FP64 adds, 120 clocks, per date, and
// 672 us for the 6400 flagged pairs of 1218 x 2000), then the centred second
// pass (compensated above T = 2048).
__global__ void __launch_bounds__(128) k_sc_fallback(const double* __restrict__ Xraw, const uint32_t* __restrict__ bits,
                                                     int T, int N, int Tp, const int* __restrict__ fb_list,
                                                     const ScSummary* __restrict__ sum, double* __restrict__ out) {
  if (out_of_domain(sum)) return;
  const int cnt = sum->flagged, W = Tp / 32, lane = static_cast<int>(threadIdx.x & 31);
  const int nw = static_cast<int>(gridDim.x * blockDim.x) >> 5;
  for (int g = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < cnt; g += nw) {
    const int cell = fb_list[g], i = cell / N, j = cell % N;
    const double* xi = Xraw + static_cast<size_t>(i) * Tp + lane;
    const double* xj = Xraw + static_cast<size_t>(j) * Tp + lane;
    const uint32_t* bi = bits + static_cast<size_t>(i) * W;
    const uint32_t* bj = bits + static_cast<size_t>(j) * W;
    int n = 0;
    // a column is constant on the joint dates when all its values equal the
    // first (bit patterns: a column of both zeros has no variance either)
    unsigned long long dx0 = 0ull, dy0 = 0ull;
    long long x0 = 0, y0 = 0;
    TwoSum kx, ky;
#pragma unroll 4
    for (int w = 0; w < W; ++w) {
      const uint32_t m = __ldg(bi + w) & __ldg(bj + w);
      const double x = __ldg(xi + w * 32), y = __ldg(xj + w * 32);
      const long long xb = __double_as_longlong(x), yb = __double_as_longlong(y);
      if (n == 0 && m != 0u) {  // uniform across the warp
        x0 = __shfl_sync(kFull, xb, __ffs(m) - 1);
        y0 = __shfl_sync(kFull, yb, __ffs(m) - 1);
      }
      n += __popc(m);
      if ((m >> lane) & 1u) {
        kx.add(x);
        ky.add(y);
        dx0 |= static_cast<unsigned long long>(xb ^ x0);
        dy0 |= static_cast<unsigned long long>(yb ^ y0);
      }
    }
    kx.warp_total();
    ky.warp_total();
    const bool varies = __any_sync(kFull, dx0 != 0ull) && __any_sync(kFull, dy0 != 0ull);
    double v = dnan();
    if (n >= 2 && varies) {  // uniform across the warp
      const double mx = kx.value() / n, my = ky.value() / n;
      double sxx = 0.0, syy = 0.0, sxy = 0.0;
      if (T > kTwoPassKahanT) {
        TwoSum ka, kb, kc;
#pragma unroll 4
        for (int w = 0; w < W; ++w)
          if (((__ldg(bi + w) & __ldg(bj + w)) >> lane) & 1u) {
            const double dx = __ldg(xi + w * 32) - mx, dy = __ldg(xj + w * 32) - my;
            ka.add(dx * dx);
            kb.add(dy * dy);
            kc.add(dx * dy);
          }
        ka.warp_total();
        kb.warp_total();
        kc.warp_total();
        sxx = ka.value();
        syy = kb.value();
        sxy = kc.value();
      } else {
#pragma unroll 4
        for (int w = 0; w < W; ++w)
          if (((__ldg(bi + w) & __ldg(bj + w)) >> lane) & 1u) {
            const double dx = __ldg(xi + w * 32) - mx, dy = __ldg(xj + w * 32) - my;
            sxx += dx * dx;
            syy += dy * dy;
            sxy += dx * dy;
          }
        sxx = warp_sum(sxx);
        syy = warp_sum(syy);
        sxy = warp_sum(sxy);
      }
      v = safe_pearson(sxy, sxx, syy);
    }
    if (lane == 0) {
      out[static_cast<size_t>(i) * N + j] = v;
      out[static_cast<size_t>(j) * N + i] = v;
    }
  }
}

int sc_chunks(int T) { return (T + kScChunk - 1) / kScChunk; }
int sc_list_cap(int T) { return (T + 16 * sc_chunks(T) + 7) / 8 * 8; }  // whole 16-byte groups, two padded runs a chunk
size_t al256(size_t x) { return (x + 255) & ~size_t(255); }
// columns of one block of pair sums: all of them, or equal blocks of whole tiles
int sc_block(int N) {
  const int nb = (N + kScBlock - 1) / kScBlock;
  return nb <= 1 ? N : ((N + nb - 1) / nb + kScTile - 1) / kScTile * kScTile;
}

// entries of the list of direct pair sums
int sc_direct_cap(int N) {
  const long long bs = sc_block(N);
  return static_cast<int>(std::min<long long>(bs * bs, kScDirect));
}

template <typename TIN>
cudaError_t sc_launch(const TIN* X, const uint8_t* mask, int T, int N, const ScWork& w, double* out, cudaStream_t s) {
  const int Tp = (T + 31) / 32 * 32, nchunk = sc_chunks(T), lcap = sc_list_cap(T);
  uint8_t* m = static_cast<uint8_t*>(w.masks);
  uint32_t* bits = reinterpret_cast<uint32_t*>(m);
  m += al256(static_cast<size_t>(N) * (Tp / 32) * 4);
  uint16_t* list = reinterpret_cast<uint16_t*>(m);
  m += al256(static_cast<size_t>(N) * lcap * 2);
  int* ptr = reinterpret_cast<int*>(m);
  m += al256(static_cast<size_t>(N) * (2 * nchunk + 1) * 4);
  int* invert = reinterpret_cast<int*>(m);
  m += al256(static_cast<size_t>(N) * 4);
  int* direct_list = reinterpret_cast<int*>(m);
  cudaError_t e = cudaMemsetAsync(w.summary, 0, sizeof(ScSummary), s);
  if (e != cudaSuccess) return e;
  k_sc_colstats<TIN><<<(N + 31) / 32, 32 * kStWarps, 0, s>>>(X, mask, T, N, w.st, w.summary);
  k_sc_transpose<TIN><<<dim3(Tp / 32, (N + 31) / 32), dim3(32, 8), 0, s>>>(X, mask, T, N, Tp, w.st, w.xraw, w.xc, bits);
  k_sc_lists<<<(N * 32 + 255) / 256, 256, 0, s>>>(w.xc, bits, T, N, Tp, nchunk, lcap, w.st, list, ptr, invert);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const int tc = std::min(T, kScChunk);
  const size_t psmem = (static_cast<size_t>(tc + 1) * 8 + static_cast<size_t>((tc + 31) / 32 + 1) * 16) * kScRows;
  const size_t gsmem = std::max(2 * sizeof(ScStage), sizeof(ScProducts));
  const bool lng = T > kTwoPassKahanT;
  auto* k_pairsum = lng ? k_sc_pairsum<TIN, true> : k_sc_pairsum<TIN, false>;
  auto* k_gram = lng ? k_sc_gram<true> : k_sc_gram<false>;
  e = cudaFuncSetAttribute(k_pairsum, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(psmem));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(gsmem));
  if (e != cudaSuccess) return e;
  bool first = true;
  auto pairsum = [&](int ia, int ib, int ja, int jb, double2* ab) -> cudaError_t {
    if (!first) {
      const cudaError_t r = cudaMemsetAsync(&w.summary->direct, 0, sizeof(int), s);
      if (r != cudaSuccess) return r;
    }
    first = false;
    const int rows = (ib - ia + kScRows - 1) / kScRows, cols = (jb - ja + 63) / 64;
    // a CTA per SM and row block; few row blocks share out the columns
    const int split = std::max(1, std::min(cols, 148 / rows));
    for (int c = 0; c < nchunk; ++c)
      k_pairsum<<<dim3(rows, split), 1024, psmem, s>>>(X, mask, w.xc, bits, w.st, list, ptr, invert, T, N, Tp, nchunk,
                                                       lcap, c, ia, ib, ja, jb, ib - ia, ab, direct_list,
                                                       w.summary);
    k_sc_direct<<<148 * 8, 256, 0, s>>>(w.xc, bits, T, Tp, ia, ja, ib - ia, direct_list, ab, w.summary);
    return cudaGetLastError();
  };
  const int bs = sc_block(N);
  for (int ia = 0; ia < N; ia += bs)
    for (int ja = ia; ja < N; ja += bs) {
      const int ib = std::min(N, ia + bs), jb = std::min(N, ja + bs);
      const long long ti = (ib - ia + kScTile - 1) / kScTile, tj = (jb - ja + kScTileJ - 1) / kScTileJ;
      double2* ab = w.ab;
      double2* ba = ia == ja ? ab : ab + static_cast<size_t>(bs) * bs;
      if ((e = pairsum(ia, ib, ja, jb, ab)) != cudaSuccess) return e;
      if (ia != ja && (e = pairsum(ja, jb, ia, ib, ba)) != cudaSuccess) return e;
      const long long tiles = ia == ja ? ti * tj - ti * (ti - 1) : ti * tj;
      k_gram<<<static_cast<unsigned>(tiles), 256, gsmem, s>>>(w.xc, bits, w.st, T, N, Tp, ia, ib, ja, jb, ab, ba, out,
                                                                 w.fb_list, w.summary);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
  // grid-stride over the device-side fallback count (no host round trip)
  k_sc_fallback<<<148 * 8, 128, 0, s>>>(w.xraw, bits, T, N, Tp, w.fb_list, w.summary, out);
  return cudaGetLastError();
}

}  // namespace

size_t sc_masks_bytes(int T, int N) {
  const size_t Tp = static_cast<size_t>((T + 31) / 32 * 32);
  return al256(N * (Tp / 32) * 4) + al256(static_cast<size_t>(N) * sc_list_cap(T) * 2) +
         al256(static_cast<size_t>(N) * (2 * sc_chunks(T) + 1) * 4) + al256(static_cast<size_t>(N) * 4) +
         al256(static_cast<size_t>(sc_direct_cap(N)) * 4);
}

size_t sc_pairs_bytes(int N) {
  const size_t bs = static_cast<size_t>(sc_block(N));
  return bs * bs * sizeof(double2) * (bs < static_cast<size_t>(N) ? 2 : 1);
}

cudaError_t launch_stock_corr(const void* X, int dtype, const uint8_t* mask, int T, int N, const ScWork& w, double* out,
                              cudaStream_t s) {
  return dtype == 0 ? sc_launch(static_cast<const float*>(X), mask, T, N, w, out, s)
                    : sc_launch(static_cast<const double*>(X), mask, T, N, w, out, s);
}

}  // namespace fcb
