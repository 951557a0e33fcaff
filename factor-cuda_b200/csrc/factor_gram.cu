// factor_gram.cu -- Gram pass of factor_corr for up to 12 factors, in
// registers, for sm_100a.
//
// A pooled row of F factor values adds one rank-1 update to the F x F moment
// sums.  A thread takes one row at a time and keeps the F (F + 1) / 2 sums of
// x'_i x'_j (x' = value minus the factor's shift, 0 where invalid) and the F
// sums of x'_i in registers: no staging, and one FP64 FMA per pair and row,
// which is what bounds the pass.  The masked sums of a pair (i, j) -- the rows
// n, sum x'_i and sum x'_i^2 where j is valid too -- are the totals less the
// rows on which j is missing.  Rows with no valid factor add nothing, and rows
// with all of them need no correction; the others (one in ten at 12 factors
// with 1 % missing cells) go on a queue per warp in shared memory, and the warp
// adds a full queue to the sums of the factors that its rows miss.  All sums
// are formed in a fixed order.
// Panels of which more than a few cells are missing take the staged pass
// instead (fc_stage_rule, decided on the device: both are launched, and one
// returns at once).
// Per block the same partials come out as from the staged pass
// (fc_gram_body): P[product][i][j] with product 0 n, 1 sum x'_i over rows where
// j is valid, 2 sum x'_i^2 likewise, 3 sum x'_i x'_j.
//
// Measured on a B200, 6.1 M rows x 12 factors f32 with a mask and 1 % missing
// cells: 143 us (the staged pass took 673; memory alone 46, the FP64 sums 35),
// factor_corr 1405 -> 219 us a call with the sampled shift and the two-pass
// recomputation kept for sums that fall short.  What bounds it is the issue of
// 300 instructions per 32 rows (102 FP64; the rest converts, tests and selects)
// and the queue, at 8 warps per SM of 255 registers: the 90 sums of a thread
// leave room for no more.
#include "corr_common.cuh"
#include "fcb_kernels.h"

namespace fcb {
namespace {

constexpr int kRegThreads = 128, kRegWarps = kRegThreads / 32;
constexpr int kQueue = 96;   // rows a warp's queue holds: flushed above 64, up to 32 arrive at a time

template <int FP>
struct RegShape {
  static constexpr int kPairs = FP * (FP + 1) / 2, kSums = kPairs + FP;
};

// One warp's shared memory.
template <int FP>
struct RegWarp {
  double2 row[kQueue][FP / 2];  // centred values, 0 where invalid
  double2 c[2][FP][FP];         // [half][j][i]: sum x'_i, sum x'_i^2 over the rows that miss j
  uint32_t cn[2][FP][FP];       // rows where i is valid and j is not; [j][j]: rows that miss j
  uint32_t valid[kQueue];
};

// Sums of M values over the warp's lanes, spread over the lanes: each step
// trades one half of the values for the other lanes' share of the other half.
// On return a lane holds the totals of values base .. base + len - 1 in v[0 ..].
template <int M, int O, int FULL>
FCB_DEV void spread_sums(double (&v)[FULL], int& base, int& len) {
  if constexpr (O > 0) {
    constexpr int H = (M + 1) / 2;
    const bool up = (lane_id() & O) != 0;
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const double hi = H + k < M ? v[H + k] : 0.0, lo = v[k];
      const double other = __shfl_xor_sync(kFull, up ? lo : hi, O);
      v[k] = (up ? hi : lo) + other;
    }
    base += up ? H : 0;
    len = up ? max(0, len - H) : min(len, H);
    spread_sums<H, O / 2, FULL>(v, base, len);
  }
}
template <int M>
constexpr int spread_len() {
  int m = M;
  for (int o = 16; o > 0; o >>= 1) m = (m + 1) / 2;
  return m;
}

// Adds the n queued rows to the warp's corrections: each half-warp takes every
// other row, lane i the factor i, and adds it to the sums of the factors that
// the row misses (one, as a rule).
template <int FP>
FCB_DEV void flush_queue(RegWarp<FP>& w, int n, uint32_t all) {
  const int h = static_cast<int>(lane_id() >> 4), i = static_cast<int>(lane_id() & 15u);
  __syncwarp();
  if (i < FP) {
    const double* rows = reinterpret_cast<const double*>(w.row);
    uint32_t valid = h < n ? w.valid[h] : all;
    double x = h < n ? rows[h * FP + i] : 0.0;
    for (int r = h; r < n; r += 2) {
      const uint32_t v = valid;
      const double y = x;
      if (r + 2 < n) {
        valid = w.valid[r + 2];
        x = rows[(r + 2) * FP + i];
      }
      for (uint32_t m = all & ~v; m != 0u; m &= m - 1u) {
        const int j = __ffs(m) - 1;
        double2 c = w.c[h][j][i];
        c.x += y;
        c.y = fma(y, y, c.y);
        w.c[h][j][i] = c;
        w.cn[h][j][i] += i == j ? 1u : (v >> i) & 1u;
      }
    }
  }
  __syncwarp();
}

// The rows of a warp's next kStages - 1 steps are on their way to shared memory
// (cp.async) while it works on the current ones: two warps per SM quadrant hide
// no memory latency by themselves.  A lane copies and reads its own row only, so
// no barrier is needed.  Element (r, f) is X[r * sr + f * sf].
constexpr int kStages = 4;

template <typename TIN, int FP, bool ROWS>
struct RowRing {
  static constexpr int VL = 16 / static_cast<int>(sizeof(TIN));  // values per 16 bytes
  static constexpr bool kWhole = ROWS && FP % VL == 0;           // 16-byte pieces when F == FP and X is aligned
  static constexpr size_t kStage = size_t(32) * FP * sizeof(TIN), kBytes = kStages * kStage;
  const TIN* X;
  long long sf, r1;
  int F;
  bool pieces;
  uint8_t* mem;  // this lane's first piece or value of stage 0

  FCB_DEV RowRing(const TIN* X_, long long sf_, long long r1_, int F_, uint8_t* ring)
      : X(X_), sf(sf_), r1(r1_), F(F_) {
    pieces = kWhole && F == FP && (reinterpret_cast<uintptr_t>(X) & 15u) == 0;
    mem = ring + lane_id() * (pieces ? 16u : static_cast<unsigned>(sizeof(TIN)));
  }
  // Row r into stage s (nothing beyond the last row: its values are not used).
  FCB_DEV void fetch(int s, long long r) {
    if (r < r1) {
      const uint32_t dst = smem_u32(mem + s * kStage);
      if (kWhole && pieces) {
        const TIN* p = X + r * F;
#pragma unroll
        for (int c = 0; c < FP / VL; ++c)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + c * 512), "l"(p + c * VL) : "memory");
      } else {
        const TIN* p = ROWS ? X + r * F : X + r;
#pragma unroll
        for (int f = 0; f < FP; ++f)
          if (f < F)
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                             dst + f * 32 * static_cast<int>(sizeof(TIN))),
                         "l"(p + (ROWS ? static_cast<long long>(f) : f * sf)), "n"(sizeof(TIN))
                         : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // The values of the oldest row in flight, which is in stage s.
  FCB_DEV void take(int s, TIN (&x)[FP]) const {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    const uint8_t* src = mem + s * kStage;
    if (kWhole && pieces) {
#pragma unroll
      for (int f = 0; f < FP; f += VL) {
        const uint4 q = *reinterpret_cast<const uint4*>(src + f / VL * 512);
        if constexpr (sizeof(TIN) == 4) {
          x[f] = __uint_as_float(q.x);
          if (f + 1 < FP) x[f + 1] = __uint_as_float(q.y);
          if (f + 2 < FP) x[f + 2] = __uint_as_float(q.z);
          if (f + 3 < FP) x[f + 3] = __uint_as_float(q.w);
        } else {
          x[f] = __hiloint2double(static_cast<int>(q.y), static_cast<int>(q.x));
          if (f + 1 < FP) x[f + 1] = __hiloint2double(static_cast<int>(q.w), static_cast<int>(q.z));
        }
      }
    } else {
#pragma unroll
      for (int f = 0; f < FP; ++f)
        x[f] = f < F ? *reinterpret_cast<const TIN*>(src + f * 32 * sizeof(TIN)) : TIN(0);
    }
  }
};

// The warps' queues and their sums, before the rings.
template <int FP>
__host__ __device__ constexpr size_t reg_sums_bytes() {
  return (kRegWarps * (sizeof(RegWarp<FP>) + (RegShape<FP>::kSums + 1) * sizeof(double)) + 15) / 16 * 16;
}

FCB_DEV bool row_finite(float x) { return fabsf(x) <= 3.402823466e38f; }
FCB_DEV bool row_finite(double x) { return KeyOf<double>::finite(x); }

// Rows [bx * rows_per_block, ...) of the pool into part + bx * 4 Fp^2.
template <typename TIN, int FP, bool ROWS>
FCB_DEV void gram_reg_body(const TIN* __restrict__ X, const uint8_t* __restrict__ mask, long long R, int F,
                           long long sf, int Fp, long long rows_per_block, const FcColStat* __restrict__ st,
                           double* __restrict__ part, int bx, uint8_t* smem) {
  using S = RegShape<FP>;
  if (st[0].staged != 0) return;  // uniform: the staged pass writes the partials
  RegWarp<FP>* warps = reinterpret_cast<RegWarp<FP>*>(smem);
  const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, wi = tid >> 5;
  RegWarp<FP>& w = warps[wi];
  for (int e = lane; e < 2 * FP * FP; e += 32) {
    (&w.c[0][0][0])[e] = make_double2(0.0, 0.0);
    (&w.cn[0][0][0])[e] = 0u;
  }
  const uint32_t all = (1u << F) - 1u;
  double shift[FP];
#pragma unroll
  for (int f = 0; f < FP; ++f) shift[f] = f < F ? st[f].mean : 0.0;
  double acc[S::kSums];
#pragma unroll
  for (int k = 0; k < S::kSums; ++k) acc[k] = 0.0;
  uint32_t rows = 0u;  // rows with some valid factor (this warp's, uniform)
  int queued = 0;
  const long long r0 = bx * rows_per_block, r1 = min(R, r0 + rows_per_block);
  RowRing<TIN, FP, ROWS> ring(X, sf, r1, F,
                              smem + reg_sums_bytes<FP>() + wi * RowRing<TIN, FP, ROWS>::kBytes);
  auto mask_of = [&](long long r) { return r < r1 ? (mask != nullptr ? __ldg(mask + r) : 1u) : 0u; };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) ring.fetch(s, r0 + tid + s * kRegThreads);
  uint32_t next_mask = mask_of(r0 + tid);
  int stage = 0;
  for (long long rb = r0; rb < r1; rb += kRegThreads) {
    const uint32_t cur_mask = next_mask;
    next_mask = mask_of(rb + kRegThreads + tid);
    uint32_t v = 0u;
    double x[FP];
    {
      TIN raw[FP];
      ring.take(stage, raw);
      ring.fetch((stage + kStages - 1) % kStages, rb + tid + (kStages - 1) * kRegThreads);
      stage = (stage + 1) % kStages;
#pragma unroll
      for (int f = 0; f < FP; ++f) {
        const bool ok = f < F && cur_mask != 0u && row_finite(raw[f]);
        x[f] = ok ? static_cast<double>(raw[f]) - shift[f] : 0.0;
        v |= ok ? 1u << f : 0u;
      }
    }
    const unsigned some = __ballot_sync(kFull, v != 0u);
    rows += __popc(some);
    if (some == 0u) continue;  // uniform across the warp
#pragma unroll
    for (int i = 0, k = 0; i < FP; ++i)
#pragma unroll
      for (int j = i; j < FP; ++j, ++k) acc[k] = fma(x[i], x[j], acc[k]);
#pragma unroll
    for (int f = 0; f < FP; ++f) acc[S::kPairs + f] += x[f];
    const unsigned q = __ballot_sync(kFull, v != 0u && v != all);
    if (q != 0u) {
      if ((q >> lane) & 1u) {
        const int at = queued + __popc(q & lanemask_lt());
#pragma unroll
        for (int f = 0; f < FP; f += 2) w.row[at][f / 2] = make_double2(x[f], x[f + 1]);
        w.valid[at] = v;
      }
      queued += __popc(q);
      if (queued > kQueue - 32) {
        flush_queue<FP>(w, queued, all);
        queued = 0;
      }
    }
  }
  flush_queue<FP>(w, queued, all);
  // the warps' sums meet in shared memory, in warp order
  constexpr int L = spread_len<S::kSums>(), TS = S::kSums + 1;
  double* t0 = reinterpret_cast<double*>(smem + kRegWarps * sizeof(RegWarp<FP>));
  int base = 0, len = S::kSums;
  spread_sums<S::kSums, 16, S::kSums>(acc, base, len);
#pragma unroll
  for (int k = 0; k < L; ++k)
    if (k < len) t0[wi * TS + base + k] = acc[k];
  if (lane == 0) t0[wi * TS + S::kSums] = static_cast<double>(rows);
  __syncthreads();
  double* P = part + static_cast<size_t>(bx) * 4 * Fp * Fp;
  for (int e = tid; e < Fp * Fp; e += kRegThreads) {
    const int i = e / Fp, j = e % Fp;
    double n = 0.0, sx = 0.0, sx2 = 0.0, sxy = 0.0;
    if (i < F && j < F) {
      const int a = i < j ? i : j, b = i < j ? j : i;
      const int kij = a * FP - a * (a - 1) / 2 + (b - a), kii = i * FP - i * (i - 1) / 2;
      for (int q = 0; q < kRegWarps; ++q) {
        const RegWarp<FP>& u = warps[q];
        const double* t = t0 + q * TS;
        n += t[S::kSums] - static_cast<double>(u.cn[0][i][i] + u.cn[1][i][i]);
        if (i != j) n -= static_cast<double>(u.cn[0][j][i] + u.cn[1][j][i]);
        sxy += t[kij];
        sx += t[S::kPairs + i] - (u.c[0][j][i].x + u.c[1][j][i].x);
        sx2 += t[kii] - (u.c[0][j][i].y + u.c[1][j][i].y);
      }
    }
    P[(0 * Fp + i) * Fp + j] = n;
    P[(1 * Fp + i) * Fp + j] = sx;
    P[(2 * Fp + i) * Fp + j] = sx2;
    P[(3 * Fp + i) * Fp + j] = sxy;
  }
}

template <typename TIN, int FP>
constexpr size_t reg_smem() {
  return reg_sums_bytes<FP>() + kRegWarps * RowRing<TIN, FP, true>::kBytes;
}

template <typename TIN, int FP, bool ROWS>
__global__ void __launch_bounds__(kRegThreads, 2)
    k_fc_gram_reg(const TIN* __restrict__ X, const uint8_t* __restrict__ mask, long long R, int F, long long sf, int Fp,
                  long long rows_per_block, const FcColStat* __restrict__ st, double* __restrict__ part) {
  extern __shared__ __align__(16) uint8_t smem[];
  gram_reg_body<TIN, FP, ROWS>(X, mask, R, F, sf, Fp, rows_per_block, st, part, blockIdx.x, smem);
}

// Many factor-plane panels: a block finds its panel by binary search.
template <typename TIN, int FP>
__global__ void __launch_bounds__(kRegThreads, 2)
    k_fcb_gram_reg(const FcBatchPanel* __restrict__ P, const int* __restrict__ off, int np) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int b = static_cast<int>(blockIdx.x);
  int lo = 0, hi = np - 1;  // largest p with off[p] <= b
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= b) lo = mid; else hi = mid - 1;
  }
  const FcBatchPanel& q = P[lo];
  gram_reg_body<TIN, FP, false>(static_cast<const TIN*>(q.X), q.mask, q.R, q.F, q.R, q.Fp, q.rpb_reg, q.w.colstat,
                                q.w.gram, b - off[lo], smem);
}

template <typename TIN, int FP>
cudaError_t reg_launch(const TIN* X, const uint8_t* mask, long long R, int F, bool rows, long long sf, int Fp,
                       long long rpb, int nblk, const FcColStat* st, double* part, cudaStream_t s) {
  auto go = [&](auto kernel) -> cudaError_t {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(reg_smem<TIN, FP>()));
    if (e != cudaSuccess) return e;
    kernel<<<nblk, kRegThreads, reg_smem<TIN, FP>(), s>>>(X, mask, R, F, sf, Fp, rpb, st, part);
    return cudaGetLastError();
  };
  return rows ? go(k_fc_gram_reg<TIN, FP, true>) : go(k_fc_gram_reg<TIN, FP, false>);
}

template <typename TIN>
cudaError_t reg_by_width(const TIN* X, const uint8_t* mask, long long R, int F, bool rows, long long sf, int Fp,
                         long long rpb, int nblk, const FcColStat* st, double* part, cudaStream_t s) {
  if (F <= 4) return reg_launch<TIN, 4>(X, mask, R, F, rows, sf, Fp, rpb, nblk, st, part, s);
  if (F <= 6) return reg_launch<TIN, 6>(X, mask, R, F, rows, sf, Fp, rpb, nblk, st, part, s);
  if (F <= 8) return reg_launch<TIN, 8>(X, mask, R, F, rows, sf, Fp, rpb, nblk, st, part, s);
  if (F <= 10) return reg_launch<TIN, 10>(X, mask, R, F, rows, sf, Fp, rpb, nblk, st, part, s);
  return reg_launch<TIN, 12>(X, mask, R, F, rows, sf, Fp, rpb, nblk, st, part, s);
}

}  // namespace

cudaError_t launch_fc_gram_reg(const void* X, int dtype, const uint8_t* mask, long long R, int F, long long sr,
                               long long sf, int Fp, long long rows_per_block, int nblk, const FcColStat* st,
                               double* part, cudaStream_t s) {
  if (F > kFcRegMaxF || !((sr == F && sf == 1) || sr == 1)) return cudaErrorInvalidValue;
  const bool rows = sr != 1 || sf == 1;  // (one factor: both layouts are the same)
  return dtype == 0 ? reg_by_width(static_cast<const float*>(X), mask, R, F, rows, sf, Fp, rows_per_block, nblk, st,
                                   part, s)
                    : reg_by_width(static_cast<const double*>(X), mask, R, F, rows, sf, Fp, rows_per_block, nblk, st,
                                   part, s);
}

int fc_reg_kind(int F) { return F <= 4 ? 0 : F <= 6 ? 1 : F <= 8 ? 2 : F <= 10 ? 3 : 4; }

cudaError_t launch_fc_gram_reg_batch(int kind, int dtype, const FcBatchPanel* panels, const int* off, int np, int blocks,
                                     cudaStream_t s) {
  auto go = [&](auto kernel, size_t smem) -> cudaError_t {
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    kernel<<<blocks, kRegThreads, smem, s>>>(panels, off, np);
    return cudaGetLastError();
  };
  const bool f32 = dtype == 0;
  switch (kind) {
    case 0: return f32 ? go(k_fcb_gram_reg<float, 4>, reg_smem<float, 4>()) : go(k_fcb_gram_reg<double, 4>, reg_smem<double, 4>());
    case 1: return f32 ? go(k_fcb_gram_reg<float, 6>, reg_smem<float, 6>()) : go(k_fcb_gram_reg<double, 6>, reg_smem<double, 6>());
    case 2: return f32 ? go(k_fcb_gram_reg<float, 8>, reg_smem<float, 8>()) : go(k_fcb_gram_reg<double, 8>, reg_smem<double, 8>());
    case 3: return f32 ? go(k_fcb_gram_reg<float, 10>, reg_smem<float, 10>()) : go(k_fcb_gram_reg<double, 10>, reg_smem<double, 10>());
    default: return f32 ? go(k_fcb_gram_reg<float, 12>, reg_smem<float, 12>()) : go(k_fcb_gram_reg<double, 12>, reg_smem<double, 12>());
  }
}

}  // namespace fcb
