// fcb_kernels.h -- internal launch interface between the kernel translation
// units and the C-ABI host drivers (capi.cu).  Not part of the public ABI.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace fcb {

// Largest cross-section the shared-memory rank kernels take (u16 column ids,
// 1024 threads x 16 items).  Larger N goes through the global-memory path.
constexpr int kSmemRankCap = 16384;
// CDF network for learned splitters: hidden width, parameter count, table knots.
constexpr int kCdfHidden = 32;
constexpr int kCdfParams = 1 + 1 * 32 + 32 + 32 * 32 + 32 + 32;  // W1,b1,W2,b2,w3,b3 = 1153
constexpr int kCdfKnots = 1024;
// Share of the buckets the tabulated CDF spreads uniformly over its knots.
constexpr float kCdfLinearShare = 0.03f;
constexpr size_t kMaxSmemPerBlock = 227 * 1024;

struct ScanOut {
  float* out[4];  // group g output panel (T,N) or nullptr when the group is inactive
};

// Default largest bucket the learned rank path ranks itself.  A bucket of b
// cells costs each of its cells b comparisons; above the cap the section goes
// to the plain kernel after the learned one (at 1218 x 5000 x 12 a cap of 64
// sent one section in 14616 there, 256 none).
constexpr int kLearnCapDefault = 256;

template <typename TF, typename TR>
struct RankIcArgs {
  const TF* X;              // (F,T,N) factor panels
  const TR* R;              // (T,N) forward returns
  const uint8_t* fmask;     // (T,N) factor mask or nullptr
  const uint8_t* rmask;     // (T,N) forward-return mask or nullptr
  int F, T, N, min_valid;
  float* ranks_out;         // (F,T,N) cs_rank ranks (valid = finite(f) & fmask) or nullptr
  double* ic_out;           // (F,T)
  double* rank_f_out;       // (F,T,N) joint-set ranks, 0 elsewhere, or nullptr
  double* rank_r_out;       // (F,T,N) joint-set ranks of the returns, or nullptr
  // learned splitters (used by the LEARNED instantiation only)
  const float* cdf_table;   // (F, kCdfKnots) tabulated monotone CDF per factor
  const float* cdf_zrange;  // (F, 2) grid range [lo, hi] in standardised units
  int learn_cap;            // largest bucket the learned path accepts
  int* learn_stats;         // (F,T,4): outcome, largest bucket, sum of squared bucket sizes, m; or nullptr
  int ic_ld;                // row stride of ic_out (0 = T)
};

struct ColStat {  // one stock_corr column
  double count, mean, min, max, min_abs, max_abs, s2, s1;
};
// stock_corr: what the device knows of the whole panel (zeroed first).
struct ScSummary {
  unsigned long long max_abs;      // bits of the largest |x| over the valid cells
  unsigned long long min_abs_inv;  // inverted bits of the smallest nonzero |x| (0: none)
  int masked;                      // some cell is invalid
  int flagged;                     // pairs that the two-pass fallback recomputes
  int gated;                       // pairs that fail the cancellation gate
  int direct;                      // pair sums to be formed over the joint dates (of one block of columns)
};
struct ScWork {
  double *xraw, *xc;  // (N,Tp) column-major values, as they are and centred; Tp = T rounded to 32
  void* masks;        // sc_masks_bytes: validity bits, date lists
  double2* ab;        // sc_pairs_bytes: pair sums
  ColStat* st;        // [N]
  ScSummary* summary;
  int* fb_list;       // [N (N-1) / 2]
};
size_t sc_masks_bytes(int T, int N);
size_t sc_pairs_bytes(int N);
// (N,N) correlations of a (T,N) panel into out (untouched when the panel is
// out of the domain, see the summary).
cudaError_t launch_stock_corr(const void* X, int dtype, const uint8_t* mask, int T, int N, const ScWork& w, double* out,
                              cudaStream_t s);
// Column statistics of the sampled rows.  In the entries of factor 0: rows,
// those with some valid factor; staged, the form of the Gram pass (fc_stage_rule).
struct FcColPart {
  double count, s, c, rows;
};
struct FcColStat {
  double count, mean;
  int staged;
};
struct FcWork {
  int nblk_cols, nblk_gram;
  FcColPart* colpart;  // [nblk_cols][F]
  FcColStat* colstat;  // [F]
  double* gram;        // [nblk_gram][4][Fp][Fp]
  int* fb_list;        // [F*F]
  int* fb_count;       // [2]: flagged pairs; column blocks that are done
  double* fb_part;     // fc_fb_part_doubles(R, F) doubles, or nullptr (single-block fallback)
};
// Up to this many factors the Gram pass keeps its sums in registers
// (factor_gram.cu).
constexpr int kFcRegMaxF = 12;
// Row blocks of factor_corr's Gram pass: staged panels of F <= 32 fill the SMs
// several times over (their tile is small); the register form takes two per SM
// of them (a block's final reduction costs as much as about ten of its rows per
// thread).  The same count everywhere keeps single-panel and batched results
// identical.
inline int fc_gram_blocks(long long R, int F) {
  const long long cap = F <= 32 ? 888 : 148;
  long long nb = R / 1024;
  if (nb < 1) nb = 1;
  return static_cast<int>(nb < cap ? nb : cap);
}
__host__ __device__ inline int fc_reg_blocks(int gram_blocks) { return gram_blocks < 296 ? gram_blocks : 296; }
// Column statistics come from a sample of the rows, every fc_col_stride-th: the
// mean is only the shift of the centred sums.  Up to kFcRegMaxF factors about
// 16384 rows, at most kFcColRows a block; above, where the Gram pass takes far
// longer, 262144: f32 values less one shift end in the same bits, so that the
// additions of a staged chain all round the same way and sum x' is off by a share
// of the rows; in a covariance that counts with the shift's distance from the
// mean (200 x 700 x 16 f32, independent factors: rms error 1.5e-18 with all rows,
// 2.0e-18 with 16384).
constexpr int kFcColRows = 256;
__host__ __device__ inline long long fc_col_stride(long long R, int F) {
  const long long ms = R / (F <= kFcRegMaxF ? 16384 : 262144);
  return ms > 1 ? ms : 1;
}
__host__ __device__ inline long long fc_col_rows(long long R, int F) {
  const long long ms = fc_col_stride(R, F);
  return (R + ms - 1) / ms;
}
inline int fc_col_blocks(long long R, int F) {
  const long long nb = fc_col_rows(R, F) / 128, cap = F <= kFcRegMaxF ? 148 : 296;
  return static_cast<int>(nb < 1 ? 1 : nb < cap ? nb : cap);
}
// Row blocks per flagged pair of the multi-block fallback (at most
// kFcFbMaxNblk), and the partials buffer it needs (doubles): kFcFbPartDoubles
// per pair and block plus 4 per pair.
constexpr int kFcFbMaxNblk = 64;
constexpr int kFcFbPartDoubles = 9;
int fc_fb_nblk(long long R, int F);
size_t fc_fb_part_doubles(long long R, int F);
// One factor-plane panel (rows at unit stride, F planes of R rows) of a
// batched factor_corr launch, with its single-panel launch geometry.
struct FcBatchPanel {
  const void* X;
  const uint8_t* mask;
  long long R;
  int F, Fp;
  long long rpb_cols, rpb_gram, rpb_reg;  // rows per column / staged / register Gram block
  int tasks_total, tasks_per_block, ytiles;
  int maxpairs, fb_nblk, fb_ysl;  // flagged-pair slots, fallback row blocks, pair slots per row block
  int large;                      // 1: multi-block fallback, 0: one block per flagged pair
  FcWork w;
  double* out;
};
// Kinds of batched grid (prefix offsets are kept per kind).
constexpr int kFcbCols = 0, kFcbColFinal = 1, kFcbGram = 2, kFcbFinal = 3, kFcbFbPass = 4, kFcbFbPair = 5,
              kFcbSmall = 6, kFcbReg = 7, kFcRegKinds = 5,  // kFcbReg: the register form, one kind per fc_reg_kind
              kFcbLow = kFcbReg + kFcRegKinds, kFcbGrids = kFcbLow + 1;  // kFcbLow: its panels, staged (fc_stage_rule)
FcBatchPanel fc_batch_panel(const void* X, const uint8_t* mask, long long R, int F, const FcWork& w, double* out);
// Blocks the panel contributes to each kind of batched grid.
void fc_batch_grids(const FcBatchPanel& q, int (&blocks)[kFcbGrids]);
// Up to ten launches for every panel: d_off holds kFcbGrids runs of np + 1
// prefix offsets, total the grid sizes (host), gram_smem the largest Gram
// staging of the panels; results equal launch_factor_corr_strided's per panel.
cudaError_t launch_factor_corr_batch(const FcBatchPanel* d_panels, int np, const int* d_off, const int* total,
                                     int dtype, size_t gram_smem, cudaStream_t s);

// factor_gram.cu: the register form of the Gram pass, F <= kFcRegMaxF, (T,N,F)
// rows (sr = F, sf = 1) or factor planes (sr = 1); partials as the staged form's.
cudaError_t launch_fc_gram_reg(const void* X, int dtype, const uint8_t* mask, long long R, int F, long long sr,
                               long long sf, int Fp, long long rows_per_block, int nblk, const FcColStat* st,
                               double* part, cudaStream_t s);
int fc_reg_kind(int F);  // 0..4: the width its panel runs at
cudaError_t launch_fc_gram_reg_batch(int kind, int dtype, const FcBatchPanel* panels, const int* off, int np, int blocks,
                                     cudaStream_t s);

// rank_plane.cu; rank_kernels.cu (one factor with learned splitters)
cudaError_t launch_cs_rank(const float* X, const uint8_t* mask, int T, int N, int desc, float* out,
                           int* status, cudaStream_t st);
cudaError_t launch_param_scan(const float* X, const uint8_t* mask, int T, int N, ScanOut outs, int* status,
                              cudaStream_t st);
size_t rank_ic_learned_smem(int N);
cudaError_t launch_rank_ic_learned(const RankIcArgs<float, float>& a, int* status, cudaStream_t st);

// rank_slices.cu: cs_rank of rows above kSmemRankCap, without scratch, for the
// calls that cs_rank_by_slices names; the others, and those in place, sort in
// global memory, one CTA a row.  A row costs the slices the reads of all its
// slices, whatever its values, and the sort a pass for each digit in which its
// values differ: full SMs of tied rows are sorted sooner (us, sort against slices,
// values in 30 steps: 300 x 17000 227 / 168, 148 x 20000 98 / 105, 64 x 40000 172 /
// 163, 148 x 40000 187 / 316, 64 x 60000 257 / 288; smooth: 469 / 165, 192 / 97,
// 350 / 142, 384 / 329, 522 / 270).
constexpr int kSliceMaxN = 65536;
inline bool cs_rank_by_slices(int T, int N) {
  return N > kSmemRankCap && (N <= 18432 || (T <= 64 && N <= 40960) || (T <= 32 && N <= kSliceMaxN));
}
cudaError_t launch_cs_rank_slices(const float* X, const uint8_t* mask, int T, int N, int desc, float* out,
                                  cudaStream_t st);

// rank_ic_pair.cu: rank + IC of one factor row against one returns row per CTA
// (any F); true when its shared-memory kernel takes N for these dtypes.
template <typename TF, typename TR>
bool rank_ic_fits(int N);
template <typename TF, typename TR>
cudaError_t launch_rank_ic(const RankIcArgs<TF, TR>& a, cudaStream_t st);

// cdf_mlp.cu
size_t cdf_train_smem();
cudaError_t launch_cdf_features(const float* X, const float* ranks, int F, int T, int N, int t0, int tcount, int S,
                                float2* samples, cudaStream_t s);
cudaError_t launch_cdf_train(float* params, float* adam, const float2* samples, int F, int nsamp, int steps, float lr,
                             int step0, float* loss_out, cudaStream_t s);
cudaError_t launch_cdf_grad(const float* params, const float* z, const float* u, int n, float* grad, float* loss,
                            cudaStream_t s);
cudaError_t launch_cdf_tabulate(const float* params, const float2* samples, int F, int nsamp, float* zrange,
                                float* table, bool linear, cudaStream_t s);

// Operands of the stock_corr precision forms, K-major (Np rows x Tp dates),
// column-centred; unused members are nullptr.
struct PrecOperands {
  __nv_bfloat16* h;  // [7][Np][Tp] bf16: mask, three limbs of x', three limbs of x'^2 (or nullptr)
  int np;            // Np (row count of each plane)
  float *x32, *q32, *m32;        // FP32 x', x'^2, mask
};

// corr_tc.cu
constexpr int kPrecTileTcM = 128, kPrecTileTcN = 64, kPrecTileFp32 = 64;
size_t prec_tc_smem();
// Tile list of a precision form (mode 0 BF16x3, 1 FP32) built on the device;
// prec_tile_count gives its length.
int prec_tile_count(int mode, int N);
cudaError_t launch_prec_tiles(int mode, int N, int2* tiles, cudaStream_t s);
// Column means (two steps; part: prec_colmean_chunks(T) * Np double2 scratch)
// and the split operands.
int prec_colmean_chunks(int T);
cudaError_t launch_prec_prep(const float* X, const uint8_t* mask, int T, int N, int Np, int Tp, float* mu,
                             double2* part, PrecOperands op, cudaStream_t s);
cudaError_t launch_corr_bf16x3(const PrecOperands& op, const int2* tiles, int ntiles, int N, int Np, int Tp,
                               double* out, int* status, cudaStream_t s);
cudaError_t launch_corr_fp32(const PrecOperands& op, const int2* tiles, int ntiles, int N, int Tp, double* out,
                             cudaStream_t s);

// corr_kernels.cu
// max |x| and min nonzero |x| over the valid cells (finite, mask true) of a
// factor_corr panel, as IEEE bit patterns in ext[0] / ext[1] (0 and +inf when
// no cell is valid).  planes = 0: (R,F) rows; planes = 1: F planes of R rows.
cudaError_t launch_corr_domain(const void* X, int dtype, const uint8_t* mask, long long R, int F, int planes,
                               unsigned long long* ext, cudaStream_t s);
size_t fc_gram_smem(int Fp, int tasks_per_block, int elem_bytes);
// Work split of the Gram pass for Fp (factors rounded to 4): tiles or tile
// units in all, per block (blockIdx.y), and the blocks along y.
void fc_gram_plan(int Fp, int* tasks_total, int* tasks_per_block, int* ytiles);
cudaError_t launch_factor_corr(const void* X, int dtype, const uint8_t* mask, long long R, int F, FcWork& w,
                               double* out, uint8_t* flags, cudaStream_t s);
// Returns of each date prepared once for the per-(date, factor) rank + IC
// kernels (rank_ic_bucket.cu).  word[t*ld + i]: bits 0-13 the position of
// stock i in the stable ascending order of the date's valid returns, bits
// 14-27 the position where its tie group starts, bit 28 returns valid, bit 29
// factor mask (N <= 16384; rows 16-byte aligned).  fb_count / fb_items: the
// sections (t*F + f) the learned kernel hands back.
struct RicPrep {
  uint32_t* word;
  int* fb_count;
  int* fb_items;
  int ld;
};
// A device list of sections (item ids) that the learned kernel hands back.
struct RicList {
  int* count;
  int* items;
};
size_t ric_prep_bytes(int T, int N, int F);
RicPrep ric_prep_carve(void* base, int T, int N, int F);
// True when the per-(date, factor) kernels take N (f32 factors and returns).
bool ric_items_fit(int N);
// Batched form: the panels of one size variant (variant v serves N up to
// ric_variant_cap(v)) in one returns launch and one rank launch; items are a
// panel's dates (returns pass) or its (date, factor) sections, in panel order.
constexpr int kRicVariants = 9;
int ric_variant_cap(int variant);
struct RicPanel {
  RankIcArgs<float, float> a;
  RicPrep rp;
};
struct RicBatchVariant {
  const RicPanel* panels;  // device, np entries
  const int* off_dates;    // device, exclusive prefix of the panels' T (np entries)
  const int* off_items;    // device, exclusive prefix of the panels' T*F (np entries)
  int np, dates, items, maxN;
};
cudaError_t launch_rank_ic_prep_batch(int variant, const RicBatchVariant& v, cudaStream_t st);
cudaError_t launch_rank_ic_items_batch(int variant, const RicBatchVariant& v, cudaStream_t st);
// Rank + IC of F >= 1 f32 factor panels against one f32 returns panel: the
// returns pass, then one CTA per (date, factor) -- value-spread buckets, or
// learned splitters (with the former taking the sections they hand back).
// Requires rank_f_out == rank_r_out == nullptr.
cudaError_t launch_rank_ic_items(const RankIcArgs<float, float>& a, RicPrep rp, bool learned, cudaStream_t st);
// Stream-ordered scratch for the entry points that take no workspace: a
// library-private memory pool per device that keeps freed blocks cached.
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s);
cudaError_t scratch_free(void* p, cudaStream_t s);
// Per-device status word of the asynchronous entry points (capi.cu).
cudaError_t dev_status_sink(int** out);
// One block waiting (at most max_polls polls) on a barrier that completes
// only if `arrive`; sets *status on timeout (selftest.cu).
cudaError_t launch_wait_probe(bool arrive, uint32_t max_polls, int* status, cudaStream_t s);
// Global-memory rank path for cross-sections the shared-memory kernels cannot
// hold (rank_global.cu).  kind 0 cs_rank, 1 parameter_scan, 2 rank+IC: bytes
// of scratch one date needs; the launchers process dates in chunks that fit
// the scratch they are given (at least one date's worth).
size_t rank_global_bytes_per_date(int kind, int N, int F, int ksz_f, int ksz_r);
cudaError_t launch_cs_rank_global(const float* X, const uint8_t* mask, int T, int N, int desc, float* out,
                                  uint8_t* scratch, size_t bytes, cudaStream_t s);
cudaError_t launch_param_scan_global(const float* X, const uint8_t* mask, int T, int N, ScanOut outs,
                                     uint8_t* scratch, size_t bytes, cudaStream_t s);
template <typename TF, typename TR>
cudaError_t launch_rank_ic_global(const RankIcArgs<TF, TR>& a, uint8_t* scratch, size_t bytes, cudaStream_t s);
// True when the one-factor learned kernel takes N.
inline bool rank_ic_learned_fits(int N) {
  return N <= kSmemRankCap && rank_ic_learned_smem(N) <= kMaxSmemPerBlock;
}
inline size_t rank_global_scratch(size_t per_date, int T) {
  size_t b = per_date * static_cast<size_t>(T);
  if (b > (size_t(1) << 30)) b = size_t(1) << 30;  // chunks of about 1 GiB
  if (b < per_date) b = per_date;
  return b + 8192;
}

// Persistent rank+IC over f64 (panel, date) items; nt in {256, 512, 1024}.  With
// occ != nullptr nothing is launched: *occ receives the CTAs per SM that fit.
size_t rank_ic_batch_smem(int nt, int maxN);
cudaError_t launch_rank_ic_batch(int nt, const RankIcArgs<double, double>* panels, const int2* items, int nitems,
                                 int* counter, int grid, size_t smem, int* status, cudaStream_t st, int* occ);
// factor_corr precision form (fc_tc.cu): BF16x3 tcgen05 moment products over
// the R pooled rows, split over one CTA per SM, FP64 finalize.  F <= kFcTcMaxF;
// element (r, f) at X[r*sr + f*sf]; work: fc_tc_work_bytes(F) bytes.
constexpr int kFcTcMaxF = 16;
size_t fc_tc_work_bytes(int F);
cudaError_t launch_factor_corr_bf16x3(const float* X, const uint8_t* mask, long long R, int F, long long sr,
                                      long long sf, void* work, double* out, int* status, cudaStream_t s);
// Same with element (r, f) at X[r*sr + f*sf].
cudaError_t launch_factor_corr_strided(const void* X, int dtype, const uint8_t* mask, long long R, int F,
                                       long long sr, long long sf, FcWork& w, double* out, uint8_t* flags,
                                       cudaStream_t s);

}  // namespace fcb
