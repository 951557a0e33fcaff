// corr_common.cuh -- what the FP64 correlations share: compensated sums, the
// Pearson finalize with its gates, and the FP64 matrix instruction.
#pragma once

#include "fcb_common.cuh"

namespace fcb {

constexpr double kBigPos = 1e300;
constexpr double kCancelRatio = 3.0;
constexpr double kConstVarRel = 1e-10;
constexpr double kTiny = 1e-300;
constexpr int kTwoPassKahanT = 2048;

struct Kahan {
  double s = 0.0, c = 0.0;
  FCB_DEV void add(double x) {
    const double y = x - c;
    const double t = s + y;
    c = (t - s) - y;
    s = t;
  }
  FCB_DEV void merge(const Kahan& o) {
    add(o.s);
    add(-o.c);
  }
};

// A sum with its rounding errors (two-sum): s + c is the sum to about twice
// the precision.
struct TwoSum {
  double s = 0.0, c = 0.0;
  FCB_DEV void add(double x) {
    const double t = s + x, b = t - s;
    c += (s - (t - b)) + (x - b);
    s = t;
  }
  FCB_DEV double value() const { return s + c; }
  // the sum less a * b, with one rounding of the size of the sum
  FCB_DEV double less_product(double a, double b) const {
    const double p = a * b, e = fma(a, b, -p);
    TwoSum r = *this;
    r.add(-p);
    return r.s + (r.c - e);
  }
  // the warp's total, the same in every lane
  FCB_DEV void warp_total() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double s2 = __shfl_xor_sync(kFull, s, o), c2 = __shfl_xor_sync(kFull, c, o);
      c += c2;
      add(s2);
    }
  }
};

FCB_DEV double dnan() { return __longlong_as_double(0x7ff8000000000000ll); }

FCB_DEV double safe_pearson(double sxy, double sxx, double syy) {
  if (!(sxx > 0.0 && syy > 0.0) || !isfinite(sxx) || !isfinite(syy) || !isfinite(sxy)) return dnan();
  const double r = (sxy / sqrt(sxx)) / sqrt(syy);
  return isfinite(r) ? r : dnan();
}

// One pair from its centred moment sums (x' = x - mux).  gate: the reference's
// cancellation gate on the uncentred sums (reconstructed) fails.  redo: the
// value must come from the two-pass recomputation.  A gated pair's value is
// kept when the centred sums carry it at full precision: the joint means lie
// within two standard deviations of the shifts, and the shifts within 1e6 of
// them from zero (beyond, the rounding of the two-pass mean itself shows).
struct PairResult {
  double r;
  bool gate, redo;
};
// cov, vx, vy: the sums about the joint means (mx, my from the shifts, rn = 1 / n).
FCB_DEV PairResult finalize_about_means(double n, double rn, double mx, double my, double sx, double sy, double cov,
                                        double vx, double vy, double sx2, double sy2, double mux, double muy) {
  // uncentred sums of the reference's one-pass Gram, reconstructed
  const double sxr = sx + n * mux;
  const double syr = sy + n * muy;
  const double sx2r = sx2 + 2.0 * mux * sx + n * mux * mux;
  const double sy2r = sy2 + 2.0 * muy * sy + n * muy * muy;
  const double qxx = sxr * sxr * rn, qyy = syr * syr * rn;
  const bool gate = (fabs(sxr * syr * rn) > kCancelRatio * fabs(cov)) || (fabs(qxx) > kCancelRatio * fabs(vx)) ||
                    (fabs(qyy) > kCancelRatio * fabs(vy));
  const double xmag = fmax(fabs(sx2r), fabs(qxx));
  const double ymag = fmax(fabs(sy2r), fabs(qyy));
  const double r = safe_pearson(cov, vx, vy);
  const bool degenerate = fabs(vx) <= kConstVarRel * (xmag + kTiny) || fabs(vy) <= kConstVarRel * (ymag + kTiny) ||
                          !isfinite(r) || fabs(r) > 1.0;
  const bool near = mx * sx <= 4.0 * vx && my * sy <= 4.0 * vy;
  const bool small = n * mux * mux <= 1e12 * vx && n * muy * muy <= 1e12 * vy;
  const bool redo = degenerate || !near || (gate && !small);
  return PairResult{redo ? dnan() : r, gate || degenerate, redo};
}

FCB_DEV PairResult finalize_pair(double n, double sx, double sy, double sxy, double sx2, double sy2, double mux,
                                 double muy) {
  if (n < 2.0) return PairResult{dnan(), false, false};
  const double rn = 1.0 / n, mx = sx * rn, my = sy * rn;  // one division for all
  return finalize_about_means(n, rn, mx, my, sx, sy, fma(-mx, sy, sxy), fma(-mx, sx, sx2), fma(-my, sy, sy2), sx2, sy2,
                              mux, muy);
}

FCB_DEV void dmma_f64(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

}  // namespace fcb
