// Bounds on the chi2 of a start from block sums, so that only the starts that
// can hold a period's minimum get their full template sums.
//
// delta(d, k) = c (2 B + c C) with B = sum_i s_i u_{k+i}, C = sum_i s_i^2
// w_{k+i}.  The template is cut into cells.  In cell q (samples q0..q1, l of
// them) it is a_q plus a remainder r, and with U, W, Q the prefix sums of u, w
// and u^2
//
//   sum_cell s u = a_q dU + rbar dU + sum (r - rbar)(u - ubar),
//   |last term| <= ||r - rbar|| sqrt(dQ - dU^2 / l)          (Cauchy-Schwarz)
//   min s^2 dW <= sum_cell s^2 w <= max s^2 dW
//
// so a few prefix values per cell bound delta from both sides.  The smallest
// upper bound of any start is an upper bound of the minimum, and a start whose
// lower bound lies above it can be left out: the minimum over the others, and
// its first location, are those over all starts.  Every rounding of the FP32
// arithmetic (prefix values, cell sums, coefficients) is added to the bounds
// (ScreenErr, kGammaF and the factors next to them), so they hold for the
// value the exact sums give, in FP64 or FP32.
//
// Two tables of cells per duration, narrower at the template's edges, where it
// is steep.  All starts that pass the depth test are bounded with about
// sqrt(width)/2 cells, a start per lane; those that this leaves with 16 to 96
// cells, a start per warp, a cell per lane.  Measured on 19,728- and
// 70,000-sample curves (5,000 to 50,000 starts a period pass): the first
// leaves 1 to 15%, the second 1 to 60 starts a period.  (One table of sqrt(width)
// cells takes 2.5 times the cell evaluations; equal cells leave 2 to 4 times
// as many starts.)
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace gtls {

constexpr int kLaneCells = 16;     // cells of the first table, at most
constexpr int kWarpCells = 96;     // cells of the second table, at most
constexpr float kGammaF = 2e-5f;   // relative rounding of the FP32 cell sums (kWarpCells terms and their factors)

// One cell of a duration's template.
struct ScreenCell {
  float a, rc;       // mean of the template, norm of the centred remainder
  float mn, mx;      // bounds of the squared template
  float l, inv_l;    // samples; 1/l, rounded down (it multiplies a subtracted square)
  float b, rb;       // coarse rows: change of a per sample of offset, bound of |rbar|
};

// One duration and table.
struct ScreenRow {
  int first, m;        // its cells
  float inv_w, os2;    // 1/width, 2 * overshoot
  float asum, tn;      // sum of |a| (and |b| times the largest offset), norm of the template
  float smn, smx;      // sums of mn and mx
  float lmn, lmx;      // sums of mn * l and mx * l
  float t2;            // sum of the squared template
  float pad;
};

// Where cell i of m ends, as a fraction of the template: z - e sin(2 pi z) / 2 pi
// at z = (i + 1) / m, so cells at the edges are 1 - e times as long as equal ones.
inline const std::vector<double>& cell_fractions(int m, bool per_lane) {
  static const std::vector<std::vector<double>> tables = [] {
    std::vector<std::vector<double>> t(2 * (kWarpCells + 1));
    const double pi = 3.14159265358979323846;
    for (int k = 0; k < 2; ++k)
      for (int c = 1; c <= kWarpCells; ++c)
        for (int i = 1; i <= c; ++i) {
          const double z = (double)i / c;
          t[2 * c + k].push_back(i == c ? 1.0 : z - (k ? 0.8 : 0.5) * std::sin(2.0 * pi * z) / (2.0 * pi));
        }
    return t;
  }();
  return tables[2 * m + (per_lane ? 1 : 0)];
}

// Cell boundaries of a template of `width` samples in steps of `g` samples (1:
// exact rows; else the window starts up to g - 1 samples into the first
// step): the ends of the cells, in steps, into `ends`.
inline void screen_cells(int width, int g, bool per_lane, std::vector<int>& ends) {
  const int top = g == 1 ? width : (width + 2 * (g - 1)) / g;   // steps that cover every offset
  const int m = per_lane ? std::min(kLaneCells, std::max(2, (int)std::lround(std::sqrt((double)width) / 2.0)))
                         : (width <= 128 ? 16 : (width <= 512 ? 32 : (width <= 2048 ? 64 : kWarpCells)));
  int prev = 0;
  for (const double f : cell_fractions(m, per_lane)) {
    const int e = std::min(top, (int)std::lround(f * top));
    if (e > prev) {
      ends.push_back(e);
      prev = e;
    }
  }
}

// Rounding of the stored prefix values: bounds of the error of a difference
// of two of them (V, U, W), and what the errors of U and Q add to a cell's
// squared norm (2 x e <= x^2/1024 + 1024 e^2 for the square of dU).
struct ScreenErr {
  float v, u, w, n2;
};
__host__ __device__ __forceinline__ ScreenErr screen_err(float v, float u, float w, float q) {
  return ScreenErr{v, u, w, fmaf(1026.f * u, u, q + 1e-30f)};
}

// Rounding of a difference of two prefix values, relative to the largest of
// them: they are summed in FP64 and rounded to FP32 once each.  (Summed in FP32
// the bound was 2^-16 of the largest; after six flares of 50% it left so many
// starts that the list ran over: 300 periods of 19,728 samples 18.5 ms, now 0.61,
// of 70,000 92 and 1.67 ms.  Without flares both take the same time.)
constexpr float kPrefixErr = 0x1.01p-23f;

struct StartBounds {
  float lb, ub;
};

__host__ __device__ __forceinline__ float screen_sqrt(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));   // 1 ulp and a bit: kGammaF covers it
  return r;
#else
  return std::sqrt(x);
#endif
}

// Running sums of a start over its cells.
struct CellSums {
  float B = 0.f, er = 0.f, cl = 0.f, cu = 0.f;
};

// Add a cell with prefix differences (dU, dW, dQ).  dW and dQ are of the
// detrended prefixes (mean weight wbar and mean square qbar taken out: their
// values stay small); wbar's part of C is added in start_bounds.  `kappa`: the
// window's offset in its first step (coarse rows, <= 0).
template <bool kCoarse, bool kUpper>
__host__ __device__ __forceinline__ void add_cell(CellSums& s, const ScreenCell& c, float dU, float dW, float dQ,
                                                  float kappa, float qbar, const ScreenErr& e) {
  // ||u - ubar||^2 of the cell from above: dQ + l qbar - dU^2/l, with 2^-10 of
  // the subtracted square kept back for dU's error
  const float n2 = fmaf(-dU * dU, c.inv_l, fmaf(c.l, qbar * 1.000002f, dQ));
  const float nn = screen_sqrt(fmaxf(n2, 0.f) + e.n2);
  const float a = kCoarse ? fmaf(c.b, kappa, c.a) : c.a;
  s.B = fmaf(a, dU, s.B);
  s.er = fmaf(c.rc, nn, s.er);
  if (kCoarse) s.er = fmaf(c.rb, fabsf(dU) + e.u, s.er);
  s.cl = fmaf(c.mn, dW, s.cl);
  if (kUpper) s.cu = fmaf(c.mx, dW, s.cu);
}

// A sample that is kept out of the prefix sums (its u and w there are 0) and lies
// in the window, where the template is s and its square s2: its products, with
// the rounding of the sums of up to `err`'s count of them.  Where all weights equal wbar,
// w is 0 here (C is wbar * t2 then).
__host__ __device__ __forceinline__ float spike_err(int count) { return 1.2e-7f * (float)(count + 8); }
__host__ __device__ __forceinline__ void add_spike(CellSums& cs, float s, float s2, float u, float w, float err) {
  const float b = s * u, c = s2 * w;
  cs.B += b;
  cs.er = fmaf(fabsf(b), err, cs.er);
  cs.cl = fmaf(c, 1.f - err, cs.cl);
  cs.cu = fmaf(c, 1.f + err, cs.cu);
}

// Bounds of delta (the upper one only with kUpper) for a window of mean depth in [mean - em, mean + em] (scaled
// units).  gamma: relative rounding of the exact sums themselves (FP32 form).
// uniform: all weights equal wbar, so C is wbar * t2.
template <bool kUpper>
__host__ __device__ __forceinline__ StartBounds start_bounds(const CellSums& s, const ScreenRow& r, float mean,
                                                             float em, float qwin, float wbar, bool uniform,
                                                             float gamma, const ScreenErr& e) {
  const float er = s.er * 1.0001f + r.tn * gamma * screen_sqrt(fmaxf(qwin, 0.f)) + r.asum * e.u;
  float cl = uniform ? wbar * r.t2 : fmaf(wbar, r.lmn, s.cl) - e.w * r.smn;
  // sums of mn dW and wbar mn l may nearly cancel: their rounding is relative to each
  cl = fmaxf(cl - (1e-5f + 2.f * gamma) * (fabsf(s.cl) + wbar * r.lmx), 0.f);
  const float x1 = r.os2 * (mean - em), x2 = r.os2 * (mean + em);
  const float w = 2e-6f * fmaxf(fabsf(x1), fabsf(x2));
  const float c1 = fminf(x1, x2) - w, c2 = fmaxf(x1, x2) + w;
  const float blo = s.B - er, bhi = s.B + er;
  const float p1 = c1 * blo, p2 = c1 * bhi, p3 = c2 * blo, p4 = c2 * bhi;
  const float plo = fminf(fminf(p1, p2), fminf(p3, p4));
  const float sq1 = c1 * c1, sq2 = c2 * c2;
  const float sqlo = (c1 > 0.f || c2 < 0.f) ? fminf(sq1, sq2) : 0.f;
  StartBounds o;
  o.lb = fmaf(2.f, plo, sqlo * cl);
  o.lb -= 4e-6f * (2.f * fabsf(plo) + sqlo * cl);
  o.ub = INFINITY;
  if (kUpper) {
    float cu = uniform ? wbar * r.t2 : fmaf(wbar, r.lmx, s.cu) + e.w * r.smx;
    cu += (1e-5f + 2.f * gamma) * (fabsf(s.cu) + wbar * r.lmx);
    const float phi = fmaxf(fmaxf(p1, p2), fmaxf(p3, p4)), sqhi = fmaxf(sq1, sq2);
    o.ub = fmaf(2.f, phi, sqhi * cu);
    o.ub += 4e-6f * (2.f * fabsf(phi) + sqhi * cu);
  }
  // fminf and fmaxf drop a NaN operand: a NaN anywhere must reach the bounds
  const float sum = s.B + s.er + s.cl + mean + qwin;
  const float nan = sum - sum;
  o.lb += nan;
  if (kUpper) o.ub += nan;
  return o;
}

}  // namespace gtls
