// Host check of the bounds of gtls_b200/csrc/screen.cuh on curves with spikes:
// samples of up to 10^8 times the others' |u| or w, kept out of the prefix sums and
// added to the windows that hold them.  Prefix sums as the kernel keeps them, in
// FP64 and rounded once, with its bound of that rounding.  The bounds of
// every start must enclose delta = c (2 B + c C) as 64-bit sums over the window
// give it, from both tables of cells, on exact and coarse prefix values, for equal and
// unequal weights.  Prints one line per violation and "ok <starts>"; exit
// status 1 on any violation.
#include <cstdio>
#include <random>

#include "screen.cuh"

using namespace gtls;

int main() {
  std::mt19937_64 rng(77);
  std::normal_distribution<double> gauss;
  std::uniform_real_distribution<double> uni(0.0, 1.0);
  long long starts = 0, held = 0, bad = 0;
  const int widths[] = {1, 2, 7, 33, 100, 128, 129, 513, 1407, 1408, 3000};
  for (int w : widths)
    for (int kind = 0; kind < 4; ++kind) {   // glitches, sure samples, both with a transit, equal weights
      const int g = w > 1407 ? 17 : 1, n = 3 * w + 300, total = n + w + 4 * g;
      std::vector<double> T(w), v(total), wt(total);
      for (int i = 0; i < w; ++i) {
        const double x = w > 1 ? 2.0 * i / (w - 1) - 1.0 : 0.0;
        T[i] = 0.5 * std::sqrt(std::max(0.0, 1.0 - x * x * 0.999));
      }
      for (int i = 0; i < total; ++i) {
        wt[i] = kind == 3 ? 0.87 : std::exp(gauss(rng));
        v[i] = gauss(rng) / std::sqrt(wt[i]) - 0.2;
        if (kind == 2 && i > n / 2 && i < n / 2 + w) v[i] -= 4.0 * T[i - n / 2];
      }
      std::vector<char> spike(total, 0);
      const int count = kind == 2 ? 40 : 6;
      for (int q = 0; q < count; ++q) {
        const int i = (int)(uni(rng) * total);
        spike[i] = 1;
        if (kind == 0 || kind == 3 || (kind == 2 && q % 2)) v[i] *= std::exp(uni(rng) * 18.0);
        else wt[i] *= std::exp(uni(rng) * 18.0);
      }
      double wbar = 0, qbar = 0, t2 = 0;
      for (int i = 0; i < n; ++i)
        if (!spike[i]) wbar += wt[i] / n, qbar += v[i] * wt[i] * v[i] * wt[i] / n;
      if (kind == 3) wbar = 0.87;
      for (double t : T) t2 += t * t;
      std::vector<float> V(total + 1), U(total + 1), W(total + 1), Q(total + 1);
      double sv = 0, su = 0, sw = 0, sq = 0, mv = 0, mu = 0, mw = 0, mq = 0;
      for (int i = 0; i < total; ++i) {
        const double wi = spike[i] ? 0.0 : wt[i], u = v[i] * wi;
        sv += v[i], su += u, sw += wi - (float)wbar, sq += u * u - (float)qbar;
        V[i + 1] = (float)sv, U[i + 1] = (float)su, W[i + 1] = (float)sw, Q[i + 1] = (float)sq;
        mv = std::max(mv, std::fabs(sv)), mu = std::max(mu, std::fabs(su));
        mw = std::max(mw, std::fabs(sw)), mq = std::max(mq, std::fabs(sq));
      }
      const ScreenErr e = screen_err((float)mv * kPrefixErr, (float)mu * kPrefixErr, (float)mw * kPrefixErr, (float)mq * kPrefixErr);
      for (int table = 0; table < 2; ++table) {
        std::vector<int> ends;
        screen_cells(w, g, table == 0, ends);
        std::vector<ScreenCell> cells;
        ScreenRow row = {};
        auto at = [&](int i) { return i >= 0 && i < w ? T[i] : 0.0; };
        for (size_t q = 0; q < ends.size(); ++q) {
          const int e0 = (q ? ends[q - 1] : 0) * g, e1 = ends[q] * g, l = e1 - e0;
          double m0 = 0, m1 = 0, rc2 = 0, rb = 0, mn = INFINITY, mx = 0;
          for (int x = e0; x < e1; ++x) m0 += at(x) / l, m1 += at(x - (g - 1)) / l;
          ScreenCell c;
          c.a = (float)m0;
          c.b = g > 1 ? (float)((m0 - m1) / (g - 1)) : 0.f;
          for (int off = 0; off < g; ++off) {
            double r1 = 0, r2 = 0;
            for (int x = e0 - off; x < e1 - off; ++x) {
              const double r = at(x) - ((double)c.a - (double)c.b * off);
              r1 += r, r2 += r * r;
              mn = std::min(mn, at(x) * at(x)), mx = std::max(mx, at(x) * at(x));
            }
            rc2 = std::max(rc2, r2 - r1 * r1 / l + 1e-14 * r2);
            rb = std::max(rb, std::fabs(r1 / l));
          }
          c.rc = (float)(std::sqrt(std::max(rc2, 0.0)) * 1.000001), c.rb = (float)(rb * 1.000001);
          c.mn = (float)mn, c.mx = (float)mx, c.l = (float)l, c.inv_l = (float)(1.0 / l * (1.0 - 0x1p-10));
          cells.push_back(c);
          row.asum += (float)((std::fabs((double)c.a) + std::fabs((double)c.b) * (g - 1) + rb) * 1.0001);
          row.smn += (float)mn, row.smx += (float)(mx * 1.0001), row.lmn += (float)(mn * l), row.lmx += (float)(mx * l);
        }
        row.m = (int)cells.size(), row.inv_w = (float)(1.0 / w), row.os2 = 2.f * 1.07f;
        row.tn = (float)(std::sqrt(t2) * 1.000001), row.t2 = (float)t2;
        for (int k = 0; k < n; k += 1 + w / 60) {
          const int q1 = k / g;
          const float kappa = (float)(q1 * g - k);
          CellSums cs;
          for (size_t q = 0; q < cells.size(); ++q) {
            const int p0 = (q1 + (q ? ends[q - 1] : 0)) * g, p1 = (q1 + ends[q]) * g;
            const float dU = U[p1] - U[p0], dW = W[p1] - W[p0], dQ = Q[p1] - Q[p0];
            if (g > 1) add_cell<true, true>(cs, cells[q], dU, dW, dQ, kappa, (float)qbar, e);
            else add_cell<false, true>(cs, cells[q], dU, dW, dQ, 0.f, (float)qbar, e);
          }
          const int span = g > 1 ? ends.back() * g : w;
          const float m = (V[k] - V[k + w]) * row.inv_w, em = std::fmaf(3e-7f, std::fabs(m), e.v * row.inv_w);
          float qwin = (Q[q1 * g + span] - Q[q1 * g]) + (float)span * (float)qbar + 4.f * e.n2;
          for (int i = 0; i < w; ++i)
            if (spike[k + i]) {
              const float u = (float)(v[k + i] * wt[k + i]);
              add_spike(cs, (float)T[i], (float)(T[i] * T[i]), u, kind == 3 ? 0.f : (float)wt[k + i], spike_err(count));
              qwin = std::fmaf(u, u, qwin);
              ++held;
            }
          const StartBounds b = start_bounds<true>(cs, row, m, em, qwin, (float)wbar, kind == 3, kGammaF, e);
          double S = 0, B = 0, C = 0;
          for (int i = 0; i < w; ++i) S += v[k + i], B += T[i] * v[k + i] * wt[k + i], C += T[i] * T[i] * wt[k + i];
          const double c = 2.0 * 1.07f * (-S / w), delta = c * (2 * B + c * C);
          ++starts;
          if (!(b.lb <= delta && delta <= b.ub))
            if (++bad <= 20) std::printf("w %d kind %d table %d start %d: %g not in [%g, %g]\n", w, kind, table, k, delta, b.lb, b.ub);
        }
      }
    }
  if (bad) return std::printf("%lld of %lld starts outside\n", bad, starts), 1;
  std::printf("ok %lld (%lld spikes in their windows)\n", starts, held);
  return 0;
}
