// Occultation of a star with quadratic limb darkening by an opaque disk, by
// the quadrature of gtls_b200/ldmodel.py (96-node Gauss-Legendre after the
// substitution r = m + h sin(theta)), in forms shared by the adjoint model
// (adjoint.cu, with derivatives in (z, p)) and the transit
// template generator (templates.cu).  ldmodel stands in for the batman light
// curve of the reference (src/gputls/transit.py:8-42).
#pragma once
#include <cuda_runtime.h>

#include <cmath>

namespace gtls {

constexpr double kPi = 3.14159265358979323846;
constexpr int kGLN = 96;

// Quadrature table: s[j] = sin(theta_j), jw[j] = cos(theta_j) * pi/2 * w_j
// with theta_j = pi/2 x_j for the Gauss-Legendre nodes x_j and weights w_j.
struct GLTable {
  double s[kGLN];
  double jw[kGLN];
};

// Gauss-Legendre nodes and weights on [-1, 1] by Newton's method on the
// three-term recurrence of the Legendre polynomials (Golub-Welsch-free
// classic; converges to a few ulp from the Tricomi starting values).
static GLTable make_gl_table() {
  GLTable g;
  const int n = kGLN;
  for (int i = 0; i < (n + 1) / 2; ++i) {
    double x = std::cos(kPi * (i + 0.75) / (n + 0.5));
    double dp = 1.0;
    for (int it = 0; it < 100; ++it) {
      double p0 = 1.0, p1 = x;
      for (int k = 2; k <= n; ++k) {
        const double p2 = ((2.0 * k - 1.0) * x * p1 - (k - 1.0) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      dp = n * (x * p1 - p0) / (x * x - 1.0);
      const double dx = p1 / dp;
      x -= dx;
      if (std::fabs(dx) < 1e-17) break;
    }
    const double w = 2.0 / ((1.0 - x * x) * dp * dp);
    // ascending order: node j = n-1-i holds +x, node i holds -x
    const int hi = n - 1 - i, lo = i;
    const double th = 0.5 * kPi * x;
    g.s[hi] = std::sin(th);
    g.jw[hi] = std::cos(th) * (0.5 * kPi) * w;
    g.s[lo] = -g.s[hi];
    g.jw[lo] = g.jw[hi];
  }
  return g;
}

static const GLTable& gl_table() {
  static const GLTable g = make_gl_table();
  return g;
}

// mu = sqrt(max(1 - r^2, 0))
__device__ __forceinline__ double mu_of(double r) {
  const double x = 1.0 - r * r;
  return x > 0.0 ? sqrt(x) : 0.0;
}
// acos of c clamped to [-1, 1]
__device__ __forceinline__ double acos_clamped(double c) {
  return c >= 1.0 ? 0.0 : (c <= -1.0 ? kPi : acos(c));
}

// Moments M0..M2 of the occulted flux: lambda = (M0 - u1 M1 - u2 M2) / (pi K),
// Mk = int (1 - mu)^k x (2 pi r over the covered disk, 2 r acos(c) over the
// partly covered annuli) dr, both by the quadrature of ldmodel.occulted_fraction
// (its nodes j0, j0 + step, ...).
__device__ __forceinline__ void occultation_moments(double z, double p, const GLTable& g, double (&M)[3], int j0 = 0,
                                                    int step = 1) {
#pragma unroll
  for (int k = 0; k < 3; ++k) M[k] = 0.0;
  // region fully covered by the planet: r in [0, min(p - z, 1)]
  if (p - z > 0.0) {
    const double half = (p - z > 1.0 ? 1.0 : p - z) * 0.5;
    for (int j = j0; j < kGLN; j += step) {
      const double r = half + half * g.s[j];
      const double om = 1.0 - mu_of(r);
      const double f = r * (half * g.jw[j]) * (2.0 * kPi);
      M[0] = M[0] + f;
      M[1] = M[1] + f * om;
      M[2] = M[2] + f * om * om;
    }
  }
  // partially covered annuli: r in [|z - p|, min(1, z + p)]
  const double lo = z >= p ? z - p : p - z;
  const double hi = z + p > 1.0 ? 1.0 : z + p;
  if (hi > lo) {
    const double mid = (lo + hi) * 0.5, half = (hi - lo) * 0.5;
    const double zs = z > 1e-300 ? z : 1e-300;
    const double zp2 = zs * zs - p * p;
    for (int j = j0; j < kGLN; j += step) {
      const double r = mid + half * g.s[j];
      const double c = (r * r + zp2) / (r * zs * 2.0);
      const double om = 1.0 - mu_of(r);
      const double f = r * acos_clamped(c) * (half * g.jw[j]) * 2.0;
      M[0] = M[0] + f;
      M[1] = M[1] + f * om;
      M[2] = M[2] + f * om * om;
    }
  }
}

// N = M0 - u1 M1 - u2 M2 with its derivatives in (z, p), and M1, M2 (which are
// minus its derivatives in u1, u2): the derivatives of the discrete quadrature
// itself, through the nodes, the limits and c.  Written out by hand, with one
// reciprocal per node where general dual numbers divide five times; where a
// square root or the acos is clamped its derivative is 0.
struct OccultationGrad {
  double N, Nz, Np, M1, M2;
};
__device__ __forceinline__ OccultationGrad occultation_grad(double z, double p, double u1, double u2,
                                                            const GLTable& g, int j0, int step) {
  OccultationGrad o{0.0, 0.0, 0.0, 0.0, 0.0};
  // one node: f and its derivatives times the intensity at r
  auto add = [&](double r, double rz, double rp, double f, double fz, double fp) {
    const double x = 1.0 - r * r;
    double mu = 0.0, k = 0.0;   // mu and r / mu = -dmu/dr
    if (x > 0.0) {
      const double s = rsqrt(x);
      mu = x * s;
      k = r * s;
    }
    const double om = 1.0 - mu;
    const double I = 1.0 - om * (u1 + u2 * om), Ir = -(u1 + 2.0 * u2 * om) * k;
    o.N = fma(f, I, o.N);
    o.Nz += fz * I + f * Ir * rz;
    o.Np += fp * I + f * Ir * rp;
    const double fo = f * om;
    o.M1 += fo;
    o.M2 = fma(fo, om, o.M2);
  };
  if (p - z > 0.0) {
    const bool whole = p - z > 1.0;
    const double half = (whole ? 1.0 : p - z) * 0.5, hz = whole ? 0.0 : -0.5;   // dhalf/dp = -hz
    for (int j = j0; j < kGLN; j += step) {
      const double s1 = 1.0 + g.s[j], jw = g.jw[j] * (2.0 * kPi);
      const double r = half * s1, wt = half * jw;
      // f = r wt: both are half times a constant
      const double fh = 2.0 * r * jw;
      add(r, hz * s1, -hz * s1, r * wt, fh * hz, -fh * hz);
    }
  }
  const bool out = z >= p, limb = z + p > 1.0;
  const double lo = out ? z - p : p - z, hi = limb ? 1.0 : z + p;
  if (hi > lo) {
    const double mid = (lo + hi) * 0.5, half = (hi - lo) * 0.5;
    const double loz = out ? 1.0 : -1.0, h1 = limb ? 0.0 : 1.0;   // dlo/dz = -dlo/dp; dhi/dz = dhi/dp
    const double mz = 0.5 * (loz + h1), mp = 0.5 * (h1 - loz), hz = 0.5 * (h1 - loz), hp = 0.5 * (h1 + loz);
    const bool centre = !(z > 1e-300);
    const double zs = centre ? 1e-300 : z, dzs = centre ? 0.0 : 1.0;
    const double zp2 = zs * zs - p * p;
    for (int j = j0; j < kGLN; j += step) {
      const double s = g.s[j], jw = 2.0 * g.jw[j];
      const double r = mid + half * s, rz = mz + hz * s, rp = mp + hp * s;
      const double inv = 1.0 / (2.0 * r * zs);
      const double c = (r * r + zp2) * inv;
      double ac = c >= 1.0 ? 0.0 : (c <= -1.0 ? kPi : c), acz = 0.0, acp = 0.0;   // (a NaN stays one)
      if (c < 1.0 && c > -1.0) {
        ac = acos(c);
        const double d = 1.0 - c * c;
        const double k = d > 0.0 ? -2.0 * inv * rsqrt(d) : 0.0;   // dacos/dc times 2 / (2 r z)
        acz = k * (r * rz + zs * dzs - c * (rz * zs + r * dzs));
        acp = k * (r * rp - p - c * rp * zs);
      }
      const double ra = r * ac, wt = half * jw;
      add(r, rz, rp, ra * wt, (rz * ac + r * acz) * wt + ra * (hz * jw), (rp * ac + r * acp) * wt + ra * (hp * jw));
    }
  }
  return o;
}

// Fraction of the stellar flux blocked by a disk of radius p at separation z
// (ldmodel.occulted_fraction): 0 unless z < 1 + p and p > 0.
__device__ __forceinline__ double occulted_fraction(double z, double p, double u1, double u2, const GLTable& g) {
  if (!(p > 0.0) || !(z < 1.0 + p)) return 0.0;
  double M[3];
  occultation_moments(z, p, g, M);
  return (M[0] - u1 * M[1] - u2 * M[2]) / (kPi * (1.0 - u1 / 3.0 - u2 / 6.0));
}

}  // namespace gtls
