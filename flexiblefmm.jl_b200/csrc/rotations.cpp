// The rotations of the FP64 M2L (m2l_rot.cu): for each symmetry class of the far offsets, the
// rotation that takes the representative offset o = (|o| sin θ cos φ, |o| sin θ sin φ, |o| cos θ)
// to the z axis, in the real Schmidt storage. The rotation about z by −φ is a 2 × 2 rotation of
// each (Re, Im) pair of order m; the rotation about y by −θ is block diagonal in the degree l and
// mixes neither real with imaginary parts nor degrees: per degree a block of l + 1 real parts and
// a block of l imaginary parts. The blocks are the projections of the rotated solid harmonics
// onto the harmonics, by a Gauss–Legendre × trapezoid rule on the sphere that integrates their
// products exactly.
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <utility>

#include "m2l_rot.h"

namespace fmmb {
namespace {

// Re, Im Υ̃_n^m(x), 0 ≤ m ≤ n ≤ p, at n(n + 1)/2 + m: the Schmidt recurrences of the P2M and L2P
// folds (src/operators/harmonics.jl:682-700)
using ld = long double;   // the blocks are formed in extended precision and rounded once
constexpr ld PI = 3.14159265358979323846264338327950288L;

void harmonics_at(ld x, ld y, ld z, int p, std::vector<ld>& vr, std::vector<ld>& vi) {
  const ld r2 = x * x + y * y + z * z;
  ld sr = 1, si = 0;
  for (int m = 0; m <= p; ++m) {
    if (m > 0) {
      const ld e = std::sqrt((ld)(2 * m - 1) / (ld)(2 * m));
      const ld nr = -e * (x * sr - y * si), ni = -e * (x * si + y * sr);
      sr = nr;
      si = ni;
    }
    ld pr = 0, pi = 0, cr = sr, ci = si;
    vr[m * (m + 1) / 2 + m] = sr;
    vi[m * (m + 1) / 2 + m] = si;
    for (int n = m + 1; n <= p; ++n) {
      const ld c = std::sqrt((ld)((n - m) * (n + m)));
      const ld az = (2 * n - 1) / c * z, br = std::sqrt((ld)((n - m - 1) * (n + m - 1))) / c * r2;
      const ld nr = az * cr - br * pr, ni = az * ci - br * pi;
      vr[n * (n + 1) / 2 + m] = nr;
      vi[n * (n + 1) / 2 + m] = ni;
      pr = cr; pi = ci; cr = nr; ci = ni;
    }
  }
}

RotLayout make_layout(int p) {
  RotLayout R;
  R.p = p;
  for (int l = 0; l <= p; ++l) {
    R.offd[l] = (uint16_t)R.nd;
    R.nd += 2 * RotLayout::ksteps(l + 1) * RotLayout::tiles(l + 1);
  }
  for (int m = 0; m <= p; ++m) {
    R.offt[m] = (uint16_t)R.nt;
    R.nt += RotLayout::ksteps(p + 1 - m) * RotLayout::tiles(p + 1 - m);
  }
  return R;
}

// the Gauss–Legendre rule on [−1, 1] of n points by Newton's iteration on P_n (the reference
// takes the Golub–Welsch eigenvalues, harmonics_yukawa.jl:89-93: the same rule to rounding)
template <class T>
void legendre_rule(int n, std::vector<T>& t, std::vector<T>& w, T pi, T eps) {
  t.assign(n, T(0));
  w.assign(n, T(0));
  for (int i = 0; i < (n + 1) / 2; ++i) {
    T x = std::cos(pi * (i + T(0.75)) / (n + T(0.5))), dp = 0;
    for (int it = 0; it < 100; ++it) {
      T p0 = 1, p1 = x;
      for (int k = 2; k <= n; ++k) {
        const T p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      dp = n * (x * p1 - p0) / (x * x - 1);
      const T dx = p1 / dp;
      x -= dx;
      if (std::fabs(dx) < eps) break;
    }
    T p0 = 1, p1 = x;
    for (int k = 2; k <= n; ++k) {
      const T p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
      p0 = p1;
      p1 = p2;
    }
    dp = n * (x * p1 - p0) / (x * x - 1);
    t[i] = -x;
    t[n - 1 - i] = x;
    w[i] = w[n - 1 - i] = 2 / ((1 - x * x) * dp * dp);
  }
}

std::shared_ptr<const RotHost> build(int p, const HostOperators& op) {
  // the classes of the far offsets, then the direction of the child slots
  std::vector<int> reps_off = op.reps_off;
  reps_off.insert(reps_off.end(), {1, 1, 1});
  auto H = std::make_shared<RotHost>();
  H->layout = make_layout(p);
  const RotLayout& R = H->layout;
  const int ntri = (p + 1) * (p + 2) / 2, nth = p + 1, nph = 2 * p + 2, nq = nth * nph;
  std::vector<ld> t, wt;
  legendre_rule<ld>(nth, t, wt, PI, 1e-19L);
  // the harmonics at the nodes, weighted and normalised: ∫ Re² = 2π/(2l + 1) for m ≥ 1, twice that
  // for m = 0
  std::vector<ld> br((size_t)ntri * nq), bi((size_t)ntri * nq), vr(ntri), vi(ntri), xs(3 * nq);
  for (int a = 0; a < nth; ++a)
    for (int b = 0; b < nph; ++b) {
      const int q = a * nph + b;
      const ld ph = 2 * PI * (b + 0.5L) / nph, st = std::sqrt(1 - t[a] * t[a]);
      xs[3 * q] = st * std::cos(ph);
      xs[3 * q + 1] = st * std::sin(ph);
      xs[3 * q + 2] = t[a];
      harmonics_at(xs[3 * q], xs[3 * q + 1], xs[3 * q + 2], p, vr, vi);
      for (int l = 0; l <= p; ++l)
        for (int m = 0; m <= l; ++m) {
          const ld g = wt[a] * (2 * PI / nph) * (2 * l + 1) / (m == 0 ? 4 * PI : 2 * PI);
          br[(size_t)(l * (l + 1) / 2 + m) * nq + q] = vr[l * (l + 1) / 2 + m] * g;
          bi[(size_t)(l * (l + 1) / 2 + m) * nq + q] = vi[l * (l + 1) / 2 + m] * g;
        }
    }
  const int ncls = (int)reps_off.size() / 3;
  H->d.assign((size_t)ncls * 32 * R.nd, 0.0);
  H->cs.assign((size_t)ncls * 2 * (p + 1), 0.0);
  std::map<std::pair<int, int>, int> seen;             // (dz², |o|²) → a class of the same angle θ
  std::vector<ld> rr((size_t)ntri * nq), ri((size_t)ntri * nq);
  for (int c = 0; c < ncls; ++c) {
    const int ox = reps_off[3 * c], oy = reps_off[3 * c + 1], oz = reps_off[3 * c + 2];
    const ld phi = std::atan2((ld)oy, (ld)ox);
    for (int m = 0; m <= p; ++m) {
      H->cs[((size_t)c * (p + 1) + m) * 2] = (double)std::cos(m * phi);
      H->cs[((size_t)c * (p + 1) + m) * 2 + 1] = (double)std::sin(m * phi);
    }
    int a2 = oz * oz, b2 = ox * ox + oy * oy + oz * oz;
    for (int g = 2; g <= a2 || (a2 == 0 && g <= b2); ++g)
      while (a2 % g == 0 && b2 % g == 0 && b2 > 1) { a2 /= g; b2 /= g; }
    const size_t nd = (size_t)32 * R.nd;
    double* D = &H->d[c * nd];
    const auto it = seen.find({a2, b2});
    if (it != seen.end()) {
      std::copy(&H->d[it->second * nd], &H->d[it->second * nd] + nd, D);
      continue;
    }
    seen[{a2, b2}] = c;
    // x → R_y(−θ) x
    const ld r = std::sqrt((ld)(ox * ox + oy * oy + oz * oz)), ct = oz / r, st = std::sqrt((ld)(ox * ox + oy * oy)) / r;
    for (int q = 0; q < nq; ++q) {
      const ld x = xs[3 * q], y = xs[3 * q + 1], z = xs[3 * q + 2];
      harmonics_at(ct * x - st * z, y, st * x + ct * z, p, vr, vi);
      for (int k = 0; k < ntri; ++k) {
        rr[(size_t)k * nq + q] = vr[k];
        ri[(size_t)k * nq + q] = vi[k];
      }
    }
    for (int l = 0; l <= p; ++l)
      for (int part = 0; part < 2; ++part) {            // real parts (orders 0..l), imaginary parts (1..l)
        const ld *rot = part ? ri.data() : rr.data(), *bas = part ? bi.data() : br.data();
        for (int k = part; k <= l; ++k)                 // column k: the input order
          for (int j = part; j <= l; ++j) {             // row j: the output order
            const ld* u = rot + (size_t)(l * (l + 1) / 2 + j) * nq;
            const ld* v = bas + (size_t)(l * (l + 1) / 2 + k) * nq;
            ld sum = 0;
            for (int q = 0; q < nq; ++q) sum += u[q] * v[q];
            D[R.rot_at(l, part, j, k)] = (double)sum;
          }
      }
  }
  H->csf.assign((size_t)NFAR * 2 * (p + 1), 0.0);
  for (int f = 0; f < NFAR; ++f) {
    const ld phi = std::atan2((ld)op.faroff[3 * f + 1], (ld)op.faroff[3 * f]);
    for (int m = 0; m <= p; ++m) {
      const ld sg = op.faroff[3 * f + 2] < 0 && (m & 1) ? -1 : 1;
      H->csf[((size_t)f * (p + 1) + m) * 2] = (double)(sg * std::cos(m * phi));
      H->csf[((size_t)f * (p + 1) + m) * 2 + 1] = (double)(sg * std::sin(m * phi));
    }
  }
  H->csk.assign((size_t)NCH * 2 * (p + 1), 0.0);
  for (int k = 0; k < NCH; ++k) {
    const ld phi = std::atan2((ld)(k >> 1 & 1) - 0.5L, (ld)(k & 1) - 0.5L);
    for (int m = 0; m <= p; ++m) {
      const ld sg = !(k >> 2) && (m & 1) ? -1 : 1;
      H->csk[((size_t)k * (p + 1) + m) * 2] = (double)(sg * std::cos(m * phi));
      H->csk[((size_t)k * (p + 1) + m) * 2 + 1] = (double)(sg * std::sin(m * phi));
    }
  }
  return H;
}

}  // namespace

void gauss_legendre(int n, std::vector<double>& t, std::vector<double>& w) {
  legendre_rule<double>(n, t, w, M_PI, 1e-16);
}

// built once per order in the process (at most PMAX of them, 2.5 MB at the largest order) and
// shared by every cache; the classes and their representatives are the same for every order
std::shared_ptr<const RotHost> rotation_tables(int p, const HostOperators& op) {
  static std::mutex mu;
  static std::map<int, std::shared_ptr<const RotHost>> store;
  std::lock_guard<std::mutex> lk(mu);
  auto& h = store[p];
  if (!h) h = build(p, op);
  return h;
}

}  // namespace fmmb
