// The rotations of the FP64 M2L (m2l_rot.cu): for each symmetry class of the far offsets, the
// rotation that takes the representative offset o = (|o| sin θ cos φ, |o| sin θ sin φ, |o| cos θ)
// to the z axis, in the real Schmidt storage. The rotation about z by −φ is a 2 × 2 rotation of
// each (Re, Im) pair of order m; the rotation about y by −θ is block diagonal in the degree l and
// mixes neither real with imaginary parts nor degrees: per degree a block of l + 1 real parts and
// a block of l imaginary parts, from Wigner's d matrices by their recurrence in the degree: O(p³) per
// angle. (Projections of the rotated harmonics by quadrature, O(p⁵), gave the same tables to rounding and
// took 15, 97 and 292 ms of one CPU thread at p = 10, 16 and 20, paid by the first state of an order in a
// process; the recurrence takes 1, 3 and 5.)
#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <utility>

#include "m2l_rot.h"

namespace fmmb {
namespace {

using ld = long double;   // the blocks are formed in extended precision and rounded once

// Wigner's d^l_{ab}(β), a ≥ |b|, for l = a..p at d[l], cb = cos β, ch and sh the cosine and sine of β/2:
// d^a_{ab} = √C(2a, a + b) ch^(a+b) (−sh)^(a−b), then the three-term recurrence in the degree
// (Varshalovich, Moskalev, Khersonskii, Quantum Theory of Angular Momentum, 1988, section 4.8; upwards, as for the
// Jacobi polynomials, the stable direction)
void wigner_d(int a, int b, int p, ld cb, ld ch, ld sh, ld* d) {
  ld v = 1;
  for (int i = 1; i <= a - b; ++i) v *= std::sqrt((ld)(a + b + i) / i) * -sh;   // C(2a, a − b) = Π (a + b + i)/i
  for (int i = 0; i < a + b; ++i) v *= ch;
  d[a] = v;
  ld prev = 0;
  for (int l = a; l < p; ++l) {
    const ld ab = l ? (ld)(a * b) / l : 0, back = l ? std::sqrt((ld)(l * l - a * a) * (l * l - b * b)) / l : 0;
    const ld next = ((2 * l + 1) * ((l + 1) * cb - ab) * d[l] - (l + 1) * back * prev) /
                    std::sqrt((ld)((l + 1) * (l + 1) - a * a) * ((l + 1) * (l + 1) - b * b));
    prev = d[l];
    d[l + 1] = next;
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

std::shared_ptr<const RotHost> build(int p, const HostOperators& op) {
  // the classes of the far offsets, then the direction of the child slots
  std::vector<int> reps_off = op.reps_off;
  reps_off.insert(reps_off.end(), {1, 1, 1});
  auto H = std::make_shared<RotHost>();
  H->layout = make_layout(p);
  const RotLayout& R = H->layout;
  const int ncls = (int)reps_off.size() / 3;
  H->d.assign((size_t)ncls * 32 * R.nd, 0.0);
  H->cs.assign((size_t)ncls * 2 * (p + 1), 0.0);
  std::map<std::pair<int, int>, int> seen;             // (dz², |o|²) → a class of the same angle θ
  std::vector<ld> dp(p + 1), dm(p + 1);
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
    // Υ^j(R_y(−θ) x) = Σ_k d_{kj}(θ) Υ^k(x), k = −l..l, in real and imaginary parts by Υ^{−k} = (−1)^k conj Υ^k
    const ld r = std::sqrt((ld)(ox * ox + oy * oy + oz * oz)), ct = oz / r;
    const ld ch = std::sqrt((r + oz) / (2 * r)), sh = std::sqrt((r - oz) / (2 * r));
    for (int j = 0; j <= p; ++j)                        // row j: the output order
      for (int k = 0; k <= p; ++k) {                    // column k: the input order
        // d_{kj} and (−1)^k d_{−k,j}, by d_{kj} = (−1)^(k−j) d_{jk} = d_{−j,−k}
        const int a = std::max(j, k), b = std::min(j, k), odd = (j + k) & 1;
        wigner_d(a, b, p, ct, ch, sh, dp.data());
        wigner_d(a, -b, p, ct, ch, sh, dm.data());
        for (int l = a; l <= p; ++l) {
          const ld plus = odd && k < j ? -dp[l] : dp[l], minus = j & 1 ? -dm[l] : dm[l];
          D[R.rot_at(l, 0, j, k)] = (double)(k == 0 ? plus : plus + minus);
          if (j && k) D[R.rot_at(l, 1, j, k)] = (double)(plus - minus);
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
