// The tables of the FP64 translations by rotations (rotations.cpp, m2l_rot.cu).
#pragma once
#include <memory>

#include "common.cuh"

namespace fmmb {

// The rotations' and translations' coefficients lie in fragments of the FP64 tensor cores' B operand
// (4 inputs × 8 outputs): lane 4n + t holds the coefficient of input 4·ks + t and output
// 8·rt + rot_out(n). The outputs of a fragment's columns are ordered so that a lane's two results
// (columns 2t, 2t + 1) are the outputs t and t + 4: four lanes then write consecutive entries.
__host__ __device__ constexpr int rot_out(int n) { return n & 1 ? 4 + n / 2 : n / 2; }
__host__ __device__ constexpr int rot_col(int out) { return out < 4 ? 2 * out : 2 * (out - 4) + 1; }

// Where the fragments of one class lie (in units of 32 doubles): per degree l, [ks][rt][part] over the
// l + 1 input and output orders (part 1: the imaginary parts, row and column 0 zero); per order m,
// [ks][rt] over the degrees m..p, the same for both parts
struct RotLayout {
  int p = 0, nd = 0, nt = 0;              // fragments per class: rotations, translations
  uint16_t offd[PMAX + 1], offt[PMAX + 1];
  static __host__ __device__ constexpr int ksteps(int s) { return (s + 3) / 4; }
  static __host__ __device__ constexpr int tiles(int s) { return (s + 7) / 8; }
  // the coefficient of input k and output j: of degree l's part, of order m (both from 0)
  __host__ __device__ int rot_at(int l, int part, int j, int k) const {
    return 32 * (offd[l] + ((k / 4) * tiles(l + 1) + j / 8) * 2 + part) + 4 * rot_col(j & 7) + (k & 3);
  }
  __host__ __device__ int trans_at(int m, int j, int k) const {
    return 32 * (offt[m] + (k / 4) * tiles(p + 1 - m) + j / 8) + 4 * rot_col(j & 7) + (k & 3);
  }
};

// The tile's row of one pair: degree l from base(l) on, the l + 1 real parts of m = 0..l, then the l
// imaginary parts; base(l) ≡ l (mod 4) and a row is an odd multiple of 4 doubles, so that the 8 pairs ×
// 4 orders (or 4 degrees of one order) a warp reads or writes at once lie in distinct banks
__host__ __device__ constexpr int rot_base(int l) { return l * l + 2 * (l / 2); }
__host__ __device__ constexpr int rot_row(int p) { return (rot_base(p + 1) + 3) / 4 * 4 | 4; }
// the row of the pair's (cos mφ, sin mφ): zeros past m = p for the padded inputs
__host__ __device__ constexpr int rot_cs(int p) { return (p + 4) / 8 * 8 + 5; }
constexpr int rot_list(int nc) { return 4 * nc + 2; }   // source, offset (bit 31: it points down), target, runs; the last run's end, their count

// fragments of a class's translations; its rotations have twice as many (RotLayout's nt and nd)
constexpr int rot_fragments(int p) {
  int n = 0;
  for (int s = 1; s <= p + 1; ++s) n += RotLayout::ksteps(s) * RotLayout::tiles(s);
  return n;
}
// the shared memory of a CTA: G groups of warps, NG groups of 8 pairs a chunk each
constexpr size_t rot_smem(int p, int NG, int G) {
  const int nc = 8 * NG, nt = rot_fragments(p);
  return sizeof(double) * ((size_t)32 * (2 * nt + G * nt) + (size_t)G * nc * (2 * rot_cs(p) + rot_row(p)) + 8) +
         sizeof(int) * (size_t)G * 2 * rot_list(nc);
}
// the CTAs of an SM: `most` (what the registers allow), or as many as fit its 228 KB, 1 KB of each the system's
constexpr int rot_resident(int p, int NG, int G, int most) {
  const int fit = (int)(size_t(228 * 1024) / (rot_smem(p, NG, G) + 1024));
  return fit < most ? fit : most;
}

struct RotHost {
  RotLayout layout;
  // per class of the far offsets, and (the last) for the direction (1, 1, 1) of the child slots:
  std::vector<double> d;                  // × 32·nd
  std::vector<double> cs;                 // × (p + 1) × (cos mφ, sin mφ), φ the representative's azimuth
  std::vector<double> csf, csk;           // the same of every far offset and child slot, times (−1)^m where it points down
};

std::shared_ptr<const RotHost> rotation_tables(int p, const HostOperators& op);

}  // namespace fmmb
