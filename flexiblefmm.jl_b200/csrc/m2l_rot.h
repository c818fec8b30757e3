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

struct RotHost {
  RotLayout layout;
  // per class of the far offsets, and (the last) for the direction (1, 1, 1) of the child slots:
  std::vector<double> d;                  // × 32·nd
  std::vector<double> cs;                 // × (p + 1) × (cos mφ, sin mφ), φ the representative's azimuth
  std::vector<double> csf, csk;           // the same of every far offset and child slot, times (−1)^m where it points down
};

std::shared_ptr<const RotHost> rotation_tables(int p, const HostOperators& op);

}  // namespace fmmb
