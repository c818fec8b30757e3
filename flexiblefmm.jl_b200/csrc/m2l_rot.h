// The tables of the FP64 M2L by rotations (rotations.cpp, m2l_rot.cu).
#pragma once
#include <memory>

#include "common.cuh"

namespace fmmb {

// a block's columns start on 16 bytes
__host__ __device__ constexpr int rot_pad(int s) { return (s + 1) & ~1; }

// Where the blocks of one class lie: per degree l the rotation's, column-major, column k (the input
// order) holding the l + 1 output orders' real parts and, for k ≥ 1, the l imaginary parts; per
// order m the translation's, column-major over the degrees m..p
struct RotLayout {
  int p = 0, nd = 0, nt = 0;              // doubles per class: rotations, translations
  uint16_t offd[PMAX + 1], offt[PMAX + 1];
  __host__ __device__ int re_col(int l, int k) const {   // the real parts of column k of degree l
    return offd[l] + k * rot_pad(l + 1) + (k ? k - 1 : 0) * rot_pad(l);
  }
};

struct RotHost {
  RotLayout layout;
  std::vector<double> d;                  // classes × nd
  std::vector<double> cs;                 // classes × (p + 1) × (cos mφ, sin mφ), φ the representative's azimuth
  std::vector<double> csf;                // the same of every far offset, times (−1)^m where it points down
};

std::shared_ptr<const RotHost> rotation_tables(int p, const HostOperators& op);
// the Gauss–Legendre rule on [−1, 1] of n points
void gauss_legendre(int n, std::vector<double>& t, std::vector<double>& w);

}  // namespace fmmb
