// The FP64 translations of the harmonic methods by rotations: M2L of the plain path (one launch for all
// levels), M2M and L2L of every path (a launch per level; src/device_passes.jl:565-580, the translations
// of harmonics.jl:531-645).
//
// Every translation operator is A = R⁻¹ T R exactly: R rotates the offset to the z axis (it mixes the
// orders of one degree), T translates along z (it mixes the degrees of one order). The dense product
// costs (p+1)⁴ multiply-adds per pair, the three factors 2(p+1)³: 2,673 against 14,641 at p = 10, 9,843
// against 83,521 at p = 16. R is a rotation by the offset's azimuth about z, a 2 × 2 rotation of each
// (n, m) by mφ (with the sign (−1)^(n+m) for offsets that point down), then one by the polar angle about
// y, which the offsets of a class share (M2M and L2L: all eight children).
// Per chunk of NC = 8·NG pairs of one class the inputs lie in a shared-memory tile [pair][entry], and the
// warps split the degrees (orders) between them:
//   rotate     per degree: z rotation of the inputs as they are read, then the product with the class's
//              (l + 1) × (l + 1) coefficients
//   translate  per order over the degrees, the real and the imaginary parts with the same coefficients
//   rotate     back with the same coefficients: R_y(−θ) = Σ R_y(θ) Σ, Σ = diag((−1)^m) (the right Σ
//              sits in T, the left one in the signs of the z rotation)
//   scatter    into the outputs: each target's entry takes its pairs one by one in the list's order,
//              starting from the value in memory (a target has one owner: deterministic, no atomics, and
//              the sums depend neither on where the chunks end nor on the other targets); the warp then
//              sends the next chunk's inputs (cp.async) into the rows it has read
// The products run on the FP64 tensor cores, 8 pairs × 4 inputs as A and the coefficients as B, laid out
// in fragments on the host; a fragment serves the NG groups of a chunk, where FMAs with a pair per lane read a
// coefficient per multiply-add (180 shared-memory wavefronts a pair at p = 10). The blocks of 1 to p + 1 pad the
// 8 × 8 × 4 tiles by half, which costs less than it saves. What bounds the kernel is the L1 / shared-memory pipe
// (two thirds busy: the tile is read and written three times) and instruction issue, not the FP64 rate (equal on
// the FMA units). Measured, M2L of a
// uniform cloud (FMAs with a pair per lane → this): 400,000 points p = 10 5.98 → 5.23 ms, p = 14 12.5 →
// 10.9, p = 16 19.8 → 15.2; 31,000 points on a sphere p = 16 0.66 → 0.55. The dense products before it:
// 9.4 ms at p = 10, 57 at p = 16. M2M and L2L (dense GEMMs → this):
// 0.146 → 0.071 and 0.103 → 0.083 ms at 400,000 points p = 10, 0.536 → 0.157 and 0.425 → 0.161 at p = 16.
// Loading the next step's operands ahead within a product spilled (5.4 → 7.7 ms).
#include <algorithm>
#include <numeric>
#include <type_traits>

#include "d4h.cuh"
#include "m2l_rot.h"
#include "passes.cuh"

namespace fmmb {

__constant__ int c_d4h[NFAR];
__constant__ int c_faroff[NFAR * 3];   // the far offsets, source cell − target cell

void upload_d4h(const HostOperators& h, cudaStream_t s) {
  std::vector<int> fac(h.d4h.begin(), h.d4h.end());
  require(fac.size() == NFAR, FMMB_ERR_DEVICE, "the D4h factor table has the wrong size");
  FMMB_CUDA(cudaMemcpyToSymbolAsync(c_d4h, fac.data(), sizeof(int) * NFAR, 0, cudaMemcpyHostToDevice, s));
  std::vector<int> off(h.faroff.begin(), h.faroff.end());
  require(off.size() == 3 * NFAR, FMMB_ERR_DEVICE, "the far offset table has the wrong size");
  FMMB_CUDA(cudaMemcpyToSymbolAsync(c_faroff, off.data(), sizeof(int) * 3 * NFAR, 0, cudaMemcpyHostToDevice, s));
}

namespace {

// the tasks by warp (largest first onto the least loaded warp): the rotations' degrees and the
// translations' orders
struct RotSched {
  RotLayout lay;
  uint8_t first[2][13];         // stage kind k, warp w: order[k][first[k][w]] .. order[k][first[k][w + 1] - 1]
  uint8_t order[2][PMAX + 1];
};

// the translation a launch performs: between far boxes, of the children's multipoles to their parent,
// of the parent's local to its children
enum : int { ROT_M2L = 0, ROT_M2M = 1, ROT_L2L = 2 };

// T of class c0 + blockIdx.x from its dense operator A (column-major, lda; stride per class):
// T^m_{ll'} = the (Re l m, Re l' m) entry of D A D⁻¹, negated for odd m on both sides' behalf (Σ
// above): a CTA per class and input degree l' = blockIdx.y, a thread per entry; T is zeroed by the caller.
// (M2M and L2L are one class each: with a CTA per class alone the first state of a cache took 1.5 ms at p = 16
// and 3.8 at p = 20, now 0.65 and 1.2.) Multipoles transform by the conjugate of the locals' rotation.
__global__ void k_rot_translations(const double* __restrict__ dense, int lda, int64_t stride, int mode, int c0,
                                   const double* __restrict__ dtab, const double* __restrict__ cstab, RotLayout lay,
                                   double* __restrict__ out) {
  const int p = lay.p, c = c0 + blockIdx.x, l2 = blockIdx.y;
  const double* A = dense + blockIdx.x * stride;
  const double sin_in = mode == ROT_L2L ? 1.0 : -1.0, sin_out = mode == ROT_M2M ? -1.0 : 1.0;
  const double* d = dtab + (int64_t)c * 32 * lay.nd;
  const double* cs = cstab + (int64_t)c * 2 * (p + 1);
  double* T = out + (int64_t)blockIdx.x * 32 * lay.nt;
  for (int i = threadIdx.x; i < (p + 1) * (p + 1); i += blockDim.x) {
    const int m = i % (p + 1), l = i / (p + 1);
    if (m > l || m > l2) continue;
    double sum = 0;
    for (int b = 0; b <= l2; ++b) {
      // the column of D⁻¹ = Z⁻¹ Σ d Σ: order b of degree l2 from (l2, m)
      const double v = d[lay.rot_at(l2, 0, b, m)] * ((m + b) & 1 ? -1.0 : 1.0);
      const double vr = cs[2 * b] * v, vi = sin_in * cs[2 * b + 1] * v;
      const double* Ar = A + (int64_t)(b == 0 ? l2 * l2 : l2 * l2 + 2 * b - 1) * lda;
      double col = 0;
      for (int a = 0; a <= l; ++a) {
        const int ra = a == 0 ? l * l : l * l + 2 * a - 1;
        double re = Ar[ra] * vr, im = a ? Ar[ra + 1] * vr : 0.0;
        if (b) {
          re += Ar[lda + ra] * vi;
          im += a ? Ar[lda + ra + 1] * vi : 0.0;
        }
        col += d[lay.rot_at(l, 0, m, a)] * (cs[2 * a] * re + sin_out * cs[2 * a + 1] * im);
      }
      sum += col;
    }
    T[lay.trans_at(m, l - m, l2 - m)] = m & 1 ? -sum : sum;
  }
}

__device__ __forceinline__ double flip(double x, int mask) {   // −x where mask is the sign bit
  return __hiloint2double(__double2hiint(x) ^ mask, __double2loint(x));
}

// one FP64 tensor-core MMA, D(8×8) += A(8×4)·B(4×8): this lane holds A[g][t], B[t][g] and
// D[g][2t], D[g][2t+1] (g = lane / 4, t = lane % 4)
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// the rotation of degree l of NG groups of 8 pairs, in place: r, cs: this lane's pair of the first
// group (pair g), PT and PM apart per pair; B: the degree's fragments at this lane; down: per group
// the sign bit where the pair's offset points down; BACK: the z rotation after the product (to the
// offset's azimuth) instead of before it. The imaginary parts of multipoles are negated on the way in
// (not in ROT_L2L, whose inputs are locals) and on the way out where the output is one (ROT_M2M):
// Tᵐ then acts on the real and the imaginary parts alike.
template <int MODE, int P, int RT, int NG, bool BACK>
__device__ __forceinline__ void rotate_degree(int l, int t, double* r, const double2* cs, const double* __restrict__ B,
                                              const int (&down)[NG]) {
  constexpr int PT = rot_row(P), PM = rot_cs(P);
  double ar[NG][RT][2], ai[NG][RT][2];
#pragma unroll
  for (int q = 0; q < NG; ++q)
#pragma unroll
    for (int i = 0; i < RT; ++i) ar[q][i][0] = ar[q][i][1] = ai[q][i][0] = ai[q][i][1] = 0.0;
  double* re = r + rot_base(l);
  double* im = re + l;                                   // the imaginary part of m at im[m]
  const int odd = l & 1;
#pragma unroll 1
  for (int k = t; k - t <= l; k += 4, B += 64 * RT) {
    double br[RT], bi[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) { br[i] = B[64 * i]; bi[i] = B[64 * i + 32]; }
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      double xr = re[8 * q * PT + k], xi = im[8 * q * PT + k];
      if (!BACK) {
        double2 z = cs[8 * q * PM + k];
        if (odd) { z.x = flip(z.x, down[q]); z.y = flip(z.y, down[q]); }
        const double x = MODE == ROT_L2L ? -xi : xi, u = z.x * xr - z.y * x;
        xi = -(z.y * xr + z.x * x);
        xr = u;
      }
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        dmma(ar[q][i], xr, br[i]);
        dmma(ai[q][i], xi, bi[i]);
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < NG; ++q)
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int m = 8 * i + t + 4 * e;
        double a = ar[q][i][e], b = ai[q][i][e];
        if (BACK && m <= l) {
          double2 z = cs[8 * q * PM + m];
          if (odd) { z.x = flip(z.x, down[q]); z.y = flip(z.y, down[q]); }
          const int sg = (m & 1) << 31;                  // Σ
          const double u = z.x * a - z.y * b, v = z.y * a + z.x * b;
          a = flip(u, sg);
          b = flip(MODE == ROT_M2M ? -v : v, sg);
        }
        if (m <= l) re[8 * q * PT + m] = a;
        if (m <= l && m > 0) im[8 * q * PT + m] = b;
      }
}

// the translation of order m over the degrees m..p, in place
template <int P, int RT, int NG>
__device__ __forceinline__ void translate_order(int m, int t, double* r, const double* __restrict__ B) {
  constexpr int p = P, PT = rot_row(P);
  double ar[NG][RT][2], ai[NG][RT][2];
#pragma unroll
  for (int q = 0; q < NG; ++q)
#pragma unroll
    for (int i = 0; i < RT; ++i) ar[q][i][0] = ar[q][i][1] = ai[q][i][0] = ai[q][i][1] = 0.0;
#pragma unroll 1
  for (int l0 = m; l0 <= p; l0 += 4, B += 32 * RT) {
    const int l = min(l0 + t, p);                        // past p: zero coefficients
    const double* x = r + rot_base(l) + m;
    const int im = m ? l : 0;                            // m = 0 has no imaginary parts
    double b[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) b[i] = B[32 * i];
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const double xr = x[8 * q * PT], xi = x[8 * q * PT + im];
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        dmma(ar[q][i], xr, b[i]);
        if (m) dmma(ai[q][i], xi, b[i]);
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int l = m + 8 * i + t + 4 * e;
      if (l <= p) {
        double* y = r + rot_base(l) + m;
#pragma unroll
        for (int q = 0; q < NG; ++q) {
          y[8 * q * PT] = ar[q][i][e];
          if (m) y[8 * q * PT + l] = ai[q][i][e];
        }
      }
    }
}

template <int MODE, int P, int NG, bool BACK>
__device__ __forceinline__ void rotate_any(int l, int t, double* r, const double2* cs, const double* B, const int (&down)[NG]) {
  if (P < 8 || l < 8) rotate_degree<MODE, P, 1, NG, BACK>(l, t, r, cs, B, down);
  else if (P < 16 || l < 16) rotate_degree<MODE, P, 2, NG, BACK>(l, t, r, cs, B, down);
  else rotate_degree<MODE, P, 3, NG, BACK>(l, t, r, cs, B, down);
}
template <int P, int NG>
__device__ __forceinline__ void translate_any(int m, int t, double* r, const double* B) {
  const int s = P + 1 - m;
  if (P < 8 || s <= 8) translate_order<P, 1, NG>(m, t, r, B);
  else if (P < 16 || s <= 16) translate_order<P, 2, NG>(m, t, r, B);
  else translate_order<P, 3, NG>(m, t, r, B);
}

__device__ __forceinline__ void cpa16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cpa8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

struct RotArgs {
  RotSched sch;
  const double* dtab;                   // the rotations' fragments by class
  const double2* cst;                   // per far offset, or child slot, (cos mφ, sin mφ)
  int LD, stokes;
  int64_t pitch;
  const double* in;                     // multipoles (the parents' locals for ROT_L2L)
  double* out;                          // locals (the parents' multipoles for ROT_M2M)
  // ROT_M2L: the blocks, `sub` parts of TB / sub targets each, and per level the translations
  int nparts, sub, TB;
  const int4* blocks;
  const int *cls_off, *rtab;
  const int2* pairs;
  const uint64_t* lv_trans;
  const double* m2l_scale;
  // ROT_M2M, ROT_L2L: the level's sibling groups (children c0 .., eight each, of the parents gp), a
  // multiple of eight children per CTA, the translation
  int c0, nchild, per;
  const int* gp;
  const double* trans;
};

// NG groups of 8 pairs per chunk, G groups of NW warps. The order is a template argument: with the tile's
// pitches known the addresses are immediates (M2L, 400,000 points, the order an argument → this: p = 3
// 2.25 → 1.88 ms, p = 6 3.34 → 2.95, p = 10 5.42 → 5.23, p = 16 16.5 → 15.2, p = 20 120,000 points 3.98 → 3.36:
// of 460 instructions a pair and warp at p = 10 two thirds were integer).
template <int MODE, int P, int NG, int G, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW * G, MINB) k_rot(const __grid_constant__ RotArgs A) {
  static_assert(MINB <= rot_resident(P, NG, G, MINB), "the CTAs that the launch counts on fit an SM");
  static_assert(MODE == ROT_M2L || G == 1, "one group of warps per CTA in the sweeps");
  const RotSched& sch = A.sch;
  constexpr int NC = 8 * NG, NT = 32 * NW, NL = rot_list(NC);
  constexpr int p = P, NP = (P + 1) * (P + 1), NE = (NP + 31) / 32, PT = rot_row(P), PM = rot_cs(P);
  const int nd = 32 * sch.lay.nd, nt = 32 * sch.lay.nt;
  const int tid = threadIdx.x % NT, grp = threadIdx.x / NT, warp = tid >> 5, lane = tid & 31;
  const int comp = blockIdx.y, psi = A.stokes && comp == 3, LD = A.LD;
  const int64_t pitch = A.pitch;
  extern __shared__ __align__(16) double sm[];
  double* D = sm;                                        // the class's rotation
  double* T = D + nd + grp * nt;                         // the group's translation
  double2* cs0 = (double2*)(D + nd + G * nt);
  double2* cs = cs0 + (size_t)grp * NC * PM;             // [pair][order]
  double* tile0 = (double*)(cs0 + (size_t)G * NC * PM);
  double* tile = tile0 + (size_t)grp * NC * PT;          // [pair][entry], 8 doubles past the last row
  int* list = (int*)(tile0 + (size_t)G * NC * PT + 8) + grp * 2 * NL;
  // the padding stays zero: it meets zero coefficients
  for (int i = threadIdx.x; i < G * NC * (2 * PM + PT) + 8; i += NT * G) ((double*)cs0)[i] = 0.0;
  __syncthreads();
  // where this lane's entries e = lane + 32k of an expansion lie in a row
  int loc[NE];
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    int n, m, part;
    coef_nmp(lane + 32 * k, n, m, part);
    loc[k] = rot_base(n) + m + (part == 2 ? n : 0);
  }
  auto gsync = [&] {
    if constexpr (G == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(NT) : "memory");
  };
  // part q of block blk: its targets [t0, t1), whose pairs are consecutive in every class
  const int part = blockIdx.x * G + grp;
  const bool on = MODE != ROT_M2L || part < A.nparts;
  int blk = 0, t0 = 0, t1 = 0;
  int4 b = make_int4(0, 0, 0, 0);
  double alpha = 1.0;
  const double* lt = A.trans;
  if constexpr (MODE == ROT_M2L) {
    blk = part / A.sub;
    t0 = part % A.sub * (A.TB / A.sub);
    t1 = t0 + A.TB / A.sub;
    if (on) b = A.blocks[blk];
    alpha = on ? A.m2l_scale[b.x & 255] : 0.0;
    lt = reinterpret_cast<const double*>(A.lv_trans[b.x & 255]);
  }
  const double* Mc = A.in + (int64_t)comp * LD;
  double* Pc = A.out + (int64_t)b.y * pitch + (int64_t)comp * LD;

  // pair j of a list: its multipole into the tile's row j, its azimuth's table into the columns j
  auto gather = [&](const int* L, int j) {
    double* row = tile + j * PT;
    const int f = L[NC + j] & 0xffff;
    const double* src = Mc + (int64_t)L[j] * pitch;
    if (psi) {
      // the Stokes Ψ̂ block takes Ψ̂ + o·Φ of a far box at offset o, ½Ψ̂ + δ̂·Φ of a child and
      // 2Ψ̂ − 2δ̂·Φ of a parent, δ̂ the child's offset (harmonics_stokes.jl:77-129)
      const double* phi = A.in + (int64_t)L[j] * pitch;
      double o[3], c = MODE == ROT_M2M ? 0.5 : (MODE == ROT_L2L ? 2.0 : 1.0);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (MODE == ROT_M2L) o[d] = c_faroff[3 * f + d];
        else o[d] = (f >> d & 1 ? 0.25 : -0.25) * (MODE == ROT_L2L ? -2.0 : 1.0);
      }
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const int e = lane + 32 * k;
        if (e < NP)
          row[loc[k]] = fma(o[2], __ldg(phi + 2 * LD + e),
                            fma(o[1], __ldg(phi + LD + e), fma(o[0], __ldg(phi + e), c * __ldg(src + e))));
      }
    } else {
#pragma unroll
      for (int k = 0; k < NE; ++k)
        if (lane + 32 * k < NP) cpa8(row + loc[k], src + lane + 32 * k);
    }
    if (lane <= p) cpa16(cs + j * PM + lane, A.cst + f * (p + 1) + lane);
  };
  // the chunk's pairs read by the group's first warp, then into the list with the runs of one target
  // (the pairs of a class are grouped by target)
  auto fetch = [&](int q0, int nc) {                     // source, offset or child slot, target (−1: none)
    if (lane >= nc) return make_int3(0, 0, -1);
    const int q = q0 + lane;
    if constexpr (MODE == ROT_M2L) {
      const int2 pr = A.pairs[b.w + q];
      return make_int3(pr.x, pr.y >> 8, pr.y & 0xff);
    } else {
      const int c = A.c0 + q, pa = A.gp[q >> 3];
      return MODE == ROT_M2M ? make_int3(c, q & 7, pa) : make_int3(pa, q & 7, c);
    }
  };
  auto commit = [&](int* L, int nc, int3 pr) {
    const int prev = __shfl_up_sync(0xffffffffu, pr.z, 1);
    const bool start = lane < nc && (lane == 0 || pr.z != prev);
    const unsigned bal = __ballot_sync(0xffffffffu, start);
    if (lane < NC) {
      const bool down = MODE == ROT_M2L ? c_faroff[3 * pr.y + 2] < 0 : !(pr.y >> 2);
      L[lane] = pr.x;
      L[NC + lane] = pr.y | (int)down << 31;
      L[2 * NC + lane] = pr.z;
    }
    if (start) L[3 * NC + __popc(bal & ((1u << lane) - 1u))] = lane;
    if (lane == 0) { L[3 * NC + __popc(bal)] = nc; L[4 * NC + 1] = __popc(bal); }
  };
  static_assert(NC <= 32, "a lane per pair of a chunk");
  const int g = lane >> 2, t = lane & 3;
  double* row0 = tile + g * PT;                          // this lane's pair of the first 8
  const double2* cs_g = cs + g * PM;

  for (int c = 0; c < (MODE == ROT_M2L ? NCLASS : 1); ++c) {
    int a0 = 0, a1 = 0;
    if constexpr (MODE == ROT_M2L) {
      const int* co = A.cls_off + (int64_t)(on ? blk : 0) * (NCLASS + 1);
      const int* rt = A.rtab + ((int64_t)blk * NCLASS + c) * A.TB;
      if (on) {
        a0 = co[c] + (t0 ? rt[t0] & 0xffff : 0);
        a1 = t1 < A.TB ? co[c] + (rt[t1] & 0xffff) : co[c + 1];
      }
    } else {
      a0 = part * A.per;
      a1 = min(A.nchild, a0 + A.per);
    }
    if constexpr (G == 1) {
      if (a0 == a1) continue;
    } else {
      if (!__syncthreads_or(a0 < a1)) continue;          // no group is still in the previous class
    }
    // the class's tables, the first chunk's list and multipoles
    {
      const double* src = A.dtab + (int64_t)(MODE == ROT_M2L ? c : NCLASS) * nd;
      for (int i = 2 * threadIdx.x; i < nd; i += 2 * NT * G) cpa16(D + i, src + i);
      const double* ts = lt + (int64_t)c * nt;
      if (a0 < a1)                                       // an idle group has no level
        for (int i = 2 * tid; i < nt; i += 2 * NT) cpa16(T + i, ts + i);
    }
    if (warp == 0 && a0 < a1) {
      commit(list, min(NC, a1 - a0), fetch(a0, min(NC, a1 - a0)));
    }
    gsync();
    for (int j = warp; j < min(NC, a1 - a0); j += NW) gather(list, j);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    int cur = 0;
    for (int q0 = a0; q0 < a1; q0 += NC, cur ^= 1) {
      const int* L = list + cur * NL;
      int* Ln = list + (cur ^ 1) * NL;
      const int nn = min(NC, a1 - q0 - NC);              // the next chunk's pairs (≤ 0: none in this class)
      int3 pr;
      if (warp == 0 && nn > 0) pr = fetch(q0 + NC, nn);
      int down[NG];
#pragma unroll
      for (int k = 0; k < NG; ++k) down[k] = L[NC + 8 * k + g] & (int)0x80000000;
#pragma unroll 1
      for (int i = sch.first[0][warp]; i < sch.first[0][warp + 1]; ++i) {
        const int l = sch.order[0][i];
        rotate_any<MODE, P, NG, false>(l, t, row0, cs_g, D + 32 * sch.lay.offd[l] + lane, down);
      }
      if (warp == 0 && nn > 0) commit(Ln, nn, pr);
      gsync();
#pragma unroll 1
      for (int i = sch.first[1][warp]; i < sch.first[1][warp + 1]; ++i) {
        const int m = sch.order[1][i];
        translate_any<P, NG>(m, t, row0, T + 32 * sch.lay.offt[m] + lane);
      }
      gsync();
#pragma unroll 1
      for (int i = sch.first[0][warp]; i < sch.first[0][warp + 1]; ++i) {
        const int l = sch.order[0][i];
        rotate_any<MODE, P, NG, true>(l, t, row0, cs_g, D + 32 * sch.lay.offd[l] + lane, down);
      }
      gsync();
      // scatter: a warp the runs w, w + NW, ..., the entries across the lanes; then the next chunk's
      // multipoles into the rows it has read
      const int nrun = L[4 * NC + 1];
      if constexpr (MODE == ROT_M2M) {
        // few runs (a parent's eight children are one): a warp a run's 32 entries at a time, and the next
        // chunk's rows over all warps. A parent's multipole starts from zero.
        for (int r = 0; r < nrun; ++r) {
          const int j0 = L[3 * NC + r], j1 = L[3 * NC + r + 1];
          double* dst = Pc + (int64_t)L[2 * NC + j0] * pitch;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            if ((r * NE + k) % NW != warp || lane + 32 * k >= NP) continue;
            double v = 0.0;
            for (int j = j0; j < j1; ++j) v = fma(alpha, tile[j * PT + loc[k]], v);
            dst[lane + 32 * k] = v;
          }
        }
        if (nn > 0) {
          gsync();
          for (int j = warp; j < nn; j += NW) gather(Ln, j);
        }
      } else {
        for (int r = warp; r < nrun; r += NW) {
          const int j0 = L[3 * NC + r], j1 = L[3 * NC + r + 1];
          double* dst = Pc + (int64_t)L[2 * NC + j0] * pitch;
          double v[NE];
#pragma unroll
          for (int k = 0; k < NE; ++k) v[k] = lane + 32 * k < NP ? dst[lane + 32 * k] : 0.0;
          for (int j = j0; j < j1; ++j)
#pragma unroll
            for (int k = 0; k < NE; ++k)
              if (lane + 32 * k < NP) v[k] = fma(alpha, tile[j * PT + loc[k]], v[k]);
#pragma unroll
          for (int k = 0; k < NE; ++k)
            if (lane + 32 * k < NP) dst[lane + 32 * k] = v[k];
          if (nn > 0) {
            __syncwarp();
            for (int j = j0; j < min(j1, nn); ++j) gather(Ln, j);
          }
        }
      }
      // rows past this chunk's last pair (a next chunk is longer only when this one is full)
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
      gsync();
    }
  }
}

// f(std::integral_constant<int, p>)
template <class F>
void for_order(int p, F&& f) {
  switch (p) {
#define X(pp) case pp: f(std::integral_constant<int, pp>()); break;
    FMMB_P_CASES(X)
#undef X
    default: throw Error(FMMB_ERR_UNSUPPORTED, "p out of range");
  }
}

RotSched schedule(const RotLayout& lay, int nw) {
  RotSched s{};
  s.lay = lay;
  for (int kind = 0; kind < 2; ++kind) {
    // the MMAs of degree l, of order m (half of them for m = 0), and a task's fixed part
    std::vector<int> cost(lay.p + 1), id(lay.p + 1);
    for (int i = 0; i <= lay.p; ++i) {
      const int q = kind == 0 ? i + 1 : lay.p + 1 - i;
      cost[i] = (kind == 1 && i == 0 ? 1 : 2) * RotLayout::ksteps(q) * RotLayout::tiles(q) + 2;
      id[i] = i;
    }
    std::stable_sort(id.begin(), id.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::vector<std::vector<int>> of(nw);
    std::vector<int> load(nw, 0);
    for (int i : id) {
      const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      of[w].push_back(i);
      load[w] += cost[i];
    }
    int k = 0;
    for (int w = 0; w < nw; ++w) {
      s.first[kind][w] = (uint8_t)k;
      for (int i : of[w]) s.order[kind][k++] = (uint8_t)i;
    }
    s.first[kind][nw] = (uint8_t)k;
  }
  return s;
}

// The parts a block is cut into: more of them fill the device and cut the heaviest block (a cluster's hold twenty
// times the average), fewer of them fill the chunks (a class's last chunk of a part is half empty, and one with
// few pairs costs a whole one): the power of two with the least time, in chunks per class, of all parts over the
// groups of warps that run at once (`slots`, `per_sm` of them on an SM) and of the heaviest block's on its own (the
// fewer groups share its SM, the faster it runs: a twelfth per group). Of a class's λ pairs on average, a part has
// any with probability 1 − e^−λ. Fitted to every power of two at 315 sets (p = 4 to 20; 1,200 to 400,000 points,
// uniform, on a sphere and in clusters; ppl 24 to 300): 2 % above the best of them on average, and nowhere above the
// rule that looked at the average block alone, which took up to 2.8 times the best. M2L, that rule → this: 150,000 points
// in clusters p = 8 3.29 → 1.93 ms, p = 14 4.99 → 3.43, p = 20 15.9 → 8.1; uniform clouds and spheres within 1 %.
int parts_per_block(const Plan& P, int nexp, int slots, int per_sm, int nc) {
  const double nb = (double)P.h_blocks.size();
  int best = 1;
  double least = 1e300;
  for (int sub = 1; sub <= P.TB / 4; sub *= 2) {
    auto chunks = [&](double pairs, double last) {
      const double lam = pairs / (sub * NCLASS), any = 1 - std::exp(-lam);
      return std::max(any, lam / nc + last * any);
    };
    const double t = std::max(nb * sub * nexp / slots * chunks(P.npairs / nb, 0.75),
                              chunks((double)P.max_block_pairs, 0.5) / (1 + 0.08 * (per_sm - 1)));
    if (t < 0.97 * least) { least = t; best = sub; }
  }
  return best;
}

template <int MODE, int P, int NG, int G, int NW, int MINB>
void start(RotArgs& A, const RotHost& R, int ctas, int nexp, cudaStream_t s) {
  A.sch = schedule(R.layout, NW);
  const size_t smem = rot_smem(P, NG, G);
  auto kern = k_rot<MODE, P, NG, G, NW, MINB>;
  FMMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<dim3(ctas, nexp), 32 * NW * G, smem, s>>>(A);
  FMMB_LAUNCH_CHECK();
}

RotArgs common_args(State& S, const double* cst, const double* in, double* out) {
  Cache& K = *S.plan->cache;
  RotArgs A{};
  A.dtab = K.rot_d.p;
  A.cst = (const double2*)cst;
  A.LD = K.ld;
  A.stokes = K.nexp == 4;
  A.pitch = (int64_t)K.nexp * K.ld;
  A.in = in;
  A.out = out;
  return A;
}

template <int ORD, int NG, int G, int NW, int MINB>
void launch(State& S) {
  Plan& P = *S.plan;
  Cache& K = *P.cache;
  const int nb = (int)P.h_blocks.size();
  if (nb == 0) return;
  RotArgs A = common_args(S, K.rot_csf.p, S.M.p, S.Pl.p);
  A.sub = parts_per_block(P, K.nexp, P.ctx->num_sms * MINB * G, MINB * G, 8 * NG);
  A.nparts = nb * A.sub;
  A.TB = P.TB;
  A.blocks = P.blocks.p;
  A.cls_off = P.cls_off.p;
  A.rtab = P.rtab.p;
  A.pairs = P.pairs.p;
  A.lv_trans = P.d_lv_rot.p;
  A.m2l_scale = P.d_m2l_scale.p;
  start<ROT_M2L, ORD, NG, G, NW, MINB>(A, *K.rot, (A.nparts + G - 1) / G, K.nexp, P.ctx->stream);
}

// the children of level l (into their parents, or from them): chunks spread over the CTAs that run at once
template <int MODE, int ORD, int NG, int NW, int MINB>
void launch_sweep(State& S, int l, const double* trans) {
  Plan& P = *S.plan;
  Cache& K = *P.cache;
  RotArgs A = MODE == ROT_M2M ? common_args(S, K.rot_csk.p, S.M.p, S.M.p) : common_args(S, K.rot_csk.p, S.Pl.p, S.Pl.p);
  A.c0 = P.level_start[l];
  A.nchild = NCH * P.level_groups[l];
  A.gp = P.group_parent[l].p;
  A.trans = trans;
  const int slots = std::max(1, P.ctx->num_sms * MINB / K.nexp), chunks = (A.nchild + 8 * NG - 1) / (8 * NG);
  A.per = 8 * NG * ((chunks + slots - 1) / slots);
  start<MODE, ORD, NG, 1, NW, MINB>(A, *K.rot, (A.nchild + A.per - 1) / A.per, K.nexp, P.ctx->stream);
}

template <int MODE>
void sweep(State& S, int l, const double* trans) {
  auto go = [&](auto order) {
    constexpr int P = decltype(order)::value, NG = P <= 15 ? 3 : 2;
    launch_sweep<MODE, P, NG, P <= 11 ? 4 : (P <= 15 ? 6 : 8), rot_resident(P, NG, 1, P <= 11 ? 4 : (P <= 15 ? 2 : 1))>(S, l, trans);
  };
  for_order(S.plan->cache->p, go);
}

// the translations along z of n classes (c0 ..) from their dense operators
void translations(Cache& C, const RotLayout& lay, int mode, int c0, int n, const double* dense, int lda, int64_t stride,
                  DBuf<double>& out, cudaStream_t s) {
  out.alloc((size_t)n * 32 * lay.nt);
  FMMB_CUDA(cudaMemsetAsync(out.p, 0, out.bytes(), s));
  k_rot_translations<<<dim3(n, lay.p + 1), 128, 0, s>>>(dense, lda, stride, mode, c0, C.rot_d.p, C.rot_cs.p, lay, out.p);
  FMMB_LAUNCH_CHECK();
}
void all_translations(Cache& C, const RotLayout& lay, const double* reps, const double* m2m, const double* l2l,
                      RotTrans& t, cudaStream_t s) {
  const int LD = C.ld;
  translations(C, lay, ROT_M2L, 0, NCLASS, reps, LD, (int64_t)LD * LD, t.m2l, s);
  // of the child slot (1, 1, 1), the last: the direction the rotation is built for
  translations(C, lay, ROT_M2M, NCLASS, 1, m2m + (int64_t)7 * LD * LD, LD, 0, t.m2m, s);
  translations(C, lay, ROT_L2L, NCLASS, 1, l2l + (int64_t)7 * LD, NCH * LD, 0, t.l2l, s);
}

}  // namespace

// the tables of the FP64 translations: the cache's rotations (uploaded with its first state) and per
// level the translations along z (the cache's for the homogeneous kernels, the level width's own for
// Yukawa3D). The cache is locked by the caller.
void prepare_rotations(Plan& P) {
  Cache& C = *P.cache;
  cudaStream_t s = P.ctx->stream;
  if (P.d_lv_rot.n) return;
  if (!C.rot) {
    auto h = rotation_tables(C.p, C.host);
    to_device(C.rot_d, h->d, s);
    to_device(C.rot_cs, h->cs, s);
    to_device(C.rot_csf, h->csf, s);
    to_device(C.rot_csk, h->csk, s);
    if (C.kernel != FMMB_KERNEL_YUKAWA3D) all_translations(C, h->layout, C.reps.p, C.m2m.p, C.l2l.p, C.rot_t, s);
    C.rot = h;
  }
  std::vector<uint64_t> t(P.L, 0);
  P.lv_rot_m2m.assign(P.L, nullptr);
  P.lv_rot_l2l.assign(P.L, nullptr);
  for (int l = 0; l < P.L; ++l) {
    const RotTrans* r = nullptr;
    if (C.kernel != FMMB_KERNEL_YUKAWA3D) {
      r = &C.rot_t;
    } else if (l >= 2 && l < (int)P.lv_yukawa.size() && P.lv_yukawa[l]) {
      YukawaLevel& Y = *P.lv_yukawa[l];
      std::lock_guard<std::mutex> lk(Y.mu);
      if (!Y.rot_t.l2l.n) {
        // shared by caches on other streams: outside the stream-ordered pool, complete before use
        const cudaStream_t keep = g_alloc_stream;
        g_alloc_stream = nullptr;
        try {
          all_translations(C, C.rot->layout, Y.reps.p, Y.m2m.p, Y.l2l.p, Y.rot_t, s);
          FMMB_CUDA(cudaStreamSynchronize(s));
        } catch (...) {
          Y.rot_t = RotTrans();
          g_alloc_stream = keep;
          throw;
        }
        g_alloc_stream = keep;
      }
      r = &Y.rot_t;
    }
    if (!r) continue;                                    // no translations touch the level
    t[l] = (uint64_t)(uintptr_t)r->m2l.p;
    P.lv_rot_m2m[l] = r->m2m.p;
    P.lv_rot_l2l[l] = r->l2l.p;
  }
  to_device(P.d_lv_rot, t, s);
}

// the children of level l + 1 into the parents of level l; the parents' locals of level l − 1 into the
// children of level l
void m2m_rot(State& S, int l) { sweep<ROT_M2M>(S, l + 1, S.plan->lv_rot_m2m[l]); }
void l2l_rot(State& S, int l) { sweep<ROT_L2L>(S, l, S.plan->lv_rot_l2l[l - 1]); }

// (Measured with the order an argument.) Chunks of 24 pairs and two to four CTAs per SM while the tiles
// and tables fit (400,000 points p = 10:
// 5.42 ms, sphere of 30,000 0.49; chunks of 16 6.42 and 0.50; two groups with chunks of 32 5.50 and 0.65.
// p = 14: 11.6; chunks of 16 14.4; four warps instead of six 13.8). Three CTAs fit at p = 11 (400,000 points: 8.33 ms, 8.49
// with the registers and parts of four; M2M and L2L 0.095 and 0.111 → 0.081 and 0.095). From p = 16 on one CTA
// runs (of chunks of 16 two would fit at p = 16 by shared memory, and one by its 209 registers a thread). At p = 16 two
// groups of warps with chunks of 24 share the rotations, one computing while the other scatters, as long as there
// are pairs enough for that many chunks (one group's time over two groups': uniform clouds 0.55 at 56,448 pairs, 0.84 at
// 184,722, 1.03 at 601,701, 1.09 at 640,584, 1.37 at 2.3M; spheres 0.94 at 308,559, 1.07 at 668,268, 1.19 at 1.4M; Gaussian
// mixtures 0.94 at 381,317, 0.96 at 627,320, 1.05 at 1.06M, 1.34 at 3.1M).
void m2l_rot(State& S) {
  const bool many = (int64_t)S.plan->npairs * S.plan->cache->nexp >= 600000;
  for_order(S.plan->cache->p, [&](auto order) {
    constexpr int P = decltype(order)::value;
    if constexpr (P <= 11) launch<P, 3, 1, 4, rot_resident(P, 3, 1, 4)>(S);
    else if constexpr (P <= 15) launch<P, 3, 1, 6, rot_resident(P, 3, 1, 2)>(S);
    else if (P == 16 && many) launch<16, 3, 2, 6, 1>(S);
    else launch<P, 2, 1, 8, 1>(S);
  });
}

}  // namespace fmmb
