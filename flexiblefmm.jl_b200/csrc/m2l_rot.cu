// M2L of the plain FP64 path by rotations: one launch for all levels, a CTA of G groups of warps,
// each group the far pairs of one block of targets (src/device_passes.jl:565-580, the class-wise
// translation of harmonics.jl:531-645).
//
// A class representative is A_c = R_cᵀ T_c R_c exactly, and so is every far offset's translation:
// R rotates the offset to the z axis (it mixes the orders of one degree), T_c translates along z (it
// mixes the degrees of one order). The dense product costs (p+1)⁴ multiply-adds per pair, the three
// factors 2(p+1)³: 2,673 against 14,641 at p = 10, 9,843 against 83,521 at p = 16. R is a rotation by
// the offset's azimuth about z, a 2 × 2 rotation of each (n, m) by mφ (with the sign (−1)^(n+m) for
// offsets that point down), then one by the polar angle about y, which the class's offsets share.
// Per class and chunk of NC = 32·C pairs the multipoles lie in a shared-memory tile [pair][entry],
// a lane owns C pairs, and the warps split the degrees (orders) between them:
//   rotate     per degree: z rotation of the column read, then y_j += d_jk x_k in registers, the
//              class's coefficients broadcast from shared memory
//   translate  per order over the degrees, the real and the imaginary parts with the same
//              coefficients
//   rotate     back with the same coefficients: R_y(−θ) = Σ R_y(θ) Σ, Σ = diag((−1)^m) (the right Σ
//              sits in T_c, the left one in the signs of the z rotation)
//   scatter    into the targets' partial locals: each target's entry takes its pairs one by one in
//              the list's order, starting from the value in memory (the block owns its targets:
//              deterministic, no atomics, and the sums depend neither on where the chunks end nor on
//              the other targets of the block); the warp then sends the next chunk's multipoles
//              (cp.async) into the rows it has read
// The products are FP64 FMAs with the pairs across the lanes: blocks of 1 to p + 1 would fill a third
// to two thirds of the 8 × 8 × 4 tiles of the FP64 tensor cores, whose rate is the FMA units'. What
// bounds it is shared memory: the tile is read and written three times per pair, and each
// coefficient's broadcast serves C pairs per lane.
#include <algorithm>
#include <numeric>

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

// T_c of one class from its dense representative: T^m_{ll'} = the (Re l m, Re l' m) entry of
// D A D⁻¹, negated for odd m on both sides' behalf (Σ above): a thread per entry
__global__ void k_rot_translations(const double* __restrict__ reps, const double* __restrict__ dtab,
                                   const double* __restrict__ cstab, RotLayout lay, int LD, double* __restrict__ out) {
  const int p = lay.p, c = blockIdx.x;
  const double* A = reps + (int64_t)c * LD * LD;
  const double* d = dtab + (int64_t)c * lay.nd;
  const double* cs = cstab + (int64_t)c * 2 * (p + 1);
  double* T = out + (int64_t)c * lay.nt;
  for (int i = threadIdx.x; i < lay.nt; i += blockDim.x) T[i] = 0.0;
  __syncthreads();
  const int np = (p + 1) * (p + 1) * (p + 1);
  for (int i = threadIdx.x; i < np; i += blockDim.x) {
    const int m = i % (p + 1), l = i / (p + 1) % (p + 1), l2 = i / ((p + 1) * (p + 1));
    if (m > l || m > l2) continue;
        double sum = 0;
    for (int b = 0; b <= l2; ++b) {
      // the column of D⁻¹ = Z⁻¹ Σ d Σ: order b of degree l2 from (l2, m)
      const double v = d[lay.re_col(l2, m) + b] * ((m + b) & 1 ? -1.0 : 1.0);
      const double vr = cs[2 * b] * v, vi = -cs[2 * b + 1] * v;
      const double* Ar = A + (int64_t)(b == 0 ? l2 * l2 : l2 * l2 + 2 * b - 1) * LD;
      double col = 0;
      for (int a = 0; a <= l; ++a) {
        const int ra = a == 0 ? l * l : l * l + 2 * a - 1;
        double re = Ar[ra] * vr, im = a ? Ar[ra + 1] * vr : 0.0;
        if (b) {
          re += Ar[LD + ra] * vi;
          im += a ? Ar[LD + ra + 1] * vi : 0.0;
        }
        col += d[lay.re_col(l, a) + m] * (cs[2 * a] * re + cs[2 * a + 1] * im);
      }
      sum += col;
    }
    // column l2 − m, row l − m of the block of order m
    T[lay.offt[m] + (l2 - m) * rot_pad(p + 1 - m) + (l - m)] = m & 1 ? -sum : sum;
  }
}

__device__ __forceinline__ double flip(double x, int mask) {   // −x where mask is the sign bit
  return __hiloint2double(__double2hiint(x) ^ mask, __double2loint(x));
}

// y[i] += col[i]·x over a column of S coefficients on 16 bytes
template <int S>
__device__ __forceinline__ void axpy_column(double (&y)[S], const double* col, double x) {
#pragma unroll
  for (int i = 0; i < S; i += 2) {
    const double2 b = *reinterpret_cast<const double2*>(col + i);
    y[i] = fma(b.x, x, y[i]);
    if (i + 1 < S) y[i + 1] = fma(b.y, x, y[i + 1]);
  }
}

// the rotation of degree L of this lane's C pairs, in place in their tile rows r (32·PT apart);
// D: the degree's coefficients; cs: the pairs' (cos mφ, sin mφ), NC apart per order; BACK: the z
// rotation after the product (to the offset's azimuth) instead of before it
template <int L, int C, bool BACK>
__device__ __forceinline__ void rotate_degree(double* r, int PT, const double* __restrict__ D,
                                              const double2* __restrict__ cs, const int (&down)[C]) {
  constexpr int NC = 32 * C, SR = rot_pad(L + 1), SI = rot_pad(L), K0 = L * L;
  double yr[C][L + 1], yi[C][L > 0 ? L : 1];
#pragma unroll
  for (int c = 0; c < C; ++c) {
#pragma unroll
    for (int i = 0; i <= L; ++i) yr[c][i] = 0.0;
#pragma unroll
    for (int i = 0; i < L; ++i) yi[c][i] = 0.0;
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    double x = r[32 * c * PT + K0];
    if (!BACK && (L & 1)) x = flip(x, down[c]);
    axpy_column<L + 1>(yr[c], D, x);
  }
  if constexpr (L > 0) {
    const double* col = D + SR;
#pragma unroll 1
    for (int k = 1; k <= L; ++k, col += SR + SI) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        double xr = r[32 * c * PT + K0 + 2 * k - 1], xi = r[32 * c * PT + K0 + 2 * k];
        if (!BACK) {
          double2 z = cs[k * NC + 32 * c];
          if (L & 1) { z.x = flip(z.x, down[c]); z.y = flip(z.y, down[c]); }
          const double t = z.x * xr - z.y * xi;
          // the imaginary parts negated: Tᵐ acts on them with the opposite sign
          xi = -(z.y * xr + z.x * xi);
          xr = t;
        }
        axpy_column<L + 1>(yr[c], col, xr);
        axpy_column<L>(yi[c], col + SR, xi);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    double* q = r + 32 * c * PT + K0;
    const int dn = L & 1 ? down[c] : 0;
    q[0] = BACK && (L & 1) ? flip(yr[c][0], dn) : yr[c][0];
#pragma unroll
    for (int j = 1; j <= L; ++j) {
      double a = yr[c][j], b = yi[c][j - 1];
      if (BACK) {
        double2 z = cs[j * NC + 32 * c];
        if (L & 1) { z.x = flip(z.x, dn); z.y = flip(z.y, dn); }
        const double u = z.x * a - z.y * b, v = z.y * a + z.x * b;
        a = j & 1 ? -u : u;                              // Σ
        b = j & 1 ? -v : v;
      }
      q[2 * j - 1] = a;
      q[2 * j] = b;
    }
  }
}

// the translation of order m over the S = p + 1 − m degrees m..p, in place; B the order's coefficients
template <int S, int C>
__device__ __forceinline__ void translate_order(double* r, int PT, int m, const double* __restrict__ B) {
  constexpr int SP = rot_pad(S);
  const int k0 = m * m + (m ? 2 * m - 1 : 0);            // degree l at l² + 2m − 1 (l² for m = 0)
  double yr[C][S], yi[C][S];
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int i = 0; i < S; ++i) yr[c][i] = yi[c][i] = 0.0;
  int k = k0, step = 2 * m + 1;
  if (m == 0) {
#pragma unroll 2
    for (int i = 0; i < S; ++i, k += step, step += 2)
#pragma unroll
      for (int c = 0; c < C; ++c) axpy_column<S>(yr[c], B + i * SP, r[32 * c * PT + k]);
  } else {
#pragma unroll 1
    for (int i = 0; i < S; ++i, k += step, step += 2)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        axpy_column<S>(yr[c], B + i * SP, r[32 * c * PT + k]);
        axpy_column<S>(yi[c], B + i * SP, r[32 * c * PT + k + 1]);
      }
  }
  k = k0;
  step = 2 * m + 1;
#pragma unroll
  for (int i = 0; i < S; ++i) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      r[32 * c * PT + k] = yr[c][i];
      if (m) r[32 * c * PT + k + 1] = yi[c][i];
    }
    k += step;
    step += 2;
  }
}

// the instance of a runtime degree or block size
template <int L, int C, bool BACK>
__device__ __forceinline__ void rotate_any(int l, double* r, int PT, const double* D, const double2* cs, const int (&down)[C]) {
  if constexpr (L > 0) {
    if (l < L) { rotate_any<L - 1, C, BACK>(l, r, PT, D, cs, down); return; }
  }
  rotate_degree<L, C, BACK>(r, PT, D, cs, down);
}
template <int S, int C>
__device__ __forceinline__ void translate_any(int s, double* r, int PT, int m, const double* B) {
  if constexpr (S > 1) {
    if (s < S) { translate_any<S - 1, C>(s, r, PT, m, B); return; }
  }
  translate_order<S, C>(r, PT, m, B);
}

// an odd row length: the lanes' rows (columns of the tile) are free of bank conflicts
__host__ __device__ constexpr int rot_row(int p) { return (p + 1) * (p + 1) | 1; }
constexpr int rot_list(int nc) { return 4 * nc + 2; }   // source, offset (bit 31: it points down), target, runs; the last run's end, their count

size_t rot_smem(const RotLayout& l, int C, int G) {
  const int nc = 32 * C;
  return sizeof(double) * ((size_t)l.nd + G * l.nt + (size_t)G * 2 * (l.p + 1) * nc + (size_t)G * nc * rot_row(l.p)) +
         sizeof(int) * (size_t)G * 2 * rot_list(nc);
}

__device__ __forceinline__ void cpa16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cpa8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// NW warps per group; LMAX ≥ p the largest degree
template <int C, int G, int NW, int LMAX, int MINB>
__global__ void __launch_bounds__(32 * NW * G, MINB)
    k_m2l_rot(const __grid_constant__ RotSched sch, int nparts, int sub, int TB, const int4* __restrict__ blocks,
              const int* __restrict__ cls_off, const int* __restrict__ rtab, const int2* __restrict__ pairs, const double* __restrict__ dtab,
              const double2* __restrict__ csf, const uint64_t* __restrict__ lv_trans, const double* __restrict__ m2l_scale,
              int LD, const double* __restrict__ M, double* __restrict__ Pl, int64_t pitch, int stokes) {
  constexpr int NC = 32 * C, NT = 32 * NW, NL = rot_list(NC);
  const int p = sch.lay.p, NP = (p + 1) * (p + 1), PT = rot_row(p), nd = sch.lay.nd, nt = sch.lay.nt;
  const int tid = threadIdx.x % NT, grp = threadIdx.x / NT, warp = tid >> 5, lane = tid & 31;
  const int comp = blockIdx.y, psi = stokes && comp == 3;
  extern __shared__ __align__(16) double sm[];
  double* D = sm;                                        // the class's rotation
  double* T = D + nd + grp * nt;                         // the group's translation
  double2* cs = (double2*)(D + nd + G * nt) + (size_t)grp * (p + 1) * NC;   // [order][pair]
  double* tile = (double*)((double2*)(D + nd + G * nt) + (size_t)G * (p + 1) * NC) + (size_t)grp * NC * PT;
  int* list = (int*)((double*)((double2*)(D + nd + G * nt) + (size_t)G * (p + 1) * NC) + (size_t)G * NC * PT) + grp * 2 * NL;
  auto gsync = [&] {
    if constexpr (G == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(NT) : "memory");
  };
  // part q of block blk: its targets [t0, t1), whose pairs are consecutive in every class
  const int part = blockIdx.x * G + grp, blk = part / sub, t0 = (part % sub) * (TB / sub), t1 = t0 + TB / sub;
  const bool on = part < nparts;
  const int4 b = on ? blocks[blk] : make_int4(0, 0, 0, 0);
  const int level = b.x & 255;
  const double alpha = on ? m2l_scale[level] : 0.0;
  const int* co = cls_off + (int64_t)(on ? blk : 0) * (NCLASS + 1);
  const double* lt = reinterpret_cast<const double*>(lv_trans[level]);
  const double* Mc = M + (int64_t)comp * LD;
  double* Pc = Pl + (int64_t)b.y * pitch + (int64_t)comp * LD;

  // pair j of a list: its multipole into the tile's row j, its azimuth's table into the columns j
  auto gather = [&](const int* L, int j) {
    double* row = tile + j * PT;
    const int f = L[NC + j] & 0xffff;
    const double* src = Mc + (int64_t)L[j] * pitch;
    if (psi) {
      // the Stokes Ψ̂ block: its source is Ψ̂ + o·Φ of the source box, o the far offset
      // (harmonics_stokes.jl: M2L Ψ̂_B = Ψ̂_A + o·Φ, linear in the source)
      const double* phi = M + (int64_t)L[j] * pitch;
      const double o0 = c_faroff[3 * f], o1 = c_faroff[3 * f + 1], o2 = c_faroff[3 * f + 2];
      for (int e = lane; e < NP; e += 32)
        row[e] = fma(o2, __ldg(phi + 2 * LD + e), fma(o1, __ldg(phi + LD + e), fma(o0, __ldg(phi + e), __ldg(src + e))));
    } else {
      for (int e = lane; e < NP; e += 32) cpa8(row + e, src + e);
    }
    for (int m = lane; m <= p; m += 32) cpa16(cs + m * NC + j, csf + f * (p + 1) + m);
  };
  // the chunk's pairs read by the group's first warp, then into the list with the runs of one target
  // (the pairs of a class are grouped by target)
  auto fetch = [&](int q0, int nc, int2 (&pr)[C]) {
#pragma unroll
    for (int c = 0; c < C; ++c) pr[c] = 32 * c + lane < nc ? pairs[b.w + q0 + 32 * c + lane] : make_int2(0, -1);
  };
  auto commit = [&](int* L, int nc, const int2 (&pr)[C]) {
    int base = 0, last = -1;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = 32 * c + lane, tg = pr[c].y < 0 ? -1 : pr[c].y & 0xff;
      int prev = __shfl_up_sync(0xffffffffu, tg, 1);
      if (lane == 0) prev = last;
      last = __shfl_sync(0xffffffffu, tg, 31);
      const bool start = j < nc && tg != prev;
      const unsigned bal = __ballot_sync(0xffffffffu, start);
      L[j] = pr[c].x;
      const int f = pr[c].y < 0 ? 0 : pr[c].y >> 8;
      L[NC + j] = f | (c_faroff[3 * f + 2] < 0) << 31;
      L[2 * NC + j] = tg;
      if (start) L[3 * NC + base + __popc(bal & ((1u << lane) - 1u))] = j;
      base += __popc(bal);
    }
    if (lane == 0) { L[3 * NC + base] = nc; L[4 * NC + 1] = base; }
  };

  for (int c = 0; c < NCLASS; ++c) {
    const int* rt = rtab + ((int64_t)blk * NCLASS + c) * TB;
    const int a0 = on ? co[c] + (t0 ? rt[t0] & 0xffff : 0) : 0, a1 = on ? (t1 < TB ? co[c] + (rt[t1] & 0xffff) : co[c + 1]) : 0;
    if constexpr (G == 1) {
      if (a0 == a1) continue;
    } else {
      if (!__syncthreads_or(a0 < a1)) continue;          // no group is still in the previous class
    }
    // the class's tables, the first chunk's list and multipoles
    {
      const double* src = dtab + (int64_t)c * nd;
      for (int i = 2 * threadIdx.x; i < nd; i += 2 * NT * G) cpa16(D + i, src + i);
      const double* ts = lt + (int64_t)c * nt;
      if (a0 < a1)                                       // an idle group has no level
        for (int i = 2 * tid; i < nt; i += 2 * NT) cpa16(T + i, ts + i);
    }
    if (warp == 0 && a0 < a1) {
      int2 pr[C];
      fetch(a0, min(NC, a1 - a0), pr);
      commit(list, min(NC, a1 - a0), pr);
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
      int2 pr[C];
      if (warp == 0 && nn > 0) fetch(q0 + NC, nn, pr);
      int down[C];
#pragma unroll
      for (int k = 0; k < C; ++k) down[k] = L[NC + 32 * k + lane] & (int)0x80000000;
#pragma unroll 1
      for (int i = sch.first[0][warp]; i < sch.first[0][warp + 1]; ++i) {
        const int l = sch.order[0][i];
        rotate_any<LMAX, C, false>(l, tile + lane * PT, PT, D + sch.lay.offd[l], cs + lane, down);
      }
      if (warp == 0 && nn > 0) commit(Ln, nn, pr);
      gsync();
#pragma unroll 1
      for (int i = sch.first[1][warp]; i < sch.first[1][warp + 1]; ++i) {
        const int m = sch.order[1][i];
        translate_any<LMAX + 1, C>(p + 1 - m, tile + lane * PT, PT, m, T + sch.lay.offt[m]);
      }
      gsync();
#pragma unroll 1
      for (int i = sch.first[0][warp]; i < sch.first[0][warp + 1]; ++i) {
        const int l = sch.order[0][i];
        rotate_any<LMAX, C, true>(l, tile + lane * PT, PT, D + sch.lay.offd[l], cs + lane, down);
      }
      gsync();
      // scatter: a warp the runs w, w + NW, ..., the entries across the lanes; then the next chunk's
      // multipoles into the rows it has read
      const int nrun = L[4 * NC + 1];
      for (int r = warp; r < nrun; r += NW) {
        const int j0 = L[3 * NC + r], j1 = L[3 * NC + r + 1];
        double* dst = Pc + (int64_t)L[2 * NC + j0] * pitch;
        for (int e0 = lane; e0 < NP; e0 += 128) {
          double v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = e0 + 32 * k < NP ? dst[e0 + 32 * k] : 0.0;
          for (int j = j0; j < j1; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (e0 + 32 * k < NP) v[k] = fma(alpha, tile[j * PT + e0 + 32 * k], v[k]);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (e0 + 32 * k < NP) dst[e0 + 32 * k] = v[k];
        }
        if (nn > 0) {
          __syncwarp();
          for (int j = j0; j < min(j1, nn); ++j) gather(Ln, j);
        }
      }
      // rows past this chunk's last pair (a next chunk is longer only when this one is full)
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
      gsync();
    }
  }
}

RotSched schedule(const RotLayout& lay, int nw) {
  RotSched s{};
  s.lay = lay;
  for (int kind = 0; kind < 2; ++kind) {
    // the work of degree l: (l + 1)² + l² products; of order m over q = p + 1 − m degrees: 2q² (q² for
    // m = 0); and the rows read and written
    std::vector<int> cost(lay.p + 1), id(lay.p + 1);
    for (int i = 0; i <= lay.p; ++i) {
      const int q = lay.p + 1 - i;
      cost[i] = kind == 0 ? (i + 1) * (i + 1) + i * i + 12 * i + 20 : (i ? 2 : 1) * q * (q + 6) + 20;
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

// The parts a block is cut into: more of them fill the device (`slots` groups run at once), fewer
// of them fill the chunks (a class's last chunk of a part is half empty on average, and one with
// few pairs costs a whole one): the power of two with the least waves × chunks per part. Measured
// at 6.04M far pairs of 293 blocks, p = 10 (1, 2, 4, 8 parts): 7.9, 6.0, 6.0, 6.3 ms; at 207,331
// pairs of a sphere: 0.77, 0.59, 0.72, 0.95 ms.
int parts_per_block(const Plan& P, int nexp, int slots) {
  const double nb = (double)P.h_blocks.size();
  int best = 1;
  double least = 1e300;
  for (int sub = 1; sub <= P.TB / 4; sub *= 2) {
    const double pairs = (double)P.npairs / (nb * sub * NCLASS);
    const double t = std::max(1.0, nb * sub * nexp / slots) * std::max(1.0, pairs / 32 + 0.5);
    if (t < 0.97 * least) { least = t; best = sub; }
  }
  return best;
}

template <int C, int G, int NW, int LMAX, int MINB>
void launch(State& S) {
  Plan& P = *S.plan;
  Cache& K = *P.cache;
  const int nb = (int)P.h_blocks.size();
  if (nb == 0) return;
  const RotSched sch = schedule(K.rot->layout, NW);
  const size_t smem = rot_smem(K.rot->layout, C, G);
  auto kern = k_m2l_rot<C, G, NW, LMAX, MINB>;
  FMMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int sub = parts_per_block(P, K.nexp, P.ctx->num_sms * MINB * G);
  kern<<<dim3((nb * sub + G - 1) / G, K.nexp), 32 * NW * G, smem, P.ctx->stream>>>(
      sch, nb * sub, sub, P.TB, P.blocks.p, P.cls_off.p, P.rtab.p, P.pairs.p, K.rot_d.p, (const double2*)K.rot_csf.p, P.d_lv_rot.p, P.d_m2l_scale.p,
      K.ld, S.M.p, S.Pl.p, (int64_t)K.nexp * K.ld, K.nexp == 4);
  FMMB_LAUNCH_CHECK();
}

void translations(Cache& C, const RotLayout& lay, const double* reps, DBuf<double>& out, cudaStream_t s) {
  out.alloc((size_t)NCLASS * lay.nt);
  k_rot_translations<<<NCLASS, 256, 0, s>>>(reps, C.rot_d.p, C.rot_cs.p, lay, C.ld, out.p);
  FMMB_LAUNCH_CHECK();
}

}  // namespace

// the tables of the FP64 M2L: the cache's rotations (uploaded with its first FP64 state) and per
// level the translations along z (the cache's for the homogeneous kernels, the level width's own
// for Yukawa3D). The cache is locked by the caller.
void prepare_rotations(Plan& P) {
  Cache& C = *P.cache;
  cudaStream_t s = P.ctx->stream;
  if (P.d_lv_rot.n) return;
  if (!C.rot) {
    auto h = rotation_tables(C.p, C.host);
    to_device(C.rot_d, h->d, s);
    to_device(C.rot_cs, h->cs, s);
    to_device(C.rot_csf, h->csf, s);
    if (C.kernel != FMMB_KERNEL_YUKAWA3D) translations(C, h->layout, C.reps.p, C.rot_t, s);
    C.rot = h;
  }
  std::vector<uint64_t> t(P.L, 0);
  for (int l = 0; l < P.L; ++l) {
    if (C.kernel != FMMB_KERNEL_YUKAWA3D) {
      t[l] = (uint64_t)(uintptr_t)C.rot_t.p;
    } else if (l >= 2 && l < (int)P.lv_yukawa.size() && P.lv_yukawa[l]) {
      YukawaLevel& Y = *P.lv_yukawa[l];
      std::lock_guard<std::mutex> lk(Y.mu);
      if (!Y.rot_t.n) {
        // shared by caches on other streams: outside the stream-ordered pool, complete before use
        const cudaStream_t keep = g_alloc_stream;
        g_alloc_stream = nullptr;
        try {
          translations(C, C.rot->layout, Y.reps.p, Y.rot_t, s);
          FMMB_CUDA(cudaStreamSynchronize(s));
        } catch (...) {
          Y.rot_t.release();
          g_alloc_stream = keep;
          throw;
        }
        g_alloc_stream = keep;
      }
      t[l] = (uint64_t)(uintptr_t)Y.rot_t.p;
    }
  }
  to_device(P.d_lv_rot, t, s);
}

void m2l_rot(State& S) {
  const int p = S.plan->cache->p;
  // four warps share a tile up to p = 13; above, the largest degree is a smaller share of the work and
  // more warps even out. At p = 16 one tile and the class's tables take 122 KB: two groups share the
  // tables (6.04M pairs: 15.0 ms, 20.0 ms with one), where there are enough blocks for both.
  if (p <= 11) launch<1, 1, 4, 11, 4>(S);
  else if (p <= 13) launch<1, 1, 4, 13, 3>(S);
  else if (p <= 15) launch<1, 1, 6, 15, 2>(S);
  else if (p == 16 && (int64_t)S.plan->h_blocks.size() * S.plan->cache->nexp >= 2 * S.plan->ctx->num_sms) launch<1, 2, 6, 16, 1>(S);
  else if (p == 16) launch<1, 1, 8, 16, 1>(S);
  else launch<1, 1, 8, 20, 1>(S);
}

}  // namespace fmmb
