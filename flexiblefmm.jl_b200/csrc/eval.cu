// Evaluation at the targets of one leaf (src/evaluate.jl:12-48, src/device.jl:89-100,185-206),
// in two kernels:
//   k_l2p   the far field: L2P of the leaf's local expansion (harmonics.jl:447-486), one warp per leaf group (a
//           CTA of four where leaves are few) with the local staged in shared memory, lanes over the targets;
//           FP64 on the plain path, FP32 on the mixed path (tolerances ≥ 1e-8); writes the outputs
//   k_near  the near field (near.cuh): the sources of the 27 colleagues, flattened into batches of 32
//           that the warps of a leaf's team stage in shared memory, lanes over the targets; adds to
//           the outputs. The self term is skipped by index (evaluate_at_sources,
//           src/evaluate.jl:1-10), checked only in the batches that hold the leaf's own points.
// Two precisions of the near field:
//   double  the plain path: absolute coordinates, the reference's FMA square norm
//           (src/kernels.jl:20-24)
//   float   the mixed path: coordinates relative to the target leaf's centre, converted from FP64
//           when staged (the FP32 differences carry an absolute error of ~2⁻²⁴·w instead of
//           2⁻²⁴·|x|, so close pairs keep their accuracy); two sources per packed f32x2
//           instruction; each batch summed in FP32, the batch sums accumulated in FP64
// Splitting the two keeps the near-field loop at a low register count (high occupancy); the
// outputs are u then u + KC·near, the same arithmetic as one fused pass.
#include "near.cuh"

namespace fmmb {
namespace {

// The leaf's local expansion prepared for L2P: the entries' eight values (l2p_values), rounded to R, m-major
template <int P, typename R>
__device__ void l2p_prepare(const double* __restrict__ L, R* __restrict__ E, int first, int step) {
  for (int q = first; q < l2p_entries<P>(); q += step) {
    double v[8];
    l2p_values<P>(L, q, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) E[8 * q + i] = (R)v[i];
  }
}

template <typename R> struct alignas(4 * sizeof(R)) Quad { R a, b, c, d; };

// L2P at x̂ from the prepared entries (potential and the gradient before the 1/w factor)
template <int P, typename R>
__device__ __forceinline__ void l2p_prepared(const R* __restrict__ E, R x, R y, R z, R& u, R& gx, R& gy, R& gz) {
  const R r2 = x * x + y * y + z * z;
  R sr = 1, si = 0;
  u = 0; gx = 0; gy = 0; gz = 0;
#pragma unroll 1
  for (int m = 0; m <= P; ++m) {
    R pr = 0, pi = 0, cr = sr, ci = si;
    const Quad<R>* Em = reinterpret_cast<const Quad<R>*>(E + 8 * l2p_entry(P, m, m));
#pragma unroll 2
    for (int n = m; n <= P; ++n) {
      R vr, vi;
      if (n == m) { vr = sr; vi = si; }
      else {
        const int t = tri(n, m);
        const R az = ctab<R>(t) * z, br = ctab<R>(TRI_MAX + t) * r2;
        vr = az * cr - br * pr; vi = az * ci - br * pi;
        pr = cr; pi = ci; cr = vr; ci = vi;
      }
      const Quad<R> a = Em[2 * (n - m)], b = Em[2 * (n - m) + 1];
      u += a.a * vr + a.b * vi;
      gx += a.c * vr + a.d * vi;
      gy += b.a * vr + b.b * vi;
      gz += b.c * vr + b.d * vi;
    }
    if (m < P) {
      const R e = ce<R>(m);
      const R nr = -e * (x * sr - y * si), ni = -e * (x * si + y * sr);
      sr = nr; si = ni;
    }
  }
}

// per-warp shared memory of k_l2p: the prepared entries, or (Yukawa3D) the local itself
template <int P, typename R, bool YK>
size_t l2p_warp_bytes(int LD) { return YK ? sizeof(R) * LD : sizeof(R) * 8 * l2p_entries<P>(); }

// YK: Yukawa3D's weighted L2P (FP64), κ̂² = kh2[level]
template <int P, typename R, bool YK>
__global__ void __launch_bounds__(256) k_l2p(const int* __restrict__ gnode, const int* __restrict__ gstart,
                                             const int* __restrict__ gcount, int ngroups, const double* __restrict__ tx,
                                             const double* __restrict__ ty, const double* __restrict__ tz,
                                             const int* __restrict__ tout, const int4* __restrict__ cell,
                                             const double* __restrict__ Pl, int LD, Geometry geo,
                                             const double* __restrict__ scale, int outputs, double* __restrict__ pot,
                                             double* __restrict__ grad, const double* __restrict__ kh2, int acc, int team) {
  extern __shared__ __align__(16) unsigned char sl_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a leaf's entries are prepared, and its targets shared out, by `team` warps: one, or all of the CTA's
  const int grp = team ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + warp;
  if (grp >= ngroups) return;
  const int leaf = gnode[grp], first = team ? threadIdx.x : lane, step = team ? blockDim.x : 32;
  R* L = reinterpret_cast<R*>(sl_raw) + (team ? 0 : warp) * (YK ? LD : 8 * l2p_entries<P>());
  if constexpr (YK) {
    for (int i = first; i < LD; i += step) L[i] = (R)Pl[(int64_t)leaf * LD + i];
  } else {
    l2p_prepare<P, R>(Pl + (int64_t)leaf * LD, L, first, step);
  }
  if (team) __syncthreads();
  else __syncwarp();
  const int4 c = cell[leaf];
  const Geometry gn = geo.at(leaf);
  const double w = ldexp(geo.W0, -c.w), s = scale[c.w];
  const double cx = gn.center(0, c.x, w), cy = gn.center(1, c.y, w), cz = gn.center(2, c.z, w);
  const int t0 = gstart[grp], nt = gcount[grp];
  for (int base = first - lane; base < nt; base += step) {
    const int k = t0 + base + lane;
    const bool act = base + lane < nt;
    const double x = act ? tx[k] : cx, y = act ? ty[k] : cy, z = act ? tz[k] : cz;
    R u, gx, gy, gz;
    if constexpr (YK) l2p_yukawa<P>(L, kh2[c.w], (x - cx) * s, (y - cy) * s, (z - cz) * s, u, gx, gy, gz);
    else l2p_prepared<P, R>(L, (R)((x - cx) * s), (R)((y - cy) * s), (R)((z - cz) * s), u, gx, gy, gz);
    if (act) {
      const int o = tout[k];
      // acc: the near field is already in the outputs (x + y = y + x: the same sums either way)
      if (outputs & FMMB_OUTPUT_POTENTIAL) pot[o] = (acc ? pot[o] : 0.0) + (double)u;
      if (outputs & FMMB_OUTPUT_GRADIENT) {
        const int64_t o3 = 3 * (int64_t)o;
        grad[o3] = (acc ? grad[o3] : 0.0) + (double)gx * s;
        grad[o3 + 1] = (acc ? grad[o3 + 1] : 0.0) + (double)gy * s;
        grad[o3 + 2] = (acc ? grad[o3 + 2] : 0.0) + (double)gz * s;
      }
    }
  }
}

// one staged source: aligned so that it is read with one 16-byte (FP32) or two 16-byte (FP64)
// shared-memory loads
template <typename R>
struct alignas(4 * sizeof(R)) R4 { R x, y, z, w; };

// the hardware reciprocal square root (PTX rsqrt.approx, relative error below 2^-22), with
// subnormal inputs flushed: squared distances of distinct points in leaf-centred coordinates are
// far above FP32's subnormal range, and the self term (r² = 0 → ∞) is masked by index
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// packed FP32 pairs (the f32x2 instructions of sm_100: two lanes of arithmetic per instruction)
__device__ __forceinline__ uint64_t pk2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// The near field of charges (near.cuh). KERNEL 0: Laplace3D; 1 (FP64): the Yukawa pair e^{−κr}/r and
// its radial derivative −e^{−κr}(1 + κr)/r² (src/kernels.jl:235-242); 2 (FP64): the Laplace2D pair
// c·log r², c = −1/(4π), as KC·(−τ log r²) and gradient −KC·(2τ/r²)·d (src/kernels.jl:58-66; the
// points share z, so r² is the planar distance). GRAD: the gradient's sums too.
template <typename R, int KERNEL, bool GRAD>
struct ChargesNear {
  using Real = R;
  static constexpr bool REL = sizeof(R) == 4;   // the mixed path works relative to the leaf's centre
  static constexpr int NA = GRAD ? 4 : 1, CH = 2, MINB = KERNEL == 2 ? 4 : 5;
  struct Args {
    const double *xs, *ys, *zs, *q;
    double kappa;
    int outputs, first;       // first: the far field comes after (and adds to) the outputs
    double *pot, *grad;
  };
  struct Src { double x, y, z, w; };
  struct Stage { R4<R> s[32]; };
  static __device__ __forceinline__ void load(const Args& a, int j, Src& v) { v = Src{a.xs[j], a.ys[j], a.zs[j], a.q[j]}; }
  static __device__ __forceinline__ void stage(Stage& st, int lane, const Src& v, double cx, double cy, double cz) {
    if constexpr (sizeof(R) == 4) {
      // source pairs {x₀ x₁ y₀ y₁}{z₀ z₁ w₀ w₁}: lane l into pair l/2, slot l%2
      float* f = reinterpret_cast<float*>(st.s) + 8 * (lane >> 1) + (lane & 1);
      f[0] = (float)(v.x - cx);
      f[2] = (float)(v.y - cy);
      f[4] = (float)(v.z - cz);
      f[6] = (float)v.w;
    } else {
      st.s[lane] = R4<R>{(R)v.x, (R)v.y, (R)v.z, (R)v.w};
    }
  }
  // m staged sources against this lane's target; CHECK skips source `is`; the lane's part of f of them
  template <bool CHECK>
  static __device__ __forceinline__ void batch(const Args& pa, const Stage& st, int m, int is, int part, int f, const R (&t)[3],
                                               double (&acc)[NA]) {
    if constexpr (sizeof(R) == 4) batch_f32x2<CHECK>(st, m, is, part, f, t, acc);
    else batch_f64<CHECK>(pa, st, m, is, part, f, t, acc);
  }
  // the plain path sums straight into the FP64 totals
  template <bool CHECK>
  static __device__ __forceinline__ void batch_f64(const Args& pa, const Stage& st, int m, int is, int part, int f,
                                                   const double (&t)[3], double (&acc)[NA]) {
    auto body = [&](int i) {
      const R4<R> sv = st.s[i];
      const double dx = t[0] - sv.x, dy = t[1] - sv.y, dz = t[2] - sv.z;
      const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
      // the potential's sums in explicit FMAs: the same bits with and without the gradient's
      double qir3 = 0;
      if constexpr (KERNEL == 2) {
        const bool self = CHECK && i == is;
        acc[0] = fma(-sv.w, self ? 0.0 : log(r2), acc[0]);
        if (GRAD) qir3 = self ? 0.0 : 2 * sv.w / r2;
      } else {
        double ir = rsqrt(r2), w = sv.w;
        if (CHECK && i == is) ir = 0.0;
        if constexpr (KERNEL == 1) {
          const double kr = __dmul_rn(pa.kappa, __dmul_rn(r2, ir));
          w = __dmul_rn(w, exp(-kr));
          if (GRAD) qir3 = w * (1 + kr) * ir * ir * ir;
        } else {
          if (GRAD) qir3 = w * ir * ir * ir;
        }
        acc[0] = fma(w, ir, acc[0]);
      }
      if constexpr (GRAD) {
        acc[1] = fma(qir3, dx, acc[1]);
        acc[2] = fma(qir3, dy, acc[2]);
        acc[3] = fma(qir3, dz, acc[3]);
      }
    };
    if (m == 32 && f == 1) {
#pragma unroll 8
      for (int i = 0; i < 32; ++i) body(i);
    } else {
#pragma unroll 4
      for (int i = part; i < m; i += f) body(i);
    }
  }
  // two sources per instruction: each pair's arithmetic in packed f32x2, the two running sums of
  // every quantity added at the end and the batch's sums accumulated in FP64; an odd last source
  // takes a scalar body
  template <bool CHECK>
  static __device__ __forceinline__ void batch_f32x2(const Stage& st, int m, int is, int part, int f, const R (&t)[3],
                                                     double (&acc)[NA]) {
    const float4* pr = reinterpret_cast<const float4*>(st.s);
    const float fx = t[0], fy = t[1], fz = t[2];
    const uint64_t fx2 = pk2(fx, fx), fy2 = pk2(fy, fy), fz2 = pk2(fz, fz);
    uint64_t p2 = pk2(0.f, 0.f), x2 = p2, y2 = p2, z2 = p2;
    const int np = m >> 1;
    auto body = [&](int k) {
      const float4 a = pr[2 * k], b = pr[2 * k + 1];
      const uint64_t dx = sub2(fx2, pk2(a.x, a.y)), dy = sub2(fy2, pk2(a.z, a.w)), dz = sub2(fz2, pk2(b.x, b.y));
      const uint64_t r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
      float ra, rb;
      upk2(r2, ra, rb);
      float ia = rsqrt_ftz(ra), ib = rsqrt_ftz(rb);
      if (CHECK && 2 * k == is) ia = 0.f;
      if (CHECK && 2 * k + 1 == is) ib = 0.f;
      const uint64_t ir = pk2(ia, ib);
      const uint64_t w = pk2(b.z, b.w);
      p2 = fma2(w, ir, p2);                        // explicit: the same bits with and without the gradient
      if constexpr (GRAD) {
        const uint64_t qir3 = mul2(mul2(mul2(w, ir), ir), ir);
        x2 = fma2(qir3, dx, x2);
        y2 = fma2(qir3, dy, y2);
        z2 = fma2(qir3, dz, z2);
      }
    };
    if (np == 16 && f == 1) {
#pragma unroll 8
      for (int k = 0; k < 16; ++k) body(k);
    } else {
#pragma unroll 2
      for (int k = part; k < np; k += f) body(k);
    }
    float bp, bx, by, bz, hi;
    upk2(p2, bp, hi); bp += hi;
    if constexpr (GRAD) {
      upk2(x2, bx, hi); bx += hi;
      upk2(y2, by, hi); by += hi;
      upk2(z2, bz, hi); bz += hi;
    }
    if ((m & 1) && part == 0) {                    // the odd last source
      const float* g = reinterpret_cast<const float*>(pr + 2 * np);
      const float dx = fx - g[0], dy = fy - g[2], dz = fz - g[4];
      float ir = rsqrt_ftz(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
      if (CHECK && m - 1 == is) ir = 0.f;
      bp = fmaf(g[6], ir, bp);
      if constexpr (GRAD) {
        const float qir3 = g[6] * ir * ir * ir;
        bx = fmaf(qir3, dx, bx);
        by = fmaf(qir3, dy, by);
        bz = fmaf(qir3, dz, bz);
      }
    }
    acc[0] += bp;
    if constexpr (GRAD) { acc[1] += bx; acc[2] += by; acc[3] += bz; }
  }
  static __device__ __forceinline__ void write(const Args& a, int o, const double (&acc)[NA]) {
    // a product and a sum, never one FMA: the near field may come before or after the far field
    if (a.outputs & FMMB_OUTPUT_POTENTIAL) a.pot[o] = __dadd_rn(a.first ? 0.0 : a.pot[o], __dmul_rn(KC, acc[0]));
    if constexpr (GRAD) {
      if (a.outputs & FMMB_OUTPUT_GRADIENT) {
        double* g = a.grad + 3 * (int64_t)o;
#pragma unroll
        for (int d = 0; d < 3; ++d) g[d] = __dadd_rn(a.first ? 0.0 : g[d], -__dmul_rn(KC, acc[1 + d]));
      }
    }
  }
};

// The kernel-independent far field (l2t, src/operators/ki_common.jl:293-327): at each target
// Σ_k G(x − y_k) L_k over the leaf's large surface y_k = c + w·ŷ_k (ŷ at width 1), times w (the
// pseudo-inverse's scale). A warp per leaf, lanes over the surface points (a lane takes every
// 32nd): each lane reads its points and densities once per batch of up to TB targets held in
// registers, then the batch's sums are reduced across the lanes in FP64. (Leaves of the adaptive
// configurations hold a few points each, so lanes over the targets would mostly idle.)
// R = float: leaf-centred FP32 terms, each lane's partial sums in FP32, the reduction in FP64;
// R = double: FP64 throughout. Writes the outputs (the near field adds to them).
template <typename R, int TB>
__device__ __forceinline__ void ki_l2t_batch(int k0, int nb, const double* __restrict__ tx, const double* __restrict__ ty,
                                             const double* __restrict__ tz, const int* __restrict__ tout,
                                             const double* __restrict__ L, const double* __restrict__ large, int nl,
                                             double w, double cx, double cy, double cz, int lane, int outputs,
                                             double* __restrict__ pot, double* __restrict__ grad) {
  R px[TB], py[TB], pz[TB], au[TB], ax[TB], ay[TB], az[TB];
#pragma unroll
  for (int i = 0; i < TB; ++i) {
    const int k = k0 + (i < nb ? i : 0);             // slots past the batch repeat its first target
    px[i] = (R)(tx[k] - cx); py[i] = (R)(ty[k] - cy); pz[i] = (R)(tz[k] - cz);
    au[i] = 0; ax[i] = 0; ay[i] = 0; az[i] = 0;
  }
  for (int q = lane; q < nl; q += 32) {
    const R yx = (R)(w * large[3 * q]), yy = (R)(w * large[3 * q + 1]), yz = (R)(w * large[3 * q + 2]);
    const R l = (R)L[q];
#pragma unroll
    for (int i = 0; i < TB; ++i) {
      const R dx = px[i] - yx, dy = py[i] - yy, dz = pz[i] - yz;
      const R ir = rsqrt(dx * dx + dy * dy + dz * dz);
      const R li = l * ir;
      au[i] += li;
      const R li3 = li * ir * ir;
      ax[i] += li3 * dx;
      ay[i] += li3 * dy;
      az[i] += li3 * dz;
    }
  }
#pragma unroll
  for (int i = 0; i < TB; ++i) {
    double u = au[i], gx = ax[i], gy = ay[i], gz = az[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      u += __shfl_xor_sync(0xffffffffu, u, o);
      gx += __shfl_xor_sync(0xffffffffu, gx, o);
      gy += __shfl_xor_sync(0xffffffffu, gy, o);
      gz += __shfl_xor_sync(0xffffffffu, gz, o);
    }
    if (lane == i && i < nb) {
      const int t = tout[k0 + i];
      if (outputs & FMMB_OUTPUT_POTENTIAL) pot[t] = KC * w * u;
      if (outputs & FMMB_OUTPUT_GRADIENT) {
        grad[3 * (int64_t)t] = -KC * w * gx;
        grad[3 * (int64_t)t + 1] = -KC * w * gy;
        grad[3 * (int64_t)t + 2] = -KC * w * gz;
      }
    }
  }
}

template <typename R>
__global__ void __launch_bounds__(128) k_ki_l2t(const int* __restrict__ gnode, const int* __restrict__ gstart,
                                                const int* __restrict__ gcount, int ngroups, const double* __restrict__ tx,
                                                const double* __restrict__ ty, const double* __restrict__ tz,
                                                const int* __restrict__ tout, const int4* __restrict__ cell,
                                                const double* __restrict__ Ll, int nl, int nld,
                                                const double* __restrict__ large, Geometry geo, int outputs,
                                                double* __restrict__ pot, double* __restrict__ grad) {
  constexpr int TB = sizeof(R) == 4 ? 8 : 4;         // targets per batch
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * (blockDim.x >> 5) + warp;
  if (grp >= ngroups) return;
  const int leaf = gnode[grp];
  const int4 c = cell[leaf];
  const Geometry gn = geo.at(leaf);
  const double w = ldexp(geo.W0, -c.w);
  const double cx = gn.center(0, c.x, w), cy = gn.center(1, c.y, w), cz = gn.center(2, c.z, w);
  const double* L = Ll + (int64_t)leaf * nld;
  const int t0 = gstart[grp], nt = gcount[grp];
  for (int b = 0; b < nt; b += TB) {
    const int nb = min(TB, nt - b);                  // uniform across the warp
    if (nb > TB / 2)
      ki_l2t_batch<R, TB>(t0 + b, nb, tx, ty, tz, tout, L, large, nl, w, cx, cy, cz, lane, outputs, pot, grad);
    else if (nb > TB / 4)
      ki_l2t_batch<R, TB / 2>(t0 + b, nb, tx, ty, tz, tout, L, large, nl, w, cx, cy, cz, lane, outputs, pot, grad);
    else
      ki_l2t_batch<R, TB / 4>(t0 + b, nb, tx, ty, tz, tout, L, large, nl, w, cx, cy, cz, lane, outputs, pot, grad);
  }
}

// The circle method's far field (l2t over the large circle, src/operators/ki_common.jl:293-327):
// Σ_k c·log|x − y_k|² L_k and its gradient Σ_k 2c (x − y_k)/|x − y_k|² L_k, y_k on the leaf's
// circle of radius (4 − √2)/2·w, FP64; writes the outputs (the near field adds to them)
__global__ void __launch_bounds__(128) k_kic_l2t(const int* __restrict__ gnode, const int* __restrict__ gstart,
                                                 const int* __restrict__ gcount, int ngroups, const double* __restrict__ tx,
                                                 const double* __restrict__ ty, const int* __restrict__ tout,
                                                 const int4* __restrict__ cell, const double* __restrict__ Ll, int N,
                                                 Geometry geo, int outputs, double* __restrict__ pot,
                                                 double* __restrict__ grad) {
  __shared__ double sL[4][64], sx[4][64], sy[4][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * 4 + warp;
  if (grp >= ngroups) return;
  const int leaf = gnode[grp];
  const int4 c = cell[leaf];
  const Geometry gn = geo.at(leaf);
  const double w = ldexp(geo.W0, -c.w);
  const double cx = gn.center(0, c.x, w), cy = gn.center(1, c.y, w);
  for (int k = lane; k < N; k += 32) {
    double sn, cs;
    sincospi(2.0 * k / N, &sn, &cs);
    sL[warp][k] = Ll[(int64_t)leaf * 64 + k];
    sx[warp][k] = cx + KIC_LARGE * w * cs;
    sy[warp][k] = cy + KIC_LARGE * w * sn;
  }
  __syncwarp();
  const int t0 = gstart[grp], nt = gcount[grp];
  for (int base = 0; base < nt; base += 32) {
    const int k = t0 + base + lane;
    const bool act = base + lane < nt;
    const double x = act ? tx[k] : cx, y = act ? ty[k] : cy;
    double u = 0, gx = 0, gy = 0;
    for (int q = 0; q < N; ++q) {
      const double dx = x - sx[warp][q], dy = y - sy[warp][q];
      const double r2 = fma(dy, dy, dx * dx);
      u = fma(sL[warp][q], log(r2), u);
      const double g = sL[warp][q] / r2;
      gx = fma(g, dx, gx);
      gy = fma(g, dy, gy);
    }
    if (act) {
      const int o = tout[k];
      if (outputs & FMMB_OUTPUT_POTENTIAL) pot[o] = -KC * u;
      if (outputs & FMMB_OUTPUT_GRADIENT) {
        grad[3 * (int64_t)o] = -2 * KC * gx;
        grad[3 * (int64_t)o + 1] = -2 * KC * gy;
        grad[3 * (int64_t)o + 2] = 0.0;
      }
    }
  }
}

// The near field of charges and dipoles (near.cuh; source_field / target_field of
// src/sources.jl:137-155 with Laplace3D): per source q/r + (d·v)/r³ and the gradient
// −q v/r³ + d/r³ − 3 v (d·v)/r⁵, v = t − s, as KC times the sums below (pot += KC·Σ, grad −= KC·Σ);
// coincident points contribute nothing. R = float: relative to the leaf's centre, batches summed in
// FP32 and their sums in FP64; the reciprocal root correctly rounded, in one step: as 1/√r², in a division and a
// root, it bounded the kernel at this frame's occupancy (500,000 points, 2·10⁶ targets p = 4, the whole evaluation: a
// warp a leaf 3.05 ms, this frame with the division 5.17, with __frsqrt_rn 2.70, five CTAs an SM and four
// sources at a time 2.42; 60,000 points at the sources p = 11 0.198, 0.225, 0.201, 0.192). FP64, 500,000 points and
// targets p = 4: two sources at a time 1.34, four 1.14, with selects 1.05 (a warp a leaf 1.89).
template <typename R>
struct DipolesNear {
  using Real = R;
  static constexpr bool REL = sizeof(R) == 4;
  static constexpr int NA = 4, CH = 2, MINB = REL ? 5 : 4;
  struct Args {
    const double *xs, *ys, *zs, *q, *d3;
    int64_t npts;
    int outputs;
    double *pot, *grad;
  };
  struct Src { double x, y, z, q, dx, dy, dz; };
  struct Stage { R4<R> p[32], d[32]; };
  static __device__ __forceinline__ void load(const Args& a, int j, Src& v) {
    v = Src{a.xs[j], a.ys[j], a.zs[j], a.q[j], a.d3[j], a.d3[a.npts + j], a.d3[2 * a.npts + j]};
  }
  static __device__ __forceinline__ void stage(Stage& st, int lane, const Src& v, double cx, double cy, double cz) {
    st.p[lane] = R4<R>{(R)(v.x - cx), (R)(v.y - cy), (R)(v.z - cz), (R)v.q};
    st.d[lane] = R4<R>{(R)v.dx, (R)v.dy, (R)v.dz, (R)0};
  }
  template <bool CHECK>
  static __device__ __forceinline__ void batch(const Args&, const Stage& st, int m, int is, int part, int f, const R (&t)[3],
                                               double (&acc)[NA]) {
    R bp = 0, bx = 0, by = 0, bz = 0;
#pragma unroll 4
    for (int i = part; i < m; i += f) {
      const R4<R> sv = st.p[i], dv = st.d[i];
      const R vx = t[0] - sv.x, vy = t[1] - sv.y, vz = t[2] - sv.z;
      const R r2 = vx * vx + vy * vy + vz * vz;
      R ir;
      if constexpr (sizeof(R) == 8) ir = rsqrt(r2);
      else ir = __frsqrt_rn(r2);
      if (!(r2 > R(0)) || (CHECK && i == is)) ir = R(0);   // selects: a branch around the root cost a tenth of the time
      const R ir2 = ir * ir, ir3 = ir2 * ir;
      const R dd = dv.x * vx + dv.y * vy + dv.z * vz;
      bp += sv.w * ir + dd * ir3;
      const R cv = sv.w * ir3 + 3 * dd * ir3 * ir2;
      bx += cv * vx - dv.x * ir3;
      by += cv * vy - dv.y * ir3;
      bz += cv * vz - dv.z * ir3;
    }
    acc[0] += bp; acc[1] += bx; acc[2] += by; acc[3] += bz;
  }
  static __device__ __forceinline__ void write(const Args& a, int o, const double (&acc)[NA]) {
    if (a.outputs & FMMB_OUTPUT_POTENTIAL) a.pot[o] += KC * acc[0];
    if (a.outputs & FMMB_OUTPUT_GRADIENT) {
      double* g = a.grad + 3 * (int64_t)o;
#pragma unroll
      for (int d = 0; d < 3; ++d) g[d] -= KC * acc[1 + d];
    }
  }
};

template <int P>
void launch_l2p(State& S, const int* gnode, const int* gstart, const int* gcount, int ng, const double* tx, const double* ty,
                const double* tz, const int* tout, int outputs, double* pot, double* grad, int acc = 0) {
  Plan& P_ = *S.plan;
  // the mixed path evaluates Laplace3D in FP32; Yukawa3D keeps its radial weights in FP64 (its
  // mixed path is the tensor-core M2L only)
  const bool yk = P_.cache->kernel == FMMB_KERNEL_YUKAWA3D;
  const bool mixed = S.precision == FMMB_PRECISION_MIXED && !yk;
  const size_t per_warp = mixed ? l2p_warp_bytes<P, float, false>(P_.cache->ld)
                                : (yk ? l2p_warp_bytes<P, double, true>(P_.cache->ld) : l2p_warp_bytes<P, double, false>(P_.cache->ld));
  // a CTA of four warps a leaf while there are no more than eight leaves an SM, which would leave its warp
  // schedulers idle (a sphere of 31,000 points p = 16: near field and L2P 0.276 → 0.233 ms; Yukawa 40,000
  // points p = 16, the whole pass 1.13 → 1.04); with more, a warp a leaf prepares its own entries without
  // waiting for others
  const int team = ng <= 8 * P_.ctx->num_sms;
  const int warps = team || per_warp > 8192 ? 4 : 8;
  const size_t smem = per_warp * (team ? 1 : warps);
  auto kern = mixed ? k_l2p<P, float, false> : (yk ? k_l2p<P, double, true> : k_l2p<P, double, false>);
  FMMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<team ? ng : (ng + warps - 1) / warps, 32 * warps, smem, P_.ctx->stream>>>(
      gnode, gstart, gcount, ng, tx, ty, tz, tout, P_.cell.p, S.Pl.p, P_.cache->ld, geometry(P_), P_.d_scale.p, outputs, pot,
      grad, P_.d_kh2.p, acc, team);
  FMMB_LAUNCH_CHECK();
}

NearArgs near_args(const Plan& P, const int* gnode, const int* gstart, const int* gcount, int ng, const double* tx,
                   const double* ty, const double* tz, const int* tout) {
  return NearArgs{gnode, gstart, gcount, ng, tx, ty, tz, tout, P.cell.p, P.plo.p, P.phi.p, P.col.p, geometry(P)};
}

template <typename R, bool SELF, int KERNEL = 0>
void launch_near(State& S, const int* gnode, const int* gstart, const int* gcount, int ng, const double* tx, const double* ty,
                 const double* tz, const int* tout, int outputs, double* pot, double* grad, int first = 0,
                 cudaStream_t st = nullptr) {
  Plan& P_ = *S.plan;
  const cudaStream_t s = st ? st : P_.ctx->stream;
  const NearArgs A = near_args(P_, gnode, gstart, gcount, ng, tx, ty, tz, tout);
  auto go = [&](auto pol) {
    using Pol = decltype(pol);
    const typename Pol::Args pa{S.xs.p, S.ys.p, S.zs.p, S.q.p, P_.cache->kappa, outputs, first, pot, grad};
    launch_near_leaves<Pol, SELF>(A, pa, P_.ctx->num_sms, s);
  };
  if (outputs & FMMB_OUTPUT_GRADIENT) go(ChargesNear<R, KERNEL, true>{});
  else go(ChargesNear<R, KERNEL, false>{});
}

template <typename R, bool SELF>
void launch_near_dip(State& S, const int* gnode, const int* gstart, const int* gcount, int ng, const double* tx,
                     const double* ty, const double* tz, const int* tout, int outputs, double* pot, double* grad) {
  Plan& P_ = *S.plan;
  using Pol = DipolesNear<R>;
  const typename Pol::Args pa{S.xs.p, S.ys.p, S.zs.p, S.q.p, S.dip.p, P_.N, outputs, pot, grad};
  launch_near_leaves<Pol, SELF>(near_args(P_, gnode, gstart, gcount, ng, tx, ty, tz, tout), pa, P_.ctx->num_sms,
                                P_.ctx->stream);
}

}  // namespace

void evaluate_groups(State& S, const int* gnode, const int* gstart, const int* gcount, int ng, const double* tx,
                     const double* ty, const double* tz, const int* tout, bool self, int outputs, double* pot, double* grad) {
  if (ng == 0) return;
  if (S.plan->cache->method == FMMB_METHOD_KI_CIRCLE) {
    Plan& P_ = *S.plan;
    k_kic_l2t<<<(ng + 3) / 4, 128, 0, P_.ctx->stream>>>(gnode, gstart, gcount, ng, tx, ty, tout, P_.cell.p, S.ki_ll.p,
                                                        P_.cache->np, geometry(P_), outputs, pot, grad);
    FMMB_LAUNCH_CHECK();
    if (self) launch_near<double, true, 2>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else launch_near<double, false, 2>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    return;
  }
  if (S.plan->cache->method == FMMB_METHOD_CUBE_KI) {
    Plan& P_ = *S.plan;
    Cache& C = *P_.cache;
    const bool mixed = S.precision == FMMB_PRECISION_MIXED;
    const int warps = 4;
    auto kern = mixed ? k_ki_l2t<float> : k_ki_l2t<double>;
    kern<<<(ng + warps - 1) / warps, 32 * warps, 0, P_.ctx->stream>>>(gnode, gstart, gcount, ng, tx, ty, tz, tout,
                                                                       P_.cell.p, S.ki_ll.p, C.ki_nl, C.ki_nld,
                                                                       C.ki_large.p, geometry(P_), outputs, pot, grad);
    FMMB_LAUNCH_CHECK();
    if (mixed && self) launch_near<float, true>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else if (mixed) launch_near<float, false>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else if (self) launch_near<double, true>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else launch_near<double, false>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    return;
  }
  switch (S.plan->cache->p) {
#define X(pp) case pp: launch_l2p<pp>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad); break;
    FMMB_P_CASES(X)
#undef X
    default: throw Error(FMMB_ERR_UNSUPPORTED, "p out of range");
  }
  const bool mixed = S.precision == FMMB_PRECISION_MIXED;
  if (S.has_dip) {
    if (mixed && self) launch_near_dip<float, true>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else if (mixed) launch_near_dip<float, false>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else if (self) launch_near_dip<double, true>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else launch_near_dip<double, false>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    return;
  }
  if (S.plan->cache->kernel == FMMB_KERNEL_YUKAWA3D) {   // the near field in FP64 on both paths
    if (self) launch_near<double, true, 1>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    else launch_near<double, false, 1>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
    return;
  }
  if (mixed && self) launch_near<float, true>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
  else if (mixed) launch_near<float, false>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
  else if (self) launch_near<double, true>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
  else launch_near<double, false>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, outputs, pot, grad);
}

// the harmonic method's evaluation at the sources in two halves: the near field on stream st
// (writing the outputs) and, after it, the far field (adding to them); charges only
bool split_evaluation(const State& S) {
  const Cache& C = *S.plan->cache;
  return C.method == FMMB_METHOD_SPHERICAL_HARMONICS && !S.has_dip &&
         (C.kernel == FMMB_KERNEL_LAPLACE3D || C.kernel == FMMB_KERNEL_YUKAWA3D);
}

void near_sources(State& S, int outputs, double* pot, double* grad, cudaStream_t st) {
  Plan& P = *S.plan;
  if (P.n_leaves == 0) return;
  const bool mixed = S.precision == FMMB_PRECISION_MIXED;
  const double *tx = S.xs.p, *ty = S.ys.p, *tz = S.zs.p;
  if (P.cache->kernel == FMMB_KERNEL_YUKAWA3D)
    launch_near<double, true, 1>(S, P.leaves.p, P.leaf_start.p, P.leaf_count.p, P.n_leaves, tx, ty, tz, P.perm.p, outputs,
                                 pot, grad, 1, st);
  else if (mixed)
    launch_near<float, true>(S, P.leaves.p, P.leaf_start.p, P.leaf_count.p, P.n_leaves, tx, ty, tz, P.perm.p, outputs, pot,
                             grad, 1, st);
  else
    launch_near<double, true>(S, P.leaves.p, P.leaf_start.p, P.leaf_count.p, P.n_leaves, tx, ty, tz, P.perm.p, outputs, pot,
                              grad, 1, st);
}

void far_sources(State& S, int outputs, double* pot, double* grad) {
  Plan& P = *S.plan;
  if (P.n_leaves == 0) return;
  switch (P.cache->p) {
#define X(pp)                                                                                                    \
  case pp:                                                                                                       \
    launch_l2p<pp>(S, P.leaves.p, P.leaf_start.p, P.leaf_count.p, P.n_leaves, S.xs.p, S.ys.p, S.zs.p, P.perm.p, outputs, \
                   pot, grad, 1);                                                                                \
    break;
    FMMB_P_CASES(X)
#undef X
    default: throw Error(FMMB_ERR_UNSUPPORTED, "p out of range");
  }
}

}  // namespace fmmb
