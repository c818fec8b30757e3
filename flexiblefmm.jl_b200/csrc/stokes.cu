// StokesHarmonics(Stokeslet3D(); p) on the plain FP64 path (src/operators/harmonics_stokes.jl):
// the Stokeslet through four Laplace potentials, Φ_k = Σ f_k/(4πr) and Ψ_c = Σ (y − c)·f/(4πr),
// u = ½[Φ − (x − c)·∇Φ + ∇Ψ_c]. Every node holds the four scalar expansions [Φ₁; Φ₂; Φ₃; Ψ̂]
// (Ψ̂ = Ψ_c/w in the box's own coordinates), nexp·LD apart; they use the scalar operators of
// SphericalHarmonics with the couplings of the reference:
//   P2M  block k: charges f_k; block 4: charges ŷ·f (ŷ = (y − c)/w)        (harmonics_stokes.jl:322-328)
//   M2M  Ψ̂_P = Σ M2M(½ Ψ̂_C + δ̂·Φ_C), δ̂ = (c_C − c_P)/w_P ∈ {±¼}³          (:136-158)
//   M2L  Ψ̂_B += T(Ψ̂_A + o·Φ_A), o the far offset                             (:77-97)
//   L2L  Ψ̂_C += L2L(2Ψ̂_P − 2 δ̂·Φ_P)                                          (:159-183)
//        (each is linear in the source: the translations' gather forms it, m2l_rot.cu)
//   L2P  u = ½[Φ − x̂·∇̂Φ + ∇̂Ψ̂] from the values and scaled gradients of the four blocks (:283-287)
//   near c(f/r + d(d·f)/r³), c = 1/(8π), self excluded by index (src/kernels.jl:253-272)
// Stresslets (f, ν) and doublets g (src/sources.jl:203-281) enter as dipole densities
// (harmonics_stokes.jl:205-216,382-393): block k takes the dipole −(f_k ν + ν_k f), block 4 the
// dipole −((ν·ŷ) f + (f·ŷ) ν) + g/w; the translations and L2P are the same. The pressure is
// −∇·Φ (−s·tr of the scaled gradients of blocks 1–3, :343-346) plus the near-field pressures
// 2c(d·f)/r³ and 4c[(f·ν)/r³ − 3(d·f)(d·ν)/r⁵] (a doublet has none).
#include <type_traits>

#include "near.cuh"

namespace fmmb {
namespace {

constexpr double KSTOKES = 0.039788735772973833942;   // 1/(8π)
constexpr int SW = 4;                                  // warps per block of the evaluation kernels

inline unsigned nblk(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// points and densities in tree order (perm: sorted position → original index), weighted: the
// Stokeslets into f3 (zeros when absent), the stresslet strengths, stressvecs and doublets into
// sd (3 × n planar each, zeros when absent) when sd is given
__global__ void k_stokes_gather(const double* __restrict__ xyz, StokesDensities d, const int* __restrict__ perm,
                                int64_t n, double* __restrict__ xs, double* __restrict__ ys, double* __restrict__ zs,
                                double* __restrict__ f3, double* __restrict__ sd) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t j = perm[i];
  xs[i] = xyz[3 * j];
  ys[i] = xyz[3 * j + 1];
  zs[i] = xyz[3 * j + 2];
  const double wt = d.weights ? d.weights[j] : 1.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) f3[k * n + i] = d.stokeslets ? wt * d.stokeslets[3 * j + k] : 0.0;
  if (sd) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      sd[k * n + i] = d.stresslets ? wt * d.stresslets[3 * j + k] : 0.0;
      sd[(3 + k) * n + i] = d.stresslets ? d.stressvecs[3 * j + k] : 0.0;
      sd[(6 + k) * n + i] = d.doublets ? wt * d.doublets[3 * j + k] : 0.0;
    }
  }
}

// the fourth P2M block's charges ŷ·f, ŷ = (y − c)·s relative to the centre c of the node whose
// multipole the point enters, s = 1/w; with DENS also the four blocks' dipoles (3 × n planar per
// block, in physical units: the P2M scales them by s): −(f_k ν + ν_k f) for block k and
// −((ν·ŷ) f + (f·ŷ) ν) + g·s for block 4 (f, ν the stresslet, g the doublet)
template <bool DENS>
__global__ void k_stokes_q4(const int* __restrict__ nodes, int nn, const int4* __restrict__ cell,
                            const int* __restrict__ plo, const int* __restrict__ phi, Geometry geo,
                            const double* __restrict__ scale, int64_t n, const double* __restrict__ xs,
                            const double* __restrict__ ys, const double* __restrict__ zs, const double* __restrict__ f3,
                            const double* __restrict__ sd, double* __restrict__ q4, double* __restrict__ dip4) {
  // one warp per childless node with sources (the nodes P2M runs on, ghost children of a leaf
  // included): Ψ̂ is centred on the node whose multipole it starts
  const int wid = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (wid >= nn) return;
  const int node = nodes[wid];
  const int4 c = cell[node];
  const Geometry gn = geo.at(node);
  const double w = ldexp(geo.W0, -c.w), s = scale[c.w];
  const double cx = gn.center(0, c.x, w), cy = gn.center(1, c.y, w), cz = gn.center(2, c.z, w);
  for (int i = plo[node] + lane; i <= phi[node]; i += 32) {
    const double y[3] = {(xs[i] - cx) * s, (ys[i] - cy) * s, (zs[i] - cz) * s};
    q4[i] = y[0] * f3[i] + y[1] * f3[n + i] + y[2] * f3[2 * n + i];
    if (DENS) {
      double f[3], nu[3], g[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        f[k] = sd[k * n + i];
        nu[k] = sd[(3 + k) * n + i];
        g[k] = sd[(6 + k) * n + i];
      }
      const double ny = nu[0] * y[0] + nu[1] * y[1] + nu[2] * y[2], fy = f[0] * y[0] + f[1] * y[1] + f[2] * y[2];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int e = 0; e < 3; ++e) dip4[(3 * k + e) * n + i] = -(f[k] * nu[e] + nu[k] * f[e]);
        dip4[(9 + k) * n + i] = -(ny * f[k] + fy * nu[k]) + g[k] * s;
      }
    }
  }
}

// The far field at the targets of one leaf: u_i = ½[Φ_i + ∂̂_iΨ̂ − Σ_k x̂_k ∂̂_iΦ_k], or with PRES the
// pressure −s·Σ_k ∂̂_kΦ_k. A CTA of four warps takes a leaf: all of them prepare its entries (m, n) in shared
// memory, NV coefficient pairs each (Φ_i + ∂̂_iΨ̂, then ∂̂_iΦ_k at 3 + 3i + k; PRES: the divergence), then a
// warp 32 targets at a time runs the recurrence once for all of them. Bound by the entries' shared-memory
// reads. Measured (four unprepared L2Ps per target, a warp a leaf → this): 13,704 leaves of twelve spheres p = 16
// 3.06 → 1.34 ms; 332 leaves and 395 of targets p = 12 0.84 → 0.072 (the whole call with densities 2.50 → 1.72).
template <int P, bool PRES>
__global__ void __launch_bounds__(SW * 32) k_stokes_l2p(const int* __restrict__ gnode, const int* __restrict__ gstart,
                                                        const int* __restrict__ gcount, const double* __restrict__ tx,
                                                        const double* __restrict__ ty, const double* __restrict__ tz,
                                                        const int* __restrict__ tout, const int4* __restrict__ cell,
                                                        const double* __restrict__ Pl, int LD, Geometry geo,
                                                        const double* __restrict__ scale, double* __restrict__ out) {
  constexpr int NV = PRES ? 1 : 12;
  extern __shared__ __align__(16) double sl[];
  double2* E = reinterpret_cast<double2*>(sl);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = blockIdx.x;
  const int leaf = gnode[grp];
  const double* L = Pl + (int64_t)leaf * 4 * LD;
  for (int q = threadIdx.x; q < l2p_entries<P>(); q += SW * 32) {
    double v[3][8], psi[8];
#pragma unroll
    for (int a = 0; a < 3; ++a) l2p_values<P>(L + a * LD, q, v[a]);
    if (PRES) {
      E[q] = make_double2(v[0][2] + v[1][4] + v[2][6], v[0][3] + v[1][5] + v[2][7]);
    } else {
      l2p_values<P>(L + 3 * LD, q, psi);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        E[NV * q + i] = make_double2(v[i][0] + psi[2 + 2 * i], v[i][1] + psi[3 + 2 * i]);
#pragma unroll
        for (int k = 0; k < 3; ++k) E[NV * q + 3 + 3 * i + k] = make_double2(v[k][2 + 2 * i], v[k][3 + 2 * i]);
      }
    }
  }
  __syncthreads();
  const int4 c = cell[leaf];
  const Geometry gn = geo.at(leaf);
  const double w = ldexp(geo.W0, -c.w), s = scale[c.w];
  const double cx = gn.center(0, c.x, w), cy = gn.center(1, c.y, w), cz = gn.center(2, c.z, w);
  const int t0 = gstart[grp], nt = gcount[grp];
  for (int base = 32 * warp; base < nt; base += 32 * SW) {
    const int k = t0 + base + lane;
    const bool act = base + lane < nt;
    const double x = act ? (tx[k] - cx) * s : 0.0, y = act ? (ty[k] - cy) * s : 0.0, z = act ? (tz[k] - cz) * s : 0.0;
    const double r2 = x * x + y * y + z * z;
    double acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = 0.0;
    double sr = 1.0, si = 0.0;
    const double2* e = E;
#pragma unroll 1
    for (int m = 0; m <= P; ++m) {
      double pr = 0.0, pi = 0.0, vr = sr, vi = si;
#pragma unroll 1
      for (int n = m; n <= P; ++n, e += NV) {
        if (n > m) {                                     // uniform
          const int t = tri(n, m);
          const double az = c_tab[t] * z, br = c_tab[TRI_MAX + t] * r2;
          const double nr = az * vr - br * pr, ni = az * vi - br * pi;
          pr = vr; pi = vi; vr = nr; vi = ni;
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const double2 a = e[i];
          acc[i] = fma(a.y, vi, fma(a.x, vr, acc[i]));
        }
      }
      if (m < P) {
        const double f = c_e[m], nr = -f * (x * sr - y * si), ni = -f * (x * si + y * sr);
        sr = nr; si = ni;
      }
    }
    if (act) {
      const int o = tout[k];
      if constexpr (PRES) {
        out[o] = -s * acc[0];
      } else {
#pragma unroll
        for (int i = 0; i < 3; ++i)
          out[3 * (int64_t)o + i] = 0.5 * (acc[i] - (x * acc[3 + 3 * i] + y * acc[4 + 3 * i] + z * acc[5 + 3 * i]));
      }
    }
  }
}

// the scaled gradient of a local expansion L of degree P as three expansions of degree P − 1 in
// the real storage (n², and re/im of order m at n² + 2m − 1, n² + 2m), from the derivative
// identities (harmonics_stokes.jl:231-240, harmonics.jl:465-486): (D₋L)_n^m = −cm(n+1, m+1) L_{n+1}^{m+1},
// (D₊L)_n^m = cp(n+1, m−1) L_{n+1}^{m−1}, (D_zL)_n^m = cz(n+1, m) L_{n+1}^m, ∂̂_x = ½(D₋ + D₊),
// ∂̂_y = (i/2)(D₊ − D₋), ∂̂_z = D_z; the lanes of a warp share the P² entries
template <int P>
__device__ void grad_sets(const double* __restrict__ L, double* __restrict__ Ax, double* __restrict__ Ay,
                          double* __restrict__ Az, int lane) {
  for (int e = lane; e < P * P; e += 32) {
    int n = (int)sqrtf((float)e);
    while (n * n > e) --n;
    while ((n + 1) * (n + 1) <= e) ++n;
    const int k = e - n * n, m = (k + 1) / 2, n1 = n + 1, b = n1 * n1;
    const bool im = k > 0 && (k & 1) == 0;
    if (m == 0) {
      const double cmv = c_tab[3 * TRI_MAX + tri(n1, 1)];
      Ax[e] = -cmv * L[b + 1];
      Ay[e] = -cmv * L[b + 2];
      Az[e] = c_tab[2 * TRI_MAX + tri(n1, 0)] * L[b];
    } else {
      const double ur = L[b + 2 * (m + 1) - 1], ui = L[b + 2 * (m + 1)];
      const double dr = m == 1 ? L[b] : L[b + 2 * (m - 1) - 1], di = m == 1 ? 0.0 : L[b + 2 * (m - 1)];
      const double cu = 0.5 * c_tab[3 * TRI_MAX + tri(n1, m + 1)], cd = 0.5 * c_tab[4 * TRI_MAX + tri(n1, m - 1)];
      const double czv = c_tab[2 * TRI_MAX + tri(n1, m)];
      Ax[e] = im ? -cu * ui + cd * di : -cu * ur + cd * dr;
      Ay[e] = im ? cu * ur + cd * dr : -(cu * ui + cd * di);
      Az[e] = czv * (im ? L[b + 2 * m] : L[b + 2 * m - 1]);
    }
  }
}

constexpr int GW = 2;   // warps per block of the velocity-gradient L2P

// the far-field velocity gradient at the targets of one leaf (harmonics_stokes.jl:347-350):
// ∂u_i/∂t_j = (s/2)[∂̂_jΦ_i − ∂̂_iΦ_j − Σ_k x̂_k ∂̂_i∂̂_jΦ_k + ∂̂_i∂̂_jΨ̂], written at 9·o + 3i + j. Per
// warp the leaf's four blocks and their twelve gradient expansions sit in shared memory; per target
// twelve degree-(P−1) L2Ps give the first and second derivatives.
template <int P>
__global__ void __launch_bounds__(GW * 32) k_stokes_l2p_grad(const int* __restrict__ gnode, const int* __restrict__ gstart,
                                                             const int* __restrict__ gcount, int ngroups,
                                                             const double* __restrict__ tx, const double* __restrict__ ty,
                                                             const double* __restrict__ tz, const int* __restrict__ tout,
                                                             const int4* __restrict__ cell, const double* __restrict__ Pl,
                                                             int LD, Geometry geo, const double* __restrict__ scale,
                                                             double* __restrict__ out) {
  extern __shared__ double sg[];
  constexpr int NG = P * P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * GW + warp;
  if (grp >= ngroups) return;
  double* L = sg + (int64_t)warp * (4 * LD + 12 * NG);
  double* A = L + 4 * LD;   // block a, direction j at A + (3a + j)·NG
  const int leaf = gnode[grp];
  for (int i = lane; i < 4 * LD; i += 32) L[i] = Pl[(int64_t)leaf * 4 * LD + i];
  __syncwarp();
  for (int a = 0; a < 4; ++a) grad_sets<P>(L + a * LD, A + 3 * a * NG, A + (3 * a + 1) * NG, A + (3 * a + 2) * NG, lane);
  __syncwarp();
  const int4 c = cell[leaf];
  const Geometry gn = geo.at(leaf);
  const double w = ldexp(geo.W0, -c.w), s = scale[c.w];
  const double cx = gn.center(0, c.x, w), cy = gn.center(1, c.y, w), cz = gn.center(2, c.z, w);
  const int t0 = gstart[grp], nt = gcount[grp];
  for (int base = 0; base < nt; base += 32) {
    const int k = t0 + base + lane;
    const bool act = base + lane < nt;
    const double xh[3] = {act ? (tx[k] - cx) * s : 0.0, act ? (ty[k] - cy) * s : 0.0, act ? (tz[k] - cz) * s : 0.0};
    double gr[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int a = 0; a < 4; ++a) {
      const double coef = a < 3 ? -xh[a] : 1.0;
      for (int j = 0; j < 3; ++j) {
        double v, h[3];
        l2p<P - 1, double>(A + (3 * a + j) * NG, xh[0], xh[1], xh[2], v, h[0], h[1], h[2]);
        if (a < 3) {   // v = ∂̂_jΦ_a: +v at (a, j), −v at (j, a)
          gr[a][j] += v;
          gr[j][a] -= v;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) gr[i][j] += coef * h[i];   // h_i = ∂̂_i∂̂_j of block a
      }
    }
    if (act) {
      const int o = tout[k];
#pragma unroll
      for (int e = 0; e < 9; ++e) out[9 * (int64_t)o + e] = 0.5 * s * gr[e / 3][e % 3];
    }
  }
}

// The near field (near.cuh): adds c·Σ to the velocities (OUT 0),
// the pressures (OUT 1) or the velocity gradients (OUT 2, ∂u_i/∂t_j at 9·o + 3i + j). DENS adds
// the stresslets and doublets of sd (3 × n planar: strengths, stressvecs, doublets) to the
// Stokeslets (src/sources.jl:203-281):
//   u = c[f/r + g/r³ + d((d·f)/r³ − 3(d·g)/r⁵ − 6(d·f_s)(d·ν)/r⁵)],  p = c[2(d·f)/r³ + 4(f_s·ν)/r³ − 12(d·f_s)(d·ν)/r⁵]
//   ∂u_i/∂t_j = c[d_i(A d_j + v_j) + w_i d_j + B δ_ij] with A = −3(d·f)/r⁵ + (30(d·f_s)(d·ν) + 15(d·g))/r⁷,
//   B = (d·f)/r³ − (6(d·f_s)(d·ν) + 3(d·g))/r⁵, v = f/r³ − 6((d·ν) f_s + (d·f_s) ν)/r⁵ − 3g/r⁵,
//   w = −f/r³ − 3g/r⁵ (the closed forms of the three gradients, summed)
template <bool DENS, int OUT>
struct StokesNear {
  using Real = double;
  static constexpr bool REL = false;
  static constexpr int NA = OUT == 2 ? 9 : (OUT == 1 ? 1 : 3), CH = DENS || OUT == 2 ? 1 : 2, MINB = 4;
  struct Args {
    const double *xs, *ys, *zs, *f3, *sd;
    int64_t n;
    double* out;
  };
  struct alignas(16) S8 { double x, y, z, fx, fy, fz; };
  struct alignas(16) S16 { double x, y, z, fx, fy, fz, sx, sy, sz, nx, ny, nz, gx, gy, gz, pad; };
  using SV = std::conditional_t<DENS, S16, S8>;
  using Src = SV;
  struct Stage { SV s[32]; };
  static __device__ __forceinline__ void load(const Args& a, int j, Src& v) {
    const int64_t n = a.n;
    if constexpr (DENS)
      v = SV{a.xs[j],         a.ys[j],         a.zs[j],         a.f3[j],         a.f3[n + j],     a.f3[2 * n + j],
             a.sd[j],         a.sd[n + j],     a.sd[2 * n + j], a.sd[3 * n + j], a.sd[4 * n + j], a.sd[5 * n + j],
             a.sd[6 * n + j], a.sd[7 * n + j], a.sd[8 * n + j], 0};
    else
      v = SV{a.xs[j], a.ys[j], a.zs[j], a.f3[j], a.f3[n + j], a.f3[2 * n + j]};
  }
  static __device__ __forceinline__ void stage(Stage& st, int lane, const Src& v, double, double, double) { st.s[lane] = v; }
  template <bool CHECK>
  static __device__ __forceinline__ void batch(const Args&, const Stage& st, int m, int is, int part, int f,
                                               const double (&t)[3], double (&acc)[NA]) {
#pragma unroll 2
    for (int i = part; i < m; i += f) {
      const SV sv = st.s[i];
      const double dx = t[0] - sv.x, dy = t[1] - sv.y, dz = t[2] - sv.z;
      const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
      double ir = rsqrt(r2);
      if (CHECK && i == is) ir = 0.0;
      const double ir3 = ir * ir * ir;
      const double df = dx * sv.fx + dy * sv.fy + dz * sv.fz;
      if constexpr (OUT == 2) {
        const double ir2 = ir * ir, ir5 = ir3 * ir2;
        const double d[3] = {dx, dy, dz};
        double A = -3.0 * df * ir5, B = df * ir3;
        double v[3] = {sv.fx * ir3, sv.fy * ir3, sv.fz * ir3}, w[3] = {-v[0], -v[1], -v[2]};
        if constexpr (DENS) {
          const double ds = dx * sv.sx + dy * sv.sy + dz * sv.sz, dn = dx * sv.nx + dy * sv.ny + dz * sv.nz;
          const double dg = dx * sv.gx + dy * sv.gy + dz * sv.gz;
          A += (30.0 * ds * dn + 15.0 * dg) * ir5 * ir2;
          B -= (6.0 * ds * dn + 3.0 * dg) * ir5;
          const double fs[3] = {sv.sx, sv.sy, sv.sz}, nu[3] = {sv.nx, sv.ny, sv.nz}, g[3] = {sv.gx, sv.gy, sv.gz};
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            v[e] -= (6.0 * (dn * fs[e] + ds * nu[e]) + 3.0 * g[e]) * ir5;
            w[e] -= 3.0 * g[e] * ir5;
          }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
#pragma unroll
          for (int b = 0; b < 3; ++b) acc[3 * a + b] += d[a] * (A * d[b] + v[b]) + w[a] * d[b] + (a == b ? B : 0.0);
        }
      } else if constexpr (DENS) {
        const double ir5 = ir3 * ir * ir;
        const double ds = dx * sv.sx + dy * sv.sy + dz * sv.sz, dn = dx * sv.nx + dy * sv.ny + dz * sv.nz;
        if constexpr (OUT == 1) {
          const double sn = sv.sx * sv.nx + sv.sy * sv.ny + sv.sz * sv.nz;
          acc[0] += 2.0 * df * ir3 + 4.0 * sn * ir3 - 12.0 * ds * dn * ir5;
        } else {
          const double dg = dx * sv.gx + dy * sv.gy + dz * sv.gz;
          const double c = df * ir3 - (3.0 * dg + 6.0 * ds * dn) * ir5;
          acc[0] += sv.fx * ir + sv.gx * ir3 + dx * c;
          acc[1] += sv.fy * ir + sv.gy * ir3 + dy * c;
          acc[2] += sv.fz * ir + sv.gz * ir3 + dz * c;
        }
      } else if constexpr (OUT == 1) {
        acc[0] += 2.0 * df * ir3;
      } else {
        const double c = df * ir3;
        acc[0] += sv.fx * ir + dx * c;
        acc[1] += sv.fy * ir + dy * c;
        acc[2] += sv.fz * ir + dz * c;
      }
    }
  }
  static __device__ __forceinline__ void write(const Args& a, int o, const double (&acc)[NA]) {
#pragma unroll
    for (int e = 0; e < NA; ++e) a.out[NA * (int64_t)o + e] += KSTOKES * acc[e];
  }
};

template <int P>
void launch_stokes_l2p(State& S, const int* gnode, const int* gstart, const int* gcount, int ng, const double* tx,
                       const double* ty, const double* tz, const int* tout, int output, double* out) {
  Plan& P_ = *S.plan;
  const int LD = P_.cache->ld;
  if (output == FMMB_STOKES_GRADIENT) {
    const size_t smem = sizeof(double) * GW * (4 * LD + 12 * P * P);
    FMMB_CUDA(cudaFuncSetAttribute(k_stokes_l2p_grad<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_stokes_l2p_grad<P><<<(ng + GW - 1) / GW, GW * 32, smem, P_.ctx->stream>>>(
        gnode, gstart, gcount, ng, tx, ty, tz, tout, P_.cell.p, S.Pl.p, LD, geometry(P_), P_.d_scale.p, out);
    FMMB_LAUNCH_CHECK();
    return;
  }
  const bool pres = output == FMMB_STOKES_PRESSURE;
  const size_t smem = sizeof(double2) * (pres ? 1 : 12) * l2p_entries<P>();
  auto kern = pres ? k_stokes_l2p<P, true> : k_stokes_l2p<P, false>;
  FMMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<ng, SW * 32, smem, P_.ctx->stream>>>(gnode, gstart, gcount, tx, ty, tz, tout, P_.cell.p, S.Pl.p, LD, geometry(P_),
                                              P_.d_scale.p, out);
  FMMB_LAUNCH_CHECK();
}

}  // namespace

// build_expansions! of a Stokes state from the densities of stokes_fmm_eval! (device, original
// order)
void stokes_build(State& S, const double* xyz_dev, const StokesDensities& d) {
  Plan& P = *S.plan;
  Cache& C = *P.cache;
  cudaStream_t s = P.ctx->stream;
  const int LD = C.ld;
  const int64_t n = P.N, pitch = 4 * (int64_t)LD;
  const bool dens = d.stresslets || d.doublets;
  if (S.f3.n < (size_t)(3 * n)) S.f3.alloc(3 * n);
  if (S.q.n < (size_t)n) S.q.alloc(n);
  if (dens && S.sd.n < (size_t)(9 * n)) S.sd.alloc(9 * n);
  if (dens && S.dip4.n < (size_t)(12 * n)) S.dip4.alloc(12 * n);
  k_stokes_gather<<<nblk(n), 256, 0, s>>>(xyz_dev, d, P.perm.p, n, S.xs.p, S.ys.p, S.zs.p, S.f3.p,
                                          dens ? S.sd.p : nullptr);
  FMMB_LAUNCH_CHECK();
  S.stokes_dens = dens;
  if (P.n_s2m > 0) {
    auto kern = dens ? k_stokes_q4<true> : k_stokes_q4<false>;
    kern<<<nblk((int64_t)P.n_s2m * 32), 256, 0, s>>>(P.s2m_nodes.p, P.n_s2m, P.cell.p, P.plo.p, P.phi.p, geometry(P),
                                                     P.d_scale.p, n, S.xs.p, S.ys.p, S.zs.p, S.f3.p,
                                                     dens ? S.sd.p : nullptr, S.q.p, dens ? S.dip4.p : nullptr);
    FMMB_LAUNCH_CHECK();
  }
  // P2M of the four blocks (charges, and the dipoles of the stresslets and doublets)
  const double *q4[4], *d4[4];
  double* M4[4];
  for (int a = 0; a < 4; ++a) {
    q4[a] = a < 3 ? S.f3.p + a * n : S.q.p;
    d4[a] = dens ? S.dip4.p + 3 * a * n : nullptr;
    M4[a] = S.M.p + (int64_t)a * LD;
  }
  p2m_blocks(S, 4, q4, d4, M4, pitch);
  // M2M, level by level, then the M2L of every block and L2L, each with the Ψ̂ coupling
  m2m_sweep(S);
  m2l_stage(S);
  l2l_sweep(S);
  S.built = true;
}

namespace {

// the far and near fields at ng groups of targets (per leaf: node, first, count), targets in
// group order with their output indices tout; self: the targets are the sources (i = j skipped)
void stokes_evaluate_groups(State& S, const int* gnode, const int* gstart, const int* gcount, int ng, const double* tx,
                            const double* ty, const double* tz, const int* tout, bool self, int output, double* out) {
  Plan& P = *S.plan;
  require(output == FMMB_STOKES_VELOCITY || output == FMMB_STOKES_PRESSURE || output == FMMB_STOKES_GRADIENT,
          FMMB_ERR_UNSUPPORTED, "Stokes outputs are the velocity, the pressure and the velocity gradient");
  if (ng == 0) return;
  switch (P.cache->p) {
#define X(pp) case pp: launch_stokes_l2p<pp>(S, gnode, gstart, gcount, ng, tx, ty, tz, tout, output, out); break;
    FMMB_P_CASES(X)
#undef X
    default: throw Error(FMMB_ERR_UNSUPPORTED, "p out of range");
  }
  const bool d = S.stokes_dens;
  const NearArgs A{gnode, gstart, gcount, ng, tx, ty, tz, tout, P.cell.p, P.plo.p, P.phi.p, P.col.p, geometry(P)};
  auto go = [&](auto pol) {
    using Pol = decltype(pol);
    const typename Pol::Args pa{S.xs.p, S.ys.p, S.zs.p, S.f3.p, d ? S.sd.p : nullptr, P.N, out};
    if (self) launch_near_leaves<Pol, true>(A, pa, P.ctx->num_sms, P.ctx->stream);
    else launch_near_leaves<Pol, false>(A, pa, P.ctx->num_sms, P.ctx->stream);
  };
  if (output == FMMB_STOKES_VELOCITY) d ? go(StokesNear<true, 0>{}) : go(StokesNear<false, 0>{});
  else if (output == FMMB_STOKES_PRESSURE) d ? go(StokesNear<true, 1>{}) : go(StokesNear<false, 1>{});
  else d ? go(StokesNear<true, 2>{}) : go(StokesNear<false, 2>{});
}

}  // namespace

// evaluate_at_sources! of a Stokes state: velocities (3 × n) or pressures (n), original order,
// device, self excluded
void stokes_evaluate_sources(State& S, int output, double* out_dev) {
  Plan& P = *S.plan;
  stokes_evaluate_groups(S, P.leaves.p, P.leaf_start.p, P.leaf_count.p, P.n_leaves, S.xs.p, S.ys.p, S.zs.p, P.perm.p, true,
                         output, out_dev);
}

// evaluate! of a Stokes state at nt targets (device, 3 × nt): velocities (3 × nt) or pressures
// (nt) in the targets' order, device
void stokes_evaluate_targets(State& S, const double* tg_dev, int64_t nt, int output, double* out_dev) {
  if (nt == 0) return;
  const int ng = group_targets(S, tg_dev, nt);
  const int* g = S.t_groups.p;
  stokes_evaluate_groups(S, g, g + nt, g + 2 * nt, ng, S.t_x.p, S.t_y.p, S.t_z.p, S.t_out.p, false, output, out_dev);
}

}  // namespace fmmb
