// P2M: the multipoles of the childless nodes with sources,
// M_n^m = Σ τ conj Υ̃_n^m((y − c)/w) (src/device_passes.jl:343-373, harmonics.jl:682-743).
//
// A warp takes a node, 32 of its sources at a time: a lane per source scales it into the box and
// forms the sectoral values Υ̃_m^m, m = 0..P (and Yukawa3D's radial weights), into shared memory; then
// the lanes are (pair of orders h and P − h) × (subset of the sources): the two recurrences over the
// degree have P + 2 steps together for every h, so the lanes stay together, the sums of the P + 2
// values live in registers, and the subsets' sums meet in shared memory once per node. Nodes with more
// than P2M_ALONE sources are shared by the four warps of the CTA, every fourth 32 sources each; nodes of at
// most 16 (8) sources share a warp by twos (fours) up to p = 15, each with its part of the lanes and subsets. How
// a node's sums are split depends on its own sources only. Dipoles are three more charge sets (and Stokes has
// four of each): where the list fills the SMs a CTA takes all sets of its nodes and stages the sources once.
// One thread per (node, order) would read every source P + 1 times from 32 scattered places per load
// instruction, and leave few threads on small trees; that bounded it. Measured (that form → this): a
// million points p = 11 in FP32 0.269 → 0.090 ms, 400,000 p = 10 in FP64 0.155 → 0.102, 400,000 p = 16
// 0.364 → 0.183, a sphere of 31,000 p = 16 0.183 → 0.030; a million points in leaves of at most 16, p = 6 in FP32,
// 0.215 → 0.160 (0.410 with a warp per node), p = 10 0.552 → 0.265; 500,000 dipoles p = 5 mixed, the whole build,
// 0.921 → 0.873 (1.024 with the sets apart and a warp per node). What bounds it now is the recurrences' FMAs and
// their shared-memory reads (2P + 5 words a source and order pair).
#include <algorithm>
#include <type_traits>

#include "passes.cuh"

namespace fmmb {
namespace {

constexpr int P2M_WARPS = 4, P2M_ALONE = 64, P2M_SETS = 16;

// the charges and where their multipoles go: of the first nnode sets node g's at out + g·pitch, of the others
// the i-th of the node list's at out + i·ipitch
struct P2MSets {
  const double* q[P2M_SETS];
  double* out[P2M_SETS];
  int64_t pitch, ipitch;
  int nnode, n;
};

template <int P, bool YK, typename R>
struct P2MShape {
  static constexpr int H = (P + 2) / 2, NS = 32 / H, K = P + 2;   // order pairs, source subsets, steps
  // per warp, 32 each: z, r², τ, the sectoral values (and the radial weights); the sums after them
  static constexpr int WARP = 32 * (3 + 2 * (P + 1) + (YK ? P + 1 : 0));
  static_assert(32 * 2 * K <= WARP, "the sums reuse the staging");
  static constexpr bool PACK = NS >= 4;                           // nodes of few sources share a warp
  static constexpr size_t smem(bool many) { return sizeof(R) * (P2M_WARPS * (WARP + (many ? 64 * K : 0)) + 2 * K * H); }
};

// npw nodes per warp (0: one per CTA). MANY: a CTA takes all sets of its nodes, one after the other, and stages
// the sources once for all of them where each warp has one batch
template <int P, bool YK, typename R, bool MANY>
__global__ void __launch_bounds__(32 * P2M_WARPS, sizeof(R) == 4 ? 5 : 3) k_p2m(const int* __restrict__ nodes, int nn, const int4* __restrict__ cell,
                                                        const int* __restrict__ plo, const int* __restrict__ phi,
                                                        const double* __restrict__ xs, const double* __restrict__ ys,
                                                        const double* __restrict__ zs, const P2MSets sets, Geometry geo,
                                                        const double* __restrict__ scale, const double* __restrict__ kh2,
                                                        int npw) {
  static_assert(!YK || sizeof(R) == 8, "Yukawa3D's P2M runs in FP64");
  using Sh = P2MShape<P, YK, R>;
  constexpr int H = Sh::H, NS = Sh::NS, K = Sh::K, SUMS = MANY ? Sh::WARP : 0, WS = Sh::WARP + (MANY ? 64 * K : 0);
  extern __shared__ __align__(16) unsigned char p2m_raw[];
  R* ab = reinterpret_cast<R*>(p2m_raw);                        // [K][H] recurrence factors (a, b)
  R* st0 = ab + 2 * K * H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = lane % H, sub = lane / H;
  R* st = st0 + warp * WS;
  R *sz = st, *sr2 = st + 32, *sq = st + 64, *ss = st + 96, *su = st + 96 + 64 * (P + 1);
  for (int i = threadIdx.x; i < K * H; i += blockDim.x) {
    const int k = i / H, hh = i % H, m = k <= P - hh ? hh : P - hh, n = k <= P - hh ? hh + k : k - 1;   // m + k − (P − h + 1) = k − 1
    ab[2 * i] = n > m ? ctab<R>(tri(n, m)) : R(0);
    ab[2 * i + 1] = n > m ? ctab<R>(TRI_MAX + tri(n, m)) : R(0);
  }
  __syncthreads();
  // the sums of set a over the batches who, who + team, ... of G nodes (G > 1: one batch), 32 / G lanes staging
  // and NS / G subsets each, into the warp's own part of shared memory; node: this lane's; ccnt: the source count
  // of the node this lane sums for; staged: the batch lies there but for the charges
  auto sums = [&](auto pack, int node, int ccnt, int who, int team, int a, bool staged) {
    constexpr int G = decltype(pack)::value, W = 32 / G, SUB = NS / G;
    const double* q = sets.q[a];
    const int4 c = cell[node];
    const Geometry gn = geo.at(node);
    const double w = ldexp(geo.W0, -c.w), s = scale[c.w];
    const double cx = gn.center(0, c.x, w), cy = gn.center(1, c.y, w), cz = gn.center(2, c.z, w);
    const int j0 = plo[node], cnt = phi[node] - j0 + 1, l = lane % W;
    R ar[K], ai[K];
#pragma unroll
    for (int k = 0; k < K; ++k) { ar[k] = 0; ai[k] = 0; }
    for (int b = 32 * who; b < (G > 1 ? 1 : cnt); b += 32 * team) {
      const int m = min(32, cnt - b), cm = G > 1 ? ccnt : m;
      __syncwarp();                                             // the previous batch is read
      if (l < m) {
        const int j = j0 + b + l;
        sq[lane] = R(q[j]);
        if (!MANY || !staged || (G == 1 && 32 * (who + team) < cnt)) {
          const R x = R((xs[j] - cx) * s), y = R((ys[j] - cy) * s), z = R((zs[j] - cz) * s);
          const R r2 = x * x + y * y + z * z;
          sz[lane] = z;
          sr2[lane] = r2;
          R sr = 1, si = 0;
          ss[lane] = sr;
          ss[32 + lane] = si;
#pragma unroll
          for (int k = 1; k <= P; ++k) {
            const R e = ce<R>(k - 1);
            const R nr = -e * (x * sr - y * si), ni = -e * (x * si + y * sr);
            sr = nr; si = ni;
            ss[64 * k + lane] = sr;
            ss[64 * k + 32 + lane] = si;
          }
          if constexpr (YK) {
            // the degree-n terms weighted by u_n(κ̂|x̂|), κ̂² = kh2[level] (harmonics_yukawa.jl:281-296)
            double u[P + 1];
            yukawa_u<P>(kh2[c.w] * (double)r2, u);
#pragma unroll
            for (int n = 0; n <= P; ++n) su[32 * n + lane] = (R)u[n];
          }
        }
      }
      __syncwarp();
      if (sub < G * SUB)
        for (int t = sub % SUB; t < cm; t += SUB) {
          const int i = sub / SUB * W + t;
          const R z = sz[i], r2 = sr2[i], tau = sq[i];
          R cr = ss[64 * h + i], ci = ss[64 * h + 32 + i], pr = 0, pi = 0;
          const R dr = ss[64 * (P - h) + i], di = ss[64 * (P - h) + 32 + i];
#pragma unroll
          for (int k = 0; k < K; ++k) {
            if (k > 0) {
              const R az = ab[2 * (k * H + h)] * z, br = ab[2 * (k * H + h) + 1] * r2;
              R nr = az * cr - br * pr, ni = az * ci - br * pi;
              pr = cr; pi = ci;
              if (k >= P - H + 2 && k == P - h + 1) { nr = dr; ni = di; pr = 0; pi = 0; }   // the second order starts
              cr = nr; ci = ni;
            }
            R tt = tau;
            if constexpr (YK) tt *= su[32 * (k <= P - h ? h + k : k - 1) + i];
            ar[k] += tt * cr;
            ai[k] -= tt * ci;
          }
        }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < K; ++k) {
      st[SUMS + 64 * k + lane] = ar[k];
      st[SUMS + 64 * k + 32 + lane] = ai[k];
    }
  };
  // outputs first, first + step, ... of set a and the node from the sums of nw warps, `n` subsets each, the first at r
  auto write = [&](auto subsets, int idx, int node, int a, const R* r, int nw, int first, int step) {
    constexpr int SUB = decltype(subsets)::value;
    double* col = sets.out[a] + (a < sets.nnode ? node * sets.pitch : idx * sets.ipitch);
    for (int o = first; o < 2 * K * H; o += step) {
      const int hh = o % H, kp = o / H, k = kp >> 1, part = kp & 1;
      const int m = k <= P - hh ? hh : P - hh, n = k <= P - hh ? hh + k : k - 1;
      if ((k > P - hh && P - hh == hh) || (part && m == 0)) continue;
      double v = 0;
      for (int w = 0; w < nw; ++w)
#pragma unroll
        for (int s = 0; s < SUB; ++s) v += (double)r[w * WS + SUMS + 32 * kp + s * H + hh];
      col[m == 0 ? n * n : n * n + 2 * m - 1 + part] = v;
    }
  };
  const int npc = npw ? P2M_WARPS * npw : 1, n0 = blockIdx.x * npc, a0 = MANY ? 0 : blockIdx.y, a1 = MANY ? sets.n : a0 + 1;
  // the warp's own nodes, lane i the i-th: those of at most 8 sources four at a time, of at most 16 two at a time
  // (each has its lanes and subsets whether or not the others are there), of at most P2M_ALONE alone
  const int mine = n0 + warp * npw, own = npw ? npw : warp == 0;
  const int nd = lane < own && mine + lane < nn ? nodes[mine + lane] : -1, cn = nd < 0 ? 0 : phi[nd] - plo[nd] + 1;
  auto packed = [&](auto pack, unsigned todo) {
    constexpr int G = decltype(pack)::value, W = 32 / G, SUB = NS / G;
    while (todo) {
      int at[G];                                                // the nodes of this turn (the first again where there are fewer)
      int n = 0;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        at[g] = todo ? __ffs(todo) - 1 : at[0];
        n += todo != 0;
        todo &= todo - 1;
      }
      int my = at[0], sum = at[0];
#pragma unroll
      for (int g = 1; g < G; ++g) {
        if (lane / W == g) my = at[g];
        if (sub / SUB == g) sum = at[g];
      }
      const int node = __shfl_sync(0xffffffffu, nd, my), ccnt = __shfl_sync(0xffffffffu, cn, sum);
#pragma unroll 1
      for (int a = a0; a < a1; ++a) {
        sums(pack, node, ccnt, 0, 1, a, a > a0);
        __syncwarp();
#pragma unroll
        for (int g = 0; g < G; ++g)
          if (g < n)
            write(std::integral_constant<int, SUB>(), mine + at[g], __shfl_sync(0xffffffffu, nd, at[g]), a, st + g * SUB * H, 1, lane, 32);
      }
    }
  };
  if constexpr (Sh::PACK) {
    packed(std::integral_constant<int, 4>(), __ballot_sync(0xffffffffu, cn > 0 && cn <= 8));
    packed(std::integral_constant<int, 2>(), __ballot_sync(0xffffffffu, cn > 8 && cn <= 16));
  }
  packed(std::integral_constant<int, 1>(), __ballot_sync(0xffffffffu, cn > (Sh::PACK ? 16 : 0) && cn <= P2M_ALONE));
  for (int i = 0; i < npc && n0 + i < nn; ++i) {
    const int node = nodes[n0 + i];
    if (phi[node] - plo[node] < P2M_ALONE) continue;            // uniform
#pragma unroll 1
    for (int a = a0; a < a1; ++a) {
      sums(std::integral_constant<int, 1>(), node, 0, warp, P2M_WARPS, a, a > a0);
      __syncthreads();
      write(std::integral_constant<int, NS>(), n0 + i, node, a, st0, P2M_WARPS, threadIdx.x, 32 * P2M_WARPS);
      __syncthreads();
    }
  }
}

// The multipoles of charges and dipoles from those of the charges and of the three components of the
// moments, taken as charges (src/operators/harmonics.jl:708-738): the derivative identities act on the
// sums, with the moments in box units d·s (harmonics.jl:436); A = (x, y, z) at degree n − 1:
//   M_n^m = Q_n^m + s·{cz(n, m) Z^m + ½cm(n, m)[−(Xr + Yi), Yr − Xi]^(m−1) + ½cp(n, m)[Xr − Yi, Yr + Xi]^(m+1)}
// (m = 0: cp(n, 0)(Xr − Yi)^1 in place of the last two). scr: X, Y, Z of the list's nodes i0 .. i0 + nn − 1,
// set-major, (P + 1)² apart; Q in place at M.
__global__ void k_p2m_dipoles(const int* __restrict__ nodes, int nn, int p, const int4* __restrict__ cell,
                              const double* __restrict__ scale, const double* __restrict__ scr, int64_t pitch,
                              double* __restrict__ M) {
  const int np = (p + 1) * (p + 1), e = blockIdx.x * blockDim.x + threadIdx.x, i = e / np, k = e % np;
  if (i >= nn || k == 0) return;
  const int node = nodes[i];
  const double s = scale[cell[node].w];
  int n = (int)sqrtf((float)k + 0.5f);
  while (n * n > k) --n;
  while ((n + 1) * (n + 1) <= k) ++n;
  const int r = k - n * n, m = (r + 1) >> 1, part = r == 0 ? 0 : 1 - (r & 1), n1 = n - 1;   // part 1: imaginary
  const double *X = scr + (int64_t)i * np, *Y = X + (int64_t)nn * np, *Z = Y + (int64_t)nn * np;
  auto at = [&](const double* A, int mm, int pt) {
    return mm == 0 ? (pt ? 0.0 : A[n1 * n1]) : A[n1 * n1 + 2 * mm - 1 + pt];
  };
  double v = 0;
  if (m <= n1) v = c_tab[2 * TRI_MAX + tri(n, m)] * at(Z, m, part);
  if (m >= 1) {
    const double cm = 0.5 * c_tab[3 * TRI_MAX + tri(n, m)];
    v += part ? cm * (at(Y, m - 1, 0) - at(X, m - 1, 1)) : -cm * (at(X, m - 1, 0) + at(Y, m - 1, 1));
    if (m + 1 <= n1) {
      const double cp = 0.5 * c_tab[4 * TRI_MAX + tri(n, m)];
      v += part ? cp * (at(Y, m + 1, 0) + at(X, m + 1, 1)) : cp * (at(X, m + 1, 0) - at(Y, m + 1, 1));
    }
  } else if (n1 >= 1) {
    v += c_tab[4 * TRI_MAX + tri(n, 0)] * (at(X, 1, 0) - at(Y, 1, 1));
  }
  M[(int64_t)node * pitch + k] += s * v;
}

// nodes [i0, i0 + nn) of the list: several per warp where there are CTAs enough for that (four per warp fill the
// device from about 128 nodes an SM on; two that share a warp, on average, from 24; one from four, or from 32 where
// nodes are large and the CTA's four would be taken one after the other by all its warps)
template <int P, bool YK, typename R, bool MANY>
void launch(State& S, int i0, int nn, const P2MSets& sets) {
  Plan& P_ = *S.plan;
  const int ny = MANY ? 1 : sets.n;
  const int64_t per_sm = (int64_t)nn * ny / P_.ctx->num_sms, avg = P_.N / P_.n_s2m;
  const bool pack = P2MShape<P, YK, R>::PACK;
  const int npw = pack && per_sm >= 128 ? 4 : (pack && avg <= 16 && per_sm >= 24 ? 2 : per_sm >= (avg <= 32 ? 4 : 32));
  const int npc = npw ? P2M_WARPS * npw : 1;
  auto kern = k_p2m<P, YK, R, MANY>;
  constexpr size_t smem = P2MShape<P, YK, R>::smem(MANY);
  FMMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<dim3((nn + npc - 1) / npc, ny), 32 * P2M_WARPS, smem, P_.ctx->stream>>>(
      P_.s2m_nodes.p + i0, nn, P_.cell.p, P_.plo.p, P_.phi.p, S.xs.p, S.ys.p, S.zs.p, sets, geometry(P_), P_.d_scale.p,
      P_.d_kh2.p, npw);
  FMMB_LAUNCH_CHECK();
}

template <int P>
void launch_kind(State& S, int i0, int nn, const P2MSets& sets, bool many) {
  const int kernel = S.plan->cache->kernel;
  // in FP32 on the mixed path of Laplace3D with charges (box-centred, scaled coordinates in [−½, ½]³,
  // written as doubles: about 2⁻²⁴ per coefficient, below the FP16x3 M2L's 2⁻²² that consumes them)
  if (kernel == FMMB_KERNEL_YUKAWA3D) launch<P, true, double, false>(S, i0, nn, sets);
  else if (S.precision == FMMB_PRECISION_MIXED && kernel == FMMB_KERNEL_LAPLACE3D && !S.has_dip)
    launch<P, false, float, false>(S, i0, nn, sets);
  else if (many) launch<P, false, double, true>(S, i0, nn, sets);
  else launch<P, false, double, false>(S, i0, nn, sets);
}

void run(State& S, int i0, int nn, const P2MSets& sets) {
  // (of a list that does not fill the SMs, a CTA per node and set: 30,000 points, the whole build, dipoles p = 12
  // in FP64 0.75 ms against 0.80 with all sets in one; 500,000 points p = 3 mixed 0.70 against 0.64. Above 32 sources
  // a node on average there is little to stage once: twelve Stokes spheres p = 16, the whole pass, 25.8 ms against 25.5)
  const bool many = sets.n > 1 && nn >= 32 * S.plan->ctx->num_sms && S.plan->N <= 32 * (int64_t)S.plan->n_s2m;
  switch (S.plan->cache->p) {
#define X(pp) case pp: launch_kind<pp>(S, i0, nn, sets, many); break;
    FMMB_P_CASES(X)
#undef X
    default: throw Error(FMMB_ERR_UNSUPPORTED, "p out of range");
  }
}

}  // namespace

// P2M of nsets ≤ 4 charge sets q[a] and, where d3[a] is given (3 × N planar), dipoles into the blocks
// at M[a] (pitch doubles per node); returns the launches
int p2m_blocks(State& S, int nsets, const double* const* q, const double* const* d3, double* const* M, int64_t pitch) {
  Plan& P = *S.plan;
  const int nn = P.n_s2m;
  if (nn == 0) return 0;
  P2MSets sets{};
  sets.pitch = pitch;
  sets.n = sets.nnode = nsets;
  for (int a = 0; a < nsets; ++a) { sets.q[a] = q[a]; sets.out[a] = M[a]; }
  if (!d3[0]) {
    run(S, 0, nn, sets);
    return 1;
  }
  // the moments' components as charges, into scratch of at most 128 MB, a range of nodes at a time
  const int64_t np = P.cache->np, N = P.N;
  const int chunk = (int)std::min<int64_t>(nn, std::max<int64_t>(1, (128ll << 20) / (8 * 3 * nsets * np)));
  DBuf<double> scr((size_t)3 * nsets * chunk * np);
  int launches = 0;
  sets.ipitch = np;
  sets.n = 4 * nsets;
  for (int i0 = 0; i0 < nn; i0 += chunk) {
    const int c = std::min(chunk, nn - i0);
    for (int a = 0; a < nsets; ++a)
      for (int k = 0; k < 3; ++k) {
        sets.q[nsets + 3 * a + k] = d3[a] + k * N;
        sets.out[nsets + 3 * a + k] = scr.p + (int64_t)(3 * a + k) * c * np;
      }
    run(S, i0, c, sets);
    for (int a = 0; a < nsets; ++a) {
      k_p2m_dipoles<<<(unsigned)((c * np + 255) / 256), 256, 0, P.ctx->stream>>>(
          P.s2m_nodes.p + i0, c, P.cache->p, P.cell.p, P.d_scale.p, scr.p + (int64_t)3 * a * c * np, pitch, M[a]);
      FMMB_LAUNCH_CHECK();
    }
    launches += 1 + nsets;
  }
  return launches;
}

}  // namespace fmmb
