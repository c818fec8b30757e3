// The near field's frame (eval.cu, stokes.cu): the sources of a leaf's colleagues (at most 27),
// flattened in colleague order into batches of 32, against the leaf's targets.
//
// A team of four warps takes a leaf, every fourth batch each: a warp stages its batch in shared
// memory while the next one's loads are in flight, and its lanes run over the targets, CH chunks of
// 32 at a time from the same staged batch. A chunk of 16 targets or fewer would leave half the lanes
// idle or more: its lanes split the batch's sources 2, 4 or 8 ways instead, and the parts are summed
// by shuffles at the end. (A leaf of a uniform cloud with ppl = 64 holds 30 points on average, and a
// third of them more than 32: the second chunk then costs an eighth to a half of the first instead of
// as much.) The warps' sums meet in shared memory in warp order. A leaf of at most NEAR_ALONE
// source-target pairs goes to one warp: a team's set-up and sums would cost more than its share.
// How the sums are split depends on the leaf's own targets and sources only, so a leaf's results are
// the same in every plan that holds it; the last bits of a target's sum depend on how many targets share its leaf. Groups per CTA (4 or 1) only place the work: 4 share the
// set-up's latency, 1 spreads few leaves over more SMs.
// The arithmetic pipe and the issue slots are each about 60 % busy (a million points), the rest is the latency of a
// pair's chain and the team's barriers. Measured, near field and L2P, a warp a leaf and no lane
// splits → this: a million points FP64 ppl = 64 p = 10 2.16 → 1.79 ms, in FP32 p = 4 0.79 → 0.74; 200,000 points FP64
// p = 4 0.70 → 0.45; a sphere of 30,000 FP64 ppl = 128 p = 16 (few full leaves) 0.68 → 0.21; 300,000 points of a Gaussian
// mixture in FP32 (many small leaves) 0.335 → 0.318. NEAR_ALONE: with teams from 256 sources on instead, the
// 400,000 FP64 points took 0.92, with every leaf alone the sphere's few leaves would leave SMs idle.
//
// A policy P gives: Args; Src (a source in registers), Stage (32 of them in shared memory); NA sums
// per target, CH chunks; REL (positions relative to the leaf's centre); load, stage, batch, write.
#pragma once
#include "passes.cuh"

namespace fmmb {
namespace {

constexpr int NEAR_TEAM = 4, NEAR_ALONE = 10000;

// the targets' groups (per leaf: node, first target, count), the targets in group order and their
// output indices, and the tree
struct NearArgs {
  const int *gnode, *gstart, *gcount;
  int ngroups;
  const double *tx, *ty, *tz;
  const int* tout;
  const int4* cell;
  const int *plo, *phi, *col;
  Geometry geo;
};

struct NearGroup {
  int lo[32];         // first point of each colleague (27 used)
  int pre[32];        // flat index of each colleague's first point (total for the unused slots)
  int S;              // sources
  int pself, loself, lenself;   // the leaf's own points among them: flat index, first point, count (pself −1: none)
  int t0, nt;
  double c[3];        // the leaf's centre (REL)
};

template <bool REL>
__device__ __forceinline__ void near_setup(const NearArgs& A, int g, int lane, NearGroup& G) {
  const int leaf = A.gnode[g];
  const int cn = lane < NCOL ? A.col[(int64_t)leaf * NCOL + lane] : -1;
  int lo = 0, len = 0;
  if (cn >= 0) {
    lo = A.plo[cn];
    len = max(0, A.phi[cn] - lo + 1);
  }
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  G.lo[lane] = lo;
  G.pre[lane] = incl - len;
  const unsigned selfm = __ballot_sync(0xffffffffu, cn == leaf);
  const int slot = selfm ? __ffs(selfm) - 1 : 0;
  if (lane == 31) G.S = incl;
  if (lane == slot) {
    G.pself = selfm ? incl - len : -1;
    G.loself = lo;
    G.lenself = selfm ? len : 0;
  }
  if (lane == 0) {
    G.t0 = A.gstart[g];
    G.nt = A.gcount[g];
    G.c[0] = G.c[1] = G.c[2] = 0.0;
    if (REL) {
      const int4 c = A.cell[leaf];
      const Geometry gn = A.geo.at(leaf);
      const double w = ldexp(A.geo.W0, -c.w);
      G.c[0] = gn.center(0, c.x, w);
      G.c[1] = gn.center(1, c.y, w);
      G.c[2] = gn.center(2, c.z, w);
    }
  }
}

// the tree index of flat source f < S of the group
__device__ __forceinline__ int near_source(const NearGroup& G, int f) {
  int idx = 0;   // the last colleague whose flat start is ≤ f
#pragma unroll
  for (int step = 16; step; step >>= 1)
    if (G.pre[idx + step] <= f) idx += step;
  return G.lo[idx] + (f - G.pre[idx]);
}

__device__ __forceinline__ bool near_alone(const NearGroup& G) { return (int64_t)G.S * G.nt <= NEAR_ALONE; }

// log2 of the ways to split a batch over the lanes of a chunk of n targets
__device__ __forceinline__ int near_split(int n) { return n > 16 ? 0 : (n > 8 ? 1 : (n > 4 ? 2 : 3)); }

// one group by `team` warps (this one's rank in it: who); red: 3 × 32·CH × NA sums of a team
template <class P, bool SELF>
__device__ __forceinline__ void near_group(const NearArgs& A, const typename P::Args& pa, const NearGroup& G, int team,
                                           int who, int lane, typename P::Stage* stg, double* red) {
  constexpr int CH = P::CH, NA = P::NA;
  using R = typename P::Real;
  const double cx = G.c[0], cy = G.c[1], cz = G.c[2];
  const int S = G.S;
  for (int base = 0; base < G.nt; base += 32 * CH) {
    int n[CH], lf[CH], fself[CH];
    R t[CH][3];
    double acc[CH][NA];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      n[c] = min(32, G.nt - base - 32 * c);
      lf[c] = near_split(n[c]);
      const int q = lane & ((32 >> lf[c]) - 1);
      const bool act = q < n[c];
      const int k = G.t0 + base + 32 * c + q;
      t[c][0] = (R)((act ? A.tx[k] : cx) - cx);
      t[c][1] = (R)((act ? A.ty[k] : cy) - cy);
      t[c][2] = (R)((act ? A.tz[k] : cz) - cz);
      fself[c] = SELF && act && G.pself >= 0 ? G.pself + (k - G.loself) : -1;
#pragma unroll
      for (int i = 0; i < NA; ++i) acc[c][i] = 0.0;
    }
    typename P::Src nxt;
    auto load = [&](int b) {
      nxt = typename P::Src{};
      if (32 * b + lane < S) P::load(pa, near_source(G, 32 * b + lane), nxt);
    };
    if (32 * who < S) load(who);
    int buf = 0;
    for (int b = who; 32 * b < S; b += team, buf ^= 1) {
      P::stage(stg[buf], lane, nxt, cx, cy, cz);
      __syncwarp();
      if (32 * (b + team) < S) load(b + team);
      const int m = min(32, S - 32 * b);
      const bool chk = SELF && G.pself >= 0 && 32 * b < G.pself + G.lenself && 32 * b + 32 > G.pself;   // uniform
#pragma unroll
      for (int c = 0; c < CH; ++c)
        if (n[c] > 0) {                                  // uniform
          const int part = lane >> (5 - lf[c]);
          if (chk) P::template batch<true>(pa, stg[buf], m, fself[c] - 32 * b, part, 1 << lf[c], t[c], acc[c]);
          else P::template batch<false>(pa, stg[buf], m, 0, part, 1 << lf[c], t[c], acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < CH; ++c)
      for (int o = 32 >> lf[c]; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < NA; ++i) acc[c][i] += __shfl_xor_sync(0xffffffffu, acc[c][i], o);
    if (team > 1) {
      if (who > 0)
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
          for (int i = 0; i < NA; ++i) red[(((who - 1) * CH + c) * NA + i) * 32 + lane] = acc[c][i];
      __syncthreads();
      if (who == 0)
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
          for (int i = 0; i < NA; ++i)
#pragma unroll
            for (int w = 0; w < NEAR_TEAM - 1; ++w) acc[c][i] += red[((w * CH + c) * NA + i) * 32 + lane];
    }
    if (who == 0)
#pragma unroll
      for (int c = 0; c < CH; ++c)
        if (lane < n[c]) P::write(pa, A.tout[G.t0 + base + 32 * c + lane], acc[c]);
    if (team > 1) __syncthreads();                       // the sums and the staging are read
    else __syncwarp();
  }
}

template <class P, bool SELF>
__global__ void __launch_bounds__(32 * NEAR_TEAM, P::MINB) k_near(const NearArgs A, const typename P::Args pa, int gpc) {
  __shared__ NearGroup grp[NEAR_TEAM];
  __shared__ typename P::Stage stg[NEAR_TEAM][2];
  __shared__ double red[(NEAR_TEAM - 1) * P::CH * P::NA * 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g0 = blockIdx.x * gpc;
  const bool mine = warp < gpc && g0 + warp < A.ngroups;
  if (mine) near_setup<P::REL>(A, g0 + warp, lane, grp[warp]);
  __syncthreads();
  // first each warp's own leaf where it takes one alone, then the others by the whole team (one call, so
  // that the loops are in the code once)
#pragma unroll 1
  for (int i = 0; i <= gpc; ++i) {
    const int g = i == 0 ? warp : i - 1;
    if (i == 0 ? !mine : g0 + g >= A.ngroups) continue;
    if (near_alone(grp[g]) != (i == 0)) continue;          // uniform over the team where i > 0
    near_group<P, SELF>(A, pa, grp[g], i == 0 ? 1 : NEAR_TEAM, i == 0 ? 0 : warp, lane, stg[warp], red);
  }
}

// 4 groups per CTA where there are CTAs enough for every SM's warps, else 1
template <class P, bool SELF>
void launch_near_leaves(const NearArgs& A, const typename P::Args& pa, int num_sms, cudaStream_t s) {
  const int gpc = A.ngroups >= 32 * num_sms ? NEAR_TEAM : 1;
  k_near<P, SELF><<<(A.ngroups + gpc - 1) / gpc, 32 * NEAR_TEAM, 0, s>>>(A, pa, gpc);
  FMMB_LAUNCH_CHECK();
}

}  // namespace
}  // namespace fmmb
