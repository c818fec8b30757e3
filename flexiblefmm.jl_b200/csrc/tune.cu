// The autotuner of the launch shapes: tile and block shapes chosen by timing them on the
// caller's own inputs (the reference has no tuner).
//
// One shape is free, in that no result depends on it (each target's sums are taken in the list's
// order whatever the blocking):
//   - the targets per M2L block (32, 64 or 128; a plan property: its blocks are re-cut from the
//     pairs per target), for both M2L kernels.
// fmmb_autotune times each candidate on the state's own inputs (CUDA events on the context's
// stream, the median of three after one warm-up), keeps the fastest, applies it, and records it
// for every later plan of the same kind: method, kernel, order and the number of points rounded down
// to a power of two. Plans created afterwards take the recorded
// block size.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "passes.cuh"

namespace fmmb {
namespace {

struct Tuned {
  int tb = 0;
};
using Kind = std::tuple<int, int, int, int>;   // method, kernel, p, log2 N

std::mutex g_mu;
std::map<Kind, Tuned> g_tuned;

int log2_floor(int64_t n) {
  int b = 0;
  while ((int64_t)1 << (b + 1) <= n) ++b;
  return b;
}

Kind kind_of(const Plan& P) {
  const Cache& C = *P.cache;
  return Kind(C.method, C.kernel, C.p, log2_floor(P.N));
}

// the median of three timed runs after one warm-up, in ms
template <class F>
double time_ms(cudaStream_t s, F&& f) {
  cudaEvent_t e0, e1;
  FMMB_CUDA(cudaEventCreate(&e0));
  FMMB_CUDA(cudaEventCreate(&e1));
  f();
  double t[3];
  for (double& x : t) {
    FMMB_CUDA(cudaEventRecord(e0, s));
    f();
    FMMB_CUDA(cudaEventRecord(e1, s));
    FMMB_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    FMMB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    x = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  std::sort(t, t + 3);
  return t[1];
}

}  // namespace

int tuned_block_size(const Plan& P) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_tuned.find(kind_of(P));
  return it == g_tuned.end() ? 0 : it->second.tb;
}

void autotune(State& S, const double* xyz, const double* tau, bool tune_blocks, double* out) {
  Plan& P = *S.plan;
  Cache& C = *P.cache;
  require(C.method == FMMB_METHOD_SPHERICAL_HARMONICS, FMMB_ERR_UNSUPPORTED, "the tuner takes the harmonic methods");
  cudaStream_t s = P.ctx->stream;
  // the multipoles of these inputs, which every M2L candidate reads (Stokeslet3D: Stokeslets)
  if (C.kernel == FMMB_KERNEL_STOKESLET3D) {
    StokesDensities d;
    d.stokeslets = tau;
    stokes_build(S, xyz, d);
  } else {
    gather_inputs(S, xyz, tau);
    upward_pass(S);
  }
  // the M2L's block sizes
  std::vector<int> tbs = {P.TB};
  if (tune_blocks) tbs = {32, 64, 128};
  double best = 1e300;
  int best_tb = P.TB;
  for (int tb : tbs) {
    if (tb != P.TB) build_blocks(P, tb);
    const double ms = time_ms(s, [&] { m2l_stage(S); });
    if (ms < best) { best = ms; best_tb = tb; }
  }
  if (P.TB != best_tb) build_blocks(P, best_tb);
  // the near field at the sources (harmonic methods with charges: Laplace3D and Yukawa3D), for the
  // caller: it has no shape to choose
  double near_ms = 0;
  if (C.kernel != FMMB_KERNEL_STOKESLET3D && P.n_leaves > 0) {
    DBuf<double> pot(P.N), grad(3 * P.N);
    near_ms = time_ms(s, [&] { near_sources(S, FMMB_OUTPUT_POTENTIAL | FMMB_OUTPUT_GRADIENT, pot.p, grad.p, s); });
    FMMB_CUDA(cudaStreamSynchronize(s));
  }
  S.built = false;                      // the timed stages left the expansions incomplete
  {
    std::lock_guard<std::mutex> lk(g_mu);
    Tuned t;
    t.tb = best_tb;
    if (tune_blocks) g_tuned[kind_of(P)] = t;
  }
  if (out) {
    out[0] = best_tb;
    out[1] = 0;                          // the FP64 M2L has one chunk width
    out[2] = 4;                          // warps of a near-field team
    out[3] = best;
    out[4] = near_ms;
  }
}

}  // namespace fmmb
