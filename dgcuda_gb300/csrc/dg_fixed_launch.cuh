// dg_fixed_launch.cuh -- launchers of the fixed-point element stage and
// traces (dg_fixed.cuh), p = 1..4; each equation is instantiated in a
// translation unit of its own (dg_fixed_<equation>.cu).
#pragma once
#include "dg_fixed.cuh"

namespace dg {
namespace fx {

template <class Eq, int P>
void run_element(const Ctx &c, const ElemArgs &a, int mode) {
  using S = Shape<Eq, P>;
  const FxTab<P> &tab = *static_cast<const FxTab<P> *>(c.fx);
  const unsigned blocks = nblk(c.m.K, kTile);
  if (mode == 0) {
    launch(k_element_fx<Eq, P, 0>, blocks, S::kThreads, c.st, tab, *c.q, a);
  } else if (mode == 1) {
    launch(k_element_fx<Eq, P, 1>, blocks, S::kThreads, c.st, tab, *c.q, a);
  } else if (mode == 3) {
    launch(k_element_fx<Eq, P, 3>, blocks, S::kThreads, c.st, tab, *c.q, a);
  } else {
    if constexpr (Eq::kFusedLimiter)
      launch(k_element_fx<Eq, P, 2>, blocks, S::kThreads, c.st, tab, *c.q, a);
  }
}

// what: 0 the traces, 1 limited and traced, 2 limited only
template <class Eq, int P>
void run_trace(const Ctx &c, double *u, int what) {
  const FxTab<P> &tab = *static_cast<const FxTab<P> *>(c.fx);
  const unsigned blocks = nblk(c.m.K, kTile);
  constexpr int T = Shape<Eq, P>::kThreads;
  if (what == 0)
    launch(k_trace_fx<Eq, P, false, true>, blocks, T, c.st, tab, *c.q, u, c.T, c.m.nbr, c.m.K,
           c.m.Kp);
  else if (what == 1)
    launch(k_trace_fx<Eq, P, true, true>, blocks, T, c.st, tab, *c.q, u, c.T, c.m.nbr, c.m.K,
           c.m.Kp);
  else
    launch(k_trace_fx<Eq, P, true, false>, blocks, T, c.st, tab, *c.q, u, c.T, c.m.nbr, c.m.K,
           c.m.Kp);
}

template <class Eq>
void element(const Ctx &c, const ElemArgs &a, int mode) {
  switch (c.p) {
    case 1: run_element<Eq, 1>(c, a, mode); break;
    case 2: run_element<Eq, 2>(c, a, mode); break;
    case 3: run_element<Eq, 3>(c, a, mode); break;
    case 4: run_element<Eq, 4>(c, a, mode); break;
  }
}

template <class Eq>
void trace(const Ctx &c, double *u, int what) {
  switch (c.p) {
    case 1: run_trace<Eq, 1>(c, u, what); break;
    case 2: run_trace<Eq, 2>(c, u, what); break;
    case 3: run_trace<Eq, 3>(c, u, what); break;
    case 4: run_trace<Eq, 4>(c, u, what); break;
  }
}

// the element stage, and with stage < 0 the start-of-run traces, of n blocks of
// blk elements from block lo of a batch's map, all of order p
template <class Eq, int P>
void run_batch(const BatchLaunch &b, cudaStream_t st, int lo, int n, int blk, int stage,
               int check) {
  using S = Shape<Eq, P>;
  const FxTab<P> &tab = *static_cast<const FxTab<P> *>(b.fx[P]);
  const int sub = blk / kTile;
  if (stage < 0)
    k_trace_batch_fx<Eq, P, false><<<n * sub, S::kThreads, 0, st>>>(
        tab, b.probs, b.eblk2prob, b.eblk0, lo, sub, 0);
  else
    k_element_batch_fx<Eq, P><<<n * sub, S::kThreads, 0, st>>>(tab, b.probs, b.eblk2prob, b.eblk0,
                                                               lo, sub, stage, check);
}

template <class Eq>
void batch_element(const BatchLaunch &b, cudaStream_t st, int p, int lo, int n, int blk,
                   int stage, int check) {
  if (p == 1) run_batch<Eq, 1>(b, st, lo, n, blk, stage, check);
  if (p == 2) run_batch<Eq, 2>(b, st, lo, n, blk, stage, check);
  if (p == 3) run_batch<Eq, 3>(b, st, lo, n, blk, stage, check);
}

// the limiter of a stage's output and its traces, of the same blocks
template <class Eq, int P>
void run_batch_limit(const BatchLaunch &b, int lo, int n, int blk, int stage) {
  const int sub = blk / kTile;
  k_trace_batch_fx<Eq, P, true><<<n * sub, Shape<Eq, P>::kThreads, 0, b.st>>>(
      *static_cast<const FxTab<P> *>(b.fx[P]), b.probs, b.eblk2prob, b.eblk0, lo, sub, stage);
}

template <class Eq>
void batch_limit(const BatchLaunch &b, int p, int lo, int n, int blk, int stage) {
  if (p == 1) run_batch_limit<Eq, 1>(b, lo, n, blk, stage);
  if (p == 2) run_batch_limit<Eq, 2>(b, lo, n, blk, stage);
  if (p == 3) run_batch_limit<Eq, 3>(b, lo, n, blk, stage);
}

}  // namespace fx
}  // namespace dg
