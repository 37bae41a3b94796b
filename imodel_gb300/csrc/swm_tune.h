// The autotuner's search over the launch configurations of the FP32 stage
// (internal header): what is timed, in which order, and what is kept.
#pragma once
#include "swm_common.cuh"

namespace imodel {

// What the handle can run: the stencil variant, the cell-centred ones; whether
// variant 1 is the fused stage, which takes no block sizes; whether the
// learned-correction kernel is in the step.
struct TuneSpace {
  bool stencil = true, cells = true, fused = false, network = false;
};

// trial(Tune) returns a step's time, 1e30 where it cannot be had.  Each
// configuration is timed once, and only those whose kernels differ: variants 1
// and 2 launch the same separate kernels unless variant 1 is fused, and block
// sizes mean nothing to the fused stage.  Where it is the fastest, the sizes kept
// beside it are the separate kernels' best, which run once an option is
// switched on.
template <class Trial>
Tune search_tune(const TuneSpace &S, Trial trial) {
  constexpr int kSizes[3] = {128, 256, 512};
  struct Best {
    Tune t;
    float ms = 1e30f;
  };
  auto take = [&](Best &b, const Tune &t) {
    const float ms = trial(t);
    if (ms < b.ms) b = {t, ms};
  };
  auto sweep = [&](int variant) {
    Best b;
    b.t.variant = variant;
    for (int n : kSizes) {
      Tune t;
      t.variant = variant;
      t.bs_tri = t.bs_pre = t.bs_cell = t.bs_edge = n;
      take(b, t);
    }
    return b;
  };
  // the block size of each kernel with the others fixed
  auto refine = [&](Best &b) {
    int Tune::*fields[4] = {&Tune::bs_tri, &Tune::bs_pre, &Tune::bs_cell, &Tune::bs_edge};
    for (int f = 0; f < 4; ++f) {
      if (f == 1 && b.t.variant >= 1) continue;
      const int timed = b.t.*fields[f];
      for (int n : kSizes) {
        if (n == timed) continue;
        Tune t = b.t;
        t.*fields[f] = n;
        take(b, t);
      }
    }
  };
  Best stencil, cells, fused;
  if (S.stencil) stencil = sweep(0);
  if (S.cells) cells = sweep(S.fused ? 2 : 1);
  if (S.cells && S.fused) take(fused, Tune());
  Best best;
  if (!S.cells || (stencil.ms < cells.ms && stencil.ms < fused.ms)) {
    best = stencil;
    refine(best);
  } else if (S.fused && fused.ms <= cells.ms) {
    best = cells;
    refine(best);
    best = {best.t, fused.ms};
    best.t.variant = 1;
  } else {
    best = cells;
    refine(best);
  }
  // the learned-correction kernel's split of warps between gathering and the
  // epilogue
  if (S.network)
    for (int g = 2; g <= 4; ++g) {
      if (best.t.mlp_gather == g) continue;
      Tune t = best.t;
      t.mlp_gather = g;
      take(best, t);
    }
  return best.t;
}

}  // namespace imodel
