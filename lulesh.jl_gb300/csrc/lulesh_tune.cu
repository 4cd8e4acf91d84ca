// Autotuner shared by the single-problem handle and the ensemble: block
// sizes of the step kernels that run one thread per node or element (k_node,
// k_material; the other two run three per element in blocks of 96).
//
// Coordinate descent: for each of them in turn, every candidate block
// size runs `cycles` full cycles on the live problem with CUDA events around
// each kernel; the fastest candidate for that kernel is kept before the next
// kernel is tuned. Every choice gives bitwise the same results. The caller
// saves and restores the state.
#include <climits>

#include "lulesh_kernels.h"

namespace lulesh {

namespace {
void launch_phase(int q, const DevDomain& d, const Params& prm, bool aux, const Tuning& t, cudaStream_t s) {
  switch (q) {
    case 0: launch_force(d, prm, s); break;
    case 1: launch_node(d, prm, aux, t, s); break;
    case 2: launch_kinematics(d, prm, aux, s); break;
    default: launch_material(d, prm, aux, t, s); break;
  }
}

// Runs 1 + cycles full cycles with tuning t (the first warms up) and adds each
// step kernel's time over the timed cycles to ms[0..3].
cudaError_t phase_times(const DevDomain& d, const Params& prm, bool aux, int ninst, cudaStream_t s, int cycles,
                        const Tuning& t, cudaEvent_t* ev, float ms[4]) {
  for (int q = 0; q < 4; ++q) ms[q] = 0.f;
  cudaError_t err = cudaSuccess;
  for (int c = 0; c <= cycles && err == cudaSuccess; ++c) {
    launch_time_increment(d.st, ninst, prm, s);
    for (int q = 0; q < 4; ++q) {
      cudaEventRecord(ev[q], s);
      launch_phase(q, d, prm, aux, t, s);
    }
    cudaEventRecord(ev[4], s);
    err = cudaEventSynchronize(ev[4]);
    if (err == cudaSuccess && c > 0) {
      for (int q = 0; q < 4; ++q) {
        float x = 0.f;
        cudaEventElapsedTime(&x, ev[q], ev[q + 1]);
        ms[q] += x;
      }
    }
  }
  return err;
}

// Coordinate descent over the block sizes.
cudaError_t descend(const DevDomain& d, const Params& prm, bool aux, int ninst, cudaStream_t s, int cycles, Tuning& t,
                    cudaEvent_t* ev) {
  static const int elem_cand[3] = {64, 128, 256};
  static const int node_cand[3] = {128, 256, 512};
  cudaError_t err = cudaSuccess;
  for (int k = 1; k < 4 && err == cudaSuccess; k += 2) {
    int* slot = k == 1 ? &t.node : &t.mat;
    const int* cand = (k == 1) ? node_cand : elem_cand;
    float best = 3.0e38f;
    int best_bs = *slot;
    for (int j = 0; j < 3 && err == cudaSuccess; ++j) {
      *slot = cand[j];
      float ms[4];
      err = phase_times(d, prm, aux, ninst, s, cycles, t, ev, ms);
      if (err == cudaSuccess && ms[k] < best) {
        best = ms[k];
        best_bs = cand[j];
      }
    }
    *slot = best_bs;
  }
  return err;
}
}  // namespace

cudaError_t autotune_blocks(const DevDomain& d, const Params& prm, bool aux, int ninst, cudaStream_t s,
                            int cycles, Tuning& t) {
  cudaEvent_t ev[5] = {};
  cudaError_t err = cudaSuccess;
  for (int i = 0; i < 5 && err == cudaSuccess; ++i) err = cudaEventCreate(&ev[i]);
  if (cycles < 1) cycles = 1;
  if (err == cudaSuccess) err = descend(d, prm, aux, ninst, s, cycles, t, ev);
  for (int i = 0; i < 5; ++i)
    if (ev[i]) cudaEventDestroy(ev[i]);
  if (err == cudaSuccess) err = cudaGetLastError();
  return err;
}

}  // namespace lulesh
