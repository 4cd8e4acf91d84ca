// Launchers of the step kernels (lulesh_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include "lulesh_internal.h"

namespace lulesh {

// Element kernels are compiled for blocks of up to kMaxElemBlock threads and
// the node kernel for up to kMaxNodeBlock (the register budget is the same
// 255 per thread either way), so the block size is a launch-time choice.
constexpr int kMaxElemBlock = 256;
constexpr int kMaxNodeBlock = 512;
// Elements per block of the kernels that run one thread per element and
// coordinate: a warp for each coordinate.
constexpr int kFixedElems = 32;

constexpr int kNodeBlock = 256, kMatBlock = 128;

// Launch configuration chosen by the caller or the autotuner (defaults are the block
// sizes that measured best for the 150^3 problem). `force`, `kin` and `geo` are the
// caller's values of lulesh_tuning, kept for lulesh_get_tuning: k_force and
// k_kinematics run blocks of 3 * kFixedElems threads, and the force geometry is
// formed in k_force whatever `geo` says.
struct Tuning {
  int force = 128;
  int node = kNodeBlock;
  int kin = 128;
  int mat = kMatBlock;
  int geo = 0;
};

// Whether two configurations launch the same kernels.
inline bool same_launches(const Tuning& a, const Tuning& b) { return a.node == b.node && a.mat == b.mat; }

// Threads per block of a kernel with one thread per unit. A block size the caller
// set is used as it is; the default is halved, down to a warp, until there are
// eight blocks per SM. A small mesh then spreads over the SMs evenly: 41.2 -> 39.9 us
// per cycle at 30^3, nothing from 64^3 up.
inline int threads_per_block(int units, int block, int by_default) {
  constexpr int kSMs = 152;
  if (block == by_default)
    while (block > 32 && (units + block - 1) / block < 8 * kSMs) block /= 2;
  return block;
}

// The first taped cycle's face diagonals and normals.
void launch_tape_geometry(const DevDomain& d, cudaStream_t s);
// with time: the cycle's time step too, in place of launch_time_increment (not
// while taping)
void launch_force(const DevDomain& d, const Params& prm, cudaStream_t s, bool time = false);
void launch_node(const DevDomain& d, const Params& prm, bool aux, const Tuning& t, cudaStream_t s);
void launch_kinematics(const DevDomain& d, const Params& prm, bool aux, cudaStream_t s);
void launch_material(const DevDomain& d, const Params& prm, bool aux, const Tuning& t, cudaStream_t s);
void launch_time_increment(DevState* st, int n, const Params& prm, cudaStream_t s);
// One problem's step state to the device, and to pinned host memory.
void launch_put_state(DevState* st, const DevState& value, cudaStream_t s);
void launch_get_state(const DevState* st, DevState* pinned, cudaStream_t s);

// Picks block sizes for the four step kernels by timing them on the live
// problem (lulesh_tune.cu); the state advances, so callers save and restore it.
cudaError_t autotune_blocks(const DevDomain& d, const Params& prm, bool aux, int ninst, cudaStream_t s,
                            int cycles, Tuning& t);

}  // namespace lulesh
