// Nodal forces without any device allocation.
//
// Who needs this: callers that keep the Domain's arrays in device memory they
// manage themselves and must not have a library allocate behind their back,
// for example a Julia program whose CuArrays come from its own memory pool,
// or a host application that budgets every byte of device memory up front.
// Such callers pass device pointers to their own inputs and outputs; the
// per-corner force scratch this computation needs lives in a fixed array
// compiled into the library (g_corner_scratch below), so nothing here calls
// cudaMalloc, cudaFree or any allocating routine.
//
// Costs and limits:
//  * the array holds kStaticMaxElems elements' corner forces (6 MiB plus a
//    status word); CUDA loads the library's device code lazily, so a device
//    commits the array at the first call made there and keeps it until the
//    process exits;
//  * all calls share it: two calls that overlap on the GPU (different
//    streams, or different host threads) race on it and give wrong forces;
//  * the first call on a device looks up the array's device address (once
//    per device); make that first call before any stream capture.
#include <cuda_runtime.h>

#include <mutex>

#include "../../include/lulesh_gb300.h"
#include "lulesh_device.cuh"
#include "lulesh_element_fp64.cuh"
#include "lulesh_fixed_force.cuh"
#include "lulesh_kernels.h"

namespace lulesh {
namespace {

constexpr int64_t kStaticMaxElems = LULESH_STATIC_MAX_ELEMS;

// [0, 24*max): corner forces, component-major, then corner-major
// (x: [0, 8*max), y: [8*max, 16*max), z: [16*max, 24*max)), index c*max + e, so
// that a warp's elements store side by side; [24*max]: status bits of the call
// in progress, [24*max + 1]: of the last finished one.
static __device__ __align__(256) double g_corner_scratch[24 * kStaticMaxElems + 32];

constexpr int kMaxDevices = 64;
void* g_scratch_addr[kMaxDevices] = {};
std::mutex g_scratch_mutex;

// Address of g_corner_scratch on the current device (looked up once).
int scratch_address(double** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return LULESH_ERR_CUDA;
  if (dev < 0 || dev >= kMaxDevices) return LULESH_ERR_ARGUMENT;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_corner_scratch) != cudaSuccess || !p) return LULESH_ERR_CUDA;
    g_scratch_addr[dev] = p;
  }
  *out = static_cast<double*>(g_scratch_addr[dev]);
  return LULESH_OK;
}

// Corner forces of 32 elements per block, three threads each: the step's
// k_force on the caller's arrays. At most 1,024 blocks, so what bounds it is
// one block's latency: the whole call at 27^3 takes 45 us, 84 with one thread
// per element in FP64, corner forces stored element-major and a memset of the
// status word.
struct NoTape {
  static constexpr bool on = false;
  __device__ void derivative(int, int, double) const {}
  __device__ void mode(int, int, double) const {}
  __device__ void sum(int, int, double) const {}
};

template <int MODE>
__global__ void __launch_bounds__(3 * kFixedElems) k_static_corner_forces(lulesh_force_args a, double* scratch,
                                                                          int64_t max_elems) {
  __shared__ fx::Num column[fx::FS_COUNT * kFixedElems];
  const int64_t E = a.num_elem;
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  const int64_t slot = (int64_t)blockIdx.x * kFixedElems + lane;
  const int64_t e = slot < E ? slot : E - 1;
  const bool live = slot < E;
  unsigned* const status = reinterpret_cast<unsigned*>(scratch + 24 * max_elems);
  const double* const X = k == 0 ? a.x : k == 1 ? a.y : a.z;
  const double* const U = k == 0 ? a.xd : k == 1 ? a.yd : a.zd;
  const fx::Slots sh{column + lane, kFixedElems};
  fx::ForceLane r;
  double v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int64_t nd = a.nodelist[8 * e + c];
    r.x[c] = X[nd];
    v[c] = U[nd];
  }
  ForceScalars c = {};
  if (k == 0) {
    c.v = a.v[e];
    const double rc = inv_cbrt(a.volo[e] * c.v);
    c.vi12 = (rc * rc) * (rc * (1.0 / 12.0));
    c.coef = a.hgcoef > 0.0 ? ((-a.hgcoef * 0.01) * a.ss[e]) * a.elemMass[e] * rc : 0.0;
    fx::force_scales(sh, gt_zero(c.v) ? c.vi12 : 0.0, c.coef);
  } else if (k == 1) {
    fx::force_stress(sh, ((-a.p[e]) - a.q[e]) * 0.125);
  }
  fx::force_load(k, sh, v, r);
  long long hm[4];
  __syncthreads();
  fx::force_diagonals(k, sh, r, hm, fx::wide());
  __syncthreads();
  fx::force_products<MODE>(k, sh, r, hm, NoTape{}, fx::wide());
  __syncthreads();
  fx::force_base(k, sh, r);
  const int others = __syncthreads_or(live && !r.ok);
  double* const out = scratch + 8 * k * max_elems + e;
  auto store = [&](int n, double f) { out[n * max_elems] = f; };
  if (live && r.ok) fx::force_corners(k, sh, r, store, NoTape{});
  if (others) {
    __syncthreads();
    c.v = a.v[e];
    const double rc = inv_cbrt(a.volo[e] * c.v);
    c.vi12 = (rc * rc) * (rc * (1.0 / 12.0));
    c.coef = ((-a.hgcoef * 0.01) * a.ss[e]) * a.elemMass[e] * rc;
    c.s8 = ((-a.p[e]) - a.q[e]) * 0.125;
    c.hourglass = a.hgcoef > 0.0;
    force_fp64<MODE>(k, RealSlots{reinterpret_cast<double*>(column) + lane, kFixedElems}, r.x, v, c, live && !r.ok,
                     status, store, NoTape{});
  }
}

// fx = sum of the node's corner forces in nodeElemCornerList order
// (src/domain.jl:1112-1127).
// It also hands the status word over and clears it for the next call (a call whose
// gather is not launched clears it itself).
__global__ void __launch_bounds__(256) k_static_gather(lulesh_force_args a, double* scratch, int64_t max_elems) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n == 0) {
    unsigned* const status = reinterpret_cast<unsigned*>(scratch + 24 * max_elems);
    status[2] = status[0];
    status[0] = 0u;
  }
  if (n >= a.num_node) return;
  const int64_t s = a.nodeElemStart[n], cnt = a.nodeElemCount[n];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  for (int64_t i = 0; i < cnt; ++i) {
    const int64_t corner = a.nodeElemCornerList[s + i] - 1;  // 8*e + c
    const int64_t k = (corner & 7) * max_elems + (corner >> 3);
    if (i == 0) {
      fx = scratch[k]; fy = scratch[8 * max_elems + k]; fz = scratch[16 * max_elems + k];
    } else {
      fx += scratch[k]; fy += scratch[8 * max_elems + k]; fz += scratch[16 * max_elems + k];
    }
  }
  a.fx[n] = fx;
  a.fy[n] = fy;
  a.fz[n] = fz;
}

}  // namespace
}  // namespace lulesh

extern "C" int lulesh_calc_force_for_nodes_static(const lulesh_force_args* args, void* stream,
                                                  int32_t* site) {
  using namespace lulesh;
  if (site) *site = LULESH_SITE_NONE;
  if (!args) return LULESH_ERR_ARGUMENT;
  const lulesh_force_args& a = *args;
  if (a.num_elem < 1 || a.num_node < 1 || a.mode < 0 || a.mode > 7 || !a.nodelist || !a.nodeElemStart ||
      !a.nodeElemCount || !a.nodeElemCornerList || !a.x || !a.y || !a.z || !a.xd || !a.yd || !a.zd ||
      !a.p || !a.q || !a.ss || !a.v || !a.volo || !a.elemMass || !a.fx || !a.fy || !a.fz)
    return LULESH_ERR_ARGUMENT;
  if (a.num_elem > kStaticMaxElems) return LULESH_ERR_ARGUMENT;  // beyond the fixed scratch
  double* scratch = nullptr;
  int rc = scratch_address(&scratch);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const unsigned* status = reinterpret_cast<const unsigned*>(scratch + 24 * kStaticMaxElems) + 2;
  const int eg = (int)((a.num_elem + kFixedElems - 1) / kFixedElems), bs = 3 * kFixedElems;
  switch (a.mode & 3) {
    case 0: k_static_corner_forces<0><<<eg, bs, 0, s>>>(a, scratch, kStaticMaxElems); break;
    case 1: k_static_corner_forces<1><<<eg, bs, 0, s>>>(a, scratch, kStaticMaxElems); break;
    case 2: k_static_corner_forces<2><<<eg, bs, 0, s>>>(a, scratch, kStaticMaxElems); break;
    default: k_static_corner_forces<3><<<eg, bs, 0, s>>>(a, scratch, kStaticMaxElems); break;
  }
  k_static_gather<<<(int)((a.num_node + 255) / 256), 256, 0, s>>>(a, scratch, kStaticMaxElems);
  if (cudaGetLastError() != cudaSuccess) {
    // one of the two was not launched: what the first may have found is no
    // one's to report
    cudaMemsetAsync(scratch + 24 * kStaticMaxElems, 0, sizeof(double), s);
    cudaStreamSynchronize(s);
    cudaGetLastError();
    return LULESH_ERR_CUDA;
  }
  unsigned bits = 0;
  if (cudaMemcpyAsync(&bits, status, sizeof(unsigned), cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return LULESH_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return LULESH_ERR_CUDA;
  if (bits & ST_EARLY) { if (site) *site = LULESH_SITE_EARLY; return LULESH_ERR_VOLUME; }
  if (bits & ST_HOURGLASS) { if (site) *site = LULESH_SITE_HOURGLASS; return LULESH_ERR_VOLUME; }
  return LULESH_OK;
}
