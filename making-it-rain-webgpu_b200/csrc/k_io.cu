// k_io.cu -- states between the device's tables and the caller's arrays.
//
// The C ABI trades xyz-interleaved doubles (StepLoop.positions(), loop.ts:900);
// the device keeps one table per component, positions and forces in 2^32
// fixed point, forces by slot.  These kernels convert and interleave on the
// device and read or write the engine's pinned host block directly, so a call
// is one launch, one wait and one host copy, in place of a blocking transfer
// per table through pageable memory and a host loop over every number (an
// upload, an evaluation and its forces: 2,652 atoms 0.50 -> 0.26 ms, 27k atoms
// 1.73 -> 1.05 ms; twenty ensemble steps and 64 systems' states 76 -> 68 ms).
// Bound by the bus: 24 bytes an atom.
#include <algorithm>

#include "device_state.h"

namespace mdb {
namespace {

constexpr int kThreads = 256;
constexpr double kFixedToNm = 1.0 / 4294967296.0;  // a power of two: the product is exact

// Threads run over the interleaved array, so the bus sees whole lines.
__global__ void __launch_bounds__(kThreads) k_positions_out(const long long* x, const long long* y, const long long* z,
                                                            int n, double* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += gridDim.x * blockDim.x) {
    const int a = i / 3, k = i - 3 * a;
    out[i] = static_cast<double>((k == 0 ? x : (k == 1 ? y : z))[a]) * kFixedToNm;
  }
}

__global__ void __launch_bounds__(kThreads) k_velocities_out(const float* x, const float* y, const float* z, int n,
                                                             double* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += gridDim.x * blockDim.x) {
    const int a = i / 3, k = i - 3 * a;
    out[i] = (k == 0 ? x : (k == 1 ? y : z))[a];
  }
}

__global__ void __launch_bounds__(kThreads) k_forces_out(Dev d, int atom_off, int slot_off, int n, double* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += gridDim.x * blockDim.x) {
    const int a = i / 3, k = i - 3 * a, gs = slot_off + d.rank[atom_off + a];
    out[i] = static_cast<double>(static_cast<long long>((k == 0 ? d.fx : (k == 1 ? d.fy : d.fz))[gs])) * kFixedToNm;
  }
}

__global__ void __launch_bounds__(kThreads) k_positions_in(Dev d, int atom_off, int n, const double* in,
                                                           int clear_residual) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += gridDim.x * blockDim.x) {
    const int k = i % 3, a = atom_off + i / 3;
    (k == 0 ? d.px : (k == 1 ? d.py : d.pz))[a] = llround(in[i] * 4294967296.0);
    if (clear_residual) (k == 0 ? d.rx : (k == 1 ? d.ry : d.rz))[a] = 0.f;
  }
}

__global__ void __launch_bounds__(kThreads) k_velocities_in(Dev d, int atom_off, int n, const double* in) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += gridDim.x * blockDim.x) {
    const int k = i % 3, a = atom_off + i / 3;
    (k == 0 ? d.vx : (k == 1 ? d.vy : d.vz))[a] = static_cast<float>(in[i]);
  }
}

__global__ void k_request_rebuild(Dev d, int s) {
  for (int k = threadIdx.x; k < d.S; k += blockDim.x)
    if (s < 0 || k == s) d.rebuild_now[k] = 1;
  if (threadIdx.x == 0) *d.any_rebuild = 1;
}

int blocks_for(int n) { return std::max(1, std::min((3 * n + kThreads - 1) / kThreads, 148 * 4)); }

}  // namespace

void launch_positions_out(const Dev& d, int atom_off, int n, double* out, cudaStream_t st) {
  k_positions_out<<<blocks_for(n), kThreads, 0, st>>>(d.px + atom_off, d.py + atom_off, d.pz + atom_off, n, out);
}
void launch_velocities_out(const Dev& d, int atom_off, int n, double* out, cudaStream_t st) {
  k_velocities_out<<<blocks_for(n), kThreads, 0, st>>>(d.vx + atom_off, d.vy + atom_off, d.vz + atom_off, n, out);
}
void launch_forces_out(const Dev& d, int atom_off, int slot_off, int n, double* out, cudaStream_t st) {
  k_forces_out<<<blocks_for(n), kThreads, 0, st>>>(d, atom_off, slot_off, n, out);
}
void launch_positions_in(const Dev& d, int atom_off, int n, const double* in, bool clear_residual, cudaStream_t st) {
  k_positions_in<<<blocks_for(n), kThreads, 0, st>>>(d, atom_off, n, in, clear_residual ? 1 : 0);
}
void launch_velocities_in(const Dev& d, int atom_off, int n, const double* in, cudaStream_t st) {
  k_velocities_in<<<blocks_for(n), kThreads, 0, st>>>(d, atom_off, n, in);
}
void launch_request_rebuild(const Dev& d, int s, cudaStream_t st) {
  k_request_rebuild<<<1, kThreads, 0, st>>>(d, s);
}

}  // namespace mdb
