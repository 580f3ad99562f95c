// fake_launchers.cu -- the kernel launchers beside fake_cuda.cpp: kernels that do
// nothing but what a test asks for (a list that overflows or times out).
#include "device_state.h"
#include "mlp.h"

extern "C" void fake_launch(const char* what, cudaStream_t s);

namespace {
int g_overflows = 0;
bool g_time_out = false;
}
extern "C" void fake_overflow_lists(int times) { g_overflows = times; }
extern "C" void fake_time_out() { g_time_out = true; }  // a grid barrier of the next list build gives up

namespace mdb {

#define LAUNCHER(name, ...) \
  void name(__VA_ARGS__, cudaStream_t s) { fake_launch(#name, s); }

LAUNCHER(launch_prune_references, const Dev&)
LAUNCHER(launch_rebuild_sort, const Dev&)
LAUNCHER(launch_inner_prune, const Dev&)
LAUNCHER(launch_nonbonded, const Dev&, bool)
LAUNCHER(launch_listed, const Dev&, bool)
LAUNCHER(launch_pme, const Dev&, bool)
LAUNCHER(launch_pme_spread, const Dev&)
LAUNCHER(launch_pme_fft, const Dev&, bool)
LAUNCHER(launch_pme_gather, const Dev&)
LAUNCHER(launch_influence, const Dev&, int)
LAUNCHER(launch_integrate, const Dev&)
LAUNCHER(launch_positions_out, const Dev&, int, int, double*)
LAUNCHER(launch_velocities_out, const Dev&, int, int, double*)
LAUNCHER(launch_forces_out, const Dev&, int, int, int, double*)
LAUNCHER(launch_positions_in, const Dev&, int, int, const double*, bool)
LAUNCHER(launch_velocities_in, const Dev&, int, int, const double*)
LAUNCHER(launch_request_rebuild, const Dev&, int)
LAUNCHER(launch_momentum, const Dev&)
LAUNCHER(launch_scale_molecules, const Dev&, int, int, double)
LAUNCHER(launch_restore_positions, const Dev&, int, int)
LAUNCHER(launch_after_box_change, const Dev&, int, int, int)
LAUNCHER(launch_molecular_offsets, const Dev&, int, int, int, double*)
LAUNCHER(launch_mlp_forward, const __nv_bfloat16*, const float*, int, float*)

void launch_rebuild_tiles(const Dev& d, cudaStream_t s) {
  fake_launch("launch_rebuild_tiles", s);
  if (g_overflows > 0) {
    --g_overflows;
    *d.halt = 1;
    d.err[0] |= kErrTileCapacity;
    d.tile_need[0] = d.sys[0].tile_cap + 1;
  }
  if (g_time_out) d.err[0] |= kErrTimeout;
  g_time_out = false;
}
bool launch_list(const Dev&, cudaStream_t) { return false; }
int prepare_list_kernel(int) { return 0; }
int allow_pme_smem(int) { return 0; }
int plane_smem(int, int) { return 0; }
int z_smem(int, int) { return 0; }
int strip_smem(int, int) { return 0; }
int molecular_offset_blocks(int) { return 1; }
cudaError_t mlp_train(const MlpDev&, const float*, const float*, int, int, uint32_t, float*, std::vector<double>*,
                      cudaStream_t s) {
  return fake_launch("mlp_train", s), cudaSuccess;
}

}  // namespace mdb
