// Internal declarations shared by the libselfgpu translation units.
#pragma once

#include <cstddef>
#include <cstdint>
#include <string>

#include "../../include/selfgpu.h"

namespace selfgpu {

// Records the calling thread's last error (read back by selfgpu_last_error).
int set_error(int code, const std::string& msg);
const char* last_error();

// Host set-up (setup_host.cpp).
void legendre_quadrature(int N, int type, double* x, double* w);
int lagrange_init(int N, int ctrlType, int M, int tgtType, double* ctrl, double* tgt, double* bw,
                  double* qw, double* iM, double* dM, double* dgM, double* bM);
int mesh2d_structured(int nx, int ny, double x0, double x1, double y0, double y1, int perX, int perY,
                      double amp, int bcid, const int* rot, double* nodeCoords, int* globalNodeIDs,
                      int* sideInfo);
// Neighbour ids may reach nNeighbours (= nEl, or nEl + halo elements).
int validate_side_info(const int* sideInfo, int nEl, int nNeighbours);
// T(k,i) = w_i sqrt((2k+1)/2) L_k(x_i): nodal -> orthonormal Legendre modes
void modal_matrix(int N, const double* x, const double* w, double* T);

// Fused stage launches (stage_fp64_prod.cu / stage_fp64.cu / stage_fp32.cu).
struct StageArgs;
struct StageLaunch {
  bool allowTma;   // use the persistent bulk-copy kernel where it applies
  int smemOptin;   // opt-in shared memory per block (bytes)
  int numSMs;
  int maxGroups;   // cap on the persistent kernel's consumer groups (0 = as many as fit)
  int l2Bytes;     // the device's L2
};
}  // namespace selfgpu

#include <cuda_runtime.h>

namespace selfgpu {
// A launch that may overlap the end of the previous kernel on the stream; the
// kernel waits for that kernel's completion itself (griddepcontrol.wait).
template <class... KArgs, class... Args>
inline cudaError_t launch_dependent_smem(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t st,
                                         Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
template <class... KArgs, class... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), int grid, int block, cudaStream_t st, Args... args) {
  return launch_dependent_smem(kernel, grid, block, 0, st, args...);
}
// production FP64 (stage_fp64_prod.cu), reference roundings (stage_fp64.cu), FP32 bulk
cudaError_t launch_stage_fp64(int model, int P, const StageArgs& a, const StageLaunch& L, cudaStream_t st,
                              int* usedTma);
cudaError_t launch_stage_fp64_ref(int model, int P, const StageArgs& a, const StageLaunch& L, cudaStream_t st,
                                  int* usedTma);
cudaError_t launch_stage_fp32(int model, int P, const StageArgs& a, const StageLaunch& L, cudaStream_t st,
                              int* usedTma);
// consumer groups the persistent kernel would run with these arguments, 0 where it does not apply
int stage_groups_fp64(int model, int P, const StageArgs& a, const StageLaunch& L);
int stage_groups_fp64_ref(int model, int P, const StageArgs& a, const StageLaunch& L);
int stage_groups_fp32(int model, int P, const StageArgs& a, const StageLaunch& L);
// all stages of an rk3 call in one cooperative launch of k_fused_resident, per form
struct ResidentArgs;
cudaError_t launch_resident_fp64(int model, int P, const StageArgs& a, ResidentArgs& ra, const StageLaunch& L,
                                 cudaStream_t st);
cudaError_t launch_resident_fp64_ref(int model, int P, const StageArgs& a, ResidentArgs& ra, const StageLaunch& L,
                                     cudaStream_t st);
cudaError_t launch_resident_fp32(int model, int P, const StageArgs& a, ResidentArgs& ra, const StageLaunch& L,
                                 cudaStream_t st);
// several RK stages in one cooperative launch of the persistent kernel
// (k_fused_stage_tma<..., true>; cudaErrorNotSupported where it does not apply)
struct TmaSteps;
cudaError_t launch_stages_tma_fp64(int model, int P, const StageArgs& a, const StageLaunch& L, const TmaSteps& ms,
                                   cudaStream_t st);
cudaError_t launch_stages_tma_fp64_ref(int model, int P, const StageArgs& a, const StageLaunch& L,
                                       const TmaSteps& ms, cudaStream_t st);
cudaError_t launch_stages_tma_fp32(int model, int P, const StageArgs& a, const StageLaunch& L, const TmaSteps& ms,
                                   cudaStream_t st);
// Artificial-viscosity closure (av_closure.cuh).
struct AvArgs;
// closure: the viscosity kernel and the viscous-term kernel of one stage
// (formNu = false: the viscous-term kernel only, with the viscosity already formed)
cudaError_t launch_av_prep_fp64(int P, const AvArgs& a, cudaStream_t st, int numSMs, bool formNu = true);
cudaError_t launch_av_prep_fp32(int P, const AvArgs& a, cudaStream_t st, int numSMs, bool formNu = true);
cudaError_t launch_element_size(const double* J, const double* qw, int P, int nEl, double* h, cudaStream_t st);
cudaError_t launch_closure_features(const double* q, int P, int nEl, const AvArgs& a, float* act, float* feat,
                                    cudaStream_t st);
}  // namespace selfgpu
