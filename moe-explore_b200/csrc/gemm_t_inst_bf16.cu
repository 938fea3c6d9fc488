// Explicit instantiations of the transposed-tile grouped GEMM: __nv_bfloat16.
#define MOE_GEMM_DEFINE_LAUNCH
#include "gemm_t_kernel.cuh"

namespace moe {
#define MOE_INST(UNIT, W_K, EPI) \
  template int launch_t<__nv_bfloat16, UNIT, W_K, EPI>(const TMaps&, const GemmArgs&, const LaunchParams&);
#define MOE_INST_UNIT(UNIT)          \
  MOE_INST(UNIT, false, EPI_ACT)     \
  MOE_INST(UNIT, false, EPI_GLU)     \
  MOE_INST(UNIT, false, EPI_ACT_AUX) \
  MOE_INST(UNIT, true, EPI_ACT)      \
  MOE_INST(UNIT, true, EPI_ACT_AUX)  \
  MOE_INST(UNIT, true, EPI_DGLU)
MOE_INST_UNIT(128)
MOE_INST_UNIT(256)
}  // namespace moe
