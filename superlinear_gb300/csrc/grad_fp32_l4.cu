// FP32-bulk parameter-gradient passes, sh_l_max = 4.
#include "grad_inst.cuh"
namespace sus2g {
SUS2G_INSTANTIATE_GRAD(float, 4)
SUS2G_INSTANTIATE_GRAD_MOMENT(4)
}  // namespace sus2g
