#include "lbmx_pair_kernels.cuh"
namespace lbmx {
LBMX_INSTANTIATE_PAIR(__nv_bfloat16)
}
