// stk_p2p_list_fp64.cu -- P2P kernels: lists, FP64 (stk_p2p_kernel.cuh).
#include "stk_p2p_kernel.cuh"

namespace stk {

STK_P2P_UNIT(list_p2p_fp64, false, false)

}  // namespace stk
