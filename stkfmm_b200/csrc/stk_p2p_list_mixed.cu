// stk_p2p_list_mixed.cu -- P2P kernels: lists, mixed precision (stk_p2p_kernel.cuh).
#include "stk_p2p_kernel.cuh"

namespace stk {

STK_P2P_UNIT(list_p2p_mixed, true, false)

}  // namespace stk
