// stk_p2p_direct_mixed.cu -- P2P kernels: direct sums, mixed precision (stk_p2p_kernel.cuh).
#include "stk_p2p_kernel.cuh"

namespace stk {

STK_P2P_UNIT(direct_p2p_mixed, true, true)

}  // namespace stk
