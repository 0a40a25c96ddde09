// stk_p2p_direct_fp64.cu -- P2P kernels: direct sums, FP64 (stk_p2p_kernel.cuh).
#include "stk_p2p_kernel.cuh"

namespace stk {

STK_P2P_UNIT(direct_p2p_fp64, false, true)

cudaError_t direct_p2p_fp64_occupancy(int uk, int &n) {
    return with_uk(uk, [&](auto id) { return occupancy<decltype(id)::value, false, true>(n); });
}

}  // namespace stk
