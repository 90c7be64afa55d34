// The tensor-core kernel for 4-bit (q4g32a.t64) weights, one instantiation per fused epilogue.
#include "k_umma.cuh"

namespace p0p {

umma_kernel_fn umma_kernel_q4(uint32_t variant, uint32_t epi) {
  static const umma_kernel_fn table[5][7] = {P0P_UMMA_ROW(P0P_ENC_Q4, 1, true, false), P0P_UMMA_ROW(P0P_ENC_Q4, 2, true, false), P0P_UMMA_ROW(P0P_ENC_Q4, 2, false, false),
                                             P0P_UMMA_ROW(P0P_ENC_Q4, 4, false, false), P0P_UMMA_ROW(P0P_ENC_Q4, 1, true, true)};
  return table[variant][epi];
}

}  // namespace p0p
