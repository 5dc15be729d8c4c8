// Instances of the tensor-core trellis GEMM for one bit width (AMP_TC_K, compiled once per width)
#include "exl3_gemm_tc.cuh"

#ifndef AMP_TC_K
#define AMP_TC_K 4
#endif

namespace amp {

#define AMP_CAT2(a, b) a##b
#define AMP_CAT(a, b) AMP_CAT2(a, b)
tg_fn AMP_CAT(tg_kernel_k, AMP_TC_K)(int cb, int form)
{
    constexpr int K = AMP_TC_K;
    static const tg_fn table[3][3] = {
        { exl3_gemm_tc_kernel<K, 0, 2, false>, exl3_gemm_tc_kernel<K, 1, 2, false>, exl3_gemm_tc_kernel<K, 2, 2, false> },
        { exl3_gemm_tc_kernel<K, 0, 1, true>, exl3_gemm_tc_kernel<K, 1, 1, true>, exl3_gemm_tc_kernel<K, 2, 1, true> },
        { exl3_gemm_tc_kernel<K, 0, 2, false, true>, exl3_gemm_tc_kernel<K, 1, 2, false, true>, exl3_gemm_tc_kernel<K, 2, 2, false, true> } };
    return table[form][cb];
}

}  // namespace amp
