// Instances of the short-batch trellis GEMM for one bit width (AMP_SHORT_K, compiled once per width)
#include "exl3_gemm_short.cuh"

#ifndef AMP_SHORT_K
#define AMP_SHORT_K 4
#endif

namespace amp {

#define AMP_CAT2(a, b) a##b
#define AMP_CAT(a, b) AMP_CAT2(a, b)
sh_fn AMP_CAT(sh_kernel_k, AMP_SHORT_K)(int cb, int grouped)
{
    constexpr int K = AMP_SHORT_K;
    static const sh_fn table[2][3] = {
        { exl3_gemm_short_kernel<K, 0, 2, false>, exl3_gemm_short_kernel<K, 1, 2, false>, exl3_gemm_short_kernel<K, 2, 2, false> },
        { exl3_gemm_short_kernel<K, 0, 1, true>, exl3_gemm_short_kernel<K, 1, 1, true>, exl3_gemm_short_kernel<K, 2, 1, true> } };
    return table[grouped][cb];
}

}  // namespace amp
