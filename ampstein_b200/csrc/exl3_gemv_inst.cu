// Kernel instances of the trellis-decode GEMV for one bitrate; compiled once per K with
// -DAMP_GEMV_K=<1..8, 17..19> (17..19: the half-integer rates) so the translation units build in parallel.
#include "exl3_gemv_kernel.cuh"
#include "exl3_gemv_tc.cuh"

#ifndef AMP_GEMV_K
#error "compile with -DAMP_GEMV_K=<bits>"
#endif

#define AMP_CAT_(a, b) a##b
#define AMP_CAT(a, b) AMP_CAT_(a, b)

namespace amp {

#if AMP_GEMV_K > 8
// half-integer bitrates (mul1 codebook): single matrices, fp16 activations
gemv_fn AMP_CAT(gemv_kernel_k, AMP_GEMV_K)(int cb, int MB, int mode, int gin)
{
    // plain input, input already rotated (no fused all-reduce: no entry takes these rates with one)
    static const gemv_fn fn[2][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 2>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 2> },
    };
    if (cb != 2 || mode || (gin != 0 && gin != 2) || MB < 1 || MB > 2) return nullptr;
    return fn[gin / 2][MB - 1];
}
#else
gemv_fn AMP_CAT(gemv_kernel_k, AMP_GEMV_K)(int cb, int MB, int mode, int gin)
{
    // input gathered from the all-reduce buffers (split exchange)
    static const gemv_fn fng[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 1>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 1> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 1>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 1> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 1>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 1> },
    };
    // input already rotated
    static const gemv_fn fnr[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 2>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 2> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 2>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 2> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 2>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 2> },
    };
    // input = silu(gate) * up, formed in the prologue
    static const gemv_fn fna[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 3>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 3> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 3>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 3> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 3>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 3> },
    };
    // input = RMSNorm(x + residual) * w, formed in the prologue
    static const gemv_fn fnn[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 4>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 4> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 4>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 4> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 4>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 4> },
    };
    // split norm: producer epilogue (5) and consumer prologue (6)
    static const gemv_fn fnp[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 5>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 5> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 5>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 5> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 5>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 5> },
    };
    static const gemv_fn fnc[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 6>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 6> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 6>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 6> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 6>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 6> },
    };
    static const gemv_fn fn[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2> },
    };
    // with the fused all-reduce: plain input (8), input already rotated (9)
    static const gemv_fn far[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 8>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 8> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 8>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 8> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 8>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 8> },
    };
    static const gemv_fn farr[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 0, 9>, exl3_gemv_kernel<AMP_GEMV_K, 0, 2, 0, 9> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 0, 9>, exl3_gemv_kernel<AMP_GEMV_K, 1, 2, 0, 9> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 0, 9>, exl3_gemv_kernel<AMP_GEMV_K, 2, 2, 0, 9> },
    };
    // grouped experts: runs from a table, and a single token (gin 7)
    static const gemv_fn moe[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 1>, exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 2> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 1>, exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 2> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 1>, exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 2> },
    };
    static const gemv_fn one[3][2] =
    {
        { exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 1, 7>, exl3_gemv_kernel<AMP_GEMV_K, 0, 1, 2, 7> },
        { exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 1, 7>, exl3_gemv_kernel<AMP_GEMV_K, 1, 1, 2, 7> },
        { exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 1, 7>, exl3_gemv_kernel<AMP_GEMV_K, 2, 1, 2, 7> },
    };
    // cb 3 = the mul1 codebook with int8 activations: one batch row, plain launches only
    if (cb == 3) return (MB == 1 && !mode && (!gin || gin == 8)) ? (gin ? exl3_gemv_kernel<AMP_GEMV_K, 3, 1, 0, 8> : exl3_gemv_kernel<AMP_GEMV_K, 3, 1>) : nullptr;
    if (cb == 4) return (MB == 1 && !mode && (!gin || gin == 8)) ? (gin ? exl3_gemv_kernel<AMP_GEMV_K, 4, 1, 0, 8> : exl3_gemv_kernel<AMP_GEMV_K, 4, 1>) : nullptr;
    if (cb < 0 || cb > 2 || MB < 1 || MB > 2 || mode < 0 || mode > 2) return nullptr;
    if (mode) return (MB == 1 && (!gin || gin == 7)) ? (gin ? one : moe)[cb][mode - 1] : nullptr;
    if (gin >= 8) return (gin == 8 ? far : farr)[cb][MB - 1];
    if (gin == 4) return fnn[cb][MB - 1];
    if (gin == 5) return fnp[cb][MB - 1];
    if (gin == 6) return fnc[cb][MB - 1];
    return gin == 3 ? fna[cb][MB - 1] : (gin == 2 ? fnr[cb][MB - 1] : (gin ? fng[cb][MB - 1] : fn[cb][MB - 1]));
}

// tensor-memory form (dense / bundle launches of up to eight rows)
gemv_fn AMP_CAT(gemv_tc_kernel_k, AMP_GEMV_K)(int cb, int ar)
{
    static const gemv_fn fn[3][2] =
    {
        { exl3_gemv_tc_kernel<AMP_GEMV_K, 0, 0>, exl3_gemv_tc_kernel<AMP_GEMV_K, 0, 1> },
        { exl3_gemv_tc_kernel<AMP_GEMV_K, 1, 0>, exl3_gemv_tc_kernel<AMP_GEMV_K, 1, 1> },
        { exl3_gemv_tc_kernel<AMP_GEMV_K, 2, 0>, exl3_gemv_tc_kernel<AMP_GEMV_K, 2, 1> },
    };
    if (cb < 0 || cb > 2) return nullptr;
    return fn[cb][ar ? 1 : 0];
}
#endif

}  // namespace amp
