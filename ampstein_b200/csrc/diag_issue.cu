// Issue-rate microbenchmark behind `python bench.py --workload issue`: how many cycles a scheduler
// needs per 8 decoded weights and lane for the decode GEMV's instruction mix, with the dot product
// fed (a) through two mma.sync m16n8k16 as in exl3_gemv_kernel, (b) through one tcgen05.st into
// tensor memory as in exl3_gemv_tc_kernel, (c) not at all (decoded words folded into a checksum),
// and (d) the two mma.sync alone. Measurement infrastructure, not part of the hot path: it backs the
// statement that on sm_100 a legacy mma.sync keeps its scheduler from issuing other instructions
// for most of the eight cycles the tensor pipe works on it. No counterpart in the reference.
#include "exl3_gemv_kernel.cuh"
#include "host_common.h"
#include <vector>

namespace amp {

constexpr int DIAG_ITERS = 1024;

// V: 0 decode + two mma.sync, 1 decode + tcgen05.st (8 registers), 2 decode + checksum (four lop3),
// 3 two mma.sync on undecoded words
template <int V>
__global__ void __launch_bounds__(128) diag_issue_kernel(uint32_t* out, long long* clk, uint32_t seed)
{
    __shared__ uint32_t s_tmem;
    uint32_t tmem = 0;
    const int warp = threadIdx.x >> 5;
    if (V == 1)
    {
        if (warp == 0)
        {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&s_tmem)), "r"(32u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem = s_tmem + ((uint32_t) (warp * 32) << 16);
    }
    uint32_t w[4], prev = seed ^ 0x9e3779b9u, cur = seed * (threadIdx.x + 1) + blockIdx.x, sink = 0;
    float d0[4] = {0, 0, 0, 0}, d1[4] = {0, 0, 0, 0};
    const uint32_t b0 = seed | 0x3c003c00u, b1 = b0 + 1;
    __syncthreads();
    const long long t0 = clock64();
    // four iterations per turn: the 32 weights of a lane's chunk of four words, as the kernel walks a tile
    for (int it = 0; it < DIAG_ITERS; it += 4)
    {
        #pragma unroll
        for (int j = 0; j < 4; ++j) { w[j] = cur; cur = cur * 1664525u + 1013904223u; }
        auto quarter = [&](auto rtag)
        {
            constexpr int R = decltype(rtag)::value;
            uint32_t a[8];
            if (V == 3)
            {
                #pragma unroll
                for (int j = 0; j < 8; ++j) a[j] = w[R] + j;
            }
            else
            {
                // the decode GEMV's own decode at 4 bits, codebook 0
                uint32_t x[8];
                products8<4, R, 0>(w, prev, x);
                #pragma unroll
                for (int j = 0; j < 8; ++j) a[j] = a_word<0>(x[j]);
            }
            if (V == 0 || V == 3)
            {
                mma_16816(d0, a[0], a[4], a[1], a[5], b0, b1);
                mma_16816(d1, a[2], a[6], a[3], a[7], b1, b0);
            }
            if (V == 1)
            {
                asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                    :: "r"(tmem + (uint32_t) ((R & 1) * 16)), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]) : "memory");
                if (R == 3 && (it & 4)) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            if (V == 2)
            {
                asm volatile("lop3.b32 %0, %0, %1, %2, 0x96;" : "+r"(sink) : "r"(a[0]), "r"(a[1]));
                asm volatile("lop3.b32 %0, %0, %1, %2, 0x96;" : "+r"(sink) : "r"(a[2]), "r"(a[3]));
                asm volatile("lop3.b32 %0, %0, %1, %2, 0x96;" : "+r"(sink) : "r"(a[4]), "r"(a[5]));
                asm volatile("lop3.b32 %0, %0, %1, %2, 0x96;" : "+r"(sink) : "r"(a[6]), "r"(a[7]));
            }
        };
        quarter(std::integral_constant<int, 0>()); quarter(std::integral_constant<int, 1>());
        quarter(std::integral_constant<int, 2>()); quarter(std::integral_constant<int, 3>());
        prev = w[3];
    }
    const long long t1 = clock64();
    out[blockIdx.x * blockDim.x + threadIdx.x] = __float_as_uint(d0[0] + d0[1] + d0[2] + d0[3] + d1[0] + d1[1] + d1[2] + d1[3]) + cur + sink;
    if (threadIdx.x == 0) clk[blockIdx.x] = t1 - t0;
    if (V == 1)
    {
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(s_tmem), "r"(32u) : "memory");
    }
}

}  // namespace amp

using namespace amp;

// variant 0..3 (see the kernel), warps_per_scheduler 1..8 (= CTAs of four warps per SM). Writes the
// average cycles one scheduler needs per iteration (8 weights per lane) to *cycles_per_iter.
// Synchronises; allocates and frees its own small buffers.
AMP_API int amp_diag_issue_cycles(int variant, int warps_per_scheduler, float* cycles_per_iter)
{
    AMP_REQUIRE(variant >= 0 && variant <= 3 && warps_per_scheduler >= 1 && warps_per_scheduler <= 8 && cycles_per_iter,
                "diag_issue: variant 0..3, 1..8 warps per scheduler");
    int dev = 0, sms = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return cuda_rc(e, "cudaGetDevice");
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int blocks = sms * warps_per_scheduler;
    uint32_t* out = nullptr; long long* clk = nullptr;
    if (cudaError_t e = cudaMalloc(&out, (size_t) blocks * 128 * 4)) return cuda_rc(e, "diag_issue alloc");
    if (cudaError_t e = cudaMalloc(&clk, (size_t) blocks * 8)) { cudaFree(out); return cuda_rc(e, "diag_issue alloc"); }
    for (int rep = 0; rep < 2; ++rep)
    {
        switch (variant)
        {
            case 0: diag_issue_kernel<0><<<blocks, 128>>>(out, clk, 12345u); break;
            case 1: diag_issue_kernel<1><<<blocks, 128>>>(out, clk, 12345u); break;
            case 2: diag_issue_kernel<2><<<blocks, 128>>>(out, clk, 12345u); break;
            default: diag_issue_kernel<3><<<blocks, 128>>>(out, clk, 12345u); break;
        }
        if (cudaError_t e = cudaDeviceSynchronize()) { cudaFree(out); cudaFree(clk); return cuda_rc(e, "diag_issue run"); }
    }
    std::vector<long long> h(blocks);
    cudaError_t e = cudaMemcpy(h.data(), clk, (size_t) blocks * 8, cudaMemcpyDeviceToHost);
    cudaFree(out); cudaFree(clk);
    if (e) return cuda_rc(e, "diag_issue copy");
    double avg = 0;
    for (long long v : h) avg += (double) v;
    avg /= blocks;
    *cycles_per_iter = (float) (avg / ((double) DIAG_ITERS * warps_per_scheduler));
    return 0;
}
