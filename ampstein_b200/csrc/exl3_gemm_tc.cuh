// What the tensor-core trellis GEMMs share: launch parameters, the slice lookup of a bundle, the swizzled
// tile layout and its descriptor, tcgen05 issue, and the decode of a packed chunk into exact fp16 weights.
#pragma once
#include "exl3_gemv_kernel.cuh"
#include "exl3_gemv_host.h"
#include "host_common.h"

namespace amp {

constexpr int TC_DECODE_WARPS = 16;           // two groups of eight that take alternate k steps
constexpr int TC_THREADS = 32 * (2 + TC_DECODE_WARPS);     // warp 0 fetches, warp 1 issues the MMAs, the rest decode
constexpr int TC_BM = 128;            // tokens per sub-tile (UMMA M)
constexpr int TC_SUB = 4;             // sub-tiles per CTA
constexpr int TC_BN = 128;            // output columns per CTA (UMMA N)
constexpr int TC_BK = 64;             // k per step (one 128-byte swizzle row)
constexpr int TC_A_SLOTS = 2, TC_B_STAGES = 3;
constexpr int TC_A_BYTES = TC_SUB * TC_BM * TC_BK * 2;     // one slot = the x~ tile of one k step: 65536
constexpr int TC_B_BYTES = TC_BN * TC_BK * 2;              // 16384
// packed trellis words travel through per-lane cp.async rings this many k steps deep (the words
// come from HBM exactly once: the ring must cover the HBM latency, a step is ~0.5 us)
__host__ __device__ constexpr int tc_p_stages(int K) { return K <= 4 ? 4 : 3; }        // per decode group: every other step
__host__ __device__ constexpr int tc_smem_bytes(int K)
{
    return 1024 + TC_A_SLOTS * TC_A_BYTES + TC_B_STAGES * TC_B_BYTES + TC_DECODE_WARPS * tc_p_stages(K) * 128 * K;
}
constexpr unsigned TC_SPIN_LIMIT = 1u << 22;   // try_wait polls before a wait is declared lost

struct TcParams
{
    const unsigned char* xt;    // rotated input, k-step-major and pre-swizzled (had_tiled_kernel): [k/64][M][128 bytes]
    const uint16_t* trellis;    // (k/16, n/16, 16K)
    const __half* svh;          // (n)
    void* c;                    // (M, n) fp16 or fp32
    int M, k, n, c_fp32;        // n: row width of the trellis / output (bundle: columns per slice)
    int sub;                    // 128-token sub-tiles per CTA: 4, or fewer when the grid would leave SMs idle
    int* status;
    int relay_release;          // pair form: the relay's remote arrival releases at cluster scope (slower; default relaxed)
    // bundle (tables == 1): several matrices or equal-width column slices in one grid, identified
    // by device pointer tables with one entry per slice, exactly as the decode kernel's table mode
    int tables;
    const long long* t_trellis;
    const long long* t_svh;
    const long long* t_c;       // may be null: outputs stacked in c as (slices, M, n)
    const int* t_stride;        // may be null: row width = n
    const int* t_src;           // may be null: rotated input of slice i is source i
    // expert groups (grouped instances of exl3_gemm_short_kernel): blockIdx.y walks a tile table
    // that a kernel in front of this one built from the routing, blockIdx.x = projection * (n / 128)
    // + column block. A tile is up to ShParams::tile consecutive rows of ONE expert in the padded,
    // expert-sorted row space of xt / c (M = its capacity); t_trellis / t_svh hold g_kinds *
    // g_experts entries, projection-major; projection p reads xt + p * M * k halves and writes
    // c + p * M * n elements.
    const int* g_ntiles;        // device: tiles in use (CTAs beyond it return at once)
    const int* g_tile_e;        // device: expert of a tile
    const int* g_tile_row0;     // device: first padded row of a tile (a multiple of 8)
    const int* g_tile_rows;     // device: valid rows of a tile (0: none)
    int g_experts;
    // experts of different bit widths: per projection a device table of the experts' widths (null:
    // all of this launch's width); a CTA whose expert has another width than this instance returns
    const unsigned char* g_bits[2];
};

// What one CTA (pair) works on: its weight, scales, output, rotated input and column block
struct TcSlice
{
    const unsigned char* trellis;
    const __half* svh;
    unsigned char* c;
    const unsigned char* xt;
    int n_row;                  // row width of trellis and output
    int nb;                     // column block (of BW columns) inside the slice
};

template <int BW>
__device__ __forceinline__ TcSlice tc_slice(const TcParams& P, int nbg)
{
    TcSlice s;
    s.trellis = reinterpret_cast<const unsigned char*>(P.trellis);
    s.svh = P.svh; s.c = reinterpret_cast<unsigned char*>(P.c); s.xt = P.xt; s.n_row = P.n; s.nb = nbg;
    if (P.tables)
    {
        const int bps = P.n / BW, slice = nbg / bps;
        s.nb = nbg - slice * bps;
        s.trellis = reinterpret_cast<const unsigned char*>(P.t_trellis[slice]);
        s.svh = reinterpret_cast<const __half*>(P.t_svh[slice]);
        s.n_row = P.t_stride ? P.t_stride[slice] : P.n;
        s.c = P.t_c ? reinterpret_cast<unsigned char*>(P.t_c[slice])
                    : reinterpret_cast<unsigned char*>(P.c) + (size_t) slice * P.M * P.n * (P.c_fp32 ? 4 : 2);
        const int src = P.t_src ? P.t_src[slice] : slice;
        s.xt = P.xt + (size_t) src * P.M * P.k * 2;
    }
    return s;
}

// K-major, 128-byte swizzle, rows of 128 bytes: byte offset of (row, 16-byte chunk)
__device__ __forceinline__ uint32_t sw128(int row, int chunk)
{
    return (uint32_t) (row * 128 + ((chunk ^ (row & 7)) << 4));
}

__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr)
{
    // start address >> 4 [0,14), LBO (1, unused for swizzled K-major) [16,30), SBO = 1024 B >> 4
    // [32,46), descriptor version 1 [46,48), layout SWIZZLE_128B (2) [61,64)
    return (uint64_t) ((smem_addr & 0x3ffff) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        :: "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
}

// 4K bytes of one lane, global -> this lane's ring slot, widest cp.async the alignment allows
template <int K>
__device__ __forceinline__ void cp_async_chunk(uint32_t dst, const unsigned char* src)
{
    if constexpr (K % 4 == 0)
    {
        #pragma unroll
        for (int i = 0; i < K / 4; ++i)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst + 16 * i), "l"(src + 16 * i) : "memory");
    }
    else if constexpr (K % 2 == 0)
    {
        #pragma unroll
        for (int i = 0; i < K / 2; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"(dst + 8 * i), "l"(src + 8 * i) : "memory");
    }
    else
    {
        #pragma unroll
        for (int i = 0; i < K; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(dst + 4 * i), "l"(src + 4 * i) : "memory");
    }
}

// two states -> two exact fp16 weights packed (a in the low half), bit-identical to the reference
template <int CB>
__device__ __forceinline__ uint32_t weights2(uint32_t sa, uint32_t sb)
{
    if constexpr (CB == 2)
    {
        const uint32_t raw = __byte_perm(cb2_raw(sa), cb2_raw(sb), 0x5410);
        const __half2 kinv = __half2half2(__ushort_as_half((unsigned short) 0x1eee));
        const __half2 kbias = __half2half2(__ushort_as_half((unsigned short) 0xc931));
        const __half2 w = __hfma2(*reinterpret_cast<const __half2*>(&raw), kinv, kbias);
        return *reinterpret_cast<const uint32_t*>(&w);
    }
    else
    {
        const uint32_t ya = cb_halves<CB>(sa), yb = cb_halves<CB>(sb);
        const uint32_t lo = __byte_perm(ya, yb, 0x5410), hi = __byte_perm(ya, yb, 0x7632);
        const __half2 w = __hadd2(*reinterpret_cast<const __half2*>(&lo), *reinterpret_cast<const __half2*>(&hi));
        return *reinterpret_cast<const uint32_t*>(&w);
    }
}

// device address of the prefill GEMMs' status word on a device (host side, cached per device)
int tc_status_ptr(int dev, int** out);

extern int g_short_split, g_short_tile;
// short-batch form; P as prepared by launch_gemm_tc. AMP_E_UNSUPPORTED: nothing launched, no plan is expected to
// take less than `limit` microseconds.
int launch_gemm_short(const TcParams& P, int K, int cb, long blocks, int sms, int dev, double limit, cudaStream_t stream);

}  // namespace amp
