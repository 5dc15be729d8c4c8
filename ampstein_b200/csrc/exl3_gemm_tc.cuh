// Trellis GEMM on the tensor cores, for every row count above the decode kernel's and for expert groups:
// C (M, n) = x~ (M, k) @ W_hat (k, n) -> Hadamard -> * svh, with W_hat decoded from the trellis into shared memory and
// multiplied by tcgen05.mma (accumulators in tensor memory). x~ = fp16(H(x * suh) / sqrt(128)) is written by the
// rotation kernel in front (had_tiled_kernel).
//
// Replaces the reference's trellis-decode GEMM (exl3_gemm_kernel, vendor/exl3/exllamav3_ext/quant/exl3_gemm_kernel.cuh:8-80,
// mma.sync, re-decoding the weights for every 16-row slab) and its reconstruct + cuBLAS path (torch_exl3_gemm_recon,
// src/torch/amp_torch.cpp:11148-11230, which writes the whole fp16 weight to global memory first).
//
// The DECODED WEIGHTS are the M operand (128 output columns per CTA) and the tokens the N operand, so that a weight
// is decoded once per tile of up to 512 tokens and the x~ tile of a step is only as tall as the batch. Three forms:
//   * dense: one CTA of 16 decode warps per SM; k is split over the CTAs of a thread-block cluster, so that a small
//     matrix or a short batch still spreads over the device (partial sums meet through distributed shared memory);
//   * pair: two CTAs (two SMs) with tcgen05 cta_group::2, 256 columns x up to 512 tokens. Each CTA decodes its 128
//     columns and fetches half of the x~ rows; the tensor cores of both read both halves. For many rows. k may be split
//     over up to four pairs of a cluster (x~ then crosses the L2 once per 256 columns also where the grid needs the split);
//   * grouped: one CTA of 8 decode warps per (expert tile, projection, 128 columns), two per SM, so that one CTA's
//     set-up and epilogue run under the other's decode.
//
// What bounds it: the decode up to about 300 tokens per tile (7.7 warp instructions per 32 weights all told where the
// decode is most of the work: 11.4 weights per clock and SM at 0.75 issue slots per scheduler, 0.40 us per 64-row step of
// a CTA), the tensor pipe above (512 tokens: 0.65 us per step, of which 0.57 is the MMAs'; active in 69 % of the cycles of
// 1024 x 4096 x 14336). What it replaced: token-major kernels whose k loop was a chain of barrier hand-overs of 0.6 -
// 0.75 us per step whatever the batch.
//
// Warps 0 .. 8 NG - 1 decode, in groups of four that take alternate 64-row steps (a warp owns two 16-column tile
// columns); one warp fetches x~ with bulk copies, one issues the MMAs (second CTA of a pair: three report its operands
// to the first CTA instead). A step's stages (decoded weights, x~) are
// freed by one tcgen05.commit.
//
// Epilogue: the accumulator's rows are output columns, its columns tokens. Every CTA lays its partial sums out
// token by token in its own shared memory and sends every CTA of the cluster the run of tokens that one
// finishes; there four lanes per token add the partials in ascending k order (bitwise reproducible), run the 128-point
// Hadamard, scale and store.
//
// Every mbarrier wait is bounded. A role whose wait ran out hands nothing over any more (no copy, no tile, no MMA, no
// arrival), so that every role that depends on it runs out as well, in the other CTA of
// a pair too; the CTAs of a split tell each other before the partial sums are added. What was not computed from complete
// operands is therefore not stored, the status word is set, and no CTA leaves before its own copies and MMAs are done.
#pragma once
#include "exl3_gemv_kernel.cuh"
#include "exl3_gemv_host.h"
#include "host_common.h"

namespace amp {

constexpr int TC_BM = 128;            // output columns per CTA (UMMA M)
constexpr int TC_BN = 128;            // ... as the bundle and grouping code counts them
constexpr int TC_BK = 64;             // k per step (one 128-byte swizzle row)
constexpr unsigned TC_SPIN_LIMIT = 1u << 22;   // try_wait polls before a wait is declared lost (about 4 us each)

struct TcParams
{
    const unsigned char* xt;    // rotated input, k-step-major and pre-swizzled (had_tiled_kernel): [k/64][M][128 bytes]
    const uint16_t* trellis;    // (k/16, n/16, 16K)
    const __half* svh;          // (n)
    void* c;                    // (M, n) fp16 or fp32
    int M, k, n, c_fp32;        // n: row width of the trellis / output (bundle: columns per slice)
    int* status;
    unsigned wait_limit, wait_limit_last;   // polls of a barrier wait; of the last CTA of a cluster or pair (amp_exl3_set_gemm_wait_limit)
    // bundle (tables == 1): several matrices or equal-width column slices in one grid, identified
    // by device pointer tables with one entry per slice, exactly as the decode kernel's table mode
    int tables;
    const long long* t_trellis;
    const long long* t_svh;
    const long long* t_c;       // may be null: outputs stacked in c as (slices, M, n)
    const int* t_stride;        // may be null: row width = n
    const int* t_src;           // may be null: rotated input of slice i is source i
    // expert groups (grouped instances of exl3_gemm_tc_kernel): blockIdx.y walks a tile table
    // that a kernel in front of this one built from the routing, blockIdx.x = projection * (n / 128)
    // + column block. A tile is up to TgParams::tile consecutive rows of ONE expert in the padded,
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

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_u32(bar)) : "memory");
}

// Shared shifts (window_product) where they take load off the integer ALU, which also packs here. At 2, 3 and 6 bits a shift and a
// mask on the other pipe per window leave it less to do in most instances. us, one each / shared (24 to 333 rows x 4096 x 14336,
// 14336 x 4096, 5120 x 25600, 2048 x 5120; expert layers of 59, 300 and 1500 tokens x top-8 of 128):
//   2 bits   24 x 4096 x 14336 27.6 / 28.4 (codebook 2 27.3 / 28.4), 200 x 5120 x 25600 74.0 / 75.4, from 333 rows on between 2 %
//            more and 1 % less (92.0 / 90.2); experts 239 / 230, 244 / 235, 318 / 310 (codebook 2 216 / 217, 225 / 224, 308 / 305)
//   3, 6     codebooks 0, 1: dense 30.2 / 30.4 and 30.4 / 32.1, experts of 59 tokens 236 / 240 and 240 / 246; codebook 2, whose masks are
//            ALU work too: 59 tokens 221 / 218 and 232 / 231, 5120 x 25600 at 6 bits, 333 rows 92.3 / 91.0, 3 bits dense level
template <int K, int CB, bool GROUPED>
constexpr bool tg_shared_phase = shared_phase<K> && (K == 2 ? GROUPED : CB == 2 || (K != 3 && K != 6));

constexpr int TG_MAX_N = 256;                 // tokens per accumulator (UMMA N)
constexpr int TG_MAX_TOKENS = 512;            // tokens per tile: two accumulators, with 16 decode warps only
constexpr int TG_MAX_STAGES = 16;
// bytes of a token's 128 partial sums in the epilogue: 16 of padding make the reads conflict-free; rows sent to a
// peer stay on 128-byte lines instead
__host__ __device__ constexpr int tg_row(int split) { return split > 1 ? 512 : 528; }
constexpr int TG_W_BYTES = TC_BN * TC_BK * 2; // decoded weights of a step: 16384

struct TgParams
{
    TcParams t;                 // pointers, sizes, bundle tables, expert tile table
    int tile;                   // tokens per tile: a multiple of 16, at most 512
    int n0;                     // tokens of the first accumulator: a multiple of 16, at most 256 (the rest: the second, at column 256)
    int split;                  // slices of k: CTAs per cluster (1: no cluster), pairs per cluster in the pair form
    int wstages, xstages;       // stages of decoded weights and of x~: wstages >= 2 NG
    int x_area;                 // expert groups: bytes of all x~ stages together (xstages then follows from the tile's rows)
    int tmem_cols;              // tensor-memory columns to allocate: a power of two >= tile, >= 32 (two accumulators: 512)
    int share;                  // tokens a CTA finishes per epilogue pass (no split, or several passes: a multiple of 16)
    int recv_off;               // where the partial sums are received: behind the stages, or 0: over them
    int pdl;                    // launched as a programmatic dependent of the kernel that writes x~
};

// warps that decode a step together (each 8 / 4 = 2 of the eight 16-column tiles of the block): per step a warp
// pays about 60 instructions of bookkeeping, so that it should not be shorter
constexpr int TG_GROUP_WARPS = 4;
// Warps of a pair's second CTA that tell the first one that a step's operands are ready. The arrival releases at cluster
// scope, which takes about 1 us (it waits for what the SM has in flight): one relay paces the pair at 1.1 us per step,
// three taking every third step each cost nothing (2048 rows, sustained, us, one relay / three / one whose arrival was
// relaxed, which no rule of the memory model covers: 4096 x 14336 at 3 bits 295 / 236 / 234, 14336 x 4096 at 4 bits 284 / 247 /
// 240, 4096 x 6144 at 5 bits 152 / 114 / 117). Two warps more fit: registers are granted to groups of four warps.
constexpr int TG_RELAYS = 3;
__host__ __device__ constexpr int tg_threads(int ng, bool pair = false) { return 32 * (8 * ng + 2 + (pair ? TG_RELAYS - 1 : 0)); }

// K words of one lane from global memory, widest loads the alignment allows. Where that takes several loads,
// each touches the same sectors of the warp's rows again and has to find them in L1 (with L1::no_allocate 5 bits
// streamed at 4.6 weights per clock and SM instead of 10.8)
template <int K>
__device__ __forceinline__ void load_chunk_g(const unsigned char* p, uint32_t (&w)[K])
{
    if constexpr (K % 4 == 0)
    {
        #pragma unroll
        for (int i = 0; i < K / 4; ++i)
            asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3]) : "l"(p + 16 * i));
    }
    else if constexpr (K % 2 == 0)
    {
        #pragma unroll
        for (int i = 0; i < K / 2; ++i)
            asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(w[2 * i]), "=r"(w[2 * i + 1]) : "l"(p + 8 * i));
    }
    else
    {
        #pragma unroll
        for (int i = 0; i < K; ++i)
            asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(w[i]) : "l"(p + 4 * i));
    }
}

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ void lds_f32x2(uint32_t addr, f32x2& a, f32x2& b)
{
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr) : "memory");
}

// Products of two weights (cb_product) -> two exact fp16 weights, packed (a in the low half), bit-identical to the reference.
// Codebooks 0 / 1: the halves of each word are added by one instruction per weight on the half-precision pipe and
// packed by one byte permute per pair (two permutes and one addition: the integer ALU is the busier pipe).
template <int CB>
__device__ __forceinline__ uint32_t tg_weights2(uint32_t xa, uint32_t xb)
{
    if constexpr (CB == 2)
    {
        const uint32_t raw = __byte_perm(cb2_raw_of(xa), cb2_raw_of(xb), 0x5410);
        const __half2 kinv = __half2half2(__ushort_as_half((unsigned short) 0x1eee));
        const __half2 kbias = __half2half2(__ushort_as_half((unsigned short) 0xc931));
        const __half2 w = __hfma2(*reinterpret_cast<const __half2*>(&raw), kinv, kbias);
        return *reinterpret_cast<const uint32_t*>(&w);
    }
    else
    {
        const uint32_t ya = cb_halves_of(xa), yb = cb_halves_of(xb);
        const __half2 ha = *reinterpret_cast<const __half2*>(&ya), hb = *reinterpret_cast<const __half2*>(&yb);
        const __half2 wa = __hadd2(__low2half2(ha), __high2half2(ha)), wb = __hadd2(__low2half2(hb), __high2half2(hb));
        return __byte_perm(*reinterpret_cast<const uint32_t*>(&wa), *reinterpret_cast<const uint32_t*>(&wb), 0x5410);
    }
}

// Whole-warp wait for an mbarrier phase, bounded, as straight-line code: the usual case (already there) is
// one instruction and a branch not taken. Returns false when a first look and `limit` more were not enough (a look at a
// phase that is not there yet lasts about 4 us).
// CLUSTER: acquires at cluster scope (the arrival comes from the other CTA of a pair).
#define AMP_TG_WAIT(sem) \
    asm volatile( \
        "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\t" \
        "mbarrier.try_wait.parity" sem ".shared::cta.b64 p, [%1], %2;\n\t" \
        "@p bra $TG_DONE_%=;\n\t" \
        "mov.u32 n, %3;\n" \
        "$TG_POLL_%=:\n\t" \
        "setp.eq.u32 q, n, 0;\n\t" \
        "@q bra $TG_DONE_%=;\n\t" \
        "sub.u32 n, n, 1;\n\t" \
        "mbarrier.try_wait.parity" sem ".shared::cta.b64 p, [%1], %2;\n\t" \
        "@!p bra $TG_POLL_%=;\n" \
        "$TG_DONE_%=:\n\t" \
        "selp.u32 %0, 1, 0, p;\n\t}" \
        : "=r"(r) : "r"(bar), "r"(parity), "r"(limit) : "memory")
template <bool CLUSTER = false>
__device__ __forceinline__ bool tg_wait(uint32_t bar, uint32_t parity, uint32_t limit)
{
    uint32_t r;
    if constexpr (CLUSTER) AMP_TG_WAIT(".acquire.cluster");
    else AMP_TG_WAIT("");
    return r != 0;
}
#undef AMP_TG_WAIT

// one look at an mbarrier phase
__device__ __forceinline__ uint32_t tg_test(uint32_t bar, uint32_t parity)
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r) : "r"(bar), "r"(parity) : "memory");
    return r;
}

// one lane of the (converged) warp
__device__ __forceinline__ bool tg_elect()
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}

template <bool PAIR>
__device__ __forceinline__ void tg_umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    if constexpr (PAIR)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

// Arrives, once every tcgen05.mma issued so far by this thread has completed, on the barrier at this shared-memory
// offset in both CTAs of a pair (an arrival multicast, not a load)
__device__ __forceinline__ void tg_commit_both(uint64_t* bar, unsigned short pair_mask)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 :: "r"(smem_u32(bar)), "h"(pair_mask) : "memory");
}

// An arrival on a barrier of the first CTA of a pair: publishes what this thread wrote or observed (releasing arrivals of
// the decode warps, completed bulk copies) to whoever acquires the phase at cluster scope. What the pair's MMAs read in this
// CTA's shared memory: x~ bytes whose bulk copy completed on the barrier the relay has acquired, and weight tiles whose
// writers each ran fence.proxy.async and a releasing arrive on another one; the first CTA's issue warp acquires this phase.
__device__ __forceinline__ void tg_arrive_cluster(uint32_t cluster_bar)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" :: "r"(cluster_bar) : "memory");
}

__device__ __forceinline__ void tg_st_cluster_u32(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t tg_cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

template <int K, int CB, int NG, bool GROUPED, bool PAIR = false>
__global__ __launch_bounds__(tg_threads(NG, PAIR), NG == 1 ? 2 : 1)
void exl3_gemm_tc_kernel(const TgParams S)
{
    const TcParams& P = S.t;
    if constexpr (GROUPED)
    {
        // the whole CTA leaves, before any barrier or allocation (the first one of the grid not before the grid in front is done:
        // a grid without any tile is over only then, see ms_begin)
        if ((int) blockIdx.y >= *P.g_ntiles || P.g_tile_rows[blockIdx.y] <= 0)
        {
            if (S.pdl && blockIdx.x == 0 && blockIdx.y == 0) pdl_wait();
            return;
        }
        const unsigned char* bits = P.g_bits[(int) blockIdx.x / (P.n / TC_BN)];
        if (bits && bits[P.g_tile_e[blockIdx.y]] != K) return;
    }
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw;
    if (smem_u32(smem_raw) & 1023)                           // (the swizzle needs the alignment the declaration asks for)
    {
        if (threadIdx.x == 0) atomicExch(P.status, 2);
        if (S.pdl) pdl_wait();
        return;
    }
    __shared__ uint64_t x_full[TG_MAX_STAGES], w_full[TG_MAX_STAGES], done[TG_MAX_STAGES], peer[PAIR ? TG_MAX_STAGES : 1];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_bad;
    __shared__ __align__(16) uint2 s_svh[32];                    // the block's output scales
    constexpr int NDEC = 8 * NG, NGR = NDEC / TG_GROUP_WARPS;    // decode warps; groups of them that take alternate steps

    // the kernel behind (as a rule the rotation of the next linear, or of the expert layer's activations) may move in as this
    // grid's CTAs leave; it waits for all of them before it does anything
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int t = threadIdx.x, lane = t & 31, warp = __shfl_sync(0xffffffffu, t >> 5, 0);
    const int split = GROUPED ? 1 : S.split;
    // place in the cluster: slice of k (crank), CTA of a pair (prank); the CTA that holds the same columns in slice i
    const int rank = PAIR || split > 1 ? (int) tg_cluster_rank() : 0;
    const int prank = PAIR ? rank & 1 : 0, crank = PAIR ? rank >> 1 : rank;
    auto peer_of = [&](int i) { return (uint32_t) (PAIR ? 2 * i + prank : i); };
    TcSlice W;
    int m0, rows;
    if constexpr (GROUPED)
    {
        const int tile = blockIdx.y, bpk = P.n / TC_BN, kind = (int) blockIdx.x / bpk;
        const size_t idx = (size_t) kind * P.g_experts + P.g_tile_e[tile];
        W.trellis = reinterpret_cast<const unsigned char*>(P.t_trellis[idx]);
        W.svh = reinterpret_cast<const __half*>(P.t_svh[idx]);
        W.c = reinterpret_cast<unsigned char*>(P.c) + (size_t) kind * P.M * P.n * (P.c_fp32 ? 4 : 2);
        W.xt = P.xt + (size_t) kind * P.M * P.k * 2;
        W.n_row = P.n;
        W.nb = (int) blockIdx.x - kind * bpk;
        m0 = P.g_tile_row0[tile];
        rows = min(P.g_tile_rows[tile], S.tile);
    }
    else
    {
        W = tc_slice<TC_BN>(P, PAIR ? (int) blockIdx.x / (2 * split) * 2 + prank : (int) blockIdx.x / split);
        m0 = (int) blockIdx.y * S.tile;
        rows = min(S.tile, P.M - m0);
    }
    const int nb = W.nb;
    const int ksteps = P.k / TC_BK;
    const int ks0 = ksteps * crank / split, nsteps = ksteps * (crank + 1) / split - ks0;     // (split <= ksteps: never empty)
    const size_t tiles_n = (size_t) W.n_row >> 4;
    // expert groups: the x~ stages are as tall as this tile, so that short tiles get more of them; pairs: half a tile
    const int x_bytes = (GROUPED ? (rows + 15) & ~15 : (PAIR ? S.tile / 2 : S.tile)) * (TC_BK * 2);
    // tokens of the two accumulators, and how many rows of each this CTA fetches (pairs: its half of the MMA's N)
    const int rows0 = min(rows, S.n0), rows1 = NG > 1 ? max(rows - S.n0, 0) : 0;
    const int n16 = (rows0 + 15) & ~15, n16b = (rows1 + 15) & ~15;
    const int WS = S.wstages, XS = GROUPED ? min(TG_MAX_STAGES, S.x_area / x_bytes) : S.xstages, DS = max(WS, XS);
    unsigned char* x_base = smem + WS * TG_W_BYTES;

    if (t == 0)
    {
        // done[i % DS]: the MMAs of step i have completed -- one commit per step frees the x~ stage and the
        // weight stage of step i; who waits for step i - XS or i - WS finds it in this ring
        for (int i = 0; i < XS; ++i) mbar_init(&x_full[i], 1);
        for (int i = 0; i < DS; ++i) mbar_init(&done[i], 1);
        // pairs: the second CTA's x~ and weights of a step are ready (first CTA only)
        if (PAIR) for (int i = 0; i < DS; ++i) mbar_init(&peer[i], 1);
        for (int i = 0; i < WS; ++i) mbar_init(&w_full[i], TG_GROUP_WARPS);
        fence_mbar_init();
        s_bad = 0;
    }
    __syncwarp();
    if (warp == NDEC)
    {
        if constexpr (PAIR)
        {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&s_tmem)), "r"((uint32_t) S.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
        else
        {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&s_tmem)), "r"((uint32_t) S.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    if (warp == NDEC + 1) s_svh[lane] = reinterpret_cast<const uint2*>(W.svh + (size_t) nb * 128)[lane];      // (8-byte aligned)
    // The decode warps' packed words go straight into registers, one step ahead of their use (two: no gain). (Not through
    // cp.async rings: the release of a step's barrier waits for the warp's copies in flight, so that every
    // step paid the HBM latency -- 1.1 us per step and warp, 20 us for 77 x 4096 x 4096 at 4 bits.)
    constexpr int GW = TG_GROUP_WARPS, NT = 8 / GW;
    const int dw = warp % GW, grp = warp / GW;                   // first tile column / NT, first step (decode warps)
    const int gq = lane >> 2, pq = lane & 3;                     // 32-weight piece of the tile, tile row of the step
    const size_t group_bytes = (size_t) NGR * 4 * tiles_n * (32 * K);                    // from one step of this warp to its next
    const unsigned char* src = W.trellis + ((size_t) ((ks0 + grp) * 4 + pq) * tiles_n + (size_t) nb * 8 + dw * NT) * (32 * K) + gq * (4 * K);
    int left = warp < NDEC ? (nsteps - grp + NGR - 1) / NGR : 0;                         // steps of this warp
    uint32_t next[NT][K];
    auto fetch_words = [&]()
    {
        #pragma unroll
        for (int c = 0; c < NT; ++c) load_chunk_g<K>(src + c * (32 * K), next[c]);
        src += group_bytes;
    };
    if (left > 0) fetch_words();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync_all();                            // both CTAs' barriers exist before anyone arrives remotely
    // (the issue warp has time: its arrival publishes s_bad = 0. From the decode warps a releasing arrival costs 0.5 us)
    else if (split > 1) { if (warp == NDEC + 1) cluster_arrive_started<true>(); else cluster_arrive_started(); }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    // 0: a wait of this role ran out. It walks on to its end, looks at later barriers once each and hands nothing over any
    // more; every barrier below is still reached.
    auto full_limit = [&]() { return !GROUPED && crank == split - 1 && (!PAIR || prank == 1) ? P.wait_limit_last : P.wait_limit; };
    unsigned limit = full_limit();
    auto wait_bar = [&](uint32_t bar, uint32_t parity)
    {
        if (!tg_wait(bar, parity, limit)) { limit = 0; s_bad = 1; }
    };
    const uint32_t w_base = smem_u32(smem), b_x = smem_u32(x_full), b_w = smem_u32(w_full), b_done = smem_u32(done), b_peer = smem_u32(peer);
    (void) b_peer;

    if (warp == NDEC)
    {
        // ---- fetch ----
        if (S.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");          // x~ comes from the kernel in front
        // entry of `done` that frees the stage of step i: step i - XS; the first XS steps find the (passing)
        // parity of a barrier nobody has arrived on yet
        int s = 0, sd = DS - XS; uint32_t phd = 1;
        if (sd == DS) { sd = 0; phd = 0; }
        // rows this CTA fetches of each accumulator: all, or in a pair one half (the other CTA's tensor core reads
        // it in place). Rows beyond the batch stay stale: their accumulator columns are never read.
        const int h0 = PAIR ? n16 / 2 : n16, h1 = PAIR ? n16b / 2 : n16b;
        const int e0 = max(0, min(rows0 - prank * h0, h0)), e1 = max(0, min(rows1 - prank * h1, h1));
        const unsigned char* xs = W.xt + (((size_t) ks0 * P.M + m0 + prank * h0) << 7);
        const size_t to1 = ((size_t) (S.n0 + prank * h1 - prank * h0)) << 7;
        const int off1 = (PAIR ? S.n0 / 2 : S.n0) * (TC_BK * 2);
        uint32_t phs = 0;
        int issued = 0;
        for (int i = 0; i < nsteps; ++i)
        {
            wait_bar(b_done + sd * 8, phd);
            if (tg_elect() && limit)
            {
                mbar_expect_tx(&x_full[s], (uint32_t) (e0 + e1) * 128);
                if (e0 > 0) bulk_g2s(x_base + s * x_bytes, xs, (uint32_t) e0 * 128, &x_full[s]);
                if (NG > 1 && e1 > 0) bulk_g2s(x_base + s * x_bytes + off1, xs + to1, (uint32_t) e1 * 128, &x_full[s]);
            }
            if (limit == 0) continue;
            ++issued;
            xs += (size_t) P.M << 7;
            if (++s == XS) { s = 0; phs ^= 1; }
            if (++sd == DS) { sd = 0; phd ^= 1; }
        }
        __syncwarp();
        // the last copies have landed before this warp leaves, whoever gave up waiting for them
        for (int j = min(issued, XS); j > 0; --j)
        {
            if (s == 0) { s = XS; phs ^= 1; }
            --s;
            tg_wait(b_x + s * 8, phs, full_limit());
        }
    }
    else if (PAIR && prank != 0 && warp > NDEC)
    {
        // ---- relay (second CTA of a pair): tell the first CTA that this CTA's halves of a step are ready; see TG_RELAYS ----
        const int r = warp - (NDEC + 1), held = min(XS, WS);
        int s = r % WS, sx = r % XS, sd = r % DS, sq = r + DS - held, last = -1;
        uint32_t ph = (r / WS) & 1, phx = (r / XS) & 1, phd = (r / DS) & 1, phq = 1, phl = 0;
        if (sq >= DS) { sq -= DS; phq = 0; }
        for (int i = r; i < nsteps; i += TG_RELAYS)
        {
            // The stages' barriers have passed the phases of the steps in front (other relays'): a phase that is two behind
            // has the same parity as the one waited for. (And no further than this step's: done needs this arrival.)
            wait_bar(b_done + sq * 8, phq);
            wait_bar(b_x + sx * 8, phx);
            wait_bar(b_w + s * 8, ph);
            if (tg_elect() && limit) tg_arrive_cluster(cluster_map(b_peer + sd * 8, (uint32_t) rank & ~1u));
            __syncwarp();
            if (limit == 0) continue;
            last = sd; phl = phd;
            s += TG_RELAYS; while (s >= WS) { s -= WS; ph ^= 1; }
            sx += TG_RELAYS; while (sx >= XS) { sx -= XS; phx ^= 1; }
            sd += TG_RELAYS; while (sd >= DS) { sd -= DS; phd ^= 1; }
            sq += TG_RELAYS; while (sq >= DS) { sq -= DS; phq ^= 1; }
        }
        // the MMAs of the steps handed over have read this CTA's shared memory before it leaves
        if (last >= 0) tg_wait(b_done + last * 8, phl, full_limit());
    }
    else if (warp == NDEC + 1)
    {
        // ---- MMA issue: D (128 columns x N tokens) += W^T (128 x 16) x~^T (16 x N). The whole warp walks
        // the loop and one elected lane issues: the operands then stay in uniform registers (a single
        // thread in a divergent branch takes ~100 cycles per tcgen05.mma, this form ~55) ----
        constexpr uint32_t M_FIELD = (uint32_t) ((PAIR ? 256 : TC_BM) >> 4) << 24;
        const uint32_t idesc = (1u << 4) | ((uint32_t) (n16 >> 3) << 17) | M_FIELD, idesc1 = (1u << 4) | ((uint32_t) (n16b >> 3) << 17) | M_FIELD;
        const uint64_t to1 = (uint64_t) ((PAIR ? S.n0 / 2 : S.n0) * 8);
        const uint64_t dw0 = make_desc(smem_u32(smem)), dx0 = make_desc(smem_u32(x_base));
        int s = 0, sx = 0, sd = 0; uint32_t ph = 0, phx = 0, phd = 0;
        for (int i = 0; i < nsteps; ++i)
        {
            wait_bar(b_x + sx * 8, phx);
            wait_bar(b_w + s * 8, ph);
            if constexpr (PAIR)
            {
                if (!tg_wait<true>(b_peer + sd * 8, phd, limit)) { limit = 0; s_bad = 1; }
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t dx = dx0 + (uint64_t) ((sx * x_bytes) >> 4), dwt = dw0 + (uint64_t) ((s * TG_W_BYTES) >> 4);
            if (tg_elect() && limit)
            {
                #pragma unroll
                for (int kk = 0; kk < TC_BK / 16; ++kk) tg_umma<PAIR>(tmem, dwt + 2 * kk, dx + 2 * kk, idesc, (i > 0 || kk > 0) ? 1u : 0u);
                if (rows1 > 0)
                    #pragma unroll
                    for (int kk = 0; kk < TC_BK / 16; ++kk)
                        tg_umma<PAIR>(tmem + TG_MAX_N, dwt + 2 * kk, dx + to1 + 2 * kk, idesc1, (i > 0 || kk > 0) ? 1u : 0u);
                if constexpr (PAIR) tg_commit_both(&done[sd], (unsigned short) (3u << (rank & ~1)));
                else umma_commit(&done[sd]);
            }
            __syncwarp();
            if (limit == 0) continue;
            if (++sd == DS) { sd = 0; phd ^= 1; }
            if (++s == WS) { s = 0; ph ^= 1; }
            if (++sx == XS) { sx = 0; phx ^= 1; }
        }
        // the MMAs of the steps that this CTA issued are done before it leaves (no step at all: the parity passes on the
        // barrier nobody has arrived on)
        tg_wait(b_done + (sd == 0 ? DS - 1 : sd - 1) * 8, sd == 0 ? phd ^ 1 : phd, full_limit());
    }
    else if (warp < NDEC)
    {
        // ---- decode ----
        const int ncol = dw * (16 * NT) + gq;
        // the four 16-byte pieces of a tile this lane stores: rows ncol and ncol + 8 (same swizzle phase),
        // chunks 2 pq and 2 pq + 1
        const uint32_t o0 = sw128(ncol, 2 * pq), o1 = sw128(ncol, 2 * pq + 1);
        uint32_t wst = w_base + grp * TG_W_BYTES, wbar = b_w + grp * 8;          // weight stage and its barrier
        // entry of `done` that frees the stage: step i - WS; the first WS steps find the (passing) parity
        // of a barrier nobody has arrived on yet
        int sd = grp - WS + DS;
        uint32_t phd = 1, publish = 0;                       // publish: barrier of a stage written but not yet handed over
        if (sd >= DS) { sd -= DS; phd = 0; }
        auto hand_over = [&]()
        {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && limit) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(publish) : "memory");
        };
        while (--left >= 0)
        {
            uint32_t w[NT][K];
            #pragma unroll
            for (int c = 0; c < NT; ++c)
                #pragma unroll
                for (int j = 0; j < K; ++j) w[c][j] = next[c][j];
            if (left > 0) fetch_words();
            // is the stage free? (asked now, looked at behind the decode of the first tile)
            const uint32_t free_now = tg_test(b_done + sd * 8, phd);
            // the word in front of this lane's piece: the last word of the lane four below (ring)
            uint32_t prev[NT];
            #pragma unroll
            for (int c = 0; c < NT; ++c) prev[c] = __shfl_sync(0xffffffffu, w[c][K - 1], (lane + 28) & 31);
            #pragma unroll
            for (int c = 0; c < NT; ++c)
            {
                uint32_t colA[8], colB[8];                   // packed pairs (k, k+1): words 0-3 = k 0..7, 4-7 = k 8..15
                auto decode_r = [&](auto rtag)
                {
                    constexpr int R = decltype(rtag)::value;
                    uint32_t st[8];
                    // (codebook 2 already has two instructions per weight on the FMA pipe: its fields are cut on the ALU)
                    products8<K, R, CB, CB != 2, tg_shared_phase<K, CB, GROUPED>>(w[c], prev[c], st);
                    colA[R] = tg_weights2<CB>(st[0], st[1]);     colA[4 + R] = tg_weights2<CB>(st[2], st[3]);
                    colB[R] = tg_weights2<CB>(st[4], st[5]);     colB[4 + R] = tg_weights2<CB>(st[6], st[7]);
                };
                decode_r(std::integral_constant<int, 0>()); decode_r(std::integral_constant<int, 1>());
                decode_r(std::integral_constant<int, 2>()); decode_r(std::integral_constant<int, 3>());
                if (c == 0)
                {
                    // hand over the tile of the previous step: its stores have long completed, so that the proxy
                    // fence costs nothing here (right behind the stores it waits for them, ~150 cycles a step)
                    if (publish) hand_over();
                    if (!free_now) wait_bar(b_done + sd * 8, phd);
                }
                const uint32_t b = wst + c * 2048;
                sts128(b + o0, colA[0], colA[1], colA[2], colA[3]);
                sts128(b + o1, colA[4], colA[5], colA[6], colA[7]);
                sts128(b + o0 + 1024, colB[0], colB[1], colB[2], colB[3]);
                sts128(b + o1 + 1024, colB[4], colB[5], colB[6], colB[7]);
            }
            publish = wbar;
            // (second CTA of a pair: at once, the way to the first CTA's MMA is a microsecond longer)
            if (PAIR && prank != 0) { hand_over(); publish = 0; }
            wst += NGR * TG_W_BYTES; wbar += NGR * 8;
            if (wst >= w_base + WS * TG_W_BYTES) { wst -= WS * TG_W_BYTES; wbar -= WS * 8; }
            sd += NGR;
            if (sd >= DS) { sd -= DS; phd ^= 1; }
        }
        if (publish) hand_over();
    }

    // ---- epilogue ----
    if (warp < NDEC) wait_bar(b_done + ((nsteps - 1) % DS) * 8, (uint32_t) (((nsteps - 1) / DS) & 1));
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (split > 1)
    {
        if constexpr (!PAIR) cluster_wait_started();         // the peers run: their shared memory is written from here on
        // nobody adds up partial sums to which a wait that ran out has contributed (read behind the barrier of the exchange)
        if (s_bad && t < split) tg_st_cluster_u32(cluster_map(smem_u32(const_cast<int*>(&s_bad)), peer_of(t)), 1);
    }
    // ... and they write into this CTA's receive buffer: where it overlaps the stages, everybody's MMAs must have read theirs
    if (split > 1 && S.recv_off == 0) cluster_sync_all();
    const int row = tg_row(split), n0 = S.n0;
    // passes of equal length, each CTA of the cluster finishing TS tokens of a pass
    const int npass = (rows + S.share * split - 1) / (S.share * split);
    const int TS = npass > 1 ? ((rows + npass * split - 1) / (npass * split) + 15) & ~15 : S.share;
    const uint32_t xbuf = smem_u32(smem) + (uint32_t) S.recv_off;             // [split][TS] rows of 128 fp32
    for (int p0 = 0; p0 < rows; p0 += TS * split)
    {
        const int np = min(TS * split, rows - p0);           // tokens of this pass
        if (warp < NDEC)
        {
            // rows of the accumulator (output columns) 32 q .. + 31 belong to the warps with warp % 4 == q
            const int q = warp & 3;
            const uint32_t col = xbuf + (uint32_t) (crank * TS * row + (q * 32 + lane) * 4);
            for (int c0 = (warp >> 2) * 16; c0 < np; c0 += NDEC * 4)
            {
                uint32_t v[16];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                               "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                             : "r"(tmem + ((uint32_t) (32 * q) << 16) + (uint32_t) (p0 + c0 + (NG > 1 && p0 + c0 >= n0 ? TG_MAX_N - n0 : 0))) : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (split == 1)
                {
                    // (a last chunk stores what lies behind its tokens too: the buffer has room for whole chunks)
                    const uint32_t at = col + (uint32_t) (c0 * 528);
                    #pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("st.shared.u32 [%0], %1;" :: "r"(at + (uint32_t) (j * 528)), "r"(v[j]) : "memory");
                    continue;
                }
                int dest = c0 / TS, tl = c0 - dest * TS;
                #pragma unroll
                for (int j = 0; j < 16; ++j)
                {
                    if (c0 + j < np)
                    {
                        const uint32_t a = col + (uint32_t) (tl * row);
                        if (dest == crank) asm volatile("st.shared.u32 [%0], %1;" :: "r"(a), "r"(v[j]) : "memory");
                        else cluster_st_f32(cluster_map(a, peer_of(dest)), __uint_as_float(v[j]));
                    }
                    if (++tl == TS) { tl = 0; ++dest; }
                }
            }
        }
        if (split > 1) cluster_sync_all(); else __syncthreads();
        const int first = crank * TS, nt = min(TS, np - first);              // this CTA's share of the pass (may be empty)
        if (warp < NDEC && !s_bad)
        {
            // four lanes per token, eight tokens per warp in flight
            const int pc = lane & 3, cl = lane >> 2;
            const uint32_t svp = smem_u32(s_svh) + 16 * pc;
            const bool wide = (reinterpret_cast<uintptr_t>(W.c) & 15) == 0;      // (a bundle's outputs may be 8-byte aligned)
            const f32x2 rs = pack_f32x2(kRScale, kRScale);
            #pragma unroll 1
            for (int r0 = warp * 8; r0 < nt; r0 += NDEC * 8)
            {
                const int r = r0 + cl;
                // partial sums of the cluster's CTAs in ascending k order
                uint32_t at_s = xbuf + (uint32_t) (min(r, nt - 1) * row + 32 * pc);
                f32x2 h[16];
                #pragma unroll
                for (int j = 0; j < 8; ++j) lds_f32x2(at_s + (j & 1) * 16 + (j >> 1) * 128, h[2 * j], h[2 * j + 1]);
                for (int i = 1; i < split; ++i)
                {
                    at_s += (uint32_t) (TS * row);
                    #pragma unroll
                    for (int j = 0; j < 8; ++j)
                    {
                        f32x2 u, v;
                        lds_f32x2(at_s + (j & 1) * 16 + (j >> 1) * 128, u, v);
                        h[2 * j] = add_f32x2(h[2 * j], u); h[2 * j + 1] = add_f32x2(h[2 * j + 1], v);
                    }
                }
                quad_had128(h, pc);
                if (r >= nt) continue;
                const size_t at = (size_t) (m0 + p0 + first + r) * W.n_row + (size_t) nb * 128 + 8 * pc;
                #pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    uint4 sv;
                    lds128(svp + 64 * j, sv.x, sv.y, sv.z, sv.w);
                    const __half2* s2 = reinterpret_cast<const __half2*>(&sv);
                    float2 v[4];
                    #pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = unpack_f32x2(mul_f32x2(h[4 * j + q], rs));
                    if (P.c_fp32)
                    {
                        float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(W.c) + at + 32 * j);
                        o[0] = make_float4(v[0].x * __low2float(s2[0]), v[0].y * __high2float(s2[0]), v[1].x * __low2float(s2[1]), v[1].y * __high2float(s2[1]));
                        o[1] = make_float4(v[2].x * __low2float(s2[2]), v[2].y * __high2float(s2[2]), v[3].x * __low2float(s2[3]), v[3].y * __high2float(s2[3]));
                    }
                    else
                    {
                        uint4 o;
                        __half2* o2 = reinterpret_cast<__half2*>(&o);
                        #pragma unroll
                        for (int q = 0; q < 4; ++q) o2[q] = __hmul2(__float22half2_rn(v[q]), s2[q]);
                        __half* dst = reinterpret_cast<__half*>(W.c) + at + 32 * j;
                        if (wide) *reinterpret_cast<uint4*>(dst) = o;
                        else { reinterpret_cast<uint2*>(dst)[0] = make_uint2(o.x, o.y); reinterpret_cast<uint2*>(dst)[1] = make_uint2(o.z, o.w); }
                    }
                }
            }
        }
        if (p0 + TS * split < rows) { if (split > 1) cluster_sync_all(); else __syncthreads(); }
    }

    if (t == 0 && s_bad) atomicExch(P.status, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR)
    {
        cluster_sync_all();                                  // neither CTA leaves while the other may still use its memory
        if (warp == NDEC)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t) S.tmem_cols) : "memory");
    }
    else if (warp == NDEC)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t) S.tmem_cols) : "memory");
}

typedef void (*tg_fn)(const TgParams);
enum { TG_DENSE = 0, TG_GROUPED = 1, TG_PAIR = 2 };
// kernel of a bit width and codebook: dense, 16 decode warps; expert groups, 8 warps and two CTAs per SM; dense CTA pairs
tg_fn tg_kernel(int K, int cb, int form);

}  // namespace amp
