// Trellis GEMM for short batches and expert groups: C (M, n) = x~ (M, k) @ W_hat (k, n) -> Hadamard -> * svh
// with the DECODED WEIGHTS as the M operand of tcgen05.mma (128 output columns) and the tokens as the N
// operand (16 .. 256 per tile). A weight is decoded once per tile of up to 256 tokens, the x~ tile of a
// step is only as tall as the batch, and k is split over the CTAs of a thread-block cluster so that a
// small matrix still spreads over the device.
//
// What bounds it: the decode (about 5.5 instructions per weight; ~18 weights per clock and SM is the
// issue limit) up to a few hundred tokens, the tensor pipe above. The token-major kernels of
// exl3_gemm_tc.cu cannot reach that at these sizes: their k loop is a chain of barrier hand-overs of
// about 0.6 us per 64-row step that is k / 64 steps long whatever the batch, and at 4096 columns only
// 32 CTAs share the work.
//
// One CTA = 128 output columns x one token tile x one slice of k. Warps 0 .. 8 NG - 1 decode, in groups
// of four that take alternate 64-row steps (a warp owns two 16-column tile columns); one thread
// fetches x~ with bulk copies, one issues the MMAs. A stage holds the x~ tile and the weight tile of a
// step and is freed by one tcgen05.commit. Several CTAs share an SM (tensor-memory columns and shared
// memory are sized by the tile), so that one CTA's set-up, waits and epilogue run under another's decode.
//
// Epilogue: the accumulator's rows are output columns, its columns tokens. Every CTA lays its partial sums out
// token by token in its own shared memory and sends every CTA of the cluster the run of tokens that one
// finishes; there four lanes per token add the partials in ascending k order (bitwise reproducible), run the 128-point
// Hadamard, scale and store. Every mbarrier wait is bounded as in the other kernels.
#pragma once
#include "exl3_gemm_tc.cuh"

namespace amp {

constexpr int SH_MAX_N = 256;                 // tokens per accumulator (UMMA N)
constexpr int SH_MAX_TOKENS = 512;            // tokens per tile: two accumulators, with 16 decode warps only
constexpr int SH_MAX_STAGES = 16;
// bytes of a token's 128 partial sums in the epilogue: 16 of padding make the reads conflict-free; rows sent to a
// peer stay on 128-byte lines instead
__host__ __device__ constexpr int sh_row(int split) { return split > 1 ? 512 : 528; }
constexpr int SH_W_BYTES = TC_BN * TC_BK * 2; // decoded weights of a step: 16384

struct ShParams
{
    TcParams t;                 // pointers, sizes, bundle tables, expert tile table
    int tile;                   // tokens per tile: a multiple of 16, at most 512
    int n0;                     // tokens of the first accumulator: a multiple of 16, at most 256 (the rest: the second, at column 256)
    int split;                  // CTAs per cluster = slices of k (1: no cluster)
    int wstages, xstages;       // stages of decoded weights and of x~: wstages >= 2 NG
    int x_area;                 // expert groups: bytes of all x~ stages together (xstages then follows from the tile's rows)
    int tmem_cols;              // tensor-memory columns to allocate: a power of two >= tile, >= 32 (two accumulators: 512)
    int share;                  // tokens a CTA finishes per epilogue pass (several passes: a multiple of 8)
    int recv_off;               // where the partial sums are received: behind the stages, or 0: over them
    int pdl;                    // launched as a programmatic dependent of the kernel that writes x~
};

// warps that decode a step together (each 8 / 4 = 2 of the eight 16-column tiles of the block): per step a warp
// pays about 60 instructions of bookkeeping, so that it should not be shorter
constexpr int SH_GROUP_WARPS = 4;
__host__ __device__ constexpr int sh_threads(int ng) { return 32 * (8 * ng + 2); }

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

__device__ __forceinline__ void lds128f(uint32_t addr, float2& a, float2& b)
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(b.x), "=f"(b.y) : "r"(addr) : "memory");
}

// Two states -> two exact fp16 weights, packed. As weights2, with the halves of each word added by one
// instruction per weight on the half-precision pipe and one byte permute per pair (weights2: two permutes
// and one addition): the integer ALU is the busier pipe.
template <int CB>
__device__ __forceinline__ uint32_t sh_weights2(uint32_t sa, uint32_t sb)
{
    if constexpr (CB == 2) return weights2<2>(sa, sb);
    else
    {
        const uint32_t ya = cb_halves<CB>(sa), yb = cb_halves<CB>(sb);
        const __half2 ha = *reinterpret_cast<const __half2*>(&ya), hb = *reinterpret_cast<const __half2*>(&yb);
        const __half2 wa = __hadd2(__low2half2(ha), __high2half2(ha)), wb = __hadd2(__low2half2(hb), __high2half2(hb));
        return __byte_perm(*reinterpret_cast<const uint32_t*>(&wa), *reinterpret_cast<const uint32_t*>(&wb), 0x5410);
    }
}

// Whole-warp wait for an mbarrier phase, bounded, as straight-line code: the usual case (already there) is
// one instruction and a branch not taken. Returns false when `limit` polls were not enough.
__device__ __forceinline__ bool sh_wait(uint32_t bar, uint32_t parity, uint32_t limit)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra $SH_DONE_%=;\n\t"
        "mov.u32 n, %3;\n"
        "$SH_POLL_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra $SH_DONE_%=;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 q, n, 0;\n\t"
        "@q bra $SH_POLL_%=;\n"
        "$SH_DONE_%=:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r) : "r"(bar), "r"(parity), "r"(limit) : "memory");
    return r != 0;
}

// one look at an mbarrier phase
__device__ __forceinline__ uint32_t sh_test(uint32_t bar, uint32_t parity)
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r) : "r"(bar), "r"(parity) : "memory");
    return r;
}

// one lane of the (converged) warp
__device__ __forceinline__ bool sh_elect()
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}

__device__ __forceinline__ void sh_umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ uint32_t sh_cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

template <int K, int CB, int NG, bool GROUPED>
__global__ __launch_bounds__(sh_threads(NG), NG == 1 ? 2 : 1)
void exl3_gemm_short_kernel(const ShParams S)
{
    const TcParams& P = S.t;
    if constexpr (GROUPED)
    {
        // the whole CTA leaves, before any barrier or allocation
        if ((int) blockIdx.y >= *P.g_ntiles || P.g_tile_rows[blockIdx.y] <= 0) return;
        const unsigned char* bits = P.g_bits[(int) blockIdx.x / (P.n / TC_BN)];
        if (bits && bits[P.g_tile_e[blockIdx.y]] != K) return;
    }
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw;
    if (smem_u32(smem_raw) & 1023)                           // (the swizzle needs the alignment the declaration asks for)
    {
        if (threadIdx.x == 0) atomicExch(P.status, 2);
        return;
    }
    __shared__ uint64_t x_full[SH_MAX_STAGES], w_full[SH_MAX_STAGES], done[SH_MAX_STAGES];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_bad;
    constexpr int NDEC = 8 * NG, NGR = NDEC / SH_GROUP_WARPS;    // decode warps; groups of them that take alternate steps

    const int t = threadIdx.x, lane = t & 31, warp = __shfl_sync(0xffffffffu, t >> 5, 0);
    const int split = GROUPED ? 1 : S.split;
    const int crank = split > 1 ? (int) sh_cluster_rank() : 0;
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
        W = tc_slice<TC_BN>(P, (int) blockIdx.x / split);
        m0 = (int) blockIdx.y * S.tile;
        rows = min(S.tile, P.M - m0);
    }
    const int nb = W.nb;
    const int ksteps = P.k / TC_BK;
    const int ks0 = ksteps * crank / split, nsteps = ksteps * (crank + 1) / split - ks0;     // (split <= ksteps: never empty)
    const size_t tiles_n = (size_t) W.n_row >> 4;
    // expert groups: the x~ stages are as tall as this tile, so that short tiles get more of them
    const int x_bytes = (GROUPED ? (rows + 15) & ~15 : S.tile) * (TC_BK * 2);
    const int WS = S.wstages, XS = GROUPED ? min(SH_MAX_STAGES, S.x_area / x_bytes) : S.xstages, DS = max(WS, XS);
    unsigned char* x_base = smem + WS * SH_W_BYTES;

    if (t == 0)
    {
        // done[i % DS]: the MMAs of step i have completed -- one commit per step frees the x~ stage and the
        // weight stage of step i; who waits for step i - XS or i - WS finds it in this ring
        for (int i = 0; i < XS; ++i) mbar_init(&x_full[i], 1);
        for (int i = 0; i < DS; ++i) mbar_init(&done[i], 1);
        for (int i = 0; i < WS; ++i) mbar_init(&w_full[i], SH_GROUP_WARPS);
        fence_mbar_init();
        s_bad = 0;
    }
    __syncwarp();
    if (warp == NDEC)
    {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&s_tmem)), "r"((uint32_t) S.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // The decode warps' packed words go straight into registers, one step ahead of their use (two: no gain). (Not through
    // cp.async rings: the release of a step's barrier waits for the warp's copies in flight, so that every
    // step paid the HBM latency -- 1.1 us per step and warp, 20 us for 77 x 4096 x 4096 at 4 bits.)
    constexpr int GW = SH_GROUP_WARPS, NT = 8 / GW;
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
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    // After a wait that ran out, later waits give up at once: the roles run on over stale data to their end
    // (nothing is stored) and every barrier below is still reached.
    unsigned limit = TC_SPIN_LIMIT;
    auto wait_bar = [&](uint32_t bar, uint32_t parity)
    {
        if (!sh_wait(bar, parity, limit)) { limit = 1; s_bad = 1; }
    };
    const uint32_t w_base = smem_u32(smem), b_x = smem_u32(x_full), b_w = smem_u32(w_full), b_done = smem_u32(done);

    if (warp == NDEC)
    {
        // ---- fetch ----
        if (S.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");          // x~ comes from the kernel in front
        // entry of `done` that frees the stage of step i: step i - XS; the first XS steps find the (passing)
        // parity of a barrier nobody has arrived on yet
        int s = 0, sd = DS - XS; uint32_t phd = 1;
        if (sd == DS) { sd = 0; phd = 0; }
        const unsigned char* xs = W.xt + (((size_t) ks0 * P.M + m0) << 7);
        for (int i = 0; i < nsteps; ++i)
        {
            wait_bar(b_done + sd * 8, phd);
            if (sh_elect())
            {
                // (rows beyond the batch stay stale: their accumulator columns are never read)
                mbar_expect_tx(&x_full[s], (uint32_t) rows * 128);
                bulk_g2s(x_base + s * x_bytes, xs, (uint32_t) rows * 128, &x_full[s]);
            }
            xs += (size_t) P.M << 7;
            if (++s == XS) s = 0;
            if (++sd == DS) { sd = 0; phd ^= 1; }
        }
        __syncwarp();
    }
    else if (warp == NDEC + 1)
    {
        // ---- MMA issue: D (128 columns x N tokens) += W^T (128 x 16) x~^T (16 x N). The whole warp walks
        // the loop and one elected lane issues: the operands then stay in uniform registers (a single
        // thread in a divergent branch takes ~100 cycles per tcgen05.mma, this form ~55) ----
        const int rows1 = NG > 1 ? rows - S.n0 : 0;         // tokens of the second accumulator
        const uint32_t n16 = (uint32_t) (min(rows, S.n0) + 15) & ~15u, n16b = rows1 > 0 ? (uint32_t) (rows1 + 15) & ~15u : 16u;
        const uint32_t idesc = (1u << 4) | ((n16 >> 3) << 17) | ((uint32_t) (TC_BM >> 4) << 24);
        const uint32_t idesc1 = (1u << 4) | ((n16b >> 3) << 17) | ((uint32_t) (TC_BM >> 4) << 24);
        const uint64_t dw0 = make_desc(smem_u32(smem)), dx0 = make_desc(smem_u32(x_base));
        int s = 0, sx = 0, sd = 0; uint32_t ph = 0, phx = 0;
        for (int i = 0; i < nsteps; ++i)
        {
            wait_bar(b_x + sx * 8, phx);
            wait_bar(b_w + s * 8, ph);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t dx = dx0 + (uint64_t) ((sx * x_bytes) >> 4), dwt = dw0 + (uint64_t) ((s * SH_W_BYTES) >> 4);
            if (sh_elect())
            {
                #pragma unroll
                for (int kk = 0; kk < TC_BK / 16; ++kk) sh_umma(tmem, dwt + 2 * kk, dx + 2 * kk, idesc, (i > 0 || kk > 0) ? 1u : 0u);
                if (rows1 > 0)
                    #pragma unroll
                    for (int kk = 0; kk < TC_BK / 16; ++kk)
                        sh_umma(tmem + SH_MAX_N, dwt + 2 * kk, dx + (uint64_t) (S.n0 * 8) + 2 * kk, idesc1, (i > 0 || kk > 0) ? 1u : 0u);
                umma_commit(&done[sd]);
            }
            __syncwarp();
            if (++sd == DS) sd = 0;
            if (++s == WS) { s = 0; ph ^= 1; }
            if (++sx == XS) { sx = 0; phx ^= 1; }
        }
    }
    else
    {
        // ---- decode ----
        const int ncol = dw * (16 * NT) + gq;
        // the four 16-byte pieces of a tile this lane stores: rows ncol and ncol + 8 (same swizzle phase),
        // chunks 2 pq and 2 pq + 1
        const uint32_t o0 = sw128(ncol, 2 * pq), o1 = sw128(ncol, 2 * pq + 1);
        uint32_t wst = w_base + grp * SH_W_BYTES, wbar = b_w + grp * 8;          // weight stage and its barrier
        // entry of `done` that frees the stage: step i - WS; the first WS steps find the (passing) parity
        // of a barrier nobody has arrived on yet
        int sd = grp - WS + DS;
        uint32_t phd = 1, publish = 0;                       // publish: barrier of a stage written but not yet handed over
        if (sd >= DS) { sd -= DS; phd = 0; }
        auto hand_over = [&]()
        {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(publish) : "memory");
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
            const uint32_t free_now = sh_test(b_done + sd * 8, phd);
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
                    states8<K, R, CB != 2>(w[c], prev[c], st);
                    colA[R] = sh_weights2<CB>(st[0], st[1]);     colA[4 + R] = sh_weights2<CB>(st[2], st[3]);
                    colB[R] = sh_weights2<CB>(st[4], st[5]);     colB[4 + R] = sh_weights2<CB>(st[6], st[7]);
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
            wst += NGR * SH_W_BYTES; wbar += NGR * 8;
            if (wst >= w_base + WS * SH_W_BYTES) { wst -= WS * SH_W_BYTES; wbar -= WS * 8; }
            sd += NGR;
            if (sd >= DS) { sd -= DS; phd ^= 1; }
        }
        if (publish) hand_over();
    }

    // ---- epilogue ----
    if (warp < NDEC) wait_bar(b_done + ((nsteps - 1) % DS) * 8, (uint32_t) (((nsteps - 1) / DS) & 1));
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // peers write into this CTA's receive buffer from here on: where it overlaps the stages, everybody's MMAs
    // must have read theirs
    if (split > 1 && S.recv_off == 0) cluster_sync_all();
    const int row = sh_row(split), n0 = S.n0, TS = S.share;                                  // tokens this CTA finishes per pass
    const uint32_t xbuf = smem_u32(smem) + (uint32_t) S.recv_off;             // [split][TS] rows of 128 fp32
    for (int p0 = 0; p0 < rows; p0 += TS * split)
    {
        const int np = min(TS * split, rows - p0);           // tokens of this pass
        if (warp < NDEC)
        {
            // rows of the accumulator (output columns) 32 q .. + 31 belong to the warps with warp % 4 == q
            const int q = warp & 3;
            const uint32_t col = xbuf + (uint32_t) (crank * TS * row + (q * 32 + lane) * 4);
            for (int c0 = (warp >> 2) * 8; c0 < np; c0 += NDEC * 2)
            {
                uint32_t v[8];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                             : "r"(tmem + ((uint32_t) (32 * q) << 16) + (uint32_t) (p0 + c0 + (NG > 1 && p0 + c0 >= n0 ? SH_MAX_N - n0 : 0))) : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (split == 1)
                {
                    #pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c0 + j < np) asm volatile("st.shared.u32 [%0], %1;" :: "r"(col + (uint32_t) ((c0 + j) * row)), "r"(v[j]) : "memory");
                    continue;
                }
                int dest = c0 / TS, tl = c0 - dest * TS;
                #pragma unroll
                for (int j = 0; j < 8; ++j)
                {
                    if (c0 + j < np)
                    {
                        const uint32_t a = col + (uint32_t) (tl * row);
                        if (dest == crank) asm volatile("st.shared.u32 [%0], %1;" :: "r"(a), "r"(v[j]) : "memory");
                        else cluster_st_f32(cluster_map(a, (uint32_t) dest), __uint_as_float(v[j]));
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
            const __half* svp = W.svh + (size_t) nb * 128 + 8 * pc;
            const bool wide = (reinterpret_cast<uintptr_t>(W.c) & 15) == 0;      // (a bundle's outputs may be 8-byte aligned)
            for (int r0 = warp * 8; r0 < nt; r0 += NDEC * 8)
            {
                const int r = r0 + cl;
                // partial sums of the cluster's CTAs in ascending k order
                uint32_t at_s = xbuf + (uint32_t) (min(r, nt - 1) * row + 32 * pc);
                float2 h[16];
                #pragma unroll
                for (int j = 0; j < 8; ++j) lds128f(at_s + (j & 1) * 16 + (j >> 1) * 128, h[2 * j], h[2 * j + 1]);
                for (int i = 1; i < split; ++i)
                {
                    at_s += (uint32_t) (TS * row);
                    #pragma unroll
                    for (int j = 0; j < 8; ++j)
                    {
                        float2 u, v;
                        lds128f(at_s + (j & 1) * 16 + (j >> 1) * 128, u, v);
                        h[2 * j] = add_f32x2(h[2 * j], u); h[2 * j + 1] = add_f32x2(h[2 * j + 1], v);
                    }
                }
                quad_had128(h, pc);
                if (r >= nt) continue;
                const size_t at = (size_t) (m0 + p0 + first + r) * W.n_row + (size_t) nb * 128 + 8 * pc;
                #pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    // (scale vectors are 8-byte aligned)
                    const uint2 sv[2] = { *reinterpret_cast<const uint2*>(svp + 32 * j), *reinterpret_cast<const uint2*>(svp + 32 * j + 4) };
                    const __half2* s2 = reinterpret_cast<const __half2*>(sv);
                    float2* v = h + 4 * j;
                    #pragma unroll
                    for (int q = 0; q < 4; ++q) { v[q].x *= kRScale; v[q].y *= kRScale; }
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
                        for (int q = 0; q < 4; ++q) o2[q] = __hmul2(__floats2half2_rn(v[q].x, v[q].y), s2[q]);
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
    if (warp == NDEC)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t) S.tmem_cols) : "memory");
}

typedef void (*sh_fn)(const ShParams);
// kernel of a bit width and codebook. grouped 0: dense, 16 decode warps; 1: expert groups, 8 warps and two CTAs per SM
sh_fn sh_kernel(int K, int cb, int grouped);

}  // namespace amp
