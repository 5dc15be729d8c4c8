// Host side of the short-batch trellis GEMM (exl3_gemm_short.cuh): tile, split and stage choice, launch.
#include "exl3_gemm_short.cuh"
#include <mutex>

namespace amp {

#define AMP_DECL(K) sh_fn sh_kernel_k##K(int cb, int grouped);
AMP_DECL(1) AMP_DECL(2) AMP_DECL(3) AMP_DECL(4) AMP_DECL(5) AMP_DECL(6) AMP_DECL(7) AMP_DECL(8)
#undef AMP_DECL

sh_fn sh_kernel(int K, int cb, int grouped)
{
    switch (K)
    {
        case 1: return sh_kernel_k1(cb, grouped);
        case 2: return sh_kernel_k2(cb, grouped);
        case 3: return sh_kernel_k3(cb, grouped);
        case 4: return sh_kernel_k4(cb, grouped);
        case 5: return sh_kernel_k5(cb, grouped);
        case 6: return sh_kernel_k6(cb, grouped);
        case 7: return sh_kernel_k7(cb, grouped);
        default: return sh_kernel_k8(cb, grouped);
    }
}

int g_short_split = 0, g_short_tile = 0;      // forced (0: by rule), see amp_exl3_set_gemm_short

constexpr int SH_STATIC = 1024;          // static shared memory of the kernel (its dynamic part is 1024-byte aligned)

static int sh_smem(int tile, int ws, int xs)
{
    return ws * SH_W_BYTES + xs * tile * TC_BK * 2;
}

// Memory plan of one tile height and number of decode groups: stages, tensor-memory columns, tokens per
// accumulator. Returns the dynamic shared memory, 0 where it does not fit.
static int sh_layout(ShParams& S, int tile, int ng)
{
    if (tile > (ng == 1 ? SH_MAX_N : SH_MAX_TOKENS)) return 0;
    S.tile = tile;
    S.n0 = tile > SH_MAX_N ? ((tile + 1) / 2 + 15) & ~15 : tile;
    int cols = 32;
    while (cols < tile) cols <<= 1;
    S.tmem_cols = cols > SH_MAX_N ? 512 : cols;
    const int budget = 228 * 1024 / (ng == 1 ? 2 : 1) - 1024 - SH_STATIC;             // two CTAs per SM / one
    // weights are handed over a step or two behind their decode; x~ comes from L2 and wants the depth
    int ws = ng == 1 ? 3 : 5, xs = 2;
    while (ws > 2 * ng && sh_smem(tile, ws, xs) > budget) --ws;
    if (sh_smem(tile, ws, xs) > budget) return 0;
    while (xs < SH_MAX_STAGES && sh_smem(tile, ws, xs + 1) <= budget) ++xs;
    S.wstages = ws; S.xstages = xs;
    return sh_smem(tile, ws, xs);
}

// Tokens a CTA finishes per epilogue pass and where their partial sums ((source, token) rows of 512 bytes) are
// received: behind the stages where that leaves three x~ stages (no barrier between the k loop and the exchange
// then), else over the stages, in several passes if need be. Returns the dynamic shared memory.
static int sh_exchange(ShParams& S, int smem)
{
    int ts = (S.tile + S.split - 1) / S.split;
    S.recv_off = 0;
    if (S.split > 1)
    {
        const int budget = smem - sh_smem(S.tile, S.wstages, 0), recv = S.split * ts * sh_row(S.split), x = S.tile * TC_BK * 2;
        const int left = (budget - recv) / x;
        if (budget > recv && left >= 3)
        {
            S.xstages = left < S.xstages ? left : S.xstages;
            S.recv_off = S.wstages * SH_W_BYTES + S.xstages * x;
        }
    }
    const int room = smem / sh_row(S.split);
    if (!S.recv_off && ts * S.split > room) ts = room / S.split & ~7;
    S.share = ts;
    return S.recv_off ? sh_smem(S.tile, S.wstages, S.xstages) + S.split * ts * sh_row(S.split) : smem;
}

// Clusters of c CTAs (one CTA per SM) the device holds at once: the SMs of a GPC come in no multiple of c
static int sh_max_clusters(int c, int sms, int dev)
{
    static int table[64][9] = {};
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    int& v = table[dev & 63][c];
    if (!v)
    {
        const int smem = 227 * 1024 - SH_STATIC;
        sh_fn fn = sh_kernel(4, 0, 0);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned) (c * sms), 1, 1);
        cfg.blockDim = dim3(sh_threads(2), 1, 1);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = c; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (ensure_smem(fn, smem, dev) || cudaOccupancyMaxActiveClusters(&n, fn, &cfg) || n < 1) { cudaGetLastError(); n = sms / c > 1 ? sms / c - 1 : 1; }
        v = n;
    }
    return v;
}

// Tile height, decode groups and k split for M rows x `blocks` column blocks: the cheapest by a model of the
// measured times (us). A 64-row step takes the slowest of the decode (0.40 per 8192 weights), the tensor pipe (0.28
// per 256 tokens) and the x~ tiles of all CTAs out of L2 (8.5 TB/s); a CTA costs 4 + 0.02 per token around its k
// loop, the exchange of a split 1.5 and 0.035 (clusters of more than four: 0.07) per token that crosses to a peer.
// One CTA of sixteen decode warps per SM: two of eight take as long per step and longer per exchange.
static int sh_plan(ShParams& S, int M, long blocks, int ksteps, int sms, int dev, double limit)
{
    double best = limit;
    int best_smem = 0;
    ShParams T = S;
    for (int tiles = (M + SH_MAX_TOKENS - 1) / SH_MAX_TOKENS; tiles <= (M + 127) / 128; ++tiles)
    {
        const int smem = sh_layout(T, g_short_tile ? g_short_tile : ((M + tiles - 1) / tiles + 15) & ~15, 2), xs = T.xstages;
        if (!smem) continue;
        for (int c = 1; c <= 8 && c <= ksteps; ++c)
        {
            T.split = c;
            T.xstages = xs;
            if (g_short_split && c != g_short_split) continue;
            const int need = sh_exchange(T, smem);
            if (T.share < 1) continue;
            const long clusters = blocks * ((M + T.tile - 1) / T.tile), fit = c > 1 ? sh_max_clusters(c, sms, dev) : sms;
            const long waves = (clusters + fit - 1) / fit, live = c * (clusters < fit ? clusters : fit);
            const double mma = 0.28 * T.tile / 256, l2 = T.tile * 128.0 * live / 8.5e6;
            const double step = mma > l2 ? (mma > 0.40 ? mma : 0.40) : (l2 > 0.40 ? l2 : 0.40);
            const double cost = waves * ((double) ((ksteps + c - 1) / c) * step + 4.0 + 0.02 * T.tile
                                         + (c > 1 ? 1.5 + (c > 4 ? 0.07 : 0.035) * T.tile * (c - 1) / c : 0.0));
            if (cost < best * 0.99) { best = cost; best_smem = need; S = T; }
        }
    }
    return best_smem;
}

int launch_gemm_short(const TcParams& P, int K, int cb, long blocks, int sms, int dev, double limit, cudaStream_t stream)
{
    ShParams S = {};
    S.t = P;
    S.pdl = g_pdl;
    const int smem = sh_plan(S, P.M, blocks, P.k / TC_BK, sms, dev, limit);
    if (!smem) return AMP_E_UNSUPPORTED;
    sh_fn fn = sh_kernel(K, cb, 0);
    if (cudaError_t e = ensure_smem(fn, smem, dev)) return cuda_rc(e, "exl3_gemm_short smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (blocks * S.split), (unsigned) ((P.M + S.tile - 1) / S.tile), 1);
    cfg.blockDim = dim3(sh_threads(2), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (S.split > 1)
    {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = S.split; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (g_pdl)
    {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return cuda_rc(cudaLaunchKernelEx(&cfg, fn, S), "exl3_gemm_short launch");
}

// Expert-grouped form for token-sorted MoE prefill: xt / c are (kinds, Mcap, k / n) in the padded, expert-sorted row
// space, the tile table lives in device memory (see TcParams). One CTA per (tile, projection, 128-column block); the
// grid is sized for G.max_tiles and the surplus returns. Eight decode warps and two CTAs per SM, so that one CTA's
// set-up and epilogue run under the other's decode.
int launch_gemm_short_grouped(const void* xt, void* c, long Mcap, int k, int n, int K, int cb, int c_fp32,
                              const long long* t_trellis, const long long* t_svh, const TcGroups& G, cudaStream_t stream)
{
    AMP_REQUIRE(xt && c && t_trellis && t_svh && G.ntiles && G.tile_e && G.tile_row0 && G.tile_rows, "exl3_moe_sorted: null pointer");
    AMP_REQUIRE(K >= 1 && K <= 8 && cb >= 0 && cb <= 2, "exl3_moe_sorted: unsupported bitrate / codebook");
    AMP_REQUIRE(Mcap >= 1 && Mcap <= 0x7fffffffL && k % 128 == 0 && n % 128 == 0 && k > 0 && n > 0, "exl3_moe_sorted: k and n must be multiples of 128");
    AMP_REQUIRE(((uintptr_t) xt & 15) == 0 && ((uintptr_t) c & 15) == 0, "exl3_moe_sorted: misaligned pointer");
    AMP_REQUIRE(G.kinds >= 1 && G.kinds <= 2 && G.tile >= 16 && G.tile <= SH_MAX_N && G.tile % 16 == 0 && G.experts >= 1, "exl3_moe_sorted: bad grouping");
    AMP_REQUIRE(G.max_tiles >= 1 && G.max_tiles <= 65535, "exl3_moe_sorted: too many row tiles");
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return cuda_rc(e, "cudaGetDevice");
    ShParams S = {};
    const int smem = sh_layout(S, G.tile, 1);
    AMP_REQUIRE(smem, "exl3_moe_sorted: tile does not fit");
    S.x_area = smem - sh_smem(G.tile, S.wstages, 0);
    S.split = 1;
    S.share = smem / sh_row(1) & ~7;
    // Dependent launch only where every grid that does anything waits for the rotation kernel: with one launch per
    // bit width a launch whose experts all have another width would be over before that kernel, and the next
    // launch's wait would be for it alone.
    S.pdl = g_pdl && !G.bits[0];
    TcParams& P = S.t;
    P.xt = (const unsigned char*) xt; P.c = c;
    P.M = (int) Mcap; P.k = k; P.n = n; P.c_fp32 = c_fp32;
    P.t_trellis = t_trellis; P.t_svh = t_svh;
    P.g_ntiles = G.ntiles; P.g_tile_e = G.tile_e; P.g_tile_row0 = G.tile_row0; P.g_tile_rows = G.tile_rows;
    P.g_experts = G.experts;
    P.g_bits[0] = G.bits[0]; P.g_bits[1] = G.bits[1];
    if (int rc = tc_status_ptr(dev, &P.status)) return rc;
    sh_fn fn = sh_kernel(K, cb, 1);
    if (cudaError_t e = ensure_smem(fn, smem, dev)) return cuda_rc(e, "exl3_moe_sorted smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (G.kinds * (n / 128)), (unsigned) G.max_tiles, 1);
    cfg.blockDim = dim3(sh_threads(1), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = S.pdl ? 1 : 0;
    return cuda_rc(cudaLaunchKernelEx(&cfg, fn, S), "exl3_moe_sorted gemm launch");
}

}  // namespace amp
