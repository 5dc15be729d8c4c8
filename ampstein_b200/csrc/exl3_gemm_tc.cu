// Host side of the tensor-core trellis GEMM (exl3_gemm_tc.cuh): form, tile, split and stage choice, launch.
#include "exl3_gemm_tc.cuh"
#include <mutex>

namespace amp {

__device__ int g_tc_status;
int g_tc_pair = 1;                            // see amp_exl3_set_gemm_pair
unsigned g_tc_wait[2] = { TC_SPIN_LIMIT, TC_SPIN_LIMIT };       // see amp_exl3_set_gemm_wait_limit
int g_tc_split = 0, g_tc_tile = 0;            // forced (0: by rule), see amp_exl3_set_gemm_plan

// address of the status word, looked up once per device (under a lock: two host threads may make their first launch
// on a device at the same time)
static int tc_status_ptr(int dev, int** out)
{
    static int* ptr[64] = {};
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    int*& p = ptr[dev & 63];
    if (!p)
        if (cudaError_t e = cudaGetSymbolAddress((void**) &p, g_tc_status)) return cuda_rc(e, "status symbol");
    *out = p;
    return 0;
}

#define AMP_DECL(K) tg_fn tg_kernel_k##K(int cb, int form);
AMP_DECL(1) AMP_DECL(2) AMP_DECL(3) AMP_DECL(4) AMP_DECL(5) AMP_DECL(6) AMP_DECL(7) AMP_DECL(8)
#undef AMP_DECL

tg_fn tg_kernel(int K, int cb, int form)
{
    switch (K)
    {
        case 1: return tg_kernel_k1(cb, form);
        case 2: return tg_kernel_k2(cb, form);
        case 3: return tg_kernel_k3(cb, form);
        case 4: return tg_kernel_k4(cb, form);
        case 5: return tg_kernel_k5(cb, form);
        case 6: return tg_kernel_k6(cb, form);
        case 7: return tg_kernel_k7(cb, form);
        default: return tg_kernel_k8(cb, form);
    }
}


constexpr int TG_STATIC = 1024;          // static shared memory of the kernel (its dynamic part is 1024-byte aligned)

// x_rows: rows of an x~ stage (the tile's, or half of them in a pair)
static int tg_smem(int x_rows, int ws, int xs)
{
    return ws * TG_W_BYTES + xs * x_rows * TC_BK * 2;
}

// Memory plan of one tile height and number of decode groups: stages, tensor-memory columns, tokens per
// accumulator. Returns the dynamic shared memory, 0 where it does not fit.
static int tg_layout(TgParams& S, int tile, int ng, bool pair = false)
{
    if (tile > (ng == 1 ? TG_MAX_N : TG_MAX_TOKENS)) return 0;
    S.tile = tile;
    S.n0 = tile > TG_MAX_N ? ((tile + 1) / 2 + 15) & ~15 : tile;
    int cols = 32;
    while (cols < tile) cols <<= 1;
    S.tmem_cols = cols > TG_MAX_N ? 512 : cols;
    const int budget = 228 * 1024 / (ng == 1 ? 2 : 1) - 1024 - TG_STATIC;             // two CTAs per SM / one
    // weights are handed over a step or two behind their decode; x~ comes from L2 and wants the depth
    int ws = ng == 1 ? 3 : 5, xs = 2;
    const int xr = pair ? tile / 2 : tile;
    while (ws > 2 * ng && tg_smem(xr, ws, xs) > budget) --ws;
    if (tg_smem(xr, ws, xs) > budget) return 0;
    while (xs < TG_MAX_STAGES && tg_smem(xr, ws, xs + 1) <= budget) ++xs;
    S.wstages = ws; S.xstages = xs;
    return tg_smem(xr, ws, xs);
}

// Tokens a CTA finishes per epilogue pass and where their partial sums ((source, token) rows of 512 bytes) are
// received: behind the stages where that leaves three x~ stages (no barrier between the k loop and the exchange
// then), else over the stages, in several passes if need be. Returns the dynamic shared memory.
static int tg_exchange(TgParams& S, int smem, bool pair)
{
    const int xr = pair ? S.tile / 2 : S.tile;
    int ts = (S.tile + S.split - 1) / S.split;
    S.recv_off = 0;
    if (S.split > 1)
    {
        const int budget = smem - tg_smem(0, S.wstages, 0), recv = S.split * ts * tg_row(S.split), x = xr * TC_BK * 2;
        const int left = (budget - recv) / x;
        if (budget > recv && left >= 3)
        {
            S.xstages = left < S.xstages ? left : S.xstages;
            S.recv_off = S.wstages * TG_W_BYTES + S.xstages * x;
        }
    }
    const int room = smem / tg_row(S.split);
    if (!S.recv_off && ts * S.split > room) ts = room / S.split & ~15;
    S.share = ts;
    return S.recv_off ? tg_smem(xr, S.wstages, S.xstages) + S.split * ts * tg_row(S.split) : smem;
}

// Clusters of c CTAs (one CTA per SM) the device holds at once: the SMs of a GPC come in no multiple of c
static int tg_max_clusters(int c, int sms, int dev)
{
    static int table[64][9] = {};
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    int& v = table[dev & 63][c];
    if (!v)
    {
        const int smem = 227 * 1024 - TG_STATIC;
        tg_fn fn = tg_kernel(4, 0, TG_DENSE);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned) (c * sms), 1, 1);
        cfg.blockDim = dim3(tg_threads(2), 1, 1);
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

// Share of a wave that clusters of an odd size take longer when they fill the device (`left` more would fit) behind a rotation
// kernel whose blocks are still leaving (a dependent launch). What the occupancy query counts fits at once only on free SMs: clusters
// that move in one by one as SMs free up leave single SMs over, and the last ones start late. Measured, us, with dependent launches /
// in plain order: 400 x 2304 with k cut in three, 41 clusters 28.7 / 33.0, 44: 34.6 / 33.0, 45 (all that fit) 43.1 / 33.0; 400 x 3840 cut
// in five, 23: 30.3 / 33.0, 25: 36.6 / 33.1, 26 (all) 46.4 / 33.3. Rotations of up to a block per SM leave no trace (40 rows: 12.2 at any
// count), nor do even sizes, nor seven (105 of 148 SMs).
static double tg_late(int c, long left, long chunks, int sms)
{
    return (c != 3 && c != 5) || chunks <= 8L * sms || left > 2 ? 0.0 : (left == 0 ? 0.4 : (left == 1 ? 0.15 : 0.04));
}

// Tile height, form and k split for M rows x `blocks` column blocks: the cheapest by a model (us) that ranks plans. A 64-row
// step takes the slowest of the decode (0.44 per 8192 weights, 0.48 in a pair with its hand-over), the tensor pipe
// (0.50 per 256 tokens, 0.66 per 512 of a pair) and the x~ tiles of all CTAs out of L2 (9.7 TB/s; the CTAs of a pair fetch half
// each); a CTA costs 3.6 + 0.0155 per token (a pair 2.8 more) around its k loop, the exchange of a split 0.72 and 0.0354 per token
// that crosses to a peer. One set of constants: over 1 .. 8 bits and the three codebooks a step's decode differs by a tenth (0.32 ..
// 0.37, pairs 0.34 .. 0.40). The sums are not times, the ranking is what was measured: fitted on 984 pairs of a shape (k 1024 .. 25600,
// n 512 .. 28672, 2 .. 8 bits, every codebook) and a row count (17 .. 2048), every form, tile height and split forced in turn. On 357
// others, on another machine, the plan taken is on average within 0.4 % of the best one, nineteen in twenty within 1.9 % (before tg_late
// and with constants fitted at 4 bits: 1.2 and 7.5 %, at worst 1.52 x); twelve are more than 5 % above it, at worst 133 x 1792 x 3584
// 14.2 us / 12.7, 1756 x 10368 x 13952 472 / 432, 698 x 14336 x 2048 59.5 / 55.1.
// One CTA of sixteen decode warps per SM: two of eight take as long per step and longer per exchange.
static int tg_plan(TgParams& S, int M, long blocks, bool pairs, int ksteps, int sms, int dev, int* form)
{
    // forced by tests and sweeps: pairs of 512- / 256-token tiles (modes 2, 3), no pairs (0), a tile height, a split
    const int tile_forced = g_tc_tile ? g_tc_tile : (pairs && g_tc_pair == 2 ? 512 : (pairs && g_tc_pair == 3 ? 256 : 0));
    const bool only_pairs = pairs && g_tc_pair >= 2, no_pairs = !pairs || !g_tc_pair || (g_tc_split && g_tc_pair < 2);
    double best = 1e30;
    int best_smem = 0;
    TgParams T = S;
    for (int tiles = (M + TG_MAX_TOKENS - 1) / TG_MAX_TOKENS; tiles <= (M + 127) / 128 && tiles < (M + TG_MAX_TOKENS - 1) / TG_MAX_TOKENS + 8; ++tiles)
        for (int pair = only_pairs ? 1 : 0; pair <= (no_pairs ? 0 : 1); ++pair)
        {
            const int smem = tg_layout(T, tile_forced ? tile_forced : ((M + tiles - 1) / tiles + 15) & ~15, 2, pair), xs = T.xstages;
            if (!smem) continue;
            for (int c = 1; c <= (pair ? 4 : 8) && c <= ksteps; ++c)
            {
                T.split = c;
                T.xstages = xs;
                if (g_tc_split && c != g_tc_split) continue;
                const int need = tg_exchange(T, smem, pair);
                if (T.share < 1) continue;
                const long clusters = (pair ? blocks / 2 : blocks) * ((M + T.tile - 1) / T.tile);
                const long fit = c > 1 || pair ? tg_max_clusters(pair ? 2 * c : c, sms, dev) : sms;
                const long waves = (clusters + fit - 1) / fit, live = (pair ? 2 : 1) * c * (clusters < fit ? clusters : fit);
                const double late = S.pdl && !pair ? tg_late(c, waves * fit - clusters, (long) M * ksteps / 2, sms) : 0.0;
                const double mma = (pair ? 0.00128 : 0.00195) * T.tile, l2 = T.tile * (pair ? 64.0 : 128.0) * live / 9.67e6, decode = pair ? 0.48 : 0.44;
                const double feed = mma > l2 ? mma : l2, step = feed > decode ? feed : decode;
                const double cost = (waves + late) * ((double) ((ksteps + c - 1) / c) * step + 3.6 + 0.0155 * T.tile + (pair ? 2.8 : 0.0)
                                             + (c > 1 ? 0.72 + 0.0354 * T.tile * (c - 1) / c : 0.0));
                if (cost < best * 0.99) { best = cost; best_smem = need; S = T; *form = pair ? TG_PAIR : TG_DENSE; }
            }
        }
    return best_smem;
}

// tiled x~ (launch_had_tiled) -> C. With T set (amp_exl3_mgemm): `n` is the width of one slice, the grid covers
// T->num slices, and trellis / svh (and c when T->c is given) are ignored in favour of the tables.
int launch_gemm_tc(const void* xh, const void* trellis, void* c, const void* svh, int M, int k, int n,
                   int K, int cb, int c_fp32, cudaStream_t stream, const TcTables* T)
{
    AMP_REQUIRE(xh && (T || (trellis && c && svh)), "exl3_gemm: null pointer");
    AMP_REQUIRE(!T || (T->num >= 1 && T->trellis && T->svh && (T->c || c)), "exl3_mgemm: pointer tables are required");
    AMP_REQUIRE(K >= 1 && K <= 8 && cb >= 0 && cb <= 2, "exl3_gemm: unsupported bitrate / codebook");
    AMP_REQUIRE(M >= 1 && k % 128 == 0 && n % 128 == 0 && k > 0 && n > 0, "exl3_gemm: k and n must be multiples of 128");
    AMP_REQUIRE(((uintptr_t) xh & 15) == 0 && ((uintptr_t) trellis & 15) == 0 && ((uintptr_t) c & 15) == 0 &&
                ((uintptr_t) svh & 7) == 0, "exl3_gemm: misaligned pointer");
    const long slices = T ? T->num : 1, blocks = slices * (n / 128);
    AMP_REQUIRE(blocks <= 0x3fffffffL / 8, "exl3_gemm: too many column blocks");
    int dev = 0, sms = 148;
    if (cudaError_t e = cudaGetDevice(&dev)) return cuda_rc(e, "cudaGetDevice");
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);

    TgParams S = {};
    TcParams& P = S.t;
    P.xt = (const unsigned char*) xh; P.trellis = (const uint16_t*) trellis; P.svh = (const __half*) svh; P.c = c;
    P.M = M; P.k = k; P.n = n; P.c_fp32 = c_fp32;
    P.tables = T ? 1 : 0;
    P.wait_limit = g_tc_wait[0]; P.wait_limit_last = g_tc_wait[1];
    if (T) { P.t_trellis = T->trellis; P.t_svh = T->svh; P.t_c = T->c; P.t_stride = T->stride; P.t_src = T->src; }
    if (int rc = tc_status_ptr(dev, &P.status)) return rc;
    S.pdl = g_pdl;
    int form = TG_DENSE;
    const int smem = tg_plan(S, M, blocks, n % 256 == 0, k / TC_BK, sms, dev, &form);
    AMP_REQUIRE(smem, "exl3_gemm: no plan for the forced split and tile");
    const long mblk = ((long) M + S.tile - 1) / S.tile;
    AMP_REQUIRE(mblk <= 65535, "exl3_gemm: too many rows");
    tg_fn fn = tg_kernel(K, cb, form);
    if (cudaError_t e = ensure_smem(fn, smem, dev)) return cuda_rc(e, "exl3_gemm smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (blocks * S.split), (unsigned) mblk, 1);
    cfg.blockDim = dim3(tg_threads(2, form == TG_PAIR), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    const int cluster = form == TG_PAIR ? 2 * S.split : S.split;
    if (cluster > 1)
    {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = cluster; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (g_pdl)
    {
        // the rotation kernel in front releases this launch at its start
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return cuda_rc(cudaLaunchKernelEx(&cfg, fn, S), "exl3_gemm launch");
}

// Expert-grouped form for token-sorted MoE prefill: xt / c are (kinds, Mcap, k / n) in the padded, expert-sorted row
// space, the tile table lives in device memory (see TcParams). One CTA per (tile, projection, 128-column block); the
// grid is sized for G.max_tiles and the surplus returns. Eight decode warps and two CTAs per SM, so that one CTA's
// set-up and epilogue run under the other's decode.
int launch_gemm_tc_grouped(const void* xt, void* c, long Mcap, int k, int n, int K, int cb, int c_fp32,
                              const long long* t_trellis, const long long* t_svh, const TcGroups& G, cudaStream_t stream)
{
    AMP_REQUIRE(xt && c && t_trellis && t_svh && G.ntiles && G.tile_e && G.tile_row0 && G.tile_rows, "exl3_moe_sorted: null pointer");
    AMP_REQUIRE(K >= 1 && K <= 8 && cb >= 0 && cb <= 2, "exl3_moe_sorted: unsupported bitrate / codebook");
    AMP_REQUIRE(Mcap >= 1 && Mcap <= 0x7fffffffL && k % 128 == 0 && n % 128 == 0 && k > 0 && n > 0, "exl3_moe_sorted: k and n must be multiples of 128");
    AMP_REQUIRE(((uintptr_t) xt & 15) == 0 && ((uintptr_t) c & 15) == 0, "exl3_moe_sorted: misaligned pointer");
    AMP_REQUIRE(G.kinds >= 1 && G.kinds <= 2 && G.tile >= 16 && G.tile <= TG_MAX_N && G.tile % 16 == 0 && G.experts >= 1, "exl3_moe_sorted: bad grouping");
    AMP_REQUIRE(G.max_tiles >= 1 && G.max_tiles <= 65535, "exl3_moe_sorted: too many row tiles");
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return cuda_rc(e, "cudaGetDevice");
    TgParams S = {};
    const int smem = tg_layout(S, G.tile, 1);
    AMP_REQUIRE(smem, "exl3_moe_sorted: tile does not fit");
    S.x_area = smem - tg_smem(0, S.wstages, 0);
    S.split = 1;
    S.share = smem / tg_row(1) & ~15;
    // Dependent launch only where the first CTA of the grid waits for the rotation kernel: with one launch per bit width a
    // launch whose experts all have another width would be over before that kernel, and the next launch's wait would be
    // for it alone.
    S.pdl = g_pdl && !G.bits[0];
    TcParams& P = S.t;
    P.xt = (const unsigned char*) xt; P.c = c;
    P.M = (int) Mcap; P.k = k; P.n = n; P.c_fp32 = c_fp32;
    P.t_trellis = t_trellis; P.t_svh = t_svh;
    P.g_ntiles = G.ntiles; P.g_tile_e = G.tile_e; P.g_tile_row0 = G.tile_row0; P.g_tile_rows = G.tile_rows;
    P.g_experts = G.experts;
    P.wait_limit = P.wait_limit_last = g_tc_wait[0];
    P.g_bits[0] = G.bits[0]; P.g_bits[1] = G.bits[1];
    if (int rc = tc_status_ptr(dev, &P.status)) return rc;
    tg_fn fn = tg_kernel(K, cb, TG_GROUPED);
    if (cudaError_t e = ensure_smem(fn, smem, dev)) return cuda_rc(e, "exl3_moe_sorted smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (G.kinds * (n / 128)), (unsigned) G.max_tiles, 1);
    cfg.blockDim = dim3(tg_threads(1), 1, 1);
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

using namespace amp;

// Reads and clears the GEMM's status word on the current device (non-zero: a bounded wait on a barrier ran out).
// Synchronises.
AMP_API int amp_exl3_gemm_status(int* out)
{
    int v = 0, zero = 0;
    if (cudaError_t e = cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int))) return cuda_rc(e, "status read");
    if (v) if (cudaError_t e = cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int))) return cuda_rc(e, "status clear");
    if (out) *out = v;
    return 0;
}

// The pair form's remote arrivals release at cluster scope, always; this used to select it. Returns 1, the setting.
AMP_API int amp_exl3_set_gemm_relay_release(int)
{
    return 1;
}

// Pair (cta_group::2) form: 0 = never, 1 = by plan (default), 2 / 3 = pairs of 512 / 256 tokens whenever n is a
// multiple of 256, with a forced split over up to four pairs (tests). Returns the previous setting.
AMP_API int amp_exl3_set_gemm_pair(int mode)
{
    const int old = g_tc_pair;
    g_tc_pair = mode < 0 ? 0 : (mode > 3 ? 3 : mode);
    return old;
}

// Forces the number of k slices (1..8) and / or the tokens per tile (a multiple of 16, up to 512) of the dense form;
// 0: by rule. For tests and sweeps.
AMP_API int amp_exl3_set_gemm_plan(int split, int tile)
{
    g_tc_split = split < 0 || split > 8 ? 0 : split;
    g_tc_tile = tile < 0 || tile > 512 ? 0 : (tile + 15) & ~15;
    return 0;
}

// Polls of a barrier wait before it is declared lost, and of the waits of the last CTA of a cluster or pair (a few
// microseconds each; 0: the default, TC_SPIN_LIMIT). For tests of what a wait that runs out leaves behind.
AMP_API int amp_exl3_set_gemm_wait_limit(int polls, int last)
{
    g_tc_wait[0] = polls > 0 ? (unsigned) polls : TC_SPIN_LIMIT;
    g_tc_wait[1] = last > 0 ? (unsigned) last : TC_SPIN_LIMIT;
    return 0;
}
