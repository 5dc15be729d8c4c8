// Token-sorted MoE dispatch in one launch: the router's picks become the expert-sorted lists that
// amp_exl3_moe_sorted (and the reference's exl3_moe) take. Integer work, bit-exact by definition:
// a stable counting sort of the assignments by local expert.
//
// Replaces, with the same name, signature and return convention (a cudaError_t), the reference's
// amp_moe_prep (src/torch/amp_kernels.cu:7024-7043, kernels :6849-7022; binding torch.moe_prep,
// src/torch/amp_torch.cpp:8164-8215). For the experts [e0, e0 + E) of this rank, with foreign picks
// in the sentinel bucket E:
//   fe[a]     bucket of assignment a = token * K + pick            order[j]  assignment at sorted position j
//   tok[j]    its token   wts[j] its weight, fp16                  inv[a]    sorted position of assignment a
//   count[b]  assignments per bucket (E + 1)   start[b] exclusive prefix sum   kind[e] = count[e] > 0
//
// One block, or a cluster of eight for longer lists (a single SM pays a global round trip per step of its warps
// and one SM's worth of scattered stores: 47 us for 12000 assignments, the cluster takes 9). The assignments are
// cut into one contiguous segment per warp of the cluster. A warp walks its segment 32 assignments at a time, four
// steps' loads in flight; __match_any_sync groups the lanes of one bucket, so a bucket's counter of the segment
// takes one update per group. Pass 1 counts; a prefix over the segments, the blocks' bucket totals (read through
// distributed shared memory) and a scan over the buckets give every (segment, bucket) its first position; pass 2
// walks the segments again and hands out positions in assignment order: earlier blocks and segments first, then
// earlier steps, then lower lanes. The number of warps is chosen so that the counters fit in shared memory
// (32 warps up to about 1500 experts, 8 at 4096), so every E up to 4096 takes the same path.
#include "host_common.h"
#include <cuda_fp16.h>
#include <stdint.h>

namespace amp {

constexpr int MP_CLUSTER = 8;              // blocks of a long list
constexpr int MP_LONG = 1024;              // assignments from which the cluster pays

__device__ __forceinline__ int mp_ld_cluster(const int* p, int rank)
{
    uint32_t a = (uint32_t) __cvta_generic_to_shared(p);
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

__device__ __forceinline__ void mp_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void moe_dispatch_kernel(const long long* __restrict__ idx, const float* __restrict__ w, int A, int K, int E, long long e0,
                                    long long* __restrict__ fe, long long* __restrict__ order, long long* __restrict__ tok,
                                    __half* __restrict__ wts, long long* __restrict__ count, long long* __restrict__ start,
                                    long long* __restrict__ inv, long long* __restrict__ kind)
{
    extern __shared__ int sh[];
    const int nb = E + 1, nw = blockDim.x >> 5, rank = blockIdx.x, nblk = gridDim.x;    // (the grid is one cluster)
    int* tot = sh;                      // [nb] assignments per bucket
    int* first = sh + nb;               // [nb] first sorted position of a bucket; then of this block's share of it
    int* mine = sh + 2 * nb;            // [nb] this block's assignments per bucket (read by the peers)
    int* seg = sh + 3 * nb;             // [nw][nb] pass 1: count of (segment, bucket); then its running offset inside the block's share
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int per = (A + nw * nblk - 1) / (nw * nblk);
    const int a0 = min((rank * nw + warp) * per, A), a1 = min(a0 + per, A);
    const unsigned below = (1u << lane) - 1u;
    constexpr int U = 4;                // steps whose loads are in flight together

    for (int i = t; i < nw * nb; i += blockDim.x) seg[i] = 0;
    __syncthreads();

    auto bucket_of = [&](long long e) {
        const long long loc = e - e0;
        return (loc >= 0 && loc < E) ? (int) loc : E;
    };

    for (int base = a0; base < a1; base += 32 * U)
    {
        long long e[U];
        #pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const int a = base + 32 * u + lane;
            e[u] = a < a1 ? idx[a] : 0;
        }
        #pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const int a = base + 32 * u + lane;
            const bool live = a < a1;
            const int b = live ? bucket_of(e[u]) : E;
            if (live) fe[a] = b;
            const unsigned peers = __match_any_sync(0xffffffffu, b) & __ballot_sync(0xffffffffu, live);
            if (live && (peers & below) == 0) seg[warp * nb + b] += __popc(peers);       // the group's lowest lane
            __syncwarp();
        }
    }
    __syncthreads();

    // per bucket: offsets of the segments inside this block's share, and the share
    for (int b = t; b < nb; b += blockDim.x)
    {
        int acc = 0;
        for (int s = 0; s < nw; ++s)
        {
            const int c = seg[s * nb + b];
            seg[s * nb + b] = acc;
            acc += c;
        }
        mine[b] = acc;
    }
    if (nblk > 1) mp_cluster_sync(); else __syncthreads();
    // totals over the blocks; `first` holds what the blocks in front contribute until the scan below
    for (int b = t; b < nb; b += blockDim.x)
    {
        int all = 0, before = 0;
        if (nblk == 1) all = mine[b];
        else
        {
            int v[MP_CLUSTER];
            #pragma unroll
            for (int r = 0; r < MP_CLUSTER; ++r) v[r] = mp_ld_cluster(mine + b, r);
            #pragma unroll
            for (int r = 0; r < MP_CLUSTER; ++r) { before += r < rank ? v[r] : 0; all += v[r]; }
        }
        tot[b] = all;
        first[b] = before;
    }
    if (nblk > 1) mp_cluster_sync(); else __syncthreads();           // (no block leaves while a peer may read its share)

    // exclusive scan over the buckets (warp 0: a contiguous run of buckets per lane)
    if (warp == 0)
    {
        const int run = (nb + 31) / 32, b0 = min(lane * run, nb), b1 = min(b0 + run, nb);
        int sum = 0;
        for (int b = b0; b < b1; ++b) sum += tot[b];
        int inc = sum;
        #pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const int o = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += o;
        }
        int acc = inc - sum;
        for (int b = b0; b < b1; ++b)
        {
            if (rank == 0) start[b] = acc;
            first[b] += acc;
            acc += tot[b];
        }
    }
    __syncthreads();

    if (rank == 0)
        for (int b = t; b < nb; b += blockDim.x)
        {
            count[b] = tot[b];
            if (b < E) kind[b] = tot[b] > 0 ? 1 : 0;
        }

    for (int base = a0; base < a1; base += 32 * U)
    {
        long long e[U];
        float wt[U];
        #pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const int a = base + 32 * u + lane;
            e[u] = a < a1 ? idx[a] : 0;
            wt[u] = a < a1 ? w[a] : 0.0f;
        }
        #pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const int a = base + 32 * u + lane;
            const bool live = a < a1;
            const int b = live ? bucket_of(e[u]) : E;
            const unsigned peers = __match_any_sync(0xffffffffu, b) & __ballot_sync(0xffffffffu, live);
            int pos = 0;
            if (live) pos = first[b] + seg[warp * nb + b] + __popc(peers & below);
            __syncwarp();                                          // every lane has read the offset before the group moves it
            if (live && (peers & below) == 0) seg[warp * nb + b] += __popc(peers);
            __syncwarp();
            if (live)
            {
                order[pos] = a;
                tok[pos] = a / K;
                wts[pos] = __float2half(wt[u]);
                inv[a] = pos;
            }
        }
    }
}

}  // namespace amp

AMP_API int amp_moe_prep(const long long* idx, const float* w, int A, int K, int E, long long e0, long long* fe,
                         long long* order, long long* tok, void* wts, long long* count, long long* start,
                         long long* inv, long long* kind, cudaStream_t stream)
{
    if (A < 1 || K < 1 || E < 1 || E > 4096 || !idx || !w || !fe || !order || !tok || !wts || !count || !start || !inv || !kind)
        return (int) cudaErrorInvalidValue;
    const size_t nb = (size_t) E + 1;
    const int blocks = A >= amp::MP_LONG ? amp::MP_CLUSTER : 1;
    int nw = 32;
    while (nw > 1 && (3 + nw) * nb * sizeof(int) > 200 * 1024) nw >>= 1;
    const size_t smem = (3 + nw) * nb * sizeof(int);
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return (int) e;
    if (smem > 48 * 1024)
        if (cudaError_t e = amp::ensure_smem(amp::moe_dispatch_kernel, (int) smem, dev)) return (int) e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) blocks, 1, 1);
    cfg.blockDim = dim3((unsigned) (nw * 32), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned) blocks; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = blocks > 1 ? 1 : 0;
    return (int) cudaLaunchKernelEx(&cfg, amp::moe_dispatch_kernel, idx, w, A, K, E, e0, fe, order, tok, (__half*) wts, count, start, inv, kind);
}
