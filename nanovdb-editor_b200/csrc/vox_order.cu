// vox_order.cu - the reference's node order (VOX_FLAG_WINDOW_ORDER).
//
// The reference builds the tree window by window: Gaussians in batches of
// 256K, each batch's bbox fragments in windows of 8M (raster/Raster.cpp:443-444),
// and per window, level by level (upper, lower, leaf), the nodes the window
// creates are appended to one node pool in (parent node_idx, n) order
// (raster/GridBuild.cpp:412-505, grid_build_scatter_new.slang:107-170).
// node_idx is a node's position in that pool, node2 addresses follow node_idx
// order, and every node's value_idx is 2 + the active voxels of the leaves
// before it in node_idx order (so uppers and lowers created in a later window
// carry the count of the earlier windows' leaves).
//
// A node is created in the first window holding a passing fragment of one of
// its voxels.  The leaf walk records that window per candidate leaf (the
// minimum over its passing pairs); lowers and uppers take the minimum over
// their children.  Per level, the order by (window, parent rank, n) gives each
// node's rank; per-window counts place the levels of a window after the
// nodes of every earlier window.  A call whose fragments fit one window has the
// canonical order (every node in window 0, so ranks go by parent and n) and
// takes none of this (vox_api.cu).
#include <cstdio>
#include <cuda_runtime.h>

#include "pnanovdb_b200.h"
#include "vox_device.cuh"
#include "vox_internal.h"
#include "vox_raster.h"

namespace vox
{

// windows of each 256K-Gaussian batch: ceil(fragments / 8M)
__global__ void k_batch_windows(const uint64_t* frag_off, const uint64_t* F_total, int64_t G, int64_t nbatch,
                                uint64_t* nwin)
{
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nbatch)
        return;
    const int64_t g0 = b * REF_PRIM_BATCH, g1 = min(G, g0 + (int64_t)REF_PRIM_BATCH);
    const uint64_t f0 = frag_off[g0], f1 = g1 < G ? frag_off[g1] : *F_total;
    nwin[b] = (f1 - f0 + REF_WINDOW - 1) / REF_WINDOW;
}

__global__ void k_leaf_wkey(int64_t L, const uint32_t* leaf_cand, const uint64_t* cand_wkey, uint64_t* leaf_wkey)
{
    const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (l < L)
        leaf_wkey[l] = cand_wkey[leaf_cand[l]];
}

// minimum over the children runs [start[i], start[i + 1]), a warp per run
// (a lower has up to 4096 leaves: one thread per run took 61 us for 8 lowers)
__global__ void k_run_min(int64_t n, const uint32_t* start, const uint64_t* child, uint64_t* out)
{
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= n)
        return;
    uint64_t m = ~0ull;
    const uint32_t c1 = start[i + 1];
#pragma unroll 4
    for (uint32_t c = start[i] + lane; c < c1; c += 32)
    {
        const uint64_t v = child[c];
        m = v < m ? v : m;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1)
    {
        const uint64_t v = __shfl_xor_sync(0xffffffffu, m, o);
        m = v < m ? v : m;
    }
    if (lane == 0)
        out[i] = m;
}

// sort key of a level: window, parent rank, n (nbits bits; pbits for the rank);
// nodes per window (lanes of one window add once)
template <class K>
__global__ void k_level_keys(int64_t n, const uint64_t* wkey, const uint32_t* parent, const uint32_t* parent_rank,
                             const uint32_t* nval, int nbits, int pbits, K* keys, uint32_t* vals, uint64_t* wcount)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const uint64_t pr = parent ? (uint64_t)parent_rank[parent[i]] : 0ull, w = wkey[i];
    keys[i] = (K)((w << (pbits + nbits)) | (pr << nbits) | (uint64_t)(nval[i] & ((1u << nbits) - 1u)));
    vals[i] = (uint32_t)i;
    const uint32_t peers = __match_any_sync(__activemask(), w);
    if ((threadIdx.x & 31) == __ffs(peers) - 1)
        atomicAdd((unsigned long long*)&wcount[w], (unsigned long long)__popc(peers));
}

__global__ void k_level_rank(int64_t n, const uint32_t* sorted_vals, uint32_t* rank)
{
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n)
        rank[sorted_vals[p]] = (uint32_t)p;
}

// A level of at most LEVEL_RANK_SMALL_MAX nodes: a node's rank is the number of smaller
// keys (the keys are distinct).  One launch of n^2 comparisons in shared memory
// (2048 nodes: 16k per thread, 10 us) for the histogram, the passes and the
// inversion of a radix sort.
__global__ void __launch_bounds__(256) k_level_rank_small(int n, const uint64_t* keys, uint32_t* rank)
{
    __shared__ uint64_t s_key[LEVEL_RANK_SMALL_MAX];
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        s_key[i] = keys[i];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const uint64_t k = s_key[i];
    uint32_t r = 0;
#pragma unroll 8
    for (int j = 0; j < n; j++)
        r += s_key[j] < k ? 1u : 0u;
    rank[i] = r;
}

// voxels of every leaf, in the level's order
__global__ void k_leaf_popc_ranked(int64_t L, const uint32_t* rank, const uint32_t* leaf_vstart, uint64_t* out)
{
    const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (l < L)
        out[rank[l]] = (uint64_t)(leaf_vstart[l + 1] - leaf_vstart[l]);
}

// node_idx, byte address and value index of every node from its level rank and
// the per-window counts (base_* = nodes of each level in earlier windows)
__global__ void k_window_place(WindowOrderParams W, NodeParams N)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t root_sz = n2_node_bytes(0), up_sz = n2_node_bytes(1), lo_sz = n2_node_bytes(2),
                   lf_sz = n2_node_bytes(3);
    const uint64_t base_addr = N.C.grid_off[0] + VOX_GRID_HEADER_BYTES + root_sz;
    // every node's value_idx is 2 + the active voxels of the leaves before it in
    // node_idx order; the uppers and lowers of window w follow the leaves of the
    // earlier windows
    if (t < (int64_t)W.U)
    {
        const uint64_t p = W.rank_u[t], w = W.wkey_u[t];
        N.upper_idx[t] = 1 + W.base_all[w] + (p - W.base_u[w]);
        N.upper_addr[t] = base_addr + p * up_sz + W.base_lo[w] * lo_sz + W.base_leaf[w] * lf_sz;
        N.upper_vidx[t] = 2 + (W.base_leaf[w] < (uint64_t)N.L ? W.leaf_voff[W.base_leaf[w]] : W.V);
    }
    if (t < N.Lo)
    {
        const uint64_t p = W.rank_lo[t], w = W.wkey_lo[t];
        const uint64_t cu = W.base_u[w + 1] - W.base_u[w];
        N.lower_idx[t] = 1 + W.base_all[w] + cu + (p - W.base_lo[w]);
        N.lower_addr[t] = base_addr + W.base_u[w + 1] * up_sz + p * lo_sz + W.base_leaf[w] * lf_sz;
        N.lower_vidx[t] = 2 + (W.base_leaf[w] < (uint64_t)N.L ? W.leaf_voff[W.base_leaf[w]] : W.V);
    }
    if (t < N.L)
    {
        const uint64_t p = W.rank_leaf[t], w = W.wkey_leaf[t];
        const uint64_t cu = W.base_u[w + 1] - W.base_u[w], clo = W.base_lo[w + 1] - W.base_lo[w];
        N.leaf_idx[t] = 1 + W.base_all[w] + cu + clo + (p - W.base_leaf[w]);
        N.leaf_addr[t] = base_addr + W.base_u[w + 1] * up_sz + W.base_lo[w + 1] * lo_sz + p * lf_sz;
        N.leaf_vidx[t] = 2 + W.leaf_voff[p];
    }
}

// nodes of each level in earlier windows: one CTA, 1024 windows at a time
__global__ void __launch_bounds__(1024) k_window_bases(int64_t nw, const uint64_t* cu, const uint64_t* clo,
                                                       const uint64_t* cleaf, uint64_t* base_u, uint64_t* base_lo,
                                                       uint64_t* base_leaf, uint64_t* base_all)
{
    __shared__ uint64_t s_warp[33];
    const uint64_t* cnt[3] = { cu, clo, cleaf };
    uint64_t* base[3] = { base_u, base_lo, base_leaf };
    uint64_t run[3] = { 0, 0, 0 };
    for (int64_t w0 = 0; w0 <= nw; w0 += blockDim.x)
    {
        const int64_t w = w0 + threadIdx.x;
        uint64_t all = 0;
        for (int k = 0; k < 3; k++)
        {
            uint64_t total;
            const uint64_t ex = run[k] + block_excl_scan_u64(w < nw ? cnt[k][w] : 0ull, s_warp, total);
            run[k] += total;
            all += ex;
            if (w <= nw)
                base[k][w] = ex;
        }
        if (w <= nw)
            base_all[w] = all;
    }
}

static unsigned blocks_for(int64_t n)
{
    return (unsigned)((n + 255) / 256 > 0 ? (n + 255) / 256 : 1);
}

void launch_batch_windows(const uint64_t* frag_off, const uint64_t* F_total, int64_t G, int64_t nbatch,
                          uint64_t* nwin, cudaStream_t s)
{
    if (nbatch <= 0)
        return;
    { k_batch_windows<<<blocks_for(nbatch), 256, 0, s>>>(frag_off, F_total, G, nbatch, nwin); count_launch(); }
}

void launch_leaf_wkey(int64_t L, const uint32_t* leaf_cand, const uint64_t* cand_wkey, uint64_t* leaf_wkey,
                      cudaStream_t s)
{
    if (L <= 0)
        return;
    { k_leaf_wkey<<<blocks_for(L), 256, 0, s>>>(L, leaf_cand, cand_wkey, leaf_wkey); count_launch(); }
}

void launch_run_min(int64_t n, const uint32_t* start, const uint64_t* child, uint64_t* out, cudaStream_t s)
{
    if (n <= 0)
        return;
    { k_run_min<<<blocks_for(32 * n), 256, 0, s>>>(n, start, child, out); count_launch(); }
}

void launch_level_keys(int64_t n, const uint64_t* wkey, const uint32_t* parent, const uint32_t* parent_rank,
                       const uint32_t* nval, int nbits, int pbits, void* keys, int key64, uint32_t* vals,
                       uint64_t* wcount, cudaStream_t s)
{
    if (n <= 0)
        return;
    if (key64)
        { k_level_keys<uint64_t><<<blocks_for(n), 256, 0, s>>>(n, wkey, parent, parent_rank, nval, nbits, pbits, (uint64_t*)keys, vals, wcount); count_launch(); }
    else
        { k_level_keys<uint32_t><<<blocks_for(n), 256, 0, s>>>(n, wkey, parent, parent_rank, nval, nbits, pbits, (uint32_t*)keys, vals, wcount); count_launch(); }
}

void launch_level_rank_small(int64_t n, const uint64_t* keys, uint32_t* rank, cudaStream_t s)
{
    if (n <= 0)
        return;
    { k_level_rank_small<<<blocks_for(n), 256, 0, s>>>((int)n, keys, rank); count_launch(); }
}

void launch_level_rank(int64_t n, const uint32_t* sorted_vals, uint32_t* rank, cudaStream_t s)
{
    if (n <= 0)
        return;
    { k_level_rank<<<blocks_for(n), 256, 0, s>>>(n, sorted_vals, rank); count_launch(); }
}

void launch_leaf_popc_ranked(int64_t L, const uint32_t* rank, const uint32_t* leaf_vstart, uint64_t* out,
                             cudaStream_t s)
{
    if (L <= 0)
        return;
    { k_leaf_popc_ranked<<<blocks_for(L), 256, 0, s>>>(L, rank, leaf_vstart, out); count_launch(); }
}

void launch_window_bases(int64_t nw, const uint64_t* cu, const uint64_t* clo, const uint64_t* cleaf, uint64_t* base_u,
                         uint64_t* base_lo, uint64_t* base_leaf, uint64_t* base_all, cudaStream_t s)
{
    { k_window_bases<<<1, 1024, 0, s>>>(nw, cu, clo, cleaf, base_u, base_lo, base_leaf, base_all); count_launch(); }
}

void launch_window_place(const WindowOrderParams& W, const NodeParams& N, cudaStream_t s)
{
    const int64_t n = N.L > N.Lo ? N.L : N.Lo;
    if (n <= 0)
        return;
    { k_window_place<<<blocks_for(n), 256, 0, s>>>(W, N); count_launch(); }
}

} // namespace vox
