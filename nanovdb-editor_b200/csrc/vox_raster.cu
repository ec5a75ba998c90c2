// vox_raster.cu - per-Gaussian records, rank tables, run detection and the
// node2 tree of the Gaussian -> node2 voxelization.
//
// Reference path (raster/Raster.cpp:420-558): two passes of fragment windows,
// each re-running gaussian_prim / fanout / gaussian_frag_{alloc,color} and an
// incremental 4-level tree build with atomics.  Here:
//   k_prep        one record per Gaussian (bbox, inverse rotation, alpha
//                 constants), footprint, touched root tiles
//   k_mark_lower  touched lower-node cells (128^3 voxels) per Gaussian bbox
//   [vox_leaf.cu] (leaf, Gaussian) pairs, sort, one CTA per candidate leaf:
//                 value masks, RGBA8, float sums
//   k_tree        the candidates' masks -> leaves, lowers, uppers, the clouds'
//                 first nodes
//   k_cloud_layout   per-cloud grid layout
//   [vox_leaf.cu] k_write_leaves: leaf nodes, values, bbox
//   k_write_nodes the other node2 nodes, headers and gaps
#include <cstdio>
#include <cuda_runtime.h>

#include "pnanovdb_b200.h"
#include "vox_device.cuh"
#include "vox_internal.h"
#include "vox_raster.h"

namespace vox
{

// Sets a bit of a bitmap that many threads mark (a cloud's Gaussians touch a
// handful of root tiles and lower cells): a word that already has it is only
// read.  Read-modify-write atomics on one word run one after another in L2,
// reads of it do not: the call on 2M Gaussians (8 root tiles) 51.84 -> 51.15 ms,
// on 64 clouds with 2M Gaussians 20.60 -> 20.19 ms.
__device__ __forceinline__ void mark_bit(unsigned long long* bits, uint64_t i)
{
    const unsigned long long b = 1ull << (i & 63);
    if (!(__ldcg(&bits[i >> 6]) & b))
        atomicOr(&bits[i >> 6], b);
}

// ------------------------------------------------------------------ prep ----
__global__ void __launch_bounds__(256) k_prep(PrepParams P, GaussRec* recs, WalkRec* walk,
                                              uint64_t* footprints, uint64_t* lcols, unsigned long long* root_bits,
                                              int* err)
{
    const int64_t g = P.g0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= (P.g1 < 0 ? P.count : P.g1))
        return;
    GaussRec R;
    int32_t bmax[3];
    uint32_t cloud = 0;
    if (P.cloud_start)
    {
        // last cloud whose start is <= g
        int64_t lo = 0, hi = P.clouds;
        while (lo < hi)
        {
            int64_t mid = (lo + hi) >> 1;
            if (P.cloud_start[mid] <= g)
                lo = mid + 1;
            else
                hi = mid;
        }
        cloud = (uint32_t)(lo - 1);
    }
    const float vs = P.cloud_vs ? P.cloud_vs[cloud] : P.voxel_size;
    uint64_t fp = make_record(P, g, vs, R, bmax);
    R.q5.w = (int32_t)cloud;
    if (fp)
    {
        int e = 0;
        for (int a = 0; a < 3; a++)
        {
            int32_t lo = (&R.q4.x)[a];
            if (lo < -65536 || bmax[a] > 65535)
                e |= ERR_RANGE;
        }
        if (fp >= (1ull << 31))
            e |= ERR_FOOTPRINT;
        if (e)
        {
            atomicOr(err, e);
            fp = 0;
            R.q4.w = 0;
        }
    }
    recs[g] = R;
    footprints[g] = fp;
    // leaf columns (lx, ly) of the bbox
    lcols[g] = fp ? (uint64_t)((bmax[0] >> 3) - (R.q4.x >> 3) + 1) * (uint64_t)((bmax[1] >> 3) - (R.q4.y >> 3) + 1) : 0ull;
    if (fp)
    {
        walk[g] = walk_record(R, vs);
        // root tiles (4096^3 voxels) spanned by the bbox
        for (int32_t x = R.q4.x >> 12; x <= (bmax[0] >> 12); x++)
            for (int32_t y = R.q4.y >> 12; y <= (bmax[1] >> 12); y++)
                for (int32_t z = R.q4.z >> 12; z <= (bmax[2] >> 12); z++)
                {
                    mark_bit(root_bits, root_index(cloud, x << 12, y << 12, z << 12));
                }
    }
}

__global__ void __launch_bounds__(256) k_mark_lower(const GaussRec* recs, int64_t G, const uint64_t* root_bits,
                                                    const uint64_t* root_prefix, unsigned long long* lower_bits)
{
    int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G)
        return;
    GaussRec R = recs[g];
    if (!R.q4.w)
        return;
    int32_t mn[3] = { R.q4.x, R.q4.y, R.q4.z };
    int32_t mx[3] = { R.q4.x + R.q5.x - 1, R.q4.y + R.q5.y - 1, R.q4.z + R.q5.z - 1 };
    for (int32_t x = mn[0] >> 7; x <= (mx[0] >> 7); x++)
        for (int32_t y = mn[1] >> 7; y <= (mx[1] >> 7); y++)
            for (int32_t z = mn[2] >> 7; z <= (mx[2] >> 7); z++)
            {
                int32_t cx = x << 7, cy = y << 7, cz = z << 7;
                uint64_t rr = bit_rank(root_bits, root_prefix, root_index(rec_cloud(R), cx, cy, cz));
                mark_bit(lower_bits, rr * 32768ull + upper_n_of(cx, cy, cz));
            }
}

// inverse tables: rank -> root_n, rank -> cell
__global__ void k_invert_bits(const uint64_t* bits, const uint64_t* prefix, int64_t words, uint32_t* out)
{
    int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= words)
        return;
    uint64_t b = bits[w];
    uint64_t r = prefix[w];
    while (b)
    {
        int bit = __ffsll((long long)b) - 1;
        out[r++] = (uint32_t)(w * 64 + bit);
        b &= b - 1;
    }
}

// ------------------------------------------------------------------ tree ----
// The tree's tables from the candidate leaves' value masks, in one pass.  The
// candidates are sorted by leaf key, so the leaves are the candidates with a
// non-empty mask, in order; a lower node starts at the leaf whose lower rank
// differs from the leaf's before, an upper node at the lower whose root tile
// does, a cloud's tables at the upper whose cloud does.  A tile counts its
// voxels, leaves, lowers and uppers (one candidate per lane), gets the four
// counts of the tiles before it by look-back (a warp each), and writes every
// table at its place.  Bound by latency: 64 B of mask and some 40 B of tables
// per candidate, 19 us for the 440k candidates of 2M Gaussians, 13 us for 20k.
// Sorted voxel keys, run detection over them and per-voxel leaf and position
// arrays, which it replaces, took 1.1 ms for 106M voxels.
constexpr int TREE_BLOCK = 256;
constexpr int TREE_ITEMS = 4;
constexpr int TREE_WARPS = TREE_BLOCK / 32;
constexpr int TREE_TILE = TREE_BLOCK * TREE_ITEMS;

__device__ __forceinline__ uint32_t cand_voxels(const uint64_t* cand_mask, int64_t c)
{
    const ulonglong2* m = reinterpret_cast<const ulonglong2*>(cand_mask + 8 * c);
    uint32_t n = 0;
#pragma unroll
    for (int w = 0; w < 4; w++)
    {
        const ulonglong2 x = m[w];
        n += __popcll(x.x) + __popcll(x.y);
    }
    return n;
}

__global__ void __launch_bounds__(TREE_BLOCK) k_tree(TreeParams T, NodeParams N)
{
    __shared__ uint32_t s_cnt[4][TREE_WARPS];
    __shared__ uint64_t s_ex[4];
    __shared__ uint32_t s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    if (threadIdx.x == 0)
        s_tile = atomicAdd(T.counter, 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    const int64_t wbase = (int64_t)tile * TREE_TILE + (int64_t)warp * (32 * TREE_ITEMS);
    // the last leaf before this warp's candidates.  Empty candidates come in short
    // runs: every Gaussian passes in the leaf of its centre, and the leaf test
    // lets through only leaves next to its ellipsoid.
    bool has_prev = false;
    uint32_t prev = 0;
    if (wbase < T.NCL)
        for (int64_t e = wbase - 1; e >= 0 && !has_prev; e -= 32)
        {
            const int64_t c = e - lane;
            const uint32_t b = __ballot_sync(0xffffffffu, c >= 0 && cand_voxels(T.cand_mask, c) > 0);
            if (b)
            {
                has_prev = true;
                prev = T.cand_key[e - (__ffs(b) - 1)];
            }
        }
    uint32_t cnt[TREE_ITEMS], vin[TREE_ITEMS], key[TREE_ITEMS], pkey[TREE_ITEMS];
    uint32_t bleaf[TREE_ITEMS], blo[TREE_ITEMS], bup[TREE_ITEMS], bprev[TREE_ITEMS];
    uint32_t tv = 0, tl = 0, tlo = 0, tu = 0;
#pragma unroll
    for (int i = 0; i < TREE_ITEMS; i++)
    {
        const int64_t c = wbase + i * 32 + lane;
        const bool valid = c < T.NCL;
        cnt[i] = valid ? cand_voxels(T.cand_mask, c) : 0u;
        key[i] = valid ? T.cand_key[c] : 0u;
        const bool leaf = cnt[i] > 0;
        bleaf[i] = __ballot_sync(0xffffffffu, leaf);
        const uint32_t before = bleaf[i] & lt;
        const uint32_t kb = __shfl_sync(0xffffffffu, key[i], before ? 31 - __clz(before) : 0);
        pkey[i] = before ? kb : prev;
        const bool hp = before || has_prev;
        const bool hlo = leaf && (!hp || (key[i] >> 12) != (pkey[i] >> 12));
        const bool hup = hlo && (!hp || (N.lower_cell[key[i] >> 12] >> 15) != (N.lower_cell[pkey[i] >> 12] >> 15));
        bprev[i] = __ballot_sync(0xffffffffu, hp);
        blo[i] = __ballot_sync(0xffffffffu, hlo);
        bup[i] = __ballot_sync(0xffffffffu, hup);
        uint32_t incl = cnt[i];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += y;
        }
        vin[i] = tv + incl;
        tv += __shfl_sync(0xffffffffu, incl, 31);
        tl += __popc(bleaf[i]);
        tlo += __popc(blo[i]);
        tu += __popc(bup[i]);
        if (bleaf[i])
        {
            has_prev = true;
            prev = __shfl_sync(0xffffffffu, key[i], 31 - __clz(bleaf[i]));
        }
    }
    if (lane == 0)
    {
        s_cnt[0][warp] = tv;
        s_cnt[1][warp] = tl;
        s_cnt[2][warp] = tlo;
        s_cnt[3][warp] = tu;
    }
    __syncthreads();
    if (warp < 4)
    {
        uint64_t agg = 0;
        for (int w = 0; w < TREE_WARPS; w++)
            agg += s_cnt[warp][w];
        const int64_t tiles = (T.NCL + TREE_TILE - 1) / TREE_TILE;
        const uint64_t e = lookback_exclusive_warp(T.status + 4 * (uint64_t)warp * tiles, tile, agg, T.epoch, T.err);
        if (lane == 0)
            s_ex[warp] = e;
    }
    __syncthreads();
    uint64_t v = s_ex[0], l = s_ex[1], lo = s_ex[2], u = s_ex[3];
    for (int w = 0; w < warp; w++)
    {
        v += s_cnt[0][w];
        l += s_cnt[1][w];
        lo += s_cnt[2][w];
        u += s_cnt[3][w];
    }
    const CloudParams& C = N.C;
    const uint32_t le = lt | (1u << lane);
#pragma unroll
    for (int i = 0; i < TREE_ITEMS; i++)
    {
        const int64_t c = wbase + i * 32 + lane;
        if (c < T.NCL)
        {
            const bool leaf = cnt[i] > 0, hp = (bprev[i] >> lane) & 1u;
            const uint64_t vx = v + vin[i] - cnt[i], li = l + __popc(bleaf[i] & lt);
            // counts up to and including this candidate
            const uint64_t loi = lo + __popc(blo[i] & le), ui = u + __popc(bup[i] & le);
            T.cand_voff[c] = vx;
            int64_t cloud = -1; // of this leaf, or of the last one before
            if (leaf || (hp && c == T.NCL - 1))
                cloud = N.root_of_rank[N.lower_cell[(leaf ? key[i] : pkey[i]) >> 12] >> 15] >> 15;
            if (leaf)
            {
                const int4 o = T.cand_org[c];
                N.leaf_vstart[li] = (uint32_t)vx;
                N.leaf_cand[li] = (uint32_t)c;
                N.leaf_lower[li] = (uint32_t)(loi - 1);
                N.leaf_lower_n[li] = key[i] & 4095u;
                N.leaf_origin[3 * li + 0] = o.x;
                N.leaf_origin[3 * li + 1] = o.y;
                N.leaf_origin[3 * li + 2] = o.z;
                C.leaf_cloud[li] = (uint32_t)cloud;
            }
            // lowers never outnumber the touched lower cells; more heads mean the
            // candidates are not sorted: report, never write past the tables
            if (loi >= T.lower_cap)
                atomicOr(T.err, ERR_ORDER);
            else
            {
                if ((blo[i] >> lane) & 1u)
                {
                    N.lower_lstart[loi - 1] = (uint32_t)li;
                    N.lower_upper_n[loi - 1] = N.lower_cell[key[i] >> 12] & 32767u;
                    N.lower_parent[loi - 1] = (uint32_t)(ui - 1);
                }
                if ((bup[i] >> lane) & 1u)
                {
                    N.upper_root_n[ui - 1] = N.root_of_rank[N.lower_cell[key[i] >> 12] >> 15];
                    N.upper_lostart[ui - 1] = (uint32_t)(loi - 1);
                    const int64_t pc = hp ? (int64_t)(N.root_of_rank[N.lower_cell[pkey[i] >> 12] >> 15] >> 15) : -1;
                    for (int64_t b = pc + 1; b <= cloud; b++)
                    {
                        C.upper_start[b] = (uint32_t)(ui - 1);
                        C.lower_start[b] = (uint32_t)(loi - 1);
                        C.leaf_start[b] = (uint32_t)li;
                        C.vstart[b] = vx;
                    }
                }
                if (c == T.NCL - 1)
                {
                    const uint64_t V = vx + cnt[i], L = li + (leaf ? 1u : 0u);
                    N.leaf_vstart[L] = (uint32_t)V;
                    N.lower_lstart[loi] = (uint32_t)L;
                    N.upper_lostart[ui] = (uint32_t)loi;
                    for (int64_t b = cloud + 1; b <= C.B; b++)
                    {
                        C.upper_start[b] = (uint32_t)ui;
                        C.lower_start[b] = (uint32_t)loi;
                        C.leaf_start[b] = (uint32_t)L;
                        C.vstart[b] = V;
                    }
                    T.counts[0] = V;
                    T.counts[1] = L;
                    T.counts[2] = loi;
                    T.counts[3] = ui;
                }
            }
        }
        l += __popc(bleaf[i]);
        lo += __popc(blo[i]);
        u += __popc(bup[i]);
    }
}

// ---------------------------------------------------------------- clouds ----
__device__ __forceinline__ uint32_t upper_cloud(const NodeParams& N, uint64_t u)
{
    return N.upper_root_n[u] >> 15;
}
__device__ __forceinline__ uint32_t lower_cloud(const NodeParams& N, uint64_t lo)
{
    return N.upper_root_n[N.lower_parent[lo]] >> 15;
}

__device__ __forceinline__ uint64_t al256(uint64_t x)
{
    return (x + 255) / 256 * 256;
}

// one CTA: per-cloud node counts -> grid layout, grid offsets and value bases
// (exclusive scans over the clouds, 1024 at a time)
__global__ void __launch_bounds__(1024) k_cloud_layout(NodeParams N)
{
    __shared__ uint64_t s_warp[33];
    __shared__ uint64_t s_carry[2];
    const CloudParams& C = N.C;
    if (threadIdx.x == 0)
        s_carry[0] = s_carry[1] = 0;
    __syncthreads();
    for (int64_t c0 = 0; c0 < C.B; c0 += blockDim.x)
    {
        const int64_t b = c0 + threadIdx.x;
        uint64_t size = 0, vc = 0;
        uint64_t node2 = 0, o_bbox = 0, o_rgba = 0, o_dens = 0, o_col = 0;
        if (b < C.B)
        {
            const uint64_t U = C.upper_start[b + 1] - C.upper_start[b];
            const uint64_t Lo = C.lower_start[b + 1] - C.lower_start[b];
            const uint64_t L = C.leaf_start[b + 1] - C.leaf_start[b];
            vc = 2 + (C.vstart[b + 1] - C.vstart[b]);
            node2 = n2_node_bytes(0) + U * n2_node_bytes(1) + Lo * n2_node_bytes(2) + L * n2_node_bytes(3);
            o_bbox = al256(VOX_GRID_HEADER_BYTES + node2);
            o_rgba = al256(o_bbox + 32);
            o_dens = al256(o_rgba + 4 * vc);
            o_col = al256(o_dens + 4 * vc);
            size = C.floats ? al256(o_col + 12 * vc) : o_dens;
            for (int a = 0; a < 6; a++)
                C.bbox[6 * b + a] = a < 3 ? 0x7FFFFFFF : (int32_t)0x80000000;
        }
        uint64_t tot_size, tot_vc;
        const uint64_t ex_size = block_excl_scan_u64(size, s_warp, tot_size);
        const uint64_t ex_vc = block_excl_scan_u64(vc, s_warp, tot_vc);
        if (b < C.B)
        {
            const uint64_t g = s_carry[0] + ex_size;
            C.grid_off[b] = g;
            C.value_base[b] = s_carry[1] + ex_vc;
            C.node2_bytes[b] = node2;
            C.bbox_off[b] = g + o_bbox;
            C.rgba_off[b] = g + o_rgba;
            C.dens_off[b] = g + o_dens;
            C.col_off[b] = g + o_col;
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            s_carry[0] += tot_size;
            s_carry[1] += tot_vc;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        C.grid_off[C.B] = s_carry[0];
        C.value_base[C.B] = s_carry[1];
    }
}

// canonical (single fragment window) node order inside every cloud's grid:
// uppers, lowers, leaves, each in hierarchical key order; node addresses
// (absolute in the output buffer) follow node_idx order
__global__ void k_canonical_order(NodeParams N, uint64_t U)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t root_sz = n2_node_bytes(0), up_sz = n2_node_bytes(1), lo_sz = n2_node_bytes(2),
                   lf_sz = n2_node_bytes(3);
    const CloudParams& C = N.C;
    if (t < (int64_t)U)
    {
        const uint32_t b = upper_cloud(N, t);
        const uint64_t local = (uint64_t)t - C.upper_start[b];
        N.upper_idx[t] = 1 + local;
        N.upper_addr[t] = C.grid_off[b] + VOX_GRID_HEADER_BYTES + root_sz + local * up_sz;
        N.upper_vidx[t] = 2;
    }
    if (t < N.Lo)
    {
        const uint32_t b = lower_cloud(N, t);
        const uint64_t Ub = C.upper_start[b + 1] - C.upper_start[b];
        const uint64_t local = (uint64_t)t - C.lower_start[b];
        N.lower_idx[t] = 1 + Ub + local;
        N.lower_addr[t] = C.grid_off[b] + VOX_GRID_HEADER_BYTES + root_sz + Ub * up_sz + local * lo_sz;
        N.lower_vidx[t] = 2;
    }
    if (t < N.L)
    {
        const uint32_t b = C.leaf_cloud[t];
        const uint64_t Ub = C.upper_start[b + 1] - C.upper_start[b];
        const uint64_t Lob = C.lower_start[b + 1] - C.lower_start[b];
        const uint64_t local = (uint64_t)t - C.leaf_start[b];
        N.leaf_idx[t] = 1 + Ub + Lob + local;
        N.leaf_addr[t] = C.grid_off[b] + VOX_GRID_HEADER_BYTES + root_sz + Ub * up_sz + Lob * lo_sz + local * lf_sz;
        N.leaf_vidx[t] = 2 + ((uint64_t)N.leaf_vstart[t] - C.vstart[b]);
    }
}

// ------------------------------------------------------------ node2 write ----
// Node2 roots, uppers and lowers, headers and the gaps between a grid's parts,
// in one launch.  A CTA writes a stretch of NODE_PART words of one node (a root
// is 542 KB, an upper 274 KB: one CTA each would run for as long as all the rest)
// and every word of it once, so nothing is cleared first.  A node's first
// stretch holds its indices, masks and prefix words
// (grid_build_count_new.slang:49-88), the others children only.  Bound by the
// latency of a lower's up to 4096 child loads; 11 us for 8 uppers, 8 full lowers
// (separate kernels that cleared the region and summed prefixes in one thread: 62 us).
constexpr int NODE_THREADS = 256;
constexpr uint32_t NODE_PART = 4352; // words: a whole lower node (4292)
__host__ __device__ constexpr uint32_t node_words(int t)
{
    return (uint32_t)(n2_node_bytes(t) / 8);
}
__host__ __device__ constexpr uint32_t node_parts(int t)
{
    return (node_words(t) + NODE_PART - 1) / NODE_PART;
}

// word w of the prefix of a mask with exclusive popcounts ex[0 .. nw) and total ex[nw]
__device__ __forceinline__ uint64_t prefix_word(const uint16_t* ex, uint32_t nw, uint32_t q)
{
    uint64_t v = q == 0 ? (uint64_t)ex[nw] : (uint64_t)ex[4 * q];
    for (uint32_t f = 1; f < 4; f++)
        v |= (uint64_t)ex[4 * q + f] << (16 * f);
    return v;
}

// the CTA's stretch of node type T; child(i) is the i-th of its `children` child words
template <int T, class Child>
__device__ __forceinline__ void write_node_part(uint64_t* W, uint32_t part, uint64_t idx, uint64_t vidx,
                                                uint32_t children, const uint64_t* s_mask, const uint16_t* s_ex,
                                                Child child)
{
    constexpr uint32_t nw = T == 2 ? 64u : 512u;
    const uint32_t w0 = part * NODE_PART, w1 = min(node_words(T), w0 + NODE_PART);
    if (part == 0)
        for (uint32_t w = threadIdx.x; w < n2_off_children(T); w += NODE_THREADS)
        {
            uint64_t v = 0;
            if (w == N2_OFF_NODE_IDX)
                v = idx;
            else if (w == N2_OFF_VALUE_IDX)
                v = vidx;
            else if (w - n2_off_child_mask(T) < nw)
                v = s_mask[w - n2_off_child_mask(T)];
            else if (w - n2_off_child_prefix(T) < nw / 4)
                v = prefix_word(s_ex, nw, w - n2_off_child_prefix(T));
            else if (T == 0 && w - N2_OFF_KEY_MASK_ROOT < nw)
                v = s_mask[w - N2_OFF_KEY_MASK_ROOT];
            else if (T == 0 && w - N2_OFF_KEY_PREFIX_ROOT < nw / 4)
                v = prefix_word(s_ex, nw, w - N2_OFF_KEY_PREFIX_ROOT);
            W[w] = v;
        }
    const uint32_t c0 = max(w0, n2_off_children(T));
#pragma unroll 4
    for (uint32_t w = c0 + threadIdx.x; w < w1; w += NODE_THREADS)
    {
        const uint32_t i = w - n2_off_children(T);
        W[w] = i < children ? child(i) : (T == 0 && i < 65536u ? N2_END_KEY : 0ull);
    }
}

// the first stretch's mask and its exclusive popcounts: slot(i) is child i's bit
template <int T, class Slot>
__device__ __forceinline__ void node_mask(uint64_t* s_mask, uint16_t* s_ex, uint64_t* s_warp, uint32_t children, Slot slot)
{
    constexpr uint32_t nw = T == 2 ? 64u : 512u;
    for (uint32_t i = threadIdx.x; i < nw; i += NODE_THREADS)
        s_mask[i] = 0;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < children; i += NODE_THREADS)
    {
        const uint32_t n = slot(i);
        // 32-bit words: a 64-bit OR in shared memory is a compare-and-swap loop
        atomicOr(reinterpret_cast<uint32_t*>(s_mask) + (n >> 5), 1u << (n & 31));
    }
    __syncthreads();
    const uint32_t w = 2 * threadIdx.x;
    const uint32_t a = w < nw ? __popcll(s_mask[w]) : 0, b = w < nw ? __popcll(s_mask[w + 1]) : 0;
    uint64_t total;
    const uint64_t ex = block_excl_scan_u64(a + b, s_warp, total);
    if (w < nw)
    {
        s_ex[w] = (uint16_t)ex;
        s_ex[w + 1] = (uint16_t)(ex + a);
    }
    if (threadIdx.x == 0)
        s_ex[nw] = (uint16_t)total;
    __syncthreads();
}

// bytes [a, b) of the output zeroed by the CTA (multiples of 4, a few hundred)
__device__ __forceinline__ void zero_words(uint8_t* out, uint64_t a, uint64_t b)
{
    for (uint64_t o = a + 4 * threadIdx.x; o < b; o += 4 * NODE_THREADS)
        *reinterpret_cast<uint32_t*>(out + o) = 0u;
}

// cloud b's header, bbox, background values (the two slots before each channel's
// first voxel) and alignment gaps
__device__ __forceinline__ void write_grid_header(const NodeParams& N, uint64_t b, uint8_t* out, vox_grid_header_t& h)
{
    const CloudParams& C = N.C;
    const uint64_t g = C.grid_off[b];
    const uint64_t vc = 2 + (C.vstart[b + 1] - C.vstart[b]);
    if (threadIdx.x == 0)
    {
        memset(&h, 0, sizeof(h));
        h.magic = VOX_GRID_MAGIC;
        h.version = 1;
        h.header_bytes = VOX_GRID_HEADER_BYTES;
        h.grid_bytes = C.grid_off[b + 1] - g;
        h.node2_offset = VOX_GRID_HEADER_BYTES;
        h.node2_bytes = C.node2_bytes[b];
        h.upper_count = C.upper_start[b + 1] - C.upper_start[b];
        h.lower_count = C.lower_start[b + 1] - C.lower_start[b];
        h.leaf_count = C.leaf_start[b + 1] - C.leaf_start[b];
        h.node_order = C.node_order;
        h.value_count = vc;
        h.bbox_offset = C.bbox_off[b] - g;
        h.rgba8_offset = C.rgba_off[b] - g;
        h.density_offset = C.floats ? C.dens_off[b] - g : 0;
        h.color_offset = C.floats ? C.col_off[b] - g : 0;
        h.voxel_size = C.cloud_vs ? C.cloud_vs[b] : C.voxel_size;
        if (vc > 2)
            for (int a = 0; a < 6; a++)
                h.bbox[a] = C.bbox[6 * b + a];
        h.pair_count = C.cloud_pairs ? C.cloud_pairs[b] : (uint64_t)C.P;
        const int64_t g0 = C.cloud_start ? C.cloud_start[b] : 0, g1 = C.cloud_start ? C.cloud_start[b + 1] : C.G;
        const uint64_t f0 = g0 < C.G ? C.frag_off[g0] : *C.F_total, f1 = g1 < C.G ? C.frag_off[g1] : *C.F_total;
        h.candidate_count = f1 - f0;
    }
    __syncthreads();
    if (threadIdx.x < sizeof(h) / 4)
        ((uint32_t*)(out + g))[threadIdx.x] = reinterpret_cast<const uint32_t*>(&h)[threadIdx.x];
    if (threadIdx.x < 6)
        ((int32_t*)(out + C.bbox_off[b]))[threadIdx.x] = h.bbox[threadIdx.x];
    zero_words(out, g + VOX_GRID_HEADER_BYTES + C.node2_bytes[b], C.bbox_off[b]);
    zero_words(out, C.bbox_off[b] + 24, C.rgba_off[b] + 8);
    if (!C.floats)
    {
        zero_words(out, C.rgba_off[b] + 4 * vc, C.grid_off[b + 1]);
        return;
    }
    zero_words(out, C.rgba_off[b] + 4 * vc, C.dens_off[b] + 8);
    zero_words(out, C.dens_off[b] + 4 * vc, C.col_off[b] + 24);
    zero_words(out, C.col_off[b] + 12 * vc, C.grid_off[b + 1]);
}
static_assert(sizeof(vox_grid_header_t) == VOX_GRID_HEADER_BYTES && VOX_GRID_HEADER_BYTES / 4 <= NODE_THREADS,
              "the header is written by one word per thread");

__global__ void __launch_bounds__(NODE_THREADS) k_write_nodes(NodeParams N, uint64_t U, uint8_t* out)
{
    __shared__ uint64_t s_mask[512];
    __shared__ uint16_t s_ex[513];
    __shared__ uint64_t s_warp[33];
    __shared__ vox_grid_header_t s_head;
    uint64_t k = blockIdx.x;
    if (k < (uint64_t)N.C.B * node_parts(0)) // roots, headers
    {
        const uint64_t b = k / node_parts(0);
        const uint32_t part = (uint32_t)(k % node_parts(0));
        const uint64_t addr = N.C.grid_off[b] + VOX_GRID_HEADER_BYTES;
        const uint32_t u0 = N.C.upper_start[b], nu = N.C.upper_start[b + 1] - u0;
        if (part == 0)
        {
            write_grid_header(N, b, out, s_head);
            node_mask<0>(s_mask, s_ex, s_warp, nu, [&](uint32_t i) { return N.upper_root_n[u0 + i] & 32767u; });
        }
        // per child its offset, then per child its key
        write_node_part<0>((uint64_t*)(out + addr), part, 0, 2, 2 * nu, s_mask, s_ex, [&](uint32_t i) -> uint64_t {
            if (i < nu)
                return N.upper_addr[u0 + i] - addr;
            int32_t o[3];
            root_tile_origin(N.upper_root_n[u0 + i - nu] & 32767u, o);
            return (uint64_t)((uint32_t)o[2] >> 12) | ((uint64_t)((uint32_t)o[1] >> 12) << 21) |
                   ((uint64_t)((uint32_t)o[0] >> 12) << 42);
        });
        return;
    }
    k -= (uint64_t)N.C.B * node_parts(0);
    if (k < U * node_parts(1)) // uppers
    {
        const uint64_t u = k / node_parts(1);
        const uint32_t part = (uint32_t)(k % node_parts(1));
        const uint64_t addr = N.upper_addr[u];
        const uint32_t lo0 = N.upper_lostart[u], n = N.upper_lostart[u + 1] - lo0;
        if (part == 0)
            node_mask<1>(s_mask, s_ex, s_warp, n, [&](uint32_t i) { return N.lower_upper_n[lo0 + i]; });
        write_node_part<1>((uint64_t*)(out + addr), part, N.upper_idx[u], N.upper_vidx[u], n, s_mask, s_ex,
                           [&](uint32_t i) { return N.lower_addr[lo0 + i] - addr; });
        return;
    }
    k -= U * node_parts(1); // lowers
    const uint64_t addr = N.lower_addr[k];
    const uint32_t l0 = N.lower_lstart[k], n = N.lower_lstart[k + 1] - l0;
    node_mask<2>(s_mask, s_ex, s_warp, n, [&](uint32_t i) { return N.leaf_lower_n[l0 + i]; });
    write_node_part<2>((uint64_t*)(out + addr), 0, N.lower_idx[k], N.lower_vidx[k], n, s_mask, s_ex,
                       [&](uint32_t i) { return N.leaf_addr[l0 + i] - addr; });
}
static_assert(node_parts(2) == 1, "a lower node is one stretch");

// =================================================================== launch
void launch_prep(const PrepParams& P, GaussRec* recs, WalkRec* walk, uint64_t* footprints, uint64_t* lcols,
                 uint64_t* root_bits, int* err, cudaStream_t s)
{
    const int64_t n = (P.g1 < 0 ? P.count : P.g1) - P.g0;
    if (n <= 0)
        return;
    { k_prep<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(P, recs, walk, footprints, lcols, (unsigned long long*)root_bits, err); count_launch(); }
}

void launch_mark_lower(const GaussRec* recs, int64_t G, const uint64_t* root_bits, const uint64_t* root_prefix,
                       uint64_t* lower_bits, cudaStream_t s)
{
    if (G <= 0)
        return;
    { k_mark_lower<<<(unsigned)((G + 255) / 256), 256, 0, s>>>(recs, G, root_bits, root_prefix,
                                                           (unsigned long long*)lower_bits); count_launch(); }
}

void launch_invert_bits(const uint64_t* bits, const uint64_t* prefix, int64_t words, uint32_t* out, cudaStream_t s)
{
    if (words <= 0)
        return;
    { k_invert_bits<<<(unsigned)((words + 255) / 256), 256, 0, s>>>(bits, prefix, words, out); count_launch(); }
}


size_t tree_status_words(int64_t NCL)
{
    return 16 * (size_t)((NCL + TREE_TILE - 1) / TREE_TILE);
}

void launch_tree(const TreeParams& T, const NodeParams& N, cudaStream_t s)
{
    if (T.NCL <= 0)
        return;
    { k_tree<<<(unsigned)((T.NCL + TREE_TILE - 1) / TREE_TILE), TREE_BLOCK, 0, s>>>(T, N); count_launch(); }
}
void launch_canonical_order(const NodeParams& N, uint64_t U, cudaStream_t s)
{
    int64_t m = N.L;
    if ((int64_t)U > m)
        m = (int64_t)U;
    if (N.Lo > m)
        m = N.Lo;
    if (m <= 0)
        return;
    { k_canonical_order<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(N, U); count_launch(); }
}
void launch_write_nodes(const NodeParams& N, uint64_t U, uint8_t* out, cudaStream_t s)
{
    const uint64_t grid = (uint64_t)N.C.B * node_parts(0) + U * node_parts(1) + (uint64_t)N.Lo;
    { k_write_nodes<<<(unsigned)grid, NODE_THREADS, 0, s>>>(N, U, out); count_launch(); }
}
void launch_cloud_layout(const NodeParams& N, cudaStream_t s)
{
    { k_cloud_layout<<<1, 1024, 0, s>>>(N); count_launch(); }
}
} // namespace vox
