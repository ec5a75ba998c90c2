// vox_leaf.cu - leaf-granular voxelization: (leaf, Gaussian) pairs, one CTA
// per candidate leaf.
//
// The reference tests every (voxel, Gaussian) fragment of a Gaussian's bbox in
// 8M-fragment windows and inserts passing voxels into its tree with atomics
// (raster/Raster.cpp:420-558, gaussian_frag_alloc.slang, grid_build_*.slang,
// gaussian_frag_color.slang).  Here the unit of sorting is the leaf (8^3
// voxels, the node2 leaf of PNanoVDBExt.h:72-81):
//   k_leaf_emit   per Gaussian, the leaf cells of its bbox whose box may reach
//       its 0.01-opacity ellipsoid (a conservative test in double), written as
//       (leaf key, Gaussian) in Gaussian-major order; a stable sort by leaf key
//       keeps each leaf's Gaussians in ascending id;
//   k_leaf_cands  runs of equal leaf keys -> candidate leaves;
//   k_leaf_pass   persistent CTAs over the candidate leaves, a leaf's Gaussians
//       in chunks: the test (gaussian_frag_alloc.slang:84-162) one (Gaussian, box
//       column) per thread, which sets the leaf's value mask, then the passing
//       pairs' RGBA8 maximum (gaussian_frag_color.slang:239-246) and float sums,
//       one pair per thread, in any order;
//   k_write_leaves   once the tree's tables stand (k_tree): staged values to
//       their value index, leaf nodes, bbox.
// The adjoint (k_leaf_backward) and the sorted pair list (k_leaf_export)
// go through the same (leaf, Gaussian) pairs.
#include <cstdio>
#include <cuda_runtime.h>

#include "vox_device.cuh"
#include "vox_internal.h"
#include "vox_raster.h"

namespace vox
{

constexpr int LP_THREADS = 256; // two voxels per thread: leaf_n = t and t + 256
constexpr int LP_CHUNK = 32;    // Gaussian records staged in shared memory per round

__device__ __forceinline__ int64_t upper_bound_u64_l(const uint64_t* a, int64_t lo, int64_t hi, uint64_t v)
{
    while (lo < hi)
    {
        int64_t mid = (lo + hi) >> 1;
        if (a[mid] <= v)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// ------------------------------------------------------------ emission ----
// May a voxel of the leaf at origin o pass the reference test?  The local AABB
// of the leaf box (monotone-corner identity, in double) contains every voxel's
// local AABB; the float test's rounding is bounded by delta = 1e-5 (1 + B), B
// bounding the magnitudes it sums (a worst-case error bound of the float test
// is below 1.1e-6 B).
__device__ __forceinline__ bool leaf_may_hit(const GaussRec& R, const RInv& M, float vsf, int32_t ox, int32_t oy,
                                             int32_t oz)
{
    const double vs = vsf;
    const int32_t o[3] = { ox, oy, oz };
    const double mu[3] = { R.q0.x, R.q0.y, R.q0.z };
    const double inv_s[3] = { R.q3.y, R.q3.z, R.q3.w };
    double lo[3], hi[3], E[3];
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        const double w0 = (double)o[a] * vs, w1 = (double)(o[a] + 8) * vs;
        lo[a] = w0 - mu[a];
        hi[a] = w1 - mu[a];
        E[a] = fmax(fabs(w0), fabs(w1)) + fabs(mu[a]) + vs;
    }
    double sum = 0.0, B = 0.0;
#pragma unroll
    for (int r = 0; r < 3; r++)
    {
        const double sc = (double)R.q0.w * inv_s[r];
        double mn = 0.0, mx = 0.0, mag = 0.0;
#pragma unroll
        for (int a = 0; a < 3; a++)
        {
            const double m = (double)M.m[r][a];
            const double p0 = lo[a] * m, p1 = hi[a] * m;
            mn += fmin(p0, p1);
            mx += fmax(p0, p1);
            mag += fabs(m) * E[a];
        }
        mn *= sc;
        mx *= sc;
        const double d = mn > 0.0 ? mn : (mx < 0.0 ? -mx : 0.0);
        sum += d * d;
        B = fmax(B, mag * sc);
    }
    const double bound = 1.0 + 1e-5 * (1.0 + B);
    return sum < bound * bound;
}

// the same from the record in global memory, out of line: for the write pass, which
// needs it in columns of more than 32 leaves alone
__device__ __noinline__ bool leaf_may_hit_at(const GaussRec* rec, float vsf, int32_t ox, int32_t oy, int32_t oz)
{
    const GaussRec R = *rec;
    return leaf_may_hit(R, rinv_of(R), vsf, ox, oy, oz);
}

// rank of the lower node of voxel (x, y, z) of a cloud, at its place in the leaf's key
__device__ __forceinline__ uint32_t lower_key_of(uint32_t cloud, int32_t x, int32_t y, int32_t z, const RankTables& T)
{
    const uint64_t rr = bit_rank(T.root_bits, T.root_prefix, root_index(cloud, x, y, z));
    const uint64_t cell = rr * 32768ull + upper_n_of(x, y, z);
    return (uint32_t)(bit_rank(T.lower_bits, T.lower_prefix, cell) << 12);
}

// the Gaussian of each 256-column tile's first column
__global__ void k_tile_gauss(const uint64_t* lcol_off, int64_t G, uint64_t NLC, int64_t* tile_g0)
{
    const uint64_t tile = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tile * 256 < NLC)
        tile_g0[tile] = upper_bound_u64_l(lcol_off, 0, G, tile * 256) - 1;
}

// One thread per leaf column (lx, ly) of a Gaussian's bbox, looping over lz.  Bound by
// the latency of the records' loads and of the double-precision chains, so by the CTAs an
// SM holds: the count pass 4 (64 registers), the write pass, which reads the box alone, 6.
// Both passes of 2M Gaussians' 29.6M pairs with their scan 1.34 -> 1.14 ms, 64 clouds 0.576
// -> 0.493 (3 CTAs each before; count 5: 1.18 ms, 6: 1.23; write 4: 1.21 with count 5).
// Blocks walk 256-column tiles; a tile's Gaussians [g0, g1] (g1 = the next
// tile's first) have their column offsets copied to shared memory, where each
// thread finds its column's Gaussian.
template <bool WRITE>
__global__ void __launch_bounds__(256, WRITE ? 6 : 4) k_leaf_emit(LeafEmitParams P, RankTables T)
{
    __shared__ uint64_t s_off[257];
    const uint64_t ntiles = (P.NLC + 255) / 256;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
    {
        const int64_t g0 = P.tile_g0[tile];
        const int64_t g1 = tile + 1 < ntiles ? P.tile_g0[tile + 1] : P.G - 1;
        const int64_t n = g1 - g0 + 1;
        if (n <= 256 && (int64_t)threadIdx.x < n)
            s_off[threadIdx.x] = P.lcol_off[g0 + threadIdx.x];
        __syncthreads();
        const uint64_t t = tile * 256 + threadIdx.x;
        if (t < P.NLC)
        {
        int64_t g;
        if (n <= 256)
        {
            int64_t lo = 0, hi = n; // upper bound of t in s_off[0, n)
            while (lo < hi)
            {
                const int64_t mid = (lo + hi) >> 1;
                if (s_off[mid] <= t)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            g = g0 + lo - 1;
        }
        else
            g = upper_bound_u64_l(P.lcol_off, g0, g1 + 1, t) - 1;
        GaussRec R;
        if (WRITE) // the box and the cloud
        {
            R.q4 = P.recs[g].q4;
            R.q5 = P.recs[g].q5;
        }
        else
            R = P.recs[g];
        const float vsf = rec_vs(R, P.voxel_size, P.cloud_vs);
        const int32_t lx0 = R.q4.x >> 3, ly0 = R.q4.y >> 3, ly1 = (R.q4.y + R.q5.y - 1) >> 3;
        const int32_t lz0 = R.q4.z >> 3, lz1 = (R.q4.z + R.q5.z - 1) >> 3;
        const uint32_t Ly = (uint32_t)(ly1 - ly0 + 1);
        const uint32_t local = (uint32_t)(t - P.lcol_off[g]);
        const int32_t ox = (lx0 + (int32_t)(local / Ly)) * 8, oy = (ly0 + (int32_t)(local % Ly)) * 8;
        uint64_t e = WRITE ? P.lc_off[t] : 0;
        uint64_t npairs = 0;
        // the write pass reuses the count pass's test results (first 32 leaves)
        const uint32_t known = WRITE ? P.lc_mask[t] : 0u;
        uint32_t mask = 0, lower = 0;
        int32_t lower_z = INT32_MIN;
        for (int32_t lz = lz0; lz <= lz1; lz++)
        {
            const int32_t oz = lz * 8;
            const int32_t i = lz - lz0;
            const bool hit = !WRITE    ? leaf_may_hit(R, rinv_of(R), vsf, ox, oy, oz)
                             : i < 32 ? ((known >> i) & 1u) != 0u
                                      : leaf_may_hit_at(&P.recs[g], vsf, ox, oy, oz);
            if (!WRITE && hit && i < 32)
                mask |= 1u << i;
            if (hit || P.check)
            {
                if (WRITE)
                {
                    if (oz >> 7 != lower_z) // a lower node is 16 leaves of the column
                    {
                        lower_z = oz >> 7;
                        lower = lower_key_of(rec_cloud(R), ox, oy, oz, T);
                    }
                    P.keys[e] = lower | lower_n_of(ox, oy, oz);
                    // the sort's value: the Gaussian itself, or the emission index where
                    // something is kept by it (the adjoint's rows, check mode's flags)
                    P.vals[e] = P.emit_gid ? (uint32_t)e : (uint32_t)g;
                    if (P.emit_gid)
                        P.emit_gid[e] = (uint32_t)g;
                    if (P.check)
                        P.emit_flag[e] = hit ? 0 : 1;
                    e++;
                }
                npairs++;
            }
        }
        if (!WRITE)
        {
            P.lc_count[t] = npairs;
            P.lc_mask[t] = mask;
        }
        }
        __syncthreads();
    }
}

// origin of the leaf with compact key lower_rank << 12 | lower_n
__device__ __forceinline__ void leaf_origin_of_key(uint32_t key, const uint32_t* lower_cell,
                                                   const uint32_t* root_of_rank, int32_t o[3])
{
    const uint32_t lr = key >> 12, ln = key & 4095u;
    const uint32_t cell = lower_cell[lr];
    const uint32_t un = cell & 32767u;
    root_tile_origin(root_of_rank[cell >> 15] & 32767u, o);
    o[0] += (int32_t)((un >> 10) & 31) * 128 + (int32_t)((ln >> 8) & 15) * 8;
    o[1] += (int32_t)((un >> 5) & 31) * 128 + (int32_t)((ln >> 4) & 15) * 8;
    o[2] += (int32_t)(un & 31) * 128 + (int32_t)(ln & 15) * 8;
}

// Candidate leaves (key, origin, first pair) from the runs of the sorted keys,
// and each sorted pair's Gaussian where the sort's values are emission indices
// (emit_gid non-null): one pass, run heads against the key before (a shuffle
// inside a warp), their count before the tile by look-back.  HBM-bound: 4 B per
// pair (flags, their scan and a compaction pass moved 40).  Sort and candidates of
// 29.6M pairs, with the sort carrying the Gaussians themselves: 1.65 -> 1.27 ms.
constexpr int LC_BLOCK = 256;
constexpr int LC_ITEMS = 8;
constexpr int LC_TILE = LC_BLOCK * LC_ITEMS;

__global__ void __launch_bounds__(LC_BLOCK) k_leaf_cands(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                                                         const uint32_t* __restrict__ emit_gid, int64_t Q,
                                                         const uint32_t* lower_cell, const uint32_t* root_of_rank,
                                                         CandParams C)
{
    __shared__ uint32_t s_cnt[LC_BLOCK / 32];
    __shared__ uint64_t s_ex;
    __shared__ uint32_t s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        s_tile = atomicAdd(C.counter, 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    const int64_t wbase = (int64_t)tile * LC_TILE + (int64_t)warp * (32 * LC_ITEMS);
    uint32_t k[LC_ITEMS], heads[LC_ITEMS];
    uint32_t carry = wbase > 0 && wbase - 1 < Q ? keys[wbase - 1] : 0u, count = 0;
#pragma unroll
    for (int i = 0; i < LC_ITEMS; i++)
    {
        const int64_t q = wbase + i * 32 + lane;
        k[i] = q < Q ? keys[q] : 0u;
        if (emit_gid && q < Q)
            C.pair_gid[q] = emit_gid[vals[q]];
    }
#pragma unroll
    for (int i = 0; i < LC_ITEMS; i++)
    {
        const int64_t q = wbase + i * 32 + lane;
        uint32_t prev = __shfl_up_sync(0xffffffffu, k[i], 1);
        if (lane == 0)
            prev = carry;
        carry = __shfl_sync(0xffffffffu, k[i], 31);
        heads[i] = __ballot_sync(0xffffffffu, q < Q && (q == 0 || k[i] != prev));
        count += __popc(heads[i]);
    }
    if (lane == 0)
        s_cnt[warp] = count;
    __syncthreads();
    if (warp == 0)
    {
        uint64_t agg = 0;
        for (int w = 0; w < LC_BLOCK / 32; w++)
            agg += s_cnt[w];
        const uint64_t e = lookback_exclusive_warp(C.status, tile, agg, C.epoch, C.err);
        if (lane == 0)
            s_ex = e;
    }
    __syncthreads();
    uint64_t at = s_ex;
    for (int w = 0; w < warp; w++)
        at += s_cnt[w];
#pragma unroll
    for (int i = 0; i < LC_ITEMS; i++)
    {
        const int64_t q = wbase + i * 32 + lane;
        const bool head = (heads[i] >> lane) & 1u;
        const uint64_t c = at + __popc(heads[i] & ((1u << lane) - 1u)); // candidates before this pair's own
        if (head)
        {
            int32_t o[3];
            leaf_origin_of_key(k[i], lower_cell, root_of_rank, o);
            C.cand_org[c] = make_int4(o[0], o[1], o[2], 0);
            C.cand_key[c] = k[i];
            C.cand_start[c] = (uint32_t)q;
        }
        if (q == Q - 1)
        {
            C.cand_start[c + (head ? 1u : 0u)] = (uint32_t)Q;
            *C.total = c + (head ? 1u : 0u);
        }
        at += __popc(heads[i]);
    }
}

// ------------------------------------------------------------ leaf walk ----
struct LeafSmem
{
    GaussRec rec[LP_CHUNK];
    uint32_t gid[LP_CHUNK];
    uint64_t mask[8];
    uint32_t cand;
};

__device__ __forceinline__ void cand_origin(const LeafPassParams& P, uint32_t key, int32_t o[3])
{
    leaf_origin_of_key(key, P.lower_cell, P.root_of_rank, o);
}

__device__ __forceinline__ bool in_bbox(const GaussRec& R, int32_t x, int32_t y, int32_t z)
{
    return (uint32_t)(x - R.q4.x) < (uint32_t)R.q5.x && (uint32_t)(y - R.q4.y) < (uint32_t)R.q5.y &&
           (uint32_t)(z - R.q4.z) < (uint32_t)R.q5.z;
}

// stage Gaussians [q0, q0 + cnt) of the sorted pair list
__device__ __forceinline__ void stage_chunk(const LeafPassParams& P, LeafSmem& S, uint32_t q0, uint32_t cnt)
{
    const int t = threadIdx.x;
    if (t < (int)cnt * 8)
    {
        const uint32_t j = (uint32_t)t >> 3, w = (uint32_t)t & 7u;
        const uint32_t g = P.pair_gid[q0 + j];
        reinterpret_cast<float4*>(&S.rec[j])[w] = reinterpret_cast<const float4*>(&P.recs[g])[w];
        if (w == 0)
            S.gid[j] = g;
    }
}

// ------------------------------------------------------ forward leaf walk
// A CTA walks a stream of candidate leaves in chunks of Gaussians (a leaf's
// Gaussians in ascending id): as many of the next LF_CHUNK as have boxes of
// lf_cap voxels together, since every voxel may pass and take a queue entry.
// Per chunk:
//   test   the part of each Gaussian's bbox inside the leaf, one (Gaussian,
//          column) per thread: the column's x / y share once, then its z run;
//          passing (Gaussian, voxel) pairs go to a shared queue;
//   alpha  one queued pair per thread: the reference's RGBA8 alpha and the
//          float channels' stable alpha, accumulated per voxel with shared
//          atomics - RGBA8 maximum, fixed-point density / colour sums (exact,
//          so independent of order);
//   flush  once a leaf's last alpha is done: its staged values, value mask
//          and pair count.
// One barrier per chunk: phase i runs the flush of the leaf that ended with
// chunk i - 2, the alpha of chunk i - 1, the test of chunk i, and the staging
// of chunk i + 1 (lanes of the last warp copy its records with cp.async and
// place its boxes).  Chunk data is triple-buffered, queues double-buffered.
// The barrier, the staging and the partly filled rounds cost the same for any
// chunk, so the larger it is the better; 56 KB of shared memory (4 CTAs per SM)
// bound it.  Against chunks of 12 Gaussians (with their whole records in each
// buffer), the walk of 200k Gaussians 3.52 -> 3.05 ms, a call on 2M 37.1 -> 32.5.
constexpr int LF_CHUNK = 24;
// the differentiable walk's chunks carry more per Gaussian and take fewer voxels
// to fit 4 CTAs as well (5120 and 3 CTAs: 2.37 instead of 2.27 ms for 500k Gaussians)
template <bool SMOOTH>
constexpr uint32_t lf_cap = SMOOTH ? 3840 : 5120;

// what the stagers read of the next chunk, each its own column (overwritten by
// its own next copies)
struct LeafStage
{
    float4 rec[6][LF_CHUNK];  // record words 0 - 5
    float4 walk[2][LF_CHUNK]; // walk constants 4, 5
};

// for the differentiable channels' kernel: record words 0 - 3, voxel size, WalkRec::w5.w
template <bool SMOOTH>
struct LeafSmooth
{
};
template <>
struct LeafSmooth<true>
{
    float4 rec[4][LF_CHUNK];
    float vs[LF_CHUNK];
    uint32_t exact_d[LF_CHUNK];
};

template <bool SMOOTH>
struct LeafChunk : LeafSmooth<SMOOTH>
{
    float4 q6[LF_CHUNK], q7[LF_CHUNK]; // record words 6, 7
    float4 walk[4][LF_CHUNK];          // walk constants 0 - 3
    // per (leaf, Gaussian)
    float4 tc[LF_CHUNK]; // the test's c at the box origin's voxel, lo_t
    float4 tb[LF_CHUNK]; // 65536 / ny rounded up (exact division below 64), ny | nz << 8 | leaf test failed << 16 (check
                         // mode), j << 9 | box origin's leaf_n, h_2
    float4 al[LF_CHUNK]; // lo0, the colour bytes of the RGBA8 value
    float4 aa[LF_CHUNK]; // 2^24 + 2 anchor x, y, z, h_2
    uint64_t win[LF_CHUNK]; // reference windows: of the box's fragments, ~0 if they lie in several
    uint32_t gid[LF_CHUNK];
    uint32_t cstart[LF_CHUNK]; // first column of box j (boxes past the chunk's count: the end)
    uint32_t cols;             // all columns
    uint32_t pad;
};

// Per-voxel sums as two 32-bit words (acc_add)
struct LeafAcc
{
    uint32_t dens[2][512];
    uint32_t col[3][2][512];
    uint32_t rgba[512];       // packed RGBA8 maximum
    unsigned long long wmin;  // creation window (reference node order)
};

template <bool SMOOTH>
struct LeafQSmem
{
    LeafStage st;
    LeafChunk<SMOOTH> ch[3];
    LeafAcc acc;
    uint32_t mask[3][16]; // value masks of the leaf being tested and of the two before it
    uint16_t queue[2][lf_cap<SMOOTH>];
    uint32_t defer[SMOOTH ? 1 : LP_THREADS / 32][64]; // per warp: the leaf's pairs whose RGBA8 byte is open
    uint32_t qn[3];
    int32_t nxt_o[2][3]; // the next chunk (by phase parity): leaf origin, sorted pair range and count
    uint32_t nxt_q0[2], nxt_p1[2], nxt_cnt[2];
    uint32_t cand_next[2];
    uint32_t cand;
};

static_assert(sizeof(LeafQSmem<false>) <= 56 * 1024 && sizeof(LeafQSmem<true>) <= 56 * 1024, "four CTAs of the leaf walk fit an SM's 228 KB (1 KB of it reserved per CTA)");

// One term of an exact fixed-point sum, (hi, lo) += (xh, xl) with the carry from
// the low word's old value: the total is the same integer in any order.  A
// 64-bit add in shared memory is a compare-and-swap loop (several round trips
// where lanes meet on a voxel); 32-bit adds are single instructions, and the
// high word is touched only when something reaches it (about once in 1 / alpha
// terms).
__device__ __forceinline__ void acc_add(uint32_t* lo, uint32_t* hi, uint32_t xl, uint32_t xh)
{
    const uint32_t old = atomicAdd(lo, xl);
    const uint32_t up = xh + (old + xl < old ? 1u : 0u);
    if (up)
        atomicAdd(hi, up);
}
__device__ __forceinline__ void acc_add(uint32_t* lo, uint32_t* hi, unsigned long long x)
{
    acc_add(lo, hi, (uint32_t)x, (uint32_t)(x >> 32));
}

// Two floats in one register pair; add and fma round each half as the scalar
// instruction does and take one issue slot for both.
struct F2
{
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi)
{
    F2 o;
    asm("mov.b64 %0, {%1, %2};" : "=l"(o.v) : "f"(lo), "f"(hi));
    return o;
}
__device__ __forceinline__ float2 f2_get(F2 a)
{
    float2 o;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(a.v));
    return o;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c)
{
    F2 o;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(o.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return o;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b)
{
    F2 o;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(o.v) : "l"(a.v), "l"(b.v));
    return o;
}

// The z run of one column (fx, fy voxels from the box's origin): which of its nz
// voxels surely pass, and which need the reference test (leaf_test_columns has
// the bounds).  q0 .. q3, h2: the test's constants (LeafChunk::tc, walk, tb).
__device__ __forceinline__ uint32_t column_test(const float4& q0, const float4& q1, const float4& q2, const float4& q3,
                                                float h2, float fx, float fy, uint32_t nz, uint32_t& unsure)
{
    const float b0 = VOX_FFMA(fy, q2.x, VOX_FFMA(fx, q1.x, q0.x)), b1 = VOX_FFMA(fy, q2.y, VOX_FFMA(fx, q1.y, q0.y)),
                b2 = VOX_FFMA(fy, q2.z, VOX_FFMA(fx, q1.z, q0.z));
    const F2 B0 = f2(b0, b0), B1 = f2(b1, b1), B2 = f2(b2, b2);
    const F2 S0 = f2(q3.x, q3.x), S1 = f2(q3.y, q3.y), S2 = f2(q3.z, q3.z);
    const F2 nlo = f2(-q0.w, -q0.w), hi2 = f2(q1.w, q1.w), m1 = f2(-1.f, -1.f), m2 = f2(-2.f, -2.f), zero = f2(0.f, 0.f);
    const float h0 = q2.w, h1 = q3.w;
    const uint32_t steps = (nz + 1u) >> 1; // voxels (2 k - 2, 2 k - 1) for k = steps .. 1
    const float ft = (float)(2u * steps);
    F2 K = f2(ft - 2.f, ft - 1.f);
    uint32_t pass = 0, fail = 0;
#pragma unroll 1
    for (uint32_t k = steps; k; k--)
    {
        const float2 c0 = f2_get(f2_fma(K, S0, B0)), c1 = f2_get(f2_fma(K, S1, B1)), c2 = f2_get(f2_fma(K, S2, B2));
        const F2 x0 = f2(__saturatef(VOX_FSUB(fabsf(c0.x), h0)), __saturatef(VOX_FSUB(fabsf(c0.y), h0)));
        const F2 x1 = f2(__saturatef(VOX_FSUB(fabsf(c1.x), h1)), __saturatef(VOX_FSUB(fabsf(c1.y), h1)));
        const F2 x2 = f2(__saturatef(VOX_FSUB(fabsf(c2.x), h2)), __saturatef(VOX_FSUB(fabsf(c2.y), h2)));
        const F2 D = f2_fma(x2, x2, f2_fma(x1, x1, f2_fma(x0, x0, zero)));
        const float2 dl = f2_get(f2_add(D, nlo)), dh = f2_get(f2_fma(D, m1, hi2));
        pass = __funnelshift_l(__float_as_uint(dl.y), pass, 1);
        pass = __funnelshift_l(__float_as_uint(dl.x), pass, 1);
        fail = __funnelshift_l(__float_as_uint(dh.y), fail, 1);
        fail = __funnelshift_l(__float_as_uint(dh.x), fail, 1);
        K = f2_add(K, m2);
    }
    const uint32_t valid = (1u << nz) - 1u;
    unsure = ~(pass | fail) & valid;
    return pass & valid;
}

// The forward walk's test: the boxes of a chunk, one box column per lane; the
// passing (Gaussian, voxel) pairs are appended to queue (entry j << 9 | leaf_n)
// and their voxels set in mask (the leaf's value mask as 32-bit words).  The
// results are voxel_local_aabb + aabb_hits_unit_sphere per voxel, decided where
// possible from the float channels' local AABB as centre and half width
// (leaf_consts; per row x = max(|c| - h, 0) is the AABB's point nearest to
// zero, 1-Lipschitz in c and h).  Per row that is within delta_r = 1.5 dab_r of
// the reference's, so the vectors of the three differ by eta <= Delta = sum
// delta_r in norm.  The reference passes a voxel when its fl-evaluated 1 - S >
// 0: surely if S < 1 - 2^-22 (three subtractions and squares of values below 1)
// and surely not if S > 1 + 2^-20.  With D the fma-summed squares of the float
// values (relative error <= 3 2^-24) and Delta <= 1/16, (sqrt(D) + eta)^2 <
// 1 - 2^-22 holds when D < 1 - (2 Delta + 2^-19), and (sqrt(D) - eta)^2 > 1 +
// 2^-20 when D > 1 + (2 Delta + Delta^2 + 2^-18) (the slack covers the
// roundings of the thresholds themselves).  The kernel holds c, h and the steps
// halved, D and the thresholds quartered: a halved x saturates at 1 (a quarter
// of D at least 1: far above the fail threshold).  Voxels between the
// thresholds, and every voxel of a (leaf, Gaussian) with Delta > 1/16 (lo_t =
// -1, hi_t = inf; also NaN), take the reference test.  In CHECK mode every
// voxel also takes it and a difference sets ERR_BOUNDS.
//
// The walk is bound by instruction issue, and integer and min / max instructions
// run at half the rate of FP32 ones, so the z loop has two voxels per step in
// packed FP32 arithmetic, |c| - h clamped by the addition itself (.sat), and the
// comparisons as sign bits of differences shifted into the masks (highest z
// first): 11 instructions per voxel for 24.  With acc_add, the constants as
// 16-byte words and the value masks set here instead of counted per pair, the
// walk of 2M Gaussians (1.6e9 pairs) 42.9 -> 34.1 ms.
template <bool CHECK, class Chunk>
__device__ __forceinline__ void leaf_test_columns(const LeafPassParams& P, const Chunk& C, const int32_t o[3],
                                                  uint16_t* queue, uint32_t* qcount, uint32_t* mask, int t, int lane,
                                                  uint32_t rot)
{
    const uint32_t T = C.cols;
    const uint32_t cs = lane < LF_CHUNK ? C.cstart[lane] : 0x7fffffffu;
    const uint32_t le = 0xffffffffu >> (31 - lane);
    // rounds of 32 columns dealt to the warps in turn, starting at warp rot (mod 8):
    // the deal continues where the alpha's rounds of 32 pairs stopped, so the warps'
    // loads in a phase differ by at most one round
    const uint32_t first = (uint32_t)(((t >> 5) - (int)(rot & 7u)) & 7);
    for (uint32_t e0 = first * 32u; e0 < T; e0 += LP_THREADS)
    {
        // j: the last box whose first column is <= e (a box with columns: every
        // emitted leaf meets its Gaussian's bbox); sj its first column
        const uint32_t rel = cs - e0;
        const uint32_t heads = __reduce_or_sync(0xffffffffu, rel - 1u < 31u ? 1u << rel : 0u);
        const uint32_t j = (uint32_t)(__popc(__ballot_sync(0xffffffffu, cs <= e0)) - 1 + __popc(heads & le)) & 31u;
        const uint32_t sj = __shfl_sync(0xffffffffu, cs, (int)j);
        const uint32_t e = e0 + (uint32_t)lane;
        uint32_t zmask = 0, ebase = 0;
        if (e < T)
        {
            const float4 q0 = C.tc[j], q1 = C.walk[0][j], q2 = C.walk[1][j], q3 = C.walk[2][j], q4 = C.tb[j];
            const uint32_t ext = __float_as_uint(q4.y), ny = ext & 255u, nz = (ext >> 8) & 255u;
            const uint32_t local = e - sj;
            const uint32_t dx = (local * __float_as_uint(q4.x)) >> 16;
            const uint32_t dy = local - dx * ny;
            ebase = __float_as_uint(q4.z) + (dx << 6) + (dy << 3);
            uint32_t unsure;
            zmask = column_test(q0, q1, q2, q3, q4.w, (float)dx, (float)dy, nz, unsure);
            // the reference test of one voxel, from the record (nothing of the column kept live)
            auto exact_voxel = [&](uint32_t k) -> uint32_t {
                const GaussRec R = P.recs[C.gid[j]];
                const uint32_t n = (ebase & 511u) + k;
                const Aabb b = voxel_local_aabb(R, rinv_of(R), P.walk[C.gid[j]].w5.z, o[0] + (int32_t)(n >> 6),
                                                o[1] + (int32_t)((n >> 3) & 7u), o[2] + (int32_t)(n & 7u));
                return aabb_hits_unit_sphere(b) ? 1u << k : 0u;
            };
            for (uint32_t m = unsure; m; m &= m - 1u)
                zmask |= exact_voxel((uint32_t)(__ffs(m) - 1));
            if (CHECK)
            {
                uint32_t ex = 0;
                for (uint32_t k = 0; k < nz; k++)
                    ex |= exact_voxel(k);
                if (ex != zmask)
                    atomicOr(P.err, ERR_BOUNDS); // a classification differs from the reference test
                if (zmask && ext >> 16)
                    atomicOr(P.err, ERR_BOUNDS); // the leaf test would have dropped a passing voxel
            }
            if (zmask)
                atomicOr(&mask[(ebase & 511u) >> 5], zmask << (ebase & 31u));
        }
        // queue slots: warp inclusive scan of the pass counts, one shared atomic per warp
        const uint32_t np = (uint32_t)__popc(zmask);
        uint32_t incl = np;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off)
                incl += y;
        }
        uint32_t qb = 0;
        if (lane == 31 && incl)
            qb = atomicAdd(qcount, incl);
        qb = __shfl_sync(0xffffffffu, qb, 31) + incl - np;
        uint16_t* dst = queue + qb;
#pragma unroll
        for (uint32_t k = 0; k < 8; k++)
            if (zmask & (1u << k))
                *dst++ = (uint16_t)(ebase + k);
    }
}

// the part of a Gaussian's bbox inside the leaf at o, leaf-relative
struct LeafBox
{
    int32_t lo[3];
    uint32_t nx, ny, nz; // nx = 0: empty
};
__device__ __forceinline__ LeafBox leaf_box(const GaussRec& R, const int32_t o[3])
{
    LeafBox b;
    const int32_t x0 = max(R.q4.x, o[0]) - o[0], x1 = min(R.q4.x + R.q5.x - 1, o[0] + 7) - o[0];
    const int32_t y0 = max(R.q4.y, o[1]) - o[1], y1 = min(R.q4.y + R.q5.y - 1, o[1] + 7) - o[1];
    const int32_t z0 = max(R.q4.z, o[2]) - o[2], z1 = min(R.q4.z + R.q5.z - 1, o[2] + 7) - o[2];
    const bool empty = x1 < x0 || y1 < y0 || z1 < z0;
    b.lo[0] = x0;
    b.lo[1] = y0;
    b.lo[2] = z0;
    b.nx = empty ? 0u : (uint32_t)(x1 - x0 + 1);
    b.ny = empty ? 1u : (uint32_t)(y1 - y0 + 1);
    b.nz = empty ? 1u : (uint32_t)(z1 - z0 + 1);
    return b;
}

// the last warp, each lane with its own box's columns and voxels (0 past the
// Gaussians at hand): the chunk takes the first boxes of lf_cap voxels together;
// its column prefix, and how many Gaussians it has
template <bool SMOOTH>
__device__ __forceinline__ uint32_t leaf_stage_prefix(LeafChunk<SMOOTH>& C, int lane, uint32_t avail, uint32_t cols, uint32_t voxels)
{
    uint32_t v = voxels;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off)
            v += y;
    }
    const uint32_t cnt = (uint32_t)__popc(__ballot_sync(0xffffffffu, (uint32_t)lane < avail && v <= lf_cap<SMOOTH>));
    const uint32_t mine = (uint32_t)lane < cnt ? cols : 0u;
    uint32_t c = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, c, off);
        if (lane >= off)
            c += y;
    }
    if (lane < LF_CHUNK)
        C.cstart[lane] = c - mine;
    if (lane == 31)
        C.cols = c;
    return cnt;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// record and walk constants of sorted leaf pair q into slot j (asynchronous); returns its Gaussian id
template <bool SMOOTH>
__device__ __forceinline__ uint32_t leaf_stage_issue(const LeafPassParams& P, LeafStage& T, LeafChunk<SMOOTH>& C, int j,
                                                     uint32_t q)
{
    const uint32_t g = P.pair_gid[q];
    const float4* rec = reinterpret_cast<const float4*>(&P.recs[g]);
    const float4* walk = reinterpret_cast<const float4*>(&P.walk[g]);
#pragma unroll
    for (int w = 0; w < 6; w++)
        cp_async16(&T.rec[w][j], rec + w);
    cp_async16(&C.q6[j], rec + 6);
    cp_async16(&C.q7[j], rec + 7);
#pragma unroll
    for (int w = 0; w < 4; w++)
        cp_async16(&C.walk[w][j], walk + w);
    cp_async16(&T.walk[0][j], walk + 4);
    cp_async16(&T.walk[1][j], walk + 5);
    if constexpr (SMOOTH)
#pragma unroll
        for (int w = 0; w < 4; w++)
            cp_async16(&C.rec[w][j], rec + w);
    return g;
}

// the reference's window of voxel (x, y, z)'s fragment of Gaussian g: its x-major
// index in the bbox (gaussian_frag_alloc.slang:55-58) after the Gaussian's batch offset
__device__ __forceinline__ uint64_t frag_window(const LeafPassParams& P, uint32_t g, const int4& b0, const int4& ext,
                                                int32_t x, int32_t y, int32_t z)
{
    const int64_t batch = (int64_t)g / REF_PRIM_BATCH;
    const uint64_t r = (uint64_t)(x - b0.x) * (uint64_t)ext.y * (uint64_t)ext.z + (uint64_t)(y - b0.y) * (uint64_t)ext.z +
                       (uint64_t)(z - b0.z);
    return P.win_before[batch] + (P.frag_off[g] - P.frag_off[batch * REF_PRIM_BATCH] + r) / REF_WINDOW;
}

// once the record landed: the chunk's constants of Gaussian j, and its box's columns and voxels
template <bool CHECK, bool WINDOW, bool SMOOTH>
__device__ __forceinline__ void leaf_stage_box(const LeafPassParams& P, const LeafStage& T, LeafChunk<SMOOTH>& C, int j, uint32_t q,
                                               uint32_t g, const int32_t o[3], uint32_t& cols, uint32_t& voxels)
{
    GaussRec R;
    R.q4 = *reinterpret_cast<const int4*>(&T.rec[4][j]);
    R.q5 = *reinterpret_cast<const int4*>(&T.rec[5][j]);
    const LeafBox b = leaf_box(R, o);
    int32_t r0[3];
#pragma unroll
    for (int a = 0; a < 3; a++)
        r0[a] = anchor_of((&R.q4.x)[a], (&R.q5.x)[a], o[a]);
    R.q0 = T.rec[0][j];
    R.q1 = T.rec[1][j];
    R.q2 = T.rec[2][j];
    R.q3.x = T.rec[3][j].x;
    const float mu[3] = { R.q0.x, R.q0.y, R.q0.z };
    const float4 w0 = C.walk[0][j], w1 = C.walk[1][j], w2 = C.walk[2][j], w4 = T.walk[0][j], w5 = T.walk[1][j];
    const LeafConst K = leaf_consts(rinv_of(R), mu, w0, w1, w2, w4, w5.z, o, r0);
    const float bx = (float)(b.lo[0] - r0[0]), by = (float)(b.lo[1] - r0[1]), bz = (float)(b.lo[2] - r0[2]);
    float c[3];
#pragma unroll
    for (int r = 0; r < 3; r++)
        c[r] = VOX_FFMA(bz, (&w2.x)[r], VOX_FFMA(by, (&w1.x)[r], VOX_FFMA(bx, (&w0.x)[r], K.c[r])));
    const uint32_t failed = CHECK ? (uint32_t)P.emit_flag[P.vals[q]] : 0u;
    C.tc[j] = make_float4(c[0], c[1], c[2], w5.x);
    C.tb[j] = make_float4(__uint_as_float((65536u + b.ny - 1u) / b.ny), __uint_as_float(b.ny | b.nz << 8 | failed << 16),
                          __uint_as_float((uint32_t)j << 9 | (uint32_t)(b.lo[0] << 6 | b.lo[1] << 3 | b.lo[2])), w4.w);
    C.al[j] = make_float4(K.lo0[0], K.lo0[1], K.lo0[2], w5.y);
    C.aa[j] = make_float4(16777216.f + (float)(2 * r0[0]), 16777216.f + (float)(2 * r0[1]), 16777216.f + (float)(2 * r0[2]),
                          w4.w);
    C.gid[j] = g;
    if constexpr (SMOOTH)
    {
        C.vs[j] = w5.z;
        C.exact_d[j] = w5.w != 0.f ? 1u : 0u;
    }
    if (WINDOW)
    {
        // fragments are numbered x-major, so the box's lie between its two corners'
        const int32_t x = o[0] + b.lo[0], y = o[1] + b.lo[1], z = o[2] + b.lo[2];
        const uint64_t first = frag_window(P, g, R.q4, R.q5, x, y, z);
        const uint64_t last = frag_window(P, g, R.q4, R.q5, x + (int32_t)b.nx - 1, y + (int32_t)b.ny - 1, z + (int32_t)b.nz - 1);
        C.win[j] = first == last ? first : ~0ull;
    }
    cols = b.nx * b.ny;
    voxels = cols * b.nz;
}

// BYTES: the RGBA8 values alone, for callers that take no float channels (the
// reference-facing entries): no sums, the alpha only as far as its byte is bounded.
// The entry on 30k host arrays 1.71 -> 1.60 ms, on 500k 8.93 -> 8.58 ms.
template <bool CHECK, bool WINDOW, bool SMOOTH, int MINB, bool BYTES>
__global__ void __launch_bounds__(LP_THREADS, MINB) k_leaf_pass(LeafPassParams P, uint32_t* counter)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LeafQSmem<SMOOTH>& S = *reinterpret_cast<LeafQSmem<SMOOTH>*>(smem_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool stager = warp == LP_THREADS / 32 - 1; // lane j < LF_CHUNK stages Gaussian j of the next chunk
    if (t == 0)
    {
        S.cand = atomicAdd(counter, 1u);
        S.cand_next[0] = atomicAdd(counter, 1u);
        S.qn[0] = S.qn[1] = S.qn[2] = 0;
        S.acc.wmin = ~0ull;
    }
    for (int i = t; i < 9 * 512; i += LP_THREADS) // the sums and the RGBA8 maxima
        (&S.acc.dens[0][0])[i] = 0;
    if (t < 48)
        S.mask[0][t] = 0;
    __syncthreads();
    // the chunk being tested (t*), the chunk whose alpha runs (a*), the leaf being flushed (f*)
    int64_t tc = S.cand;
    if (tc >= P.NCL)
        return;
    int64_t cn = S.cand_next[0];
    int32_t to[3];
    {
        const int4 o4 = P.cand_org[tc];
        to[0] = o4.x;
        to[1] = o4.y;
        to[2] = o4.z;
    }
    // stagers: the next leaf's origin and pair range, loaded as soon as the leaf
    // is known and used at the current leaf's end; lane 0 claims the leaf after
    // it just as early, so no leaf end waits on global memory
    int4 pre_org = make_int4(0, 0, 0, 0);
    uint32_t pre_q0 = 0, pre_p1 = 0, cn2 = 0;
    bool cn_fresh = true;
    uint32_t tq0 = P.cand_start[tc], tp1 = P.cand_start[tc + 1];
    if (stager)
    {
        uint32_t cols = 0, voxels = 0;
        const uint32_t avail = min((uint32_t)LF_CHUNK, tp1 - tq0);
        if ((uint32_t)lane < avail)
        {
            const uint32_t g = leaf_stage_issue<SMOOTH>(P, S.st, S.ch[0], lane, tq0 + (uint32_t)lane);
            cp_async_wait_all();
            leaf_stage_box<CHECK, WINDOW>(P, S.st, S.ch[0], lane, tq0 + (uint32_t)lane, g, to, cols, voxels);
        }
        const uint32_t cnt = leaf_stage_prefix(S.ch[0], lane, avail, cols, voxels);
        if (lane == 0)
            S.nxt_cnt[1] = cnt;
    }
    __syncthreads();
    uint32_t tcnt = S.nxt_cnt[1]; // (phase 0 fills the other)
    bool t_valid = true, a_valid = false, f_valid = false, a_leaf_end = false;
    int tm = 0, am = 0, fm = 0; // value mask buffers, one per leaf in turn
    int64_t ac = 0, fc = 0;
    int32_t ao[3] = { 0, 0, 0 };
    unsigned long long leaf_pairs = 0, all_pairs = 0; // thread 0's
    uint32_t tleaf0 = tq0, aleaf0 = 0, alocal = 0;    // first pair of the leaf; the alpha's chunk's place after it
    uint32_t dn = 0;                                  // this warp's deferred pairs (warp-uniform)
    uint32_t i = 0; // phase
    while (t_valid || a_valid || f_valid)
    {
        const int tb = (int)(i % 3u), ab = (int)((i + 2u) % 3u), nb = (int)((i + 1u) % 3u);
        const bool t_leaf_end = t_valid && tq0 + tcnt >= tp1;
        const int64_t nc = t_leaf_end ? cn : tc;
        const bool n_valid = t_valid && nc < P.NCL;
        if (stager && cn_fresh)
        {
            if (cn < P.NCL)
            {
                pre_org = P.cand_org[cn];
                pre_q0 = P.cand_start[cn];
                pre_p1 = P.cand_start[cn + 1];
                if (lane == 0)
                    cn2 = atomicAdd(counter, 1u);
            }
        }
        cn_fresh = false;
        // ---- stagers: the next chunk's pair range, its record copies
        uint32_t nq0 = 0, np1 = 0, avail = 0, ng = 0;
        if (stager && n_valid)
        {
            nq0 = t_leaf_end ? pre_q0 : tq0 + tcnt;
            np1 = t_leaf_end ? pre_p1 : tp1;
            avail = min((uint32_t)LF_CHUNK, np1 - nq0);
            if ((uint32_t)lane < avail)
                ng = leaf_stage_issue<SMOOTH>(P, S.st, S.ch[nb], lane, nq0 + (uint32_t)lane);
        }
        // ---- flush of the leaf whose last alpha ran in the previous phase
        if (f_valid)
        {
            LeafAcc& A = S.acc;
            const uint32_t* mask = S.mask[fm];
#pragma unroll
            for (int h = 0; h < 2; h++)
            {
                const uint32_t n = (uint32_t)(t + 256 * h);
                if ((mask[warp + 8 * h] >> lane) & 1u)
                {
                    const uint64_t slot = (uint64_t)fc * 512u + n;
                    P.s_rgba[slot] = A.rgba[n];
                    A.rgba[n] = 0;
                    if constexpr (!BYTES)
                    {
                        const float ds = fx_to_float((unsigned long long)A.dens[1][n] << 32 | A.dens[0][n]);
                        float col[3];
#pragma unroll
                        for (int k = 0; k < 3; k++)
                        {
                            col[k] = fx_to_float((unsigned long long)A.col[k][1][n] << 32 | A.col[k][0][n]);
                            if (!SMOOTH)
                                col[k] = ds > 0.f ? VOX_FDIV(col[k], ds) : 0.f;
                        }
                        P.s_dens[slot] = ds;
                        P.s_col[3 * slot + 0] = col[0];
                        P.s_col[3 * slot + 1] = col[1];
                        P.s_col[3 * slot + 2] = col[2];
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            (&A.dens[0][0])[512 * k + n] = 0;
                    }
                }
            }
            if (t < 16)
                reinterpret_cast<uint32_t*>(P.cand_mask + 8 * (uint64_t)fc)[t] = mask[t];
            if (t == 0)
            {
                P.cand_pairs[fc] = leaf_pairs;
                all_pairs += leaf_pairs;
                leaf_pairs = 0;
                if (WINDOW)
                {
                    P.cand_wkey[fc] = A.wmin;
                    A.wmin = ~0ull;
                }
            }
            __syncthreads(); // the next leaf's alpha reuses the accumulators
            if (t < 16)
                S.mask[fm][t] = 0; // filled again by the leaf after next, from the next phase on
        }
        const uint32_t a_rounds = a_valid ? (S.qn[ab] + 31u) / 32u : 0u; // the alpha's rounds of 32 pairs
        // ---- alpha of the previous chunk, one queued pair per thread.  A pair whose
        // RGBA8 byte the bound leaves open (1 - 2%) and that may be its voxel's
        // maximum goes to its warp's list, which lasts through the leaf, and the
        // reference's byte is evaluated 32 pairs at a time (from the records in global
        // memory) or at the leaf's end, each warp its own: one warp taking all that
        // were left held the others up at the barrier (walk of 4999 Gaussians 120 us,
        // now 111; of 64 clouds 8.11 ms, now 7.88; with each pair evaluated on the spot
        // 102 us and 8.00 ms, but 100k 600 us for 565).  The smooth mode, whose records
        // are in shared memory, evaluates on the spot (500k 2.14 -> 2.05 ms).
        if (a_valid)
        {
            const LeafChunk<SMOOTH>& C = S.ch[ab];
            LeafAcc& A = S.acc;
            const uint16_t* queue = S.queue[(i + 1u) & 1u];
            const uint32_t qn = S.qn[ab];
            if (t == 0)
                leaf_pairs += qn;
            uint32_t* dq = S.defer[SMOOTH ? 0 : warp];
            // the reference's byte of voxel n and the leaf's Gaussian at position l of its pairs
            auto ref_byte = [&](uint32_t l, uint32_t n) {
                const uint32_t g = P.pair_gid[aleaf0 + l];
                const GaussRec R = P.recs[g];
                const uint32_t a8 = ref_alpha_byte(R, P.walk[g].w5.z, ao[0] + (int32_t)(n >> 6),
                                                   ao[1] + (int32_t)((n >> 3) & 7u), ao[2] + (int32_t)(n & 7u));
                atomicMax(&A.rgba[n], (a8 << 24) | __float_as_uint(P.walk[g].w5.y));
            };
            for (uint32_t e0 = (uint32_t)(t & ~31); e0 < qn; e0 += LP_THREADS) // warp-uniform trip count
            {
                const uint32_t e = e0 + (uint32_t)lane;
                bool defer = false;
                uint32_t q = 0;
                if (e < qn)
                {
                    q = queue[e];
                    const uint32_t j = q >> 9, n = q & 511u;
                    const float4 al = C.al[j], q7 = C.q7[j], w3 = C.walk[3][j], w0 = C.walk[0][j], w1 = C.walk[1][j],
                                 w2 = C.walk[2][j], aa = C.aa[j], q6 = C.q6[j];
                    float a;
                    AlphaF af;
                    {
                        const float lo0[3] = { al.x, al.y, al.z }, W4[3] = { w1.w, w2.w, aa.w };
                        const float h[3][3] = { { w0.x, w1.x, w2.x }, { w0.y, w1.y, w2.y }, { w0.z, w1.z, w2.z } };
                        // twice the voxels from the anchor, exactly (a last place is 2 from 2^24 on)
                        const float fx = VOX_FSUB(__uint_as_float(0x4b800000u | (n >> 6)), aa.x),
                                    fy = VOX_FSUB(__uint_as_float(0x4b800000u | ((n >> 3) & 7u)), aa.y),
                                    fz = VOX_FSUB(__uint_as_float(0x4b800000u | (n & 7u)), aa.z);
                        const Aabb box = stable_leaf_aabb(lo0, W4, h, fx, fy, fz);
                        if constexpr (SMOOTH || BYTES)
                            af = pair_alpha_approx(q6, box);
                        else
                            af = pair_alpha_f_ex(q6, box);
                    }
                    bool decided;
                    uint32_t most;
                    uint32_t a8 = alpha_byte_bound<SMOOTH || BYTES>(q6, q7.w, af, w3, decided, most);
                    // an open pair that cannot exceed the voxel's maximum so far needs no byte
                    // (a8 <= most: the maximum below changes nothing).  Of a voxel's k-th pair
                    // that holds but for about one in k: the walk of 2M Gaussians 26.8 -> 26.1 ms
                    defer = !decided && *(volatile uint32_t*)&A.rgba[n] < (most | __float_as_uint(al.w));
                    if (CHECK && decided &&
                        a8 >> 24 != ref_alpha_byte(P.recs[C.gid[j]], P.walk[C.gid[j]].w5.z, ao[0] + (int32_t)(n >> 6),
                                                   ao[1] + (int32_t)((n >> 3) & 7), ao[2] + (int32_t)(n & 7)))
                        atomicOr(P.err, ERR_BOUNDS); // the margin failed to cover the reference's byte
                    if constexpr (SMOOTH)
                    {
                        const int32_t x = ao[0] + (int32_t)(n >> 6), yy = ao[1] + (int32_t)((n >> 3) & 7),
                                      zz = ao[2] + (int32_t)(n & 7);
                        GaussRec R;
                        R.q0 = C.rec[0][j];
                        R.q1 = C.rec[1][j];
                        R.q2 = C.rec[2][j];
                        R.q3 = C.rec[3][j];
                        const float mu[3] = { R.q0.x, R.q0.y, R.q0.z }, inv_s[3] = { R.q3.y, R.q3.z, R.q3.w };
                        SmoothTerms st;
                        a = smooth_kernel(mu, inv_s, q6.x, rinv_of(R), C.vs[j], C.exact_d[j] != 0u, x, yy, zz, st);
                        if (defer) // the records are at hand
                        {
                            R.q6 = q6;
                            R.q7 = q7;
                            a8 = ref_alpha_byte(R, C.vs[j], x, yy, zz) << 24;
                            defer = false;
                        }
                    }
                    else if constexpr (!BYTES)
                        a = q7.w != 0.f ? 0.f : af.a1;
                    if (!defer)
                        atomicMax(&A.rgba[n], a8 | __float_as_uint(al.w));
                    if constexpr (!BYTES)
                    {
                        if (a < 1.f && (int32_t)__float_as_uint(w3.w) >= 0)
                        {
                            // the colours and the opacity in [0, 1], so alpha and terms in [0, 1):
                            // below 2^32 units
                            const float c0 = VOX_FMUL(a, q7.x), c1 = VOX_FMUL(a, q7.y), c2 = VOX_FMUL(a, q7.z);
                            acc_add(&A.dens[0][n], &A.dens[1][n], __float2uint_rn(VOX_FMUL(a, FX_SCALE)), 0u);
                            acc_add(&A.col[0][0][n], &A.col[0][1][n], __float2uint_rn(VOX_FMUL(c0, FX_SCALE)), 0u);
                            acc_add(&A.col[1][0][n], &A.col[1][1][n], __float2uint_rn(VOX_FMUL(c1, FX_SCALE)), 0u);
                            acc_add(&A.col[2][0][n], &A.col[2][1][n], __float2uint_rn(VOX_FMUL(c2, FX_SCALE)), 0u);
                        }
                        else
                        {
                            // where the power's base b in pair_alpha_f_ex is negative (near the
                            // centre of an opacity above 1), or 1 with an infinite exponent, the
                            // alpha is 0, as the oracle's (a base of 1 and a finite one give 0 too)
                            const float b = VOX_FSUB(1.f, af.a);
                            if (!SMOOTH && (b < 0.f || b == 1.f))
                                a = 0.f;
                            acc_add(&A.dens[0][n], &A.dens[1][n], fx_of_unit(a));
                            acc_add(&A.col[0][0][n], &A.col[0][1][n], fx_of(VOX_FMUL(a, q7.x)));
                            acc_add(&A.col[1][0][n], &A.col[1][1][n], fx_of(VOX_FMUL(a, q7.y)));
                            acc_add(&A.col[2][0][n], &A.col[2][1][n], fx_of(VOX_FMUL(a, q7.z)));
                        }
                    }
                    if (WINDOW)
                    {
                        unsigned long long wk = C.win[j];
                        if (wk == ~0ull)
                        {
                            const GaussRec& R = P.recs[C.gid[j]];
                            wk = frag_window(P, C.gid[j], R.q4, R.q5, ao[0] + (int32_t)(n >> 6),
                                             ao[1] + (int32_t)((n >> 3) & 7), ao[2] + (int32_t)(n & 7));
                        }
                        // read first: a 64-bit minimum in shared memory is a compare-and-swap loop,
                        // and nearly every pair's window is no earlier than the one there
                        if (wk < *(volatile unsigned long long*)&A.wmin)
                            atomicMin(&A.wmin, wk);
                    }
                }
                if constexpr (!SMOOTH)
                {
                    // a list entry holds the pair's position among the leaf's pairs in 23 bits;
                    // a leaf of more pairs evaluates the rest at once
                    const uint32_t l = alocal + (q >> 9);
                    if (defer && l >= 1u << 23)
                    {
                        ref_byte(l, q & 511u);
                        defer = false;
                    }
                    const uint32_t bal = __ballot_sync(0xffffffffu, defer);
                    if (bal)
                    {
                        if (defer)
                            dq[dn + (uint32_t)__popc(bal & ((1u << lane) - 1u))] = l << 9 | (q & 511u);
                        dn += (uint32_t)__popc(bal);
                        if (dn >= 32u) // dn <= 63: a batch of 32, the rest moved to the front
                        {
                            __syncwarp();
                            const uint32_t d = dq[lane];
                            ref_byte(d >> 9, d & 511u);
                            const uint32_t rest = dn - 32u;
                            const uint32_t mv = (uint32_t)lane < rest ? dq[32 + lane] : 0u;
                            __syncwarp();
                            if ((uint32_t)lane < rest)
                                dq[lane] = mv;
                            __syncwarp();
                            dn = rest;
                        }
                    }
                }
            }
            // at the leaf's end, the open pairs left in the warp's list (fewer than 32)
            if (a_leaf_end && dn)
            {
                __syncwarp();
                if ((uint32_t)lane < dn)
                {
                    const uint32_t d = dq[lane];
                    ref_byte(d >> 9, d & 511u);
                }
                dn = 0;
                __syncwarp();
            }
        }
        // ---- test of this chunk
        if (t_valid)
            leaf_test_columns<CHECK>(P, S.ch[tb], to, S.queue[i & 1u], &S.qn[tb], S.mask[tm], t, lane, a_rounds);
        // the counter the test of phase i + 1 fills: last read by the alpha of phase i - 1
        if (t == 0)
            S.qn[nb] = 0;
        // ---- stagers: the next chunk's boxes (their own copies have landed)
        if (stager && n_valid)
        {
            int32_t no[3] = { to[0], to[1], to[2] };
            if (t_leaf_end)
            {
                no[0] = pre_org.x;
                no[1] = pre_org.y;
                no[2] = pre_org.z;
            }
            uint32_t cols = 0, voxels = 0;
            if ((uint32_t)lane < avail)
            {
                cp_async_wait_all();
                leaf_stage_box<CHECK, WINDOW>(P, S.st, S.ch[nb], lane, nq0 + (uint32_t)lane, ng, no, cols, voxels);
            }
            const uint32_t ncnt = leaf_stage_prefix(S.ch[nb], lane, avail, cols, voxels);
            if (lane == 0)
            {
                const int pp = (int)(i & 1u);
                S.nxt_o[pp][0] = no[0];
                S.nxt_o[pp][1] = no[1];
                S.nxt_o[pp][2] = no[2];
                S.nxt_q0[pp] = nq0;
                S.nxt_p1[pp] = np1;
                S.nxt_cnt[pp] = ncnt;
                if (t_leaf_end)
                    S.cand_next[pp] = cn2;
            }
        }
        __syncthreads();
        // ---- advance: flush <- alpha (at a leaf end), alpha <- test, test <- next
        f_valid = a_valid && a_leaf_end;
        fc = ac;
        fm = am;
        a_valid = t_valid;
        a_leaf_end = t_leaf_end;
        ac = tc;
        am = tm;
        aleaf0 = tleaf0;
        alocal = tq0 - tleaf0;
        ao[0] = to[0];
        ao[1] = to[1];
        ao[2] = to[2];
        if (n_valid)
        {
            const int pp = (int)(i & 1u);
            if (t_leaf_end)
            {
                cn = S.cand_next[pp];
                cn_fresh = true;
                tm = tm == 2 ? 0 : tm + 1;
            }
            tc = nc;
            tq0 = S.nxt_q0[pp];
            tp1 = S.nxt_p1[pp];
            tcnt = S.nxt_cnt[pp];
            if (t_leaf_end)
                tleaf0 = tq0;
            to[0] = S.nxt_o[pp][0];
            to[1] = S.nxt_o[pp][1];
            to[2] = S.nxt_o[pp][2];
        }
        t_valid = n_valid;
        i++;
    }
    if (t == 0 && all_pairs)
        atomicAdd((unsigned long long*)P.total_pairs, all_pairs);
}

__device__ __forceinline__ uint32_t mask_rank(const uint64_t* m, uint32_t n)
{
    uint32_t r = 0;
    for (uint32_t w = 0; w < (n >> 6); w++)
        r += __popcll(m[w]);
    return r + __popcll(m[n >> 6] & ((1ull << (n & 63)) - 1ull));
}

// The adjoint: per (leaf, Gaussian) pair, the sums of its voxel pairs' terms
// (vox_backward.cu), stored by the pair's emission index.  A warp takes 32
// consecutive sorted pairs: their constants once, a pair per lane; then, in batches
// of as many pairs as have boxes of BW_CAP voxels together, the forward's column
// test (the same pairs pass) with the batch's columns packed into the lanes, and
// pair by pair the passing voxels' terms a voxel per lane and the pair's sums
// across the warp.  RAW: 13 sums; without it, 19 (bwd_nacc).  Every sum has a fixed order (deterministic, no atomics), and no
// warp waits for another.  Bound by instruction issue (70% of the slots; gathers of
// the upstream gradients behind them): 0.78 ms for 200k Gaussians (1.17M pairs, 33M
// voxel pairs).  With the columns tested pair by pair 16 clouds took 1.20 ms for
// 1.08, 20k Gaussians 106 us for 99, 500k 1.98 ms for 1.94; batches of 512 voxels
// 1.09 ms, 100 us, 1.98 ms.
constexpr int BW_WARPS = 4;
constexpr uint32_t BW_CAP = 1024;

struct BwdWarp
{
    // constants of the 32 pairs
    float4 tc[32], tb[32], w0[32], w1[32], w2[32]; // the test's (LeafChunk)
    float4 m0[32], m1[32], m2[32], m3[32];         // mu, opacity; rows of the inverse rotation, each with its 1 / s
    float4 rgb[32];                                // colour, voxel size
    uint32_t eidx[32], gid[32], cand[32];
    uint32_t mask[16], before[16]; // the leaf's value mask and the voxels before each word
    uint32_t qs[33];               // first queue entry of each pair of the batch, and the end
    uint16_t queue[BW_CAP];        // the passing voxels of a batch of pairs
};

// v[0 .. N) summed across the warp's lanes: at each step lanes that differ in one
// bit of their number split the values, so N + N / 2 + ... shuffles do for N.
// Afterwards lane l holds the sum of value k(l) in v[0]; returns k(l) (>= N: none).
// (One instance per step, so that every index is a constant: as a loop over the
// steps 19 values were selected by comparisons, 2,000 instructions per sum.)
template <int N, int BIT = 16>
__device__ __forceinline__ void warp_sum_steps(float* v, int lane, int& first, int& width)
{
    if constexpr (BIT > 0)
    {
        constexpr int half = (N + 1) / 2;
        const bool up = (lane & BIT) != 0;
#pragma unroll
        for (int i = 0; i < half; i++)
        {
            const float hi = half + i < N ? v[half + i] : 0.f;
            const float give = up ? v[i] : hi;
            v[i] = (up ? hi : v[i]) + __shfl_xor_sync(0xffffffffu, give, BIT);
        }
        first += up ? half : 0;
        width = up ? width - half : min(width, half);
        warp_sum_steps<half, BIT / 2>(v, lane, first, width);
    }
}
template <int N>
__device__ __forceinline__ int warp_sum_split(float* v, int lane)
{
    int first = 0, width = N; // this lane's share
    warp_sum_steps<N>(v, lane, first, width);
    return width > 0 ? first : N;
}

template <bool RAW>
__global__ void __launch_bounds__(BW_WARPS * 32) k_leaf_backward(LeafPassParams P, int64_t Q)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    BwdWarp& S = reinterpret_cast<BwdWarp*>(smem_raw)[warp];
    const int64_t base = ((int64_t)blockIdx.x * BW_WARPS + warp) * 32;
    if (base >= Q)
        return;
    const int items = (int)min((int64_t)32, Q - base);
    if (lane < items)
    {
        const uint32_t q = (uint32_t)(base + lane);
        // its leaf: the last candidate whose first pair is <= q
        int64_t lo = 0, hi = P.NCL;
        while (lo < hi)
        {
            const int64_t mid = (lo + hi) >> 1;
            if (P.cand_start[mid] <= q)
                lo = mid + 1;
            else
                hi = mid;
        }
        const int4 o4 = P.cand_org[lo - 1];
        const int32_t o[3] = { o4.x, o4.y, o4.z };
        const uint32_t g = P.pair_gid[q];
        const GaussRec R = P.recs[g];
        const WalkRec W = P.walk[g];
        const LeafBox b = leaf_box(R, o);
        int32_t r0[3];
#pragma unroll
        for (int a = 0; a < 3; a++)
            r0[a] = anchor_of((&R.q4.x)[a], (&R.q5.x)[a], o[a]);
        const float mu[3] = { R.q0.x, R.q0.y, R.q0.z };
        const LeafConst K = leaf_consts(rinv_of(R), mu, W.w0, W.w1, W.w2, W.w4, W.w5.z, o, r0);
        const float bx = (float)(b.lo[0] - r0[0]), by = (float)(b.lo[1] - r0[1]), bz = (float)(b.lo[2] - r0[2]);
        float c[3];
#pragma unroll
        for (int r = 0; r < 3; r++)
            c[r] = VOX_FFMA(bz, (&W.w2.x)[r], VOX_FFMA(by, (&W.w1.x)[r], VOX_FFMA(bx, (&W.w0.x)[r], K.c[r])));
        S.tc[lane] = make_float4(c[0], c[1], c[2], W.w5.x);
        S.tb[lane] = make_float4(__uint_as_float((65536u + b.ny - 1u) / b.ny),
                                 __uint_as_float(b.ny | b.nz << 8 | (W.w5.w != 0.f ? 1u : 0u) << 16 | (b.nx * b.ny) << 17),
                                 __uint_as_float((uint32_t)(b.lo[0] << 6 | b.lo[1] << 3 | b.lo[2])), W.w4.w);
        S.w0[lane] = W.w0;
        S.w1[lane] = W.w1;
        S.w2[lane] = W.w2;
        S.m0[lane] = make_float4(mu[0], mu[1], mu[2], R.q6.x);
        S.m1[lane] = make_float4(R.q1.x, R.q1.y, R.q1.z, R.q3.y);
        S.m2[lane] = make_float4(R.q1.w, R.q2.x, R.q2.y, R.q3.z);
        S.m3[lane] = make_float4(R.q2.z, R.q2.w, R.q3.x, R.q3.w);
        S.rgb[lane] = make_float4(R.q7.x, R.q7.y, R.q7.z, W.w5.z);
        S.gid[lane] = g;
        S.cand[lane] = (uint32_t)(lo - 1);
        S.eidx[lane] = P.vals[q];
    }
    __syncwarp();
    uint32_t cur = ~0u;
    uint64_t vbase = 0;
    int32_t o[3] = { 0, 0, 0 };
    // per lane: its pair's voxels (bits 0 - 15) and columns, and the sums of both up to it
    uint32_t own = 0;
    if (lane < items)
    {
        const uint32_t ext = __float_as_uint(S.tb[lane].y), cols = ext >> 17;
        own = cols * ((ext >> 8) & 255u) | cols << 16;
    }
    uint32_t upto = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, upto, off);
        if (lane >= off)
            upto += y;
    }
    const uint32_t le = 0xffffffffu >> (31 - lane);
    for (int first = 0, last; first < items; first = last)
    {
        // ---- the batch: as many pairs as have boxes of BW_CAP voxels together
        const uint32_t before = __shfl_sync(0xffffffffu, upto - own, first);
        const uint32_t voxels = (upto & 0xffffu) - (before & 0xffffu);
        last = first + __popc(__ballot_sync(0xffffffffu, lane >= first && lane < items && voxels <= BW_CAP));
        const uint32_t T = (__shfl_sync(0xffffffffu, upto, last - 1) >> 16) - (before >> 16);
        // its pair's first column (0 before the batch, none after it)
        const uint32_t cs = lane < first ? 0u : lane < last ? ((upto - own) >> 16) - (before >> 16) : 0x7fffffffu;
        uint32_t qn = 0;
        for (uint32_t e0 = 0; e0 < T; e0 += 32)
        {
            // j: the last pair whose first column is <= e (every box has columns)
            const uint32_t rel = cs - e0;
            const uint32_t heads = __reduce_or_sync(0xffffffffu, rel - 1u < 31u ? 1u << rel : 0u);
            const uint32_t j = (uint32_t)(__popc(__ballot_sync(0xffffffffu, cs <= e0)) - 1 + __popc(heads & le)) & 31u;
            const uint32_t sj = __shfl_sync(0xffffffffu, cs, (int)j);
            const uint32_t e = e0 + (uint32_t)lane;
            uint32_t zmask = 0, n0 = 0;
            if (e < T)
            {
                const float4 tb = S.tb[j];
                const uint32_t ext = __float_as_uint(tb.y), ny = ext & 255u, nz = (ext >> 8) & 255u, local = e - sj;
                const uint32_t dx = (local * __float_as_uint(tb.x)) >> 16, dy = local - dx * ny;
                n0 = __float_as_uint(tb.z) + (dx << 6) + (dy << 3);
                uint32_t unsure;
                zmask = column_test(S.tc[j], S.w0[j], S.w1[j], S.w2[j], tb.w, (float)dx, (float)dy, nz, unsure);
                for (uint32_t m = unsure; m; m &= m - 1u)
                {
                    const uint32_t k = (uint32_t)(__ffs(m) - 1), n = n0 + k;
                    const GaussRec R = P.recs[S.gid[j]];
                    const int4 org = P.cand_org[S.cand[j]];
                    const Aabb b = voxel_local_aabb(R, rinv_of(R), S.rgb[j].w, org.x + (int32_t)(n >> 6),
                                                    org.y + (int32_t)((n >> 3) & 7u), org.z + (int32_t)(n & 7u));
                    zmask |= aabb_hits_unit_sphere(b) ? 1u << k : 0u;
                }
            }
            const uint32_t np = (uint32_t)__popc(zmask);
            uint32_t incl = np;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1)
            {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off)
                    incl += y;
            }
            const uint32_t q0 = qn + incl - np;
            if (e == sj)
                S.qs[j] = q0;
            uint16_t* dst = S.queue + q0;
#pragma unroll
            for (uint32_t k = 0; k < 8; k++)
                if (zmask & (1u << k))
                    *dst++ = (uint16_t)(n0 + k);
            qn += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0)
            S.qs[last] = qn;
        __syncwarp();
        // ---- each pair's terms and sums
        for (int it = first; it < last; it++)
        {
            const uint32_t c = S.cand[it];
            if (c != cur)
            {
                cur = c;
                const int4 o4 = P.cand_org[c];
                o[0] = o4.x;
                o[1] = o4.y;
                o[2] = o4.z;
                vbase = P.cand_vbase[c];
                const uint32_t m = lane < 16 ? reinterpret_cast<const uint32_t*>(P.cand_mask + 8 * (uint64_t)c)[lane] : 0u;
                uint32_t incl = __popc(m);
#pragma unroll
                for (int off = 1; off < 16; off <<= 1)
                {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
                    if (lane >= off)
                        incl += y;
                }
                if (lane < 16)
                {
                    S.mask[lane] = m;
                    S.before[lane] = incl - __popc(m);
                }
                __syncwarp();
            }
            const uint32_t end = S.qs[it + 1];
            const bool exact_d = (__float_as_uint(S.tb[it].y) >> 16) & 1u;
            constexpr int NACC = bwd_nacc<RAW>;
            float acc[NACC];
#pragma unroll
            for (int k = 0; k < NACC; k++)
                acc[k] = 0.f;
            for (uint32_t p = S.qs[it] + (uint32_t)lane; p < end; p += 32)
            {
                const uint32_t n = S.queue[p];
                const float4 m0 = S.m0[it], m1 = S.m1[it], m2 = S.m2[it], m3 = S.m3[it], col = S.rgb[it];
                const float mu[3] = { m0.x, m0.y, m0.z }, inv_s[3] = { m1.w, m2.w, m3.w };
                RInv M;
                M.m[0][0] = m1.x;
                M.m[0][1] = m1.y;
                M.m[0][2] = m1.z;
                M.m[1][0] = m2.x;
                M.m[1][1] = m2.y;
                M.m[1][2] = m2.z;
                M.m[2][0] = m3.x;
                M.m[2][1] = m3.y;
                M.m[2][2] = m3.z;
                SmoothTerms st;
                const float Kw = smooth_kernel(mu, inv_s, m0.w, M, col.w, exact_d, o[0] + (int32_t)(n >> 6),
                                               o[1] + (int32_t)((n >> 3) & 7), o[2] + (int32_t)(n & 7), st);
                if (st.e > SMOOTH_TAU)
                {
                    const uint64_t vi = vbase + S.before[n >> 5] + __popc(S.mask[n >> 5] & ((1u << (n & 31u)) - 1u));
                    const float gd = P.grad_density ? P.grad_density[vi] : 0.f;
                    float gc[3] = { 0.f, 0.f, 0.f };
                    if (P.grad_color)
#pragma unroll
                        for (int k = 0; k < 3; k++)
                            gc[k] = P.grad_color[3 * vi + k];
                    const float f = -(gd + gc[0] * col.x + gc[1] * col.y + gc[2] * col.z) * st.e;
                    const float f0 = f * st.z[0], f1 = f * st.z[1], f2 = f * st.z[2];
                    acc[0] += f;
                    acc[1] += f0;
                    acc[2] += f1;
                    acc[3] += f2;
                    acc[4] += f0 * st.z[0];
                    acc[5] += f1 * st.z[1];
                    acc[6] += f2 * st.z[2];
                    if constexpr (RAW)
                    {
                        acc[7] += f0 * st.z[1];
                        acc[8] += f0 * st.z[2];
                        acc[9] += f1 * st.z[2];
                    }
                    else
#pragma unroll
                        for (int a = 0; a < 3; a++)
                        {
                            acc[7 + a] += f0 * st.d[a];
                            acc[10 + a] += f1 * st.d[a];
                            acc[13 + a] += f2 * st.d[a];
                        }
                    acc[NACC - 3] += Kw * gc[0];
                    acc[NACC - 2] += Kw * gc[1];
                    acc[NACC - 1] += Kw * gc[2];
                }
            }
            const int k = warp_sum_split<NACC>(acc, lane);
            if (k < NACC)
                P.partials[(uint64_t)S.eidx[it] * bwd_stride<RAW> + k] = acc[0];
            __syncwarp(); // the leaf's mask and, at the end, the queue are filled again
        }
    }
}

// the sorted (voxel key, Gaussian id) pair list: per voxel, its Gaussians in
// ascending id, at the voxel's pair offset (COUNT: only the pairs per voxel)
template <bool COUNT>
__global__ void __launch_bounds__(LP_THREADS) k_leaf_export(LeafPassParams P, uint64_t* vpairs, uint32_t* counter)
{
    __shared__ LeafSmem S;
    const int t = threadIdx.x;
    while (true)
    {
        if (t == 0)
            S.cand = atomicAdd(counter, 1u);
        __syncthreads();
        const int64_t c = S.cand;
        if (c >= P.NCL)
            break;
        if (t < 8)
            S.mask[t] = P.cand_mask[8 * (uint64_t)c + t];
        const uint32_t key = P.cand_key[c];
        int32_t o[3];
        cand_origin(P, key, o);
        __syncthreads();
        const int32_t xa = o[0] + (t >> 6), y = o[1] + ((t >> 3) & 7), z = o[2] + (t & 7), xb = xa + 4;
        uint64_t dst[2] = { 0, 0 };
        bool act[2];
#pragma unroll
        for (int h = 0; h < 2; h++)
        {
            const uint32_t n = (uint32_t)(t + 256 * h);
            act[h] = (S.mask[n >> 6] >> (n & 63)) & 1ull;
            if (act[h] && !COUNT)
                dst[h] = P.pair_off[P.cand_voff[c] + mask_rank(S.mask, n)];
        }
        const uint32_t p0 = P.cand_start[c], p1 = P.cand_start[c + 1];
        for (uint32_t q0 = p0; q0 < p1; q0 += LP_CHUNK)
        {
            const uint32_t cnt = min((uint32_t)LP_CHUNK, p1 - q0);
            stage_chunk(P, S, q0, cnt);
            __syncthreads();
            for (uint32_t j = 0; j < cnt; j++)
            {
                const GaussRec& R = S.rec[j];
                const RInv M = rinv_of(R);
                const float vsf = rec_vs(R, P.voxel_size, P.cloud_vs);
#pragma unroll
                for (int h = 0; h < 2; h++)
                {
                    const int32_t x = h ? xb : xa;
                    if (!act[h] || !in_bbox(R, x, y, z))
                        continue;
                    if (!aabb_hits_unit_sphere(voxel_local_aabb(R, M, vsf, x, y, z)))
                        continue;
                    if (!COUNT)
                    {
                        const uint64_t k = ((uint64_t)key << 9) | (uint32_t)(t + 256 * h);
                        if (P.key64)
                            ((uint64_t*)P.out_keys)[dst[h]] = k;
                        else
                            ((uint32_t*)P.out_keys)[dst[h]] = (uint32_t)k;
                        P.out_ids[dst[h]] = S.gid[j];
                    }
                    dst[h]++;
                }
            }
            __syncthreads();
        }
        if (COUNT)
        {
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (act[h])
                    vpairs[P.cand_voff[c] + mask_rank(S.mask, (uint32_t)(t + 256 * h))] = dst[h];
            __syncthreads(); // the mask is reloaded for the next candidate
        }
    }
}

// ------------------------------------------------------------ leaf output ----
// lane r of a warp (r < 16): word r of a leaf's value mask as 32-bit words and
// the active voxels in the words before it
__device__ __forceinline__ uint32_t leaf_mask_word(const NodeParams& N, int64_t l, int lane, uint32_t& before)
{
    const uint32_t* m32 = reinterpret_cast<const uint32_t*>(N.cand_mask + 8 * (uint64_t)N.leaf_cand[l]);
    const uint32_t m = lane < 16 ? m32[lane] : 0u;
    uint32_t incl = __popc(m);
#pragma unroll
    for (int o = 1; o < 16; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += y;
    }
    before = incl - __popc(m);
    return m;
}

// One warp per leaf (a CTA's warps take consecutive leaves): the leaf's staged
// values to its value indices, its node2 node (grid_build_finalize.slang) and
// its share of the cloud's bbox (grid_build_compute_bbox.slang).  A round takes
// 32 slots of the leaf: staged reads and value writes are runs of consecutive
// words.  HBM-bound: 20 B read and 20 B written per voxel, 1.04 ms for 106M
// voxels (4.5 TB/s; the loads of 2 / 4 / 8 rounds in flight: 1.11 / 1.04 / 1.12 ms,
// of one 1.76 ms).
constexpr int WL_THREADS = 256;
constexpr int WL_ROUNDS = 4; // rounds whose loads are in flight together

template <bool FLOATS>
__global__ void __launch_bounds__(WL_THREADS) k_write_leaves(ValueParams A, NodeParams N, int per_warp)
{
    __shared__ int32_t s_bb[6];
    __shared__ unsigned long long s_pairs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const CloudParams& C = N.C;
    const int64_t l0 = (int64_t)blockIdx.x * (WL_THREADS / 32) * per_warp;
    const uint32_t cb = C.leaf_cloud[l0]; // the CTA's first leaf's cloud: its sums stay in shared memory
    if (threadIdx.x < 6)
        s_bb[threadIdx.x] = threadIdx.x < 3 ? 0x7FFFFFFF : (int32_t)0x80000000;
    if (threadIdx.x == 0)
        s_pairs = 0;
    __syncthreads();
    for (int k = 0; k < per_warp; k++)
    {
        const int64_t l = l0 + (int64_t)warp * per_warp + k;
        if (l >= N.L)
            break;
        const uint32_t b = C.leaf_cloud[l], c = N.leaf_cand[l];
        uint32_t before;
        const uint32_t mine = leaf_mask_word(N, l, lane, before);
        const uint64_t vidx = N.leaf_vidx[l];
        uint32_t* rgba = (uint32_t*)(A.out + C.rgba_off[b]) + vidx;
        float* dens = (float*)(A.out + C.dens_off[b]) + vidx;
        float* col = (float*)(A.out + C.col_off[b]) + 3 * vidx;
#pragma unroll 1
        for (int r0 = 0; r0 < 16; r0 += WL_ROUNDS)
        {
            uint32_t at[WL_ROUNDS], vr[WL_ROUNDS];
            float vd[WL_ROUNDS], vc[WL_ROUNDS][3];
#pragma unroll
            for (int i = 0; i < WL_ROUNDS; i++)
            {
                const uint32_t bits = __shfl_sync(0xffffffffu, mine, r0 + i);
                const uint32_t base = __shfl_sync(0xffffffffu, before, r0 + i);
                at[i] = (bits >> lane) & 1u ? base + __popc(bits & lt) : ~0u;
                const uint64_t slot = (uint64_t)c * 512u + (uint32_t)(32 * (r0 + i) + lane);
                if (at[i] != ~0u)
                {
                    vr[i] = __ldcs(A.s_rgba + slot);
                    if constexpr (FLOATS)
                    {
                        vd[i] = __ldcs(A.s_dens + slot);
#pragma unroll
                        for (int k2 = 0; k2 < 3; k2++)
                            vc[i][k2] = __ldcs(A.s_col + 3 * slot + k2);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < WL_ROUNDS; i++)
                if (at[i] != ~0u)
                {
                    __stcs(rgba + at[i], vr[i]);
                    if constexpr (FLOATS)
                    {
                        __stcs(dens + at[i], vd[i]);
#pragma unroll
                        for (int k2 = 0; k2 < 3; k2++)
                            __stcs(col + 3 * at[i] + k2, vc[i][k2]);
                    }
                }
        }
        // the node: index, value index, prefix words, mask (128 B)
        const uint32_t total = __shfl_sync(0xffffffffu, before + __popc(mine), 15);
        uint64_t word = 0;
        const uint64_t m_lo = __shfl_sync(0xffffffffu, mine, (2 * (lane - 8)) & 31);
        const uint64_t m_hi = __shfl_sync(0xffffffffu, mine, (2 * (lane - 8) + 1) & 31);
        uint64_t prefix[2] = { total & 0xFFFFu, 0 };
#pragma unroll
        for (int q = 1; q < 8; q++)
            prefix[q >> 2] |= (uint64_t)(__shfl_sync(0xffffffffu, before, 2 * q) & 0xFFFFu) << (16 * (q & 3));
        if (lane == 0)
        {
            word = N.leaf_idx[l];
            A.cand_vbase[c] = C.value_base[b] + vidx;
        }
        else if (lane == 1)
            word = vidx;
        else if (lane == 6 || lane == 7)
            word = prefix[lane - 6];
        else if (lane >= 8)
            word = m_lo | (m_hi << 32);
        if (lane < 16)
            ((uint64_t*)(A.out + N.leaf_addr[l]))[lane] = word;
        // bbox: x from the mask words with a voxel, y and z from their union
        const uint32_t even = __reduce_or_sync(0xffffffffu, (lane & 1) ? 0u : mine),
                       odd = __reduce_or_sync(0xffffffffu, (lane & 1) ? mine : 0u);
        const uint32_t nz = __ballot_sync(0xffffffffu, mine != 0u);
        uint32_t ym = 0, zm = even | odd;
        zm |= zm >> 16;
        zm = (zm | (zm >> 8)) & 0xffu;
#pragma unroll
        for (int q = 0; q < 4; q++)
            ym |= ((even >> (8 * q)) & 0xffu ? 1u : 0u) << q | ((odd >> (8 * q)) & 0xffu ? 1u : 0u) << (q + 4);
        if (lane < 6)
        {
            const int a = lane % 3;
            const int32_t lo = a == 0 ? (__ffs(nz) - 1) >> 1 : __ffs(a == 1 ? ym : zm) - 1;
            const int32_t hi = a == 0 ? (31 - __clz(nz)) >> 1 : 31 - __clz(a == 1 ? ym : zm);
            int32_t* bb = b == cb ? s_bb : C.bbox + 6 * (uint64_t)b;
            const int32_t o = N.leaf_origin[3 * l + a];
            if (lane < 3)
                atomicMin(&bb[a], o + lo);
            else
                atomicMax(&bb[3 + a], o + hi);
        }
        if (A.cloud_pairs && lane == 0)
            atomicAdd(b == cb ? &s_pairs : (unsigned long long*)&A.cloud_pairs[b], (unsigned long long)A.cand_pairs[c]);
    }
    __syncthreads();
    if (threadIdx.x < 3)
        atomicMin(&C.bbox[6 * (uint64_t)cb + threadIdx.x], s_bb[threadIdx.x]);
    else if (threadIdx.x < 6)
        atomicMax(&C.bbox[6 * (uint64_t)cb + threadIdx.x], s_bb[threadIdx.x]);
    if (threadIdx.x == 0 && A.cloud_pairs && s_pairs)
        atomicAdd((unsigned long long*)&A.cloud_pairs[cb], s_pairs);
}

// f(voxel in canonical order, leaf, leaf_n) for every active voxel, a warp per leaf
template <class F>
__device__ __forceinline__ void each_voxel(const NodeParams& N, F f)
{
    const int64_t l = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (l >= N.L)
        return;
    uint32_t before;
    const uint32_t mine = leaf_mask_word(N, l, lane, before);
    const uint64_t v0 = N.leaf_vstart[l];
    for (int r = 0; r < 16; r++)
    {
        const uint32_t bits = __shfl_sync(0xffffffffu, mine, r), base = __shfl_sync(0xffffffffu, before, r);
        if ((bits >> lane) & 1u)
            f(v0 + base + __popc(bits & ((1u << lane) - 1u)), l, (uint32_t)(32 * r + lane));
    }
}

// coordinates of the active voxels by value index (clouds back to back)
__global__ void k_voxel_coords(NodeParams N, int32_t* out)
{
    each_voxel(N, [&](uint64_t v, int64_t l, uint32_t n) {
        const uint64_t at = N.C.value_base[N.C.leaf_cloud[l]] + N.leaf_vidx[l] + (v - N.leaf_vstart[l]);
        out[3 * at + 0] = N.leaf_origin[3 * l + 0] + (int32_t)(n >> 6);
        out[3 * at + 1] = N.leaf_origin[3 * l + 1] + (int32_t)((n >> 3) & 7);
        out[3 * at + 2] = N.leaf_origin[3 * l + 2] + (int32_t)(n & 7);
    });
}

// ---------------------------------------------------------------- launch ----
void launch_tile_gauss(const uint64_t* lcol_off, int64_t G, uint64_t NLC, int64_t* tile_g0, cudaStream_t s)
{
    if (NLC == 0)
        return;
    const uint64_t ntiles = (NLC + 255) / 256;
    { k_tile_gauss<<<(unsigned)((ntiles + 255) / 256), 256, 0, s>>>(lcol_off, G, NLC, tile_g0); count_launch(); }
}

void launch_leaf_emit(const LeafEmitParams& P, const RankTables& T, bool write, cudaStream_t s)
{
    if (P.NLC == 0)
        return;
    uint64_t blocks = (P.NLC + 255) / 256;
    if (blocks > 148ull * 64)
        blocks = 148ull * 64;
    if (write)
        { k_leaf_emit<true><<<(unsigned)blocks, 256, 0, s>>>(P, T); count_launch(); }
    else
        { k_leaf_emit<false><<<(unsigned)blocks, 256, 0, s>>>(P, T); count_launch(); }
}

size_t cand_status_words(int64_t Q)
{
    return 4 * (size_t)((Q + LC_TILE - 1) / LC_TILE);
}

void launch_leaf_cands(const uint32_t* keys, const uint32_t* vals, const uint32_t* emit_gid, int64_t Q,
                       const uint32_t* lower_cell, const uint32_t* root_of_rank, const CandParams& C, cudaStream_t s)
{
    if (Q <= 0)
        return;
    { k_leaf_cands<<<(unsigned)((Q + LC_TILE - 1) / LC_TILE), LC_BLOCK, 0, s>>>(keys, vals, emit_gid, Q, lower_cell, root_of_rank, C); count_launch(); }
}

static unsigned walk_grid(int64_t NCL, int num_sms)
{
    int64_t g = (int64_t)num_sms * 8;
    return (unsigned)(g < NCL ? g : (NCL > 0 ? NCL : 1));
}

template <bool CHECK, bool WINDOW, bool SMOOTH, int MINB, bool BYTES = false>
static int launch_walk(const LeafPassParams& P, uint32_t* counter, int num_sms, cudaStream_t s)
{
    auto kern = k_leaf_pass<CHECK, WINDOW, SMOOTH, MINB, BYTES>;
    const size_t smem = sizeof(LeafQSmem<SMOOTH>);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, LP_THREADS, smem);
    int64_t grid = (int64_t)num_sms * (per_sm > 0 ? per_sm : 1);
    if (grid > P.NCL)
        grid = P.NCL;
    { kern<<<(unsigned)grid, LP_THREADS, smem, s>>>(P, counter); count_launch(); }
    return per_sm;
}

int launch_leaf_pass(const LeafPassParams& P, uint32_t* counter, int num_sms, cudaStream_t s, int variant)
{
    if (P.NCL <= 0)
        return 0;
    if (P.smooth)
        return P.emit_flag ? (P.window ? launch_walk<true, true, true, 4>(P, counter, num_sms, s)
                                       : launch_walk<true, false, true, 4>(P, counter, num_sms, s))
                           : (P.window ? launch_walk<false, true, true, 4>(P, counter, num_sms, s)
                                       : launch_walk<false, false, true, 4>(P, counter, num_sms, s));
    if (P.bytes)
        return P.emit_flag ? (P.window ? launch_walk<true, true, false, 4, true>(P, counter, num_sms, s)
                                       : launch_walk<true, false, false, 4, true>(P, counter, num_sms, s))
                           : (P.window ? launch_walk<false, true, false, 4, true>(P, counter, num_sms, s)
                                       : launch_walk<false, false, false, 4, true>(P, counter, num_sms, s));
    if (P.emit_flag)
        return P.window ? launch_walk<true, true, false, 4>(P, counter, num_sms, s)
                        : launch_walk<true, false, false, 4>(P, counter, num_sms, s);
    if (variant == 1)
        return P.window ? launch_walk<false, true, false, 3>(P, counter, num_sms, s)
                        : launch_walk<false, false, false, 3>(P, counter, num_sms, s);
    return P.window ? launch_walk<false, true, false, 4>(P, counter, num_sms, s)
                    : launch_walk<false, false, false, 4>(P, counter, num_sms, s);
}

void launch_leaf_backward(const LeafPassParams& P, int64_t Q, bool raw, cudaStream_t s)
{
    if (Q <= 0)
        return;
    const size_t smem = sizeof(BwdWarp) * BW_WARPS;
    auto kern = raw ? k_leaf_backward<true> : k_leaf_backward<false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int64_t per = 32 * BW_WARPS;
    { kern<<<(unsigned)((Q + per - 1) / per), BW_WARPS * 32, smem, s>>>(P, Q); count_launch(); }
}

void launch_leaf_export(const LeafPassParams& P, uint64_t* vpairs, uint32_t* counter, int num_sms, cudaStream_t s)
{
    if (P.NCL <= 0)
        return;
    cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
    if (vpairs)
        { k_leaf_export<true><<<walk_grid(P.NCL, num_sms), LP_THREADS, 0, s>>>(P, vpairs, counter); count_launch(); }
    else
        { k_leaf_export<false><<<walk_grid(P.NCL, num_sms), LP_THREADS, 0, s>>>(P, nullptr, counter); count_launch(); }
}

void launch_write_leaves(const ValueParams& A, const NodeParams& N, int num_sms, cudaStream_t s)
{
    if (N.L <= 0)
        return;
    // up to 8 leaves per warp (its CTA adds 64 leaves to the bbox at once), but no
    // more than leave every SM its 8 CTAs
    const int64_t per_cta = WL_THREADS / 32;
    int64_t per_warp = N.L / (per_cta * 8 * num_sms);
    per_warp = per_warp < 1 ? 1 : per_warp > 8 ? 8 : per_warp;
    const int64_t grid = (N.L + per_cta * per_warp - 1) / (per_cta * per_warp);
    if (A.s_dens)
        { k_write_leaves<true><<<(unsigned)grid, WL_THREADS, 0, s>>>(A, N, (int)per_warp); count_launch(); }
    else
        { k_write_leaves<false><<<(unsigned)grid, WL_THREADS, 0, s>>>(A, N, (int)per_warp); count_launch(); }
}

void launch_voxel_coords(const NodeParams& N, int32_t* out, cudaStream_t s)
{
    if (N.L <= 0)
        return;
    { k_voxel_coords<<<(unsigned)((N.L + 7) / 8), 256, 0, s>>>(N, out); count_launch(); }
}

} // namespace vox
