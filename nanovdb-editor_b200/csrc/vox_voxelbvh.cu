// vox_voxelbvh.cu - VoxelBVH Gaussian ingestion: per Gaussian, the finest
// power-of-two cell level at which at most 8 cells overlap its 0.01-opacity
// ellipsoid, those cells as 64-bit keys i << 48 | j << 32 | k << 16 | level,
// and after the key sort the [start, end) range of every distinct key
// (raster/VoxelBVH.cpp:1225-1435, ijkl_from_gaussians).
//
// Kernels, all on the caller's stream:
//   k_vb_init           world-box accumulator = (+inf, -inf)
//   k_vb_box            per-Gaussian transformed 8-corner box, warp-reduced,
//                       one atomicMin / atomicMax per warp on order-preserving
//                       integer keys (deterministic; -0 orders below +0)
//                       (voxelbvh_gaussians_bbox_reduce1/2.slang)
//   k_vb_keys           the level search from 11 down, stopping once more
//                       than 8 cells overlap; 8 keys and 8 ids per Gaussian
//                       (voxelbvh_gaussians_to_ijkl.slang:25-250)
//   (scan)              the used slots (a prefix of each Gaussian's 8)
//   k_vb_compress_used  their keys compressed to 4 + bits(i) + bits(j) +
//                       bits(k) bits (32-bit when they fit), sized by the
//                       emitted cells' range the search reduces: the same
//                       order in fewer radix passes, and compacted (the
//                       unused slots, all-ones key and id, are the sorted tail)
//   (sort)              stable LSD sort of the used compressed keys (of all
//                       64-bit keys when a cell lies outside [0, 2^16))
//   k_vb_ranges         headers [2r] = start, [2r + 1] = end (the others are
//                       zero), the sorted keys as 64-bit keys, the unused
//                       tail's keys and ids all ones, its run the last range
//                       (voxelbvh_find_range_starts.slang,
//                       voxelbvh_scatter_range_headers.slang)
//
// Float arithmetic: every operation that decides a key is one IEEE
// round-to-nearest intrinsic in the order the shaders write it (no
// contraction), or a cheaper form whose distance from it is bounded and whose
// decision is taken only outside that distance (k_vb_keys), so the keys are the
// same bits as the C restatement's.
#include <cuda_runtime.h>

#include "vox_device.cuh"
#include "vox_internal.h"
#include "vox_raster.h"

namespace vox
{

namespace
{

constexpr int VB_THREADS = 256;
constexpr int VB_TILE = 2048; // keys per range tile (8 per thread)
constexpr float VB_CELL_LIMIT = 65536.f;
// a level whose cell box exceeds this is reported (VOX_ERR_RANGE) instead of
// searched: it bounds the search, and no Gaussian whose box is its own
// ellipsoid's reaches it (more than 8 of its cells overlap long before)
constexpr int64_t VB_MAX_CELLS = 1ll << 24;

__device__ __forceinline__ uint32_t vb_fkey(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float vb_funkey(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct VbGauss
{
    float mu[3];
    float R[3][3]; // forward rotation rows; the inverse is the transpose
    float e[3];    // scale * local_scale
    float inv[3];  // 1 / (local_scale * scale)
};

__device__ __forceinline__ void vb_load(const VoxelBvhParams& P, int64_t g, VbGauss& G)
{
    for (int a = 0; a < 3; a++)
        G.mu[a] = P.means[3 * g + a];
    const float w = P.quats[4 * g + 0], x = P.quats[4 * g + 1], y = P.quats[4 * g + 2], z = P.quats[4 * g + 3];
    float s[3];
    for (int a = 0; a < 3; a++)
        s[a] = P.scales[3 * g + a];
    const float op = P.opac[g];
    const float o = 0.01f > op ? 0.01f : op;
    const float ls = __fsqrt_rn(__fmul_rn(2.f, vox_logf(__fdiv_rn(o, 0.01f))));
    G.R[0][0] = __fsub_rn(1.f, __fmul_rn(2.f, __fadd_rn(__fmul_rn(y, y), __fmul_rn(z, z))));
    G.R[0][1] = __fmul_rn(2.f, __fsub_rn(__fmul_rn(x, y), __fmul_rn(z, w)));
    G.R[0][2] = __fmul_rn(2.f, __fadd_rn(__fmul_rn(x, z), __fmul_rn(y, w)));
    G.R[1][0] = __fmul_rn(2.f, __fadd_rn(__fmul_rn(x, y), __fmul_rn(z, w)));
    G.R[1][1] = __fsub_rn(1.f, __fmul_rn(2.f, __fadd_rn(__fmul_rn(x, x), __fmul_rn(z, z))));
    G.R[1][2] = __fmul_rn(2.f, __fsub_rn(__fmul_rn(y, z), __fmul_rn(x, w)));
    G.R[2][0] = __fmul_rn(2.f, __fsub_rn(__fmul_rn(x, z), __fmul_rn(y, w)));
    G.R[2][1] = __fmul_rn(2.f, __fadd_rn(__fmul_rn(y, z), __fmul_rn(x, w)));
    G.R[2][2] = __fsub_rn(1.f, __fmul_rn(2.f, __fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y))));
    for (int a = 0; a < 3; a++)
    {
        G.e[a] = __fmul_rn(s[a], ls);
        G.inv[a] = __fdiv_rn(1.f, __fmul_rn(ls, s[a]));
    }
}

// p' = [p 1] T (row vector), sums left to right
__device__ __forceinline__ float vb_xf(const float* T, float p0, float p1, float p2, int c)
{
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p0, T[c]), __fmul_rn(p1, T[4 + c])), __fmul_rn(p2, T[8 + c])),
                     T[12 + c]);
}

__device__ __forceinline__ bool vb_finite(float x)
{
    return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u;
}

// transformed 8-corner box of the local_scale cube; minima / maxima as keys.
// Returns false when a corner is not finite (the keys then cover the finite
// corners only): the caller reports an error, since NaN has no place in the
// order the keys encode.
__device__ __forceinline__ bool vb_box_keys(const VoxelBvhParams& P, const VbGauss& G, uint32_t kmn[3], uint32_t kmx[3])
{
    bool finite = true;
    float pr[3][3]; // pr[c][a] = e[a] * R[c][a]; the -e corner's product is its negation
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int a = 0; a < 3; a++)
            pr[c][a] = __fmul_rn(G.e[a], G.R[c][a]);
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        kmn[a] = 0xffffffffu;
        kmx[a] = 0u;
    }
#pragma unroll
    for (int v = 0; v < 8; v++)
    {
        float wp[3];
#pragma unroll
        for (int c = 0; c < 3; c++)
        {
            const float t0 = (v & 1) ? pr[c][0] : -pr[c][0];
            const float t1 = (v & 2) ? pr[c][1] : -pr[c][1];
            const float t2 = (v & 4) ? pr[c][2] : -pr[c][2];
            wp[c] = __fadd_rn(__fadd_rn(__fadd_rn(t0, t1), t2), G.mu[c]);
        }
        float tp[3];
        if (P.has_xform)
        {
#pragma unroll
            for (int c = 0; c < 3; c++)
                tp[c] = vb_xf(P.t, wp[0], wp[1], wp[2], c);
        }
        else
        {
#pragma unroll
            for (int c = 0; c < 3; c++)
                tp[c] = wp[c];
        }
#pragma unroll
        for (int a = 0; a < 3; a++)
        {
            if (!vb_finite(tp[a]))
            {
                finite = false;
                continue;
            }
            const uint32_t k = vb_fkey(tp[a]);
            kmn[a] = k < kmn[a] ? k : kmn[a];
            kmx[a] = k > kmx[a] ? k : kmx[a];
        }
    }
    return finite;
}

// Voxel-to-world coordinate of one cell boundary on axis a:
// (v - offset) / scale, v = the boundary's voxel coordinate.
__device__ __forceinline__ float vb_lp(const float w2v[4], float v, int a)
{
    return __fdiv_rn(__fsub_rn(v, w2v[a]), w2v[3]);
}

__global__ void k_vb_init(uint32_t* box_keys, int* cell_minmax)
{
    if (threadIdx.x < 3)
        box_keys[threadIdx.x] = 0xff800000u; // key of +inf
    else if (threadIdx.x < 6)
        box_keys[threadIdx.x] = 0x007fffffu; // key of -inf
    if (threadIdx.x < 3)
        cell_minmax[threadIdx.x] = 0x7fffffff;
    else if (threadIdx.x < 6)
        cell_minmax[threadIdx.x] = (int)0x80000000;
}

__global__ void __launch_bounds__(VB_THREADS) k_vb_box(VoxelBvhParams P)
{
    uint32_t mn[3] = { 0xff800000u, 0xff800000u, 0xff800000u }, mx[3] = { 0x007fffffu, 0x007fffffu, 0x007fffffu };
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < P.n; g += (int64_t)gridDim.x * blockDim.x)
    {
        VbGauss G;
        vb_load(P, g, G);
        uint32_t a0[3], a1[3];
        if (!vb_box_keys(P, G, a0, a1))
            atomicOr(P.err, ERR_RANGE);
#pragma unroll
        for (int a = 0; a < 3; a++)
        {
            mn[a] = a0[a] < mn[a] ? a0[a] : mn[a];
            mx[a] = a1[a] > mx[a] ? a1[a] : mx[a];
        }
    }
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        const uint32_t wmn = __reduce_min_sync(0xffffffffu, mn[a]);
        const uint32_t wmx = __reduce_max_sync(0xffffffffu, mx[a]);
        if ((threadIdx.x & 31) == 0)
        {
            atomicMin(&P.box_keys[a], wmn);
            atomicMax(&P.box_keys[3 + a], wmx);
        }
    }
}

__device__ __forceinline__ bool vb_cell_ok(float v)
{
    return v >= -VB_CELL_LIMIT && v <= VB_CELL_LIMIT; // false for NaN
}

// voxel_ellipsoid_overlap (voxelbvh_gaussians_to_ijkl.slang:25-109) of the cell
// of edge 2^level at (i, j, k), the shader's arithmetic
template <bool XF>
__device__ __noinline__ bool vb_overlap_cell(const VoxelBvhParams& P, int64_t g, float off0, float off1, float off2, float sc,
                                             int i, int j, int k, uint32_t level)
{
    VbGauss G;
    vb_load(P, g, G);
    const float w2v[4] = { off0, off1, off2, sc };
    const float step = (float)(1u << level);
    const int ijk[3] = { i, j, k };
    float lp[3][2];
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        const float v0 = (float)ijk[a];
        lp[a][0] = vb_lp(w2v, v0, a);
        lp[a][1] = vb_lp(w2v, __fadd_rn(v0, step), a);
    }
    float vmin[3] = { 0.f, 0.f, 0.f }, vmax[3] = { 0.f, 0.f, 0.f };
#pragma unroll 1
    for (int v = 0; v < 8; v++)
    {
        const int b0 = v & 1, b1 = (v >> 1) & 1, b2 = (v >> 2) & 1;
        const float p0 = b0 ? lp[0][1] : lp[0][0], p1 = b1 ? lp[1][1] : lp[1][0], p2 = b2 ? lp[2][1] : lp[2][0];
        float d[3];
        if (XF)
        {
#pragma unroll
            for (int c = 0; c < 3; c++)
                d[c] = __fsub_rn(vb_xf(P.ti, p0, p1, p2, c), G.mu[c]);
        }
        else
        {
            d[0] = __fsub_rn(p0, G.mu[0]);
            d[1] = __fsub_rn(p1, G.mu[1]);
            d[2] = __fsub_rn(p2, G.mu[2]);
        }
#pragma unroll
        for (int r = 0; r < 3; r++)
        {
            const float lr = __fadd_rn(__fadd_rn(__fmul_rn(d[0], G.R[0][r]), __fmul_rn(d[1], G.R[1][r])),
                                       __fmul_rn(d[2], G.R[2][r]));
            const float x = __fmul_rn(lr, G.inv[r]);
            if (v == 0 || x < vmin[r])
                vmin[r] = x;
            if (v == 0 || x > vmax[r])
                vmax[r] = x;
        }
    }
    float dist2 = 1.f;
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        if (0.f < vmin[a])
            dist2 = __fsub_rn(dist2, __fmul_rn(vmin[a], vmin[a]));
        else if (0.f > vmax[a])
            dist2 = __fsub_rn(dist2, __fmul_rn(vmax[a], vmax[a]));
    }
    return dist2 > 0.f;
}

__device__ __forceinline__ int64_t vb_level_cells(const int lo[3], const int hi[3], uint32_t level)
{
    int64_t cells = 1;
#pragma unroll
    for (int a = 0; a < 3; a++)
        cells *= (int64_t)((hi[a] >> level) - (lo[a] >> level)) + 1;
    return cells;
}

// The level search, a thread per Gaussian.  Only "more than 8 cells overlap"
// matters, so a level whose box holds at most 8 cells is decided without a test
// and a count stops at 9.
//
// A cell's local AABB is its centre plus and minus a half width (the map from
// cells to the Gaussian's unit-sphere space is affine, with or without a
// transform): row r, for a cell at offset o from the box's corner cell lo, centre
// base_r + sum_a B_ra (o_a + st / 2), half width st / 2 sum_a |B_ra|.  That takes
// 18 instructions where the shader's corners take 50 (400 with a transform), and
// decides every cell whose squared distance D from the unit sphere's centre is
// not near 1.  In units of 2^-24, with lp the cell corners' world coordinates,
// d their offsets from the mean, X the box's extent there (with a transform: M
// = sum |lp t| + |t_3|, X through |t|), the shader's row values are within inv_r
// sum |R| (2 |lp| + 5 |d|) (transform: 6 M + 5 |d|) of exact; this form's base
// within the same, its B (two products and 1 / sc, each rounded once) within 3 X
// (6 X), the sums 3 (|d| + X), the half width 6 X (9 X), the difference |d| + 2 X.
// delta_r = inv_r sum |R| (5 |lp| + 16 |d| + 16 X), or (14 M + 16 |d| + 24 X), covers
// both; Delta = sum_r delta_r gives the thresholds on D exactly as in the leaf test
// (vox_leaf.cu), and what lies between them, or a Gaussian with Delta > 1/16, takes
// the shader's arithmetic.  So does one whose cells or ellipsoid are below 2^-100:
// products that leave the normal range have roundings that are not relative (1 / sc
// itself does from 2^126 on).
// Everything is held halved (D quartered), so that a saturating difference is
// max(|c| - h, 0) up to far above the threshold.
//
// The three levels of loops are one loop over cells, so lanes at different
// levels or in different phases (counting, emitting) go on together.  Bound by
// instruction issue; the keys
// stage of 2M Gaussians at resolution 512 1.16 -> 0.46 ms, of 20k with a transform
// 0.100 -> 0.038 (3 CTAs per SM; 4 spill, 0.47 and 0.040).
template <bool XF>
__global__ void __launch_bounds__(VB_THREADS, 3) k_vb_keys(const __grid_constant__ VoxelBvhParams P)
{
    // compute_world_to_voxel (voxelbvh_gaussians_to_ijkl.slang:111-118)
    float wmin[3], wmax[3];
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        wmin[a] = vb_funkey(P.box_keys[a]);
        wmax[a] = vb_funkey(P.box_keys[3 + a]);
    }
    if (blockIdx.x == 0 && threadIdx.x < 6)
        P.world_bbox[threadIdx.x] = threadIdx.x < 3 ? wmin[threadIdx.x] : wmax[threadIdx.x - 3];
    const float d0 = __fsub_rn(wmax[0], wmin[0]), d1 = __fsub_rn(wmax[1], wmin[1]), d2 = __fsub_rn(wmax[2], wmin[2]);
    const float dyz = d1 > d2 ? d1 : d2;
    const float dmax = d0 > dyz ? d0 : dyz;
    const float sc = __fdiv_rn((float)(P.resolution - 1u), dmax);
    const float w2v[4] = { __fadd_rn(__fmul_rn(-wmin[0], sc), 0.5f), __fadd_rn(__fmul_rn(-wmin[1], sc), 0.5f),
                           __fadd_rn(__fmul_rn(-wmin[2], sc), 0.5f), sc };

    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = g < P.n;
    bool ok = valid;
    int lo[3] = { 0, 0, 0 }, hi[3] = { 0, 0, 0 };
    uint32_t level = 11u, last_good = 11u;
    bool emit = false;
    float B[3][3] = {}, base[3] = {};
    float lo_t = -1.f, hi_t = __int_as_float(0x7f800000); // every cell takes the shader's arithmetic
    if (valid)
    {
        VbGauss G;
        vb_load(P, g, G);
        uint32_t kmn[3], kmx[3];
        ok = vb_box_keys(P, G, kmn, kmx);
#pragma unroll
        for (int a = 0; a < 3; a++)
        {
            const float fl = floorf(__fadd_rn(__fmul_rn(sc, vb_funkey(kmn[a])), w2v[a]));
            const float fh = floorf(__fadd_rn(__fmul_rn(sc, vb_funkey(kmx[a])), w2v[a]));
            ok = ok && vb_cell_ok(fl) && vb_cell_ok(fh);
            lo[a] = (int)fl;
            hi[a] = (int)fh;
        }
        if (ok)
        {
            // down to the first level that needs a test, or to level 0, emitted untested
            while (true)
            {
                const int64_t cells = vb_level_cells(lo, hi, level);
                ok = cells <= VB_MAX_CELLS;
                emit = cells <= 8;
                if (!ok || !emit || level == 0u)
                    break;
                last_good = level;
                level -= 1u;
            }
        }
        if (ok)
        {
            // the coarsest level whose cells may be tested bounds all of them
            const uint32_t top = level < 11u ? level + 1u : 11u;
            const int st = 1 << top, msk = -st;
            float lp[3], ext[3], at[3];
#pragma unroll
            for (int a = 0; a < 3; a++)
            {
                const float c0 = vb_lp(w2v, (float)(lo[a] & msk), a), c1 = vb_lp(w2v, (float)((hi[a] & msk) + st), a);
                lp[a] = fmaxf(fabsf(c0), fabsf(c1));
                ext[a] = fabsf(c1 - c0);
                at[a] = vb_lp(w2v, (float)lo[a], a); // the corner cell's corner
            }
            float Dl = 0.f;
            float w[3], M[3], X[3];
#pragma unroll
            for (int c = 0; c < 3; c++)
            {
                if (XF)
                {
                    w[c] = at[0] * P.ti[c] + at[1] * P.ti[4 + c] + at[2] * P.ti[8 + c] + P.ti[12 + c];
                    M[c] = lp[0] * fabsf(P.ti[c]) + lp[1] * fabsf(P.ti[4 + c]) + lp[2] * fabsf(P.ti[8 + c]) + fabsf(P.ti[12 + c]);
                    X[c] = ext[0] * fabsf(P.ti[c]) + ext[1] * fabsf(P.ti[4 + c]) + ext[2] * fabsf(P.ti[8 + c]);
                }
                else
                {
                    w[c] = at[c];
                    M[c] = lp[c];
                    X[c] = ext[c];
                }
                w[c] -= G.mu[c];
                M[c] = XF ? 14.f * M[c] + 16.f * (fabsf(w[c]) + X[c]) + 24.f * X[c]
                          : 5.f * M[c] + 16.f * (fabsf(w[c]) + X[c]) + 16.f * X[c];
            }
            const float rs = __fdiv_rn(1.f, sc);
            float big = sc;
#pragma unroll
            for (int r = 0; r < 3; r++)
            {
                base[r] = 0.5f * G.inv[r] * (G.R[0][r] * w[0] + G.R[1][r] * w[1] + G.R[2][r] * w[2]);
#pragma unroll
                for (int a = 0; a < 3; a++)
                {
                    const float m = XF ? G.R[0][r] * P.ti[4 * a] + G.R[1][r] * P.ti[4 * a + 1] + G.R[2][r] * P.ti[4 * a + 2]
                                       : G.R[a][r];
                    B[r][a] = 0.5f * G.inv[r] * m * rs;
                }
                big = fmaxf(big, G.inv[r]);
                Dl += G.inv[r] * (fabsf(G.R[0][r]) * M[0] + fabsf(G.R[1][r]) * M[1] + fabsf(G.R[2][r]) * M[2]);
            }
            Dl *= 0x1.02p-24f;
            if (Dl <= 0.0625f && big < 0x1p100f) // false for NaN
            {
                lo_t = 0.25f * (1.f - (2.f * Dl + 0x1p-19f));
                hi_t = 0.25f * (1.f + (2.f * Dl + Dl * Dl + 0x1p-18f));
            }
        }
    }
    uint32_t count = 0;
    uint64_t* out = P.keys + 8 * g;
    bool busy = valid && ok, start = true;
    float st = 0.f, i0 = 0.f, i1 = 0.f, j0 = 0.f, j1 = 0.f, k0 = 0.f, k1 = 0.f; // cells of the level, from lo
    float i = 0.f, j = 0.f, k = 0.f, b[3] = {}, h[3] = {};
    while (busy)
    {
        if (start)
        {
            const int s1 = 1 << level, msk = -s1;
            st = (float)s1;
            i = i0 = (float)((lo[0] & msk) - lo[0]);
            j = j0 = (float)((lo[1] & msk) - lo[1]);
            k = k0 = (float)((lo[2] & msk) - lo[2]);
            i1 = (float)((hi[0] & msk) - lo[0]);
            j1 = (float)((hi[1] & msk) - lo[1]);
            k1 = (float)((hi[2] & msk) - lo[2]);
#pragma unroll
            for (int r = 0; r < 3; r++)
            {
                b[r] = base[r] + 0.5f * st * (B[r][0] + B[r][1] + B[r][2]);
                h[r] = 0.5f * st * (fabsf(B[r][0]) + fabsf(B[r][1]) + fabsf(B[r][2]));
            }
            count = 0;
            start = false;
        }
        float D = 0.f;
#pragma unroll
        for (int r = 0; r < 3; r++)
        {
            const float c = VOX_FFMA(B[r][2], k, VOX_FFMA(B[r][1], j, VOX_FFMA(B[r][0], i, b[r])));
            const float x = __saturatef(VOX_FSUB(fabsf(c), h[r]));
            D = VOX_FFMA(x, x, D);
        }
        bool hit = D < lo_t;
        if (!hit && !(D > hi_t))
            hit = vb_overlap_cell<XF>(P, g, w2v[0], w2v[1], w2v[2], sc, lo[0] + (int)i, lo[1] + (int)j, lo[2] + (int)k, level);
        if (hit)
        {
            if (emit)
                out[count] = ((uint64_t)(int64_t)(lo[0] + (int)i) << 48) | ((uint64_t)(int64_t)(lo[1] + (int)j) << 32) |
                             ((uint64_t)(int64_t)(lo[2] + (int)k) << 16) | (uint64_t)level;
            count++;
        }
        k += st;
        if (k > k1)
        {
            k = k0;
            j += st;
            if (j > j1)
            {
                j = j0;
                i += st;
            }
        }
        if (i > i1 || count >= (emit ? 8u : 9u))
        {
            // the level is done
            start = true;
            if (emit)
                busy = false;
            else if (count > 8u) // too many: the last level that was not
            {
                level = last_good;
                emit = true;
            }
            else if (level == 0u)
                emit = true;
            else
            {
                last_good = level;
                level -= 1u; // its box holds no fewer cells
                if (vb_level_cells(lo, hi, level) > VB_MAX_CELLS)
                {
                    ok = false;
                    busy = false;
                }
            }
        }
    }
    if (valid && !ok) // not finite, out of range or unbounded: unused slots, error
        atomicOr(P.err, ERR_RANGE);
    const uint32_t nkeys = valid && ok ? count : 0u;
    if (valid)
    {
#pragma unroll
        for (uint32_t s = 0; s < 8; s++)
            if (s >= nkeys)
                out[s] = ~0ull;
        P.used[g] = nkeys;
        const uint32_t id = (uint32_t)g;
        uint4* idd = reinterpret_cast<uint4*>(P.ids + 8 * g);
        idd[0] = make_uint4(nkeys > 0 ? id : ~0u, nkeys > 1 ? id : ~0u, nkeys > 2 ? id : ~0u, nkeys > 3 ? id : ~0u);
        idd[1] = make_uint4(nkeys > 4 ? id : ~0u, nkeys > 5 ? id : ~0u, nkeys > 6 ? id : ~0u, nkeys > 7 ? id : ~0u);
    }
    // the range of the emitted levels' cells (sizes the compressed sort key)
    const int msk = -(1 << level);
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        const int wmn = __reduce_min_sync(0xffffffffu, nkeys ? lo[a] & msk : 0x7fffffff);
        const int wmx = __reduce_max_sync(0xffffffffu, nkeys ? hi[a] & msk : (int)0x80000000);
        if ((threadIdx.x & 31) == 0)
        {
            // (read first: most warps lie inside the range found so far)
            if (wmn < *(volatile int*)&P.cell_minmax[a])
                atomicMin(&P.cell_minmax[a], wmn);
            if (wmx > *(volatile int*)&P.cell_minmax[3 + a])
                atomicMax(&P.cell_minmax[3 + a], wmx);
        }
    }
}

// 64-bit key of a compressed key (VbRangeParams::bits)
template <class K>
__device__ __forceinline__ uint64_t vb_expand(K c, const VbRangeParams& R)
{
    if ((uint64_t)c == R.sentinel)
        return ~0ull;
    const uint64_t u = (uint64_t)c;
    const uint64_t level = u & 15u;
    const uint64_t k = (u >> 4) & ((1ull << R.bits[2]) - 1);
    const uint64_t j = (u >> (4 + R.bits[2])) & ((1ull << R.bits[1]) - 1);
    const uint64_t i = u >> (4 + R.bits[2] + R.bits[1]);
    return (i << 48) | (j << 32) | (k << 16) | level;
}

// Headers of the U sorted keys' runs ([2r] = start, [2r + 1] = end; the array is
// zero before) and, from U on, the unused slots: keys and ids all ones, their run
// the last range.  With R.expand the sorted compressed keys are written out as
// 64-bit keys, and the ids copied when the sort left them in its second buffer.
// One pass: a run's start is a key unlike the one before, its number the starts
// before it (look-back across tiles), and it ends the run before.  HBM-bound: at
// 2M Gaussians 360 MB with the headers' memset; counting, scanning, scattering
// and the tail in separate kernels, 8 keys per thread: 0.27 -> 0.16 ms.
constexpr int VB_ITEMS = VB_TILE / VB_THREADS;

template <class K>
__global__ void __launch_bounds__(VB_THREADS) k_vb_ranges(const K* __restrict__ keys, int64_t U, int64_t N, VbRangeParams R)
{
    __shared__ uint32_t s_cnt[VB_THREADS / 32];
    __shared__ uint64_t s_ex;
    __shared__ uint32_t s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        s_tile = atomicAdd(R.counter, 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    const int64_t wbase = (int64_t)tile * VB_TILE + (int64_t)warp * (32 * VB_ITEMS);
    K k[VB_ITEMS];
    uint32_t heads[VB_ITEMS], count = 0;
    K carry = wbase > 0 && wbase - 1 < U ? keys[wbase - 1] : K(0);
#pragma unroll
    for (int i = 0; i < VB_ITEMS; i++)
    {
        const int64_t q = wbase + i * 32 + lane;
        k[i] = q < U ? keys[q] : K(0);
    }
#pragma unroll
    for (int i = 0; i < VB_ITEMS; i++)
    {
        const int64_t q = wbase + i * 32 + lane;
        K prev = __shfl_up_sync(0xffffffffu, k[i], 1);
        if (lane == 0)
            prev = carry;
        carry = __shfl_sync(0xffffffffu, k[i], 31);
        heads[i] = __ballot_sync(0xffffffffu, q < U && (q == 0 || k[i] != prev));
        count += __popc(heads[i]);
    }
    if (lane == 0)
        s_cnt[warp] = count;
    __syncthreads();
    if ((int64_t)tile * VB_TILE < U) // (a tile of unused slots has no runs and no successor that needs it)
    {
        if (warp == 0)
        {
            uint64_t agg = 0;
            for (int w = 0; w < VB_THREADS / 32; w++)
                agg += s_cnt[w];
            const uint64_t e = lookback_narrow_warp<false>(R.status, tile, agg, R.epoch, R.err);
            if (lane == 0)
                s_ex = e;
        }
        __syncthreads();
    }
    uint64_t at = s_ex;
    for (int w = 0; w < warp; w++)
        at += s_cnt[w];
#pragma unroll
    for (int i = 0; i < VB_ITEMS; i++)
    {
        const int64_t q = wbase + i * 32 + lane;
        if (q < U)
        {
            const bool head = (heads[i] >> lane) & 1u;
            const uint64_t r = at + __popc(heads[i] & ((1u << lane) - 1u)); // runs started before this key
            if (head)
            {
                R.range[2 * r] = (uint32_t)q;
                if (r > 0)
                    R.range[2 * r - 1] = (uint32_t)q;
            }
            if (q == U - 1)
            {
                // key 0 starts a run, so there is one, unless the look-back gave up and the
                // prefix lacks it: nothing is written then (the call reports the wait)
                const uint64_t runs = r + (head ? 1u : 0u);
                if (runs == 0)
                    atomicOr(R.err, ERR_BOUNDS);
                else
                {
                    R.range[2 * runs - 1] = (uint32_t)U;
                    if (U < N)
                    {
                        R.range[2 * runs] = (uint32_t)U;
                        R.range[2 * runs + 1] = (uint32_t)N;
                    }
                    *R.total = runs + (U < N ? 1u : 0u);
                }
            }
            if (R.expand)
                R.keys_out[q] = vb_expand(k[i], R);
            if (R.ids_src)
                R.ids_out[q] = R.ids_src[q];
        }
        else if (q < N)
        {
            R.keys_out[q] = ~0ull;
            R.ids_out[q] = ~0u;
        }
        at += __popc(heads[i]);
    }
}

// Compaction of the used slots before the sort: a Gaussian's used slots are
// the first of its 8 (the unused ones carry key ~0 and id ~0, identical pairs,
// so after a stable sort they simply fill the tail).  The compressed key
// holds i, j, k in bits[0], bits[1], bits[2] bits above a 4-bit level, in the
// order of the 64-bit key for cells in [0, 2^bits).  k_vb_compress_used: the
// used slots' compressed keys and ids at their scanned positions.
template <class K>
__global__ void __launch_bounds__(VB_THREADS) k_vb_compress_used(const uint64_t* __restrict__ keys,
                                                                   const uint32_t* __restrict__ ids, int64_t count,
                                                                   const uint32_t* __restrict__ used,
                                                                   const uint32_t* __restrict__ off, VbRangeParams R,
                                                                   K* __restrict__ out_keys, uint32_t* __restrict__ out_ids)
{
    const int64_t N = 8 * count;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (int64_t)gridDim.x * blockDim.x)
    {
        const int64_t g = t >> 3;
        const uint32_t slot = (uint32_t)(t & 7);
        if (slot >= used[g])
            continue;
        const uint64_t u = keys[t];
        const uint64_t i = (u >> 48) & 0xffffu, j = (u >> 32) & 0xffffu, k = (u >> 16) & 0xffffu, level = u & 15u;
        const int64_t dst = (int64_t)off[g] + slot;
        out_keys[dst] = (K)((((i << R.bits[1] | j) << R.bits[2] | k) << 4) | level);
        out_ids[dst] = ids[t];
    }
}

} // namespace

void launch_vb_compress_used(const uint64_t* keys, const uint32_t* ids, int64_t count, const uint32_t* used,
                             const uint32_t* off, const VbRangeParams& R, void* out_keys, uint32_t* out_ids, int key32,
                             int num_sms, cudaStream_t s)
{
    if (count <= 0)
        return;
    int64_t grid = (8 * count + VB_THREADS - 1) / VB_THREADS;
    const int64_t cap = (int64_t)num_sms * 16;
    if (grid > cap)
        grid = cap;
    if (key32)
        k_vb_compress_used<uint32_t><<<(unsigned)grid, VB_THREADS, 0, s>>>(keys, ids, count, used, off, R,
                                                                           (uint32_t*)out_keys, out_ids);
    else
        k_vb_compress_used<uint64_t><<<(unsigned)grid, VB_THREADS, 0, s>>>(keys, ids, count, used, off, R,
                                                                           (uint64_t*)out_keys, out_ids);
    count_launch();
}

void launch_vb_init(uint32_t* box_keys, int* cell_minmax, cudaStream_t s)
{
    k_vb_init<<<1, 32, 0, s>>>(box_keys, cell_minmax);
    count_launch();
}

void launch_vb_box(const VoxelBvhParams& P, int num_sms, cudaStream_t s)
{
    if (P.n <= 0)
        return;
    int64_t grid = (P.n + VB_THREADS - 1) / VB_THREADS;
    const int64_t cap = (int64_t)num_sms * 8;
    if (grid > cap)
        grid = cap;
    k_vb_box<<<(unsigned)grid, VB_THREADS, 0, s>>>(P);
    count_launch();
}

void launch_vb_keys(const VoxelBvhParams& P, cudaStream_t s)
{
    // one block even for n = 0: it writes the world box
    const int64_t grid = P.n > 0 ? (P.n + VB_THREADS - 1) / VB_THREADS : 1;
    if (P.has_xform)
        k_vb_keys<true><<<(unsigned)grid, VB_THREADS, 0, s>>>(P);
    else
        k_vb_keys<false><<<(unsigned)grid, VB_THREADS, 0, s>>>(P);
    count_launch();
}

size_t vb_range_status_words(int64_t N)
{
    return (size_t)((N + VB_TILE - 1) / VB_TILE) + 1;
}

void launch_vb_ranges(const void* keys, int key32, int64_t U, int64_t N, const VbRangeParams& R, cudaStream_t s)
{
    if (N <= 0)
        return;
    cudaMemsetAsync(R.range, 0, 8 * (size_t)N, s);
    const unsigned grid = (unsigned)((N + VB_TILE - 1) / VB_TILE);
    if (key32)
        k_vb_ranges<uint32_t><<<grid, VB_THREADS, 0, s>>>((const uint32_t*)keys, U, N, R);
    else
        k_vb_ranges<uint64_t><<<grid, VB_THREADS, 0, s>>>((const uint64_t*)keys, U, N, R);
    count_launch();
}

} // namespace vox
