// vox_optim.cu - the fitting loop's own kernels:
//   k_adam_bf16      Adam over the voxelizer's attribute arrays, FP32 master
//                    copies and moments, bfloat16 attributes out, one pass.
//                    Elementwise and HBM-bound (30 bytes per parameter: 16 read,
//                    14 written); grid-stride over the SMs.
//   k_target_lookup  a target grid's density at a list of voxels.
#include <cmath>
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "pnanovdb_b200.h"
#include "vox_internal.h"

namespace vox
{

__global__ void __launch_bounds__(256) k_adam_bf16(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                                                    const float* __restrict__ grad, __nv_bfloat16* __restrict__ out,
                                                    int64_t n, float lr_t, float beta1, float beta2, float eps_t)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
        const float g = grad[i];
        const float mi = beta1 * m[i] + (1.f - beta1) * g;
        const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
        // lr (m / c1) / (sqrt(v / c2) + eps) = lr_t m / (sqrt(v) + eps_t), lr_t = lr sqrt(c2) / c1, eps_t = eps sqrt(c2)
        const float p = master[i] - lr_t * mi / (sqrtf(vi) + eps_t);
        m[i] = mi;
        v[i] = vi;
        master[i] = p;
        out[i] = __float2bfloat16_rn(p);
    }
}

// The target's density at every query voxel: the key (from int32 coordinates, or
// given), its lower bound among the sorted keys, the density where it is the same
// key.  One pass for what was twelve elementwise, search and gather launches with
// 64-bit intermediates of 3 words per voxel.
//
// The search is bound by its chain of dependent loads (22 for 3M keys), so each
// block keeps 2^TL_LOG evenly spaced keys in shared memory and bisects those
// first: half of the chain costs shared-memory latency, and the rest stays inside a
// range of a few KB that a warp's queries (neighbouring voxels of a leaf) share in
// L1.  The blocks are persistent, 8 to an SM, and a block that would see few
// queries loads fewer splitters.  Idx: 32-bit positions where the counts allow.
// 10.8M voxels among as many keys: 180 us (by torch's operators 897 us; with the warp's
// common range found 17 ways per round instead of the splitters 405 us, its 64-bit
// divisions and votes costing more than the loads they save); 1.5M: 28 us (139).
constexpr int TL_LOG = 11;
constexpr int TL_BLOCKS = 8; // per SM: 8 * 16 KB
template <bool PACK, class Idx>
__global__ void __launch_bounds__(256) k_target_lookup(const int64_t* __restrict__ keys, const float* __restrict__ density,
                                                        Idx count, const int32_t* __restrict__ ijk,
                                                        const int64_t* __restrict__ query, int64_t n, int splits, Idx gap,
                                                        float* __restrict__ value, uint8_t* __restrict__ hit)
{
    // splitter s: keys[s gap + gap - 1], the last key of part s (the largest integer past the end)
    __shared__ int64_t s_split[1 << TL_LOG];
    for (int s = threadIdx.x; s < splits; s += 256)
    {
        const int64_t at = (int64_t)s * gap + gap - 1;
        s_split[s] = at < (int64_t)count ? keys[at] : 0x7fffffffffffffffll;
    }
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256)
    {
        int64_t k;
        if (PACK)
        {
            // 21 bits per axis, shifted and joined as 64-bit integers
            const int64_t x = (int64_t)ijk[3 * i] + (1 << 20), y = (int64_t)ijk[3 * i + 1] + (1 << 20),
                          z = (int64_t)ijk[3 * i + 2] + (1 << 20);
            k = (int64_t)((uint64_t)x << 42 | (uint64_t)y << 21 | (uint64_t)z);
        }
        else
            k = query[i];
        // the part whose last key is the first one >= k (splits is a power of two)
        int part = 0;
        for (int step = splits >> 1; step; step >>= 1)
            part += s_split[part + step - 1] < k ? step : 0;
        // the lower bound lies in [first, first + len], len the part's keys (the last part
        // may end past the array, or be empty)
        const int64_t start = (int64_t)part * gap;
        Idx first = start < (int64_t)count ? (Idx)start : count;
        Idx len = count - first < gap ? count - first : gap;
        while (len > 0)
        {
            const Idx half = len >> 1;
            const bool below = keys[first + half] < k;
            first = below ? first + half + 1 : first;
            len = below ? len - half - 1 : half;
        }
        const bool same = first < count && keys[first] == k;
        value[i] = same ? density[first] : 0.f;
        if (hit)
            hit[i] = same ? 1 : 0;
    }
}

template <bool PACK, class Idx>
static void launch_target_lookup(const int64_t* keys, const float* density, int64_t count, const int32_t* ijk,
                                 const int64_t* query, int64_t n, float* value, uint8_t* hit, cudaStream_t s)
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t blocks = (n + 255) / 256;
    if (blocks > (int64_t)sms * TL_BLOCKS)
        blocks = (int64_t)sms * TL_BLOCKS;
    // a block of q queries spends q log2(splits) shared loads instead of cached ones for
    // splits / 256 loads per thread: as many splitters as it has queries, and no more than keys
    const int64_t q = (n + blocks - 1) / blocks;
    int splits = 1;
    while (splits < (1 << TL_LOG) && 2 * splits <= q && 2 * splits <= count)
        splits *= 2;
    const int64_t gap = count > 0 ? (count + splits - 1) / splits : 1; // (no keys: one empty part)
    k_target_lookup<PACK, Idx><<<(unsigned)blocks, 256, 0, s>>>(keys, density, (Idx)count, ijk, query, n, splits, (Idx)gap,
                                                                 value, hit);
    count_launch();
}

} // namespace vox

extern "C" int vox_target_lookup(const int64_t* keys, const float* density, int64_t count, const int32_t* ijk,
                                 const int64_t* query, int64_t n, float* value, uint8_t* hit, void* stream)
{
    if (n < 0 || count < 0 || (count > 0 && (!keys || !density)) || (n > 0 && (!value || !ijk == !query)))
        return VOX_ERR_ARGS;
    if (n == 0)
        return VOX_OK;
    const cudaStream_t s = (cudaStream_t)stream;
    const bool narrow = count < 1ll << 31;
    if (ijk && narrow)
        vox::launch_target_lookup<true, uint32_t>(keys, density, count, ijk, query, n, value, hit, s);
    else if (ijk)
        vox::launch_target_lookup<true, int64_t>(keys, density, count, ijk, query, n, value, hit, s);
    else if (narrow)
        vox::launch_target_lookup<false, uint32_t>(keys, density, count, ijk, query, n, value, hit, s);
    else
        vox::launch_target_lookup<false, int64_t>(keys, density, count, ijk, query, n, value, hit, s);
    return cudaGetLastError() == cudaSuccess ? VOX_OK : VOX_ERR_CUDA;
}

extern "C" int vox_adam_bf16(float* master, float* m, float* v, const float* grad, uint16_t* out_bf16, int64_t n,
                             float lr, float beta1, float beta2, float eps, int64_t step, void* stream)
{
    if (n < 0 || (n > 0 && (!master || !m || !v || !grad || !out_bf16)) || step < 1 || !(beta1 >= 0.f && beta1 < 1.f) ||
        !(beta2 >= 0.f && beta2 < 1.f))
        return VOX_ERR_ARGS;
    if (n == 0)
        return VOX_OK;
    const double c1 = 1.0 - pow((double)beta1, (double)step), c2 = 1.0 - pow((double)beta2, (double)step);
    const float lr_t = (float)((double)lr * sqrt(c2) / c1), eps_t = (float)((double)eps * sqrt(c2));
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t blocks = (n + 255) / 256;
    if (blocks > (int64_t)sms * 8)
        blocks = (int64_t)sms * 8;
    vox::k_adam_bf16<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(master, m, v, grad, (__nv_bfloat16*)out_bf16, n, lr_t,
                                                                          beta1, beta2, eps_t);
    vox::count_launch();
    return cudaGetLastError() == cudaSuccess ? VOX_OK : VOX_ERR_CUDA;
}
