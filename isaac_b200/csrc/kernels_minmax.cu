// Min/max of a source after its functor chain: MinMaxKernel / MinMaxParticleKernel
// (lib/isaac/isaac_min_max_kernel.hpp:22-97) followed by the host scan of
// CalcMinMaxIterator (lib/isaac.hpp:372-497).
//
// The reference keeps, per column, the first value in scan order among equal
// candidates (glm::min(a,b) = b<a ? b : a, and a strict '<' in the host scan),
// never lets NaN in, and starts from +/-FLT_MAX.  A single-pass grid reduction
// with the same comparison yields the same value for every input; the only
// values that compare equal yet differ in bits are +0 and -0, so when the
// result is zero a second pass finds which zero comes first in the reference's
// scan order (column x + y*X, then z, then particle index).
#include "isaacb_internal.h"

#include <algorithm>
#include <cfloat>

namespace isaacb
{
    constexpr int kMMThreads = 256;

    // voxel i of the interior in x, y, z order.  PLAIN: no ghost cells
    template<bool PLAIN>
    __device__ __forceinline__ float mm_value(const MinMaxParams& p, size_t i)
    {
        float v[4];
        if(!PLAIN)
        {
            const size_t row = i / size_t(p.g.ls[0]), z = row / size_t(p.g.ls[1]);
            i = z * p.pitchZ + (row - z * size_t(p.g.ls[1])) * p.pitchY + (i - row * size_t(p.g.ls[0]));
        }
        const float* sp = p.src + i * p.fdim;
        v[0] = __ldg(sp);
        v[1] = p.fdim > 1 ? __ldg(sp + 1) : 0.0f;
        v[2] = p.fdim > 2 ? __ldg(sp + 2) : 0.0f;
        v[3] = p.fdim > 3 ? __ldg(sp + 3) : 0.0f;
        return apply_chain(v, p.fdim, p.chain);
    }
    __device__ __forceinline__ float mm_particle(const MinMaxParams& p, uint32_t k)
    {
        float v[4];
        const float* sp = p.attr + size_t(k) * p.fdim;
        v[0] = __ldg(sp);
        v[1] = p.fdim > 1 ? __ldg(sp + 1) : 0.0f;
        v[2] = p.fdim > 2 ? __ldg(sp + 2) : 0.0f;
        v[3] = p.fdim > 3 ? __ldg(sp + 3) : 0.0f;
        return apply_chain(v, p.fdim, p.chain);
    }

    __device__ __forceinline__ void block_reduce(float& lo, float& hi, float* out)
    {
        __shared__ float sLo[kMMThreads / 32], sHi[kMMThreads / 32];
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
        {
            lo = gmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = gmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        const int w = threadIdx.x >> 5;
        if((threadIdx.x & 31) == 0)
        {
            sLo[w] = lo;
            sHi[w] = hi;
        }
        __syncthreads();
        if(threadIdx.x == 0)
        {
            float a = sLo[0], b = sHi[0];
            for(int i = 1; i < kMMThreads / 32; ++i)
            {
                a = gmin(a, sLo[i]);
                b = gmax(b, sHi[i]);
            }
            out[0] = a;
            out[1] = b;
        }
    }

    // The block's result joins the others': the last block to arrive reduces them all and
    // leaves the ticket at zero for the next launch.
    __device__ __forceinline__ void mm_finish(const MinMaxParams& p, float lo, float hi)
    {
        __shared__ bool last;
        block_reduce(lo, hi, p.partial + 2 * blockIdx.x);
        if(threadIdx.x == 0)
        {
            __threadfence();
            last = atomicAdd(p.ticket, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if(!last)
            return;
        __threadfence();
        lo = FLT_MAX;
        hi = -FLT_MAX;
        for(unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x)
        {
            lo = gmin(lo, __ldcg(p.partial + 2 * i));
            hi = gmax(hi, __ldcg(p.partial + 2 * i + 1));
        }
        block_reduce(lo, hi, p.result);
        if(threadIdx.x == 0)
            *p.ticket = 0u;
    }

    // any source or particle source, one value at a time.  PLAIN: no ghost cells (a pow chain
    // over 400 x 400 x 300 voxels 0.64 ms, 0.68 with the pitches asked for each value)
    template<bool PLAIN>
    __global__ void __launch_bounds__(kMMThreads) k_minmax(const __grid_constant__ MinMaxParams p)
    {
        float lo = FLT_MAX, hi = -FLT_MAX;
        if(!p.particle)
        {
            const size_t n = size_t(p.g.ls[0]) * p.g.ls[1] * p.g.ls[2];
            for(size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
            {
                const float v = mm_value<PLAIN>(p, i);
                lo = gmin(lo, v);
                hi = gmax(hi, v);
            }
        }
        else
        {
            const size_t n = size_t(p.g.lps[0]) * p.g.lps[1] * p.g.lps[2];
            for(size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x)
            {
                for(uint32_t k = __ldg(p.offsets + c); k < __ldg(p.offsets + c + 1); ++k)
                {
                    const float v = mm_particle(p, k);
                    lo = gmin(lo, v);
                    hi = gmax(hi, v);
                }
            }
        }
        mm_finish(p, lo, hi);
    }

    // A source without ghost cells, 16-byte aligned, its chain a LineChain: 4 voxels are FD
    // 16-byte loads, and a thread issues those of UNROLL groups before it uses one, 64 bytes
    // or more in flight each.  Bound by memory: one value at a time took 0.54 ms for a 512^3
    // scalar and 0.66 ms for a vector field, both together 1.26 ms with their reads; this takes
    // 0.36 ms for both, 5.9 TB/s.
    template<int FD, bool CHAIN>
    __global__ void __launch_bounds__(kMMThreads) k_minmax_vec(const __grid_constant__ MinMaxParams p, const __grid_constant__ LineChain chain)
    {
        constexpr int UNROLL = FD == 1 ? 4 : 2;
        float lo = FLT_MAX, hi = -FLT_MAX;
        const size_t n = size_t(p.g.ls[0]) * p.g.ls[1] * p.g.ls[2], groups = n / 4;
        const float4* src = reinterpret_cast<const float4*>(p.src);
        auto take = [&](float (&v)[4][FD]) {
            if(CHAIN)
                line_chain<4, FD>(v, FD, chain);
#pragma unroll
            for(int j = 0; j < 4; ++j)
            {
                lo = gmin(lo, v[j][0]);
                hi = gmax(hi, v[j][0]);
            }
        };
        const size_t stride = size_t(gridDim.x) * kMMThreads;
        for(size_t q = blockIdx.x * size_t(kMMThreads) + threadIdx.x; q < groups; q += UNROLL * stride)
        {
            float4 raw[UNROLL][FD];
#pragma unroll
            for(int u = 0; u < UNROLL; ++u)
#pragma unroll
                for(int c = 0; c < FD; ++c) // a group past the end repeats the first
                    raw[u][c] = __ldg(src + (q + u * stride < groups ? q + u * stride : q) * FD + c);
#pragma unroll
            for(int u = 0; u < UNROLL; ++u)
            {
                float f[4 * FD], v[4][FD];
#pragma unroll
                for(int c = 0; c < FD; ++c)
                    f[4 * c] = raw[u][c].x, f[4 * c + 1] = raw[u][c].y, f[4 * c + 2] = raw[u][c].z, f[4 * c + 3] = raw[u][c].w;
#pragma unroll
                for(int j = 0; j < 4; ++j)
#pragma unroll
                    for(int c = 0; c < FD; ++c)
                        v[j][c] = f[j * FD + c];
                take(v);
            }
        }
        if(blockIdx.x == 0 && threadIdx.x < n - 4 * groups)
        {
            const float v = mm_value<true>(p, 4 * groups + threadIdx.x);
            lo = gmin(lo, v);
            hi = gmax(hi, v);
        }
        mm_finish(p, lo, hi);
    }

    int minmax_blocks(const MinMaxParams& p, size_t perThread = 1)
    {
        const size_t n = p.particle ? size_t(p.g.lps[0]) * p.g.lps[1] * p.g.lps[2]
                                    : size_t(p.g.ls[0]) * p.g.ls[1] * p.g.ls[2];
        const size_t per = kMMThreads * perThread;
        return int(std::max<size_t>(1, std::min<size_t>((n + per - 1) / per, kMinMaxBlocks)));
    }

    void launch_minmax(const MinMaxParams& p, cudaStream_t s)
    {
        LineChain line;
        const bool plain = p.particle || p.pitchY == size_t(p.g.ls[0]);
        const bool vec = !p.particle && plain && (reinterpret_cast<uintptr_t>(p.src) & 15u) == 0
            && line_chain_of(p.chain, line);
        if(!vec)
        {
            if(plain)
                k_minmax<true><<<minmax_blocks(p), kMMThreads, 0, s>>>(p);
            else
                k_minmax<false><<<minmax_blocks(p), kMMThreads, 0, s>>>(p);
            return;
        }
        const int blocks = minmax_blocks(p, 4);
        switch(p.fdim)
        {
        case 1: line.idem ? k_minmax_vec<1, false><<<blocks, kMMThreads, 0, s>>>(p, line) : k_minmax_vec<1, true><<<blocks, kMMThreads, 0, s>>>(p, line); break;
        case 2: line.idem ? k_minmax_vec<2, false><<<blocks, kMMThreads, 0, s>>>(p, line) : k_minmax_vec<2, true><<<blocks, kMMThreads, 0, s>>>(p, line); break;
        case 3: line.idem ? k_minmax_vec<3, false><<<blocks, kMMThreads, 0, s>>>(p, line) : k_minmax_vec<3, true><<<blocks, kMMThreads, 0, s>>>(p, line); break;
        default: line.idem ? k_minmax_vec<4, false><<<blocks, kMMThreads, 0, s>>>(p, line) : k_minmax_vec<4, true><<<blocks, kMMThreads, 0, s>>>(p, line); break;
        }
    }

    // Reference scan-order key of the first +0 and the first -0:
    // keys[0] = first +0, keys[1] = first -0 (64-bit order keys, ULLONG_MAX if none)
    template<bool PLAIN>
    __global__ void __launch_bounds__(kMMThreads) k_minmax_zero_keys(const __grid_constant__ MinMaxParams p)
    {
        if(!p.particle)
        {
            const int LX = p.g.ls[0], LY = p.g.ls[1], LZ = p.g.ls[2];
            const size_t n = size_t(LX) * LY * LZ;
            for(size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
            {
                const float v = mm_value<PLAIN>(p, i);
                if(v == 0.0f)
                {
                    const size_t x = i % LX, y = (i / LX) % LY, z = i / (size_t(LX) * LY);
                    const unsigned long long key = (unsigned long long) ((y * LX + x) * LZ + z);
                    atomicMin(&p.keys[signbit(v) ? 1 : 0], key);
                }
            }
        }
        else
        {
            const int PX = p.g.lps[0], PY = p.g.lps[1], PZ = p.g.lps[2];
            const size_t n = size_t(PX) * PY * PZ;
            for(size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x)
            {
                const uint32_t k0 = __ldg(p.offsets + c), k1 = __ldg(p.offsets + c + 1);
                for(uint32_t k = k0; k < k1; ++k)
                {
                    const float v = mm_particle(p, k);
                    if(v == 0.0f)
                    {
                        const size_t x = c % PX, y = (c / PX) % PY, z = c / (size_t(PX) * PY);
                        // column, then z, then position in the cell (< 2^32 particles per cell)
                        const unsigned long long key
                            = ((unsigned long long) ((y * PX + x) * PZ + z) << 32) | (unsigned long long) (k - k0);
                        atomicMin(&p.keys[signbit(v) ? 1 : 0], key);
                    }
                }
            }
        }
    }

    void launch_minmax_zero_keys(const MinMaxParams& p, cudaStream_t s)
    {
        if(p.particle || p.pitchY == size_t(p.g.ls[0]))
            k_minmax_zero_keys<true><<<minmax_blocks(p), kMMThreads, 0, s>>>(p);
        else
            k_minmax_zero_keys<false><<<minmax_blocks(p), kMMThreads, 0, s>>>(p);
    }
} // namespace isaacb
