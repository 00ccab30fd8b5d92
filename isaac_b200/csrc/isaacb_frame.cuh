// Per-pixel helpers shared by the combined and the per-source frame kernels.
#pragma once

#include "isaacb_internal.h"

#include <cfloat>

namespace isaacb
{
    __device__ __forceinline__ size_t pix(const FrameParams& p, int x, int y)
    {
        return size_t(y) * p.v.W + x;
    }

    __device__ __forceinline__ void count_samples(unsigned long long* ctr, unsigned long long n)
    {
        // one atomic per warp
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            n += __shfl_xor_sync(0xffffffffu, n, o);
        if((threadIdx.x & 31) == 0 && n)
            atomicAdd(ctr, n);
    }

    // ------------------------------------------------------------------ shading + volume
    // ShadingKernel (lib/isaac/isaac_common_kernel.hpp:220-320) for rank 0
    __device__ __forceinline__ float4 hsva_rank0(float a)
    {
        // getHSVA(halton(0,3)*2pi, 1, 1, a) = (1, 0, 0, a)
        return make_float4(1.0f, 0.0f, 0.0f, a);
    }

    // the settings ShadingKernel reads
    struct ShadeParams
    {
        int32_t renderMode;
        float aoWeight;
        float4 bg;
    };

    // ShadingKernel on one pixel's G-buffer values along its ray direction: colour and depth
    // are updated in place.  A zero normal (no surface) has light and specular terms of
    // exactly 0 for any direction of length 1, so they are not formed.
    __device__ __forceinline__ void shade_values(
        const ShadeParams& sp,
        const Geom& g,
        float3 dir,
        uchar4& gcolor,
        float3 normal,
        float aoRaw,
        float& depth)
    {
        float4 color = from_byte4(gcolor);
        const float aoStrength = 1.0f - aoRaw;
        const int mode = sp.renderMode;
        if(mode == 7)
            color = hsva_rank0(color.w);
        if(mode < 3 || mode == 7)
        {
            float lightFactor = 0.0f, specular = 0.0f;
            // (a direction that is not a number must reach the general terms)
            if(normal.x != 0.0f || normal.y != 0.0f || normal.z != 0.0f || !(dot3(dir, dir) > 0.5f))
            {
                const float3 lightDir = neg3(dir);
                lightFactor = fabsf(dot3(normal, lightDir));
                const float3 halfVector = normalize3(add3(neg3(dir), lightDir));
                specular = dot3(normal, halfVector);
                const double s2 = double(specular) * double(specular);
                specular = float(s2 * s2);
                specular *= 0.5f;
                if(mode == 1)
                    specular = 0.0f;
            }
            const float w = sp.aoWeight;
            const float aoFactor = ((1.0f - w) + w * aoStrength);
            lightFactor += aoFactor;
            lightFactor *= 0.5f;
            float4 sh;
            sh.x = gmin(color.x * lightFactor + specular, 1.0f);
            sh.y = gmin(color.y * lightFactor + specular, 1.0f);
            sh.z = gmin(color.z * lightFactor + specular, 1.0f);
            sh.w = color.w;
            gcolor = to_byte4(sh);
            if(mode == 2 || mode == 7)
                depth = 0.0f;
        }
        else if(mode == 3)
        {
            gcolor = to_byte4(make_float4(sp.bg.w, sp.bg.z, sp.bg.y, color.w));
        }
        else if(mode == 4)
        {
            gcolor = to_byte4(make_float4(normal.x * 0.5f + 0.5f, normal.y * 0.5f + 0.5f, normal.z * 0.5f + 0.5f, color.w));
            depth = 0.0f;
        }
        else if(mode == 5)
        {
            const float d = depth / float(g.maxGss);
            gcolor = to_byte4(make_float4(d, d, d, color.w));
            depth = 0.0f;
        }
        else if(mode == 6)
        {
            const float w = sp.aoWeight;
            const float aoFactor = ((1.0f - w) + w * aoStrength);
            gcolor = to_byte4(make_float4(aoFactor, aoFactor, aoFactor, color.w));
            depth = 0.0f;
        }
        else if(mode == 8)
        {
            gcolor = to_byte4(hsva_rank0(1.0f));
            depth = 0.0f;
        }
    }

    // the cleared G-buffer beside the colour (ClearBufferKernel,
    // lib/isaac/isaac_common_kernel.hpp:195-217)
    __device__ __forceinline__ void store_clear(const FrameParams& p, size_t o, float depth)
    {
        p.normal[3 * o] = 0.0f;
        p.normal[3 * o + 1] = 0.0f;
        p.normal[3 * o + 2] = 0.0f;
        p.depth[o] = depth;
        p.ao[o] = 0.0f;
    }
    // Shades pixel o in place along its ray direction and returns its depth.  CLEAN: no pass
    // has drawn a surface, so that the pixel has the clear values, which are written here
    // instead of by a pass of their own.  The results go to memory rather than stay in
    // registers, of which the march that follows needs every one.
    template<bool CLEAN>
    __device__ __forceinline__ float shade_surface(const FrameParams& p, float3 dir, size_t o)
    {
        const ShadeParams sp{p.renderMode, p.aoWeight, p.bg};
        uchar4 c = CLEAN ? to_byte4(p.bgSwizzled) : p.color[o];
        float depth = CLEAN ? FLT_MAX : p.depth[o];
        const float3 n = CLEAN ? f3(0, 0, 0) : f3(p.normal[3 * o], p.normal[3 * o + 1], p.normal[3 * o + 2]);
        shade_values(sp, p.g, dir, c, n, CLEAN ? 0.0f : p.ao[o], depth);
        p.color[o] = c;
        if(CLEAN)
            store_clear(p, o, depth);
        else if(p.shadeDepth)
            p.depth[o] = depth;
        return depth;
    }
    // front colour over the shaded surface
    __device__ __forceinline__ uchar4 over_surface(float4 c, uchar4 surface)
    {
        const float4 solid = from_byte4(surface);
        const float r = 1.0f - c.w;
        return to_byte4(make_float4(c.x + r * solid.x, c.y + r * solid.y, c.z + r * solid.z, c.w + r * solid.w));
    }
} // namespace isaacb
