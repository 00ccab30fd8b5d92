// The combined-texture ray-march shared by the single-view and the batched
// kernels.  Included by the kernel translation units only.
#pragma once

#include "isaacb_internal.h"

namespace isaacb
{
    // the texture a march reads: geometry, quad bricks and per-brick emptiness
    struct VolTexRef
    {
        Geom g;
        const uint4* volQ;
        const uint8_t* volFlag;
        float negZero; // -0.0f from a kernel parameter (f2p_mul_exact), for march_ahead
    };

    // the last step index, at least fi and at most fe, whose position c0 + sv * i stays inside
    // the sample region [8b-1, 8b+7) of the brick of apron-shifted texel (ax, ay, az)
    __device__ __forceinline__ float last_step_in_brick(int ax, int ay, int az, const float (&c0)[3], const float (&sv)[3], float fi, float fe)
    {
        float tEnd = 3.0e38f;
        const float bl[3] = {float(ax & ~7) - 1.0f, float(ay & ~7) - 1.0f, float(az & ~7) - 1.0f};
#pragma unroll
        for(int a = 0; a < 3; ++a)
        {
            if(sv[a] > 0.0f)
                tEnd = fminf(tEnd, (bl[a] + 8.0f - c0[a]) / sv[a]);
            else if(sv[a] < 0.0f)
                tEnd = fminf(tEnd, (bl[a] - c0[a]) / sv[a]);
        }
        // margin: 1e-3 steps plus the float rounding of tEnd itself
        return fminf(fmaxf(floorf(tEnd - (1.0e-3f + 1.0e-6f * fabsf(tEnd))), fi), fe);
    }

    // a slot's load that stays where it is written: the compiler moves an ordinary one past
    // the exits between the samples of a trip, next to its use, and nothing is ahead any more
    __device__ __forceinline__ uint4 load_slot_here(const uint4* at)
    {
        uint4 v;
        asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(at));
        return v;
    }

    // the weight words of two samples at once, one per packed lane, at the fractional
    // positions (fx, fy, fz): w[l][0..3] are lane l's 16-bit fixed-point weight pairs
    // (texel x0 | texel x0 + 1 << 16) of rows y0 and y0 + 1 of plane z0, then of z0 + 1.
    // With the samples in the lanes every product of the chain is packed and no weight has
    // to be broadcast into a pair; each lane rounds like the scalar operations.
    __device__ __forceinline__ void trilinear_weights2(f2p fx, f2p fy, f2p fz, f2p negZero, uint32_t (&w)[2][4])
    {
        constexpr float kUnit = 65535.0f;
        const f2p one = f2p_make(1.0f, 1.0f), unit = f2p_make(kUnit, kUnit);
        const f2p gx = f2p_sub(one, fx), gy = f2p_sub(one, fy);
        // a product that feeds a subtraction: rounded on its own (f2p_mul_exact)
        const f2p fzU = f2p_mul_exact(fz, unit, negZero), gzU = f2p_sub(unit, fzU);
        const f2p r[4] = {f2p_mul(gx, gy), f2p_mul(fx, gy), f2p_mul(gx, fy), f2p_mul(fx, fy)};
        // round(w * 65535) lands in the low bits of 2^23 + w * 65535 (one rounding per lane,
        // to nearest, as the scalar fmaf); <= 65535, so the low 16 bits are the weight
        const f2p M = f2p_make(8388608.0f, 8388608.0f);
#pragma unroll
        for(int q = 0; q < 4; ++q)
        {
            const f2p z = q < 2 ? gzU : fzU;
            float a0, a1, b0, b1;
            f2p_split(f2p_fma(r[2 * (q & 1)], z, M), a0, a1);
            f2p_split(f2p_fma(r[2 * (q & 1) + 1], z, M), b0, b1);
            w[0][q] = __byte_perm(__float_as_uint(a0), __float_as_uint(b0), 0x5410u);
            w[1][q] = __byte_perm(__float_as_uint(a1), __float_as_uint(b1), 0x5410u);
        }
    }

    // the trilinear sample of channel-major slots A (plane z0) and B (plane z0 + 1) with the
    // weight words w, in units of 1/65535 byte: an exact integer sum of 16-bit fixed-point
    // weights times bytes (the weights sum to at most 65535 + 4, so it stays below 2^24)
    __device__ __forceinline__ float4 trilinear_dp2a(uint4 A, uint4 B, const uint32_t (&w)[4])
    {
        auto tri = [&](uint32_t a, uint32_t b) {
            return __uint2float_rn(dp2a_hi(w[3], b, dp2a_lo(w[2], b, dp2a_hi(w[1], a, dp2a_lo(w[0], a, 0u)))));
        };
        return make_float4(tri(A.x, B.x), tri(A.y, B.y), tri(A.z, B.z), tri(A.w, B.w));
    }

    // Front-to-back march of CombinedVolumeRenderKernel (lib/isaac/isaac_volume_kernel.hpp:61-87)
    // at the reference's sample positions.  Differences from the exact form, all far
    // below one output LSB and covered by the parity tests:
    //  * pos - 0.5 is one fmaf per axis and the /255 normalisation is folded into the
    //    per-ray factor;
    //  * the trilinear is an integer dot product: the 8 FP32 weights are rounded to
    //    16-bit fixed point (w * 65535), and each channel-major slot word (channel c of
    //    the 2x2 texels of one plane) is weighed whole by dp2a.lo + dp2a.hi.  The sums
    //    are exact integers below 2^24, so the only error is the weights' rounding,
    //    at most 8 * 0.5 / 65535 * 255 = 0.016 byte units per sample;
    //  * empty-space skipping: a brick whose texels (apron included) are all zero
    //    yields exactly zero samples, so the samples inside it are counted but not
    //    evaluated -- adding zero leaves the colour unchanged.
    // CLAMP keeps every coordinate inside the volume; a LINEAR ray whose first and
    // last sample lie strictly inside needs no per-sample clamp (positions are affine
    // in the step index, rounding is far below the 1e-3 margin).
    // YFAST: the texture's slots are y fastest (Geom::yfast), else x fastest.
    //
    // A trip takes 2 * PAIRS samples, all their slots loading before any is weighed.  Two
    // consecutive samples are the two lanes of every packed position and weight operation
    // (f32x2); they are composited one after the other, in order, and a sample past the last
    // step or the opacity limit takes the factor 0 and adds exactly nothing.  There is no
    // branch between a trip's samples: with one, the compiler moved each sample's loads
    // behind it and a ray waited for every sample's loads in turn.
    template<bool LINEAR, bool CLAMP, bool SKIP, bool YFAST, int PAIRS>
    __device__ __forceinline__ float4 march_combined(
        const VolTexRef& p,
        const March& m,
        float factor,
        unsigned long long& count)
    {
        const Geom& g = p.g;
        const float k = factor / 255.0f;
        // trilinear samples come out scaled by the weights' fixed-point unit 65535
        constexpr float kUnit = 65535.0f;
        const float kS = LINEAR ? k / kUnit : k;
        const float off = LINEAR ? 0.5f : 0.0f;
        const float c0x = m.startU.x - off, c0y = m.startU.y - off, c0z = m.startU.z - off;
        const float svx = m.stepVec.x, svy = m.stepVec.y, svz = m.stepVec.z;
        const float lo = LINEAR ? -1.0f : 0.0f;
        const float hx = float(g.ls[0] - 1), hy = float(g.ls[1] - 1), hz = float(g.ls[2] - 1);
        const int nb0 = g.nb[0], nb1 = g.nb[1];
        // the slot of apron-shifted coordinates as a sum over the axes: with b = a >> 3 and
        // l = a & 7 per axis, b * stride + l * step == a * step + b * (stride - 8 * step);
        // the in-brick steps of x and y are (1, 8), or (8, 1) for y-fastest slots
        constexpr uint32_t stepX = YFAST ? 8u : 1u, stepY = YFAST ? 1u : 8u, kx = 576u - 8u * stepX;
        const uint32_t sy = uint32_t(nb0) * uint32_t(kSlotsPerBrick) - 8u * stepY;
        const uint32_t sz = uint32_t(nb1) * uint32_t(nb0) * uint32_t(kSlotsPerBrick) - 512u;
        // floor(c) + 1, the apron-shifted coordinate a, by a round-down add of 1.5 * 2^23 + 1:
        // the sum's bits are kBits + a, and kBits is a multiple of 8, so bits >> 3 is
        // (kBits >> 3) + (a >> 3) and the constants leave the slot as one offset (mod 2^32)
        constexpr float kFloor = 12582913.0f;
        constexpr uint32_t kBits = 0x4B400000u;
        const uint32_t slot0 = 0u - (stepX + stepY + 64u) * kBits - (kx + sy + sz) * (kBits >> 3);
        const f2p sv2[3] = {f2p_make(svx, svx), f2p_make(svy, svy), f2p_make(svz, svz)};
        const f2p c02[3] = {f2p_make(c0x, c0x), f2p_make(c0y, c0y), f2p_make(c0z, c0z)};
        const f2p floor2 = f2p_make(kFloor, kFloor), nz = f2p_make(p.negZero, p.negZero);
        f2p rg = f2p_make(0.0f, 0.0f), ba = rg; // colour so far: (red, green), (blue, alpha)
        float alpha = 0.0f;
        int curBrick = -1;
        bool empty = false;
        const float fs = float(m.startSteps), fe = float(m.endSteps);
        float fi = fs;
        while(fi <= fe)
        {
            f2p fr[PAIRS][3];
            uint32_t slot[2 * PAIRS];
            int brick = 0, ax = 0, ay = 0, az = 0; // of the first sample
#pragma unroll
            for(int q = 0; q < PAIRS; ++q)
            {
                const f2p fq = f2p_make(q == 0 ? fi : fminf(fi + float(2 * q), fe), fminf(fi + float(2 * q + 1), fe));
                uint32_t tb[3][2];
#pragma unroll
                for(int a = 0; a < 3; ++a)
                {
                    f2p c = f2p_fma(sv2[a], fq, c02[a]);
                    if(CLAMP)
                    {
                        const float h = a == 0 ? hx : a == 1 ? hy : hz;
                        float u, v;
                        f2p_split(c, u, v);
                        c = f2p_make(fminf(fmaxf(u, lo), h), fminf(fmaxf(v, lo), h));
                    }
                    const f2p t = f2p_add_rd(c, floor2);
                    fr[q][a] = f2p_sub(c, f2p_sub(t, floor2));
                    float t0, t1;
                    f2p_split(t, t0, t1);
                    tb[a][0] = __float_as_uint(t0);
                    tb[a][1] = __float_as_uint(t1);
                }
#pragma unroll
                for(int l = 0; l < 2; ++l)
                    slot[2 * q + l] = (tb[0][l] >> 3) * kx + (tb[0][l] * stepX + slot0) + ((tb[1][l] >> 3) * sy + tb[1][l] * stepY)
                        + ((tb[2][l] >> 3) * sz + tb[2][l] * 64u);
                if(SKIP && q == 0)
                {
                    ax = int(tb[0][0] - kBits), ay = int(tb[1][0] - kBits), az = int(tb[2][0] - kBits);
                    brick = ((az >> 3) * nb1 + (ay >> 3)) * nb0 + (ax >> 3);
                }
            }
            // an empty brick under the first sample of the trip ends it; a later sample of
            // the trip in one is weighed and adds exactly zero
            if(SKIP && brick != curBrick)
            {
                curBrick = brick;
                empty = __ldg(p.volFlag + brick) == 0;
            }
            if(SKIP && empty)
            {
                const float sv[3] = {svx, svy, svz};
                const float c0[3] = {c0x, c0y, c0z};
                const float last = last_step_in_brick(ax, ay, az, c0, sv, fi, fe);
                fi = last + 1.0f;
                continue;
            }
            // channel-major slots: A.c / B.c = channel c of the 2x2 texels of planes z0 / z0+1
            uint4 A[2 * PAIRS], B[2 * PAIRS];
#pragma unroll
            for(int j = 0; j < 2 * PAIRS; ++j)
            {
                A[j] = load_slot_here(p.volQ + slot[j]);
                if(LINEAR)
                    B[j] = load_slot_here(p.volQ + slot[j] + 64);
            }
            uint32_t w[PAIRS][2][4];
            if(LINEAR)
#pragma unroll
                for(int q = 0; q < PAIRS; ++q)
                    trilinear_weights2(fr[q][0], fr[q][1], fr[q][2], nz, w[q]);
            // a sample past the last step or the opacity limit takes the factor 0 and adds
            // exactly nothing: no branch parts the trip's loads from their uses
            bool done = false;
#pragma unroll
            for(int j = 0; j < 2 * PAIRS; ++j)
            {
                float4 r;
                if(LINEAR)
                    r = trilinear_dp2a(A[j], B[j], w[j >> 1][j & 1]);
                else // texel (x0, y0) of the slot: byte 0 of each channel word
                    r = make_float4(ubyte_f(A[j].x, 0), ubyte_f(A[j].y, 0), ubyte_f(A[j].z, 0), ubyte_f(A[j].w, 0));
                const bool take = j == 0 || (!done && fi <= fe);
                const float s = take ? (1.0f - alpha) * kS : 0.0f;
                rg = f2p_fma(f2p_make(s, s), f2p_make(r.x, r.y), rg);
                ba = f2p_fma(f2p_make(s, s), f2p_make(r.z, r.w), ba);
                float blue;
                f2p_split(ba, blue, alpha);
                fi += take ? 1.0f : 0.0f;
                done = done || alpha > 0.99f;
            }
            if(done)
                break;
        }
        count += (unsigned long long) (fminf(fi, fe + 1.0f) - fs);
        float4 color;
        f2p_split(rg, color.x, color.y);
        f2p_split(ba, color.z, color.w);
        return color;
    }

    // a LINEAR ray needs no clamp if both end samples are inside [-1, L) by a margin
    __device__ __forceinline__ bool march_in_range(const Geom& g, const March& m)
    {
        const float fs = float(m.startSteps), fe = float(m.endSteps);
        const float c0[3] = {m.startU.x - 0.5f, m.startU.y - 0.5f, m.startU.z - 0.5f};
        const float sv[3] = {m.stepVec.x, m.stepVec.y, m.stepVec.z};
        bool ok = true;
#pragma unroll
        for(int a = 0; a < 3; ++a)
        {
            const float a0 = fmaf(sv[a], fs, c0[a]), a1 = fmaf(sv[a], fe, c0[a]);
            ok = ok && fminf(a0, a1) >= -0.999f && fmaxf(a0, a1) <= float(g.ls[a]) - 0.001f;
        }
        return ok;
    }

} // namespace isaacb
