// Launch interface of the tensor-core convolution kernels (recon_gemm.cu),
// shared with the frame reconstructor (recon.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace isaacb
{
    // forward / input-gradient implicit GEMM (see recon_gemm.cu)
    struct ConvGemmParams
    {
        const __nv_bfloat16* x; // gather source, NHWC [B][H][W][Cg]
        const __nv_bfloat16* w; // packed weights [Npad][Kpad]
        const float* bias; // [Cout] or null
        __nv_bfloat16* y; // NHWC [B][Ho][Wo][Cout] (unless yf)
        float* yf; // FP32 output instead of y
        const __nv_bfloat16* mask; // output *= (mask > 0), NHWC like y, or null
        int B, H, W, Cg;
        int Ho, Wo, Cout, Npad, Kpad;
        int ks, stride, pad, transposed;
        int relu, accumulate;
        int step, tiles; // set by the launcher: residue classes per axis of the output pixels, and all classes' tiles
        int* errorFlag;
        // failure-detection check: non-zero = before any copy or MMA, wait this many ns on
        // an mbarrier that nothing arrives at, raise errorFlag, release TMEM and return
        unsigned long long waitCheckNs;
        // row-tile kernel only (k_conv_row):
        // implicit concatenation (cp.async producer, 1x1): the first upC input channels
        // come from xUp, [B][upInH][upInW][upC], read at the nearest coarse pixel
        // (min(y/2, upInH-1), min(x/2, upInW-1)); the other Cg - upC from x, whose pixels
        // then hold Cg - upC channels; null = off
        const __nv_bfloat16* xUp;
        int upC, upInH, upInW;
        // host launch hint (row-tile kernel): launch as a programmatic dependent of the
        // stream's previous kernel, so that its CTAs load their weights while that kernel
        // drains; the kernel reads its input only after griddepcontrol.wait
        int pdl;
    };

    // v / 255 rounded to nearest, for v in quarters from 0 to 255 (Markstein's correction of
    // v times the rounded reciprocal; the 1021 values give the quotient, bit for bit)
    __device__ __forceinline__ float div255(float v)
    {
        constexpr float rcp = 1.0f / 255.0f;
        const float q = __fmul_rn(v, rcp);
        return __fmaf_rn(__fmaf_rn(-255.0f, q, v), rcp, q);
    }

    // bilinear x2 of a half-size RGBA8 frame at full-size pixel (X, Y), aligned with the
    // renderer's pixel positions (integer coordinates): even pixels copy, odd ones
    // average two neighbours; values in [0, 1]
    __device__ __forceinline__ float4 bilinear2_rgba(const uchar4* __restrict__ low, int h, int w, int X, int Y)
    {
        const int ya = Y >> 1, yb = min((Y + 1) >> 1, h - 1);
        const int xa = X >> 1, xb = min((X + 1) >> 1, w - 1);
        const float wy = (Y & 1) ? 0.5f : 0.0f, wx = (X & 1) ? 0.5f : 0.0f;
        const uchar4 a = __ldg(low + size_t(ya) * w + xa), b = __ldg(low + size_t(ya) * w + xb);
        const uchar4 c = __ldg(low + size_t(yb) * w + xa), d = __ldg(low + size_t(yb) * w + xb);
        auto mix = [&](float va, float vb, float vc, float vd) {
            const float r0 = va * (1.0f - wx) + vb * wx;
            const float r1 = vc * (1.0f - wx) + vd * wx;
            return div255(r0 * (1.0f - wy) + r1 * wy);
        };
        return make_float4(mix(a.x, b.x, c.x, d.x), mix(a.y, b.y, c.y, d.y), mix(a.z, b.z, c.z, d.z), mix(a.w, b.w, c.w, d.w));
    }
    // the four full-size pixels (2x + (k & 1), 2y + (k >> 1)) of half-size pixel (x, y): the
    // same values (sums of bytes in quarters are exact) from one load of each neighbour.  The
    // frame and loss kernels took most of their time in 16 and 32 IEEE divisions a half-size
    // pixel and in loading each neighbour up to four times: 960x540 inference 240 -> 233 us,
    // a step of 16 128 x 128 pairs 702 -> 687 us.
    __device__ __forceinline__ void bilinear2_quad(const uchar4* __restrict__ low, int h, int w, int x, int y, float4 (&o)[4])
    {
        const int x1 = min(x + 1, w - 1);
        const uchar4* row0 = low + size_t(y) * w;
        const uchar4* row1 = low + size_t(min(y + 1, h - 1)) * w;
        const uchar4 a = __ldg(row0 + x), b = __ldg(row0 + x1), c = __ldg(row1 + x), d = __ldg(row1 + x1);
        auto mix = [&](uint8_t va, uint8_t vb, uint8_t vc, uint8_t vd, float& o0, float& o1, float& o2, float& o3) {
            const uint32_t ab = uint32_t(va) + vb, ac = uint32_t(va) + vc;
            o0 = div255(float(va));
            o1 = div255(0.5f * float(ab));
            o2 = div255(0.5f * float(ac));
            o3 = div255(0.25f * float(ab + vc + vd));
        };
        mix(a.x, b.x, c.x, d.x, o[0].x, o[1].x, o[2].x, o[3].x);
        mix(a.y, b.y, c.y, d.y, o[0].y, o[1].y, o[2].y, o[3].y);
        mix(a.z, b.z, c.z, d.z, o[0].z, o[1].z, o[2].z, o[3].z);
        mix(a.w, b.w, c.w, d.w, o[0].w, o[1].w, o[2].w, o[3].w);
    }

    // a value in [0, 1] as a byte: round to nearest, clamped
    __device__ __forceinline__ uint8_t unit_byte(float v)
    {
        return uint8_t(__float2int_rn(fminf(fmaxf(v * 255.0f, 0.0f), 255.0f)));
    }

    // weight gradient (see recon_gemm.cu)
    struct WgradParams
    {
        const __nv_bfloat16* x; // layer input [B][H][W][Cin]
        const __nv_bfloat16* dy; // output gradient [B][Ho][Wo][Cout]
        float* dw; // [Mtot][Npad], accumulated
        int B, H, W, Cin, Ho, Wo, Cout, Npad;
        int ks, stride, pad;
        int Mtot; // ks*ks*Cin
        // implicit concatenation as in ConvGemmParams (1x1): the first upC input channels come
        // from xUp at the nearest coarse pixel, the other Cin - upC from x; null = off
        const __nv_bfloat16* xUp;
        int upC, upInH, upInW;
        int chunksPerSplit, mTiles; // set by the launcher
        int* errorFlag;
    };
    // the layers of one launch; CTA i works on layer l with first[l] <= i < first[l + 1]
    constexpr int kWgradLayers = 12;
    struct WgradTable
    {
        WgradParams layer[kWgradLayers];
        int first[kWgradLayers + 1];
    };

    size_t conv_gemm_smem(int Npad, int Kpad);
    // the row-tile kernel takes this convolution (and then honours xUp)
    bool row_tiles_apply(const ConvGemmParams& p);
    // false where no kernel takes it: nothing was launched
    bool launch_conv_gemm(ConvGemmParams p, cudaStream_t s);
    // the weight gradients of n layers (1 to kWgradLayers) in one launch; false as above
    bool launch_conv_wgrad(const WgradParams* layers, int n, cudaStream_t s);
} // namespace isaacb
