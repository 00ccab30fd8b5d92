// Many views of one or more contexts (e.g. the timesteps of a simulation) in
// one persistent launch.  No counterpart in the reference, which renders one
// view per doVisualization (lib/isaac.hpp:2008-2061).
//
// Every CTA pulls 32x8-pixel-sized tiles (any 256-pixel shape) from an atomic
// work queue over all views, stages the tile's view and context in shared
// memory, and renders each pixel exactly as the single-view pipeline does for a
// volume-only context: clear (ClearBufferKernel), shading of the empty G-buffer
// (ShadingKernel) and the combined volume march.  The frames are therefore
// bit-identical to isaacb_render's.
#include "isaacb_frame.cuh"
#include "isaacb_march.cuh"

#include <cfloat>
#include <type_traits>

namespace isaacb
{
    // the pixel without a volume: the shaded background, and its depth
    __device__ __forceinline__ uchar4 batch_surface(const BatchCtx& c, float3 dir, float& depth)
    {
        uchar4 col = to_byte4(c.bgSwizzled);
        depth = FLT_MAX;
        const ShadeParams sp{c.renderMode, c.aoWeight, c.bg};
        shade_values(sp, c.g, dir, col, f3(0, 0, 0), 0.0f, depth);
        return col;
    }

    // A view's buffer is stored to once a pixel and never read: it may be host or peer memory,
    // or another view's as well.  The march needs the registers that the surface would take
    // meanwhile, so the surface, the same for every direction that is a number, is formed again
    // after it (four 1080p views of 512^3 textures 13.7 ms; kept in a register 14.9, in shared
    // memory 14.0, read back from the buffer 13.5).
    template<bool LINEAR, bool SKIP, bool YFAST>
    __device__ __forceinline__ void batch_pixel(
        const BatchCtx& c, const View& v, float negZero, int px, int py, uchar4* out, unsigned long long& n)
    {
        float depth;
        Ray ray = pixel_to_ray(v, c.g, px, py);
        const uchar4 col = batch_surface(c, ray.dir, depth);
        if(!c.volume || !clip_ray(ray, v, c.g))
        {
            *out = col;
            return;
        }
        ray.endDepth = gmin(ray.endDepth, depth);
        if(ray.endDepth <= ray.startDepth)
        {
            *out = col;
            return;
        }
        if(ray.dir.x != ray.dir.x)
        {
            // not a number (a singular camera), nor is the colour of the one sample that the
            // march would take, in brick 0, unless it skips that
            const float q = SKIP && __ldg(c.volFlag) == 0 ? 0.0f : ray.dir.x;
            *out = over_surface(make_float4(q, q, q, q), col);
            n += 1;
            return;
        }
        const March m = march_setup(ray, c.g, v.scale, c.step);
        const float factor = m.factor * c.totalWeightAll;
        const VolTexRef tex{c.g, c.volQ, c.volFlag, negZero};
        float4 color;
        if(LINEAR && march_in_range(c.g, m))
            color = march_combined<LINEAR, false, SKIP, YFAST, 1>(tex, m, factor, n);
        else
            color = march_combined<LINEAR, true, SKIP, YFAST, 1>(tex, m, factor, n);
        *out = over_surface(color, batch_surface(c, f3(0, 0, 1), depth));
    }

    // 4 CTAs per SM (64 registers): two merges and 8 views of 512^3 textures take 20.9 ms; 3
    // CTAs at 80 registers 21.5, 5 at 48 with spills 22.8
    __global__ void __launch_bounds__(256, 4) k_batch(const __grid_constant__ BatchParams bp)
    {
        __shared__ View sv;
        __shared__ BatchCtx sc;
        __shared__ int sTile, sView;
        unsigned long long n = 0;
        const int t = threadIdx.x;
        for(;;)
        {
            if(t == 0)
            {
                const int tile = atomicAdd(bp.counter, 1);
                int v = -1;
                if(tile < bp.totalTiles)
                    for(int i = 0; i < bp.nViews; ++i)
                        if(tile >= bp.views[i].tileBase && tile < bp.views[i].tileBase + bp.views[i].tiles)
                        {
                            v = i;
                            break;
                        }
                sTile = tile;
                sView = v;
            }
            __syncthreads();
            const int tile = sTile, vi = sView;
            if(tile >= bp.totalTiles || vi < 0)
                break;
            const BatchView& bv = bp.views[vi];
            // stage the view and its context in shared memory
            {
                const int* src = reinterpret_cast<const int*>(&bp.ctxs[bv.ctx]);
                int* dst = reinterpret_cast<int*>(&sc);
                for(int i = t; i < int(sizeof(BatchCtx) / 4); i += blockDim.x)
                    dst[i] = src[i];
                if(t < 16)
                    sv.inv[t] = bv.inv[t];
                if(t == 0)
                {
                    sv.W = bv.W;
                    sv.H = bv.H;
                }
            }
            __syncthreads();
            if(t == 0)
            {
                sv.scale = sc.scale;
                sv.clipCount = sc.clipCount;
            }
            for(int i = t; i < kMaxClip * 3; i += blockDim.x)
            {
                sv.clipPos[i / 3][i % 3] = sc.clipPos[i / 3][i % 3];
                sv.clipNrm[i / 3][i % 3] = sc.clipNrm[i / 3][i % 3];
            }
            __syncthreads();
            // pixel of this thread inside the tile: 8 x 4 pixels a warp, lanes along rows, for
            // x-fastest slots; 4 x 8 where the tile has them for y-fastest ones, lanes down
            // columns or along rows by the view (k_shade_volume)
            const bool yfast = sc.g.yfast != 0, tall = yfast && (bp.tileH & 7) == 0, down = yfast && bv.laneColumns != 0;
            const int ww = tall ? 4 : 8, wh = tall ? 8 : 4, warpsX = bp.tileW / ww;
            const int w = t >> 5, l = t & 31;
            const int ox = (w % warpsX) * ww + (down ? l / wh : l % ww);
            const int oy = (w / warpsX) * wh + (down ? l % wh : l / ww);
            const int local = tile - bv.tileBase;
            const int px = (local % bv.tilesX) * bp.tileW + ox;
            const int py = (local / bv.tilesX) * bp.tileH + oy;
            if(px < sv.W && py < sv.H)
            {
                // auto (-1): skip when the context's last merge found empty bricks
                const bool skip = sc.skipEmpty >= 0 ? sc.skipEmpty != 0 : __ldg(sc.emptyCount) != 0u;
                uchar4* out = bv.out + (size_t(py) * sv.W + px);
                auto pixel = [&](auto linear, auto y) {
                    if(skip)
                        batch_pixel<decltype(linear)::value, true, decltype(y)::value>(sc, sv, bp.negZero, px, py, out, n);
                    else
                        batch_pixel<decltype(linear)::value, false, decltype(y)::value>(sc, sv, bp.negZero, px, py, out, n);
                };
                const std::true_type yes;
                const std::false_type no;
                if(sc.interpolation)
                    yfast ? pixel(yes, yes) : pixel(yes, no);
                else
                    yfast ? pixel(no, yes) : pixel(no, no);
            }
            __syncthreads();
        }
        if(bp.samples)
            count_samples(bp.samples, n);
    }

    void launch_batch(const BatchParams& p, int blocks, cudaStream_t s)
    {
        k_batch<<<blocks, 256, 0, s>>>(p);
    }

    int batch_max_blocks_per_sm()
    {
        int n = 0;
        if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_batch, 256, 0) != cudaSuccess)
            return 1;
        return n > 0 ? n : 1;
    }
} // namespace isaacb
