// Convolutions as implicit GEMMs on the sm_100a tensor cores (tcgen05).
//
// Forward and input-gradient ("dgrad") passes share k_conv_gemm:
//   Y[p][n] = sum_k A[p][k] * Wp[n][k],  k = tap * Cg + c,
// where A is the im2col gather of the NHWC bf16 source (never materialised:
// each CTA gathers its 128-row x 64-column K-slices straight into shared
// memory with zero-filling cp.async), Wp is the packed bf16 weight matrix
// held whole in shared memory, and the FP32 accumulator lives in TMEM.  One
// thread issues the MMAs (M=128, N=Npad, K=16 per instruction) and commits
// them to per-stage mbarriers that recycle the shared-memory stages; the
// epilogue reads TMEM with tcgen05.ld and fuses bias, ReLU, the ReLU mask of
// the backward pass, accumulation into an existing gradient and the bf16 or
// FP32 store.  The gather has two forms:
//   forward     input pixel = out * stride - pad + tap
//   transposed  input pixel = (out + pad - tap) / stride when divisible
// The transposed form with the per-tap transposed weights is the gradient
// of the forward form with respect to its input.
//
// The weight gradient ("wgrad") is k_conv_wgrad:
//   dW[(tap, ci)][co] = sum_p X[in(p, tap)][ci] * dY[p][co]
// with both operands MN-major (channels contiguous in NHWC), the pixel axis
// as the reduction split over CTAs, and FP32 partial sums added atomically.
//
// Every mbarrier wait is bounded; on a timeout the kernel raises the error
// flag, stops issuing work, waits (bounded) for its MMAs and frees its TMEM.
#include "../../include/isaac_b200.h"
#include "isaacb_internal.h"
#include "isaacb_conv.h"
#include "isaacb_tc.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <string>

namespace isaacb
{
    void set_global_error(const std::string& msg);

    namespace
    {
        using bf16 = __nv_bfloat16;
        constexpr int kThreads = 256;
        constexpr int kStages = 4;
        constexpr int kTileM = 128;
        constexpr int kChunkK = 64; // K elements per pipeline stage
        constexpr int kStageBytesA = kTileM * kChunkK * 2; // 16 KiB

        __host__ __device__ inline uint32_t tmem_columns(int n)
        {
            uint32_t c = 32;
            while(c < uint32_t(n))
                c <<= 1;
            return c;
        }

        __device__ __forceinline__ void raise_error(int* flag, bool& abortLocal)
        {
            abortLocal = true;
            if(flag)
                atomicExch(flag, 1);
        }

        __device__ __forceinline__ uint4 pack_bf16x8(const float (&v)[8])
        {
            uint4 o;
            __nv_bfloat162 h;
            h = __floats2bfloat162_rn(v[0], v[1]);
            o.x = *reinterpret_cast<uint32_t*>(&h);
            h = __floats2bfloat162_rn(v[2], v[3]);
            o.y = *reinterpret_cast<uint32_t*>(&h);
            h = __floats2bfloat162_rn(v[4], v[5]);
            o.z = *reinterpret_cast<uint32_t*>(&h);
            h = __floats2bfloat162_rn(v[6], v[7]);
            o.w = *reinterpret_cast<uint32_t*>(&h);
            return o;
        }
        __device__ __forceinline__ void unpack_bf16x8(uint4 u, float (&v)[8])
        {
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for(int i = 0; i < 4; ++i)
            {
                v[2 * i] = __uint_as_float(w[i] << 16);
                v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
            }
        }

        // ------------------------------------------------------------------ forward / dgrad
        __global__ void __launch_bounds__(kThreads, 1) k_conv_gemm(const __grid_constant__ ConvGemmParams p)
        {
            extern __shared__ unsigned char dsm[];
            __shared__ uint32_t sTmem;
            __shared__ __align__(8) uint64_t sEmpty[kStages];
            __shared__ __align__(8) uint64_t sDone;
            unsigned char* base = dsm + ((128u - (tc::smem_addr(dsm) & 127u)) & 127u);
            const uint32_t sB = tc::smem_addr(base);
            const uint32_t sA = sB + uint32_t(p.Npad) * uint32_t(p.Kpad) * 2u;
            const int tid = threadIdx.x;
            const uint32_t cols = tmem_columns(p.Npad);
            if(tid < 32)
            {
                tc::tmem_alloc(&sTmem, cols);
                tc::tmem_relinquish();
            }
            if(tid == 0)
            {
                for(int s = 0; s < kStages; ++s)
                    tc::mbar_init(&sEmpty[s], 1);
                tc::mbar_init(&sDone, 1);
                tc::mbar_init_fence();
            }
            bool abortLocal = false, aborted = false;
            // the whole packed weight matrix, canonical K-major: core (n/8, k/8) at (n/8)*Kpad*16 + (k/8)*128
            {
                const int kb = p.Kpad / 8;
                const int pieces = p.Npad * kb;
                for(int i = tid; i < pieces; i += kThreads)
                {
                    const int n = i / kb, k8 = i - n * kb;
                    const uint32_t dst = sB + uint32_t(n >> 3) * uint32_t(p.Kpad) * 16u + uint32_t(k8) * 128u + uint32_t(n & 7) * 16u;
                    tc::cp_async16(dst, p.w + size_t(n) * p.Kpad + size_t(k8) * 8, 16);
                }
                tc::cp_async_commit();
                tc::cp_async_wait<0>();
                tc::fence_async_smem();
            }
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();
            const uint32_t tmem = sTmem;
            if(p.waitCheckNs != 0)
            {
                // failure-detection check: sDone has had no arrival, so this bounded wait
                // runs out; no copy or MMA is in flight when the TMEM is released
                if(tid == 0 && !tc::mbar_wait(&sDone, 0, p.waitCheckNs) && p.errorFlag)
                    atomicExch(p.errorFlag, 1);
                tc::fence_before_sync();
                __syncthreads();
                if(tid < 32)
                    tc::tmem_dealloc(tmem, cols);
                return;
            }

            // Output pixels go by residue class (y mod step, x mod step): an input gradient of
            // stride s reaches a pixel only through the taps of its class, so with step = s a
            // tile walks those taps alone ((ks / s)^2 on average) instead of all ks^2 with the
            // others multiplied as zeros.  Every other convolution is one class of all taps.
            const int step = p.step;
            const int m = tid & (kTileM - 1);
            const int jBase = tid >> 7;
            const uint32_t idesc = tc::idesc_bf16(kTileM, p.Npad, false, false);
            const uint32_t sboB = uint32_t(p.Kpad) * 16u;
            uint32_t G0 = 0;
            uint32_t donePhase = 0;

            for(int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x)
            {
                // the tile's class (cy, cx), its Hc x Wc grid of pixels and its taps
                int cy = 0, cx = 0, Hc = p.Ho, Wc = p.Wo, local = tile;
                for(int c = 0; c < step * step; ++c)
                {
                    cy = c / step;
                    cx = c - cy * step;
                    Hc = (p.Ho - cy + step - 1) / step;
                    Wc = (p.Wo - cx + step - 1) / step;
                    const int n = (p.B * Hc * Wc + kTileM - 1) / kTileM;
                    if(local < n)
                        break;
                    local -= n;
                }
                const int ty0 = step > 1 ? (cy + p.pad) % step : 0, tx0 = step > 1 ? (cx + p.pad) % step : 0;
                const int nty = max(0, (p.ks - ty0 + step - 1) / step), ntx = max(0, (p.ks - tx0 + step - 1) / step);
                const int kTotal = nty * ntx * p.Cg;
                const int nk = (kTotal + kChunkK - 1) / kChunkK;
                const int pc = local * kTileM + m;
                const bool valid = pc < p.B * Hc * Wc;
                int b = 0, oy = 0, ox = 0;
                if(valid)
                {
                    ox = pc % Wc;
                    const int t = pc / Wc;
                    oy = t % Hc;
                    b = t / Hc;
                    ox = cx + step * ox;
                    oy = cy + step * oy;
                }
                const int pix = (b * p.Ho + oy) * p.Wo + ox;
                // a thread's four 16-byte pieces of a chunk: tap (its place in the class's
                // list, by row and column) and channel, advanced chunk by chunk
                int pty[4], ptx[4], pch[4];
#pragma unroll
                for(int q = 0; q < 4; ++q)
                {
                    pty[q] = ptx[q] = 0;
                    pch[q] = (jBase + 2 * q) * 8;
                }
                auto load_chunk = [&](uint32_t G) {
                    const uint32_t stage = sA + (G % kStages) * uint32_t(kStageBytesA);
#pragma unroll
                    for(int q = 0; q < 4; ++q)
                    {
                        while(pch[q] >= p.Cg)
                        {
                            pch[q] -= p.Cg;
                            if(++ptx[q] == ntx)
                            {
                                ptx[q] = 0;
                                ++pty[q];
                            }
                        }
                        const bf16* src = p.x;
                        uint32_t bytes = 0;
                        if(valid && pty[q] < nty)
                        {
                            const int ty = ty0 + step * pty[q], tx = tx0 + step * ptx[q];
                            int iy, ix;
                            bool ok;
                            if(!p.transposed)
                            {
                                iy = oy * p.stride - p.pad + ty;
                                ix = ox * p.stride - p.pad + tx;
                                ok = iy >= 0 && ix >= 0 && iy < p.H && ix < p.W;
                            }
                            else
                            {
                                const int ny = oy + p.pad - ty, nx = ox + p.pad - tx;
                                ok = ny >= 0 && nx >= 0 && (ny % p.stride) == 0 && (nx % p.stride) == 0;
                                iy = ny / p.stride;
                                ix = nx / p.stride;
                                ok = ok && iy < p.H && ix < p.W;
                            }
                            if(ok)
                            {
                                src = p.x + ((size_t(b) * p.H + iy) * p.W + ix) * p.Cg + pch[q];
                                bytes = 16;
                            }
                        }
                        const int j = jBase + 2 * q;
                        const uint32_t dst = stage + uint32_t(m >> 3) * 1024u + uint32_t(j) * 128u + uint32_t(m & 7) * 16u;
                        tc::cp_async16(dst, src, bytes);
                        pch[q] += kChunkK;
                    }
                };

                for(int c = 0; c < kStages - 1; ++c)
                {
                    if(c < nk)
                    {
                        const uint32_t G = G0 + c;
                        if(G >= kStages && !tc::mbar_wait(&sEmpty[G % kStages], ((G / kStages) - 1) & 1))
                            raise_error(p.errorFlag, abortLocal);
                        load_chunk(G);
                    }
                    tc::cp_async_commit();
                }
                for(int kc = 0; kc < nk; ++kc)
                {
                    const int kn = kc + kStages - 1;
                    if(kn < nk)
                    {
                        const uint32_t G = G0 + kn;
                        if(G >= kStages && !tc::mbar_wait(&sEmpty[G % kStages], ((G / kStages) - 1) & 1))
                            raise_error(p.errorFlag, abortLocal);
                        load_chunk(G);
                    }
                    tc::cp_async_commit();
                    tc::cp_async_wait<kStages - 1>();
                    tc::fence_async_smem();
                    if(__syncthreads_or(abortLocal))
                    {
                        aborted = true;
                        break;
                    }
                    if(tid == 0)
                    {
                        tc::fence_after_sync();
                        const uint32_t G = G0 + kc;
                        const uint32_t stage = sA + (G % kStages) * uint32_t(kStageBytesA);
#pragma unroll
                        for(int j = 0; j < kChunkK / 16; ++j)
                        {
                            // this step's place among the packed weights (a class of several
                            // takes whole taps of a multiple of 16 channels)
                            int kw = kc * kChunkK + j * 16;
                            if(kw >= kTotal)
                                break;
                            if(step > 1)
                            {
                                const int t = kw / p.Cg, tr = t / ntx;
                                kw += ((ty0 + step * tr) * p.ks + tx0 + step * (t - tr * ntx) - t) * p.Cg;
                            }
                            const uint64_t ad = tc::smem_desc(stage + uint32_t(j) * 256u, 128u, 1024u);
                            const uint64_t bd = tc::smem_desc(sB + uint32_t(kw / 8) * 128u, 128u, sboB);
                            tc::mma_bf16(tmem, ad, bd, idesc, (kc | j) != 0 ? 1u : 0u);
                        }
                        tc::mma_commit(&sEmpty[G % kStages]);
                    }
                }
                tc::cp_async_wait<0>();
                if(tid == 0)
                    tc::mma_commit(&sDone);
                if(!tc::mbar_wait(&sDone, donePhase))
                    raise_error(p.errorFlag, abortLocal);
                donePhase ^= 1u;
                G0 += uint32_t(nk);
                if(__syncthreads_or(abortLocal))
                {
                    aborted = true;
                    break;
                }
                tc::fence_after_sync();

                // epilogue: thread = TMEM lane = tile row; the two warpgroups split the columns
                {
                    const int warp = tid >> 5;
                    const uint32_t lane0 = uint32_t(warp & 3) * 32u;
                    const int half = warp >> 2;
                    const int cpw = p.Npad / 2;
                    for(int c0 = half * cpw; c0 < (half + 1) * cpw; c0 += 8)
                    {
                        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                        if(nk > 0) // a class without a tap has no accumulator
                        {
                            tc::tmem_ld8(tmem + (lane0 << 16) + uint32_t(c0), v);
                            tc::tmem_wait_ld();
                        }
                        if(!valid || c0 >= p.Cout)
                            continue;
                        const size_t o = size_t(pix) * p.Cout + c0;
                        if(p.bias)
                        {
#pragma unroll
                            for(int i = 0; i < 8; ++i)
                                v[i] += __ldg(p.bias + c0 + i);
                        }
                        if(p.relu)
                        {
#pragma unroll
                            for(int i = 0; i < 8; ++i)
                                v[i] = fmaxf(v[i], 0.0f);
                        }
                        if(p.mask)
                        {
                            float mk[8];
                            unpack_bf16x8(__ldg(reinterpret_cast<const uint4*>(p.mask + o)), mk);
#pragma unroll
                            for(int i = 0; i < 8; ++i)
                                v[i] = mk[i] > 0.0f ? v[i] : 0.0f;
                        }
                        if(p.yf)
                        {
                            float4* dst = reinterpret_cast<float4*>(p.yf + o);
                            if(p.accumulate)
                            {
                                const float4 a = dst[0], bq = dst[1];
                                v[0] += a.x, v[1] += a.y, v[2] += a.z, v[3] += a.w;
                                v[4] += bq.x, v[5] += bq.y, v[6] += bq.z, v[7] += bq.w;
                            }
                            dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                            dst[1] = make_float4(v[4], v[5], v[6], v[7]);
                        }
                        else
                        {
                            uint4* dst = reinterpret_cast<uint4*>(p.y + o);
                            if(p.accumulate)
                            {
                                float a[8];
                                unpack_bf16x8(*dst, a);
#pragma unroll
                                for(int i = 0; i < 8; ++i)
                                    v[i] += a[i];
                            }
                            *dst = pack_bf16x8(v);
                        }
                    }
                }
                tc::fence_before_sync();
                __syncthreads();
            }
            // drain: every MMA this CTA issued has completed before TMEM is released
            if(aborted)
            {
                if(tid == 0)
                    tc::mma_commit(&sDone);
                tc::mbar_wait(&sDone, donePhase);
            }
            tc::fence_before_sync();
            __syncthreads();
            if(tid < 32)
                tc::tmem_dealloc(tmem, cols);
        }

        // ------------------------------------------------------------------ row tiles
        // Convolutions of stride 1 (forward, or the input gradient with `transposed`) or
        // stride 2 (forward) whose gathered channel count is a multiple of 16.  A tile is
        // 128 consecutive output pixels of one image row.  Its input rows (ks of them)
        // are loaded into shared memory once, channel chunks of 8 stored as separate
        // runs of 16-byte pixels; for stride 2 each run is split into its even and odd
        // input columns.  Every tap then reads the same halo through a descriptor whose
        // start is shifted by the tap's column offset: the no-swizzle core matrix is 8
        // consecutive 16-byte rows, and consecutive output pixels are consecutive
        // entries of a run (of a parity plane for stride 2).  Warp roles:
        //   warps 0-3  epilogue (TMEM lane = pixel), double-buffered accumulators
        //   warps 4-7  producers: cp.async of the halo, arrival on the stage's mbarrier
        //   warp 8     one thread issues the MMAs and commits them
        // With TMA the halo comes in one tiled bulk-tensor load per run (a box of 8 channels
        // x the run's pixels) issued by one thread of warp 9, and warps 4-7 join the
        // epilogue: warps 0-3 take the first half of the accumulator columns, warps 4-7 the
        // second (a warp reads TMEM lanes 32*(w%4)..+31, so both groups see every pixel).
        constexpr int kRowThreads = 288;
        template<bool TMA>
        __host__ __device__ constexpr int row_threads()
        {
            return TMA ? 320 : kRowThreads;
        }

        struct RowGeom
        {
            int S; // stride: 1 or 2
            int HWp; // entries between runs (per parity plane for stride 2)
            int HWn; // entries a run needs (<= HWp, which holds a full tile's, padded to 8 for TMA destinations)
            int stages; // halo buffers: 1 or 2
            int rowB; // swizzled staging: bytes per staged pixel (Cg * 2 = 32, 64 or 128); 0 = chunked runs
            // implicit concatenation by TMA (1x1, xUp): channel chunks of cwc (coarse) and cwf
            // (fine) channels, each staged as 128 swizzled rows; 0 = off
            int cwc, cwf;
        };

        // width: output pixels of a row (of a parity's, for stride-2 input gradients)
        inline RowGeom row_geom(int stride, int ks, int pad, int width, int stages, bool tma)
        {
            RowGeom g;
            g.S = stride;
            const int more = stride == 1 ? 2 * pad : (ks - 1) / 2 + 1;
            // a row narrower than a tile needs its own columns only; the MMA's other rows read
            // what the buffer holds, and nothing stores them
            g.HWn = (width < kTileM ? width : kTileM) + more;
            // a TMA destination starts on a 128-byte boundary: runs of a multiple of 8 entries
            g.HWp = tma ? (kTileM + more + 7) / 8 * 8 : kTileM + more;
            g.stages = stages;
            g.rowB = 0;
            g.cwc = g.cwf = 0;
            return g;
        }
        // Input gradients of stride 2 go by output parity: output row y takes the tap rows
        // ty = (y + pad) mod 2, + 2, ... at input rows (y + pad - ty) / 2, and its even and
        // odd columns x = 2u, 2u + 1 are two stride-1 convolutions in u over the same halo
        // (taps tx of their parity at input column u + (x mod 2 + pad - tx) / 2, within one
        // of u), accumulated side by side in TMEM.
        __host__ __device__ inline bool parity_tiles(const ConvGemmParams& p)
        {
            return p.transposed && p.stride == 2;
        }
        // input rows of a tile's halo, at most
        __host__ __device__ inline int halo_rows(const ConvGemmParams& p)
        {
            return parity_tiles(p) ? (p.ks + 1) / 2 : p.ks;
        }
        __host__ __device__ inline int row_tile_count(const ConvGemmParams& p)
        {
            return ((parity_tiles(p) ? (p.Wo + 1) / 2 : p.Wo) + kTileM - 1) / kTileM;
        }
        __host__ __device__ inline int accumulator_columns(const ConvGemmParams& p)
        {
            return parity_tiles(p) ? 2 * p.Npad : p.Npad;
        }
        inline RowGeom row_geom_of(const ConvGemmParams& p, int stages, bool tma)
        {
            return parity_tiles(p) ? row_geom(1, p.ks, 1, (p.Wo + 1) / 2, stages, tma) : row_geom(p.stride, p.ks, p.pad, p.Wo, stages, tma);
        }

        // 16 bytes, or zeros; issued where it stands
        __device__ __forceinline__ uint4 load_piece(const bf16* src, bool ok)
        {
            uint4 v = make_uint4(0, 0, 0, 0);
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
                : "l"(src), "r"(int(ok)));
            return v;
        }
        // 16 bytes of a tensor that this kernel also writes
        __device__ __forceinline__ uint4 load_own(const bf16* src)
        {
            uint4 v;
            asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(src) : "memory");
            return v;
        }

        // Epilogue of one 128-pixel output tile (row y of image b): this thread's column x,
        // accumulator columns [cBeg, cBeg + colsPer) of the TMEM tile at tAcc (this warp's
        // lanes), which are complete when `full` reaches `phase`; bias, ReLU, mask, then the
        // bf16 / FP32 store.  What it reads of a mask or of the tensor it adds to is loaded one
        // group of columns ahead, the first group's before the wait: with each group's loads
        // after the last one's stores a tile waited for memory once a group (the three
        // stride-2 gradients of a step of 16 128 x 128 pairs: 136 -> 92 us).
        // False when the wait ran out.
        template<bool READS>
        __device__ __forceinline__ bool row_epilogue(
            const ConvGemmParams& p,
            uint64_t* full,
            uint32_t phase,
            uint32_t tAcc,
            int x,
            int b,
            int y,
            int cBeg,
            int colsPer,
            const float* sBias)
        {
            const bool valid = x < p.Wo;
            const size_t pix = (size_t(b) * p.Ho + y) * p.Wo + x;
            const int cEnd = min(cBeg + colsPer, p.Cout);
            const bool masked = READS && valid && p.mask, added = READS && valid && p.accumulate && !p.yf;
            uint4 mk[2] = {}, ad[2] = {};
            auto fetch = [&](int c16) {
#pragma unroll
                for(int hh = 0; hh < 2; ++hh)
                {
                    const int c0 = c16 + 8 * hh;
                    if(masked && c0 < cEnd)
                        mk[hh] = load_piece(p.mask + pix * p.Cout + c0, true);
                    if(added && c0 < cEnd)
                        ad[hh] = load_own(p.y + pix * p.Cout + c0);
                }
            };
            fetch(cBeg);
            if(!tc::mbar_wait(full, phase))
                return false;
            tc::fence_after_sync();
            // 16 accumulator columns per TMEM wait (8 where a column group ends)
            for(int c16 = cBeg; c16 < cBeg + colsPer; c16 += 16)
            {
                const bool two = c16 + 16 <= cBeg + colsPer;
                float v[2][8];
                const uint32_t ta = tAcc + uint32_t(c16);
                tc::tmem_ld8(ta, v[0]);
                if(two)
                    tc::tmem_ld8(ta + 8u, v[1]);
                tc::tmem_wait_ld();
                const uint4 mkNow[2] = {mk[0], mk[1]}, adNow[2] = {ad[0], ad[1]};
                fetch(c16 + 16);
                if(!valid)
                    continue;
#pragma unroll
                for(int hh = 0; hh < 2; ++hh)
                {
                    const int c0 = c16 + 8 * hh;
                    if(c0 >= cEnd)
                        break;
                    float(&w)[8] = v[hh];
                    const size_t o = pix * p.Cout + c0;
                    if(p.bias)
                    {
#pragma unroll
                        for(int k = 0; k < 8; ++k)
                            w[k] += sBias[c0 + k];
                    }
                    if(p.relu)
                    {
#pragma unroll
                        for(int k = 0; k < 8; ++k)
                            w[k] = fmaxf(w[k], 0.0f);
                    }
                    if(READS && p.mask)
                    {
                        float m8[8];
                        unpack_bf16x8(mkNow[hh], m8);
#pragma unroll
                        for(int k = 0; k < 8; ++k)
                            w[k] = m8[k] > 0.0f ? w[k] : 0.0f;
                    }
                    if(p.yf)
                    {
                        float4* dst = reinterpret_cast<float4*>(p.yf + o);
                        if(READS && p.accumulate)
                        {
                            const float4 u = dst[0], t2 = dst[1];
                            w[0] += u.x, w[1] += u.y, w[2] += u.z, w[3] += u.w;
                            w[4] += t2.x, w[5] += t2.y, w[6] += t2.z, w[7] += t2.w;
                        }
                        dst[0] = make_float4(w[0], w[1], w[2], w[3]);
                        dst[1] = make_float4(w[4], w[5], w[6], w[7]);
                    }
                    else
                    {
                        if(READS && p.accumulate)
                        {
                            float u[8];
                            unpack_bf16x8(adNow[hh], u);
#pragma unroll
                            for(int k = 0; k < 8; ++k)
                                w[k] += u[k];
                        }
                        *reinterpret_cast<uint4*>(p.y + o) = pack_bf16x8(w);
                    }
                }
            }
            return true;
        }

        // PAR: parity_tiles.  READS: the epilogue reads a mask or the tensor it adds to.  Each is
        // compiled apart: a plain convolution keeps three blocks an SM by registers.
        template<bool TMA, bool PAR, bool READS>
        __global__ void __launch_bounds__(row_threads<TMA>(), 1)
            k_conv_row(const __grid_constant__ ConvGemmParams p, const RowGeom rg, const __grid_constant__ CUtensorMap tmap,
                       const __grid_constant__ CUtensorMap tmapUp)
        {
            extern __shared__ unsigned char dsm[];
            __shared__ uint32_t sTmem;
            __shared__ float sBias[256];
            __shared__ __align__(8) uint64_t sFull[2];
            __shared__ __align__(8) uint64_t sEmpty[2];
            __shared__ __align__(8) uint64_t sAccFull[2];
            __shared__ __align__(8) uint64_t sAccEmpty[2];
            __shared__ __align__(8) uint64_t sDrain;
            unsigned char* base = dsm + ((128u - (tc::smem_addr(dsm) & 127u)) & 127u);
            const uint32_t sB = tc::smem_addr(base);
            const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
            const int pad = p.pad, ks = p.ks, S = rg.S, HWp = rg.HWp, NS = rg.stages;
            constexpr bool par = PAR;
            const int rows = halo_rows(p), left = par ? 1 : pad; // columns of the halo before the tile's first
            const int nC = p.Cg / 8;
            const uint32_t runBytes = uint32_t(HWp) * 16u;
            // swizzled staging: each input row is HWp pixels of rowB bytes, the row buffers
            // and the halo start on multiples of the swizzle pattern's period (8 rows)
            const int rowB = rg.rowB;
            const bool cat = TMA && rg.cwc != 0;
            const uint32_t swSpan = cat ? 1024u : 8u * uint32_t(rowB);
            const uint32_t rowPitch = rowB ? (uint32_t(HWp * rowB) + swSpan - 1u) / swSpan * swSpan : 0u;
            const uint32_t haloBytes = rowB ? uint32_t(rows * S) * rowPitch : uint32_t(rows * nC * S) * runBytes;
            const uint32_t wEnd = sB + uint32_t(p.Npad) * uint32_t(p.Kpad) * 2u;
            const uint32_t sH = (rowB || cat) ? (wEnd + swSpan - 1u) / swSpan * swSpan : wEnd;
            const uint32_t half = tmem_columns(accumulator_columns(p));
            const uint32_t cols = 2 * half;
            if(warp == 0)
            {
                tc::tmem_alloc(&sTmem, cols);
                tc::tmem_relinquish();
            }
            if(tid == 0)
            {
                for(int s = 0; s < 2; ++s)
                {
                    tc::mbar_init(&sFull[s], TMA ? 1 : 128);
                    tc::mbar_init(&sEmpty[s], 1);
                    tc::mbar_init(&sAccFull[s], 1);
                    tc::mbar_init(&sAccEmpty[s], TMA ? 256 : 128);
                }
                tc::mbar_init(&sDrain, 1);
                tc::mbar_init_fence();
            }
            {
                const int kb = p.Kpad / 8;
                const int pieces = p.Npad * kb;
                for(int i = tid; i < pieces; i += row_threads<TMA>())
                {
                    const int n = i / kb, k8 = i - n * kb;
                    const uint32_t dst = sB + uint32_t(n >> 3) * uint32_t(p.Kpad) * 16u + uint32_t(k8) * 128u + uint32_t(n & 7) * 16u;
                    tc::cp_async16(dst, p.w + size_t(n) * p.Kpad + size_t(k8) * 8, 16);
                }
                tc::cp_async_commit();
                // the per-channel bias, read by every epilogue thread for every pixel
                for(int c = tid; c < p.Npad && c < 256; c += row_threads<TMA>())
                    sBias[c] = (p.bias && c < p.Cout) ? __ldg(p.bias + c) : 0.0f;
                tc::cp_async_wait<0>();
                tc::fence_async_smem();
            }
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();
            // everything above (weights, bias, barriers, TMEM) is independent of the
            // previous layer; its output is read only from here on
            tc::grid_dependency_wait();
            tc::grid_launch_dependents();
            const uint32_t tmem = sTmem;
            if(p.waitCheckNs != 0)
            {
                // failure-detection check: sDrain has had no arrival, so this bounded wait
                // runs out; no copy or MMA is in flight when the TMEM is released
                if(tid == 0 && !tc::mbar_wait(&sDrain, 0, p.waitCheckNs) && p.errorFlag)
                    atomicExch(p.errorFlag, 1);
                tc::fence_before_sync();
                __syncthreads();
                if(warp == 0)
                    tc::tmem_dealloc(tmem, cols);
                return;
            }
            const int tilesPerRow = row_tile_count(p);
            const int nTiles = p.B * p.Ho * tilesPerRow;

            if(TMA && warp == 9)
            {
                // entry (ty, chunk j, parity q, idx) holds input column S*x0 - pad + S*idx + q:
                // one box per run.  Stride 1: map (C, W, H, B), box (8, HWn, 1, 1) at
                // (8j, x0 - pad, row, b).  Stride 2: map (C, 2, W/2, H, B), the column split
                // into its parity and half, box (8, 1, HWn, 1, 1) at (8j, c & 1, c >> 1, row,
                // b) with c = 2*x0 - pad + q.  Swizzled staging (16-64 channels): one box of
                // all channels per run, (C, HWn, 1, 1) at (0, x0 - pad, row, b) or
                // (C, 1, HWn, 1, 1) at (0, c & 1, c >> 1, row, b), written with the map's
                // 32/64/128-byte swizzle.  Rows and columns outside the image read zeros.
                if(lane == 0)
                {
                    const uint32_t rowTx = rowB ? uint32_t(S * rg.HWn * rowB) : uint32_t(nC * S * rg.HWn) * 16u;
                    int i = 0;
                    for(int tile = blockIdx.x; tile < nTiles; tile += gridDim.x, ++i)
                    {
                        const int s = i % NS, n = i / NS;
                        if(n >= 1 && !tc::mbar_wait(&sEmpty[s], uint32_t(n - 1) & 1u))
                        {
                            if(p.errorFlag)
                                atomicExch(p.errorFlag, 1);
                            break;
                        }
                        const int xt = tile % tilesPerRow;
                        const int row = tile / tilesPerRow;
                        const int y = row % p.Ho, b = row / p.Ho;
                        const int x0 = xt * kTileM;
                        const uint32_t st = sH + uint32_t(s) * haloBytes;
                        const int ty0 = par ? (y + pad) & 1 : 0;
                        const int nRows = par ? (ks - ty0 + 1) / 2 : ks;
                        tc::mbar_arrive_expect_tx(&sFull[s], cat ? uint32_t(kTileM * p.Cg * 2) : uint32_t(nRows) * rowTx);
                        if(cat)
                        {
                            // tile rows in parity order: row m < 64 is pixel x0 + 2m, row 64 + m
                            // is pixel x0 + 2m + 1; both halves read coarse pixel x0/2 + m, so
                            // the coarse chunk is copied to both, the fine chunk by parity
                            uint32_t dst = st;
                            const int yc = min(y >> 1, p.upInH - 1); // the nearest coarse row, clamped
                            for(int c = 0; c < p.upC; c += rg.cwc)
                            {
                                for(int h = 0; h < 2; ++h)
                                    tc::tma_load_4d(dst + uint32_t(h * 64 * rg.cwc * 2), &tmapUp, c, x0 >> 1, yc, b, &sFull[s]);
                                dst += uint32_t(kTileM * rg.cwc * 2);
                            }
                            for(int c = 0; c < p.Cg - p.upC; c += rg.cwf)
                            {
                                for(int q = 0; q < 2; ++q)
                                    tc::tma_load_5d(dst + uint32_t(q * 64 * rg.cwf * 2), &tmap, c, q, x0 >> 1, y, b, &sFull[s]);
                                dst += uint32_t(kTileM * rg.cwf * 2);
                            }
                            continue;
                        }
                        for(int ty = 0; ty < nRows; ++ty)
                        {
                            const int iy = par ? ((y + pad - ty0) >> 1) - ty : p.transposed ? y + pad - ty : S * y - pad + ty;
                            if(rowB)
                            {
                                if(S == 1)
                                    tc::tma_load_4d(st + uint32_t(ty) * rowPitch, &tmap, 0, x0 - left, iy, b, &sFull[s]);
                                else
                                    for(int q = 0; q < 2; ++q)
                                    {
                                        const int c = 2 * x0 - pad + q;
                                        tc::tma_load_5d(st + uint32_t(ty * 2 + q) * rowPitch, &tmap, 0, c & 1, c >> 1, iy, b,
                                                        &sFull[s]);
                                    }
                                continue;
                            }
                            for(int j = 0; j < nC; ++j)
                                for(int q = 0; q < S; ++q)
                                {
                                    const uint32_t dst = st + uint32_t((ty * nC + j) * S + q) * runBytes;
                                    if(S == 1)
                                        tc::tma_load_4d(dst, &tmap, 8 * j, x0 - left, iy, b, &sFull[s]);
                                    else
                                    {
                                        const int c = 2 * x0 - pad + q;
                                        tc::tma_load_5d(dst, &tmap, 8 * j, c & 1, c >> 1, iy, b, &sFull[s]);
                                    }
                                }
                        }
                    }
                }
            }
            else if(!TMA && warp >= 4 && warp < 8)
            {
                // producers: entry (ty, chunk j, parity q, idx) holds input column S*x0 - pad + S*idx + q
                const int pt = tid - 128;
                const int dj = 128 % nC, dc = 128 / nC;
                int i = 0;
                for(int tile = blockIdx.x; tile < nTiles; tile += gridDim.x, ++i)
                {
                    const int s = i % NS, n = i / NS;
                    if(n >= 1 && !tc::mbar_wait(&sEmpty[s], uint32_t(n - 1) & 1u))
                    {
                        if(p.errorFlag)
                            atomicExch(p.errorFlag, 1);
                        break;
                    }
                    const int xt = tile % tilesPerRow;
                    const int row = tile / tilesPerRow;
                    const int y = row % p.Ho, b = row / p.Ho;
                    const int x0 = xt * kTileM;
                    const uint32_t st = sH + uint32_t(s) * haloBytes;
                    // flat index g = (c * nC + j) within one halo row, c = S*idx + q the input column
                    // offset; consecutive threads take consecutive 16-byte pieces of global memory and
                    // step by 128 pieces, so j and c advance by fixed amounts
                    const int perRow = nC * S * HWp;
                    const int ty0 = par ? (y + pad) & 1 : 0;
                    const int nRows = par ? (ks - ty0 + 1) / 2 : ks;
                    for(int ty = 0; ty < nRows; ++ty)
                    {
                        const int iy = par ? ((y + pad - ty0) >> 1) - ty : p.transposed ? y + pad - ty : S * y - pad + ty;
                        const bool rowOk = iy >= 0 && iy < p.H;
                        // implicit concatenation: chunks below nUp come from the coarse tensor at
                        // the nearest coarse pixel, the rest from x, whose pixels hold cX channels
                        const int nUp = p.xUp ? p.upC / 8 : 0;
                        const int cX = p.Cg - 8 * nUp;
                        const bf16* rowPtr = p.x + (size_t(b) * p.H + (rowOk ? iy : 0)) * p.W * cX;
                        const bf16* upRow = p.xUp
                            ? p.xUp + (size_t(b) * p.upInH + min((rowOk ? iy : 0) >> 1, p.upInH - 1)) * p.upInW * p.upC
                            : nullptr;
                        const uint32_t rowBase = st + uint32_t(ty * nC * S) * runBytes;
                        int j = pt % nC, c = pt / nC;
                        for(int g = pt; g < perRow; g += 128)
                        {
                            const int ix = S * x0 - left + c;
                            const int q = c & (S - 1), idx = S == 1 ? c : (c >> 1);
                            const bool ok = rowOk && ix >= 0 && ix < p.W;
                            const bf16* src = !ok ? p.x
                                : j < nUp ? upRow + size_t(min(ix >> 1, p.upInW - 1)) * p.upC + j * 8
                                          : rowPtr + size_t(ix) * cX + (j - nUp) * 8;
                            tc::cp_async16(rowBase + uint32_t(j * S + q) * runBytes + uint32_t(idx) * 16u, src, ok ? 16u : 0u);
                            j += dj;
                            c += dc;
                            if(j >= nC)
                            {
                                j -= nC;
                                ++c;
                            }
                        }
                    }
                    tc::cp_async_arrive(&sFull[s]);
                }
                tc::cp_async_wait<0>();
            }
            else if(warp == 8)
            {
                if(lane == 0)
                {
                    const uint32_t idesc = tc::idesc_bf16(kTileM, p.Npad, false, false);
                    const uint32_t lboA = uint32_t(S) * runBytes;
                    const uint32_t sboB = uint32_t(p.Kpad) * 16u;
                    int i = 0;
                    for(int tile = blockIdx.x; tile < nTiles; tile += gridDim.x, ++i)
                    {
                        const int s = i % NS, n = i / NS;
                        const int a = i & 1, na = i >> 1;
                        if(!tc::mbar_wait(&sFull[s], uint32_t(n) & 1u)
                           || (na >= 1 && !tc::mbar_wait(&sAccEmpty[a], uint32_t(na - 1) & 1u)))
                        {
                            if(p.errorFlag)
                                atomicExch(p.errorFlag, 1);
                            break;
                        }
                        tc::fence_async_smem();
                        tc::fence_after_sync();
                        const uint32_t st = sH + uint32_t(s) * haloBytes;
                        const uint32_t dTile = tmem + uint32_t(a) * half;
                        const int y = (tile / tilesPerRow) % p.Ho;
                        const int ty0 = par ? (y + pad) & 1 : 0, nRows = par ? (ks - ty0 + 1) / 2 : ks;
                        const int nPar = par ? 2 : 1, tapStep = nPar;
                        // descriptors differ only in their start field (16-byte units), so the
                        // loop adds offsets to two base descriptors
                        const uint64_t aBase = tc::smem_desc(st, lboA, 128u);
                        const uint64_t bBase = tc::smem_desc(sB, 128u, sboB);
                        uint32_t acc = 0;
                        if(cat)
                        {
                            // the chunks in channel order (coarse, then fine), each 128 rows of
                            // cw * 2 bytes with that width's swizzle
                            uint32_t region = st, bOff = 0;
                            for(int part = 0; part < 2; ++part)
                            {
                                const int cw = part == 0 ? rg.cwc : rg.cwf;
                                const int cN = part == 0 ? p.upC : p.Cg - p.upC;
                                const uint32_t rb = uint32_t(cw * 2);
                                const uint64_t swDesc = (tc::smem_desc(0, 16u, 8u * rb) & ~uint64_t(0x3FFF))
                                    | (uint64_t(rb == 32 ? 6 : rb == 64 ? 4 : 2) << 61);
                                for(int c = 0; c < cN; c += cw)
                                {
                                    for(int jp = 0; jp < cw / 16; ++jp)
                                    {
                                        const uint32_t addr = region + uint32_t(jp) * 32u;
                                        tc::mma_bf16(dTile, swDesc | uint64_t((addr >> 4) & 0x3FFFu), bBase + bOff, idesc, acc);
                                        acc = 1;
                                        bOff += 16u;
                                    }
                                    region += uint32_t(kTileM) * rb;
                                }
                            }
                        }
                        else if(rowB)
                        {
                            // K-major A with the rows' own swizzle (layout 6 / 4 / 2 = 32 / 64 /
                            // 128 bytes), 8-row groups swSpan apart; tap (ty, tx) starts idx0 rows
                            // into run (ty, q) and each K step of 16 channels 32 bytes further.
                            // The swizzle follows the absolute shared-memory address, as the TMA
                            // copy wrote it, so the base-offset field stays 0.
                            const uint64_t swDesc = (tc::smem_desc(0, 16u, swSpan) & ~uint64_t(0x3FFF))
                                | (uint64_t(rowB == 32 ? 6 : rowB == 64 ? 4 : 2) << 61);
                            for(int cx = 0; cx < nPar; ++cx, acc = 0)
                                for(int ty = 0; ty < nRows; ++ty)
                                    for(int tx = par ? (cx + pad) & 1 : 0; tx < ks; tx += tapStep)
                                    {
                                        const int col = par ? ((cx + pad - tx) >> 1) + 1 : p.transposed ? 2 * pad - tx : tx;
                                        const int q = col & (S - 1), idx0 = S == 1 ? col : (col >> 1);
                                        const uint32_t d = dTile + uint32_t(cx * p.Npad);
                                        uint32_t addr = st + uint32_t(ty * S + q) * rowPitch + uint32_t(idx0 * rowB);
                                        uint32_t bOff = uint32_t(((ty0 + tapStep * ty) * ks + tx) * p.Cg);
                                        for(int jp = 0; jp < nC / 2; ++jp)
                                        {
                                            tc::mma_bf16(d, swDesc | uint64_t((addr >> 4) & 0x3FFFu), bBase + bOff, idesc, acc);
                                            acc = 1;
                                            addr += 32u;
                                            bOff += 16u;
                                        }
                                    }
                        }
                        else
                            for(int cx = 0; cx < nPar; ++cx, acc = 0)
                                for(int ty = 0; ty < nRows; ++ty)
                                    for(int tx = par ? (cx + pad) & 1 : 0; tx < ks; tx += tapStep)
                                    {
                                        const int col = par ? ((cx + pad - tx) >> 1) + 1 : p.transposed ? 2 * pad - tx : tx;
                                        const int q = col & (S - 1), idx0 = S == 1 ? col : (col >> 1);
                                        const uint32_t d = dTile + uint32_t(cx * p.Npad);
                                        uint32_t aOff = uint32_t((ty * nC * S + q) * HWp + idx0);
                                        uint32_t bOff = uint32_t(((ty0 + tapStep * ty) * ks + tx) * p.Cg);
                                        for(int jp = 0; jp < nC / 2; ++jp)
                                        {
                                            tc::mma_bf16(d, aBase + aOff, bBase + bOff, idesc, acc);
                                            acc = 1;
                                            aOff += uint32_t(2 * S * HWp);
                                            bOff += 16u;
                                        }
                                    }
                        tc::mma_commit(&sEmpty[s]);
                        tc::mma_commit(&sAccFull[a]);
                    }
                    // every MMA of this CTA has completed before TMEM is released
                    tc::mma_commit(&sDrain);
                    tc::mbar_wait(&sDrain, 0);
                }
                __syncwarp();
            }
            else
            {
                // epilogue: thread = TMEM lane = pixel of the tile; with TMA two groups of four
                // warps split the accumulator columns
                const uint32_t lane0 = uint32_t(warp & 3) * 32u;
                const int group = TMA ? warp >> 2 : 0;
                const int colsPer = TMA && !par ? p.Npad / 2 : p.Npad; // a multiple of 8
                const int cBeg = group * colsPer;
                int i = 0;
                for(int tile = blockIdx.x; tile < nTiles; tile += gridDim.x, ++i)
                {
                    const int a = i & 1;
                    const int xt = tile % tilesPerRow;
                    const int row = tile / tilesPerRow;
                    const int m = tid & 127;
                    const int px = cat ? (m < 64 ? 2 * m : 2 * (m - 64) + 1) : m; // parity-ordered rows
                    const uint32_t tAcc = tmem + uint32_t(a) * half + (lane0 << 16), phase = uint32_t(i >> 1) & 1u;
                    bool ok = true;
                    if(par) // a parity's columns each, with TMA a group of warps each
                        for(int cx = group; cx < 2; cx += TMA ? 2 : 1)
                            ok = ok && row_epilogue<READS>(p, &sAccFull[a], phase, tAcc + uint32_t(cx * p.Npad), 2 * (xt * kTileM + px) + cx,
                                                    row / p.Ho, row % p.Ho, 0, p.Npad, sBias);
                    else
                        ok = row_epilogue<READS>(p, &sAccFull[a], phase, tAcc, xt * kTileM + px, row / p.Ho, row % p.Ho, cBeg, colsPer, sBias);
                    if(!ok)
                    {
                        if(p.errorFlag)
                            atomicExch(p.errorFlag, 1);
                        break;
                    }
                    tc::fence_before_sync();
                    tc::mbar_arrive(&sAccEmpty[a]);
                }
            }
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();
            if(warp == 0)
                tc::tmem_dealloc(tmem, cols);
        }

        constexpr int kWgradStages = 2;
        // bytes from one 8-channel block of 64 pixels to the next: 32 more than the block, so
        // that the 8 lanes of a 16-byte store phase (2 pixels x 4 blocks) meet all banks
        constexpr uint32_t kBlockPitch = kChunkK * 16 + 32;

        __device__ __forceinline__ void store_piece(uint32_t at, uint4 v)
        {
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
        }

        // ------------------------------------------------------------------ weight gradient
        // All layers of a network in one launch: their CTAs fill the device together, and there
        // is one tail instead of one per layer (a step of 16 128 x 128 pairs: eleven launches of
        // 14-55 us, 362 us together, to one of 329 us).  What bounds a CTA is bringing the tiles to
        // shared memory, pixels' channels into 8-channel blocks: cp.async writes each 16-byte
        // piece of its own line in its own shared-memory cycle (30 a request, half of the time),
        // so a thread loads its pieces of the next chunk into registers while the MMAs of this
        // one run, and stores them 8 lanes a cycle: 329 -> 213 us; addresses as 32-bit piece
        // counts from the pixel's: 177 us.  Three CTAs an SM (two 3533, three 3374, four, with
        // 62 registers, 3430 us per four steps), twelve an SM in all (three 3410, six 3374,
        // twelve 3359 us): the layers' CTAs differ in cost and the last ones stay short.
        template<int NB>
        __global__ void __launch_bounds__(kThreads, NB == 4 ? 3 : 2) k_conv_wgrad(const __grid_constant__ WgradTable T)
        {
            extern __shared__ unsigned char dsm[];
            __shared__ uint32_t sTmem;
            __shared__ __align__(8) uint64_t sEmpty[kWgradStages];
            __shared__ __align__(8) uint64_t sDone;
            int layer = 0;
            while(int(blockIdx.x) >= T.first[layer + 1])
                ++layer;
            const WgradParams& p = T.layer[layer];
            const int local = int(blockIdx.x) - T.first[layer];
            constexpr uint32_t stages = kWgradStages;
            unsigned char* base = dsm + ((128u - (tc::smem_addr(dsm) & 127u)) & 127u);
            const uint32_t stageBytes = (16u + uint32_t(p.Npad) / 8u) * kBlockPitch;
            const uint32_t s0 = tc::smem_addr(base);
            const int tid = threadIdx.x;
            const uint32_t cols = tmem_columns(p.Npad);
            if(tid < 32)
            {
                tc::tmem_alloc(&sTmem, cols);
                tc::tmem_relinquish();
            }
            if(tid == 0)
            {
                for(int s = 0; s < kWgradStages; ++s)
                    tc::mbar_init(&sEmpty[s], 1);
                tc::mbar_init(&sDone, 1);
                tc::mbar_init_fence();
            }
            bool abortLocal = false, aborted = false;
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();
            const uint32_t tmem = sTmem;

            const int P = p.B * p.Ho * p.Wo;
            const int nChunks = (P + kChunkK - 1) / kChunkK;
            const int split = local / p.mTiles;
            const int c0 = split * p.chunksPerSplit;
            const int c1 = min(nChunks, c0 + p.chunksPerSplit);
            const int nk = c1 - c0;
            const int mTile = local - split * p.mTiles;
            const uint32_t idesc = tc::idesc_bf16(kTileM, p.Npad, true, true);

            // A thread carries, for pixel px of every chunk, the row blocks (8 channels of one
            // tap) mb0 + 4 q and the column blocks mb0 + 4 i of dY.  The chunks are taken in
            // order, so the pixel's place in the image and the blocks' taps need no division
            // inside the loop.
            const int px = tid >> 2, mb0 = tid & 3;
            // Addresses in 16-byte pieces: a tensor's fit 32 bits (2^26 pixels of at most 28).
            const int cX = (p.Cin - p.upC) / 8, cD = p.Cout / 8, cU = p.upC / 8;
            int ty[4], tx[4];
            int inUp = 0; // bit q: row block q is of the coarse tensor
            uint32_t delta[4]; // the tap's and channel's pieces from the pixel's first
#pragma unroll
            for(int q = 0; q < 4; ++q)
            {
                const int r0 = mTile * kTileM + (mb0 + 4 * q) * 8;
                const int t = r0 / p.Cin, ch = (r0 - t * p.Cin) / 8;
                ty[q] = r0 < p.Mtot ? t / p.ks - p.pad : 1 << 30; // past the last row: outside always (H < 2^28)
                tx[q] = t % p.ks - p.pad;
                // of the coarse tensor (1x1 layers: the tap is the pixel) or of x
                inUp |= int(ch < cU) << q;
                delta[q] = ch < cU ? uint32_t(ch) : (uint32_t(ty[q]) * uint32_t(p.W) + uint32_t(tx[q])) * uint32_t(cX) + uint32_t(ch - cU);
            }
            const bool up = cU > 0;
            int pix = c0 * kChunkK + px;
            int ox = pix % p.Wo, oy = (pix / p.Wo) % p.Ho, b = pix / p.Wo / p.Ho;
            uint4 ra[4], rb[NB];
            auto fetch = [&]() {
                const int x0 = ox * p.stride, y0 = pix < P ? oy * p.stride : -(1 << 20); // past the last pixel: no row
                const uint32_t at = (uint32_t(b * p.H + y0) * uint32_t(p.W) + uint32_t(x0)) * uint32_t(cX);
                uint32_t atUp = 0;
                if(up) // nearest coarse pixel
                    atUp = (uint32_t(b * p.upInH + min(y0 >> 1, p.upInH - 1)) * uint32_t(p.upInW)
                            + uint32_t(min(x0 >> 1, p.upInW - 1))) * uint32_t(cU);
#pragma unroll
                for(int q = 0; q < 4; ++q)
                {
                    const bool ok = uint32_t(y0 + ty[q]) < uint32_t(p.H) && uint32_t(x0 + tx[q]) < uint32_t(p.W);
                    const bool coarse = inUp >> q & 1;
                    ra[q] = load_piece((coarse ? p.xUp : p.x) + size_t((coarse ? atUp : at) + delta[q]) * 8, ok);
                }
                // B: Npad/8 column blocks x 64 pixels of dY
#pragma unroll
                for(int i = 0; i < NB; ++i)
                {
                    const int nb = mb0 + 4 * i;
                    rb[i] = load_piece(p.dy + (size_t(uint32_t(pix) * uint32_t(cD)) + nb) * 8, pix < P && nb < cD);
                }
                pix += kChunkK;
                ox += kChunkK;
                while(ox >= p.Wo)
                {
                    ox -= p.Wo;
                    if(++oy == p.Ho)
                    {
                        oy = 0;
                        ++b;
                    }
                }
            };

            const uint32_t at = uint32_t(mb0) * kBlockPitch + uint32_t(px) * 16u;
            if(nk > 0)
                fetch();
            for(int kc = 0; kc < nk; ++kc)
            {
                const uint32_t G = uint32_t(kc);
                if(G >= stages && !tc::mbar_wait(&sEmpty[G % stages], ((G / stages) - 1) & 1))
                    raise_error(p.errorFlag, abortLocal);
                const uint32_t st = s0 + (G % stages) * stageBytes + at;
#pragma unroll
                for(int q = 0; q < 4; ++q)
                    store_piece(st + uint32_t(4 * q) * kBlockPitch, ra[q]);
#pragma unroll
                for(int i = 0; i < NB; ++i)
                    if(mb0 + 4 * i < p.Npad / 8)
                        store_piece(st + uint32_t(16 + 4 * i) * kBlockPitch, rb[i]);
                tc::fence_async_smem();
                if(kc + 1 < nk) // in flight over the barrier and the next wait
                    fetch();
                if(__syncthreads_or(abortLocal))
                {
                    aborted = true;
                    break;
                }
                if(tid == 0)
                {
                    tc::fence_after_sync();
                    const uint32_t stA = s0 + (uint32_t(kc) % stages) * stageBytes;
                    const uint32_t stB = stA + 16u * kBlockPitch;
#pragma unroll
                    for(int j = 0; j < kChunkK / 16; ++j)
                    {
                        const uint64_t ad = tc::smem_desc(stA + uint32_t(j) * 256u, 128u, kBlockPitch);
                        const uint64_t bd = tc::smem_desc(stB + uint32_t(j) * 256u, 128u, kBlockPitch);
                        tc::mma_bf16(tmem, ad, bd, idesc, (kc | j) != 0 ? 1u : 0u);
                    }
                    tc::mma_commit(&sEmpty[uint32_t(kc) % stages]);
                }
            }
            if(tid == 0)
                tc::mma_commit(&sDone);
            if(!aborted && !tc::mbar_wait(&sDone, 0))
                raise_error(p.errorFlag, abortLocal);
            aborted = __syncthreads_or(abortLocal) != 0;
            tc::fence_after_sync();
            if(aborted)
            {
                // one more bounded wait: the MMAs must be done before TMEM is released
                if(tid == 0)
                    tc::mma_commit(&sDone);
                tc::mbar_wait(&sDone, 1);
            }
            else if(nk > 0)
            {
                const int warp = tid >> 5;
                const uint32_t lane0 = uint32_t(warp & 3) * 32u;
                const int half = warp >> 2;
                const int cpw = p.Npad / 2;
                const int row = mTile * kTileM + (tid & (kTileM - 1));
                const bool vec4 = (reinterpret_cast<uintptr_t>(p.dw) & 15u) == 0; // rows are multiples of 16 floats
                for(int cc = half * cpw; cc < (half + 1) * cpw; cc += 8)
                {
                    float v[8];
                    tc::tmem_ld8(tmem + (lane0 << 16) + uint32_t(cc), v);
                    tc::tmem_wait_ld();
                    if(row >= p.Mtot)
                        continue;
                    if(cc >= p.Cout) // channel counts are multiples of 8
                        continue;
                    float* dst = p.dw + size_t(row) * p.Npad + cc;
                    if(vec4)
                    {
                        atomicAdd(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
                        atomicAdd(reinterpret_cast<float4*>(dst) + 1, make_float4(v[4], v[5], v[6], v[7]));
                    }
                    else
#pragma unroll
                        for(int i = 0; i < 8; ++i)
                            atomicAdd(dst + i, v[i]);
                }
            }
            tc::fence_before_sync();
            __syncthreads();
            if(tid < 32)
                tc::tmem_dealloc(tmem, cols);
        }

        int num_sms()
        {
            static int n = 0;
            if(n == 0)
            {
                int dev = 0;
                cudaGetDevice(&dev);
                cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
                if(n <= 0)
                    n = 148;
            }
            return n;
        }
    } // namespace

    size_t conv_gemm_smem(int Npad, int Kpad)
    {
        return size_t(Npad) * Kpad * 2 + size_t(kStages) * kStageBytesA + 128;
    }
    bool row_tiles_apply(const ConvGemmParams& p)
    {
        if(p.xUp && (p.ks != 1 || p.stride != 1 || p.upC % 8 != 0 || p.transposed))
            return false;
        return p.Cg % 16 == 0 && p.Npad <= 256
            && ((p.stride == 1 && 2 * p.pad == p.ks - 1) || (p.stride == 2 && !p.transposed && p.ks <= 3 && p.pad <= 1)
                // both parities' accumulators, twice, fill 512 TMEM columns at 128; of one tap
                // a parity would have none; and a narrow row leaves most of a tile's pixels
                // unused: a 2x2 gradient of 32 columns took 27 us here and 22 us by residue
                // classes (k_conv_gemm), a 3x3 of 64 columns 36 and 67 us, of 128 columns 29
                // and 90 us
                || (parity_tiles(p) && p.Npad <= 128 && (p.ks == 2 || p.ks == 3) && p.pad <= 1 && p.Wo >= 64));
    }
    // Swizzled staging for the TMA producer: 16, 32 or 64 channels, each run (an input row,
    // or one parity plane of it at stride 2) one box of Cg * 2-byte pixels, instead of one
    // box per 8-channel chunk (the narrow chunk boxes kept the copy engine busy).  Returns
    // the bytes per staged pixel, 0 where the chunked runs are used.
    inline int swizzle_row_bytes(const ConvGemmParams& p)
    {
        return (p.Cg == 16 || p.Cg == 32 || p.Cg == 64) ? p.Cg * 2 : 0;
    }
    size_t conv_row_smem(const ConvGemmParams& p, int stages, bool tma = false)
    {
        const RowGeom g = row_geom_of(p, stages, tma);
        const int rowB = tma ? swizzle_row_bytes(p) : 0;
        if(rowB)
        {
            const size_t span = size_t(8) * rowB, pitch = (size_t(g.HWp) * rowB + span - 1) / span * span;
            return size_t(p.Npad) * p.Kpad * 2 + span + size_t(stages) * halo_rows(p) * g.S * pitch + 128;
        }
        return size_t(p.Npad) * p.Kpad * 2 + size_t(stages) * halo_rows(p) * (p.Cg / 8) * g.S * g.HWp * 16 + 128;
    }

    namespace
    {
        PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
        {
            static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
            static bool tried = false;
            if(!tried)
            {
                tried = true;
                void* f = nullptr;
                cudaDriverEntryPointQueryResult q{};
                if(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess
                   && q == cudaDriverEntryPointSuccess)
                    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
            }
            return fn;
        }

        // The tensor map of a row-tile convolution's input for the TMA producer (layouts at
        // k_conv_row); false when the input does not fit one (then the cp.async producer runs)
        bool encode_row_map(const ConvGemmParams& p, const RowGeom& g, CUtensorMap& m)
        {
            auto enc = tensor_map_encoder();
            if(!enc || (reinterpret_cast<uintptr_t>(p.x) & 15u) != 0 || p.Cg % 8 != 0)
                return false;
            const cuuint64_t C = cuuint64_t(p.Cg), W = cuuint64_t(p.W), H = cuuint64_t(p.H), B = cuuint64_t(p.B);
            cuuint32_t estr[5] = {1, 1, 1, 1, 1};
            CUresult r;
            if(g.rowB)
            {
                const CUtensorMapSwizzle sw = g.rowB == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                    : g.rowB == 64                         ? CU_TENSOR_MAP_SWIZZLE_64B
                                                           : CU_TENSOR_MAP_SWIZZLE_128B;
                if(g.S == 1)
                {
                    cuuint64_t dims[4] = {C, W, H, B};
                    cuuint64_t strides[3] = {C * 2, W * C * 2, H * W * C * 2};
                    cuuint32_t box[4] = {cuuint32_t(C), cuuint32_t(g.HWn), 1, 1};
                    r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(p.x), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
                }
                else
                {
                    if(p.W % 2 != 0)
                        return false; // the parity split views W as (W/2, 2)
                    cuuint64_t dims[5] = {C, 2, W / 2, H, B};
                    cuuint64_t strides[4] = {C * 2, 2 * C * 2, W * C * 2, H * W * C * 2};
                    cuuint32_t box[5] = {cuuint32_t(C), 1, cuuint32_t(g.HWn), 1, 1};
                    r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(p.x), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
                }
            }
            else if(g.S == 1)
            {
                cuuint64_t dims[4] = {C, W, H, B};
                cuuint64_t strides[3] = {C * 2, W * C * 2, H * W * C * 2};
                cuuint32_t box[4] = {8, cuuint32_t(g.HWn), 1, 1};
                r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(p.x), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            }
            else
            {
                if(p.W % 2 != 0)
                    return false; // the parity split views W as (W/2, 2)
                cuuint64_t dims[5] = {C, 2, W / 2, H, B};
                cuuint64_t strides[4] = {C * 2, 2 * C * 2, W * C * 2, H * W * C * 2};
                cuuint32_t box[5] = {8, 1, cuuint32_t(g.HWn), 1, 1};
                r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(p.x), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            }
            return r == CUDA_SUCCESS;
        }

        inline int chunk_width(int c)
        {
            return c % 64 == 0 ? 64 : c % 32 == 0 ? 32 : c % 16 == 0 ? 16 : 0;
        }
        inline CUtensorMapSwizzle swizzle_of(int rowBytes)
        {
            return rowBytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : rowBytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
        }

        // The two tensor maps of the implicit concatenation by TMA (layout at k_conv_row):
        // the fine tensor split by column parity, the coarse one plain; false when the layer
        // does not fit (then the cp.async producer gathers it)
        bool encode_cat_maps(const ConvGemmParams& p, RowGeom& g, CUtensorMap& fine, CUtensorMap& coarse)
        {
            auto enc = tensor_map_encoder();
            const int cf = p.Cg - p.upC;
            // columns past the coarse width would read zeros where the gather clamps, so the
            // coarse width must cover W / 2; rows are clamped in the kernel
            if(!enc || !p.xUp || p.ks != 1 || p.stride != 1 || p.pad != 0 || p.transposed || p.W % 2 != 0 || p.Wo != p.W
               || p.Ho != p.H || 2 * p.upInW < p.W || p.upInH < 1 || p.upC <= 0 || cf <= 0 || !chunk_width(p.upC)
               || !chunk_width(cf) || (reinterpret_cast<uintptr_t>(p.x) & 15u) != 0
               || (reinterpret_cast<uintptr_t>(p.xUp) & 15u) != 0)
                return false;
            g.cwc = chunk_width(p.upC);
            g.cwf = chunk_width(cf);
            cuuint32_t estr[5] = {1, 1, 1, 1, 1};
            const cuuint64_t C = cuuint64_t(cf), W = cuuint64_t(p.W), H = cuuint64_t(p.H), B = cuuint64_t(p.B);
            cuuint64_t dims[5] = {C, 2, W / 2, H, B};
            cuuint64_t strides[4] = {C * 2, 2 * C * 2, W * C * 2, H * W * C * 2};
            cuuint32_t box[5] = {cuuint32_t(g.cwf), 1, 64, 1, 1};
            if(enc(&fine, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(p.x), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_of(2 * g.cwf), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
               != CUDA_SUCCESS)
                return false;
            const cuuint64_t Cc = cuuint64_t(p.upC), Wc = cuuint64_t(p.upInW), Hc = cuuint64_t(p.upInH);
            cuuint64_t dimsC[4] = {Cc, Wc, Hc, B};
            cuuint64_t stridesC[3] = {Cc * 2, Wc * Cc * 2, Hc * Wc * Cc * 2};
            cuuint32_t boxC[4] = {cuuint32_t(g.cwc), 64, 1, 1};
            return enc(&coarse, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(p.xUp), dimsC, stridesC, boxC, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_of(2 * g.cwc), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                == CUDA_SUCCESS;
        }

        template<bool TMA, bool PAR, bool READS>
        void launch_row_as(const ConvGemmParams& p, int stages, const CUtensorMap& m, cudaStream_t s, int rowB,
                           const CUtensorMap* m2, int cwc, int cwf)
        {
            const size_t smem = conv_row_smem(p, stages, TMA) + (cwc ? 1024 : 0);
            cudaFuncSetAttribute(k_conv_row<TMA, PAR, READS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            cudaFuncSetAttribute(k_conv_row<TMA, PAR, READS>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
            const int tiles = p.B * p.Ho * row_tile_count(p);
            int perSm = ctas_per_sm(k_conv_row<TMA, PAR, READS>, row_threads<TMA>(), smem);
            while(perSm > 1 && perSm * 2 * int(tmem_columns(accumulator_columns(p))) > 512)
                --perSm;
            const int slots = num_sms() * perSm;
            RowGeom g = row_geom_of(p, stages, TMA);
            g.rowB = TMA ? rowB : 0;
            g.cwc = TMA ? cwc : 0;
            g.cwf = TMA ? cwf : 0;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(unsigned(tiles < slots ? tiles : slots));
            cfg.blockDim = dim3(unsigned(row_threads<TMA>()));
            cfg.dynamicSmemBytes = smem;
            cfg.stream = s;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = p.pdl ? 1 : 0;
            cudaLaunchKernelEx(&cfg, k_conv_row<TMA, PAR, READS>, p, g, m, m2 ? *m2 : m);
        }
        template<bool TMA>
        void launch_row(const ConvGemmParams& p, int stages, const CUtensorMap& m, cudaStream_t s, int rowB = 0,
                        const CUtensorMap* m2 = nullptr, int cwc = 0, int cwf = 0)
        {
            if(parity_tiles(p))
                launch_row_as<TMA, true, true>(p, stages, m, s, rowB, m2, cwc, cwf);
            else if(p.mask || p.accumulate)
                launch_row_as<TMA, false, true>(p, stages, m, s, rowB, m2, cwc, cwf);
            else
                launch_row_as<TMA, false, false>(p, stages, m, s, rowB, m2, cwc, cwf);
        }
    } // namespace

    bool g_rowTma = true; // the TMA producer where the input allows it
    bool launch_conv_gemm(ConvGemmParams p, cudaStream_t s)
    {
        if(row_tiles_apply(p))
        {
            int stages = 2;
            if(conv_row_smem(p, 2, true) > 227 * 1024)
                stages = 1;
            if(conv_row_smem(p, stages, true) <= 227 * 1024)
            {
                CUtensorMap m{};
                RowGeom g = row_geom_of(p, stages, true);
                g.rowB = swizzle_row_bytes(p);
                CUtensorMap m2{};
                if(g_rowTma && p.xUp && conv_row_smem(p, stages, true) + 1024 <= 227 * 1024 && encode_cat_maps(p, g, m, m2))
                    launch_row<true>(p, stages, m, s, 0, &m2, g.cwc, g.cwf);
                else if(g_rowTma && !p.xUp && encode_row_map(p, g, m))
                    launch_row<true>(p, stages, m, s, g.rowB);
                else
                    launch_row<false>(p, stages, m, s);
                return true;
            }
        }
        // k_conv_gemm knows no second input: it would read x as if that held all Cg channels
        const size_t smem = conv_gemm_smem(p.Npad, p.Kpad);
        if(smem > 227 * 1024 || p.xUp)
            return false;
        cudaFuncSetAttribute(k_conv_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        cudaFuncSetAttribute(k_conv_gemm, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        // output pixels by residue class: whole taps of 16-channel steps only, so that an MMA
        // step never crosses from one tap to the next of its class
        p.step = p.transposed && p.Cg % 16 == 0 ? p.stride : 1;
        p.tiles = 0;
        for(int c = 0; c < p.step * p.step; ++c)
        {
            const int hc = (p.Ho - c / p.step + p.step - 1) / p.step, wc = (p.Wo - c % p.step + p.step - 1) / p.step;
            p.tiles += (p.B * hc * wc + kTileM - 1) / kTileM;
        }
        const int tiles = p.tiles;
        // as many persistent CTAs as fit on an SM (shared memory and TMEM permitting), so one
        // CTA's epilogue and gathers overlap another's MMAs
        int perSm = ctas_per_sm(k_conv_gemm, kThreads, smem);
        while(perSm > 1 && perSm * int(tmem_columns(p.Npad)) > 512)
            --perSm;
        const int slots = num_sms() * perSm;
        const int grid = tiles < slots ? tiles : slots;
        k_conv_gemm<<<grid, kThreads, smem, s>>>(p);
        return true;
    }

    namespace
    {
        template<int NB>
        void launch_wgrad(const WgradTable& T, int grid, size_t smem, cudaStream_t s)
        {
            cudaFuncSetAttribute(k_conv_wgrad<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            cudaFuncSetAttribute(k_conv_wgrad<NB>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
            k_conv_wgrad<NB><<<grid, kThreads, smem, s>>>(T);
        }
    } // namespace

    bool launch_conv_wgrad(const WgradParams* layers, int n, cudaStream_t s)
    {
        if(n < 1 || n > kWgradLayers)
            return false;
        WgradTable T{};
        size_t smem = 0, work = 0;
        int npad = 0;
        for(int l = 0; l < n; ++l)
        {
            WgradParams& p = T.layer[l];
            p = layers[l];
            p.mTiles = (p.Mtot + kTileM - 1) / kTileM;
            npad = std::max(npad, p.Npad);
            work += size_t(p.mTiles) * ((size_t(p.B) * p.Ho * p.Wo + kChunkK - 1) / kChunkK);
        }
        if(npad > 256)
            return false;
        smem = size_t(kWgradStages) * (16 + npad / 8) * kBlockPitch + 128;
        // beyond 128 columns a CTA holds 256 TMEM columns: no more than two on an SM
        if(npad > 128)
            smem = std::max(smem, size_t(80) * 1024);
        // three CTAs fit on an SM; about four such waves of equal work, at least 4 chunks each
        const size_t ctas = size_t(12) * num_sms();
        const int per = std::max(4, int((work + ctas - 1) / ctas));
        for(int l = 0; l < n; ++l)
        {
            WgradParams& p = T.layer[l];
            const int chunks = (p.B * p.Ho * p.Wo + kChunkK - 1) / kChunkK;
            p.chunksPerSplit = per;
            T.first[l + 1] = T.first[l] + p.mTiles * ((chunks + per - 1) / per);
        }
        for(int l = n; l < kWgradLayers; ++l)
            T.first[l + 1] = T.first[n];
        if(npad > 128)
            launch_wgrad<8>(T, T.first[n], smem, s);
        else
            launch_wgrad<4>(T, T.first[n], smem, s);
        return true;
    }
} // namespace isaacb

using namespace isaacb;

namespace
{
    int round_up(int v, int m)
    {
        return (v + m - 1) / m * m;
    }

    isaacb_status check_conv(const isaacb_conv_args* a, bool wgrad)
    {
        if(!a)
            return ISAACB_INVALID_ARG;
        if(a->batch == 0 || a->in_h == 0 || a->in_w == 0 || a->out_h == 0 || a->out_w == 0 || a->c_in == 0 || a->c_out == 0)
            return ISAACB_INVALID_ARG;
        if(a->c_in % 8 != 0 || a->c_out % 8 != 0 || a->c_out > 256 || a->ksize < 1 || a->ksize > 7 || a->stride < 1
           || a->stride > 4)
            return ISAACB_INVALID_ARG;
        const uint64_t pin = uint64_t(a->batch) * a->in_h * a->in_w, pout = uint64_t(a->batch) * a->out_h * a->out_w;
        if(pin * a->c_in >= (1ull << 31) || pout * a->c_out >= (1ull << 31))
            return ISAACB_INVALID_ARG;
        if(wgrad ? (!a->x || !a->dy || !a->dw) : (!a->x || !a->w || (!a->y && !a->y_f32)))
            return ISAACB_INVALID_ARG;
        return ISAACB_OK;
    }
} // namespace

extern "C"
{
    isaacb_status isaacb_conv_forward(const isaacb_conv_args* a, void* stream)
    {
        if(check_conv(a, false) != ISAACB_OK)
        {
            set_global_error("isaacb_conv_forward: invalid arguments");
            return ISAACB_INVALID_ARG;
        }
        ConvGemmParams p{};
        p.x = static_cast<const __nv_bfloat16*>(a->x);
        p.w = static_cast<const __nv_bfloat16*>(a->w);
        p.bias = a->bias;
        p.y = static_cast<__nv_bfloat16*>(a->y);
        p.yf = a->y_f32;
        p.mask = static_cast<const __nv_bfloat16*>(a->mask);
        p.B = int(a->batch);
        p.H = int(a->in_h);
        p.W = int(a->in_w);
        p.Cg = int(a->c_in);
        p.Ho = int(a->out_h);
        p.Wo = int(a->out_w);
        p.Cout = int(a->c_out);
        p.Npad = round_up(int(a->c_out), 16);
        p.Kpad = round_up(int(a->ksize * a->ksize * a->c_in), 64);
        p.ks = int(a->ksize);
        p.stride = int(a->stride);
        p.pad = int(a->pad);
        p.transposed = a->transposed ? 1 : 0;
        p.relu = a->relu ? 1 : 0;
        p.accumulate = a->accumulate ? 1 : 0;
        p.errorFlag = a->error_flag;
        p.waitCheckNs = 1000ull * a->wait_check_us;
        if(!launch_conv_gemm(p, (cudaStream_t) stream))
        {
            set_global_error("isaacb_conv_forward: weights do not fit in shared memory");
            return ISAACB_INVALID_ARG;
        }
        const cudaError_t e = cudaGetLastError();
        if(e != cudaSuccess)
        {
            set_global_error(std::string("isaacb_conv_forward: ") + cudaGetErrorString(e));
            return ISAACB_CUDA_ERROR;
        }
        return ISAACB_OK;
    }

    isaacb_status isaacb_conv_set_producer(int32_t tma)
    {
        g_rowTma = tma != 0;
        return ISAACB_OK;
    }

    isaacb_status isaacb_conv_wgrad(const isaacb_conv_args* a, void* stream)
    {
        if(check_conv(a, true) != ISAACB_OK)
        {
            set_global_error("isaacb_conv_wgrad: invalid arguments");
            return ISAACB_INVALID_ARG;
        }
        WgradParams p{};
        p.x = static_cast<const __nv_bfloat16*>(a->x);
        p.dy = static_cast<const __nv_bfloat16*>(a->dy);
        p.dw = a->dw;
        p.B = int(a->batch);
        p.H = int(a->in_h);
        p.W = int(a->in_w);
        p.Cin = int(a->c_in);
        p.Ho = int(a->out_h);
        p.Wo = int(a->out_w);
        p.Cout = int(a->c_out);
        p.Npad = round_up(int(a->c_out), 16);
        p.ks = int(a->ksize);
        p.stride = int(a->stride);
        p.pad = int(a->pad);
        p.Mtot = int(a->ksize * a->ksize * a->c_in);
        p.errorFlag = a->error_flag;
        if(!launch_conv_wgrad(&p, 1, (cudaStream_t) stream))
        {
            set_global_error("isaacb_conv_wgrad: tile does not fit in shared memory");
            return ISAACB_INVALID_ARG;
        }
        const cudaError_t e = cudaGetLastError();
        if(e != cudaSuccess)
        {
            set_global_error(std::string("isaacb_conv_wgrad: ") + cudaGetErrorString(e));
            return ISAACB_CUDA_ERROR;
        }
        return ISAACB_OK;
    }
}
