// Implicit-GEMM convolutions of the learned flow initialiser on the tcgen05 tensor core.
//
// Activations are bf16, their channels a multiple of 16, in one of two layouts: NHWC, or in planes
// of 8 channels, [n][c / 8][h][w][8].  The products read 8 channels of a pixel as one 16-byte row;
// a TMA box of NHWC data is made of such rows, at about 1.6 cycles each the bound of the wide
// layers, while a box of planes has rows of as many pixels as it is wide (seen as pairs of 64-bit
// elements).  The network keeps its tensors in planes (a training step of 8 images at 480x272 1.58 -> 1.48 ms).  Weights are kept as
// f32 masters [cout][tap][cin] (tap = 3 * (dy + 1) + (dx + 1) for 3x3, 0 for 1x1) and
// packed to bf16 operand images by pack_kernel.
//
// conv_kernel (forward, and the data gradient with packed transposed weights): persistent CTAs of
// 192 threads, each computing tiles of 128 output pixels (16 x 8; 128 x 1 in 1x1 layers between
// planes; M = 128) x all output channels (N = cout <= 256) into TMEM.  The K loop runs over (tap,
// chunk of ck input channels) stages through a ring in shared memory; producer and MMA issuer are
// whole warps in step, one elected lane executing the copies and MMAs (isti_tc.cuh):
//   warp 0: per stage, one TMA box of ck channels x the tile's pixels of the input at the tap's
//     offset (zero fill outside the image = the convolution's zero padding; NHWC without 5-D
//     maps: ck / 8 boxes) and one bulk copy of the stage's packed weights, completion on full[s];
//   warp 1: waits full[s], issues ck / 16 tcgen05.mma (K = 16 each) and commits to empty[s], which
//     frees the stage for the producer; after a tile's last stage, commits to acc_full of its
//     accumulator, one of two;
//   warps 2-5 (epilogue): wait acc_full, read their 32 TMEM lanes (= tile rows) with tcgen05.ld,
//     add the bias, apply ReLU and/or the gradient mask (x > 0 of a saved activation), convert to
//     bf16, store the pixel's channels and free the accumulator, while the next tile goes into the
//     other one.
// Every mbarrier wait is bounded; on timeout the status word is set, the loops stop, the
// producer waits (bounded) for the copies it issued, and TMEM is freed before returning.
//
// wgrad_kernel (weight gradient): K = pixels, both operands MN-major (the channel runs along the
// 16-byte row; for them the descriptor's LBO steps along K and its SBO along M/N, checked
// against torch).  A CTA covers a range of row segments and writes its partial sums; a second
// kernel adds the partials in a fixed order (deterministic).
#pragma once

#include "isti_pdl.cuh"
#include "isti_tc.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <algorithm>

namespace isti_unet
{
using namespace isti_tc;
using isti::dependents_may_launch;
using isti::wait_for_prerequisites;

constexpr size_t SMEM_BUDGET = 200 * 1024; // shared memory of a CTA that has the SM to itself
constexpr int TILE_W = 16, TILE_H = 8, TILE_M = TILE_W * TILE_H;
constexpr uint32_t BOX_BYTES = TILE_M * 16; // one TMA box: 8 channels x 128 pixels

__host__ __device__ constexpr uint32_t tmem_cols(int n)
{
    uint32_t c = 32;
    while (c < (uint32_t)n)
        c <<= 1;
    return c;
}

struct ConvParams
{
    const __nv_bfloat16 *wpack; // packed weights: per stage ck x cout, K-major core matrices [ck/8][cout/8][8][8]
    const float *bias;          // cout, or null
    const __nv_bfloat16 *mask;  // cout channels: output *= (mask > 0); or null
    __nv_bfloat16 *out;         // cout channels
    int32_t *status;
    int w, h, b;
    int cin, cout, ck;          // ck: input channels per stage (16 or 32)
    int tiles_x, tiles_y, n_tiles;
    int tile_shift;             // conv_kernel: log2 of the tile's width (4: 16 x 8 pixels; 7: 128 x 1, 1x1 layers in planes)
    int relu;
    int stages;                 // depth of the shared-memory ring
    int in_planes, out_planes;  // layouts of the input; of the output and the mask
    int chunked_map;            // NHWC input: 1: one 5-D box per stage (channel chunks outermost); 0: ck / 8 4-D boxes
    int halo, seg_out;          // row_conv_kernel: pixels per fetched row and outputs per unit
    // 1x1 output head fused into the epilogue (row_conv_kernel, inference): when head_w is
    // set, each pixel's bf16 outputs feed HEAD outputs = head_b + head_w . out (f32, fused
    // multiply-adds in channel order) written to head_flow (f32) and/or head_flow16 (f16),
    // and `out` is not written
    const float *head_w;        // [HEAD][cout]
    const float *head_b;        // [HEAD]
    float *head_flow;           // [pixel][HEAD], or null
    __half *head_flow16;        // [pixel][HEAD], or null
};

constexpr int CONV_HEAD = 4; // outputs of a fused head

__host__ __device__ constexpr uint32_t conv_stage_bytes(int ck, int cout) { return (uint32_t)ck * 256u + (uint32_t)ck * cout * 2u; }

// bf16 > 0 (positive, non-zero, not NaN)
__device__ __forceinline__ bool bf16_positive(uint16_t b) { return (b & 0x8000u) == 0 && (b & 0x7fffu) != 0 && (b & 0x7fffu) <= 0x7f80u; }

// The producer, MMA and epilogue loops run on one thread or four warps of a CTA, at the latency of
// every instruction: divisions are done once and positions then stepped along.

// Position in a ring of S stages: stage and phase (how often the ring wrapped, mod 2).
struct RingPos
{
    uint32_t s = 0, phase = 0;
    __device__ __forceinline__ void next(uint32_t S)
    {
        if (++s == S)
        {
            s = 0;
            phase ^= 1u;
        }
    }
};

// Unit u = (bi * ny + y) * nx + x, stepped by `step` units at a time.
struct UnitPos
{
    int x, y, b, dx, dy, db, nx, ny;
    __device__ __forceinline__ UnitPos(int u, int step, int nx_, int ny_) : nx(nx_), ny(ny_)
    {
        x = u % nx, u /= nx, y = u % ny, b = u / ny;
        dx = step % nx, step /= nx, dy = step % ny, db = step / ny;
    }
    __device__ __forceinline__ void next()
    {
        x += dx, y += dy, b += db;
        if (x >= nx)
            x -= nx, y++;
        if (y >= ny)
            y -= ny, b++;
    }
};

// What the epilogue reads for every pixel: bias, and the weights and bias of a fused head.
constexpr int CONV_MAX_COUT = 256;
struct EpilogueTable
{
    float bias[CONV_MAX_COUT];
    float head[CONV_HEAD * CONV_MAX_COUT], head_bias[CONV_HEAD];
    __device__ __forceinline__ void fill(const ConvParams &p) // whole block; complete before the kernel started (forward in isti_flownet.cu)
    {
        for (int i = threadIdx.x; i < p.cout; i += blockDim.x)
            bias[i] = p.bias ? __ldg(p.bias + i) : 0.0f;
        if (!p.head_w)
            return;
        for (int i = threadIdx.x; i < CONV_HEAD * p.cout; i += blockDim.x)
            head[i] = __ldg(p.head_w + i);
        if (threadIdx.x < CONV_HEAD)
            head_bias[threadIdx.x] = __ldg(p.head_b + threadIdx.x);
    }
};

// Drains the accumulator of one pixel per lane (warp-collective; columns taddr .. taddr + cout - 1):
// bias, ReLU, gradient mask, bf16, 16-byte stores or the fused head.  pix: the pixel within image bi;
// store: whether this lane's pixel exists.
__device__ __forceinline__ void epilogue_pixel(const ConvParams &p, const EpilogueTable &t, uint32_t taddr, int bi, uint32_t pix, bool store)
{
    // 16-byte groups of 8 channels: the pixel's first, and the distance to the next
    const size_t image = (size_t)p.h * p.w, groups = (size_t)(p.cout / 8);
    size_t group = p.out_planes ? (size_t)bi * groups * image + pix : ((size_t)bi * image + pix) * groups;
    const size_t step = p.out_planes ? image : 1;
    float hacc[CONV_HEAD];
    if (p.head_w)
#pragma unroll
        for (int q = 0; q < CONV_HEAD; q++)
            hacc[q] = t.head_bias[q];
#pragma unroll 1
    for (int c0 = 0; c0 < p.cout; c0 += 32)
    {
        uint32_t r[2][16];
        const int halves = c0 + 16 < p.cout ? 2 : 1;
        tmem_ld16(taddr + (uint32_t)c0, r[0]);
        if (halves == 2)
            tmem_ld16(taddr + (uint32_t)c0 + 16u, r[1]);
        tmem_ld_wait();
        if (!store)
            continue;
#pragma unroll
        for (int half = 0; half < 2; half++)
        {
            if (half == halves)
                break;
            const int c = c0 + 16 * half;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; j++)
                v[j] = __uint_as_float(r[half][j]);
            if (p.bias)
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                {
                    const float4 b = *reinterpret_cast<const float4 *>(t.bias + c + j);
                    v[j] += b.x, v[j + 1] += b.y, v[j + 2] += b.z, v[j + 3] += b.w;
                }
            if (p.relu)
#pragma unroll
                for (int j = 0; j < 16; j++)
                    v[j] = fmaxf(v[j], 0.0f);
            if (p.mask)
            {
                const uint4 *mk = reinterpret_cast<const uint4 *>(p.mask) + group;
                const uint4 m0 = mk[0], m1 = mk[step]; // plain loads: a previous kernel wrote them, perhaps after this launch
                const uint32_t mw[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (!bf16_positive((uint16_t)(mw[j / 2] >> (16 * (j % 2)))))
                        v[j] = 0.0f;
            }
            uint32_t o[8];
#pragma unroll
            for (int j = 0; j < 8; j++)
            {
                const __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                o[j] = *reinterpret_cast<const uint32_t *>(&h2);
            }
            if (p.head_w)
            {
#pragma unroll
                for (int j = 0; j < 8; j += 2)
                {
                    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&o[j]));
                    const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&o[j + 1]));
#pragma unroll
                    for (int q = 0; q < CONV_HEAD; q++)
                    {
                        const float4 w = *reinterpret_cast<const float4 *>(t.head + q * p.cout + c + 2 * j);
                        hacc[q] = fmaf(w.x, f.x, hacc[q]);
                        hacc[q] = fmaf(w.y, f.y, hacc[q]);
                        hacc[q] = fmaf(w.z, g.x, hacc[q]);
                        hacc[q] = fmaf(w.w, g.y, hacc[q]);
                    }
                }
            }
            else
            {
                uint4 *dst = reinterpret_cast<uint4 *>(p.out) + group;
                dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
                dst[step] = make_uint4(o[4], o[5], o[6], o[7]);
            }
            group += 2 * step;
        }
    }
    if (p.head_w && store)
    {
        const size_t hp = (size_t)bi * image + pix;
        if (p.head_flow)
            *reinterpret_cast<float4 *>(p.head_flow + hp * CONV_HEAD) = make_float4(hacc[0], hacc[1], hacc[2], hacc[3]);
        if (p.head_flow16)
        {
            const __half2 h0 = __floats2half2_rn(hacc[0], hacc[1]), h1 = __floats2half2_rn(hacc[2], hacc[3]);
            *reinterpret_cast<uint2 *>(p.head_flow16 + hp * CONV_HEAD) =
                make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
        }
    }
}

constexpr int PCONV_THREADS = 192; // warp 0: TMA producer, warp 1: MMA issuer, warps 2-5: epilogue

// Persistent convolution: each CTA works through tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// The producer runs ahead through the ring across tiles; the MMA issuer accumulates tile i into
// TMEM buffer i % 2 while the epilogue warps drain buffer (i - 1) % 2 (acc_full / acc_empty
// barriers), so stores overlap the next tile's loads and MMAs.
template <int TAPS>
__global__ void __launch_bounds__(PCONV_THREADS, 1) conv_kernel(const __grid_constant__ ConvParams p, const __grid_constant__ CUtensorMap xmap)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(16) EpilogueTable table;
    const int S = p.stages;
    const uint32_t a_bytes = (uint32_t)p.ck * 256u, b_bytes = (uint32_t)p.ck * p.cout * 2u, stage_bytes = a_bytes + b_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)S * stage_bytes);
    uint64_t *empty = full + S;
    uint64_t *acc_full = empty + S;
    uint64_t *acc_empty = acc_full + 2;
    uint64_t *mma_done = acc_empty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mma_done + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0), lane = threadIdx.x % 32; // warp: known to be uniform
    const uint32_t acc_cols = tmem_cols(p.cout), ncols = 2 * acc_cols;

    table.fill(p);
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < S; s++)
        {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++)
        {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4); // one arrival per epilogue warp
        }
        mbar_init(mma_done, 1);
        fence_barrier_init();
    }
    if (warp == 0)
        tmem_alloc(tmem_slot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int chunks = p.cin / p.ck;
    if (threadIdx.x == 0)
        dependents_may_launch(); // the next layer may set up while this one runs

    if (warp == 0)
    {
        const uint32_t leader = elect_one();
        wait_for_prerequisites(); // the previous layer's output is complete (every load below is later)
        fence_proxy_async_global();
        uint32_t g = 0; // stages filled
        RingPos ring;
        UnitPos at(blockIdx.x, gridDim.x, p.tiles_x, p.tiles_y);
        bool stop = false;
        for (int t = blockIdx.x; t < p.n_tiles && !stop; t += gridDim.x, at.next())
        {
            const int x0 = at.x << p.tile_shift, y0 = at.y * (TILE_M >> p.tile_shift);
            const __nv_bfloat16 *weights = p.wpack;
            for (int tap = 0; tap < TAPS && !stop; tap++)
            {
                const int dy = TAPS == 9 ? tap / 3 - 1 : 0, dx = TAPS == 9 ? tap % 3 - 1 : 0;
                for (int c = 0; c < chunks; c++, g++, ring.next(S), weights += p.ck * p.cout)
                {
                    const uint32_t s = ring.s;
                    if (!mbar_wait_warp(&empty[s], ring.phase ^ 1u, p.status)) // (the first round's waits return at once)
                    {
                        stop = true;
                        break;
                    }
                    const uint32_t st = smem_u32(smem) + s * stage_bytes;
                    mbar_expect_tx_if(leader, &full[s], stage_bytes);
                    if (p.in_planes)
                        tma_load_4d(leader, st, &xmap, 2 * (x0 + dx), y0 + dy, c * (p.ck / 8), at.b, &full[s]);
                    else if (p.chunked_map)
                        tma_load_5d(leader, st, &xmap, 0, x0 + dx, y0 + dy, c * (p.ck / 8), at.b, &full[s]);
                    else
                        for (int j = 0; j < p.ck / 8; j++)
                            tma_load_4d(leader, st + j * BOX_BYTES, &xmap, c * p.ck + 8 * j, x0 + dx, y0 + dy, at.b, &full[s]);
                    bulk_load(leader, st + a_bytes, weights, b_bytes, &full[s]);
                }
            }
        }
        for (uint32_t q = g > (uint32_t)S ? g - (uint32_t)S : 0u; q < g; q++) // copies still landing
            if (!mbar_wait_warp(&full[q % (uint32_t)S], (q / (uint32_t)S) & 1u, p.status))
                break;
    }
    else if (warp == 1)
    {
        const uint32_t leader = elect_one();
        const uint32_t idesc = idesc_bf16(TILE_M, (uint32_t)p.cout, 0, 0);
        const uint32_t lbo_b = (uint32_t)(p.cout / 8) * 128u;
        const int iters = TAPS * chunks;
        RingPos ring;
        int i = 0;
        bool stop = false;
        for (int t = blockIdx.x; t < p.n_tiles && !stop; t += gridDim.x, i++)
        {
            const int buf = i & 1;
            if (i >= 2 && !mbar_wait_warp(&acc_empty[buf], (uint32_t)(((i >> 1) - 1) & 1), p.status))
                break;
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)buf * acc_cols;
            for (int it = 0; it < iters; it++, ring.next(S))
            {
                const uint32_t s = ring.s;
                if (!mbar_wait_warp(&full[s], ring.phase, p.status))
                {
                    stop = true;
                    break;
                }
                tc_fence_after();
                const uint32_t a0 = smem_u32(smem) + s * stage_bytes;
                const Desc da(a0, BOX_BYTES, 128), db(a0 + a_bytes, lbo_b, 128);
                mma_bf16(leader, d, da, db, idesc, it > 0);
                if (p.ck == 32)
                    mma_bf16(leader, d, da + 2u * BOX_BYTES, db + 2u * lbo_b, idesc, true);
                mma_commit(leader, &empty[s]);
            }
            if (!stop)
                mma_commit(leader, &acc_full[buf]);
        }
        mma_commit(leader, mma_done);
    }
    else if (warp >= 2)
    {
        wait_for_prerequisites(); // the mask is complete
        const int q = warp % 4; // the TMEM lane quadrant this warp may read
        const int m = q * 32 + lane, mx = m & ((1 << p.tile_shift) - 1), my = m >> p.tile_shift;
        UnitPos at(blockIdx.x, gridDim.x, p.tiles_x, p.tiles_y);
        int i = 0;
        for (int t = blockIdx.x; t < p.n_tiles; t += gridDim.x, i++, at.next())
        {
            const int buf = i & 1;
            if (!mbar_wait(&acc_full[buf], (uint32_t)((i >> 1) & 1), p.status))
                break;
            tc_fence_after();
            const int px = (at.x << p.tile_shift) + mx, py = at.y * (TILE_M >> p.tile_shift) + my;
            epilogue_pixel(p, table, tmem + (uint32_t)buf * acc_cols + ((uint32_t)(q * 32) << 16), at.b, (uint32_t)py * (uint32_t)p.w + (uint32_t)px,
                           px < p.w && py < p.h);
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    if (warp == 0)
    {
        if (lane == 0)
            mbar_wait(mma_done, 0, p.status); // no MMA may still write TMEM when it is freed
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
    {
        tc_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// ---- row-tile 3x3 convolution for the wide, thin layers ----
//
// A unit is up to 128 consecutive output pixels of one row (M = 128).  Per chunk of ck input
// channels one TMA copy lands the unit's halo -- 3 input rows, channel groups of 8 outermost -- and
// the 9 taps are 9 descriptor start offsets into it ((dy + 1) rows and (dx + 1) pixels on, 16
// bytes per pixel and group), so every input pixel is fetched for 3 units instead of 9 taps.  From
// planes the copy is 128 pixels wide (a TMA box has at most 256 elements) for 126 outputs: the
// products of the last two pixels read past their row and are not stored.  From NHWC it is 130
// pixels wide for 128 outputs.  The weights of all taps and chunks stay in shared memory for the
// CTA's lifetime (one bulk copy).  Roles and the double-buffered TMEM accumulators are those of
// conv_kernel.
constexpr int ROW_M = 128, ROW_HALO = ROW_M + 2;
__host__ __device__ constexpr uint32_t row_chunk_bytes(int halo) { return 3u * halo * 16u; } // one 8-channel group
// (32 bytes more than the groups: the unstored products read that far)
__host__ __device__ constexpr uint32_t row_stage_bytes(int ck, int halo) { return ((uint32_t)(ck / 8) * row_chunk_bytes(halo) + 32u + 1023u) / 1024u * 1024u; }

template <int UNUSED = 0>
__global__ void __launch_bounds__(PCONV_THREADS, 1) row_conv_kernel(const __grid_constant__ ConvParams p, const __grid_constant__ CUtensorMap xmap)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(16) EpilogueTable table;
    const int S = p.stages;
    const int chunks = p.cin / p.ck;
    const uint32_t w_bytes = 9u * (uint32_t)p.cin * p.cout * 2u; // every tap and chunk, packed
    const uint32_t w_region = (w_bytes + 1023u) / 1024u * 1024u;
    const uint32_t chunk_bytes = row_chunk_bytes(p.halo), a_bytes = (uint32_t)(p.ck / 8) * chunk_bytes, stage_bytes = row_stage_bytes(p.ck, p.halo);
    uint8_t *wsm = smem;
    uint8_t *ring = smem + w_region;
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + (size_t)S * stage_bytes);
    uint64_t *empty = full + S;
    uint64_t *acc_full = empty + S;
    uint64_t *acc_empty = acc_full + 2;
    uint64_t *mma_done = acc_empty + 2;
    uint64_t *wbar = mma_done + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(wbar + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0), lane = threadIdx.x % 32; // warp: known to be uniform
    const uint32_t acc_cols = tmem_cols(p.cout), ncols = 2 * acc_cols;
    const int segs = (p.w + p.seg_out - 1) / p.seg_out;
    const int n_units = p.b * p.h * segs;

    table.fill(p);
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < S; s++)
        {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++)
        {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);
        }
        mbar_init(mma_done, 1);
        mbar_init(wbar, 1);
        fence_barrier_init();
    }
    if (warp == 0)
        tmem_alloc(tmem_slot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (threadIdx.x == 0)
        dependents_may_launch(); // the next layer may set up while this one runs
    if (warp == 0)
    {
        const uint32_t leader = elect_one();
        mbar_expect_tx_if(leader, wbar, w_bytes);
        for (uint32_t o = 0; o < w_bytes; o += 32768u) // pieces of at most 32 KiB (the weights are complete, forward in isti_flownet.cu)
            bulk_load(leader, smem_u32(wsm) + o, reinterpret_cast<const uint8_t *>(p.wpack) + o, min(32768u, w_bytes - o), wbar);
        wait_for_prerequisites(); // the previous layer's output is complete (every activation load below is later)
        fence_proxy_async_global();
        uint32_t g = 0;
        RingPos pos;
        UnitPos at(blockIdx.x, gridDim.x, segs, p.h);
        bool stop = false;
        for (int u = blockIdx.x; u < n_units && !stop; u += gridDim.x, at.next())
            for (int c = 0; c < chunks; c++, g++, pos.next(S))
            {
                const uint32_t s = pos.s;
                if (!mbar_wait_warp(&empty[s], pos.phase ^ 1u, p.status))
                {
                    stop = true;
                    break;
                }
                mbar_expect_tx_if(leader, &full[s], a_bytes);
                if (p.in_planes)
                    tma_load_4d(leader, smem_u32(ring) + s * stage_bytes, &xmap, 2 * (at.x * p.seg_out - 1), at.y - 1, c * (p.ck / 8), at.b, &full[s]);
                else
                    tma_load_5d(leader, smem_u32(ring) + s * stage_bytes, &xmap, 0, at.x * p.seg_out - 1, at.y - 1, c * (p.ck / 8), at.b, &full[s]);
            }
        for (uint32_t q = g > (uint32_t)S ? g - (uint32_t)S : 0u; q < g; q++)
            if (!mbar_wait_warp(&full[q % (uint32_t)S], (q / (uint32_t)S) & 1u, p.status))
                break;
        mbar_wait_warp(wbar, 0, p.status);
    }
    else if (warp == 1)
    {
        const uint32_t leader = elect_one();
        const uint32_t idesc = idesc_bf16(ROW_M, (uint32_t)p.cout, 0, 0);
        const uint32_t lbo_b = (uint32_t)(p.cout / 8) * 128u;
        const uint32_t wtap_bytes = (uint32_t)p.ck * p.cout * 2u; // packed weights of one tap and chunk
        const Desc db0(smem_u32(wsm), lbo_b, 128);
        RingPos pos;
        int i = 0;
        bool stop = !mbar_wait_warp(wbar, 0, p.status);
        for (int u = blockIdx.x; u < n_units && !stop; u += gridDim.x, i++)
        {
            const int buf = i & 1;
            if (i >= 2 && !mbar_wait_warp(&acc_empty[buf], (uint32_t)(((i >> 1) - 1) & 1), p.status))
                break;
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)buf * acc_cols;
            for (int c = 0; c < chunks; c++, pos.next(S))
            {
                const uint32_t s = pos.s;
                if (!mbar_wait_warp(&full[s], pos.phase, p.status))
                {
                    stop = true;
                    break;
                }
                tc_fence_after();
                const Desc da(smem_u32(ring) + s * stage_bytes, chunk_bytes, 128);
                Desc db = db0 + (uint32_t)c * wtap_bytes;
#pragma unroll
                for (int tap = 0; tap < 9; tap++, db = db + (uint32_t)chunks * wtap_bytes)
                {
                    const Desc dt = da + (uint32_t)((tap / 3) * p.halo + (tap % 3)) * 16u;
                    mma_bf16(leader, d, dt, db, idesc, c > 0 || tap > 0);
                    if (p.ck == 32)
                        mma_bf16(leader, d, dt + 2u * chunk_bytes, db + 2u * lbo_b, idesc, true);
                }
                mma_commit(leader, &empty[s]);
            }
            if (!stop)
                mma_commit(leader, &acc_full[buf]);
        }
        mma_commit(leader, mma_done);
    }
    else if (warp >= 2)
    {
        wait_for_prerequisites(); // the mask is complete
        const int q = warp % 4;
        const int m = q * 32 + lane;
        UnitPos at(blockIdx.x, gridDim.x, segs, p.h);
        int i = 0;
        for (int u = blockIdx.x; u < n_units; u += gridDim.x, i++, at.next())
        {
            const int buf = i & 1;
            if (!mbar_wait(&acc_full[buf], (uint32_t)((i >> 1) & 1), p.status))
                break;
            tc_fence_after();
            const int px = at.x * p.seg_out + m;
            epilogue_pixel(p, table, tmem + (uint32_t)buf * acc_cols + ((uint32_t)(q * 32) << 16), at.b, (uint32_t)at.y * (uint32_t)p.w + (uint32_t)px,
                           m < p.seg_out && px < p.w);
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    if (warp == 0)
    {
        if (lane == 0)
            mbar_wait(mma_done, 0, p.status);
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
    {
        tc_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// ---- weight gradient ----
//
// dW[co][tap][ci] = sum over pixels p of dY[p + s][co] * X[p + dy rows][ci] with tap = (dy, dx = -s):
// the horizontal offset is taken on dY's side.  A unit is KSEG consecutive pixels of a row, the
// K of the products.  A = the rows (s, co) of dY, its three shifted copies one after another (each a
// TMA copy of the same pixels at another x), packed into M blocks of 128 -- 96 of 128 rows used for
// 32 output channels, where one tap per product would use 32.  B = the channels of the X rows
// y - 1 .. y + 1 (one copy), each row a product of its own with N = cin.  So dY and X are fetched
// three times per pixel instead of once per tap, and a unit takes 3 products per M block instead of 9.
// The bias gradient (the column sums of dY) rides along: the row of dy = 0 has 16 more columns of
// ones behind its channels.  Both operands are MN-major (the channel runs along the 16-byte row).
// A CTA keeps every accumulator in TMEM: M blocks x (rows x cin + 16) columns; where that exceeds
// 512 the grid's y takes one dy each, and its z one M block each (wgrad_config in isti_unet.cu;
// N_DY X rows and N_MB M blocks per CTA).
// 1x1 layers: one row, no shift, an image one row of pixels.
//
// Bound by the issue of narrow MMAs (about 75 cycles each) and by shared-memory operand reads (4 KB
// of A per K = 16 step).  8 images of 480x272: 32 -> 32 channels 407 -> 50 us, 16 -> 32 358 -> 41,
// 64 -> 64 at half size 154 -> 37; the bias gradients had passes over dY of their own, 0.7 ms of a
// 3.0 ms step.
struct WgradParams
{
    float *partial;  // [splits][cout][TAPS][cin]
    float *bpartial; // [splits][cout], or null: no bias gradient
    int32_t *status;
    int w, h, b;
    int cin, cout;
    int kseg, segs, n_units, units_per_split;
    int dy_planes, x_planes; // layouts
    int box_chunks; // channel chunks (of 8) per TMA box of dY: cout / 8, or 1 where an M block may start inside a shift
    int stages;
};

__host__ __device__ constexpr uint32_t wgrad_a_bytes(int n_mb, int kseg) { return (uint32_t)n_mb * 16u * kseg * 16u; }
__host__ __device__ constexpr uint32_t wgrad_stage_bytes(int cin, int n_dy, int n_mb, int kseg)
{
    return wgrad_a_bytes(n_mb, kseg) + (uint32_t)(cin / 8 + 2) * n_dy * kseg * 16u; // two chunks of ones behind X's
}
__host__ __device__ constexpr int wgrad_mb_cols(int cin, int n_dy) { return n_dy * cin + 16; }

// The work split of wgrad_kernel.  Every split has units (tests/cpp/wgrad_splits_test.cu): one without
// would write its zeros, and be added up, for nothing.
struct WgradConfig
{
    int n, h, w;              // the images, those of 1x1 layers as one row of pixels each
    int kseg, segs, n_units;
    int n_dy, n_mb;           // per CTA
    int grid_y, grid_z, splits, units_per_split, stages;
    size_t smem;
};

inline bool wgrad_config(int taps, int n, int h, int w, int cin, int cout, WgradConfig &c)
{
    c = WgradConfig{};
    c.n = n;
    c.h = taps == 9 ? h : 1;
    const long long row = taps == 9 ? w : (long long)h * w;
    if (row > INT32_MAX / 2 - 256)
        return false;
    c.w = (int)row;
    const int mblocks = ((taps == 9 ? 3 : 1) * cout + 127) / 128;
    c.n_dy = taps == 9 ? 3 : 1;
    c.n_mb = mblocks;
    // all accumulators of a CTA in the 512 TMEM columns: else one row (dy) per CTA, then one M block
    if (c.n_dy == 3 && c.n_mb * wgrad_mb_cols(cin, 3) > 512)
        c.n_dy = 1;
    if (c.n_mb * wgrad_mb_cols(cin, c.n_dy) > 512)
        c.n_mb = 1;
    c.grid_y = taps == 9 && c.n_dy == 1 ? 3 : 1;
    c.grid_z = mblocks / c.n_mb;
    // 128 pixels per unit where three stages of them fit and the rows are that long, else 64
    for (c.kseg = 128;; c.kseg = 64)
    {
        const size_t sb = wgrad_stage_bytes(cin, c.n_dy, c.n_mb, c.kseg);
        c.stages = (int)std::min<size_t>(6, (SMEM_BUDGET - 256) / sb);
        if (c.kseg == 64 || (c.stages >= 3 && c.w > 64))
        {
            c.smem = c.stages * sb + (2 * c.stages + 1) * 8 + 16;
            break;
        }
    }
    c.segs = (c.w + c.kseg - 1) / c.kseg;
    c.n_units = c.n * c.h * c.segs;
    // at most one CTA per SM, at least 4 units each (the last one takes what is left)
    const int most = std::max(1, std::min(152 / (c.grid_y * c.grid_z), (c.n_units + 3) / 4));
    c.units_per_split = (c.n_units + most - 1) / most;
    c.splits = (c.n_units + c.units_per_split - 1) / c.units_per_split;
    return c.stages >= 2;
}

constexpr int WGRAD_THREADS = 128; // warp 0 producer, warp 1 MMA, all four epilogue

template <int TAPS, int N_DY, int N_MB>
__global__ void __launch_bounds__(WGRAD_THREADS) wgrad_kernel(const __grid_constant__ WgradParams p, const __grid_constant__ CUtensorMap dymap,
                                                              const __grid_constant__ CUtensorMap xmap)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int SHIFTS = TAPS == 9 ? 3 : 1;
    const int S = p.stages;
    const uint32_t px_bytes = (uint32_t)p.kseg * 16u; // one channel chunk of a unit's pixels
    const uint32_t a_bytes = wgrad_a_bytes(N_MB, p.kseg), stage_bytes = wgrad_stage_bytes(p.cin, N_DY, N_MB, p.kseg);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)S * stage_bytes);
    uint64_t *empty = full + S;
    uint64_t *done = empty + S;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0), lane = threadIdx.x % 32; // warp: known to be uniform
    const int split = blockIdx.x, dy0 = TAPS == 9 ? (int)blockIdx.y : 1, mb0 = (int)blockIdx.z * N_MB; // dy0: first row, 0..2
    const int u_begin = split * p.units_per_split, u_end = min(p.n_units, u_begin + p.units_per_split);
    const int iters = max(0, u_end - u_begin);
    const int co_chunks = p.cout / 8;
    const int boxes = min(N_MB * 16, SHIFTS * co_chunks - mb0 * 16) / p.box_chunks; // dY boxes of this CTA
    const uint32_t ncols = tmem_cols(N_MB * wgrad_mb_cols(p.cin, N_DY));
    const uint32_t b_rows_bytes = (uint32_t)N_DY * px_bytes; // one channel chunk of X
    // columns of row d within an M block: the row of dy = 0 has 16 more
    auto row_col = [&](int d) { return d * p.cin + (dy0 + d > 1 && d > 0 ? 16 : 0); };

    // rows of A past the last channel and the ones behind X's channels are never loaded: set once,
    // for every stage
    for (uint32_t i = threadIdx.x * 16u; i < (uint32_t)S * stage_bytes; i += WGRAD_THREADS * 16u)
    {
        const uint32_t v = i % stage_bytes >= a_bytes + (uint32_t)(p.cin / 8) * b_rows_bytes ? 0x3f803f80u : 0u;
        *reinterpret_cast<uint4 *>(smem + i) = make_uint4(v, v, v, v);
    }
    fence_proxy_async();
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < S; s++)
        {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        fence_barrier_init();
    }
    if (warp == 0)
        tmem_alloc(tmem_slot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (threadIdx.x == 0)
        dependents_may_launch();
    if (warp == 0)
    {
        const uint32_t leader = elect_one();
        wait_for_prerequisites(); // dY and X are complete (every load below is later)
        fence_proxy_async_global();
        const uint32_t tx_bytes = (uint32_t)(boxes * p.box_chunks) * px_bytes + (uint32_t)(p.cin / 8) * b_rows_bytes;
        const int shift0 = mb0 * 16 / co_chunks, group0 = mb0 * 16 % co_chunks; // of the first box
        RingPos ring;
        UnitPos at(u_begin, 1, p.segs, p.h);
        int issued = 0;
        for (int it = 0; it < iters; it++, ring.next(S), at.next())
        {
            const uint32_t s = ring.s;
            if (!mbar_wait_warp(&empty[s], ring.phase ^ 1u, p.status)) // (the first round's waits return at once)
                break;
            const int x0 = at.x * p.kseg;
            const uint32_t st = smem_u32(smem) + s * stage_bytes;
            mbar_expect_tx_if(leader, &full[s], tx_bytes);
            int shift = TAPS == 9 ? shift0 - 1 : 0, group = group0;
            for (int b = 0; b < boxes; b++)
            {
                const uint32_t dst = st + (uint32_t)(b * p.box_chunks) * px_bytes;
                if (p.dy_planes)
                    tma_load_4d(leader, dst, &dymap, 2 * (x0 + shift), at.y, group, at.b, &full[s]);
                else
                    tma_load_5d(leader, dst, &dymap, 0, x0 + shift, at.y, group, at.b, &full[s]);
                group += p.box_chunks;
                if (group >= co_chunks)
                    group = 0, shift++;
            }
            if (p.x_planes)
                tma_load_4d(leader, st + a_bytes, &xmap, 2 * x0, at.y + dy0 - 1, 0, at.b, &full[s]);
            else
                tma_load_5d(leader, st + a_bytes, &xmap, 0, x0, at.y + dy0 - 1, 0, at.b, &full[s]);
            issued = it + 1;
        }
        for (int it = issued > S ? issued - S : 0; it < issued; it++)
            if (!mbar_wait_warp(&full[it % S], (uint32_t)((it / S) & 1), p.status))
                break;
    }
    else if (warp == 1)
    {
        const uint32_t leader = elect_one();
        // MN-major operands: LBO = distance between core matrices adjacent in K (the next 8
        // pixels, 128 bytes on), SBO = between core matrices adjacent in M/N (the next 8 channels)
        const uint32_t idesc_side = idesc_bf16(128, (uint32_t)p.cin, 1, 1);
        const uint32_t idesc_centre = idesc_bf16(128, (uint32_t)p.cin + (p.bpartial ? 16u : 0u), 1, 1);
        const uint32_t mb_cols = (uint32_t)wgrad_mb_cols(p.cin, N_DY);
        uint32_t row_cols[N_DY];
#pragma unroll
        for (int d = 0; d < N_DY; d++)
            row_cols[d] = (uint32_t)row_col(d);
        RingPos ring;
        for (int it = 0; it < iters; it++, ring.next(S))
        {
            const uint32_t s = ring.s;
            if (!mbar_wait_warp(&full[s], ring.phase, p.status))
                break;
            tc_fence_after();
            const uint32_t a0 = smem_u32(smem) + s * stage_bytes, b0 = a0 + a_bytes;
            const Desc da(a0, 128u, px_bytes), db(b0, 128u, b_rows_bytes);
            // K = 16 pixels per MMA: two 8-pixel core-matrix groups, 256 bytes on.  The accumulators in
            // turn, an MMA into the one before's waits for it; unrolled, the loop costs more than that
            for (uint32_t k0 = 0; k0 < px_bytes; k0 += 1024u)
            {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int mb = 0; mb < N_MB; mb++)
#pragma unroll
                        for (int d = 0; d < N_DY; d++)
                        {
                            const uint32_t k = k0 + 256u * q;
                            mma_bf16(leader, tmem + (uint32_t)mb * mb_cols + row_cols[d], da + (uint32_t)mb * 16u * px_bytes + k,
                                     db + (uint32_t)d * px_bytes + k, dy0 + d == 1 ? idesc_centre : idesc_side, it > 0 || k0 > 0 || q > 0);
                        }
            }
            mma_commit(leader, &empty[s]);
        }
        mma_commit(leader, done);
    }
    __syncwarp();

    // The scratch is one for all layers, and the kernels between let this one start before they
    // waited themselves: the reduction of the layer before may still read it.  (Warp 0's wait
    // orders a CTA's stores by way of its copies and products only where it has units.)
    wait_for_prerequisites();
    const bool ok = mbar_wait(done, 0, p.status);
    tc_fence_after();
    if (ok)
        for (int mb = 0; mb < N_MB; mb++)
        {
            const int m = (mb0 + mb) * 128 + warp * 32 + lane; // row (shift, co)
            const int shift = m / p.cout, co = m % p.cout;
            for (int d = 0; d < N_DY; d++)
            {
                const int tap = TAPS == 9 ? (dy0 + d) * 3 + (2 - shift) : 0;
                const bool ones = p.bpartial && dy0 + d == 1;
                for (int c0 = 0; c0 < p.cin + (ones ? 16 : 0); c0 += 16)
                {
                    uint32_t r[16];
                    tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(mb * wgrad_mb_cols(p.cin, N_DY) + row_col(d) + c0), r);
                    tmem_ld_wait();
                    if (shift >= SHIFTS)
                        continue;
                    if (c0 == p.cin)
                    {
                        if (shift == SHIFTS / 2)
                            p.bpartial[(size_t)split * p.cout + co] = iters > 0 ? __uint_as_float(r[0]) : 0.0f;
                        continue;
                    }
                    float4 *dst = reinterpret_cast<float4 *>(p.partial + (((size_t)split * p.cout + co) * TAPS + tap) * p.cin + c0);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        dst[i] = iters > 0 ? make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                                                         __uint_as_float(r[4 * i + 3]))
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        tmem_dealloc(tmem, ncols);
}

// dW (+)= sum over splits of the partials, in a fixed order: eight threads per value add every
// eighth split, then their sums are added.  The bias gradients db follow the n weights (db may be null).
constexpr int WREDUCE_PARTS = 8;
__global__ void __launch_bounds__(32 * WREDUCE_PARTS) wgrad_reduce_kernel(const float *partial, const float *bpartial, int splits, int n, int nb,
                                                                          float *dw, float *db, int accumulate)
{
    __shared__ float part[WREDUCE_PARTS][32];
    dependents_may_launch();
    wait_for_prerequisites();
    const int i = blockIdx.x * 32 + threadIdx.x;
    const bool weight = i < n, used = weight || (db && i < n + nb);
    float s = 0.0f;
    if (used)
    {
        const float *src = weight ? partial + i : bpartial + (i - n);
        const size_t stride = weight ? n : nb;
#pragma unroll 4
        for (int k = threadIdx.y; k < splits; k += WREDUCE_PARTS)
            s += src[k * stride];
    }
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y != 0 || !used)
        return;
    float *out = weight ? dw + i : db + (i - n);
    float total = accumulate ? *out : 0.0f;
#pragma unroll
    for (int k = 0; k < WREDUCE_PARTS; k++)
        total += part[k][threadIdx.x];
    *out = total;
}

// Packs f32 weights [cout][taps][cin] into the bf16 operand image of conv_kernel:
// per stage (tap, chunk of ck input channels) a K-major block [ck/8][cout/8][8 rows = out
// channel][8 = in channel].  transpose != 0 packs the data-gradient convolution instead:
// its inputs are the forward's outputs and its taps mirrored (dX = conv(dY, W^T flipped)).
__global__ void pack_kernel(const float *w, int taps, int cin, int cout, int transpose, __nv_bfloat16 *wpack)
{
    const int n = taps * cin * cout;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const int co = i / (taps * cin), tap = (i / cin) % taps, ci = i % cin;
    // the packed convolution's (input channel, tap, output channel)
    const int pin = transpose ? co : ci, pout = transpose ? ci : co, ptap = transpose ? taps - 1 - tap : tap;
    const int pcin = transpose ? cout : cin, pcout = transpose ? cin : cout;
    const int ck = pcin % 32 == 0 ? 32 : 16;
    const int stage = ptap * (pcin / ck) + pin / ck;
    const int kin = pin % ck;
    const size_t off = (size_t)stage * ck * pcout + (((size_t)(kin / 8) * (pcout / 8) + pout / 8) * 8 + pout % 8) * 8 + kin % 8;
    wpack[off] = __float2bfloat16_rn(w[i]);
}
} // namespace isti_unet
