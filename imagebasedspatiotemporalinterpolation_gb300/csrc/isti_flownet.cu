// The learned flow initialiser network: layers, forward pass, training backward pass and
// Adam, over the tcgen05 convolution operators (isti_unet.cu) and the CUDA-core kernels
// below (pooling, upsampling skips, gradient masks, the 1x1 output head, loss, bias
// gradients, optimiser).  C ABI: include/isti_unet.h.
//
// Architecture (H, W: the quarter-resolution input size, multiples of 8):
//   x0  [H,W,16]  inputs (isti_flownet_input_channels)
//   e1 = relu(conv3x3 16->32)(x0)          q1 = avgpool2(e1)   [H/2]
//   e2 = relu(conv3x3 32->64)(q1)          q2 = avgpool2(e2)   [H/4]
//   e3 = relu(conv3x3 64->96)(q2)          q3 = avgpool2(e3)   [H/8]
//   e4 = relu(conv3x3 96->128)(q3)
//   s3 = up2(conv1x1 128->96 (e4)) + e3    d3 = relu(conv3x3 96->96)(s3)
//   s2 = up2(conv1x1 96->64 (d3)) + e2     d2 = relu(conv3x3 64->64)(s2)
//   s1 = up2(conv1x1 64->32 (d2)) + e1     d1 = relu(conv3x3 32->32)(s1)
//   flow = conv1x1 32->4 (d1)              [H,W,4] f32
// 10 tensor-core layers + the head: 339,268 parameters.
#include "isti_pdl.cuh"
#include "isti_tc.cuh"
#include "isti_unet.h"
#include "isti_unet_ops.h"
#include "host/isti_error.hpp"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace
{
using bf16 = __nv_bfloat16;

struct LayerDef
{
    int taps, cin, cout, relu;
};

constexpr int N_CONV = 10;
constexpr LayerDef LAYERS[N_CONV] = {
    {9, 16, 32, 1},   // 0 e1
    {9, 32, 64, 1},   // 1 e2
    {9, 64, 96, 1},   // 2 e3
    {9, 96, 128, 1},  // 3 e4
    {1, 128, 96, 0},  // 4 p3
    {9, 96, 96, 1},   // 5 d3
    {1, 96, 64, 0},   // 6 p2
    {9, 64, 64, 1},   // 7 d2
    {1, 64, 32, 0},   // 8 p1
    {9, 32, 32, 1},   // 9 d1
};
constexpr int HEAD_CIN = 32, HEAD_COUT = 4;
constexpr int IN_CH = 16;

isti_status cuda_fail(cudaError_t e, const char *what) { return isti::set_error(ISTI_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e)); }

// ---- elementwise kernels on bf16, 8 channels (16 bytes) at a time ----

__device__ __forceinline__ void unpack8(uint4 u, float (&f)[8])
{
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; i++)
    {
        const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&w[i]);
        const float2 v = __bfloat1622float2(h);
        f[2 * i] = v.x;
        f[2 * i + 1] = v.y;
    }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8])
{
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
    {
        const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// The elementwise kernels work on tensors in planes of 8 channels ([n][c / 8][h][w][8],
// isti_unet_conv.cuh): a thread takes one 16-byte group of a half-resolution pixel and the 2x2
// block of the full resolution under it.  planes = n * c / 8; ho, wo: the half resolution.
// f(index of the half-resolution group, index of the block's first group, the full row's groups).
constexpr int EW_X = 64, EW_Y = 4;
template <class F>
__device__ __forceinline__ void for_each_block(uint32_t planes, uint32_t ho, uint32_t wo, F f)
{
    for (uint32_t r = blockIdx.x * EW_Y + threadIdx.y; r < planes * ho; r += gridDim.x * EW_Y)
    {
        const uint32_t plane = r / ho, yo = r - plane * ho;
        for (uint32_t x = threadIdx.x; x < wo; x += EW_X)
            f((size_t)r * wo + x, ((size_t)plane * ho + yo) * 4 * wo + 2 * x, (size_t)2 * wo);
    }
}

__device__ __forceinline__ void add8(float (&acc)[8], const bf16 *x, size_t group)
{
    float f[8];
    unpack8(reinterpret_cast<const uint4 *>(x)[group], f); // plain load: the previous kernel may still run at launch
#pragma unroll
    for (int k = 0; k < 8; k++)
        acc[k] += f[k];
}

// r = scale * the sum of x over 2x2 blocks: average pooling (0.25), gradient of nearest upsampling (1)
__global__ void __launch_bounds__(EW_X * EW_Y) blocksum_kernel(const bf16 *x, uint32_t planes, uint32_t ho, uint32_t wo, float scale, bf16 *r)
{
    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    for_each_block(planes, ho, wo, [&](size_t half, size_t full, size_t row) {
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        add8(acc, x, full);
        add8(acc, x, full + 1);
        add8(acc, x, full + row);
        add8(acc, x, full + row + 1);
#pragma unroll
        for (int k = 0; k < 8; k++)
            acc[k] *= scale;
        reinterpret_cast<uint4 *>(r)[half] = pack8(acc);
    });
}

// s[h, w] = a[h/2, w/2] (nearest upsampling) + b[h, w]
__global__ void __launch_bounds__(EW_X * EW_Y) upadd_kernel(const bf16 *a, const bf16 *b, uint32_t planes, uint32_t ho, uint32_t wo, bf16 *s)
{
    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    for_each_block(planes, ho, wo, [&](size_t half, size_t full, size_t row) {
        const uint4 ua = reinterpret_cast<const uint4 *>(a)[half];
        uint4 ub[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            ub[q] = reinterpret_cast<const uint4 *>(b)[full + (q / 2) * row + q % 2];
        float fa[8];
        unpack8(ua, fa);
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            float fb[8];
            unpack8(ub[q], fb);
#pragma unroll
            for (int k = 0; k < 8; k++)
                fb[k] = fa[k] + fb[k];
            reinterpret_cast<uint4 *>(s)[full + (q / 2) * row + q % 2] = pack8(fb);
        }
    });
}

// ge[h, w] = (gskip[h, w] + gq[h/2, w/2] / 4) * (act > 0): the gradient of an encoder
// activation that feeds both a skip connection and the 2x2 average pool, through its ReLU
__global__ void __launch_bounds__(EW_X * EW_Y) poolback_kernel(const bf16 *gskip, const bf16 *gq, const bf16 *act, uint32_t planes, uint32_t ho,
                                                               uint32_t wo, bf16 *ge)
{
    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    for_each_block(planes, ho, wo, [&](size_t half, size_t full, size_t row) {
        uint4 us[4], ua[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            us[q] = reinterpret_cast<const uint4 *>(gskip)[full + (q / 2) * row + q % 2];
            ua[q] = reinterpret_cast<const uint4 *>(act)[full + (q / 2) * row + q % 2];
        }
        float fq[8];
        unpack8(reinterpret_cast<const uint4 *>(gq)[half], fq);
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            float fs[8], fa[8];
            unpack8(us[q], fs);
            unpack8(ua[q], fa);
#pragma unroll
            for (int k = 0; k < 8; k++)
                fs[k] = fa[k] > 0.0f ? fs[k] + 0.25f * fq[k] : 0.0f;
            reinterpret_cast<uint4 *>(ge)[full + (q / 2) * row + q % 2] = pack8(fs);
        }
    });
}

// 16-byte group q of pixel p (of all images) of a tensor in planes with `groups` groups
__device__ __forceinline__ size_t plane_group(size_t p, size_t image, int groups, int q)
{
    const size_t b = p / image;
    return (b * groups + q) * image + (p - b * image);
}

// flow[p][0..3] = hb + hw . d1[p]  (the 1x1 output head, f32); optionally also f16
__global__ void head_kernel(const bf16 *d1, size_t npix, size_t image, const float *hw, const float *hb, float *flow, __half *flow16)
{
    __shared__ float sw[HEAD_COUT * HEAD_CIN + HEAD_COUT];
    for (int i = threadIdx.x; i < HEAD_COUT * HEAD_CIN; i += blockDim.x)
        sw[i] = hw[i];
    if (threadIdx.x < HEAD_COUT)
        sw[HEAD_COUT * HEAD_CIN + threadIdx.x] = hb[threadIdx.x];
    isti::dependents_may_launch();
    isti::wait_for_prerequisites(); // the weights above are no previous kernel's output; d1 is
    __syncthreads();
    for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += (size_t)gridDim.x * blockDim.x)
    {
        float f[HEAD_CIN];
        const uint4 *src = reinterpret_cast<const uint4 *>(d1) + plane_group(p, image, HEAD_CIN / 8, 0);
#pragma unroll
        for (int q = 0; q < HEAD_CIN / 8; q++)
        {
            float t[8];
            unpack8(src[q * image], t); // plain load: written by the previous kernel, which may still run at launch
#pragma unroll
            for (int k = 0; k < 8; k++)
                f[8 * q + k] = t[k];
        }
        float o[HEAD_COUT];
#pragma unroll
        for (int j = 0; j < HEAD_COUT; j++)
        {
            float a = sw[HEAD_COUT * HEAD_CIN + j];
#pragma unroll
            for (int k = 0; k < HEAD_CIN; k++)
                a = fmaf(sw[j * HEAD_CIN + k], f[k], a); // fused multiply-adds in channel order, as the fused head
            o[j] = a;
        }
        if (flow)
            *reinterpret_cast<float4 *>(flow + p * 4) = make_float4(o[0], o[1], o[2], o[3]);
        if (flow16)
        {
            __half2 a = __floats2half2_rn(o[0], o[1]), b = __floats2half2_rn(o[2], o[3]);
            uint2 u;
            u.x = *reinterpret_cast<uint32_t *>(&a);
            u.y = *reinterpret_cast<uint32_t *>(&b);
            *reinterpret_cast<uint2 *>(flow16 + p * 4) = u;
        }
    }
}

// Loss and head backward.  Loss = sum over labelled entries of huber(flow - label) / npix
// (label NaN = not labelled; huber with delta 1: 0.5 d^2 for |d| < 1, |d| - 0.5 beyond).
// Writes the gradient of the head's input through d1's ReLU (bf16), and per block the partials of
// the head's weight and bias gradients and of the loss, [block][4 * 32 + 4 + 1].
//
// A block works through tiles of 256 pixels in two steps: a thread per pixel (flow, loss, the
// gradient of the head's input; the output gradients go to shared memory), then a thread per
// channel group and pixel for the head's gradients, with 36 sums per thread.  (All 132 sums in the
// thread of a pixel left 8 warps per SM: 8 images of 480x272 97 -> 55 us.)
constexpr int HEAD_GRADS = HEAD_COUT * HEAD_CIN + HEAD_COUT, HEAD_VALUES = HEAD_GRADS + 1;
constexpr int HEAD_GROUPS = HEAD_CIN / 8, HEAD_TILE = 256, HEAD_LANES = HEAD_TILE / HEAD_GROUPS;
__global__ void __launch_bounds__(HEAD_TILE, 2) head_back_kernel(const bf16 *d1, size_t npix, size_t image, const float *hw, const float *hb,
                                                                 const float *label, float inv_norm, bf16 *g_d1, float *partial)
{
    __shared__ __align__(16) float sw[HEAD_GRADS];
    __shared__ float4 gout[2][HEAD_TILE];
    __shared__ float warp_sums[HEAD_TILE / 32][HEAD_COUT * 8 + HEAD_COUT + 1];
    for (int i = threadIdx.x; i < HEAD_COUT * HEAD_CIN; i += HEAD_TILE)
        sw[i] = hw[i];
    if (threadIdx.x < HEAD_COUT)
        sw[HEAD_COUT * HEAD_CIN + threadIdx.x] = hb[threadIdx.x];
    isti::dependents_may_launch();
    isti::wait_for_prerequisites(); // the weights above are no previous kernel's output; d1 is
    __syncthreads();
    const bool label_vec = (reinterpret_cast<uintptr_t>(label) & 15u) == 0;
    const int q = threadIdx.x / HEAD_LANES, lane = threadIdx.x % HEAD_LANES; // second step: channel group, pixel lane
    float my_loss = 0.0f, my_w[HEAD_COUT][8] = {}, my_b[HEAD_COUT] = {};
    int buf = 0;
    for (size_t p0 = (size_t)blockIdx.x * HEAD_TILE; p0 < npix; p0 += (size_t)gridDim.x * HEAD_TILE, buf ^= 1)
    {
        const size_t p = p0 + threadIdx.x;
        float go[HEAD_COUT] = {};
        if (p < npix)
        {
            const size_t group = plane_group(p, image, HEAD_GROUPS, 0);
            const uint4 *src = reinterpret_cast<const uint4 *>(d1) + group;
            float l[HEAD_COUT];
            if (label_vec)
            {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(label) + p);
                l[0] = v.x, l[1] = v.y, l[2] = v.z, l[3] = v.w;
            }
            else
#pragma unroll
                for (int j = 0; j < HEAD_COUT; j++)
                    l[j] = __ldg(label + p * HEAD_COUT + j);
            float f[HEAD_CIN];
#pragma unroll
            for (int g = 0; g < HEAD_GROUPS; g++)
            {
                float t[8];
                unpack8(src[g * image], t);
#pragma unroll
                for (int k = 0; k < 8; k++)
                    f[8 * g + k] = t[k];
            }
#pragma unroll
            for (int j = 0; j < HEAD_COUT; j++)
            {
                float a = sw[HEAD_COUT * HEAD_CIN + j];
#pragma unroll
                for (int k = 0; k < HEAD_CIN; k++)
                    a = fmaf(sw[j * HEAD_CIN + k], f[k], a); // fused multiply-adds in channel order, as the fused head
                if (!isnan(l[j]))
                {
                    const float d = a - l[j], ad = fabsf(d);
                    my_loss += (ad < 1.0f ? 0.5f * d * d : ad - 0.5f) * inv_norm;
                    go[j] = fminf(1.0f, fmaxf(-1.0f, d)) * inv_norm;
                }
            }
            asm volatile("" ::: "memory"); // the weights are read again: kept, all 128 would stay in registers
            uint4 *dst = reinterpret_cast<uint4 *>(g_d1) + group;
#pragma unroll
            for (int g = 0; g < HEAD_GROUPS; g++)
            {
                float t[8];
#pragma unroll
                for (int k = 0; k < 8; k++)
                {
                    float s = 0.0f;
#pragma unroll
                    for (int j = 0; j < HEAD_COUT; j++)
                        s += sw[j * HEAD_CIN + 8 * g + k] * go[j];
                    t[k] = f[8 * g + k] > 0.0f ? s : 0.0f;
                }
                dst[g * image] = pack8(t);
            }
        }
        gout[buf][threadIdx.x] = make_float4(go[0], go[1], go[2], go[3]);
        __syncthreads(); // (the other buffer is free by the next tile's barrier)
#pragma unroll
        for (int i = 0; i < HEAD_TILE / HEAD_LANES; i++)
        {
            const int t = i * HEAD_LANES + lane;
            if (p0 + t >= npix)
                break;
            const float4 g4 = gout[buf][t];
            const float g[HEAD_COUT] = {g4.x, g4.y, g4.z, g4.w};
            float f[8];
            unpack8(reinterpret_cast<const uint4 *>(d1)[plane_group(p0 + t, image, HEAD_GROUPS, q)], f);
#pragma unroll
            for (int j = 0; j < HEAD_COUT; j++)
            {
#pragma unroll
                for (int k = 0; k < 8; k++)
                    my_w[j][k] += g[j] * f[k];
                my_b[j] += g[j];
            }
        }
    }
    // block sums: warp shuffles, then the warps of a channel group (of all pixels for the loss) in order
    const int warp = threadIdx.x / 32;
    auto warp_total = [&](float v, int slot) {
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x % 32 == 0)
            warp_sums[warp][slot] = v;
    };
#pragma unroll
    for (int j = 0; j < HEAD_COUT; j++)
    {
#pragma unroll
        for (int k = 0; k < 8; k++)
            warp_total(my_w[j][k], j * 8 + k);
        warp_total(my_b[j], HEAD_COUT * 8 + j);
    }
    warp_total(my_loss, HEAD_COUT * 8 + HEAD_COUT);
    __syncthreads();
    constexpr int GROUP_WARPS = HEAD_LANES / 32;
    for (int i = threadIdx.x; i < HEAD_VALUES; i += HEAD_TILE)
    {
        const bool weight = i < HEAD_COUT * HEAD_CIN, loss = i == HEAD_GRADS;
        const int j = i / HEAD_CIN, k = i % HEAD_CIN;
        const int slot = weight ? j * 8 + k % 8 : HEAD_COUT * 8 + (loss ? HEAD_COUT : i - HEAD_COUT * HEAD_CIN);
        const int first = weight ? (k / 8) * GROUP_WARPS : 0, n = loss ? HEAD_TILE / 32 : GROUP_WARPS; // biases: the first group's
        float s = 0.0f;
        for (int w = 0; w < n; w++)
            s += warp_sums[first + w][slot];
        partial[(size_t)blockIdx.x * HEAD_VALUES + i] = s;
    }
}

// The head's gradients and the loss: sums over blocks of head_back_kernel's partials in a fixed
// order (eight threads per value take every eighth block, then their sums are added).
constexpr int SUM_PARTS = 8;
__global__ void __launch_bounds__(32 * SUM_PARTS) head_sums_kernel(const float *partial, int blocks, float *grads, float *loss)
{
    __shared__ float part[SUM_PARTS][32];
    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    const int i = blockIdx.x * 32 + threadIdx.x;
    float s = 0.0f;
    if (i < HEAD_VALUES)
#pragma unroll 4
        for (int b = threadIdx.y; b < blocks; b += SUM_PARTS)
            s += partial[(size_t)b * HEAD_VALUES + i];
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y != 0 || i >= HEAD_VALUES)
        return;
    float total = 0.0f;
#pragma unroll
    for (int k = 0; k < SUM_PARTS; k++)
        total += part[k][threadIdx.x];
    *(i < HEAD_GRADS ? grads + i : loss) = total;
}

// Adam on f32 parameters (bias-corrected; beta1 0.9, beta2 0.999, eps 1e-8)
__global__ void adam_kernel(float *w, const float *g, float *m, float *v, size_t n, float lr, float c1, float c2)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float gi = g[i];
    const float mi = 0.9f * m[i] + 0.1f * gi, vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
}

unsigned grid_for(size_t work) { return (unsigned)std::max<size_t>(1, std::min<size_t>((work + 255) / 256, 152 * 8)); }

// grid of the elementwise kernels over `rows` half-resolution rows of all planes
dim3 rows_grid(int rows) { return dim3((unsigned)std::max(1, std::min((rows + EW_Y - 1) / EW_Y, 152 * 8))); }

constexpr int HEAD_BLOCKS = 152 * 2; // of head_back_kernel: two per SM
} // namespace

struct isti_flownet
{
    int device = 0;
    // parameters: f32 [w_0 b_0 w_1 b_1 ... w_9 b_9 head_w head_b], grads and Adam moments alike
    size_t n_params = 0;
    size_t w_off[N_CONV + 1] = {}, b_off[N_CONV + 1] = {};
    float *params = nullptr, *grads = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    int adam_step = 0;
    // packed bf16 operand images (forward and data-gradient) per layer
    size_t pk_off[N_CONV] = {}, pkt_off[N_CONV] = {};
    bf16 *packs = nullptr;
    int32_t *status = nullptr;
    float *loss = nullptr;     // device scalar of the last training step
    // activation / gradient arena for the current shape
    int n = 0, h = 0, w = 0;
    void *arena = nullptr;
    size_t arena_bytes = 0;
};

namespace
{
// activations and gradients of one shape, carved from the arena
struct Buffers
{
    bf16 *e1, *q1, *e2, *q2, *e3, *q3, *e4, *p3, *s3, *d3, *p2, *s2, *d2, *p1, *s1, *d1;
    bf16 *g_d1, *g_s1, *g_p1, *g_d2, *g_s2, *g_p2, *g_d3, *g_s3, *g_p3, *g_e4, *g_q3, *g_e3, *g_q2, *g_e2, *g_q1, *g_e1;
    float *flow, *partial, *wscratch;
    size_t wscratch_bytes;
};

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

// Lays out (or, with base == nullptr, measures) the buffers of an n x h x w input.
size_t layout(Buffers &b, char *base, int n, int h, int w)
{
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += align256(bytes);
        return p;
    };
    const size_t p1 = (size_t)n * h * w, p2 = p1 / 4, p3 = p1 / 16, p4 = p1 / 64;
    auto t = [&](size_t pix, int c) { return reinterpret_cast<bf16 *>(take(pix * c * 2)); };
    b.e1 = t(p1, 32), b.q1 = t(p2, 32), b.e2 = t(p2, 64), b.q2 = t(p3, 64), b.e3 = t(p3, 96), b.q3 = t(p4, 96), b.e4 = t(p4, 128);
    b.p3 = t(p4, 96), b.s3 = t(p3, 96), b.d3 = t(p3, 96), b.p2 = t(p3, 64), b.s2 = t(p2, 64), b.d2 = t(p2, 64), b.p1 = t(p2, 32);
    b.s1 = t(p1, 32), b.d1 = t(p1, 32);
    b.g_d1 = t(p1, 32), b.g_s1 = t(p1, 32), b.g_p1 = t(p2, 32), b.g_d2 = t(p2, 64), b.g_s2 = t(p2, 64), b.g_p2 = t(p3, 64);
    b.g_d3 = t(p3, 96), b.g_s3 = t(p3, 96), b.g_p3 = t(p4, 96), b.g_e4 = t(p4, 128), b.g_q3 = t(p4, 96), b.g_e3 = t(p3, 96);
    b.g_q2 = t(p3, 64), b.g_e2 = t(p2, 64), b.g_q1 = t(p2, 32), b.g_e1 = t(p1, 32);
    b.flow = reinterpret_cast<float *>(take(p1 * 4 * sizeof(float)));
    b.partial = reinterpret_cast<float *>(take((size_t)HEAD_BLOCKS * HEAD_VALUES * sizeof(float)));
    size_t ws = 0;
    const int hs[N_CONV] = {h, h / 2, h / 4, h / 8, h / 8, h / 4, h / 4, h / 2, h / 2, h};
    const int wsz[N_CONV] = {w, w / 2, w / 4, w / 8, w / 8, w / 4, w / 4, w / 2, w / 2, w};
    for (int l = 0; l < N_CONV; l++)
        ws = std::max(ws, isti_unet::wgrad_scratch(LAYERS[l].taps, n, hs[l], wsz[l], LAYERS[l].cin, LAYERS[l].cout));
    b.wscratch_bytes = ws;
    b.wscratch = reinterpret_cast<float *>(take(ws));
    return off;
}

isti_status ensure_arena(isti_flownet *net, int n, int h, int w, Buffers &b)
{
    Buffers tmp{};
    const size_t need = layout(tmp, nullptr, n, h, w);
    if (need > net->arena_bytes)
    {
        if (net->arena)
            cudaFree(net->arena);
        net->arena = nullptr;
        net->arena_bytes = 0;
        const cudaError_t e = cudaMalloc(&net->arena, need);
        if (e != cudaSuccess)
            return e == cudaErrorMemoryAllocation ? isti::set_error(ISTI_ERR_OOM, "flownet: activation arena") : cuda_fail(e, "cudaMalloc");
        net->arena_bytes = need;
    }
    net->n = n;
    net->h = h;
    net->w = w;
    layout(b, static_cast<char *>(net->arena), n, h, w);
    return ISTI_OK;
}

isti_status repack(isti_flownet *net, cudaStream_t s)
{
    for (int l = 0; l < N_CONV; l++)
    {
        const LayerDef &d = LAYERS[l];
        isti_status st = isti_unet::pack_launch(d.taps, net->params + net->w_off[l], d.cin, d.cout, 0, net->packs + net->pk_off[l], s);
        if (st == ISTI_OK && l > 0) // the first layer's data gradient is never needed
            st = isti_unet::pack_launch(d.taps, net->params + net->w_off[l], d.cin, d.cout, 1, net->packs + net->pkt_off[l], s);
        if (st != ISTI_OK)
            return st;
    }
    return ISTI_OK;
}

isti_status conv(isti_flownet *net, int l, const bf16 *x, int n, int h, int w, const bf16 *mask, bf16 *out, cudaStream_t s, bool pdl = false,
                 const isti_unet::ConvHead *head = nullptr, bool *head_fused = nullptr)
{
    const LayerDef &d = LAYERS[l];
    // every tensor but the network's input (NHWC) is in planes
    return isti_unet::conv_launch(d.taps, x, n, h, w, d.cin, net->packs + net->pk_off[l], net->params + net->b_off[l], mask, d.relu, out, d.cout,
                                  net->status, s, l == 0 ? isti_unet::OUT_PLANES : isti_unet::IN_PLANES | isti_unet::OUT_PLANES, pdl, head,
                                  head_fused);
}

// data gradient of layer l: g_in = conv(g_out, W^T flipped), masked by (mask > 0) when given
isti_status dgrad(isti_flownet *net, int l, const bf16 *g_out, int n, int h, int w, const bf16 *mask, bf16 *g_in, cudaStream_t s)
{
    const LayerDef &d = LAYERS[l];
    return isti_unet::conv_launch(d.taps, g_out, n, h, w, d.cout, net->packs + net->pkt_off[l], nullptr, mask, 0, g_in, d.cin, net->status, s,
                                  isti_unet::IN_PLANES | isti_unet::OUT_PLANES, true);
}

isti_status wgrad(isti_flownet *net, int l, const bf16 *g_out, const bf16 *x, int n, int h, int w, Buffers &b, cudaStream_t s)
{
    const LayerDef &d = LAYERS[l];
    return isti_unet::wgrad_launch(d.taps, g_out, x, n, h, w, d.cin, d.cout, net->grads + net->w_off[l], net->grads + net->b_off[l], 0, b.wscratch,
                                   b.wscratch_bytes, net->status, s,
                                   l == 0 ? isti_unet::OUT_PLANES : isti_unet::IN_PLANES | isti_unet::OUT_PLANES, true);
}

#define ISTI_TRY(x)                                                                                                                             \
    do                                                                                                                                          \
    {                                                                                                                                           \
        const isti_status st_ = (x);                                                                                                            \
        if (st_ != ISTI_OK)                                                                                                                     \
            return st_;                                                                                                                         \
    } while (0)

// Every launch but the first is a programmatic dependent of the one before (each kernel sets up while
// its predecessor finishes).  Weights and biases are read before a kernel's wait, so the first one
// follows in full order what may have written them (Adam, the packing kernels, the caller), whatever
// dependents were launched in between; the others start after it has (learned call at 1080p: 439 us,
// 436 without that order).
isti_status forward(isti_flownet *net, const bf16 *x0, int n, int h, int w, Buffers &b, float *flow, __half *flow16, cudaStream_t s)
{
    constexpr bool pdl = true;
    const int h2 = h / 2, w2 = w / 2, h4 = h / 4, w4 = w / 4, h8 = h / 8, w8 = w / 8;
    const dim3 blk(EW_X, EW_Y);
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t x) {
        if (e == cudaSuccess)
            e = x;
        return e == cudaSuccess;
    };
    ISTI_TRY(conv(net, 0, x0, n, h, w, nullptr, b.e1, s));
    ok(isti::launch_after(pdl, blocksum_kernel, rows_grid(n * 4 * h2), blk, 0, s, (const bf16 *)b.e1, (uint32_t)(n * 4), (uint32_t)h2, (uint32_t)w2, 0.25f, b.q1));
    ISTI_TRY(conv(net, 1, b.q1, n, h2, w2, nullptr, b.e2, s, pdl));
    ok(isti::launch_after(pdl, blocksum_kernel, rows_grid(n * 8 * h4), blk, 0, s, (const bf16 *)b.e2, (uint32_t)(n * 8), (uint32_t)h4, (uint32_t)w4, 0.25f, b.q2));
    ISTI_TRY(conv(net, 2, b.q2, n, h4, w4, nullptr, b.e3, s, pdl));
    ok(isti::launch_after(pdl, blocksum_kernel, rows_grid(n * 12 * h8), blk, 0, s, (const bf16 *)b.e3, (uint32_t)(n * 12), (uint32_t)h8, (uint32_t)w8, 0.25f, b.q3));
    ISTI_TRY(conv(net, 3, b.q3, n, h8, w8, nullptr, b.e4, s, pdl));
    ISTI_TRY(conv(net, 4, b.e4, n, h8, w8, nullptr, b.p3, s, pdl));
    ok(isti::launch_after(pdl, upadd_kernel, rows_grid(n * 12 * h8), blk, 0, s, (const bf16 *)b.p3, (const bf16 *)b.e3, (uint32_t)(n * 12), (uint32_t)h8, (uint32_t)w8,
                     b.s3));
    ISTI_TRY(conv(net, 5, b.s3, n, h4, w4, nullptr, b.d3, s, pdl));
    ISTI_TRY(conv(net, 6, b.d3, n, h4, w4, nullptr, b.p2, s, pdl));
    ok(isti::launch_after(pdl, upadd_kernel, rows_grid(n * 8 * h4), blk, 0, s, (const bf16 *)b.p2, (const bf16 *)b.e2, (uint32_t)(n * 8), (uint32_t)h4, (uint32_t)w4,
                     b.s2));
    ISTI_TRY(conv(net, 7, b.s2, n, h2, w2, nullptr, b.d2, s, pdl));
    ISTI_TRY(conv(net, 8, b.d2, n, h2, w2, nullptr, b.p1, s, pdl));
    ok(isti::launch_after(pdl, upadd_kernel, rows_grid(n * 4 * h2), blk, 0, s, (const bf16 *)b.p1, (const bf16 *)b.e1, (uint32_t)(n * 4), (uint32_t)h2, (uint32_t)w2,
                     b.s1));
    // inference: the 1x1 head in d1's epilogue where the row-tile kernel runs d1 (d1 itself is
    // then not stored), else its own kernel
    const isti_unet::ConvHead head{net->params + net->w_off[N_CONV], net->params + net->b_off[N_CONV], flow, flow16};
    bool fused = false;
    ISTI_TRY(conv(net, 9, b.s1, n, h, w, nullptr, b.d1, s, pdl, flow || flow16 ? &head : nullptr, &fused));
    if ((flow || flow16) && !fused)
        ok(isti::launch_after(pdl, head_kernel, dim3(grid_for((size_t)n * h * w)), dim3(256), 0, s, (const bf16 *)b.d1, (size_t)n * h * w, (size_t)h * w,
                         (const float *)(net->params + net->w_off[N_CONV]), (const float *)(net->params + net->b_off[N_CONV]), flow, flow16));
    if (e == cudaSuccess)
        e = cudaGetLastError();
    return e == cudaSuccess ? ISTI_OK : cuda_fail(e, "flownet forward");
}

isti_status backward(isti_flownet *net, const bf16 *x0, const float *label, int n, int h, int w, Buffers &b, cudaStream_t s)
{
    const int h2 = h / 2, w2 = w / 2, h4 = h / 4, w4 = w / 4, h8 = h / 8, w8 = w / 8;
    const size_t npix = (size_t)n * h * w;
    const int blocks = (int)std::min<size_t>(HEAD_BLOCKS, (npix + HEAD_TILE - 1) / HEAD_TILE);
    cudaError_t e = cudaSuccess;
    // every launch a programmatic dependent of the one before
    auto launch = [&](auto kernel, dim3 grid, dim3 block, auto... args) {
        const cudaError_t x = isti::launch_after(true, kernel, grid, block, 0, s, args...);
        if (e == cudaSuccess)
            e = x;
    };
    const dim3 blk(EW_X, EW_Y);
    launch(head_back_kernel, dim3(blocks), dim3(HEAD_TILE), b.d1, npix, (size_t)h * w, net->params + net->w_off[N_CONV],
           net->params + net->b_off[N_CONV], label, 1.0f / (float)npix, b.g_d1, b.partial);
    launch(head_sums_kernel, dim3((HEAD_VALUES + 31) / 32), dim3(32, SUM_PARTS), b.partial, blocks, net->grads + net->w_off[N_CONV], net->loss);
    // level 1 decoder
    ISTI_TRY(wgrad(net, 9, b.g_d1, b.s1, n, h, w, b, s));
    ISTI_TRY(dgrad(net, 9, b.g_d1, n, h, w, nullptr, b.g_s1, s));
    launch(blocksum_kernel, rows_grid(n * 4 * h2), blk, b.g_s1, n * 4, h2, w2, 1.0f, b.g_p1);
    ISTI_TRY(wgrad(net, 8, b.g_p1, b.d2, n, h2, w2, b, s));
    ISTI_TRY(dgrad(net, 8, b.g_p1, n, h2, w2, b.d2, b.g_d2, s));
    // level 2 decoder
    ISTI_TRY(wgrad(net, 7, b.g_d2, b.s2, n, h2, w2, b, s));
    ISTI_TRY(dgrad(net, 7, b.g_d2, n, h2, w2, nullptr, b.g_s2, s));
    launch(blocksum_kernel, rows_grid(n * 8 * h4), blk, b.g_s2, n * 8, h4, w4, 1.0f, b.g_p2);
    ISTI_TRY(wgrad(net, 6, b.g_p2, b.d3, n, h4, w4, b, s));
    ISTI_TRY(dgrad(net, 6, b.g_p2, n, h4, w4, b.d3, b.g_d3, s));
    // level 3 decoder
    ISTI_TRY(wgrad(net, 5, b.g_d3, b.s3, n, h4, w4, b, s));
    ISTI_TRY(dgrad(net, 5, b.g_d3, n, h4, w4, nullptr, b.g_s3, s));
    launch(blocksum_kernel, rows_grid(n * 12 * h8), blk, b.g_s3, n * 12, h8, w8, 1.0f, b.g_p3);
    ISTI_TRY(wgrad(net, 4, b.g_p3, b.e4, n, h8, w8, b, s));
    ISTI_TRY(dgrad(net, 4, b.g_p3, n, h8, w8, b.e4, b.g_e4, s));
    // bottleneck and encoder
    ISTI_TRY(wgrad(net, 3, b.g_e4, b.q3, n, h8, w8, b, s));
    ISTI_TRY(dgrad(net, 3, b.g_e4, n, h8, w8, nullptr, b.g_q3, s));
    launch(poolback_kernel, rows_grid(n * 12 * h8), blk, b.g_s3, b.g_q3, b.e3, n * 12, h8, w8, b.g_e3);
    ISTI_TRY(wgrad(net, 2, b.g_e3, b.q2, n, h4, w4, b, s));
    ISTI_TRY(dgrad(net, 2, b.g_e3, n, h4, w4, nullptr, b.g_q2, s));
    launch(poolback_kernel, rows_grid(n * 8 * h4), blk, b.g_s2, b.g_q2, b.e2, n * 8, h4, w4, b.g_e2);
    ISTI_TRY(wgrad(net, 1, b.g_e2, b.q1, n, h2, w2, b, s));
    ISTI_TRY(dgrad(net, 1, b.g_e2, n, h2, w2, nullptr, b.g_q1, s));
    launch(poolback_kernel, rows_grid(n * 4 * h2), blk, b.g_s1, b.g_q1, b.e1, n * 4, h2, w2, b.g_e1);
    ISTI_TRY(wgrad(net, 0, b.g_e1, x0, n, h, w, b, s));
    if (e == cudaSuccess)
        e = cudaGetLastError();
    return e == cudaSuccess ? ISTI_OK : cuda_fail(e, "flownet backward");
}

isti_status check_shape(const void *x, int n, int h, int w)
{
    if (!x || n < 1 || h < 8 || w < 16 || h % 8 || w % 8)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "flownet: input must be n x h x w x 16 with h, w multiples of 8 (w >= 16)");
    return ISTI_OK;
}
} // namespace

extern "C" {

int32_t isti_flownet_input_channels(void) { return IN_CH; }
int32_t isti_flownet_output_channels(void) { return HEAD_COUT; }
int32_t isti_flownet_num_layers(void) { return N_CONV + 1; }

isti_status isti_flownet_layer(int32_t index, int32_t *taps, int32_t *cin, int32_t *cout, int32_t *relu)
{
    if (index < 0 || index > N_CONV)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "flownet: layer index out of range");
    const LayerDef d = index < N_CONV ? LAYERS[index] : LayerDef{1, HEAD_CIN, HEAD_COUT, 0};
    if (taps)
        *taps = d.taps;
    if (cin)
        *cin = d.cin;
    if (cout)
        *cout = d.cout;
    if (relu)
        *relu = d.relu;
    return ISTI_OK;
}

isti_status isti_flownet_create(isti_flownet **out, uint64_t seed)
{
    if (!out)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "out is NULL");
    isti_flownet *net = new (std::nothrow) isti_flownet();
    if (!net)
        return isti::set_error(ISTI_ERR_OOM, "host allocation failed");
    cudaGetDevice(&net->device);
    size_t off = 0, pk = 0;
    for (int l = 0; l <= N_CONV; l++)
    {
        const LayerDef d = l < N_CONV ? LAYERS[l] : LayerDef{1, HEAD_CIN, HEAD_COUT, 0};
        net->w_off[l] = off;
        off += (size_t)d.taps * d.cin * d.cout;
        net->b_off[l] = off;
        off += (size_t)d.cout;
        off = (off + 3) / 4 * 4; // 16-byte aligned tensors
        if (l < N_CONV)
        {
            net->pk_off[l] = pk;
            pk += (size_t)d.taps * d.cin * d.cout;
            net->pkt_off[l] = pk;
            pk += (size_t)d.taps * d.cin * d.cout;
        }
    }
    net->n_params = off;
    // He-normal weights, zero biases (host PRNG: reproducible for a seed)
    std::vector<float> host(off, 0.0f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l <= N_CONV; l++)
    {
        const LayerDef d = l < N_CONV ? LAYERS[l] : LayerDef{1, HEAD_CIN, HEAD_COUT, 0};
        const float sd = l < N_CONV ? std::sqrt(2.0f / (float)(d.taps * d.cin)) : 0.01f;
        std::normal_distribution<float> nd(0.0f, sd);
        for (size_t i = 0; i < (size_t)d.taps * d.cin * d.cout; i++)
            host[net->w_off[l] + i] = nd(rng);
    }
    cudaError_t e = cudaMalloc(&net->params, off * sizeof(float) * 4);
    if (e == cudaSuccess)
        e = cudaMalloc(&net->packs, pk * sizeof(bf16));
    if (e == cudaSuccess)
        e = cudaMalloc(&net->status, 256);
    if (e != cudaSuccess)
    {
        isti_flownet_destroy(net);
        return isti::set_error(ISTI_ERR_OOM, "flownet: parameter allocation");
    }
    net->grads = net->params + off;
    net->adam_m = net->grads + off;
    net->adam_v = net->adam_m + off;
    net->loss = reinterpret_cast<float *>(net->status + 32);
    cudaMemset(net->params, 0, off * sizeof(float) * 4);
    cudaMemset(net->status, 0, 256);
    cudaMemcpy(net->params, host.data(), off * sizeof(float), cudaMemcpyHostToDevice);
    isti_status st = repack(net, nullptr);
    if (st == ISTI_OK)
    {
        e = cudaDeviceSynchronize();
        if (e != cudaSuccess)
            st = cuda_fail(e, "flownet init");
    }
    if (st != ISTI_OK)
    {
        isti_flownet_destroy(net);
        return st;
    }
    *out = net;
    return ISTI_OK;
}

isti_status isti_flownet_destroy(isti_flownet *net)
{
    if (!net)
        return ISTI_OK;
    cudaFree(net->params);
    cudaFree(net->packs);
    cudaFree(net->status);
    cudaFree(net->arena);
    delete net;
    return ISTI_OK;
}

isti_status isti_flownet_tensors(isti_flownet *net, float **params, float **grads, size_t *count)
{
    if (!net)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "flownet is NULL");
    if (params)
        *params = net->params;
    if (grads)
        *grads = net->grads;
    if (count)
        *count = net->n_params;
    return ISTI_OK;
}

isti_status isti_flownet_param_offsets(const isti_flownet *net, int32_t layer, size_t *w_off, size_t *b_off)
{
    if (!net || layer < 0 || layer > N_CONV)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "flownet: bad layer");
    if (w_off)
        *w_off = net->w_off[layer];
    if (b_off)
        *b_off = net->b_off[layer];
    return ISTI_OK;
}

isti_status isti_flownet_sync_params(isti_flownet *net, void *stream)
{
    if (!net)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "flownet is NULL");
    return repack(net, static_cast<cudaStream_t>(stream));
}

isti_status isti_flownet_forward(isti_flownet *net, const void *x, int32_t n, int32_t h, int32_t w, float *flow, void *flow_f16, void *stream)
{
    if (!net)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "flownet is NULL");
    ISTI_TRY(check_shape(x, n, h, w));
    Buffers b{};
    ISTI_TRY(ensure_arena(net, n, h, w, b));
    return forward(net, static_cast<const bf16 *>(x), n, h, w, b, flow, static_cast<__half *>(flow_f16), static_cast<cudaStream_t>(stream));
}

isti_status isti_flownet_backward(isti_flownet *net, const void *x, const float *label, int32_t n, int32_t h, int32_t w, void *stream)
{
    if (!net || !label)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "NULL argument");
    ISTI_TRY(check_shape(x, n, h, w));
    Buffers b{};
    ISTI_TRY(ensure_arena(net, n, h, w, b));
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    ISTI_TRY(forward(net, static_cast<const bf16 *>(x), n, h, w, b, nullptr, nullptr, s));
    return backward(net, static_cast<const bf16 *>(x), label, n, h, w, b, s);
}

isti_status isti_flownet_adam(isti_flownet *net, float lr, void *stream)
{
    if (!net)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "flownet is NULL");
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    net->adam_step++;
    const float c1 = 1.0f - std::pow(0.9f, (float)net->adam_step), c2 = 1.0f - std::pow(0.999f, (float)net->adam_step);
    adam_kernel<<<(unsigned)((net->n_params + 255) / 256), 256, 0, s>>>(net->params, net->grads, net->adam_m, net->adam_v, net->n_params, lr, c1,
                                                                        c2);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return cuda_fail(e, "flownet adam");
    return repack(net, s);
}

isti_status isti_flownet_loss(isti_flownet *net, float **loss_device)
{
    if (!net || !loss_device)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "NULL argument");
    *loss_device = net->loss;
    return ISTI_OK;
}

isti_status isti_flownet_device_status(isti_flownet *net, int32_t *status)
{
    if (!net || !status)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "NULL argument");
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess)
        e = cudaMemcpy(status, net->status, sizeof(int32_t), cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? ISTI_OK : cuda_fail(e, "flownet status");
}

} // extern "C"
