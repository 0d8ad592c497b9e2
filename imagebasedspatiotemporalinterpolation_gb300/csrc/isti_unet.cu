// Host side of the learned flow initialiser: tensor maps and launches of the tcgen05
// convolution kernels (isti_unet_conv.cuh) and the C ABI of include/isti_unet.h.
#include "isti_unet.h"
#include "isti_unet_conv.cuh"
#include "isti_unet_ops.h"
#include "host/isti_error.hpp"

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

namespace
{
using namespace isti_unet;

isti_status cuda_fail(cudaError_t e, const char *what) { return isti::set_error(ISTI_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e)); }

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                   const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled()
{
    static EncodeTiledFn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (EncodeTiledFn) nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}

// 4-D map over an NHWC bf16 tensor: dims (c, w, h, n), box {8 channels, 16 x, 8 y, 1}.
isti_status nhwc_map(CUtensorMap &m, const void *base, int n, int h, int w, int c)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc)
        return isti::set_error(ISTI_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
    if (((uintptr_t)base & 15u) || c % 8)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "NHWC tensor: base 16-byte aligned, channels a multiple of 8");
    const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint64_t strides[3] = {(cuuint64_t)c * 2u, (cuuint64_t)w * c * 2u, (cuuint64_t)h * w * c * 2u};
    const cuuint32_t box[4] = {8, (cuuint32_t)TILE_W, (cuuint32_t)TILE_H, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    if (enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "cuTensorMapEncodeTiled rejected an NHWC tensor");
    return ISTI_OK;
}

// Map of a box of `px` x `rows` pixels x `groups` channel groups of 8.  NHWC: 5-D over (8, w, h,
// c / 8, n); planes: 4-D over (2 w, h, c / 8, n) 64-bit elements, so that a box row is one run of
// px * 16 bytes.  Either lands the groups one after another, pixels of 16 bytes within.
isti_status box_map(CUtensorMap &m, const void *base, bool planes, int n, int h, int w, int c, int px, int rows, int groups)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc)
        return isti::set_error(ISTI_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
    if (((uintptr_t)base & 15u) || c % 8)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "activation tensor: base 16-byte aligned, channels a multiple of 8");
    const cuuint64_t W = (cuuint64_t)w, H = (cuuint64_t)h, G = (cuuint64_t)(c / 8), N = (cuuint64_t)n;
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r;
    if (planes)
    {
        const cuuint64_t dims[4] = {2 * W, H, G, N}, strides[3] = {16 * W, 16 * W * H, 16 * W * H * G};
        const cuuint32_t box[4] = {2 * (cuuint32_t)px, (cuuint32_t)rows, (cuuint32_t)groups, 1};
        r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    else
    {
        const cuuint64_t dims[5] = {8, W, H, G, N}, strides[4] = {16 * G, 16 * G * W, 16u, 16 * G * W * H};
        const cuuint32_t box[5] = {8, (cuuint32_t)px, (cuuint32_t)rows, (cuuint32_t)groups, 1};
        r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    return r == CUDA_SUCCESS ? ISTI_OK : isti::set_error(ISTI_ERR_INVALID_ARG, "cuTensorMapEncodeTiled rejected an activation tensor");
}

int sm_count()
{
    static int n[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
        return 152;
    if (!n[dev & 63])
    {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        n[dev & 63] = v > 0 ? v : 152;
    }
    return n[dev & 63];
}

// A kernel's dynamic shared-memory limit, raised once per kernel and device to the largest
// size asked (keyed by the kernel's address: instances of one template share a type).
template <class K>
cudaError_t smem_limit(K kernel, size_t bytes)
{
    struct Entry
    {
        const void *fn;
        int dev;
        size_t bytes;
    };
    static std::mutex mu;
    static std::vector<Entry> set;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || bytes <= 48 * 1024)
        return e;
    std::lock_guard<std::mutex> lock(mu);
    const void *fn = reinterpret_cast<const void *>(kernel);
    for (Entry &x : set)
        if (x.fn == fn && x.dev == dev)
        {
            if (bytes > x.bytes)
            {
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
                if (e == cudaSuccess)
                    x.bytes = bytes;
            }
            return e;
        }
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess)
        set.push_back({fn, dev, bytes});
    return e;
}

int32_t *g_null_status = nullptr; // device word for callers that pass no status

isti_status status_word(int32_t *&status)
{
    if (status)
        return ISTI_OK;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (!g_null_status)
    {
        cudaError_t e = cudaMalloc(&g_null_status, 256);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaMalloc(status word)");
        cudaMemset(g_null_status, 0, 256);
    }
    status = g_null_status;
    return ISTI_OK;
}
} // namespace

namespace isti_unet
{
// Launch of conv_kernel<taps> (shared with the network code in isti_flownet.cu).
isti_status conv_launch(int taps, const void *x, int n, int h, int w, int cin, const void *wpack, const float *bias, const void *mask, int relu,
                        void *out, int cout, int32_t *status, cudaStream_t stream, int planes, bool pdl, const ConvHead *head, bool *head_fused)
{
    if (head_fused)
        *head_fused = false;
    if (head && (!head->w || !head->b || (!head->flow && !head->flow16) || ((uintptr_t)head->flow & 15u) || ((uintptr_t)head->flow16 & 7u)))
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_conv: fused head needs weights, bias and an aligned output");
    if ((taps != 9 && taps != 1) || n < 1 || h < 1 || w < 1 || cin % 16 || cout % 16 || cout < 16 || cout > 256 || !x || !wpack || !out)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_conv: bad shape or NULL buffer");
    if (((uintptr_t)out & 15u) || ((uintptr_t)mask & 15u) || ((uintptr_t)wpack & 15u))
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_conv: buffers must be 16-byte aligned");
    isti_status st = status_word(status);
    if (st != ISTI_OK)
        return st;
    ConvParams p{};
    p.wpack = static_cast<const __nv_bfloat16 *>(wpack);
    p.bias = bias;
    p.mask = static_cast<const __nv_bfloat16 *>(mask);
    p.out = static_cast<__nv_bfloat16 *>(out);
    p.status = status;
    p.w = w;
    p.h = h;
    p.b = n;
    p.cin = cin;
    p.cout = cout;
    p.ck = cin % 32 == 0 ? 32 : 16;
    p.in_planes = (planes & IN_PLANES) != 0;
    p.out_planes = (planes & OUT_PLANES) != 0;
    p.halo = p.in_planes ? ROW_M : ROW_HALO;
    p.seg_out = p.halo - 2;
    p.tile_shift = 4;
    // 1x1 layers in planes: an image is one row of pixels, a tile 128 of them
    if (taps == 1 && p.in_planes && p.out_planes && (size_t)h * w <= (size_t)INT32_MAX / 2)
    {
        p.tile_shift = 7;
        p.w = w = h * w;
        p.h = h = 1;
    }
    const int tile_w = 1 << p.tile_shift, tile_h = TILE_M / tile_w;
    p.tiles_x = (w + tile_w - 1) / tile_w;
    p.tiles_y = (h + tile_h - 1) / tile_h;
    p.n_tiles = n * p.tiles_x * p.tiles_y;
    p.relu = relu;
    CUtensorMap xmap;
    // wide, thin 3x3 layers: row-tile kernel with a loaded-once halo and resident weights
    const uint32_t w_bytes = 9u * (uint32_t)cin * cout * 2u;
    if (taps == 9 && w >= ROW_M && w_bytes <= 96u * 1024u && box_map(xmap, x, p.in_planes, n, h, w, cin, p.halo, 3, p.ck / 8) == ISTI_OK)
    {
        const size_t w_region = (w_bytes + 1023) / 1024 * 1024, sb = row_stage_bytes(p.ck, p.halo), tail = 16 * 8 + 16;
        int per_sm = 2;
        size_t stages = w_region + 2 * sb + 2 * 16 + tail <= 100 * 1024 ? (100 * 1024 - w_region - tail) / (sb + 16) : 0;
        if (stages < 2)
        {
            per_sm = 1;
            stages = (SMEM_BUDGET - w_region - tail) / (sb + 16);
        }
        p.stages = (int)std::min<size_t>(8, stages);
        if (p.stages >= 2)
        {
            if (head)
            {
                p.head_w = head->w;
                p.head_b = head->b;
                p.head_flow = head->flow;
                p.head_flow16 = static_cast<__half *>(head->flow16);
            }
            const size_t smem = w_region + (size_t)p.stages * sb + (2 * p.stages + 6) * 8 + 16;
            const int units = n * h * ((w + p.seg_out - 1) / p.seg_out);
            const int grid = std::min(units, sm_count() * per_sm);
            cudaError_t e = smem_limit(row_conv_kernel<0>, smem);
            if (e == cudaSuccess)
                e = isti::launch_after(pdl, row_conv_kernel<0>, dim3((unsigned)grid), dim3(PCONV_THREADS), smem, stream, p, xmap);
            if (e == cudaSuccess && head && head_fused)
                *head_fused = true;
            return e == cudaSuccess ? ISTI_OK : cuda_fail(e, "isti_unet_conv launch");
        }
    }
    st = box_map(xmap, x, p.in_planes, n, h, w, cin, tile_w, tile_h, p.ck / 8);
    p.chunked_map = !p.in_planes && st == ISTI_OK;
    if (st != ISTI_OK && (p.in_planes || (st = nhwc_map(xmap, x, n, h, w, cin)) != ISTI_OK))
        return st;
    // ring: about 100 KB, so that two CTAs share an SM; the ring runs across tiles
    const uint32_t sb = conv_stage_bytes(p.ck, cout);
    p.stages = (int)std::min<size_t>(16, std::max<size_t>(2, (100 * 1024) / sb));
    const size_t smem = (size_t)p.stages * sb + (2 * p.stages + 5) * 8 + 16;
    if (smem > SMEM_BUDGET)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_conv: stage does not fit in shared memory");
    const uint32_t ncols = 2 * tmem_cols(cout);
    const int per_sm = std::max(1, std::min(2, (int)(512 / ncols)));
    const int grid = std::min(p.n_tiles, sm_count() * per_sm);
    cudaError_t e;
    if (taps == 9)
    {
        e = smem_limit(conv_kernel<9>, smem);
        if (e == cudaSuccess)
            e = isti::launch_after(pdl, conv_kernel<9>, dim3((unsigned)grid), dim3(PCONV_THREADS), smem, stream, p, xmap);
    }
    else
    {
        e = smem_limit(conv_kernel<1>, smem);
        if (e == cudaSuccess)
            e = isti::launch_after(pdl, conv_kernel<1>, dim3((unsigned)grid), dim3(PCONV_THREADS), smem, stream, p, xmap);
    }
    if (e == cudaSuccess)
        e = cudaGetLastError();
    return e == cudaSuccess ? ISTI_OK : cuda_fail(e, "isti_unet_conv launch");
}

// Bytes of scratch: every split's partial sums.
size_t wgrad_scratch(int taps, int n, int h, int w, int cin, int cout)
{
    WgradConfig c;
    if ((taps != 9 && taps != 1) || n < 1 || h < 1 || w < 1 || cin < 16 || cout < 16 || !wgrad_config(taps, n, h, w, cin, cout, c))
        return 0;
    return (size_t)c.splits * cout * ((size_t)taps * cin + 1) * sizeof(float);
}

isti_status wgrad_launch(int taps, const void *dy, const void *x, int n, int h, int w, int cin, int cout, float *dw, float *db, int accumulate,
                         void *scratch, size_t scratch_bytes, int32_t *status, cudaStream_t stream, int planes, bool pdl)
{
    if ((taps != 9 && taps != 1) || n < 1 || h < 1 || w < 1 || cin % 16 || cout % 16 || cin < 16 || cin > 256 || cout < 16 || cout > 128 || !dy ||
        !x || !dw || !scratch || (db && cin > 240))
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_wgrad: bad shape or NULL buffer");
    WgradConfig c;
    if (!wgrad_config(taps, n, h, w, cin, cout, c))
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_wgrad: image too large");
    if (scratch_bytes < wgrad_scratch(taps, n, h, w, cin, cout))
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_wgrad: scratch too small");
    isti_status st = status_word(status);
    if (st != ISTI_OK)
        return st;
    WgradParams p{};
    p.partial = static_cast<float *>(scratch);
    p.bpartial = db ? p.partial + (size_t)c.splits * cout * taps * cin : nullptr;
    p.status = status;
    p.w = c.w;
    p.h = c.h;
    p.b = c.n;
    p.cin = cin;
    p.cout = cout;
    p.kseg = c.kseg;
    p.segs = c.segs;
    p.n_units = c.n_units;
    p.units_per_split = c.units_per_split;
    p.box_chunks = c.grid_z == 1 ? cout / 8 : 1;
    p.stages = c.stages;
    p.dy_planes = (planes & OUT_PLANES) != 0;
    p.x_planes = (planes & IN_PLANES) != 0;
    CUtensorMap dymap, xmap;
    if ((st = box_map(dymap, dy, p.dy_planes, c.n, c.h, c.w, cout, c.kseg, 1, p.box_chunks)) != ISTI_OK ||
        (st = box_map(xmap, x, p.x_planes, c.n, c.h, c.w, cin, c.kseg, c.n_dy, cin / 8)) != ISTI_OK)
        return st;
    const dim3 grid((unsigned)c.splits, (unsigned)c.grid_y, (unsigned)c.grid_z);
    using Kernel = void (*)(WgradParams, CUtensorMap, CUtensorMap);
    constexpr Kernel rows3[3] = {wgrad_kernel<9, 3, 1>, wgrad_kernel<9, 3, 2>, wgrad_kernel<9, 3, 3>};
    constexpr Kernel rows1[3] = {wgrad_kernel<9, 1, 1>, wgrad_kernel<9, 1, 2>, wgrad_kernel<9, 1, 3>};
    const Kernel kernel = taps == 1 ? wgrad_kernel<1, 1, 1> : (c.n_dy == 3 ? rows3 : rows1)[c.n_mb - 1];
    cudaError_t e = smem_limit(kernel, c.smem);
    if (e == cudaSuccess)
    {
        e = isti::launch_after(pdl, kernel, grid, dim3(WGRAD_THREADS), c.smem, stream, p, dymap, xmap);
        const int nw = cout * taps * cin;
        if (e == cudaSuccess)
            e = isti::launch_after(pdl, wgrad_reduce_kernel, dim3((unsigned)((nw + (db ? cout : 0) + 31) / 32)), dim3(32, WREDUCE_PARTS), 0, stream,
                              (const float *)p.partial, (const float *)p.bpartial, c.splits, nw, cout, dw, db, accumulate);
    }
    if (e == cudaSuccess)
    {
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? ISTI_OK : cuda_fail(e, "isti_unet_wgrad launch");
}

isti_status pack_launch(int taps, const float *w, int cin, int cout, int transpose, void *wpack, cudaStream_t stream)
{
    if ((taps != 9 && taps != 1) || cin % 16 || cout % 16 || !w || !wpack)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_unet_pack: bad shape or NULL buffer");
    const int n = taps * cin * cout;
    pack_kernel<<<(n + 255) / 256, 256, 0, stream>>>(w, taps, cin, cout, transpose, static_cast<__nv_bfloat16 *>(wpack));
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ISTI_OK : cuda_fail(e, "isti_unet_pack launch");
}
} // namespace isti_unet

extern "C" {

size_t isti_unet_packed_bytes(int32_t taps, int32_t cin, int32_t cout) { return (size_t)taps * cin * cout * 2u; }

isti_status isti_unet_pack(int32_t taps, const float *w, int32_t cin, int32_t cout, int32_t transpose, void *wpack, void *stream)
{
    return isti_unet::pack_launch(taps, w, cin, cout, transpose, wpack, static_cast<cudaStream_t>(stream));
}

isti_status isti_unet_conv(int32_t taps, const void *x, int32_t n, int32_t h, int32_t w, int32_t cin, const void *wpack, const float *bias,
                           const void *mask, int32_t relu, void *out, int32_t cout, int32_t *status, void *stream)
{
    return isti_unet::conv_launch(taps, x, n, h, w, cin, wpack, bias, mask, relu, out, cout, status, static_cast<cudaStream_t>(stream));
}

size_t isti_unet_wgrad_scratch_bytes(int32_t taps, int32_t n, int32_t h, int32_t w, int32_t cin, int32_t cout)
{
    return isti_unet::wgrad_scratch(taps, n, h, w, cin, cout);
}

isti_status isti_unet_wgrad(int32_t taps, const void *dy, const void *x, int32_t n, int32_t h, int32_t w, int32_t cin, int32_t cout,
                            float *dw, int32_t accumulate, void *scratch, size_t scratch_bytes, int32_t *status, void *stream)
{
    return isti_unet::wgrad_launch(taps, dy, x, n, h, w, cin, cout, dw, nullptr, accumulate, scratch, scratch_bytes, status,
                                   static_cast<cudaStream_t>(stream));
}

} // extern "C"
