// PSNR and SSIM of RGBA8 image pairs (include/isti_metrics.h): the metrics of
// the reference's evaluation script (scripts/eval.py:66-132,
// scripts/loss_utils.py:17-57), as two kernels.
//
// quality_tile_kernel: one block per 32x32 output tile.  For each colour
// channel the tile plus a 5-pixel halo of both images is staged in shared
// memory as floats in [0, 1] (zero outside the image: the reference's zero
// padding), the five moments x, y, x^2, y^2, xy are filtered horizontally
// into shared memory and then vertically per output pixel, and the SSIM
// value is accumulated; the squared error is accumulated exactly in
// integers.  Each block writes its two partial sums.
// quality_final_kernel: one block adds the partial sums in a fixed order.
#include "isti_metrics.h"
#include "host/isti_error.hpp"
#include "isti_device.cuh"
#include "isti_pdl.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

namespace
{
constexpr int TW = 32, TH = 32, R = 5, WIN = 2 * R + 1;
constexpr int SW = TW + 2 * R, SH = TH + 2 * R;
constexpr int THREADS = 256;   // final kernels, FLIP tiles
constexpr int Q_THREADS = 128; // SSIM tiles

struct Gauss
{
    float2 g[WIN]; // each tap twice: the packed operations take a pair
};

// v / 255 for an integer v in 0..255, correctly rounded
__device__ __forceinline__ float byte_to_unit(uint32_t v)
{
    return isti::divided_by<255>((float)v);
}

// Both passes are bound by FMA issue and shared-memory reads, so a thread filters several
// neighbouring outputs from one set of reads (4 along a row, then 8 down a column), and the
// images' moments travel as pairs (x, y), (x^2, y^2) through the packed fma.rn.f32x2.  Rows
// are spread over the lanes in the horizontal pass: the pitches (21 and 17 sixteen-byte words,
// 9 for the single plane) are odd, so their 16-byte accesses meet no bank conflict.
// 1080p: 112 -> 66 us (one output per thread and pass, 32x16 tiles, scalar operations before).
constexpr int Q_PITCH = TW + 2, Q_PITCH1 = TW + 4;
__global__ void __launch_bounds__(Q_THREADS) quality_tile_kernel(const uint32_t *a, const uint32_t *b, int w, int h, double *partials,
                                                                 const __grid_constant__ Gauss gw)
{
    __shared__ __align__(16) float2 xy[SH * SW];
    __shared__ __align__(16) float2 hm[SH * Q_PITCH], hq[SH * Q_PITCH]; // horizontally filtered (x, y) and (x^2, y^2)
    __shared__ __align__(16) float hc[SH * Q_PITCH1];                   // and xy
    constexpr int PER = (SH * SW + Q_THREADS - 1) / Q_THREADS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int x0 = blockIdx.x * TW, y0 = blockIdx.y * TH;

    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    uint32_t pa[PER], pb[PER]; // this thread's staged pixels, read once for the three channels
    uint32_t sq = 0;
#pragma unroll
    for (int i = 0; i < PER; i++)
    {
        const int e = tid + i * Q_THREADS, yy = e / SW, xx = e % SW;
        const int gx = x0 + xx - R, gy = y0 + yy - R;
        pa[i] = pb[i] = 0u;
        if (e < SH * SW && gx >= 0 && gx < w && gy >= 0 && gy < h)
        {
            const size_t idx = (size_t)gy * w + gx;
            pa[i] = a[idx];
            pb[i] = b[idx];
            if (xx >= R && xx < R + TW && yy >= R && yy < R + TH)
            {
                const uint32_t d = __vabsdiffu4(pa[i], pb[i]) & 0xffffffu;
                sq = __dp4a(d, d, sq);
            }
        }
    }
    isti::ExactSum ssim;
#pragma unroll 1
    for (int c = 0; c < 3; c++)
    {
        const int shift = 8 * c;
#pragma unroll
        for (int i = 0; i < PER; i++)
            if (tid + i * Q_THREADS < SH * SW)
                xy[tid + i * Q_THREADS] = make_float2(byte_to_unit((pa[i] >> shift) & 255u), byte_to_unit((pb[i] >> shift) & 255u));
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < SH * (TW / 4); i += Q_THREADS)
        {
            const int col = i / SH * 4, row = i % SH;
            const float4 *src = reinterpret_cast<const float4 *>(xy + row * SW + col);
            float2 m[4] = {}, q[4] = {};
            float x12[4] = {};
#pragma unroll
            for (int t = 0; t < WIN + 3; t += 2)
            {
                const float4 two = src[t / 2];
                const float2 v[2] = {make_float2(two.x, two.y), make_float2(two.z, two.w)};
#pragma unroll
                for (int s = 0; s < 2; s++)
                {
                    const float2 v2 = __fmul2_rn(v[s], v[s]);
                    const float vc = v[s].x * v[s].y;
#pragma unroll
                    for (int j = 0; j < 4; j++)
                    {
                        const int k = t + s - j;
                        if (k < 0 || k >= WIN)
                            continue;
                        m[j] = __ffma2_rn(gw.g[k], v[s], m[j]);
                        q[j] = __ffma2_rn(gw.g[k], v2, q[j]);
                        x12[j] = fmaf(gw.g[k].x, vc, x12[j]);
                    }
                }
            }
            float4 *om = reinterpret_cast<float4 *>(hm + row * Q_PITCH + col), *oq = reinterpret_cast<float4 *>(hq + row * Q_PITCH + col);
            om[0] = make_float4(m[0].x, m[0].y, m[1].x, m[1].y);
            om[1] = make_float4(m[2].x, m[2].y, m[3].x, m[3].y);
            oq[0] = make_float4(q[0].x, q[0].y, q[1].x, q[1].y);
            oq[1] = make_float4(q[2].x, q[2].y, q[3].x, q[3].y);
            *reinterpret_cast<float4 *>(hc + row * Q_PITCH1 + col) = make_float4(x12[0], x12[1], x12[2], x12[3]);
        }
        __syncthreads();
        constexpr int ROWS_EACH = TH / (Q_THREADS / 32);
        float2 m[ROWS_EACH] = {}, q[ROWS_EACH] = {};
        float x12[ROWS_EACH] = {};
#pragma unroll
        for (int t = 0; t < ROWS_EACH + WIN - 1; t++)
        {
            const int row = warp * ROWS_EACH + t;
            const float2 vm = hm[row * Q_PITCH + lane], vq = hq[row * Q_PITCH + lane];
            const float vc = hc[row * Q_PITCH1 + lane];
#pragma unroll
            for (int j = 0; j < ROWS_EACH; j++)
            {
                const int k = t - j;
                if (k < 0 || k >= WIN)
                    continue;
                m[j] = __ffma2_rn(gw.g[k], vm, m[j]);
                q[j] = __ffma2_rn(gw.g[k], vq, q[j]);
                x12[j] = fmaf(gw.g[k].x, vc, x12[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < ROWS_EACH; j++)
        {
            if (x0 + lane >= w || y0 + warp * ROWS_EACH + j >= h)
                continue;
            constexpr float C1 = 0.01f * 0.01f, C2 = 0.03f * 0.03f;
            const float m1s = m[j].x * m[j].x, m2s = m[j].y * m[j].y, m12 = m[j].x * m[j].y;
            const float v1 = q[j].x - m1s, v2 = q[j].y - m2s, v12 = x12[j] - m12;
            const float num = (2.0f * m12 + C1) * (2.0f * v12 + C2);
            const float den = (m1s + m2s + C1) * (v1 + v2 + C2);
            ssim.add(__fdiv_rn(num, den)); // (about -1..1)
        }
        // the next channel's staging writes xy, which every thread has read before the last
        // barrier; its horizontal pass writes hm, hq and hc after the next one
    }

    // block reduction (warp shuffles, then one value per warp)
    double ssim_sum = ssim.value();
    for (int o = 16; o > 0; o >>= 1)
        ssim_sum += __shfl_down_sync(0xffffffffu, ssim_sum, o);
    sq = __reduce_add_sync(0xffffffffu, sq); // a tile has 1024 pixels: 1024 * 3 * 65025 < 2^32
    __shared__ double ws[Q_THREADS / 32];
    __shared__ uint32_t wq[Q_THREADS / 32];
    if (lane == 0)
    {
        ws[warp] = ssim_sum;
        wq[warp] = sq;
    }
    __syncthreads();
    if (tid == 0)
    {
        double s = 0.0;
        unsigned long long q = 0;
        for (int k = 0; k < Q_THREADS / 32; k++)
        {
            s += ws[k];
            q += wq[k];
        }
        const size_t blk = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
        partials[2 * blk] = s;
        partials[2 * blk + 1] = (double)q; // exact: at most 3 * 1024 * 65025 per block
    }
}

__global__ void __launch_bounds__(THREADS) quality_final_kernel(const double *partials, size_t n_blocks,
                                                                double n_values, isti_quality *out)
{
    __shared__ double ss[THREADS], sq[THREADS];
    double s = 0.0, q = 0.0;
    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    for (size_t i = threadIdx.x; i < n_blocks; i += THREADS) // fixed assignment and order: deterministic
    {
        s += partials[2 * i];
        q += partials[2 * i + 1];
    }
    ss[threadIdx.x] = s;
    sq[threadIdx.x] = q;
    __syncthreads();
    for (int o = THREADS / 2; o > 0; o >>= 1)
    {
        if ((int)threadIdx.x < o)
        {
            ss[threadIdx.x] += ss[threadIdx.x + o];
            sq[threadIdx.x] += sq[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        const double mse = sq[0] / (n_values * 65025.0);
        out->mse = mse;
        out->psnr = mse > 0.0 ? -10.0 * log10(mse) : INFINITY;
        out->ssim = ss[0] / n_values;
    }
}

// ---------------------------------------------------------------- LDR-FLIP
//
// scripts/flip_loss.py (the published LDR-FLIP, Andersson et al. 2020).  Every 2-D
// kernel of the reference is a sum of products f(x) g(y): the contrast-sensitivity
// filters are (sums of) normalised Gaussians, the edge / point detectors a derivative
// of a Gaussian in x times a Gaussian in y, normalised per sign of the x factor.  So
// each is applied as a horizontal then a vertical 1-D pass, all taps padded to a
// common radius R (the reference pads every filter by the largest radius, replicating
// the border).

constexpr int FR_MAX = ISTI_FLIP_MAX_RADIUS;
constexpr int FTAPS = 2 * FR_MAX + 1;
constexpr int FGROUPS_MAX = (FTAPS + 3) / 4; // taps are applied in groups of 4, the last one padded with zeros
constexpr int FTW = 32, FTH = 32;

enum FlipFilter
{
    CSF_A,   // achromatic CSF, 1-D factor
    CSF_RG,  // red-green CSF
    CSF_BY1, // blue-yellow CSF = by1(x) by1(y) + by2(x) by2(y)
    CSF_BY2,
    GAUSS,   // feature detectors: normalised Gaussian factor
    EDGE,    // d/dx factor of the edge detector
    POINT,   // d2/dx2 factor of the point detector
    N_FLIP_FILTERS
};

struct FlipFilters
{
    int r;      // common radius of every 1-D filter
    int groups; // groups of 4 taps: (2 r + 1) rounded up
    float cmax; // maximum HyAB^qc (green vs blue), redistribute_errors
    float2 tap[N_FLIP_FILTERS][4 * FGROUPS_MAX]; // tap k (offset k - r) twice, for the packed operations; zeros past 2 r
};

// Shared memory of a FLIP tile: the (reference, test) pixels, one plane of them at a time (Cz, Cx, Y,
// the normalised Y) as pairs, two buffers of horizontally filtered rows, the sRGB table.  The third
// buffer of the feature detectors lies over the pixels, not needed by then.
struct FlipTile
{
    int sh, sw, pitch, hrows; // input rows and columns; input pitch; rows of a filtered buffer (padded taps read past sh)
    __host__ __device__ explicit FlipTile(int r, int groups)
        : sh(FTH + 2 * r), sw(FTW + 2 * r), pitch(sw + (sw % 4 == 0 ? 2 : 0)), hrows(FTH + 4 * groups)
    {
    }
    __host__ __device__ int plane() const { return sh * pitch; }
    __host__ __device__ int hplane() const { return hrows * FH_PITCH; }
    __host__ __device__ int pixels() const { return plane() > hplane() ? plane() : hplane(); }
    __host__ __device__ int padded_plane() const { return plane() + ROW_SLACK; }
    __host__ __device__ size_t bytes() const
    {
        return (size_t)(pixels() + padded_plane() + 2 * hplane()) * sizeof(float2) + 256 * sizeof(float);
    }
    static constexpr int FH_PITCH = FTW + 2;
    static constexpr int ROW_SLACK = 4; // padded (zero) taps read up to 4 pairs past a row
};

constexpr float FLIP_QC = 0.7f, FLIP_PC = 0.4f, FLIP_PT = 0.95f, FLIP_EPS = 1e-15f;

// linear RGB -> XYZ (D65), the reference's rational constants rounded to float
__constant__ float L2X[3][3] = {{(float)(10135552.0 / 24577794.0), (float)(8788810.0 / 24577794.0), (float)(4435075.0 / 24577794.0)},
                             {(float)(2613072.0 / 12288897.0), (float)(8788810.0 / 12288897.0), (float)(887015.0 / 12288897.0)},
                             {(float)(1425312.0 / 73733382.0), (float)(8788810.0 / 73733382.0), (float)(70074185.0 / 73733382.0)}};

__device__ __forceinline__ float3 lin_to_xyz_scaled(float r, float g, float b)
{
    // XYZ divided by the D65 white (the reference's inv_reference_illuminant)
    return make_float3((L2X[0][0] * r + L2X[0][1] * g + L2X[0][2] * b) * 1.052156925f, L2X[1][0] * r + L2X[1][1] * g + L2X[1][2] * b,
                       (L2X[2][0] * r + L2X[2][1] * g + L2X[2][2] * b) * 0.918357670f);
}

// sRGB byte -> linear
__device__ __forceinline__ float srgb8_to_linear(uint32_t byte)
{
    const float v = (float)byte / 255.0f;
    return v > 0.04045f ? powf((fmaxf(v, 0.04045f) + 0.055f) / 1.055f, 2.4f) : v / 12.92f;
}

// sRGB pixel -> one component of YCxCz (color_space_transform 'srgb2ycxcz'); lin: srgb8_to_linear of every byte
enum FlipPlane
{
    PLANE_Y,
    PLANE_CX,
    PLANE_CZ
};
template <FlipPlane C>
__device__ __forceinline__ float srgb8_to_ycxcz(uint32_t p, const float *lin)
{
    const float3 xyz = lin_to_xyz_scaled(lin[p & 255u], lin[(p >> 8) & 255u], lin[(p >> 16) & 255u]);
    return C == PLANE_Y ? 116.0f * xyz.y - 16.0f : C == PLANE_CX ? 500.0f * (xyz.x - xyz.y) : 200.0f * (xyz.y - xyz.z);
}

// filtered YCxCz -> linear RGB clamped to the unit cube -> L*a*b* -> Hunt-adjusted
__device__ __forceinline__ float3 ycxcz_to_hunt_lab(float Y, float Cx, float Cz)
{
    const float yy = isti::divided_by<116>(Y + 16.0f);
    const float X = (yy + isti::divided_by<500>(Cx)) * 0.950428545f, Yv = yy, Z = (yy - isti::divided_by<200>(Cz)) * 1.088900371f;
    float rgb[3] = {3.241003275f * X - 1.537398934f * Yv - 0.498615861f * Z, -0.969224334f * X + 1.875930071f * Yv + 0.041554224f * Z,
                    0.055639423f * X - 0.204011202f * Yv + 1.057148933f * Z};
#pragma unroll
    for (int k = 0; k < 3; k++)
        rgb[k] = fminf(fmaxf(rgb[k], 0.0f), 1.0f);
    const float3 s = lin_to_xyz_scaled(rgb[0], rgb[1], rgb[2]);
    float xyz[3] = {s.x, s.y, s.z};
    constexpr float d3 = (6.0f / 29.0f) * (6.0f / 29.0f) * (6.0f / 29.0f);
    constexpr float factor = 1.0f / (3.0f * (6.0f / 29.0f) * (6.0f / 29.0f));
#pragma unroll
    for (int k = 0; k < 3; k++)
        xyz[k] = xyz[k] > d3 ? powf(fmaxf(xyz[k], d3), 1.0f / 3.0f) : factor * xyz[k] + 4.0f / 29.0f;
    const float L = 116.0f * xyz[1] - 16.0f;
    const float a = 500.0f * (xyz[0] - xyz[1]), b = 200.0f * (xyz[1] - xyz[2]);
    return make_float3(L, 0.01f * L * a, 0.01f * L * b);
}

// The horizontal pass of NF filters over one plane: a thread filters 4 neighbouring outputs of a
// row from one window of the row, 4 taps at a time.
template <int NF>
__device__ __forceinline__ void flip_rows(const FlipFilters &f, const FlipTile &t, const float2 *plane, const FlipFilter (&which)[NF],
                                          float2 *const (&out)[NF])
{
#pragma unroll 1
    for (int i = threadIdx.x; i < t.sh * (FTW / 4); i += THREADS)
    {
        // lanes take different rows: pitches of an odd number of 16-byte words, no bank conflicts
        const int g = i / t.sh, row = i - g * t.sh;
        const float4 *src = reinterpret_cast<const float4 *>(plane + row * t.pitch + 4 * g);
        float2 acc[NF][4] = {}, v[8];
        auto load = [&](int at, int n) {
            const float4 a = src[2 * n], b = src[2 * n + 1];
            v[at] = make_float2(a.x, a.y);
            v[at + 1] = make_float2(a.z, a.w);
            v[at + 2] = make_float2(b.x, b.y);
            v[at + 3] = make_float2(b.z, b.w);
        };
        load(0, 0);
#pragma unroll 2
        for (int n = 0; n < f.groups; n++)
        {
            load(4, n + 1);
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int q = 0; q < NF; q++)
                {
                    const float2 c = f.tap[which[q]][4 * n + k];
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        acc[q][j] = __ffma2_rn(c, v[k + j], acc[q][j]);
                }
#pragma unroll
            for (int k = 0; k < 4; k++)
                v[k] = v[4 + k];
        }
#pragma unroll
        for (int q = 0; q < NF; q++)
        {
            float4 *o = reinterpret_cast<float4 *>(out[q] + row * FlipTile::FH_PITCH + 4 * g);
            o[0] = make_float4(acc[q][0].x, acc[q][0].y, acc[q][1].x, acc[q][1].y);
            o[1] = make_float4(acc[q][2].x, acc[q][2].y, acc[q][3].x, acc[q][3].y);
        }
    }
}

constexpr int F_ROWS_EACH = FTH / (THREADS / 32);

// The vertical pass: a thread filters F_ROWS_EACH outputs of its column.  Term q is filter
// which[q] over buffer rows[from[q]], added to acc[to[q]]; terms of one sum alternate tap by tap.
template <int NB, int NF, int NA>
__device__ __forceinline__ void flip_columns(const FlipFilters &f, const float2 *const (&rows)[NB], const int (&from)[NF],
                                             const FlipFilter (&which)[NF], const int (&to)[NF], float2 (&acc)[NA][F_ROWS_EACH])
{
    static_assert(F_ROWS_EACH == 4, "the window holds 4 outputs and 4 taps");
    const int at = (threadIdx.x >> 5) * F_ROWS_EACH * FlipTile::FH_PITCH + (threadIdx.x & 31);
    float2 v[NB][8];
#pragma unroll
    for (int b = 0; b < NB; b++)
#pragma unroll
        for (int k = 0; k < 4; k++)
            v[b][k] = rows[b][at + k * FlipTile::FH_PITCH];
#pragma unroll 2
    for (int n = 0; n < f.groups; n++)
    {
#pragma unroll
        for (int b = 0; b < NB; b++)
#pragma unroll
            for (int k = 0; k < 4; k++)
                v[b][4 + k] = rows[b][at + (4 * (n + 1) + k) * FlipTile::FH_PITCH];
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int q = 0; q < NF; q++)
            {
                const float2 c = f.tap[which[q]][4 * n + k];
#pragma unroll
                for (int j = 0; j < F_ROWS_EACH; j++)
                    acc[to[q]][j] = __ffma2_rn(c, v[from[q]][k + j], acc[to[q]][j]);
            }
#pragma unroll
        for (int b = 0; b < NB; b++)
#pragma unroll
            for (int k = 0; k < 4; k++)
                v[b][k] = v[b][4 + k];
    }
}

// One block per 32x32 output tile.  Both images travel together as (reference, test) pairs:
// every filter step is one packed fma.rn.f32x2 for both.  The tile's pixels and an R-pixel
// replicate-padded halo are staged once; plane by plane they are converted, rows are filtered into
// shared memory, then columns per output pixel, while the next plane is converted.
// Bound by issue and its latencies (8 powers a pixel, the filters' FMAs and shared-memory reads; not by
// HBM: 2 x 4 bytes a pixel): the register windows read each staged value once per 4 outputs, and a
// 21-tap tile takes a third of an SM.  1080p: 510 us with the images in turn, one output per thread
// and pass and a power per staged colour value; 238 with all three planes staged and two tiles per
// SM; 211 with three tiles, 198 with divisions by constants and roots instead of powers.
__global__ void __launch_bounds__(THREADS, 3) flip_tile_kernel(const uint32_t *test, const uint32_t *ref, int w, int h,
                                                               const __grid_constant__ FlipFilters f, double *partials, float *map)
{
    extern __shared__ __align__(16) float2 fsm[];
    const FlipTile t(f.r, f.groups);
    uint2 *pixels = reinterpret_cast<uint2 *>(fsm); // (reference, test)
    float2 *plane = fsm + t.pixels();
    float2 *h0 = plane + t.padded_plane(), *h1 = h0 + t.hplane(), *h2 = fsm;
    float *lin = reinterpret_cast<float *>(h1 + t.hplane());
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * FTW, y0 = blockIdx.y * FTH;
    const float2 zero = make_float2(0.0f, 0.0f);
    auto clear_tail = [&](float2 *rows) { // rows past the input's, read by padded (zero) taps
        for (int i = t.sh * FlipTile::FH_PITCH + tid; i < t.hplane(); i += THREADS)
            rows[i] = zero;
    };

    static_assert(THREADS == 256, "one table entry per thread");
    lin[tid] = srgb8_to_linear((uint32_t)tid);
    clear_tail(h0);
    clear_tail(h1);
    if (tid < FlipTile::ROW_SLACK)
        plane[t.plane() + tid] = zero;
    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    const int step_y = THREADS / t.pitch, step_x = THREADS - step_y * t.pitch;
    for (int i = tid, yy = tid / t.pitch, xx = tid - yy * t.pitch; i < t.plane(); i += THREADS)
    {
        const int gx = min(max(x0 + xx - f.r, 0), w - 1), gy = min(max(y0 + yy - f.r, 0), h - 1);
        const size_t idx = (size_t)gy * w + gx;
        pixels[i] = make_uint2(ref[idx], test[idx]);
        xx += step_x;
        yy += step_y;
        if (xx >= t.pitch)
        {
            xx -= t.pitch;
            yy++;
        }
    }
    __syncthreads();
    // (a thread converts the pixels that it staged)
    auto convert = [&]<FlipPlane C>() {
        for (int i = tid; i < t.plane(); i += THREADS)
            plane[i] = make_float2(srgb8_to_ycxcz<C>(pixels[i].x, lin), srgb8_to_ycxcz<C>(pixels[i].y, lin));
    };
    convert.template operator()<PLANE_CZ>();
    __syncthreads();

    float2 by[1][F_ROWS_EACH] = {}, rg[1][F_ROWS_EACH] = {}, la[1][F_ROWS_EACH] = {};
    flip_rows<2>(f, t, plane, {CSF_BY1, CSF_BY2}, {h0, h1});
    __syncthreads();
    flip_columns<2, 2>(f, {h0, h1}, {0, 1}, {CSF_BY1, CSF_BY2}, {0, 0}, by);
    convert.template operator()<PLANE_CX>();
    __syncthreads();
    flip_rows<1>(f, t, plane, {CSF_RG}, {h0});
    __syncthreads();
    flip_columns<1, 1>(f, {h0}, {0}, {CSF_RG}, {0}, rg);
    convert.template operator()<PLANE_Y>();
    __syncthreads();
    flip_rows<1>(f, t, plane, {CSF_A}, {h1});
    clear_tail(h2);
    __syncthreads();
    flip_columns<1, 1>(f, {h1}, {0}, {CSF_A}, {0}, la);
    for (int i = tid; i < t.plane(); i += THREADS)
        plane[i] = make_float2(isti::divided_by<116>(plane[i].x + 16.0f), isti::divided_by<116>(plane[i].y + 16.0f));
    __syncthreads();
    flip_rows<3>(f, t, plane, {GAUSS, EDGE, POINT}, {h0, h1, h2});
    __syncthreads();
    float2 gy[2][F_ROWS_EACH] = {}, ex[1][F_ROWS_EACH] = {}, fx[1][F_ROWS_EACH] = {}; // gy: edge and point along y
    flip_columns<1, 2>(f, {h0}, {0, 0}, {EDGE, POINT}, {0, 1}, gy);
    flip_columns<1, 1>(f, {h1}, {0}, {GAUSS}, {0}, ex);
    flip_columns<1, 1>(f, {h2}, {0}, {GAUSS}, {0}, fx);

    isti::ExactSum sum_v;
    const float pccmax = FLIP_PC * f.cmax;
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int r = 0; r < F_ROWS_EACH; r++)
    {
        const int gx = x0 + lane, gyy = y0 + warp * F_ROWS_EACH + r;
        if (gx >= w || gyy >= h)
            continue;
        const float3 lr = ycxcz_to_hunt_lab(la[0][r].x, rg[0][r].x, by[0][r].x), lt = ycxcz_to_hunt_lab(la[0][r].y, rg[0][r].y, by[0][r].y);
        // color pipeline: HyAB(reference, test) of the Hunt-adjusted colours
        const float dL = lr.x - lt.x, da = lr.y - lt.y, db = lr.z - lt.z;
        // (the root of a rounded square is the number again)
        const float hy = (dL * dL > FLIP_EPS ? fabsf(dL) : sqrtf(FLIP_EPS)) + sqrtf(da * da + db * db);
        const float power = powf(hy, FLIP_QC);
        const float dec = power < pccmax ? (FLIP_PT / pccmax) * power
                                         : FLIP_PT + ((power - pccmax) / (f.cmax - pccmax)) * (1.0f - FLIP_PT);
        // feature pipeline
        const float er = sqrtf(ex[0][r].x * ex[0][r].x + gy[0][r].x * gy[0][r].x), et = sqrtf(ex[0][r].y * ex[0][r].y + gy[0][r].y * gy[0][r].y);
        const float pr = sqrtf(fx[0][r].x * fx[0][r].x + gy[1][r].x * gy[1][r].x), pt = sqrtf(fx[0][r].y * fx[0][r].y + gy[1][r].y * gy[1][r].y);
        float def = fmaxf(fabsf(er - et), fabsf(pt - pr));
        def = fmaxf(def, FLIP_EPS);
        def = sqrtf(0.70710678f * def); // to the power qf = 1/2
        const float v = powf(dec, 1.0f - def);
        sum_v.add(v); // (about 0..1)
        if (map)
            map[(size_t)gyy * w + gx] = v;
    }
    double sum = sum_v.value();
    for (int o = 16; o > 0; o >>= 1)
        sum += __shfl_down_sync(0xffffffffu, sum, o);
    __shared__ double ws[THREADS / 32];
    if ((tid & 31) == 0)
        ws[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0)
    {
        double s = 0.0;
        for (int k = 0; k < THREADS / 32; k++)
            s += ws[k];
        partials[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(THREADS) flip_final_kernel(const double *partials, size_t n_blocks, double n_px,
                                                             double *out)
{
    __shared__ double ss[THREADS];
    double s = 0.0;
    isti::dependents_may_launch();
    isti::wait_for_prerequisites();
    for (size_t i = threadIdx.x; i < n_blocks; i += THREADS)
        s += partials[i];
    ss[threadIdx.x] = s;
    __syncthreads();
    for (int o = THREADS / 2; o > 0; o >>= 1)
    {
        if ((int)threadIdx.x < o)
            ss[threadIdx.x] += ss[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *out = ss[0] / n_px;
}

// The reference's filter definitions (generate_spatial_filter, feature_detection) as
// 1-D factors, in double, centred at FR_MAX.  Returns false when a filter's radius
// exceeds FR_MAX.
bool make_flip_filters(double ppd, FlipFilters &f)
{
    std::memset(&f, 0, sizeof f);
    const double pi = 3.14159265358979323846;
    const int rc = (int)std::ceil(3.0 * std::sqrt(0.04 / (2.0 * pi * pi)) * ppd); // max CSF scale parameter 0.04
    const double sd = 0.5 * 0.082 * ppd;
    const int rf = (int)std::ceil(3.0 * sd);
    if (rc > FR_MAX || rf > FR_MAX || rc < 0 || rf < 0)
        return false;
    f.r = std::max(rc, rf);
    f.groups = (2 * f.r + 1 + 3) / 4;
    auto tap = [&](FlipFilter which, int t) -> float2 & { return f.tap[which][t - FR_MAX + f.r]; }; // t - FR_MAX: the offset, -r..r
    auto set = [&](FlipFilter which, int t, double v) { tap(which, t) = make_float2((float)v, (float)v); };
    const double dx = 1.0 / ppd;
    auto gauss_1d = [&](double b, std::vector<double> &e) {
        e.assign(FTAPS, 0.0);
        double s = 0.0;
        for (int x = -rc; x <= rc; x++)
            s += (e[FR_MAX + x] = std::exp(-pi * pi * (x * dx) * (x * dx) / b));
        return s;
    };
    std::vector<double> ea, erg, e1, e2;
    const double sa = gauss_1d(0.0047, ea), srg = gauss_1d(0.0053, erg), s1 = gauss_1d(0.04, e1), s2 = gauss_1d(0.025, e2);
    // BY: 34.1 sqrt(pi / 0.04) e1(x) e1(y) + 13.5 sqrt(pi / 0.025) e2(x) e2(y), normalised to sum 1
    const double w1 = 34.1 * std::sqrt(pi / 0.04), w2 = 13.5 * std::sqrt(pi / 0.025);
    const double norm = w1 * s1 * s1 + w2 * s2 * s2;
    for (int t = FR_MAX - f.r; t <= FR_MAX + f.r; t++)
    {
        set(CSF_A, t, ea[t] / sa);
        set(CSF_RG, t, erg[t] / srg);
        set(CSF_BY1, t, e1[t] * std::sqrt(w1 / norm));
        set(CSF_BY2, t, e2[t] * std::sqrt(w2 / norm));
    }
    std::vector<double> g(FTAPS, 0.0), de(FTAPS, 0.0), dp(FTAPS, 0.0);
    double gs = 0.0, pos_e = 0.0, neg_e = 0.0, pos_p = 0.0, neg_p = 0.0;
    for (int x = -rf; x <= rf; x++)
    {
        const double e = std::exp(-(double)(x * x) / (2.0 * sd * sd));
        g[FR_MAX + x] = e;
        gs += e;
        de[FR_MAX + x] = -x * e;
        dp[FR_MAX + x] = ((double)(x * x) / (sd * sd) - 1.0) * e;
        (de[FR_MAX + x] < 0 ? neg_e : pos_e) += std::fabs(de[FR_MAX + x]);
        (dp[FR_MAX + x] < 0 ? neg_p : pos_p) += std::fabs(dp[FR_MAX + x]);
    }
    for (int t = FR_MAX - f.r; t <= FR_MAX + f.r; t++)
    {
        set(GAUSS, t, g[t] / gs);
        set(EDGE, t, de[t] / (de[t] < 0 ? neg_e : pos_e));
        set(POINT, t, dp[t] / (dp[t] < 0 ? neg_p : pos_p));
    }
    // cmax = HyAB(hunt(lab(green)), hunt(lab(blue)))^qc
    auto hunt_lab = [&](double r, double gg, double b, double out[3]) {
        static const double M[3][3] = {{10135552.0 / 24577794, 8788810.0 / 24577794, 4435075.0 / 24577794},
                                       {2613072.0 / 12288897, 8788810.0 / 12288897, 887015.0 / 12288897},
                                       {1425312.0 / 73733382, 8788810.0 / 73733382, 70074185.0 / 73733382}};
        static const double inv_illum[3] = {1.052156925, 1.0, 0.918357670};
        double v[3];
        for (int k = 0; k < 3; k++)
        {
            const double c = (M[k][0] * r + M[k][1] * gg + M[k][2] * b) * inv_illum[k];
            const double d = 6.0 / 29.0;
            v[k] = c > d * d * d ? std::cbrt(c) : c / (3 * d * d) + 4.0 / 29.0;
        }
        const double L = 116 * v[1] - 16;
        out[0] = L;
        out[1] = 0.01 * L * 500 * (v[0] - v[1]);
        out[2] = 0.01 * L * 200 * (v[1] - v[2]);
    };
    double gl[3], bl[3];
    hunt_lab(0, 1, 0, gl);
    hunt_lab(0, 0, 1, bl);
    const double hy = std::sqrt(std::max((gl[0] - bl[0]) * (gl[0] - bl[0]), 1e-15)) +
                      std::sqrt((gl[1] - bl[1]) * (gl[1] - bl[1]) + (gl[2] - bl[2]) * (gl[2] - bl[2]));
    f.cmax = (float)std::pow(hy, 0.7);
    return true;
}

size_t flip_tiles(int32_t w, int32_t h) { return (size_t)((w + FTW - 1) / FTW) * (size_t)((h + FTH - 1) / FTH); }

Gauss make_gauss()
{
    // loss_utils.gaussian(11, 1.5): float32 of exp(-(x - 5)^2 / (2 sigma^2)), divided by its float32 sum
    Gauss g;
    float sum = 0.0f;
    for (int k = 0; k < WIN; k++)
    {
        g.g[k].x = (float)std::exp(-double((k - R) * (k - R)) / (2.0 * 1.5 * 1.5));
        sum += g.g[k].x;
    }
    for (float2 &v : g.g)
        v.y = v.x = v.x / sum;
    return g;
}

size_t n_tiles(int32_t w, int32_t h) { return (size_t)((w + TW - 1) / TW) * (size_t)((h + TH - 1) / TH); }
} // namespace

extern "C" {

size_t isti_quality_scratch_bytes(int32_t width, int32_t height)
{
    if (width <= 0 || height <= 0)
        return 0;
    return n_tiles(width, height) * 2 * sizeof(double);
}

isti_status isti_quality_rgba8(const void *a, const void *b, int32_t width, int32_t height, void *scratch,
                               isti_quality *out, void *stream)
{
    if (!a || !b || !scratch || !out || width <= 0 || height <= 0 || width > 65535 || height > 65535)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_quality_rgba8: bad argument");
    if (((uintptr_t)a | (uintptr_t)b) & 3u)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_quality_rgba8: images must be 4-byte aligned");
    if (((uintptr_t)scratch | (uintptr_t)out) & 7u)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_quality_rgba8: scratch and out must be 8-byte aligned");
    static const Gauss gw = make_gauss();
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid((width + TW - 1) / TW, (height + TH - 1) / TH);
    // (every launch a programmatic dependent of what was before it)
    cudaError_t e = isti::launch_after(true, quality_tile_kernel, grid, Q_THREADS, 0, s, static_cast<const uint32_t *>(a),
                                             static_cast<const uint32_t *>(b), width, height, static_cast<double *>(scratch), gw);
    if (e == cudaSuccess)
        e = isti::launch_after(true, quality_final_kernel, 1, THREADS, 0, s, static_cast<const double *>(scratch),
                                     n_tiles(width, height), 3.0 * (double)width * (double)height, out);
    if (e != cudaSuccess)
        return isti::set_error(ISTI_ERR_CUDA, std::string("isti_quality_rgba8: ") + cudaGetErrorString(e));
    return ISTI_OK;
}

size_t isti_flip_scratch_bytes(int32_t width, int32_t height)
{
    if (width <= 0 || height <= 0)
        return 0;
    return flip_tiles(width, height) * sizeof(double);
}

isti_status isti_flip_rgba8(const void *test, const void *reference, int32_t width, int32_t height, float pixels_per_degree,
                            void *scratch, double *out_mean, float *out_map, void *stream)
{
    if (!test || !reference || !scratch || !out_mean || width <= 0 || height <= 0 || width > 65535 || height > 65535 ||
        !(pixels_per_degree > 0.0f))
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_flip_rgba8: bad argument");
    if (((uintptr_t)test | (uintptr_t)reference | (uintptr_t)out_map) & 3u || ((uintptr_t)scratch | (uintptr_t)out_mean) & 7u)
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_flip_rgba8: misaligned pointer");
    FlipFilters f;
    if (!make_flip_filters((double)pixels_per_degree, f))
        return isti::set_error(ISTI_ERR_INVALID_ARG, "isti_flip_rgba8: pixels_per_degree too large for the filter radius limit");
    const size_t smem = FlipTile(f.r, f.groups).bytes();
    static std::once_flag attr_once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(attr_once, [] {
        const size_t max_smem = FlipTile(FR_MAX, FGROUPS_MAX).bytes();
        attr_err = cudaFuncSetAttribute(flip_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem);
    });
    if (attr_err != cudaSuccess)
        return isti::set_error(ISTI_ERR_CUDA, std::string("isti_flip_rgba8: ") + cudaGetErrorString(attr_err));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid((width + FTW - 1) / FTW, (height + FTH - 1) / FTH);
    cudaError_t e = isti::launch_after(true, flip_tile_kernel, grid, THREADS, smem, s, static_cast<const uint32_t *>(test),
                                             static_cast<const uint32_t *>(reference), width, height, f, static_cast<double *>(scratch), out_map);
    if (e == cudaSuccess)
        e = isti::launch_after(true, flip_final_kernel, 1, THREADS, 0, s, static_cast<const double *>(scratch),
                                     flip_tiles(width, height), (double)width * (double)height, out_mean);
    if (e != cudaSuccess)
        return isti::set_error(ISTI_ERR_CUDA, std::string("isti_flip_rgba8: ") + cudaGetErrorString(e));
    return ISTI_OK;
}

} // extern "C"
