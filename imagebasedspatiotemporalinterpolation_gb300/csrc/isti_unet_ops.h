// Launches of the tcgen05 convolution operators (isti_unet.cu), shared with the
// network code (isti_flownet.cu).
#pragma once

#include "isti.h"

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace isti_unet
{
// A 1x1 head of 4 outputs (f32 weights [4][cout] and bias) to fuse into a convolution's
// epilogue: its outputs go to flow (f32) and/or flow16 (f16), [pixel][4].
struct ConvHead
{
    const float *w, *b;
    float *flow;
    void *flow16;
};

// planes: which tensors are in planes of 8 channels ([n][c / 8][h][w][8], isti_unet_conv.cuh) rather
// than NHWC -- IN_PLANES the layer's input (x, of the weight gradient too), OUT_PLANES its output
// (out and mask; dy of the weight gradient).
constexpr int IN_PLANES = 1, OUT_PLANES = 2;

// pdl: launch as a programmatic dependent of the previous kernel in `stream` (it prepares while
// that kernel finishes, isti_pdl.cuh).  It then reads wpack, bias and the head before it waits: only
// behind a kernel that was itself launched after they were complete.  head: fuse that head into
// the epilogue where the row-tile kernel runs the layer (then `out` is not written and
// *head_fused is set); otherwise the layer runs as usual and *head_fused is cleared.
isti_status conv_launch(int taps, const void *x, int n, int h, int w, int cin, const void *wpack, const float *bias, const void *mask, int relu,
                        void *out, int cout, int32_t *status, cudaStream_t stream, int planes = 0, bool pdl = false,
                        const ConvHead *head = nullptr, bool *head_fused = nullptr);

// db (may be null): the bias gradient, the column sums of dy
isti_status wgrad_launch(int taps, const void *dy, const void *x, int n, int h, int w, int cin, int cout, float *dw, float *db, int accumulate,
                         void *scratch, size_t scratch_bytes, int32_t *status, cudaStream_t stream, int planes = 0, bool pdl = false);
isti_status pack_launch(int taps, const float *w, int cin, int cout, int transpose, void *wpack, cudaStream_t stream);
size_t wgrad_scratch(int taps, int n, int h, int w, int cin, int cout);
} // namespace isti_unet
