// pt_internal.h -- launchers shared by the kernel and host translation units.
#pragma once

#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#include <vector>

#include "pt_types.h"

namespace pt {

// Gaussian weights of radius r, sigma = r / 3, as allocateGaussianKernel
// (src/PaintTweenCUDA/convolution.cu:37-60) forms them: the exponential in
// float, and with `normalize` the division by sqrt(2*pi)*sigma in double
// (M_PI promotes the expression) rounded back to float.  w has 2r+1 entries.
inline void gaussian_weights(int r, bool normalize, float* w) {
    float sigma = (float)r / 3.0f, s2 = sigma * sigma;
    for (int i = 0; i <= r; i++) {
        float v = expf(-(float)(i * i) / (2.f * s2));
        if (normalize) v = (float)((double)v / (std::sqrt(2.0 * M_PI) * (double)sigma));
        w[r + i] = v;
        w[r - i] = v;
    }
}

#ifdef __CUDACC__
// With `dependent`, a launch whose blocks may start before the stream's
// previous kernel has ended; the kernel calls pdl_start before it touches
// global memory, and the previous one is of the same chain (pt_ctx::chained).
// Measured on whole syntheses: 128x128 still 5.38 -> 5.00 ms, four 512x512
// frames 87.7 -> 81.6 ms.  Larger grids than these hide a launch behind the
// last blocks of the one before anyway, and the blocks that wait take places
// from them: with all launches dependent two 1080p frames took 257 ms against
// 251 with none and 248 with this limit.
constexpr size_t kDependentBlocks = 3000;
template <class... K, class... A>
inline cudaError_t launch_dependent(bool dependent, void (*kernel)(K...), dim3 g, dim3 b, size_t smem, cudaStream_t s,
                                    A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = g;
    c.blockDim = b;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = at;
    c.numAttrs = dependent && (size_t)g.x * g.y <= kDependentBlocks ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, args...);
}
#endif

using ptk::Arr;
using ptk::ConvKernel;
using ptk::ExView;
using ptk::Params;
using ptk::PatchPlanes;
using ptk::TileMaps;

using ptk::KeyView;
using ptk::Ribbon;

cudaError_t launch_propagate(const Params& P, PatchPlanes work, int jump, int key, cudaStream_t s);
cudaError_t launch_scatter(const Params& P, PatchPlanes work, int write_all, uint32_t pass_id, int key,
                           cudaStream_t s);
// keyframe interpolation (pt_keys.cu)
cudaError_t launch_propagate_keys(const Params& P, PatchPlanes work, int jump, int key, const KeyView& K,
                                  cudaStream_t s);
cudaError_t launch_scatter_keys(const Params& P, PatchPlanes work, int write_all, int key, const KeyView& K,
                                cudaStream_t s);
cudaError_t launch_accumulate_ribbon(const Params& P, int forwards, Ribbon* dest, const Ribbon* src, int time_step,
                                     int overwrite, cudaStream_t s);
cudaError_t launch_ribbon_output(const Params& P, const Ribbon* rib, const float4* canvas, float4* out,
                                 cudaStream_t s);
cudaError_t launch_frame_to_key(const Params& P, PatchPlanes work, int look_forwards, const KeyView& K,
                                cudaStream_t s);
cudaError_t launch_merge_advected(const Params& P, int fallback, PatchPlanes work, cudaStream_t s);
cudaError_t launch_fill_ribbons(Ribbon* r, size_t n, int layer, cudaStream_t s);
cudaError_t launch_ribbon_pack(const Ribbon* src, int w, int h, float4* dst, cudaStream_t s);
cudaError_t launch_ribbon_down(const float4* src, int sw, float4* dst, int w, int h, cudaStream_t s);
cudaError_t launch_residual(const Params& P, float* out, cudaStream_t s);
cudaError_t launch_canvas(const Params& P, float4* canvas, bool dependent, cudaStream_t s);
// the tiles (kTileW x tile_h) with a pixel that is not culled (IncView::tiles)
cudaError_t launch_active_tiles(const Params& P, int tile_h, int* list, cudaStream_t s);
cudaError_t launch_random_offsets(const Params& P, PatchPlanes work, cudaStream_t s);
cudaError_t launch_upsample(const Params& P, PatchPlanes work, PatchPlanes border_src, int copy_border,
                            float* res_out, cudaStream_t s);
cudaError_t launch_advect(const Params& P, int d, int forwards, int time_step, int flags, cudaStream_t s);
cudaError_t launch_merge_random(const Params& P, int d, int forwards, float weight, int force, PatchPlanes work,
                                cudaStream_t s);
cudaError_t launch_merge_residual(const Params& P, int d, PatchPlanes work, cudaStream_t s);
cudaError_t launch_conv(const float* src, float* dst, int w, int h, int pitch, int rows, const ConvKernel& kw,
                        cudaStream_t s);
// both passes of the separable Gaussian at once (src and dst do not overlap)
cudaError_t launch_blur(const float* src, float* dst, int w, int h, int pitch, const ConvKernel& kw, cudaStream_t s);
cudaError_t launch_copy_patch(const Params& P, PatchPlanes dst, PatchPlanes src, cudaStream_t s);
cudaError_t launch_copy_float(const Params& P, float* dst, const float* src, cudaStream_t s);
cudaError_t launch_unpack_patch(const Params& P, const pt_patchxf* src, PatchPlanes dst, cudaStream_t s);
cudaError_t launch_pack_patch(const Params& P, PatchPlanes src, pt_patchxf* dst, cudaStream_t s);
cudaError_t launch_load_residual(const Params& P, const float* src, float* dst, cudaStream_t s);
cudaError_t launch_gather_level(const Params& P, const float* src, int ch, float* dst, cudaStream_t s);
cudaError_t launch_down_avg(const float* src, int w, int h, int ch, int vel, float* dst, cudaStream_t s);
cudaError_t launch_down_vote(const int* src, int w, int h, int* dst, cudaStream_t s);
cudaError_t launch_tensor_angle(const float* t3, int n, float* out, cudaStream_t s);
// the random level (pt_random.cu): L.nk > 0 with keyframe interpolation
struct RandomLevel {
    int w, h, mx, my;
    int transparencyOk, orientationEnabled;
    Arr<float4> img;
    Arr<float> iorient;
    ExView ex;
    float4* out;
    int nk, first_key;
};
using ptk::GlibcState;
using ptk::Walk;
// the powers step^(segment * 2^b), b < count, of glibc's generator, each transposed (31 x 31)
std::vector<uint32_t> glibc_powers(int segment, int count);
// Pixels that cannot retry: four draws each, no scratch but `last` (31 words).
// *launches grows by the kernels launched.
cudaError_t launch_random_level(const RandomLevel& L, const GlibcState& s0, uint32_t* last, int* launches,
                                cudaStream_t s);
// With retries or keys: windows of the stream up to `total` draws in all (what
// these do not suffice for is drawn serially); draws and trials: `window`
// elements, a size that random_window gave, or null (all is drawn serially);
// last: 31 words.
constexpr size_t kRandomWindow = 1 << 20;  // 5 MB of scratch
size_t random_window(size_t n);
cudaError_t launch_random_level_retry(const RandomLevel& L, const GlibcState& s0, size_t total, uint32_t* draws,
                                      uint8_t* trials, size_t window, uint32_t* last, Walk* walk, int* launches,
                                      cudaStream_t s);
cudaError_t launch_random_level_counter(const RandomLevel& L, uint32_t seed, cudaStream_t s);
cudaError_t launch_count_transparent(const float4* out, size_t n, int* count, cudaStream_t s);
cudaError_t launch_interleave_texels(const float4* base, const float4* out, const float* dt, float4* bo, int* flags,
                                     size_t n, cudaStream_t s);

// tiled patch-distance kernels for patch radius 2, 3, 4 (pt_tiled_r*.cu):
// kind 0 = propagate (arg = jump), 1 = scatter (arg = write_all),
// 2 = residual (into out); tm 0 = no temporal terms, 1 = forward, 2 = backward;
// M: the tensor maps of the staged planes (M.on = 0: staged by plain loads);
// wide: four lanes per pixel instead of two (propagate, scatter) or instead of
// one or two (residual); same results; dependent: launch_dependent
cudaError_t launch_tiled_2(int kind, int tm, const Params& P, const TileMaps& M, PatchPlanes work, int arg,
                           uint32_t pass_id, float* out, int wide, bool dependent, cudaStream_t s);
cudaError_t launch_tiled_3(int kind, int tm, const Params& P, const TileMaps& M, PatchPlanes work, int arg,
                           uint32_t pass_id, float* out, int wide, bool dependent, cudaStream_t s);
cudaError_t launch_tiled_4(int kind, int tm, const Params& P, const TileMaps& M, PatchPlanes work, int arg,
                           uint32_t pass_id, float* out, int wide, bool dependent, cudaStream_t s);
}  // namespace pt
