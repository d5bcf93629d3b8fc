// pt_random.cu -- the random-offset level (SynthesisFrame::
// createRandomPyramid, synthesisFrame.cpp:66-150).
//
// The reference draws it from glibc's rand() in one serial order: per pixel
// (with keyframes a draw for the key layer, then) pairs of draws for the
// offset until it hits a painted texel (opaque pixels only, at most 50
// trials), then two draws for the fractions.  Here the stream is cut into
// segments that are generated in parallel, each from its state, which the
// powers of the generator's step matrix give (k_glibc_states, k_glibc_draws).
// Without retries pixel k's draws are the k-th four.  With them, window by
// window of the stream, so that the scratch stays small (5 bytes a draw):
//  * k_trials: for every place in the stream, how many trials an opaque pixel
//    that starts there takes;
//  * k_starts: the one serial part, a warp that follows the places from
//    pixel to pixel, 32 pixels or up to the next retry at a step;
//  * k_texels: every pixel from its place.
// Before this, one thread stepped a row, or with retries or keys one thread
// the level.  Measured: a 1024x1024 level without retries 431 -> 41 us (and
// 1 ms of host work and a synchronisation less), a 192x160 level of an
// exemplar with a fifth of it unpainted 18.6 -> 0.89 ms, bounded by k_starts'
// chain of about 60 cycles a retry; a 1024x1024 level with half of it
// unpainted takes 72 ms.
#include <algorithm>
#include <mutex>
#include <vector>

#include "pt_common.cuh"
#include "pt_device.cuh"
#include "pt_internal.h"

namespace ptk {

constexpr int kSegment = 496;  // draws of a segment: 16 turns of the 31-word state

// The powers step^(kSegment 2^b) of the generator's step, each transposed, in
// the library's own device memory (no context's budget pays for them), filled
// once a device.  Streams of up to 2^31 draws need 23.
constexpr int kPowers = 23;
__device__ uint32_t g_powers[kPowers * 961];

struct RandParams {
    int w, h, mx, my;
    int transparencyOk, orientationEnabled;
    Arr<float4> img;     // level-size input colour (alpha)
    Arr<float> iorient;  // level-size input orientation
    ExView ex;           // exemplar level
    float4* out;
    int lead;            // draws before a pixel's trials: 1 with keys (its layer), else 0
    int nk, first_key;   // with keys
};

__device__ __forceinline__ uint32_t offset_texel(const RandParams& R, uint32_t d0, uint32_t d1, int* ox, int* oy) {
    *ox = (int)((d0 >> 1) % (uint32_t)R.mx);
    *oy = (int)((d1 >> 1) % (uint32_t)R.my);
    return (uint32_t)*oy * (uint32_t)R.ex.w + (uint32_t)*ox;
}
// the exemplar layer that a pixel's draw for its key gives
__device__ __forceinline__ int style_of(const RandParams& R, uint32_t d) {
    return (int)((d >> 1) % (uint32_t)R.nk) + R.first_key;
}
__device__ __forceinline__ const float4* layer_out(const RandParams& R, int style) {
    return R.ex.out + (size_t)clampi(style, 0, R.ex.ns - 1) * R.ex.w * R.ex.h;
}
__device__ __forceinline__ float4 random_texel(const RandParams& R, int x, int y, int style, uint32_t d0, uint32_t d1,
                                                uint32_t d2, uint32_t d3) {
    int ox, oy;
    const uint32_t t = offset_texel(R, d0, d1, &ox, &oy);
    const size_t L = (size_t)clampi(style, 0, R.ex.ns - 1) * R.ex.w * R.ex.h;
    const float orient = R.orientationEnabled
                             ? __ldg(R.iorient.p + (size_t)y * R.iorient.w + x) - __ldg(R.ex.orient + L + t)
                             : 0.f;
    const float rx = (float)(d2 >> 1) / (float)2147483647;
    const float ry = (float)(d3 >> 1) / (float)2147483647;
    return f4((float)ox + rx, (float)oy + ry, orient, (float)style);
}
__device__ __forceinline__ bool opaque_pixel(const RandParams& R, int k) {
    if (R.transparencyOk) return false;
    const int x = k % R.w, y = k / R.w;
    return __ldg(R.img.p + (size_t)y * R.img.w + x).w > kAlphaThreshold;
}

// The state at the start of each segment: segment g of the stream starts g *
// kSegment steps on, so its state is the product of the powers of g's bits
// with the seed's state.  A warp a segment.  The states lie where the draws
// will be, each at its segment's start; the last segment's, whose draws may
// be fewer than 31, in `last`.
__device__ __forceinline__ uint32_t* segment_state(uint32_t* draws, uint32_t* last, int segments, int i) {
    return i == segments - 1 ? last : draws + (size_t)i * kSegment;
}
// (walk: with retries; nothing is left to do once every pixel has its place)
__device__ __forceinline__ bool walk_done(const Walk* walk, int px) { return walk && walk->next >= px; }

__global__ void __launch_bounds__(256) k_glibc_states(const GlibcState s0, int first, int segments, uint32_t* draws,
                                                      uint32_t* last, const Walk* walk, int px) {
    const int seg = blockIdx.x * 8 + threadIdx.x / 32, i = threadIdx.x % 32;
    if (seg >= segments || walk_done(walk, px)) return;
    const int g = first + seg;
    uint32_t s = i < 31 ? s0.s[i] : 0u;
    for (int b = 0; g >> b; b++) {
        if (!((g >> b) & 1)) continue;
        const uint32_t* M = g_powers + (size_t)b * 961;
        uint32_t acc = 0;
#pragma unroll
        for (int k = 0; k < 31; k++) {
            const uint32_t m = i < 31 ? __ldg(M + k * 31 + i) : 0u;
            acc += m * __shfl_sync(0xffffffffu, s, k);
        }
        s = acc;
    }
    if (i < 31) segment_state(draws, last, segments, seg)[i] = s;
}

// The draws of each segment, a thread a segment with the 31-word state of
// r[i] = r[i-31] + r[i-3] in registers; each turn's 31 words go through
// shared memory so that a warp writes whole runs.
__global__ void __launch_bounds__(32) k_glibc_draws(int segments, size_t n, uint32_t* draws, uint32_t* last,
                                                    const Walk* walk, int px) {
    __shared__ uint32_t out[32][33];
    const int lane = threadIdx.x, g0 = blockIdx.x * 32, g = g0 + lane;
    if (walk_done(walk, px)) return;
    const uint32_t* state = segment_state(draws, last, segments, min(g, segments - 1));
    uint32_t r[31];
#pragma unroll
    for (int i = 0; i < 31; i++) r[i] = state[i];
    __syncwarp();  // (the warp's draws go over its segments' states)
#pragma unroll 1
    for (int turn = 0; turn < kSegment / 31; turn++) {
#pragma unroll
        for (int i = 0; i < 31; i++) {
            r[i] += r[i < 3 ? i + 28 : i - 3];
            out[lane][i] = r[i];
        }
        __syncwarp();
#pragma unroll 8
        for (int t = 0; t < 32; t++) {
            const size_t at = (size_t)(g0 + t) * kSegment + turn * 31 + lane;
            if (lane < 31 && g0 + t < segments && at < n) draws[at] = out[t][lane];
        }
        __syncwarp();
    }
}

// without retries: pixel k's four draws (in place) to its texel
__global__ void __launch_bounds__(256) k_texels_plain(const RandParams R) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= R.w * R.h) return;
    const uint4 d = reinterpret_cast<const uint4*>(R.out)[k];
    R.out[k] = random_texel(R, k % R.w, k / R.w, 0, d.x, d.y, d.z, d.w);
}

// trials of an opaque pixel that starts at draw a (draws past n count as
// painted: k_starts does not go there)
__global__ void __launch_bounds__(256) k_trials(const RandParams R, const uint32_t* __restrict__ draws, int n,
                                                uint8_t* trials, const Walk* walk) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n || walk_done(walk, R.w * R.h)) return;
    int t = 1;
    if (R.lead || !(a & 1)) {  // (without keys every pixel starts at an even place)
        const float4* L = layer_out(R, R.lead ? style_of(R, draws[a]) : 0);
        for (int p = a + R.lead; t < 50 && p + 1 < n; t++, p += 2) {
            int ox, oy;
            const uint32_t at = offset_texel(R, draws[p], draws[p + 1], &ox, &oy);
            if (!(__ldg(&L[at].w) < kAlphaThreshold)) break;
        }
    }
    trials[a] = (uint8_t)t;
}

// The place among the window's n draws at which each pixel starts, left in
// the bits of its texel's first word.  One block; its first warp walks, the
// others help to stage parts of `trials` and of the pixels' opacity.  A lane
// takes a pixel as if those before it in the step had no retry; the step ends
// at the first that has one.  The walk goes on from the window before, whose
// draws began `back` places earlier; it ends with less than a reserve of
// draws left, and windows overlap by a segment, which is more, so the place
// it ends at is one of the next window's.
constexpr int kWalkWindow = 1 << 15, kWalkReserve = 1 + 2 * 50 + 2 + 5 * 32;
static_assert(kSegment >= kWalkReserve + 31, "the next window holds the walk's place and the 31 draws before it");
__global__ void __launch_bounds__(512) k_starts(const RandParams R, const uint8_t* __restrict__ trials, int n,
                                                int back, Walk* walk) {
    __shared__ __align__(16) uint8_t T[kWalkWindow];
    __shared__ uint32_t O[kWalkWindow / 4 / 32 + 1];
    __shared__ int at[2];  // the next pixel and its place
    const int px = R.w * R.h, c = R.lead + 4, tid = threadIdx.x, lane = tid % 32;
    const int k0 = walk->next;
    int k = k0, a = walk->place - back;
    while (k < px) {
        const int count = min(n - a, kWalkWindow), pixels = min(px - k, kWalkWindow / 4);
        for (int i = tid; i < count; i += blockDim.x) T[i] = trials[a + i];
        for (int i = tid; i < (pixels + 31) / 32 * 32; i += blockDim.x) {
            const unsigned o = __ballot_sync(0xffffffffu, i < pixels && opaque_pixel(R, k + i));
            if (lane == 0) O[i / 32] = o;
        }
        __syncthreads();
        if (tid < 32) {
            int dk = 0, da = 0;
            while (dk < pixels && da + kWalkReserve <= count) {
                const int m = min(32, pixels - dk);
                const int j = dk + lane;
                const bool in = lane < m;
                const int t = in && ((O[j / 32] >> (j % 32)) & 1) ? T[da + c * lane] : 1;
                const unsigned retry = __ballot_sync(0xffffffffu, t != 1);
                const int s = retry ? __ffs(retry) - 1 : m - 1;  // the step's last pixel
                if (lane <= s) R.out[k + j].x = __int_as_float(a + da + c * lane);
                da += c * s + R.lead + 2 + 2 * __shfl_sync(0xffffffffu, t, s);
                dk += s + 1;
            }
            if (lane == 0) {
                at[0] = k + dk;
                at[1] = a + da;
            }
        }
        __syncthreads();
        const int k1 = at[0], a1 = at[1];
        __syncthreads();
        const bool stuck = k1 == k;  // fewer than a reserve of draws left
        k = k1;
        a = a1;
        if (stuck) break;
    }
    __syncthreads();  // (all have read the walk)
    if (tid == 0) {
        walk->first = k0;
        walk->next = k;
        walk->place = k < px ? a : back;
    }
}

// every pixel that k_starts placed in this window, from its place
__global__ void __launch_bounds__(256) k_texels(const RandParams R, const uint32_t* __restrict__ draws,
                                                const uint8_t* __restrict__ trials, const Walk* walk) {
    const int k = walk->first + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= walk->next) return;
    const int a = __float_as_int(R.out[k].x), t = opaque_pixel(R, k) ? trials[a] : 1;
    const uint32_t* d = draws + a + R.lead + 2 * (t - 1);
    R.out[k] = random_texel(R, k % R.w, k / R.w, R.lead ? style_of(R, draws[a]) : 0, d[0], d[1], d[2], d[3]);
}

// The pixels that the windows' draws did not suffice for (an exemplar with
// hardly a painted texel), one thread on from where k_starts ended: the 31
// draws before that place in the last window are the state there.  Without
// any draws (no scratch to be had), the whole level from the seed.
__global__ void k_rest(const RandParams R, const GlibcState s0, const uint32_t* draws, const Walk* walk) {
    const int px = R.w * R.h;
    int k = draws ? walk->next : 0;
    if (k >= px) return;
    uint32_t ring[31];
    for (int i = 0; i < 31; i++) ring[i] = draws ? draws[walk->place - 31 + i] : s0.s[i];
    int head = 0;
    auto next = [&]() -> uint32_t {
        int h28 = head + 28;
        if (h28 >= 31) h28 -= 31;
        const uint32_t v = ring[head] + ring[h28];
        ring[head] = v;
        head = (head == 30) ? 0 : head + 1;
        return v;
    };
    for (; k < px; k++) {
        const int style = R.lead ? style_of(R, next()) : 0;
        const float4* L = layer_out(R, style);
        const bool opaque = opaque_pixel(R, k);
        uint32_t d0, d1;
        int trial = 0;
        bool again;
        do {
            d0 = next();
            d1 = next();
            int ox, oy;
            const uint32_t t = offset_texel(R, d0, d1, &ox, &oy);
            trial++;
            again = opaque && __ldg(&L[t].w) < kAlphaThreshold && trial < 50;
        } while (again);
        const uint32_t d2 = next(), d3 = next();
        R.out[k] = random_texel(R, k % R.w, k / R.w, style, d0, d1, d2, d3);
    }
}

// counter-based random level: four hashed draws per pixel and trial
__global__ void k_counter_random(const RandParams R, uint32_t seed) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= R.w || y >= R.h) return;
    float ia = __ldg(R.img.p + (size_t)y * R.img.w + x).w;
    uint32_t base = hash32(seed ^ hash32(x * 0x85EBCA6BU ^ hash32(y * 0xC2B2AE35U)));
    uint32_t d0, d1;
    int trial = 0;
    bool again;
    do {
        d0 = hash32(base + 4u * trial);
        d1 = hash32(base + 4u * trial + 1u);
        trial++;
        int ox, oy;
        const uint32_t t = offset_texel(R, d0, d1, &ox, &oy);
        float ea = __ldg(&R.ex.out[t].w);
        again = !R.transparencyOk && ia > kAlphaThreshold && ea < kAlphaThreshold && trial < 50;
    } while (again);
    uint32_t d2 = hash32(base + 0x40000000u), d3 = hash32(base + 0x40000001u);
    R.out[(size_t)y * R.w + x] = random_texel(R, x, y, 0, d0, d1, d2, d3);
}

// the exemplar output texels with alpha < 0.99 (whether the random level's
// pixels may retry, and how often)
__global__ void k_count_transparent(const float4* out, size_t n, int* count) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    int c = 0;
    for (; i < n; i += (size_t)gridDim.x * blockDim.x) c += __ldg(&out[i].w) < kAlphaThreshold;
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

}  // namespace ptk

namespace pt {

using namespace ptk;

static RandParams rand_params(const RandomLevel& L) {
    RandParams R;
    R.w = L.w; R.h = L.h; R.mx = L.mx; R.my = L.my;
    R.transparencyOk = L.transparencyOk; R.orientationEnabled = L.orientationEnabled;
    R.img = L.img; R.iorient = L.iorient; R.ex = L.ex; R.out = L.out;
    R.lead = L.nk > 0 ? 1 : 0;
    R.nk = L.nk; R.first_key = L.first_key;
    return R;
}

// g_powers of the current device
static cudaError_t powers_ready(cudaStream_t s) {
    static std::mutex m;
    static uint64_t done = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(m);
    if (dev < 64 && (done >> dev & 1)) return cudaSuccess;
    const std::vector<uint32_t> all = glibc_powers(kSegment, kPowers);
    e = cudaMemcpyToSymbolAsync(g_powers, all.data(), all.size() * sizeof(uint32_t), 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // (other contexts' streams read them next)
    if (e == cudaSuccess && dev < 64) done |= 1ull << dev;
    return e;
}

// n draws of the stream from segment `first` on
static cudaError_t draw_stream(const GlibcState& s0, int first, size_t n, uint32_t* draws, uint32_t* last,
                               const Walk* walk, int px, cudaStream_t s) {
    const int seg = (int)((n + kSegment - 1) / kSegment);
    k_glibc_states<<<(seg + 7) / 8, 256, 0, s>>>(s0, first, seg, draws, last, walk, px);
    k_glibc_draws<<<(seg + 31) / 32, 32, 0, s>>>(seg, n, draws, last, walk, px);
    return cudaGetLastError();
}

cudaError_t launch_random_level(const RandomLevel& L, const GlibcState& s0, uint32_t* last, int* launches,
                                cudaStream_t s) {
    const RandParams R = rand_params(L);
    const size_t px = (size_t)L.w * L.h;
    cudaError_t e = powers_ready(s);
    if (e == cudaSuccess) e = draw_stream(s0, 0, 4 * px, (uint32_t*)L.out, last, nullptr, 0, s);
    if (e != cudaSuccess) return e;
    k_texels_plain<<<(unsigned)((px + 255) / 256), 256, 0, s>>>(R);
    *launches += 3;
    return cudaGetLastError();
}

size_t random_window(size_t n) {
    const size_t least = 8, most = (kRandomWindow + kSegment - 1) / kSegment;
    return std::min(std::max((n + kSegment - 1) / kSegment, least), most) * kSegment;
}

cudaError_t launch_random_level_retry(const RandomLevel& L, const GlibcState& s0, size_t total, uint32_t* draws,
                                      uint8_t* trials, size_t window, uint32_t* last, Walk* walk, int* launches,
                                      cudaStream_t s) {
    const RandParams R = rand_params(L);
    const int px = L.w * L.h, n = (int)window;
    if (!draws) {
        k_rest<<<1, 1, 0, s>>>(R, s0, nullptr, nullptr);
        *launches += 1;
        return cudaGetLastError();
    }
    cudaError_t e = powers_ready(s);
    if (e == cudaSuccess) e = cudaMemsetAsync(walk, 0, sizeof(Walk), s);
    // (at least four draws a pixel)
    const unsigned texels = (unsigned)((std::min(px, n / 4 + 1) + 255) / 256);
    int back = 0;
    for (size_t at = 0; e == cudaSuccess; at += back) {
        e = draw_stream(s0, (int)(at / kSegment), n, draws, last, walk, px, s);
        if (e != cudaSuccess) return e;
        k_trials<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(R, draws, n, trials, walk);
        k_starts<<<1, 512, 0, s>>>(R, trials, n, back, walk);
        k_texels<<<texels, 256, 0, s>>>(R, draws, trials, walk);
        *launches += 5;
        e = cudaGetLastError();
        back = n - kSegment;
        if (at + n >= total) break;
    }
    if (e != cudaSuccess) return e;
    k_rest<<<1, 1, 0, s>>>(R, s0, draws, walk);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_random_level_counter(const RandomLevel& L, uint32_t seed, cudaStream_t s) {
    const RandParams R = rand_params(L);
    const dim3 b(32, 4), g((L.w + 31) / 32, (L.h + 3) / 4);
    k_counter_random<<<g, b, 0, s>>>(R, seed);
    return cudaGetLastError();
}

cudaError_t launch_count_transparent(const float4* out, size_t n, int* count, cudaStream_t s) {
    k_count_transparent<<<152 * 4, 256, 0, s>>>(out, n, count);
    return cudaGetLastError();
}

}  // namespace pt
