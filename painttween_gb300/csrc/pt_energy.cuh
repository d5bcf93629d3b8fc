// pt_energy.cuh -- the tiled patch-distance kernels (propagate, scatter,
// residual) for a compile-time patch radius R and temporal mode TM.
//
// Same per-pixel semantics and the same FP32 arithmetic, operation by
// operation, as the generic kernels in pt_kernels.cu (which restate
// calculateResidual and its callers, src/PaintTweenCUDA/texSynth_kernel.cu:
// 537-952), organised for sm_103a:
//  * a block owns a tile 32 pixels wide and two or four high; the pixel-side
//    inputs of every tap (input colour, canvas, and for temporal passes the
//    advected colours and validity) are staged once into shared memory with an
//    R-pixel halo;
//  * several lanes share a pixel: they take its candidates, or the taps of one
//    candidate, side by side; taps outside the level rectangle count as zeros,
//    which leaves the sums exactly as skipping them would;
//  * an exemplar texel is 32 bytes (base RGBA, output RGBA), one sector per
//    texel of the bilinear footprint; when a candidate's whole footprint lies inside the
//    exemplar (decided for the whole warp), the wrap and clamp steps -- which
//    are then no-ops -- are left out.
#pragma once

#include <atomic>
#include <climits>

#include "pt_common.cuh"
#include "pt_internal.h"

namespace ptk {

// Propagate's blocks per SM, which set its registers: the kernel waits for its
// fetches, so more warps help until they spill.  Measured (summed launches):
// without temporal terms three blocks of two candidates a lane (80 registers)
// 11.6 ms against 13.8 with two (1024x1024 still); with them two blocks (128)
// 167 against 174 ms (two 1080p frames); with the exact filter, whose samples
// hold eight texels, two 50 against 70 ms (640x360, radius 4).
template <int CPL, int TM, int HW>
struct PropShape {
    static constexpr int kBlocks = (HW == 0 || TM) ? (CPL == 1 ? 1 : 2) : (CPL == 1 ? 2 : 3);
};

// The residual's, by lanes per pixel.
template <int LPP, int HW>
struct ResidShape {
    static constexpr int kBlocks = LPP == 1 ? 4 : LPP == 2 ? 2 : 3;
};

enum { TM_NONE = 0, TM_FWD = 1, TM_BWD = 2 };

// The staged planes start on 128-byte boundaries (tensor copies write
// there); a tile row is TW texels, as a tensor copy's box row is.
template <int R, int TM, int H>
struct TileSmem {
    static constexpr int TW = kTileW + 2 * R;
    static constexpr int TH = H + 2 * R;
    static constexpr int N = TW * TH;
    alignas(128) float4 base[N];
    alignas(128) float4 canvas[N];
    alignas(128) float4 pbase[TM ? N : 1];
    alignas(128) float4 pout[TM ? N : 1];
    unsigned long long bar;          // completion barrier of the tensor copies
    uint8_t pvalid[TM ? N : 1];      // the advected record is valid (hysteresis > 0)
};

// both colours of one exemplar texel: a 32-byte record of the interleaved
// copy, one 256-bit read-only load (records start on 32-byte boundaries)
__device__ __forceinline__ void ld_texel(const float4* p, float4* b, float4* o) {
    float r0, r1, r2, r3, r4, r5, r6, r7;
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(r0), "=f"(r1), "=f"(r2), "=f"(r3), "=f"(r4), "=f"(r5), "=f"(r6), "=f"(r7)
        : "l"(p));
    *b = make_float4(r0, r1, r2, r3);
    *o = make_float4(r4, r5, r6, r7);
}

// bilinear base+output at (u, v) of one exemplar layer (LBO: its interleaved
// records); fast (warp-uniform): the footprint is known to be inside
// [0, w-1] x [0, h-1], so the clamps are no-ops and are skipped
// With HW (PT_FILTER_TEXTURE, textures bound) both colours come from the
// texture unit: layered fetches of layer `li` (the clamped style layer) at the
// texture coordinate u + 0.5, which is the reference's own sampling
// (PYRAMID_FETCH_LAYER, texSynth_kernel.cu:600-601).  The level sits in the
// corner of a larger array with its edge texels repeated once beyond, so
// outside the fast case the coordinate is clamped to [0, w-1] x [0, h-1]
// first (NaN to 0): that fetches the texels, with the weights, that clamp
// addressing on a w x h array would.
template <bool PK, int HW>
__device__ __forceinline__ void sample2(const ExView& E, int li, const float4* LBO, float u, float v, float4* base,
                                        float4* out, bool fast) {
    const int w = E.w, h = E.h;
    if (HW) {
        if (!fast) {  // (ex_tex's clamp)
            u = fminf(fmaxf(u, 0.0f), (float)(w - 1));
            v = fminf(fmaxf(v, 0.0f), (float)(h - 1));
        }
        const float xs = u + 0.5f, ys = v + 0.5f;
        *base = tex2DLayered<float4>(E.tbase, xs, ys, li);
        *out = tex2DLayered<float4>(E.tout, xs, ys, li);
        return;
    }
    float xs = u + 0.5f, ys = v + 0.5f;
    float xb = xs - 0.5f, yb = ys - 0.5f;
    float fx = floorf(xb), fy = floorf(yb);
    float a = xb - fx, c = yb - fy;
    int x0, x1, y0, y1;
    if (fast) {
        x0 = (int)fx; y0 = (int)fy; x1 = x0 + 1; y1 = y0 + 1;
    } else {
        fx = fminf(fmaxf(fx, -1.0f), (float)w);
        fy = fminf(fmaxf(fy, -1.0f), (float)h);
        int ix = (int)fx, iy = (int)fy;
        x0 = clampi(ix, 0, w - 1); x1 = clampi(ix + 1, 0, w - 1);
        y0 = clampi(iy, 0, h - 1); y1 = clampi(iy + 1, 0, h - 1);
    }
    float oa = 1.0f - a, oc = 1.0f - c;
    Bl bw;
    bw.w00 = oa * oc; bw.w10 = a * oc; bw.w01 = oa * c; bw.w11 = a * c;
    const size_t r0 = (size_t)y0 * w, r1 = (size_t)y1 * w;
    float4 b00, b10, b01, b11, o00, o10, o01, o11;
    ld_texel(LBO + 2 * (r0 + x0), &b00, &o00);
    ld_texel(LBO + 2 * (r0 + x1), &b10, &o10);
    ld_texel(LBO + 2 * (r1 + x0), &b01, &o01);
    ld_texel(LBO + 2 * (r1 + x1), &b11, &o11);
    *base = PK ? bl4p(bw, b00, b10, b01, b11) : bl4(bw, b00, b10, b01, b11);
    *out = PK ? bl4p(bw, o00, o10, o01, o11) : bl4(bw, o00, o10, o01, o11);
}

// the exemplar view with its filter mode fixed at compile time (the tiled
// kernels are instantiated per mode, so the other mode's code is dropped)
template <int HW>
__device__ __forceinline__ ExView ex_mode(const ExView& e) {
    ExView v = e;
    v.hw = HW;
    return v;
}

struct Cand {
    float x, y, theta, su, sv;
    int layer;
};

// per-pixel state of the tiled kernels
struct PixT {
    int x, y;          // level coordinates
    int sidx;          // shared-memory index of the pixel
    int imin, imax, jmin, jmax;  // taps inside the level rectangle
    bool hyst_on;      // advected-F centre valid (hysteresis term subtracted)
    float hyst;
    bool temporal;     // temporal terms of direction TM apply at this pixel
    Patch prev;        // advected offset at the pixel (direction TM)
    float2 pb0, pb1;   // its basis
    bool prev_fast;    // its footprint is inside the exemplar
    float sumW;        // sum of the valid taps' weights, in tap order (the same for every candidate)
};

// does the footprint of a patch at (x, y) with basis (b0, b1) stay inside
// [1, w-3] x [1, h-3] (so every tap's 2x2 texels are in range and no wrap
// applies, since the wrap period is at least the exemplar size)
template <int R>
__device__ __forceinline__ bool footprint_inside(float x, float y, float2 b0, float2 b1, int w, int h) {
    float bx = (float)R * (fabsf(b0.x) + fabsf(b1.x)) + 1.0f;
    float by = (float)R * (fabsf(b0.y) + fabsf(b1.y)) + 1.0f;
    return (x - bx >= 0.0f) && (x + bx <= (float)(w - 2)) && (y - by >= 0.0f) && (y + by <= (float)(h - 2));
}

// Early exit.  When every per-tap term is >= 0 (Params::earlyExit), the
// running sum of a candidate never decreases (each fmaf adds a non-negative
// product and rounding is monotone), and the final energy is that sum divided
// by the pixel's constant tap-weight sum.  Once the running sum reaches
// thr2 = best * sumW rounded up, the energy is >= best whatever the remaining
// taps add, so the reference's strict "<" test rejects the candidate: its
// remaining taps are skipped and it returns +inf, which every caller rejects
// the same way.  A candidate that is still below thr2 at the end returns
// exactly sum / sumW.  A NaN thr2 (no early exit, or best = kNoBest) never
// stops a sum, so the energy is computed in full, NaN and inf included.
constexpr float kNoBest = __builtin_nanf("");
__device__ __forceinline__ void count_taps(const Params& P, unsigned taps, bool temporal) {
    unsigned mask = __activemask();
    unsigned tsum = __reduce_add_sync(mask, taps);
    unsigned ttsum = __reduce_add_sync(mask, temporal ? taps : 0u);
    if (lane_id() == (unsigned)(__ffs(mask) - 1)) {
        atomicAdd(&P.counters[1], (unsigned long long)tsum);
        atomicAdd(&P.counters[2], (unsigned long long)ttsum);
    }
}

// Tensor copies into shared memory (cp.async.bulk.tensor) completing on an
// mbarrier.  Every wait is bounded: kWaitLimit polls of mbarrier.try_wait,
// each of which may suspend the thread for a short hardware time limit.
constexpr int kWaitLimit = 1 << 20;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// box (x, y) of a 2-D tensor map into shared memory at dst, counted on bar
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// waits for the barrier's phase `parity` to complete; false if it did not
// within the limit
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
#pragma unroll 1
    for (int i = 0; i < kWaitLimit; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// The tile of this block: of a list of active tiles, or of the whole grid.
// False past the list's end.
__device__ __forceinline__ bool block_tile(const int* list, int2* tile) {
    if (!list) {
        *tile = make_int2(blockIdx.x, blockIdx.y);
        return true;
    }
    const int i = blockIdx.y * gridDim.x + blockIdx.x;
    const int n = list[0], id = list[1 + i];  // (the list has room for every tile)
    *tile = make_int2(id & 0xffff, id >> 16);
    return i < n;
}

// Stages the tile (and halo) of the pixel-side inputs (`changed`: the records
// whose canvas is formed here, a bit each by row; plain loads only) and fills the
// state of pixel `pid` of the tile (several threads of the block's NT may ask
// for the same pixel).  Returns false for
// threads whose pixel is outside the level rectangle.  A tile whose halo lies inside the level rectangle, where
// the clamps are no-ops, is copied by tensor copies when the maps are on
// (one thread issues them; the texture mode's flush of subnormal input
// colours follows in shared memory); the others load texel by texel with
// the clamp rules.  *abort is set (for the whole block) when the copies did
// not complete within two bounded waits; the block must then return.
template <int R, int TM, int NT, int H>
__device__ __forceinline__ bool stage_tile(const Params& P, const TileMaps& M, TileSmem<R, TM, H>& T, int2 tile,
                                           int pid, PixT* px, bool* abort,
                                           const unsigned long long* changed = nullptr) {
    constexpr int TW = TileSmem<R, TM, H>::TW, TH = TileSmem<R, TM, H>::TH, N = TileSmem<R, TM, H>::N;
    const int tid = threadIdx.x + threadIdx.y * kTileW;
    const int lx = pid % kTileW, ly = pid / kTileW;
    const int x0 = tile.x * kTileW - R, y0 = tile.y * H - R;
    *abort = false;
    const bool interior = M.on && x0 >= 0 && y0 >= 0 && x0 + TW <= P.lw && y0 + TH <= P.lh;  // (block-uniform)
    if (interior) {
        const uint32_t bar = smem_addr(&T.bar);
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0) {
            const uint32_t bytes = (uint32_t)(N * sizeof(float4)) * (TM ? 4u : 2u);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            // x in FLOAT32 elements: 4 per texel, so x * 4 bytes is a multiple of 16
            tma_load_2d(T.base, &M.base, 4 * x0, y0, bar);
            tma_load_2d(T.canvas, &M.canvas, 4 * x0, y0, bar);
            if (TM) {
                tma_load_2d(T.pbase, &M.pbase, 4 * x0, y0, bar);
                tma_load_2d(T.pout, &M.pout, 4 * x0, y0, bar);
            }
        }
    } else {
        const Arr<float4>& ib = P.img.base[P.img.cur];
        for (int q = tid; q < N; q += NT) {
            int gx = clampi(x0 + q % TW, 0, P.lw - 1);
            int gy = clampi(y0 + q / TW, 0, P.lh - 1);
            size_t k = (size_t)gy * P.W + gx;
            T.base[q] = lin_texel_of(__ldg(ib.p + (size_t)gy * ib.w + gx), P.hwFilter);
            if (changed && ((changed[q / TW] >> (q % TW)) & 1)) {
                // formed here, and written where the record is of this tile;
                // no block of the launch reads the old value
                const float4 cv = canvas_of(P, k);
                const int lx = q % TW - R, ly = q / TW - R;
                T.canvas[q] = cv;
                if (lx >= 0 && ly >= 0 && lx < kTileW && ly < H && tile.x * kTileW + lx < P.lw &&
                    tile.y * H + ly < P.lh)
                    const_cast<float4*>(P.canvas)[k] = cv;
            } else {
                T.canvas[q] = P.canvas[k];
            }
            if (TM) {
                const AdvView& A = P.adv[TM == TM_FWD ? 0 : 1];
                T.pbase[q] = __ldg(A.base + k);
                T.pout[q] = __ldg(A.out + k);
            }
        }
    }
    if (TM) {
        const PatchPlanes& O = P.adv[TM == TM_FWD ? 0 : 1].off;
        for (int q = tid; q < N; q += NT) {
            const int gx = clampi(x0 + q % TW, 0, P.lw - 1), gy = clampi(y0 + q / TW, 0, P.lh - 1);
            T.pvalid[q] = __ldg(&O.B[(size_t)gy * P.W + gx].x) > 0;
        }
    }
    // the per-pixel state reads global memory only: with tensor copies it is
    // computed while they are in flight
    const int x = tile.x * kTileW + lx, y = tile.y * H + ly;
    const bool in = x < P.lw && y < P.lh;
    if (in) {
        px->x = x;
        px->y = y;
        px->sidx = (ly + R) * TW + lx + R;
        px->imin = max(-R, -x); px->imax = min(R, P.lw - 1 - x);
        px->jmin = max(-R, -y); px->jmax = min(R, P.lh - 1 - y);
        if (px->imin == -R && px->imax == R && px->jmin == -R && px->jmax == R) {
            px->sumW = P.sumW;
        } else {
            float sw = 0.0f;
#pragma unroll 1
            for (int i = -R; i <= R; i++)
#pragma unroll
                for (int j = -R; j <= R; j++) {
                    const bool valid = (i >= px->imin) && (i <= px->imax) && (j >= px->jmin) && (j <= px->jmax);
                    const float w = P.gauss[i + R] * P.gauss[j + R];
                    sw = valid ? sw + w : sw;
                }
            px->sumW = sw;
        }
        const size_t k = (size_t)y * P.W + x;
        px->hyst_on = false;
        px->hyst = 0.0f;
        if (P.hysteresisWeight != 0.0f) {
            px->hyst_on = __ldg(&P.adv[0].off.B[k].x) > 0;
            if (px->hyst_on) px->hyst = hysteresis_term(P, x, y);
        }
        px->temporal = false;
        px->prev_fast = false;
        if (TM) {
            px->prev = load_patch(P.adv[TM == TM_FWD ? 0 : 1].off, k);
            bool td = (P.tdIn > 0.f || P.tdOut > 0.f || P.tc > 0.f);
            px->temporal = td && px->prev.hyst > 0;
            if (px->temporal) {
                float a = screen_to_exemplar_angle(P, x, y, px->prev.x, px->prev.y, px->prev.layer);
                basis(a, P.scaleWU * px->prev.su, P.scaleWV * px->prev.sv, &px->pb0, &px->pb1);
                px->prev_fast = footprint_inside<R>(px->prev.x, px->prev.y, px->pb0, px->pb1, P.ex.w, P.ex.h);
            }
        }
    }
    if (interior) {
        const uint32_t bar = smem_addr(&T.bar);
        bool ok = mbar_wait(bar, 0);
        if (!ok) ok = mbar_wait(bar, 0);  // the copies still in flight, once more
        if (__syncthreads_or(!ok)) {
            if (tid == 0 && M.err) atomicExch(M.err, 1);
            *abort = true;
            return false;
        }
        if (P.hwFilter)
            for (int q = tid; q < N; q += NT) T.base[q] = lin_texel_of(T.base[q], 1);
    }
    __syncthreads();
    return in;
}

// A block whose pixels need no energy (change tracking skipped all their
// candidates) copies its records and stops before staging its tile.
// (write: the working buffer needs every record written)
__device__ __forceinline__ bool block_idle(const Params& P, PatchPlanes work, bool need, bool in, size_t k,
                                           bool write = true) {
    if (__syncthreads_or(need)) return false;
    if (in) {
        if (write) store_patch(work, k, load_patch(P.off, k));
        P.inc.chg[k] = 0;
    }
    return true;
}

constexpr unsigned kFull = 0xffffffffu;
// (1 -/+ 2^-17): bounds of the rounding of a reference-order sum of <= 81 terms
constexpr float kBoundLo = 1.0f - 1.0f / 131072.0f;
constexpr float kBoundHi = 1.0f + 1.0f / 131072.0f;
// pixel side of an evaluation
struct LanePix {
    int x, y, sidx;
    int imin, imax, jmin, jmax;
    float sum0, sumW;
    bool temporal, prev_fast;
    float prevx, prevy;
    int prevlayer;  // clamped to the exemplar's layers
    float2 pb0, pb1;
};

template <int R>
__device__ __forceinline__ LanePix lane_pix(const Params& P, const PixT& px) {
    LanePix q;
    q.x = px.x; q.y = px.y; q.sidx = px.sidx;
    q.imin = px.imin; q.imax = px.imax; q.jmin = px.jmin; q.jmax = px.jmax;
    q.sum0 = px.hyst_on ? 0.0f - px.hyst : 0.0f;
    q.sumW = px.sumW;
    q.temporal = px.temporal;
    q.prev_fast = px.prev_fast;
    q.prevx = px.prev.x; q.prevy = px.prev.y;
    q.prevlayer = ex_layer(P.ex, px.prev.layer);
    q.pb0 = px.pb0; q.pb1 = px.pb1;
    return q;
}

// the pixel contexts of a tile of NP pixels in shared memory
template <int NP>
struct PixShared {
    float4 a[NP];  // sum0, sumW, prev x, prev y
    float4 b[NP];  // prev basis
    int bits[NP];  // window bounds + R (4 bits each), temporal, prev_fast, prev layer
};

template <int R, int NP>
__device__ __forceinline__ void put_pix(PixShared<NP>& S, int pid, const LanePix& q) {
    S.a[pid] = make_float4(q.sum0, q.sumW, q.prevx, q.prevy);
    S.b[pid] = make_float4(q.pb0.x, q.pb0.y, q.pb1.x, q.pb1.y);
    S.bits[pid] = (q.imin + R) | ((q.imax + R) << 4) | ((q.jmin + R) << 8) | ((q.jmax + R) << 12) |
                  (q.temporal ? 1 << 16 : 0) | (q.prev_fast ? 1 << 17 : 0) | (q.prevlayer << 18);
}

template <int R, int TM, int NP>
__device__ __forceinline__ LanePix get_pix(const Params& P, const PixShared<NP>& S, int2 tile, int pid) {
    constexpr int TW = TileSmem<R, TM, NP / kTileW>::TW;
    LanePix q;
    const int lx = pid % kTileW, ly = pid / kTileW;
    q.x = tile.x * kTileW + lx;
    q.y = tile.y * (NP / kTileW) + ly;
    q.sidx = (ly + R) * TW + lx + R;
    const float4 a = S.a[pid], b = S.b[pid];
    const int bits = S.bits[pid];
    q.imin = (bits & 15) - R; q.imax = ((bits >> 4) & 15) - R;
    q.jmin = ((bits >> 8) & 15) - R; q.jmax = ((bits >> 12) & 15) - R;
    q.temporal = (bits >> 16) & 1;
    q.prev_fast = (bits >> 17) & 1;
    q.prevlayer = bits >> 18;
    q.sum0 = a.x; q.sumW = a.y; q.prevx = a.z; q.prevy = a.w;
    q.pb0 = make_float2(b.x, b.y); q.pb1 = make_float2(b.z, b.w);
    return q;
}

// ---------------------------------------------------------------------------
// Candidate evaluation in two parts.
//
// Nineteen of twenty candidates lose, so a candidate is first held against a
// lower bound of its energy over the taps in the order of their weight.  The
// reference forms its sum in tap order with round-to-nearest fmaf over at
// most 81 non-negative terms, which is at least (1 - 2^-17) times the exact
// sum of those terms, plus its start sum (the hysteresis term, <= 0) scaled by
// at most (1 + 2^-17).  So once (1 - 2^-17) * bound + that start-sum share
// reaches thr2 = best * sumW rounded up, the reference-order
// energy is >= best and the strict "<" rejects the candidate; the bound is
// formed with round-down products and sums, in any order.  Only where the
// threshold is so small (|thr2| < 2^-100) that subnormal rounding could
// matter, or is none at all, no candidate is rejected by it.
//  * The front pass (front_taps) takes the heaviest taps, the 3 x 3 in the
//    middle, for all of a lane's candidates of its pixel at once: the
//    pixel-side texels and the previous frame's samples of a tap are read
//    once for them.  Measured on whole syntheses: 82-89 % of the candidates end
//    here at radius 2, 66-68 % at radius 3, 45-57 % at radius 4.
//  * The survivors of a warp are packed into a queue of its own (WarpQueue),
//    from which groups of eight lanes take one candidate each (eval_queue):
//    eight further taps at a time in the order of their weight, the bound
//    tested after each eight.  Every tap's value is kept, so that a candidate
//    that no bound rejects (5-9 %) has its energy summed from them in the
//    reference's order: no tap is fetched again for the exact sum.
// Before this, each candidate was summed in the reference's order from the
// first column on, whose taps are the lightest, and left at the threshold:
// 15.7 / 28.4 / 48.1 taps fetched per candidate at radius 2 / 3 / 4 (now 7.5 /
// 12.0 / 24.6), each with its own read of the pixel side.  Measured, summed
// launches: propagate of a 1024x1024 still (radius 2) 21.5 -> 11.6 ms, of two
// 1080p frames (radius 3) 288 -> 167 ms, of a 128x128 still 5.5 -> 2.5 ms.
// What bounds it now (launches of the finest level, three in a row): warps wait
// for the fetches of one tap at a time, 4.8 of 10.2 cycles an instruction on a
// 1080p level and 6.3 of 11.8 on a 1024x1024 one, with the texture unit's data
// pipe at 33-45 and 26-40 % of its peak (74 % before); hence as many warps as
// the registers allow (PropShape).  Groups of 4 lanes measured the same, of 16
// 7 % slower; a front of 5 taps 1-7 % slower than 9.
// ---------------------------------------------------------------------------

constexpr int kFront = 9;   // taps of the front pass: the 3 x 3 in the middle
constexpr int kGroup = 8;   // lanes that evaluate one surviving candidate
constexpr int kGroups = 32 / kGroup;

// One tap of the weight order: its place (i, j), weight and index in the
// reference's (column-major) order.
struct Tap {
    float fi, fj, w;
    int code;  // (i + R) | (j + R) << 4 | t << 8 | place in a tile (j * TW + i) << 16
};
template <int R>
struct TapList {
    Tap tap[(2 * R + 1) * (2 * R + 1)];
    alignas(16) float w[(2 * R + 1) * (2 * R + 1)];  // the weights in the reference's order
};
template <int R>
__device__ __forceinline__ void load_tap_list(const Params& P, TapList<R>& L, int tid) {
    constexpr int n = 2 * R + 1, K = n * n;
    if (tid < K) {
        const int t = P.tapOrder[tid], i = t / n, j = t % n;
        Tap a;
        a.fi = (float)(i - R);
        a.fj = (float)(j - R);
        a.w = P.gauss[i] * P.gauss[j];
        a.code = i | (j << 4) | (t << 8) | (((j - R) * (kTileW + 2 * R) + i - R) * 65536);
        L.tap[tid] = a;
        L.w[t] = a.w;
    }
}

// the taps in the reference's order
template <int R>
struct TapPlace {
    Tap tap[(2 * R + 1) * (2 * R + 1)];
    float w[(2 * R + 1) * (2 * R + 1)];
};
template <int R>
__device__ __forceinline__ void load_tap_place(const Params& P, TapPlace<R>& L, int tid) {
    constexpr int n = 2 * R + 1;
    if (tid < n * n) {
        const int i = tid / n, j = tid % n;
        Tap a;
        a.fi = (float)(i - R);
        a.fj = (float)(j - R);
        a.w = P.gauss[i] * P.gauss[j];
        a.code = i | (j << 4) | (tid << 8) | (((j - R) * (kTileW + 2 * R) + i - R) * 65536);
        L.tap[tid] = a;
        L.w[tid] = a.w;
    }
}

// the candidate side of an evaluation
struct CandPos {
    float x, y;
    float2 b0, b1;
    int layer;
};

// exemplar samples of one tap
struct ExSample {
    float4 tb, to;
};

template <int HW>
__device__ __forceinline__ ExSample cand_fetch(const Params& P, const CandPos& c, float fi, float fj, bool fast,
                                               float* ptx, float* pty) {
    const size_t lsz = (size_t)P.ex.w * P.ex.h;
    const int li = ex_layer(P.ex, c.layer);
    const float hw = (float)P.histW, hh = (float)P.histH;
    float tx = c.x + fmaf(fi, c.b0.x, fj * c.b1.x);
    float ty = c.y + fmaf(fi, c.b0.y, fj * c.b1.y);
    if (!fast) {
        if (tx >= hw) tx -= hw; else if (tx < 0) tx += hw;
        if (ty >= hh) ty -= hh; else if (ty < 0) ty += hh;
    }
    ExSample s;
    sample2<true, HW>(P.ex, li, P.ex.bo + 2 * (size_t)li * lsz, tx, ty, &s.tb, &s.to, fast);
    *ptx = tx;
    *pty = ty;
    return s;
}

// the previous frame's samples of one tap (temporal passes)
template <int HW>
__device__ __forceinline__ ExSample prev_fetch(const Params& P, const LanePix& q, float fi, float fj, bool fastp) {
    const size_t lsz = (size_t)P.ex.w * P.ex.h;
    const float x = q.prevx + fmaf(fi, q.pb0.x, fj * q.pb1.x);
    const float y = q.prevy + fmaf(fi, q.pb0.y, fj * q.pb1.y);
    ExSample s;
    sample2<true, HW>(P.ex, q.prevlayer, P.ex.bo + 2 * (size_t)q.prevlayer * lsz, x, y, &s.tb, &s.to, fastp);
    return s;
}

// whether a tap of pixel q lies inside the level rectangle
template <int R>
__device__ __forceinline__ bool tap_inside(const LanePix& q, const Tap& tp) {
    const int i = (tp.code & 15) - R, j = ((tp.code >> 4) & 15) - R;
    return (i >= q.imin) && (i <= q.imax) && (j >= q.jmin) && (j <= q.jmax);
}

// the pixel side of one tap
struct PixSample {
    float4 base, canvas, pout;
    float4 dbase, dcanvas;  // temporal: base - pbase, canvas - pout
    bool prev;              // the temporal terms apply at this tap
};
template <int R, int TM, int H>
__device__ __forceinline__ PixSample pix_sample(const TileSmem<R, TM, H>& T, const LanePix& q, int s) {
    PixSample p;
    p.base = T.base[s];
    p.canvas = T.canvas[s];
    p.prev = false;
    if (TM && q.temporal) {
        p.pout = T.pout[s];
        p.prev = T.pvalid[s] != 0;
        p.dbase = sub4p(p.base, T.pbase[s]);
        p.dcanvas = sub4p(p.canvas, p.pout);
    }
    return p;
}

// calculateResidual's value at one tap before its Gaussian weight
// (texSynth_kernel.cu:537-659), without the terms of the middle tap;
// `center`: the middle tap, which leaves out the canvas term
template <int TM>
__device__ __forceinline__ float tap_terms(const Params& P, const PixSample& p, const ExSample& c, const ExSample& v,
                                           bool center) {
    float res = ssd_ap(p.base, c.tb, P.alphaWeight) * P.inputAnalogyWeight;
    if (TM) {
        float r = ssdp(p.dbase, sub4p(c.tb, v.tb)) * P.tdIn;
        r = fmaf(ssdp(p.dcanvas, sub4p(c.to, v.to)), P.tdOut, r);
        r = fmaf(ssdp(p.pout, c.to), P.tc, r);
        res = p.prev ? res + r : res;
    }
    return center ? res : fmaf(ssd_ap(p.canvas, c.to, P.alphaWeight), P.canvasOutputWeight, res);
}

// the terms of the middle tap added to its value: distance transform,
// histogram, object ids (texSynth_kernel.cu:640-655)
template <int HW>
__device__ __forceinline__ float center_terms(const Params& P, const LanePix& q, int layer, float sv, float tx,
                                              float ty, float res) {
    if (P.distTransWeight > 0.f) {
        float de = ex_sample_dt(ex_mode<HW>(P.ex), tx, ty, layer) / sv;
        float di = lay_texel(P.img.dt[P.img.cur], P, q.x, q.y);
        float diff = fmaxf(0.0f, fminf(fabsf(de - di), 10.0f));  // clamp(diff, 0, 10): a NaN difference gives 10
        res = res + diff * P.distTransWeight;
    }
    {
        int Lh = clampi(layer, 0, PT_MAX_STYLES - 1);
        float sh = (float)(P.histH / P.numStyles);
        int hx = clampi((int)tx, 0, P.histPitch - 1);
        int hy = clampi((int)(ty + sh * (float)layer), 0, P.histRows - 1);
        float h = __ldg(P.hist + (size_t)hy * P.histPitch + hx);
        float thr = P.histThreshold[Lh];
        res = res + ((h > thr) ? (h - thr) * P.histSlope[Lh] : 0.0f);
    }
    if (P.styleObjIdWeight > 0.f) {
        int imgID = lvl_texel(P.img.ids, q.x, q.y);
        int styleID = ex_point_id(P.ex, tx, ty, layer);
        res = res + ((imgID != styleID) ? P.styleObjIdWeight : 0.0f);
    }
    return res;
}

// calculateResidual's value at one tap, before its weight, of record c at its
// pixel q
template <int R, int TM, int HW, int H>
__device__ __forceinline__ float own_tap(const Params& P, const TileSmem<R, TM, H>& T, const LanePix& q,
                                         const CandPos& c, float sv, const Tap& tp, bool fast, bool fastp) {
    const PixSample p = pix_sample<R, TM, H>(T, q, q.sidx + (tp.code >> 16));
    ExSample v;
    float tx, ty;
    if (TM && p.prev) v = prev_fetch<HW>(P, q, tp.fi, tp.fj, fastp);
    const ExSample s = cand_fetch<HW>(P, c, tp.fi, tp.fj, fast, &tx, &ty);
    const bool center = tp.fi == 0.0f && tp.fj == 0.0f;
    const float r = tap_terms<TM>(P, p, s, v, center);
    return center ? center_terms<HW>(P, q, c.layer, sv, tx, ty, r) : r;
}

// thr2 and the bound pass's threshold of a pixel whose energy to beat is
// `best` (see kNoBest): the latter is NaN, which rejects nothing,
// where the bound is not used
struct Threshold {
    float thr2, bound;
};
__device__ __forceinline__ Threshold threshold_of(const Params& P, const LanePix& q, float best) {
    Threshold t;
    t.thr2 = (P.earlyExit && q.sumW >= kEpsilon) ? __fmul_ru(best, q.sumW) : kNoBest;
    // the start sum's share of the reference-order sum, from below
    const float s0lo = q.sum0 >= 0.0f ? __fmul_rd(q.sum0, kBoundLo) : __fmul_rd(q.sum0, kBoundHi);
    // (thr2 - s0lo) / (1 - 2^-17) from above: 1 / (1 - 2^-17) < 1 + 2^-16
    const float need = __fsub_ru(t.thr2, s0lo);
    t.bound = fabsf(t.thr2) >= 0x1p-100f ? (need > 0.0f ? __fmul_ru(need, 1.0f + 1.0f / 65536.0f) : need) : kNoBest;
    return t;
}

// The surviving candidates of one warp.
template <int CAP>
struct WarpQueue {
    float4 a[CAP];     // x, y, b0
    float4 b[CAP];     // b1, the bound so far, layer bits
    float v0[CAP];     // the middle tap's value
    uint16_t id[CAP];  // pid * CH + slot | fast << 15
};

// The front pass over NC candidates of pixel q (bit c of `alive`: candidate c
// is evaluated), the warp's lanes together.  Returns the candidates still
// alive; their bounds are in sum[], the middle tap's values in v0[].
template <int R, int TM, int HW, int NC, int H>
__device__ __forceinline__ unsigned front_taps(const Params& P, const TileSmem<R, TM, H>& T, const TapList<R>& L,
                                               const LanePix& q, const Threshold& th, const CandPos (&c)[NC],
                                               const float (&sv)[NC], unsigned alive, float (&sum)[NC],
                                               float (&v0)[NC]) {
    bool fast[NC];  // all of the warp's footprints of this candidate inside the exemplar
#pragma unroll
    for (int k = 0; k < NC; k++) {
        fast[k] = __all_sync(kFull, !((alive >> k) & 1) || footprint_inside<R>(c[k].x, c[k].y, c[k].b0, c[k].b1,
                                                                              P.ex.w, P.ex.h));
        sum[k] = 0.0f;
        v0[k] = 0.0f;
    }
    const bool fastp = TM ? __all_sync(kFull, !alive || !q.temporal || q.prev_fast) : true;
    const bool bounded = th.bound == th.bound;
    unsigned taps = 0;
#pragma unroll 1
    for (int t = 0; t < kFront; t++) {
        const unsigned on = (t == 0 || bounded) ? alive : 0u;
        if (!__any_sync(kFull, on)) break;
        const Tap tp = L.tap[t];
        if (!on || !tap_inside<R>(q, tp)) continue;
        const PixSample p = pix_sample<R, TM, H>(T, q, q.sidx + (tp.code >> 16));
        ExSample s[NC], v;
        float tx[NC], ty[NC];
        if (TM && p.prev) v = prev_fetch<HW>(P, q, tp.fi, tp.fj, fastp);
#pragma unroll
        for (int k = 0; k < NC; k++)
            if ((on >> k) & 1) s[k] = cand_fetch<HW>(P, c[k], tp.fi, tp.fj, fast[k], &tx[k], &ty[k]);
#pragma unroll
        for (int k = 0; k < NC; k++)
            if ((on >> k) & 1) {
                float r = tap_terms<TM>(P, p, s[k], v, t == 0);
                if (t == 0) {
                    r = center_terms<HW>(P, q, c[k].layer, sv[k], tx[k], ty[k], r);
                    v0[k] = r;
                }
                sum[k] = __fmaf_rd(r, tp.w, sum[k]);
                if (sum[k] >= th.bound) alive &= ~(1u << k);
            }
        taps += __popc(on);
    }
    if (P.counters) count_taps(P, taps, q.temporal);
    return alive;
}

// The lane's surviving candidates appended to its warp's queue; returns the
// queue's length (the same for every lane).
template <int R, int NC, int CAP>
__device__ __forceinline__ int queue_survivors(const Params& P, WarpQueue<CAP>& Q, int id0, unsigned alive,
                                               const CandPos (&c)[NC], const float (&sum)[NC], const float (&v0)[NC]) {
    const int n = __popc(alive);
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if ((int)lane_id() >= o) incl += v;
    }
    int w = incl - n;
#pragma unroll
    for (int k = 0; k < NC; k++)
        if ((alive >> k) & 1) {
            const bool in = footprint_inside<R>(c[k].x, c[k].y, c[k].b0, c[k].b1, P.ex.w, P.ex.h);
            Q.a[w] = make_float4(c[k].x, c[k].y, c[k].b0.x, c[k].b0.y);
            Q.b[w] = make_float4(c[k].b1.x, c[k].b1.y, sum[k], __int_as_float(c[k].layer));
            Q.v0[w] = v0[k];
            Q.id[w] = (uint16_t)((id0 + k) | (in ? 1 << 15 : 0));
            w++;
        }
    __syncwarp();
    return __shfl_sync(kFull, incl, 31);
}

// Evaluates the first n candidates of the warp's queue, a group of kGroup
// lanes each; energies of those that no bound rejects into energy[pid * CH +
// slot].  thr: the energy to beat of each pixel of the tile; V: the tap values
// of each of the warp's groups.
template <int R, int TM, int HW, int H, int CAP, int CH>
__device__ __forceinline__ void eval_queue(const Params& P, const TileSmem<R, TM, H>& T,
                                           const PixShared<kTileW * H>& S, const TapList<R>& L,
                                           const WarpQueue<CAP>& Q, int2 tile, int n, const float* thr,
                                           float* V, float* energy) {
    constexpr int K = (2 * R + 1) * (2 * R + 1);
    constexpr int kStride = (K + 3) / 4 * 4;
    constexpr int kRest = (K - kFront + kGroup - 1) / kGroup;        // steps past the front
    constexpr int kLast = kRest + (kFront - 1 + kGroup - 1) / kGroup;  // and of the front's other taps
    const int lane = (int)lane_id(), g = lane / kGroup, l = lane % kGroup;
    float* val = V + g * kStride;
    bool act = false, cfast = false;
    int next = 0, step = 0, id = 0;
    float sum = 0.0f;
    LanePix q;
    CandPos c;
    Threshold th;
    q.temporal = false;
    q.prev_fast = true;
#pragma unroll 1
    while (true) {
        const unsigned idle = __ballot_sync(kFull, !act);
        if (!act) {
            const int t = next + __popc(idle & ((1u << (g * kGroup)) - 1u)) / kGroup;
            if (t < n) {
                const float4 a = Q.a[t], b = Q.b[t];
                id = Q.id[t];
                cfast = (id >> 15) & 1;
                id &= 0x7fff;
                c.x = a.x; c.y = a.y;
                c.b0 = make_float2(a.z, a.w);
                c.b1 = make_float2(b.x, b.y);
                c.layer = __float_as_int(b.w);
                sum = b.z;
                q = get_pix<R, TM>(P, S, tile, id / CH);
                th = threshold_of(P, q, thr[id / CH]);
                if (l == 0) val[K / 2] = Q.v0[t];
                step = 0;
                act = true;
            }
        }
        next += __popc(idle) / kGroup;
        if (!__any_sync(kFull, act)) break;
        const bool fast = __all_sync(kFull, !act || cfast);
        const bool fastp = TM ? __all_sync(kFull, !act || !q.temporal || q.prev_fast) : true;
        // steps 0 .. kRest-1: the taps past the front; then the front's other
        // taps, for the exact sum
        float part = 0.0f;
        const int pos = step < kRest ? kFront + step * kGroup + l : 1 + (step - kRest) * kGroup + l;
        if (act && pos < (step < kRest ? K : kFront)) {
            const Tap tp = L.tap[pos];
            const int t = (tp.code >> 8) & 255;
            val[t] = 0.0f;  // (a tap outside the level rectangle adds nothing)
            if (tap_inside<R>(q, tp)) {
                const PixSample p = pix_sample<R, TM, H>(T, q, q.sidx + (tp.code >> 16));
                ExSample v;
                float tx, ty;
                if (TM && p.prev) v = prev_fetch<HW>(P, q, tp.fi, tp.fj, fastp);
                const ExSample s = cand_fetch<HW>(P, c, tp.fi, tp.fj, fast, &tx, &ty);
                const float r = tap_terms<TM>(P, p, s, v, false);
                val[t] = r;
                if (step < kRest) part = __fmul_rd(r, tp.w);
            }
            if (P.counters) count_taps(P, 1u, q.temporal);
        }
#pragma unroll
        for (int o = 1; o < kGroup; o <<= 1) part = __fadd_rd(part, __shfl_xor_sync(kFull, part, o));
        const bool last = act && step == kLast - 1;
        sum = __fadd_rd(sum, part);
        step++;
        if (act && !last && sum >= th.bound) act = false;
        if (__any_sync(kFull, last)) {
            __syncwarp();
            if (last) {
                // the exact sum, in the reference's order
                float e = q.sum0;
#pragma unroll
                for (int t = 0; t + 3 < K; t += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(val + t);
                    const float4 w = *reinterpret_cast<const float4*>(L.w + t);
                    e = fmaf(v.x, w.x, e);
                    e = fmaf(v.y, w.y, e);
                    e = fmaf(v.z, w.z, e);
                    e = fmaf(v.w, w.w, e);
                }
                static_assert(K % 4 == 1, "one tap past the fours");
                e = fmaf(val[K - 1], L.w[K - 1], e);
                if (l == 0)
                    energy[id] = (q.sumW < kEpsilon) ? kBigResidual : (e >= th.thr2) ? INFINITY : e / q.sumW;
                act = false;
            }
            __syncwarp();
        }
    }
}

// the energy phase's shared state of a block of NW warps over NP pixels, each
// warp with up to CAP surviving candidates
template <int R, int NW, int NP, int CAP, int CH>
struct EvalSmem {
    PixShared<NP> S;
    WarpQueue<CAP> Q[NW];
    TapList<R> L;
    alignas(16) float V[NW][kGroups * (((2 * R + 1) * (2 * R + 1) + 3) / 4 * 4)];
    float thr[NP];                    // the energy each pixel has to beat
    alignas(16) float energy[NP * CH];  // per candidate (CH a pixel): its energy, +inf where it lost or is none
};

// calculatePropagateOffset, texSynth_kernel.cu:956-982 (propagate_offset), for
// CPL of a pixel's sources at once, in steps whose loads do not wait for one
// another: the sources' records and scales, the exemplar orientations under
// the moved offsets, then the angles and bases.
struct PropCand {
    CandPos c;
    float theta;
};
template <int CPL>
__device__ __forceinline__ void propagate_candidates(const Params& P, int x, int y, int slot0, int jump,
                                                     float2 scale, PropCand (&o)[CPL]) {
    float4 a[CPL];
    float2 sc[CPL];
    float dx[CPL], dy[CPL];
#pragma unroll
    for (int i = 0; i < CPL; i++) {
        int tx, ty;
        propagate_source(slot0 + i, x, y, jump, &tx, &ty);
        dx[i] = (float)x - (float)tx;
        dy[i] = (float)y - (float)ty;
        a[i] = P.off.A[pixel_wrap_index(P, tx, ty)];
        sc[i] = lvl_texel_lin(P.img.scale, tx, ty, P.hwFilter);
    }
    float eo[CPL];
#pragma unroll
    for (int i = 0; i < CPL; i++) {
        float2 b0, b1;
        basis(a[i].z, P.scaleWU * sc[i].x, P.scaleWV * sc[i].y, &b0, &b1);
        CandPos& c = o[i].c;
        new_coord(dx[i], dy[i], a[i].x, a[i].y, b0, b1, &c.x, &c.y);
        clamp_to_exemplar(&c.x, &c.y, P.ex.w, P.ex.h);
        c.layer = __float_as_int(a[i].w);
        eo[i] = P.orientationEnabled ? ex_point_orient(P.ex, c.x, c.y, c.layer) : 0.0f;
    }
    const float io = P.orientationEnabled ? lvl_texel(P.img.orient, x, y) : 0.0f;
#pragma unroll
    for (int i = 0; i < CPL; i++) {
        o[i].theta = P.orientationEnabled ? fold_angle(eo[i] - io) : 0.0f;
        basis(o[i].theta, P.scaleWU * scale.x, P.scaleWV * scale.y, &o[i].c.b0, &o[i].c.b1);
    }
}

// propagate_kernel, texSynth_kernel.cu:956-982,1112-1219, over tiles of 32 x H
// pixels.  A lane takes CPL of its pixel's four candidates (a warp covers
// 8 * CPL pixels), and a warp goes through its candidates alone, from the
// front pass to its pixels' results, without a barrier of the block.
template <int R, int TM, int HW, int CPL, int H>
__global__ void __launch_bounds__(kTileW * H * 4 / CPL, PropShape<CPL, TM, HW>::kBlocks)
    kt_propagate(const Params P, const __grid_constant__ TileMaps M, PatchPlanes work, int jump) {
    constexpr int NP = kTileW * H, NT = NP * 4 / CPL, NW = NT / 32, PPW = 8 * CPL;  // PPW: pixels per warp
    using Tile = TileSmem<R, TM, H>;
    using Eval = EvalSmem<R, NW, NP, 32 * CPL, 4>;
    extern __shared__ __align__(128) unsigned char dyn[];
    Tile& T = *reinterpret_cast<Tile*>(dyn);
    Eval& E = *reinterpret_cast<Eval*>(dyn + (sizeof(Tile) + 127) / 128 * 128);
    pdl_start();
    int2 tile;
    if (P.inc.rtiles && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) P.inc.rtiles[0] = 0;
    if (!block_tile(P.inc.tiles, &tile)) return;
    const int tid = threadIdx.x + threadIdx.y * kTileW, warp = tid / 32, lane = tid % 32;
    const int pid = warp * PPW + lane % PPW, slot0 = lane / PPW * CPL;  // the lane's pixel and first candidate
    const bool head = slot0 == 0;                                      // the lane that writes its pixel
    // Change tracking: a candidate whose source record and whose target's
    // patch window are unchanged since the previous pass with this jump was
    // rejected there against the same residual and is skipped (bit i of
    // `skip`); a pass without a previous one skips nothing.
    unsigned skip = 0;
    if (P.inc.on) {
        const int x = tile.x * kTileW + pid % kTileW, y = tile.y * H + pid / kTileW;
        const bool in = x < P.lw && y < P.lh;
        const size_t k = (size_t)y * P.W + x;
        bool need = in;
        if (in && P.inc.prev != INT_MIN) {
            int last[CPL];
#pragma unroll
            for (int i = 0; i < CPL; i++) {
                int tx, ty;
                propagate_source(slot0 + i, x, y, jump, &tx, &ty);
                last[i] = P.inc.last[pixel_wrap_index(P, tx, ty)];
            }
            if (P.inc.win[k] < P.inc.prev) {
#pragma unroll
                for (int i = 0; i < CPL; i++)
                    if (last[i] < P.inc.prev) skip |= 1u << i;
                need = skip != (1u << CPL) - 1u && !image_culled(P, x, y);
            }
        }
        if (block_idle(P, work, need, in && head, k)) return;
    }
    load_tap_list<R>(P, E.L, tid);
    PixT px;
    bool abort;
    const bool in = stage_tile<R, TM, NT, H>(P, M, T, tile, pid, &px, &abort);  // (synchronises the block)
    if (abort) return;
    const int x = px.x, y = px.y;
    const size_t k = in ? (size_t)y * P.W + x : 0;
    // the candidates, in the reference's order (repeats and test_offset
    // rejections resolved here)
    CandPos c[CPL];
    float sv[CPL];
    unsigned alive = 0;
    bool own = false;
    LanePix q;
    Threshold th;
    q.temporal = false;
    q.prev_fast = true;
    th.thr2 = th.bound = kNoBest;
    float best = 0.0f;
    if (in) {
        if (image_culled(P, x, y)) {
            if (head) {
                const Patch z = make_patch(0, 0, 0, 0, 0, 1.f, 1.f);
                if (P.inc.on) P.inc.chg[k] = same_record(z, load_patch(P.off, k)) ? 0 : 1;
                store_patch(work, k, z);
            }
        } else {
            own = true;
            best = P.res[k];
            const float2 scale = lvl_texel_lin(P.img.scale, x, y, P.hwFilter);
            PropCand pc[CPL];
            propagate_candidates<CPL>(P, x, y, slot0, jump, scale, pc);
            const bool opaque = P.transparencyOk || !exemplar_transparent(P.ex);
            const bool culls = exemplar_culls(P.ex, P.exCull);
            const float ia = T.base[px.sidx].w;
#pragma unroll
            for (int i = 0; i < CPL; i++) {
                c[i] = pc[i].c;
                sv[i] = scale.y;
                float e = INFINITY;  // skipped, a repeat, or lost: rejected by "<"
                bool dup = false;
#pragma unroll
                for (int h = 0; h < i; h++)
                    dup |= !((skip >> h) & 1) && __float_as_uint(c[h].x) == __float_as_uint(c[i].x) &&
                           __float_as_uint(c[h].y) == __float_as_uint(c[i].y) &&
                           __float_as_uint(pc[h].theta) == __float_as_uint(pc[i].theta) && c[h].layer == c[i].layer;
                if (!((skip >> i) & 1) && !dup) {
                    bool ok = !culls ||
                              !(ex_texel_dt(ex_mode<HW>(P.ex), (int)c[i].x, (int)c[i].y, c[i].layer) > P.exCull);
                    if (ok && !opaque && ia > kAlphaThreshold)
                        ok = !(ex_sample_out_alpha(ex_mode<HW>(P.ex), c[i].x, c[i].y, c[i].layer) < kAlphaThreshold);
                    if (ok) {
                        alive |= 1u << i;
                        if (P.counters) count_eval(P, x, y, px.temporal, false);
                    } else {
                        e = kBigResidual;  // rejected before the energy: competes with 1e31
                    }
                }
                E.energy[pid * 4 + slot0 + i] = e;
            }
            q = lane_pix<R>(P, px);
            th = threshold_of(P, q, best);
            if (head) {
                E.thr[pid] = best;
                put_pix<R>(E.S, pid, q);
            }
        }
    }
    float sum[CPL], v0[CPL];
    alive = front_taps<R, TM, HW, CPL, H>(P, T, E.L, q, th, c, sv, alive, sum, v0);
    const int n = queue_survivors<R, CPL>(P, E.Q[warp], pid * 4 + slot0, alive, c, sum, v0);
    eval_queue<R, TM, HW, H, 32 * CPL, 4>(P, T, E.S, E.L, E.Q[warp], tile, n, E.thr, E.V[warp], E.energy);
    __syncwarp();
    // each pixel takes the first candidate, in the reference's order, that
    // beats its running best
    if (own && head) {
        int win = -1;
        const float4 e4 = *reinterpret_cast<const float4*>(&E.energy[pid * 4]);
        const float e[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
        for (int cdx = 0; cdx < 4; cdx++)
            if (e[cdx] < best) { best = e[cdx]; win = cdx; }
        const Patch old = load_patch(P.off, k);
        if (win >= 0) {
            int tx, ty;
            propagate_source(win, x, y, jump, &tx, &ty);
            const Patch ow = propagate_offset(P, tx, ty, x, y);
            if (P.inc.on) P.inc.chg[k] = same_record(ow, old) ? 0 : 1;
            store_patch(work, k, ow);
        } else {
            if (P.inc.on) P.inc.chg[k] = 0;
            store_patch(work, k, old);
        }
    }
}

// scatter_kernel + averageOffset, texSynth_kernel.cu:841-952, over tiles of
// 32 x H pixels.  A pixel's chain is up to 25 candidates around its running
// best offset, then the average of its neighbours.  Few of them win, so LPP
// lanes of the pixel's own take the next LPP * NC of them at once, as they
// follow if none of those before wins; the first, in the chain's order, that
// beats the best is taken, and the chain goes on behind it from there.  Their
// energies go the way of propagate's candidates (front pass, then the warp's
// queue).
// Before this, a lane ran its pixel's chain one candidate after the other, so
// a launch took as long as the longest chains of its warps.  Measured, summed
// launches: 128x128 still 1.90 -> 0.44 ms, 1024x1024 still 5.6 -> 3.1 ms, two
// 1080p frames 67 -> 49 ms.  Eight lanes a pixel measured 41-55 % slower than
// four, tiles of eight rows 5-9 % slower than four with two lanes, three
// blocks an SM (80 registers) 9-30 % slower than two.
template <int R, int TM, int HW, int LPP, int H>
__global__ void __launch_bounds__(kTileW * H * LPP, 2)
    kt_scatter(const Params P, const __grid_constant__ TileMaps M, PatchPlanes work, int write_all,
               uint32_t pass_id) {
    constexpr int NC = 2, CH = NC * LPP;
    constexpr int NP = kTileW * H, NT = NP * LPP, NW = NT / 32, PPW = 32 / LPP;
    using Tile = TileSmem<R, TM, H>;
    using Eval = EvalSmem<R, NW, NP, 32 * NC, CH>;
    extern __shared__ __align__(128) unsigned char dyn[];
    Tile& T = *reinterpret_cast<Tile*>(dyn);
    Eval& E = *reinterpret_cast<Eval*>(dyn + (sizeof(Tile) + 127) / 128 * 128);
    pdl_start();
    int2 tile;
    if (P.inc.rtiles && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) P.inc.rtiles[0] = 0;
    if (!block_tile(P.inc.tiles, &tile)) return;
    const int tid = threadIdx.x + threadIdx.y * kTileW, warp = tid / 32, lane = tid % 32;
    const int pid = warp * PPW + lane % PPW, sub = lane / PPW;
    const bool head = sub == 0;  // the lane that writes its pixel
    // Change tracking: with the reference's generator a pixel's candidates
    // follow from its own record and its 3x3 neighbours, so a pixel whose
    // patch window is unchanged since the previous scatter of the loop had
    // every candidate rejected there against the same residual, and again now.
    bool stable = false;
    if (P.inc.on) {
        const int x = tile.x * kTileW + pid % kTileW, y = tile.y * H + pid / kTileW;
        const bool in = x < P.lw && y < P.lh;
        const size_t k = (size_t)y * P.W + x;
        stable = in && P.inc.prev != INT_MIN && P.inc.win[k] < P.inc.prev;
        if (block_idle(P, work, in && !stable, in && head, k, write_all != 0)) return;
    }
    load_tap_list<R>(P, E.L, tid);
    PixT px;
    bool abort;
    const bool in = stage_tile<R, TM, NT, H>(P, M, T, tile, pid, &px, &abort);  // (synchronises the block)
    if (abort) return;
    const int x = px.x, y = px.y;
    const size_t k = in ? (size_t)y * P.W + x : 0;
    bool own = false;
    if (in) {
        if (stable || image_culled(P, x, y)) {
            if (head) {
                if (write_all) store_patch(work, k, load_patch(P.off, k));
                if (P.inc.on) P.inc.chg[k] = 0;
            }
        } else {
            own = true;
        }
    }
    // chain state (the reference's loop, :896-937), the same in all of the
    // pixel's lanes
    const float closest = 10.f, factor = 0.9f;
    const float cached = own ? P.res[k] : 0.0f;
    float best = (float)((double)cached + 10e-7);
    float owx = 0.f, owy = 0.f, owt = 0.f;  // running best offset
    int wkind = 0;                           // 0: the pixel's own, 1: a chain candidate, 2: the average
    float ia = 0.f, dist = 0.f;
    float2 sc = make_float2(1.f, 1.f);
    float avgx = 0.f, avgy = 0.f;
    LanePix q;
    q.temporal = false;
    q.prev_fast = true;
    if (own) {
        const float4 a = P.off.A[k];
        owx = a.x; owy = a.y;
        ia = T.base[px.sidx].w;
        dist = (float)(P.ex.w > P.ex.h ? P.ex.w : P.ex.h);
        sc = lvl_texel_lin(P.img.scale, x, y, P.hwFilter);
        // averageOffset of the base field (:841-861)
        int na = 0;
#pragma unroll
        for (int i = -1; i <= 1; i++)
#pragma unroll
            for (int j = -1; j <= 1; j++) {
                if (!in_rect(P, x + i, y + j) || (i == 0 && j == 0)) continue;
                const float4 nb = P.off.A[(size_t)(y + j) * P.W + (x + i)];
                if (__float_as_int(nb.w) != 0) continue;
                avgx = avgx + nb.x;
                avgy = avgy + nb.y;
                na++;
            }
        avgx = avgx / (float)na;
        avgy = avgy / (float)na;
        q = lane_pix<R>(P, px);
        if (head) put_pix<R>(E.S, pid, q);
    }
    const bool opaque = P.transparencyOk || !exemplar_transparent(P.ex) || !(ia > kAlphaThreshold);
    const bool culls = exemplar_culls(P.ex, P.exCull);
    uint32_t lastx = 0xffffffffu, lasty = 0xffffffffu;
    int next = 0;                 // the chain's next candidate
    bool avg_pending = true, more = own;
#pragma unroll 1
    while (__any_sync(kFull, more)) {
        // the next CH candidates; the lane keeps its own NC
        CandPos c[NC];
        float sv[NC], theta[NC], cdist[NC];
        int kind[NC], cnext[NC];  // 0: none; where the chain goes on behind the candidate
#pragma unroll
        for (int s = 0; s < NC; s++) {
            c[s] = CandPos{0.f, 0.f, make_float2(0.f, 0.f), make_float2(0.f, 0.f), 0};
            sv[s] = 1.f;
            theta[s] = cdist[s] = 0.f;
            kind[s] = cnext[s] = 0;
        }
        const uint32_t lastx0 = lastx, lasty0 = lasty;
        bool any = false;
        if (more) {
#pragma unroll 1
            for (int s = 0; s < CH; s++) {
                bool have = false;
                float ex = 0.f, ey = 0.f;
#pragma unroll 1
                while (next < P.scatterSamples && dist * factor >= closest) {
                    const float dmin = dist * factor;
                    if (P.rngMode == PT_RNG_COUNTER) {
                        if (s / NC == sub) {
                            const float rr = counter_u01(P.rngSeed, pass_id, x, y, 2 * next);
                            const float th = counter_u01(P.rngSeed, pass_id, x, y, 2 * next + 1) * 6.28318530717958647692f;
                            float sn, cs;
                            sincos_poly(th, &sn, &cs);
                            const float len = fmaf(rr, dist - dmin, dmin);
                            ex = fmaf(cs, len, owx);
                            ey = fmaf(sn, len, owy);
                            clamp_to_exemplar(&ex, &ey, P.ex.w, P.ex.h);
                        }
                        next++;
                        dist *= factor;
                        have = true;
                        break;
                    }
                    ex = owx + dmin;
                    ey = owy + 0.0f;
                    clamp_to_exemplar(&ex, &ey, P.ex.w, P.ex.h);
                    next++;
                    dist *= factor;
                    // an exact repeat of the previous candidate has its energy
                    // and is rejected by the strict "<"
                    if (__float_as_uint(ex) == lastx && __float_as_uint(ey) == lasty) continue;
                    lastx = __float_as_uint(ex);
                    lasty = __float_as_uint(ey);
                    have = true;
                    break;
                }
                int kd = 1;
                if (!have) {
                    if (!avg_pending) break;
                    avg_pending = false;
                    kd = 2;
                    ex = avgx;
                    ey = avgy;
                }
                any = true;
#pragma unroll
                for (int z = 0; z < NC; z++)
                    if (s == sub * NC + z) {
                        c[z].x = ex;
                        c[z].y = ey;
                        kind[z] = kd;
                        cnext[z] = next;
                        cdist[z] = dist;
                    }
            }
        }
        unsigned alive = 0;
#pragma unroll
        for (int z = 0; z < NC; z++) {
            float e = INFINITY;
            if (kind[z]) {
                theta[z] = screen_to_exemplar_angle(P, x, y, c[z].x, c[z].y, 0);
                const float su = kind[z] == 1 ? sc.x : 1.f;
                sv[z] = kind[z] == 1 ? sc.y : 1.f;
                basis(theta[z], P.scaleWU * su, P.scaleWV * sv[z], &c[z].b0, &c[z].b1);
                bool ok = !culls || !(ex_texel_dt(ex_mode<HW>(P.ex), (int)c[z].x, (int)c[z].y, 0) > P.exCull);
                if (ok && !opaque) ok = !(ex_sample_out_alpha(ex_mode<HW>(P.ex), c[z].x, c[z].y, 0) < kAlphaThreshold);
                if (ok) {
                    alive |= 1u << z;
                    if (P.counters) count_eval(P, x, y, px.temporal, false);
                } else {
                    e = kBigResidual;  // rejected before the energy: competes with 1e31
                }
            }
            if (more) E.energy[pid * CH + sub * NC + z] = e;
        }
        const Threshold th = threshold_of(P, q, more ? best : kNoBest);
        if (more && head) E.thr[pid] = best;
        float sum[NC], v0[NC];
        alive = front_taps<R, TM, HW, NC, H>(P, T, E.L, q, th, c, sv, alive, sum, v0);
        const int n = queue_survivors<R, NC>(P, E.Q[warp], pid * CH + sub * NC, alive, c, sum, v0);
        eval_queue<R, TM, HW, H, 32 * NC, CH>(P, T, E.S, E.L, E.Q[warp], tile, n, E.thr, E.V[warp], E.energy);
        __syncwarp();
        // the first candidate that beats the best, if any
        int win = -1;
        if (more) {
#pragma unroll
            for (int s = CH - 1; s >= 0; s--) {
                const float r = E.energy[pid * CH + s];
                win = r < best ? s : win;
            }
        }
        const int src = (win < 0 ? sub : win / NC) * PPW + lane % PPW;
        float wx = 0.f, wy = 0.f, wt = 0.f, wd = 0.f;
        int wn = 0, wk = 0;
#pragma unroll
        for (int z = 0; z < NC; z++) {
            const float tx = __shfl_sync(kFull, c[z].x, src), ty = __shfl_sync(kFull, c[z].y, src);
            const float tt = __shfl_sync(kFull, theta[z], src), td = __shfl_sync(kFull, cdist[z], src);
            const int tn = __shfl_sync(kFull, cnext[z], src), tk = __shfl_sync(kFull, kind[z], src);
            if (win % NC == z) { wx = tx; wy = ty; wt = tt; wd = td; wn = tn; wk = tk; }
        }
        if (more) {
            if (win >= 0) {
                best = E.energy[pid * CH + win];
                owx = wx; owy = wy; owt = wt;
                wkind = wk;
                next = wn;
                dist = wd;
                avg_pending = wk != 2;
                lastx = __float_as_uint(wx);
                lasty = __float_as_uint(wy);
                if (wk == 2) { lastx = lastx0; lasty = lasty0; }
            }
            more = any && (avg_pending || next < P.scatterSamples && dist * factor >= closest);
        }
        __syncwarp();
    }
    if (!own || !head) return;
    const Patch off = load_patch(P.off, k);
    Patch ow = off;
    if (wkind == 1) ow = make_patch(owx, owy, owt, 0.0f, 0, sc.x, sc.y);
    else if (wkind == 2) ow = make_patch(owx, owy, owt, 1.f, 0, 1.f, 1.f);
    const bool take = best < cached;
    if (P.inc.on) P.inc.chg[k] = (take && !same_record(ow, off)) ? 1 : 0;
    if (take) store_patch(work, k, ow);
    else if (write_all) store_patch(work, k, off);
}

// updateResidualCache_kernel, texSynth_kernel.cu:661-693, over tiles of 32 x H
// pixels.  The residual is the reference-order weighted sum of per-tap values;
// LPP lanes of a pixel take its taps side by side, the values are kept and
// then summed in order.
//
// KEEP: inside a tracked propagate/scatter loop the values stay in P.inc.taps.
// A tap's value changes only when the pixel's own record changed (all taps) or
// the record of the pixel under the tap changed (its canvas), so only those
// taps are recomputed, queued per warp tap by tap so that neighbouring lanes
// sample neighbouring texels, and the sum is then taken again over the stored
// values: the same operations on the same values, so the same bits.  With
// `fill` every tap of every pixel is computed (the loop's first residual).
// Otherwise the values stay in shared memory.
//
// What bounds it is the time of the checks, loads and barriers around few
// taps: most tiles have none or a handful to recompute.  So tiles come from
// the canvas kernel's list on large levels, the changed records are a bit
// each, from which a row of a window is a shift, and a warp queues and sums
// alone.  Before: a lane a pixel over 32 x 8 tiles, the changed records a byte
// each, one queue a block between barriers.  Measured, summed launches: two
// 1080p frames 56.6 -> 47.7 ms, radius 4 at 192x160 4.8 -> 4.1 ms; without the
// lists the same kernel took 70 ms.  ResidShape: with one lane a pixel four
// blocks an SM 49.8, five 50.2, six 55.2 ms (two 1080p frames).
template <int R, int NW, int NP, bool KEEP>
struct ResidSmem {
    static constexpr int K = (2 * R + 1) * (2 * R + 1);
    PixShared<NP> S;
    float4 own[NP];   // the pixel's record: x, y, basis b0
    float4 own2[NP];  // basis b1, sv, layer bits
    uint8_t fast[NP];  // its footprint is inside the exemplar
    TapPlace<R> L;
    uint16_t list[KEEP ? NW : 1][KEEP ? NP / NW * K : 1];  // pixel of the warp << 8 | tap
    float v[KEEP ? 1 : NP][KEEP ? 1 : K];
    unsigned long long chg[NP / kTileW + 2 * R];  // the changed records of each row of tile and halo, a bit each
};

template <int R, int TM, int HW, int LPP, int H, bool KEEP>
__global__ void __launch_bounds__(kTileW * H * LPP, ResidShape<LPP, HW>::kBlocks)
    kt_residual(const Params P, const __grid_constant__ TileMaps M, float* out) {
    constexpr int NP = kTileW * H, NT = NP * LPP, NW = NT / 32, PPW = 32 / LPP;
    constexpr int n1 = 2 * R + 1, K = n1 * n1;
    using Tile = TileSmem<R, TM, H>;
    using Shared = ResidSmem<R, NW, NP, KEEP>;
    extern __shared__ __align__(128) unsigned char dyn[];
    Tile& T = *reinterpret_cast<Tile*>(dyn);
    Shared& E = *reinterpret_cast<Shared*>(dyn + (sizeof(Tile) + 127) / 128 * 128);
    constexpr int TW = Tile::TW, N = Tile::N;
    pdl_start();
    int2 tile;
    if (!block_tile(P.inc.fill ? nullptr : P.inc.rtiles, &tile)) return;
    const int tid = threadIdx.x + threadIdx.y * kTileW, warp = tid / 32, lane = tid % 32;
    const int lp = lane % PPW, pid = warp * PPW + lp, sub = lane / PPW;
    const int lx = pid % kTileW, ly = pid / kTileW;
    const int x = tile.x * kTileW + lx, y = tile.y * H + ly;
    const bool in = x < P.lw && y < P.lh;
    const size_t k = in ? (size_t)y * P.W + x : 0;
    const size_t plane = (size_t)P.W * P.H;
    const bool dense = !KEEP || P.inc.fill;  // every tap of every pixel
    bool own = in, any = in;
    load_tap_place<R>(P, E.L, tid);
    if (!dense) {
        const int x0 = tile.x * kTileW - R, y0 = tile.y * H - R;
        if (tid < Tile::TH) E.chg[tid] = 0;
        __syncthreads();
        bool some = false;
        for (int q = tid; q < N; q += NT) {
            const int gx = clampi(x0 + q % TW, 0, P.lw - 1), gy = clampi(y0 + q / TW, 0, P.lh - 1);
            if (P.inc.chg[(size_t)gy * P.W + gx]) {
                atomicOr(&E.chg[q / TW], 1ull << (q % TW));
                some = true;
            }
        }
        if (!__syncthreads_or(some)) return;
        unsigned all = 0;
#pragma unroll
        for (int j = 0; j < n1; j++) all |= (unsigned)(E.chg[ly + j] >> lx);
        own = in && ((E.chg[ly + R] >> (lx + R)) & 1);
        any = in && (all & ((1u << n1) - 1u));
        if (sub == 0) {
            if (own) P.inc.last[k] = P.inc.pi;
            if (any) P.inc.win[k] = P.inc.pi;
        }
    }
    PixT px;
    bool abort;
    // (synchronises the block)
    stage_tile<R, TM, NT, H>(P, M, T, tile, pid, &px, &abort, !dense && P.inc.canvas ? E.chg : nullptr);
    if (abort) return;
    bool mine = false;
    LanePix q;
    CandPos c;
    float sv = 1.0f;
    bool fast = true;
    q.temporal = false;
    q.prev_fast = true;
    if (any) {
        if (image_culled(P, x, y)) {
            if (sub == 0) out[k] = 0.0f;
        } else {
            mine = true;
            q = lane_pix<R>(P, px);
            const Patch o = load_patch(P.off, k);
            c.x = o.x; c.y = o.y; c.layer = o.layer;
            sv = o.sv;
            basis(o.theta, P.scaleWU * o.su, P.scaleWV * o.sv, &c.b0, &c.b1);
            fast = footprint_inside<R>(c.x, c.y, c.b0, c.b1, P.ex.w, P.ex.h);
            if (sub == 0 && !dense) {
                put_pix<R>(E.S, pid, q);
                E.own[pid] = make_float4(c.x, c.y, c.b0.x, c.b0.y);
                E.own2[pid] = make_float4(c.b1.x, c.b1.y, sv, __int_as_float(c.layer));
                E.fast[pid] = fast;
            }
            if (P.counters && own && sub == 0) count_eval(P, x, y, px.temporal, false);
        }
    }
    if (dense) {
        // the lane's own pixel, every LPP-th tap
        const bool wfast = __all_sync(kFull, !mine || fast);
        const bool fastp = TM ? __all_sync(kFull, !mine || !q.temporal || q.prev_fast) : true;
        unsigned taps = 0;
#pragma unroll 2
        for (int t = sub; t < K; t += LPP) {
            const Tap tp = E.L.tap[t];
            if (mine && tap_inside<R>(q, tp)) {
                const float r = own_tap<R, TM, HW, H>(P, T, q, c, sv, tp, wfast, fastp);
                if (KEEP) P.inc.taps[(size_t)t * plane + k] = r;
                else E.v[pid][t] = r;
                taps++;
            }
        }
        if (P.counters) count_taps(P, taps, q.temporal);
    } else {
        // the warp's affected taps, tap by tap
        int n = 0;
        uint16_t* list = E.list[warp];
        const unsigned cols = mine ? ((2u << (q.imax + R)) - 1u) & ~((1u << (q.imin + R)) - 1u) : 0u;
#pragma unroll 1
        for (int j0 = 0; j0 < n1; j0 += LPP) {
            const int j = j0 + sub;  // the lane's row of the window
            unsigned bits = 0;
            if (mine && j - R >= q.jmin && j - R <= q.jmax)
                bits = own ? cols : (unsigned)(E.chg[ly + j] >> lx) & cols;
            if (!__any_sync(kFull, bits)) continue;
#pragma unroll
            for (int i = 0; i < n1; i++) {
                const bool b = (bits >> i) & 1;
                const unsigned m = __ballot_sync(kFull, b);
                if (b) list[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(lp << 8 | (i * n1 + j));
                n += __popc(m);
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int i0 = 0; i0 < n; i0 += 32) {
            const bool act = i0 + lane < n;
            int t = 0, op = 0;
            LanePix a;
            CandPos ac;
            float asv = 1.0f;
            bool af = true;
            a.temporal = false;
            a.prev_fast = true;
            if (act) {
                const int v = list[i0 + lane];
                t = v & 255;
                op = warp * PPW + (v >> 8);
                a = get_pix<R, TM>(P, E.S, tile, op);
                const float4 o = E.own[op], o2 = E.own2[op];
                ac.x = o.x; ac.y = o.y;
                ac.b0 = make_float2(o.z, o.w);
                ac.b1 = make_float2(o2.x, o2.y);
                asv = o2.z;
                ac.layer = __float_as_int(o2.w);
                af = E.fast[op] != 0;
            }
            const bool wfast = __all_sync(kFull, af);
            const bool fastp = TM ? __all_sync(kFull, !a.temporal || a.prev_fast) : true;
            if (act)
                P.inc.taps[(size_t)t * plane + (size_t)a.y * P.W + a.x] =
                    own_tap<R, TM, HW, H>(P, T, a, ac, asv, E.L.tap[t], wfast, fastp);
            if (P.counters) count_taps(P, act ? 1u : 0u, a.temporal);
        }
    }
    __syncwarp();
    // the residual: the values summed in the reference's order
    if (mine && sub == 0) {
        float sum = q.sum0;
        const float* v = KEEP ? P.inc.taps + k : E.v[pid];
        const size_t step = KEEP ? plane : 1;
        const bool whole = q.imin == -R && q.imax == R && q.jmin == -R && q.jmax == R;
        if (whole) {
#pragma unroll n1
            for (int t = 0; t < K; t++) sum = fmaf(v[t * step], E.L.w[t], sum);
        } else {
#pragma unroll 1
            for (int t = 0; t < K; t++)
                if (tap_inside<R>(q, E.L.tap[t])) sum = fmaf(v[t * step], E.L.w[t], sum);
        }
        out[k] = (q.sumW < kEpsilon) ? kBigResidual : sum / q.sumW;
    }
}

// Kernels with more shared memory than a static array may have: the
// attribute that allows it is set once per kernel and device.
template <class F>
static cudaError_t allow_smem(F* kernel, size_t smem, std::atomic<uint64_t>& done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || (dev < 64 && (done.load(std::memory_order_acquire) >> dev & 1))) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
    return e;
}

template <int R, int TM, int HW, int CPL, int H>
static cudaError_t launch_propagate_t(const Params& P, const TileMaps& M, PatchPlanes work, int jump,
                                      bool dependent, cudaStream_t s) {
    constexpr int NP = kTileW * H, NT = NP * 4 / CPL;
    constexpr size_t smem =
        (sizeof(TileSmem<R, TM, H>) + 127) / 128 * 128 + sizeof(EvalSmem<R, NT / 32, NP, 32 * CPL, 4>);
    static std::atomic<uint64_t> done{0};
    const cudaError_t e = allow_smem(kt_propagate<R, TM, HW, CPL, H>, smem, done);
    if (e != cudaSuccess) return e;
    const dim3 g((P.lw + kTileW - 1) / kTileW, (P.lh + H - 1) / H);
    return pt::launch_dependent(dependent, kt_propagate<R, TM, HW, CPL, H>, g, dim3(kTileW, NT / kTileW), smem, s, P, M,
                                work, jump);
}

template <int R, int TM, int HW, int LPP, int H>
static cudaError_t launch_scatter_t(const Params& P, const TileMaps& M, PatchPlanes work, int write_all,
                                    uint32_t pass_id, bool dependent, cudaStream_t s) {
    constexpr int NP = kTileW * H, NT = NP * LPP;
    constexpr size_t smem =
        (sizeof(TileSmem<R, TM, H>) + 127) / 128 * 128 + sizeof(EvalSmem<R, NT / 32, NP, 64, 2 * LPP>);
    static std::atomic<uint64_t> done{0};
    const cudaError_t e = allow_smem(kt_scatter<R, TM, HW, LPP, H>, smem, done);
    if (e != cudaSuccess) return e;
    const dim3 g((P.lw + kTileW - 1) / kTileW, (P.lh + H - 1) / H);
    return pt::launch_dependent(dependent, kt_scatter<R, TM, HW, LPP, H>, g, dim3(kTileW, NT / kTileW), smem, s, P, M,
                                work, write_all, pass_id);
}

template <int R, int TM, int HW, int LPP, int H, bool KEEP>
static cudaError_t launch_residual_t(const Params& P, const TileMaps& M, float* out, bool dependent, cudaStream_t s) {
    constexpr int NP = kTileW * H, NT = NP * LPP;
    constexpr size_t smem = (sizeof(TileSmem<R, TM, H>) + 127) / 128 * 128 + sizeof(ResidSmem<R, NT / 32, NP, KEEP>);
    static std::atomic<uint64_t> done{0};
    const cudaError_t e = allow_smem(kt_residual<R, TM, HW, LPP, H, KEEP>, smem, done);
    if (e != cudaSuccess) return e;
    const dim3 g((P.lw + kTileW - 1) / kTileW, (P.lh + H - 1) / H);
    return pt::launch_dependent(dependent, kt_residual<R, TM, HW, LPP, H, KEEP>, g, dim3(kTileW, NT / kTileW), smem, s,
                                P, M, out);
}

template <int R>
cudaError_t launch_tiled_r(int kind, int tm, const Params& P, const TileMaps& M, PatchPlanes work, int arg,
                           uint32_t pass_id, float* out, int wide, bool dependent, cudaStream_t s) {
    // the texture-unit kernels fetch through the exemplar's textures, which
    // must be bound
    if (P.ex.hw && (!P.ex.tbase || !P.ex.tout)) return cudaErrorInvalidValue;
#define PT_TILED_DISPATCH(TMV, HWV)                                                                           \
    if (kind == 0 && wide) return launch_propagate_t<R, TMV, HWV, 1, kPropH>(P, M, work, arg, dependent, s);  \
    else if (kind == 0) return launch_propagate_t<R, TMV, HWV, 2, kPropH>(P, M, work, arg, dependent, s);     \
    else if (kind == 1 && wide)                                                                               \
        return launch_scatter_t<R, TMV, HWV, 4, kScatHWide>(P, M, work, arg, pass_id, dependent, s);          \
    else if (kind == 1) return launch_scatter_t<R, TMV, HWV, 2, kScatH>(P, M, work, arg, pass_id, dependent, s);\
    else if (wide && (P.inc.on || P.inc.fill))                                                                \
        return launch_residual_t<R, TMV, HWV, 4, kResidHWide, true>(P, M, out, dependent, s);                 \
    else if (wide) return launch_residual_t<R, TMV, HWV, 4, kResidHWide, false>(P, M, out, dependent, s);     \
    else if (P.inc.on || P.inc.fill)                                                                          \
        return launch_residual_t<R, TMV, HWV, HWV ? 1 : 2, kResidH, true>(P, M, out, dependent, s);           \
    else return launch_residual_t<R, TMV, HWV, HWV ? 1 : 2, kResidH, false>(P, M, out, dependent, s);
    if (P.ex.hw) {
        if (tm == TM_NONE) { PT_TILED_DISPATCH(TM_NONE, 1) }
        else if (tm == TM_FWD) { PT_TILED_DISPATCH(TM_FWD, 1) }
        else { PT_TILED_DISPATCH(TM_BWD, 1) }
    } else {
        if (tm == TM_NONE) { PT_TILED_DISPATCH(TM_NONE, 0) }
        else if (tm == TM_FWD) { PT_TILED_DISPATCH(TM_FWD, 0) }
        else { PT_TILED_DISPATCH(TM_BWD, 0) }
    }
#undef PT_TILED_DISPATCH
    return cudaGetLastError();
}

}  // namespace ptk
