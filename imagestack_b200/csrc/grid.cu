// The bilateral grid on the GPU: the GRID branch of GaussTransform::apply
// (src/GaussTransform.cpp:227-290), which JointBilateral::apply picks by default for at
// most four position channels (:553-564), with the reference's DenseGrid
// (src/DenseGrid.h): a dense grid over the positions' bounding box, multilinear splatting
// into the 2^d corners of each point's cell, two [1 2 1]/4 passes per dimension (taps 5),
// and multilinear slicing.
//
//   preview  min and max of every scaled guide channel (block reduction, then
//            order-preserving integer atomics: exact in any order); pixel coordinates grow
//            with the pixel, so the host takes theirs from the image's ends
//   splat    one to four pixels per thread; FP32 reductions into the corners (the reference
//            adds in point order, so sums agree to rounding)
//   blur     one launch per dimension, one thread per grid value: the reference's two
//            in-place passes (src/DenseGrid.h:199-236) evaluated out of place, cell by cell,
//            with their exact arithmetic, including the last cell's double-precision step
//   slice    one thread per point; the corners gathered in the reference's order
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "engine.h"

namespace pgpu {
namespace {

constexpr int kGridTaps = 5;        // GaussTransform::apply builds DenseGrid(d, vd, 5)
constexpr int kGridMaxD = 5;        // 2^d corners per point; the reference's AUTO uses d <= 4
constexpr int kGridMaxVd = 8;
constexpr int kGridThreads = 256;
constexpr long long kGridMaxCells = 1LL << 30;   // floats in the grid

struct GridArgs {
    int vd;
    float sf;                            // scaleFactor, the same in every dimension
    float minp[kGridMaxD];               // minPosition
    int sizes[kGridMaxD];
    uint32_t stride[kGridMaxD + 1];      // stride[0] = vd; grids hold at most 2^30 values
    float* grid;
    // Splat in pairs (two values per cell): grid[2*offset..] holds, for the cell at offset, its
    // own two values and what its points add to the next cell along dimension 0, so that
    // a point's two corners there take one reduction of four floats.
    int pairs;
};

// float <-> unsigned mapping that preserves order, for min/max by integer atomics
__device__ __forceinline__ unsigned ordered_bits(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
float unordered_float(unsigned u) {
    const unsigned b = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
    float f;
    memcpy(&f, &b, 4);
    return f;
}

// DenseGrid::preview (src/DenseGrid.h:142-160): the bounding box of position * scaleFactor, guide
// channels only.  Blocks stride over pieces of kMinmaxPixels pixels of a row.
constexpr uint32_t kMinmaxPixels = 4 * kGridThreads;
template <int D>
__global__ void __launch_bounds__(kGridThreads) grid_minmax_kernel(PointSource src, float sf, uint32_t pieces,
                                                                   uint32_t total, unsigned* mm) {
    __shared__ unsigned smin[D], smax[D];
    if (threadIdx.x < D) {
        smin[threadIdx.x] = 0xFFFFFFFFu;
        smax[threadIdx.x] = 0u;
    }
    __syncthreads();
    unsigned lo[D], hi[D];
#pragma unroll
    for (int c = 0; c < D; ++c) lo[c] = 0xFFFFFFFFu, hi[c] = 0u;
    // (64 bits: total may be as large as 2^32 - 1, which a 32-bit count would step over)
    for (uint64_t next = blockIdx.x; next < total; next += gridDim.x) {
        const uint32_t b = (uint32_t)next;
        const uint32_t row = b / pieces, x0 = (b - row * pieces) * kMinmaxPixels + threadIdx.x;
        const uint32_t t = row / (uint32_t)src.height, y = row - t * (uint32_t)src.height;
        const float* at = src.pos.base + (long long)t * src.pos.tstride + (long long)y * src.pos.ystride;
#pragma unroll
        for (int c = 0; c < D; ++c, at += src.pos.cstride) {
            if (c >= src.pos_channels) break;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t x = x0 + k * kGridThreads;
                if (x >= (uint32_t)src.width) break;
                const unsigned o = ordered_bits(__fmul_rn(__fmul_rn(__ldg(at + x), src.pos_scale[c]), sf));
                lo[c] = min(lo[c], o);
                hi[c] = max(hi[c], o);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < D; ++c) {
        if (c >= src.pos_channels) break;
        lo[c] = __reduce_min_sync(0xFFFFFFFFu, lo[c]);
        hi[c] = __reduce_max_sync(0xFFFFFFFFu, hi[c]);
        if ((threadIdx.x & 31u) == 0) {
            atomicMin(&smin[c], lo[c]);
            atomicMax(&smax[c], hi[c]);
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < src.pos_channels) {
        atomicMin(&mm[threadIdx.x], smin[threadIdx.x]);
        atomicMax(&mm[D + threadIdx.x], smax[threadIdx.x]);
    }
}

// DenseGrid::query (src/DenseGrid.h:240-285): integral cell and fractions of one point
template <int D>
__device__ __forceinline__ void grid_cell(const GridArgs& g, const float (&p)[D], int (&I)[D], float (&F)[D],
                                          float (&Fi)[D]) {
#pragma unroll
    for (int c = 0; c < D; ++c) {
        const float f = __fsub_rn(__fmul_rn(p[c], g.sf), g.minp[c]);
        I[c] = (int)(short)floorf(f);
        F[c] = __fsub_rn(f, (float)I[c]);
        Fi[c] = __fsub_rn(1.0f, F[c]);
    }
}

// The cell's base offset, and which of its upper corners lie inside the grid (bit j: the
// corners one step up along dimension j); false if the cell itself is outside.  A corner
// past the grid's last cell has weight exactly 0 (the point lies on the last plane) and is
// skipped, as DenseGrid::query's bounds checks do.
template <int D>
__device__ __forceinline__ bool grid_base(const GridArgs& g, const int (&I)[D], uint32_t& base, unsigned& hi_ok) {
    base = 0;
    hi_ok = 0;
    bool ok = true;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        ok = ok && I[j] >= 0 && I[j] < g.sizes[j];
        base += (uint32_t)I[j] * g.stride[j];
        if (I[j] + 1 < g.sizes[j]) hi_ok |= 1u << j;
    }
    return ok;
}

// Corner `corner` of the cell (unrolled by the caller): its weight in the reference's
// product order and its offset from the cell's base.  (Corners share the first products.)
template <int D>
__device__ __forceinline__ float grid_corner_weight(const float (&F)[D], const float (&Fi)[D], int corner) {
    float w = (corner & 1) ? F[0] : Fi[0];   // 1 * it
#pragma unroll
    for (int j = 1; j < D; ++j) w = __fmul_rn(w, ((corner >> j) & 1) ? F[j] : Fi[j]);
    return w;
}
template <int D>
__device__ __forceinline__ uint32_t grid_corner_offset(const GridArgs& g, int corner) {
    uint32_t off = 0;
#pragma unroll
    for (int j = 0; j < D; ++j)
        if ((corner >> j) & 1) off += g.stride[j];
    return off;
}

// Blocks of the splat and slice: tiles of (bw * kp) x (kGridThreads/bw) pixels of one frame
// (bw = 32 for images, kGridThreads for point lists of one row; kp consecutive pixels of a
// row per thread), so a thread finds its pixels without dividing.
struct PixelTiles {
    unsigned bshift;   // log2 of bw
    dim3 grid;
};
PixelTiles pixel_tiles(const PointSource& s, unsigned kp) {
    PixelTiles t;
    t.bshift = s.height == 1 ? 8u : 5u;
    static_assert(kGridThreads == 256, "bw of a one-row tile");
    const unsigned bw = 1u << t.bshift, bh = kGridThreads / bw, w = bw * kp;
    t.grid = dim3(((unsigned)s.width + w - 1) / w, ((unsigned)s.height + bh - 1) / bh, (unsigned)s.frames);
    return t;
}

// the splat's reduction of one corner: VD values of a cell are 8- or 16-byte aligned when VD is
// 2 or 4, so one vector reduction adds them; otherwise one float atomic per value
__device__ __forceinline__ void red4(float* p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                 :: "l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
template <int VD>
__device__ __forceinline__ void grid_add(const GridArgs& g, uint32_t off, const float* c) {
    if constexpr (VD == 2) {
        asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" :: "l"(g.grid + off), "f"(c[0]), "f"(c[1]) : "memory");
    } else if constexpr (VD == 4) {
        red4(g.grid + off, c[0], c[1], c[2], c[3]);
    } else {
#pragma unroll
        for (int k = 0; k < kGridMaxVd; ++k)
            if (k < g.vd) atomicAdd(g.grid + off + k, c[k]);
    }
}

// KP consecutive pixels of a row per thread.  With KP > 1 (small grids: the 2^D corners x
// VD values fit in registers) a run of pixels that fall into the same cell is summed in
// registers first and sent as one set of corner reductions: neighbouring pixels share cells,
// and the splat is bound by the reductions' rate.  The sums differ from the reference's
// point-by-point additions only in rounding order.  PAIRS: GridArgs::pairs, half as many
// reductions (4K grey d=3: see run_grid).
template <int D, int VD, int KP, bool PAIRS>
__global__ void __launch_bounds__(kGridThreads) grid_splat_kernel(PointSource src, unsigned bshift, GridArgs g) {
    static_assert(!PAIRS || (VD == 2 && KP > 1), "pairs hold two values per cell");
    constexpr int NC = 1 << D;
    constexpr int NV = VD > 0 ? VD : kGridMaxVd;
    const uint32_t x0 = ((blockIdx.x << bshift) + (threadIdx.x & ((1u << bshift) - 1u))) * KP;
    const uint32_t y = blockIdx.y * (kGridThreads >> bshift) + (threadIdx.x >> bshift);
    if (x0 >= (uint32_t)src.width || y >= (uint32_t)src.height) return;
    float acc[KP > 1 ? NC : 1][NV];
    uint32_t run_base = 0xFFFFFFFFu;   // no run: no grid has this offset
    unsigned run_hi = 0;
    auto flush = [&]() {
        if (run_base == 0xFFFFFFFFu) return;
#pragma unroll
        for (int corner = 0; corner < NC; ++corner) {
            if (PAIRS && (corner & 1)) continue;
            if (corner & ~run_hi) continue;
            const uint32_t off = run_base + grid_corner_offset<D>(g, corner);
            // (the next cell's half of a pair whose next cell lies outside is never read)
            if constexpr (PAIRS) {
                const float* lo = acc[KP > 1 ? corner : 0];
                const float* hi = acc[KP > 1 ? corner + 1 : 0];
                red4(g.grid + 2 * (size_t)off, lo[0], lo[1], hi[0], hi[1]);
            } else {
                grid_add<VD>(g, off, acc[KP > 1 ? corner : 0]);
            }
        }
    };
#pragma unroll
    for (int kp = 0; kp < KP; ++kp) {
        const uint32_t x = x0 + kp;
        if (x >= (uint32_t)src.width) break;
        float p[D], v[NV];
        load_point_xyt<D, NV>(src, x, y, blockIdx.z, p, v);
        int I[D];
        float F[D], Fi[D];
        grid_cell<D>(g, p, I, F, Fi);
        uint32_t base;
        unsigned hi_ok;
        if (!grid_base<D>(g, I, base, hi_ok)) continue;
        if constexpr (KP > 1) {
            if (base != run_base) {   // a new cell: send the run so far, start a new one
                flush();
                run_base = base;
                run_hi = hi_ok;
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int k = 0; k < NV; ++k) acc[c][k] = 0.0f;
            }
#pragma unroll
            for (int corner = 0; corner < NC; ++corner) {
                const float w = grid_corner_weight<D>(F, Fi, corner);
#pragma unroll
                for (int k = 0; k < NV; ++k) acc[corner][k] = __fadd_rn(acc[corner][k], __fmul_rn(w, v[k]));
            }
        } else {
#pragma unroll
            for (int corner = 0; corner < NC; ++corner) {
                if (corner & ~hi_ok) continue;
                const float w = grid_corner_weight<D>(F, Fi, corner);
                float c[NV];
#pragma unroll
                for (int k = 0; k < NV; ++k) c[k] = __fmul_rn(w, v[k]);
                grid_add<VD>(g, base + grid_corner_offset<D>(g, corner), c);
            }
        }
    }
    if constexpr (KP > 1) flush();
}

// The two [1 2 1]/4 passes of DenseGrid::blur_ (src/DenseGrid.h:186-238) along dimension j
// (taps 5: taps/2 passes).  The reference walks each row in place, but every value a pass
// writes depends only on values from before that pass (row[x] is overwritten after both
// row[x] and row[x+1] were read, and the running tmp carries 0.5*(old[x-1] + old[x])), so
// each cell is computed independently here, out of place, with the same single-precision
// operations in the same order:
//   x = 0:           0.5*(old[0]/2 + 0.5*(old[0] + old[1]))
//   0 < x < len-1:   0.5*(0.5*(old[x-1] + old[x]) + 0.5*(old[x] + old[x+1]))
//   x = len-1:       0.5*(tmp + 0.5*old[len-1]) in double (the reference's double literals),
//                    tmp = 0.5*(old[len-2] + old[len-1]) in single, or old[0]/2 when len == 1
// The second pass at x needs the first pass at x-1, x and x+1, which each thread evaluates
// from the five values around x.  One thread per grid value; consecutive threads are
// consecutive values, so every access is coalesced whatever the dimension.
__device__ __forceinline__ float grid_pass_value(float left, float here, float right, uint32_t x, uint32_t len) {
    // (here / 2 and 0.5 * here round alike)
    const float t1 = x == 0 ? __fmul_rn(0.5f, here) : __fmul_rn(0.5f, __fadd_rn(left, here));
    if (x == len - 1) return (float)__dmul_rn(0.5, __dadd_rn((double)t1, __dmul_rn(0.5, (double)here)));
    return __fmul_rn(0.5f, __fadd_rn(t1, __fmul_rn(0.5f, __fadd_rn(here, right))));
}

// ms, ml: floor(2^32 / stride) and floor(2^32 / len) (div_magic).  pairs: dimension 0 of a grid
// splatted in pairs.
__global__ void __launch_bounds__(kGridThreads) grid_blur_kernel(const float* src, float* dst, uint32_t total,
                                                                 uint32_t s, uint32_t ms, uint32_t len, uint32_t ml,
                                                                 int pairs) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;   // grids hold at most 2^30 values
    if (t >= total) return;
    uint32_t rem, x;
    div_magic(div_magic(t, s, ms, &rem), len, ml, &x);
    // old values at x-2 .. x+2 (those outside the row are never used)
    float o[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int xx = (int)x + k - 2;
        o[k] = 0.0f;
        if (xx < 0 || xx >= (int)len) continue;
        const int64_t at = (int64_t)t + (int64_t)(k - 2) * s;
        if (pairs) {   // s == 2: the cell's own two values, and the previous cell's for it
            const int64_t cell = at >> 1, c = at & 1;
            o[k] = src[4 * cell + c];
            if (xx > 0) o[k] = __fadd_rn(o[k], src[4 * (cell - 1) + 2 + c]);
        } else {
            o[k] = src[at];
        }
    }
    // first pass at x-1, x, x+1, then the second pass at x
    float p1[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int xx = (int)x + k - 1;
        p1[k] = (xx >= 0 && xx < (int)len) ? grid_pass_value(o[k], o[k + 1], o[k + 2], (uint32_t)xx, len) : 0.0f;
    }
    dst[t] = grid_pass_value(p1[0], p1[1], p1[2], x, len);
}

template <int D, int VD>
__global__ void __launch_bounds__(kGridThreads) grid_slice_kernel(PointSource src, unsigned bshift, GridArgs g,
                                                                  OutView out) {
    constexpr int NV = VD > 0 ? VD : kGridMaxVd;
    const int vd = VD > 0 ? VD : g.vd;
    const uint32_t x = (blockIdx.x << bshift) + (threadIdx.x & ((1u << bshift) - 1u));
    const uint32_t y = blockIdx.y * (kGridThreads >> bshift) + (threadIdx.x >> bshift);
    if (x >= (uint32_t)src.width || y >= (uint32_t)src.height) return;
    float p[D];
    load_position_xyt<D>(src, x, y, blockIdx.z, p);
    int I[D];
    float F[D], Fi[D];
    grid_cell<D>(g, p, I, F, Fi);
    float acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0f;
    uint32_t base;
    unsigned hi_ok;
    const bool inside = grid_base<D>(g, I, base, hi_ok);
#pragma unroll
    for (int corner = 0; corner < (1 << D); ++corner) {
        if (!inside || (corner & ~hi_ok)) continue;
        const float w = grid_corner_weight<D>(F, Fi, corner);
        const float* cell = g.grid + base + grid_corner_offset<D>(g, corner);
        float c[NV];
        if constexpr (VD == 2) {
            const float2 q = __ldg(reinterpret_cast<const float2*>(cell));
            c[0] = q.x, c[1] = q.y;
        } else if constexpr (VD == 4) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(cell));
            c[0] = q.x, c[1] = q.y, c[2] = q.z, c[3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < NV; ++k) c[k] = k < vd ? cell[k] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < NV; ++k)
            if (k < vd) acc[k] = __fadd_rn(acc[k], __fmul_rn(w, c[k]));
    }
    float* o = out.base + (long long)blockIdx.z * out.tstride + (long long)y * out.ystride + x;
    float wsum = acc[0];
#pragma unroll
    for (int k = 0; k < NV; ++k) if (k == vd - 1) wsum = acc[k];
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (k < out.channels) o[(long long)k * out.cstride] = out.normalize ? acc[k] / wsum : acc[k];
}

template <int D>
void launch_minmax(const PointSource& s, float sf, unsigned* mm, int sms, cudaStream_t st) {
    const uint32_t pieces = ((uint32_t)s.width + kMinmaxPixels - 1) / kMinmaxPixels;
    const uint32_t total = pieces * (uint32_t)s.height * (uint32_t)s.frames;   // at most the points
    const uint32_t blocks = std::min(total, (uint32_t)sms * 8u);
    grid_minmax_kernel<D><<<blocks, kGridThreads, 0, st>>>(s, sf, pieces, total, mm);
}
// Pixels of a run are summed in registers where the corner sums fit (2^d x vd <= 16), and
// pairs halve the reductions of two values per cell (4K grey d=3: 66 M reductions of two floats
// one by one 0.90 ms, runs 0.23 ms, runs in pairs 0.11).
bool splat_in_pairs(int d, int vd, long long values) {
    return vd == 2 && d <= 3 && values <= (1LL << 28);   // the pairs take twice the grid's memory
}
template <int D>
void launch_splat(const PointSource& s, uint32_t n, const GridArgs& g, cudaStream_t st) {
    if (!n) return;
    if constexpr (D <= 3) {
        if (g.vd == 2) {
            const PixelTiles t = pixel_tiles(s, 4);
            if (g.pairs) grid_splat_kernel<D, 2, 4, true><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g);
            else grid_splat_kernel<D, 2, 4, false><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g);
            return;
        }
    }
    if constexpr (D <= 2) {
        if (g.vd == 4) {
            const PixelTiles t = pixel_tiles(s, 4);
            grid_splat_kernel<D, 4, 4, false><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g);
            return;
        }
    }
    const PixelTiles t = pixel_tiles(s, 1);
    if (g.vd == 2) grid_splat_kernel<D, 2, 1, false><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g);
    else if (g.vd == 4) grid_splat_kernel<D, 4, 1, false><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g);
    else grid_splat_kernel<D, 0, 1, false><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g);
}
template <int D>
void launch_slice(const PointSource& s, uint32_t n, const GridArgs& g, const OutView& o, cudaStream_t st) {
    if (!n) return;
    const PixelTiles t = pixel_tiles(s, 1);
    if (g.vd == 2) grid_slice_kernel<D, 2><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g, o);
    else if (g.vd == 4) grid_slice_kernel<D, 4><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g, o);
    else grid_slice_kernel<D, 0><<<t.grid, kGridThreads, 0, st>>>(s, t.bshift, g, o);
}

// Bounds of the pixel-coordinate dimensions of s, folded into lo and hi: x * scale * scaleFactor,
// with the kernels' roundings, never decreases (scale > 0) or increases from pixel to pixel.
void coordinate_bounds(const PointSource& s, float sf, float* lo, float* hi, bool first) {
    const int last[3] = {s.width - 1, s.height - 1, s.frames - 1};
    int c = s.pos_channels;
    for (int k = 0; k < 3; ++k) {
        if (!((s.coord_mask >> k) & 1)) continue;
        for (int end = 0; end < 2; ++end) {
            volatile float p = (float)(uint32_t)(end ? last[k] : 0) * s.coord_scale[k];
            volatile float q = p * sf;
            const float v = q;
            if ((first && end == 0) || v < lo[c] || !std::isfinite(v)) lo[c] = v;
            if ((first && end == 0) || v > hi[c] || !std::isfinite(v)) hi[c] = v;
        }
        ++c;
    }
}

#define PGPU_GRID_DISPATCH(d, call)          \
    switch (d) {                             \
    case 1: { constexpr int DD = 1; call; } break; \
    case 2: { constexpr int DD = 2; call; } break; \
    case 3: { constexpr int DD = 3; call; } break; \
    case 4: { constexpr int DD = 4; call; } break; \
    case 5: { constexpr int DD = 5; call; } break; \
    }

}  // namespace

int run_grid(Engine& E, const LatticeJob& J, cudaStream_t st) {
    const int d = J.d, vd = J.vd;
    if (d < 1 || d > kGridMaxD)
        return fail(PGPU_ERR_UNSUPPORTED, "the grid method takes 1..%d position dimensions (got %d)",
                    kGridMaxD, d);
    if (vd < 1 || vd > kGridMaxVd) return fail(PGPU_ERR_UNSUPPORTED, "%d value channels", vd);
    if (J.payload != kPayloadF32) return fail(PGPU_ERR_UNSUPPORTED, "the grid method computes in FP32 only");
    for (const PointSource* ps : {&J.splat, &J.slice}) {   // the launches' grid dimensions
        if (ps == &J.slice && J.replay) continue;
        if (ps->frames > 65535 || (ps->height > 1 && ps->height > 65535 * (kGridThreads / 32)))
            return fail(PGPU_ERR_UNSUPPORTED, "the grid method takes at most 65535 frames and %d rows",
                        65535 * (kGridThreads / 32));
    }
    // DenseGrid's constructor (src/DenseGrid.h:111-127): sqrtf(1.0/3 + (taps-1)*0.25)
    const float sf = sqrtf((float)(1.0 / 3 + (kGridTaps - 1) * 0.25));
    const PointSource& sl = J.replay ? J.splat : J.slice;
    const uint32_t nsl = J.replay ? J.n : J.n_slice;
    int rc;
    if ((rc = E.meta.ensure(64))) return rc;
    unsigned* mm = (unsigned*)E.meta.p;
    CUDA_TRY(cudaEventRecord(E.ev[0], st));
    CUDA_TRY(cudaMemsetAsync(mm, 0xFF, sizeof(unsigned) * d, st));
    CUDA_TRY(cudaMemsetAsync(mm + d, 0, sizeof(unsigned) * d, st));
    if (J.splat.pos_channels) {
        PGPU_GRID_DISPATCH(d, launch_minmax<DD>(J.splat, sf, mm, E.sms, st));
        if (!J.replay) PGPU_GRID_DISPATCH(d, launch_minmax<DD>(sl, sf, mm, E.sms, st));
    }
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(E.hstat, mm, sizeof(unsigned) * 2 * d, cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    float lows[kGridMaxD], highs[kGridMaxD];
    for (int i = 0; i < J.splat.pos_channels; ++i) {
        lows[i] = unordered_float(E.hstat[i]);
        highs[i] = unordered_float(E.hstat[d + i]);
    }
    coordinate_bounds(J.splat, sf, lows, highs, true);
    if (!J.replay) coordinate_bounds(sl, sf, lows, highs, false);

    GridArgs g;
    memset(&g, 0, sizeof(g));
    g.vd = vd;
    g.sf = sf;
    g.stride[0] = (uint32_t)vd;
    long long cells = vd;   // values in the grid
    for (int i = 0; i < d; ++i) {
        const float lo = lows[i], hi = highs[i];
        if (!std::isfinite(lo) || !std::isfinite(hi))
            return fail(PGPU_ERR_ARGUMENT, "positions are not finite");
        g.minp[i] = lo;
        const float span = hi - lo;   // float subtraction, as maxPosition[i] - minPosition[i]
        g.sizes[i] = (int)(std::ceil(span) + 1);
        cells *= g.sizes[i];
        if (g.sizes[i] < 1 || cells > kGridMaxCells)
            return fail(PGPU_ERR_CAPACITY, "the grid would need more than %lld cells", kGridMaxCells);
        g.stride[i + 1] = (uint32_t)cells;
    }
    g.pairs = splat_in_pairs(d, vd, cells) ? 1 : 0;
    const size_t splat_values = (size_t)cells << g.pairs;
    if ((rc = E.grid.ensure(splat_values * sizeof(float))) ||
        (rc = E.grid2.ensure((size_t)cells * sizeof(float))))
        return rc;
    g.grid = (float*)E.grid.p;
    CUDA_TRY(cudaMemsetAsync(g.grid, 0, splat_values * sizeof(float), st));
    CUDA_TRY(cudaEventRecord(E.ev[1], st));
    PGPU_GRID_DISPATCH(d, launch_splat<DD>(J.splat, J.n, g, st));
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaEventRecord(E.ev[3], st));
    // one launch per dimension (both of its passes), ping-ponging between the grid and a
    // second buffer
    static_assert(kGridTaps / 2 == 2, "grid_blur_kernel fuses exactly two passes");
    float* bufs[2] = {g.grid, (float*)E.grid2.p};
    int cur = 0;
    const unsigned blur_blocks = (unsigned)((cells + kGridThreads - 1) / kGridThreads);
    for (int j = 0; j < d; ++j, cur ^= 1)
        grid_blur_kernel<<<blur_blocks, kGridThreads, 0, st>>>(
            bufs[cur], bufs[cur ^ 1], (uint32_t)cells, g.stride[j], magic_of(g.stride[j]), (uint32_t)g.sizes[j],
            magic_of((uint32_t)g.sizes[j]), j == 0 ? g.pairs : 0);
    g.grid = bufs[cur];
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaEventRecord(E.ev[4], st));
    PGPU_GRID_DISPATCH(d, launch_slice<DD>(sl, nsl, g, J.out, st));
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaEventRecord(E.ev[5], st));
    CUDA_TRY(cudaStreamSynchronize(st));

    pgpu_stats s;
    memset(&s, 0, sizeof(s));
    s.points = J.n;
    s.vertices = cells / vd;        // grid cells
    s.capacity = cells / vd;
    s.d = d;
    s.vd = vd;
    s.payload = J.payload;
    cudaEventElapsedTime(&s.ms_splat, E.ev[1], E.ev[3]);
    cudaEventElapsedTime(&s.ms_compact, E.ev[0], E.ev[1]);   // the bounding-box preview
    cudaEventElapsedTime(&s.ms_blur, E.ev[3], E.ev[4]);
    cudaEventElapsedTime(&s.ms_slice, E.ev[4], E.ev[5]);
    cudaEventElapsedTime(&s.ms_total, E.ev[0], E.ev[5]);
    set_stats(s);
    return PGPU_OK;
}

}  // namespace pgpu
