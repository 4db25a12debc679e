// Per-dimension instantiation of the splat, neighbour and slice kernels.  This file is
// compiled once for each d in 1..16 with -DPGPU_D=d, so the sixteen variants build in
// parallel and each keeps its per-point arrays in registers.
#include "lattice_ops.h"

#ifndef PGPU_D
#error "compile with -DPGPU_D=<number of position dimensions>"
#endif

namespace pgpu {
namespace {

constexpr int D = PGPU_D;

int grid_cap(uint64_t work, int threads, int sms) {
    uint64_t g = (work + threads - 1) / threads;
    const uint64_t cap = (uint64_t)sms * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

SegSource<true> param_segs(const Segment* segs, int nseg) {
    SegSource<true> p;
    for (int k = 0; k < nseg; ++k) p.seg[k] = segs[k];
    return p;
}

template <int VDP, typename Acc>
void splat_t(const SplatArgs& a, cudaStream_t st) {
    if (a.blocks) splat_kernel<D, VDP, Acc><<<a.blocks, kSplatThreads, 0, st>>>(a);
}

template <int VDP>
void wide_tile_t(const SplatArgs& a, cudaStream_t st) {
    if constexpr (key_words(D) == 1)
        if (a.tile_blocks) wide_tile_kernel<D, VDP><<<a.tile_blocks, kWideTileThreads, 0, st>>>(a);
}

bool splat(const SplatArgs& a, int vdp, int payload, cudaStream_t st) {
    const bool f64 = payload == kPayloadF64;
    if (a.tile_blocks && (f64 || key_words(D) > 1)) return false;
    switch (vdp) {
    case 2: wide_tile_t<2>(a, st); break;
    case 4: wide_tile_t<4>(a, st); break;
    case 8: wide_tile_t<8>(a, st); break;
    }
    switch (vdp) {
    case 2: f64 ? splat_t<2, double>(a, st) : splat_t<2, float>(a, st); return true;
    case 4: f64 ? splat_t<4, double>(a, st) : splat_t<4, float>(a, st); return true;
    case 8: f64 ? splat_t<8, double>(a, st) : splat_t<8, float>(a, st); return true;
    }
    return false;
}

// One vertex per thread, in block order: the vertices looked up together are neighbours in the
// numbering and share the table's and the pairs' sectors, which blocks that stride over all of
// them lose once the table is larger than L2.  16 striding blocks per SM -> this: 14.3 M
// vertices of d=7 4.67 -> 3.62 ms, 10.2 M 2.93 -> 2.31, 1.0 M 0.099 -> 0.099; 5.4 M of d=10
// 1.39 -> 1.29.
void neighbours(const NbrArgs& a, uint32_t vmax, int, cudaStream_t st) {
    neighbours_kernel<D><<<vmax / 256 + 1, 256, 0, st>>>(a);
}

template <int VDP, typename A>
void slice_t(const SliceArgs& a, cudaStream_t st) {
    if (!a.blocks) return;
    if (a.rec && a.host_segs)
        slice_replay_kernel<D, VDP, A, true><<<a.blocks, kSliceThreads, 0, st>>>(a, param_segs(a.host_segs, a.nseg));
    else if (a.rec)
        slice_replay_kernel<D, VDP, A, false><<<a.blocks, kSliceThreads, 0, st>>>(a, SegSource<false>{});
    else
        slice_kernel<D, VDP, A><<<a.blocks, kSliceThreads, 0, st>>>(a);
}

// the slice reads the last blur pass's rows, plain (not homogeneous) products: FP64 for
// the FP64 lattice, FP32 otherwise; homogeneous lattices exist only for 16-bit payloads
template <int VDP>
bool slice_p(const SliceArgs& a, int payload, bool homog, cudaStream_t st) {
    switch (payload) {
    case kPayloadF32: slice_t<VDP, float>(a, st); return !homog;
    case kPayloadF16:
    case kPayloadBF16: slice_t<VDP, float>(a, st); return true;
    case kPayloadF64: slice_t<VDP, double>(a, st); return !homog;
    }
    return false;
}

bool slice(const SliceArgs& a, int vdp, int payload, bool homog, cudaStream_t st) {
    switch (vdp) {
    case 2: return slice_p<2>(a, payload, homog, st);
    case 4: return slice_p<4>(a, payload, homog, st);
    case 8: return slice_p<8>(a, payload, homog, st);
    }
    return false;
}

template <int VDP, int NP>
void compact_tile_t(const CompactSplatArgs& a, cudaStream_t st) {
    if constexpr (CompactKey<D>::kOneWord) {
        const size_t smem = tile_smem_bytes(D, NP);
        if (a.host_segs)
            compact_tile_kernel<D, VDP, NP, true><<<a.tile_blocks, kTileThreads, smem, st>>>(
                a, param_segs(a.host_segs, a.nseg));
        else
            compact_tile_kernel<D, VDP, NP, false><<<a.tile_blocks, kTileThreads, smem, st>>>(a, SegSource<false>{});
    }
}

template <int VDP>
bool compact_splat_t(const CompactSplatArgs& a, cudaStream_t st) {
    if (a.blocks) compact_direct_kernel<D, VDP><<<a.blocks, kDirectThreads, direct_smem_bytes(D), st>>>(a);
    if constexpr (CompactKey<D>::kOneWord) {
        if (a.tile_blocks) {
            if (a.tile_px == 1) compact_tile_t<VDP, 1>(a, st);
            else if (a.tile_px == 2) compact_tile_t<VDP, 2>(a, st);
            else return false;
        }
        return true;
    }
    return a.tile_blocks == 0;
}

bool compact_splat(const CompactSplatArgs& a, int vdp, cudaStream_t st) {
    switch (vdp) {
    case 2: return compact_splat_t<2>(a, st);
    case 4: return compact_splat_t<4>(a, st);
    case 8: return compact_splat_t<8>(a, st);
    }
    return false;
}

void compact_rank(const CompactRankArgs& a, int sms, cudaStream_t st) {
    compact_rank_kernel<D><<<grid_cap(a.cap, 256, sms), 256, 0, st>>>(a);
}

void compact_neighbours(const CompactNbrArgs& a, uint32_t vmax, int sms, cudaStream_t st) {
    compact_neighbours_kernel<D><<<grid_cap(vmax, 256, sms), 256, 0, st>>>(a);
}

template <int VDP>
void compact_slice_t(const CompactSliceArgs& a, cudaStream_t st) {
    if (!a.blocks) return;
    if constexpr (CompactKey<D>::kOneWord)
        compact_tile_slice_kernel<D, VDP><<<a.blocks, kTileThreads, tile_smem_bytes(D, kTileSlicePx), st>>>(a);
    else
        compact_slice_kernel<D, VDP><<<a.blocks, kSliceThreads, (size_t)(D + 1) * kSliceThreads * sizeof(uint2), st>>>(a);
}

bool compact_slice(const CompactSliceArgs& a, int vdp, cudaStream_t st) {
    switch (vdp) {
    case 2: compact_slice_t<2>(a, st); return true;
    case 4: compact_slice_t<4>(a, st); return true;
    case 8: compact_slice_t<8>(a, st); return true;
    }
    return false;
}

const DimOps kOps = {splat, neighbours, slice, compact_splat, compact_rank, compact_neighbours, compact_slice,
                     CompactKey<D>::kMaxQ};

}  // namespace

#define PGPU_CAT2(a, b) a##b
#define PGPU_CAT(a, b) PGPU_CAT2(a, b)
const DimOps* PGPU_CAT(dim_ops_, PGPU_D)() { return &kOps; }

}  // namespace pgpu
