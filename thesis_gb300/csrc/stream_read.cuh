// stream_read.cuh -- a 3-D FP32 grid read once by the streaming sweep's code
// (stream_body.cuh) for something else than a sweep: the residual norm
// (k_util.cu) and the refinement's residual (k_ir.cu).
#pragma once

#include <algorithm>

#include "host.hpp"
#include "stream_body.cuh"

namespace st {

// One row per thread: with two (as the sweeps of large grids at R >= 3) the
// outputs' own work makes the passes 5 to 10 % slower.
template <int R> struct ReadTile {
    static constexpr int TY = 16, RY = 1, NS = R <= 2 ? 16 : 8;
};
template <int R>
using ReadShape = StreamShape<R, 128, ReadTile<R>::TY, ReadTile<R>::RY, ReadTile<R>::NS>;

// Out: a thread's share of the result, made from its arguments (Out::Args)
// and given its rows (see stream3d_sweeps); finish() is called by the whole
// CTA at the end.
template <int R, class Out>
__global__ void __launch_bounds__(ReadShape<R>::THREADS, ReadShape<R>::MIN_BLOCKS)
    k_stream_read(const __grid_constant__ CUtensorMap map, Geom g, int tiles_x, int tiles_y, int zchunk,
                  int items, typename Out::Args a) {
    using S = ReadShape<R>;
    constexpr int NS = ReadTile<R>::NS;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float *ring = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) &
                                            ~static_cast<uintptr_t>(127));
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + NS * S::SLOT_FLOATS);
    uint64_t *empty = full + NS, *swept = empty + NS;
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map);
        for (int s = 0; s < NS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], S::CWARPS);
        }
        fence_mbar_init();
    }
    __syncthreads();
    Out out(a, g);
    stream3d_sweeps<R, 128, ReadTile<R>::TY, ReadTile<R>::RY, NS, false, false, Out>(ring, full, empty, swept, &map, &map, nullptr, nullptr,
                                                          g, tiles_x, tiles_y, zchunk, items, 1, nullptr, 0u,
                                                          blockIdx.x, gridDim.x, false, &out);
    __syncthreads();
    out.finish();
}

// On at most max_ctas CTAs; *ctas: as many as were launched.
template <int R, class Out>
int launch_stream_read(const Geom &g, const float *u, typename Out::Args a, int max_ctas, cudaStream_t s, int *ctas) {
    using S = ReadShape<R>;
    const void *fn = reinterpret_cast<const void *>(k_stream_read<R, Out>);
    int resident = 0, tiles_x, tiles_y, zchunk, items;
    int rc = grid_resident_ctas(fn, S::THREADS, S::SMEM_BYTES, &resident);
    if (rc) return rc;
    if (resident < 1) return fail(STENCIL_EUNSUPPORTED, "stream kernel does not fit on an SM");
    resident = std::min(resident, max_ctas);
    stream3d_plan(g, 128, ReadTile<R>::TY, resident, &tiles_x, &tiles_y, &zchunk, &items);
    *ctas = std::min(items, resident);
    CUtensorMap map;
    const long long dims[3] = {g.nx, g.ny, g.nz};
    const int box[3] = {S::PW, S::PH, 1};
    rc = make_tensor_map(&map, u, 3, dims, box, g.sy, true);
    if (rc) return rc;
    Geom gg = g;
    void *args[] = {&map, &gg, &tiles_x, &tiles_y, &zchunk, &items, &a};
    ST_CUDA(cudaLaunchKernel(fn, dim3(*ctas), dim3(S::THREADS), args, S::SMEM_BYTES, s));
    return STENCIL_OK;
}

}  // namespace st
