// reg2d_body.cuh -- every sweep of a small 2-D grid (R = 1, JACOBI) by one
// CTA with the grid in registers.
//
// A row of at most 4 * LW cells lies across LW lanes (4 consecutive cells
// each), a thread holds its chunk column of a block of RW rows, and the
// blocks of the CTA's NT / LW lane groups cover the grid.  In a sweep the
// y-neighbours inside a block are the thread's own registers, the
// x-neighbours come from the adjacent lanes by shuffles, and only the first
// and last row of each block go through shared memory (double-buffered by
// sweep parity, so one CTA barrier per sweep).  A sweep from shared memory
// spends three 16-byte loads and a 16-byte store per 4 cells (16 wavefronts, of
// which an SM serves one a cycle); here it is 16 FP32 instructions and two
// shuffles over four schedulers, and FP32 issue bounds it.  GB300, 304 grids of
// 128^2, GCell/s: 12 warps of 11 rows, one CTA per SM 5216 (4853 without the
// inner rows first); 16 warps of 8 rows 4829; two CTAs per SM of 8 warps of 16
// rows 4013 and of 16 warps of 8 rows 3502 (registers spill at their limits);
// packed f32x2 sums 4835 (the sums' pairs are not aligned).  From shared memory
// the same batch ran at 975.
//
// The border band must be equal in both buffers (bit for bit), since the
// registers hold one state; the caller takes another path where
// reg2d_borders_equal says otherwise.  Sums keep the reference's order (left,
// right, row above, row below); the sum starts from its first term and the
// division is fma(s, 1/4, +0): the reference's leading +0 only matters for an
// all-(-0) sum, which the +0 addend maps to +0.
#pragma once

#include "common.cuh"

namespace st {

// Whether the border bands (width 1) of the nx x ny grids a and b (row pitch
// px) hold the same bits; the CTA's threads agree.
__device__ __forceinline__ bool reg2d_borders_equal(const float *a, const float *b, int nx, int ny, int px) {
    const unsigned *ua = reinterpret_cast<const unsigned *>(a), *ub = reinterpret_cast<const unsigned *>(b);
    bool same = true;
    for (int x = threadIdx.x; x < nx; x += blockDim.x) {
        const int last = (ny - 1) * px + x;
        same &= ua[x] == ub[x] && ua[last] == ub[last];
    }
    for (int y = threadIdx.x; y < ny; y += blockDim.x) {
        const int first = y * px, last = first + nx - 1;
        same &= ua[first] == ub[first] && ua[last] == ub[last];
    }
    return __syncthreads_and(same) != 0;
}

// The update of one chunk: left and right neighbours l and r, rows above and
// below.  Cells outside the mask keep their value; where ALL is not set, only
// the first and last cell of a chunk can be outside (a width that is a
// multiple of 4).
template <bool ALL>
__device__ __forceinline__ float4 reg2d_chunk(float4 c, float4 up, float4 dn, float l, float r, unsigned mask) {
    const float x = fmaf(((l + c.y) + up.x) + dn.x, 0.25f, 0.0f), y = fmaf(((c.x + c.z) + up.y) + dn.y, 0.25f, 0.0f);
    const float z = fmaf(((c.y + c.w) + up.z) + dn.z, 0.25f, 0.0f), w = fmaf(((c.z + r) + up.w) + dn.w, 0.25f, 0.0f);
    return make_float4(mask & 1u ? x : c.x, !ALL || (mask & 2u) ? y : c.y, !ALL || (mask & 4u) ? z : c.z,
                       mask & 8u ? w : c.w);
}

// Shared memory of a CTA of NT threads: per sweep parity, every thread's
// first and last row, and before the last rows the grid's first row.
template <int NT>
struct Reg2dHalo {
    float4 first[2][NT + 32], last[2][NT + 32];
};

// iters sweeps of the nx x ny grid (row pitch px, a multiple of 4 and at most
// 4 * LW; ny - 1 at most RW * NT / LW) between a (the initial state) and b,
// which end as the ping-pong loop leaves them.  ALL: nx is not a multiple of
// 4.  Every thread of the CTA (NT of them) calls it.
template <int LW, int RW, int NT, bool ALL>
__device__ __forceinline__ void reg2d_sweeps(float *a, float *b, int nx, int ny, int px, int iters,
                                             Reg2dHalo<NT> &halo) {
    static_assert(RW >= 3 && NT % LW == 0, "row blocks with inner rows");
    if (iters < 1) return;
    const int tid = threadIdx.x, lane = tid % LW, x0 = 4 * lane;
    const int y0 = 1 + tid / LW * RW;  // row 0 never changes: it stays in shared memory
    unsigned mask = 0;                 // this lane's cells inside the update region
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (x0 + e >= 1 && x0 + e < nx - 1) mask |= 1u << e;
    const int nlive = min(max(ny - 1 - y0, 0), RW);  // rows of the block inside it
    float4 v[RW];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        v[r] = zero;
        if (y0 + r < ny && x0 < px) v[r] = *reinterpret_cast<const float4 *>(a + (y0 + r) * px + x0);
    }
    if (tid < LW) {
        const float4 top = x0 < px ? *reinterpret_cast<const float4 *>(a + x0) : zero;
        halo.last[0][tid] = halo.last[1][tid] = top;
        halo.first[0][NT + tid] = halo.first[1][NT + tid] = zero;  // below the last block: no update reads it
    }
    auto store = [&](float *g) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
            if (r < nlive && x0 < px) *reinterpret_cast<float4 *>(g + (y0 + r) * px + x0) = v[r];
    };
    // rows of the warp's fullest block, and whether all its blocks have them
    const int rows = __reduce_max_sync(0xffffffffu, nlive);
    const bool even = __all_sync(0xffffffffu, nlive == rows);
    auto row = [&](const float4 &c, const float4 &up, const float4 &dn) {
        const float l = __shfl_up_sync(0xffffffffu, c.w, 1, LW);
        const float q = __shfl_down_sync(0xffffffffu, c.x, 1, LW);
        return reg2d_chunk<ALL>(c, up, dn, l, q, mask);
    };
    auto sweep = [&](const float4 &up, const float4 &dn) {
        if (even && rows == RW) {
            // inner rows first: the rows from shared memory arrive meanwhile
            const float4 old1 = v[1], old2 = v[RW - 2];
            float4 prev = v[0];
#pragma unroll
            for (int r = 1; r < RW - 1; ++r) {
                const float4 c = v[r];
                v[r] = row(c, prev, v[r + 1]);
                prev = c;
            }
            v[0] = row(v[0], up, old1);
            v[RW - 1] = row(v[RW - 1], old2, dn);
            return;
        }
        float4 prev = up;
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            if (r >= rows) break;
            const float4 c = v[r];
            const float4 n = row(c, prev, r + 1 < RW ? v[r + 1] : dn);
            if (LW == 32 || even || r < nlive) v[r] = n;
            prev = c;
        }
    };
    // all sweeps but the last, the state before the last to its buffer, the
    // last sweep, the result
    int par = 0;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll 1
        for (int it = pass ? 1 : iters - 1; it > 0; --it, par ^= 1) {
            halo.first[par][tid] = v[0];
            halo.last[par][LW + tid] = v[RW - 1];
            __syncthreads();
            const float4 up = halo.last[par][tid], dn = halo.first[par][tid + LW];
            sweep(up, dn);
        }
        store((iters & 1) == pass ? b : a);
    }
    __syncthreads();  // the halo rows are reused by the next grid
}

}  // namespace st
