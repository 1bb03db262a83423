// rows_body.cuh -- one sweep of a 2-D grid by register-queue chunk columns,
// the per-CTA part of the persistent 2-D rows kernel (k_rows2d.cu) and of the
// one-launch batch kernel (k_batch1.cu).
//
// A thread owns one float4 chunk column of a block of hb rows: it keeps the
// column's rows j-R .. j+R in a register queue (one new 16-byte load per
// row, the smem_register idea of src/stencils.cu:71-83 on registers) and
// takes the x-neighbours from the lanes beside it, so a 4-cell update costs
// one 16-byte load at any R <= 4.  Items (chunk column, row block) are spread
// over the nctas CTAs that share the grid with a grid stride; consecutive
// threads take consecutive chunk columns, so a warp's loads and stores are
// contiguous 512-byte segments.  Loads are ld.global.cg (L2) or, with L1,
// plain L1-cached loads: a buffer is rewritten every other sweep inside one
// launch, and the plain form relies on every read of another CTA's writes
// following an acquire at GPU scope and a CTA barrier (then weak loads
// observe those writes).  Every cell keeps the
// reference's summation order (axis i offsets -R..-1, +1..+R, then axis j,
// from +0) and division; cells outside the update region are never written.
#pragma once

#include "common.cuh"

namespace st {

// What a chunk's x-neighbours give: R cells, read by the first and the last
// lane of a warp only.
template <int R> struct RowsEdge { using V = float4; };
template <> struct RowsEdge<1> { using V = float; };
template <> struct RowsEdge<2> { using V = float2; };

// One sweep src -> dst of a 2-D grid (g.sy: the row pitch, a multiple of 4;
// the chunk columns cover it) by CTA `cta` of the nctas CTAs of NT threads
// that share it; hb rows per block, nblk blocks.  The loads of D rows are in
// flight ahead of the row that is computed: its rows and those make one ring
// of K registers, whose index is static (the row loop is unrolled K times).
// Every lane of a warp walks the same number of rows, also where it has
// nothing to store, because its neighbours take their x-neighbours from it.
template <int R, int NT, int D, bool L1 = false>
__device__ __forceinline__ void rows2d_sweep(const float *src, float *dst, const Geom g, int hb,
                                             int nblk, unsigned cta, unsigned nctas) {
    using Edge = typename RowsEdge<R>::V;
    auto ld = [](const auto *p) {
        if constexpr (L1) return *p;
        else return __ldcg(p);
    };
    constexpr int C = 4 * R, K = 2 * R + 1 + D;
    // nx: the width (update region x < nx - R); px: the row pitch
    const int nx = g.nx, ny = g.ny, px = (int)g.sy, nch = px >> 2;
    const int items = nch * nblk, lane = threadIdx.x & 31;
    for (int w0 = (int)(cta * NT + (threadIdx.x & ~31u)); w0 < items; w0 += (int)(nctas * NT)) {
        const int it = w0 + lane;
        const int c = it % nch, rb = it / nch, x0 = 4 * c;
        const int j0 = R + rb * hb, rows = it < items ? min(hb, ny - R - j0) : 0;
        const int steps = __reduce_max_sync(~0u, rows);
        const bool any = x0 + 3 >= R && x0 < nx - R;
        const bool full = x0 >= R && x0 + 3 < nx - R;
        // the cells left of lane 0's chunk, right of lane 31's
        const bool edge = (lane == 0 && c > 0) || (lane == 31 && c + 1 < nch);
        const float *col = src + (long long)j0 * px + x0;
        const float *ecol = col + (lane == 0 ? -(int)(sizeof(Edge) / 4) : 4);
        float *dcol = dst + (long long)j0 * px + x0;
        float4 q[K];  // row j0 + i of this chunk column: q[(i + R) % K]
        Edge e[K];    // row j0 + i's edge: e[i % K]
#pragma unroll
        for (int k = 0; k < 2 * R + D; ++k) {
            q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < rows + 2 * R && rows) q[k] = ld(reinterpret_cast<const float4 *>(col + (long long)(k - R) * px));
        }
#pragma unroll
        for (int k = 0; k < D; ++k) {
            e[k] = Edge{};
            if (edge && k < rows) e[k] = ld(reinterpret_cast<const Edge *>(ecol + (long long)k * px));
        }
        for (int i0 = 0; i0 < steps; i0 += K) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int i = i0 + k;
                if (i >= steps) break;
                if (i + D < rows) {
                    q[(k + 2 * R + D) % K] = ld(reinterpret_cast<const float4 *>(col + (long long)(R + D) * px));
                    if (edge) e[(k + D) % K] = ld(reinterpret_cast<const Edge *>(ecol + (long long)D * px));
                }
                const float4 m4 = q[(k + R) % K];
                const float m[4] = {m4.x, m4.y, m4.z, m4.w};
                float w[4 + 2 * R];  // cells x0 - R .. x0 + 3 + R
#pragma unroll
                for (int o = 0; o < 4; ++o) w[R + o] = m[o];
                float ev[4] = {0.f, 0.f, 0.f, 0.f};
                if constexpr (R == 1) ev[0] = e[k];
                else if constexpr (R == 2) ev[0] = e[k].x, ev[1] = e[k].y;
                else ev[0] = e[k].x, ev[1] = e[k].y, ev[2] = e[k].z, ev[3] = e[k].w;
#pragma unroll
                for (int o = 0; o < R; ++o) {
                    const float l = __shfl_up_sync(~0u, m[4 - R + o], 1), r = __shfl_down_sync(~0u, m[o], 1);
                    w[o] = lane == 0 ? ev[(R == 3 ? 1 : 0) + o] : l;
                    w[R + 4 + o] = lane == 31 ? ev[o] : r;
                }
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int o = -R; o <= R; ++o) {
                    if (!o) continue;
#pragma unroll
                    for (int x = 0; x < 4; ++x) acc[x] += w[R + x + o];
                }
#pragma unroll
                for (int o = -R; o <= R; ++o) {
                    if (!o) continue;
                    const float4 v = q[(k + R + o + K) % K];
                    acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w;
                }
                float out[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    out[x] = div_coeff<C>(acc[x]);
                    if (g.legacy) out[x] -= m[x];
                }
                if (i < rows) {
                    if (full) {
                        *reinterpret_cast<float4 *>(dcol) = make_float4(out[0], out[1], out[2], out[3]);
                    } else if (any) {
#pragma unroll
                        for (int x = 0; x < 4; ++x)
                            if (in_range(x0 + x, nx, R)) dcol[x] = out[x];
                    }
                }
                col += px;
                ecol += px;
                dcol += px;
            }
        }
    }
}

// One sweep of a 2-D grid whose rows are not 16-byte aligned (any pitch): a
// thread owns one column of a block of hb rows, its rows j-R .. j+R in a
// register queue and the x-neighbours loaded 4 bytes each (L1 hits: they are
// the neighbouring lanes' columns), the next row's loads issued before the
// current row is computed.  Plain loads, as the L1 form above.  GB300, R = 1:
// 850 x 2933 7.5 us a sweep (a launch per sweep of one thread per cell: 26.6),
// 8191 x 8190 228 us (765).
template <int R, int NT>
__device__ __forceinline__ void rows2d_sweep_any(const float *src, float *dst, const Geom g, int hb, int nblk,
                                                 unsigned cta, unsigned nctas) {
    constexpr int C = 4 * R;
    const int nx = g.nx, ny = g.ny, cols = nx - 2 * R;
    const long long pitch = g.sy;
    const int items = cols * nblk;
    for (int it = (int)(cta * NT + threadIdx.x); it < items; it += (int)(nctas * NT)) {
        const int x = R + it % cols, rb = it / cols;
        const int j0 = R + rb * hb, j1 = min(j0 + hb, ny - R);
        const float *col = src + x;
        float q[2 * R + 1], nq, nw[2 * R];  // the column's rows; row j+1's loads
#pragma unroll
        for (int k = 0; k < 2 * R; ++k) q[k] = col[(j0 - R + k) * pitch];
        auto fetch = [&](int j) {
            const float *row = col + j * pitch;
            nq = row[R * pitch];
#pragma unroll
            for (int o = 0; o < R; ++o) nw[o] = row[o - R], nw[R + o] = row[1 + o];
        };
        fetch(j0);
        for (int j = j0; j < j1; ++j) {
            q[2 * R] = nq;
            float acc = 0.f;
#pragma unroll
            for (int o = 0; o < 2 * R; ++o) acc += nw[o];
            if (j + 1 < j1) fetch(j + 1);
#pragma unroll
            for (int o = -R; o <= R; ++o)
                if (o) acc += q[R + o];
            float v = div_coeff<C>(acc);
            if (g.legacy) v -= q[R];
            dst[j * pitch + x] = v;
#pragma unroll
            for (int k = 0; k < 2 * R; ++k) q[k] = q[k + 1];
        }
    }
}

}  // namespace st
