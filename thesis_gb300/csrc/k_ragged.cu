// k_ragged.cu -- 3-D grids whose rows are not 16-byte aligned (nx % 4 != 0):
// every sweep in one cooperative launch ("smem_register" role of
// src/stencil_kernel_smem_register.cu:8-62 for shapes that the stream kernel's
// tensor maps cannot describe).
//
// The structure is the stream kernel's (stream_body.cuh): a CTA owns an x-y
// tile and a chunk of z-planes, producer warps stream plane tiles with
// their halo into a ring of shared-memory slots (full/empty mbarriers), the
// consumers keep the z-neighbours in a register queue, and between sweeps the
// CTAs meet at a bounded grid barrier.  What differs:
//   * a plane tile is one cp.async.bulk per row (shared out over two or four
//     producer warps), from the 16-byte boundary at or before its first cell
//     to the one at or after its last.  The slot's row pitch is congruent to nx
//     modulo 4, so every cell of a plane sits at its place plus one shift
//     (0..3) that depends on the plane alone, and the copies keep 16-byte
//     alignment on both sides;
//   * a thread owns one column of RY rows and reads shared memory 4 bytes at a
//     time (32 consecutive words of any alignment are free of bank conflicts),
//     and stores 4 bytes (a warp's 128 bytes in a row).
// Per 32 cells that is 1 + 2R + 2R/RY shared-memory wavefronts; the sweep is
// bound by HBM at R = 1 and by instruction issue at larger radii (about twice
// the instructions per cell of the stream kernel's 4-cell vectors).  GB300, us
// per sweep, against a launch per sweep of one thread per cell: 509 x 511 x 510
// R = 1 194 (1303; the stream kernel's 512^3: 182), 205 x 301 x 253 R = 2 30.7
// (177), 99 x 505 x 205 R = 3 32.5 (157), 511 x 510 x 509 R = 4 313 (2033), 61^3
// R = 1 5.5 (7.9).  With two producer warps at every radius: packed sums
// against scalar ones R = 4 313 / 342, R = 2 33.4 / 35.1; one CTA per SM against
// two at R = 2 (whose 56 registers spill) 205 x 301 x 253 33.4 / 35.7, 511 x 510 x
// 509 259 / 249 (one CTA with four producer warps 30.9 and 230).
#include <algorithm>
#include <mutex>
#include <vector>

#include "host.hpp"
#include "stream_body.cuh"

namespace st {

namespace {

template <int R, int WX, int M>
struct RaggedShape {
    static constexpr int RY = 4, WARPS = 16, CONSUMERS = 32 * WARPS, PW_WARPS = R == 1 ? 2 : 4;  // consumer rows per thread; producer warps
    static constexpr int THREADS = CONSUMERS + 32 * PW_WARPS;
    static constexpr int TX = 32 * WX, TY = RY * (WARPS / WX);
    static constexpr int PH = TY + 2 * R;
    // room for the copies' ends (up to 3 cells before and after), congruent to
    // nx modulo 4
    static constexpr int PW = (TX + 2 * R + 6 + 3) / 4 * 4 + M;
    static constexpr int SLOT = (PH * PW + 8 + 31) / 32 * 32;  // floats
    static constexpr int NS = 8;
    static constexpr int SMEM = NS * SLOT * 4 + 2 * NS * 8 + 128;
    static constexpr int MIN_BLOCKS = R == 1 ? 2 : 1;
    static_assert(NS >= R + 2, "ring");
};

template <int R, int WX, int M>
__global__ void __launch_bounds__(RaggedShape<R, WX, M>::THREADS, RaggedShape<R, WX, M>::MIN_BLOCKS)
    k_ragged3d(float *a, float *b, Geom g, int tiles_x, int tiles_y, int zchunk, int items, int sweeps, unsigned *grid_bar) {
    using S = RaggedShape<R, WX, M>;
    constexpr int C = 6 * R, QN = 2 * R + 1, RY = S::RY, NS = S::NS, PW = S::PW;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float *ring = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + NS * S::SLOT), *empty = full + NS;
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int ntiles = tiles_x * tiles_y;
    const long long total = g.sz * g.nz;
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&full[s], S::PW_WARPS);
            mbar_init(&empty[s], S::WARPS);
        }
        fence_mbar_init();
    }
    __syncthreads();

    if (warp >= S::WARPS) {
        // ---------------- producers ----------------
        // Each of the PW_WARPS warps copies every PW_WARPS-th row.  The whole
        // warp runs the loop and one lane is elected to issue, so that the
        // addresses stay in uniform registers (a lane per row made a plane of
        // 20 rows cost 2000 cycles).
        const int wp = warp - S::WARPS;
        const uint32_t on = elect_lane();
        uint32_t q = 0;
        for (int sw = 0; sw < sweeps; ++sw) {
            // sweep sw reads what every CTA wrote in sweep sw - 1: the elected
            // lane's acquire and fence (in the wait) come before its copies
            if (sw > 0 && !__all_sync(0xffffffffu, grid_wait_bounded(grid_bar, (unsigned)sw * gridDim.x))) return;
            const float *src = (sw & 1) ? b : a;
            for (int item = blockIdx.x; item < items; item += gridDim.x) {
                const int t = item % ntiles, ch = item / ntiles;
                const int x0 = (t % tiles_x) * S::TX, y0 = (t / tiles_x) * S::TY;
                const int z0 = R + ch * zchunk, z1 = min(z0 + zchunk, g.nz - R);
                const int np = (z1 - z0) + 2 * R;
                const int xa = max(x0 - R, 0), xb = min(x0 + S::TX + R, g.nx);
                for (int p = 0; p < np; ++p, ++q) {
                    const int s = q & (NS - 1);
                    const uint32_t use = q / NS;
                    if (use > 0 && !warp_wait_bounded(&empty[s], (use - 1) & 1)) return;
                    fence_proxy_async();  // the consumers' reads of the slot before the copies
                    const long long plane = (long long)(z0 - R + p) * g.sz;
                    // cell (x, row r) sits at slot + shift + r * PW + x - x0 + R,
                    // shift = its plane's global index of (x0 - R, y0 - R) mod 4
                    const long long org = plane + (long long)(y0 - R) * g.nx + x0 - R;
                    const uint32_t bar = smem_u32(&full[s]);
                    // byte addresses of cell xa of row r, in memory and in the slot
                    int r = wp + max(0, (R - y0 - wp + S::PW_WARPS - 1) / S::PW_WARPS) * S::PW_WARPS;  // first row >= 0
                    const int yend = min(y0 + S::TY + R, plane + g.sz == total ? g.ny - 1 : g.ny) - (y0 - R);
                    uint64_t from = reinterpret_cast<uint64_t>(src) + 4 * (plane + (long long)(y0 - R + r) * g.nx + xa);
                    uint32_t to = smem_u32(ring + s * S::SLOT) + 4 * (4 + (int)(org & 3) + r * PW + xa - (x0 - R));
                    uint32_t sum = 0;
                    // the grid's last row has no cell that a star needs, and the
                    // 16 bytes at its end may lie past the buffer's: not copied
                    for (; r < yend; r += S::PW_WARPS) {
                        const uint32_t sh = (uint32_t)from & 12u, bytes = (4u * (xb - xa) + sh + 15u) & ~15u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                            "@p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(
                                to - sh),
                            "l"(from - sh), "r"(bytes), "r"(bar), "r"(on)
                            : "memory");
                        sum += bytes;
                        from += 4ull * S::PW_WARPS * g.nx;
                        to += 4u * S::PW_WARPS * PW;
                    }
                    expect_tx_if(on, bar, sum);
                }
            }
        }
        return;
    }

    // ---------------- consumers ----------------
    const int cx = (warp % WX) * 32 + lane, cy = (warp / WX) * RY;
    const int own = 4 + (cy + R) * PW + cx + R;  // slot offset of row 0 (without the plane's shift)
    auto release = [&](int s) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
    };
    // z register queue of row pairs, rotated by unrolling: plane z+k-R sits at
    // index (z-z0+k) % QN
    float2 qz[RY / 2][QN];
    uint32_t qb = 0;   // sequence number of plane 0 of the current item
    bool ok = true;    // false once a bounded wait gave up
    const int dz = (int)(g.sz & 3);
    for (int sw = 0; sw < sweeps && ok; ++sw) {
        float *dst = (sw & 1) ? a : b;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            const int t = item % ntiles, ch = item / ntiles;
            const int x0 = (t % tiles_x) * S::TX, y0 = (t / tiles_x) * S::TY;
            const int z0 = R + ch * zchunk, z1 = min(z0 + zchunk, g.nz - R);
            const int np = (z1 - z0) + 2 * R;
            const int x = x0 + cx, y = y0 + cy;
            unsigned live = 0;  // this thread's cells inside the update region
#pragma unroll
            for (int r = 0; r < RY; ++r)
                if (in_range(x, g.nx, R) && in_range(y + r, g.ny, R)) live |= 1u << r;
            // shift of plane 0 of the item; plane p's is (c0 + p * dz) & 3
            const int c0 = (int)(((long long)(z0 - R) * g.sz + (long long)(y0 - R) * g.nx + x0 - R) & 3);
#pragma unroll
            for (int p = 0; p < 2 * R; ++p) {
                const uint32_t q = qb + p;
                const int s = q & (NS - 1);
                if (!mbar_wait_bounded(&full[s], (q / NS) & 1)) { ok = false; break; }
                const float *sl = ring + s * S::SLOT + own + ((c0 + p * dz) & 3);
#pragma unroll
                for (int r = 0; r < RY / 2; ++r) qz[r][p] = make_float2(sl[2 * r * PW], sl[(2 * r + 1) * PW]);
                if (p < R || p >= np - R) release(s);
            }
            if (!ok) break;
            float *drow = dst + (long long)z0 * g.sz + (long long)y * g.nx + x;
            for (int zb = z0; zb < z1 && ok; zb += QN) {
#pragma unroll
                for (int ph = 0; ph < QN; ++ph) {
                    const int z = zb + ph;
                    if (z >= z1) break;
                    const int step = z - z0;
                    const int sc = (qb + step + R) & (NS - 1);
                    const float *cb = ring + sc * S::SLOT + own + ((c0 + (step + R) * dz) & 3);
                    // the column's rows -R .. RY-1+R: its own from the queue
                    float col[RY + 2 * R];
#pragma unroll
                    for (int k = 0; k < RY + 2 * R; ++k) {
                        if (k >= R && k < R + RY) {
                            const float2 v = qz[(k - R) / 2][(ph + R) % QN];
                            col[k] = (k - R) & 1 ? v.y : v.x;
                        } else {
                            col[k] = cb[(k - R) * PW];
                        }
                    }
                    // sums of two rows at a time along x and z (fadd2), started
                    // from the first term (div_slow_from_first)
                    float2 acc[RY / 2];
#pragma unroll
                    for (int r = 0; r < RY / 2; ++r) {
                        const float *c0r = cb + 2 * r * PW, *c1r = c0r + PW;
                        acc[r] = make_float2(c0r[-R], c1r[-R]);
#pragma unroll
                        for (int o = -R + 1; o <= R; ++o)
                            if (o) acc[r] = fadd2(acc[r], make_float2(c0r[o], c1r[o]));
#pragma unroll
                        for (int o = -R; o <= R; ++o)
                            if (o) acc[r].x += col[2 * r + R + o], acc[r].y += col[2 * r + 1 + R + o];
#pragma unroll
                        for (int o = -R; o <= -1; ++o) acc[r] = fadd2(acc[r], qz[r][(ph + R + o + QN) % QN]);
                    }
                    release(sc);
                    {
                        const int pn = step + 2 * R;
                        const uint32_t q = qb + pn;
                        const int s = q & (NS - 1);
                        if (!mbar_wait_bounded(&full[s], (q / NS) & 1)) { ok = false; break; }
                        const float *sl = ring + s * S::SLOT + own + ((c0 + pn * dz) & 3);
#pragma unroll
                        for (int r = 0; r < RY / 2; ++r)
                            qz[r][(ph + 2 * R) % QN] = make_float2(sl[2 * r * PW], sl[(2 * r + 1) * PW]);
                        if (pn >= np - R) release(s);
                    }
#pragma unroll
                    for (int r = 0; r < RY / 2; ++r)
#pragma unroll
                        for (int o = 1; o <= R; ++o) acc[r] = fadd2(acc[r], qz[r][(ph + R + o) % QN]);
                    // correctly rounded division by 6R: the fast path where every
                    // stored sum lies in its range, else the warp divides
                    float lo = 0x1p-100f, hi = 0x1p+120f;
#pragma unroll
                    for (int r = 0; r < RY; ++r)
                        if (live & (1u << r)) {
                            const float v = fabsf(r & 1 ? acc[r / 2].y : acc[r / 2].x);
                            lo = fminf(lo, v);
                            hi = fmaxf(hi, v);
                        }
                    if (__all_sync(0xffffffffu, lo >= 0x1p-100f && hi <= 0x1p+120f)) {
#pragma unroll
                        for (int r = 0; r < RY / 2; ++r) acc[r] = div_fast2<C>(acc[r]);
                    } else {
#pragma unroll
                        for (int r = 0; r < RY / 2; ++r)
                            acc[r] = make_float2(div_slow_from_first<C>(acc[r].x), div_slow_from_first<C>(acc[r].y));
                    }
#pragma unroll
                    for (int r = 0; r < RY; ++r) {
                        float v = r & 1 ? acc[r / 2].y : acc[r / 2].x;
                        if (g.legacy) v -= col[r + R];
                        if (live & (1u << r)) drow[r * g.nx] = v;
                    }
                    drow += g.sz;
                }
            }
            qb += np;
        }
        if (sw + 1 < sweeps) {
            // once every consumer of this CTA has stored its part of sweep sw
            // (or given up), one thread arrives at the grid barrier
            ok = named_barrier_and(1, S::CONSUMERS, ok);
            if (ok && tid == 0) grid_arrive(grid_bar);
        }
    }
}

struct RaggedKernel {
    const void *fn;
    int tx, ty, threads, smem;
};

template <int R, int WX, int M>
RaggedKernel rk() {
    using S = RaggedShape<R, WX, M>;
    return {reinterpret_cast<const void *>(k_ragged3d<R, WX, M>), S::TX, S::TY, S::THREADS, S::SMEM};
}

template <int R, int WX>
RaggedKernel pick_m(int m) {
    return m == 1 ? rk<R, WX, 1>() : m == 2 ? rk<R, WX, 2>() : rk<R, WX, 3>();
}

// Tiles of 128 x 16 or 64 x 32 cells: the ones that cover nx x ny with fewer
// cells (a tie: the wider).
RaggedKernel pick(const Geom &g) {
    auto cells = [&](int tx, int ty) { return (long long)((g.nx + tx - 1) / tx * tx) * ((g.ny + ty - 1) / ty * ty); };
    const bool wide = cells(128, 16) <= cells(64, 32);
    const int m = g.nx & 3;
    switch (g.radius) {
        case 1: return wide ? pick_m<1, 4>(m) : pick_m<1, 2>(m);
        case 2: return wide ? pick_m<2, 4>(m) : pick_m<2, 2>(m);
        case 3: return wide ? pick_m<3, 4>(m) : pick_m<3, 2>(m);
        default: return wide ? pick_m<4, 4>(m) : pick_m<4, 2>(m);
    }
}

}  // namespace

bool ragged3d_supported(const Geom &g, int dims) {
    return dims == 3 && g.nx % 4 != 0 && g.sy == g.nx && g.radius >= 1 && g.radius <= 4;
}

// A launch per sweep takes 4.2 to 6.3 us a sweep up to about 10^5 cells, the
// persistent sweeps 5.6 (R = 1), 5.5, 6.4 or 7.4 us (R = 4) as soon as the CTAs
// have a plane each.  GB300, us a sweep in a call of 8 sweeps, a launch each /
// persistent: R = 1 37^3 5.95 / 6.20, 45^3 6.47 / 6.22, 61^3 8.45 / 6.21; R = 2
// 33^3 5.45 / 6.00, 37^3 6.44 / 5.95; R = 3 45^3 6.48 / 7.00, 49^3 8.52 / 7.06; R =
// 4 33^3 6.45 / 7.98, 17 x 65 x 129 6.49 / 8.25, 61^3 9.72 / 8.09.  (On four
// streams at once, us a sweep and grid: 49^3 R = 2 2.66 / 1.56, 101 x 99 x 97 R = 2
// 12.3 / 6.3, but 63 x 65 x 67 R = 4 5.0 / 6.8, alone 10.4 / 6.9.)
long long ragged3d_least_cells(int radius) {
    return radius == 1 ? 80000 : radius == 2 ? 45000 : radius == 3 ? 110000 : 150000;
}

int run_ragged3d(const Geom &g, float *a, float *b, int iters, cudaStream_t s, float **res) {
    if (res) *res = (iters & 1) ? b : a;
    if (iters <= 0) return STENCIL_OK;
    const RaggedKernel k = pick(g);
    int resident = 0;
    int rc = grid_resident_ctas(k.fn, k.threads, k.smem, &resident);
    if (rc) return rc;
    if (resident < 1) return fail(STENCIL_EUNSUPPORTED, "ragged stream kernel does not fit on an SM");
    int tiles_x = 0, tiles_y = 0, zchunk = 0, items = 0;
    stream3d_plan(g, k.tx, k.ty, resident, &tiles_x, &tiles_y, &zchunk, &items);
    LaunchSlot slot;
    rc = take_barrier(s, &slot);
    if (rc) return rc;
    unsigned *bar = static_cast<unsigned *>(slot.mem());
    Geom gg = g;
    int sw = iters;
    void *args[] = {&a, &b, &gg, &tiles_x, &tiles_y, &zchunk, &items, &sw, &bar};
    ST_CUDA(cudaLaunchCooperativeKernel(k.fn, dim3(std::min(items, resident)), dim3(k.threads), args, k.smem, s));
    note_launches("ragged3d-persistent", 1);
    return STENCIL_OK;
}

}  // namespace st
