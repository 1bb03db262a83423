// k_rows2d.cu -- 2-D grids too large for one tile per SM: every sweep in one
// cooperative launch over the whole GPU ("coop" role,
// src/stencil_kernel_coop.cu:5-49), with a bounded grid-wide barrier between
// sweeps instead of a launch per sweep.
//
// A thread owns one float4 chunk column of a block of HB rows: it keeps the
// column's rows j-R .. j+R in a register queue (one new 16-byte load per
// row, the smem_register idea of src/stencils.cu:71-83 on registers) and
// takes the x-neighbours from the lanes beside it, so a 4-cell update costs
// one 16-byte load at any R <= 4 (the base kernel: 3 + 2R) and one short load
// in a warp's first and last lane.  Items (chunk column, row block) are spread
// over the resident CTAs with a grid stride; consecutive threads take
// consecutive chunk columns, so a warp's loads and stores are contiguous
// 512-byte segments.
//
// Bounds: device memory above the L2's size (91 % of a plain copy's rate at
// R = 1), L2 reads and the barrier below it.  What was in the way was bytes
// in flight: with the left and right chunks loaded too, registers allowed one
// row ahead (16 KB an SM), and hb blocks that left a nearly empty last wave.
// GB300, microseconds a sweep before -> now: R = 1 1024^2 3.07 -> 3.00, 2048^2
// 6.23 -> 5.4, 4096^2 26.1 -> 22.3, 8192^2 111.8 -> 86.6, 16384^2 401 -> 336;
// 8192^2 R = 2 114.7 -> 88.8, R = 3 216 -> 146, R = 4 186 -> 109.
//
// Loads are plain (L1-cached): a buffer is rewritten every other sweep
// inside the launch, and every read of another CTA's writes follows the grid
// barrier's acquire at GPU scope and a CTA barrier, after which weak loads
// observe those writes (PTX memory model).  Every cell keeps the reference's summation order (axis i
// offsets -R..-1, +1..+R, then axis j, from +0) and division, so results are
// bit-identical to single sweeps; cells outside the update region are never
// written.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "host.hpp"
#include "rows_body.cuh"

namespace st {
namespace {

constexpr int kRowsThreads = 512;

// Rows in flight ahead of the row being computed: as many as leave two CTAs
// (R <= 2) or one CTA of 16 warps on an SM without spills in the loop.  GB300,
// GCell/s for 1 / 2 / 3 / 4 rows, R = 1 8192^2: - / 739 / 775 / 731; R = 2:
// 707 / 755; R = 3: 388 / 445 / 460; R = 4: 514 / 574 / 615.
template <int R> constexpr int kRowsAhead = R == 2 ? 2 : 3;

// ANY: rows that are not 16-byte aligned, one column per thread
// (rows2d_sweep_any).
template <int R, bool L1, bool ANY = false>
__global__ void __launch_bounds__(kRowsThreads, R <= 2 || ANY ? 2 : 1)
    k_rows2d(float *a, float *b, Geom g, int hb, int nblk, int iters, unsigned *bar) {
    __shared__ int s_ok;
    for (int sw = 0; sw < iters; ++sw) {
        const float *src = (sw & 1) ? b : a;
        float *dst = (sw & 1) ? a : b;
        if constexpr (ANY) rows2d_sweep_any<R, kRowsThreads>(src, dst, g, hb, nblk, blockIdx.x, gridDim.x);
        else rows2d_sweep<R, kRowsThreads, kRowsAhead<R>, L1>(src, dst, g, hb, nblk, blockIdx.x, gridDim.x);
        if (sw + 1 < iters) {
            // every CTA's writes of this sweep before any CTA's next reads
            __syncthreads();
            if (threadIdx.x == 0) {
                grid_arrive(bar);
                s_ok = grid_wait_bounded(bar, (unsigned)(sw + 1) * gridDim.x) ? 1 : 0;
            }
            __syncthreads();
            if (!s_ok) return;
        }
    }
}

using RowsFn = void (*)(float *, float *, Geom, int, int, int, unsigned *);

// Loads: plain, L1-cached (a warp's edge cells are its neighbour warp's
// chunks), legal because every read of another CTA's writes follows the grid
// barrier's acquire and a CTA barrier; STENCIL_ROWS_L1=0 (read at each
// launch) selects ld.global.cg.
RowsFn rows_fn(int r, bool l1) {
    switch (r * 2 + (l1 ? 1 : 0)) {
        case 2: return k_rows2d<1, false>;
        case 3: return k_rows2d<1, true>;
        case 4: return k_rows2d<2, false>;
        case 5: return k_rows2d<2, true>;
        case 6: return k_rows2d<3, false>;
        case 7: return k_rows2d<3, true>;
        case 8: return k_rows2d<4, false>;
        case 9: return k_rows2d<4, true>;
        default: return nullptr;
    }
}

RowsFn rows_any_fn(int r) {
    return r == 1 ? k_rows2d<1, true, true> : r == 2 ? k_rows2d<2, true, true>
         : r == 3 ? k_rows2d<3, true, true> : k_rows2d<4, true, true>;
}

bool rows_l1() {
    const char *e = std::getenv("STENCIL_ROWS_L1");
    return !(e && e[0] == '0');
}

// Resident CTAs of the kernel that is launched (once per kernel and device).
int rows_ctas(RowsFn fn) {
    static std::mutex mu;
    static std::vector<std::pair<std::pair<RowsFn, int>, int>> cache;
    const int dev = current_device();
    std::lock_guard<std::mutex> lock(mu);
    for (auto &c : cache)
        if (c.first.first == fn && c.first.second == dev) return c.second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, reinterpret_cast<const void *>(fn), kRowsThreads, 0) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    const int ctas = n * num_sms();
    cache.push_back({{fn, dev}, ctas});
    return ctas;
}

}  // namespace

bool rows2d_supported(const Geom &g, int dims) {
    return dims == 2 && g.sy % 4 == 0 && g.radius >= 1 && g.radius <= 4 &&
           (long long)(g.sy / 4) * (g.ny - 2 * g.radius) < (1LL << 31) && rows_ctas(rows_fn(g.radius, rows_l1())) > 0;
}

// Rows that are not 16-byte aligned: fewer than 2^31 (column, row) pairs, and
// row offsets that the kernel's 64-bit products hold.
bool rows2d_any_supported(const Geom &g, int dims) {
    return dims == 2 && g.sy % 4 != 0 && g.radius >= 1 && g.radius <= 4 &&
           (long long)g.nx * g.ny < (1LL << 31) && rows_ctas(rows_any_fn(g.radius)) > 0;
}

int rows2d_capacity(const Geom &g) { return rows_ctas(rows_fn(g.radius, rows_l1())); }

// Row blocks of a rows sweep of g on `threads` threads: the height, at most
// 64 rows and at least 4 (R = 1) or 8, that costs the busiest thread the
// fewest rows, each of its items counted with its 2R halo rows and about
// three rows' time for the first load.  (About four items per thread, as
// before, left one more, nearly empty wave: 4.14 items per thread on 8192^2.
// Limits of 128 rows and 1 or 6 rows for the first load measured within 1 %.)
void rows2d_plan(const Geom &g, long long threads, int *hb, int *nblk) {
    const int nch = (int)(g.sy / 4), rows = g.ny - 2 * g.radius;
    const int lo = std::min(rows, g.radius == 1 ? 4 : 8), hi = std::min(rows, 64);
    threads = std::max(1LL, threads);
    double best = 1e300;
    for (int h = hi; h >= lo; --h) {
        const int n = (rows + h - 1) / h;
        const long long waves = ((long long)nch * n + threads - 1) / threads;
        const double cost = (double)waves * (h + 3 + 2 * g.radius);
        if (cost < best) { best = cost; *hb = h; *nblk = n; }
    }
}

// The persistent rows kernel on rows that are not 16-byte aligned.  Row blocks
// as rows2d_plan's, for one column per thread: about four items per thread, 4
// to 64 rows.
int run_rows2d_any(const Geom &g, float *a, float *b, int iters, cudaStream_t s, float **res) {
    if (res) *res = (iters & 1) ? b : a;
    if (iters <= 0) return STENCIL_OK;
    const int ctas = rows_ctas(rows_any_fn(g.radius));
    const int cols = g.nx - 2 * g.radius, rows = g.ny - 2 * g.radius;
    int hb = (int)std::min<long long>(64, std::max<long long>(4, (long long)cols * rows / (4LL * ctas * kRowsThreads)));
    hb = std::min(hb, rows);
    int nblk = (rows + hb - 1) / hb;
    const int grid = (int)std::min<long long>(ctas, ((long long)cols * nblk + kRowsThreads - 1) / kRowsThreads);
    LaunchSlot slot;
    int rc = take_barrier(s, &slot);
    if (rc) return rc;
    unsigned *bar = static_cast<unsigned *>(slot.mem());
    Geom gg = g;
    int n = iters;
    void *args[] = {&a, &b, &gg, &hb, &nblk, &n, &bar};
    ST_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(rows_any_fn(g.radius)), dim3(grid),
                                        dim3(kRowsThreads), args, 0, s));
    note_launches("rows2d-persistent", 1);
    return STENCIL_OK;
}

int run_rows2d(const Geom &g, float *a, float *b, int iters, cudaStream_t s, float **res,
               int max_ctas) {
    if (!rows2d_supported(g, 2))
        return fail(STENCIL_EUNSUPPORTED, "persistent 2-D rows kernel: row pitch %% 4 == 0, R <= 4");
    if (res) *res = (iters & 1) ? b : a;
    if (iters <= 0) return STENCIL_OK;
    const RowsFn fn = rows_fn(g.radius, rows_l1());
    const int resident = rows_ctas(fn), ctas = max_ctas > 0 ? std::min(max_ctas, resident) : resident;
    const int nch = (int)(g.sy / 4);
    int hb = 0, nblk = 0;
    rows2d_plan(g, (long long)ctas * kRowsThreads, &hb, &nblk);
    const int items = nch * nblk;
    const int grid = (int)std::max<long long>(1, std::min<long long>(ctas, (items + kRowsThreads - 1) / kRowsThreads));
    LaunchSlot slot;
    int rc = take_barrier(s, &slot);
    if (rc) return rc;
    unsigned *bar = static_cast<unsigned *>(slot.mem());
    Geom gg = g;
    int hb_ = hb, nb_ = nblk, n = iters;
    void *args[] = {&a, &b, &gg, &hb_, &nb_, &n, &bar};
    ST_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(fn), dim3(grid), dim3(kRowsThreads), args, 0, s));
    note_launches("rows2d-persistent", 1);
    return STENCIL_OK;
}

}  // namespace st
