// unet.cu -- kernels of the learned-warm-start U-Net (include/unet.h).
//
// Convolutions are implicit GEMMs on the BF16 tensor cores with FP32
// accumulation:
//   forward / data gradient:  M = pixels, N = output channels, K = 9 x input
//     channels (taps outer, channels inner), zero padding;
//   weight gradient:          M = input channels of three taps, N = output
//     channels, K = pixels (split across CTAs, FP32 atomics).
// The default engine is tcgen05 (TMA-fed, TMEM accumulators); the mma.sync one
// (cp.async-fed, ldmatrix) is kept as an engine a caller may choose and serves
// weight gradients that the other does not take.
// Everything else (pooling, upsampling, ReLU gradient, head, loss, Adam,
// features) is bandwidth-bound element-wise work on 16-byte vectors.
#include <cuda_bf16.h>

#include "../../include/unet.h"
#include "host.hpp"

namespace st {
namespace {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid) {
    const uint32_t s = smem_u32(smem);
    const int n = valid ? 16 : 0;  // zero-fill when the source is outside the tensor
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2,
                                        uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2,
                                          uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void mma16816(float *d, const uint32_t *a, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct Act {
    bf16 *p;
    int n, h, w, cs, co, c;
};

Act to_act(const unet_act &a) { return {static_cast<bf16 *>(a.ptr), a.n, a.h, a.w, a.c_stride, a.c_off, a.c}; }

// v where the gate's value is positive, else 0 (the ReLU gradient), for eight
// BF16 values.
__device__ __forceinline__ uint4 gate8(uint4 v, uint4 gate) {
    uint32_t *w = reinterpret_cast<uint32_t *>(&v);
    const __nv_bfloat162 *g = reinterpret_cast<const __nv_bfloat162 *>(&gate);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(g[k]);
        w[k] &= (f.x > 0.f ? 0x0000FFFFu : 0u) | (f.y > 0.f ? 0xFFFF0000u : 0u);
    }
    return v;
}

// ---------------------------------------------------------------------------
// 3x3 convolution, forward (also the data gradient with flipped weights).
// Block: 128 threads = 2 x 2 warps; tile BM = 128 pixels x BN output channels,
// K chunk BK = 32 input channels of one tap; two cp.async stages.
// ---------------------------------------------------------------------------
constexpr int BM = 128, BK = 32, PITCH = BK + 8;  // 80-byte rows: conflict-free ldmatrix

template <int BN>
__global__ void __launch_bounds__(128)
    k_conv3x3(Act x, const bf16 *__restrict__ w, const float *__restrict__ bias, Act y, int relu,
              int dil) {
    __shared__ __align__(128) bf16 As[2][BM][PITCH];
    __shared__ __align__(128) bf16 Bs[2][BN][PITCH];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp & 1, wn = warp >> 1;
    const long long P = (long long)x.n * x.h * x.w;
    const long long m0 = (long long)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN;
    const int cin = x.c, cout = y.c;
    const int nc = cin / BK, KB = 9 * nc;
    // Rows this thread loads for A: idx = tid + 128*i, row = idx / 4, part = idx % 4.
    int a_n[4], a_y[4], a_x[4];
    bool a_ok[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = (tid + 128 * i) >> 2;
        const long long p = m0 + row;
        a_ok[i] = p < P;
        const long long pp = a_ok[i] ? p : 0;
        a_x[i] = (int)(pp % x.w);
        a_y[i] = (int)((pp / x.w) % x.h);
        a_n[i] = (int)(pp / ((long long)x.w * x.h));
    }
    auto load = [&](int kb, int st) {
        const int tap = kb / nc, c0 = (kb % nc) * BK;
        const int dy = (tap / 3 - 1) * dil, dx = (tap % 3 - 1) * dil;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = tid + 128 * i, row = idx >> 2, part = idx & 3;
            const int yy = a_y[i] + dy, xx = a_x[i] + dx;
            const bool v = a_ok[i] && yy >= 0 && yy < x.h && xx >= 0 && xx < x.w;
            const bf16 *src = x.p + (((long long)a_n[i] * x.h + (v ? yy : 0)) * x.w + (v ? xx : 0)) * x.cs +
                              x.co + c0 + part * 8;
            cp_async16(&As[st][row][part * 8], src, v);
        }
#pragma unroll
        for (int i = 0; i < (BN * 4) / 128; ++i) {
            const int idx = tid + 128 * i, row = idx >> 2, part = idx & 3;
            const int co = n0 + row;
            const bool v = co < cout;
            const bf16 *src = w + ((long long)(v ? co : 0) * 9 + tap) * cin + c0 + part * 8;
            cp_async16(&Bs[st][row][part * 8], src, v);
        }
        cp_async_commit();
    };
    constexpr int NT = BN / 16;  // n8 tiles per warp (warp covers BN/2 channels)
    float acc[4][NT][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    load(0, 0);
    for (int kb = 0; kb < KB; ++kb) {
        const int st = kb & 1;
        cp_async_wait_all();
        __syncthreads();
        if (kb + 1 < KB) load(kb + 1, st ^ 1);
#pragma unroll
        for (int ks = 0; ks < BK; ks += 16) {
            uint32_t af[4][4];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) {
                const int row = wm * 64 + mi * 16 + (lane & 7) + 8 * ((lane >> 3) & 1);
                const int col = ks + 8 * (lane >> 4);
                ldsm_x4(smem_u32(&As[st][row][col]), af[mi][0], af[mi][1], af[mi][2], af[mi][3]);
            }
#pragma unroll
            for (int nj = 0; nj < NT / 2; ++nj) {
                const int nrow = wn * (BN / 2) + nj * 16 + (lane & 7) + 8 * (lane >> 4);
                const int col = ks + 8 * ((lane >> 3) & 1);
                uint32_t b0, b1, b2, b3;
                ldsm_x4(smem_u32(&Bs[st][nrow][col]), b0, b1, b2, b3);
#pragma unroll
                for (int mi = 0; mi < 4; ++mi) {
                    mma16816(acc[mi][2 * nj], af[mi], b0, b1);
                    mma16816(acc[mi][2 * nj + 1], af[mi], b2, b3);
                }
            }
        }
        __syncthreads();
    }
    // Epilogue: bias, ReLU, BF16 pairs.
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int nj = 0; nj < NT; ++nj)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const long long p = m0 + wm * 64 + mi * 16 + (lane >> 2) + 8 * hh;
                const int co = n0 + wn * (BN / 2) + nj * 8 + (lane & 3) * 2;
                if (p >= P || co >= cout) continue;
                float v0 = acc[mi][nj][2 * hh], v1 = acc[mi][nj][2 * hh + 1];
                if (bias) { v0 += bias[co]; v1 += bias[co + 1]; }
                if (relu) { v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); }
                *reinterpret_cast<__nv_bfloat162 *>(y.p + p * y.cs + y.co + co) =
                    __floats2bfloat162_rn(v0, v1);
            }
}

// ---------------------------------------------------------------------------
// 3x3 convolution, forward / data gradient, on the 5th-generation tensor
// cores: tcgen05.mma (kind::f16, BF16 operands, FP32 accumulator in tensor
// memory), completion tracked by tcgen05.commit on mbarriers.
//   D[128 pixels x BN channels] (TMEM, BN columns) += A[128 x 16] B[BN x 16]^T
// per instruction; K runs over taps, then channels.  A is the shifted input
// pixels (zero outside the image), B the weights of one tap.  The epilogue
// reads the accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 =
// pixels), adds the bias, applies ReLU and stores BF16.  Every mbarrier wait
// is bounded.
// ---------------------------------------------------------------------------
template <int BN>
__device__ __forceinline__ constexpr uint32_t umma_idesc() {
    // D FP32, A and B BF16, both K-major, N = BN, M = 128
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit_if(uint32_t on, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t"
        "@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
        "r"(on)
        : "memory");
}

__device__ __forceinline__ void mma_f16_if(uint32_t on, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc),
        "r"(acc), "r"(on)
        : "memory");
}

__device__ __forceinline__ void tma_load_4d_if(uint32_t on, uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0,
                                               int c1, int c2, int c3) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %7, 0;\n\t"
        "@p cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];\n\t}" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(on)
        : "memory");
}

__device__ __forceinline__ void tma_load_5d_if(uint32_t on, uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0,
                                               int c1, int c2, int c3, int c4) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %8, 0;\n\t"
        "@p cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];\n\t}" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(on)
        : "memory");
}

// ---------------------------------------------------------------------------
// Tiles fed by TMA.  A tile is 128 pixels, 128 /
// tile_w rows of tile_w columns of one image.  One warp streams each K chunk
// as two tensor-map loads -- a 4-D box of BC channels x the tile's pixels
// shifted by the tap (its out-of-bounds cells arrive as zeros, which is the
// convolution's padding and fills tiles that reach past the image) and a 3-D
// box of the weights -- with a swizzle of BC channels (64 or 128 bytes), which
// is the layout the UMMA descriptors below describe; one warp issues the
// MMAs; 4 warps run the epilogue.  Warps: 0-3 epilogue, 4 TMA producer, 5 MMA
// issuer.  K runs over taps, then channels, in either form.
// What bounds it: TMA, at about three cycles per box row of 64 or 128 bytes
// (the input nine times, the weights once per tile), hence 64 channels a row
// where the layer has them; and, with few tiles, the latency of the K chain.
// ---------------------------------------------------------------------------
// K-major descriptor of BC-channel rows (64- or 128-byte swizzle): 8-row
// groups 8 rows apart, version 1.
template <int BC>
__device__ __forceinline__ uint64_t umma_desc_k(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | (1ull << 16) | ((uint64_t)(BC * 16 >> 4) << 32) | (1ull << 46) |
           ((BC == 64 ? 2ull : 4ull) << 61);
}

struct ConvTiles {
    int cin, H, W, tile_w, tiles_x, tiles_y, relu, dil, stages;
};

template <int BN, int BC>
__global__ void __launch_bounds__(192)
    k_conv3x3_tma(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                  const float *__restrict__ bias, Act y, Act gate, ConvTiles p) {
    extern __shared__ __align__(1024) unsigned char tm_smem[];
    constexpr int A_BYTES = BM * BC * 2, STAGE = A_BYTES + BN * BC * 2;
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(tm_smem) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(base + p.stages * STAGE);
    uint64_t *empty = full + p.stages;
    uint64_t *accd = empty + p.stages;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(accd + 1);
    int *bad = reinterpret_cast<int *>(tslot + 1);
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int n0 = blockIdx.y * BN;
    const int nc = p.cin / BC;
    // tile origin: image n, row h0, column w0
    const int tx = blockIdx.x % p.tiles_x, t = blockIdx.x / p.tiles_x;
    const int n = t / p.tiles_y, h0 = t % p.tiles_y * (BM / p.tile_w), w0 = tx * p.tile_w;

    if (tid == 0) {
        prefetch_tensormap(&xmap);
        prefetch_tensormap(&wmap);
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(accd, 1);
        *bad = 0;
        fence_mbar_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    if (warp == 4) {
        const uint32_t on = elect_lane(), ring = smem_u32(base), fb = smem_u32(full);
        RingPos q;
        bool ok = true, wrap = false;  // wrap: the stages have been used before
        for (int tap = 0; tap < 9 && ok; ++tap) {
            const int dy = (tap / 3 - 1) * p.dil, dx = (tap % 3 - 1) * p.dil;
            for (int c = 0; c < nc; ++c) {
                if (wrap && !warp_wait_bounded(&empty[q.slot], q.parity ^ 1)) { ok = false; break; }
                const uint32_t a = ring + q.slot * STAGE, bar = fb + 8 * q.slot;
                expect_tx_if(on, bar, STAGE);
                tma_load_4d_if(on, a, &xmap, bar, c * BC, w0 + dx, h0 + dy, n);
                tma_load_3d_if(on, a + A_BYTES, &wmap, bar, c * BC, tap, n0);
                q.next(p.stages);
                wrap |= q.slot == 0;
            }
        }
        if (!ok && on) *bad = 1;
    } else if (warp == 5) {
        constexpr uint32_t IDESC = umma_idesc<BN>();
        const uint32_t on = elect_lane(), eb = smem_u32(empty);
        const uint64_t ad0 = umma_desc_k<BC>(smem_u32(base)), bd0 = umma_desc_k<BC>(smem_u32(base) + A_BYTES);
        RingPos q;
        bool ok = true;
        uint32_t acc = 0;
        for (int k = 0; k < 9 * nc; ++k) {
            if (!warp_wait_bounded(&full[q.slot], q.parity)) { ok = false; break; }
            tc_fence_after();
            const uint32_t off = q.slot * (STAGE >> 4);
#pragma unroll
            for (int j = 0; j < BC / 16; ++j) {
                mma_f16_if(on, tmem, ad0 + off + 2 * j, bd0 + off + 2 * j, IDESC, acc);
                acc = 1;
            }
            tc_commit_if(on, eb + 8 * q.slot);
            q.next(p.stages);
        }
        if (!ok && on) *bad = 1;
        tc_commit_if(on, smem_u32(accd));  // arrives once every MMA issued above has completed
    } else {
        // epilogue warps 0-3: TMEM lanes 32w .. 32w+31 = the tile's pixels 32w + lane
        const bool done = mbar_wait_bounded(accd, 0);
        tc_fence_after();
        if (done && !*reinterpret_cast<volatile int *>(bad)) {
            const int m = warp * 32 + lane, row = h0 + m / p.tile_w, col = w0 + m % p.tile_w;
            const bool in = row < p.H && col < p.W;
            const long long px = ((long long)n * p.H + row) * p.W + col;
            bf16 *out = y.p + px * y.cs + y.co + n0;
            const bf16 *gt = gate.p + px * gate.cs + gate.co + n0;
#pragma unroll
            for (int c = 0; c < BN; c += 8) {
                uint32_t r[8];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                      "=r"(r[7])
                    : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    v[e] = __uint_as_float(r[e]) + (bias ? bias[n0 + c + e] : 0.f);
                    if (p.relu) v[e] = fmaxf(v[e], 0.f);
                }
                uint4 q;
                __nv_bfloat162 h0v = __floats2bfloat162_rn(v[0], v[1]), h1v = __floats2bfloat162_rn(v[2], v[3]);
                __nv_bfloat162 h2v = __floats2bfloat162_rn(v[4], v[5]), h3v = __floats2bfloat162_rn(v[6], v[7]);
                q.x = *reinterpret_cast<uint32_t *>(&h0v);
                q.y = *reinterpret_cast<uint32_t *>(&h1v);
                q.z = *reinterpret_cast<uint32_t *>(&h2v);
                q.w = *reinterpret_cast<uint32_t *>(&h3v);
                if (in) {
                    if (gate.p) q = gate8(q, *reinterpret_cast<const uint4 *>(gt + c));
                    *reinterpret_cast<uint4 *>(out + c) = q;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
    }
}

// ---------------------------------------------------------------------------
// The same convolution for few channels on wide images (rows longer than 64
// pixels; all the weights of up to 128 output channels in shared memory): one
// CTA marches down the rows of 128-pixel columns.  Each input row is loaded
// once with its column halo into a ring of rows; a tap's A operand is the
// row's slot started dx pixels (rows of 64 bytes) later, so a row serves all
// nine taps, where the tiled form loads it nine times and the weights once
// per tile.  Accumulators alternate between two TMEM buffers, so that the
// epilogue of one row runs under the MMAs of the next.  What bounds it: the
// operand reads of the MMAs (5 KB of shared memory each for 32 output
// channels) and HBM.  Warps: 0-3 epilogue, 4 TMA producer, 5 MMA issuer.
// ---------------------------------------------------------------------------
struct ConvMarch {
    int cin, H, W, n, relu, dil;
    int rows;      // row tiles in all
    int slots;     // ring slots, each one row of every 32-channel chunk
    int rowbytes;  // bytes of one chunk's row in a slot
};

template <int BN>
__global__ void __launch_bounds__(192)
    k_conv3x3_march(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                    const float *__restrict__ bias, Act y, Act gate, ConvMarch p) {
    extern __shared__ __align__(1024) unsigned char mc_smem[];
    constexpr int WT = BN * BK * 2;  // weights of one tap and chunk
    constexpr uint32_t TCOLS = BN <= 32 ? 64 : BN <= 64 ? 128 : 256;
    unsigned char *wsm = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(mc_smem) + 1023) & ~static_cast<uintptr_t>(1023));
    const int nc = p.cin / BK, slot = nc * p.rowbytes, dil = p.dil;
    unsigned char *ring = wsm + 9 * nc * WT;
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + p.slots * slot);
    uint64_t *empty = full + p.slots, *wfull = empty + p.slots, *accf = wfull + 1, *acce = accf + 2;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + 2);
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int n0 = blockIdx.y * BN;
    const int r0 = (int)((long long)p.rows * blockIdx.x / gridDim.x);
    const int r1 = (int)((long long)p.rows * (blockIdx.x + 1) / gridDim.x);

    if (tid == 0) {
        prefetch_tensormap(&xmap);
        prefetch_tensormap(&wmap);
        for (int s = 0; s < p.slots; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(wfull, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&accf[s], 1);
            mbar_init(&acce[s], 4);
        }
        fence_mbar_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(TCOLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    // Row tile r: column segment, image and row; a run of tiles that stays in
    // one image's column is one march.
    if (warp == 4) {
        const uint32_t on = elect_lane(), rs = smem_u32(ring), ws = smem_u32(wsm), fb = smem_u32(full);
        const uint32_t rowtx = nc * (128 + 2 * dil) * BK * 2;
        expect_tx_if(on, smem_u32(wfull), 9 * nc * WT);
        for (int k = 0; k < 9 * nc; ++k)
            tma_load_3d_if(on, ws + k * WT, &wmap, smem_u32(wfull), k % nc * BK, k / nc, n0);
        RingPos q;
        bool ok = true, wrap = false;  // wrap: the slots have been used before
        for (int r = r0; r < r1 && ok;) {
            const int img = r / p.H, y0 = r - img * p.H, y1 = min(p.H, y0 + (r1 - r));
            const int im = img % p.n, w0 = img / p.n * 128 - dil;
            for (int row = y0 - dil; row < y1 + dil; ++row) {
                if (wrap && !warp_wait_bounded(&empty[q.slot], q.parity ^ 1)) { ok = false; break; }
                const uint32_t bar = fb + 8 * q.slot;
                expect_tx_if(on, bar, rowtx);
                for (int c = 0; c < nc; ++c)
                    tma_load_4d_if(on, rs + q.slot * slot + c * p.rowbytes, &xmap, bar, c * BK, w0, row, im);
                q.next(p.slots);
                wrap |= q.slot == 0;
            }
            r += y1 - y0;
        }
    } else if (warp == 5) {
        constexpr uint32_t IDESC = umma_idesc<BN>();
        const uint32_t on = elect_lane(), eb = smem_u32(empty), afb = smem_u32(accf);
        const uint64_t ad0 = umma_desc_k<BK>(smem_u32(ring)), bd0 = umma_desc_k<BK>(smem_u32(wsm));
        RingPos got, acc;
        int first = 0;  // slot of input row y - dil
        bool ok = warp_wait_bounded(wfull, 0), again = false;
        for (int r = r0; r < r1 && ok;) {
            const int y0 = r % p.H, np = min(p.H - y0, r1 - r);
            for (int i = -2 * dil; i < np; ++i) {
                if (!warp_wait_bounded(&full[got.slot], got.parity)) { ok = false; break; }
                got.next(p.slots);
                if (i < 0) continue;
                if (again && !warp_wait_bounded(&acce[acc.slot], acc.parity ^ 1)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem + acc.slot * (TCOLS / 2);
                uint64_t b = bd0;
                int s = first;
                uint32_t more = 0;
                for (int ty = 0; ty < 3; ++ty) {
                    const uint64_t arow = ad0 + s * (slot >> 4);
                    for (int dx = 0; dx < 3; ++dx) {
                        uint64_t a = arow + dx * dil * (BK * 2 / 16);
                        for (int c = 0; c < nc; ++c, a += p.rowbytes >> 4, b += WT >> 4) {
                            mma_f16_if(on, d, a, b, IDESC, more);
                            mma_f16_if(on, d, a + 2, b + 2, IDESC, 1);
                            more = 1;
                        }
                    }
                    s += dil;
                    if (s >= p.slots) s -= p.slots;
                }
                tc_commit_if(on, afb + 8 * acc.slot);
                tc_commit_if(on, eb + 8 * first);
                acc.next(2);
                again |= acc.slot == 0;
                if (++first == p.slots) first = 0;
            }
            if (!ok) break;
            for (int i = 0; i < 2 * dil; ++i) {
                tc_commit_if(on, eb + 8 * first);
                if (++first == p.slots) first = 0;
            }
            r += np;
        }
    } else {
        RingPos acc;
        for (int r = r0; r < r1; ++r) {
            if (!warp_wait_bounded(&accf[acc.slot], acc.parity)) break;
            tc_fence_after();
            const int img = r / p.H, row = r - img * p.H, col = img / p.n * 128 + warp * 32 + lane;
            const bool in = col < p.W;
            const long long px = ((long long)(img % p.n) * p.H + row) * p.W + col;
            bf16 *out = y.p + px * y.cs + y.co + n0;
            const bf16 *gt = gate.p + px * gate.cs + gate.co + n0;
            const uint32_t t = tmem + ((uint32_t)(warp * 32) << 16) + acc.slot * (TCOLS / 2);
#pragma unroll
            for (int c = 0; c < BN; c += 32) {
                uint32_t v[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
                    "[%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                      "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                      "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(t + c));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (c + 32 >= BN) {  // read: the buffer may be written again
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[acc.slot]);
                }
#pragma unroll
                for (int g = 0; g < 32; g += 8) {
                    uint4 q;
                    uint32_t *h = reinterpret_cast<uint32_t *>(&q);
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        float a0 = __uint_as_float(v[g + e]) + (bias ? bias[n0 + c + g + e] : 0.f);
                        float a1 = __uint_as_float(v[g + e + 1]) + (bias ? bias[n0 + c + g + e + 1] : 0.f);
                        if (p.relu) a0 = fmaxf(a0, 0.f), a1 = fmaxf(a1, 0.f);
                        const __nv_bfloat162 b2 = __floats2bfloat162_rn(a0, a1);
                        h[e / 2] = *reinterpret_cast<const uint32_t *>(&b2);
                    }
                    if (in) {
                        if (gate.p) q = gate8(q, *reinterpret_cast<const uint4 *>(gt + c + g));
                        *reinterpret_cast<uint4 *>(out + c + g) = q;
                    }
                }
            }
            acc.next(2);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Weight gradient on tcgen05:
//   dW[co][tap][ci] += sum_p dy[p][co] x[p + tap][ci],  db[co] += sum_p dy[p][co]
// as GEMMs with K = pixels, both operands MN-major: channels are innermost in
// the NHWC views, so a TMA box of 32 channels x a run of pixels of one image
// row (64-byte swizzle) is an operand as it lands, with no transposed copy.
// One CTA owns 32 input channels, up to 128 output channels and the three taps
// of one column shift, and marches down image rows: each input row is loaded
// once, shifted by -dil, 0 or +dil columns (out-of-bounds zeros are the
// padding), into a ring of rows; output row y multiplies dy's row with the
// input rows y - dil, y and y + dil, which are dil ring slots apart: three of
// the four 32-row blocks of an M = 128 instruction (the fourth reads what lies
// behind them; its result rows are not used).  The ring's first 2 * dil slots
// are loaded a second time behind its end, so that the three rows always lie
// in line.  The accumulator [(tap row, ci)][co] in tensor memory ends in FP32
// atomics on dW, coalesced over ci.  In the CTAs of the first channel block the
// idle epilogue warps sum every third row of dy for the bias while it is in
// shared memory (all rows in the CTAs of one shift made those the slowest: 119
// us against 86 on 64 x 128^2, 32 -> 32 channels; rows shared out over all
// channel blocks' CTAs cost more in atomics on the few bias words).
// A step loads rs input rows and the rs rows of dy that they complete (about
// 128 pixels by two 32-channel blocks), with one barrier to wait for and one
// commit, since a wait and a commit cost the issuing warp some 200 cycles.
// What bounds it: the issue of eight MMAs per 128 pixels of a row (5 to 8 KB
// of operands each) behind those, and the few slices of the widest layers.
// Ring positions are counted and never divided (a division per slot made every
// row cost 3500 cycles).  Measured and not kept: dy by cp.async or through
// registers from the idle warps (64 x 128^2, 32 -> 32 channels: 281 and 270 us
// where both operands by TMA took 127).
// Warps: 0-3 bias and epilogue, 4 TMA producer, 5 MMA issuer.
// ---------------------------------------------------------------------------
struct WgradRows {
    int cin, cout, n, H, W, dil;
    int wp, rs;      // a step: rs rows of segments of wp pixels (a multiple of 16, at most 128)
    int rows;        // row segments in all
    int slices;      // CTAs that share them
    int stages;      // steps in flight
    int lag;         // steps between a row's arrival and its last use
    int dslot;       // bytes of a step of dy
    int march;       // dil: a row serves three output rows; 0: its three rows are loaded with each
    int xrows;       // rows of x in shared memory
};

__device__ __forceinline__ uint64_t umma_desc_mn64(uint32_t saddr, uint32_t block_bytes) {
    // MN-major, 64-byte swizzle: 32-element blocks block_bytes apart, groups
    // of 8 K rows 512 bytes apart, version 1
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(block_bytes >> 4) << 16) |
           ((uint64_t)(512 >> 4) << 32) | (1ull << 46) | (4ull << 61);
}

__global__ void __launch_bounds__(192, 2)
    k_wgrad_rows(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap gmap,
                 float *__restrict__ dw, float *__restrict__ db, WgradRows p) {
    extern __shared__ __align__(1024) unsigned char wr_smem[];
    __shared__ float bsum[4][128];
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(wr_smem) + 1023) & ~static_cast<uintptr_t>(1023));
    const int tile = p.wp * 64, dil = p.dil, rs = p.rs, nst = p.stages, nx = nst + p.lag, march = p.march;
    const int xstep = march ? rs : 3 * rs, xend = march ? nx * rs : 1 << 30;  // ring rows of a step; where they wrap
    unsigned char *xring = base, *dring = base + (size_t)p.xrows * tile;
    uint64_t *full = reinterpret_cast<uint64_t *>(dring + (size_t)nst * p.dslot);
    uint64_t *empty = full + nst, *accd = empty + nst;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(accd + 1);
    int *bad = reinterpret_cast<int *>(tslot + 1);
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int shift = blockIdx.y % 3, ci0 = blockIdx.y / 3 * 32, co0 = blockIdx.z * 128;
    const int ncols = min(128, p.cout - co0), nb = ncols / 32;
    const int drow = p.dslot / rs;  // bytes of a row of dy
    const bool bias = db != nullptr && ci0 == 0;
    const int r0 = (int)((long long)p.rows * blockIdx.x / gridDim.x);
    const int r1 = (int)((long long)p.rows * (blockIdx.x + 1) / gridDim.x);
    const uint32_t tcols = ncols <= 32 ? 32 : ncols <= 64 ? 64 : 128;

    if (tid == 0) {
        prefetch_tensormap(&xmap);
        prefetch_tensormap(&gmap);
        for (int s = 0; s < nst; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], bias ? 5 : 1);
        }
        mbar_init(accd, 1);
        *bad = 0;
        fence_mbar_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(tcols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    // Row segment r: segment column, image and row; a run of segments that
    // stays in one image's column (output rows y0 .. y1 - 1) is one march.
    // Its step g brings input rows y0 - dil + g * rs ... and dy's rows that
    // these complete, y0 - 2 * dil + g * rs ..., of which the ones in the
    // march are used.  Where the rows of one march do not fit shared memory
    // (wide dilations) a step brings its rs rows of dy and the three times rs
    // input rows that they meet, one after the other.
    if (warp == 4) {
        const uint32_t on = elect_lane(), xs = smem_u32(xring), ds = smem_u32(dring), fb = smem_u32(full);
        RingPos q;
        int xslot = 0;
        bool ok = true, wrap = false;  // wrap: the stages have been used before
        for (int r = r0; r < r1 && ok;) {
            const int img = r / p.H, y0 = r - img * p.H, y1 = min(p.H, y0 + (r1 - r));
            const int im = img % p.n, w0 = img / p.n * p.wp, xw = w0 + (shift - 1) * dil;
            for (int row = y0 - march; row < y1 + march; row += rs) {
                if (wrap && !warp_wait_bounded(&empty[q.slot], q.parity ^ 1)) { ok = false; break; }
                if (bias) fence_proxy_async();  // the bias warps' reads of the slot before the TMA write
                const uint32_t bar = fb + 8 * q.slot, to = xs + xslot * xstep * tile;
                const bool twice = xslot < p.lag;
                expect_tx_if(on, bar, p.dslot + (march ? twice ? 2 : 1 : 3) * rs * tile);
                tma_load_4d_if(on, to, &xmap, bar, ci0, xw, march ? row : row - dil, im);
                tma_load_5d_if(on, ds + q.slot * p.dslot, &gmap, bar, 0, w0, co0 / 32, row - march, im);
                if (!march) {
                    tma_load_4d_if(on, to + rs * tile, &xmap, bar, ci0, xw, row, im);
                    tma_load_4d_if(on, to + 2 * rs * tile, &xmap, bar, ci0, xw, row + dil, im);
                }
                if (twice) tma_load_4d_if(on, to + nx * rs * tile, &xmap, bar, ci0, xw, row, im);
                if (++xslot == nx) xslot = 0;
                q.next(nst);
                wrap |= q.slot == 0;
            }
            r += y1 - y0;
        }
        if (!ok && on) *bad = 1;
    } else if (warp == 5) {
        // D FP32, A and B BF16, both MN-major, N = ncols, M = 128
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                               ((uint32_t)(ncols >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        const uint64_t adesc = umma_desc_mn64(smem_u32(xring), (march ? dil : rs) * tile), bdesc = umma_desc_mn64(smem_u32(dring), tile);
        const uint32_t astep = tile >> 4, ks = p.wp / 16, on = elect_lane(), fb = smem_u32(empty);
        RingPos q;
        int xslot = 0;
        uint32_t acc = 0;
        bool ok = true;
        for (int r = r0; r < r1 && ok;) {
            const int y0 = r % p.H, np = min(p.H - y0, r1 - r);
            int first = xslot * rs;  // ring row of input row y - dil
            for (int i = -2 * march; i < np; i += rs) {
                if (!warp_wait_bounded(&full[q.slot], q.parity)) { ok = false; break; }
                tc_fence_after();
                if (!march) first = xslot * xstep;
                uint64_t b = bdesc + q.slot * (p.dslot >> 4);
                for (int j = i; j < i + rs; ++j, b += drow >> 4) {
                    if (j < 0 || j >= np) continue;
                    const uint64_t a = adesc + first * astep;
#pragma unroll 4
                    for (uint32_t k = 0; k < ks; ++k) {
                        mma_f16_if(on, tmem, a + k * 64, b + k * 64, idesc, acc);
                        acc = 1;
                    }
                    if (++first == xend) first = 0;
                }
                tc_commit_if(on, fb + 8 * q.slot);
                if (++xslot == nx) xslot = 0;
                q.next(nst);
            }
            r += np;
        }
        if (!ok && on) *bad = 1;
        tc_commit_if(on, smem_u32(accd));  // arrives once every MMA issued above has completed
    } else {
        if (bias) {
            // thread -> 8 channels (a 16-byte chunk) of every 32nd pixel of
            // this CTA's share of the rows
            float s[4][8] = {};
            const int c = tid & 3;
            const unsigned char *own = dring + (tid >> 2) * 64 + ((c ^ ((tid >> 3) & 3)) << 4);  // 64-byte swizzle
            RingPos q;
            bool ok = true;
            for (int r = r0; r < r1 && ok;) {
                const int y0 = r % p.H, np = min(p.H - y0, r1 - r);
                for (int i = -2 * march; i < np; i += rs) {
                    if (!warp_wait_bounded(&full[q.slot], q.parity)) { ok = false; break; }
                    for (int j = max(i, 0); j < min(i + rs, np); ++j) {
                        if ((y0 + j) % 3 != shift) continue;
                        const unsigned char *t = own + q.slot * p.dslot + (j - i) * drow;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (k >= nb) break;
                            uint4 v[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                v[u] = make_uint4(0, 0, 0, 0);
                                if ((tid >> 2) + 32 * u < p.wp)
                                    v[u] = *reinterpret_cast<const uint4 *>(t + k * tile + u * 2048);
                            }
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v[u]);
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const float2 f = __bfloat1622float2(h[e]);
                                    s[k][2 * e] += f.x;
                                    s[k][2 * e + 1] += f.y;
                                }
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[q.slot]);
                    q.next(nst);
                }
                r += np;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    for (int o = 4; o < 32; o <<= 1) s[k][e] += __shfl_xor_sync(0xffffffffu, s[k][e], o);
                    if (lane < 4) bsum[warp][32 * k + 8 * c + e] = s[k][e];
                }
            named_barrier_and(1, 128, true);  // the four warps' sums, then one atomic per channel
            if (tid < ncols) atomicAdd(db + co0 + tid, (bsum[0][tid] + bsum[1][tid]) + (bsum[2][tid] + bsum[3][tid]));
        }
        const bool done = mbar_wait_bounded(accd, 0);
        tc_fence_after();
        if (warp < 3 && done && r1 > r0 && !*reinterpret_cast<volatile int *>(bad)) {
            // warp = tap row, lane = input channel
            float *d = dw + ((long long)co0 * 9 + warp * 3 + shift) * p.cin + ci0 + lane;
            for (int c = 0; c < ncols; c += 8) {
                uint32_t r[8];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                      "=r"(r[7])
                    : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int e = 0; e < 8; ++e) atomicAdd(d + (long long)(c + e) * 9 * p.cin, __uint_as_float(r[e]));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Weight gradient: dW[co][tap][ci] += sum_p dy[p][co] x[p + tap][ci].
// Block: 128 threads = 2 x 2 warps, tile 64 (co) x 64 (ci), K = pixels in
// chunks of 32 from this block's pixel range; grid.z = tap.
// ---------------------------------------------------------------------------
constexpr int WK = 32, WPITCH = 64 + 8;

__global__ void __launch_bounds__(128)
    k_wgrad(Act x, Act dy, float *__restrict__ dw, long long pix_per_block, int dil) {
    __shared__ __align__(128) bf16 As[2][WK][WPITCH];  // [p][co]
    __shared__ __align__(128) bf16 Bs[2][WK][WPITCH];  // [p][ci]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp & 1, wn = warp >> 1;
    const int co0 = blockIdx.x * 64, ci0 = blockIdx.y * 64;
    const int tap = blockIdx.z % 9, split = blockIdx.z / 9;
    const int ddy = (tap / 3 - 1) * dil, ddx = (tap % 3 - 1) * dil;
    const long long P = (long long)x.n * x.h * x.w;
    const long long pb = split * pix_per_block, pe = min(P, pb + pix_per_block);
    if (pb >= pe) return;
    const int KB = (int)((pe - pb + WK - 1) / WK);
    auto load = [&](int kb, int st) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int idx = tid + 128 * i, row = idx >> 3, part = idx & 7;
            const long long p = pb + (long long)kb * WK + row;
            const bool pv = p < pe;
            const long long pp = pv ? p : 0;
            // dy row
            const int co = co0 + part * 8;
            const bool av = pv && co < dy.c;
            cp_async16(&As[st][row][part * 8], dy.p + pp * dy.cs + dy.co + (av ? co : 0), av);
            // shifted x row
            const int xx = (int)(pp % x.w) + ddx;
            const int yy = (int)((pp / x.w) % x.h) + ddy;
            const int nn = (int)(pp / ((long long)x.w * x.h));
            const int ci = ci0 + part * 8;
            const bool bv = pv && ci < x.c && xx >= 0 && xx < x.w && yy >= 0 && yy < x.h;
            const bf16 *src = x.p + (((long long)nn * x.h + (bv ? yy : 0)) * x.w + (bv ? xx : 0)) * x.cs +
                              x.co + (bv ? ci : 0);
            cp_async16(&Bs[st][row][part * 8], src, bv);
        }
        cp_async_commit();
    };
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    load(0, 0);
    for (int kb = 0; kb < KB; ++kb) {
        const int st = kb & 1;
        cp_async_wait_all();
        __syncthreads();
        if (kb + 1 < KB) load(kb + 1, st ^ 1);
#pragma unroll
        for (int ks = 0; ks < WK; ks += 16) {
            uint32_t af[2][4];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) {
                const int q = lane >> 3, r = lane & 7;
                const int krow = ks + r + 8 * (q >> 1);
                const int mcol = wm * 32 + mi * 16 + 8 * (q & 1);
                ldsm_x4_t(smem_u32(&As[st][krow][mcol]), af[mi][0], af[mi][1], af[mi][2], af[mi][3]);
            }
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                const int q = lane >> 3, r = lane & 7;
                const int krow = ks + r + 8 * (q & 1);
                const int ncol = wn * 32 + nj * 16 + 8 * (q >> 1);
                uint32_t b0, b1, b2, b3;
                ldsm_x4_t(smem_u32(&Bs[st][krow][ncol]), b0, b1, b2, b3);
#pragma unroll
                for (int mi = 0; mi < 2; ++mi) {
                    mma16816(acc[mi][2 * nj], af[mi], b0, b1);
                    mma16816(acc[mi][2 * nj + 1], af[mi], b2, b3);
                }
            }
        }
        __syncthreads();
    }
    const int cin = x.c;
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int nj = 0; nj < 4; ++nj)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int co = co0 + wm * 32 + mi * 16 + (lane >> 2) + 8 * hh;
                const int ci = ci0 + wn * 32 + nj * 8 + (lane & 3) * 2;
                if (co >= dy.c || ci >= cin) continue;
                float *d = dw + ((long long)co * 9 + tap) * cin + ci;
                atomicAdd(d, acc[mi][nj][2 * hh]);
                atomicAdd(d + 1, acc[mi][nj][2 * hh + 1]);
            }
}

// Bias gradient: db[c] += sum_p dy[p][c]; one block per 32-channel group.
__global__ void k_bias_grad(Act dy, float *db) {
    __shared__ float sh[8][33];
    const int c = blockIdx.y * 32 + (threadIdx.x & 31);
    const int r = threadIdx.x >> 5;  // 8 warps
    const long long P = (long long)dy.n * dy.h * dy.w;
    float s = 0.f;
    if (c < dy.c)
        for (long long p = blockIdx.x * 8 + r; p < P; p += (long long)gridDim.x * 8)
            s += __bfloat162float(dy.p[p * dy.cs + dy.co + c]);
    sh[r][threadIdx.x & 31] = s;
    __syncthreads();
    if (r == 0 && c < dy.c) {
        float t = 0.f;
        for (int k = 0; k < 8; ++k) t += sh[k][threadIdx.x];
        atomicAdd(&db[c], t);
    }
}

// Weights [co][tap][ci] -> [ci][8 - tap][co] (ky -> 2-ky, kx -> 2-kx) of up to
// kFlipMax layers in one launch: block (32-channel tiles of the layers in
// turn, tap), through shared memory so that both sides are coalesced.
constexpr int kFlipMax = 32;
struct FlipTable {
    const bf16 *w[kFlipMax];
    bf16 *wt[kFlipMax];
    int cout[kFlipMax], cin[kFlipMax];
    int first[kFlipMax + 1];  // tiles of the layers before
    int n;
};
__global__ void __launch_bounds__(256) k_flip(FlipTable t) {
    __shared__ bf16 v[32][33];
    int l = 0;
    while (l + 1 < t.n && (int)blockIdx.x >= t.first[l + 1]) ++l;
    const int cout = t.cout[l], cin = t.cin[l], tile = (int)blockIdx.x - t.first[l], nci = (cin + 31) / 32;
    const int co0 = tile / nci * 32, ci0 = tile % nci * 32, tap = blockIdx.y;
    const int a = (int)threadIdx.x & 31;
    for (int b = (int)threadIdx.x >> 5; b < 32; b += 8)
        if (co0 + b < cout && ci0 + a < cin) v[b][a] = t.w[l][((long long)(co0 + b) * 9 + tap) * cin + ci0 + a];
    __syncthreads();
    for (int b = (int)threadIdx.x >> 5; b < 32; b += 8)
        if (ci0 + b < cin && co0 + a < cout)
            t.wt[l][((long long)(ci0 + b) * 9 + (8 - tap)) * cout + co0 + a] = v[a][b];
}

// Element-wise kernels over 8-channel vectors of a view.
__device__ __forceinline__ long long vec_count(const Act &a) {
    return (long long)a.n * a.h * a.w * (a.c / 8);
}
__device__ __forceinline__ uint4 *vec_at(const Act &a, long long v) {
    const long long p = v / (a.c / 8);
    const int c8 = (int)(v % (a.c / 8));
    return reinterpret_cast<uint4 *>(a.p + p * a.cs + a.co + c8 * 8);
}

__global__ void k_relu_bwd(Act g, Act y) {
    const long long n = vec_count(g);
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n;
         v += (long long)gridDim.x * blockDim.x) {
        uint4 gv = *vec_at(g, v);
        const uint4 yv = *vec_at(y, v);
        __nv_bfloat162 *gp = reinterpret_cast<__nv_bfloat162 *>(&gv);
        const __nv_bfloat162 *yp = reinterpret_cast<const __nv_bfloat162 *>(&yv);
        const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 yf = __bfloat1622float2(yp[k]);
            float2 gf = __bfloat1622float2(gp[k]);
            gf.x = yf.x > 0.f ? gf.x : 0.f;
            gf.y = yf.y > 0.f ? gf.y : 0.f;
            gp[k] = __float22bfloat162_rn(gf);
        }
        (void)zero;
        *vec_at(g, v) = gv;
    }
}

__global__ void k_add(Act a, Act b) {
    const long long n = vec_count(a);
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n;
         v += (long long)gridDim.x * blockDim.x) {
        uint4 av = *vec_at(a, v);
        const uint4 bv = *vec_at(b, v);
        __nv_bfloat162 *ap = reinterpret_cast<__nv_bfloat162 *>(&av);
        const __nv_bfloat162 *bp = reinterpret_cast<const __nv_bfloat162 *>(&bv);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 x = __bfloat1622float2(ap[k]), y = __bfloat1622float2(bp[k]);
            ap[k] = __floats2bfloat162_rn(x.x + y.x, x.y + y.y);
        }
        *vec_at(a, v) = av;
    }
}

// y (h/2 x w/2) = max over 2x2 blocks of x.
__global__ void k_pool_fwd(Act x, Act y) {
    const long long n = vec_count(y);
    const int c8n = y.c / 8;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n;
         v += (long long)gridDim.x * blockDim.x) {
        const int c8 = (int)(v % c8n);
        const long long p = v / c8n;
        const int ox = (int)(p % y.w), oy = (int)((p / y.w) % y.h), nn = (int)(p / ((long long)y.w * y.h));
        float m[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) m[k] = -3.0e38f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const long long ip = ((long long)nn * x.h + 2 * oy + (q >> 1)) * x.w + 2 * ox + (q & 1);
            const uint4 xv = *reinterpret_cast<const uint4 *>(x.p + ip * x.cs + x.co + c8 * 8);
            const __nv_bfloat162 *xp = reinterpret_cast<const __nv_bfloat162 *>(&xv);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(xp[k]);
                m[2 * k] = fmaxf(m[2 * k], f.x);
                m[2 * k + 1] = fmaxf(m[2 * k + 1], f.y);
            }
        }
        uint4 ov;
        __nv_bfloat162 *op = reinterpret_cast<__nv_bfloat162 *>(&ov);
#pragma unroll
        for (int k = 0; k < 4; ++k) op[k] = __floats2bfloat162_rn(m[2 * k], m[2 * k + 1]);
        *reinterpret_cast<uint4 *>(y.p + p * y.cs + y.co + c8 * 8) = ov;
    }
}

// dx = dy routed to the first input of each 2x2 block equal to the max (y);
// with a skip gradient (skip.p), that is added (one rounding to BF16, as a sum
// of two stored gradients) and the result passes where x > 0.
__global__ void k_pool_bwd(Act x, Act y, Act dy, Act skip, Act dx) {
    const long long n = vec_count(y);
    const int c8n = y.c / 8;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n;
         v += (long long)gridDim.x * blockDim.x) {
        const int c8 = (int)(v % c8n);
        const long long p = v / c8n;
        const int ox = (int)(p % y.w), oy = (int)((p / y.w) % y.h), nn = (int)(p / ((long long)y.w * y.h));
        const uint4 yv = *reinterpret_cast<const uint4 *>(y.p + p * y.cs + y.co + c8 * 8);
        const uint4 gv = *reinterpret_cast<const uint4 *>(dy.p + p * dy.cs + dy.co + c8 * 8);
        const bf16 *yb = reinterpret_cast<const bf16 *>(&yv);
        const bf16 *gb = reinterpret_cast<const bf16 *>(&gv);
        bool taken[8] = {false, false, false, false, false, false, false, false};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const long long ip = ((long long)nn * x.h + 2 * oy + (q >> 1)) * x.w + 2 * ox + (q & 1);
            const uint4 xv = *reinterpret_cast<const uint4 *>(x.p + ip * x.cs + x.co + c8 * 8);
            const bf16 *xb = reinterpret_cast<const bf16 *>(&xv);
            uint4 ov;
            bf16 *ob = reinterpret_cast<bf16 *>(&ov);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const bool hit = !taken[k] && __bfloat162float(xb[k]) == __bfloat162float(yb[k]);
                taken[k] = taken[k] || hit;
                ob[k] = hit ? gb[k] : __float2bfloat16_rn(0.f);
            }
            if (skip.p) {
                const uint4 sv = *reinterpret_cast<const uint4 *>(skip.p + ip * skip.cs + skip.co + c8 * 8);
                __nv_bfloat162 *op = reinterpret_cast<__nv_bfloat162 *>(&ov);
                const __nv_bfloat162 *sp = reinterpret_cast<const __nv_bfloat162 *>(&sv);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 a = __bfloat1622float2(op[k]), b = __bfloat1622float2(sp[k]);
                    op[k] = __floats2bfloat162_rn(a.x + b.x, a.y + b.y);
                }
                ov = gate8(ov, xv);
            }
            *reinterpret_cast<uint4 *>(dx.p + ip * dx.cs + dx.co + c8 * 8) = ov;
        }
    }
}

__global__ void k_up_fwd(Act x, Act y) {
    const long long n = vec_count(y);
    const int c8n = y.c / 8;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n;
         v += (long long)gridDim.x * blockDim.x) {
        const int c8 = (int)(v % c8n);
        const long long p = v / c8n;
        const int ox = (int)(p % y.w), oy = (int)((p / y.w) % y.h), nn = (int)(p / ((long long)y.w * y.h));
        const long long ip = ((long long)nn * x.h + oy / 2) * x.w + ox / 2;
        *reinterpret_cast<uint4 *>(y.p + p * y.cs + y.co + c8 * 8) =
            *reinterpret_cast<const uint4 *>(x.p + ip * x.cs + x.co + c8 * 8);
    }
}

// gate.p: the result passes where the gate is positive.
__global__ void k_up_bwd(Act dy, Act gate, Act dx) {
    const long long n = vec_count(dx);
    const int c8n = dx.c / 8;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n;
         v += (long long)gridDim.x * blockDim.x) {
        const int c8 = (int)(v % c8n);
        const long long p = v / c8n;
        const int ox = (int)(p % dx.w), oy = (int)((p / dx.w) % dx.h), nn = (int)(p / ((long long)dx.w * dx.h));
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const long long ip = ((long long)nn * dy.h + 2 * oy + (q >> 1)) * dy.w + 2 * ox + (q & 1);
            const uint4 gv = *reinterpret_cast<const uint4 *>(dy.p + ip * dy.cs + dy.co + c8 * 8);
            const __nv_bfloat162 *gp = reinterpret_cast<const __nv_bfloat162 *>(&gv);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(gp[k]);
                s[2 * k] += f.x;
                s[2 * k + 1] += f.y;
            }
        }
        uint4 ov;
        __nv_bfloat162 *op = reinterpret_cast<__nv_bfloat162 *>(&ov);
#pragma unroll
        for (int k = 0; k < 4; ++k) op[k] = __floats2bfloat162_rn(s[2 * k], s[2 * k + 1]);
        if (gate.p) ov = gate8(ov, *reinterpret_cast<const uint4 *>(gate.p + p * gate.cs + gate.co + c8 * 8));
        *reinterpret_cast<uint4 *>(dx.p + p * dx.cs + dx.co + c8 * 8) = ov;
    }
}

// Head: one warp per pixel group; channel count <= 256 (multiple of 8).
__global__ void k_head_fwd(Act x, const float *__restrict__ w, const float *__restrict__ b,
                           float *__restrict__ y) {
    const long long P = (long long)x.n * x.h * x.w;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
         p += (long long)gridDim.x * blockDim.x) {
        float s = b[0];
        for (int c = 0; c < x.c; c += 8) {
            const uint4 xv = *reinterpret_cast<const uint4 *>(x.p + p * x.cs + x.co + c);
            const __nv_bfloat162 *xp = reinterpret_cast<const __nv_bfloat162 *>(&xv);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(xp[k]);
                s = fmaf(f.x, w[c + 2 * k], s);
                s = fmaf(f.y, w[c + 2 * k + 1], s);
            }
        }
        y[p] = s;
    }
}

// Head gradient: dx = dy w (where x > 0 with GATE), dw += sum dy x, db += sum
// dy.  A thread owns 8 channels of every groups-th pixel and keeps their sums
// in registers; bound by HBM (64 x 128^2 x 32 channels: 502 us with an atomic
// on shared memory per value, 42 us so).
template <bool GATE>
__global__ void __launch_bounds__(256) k_head_bwd(Act x, const float *__restrict__ w, const float *__restrict__ dy, Act dx,
                                                  float *__restrict__ dw, float *__restrict__ db) {
    __shared__ float sdw[256];
    __shared__ float sdb;
    sdw[threadIdx.x] = 0.f;
    if (threadIdx.x == 0) sdb = 0.f;
    __syncthreads();
    const int c8n = x.c / 8, groups = 256 / c8n, c = (int)threadIdx.x % c8n * 8, grp = (int)threadIdx.x / c8n;
    const long long P = (long long)x.n * x.h * x.w;
    float wv[8], s[8] = {}, sb = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) wv[k] = w[c + k];
    if (grp < groups)
        for (long long p = (long long)blockIdx.x * groups + grp; p < P; p += (long long)gridDim.x * groups) {
            const float g = dy[p];
            if (c == 0) sb += g;
            const uint4 xv = *reinterpret_cast<const uint4 *>(x.p + p * x.cs + x.co + c);
            const __nv_bfloat162 *xp = reinterpret_cast<const __nv_bfloat162 *>(&xv);
            uint4 ov;
            __nv_bfloat162 *op = reinterpret_cast<__nv_bfloat162 *>(&ov);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(xp[k]);
                s[2 * k] += g * f.x;
                s[2 * k + 1] += g * f.y;
                op[k] = __floats2bfloat162_rn(g * wv[2 * k], g * wv[2 * k + 1]);
            }
            if (GATE) ov = gate8(ov, xv);
            *reinterpret_cast<uint4 *>(dx.p + p * dx.cs + dx.co + c) = ov;
        }
    if (grp < groups) {
#pragma unroll
        for (int k = 0; k < 8; ++k) atomicAdd(&sdw[c + k], s[k]);
        if (c == 0) atomicAdd(&sdb, sb);
    }
    __syncthreads();
    if ((int)threadIdx.x < x.c) atomicAdd(&dw[threadIdx.x], sdw[threadIdx.x]);
    if (threadIdx.x == 0) atomicAdd(db, sdb);
}

// Features: ch0 border field, ch1 mask, ch2 Coons patch, other channels 0.
__global__ void k_features(const float *__restrict__ f, int n, int h, int w, Act x,
                           float *__restrict__ coons) {
    const long long P = (long long)n * h * w;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
         p += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(p % w), j = (int)((p / w) % h), nn = (int)(p / ((long long)w * h));
        const float *g = f + (long long)nn * h * w;
        const bool bnd = i == 0 || j == 0 || i == w - 1 || j == h - 1;
        const float s = (float)i / (w - 1), t = (float)j / (h - 1);
        const float B = g[i], T = g[(long long)(h - 1) * w + i];
        const float L = g[(long long)j * w], Rr = g[(long long)j * w + w - 1];
        const float c00 = g[0], c10 = g[w - 1], c01 = g[(long long)(h - 1) * w], c11 = g[(long long)h * w - 1];
        float cp = (1 - t) * B + t * T + (1 - s) * L + s * Rr -
                   ((1 - s) * (1 - t) * c00 + s * (1 - t) * c10 + (1 - s) * t * c01 + s * t * c11);
        if (bnd) cp = g[(long long)j * w + i];
        if (coons) coons[p] = cp;
        bf16 *o = x.p + p * x.cs + x.co;
        for (int c = 0; c < x.c; c += 8) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (c == 0) {
                __nv_bfloat162 *vp = reinterpret_cast<__nv_bfloat162 *>(&v);
                vp[0] = __floats2bfloat162_rn(bnd ? g[(long long)j * w + i] : 0.f, bnd ? 1.f : 0.f);
                vp[1] = __floats2bfloat162_rn(cp, 0.f);
            }
            *reinterpret_cast<uint4 *>(o + c) = v;
        }
    }
}

__global__ void k_mse(const float *__restrict__ out, const float *__restrict__ coons,
                      const float *__restrict__ target, int n, int h, int w, float scale,
                      float *loss, float *__restrict__ dout) {
    const long long P = (long long)n * h * w;
    float s = 0.f;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
         p += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(p % w), j = (int)((p / w) % h);
        const bool bnd = i == 0 || j == 0 || i == w - 1 || j == h - 1;
        float g = 0.f;
        if (!bnd) {
            const float d = coons[p] + out[p] - target[p];
            s += d * d;
            g = 2.f * d * scale;
        }
        dout[p] = g;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, s);
}

__global__ void k_adam(float *p, const float *g, float *m, float *v, bf16 *pb, long long n, float lr,
                       float b1, float b2, float eps, float c1, float c2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        if (pb) pb[i] = __float2bfloat16_rn(pi);
    }
}

__global__ void k_assemble(const float *f, const float *coons, const float *out, int n, int h, int w,
                           float *u) {
    const long long P = (long long)n * h * w;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
         p += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(p % w), j = (int)((p / w) % h);
        const bool bnd = i == 0 || j == 0 || i == w - 1 || j == h - 1;
        u[p] = bnd ? f[p] : coons[p] + out[p];
    }
}

// Transfinite (Coons) interpolation of each field's border on its interior,
// the border band copied (the formula of k_features' channel 2).
__global__ void k_coons_fill(const float *__restrict__ f, int n, int h, int w, float *__restrict__ u) {
    const long long P = (long long)n * h * w;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
         p += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(p % w), j = (int)((p / w) % h), nn = (int)(p / ((long long)w * h));
        const float *g = f + (long long)nn * h * w;
        const bool bnd = i == 0 || j == 0 || i == w - 1 || j == h - 1;
        const float s = (float)i / (w - 1), t = (float)j / (h - 1);
        const float B = g[i], T = g[(long long)(h - 1) * w + i];
        const float L = g[(long long)j * w], Rr = g[(long long)j * w + w - 1];
        const float c00 = g[0], c10 = g[w - 1], c01 = g[(long long)(h - 1) * w], c11 = g[(long long)h * w - 1];
        const float cp = (1 - t) * B + t * T + (1 - s) * L + s * Rr -
                         ((1 - s) * (1 - t) * c00 + s * (1 - t) * c10 + (1 - s) * t * c01 + s * t * c11);
        u[p] = bnd ? g[(long long)j * w + i] : cp;
    }
}

// Nearest source index of coarse index k when k = 0..m-1 spans 0..M-1:
// round(k (M-1) / (m-1)), ties up.
__device__ __forceinline__ int nearest_index(int k, int m, int M) {
    return m > 1 ? (int)((2LL * k * (M - 1) + (m - 1)) / (2LL * (m - 1))) : 0;
}

// Coarse h x w problems from fine H x W borders: each coarse border cell
// takes the fine border value at the nearest position; interior zero.
__global__ void k_resample_border(const float *__restrict__ f, int n, int H, int W, int h, int w,
                                  float *__restrict__ c) {
    const long long P = (long long)n * h * w;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
         p += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(p % w), j = (int)((p / w) % h), nn = (int)(p / ((long long)w * h));
        const bool bnd = i == 0 || j == 0 || i == w - 1 || j == h - 1;
        float v = 0.0f;
        if (bnd)
            v = f[(long long)nn * H * W + (long long)nearest_index(j, h, H) * W + nearest_index(i, w, W)];
        c[p] = v;
    }
}

// Fine H x W fields from coarse h x w ones: bilinear interpolation with the
// corner cells aligned (fine index I maps to I (w-1)/(W-1)) on the interior;
// the fine border band is copied from f.
__global__ void k_upsample_bilinear(const float *__restrict__ c, int n, int h, int w,
                                    const float *__restrict__ f, int H, int W, float *__restrict__ u) {
    const long long P = (long long)n * H * W;
    const float sx = W > 1 ? (float)(w - 1) / (float)(W - 1) : 0.0f;
    const float sy = H > 1 ? (float)(h - 1) / (float)(H - 1) : 0.0f;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
         p += (long long)gridDim.x * blockDim.x) {
        const int I = (int)(p % W), J = (int)((p / W) % H), nn = (int)(p / ((long long)W * H));
        if (I == 0 || J == 0 || I == W - 1 || J == H - 1) {
            u[p] = f[p];
            continue;
        }
        const float x = I * sx, y = J * sy;
        const int x0 = min((int)x, w - 2), y0 = min((int)y, h - 2);
        const float ax = x - x0, ay = y - y0;
        const float *g = c + (long long)nn * h * w + (long long)y0 * w + x0;
        const float top = (1.0f - ax) * g[0] + ax * g[1];
        const float bot = (1.0f - ax) * g[w] + ax * g[w + 1];
        u[p] = (1.0f - ay) * top + ay * bot;
    }
}

__global__ void k_to_bf16(const float *s, bf16 *d, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        d[i] = __float2bfloat16_rn(s[i]);
}

int check_act(const unet_act *a, const char *what) {
    if (!a || !a->ptr) return fail(STENCIL_EINVAL, "%s: null view", what);
    if (a->n < 1 || a->h < 1 || a->w < 1 || a->c < 8 || a->c % 8 || a->c_stride % 8 ||
        a->c_off % 8 || a->c_off + a->c > a->c_stride)
        return fail(STENCIL_EINVAL, "%s: bad view (c %d, stride %d, off %d)", what, a->c, a->c_stride, a->c_off);
    if (reinterpret_cast<uintptr_t>(a->ptr) & 15) return fail(STENCIL_EINVAL, "%s: 16-byte alignment", what);
    return STENCIL_OK;
}

int grid_for(long long n) {
    long long b = (n + 255) / 256;
    const long long cap = 16LL * num_sms();
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace
}  // namespace st

using namespace st;

#define CHECK_VIEW(v) \
    do { int rc_ = check_act(v, #v); if (rc_) return rc_; } while (0)
#define STREAM(s) reinterpret_cast<cudaStream_t>(s)

// Columns of a 128-pixel tile (its rows: 128 over that) that cover an H x W
// image with the fewest tiles.
int tma_tile_w(int H, int W) {
    int best = 128, count = 1 << 30;
    for (int tw : {128, 64, 32, 16, 8}) {
        const int th = BM / tw, n = ((W + tw - 1) / tw) * ((H + th - 1) / th);
        if (n < count) count = n, best = tw;
    }
    return best;
}

template <int BN, int BC>
int launch_conv_tma(const unet_act *x, const bf16 *wb, const float *b, const Act &ya, const Act &gate, int relu,
                    int dil, cudaStream_t s) {
    constexpr int STAGE = (BM + BN) * BC * 2, SMEM_MAX = 200 * 1024;
    static bool attr[64] = {false};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && !attr[dev]) {
        ST_CUDA(cudaFuncSetAttribute(k_conv3x3_tma<BN, BC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SMEM_MAX + 2048));
        attr[dev] = true;
    }
    const int cin = x->c, cout = ya.c, tw = tma_tile_w(x->h, x->w), th = BM / tw;
    CUtensorMap xm, wm;
    const unsigned long long cs2 = (unsigned long long)x->c_stride * 2;
    const unsigned long long xd[4] = {(unsigned long long)cin, (unsigned long long)x->w,
                                      (unsigned long long)x->h, (unsigned long long)x->n};
    const unsigned long long xs[3] = {cs2, cs2 * x->w, cs2 * x->w * x->h};
    const unsigned xb[4] = {(unsigned)BC, (unsigned)tw, (unsigned)th, 1u};
    const bf16 *xbase = static_cast<const bf16 *>(x->ptr) + x->c_off;
    const CUtensorMapSwizzle swz = BC == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    int rc = make_tensor_map_general(&xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, xbase, xd, xs, xb, swz);
    if (rc) return rc;
    const unsigned long long wd[3] = {(unsigned long long)cin, 9ull, (unsigned long long)cout};
    const unsigned long long ws[2] = {(unsigned long long)cin * 2, 9ull * cin * 2};
    const unsigned wbx[3] = {(unsigned)BC, 1u, (unsigned)BN};
    rc = make_tensor_map_general(&wm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, wb, wd, ws, wbx, swz);
    if (rc) return rc;
    ConvTiles p = {cin, x->h, x->w, tw, (x->w + tw - 1) / tw, (x->h + th - 1) / th, relu, dil, 0};
    const dim3 grid((unsigned)((long long)p.tiles_x * p.tiles_y * x->n), cout / BN);
    // a lone CTA per SM gets a deep ring; otherwise several share the SM, the
    // more the fewer channels a tile has (64^2, 64 -> 64: 41 us with two stages,
    // 48 with four; 32^2, 384 -> 128: 66 us with two, 53 with three)
    const int budget = (long long)grid.x * grid.y <= num_sms() ? SMEM_MAX : BN == 128 ? 100 * 1024 : 48 * 1024;
    p.stages = std::max(2, std::min(9 * cin / BC, std::min(8, budget / STAGE)));
    const int smem = p.stages * STAGE + (2 * p.stages + 1) * 8 + 16 + 1024;
    k_conv3x3_tma<BN, BC><<<grid, 192, smem, s>>>(xm, wm, b, ya, gate, p);
    return cuda_fail(cudaGetLastError(), "conv3x3 (tcgen05, TMA) launch");
}

// Tiles of BN output channels, or of half as many as long as all their CTAs
// still find an SM of their own: a lone CTA's time is its chain of K chunks,
// each as long as its TMA rows (128 of the input, BN of the weights) take.
// One image, us: 32^2 384 -> 128 14.9 -> 8.9 with 32 output channels a tile
// instead of 128, 16^2 256 -> 256 16.3 -> 9.5, 64^2 192 -> 64 9.5 -> 7.8.
template <int BN>
int launch_conv_tma(const unet_act *x, const bf16 *wb, const float *b, const Act &ya, const Act &gate, int relu,
                    int dil, cudaStream_t s) {
    if constexpr (BN > 32) {
        const int tw = tma_tile_w(x->h, x->w), th = BM / tw;
        const long long tiles = (long long)((x->w + tw - 1) / tw) * ((x->h + th - 1) / th) * x->n;
        if (2 * tiles * (ya.c / BN) <= num_sms()) return launch_conv_tma<BN / 2>(x, wb, b, ya, gate, relu, dil, s);
    }
    return x->c % 64 == 0 ? launch_conv_tma<BN, 64>(x, wb, b, ya, gate, relu, dil, s)
                          : launch_conv_tma<BN, 32>(x, wb, b, ya, gate, relu, dil, s);
}

// Whether the marching form takes the layer, and its plan: rows of more than
// 64 pixels (a tile is 128 pixels of one row), two row tiles per SM or more,
// and weights plus 2 * dil + 2 rows in shared memory.  Six slots let three
// CTAs share an SM at 32 -> 32 channels (39 us against 43 with eight slots and
// two CTAs); with 96 outputs one CTA with eight slots is faster than two (93 /
// 103 us).
constexpr int CM_SMEM = 200 * 1024;
template <int BN>
bool conv_march_plan(const unet_act *x, int relu, int dil, ConvMarch *p) {
    if (x->w <= 64 || dil > 32) return false;
    const int nc = x->c / BK, rowbytes = ((128 + 2 * dil) * BK * 2 + 1023) / 1024 * 1024;
    const int slots = std::min(BN <= 64 ? 6 : 8, (CM_SMEM - 9 * nc * BN * BK * 2) / (nc * rowbytes));
    if (slots < 2 * dil + 2) return false;
    const long long rows = (long long)x->n * x->h * ((x->w + 127) / 128);
    if (rows < 2LL * num_sms() || rows >= (1LL << 31)) return false;
    *p = {x->c, x->h, x->w, x->n, relu, dil, (int)rows, slots, rowbytes};
    return true;
}

template <int BN>
int launch_conv_march(const unet_act *x, const bf16 *wb, const float *b, const Act &ya, const Act &gate,
                      const ConvMarch &p, cudaStream_t s) {
    static bool attr[64] = {false};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && !attr[dev]) {
        ST_CUDA(cudaFuncSetAttribute(k_conv3x3_march<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, CM_SMEM + 2048));
        attr[dev] = true;
    }
    typedef unsigned long long u64;
    CUtensorMap xm, wm;
    const u64 cs2 = 2ull * x->c_stride, cin = x->c;
    const u64 xd[4] = {cin, (u64)x->w, (u64)x->h, (u64)x->n}, xs[3] = {cs2, cs2 * x->w, cs2 * x->w * x->h};
    const unsigned xb[4] = {(unsigned)BK, (unsigned)(128 + 2 * p.dil), 1u, 1u};
    int rc = make_tensor_map_general(&xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, static_cast<const bf16 *>(x->ptr) + x->c_off,
                                     xd, xs, xb, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
    const u64 wd[3] = {cin, 9, (u64)ya.c}, ws[2] = {cin * 2, 9 * cin * 2};
    const unsigned wbx[3] = {(unsigned)BK, 1u, (unsigned)BN};
    rc = make_tensor_map_general(&wm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, wb, wd, ws, wbx, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
    const int nc = p.cin / BK;
    const int smem = 9 * nc * BN * BK * 2 + p.slots * nc * p.rowbytes + 1024 + (2 * p.slots + 5) * 8 + 16;
    const int per_sm = std::max(1, std::min(512 / (BN <= 32 ? 64 : BN <= 64 ? 128 : 256), (227 * 1024) / (smem + 1024)));
    const int ctas = std::max(1, std::min(p.rows, per_sm * num_sms() / (ya.c / BN)));
    k_conv3x3_march<BN><<<dim3(ctas, ya.c / BN), 192, smem, s>>>(xm, wm, b, ya, gate, p);
    return cuda_fail(cudaGetLastError(), "conv3x3 (tcgen05, rows) launch");
}

template <int BN>
int launch_conv(const unet_act *x, const bf16 *wb, const float *b, const Act &ya, const Act &gate, int relu, int dil,
                cudaStream_t s) {
    ConvMarch m;
    if (conv_march_plan<BN>(x, relu, dil, &m)) return launch_conv_march<BN>(x, wb, b, ya, gate, m, s);
    // tiles of at most 128 channels whose number divides the layer's
    if constexpr (BN == 96) return launch_conv_tma<32>(x, wb, b, ya, gate, relu, dil, s);
    else return launch_conv_tma<BN>(x, wb, b, ya, gate, relu, dil, s);
}

// The tcgen05 convolution; gate.p null: none.
int conv_tcgen05(const unet_act *x, const bf16 *wb, const float *b, const Act &ya, const Act &gate, int relu, int dil,
                 cudaStream_t s) {
    if (ya.c % 128 == 0) return launch_conv<128>(x, wb, b, ya, gate, relu, dil, s);
    if (ya.c == 96) return launch_conv<96>(x, wb, b, ya, gate, relu, dil, s);
    if (ya.c == 64) return launch_conv<64>(x, wb, b, ya, gate, relu, dil, s);
    if (ya.c == 32) return launch_conv<32>(x, wb, b, ya, gate, relu, dil, s);
    return ya.c % 64 == 0 ? launch_conv_tma<64>(x, wb, b, ya, gate, relu, dil, s)
                          : launch_conv_tma<32>(x, wb, b, ya, gate, relu, dil, s);
}

extern "C" int unet_conv3x3_fwd_engine(const unet_act *x, const void *w, const float *b,
                                       const unet_act *y, int relu, int dilation, int engine,
                                       stencil_stream_t s) {
    CHECK_VIEW(x);
    CHECK_VIEW(y);
    if (!w) return fail(STENCIL_EINVAL, "null weights");
    if (dilation < 1) return fail(STENCIL_EINVAL, "dilation must be >= 1");
    if (engine < 0 || engine > 2) return fail(STENCIL_EINVAL, "engine must be 0, 1 or 2");
    if (x->c % 32 || y->c % 32) return fail(STENCIL_EINVAL, "channels must be multiples of 32");
    if (x->n != y->n || x->h != y->h || x->w != y->w) return fail(STENCIL_EINVAL, "shape mismatch");
    const long long P = (long long)x->n * x->h * x->w;
    const Act xa = to_act(*x), ya = to_act(*y);
    const bf16 *wb = static_cast<const bf16 *>(w);
    // tcgen05 with TMA-fed operands for every shape (bit for bit the mma.sync
    // engine's results, 1.6 to 5 times as fast on the U-Net's layers); the
    // marching form where it fits and its row tiles fill the GPU more than
    // once (64 x 128^2, us, marching / tiled / mma.sync: 32 -> 32 channels 39 /
    // 74 / 149, 96 -> 32 96 / 146 / 349, 32 -> 96 93 / 231 / 425; one 128^2
    // image 8 / 7 / 12)
    if (engine != 2) return conv_tcgen05(x, wb, b, ya, Act{}, relu, dilation, STREAM(s));
    if (y->c % 64 == 0) {
        dim3 grid((unsigned)((P + BM - 1) / BM), y->c / 64);
        k_conv3x3<64><<<grid, 128, 0, STREAM(s)>>>(xa, wb, b, ya, relu, dilation);
    } else {
        dim3 grid((unsigned)((P + BM - 1) / BM), y->c / 32);
        k_conv3x3<32><<<grid, 128, 0, STREAM(s)>>>(xa, wb, b, ya, relu, dilation);
    }
    return cuda_fail(cudaGetLastError(), "conv3x3 launch");
}

extern "C" int unet_conv3x3_dgrad_relu(const unet_act *dy, const void *wt, const unet_act *gate, const unet_act *dx,
                                       int dilation, stencil_stream_t s) {
    CHECK_VIEW(dy);
    CHECK_VIEW(gate);
    CHECK_VIEW(dx);
    if (!wt) return fail(STENCIL_EINVAL, "null weights");
    if (dilation < 1) return fail(STENCIL_EINVAL, "dilation must be >= 1");
    if (dy->c % 32 || dx->c % 32) return fail(STENCIL_EINVAL, "channels must be multiples of 32");
    if (dy->n != dx->n || dy->h != dx->h || dy->w != dx->w || gate->n != dx->n || gate->h != dx->h ||
        gate->w != dx->w || gate->c != dx->c)
        return fail(STENCIL_EINVAL, "shape mismatch");
    return conv_tcgen05(dy, static_cast<const bf16 *>(wt), nullptr, to_act(*dx), to_act(*gate), 0, dilation, STREAM(s));
}

extern "C" int unet_conv3x3_fwd_dil(const unet_act *x, const void *w, const float *b,
                                    const unet_act *y, int relu, int dilation, stencil_stream_t s) {
    return unet_conv3x3_fwd_engine(x, w, b, y, relu, dilation, 0, s);
}

extern "C" int unet_conv3x3_fwd(const unet_act *x, const void *w, const float *b, const unet_act *y,
                                int relu, stencil_stream_t s) {
    return unet_conv3x3_fwd_dil(x, w, b, y, relu, 1, s);
}

extern "C" int unet_flip_weights_many(const unet_flip *layers, int count, stencil_stream_t s) {
    if (count < 0 || (count && !layers)) return fail(STENCIL_EINVAL, "bad arguments");
    for (int k = 0; k < count; ++k)
        if (!layers[k].w || !layers[k].wt || layers[k].cout < 1 || layers[k].cin < 1)
            return fail(STENCIL_EINVAL, "bad arguments (layer %d)", k);
    for (int k0 = 0; k0 < count; k0 += kFlipMax) {
        FlipTable t;
        t.n = std::min(kFlipMax, count - k0);
        t.first[0] = 0;
        for (int k = 0; k < t.n; ++k) {
            const unet_flip &f = layers[k0 + k];
            t.w[k] = static_cast<const bf16 *>(f.w);
            t.wt[k] = static_cast<bf16 *>(f.wt);
            t.cout[k] = f.cout;
            t.cin[k] = f.cin;
            t.first[k + 1] = t.first[k] + (f.cout + 31) / 32 * ((f.cin + 31) / 32);
        }
        k_flip<<<dim3(t.first[t.n], 9), 256, 0, STREAM(s)>>>(t);
        int rc = cuda_fail(cudaGetLastError(), "flip launch");
        if (rc) return rc;
    }
    return STENCIL_OK;
}

extern "C" int unet_flip_weights(const void *w, void *wt, int cout, int cin, stencil_stream_t s) {
    const unet_flip f = {w, wt, cout, cin};
    return unet_flip_weights_many(&f, 1, s);
}

namespace {

// The row-marching weight gradient's plan for a layer; false where its channels
// are not multiples of 32.  Two CTAs share an SM where the rings allow it.
// Dilations beyond about 20, of which no march fits shared memory in segments
// of 16 pixels, load their input rows three times (64 x 128^2, 32 -> 32 channels,
// dilation 32: 86 us; mma.sync 1026; dilation 1, marching, 91).
constexpr int WR_SMEM = 107 * 1024, WR_SMEM_MAX = 218 * 1024;
bool wgrad_rows_plan(const unet_act *x, const unet_act *dy, int dil, WgradRows *p) {
    if (x->c % 32 || dy->c % 32 || (long long)x->n * x->h * ((x->w + 15) / 16) >= (1LL << 31)) return false;
    const int nb = std::min(dy->c, 128) / 32;
    for (int n = 0; n < 4; ++n)
        for (int wp : {128, 64, 32, 16}) {
            const int budget = n % 2 ? WR_SMEM_MAX : WR_SMEM, march = n < 2 ? dil : 0;
            if ((long long)march * 128 > WR_SMEM_MAX) continue;
            // the shortest segment that covers a row, else the longest that fits
            if (wp > 16 && wp / 2 >= x->w) continue;
            wp = std::min(wp, (x->w + 15) / 16 * 16);
            const int rs = std::max(1, 256 / (wp * nb)), tile = wp * 64, lag = (2 * march + rs - 1) / rs;
            const int dslot = rs * nb * tile, fixed = 2 * lag * rs + march, xstep = march ? rs : 3 * rs;
            const int stages = std::min(8, (budget - fixed * tile) / (dslot + xstep * tile));
            if (stages < 3) continue;
            *p = {x->c, dy->c, x->n, x->h, x->w, dil, wp, rs, (x->w + wp - 1) / wp * x->n * x->h, 1, stages, lag, dslot,
                  march, stages * xstep + fixed};
            // Slices of the rows.  The tensor core truncates: a sum of k
            // steps of 16 pixels ends about 1.5e-8 k below its exact value
            // (measured, positive activations), so few slices cost accuracy
            // and many cost atomics.  About two CTAs per SM for the nine taps
            // of a 128 x 128 (widths that are multiples of 32) or four for
            // those of a 64 x 64 channel block.
            const long long px = (long long)x->n * x->h * x->w;
            long long blocks, splits, least;  // least pixels of a slice
            if (x->w % 32 == 0) {
                blocks = (dy->c + 127) / 128 * (x->c % 128 == 0 ? x->c / 128 : x->c % 64 == 0 ? x->c / 64 : x->c / 32);
                splits = (2LL * num_sms() + 9 * blocks - 1) / (9 * blocks), least = 512;
            } else {
                blocks = (long long)((dy->c + 63) / 64) * ((x->c + 63) / 64);
                splits = (4LL * num_sms() + 9 * blocks - 1) / (9 * blocks), least = 32;
            }
            const long long per = std::max(least, (px + splits - 1) / splits);
            p->slices = (int)std::max(1LL, std::min((long long)p->rows, (px + per - 1) / per));
            return true;
        }
    return false;
}

int launch_wgrad_rows(const unet_act *x, const unet_act *dy, float *dw, float *db, const WgradRows &p,
                      cudaStream_t s) {
    static bool attr[64] = {false};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && !attr[dev]) {
        ST_CUDA(cudaFuncSetAttribute(k_wgrad_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, WR_SMEM_MAX + 2048));
        attr[dev] = true;
    }
    CUtensorMap xm, gm;
    typedef unsigned long long u64;
    const u64 W = p.W, H = p.H, N = p.n, xc = 2ull * x->c_stride, gc = 2ull * dy->c_stride;
    const u64 xd[4] = {(u64)p.cin, W, H, N}, xs[3] = {xc, xc * W, xc * W * H};
    const unsigned xb[4] = {32u, (unsigned)p.wp, (unsigned)p.rs, 1u};
    int rc = make_tensor_map_general(&xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, static_cast<const bf16 *>(x->ptr) + x->c_off,
                                     xd, xs, xb, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
    // dy's channels in blocks of 32: one box holds every block of a step
    const u64 gd[5] = {32, W, (u64)p.cout / 32, H, N}, gs[4] = {gc, 64, gc * W, gc * W * H};
    const unsigned gb[5] = {32u, (unsigned)p.wp, (unsigned)(p.dslot / (p.rs * p.wp * 64)), (unsigned)p.rs, 1u};
    rc = make_tensor_map_general(&gm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, static_cast<const bf16 *>(dy->ptr) + dy->c_off,
                                 gd, gs, gb, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
    const int smem = p.xrows * p.wp * 64 + p.stages * p.dslot + 1024 + (2 * p.stages + 1) * 8 + 16;
    k_wgrad_rows<<<dim3(p.slices, 3 * (p.cin / 32), (p.cout + 127) / 128), 192, smem, s>>>(xm, gm, dw, db, p);
    return cuda_fail(cudaGetLastError(), "wgrad (tcgen05) launch");
}

}  // namespace

extern "C" int unet_wgrad_workspace_bytes(const unet_act *x, const unet_act *dy, size_t *bytes) {
    CHECK_VIEW(x);
    CHECK_VIEW(dy);
    if (!bytes) return fail(STENCIL_EINVAL, "null bytes");
    *bytes = (size_t)(3 * x->c + dy->c) * (size_t)x->n * x->h * x->w * 2;
    return STENCIL_OK;
}

extern "C" int unet_conv3x3_wgrad_engine(const unet_act *x, const unet_act *dy, float *dw, float *db,
                                         int dilation, int engine, void *workspace,
                                         size_t workspace_bytes, stencil_stream_t s) {
    CHECK_VIEW(x);
    CHECK_VIEW(dy);
    if (!dw) return fail(STENCIL_EINVAL, "null dw");
    if (dilation < 1) return fail(STENCIL_EINVAL, "dilation must be >= 1");
    if (engine < 0 || engine > 2) return fail(STENCIL_EINVAL, "engine must be 0, 1 or 2");
    if (x->n != dy->n || x->h != dy->h || x->w != dy->w) return fail(STENCIL_EINVAL, "shape mismatch");
    const size_t need = (size_t)(3 * x->c + dy->c) * (size_t)x->n * x->h * x->w * 2;
    const bool fits = x->w % 32 == 0 && x->c % 32 == 0 && dy->c % 32 == 0 && workspace &&
                      workspace_bytes >= need && (reinterpret_cast<uintptr_t>(workspace) & 255) == 0;
    if (engine == 1 && !fits)
        return fail(STENCIL_EINVAL, "tcgen05 weight gradient needs W %% 32 == 0 and a %zu-byte workspace", need);
    // tcgen05 wherever the channels allow it
    WgradRows p;
    if (engine != 2 && wgrad_rows_plan(x, dy, dilation, &p)) return launch_wgrad_rows(x, dy, dw, db, p, STREAM(s));
    return unet_conv3x3_wgrad_dil(x, dy, dw, db, dilation, s);
}

extern "C" int unet_conv3x3_wgrad_dil(const unet_act *x, const unet_act *dy, float *dw, float *db,
                                      int dilation, stencil_stream_t s) {
    CHECK_VIEW(x);
    CHECK_VIEW(dy);
    if (!dw) return fail(STENCIL_EINVAL, "null dw");
    if (dilation < 1) return fail(STENCIL_EINVAL, "dilation must be >= 1");
    if (x->n != dy->n || x->h != dy->h || x->w != dy->w) return fail(STENCIL_EINVAL, "shape mismatch");
    const long long P = (long long)x->n * x->h * x->w;
    const int mt = (dy->c + 63) / 64, nt = (x->c + 63) / 64;
    // Split the pixels so that about 4 blocks per SM run.
    long long splits = (4LL * num_sms() + 9LL * mt * nt - 1) / (9LL * mt * nt);
    if (splits < 1) splits = 1;
    long long per = (P + splits - 1) / splits;
    per = ((per + WK - 1) / WK) * WK;
    splits = (P + per - 1) / per;
    dim3 grid(mt, nt, (unsigned)(9 * splits));
    k_wgrad<<<grid, 128, 0, STREAM(s)>>>(to_act(*x), to_act(*dy), dw, per, dilation);
    int rc = cuda_fail(cudaGetLastError(), "wgrad launch");
    if (rc || !db) return rc;
    dim3 g2((unsigned)std::min<long long>(1024, (P + 255) / 256), (dy->c + 31) / 32);
    k_bias_grad<<<g2, 256, 0, STREAM(s)>>>(to_act(*dy), db);
    return cuda_fail(cudaGetLastError(), "bias grad launch");
}

extern "C" int unet_conv3x3_wgrad(const unet_act *x, const unet_act *dy, float *dw, float *db,
                                  stencil_stream_t s) {
    return unet_conv3x3_wgrad_dil(x, dy, dw, db, 1, s);
}

extern "C" int unet_relu_bwd(const unet_act *g, const unet_act *y, stencil_stream_t s) {
    CHECK_VIEW(g);
    CHECK_VIEW(y);
    const Act ga = to_act(*g);
    k_relu_bwd<<<grid_for((long long)g->n * g->h * g->w * (g->c / 8)), 256, 0, STREAM(s)>>>(ga, to_act(*y));
    return cuda_fail(cudaGetLastError(), "relu_bwd launch");
}

extern "C" int unet_maxpool2_fwd(const unet_act *x, const unet_act *y, stencil_stream_t s) {
    CHECK_VIEW(x);
    CHECK_VIEW(y);
    if (x->h != 2 * y->h || x->w != 2 * y->w || x->c != y->c) return fail(STENCIL_EINVAL, "pool shapes");
    k_pool_fwd<<<grid_for((long long)y->n * y->h * y->w * (y->c / 8)), 256, 0, STREAM(s)>>>(to_act(*x), to_act(*y));
    return cuda_fail(cudaGetLastError(), "pool launch");
}

extern "C" int unet_maxpool2_bwd(const unet_act *x, const unet_act *y, const unet_act *dy,
                                 const unet_act *dx, stencil_stream_t s) {
    CHECK_VIEW(x);
    CHECK_VIEW(y);
    CHECK_VIEW(dy);
    CHECK_VIEW(dx);
    k_pool_bwd<<<grid_for((long long)y->n * y->h * y->w * (y->c / 8)), 256, 0, STREAM(s)>>>(
        to_act(*x), to_act(*y), to_act(*dy), Act{}, to_act(*dx));
    return cuda_fail(cudaGetLastError(), "pool bwd launch");
}

extern "C" int unet_maxpool2_bwd_skip_relu(const unet_act *x, const unet_act *y, const unet_act *dy,
                                           const unet_act *skip, const unet_act *dx, stencil_stream_t s) {
    const unet_act *v[5] = {x, y, dy, skip, dx};
    for (const unet_act *a : v) {
        int rc = check_act(a, "pool bwd");
        if (rc) return rc;
        const int f = a == y || a == dy ? 2 : 1;
        if (a->n != x->n || a->h * f != x->h || a->w * f != x->w || a->c != x->c)
            return fail(STENCIL_EINVAL, "pool shapes");
    }
    k_pool_bwd<<<grid_for((long long)y->n * y->h * y->w * (y->c / 8)), 256, 0, STREAM(s)>>>(
        to_act(*x), to_act(*y), to_act(*dy), to_act(*skip), to_act(*dx));
    return cuda_fail(cudaGetLastError(), "pool bwd launch");
}

extern "C" int unet_upsample2_fwd(const unet_act *x, const unet_act *y, stencil_stream_t s) {
    CHECK_VIEW(x);
    CHECK_VIEW(y);
    if (y->h != 2 * x->h || y->w != 2 * x->w || x->c != y->c) return fail(STENCIL_EINVAL, "upsample shapes");
    k_up_fwd<<<grid_for((long long)y->n * y->h * y->w * (y->c / 8)), 256, 0, STREAM(s)>>>(to_act(*x), to_act(*y));
    return cuda_fail(cudaGetLastError(), "upsample launch");
}

extern "C" int unet_upsample2_bwd(const unet_act *dy, const unet_act *dx, stencil_stream_t s) {
    CHECK_VIEW(dy);
    CHECK_VIEW(dx);
    k_up_bwd<<<grid_for((long long)dx->n * dx->h * dx->w * (dx->c / 8)), 256, 0, STREAM(s)>>>(to_act(*dy), Act{}, to_act(*dx));
    return cuda_fail(cudaGetLastError(), "upsample bwd launch");
}

extern "C" int unet_upsample2_bwd_relu(const unet_act *dy, const unet_act *gate, const unet_act *dx, stencil_stream_t s) {
    CHECK_VIEW(dy);
    CHECK_VIEW(gate);
    CHECK_VIEW(dx);
    if (dy->n != dx->n || dy->h != 2 * dx->h || dy->w != 2 * dx->w || dy->c != dx->c || gate->n != dx->n ||
        gate->h != dx->h || gate->w != dx->w || gate->c != dx->c)
        return fail(STENCIL_EINVAL, "upsample shapes");
    k_up_bwd<<<grid_for((long long)dx->n * dx->h * dx->w * (dx->c / 8)), 256, 0, STREAM(s)>>>(
        to_act(*dy), to_act(*gate), to_act(*dx));
    return cuda_fail(cudaGetLastError(), "upsample bwd launch");
}

extern "C" int unet_add(const unet_act *a, const unet_act *b, stencil_stream_t s) {
    CHECK_VIEW(a);
    CHECK_VIEW(b);
    k_add<<<grid_for((long long)a->n * a->h * a->w * (a->c / 8)), 256, 0, STREAM(s)>>>(to_act(*a), to_act(*b));
    return cuda_fail(cudaGetLastError(), "add launch");
}

extern "C" int unet_head_fwd(const unet_act *x, const float *w, const float *b, float *y,
                             stencil_stream_t s) {
    CHECK_VIEW(x);
    if (!w || !b || !y) return fail(STENCIL_EINVAL, "null pointer");
    k_head_fwd<<<grid_for((long long)x->n * x->h * x->w), 256, 0, STREAM(s)>>>(to_act(*x), w, b, y);
    return cuda_fail(cudaGetLastError(), "head launch");
}

static int head_bwd(const unet_act *x, const float *w, const float *dy, const unet_act *dx, float *dw, float *db,
                    bool gate, cudaStream_t s) {
    CHECK_VIEW(x);
    CHECK_VIEW(dx);
    if (!w || !dy || !dw || !db || x->c > 256) return fail(STENCIL_EINVAL, "bad head arguments");
    const long long px = (long long)x->n * x->h * x->w, per = 256 / (x->c / 8);
    const int blocks = (int)std::min(8LL * num_sms(), (px + per - 1) / per);
    if (gate) k_head_bwd<true><<<blocks, 256, 0, s>>>(to_act(*x), w, dy, to_act(*dx), dw, db);
    else k_head_bwd<false><<<blocks, 256, 0, s>>>(to_act(*x), w, dy, to_act(*dx), dw, db);
    return cuda_fail(cudaGetLastError(), "head bwd launch");
}

extern "C" int unet_head_bwd(const unet_act *x, const float *w, const float *dy, const unet_act *dx,
                             float *dw, float *db, stencil_stream_t s) {
    return head_bwd(x, w, dy, dx, dw, db, false, STREAM(s));
}

extern "C" int unet_head_bwd_relu(const unet_act *x, const float *w, const float *dy, const unet_act *dx,
                                  float *dw, float *db, stencil_stream_t s) {
    return head_bwd(x, w, dy, dx, dw, db, true, STREAM(s));
}

extern "C" int unet_features(const float *fields, int n, int h, int w, const unet_act *x, float *coons,
                             stencil_stream_t s) {
    CHECK_VIEW(x);
    if (!fields || x->n != n || x->h != h || x->w != w || h < 3 || w < 3)
        return fail(STENCIL_EINVAL, "feature shapes");
    k_features<<<grid_for((long long)n * h * w), 256, 0, STREAM(s)>>>(fields, n, h, w, to_act(*x), coons);
    return cuda_fail(cudaGetLastError(), "features launch");
}

extern "C" int unet_mse(const float *out, const float *coons, const float *target, int n, int h, int w,
                        float scale, float *loss_sum, float *dout, stencil_stream_t s) {
    if (!out || !coons || !target || !loss_sum || !dout) return fail(STENCIL_EINVAL, "null pointer");
    k_mse<<<grid_for((long long)n * h * w), 256, 0, STREAM(s)>>>(out, coons, target, n, h, w, scale, loss_sum, dout);
    return cuda_fail(cudaGetLastError(), "mse launch");
}

extern "C" int unet_adam(float *p, const float *g, float *m, float *v, void *p_bf16, long long count,
                         float lr, float beta1, float beta2, float eps, int step, stencil_stream_t s) {
    if (!p || !g || !m || !v || count < 0 || step < 1) return fail(STENCIL_EINVAL, "bad adam arguments");
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    k_adam<<<grid_for(count), 256, 0, STREAM(s)>>>(p, g, m, v, static_cast<bf16 *>(p_bf16), count, lr, beta1,
                                                    beta2, eps, c1, c2);
    return cuda_fail(cudaGetLastError(), "adam launch");
}

extern "C" int unet_assemble(const float *fields, const float *coons, const float *out, int n, int h, int w,
                             float *u, stencil_stream_t s) {
    if (!fields || !coons || !out || !u) return fail(STENCIL_EINVAL, "null pointer");
    k_assemble<<<grid_for((long long)n * h * w), 256, 0, STREAM(s)>>>(fields, coons, out, n, h, w, u);
    return cuda_fail(cudaGetLastError(), "assemble launch");
}

extern "C" int unet_coons_fill(const float *fields, int n, int h, int w, float *u, stencil_stream_t s) {
    if (!fields || !u || n < 0 || h < 2 || w < 2) return fail(STENCIL_EINVAL, "bad arguments");
    k_coons_fill<<<grid_for((long long)n * h * w), 256, 0, STREAM(s)>>>(fields, n, h, w, u);
    return cuda_fail(cudaGetLastError(), "coons_fill launch");
}

extern "C" int unet_resample_border(const float *fields, int n, int H, int W, int h, int w,
                                    float *coarse, stencil_stream_t s) {
    if (!fields || !coarse || n < 0 || H < 2 || W < 2 || h < 2 || w < 2)
        return fail(STENCIL_EINVAL, "bad arguments");
    k_resample_border<<<grid_for((long long)n * h * w), 256, 0, STREAM(s)>>>(fields, n, H, W, h, w, coarse);
    return cuda_fail(cudaGetLastError(), "resample_border launch");
}

extern "C" int unet_upsample_bilinear(const float *coarse, int n, int h, int w, const float *fields,
                                      int H, int W, float *u, stencil_stream_t s) {
    if (!coarse || !fields || !u || n < 0 || H < 2 || W < 2 || h < 2 || w < 2)
        return fail(STENCIL_EINVAL, "bad arguments");
    k_upsample_bilinear<<<grid_for((long long)n * H * W), 256, 0, STREAM(s)>>>(coarse, n, h, w, fields, H,
                                                                             W, u);
    return cuda_fail(cudaGetLastError(), "upsample_bilinear launch");
}

extern "C" int unet_to_bf16(const float *src, void *dst, long long count, stencil_stream_t s) {
    if (!src || !dst || count < 0) return fail(STENCIL_EINVAL, "bad arguments");
    k_to_bf16<<<grid_for(count), 256, 0, STREAM(s)>>>(src, static_cast<bf16 *>(dst), count);
    return cuda_fail(cudaGetLastError(), "to_bf16 launch");
}
