// BF16 implicit-GEMM 3x3 / 1x1 convolutions on the tcgen05 tensor cores
// (FP32 accumulation in tensor memory), for the warm-start network.
//
// Activations are NHWC bf16; weights [Cout][taps][Cin] bf16.
//
//   conv_halo (3x3 forward and data gradient, narrow layers) and
//   conv_gemm_persistent (every other forward): D[pixel][co] = sum over taps t
//     and input channels ci of A[pixel + off(t)][ci] * B[co][t][ci], taps
//     outermost, so both give the same sums.  Both operands are K-major.  The
//     epilogue adds the bias and an optional skip tensor, applies ReLU, zeroes
//     where a mask tensor is <= 0 (the ReLU derivative of the data gradient)
//     and stores bf16 (and/or fp32).
//   conv_wgrad_kernel (weight and bias gradient): D[ci][co] = sum over pixels
//     p of X[p + off(t)][ci] * G[p][co], all taps in one CTA.  K runs over
//     pixels, so both operands are MN-major (channels contiguous); the pixels
//     are split over CTAs and the FP32 partial sums are added into dW with
//     atomics.
//
// Tiles come in by 4-D TMA boxes whose out-of-image part arrives as zeros
// (the convolution's zero padding).  The swizzle of a staged box is a
// function of the shared-memory address alone, so an operand may start at any
// of its pixels: the nine taps of a tile are nine start addresses into one
// box with a one-pixel border.
//
// Every mbarrier wait is bounded: on a timeout the CTA records an error in
// *status and finishes without hanging.  A role ends at the first of its own
// waits that gives up (the others' waits then run out too), and one that runs on
// a whole warp with all lanes together (warp_wait): its MMAs, commits and
// tensor-memory loads wait for every lane of the warp.
#include "fmvd_internal.h"
#include "smem_opt_in.h"
#include "tma_util.cuh"
#include "umma.cuh"
#include "unet.h"

#include <cuda_bf16.h>
#include <stdio.h>
#include <algorithm>
#include <atomic>

namespace fmvd {
namespace unet {

using bf16 = __nv_bfloat16;
__host__ __device__ constexpr uint32_t align1k(uint32_t b) { return (b + 1023u) & ~1023u; }

__device__ __forceinline__ void tap_offset(int taps, int t, int &dy, int &dx)
{
    if (taps == 9) {
        dy = t / 3 - 1;
        dx = t % 3 - 1;
    } else {
        dy = dx = 0;
    }
}

// Bounded wait of a whole, converged warp: lanes poll for themselves, and one
// that gave up decides for all.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity)
{
    return __all_sync(0xffffffffu, umma::bar_wait(bar, parity));
}

// Sixteen bf16 values as floats (vec: p on a 32-byte boundary).
__device__ __forceinline__ void load16(const bf16 *p, int vec, float (&f)[16])
{
    if (vec) {
        uint32_t w[8];
        umma::ldg32(p, w);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++)
            f[i] = __bfloat162float(p[i]);
    }
}

// Epilogue of sixteen accumulator columns co.. of pixel pix: bias, skip
// tensor, ReLU, mask, stores.  g.vec: every tensor may be accessed 32 bytes
// (whole sectors) at a time.
__device__ __forceinline__ void epilogue16(const GemmArgs &g, size_t pix, int co, float (&v)[16])
{
    float t[16];
    if (g.bias) {
        if (g.vec) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                *reinterpret_cast<float4 *>(t + 4 * i) = __ldg(reinterpret_cast<const float4 *>(g.bias + co) + i);
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++)
                t[i] = g.bias[co + i];
        }
#pragma unroll
        for (int i = 0; i < 16; i++)
            v[i] += t[i];
    }
    if (g.add) {
        load16(g.add + pix * g.add_ld + co, g.vec, t);
#pragma unroll
        for (int i = 0; i < 16; i++)
            v[i] += t[i];
    }
    if (g.relu) {
#pragma unroll
        for (int i = 0; i < 16; i++)
            v[i] = fmaxf(v[i], 0.f);
    }
    if (g.mask) {
        load16(g.mask + pix * g.mask_ld + co, g.vec, t);
#pragma unroll
        for (int i = 0; i < 16; i++)
            v[i] = t[i] > 0.f ? v[i] : 0.f;
    }
    if (g.out) {
        uint32_t h[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            h[i] = *reinterpret_cast<const uint32_t *>(&b);
        }
        bf16 *dst = g.out + pix * g.out_ld + g.out_coff + co;
        if (g.vec) {
            umma::stg32(dst, h);
        } else {
            reinterpret_cast<uint4 *>(dst)[0] = make_uint4(h[0], h[1], h[2], h[3]);
            reinterpret_cast<uint4 *>(dst)[1] = make_uint4(h[4], h[5], h[6], h[7]);
        }
    }
    if (g.out_f32) {
        float4 *dst = reinterpret_cast<float4 *>(g.out_f32 + pix * g.outf_ld + co);
#pragma unroll
        for (int i = 0; i < 4; i++)
            dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
}

// Persistent forward / data-gradient GEMM.  Each CTA
// walks tiles blockIdx.x, blockIdx.x + gridDim.x, ... of the 128-pixel x BN
// output; the K blocks of consecutive tiles flow through one TMA stage ring
// without a break, and the accumulator is double-buffered in tensor memory,
// so the epilogue of a tile overlaps the MMAs of the next.  Warps 0-3: the
// epilogue (warp w reads accumulator lanes 32w..32w+31); warp 4: tensor
// memory allocation and, in lane 0, the TMA producer; warp 5 lane 0: the MMA
// issuer.
constexpr int kPersistentThreads = 192;

template <int CB, int BN>
struct PersistCfg {
    static constexpr int R = CB * 2;
    static constexpr uint32_t SA = 128u * R, SB = (uint32_t)BN * R;
    static constexpr uint32_t STAGE = align1k(SA) + align1k(SB);
    static constexpr int ACC_COLS = BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
    static constexpr int TCOLS = 2 * ACC_COLS;  // two accumulators
    // one CTA per SM when its accumulators take all of tensor memory: then
    // the stage ring may use most of shared memory
    static constexpr uint32_t BUDGET = TCOLS == 512 ? 196608u : 98304u;
    static constexpr int STAGES = BUDGET / STAGE >= 6 ? 6 : (BUDGET / STAGE >= 2 ? (int)(BUDGET / STAGE) : 2);
    static constexpr uint32_t SMEM = STAGES * STAGE + 1024;
    static constexpr int KSTEPS = CB / 16;
};

template <int CB, int BN>
__global__ void __launch_bounds__(kPersistentThreads, 1)
    conv_gemm_persistent(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const GemmArgs g, int ntiles, int ntiles_n)
{
    using C = PersistCfg<CB, BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[C::STAGES], empty[C::STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_sh;
    __shared__ int fail_store;
    volatile int &fail_sh = fail_store;  // set by any role that gave up waiting
    const int warp = umma::warp_index(), lane = threadIdx.x & 31;
    const int tx = g.W / g.bw, ty = g.H / g.bh;
    const int nk = g.taps * (g.cin / CB);
    const int cblocks = g.cin / CB;

    if (threadIdx.x == 0) {
        for (int i = 0; i < C::STAGES; i++) {
            umma::bar_init(&full[i], 1);
            umma::bar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            umma::bar_init(&acc_full[i], 1);
            umma::bar_init(&acc_empty[i], 4);  // one arrival per epilogue warp
        }
        umma::bar_fence_init();
        fail_sh = 0;
    }
    if (warp == 4) {
        umma::tmem_alloc(&tmem_sh, C::TCOLS);
        umma::tmem_relinquish();
    }
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tmem_sh;

    auto tile_coords = [&](int tile, int &n, int &y0, int &x0, int &co0) {
        const int tp = tile / ntiles_n, tn = tile % ntiles_n;
        n = tp / (tx * ty);
        const int r = tp % (tx * ty);
        y0 = (r / tx) * g.bh;
        x0 = (r % tx) * g.bw;
        co0 = tn * BN;
    };

    if (warp == 4) {
        if (lane == 0) {
            // ---- producer
            int gk = 0;
            for (int tile = blockIdx.x; tile < ntiles && !fail_sh; tile += gridDim.x) {
                int n, y0, x0, co0;
                tile_coords(tile, n, y0, x0, co0);
                for (int kb = 0; kb < nk; kb++, gk++) {
                    const int s = gk % C::STAGES, round = gk / C::STAGES;
                    if (round > 0 && !umma::bar_wait(&empty[s], (round - 1) & 1)) {
                        fail_sh = 1;
                        break;
                    }
                    umma::bar_expect_tx(&full[s], C::SA + C::SB);
                    uint8_t *a = smem + s * C::STAGE;
                    uint8_t *b = a + align1k(C::SA);
                    const int t = kb / cblocks, cb = kb % cblocks;
                    int dy, dx;
                    tap_offset(g.taps, t, dy, dx);
                    umma::tma_load_4d(a, &tmA, cb * CB, x0 + dx, y0 + dy, n, &full[s]);
                    umma::tma_load_2d(b, &tmB, kb * CB, co0, &full[s]);
                }
            }
        }
    } else if (warp == 5) {
        // ---- MMA issue
        const uint32_t idesc = umma::make_idesc(128, BN, 0, 0);
        int gk = 0, it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, it++) {
            const int ab = it & 1;
            ok = it < 2 || warp_wait(&acc_empty[ab], ((it >> 1) - 1) & 1);
            if (!ok)
                break;
            umma::tc_fence_after();
            const uint32_t acc = tmem + ab * C::ACC_COLS;
            for (int kb = 0; kb < nk; kb++, gk++) {
                const int s = gk % C::STAGES, round = gk / C::STAGES;
                ok = warp_wait(&full[s], round & 1);
                if (!ok)
                    break;
                umma::tc_fence_after();
                const uint32_t a0 = umma::smem_addr(smem) + s * C::STAGE;
                const umma::Desc ad = umma::make_desc(a0, 16, 8 * C::R, C::R);
                const umma::Desc bd = umma::make_desc(a0 + align1k(C::SA), 16, 8 * C::R, C::R);
#pragma unroll
                for (int kk = 0; kk < C::KSTEPS; kk++)
                    umma::mma_bf16(acc, ad + kk * 32, bd + kk * 32, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
                umma::mma_commit(&empty[s]);
            }
            umma::mma_commit(&acc_full[ab]);
        }
        if (!ok)
            fail_sh = 1;
    } else {
        // ---- epilogue: warp w owns accumulator rows 32w..32w+31
        const int row = warp * 32 + lane;
        int it = 0;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
            const int ab = it & 1;
            if (!warp_wait(&acc_full[ab], (it >> 1) & 1)) {
                fail_sh = 1;
                break;
            }
            umma::tc_fence_after();
            int n, y0, x0, co0;
            tile_coords(tile, n, y0, x0, co0);
            const int y = y0 + row / g.bw, x = x0 + row % g.bw;
            const size_t pix = ((size_t)n * g.H + y) * g.W + x;
            const uint32_t trow = tmem + ab * C::ACC_COLS + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 16) {
                float v[16];
                umma::tmem_ld16(trow + c0, v);
                epilogue16(g, pix, co0 + c0, v);
            }
            umma::tc_fence_before();
            __syncwarp();
            if (lane == 0)
                umma::bar_arrive(&acc_empty[ab]);
        }
    }
    __syncwarp();
    umma::tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && fail_sh && g.status)
        atomicExch(g.status, 1);
    if (warp == 4) {
        umma::tc_fence_after();
        umma::tmem_dealloc(tmem, C::TCOLS);
    }
}

// 3x3 forward / data-gradient GEMM of the narrow layers (cin = CB * NB up to
// 128, cout = BN up to 128 with the weights within shared memory).  A tile is
// 8 x 16 pixels; its input comes in once, with a one-pixel border (10 x 18
// pixels per channel block), and the nine taps read it at nine start
// addresses: 128 output pixels load 180 pixels instead of 9 x 128, and the
// weights are loaded once per CTA.  An 8-row group of the A operand is one
// row of the tile, so the group stride is the border box's row pitch.  Roles
// as in conv_gemm_persistent.
// Four 512 x 512 planes: 32 -> 32 channels 39 us (one CTA per tile and every
// tap loaded on its own: 91 us), 64 -> 32 77 us; 64 -> 64 at 256 x 256 33 us
// (45 us).  What bounds it: loads, stores and their latencies (with one tap
// instead of nine the network's forward pass is 6 % faster, without the stores
// 14 %).
constexpr int kTileW = 8, kTileH = 16, kBoxW = kTileW + 2, kBoxH = kTileH + 2;
constexpr uint32_t kSmemOne = 226u * 1024u, kSmemTwo = 113u * 1024u;  // per CTA, one or two CTAs on an SM

template <int CB, int NB, int BN>
struct HaloCfg {
    static constexpr uint32_t R = CB * 2;
    static constexpr uint32_t BOX = kBoxW * kBoxH * R, SLOT = align1k(BOX);
    static constexpr uint32_t WB = align1k((uint32_t)BN * R), WEIGHTS = 9u * NB * WB;
    static constexpr uint32_t BUDGET = (WEIGHTS + (NB + 1) * SLOT + 1024u <= kSmemTwo ? kSmemTwo : kSmemOne) - 1024u;
    static constexpr int FIT = (int)((BUDGET - WEIGHTS) / SLOT);
    static constexpr int SLOTS = FIT < 2 * NB + 2 ? FIT : 2 * NB + 2;
    static constexpr uint32_t SMEM = WEIGHTS + SLOTS * SLOT + 1024;
    static constexpr int ACC_COLS = BN <= 32 ? 32 : (BN <= 64 ? 64 : 128);
    static constexpr int TCOLS = 2 * ACC_COLS;
    static_assert(SLOTS >= NB + 1, "a tile's channel blocks and the next one's first are in flight");
};

template <int CB, int NB, int BN>
__global__ void __launch_bounds__(kPersistentThreads, 1)
    conv_halo(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g,
              int ntiles)
{
    using C = HaloCfg<CB, NB, BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *wsm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *slots = wsm + C::WEIGHTS;
    __shared__ __align__(8) uint64_t wfull, full[C::SLOTS], empty[C::SLOTS], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_sh;
    __shared__ int fail_store;
    volatile int &fail_sh = fail_store;  // set by any role that gave up waiting
    const int warp = umma::warp_index(), lane = threadIdx.x & 31;
    const int tx = g.W / kTileW, ty = (g.H + kTileH - 1) / kTileH;

    if (threadIdx.x == 0) {
        umma::bar_init(&wfull, 1);
        for (int i = 0; i < C::SLOTS; i++) {
            umma::bar_init(&full[i], 1);
            umma::bar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            umma::bar_init(&acc_full[i], 1);
            umma::bar_init(&acc_empty[i], 4);  // one arrival per epilogue warp
        }
        umma::bar_fence_init();
        fail_sh = 0;
    }
    if (warp == 4) {
        umma::tmem_alloc(&tmem_sh, C::TCOLS);
        umma::tmem_relinquish();
    }
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tmem_sh;

    auto tile_coords = [&](int tile, int &n, int &y0, int &x0) {
        n = tile / (tx * ty);
        const int r = tile % (tx * ty);
        y0 = (r / tx) * kTileH;
        x0 = (r % tx) * kTileW;
    };

    if (warp == 4) {
        if (lane == 0) {
            // ---- producer: the weights once, then the tiles' input boxes
            umma::bar_expect_tx(&wfull, 9u * NB * BN * C::R);
            for (int k = 0; k < 9 * NB; k++)
                umma::tma_load_2d(wsm + k * C::WB, &tmB, k * CB, 0, &wfull);
            int gs = 0;
            for (int tile = blockIdx.x; tile < ntiles && !fail_sh; tile += gridDim.x) {
                int n, y0, x0;
                tile_coords(tile, n, y0, x0);
                for (int cb = 0; cb < NB; cb++, gs++) {
                    const int s = gs % C::SLOTS, round = gs / C::SLOTS;
                    if (round > 0 && !umma::bar_wait(&empty[s], (round - 1) & 1)) {
                        fail_sh = 1;
                        break;
                    }
                    umma::bar_expect_tx(&full[s], C::BOX);
                    umma::tma_load_4d(slots + s * C::SLOT, &tmA, cb * CB, x0 - 1, y0 - 1, n, &full[s]);
                }
            }
        }
    } else if (warp == 5) {
        // ---- MMA issue
        const uint32_t idesc = umma::make_idesc(128, BN, 0, 0);
        const umma::Desc bd = umma::make_desc(umma::smem_addr(wsm), 16, 8 * C::R, C::R);
        bool ok = warp_wait(&wfull, 0);
        int gs = 0, it = 0;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, it++, gs += NB) {
            const int ab = it & 1;
            ok = it < 2 || warp_wait(&acc_empty[ab], ((it >> 1) - 1) & 1);
            const uint32_t acc = tmem + ab * C::ACC_COLS;
            umma::Desc ad[NB];
#pragma unroll
            for (int cb = 0; cb < NB; cb++) {
                const int s = (gs + cb) % C::SLOTS, round = (gs + cb) / C::SLOTS;
                ok = ok && warp_wait(&full[s], round & 1);
                ad[cb] = umma::make_desc(umma::smem_addr(slots) + s * C::SLOT, 16, kBoxW * C::R, C::R);
            }
            if (!ok)
                break;
            umma::tc_fence_after();
#pragma unroll
            for (int t = 0; t < 9; t++)
#pragma unroll
                for (int cb = 0; cb < NB; cb++)
#pragma unroll
                    for (int kk = 0; kk < CB / 16; kk++)
                        umma::mma_bf16(acc, ad[cb] + (((t / 3) * kBoxW + t % 3) * C::R + kk * 32),
                                       bd + ((t * NB + cb) * C::WB + kk * 32), idesc,
                                       (t > 0 || cb > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
            for (int cb = 0; cb < NB; cb++)
                umma::mma_commit(&empty[(gs + cb) % C::SLOTS]);
            umma::mma_commit(&acc_full[ab]);
        }
        if (!ok)
            fail_sh = 1;
    } else {
        // ---- epilogue: warp w owns accumulator rows 32w..32w+31
        const int row = warp * 32 + lane;
        int it = 0;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
            const int ab = it & 1;
            if (!warp_wait(&acc_full[ab], (it >> 1) & 1)) {
                fail_sh = 1;
                break;
            }
            umma::tc_fence_after();
            int n, y0, x0;
            tile_coords(tile, n, y0, x0);
            const int y = y0 + row / kTileW, x = x0 + row % kTileW;
            const size_t pix = ((size_t)n * g.H + y) * g.W + x;
            const uint32_t trow = tmem + ab * C::ACC_COLS + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 16) {
                float v[16];
                umma::tmem_ld16(trow + c0, v);
                if (y < g.H)
                    epilogue16(g, pix, c0, v);
                __syncwarp();  // rows past the image skip the stores
            }
            umma::tc_fence_before();
            __syncwarp();
            if (lane == 0)
                umma::bar_arrive(&acc_empty[ab]);
        }
    }
    __syncwarp();
    umma::tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && fail_sh && g.status)
        atomicExch(g.status, 1);
    if (warp == 4) {
        umma::tc_fence_after();
        umma::tmem_dealloc(tmem, C::TCOLS);
    }
}

// Weight and bias gradient: D[ci][co] = sum over pixels p of
// X[p + off(t)][ci] G[p][co] for every tap t of a 128 x BN tile of (ci, co),
// over this CTA's share of the pixels.  A tile is 16 x 8 pixels; X comes in
// with a one-pixel border (18 x 10) and the taps are start addresses into it,
// so X and G are loaded once instead of once per tap.  M = 128 rows are
//   cin >= 128: 128 channels (two 64-channel groups), one tap per MMA;
//   cin = 64:   64 channels at two neighbouring pixels (PACK = 2), the taps
//               dx = -1, 0 of a row in one MMA and dx = 1 in a second;
//   cin = 32:   32 channels at four neighbouring pixels (PACK = 4), the three
//               taps of a row in one MMA.
// The neighbouring pixel is one row of the staged box further: the M-group
// stride of the operand's descriptor.  Rows beyond dx = 1 are not read back.
// Warp 0 issues the TMA ring, warp 1 the MMAs; warps 2 and 3 sum the staged G
// for the bias gradient; at the end all four read tensor memory and add the
// sums with atomics, consecutive lanes consecutive ci.
// The tensor cores' FP32 accumulation rounds towards zero: a sum of n pixels
// comes out about 1.2e-9 n too small.  A CTA's share (launch_wgrad) grows with
// the batch: 31.9 k pixels, 3.7e-5, at 16 planes of 512 x 512, four times that
// at 64.  The bias
// sums, which cancel more, are ordinary FP32 additions (as an MMA with a
// matrix of ones they were 4.7e-5 off).
// Four 512 x 512 planes: 32 -> 32 channels 69 us (280 us with one tap per CTA),
// 64 -> 32 112 us (288); 64 -> 64 at 256 x 256 41 us (106); 128 -> 128 at 128 x
// 128 53 us (98); the bias sums are part of it (they were passes of their own
// over G).  What bounds it: the MMAs (about 90 cycles each, few CTAs).
constexpr int kGradW = 16, kGradH = 8;

template <int CB, int GROUPS, int PACK, int BN, int TAPS>
struct WgradCfg {
    static constexpr int NACC = TAPS == 1 ? 1 : PACK == 4 ? 3 : PACK == 2 ? 6 : 9;
    static constexpr int XW = TAPS == 1 ? kGradW : kGradW + 2, XH = TAPS == 1 ? kGradH : kGradH + 2;
    static constexpr uint32_t R = CB * 2, XBOX = XW * XH * R, XS = align1k(XBOX);
    static constexpr int CBG = BN >= 64 ? 64 : 32, NG = BN / CBG;
    static constexpr uint32_t RG = CBG * 2, GBOX = kGradW * kGradH * RG;
    static constexpr uint32_t STAGE = GROUPS * XS + NG * GBOX;
    static constexpr int COLS = NACC * BN;
    static constexpr int TCOLS = COLS <= 64 ? 64 : COLS <= 128 ? 128 : COLS <= 256 ? 256 : 512;
    static constexpr bool TWO = TCOLS <= 256 && 3 * STAGE + 1024 <= kSmemTwo;
    static constexpr uint32_t BUDGET = (TWO ? kSmemTwo : kSmemOne) - 1024;
    static constexpr int STAGES = BUDGET / STAGE >= 4 ? 4 : (int)(BUDGET / STAGE);
    static constexpr uint32_t SMEM = STAGES * STAGE + 1024;
    static constexpr int PER_SM = TWO ? 2 : 1;
    static_assert(CB * GROUPS * PACK == 128 && STAGES >= 2 && COLS <= 512, "tile");
    // the last PACK - 1 pixels of the last K step lie past the box
    static_assert(TAPS == 1 || PACK == 1 || XS >= XBOX + R, "reads past the box stay in its stage");
};

// first tap offset of accumulator a
template <int PACK, int TAPS>
__host__ __device__ constexpr int acc_dy(int a) { return TAPS == 1 ? 0 : PACK == 4 ? a - 1 : PACK == 2 ? a / 2 - 1 : a / 3 - 1; }
template <int PACK, int TAPS>
__host__ __device__ constexpr int acc_dx(int a) { return TAPS == 1 ? 0 : PACK == 4 ? -1 : PACK == 2 ? (a & 1 ? 1 : -1) : a % 3 - 1; }

template <int CB, int GROUPS, int PACK, int BN, int TAPS>
__global__ void __launch_bounds__(128, 1)
    conv_wgrad_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmG,
                      const GemmArgs g, int ntiles, int chunk)
{
    using C = WgradCfg<CB, GROUPS, PACK, BN, TAPS>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *stages = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[C::STAGES], empty[C::STAGES], done;
    __shared__ uint32_t tmem_sh;
    __shared__ int fail_sh;
    const int warp = umma::warp_index(), lane = threadIdx.x & 31;
    const int co0 = blockIdx.y * BN, ci0 = blockIdx.z * CB * GROUPS;
    const int k0 = blockIdx.x * chunk, nk = min(chunk, ntiles - k0);
    const bool bias = g.db && blockIdx.z == 0;
    const int tx = (g.W + kGradW - 1) / kGradW, ty = (g.H + kGradH - 1) / kGradH;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; s++) {
            umma::bar_init(&full[s], 1);
            umma::bar_init(&empty[s], bias ? 3 : 1);  // the MMAs, and the two warps that sum G
        }
        umma::bar_init(&done, 1);
        umma::bar_fence_init();
        fail_sh = 0;
    }
    if (warp == 0) {
        umma::tmem_alloc(&tmem_sh, C::TCOLS);
        umma::tmem_relinquish();
    }
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tmem_sh;

    if (warp == 0 && lane == 0) {
        for (int k = 0; k < nk; k++) {
            const int s = k % C::STAGES, round = k / C::STAGES;
            if (round > 0 && !umma::bar_wait(&empty[s], (round - 1) & 1)) {
                fail_sh = 1;
                break;
            }
            const int tile = k0 + k, n = tile / (tx * ty), r = tile % (tx * ty);
            const int y0 = (r / tx) * kGradH, x0 = (r % tx) * kGradW;
            constexpr int halo = TAPS == 1 ? 0 : 1;
            umma::bar_expect_tx(&full[s], GROUPS * C::XBOX + C::NG * C::GBOX);
            uint8_t *st = stages + s * C::STAGE;
#pragma unroll
            for (int j = 0; j < GROUPS; j++)
                umma::tma_load_4d(st + j * C::XS, &tmX, ci0 + j * CB, x0 - halo, y0 - halo, n, &full[s]);
#pragma unroll
            for (int j = 0; j < C::NG; j++)
                umma::tma_load_4d(st + GROUPS * C::XS + j * C::GBOX, &tmG, co0 + j * C::CBG, x0, y0, n, &full[s]);
        }
    } else if (warp == 1) {
        const uint32_t idesc = umma::make_idesc(128, BN, 1, 1);
        for (int k = 0; k < nk; k++) {
            const int s = k % C::STAGES, round = k / C::STAGES;
            if (!warp_wait(&full[s], round & 1)) {
                fail_sh = 1;
                break;
            }
            umma::tc_fence_after();
            const uint32_t x0 = umma::smem_addr(stages) + s * C::STAGE;
            umma::Desc xd = umma::make_desc(x0, PACK > 1 ? C::R : C::XS, 8 * C::R, C::R);
            umma::Desc gd = umma::make_desc(x0 + GROUPS * C::XS, C::GBOX, 8 * C::RG, C::RG);
#pragma unroll 1
            for (int r = 0; r < kGradH; r++) {
#pragma unroll
                for (int a = 0; a < C::NACC; a++) {
                    constexpr int o = TAPS == 1 ? 0 : 1;
                    const int at = (acc_dy<PACK, TAPS>(a) + o) * C::XW + acc_dx<PACK, TAPS>(a) + o;
                    umma::mma_bf16(tmem + a * BN, xd + at * C::R, gd, idesc, (k > 0 || r > 0) ? 1u : 0u);
                }
                xd = xd + C::XW * C::R;
                gd = gd + kGradW * C::RG;
            }
            umma::mma_commit(&empty[s]);
        }
        umma::mma_commit(&done);
    } else if (warp >= 2 && bias) {
        // thread: eight channels (chunk cc) of pixels p0, p0 + step, ...
        constexpr int CH = BN / 8, step = 64 / CH;
        const int cc = lane % CH, c = cc % (C::CBG / 8), p0 = (threadIdx.x - 64) / CH;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < nk; k++) {
            const int s = k % C::STAGES, round = k / C::STAGES;
            if (!warp_wait(&full[s], round & 1)) {
                fail_sh = 1;
                break;
            }
            const uint8_t *gs = stages + s * C::STAGE + GROUPS * C::XS + (cc * 8 / C::CBG) * C::GBOX;
#pragma unroll 4
            for (int p = p0; p < kGradW * kGradH; p += step) {
                // the 16-byte units of a staged pixel are swizzled by its address
                const int u = c ^ (C::RG == 128 ? p & 7 : (p >> 1) & 3);
                const uint4 q = *reinterpret_cast<const uint4 *>(gs + p * C::RG + 16 * u);
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    acc[2 * i] += __uint_as_float(w[i] << 16);
                    acc[2 * i + 1] += __uint_as_float(w[i] & 0xFFFF0000u);
                }
            }
            __syncwarp();
            if (lane == 0)
                umma::bar_arrive(&empty[s]);
        }
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 8; e++) {
            for (int o = CH; o < 32; o <<= 1)
                acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
            if (lane < CH)
                atomicAdd(g.db + co0 + 8 * cc + e, acc[e]);
        }
    }
    __syncwarp();

    // accumulator rows are TMEM lanes (warp w: lanes 32w..)
    if (!warp_wait(&done, 0))
        fail_sh = 1;
    umma::tc_fence_after();
    const int row = warp * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    const int j = PACK > 1 ? row / CB : 0, ci = ci0 + (PACK > 1 ? row % CB : row);
#pragma unroll 1
    for (int a = 0; a < C::NACC; a++) {
        const int dx = acc_dx<PACK, TAPS>(a) + j, tap = TAPS == 1 ? 0 : (acc_dy<PACK, TAPS>(a) + 1) * 3 + dx + 1;
        if (dx > (TAPS == 1 ? 0 : 1))  // the same for a whole warp
            continue;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            float v[16];
            umma::tmem_ld16(trow + a * BN + c0, v);
            float *dst = g.dw + ((size_t)(co0 + c0) * TAPS + tap) * g.cin + ci;
#pragma unroll
            for (int i = 0; i < 16; i++)
                atomicAdd(dst + (size_t)i * TAPS * g.cin, v[i]);
        }
    }
    umma::tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && fail_sh && g.status)
        atomicExch(g.status, 1);
    if (warp == 0)
        umma::tmem_dealloc(tmem, C::TCOLS);
}

// ------------------------------------------------------------------ host
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encoder()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

CUtensorMapSwizzle swizzle_for(int cb) { return cb == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B; }

// NHWC activation tensor as a 4-D map {C, W, H, N}, box {cb, bw, bh, 1}.
bool map_nhwc(CUtensorMap *m, const void *base, int C, int W, int H, int N, int cb, int bw, int bh)
{
    cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
    cuuint32_t box[4] = {(cuuint32_t)cb, (cuuint32_t)bw, (cuuint32_t)bh, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(cb), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Row-major [rows][cols] bf16 matrix as a 2-D map, box {cb, brows}.
bool map_matrix(CUtensorMap *m, const void *base, int cols, int rows, int cb, int brows)
{
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)cb, (cuuint32_t)brows};
    cuuint32_t es[2] = {1, 1};
    return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(cb), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// pixel box of 'count' pixels on a W-wide image
void pixel_box(int W, int count, int &bw, int &bh)
{
    bw = W < count ? W : count;
    bh = count / bw;
}

// Opts a kernel in to its dynamic shared memory on the current device and reads
// the device's multiprocessor count.
template <typename K>
bool configure(K kern, uint32_t smem, std::atomic<unsigned long long> &devices, int &sms)
{
    int dev = 0;
    return FMVD_CHECK(cudaGetDevice(&dev)) &&
           FMVD_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) &&
           FMVD_CHECK(allow_smem(kern, smem, devices));
}

template <int CB, int BN>
bool launch_persistent(const CUtensorMap &ta, const CUtensorMap &tb, const GemmArgs &g, int ntiles, int ntiles_n,
                       cudaStream_t s)
{
    using C = PersistCfg<CB, BN>;
    auto k = conv_gemm_persistent<CB, BN>;
    static std::atomic<unsigned long long> devices{0};
    int sms = 0;
    if (!configure(k, C::SMEM, devices, sms))
        return false;
    // CTAs per SM: tensor memory (512 columns) and shared memory allow
    const int by_tmem = 512 / C::TCOLS;
    const int by_smem = (int)(200u * 1024u / C::SMEM);
    const int per_sm = by_tmem < by_smem ? by_tmem : by_smem;
    int grid = sms * (per_sm < 1 ? 1 : per_sm);
    if (grid > ntiles)
        grid = ntiles;
    k<<<grid, kPersistentThreads, C::SMEM, s>>>(ta, tb, g, ntiles, ntiles_n);
    rl_count_launch(1);
    return FMVD_CHECK(cudaGetLastError());
}

#define FMVD_BN_CASES(F) F(16) F(32) F(64) F(128) F(256)

template <int CB>
bool dispatch_persistent(int bn, const CUtensorMap &ta, const CUtensorMap &tb, const GemmArgs &g, int ntiles,
                         int ntiles_n, cudaStream_t s)
{
    switch (bn) {
#define X(B) \
    case B: return launch_persistent<CB, B>(ta, tb, g, ntiles, ntiles_n, s);
        FMVD_BN_CASES(X)
#undef X
    default: report_error("fmvd: unsupported GEMM N tile"); return false;
    }
}

bool aligned32(const void *p) { return reinterpret_cast<uintptr_t>(p) % 32 == 0; }

template <int CB, int NB, int BN>
bool launch_halo(const CUtensorMap &ta, const CUtensorMap &tb, const GemmArgs &g, cudaStream_t s)
{
    using C = HaloCfg<CB, NB, BN>;
    auto k = conv_halo<CB, NB, BN>;
    static std::atomic<unsigned long long> devices{0};
    int sms = 0;
    if (!configure(k, C::SMEM, devices, sms))
        return false;
    const int ntiles = g.N * ((g.H + kTileH - 1) / kTileH) * (g.W / kTileW);
    // CTAs per SM: tensor memory (512 columns), shared memory (228 KB, 1 KB of
    // it per CTA reserved), registers
    int per_sm = (int)(228u * 1024u / (C::SMEM + 1024u));
    per_sm = std::max(1, std::min(per_sm, std::min(512 / C::TCOLS, 3)));
    k<<<std::min(ntiles, sms * per_sm), kPersistentThreads, C::SMEM, s>>>(ta, tb, g, ntiles);
    rl_count_launch(1);
    return FMVD_CHECK(cudaGetLastError());
}

// The halo kernel for this layer, or null where its weights do not fit.
using HaloLaunch = bool (*)(const CUtensorMap &, const CUtensorMap &, const GemmArgs &, cudaStream_t);
HaloLaunch halo_for(int cin, int cout)
{
    switch (cin * 1024 + cout) {
#define X(CI, CB, NB, BN) \
    case CI * 1024 + BN: return launch_halo<CB, NB, BN>;
        X(32, 32, 1, 16) X(32, 32, 1, 32) X(32, 32, 1, 64) X(32, 32, 1, 128)
        X(64, 64, 1, 16) X(64, 64, 1, 32) X(64, 64, 1, 64) X(64, 64, 1, 128)
        X(128, 64, 2, 32) X(128, 64, 2, 64)
#undef X
    default: return nullptr;
    }
}

template <int CB, int GROUPS, int PACK, int BN, int TAPS>
bool launch_wgrad(const CUtensorMap &tx, const CUtensorMap &tg, const GemmArgs &g, cudaStream_t s)
{
    using C = WgradCfg<CB, GROUPS, PACK, BN, TAPS>;
    auto k = conv_wgrad_kernel<CB, GROUPS, PACK, BN, TAPS>;
    static std::atomic<unsigned long long> devices{0};
    int sms = 0;
    if (!configure(k, C::SMEM, devices, sms))
        return false;
    const int ntiles = g.N * ((g.H + kGradH - 1) / kGradH) * ((g.W + kGradW - 1) / kGradW);
    // pixels per CTA: at least 8 tiles, and for larger batches so many that the
    // grid covers the GPU a few times over
    const long long parts = (long long)g.taps * ((g.cout + 127) / 128) * ((g.cin + 255) / 256);
    const int chunk = (int)std::min<long long>(ntiles, std::max<long long>(8, (ntiles * parts + 1183) / 1184));
    const dim3 grid((ntiles + chunk - 1) / chunk, g.cout / BN, g.cin / (CB * GROUPS));
    k<<<grid, 128, C::SMEM, s>>>(tx, tg, g, ntiles, chunk);
    rl_count_launch(1);
    return FMVD_CHECK(cudaGetLastError());
}

template <int CB, int GROUPS, int PACK, int BN>
bool wgrad_taps(const CUtensorMap &tx, const CUtensorMap &tg, const GemmArgs &g, cudaStream_t s)
{
    return g.taps == 9 ? launch_wgrad<CB, GROUPS, PACK, BN, 9>(tx, tg, g, s)
                       : launch_wgrad<CB, GROUPS, PACK, BN, 1>(tx, tg, g, s);
}

} // namespace

bool conv_forward(const ConvDesc &c, cudaStream_t s)
{
    // D[pixel][co]: A = input activations (cin channels), B = weights [cout][taps][cin]
    if (!encoder()) {
        report_error("fmvd: cuTensorMapEncodeTiled is unavailable");
        return false;
    }
    const int cb = c.cin >= 64 ? 64 : 32;
    const int bn = c.cout > 256 ? 256 : c.cout;
    if (c.cin % cb || c.cout % bn || bn % 16 || (c.taps != 1 && c.taps != 9) || c.W % 8 || c.H * c.W < 128 ||
        (c.W < 128 ? 128 % c.W : c.W % 128) || (c.W < 128 && c.H % (128 / c.W))) {
        report_error("fmvd: unsupported convolution geometry");
        return false;
    }
    int bw, bh;
    pixel_box(c.W, 128, bw, bh);
    const HaloLaunch halo = c.taps == 9 ? halo_for(c.cin, c.cout) : nullptr;
    CUtensorMap ta, tb;
    if (!map_nhwc(&ta, c.in, c.cin, c.W, c.H, c.N, cb, halo ? kBoxW : bw, halo ? kBoxH : bh) ||
        !map_matrix(&tb, c.weight, c.taps * c.cin, c.cout, cb, bn)) {
        report_error("fmvd: tensor map encoding failed");
        return false;
    }
    GemmArgs g{};
    g.N = c.N;
    g.H = c.H;
    g.W = c.W;
    g.bw = bw;
    g.bh = bh;
    g.taps = c.taps;
    g.cin = c.cin;
    g.cout = c.cout;
    g.out = c.out;
    g.out_ld = c.out_ld ? c.out_ld : c.cout;
    g.out_coff = c.out_coff;
    g.out_f32 = c.out_f32;
    g.outf_ld = c.outf_ld ? c.outf_ld : c.cout;
    g.bias = c.bias;
    g.add = c.add;
    g.add_ld = c.add_ld ? c.add_ld : c.cout;
    g.mask = c.mask;
    g.mask_ld = c.mask_ld ? c.mask_ld : c.cout;
    g.relu = c.relu;
    g.status = c.status;
    // 32-byte accesses in the epilogue where sixteen channels of every tensor
    // start on a 32-byte boundary (the channel counts are multiples of 16)
    g.vec = aligned32(c.bias) && aligned32(c.add) && aligned32(c.mask) && aligned32(c.out) &&
            (g.add_ld | g.mask_ld | g.out_ld | g.out_coff) % 16 == 0;
    if (halo)
        return halo(ta, tb, g, s);
    const int ntiles_n = c.cout / bn;
    const int ntiles = c.N * (c.H / bh) * (c.W / bw) * ntiles_n;
    return cb == 64 ? dispatch_persistent<64>(bn, ta, tb, g, ntiles, ntiles_n, s)
                    : dispatch_persistent<32>(bn, ta, tb, g, ntiles, ntiles_n, s);
}

bool conv_wgrad(const WgradDesc &c, cudaStream_t s)
{
    // dW[co][t][ci] += sum_p G[p][co] X[p + off(t)][ci]
    if (!encoder()) {
        report_error("fmvd: cuTensorMapEncodeTiled is unavailable");
        return false;
    }
    const int cba = c.cout >= 64 ? 64 : 32;
    const int cbb = c.cin >= 64 ? 64 : 32;
    const int bn = c.cin > 256 ? 256 : c.cin;
    if (c.cout % cba || c.cin % cbb || c.cin % bn || (bn != 32 && bn != 64 && bn != 128 && bn != 256) ||
        (c.taps != 1 && c.taps != 9) || (c.H * c.W) % 64 || (c.W < 64 ? 64 % c.W : c.W % 64)) {
        report_error("fmvd: unsupported weight-gradient geometry");
        return false;
    }
    // N tile (output channels): what tensor memory holds beside every tap
    const int nt = c.cin >= 128 ? 32 : c.cin == 64 ? (cba == 64 ? 64 : 32)
                                                   : (c.cout % 128 == 0 ? 128 : cba == 64 ? 64 : 32);
    const int halo = c.taps == 9 ? 2 : 0;
    CUtensorMap tx, tg;
    if (!map_nhwc(&tx, c.in, c.cin, c.W, c.H, c.N, cbb, kGradW + halo, kGradH + halo) ||
        !map_nhwc(&tg, c.grad, c.cout, c.W, c.H, c.N, nt >= 64 ? 64 : 32, kGradW, kGradH)) {
        report_error("fmvd: tensor map encoding failed");
        return false;
    }
    GemmArgs g{};
    g.N = c.N;
    g.H = c.H;
    g.W = c.W;
    g.taps = c.taps;
    g.cin = c.cin;
    g.cout = c.cout;
    g.dw = c.dw;
    g.db = c.db;
    g.status = c.status;
    if (c.cin >= 128)
        return wgrad_taps<64, 2, 1, 32>(tx, tg, g, s);
    if (c.cin == 64)
        return nt == 64 ? wgrad_taps<64, 1, 2, 64>(tx, tg, g, s) : wgrad_taps<64, 1, 2, 32>(tx, tg, g, s);
    return nt == 128 ? wgrad_taps<32, 1, 4, 128>(tx, tg, g, s)
                     : nt == 64 ? wgrad_taps<32, 1, 4, 64>(tx, tg, g, s) : wgrad_taps<32, 1, 4, 32>(tx, tg, g, s);
}

} // namespace unet
} // namespace fmvd
