// Fused per-plane Richardson-Lucy passes on sm_100a.
//
// One RL view update of the reference (fmvd_deconvolve.impl.cpp:264-272:
// R2C, modulate, C2R, divide, R2C, modulate, C2R, multiply32 = 4 FFTs and 4
// element-wise sweeps, 8 launches per plane) becomes four launches over a
// whole batch of plane pairs:
//
//   row pass  "divide": inverse row FFT of the blurred estimate, the data/blur
//             ratio (the reference's q > 1 rule), forward row FFT of the ratio
//   col pass : forward column FFT, times the view's kernel-2 spectrum,
//             inverse column FFT
//   row pass  "update": inverse row FFT (correction r), the weighted
//             multiplicative update e += w (e r - e), forward row FFT of the
//             new estimate (or, after the last update, the cropped, clipped,
//             truncated sample output)
//   col pass : forward column FFT, times the next view's kernel-1 spectrum,
//             inverse column FFT
//
// Two real planes share one complex transform (real part = plane 2p,
// imaginary part = plane 2p+1): convolution with a real kernel acts on both
// parts independently, so every FFT does the work of two real transforms.
// Each pass keeps its lines in shared memory and registers; between passes
// the batch's complex planes are the only traffic, sized by the host to stay
// resident in L2.
#include "fft_engine.cuh"
#include "rl_kernels.h"
#include "warp_fft.cuh"
#include "tma_util.cuh"

#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <type_traits>
#include <vector>

namespace fmvd {

// Kernel launches issued by this library (host-side count, for reporting).
static unsigned long long g_launches = 0;
unsigned long long rl_launch_count() { return g_launches; }
void rl_count_launch(unsigned long long n) { g_launches += n; }

// Work planes are row-major, element (y, x) of pair p at
// C[(p * H + y) * W + x], but for planes of 1024 rows: there x is exchanged
// within its column block for x ^ f(y), f the bank swizzle of the column
// pass's tile.  That costs the row passes nothing (f is fixed per row, so a
// lane's elements stay T apart), and the column pass fills its tile with
// 16-byte copies that need no swizzle of their own.
struct RowSwizzle {
    int shift, mask;  // f(y) = (y >> shift) & mask; mask 0: none
    __device__ __forceinline__ int f(int y) const { return (y >> shift) & mask; }
};

__device__ __forceinline__ int clamp_src(int i, int n, int border)
{
    // i < n: i; n <= i < n + border: n - 1; beyond: 0 (i >= 0)
    const int c = min(i, n - 1);
    return i < n + border ? c : 0;
}

// Programmatic dependent launch.  Every pass lets the next kernel of its
// stream launch as soon as all of its own blocks have started
// (launch_dependents), and waits for the previous kernel to complete, with
// its writes visible, before it reads anything an earlier kernel produced
// (dependency_wait).  Work on constant operands (weights, spectra) may run
// before the wait, so the next pass's blocks set up while the tail of the
// previous one finishes.  Launched without the attribute, both are no-ops.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Requests the 128-byte line holding p into L1 (no result, no wait).
__device__ __forceinline__ void prefetch_l1(const void *p)
{
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Shared-memory loads by 32-bit shared-window address.
__device__ __forceinline__ float lds_f32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 lds_f32x2(uint32_t addr)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
template <int BITS>
__device__ __forceinline__ float lds_sample(uint32_t row, int sx)
{
    uint32_t v;
    if constexpr (BITS == 16)
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(row + 2u * sx) : "memory");
    else
        asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(row + (uint32_t)sx) : "memory");
    return (float)v;
}

// ----------------------------------------------------------- row passes
enum RowMode { ROW_INIT = 0, ROW_DIVIDE = 1, ROW_UPDATE = 2 };

struct RowArgs {
    RlDims d;
    RlBatch b;
    const float2 *tw;
    int view;
    int last;
    int bulk_data;      // data rows may be fetched with 16-byte bulk copies
    int group_floats;   // warp engine: shared floats per group (transpose + prefetch)
    RowSwizzle sw;      // storage order of the work planes' rows
    const float2 *twN;  // lines above 1024: exp(-2 pi i n / W), n < W
};

// Float to sample as the reference's unpad kernel: clip at the maximum,
// then convert with truncation (saturating at 0 for negatives).
__device__ __forceinline__ void store_sample(void *base, size_t idx, float v, int bits)
{
    if (bits == 16) {
        if (v > 65535.f) v = 65535.f;
        reinterpret_cast<unsigned short *>(base)[idx] = (unsigned short)__float2uint_rz(v);
    } else {
        if (v > 255.f) v = 255.f;
        reinterpret_cast<unsigned char *>(base)[idx] = (unsigned char)__float2uint_rz(v);
    }
}

// Element-wise work of the row passes on row y of pair p (row-invariant
// pointers computed once):
//   INIT:   estimate = 10 * nViews (imaginary part 0 for a missing second plane)
//   DIVIDE: blur b -> data / b where b > 1, else b (divide_kernel, the
//           reference's in-place quirk)
//   UPDATE: correction r -> e + w (e r - e) (multiply32_kernel); after the
//           last view of the last iteration also the output samples
// BITS: the sample width (8 or 16; 0 in the INIT pass, which has no samples),
// so the element-wise step has no per-element branches.  NOOUT: an update pass
// known at compile time not to be the last one, so the output-sample code is
// left out.  SMEM: the operand row is in shared memory at the s_* addresses
// (the data rows in the divide pass, where their alignment allows the bulk
// copy; the weight row in the update pass, always, and the estimate row too
// when EST_S).  Weight rows lie a multiple of 16 bytes apart so that the bulk
// copy takes any plane width: with widths that are not a multiple of four the
// rows used to be read element by element through generic pointers, 22.7 us
// for an update of 8 pairs of 512 x 512 against 14.6.  (Rows padded to W,
// which save the border arithmetic, cost more than they give: 4.2 % of a
// 1024-point step, since the larger shared memory leaves less L1 for the
// twiddle tables.)  Estimate traffic is streamed (evict-first in L2) so that
// the batch's complex work planes stay resident between passes.
template <int MODE, int BITS = 0, bool NOOUT = false, bool SMEM = false, bool EST_S = SMEM>
struct RowWork {
    const RlDims &d;
    float2 *est;             // row y of the pair's estimate (global)
    const void *src0, *src1; // data rows (clamped) of planes 2p and 2p+1, view a.view
    const float *wrow;       // weight row (clamped)
    void *out0, *out1;       // output rows, or null
    bool has1;
    float init0, init1;
    const float *initr0, *initr1;  // rows of a given initial estimate, or null
    uint32_t s_src0, s_src1, s_w, s_est;  // shared-memory rows (SMEM)

    __device__ __forceinline__ RowWork(const RowArgs &a, int p, int y) : d(a.d)
    {
        const int W = d.W;
        has1 = 2 * p + 1 < a.b.nplanes;
        est = a.b.est + ((size_t)p * d.H + y) * W;
        init0 = a.b.init_value;
        init1 = has1 ? a.b.init_value : 0.f;
        initr0 = initr1 = nullptr;
        if (MODE == ROW_INIT && a.b.init) {
            initr0 = a.b.init + ((size_t)(2 * p) * d.H + y) * W;
            initr1 = has1 ? a.b.init + ((size_t)(2 * p + 1) * d.H + y) * W : nullptr;
        }
        const size_t es = d.bits == 16 ? 2 : 1;
        src0 = src1 = nullptr;
        wrow = nullptr;
        out0 = out1 = nullptr;
        if (MODE == ROW_DIVIDE) {
            const size_t base = (size_t)a.view * a.b.view_stride + (size_t)clamp_src(y, d.dataH, d.byD) * d.dataW;
            src0 = (const char *)a.b.data + (base + (size_t)(2 * p) * a.b.plane_stride) * es;
            src1 = has1 ? (const char *)a.b.data + (base + (size_t)(2 * p + 1) * a.b.plane_stride) * es : src0;
        }
        if (MODE == ROW_UPDATE) {
            wrow = a.b.weights + ((size_t)a.view * d.dataH + clamp_src(y, d.dataH, d.byW)) * d.wpitch;
            if (a.last && y < d.dataH) {
                out0 = (char *)a.b.out + ((size_t)(2 * p) * a.b.plane_stride + (size_t)y * d.dataW) * es;
                if (has1)
                    out1 = (char *)a.b.out + ((size_t)(2 * p + 1) * a.b.plane_stride + (size_t)y * d.dataW) * es;
            }
        }
    }

    __device__ __forceinline__ float sample(const void *row, int sx) const
    {
        if constexpr (BITS == 16)
            return (float)reinterpret_cast<const unsigned short *>(row)[sx];
        else
            return (float)reinterpret_cast<const unsigned char *>(row)[sx];
    }

    // The operands of position x that come from global memory (the estimate;
    // the two planes' samples), to be requested ahead of the element-wise step.
    __device__ __forceinline__ float2 fetch(int x) const
    {
        if constexpr (MODE == ROW_UPDATE && !EST_S)
            return est[x];
        if constexpr (MODE == ROW_DIVIDE && !SMEM) {
            const int sx = clamp_src(x, d.dataW, d.bxD);
            return make_float2(sample(src0, sx), has1 ? sample(src1, sx) : 0.f);
        }
        return make_float2(0.f, 0.f);
    }

    __device__ __forceinline__ void apply(int x, float2 &v) const { apply(x, v, fetch(x)); }

    __device__ __forceinline__ void apply(int x, float2 &v, float2 c) const
    {
        if (MODE == ROW_INIT) {
            v = initr0 ? make_float2(__ldcs(initr0 + x), initr1 ? __ldcs(initr1 + x) : 0.f)
                       : make_float2(init0, init1);
            __stcs(est + x, v);
        } else if (MODE == ROW_DIVIDE) {
            // q > 1 keeps the divisor in the range where the fast division is
            // within 2 ulp of the IEEE quotient
            if constexpr (SMEM) {
                const int sx = clamp_src(x, d.dataW, d.bxD);
                c.x = lds_sample<BITS>(s_src0, sx);
                const float s1 = lds_sample<BITS>(s_src1, sx);
                c.y = has1 ? s1 : 0.f;
            }
            float2 q = v;
            q.x = q.x > 1.f ? __fdividef(c.x, q.x) : q.x;
            q.y = q.y > 1.f ? __fdividef(c.y, q.y) : q.y;
            v = q;
        } else {
            static_assert(MODE != ROW_UPDATE || SMEM, "the update pass reads its weight row from shared memory");
            const float w = lds_f32(s_w + 4u * clamp_src(x, d.dataW, d.bxW));
            if constexpr (EST_S)
                c = lds_f32x2(s_est + 8u * x);
            const float2 r = v;
            c.x += w * (c.x * r.x - c.x);
            c.y += w * (c.y * r.y - c.y);
            __stcs(est + x, c);
            v = c;
            if (!NOOUT && out0 && x < d.dataW) {
                store_sample(out0, x, c.x, BITS);
                if (out1)
                    store_sample(out1, x, c.y, BITS);
            }
        }
    }
};

// Row pass for W <= 1024: one group of T lanes per row, warp FFT, no block
// synchronisation.  Rows beyond H (only for tiny planes) compute on row H-1
// and store nothing.
// Occupancy knobs of the warp-engine passes (blocks per SM the register
// allocation must allow, and the widest column block).
#ifndef FMVD_ROW_MIN_BLOCKS
#define FMVD_ROW_MIN_BLOCKS 4
#endif
#ifndef FMVD_COL_MIN_BLOCKS
#define FMVD_COL_MIN_BLOCKS 2
#endif
#ifndef FMVD_COL_MAX_WARPS
#define FMVD_COL_MAX_WARPS 8
#endif
constexpr int kRowWarps = 4;
constexpr int kSms = 148;  // multiprocessors of a B200

template <int W, int MODE, int BITS, bool NOOUT, bool SMEM>
__global__ void __launch_bounds__(kRowWarps * 32, FMVD_ROW_MIN_BLOCKS) row_pass_w(const RowArgs a)
{
    using WF = WarpFft<W>;
    constexpr int T = WF::T, E = WF::E, G = 32 / T;
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(8) uint64_t bars[kRowWarps * G];
    __shared__ __align__(8) uint64_t ebars[MODE == ROW_UPDATE ? kRowWarps * G : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane / T, t = lane % T;
    const int gi = warp * G + g;
    float *gbase = smem + (size_t)gi * a.group_floats;
    float2 *tbuf = reinterpret_cast<float2 *>(gbase);                // padded transpose buffer
    char *pf = reinterpret_cast<char *>(gbase + WF::padded_floats);  // prefetch area, 16-byte aligned
    const int H = a.d.H;
    const int yr = blockIdx.x * (kRowWarps * G) + warp * G + g;
    const bool valid = yr < H;
    const int y = valid ? yr : H - 1;
    const int p = blockIdx.y;
    // element x = t + T m; the swizzle is below 8, so lanes stay among the T
    // of one m, but for T = 4 its upper bit picks the neighbouring m
    float2 *row = a.b.C + ((size_t)p * H + y) * W;
    const int sw = a.sw.f(y), tsw = t ^ (sw & (T - 1)), msw = T < 8 ? sw / T : 0;
    RowWork<MODE, BITS, NOOUT, SMEM> work(a, p, y);

    // Rows the element-wise step needs are fetched by the bulk-copy engine
    // while the inverse transform runs: the weight row in the update pass,
    // the two data rows in the divide pass.  The update pass's estimate row
    // lands in the transpose buffer itself, issued once the inverse
    // transform has read its transpose back, so it takes no shared memory
    // of its own.
    // SMEM is set in the update pass, and in the divide pass exactly when the
    // launch allows the bulk copies of the data rows
    constexpr bool prefetch = SMEM && MODE != ROW_INIT;
    uint64_t *bar = &bars[gi];
    uint64_t *ebar = &ebars[MODE == ROW_UPDATE ? gi : 0];
    pdl_launch_dependents();
    if (prefetch || MODE == ROW_UPDATE) {
        if (t == 0) {
            mbar_init(bar, 1);
            if (MODE == ROW_UPDATE)
                mbar_init(ebar, 1);
            mbar_fence_init();
        }
        __syncwarp();
    }
    if (prefetch && MODE == ROW_UPDATE && t == 0) {
        // the weight row is a plan constant: requested before the wait
        const uint32_t wb = a.d.wpitch * sizeof(float);
        mbar_arrive_expect_tx(bar, wb);
        bulk_load(pf, work.wrow, wb, bar);
    }
    pdl_wait();
    if (prefetch && MODE == ROW_DIVIDE && t == 0) {
        const int es = a.d.bits == 16 ? 2 : 1;
        const uint32_t rb = a.d.dataW * es;
        const uint32_t rs = (rb + 15) & ~15u;
        mbar_arrive_expect_tx(bar, work.has1 ? 2 * rb : rb);
        bulk_load(pf, work.src0, rb, bar);
        if (work.has1)
            bulk_load(pf + rs, work.src1, rb, bar);
    }

    // One copy of the transform code serves both directions: the inverse is
    // conj(DFT(conj(x))), so pass 0 (inverse of the loaded row) and pass 1
    // (forward) run the same loop body; keeping it rolled halves the code the
    // instruction cache must hold.
    float2 v[E];
    if (MODE == ROW_INIT) {
#pragma unroll
        for (int m = 0; m < E; m++)
            v[m] = make_float2(0.f, 0.f);
        if (valid) {
#pragma unroll
            for (int m = 0; m < E; m++)
                work.apply(t + T * m, v[m]);
        }
    }
    int pass = MODE == ROW_INIT ? 1 : 0;
    const auto estimate_to_tbuf = [&]() {
        if (MODE == ROW_UPDATE && pass == 0 && t == 0) {
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(ebar, W * sizeof(float2));
            bulk_load(tbuf, work.est, W * sizeof(float2), ebar);
        }
    };
#pragma unroll 1
    for (; pass < 2; pass++) {
        if (pass == 0) {
#pragma unroll
            for (int m = 0; m < E; m++) {
                const float2 x = row[tsw + T * (T < 8 ? m ^ msw : m)];
                v[m] = make_float2(x.x, -x.y);
            }
        }
        WF::template run_padded<-1>(v, a.tw, tbuf, t, estimate_to_tbuf);
        if (pass == 1)
            break;
#pragma unroll
        for (int m = 0; m < E; m++)
            v[m].y = -v[m].y;
    if (MODE == ROW_UPDATE) {
        const bool ok_w = mbar_wait(bar, 0);
        const bool ok_e = mbar_wait(ebar, 0);
        if (!ok_w || !ok_e) {
            // a copy did not land in time: flag it (the host reports the
            // batch as failed) and wait once more so no copy is left in flight
            if (t == 0)
                atomicExch(a.b.status, 1);
            if (!ok_w)
                mbar_wait(bar, 0);
            if (!ok_e)
                mbar_wait(ebar, 0);
        }
        work.s_est = smem_u32addr(tbuf);
        work.s_w = smem_u32addr(pf);
    } else if (prefetch) {
        if (!mbar_wait(bar, 0)) {
            // the copy did not land in time: flag it (the host reports the
            // batch as failed) and wait once more so no copy is left in flight
            if (t == 0)
                atomicExch(a.b.status, 1);
            mbar_wait(bar, 0);
        }
        const int es = a.d.bits == 16 ? 2 : 1;
        const uint32_t rs = (a.d.dataW * es + 15) & ~15u;
        work.s_src0 = smem_u32addr(pf);
        work.s_src1 = work.has1 ? smem_u32addr(pf + rs) : work.s_src0;
    }
    if (valid) {
#pragma unroll
        for (int m = 0; m < E; m++)
            work.apply(t + T * m, v[m]);
    }
    if (MODE == ROW_UPDATE && !NOOUT && a.last)
        return;
    if (MODE == ROW_UPDATE)
        __syncwarp();  // the estimate row in tbuf is read before the forward transform writes it
    }
    if (valid) {
#pragma unroll
        for (int m = 0; m < E; m++)
            row[tsw + T * (T < 8 ? m ^ msw : m)] = v[m];
    }
}

// --------------------------------------------------------- column pass
struct ColArgs {
    float2 *C;
    const float2 *spec;  // column-pass launch layout
    const float2 *tw;    // warp-FFT twiddles (of kLineM above 1024)
    int H, W;
    const float2 *twN;   // columns above 1024: exp(-2 pi i n / H), n < H
};

__global__ void write_estimate_kernel(const RlDims d, const RlBatch b)
{
    const size_t plane = (size_t)d.dataH * d.dataW;
    const size_t total = plane * b.nplanes;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int z = (int)(i / plane);
        const int y = (int)((i % plane) / d.dataW), x = (int)(i % d.dataW);
        const float2 e = b.est[(size_t)(z >> 1) * d.H * d.W + (size_t)y * d.W + x];
        store_sample(b.out, i, (z & 1) ? e.y : e.x, d.bits);
    }
}

__global__ void split_estimate_kernel(const float2 *__restrict__ est, int nplanes, size_t plane, float *__restrict__ out)
{
    const size_t total = plane * nplanes;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t z = i / plane, r = i % plane;
        const float2 e = est[(z >> 1) * plane + r];
        out[i] = (z & 1) ? e.y : e.x;
    }
}

// float2 shared-memory access by 32-bit shared-window address.
__device__ __forceinline__ void sts2(uint32_t addr, float2 v)
{
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t addr, float4 v)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}
__device__ __forceinline__ float4 lds4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 lds2(uint32_t addr)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}

// Column tile of the warp engine (lengths up to 1024): FC columns as
// interleaved float2, row y at byte 8 FC y, element (y, c) in 8-byte slot
// c ^ f(y) of its row.  The engine moves 8-byte elements, sixteen lanes (one
// 128-byte wavefront) at a time, and f spreads every access of a transform
// over the sixteen slots of that wavefront:
//   T = 32: sixteen lanes hold sixteen consecutive rows of one column, so f
//     steps by one slot per 128 bytes of rows.  It separates column pairs, so
//     the work plane itself is stored in this order (RowSwizzle);
//   T < 32: sixteen lanes hold eight (T = 4: four) rows of two (four)
//     neighbouring columns, so f steps by two (four) slots and a column pair
//     stays one aligned 16-byte unit.
// Either way the tile is filled and written back 16 bytes at a time (8-byte
// copies take a shared-memory cycle per row they touch: 0.75 M conflicts per
// launch of three 1024 x 1024 pairs).
// With T = 16 the two lines of a warp are interleaved lane by lane (line =
// lane & 1) to get eight rows of two columns in a half-warp.
// f uses the low bits of y only, so that for u, k < T it is linear in XOR:
// with the tile on a T * 8 FC byte boundary, the byte address of row
// T a + (u ^ k) is 8 FC T a + (Q(u) ^ R(k)), Q(u) = 8 FC u + 8 (c ^ f(u)),
// R(k) = 8 FC k + 8 f(k): one logic instruction on a lane constant and an
// immediate offset per transpose access.
template <int H, int FC>
struct ColTile {
    static constexpr int T = warp_fft_lanes(H);
    static constexpr int RB = 8 * FC;                     // bytes per row
    static constexpr int rows = T == 32 ? 32 : T < 8 ? 4 : 8;  // rows of a column that f tells apart
    static constexpr int step = T == 32 ? 1 : 16 / rows;
    static constexpr int sh = FC >= 16 ? 0 : FC == 8 ? 1 : FC == 4 ? 2 : 3;
    static constexpr bool pairs = step > 1;               // column pairs stay adjacent
    static constexpr uint32_t align = T * RB;
    static constexpr size_t bytes = (size_t)H * RB + align;
    static __host__ __device__ constexpr uint32_t f(int y) { return (((y & (rows - 1)) >> sh) * step) & (FC - 1); }
    static __host__ __device__ constexpr uint32_t R(int k) { return (uint32_t)RB * k + 8u * f(k); }
    // line (column of the warp) and lane inside the line
    static __device__ __forceinline__ int line(int lane) { return T == 16 ? lane & 1 : lane / T; }
    static __device__ __forceinline__ int pos(int lane) { return T == 16 ? lane >> 1 : lane % T; }
};

// H-point transform of one tile column (the WarpFft<H> four-step): wbase =
// tile + Q(t) (transpose writes, element k1 at row T k1 + (t ^ k1 mod T)),
// rbase = wbase + 8 FC T t (reads of row-block t).
template <int H, int FC, int DIR>
__device__ __forceinline__ void col_fft(float2 *v, const float2 *__restrict__ tw, uint32_t wbase, uint32_t rbase, int t)
{
    using WF = WarpFft<H>;
    using TL = ColTile<H, FC>;
    constexpr int T = WF::T, E = WF::E, S = WF::S;
    Dft<E, DIR>::run(v);
    WF::template twiddle<DIR>(v, tw, t);
#pragma unroll
    for (int k1 = 0; k1 < E; k1++)
        sts2((wbase ^ TL::R(k1 & (T - 1))) + (uint32_t)(T * TL::RB) * k1, v[k1]);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < S; s++)
#pragma unroll
        for (int j = 0; j < T; j++)
            v[s * T + j] = lds2((rbase ^ TL::R(j)) + (uint32_t)(T * T * TL::RB) * s);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < S; s++)
        Dft<T, DIR>::run(v + s * T);
    WF::reorder(v);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// Column pass for H <= 1024: CW warps per block, G = 32 / T columns per
// warp, FC = CW * G columns per block.  The FC-column tile is filled by
// cp.async (whole rows of the tile, 16 to 128 bytes, coalesced), each group
// transforms its column in registers using its own column of the tile as
// transpose buffer, and the tile is written back.  Spectrum in launch layout:
// warp w of the plane (columns G w .. G w + G - 1), register m, lane l at
// spec[(w * E + m) * 32 + l], whatever the block's width.
// Issue is active in 58 % of the cycles, the rest is load phases and barriers
// with few other blocks to run: with the interleaved
// XOR-swizzled tile a 512 x 512 launch of 12 plane pairs takes 19.0 us
// (27.6 us with separate real and imaginary planes of padded rows, whose
// scalar accesses cost twice the shared-memory instructions and 1.7 M bank
// conflicts).
template <int H, int CW>
__global__ void __launch_bounds__(CW * 32, FMVD_COL_MIN_BLOCKS * (8 / CW)) col_pass_w(const ColArgs a)
{
    using WF = WarpFft<H>;
    constexpr int T = WF::T, E = WF::E, G = 32 / T, FC = CW * G, NT = CW * 32;
    using TL = ColTile<H, FC>;
    extern __shared__ __align__(16) float smem[];
    const int W = a.W;
    const int p = blockIdx.y;
    float2 *C = a.C + (size_t)p * H * W + blockIdx.x * FC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float2 *sp = a.spec + (size_t)(blockIdx.x * CW + warp) * E * 32 + lane;
    // this block's slice of the spectrum (contiguous in the launch layout)
    // is brought into L2 while the tile loads and the first transform runs
    pdl_launch_dependents();
    if (threadIdx.x == 0)
        bulk_prefetch_l2(sp, (uint32_t)(E * NT * sizeof(float2)));
    pdl_wait();

    const uint32_t s0 = smem_u32addr(smem);
    const uint32_t base = (s0 + TL::align - 1) & ~(TL::align - 1);
    // fill in 16-byte units (a column pair): a thread keeps its unit of the
    // row and steps RI rows at a time, a multiple of the rows f tells apart,
    // so its swizzle is a constant (none with T = 32, where the plane is
    // stored swizzled)
    constexpr int PR = TL::RB / 16, RI = NT / PR;
    static_assert(RI % TL::rows == 0 && H % RI == 0, "a thread's rows share one swizzle");
    {
        const int y = threadIdx.x / PR, u = threadIdx.x % PR;
        const uint32_t dst = base + TL::RB * y + (TL::pairs ? (16u * u) ^ (8u * TL::f(y)) : 16u * u);
        const char *src = reinterpret_cast<const char *>(C + (size_t)y * W) + 16 * u;
        const size_t pitch = (size_t)RI * W * sizeof(float2);
#pragma unroll 8
        for (int i = 0; i < H / RI; i++)
            cp_async16(dst + RI * TL::RB * i, src + pitch * i);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    const int t = TL::pos(lane), c = warp * G + TL::line(lane);
    const uint32_t q = TL::RB * t + 8u * (c ^ TL::f(t));
    uint32_t wbase = base + q, rbase = wbase + TL::align * t;
    const float2 *tw = a.tw;
    float2 v[E];
#pragma unroll
    for (int m = 0; m < E; m++)
        v[m] = lds2(wbase + TL::align * m);  // row t + T m
    // pass 0: forward transform, times the spectrum, conjugated; pass 1: the
    // same forward code gives the conjugate of the inverse transform
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        // opaque per pass: addresses and twiddles are formed where they are
        // used instead of being kept in registers across the loop
        asm volatile("" : "+r"(wbase), "+r"(rbase), "+l"(tw));
        col_fft<H, FC, -1>(v, tw, wbase, rbase, t);
        if (pass == 1)
            break;
#pragma unroll
        for (int m0 = 0; m0 < E; m0 += 8) {
            asm volatile("" ::: "memory");
#pragma unroll
            for (int m = m0; m < m0 + 8 && m < E; m++) {
                const float2 z = cmul(v[m], __ldg(sp + m * 32));
                v[m] = make_float2(z.x, -z.y);
            }
        }
        asm volatile("" ::: "memory");
    }
#pragma unroll
    for (int m = 0; m < E; m++)
        sts2(wbase + TL::align * m, make_float2(v[m].x, -v[m].y));
    __syncthreads();
#pragma unroll 4
    for (int n = threadIdx.x; n < H * PR; n += NT) {
        const int y = n / PR, u = n % PR;
        const float4 e = lds4(base + TL::RB * y + (TL::pairs ? (16u * u) ^ (8u * TL::f(y)) : 16u * u));
        *reinterpret_cast<float4 *>(C + (size_t)y * W + 2 * u) = e;
    }
}

// -------------------------------------- lines above 1024: R x 512 engine
// A line of N = R * kLineM points (R = 3..8, every supported length above
// 1024) is split over R groups of 16 lanes (half-warps), each running the
// 512-point warp FFT on one sub-line.  Frequencies R k1 + r live in sub-line
// r at position k1 (the work planes keep rows in this order between passes,
// and the column pass's spectrum follows it); space positions n1 + 512 q
// live in group q:
//   frequency -> space:  Z_r = FFT512(sub-line r), Z_r[n1] *= w_N^(r n1),
//                        x[n1 + 512 q] = sum_r Z_r[n1] w_R^(q r)
//   space -> frequency:  u_r[n1] = sum_q x[n1 + 512 q] w_R^(q r),
//                        u_r[n1] *= w_N^(r n1), sub-line r = FFT512(u_r)
// (forward sign; the inverse is conj(forward(conj))).  The sums over the R
// groups go through shared memory between two block barriers.

// v[m] *= w_N^(r n1), n1 = t + 16 m (twN: w_N^n, n < N): the table value
// for every eighth m, times powers of w_N^(16 r) in between (at most seven
// rounding steps; few table addresses live at once)
__device__ __forceinline__ void line_twiddle(float2 *v, const float2 *__restrict__ twN, int r, int t)
{
    const float2 step = __ldg(twN + 16 * r);
#pragma unroll
    for (int m0 = 0; m0 < 32; m0 += 8) {
        float2 w = __ldg(twN + r * (t + 16 * m0));
#pragma unroll
        for (int m = m0; m < m0 + 8; m++) {
            v[m] = cmul(v[m], w);
            if (m + 1 < m0 + 8)
                w = cmul(w, step);
        }
    }
}

// w_R^(r j) (twN: w_N^n with N = R * kLineM)
template <int R>
__device__ __forceinline__ float2 line_coefficient(const float2 *__restrict__ twN, int r, int j)
{
    return __ldg(twN + ((r * j) % R) * kLineM);
}

// Row pass for W = R * 512: R warps, two rows per block (half-warp h of warp
// r is group r of row h).
// SMEM: the launch bulk-copies each row's weight row (update) or data rows
// (divide) into shared memory after the buffers.
// DSTEP: the radix-R step as R-point DFTs per position (true) or as each
// group's weighted sum over all R sub-lines (false); the two schedules give
// the same transform with different instruction mixes (autotuner knob).  With
// the DFTs the update pass runs the element-wise step between the inverse and
// the forward one in the same thread: two block barriers and eight
// shared-memory accesses per point instead of four and twelve (5 to 7 % of a
// step at R = 3 to 7).  The divide pass and R = 8 keep the separate steps:
// merged, the compiler fuses other products of their transforms, and samples
// at a rounding boundary change.
template <int R, int MODE, int BITS, bool NOOUT, bool SMEM, bool DSTEP>
__global__ void __launch_bounds__(R * 32, 16 / R) row_pass_r(const RowArgs a)
{
    using WF = WarpFft<kLineM>;
    constexpr int T = WF::T, E = WF::E, PF2 = WF::padded_f2, N = R * kLineM;
    static_assert(T == 16 && E == 32, "sub-lines are 512-point half-warp transforms");
    extern __shared__ __align__(16) float smem[];
    const int r = threadIdx.x >> 5;
    const int h = (threadIdx.x >> 4) & 1;
    const int t = threadIdx.x & 15;
    float2 *const lbuf = reinterpret_cast<float2 *>(smem) + (size_t)h * R * PF2;  // the row's R buffers
    float2 *const buf = lbuf + (size_t)r * PF2;
    const int y = blockIdx.x * 2 + h;
    const int p = blockIdx.y;
    float2 *row = a.b.C + ((size_t)p * a.d.H + y) * N + r * kLineM + (t ^ a.sw.f(y));  // element t + 16 m at row[16 m]
    RowWork<MODE, BITS, NOOUT, SMEM, false> work(a, p, y);

    // operand rows staged by bulk copies, issued now by one thread per row
    // (the weight row, a plan constant, before the dependency wait)
    constexpr bool staged = SMEM && MODE != ROW_INIT;
    __shared__ __align__(8) uint64_t sbar[2];
    const uint32_t rb = MODE == ROW_UPDATE ? a.d.wpitch * (uint32_t)sizeof(float) : a.d.dataW * (BITS == 8 ? 1u : 2u);
    const uint32_t rs = (rb + 15) & ~15u;
    char *const st = reinterpret_cast<char *>(smem) + sizeof(float2) * 2 * R * PF2 +
                     (size_t)h * (MODE == ROW_UPDATE ? rs : 2 * rs);
    pdl_launch_dependents();
    if (staged && threadIdx.x == 16 * h) {
        mbar_init(&sbar[h], 1);
        mbar_fence_init();
        if (MODE == ROW_UPDATE) {
            mbar_arrive_expect_tx(&sbar[h], rb);
            bulk_load(st, work.wrow, rb, &sbar[h]);
        }
    }
    pdl_wait();
    if (staged && MODE == ROW_DIVIDE && threadIdx.x == 16 * h) {
        mbar_arrive_expect_tx(&sbar[h], work.has1 ? 2 * rb : rb);
        bulk_load(st, work.src0, rb, &sbar[h]);
        if (work.has1)
            bulk_load(st + rs, work.src1, rb, &sbar[h]);
    }

    const auto operands_landed = [&]() {
        if (staged) {
            if (!mbar_wait(&sbar[h], 0)) {
                // the copy did not land in time: flag it (the host reports the
                // batch as failed) and wait once more so no copy is left in flight
                if (threadIdx.x == 16 * h)
                    atomicExch(a.b.status, 1);
                mbar_wait(&sbar[h], 0);
            }
            if (MODE == ROW_UPDATE) {
                work.s_w = smem_u32addr(st);
            } else {
                work.s_src0 = smem_u32addr(st);
                work.s_src1 = work.has1 ? smem_u32addr(st + rs) : work.s_src0;
            }
        }
    };
    constexpr bool MERGE = DSTEP && MODE != ROW_DIVIDE && R != 8;
    const bool no_forward = MODE == ROW_UPDATE && !NOOUT && a.last;  // the output is written, nothing follows

    // MERGE: everything between the 512-point transforms.  Every group has its
    // sub-line in its buffer (position n1); a half-warp takes blocks of 16
    // positions n1 of its row (block b = r, r + R, ...), and one thread runs the
    // R-point DFT over the R buffers, which gives it the space positions
    // n1 + 512 q, the element-wise step on them, and the R-point DFT of the
    // forward transform, back into the same places.  The next block's operands
    // from global memory are requested before the current one is worked on.
    const auto middle = [&]() {
        float2 c[R];
#pragma unroll
        for (int q = 0; q < R; q++)
            c[q] = work.fetch(q * kLineM + 16 * r + t);
#pragma unroll 1
        for (int b = r; b < kLineM / 16; b += R) {
            float2 z[R], next[R];
            const int bn = b + R < kLineM / 16 ? b + R : b;
#pragma unroll
            for (int q = 0; q < R; q++) {
                next[q] = work.fetch(q * kLineM + 16 * bn + t);
                z[q] = MODE == ROW_INIT ? make_float2(0.f, 0.f) : lbuf[q * PF2 + 16 * b + t];
            }
            if (MODE != ROW_INIT) {
                SmallDft<R>::run(z);
#pragma unroll
                for (int q = 0; q < R; q++) {
                    asm volatile("" : "+f"(z[q].x), "+f"(z[q].y));  // rounded here, as where it was stored
                    z[q].y = -z[q].y;
                }
            }
#pragma unroll
            for (int q = 0; q < R; q++) {
                work.apply(q * kLineM + 16 * b + t, z[q], c[q]);
                c[q] = next[q];
            }
            if (!no_forward) {
#pragma unroll
                for (int q = 0; q < R; q++)
                    asm volatile("" : "+f"(z[q].x), "+f"(z[q].y));
                SmallDft<R>::run(z);
#pragma unroll
                for (int q = 0; q < R; q++)
                    lbuf[q * PF2 + 16 * b + t] = z[q];
            }
        }
    };

    // The step by itself, v[m] <- sum_j (group j's v[m]) w_R^(r j): every group
    // puts its sub-line in its buffer (position n1); then (DSTEP) each half-warp
    // of the row runs the R-point DFT over the R buffers in place and every
    // group reads its own buffer back, or (!DSTEP) each group sums all R
    // sub-lines at its own positions.
    const auto line_dft = [&](float2 *v) {
#pragma unroll
        for (int m = 0; m < E; m++)
            buf[t + T * m] = v[m];
        __syncthreads();
        if constexpr (!DSTEP) {
            // each group sums all R sub-lines at its own positions
#pragma unroll
            for (int m = 0; m < E; m++)
                v[m] = lbuf[t + T * m];
#pragma unroll
            for (int j = 1; j < R; j++) {
                const float2 cj = line_coefficient<R>(a.twN, r, j);
#pragma unroll
                for (int m = 0; m < E; m++)
                    v[m] = cadd(v[m], cmul(lbuf[j * PF2 + t + T * m], cj));
            }
            __syncthreads();
        } else {
#pragma unroll 1
            for (int b = r; b < kLineM / 16; b += R) {
                float2 z[R];
#pragma unroll
                for (int q = 0; q < R; q++)
                    z[q] = lbuf[q * PF2 + 16 * b + t];
                SmallDft<R>::run(z);
#pragma unroll
                for (int q = 0; q < R; q++)
                    lbuf[q * PF2 + 16 * b + t] = z[q];
            }
            __syncthreads();
#pragma unroll
            for (int m = 0; m < E; m++)
                v[m] = buf[t + T * m];
        }
    };

    // pass 0: frequency -> space (the inverse as conj(forward(conj))) and
    // the element-wise step; pass 1: space -> frequency.  The rolled loop
    // keeps one copy of the 512-point transform.
    float2 v[E];
    if (MODE == ROW_INIT) {
        if constexpr (MERGE) {
            middle();
        } else {
#pragma unroll
            for (int m = 0; m < E; m++) {
                v[m] = make_float2(0.f, 0.f);
                work.apply(r * kLineM + t + T * m, v[m]);
            }
        }
    } else {
#pragma unroll
        for (int m = 0; m < E; m++) {
            const float2 x = row[T * m];
            v[m] = make_float2(x.x, -x.y);
        }
    }
#pragma unroll 1
    for (int pass = MODE == ROW_INIT ? 1 : 0; pass < 2; pass++) {
        if (pass == 1) {
            if constexpr (MERGE) {
                __syncthreads();
#pragma unroll
                for (int m = 0; m < E; m++)
                    v[m] = buf[t + T * m];
                __syncwarp();
            } else {
                line_dft(v);
            }
            line_twiddle(v, a.twN, r, t);
        }
        WF::template run_padded<-1>(v, a.tw, buf, t);
        if (pass == 1)
            break;
        // the operand rows of this group's space block (positions r * 512 ..
        // r * 512 + 511) are requested into L1 here and read after the sum
        if (MODE == ROW_UPDATE) {
            prefetch_l1(work.est + r * kLineM + 16 * t);
            prefetch_l1(work.est + r * kLineM + 16 * (t + 16));
        } else if (MODE == ROW_DIVIDE && !staged) {
            const int sx = clamp_src(r * kLineM + 64 * (t & 7), a.d.dataW, a.d.bxD);
            prefetch_l1((const char *)(t < 8 ? work.src0 : work.src1) + (size_t)sx * (BITS == 8 ? 1 : 2));
        }
        line_twiddle(v, a.twN, r, t);
        if constexpr (MERGE) {
#pragma unroll
            for (int m = 0; m < E; m++)
                buf[t + T * m] = v[m];
            __syncthreads();
            operands_landed();
            middle();
        } else {
            line_dft(v);
            operands_landed();
#pragma unroll
            for (int m = 0; m < E; m++) {
                v[m].y = -v[m].y;
                work.apply(r * kLineM + t + T * m, v[m]);
            }
        }
        if (no_forward)
            return;
    }
#pragma unroll
    for (int m = 0; m < E; m++)
        row[T * m] = v[m];
}

// Column tile of the line engine: four columns, row y at byte 32 y, element
// (y, c) in slot c ^ f(y), f(y) = 2 ((y >> 2) & 1).  Lane l of a warp holds
// column l & 1 of the warp's pair at position l >> 1, so sixteen lanes hold
// eight rows of two columns, and f puts them in sixteen distinct slots of a
// wavefront.  Column pairs stay together (16-byte fill and write-back).  Row
// y = 512 r + 16 a + (t ^ k) (t, k < 16) is at byte
// 16384 r + 512 a + (Q(t) ^ R(k)), Q(t) = 32 t + 8 (c ^ f(t)),
// R(k) = 32 k + 8 f(k).
struct LineTile {
    static constexpr int RB = 32;
    static __host__ __device__ constexpr uint32_t f(int y) { return 2u * ((y >> 2) & 1); }
    static __host__ __device__ constexpr uint32_t R(int k) { return (uint32_t)RB * k + 8u * f(k); }
};

// 512-point transform (WarpFft<512>: T = 16, E = 32) of one sub-line of a
// line-engine column tile, its own rows as transpose space: wbase = sub-line
// start + Q(t), rbase = wbase + 512 t.
template <int DIR, typename TW>
__device__ __forceinline__ void col_fft_512(float2 *v, const TW &tw, uint32_t wbase, uint32_t rbase, int t)
{
    using WF = WarpFft<kLineM>;
    using TL = LineTile;
    Dft<32, DIR>::run(v);
    WF::template twiddle<DIR>(v, tw, t);
#pragma unroll
    for (int k1 = 0; k1 < 32; k1++)
        sts2((wbase ^ TL::R(k1 & 15)) + 16u * TL::RB * k1, v[k1]);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int j = 0; j < 16; j++)
            v[s * 16 + j] = lds2((rbase ^ TL::R(j)) + 256u * TL::RB * s);
    __syncwarp();
    Dft<16, DIR>::run(v);
    Dft<16, DIR>::run(v + 16);
    WF::reorder(v);
}

// Column pass for H = R * 512: R warps per column pair (lane l of the warp
// (r, pair) is in group r of column 2 pair + (l & 1)), four columns per block,
// so that a row of the tile is a whole 32-byte sector and comes by 16-byte
// copies.  A launch of one 2560 x 2560 pair takes 62 us and 366 MB of L2
// traffic (79 us and 510 MB with two columns per block, filled eight bytes at a
// time), one of 1536 x 1536 23 us (32 us).  Against two columns filled by
// 16-byte copies the step is 13 % faster at R = 3, 9 % at 4, 11 % at 5, 3 % at
// 6, 5 % at 8, 0.6 % slower at 7.  Bound by its block barriers, shared-memory
// accesses and L2 latency (43 % issue active).
// Spectrum in launch layout: warp w = pair * R + r of the plane, register m,
// lane l at spec[(w * 32 + m) * 32 + l].
constexpr int kLineColumns = 4;
// Resident blocks per SM, which cap the registers of a thread.  A launch of at
// most one block per multiprocessor has nothing to share an SM with, and takes
// the kernel compiled for one (R = 3 to 5: 165 to 189 registers instead of 96
// to 128, so more loads in flight per thread; from R = 6 on they are the same).
// Five iterations of two views (us, shared / one block, and two columns per
// block as before): one pair of 1536 x 256 (64 blocks) 437 / 280, 435; three of
// 1536 x 64 (48) 407 / 269, 366; one of 2048 x 512 (128) 528 / 429, 696; one of
// 2560 x 512 (128) 657 / 486, 771; one of 1536 x 128 (32) 317 / 290, 248.
// Beyond a block per SM the shared one is as good or better: three pairs of
// 2048 x 256 (192) 502 / 544, two of 2048 x 512 (256) 576 / 632, three of
// 2560 x 256 (192) 620 / 669.
template <int R>
__host__ __device__ constexpr int col_r_blocks() { return R == 3 ? 3 : R <= 5 ? 2 : 1; }

template <int R, bool DSTEP, int BLOCKS>
__global__ void __launch_bounds__(R * 16 * kLineColumns, BLOCKS) col_pass_r(const ColArgs a)
{
    using WF = WarpFft<kLineM>;
    static_assert(WF::T == 16 && WF::E == 32, "sub-lines are 512-point half-warp transforms");
    constexpr int E = WF::E, H = R * kLineM, FC = kLineColumns, PAIRS = FC / 2, NT = R * 32 * PAIRS;
    using TL = LineTile;
    constexpr uint32_t RB = TL::RB;
    extern __shared__ __align__(16) float smem[];
    const uint32_t s0 = smem_u32addr(smem);
    const uint32_t base = (s0 + 511u) & ~511u;
    const int W = a.W;
    const int p = blockIdx.y;
    float2 *C = a.C + (size_t)p * H * W + FC * blockIdx.x;
    const int lane = threadIdx.x & 31;
    const int pair = (threadIdx.x >> 5) / R, r = (threadIdx.x >> 5) % R;
    const float2 *sp = a.spec + (size_t)(blockIdx.x * (PAIRS * R) + (threadIdx.x >> 5)) * (E * 32) + lane;
    // this block's slice of the spectrum (contiguous in the launch layout)
    // is brought into L2 while the tile loads and the first transform runs
    pdl_launch_dependents();
    if (threadIdx.x == 0)
        bulk_prefetch_l2(sp, (uint32_t)(E * NT * sizeof(float2)));
    pdl_wait();
    // DSTEP: one thread runs the R-point DFTs of a column pair at a position n1
    // (rows 512 q + n1), 16 bytes at a time: in place in the tile before the
    // transforms, and from the tile straight to the plane after them.  (The
    // first step straight from the plane as well costs 3 to 15 %: its loads are
    // not asynchronous.)
    const auto pair_dft = [&](float4 *e) {
        float2 z0[R], z1[R];
#pragma unroll
        for (int q = 0; q < R; q++) {
            z0[q] = make_float2(e[q].x, e[q].y);
            z1[q] = make_float2(e[q].z, e[q].w);
        }
        SmallDft<R>::run(z0);
        SmallDft<R>::run(z1);
#pragma unroll
        for (int q = 0; q < R; q++)
            e[q] = make_float4(z0[q].x, z0[q].y, z1[q].x, z1[q].y);
    };
#pragma unroll 8
    for (int n = threadIdx.x; n < H * PAIRS; n += NT) {
        const int y = n / PAIRS, u = n % PAIRS;
        cp_async16(base + RB * y + ((16u * u) ^ (8u * TL::f(y))), C + (size_t)y * W + 2 * u);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if constexpr (DSTEP) {
        __syncthreads();
#pragma unroll 1
        for (int n = threadIdx.x; n < kLineM * PAIRS; n += NT) {
            const int n1 = n / PAIRS, u = n % PAIRS;
            const uint32_t at = base + RB * n1 + ((16u * u) ^ (8u * TL::f(n1)));
            float4 e[R];
#pragma unroll
            for (int q = 0; q < R; q++)
                e[q] = lds4(at + kLineM * RB * q);
            pair_dft(e);
#pragma unroll
            for (int q = 0; q < R; q++)
                sts4(at + kLineM * RB * q, e[q]);
        }
    }
    __syncthreads();
    const int t = lane >> 1;
    const uint32_t q = RB * t + 8u * ((2 * pair + (lane & 1)) ^ TL::f(t));
    const uint32_t col = base + q;                  // + 512 RB j + 16 RB m: row 512 j + t + 16 m
    const uint32_t seg = base + 512u * RB * r;      // this group's sub-line
    const uint32_t wbase = seg + q, rbase = wbase + 16u * RB * t;

    // !DSTEP: v[m] = sum_j (row 512 j + t + 16 m of this column) w_R^(r j)
    const auto column_sum = [&](float2 *v) {
#pragma unroll
        for (int m = 0; m < E; m++)
            v[m] = lds2(col + 16u * RB * m);
#pragma unroll
        for (int j = 1; j < R; j++) {
            const float2 cj = line_coefficient<R>(a.twN, r, j);
#pragma unroll
            for (int m0 = 0; m0 < E; m0 += 8) {
                asm volatile("" ::: "memory");  // bounds the loads in flight
#pragma unroll
                for (int m = m0; m < m0 + 8; m++)
                    v[m] = cadd(v[m], cmul(lds2(col + 512u * RB * j + 16u * RB * m), cj));
            }
        }
        asm volatile("" ::: "memory");
    };

    float2 v[E];
    // pass 0: space -> frequency, times the spectrum, conjugated; pass 1:
    // the same forward pipeline then runs frequency -> space.  The rolled
    // loop keeps one copy of the transform (its table loads are not kept
    // live from one copy to the next).
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        if (pass == 0) {
            if constexpr (DSTEP) {
#pragma unroll
                for (int m = 0; m < E; m++)
                    v[m] = lds2(wbase + 16u * RB * m);  // row 512 r + t + 16 m: this group's sub-line
                __syncwarp();  // read before this warp's transposes overwrite its segment
            } else {
                column_sum(v);
                __syncthreads();  // every group has read the column before transposes overwrite it
            }
            line_twiddle(v, a.twN, r, t);
        }
        col_fft_512<-1>(v, a.tw, wbase, rbase, t);
        if (pass == 1)
            break;
#pragma unroll
        for (int m0 = 0; m0 < E; m0 += 8) {
            asm volatile("" ::: "memory");
#pragma unroll
            for (int m = m0; m < m0 + 8; m++) {
                const float2 z = cmul(v[m], __ldg(sp + 32 * m));
                v[m] = make_float2(z.x, -z.y);
            }
        }
        asm volatile("" ::: "memory");
    }
    line_twiddle(v, a.twN, r, t);
#pragma unroll
    for (int m = 0; m < E; m++)
        sts2(wbase + 16u * RB * m, v[m]);  // row 512 r + t + 16 m
    __syncthreads();
    if constexpr (DSTEP) {
#pragma unroll 2
        for (int n = threadIdx.x; n < kLineM * PAIRS; n += NT) {
            const int n1 = n / PAIRS, u = n % PAIRS;
            const uint32_t at = base + RB * n1 + ((16u * u) ^ (8u * TL::f(n1)));
            float4 e[R];
#pragma unroll
            for (int q = 0; q < R; q++)
                e[q] = lds4(at + kLineM * RB * q);
            pair_dft(e);
#pragma unroll
            for (int q = 0; q < R; q++)
                *reinterpret_cast<float4 *>(C + (size_t)(kLineM * q + n1) * W + 2 * u) =
                    make_float4(e[q].x, -e[q].y, e[q].z, -e[q].w);
        }
        return;
    }
    column_sum(v);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < E; m++)
        sts2(wbase + 16u * RB * m, make_float2(v[m].x, -v[m].y));
    __syncthreads();
#pragma unroll 4
    for (int n = threadIdx.x; n < H * PAIRS; n += NT) {
        const int y = n / PAIRS, u = n % PAIRS;
        *reinterpret_cast<float4 *>(C + (size_t)y * W + 2 * u) = lds4(base + RB * y + ((16u * u) ^ (8u * TL::f(y))));
    }
}

// Frequency of stored column (or row position) j of a line of length n:
// natural up to 1024, the R x 512 order above.
__host__ __device__ __forceinline__ int stored_frequency(int j, int n)
{
    if (n <= 1024)
        return j;
    const int R = n / kLineM;
    return R * (j % kLineM) + j / kLineM;
}

// Launch layout of the line engine's column-pass spectrum (see col_pass_r):
// warp w = pair * R + r, register m, lane l holds frequency
// ky = R (t + 16 m) + r, t = l >> 1, of stored column 2 pair + (l & 1).
__global__ void permute_spectrum_r(const float2 *__restrict__ nat, float2 *__restrict__ out, int H, int W, float scale)
{
    const int R = H / kLineM;
    const size_t total = (size_t)H * W;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int lane = (int)(i % 32);
        const int m = (int)((i / 32) % 32);
        const int w = (int)(i / 1024);
        const int ky = R * ((lane >> 1) + 16 * m) + w % R;
        const int kx = stored_frequency(2 * (w / R) + (lane & 1), W);
        const float2 k = nat[(size_t)ky * W + kx];
        out[i] = make_float2(k.x * scale, k.y * scale);
    }
}

// Launch layout of the column-pass spectrum for the warp engine: warp w of
// the plane, register m, lane l (see col_pass_w).
template <int H>
__global__ void permute_spectrum_w(const float2 *__restrict__ nat, float2 *__restrict__ out, int W, float scale)
{
    constexpr int T = warp_fft_lanes(H), E = H / T, G = 32 / T;
    using TL = ColTile<H, 2 * G>;
    const size_t total = (size_t)H * W;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int lane = (int)(i % 32);
        const int m = (int)((i / 32) % E);
        const int warp = (int)(i / (32 * E));
        const int n = TL::pos(lane) + T * m;
        const int col = stored_frequency(warp * G + TL::line(lane), W);
        const float2 k = nat[(size_t)n * W + col];
        out[i] = make_float2(k.x * scale, k.y * scale);
    }
}

// Plan-time kernels in FP32 (the reference builds its kernel spectra with an
// FP32 cuFFT, fmvd_deconvolve.impl.cpp:66-76).  Sums use compensated
// (Kahan) accumulation with explicitly rounded operations, so that the
// spectra carry about FP32 rounding of the exact value whatever the kernel
// size.
struct KahanSum {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float v)
    {
        const float y = __fsub_rn(v, c);
        const float t = __fadd_rn(s, y);
        c = __fsub_rn(__fsub_rn(t, s), y);
        s = t;
    }
};

// Separable direct DFT of a small kernel placed at (y - kH/2, x - kW/2) mod (H, W).
// Step 1: A[y][v] = sum_x k[y][x] exp(-2 pi i v (x - cx) / W)
__global__ void kspec_rows(const float *__restrict__ k, int kH, int kW, int W, const float2 *__restrict__ twW,
                           float2 *__restrict__ A)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (v >= W)
        return;
    KahanSum re, im;
    const int cx = kW / 2;
    for (int x = 0; x < kW; x++) {
        const long long ph = ((long long)v * (x - cx)) % W;
        const float2 t = twW[ph < 0 ? ph + W : ph];
        const float kv = k[y * kW + x];
        re.add(__fmul_rn(kv, t.x));
        im.add(__fmul_rn(kv, t.y));
    }
    A[(size_t)y * W + v] = make_float2(re.s, im.s);
}

// Step 2: K[u][v] = sum_y A[y][v] exp(-2 pi i u (y - cy) / H)
__global__ void kspec_cols(const float2 *__restrict__ A, int kH, int H, int W, const float2 *__restrict__ twH,
                           float2 *__restrict__ K)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int u = blockIdx.y;
    if (v >= W)
        return;
    KahanSum re, im;
    const int cy = kH / 2;
    for (int y = 0; y < kH; y++) {
        const long long ph = ((long long)u * (y - cy)) % H;
        const float2 t = twH[ph < 0 ? ph + H : ph];
        const float2 a = A[(size_t)y * W + v];
        re.add(__fmul_rn(a.x, t.x));
        re.add(-__fmul_rn(a.y, t.y));
        im.add(__fmul_rn(a.x, t.y));
        im.add(__fmul_rn(a.y, t.x));
    }
    K[(size_t)u * W + v] = make_float2(re.s, im.s);
}

// Weights normalised over views, rows wpitch apart (the floats past dataW
// are zero and never used).
__global__ void normalize_weights_kernel(const float *__restrict__ in, float *__restrict__ out, const RlDims d)
{
    const size_t n = (size_t)d.dataH * d.dataW, pitched = (size_t)d.dataH * d.wpitch;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < pitched; i += (size_t)gridDim.x * blockDim.x) {
        const int y = (int)(i / d.wpitch), x = (int)(i % d.wpitch);
        const size_t j = (size_t)y * d.dataW + x;
        float s = 0.f;
        for (int v = 0; v < d.V && x < d.dataW; v++)
            s += in[(size_t)v * n + j];
        for (int v = 0; v < d.V; v++) {
            const float w = x < d.dataW ? in[(size_t)v * n + j] : 0.f;
            out[(size_t)v * pitched + i] = s > 0.f ? w / s : w;
        }
    }
}

__device__ __forceinline__ int clamp_src_d(int i, int n, int border)
{
    return i < n ? i : (i < n + border ? n - 1 : 0);
}

__global__ void conv_same_kernel(const float *__restrict__ img, int dH, int dW, const float *__restrict__ k, int kH,
                                 int kW, int fH, int fW, float *__restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= dW || y >= dH)
        return;
    KahanSum acc;
    for (int ky = 0; ky < kH; ky++) {
        int py = (y - (ky - kH / 2)) % fH;
        if (py < 0)
            py += fH;
        const int sy = clamp_src_d(py, dH, kH / 2);
        for (int kx = 0; kx < kW; kx++) {
            int px = (x - (kx - kW / 2)) % fW;
            if (px < 0)
                px += fW;
            const int sx = clamp_src_d(px, dW, kW / 2);
            acc.add(__fmul_rn(img[(size_t)sy * dW + sx], k[ky * kW + kx]));
        }
    }
    out[(size_t)y * dW + x] = acc.s;
}

// ------------------------------------------------------------ dispatch
#define FMVD_FOR_EACH_LENGTH(X) \
    X(16) X(32) X(64) X(128) X(256) X(512) X(1024) X(1536) X(2048) X(2560) X(3072) X(3584) X(4096)

bool rl_length_supported(int n)
{
    switch (n) {
#define X(N) case N:
        FMVD_FOR_EACH_LENGTH(X)
#undef X
        return true;
    default:
        return false;
    }
}

int snap_transform_size(int n)
{
    // fmvd_deconvolve.cpp:22-51
    auto align = [](int a, int b) { return (a % b != 0) ? (a - a % b + b) : a; };
    n = align(n, 16);
    int hibit = 31;
    while (hibit >= 0 && !(n & (1u << hibit)))
        hibit--;
    unsigned lo = 1u << hibit;
    if (lo == (unsigned)n)
        return n;
    unsigned hi = 1u << (hibit + 1);
    if (hi <= 1024)
        return (int)hi;
    return align(n, 512);
}


// Warps per column block of the warp engine: the largest of 8, 4, 2 whose
// columns per block divide W.
static int col_warps(int H, int W)
{
    const int G = 32 / warp_fft_lanes(H);
    for (int cw = FMVD_COL_MAX_WARPS; cw > 1; cw /= 2)
        if (W % (cw * G) == 0)
            return cw;
    return 1;
}

int rl_col_warps(int H, int W, int requested)
{
    if (H > 1024)
        return 0;  // line engine: fixed four-column tile
    if (requested == 0)
        return col_warps(H, W);
    const int G = 32 / warp_fft_lanes(H);
    const bool ok = (requested == 2 || requested == 4 || requested == 8) && requested <= FMVD_COL_MAX_WARPS &&
                    W % (requested * G) == 0;
    return ok ? requested : -1;
}

size_t rl_spectrum_elems(int H, int W) { return (size_t)H * W; }

// Column-pass warps of a launch.  Four-warp blocks where eight-warp ones would
// number fewer than 64: twice as many multiprocessors then share the
// transforms.  Ten iterations of two views (us, 4 / 8 warps): one 512 x 512
// pair (32 blocks of 8 warps) 519 / 643, two 128 x 128 pairs (8) 234 / 262, two
// 256 x 256 pairs (32) 390 / 399; but two 512 x 512 pairs (64) 865 / 814 and
// eight 256 x 256 pairs (128) 523 / 502.  Two warps were never best beyond
// noise.  Not for 1024 rows, where a warp is one column and four of them read
// 32 bytes of a row instead of 64 (five iterations of two views, 4 / 8 warps): one 1024 x 256 pair 291 / 239, four 1024 x 64 pairs 291 / 236, one
// 1024 x 128 pair 247 / 236.
static int launch_col_warps(const RlDims &d, int npairs)
{
    if (d.col_auto && d.H < 1024 && d.col_warps == 8 && d.W / (8 * (32 / warp_fft_lanes(d.H))) * npairs < 64)
        return 4;
    return d.col_warps;
}

// Storage order of the work planes' rows between the passes.
static RowSwizzle row_swizzle(const RlDims &d)
{
    if (d.H != 1024)
        return RowSwizzle{0, 0};
    switch (d.col_warps) {  // ColTile<1024, 8, 4, 2>::f
    case 8: return RowSwizzle{ColTile<1024, 8>::sh, 7};
    case 4: return RowSwizzle{ColTile<1024, 4>::sh, 3};
    default: return RowSwizzle{ColTile<1024, 2>::sh, 1};
    }
}

// Launch of an RL pass with programmatic dependent launch on stream s (the
// pass's blocks may start while the previous kernel of the stream finishes;
// the pass waits for it before reading its results).  Falls back to a plain
// launch if the attribute is refused.
template <typename A>
static void launch_pass(void (*kern)(const A), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A &args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, args) != cudaSuccess) {
        cudaGetLastError();  // clear the refusal; launch without the attribute
        kern<<<grid, block, smem, s>>>(args);
    }
}

// Dynamic shared memory above 48 KB needs an opt-in per function and device.
template <typename K>
static void configure_smem(K kern, size_t bytes, unsigned &mask)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned bit = 1u << (dev & 31);
    if (!(mask & bit)) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        mask |= bit;
    }
}

static bool aligned16(const void *p, size_t bytes) { return ((uintptr_t)p % 16 == 0) && bytes % 16 == 0; }

// Row-pass variant for a launch: update passes per last / not last, divide
// passes per data rows in shared memory or not.
template <int W, int MODE, int BITS>
static void pick_row_w(const RowArgs &a, void (*&kern)(const RowArgs), unsigned *&m)
{
    static unsigned mask[2] = {0, 0};
    if constexpr (MODE == ROW_UPDATE) {
        kern = a.last ? row_pass_w<W, MODE, BITS, false, true> : row_pass_w<W, MODE, BITS, true, true>;
        m = &mask[a.last ? 1 : 0];
    } else {
        kern = a.bulk_data ? row_pass_w<W, MODE, BITS, false, true> : row_pass_w<W, MODE, BITS, false, false>;
        m = &mask[a.bulk_data ? 1 : 0];
    }
}

template <int R, int MODE, int BITS, bool DSTEP>
static void pick_row_r_bits(const RowArgs &a, void (*&kern)(const RowArgs), unsigned *&m)
{
    static unsigned mask[2] = {0, 0};
    if constexpr (MODE == ROW_UPDATE) {
        kern = a.last ? row_pass_r<R, MODE, BITS, false, true, DSTEP> : row_pass_r<R, MODE, BITS, true, true, DSTEP>;
        m = &mask[a.last ? 1 : 0];
    } else {
        kern = a.bulk_data ? row_pass_r<R, MODE, BITS, false, true, DSTEP>
                           : row_pass_r<R, MODE, BITS, false, false, DSTEP>;
        m = &mask[a.bulk_data ? 1 : 0];
    }
}

template <int R, int MODE, bool DSTEP>
static void pick_row_r(const RowArgs &a, void (*&kern)(const RowArgs), unsigned *&m)
{
    static unsigned mask0 = 0;
    if constexpr (MODE == ROW_INIT) {
        kern = row_pass_r<R, MODE, 0, false, false, DSTEP>;
        m = &mask0;
    } else if (a.d.bits == 16) {
        pick_row_r_bits<R, MODE, 16, DSTEP>(a, kern, m);
    } else {
        pick_row_r_bits<R, MODE, 8, DSTEP>(a, kern, m);
    }
}

template <int W, int MODE>
static void launch_row(const RowArgs &a0, cudaStream_t s)
{
    RowArgs a = a0;
    const size_t es = a.d.bits == 16 ? 2 : 1;
    a.bulk_data = aligned16(a.b.data, a.d.dataW * es) && (a.b.view_stride * es) % 16 == 0 &&
                  (a.b.plane_stride * es) % 16 == 0;
    const size_t data_row = (a.d.dataW * es + 15) & ~(size_t)15;
    // operand rows in shared memory, per line
    const size_t operands =
        MODE == ROW_UPDATE ? a.d.wpitch * sizeof(float) : (MODE == ROW_DIVIDE && a.bulk_data ? 2 * data_row : 0);
    void (*kern)(const RowArgs);
    unsigned *m;
    if constexpr (W <= 1024) {
        using WF = WarpFft<W>;
        constexpr int G = 32 / WF::T;
        static_assert(WF::padded_f2 >= W, "the update pass lands the estimate row in the transpose buffer");
        a.group_floats = WF::padded_floats + (int)(operands / sizeof(float));
        const size_t smem = sizeof(float) * kRowWarps * G * (size_t)a.group_floats;
        if constexpr (MODE == ROW_INIT) {
            static unsigned mask0 = 0;
            kern = row_pass_w<W, MODE, 0, false, false>;
            m = &mask0;
        } else if (a.d.bits == 16) {
            pick_row_w<W, MODE, 16>(a, kern, m);
        } else {
            pick_row_w<W, MODE, 8>(a, kern, m);
        }
        configure_smem(kern, 200 * 1024, *m);
        dim3 grid((a.d.H + kRowWarps * G - 1) / (kRowWarps * G), a.b.npairs);
        launch_pass(kern, grid, dim3(kRowWarps * 32), smem, s, a);
    } else {
        constexpr int R = W / kLineM;
        static_assert(W % kLineM == 0 && R >= 3 && R <= 8, "rows above 1024 are 3..8 sub-lines of 512");
        const size_t smem = sizeof(float2) * 2 * R * WarpFft<kLineM>::padded_f2 + 2 * operands;
        if (a.d.radix_step == kRadixSums)
            pick_row_r<R, MODE, false>(a, kern, m);
        else
            pick_row_r<R, MODE, true>(a, kern, m);
        configure_smem(kern, 200 * 1024, *m);
        dim3 grid(a.d.H / 2, a.b.npairs);
        launch_pass(kern, grid, dim3(R * 32), smem, s, a);
    }
    g_launches++;
}

template <int H, int CW>
static void launch_col_w(const ColArgs &a, int npairs, cudaStream_t s)
{
    constexpr int FC = CW * (32 / warp_fft_lanes(H));
    constexpr size_t smem = ColTile<H, FC>::bytes;
    auto kern = col_pass_w<H, CW>;
    static unsigned mask = 0;
    configure_smem(kern, smem, mask);
    dim3 grid(a.W / FC, npairs);
    launch_pass(kern, grid, dim3(CW * 32), smem, s, a);
}

template <int H>
static void launch_col(const ColArgs &a, int npairs, int cw, int radix_step, cudaStream_t s)
{
    if constexpr (H <= 1024) {
        switch (cw) {
        case 8: launch_col_w<H, 8>(a, npairs, s); break;
        case 4: launch_col_w<H, 4>(a, npairs, s); break;
        default: launch_col_w<H, 2>(a, npairs, s); break;
        }
    } else {
        constexpr int R = H / kLineM;
        static_assert(H % kLineM == 0 && R >= 3 && R <= 8, "columns above 1024 are 3..8 sub-lines of 512");
        constexpr int FC = kLineColumns;
        constexpr size_t smem = sizeof(float2) * FC * H + 512;  // tile aligned to 512 bytes in the kernel
        const bool sums = radix_step == kRadixSums, few = a.W / FC * npairs <= kSms;
        constexpr int B = col_r_blocks<R>();
        auto kern = sums ? (few ? col_pass_r<R, false, 1> : col_pass_r<R, false, B>)
                         : (few ? col_pass_r<R, true, 1> : col_pass_r<R, true, B>);
        static unsigned mask[4] = {0, 0, 0, 0};
        configure_smem(kern, smem, mask[(sums ? 2 : 0) + (few ? 1 : 0)]);
        dim3 grid(a.W / FC, npairs);
        launch_pass(kern, grid, dim3(R * 16 * FC), smem, s, a);
    }
    g_launches++;
}

template <int MODE>
static void dispatch_row(const RowArgs &a, cudaStream_t s)
{
    switch (a.d.W) {
#define X(N) \
    case N: launch_row<N, MODE>(a, s); break;
        FMVD_FOR_EACH_LENGTH(X)
#undef X
    default: break;
    }
}

size_t rl_wave_points(int H)
{
    // up to 1024 rows two blocks of 256 threads and 32 values each per SM (at
    // 512 and 1024 rows; shorter columns, with 16 values or fewer per thread,
    // take two waves of shorter blocks to the same line)
    size_t per_sm = 2 * 256 * 32;
    switch (H) {
#define X(N) \
    case N: \
        if constexpr (N > 1024) \
            per_sm = (size_t)col_r_blocks<N / kLineM>() * kLineColumns * N; \
        break;
        FMVD_FOR_EACH_LENGTH(X)
#undef X
    default: break;
    }
    return kSms * per_sm;
}

void rl_init(const RlDims &d, const RlBatch &b, const RlTables &t, cudaStream_t s)
{
    RowArgs a{d, b, t.wtwW, 0, 0, 0, 0, row_swizzle(d), t.twW};
    dispatch_row<ROW_INIT>(a, s);
}

void rl_divide(const RlDims &d, const RlBatch &b, const RlTables &t, int view, cudaStream_t s)
{
    RowArgs a{d, b, t.wtwW, view, 0, 0, 0, row_swizzle(d), t.twW};
    dispatch_row<ROW_DIVIDE>(a, s);
}

void rl_update(const RlDims &d, const RlBatch &b, const RlTables &t, int view, bool last, cudaStream_t s)
{
    RowArgs a{d, b, t.wtwW, view, last ? 1 : 0, 0, 0, row_swizzle(d), t.twW};
    dispatch_row<ROW_UPDATE>(a, s);
}

void rl_col(const RlDims &d, const RlBatch &b, const RlTables &t, const float2 *spectrum, cudaStream_t s)
{
    ColArgs a{b.C, spectrum, t.wtwH, d.H, d.W, t.twH};
    const int cw = launch_col_warps(d, b.npairs);
    switch (d.H) {
#define X(N) \
    case N: launch_col<N>(a, b.npairs, cw, d.radix_step, s); break;
        FMVD_FOR_EACH_LENGTH(X)
#undef X
    default: break;
    }
}

int rl_warp_lanes(int n) { return n <= 1024 ? warp_fft_lanes(n) : 0; }

int rl_warp_twiddle_entries(int n)
{
    if (n > 1024)
        return rl_warp_twiddle_entries(kLineM);
    const int T = rl_warp_lanes(n);
    if (T == 0)
        return n;
    const int E = n / T, R = E < kWarpTwiddleRun ? E : kWarpTwiddleRun;
    const int used = (E / R + 1) * T;
    return used > n ? used : n;
}

void rl_kernel_spectrum(const float *d_kernel, int kH, int kW, int H, int W, const float2 *twH, const float2 *twW,
                        float2 *work, float2 *d_out, cudaStream_t s)
{
    float2 *A = work;
    float2 *K = work + (size_t)kH * W;
    kspec_rows<<<dim3((W + 127) / 128, kH), 128, 0, s>>>(d_kernel, kH, kW, W, twW, A);
    kspec_cols<<<dim3((W + 127) / 128, H), 128, 0, s>>>(A, kH, H, W, twH, K);
    const size_t total = rl_spectrum_elems(H, W);
    const int blocks = (int)((total + 255) / 256 > 4096 ? 4096 : (total + 255) / 256);
    // 1 / (H W), rounded once to float (the reference's modulateAndNormalize
    // factor, fmvd_deconvolve_cuda.cu:369)
    const float scale = (float)(1.0 / ((double)H * (double)W));
    switch (H) {
#define X(N) \
    case N: \
        if constexpr (N <= 1024) \
            permute_spectrum_w<N><<<blocks, 256, 0, s>>>(K, d_out, W, scale); \
        else \
            permute_spectrum_r<<<blocks, 256, 0, s>>>(K, d_out, H, W, scale); \
        break;
        FMVD_FOR_EACH_LENGTH(X)
#undef X
    default: break;
    }
}

void rl_write_estimate(const RlDims &d, const RlBatch &b, cudaStream_t s)
{
    write_estimate_kernel<<<1024, 256, 0, s>>>(d, b);
    g_launches++;
}

void rl_split_estimate(const RlDims &d, const float2 *est, int nplanes, float *out, cudaStream_t s)
{
    split_estimate_kernel<<<1024, 256, 0, s>>>(est, nplanes, (size_t)d.H * d.W, out);
    g_launches++;
}

void rl_normalize_weights(const RlDims &d, const float *d_in, float *d_out, cudaStream_t s)
{
    const size_t n = (size_t)d.dataH * d.wpitch;
    const int blocks = (int)((n + 255) / 256 > 4096 ? 4096 : (n + 255) / 256);
    normalize_weights_kernel<<<blocks, 256, 0, s>>>(d_in, d_out, d);
}

void rl_conv_same(const float *d_img, int dH, int dW, const float *d_k, int kH, int kW, float *d_out, cudaStream_t s)
{
    const int fH = snap_transform_size(dH + kH - 1);
    const int fW = snap_transform_size(dW + kW - 1);
    conv_same_kernel<<<dim3((dW + 127) / 128, dH), 128, 0, s>>>(d_img, dH, dW, d_k, kH, kW, fH, fW, d_out);
}

} // namespace fmvd
