// Runs the convolution GEMM kernels' control flow on the CPU: one host thread
// per GPU thread, the device half of unet_gemm.cu as it is (device.inc), and
// stand-ins for the tcgen05 / mbarrier / TMA helpers that move no data.  Every
// operation that needs a whole warp (elect.sync before an MMA or a commit, a
// tensor-memory access, votes, shuffles, __syncwarp) is a meeting of the
// warp's 32 threads at the same operation; a lane that meets another operation,
// or never comes, ends the run with exit code 2: on the GPU the others would
// wait for it for good.  A chosen wait of chosen lanes "times out", and lanes
// run apart by random delays, so that they see a flag set by another warp at
// different times.
//
// emulator KERNEL WARP LANEMASK CALL SEEDS: the CALL-th wait of those lanes
// fails (CALL < 0: none does); prints the number of runs whose status was set.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#include "unet.h"

struct Index {
    int x = 0, y = 0, z = 0;
};
static thread_local Index threadIdx;
static Index blockIdx, gridDim{1, 1, 1};
static thread_local std::mt19937 *rng;

static uint8_t smem_block[256 * 1024 + 1024];
static int fail_warp, fail_call;
static uint32_t fail_lanes;
static thread_local int calls;

static void pause_randomly() { usleep((*rng)() % 60); }

struct Meeting {
    std::mutex m;
    std::condition_variable cv;
    const char *op = nullptr;
    int arrived = 0;
    unsigned generation = 0;
    bool all = true, any = false, result_all = true, result_any = false;
    void meet(int size, const char *what, bool v, bool &all_out, bool &any_out)
    {
        {
            std::unique_lock<std::mutex> l(m);
            if (arrived == 0) {
                op = what;
                all = true;
                any = false;
            } else if (strcmp(op, what)) {
                fprintf(stderr, "thread %d is at %s, others of its group at %s\n", threadIdx.x, what, op);
                _exit(2);
            }
            all = all && v;
            any = any || v;
            if (++arrived == size) {
                arrived = 0;
                result_all = all;
                result_any = any;
                generation++;
                cv.notify_all();
            } else {
                const unsigned g = generation;
                if (!cv.wait_for(l, std::chrono::seconds(20), [&] { return generation != g; })) {
                    fprintf(stderr, "thread %d waits at %s for lanes that do not come\n", threadIdx.x, what);
                    _exit(2);
                }
            }
            all_out = result_all;
            any_out = result_any;
        }
        pause_randomly();
    }
};
static Meeting warps[8], block;
static int block_threads;

static void warp_op(const char *what)
{
    bool a, b;
    warps[threadIdx.x / 32].meet(32, what, true, a, b);
}
static void __syncwarp() { warp_op("syncwarp"); }
static void __syncthreads()
{
    bool a, b;
    block.meet(block_threads, "syncthreads", true, a, b);
}
static bool __all_sync(unsigned, bool v)
{
    bool a, b;
    warps[threadIdx.x / 32].meet(32, "vote", v, a, b);
    return a;
}
static bool __any_sync(unsigned, bool v)
{
    bool a, b;
    warps[threadIdx.x / 32].meet(32, "vote", v, a, b);
    return b;
}
static float __shfl_xor_sync(unsigned, float v, int)
{
    warp_op("shuffle");
    return v;
}
static int min(int a, int b) { return a < b ? a : b; }
static float __uint_as_float(uint32_t u)
{
    float f;
    memcpy(&f, &u, 4);
    return f;
}
template <typename T>
static T __ldg(const T *p) { return *p; }
static void atomicAdd(float *, float) {}
static std::atomic<int> status;
static int atomicExch(int *, int v) { return status.exchange(v); }
#undef __grid_constant__
#define __grid_constant__

namespace fmvd {
namespace umma {
struct Desc {
    Desc operator+(uint32_t) const { return *this; }
};
static uint32_t smem_addr(const void *) { return 0; }
static Desc make_desc(uint32_t, uint32_t, uint32_t, int) { return Desc(); }
static uint32_t make_idesc(int, int, int, int) { return 0; }
static int warp_index() { return threadIdx.x / 32; }
static void bar_init(uint64_t *, uint32_t) {}
static void bar_fence_init() {}
static void bar_expect_tx(uint64_t *, uint32_t) {}
static void bar_arrive(uint64_t *) {}
static bool bar_wait(uint64_t *, uint32_t)
{
    pause_randomly();
    const int lane = threadIdx.x % 32;
    return !(calls++ == fail_call && threadIdx.x / 32 == fail_warp && (fail_lanes >> lane & 1));
}
static void tma_load_2d(void *, const CUtensorMap *, int, int, uint64_t *) {}
static void tma_load_4d(void *, const CUtensorMap *, int, int, int, int, uint64_t *) {}
static void tc_fence_before() {}
static void tc_fence_after() {}
static void tmem_alloc(uint32_t *p, uint32_t)
{
    warp_op("alloc");
    *p = 0;
}
static void tmem_relinquish() { warp_op("relinquish"); }
static void tmem_dealloc(uint32_t, uint32_t) { warp_op("dealloc"); }
static void mma_bf16(uint32_t, Desc, Desc, uint32_t, uint32_t) { warp_op("mma"); }
static void mma_commit(uint64_t *) { warp_op("commit"); }
static void tmem_ld16(uint32_t, float (&v)[16])
{
    warp_op("tensor-memory load");
    for (float &x : v)
        x = 0.f;
}
static void ldg32(const void *, uint32_t (&)[8]) {}
static void stg32(void *, const uint32_t (&)[8]) {}
} // namespace umma
} // namespace fmvd

#include "device.inc"

int main(int argc, char **argv)
{
    using namespace fmvd::unet;
    if (argc != 6)
        return 1;
    fail_warp = atoi(argv[2]);
    fail_lanes = (uint32_t)strtoul(argv[3], nullptr, 0);
    fail_call = atoi(argv[4]);
    int set = 0;
    for (int seed = 0; seed < atoi(argv[5]); seed++) {
        GemmArgs g{};
        int dummy;
        float bias_sums[64];
        g.N = 1;
        g.H = g.W = 32;
        g.bw = 32;
        g.bh = 4;
        g.taps = 9;
        g.cin = g.cout = 32;
        g.dw = g.db = bias_sums;
        g.status = &dummy;
        status = 0;
        const CUtensorMap map{};
        const int tiles = 9;
        const bool wgrad = !strcmp(argv[1], "wgrad");
        block_threads = wgrad ? 128 : kPersistentThreads;
        std::vector<std::thread> threads;
        for (int t = 0; t < block_threads; t++)
            threads.emplace_back([&, t] {
                std::mt19937 r(seed * 1000 + t);
                rng = &r;
                threadIdx.x = t;
                calls = 0;
                if (wgrad)
                    conv_wgrad_kernel<32, 1, 4, 32, 9>(map, map, g, tiles, tiles);
                else if (!strcmp(argv[1], "halo"))
                    conv_halo<32, 1, 32>(map, map, g, tiles);
                else
                    conv_gemm_persistent<32, 32>(map, map, g, tiles, 1);
            });
        for (auto &t : threads)
            t.join();
        set += status.load() != 0;
    }
    printf("%d\n", set);
    return 0;
}
