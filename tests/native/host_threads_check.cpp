// Two host threads, each with its own stream and its own periodic uniform cubic plan: the plans share
// their kernels and need very different amounts of shared memory. Every call has to succeed, and every
// thread's last result has to be its first one, bit for bit. Arguments: cells and lines of either
// thread, calls, and 1 for the refined builder.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/ddcb.h"

static std::atomic<int> waiting {2}, failures {0};

static void fail(const char* what, const char* why)
{
    if (failures++ < 5) std::printf("FAIL %s: %s\n", what, why);
}

static void work(int nc, int lines, int calls, int precision)
{
    ddcb_bsplines bs = nullptr;
    ddcb_builder b = nullptr;
    std::vector<double> pts(nc);
    int64_t n = 0;
    ddcb_builder_options opt {};
    opt.precision = precision;
    bool ok = ddcb_bsplines_create_uniform(3, 1, 0.0, 1.0, nc, &bs) == DDCB_SUCCESS
              && ddcb_greville_points(bs, DDCB_PERIODIC, DDCB_PERIODIC, pts.data(), nc, &n) == DDCB_SUCCESS
              && ddcb_builder_create(bs, pts.data(), nc, DDCB_PERIODIC, DDCB_PERIODIC, &opt, &b) == DDCB_SUCCESS;
    if (!ok) fail("create", ddcb_last_error_message());
    size_t const in = size_t(nc) * lines, out = size_t(nc + 3) * lines;
    std::vector<double> v(in), first(out), last(out);
    for (size_t i = 0; i < in; ++i) v[i] = double((i * 2654435761u) % 1000) / 500.0 - 1.0;
    double *dv = nullptr, *dc = nullptr;
    cudaStream_t s = nullptr;
    ok = ok && cudaMalloc(&dv, in * 8) == cudaSuccess && cudaMalloc(&dc, out * 8) == cudaSuccess
         && cudaMemcpy(dv, v.data(), in * 8, cudaMemcpyHostToDevice) == cudaSuccess && cudaStreamCreate(&s) == cudaSuccess;
    --waiting;
    while (waiting.load() > 0) std::this_thread::yield();
    ddcb_lines const lv {nc, lines, lines, 1, 0}, lc {nc + 3, lines, lines, 1, 0}, none {0, 1, 0, 0, 0};
    for (int i = 0; ok && i < calls; ++i) {
        if (ddcb_build(b, dc, lc, dv, lv, nullptr, none, nullptr, none, s) != DDCB_SUCCESS) fail("build", ddcb_last_error_message());
        if (i == 0) cudaMemcpyAsync(first.data(), dc, out * 8, cudaMemcpyDeviceToHost, s);
    }
    if (ok) {
        cudaMemcpyAsync(last.data(), dc, out * 8, cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) fail("stream", "an error in the queued work");
        if (std::memcmp(first.data(), last.data(), out * 8) != 0) fail("result", "the last call differs from the first");
    }
    cudaFree(dv);
    cudaFree(dc);
    if (b) ddcb_builder_destroy(b);
    if (bs) ddcb_bsplines_destroy(bs);
}

int main(int argc, char** argv)
{
    if (argc < 7) return 2;
    int a[6];
    for (int i = 0; i < 6; ++i) a[i] = std::atoi(argv[i + 1]);
    std::thread one(work, a[0], a[1], a[4], a[5]), two(work, a[2], a[3], a[4], a[5]);
    one.join();
    two.join();
    std::printf("%d failures\n", failures.load());
    return failures.load() ? 1 : 0;
}
