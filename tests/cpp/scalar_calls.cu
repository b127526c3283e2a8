// Calls that return a scalar to the host, seen from a program that shares the context's stream:
//   idle      how often the stream still has work when vec_norm2, vec_dot or diag_eval returns (expected 0)
//   blocking  with the device set to block its waiting threads: the share of a long wait that the thread spent running
#include <cstdio>
#include <cstring>
#include <ctime>

#include <cuda_runtime.h>

#include "numa_gpu.h"

static int check(int rc, const char* what) {
    if (rc != NUMA_GPU_OK) std::printf("%s: status %d\n", what, rc);
    return rc;
}

static int idle() {
    const size_t n = 15, N = n * n * n;
    numa_gpu_ctx* ctx;
    numa_gpu_vec *x, *y;
    numa_gpu_bratu3d* op;
    void* stream;
    if (check(numa_gpu_ctx_create(0, &ctx), "ctx") || check(numa_gpu_vec_create(ctx, N, &x), "vec") ||
        check(numa_gpu_vec_create(ctx, N, &y), "vec") || check(numa_gpu_bratu3d_create(ctx, n, 1.0, &op), "op") ||
        check(numa_gpu_ctx_stream(ctx, &stream), "stream"))
        return 1;
    int busy[3] = {};
    double v;
    for (int i = 0; i < 2000; ++i) {
        if (check(numa_gpu_vec_norm2(x, &v), "norm2")) return 1;
        busy[0] += cudaStreamQuery((cudaStream_t)stream) == cudaErrorNotReady;
        if (check(numa_gpu_vec_dot(x, y, &v), "dot")) return 1;
        busy[1] += cudaStreamQuery((cudaStream_t)stream) == cudaErrorNotReady;
        if (check(numa_gpu_diag_eval(op, x, NUMA_GPU_FP64, y, &v), "eval")) return 1;
        busy[2] += cudaStreamQuery((cudaStream_t)stream) == cudaErrorNotReady;
    }
    std::printf("%d %d %d\n", busy[0], busy[1], busy[2]);
    numa_gpu_bratu3d_destroy(op);
    numa_gpu_vec_destroy(x);
    numa_gpu_vec_destroy(y);
    numa_gpu_ctx_destroy(ctx);
    return 0;
}

static double seconds(clockid_t c) {
    timespec t;
    clock_gettime(c, &t);
    return (double)t.tv_sec + 1e-9 * (double)t.tv_nsec;
}

static int blocking() {
    if (cudaSetDeviceFlags(cudaDeviceScheduleBlockingSync) != cudaSuccess) return 1;
    const size_t n = 127, N = n * n * n;
    numa_gpu_ctx* ctx;
    numa_gpu_vec *r, *z;
    numa_gpu_mg* mg;
    if (check(numa_gpu_ctx_create(0, &ctx), "ctx") || check(numa_gpu_vec_create(ctx, N, &r), "vec") ||
        check(numa_gpu_vec_create(ctx, N, &z), "vec") || check(numa_gpu_mg_create(ctx, n, 2, 2, &mg), "mg"))
        return 1;
    double v, wall = 0.0, cpu = 0.0;
    for (int rep = 0; rep < 2; ++rep) {  // the second is timed
        for (int i = 0; i < 300; ++i)    // tens of milliseconds
            if (check(numa_gpu_mg_apply(mg, r, z), "apply")) return 1;
        wall = -seconds(CLOCK_MONOTONIC);
        cpu = -seconds(CLOCK_THREAD_CPUTIME_ID);
        if (check(numa_gpu_vec_norm2(z, &v), "norm2")) return 1;
        cpu += seconds(CLOCK_THREAD_CPUTIME_ID);
        wall += seconds(CLOCK_MONOTONIC);
    }
    std::printf("%g %g\n", cpu / wall, wall);
    numa_gpu_mg_destroy(mg);
    numa_gpu_vec_destroy(r);
    numa_gpu_vec_destroy(z);
    numa_gpu_ctx_destroy(ctx);
    return 0;
}

int main(int argc, char** argv) {
    if (argc > 1 && !std::strcmp(argv[1], "idle")) return idle();
    if (argc > 1 && !std::strcmp(argv[1], "blocking")) return blocking();
    return 2;
}
