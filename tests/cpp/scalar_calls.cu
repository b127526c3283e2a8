// Calls that return a scalar to the host, seen from a program that shares the context's stream:
//   idle      how often the stream still has work when vec_norm2, vec_dot or diag_eval returns (expected 0)
#include <cstdio>
#include <cstring>

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

int main(int argc, char** argv) {
    if (argc > 1 && !std::strcmp(argv[1], "idle")) return idle();
    return 2;
}
