// The announced read-back of a device scalar (Announced, csrc/common.cuh): an announcement that an exception cut off
// after its kernel had taken it must not answer a later fetch of the same scalar.  Prints what a plain fetch, a
// renewed announcement and one with a plain fetch in between return; the expected values are 2, 3 and 4.
#include <cstdio>

#include "numa_internal.hpp"

using namespace numa::gpu;

int main() {
    Context ctx(0);
    const size_t N = 1000;
    DeviceArray<double> v(N);
    double* s = ctx.scalar(kSlotNormF);
    const auto fill_with_norm = [&](double norm) {
        dev_fill(ctx, v.p, 0.0, N);
        dev_fill(ctx, v.p + 17, norm, 1);
    };
    fill_with_norm(1.0);
    try {
        Announced a(ctx, s, 1);
        dev_norm2(ctx, v.p, N, s);  // takes the announcement
        ctx.sync();
        throw 0;
    } catch (int) {
    }
    fill_with_norm(2.0);
    dev_norm2(ctx, v.p, N, s);
    const double plain = ctx.fetch1(s);
    fill_with_norm(3.0);
    Announced b(ctx, s, 1);
    dev_norm2(ctx, v.p, N, s);
    const double renewed = b.fetch1();
    Announced c(ctx, s, 1);
    dev_norm2(ctx, v.p, N, s);
    ctx.fetch1(ctx.scalar(kSlotTmp0));
    fill_with_norm(4.0);
    dev_norm2(ctx, v.p, N, s);
    std::printf("%.17g %.17g %.17g\n", plain, renewed, c.fetch1());
    return 0;
}
