// brusselator.cu — the Brusselator family on the GPU.
//
// * Brusselator1D: the reference's Brusselator1DStep (problems/brusselator1d.hpp:22-192), one
//   implicit-Euler step of the 1D reaction-diffusion system with Dirichlet u = 1, v = 3, and its
//   point-block Jacobi preconditioner BrusselatorJacobi (:194-222).  Every expression follows the
//   reference's order of operations (the library is compiled without FMA contraction), so F, J v,
//   F'' and the block solves are bit-identical to the reference.
// * Brusselator2D: the same reaction terms with parameters A, B, D_u, D_v, dt on an n x n periodic
//   grid of the unit square (h = 1/n), the 2-species reaction-diffusion configuration; and
//   BrussMG2D, a geometric multigrid for the coupled 2x2-block Jacobian K(w) - diag(D_u, D_v) Lap_h,
//   in FP64 (bit-identical to the CPU restatement) or FP32.
//
// Layouts.  Operator vectors are the reference's: w = (u, v) component-major, each plane
// row-major (i * n + j).  Inside BrussMG2D every level keeps (u, v) interleaved per point (one
// 8-byte FP32 or 16-byte FP64 pair) and the 2x2 block (k11, k12, k21, k22) per point (16 or 32
// bytes), so a point-block update is one vector load of each; the points are stored colour-split
// (each colour's points together, row-major), so a colour pass reads and writes only the cache
// lines of the colours it touches.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "numa_internal.hpp"

namespace numa::gpu {

namespace {

// ============================================================================== Brusselator1D
struct B1Geom {
    int n;
    double invdt, h2inv, alpha, A, B, base;
};

// F(w) (brusselator1d.hpp:47-69): boundary values u = 1, v = 3 outside the grid.
__global__ void __launch_bounds__(256) k_b1_eval(const double* __restrict__ w, const double* __restrict__ prev,
                                                 double* __restrict__ out, B1Geom G) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = G.n;
    if (i >= n) return;
    const double u = w[i], v = w[n + i];
    const double um = i > 0 ? w[i - 1] : 1.0, up = i + 1 < n ? w[i + 1] : 1.0;
    const double vm = i > 0 ? w[n + i - 1] : 3.0, vp = i + 1 < n ? w[n + i + 1] : 3.0;
    const double lu = (um - 2.0 * u + up) * G.h2inv;
    const double lv = (vm - 2.0 * v + vp) * G.h2inv;
    out[i] = (u - prev[i]) * G.invdt - G.alpha * lu - G.A - u * u * v + (G.B + 1.0) * u;
    out[n + i] = (v - prev[n + i]) * G.invdt - G.alpha * lv - G.B * u + u * u * v;
}

// F'(w) d (:71-98): a direction is zero outside the grid.
__global__ void __launch_bounds__(256) k_b1_jvp(const double* __restrict__ w, const double* __restrict__ d,
                                                double* __restrict__ out, B1Geom G) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = G.n;
    if (i >= n) return;
    const double u = w[i], v = w[n + i], du = d[i], dv = d[n + i];
    const double dum = i > 0 ? d[i - 1] : 0.0, dup = i + 1 < n ? d[i + 1] : 0.0;
    const double dvm = i > 0 ? d[n + i - 1] : 0.0, dvp = i + 1 < n ? d[n + i + 1] : 0.0;
    const double ldu = (dum - 2.0 * du + dup) * G.h2inv;
    const double ldv = (dvm - 2.0 * dv + dvp) * G.h2inv;
    out[i] = G.invdt * du - G.alpha * ldu - (2.0 * u * v) * du - u * u * dv + (G.B + 1.0) * du;
    out[n + i] = G.invdt * dv - G.alpha * ldv - G.B * du + (2.0 * u * v) * du + u * u * dv;
}

// F''(w)[d, d] = (-q, q), q = 2 v du^2 + 4 u du dv (:100-118).  Also the 2D operator's (any plane size).
__global__ void __launch_bounds__(256) k_bruss_d2(const double* __restrict__ w, const double* __restrict__ d,
                                                  double* __restrict__ out, size_t m) {
    pdl_wait();
    pdl_trigger();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const double u = w[i], v = w[m + i], du = d[i], dv = d[m + i];
    const double q = 2.0 * v * du * du + 4.0 * u * du * dv;
    out[i] = -q;
    out[m + i] = q;
}

// The 2x2 point blocks without the off-diagonal diffusion (:120-141), one plane each.
__global__ void __launch_bounds__(256) k_b1_blocks(const double* __restrict__ w, double* __restrict__ a, B1Geom G) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = G.n;
    if (i >= n) return;
    const double u = w[i], v = w[n + i];
    a[i] = G.base - 2.0 * u * v + (G.B + 1.0);
    a[n + i] = -u * u;
    a[2 * n + i] = -G.B + 2.0 * u * v;
    a[3 * n + i] = G.base + u * u;
}

// BrusselatorJacobi::Bound (:198-214): z = block^-1 r, or z = r where the determinant is not
// finite or below 1e-14 in magnitude.
__global__ void __launch_bounds__(256) k_b1_block_apply(const double* __restrict__ a, const double* __restrict__ r,
                                                        double* __restrict__ z, int n) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a11 = a[i], a12 = a[n + i], a21 = a[2 * n + i], a22 = a[3 * n + i];
    const double ru = r[i], rv = r[n + i];
    const double det = a11 * a22 - a12 * a21;
    if (!isfinite(det) || fabs(det) < 1e-14) {
        z[i] = ru;
        z[n + i] = rv;
        return;
    }
    z[i] = (a22 * ru - a12 * rv) / det;
    z[n + i] = (-a21 * ru + a11 * rv) / det;
}

// ============================================================================== Brusselator2D
struct B2Geom {
    int n;
    double invdt, A, B, Bp1, c1, duh, dvh;  // 1/dt, A, B, B + 1, 1/dt + (B + 1), D_u h^-2, D_v h^-2
};

// ((W - c) + (E - c)) + ((S - c) + (N - c)) on the periodic grid: for a smooth state every
// difference of neighbours is exact, so F keeps no rounding floor of order eps * D h^-2 (the form
// Sum - 4c would cancel values near 1 before the multiplication by D h^-2).
__device__ __forceinline__ double lap5(const double* __restrict__ a, int n, int i, int j, double c) {
    const int jm = j == 0 ? n - 1 : j - 1, jp = j + 1 == n ? 0 : j + 1;
    const int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
    const size_t r = (size_t)i * n;
    return ((a[r + jm] - c) + (a[r + jp] - c)) + ((a[(size_t)im * n + j] - c) + (a[(size_t)ip * n + j] - c));
}

// F(w) = (w - w_prev)/dt - diag(D_u, D_v) h^-2 L w - reaction, as FMA chains (the kernel is bound
// by the FP64 pipe, not by HBM):
//   F_u = fma(B+1, u, fma(-u^2, v, fma(-D_u h^-2, L u, fma(u - u_prev, 1/dt, -A))))
//   F_v = fma(u^2, v, fma(-B, u, fma(-D_v h^-2, L v, (v - v_prev) / dt)));
// optionally ||F||.  L u is lap5's ((W - c) + (E - c)) + ((S - c) + (N - c)), with each neighbour
// difference computed once and shared: a point forms its east difference E - c and takes its west
// one as minus the east difference of the lane to its left (RN(a - b) = -RN(b - a) exactly), and
// forms its north difference N - c, keeping it as the next row's minus-south difference while the
// thread marches down its rows.  Five FP64 instructions for each Laplacian instead of seven, the
// same bits.  A warp covers 31 columns: lane 0 is the halo column whose east difference lane 1 needs.
// FIXED (the mixed path's evaluation): each Laplacian as W + E + S + N - 4c in 64-bit fixed point, rounded
// once (lap5_fixed, common.cuh; more accurate than the sum of rounded differences), on the integer pipe
// instead of five FP64 instructions a species.
template <bool NORM, bool FIXED = false>
__global__ void __launch_bounds__(256) k_b2_eval(const double* __restrict__ w, const double* __restrict__ prev,
                                                 double* __restrict__ out, B2Geom G, int rows, RedArgs red,
                                                 double* norm_out, HostOut host) {
    pdl_wait();
    pdl_trigger();
    const int n = G.n;
    const size_t nn = (size_t)n * n;
    const int lane = threadIdx.x;
    const int jr = (int)blockIdx.x * 31 + lane - 1;  // lane 0: the column left of the warp's 31
    const int j = ((jr % n) + n) % n, jp = j + 1 == n ? 0 : j + 1;  // lanes past the grid wrap (any n)
    const bool owner = lane >= 1 && jr < n;
    const double* wu = w;
    const double* wv = w + nn;
    double acc[1] = {0.0};
    const int i0 = ((int)blockIdx.y * 8 + (int)threadIdx.y) * rows, i1 = min(i0 + rows, n);
    if (i0 < n) {
        const int im0 = i0 == 0 ? n - 1 : i0 - 1;
        double u = wu[(size_t)i0 * n + j], v = wv[(size_t)i0 * n + j];
        double su = 0.0, sv = 0.0;  // S - c of row i0 (FIXED: S itself)
        if (FIXED) {
            su = wu[(size_t)im0 * n + j];
            sv = wv[(size_t)im0 * n + j];
        } else {
            su = wu[(size_t)im0 * n + j] - u;
            sv = wv[(size_t)im0 * n + j] - v;
        }
        for (int i = i0; i < i1; ++i) {
            const size_t r = (size_t)i * n, p = r + j;
            const size_t rn = (size_t)(i + 1 == n ? 0 : i + 1) * n;
            const double un = wu[rn + j], vn = wv[rn + j];
            double lu, lv, nu_ = 0.0, nv_ = 0.0;
            if (FIXED) {
                const double Eu = wu[r + jp], Ev = wv[r + jp];
                const double Wu = __shfl_up_sync(0xffffffffu, u, 1), Wv = __shfl_up_sync(0xffffffffu, v, 1);
                lu = lap5_fixed(u, Wu, Eu, su, un);
                lv = lap5_fixed(v, Wv, Ev, sv, vn);
            } else {
                const double eu = wu[r + jp] - u, ev = wv[r + jp] - v;                  // E - c
                const double wu_ = -__shfl_up_sync(0xffffffffu, eu, 1), wv_ = -__shfl_up_sync(0xffffffffu, ev, 1);  // W - c
                nu_ = un - u;                                                           // N - c
                nv_ = vn - v;
                lu = (wu_ + eu) + (su + nu_);
                lv = (wv_ + ev) + (sv + nv_);
            }
            const double uu = u * u;
            const double fu =
                __fma_rn(G.Bp1, u, __fma_rn(-uu, v, __fma_rn(-G.duh, lu, __fma_rn(u - prev[p], G.invdt, -G.A))));
            const double fv = __fma_rn(uu, v, __fma_rn(-G.B, u, __fma_rn(-G.dvh, lv, (v - prev[nn + p]) * G.invdt)));
            if (owner) {
                out[p] = fu;
                out[nn + p] = fv;
                if (NORM) acc[0] = __fma_rn(fv, fv, __fma_rn(fu, fu, acc[0]));
            }
            if (FIXED) {  // the next row's S
                su = u;
                sv = v;
            } else {      // the next row's S - c
                su = -nu_;
                sv = -nv_;
            }
            u = un;
            v = vn;
        }
    }
    if (NORM) {
        block_sum<1>(acc);
        grid_reduce_finish<1>(acc, red, [norm_out] __device__(const double(&t)[1]) { *norm_out = __dsqrt_rn(t[0]); }, host);
    }
}

// The rows a thread marches, and the grid.  Four blocks of this kernel fit an SM; the row chunks are chosen so that
// the blocks fill whole waves of them: 32 rows always left 2048^2 with 3.5 blocks an SM (four on half of them: 147 us;
// with 29 rows 139 us, the FP64 pipe) and 512^2 with 34 blocks in all.
dim3 b2_eval_grid(int n, int sm_count, int& rows) {
    const int kb = (n + 30) / 31, wave = 4 * sm_count, most = (n + 7) / 8;  // at least a row a thread
    int best = 1;
    double best_fill = 0.0;
    for (int w = 1; w <= 4; ++w) {
        const int chunks = std::max(1, std::min(w * wave / kb, most));
        const int waves = (kb * chunks + wave - 1) / wave;
        const double fill = (double)kb * chunks / ((double)waves * wave);
        if (fill > best_fill + 0.01) {
            best = chunks;
            best_fill = fill;
        }
    }
    rows = (n + 8 * best - 1) / (8 * best);
    return dim3((unsigned)kb, (unsigned)((n + 8 * rows - 1) / (8 * rows)));
}

// J d with the point block [[c1 - 2uv, -u^2], [2uv - B, 1/dt + u^2]]:
//   (J d)_u = fma(-u^2, dv, fma(-D_u h^-2, L du, a11 du)),  (J d)_v = fma(a22, dv, fma(a21, du, -D_v h^-2 L dv)).
__global__ void __launch_bounds__(256) k_b2_jvp(const double* __restrict__ w, const double* __restrict__ d,
                                                double* __restrict__ out, B2Geom G) {
    pdl_wait();
    pdl_trigger();
    const int n = G.n;
    const size_t nn = (size_t)n * n;
    const int j = blockIdx.x * 32 + threadIdx.x;
    if (j >= n) return;
    for (int i = blockIdx.y * 8 + threadIdx.y; i < n; i += gridDim.y * 8) {
        const size_t p = (size_t)i * n + j;
        const double u = w[p], v = w[nn + p], du = d[p], dv = d[nn + p];
        const double lu = lap5(d, n, i, j, du), lv = lap5(d + nn, n, i, j, dv);
        const double u2 = 2.0 * u, uu = u * u;
        const double a11 = __fma_rn(-u2, v, G.c1), a21 = __fma_rn(u2, v, -G.B), a22 = G.invdt + uu;
        out[p] = __fma_rn(-uu, dv, __fma_rn(-G.duh, lu, a11 * du));
        out[nn + p] = __fma_rn(a22, dv, __fma_rn(a21, du, -G.dvh * lv));
    }
}

// The FP32 Jacobian product's coefficients at the iterate: (2uv, u^2) per point, in FP32 arithmetic.
__global__ void __launch_bounds__(256) k_b2_coef32(const double* __restrict__ w, size_t nn, float2* __restrict__ c) {
    pdl_wait();
    pdl_trigger();
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nn) return;
    const float u = f64_to_f32(w[p]), v = f64_to_f32(w[nn + p]);  // FP32 from the rounded state
    c[p] = make_float2((2.0f * u) * v, u * u);
}

struct B2Geom32 {
    int n;
    float invdt, B, c1, duh, dvh;
};

__device__ __forceinline__ float to_f32(double x) { return f64_to_f32(x); }
__device__ __forceinline__ float to_f32(float x) { return x; }

// J d in FP32 arithmetic (FP64 out; d in FP64 or already in FP32): a 32 x 8 tile of both components
// with its one-point periodic halo is rounded to FP32 once per point (integer-pipe conversion) into
// shared memory.
template <class VT>
__global__ void __launch_bounds__(256) k_b2_jvp32(const float2* __restrict__ coef, const VT* __restrict__ d,
                                                  double* __restrict__ out, B2Geom32 G) {
    pdl_wait();
    pdl_trigger();
    constexpr int TX = 32, TY = 8;
    __shared__ float tu[TY + 2][TX + 3], tv[TY + 2][TX + 3];
    const int n = G.n;
    const size_t nn = (size_t)n * n;
    const int i0 = blockIdx.y * TY, j0 = blockIdx.x * TX;
    const int tid = threadIdx.y * TX + threadIdx.x;
    for (int idx = tid; idx < (TY + 2) * (TX + 2); idx += TX * TY) {
        const int a = idx / (TX + 2), b = idx - a * (TX + 2);
        const int gi = (i0 - 1 + a + n) % n, gj = (j0 - 1 + b + n) % n;
        const size_t q = (size_t)gi * n + gj;
        tu[a][b] = to_f32(d[q]);
        tv[a][b] = to_f32(d[nn + q]);
    }
    __syncthreads();
    const int i = i0 + threadIdx.y, j = j0 + threadIdx.x;
    if (i >= n || j >= n) return;
    const int a = threadIdx.y + 1, b = threadIdx.x + 1;
    const float du = tu[a][b], dv = tv[a][b];
    const float lu = ((tu[a][b - 1] - du) + (tu[a][b + 1] - du)) + ((tu[a - 1][b] - du) + (tu[a + 1][b] - du));
    const float lv = ((tv[a][b - 1] - dv) + (tv[a][b + 1] - dv)) + ((tv[a - 1][b] - dv) + (tv[a + 1][b] - dv));
    const size_t p = (size_t)i * n + j;
    const float2 c = coef[p];
    const float a11 = G.c1 - c.x, a21 = c.x - G.B, a22 = G.invdt + c.y;
    const float ou = __fmaf_rn(-c.y, dv, __fmaf_rn(-G.duh, lu, a11 * du));
    const float ov = __fmaf_rn(a22, dv, __fmaf_rn(a21, du, -G.dvh * lv));
    out[p] = f32_to_f64(ou);
    out[nn + p] = f32_to_f64(ov);
}

dim3 b2_grid(int n) {
    const unsigned gx = (unsigned)((n + 31) / 32);
    const unsigned rows = (unsigned)((n + 7) / 8);
    const unsigned gy = std::max(1u, std::min(rows, (unsigned)kMaxRedBlocks / gx));
    return dim3(gx, gy);
}

// The same product from an FP32 d (the multigrid's output): no conversion, so no shared-memory
// tile — neighbours come through L1; the arithmetic is k_b2_jvp32's, operation for operation.  OT =
// float stores the FP32 result as it is, OT = double widens it.
template <class OT>
__global__ void __launch_bounds__(256) k_b2_jvp32f(const float2* __restrict__ coef, const float* __restrict__ d,
                                                   OT* __restrict__ out, B2Geom32 G) {
    pdl_wait();
    pdl_trigger();
    const int n = G.n;
    const size_t nn = (size_t)n * n;
    const int j = blockIdx.x * 32 + threadIdx.x;
    if (j >= n) return;
    const int jm = j == 0 ? n - 1 : j - 1, jp = j + 1 == n ? 0 : j + 1;
    for (int i = blockIdx.y * 8 + threadIdx.y; i < n; i += gridDim.y * 8) {
        const int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
        const size_t r = (size_t)i * n, p = r + j;
        const float du = d[p], dv = d[nn + p];
        const float lu = ((d[r + jm] - du) + (d[r + jp] - du)) + ((d[(size_t)im * n + j] - du) + (d[(size_t)ip * n + j] - du));
        const float* e = d + nn;
        const float lv = ((e[r + jm] - dv) + (e[r + jp] - dv)) + ((e[(size_t)im * n + j] - dv) + (e[(size_t)ip * n + j] - dv));
        const float2 c = coef[p];
        const float a11 = G.c1 - c.x, a21 = c.x - G.B, a22 = G.invdt + c.y;
        const float ru = __fmaf_rn(-c.y, dv, __fmaf_rn(-G.duh, lu, a11 * du));
        const float rv = __fmaf_rn(a22, dv, __fmaf_rn(a21, du, -G.dvh * lv));
        if constexpr (sizeof(OT) == 4) {
            out[p] = ru;
            out[nn + p] = rv;
        } else {
            out[p] = f32_to_f64(ru);
            out[nn + p] = f32_to_f64(rv);
        }
    }
}

// ============================================================================== BrussMG2D kernels
template <class T> struct P2;
template <> struct P2<float> { using t = float2; };
template <> struct P2<double> { using t = double2; };

template <class T>
struct Blk {
    T k11, k12, k21, k22;
};

__device__ __forceinline__ Blk<float> load_blk(const float* __restrict__ K, size_t p) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(K) + p);
    return {q.x, q.y, q.z, q.w};
}
__device__ __forceinline__ Blk<double> load_blk(const double* __restrict__ K, size_t p) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(K) + 2 * p);
    const double2 b = __ldg(reinterpret_cast<const double2*>(K) + 2 * p + 1);
    return {a.x, a.y, b.x, b.y};
}
// the same from shared memory (no read-only-cache path)
__device__ __forceinline__ Blk<float> load_blk_s(const float* K, size_t p) {
    const float4 q = reinterpret_cast<const float4*>(K)[p];
    return {q.x, q.y, q.z, q.w};
}
__device__ __forceinline__ Blk<double> load_blk_s(const double* K, size_t p) {
    const double2 a = reinterpret_cast<const double2*>(K)[2 * p];
    const double2 b = reinterpret_cast<const double2*>(K)[2 * p + 1];
    return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void store_blk(float* K, size_t p, const Blk<float>& k) {
    reinterpret_cast<float4*>(K)[p] = make_float4(k.k11, k.k12, k.k21, k.k22);
}
__device__ __forceinline__ void store_blk(double* K, size_t p, const Blk<double>& k) {
    reinterpret_cast<double2*>(K)[2 * p] = make_double2(k.k11, k.k12);
    reinterpret_cast<double2*>(K)[2 * p + 1] = make_double2(k.k21, k.k22);
}

template <class T>
__device__ __forceinline__ typename P2<T>::t ld2(const T* a, size_t p) {
    return reinterpret_cast<const typename P2<T>::t*>(a)[p];
}
template <class T>
__device__ __forceinline__ void st2(T* a, size_t p, T u, T v) {
    typename P2<T>::t q;
    q.x = u;
    q.y = v;
    reinterpret_cast<typename P2<T>::t*>(a)[p] = q;
}

// Point-block Gauss-Seidel update: (K + 4 diag(s_u, s_v)) (u, v) = (b_u + s_u S_u, b_v + s_v S_v),
// S = ((W + E) + S) + N, by Cramer's rule with two divisions.
template <class T>
__device__ __forceinline__ void block_update(const Blk<T>& k, T su, T sv, T su4, T sv4, T bu, T bv, T Su, T Sv,
                                             T& u, T& v) {
    const T ru = bu + su * Su;
    const T rv = bv + sv * Sv;
    const T m11 = k.k11 + su4, m22 = k.k22 + sv4;
    const T det = m11 * m22 - k.k12 * k.k21;
    u = (m22 * ru - k.k12 * rv) / det;
    v = (m11 * rv - k.k21 * ru) / det;
}

// One level's constants in the multigrid's precision, formed on the host: a kernel converting
// doubles per thread would spend GB300's narrow FP64 pipe on it (a few FP64 instructions per
// thread bound a one-point-per-thread FP32 pass).
template <class T>
struct LvlArgs {
    int n;
    T su, sv, su4, sv4;  // s_u = D_u h^-2, s_v, 4 s_u, 4 s_v
};

// FP64 <-> T without the FP64 pipe for T = float (integer-path conversions, same rounding).
template <class T> __device__ __forceinline__ T from_f64(double x);
template <> __device__ __forceinline__ float from_f64<float>(double x) { return f64_to_f32(x); }
template <> __device__ __forceinline__ double from_f64<double>(double x) { return x; }
// a right-hand side read as FP64 or as FP32 into the level type
template <class T> __device__ __forceinline__ T from_in(double x) { return from_f64<T>(x); }
template <class T> __device__ __forceinline__ T from_in(float x) {
    if constexpr (sizeof(T) == 4) return x;
    else return f32_to_f64(x);
}
__device__ __forceinline__ double to_f64(float x) { return f32_to_f64(x); }
__device__ __forceinline__ double to_f64(double x) { return x; }

// Storage index of point (i, j) of an n x n level (n even): colour-split, each colour's points in
// row-major order, colour (i + j) & 1 first-half / second-half — a colour pass then reads and
// writes only whole cache lines of the colours it touches.  The four neighbours of a point are all
// of the other colour, in its rows i and i +- 1 at column index j/2 or j/2 +- 1.
__device__ __forceinline__ size_t pidx(int n, int i, int j) {
    const int half = n >> 1;
    return (size_t)((i + j) & 1) * ((size_t)n * half) + (size_t)i * half + (j >> 1);
}

template <class T>
__device__ __forceinline__ void nbr_sums(const T* __restrict__ X, int n, int i, int j, T& Su, T& Sv) {
    const int jm = j == 0 ? n - 1 : j - 1, jp = j + 1 == n ? 0 : j + 1;
    const int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
    const auto w = ld2(X, pidx(n, i, jm)), e = ld2(X, pidx(n, i, jp)), s = ld2(X, pidx(n, im, j)),
               nn = ld2(X, pidx(n, ip, j));
    Su = ((w.x + e.x) + s.x) + nn.x;
    Sv = ((w.y + e.y) + s.y) + nn.y;
}

enum { kBPassNormal = 0, kBPassFirst = 1, kBPassLast = 2 };

// One colour of red-black point-block Gauss-Seidel on one level.  Thread (jj, i) owns the pair
// of row i's points 2jj and 2jj + 1 (one of each colour) and updates the one of this colour; a warp
// covers 32 consecutive points of one colour.
//  Normal: x_c updated from the other colour.
//  First (colour 0, x = 0 before the pass): x_0 = block^-1 b (neighbour sums are zeros); x_1 is left as it is,
//    as the colour-1 pass that follows writes all of it and reads none;
//    on the finest level the right-hand side is read from r (FP64 planes) and stored as b.
//  Last (finest level, colour 0, the cycle's final pass): also writes z (FP64 planes) for both points,
//    or, for an FP32 consumer, the same values as FP32 planes z32.
template <class T, int MODE, class RT = double>
__global__ void __launch_bounds__(256) k_bmg_pass(T* __restrict__ X, T* __restrict__ Bv, const T* __restrict__ K,
                                                  LvlArgs<T> L, int colour, const RT* __restrict__ r64,
                                                  double* __restrict__ z64, float* __restrict__ z32 = nullptr) {
    pdl_wait();
    pdl_trigger();
    const int n = L.n;
    const int jj = blockIdx.x * 32 + threadIdx.x;
    const int i = blockIdx.y * 8 + threadIdx.y;
    if (i >= n || 2 * jj >= n) return;
    const T su = L.su, sv = L.sv, su4 = L.su4, sv4 = L.sv4;
    const int j = 2 * jj + ((i + colour) & 1);
    const int jo = 2 * jj + 1 - ((i + colour) & 1);
    const size_t p = pidx(n, i, j), po = pidx(n, i, jo);                // level storage
    const size_t pn = (size_t)i * n + j, pon = (size_t)i * n + jo;      // r and z: natural planes
    const size_t nn = (size_t)n * n;
    T bu, bv;
    if (MODE == kBPassFirst && r64) {
        bu = from_in<T>(r64[pn]);
        bv = from_in<T>(r64[nn + pn]);
        st2(Bv, p, bu, bv);
        st2(Bv, po, from_in<T>(r64[pon]), from_in<T>(r64[nn + pon]));
    } else {
        const auto b = ld2(Bv, p);
        bu = b.x;
        bv = b.y;
    }
    T Su, Sv;
    if (MODE == kBPassFirst) {
        Su = T(0);
        Sv = T(0);
    } else {
        nbr_sums(X, n, i, j, Su, Sv);
    }
    T u, v;
    block_update(load_blk(K, p), su, sv, su4, sv4, bu, bv, Su, Sv, u, v);
    st2(X, p, u, v);
    if (MODE == kBPassLast) {
        const auto o = ld2(X, po);
        if (z64) {
            z64[pn] = to_f64(u);
            z64[nn + pn] = to_f64(v);
            z64[pon] = to_f64(o.x);
            z64[nn + pon] = to_f64(o.y);
        }
        if constexpr (sizeof(T) == 4) {
            if (z32) {  // or the values unwidened, for an FP32 consumer
                z32[pn] = u;
                z32[nn + pn] = v;
                z32[pon] = o.x;
                z32[nn + pon] = o.y;
            }
        }
    }
}

// Residual r = b - (K x - diag(s) (S - 4x)) of one level at point (i, j).
template <class T, class P>
__device__ __forceinline__ void resid_value(const Blk<T>& k, P x, P bb, T Su, T Sv, T su, T sv, T& ru, T& rv) {
    ru = bb.x - ((k.k11 * x.x + k.k12 * x.y) + su * (T(4) * x.x - Su));
    rv = bb.y - ((k.k21 * x.x + k.k22 * x.y) + sv * (T(4) * x.y - Sv));
}
template <class T, bool SMEM_K = false>
__device__ __forceinline__ void resid_at(const T* X, const T* Bv, const T* K, int n, int i, int j, T su, T sv, T& ru,
                                         T& rv) {
    const size_t p = pidx(n, i, j);
    const auto x = ld2(X, p);
    const auto bb = ld2(Bv, p);
    const Blk<T> k = SMEM_K ? load_blk_s(K, p) : load_blk(K, p);
    T Su, Sv;
    nbr_sums(X, n, i, j, Su, Sv);
    resid_value(k, x, bb, Su, Sv, su, sv, ru, rv);
}

// 9-point full weighting ((4c + 2((W + E) + (S + N))) + (((SW + SE) + NW) + NE)) / 16; S is row i-1.
template <class T>
__device__ __forceinline__ T fw9(T c, T w, T e, T s, T n, T sw, T se, T nw, T ne) {
    const T edge = (w + e) + (s + n);
    const T corner = ((sw + se) + nw) + ne;
    return ((T(4) * c + T(2) * edge) + corner) * T(0.0625);
}

// Residual of the finest-level points that a 16 x 16 tile of coarse points covers (33 x 33,
// periodic), kept in shared memory, then full weighting into the coarse right-hand side: FP64's restriction, bound
// by the FP64 pipe (1.06 residuals formed a point; the march below forms 1.1 to 1.5: 278 us against 239 on 2048^2,
// 20 against 12 on 128^2).
template <class T>
__global__ void __launch_bounds__(256) k_bmg_restrict(const T* __restrict__ X, const T* __restrict__ Bv,
                                                      const T* __restrict__ K, LvlArgs<T> L, T* __restrict__ Bc) {
    pdl_wait();
    pdl_trigger();
    constexpr int TS = 16, FS = 2 * TS + 1;
    __shared__ T su_s[FS][FS + 1], sv_s[FS][FS + 1];
    const int nf = L.n, nc = nf / 2;
    const int I0 = blockIdx.y * TS, J0 = blockIdx.x * TS;
    const int tid = threadIdx.y * TS + threadIdx.x;
    const T su = L.su, sv = L.sv;
    for (int idx = tid; idx < FS * FS; idx += TS * TS) {
        const int a = idx / FS, b = idx - a * FS;
        const int fi = (2 * I0 - 1 + a + nf) % nf, fj = (2 * J0 - 1 + b + nf) % nf;
        resid_at(X, Bv, K, nf, fi, fj, su, sv, su_s[a][b], sv_s[a][b]);
    }
    __syncthreads();
    const int I = I0 + threadIdx.y, J = J0 + threadIdx.x;
    if (I >= nc || J >= nc) return;
    const int a = 2 * threadIdx.y + 1, b = 2 * threadIdx.x + 1;
    auto fw = [a, b](const T (*f)[FS + 1]) {
        return fw9(f[a][b], f[a][b - 1], f[a][b + 1], f[a - 1][b], f[a + 1][b], f[a - 1][b - 1], f[a - 1][b + 1],
                   f[a + 1][b - 1], f[a + 1][b + 1]);
    };
    st2(Bc, pidx(nc, I, J), fw(su_s), fw(sv_s));
}

// FP32's restriction: the residual of a level, full-weighted into the next level's right-hand side.  FIRST_X: also
// that level's first smoothing pass (colour 0 from x = 0), where it is a launched level with a coarser one below: the
// pass reads nothing but b and K of its own point, so its launch and its reading of b go.
// Bound by L2 and HBM traffic (2048^2 FP32: x, b and K once are 134 MB).  A warp owns 31 coarse columns (lane 0 is
// the column before them) and marches `rows` coarse rows: each step forms the residuals of the fine points
// (2I + {0, 1}, 2J + {0, 1}) of its coarse point from 12 loaded pairs, takes those of the column before from the lane
// to the left and those of the row before from its last step.  No shared memory and no barrier, and all of a step's
// loads independent.  The tile
// form's five rounds of points a block, with two integer divisions a point, took 34.2 us on 2048^2 and 10.0 on
// 1024^2, and the pass after it 6.3 and 1.8: 33.0 and 7.2 for both.
template <class T, bool FIRST_X>
__global__ void __launch_bounds__(128) k_bmg_restrict_march(const T* __restrict__ X, const T* __restrict__ Bv,
                                                            const T* __restrict__ K, LvlArgs<T> L, int rows,
                                                            T* __restrict__ Bc, const T* __restrict__ Kc,
                                                            T* __restrict__ Xc, LvlArgs<T> Lc) {
    using P = typename P2<T>::t;
    pdl_wait();
    pdl_trigger();
    const int nf = L.n, nc = nf / 2;
    const int lane = threadIdx.x;
    const int Jr = (int)blockIdx.x * 31 + lane - 1;
    const int J = Jr < 0 ? nc - 1 : Jr < nc ? Jr : Jr - nc < nc ? Jr - nc : 0;  // lanes past the grid repeat columns
    const bool owner = lane >= 1 && Jr < nc;
    const int Jm = J == 0 ? nc - 1 : J - 1, Jp = J + 1 == nc ? 0 : J + 1;
    const int I0 = ((int)blockIdx.y * 4 + (int)threadIdx.y) * rows, I1 = min(I0 + rows, nc);
    if (I0 >= nc) return;  // whole warps
    const T su = L.su, sv = L.sv;
    // the colour halves of x, b and K, rows of nc points: (i, j) of colour 0 / 1 at i nc + j / 2
    const size_t h = (size_t)nf * nc;
    P p10, p11;  // the residuals of the row before: at (2I - 1, 2J) and (2I - 1, 2J + 1)
    {
        const int i = 2 * (I0 == 0 ? nc - 1 : I0 - 1) + 1;
        resid_at(X, Bv, K, nf, i, 2 * J, su, sv, p10.x, p10.y);
        resid_at(X, Bv, K, nf, i, 2 * J + 1, su, sv, p11.x, p11.y);
    }
    for (int I = I0; I < I1; ++I) {
        const int im = I == 0 ? nf - 1 : 2 * I - 1, ip = I + 1 == nc ? 0 : 2 * I + 2;
        const size_t q0 = (size_t)(2 * I) * nc, q1 = q0 + nc, qm = (size_t)im * nc + J, qp = (size_t)ip * nc + J;
        const size_t q = pidx(nc, I, J);
        const bool first = FIRST_X && ((I + J) & 1) == 0;
        Blk<T> kc{};
        if (first) kc = load_blk(Kc, q);
        const auto x00 = ld2(X, q0 + J), x01 = ld2(X, h + q0 + J), x10 = ld2(X, h + q1 + J), x11 = ld2(X, q1 + J);
        const auto w00 = ld2(X, h + q0 + Jm), w10 = ld2(X, q1 + Jm), e01 = ld2(X, q0 + Jp), e11 = ld2(X, h + q1 + Jp);
        const auto s00 = ld2(X, h + qm), s01 = ld2(X, qm), n10 = ld2(X, qp), n11 = ld2(X, h + qp);
        const auto b00 = ld2(Bv, q0 + J), b01 = ld2(Bv, h + q0 + J), b10 = ld2(Bv, h + q1 + J), b11 = ld2(Bv, q1 + J);
        P r00, r01, r10, r11;
        resid_value(load_blk(K, q0 + J), x00, b00, ((w00.x + x01.x) + s00.x) + x10.x,
                    ((w00.y + x01.y) + s00.y) + x10.y, su, sv, r00.x, r00.y);
        resid_value(load_blk(K, h + q0 + J), x01, b01, ((x00.x + e01.x) + s01.x) + x11.x,
                    ((x00.y + e01.y) + s01.y) + x11.y, su, sv, r01.x, r01.y);
        resid_value(load_blk(K, h + q1 + J), x10, b10, ((w10.x + x11.x) + x00.x) + n10.x,
                    ((w10.y + x11.y) + x00.y) + n10.y, su, sv, r10.x, r10.y);
        resid_value(load_blk(K, q1 + J), x11, b11, ((x10.x + e11.x) + x01.x) + n11.x,
                    ((x10.y + e11.y) + x01.y) + n11.y, su, sv, r11.x, r11.y);
        auto left = [](P a) {
            a.x = __shfl_up_sync(0xffffffffu, a.x, 1);
            a.y = __shfl_up_sync(0xffffffffu, a.y, 1);
            return a;
        };
        const P w = left(r01), nw = left(r11), sw = left(p11);
        const T bu = fw9(r00.x, w.x, r01.x, p10.x, r10.x, sw.x, p11.x, nw.x, r11.x);
        const T bv = fw9(r00.y, w.y, r01.y, p10.y, r10.y, sw.y, p11.y, nw.y, r11.y);
        if (owner) {
            st2(Bc, q, bu, bv);
            if (first) {
                T u, v;
                block_update(kc, Lc.su, Lc.sv, Lc.su4, Lc.sv4, bu, bv, T(0), T(0), u, v);
                st2(Xc, q, u, v);
            }
        }
        p10 = r10;
        p11 = r11;
    }
}

// The coarse rows a warp of k_bmg_restrict_march marches: as many (up to 8) as leave 24 warps an SM.
int bmg_march_rows(int nc, int sm_count) {
    const int most = (int)((size_t)nc * ((nc + 30) / 31) / ((size_t)sm_count * 24));
    return std::max(1, std::min(8, most));
}

// The bilinear periodic interpolation of x_coarse at the fine point (2I + 1, 2J + 1), from the four coarse points
// (I, J), (I + 1, J), (I, J + 1), (I + 1, J + 1).
template <class P>
__device__ __forceinline__ P interp11(P c00, P c10, P c01, P c11) {
    using T = decltype(c00.x);
    P r;
    r.x = T(0.25) * (((c00.x + c10.x) + c01.x) + c11.x);
    r.y = T(0.25) * (((c00.y + c10.y) + c01.y) + c11.y);
    return r;
}
template <class P>
__device__ __forceinline__ P add2(P a, P b) {
    P r;
    r.x = a.x + b.x;
    r.y = a.y + b.y;
    return r;
}

// x_fine += the interpolation of x_coarse at the fine points (2I, 2J) and (2I + 1, 2J + 1): those of colour 0.
// The first post-smoothing pass writes every colour-1 point and reads none of them, so they take no correction.
template <class T>
__device__ __forceinline__ void prolong_point(const T* Xc, int nc, int I, int J, T* Xf) {
    const int I1 = I + 1 == nc ? 0 : I + 1, J1 = J + 1 == nc ? 0 : J + 1;
    const auto c00 = ld2(Xc, pidx(nc, I, J)), c10 = ld2(Xc, pidx(nc, I1, J));
    const auto c01 = ld2(Xc, pidx(nc, I, J1)), c11 = ld2(Xc, pidx(nc, I1, J1));
    const size_t f00 = (size_t)(2 * I) * nc + J, f11 = f00 + nc;
    const auto x00 = add2(ld2(Xf, f00), c00), x11 = add2(ld2(Xf, f11), interp11(c00, c10, c01, c11));
    st2(Xf, f00, x00.x, x00.y);
    st2(Xf, f11, x11.x, x11.y);
}

template <class T>
__global__ void __launch_bounds__(256) k_bmg_prolong(const T* __restrict__ Xc, int nc, T* __restrict__ Xf) {
    pdl_wait();
    pdl_trigger();
    const int J = blockIdx.x * 32 + threadIdx.x;
    const int I = blockIdx.y * 8 + threadIdx.y;
    if (I >= nc || J >= nc) return;
    prolong_point(Xc, nc, I, J, Xf);
}

// The prolongation and the first post-smoothing pass (colour 1) of a level in one kernel (FP32; in FP64 its
// repeated interpolations and two serial block updates a thread cost more than the launch: 9.1 us against 3.1 + 3.6
// on 128^2, 219 against 49 + 144 on 2048^2).  The pass reads the
// corrected colour-0 points and writes the colour-1 points; the pass after it writes every colour-0 point and reads
// none of them: the corrected values need not be stored at all.  Thread (x, y) owns coarse point (I, J) and updates
// the fine points (2I, 2J + 1) and (2I + 1, 2J) from their six colour-0 neighbours, corrected from eight coarse
// points as they are read.
// Bound by L2 and HBM traffic, as the passes are; the prolongation by itself read and wrote all of x again, and
// cost its launch on the smaller levels: 2048^2 12.1 + 13.2 us -> 19.8, 1024^2 2.7 + 3.5 -> 4.5.
template <class T>
__global__ void __launch_bounds__(256) k_bmg_prolong_pass(const T* __restrict__ Xc, T* __restrict__ X,
                                                          const T* __restrict__ Bv, const T* __restrict__ K,
                                                          LvlArgs<T> L) {
    pdl_wait();
    pdl_trigger();
    const int nc = L.n / 2;
    const int J = blockIdx.x * 32 + threadIdx.x;
    const int I = blockIdx.y * 8 + threadIdx.y;
    if (I >= nc || J >= nc) return;
    const int Im = I == 0 ? nc - 1 : I - 1, Ip = I + 1 == nc ? 0 : I + 1;
    const int Jm = J == 0 ? nc - 1 : J - 1, Jp = J + 1 == nc ? 0 : J + 1;
    const auto c00 = ld2(Xc, pidx(nc, I, J)), c10 = ld2(Xc, pidx(nc, Ip, J));
    const auto c01 = ld2(Xc, pidx(nc, I, Jp)), c11 = ld2(Xc, pidx(nc, Ip, Jp));
    const auto cm0 = ld2(Xc, pidx(nc, Im, J)), cm1 = ld2(Xc, pidx(nc, Im, Jp));
    const auto c0m = ld2(Xc, pidx(nc, I, Jm)), c1m = ld2(Xc, pidx(nc, Ip, Jm));
    const size_t q0 = (size_t)(2 * I) * nc, q1 = q0 + nc;
    // the corrected colour-0 points: own (0, 0) and (1, 1), (0, 0) of the cells after it in J and in I, (1, 1) of
    // the cells before it in I and in J
    const auto x00 = add2(ld2(X, q0 + J), c00), x11 = add2(ld2(X, q1 + J), interp11(c00, c10, c01, c11));
    const auto xe = add2(ld2(X, q0 + Jp), c01), xn = add2(ld2(X, (size_t)(2 * Ip) * nc + J), c10);
    const auto xs = add2(ld2(X, (size_t)(2 * Im + 1) * nc + J), interp11(cm0, c00, cm1, c01));
    const auto xw = add2(ld2(X, q1 + Jm), interp11(c0m, c1m, c00, c10));
    const size_t p01 = (size_t)L.n * nc + q0 + J, p10 = p01 + nc;
    const auto b01 = ld2(Bv, p01), b10 = ld2(Bv, p10);
    T u, v;
    block_update(load_blk(K, p01), L.su, L.sv, L.su4, L.sv4, b01.x, b01.y, ((x00.x + xe.x) + xs.x) + x11.x,
                 ((x00.y + xe.y) + xs.y) + x11.y, u, v);
    st2(X, p01, u, v);
    block_update(load_blk(K, p10), L.su, L.sv, L.su4, L.sv4, b10.x, b10.y, ((xw.x + x11.x) + x00.x) + xn.x,
                 ((xw.y + x11.y) + x00.y) + xn.y, u, v);
    st2(X, p10, u, v);
}

// The middle levels of the FP32 cycle (kBTileTail < n <= kBTileTop below the finest, a coarser one below) in two
// kernels each, one on the way down (pre-smoothing from x = 0, residual, restriction) and one on the way up
// (prolongation, post-smoothing).  A block owns T x T coarse points and the fine points (2I + {0, 1}, 2J + {0, 1}) of
// them, and runs every pass on a region that shrinks by a point on each side a pass: it computes the points around its
// own again instead of waiting for other blocks.  Thread (i, jj) of the region, in linear order, holds b and K of a
// pair of neighbouring points; x is in shared memory.  x goes down in one array and comes up in another, as the blocks
// around read it.  The arithmetic is the launched kernels' operation for operation.
// Bound by the latency of a pass and its barrier: 4.2 + 3.0 us on 256^2, 2.4 + 2.1 on 32^2, for eight launches a level
// (256^2 15 us) or 20 us of the one-CTA tail (64^2).  512^2 needs two waves of blocks and stays launched.
constexpr int kBTileTop = 256, kBTileTail = 16;
struct BTile {
    LvlArgs<float> L;
    int T, S, np, sweeps;  // S x S points of the region, np = (S + 1) / 2 pairs a row
};
inline BTile btile(const LvlArgs<float>& L, int T, int sweeps, bool down) {
    const int S = 2 * T + 4 * sweeps + (down ? 1 : 0);
    return BTile{L, T, S, (S + 1) / 2, sweeps};
}
inline int btile_threads(const BTile& t) { return (t.S * t.np + 31) / 32 * 32; }
inline size_t btile_smem(const BTile& t) {
    return ((size_t)t.S * t.S + (size_t)(2 * t.T + 1) * (2 * t.T + 1)) * sizeof(float2);
}
// T of a level, 0 where the tiled kernels do not take it: the smallest whose blocks all have an SM to themselves.
inline int btile_size(int n, int pre, int post, int sm_count) {
    if (n <= kBTileTail || n > kBTileTop || pre > 3 || post > 3) return 0;
    const int nc = n / 2;
    int T = 1;
    while (((nc + T - 1) / T) * ((nc + T - 1) / T) > sm_count) ++T;
    const LvlArgs<float> L{};
    return std::max(btile_threads(btile(L, T, pre, true)), btile_threads(btile(L, T, post, false))) <= 1024 ? T : 0;
}

__device__ __forceinline__ int wrap(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

// ((W + E) + S) + N around a point of the region
__device__ __forceinline__ float2 btile_sum(const float2* X, int S) {
    const float2 w = X[-1], e = X[1], s = X[-S], n = X[S];
    return make_float2(((w.x + e.x) + s.x) + n.x, ((w.y + e.y) + s.y) + n.y);
}

extern __shared__ __align__(16) float2 btile_smem_x[];

__global__ void __launch_bounds__(1024) k_btile_down(const float* __restrict__ Bv, const float* __restrict__ K,
                                                     float* __restrict__ Y, float* __restrict__ Bc,
                                                     const __grid_constant__ BTile t) {
    float2* X = btile_smem_x;        // S^2
    float2* R = X + t.S * t.S;       // (2T + 1)^2: rows and columns 2 C0 - 1 .. 2 C0 + 2T - 1
    const int n = t.L.n, nc = n / 2, S = t.S, h = 2 * t.sweeps, rn = 2 * t.T + 1;
    const int C0i = blockIdx.y * t.T, C0j = blockIdx.x * t.T;
    const int ri = (int)threadIdx.x / t.np, rj = 2 * ((int)threadIdx.x - ri * t.np);
    const int i = 2 * C0i - h - 1 + ri, j0 = 2 * C0j - h - 1 + rj;
    const int iw = wrap(i, n);
    float2 b[2];
    Blk<float> k[2];
    bool in[2];
    pdl_wait();
    pdl_trigger();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        in[q] = ri < S && rj + q < S;
        if (!in[q]) continue;
        const size_t p = pidx(n, iw, wrap(j0 + q, n));
        b[q] = ld2(Bv, p);
        k[q] = load_blk(K, p);
    }
    float2* Xp = X + ri * S + rj;
#pragma unroll 1
    for (int p = 0; p < h; ++p) {  // colours 0, 1, 0, 1, ...
        const int q = (i + j0 + p) & 1, c = rj + q;
        if (ri >= p && ri < S - p && c >= p && c < S - p) {
            const float2 s = p == 0 ? make_float2(0.0f, 0.0f) : btile_sum(Xp + q, S);
            float u, v;
            block_update(q ? k[1] : k[0], t.L.su, t.L.sv, t.L.su4, t.L.sv4, q ? b[1].x : b[0].x, q ? b[1].y : b[0].y, s.x,
                         s.y, u, v);
            Xp[q] = make_float2(u, v);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int a = ri - h, c = rj + q - h;
        if (!in[q] || a < 0 || a >= rn || c < 0 || c >= rn) continue;
        const float2 x = Xp[q], s = btile_sum(Xp + q, S);
        float2 r;
        resid_value(k[q], x, b[q], s.x, s.y, t.L.su, t.L.sv, r.x, r.y);
        R[a * rn + c] = r;
        if (a > 0 && c > 0 && i < n && j0 + q < n) st2(Y, pidx(n, i, j0 + q), x.x, x.y);
    }
    __syncthreads();
    const int I = (int)threadIdx.x / t.T, J = (int)threadIdx.x - I * t.T;
    if (I < t.T && C0i + I < nc && C0j + J < nc) {
        const float2* f = R + (2 * I + 1) * rn + 2 * J + 1;
        const float u = fw9(f[0].x, f[-1].x, f[1].x, f[-rn].x, f[rn].x, f[-rn - 1].x, f[-rn + 1].x, f[rn - 1].x,
                            f[rn + 1].x);
        const float v = fw9(f[0].y, f[-1].y, f[1].y, f[-rn].y, f[rn].y, f[-rn - 1].y, f[-rn + 1].y, f[rn - 1].y,
                            f[rn + 1].y);
        st2(Bc, pidx(nc, C0i + I, C0j + J), u, v);
    }
}

__global__ void __launch_bounds__(1024) k_btile_up(const float* __restrict__ Bv, const float* __restrict__ K,
                                                   const float* __restrict__ Y, const float* __restrict__ Xc,
                                                   float* __restrict__ Xo, const __grid_constant__ BTile t) {
    float2* X = btile_smem_x;
    const int n = t.L.n, nc = n / 2, S = t.S, h = 2 * t.sweeps;
    const int ri = (int)threadIdx.x / t.np, rj = 2 * ((int)threadIdx.x - ri * t.np);
    const int i = 2 * (int)blockIdx.y * t.T - h + ri, j0 = 2 * (int)blockIdx.x * t.T - h + rj;
    const int iw = wrap(i, n);
    const bool row = ri < S;  // (S is even: both points of a pair are in the region)
    float2 b[2];
    Blk<float> k[2];
    pdl_wait();
    pdl_trigger();
    float2* Xp = X + ri * S + rj;
    if (row) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const size_t p = pidx(n, iw, wrap(j0 + q, n));
            b[q] = ld2(Bv, p);
            k[q] = load_blk(K, p);
        }
        // the pair's colour-0 point, corrected: (even, even) or (odd, odd)
        const int q = (i + j0) & 1, jw = wrap(j0 + q, n);
        const int I = iw >> 1, J = jw >> 1;
        const float2 x = ld2(Y, pidx(n, iw, jw)), c00 = ld2(Xc, pidx(nc, I, J));
        float2 d = c00;
        if (iw & 1) {
            const int I1 = I + 1 == nc ? 0 : I + 1, J1 = J + 1 == nc ? 0 : J + 1;
            d = interp11(c00, ld2(Xc, pidx(nc, I1, J)), ld2(Xc, pidx(nc, I, J1)), ld2(Xc, pidx(nc, I1, J1)));
        }
        Xp[q] = add2(x, d);
    }
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < h; ++p) {  // colours 1, 0, 1, 0, ...
        const int q = (i + j0 + p + 1) & 1, c = rj + q, e = p + 1;
        if (ri >= e && ri < S - e && c >= e && c < S - e) {
            const float2 s = btile_sum(Xp + q, S);
            float u, v;
            block_update(q ? k[1] : k[0], t.L.su, t.L.sv, t.L.su4, t.L.sv4, q ? b[1].x : b[0].x, q ? b[1].y : b[0].y, s.x,
                         s.y, u, v);
            Xp[q] = make_float2(u, v);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int a = ri - h, c = rj + q - h;
        if (a < 0 || a >= 2 * t.T || c < 0 || c >= 2 * t.T || i >= n || j0 + q >= n) continue;
        st2(Xo, pidx(n, i, j0 + q), Xp[q].x, Xp[q].y);
    }
}

// The coarsest level in one block: x = 0, then `sweeps` red-black sweeps (colour 0, 1).
template <class T>
__global__ void __launch_bounds__(1024) k_bmg_coarsest(T* __restrict__ X, const T* __restrict__ Bv,
                                                       const T* __restrict__ K, LvlArgs<T> L, int sweeps) {
    pdl_wait();
    pdl_trigger();
    const int n = L.n;
    const int nn = n * n;
    const T su = L.su, sv = L.sv, su4 = L.su4, sv4 = L.sv4;
    for (int p = threadIdx.x; p < nn; p += blockDim.x) st2(X, p, T(0), T(0));
    __syncthreads();
    for (int s = 0; s < sweeps; ++s) {
        for (int c = 0; c < 2; ++c) {
            for (int p = threadIdx.x; p < nn; p += blockDim.x) {
                const int i = p / n, j = p - i * n;
                if (((i + j) & 1) != c) continue;
                const size_t q = pidx(n, i, j);
                T Su, Sv, u, v;
                nbr_sums(X, n, i, j, Su, Sv);
                const auto b = ld2(Bv, q);
                block_update(load_blk(K, q), su, sv, su4, sv4, b.x, b.y, Su, Sv, u, v);
                st2(X, q, u, v);
            }
            __syncthreads();
        }
    }
}

// The small levels below the finest (n <= 64 in FP32, n <= 32 in FP64) as one block: every tail
// level's pairs x, b and blocks K live in shared memory (8 n^2 values a level, at most 175 KB), and
// the block runs their whole V-cycle — the same per-point arithmetic as the level kernels, so the
// result is the same to the bit.  desc[k] describes tail level k (k = 0 the finest of them): its
// n, the offset of its x in the shared buffer (b follows at offset + 2 n^2, K at offset + 4 n^2),
// s_u, s_v and its blocks in global memory (copied in at the start).
struct TailLvl {
    int n, off;
    const void* K;
    LvlArgs<double> d;  // the level's constants in FP64 and in FP32 (formed on the host: one SM's
    LvlArgs<float> f;   // FP64 pipe would take tens of microseconds to convert them per pass)
};
constexpr int kBmgTailLevels = 6;  // at most 64, 32, 16, 8, 4
template <class T> __device__ __forceinline__ const LvlArgs<T>& tail_args(const TailLvl& L);
template <> __device__ __forceinline__ const LvlArgs<double>& tail_args<double>(const TailLvl& L) { return L.d; }
template <> __device__ __forceinline__ const LvlArgs<float>& tail_args<float>(const TailLvl& L) { return L.f; }

// The coarsest level of a tail by one warp (n even, n <= 8): x = 0, then `sweeps` red-black sweeps.  A lane holds one
// point of each colour, with its b, K and determinant, and takes its neighbours' values from their lanes; a pass is
// the latency of eight shuffles and a block update.  (With the values in shared memory and the addresses formed again
// each pass, 60 passes on 4 x 4 points made the tail of 16^2 24.5 us; so 15.7.)
template <class T>
__device__ __forceinline__ void tail_coarsest_warp(T* X, int n, const LvlArgs<T>& A, int sweeps) {
    const int half = n / 2, cnt = n * half;
    const int lane = threadIdx.x, idx = lane < cnt ? lane : 0;
    const int i = idx / half, jj = idx - i * half;
    const int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
    const int ls = im * half + jj, ln = ip * half + jj;
    const T* Bv = X + 2 * n * n;
    const T* K = X + 4 * n * n;
    T bu[2], bv[2], m11[2], m22[2], k12[2], k21[2], det[2], xu[2], xv[2];
    int lw[2], le[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const auto b = ld2(Bv, c * cnt + idx);
        const Blk<T> k = load_blk_s(K, c * cnt + idx);
        bu[c] = b.x;
        bv[c] = b.y;
        m11[c] = k.k11 + A.su4;
        m22[c] = k.k22 + A.sv4;
        k12[c] = k.k12;
        k21[c] = k.k21;
        det[c] = m11[c] * m22[c] - k12[c] * k21[c];
        xu[c] = xv[c] = T(0);
        const bool right = (i + c) & 1;  // the point's j is 2jj + 1
        lw[c] = i * half + (right ? jj : jj == 0 ? half - 1 : jj - 1);
        le[c] = i * half + (!right ? jj : jj + 1 == half ? 0 : jj + 1);
    }
    constexpr unsigned all = 0xffffffffu;
#pragma unroll 1
    for (int s = 0; s < sweeps; ++s) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const T ou = xu[c ^ 1], ov = xv[c ^ 1];
            const T Su = ((__shfl_sync(all, ou, lw[c]) + __shfl_sync(all, ou, le[c])) + __shfl_sync(all, ou, ls)) +
                         __shfl_sync(all, ou, ln);
            const T Sv = ((__shfl_sync(all, ov, lw[c]) + __shfl_sync(all, ov, le[c])) + __shfl_sync(all, ov, ls)) +
                         __shfl_sync(all, ov, ln);
            const T ru = bu[c] + A.su * Su, rv = bv[c] + A.sv * Sv;  // block_update's steps
            xu[c] = (m22[c] * ru - k12[c] * rv) / det[c];
            xv[c] = (m11[c] * rv - k21[c] * ru) / det[c];
        }
    }
    if (lane < cnt) {
        st2(X, idx, xu[0], xv[0]);
        st2(X, cnt + idx, xu[1], xv[1]);
    }
    __syncwarp();
}

// threads of the one-CTA tail: 1024 in FP32 (64 registers, no spills), 512 in FP64 (which would spill at 1024)
template <class T>
constexpr int kBmgTailThreads = sizeof(T) == 4 ? 1024 : 512;
template <class T>
__global__ void __launch_bounds__(kBmgTailThreads<T>, 1) k_bmg_tail(const TailLvl* __restrict__ descs, int count, int pre, int post,
                                                     int sweeps, const T* __restrict__ Bin, T* __restrict__ Xout) {
    __shared__ TailLvl desc[kBmgTailLevels];  // (written once, when the hierarchy is made)
    for (int q = threadIdx.x; q < count * (int)(sizeof(TailLvl) / 4); q += blockDim.x)
        reinterpret_cast<int*>(desc)[q] = reinterpret_cast<const int*>(descs)[q];
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char bmg_smem[];
    T* base = reinterpret_cast<T*>(bmg_smem);
    // Levels with n <= 8 (at most 32 points of a colour) are run by warp 0 alone, separated by
    // __syncwarp instead of block barriers; `kw` is the first of them (count if none).
    int kw = count;
    for (int k = 0; k < count; ++k)
        if (desc[k].n <= 8) {
            kw = k;
            break;
        }
    const bool warp0 = threadIdx.x < 32;
    // one colour pass of level L (a copy in registers: from shared memory its constants would be loaded again behind
    // every barrier) by the block, or by warp 0 (small); then the barrier of that group
    auto pass = [&](const TailLvl& L, bool small, int colour, bool first) {
        const int tid = threadIdx.x, nt = small ? 32 : blockDim.x;
        const int n = L.n, half = n / 2;
        T* X = base + L.off;
        const T* Bv = X + 2 * n * n;
        const T* K = X + 4 * n * n;
        const LvlArgs<T>& A = tail_args<T>(L);
        for (int idx = tid; idx < n * half; idx += nt) {
            const int i = idx / half, jj = idx - i * half;
            const int j = 2 * jj + ((i + colour) & 1);
            const size_t p = pidx(n, i, j);
            const auto b = ld2(Bv, p);
            T Su = T(0), Sv = T(0), u, v;
            if (!first) nbr_sums(X, n, i, j, Su, Sv);
            block_update(load_blk_s(K, p), A.su, A.sv, A.su4, A.sv4, b.x, b.y, Su, Sv, u, v);
            st2(X, p, u, v);
        }
        if (small) __syncwarp();
        else __syncthreads();
    };
    // residual of level k, full-weighted into the right-hand side of level k + 1
    auto restrict_to = [&](int k) {
        const bool small = k + 1 >= kw && k >= kw;
        const int tid = threadIdx.x, nt = small ? 32 : blockDim.x;
        const TailLvl L = desc[k], C = desc[k + 1];
        const int nf = L.n, nc = C.n;
        const T* X = base + L.off;
        const T* Bv = X + 2 * nf * nf;
        const T* K = X + 4 * nf * nf;
        T* Bc = base + C.off + 2 * nc * nc;
        const T su = tail_args<T>(L).su, sv = tail_args<T>(L).sv;
        for (int idx = tid; idx < nc * nc; idx += nt) {
            const int I = idx / nc, J = idx - I * nc;
            const int i = 2 * I, j = 2 * J;
            const int im = i == 0 ? nf - 1 : i - 1, ip = i + 1, jm = j == 0 ? nf - 1 : j - 1, jp = j + 1;
            // fw9's sums in its order, accumulated as the residuals are formed (fewer live registers)
            T cu, cv, au, av, bu, bv;
            resid_at<T, true>(X, Bv, K, nf, i, j, su, sv, cu, cv);
            resid_at<T, true>(X, Bv, K, nf, i, jm, su, sv, au, av);
            resid_at<T, true>(X, Bv, K, nf, i, jp, su, sv, bu, bv);
            const T weu = au + bu, wev = av + bv;
            resid_at<T, true>(X, Bv, K, nf, im, j, su, sv, au, av);
            resid_at<T, true>(X, Bv, K, nf, ip, j, su, sv, bu, bv);
            const T edgeu = weu + (au + bu), edgev = wev + (av + bv);
            resid_at<T, true>(X, Bv, K, nf, im, jm, su, sv, au, av);
            resid_at<T, true>(X, Bv, K, nf, im, jp, su, sv, bu, bv);
            T coru = au + bu, corv = av + bv;
            resid_at<T, true>(X, Bv, K, nf, ip, jm, su, sv, au, av);
            coru = coru + au;
            corv = corv + av;
            resid_at<T, true>(X, Bv, K, nf, ip, jp, su, sv, au, av);
            coru = coru + au;
            corv = corv + av;
            st2(Bc, pidx(nc, I, J), ((T(4) * cu + T(2) * edgeu) + coru) * T(0.0625),
                ((T(4) * cv + T(2) * edgev) + corv) * T(0.0625));
        }
        if (small) __syncwarp();
        else __syncthreads();
    };
    auto prolong_from = [&](int k) {  // level k + 1 into level k
        const bool small = k >= kw;
        const int tid = threadIdx.x, nt = small ? 32 : blockDim.x;
        const int nc = desc[k + 1].n;
        const T* Xc = base + desc[k + 1].off;
        T* Xf = base + desc[k].off;
        for (int idx = tid; idx < nc * nc; idx += nt) prolong_point(Xc, nc, idx / nc, idx % nc, Xf);
        if (small) __syncwarp();
        else __syncthreads();
    };
    auto down = [&](int k) {
        const TailLvl L = desc[k];
        const bool small = k >= kw;
        pass(L, small, 0, true);
        pass(L, small, 1, false);
        for (int s = 1; s < pre; ++s) {
            pass(L, small, 0, false);
            pass(L, small, 1, false);
        }
        restrict_to(k);
    };
    auto up = [&](int k) {
        prolong_from(k);
        const TailLvl L = desc[k];
        const bool small = k >= kw;
        for (int s = 0; s < post; ++s) {
            pass(L, small, 1, false);
            pass(L, small, 0, false);
        }
    };
    auto coarsest = [&]() {
        const int kc = count - 1, n = desc[kc].n;
        T* X = base + desc[kc].off;
        if (kc >= kw) {  // n <= 8, warp 0: a lane has one point of each colour
            tail_coarsest_warp(X, n, tail_args<T>(desc[kc]), sweeps);
            return;
        }
        for (int q = threadIdx.x; q < 2 * n * n; q += blockDim.x) X[q] = T(0);
        __syncthreads();
        const TailLvl L = desc[kc];
        for (int s = 0; s < sweeps; ++s) {
            pass(L, false, 0, false);
            pass(L, false, 1, false);
        }
    };
    {
        const int n0 = desc[0].n;
        T* B0 = base + desc[0].off + 2 * n0 * n0;
        for (int q = threadIdx.x; q < 2 * n0 * n0; q += blockDim.x) B0[q] = Bin[q];
        for (int k = 0; k < count; ++k) {
            const int nk = desc[k].n;
            const float4* src = static_cast<const float4*>(desc[k].K);
            float4* dst = reinterpret_cast<float4*>(base + desc[k].off + 4 * nk * nk);
            const int n16 = (int)(4 * (size_t)nk * nk * sizeof(T) / 16);
            for (int q = threadIdx.x; q < n16; q += blockDim.x) dst[q] = __ldg(src + q);
        }
    }
    __syncthreads();
    // block-wide levels down to kw (restricting into kw last)
    for (int k = 0; k + 1 < count && k < kw; ++k) down(k);
    if (kw < count) {
        // the warp-sized levels: the rest of the V-cycle from level kw down and back up, warp 0 only
        if (warp0) {
            for (int k = kw; k + 1 < count; ++k) down(k);
            coarsest();
            for (int k = count - 2; k >= kw; --k) up(k);
        }
        __syncthreads();
    } else {
        coarsest();
    }
    for (int k = (kw < count - 1 ? kw : count - 1) - 1; k >= 0; --k) up(k);
    const int n0 = desc[0].n;
    const T* X0 = base + desc[0].off;
    for (int q = threadIdx.x; q < 2 * n0 * n0; q += blockDim.x) Xout[q] = X0[q];
}

// K at the finest level from the FP64 state: [[1/dt + B + 1 - 2uv, -u^2], [2uv - B, 1/dt + u^2]];
// in FP64 for the FP64 multigrid, in FP32 from the rounded state for the FP32 one (a preconditioner
// needs no more, and FP64 arithmetic would bound the kernel).
__device__ __forceinline__ void kfine_point(double u, double v, double c1, double c2, double B, Blk<double>& k) {
    k.k11 = c1 - (2.0 * u) * v;
    k.k12 = -(u * u);
    k.k21 = (2.0 * u) * v - B;
    k.k22 = c2 + u * u;
}
__device__ __forceinline__ void kfine_point(double u, double v, float c1, float c2, float B, Blk<float>& k) {
    const float u32 = f64_to_f32(u), v32 = f64_to_f32(v);
    const float uv2 = (2.0f * u32) * v32, uu = u32 * u32;
    k.k11 = c1 - uv2;
    k.k12 = -uu;
    k.k21 = uv2 - B;
    k.k22 = c2 + uu;
}

// c1 = 1/dt + (B + 1), c2 = 1/dt and B in the multigrid's precision (rounded on the host)
template <class T>
__global__ void __launch_bounds__(256) k_bmg_kfine(const double* __restrict__ w, int n, T c1, T c2, T B,
                                                   T* __restrict__ K) {
    pdl_wait();
    pdl_trigger();
    const size_t nn = (size_t)n * n;
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nn) return;
    const int i = (int)(p / n), j = (int)(p - (size_t)i * n);
    Blk<T> k;
    kfine_point(w[p], w[nn + p], c1, c2, B, k);
    store_blk(K, pidx(n, i, j), k);
}

// Full weighting of the four block components to the next coarser level.
template <class T>
__global__ void __launch_bounds__(256) k_bmg_krestrict(const T* __restrict__ Kf, int nf, T* __restrict__ Kc) {
    pdl_wait();
    pdl_trigger();
    const int nc = nf / 2;
    const int J = blockIdx.x * 32 + threadIdx.x;
    const int I = blockIdx.y * 8 + threadIdx.y;
    if (I >= nc || J >= nc) return;
    const int i = 2 * I, j = 2 * J;
    const int im = i == 0 ? nf - 1 : i - 1, ip = i + 1, jm = j == 0 ? nf - 1 : j - 1, jp = j + 1;
    auto at = [Kf, nf](int a, int b) { return load_blk(Kf, pidx(nf, a, b)); };
    const Blk<T> c = at(i, j), w = at(i, jm), e = at(i, jp), s = at(im, j), nth = at(ip, j);
    const Blk<T> sw = at(im, jm), se = at(im, jp), nw = at(ip, jm), ne = at(ip, jp);
    auto fw = [](T ctr, T w_, T e_, T s_, T n_, T sw_, T se_, T nw_, T ne_) {
        const T edge = (w_ + e_) + (s_ + n_);
        const T corner = ((sw_ + se_) + nw_) + ne_;
        return ((T(4) * ctr + T(2) * edge) + corner) * T(0.0625);
    };
    Blk<T> o;
    o.k11 = fw(c.k11, w.k11, e.k11, s.k11, nth.k11, sw.k11, se.k11, nw.k11, ne.k11);
    o.k12 = fw(c.k12, w.k12, e.k12, s.k12, nth.k12, sw.k12, se.k12, nw.k12, ne.k12);
    o.k21 = fw(c.k21, w.k21, e.k21, s.k21, nth.k21, sw.k21, se.k21, nw.k21, ne.k21);
    o.k22 = fw(c.k22, w.k22, e.k22, s.k22, nth.k22, sw.k22, se.k22, nw.k22, ne.k22);
    store_blk(Kc, pidx(nc, I, J), o);
}

// FP64 planes <-> interleaved level pairs (used only when the finest level is also the coarsest).
template <class T, class RT = double>
__global__ void k_bmg_in(const RT* __restrict__ r, int n, T* __restrict__ B) {
    pdl_wait();
    pdl_trigger();
    const size_t nn = (size_t)n * n;
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nn) return;
    const int i = (int)(p / n), j = (int)(p - (size_t)i * n);
    st2(B, pidx(n, i, j), from_in<T>(r[p]), from_in<T>(r[nn + p]));
}
template <class T>
__global__ void k_bmg_out(const T* __restrict__ X, int n, double* __restrict__ z) {
    pdl_wait();
    pdl_trigger();
    const size_t nn = (size_t)n * n;
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nn) return;
    const int i = (int)(p / n), j = (int)(p - (size_t)i * n);
    const auto x = ld2(X, pidx(n, i, j));
    z[p] = to_f64(x.x);
    z[nn + p] = to_f64(x.y);
}

constexpr int kBmgCoarsestSweeps = 30;
constexpr int kBmgOneBlockPoints = 4096;
constexpr int kBmgTailMaxN = 64;  // levels this small (below the finest; half in FP64) run in the one-block tail
static_assert((4 << (kBmgTailLevels - 1)) >= kBmgTailMaxN, "a tail halves down to 4 points a side");

}  // namespace

// ============================================================================== Brusselator1D
Brusselator1D::Brusselator1D(Context& ctx, size_t n, double dt) : NonlinearOp(ctx), n_(n), dt_(dt) {
    if (n == 0 || !(dt > 0.0) || !std::isfinite(dt))
        throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "Brusselator1DStep requires valid n and dt");
    if (n > (size_t)1 << 28) throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "Brusselator1DStep grid too large");
    h_ = 1.0 / (static_cast<double>(n) + 1.0);
    h2inv_ = 1.0 / (h_ * h_);
    // previous state u = 1 + sin(2 pi x), v = 3 at x = (i + 1) h (brusselator1d.hpp:30-37)
    std::vector<double> prev(2 * n);
    const double pi = std::acos(-1.0);
    for (size_t i = 0; i < n; ++i) {
        const double x = (static_cast<double>(i) + 1.0) * h_;
        prev[i] = 1.0 + std::sin(2.0 * pi * x);
        prev[n + i] = 3.0;
    }
    prev_.resize(2 * n);
    NUMA_CUDA(cudaMemcpyAsync(prev_.p, prev.data(), 2 * n * sizeof(double), cudaMemcpyHostToDevice, ctx_.stream));
    ctx_.sync();
}

static B1Geom b1_geom(size_t n, double dt, double h2inv) {
    B1Geom G;
    G.n = (int)n;
    G.invdt = 1.0 / dt;
    G.h2inv = h2inv;
    G.alpha = Brusselator1D::kAlpha;
    G.A = Brusselator1D::kA;
    G.B = Brusselator1D::kB;
    G.base = 1.0 / dt + 2.0 * Brusselator1D::kAlpha * h2inv;
    return G;
}

void Brusselator1D::eval(const double* x, double* out, double*, double* norm_out) {
    launch_pdl(k_b1_eval, (unsigned)((n_ + 255) / 256), 256, 0, ctx_.stream, x, prev_.p, out, b1_geom(n_, dt_, h2inv_));
    ctx_.count_launch();
    ctx_.check_launch("Brusselator1D eval");
    if (norm_out) dev_norm2(ctx_, out, size(), norm_out);
}

void Brusselator1D::jvp_at(const double* x, const double* v, double* out) {
    launch_pdl(k_b1_jvp, (unsigned)((n_ + 255) / 256), 256, 0, ctx_.stream, x, v, out, b1_geom(n_, dt_, h2inv_));
    ctx_.count_launch();
    ctx_.check_launch("Brusselator1D jvp");
}

void Brusselator1D::d2(const double* x, const double*, const double* v, double* out) {
    launch_pdl(k_bruss_d2, (unsigned)((n_ + 255) / 256), 256, 0, ctx_.stream, x, v, out, n_);
    ctx_.count_launch();
    ctx_.check_launch("Brusselator1D d2");
}

void Brusselator1D::blocks(const double* x, double* a) {
    launch_pdl(k_b1_blocks, (unsigned)((n_ + 255) / 256), 256, 0, ctx_.stream, x, a, b1_geom(n_, dt_, h2inv_));
    ctx_.count_launch();
    ctx_.check_launch("Brusselator1D blocks");
}

void brusselator_block_apply(Context& ctx, const double* a, const double* r, double* z, size_t n) {
    launch_pdl(k_b1_block_apply, (unsigned)((n + 255) / 256), 256, 0, ctx.stream, a, r, z, (int)n);
    ctx.count_launch();
    ctx.check_launch("BrusselatorJacobi apply");
}

namespace {
// BrusselatorJacobi (brusselator1d.hpp:194-222): make(x) forms the point blocks at x.
class BrussJacobiProvider final : public Provider {
public:
    explicit BrussJacobiProvider(Brusselator1D& op) : op_(op) { a_.resize(4 * op.grid()); }
    void make(const double* x, const double*) override { op_.blocks(x, a_.p); }
    void apply(const double* r, double* z) override { brusselator_block_apply(op_.ctx(), a_.p, r, z, op_.grid()); }
    int kind() const override { return NUMA_GPU_PRECOND_BRUSS_JACOBI; }

private:
    Brusselator1D& op_;
    DeviceArray<double> a_;
};
}  // namespace

std::unique_ptr<Provider> make_bruss_jacobi_provider(Brusselator1D& op) {
    return std::make_unique<BrussJacobiProvider>(op);
}

// ============================================================================== Brusselator2D
Brusselator2D::Brusselator2D(Context& ctx, size_t n, const numa_brusselator2d_params& p)
    : NonlinearOp(ctx), n_(n), P_(p) {
    if (n < 3 || !(p.dt > 0.0) || !std::isfinite(p.dt) || !(p.Du >= 0.0) || !(p.Dv >= 0.0) || !std::isfinite(p.A) ||
        !std::isfinite(p.B) || !std::isfinite(p.Du) || !std::isfinite(p.Dv))
        throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "Brusselator2D requires n >= 3, dt > 0, D >= 0");
    if (n > 46340) throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "Brusselator2D grid too large");
    prev_.resize(2 * n * n);
    dev_fill(ctx_, prev_.p, 0.0, 2 * n * n);
}

static B2Geom b2_geom(size_t n, const numa_brusselator2d_params& P) {
    B2Geom G;
    G.n = (int)n;
    const double h2inv = static_cast<double>(n) * static_cast<double>(n);
    G.invdt = 1.0 / P.dt;
    G.A = P.A;
    G.B = P.B;
    G.Bp1 = P.B + 1.0;
    G.c1 = G.invdt + (P.B + 1.0);
    G.duh = P.Du * h2inv;
    G.dvh = P.Dv * h2inv;
    return G;
}

void Brusselator2D::set_previous(const double* w) { dev_copy(ctx_, w, prev_.p, size()); }

void Brusselator2D::eval(const double* x, double* out, double*, double* norm_out) {
    int rows = 0;
    const dim3 grid = b2_eval_grid((int)n_, ctx_.sm_count, rows);
    if ((n_ + 30) / 31 * ((n_ + 255) / 256) > (size_t)kMaxRedBlocks)  // (the grid itself stays smaller)
        throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "Brusselator2D grid too large");
    const B2Geom G = b2_geom(n_, P_);
    if (norm_out && fixed_sum_)
        launch_pdl(k_b2_eval<true, true>, grid, dim3(32, 8), 0, ctx_.stream, x, prev_.p, out, G, rows, ctx_.red, norm_out,
                   ctx_.take(norm_out));
    else if (norm_out)
        launch_pdl(k_b2_eval<true>, grid, dim3(32, 8), 0, ctx_.stream, x, prev_.p, out, G, rows, ctx_.red, norm_out,
                   ctx_.take(norm_out));
    else  // an evaluation without the norm (the reference-facing F) keeps the FP64 differences
        launch_pdl(k_b2_eval<false>, grid, dim3(32, 8), 0, ctx_.stream, x, prev_.p, out, G, rows, ctx_.red, nullptr,
                   HostOut{});
    ctx_.count_launch();
    ctx_.check_launch("Brusselator2D eval");
}

void Brusselator2D::bind(const double* x, const double*, int precision) {
    bound_x_ = x;
    bound_precision_ = precision;
    if (precision == NUMA_GPU_FP32) {
        const size_t nn = n_ * n_;
        coef32_.resize(nn);  // one float2 per point
        launch_pdl(k_b2_coef32, (unsigned)((nn + 255) / 256), 256, 0, ctx_.stream, x, nn,
                                                                          reinterpret_cast<float2*>(coef32_.p));
        ctx_.count_launch();
        ctx_.check_launch("Brusselator2D bind");
    }
}

void Brusselator2D::jvp_bound(const double* v, double* out) {
    if (bound_precision_ != NUMA_GPU_FP32) {
        jvp_at(bound_x_, v, out);
        return;
    }
    const B2Geom G = b2_geom(n_, P_);
    const B2Geom32 G32{(int)n_, (float)G.invdt, (float)G.B, (float)G.c1, (float)G.duh, (float)G.dvh};
    const dim3 grid((unsigned)((n_ + 31) / 32), (unsigned)((n_ + 7) / 8));
    launch_pdl(k_b2_jvp32<double>, grid, dim3(32, 8), 0, ctx_.stream, reinterpret_cast<const float2*>(coef32_.p), v, out,
                                                              G32);
    ctx_.count_launch();
    ctx_.check_launch("Brusselator2D jvp32");
}

void Brusselator2D::jvp_bound32(const float* v32, double* out) {
    if (bound_precision_ != NUMA_GPU_FP32)
        throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "Brusselator2D: no FP32 product bound");
    const B2Geom G = b2_geom(n_, P_);
    const B2Geom32 G32{(int)n_, (float)G.invdt, (float)G.B, (float)G.c1, (float)G.duh, (float)G.dvh};
    launch_pdl(k_b2_jvp32f<double>, b2_grid((int)n_), dim3(32, 8), 0, ctx_.stream,
               reinterpret_cast<const float2*>(coef32_.p), v32, out, G32);
    ctx_.count_launch();
    ctx_.check_launch("Brusselator2D jvp32 (fp32 input)");
}

void Brusselator2D::jvp_bound32f(const float* v32, float* out32) {
    if (bound_precision_ != NUMA_GPU_FP32)
        throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "Brusselator2D: no FP32 product bound");
    const B2Geom G = b2_geom(n_, P_);
    const B2Geom32 G32{(int)n_, (float)G.invdt, (float)G.B, (float)G.c1, (float)G.duh, (float)G.dvh};
    launch_pdl(k_b2_jvp32f<float>, b2_grid((int)n_), dim3(32, 8), 0, ctx_.stream,
               reinterpret_cast<const float2*>(coef32_.p), v32, out32, G32);
    ctx_.count_launch();
    ctx_.check_launch("Brusselator2D jvp32 (fp32 input and output)");
}

void Brusselator2D::jvp_at(const double* x, const double* v, double* out) {
    launch_pdl(k_b2_jvp, b2_grid((int)n_), dim3(32, 8), 0, ctx_.stream, x, v, out, b2_geom(n_, P_));
    ctx_.count_launch();
    ctx_.check_launch("Brusselator2D jvp");
}

void Brusselator2D::d2(const double* x, const double*, const double* v, double* out) {
    const size_t nn = n_ * n_;
    launch_pdl(k_bruss_d2, (unsigned)((nn + 255) / 256), 256, 0, ctx_.stream, x, v, out, nn);
    ctx_.count_launch();
    ctx_.check_launch("Brusselator2D d2");
}

// ============================================================================== BrussMG2D
struct BrussMG2D::Level {
    int n;
    double su, sv;
    DeviceArray<double> x, b, k;  // level pairs and blocks in the multigrid's precision
    int T = 0;                    // > 0: run by the tiled kernels, T x T coarse points a block
    DeviceArray<double> y;        // tiled: x on its way down
};

BrussMG2D::BrussMG2D(Context& ctx, size_t n, const numa_brusselator2d_params& p, int precision, int pre, int post)
    : ctx_(ctx), n0_(n), P_(p), precision_(precision), pre_(pre), post_(post) {
    if (n < 4 || n % 2 != 0) throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "BrussMG2D needs an even n >= 4");
    if (n > 46340) throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "BrussMG2D grid too large");
    if (pre < 1 || post < 1) throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "BrussMG2D needs pre >= 1 and post >= 1");
    if (precision != NUMA_GPU_FP64 && precision != NUMA_GPU_FP32)
        throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "BrussMG2D precision must be FP64 or FP32");
    if (!(p.dt > 0.0) || !(p.Du >= 0.0) || !(p.Dv >= 0.0))
        throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "BrussMG2D requires dt > 0 and D >= 0");
    const size_t esz = precision == NUMA_GPU_FP64 ? 8 : 4;
    size_t m = n;
    for (;;) {
        auto L = std::make_unique<Level>();
        L->n = (int)m;
        L->su = p.Du * (static_cast<double>(m) * static_cast<double>(m));
        L->sv = p.Dv * (static_cast<double>(m) * static_cast<double>(m));
        const size_t mm = m * m;
        L->x.resize((2 * mm * esz + 7) / 8);
        L->b.resize((2 * mm * esz + 7) / 8);
        L->k.resize((4 * mm * esz + 7) / 8);
        levels_.push_back(std::move(L));
        if (m % 4 != 0 || m / 2 < 4) break;
        m /= 2;
    }
    // levels below the finest with n <= 64 (FP32) or n <= 32 (FP64) run as one block: x, b and K,
    // 8 (64^2 + 32^2 + ...) values, at most 175 KB of shared memory
    const int tail_max_n = precision == NUMA_GPU_FP64 ? kBmgTailMaxN / 2 : kBmgTailMaxN;
    for (size_t l = 1; l < levels_.size(); ++l) {
        Level& L = *levels_[l];
        if (precision == NUMA_GPU_FP32 && l + 1 < levels_.size()) L.T = btile_size(L.n, pre, post, ctx.sm_count);
        if (L.T) {
            L.y.resize(L.x.n);
        } else if (L.n <= tail_max_n) {
            tail_first_ = (int)l;
            break;
        }
    }
    if (tail_first_ > 0) {
        std::vector<TailLvl> d;
        size_t off = 0;
        for (size_t l = (size_t)tail_first_; l < levels_.size(); ++l) {
            const Level& L = *levels_[l];
            d.push_back(TailLvl{L.n, (int)off, L.k.p, LvlArgs<double>{L.n, L.su, L.sv, 4.0 * L.su, 4.0 * L.sv},
                                LvlArgs<float>{L.n, (float)L.su, (float)L.sv, (float)(4.0 * L.su),
                                               (float)(4.0 * L.sv)}});
            off += 8 * (size_t)L.n * L.n;
        }
        tail_count_ = (int)d.size();
        tail_smem_ = off * esz;
        tail_desc_.resize((d.size() * sizeof(TailLvl) + 7) / 8);
        NUMA_CUDA(cudaMemcpyAsync(tail_desc_.p, d.data(), d.size() * sizeof(TailLvl), cudaMemcpyHostToDevice,
                                  ctx_.stream));
        ctx_.sync();
        const int lim = precision == NUMA_GPU_FP64 ? set_dynamic_smem_limit(ctx_, k_bmg_tail<double>)
                                                   : set_dynamic_smem_limit(ctx_, k_bmg_tail<float>);
        if (tail_smem_ > (size_t)lim) throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "BrussMG2D tail exceeds shared memory");
    }
}

BrussMG2D::~BrussMG2D() {
    if (coarse_exec_) cudaGraphExecDestroy(coarse_exec_);
}

template <class T>
static T* tp(DeviceArray<double>& a) {
    return reinterpret_cast<T*>(a.p);
}

void BrussMG2D::set_state(const double* w) {
    state_set_ = true;
    const size_t nn = n0_ * n0_;
    const double c1 = 1.0 / P_.dt + (P_.B + 1.0), c2 = 1.0 / P_.dt;
    const unsigned g = (unsigned)((nn + 255) / 256);
    if (precision_ == NUMA_GPU_FP64)
        launch_pdl(k_bmg_kfine<double>, g, 256, 0, ctx_.stream, w, (int)n0_, c1, c2, P_.B, tp<double>(levels_[0]->k));
    else
        launch_pdl(k_bmg_kfine<float>, g, 256, 0, ctx_.stream, w, (int)n0_, (float)c1, (float)c2, (float)P_.B,
                                                       tp<float>(levels_[0]->k));
    ctx_.count_launch();
    for (size_t l = 0; l + 1 < levels_.size(); ++l) {
        const int nc = levels_[l + 1]->n;
        const dim3 grid((unsigned)((nc + 31) / 32), (unsigned)((nc + 7) / 8));
        if (precision_ == NUMA_GPU_FP64)
            launch_pdl(k_bmg_krestrict<double>, grid, dim3(32, 8), 0, ctx_.stream, tp<double>(levels_[l]->k), levels_[l]->n,
                                                                          tp<double>(levels_[l + 1]->k));
        else
            launch_pdl(k_bmg_krestrict<float>, grid, dim3(32, 8), 0, ctx_.stream, tp<float>(levels_[l]->k), levels_[l]->n,
                                                                         tp<float>(levels_[l + 1]->k));
        ctx_.count_launch();
    }
    ctx_.check_launch("BrussMG2D set_state");
}

// Whether level l's first smoothing pass is done by the restriction that forms its right-hand side.
template <class T>
bool BrussMG2D::first_fused(size_t l) const {
    return sizeof(T) == 4 && l > 0 && (int)l != tail_first_ && !levels_[l]->T && l + 1 < levels_.size();
}

template <class T>
void BrussMG2D::cycle(size_t l) {
    Level& L = *levels_[l];
    const int n = L.n;
    const bool finest = l == 0;
    const bool coarsest = l + 1 == levels_.size();
    cudaStream_t s = ctx_.stream;
    T* X = tp<T>(L.x);
    T* Bv = tp<T>(L.b);
    const T* K = tp<T>(L.k);
    const LvlArgs<T> A{n, (T)L.su, (T)L.sv, (T)(4.0 * L.su), (T)(4.0 * L.sv)};
    const dim3 blk(32, 8);
    const dim3 pgrid((unsigned)((n / 2 + 31) / 32), (unsigned)((n + 7) / 8));
    const size_t nn = (size_t)n * n;
    if ((int)l == tail_first_) {
        launch_pdl(k_bmg_tail<T>, 1, kBmgTailThreads<T>, tail_smem_, s, reinterpret_cast<const TailLvl*>(tail_desc_.p), tail_count_, pre_,
                                                  post_, kBmgCoarsestSweeps, Bv, X);
        ctx_.count_launch();
        return;
    }
    if constexpr (sizeof(T) == 4) {
        if (L.T) {
            Level& C = *levels_[l + 1];
            const unsigned g = (unsigned)((C.n + L.T - 1) / L.T);
            const BTile down = btile(A, L.T, pre_, true), up = btile(A, L.T, post_, false);
            launch_pdl(k_btile_down, dim3(g, g), btile_threads(down), btile_smem(down), s, (const T*)Bv, K, tp<T>(L.y),
                       tp<T>(C.b), down);
            ctx_.count_launch();
            cycle<T>(l + 1);
            launch_pdl(k_btile_up, dim3(g, g), btile_threads(up), btile_smem(up), s, (const T*)Bv, K,
                       (const T*)tp<T>(L.y), (const T*)tp<T>(C.x), X, up);
            ctx_.count_launch();
            return;
        }
    }
    if (coarsest) {
        if (finest) {
            if (r32_) launch_pdl(k_bmg_in<T, float>, (unsigned)((nn + 255) / 256), 256, 0, s, r32_, n, Bv);
            else launch_pdl(k_bmg_in<T>, (unsigned)((nn + 255) / 256), 256, 0, s, r0_, n, Bv);
            ctx_.count_launch();
        }
        if (nn <= (size_t)kBmgOneBlockPoints) {
            launch_pdl(k_bmg_coarsest<T>, 1, 1024, 0, s, X, Bv, K, A, kBmgCoarsestSweeps);
            ctx_.count_launch();
        } else {
            launch_pdl(k_bmg_pass<T, kBPassFirst>, pgrid, blk, 0, s, X, Bv, K, A, 0, nullptr, nullptr, nullptr);
            launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 1, nullptr, nullptr, nullptr);
            ctx_.count_launch(2);
            for (int k = 1; k < kBmgCoarsestSweeps; ++k) {
                launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 0, nullptr, nullptr, nullptr);
                launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 1, nullptr, nullptr, nullptr);
                ctx_.count_launch(2);
            }
        }
        if (finest) {
            launch_pdl(k_bmg_out<T>, (unsigned)((nn + 255) / 256), 256, 0, s, X, n, z0_);
            ctx_.count_launch();
        }
        return;
    }
    // pre-smoothing: colours 0, 1; the first pass starts from x = 0 (in FP32 the restriction that formed b
    // has done it below the finest level)
    if (finest && r32_) {
        launch_pdl(k_bmg_pass<T, kBPassFirst, float>, pgrid, blk, 0, s, X, Bv, K, A, 0, r32_, nullptr, nullptr);
        ctx_.count_launch();
    } else if (!first_fused<T>(l)) {
        launch_pdl(k_bmg_pass<T, kBPassFirst>, pgrid, blk, 0, s, X, Bv, K, A, 0, finest ? r0_ : nullptr, nullptr, nullptr);
        ctx_.count_launch();
    }
    launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 1, nullptr, nullptr, nullptr);
    ctx_.count_launch();
    for (int k = 1; k < pre_; ++k) {
        launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 0, nullptr, nullptr, nullptr);
        launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 1, nullptr, nullptr, nullptr);
        ctx_.count_launch(2);
    }
    Level& C = *levels_[l + 1];
    const int nc = C.n;
    if constexpr (sizeof(T) == 4) {
        const int rows = bmg_march_rows(nc, ctx_.sm_count);
        const dim3 rgrid((unsigned)((nc + 30) / 31), (unsigned)((nc + 4 * rows - 1) / (4 * rows))), rblk(32, 4);
        const LvlArgs<T> Ac{nc, (T)C.su, (T)C.sv, (T)(4.0 * C.su), (T)(4.0 * C.sv)};
        if (first_fused<T>(l + 1))
            launch_pdl(k_bmg_restrict_march<T, true>, rgrid, rblk, 0, s, X, Bv, K, A, rows, tp<T>(C.b), tp<T>(C.k),
                       tp<T>(C.x), Ac);
        else
            launch_pdl(k_bmg_restrict_march<T, false>, rgrid, rblk, 0, s, X, Bv, K, A, rows, tp<T>(C.b), nullptr,
                       nullptr, Ac);
    } else {
        launch_pdl(k_bmg_restrict<T>, dim3((unsigned)((nc + 15) / 16), (unsigned)((nc + 15) / 16)), dim3(16, 16), 0, s,
                   X, Bv, K, A, tp<T>(C.b));
    }
    ctx_.count_launch();
    if (finest) coarse_cycle();
    else cycle<T>(l + 1);
    const dim3 cgrid((unsigned)((nc + 31) / 32), (unsigned)((nc + 7) / 8));
    constexpr bool fused_prolong = sizeof(T) == 4;
    if constexpr (!fused_prolong) {
        launch_pdl(k_bmg_prolong<T>, cgrid, blk, 0, s, tp<T>(C.x), nc, X);
        ctx_.count_launch();
    }
    // post-smoothing: colours 1, 0; the very last pass of the finest level writes z
    for (int k = 0; k < post_; ++k) {
        bool corrected = false;
        if constexpr (fused_prolong) {
            if (k == 0) {
                launch_pdl(k_bmg_prolong_pass<T>, cgrid, blk, 0, s, tp<T>(C.x), X, Bv, K, A);
                corrected = true;
            }
        }
        if (!corrected)
            launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 1, nullptr, nullptr, nullptr);
        if (finest && k + 1 == post_)
            launch_pdl(k_bmg_pass<T, kBPassLast>, pgrid, blk, 0, s, X, Bv, K, A, 0, nullptr, z0_, z32_);
        else
            launch_pdl(k_bmg_pass<T, kBPassNormal>, pgrid, blk, 0, s, X, Bv, K, A, 0, nullptr, nullptr, nullptr);
        ctx_.count_launch(2);
    }
}

// Levels 1 and below as one CUDA graph: their arrays never move, and the blocks K are updated in
// place by set_state, so the graph captured on first use stays valid.
void BrussMG2D::coarse_cycle() {
    if (!coarse_exec_) {
        std::lock_guard<std::recursive_mutex> lk(alloc_capture_mutex());
        const uint64_t before = ctx_.launches;
        NUMA_CUDA(cudaStreamBeginCapture(ctx_.stream, cudaStreamCaptureModeThreadLocal));
        cudaGraph_t graph = nullptr;
        try {
            if (precision_ == NUMA_GPU_FP64) cycle<double>(1);
            else cycle<float>(1);
        } catch (...) {
            cudaStreamEndCapture(ctx_.stream, &graph);
            if (graph) cudaGraphDestroy(graph);
            cudaGetLastError();
            throw;
        }
        NUMA_CUDA(cudaStreamEndCapture(ctx_.stream, &graph));
        const cudaError_t e = cudaGraphInstantiate(&coarse_exec_, graph, 0);
        cudaGraphDestroy(graph);
        NUMA_CUDA(e);
        coarse_kernels_ = ctx_.launches - before;
        ctx_.launches = before;
    }
    NUMA_CUDA(cudaGraphLaunch(coarse_exec_, ctx_.stream));
    ctx_.count_launch(static_cast<unsigned>(coarse_kernels_));
}

// Average duration of one colour pass on the finest level (the V-cycle's dominant kernel), over
// reps back-to-back launches timed with CUDA events on the context's stream; the blocks must have
// been set.
double BrussMG2D::time_finest_pass(int reps) {
    if (!state_set_) throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "BrussMG2D: set_state before timing");
    Level& L = *levels_[0];
    const int n = L.n;
    const LvlArgs<double> A64{n, L.su, L.sv, 4.0 * L.su, 4.0 * L.sv};
    const LvlArgs<float> A32{n, (float)L.su, (float)L.sv, (float)(4.0 * L.su), (float)(4.0 * L.sv)};
    const dim3 blk(32, 8), pgrid((unsigned)((n / 2 + 31) / 32), (unsigned)((n + 7) / 8));
    const size_t esz = precision_ == NUMA_GPU_FP64 ? 8 : 4;
    NUMA_CUDA(cudaMemsetAsync(L.x.p, 0, 2 * (size_t)n * n * esz, ctx_.stream));
    NUMA_CUDA(cudaMemsetAsync(L.b.p, 0, 2 * (size_t)n * n * esz, ctx_.stream));
    cudaEvent_t a, b;
    NUMA_CUDA(cudaEventCreate(&a));
    NUMA_CUDA(cudaEventCreate(&b));
    auto launch = [&](int colour) {
        if (precision_ == NUMA_GPU_FP64)
            launch_pdl(k_bmg_pass<double, kBPassNormal>, pgrid, blk, 0, ctx_.stream, tp<double>(L.x),
                       tp<double>(L.b), tp<double>(L.k), A64, colour, nullptr, nullptr, nullptr);
        else
            launch_pdl(k_bmg_pass<float, kBPassNormal>, pgrid, blk, 0, ctx_.stream, tp<float>(L.x), tp<float>(L.b),
                       tp<float>(L.k), A32, colour, nullptr, nullptr, nullptr);
    };
    launch(0);
    NUMA_CUDA(cudaEventRecord(a, ctx_.stream));
    for (int r = 0; r < reps; ++r) launch(r & 1);
    NUMA_CUDA(cudaEventRecord(b, ctx_.stream));
    NUMA_CUDA(cudaEventSynchronize(b));
    float ms = 0.f;
    NUMA_CUDA(cudaEventElapsedTime(&ms, a, b));
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    ctx_.count_launch(reps + 1);
    ctx_.check_launch("BrussMG2D time_finest_pass");
    return reps > 0 ? ms / reps : 0.0;
}

void BrussMG2D::apply32(const double* r, float* z32) {
    if (!supports_out32()) throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "BrussMG2D: no FP32 output for this hierarchy");
    z32_ = z32;
    try {
        apply(r, nullptr);
    } catch (...) {
        z32_ = nullptr;
        throw;
    }
    z32_ = nullptr;
}

void BrussMG2D::apply32f(const float* r32, float* z32) {
    if (!supports_out32()) throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "BrussMG2D: no FP32 output for this hierarchy");
    r0_ = nullptr;
    r32_ = r32;
    z0_ = nullptr;
    z32_ = z32;
    try {
        cycle<float>(0);
    } catch (...) {
        r32_ = nullptr;
        z32_ = nullptr;
        throw;
    }
    r32_ = nullptr;
    z32_ = nullptr;
    ctx_.check_launch("BrussMG2D apply32f");
}

void BrussMG2D::apply(const double* r, double* z) {
    const size_t N = size();
    // the finest pass reads r while the last one writes z: an aliased call goes through a copy
    const double* rin = r;
    if (r == z) {
        alias_.resize(N);
        dev_copy(ctx_, r, alias_.p, N);
        rin = alias_.p;
    }
    r0_ = rin;
    z0_ = z;
    if (precision_ == NUMA_GPU_FP64) cycle<double>(0);
    else cycle<float>(0);
    ctx_.check_launch("BrussMG2D apply");
}

namespace {
// Provider over BrussMG2D: make(x) sets the blocks at the Newton iterate.
class BrussMGProvider final : public Provider {
public:
    BrussMGProvider(Context& ctx, size_t n, const numa_brusselator2d_params& p, int precision, int pre, int post)
        : mg_(ctx, n, p, precision, pre, post) {}
    void make(const double* x, const double*) override { mg_.set_state(x); }
    void apply(const double* r, double* z) override { mg_.apply(r, z); }
    // the FP32 cycle can hand its result over unwidened
    bool has_apply32() const override { return mg_.supports_out32(); }
    void apply32(const double* r, float* z32) override { mg_.apply32(r, z32); }
    bool has_apply32f() const override { return mg_.supports_out32(); }
    void apply32f(const float* r32, float* z32) override { mg_.apply32f(r32, z32); }
    int kind() const override { return NUMA_GPU_PRECOND_BRUSS_MG; }

private:
    BrussMG2D mg_;
};
}  // namespace

std::unique_ptr<Provider> make_bruss_mg_provider(Context& ctx, size_t n, const numa_brusselator2d_params& p,
                                                 int precision, int pre, int post) {
    return std::make_unique<BrussMGProvider>(ctx, n, p, precision, pre, post);
}

}  // namespace numa::gpu
