// hmg2d.cu — the 2D geometric-multigrid V-cycle for alpha I - nu Lap_h
// (linalg/helmholtz_mg2d.hpp) and the Burgers2D preconditioner provider built on it
// (problems/burgers2d.hpp:220-246), FP64.
//
// Same hierarchy (levels while n is odd, s = nu h^-2 quartered per level), red-black
// Gauss-Seidel with colour (i+j)&1 and the reference's colour orders, 9-point full weighting,
// bilinear additive prolongation, coarsest level exact at n = 1 else 30 alternating sweeps.  The
// arithmetic follows the reference operation for operation (the neighbour sum starts from 0.0,
// the update divides by alpha + 4s), so the cycle equals the reference's bit for bit.  As in the
// 3D cycle, the first colour pass of a level reads no neighbours (its x is zero there), and the
// prolongation is added only at colour-0 points when post-smoothing follows.
//
// A cycle is many short steps (11 a level), so what bounds it is launches: one host launch a step and field
// took 17.4 ms of a Burgers solve at 255^2 whose kernels ran 9 ms.  Hence: u and v go through one cycle
// together (blockIdx.z = field); programmatic dependent launch; the levels below the finest in one CUDA graph; the
// levels of 15 < n <= 127 in two tiled kernels each, on as many SMs as there are, where a step is a block barrier; and
// the levels below in one CTA a field, in shared memory (k_hmg_tail).  The Burgers solve at 255^2 went from 17.5 to
// 3.2 ms; a cycle of both fields is 82 us there (110 with 63^2 and 127^2 launched pass by pass and 31^2 in the tail):
// 30 of them the finest level's 11 launches, 16 the tail (steps bound by the latency of their nine dependent FP64
// operations), 11 each the levels between.
#include <cmath>
#include <limits>

#include "numa_internal.hpp"

namespace numa::gpu {

struct HelmholtzMG2D::Level {
    int n = 0;
    double s = 0.0;  // nu / h^2 of this level
    DeviceArray<double> x, b;
    int T = 0;              // > 0: run by the tiled kernels, T x T coarse points a block
    DeviceArray<double> y;  // tiled: x on its way down
};

namespace {

constexpr int BX = 32, BY = 8;

// A level's constants: s = nu h^-2, den = alpha + 4 s and its reciprocal for div_by_recip (the IEEE quotient in
// three operations).
struct HLvl {
    int n;
    double s, alpha, den, rden;
};

// x = (b + s * nb) / (alpha + 4 s), nb = 0 + x_{i-1} + x_{i+1} + x_{j-1} + x_{j+1}
// (helmholtz_mg2d.hpp:51-70).  FIRST: x is zero before the pass.  blockIdx.z: the field, n^2 values apart.
template <bool FIRST>
__global__ void __launch_bounds__(BX* BY) k_hsmooth(double* __restrict__ x, const double* __restrict__ b, HLvl L,
                                                    int colour) {
    pdl_wait();
    pdl_trigger();
    const int n = L.n;
    const int jj = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    if (i >= n) return;
    const int j = 2 * jj + ((i + colour) & 1);
    if (j >= n) return;
    const size_t p = ((size_t)blockIdx.z * n + i) * n + j;
    double nb = 0.0;
    if (!FIRST) {
        const double xu = i > 0 ? x[p - n] : 0.0, xd = i + 1 < n ? x[p + n] : 0.0;
        const double xl = j > 0 ? x[p - 1] : 0.0, xr = j + 1 < n ? x[p + 1] : 0.0;
        nb = nb + xu;
        nb = nb + xd;
        nb = nb + xl;
        nb = nb + xr;
    }
    x[p] = div_by_recip(b[p] + L.s * nb, L.den, L.rden);
}

// r = b - (alpha x + s (4x - nb)) (helmholtz_mg2d.hpp:72-87)
__global__ void __launch_bounds__(BX* BY) k_hresidual(const double* __restrict__ x, const double* __restrict__ b,
                                                      double* __restrict__ r, HLvl L) {
    pdl_wait();
    pdl_trigger();
    const int n = L.n;
    const int j = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    if (i >= n || j >= n) return;
    const size_t p = ((size_t)blockIdx.z * n + i) * n + j;
    const double xu = i > 0 ? x[p - n] : 0.0, xd = i + 1 < n ? x[p + n] : 0.0;
    const double xl = j > 0 ? x[p - 1] : 0.0, xr = j + 1 < n ? x[p + 1] : 0.0;
    double nb = 0.0;
    nb = nb + xu;
    nb = nb + xd;
    nb = nb + xl;
    nb = nb + xr;
    r[p] = b[p] - (L.alpha * x[p] + L.s * (4.0 * x[p] - nb));
}

// coarse b = sum_{a,b} (w_a w_b) r(2I+a, 2J+b), weights (1/4,1/2,1/4) (helmholtz_mg2d.hpp:89-108);
// each weight product is a power of two, so the FMA equals the reference's multiply-then-add.  A coarser level
// has nf = 2 nc + 1: every fine point exists.
__global__ void __launch_bounds__(BX* BY) k_hrestrict(const double* __restrict__ rf, double* __restrict__ bc, int nf,
                                                      int nc) {
    pdl_wait();
    pdl_trigger();
    const int J = blockIdx.x * BX + threadIdx.x;
    const int I = blockIdx.y * BY + threadIdx.y;
    if (I >= nc || J >= nc) return;
    const double* row = rf + ((size_t)blockIdx.z * nf + 2 * I) * nf + 2 * J;
    const double w[3] = {0.25, 0.5, 0.25};
    double v[9];
#pragma unroll
    for (int a = 0; a < 9; ++a) v[a] = row[(a / 3) * nf + a % 3];
    double acc = 0.0;
#pragma unroll
    for (int a = 0; a < 9; ++a) acc = __fma_rn(w[a / 3] * w[a % 3], v[a], acc);
    bc[((size_t)blockIdx.z * nc + I) * nc + J] = acc;
}

// fine x += bilinear interpolation of coarse x (helmholtz_mg2d.hpp:110-136): an odd index has the coarse
// neighbour (f - 1) / 2 with weight 1, an even one f / 2 - 1 and f / 2 with weight 1/2 (an absent one adds
// +0.0).  COLOUR0_ONLY: only points with (i+j) even.
template <bool COLOUR0_ONLY>
__global__ void __launch_bounds__(BX* BY) k_hprolong(const double* __restrict__ xc, double* __restrict__ xf, int nc,
                                                     int nf) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    if (i >= nf) return;
    const int j = COLOUR0_ONLY ? 2 * t + (i & 1) : t;
    if (j >= nf) return;
    const int I0 = ((i + 1) >> 1) - 1, J0 = ((j + 1) >> 1) - 1;
    const double w = (i & 1 ? 1.0 : 0.5) * (j & 1 ? 1.0 : 0.5);
    double v[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const int I = I0 + (h >> 1), J = J0 + (h & 1);
        const bool in = !((h >> 1) && (i & 1)) && !((h & 1) && (j & 1)) && I >= 0 && I < nc && J >= 0 && J < nc;
        v[h] = in ? xc[((size_t)blockIdx.z * nc + I) * nc + J] : 0.0;
    }
    double acc = 0.0;
#pragma unroll
    for (int h = 0; h < 4; ++h) acc = __fma_rn(w, v[h], acc);
    const size_t p = ((size_t)blockIdx.z * nf + i) * nf + j;
    xf[p] = xf[p] + acc;
}

// ------------------------------------------------------------------------------------------
// The levels of n <= kTileTail (kTailTop where no tiled level applies) in one CTA a field: x of each level with a halo of zeros, pitch m = (n + 2) | 1, the
// two parities of the padded index (the colours) stored apart, so that a pass reads one half and writes the other;
// b and the residual in natural order.  The arithmetic is the launched kernels' operation for operation.
constexpr int kTailTop = 31, kTailMax = 6, kTailThreads = 512;  // 31, 15, 7, 3, 1
constexpr int kTileTop = 127, kTileTail = 15;                   // the levels of the tiled kernels, below
struct HTailLvl {
    HLvl L;
    int m, H, offX, offB;  // pitch, elements of one parity of x, element offsets in shared memory
};
struct HTail {
    int levels, pre, post, offR, total;
    HTailLvl T[kTailMax];
};

extern __shared__ __align__(16) double htail_smem[];

// ------------------------------------------------------------------------------------------
// Levels of kTileTail < n <= kTileTop in two kernels, one on the way down (pre-smoothing from x = 0, residual,
// restriction) and one on the way up (prolongation, post-smoothing).  A block owns T x T coarse points and the fine
// points 2I, 2I + 1 of them (its last row and column also 2I + 2), and runs every pass on a region that shrinks by a
// point on each side a pass, so that no block needs another's values within the kernel: the points around its own are
// computed again.  Thread (i, jj) of the region, in linear order, holds b of the pair of points 2jj, 2jj + 1 of row i;
// x is in shared memory with zeros around it and outside the grid.  The arithmetic is the launched kernels' operation
// for operation.  x goes down in one array and comes up in another, as neighbours read it.
// Bound by the latency of a pass's nine dependent FP64 operations (63^2 and below) or the FP64 pipe.  A cycle of two
// fields: 31^2 37 -> 28.4 us, 63^2 and 127^2 11 to 12 us a level (11 launches: 24).
struct HTile {
    HLvl L;
    int nc, T, S, np, sweeps;  // S x S fine points of the region, np = (S + 1) / 2 pairs a row
};

__device__ __forceinline__ void htile_pass(double* X, int P, double b, const HLvl& L, bool first) {
    double nb = 0.0;
    if (!first) {
        const int m = P;
        nb = nb + X[-m];
        nb = nb + X[m];
        nb = nb + X[-1];
        nb = nb + X[1];
    }
    *X = div_by_recip(b + L.s * nb, L.den, L.rden);
}

__global__ void __launch_bounds__(1024) k_htile_down(const double* __restrict__ b, double* __restrict__ x,
                                                     double* __restrict__ bc, const __grid_constant__ HTile t) {
    const int n = t.L.n, nc = t.nc, S = t.S, m = S + 2, h = 2 * t.sweeps;
    double* X = htail_smem;           // (S + 2)^2
    double* R = htail_smem + m * m;   // (2T + 1)^2
    const int nt = blockDim.x, tid = threadIdx.x;
    for (int q = tid; q < m * m; q += nt) X[q] = 0.0;
    const int C0i = blockIdx.y * t.T, C0j = blockIdx.x * t.T;
    const int ri = tid / t.np, rj = 2 * (tid - ri * t.np);      // region row, first column of the pair
    const int i = 2 * C0i - h + ri, j0 = 2 * C0j - h + rj;      // grid row, column
    const bool row = ri < S && i >= 0 && i < n;
    bool in[2];
    double bv[2], xv[2];
    pdl_wait();
    pdl_trigger();
    const size_t f0 = (size_t)blockIdx.z * n * n;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        in[q] = row && rj + q < S && j0 + q >= 0 && j0 + q < n;
        bv[q] = in[q] ? b[f0 + (size_t)i * n + j0 + q] : 0.0;
        xv[q] = 0.0;
    }
    double* Xp = X + (ri + 1) * m + rj + 1;
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < h; ++p) {  // colours 0, 1, 0, 1, ...; the region of pass p starts p points further in
        const int q = (i + j0 + p) & 1;  // the member of the pair of this colour
        const int c = rj + q;
        if ((q ? in[1] : in[0]) && ri >= p && ri < S - p && c >= p && c < S - p)
            htile_pass(Xp + q, m, q ? bv[1] : bv[0], t.L, p == 0);
        __syncthreads();
    }
    // the residual of rows and columns 2 C0 .. 2 C0 + 2T
    const int rn = 2 * t.T + 1;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int a = ri - h, c = rj + q - h;
        if (!in[q] || a < 0 || a >= rn || c < 0 || c >= rn) continue;
        const double* P = Xp + q;
        const double xc = *P;
        double nb = 0.0;
        nb = nb + P[-m];
        nb = nb + P[m];
        nb = nb + P[-1];
        nb = nb + P[1];
        R[a * rn + c] = bv[q] - (t.L.alpha * xc + t.L.s * (4.0 * xc - nb));
        const bool oi = a < rn - 1 || C0i + t.T >= nc, oj = c < rn - 1 || C0j + t.T >= nc;
        if (oi && oj) x[f0 + (size_t)i * n + j0 + q] = xc;
    }
    __syncthreads();
    const int I = tid / t.T, J = tid - I * t.T;
    if (I < t.T && C0i + I < nc && C0j + J < nc) {
        const double w[3] = {0.25, 0.5, 0.25};
        const double* r = R + 2 * I * rn + 2 * J;
        double acc = 0.0;
#pragma unroll
        for (int a = 0; a < 9; ++a) acc = __fma_rn(w[a / 3] * w[a % 3], r[(a / 3) * rn + a % 3], acc);
        bc[((size_t)blockIdx.z * nc + C0i + I) * nc + C0j + J] = acc;
    }
}

__global__ void __launch_bounds__(1024) k_htile_up(const double* __restrict__ b, const double* __restrict__ xd,
                                                   const double* __restrict__ xc, double* __restrict__ x,
                                                   const __grid_constant__ HTile t) {
    const int n = t.L.n, nc = t.nc, S = t.S, m = S + 2, h = 2 * t.sweeps;
    double* X = htail_smem;
    const int nt = blockDim.x, tid = threadIdx.x;
    for (int q = tid; q < m * m; q += nt) X[q] = 0.0;
    const int C0i = blockIdx.y * t.T, C0j = blockIdx.x * t.T;
    const int ri = tid / t.np, rj = 2 * (tid - ri * t.np);
    const int i = 2 * C0i - h + ri, j0 = 2 * C0j - h + rj;
    const bool row = ri < S && i >= 0 && i < n;
    bool in[2];
    double bv[2];
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const size_t f0 = (size_t)blockIdx.z * n * n;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        in[q] = row && rj + q < S && j0 + q >= 0 && j0 + q < n;
        bv[q] = in[q] ? b[f0 + (size_t)i * n + j0 + q] : 0.0;
    }
    double* Xp = X + (ri + 1) * m + rj + 1;
    {  // the colour-0 point of the pair, corrected as k_hprolong does
        const int q = (i + j0) & 1, j = j0 + q;
        if (q ? in[1] : in[0]) {
            const int I0 = ((i + 1) >> 1) - 1, J0 = ((j + 1) >> 1) - 1;
            const double w = (i & 1 ? 1.0 : 0.5) * (j & 1 ? 1.0 : 0.5);
            double v[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int I = I0 + (g >> 1), J = J0 + (g & 1);
                const bool has = !((g >> 1) && (i & 1)) && !((g & 1) && (j & 1)) && I >= 0 && I < nc && J >= 0 && J < nc;
                v[g] = has ? xc[((size_t)blockIdx.z * nc + I) * nc + J] : 0.0;
            }
            const double xo = xd[f0 + (size_t)i * n + j];
            double acc = 0.0;
#pragma unroll
            for (int g = 0; g < 4; ++g) acc = __fma_rn(w, v[g], acc);
            Xp[q] = xo + acc;
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < h; ++p) {  // colours 1, 0, 1, 0, ...
        const int q = (i + j0 + p + 1) & 1, c = rj + q, d = p + 1;
        if ((q ? in[1] : in[0]) && ri >= d && ri < S - d && c >= d && c < S - d)
            htile_pass(Xp + q, m, q ? bv[1] : bv[0], t.L, false);
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int a = ri - h, c = rj + q - h, rn = 2 * t.T + 1;
        if (!in[q] || a < 0 || a >= rn || c < 0 || c >= rn) continue;
        const bool oi = a < rn - 1 || C0i + t.T >= nc, oj = c < rn - 1 || C0j + t.T >= nc;
        if (oi && oj) x[f0 + (size_t)i * n + j0 + q] = Xp[q];
    }
}

static_assert(kTailTop * ((kTailTop + 1) / 2) <= kTailThreads && (kTailTop / 2) * (kTailTop / 2) <= kTailThreads,
              "htail_sweeps and htail_restrict: a thread for each pair, and for each coarse point");

// x at padded index P
__device__ __forceinline__ double& hx(double* X, int H, int P) { return X[(P & 1) * H + (P >> 1)]; }

__device__ __noinline__ void htail_sweeps(const HTailLvl& T, int sweeps, int order, bool alternate, bool first) {
    const HLvl L = T.L;
    const int n = L.n, m = T.m, H = T.H, np = (n + 1) >> 1;
    double* X = htail_smem + T.offX;
    const double* B = htail_smem + T.offB;
    const int i = (int)threadIdx.x / np, j0 = 2 * ((int)threadIdx.x - i * np);
#pragma unroll 1
    for (int p = 0; p < 2 * sweeps; ++p) {
        const int colour = (p & 1) ^ (alternate ? (p >> 1) & 1 : order);
        const int j = j0 + ((i + colour) & 1);
        if (i < n && j < n) {
            const int q = ((i + 1) * m + j + 1) >> 1;
            const double* o = X + (colour ^ 1) * H + q;
            double nb = 0.0;
            if (!first || p > 0) {
                nb = nb + o[(colour - m) >> 1];
                nb = nb + o[(colour + m) >> 1];
                nb = nb + o[(colour - 1) >> 1];
                nb = nb + o[(colour + 1) >> 1];
            }
            X[colour * H + q] = div_by_recip(B[i * n + j] + L.s * nb, L.den, L.rden);
        }
        __syncthreads();
    }
}

__device__ __noinline__ void htail_residual(const HTailLvl& T, double* R) {
    const HLvl L = T.L;
    const int n = L.n, m = T.m, H = T.H;
    double* X = htail_smem + T.offX;
    const double* B = htail_smem + T.offB;
#pragma unroll 1
    for (int t = threadIdx.x; t < n * n; t += kTailThreads) {
        const int i = t / n, P = (i + 1) * m + t - i * n + 1;
        const double x = hx(X, H, P);
        double nb = 0.0;
        nb = nb + hx(X, H, P - m);
        nb = nb + hx(X, H, P + m);
        nb = nb + hx(X, H, P - 1);
        nb = nb + hx(X, H, P + 1);
        R[t] = B[t] - (L.alpha * x + L.s * (4.0 * x - nb));
    }
    __syncthreads();
}

__device__ __noinline__ void htail_restrict(const double* R, int nf, double* B, int nc) {
    const double w[3] = {0.25, 0.5, 0.25};
    const int t = threadIdx.x;
    if (t < nc * nc) {
        const int I = t / nc, J = t - I * nc;
        const double* row = R + 2 * I * nf + 2 * J;
        double acc = 0.0;
#pragma unroll
        for (int a = 0; a < 9; ++a) acc = __fma_rn(w[a / 3] * w[a % 3], row[(a / 3) * nf + a % 3], acc);
        B[t] = acc;
    }
    __syncthreads();
}

__device__ __noinline__ void htail_prolong(const HTailLvl& F, const HTailLvl& C, bool both) {
    const int n = F.L.n, m = F.m, mc = C.m, Hc = C.H;
    double* X = htail_smem + F.offX;
    double* XC = htail_smem + C.offX;
#pragma unroll 1
    for (int t = threadIdx.x; t < n * n; t += kTailThreads) {
        const int i = t / n, j = t - i * n;
        if (!both && ((i + j) & 1)) continue;
        const double w = (i & 1 ? 1.0 : 0.5) * (j & 1 ? 1.0 : 0.5);
        const int Pc = ((i + 1) >> 1) * mc + ((j + 1) >> 1);  // padded: coarse (I0, J0)
        double acc = 0.0;
        acc = __fma_rn(w, hx(XC, Hc, Pc), acc);
        if (!(j & 1)) acc = __fma_rn(w, hx(XC, Hc, Pc + 1), acc);
        if (!(i & 1)) acc = __fma_rn(w, hx(XC, Hc, Pc + mc), acc);
        if (!((i | j) & 1)) acc = __fma_rn(w, hx(XC, Hc, Pc + mc + 1), acc);
        double& x = hx(X, F.H, (i + 1) * m + j + 1);
        x = x + acc;
    }
    __syncthreads();
}

// x = the cycle's levels below and including the top one, applied to b (n^2 values a field, blockIdx.x = field;
// x and b may be the same array).
__global__ void __launch_bounds__(kTailThreads) k_hmg_tail(const double* b, double* x,
                                                           const __grid_constant__ HTail tp) {
    __shared__ HTailLvl lv[kTailMax];
    for (int t = threadIdx.x; t < (int)(sizeof(lv) / 4); t += kTailThreads)
        reinterpret_cast<int*>(lv)[t] = reinterpret_cast<const int*>(tp.T)[t];
    for (int t = threadIdx.x; t < tp.total; t += kTailThreads) htail_smem[t] = 0.0;  // the halos stay zero
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const int n = tp.T[0].L.n, last = tp.levels - 1;
    const size_t f0 = (size_t)blockIdx.x * n * n;
    double* R = htail_smem + tp.offR;
    for (int t = threadIdx.x; t < n * n; t += kTailThreads) htail_smem[tp.T[0].offB + t] = b[f0 + t];
    __syncthreads();
#pragma unroll 1
    for (int l = 0; l < last; ++l) {
        htail_sweeps(lv[l], tp.pre, 0, false, true);
        htail_residual(lv[l], R);
        htail_restrict(R, lv[l].L.n, htail_smem + lv[l + 1].offB, lv[l + 1].L.n);
    }
    // the coarsest: x = b / (alpha + 4 s) at n = 1 (a sweep of its one point), else 30 alternating sweeps
    htail_sweeps(lv[last], lv[last].L.n == 1 ? 1 : 30, 0, true, true);
#pragma unroll 1
    for (int l = last - 1; l >= 0; --l) {
        htail_prolong(lv[l], lv[l + 1], tp.post == 0);
        htail_sweeps(lv[l], tp.post, 1, false, false);
    }
    for (int t = threadIdx.x; t < n * n; t += kTailThreads) {
        const int i = t / n;
        x[f0 + t] = hx(htail_smem + lv[0].offX, lv[0].H, (i + 1) * lv[0].m + t - i * n + 1);
    }
}

}  // namespace

// The coarse points T a side of a tile block, 0 for a level that the tiled kernels do not take: the smallest T whose
// blocks all have an SM to themselves, for 1 to 3 sweeps and kTileTail < n <= kTileTop.  Above, the points computed
// again cost the FP64 pipe more than the launches did (255^2, 1.6 times the points: the cycle 90 us against 82); below,
// one CTA's tail is faster (15^2: 19.5 us against 21.0).
static int tile_size(int n, int fields, int pre, int post, int sm_count) {
    if (n > kTileTop || n <= kTileTail || pre < 1 || pre > 3 || post < 1 || post > 3) return 0;
    const int nc = (n - 1) / 2;
    int T = 1;
    while ((long long)((nc + T - 1) / T) * ((nc + T - 1) / T) * fields > sm_count) {
        if (++T > nc) return 0;
    }
    const int S = 2 * T + 1 + 4 * std::max(pre, post);
    return S * ((S + 1) / 2) <= 1024 ? T : 0;
}

static HLvl hlvl(int n, double s, double alpha) {
    const double den = alpha + 4.0 * s;
    // recip_for_div on the host: RN(1/den) inside the exponent range the correction needs, else 0
    const double a = std::fabs(den);
    return HLvl{n, s, alpha, den, a >= 0x1p-960 && a <= 0x1p960 ? 1.0 / den : 0.0};
}

HelmholtzMG2D::HelmholtzMG2D(Context& ctx, size_t n, double alpha, double nu, int pre, int post, int fields)
    : ctx_(ctx), N0_(n * n), fields_(fields), alpha_(alpha), pre_(pre), post_(post) {
    if (n == 0) throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "HelmholtzMG2D requires a positive grid size");
    if (pre < 0 || post < 0) throw Status(NUMA_GPU_ERR_INVALID_ARGUMENT, "negative sweep count");
    if (n > 46340) throw Status(NUMA_GPU_ERR_NOT_SUPPORTED, "HelmholtzMG2D grid too large");
    size_t m = n;
    double s = nu * (static_cast<double>(n) + 1.0) * (static_cast<double>(n) + 1.0);
    for (;;) {
        auto L = std::make_unique<Level>();
        L->n = static_cast<int>(m);
        L->s = s;
        levels_.push_back(std::move(L));
        if (m % 2 == 0 || m <= 1) break;
        m = (m - 1) / 2;
        s /= 4.0;
    }
    for (size_t l = 0; l < levels_.size(); ++l) {
        Level& L = *levels_[l];
        const bool coarser = l + 1 < levels_.size();
        L.T = coarser ? tile_size(L.n, fields, pre, post, ctx.sm_count) : 0;
        if (L.n <= (L.T ? kTileTail : kTailTop)) {  // (at most 31, 15, 7, 3, 1 follow)
            L.T = 0;
            tail_l_ = l;
            break;
        }
        if (L.T) L.y.resize((size_t)fields * L.n * L.n);
    }
    for (size_t l = 1; l < levels_.size() && l <= tail_l_; ++l) {
        const size_t Nl = (size_t)fields * levels_[l]->n * levels_[l]->n;
        levels_[l]->x.resize(Nl);
        levels_[l]->b.resize(Nl);
    }
    if (tail_l_ > 0 && !levels_[0]->T) resid_.resize(fields * N0_);
    set_dynamic_smem_limit(ctx_, k_hmg_tail);
}

HelmholtzMG2D::~HelmholtzMG2D() {
    if (exec_) cudaGraphExecDestroy(exec_);
}

void HelmholtzMG2D::launch_tail(const double* b, double* x) {
    HTail tp{};
    tp.levels = (int)(levels_.size() - tail_l_);
    tp.pre = pre_;
    tp.post = post_;
    int off = 0;
    for (int l = 0; l < tp.levels; ++l) {
        const Level& L = *levels_[tail_l_ + l];
        HTailLvl& T = tp.T[l];
        T.L = hlvl(L.n, L.s, alpha_);
        T.m = (L.n + 2) | 1;
        T.H = ((L.n + 2) * T.m + 2) / 2;
        T.offX = off;
        T.offB = off + 2 * T.H;
        off = T.offB + L.n * L.n;
    }
    tp.offR = off;
    tp.total = off + levels_[tail_l_]->n * levels_[tail_l_]->n;
    launch_pdl(k_hmg_tail, fields_, kTailThreads, tp.total * sizeof(double), ctx_.stream, b, x, tp);
    ctx_.count_launch();
    ctx_.check_launch("hmg2d tail");
}

// The levels below the finest touch only the hierarchy's own arrays: captured once, then one launch.  Inside a caller's
// own capture of the stream their kernels go into that graph.
void HelmholtzMG2D::coarse_cycle() {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    NUMA_CUDA(cudaStreamIsCapturing(ctx_.stream, &cap));
    if (tail_l_ == 1 || cap != cudaStreamCaptureStatusNone) {  // (or one kernel: no graph)
        cycle(1);
        return;
    }
    if (!exec_) {
        // no other thread may allocate or free (and so synchronise the device) during the capture
        std::lock_guard<std::recursive_mutex> lk(alloc_capture_mutex());
        const uint64_t before = ctx_.launches;
        NUMA_CUDA(cudaStreamBeginCapture(ctx_.stream, cudaStreamCaptureModeThreadLocal));
        cudaGraph_t graph = nullptr;
        try {
            cycle(1);
        } catch (...) {
            cudaStreamEndCapture(ctx_.stream, &graph);
            if (graph) cudaGraphDestroy(graph);
            cudaGetLastError();
            throw;
        }
        NUMA_CUDA(cudaStreamEndCapture(ctx_.stream, &graph));
        const cudaError_t e = cudaGraphInstantiate(&exec_, graph, 0);
        cudaGraphDestroy(graph);
        NUMA_CUDA(e);
        graph_kernels_ = ctx_.launches - before;
        ctx_.launches = before;
    }
    NUMA_CUDA(cudaGraphLaunch(exec_, ctx_.stream));
    ctx_.count_launch(static_cast<unsigned>(graph_kernels_));
}

void HelmholtzMG2D::cycle(size_t l) {
    Level& L = *levels_[l];
    const int n = L.n;
    double* x = l == 0 ? x0_ : L.x.p;
    const double* b = l == 0 ? b0_ : L.b.p;
    if (l == tail_l_) {
        launch_tail(b, x);
        return;
    }
    const HLvl K = hlvl(n, L.s, alpha_);
    cudaStream_t st = ctx_.stream;
    if (L.T) {
        Level& C = *levels_[l + 1];
        auto tile = [&](int sweeps) {
            const int S = 2 * L.T + 1 + 4 * sweeps;
            return HTile{K, C.n, L.T, S, (S + 1) / 2, sweeps};
        };
        const unsigned k = (unsigned)((C.n + L.T - 1) / L.T);
        const dim3 grid(k, k, (unsigned)fields_);
        auto threads = [](const HTile& t) { return dim3((unsigned)((t.S * t.np + 31) / 32 * 32)); };
        auto smem = [](const HTile& t) { return ((size_t)(t.S + 2) * (t.S + 2) + (2 * t.T + 1) * (2 * t.T + 1)) * sizeof(double); };
        const HTile down = tile(pre_), up = tile(post_);
        launch_pdl(k_htile_down, grid, threads(down), smem(down), st, b, L.y.p, C.b.p, down);
        ctx_.count_launch();
        if (l == 0) coarse_cycle();
        else cycle(l + 1);
        launch_pdl(k_htile_up, grid, threads(up), smem(up), st, b, (const double*)L.y.p, (const double*)C.x.p, x, up);
        ctx_.count_launch();
        ctx_.check_launch("hmg2d tiled level");
        return;
    }
    const dim3 blk(BX, BY);
    const unsigned nf = (unsigned)fields_;
    const dim3 cg(((n + 1) / 2 + BX - 1) / BX, (n + BY - 1) / BY, nf);
    auto pass = [&](int colour, bool first) {
        if (first) launch_pdl(k_hsmooth<true>, cg, blk, 0, st, x, b, K, colour);
        else launch_pdl(k_hsmooth<false>, cg, blk, 0, st, x, b, K, colour);
        ctx_.count_launch();
    };
    auto sweep = [&](int order, bool first) {
        const int c0 = order == 0 ? 0 : 1;
        pass(c0, first);
        pass(1 - c0, false);
    };
    if (l + 1 == levels_.size()) {  // an even grid above kTailTop
        for (int sw = 0; sw < 30; ++sw) sweep(sw % 2, sw == 0);
        ctx_.check_launch("hmg2d coarsest");
        return;
    }
    for (int sw = 0; sw < pre_; ++sw) sweep(0, sw == 0);
    if (pre_ == 0) NUMA_CUDA(cudaMemsetAsync(x, 0, (size_t)fields_ * n * n * sizeof(double), st));
    const dim3 fg((n + BX - 1) / BX, (n + BY - 1) / BY, nf);
    launch_pdl(k_hresidual, fg, blk, 0, st, (const double*)x, b, resid_.p, K);
    Level& C = *levels_[l + 1];
    const int nc = C.n;
    launch_pdl(k_hrestrict, dim3((nc + BX - 1) / BX, (nc + BY - 1) / BY, nf), blk, 0, st, (const double*)resid_.p, C.b.p, n,
               nc);
    ctx_.count_launch(2);
    if (l == 0) coarse_cycle();
    else cycle(l + 1);
    if (post_ > 0) launch_pdl(k_hprolong<true>, cg, blk, 0, st, (const double*)C.x.p, x, nc, n);
    else launch_pdl(k_hprolong<false>, fg, blk, 0, st, (const double*)C.x.p, x, nc, n);
    ctx_.count_launch();
    for (int sw = 0; sw < post_; ++sw) sweep(1, false);
    ctx_.check_launch("hmg2d cycle");
}

void HelmholtzMG2D::apply(const double* r, double* z) {
    const double* b = r;
    if (r == z && tail_l_ != 0) {
        alias_.resize(fields_ * N0_);
        dev_copy(ctx_, r, alias_.p, fields_ * N0_);
        b = alias_.p;
    }
    x0_ = z;
    b0_ = b;
    cycle(0);
}

namespace {

// BurgersMGProvider: M^-1 applied to u and to v (burgers2d.hpp:228-243), the two halves of the vectors, as the
// two fields of one cycle.
class BurgersMGProvider : public Provider {
public:
    BurgersMGProvider(Context& ctx, size_t n, double nu, double dt, int pre, int post)
        : mg_(ctx, n, 1.0 / dt, nu, pre, post, 2) {}
    void make(const double*, const double*) override {}
    void apply(const double* r, double* z) override { mg_.apply(r, z); }
    int kind() const override { return NUMA_GPU_PRECOND_POISSON_MG; }

private:
    HelmholtzMG2D mg_;
};

}  // namespace

std::unique_ptr<Provider> make_burgers_mg_provider(Context& ctx, size_t n, double nu, double dt, int pre, int post) {
    return std::make_unique<BurgersMGProvider>(ctx, n, nu, dt, pre, post);
}

}  // namespace numa::gpu
