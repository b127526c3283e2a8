// mg_chain.cuh — the coarse end (31, 15, 7, 3, 1 or 15, 7, 3, 1) of a V-cycle whose grids are all 2^k - 1, in one
// kernel with every size at compile time.
//
// mg_coarse.cuh says why the coarse levels belong in one kernel; this is the form for the usual hierarchies.  On
// levels this small a step is bound by the latency of its dependent instructions (an FP64 operation takes ~65
// cycles, any other ~5), so everything a step would compute besides the points' own arithmetic is a constant or
// held in a register: a pass loads from one address register per colour with immediate offsets.
//
// Split.  FP32: 31^3 over a cluster of 8 CTAs (4 planes each), 15^3 and below in CTA 0.  FP64, whose pipe is 1/64
// as wide: 15^3 over 8 CTAs (2 planes each), 7^3 and below in CTA 0.  The levels of one CTA narrow with the grid:
// 15^3 on 16 warps, 7^3 on 7 behind a named barrier, 3^3 and the single point on one warp.  A slab's edge
// planes of x, and its first plane of the residual, are also written into the neighbour's halo (distributed
// shared memory), so that restriction and smoothing read their own CTA's memory only; the coarse b goes
// straight to CTA 0, and each CTA copies the coarse planes its interpolation reads.
//
// Layout.  x, b, r (and c h^2, 1 / (6 - c h^2) of Jacobian-aware levels) of a slab share one index: planes, rows and
// columns padded by a halo (of zeros for x: the Dirichlet values), pitch M = n + 2 odd, so the parity of a
// point's index P is its colour (plus one) and the two parities are stored apart (at par H + (P >> 1)): a pass
// writes one half and reads the other, each neighbour at a constant offset.
//
// The arithmetic is that of the launched kernels (mg_kernels.cuh) operation for operation: the same bits.
// acc / (6 - c h^2) is formed from d = 6 - c h^2 and RN(1/d) by Markstein's correction, the correctly rounded
// quotient inside the exponent range where the correction is exact, and by a division outside.
#pragma once

#include <cooperative_groups.h>

#include "mg_kernels.cuh"

namespace numa::gpu {

// Input of the top level: colour-split FP32, natural in the cycle's type, natural FP64 rounded to FP32.
enum ChainIn { kChainSplit = 0, kChainSame = 1, kChainF64 = 2 };

// What a launch reads and writes (null outputs: not written); c: the coefficients of -Lap_h - c on 15^3, 7^3, 3^3
// and the point (natural layout), for the Jacobian-aware form.
struct ChainIo {
    int in_kind, pre, post;
    int half;  // colour-0 points of the top level
    const void* b;
    float* x_split;
    void* x_nat;
    double* z64;
    const float* c[4];
};

namespace {

constexpr int kChainThreads = 512, kChainCluster = 8;

enum ChainBar { kBarCta, kBarGroup, kBarWarp, kBarCluster };
constexpr int kGroupThreads = 224;  // the warps of a 7^3 level

template <int BAR>
__device__ __forceinline__ void chain_sync() {
    if constexpr (BAR == kBarCluster) cooperative_groups::this_cluster().sync();
    else if constexpr (BAR == kBarCta) __syncthreads();
    else if constexpr (BAR == kBarGroup) asm volatile("bar.sync 1, %0;" ::"n"(kGroupThreads) : "memory");
    else __syncwarp();
}

// A level: N points a side, PL planes in a CTA, its arrays from element OFF of the shared memory on.
template <class T_, int N_, int PL_, bool WIDE_, int BAR_, bool SHIFT_, int OFF_>
struct ChainLv {
    using T = T_;
    static constexpr int N = N_, PL = PL_, BAR = BAR_;
    static constexpr bool WIDE = WIDE_, SHIFT = SHIFT_;
    static constexpr int M = N + 2, M2 = M * M, NP = (N + 1) / 2, COLS = N * NP;
    static constexpr int G = kChainThreads / COLS < PL ? kChainThreads / COLS : PL;  // plane groups
    static constexpr int U = (PL + G - 1) / G;                                      // planes a thread
    static constexpr int H = ((PL + 2) * M2 + 2) / 2;  // one parity
    // a point past the grid (masked at the store) may be loaded up to U G - PL planes behind the slab
    static constexpr int PAD = (U * G - PL) * M2 / 2 + M + 2;
    static constexpr int OX = OFF_, OB = OX + 2 * H + PAD, OC = OB + 2 * H + PAD;
    static constexpr int ORD = SHIFT ? OC + 2 * H + PAD : OC, END = SHIFT ? ORD + 2 * H + PAD : OC;
    static constexpr double H2 = double(N + 1) * (N + 1);  // h^-2 (a power of two, and so is its inverse)
    static_assert(!WIDE || PL % 2 == 0);
};

extern __shared__ __align__(16) unsigned char chain_smem[];
template <class T>
__device__ __forceinline__ T* chain_base() {
    return reinterpret_cast<T*>(chain_smem);
}

__device__ __forceinline__ unsigned chain_addr(const void* p, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void chain_store(unsigned a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void chain_store(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ float chain_load(unsigned a, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ double chain_load(unsigned a, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}

// A thread's column: row j, the points k = 2kk and 2kk + 1, planes g + u G.  e[c] = which of the two has colour c in
// plane g, q[c] its index there.
template <class L>
struct ChainCol {
    int g, j, kk, e0, q0, q1;  // colour 1's member is 1 - e0
    __device__ __forceinline__ ChainCol() {
        const int t = threadIdx.x;
        g = t / L::COLS;
        const int r = t - g * L::COLS;
        j = r / L::NP;
        kk = r - j * L::NP;
        const int P0 = ((g + 1) * L::M + j + 1) * L::M + 2 * kk + 1;
        e0 = (P0 ^ 1) & 1;  // colour 0 has parity 1
        q0 = (P0 + e0) >> 1;
        q1 = (P0 + 1 - e0) >> 1;
        if (g >= L::G) g = 1 << 16;  // no work
    }
    template <int C>
    __device__ __forceinline__ int member(int u) const {  // 0 or 1: the pair's member of colour C in plane g + u G
        return (C ? 1 - e0 : e0) ^ ((u * L::G) & 1);
    }
    // index (within its parity) of the point of colour C in plane g + u G
    template <int C>
    __device__ __forceinline__ int at(int u) const {
        const int odd = (u * L::G) & 1, first = C ? 1 - e0 : e0;
        return (C ? q1 : q0) + (u * L::G * L::M2 + odd) / 2 - (odd ? first : 0);
    }
    template <int C>
    __device__ __forceinline__ bool valid(int u, int my) const {
        return g + u * L::G < my && !(member<C>(u) && kk == L::NP - 1);
    }
};

// Stores x's value v of parity PAR at index i of plane li, and in the neighbours' halo planes.
template <class L, int PAR>
__device__ __forceinline__ void chain_put(typename L::T* X, int i, int li, int my, int rank, typename L::T v) {
    X[PAR * L::H + i] = v;
    if constexpr (L::WIDE) {
        constexpr int S = L::PL * L::M2 / 2;
        if (li == 0 && rank > 0) chain_store(chain_addr(X + PAR * L::H + i + S, rank - 1), v);
        if (li == L::PL - 1 && (rank + 1) * L::PL < L::N) chain_store(chain_addr(X + PAR * L::H + i - S, rank + 1), v);
    }
}

// Quotients a / d of a Jacobian-aware level, from rd = RN(1/d) and q = RN(a rd): the residual a - q d is exact, and the
// corrected quotient RN(a / d), where neither underflows.  chain_exact says so for |d| in [2^-20, 2^20] (elsewhere
// chain_recip gives a NaN): false for a too small, a zero, an infinity or a NaN.
__device__ __forceinline__ float chain_recip(float d) {
    return fabsf(d) >= 0x1p-20f && fabsf(d) <= 0x1p20f ? __frcp_rn(d) : __int_as_float(0x7fffffff);
}
__device__ __forceinline__ bool chain_exact(float a, float q) { return fabsf(a) >= 0x1p-100f && fabsf(q) <= 0x1p100f; }

// The pass at the thread's points by divisions: rare, behind the stores of the corrected quotients (no other thread reads
// those before the barrier) and out of line, so that the usual pass waits for nothing but the tests.  A V-cycle at 63^3
// takes 46.0 us, 45.65 without the tests and 46.85 with the divisions in the pass.
template <class L, int C>
__device__ __noinline__ void chain_pass_div(ChainCol<L> col, int my, bool zero_x) {
    using T = typename L::T;
    constexpr int PAR = 1 - C, M = L::M, M2 = L::M2;
    T* X = chain_base<T>() + L::OX;
    const T* o = X + (1 - PAR) * L::H;
    const T* B = chain_base<T>() + L::OB + PAR * L::H;
    constexpr T inv = T(1.0 / L::H2);
#pragma unroll 1
    for (int u = 0; u < L::U; ++u) {
        const int gu = col.g + u * L::G;
        if (gu >= my) break;
        const int P0 = ((gu + 1) * M + col.j + 1) * M + 2 * col.kk + 1;
        const int e = ((P0 ^ 1) & 1) ^ C;
        if (e && col.kk == L::NP - 1) continue;
        const int i = (P0 + e) >> 1;
        T acc = B[i] * inv;
        if (!zero_x) {
            acc = acc + o[i + ((PAR - M2) >> 1)];
            acc = acc + o[i + ((PAR + M2) >> 1)];
            acc = acc + o[i + ((PAR - M) >> 1)];
            acc = acc + o[i + ((PAR + M) >> 1)];
            acc = acc + o[i + ((PAR - 1) >> 1)];
            acc = acc + o[i + ((PAR + 1) >> 1)];
        }
        X[PAR * L::H + i] = acc / (T(6) - chain_base<T>()[L::OC + PAR * L::H + i]);
    }
}

template <class L, int C>
__device__ __forceinline__ void chain_pass(const ChainCol<L>& col, int my, int rank, bool zero_x) {
    using T = typename L::T;
    constexpr int PAR = 1 - C, M = L::M, M2 = L::M2;
    T* X = chain_base<T>() + L::OX;
    const T* o = X + (1 - PAR) * L::H;
    const T* B = chain_base<T>() + L::OB + PAR * L::H;
    constexpr T inv = T(1.0 / L::H2);
    if (col.g >= L::G) return;  // (in FP64 a warp's idle arithmetic would hold the pipe)
    T v[L::U];
    unsigned inexact = 0;
#pragma unroll
    for (int u = 0; u < L::U; ++u) {
        const int i = col.template at<C>(u);
        T acc = B[i] * inv;
        if (!zero_x) {
            // (PAR + d) >> 1 for odd d
            acc = acc + o[i + ((PAR - M2) >> 1)];
            acc = acc + o[i + ((PAR + M2) >> 1)];
            acc = acc + o[i + ((PAR - M) >> 1)];
            acc = acc + o[i + ((PAR + M) >> 1)];
            acc = acc + o[i + ((PAR - 1) >> 1)];
            acc = acc + o[i + ((PAR + 1) >> 1)];
        }
        if constexpr (L::SHIFT) {
            const T d = T(6) - chain_base<T>()[L::OC + PAR * L::H + i], rd = chain_base<T>()[L::ORD + PAR * L::H + i];
            const T qt = acc * rd;
            v[u] = fma_t(fma_t(-qt, d, acc), rd, qt);
            inexact |= (unsigned)(!chain_exact(acc, qt)) & (unsigned)col.template valid<C>(u, my);
        } else {
            v[u] = div6(acc);
        }
    }
#pragma unroll
    for (int u = 0; u < L::U; ++u)
        if (col.template valid<C>(u, my))
            chain_put<L, PAR>(X, col.template at<C>(u), col.g + u * L::G, my, rank, v[u]);
    if constexpr (L::SHIFT)
        if (inexact) chain_pass_div<L, C>(col, my, zero_x);
}

// `passes` colour passes, the first of colour c0; zero_x: x is zero before the first.
template <class L>
__device__ __noinline__ void chain_sweeps(int my, int rank, int passes, int c0, bool zero_x) {
    const ChainCol<L> col;
#pragma unroll 1
    for (int p = 0; p < passes; ++p) {
        if ((p ^ c0) & 1) chain_pass<L, 1>(col, my, rank, false);
        else chain_pass<L, 0>(col, my, rank, zero_x && p == 0);
        chain_sync<L::BAR>();
    }
}

// The residual at the thread's points of colour C
template <class L, int C>
__device__ __forceinline__ void chain_residual(const ChainCol<L>& col, typename L::T (&v)[L::U]) {
    using T = typename L::T;
    constexpr int PAR = 1 - C, M = L::M, M2 = L::M2;
    const T* X = chain_base<T>() + L::OX;
    const T* o = X + (1 - PAR) * L::H;
    const T* B = chain_base<T>() + L::OB + PAR * L::H;
    constexpr T h2inv = T(L::H2);
#pragma unroll
    for (int u = 0; u < L::U; ++u) {
        const int i = col.template at<C>(u);
        const T x = X[PAR * L::H + i];
        T s = T(6) * x;
        s = s - o[i + ((PAR - M2) >> 1)];
        s = s - o[i + ((PAR + M2) >> 1)];
        s = s - o[i + ((PAR - M) >> 1)];
        s = s - o[i + ((PAR + M) >> 1)];
        s = s - o[i + ((PAR - 1) >> 1)];
        s = s - o[i + ((PAR + 1) >> 1)];
        if constexpr (L::SHIFT) s = s - chain_base<T>()[L::OC + PAR * L::H + i] * x;
        v[u] = B[i] - h2inv * s;
    }
}

template <class L, int OR, int C>
__device__ __forceinline__ void chain_residual_put(const ChainCol<L>& col, int my, int rank,
                                                   const typename L::T (&v)[L::U]) {
    using T = typename L::T;
    T* R = chain_base<T>() + OR + (1 - C) * L::H;
#pragma unroll
    for (int u = 0; u < L::U; ++u) {
        if (!col.template valid<C>(u, my)) continue;
        const int i = col.template at<C>(u);
        R[i] = v[u];
        if constexpr (L::WIDE)  // plane 0 is the lower neighbour's plane PL
            if (col.g + u * L::G == 0 && rank > 0) chain_store(chain_addr(R + i + L::PL * L::M2 / 2, rank - 1), v[u]);
    }
}

// The residual of level F and its full weighting into b of level C (CTA 0's): the coarse plane I is formed by the
// CTA that holds fine planes 2I and 2I + 1.
template <class F, class C, int OR>
__device__ __noinline__ void chain_restrict(int my, int rank) {
    using T = typename F::T;
    {
        const ChainCol<F> col;
        if (col.g < F::G) {
            T v0[F::U], v1[F::U];
            chain_residual<F, 0>(col, v0);
            chain_residual<F, 1>(col, v1);
            chain_residual_put<F, OR, 0>(col, my, rank, v0);
            chain_residual_put<F, OR, 1>(col, my, rank, v1);
        }
    }
    chain_sync<F::BAR>();
    constexpr int NC = C::N, planes = F::WIDE ? F::PL / 2 : NC;
    constexpr int rounds = (planes * NC * NC + kChainThreads - 1) / kChainThreads;
#pragma unroll
    for (int round = 0; round < rounds; ++round) {
        const int t = threadIdx.x + round * kChainThreads, I = t / (NC * NC), r = t - I * NC * NC, J = r / NC, K = r - J * NC;
        const int Ig = F::WIDE ? rank * planes + I : I;
        if (I < planes && Ig < NC) {
            // padded index of fine point (2I, 2J, 2K): odd, so offset d has parity (1 + d) & 1
            const T* R = chain_base<T>() + OR + ((((2 * I + 1) * F::M + 2 * J + 1) * F::M + 2 * K + 1) >> 1);
            constexpr T w[3] = {T(0.25), T(0.5), T(0.25)};
            T acc = zero<T>();
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const int d = (a * F::M + b) * F::M + c;
                        acc = fma_t(w[a] * w[b] * w[c], R[((1 + d) & 1) * F::H + ((1 + d) >> 1)], acc);
                    }
            const int P = ((Ig + 1) * C::M + J + 1) * C::M + K + 1;
            T* B = chain_base<T>() + C::OB + (P & 1) * C::H + (P >> 1);
            if constexpr (F::WIDE) chain_store(chain_addr(B, 0), acc);
            else *B = acc;
        }
    }
    chain_sync<F::BAR>();
}

// x of level F += trilinear interpolation of level C's x at the points of colour 0.  A thread owns the coarse cell (I,
// J, K), the fine points (2I + a, 2J + b, 2K + c); absent coarse neighbours are halo zeros.
template <class F, class C, int OR>
__device__ __noinline__ void chain_prolong(int my, int rank) {
    using T = typename F::T;
    constexpr int NC1 = C::N + 1, cellp = F::WIDE ? F::PL / 2 : NC1;
    constexpr int rounds = (cellp * NC1 * NC1 + kChainThreads - 1) / kChainThreads;
    const T* XC = chain_base<T>() + C::OX;
    constexpr int HS = F::WIDE ? ((F::PL / 2 + 1) * C::M2 + 2) / 2 : C::H;
    const int t = threadIdx.x;
    if constexpr (F::WIDE) {
        // coarse planes PL/2 rank - 1 ... PL/2 rank + PL/2 - 1 (padded from PL/2 rank), parity by parity
        T* dst = chain_base<T>() + OR;
        const int Ps = rank * (F::PL / 2) * C::M2, odd = Ps & 1;
#pragma unroll
        for (int s = 0; s < (2 * HS + kChainThreads - 1) / kChainThreads; ++s) {
            const int q = t + s * kChainThreads, par = q >= HS, e = q - par * HS, se = e + ((Ps + par) >> 1);
            if (q < 2 * HS)
                dst[q] = se < C::H ? chain_load(chain_addr(XC + (par ^ odd) * C::H + se, 0), T(0)) : zero<T>();
        }
        XC = dst;
        __syncthreads();
    }
#pragma unroll
    for (int round = 0; round < rounds; ++round) {
        const int tc = t + round * kChainThreads, I = tc / (NC1 * NC1), r = tc - I * NC1 * NC1, J = r / NC1, K = r - J * NC1;
        if (I < cellp && 2 * I < my) {
            const int Pc = (I * C::M + J) * C::M + K, p0 = Pc & 1;
            const T* even = XC + p0 * HS + (Pc >> 1);              // even offsets d at d / 2
            const T* oddp = XC + (1 - p0) * HS + (Pc >> 1) + p0;   // odd ones at (d - 1) / 2
            T v[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                const int d = ((h >> 2) * C::M + ((h >> 1) & 1)) * C::M + (h & 1);
                v[h] = (d & 1) ? oddp[(d - 1) / 2] : even[d / 2];
            }
            T* X = chain_base<T>() + F::OX;
            const int P = (((2 * I + 1) * F::M + 2 * J + 1) * F::M + 2 * K + 1) >> 1;  // odd: parity 1 is colour 0
            const bool in[3] = {2 * I + 1 < my, J < C::N, K < C::N};
#pragma unroll
            for (int f = 0; f < 8; ++f) {
                const int a = f >> 2, b = (f >> 1) & 1, c = f & 1;
                if ((a + b + c) & 1) continue;
                const T w = (a ? T(1) : T(0.5)) * (b ? T(1) : T(0.5)) * (c ? T(1) : T(0.5));
                T acc = zero<T>();
#pragma unroll
                for (int h = 0; h < 8; ++h)
                    if (!((a && !(h >> 2)) || (b && !((h >> 1) & 1)) || (c && !(h & 1)))) acc = fma_t(w, v[h], acc);
                const int i = P + ((a * F::M + b) * F::M + c) / 2;
                if ((!a || in[0]) && (!b || in[1]) && (!c || in[2]))
                    chain_put<F, 1>(X, i, 2 * I + a, my, rank, X[F::H + i] + acc);
            }
        }
    }
    chain_sync<F::BAR>();
}

// c h^2 and RN(1 / (6 - c h^2)) of a Jacobian-aware level
template <class L>
__device__ __forceinline__ void chain_coef(const float* c) {
    for (int t = threadIdx.x; t < L::N * L::N * L::N; t += kChainThreads) {
        const int i = t / (L::N * L::N), r = t - i * L::N * L::N, j = r / L::N, k = r - j * L::N;
        const int P = ((i + 1) * L::M + j + 1) * L::M + k + 1, q = (P & 1) * L::H + (P >> 1);
        const float cs = c[t] * float(1.0 / L::H2);
        chain_base<float>()[L::OC + q] = cs;
        chain_base<float>()[L::ORD + q] = chain_recip(6.0f - cs);
    }
}

// b / 24: (b / 6) / 4 has one rounding where div6 is exact and the quarter does not underflow.
__device__ __forceinline__ float chain_div24(float b) {
    return fabsf(b) >= 0x1p-100f && fabsf(b) <= 0x1p127f ? div6(b) * 0.25f : b / 24.0f;
}
__device__ __forceinline__ double chain_div24(double b) {
    return fabs(b) >= 0x1p-960 && fabs(b) <= 0x1p1023 ? div6(b) * 0.25 : b / 24.0;
}

// The levels CTA 0 holds below level A (which it has restricted): 7^3 on its warps, 3^3 and the point on warp 0.
template <class L7, class L3, class L1, int OR>
__device__ __forceinline__ void chain_tail(const ChainIo& io, const float* c1) {
    using T = typename L7::T;
    if (threadIdx.x >= kGroupThreads) return;
    chain_sweeps<L7>(7, 0, 2 * io.pre, 0, true);
    chain_restrict<L7, L3, OR>(7, 0);
    if (threadIdx.x < 32) {
        chain_sweeps<L3>(3, 0, 2 * io.pre, 0, true);
        chain_restrict<L3, L1, OR>(3, 0);
        if (threadIdx.x == 0) {
            constexpr int q = L1::H + ((13 - 1) >> 1);  // the point's padded index is 13: parity 1
            const T b = chain_base<T>()[L1::OB + q];
            T v;
            if constexpr (L7::SHIFT) v = b / (T(24) - *c1);
            else v = chain_div24(b);
            chain_base<T>()[L1::OX + q] = v;
        }
        __syncwarp();
        chain_prolong<L3, L1, OR>(3, 0);
        chain_sweeps<L3>(3, 0, 2 * io.post, 1, false);
    }
    chain_sync<kBarGroup>();
    chain_prolong<L7, L3, OR>(7, 0);
    chain_sweeps<L7>(7, 0, 2 * io.post, 1, false);
}

// The top level's b from global memory, x to it: a thread's own points, all loads ahead of the stores.
template <class L>
__device__ __noinline__ void chain_load_top(int in_kind, int half, const void* b, int my, int rank) {
    using T = typename L::T;
    const ChainCol<L> col;
    if (col.g >= L::G) return;
    T v[L::U][2];
#pragma unroll
    for (int u = 0; u < L::U; ++u)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int li = col.g + u * L::G, g = ((rank * L::PL + li) * L::N + col.j) * L::N + 2 * col.kk + e;
            v[u][e] = zero<T>();
            if (li >= my || (e && col.kk == L::NP - 1)) continue;
            if (sizeof(T) == 4 && in_kind == kChainF64) v[u][e] = (T)f64_to_f32(static_cast<const double*>(b)[g]);
            else v[u][e] = static_cast<const T*>(b)[in_kind == kChainSplit ? split_at(g, half) : g];
        }
    T* B = chain_base<T>() + L::OB;
#pragma unroll
    for (int u = 0; u < L::U; ++u) {
        const int m0 = col.template member<0>(u);  // the pair's member of colour 0
        if (col.template valid<0>(u, my)) B[L::H + col.template at<0>(u)] = m0 ? v[u][1] : v[u][0];
        if (col.template valid<1>(u, my)) B[col.template at<1>(u)] = m0 ? v[u][0] : v[u][1];
    }
}
template <class L>
__device__ __noinline__ void chain_store_top(int half, float* x_split, void* x_nat, double* z64, int my, int rank) {
    using T = typename L::T;
    const ChainCol<L> col;
    if (col.g >= L::G) return;
    const T* X = chain_base<T>() + L::OX;
#pragma unroll
    for (int u = 0; u < L::U; ++u) {
        const int li = col.g + u * L::G, g0 = ((rank * L::PL + li) * L::N + col.j) * L::N + 2 * col.kk;
        const auto put = [&](int g, T v) {
            if constexpr (sizeof(T) == 4) {
                if (x_split) x_split[split_at(g, half)] = v;
                if (z64) z64[g] = f32_to_f64(v);
            }
            if (x_nat) static_cast<T*>(x_nat)[g] = v;
        };
        const int m0 = col.template member<0>(u);
        if (col.template valid<0>(u, my)) put(g0 + m0, X[L::H + col.template at<0>(u)]);
        if (col.template valid<1>(u, my)) put(g0 + 1 - m0, X[col.template at<1>(u)]);
    }
}

// The level tables: FP32 with 31^3 on top (PL planes a CTA), FP64 with 15^3.
template <bool SHIFT, int PL = 4>
struct Chain32 {
    using T = float;
    using L31 = ChainLv<float, 31, PL, true, kBarCluster, false, 0>;
    using L15 = ChainLv<float, 15, 15, false, kBarCta, SHIFT, L31::END>;
    using L7 = ChainLv<float, 7, 7, false, kBarGroup, SHIFT, L15::END>;
    using L3 = ChainLv<float, 3, 3, false, kBarWarp, SHIFT, L7::END>;
    using L1 = ChainLv<float, 1, 1, false, kBarWarp, false, L3::END>;
    static constexpr int OR = L1::END, TOTAL = OR + 2 * (L31::H + L31::PAD);
};
struct Chain64 {
    using T = double;
    using L15 = ChainLv<double, 15, 2, true, kBarCluster, false, 0>;
    using L7 = ChainLv<double, 7, 7, false, kBarGroup, false, L15::END>;
    using L3 = ChainLv<double, 3, 3, false, kBarWarp, false, L7::END>;
    using L1 = ChainLv<double, 1, 1, false, kBarWarp, false, L3::END>;
    static constexpr int OR = L1::END, R15 = L15::H + L15::PAD, R7 = L7::H + L7::PAD;
    static constexpr int TOTAL = OR + 2 * (R15 > R7 ? R15 : R7);
};

// x must start from zero halos; everything else is written before it is read (points past the grid may be
// loaded but never stored).
template <class L>
__device__ __forceinline__ void chain_clear() {
    typename L::T* X = chain_base<typename L::T>() + L::OX;
    for (int t = threadIdx.x; t < 2 * L::H; t += kChainThreads) X[t] = zero<typename L::T>();
}
template <class K>
__device__ __forceinline__ void chain_clear_below31() {
    chain_clear<typename K::L15>();
    chain_clear<typename K::L7>();
    chain_clear<typename K::L3>();
    chain_clear<typename K::L1>();
}

// 15^3 and below in one CTA (FP32).
template <class K, bool SHIFT>
__device__ __forceinline__ void chain_solo15(const ChainIo& io, const float* c1) {
    using L15 = typename K::L15;
    using L7 = typename K::L7;
    chain_sweeps<L15>(15, 0, 2 * io.pre, 0, true);
    chain_restrict<L15, L7, K::OR>(15, 0);
    chain_tail<L7, typename K::L3, typename K::L1, K::OR>(io, c1);
    __syncthreads();
    chain_prolong<L15, L7, K::OR>(15, 0);
    chain_sweeps<L15>(15, 0, 2 * io.post, 1, false);
}

// (q: the grid of a batch)
template <class K, bool SHIFT>
__device__ __forceinline__ void chain_coefs(const ChainIo& io, size_t q) {
    if constexpr (SHIFT) {
        chain_coef<typename K::L15>(io.c[0] + q * 3375);
        chain_coef<typename K::L7>(io.c[1] + q * 343);
        chain_coef<typename K::L3>(io.c[2] + q * 27);
    }
}

// The cycle from 31^3 (b loaded) on a cluster, in FP32.
template <bool SHIFT, int PL = 4>
__device__ __forceinline__ void chain_cycle31(const ChainIo& io, const float* c1, int my, int rank) {
    using K = Chain32<SHIFT, PL>;
    using L31 = typename K::L31;
    chain_sweeps<L31>(my, rank, 2 * io.pre, 0, true);
    chain_restrict<L31, typename K::L15, K::OR>(my, rank);
    if (rank == 0) chain_solo15<K, SHIFT>(io, c1);
    cooperative_groups::this_cluster().sync();
    chain_prolong<L31, typename K::L15, K::OR>(my, rank);
    chain_sweeps<L31>(my, rank, 2 * io.post, 1, false);
}

// 31, 15, 7, 3, 1 in FP32 on a cluster of 8
template <bool SHIFT>
__global__ void __launch_bounds__(kChainThreads, 1) k_chain32(const __grid_constant__ ChainIo io) {
    using K = Chain32<SHIFT>;
    using L31 = typename K::L31;
    const int rank = (int)cooperative_groups::this_cluster().block_rank(), my = min(4, 31 - 4 * rank);
    chain_clear<L31>();
    if (rank == 0) chain_clear_below31<K>();
    cooperative_groups::this_cluster().sync();  // a neighbour's first halo store comes after the clearing
    pdl_wait();
    pdl_trigger();
    chain_load_top<L31>(io.in_kind, io.half, io.b, my, rank);
    if (rank == 0) chain_coefs<K, SHIFT>(io, 0);
    __syncthreads();
    chain_cycle31<SHIFT>(io, SHIFT ? io.c[3] : nullptr, my, rank);
    chain_store_top<L31>(io.half, io.x_split, io.x_nat, io.z64, my, rank);
    cooperative_groups::this_cluster().sync();  // no CTA leaves while another may write its halo
}

// 15, 7, 3, 1 in FP64 on a cluster of 8
__global__ void __launch_bounds__(kChainThreads, 1) k_chain64(const __grid_constant__ ChainIo io) {
    using K = Chain64;
    using L15 = K::L15;
    const int rank = (int)cooperative_groups::this_cluster().block_rank(), my = min(2, 15 - 2 * rank);
    chain_clear_below31<K>();
    cooperative_groups::this_cluster().sync();
    pdl_wait();
    pdl_trigger();
    chain_load_top<L15>(io.in_kind, io.half, io.b, my, rank);
    __syncthreads();
    chain_sweeps<L15>(my, rank, 2 * io.pre, 0, true);
    chain_restrict<L15, K::L7, K::OR>(my, rank);
    if (rank == 0) chain_tail<K::L7, K::L3, K::L1, K::OR>(io, nullptr);
    cooperative_groups::this_cluster().sync();
    chain_prolong<L15, K::L7, K::OR>(my, rank);
    chain_sweeps<L15>(my, rank, 2 * io.post, 1, false);
    chain_store_top<L15>(io.half, nullptr, io.x_nat, nullptr, my, rank);
    cooperative_groups::this_cluster().sync();
}

}  // namespace
}  // namespace numa::gpu
