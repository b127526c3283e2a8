// mg_coarse.cuh — the coarse end of an FP64 Poisson V-cycle as one kernel: every level from the first of
// n <= 15 points a side down to the coarsest and back, in the shared memory of one thread-block cluster.
//
// Why.  A launched pass over such a level costs its launch (2.2-2.6 us with programmatic dependent launch
// inside a graph), not its work, and a level is 11 such steps (60 passes more where the hierarchy ends in an
// even grid).  Here a step is a barrier: a V(2,2) at 7^3 takes 19 us instead of 37, at 11^3 (11, 5, 2) 31 instead of
// 103, at 23^3 (23, 11, 5, 2) 54 instead of 134, at 95^3 202 instead of 259.  What bounds it now is latency: the eight
// dependent FP64 operations of a point are ~520 of a pass's ~1,000 cycles on the small levels.  (Hierarchies of 2^k - 1
// points down to one, from 15^3 on, take mg_chain.cuh's form with its sizes at compile time.)
//
// Split of the work.  FP64 runs at two operations a clock on an SM, so one SM's pass over 15^3 takes 6,700
// cycles: the top level, where it is larger than 7 points a side, is cut into slabs of pl i-planes (an
// even number), one per CTA of a cluster of 8 (16 CTAs measured the same: barriers then cost what the
// halved work saves).  A point on a slab's edge is also written into the neighbour's halo plane (distributed
// shared memory) by the pass that updates it; the cluster barrier after the pass (~550 cycles) makes it
// visible.  The smaller levels live in CTA 0 behind block barriers (~100 cycles); the other CTAs wait at the
// next cluster barrier.  Both ends of the step between the slabs and CTA 0 are spread: each CTA restricts its
// own planes' part into CTA 0's b, and copies the planes of CTA 0's x that its own interpolation reads (one
// SM reading all the others' planes, or all of them reading one SM's, took 13 us at 31^3).
// The same kernel in FP32 was no faster than the launched levels and their one-CTA tail (k_mg_tail), whose
// arithmetic costs so little that its compile-time sizes decide; a top level of 31^3 was no faster either.
//
// Layout.  x of a slab has a halo of zeros on every side (the Dirichlet values: adding +0.0 is what the
// launched kernels' selects do), pitch m = (n + 2) | 1 in k and j, so plane and row strides are odd and
// the parity of a point's padded index is its colour up to a constant of the slab.  The two parities are
// stored apart: a colour pass reads one half and writes the other with unit stride, each neighbour
// at a fixed offset ((par + d) >> 1 for d = +-1, +-m, +-m^2).  b and r are in natural order.  A thread
// owns a (j, k-pair) column of every G-th plane.  Each operation exists once, in a function that is not
// inlined: with unrolled, inlined passes the warps waited for instructions (9.5 of 14 warps in the profile).
//
// The arithmetic of every step is that of the launched kernels (mg_kernels.cuh) operation for
// operation, so the cycle has the same bits whichever way its levels run.
#pragma once

#include <cooperative_groups.h>

#include <algorithm>

#include "mg_kernels.cuh"

namespace numa::gpu {

constexpr int kCoarseMax = 8;  // levels of one launch
// Sizes: the cycle runs in the coarse kernel from the first level of n <= top; its levels of n <= solo are
// held by one CTA.
constexpr int kCoarseTop = 15, kCoarseSolo = 7;
constexpr int kCoarseCluster = 8;
constexpr int kCoarseThreads = 512;
static_assert(kCoarseTop * ((kCoarseTop + 1) / 2) <= kCoarseThreads, "a thread for each pair of a plane");

struct CoarseLvl {
    int n, m, pl, owners;  // pitch, planes a CTA, CTAs that own planes
    int H;                 // elements of one parity of x (x: 2 H)
    int offX, offB;        // element offsets in the CTA's shared memory
    int cols, G;           // (j, k-pair) columns of a plane, groups of threads that share out the planes
    unsigned mnp, mn, mcols, mcell;  // ceil(2^32 / d) for d = pairs a row, n, cols, n + 1 (0: d = 1)
    double h2inv, inv;               // h^-2, 1 / h^-2
};

struct CoarseParams {
    int levels, pre, post;
    int cluster;  // CTAs
    int offR;     // residual scratch; the copy of a coarse level's planes
    int total;    // elements of shared memory
    CoarseLvl L[kCoarseMax];
};

namespace {

// The kernel's state in shared memory: the parameters (dynamic indexing from registers would go through
// local memory) and the arrays behind them.
struct CoarseShared {
    CoarseParams cp;
    int rank, size;  // of the cluster
};

extern __shared__ __align__(16) unsigned char coarse_smem[];
__device__ __forceinline__ CoarseShared& coarse_sh() {
    return *reinterpret_cast<CoarseShared*>(coarse_smem);
}
constexpr int kCoarseHeader = (int)((sizeof(CoarseShared) + 15) / 16 * 16);
__device__ __forceinline__ double* coarse_base() {
    return reinterpret_cast<double*>(coarse_smem + kCoarseHeader);
}

// Shared-memory addresses of the cluster's CTAs, and accesses to them (a CTA's own addresses are valid there).
__device__ __forceinline__ unsigned cl_addr(const void* p, int rank, int size) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p);
    if (size > 1) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(a), "r"(rank));
    return a;
}
__device__ __forceinline__ void cl_store(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// (not volatile, so that a thread's loads overlap: the functions that use them contain no barrier)
__device__ __forceinline__ void cl_load(unsigned a, double& v) {
    asm("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
}

__device__ __forceinline__ int fast_div(int t, unsigned magic) { return magic ? (int)__umulhi((unsigned)t, magic) : t; }

// Planes of level L in CTA rank's slab (<= 0: none).
__device__ __forceinline__ int coarse_planes(const CoarseLvl& L, int rank) {
    return min(L.pl, L.n - rank * L.pl);
}

// A thread's column of a level: row j, the points k = 2kk and 2kk + 1, planes g, g + G, ... of the slab (g >= the
// slab's planes: no work).  P0, nat0: padded and natural index of k = 2kk in plane 0.
struct CoarseCol {
    int g, G, j, k0, P0, nat0;
    bool two;  // the second point is inside the grid
};
__device__ __forceinline__ CoarseCol coarse_col(const CoarseLvl& L) {
    const int n = L.n, np = (n + 1) >> 1;
    CoarseCol c;
    c.G = L.G;
    c.g = fast_div((int)threadIdx.x, L.mcols);
    const int t = (int)threadIdx.x - c.g * L.cols;
    if (c.g >= c.G) c.g = 1 << 20;
    c.j = fast_div(t, L.mnp);
    c.k0 = 2 * (t - c.j * np);
    c.P0 = (L.m + c.j + 1) * L.m + c.k0 + 1;
    c.nat0 = c.j * n + c.k0;
    c.two = c.k0 + 1 < n;
    return c;
}

// Stores v at padded index P of the level and in the neighbours' halo planes: plane 0 of my slab is plane
// pl + 1 of the lower neighbour's, my last plane (pl) is plane 0 of the upper one's.
__device__ __forceinline__ void coarse_put(const CoarseLvl& L, double* X, int rank, int size, int my, int li, int P, double v) {
    X[(P & 1) * L.H + (P >> 1)] = v;
    if (L.owners > 1) {
        const int shift = L.pl * L.m * L.m;
        if (li == 0 && rank > 0) {
            const int Q = P + shift;
            cl_store(cl_addr(X + (Q & 1) * L.H + (Q >> 1), rank - 1, size), v);
        }
        if (li == my - 1 && rank + 1 < L.owners) {
            const int Q = P - shift;
            cl_store(cl_addr(X + (Q & 1) * L.H + (Q >> 1), rank + 1, size), v);
        }
    }
}

// After a step of a level cut over the cluster (wide), or of one that CTA 0 holds.
__device__ __forceinline__ void coarse_sync(bool wide) {
    if (wide) cooperative_groups::this_cluster().sync();
    else __syncthreads();
}

// Sweeps of level l: x = (b h^2 + the six neighbours) / 6, or / (6 - c h^2), colour order 0, 1 (order 0) or
// 1, 0; alternate: the order changes from sweep to sweep (the coarsest level); first: the first pass starts
// from x = 0 and reads no neighbours.
__device__ __noinline__ void coarse_sweeps(int l, int sweeps, int order, bool alternate, bool first) {
    const CoarseShared& S = coarse_sh();
    const CoarseLvl L = S.cp.L[l];  // a copy: the stores below could alias the shared table
    const int rank = S.rank, size = S.size;
    const CoarseCol col = coarse_col(L);
    double* base = coarse_base();
    const int my = coarse_planes(L, rank);
    const int n2 = L.n * L.n, m = L.m, M2 = m * m;
    double* X = base + L.offX;
    const double* B = base + L.offB;
    const double inv = L.inv;
#pragma unroll 1
    for (int p = 0; p < 2 * sweeps; ++p) {
        const int colour = (p & 1) ^ (alternate ? (p >> 1) & 1 : order);
        const int par = (1 + colour + rank * L.pl) & 1;  // parity of the pass's points
        const double* oth = X + (par ^ 1) * L.H;
        const int ip = (par + M2) >> 1, im = (par - M2) >> 1, jp = (par + m) >> 1, jm = (par - m) >> 1;
        const int kp = (par + 1) >> 1, km = (par - 1) >> 1;
#pragma unroll 1
        for (int li = col.g; li < my; li += col.G) {
            const int P = col.P0 + li * M2, e = (P ^ par) & 1;
            if (e && !col.two) continue;
            double acc = B[col.nat0 + li * n2 + e] * inv;
            if (!first || p > 0) {
                const double* o = oth + ((P + e) >> 1);
                acc = acc + o[im];
                acc = acc + o[ip];
                acc = acc + o[jm];
                acc = acc + o[jp];
                acc = acc + o[km];
                acc = acc + o[kp];
            }
            coarse_put(L, X, rank, size, my, li, P + e, div6(acc));
        }
        coarse_sync(L.owners > 1);
    }
}

// The 30 alternating sweeps of a coarsest level of 2^3 points (in CTA 0): lane p of warp 0 holds point p = 4i + 2j + k,
// whose only neighbours are p ^ 4, p ^ 2 and p ^ 1 (i, j, k in that order; the absent ones would add +0.0).  Sixty
// passes of the general form took 33 us a cycle, most of it indexing and FP64 additions of zeros.
__device__ __noinline__ void coarse_sweeps2(int l) {
    const CoarseLvl L = coarse_sh().cp.L[l];
    double* base = coarse_base();
    if (threadIdx.x < 32) {
        const int p = threadIdx.x & 7, colour = __popc(p) & 1;
        const double bs = base[L.offB + p] * L.inv;
        double x = 0.0;
#pragma unroll 1
        for (int pass = 0; pass < 60; ++pass) {
            const int c = (pass & 1) ^ ((pass >> 1) & 1);
            double acc = bs;
            acc = acc + __shfl_xor_sync(0xffffffffu, x, 4);
            acc = acc + __shfl_xor_sync(0xffffffffu, x, 2);
            acc = acc + __shfl_xor_sync(0xffffffffu, x, 1);
            if (c == colour) x = div6(acc);
        }
        if (threadIdx.x < 8) {
            const int P = ((1 + (p >> 2)) * L.m + 1 + ((p >> 1) & 1)) * L.m + 1 + (p & 1);
            base[L.offX + (P & 1) * L.H + (P >> 1)] = x;
        }
    }
    __syncthreads();
}

// r = b - h^-2 (6x - sum of neighbours) at the slab's points
__device__ __noinline__ void coarse_residual(int l) {
    const CoarseShared& S = coarse_sh();
    const CoarseLvl L = S.cp.L[l];
    const CoarseCol col = coarse_col(L);
    double* base = coarse_base();
    const int my = coarse_planes(L, S.rank);
    const int n2 = L.n * L.n, m = L.m, M2 = m * m;
    const double* __restrict__ X = base + L.offX;
    const double* __restrict__ B = base + L.offB;
    double* __restrict__ R = base + S.cp.offR;
    const double h2inv = L.h2inv;
#pragma unroll 1
    for (int l0 = col.g; l0 < my; l0 += 2 * col.G) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // two planes, both points of the pair (x is only read: no store waits)
            const int li = l0 + (u >> 1) * col.G, h = u & 1;
            if (li >= my || (h && !col.two)) continue;
            const int P = col.P0 + li * M2 + h, par = P & 1, q = P >> 1, nat = col.nat0 + li * n2 + h;
            const double* o = X + (par ^ 1) * L.H + q;
            const double x = X[par * L.H + q];
            double s = 6.0 * x;
            s = s - o[(par - M2) >> 1];
            s = s - o[(par + M2) >> 1];
            s = s - o[(par - m) >> 1];
            s = s - o[(par + m) >> 1];
            s = s - o[(par - 1) >> 1];
            s = s - o[(par + 1) >> 1];
            R[nat] = B[nat] - h2inv * s;
        }
    }
    coarse_sync(L.owners > 1);
}

// b of level l + 1 (in CTA 0): the 27-point full weighting of level l's residual in k_restrict's order (nf =
// 2 nc + 1, so every fine point exists).  The coarse plane I is formed by the CTA that holds fine planes 2I
// and 2I + 1; plane 2I + 2 may be the next CTA's first.
__device__ __noinline__ void coarse_restrict(int l) {
    const CoarseShared& S = coarse_sh();
    const CoarseLvl F = S.cp.L[l], C = S.cp.L[l + 1];
    const int rank = S.rank, size = S.size;
    double* base = coarse_base();
    const bool wide = F.owners > 1;
    const int nc = C.n, nf = F.n, nn = nc * nc;
    const int I0 = wide ? rank * (F.pl >> 1) : 0, I1 = wide ? min(I0 + (F.pl >> 1), nc) : nc;
    const double* R = base + S.cp.offR;
    const unsigned Bc = cl_addr(base + C.offB, 0, size);
#pragma unroll 1
    for (int t = threadIdx.x; t < (I1 - I0) * nn; t += kCoarseThreads) {
        const int row = fast_div(t, C.mn), K = t - row * nc;
        const int li = fast_div(row, C.mn), J = row - li * nc;
        double acc = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            int fi = 2 * li + a, o = rank;  // plane within the slab
            if (wide && fi == F.pl) {
                fi = 0;
                o = rank + 1;
            }
            const unsigned pln = cl_addr(R + (fi * nf + 2 * J) * nf + 2 * K, o, size);
            const double wa = a == 1 ? 0.5 : 0.25;
            double v[9];
#pragma unroll
            for (int b = 0; b < 3; ++b)
#pragma unroll
                for (int c = 0; c < 3; ++c) cl_load(pln + (unsigned)((b * nf + c) * sizeof(double)), v[b * 3 + c]);
#pragma unroll
            for (int b = 0; b < 3; ++b)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    acc = fma_t(wa * (b == 1 ? 0.5 : 0.25) * (c == 1 ? 0.5 : 0.25), v[b * 3 + c], acc);
        }
        cl_store(Bc + (unsigned)((I0 * nn + t) * sizeof(double)), acc);
    }
    coarse_sync(wide);
}

// x of level l += trilinear interpolation of level l + 1's x (in CTA 0), in k_prolong's order: at the points of
// colour 0, or at all (`both`).  An absent coarse neighbour is a halo zero (its term adds +0.0).  A slab reads
// the coarse planes pl/2 rank - 1 ... pl/2 rank + pl/2 - 1, which its CTA first copies beside it.
__device__ __noinline__ void coarse_prolong(int l, bool both) {
    const CoarseShared& S = coarse_sh();
    const CoarseLvl F = S.cp.L[l], C = S.cp.L[l + 1];
    const int rank = S.rank, size = S.size;
    double* base = coarse_base();
    const bool wide = F.owners > 1;
    const int my = coarse_planes(F, rank);
    const int M2c = C.m * C.m;
    double* X = base + F.offX;
    const double* XC = base + C.offX;
    int Hc = C.H, Ic = -1;  // XC holds the coarse planes Ic, Ic + 1, ...
    if (wide) {
        Ic = rank * (F.pl >> 1) - 1;
        const int Ps = (Ic + 1) * M2c, len = ((F.pl >> 1) + 1) * M2c;  // padded range of those planes
        // parity by parity: element e of the copy is element e + (Ps >> 1) of CTA 0's (one more where Ps is odd)
        Hc = (len + 2) >> 1;
        double* dst = base + S.cp.offR;
        const unsigned src = cl_addr(XC, 0, size);
        const int odd = Ps & 1;
#pragma unroll 2
        for (int t = threadIdx.x; t < 2 * Hc; t += kCoarseThreads) {
            const int par = t >= Hc, e = t - par * Hc;  // parity within the copy
            const int sp = par ^ odd, se = e + ((Ps + par) >> 1);
            double v = 0.0;
            if (rank * F.pl < F.n && se < C.H) cl_load(src + (unsigned)((sp * C.H + se) * sizeof(double)), v);
            dst[t] = v;
        }
        XC = dst;
        __syncthreads();
    }
    // a thread owns the coarse cell (I, J, K), i.e. the fine points (2I + a, 2J + b, 2K + c) inside the grid: an
    // even index has the coarse neighbours f/2 - 1 and f/2 with weight 1/2, an odd one (f - 1)/2 with weight 1
    const int nc1 = C.n + 1, cells = nc1 * nc1;
    const int cellI0 = wide ? rank * (F.pl >> 1) : 0;
    const int cnt = max(0, (my + 1) >> 1);  // cell planes of the slab
#pragma unroll 1
    for (int t = threadIdx.x; t < cnt * cells; t += kCoarseThreads) {
        const int row = fast_div(t, C.mcell), K = t - row * nc1;
        const int lI = fast_div(row, C.mcell), J = row - lI * nc1;
        const int Pc = ((cellI0 + lI - 1 - Ic) * C.m + J) * C.m + K;  // padded: coarse (I - 1, J - 1, K - 1)
        double v[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            const int Q = Pc + (h >> 2) * M2c + ((h >> 1) & 1) * C.m + (h & 1);
            v[h] = XC[(Q & 1) * Hc + (Q >> 1)];
        }
        const int P00 = ((2 * lI + 1) * F.m + 2 * J + 1) * F.m + 2 * K + 1;
        const bool in[3] = {2 * lI + 1 < my, 2 * J + 1 < F.n, 2 * K + 1 < F.n};
#pragma unroll
        for (int f = 0; f < 8; ++f) {
            const int a = f >> 2, b = (f >> 1) & 1, c = f & 1;
            if (((a + b + c) & 1) && !both) continue;
            if ((a && !in[0]) || (b && !in[1]) || (c && !in[2])) continue;
            const double w = (a ? 1.0 : 0.5) * (b ? 1.0 : 0.5) * (c ? 1.0 : 0.5);
            double acc = 0.0;
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                if ((a && !(h >> 2)) || (b && !((h >> 1) & 1)) || (c && !(h & 1))) continue;
                acc = fma_t(w, v[h], acc);
            }
            const int P = P00 + (a * F.m + b) * F.m + c;
            coarse_put(F, X, rank, size, my, 2 * lI + a, P, X[(P & 1) * F.H + (P >> 1)] + acc);
        }
    }
    coarse_sync(wide);
}

// The top level's b from global memory into the slab's buffer.
__device__ __noinline__ void coarse_load_top(const double* b_in) {
    const CoarseShared& S = coarse_sh();
    const CoarseLvl& L = S.cp.L[0];
    double* B = coarse_base() + L.offB;
    const int nn = L.n * L.n, total = coarse_planes(L, S.rank) * nn, g0 = S.rank * L.pl * nn;
#pragma unroll 4
    for (int t = threadIdx.x; t < total; t += kCoarseThreads) B[t] = b_in[g0 + t];
}

// The top level's x to global memory.
__device__ __noinline__ void coarse_store_top(double* x_out) {
    const CoarseShared& S = coarse_sh();
    const CoarseLvl L = S.cp.L[0];
    const double* X = coarse_base() + L.offX;
    const int n = L.n, nn = n * n, total = coarse_planes(L, S.rank) * nn, g0 = S.rank * L.pl * nn;
#pragma unroll 1
    for (int t = threadIdx.x; t < total; t += kCoarseThreads) {
        const int row = fast_div(t, L.mn), li = fast_div(row, L.mn), k = t - row * n;
        const int P = (row + li * (L.m - n) + L.m + 1) * L.m + k + 1;
        x_out[g0 + t] = X[(P & 1) * L.H + (P >> 1)];
    }
}

// The cycle x_out = V(b_in), natural order (b_in and x_out may be the same array: a CTA has its b before it
// writes its x).  Called by every thread of every CTA of the cluster after coarse_begin and pdl_wait.
__device__ __forceinline__ void coarse_cycle(const double* b_in, double* x_out) {
    const CoarseShared& S = coarse_sh();
    const CoarseParams& cp = S.cp;
    double* base = coarse_base();
    const int rank = S.rank, last = cp.levels - 1;
    coarse_load_top(b_in);
    __syncthreads();
    const bool wide = cp.L[0].owners > 1;
#pragma unroll 1
    for (int l = 0; l < last; ++l) {
        coarse_sweeps(l, cp.pre, 0, false, true);  // (pre = 0: x is zero, as coarse_begin left it)
        coarse_residual(l);
        coarse_restrict(l);
        if (rank != 0) break;  // the levels below the top are CTA 0's
    }
    if (rank == 0 || last == 0) {
        const CoarseLvl& C = cp.L[last];
        if (C.n == 1) {
            if (threadIdx.x == 0) {
                const int P = (C.m + 1) * C.m + 1;
                base[C.offX + (P & 1) * C.H + (P >> 1)] = base[C.offB] / (6.0 * C.h2inv);
            }
            __syncthreads();
        } else if (C.n == 2) {
            coarse_sweeps2(last);
        } else {
            coarse_sweeps(last, 30, 0, true, true);
        }
    }
#pragma unroll 1
    for (int l = rank == 0 ? last - 1 : (last > 0 ? 0 : -1); l >= 0; --l) {
        if (l == 0 && wide) coarse_sync(true);  // CTA 0 has finished the levels it holds
        coarse_prolong(l, cp.post == 0);
        coarse_sweeps(l, cp.post, 1, false, false);
    }
    coarse_store_top(x_out);
    if (S.size > 1) cooperative_groups::this_cluster().sync();  // no CTA leaves while another reads its memory
}

// Copies the parameters in and clears the arrays (the halos must be zero); the cluster barrier keeps a
// neighbour's first halo store behind the clearing.  Touches shared memory only, so it may run before pdl_wait.
__device__ __forceinline__ void coarse_begin(const CoarseParams& cp, int rank, int size) {
    CoarseShared& S = coarse_sh();
    double* base = coarse_base();
    const int* src = reinterpret_cast<const int*>(&cp);
    int* dst = reinterpret_cast<int*>(&S.cp);
    for (int t = threadIdx.x; t < (int)(sizeof(cp) / 4); t += kCoarseThreads) dst[t] = src[t];
    if (threadIdx.x == 0) {
        S.rank = rank;
        S.size = size;
    }
    for (int t = threadIdx.x; t < cp.total; t += kCoarseThreads) base[t] = 0.0;
    coarse_sync(size > 1);
}

__global__ void __launch_bounds__(kCoarseThreads, 1) k_mg_coarse(const __grid_constant__ CoarseParams cp,
                                                                 const double* b_in, double* x_out) {
    coarse_begin(cp, (int)cooperative_groups::this_cluster().block_rank(), (int)gridDim.x);
    pdl_wait();
    pdl_trigger();
    coarse_cycle(b_in, x_out);
}

// ------------------------------------------------------------------------------ host side
inline unsigned magic_div(int d) { return d > 1 ? 0xFFFFFFFFu / (unsigned)d + 1u : 0u; }

// Fills the level table and the shared-memory layout for the sizes n[0..levels) of the cycle; returns the bytes
// of shared memory a CTA needs.
inline size_t coarse_layout(CoarseParams& cp, const int* n, const double* h2inv, int levels) {
    cp.levels = levels;
    cp.cluster = n[0] <= kCoarseSolo ? 1 : kCoarseCluster;
    int off = 0, r = 0;
    for (int l = 0; l < levels; ++l) {
        CoarseLvl& L = cp.L[l];
        L.n = n[l];
        L.m = (n[l] + 2) | 1;
        const int C = n[l] <= kCoarseSolo ? 1 : kCoarseCluster;
        L.pl = C == 1 ? n[l] : ((n[l] + C - 1) / C + 1) / 2 * 2;  // even: fine planes 2I, 2I + 1 in one slab
        L.owners = (n[l] + L.pl - 1) / L.pl;
        L.H = ((L.pl + 2) * L.m * L.m + 2) / 2;
        L.cols = n[l] * ((n[l] + 1) / 2);
        L.G = kCoarseThreads / L.cols;
        L.mnp = magic_div((n[l] + 1) / 2);
        L.mn = magic_div(n[l]);
        L.mcols = magic_div(L.cols);
        L.mcell = magic_div(n[l] + 1);
        L.h2inv = h2inv[l];
        L.inv = (1.0 / h2inv[l]);
        L.offX = off;
        off += 2 * L.H;
        L.offB = off;
        off += L.pl * n[l] * n[l];
        // residual scratch, or the copy of the coarse planes a slab interpolates from
        r = std::max(r, L.pl * n[l] * n[l]);
        if (L.owners > 1 && l + 1 < levels) {
            const int mc = (n[l + 1] + 2) | 1;
            r = std::max(r, (L.pl / 2 + 1) * mc * mc + 4);
        }
    }
    cp.offR = off;
    off += r;
    cp.total = off;
    return (size_t)kCoarseHeader + (size_t)off * sizeof(double);
}

}  // namespace
}  // namespace numa::gpu
