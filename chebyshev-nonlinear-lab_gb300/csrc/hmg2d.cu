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
// together (blockIdx.z = field); programmatic dependent launch; the levels below the finest in one CUDA
// graph; and the levels of n <= 31 in one CTA a field, in shared memory (k_hmg_tail), where a step
// is a block barrier.  At 31^2 a pass is 2,200 cycles of one SM's FP64 pipe, about what a launch costs;
// at 63^2 it would be four times that, so that level stays launched.  The Burgers solve at 255^2 went from 17.5
// to 4.3 ms; a cycle of both fields is ~110 us there, 37 of them the tail (44 steps, each bound by the
// latency of its nine dependent FP64 operations or, at 31^2, by the FP64 pipe).
#include <cmath>
#include <limits>


#include "numa_internal.hpp"

namespace numa::gpu {

struct HelmholtzMG2D::Level {
    int n = 0;
    double s = 0.0;  // nu / h^2 of this level
    DeviceArray<double> x, b;
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
// The levels of n <= kTailTop in one CTA a field: x of each level with a halo of zeros, pitch m = (n + 2) | 1, the
// two parities of the padded index (the colours) stored apart, so that a pass reads one half and writes the other;
// b and the residual in natural order.  The arithmetic is the launched kernels' operation for operation.
constexpr int kTailTop = 31, kTailMax = 6, kTailThreads = 512;  // 31, 15, 7, 3, 1
struct HTailLvl {
    HLvl L;
    int m, H, offX, offB;  // pitch, elements of one parity of x, element offsets in shared memory
};
struct HTail {
    int levels, pre, post, offR, total;
    HTailLvl T[kTailMax];
};

extern __shared__ __align__(16) double htail_smem[];

// x at padded index P
__device__ __forceinline__ double& hx(double* X, int H, int P) { return X[(P & 1) * H + (P >> 1)]; }

__device__ __noinline__ void htail_sweeps(const HTailLvl& T, int sweeps, int order, bool alternate, bool first) {
    const HLvl L = T.L;
    const int n = L.n, m = T.m, H = T.H, np = (n + 1) >> 1;
    double* X = htail_smem + T.offX;
    const double* B = htail_smem + T.offB;
    const int i = (int)threadIdx.x / np, j0 = 2 * ((int)threadIdx.x - i * np);  // n np <= kTailThreads
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
    const int t = threadIdx.x;  // nc <= 15
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
    for (size_t l = 0; l < levels_.size(); ++l)
        if (levels_[l]->n <= kTailTop) {  // (at most 31, 15, 7, 3, 1 follow)
            tail_l_ = l;
            break;
        }
    for (size_t l = 1; l < levels_.size() && l <= tail_l_; ++l) {
        const size_t Nl = (size_t)fields * levels_[l]->n * levels_[l]->n;
        levels_[l]->x.resize(Nl);
        levels_[l]->b.resize(Nl);
    }
    if (tail_l_ > 0) resid_.resize(fields * N0_);
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

// The levels below the finest touch only the hierarchy's own arrays: captured once, then one launch.
void HelmholtzMG2D::coarse_cycle() {
    if (tail_l_ == 1) {  // one kernel: no graph
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
