// hfx_sp2.cu -- occupied-space projector by trace-correcting SP2 (see
// hfx_sp2.hpp).
//
// One step computes X_j from X_{j-1} and X_{j-1}^2 (X_j = X^2 or 2X - X^2)
// and then X_j^2, as an 8 x 8 output tile per block over the upper triangle
// (the mirror tile is written from the same values, so every X_j and X_j^2 is
// exactly symmetric).  A block stages the two 8-row panels of X_j it needs in
// shared memory, forming them on the fly from the previous step's matrices.
// The recursion's control -- which branch, when to stop -- depends only on
// tr(X_{j-1}) and tr(X_{j-1}^2), summed in a fixed order from per-tile
// partial traces by every block alike, so all blocks agree without a grid
// barrier and the result is deterministic.  Matrices alternate between two
// buffers by step parity.
#include <algorithm>
#include <cmath>

#include "hfx_sp2.hpp"

namespace hfx {
namespace {

constexpr int kTile = 8;
constexpr int kThreads = 256;       // 64 outputs x 4 slices of the inner dimension
// Stop two steps after sum_i lambda_i (1 - lambda_i) = tr(X) - tr(X^2) falls
// below this: each of the two steps squares the larger of the occupied and
// virtual deviations, leaving them at rounding level.  The traces' own
// rounding is ~1e-13 for n <= 1024.
constexpr double kIdemTol = 1e-10;
constexpr double kTraceTol = 1e-6;  // tr(D) = nocc: otherwise no gap (fractional occupation)

// The projections of one run (blockIdx.y).
struct Sp2Set {
    const double* F;
    double *X[2], *X2[2];
    double *bounds, *traces, *D, *status;
    int* state;
    int nocc;
};
struct Sp2Sets {
    Sp2Set s[2];
};

// Gershgorin bounds of sym(F) = (F + F^T) / 2, one warp per row:
// bounds[0] = min_i (f_ii - r_i), bounds[1] = max_i (f_ii + r_i).
__global__ void __launch_bounds__(1024) k_sp2_bounds(int n, Sp2Sets sets)
{
    const double* __restrict__ F = sets.s[blockIdx.y].F;
    double* bounds = sets.s[blockIdx.y].bounds;
    __shared__ double lo_w[32], hi_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double lo = INFINITY, hi = -INFINITY;
    for (int i = warp; i < n; i += nw) {
        double r = 0.0;
        for (int c = lane; c < n; c += 32)
            if (c != i) r += fabs(0.5 * (F[(size_t)i * n + c] + F[(size_t)c * n + i]));
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        const double d = F[(size_t)i * n + i];
        lo = fmin(lo, d - r);
        hi = fmax(hi, d + r);
    }
    if (lane == 0) {
        lo_w[warp] = lo;
        hi_w[warp] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < nw; ++w) {
            lo = fmin(lo, lo_w[w]);
            hi = fmax(hi, hi_w[w]);
        }
        bounds[0] = lo;
        bounds[1] = hi;
    }
}

struct Sp2Decision {
    int branch;  // 0: X_0 from F; 1: X <- X^2; 2: X <- 2X - X^2
    int kstar;   // first step with tr(X) - tr(X^2) < kIdemTol (-1: none yet)
    int answer;  // step whose X is the projector (-1: not yet)
};

// Fixed-order sums of the first m entries of v over one warp (lane 0's
// reduction order, broadcast), so that every block obtains the same bits.
__device__ __forceinline__ double warp_sum_fixed(const double* v, int m)
{
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    for (int t = lane; t < m; t += 32) s += v[t];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    return __shfl_sync(0xffffffffu, s, 0);
}

// The recursion's control before step j, from the state and traces that step
// j-1 left.  Called by one whole warp; the same result in every block.
__device__ Sp2Decision sp2_decide(int j, int nt, int nocc, const double* traces, const int* state)
{
    Sp2Decision d{0, -1, -1};
    if (j == 0) return d;
    d.kstar = state[2 * (j - 1)];
    d.answer = state[2 * (j - 1) + 1];
    if (d.answer >= 0) return d;  // step j-1 did nothing, its traces are not written
    const double* px = traces + (size_t)(j - 1) * 2 * nt;
    const double sx = warp_sum_fixed(px, nt);
    const double sx2 = warp_sum_fixed(px + nt, nt);
    if (d.kstar < 0 && sx - sx2 < kIdemTol) d.kstar = j - 1;
    if (d.kstar >= 0 && j - 1 >= d.kstar + 2) d.answer = j - 1;
    d.branch = fabs(sx2 - nocc) < fabs(2.0 * sx - sx2 - nocc) ? 1 : 2;
    return d;
}

// element (r, c) of X_j
__device__ __forceinline__ double sp2_form(int branch, int n, int r, int c, const double* F, double emax,
                                           double inv_w, const double* Xp, const double* X2p)
{
    const size_t e = (size_t)r * n + c;
    if (branch == 0) {
        const double f = 0.5 * (F[e] + F[(size_t)c * n + r]);
        return ((r == c ? emax : 0.0) - f) * inv_w;
    }
    if (branch == 1) return X2p[e];
    return 2.0 * Xp[e] - X2p[e];
}

__global__ void __launch_bounds__(kThreads) k_sp2_step(int n, int nt, int j, Sp2Sets sets)
{
    const Sp2Set& set = sets.s[blockIdx.y];
    const double* __restrict__ F = set.F;
    const double* bounds = set.bounds;
    const double *Xp = set.X[(j & 1) ^ 1], *X2p = set.X2[(j & 1) ^ 1];
    double *Xo = set.X[j & 1], *X2o = set.X2[j & 1];
    double* traces = set.traces;
    int* state = set.state;
    const int nocc = set.nocc;
    // Programmatic dependent launch: the next step's blocks may be scheduled
    // from here on and wait at their own dependency point, so that the ~45
    // dependent launches of a projection do not each pay a launch gap.
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    extern __shared__ double sm[];
    const int ld = n + 1;  // odd row stride: the 8 rows of a panel fall in distinct banks
    double* A = sm;
    double* B = sm + kTile * ld;
    double* red = B + kTile * ld;
    __shared__ int s_branch, s_kstar, s_answer;
    if (threadIdx.x < 32) {
        const Sp2Decision d = sp2_decide(j, nt, nocc, traces, state);
        if (threadIdx.x == 0) {
            s_branch = d.branch;
            s_kstar = d.kstar;
            s_answer = d.answer;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        state[2 * j] = s_kstar;
        state[2 * j + 1] = s_answer;
    }
    if (s_answer >= 0) return;
    const int branch = s_branch;
    // tile (I, J), I <= J, in row-major order of the upper triangle
    int b = blockIdx.x, I = 0;
    while (b >= nt - I) {
        b -= nt - I;
        ++I;
    }
    const int J = I + b;
    const double emax = bounds[1];
    const double inv_w = 1.0 / (bounds[1] - bounds[0]);
    for (int e = threadIdx.x; e < kTile * n; e += kThreads) {
        const int r = e / n, c = e - r * n;
        const int ra = I * kTile + r, rb = J * kTile + r;
        A[r * ld + c] = ra < n ? sp2_form(branch, n, ra, c, F, emax, inv_w, Xp, X2p) : 0.0;
        B[r * ld + c] = rb < n ? sp2_form(branch, n, rb, c, F, emax, inv_w, Xp, X2p) : 0.0;
    }
    __syncthreads();
    const int o = threadIdx.x & 63, ks = threadIdx.x >> 6;
    const int a = o >> 3, bb = o & 7;
    const double* Ar = A + a * ld;
    const double* Br = B + bb * ld;  // X_j is symmetric: row panel J is column panel J
    double acc = 0.0;
    for (int k = ks; k < n; k += 4) acc = fma(Ar[k], Br[k], acc);
    red[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x < 64) {
        const double v = (red[o] + red[o + 64]) + (red[o + 128] + red[o + 192]);
        const int row = I * kTile + a, col = J * kTile + bb;
        if (row < n && col < n) {
            const double x = A[a * ld + col];
            X2o[(size_t)row * n + col] = v;
            Xo[(size_t)row * n + col] = x;
            if (I != J) {
                X2o[(size_t)col * n + row] = v;
                Xo[(size_t)col * n + row] = x;
            }
        }
        red[o] = v;  // each thread reads and writes only its own o entries
    }
    if (I == J) {  // block-uniform
        __syncthreads();
        if (threadIdx.x == 0) {
            double tx = 0.0, tx2 = 0.0;
            for (int q = 0; q < kTile && I * kTile + q < n; ++q) {
                tx += A[q * ld + I * kTile + q];
                tx2 += red[q * kTile + q];
            }
            traces[(size_t)j * 2 * nt + I] = tx;
            traces[(size_t)j * 2 * nt + nt + I] = tx2;
        }
    }
}

__global__ void __launch_bounds__(256) k_sp2_finish(int n, int nt, int steps, Sp2Sets sets)
{
    const Sp2Set& set = sets.s[blockIdx.y];
    const double* traces = set.traces;
    const int nocc = set.nocc;
    double* D = set.D;
    __shared__ int s_answer;
    if (threadIdx.x < 32) {
        const Sp2Decision d = sp2_decide(steps, nt, nocc, traces, set.state);
        int ans = d.answer;
        if (ans >= 0) {
            const double tr = warp_sum_fixed(traces + (size_t)ans * 2 * nt, nt);
            if (!(fabs(tr - nocc) < kTraceTol)) ans = -1;
        }
        if (threadIdx.x == 0) s_answer = ans;
    }
    __syncthreads();
    const int ans = s_answer;
    if (blockIdx.x == 0 && threadIdx.x == 0) *set.status = ans >= 0 ? (double)(ans + 1) : 0.0;
    if (ans < 0) return;
    const double* X = set.X[ans & 1];
    const size_t total = (size_t)n * n;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x)
        D[e] = X[e];
}

}  // namespace

Sp2Projector::Sp2Projector(int n) : n_(n), nt_((n + kTile - 1) / kTile)
{
    if (n < 1 || n > kMaxN) throw Error(HFX_ERR_INVALID, "SP2 projector: matrix dimension out of range");
    smem_ = sizeof(double) * ((size_t)2 * kTile * (n + 1) + kThreads);
    // The limit is a property of the kernel, shared by every projector in the
    // process: always raise it to what the largest n needs, never to this n's
    // figure, which would lower it under a concurrent projector of larger n.
    const size_t smem_max = sizeof(double) * ((size_t)2 * kTile * (kMaxN + 1) + kThreads);
    cuda_check(cudaFuncSetAttribute(k_sp2_step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max),
               "SP2 shared memory");
}

void Sp2Projector::run(const Task* tasks, int count, cudaStream_t st, int max_steps)
{
    if (count < 1 || count > 2) throw Error(HFX_ERR_INVALID, "SP2 projector: one or two projections");
    const size_t nn = (size_t)n_ * n_;
    Sp2Sets sets{};
    for (int t = 0; t < count; ++t) {
        if (tasks[t].nocc <= 0 || tasks[t].nocc >= n_) throw Error(HFX_ERR_INVALID, "SP2 projector: occupation out of range");
        Sp2Set& s = sets.s[t];
        for (int p = 0; p < 2; ++p) {
            X_[t][p].alloc(nn);
            X2_[t][p].alloc(nn);
            s.X[p] = X_[t][p].p;
            s.X2[p] = X2_[t][p].p;
        }
        bounds_[t].alloc(2);
        traces_[t].alloc((size_t)kMaxSteps * 2 * nt_);
        state_[t].alloc((size_t)kMaxSteps * 2);
        s.F = tasks[t].F;
        s.nocc = tasks[t].nocc;
        s.D = tasks[t].D;
        s.status = tasks[t].status;
        s.bounds = bounds_[t].p;
        s.traces = traces_[t].p;
        s.state = state_[t].p;
    }
    const int steps = std::max(1, std::min(max_steps, kMaxSteps));
    k_sp2_bounds<<<dim3(1, count), 1024, 0, st>>>(n_, sets);
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(nt_ * (nt_ + 1) / 2), (unsigned)count);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    for (int j = 0; j < steps; ++j)
        cuda_check(cudaLaunchKernelEx(&cfg, k_sp2_step, n_, nt_, j, sets), "SP2 step");
    const int grid = (int)std::min<size_t>(1024, (nn + 255) / 256);
    k_sp2_finish<<<dim3(grid, count), 256, 0, st>>>(n_, nt_, steps, sets);
    cuda_check(cudaGetLastError(), "SP2 projector");
}

}  // namespace hfx
