// Per-voxel Levenberg-Marquardt in FP64 on the device: the step and the
// accept/damping decision of the reference's GaussNewton under a TrustRegion
// (recon/_gauss_newton.py:475-631, TrustRegion 366-415), one thread per
// voxel, over normal equations that the GN evaluation sweep reduced.
//
// Variables are the unconstrained images of the bounded properties
// (_bounds.py:77-199): a two-sided bound maps through a sigmoid, a one-sided
// one through softplus, and the Jacobian is widened by the chain factor. The
// reference solves the damped step as the augmented least-squares problem
// [J^T; sqrt(a) I] d = [r; 0] in FP32 (direct, _gauss_newton.py:247-307);
// here its normal equations (J^T J + a I) d = -J^T r are solved by a 3x3
// Cholesky factorisation in FP64.
#include <math.h>

#include "tsg_internal.h"

namespace tsg {
namespace {

constexpr double kTiny = 1.1754943508222875e-38;  // smallest normal float

__device__ __forceinline__ double sigmoid(double u) { return 1.0 / (1.0 + exp(-u)); }

__device__ __forceinline__ double softplus(double u) {
    return u > 30.0 ? u : log1p(exp(u));
}

__device__ __forceinline__ void to_natural(const tsg_gn_config& c, const double* u, double* x) {
    for (int k = 0; k < 3; ++k) {
        const double lo = c.low[k], hi = c.high[k];
        const bool has_lo = isfinite(lo), has_hi = isfinite(hi);
        if (has_lo && has_hi)
            x[k] = lo + (hi - lo) * sigmoid(u[k]);
        else if (has_lo)
            x[k] = lo + softplus(u[k]);
        else if (has_hi)
            x[k] = hi - softplus(-u[k]);
        else
            x[k] = u[k];
    }
}

__device__ __forceinline__ void widen(const tsg_gn_config& c, const double* u, double* w) {
    for (int k = 0; k < 3; ++k) {
        const double lo = c.low[k], hi = c.high[k];
        const bool has_lo = isfinite(lo), has_hi = isfinite(hi);
        if (has_lo && has_hi) {
            const double s = sigmoid(u[k]);
            w[k] = (hi - lo) * s * (1.0 - s);
        } else if (has_lo) {
            w[k] = sigmoid(u[k]);
        } else if (has_hi) {
            w[k] = sigmoid(-u[k]);
        } else {
            w[k] = 1.0;
        }
    }
}

// Free-variable normal equations from natural ones: A_f = W A W, g_f = W g.
__device__ __forceinline__ void free_system(const double* ne, const double* w, double A[3][3],
                                            double* g) {
    const double a11 = ne[1], a12 = ne[2], a13 = ne[3], a22 = ne[4], a23 = ne[5], a33 = ne[6];
    A[0][0] = w[0] * w[0] * a11;
    A[0][1] = A[1][0] = w[0] * w[1] * a12;
    A[0][2] = A[2][0] = w[0] * w[2] * a13;
    A[1][1] = w[1] * w[1] * a22;
    A[1][2] = A[2][1] = w[1] * w[2] * a23;
    A[2][2] = w[2] * w[2] * a33;
    // ne holds sum dv*(v + y): the gradient of the cost in s = -v is J_s^T r
    // with J_s = -dv and r = -(v + y), i.e. the same sum.
    g[0] = w[0] * ne[7];
    g[1] = w[1] * ne[8];
    g[2] = w[2] * ne[9];
}

// Solves (A + lambda I) d = -g; false when the matrix is not positive definite.
__device__ bool damped_solve(const double A[3][3], const double* g, double lambda, double* d) {
    double L[3][3] = {};
    double M[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) M[i][j] = A[i][j] + (i == j ? lambda : 0.0);
    for (int j = 0; j < 3; ++j) {
        double s = M[j][j];
        for (int k = 0; k < j; ++k) s -= L[j][k] * L[j][k];
        if (!(s > 0.0) || !isfinite(s)) return false;
        L[j][j] = sqrt(s);
        for (int i = j + 1; i < 3; ++i) {
            double t = M[i][j];
            for (int k = 0; k < j; ++k) t -= L[i][k] * L[j][k];
            L[i][j] = t / L[j][j];
        }
    }
    double y[3];
    for (int i = 0; i < 3; ++i) {
        double t = -g[i];
        for (int k = 0; k < i; ++k) t -= L[i][k] * y[k];
        y[i] = t / L[i][i];
    }
    for (int i = 2; i >= 0; --i) {
        double t = y[i];
        for (int k = i + 1; k < 3; ++k) t -= L[k][i] * d[k];
        d[i] = t / L[i][i];
    }
    return isfinite(d[0]) && isfinite(d[1]) && isfinite(d[2]);
}

// The voxels a launch works on: all n, or the first *count of a device list.
struct VoxelList {
    const int32_t* index;
    const int32_t* count;
};

__device__ __forceinline__ int64_t listed_voxel(const VoxelList& list, int64_t n) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (list.index == nullptr) return i < n ? i : -1;
    return i < *list.count ? list.index[i] : -1;
}

__global__ void gn_step_kernel(tsg_gn_state s, int64_t n, tsg_gn_config c, VoxelList list) {
    const int64_t i = listed_voxel(list, n);
    if (i < 0) return;
    const int status = s.status[i];
    if (status == TSG_GN_DONE) return;
    double u[3] = {s.u[3 * i], s.u[3 * i + 1], s.u[3 * i + 2]};
    double cand[3] = {u[0], u[1], u[2]};
    if (status == TSG_GN_LIVE) {
        const double* ne = s.normal + 10 * i;
        double w[3], A[3][3], g[3];
        widen(c, u, w);
        free_system(ne, w, A, g);
        // A voxel whose gradient is flat is finished before it steps
        // (_gauss_newton.py:560-565).
        const double gmax = fmax(fabs(g[0]), fmax(fabs(g[1]), fabs(g[2])));
        if (gmax < c.gradient_tolerance) {
            s.status[i] = TSG_GN_DONE;
            return;
        }
        const double lambda = s.damping[i];
        double d[3];
        const bool ok = damped_solve(A, g, lambda, d);
        int flags = 0;
        if (!ok) {
            flags |= 2;  // singular: the step is not taken
            d[0] = d[1] = d[2] = nan("");
        }
        double pred = 0.0, walked = 0.0, norm_u = 0.0;
        for (int k = 0; k < 3; ++k) {
            pred += d[k] * (lambda * d[k] - g[k]);
            walked += d[k] * d[k];
            norm_u += u[k] * u[k];
            cand[k] = u[k] + d[k];
        }
        walked = sqrt(walked);
        norm_u = sqrt(norm_u);
        if (ok && walked < c.step_tolerance * (norm_u + c.step_tolerance)) flags |= 1;
        s.predicted[i] = pred;
        s.flags[i] = flags;
    }
    for (int k = 0; k < 3; ++k) s.cand[3 * i + k] = cand[k];
    double x[3];
    to_natural(c, cand, x);
    s.t1[i] = float(x[0]);
    s.t2[i] = float(x[1]);
    s.m0[i] = float(x[2]);
}

__device__ void gn_judge(const tsg_gn_state& s, const tsg_gn_config& c, int64_t i) {
    const int status = s.status[i];
    if (status == TSG_GN_DONE) return;
    const double* tr = s.trial + 10 * i;
    double* ne = s.normal + 10 * i;
    if (status == TSG_GN_FIRST) {
        // The first evaluation is taken as it stands and sets the damping
        // from the curvature there (TrustRegion.begin, :389-393).
        for (int k = 0; k < 10; ++k) ne[k] = tr[k];
        s.cost[i] = tr[0];
        double u[3] = {s.u[3 * i], s.u[3 * i + 1], s.u[3 * i + 2]};
        double w[3], A[3][3], g[3];
        widen(c, u, w);
        free_system(ne, w, A, g);
        s.damping[i] = c.tau * fmax(A[0][0], fmax(A[1][1], A[2][2]));
        s.rising[i] = 2.0;
        s.iterations[i] = 0;
        s.status[i] = TSG_GN_LIVE;
        return;
    }
    const int flags = s.flags[i];
    const bool singular = (flags & 2) != 0;
    const bool is_short = (flags & 1) != 0;
    const double pred = s.predicted[i];
    const double cost = s.cost[i];
    const double trial_cost = tr[0];
    const double gain = pred > 0.0 ? (cost - trial_cost) / fmax(pred, kTiny) : 0.0;
    const bool better = gain > 0.0 && !singular;
    // Nielsen's update (TrustRegion.judge, :395-411).
    const double lambda = s.damping[i];
    const double rising = s.rising[i];
    const double q = 2.0 * gain - 1.0;
    const double lowered = lambda * fmax(1.0 - q * q * q, 1.0 / 3.0);
    s.damping[i] = better ? lowered : lambda * rising;
    s.rising[i] = better ? 2.0 : rising * 2.0;
    if (better) {
        for (int k = 0; k < 3; ++k) s.u[3 * i + k] = s.cand[3 * i + k];
        for (int k = 0; k < 10; ++k) ne[k] = tr[k];
        s.cost[i] = trial_cost;
    }
    const int it = s.iterations[i] + 1;
    s.iterations[i] = it;
    if (is_short && !singular) {
        s.status[i] = TSG_GN_DONE;
    } else if (it >= c.max_iterations) {
        s.status[i] = TSG_GN_DONE;
        s.flags[i] = flags | 4;  // stopped by the step limit: unconverged
    }
}

__global__ void gn_judge_kernel(tsg_gn_state s, int64_t n, tsg_gn_config c) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) gn_judge(s, c, i);
}

constexpr int kSolveThreads = 128;

// The judgement of a solve's iteration, and the list of voxels for the next
// one: a block's survivors keep their order, the blocks' runs come in the
// order they reserve their places. A voxel's arithmetic does not depend on
// its place.
__global__ void __launch_bounds__(kSolveThreads)
    gn_judge_list_kernel(tsg_gn_state s, int64_t n, tsg_gn_config c, VoxelList list,
                         int32_t* next, int32_t* next_count) {
    __shared__ int s_warp[kSolveThreads / 32];
    __shared__ int s_base;
    const int64_t i = listed_voxel(list, n);
    bool live = false;
    if (i >= 0) {
        gn_judge(s, c, i);
        live = s.status[i] != TSG_GN_DONE;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned votes = __ballot_sync(0xffffffffu, live);
    if (lane == 0) s_warp[warp] = __popc(votes);
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
        for (int w = 0; w < kSolveThreads / 32; ++w) {
            const int k = s_warp[w];
            s_warp[w] = total;
            total += k;
        }
        s_base = total > 0 ? atomicAdd(next_count, total) : 0;
    }
    __syncthreads();
    if (live) next[s_base + s_warp[warp] + __popc(votes & ((1u << lane) - 1u))] = int32_t(i);
}

// Sums of the cost over all voxels and of the damping over the live ones, as
// one pair per block, each over a fixed share of the voxels in a fixed order.
constexpr int kTotalBlocks = 64;
constexpr int kTotalThreads = 256;
__global__ void __launch_bounds__(kTotalThreads)
    gn_totals_kernel(tsg_gn_state s, int64_t n, double* out) {
    __shared__ double s_part[2][kTotalThreads];
    double cost = 0.0, damping = 0.0;
    for (int64_t i = int64_t(blockIdx.x) * kTotalThreads + threadIdx.x; i < n;
         i += int64_t(kTotalBlocks) * kTotalThreads) {
        cost += s.cost[i];
        if (s.status[i] == TSG_GN_LIVE) damping += s.damping[i];
    }
    s_part[0][threadIdx.x] = cost;
    s_part[1][threadIdx.x] = damping;
    for (int half = kTotalThreads / 2; half > 0; half >>= 1) {
        __syncthreads();
        if (threadIdx.x < half) {
            s_part[0][threadIdx.x] += s_part[0][threadIdx.x + half];
            s_part[1][threadIdx.x] += s_part[1][threadIdx.x + half];
        }
    }
    __syncthreads();  // thread 1 writes the total that thread 0 summed
    if (threadIdx.x < 2) out[2 * blockIdx.x + threadIdx.x] = s_part[threadIdx.x][0];
}

__global__ void gn_natural_kernel(const double* u, int64_t n, tsg_gn_config c, float* out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double uu[3] = {u[3 * i], u[3 * i + 1], u[3 * i + 2]};
    double x[3];
    to_natural(c, uu, x);
    for (int k = 0; k < 3; ++k) out[3 * i + k] = float(x[k]);
}

bool valid(const tsg_gn_state* s) {
    return s && s->u && s->cand && s->cost && s->normal && s->trial && s->damping && s->rising &&
           s->predicted && s->status && s->flags && s->iterations && s->t1 && s->t2 && s->m0;
}

}  // namespace
}  // namespace tsg

using namespace tsg;

extern "C" int tsg_gn_step(const tsg_gn_state* state, int64_t voxel_count,
                           const tsg_gn_config* config, void* stream) {
    if (voxel_count < 0 || !config || (voxel_count > 0 && !valid(state)))
        return fail(TSG_ERR_ARGUMENT, "invalid Gauss-Newton state");
    if (voxel_count == 0) return TSG_OK;
    gn_step_kernel<<<unsigned((voxel_count + 127) / 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        *state, voxel_count, *config, VoxelList{nullptr, nullptr});
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

extern "C" int tsg_gn_judge(const tsg_gn_state* state, int64_t voxel_count,
                            const tsg_gn_config* config, void* stream) {
    if (voxel_count < 0 || !config || (voxel_count > 0 && !valid(state)))
        return fail(TSG_ERR_ARGUMENT, "invalid Gauss-Newton state");
    if (voxel_count == 0) return TSG_OK;
    gn_judge_kernel<<<unsigned((voxel_count + 127) / 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        *state, voxel_count, *config);
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

extern "C" int tsg_gn_natural(const double* free_variables, int64_t voxel_count,
                              const tsg_gn_config* config, float* natural, void* stream) {
    if (voxel_count < 0 || !config || (voxel_count > 0 && (!free_variables || !natural)))
        return fail(TSG_ERR_ARGUMENT, "invalid arguments");
    if (voxel_count == 0) return TSG_OK;
    gn_natural_kernel<<<unsigned((voxel_count + 127) / 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        free_variables, voxel_count, *config, natural);
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

// A run of a solve's iterations queued on the stream: per iteration the step,
// the evaluation, the judgement with the next voxel list, and the sums. Nothing
// is read back, so the launches of all its iterations are queued at once (a copy
// of the pool's rows per iteration and one wait each took as long as the
// sweeps); the grids cover every voxel and blocks past the live ones end at
// once.
extern "C" int tsg_gn_solve_part(const tsg_program* program, const tsg_gn_state* state,
                                 const float* b1, int64_t voxel_count, int64_t state_count,
                                 const void* measured, const tsg_gn_config* config, int first,
                                 int iterations, int32_t* lists, int32_t* counts, double* totals,
                                 const tsg_launch* launch_shape, void* stream) {
    if (voxel_count < 0 || !config || (voxel_count > 0 && !valid(state)))
        return fail(TSG_ERR_ARGUMENT, "invalid Gauss-Newton state");
    if (config->max_iterations < 1) return fail(TSG_ERR_ARGUMENT, "max_iterations must be positive");
    if (first < 0 || iterations < 0 || first > config->max_iterations ||
        iterations > config->max_iterations + 1 - first)
        return fail(TSG_ERR_ARGUMENT, "a solve has iterations 0 to max_iterations");
    if (voxel_count > 0x7fffffffLL) return fail(TSG_ERR_CAPACITY, "too many voxels for one solve");
    if (voxel_count == 0) return TSG_OK;
    if (!lists || !counts || !totals) return fail(TSG_ERR_ARGUMENT, "null solve buffer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned blocks = unsigned((voxel_count + kSolveThreads - 1) / kSolveThreads);
    TSG_CUDA(cudaMemsetAsync(counts + first, 0, sizeof(int32_t) * iterations, s));
    const tsg_tissue tissue{state->t1, state->t2, state->m0, b1, nullptr};
    for (int it = first; it < first + iterations; ++it) {
        VoxelList list{nullptr, nullptr};
        if (it > 0) list = {lists + (it & 1) * voxel_count, counts + it - 1};
        gn_step_kernel<<<blocks, kSolveThreads, 0, s>>>(*state, voxel_count, *config, list);
        TSG_CUDA(cudaGetLastError());
        const int rc = gn_evaluate_list(program, &tissue, voxel_count, state_count, measured, nullptr,
                                        list.index, list.count, state->trial, launch_shape, stream);
        if (rc) return rc;
        gn_judge_list_kernel<<<blocks, kSolveThreads, 0, s>>>(
            *state, voxel_count, *config, list, lists + ((it + 1) & 1) * voxel_count, counts + it);
        TSG_CUDA(cudaGetLastError());
        gn_totals_kernel<<<kTotalBlocks, kTotalThreads, 0, s>>>(
            *state, voxel_count, totals + int64_t(it) * 2 * kTotalBlocks);
        TSG_CUDA(cudaGetLastError());
    }
    return TSG_OK;
}

extern "C" int tsg_gn_solve(const tsg_program* program, const tsg_gn_state* state,
                            const float* b1, int64_t voxel_count, int64_t state_count,
                            const void* measured, const tsg_gn_config* config, int32_t* lists,
                            int32_t* counts, double* totals, const tsg_launch* launch_shape,
                            void* stream) {
    return tsg_gn_solve_part(program, state, b1, voxel_count, state_count, measured, config, 0,
                             config ? config->max_iterations + 1 : 0, lists, counts, totals,
                             launch_shape, stream);
}

extern "C" int tsg_gn_total_parts(void) { return kTotalBlocks; }
