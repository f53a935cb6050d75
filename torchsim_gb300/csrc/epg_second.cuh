// Second order: the adjoint of the tangent sweep, for K directions at once.
//
// The reference differentiates its first-order adjoint along ONE direction
// in dual numbers (forward over reverse, simulate_real_vjp_jvp_range,
// src/torchsim/_epg_cpu.cpp:7028-7330), and a design cost over a K-column
// Jacobian pays K such calls (sequence/_accelerators.py:1780-1800, one per
// column of model/_signal.py:255-268). Here the same derivatives come from
// the reverse sweep of the K-direction tangent system, in one pass:
//
//   forward   x' = A(p) x + b,   t_k' = A t_k + (dA/dp . d_k) x + db . d_k,
//             samples s = m0 F+[0](x),  j_k = m0 F+[0](t_k) + dm0_k F+[0](x)
//   loss      L = <g0, s> + sum_k <g_k, j_k>
//   reverse   mu_k  <- A^T mu_k + (record of g_k)
//             lam   <- A^T lam + sum_k (dA . d_k)^T mu_k + (record of g0, g_k)
//
// mu_k is the reference's dual value (the adjoint of seed g_k) and lam its
// tangent summed over the directions. The gradient of L with respect to the
// directions (J^T g_k, the reference's "value" side) and with respect to the
// inputs (its "curvature" side, plus J^T g0) follow per micro-step:
//
//   rotation R by a = flip*b1, a'_k = dflip_k*b1 + flip*db1_k; R commutes
//   with its generator K (R' = K R = R K), so with the pre-RF state x, t_k and
//   the cotangents taken back through the pulse, mu_k = R^T mu_k and lam =
//   R^T lam + sum_k a'_k K^T mu_k:
//     G_k = mu_k . K x            (dL/da'_k)
//     dL/da = lam . K x + sum_k mu_k . K t_k
//   in w = F+ - F- and Z (F+ + F- stays): K x = (-2 Z, w / 2).
//   relaxation E = exp(-r dt), eps_k = E'_k / E = -(r'_k dt + r ddt_k),
//   with the pre-RF states and cotangents (a shift between relaxation and
//   pulse leaves the inner products unchanged):
//     Q = lam . (x - e0) + sum_k mu_k . t_k,   C_k = mu_k . (x - e0)
//     dL/dr += -dt Q - sum_k C_k ddt_k,  dL/dr'_k += -dt C_k,
//     dL/ddt += -r Q - sum_k C_k r'_k,   dL/dddt_k += -r C_k
//   (per plane pair: transverse with r2, longitudinal with r1 and the
//   recovery e0 at order 0), and r = 1000/T, r' = -1000 T'/T^2 chain to T.
//
// The forward stores every EVEN op's entry state of x and of each t_k (the
// trajectory, one tile per warp: per stored op, state and plane the warp's 32
// lanes' order pairs are 32 * RP consecutive float2, so every store and every
// load is a whole, aligned line) and every recorded F+[0]; the reverse
// streams them back through a cp.async ring and runs the even op forward once
// for the entry state of the odd op after it. Per-event partials are summed
// over the warp with shuffles in a fixed order after each op; tissue gradients
// are summed over a voxel's lanes with shuffles. No atomics: results are
// deterministic.
//
// Bound and measured at 16,384 voxels x 601 ops x 20 orders, T1, T2 and B1: the
// forward by its stores (5.2 GB of trajectory, 0.89 ms; with every op stored
// and samples stored op by op 2.21 ms), the reverse by instruction issue and
// latency at 16 warps an SM (1.77 ms). The re-run of the even ops costs the
// reverse about 0.25 ms and saves the forward about 0.6; the pulses' (u, w)
// form and the plain ops' own copy of the step take 0.45 off the reverse, the
// records read as rows 0.17. Held to nine or ten blocks an SM it spills (2.2
// ms), and four orders per lane take too many registers (2.1 ms).
#pragma once
#include "epg_adjoint.cuh"
#include <type_traits>

namespace tsg {

constexpr int kSecondMaxK = 3;
// An op of a fingerprinting train: relaxation, pulse, sample, shift.
constexpr uint32_t kPlainOp = kFastBits | OP_RECORD;
constexpr int kSecondRing = 2;
constexpr int kSecondWarps = 2;

struct SecondArgs {
    const Op* ops;
    const float2* op_dir;  // [K][train][ops] (d dt, d flip), or null (zero)
    int n_ops;
    int64_t atoms;
    int states;
    int outputs;
    const float* t1;
    const float* t2;
    const float* m0;
    const float* b1;
    const float* inv;
    // Per direction: tangents of t1, t2, m0, b1, inversion (nullable: zero).
    const float* dir[kSecondMaxK][5];
    // Forward outputs (nullable): signal (train, atom, output) and the K
    // derivatives, then with `with_m0` the derivative along M0 (F+[0]
    // itself): (train, atom, K + with_m0, output).
    int layout;
    int with_m0;
    float* sig_a;
    float* sig_b;
    float* jac_a;
    float* jac_b;
    // Trajectory: [train][warp][op / 2][state][plane][lane][RP] float2 (state
    // 0 = x, k + 1 = t_k; warp = atom / (32 / lanes_per_voxel)), and the
    // recorded F+[0] of each state, [train][state][atom][output].
    float2* traj;
    float* traj_rec;
    // Reverse: cotangents of the signal (nullable) and of the derivatives
    // (laid out as the forward writes them).
    const float* seed0;
    const float* seed;
    int seed_layout;
    // Per (train, atom): curvature t1, t2, m0, b1, inversion, then per
    // direction the values t1, t2, m0, b1, inversion.
    float* tissue_partial;
    // Per (train, warp, op): the curvature (flip, duration), then for K == 1
    // the values (flip, duration).
    float2* event_partial;
    int64_t warps_per_train;
};

// Warps (trajectory tiles) per train for lanes_per_voxel lanes a voxel.
inline int64_t second_warps(int64_t atoms, int lanes_per_voxel) {
    const int64_t vpw = 32 / lanes_per_voxel;
    return (atoms + vpw - 1) / vpw;
}

inline int64_t second_trajectory_floats(int64_t trains, int64_t atoms, int64_t ops,
                                        int lanes_per_voxel, int orders_per_lane, int k) {
    return trains * second_warps(atoms, lanes_per_voxel) * ((ops + 1) / 2) * (k + 1) * 3 * 32 *
           int64_t(orders_per_lane);
}

// Ops whose transcendentals a voxel's lanes evaluate at once in the reverse:
// one each, an even number so that a pair of ops is never split (a lone lane
// takes two).
__host__ __device__ constexpr int second_group(int lanes) { return lanes < 2 ? 2 : lanes & ~1; }

// Records held in shared memory per warp (fewer where a warp holds more
// voxels), and the reverse's values of each: a cotangent per state and M0's
// curvature, with general directions M0's K derivatives too.
__host__ __device__ constexpr int second_records(int lanes) {
    return lanes >= 8 ? 16 : lanes >= 4 ? 8 : 4;
}
__host__ __device__ constexpr int second_record_items(int k, int hot) {
    return k + 2 + (hot ? 0 : k);
}

inline int64_t second_record_floats(int64_t trains, int64_t atoms, int64_t outputs, int k) {
    return trains * outputs * (k + 1) * atoms;
}

namespace second_detail {

// One recorded sample in the given output layout (TSG_LAYOUT_*).
__device__ __forceinline__ void store_sample(int layout, float* a, float* b, int64_t idx, float v) {
    if (layout == TSG_LAYOUT_PLANES) {
        if (a) a[idx] = 0.f;
        b[idx] = v;
    } else if (layout == TSG_LAYOUT_COMPLEX) {
        reinterpret_cast<float2*>(a)[idx] = make_float2(0.f, v);
    } else {
        reinterpret_cast<float2*>(a)[idx] = make_float2(-v, 0.f);
    }
}

// A one-hot direction set (HOT != 0): direction k is the unit tangent of
// one property, (HOT >> 2k) & 3 = 1 T1, 2 T2, 3 B1, with no event
// directions; its zero terms are left out at compile time. HOT == 0: general
// directions.
__host__ __device__ constexpr int hot_dir(int hot, int k) { return (hot >> (2 * k)) & 3; }

// The voxel constants both sweeps use.
template <int K>
struct Voxel {
    float t1, t2, m0, b1, eff, r1, r2, w1, w2;
    float dt1[K], dt2[K], dm0[K], db1[K], deff[K];
};

template <int K, int HOT>
__device__ __forceinline__ Voxel<K> load_voxel(const SecondArgs& a, int64_t ac) {
    Voxel<K> v;
    v.t1 = a.t1[ac];
    v.t2 = a.t2[ac];
    v.m0 = a.m0 ? a.m0[ac] : 1.f;
    v.b1 = a.b1 ? a.b1[ac] : 1.f;
    v.eff = a.inv ? a.inv[ac] : 1.f;
    v.r1 = 1000.f / v.t1;
    v.r2 = 1000.f / v.t2;
    v.w1 = 1000.f / (v.t1 * v.t1);
    v.w2 = 1000.f / (v.t2 * v.t2);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (HOT) {
            v.dt1[k] = hot_dir(HOT, k) == 1 ? 1.f : 0.f;
            v.dt2[k] = hot_dir(HOT, k) == 2 ? 1.f : 0.f;
            v.db1[k] = hot_dir(HOT, k) == 3 ? 1.f : 0.f;
            v.dm0[k] = v.deff[k] = 0.f;
            continue;
        }
        v.dt1[k] = a.dir[k][0] ? a.dir[k][0][ac] : 0.f;
        v.dt2[k] = a.dir[k][1] ? a.dir[k][1][ac] : 0.f;
        // m0, b1 and the inversion efficiency carry a direction only where
        // the property itself is given (the reference's feature flags).
        v.dm0[k] = (a.m0 && a.dir[k][2]) ? a.dir[k][2][ac] : 0.f;
        v.db1[k] = (a.b1 && a.dir[k][3]) ? a.dir[k][3][ac] : 0.f;
        v.deff[k] = (a.inv && a.dir[k][4]) ? a.dir[k][4][ac] : 0.f;
    }
    return v;
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// Relaxation of x and the tangents over one op: t_k <- E (t_k + eps_k (x -
// e0)), x <- E x + (1 - E1) e0, e0 the recovery target (Z at order 0, held
// by lane 0's first slot).
template <int RP, int K, int HOT>
__device__ __forceinline__ void relax_all(float2 (&P)[K + 1][RP], float2 (&M)[K + 1][RP],
                                          float2 (&Z)[K + 1][RP], float e1, float e2,
                                          const float (&eps1)[K], const float (&eps2)[K], int q) {
    const float2 E1 = dup(e1), E2 = dup(e2);
    const float z0 = Z[0][0].x - (q == 0 ? 1.f : 0.f);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const float2 a1 = dup(eps1[k]), a2 = dup(eps2[k]);
        const bool e2k = !HOT || hot_dir(HOT, k) == 2;
        const bool e1k = !HOT || hot_dir(HOT, k) == 1;
#pragma unroll
        for (int kk = 0; kk < RP; ++kk) {
            if (e2k) {
                P[k + 1][kk] = mul2(E2, fma2(a2, P[0][kk], P[k + 1][kk]));
                M[k + 1][kk] = mul2(E2, fma2(a2, M[0][kk], M[k + 1][kk]));
            } else {
                P[k + 1][kk] = mul2(E2, P[k + 1][kk]);
                M[k + 1][kk] = mul2(E2, M[k + 1][kk]);
            }
            if (e1k) {
                float2 zx = Z[0][kk];
                if (kk == 0) zx.x = z0;
                Z[k + 1][kk] = mul2(E1, fma2(a1, zx, Z[k + 1][kk]));
            } else {
                Z[k + 1][kk] = mul2(E1, Z[k + 1][kk]);
            }
        }
    }
#pragma unroll
    for (int kk = 0; kk < RP; ++kk) {
        P[0][kk] = mul2(P[0][kk], E2);
        M[0][kk] = mul2(M[0][kk], E2);
        Z[0][kk] = mul2(Z[0][kk], E1);
    }
    if (q == 0) Z[0][0].x += 1.f - e1;
}

template <int RP, int L, int K>
__device__ __forceinline__ void shift_all(float2 (&P)[K + 1][RP], float2 (&M)[K + 1][RP], int q,
                                          bool kill, int kill_r) {
#pragma unroll
    for (int s = 0; s <= K; ++s) shift_fwd<RP, L>(P[s], M[s], q, kill, kill_r);
}

template <int RP, int L, int K>
__device__ __forceinline__ void shift_adjoint_all(float2 (&P)[K + 1][RP], float2 (&M)[K + 1][RP],
                                                  int q, bool kill, int kill_r) {
#pragma unroll
    for (int s = 0; s <= K; ++s) shift_adjoint<RP, L>(P[s], M[s], q, kill, kill_r);
}

template <int RP, int K>
__device__ __forceinline__ void spoil_all(float2 (&P)[K + 1][RP], float2 (&M)[K + 1][RP]) {
#pragma unroll
    for (int s = 0; s <= K; ++s)
#pragma unroll
        for (int kk = 0; kk < RP; ++kk) P[s][kk] = M[s][kk] = dup(0.f);
}

// The pulse on x and the tangents, (sin, cos) of its angle.
template <int RP, int K, int HOT>
__device__ __forceinline__ void rotate_all(float2 (&P)[K + 1][RP], float2 (&M)[K + 1][RP],
                                           float2 (&Z)[K + 1][RP], float si, float co,
                                           const float (&dal)[K]) {
    const float2 ch = dup(0.5f * (1.f + co)), sh = dup(0.5f * (1.f - co));
    const float2 hs = dup(0.5f * si), nhs = dup(-0.5f * si), hc = dup(0.5f * co);
    const float2 si2 = dup(si), nsi2 = dup(-si), co2 = dup(co);
    const float2 neg1 = dup(-1.f);
#pragma unroll
    for (int kk = 0; kk < RP; ++kk) {
        const float2 p = P[0][kk], m = M[0][kk], z = Z[0][kk];
        const float2 w = fma2(neg1, m, p);
        // R'x: (-hs w - co z, hs w + co z, hc w - si z).
        const float2 dM = fma2(hs, w, mul2(co2, z));
        const float2 dZ = fma2(hc, w, mul2(nsi2, z));
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float2 tp = P[k + 1][kk], tm = M[k + 1][kk], tz = Z[k + 1][kk];
            if (!HOT || hot_dir(HOT, k) == 3) {
                const float2 al = dup(dal[k]);
                const float2 aM = mul2(al, dM);
                P[k + 1][kk] = fma2(ch, tp, fma2(sh, tm, fma2(nsi2, tz, mul2(neg1, aM))));
                M[k + 1][kk] = fma2(sh, tp, fma2(ch, tm, fma2(si2, tz, aM)));
                Z[k + 1][kk] = fma2(hs, tp, fma2(nhs, tm, fma2(co2, tz, mul2(al, dZ))));
            } else {
                P[k + 1][kk] = fma2(ch, tp, fma2(sh, tm, mul2(nsi2, tz)));
                M[k + 1][kk] = fma2(sh, tp, fma2(ch, tm, mul2(si2, tz)));
                Z[k + 1][kk] = fma2(hs, tp, fma2(nhs, tm, mul2(co2, tz)));
            }
        }
        P[0][kk] = fma2(ch, p, fma2(sh, m, mul2(nsi2, z)));
        M[0][kk] = fma2(sh, p, fma2(ch, m, mul2(si2, z)));
        Z[0][kk] = fma2(hs, w, mul2(co2, z));
    }
}

// The inversion of x and the tangents.
template <int RP, int K, int HOT>
__device__ __forceinline__ void invert_all(float2 (&Z)[K + 1][RP], const Voxel<K>& v) {
    const float2 f = dup(-v.eff);
#pragma unroll
    for (int kk = 0; kk < RP; ++kk) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            Z[k + 1][kk] = HOT ? mul2(f, Z[k + 1][kk])
                               : fma2(f, Z[k + 1][kk], mul2(dup(-v.deff[k]), Z[0][kk]));
        Z[0][kk] = mul2(Z[0][kk], f);
    }
}

// One op's per-direction scalars: eps1_k, eps2_k (relaxation) and a'_k
// (rotation); ddt_k and dflip_k from the op's directions.
template <int K, int HOT>
__device__ __forceinline__ void op_directions(const SecondArgs& a, const float2* dirs, int64_t n,
                                              int o, const Op& op, const Voxel<K>& v,
                                              float (&ddt)[K], float (&eps1)[K], float (&eps2)[K],
                                              float (&dal)[K], float (&dfl)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (HOT) {
            ddt[k] = dfl[k] = 0.f;
            eps1[k] = hot_dir(HOT, k) == 1 ? v.w1 * op.dt : 0.f;
            eps2[k] = hot_dir(HOT, k) == 2 ? v.w2 * op.dt : 0.f;
            dal[k] = hot_dir(HOT, k) == 3 ? op.flip : 0.f;
            continue;
        }
        const float2 d = dirs ? dirs[k * n + o] : make_float2(0.f, 0.f);
        ddt[k] = d.x;
        dfl[k] = d.y;
        eps1[k] = v.w1 * v.dt1[k] * op.dt - v.r1 * d.x;
        eps2[k] = v.w2 * v.dt2[k] * op.dt - v.r2 * d.x;
        dal[k] = d.y * v.b1 + op.flip * v.db1[k];
    }
}

}  // namespace second_detail

using namespace second_detail;

// ---- forward: x and K tangents, storing the trajectory ---------------------

// Static shared memory: a chunk of ops and of each direction's per-op
// (d dt, d flip).
template <int RP, int L, int K, int HOT>
__global__ void __launch_bounds__(128) second_forward_kernel(const SecondArgs a) {
    constexpr int R = 2 * RP;
    constexpr int VPW = 32 / L;
    constexpr int NS = K + 1;
    __shared__ Op s_ops[kOpChunk];
    __shared__ float2 s_dir[K][kOpChunk];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int q = lane % L;
    const int slot = lane / L;
    const int64_t atom = (int64_t(blockIdx.x) * (blockDim.x >> 5) + warp) * VPW + slot;
    const int64_t train = blockIdx.y;
    const bool active = slot < VPW && atom < a.atoms;
    const int64_t ac = active ? atom : 0;
    const int S = a.states;
    const bool kill = L * R > S;
    const int kill_r = S - q * R;
    const Voxel<K> v = load_voxel<K, HOT>(a, ac);

    float2 P[NS][RP], M[NS][RP], Z[NS][RP];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int kk = 0; kk < RP; ++kk) P[s][kk] = M[s][kk] = Z[s][kk] = dup(0.f);
    if (q == 0) Z[0][0].x = 1.f;

    const Op* ops = a.ops + train * a.n_ops;
    const int64_t n_all = int64_t(gridDim.y) * a.n_ops;  // ops of all trains, per direction
    const float2* dirs = a.op_dir ? a.op_dir + train * a.n_ops : nullptr;
    // This warp's tile; lanes of a warp past the last voxel store nothing.
    const int64_t n_warps = (a.atoms + VPW - 1) / VPW;
    const int64_t warp_global = int64_t(blockIdx.x) * (blockDim.x >> 5) + warp;
    const int64_t op_stride = int64_t(NS) * 3 * 32 * RP;
    float2* lane_traj = (a.traj && warp_global < n_warps)
                            ? a.traj + (train * n_warps + warp_global) * ((a.n_ops + 1) >> 1) *
                                           op_stride +
                                  lane * RP
                            : nullptr;
    const bool lane0 = active && q == 0;
    // Samples: the recorded F+[0] of x and of each t_k wait in shared memory,
    // EC at a time, and leave as rows (the signal, the derivative columns, the
    // M0 column, and what the reverse sweep reads of every state). Stored
    // where they are recorded they were 2 K + 3 partial sectors a voxel and
    // op, which bound the sweep (1.57 ms; 0.89 ms in rows). With fewer than
    // four lanes a voxel, a warp's rows are not worth their shared memory.
    constexpr bool STAGED = L >= 4;
    constexpr int EC = second_records(L);
    __shared__ float s_rec[STAGED ? 4 : 1][STAGED ? VPW * NS * (EC + 1) : 1];
    __shared__ int s_index[4][EC];
    float* rec_raw = s_rec[STAGED ? warp : 0];
    int held = 0;
    const bool with_sig = a.layout == TSG_LAYOUT_PLANES ? a.sig_b != nullptr : a.sig_a != nullptr;
    const bool with_jac = a.layout == TSG_LAYOUT_PLANES ? a.jac_b != nullptr : a.jac_a != nullptr;
    const int jac_cols = K + a.with_m0;
    // One voxel's outputs of one record, from the recorded values raw[state].
    auto put_record = [&](int64_t voxel, int64_t rec, const float (&raw)[NS], float m0,
                          const float (&dm0)[K]) {
        const int64_t out = train * a.atoms + voxel;
        if (with_sig)
            store_sample(a.layout, a.sig_a, a.sig_b, out * a.outputs + rec, m0 * raw[0]);
        if (with_jac) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                store_sample(a.layout, a.jac_a, a.jac_b, (out * jac_cols + k) * a.outputs + rec,
                             HOT ? m0 * raw[k + 1] : fmaf(m0, raw[k + 1], dm0[k] * raw[0]));
            if (a.with_m0)
                store_sample(a.layout, a.jac_a, a.jac_b, (out * jac_cols + K) * a.outputs + rec,
                             raw[0]);
        }
        if (a.traj_rec) {
#pragma unroll
            for (int s = 0; s < NS; ++s)
                a.traj_rec[((train * NS + s) * a.atoms + voxel) * a.outputs + rec] = raw[s];
        }
    };
    auto flush = [&]() {
        __syncwarp();
        const int col = lane % EC;
#pragma unroll 1
        for (int first = 0; first < VPW; first += 32 / EC) {
            const int vv = first + lane / EC;
            const int from = min(vv, VPW - 1) * L;
            const float m0 = __shfl_sync(0xffffffffu, v.m0, from);
            float dm0[K];
#pragma unroll
            for (int k = 0; k < K; ++k)
                dm0[k] = HOT ? 0.f : __shfl_sync(0xffffffffu, v.dm0[k], from);
            const int64_t voxel = warp_global * VPW + vv;
            if (vv >= VPW || voxel >= a.atoms || col >= held) continue;
            float raw[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) raw[s] = rec_raw[(vv * NS + s) * (EC + 1) + col];
            put_record(voxel, s_index[warp][col], raw, m0, dm0);
        }
        __syncwarp();
        held = 0;
    };

    // One op; of a plain one (kPlainOp, most ops of a fingerprinting train) the
    // steps are known when this is compiled.
    int op_base = 0;
    auto step = [&](auto plain, int i, const Op& op, const float4& tr) {
        const uint32_t code = decltype(plain)::value ? kPlainOp : op.code;
        if (lane_traj && !((op_base + i) & 1)) {
            float2* dst = lane_traj + int64_t((op_base + i) >> 1) * op_stride;
#pragma unroll
            for (int s = 0; s < NS; ++s)
#pragma unroll
                for (int kk = 0; kk < RP; ++kk) {
                    dst[(s * 3 + 0) * 32 * RP + kk] = P[s][kk];
                    dst[(s * 3 + 1) * 32 * RP + kk] = M[s][kk];
                    dst[(s * 3 + 2) * 32 * RP + kk] = Z[s][kk];
                }
        }
        float ddt[K], eps1[K], eps2[K], dal[K], dfl[K];
        op_directions<K, HOT>(a, HOT ? nullptr : &s_dir[0][0], kOpChunk, i, op, v, ddt, eps1,
                              eps2, dal, dfl);
        if (code & OP_RELAX)
            relax_all<RP, K, HOT>(P, M, Z, tr.z, tr.w, eps1, eps2, q);
        for (int s = 0; s < op_shift1(code); ++s) shift_all<RP, L, K>(P, M, q, kill, kill_r);
        const int rf = op_rf(code);
        if (rf == RF_ROTATE) {
            rotate_all<RP, K, HOT>(P, M, Z, tr.x, tr.y, dal);
        } else if (rf == RF_INVERT) {
            invert_all<RP, K, HOT>(Z, v);
        }
        for (int s = 0; s < op_shift2(code); ++s) shift_all<RP, L, K>(P, M, q, kill, kill_r);
        if (code & OP_SPOIL1) spoil_all<RP, K>(P, M);
        if (code & OP_RECORD) {
            if constexpr (STAGED) {
                if (q == 0 && slot < VPW) {
#pragma unroll
                    for (int s = 0; s < NS; ++s)
                        rec_raw[(slot * NS + s) * (EC + 1) + held] = P[s][0].x;
                }
                if (lane == 0) s_index[warp][held] = op.record;
                if (++held == EC) flush();
            } else if (lane0) {
                float raw[NS];
#pragma unroll
                for (int s = 0; s < NS; ++s) raw[s] = P[s][0].x;
                put_record(atom, op.record, raw, v.m0, v.dm0);
            }
        }
        for (int s = 0; s < op_shift3(code); ++s) shift_all<RP, L, K>(P, M, q, kill, kill_r);
        if (code & OP_SPOIL2) spoil_all<RP, K>(P, M);
    };

    float4 my = make_float4(0.f, 1.f, 1.f, 1.f);  // (sin, cos, E1, E2) of this lane's op
    for (int base = 0; base < a.n_ops; base += kOpChunk) {
        const int count = min(kOpChunk, a.n_ops - base);
        op_base = base;
        __syncthreads();
        for (int i = threadIdx.x; i < count; i += blockDim.x) {
            s_ops[i] = ops[base + i];
#pragma unroll
            for (int k = 0; k < K; ++k)
                s_dir[k][i] = dirs ? dirs[k * n_all + base + i] : make_float2(0.f, 0.f);
        }
        __syncthreads();
        for (int i = 0; i < count; ++i) {
            const Op op = s_ops[i];
            // Lane q of a voxel evaluates the transcendentals of one of the
            // next L ops; the lanes exchange them by shuffle.
            const int g = i % L;
            if (g == 0 && i + q < count) {
                const Op next = s_ops[i + q];
                my = make_float4(0.f, 1.f, expf(-v.r1 * next.dt), expf(-v.r2 * next.dt));
                if (op_rf(next.code) == RF_ROTATE) sincosf(next.flip * v.b1, &my.x, &my.y);
            }
            float4 tr;
            tr.x = __shfl_sync(0xffffffffu, my.x, lane - q + g);
            tr.y = __shfl_sync(0xffffffffu, my.y, lane - q + g);
            tr.z = __shfl_sync(0xffffffffu, my.z, lane - q + g);
            tr.w = __shfl_sync(0xffffffffu, my.w, lane - q + g);
            if (op.code == kPlainOp)
                step(std::true_type{}, i, op, tr);
            else
                step(std::false_type{}, i, op, tr);
        }
    }
    if (STAGED && held > 0) flush();
}

// ---- reverse ---------------------------------------------------------------

// Dynamic shared memory: entry states of the even op [D][NS][3][RP][T] float2
// (a ring slot per pair of ops), transcendentals [G][VPB] float4, the records'
// values [W][VPW][NI][EC] float and indexes [W][EC] int, ops [n_ops],
// per-direction op directions [K][n_ops] float2 (only with event directions).
template <int RP, int L, int K, int HOT>
__global__ void __launch_bounds__(32 * kSecondWarps) second_reverse_kernel(const SecondArgs a) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    constexpr int W = kSecondWarps;
    constexpr int T = 32 * W;
    constexpr int R = 2 * RP;
    constexpr int VPW = 32 / L;
    constexpr int NS = K + 1;
    constexpr int D = kSecondRing;
    constexpr int NE2 = (K == 1 && !HOT) ? 2 : 1;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int q = lane % L;
    const int slot = lane / L;
    const int64_t warp_global = int64_t(blockIdx.x) * W + warp;
    const int64_t atom = warp_global * VPW + slot;
    const int64_t train = blockIdx.y;
    const bool active = slot < VPW && atom < a.atoms;
    const int64_t ac = active ? atom : 0;
    const int S = a.states;
    const int n_ops = a.n_ops;
    const bool kill = L * R > S;
    const int kill_r = S - q * R;
    const bool lane0 = active && q == 0;
    const int64_t n = a.atoms;
    const int64_t row = train * n + atom;
    const int vslot = warp * VPW + (slot < VPW ? slot : VPW - 1);

    constexpr int VPB = W * VPW;  // transcendentals are per voxel slot
    constexpr int EC = second_records(L), NI = second_record_items(K, HOT);
    float2* s_ring = reinterpret_cast<float2*>(s_raw);                    // [D][NS*3][T][RP]
    constexpr int G = second_group(L);
    float4* s_tring = reinterpret_cast<float4*>(s_ring + D * NS * 3 * RP * T);  // [G][VPB]
    float* s_seed = reinterpret_cast<float*>(s_tring + G * VPB);          // [W][VPW][NI][EC]
    int* s_index = reinterpret_cast<int*>(s_seed + W * VPW * NI * EC);     // [W][EC]
    Op* s_ops = reinterpret_cast<Op*>(s_index + W * EC);                   // [n_ops]
    float2* s_dir = reinterpret_cast<float2*>(s_ops + n_ops);              // [K][n_ops]

    const Voxel<K> v = load_voxel<K, HOT>(a, ac);
    {
        const Op* ops = a.ops + train * n_ops;
        for (int i = threadIdx.x; i < n_ops; i += T) s_ops[i] = ops[i];
        if (!HOT && a.op_dir) {
            const int64_t n_all = int64_t(gridDim.y) * n_ops;
            for (int i = threadIdx.x; i < K * n_ops; i += T) {
                const int k = i / n_ops, o = i - k * n_ops;
                s_dir[i] = a.op_dir[k * n_all + train * n_ops + o];
            }
        }
        __syncthreads();
    }

    // Cotangents: lam (state 0) and mu_k (state k + 1).
    float2 pb[NS][RP], mb[NS][RP], zb[NS][RP];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int kk = 0; kk < RP; ++kk) pb[s][kk] = mb[s][kk] = zb[s][kk] = dup(0.f);

    // Accumulated per lane: dL/dr1, dL/dr2, dL/dr1'_k, dL/dr2'_k; the
    // curvature of m0, b1, inversion; the values of m0, b1, inversion.
    float g_r1 = 0.f, g_r2 = 0.f, c_m0 = 0.f, c_b1 = 0.f, c_inv = 0.f;
    float g_rd1[K], g_rd2[K], v_m0[K], v_b1[K], v_inv[K];
#pragma unroll
    for (int k = 0; k < K; ++k) g_rd1[k] = g_rd2[k] = v_m0[k] = v_b1[k] = v_inv[k] = 0.f;

    const bool planes = a.seed_layout == TSG_LAYOUT_PLANES;
    const int seed_stride = planes ? 1 : 2;
    const float seed_sign = planes ? 1.f : -1.f;
    const int jc = K + a.with_m0;
    float* seeds = s_seed + warp * VPW * NI * EC;
    int* index = s_index + warp * EC;
    // The next records of the reverse sweep, from op o down, up to EC: their
    // cotangents of F+[0] of every state and their parts of the M0 sums,
    // read as rows. (Read one by one where they were used, they were 2 K + 3
    // copies of four bytes for each voxel and op.)
    int left = 0, at = 0;
    auto refill = [&](int o) {
        __syncwarp();
        const int j = o - lane;
        const bool rec = j >= 0 && (s_ops[j].code & OP_RECORD);
        const unsigned set = __ballot_sync(0xffffffffu, rec);
        const int rank = __popc(set & ((1u << lane) - 1u));
        if (rec && rank < EC) index[rank] = s_ops[j].record;
        left = min(__popc(set), EC);
        at = 0;
        __syncwarp();
        const int col = lane % EC;
#pragma unroll 1
        for (int first = 0; first < VPW; first += 32 / EC) {
            const int vv = first + lane / EC;
            const int from = min(vv, VPW - 1) * L;
            const float m0 = __shfl_sync(0xffffffffu, v.m0, from);
            float dm0[K];
#pragma unroll
            for (int k = 0; k < K; ++k)
                dm0[k] = HOT ? 0.f : __shfl_sync(0xffffffffu, v.dm0[k], from);
            const int64_t voxel = warp_global * VPW + vv;
            if (vv >= VPW || voxel >= n || col >= left) continue;
            const int64_t r = index[col];
            const int64_t out = train * n + voxel;
            const float* x = a.traj_rec + (train * NS * n + voxel) * a.outputs + r;
            const float* g = a.seed + (out * jc * a.outputs + r) * seed_stride;
            float* dst = seeds + vv * NI * EC + col;
            // With one or two directions all loads come first, so that they are
            // one wait (3,000 voxels x 300 x 6 states, T1 and T2: 376 and 302 us);
            // with three the compiler does better where they are used (16,384 x
            // 300 x 20: 899 and 917 us).
            constexpr bool kFirst = K < 3;
            float xs[NS], gs[K];
            if constexpr (kFirst) {
#pragma unroll
                for (int s = 0; s < NS; ++s) xs[s] = x[s * n * a.outputs];
#pragma unroll
                for (int k = 0; k < K; ++k) gs[k] = g[int64_t(k) * a.outputs * seed_stride];
            }
            auto recorded = [&](int s) { return kFirst ? xs[s] : x[s * n * a.outputs]; };
            const float x0 = recorded(0);
            const float g0 = a.seed0 ? seed_sign * a.seed0[(out * a.outputs + r) * seed_stride] : 0.f;
            // The M0 derivative is F+[0] itself: its seed acts unscaled.
            float add0 = g0 * m0, m0_sum = g0 * x0;
            if (a.with_m0)
                add0 = fmaf(seed_sign, g[int64_t(K) * a.outputs * seed_stride], add0);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const float gk = seed_sign * (kFirst ? gs[k] : g[int64_t(k) * a.outputs * seed_stride]);
                if (!HOT) {
                    add0 = fmaf(gk, dm0[k], add0);
                    dst[(NS + 1 + k) * EC] = gk * x0;
                }
                dst[(k + 1) * EC] = gk * m0;
                m0_sum = fmaf(gk, recorded(k + 1), m0_sum);
            }
            dst[0] = add0;
            dst[NS * EC] = m0_sum;
        }
        __syncwarp();
    };

    // This warp's tile (a warp past the last voxel reads tile 0 and keeps
    // nothing of it).
    const int64_t n_warps = (n + VPW - 1) / VPW;
    const int64_t op_stride = int64_t(NS) * 3 * 32 * RP;
    const float2* lane_traj =
        a.traj + (train * n_warps + (warp_global < n_warps ? warp_global : 0)) *
                     ((n_ops + 1) >> 1) * op_stride +
        lane * RP;
    const unsigned ring_base =
        static_cast<unsigned>(__cvta_generic_to_shared(s_ring + threadIdx.x * RP));

    // Pair i (ops 2 i, 2 i + 1) into ring slot rs: the even op's entry states.
    auto fetch = [&](int i, int rs) {
        const float2* src_op = lane_traj + i * op_stride;
        const unsigned dst_op = ring_base + unsigned(rs * NS * 3 * RP * T) * 8u;
#pragma unroll
        for (int sp = 0; sp < NS * 3; ++sp) {
            const float2* src = src_op + sp * 32 * RP;
            const unsigned dst = dst_op + unsigned(sp * T * RP) * 8u;
            if constexpr (RP == 2) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src)
                             : "memory");
            } else {
#pragma unroll
                for (int kk = 0; kk < RP; ++kk)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst + 8u * kk),
                                 "l"(src + kk)
                                 : "memory");
            }
        }
    };

    const int n_pairs = (n_ops + 1) >> 1;
#pragma unroll
    for (int j = 1; j < D; ++j) {
        if (n_pairs - j >= 0) fetch(n_pairs - j, j - 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    float2* event_out =
        a.event_partial + (train * a.warps_per_train + warp_global) * int64_t(n_ops) * NE2;
    const float2* dirs = a.op_dir ? s_dir : nullptr;
    int use_slot = 0, fill_slot = D - 1;
    const float2 neg1 = dup(-1.f);

    // One op in reverse; of a plain one (as is an odd op's even one then) the
    // steps are known when this is compiled.
    auto step = [&](auto plain, int o, int cur, const Op& op) {
        const uint32_t code = decltype(plain)::value ? kPlainOp : op.code;
        const bool odd = o & 1;
        const float4 tr = s_tring[(o % G) * VPB + vslot];
        const float2* ring = s_ring + cur * (NS * 3 * RP * T) + threadIdx.x * RP;

        // The pre-RF states: entry states (an odd op's by running the even op
        // before it), relaxed and pre-shifted.
        float2 P[NS][RP], M[NS][RP], Z[NS][RP];
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int kk = 0; kk < RP; ++kk) {
                P[s][kk] = ring[(s * 3 + 0) * T * RP + kk];
                M[s][kk] = ring[(s * 3 + 1) * T * RP + kk];
                Z[s][kk] = ring[(s * 3 + 2) * T * RP + kk];
            }
        float ddt[K], eps1[K], eps2[K], dal[K], dfl[K];
        if (odd) {
            const Op even = s_ops[o - 1];
            const uint32_t even_code = decltype(plain)::value ? kPlainOp : even.code;
            const float4 te = s_tring[((o - 1) % G) * VPB + vslot];
            op_directions<K, HOT>(a, dirs, n_ops, o - 1, even, v, ddt, eps1, eps2, dal, dfl);
            if (even_code & OP_RELAX) relax_all<RP, K, HOT>(P, M, Z, te.z, te.w, eps1, eps2, q);
            for (int s = 0; s < op_shift1(even_code); ++s) shift_all<RP, L, K>(P, M, q, kill, kill_r);
            if (op_rf(even_code) == RF_ROTATE)
                rotate_all<RP, K, HOT>(P, M, Z, te.x, te.y, dal);
            else if (op_rf(even_code) == RF_INVERT)
                invert_all<RP, K, HOT>(Z, v);
            for (int s = 0; s < op_shift2(even_code); ++s) shift_all<RP, L, K>(P, M, q, kill, kill_r);
            if (even_code & OP_SPOIL1) spoil_all<RP, K>(P, M);
            for (int s = 0; s < op_shift3(even_code); ++s) shift_all<RP, L, K>(P, M, q, kill, kill_r);
            if (even_code & OP_SPOIL2) spoil_all<RP, K>(P, M);
        }
        op_directions<K, HOT>(a, dirs, n_ops, o, op, v, ddt, eps1, eps2, dal, dfl);
        const bool relax = (code & OP_RELAX) != 0;
        if (relax) relax_all<RP, K, HOT>(P, M, Z, tr.z, tr.w, eps1, eps2, q);
        for (int s = 0; s < op_shift1(code); ++s) shift_all<RP, L, K>(P, M, q, kill, kill_r);

        // Reverse of the op's micro-steps after the pulse.
        if (code & OP_SPOIL2) spoil_all<RP, K>(pb, mb);
        for (int s = 0; s < op_shift3(code); ++s) shift_adjoint_all<RP, L, K>(pb, mb, q, kill, kill_r);
        if (code & OP_RECORD) {
            if (left == 0) refill(o);
            if (lane0) {
                const float* sv = seeds + slot * NI * EC + at;
#pragma unroll
                for (int s = 0; s < NS; ++s) pb[s][0].x += sv[s * EC];
                c_m0 += sv[NS * EC];
                if (!HOT)
#pragma unroll
                    for (int k = 0; k < K; ++k) v_m0[k] += sv[(NS + 1 + k) * EC];
            }
            ++at;
            --left;
        }
        if (code & OP_SPOIL1) spoil_all<RP, K>(pb, mb);
        for (int s = 0; s < op_shift2(code); ++s) shift_adjoint_all<RP, L, K>(pb, mb, q, kill, kill_r);

        float e_flip = 0.f, e_dt = 0.f;  // this lane's curvature of the op
        float ev_flip = 0.f, ev_dt = 0.f;  // value (K == 1)
        const int rf = op_rf(code);
        if (rf == RF_INVERT) {
            const float2 f = dup(-v.eff);
            float2 acc = dup(0.f);
            float2 vk[K];
#pragma unroll
            for (int k = 0; k < K; ++k) vk[k] = dup(0.f);
#pragma unroll
            for (int kk = 0; kk < RP; ++kk) {
                acc = fma2(zb[0][kk], Z[0][kk], acc);
                float2 nz = mul2(zb[0][kk], f);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const float2 zbk = zb[k + 1][kk];
                    acc = fma2(zbk, Z[k + 1][kk], acc);
                    if (!HOT) {
                        vk[k] = fma2(zbk, Z[0][kk], vk[k]);
                        nz = fma2(dup(-v.deff[k]), zbk, nz);
                    }
                    zb[k + 1][kk] = mul2(zbk, f);
                }
                zb[0][kk] = nz;
            }
            c_inv -= acc.x + acc.y;
            if (!HOT)
#pragma unroll
                for (int k = 0; k < K; ++k) v_inv[k] -= vk[k].x + vk[k].y;
        }
        // The pulse, in u = F+ + F-, w = F+ - F- (a pulse leaves u and turns
        // (w, Z), commuting with its generator w -> -2 Z, Z -> w / 2) and
        // their cotangents U, W = (F+_bar +- F-_bar) / 2; and at the point
        // before it the relaxation's inner products.
        const bool rotate = rf == RF_ROTATE;
        const float si = tr.x, co = tr.y;
        const float2 half = dup(0.5f), nhalf = dup(-0.5f);
        const float2 co2 = dup(co), hs = dup(0.5f * si), ns2 = dup(-2.f * si);
        float2 wz = dup(0.f), zw = dup(0.f);  // of dL/da
        float2 q2 = dup(0.f), q1 = dup(0.f);
        float2 gwz[K], gzw[K], c2[K], c1[K];  // of G_k; C2_k and C1_k
#pragma unroll
        for (int k = 0; k < K; ++k) gwz[k] = gzw[k] = c2[k] = c1[k] = dup(0.f);
#pragma unroll
        for (int kk = 0; kk < RP; ++kk) {
            const float2 ux = add2(P[0][kk], M[0][kk]), wx = fma2(neg1, M[0][kk], P[0][kk]);
            const float2 zx = Z[0][kk];
            float2 more_w = dup(0.f), more_z = dup(0.f);  // K^T mu_k a'_k
#pragma unroll
            for (int s = K; s >= 0; --s) {
                const int k = s - 1;
                const float2 u = s ? add2(P[s][kk], M[s][kk]) : ux;
                const float2 w = s ? fma2(neg1, M[s][kk], P[s][kk]) : wx;
                const float2 z = Z[s][kk];
                const float2 hp = mul2(half, pb[s][kk]);
                const float2 U = fma2(half, mb[s][kk], hp);
                float2 W = fma2(nhalf, mb[s][kk], hp), Zb = zb[s][kk];
                if (rotate) {
                    float2 W1 = mul2(co2, W), Z1 = mul2(ns2, W);
                    if (!s) {
                        W1 = add2(W1, more_w);
                        Z1 = add2(Z1, more_z);
                    }
                    W = fma2(hs, Zb, W1);
                    Zb = fma2(co2, Zb, Z1);
                    wz = fma2(W, z, wz);
                    zw = fma2(Zb, w, zw);
                }
                if (s && (!HOT || hot_dir(HOT, k) == 3) && rotate) {
                    gwz[k] = fma2(W, zx, gwz[k]);
                    gzw[k] = fma2(Zb, wx, gzw[k]);
                    more_w = fma2(dup(0.5f * dal[k]), Zb, more_w);
                    more_z = fma2(dup(-2.f * dal[k]), W, more_z);
                }
                q2 = fma2(U, u, fma2(W, w, q2));
                q1 = fma2(Zb, z, q1);
                if (s && (!HOT || hot_dir(HOT, k) == 2)) c2[k] = fma2(U, ux, fma2(W, wx, c2[k]));
                if (s && (!HOT || hot_dir(HOT, k) == 1)) c1[k] = fma2(Zb, zx, c1[k]);
                pb[s][kk] = add2(U, W);
                mb[s][kk] = fma2(neg1, W, U);
                zb[s][kk] = Zb;
            }
        }
        if (rotate) {
            const float gsum = 0.5f * (zw.x + zw.y) - 2.f * (wz.x + wz.y);
            float gf = gsum * v.b1, gb = gsum * op.flip;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const float g = 0.5f * (gzw[k].x + gzw[k].y) - 2.f * (gwz[k].x + gwz[k].y);
                if (HOT) {
                    if (hot_dir(HOT, k) == 3) gf += g;
                    continue;
                }
                gf = fmaf(g, v.db1[k], gf);
                gb = fmaf(g, dfl[k], gb);
                v_b1[k] = fmaf(g, op.flip, v_b1[k]);
                if (K == 1) ev_flip = g * v.b1;
            }
            e_flip = gf;
            c_b1 += gb;
        }
        if (relax) {
            const float Q2 = q2.x + q2.y;
            float Q1 = q1.x + q1.y;
            // The recovery target's part of lam.(x - e0).
            if (q == 0) Q1 -= zb[0][0].x;
            float dtc = 0.f;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                // A one-hot direction needs only its own.
                const bool n2 = !HOT || hot_dir(HOT, k) == 2;
                const bool n1 = !HOT || hot_dir(HOT, k) == 1;
                const float C2 = n2 ? c2[k].x + c2[k].y : 0.f;
                const float C1 = n1 ? c1[k].x + c1[k].y - (q == 0 ? zb[k + 1][0].x : 0.f) : 0.f;
                if (HOT) {
                    // r'_k = -w for the unit tangent of T1 (or T2).
                    if (n2) {
                        g_rd2[k] = fmaf(-op.dt, C2, g_rd2[k]);
                        dtc = fmaf(C2, v.w2, dtc);
                    }
                    if (n1) {
                        g_rd1[k] = fmaf(-op.dt, C1, g_rd1[k]);
                        dtc = fmaf(C1, v.w1, dtc);
                    }
                    continue;
                }
                g_r2 = fmaf(-C2, ddt[k], g_r2);
                g_r1 = fmaf(-C1, ddt[k], g_r1);
                g_rd2[k] = fmaf(-op.dt, C2, g_rd2[k]);
                g_rd1[k] = fmaf(-op.dt, C1, g_rd1[k]);
                // r'_k = -w T'_k.
                dtc = fmaf(C2, v.w2 * v.dt2[k], fmaf(C1, v.w1 * v.dt1[k], dtc));
                if (K == 1) ev_dt = -v.r2 * C2 - v.r1 * C1;
            }
            g_r2 = fmaf(-op.dt, Q2, g_r2);
            g_r1 = fmaf(-op.dt, Q1, g_r1);
            e_dt = -v.r2 * Q2 - v.r1 * Q1 + dtc;
        }
        for (int s = 0; s < op_shift1(code); ++s) shift_adjoint_all<RP, L, K>(pb, mb, q, kill, kill_r);
        if (relax) {
            const float2 E1 = dup(tr.z), E2 = dup(tr.w);
#pragma unroll
            for (int kk = 0; kk < RP; ++kk) {
                float2 lp = mul2(pb[0][kk], E2), lm = mul2(mb[0][kk], E2), lz = mul2(zb[0][kk], E1);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    pb[k + 1][kk] = mul2(pb[k + 1][kk], E2);
                    mb[k + 1][kk] = mul2(mb[k + 1][kk], E2);
                    zb[k + 1][kk] = mul2(zb[k + 1][kk], E1);
                    if (!HOT || hot_dir(HOT, k) == 2) {
                        lp = fma2(dup(eps2[k]), pb[k + 1][kk], lp);
                        lm = fma2(dup(eps2[k]), mb[k + 1][kk], lm);
                    }
                    if (!HOT || hot_dir(HOT, k) == 1) lz = fma2(dup(eps1[k]), zb[k + 1][kk], lz);
                }
                pb[0][kk] = lp;
                mb[0][kk] = lm;
                zb[0][kk] = lz;
            }
        }
        // The op's event partials summed over the warp in a fixed order: one
        // exchange (two for four values) leaves each lane one of the values,
        // the rest sum it. Nothing on the state recursion waits for it.
        float f0 = active ? e_flip : 0.f, f1 = active ? e_dt : 0.f;
        const bool upper = lane & 16, high = lane & 8;
        if constexpr (NE2 == 2) {
            float f2 = active ? ev_flip : 0.f, f3 = active ? ev_dt : 0.f;
            const float x0 = __shfl_xor_sync(0xffffffffu, upper ? f0 : f2, 16);
            const float x1 = __shfl_xor_sync(0xffffffffu, upper ? f1 : f3, 16);
            f0 = (upper ? f2 : f0) + x0;
            f1 = (upper ? f3 : f1) + x1;
            f0 = (high ? f1 : f0) + __shfl_xor_sync(0xffffffffu, high ? f0 : f1, 8);
        } else {
            f0 = (upper ? f1 : f0) + __shfl_xor_sync(0xffffffffu, upper ? f0 : f1, 16);
            f0 += __shfl_xor_sync(0xffffffffu, f0, 8);
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) f0 += __shfl_xor_sync(0xffffffffu, f0, off);
        constexpr int kHolders = 16 / NE2;  // lanes that hold one value
        if (lane % kHolders == 0)
            reinterpret_cast<float*>(event_out + int64_t(o) * NE2)[lane / kHolders] = f0;
    };

    for (int o = n_ops - 1; o >= 0; --o) {
        const bool odd = o & 1;
        const bool new_pair = odd || o == n_ops - 1;
        if (new_pair) {
            if (o % G == G - 1 || o == n_ops - 1) {
                // The transcendentals of the group of G ops that ends here:
                // lane q of a voxel evaluates the group's op q (a lone lane
                // both), so one pass of the warp covers them. (Their last
                // readers are done.)
                __syncwarp();
#pragma unroll
                for (int e = 0; e < (L < 2 ? 2 : 1); ++e) {
                    const int oq = o - o % G + q + e;
                    if (slot < VPW && q < G && oq <= o) {
                        const Op opq = s_ops[oq];
                        float si = 0.f, co = 1.f;
                        if (op_rf(opq.code) == RF_ROTATE) sincosf(opq.flip * v.b1, &si, &co);
                        s_tring[(oq % G) * VPB + vslot] =
                            make_float4(si, co, expf(-v.r1 * opq.dt), expf(-v.r2 * opq.dt));
                    }
                }
            }
            // Orders the lanes' reads of the slot this fetch refills (used by
            // the last pair) and the transcendentals written above.
            __syncwarp();
            if ((o >> 1) - (D - 1) >= 0) fetch((o >> 1) - (D - 1), fill_slot);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            fill_slot = fill_slot + 1 == D ? 0 : fill_slot + 1;
            asm volatile("cp.async.wait_group %0;\n" ::"n"(D - 1) : "memory");
            __syncwarp();  // the transcendentals another lane wrote
        }
        const Op op = s_ops[o];
        const int cur = use_slot;
        if (!odd) use_slot = use_slot + 1 == D ? 0 : use_slot + 1;
        if (op.code == kPlainOp && (!odd || s_ops[o - 1].code == kPlainOp))
            step(std::true_type{}, o, cur, op);
        else
            step(std::false_type{}, o, cur, op);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");

    // Tissue: r = 1000/T, r'_k = -1000 T'_k/T^2, summed over the voxel's lanes.
    // One-hot directions write the curvature only.
    constexpr int NV = HOT ? 5 : 5 * (1 + K);
    float out[NV];
    {
        float gt1 = -v.w1 * g_r1, gt2 = -v.w2 * g_r2;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (HOT) {
                if (hot_dir(HOT, k) == 1) gt1 = fmaf(g_rd1[k], 2.f * v.w1 / v.t1, gt1);
                if (hot_dir(HOT, k) == 2) gt2 = fmaf(g_rd2[k], 2.f * v.w2 / v.t2, gt2);
                continue;
            }
            gt1 = fmaf(g_rd1[k], 2.f * v.w1 * v.dt1[k] / v.t1, gt1);
            gt2 = fmaf(g_rd2[k], 2.f * v.w2 * v.dt2[k] / v.t2, gt2);
        }
        out[0] = gt1;
        out[1] = gt2;
        out[2] = c_m0;
        out[3] = c_b1;
        out[4] = c_inv;
        if constexpr (!HOT) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                out[5 + 5 * k + 0] = -v.w1 * g_rd1[k];
                out[5 + 5 * k + 1] = -v.w2 * g_rd2[k];
                out[5 + 5 * k + 2] = v_m0[k];
                out[5 + 5 * k + 3] = v_b1[k];
                out[5 + 5 * k + 4] = v_inv[k];
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const float x = active ? out[j] : 0.f;
        float sum = 0.f;
#pragma unroll
        for (int l = 0; l < L; ++l) sum += __shfl_sync(0xffffffffu, x, lane - q + l);
        out[j] = sum;
    }
    if (lane0) {
        float* dst = a.tissue_partial + row * NV;
#pragma unroll
        for (int j = 0; j < NV; ++j) dst[j] = out[j];
    }
}

template <int RP, int L, int K, int HOT>
void launch_second_forward(const SecondArgs& a, dim3 grid, dim3 block, size_t smem,
                           cudaStream_t s) {
    second_forward_kernel<RP, L, K, HOT><<<grid, block, smem, s>>>(a);
}

template <int RP, int L, int K, int HOT>
void launch_second_reverse(const SecondArgs& a, dim3 grid, dim3 block, size_t smem,
                           cudaStream_t s) {
    second_reverse_kernel<RP, L, K, HOT><<<grid, block, smem, s>>>(a);
}

// One (orders per lane, lanes per voxel) shape for K directions, general
// (hot == 0) or one-hot (the direction code of hot_dir).
struct SecondEntry {
    int orders_per_lane;
    int lanes_per_voxel;
    int directions;
    int hot;
    void (*forward)(const SecondArgs&, dim3, dim3, size_t, cudaStream_t);
    void (*reverse)(const SecondArgs&, dim3, dim3, size_t, cudaStream_t);
    const void* reverse_fn;
};

#define TSG_SECOND_ENTRY(R, L, K, HOT)                                                  \
    {R,                                                                                 \
     L,                                                                                 \
     K,                                                                                 \
     HOT,                                                                               \
     &launch_second_forward<(R) / 2, L, K, HOT>,                                        \
     &launch_second_reverse<(R) / 2, L, K, HOT>,                                        \
     reinterpret_cast<const void*>(&second_reverse_kernel<(R) / 2, L, K, HOT>)}

// The shapes instantiated per direction set: general directions take every
// shape, one-hot sets the ones measured useful.
#define TSG_SECOND_SHAPES_HOT(K, HOT)                                                     \
    TSG_SECOND_ENTRY(2, 4, K, HOT), TSG_SECOND_ENTRY(2, 5, K, HOT),                       \
        TSG_SECOND_ENTRY(2, 8, K, HOT), TSG_SECOND_ENTRY(2, 10, K, HOT),                  \
        TSG_SECOND_ENTRY(2, 16, K, HOT), TSG_SECOND_ENTRY(2, 32, K, HOT),                 \
        TSG_SECOND_ENTRY(4, 1, K, HOT), TSG_SECOND_ENTRY(4, 2, K, HOT),                   \
        TSG_SECOND_ENTRY(4, 4, K, HOT), TSG_SECOND_ENTRY(4, 5, K, HOT),                   \
        TSG_SECOND_ENTRY(4, 8, K, HOT)

// Every table of one translation unit.
const SecondEntry* second_table(int k, int hot, int* count);

}  // namespace tsg
