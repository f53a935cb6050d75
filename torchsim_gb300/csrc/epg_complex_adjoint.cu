// The first-order adjoint of the complex EPG sweep (one pool, instant RF):
// gradients with respect to T1, T2, M0, B1, the inversion efficiency, the
// transmit phase (B1phase) and off-resonance (B0) per voxel, and the flip,
// duration and phase of every event -- the reference's complex
// simulate_vjp_range<INSTANT, ONE> (src/torchsim/_epg_cpu.cpp:4840-5985).
//
// Trajectory mode, as the real adjoint's: a forward sweep stores every op's
// entry state (the six real planes F+ re/im, F- re/im, Z re/im of each lane's
// order pairs, one tile per warp so that stores and loads are whole lines)
// and every recorded F+[0]; the reverse sweep streams them back through a
// cp.async ring and re-applies only each op's relaxation and pre-shift. Both
// hold a voxel's order pairs one after the other, so the forward can run on
// twice the lanes of the reverse.
//
// The states are held in the frame of the last pulse, F+ e^{-i phi} and
// F- e^{i phi}: the turn from one pulse's frame to the next joins the
// relaxation's complex factor, B1phase (the same turn for every pulse) leaves
// the states altogether, and the pulse has real coefficients. With u = F+ + F-
// and w = F+ - F- it leaves u and turns (w, Z) alone:
//   wr' = cos a wr + 2 sin a Zi,  Zi' = cos a Zi - sin a / 2 wr
//   wi' = cos a wi - 2 sin a Zr,  Zr' = cos a Zr + sin a / 2 wi
// so it is half the arithmetic of the general complex 3x3 and commutes with
// its derivative.
//
// Adjoint algebra (complex cotangents y_bar = dL/dRe y + i dL/dIm y; for
// y = a x the cotangent is x_bar = conj(a) y_bar, and a parameter p of a
// contributes Re(sum conj(y_bar) (da/dp) x)). U, W = (F+_bar +- F-_bar) / 2,
// everything before the pulse:
//   pulse    (W, Z_bar) turn back; dL/dalpha = <x_bar, K x> with K the
//            pulse's generator = 2 (Wr Zi - Wi Zr) + (Zr_bar wi - Zi_bar wr) / 2.
//   record   v = m0 F+[0] e^{-i phi_r}: F+[0]_bar += m0 e^{i phi_r} g;
//            dL/dm0 = Re(conj(g) F+[0] e^{-i phi_r}), dL/dphi_r = Re(conj(g) (-i v)).
//   relax    F+ *= T, F- *= conj(T), T = e2 e^{i off}, off = -2 pi B0 dt;
//            with the pre-pulse states and cotangents (the shift commutes
//            with these inner products): dL/dlog e2 = <U, u> + <W, w>,
//            dL/doff = Q = Ui wr + Wi ur - Ur wi - Wr ui, dL/dlog e1 =
//            <zb, z> - Re zb[0].
//   phase    T(phi) = D T(0) D^-1: dL/dphi is Q after the pulse less Q
//            before it, so Ui dwr + ur dWi - Ur dwi - ui dWr with the
//            pulse's own changes of w and W.
#include "epg_complex.cuh"

#include <type_traits>

namespace tsg {

namespace {

using namespace complex_detail;

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

constexpr uint32_t kPlainOp = kFastBits | OP_RECORD;
constexpr int kCxWarps = 2;
constexpr int kCxRing = 2;

struct ComplexAdjointArgs {
    const Op* ops;
    const float2* phase;  // [train][ops]: (pulse phase, receiver phase)
    int n_ops;
    int64_t atoms;
    int states;
    int outputs;
    const float* t1;
    const float* t2;
    const float* m0;
    const float* b1;
    const float* inv;
    const float* b1_phase;
    const float* b0;
    // Forward: the signal (nullable), the trajectory
    // [train][warp][op][6 planes][lane][RP] float2 with the forward's warps,
    // a voxel's order pairs one after the other, and the recorded F+[0]
    // [train][output][atom] float2.
    int layout;
    float* out_a;
    float* out_b;
    float2* traj;
    int tile_voxels;  // of a forward warp
    int plane_pairs;  // its 32 RP
    float2* traj_rec;
    // Reverse: the complex seed (planes or interleaved complex), partials
    // per (train, warp, op) 2 float2 (flip, duration), (pulse phase,
    // receiver phase) and per (train, atom) 7 floats (t1, t2, m0, b1,
    // inversion, b1 phase, b0).
    const float* seed_a;
    const float* seed_b;
    int seed_layout;
    float2* event_partial;
    float* tissue_partial;
    int64_t warps_per_train;
};

// Transpose of shift_complex on the cotangents: F+ cotangents move one order
// down, F- cotangents one order up, and F+[0] = conj(F-[0]) returns
// conj(pb[0]) to the F- order that became F-[0]. The slot at order `states`
// only receives F- cotangent from below; it is kept empty.
template <int RP, int L>
__device__ __forceinline__ void shift_complex_adjoint(float2 (&pr)[RP], float2 (&pi)[RP],
                                                      float2 (&mr)[RP], float2 (&mi)[RP], int q,
                                                      bool kill, int kill_r) {
    const float carry_r = pr[0].x, carry_i = -pi[0].x;
    float in_pr = 0.f, in_pi = 0.f, in_mr = 0.f, in_mi = 0.f;
    if constexpr (L > 1) {
        in_pr = __shfl_down_sync(0xffffffffu, pr[0].x, 1);
        in_pi = __shfl_down_sync(0xffffffffu, pi[0].x, 1);
        in_mr = __shfl_up_sync(0xffffffffu, mr[RP - 1].y, 1);
        in_mi = __shfl_up_sync(0xffffffffu, mi[RP - 1].y, 1);
    }
    const bool top_lane = L == 1 || q == L - 1;
#pragma unroll
    for (int k = 0; k < RP; ++k) {
        pr[k].x = pr[k].y;
        pi[k].x = pi[k].y;
        pr[k].y = (k + 1 < RP) ? pr[k + 1].x : (top_lane ? 0.f : in_pr);
        pi[k].y = (k + 1 < RP) ? pi[k + 1].x : (top_lane ? 0.f : in_pi);
    }
    const bool first = L == 1 || q == 0;
#pragma unroll
    for (int k = RP - 1; k >= 0; --k) {
        mr[k].y = mr[k].x;
        mi[k].y = mi[k].x;
        mr[k].x = (k > 0) ? mr[k - 1].y : (first ? 0.f : in_mr);
        mi[k].x = (k > 0) ? mi[k - 1].y : (first ? 0.f : in_mi);
    }
    if (first) {
        mr[0].y += carry_r;
        mi[0].y += carry_i;
    }
    if (kill) {
#pragma unroll
        for (int k = 0; k < RP; ++k) {
            if (2 * k == kill_r) mr[k].x = mi[k].x = 0.f;
            if (2 * k + 1 == kill_r) mr[k].y = mi[k].y = 0.f;
        }
    }
}

// Turns staged phases (pulse, receiver) into every op's two angles in the
// frame of the last pulse: how far its own pulse turns that frame (0 without
// one), and its receiver phase in it. (Nothing is transverse before the first
// pulse, so the first frame is free.) One warp does it, 32 ops at a time;
// `last` and `any` carry the last pulse's phase, and whether there was one,
// from chunk to chunk.
__device__ __forceinline__ void frame_angles(const Op* ops, float2* ph, int count, int lane,
                                             float& last, bool& any) {
    for (int base = 0; base < count; base += 32) {
        const int i = base + lane;
        const float2 x = i < count ? ph[i] : make_float2(0.f, 0.f);
        const bool pulse = i < count && op_rf(ops[i].code) == RF_ROTATE;
        const unsigned set = __ballot_sync(0xffffffffu, pulse);
        const unsigned below = set & ((1u << lane) - 1u);
        const float near = __shfl_sync(0xffffffffu, x.x, below ? 31 - __clz(below) : 0);
        const float before = below ? near : any ? last : pulse ? x.x : 0.f;
        if (i < count) ph[i] = make_float2(pulse ? x.x - before : 0.f, x.y - (pulse ? x.x : before));
        const float latest = __shfl_sync(0xffffffffu, x.x, set ? 31 - __clz(set) : 0);
        if (set) last = latest;
        any |= set != 0;
    }
}

// The transcendentals of one op for one voxel: e1, the F+ factor tr + i ti
// (relaxation, off-resonance and the turn of the frame), the flip's and the
// receiver's sine and cosine.
struct FrameTrig {
    float e1 = 1.f, tr = 1.f, ti = 0.f;
    float sa = 0.f, ca = 1.f;
    float sr = 0.f, cr = 1.f;
};

__device__ __forceinline__ FrameTrig frame_trig(const Op& op, float2 angle, float r1, float r2,
                                                float b1, float b1_phase, float b0, bool off_axis) {
    FrameTrig t;
    const uint32_t code = op.code;
    if (code & OP_RELAX) {
        t.e1 = expf(-r1 * op.dt);
        t.tr = expf(-r2 * op.dt);
        if (off_axis) {
            float so, co;
            sincosf(-2.f * 3.14159265358979323846f * b0 * op.dt, &so, &co);
            t.ti = t.tr * so;
            t.tr *= co;
        }
    }
    if (angle.x != 0.f) {
        float sp, cp;
        sincosf(angle.x, &sp, &cp);
        const float re = t.tr, im = t.ti;
        t.tr = re * cp + im * sp;
        t.ti = im * cp - re * sp;
    }
    if (op_rf(code) == RF_ROTATE) sincosf(op.flip * b1, &t.sa, &t.ca);
    if (code & OP_RECORD) sincosf(angle.y - b1_phase, &t.sr, &t.cr);
    return t;
}

// Forward storing the trajectory.
template <int RP, int L>
__global__ void __launch_bounds__(128) complex_forward_traj_kernel(const ComplexAdjointArgs a) {
    constexpr int R = 2 * RP;
    constexpr int VPW = 32 / L;
    __shared__ Op s_ops[kComplexOpChunk];
    __shared__ float2 s_ph[kComplexOpChunk];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int q = lane % L;
    const int slot = lane / L;
    const int64_t warp_global = int64_t(blockIdx.x) * (blockDim.x >> 5) + warp;
    const int64_t atom = warp_global * VPW + slot;
    const int64_t train = blockIdx.y;
    const bool active = slot < VPW && atom < a.atoms;
    const int64_t ac = active ? atom : 0;
    const float r1 = 1000.f / a.t1[ac];
    const float r2 = 1000.f / a.t2[ac];
    const float m0 = a.m0 ? a.m0[ac] : 1.f;
    const float b1 = a.b1 ? a.b1[ac] : 1.f;
    const float eff = a.inv ? a.inv[ac] : 1.f;
    const float b1_phase = a.b1_phase ? a.b1_phase[ac] : 0.f;
    const float b0 = a.b0 ? a.b0[ac] : 0.f;
    const bool kill = L * R > a.states;
    const int kill_r = a.states - q * R;

    float2 X[6][RP];  // Pr, Pi, Mr, Mi, Zr, Zi
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int k = 0; k < RP; ++k) X[p][k] = dup(0.f);
    if (q == 0) X[4][0].x = 1.f;

    const Op* ops = a.ops + train * a.n_ops;
    const float2* phase = a.phase + train * a.n_ops;
    const int64_t row = train * a.atoms + atom;
    const int64_t n_warps = (a.atoms + VPW - 1) / VPW;
    const int64_t op_stride = 6 * 32 * RP;
    float2* lane_traj = warp_global < n_warps
                            ? a.traj + (train * n_warps + warp_global) * a.n_ops * op_stride + lane * RP
                            : nullptr;

    // Each op's transcendentals are the same for the L lanes of a voxel:
    // lane q evaluates them for one of the next L ops and the lanes exchange
    // them by shuffle.
    const int first_lane = lane - q;
    const bool off_axis = a.b0 != nullptr;
    FrameTrig mine;
    float frame = 0.f;
    bool framed = false;

    for (int base = 0; base < a.n_ops; base += kComplexOpChunk) {
        const int count = min(kComplexOpChunk, a.n_ops - base);
        __syncthreads();
        for (int i = threadIdx.x; i < count; i += blockDim.x) {
            s_ops[i] = ops[base + i];
            s_ph[i] = phase[base + i];
        }
        __syncthreads();
        if (warp == 0) frame_angles(s_ops, s_ph, count, lane, frame, framed);
        __syncthreads();
        for (int i = 0; i < count; ++i) {
            const Op op = s_ops[i];
            const uint32_t code = op.code;
            const int src = first_lane + i % L;
            if constexpr (L > 1) {
                if (i % L == 0) {
                    const int j = i + q;
                    mine = j < count ? frame_trig(s_ops[j], s_ph[j], r1, r2, b1, b1_phase, b0, off_axis)
                                     : FrameTrig{};
                }
            } else {
                mine = frame_trig(op, s_ph[i], r1, r2, b1, b1_phase, b0, off_axis);
            }
            // This op's value of one field (shuffled where it is used, so the
            // fields are live only there; every lane takes part).
            auto tv = [&](float v) { return L > 1 ? __shfl_sync(0xffffffffu, v, src) : v; };
            if (lane_traj) {
                float2* dst = lane_traj + int64_t(base + i) * op_stride;
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int k = 0; k < RP; ++k) dst[p * 32 * RP + k] = X[p][k];
            }
            if ((code & OP_RELAX) || s_ph[i].x != 0.f) {
                const float e1 = tv(mine.e1), tr = tv(mine.tr), ti = tv(mine.ti);
                const float2 T = dup(tr), Ti = dup(ti), nTi = dup(-ti), E1 = dup(e1);
#pragma unroll
                for (int k = 0; k < RP; ++k) {
                    const float2 pr = X[0][k], pi = X[1][k], mr = X[2][k], mi = X[3][k];
                    X[0][k] = fma2(nTi, pi, mul2(T, pr));
                    X[1][k] = fma2(Ti, pr, mul2(T, pi));
                    X[2][k] = fma2(Ti, mi, mul2(T, mr));
                    X[3][k] = fma2(nTi, mr, mul2(T, mi));
                    X[4][k] = mul2(X[4][k], E1);
                    X[5][k] = mul2(X[5][k], E1);
                }
                if (q == 0) X[4][0].x += 1.f - e1;
            }
            for (int s = 0; s < op_shift1(code); ++s)
                shift_complex<RP, L>(X[0], X[1], X[2], X[3], q, kill, kill_r);
            const int rf = op_rf(code);
            if (rf == RF_ROTATE) {
                const float sa = tv(mine.sa), ca = tv(mine.ca);
                const float2 co = dup(ca), s2 = dup(2.f * sa), ns2 = dup(-2.f * sa);
                const float2 hs = dup(0.5f * sa), nhs = dup(-0.5f * sa);
                const float2 half = dup(0.5f), nhalf = dup(-0.5f), minus = dup(-1.f);
#pragma unroll
                for (int k = 0; k < RP; ++k) {
                    const float2 hur = mul2(half, add2(X[0][k], X[2][k]));
                    const float2 hui = mul2(half, add2(X[1][k], X[3][k]));
                    const float2 wr = fma2(minus, X[2][k], X[0][k]);
                    const float2 wi = fma2(minus, X[3][k], X[1][k]);
                    const float2 zr = X[4][k], zi = X[5][k];
                    const float2 vr = fma2(s2, zi, mul2(co, wr)), vi = fma2(ns2, zr, mul2(co, wi));
                    X[4][k] = fma2(hs, wi, mul2(co, zr));
                    X[5][k] = fma2(nhs, wr, mul2(co, zi));
                    X[0][k] = fma2(half, vr, hur);
                    X[1][k] = fma2(half, vi, hui);
                    X[2][k] = fma2(nhalf, vr, hur);
                    X[3][k] = fma2(nhalf, vi, hui);
                }
            } else if (rf == RF_INVERT) {
                const float2 f = dup(-eff);
#pragma unroll
                for (int k = 0; k < RP; ++k) {
                    X[4][k] = mul2(X[4][k], f);
                    X[5][k] = mul2(X[5][k], f);
                }
            }
            for (int s = 0; s < op_shift2(code); ++s)
                shift_complex<RP, L>(X[0], X[1], X[2], X[3], q, kill, kill_r);
            if (code & OP_SPOIL1) {
#pragma unroll
                for (int k = 0; k < RP; ++k) X[0][k] = X[1][k] = X[2][k] = X[3][k] = dup(0.f);
            }
            float sr = 0.f, cr = 1.f;
            if (code & OP_RECORD) {
                sr = tv(mine.sr);
                cr = tv(mine.cr);
            }
            if ((code & OP_RECORD) && q == 0 && active) {
                const float xr = X[0][0].x, xi = X[1][0].x;
                a.traj_rec[(train * a.outputs + op.record) * a.atoms + atom] = make_float2(xr, xi);
                if (a.out_a)
                    put(a.layout, a.out_a, a.out_b, row * a.outputs + op.record,
                        m0 * (xr * cr + xi * sr), m0 * (xi * cr - xr * sr));
            }
            for (int s = 0; s < op_shift3(code); ++s)
                shift_complex<RP, L>(X[0], X[1], X[2], X[3], q, kill, kill_r);
            if (code & OP_SPOIL2) {
#pragma unroll
                for (int k = 0; k < RP; ++k) X[0][k] = X[1][k] = X[2][k] = X[3][k] = dup(0.f);
            }
        }
    }
}

// <y, x> summed over a lane's pairs: the real inner product of two planes.
template <int RP>
__device__ __forceinline__ float2 dot_acc(const float2 (&y)[RP], const float2 (&x)[RP], float2 acc) {
#pragma unroll
    for (int k = 0; k < RP; ++k) acc = fma2(y[k], x[k], acc);
    return acc;
}

// The reverse sweep. Dynamic shared memory: the entry-state ring
// [D][6][T][RP] float2, then the ops [n_ops] and their phases [n_ops].
// Two orders per lane hold the reverse step in 96 registers, ten blocks per
// SM; four orders per lane (the default shapes where they fit) take what they
// need: held to 128 registers they spill, 1.24 to 1.43 ms at 16,384 voxels x
// 601 ops x 20 states.
//
// Bound: the latency of an op's chain at two warps a scheduler (0.47 issued a
// cycle); the trajectory's 5 GB there are 0.75 ms. With the
// general 3x3 pulse (states outside its frame, derivatives by applying their
// own matrices), seeds read where they are used and two orders per lane it was
// 2.13 ms; the frame takes 0.30 off, the seeds 0.26, four orders 0.33 and the
// plain ops' own copy of the step 0.09 (1.16 ms).
//
// WIDE: a lane's two pairs are copied as one 16-byte piece, for which the
// trajectory has to be 16-byte aligned; else pair by pair.
template <int RP, int L, bool WIDE>
__global__ void __launch_bounds__(32 * kCxWarps, RP == 1 ? 10 : 1)
    complex_adjoint_kernel(const ComplexAdjointArgs a) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    constexpr int W = kCxWarps;
    constexpr int T = 32 * W;
    constexpr int R = 2 * RP;
    constexpr int VPW = 32 / L;
    constexpr int D = kCxRing;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int q = lane % L;
    const int slot = lane / L;
    const int64_t warp_global = int64_t(blockIdx.x) * W + warp;
    const int64_t atom = warp_global * VPW + slot;
    const int64_t train = blockIdx.y;
    const bool active = slot < VPW && atom < a.atoms;
    const int64_t ac = active ? atom : 0;
    const bool lane0 = active && q == 0;
    const int n_ops = a.n_ops;
    const int64_t n = a.atoms;
    const int64_t row = train * n + atom;
    const float t1 = a.t1[ac], t2 = a.t2[ac];
    const float r1 = 1000.f / t1, r2 = 1000.f / t2;
    const float w1 = 1000.f / (t1 * t1), w2 = 1000.f / (t2 * t2);
    const float m0 = a.m0 ? a.m0[ac] : 1.f;
    const float b1 = a.b1 ? a.b1[ac] : 1.f;
    const float eff = a.inv ? a.inv[ac] : 1.f;
    const float b1_phase = a.b1_phase ? a.b1_phase[ac] : 0.f;
    const float b0 = a.b0 ? a.b0[ac] : 0.f;
    const bool kill = L * R > a.states;
    const int kill_r = a.states - q * R;
    constexpr float kTwoPi = 6.28318530717958647692f;

    float2* s_ring = reinterpret_cast<float2*>(s_raw);           // [D][6][T][RP]
    Op* s_ops = reinterpret_cast<Op*>(s_ring + D * 6 * T * RP);  // [n_ops]
    float2* s_ph = reinterpret_cast<float2*>(s_ops + n_ops);     // [n_ops]
    {
        const Op* ops = a.ops + train * n_ops;
        const float2* ph = a.phase + train * n_ops;
        for (int i = threadIdx.x; i < n_ops; i += T) {
            s_ops[i] = ops[i];
            s_ph[i] = ph[i];
        }
        __syncthreads();
        float frame = 0.f;
        bool framed = false;
        if (warp == 0) frame_angles(s_ops, s_ph, n_ops, lane, frame, framed);
        __syncthreads();
    }

    // (Lanes without a voxel read the first one's.)
    const int64_t n_tiles = (n + a.tile_voxels - 1) / a.tile_voxels;
    const int64_t tile = ac / a.tile_voxels;
    const int plane = a.plane_pairs;
    const int64_t op_stride = 6 * plane;
    const float2* lane_traj = a.traj + (train * n_tiles + tile) * n_ops * op_stride +
                              (ac - tile * a.tile_voxels) * (L * RP) + q * RP;
    const unsigned ring_base =
        static_cast<unsigned>(__cvta_generic_to_shared(s_ring + threadIdx.x * RP));
    auto fetch = [&](int o, int rs) {
        const float2* src = lane_traj + o * op_stride;
        const unsigned dst = ring_base + unsigned(rs * 6 * T * RP) * 8u;
#pragma unroll
        for (int p = 0; p < 6; ++p) {
            if constexpr (WIDE) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                                 dst + unsigned(p * T * RP) * 8u),
                             "l"(src + p * plane)
                             : "memory");
            } else {
#pragma unroll
                for (int k = 0; k < RP; ++k)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                                     dst + unsigned(p * T * RP + k) * 8u),
                                 "l"(src + p * plane + k)
                                 : "memory");
            }
        }
    };

    // Seeds: planes (re plane, im plane) or interleaved complex.
    const bool planes = a.seed_layout == TSG_LAYOUT_PLANES;
    const float2* rec_col = a.traj_rec + train * int64_t(a.outputs) * n + ac;

    float2 B[6][RP];  // cotangents Pr, Pi, Mr, Mi, Zr, Zi
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int k = 0; k < RP; ++k) B[p][k] = dup(0.f);
    float g_t1 = 0.f, g_t2 = 0.f, g_m0 = 0.f, g_b1 = 0.f, g_inv = 0.f, g_b1p = 0.f, g_b0 = 0.f;

#pragma unroll
    for (int j = 1; j < D; ++j) {
        if (n_ops - j >= 0) fetch(n_ops - j, j - 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    float2* event_out = a.event_partial + (train * a.warps_per_train + warp_global) * int64_t(n_ops) * 2;
    int use_slot = 0, fill_slot = D - 1;
    // Each op's transcendentals, evaluated once per voxel: lane q takes one
    // of the next L ops of the reverse sweep (op o - q) and the lanes
    // exchange them by shuffle.
    const int first_lane = lane - q;
    const bool off_axis = a.b0 != nullptr;
    FrameTrig mine;
    // An op's seed and recorded F+[0], read while the op after it runs.
    float2 next_seed = dup(0.f), next_x0 = dup(0.f);
    auto read_record = [&](int o) {
        if (o < 0 || !lane0 || !(s_ops[o].code & OP_RECORD)) return;
        const int64_t r = s_ops[o].record;
        const int64_t idx = row * a.outputs + r;
        next_seed = planes ? make_float2(a.seed_a[idx], a.seed_b[idx])
                           : reinterpret_cast<const float2*>(a.seed_a)[idx];
        next_x0 = rec_col[r * n];
    };
    read_record(n_ops - 1);

    // One op in reverse; of a plain one (relaxation, pulse, sample, shift: most
    // ops of a fingerprinting train) the steps are known when this is compiled.
    auto step = [&](auto plain, int o, const Op& op) {
        const float2 seed = next_seed, rec0 = next_x0;
        read_record(o - 1);
        if (o - (D - 1) >= 0) fetch(o - (D - 1), fill_slot);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        fill_slot = fill_slot + 1 == D ? 0 : fill_slot + 1;
        const float2 ph = s_ph[o];
        const uint32_t code = decltype(plain)::value ? kPlainOp : op.code;
        const int g = (n_ops - 1 - o) % L;
        const int src = first_lane + g;
        if constexpr (L > 1) {
            if (g == 0) {
                const int j = o - q;
                mine = j >= 0 ? frame_trig(s_ops[j], s_ph[j], r1, r2, b1, b1_phase, b0, off_axis)
                              : FrameTrig{};
            }
        } else {
            mine = frame_trig(op, ph, r1, r2, b1, b1_phase, b0, off_axis);
        }
        // This op's value of one field (shuffled where it is used, so the
        // fields are live only there; every lane takes part).
        auto tv = [&](float v) { return L > 1 ? __shfl_sync(0xffffffffu, v, src) : v; };
        asm volatile("cp.async.wait_group %0;\n" ::"n"(D - 1) : "memory");
        const float2* ring = s_ring + use_slot * (6 * T * RP) + threadIdx.x * RP;
        use_slot = use_slot + 1 == D ? 0 : use_slot + 1;
        float2 X[6][RP];
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int k = 0; k < RP; ++k) X[p][k] = ring[p * T * RP + k];

        // Replay the relaxation (and the turns) and the pre-shift.
        const bool relax = (code & OP_RELAX) != 0;
        const bool turn = relax || ph.x != 0.f;
        float e1 = 1.f, tr = 1.f, ti = 0.f;
        if (turn) {
            e1 = tv(mine.e1);
            tr = tv(mine.tr);
            ti = tv(mine.ti);
            const float2 Tr = dup(tr), Ti = dup(ti), nTi = dup(-ti), E1 = dup(e1);
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                const float2 pr = X[0][k], pi = X[1][k], mr = X[2][k], mi = X[3][k];
                X[0][k] = fma2(nTi, pi, mul2(Tr, pr));
                X[1][k] = fma2(Ti, pr, mul2(Tr, pi));
                X[2][k] = fma2(Ti, mi, mul2(Tr, mr));
                X[3][k] = fma2(nTi, mr, mul2(Tr, mi));
                X[4][k] = mul2(X[4][k], E1);
                X[5][k] = mul2(X[5][k], E1);
            }
            if (q == 0) X[4][0].x += 1.f - e1;
        }
        for (int s = 0; s < op_shift1(code); ++s)
            shift_complex<RP, L>(X[0], X[1], X[2], X[3], q, kill, kill_r);

        // The op's micro-steps after the pulse, reversed.
        if (code & OP_SPOIL2) {
#pragma unroll
            for (int k = 0; k < RP; ++k) B[0][k] = B[1][k] = B[2][k] = B[3][k] = dup(0.f);
        }
        for (int s = 0; s < op_shift3(code); ++s)
            shift_complex_adjoint<RP, L>(B[0], B[1], B[2], B[3], q, kill, kill_r);
        float e_rec = 0.f;  // this lane's d/d(receiver phase)
        float sr = 0.f, cr = 1.f;
        if (code & OP_RECORD) {
            sr = tv(mine.sr);
            cr = tv(mine.cr);
        }
        if ((code & OP_RECORD) && lane0) {
            const float gr = seed.x, gi = seed.y;
            // d = e^{-i phi_r}: F+[0] d, and v = m0 F+[0] d.
            const float fr = rec0.x * cr + rec0.y * sr, fi = rec0.y * cr - rec0.x * sr;
            g_m0 = fmaf(gr, fr, fmaf(gi, fi, g_m0));
            // dv/dphi_r = -i v: Re(conj(g) (-i v)) = m0 (gr fi - gi fr).
            e_rec = m0 * (gr * fi - gi * fr);
            // F+[0]_bar += m0 conj(d) g = m0 e^{i phi_r} g.
            B[0][0].x += m0 * (cr * gr - sr * gi);
            B[1][0].x += m0 * (cr * gi + sr * gr);
        }
        if (code & OP_SPOIL1) {
#pragma unroll
            for (int k = 0; k < RP; ++k) B[0][k] = B[1][k] = B[2][k] = B[3][k] = dup(0.f);
        }
        for (int s = 0; s < op_shift2(code); ++s)
            shift_complex_adjoint<RP, L>(B[0], B[1], B[2], B[3], q, kill, kill_r);

        // The pulse and, at the point before it, the relaxation's and the
        // turn's inner products.
        float e_flip = 0.f, e_rf = 0.f, e_dt = 0.f;
        const int rf = op_rf(code);
        if (rf == RF_INVERT) {
            const float2 f = dup(-eff);
            float2 acc = dup(0.f);
            acc = dot_acc<RP>(B[4], X[4], acc);
            acc = dot_acc<RP>(B[5], X[5], acc);
            g_inv -= acc.x + acc.y;
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                B[4][k] = mul2(B[4][k], f);
                B[5][k] = mul2(B[5][k], f);
            }
        }
        const bool rotate = rf == RF_ROTATE;
        float sa = 0.f, ca = 1.f;
        if (rotate) {
            sa = tv(mine.sa);
            ca = tv(mine.ca);
        }
        const float2 half = dup(0.5f), nhalf = dup(-0.5f), minus = dup(-1.f);
        float2 wz = dup(0.f), zw = dup(0.f), nwz = dup(0.f), nzw = dup(0.f);  // of dL/dalpha
        float2 pp = dup(0.f), pn = dup(0.f);                                  // of dL/dphi
        float2 q2 = dup(0.f), qp = dup(0.f), qn = dup(0.f), q1 = dup(0.f);
#pragma unroll
        for (int k = 0; k < RP; ++k) {
            const float2 ur = add2(X[0][k], X[2][k]), ui = add2(X[1][k], X[3][k]);
            const float2 wr = fma2(minus, X[2][k], X[0][k]), wi = fma2(minus, X[3][k], X[1][k]);
            const float2 zr = X[4][k], zi = X[5][k];
            const float2 tr2 = mul2(half, B[0][k]), ti2 = mul2(half, B[1][k]);
            const float2 Ur = fma2(half, B[2][k], tr2), Ui = fma2(half, B[3][k], ti2);
            float2 Wr = fma2(nhalf, B[2][k], tr2), Wi = fma2(nhalf, B[3][k], ti2);
            float2 Zr = B[4][k], Zi = B[5][k];
            if (rotate) {
                // Changes of w through the pulse, and of W back through it.
                const float2 co = dup(ca), less = dup(ca - 1.f), s2 = dup(2.f * sa),
                             ns2 = dup(-2.f * sa), hs = dup(0.5f * sa), nhs = dup(-0.5f * sa);
                const float2 dwr = fma2(s2, zi, mul2(less, wr)), dwi = fma2(ns2, zr, mul2(less, wi));
                const float2 dWr = fma2(nhs, Zi, mul2(less, Wr)), dWi = fma2(hs, Zr, mul2(less, Wi));
                Zr = fma2(ns2, Wi, mul2(co, Zr));
                Zi = fma2(s2, Wr, mul2(co, Zi));
                Wr = add2(Wr, dWr);
                Wi = add2(Wi, dWi);
                // (dWr, dWi run against the pulse.)
                pp = fma2(Ui, dwr, fma2(ui, dWr, pp));
                pn = fma2(Ur, dwi, fma2(ur, dWi, pn));
                wz = fma2(Wr, zi, wz);
                nwz = fma2(Wi, zr, nwz);
                zw = fma2(Zr, wi, zw);
                nzw = fma2(Zi, wr, nzw);
                B[4][k] = Zr;
                B[5][k] = Zi;
            }
            q2 = fma2(Ur, ur, fma2(Ui, ui, fma2(Wr, wr, fma2(Wi, wi, q2))));
            qp = fma2(Ui, wr, fma2(Wi, ur, qp));
            qn = fma2(Ur, wi, fma2(Wr, ui, qn));
            q1 = fma2(Zr, zr, fma2(Zi, zi, q1));
            B[0][k] = add2(Ur, Wr);
            B[1][k] = add2(Ui, Wi);
            B[2][k] = fma2(minus, Wr, Ur);
            B[3][k] = fma2(minus, Wi, Ui);
        }
        if (rotate) {
            const float gsa = 2.f * ((wz.x - nwz.x) + (wz.y - nwz.y)) +
                              0.5f * ((zw.x - nzw.x) + (zw.y - nzw.y));
            const float gsp = (pp.x - pn.x) + (pp.y - pn.y);
            e_flip = gsa * b1;
            g_b1 = fmaf(gsa, op.flip, g_b1);
            e_rf = gsp;
            g_b1p += gsp;
        }
        if (relax) {
            const float G2 = q2.x + q2.y, Go = (qp.x - qn.x) + (qp.y - qn.y);
            const float G1 = q1.x + q1.y - (q == 0 ? B[4][0].x : 0.f);
            g_t2 = fmaf(G2, op.dt * w2, g_t2);
            g_t1 = fmaf(G1, op.dt * w1, g_t1);
            g_b0 = fmaf(Go, -kTwoPi * op.dt, g_b0);
            e_dt = -r2 * G2 - r1 * G1 - kTwoPi * b0 * Go;
        }
        for (int s = 0; s < op_shift1(code); ++s)
            shift_complex_adjoint<RP, L>(B[0], B[1], B[2], B[3], q, kill, kill_r);
        if (turn) {
            // F+_bar *= conj(T), F-_bar *= T, Z_bar *= e1.
            const float2 Tr = dup(tr), Ti = dup(ti), nTi = dup(-ti), E1 = dup(e1);
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                const float2 pr = B[0][k], pi = B[1][k], mr = B[2][k], mi = B[3][k];
                B[0][k] = fma2(Ti, pi, mul2(Tr, pr));
                B[1][k] = fma2(nTi, pr, mul2(Tr, pi));
                B[2][k] = fma2(nTi, mi, mul2(Tr, mr));
                B[3][k] = fma2(Ti, mr, mul2(Tr, mi));
                B[4][k] = mul2(B[4][k], E1);
                B[5][k] = mul2(B[5][k], E1);
            }
        }
        // The op's event partials summed over the warp: two exchanges leave
        // each lane one of the four values, three more sum it (in a fixed
        // order).
        float f0 = active ? e_flip : 0.f, f1 = active ? e_dt : 0.f, f2 = active ? e_rf : 0.f,
              f3 = active ? e_rec : 0.f;
        const bool upper = lane & 16, odd = lane & 8;
        const float x0 = __shfl_xor_sync(0xffffffffu, upper ? f0 : f2, 16);
        const float x1 = __shfl_xor_sync(0xffffffffu, upper ? f1 : f3, 16);
        f0 = (upper ? f2 : f0) + x0;
        f1 = (upper ? f3 : f1) + x1;
        f0 = (odd ? f1 : f0) + __shfl_xor_sync(0xffffffffu, odd ? f0 : f1, 8);
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) f0 += __shfl_xor_sync(0xffffffffu, f0, off);
        if ((lane & 7) == 0)
            reinterpret_cast<float*>(event_out + int64_t(o) * 2)[lane >> 3] = f0;
    };
    for (int o = n_ops - 1; o >= 0; --o) {
        const Op op = s_ops[o];
        if (op.code == kPlainOp)
            step(std::true_type{}, o, op);
        else
            step(std::false_type{}, o, op);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    float out[7] = {g_t1, g_t2, g_m0, g_b1, g_inv, g_b1p, g_b0};
#pragma unroll
    for (int j = 0; j < 7; ++j) {
        const float x = active ? out[j] : 0.f;
        float sum = 0.f;
#pragma unroll
        for (int l = 0; l < L; ++l) sum += __shfl_sync(0xffffffffu, x, lane - q + l);
        out[j] = sum;
    }
    if (lane0) {
        float* dst = a.tissue_partial + row * 7;
#pragma unroll
        for (int j = 0; j < 7; ++j) dst[j] = out[j];
    }
}

// Sums the per-warp event partials (one block per op and train, a fixed
// tree) and scatters them: flip and duration to the op's RF and dt events,
// the pulse phase to its RF event, the receiver phase to its record event.
__global__ void __launch_bounds__(kEventReduceThreads)
    reduce_complex_events(const float2* partial, int64_t warps, int64_t n_ops, int64_t events,
                          const OpSource* src, float* g_flip, float* g_dt, float* g_phase) {
    __shared__ float4 s_sum[kEventReduceThreads];
    const int64_t op = blockIdx.x;
    const int64_t t = blockIdx.y;
    const float2* p = partial + (t * warps * n_ops + op) * 2;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int64_t w = threadIdx.x; w < warps; w += kEventReduceThreads) {
        const float2 x = p[w * n_ops * 2], y = p[w * n_ops * 2 + 1];
        acc.x += x.x;
        acc.y += x.y;
        acc.z += y.x;
        acc.w += y.y;
    }
    s_sum[threadIdx.x] = acc;
    __syncthreads();
    for (int half = kEventReduceThreads / 2; half > 0; half >>= 1) {
        if (threadIdx.x < half) {
            float4& d = s_sum[threadIdx.x];
            const float4 e = s_sum[threadIdx.x + half];
            d.x += e.x;
            d.y += e.y;
            d.z += e.z;
            d.w += e.w;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const float4 c = s_sum[0];
        const OpSource s = src[t * n_ops + op];
        if (s.rf_event >= 0) {
            if (g_flip) g_flip[t * events + s.rf_event] += c.x;
            if (g_phase) g_phase[t * events + s.rf_event] += c.z;
        }
        if (s.dt_event >= 0 && g_dt) g_dt[t * events + s.dt_event] += c.y;
        if (s.rec_event >= 0 && g_phase) g_phase[t * events + s.rec_event] += c.w;
    }
}

// The seven per-atom gradient slots (t1, t2, m0, b1, inversion, b1 phase,
// b0), passed by value.
struct TissueSlots7 {
    float* p[7];
};

// Per atom, the trains' tissue partials in train order, added into the
// gradients.
__global__ void reduce_complex_tissue(const float* partial, int64_t atoms, int64_t trains,
                                      TissueSlots7 out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= atoms) return;
    for (int j = 0; j < 7; ++j) {
        float sum = 0.f;
        for (int64_t t = 0; t < trains; ++t) sum += partial[(t * atoms + i) * 7 + j];
        if (out.p[j]) out.p[j][i] += sum;
    }
}

struct CxEntry {
    int orders_per_lane;
    int lanes_per_voxel;
    void (*forward)(const ComplexAdjointArgs&, dim3, dim3, cudaStream_t);
    // The reverse for trajectories of any (8-byte) alignment and of 16 bytes.
    void (*reverse[2])(const ComplexAdjointArgs&, dim3, dim3, size_t, cudaStream_t);
    const void* reverse_fn[2];
};

template <int RP, int L>
void launch_cx_forward(const ComplexAdjointArgs& a, dim3 g, dim3 b, cudaStream_t s) {
    complex_forward_traj_kernel<RP, L><<<g, b, 0, s>>>(a);
}
template <int RP, int L, bool WIDE>
void launch_cx_reverse(const ComplexAdjointArgs& a, dim3 g, dim3 b, size_t smem, cudaStream_t s) {
    complex_adjoint_kernel<RP, L, WIDE><<<g, b, smem, s>>>(a);
}

#define TSG_CX_ENTRY(R, L)                                                                       \
    {R, L, &launch_cx_forward<(R) / 2, L>,                                                       \
     {&launch_cx_reverse<(R) / 2, L, false>, &launch_cx_reverse<(R) / 2, L, (R) == 4>},          \
     {reinterpret_cast<const void*>(&complex_adjoint_kernel<(R) / 2, L, false>),                 \
      reinterpret_cast<const void*>(&complex_adjoint_kernel<(R) / 2, L, (R) == 4>)}}

const CxEntry kCx[] = {
    TSG_CX_ENTRY(2, 2),  TSG_CX_ENTRY(2, 4),  TSG_CX_ENTRY(2, 5),  TSG_CX_ENTRY(2, 8),
    TSG_CX_ENTRY(2, 10), TSG_CX_ENTRY(2, 16), TSG_CX_ENTRY(2, 32), TSG_CX_ENTRY(4, 1),
    TSG_CX_ENTRY(4, 2),  TSG_CX_ENTRY(4, 4),  TSG_CX_ENTRY(4, 5),  TSG_CX_ENTRY(4, 8),
    TSG_CX_ENTRY(4, 16),
};

struct CxPlan {
    const CxEntry* forward = nullptr;
    const CxEntry* reverse = nullptr;
    int64_t blocks = 0;  // of the reverse sweep
    int64_t warps_per_train = 0;
    int64_t state_bytes = 0;
    int64_t trajectory_bytes = 0;
    int64_t event_bytes = 0;
    int64_t workspace_bytes = 0;
    size_t smem = 0;
};

int cx_plan(const tsg_program* prog, int64_t atoms, int64_t states, const tsg_launch* want,
            CxPlan* plan) {
    if (!prog) return fail(TSG_ERR_ARGUMENT, "null program");
    if (atoms < 0 || states < 1) return fail(TSG_ERR_ARGUMENT, "invalid EPG buffer dimensions");
    if (states > 64) return fail(TSG_ERR_CAPACITY, "the complex adjoint takes at most 64 states");
    if (!prog->d_phase && prog->host.ops > 0)
        return fail(TSG_ERR_ARGUMENT, "the complex path needs a program built with event phases");
    const CxEntry* best = nullptr;
    for (const CxEntry& e : kCx) {
        if (want && want->lanes_per_voxel > 0 && e.lanes_per_voxel != want->lanes_per_voxel) continue;
        if (want && want->orders_per_lane > 0 && e.orders_per_lane != want->orders_per_lane) continue;
        if (e.lanes_per_voxel * e.orders_per_lane < states) continue;
        // Two orders per lane on the fewest lanes; four where two would need
        // more than 32 lanes.
        if (!best || e.orders_per_lane < best->orders_per_lane ||
            (e.orders_per_lane == best->orders_per_lane && e.lanes_per_voxel < best->lanes_per_voxel))
            best = &e;
    }
    if (!best) return fail(TSG_ERR_UNSUPPORTED, "no complex adjoint kernel for this state count / launch shape");
    plan->forward = plan->reverse = best;
    // The reverse sweep takes the same orders as four per lane: its work per
    // op besides the orders (the op's scalars, the event partials) halves. The
    // forward, a shorter chain that stores what it steps, does not. Measured at
    // 20 states x 601 ops, reverse on ten and on five lanes: 1.57 and 1.24 ms
    // at 16,384 voxels, 0.53 and 0.50 at 512; forward 0.91 and 0.99, 0.26 and
    // 0.36.
    if (!want || (want->lanes_per_voxel <= 0 && want->orders_per_lane <= 0))
        for (const CxEntry& e : kCx)
            if (best->orders_per_lane == 2 && e.orders_per_lane == 4 &&
                2 * e.lanes_per_voxel == best->lanes_per_voxel)
                plan->reverse = &e;
    best = plan->reverse;
    const int64_t ops = prog->host.ops, trains = prog->host.trains;
    const int vpb = kCxWarps * (32 / best->lanes_per_voxel);
    const int tile = 32 / plan->forward->lanes_per_voxel;
    plan->blocks = (atoms + vpb - 1) / vpb;
    plan->warps_per_train = plan->blocks * kCxWarps;
    plan->state_bytes = trains * ((atoms + tile - 1) / tile) * ops * 6 * 32 *
                        int64_t(plan->forward->orders_per_lane / 2) * 8;
    plan->trajectory_bytes =
        align256(plan->state_bytes) + trains * prog->host.outputs * atoms * int64_t(sizeof(float2));
    plan->event_bytes = align256(trains * plan->warps_per_train * ops * 2 * int64_t(sizeof(float2)));
    plan->workspace_bytes = plan->event_bytes + trains * atoms * 7 * int64_t(sizeof(float));
    plan->smem = size_t(kCxRing) * 6 * 32 * kCxWarps * size_t(best->orders_per_lane / 2) * 8 +
                 size_t(ops) * (sizeof(Op) + sizeof(float2));
    if (plan->smem > 226 * 1024)
        return fail(TSG_ERR_CAPACITY, "the program does not fit in shared memory for the reverse sweep");
    if (plan->blocks > 0x7fffffffLL || trains > 65535) return fail(TSG_ERR_CAPACITY, "launch too large");
    return TSG_OK;
}

ComplexAdjointArgs cx_args(const tsg_program* prog, const tsg_tissue* tissue,
                           const tsg_offaxis* off, int64_t atoms, int64_t states) {
    ComplexAdjointArgs a{};
    a.ops = prog->d_ops;
    a.phase = prog->d_phase;
    a.n_ops = int(prog->host.ops);
    a.atoms = atoms;
    a.states = int(states);
    a.outputs = int(prog->host.outputs);
    a.t1 = tissue->t1_ms;
    a.t2 = tissue->t2_ms;
    a.m0 = tissue->m0;
    a.b1 = tissue->b1;
    a.inv = tissue->inversion;
    a.b1_phase = off ? off->b1_phase_rad : nullptr;
    a.b0 = off ? off->b0_hz : nullptr;
    return a;
}

int cx_check(const tsg_program* prog, const tsg_tissue* tissue, int64_t atoms) {
    if (!prog) return fail(TSG_ERR_ARGUMENT, "null program");
    if (!tissue || (atoms > 0 && (!tissue->t1_ms || !tissue->t2_ms)))
        return fail(TSG_ERR_ARGUMENT, "t1 and t2 are required");
    return TSG_OK;
}

}  // namespace

}  // namespace tsg

using namespace tsg;

extern "C" int tsg_epg_complex_adjoint_plan(const tsg_program* program, int64_t atom_count,
                                            int64_t state_count, const tsg_launch* launch,
                                            int64_t* trajectory_bytes, int64_t* workspace_bytes) {
    CxPlan plan;
    int rc = cx_plan(program, atom_count, state_count, launch, &plan);
    if (rc) return rc;
    if (trajectory_bytes) *trajectory_bytes = plan.trajectory_bytes;
    if (workspace_bytes) *workspace_bytes = plan.workspace_bytes;
    return TSG_OK;
}

extern "C" int tsg_epg_forward_complex_trajectory(const tsg_program* program,
                                                  const tsg_tissue* tissue,
                                                  const tsg_offaxis* offaxis, int64_t atom_count,
                                                  int64_t state_count, int layout, float* out_a,
                                                  float* out_b, void* trajectory,
                                                  const tsg_launch* launch, void* stream) {
    int rc = cx_check(program, tissue, atom_count);
    if (rc) return rc;
    CxPlan plan;
    rc = cx_plan(program, atom_count, state_count, launch, &plan);
    if (rc) return rc;
    if (layout != TSG_LAYOUT_PLANES && layout != TSG_LAYOUT_COMPLEX_IJ && layout != TSG_LAYOUT_COMPLEX)
        return fail(TSG_ERR_ARGUMENT, "unknown output layout");
    if (layout == TSG_LAYOUT_PLANES && out_a && !out_b)
        return fail(TSG_ERR_ARGUMENT, "the planes layout writes both planes");
    if (atom_count == 0 || program->host.ops == 0) return TSG_OK;
    if (!trajectory) return fail(TSG_ERR_ARGUMENT, "null trajectory");
    ComplexAdjointArgs a = cx_args(program, tissue, offaxis, atom_count, state_count);
    a.layout = layout;
    a.out_a = out_a;
    a.out_b = out_b;
    a.traj = static_cast<float2*>(trajectory);
    a.traj_rec = reinterpret_cast<float2*>(static_cast<char*>(trajectory) + align256(plan.state_bytes));
    const int vpb = 4 * (32 / plan.forward->lanes_per_voxel);
    const int64_t blocks = (atom_count + vpb - 1) / vpb;
    if (blocks > 0x7fffffffLL) return fail(TSG_ERR_CAPACITY, "too many voxels for one launch");
    plan.forward->forward(a, dim3(unsigned(blocks), unsigned(program->host.trains)), dim3(128),
                        static_cast<cudaStream_t>(stream));
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

extern "C" int tsg_epg_adjoint_complex(const tsg_program* program, const tsg_tissue* tissue,
                                       const tsg_offaxis* offaxis, int64_t atom_count,
                                       int64_t state_count, const float* seed_a,
                                       const float* seed_b, int seed_layout,
                                       const void* trajectory, const tsg_gradients* gradients,
                                       const tsg_offaxis_gradients* offaxis_gradients,
                                       void* workspace, int64_t workspace_bytes,
                                       const tsg_launch* launch, void* stream) {
    int rc = cx_check(program, tissue, atom_count);
    if (rc) return rc;
    CxPlan plan;
    rc = cx_plan(program, atom_count, state_count, launch, &plan);
    if (rc) return rc;
    if (atom_count == 0 || program->host.ops == 0) return TSG_OK;
    if (!trajectory || !workspace || !seed_a) return fail(TSG_ERR_ARGUMENT, "null trajectory, workspace or seed");
    if (seed_layout != TSG_LAYOUT_PLANES && seed_layout != TSG_LAYOUT_COMPLEX)
        return fail(TSG_ERR_ARGUMENT, "the complex seed is planes or interleaved complex");
    if (seed_layout == TSG_LAYOUT_PLANES && !seed_b) return fail(TSG_ERR_ARGUMENT, "null seed plane");
    if (workspace_bytes < plan.workspace_bytes) return fail(TSG_ERR_ARGUMENT, "workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ComplexAdjointArgs a = cx_args(program, tissue, offaxis, atom_count, state_count);
    a.traj = const_cast<float2*>(static_cast<const float2*>(trajectory));
    a.traj_rec = reinterpret_cast<float2*>(const_cast<char*>(static_cast<const char*>(trajectory)) +
                                           align256(plan.state_bytes));
    a.tile_voxels = 32 / plan.forward->lanes_per_voxel;
    a.plane_pairs = 16 * plan.forward->orders_per_lane;
    a.seed_a = seed_a;
    a.seed_b = seed_b;
    a.seed_layout = seed_layout;
    char* ws = static_cast<char*>(workspace);
    a.event_partial = reinterpret_cast<float2*>(ws);
    a.tissue_partial = reinterpret_cast<float*>(ws + plan.event_bytes);
    a.warps_per_train = plan.warps_per_train;
    const int wide = (reinterpret_cast<uintptr_t>(trajectory) & 15) == 0;
    if (plan.smem > 48 * 1024)
        TSG_CUDA(cudaFuncSetAttribute(plan.reverse->reverse_fn[wide],
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, int(plan.smem)));
    plan.reverse->reverse[wide](a, dim3(unsigned(plan.blocks), unsigned(program->host.trains)),
                        dim3(32 * kCxWarps), plan.smem, s);
    TSG_CUDA(cudaGetLastError());
    const int64_t ops = program->host.ops;
    float* g_phase = offaxis_gradients ? offaxis_gradients->phase_rad : nullptr;
    reduce_complex_events<<<dim3(unsigned(ops), unsigned(program->host.trains)),
                            kEventReduceThreads, 0, s>>>(
        a.event_partial, plan.warps_per_train, ops, program->host.events, program->d_src,
        gradients ? gradients->flip_rad : nullptr, gradients ? gradients->duration_s : nullptr,
        g_phase);
    TSG_CUDA(cudaGetLastError());
    TissueSlots7 slots{};
    if (gradients) {
        slots.p[0] = gradients->t1_ms;
        slots.p[1] = gradients->t2_ms;
        slots.p[2] = gradients->m0;
        slots.p[3] = gradients->b1;
        slots.p[4] = gradients->inversion;
    }
    if (offaxis_gradients) {
        slots.p[5] = offaxis_gradients->b1_phase_rad;
        slots.p[6] = offaxis_gradients->b0_hz;
    }
    reduce_complex_tissue<<<unsigned((atom_count + 127) / 128), 128, 0, s>>>(
        a.tissue_partial, atom_count, program->host.trains, slots);
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}
