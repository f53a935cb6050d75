// The sweep of a plain recorded train: after at most one leading inversion
// every op is relax, rotate, record, one shift (an MRF repetition; the first may
// have nothing to relax), and op i records sample i. Every event stream of the MRF builder with one playing
// compiles to this; other programs run epg_sweep.cuh.
//
// Thread mapping and state layout are the general sweep's (one voxel's orders
// over L lanes, 2 RP orders per lane as strided float2 pairs). What differs:
//
// * No op decoding: the loop body is the op.
// * Coefficients by the voxel's lanes: lane q of a voxel evaluates the
//   sin/cos/exp and the products of one op in every group of G ops and leaves
//   them, each already duplicated into a pair, in shared memory one group
//   ahead of use, so the transcendentals are off the recursion's dependency
//   chain, cost one evaluation per voxel and op instead of one per lane, and
//   a step loads its coefficients as ready operands.
// * Relaxation folded into the rotation everywhere, the recovery of order 0
//   through the addend of a product that is there anyway, and eight paired
//   instructions per order pair instead of nine: F- is held negated (n = -m),
//   so that with s = p - n, d = p + n and B = E2 cos d / 2 - E1 sin z the
//   rotated state is p' = E2 s / 2 + B, n' = -E2 s / 2 + B,
//   z' = E2 sin d / 2 + E1 cos z.
// * Records go to shared memory and leave for HBM about 32 samples of one row
//   at a time, a whole contiguous run per store instruction (one sample per
//   op and lane writes an 8-byte piece of a 32-byte sector each time).
//
// Bound: with many voxels the FMA pipe and its register ports (ncu, T1/T2/B1
// at 20 states: FMA pipe 61% active, issue 63%, math-pipe throttle and fixed
// latencies the leading stalls; more warps per SM measured no faster); with
// few, one op's chain of paired FMAs and two shuffles. Measured against the
// general sweep on the same trains: signal of 1,024 voxels x 880 pulses x 10
// states 321 -> 61 us, with T1 and T2 568 -> 94 us; 100,000 x 500 x 32 signal
// 1,256 -> 705 us (41 TFLOP/s of 18 per order and pulse), with T1 and T2
// 2,166 -> 1,757 us; 262,144 x 880 x 20 with T1, T2 and B1 10.12 -> 7.99 ms
// (83 TFLOP/s of 144 per order and pulse, above the pipe's 78 because the
// folded step needs fewer); Gauss-Newton sums of 16,384 x 880 x 10
// 606 -> 330 us.
//
// Each order's arithmetic is the same sequence of roundings at every (L, RP),
// so a voxel's samples do not depend on the launch shape.
#pragma once

#include "epg_sweep.cuh"

namespace tsg {

constexpr int kTrainChunk = 960;  // ops staged at a time: a multiple of every group and record run

__host__ __device__ constexpr int train_group(int L) { return L == 1 ? 1 : (L <= 10 ? L : 8); }
__host__ __device__ constexpr int train_records(int L) {
    return train_group(L) * (32 / train_group(L));
}
// float4s of one op's coefficients (odd, so voxels spread over the banks).
__host__ __device__ constexpr int train_coefs(int TM) { return TM == 0 ? 3 : 5; }

// Dynamic shared memory of a block of `warps` warps: the staged ops, then per
// warp the double-buffered coefficients and the records, then the GN sums.
template <int L, int TM, bool GN>
constexpr size_t train_smem(int warps) {
    constexpr int NT = SystemLayout<TM, false>::N;
    constexpr int VPW = 32 / L;
    const size_t coefs = L == 1 ? 0 : size_t(2) * train_group(L) * VPW * train_coefs(TM) * 16;
    const size_t recs = size_t(VPW + 1) * (NT + 1) * (train_records(L) + 1) * 4;
    return kTrainChunk * 8 + warps * (coefs + (recs + 15) / 16 * 16) + (GN ? size_t(warps) * 32 * 80 : 0);
}

// One op's coefficients as pairs, and the order-0 addends.
struct TrainCoef {
    float2 h, nh, hco, nsi, hsi, ce;  // E2/2, -E2/2, E2 cos/2, -E1 sin, E2 sin/2, E1 cos
    float nb, zb;                 // -sin (1 - E1), cos (1 - E1)
    float2 g1, g2;                // dt 1000 / T1^2, dt 1000 / T2^2
    float2 at, nat;               // flip, -flip
};

template <int RP, int L, int TM, bool KILL, bool GN, int MINB>
__global__ void __launch_bounds__(128, MINB) epg_train_kernel(const SweepArgs a) {
    using S = SystemLayout<TM, false>;
    constexpr int NT = S::N;
    constexpr int NC = NT + 1;
    constexpr int R = 2 * RP;
    constexpr int VPW = 32 / L;
    constexpr int G = train_group(L);
    constexpr int KB = train_records(L);
    constexpr int Q = train_coefs(TM);
    extern __shared__ __align__(16) unsigned char s_raw[];

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int q = lane % L;
    const int slot = lane / L;
    const bool holds = slot < VPW;  // lanes past the last whole voxel idle
    const int vslot = holds ? slot : 0;
    const int64_t warp_atom = (int64_t(blockIdx.x) * (blockDim.x >> 5) + warp) * VPW;
    const int64_t train = blockIdx.y;
    int64_t atom = warp_atom + slot;
    bool active = holds && atom < a.atoms;
    if constexpr (GN) {
        if (a.voxel_list != nullptr) {
            const int n = *a.voxel_list_count;
            if (int64_t(blockIdx.x) * (blockDim.x >> 5) * VPW >= n) return;
            active = holds && atom < n;
            atom = a.voxel_list[active ? atom : 0];
        }
    }
    const int64_t ac = active ? atom : 0;

    float2* s_ops = reinterpret_cast<float2*>(s_raw);  // (dt, flip)
    constexpr size_t kCoefBytes = L == 1 ? 0 : size_t(2) * G * VPW * Q * 16;
    constexpr size_t kRecBytes = (size_t(VPW + 1) * NC * (KB + 1) * 4 + 15) / 16 * 16;
    unsigned char* s_warp = s_raw + kTrainChunk * 8 + size_t(warp) * (kCoefBytes + kRecBytes);
    float4* s_coef = reinterpret_cast<float4*>(s_warp);
    float* s_rec = reinterpret_cast<float*>(s_warp + kCoefBytes);
    // GN only: sum k of this thread at cd[k * blockDim.x].
    double* cd = reinterpret_cast<double*>(s_raw + kTrainChunk * 8 +
                                           size_t(blockDim.x >> 5) * (kCoefBytes + kRecBytes)) +
                 threadIdx.x;

    const float t1 = a.t1[ac];
    const float t2 = a.t2[ac];
    const float m0 = a.m0 ? a.m0[ac] : 1.f;
    const float b1 = a.b1 ? a.b1[ac] : 1.f;
    const float nr1 = -(1000.f / t1);
    const float nr2 = -(1000.f / t2);
    const float w1 = 1000.f / (t1 * t1);
    const float w2 = 1000.f / (t2 * t2);
    const float first = q == 0 ? 1.f : 0.f;  // this lane holds order 0
    // The pair whose .x or .y is order `states`, where this lane holds it.
    const int kill_r = KILL ? a.states - q * R : -1;
    const int kill_x = kill_r >= 0 && kill_r < RP ? kill_r : -1;
    const int kill_y = kill_r >= RP && kill_r < R ? kill_r - RP : -1;
    const float2 neg1 = dup(-1.f);

    float2 P[RP], N[RP], Z[RP];  // F+, -F-, Z
    float2 dP[S::NA][RP], dN[S::NA][RP], dZ[S::NA][RP];
#pragma unroll
    for (int k = 0; k < RP; ++k) {
        P[k] = N[k] = Z[k] = dup(0.f);
#pragma unroll
        for (int j = 0; j < S::NA; ++j) dP[j][k] = dN[j][k] = dZ[j][k] = dup(0.f);
    }
    // The leading inversion on the equilibrium state: Z -> -eff Z.
    const int begin = a.train_first;
    if (q == 0) {
        Z[0].x = begin ? -(a.inv ? a.inv[ac] : 1.f) : 1.f;
        if constexpr (S::INV) dZ[S::I_INV][0].x = begin ? -1.f : 0.f;
    }

    float cs[10];
    int flushes = 0;
    const float2* yrow = nullptr;
    if constexpr (GN) {
#pragma unroll
        for (int k = 0; k < 10; ++k) {
            cs[k] = 0.f;
            cd[k * blockDim.x] = 0.0;
        }
        const int64_t mrow = a.measured_rows ? a.measured_rows[ac] : (train * a.atoms + ac);
        yrow = a.measured + mrow * a.outputs;
    }

    // The coefficients of one op for this lane's voxel, as scalars. `still`: an
    // op that does not wait (a train's first, find_train) leaves the state alone
    // whatever the relaxation times; the product of its interval with the rate
    // of a time of zero would be NaN.
    struct Raw {
        float h, hco, nsi, hsi, ce, nb, zb, g1, g2, at;
    };
    auto evaluate = [&](const float2 op, bool still) {
        const float n1 = still ? 0.f : nr1, n2 = still ? 0.f : nr2;
        const float d1 = still ? 0.f : w1, d2 = still ? 0.f : w2;
        float si, co;
        sincosf(__fmul_rn(op.y, b1), &si, &co);
        const float e1 = expf(__fmul_rn(n1, op.x)), e2 = expf(__fmul_rn(n2, op.x));
        const float h = 0.5f * e2, rec = 1.f - e1;
        return Raw{h, __fmul_rn(h, co), -__fmul_rn(e1, si), __fmul_rn(h, si), __fmul_rn(e1, co),
                   -__fmul_rn(si, rec), __fmul_rn(co, rec), __fmul_rn(op.x, d1),
                   __fmul_rn(op.x, d2), op.y};
    };
    // Lane q takes op base + q of a group and leaves its coefficients in
    // buffer `buf`. `start`: op 0 of the group is the train's first. Without a
    // B1 column the look at the first op alone costs nothing, at every op 1 to
    // 2% (100,000 voxels x 500 x 32: 703 and 711 us); with one the compiler's
    // schedule makes it the other way round (100,000 x 500 x 20: every op 1,786
    // us, the first 1,847, none 1,781).
    auto prepare = [&](int base, int count, int buf, bool start) {
        const int j = base + q;
        if (holds && q < G && j < count) {
            const Raw c = evaluate(s_ops[j], (S::B1 || (start && q == 0)) && s_ops[j].x == 0.f);
            float4* dst = s_coef + ((buf * G + q) * VPW + slot) * Q;
            dst[0] = make_float4(c.h, c.h, c.hco, c.hco);
            dst[1] = make_float4(c.nsi, c.nsi, c.hsi, c.hsi);
            dst[2] = make_float4(c.ce, c.ce, c.nb, c.zb);
            if constexpr (S::T1 || S::T2) dst[3] = make_float4(c.g1, c.g1, c.g2, c.g2);
            if constexpr (S::B1) dst[4] = make_float4(c.at, c.at, -c.at, -c.at);
        }
    };
    auto load = [&](int buf, int g) {
        const float4* src = s_coef + ((buf * G + g) * VPW + vslot) * Q;
        TrainCoef c;
        const float4 x0 = src[0], x1 = src[1], x2 = src[2];
        c.h = make_float2(x0.x, x0.y);
        c.nh = make_float2(-x0.x, -x0.x);
        c.hco = make_float2(x0.z, x0.w);
        c.nsi = make_float2(x1.x, x1.y);
        c.hsi = make_float2(x1.z, x1.w);
        c.ce = make_float2(x2.x, x2.y);
        c.nb = x2.z;
        c.zb = x2.w;
        if constexpr (S::T1 || S::T2) {
            const float4 x3 = src[3];
            c.g1 = make_float2(x3.x, x3.y);
            c.g2 = make_float2(x3.z, x3.w);
        }
        if constexpr (S::B1) {
            const float4 x4 = src[4];
            c.at = make_float2(x4.x, x4.y);
            c.nat = make_float2(x4.z, x4.w);
        }
        return c;
    };

    // One gradient shift of a plane pair: F- moves one order down (zero
    // enters at the voxel's top), F+ one up with F+[0] = -F-[0], the order
    // `states` is cleared.
    auto shift_one = [&](float2 (&p)[RP], float2 (&n)[RP]) {
        float in_p = 0.f, top = 0.f;
        if constexpr (L > 1) {
            in_p = __shfl_up_sync(0xffffffffu, p[RP - 1].y, 1);
            const float in_n = __shfl_down_sync(0xffffffffu, n[0].x, 1);
            top = q == L - 1 ? 0.f : in_n;
        }
        const float n_edge = n[0].y;
#pragma unroll
        for (int k = 0; k + 1 < RP; ++k) n[k] = n[k + 1];
        n[RP - 1] = make_float2(n_edge, top);
        const float bottom = L == 1 || q == 0 ? n[0].x : in_p;
        const float p_edge = p[RP - 1].x;
#pragma unroll
        for (int k = RP - 1; k > 0; --k) p[k] = p[k - 1];
        p[0] = make_float2(bottom, p_edge);
        if constexpr (KILL) {
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                p[k].x = k == kill_x ? 0.f : p[k].x;
                p[k].y = k == kill_y ? 0.f : p[k].y;
            }
        }
    };

    // One op: the pulse on the relaxed state, the record, the shift. `sample`
    // is the op's place in the record buffer.
    // Lanes that do not hold an order 0 write to a spare row, so the store
    // needs no branch.
    float* rec_dst = s_rec + (q == 0 && holds ? slot : VPW) * NC * (KB + 1);
    auto step = [&](const TrainCoef& c, int sample) {
        const float2 bias_b = make_float2(__fmul_rn(first, c.nb), 0.f);
        const float2 bias_z = make_float2(__fmul_rn(first, c.zb), 0.f);
        // Stage by stage over every system and pair, so that consecutive
        // instructions share their coefficient operand.
        constexpr int NS = NT + 1;
        auto X = [&](float2 (&sig)[RP], float2 (&tan)[S::NA][RP], int j) -> float2 (&)[RP] {
            return j == 0 ? sig : tan[j - 1];
        };
        float2 B[NS][RP];
        if constexpr (S::T2) {
#pragma unroll
            for (int k = 0; k < RP; ++k) dP[S::I_T2][k] = fma2(c.g2, P[k], dP[S::I_T2][k]);
#pragma unroll
            for (int k = 0; k < RP; ++k) dN[S::I_T2][k] = fma2(c.g2, N[k], dN[S::I_T2][k]);
        }
        if constexpr (S::T1) {
            // dE1/dT1 = E1 g1 acts on z - 1 at order 0 (the recovery).
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                const float2 zt = k == 0 ? make_float2(__fadd_rn(Z[0].x, -first), Z[0].y) : Z[k];
                dZ[S::I_T1][k] = fma2(c.g1, zt, dZ[S::I_T1][k]);
            }
        }
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                float2 &p = X(P, dP, j)[k], &n = X(N, dN, j)[k];
                // A paired FMA on three distinct operands takes three cycles of
                // the register ports, two scalar subtractions two; the extra
                // issue slot is free where a lane holds few pairs.
                const float2 sum = RP <= 2 ? make_float2(__fadd_rn(p.x, -n.x), __fadd_rn(p.y, -n.y))
                                           : fma2(neg1, n, p);
                n = add2(p, n);
                p = sum;
            }
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
            for (int k = 0; k < RP; ++k)
                B[j][k] = j == 0 && k == 0 ? fma2(c.nsi, Z[0], bias_b) : mul2(c.nsi, X(Z, dZ, j)[k]);
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
            for (int k = 0; k < RP; ++k) B[j][k] = fma2(c.hco, X(N, dN, j)[k], B[j][k]);
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                float2& z = X(Z, dZ, j)[k];
                z = j == 0 && k == 0 ? fma2(c.ce, z, bias_z) : mul2(c.ce, z);
            }
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                float2& z = X(Z, dZ, j)[k];
                z = fma2(c.hsi, X(N, dN, j)[k], z);
            }
        if constexpr (S::B1) {
            // d/dalpha of the pulse: (-Z', Z', B) of the signal.
#pragma unroll
            for (int k = 0; k < RP; ++k) B[1 + S::I_B1][k] = fma2(c.nat, Z[k], B[1 + S::I_B1][k]);
#pragma unroll
            for (int k = 0; k < RP; ++k) dZ[S::I_B1][k] = fma2(c.at, B[0][k], dZ[S::I_B1][k]);
        }
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
            for (int k = 0; k < RP; ++k) {
                float2 &p = X(P, dP, j)[k], &n = X(N, dN, j)[k];
                n = fma2(c.nh, p, B[j][k]);
                p = fma2(c.h, p, B[j][k]);
            }
        rec_dst[sample] = P[0].x;
#pragma unroll
        for (int j = 0; j < NT; ++j) rec_dst[(1 + j) * (KB + 1) + sample] = dP[j][0].x;
        shift_one(P, N);
#pragma unroll
        for (int j = 0; j < NT; ++j) shift_one(dP[j], dN[j]);
    };

    // `n` buffered samples of every row of the warp, from sample `sample0` on.
    auto flush = [&](int sample0, int n) {
        if constexpr (GN) {
            // The voxel's L lanes take its samples in turn: API signal s = -v
            // (v = m0 F+[0]), r = s - y; columns of dv are T1, T2 and F+[0].
            constexpr int kPer = (KB + L - 1) / L;
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const int s = i * L + q;
                if (active && s < n) {
                    const float2 y = yrow[sample0 + s];
                    const float* src = s_rec + vslot * NC * (KB + 1) + s;
                    const float p0 = src[0];
                    const float res = __fmaf_rn(m0, p0, y.x);  // -(r.real)
                    const float j1 = m0 * src[(1 + S::I_T1) * (KB + 1)];
                    const float j2 = m0 * src[(1 + S::I_T2) * (KB + 1)];
                    const float j3 = p0;
                    cs[0] = fmaf(res, res, fmaf(y.y, y.y, cs[0]));
                    cs[1] = fmaf(j1, j1, cs[1]);
                    cs[2] = fmaf(j1, j2, cs[2]);
                    cs[3] = fmaf(j1, j3, cs[3]);
                    cs[4] = fmaf(j2, j2, cs[4]);
                    cs[5] = fmaf(j2, j3, cs[5]);
                    cs[6] = fmaf(j3, j3, cs[6]);
                    cs[7] = fmaf(j1, res, cs[7]);
                    cs[8] = fmaf(j2, res, cs[8]);
                    cs[9] = fmaf(j3, res, cs[9]);
                }
            }
            // Into the doubles after at most 32 samples a lane.
            if (++flushes == L) {
                flushes = 0;
#pragma unroll
                for (int k = 0; k < 10; ++k) {
                    cd[k * blockDim.x] += double(cs[k]);
                    cs[k] = 0.f;
                }
            }
        } else {
            const int64_t row0 = train * a.atoms + warp_atom;
            const int rows = int(min(int64_t(VPW), a.atoms - warp_atom));
            const bool mine = lane < n;
            const bool planes = a.layout == TSG_LAYOUT_PLANES;
            const bool imag = a.layout == TSG_LAYOUT_COMPLEX;
            const bool signal = planes ? a.sig_b != nullptr : a.sig_a != nullptr;
            // Element offsets of this lane's sample: in the signal row and in
            // the voxel's block of columns.
            int64_t at = row0 * a.outputs + sample0 + lane;
            int64_t jat = row0 * a.jac_cols * a.outputs + sample0 + lane;
            const int64_t jstep = int64_t(a.jac_cols) * a.outputs;
            const float* src = s_rec + lane;
            auto write = [&](float* pa, float* pb, int64_t i, float v) {
                if (planes)
                    put_sample(TSG_LAYOUT_PLANES, pa, pb, i, v);
                else
                    __stcs(reinterpret_cast<float2*>(pa) + i,
                           make_float2(imag ? 0.f : -v, imag ? v : 0.f));
            };
            for (int v = 0; v < rows; ++v) {
                const float vm0 = __shfl_sync(0xffffffffu, m0, v * L);
                if (mine) {
                    const float p0 = src[0];
                    if (signal) write(a.sig_a, a.sig_b, at, vm0 * p0);
                    if (a.col_m0 >= 0) write(a.jac_a, a.jac_b, jat + a.col_m0 * a.outputs, p0);
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        int col = -1;
                        if (S::T1 && j == S::I_T1) col = a.col_t1;
                        if (S::T2 && j == S::I_T2) col = a.col_t2;
                        if (S::B1 && j == S::I_B1) col = a.col_b1;
                        if (S::INV && j == S::I_INV) col = a.col_inv;
                        if (col >= 0)
                            write(a.jac_a, a.jac_b, jat + col * a.outputs,
                                  vm0 * src[(1 + j) * (KB + 1)]);
                    }
                }
                at += a.outputs;
                jat += jstep;
                src += NC * (KB + 1);
            }
        }
    };

    const Op* ops = a.ops + train * a.n_ops + begin;
    const int n_ops = a.n_ops - begin;
    for (int base = 0; base < n_ops; base += kTrainChunk) {
        const int count = min(kTrainChunk, n_ops - base);
        __syncthreads();
        for (int i = threadIdx.x; i < count; i += blockDim.x) {
            const Op op = ops[base + i];
            s_ops[i] = make_float2((op.code & OP_RELAX) ? op.dt : 0.f, op.flip);
        }
        __syncthreads();
        int held = 0;  // buffered samples
        if constexpr (L == 1) {
            auto widen = [](const Raw& r) {
                return TrainCoef{dup(r.h), dup(-r.h), dup(r.hco), dup(r.nsi), dup(r.hsi), dup(r.ce), r.nb, r.zb,
                                 dup(r.g1), dup(r.g2),  dup(r.at),  dup(-r.at)};
            };
            Raw next = evaluate(s_ops[0], base == 0 && s_ops[0].x == 0.f);
#pragma unroll 1
            for (int i = 0; i < count; ++i) {
                const Raw now = next;
                next = evaluate(s_ops[min(i + 1, count - 1)], false);
                step(widen(now), held);
                if (++held == KB || i + 1 == count) {
                    __syncwarp();
                    flush(base + i + 1 - held, held);
                    __syncwarp();
                    held = 0;
                }
            }
        } else {
            prepare(0, count, 0, base == 0);
            __syncwarp();
            int buf = 0;
#pragma unroll 1
            for (int i = 0; i < count; i += G, buf ^= 1) {
                if (i + G < count) prepare(i + G, count, buf ^ 1, false);
                const int here = min(G, count - i);
                if (here == G) {
                    TrainCoef c = load(buf, 0);
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        TrainCoef n = c;
                        if (g + 1 < G) n = load(buf, g + 1);
                        step(c, held + g);
                        c = n;
                    }
                } else {
#pragma unroll 1
                    for (int g = 0; g < here; ++g) step(load(buf, g), held + g);
                }
                held += here;
                __syncwarp();
                if (held == KB || i + G >= count) {
                    flush(base + i + here - held, held);
                    __syncwarp();
                    held = 0;
                }
            }
        }
    }
    if constexpr (GN) {
        const int64_t row = train * a.atoms + atom;
        double* dst = a.gn_out + row * 10;
#pragma unroll 1
        for (int k = 0; k < 10; ++k) {
            const double mine = cd[k * blockDim.x] + double(cs[k]);
            double total = mine;
#pragma unroll 1
            for (int l = 1; l < L; ++l) {
                const double other = __shfl_down_sync(0xffffffffu, mine, l);
                total += other;  // used on the voxel's first lane only
            }
            if (q == 0 && active) dst[k] = total;
        }
    }
}

template <int RP, int L, int TM, bool GN, int MINB>
void launch_train(const SweepArgs& a, dim3 grid, dim3 block, size_t, cudaStream_t stream) {
    const size_t smem = train_smem<L, TM, GN>(int(block.x) / 32);
    const bool kill = 2 * RP * L > a.states;
    auto kernel = kill ? &epg_train_kernel<RP, L, TM, true, GN, MINB>
                       : &epg_train_kernel<RP, L, TM, false, GN, MINB>;
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    kernel<<<grid, block, smem, stream>>>(a);
}

}  // namespace tsg

// Entries take orders per lane R (even) and lanes per voxel L.
#define TSG_TRAIN_ENTRY(MODE, R, L, TM, MINB) \
    {MODE, R, L, &::tsg::launch_train<(R) / 2, L, TM, false, MINB>, 0}
#define TSG_TRAIN_GN_ENTRY(R, L, MINB) \
    {::tsg::MODE_GN, R, L, &::tsg::launch_train<(R) / 2, L, 3, true, MINB>, 0}
