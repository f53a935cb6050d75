// CPMG trains off the real subspace: refocusing pulses of one phase, 90
// degrees from the excitation's (FSESimulator's default), signal and T1 / T2 /
// B1 columns.
//
// In the frame of the refocusing pulses such a train splits. The excitation
// leaves F real; the pulses keep F real and Z imaginary, and take the
// recovered magnetisation (Z real, from order 0) through F imaginary and Z
// real. Both shifts of an echo interval together move by two orders, so what
// the excitation made stays on odd orders before every pulse and meets order
// 0 at the echoes, and what recovers stays on even orders and never does. So
// the recorded samples need one real number per odd order, F+ (P), -F- (N)
// and i Z (Z) below, where the complex sweep (epg_complex.cu) carries six per
// order: a quarter of its state and an eighth of its products.
//
// Odd order 2 m + 1 is slot m. A pulse with the relaxation folded in, and the
// two shifts after it:
//   s = P - N, d = P + N, B = E2/2 cos a d - E1 sin a Z
//   P[m + 1] = E2/2 s + B,  N[m - 1] = -E2/2 s + B,  P[0] = -N'[0]
//   Z[m] = E2/2 sin a d + E1 cos a Z
// and the echo is -N'[0] e2. A T1 or T2 column is the same step on (dP, dN,
// dZ) after dZ += r1' Z or (ds, dd) += r2' (s, d); a B1 column needs two more
// products, since the step's derivative in a takes B to -Z' and Z' to B.
// Slots above min(states, echoes + 1) / 2 either are cut off by the state
// limit or cannot come back to an echo.
//
// Layout: a voxel's slots over L lanes, 2 RP per lane as pairs (r, RP + r):
// a shift renames whole pairs and moves one value per array between lanes.
// The L lanes share the pulses' sincosf. Samples go to shared memory and leave
// 16 echoes at a time.
//
// Bound: the latency of an echo's chain at three warps a scheduler (0.51
// issued a cycle; 55% of the instructions are the paired products). Measured at
// 65,536 voxels x 48 echoes x 32 states, signal with T1 and T2 columns:
// 104 us (the complex sweep: 1,220 us); at 8,192 voxels 33 us.
#include "epg_complex.cuh"

#include <cmath>

namespace tsg {
namespace {

using namespace complex_detail;

constexpr int kCpmgChunk = 256;   // echoes staged in shared memory
constexpr int kCpmgEchoes = 16;   // samples held per voxel and array
constexpr int kCpmgWarps = 4;

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    return make_float2(__fadd_rn(a.x, -b.x), __fadd_rn(a.y, -b.y));
}

// Both shifts of an echo interval: P a slot up, N a slot down, P[0] = -N[0].
template <int RP, int L>
__device__ __forceinline__ void shift_slots(float2 (&P)[RP], float2 (&N)[RP], int q, int kill_r) {
    const float first = N[0].x;
    float below = P[RP - 1].y, above = 0.f;
    if constexpr (L > 1) {
        below = __shfl_up_sync(0xffffffffu, below, 1);
        above = __shfl_down_sync(0xffffffffu, first, 1);
        if (q == L - 1) above = 0.f;
    }
    const float top = P[RP - 1].x;
#pragma unroll
    for (int r = RP - 1; r > 0; --r) P[r] = P[r - 1];
    P[0] = make_float2(L == 1 || q == 0 ? -first : below, top);
    const float next = N[0].y;
#pragma unroll
    for (int r = 0; r + 1 < RP; ++r) N[r] = N[r + 1];
    N[RP - 1] = make_float2(next, above);
    if (kill_r < 2 * RP) {
#pragma unroll
        for (int r = 0; r < RP; ++r) {
            if (r == kill_r) P[r].x = 0.f;
            if (RP + r == kill_r) P[r].y = 0.f;
        }
    }
}

template <int RP, int L, int TM>
__global__ void __launch_bounds__(32 * kCpmgWarps) epg_cpmg_kernel(const ComplexArgs a) {
    constexpr bool T1 = (TM & 1) != 0, T2 = (TM & 2) != 0, B1 = (TM & 4) != 0;
    constexpr int NS = 1 + T1 + T2 + B1;
    constexpr int I1 = 1, I2 = 1 + T1, IB = 1 + T1 + T2;
    constexpr int VPW = 32 / L;
    constexpr int ROW = kCpmgEchoes + 1;
    // Per echo: flip, the interval before its pulse, the one before its sample.
    __shared__ float4 s_echo[kCpmgChunk];
    __shared__ float s_rec[kCpmgWarps][NS * VPW * ROW];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int q = lane % L;
    const int slot = lane / L;
    const int64_t first_atom = (int64_t(blockIdx.x) * kCpmgWarps + warp) * VPW;
    const int rows = int(max(int64_t(0), min(int64_t(VPW), a.atoms - first_atom)));
    const int64_t train = blockIdx.y;
    const int64_t atom = slot < rows ? first_atom + slot : 0;
    const float t1 = a.t1[atom], t2 = a.t2[atom];
    const float r1 = 1000.f / t1, r2 = 1000.f / t2;
    const float w1 = 1000.f / (t1 * t1), w2 = 1000.f / (t2 * t2);
    const float m0 = a.m0 ? a.m0[atom] : 1.f;
    const float b1 = a.b1 ? a.b1[atom] : 1.f;
    const int slots = a.states >> 1;  // odd orders below the state limit
    const int kill_r = L * 2 * RP > slots ? slots - q * 2 * RP : 2 * RP;
    const Op* ops = a.ops + train * a.n_ops;
    const float2* phase = a.phase + train * a.n_ops;
    const int echoes = a.n_ops >> 1;
    float* rec = s_rec[warp];

    float2 P[NS][RP], N[NS][RP], Z[NS][RP];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int r = 0; r < RP; ++r) P[s][r] = N[s][r] = Z[s][r] = dup(0.f);
    const float turn = phase[1].x;  // the frame's
    {
        // The excitation of the equilibrium, then the first shift.
        const float flip = ops[0].flip;
        const float side = sinf(phase[0].x - turn);
        float si, co;
        sincosf(flip * b1, &si, &co);
        if (q == 0) {
            P[0][0].x = side * si;
            if constexpr (B1) P[IB][0].x = side * (flip * co);
        }
    }
    float last_dt = __int_as_float(0x7fffffff), last_rec = last_dt;
    float e1 = 1.f, h = 0.5f, k1 = 0.f, k2 = 0.f, e2_rec = 1.f, k2_rec = 0.f;
    float my_si = 0.f, my_co = 1.f;
    int held = 0;
    for (int base = 0; base < echoes; base += kCpmgChunk) {
        const int count = min(kCpmgChunk, echoes - base);
        __syncthreads();
        for (int i = threadIdx.x; i < count; i += blockDim.x) {
            const int e = base + i;
            const Op pulse = ops[2 * e + 1];
            // What passes between pulses: this op's interval and the one of
            // the sample before it.
            const float before = e > 0 ? ops[2 * e].dt : 0.f;
            s_echo[i] = make_float4(pulse.flip, before + pulse.dt, ops[2 * e + 2].dt, 0.f);
        }
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < count; ++i) {
            const float4 echo = s_echo[i];
            float si, co;
            if constexpr (L > 1) {
                const int g = i % L;
                if (g == 0) sincosf(s_echo[min(i + q, count - 1)].x * b1, &my_si, &my_co);
                si = __shfl_sync(0xffffffffu, my_si, lane - q + g);
                co = __shfl_sync(0xffffffffu, my_co, lane - q + g);
            } else {
                sincosf(echo.x * b1, &si, &co);
            }
            if (echo.y != last_dt) {
                last_dt = echo.y;
                e1 = expf(-r1 * last_dt);
                h = 0.5f * expf(-r2 * last_dt);
                k1 = last_dt * w1;
                k2 = last_dt * w2;
            }
            if (echo.z != last_rec) {
                last_rec = echo.z;
                e2_rec = expf(-r2 * last_rec);
                k2_rec = last_rec * w2;
            }
            const float2 H = dup(h), nH = dup(-h), hco = dup(h * co), hsi = dup(h * si);
            const float2 nsi = dup(-e1 * si), ce = dup(e1 * co);
            // s and d in the places of P and N; the columns' sources.
#pragma unroll
            for (int r = 0; r < RP; ++r) {
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const float2 p = P[s][r], n = N[s][r];
                    P[s][r] = sub2(p, n);
                    N[s][r] = add2(p, n);
                }
                if constexpr (T2) {
                    P[I2][r] = fma2(dup(k2), P[0][r], P[I2][r]);
                    N[I2][r] = fma2(dup(k2), N[0][r], N[I2][r]);
                }
                if constexpr (T1) Z[I1][r] = fma2(dup(k1), Z[0][r], Z[I1][r]);
            }
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                float2 b0 = dup(0.f), z0 = dup(0.f);
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const float2 d = N[s][r], st = P[s][r];
                    float2 b = fma2(hco, d, mul2(nsi, Z[s][r]));
                    float2 z = fma2(hsi, d, mul2(ce, Z[s][r]));
                    if (s == 0) {
                        b0 = b;
                        z0 = z;
                    }
                    if (B1 && s == IB) {
                        b = fma2(dup(-echo.x), z0, b);
                        z = fma2(dup(echo.x), b0, z);
                    }
                    P[s][r] = fma2(H, st, b);
                    N[s][r] = fma2(nH, st, b);
                    Z[s][r] = z;
                }
            }
            if (q == 0) {
                // The sample, a half interval after the pulse.
                const float x = -e2_rec * N[0][0].x;
                rec[slot * ROW + held] = x;
                if constexpr (T1) rec[(I1 * VPW + slot) * ROW + held] = -e2_rec * N[I1][0].x;
                if constexpr (T2)
                    rec[(I2 * VPW + slot) * ROW + held] = fmaf(k2_rec, x, -e2_rec * N[I2][0].x);
                if constexpr (B1) rec[(IB * VPW + slot) * ROW + held] = -e2_rec * N[IB][0].x;
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) shift_slots<RP, L>(P[s], N[s], q, kill_r);
            if (++held == kCpmgEchoes || base + i + 1 == echoes) {
                __syncwarp();
                // Lane -> sample column, sixteen to a row, two rows at once.
                const int col = lane % kCpmgEchoes;
                const int output = base + i + 1 - held + col;
                float ci = 0.f, cr = 1.f;
                if (col < held) sincosf(turn - phase[2 * output + 2].y, &ci, &cr);
#pragma unroll 1
                for (int v = lane / kCpmgEchoes; v < VPW; v += 32 / kCpmgEchoes) {
                    const float m = __shfl_sync(0xffffffffu, m0, v * L);
                    if (v >= rows || col >= held) continue;
                    const int64_t row = train * a.atoms + first_atom + v;
                    const float x = rec[v * ROW + col];
                    if (a.out_a) {
                        const float y = m * x;
                        put(a.layout, a.out_a, a.out_b, row * a.outputs + output, y * cr, y * ci);
                    }
                    if constexpr (NS > 1) {
                        const int64_t jac = row * a.jac_cols;
                        auto column = [&](int c, float y) {
                            if (c >= 0)
                                put(a.layout, a.jac_a, a.jac_b, (jac + c) * a.outputs + output,
                                    y * cr, y * ci);
                        };
                        column(a.col_m0, x);
                        if constexpr (T1) column(a.col_t1, m * rec[(I1 * VPW + v) * ROW + col]);
                        if constexpr (T2) column(a.col_t2, m * rec[(I2 * VPW + v) * ROW + col]);
                        if constexpr (B1) column(a.col_b1, m * rec[(IB * VPW + v) * ROW + col]);
                    }
                }
                __syncwarp();
                held = 0;
            }
        }
    }
}

struct CpmgEntry {
    int pairs, lanes;
    void (*launch[3])(const ComplexArgs&, dim3, cudaStream_t);  // no columns, T1 T2, T1 T2 B1
};

template <int RP, int L, int TM>
void launch_cpmg(const ComplexArgs& a, dim3 grid, cudaStream_t s) {
    epg_cpmg_kernel<RP, L, TM><<<grid, 32 * kCpmgWarps, 0, s>>>(a);
}

#define TSG_CPMG_ENTRY(RP, L) \
    {RP, L, {&launch_cpmg<RP, L, 0>, &launch_cpmg<RP, L, 3>, &launch_cpmg<RP, L, 7>}}

// By rising slot count.
const CpmgEntry kCpmg[] = {TSG_CPMG_ENTRY(2, 1), TSG_CPMG_ENTRY(3, 1), TSG_CPMG_ENTRY(4, 1),
                           TSG_CPMG_ENTRY(3, 2), TSG_CPMG_ENTRY(4, 2), TSG_CPMG_ENTRY(3, 4),
                           TSG_CPMG_ENTRY(4, 4)};

}  // namespace

bool find_cpmg(const HostProgram& program) {
    if (program.phase.empty() || program.ops < 3 || !(program.ops & 1)) return false;
    if (program.outputs != program.ops >> 1) return false;
    constexpr uint32_t rotate = uint32_t(RF_ROTATE) << OP_RF_SHIFT;
    constexpr uint32_t refocus = OP_RELAX | (1u << OP_SHIFT1_SHIFT) | rotate | (1u << OP_SHIFT2_SHIFT);
    for (int64_t t = 0; t < program.trains; ++t) {
        const Op* ops = program.op.data() + t * program.ops;
        const float2* phase = program.phase.data() + t * program.ops;
        // (An interval before the excitation leaves the equilibrium as it is.)
        if ((ops[0].code & ~uint32_t(OP_RELAX)) != rotate) return false;
        for (int64_t i = 1; i < program.ops; ++i) {
            // An op without a relaxation is one of zero duration.
            if ((ops[i].code | OP_RELAX) != ((i & 1) ? refocus : uint32_t(OP_RELAX | OP_RECORD))) return false;
            if (!(i & 1) && ops[i].record != (i >> 1) - 1) return false;
            if ((i & 1) && phase[i].x != phase[1].x) return false;
        }
        // The component that the split leaves out is below the samples'
        // rounding.
        const double angle = double(phase[0].x) - double(phase[1].x);
        if (!(std::fabs(std::cos(angle)) <= 0x1p-23)) return false;
    }
    return true;
}

int launch_cpmg(const tsg_program* program, const complex_detail::ComplexArgs& a, int tangents, cudaStream_t stream,
                bool* taken) {
    *taken = false;
    if (!program->host.cpmg || a.b1_phase || a.b0 || a.states < 2) return TSG_OK;
    const int64_t echoes = program->host.ops >> 1;
    const int64_t needed = std::min<int64_t>(a.states / 2, (echoes + 1) / 2);
    const CpmgEntry* entry = nullptr;
    for (const CpmgEntry& e : kCpmg)
        if (!entry && 2 * e.pairs * e.lanes >= needed) entry = &e;
    if (!entry) return TSG_OK;
    const int vpb = kCpmgWarps * (32 / entry->lanes);
    const int64_t blocks = (a.atoms + vpb - 1) / vpb;
    if (blocks > 0x7fffffffLL) return TSG_OK;
    *taken = true;
    entry->launch[tangents == 0 ? 0 : tangents == 3 ? 1 : 2](
        a, dim3(unsigned(blocks), unsigned(program->host.trains)), stream);
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

}  // namespace tsg
