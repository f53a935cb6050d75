// CPMG trains of a batch, two voxels per lane, every order in registers.
//
// An echo train touches few orders at a time. Both shifts of an echo interval
// together move by two orders, so what the excitation made stays on odd orders
// before every pulse and is recorded, and what recovers from order 0 stays on
// even orders and never reaches an echo: only order 2 m + 1, m = 0, 1, ...
// counts. Before echo e's pulse m reaches e, and what sits above
// echoes - 1 - e cannot come back any more. So an eighth of the 2 x echoes
// states x echoes such a train is given matters; the rest is zero or never
// read. The sequences' orders spread over lanes (epg_batched.cu) cannot skip
// it, since the active orders would sit in few of a voxel's lanes.
//
// Here a lane holds F+, -F- and Z of every m for two voxels of a sequence as
// pairs: the paired products need no order's neighbour, and the shift moves F+
// up and F- down by one whole pair, so a rotated pair is written where the
// next echo reads it and no lane talks to another. The orders run in chunks
// of four behind a uniform branch, stage by stage within a chunk. Relaxation
// is folded into the pulse (the factors are fixed along the train, e at the
// first echo and e^2 after). Echoes go to shared memory and leave 32 at a time.
//
// Bound: the FMA pipe, with the sine and cosine of each pulse and voxel next.
// Measured on 96 CPMG protocols of 4 to 64 echoes, 1.5 million voxels: 2.21 ms
// with the orders spread over lanes, 0.75 ms with every order of one voxel in
// a lane's pairs, 0.46 ms here with sincosf and 0.43 with turn2().
//
// With few units one warp's chain decides, all chunks of an echo one after the
// other, and with few voxels in each unit most lanes idle: there the chunks of
// two voxels go to lanes of their own (epg_echo_few_kernel), with the same
// arithmetic and so the same bits. (Without it such a batch took longer than with the
// orders spread over lanes: one train of 64 echoes 33 and 21 us, 2,000 of them
// with four voxels each 84 and 47.)
#include "tsg_internal.h"

namespace tsg {
namespace {

constexpr int kSlots = 32;       // odd orders below 64: trains of up to 64 echoes
constexpr int kChunk = 4;        // orders at a time
constexpr int kEchoRecords = 32;

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// The sines and cosines of two angles without a branch, for |x| <= 2^20:
// reduction to |r| <= pi/4 by a three-part pi/2 (W. J. Cody and W. Waite,
// Software Manual for the Elementary Functions, 1980; with fused products the
// first difference is exact) and the Taylor series to r^9 and r^10, whose
// remainders there are 2e-9 and 2e-10. Against extended precision its steps are
// within 1.5 ulp up to 1e5 rad and within 2 ulp over the range.
// kTurnLimit bounds a flip in rad and a B1 factor each; a voxel or echo beyond
// it, or NaN, calls sincosf.
constexpr float kTurnLimit = 1024.f;

__device__ __forceinline__ bool turns_wild(float x) { return !(fabsf(x) <= kTurnLimit); }

__device__ __forceinline__ void place_turn(int quadrant, float s, float c, float* si, float* co) {
    const bool swap = quadrant & 1;
    const float a = swap ? c : s, b = swap ? s : c;
    *si = __int_as_float(__float_as_int(a) ^ ((quadrant & 2) << 30));
    *co = __int_as_float(__float_as_int(b) ^ (((quadrant + 1) & 2) << 30));
}

__device__ __forceinline__ void turn2(float2 x, float2* si, float2* co) {
    const float2 shifted = fma2(x, dup(0x1.45f306p-1f), dup(12582912.f));  // 2/pi; 1.5 * 2^23
    const float2 n = add2(shifted, dup(-12582912.f));
    float2 r = fma2(n, dup(-0x1.921fb6p+0f), x);
    r = fma2(n, dup(0x1.777a5cp-25f), r);
    r = fma2(n, dup(0x1.ee59dap-50f), r);
    const float2 t = mul2(r, r);
    float2 s = fma2(t, dup(1.f / 362880.f), dup(-1.f / 5040.f));
    float2 c = fma2(t, dup(-1.f / 3628800.f), dup(1.f / 40320.f));
    s = fma2(t, s, dup(1.f / 120.f));
    c = fma2(t, c, dup(-1.f / 720.f));
    s = fma2(t, s, dup(-1.f / 6.f));
    c = fma2(t, c, dup(1.f / 24.f));
    s = fma2(mul2(t, r), s, r);
    c = fma2(t, c, dup(-0.5f));
    c = fma2(t, c, dup(1.f));
    place_turn(__float_as_int(shifted.x), s.x, c.x, &si->x, &co->x);
    place_turn(__float_as_int(shifted.y), s.y, c.y, &si->y, &co->y);
}

// Both voxels' sample `held`, voxel-major.
__device__ __forceinline__ void rec_store(float* rec, int lane, int held, float2 y) {
    rec[lane * (kEchoRecords + 1) + held] = y.x;
    rec[(lane + 32) * (kEchoRecords + 1) + held] = y.y;
}

__global__ void __launch_bounds__(32, 8) epg_echo_kernel(
    const Op* __restrict__ ops, const tsg_batch_sequence* __restrict__ seqs,
    const tsg_batch_unit* __restrict__ units, const float* __restrict__ t1v,
    const float* __restrict__ t2v, const float* __restrict__ m0v, const float* __restrict__ b1v,
    float2* __restrict__ out) {
    __shared__ float s_flip[2 * kSlots];
    __shared__ float s_rec[64 * (kEchoRecords + 1)];
    const int lane = threadIdx.x;
    const tsg_batch_unit u = units[blockIdx.x];
    const tsg_batch_sequence sq = seqs[u.sequence];
    const Op* train = ops + sq.op_offset;
    const int echoes = sq.op_count >> 1;
    bool far = false;
    for (int e = lane; e < echoes; e += 32) {
        s_flip[e] = train[2 * e + 1].flip;
        far |= turns_wild(s_flip[e]);
    }
    // This lane's voxels: lane and lane + 32 of the unit.
    const int voxels = min(u.voxel_count, 64);
    const int64_t first = sq.voxel_offset + u.voxel_begin;
    const int64_t va = first + (lane < voxels ? lane : 0);
    const int64_t vb = first + (lane + 32 < voxels ? lane + 32 : 0);
    const float dt = train[1].dt;
    const float2 b1 = b1v ? make_float2(b1v[va], b1v[vb]) : dup(1.f);
    // An angle that turn2() does not take.
    const bool wild = __any_sync(0xffffffffu, far || turns_wild(b1.x) || turns_wild(b1.y));
    __syncwarp();
    const float2 m0 = m0v ? make_float2(m0v[va], m0v[vb]) : dup(1.f);
    const float2 f1 = make_float2(expf(__fmul_rn(-(1000.f / t1v[va]), dt)),
                                  expf(__fmul_rn(-(1000.f / t1v[vb]), dt)));
    const float2 f2 = make_float2(expf(__fmul_rn(-(1000.f / t2v[va]), dt)),
                                  expf(__fmul_rn(-(1000.f / t2v[vb]), dt)));
    const float2 m0f2 = mul2(m0, f2);
    const int slots = sq.states >> 1;  // odd orders below the state limit
    // Only a train with fewer states than it reaches meets its truncation.
    const bool capped = 2 * slots < echoes;

    float2 P[kSlots], N[kSlots], Z[kSlots];
#pragma unroll
    for (int m = 0; m < kSlots; ++m) P[m] = N[m] = Z[m] = dup(0.f);
    {
        // The excitation of the equilibrium, then the first shift.
        const float2 a = mul2(dup(train[0].flip), b1);
        if (slots > 0) P[0] = make_float2(-sinf(a.x), -sinf(a.y));
    }
    float2 w1 = f1, h = mul2(dup(0.5f), f2);
    int held = 0;
#pragma unroll 1
    for (int e = 0; e < echoes; ++e) {
        const float2 angle = mul2(dup(s_flip[e]), b1);
        float2 si, co;
        turn2(angle, &si, &co);
        if (wild) {
            if (turns_wild(s_flip[e]) || turns_wild(b1.x)) sincosf(angle.x, &si.x, &co.x);
            if (turns_wild(s_flip[e]) || turns_wild(b1.y)) sincosf(angle.y, &si.y, &co.y);
        }
        const float2 H = h, nH = make_float2(-h.x, -h.y), hco = mul2(h, co), hsi = mul2(h, si);
        const float2 wsi = mul2(w1, si), nsi = make_float2(-wsi.x, -wsi.y), ce = mul2(w1, co);
        const int top = min(min(e, echoes - 1 - e), slots - 1);  // the last order
        float2 carry = dup(0.f);  // goes to the next chunk's first place
        float2 echo = dup(0.f);
#pragma unroll
        for (int c = 0; c < kSlots; c += kChunk) {
            if (c <= top) {
                float2 s[kChunk], d[kChunk], B[kChunk];
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    const float2 p = P[c + j], n = N[c + j];
                    s[j] = make_float2(__fadd_rn(p.x, -n.x), __fadd_rn(p.y, -n.y));
                    d[j] = add2(p, n);
                }
#pragma unroll
                for (int j = 0; j < kChunk; ++j) B[j] = fma2(hco, d[j], mul2(nsi, Z[c + j]));
#pragma unroll
                for (int j = 0; j < kChunk; ++j) Z[c + j] = fma2(hsi, d[j], mul2(ce, Z[c + j]));
                // -F- moves down, F+ up.
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    const float2 n = fma2(nH, s[j], B[j]);
                    if (c + j == 0) echo = n;
                    else N[c + j - 1] = n;
                }
                N[c + kChunk - 1] = dup(0.f);
                if (c > 0) P[c] = carry;
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    const float2 p = fma2(H, s[j], B[j]);
                    if (j + 1 < kChunk) P[c + j + 1] = p;
                    else carry = p;
                }
                if (capped) {
#pragma unroll
                    for (int j = 1; j < kChunk; ++j)
                        if (c + j >= slots) P[c + j] = dup(0.f);
                    if (c + kChunk >= slots) carry = dup(0.f);
                }
            } else if (c <= top + kChunk) {
                P[c] = carry;
            }
        }
        // The shift after the pulse brings F-[1] to order 0, where it is
        // recorded, and the next one takes F+[0] = -F-[0] up.
        P[0] = slots > 0 ? echo : dup(0.f);
        rec_store(s_rec, lane, held, mul2(m0f2, echo));
        if (++held == kEchoRecords || e + 1 == echoes) {
            __syncwarp();
            float2* dst = out + sq.output_offset + int64_t(u.voxel_begin) * sq.outputs +
                          (e + 1 - held) + lane;
            if (lane < held)
                for (int v = 0; v < voxels; ++v)
                    __stcs(dst + int64_t(v) * sq.outputs,
                           make_float2(0.f, s_rec[v * (kEchoRecords + 1) + lane]));
            __syncwarp();
            held = 0;
        }
        w1 = mul2(f1, f1);
        h = mul2(dup(0.5f), mul2(f2, f2));
    }
}

// The same trains with a chunk of orders per lane: lane q of kFewLanes holds
// orders 4 q to 4 q + 3 of two voxels and evaluates the sines and cosines of every
// kFewLanes-th echo; the pair that crosses a chunk's edge moves by shuffle. A unit
// has up to 64 / kFewLanes voxels. Bound: the chain of one echo, about 0.18 us: 64
// echoes of 64 voxels 18.4 us with the coefficients and selects on it, 16.4 here;
// with many units the paired FMAs (47% active, 0.64 issued a cycle), on eight
// lanes at twice the other kernel's time for a dense unit. (The lines between the
// two: torchsim_gb300/batching.py.)
template <int kFewLanes>
__global__ void __launch_bounds__(32) epg_echo_few_kernel(
    const Op* __restrict__ ops, const tsg_batch_sequence* __restrict__ seqs,
    const tsg_batch_unit* __restrict__ units, const float* __restrict__ t1v,
    const float* __restrict__ t2v, const float* __restrict__ m0v, const float* __restrict__ b1v,
    float2* __restrict__ out) {
    constexpr int kFewVoxels = 2 * 32 / kFewLanes;
    __shared__ float s_flip[2 * kSlots];
    __shared__ float s_rec[kFewVoxels * (kEchoRecords + 1)];
    const int lane = threadIdx.x;
    const int q = lane % kFewLanes, pair = lane / kFewLanes;
    const tsg_batch_unit u = units[blockIdx.x];
    const int voxels = min(u.voxel_count, kFewVoxels);
    const tsg_batch_sequence sq = seqs[u.sequence];
    const Op* train = ops + sq.op_offset;
    const int echoes = sq.op_count >> 1;
    for (int e = lane; e < echoes; e += 32) s_flip[e] = train[2 * e + 1].flip;
    __syncwarp();
    // This group's voxels: pair and pair + kFewVoxels / 2 of the unit.
    const int64_t first = sq.voxel_offset + u.voxel_begin;
    const int other = pair + kFewVoxels / 2;
    const int64_t va = first + (pair < voxels ? pair : 0);
    const int64_t vb = first + (other < voxels ? other : 0);
    const float dt = train[1].dt;
    const float2 b1 = b1v ? make_float2(b1v[va], b1v[vb]) : dup(1.f);
    const float2 m0 = m0v ? make_float2(m0v[va], m0v[vb]) : dup(1.f);
    const float2 f1 = make_float2(expf(__fmul_rn(-(1000.f / t1v[va]), dt)),
                                  expf(__fmul_rn(-(1000.f / t1v[vb]), dt)));
    const float2 f2 = make_float2(expf(__fmul_rn(-(1000.f / t2v[va]), dt)),
                                  expf(__fmul_rn(-(1000.f / t2v[vb]), dt)));
    const float2 m0f2 = mul2(m0, f2);
    const int slots = sq.states >> 1;
    // All orders run at every echo: the ones that matter meet only each other.
    // Masks instead of selects keep the truncation and the last lane's edge off
    // the predicates.
    int keep[kChunk];
#pragma unroll
    for (int j = 0; j < kChunk; ++j)
        keep[j] = 2 * slots < echoes && q * kChunk + j + 1 >= slots ? 0 : -1;
    const int inner = q == kFewLanes - 1 ? 0 : -1;
    auto masked = [](float2 v, int mask) {
        return make_float2(__int_as_float(__float_as_int(v.x) & mask),
                           __int_as_float(__float_as_int(v.y) & mask));
    };

    float2 P[kChunk], N[kChunk], Z[kChunk];
#pragma unroll
    for (int j = 0; j < kChunk; ++j) P[j] = N[j] = Z[j] = dup(0.f);
    {
        const float2 a = mul2(dup(train[0].flip), b1);
        if (q == 0 && slots > 0) P[0] = make_float2(-sinf(a.x), -sinf(a.y));
    }
    // The pulse of echo e with the relaxation before it (w1, h) folded in.
    float2 my_si = dup(0.f), my_co = dup(0.f);
    float2 hco, hsi, nsi, ce;
    auto coefficients = [&](int e, float2 w1, float2 h) {
        const int g = e % kFewLanes;
        if (g == 0) {
            const float flip = s_flip[min(e + q, echoes - 1)];
            const float2 angle = mul2(dup(flip), b1);
            turn2(angle, &my_si, &my_co);
            if (turns_wild(flip) || turns_wild(b1.x)) sincosf(angle.x, &my_si.x, &my_co.x);
            if (turns_wild(flip) || turns_wild(b1.y)) sincosf(angle.y, &my_si.y, &my_co.y);
        }
        const float2 si = make_float2(__shfl_sync(0xffffffffu, my_si.x, g, kFewLanes),
                                      __shfl_sync(0xffffffffu, my_si.y, g, kFewLanes));
        const float2 co = make_float2(__shfl_sync(0xffffffffu, my_co.x, g, kFewLanes),
                                      __shfl_sync(0xffffffffu, my_co.y, g, kFewLanes));
        const float2 wsi = mul2(w1, si);
        hco = mul2(h, co);
        hsi = mul2(h, si);
        nsi = make_float2(-wsi.x, -wsi.y);
        ce = mul2(w1, co);
    };
    float2 h = mul2(dup(0.5f), f2);
    const float2 w_later = mul2(f1, f1), h_later = mul2(dup(0.5f), mul2(f2, f2));
    coefficients(0, f1, h);
    int held = 0;
#pragma unroll 1
    for (int e = 0; e < echoes; ++e) {
        const float2 nH = make_float2(-h.x, -h.y);
        float2 n[kChunk], p[kChunk];
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
            const float2 s = make_float2(__fadd_rn(P[j].x, -N[j].x), __fadd_rn(P[j].y, -N[j].y));
            const float2 d = add2(P[j], N[j]);
            const float2 B = fma2(hco, d, mul2(nsi, Z[j]));
            Z[j] = fma2(hsi, d, mul2(ce, Z[j]));
            n[j] = fma2(nH, s, B);
            p[j] = masked(fma2(h, s, B), keep[j]);
        }
        // -F- moves down, F+ up.
        const float2 above = make_float2(__shfl_down_sync(0xffffffffu, n[0].x, 1, kFewLanes),
                                         __shfl_down_sync(0xffffffffu, n[0].y, 1, kFewLanes));
        const float2 below = make_float2(__shfl_up_sync(0xffffffffu, p[kChunk - 1].x, 1, kFewLanes),
                                         __shfl_up_sync(0xffffffffu, p[kChunk - 1].y, 1, kFewLanes));
        // The next echo's coefficients meanwhile.
        h = h_later;
        coefficients(e + 1, w_later, h_later);
        if (q == 0) {
            const float2 y = mul2(m0f2, n[0]);
            s_rec[pair * (kEchoRecords + 1) + held] = y.x;
            s_rec[other * (kEchoRecords + 1) + held] = y.y;
        }
        P[0] = q == 0 ? (slots > 0 ? n[0] : dup(0.f)) : below;
#pragma unroll
        for (int j = 0; j + 1 < kChunk; ++j) {
            N[j] = n[j + 1];
            P[j + 1] = p[j];
        }
        N[kChunk - 1] = masked(above, inner);
        if (++held == kEchoRecords || e + 1 == echoes) {
            __syncwarp();
            float2* dst = out + sq.output_offset + int64_t(u.voxel_begin) * sq.outputs +
                          (e + 1 - held) + lane;
            if (lane < held)
                for (int v = 0; v < voxels; ++v)
                    __stcs(dst + int64_t(v) * sq.outputs,
                           make_float2(0.f, s_rec[v * (kEchoRecords + 1) + lane]));
            __syncwarp();
            held = 0;
        }
    }
}

}  // namespace
}  // namespace tsg

using namespace tsg;

namespace {

int launch_echo(decltype(&epg_echo_kernel) kernel, const void* ops, const tsg_batch_sequence* sequences,
                const tsg_batch_unit* units, int64_t unit_count, const tsg_tissue* tissue, void* out,
                void* stream) {
    if (unit_count < 0 || (unit_count > 0 && (!ops || !sequences || !units || !out)))
        return fail(TSG_ERR_ARGUMENT, "null batch buffer");
    if (!tissue || (unit_count > 0 && (!tissue->t1_ms || !tissue->t2_ms)))
        return fail(TSG_ERR_ARGUMENT, "t1 and t2 are required");
    if (tissue->inversion) return fail(TSG_ERR_UNSUPPORTED, "batched sequences take no inversion map");
    if (unit_count > 0x7fffffffLL) return fail(TSG_ERR_CAPACITY, "too many units for one launch");
    if (unit_count == 0) return TSG_OK;
    kernel<<<unsigned(unit_count), 32, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const Op*>(ops), sequences, units, tissue->t1_ms, tissue->t2_ms, tissue->m0,
        tissue->b1, static_cast<float2*>(out));
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

}  // namespace

extern "C" int tsg_epg_echo_forward(const void* ops, const tsg_batch_sequence* sequences,
                                    const tsg_batch_unit* units, int64_t unit_count,
                                    const tsg_tissue* tissue, void* out, void* stream) {
    return launch_echo(&epg_echo_kernel, ops, sequences, units, unit_count, tissue, out, stream);
}

extern "C" int tsg_epg_echo_few_forward(const void* ops, const tsg_batch_sequence* sequences,
                                        const tsg_batch_unit* units, int64_t unit_count,
                                        const tsg_tissue* tissue, void* out, int lanes,
                                        void* stream) {
    switch (lanes) {
        case 1: return launch_echo(&epg_echo_few_kernel<1>, ops, sequences, units, unit_count, tissue, out, stream);
        case 2: return launch_echo(&epg_echo_few_kernel<2>, ops, sequences, units, unit_count, tissue, out, stream);
        case 4: return launch_echo(&epg_echo_few_kernel<4>, ops, sequences, units, unit_count, tissue, out, stream);
        case 8: return launch_echo(&epg_echo_few_kernel<8>, ops, sequences, units, unit_count, tissue, out, stream);
    }
    return fail(TSG_ERR_ARGUMENT, "1, 2, 4 or 8 lanes for a voxel's orders");
}

// A train the echo kernel runs: the excitation alone, then per echo the
// refocusing op (relax, shift, rotate, shift) and the recording op, echo e
// recorded as sample e, one interval throughout, at most 64 echoes.
extern "C" int tsg_echo_train(const void* host_ops, int64_t op_count) {
    const Op* ops = static_cast<const Op*>(host_ops);
    if (!ops || op_count < 3 || !(op_count & 1) || op_count > 2 * 2 * kSlots + 1) return 0;
    constexpr uint32_t rotate = uint32_t(RF_ROTATE) << OP_RF_SHIFT;
    constexpr uint32_t refocus = OP_RELAX | (1u << OP_SHIFT1_SHIFT) | rotate | (1u << OP_SHIFT2_SHIFT);
    if (ops[0].code != rotate) return 0;
    for (int64_t i = 1; i < op_count; ++i) {
        if (ops[i].dt != ops[1].dt) return 0;
        if (ops[i].code != ((i & 1) ? refocus : uint32_t(OP_RELAX | OP_RECORD))) return 0;
        if (!(i & 1) && ops[i].record != (i >> 1) - 1) return 0;
    }
    return 1;
}
