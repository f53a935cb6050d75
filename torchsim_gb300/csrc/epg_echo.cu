// CPMG trains of a batch, one voxel per lane, every order in registers.
//
// An echo train touches few orders at a time: before echo e's pulse the
// states reach order 2 e + 1, and what sits above order 2 (echoes - e) - 1
// cannot come back to an echo any more. With the 2 x echoes states such a
// train is given, a quarter of orders x echoes matters; the rest is zero or
// never read. The sequences' orders spread over lanes (epg_batched.cu) cannot
// skip it, since the active orders would sit in few of a voxel's lanes.
//
// Here a lane holds order pairs (2 j, 2 j + 1) of F+, -F- and Z, and the two
// shifts of an echo (one before its pulse, one after) taken together move F+
// up and F- down by one whole pair: a rotated pair is written where the next
// echo reads it, and no lane talks to another. The pairs run in chunks of
// four behind a uniform branch, stage by stage within a chunk. Relaxation is
// folded into the pulse (the factors are fixed along the train, e at the
// first echo and e^2 after), the recovery into the addend of order 0
// (epg_train.cuh's form). Echoes go to shared memory and leave 32 at a time.
//
// Bound: the FMA pipe, with the chunk's unused pairs and the per-lane sin/cos
// as overhead.
#include "tsg_internal.h"

namespace tsg {
namespace {

constexpr int kPairs = 32;       // orders below 64: trains of up to 64 echoes
constexpr int kChunk = 4;        // pairs at a time
constexpr int kEchoRecords = 32;

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

__global__ void __launch_bounds__(64, 4) epg_echo_kernel(
    const Op* __restrict__ ops, const tsg_batch_sequence* __restrict__ seqs,
    const tsg_batch_unit* __restrict__ units, const float* __restrict__ t1v,
    const float* __restrict__ t2v, const float* __restrict__ m0v, const float* __restrict__ b1v,
    float2* __restrict__ out) {
    __shared__ float s_flip[64];
    __shared__ float s_rec[2][32 * (kEchoRecords + 1)];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const tsg_batch_unit u = units[blockIdx.x];
    const tsg_batch_sequence sq = seqs[u.sequence];
    const Op* train = ops + sq.op_offset;
    const int echoes = sq.op_count >> 1;
    for (int e = threadIdx.x; e < echoes; e += blockDim.x) s_flip[e] = train[2 * e + 1].flip;
    __syncthreads();
    const int local = warp * 32 + lane;
    const bool active = local < u.voxel_count;
    const int64_t voxel = sq.voxel_offset + u.voxel_begin + (active ? local : 0);
    const float t1 = t1v[voxel], t2 = t2v[voxel];
    const float m0 = m0v ? m0v[voxel] : 1.f;
    const float b1 = b1v ? b1v[voxel] : 1.f;
    const float dt = train[1].dt;
    const float f1 = expf(__fmul_rn(-(1000.f / t1), dt)), f2 = expf(__fmul_rn(-(1000.f / t2), dt));
    const float m0f2 = __fmul_rn(m0, f2);
    const int last_order = sq.states - 1;
    // Only a train with fewer states than it reaches meets its truncation.
    const bool capped = last_order < echoes;
    float* rec = s_rec[warp];

    float2 P[kPairs], N[kPairs], Z[kPairs];
#pragma unroll
    for (int j = 0; j < kPairs; ++j) P[j] = N[j] = Z[j] = dup(0.f);
    {
        // The excitation of the equilibrium, then the first shift.
        float si, co;
        sincosf(__fmul_rn(train[0].flip, b1), &si, &co);
        P[0].y = last_order >= 1 ? -si : 0.f;
        Z[0].x = co;
    }
    float w1 = f1, h = 0.5f * f2;
    int held = 0;
#pragma unroll 1
    for (int e = 0; e < echoes; ++e) {
        float si, co;
        sincosf(__fmul_rn(s_flip[e], b1), &si, &co);
        const float r = 1.f - w1;
        const float2 H = dup(h), nH = dup(-h), hco = dup(__fmul_rn(h, co)), hsi = dup(__fmul_rn(h, si));
        const float2 nsi = dup(-__fmul_rn(w1, si)), ce = dup(__fmul_rn(w1, co));
        const float2 bias_b = make_float2(-__fmul_rn(si, r), 0.f);
        const float2 bias_z = make_float2(__fmul_rn(co, r), 0.f);
        const int top = min(min(2 * e + 1, 2 * (echoes - e) - 1), last_order) >> 1;  // last pair
        float2 carry = dup(0.f);  // the pair that goes to the next chunk's first place
        float first_y = 0.f, second_x = 0.f;
#pragma unroll
        for (int c = 0; c < kPairs; c += kChunk) {
            if (c <= top) {
                float2 s[kChunk], d[kChunk], B[kChunk];
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    const float2 p = P[c + j], n = N[c + j];
                    s[j] = make_float2(__fadd_rn(p.x, -n.x), __fadd_rn(p.y, -n.y));
                    d[j] = add2(p, n);
                }
#pragma unroll
                for (int j = 0; j < kChunk; ++j)
                    B[j] = c + j == 0 ? fma2(nsi, Z[0], bias_b) : mul2(nsi, Z[c + j]);
#pragma unroll
                for (int j = 0; j < kChunk; ++j) B[j] = fma2(hco, d[j], B[j]);
#pragma unroll
                for (int j = 0; j < kChunk; ++j)
                    Z[c + j] = c + j == 0 ? fma2(ce, Z[0], bias_z) : mul2(ce, Z[c + j]);
#pragma unroll
                for (int j = 0; j < kChunk; ++j) Z[c + j] = fma2(hsi, d[j], Z[c + j]);
                // -F- moves a pair down, F+ a pair up.
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    const float2 n = fma2(nH, s[j], B[j]);
                    if (c + j == 0) first_y = n.y;
                    if (c + j == 1) second_x = n.x;
                    if (c + j > 0) N[c + j - 1] = n;
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
                    for (int j = 1; j < kChunk; ++j) {
                        if (2 * (c + j) > last_order) P[c + j].x = 0.f;
                        if (2 * (c + j) + 1 > last_order) P[c + j].y = 0.f;
                    }
                    if (2 * (c + kChunk) > last_order) carry.x = 0.f;
                    if (2 * (c + kChunk) + 1 > last_order) carry.y = 0.f;
                }
            } else if (c <= top + kChunk) {
                P[c] = carry;
            }
        }
        // The shift after the pulse brings F-[1] to order 0, the next one
        // F-[2]: F+[0] = -F-[0] each time.
        P[0] = make_float2(second_x, last_order >= 1 ? first_y : 0.f);
        rec[lane * (kEchoRecords + 1) + held] = __fmul_rn(m0f2, first_y);
        if (++held == kEchoRecords || e + 1 == echoes) {
            __syncwarp();
            const int first = u.voxel_begin + warp * 32;
            const int rows = min(32, u.voxel_count - warp * 32);
            float2* dst = out + sq.output_offset + int64_t(first) * sq.outputs + (e + 1 - held) + lane;
            if (lane < held)
                for (int v = 0; v < rows; ++v)
                    __stcs(dst + int64_t(v) * sq.outputs,
                           make_float2(0.f, rec[v * (kEchoRecords + 1) + lane]));
            __syncwarp();
            held = 0;
        }
        w1 = __fmul_rn(f1, f1);
        h = 0.5f * __fmul_rn(f2, f2);
    }
}

}  // namespace
}  // namespace tsg

using namespace tsg;

extern "C" int tsg_epg_echo_forward(const void* ops, const tsg_batch_sequence* sequences,
                                    const tsg_batch_unit* units, int64_t unit_count,
                                    const tsg_tissue* tissue, void* out, void* stream) {
    if (unit_count < 0 || (unit_count > 0 && (!ops || !sequences || !units || !out)))
        return fail(TSG_ERR_ARGUMENT, "null batch buffer");
    if (!tissue || (unit_count > 0 && (!tissue->t1_ms || !tissue->t2_ms)))
        return fail(TSG_ERR_ARGUMENT, "t1 and t2 are required");
    if (tissue->inversion) return fail(TSG_ERR_UNSUPPORTED, "batched sequences take no inversion map");
    if (unit_count > 0x7fffffffLL) return fail(TSG_ERR_CAPACITY, "too many units for one launch");
    if (unit_count == 0) return TSG_OK;
    epg_echo_kernel<<<unsigned(unit_count), 64, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const Op*>(ops), sequences, units, tissue->t1_ms, tissue->t2_ms, tissue->m0,
        tissue->b1, static_cast<float2*>(out));
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

// A train the echo kernel runs: the excitation alone, then per echo the
// refocusing op (relax, shift, rotate, shift) and the recording op, echo e
// recorded as sample e, one interval throughout, at most 64 echoes.
extern "C" int tsg_echo_train(const void* host_ops, int64_t op_count) {
    const Op* ops = static_cast<const Op*>(host_ops);
    if (!ops || op_count < 3 || !(op_count & 1) || op_count > 2 * 2 * kPairs + 1) return 0;
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
