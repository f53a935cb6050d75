// The steady state of a fast spin echo over its repetition time, applied to
// the recorded train and its columns in one pass (the reference's evaluate,
// simulators/fse.py:110-133, and its chain rule):
//   s = -1j x,  rec = exp(-(TR - ESP n) / T1),  y = M0 s (1 - rec) / (1 - rec s)
//   dy/dp = M0 (1 - rec) / (1 - rec s)^2 ds/dp, for T1 also
//           M0 s (s - 1) / (1 - rec s)^2 drec/dT1;  dy/dM0 = y / M0
// Written as one elementwise kernel because as tensor operations it was some
// forty launches, 0.3 ms on the device and 0.58 ms of host time at 65,536
// voxels x 48 echoes with two columns. A warp per row, its lanes along the
// echoes: 50 us there for 151 MB. (A thread per sample, which found its row by
// a 64-bit division and divided three times by complex numbers, took 92 us.)
#include "tsg_internal.h"

namespace tsg {
namespace {

constexpr int kRecoveryColumns = 16;

struct RecoveryColumns {
    int source[kRecoveryColumns];  // column of `jac_in`; -1: M0's
    int t1;                        // the output column that is T1's, or -1
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// 1 / a by Smith's division: no overflow of the squared magnitude.
__device__ __forceinline__ float2 creciprocal(float2 a) {
    const bool wide = fabsf(a.x) >= fabsf(a.y);
    const float r = wide ? a.y / a.x : a.x / a.y;
    const float d = 1.f / (wide ? a.x + a.y * r : a.x * r + a.y);
    return wide ? make_float2(d, -r * d) : make_float2(r * d, -d);
}

// A warp per row, its lanes along the echoes.
__global__ void __launch_bounds__(256) fse_recovery_kernel(
    const float2* __restrict__ signal, const float2* __restrict__ jac_in, int64_t rows, int echoes,
    int columns_in, int columns, RecoveryColumns map, const float* __restrict__ t1v, int t1_step,
    const float* __restrict__ m0v, int m0_step, float m0_value, float left_ms,
    float2* __restrict__ out, float2* __restrict__ jac_out) {
    const int64_t row = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const float t1 = t1v[row * t1_step];
    const float m0 = m0v ? m0v[row * m0_step] : m0_value;
    const float rec = expf(-1000.f / t1 * left_ms * 1e-3f);
    const float gone = 1.f - rec;
    const float k = rec * left_ms / (t1 * t1);
    const float2* x_row = signal + row * echoes;
    const float2* in = jac_in + row * columns_in * echoes;
    float2* y_row = out + row * echoes;
    float2* to = jac_out + row * columns * echoes;
    for (int e = threadIdx.x & 31; e < echoes; e += 32) {
        const float2 x = x_row[e];
        const float2 s = make_float2(x.y, -x.x);
        const float2 inverse = creciprocal(make_float2(1.f - rec * s.x, -rec * s.y));
        const float2 over_m0 = cmul(make_float2(s.x * gone, s.y * gone), inverse);
        y_row[e] = make_float2(m0 * over_m0.x, m0 * over_m0.y);
        if (columns == 0) continue;
        const float2 slope = cmul(make_float2(m0 * gone * inverse.x, m0 * gone * inverse.y), inverse);
        for (int c = 0; c < columns; ++c) {
            float2 y = over_m0;
            if (map.source[c] >= 0) {
                const float2 d = in[int64_t(map.source[c]) * echoes + e];
                y = cmul(slope, make_float2(d.y, -d.x));
                if (c == map.t1) {
                    const float2 a = cmul(make_float2(m0 * s.x, m0 * s.y), inverse);
                    const float2 g = cmul(cmul(a, make_float2(s.x - 1.f, s.y)), inverse);
                    y.x += g.x * k;
                    y.y += g.y * k;
                }
            }
            to[int64_t(c) * echoes + e] = y;
        }
    }
}

}  // namespace
}  // namespace tsg

using namespace tsg;

extern "C" int tsg_fse_recovery(const void* signal, const void* jacobian, int64_t rows,
                                int64_t echoes, int32_t columns_in, int32_t columns,
                                const int32_t* sources, int32_t t1_column, const float* t1_ms,
                                int64_t t1_count, const float* m0, int64_t m0_count, float m0_value,
                                float left_ms, void* out, void* jacobian_out, void* stream) {
    if (rows < 0 || echoes < 0 || columns < 0 || columns_in < 0)
        return fail(TSG_ERR_ARGUMENT, "invalid echo train dimensions");
    if (columns > kRecoveryColumns) return fail(TSG_ERR_CAPACITY, "more than 16 columns");
    if (rows * echoes == 0) return TSG_OK;
    if (!signal || !t1_ms || !out || (columns > 0 && (!sources || !jacobian_out)))
        return fail(TSG_ERR_ARGUMENT, "null echo train buffer");
    if ((t1_count != 1 && t1_count != rows) || (m0 && m0_count != 1 && m0_count != rows))
        return fail(TSG_ERR_ARGUMENT, "one T1 and M0, or one for each row");
    RecoveryColumns map{};
    map.t1 = t1_column;
    for (int c = 0; c < columns; ++c) {
        map.source[c] = sources[c];
        if (sources[c] >= columns_in || (sources[c] >= 0 && !jacobian))
            return fail(TSG_ERR_ARGUMENT, "column out of range");
    }
    const int64_t blocks = (rows + 7) / 8;
    if (echoes > 0x7fffffffLL || blocks > 0x7fffffffLL)
        return fail(TSG_ERR_CAPACITY, "launch too large");
    fse_recovery_kernel<<<unsigned(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const float2*>(signal), static_cast<const float2*>(jacobian), rows, int(echoes),
        columns_in, columns, map, t1_ms, t1_count == 1 ? 0 : 1, m0, m0_count == 1 ? 0 : 1, m0_value,
        left_ms, static_cast<float2*>(out), static_cast<float2*>(jacobian_out));
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}
