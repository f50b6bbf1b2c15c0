// Fixed-point phases of the FP64 form, shared by the coherent sum and the incoherent transforms:
// phi = sum_c Q_c R_c mod 1 as a 64-bit fraction of a revolution (see phase_fx.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sassgpu {
namespace {

constexpr int kFxTable = 1024;            // grid angles per revolution
constexpr unsigned kFxBig = 0x49800000u;  // float bits of 2^20: larger coordinates are evaluated in FP64

struct FxQ {
    unsigned w1[3], w2[3];  // Q in units of 2^-(33 + E) (integer part, 64 bits)
    float w0[3];            // its next 32 bits, times 2^-32
    unsigned hi0, lo0;      // minus the phase of the coordinates' offset 2^31
};

// Q at block exponent E (coordinates below 2^E): the 2^-96 words shifted down by 31 - E.
__device__ __forceinline__ void fx_shift_q(const uint4* __restrict__ t, int E, FxQ& q) {
    const int s = 31 - E;  // 11 .. 31
    unsigned long long p0 = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint4 w = __ldg(t + c);
        q.w0[c] = __uint2float_rn(__funnelshift_r(w.x, w.y, s)) * 2.3283064365386963e-10f;
        q.w1[c] = __funnelshift_r(w.y, w.z, s);
        q.w2[c] = __funnelshift_r(w.z, w.w, s);
        p0 -= (((unsigned long long)q.w2[c] << 32) | q.w1[c]) << 31;
    }
    q.hi0 = (unsigned)(p0 >> 32);
    q.lo0 = (unsigned)p0;
}

}  // namespace
}  // namespace sassgpu
