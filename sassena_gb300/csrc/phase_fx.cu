// Phase sum of the FP64 form in fixed point.
//
// The FP64 form evaluates sum_j b_j exp(i q.r_j) to FP64 accuracy
// (AllVectorsScatterDevice::scatter, src/scatter_devices/all_vectors_scatter_device.cpp:388-439).
// GB300's FP64 pipe gives 1.7 results per clock and SM, so an FP64 sincos of about 29 FP64
// instructions costs 550 clocks of an SM per 32 terms. The same accuracy is reached here on
// the integer and FP32 pipes (64 and 128 results per clock and SM):
//   * the phase in revolutions is a 64-bit fraction, phi = sum_c Q_c R_c mod 1, with R_c the
//     coordinate in 32 bits (exact: a float has 24) and Q_c = q_c / 2 pi in 96 bits. Whole
//     revolutions drop out of the integer arithmetic, so phi is good to about 2^-60 where
//     FP64 rounds q.r itself (2^-47 at 100 rad);
//   * phi = i / 1024 + d: cos and sin of the grid angle come from a table in units of 2^-55
//     (kept in shared memory in eight copies, one for each lane of a quarter warp, so that the
//     128-bit reads have no bank conflicts), |x| = 2 pi |d| < 2^-8.3 is added by
//       cos = C - (S sin x + C (1 - cos x)),  sin = S + (C sin x - S (1 - cos x));
//   * what is summed: the table values and the products S d, C d of their upper halves with
//     the upper 22 bits of d exactly in 64-bit integers (2 pi is applied once per 128 atoms);
//     the rest (below 2^-17) rounded to multiples of 2^-39 in 32-bit integers, and what that
//     rounding leaves (below 2^-35) in FP32.
// Per term the errors add to 1.6e-16 rms (FP32 rounding of the cubic term of sin x and of the low
// phase words). Amplitudes against 80-bit arithmetic, rms: 300 atoms at q r <= 20 2.8e-14 (FP64
// kernel 7.6e-14), 2,000 atoms at q r <= 250 7.7e-14 (2.1e-12: FP64 rounds q.r). Measured on a
// GB300, 3,000 atoms x 250 frames x 12 shells x 60 directions: FP64 kernel 39.9 ms, this one
// 1.57 ms (3.4e11 terms/s, 29 clocks of an SM per 32 terms: the FMA pipe, which also takes the
// integer products, and the issue slots are both near three quarters busy). S(q,t) is off by 4.5e-16 of
// its norm with the last lags summed directly (correlate.cu), 2.0e-15 without; the FP64 kernel's by 1.3e-15.
//
// A warp owns 32 q-vectors (any shells: the factor is read per lane) and one frame, and
// streams the atoms in class order in blocks of 32: the lanes convert one atom each to the
// fixed-point record in shared memory, then all lanes read every record. Sums are taken to
// FP64 and multiplied by the class factor where the class changes and at least every 128
// atoms. Blocks with a coordinate that is not finite or not below 2^20, and q-vectors beyond
// 2^20 revolutions per length unit, are evaluated in FP64 as before.
#include <algorithm>

#include "common.cuh"
#include "fx.cuh"
#include "kernels.h"

namespace sassgpu {

namespace {

constexpr int kFxWarps = 24;           // one CTA per SM
constexpr int kFxFold = 4;             // blocks of 32 atoms per fold: 2^62 in units of 2^-55
constexpr int kFxTableBytes = kFxTable * 128;
constexpr int kFxRecord = 32 * 48;     // a block's records: integers, floats, residuals
constexpr int kFxSmem = kFxTableBytes + kFxWarps * kFxRecord;

// (cos, sin)(2 pi i / 1024) in units of 2^-55: Taylor series in 2^-62 on the first octant.
__global__ void fx_table_kernel(longlong2* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kFxTable; i += gridDim.x * blockDim.x) {
        const int quad = i >> 8, j = i & 255;
        const int k = j <= 128 ? j : 256 - j;                         // 0 .. 128: up to pi / 4
        const long long two_pi_60 = 0x6487ed5110b4611all;             // 2 pi 2^60
        const long long x = (two_pi_60 >> 8) * k + (((two_pi_60 & 255) * k) >> 8);  // 2 pi k / 1024 in 2^-62
        const long long x2 = __mul64hi(x, x) << 2;                    // 2^-62
        const long long one = 1ll << 62;
        long long c = one, s = one;
        for (int n = 11; n >= 1; --n) {  // x^24 / 24! is below 2^-88
            c = one - (__mul64hi(x2, c) << 2) / ((2 * n - 1) * (2 * n));
            s = one - (__mul64hi(x2, s) << 2) / ((2 * n) * (2 * n + 1));
        }
        s = __mul64hi(s, x) << 2;
        c = (c + 64) >> 7;
        s = (s + 64) >> 7;
        if (k == 0) {
            c = 1ll << 55;
            s = 0;
        }
        long long a = j <= 128 ? c : s, b = j <= 128 ? s : c;  // cos, sin of j / 1024
        if (quad & 1) {
            const long long t = a;
            a = -b;
            b = t;
        }
        if (quad & 2) {
            a = -a;
            b = -b;
        }
        out[i] = make_longlong2(a, b);
    }
}

// q / 2 pi in units of 2^-96 (two's complement, 128 bits) per component, and whether the
// vector is outside the fixed-point range: four uint4 per q-vector.
__global__ void fx_q_kernel(const double* __restrict__ qv, size_t nv, uint4* __restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < 3 * nv; i += (size_t)gridDim.x * blockDim.x) {
        const size_t v = i / 3;
        const int c = (int)(i - 3 * v);
        const unsigned long long bits = (unsigned long long)__double_as_longlong(qv[i]);
        const int be = (int)(bits >> 52) & 0x7ff;
        unsigned long long m = bits & 0xfffffffffffffull;
        if (be) m |= 1ull << 52;
        const int sh = 32 - ((be ? be : 1) - 1075);  // q = m 2^(be - 1075); T = (m I) >> sh, I = 2^128 / 2 pi
        unsigned long long w[4] = {0, 0, 0, 0};
        bool bad = be >= 1023 + 22;  // |q| >= 2^22 (and infinities, NaN)
        if (!bad && sh < 192) {      // sh > 0 since |q| < 2^22
            const unsigned long long ih = 0x28be60db9391054aull, il = 0x7f09d5f47d4d3770ull;
            unsigned long long p[4];
            p[0] = m * il;
            const unsigned long long t0 = __umul64hi(m, il), t1 = m * ih;
            p[1] = t0 + t1;
            p[2] = __umul64hi(m, ih) + (p[1] < t0 ? 1ull : 0ull);
            p[3] = 0;
            const int ws = sh >> 6, bs = sh & 63;
            for (int k = 0; k < 2; ++k) {
                const unsigned long long lo = k + ws < 4 ? p[k + ws] : 0, hi = k + ws + 1 < 4 ? p[k + ws + 1] : 0;
                w[k] = bs ? (lo >> bs) | (hi << (64 - bs)) : lo;
            }
        }
        if (bits >> 63) {  // negate
            w[0] = ~w[0] + 1;
            w[1] = ~w[1] + (w[0] == 0 ? 1ull : 0ull);
        }
        out[4 * v + c] = make_uint4((unsigned)w[0], (unsigned)(w[0] >> 32), (unsigned)w[1], (unsigned)(w[1] >> 32));
        if (bad) {
            out[4 * v + 3].x = 1u;  // every writer stores the same value; cleared before the launch
        }
    }
}

struct FxSums {
    long long c, s;       // table values, 2^-55
    long long lc, ls;     // upper half of C (S) times the upper bits of d, 2^-65 revolutions
    unsigned gc, gs;      // the rest on the 2^-39 grid (bit patterns of magic sums)
    float2 f;             // what the grid leaves, units of 2^-23
    __device__ __forceinline__ void clear() {
        c = s = lc = ls = 0;
        gc = gs = 0u;
        f = make_float2(0.f, 0.f);
    }
};

constexpr float kFxMagic = 192.f;  // 1.5 2^7: its last bit is 2^-16, 2^-39 in units of 2^-23

// One term: adds cos and sin of (phi + dt 2^-64) revolutions.
__device__ __forceinline__ void fx_term(unsigned hi, unsigned lo, float dt, const unsigned char* __restrict__ tab,
                                        FxSums& a) {
    const int sh = (int)(hi << 10);
    const uint4 e = *reinterpret_cast<const uint4*>(tab + (((hi + 0x200000u) >> 15) & 0x1ff80u));
    const int chi = (int)e.y, shi = (int)e.w;
    const float d1 = __int2float_rn(sh);                   // 22 bits: exact
    // x = 2 pi (d1 2^-42 + (lo + dt) 2^-64) as xh + xl; y is the part of x beyond d1's
    constexpr float P1 = 1.42863098e-12f;                  // 2 pi 2^-42 rounded
    constexpr float P2 = (float)(6.283185307179586476925 / 4398046511104.0 - (double)P1);
    constexpr float P3 = (float)(6.283185307179586476925 / 18446744073709551616.0);
    const float y = __fmul_rn(__fadd_rn(__uint2float_rn(lo), dt), P3);
    const float xh = __fmul_rn(d1, P1);
    const float xl = __fadd_rn(fmaf(d1, P2, fmaf(d1, P1, -xh)), y);
    // u = 1 - cos x = uh + ul; sin x - (its linear part) = ys
    const float hx = __fmul_rn(0.5f, xh);
    const float uh = __fmul_rn(hx, xh);
    const float ul = fmaf(uh, __fmul_rn(uh, -1.f / 6.f), fmaf(xh, xl, fmaf(hx, xh, -uh)));
    const float ys = fmaf(-uh, xl, fmaf(xh, __fmul_rn(uh, fmaf(uh, 1.f / 30.f, -1.f / 3.f)), y));
    const float ch = __int2float_rn(chi), sn = __int2float_rn(shi);     // units of 2^-23, exact
    const float uhs = __fmul_rn(uh, 2.3283064365386963e-10f);
    const float xhs = __fmul_rn(__fadd_rn(xh, xl), 2.3283064365386963e-10f);
    const float cl = __uint2float_rn(e.x), sl = __uint2float_rn(e.z);   // units of 2^-55
    a.c += (long long)(((unsigned long long)e.y << 32) | e.x);
    a.s += (long long)(((unsigned long long)e.w << 32) | e.z);
    a.lc += (long long)chi * sh;
    a.ls += (long long)shi * sh;
    // to subtract from cos: C u + S ys + Sl x; from sin: S u - C ys - Cl x: the halves of paired
    // instructions (14 for 28; 1.75 -> 1.57 ms with sixteen terms a turn)
    const float2 A = make_float2(ch, sn), B = make_float2(sn, -ch), D = make_float2(sl, -cl), m1 = make_float2(-1.f, -1.f);
    const float2 u2 = make_float2(uh, uh), y2 = make_float2(ys, ys), x2 = make_float2(xhs, xhs);
    const float2 g1 = __ffma2_rn(A, u2, make_float2(kFxMagic, kFxMagic));
    const float2 r1 = __ffma2_rn(A, u2, __ffma2_rn(g1, m1, make_float2(kFxMagic, kFxMagic)));
    const float2 g2 = __ffma2_rn(B, y2, g1), r2 = __ffma2_rn(B, y2, __ffma2_rn(g2, m1, g1));
    const float2 g3 = __ffma2_rn(D, x2, g2), r3 = __ffma2_rn(D, x2, __ffma2_rn(g3, m1, g2));
    a.gc += __float_as_uint(g3.x);
    a.gs += __float_as_uint(g3.y);
    const float2 t = __fadd2_rn(__fadd2_rn(__ffma2_rn(make_float2(cl, sl), make_float2(uhs, uhs),
                                                      __ffma2_rn(A, make_float2(ul, ul), r1)), r2), r3);
    a.f = __fadd2_rn(a.f, t);
}

// The sums of n atoms (npad of them padding: phase 0) in units of 2^-55.
__device__ __forceinline__ void fx_total(const FxSums& a, int n, int npad, long long& tc, long long& ts) {
    const long long k2pi = 0x1921fb54442d184ll;  // 2 pi 2^54: 2^-65 revolutions to 2^-55
    const unsigned off = (unsigned)n * __float_as_uint(kFxMagic);
    tc = a.c - ((long long)npad << 55) - __mul64hi(a.ls, k2pi) - ((long long)(int)(a.gc - off) << 16) -
         __float2ll_rn(a.f.x * 4294967296.f);
    ts = a.s + __mul64hi(a.lc, k2pi) - ((long long)(int)(a.gs - off) << 16) - __float2ll_rn(a.f.y * 4294967296.f);
}

__global__ void __launch_bounds__(kFxWarps * 32, 1) phase_fx_kernel(const FxLaunch a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {   // the table, eight copies
        const uint4* src = reinterpret_cast<const uint4*>(a.table);
        for (int i = threadIdx.x; i < kFxTable * 8; i += kFxWarps * 32)
            reinterpret_cast<uint4*>(smem)[i] = __ldg(src + (i >> 3));
    }
    __syncthreads();
    const unsigned char* tab = smem + (lane & 7) * 16;
    uint4* ri = reinterpret_cast<uint4*>(smem + kFxTableBytes + warp * kFxRecord);
    float4* rf = reinterpret_cast<float4*>(ri + 32);
    int4* rr = reinterpret_cast<int4*>(ri + 64);
    const long long nunits = (long long)a.ntiles * 8;

    for (;;) {
        unsigned unit = 0;
        if (lane == 0) unit = atomicAdd(a.counter, 1u);
        unit = __shfl_sync(0xffffffffu, unit, 0);
        if ((long long)unit >= nunits) break;
        const FxTileDesc td = a.tiles[unit >> 3];
        const FxSystem sys = a.systems[td.system];
        const int f = td.f0 + (int)(unit & 7);
        if (f >= sys.nf) continue;
        const int v = td.v0 + min(lane, td.nv - 1);
        int shell = 0;  // the q-vector's shell: largest with shell_v[shell] <= v
        for (int hi = sys.nshell; hi - shell > 1;) {
            const int mid = (shell + hi) >> 1;
            if (__ldg(sys.shell_v + mid) <= v) shell = mid;
            else hi = mid;
        }
        const double* cf = sys.cf + (size_t)shell * sys.nclass;
        const uint4* qw = sys.qw + 4 * (size_t)v;
        const bool qbad = __any_sync(0xffffffffu, __ldg(qw + 3).x != 0u);
        const float4* row = sys.xyz + (size_t)f * sys.na_pad;

        double re = 0.0, im = 0.0;
        FxSums sums;
        sums.clear();
        int n = 0, npad = 0, E = -1;
        FxQ q;
        int j = __ldg(sys.map + td.b_begin * 32 + lane);
        float4 r = j >= 0 ? __ldg(row + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        int info = __ldg(sys.block_info + td.b_begin);
        for (int b = td.b_begin; b < td.b_end; ++b) {
            const unsigned mx = __reduce_max_sync(
                0xffffffffu, max(max(__float_as_uint(fabsf(r.x)), __float_as_uint(fabsf(r.y))),
                                 __float_as_uint(fabsf(r.z))));
            const bool bad = qbad || mx >= kFxBig;
            bool resid = false;
            __syncwarp();
            if (bad) {
                rf[lane] = make_float4(r.x, r.y, r.z, j >= 0 ? 1.f : 0.f);
            } else {
                const int Eb = max(0, (int)(mx >> 23) - 126);
                if (Eb != E) {
                    E = Eb;
                    fx_shift_q(qw, E, q);
                }
                const float sc = __uint_as_float((unsigned)(127 + 31 - E) << 23);
                const float vx = r.x * sc, vy = r.y * sc, vz = r.z * sc;
                const int ix = __float2int_rn(vx), iy = __float2int_rn(vy), iz = __float2int_rn(vz);
                const float ex = vx - (float)ix, ey = vy - (float)iy, ez = vz - (float)iz;
                const bool mine = ex != 0.f || ey != 0.f || ez != 0.f;
                resid = __any_sync(0xffffffffu, mine);
                ri[lane] = make_uint4((unsigned)ix ^ 0x80000000u, (unsigned)iy ^ 0x80000000u,
                                      (unsigned)iz ^ 0x80000000u, mine ? 1u : 0u);
                rf[lane] = make_float4(vx, vy, vz, 0.f);
                if (resid)
                    rr[lane] = make_int4(__float2int_rn(ex * 4294967296.f), __float2int_rn(ey * 4294967296.f),
                                         __float2int_rn(ez * 4294967296.f), 0);
            }
            __syncwarp();
            const int cur = info;
            if (b + 1 < td.b_end) {  // the next block's atoms, in flight during this one
                j = __ldg(sys.map + (b + 1) * 32 + lane);
                info = __ldg(sys.block_info + b + 1);
                r = j >= 0 ? __ldg(row + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (bad) {
                // FP64, as the direct kernel evaluates it
                const double* qv = sys.qv + 3 * (size_t)v;
                const double qx = qv[0], qy = qv[1], qz = qv[2], bf = __ldg(cf + (cur & 0xffff));
                for (int jj = 0; jj < 32; ++jj) {
                    const float4 p = rf[jj];
                    if (p.w == 0.f) continue;
                    const double ph = __dadd_rn(__dadd_rn(__dmul_rn((double)p.x, qx), __dmul_rn((double)p.y, qy)),
                                                __dmul_rn((double)p.z, qz));
                    double s, c;
                    sincos(ph, &s, &c);
                    re = __dadd_rn(re, __dmul_rn(bf, c));
                    im = __dadd_rn(im, __dmul_rn(bf, s));
                }
            } else {
                n += 32;
                npad += cur >> 16;
#pragma unroll 16
                for (int jj = 0; jj < 32; ++jj) {
                    const uint4 R = ri[jj];
                    const float4 F = rf[jj];
                    unsigned long long ph = ((unsigned long long)q.hi0 << 32) | q.lo0;
                    ph += (unsigned long long)q.w1[0] * R.x;
                    ph += (unsigned long long)q.w1[1] * R.y;
                    ph += (unsigned long long)q.w1[2] * R.z;
                    unsigned lo = (unsigned)ph;
                    unsigned hi = (unsigned)(ph >> 32) + q.w2[0] * R.x + q.w2[1] * R.y + q.w2[2] * R.z;
                    const float dt = fmaf(q.w0[0], F.x, fmaf(q.w0[1], F.y, __fmul_rn(q.w0[2], F.z)));
                    if (resid && R.w) {  // coordinates with bits below the 32-bit grid (near 0)
                        const int4 t = rr[jj];
                        const int tt[3] = {t.x, t.y, t.z};
                        unsigned long long p = ((unsigned long long)hi << 32) | lo;
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            p += (unsigned long long)(((long long)q.w1[c] * tt[c] >> 32) +
                                                      (long long)(int)q.w2[c] * tt[c]);
                        hi = (unsigned)(p >> 32);
                        lo = (unsigned)p;
                    }
                    fx_term(hi, lo, dt, tab, sums);
                }
            }
            const bool last = b + 1 == td.b_end;
            if (n && (last || n >= 32 * kFxFold || (info & 0xffff) != (cur & 0xffff))) {
                long long tc, ts;
                fx_total(sums, n, npad, tc, ts);
                const double bf = __ldg(cf + (cur & 0xffff)) * 2.77555756156289135e-17;  // 2^-55
                re = fma(bf, (double)tc, re);
                im = fma(bf, (double)ts, im);
                sums.clear();
                n = npad = 0;
            }
        }
        if (lane < td.nv) sys.out[(size_t)td.split * sys.split_stride + (size_t)v * sys.nf + f] = make_double2(re, im);
    }
}

}  // namespace

cudaError_t launch_fx_table(void* table, cudaStream_t st) {
    fx_table_kernel<<<8, 128, 0, st>>>(reinterpret_cast<longlong2*>(table));
    return cudaGetLastError();
}

cudaError_t launch_fx_q(const double* qv, size_t nv, void* qw, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(qw, 0, nv * kFxQBytes, st);
    if (e != cudaSuccess) return e;
    fx_q_kernel<<<grid_blocks(3 * nv, 256, 8), 256, 0, st>>>(qv, nv, reinterpret_cast<uint4*>(qw));
    return cudaGetLastError();
}

cudaError_t launch_phase_fx(const FxLaunch& a, cudaStream_t st) {
    if (a.ntiles <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(phase_fx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFxSmem);
    if (e != cudaSuccess) return e;
    const long long need = ((long long)a.ntiles * 8 + kFxWarps - 1) / kFxWarps;
    const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(current_sms(), need));
    phase_fx_kernel<<<grid, kFxWarps * 32, kFxSmem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace sassgpu
