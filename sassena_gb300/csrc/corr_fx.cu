// Incoherent autocorrelation of the FP64 form in fixed point, padded lengths 64, 128 and 256.
//
// Each (atom, direction) pair has its own series exp(i q.r(t)), padded to L >= 2 NF points and
// transformed (SelfVectorsScatterDevice::scatter and dsp, self_vectors_scatter_device.cpp:288-322,
// smath.cpp:141-156). On GB300's FP64 pipe (19 clocks of an SM per warp instruction) a series of
// 256 points took 4,800 clocks of sincos and butterflies. Here a number is a 64-bit integer and the
// work runs on the integer and FP32 pipes:
//   * a point is cos and sin of a 64-bit phase in units of 2^-55, by the table and the short
//     series of the coherent sum (phase_fx.cu; the table in two copies here);
//   * the transform is exact in its additions; products with a twiddle in units of 2^-62 are three
//     32-bit multiplications each (the low halves' product, below 2^-60, is left out). Every partial
//     sum of a series of at most 128 unit terms fits: |X| <= 2^7 2^55;
//   * points are scaled so that a still atom's |X| is 2^62; powers |X|^2 are summed over a few
//     series in 64 bits and taken to FP64 times b^2 where the atom changes; the series' means
//     over lags, sum_k P_k K_k, are integers too, their squares FP64.
//
// The layout is that of the transposed register transform (L = 16 C, n = a + C b, k = k_b + 16 k_a):
// a lane generates column a of its series, runs the 16-point transform over b in registers, the
// warp transposes through shared memory and lanes run the C-point transforms over a. A warp's
// G = 32 / C series are directions of one atom; each warp walks a contiguous range of a chunk's
// (atom, direction) pairs. Constants are chosen at compile time.
//
// Measured on a GB300, 10^6 series of 256 points: 31.8 ms before, 2.7 ms here.
#include <algorithm>

#include "common.cuh"
#include "fx.cuh"
#include "kernels.h"

namespace sassgpu {

namespace {

typedef long long i64;
struct zi {
    i64 x, y;
};

constexpr int kCfxWarps = 12, kCfxThreads = kCfxWarps * 32, kCfxCopies = 2;  // copies of the sincos table

template <int LG>
struct CfxShape {
    static constexpr int L = 1 << LG, C = L / 16, G = 32 / C, RPL = G / 2, NF = L / 2;
    static constexpr int ROW = C + 1, SER = 16 * ROW;  // in zi: rows padded by one
    static constexpr int UP = 8 - LG;                  // points in units of 2^-(55 + UP)
    static constexpr int PS = 62 - 2 * LG;             // powers in units of 2^-PS, at most 2^60 a series
    static constexpr int FOLD = RPL > 1 ? (RPL > 2 ? 1 : 3) : 7;  // rounds whose powers fit 63 bits
    // shared memory in bytes: sincos table, twiddles, store kernel, then per warp tile, bins, frames
    static constexpr int kTab = 0, kTw = kTab + kFxTable * 16 * kCfxCopies, kK = kTw + L * 16, kRed = kK + L * 16;
    static constexpr int kTile = kRed + kCfxWarps * 32;
    static constexpr int kBins = kTile + kCfxWarps * G * SER * 16;
    static constexpr int kRec = kBins + kCfxWarps * L * 8;
    static constexpr int kBytes = kRec + kCfxWarps * NF * 32;
};

// w in units of 2^-62 as h 2^31 + 2 l, l of 30 bits
__host__ __device__ constexpr int w_hi(i64 w) { return (int)(w >> 31); }
__host__ __device__ constexpr int w_lo(i64 w) { return (int)((w & 0x7fffffff) >> 1); }
constexpr i64 kCos8 = 4260642322793532497ll;   // cos(pi / 8) 2^62
constexpr i64 kSin8 = 1764815834521887442ll;   // sin(pi / 8) 2^62
constexpr i64 kSqrtH = 3260954456333195553ll;  // sqrt(1 / 2) 2^62

__device__ __forceinline__ int z_hi(i64 v) { return (int)(v >> 31); }
__device__ __forceinline__ int z_lo(i64 v) { return (int)(((unsigned)v >> 1) & 0x3fffffffu); }

// a b + c. Written out: left to the compiler, sums of 32 x 32 -> 64-bit products cost about half as
// many instructions again (this kernel 3.7 ms instead of 2.7).
__device__ __forceinline__ i64 wide(int a, int b, i64 c) {
    i64 r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

// v w / 2^62 for |v| < 2^62, |w| < 2^62
__device__ __forceinline__ i64 smul(i64 v, int h, int l) {
    const int vh = z_hi(v), vl = z_lo(v);
    const i64 lo = wide(vh, l, wide(vl, h, 1 << 29));
    return wide(vh, h, lo >> 30);
}

__device__ __forceinline__ zi zmul(zi v, int ch, int cl, int sh, int sl) {
    const int xh = z_hi(v.x), xl = z_lo(v.x), yh = z_hi(v.y), yl = z_lo(v.y);
    const i64 rl = wide(xh, cl, wide(xl, ch, 0)) - wide(yh, sl, wide(yl, sh, -(1 << 29)));
    const i64 il = wide(xh, sl, wide(xl, sh, 0)) + wide(yh, cl, wide(yl, ch, 1 << 29));
    zi r;
    r.x = wide(xh, ch, 0) - wide(yh, sh, 0) + (rl >> 30);
    r.y = wide(xh, sh, 0) + wide(yh, ch, 0) + (il >> 30);
    return r;
}

// v W_16^J, W_16 = exp(-2 pi i / 16)
template <int J>
__device__ __forceinline__ zi zmul16(zi v) {
    constexpr int j = J & 15;
    if constexpr (j == 0) return v;
    else if constexpr (j == 4) return zi{v.y, -v.x};
    else if constexpr (j == 8) return zi{-v.x, -v.y};
    else if constexpr (j == 12) return zi{-v.y, v.x};
    else if constexpr ((j & 3) == 2) {
        const i64 s = smul(v.x + v.y, w_hi(kSqrtH), w_lo(kSqrtH)), d = smul(v.y - v.x, w_hi(kSqrtH), w_lo(kSqrtH));
        if constexpr (j == 2) return zi{s, d};
        else if constexpr (j == 6) return zi{d, -s};
        else if constexpr (j == 10) return zi{-s, -d};
        else return zi{-d, s};
    } else {
        // cos, sin of -2 pi j / 16
        constexpr int m = j & 7;
        constexpr i64 c0 = (m == 1) ? kCos8 : (m == 3) ? kSin8 : (m == 5) ? -kSin8 : -kCos8;
        constexpr i64 s0 = (m == 1 || m == 7) ? -kSin8 : -kCos8;
        constexpr i64 c = j < 8 ? c0 : -c0, s = j < 8 ? s0 : -s0;
        return zmul(v, w_hi(c), w_lo(c), w_hi(s), w_lo(s));
    }
}

__device__ __forceinline__ zi zadd(zi a, zi b) { return zi{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ zi zsub(zi a, zi b) { return zi{a.x - b.x, a.y - b.y}; }

// Radix-2 DIF stages of span H .. 1 over x[OFF .. OFF + N), bit-reversed order out.
template <int N, int OFF, int H, int M>
__device__ __forceinline__ void z_stage(zi (&x)[16]) {
    if constexpr (M < N) {
        if constexpr ((M & H) == 0) {
            const zi u = x[OFF + M], w = x[OFF + M + H];
            x[OFF + M] = zadd(u, w);
            x[OFF + M + H] = zmul16<(M & (H - 1)) * (8 / H)>(zsub(u, w));
        }
        z_stage<N, OFF, H, M + 1>(x);
    }
}
template <int N, int OFF, int H>
__device__ __forceinline__ void z_dif(zi (&x)[16]) {
    if constexpr (H >= 1) {
        z_stage<N, OFF, H, 0>(x);
        z_dif<N, OFF, H / 2>(x);
    }
}
template <int C, int RPL, int J = 0>
__device__ __forceinline__ void z_rows(zi (&x)[16]) {
    if constexpr (J < RPL) {
        z_dif<C, J * C, C / 2>(x);
        z_rows<C, RPL, J + 1>(x);
    }
}
template <int B = 0>
__device__ __forceinline__ void z_fold(zi (&x)[16]) {  // first stage, upper half zero
    if constexpr (B < 8) {
        x[B + 8] = zmul16<B>(x[B]);
        z_fold<B + 1>(x);
    }
}
__host__ __device__ constexpr int cfx_brev(int v, int bits) {
    return bits == 0 ? 0 : (((v & 1) << (bits - 1)) | cfx_brev(v >> 1, bits - 1));
}
template <int ROW, int P = 0>
__device__ __forceinline__ void z_store(zi* base, const zi (&x)[16]) {
    if constexpr (P < 16) {
        *reinterpret_cast<longlong2*>(base + cfx_brev(P, 4) * ROW) = make_longlong2(x[P].x, x[P].y);
        z_store<ROW, P + 1>(base, x);
    }
}

__device__ __forceinline__ int brev16(int p) { return (int)(__brev((unsigned)p) >> 28); }

// cos and sin of (phi + dt 2^-64) revolutions in units of 2^-55. As fx_term of the coherent sum,
// with the angle past the grid in radians: x = X 2^-39 + xr, X a 32-bit integer, so that the
// products with the table's upper halves are exact.
__device__ __forceinline__ zi fx_sincos(unsigned hi, unsigned lo, float dt, const unsigned char* __restrict__ tab) {
    const int D = (int)__funnelshift_l(lo, hi, 10);  // the angle in 2^-42 revolutions
    const uint4 e = *reinterpret_cast<const uint4*>(tab + ((hi + 0x200000u) >> 22) * (16 * kCfxCopies));
    const int chi = (int)e.y, shi = (int)e.w;
    constexpr double kX = 0.78539816339744830962 * 2147483648.0;  // 2 pi 2^-42 in 2^-39 radians, times 2^31
    constexpr int KX = (int)kX;
    const i64 pr = wide(D, KX, 0);
    const int X = (int)(pr >> 31);
    constexpr float F1 = (float)(1.0 / 1180591620717411303424.0);               // 2^-70
    constexpr float F2 = (float)((kX - (double)KX) / 1180591620717411303424.0);  // (kX - KX) 2^-70
    constexpr float F3 = (float)(6.283185307179586476925 / 18889465931478580854784.0);  // 2 pi 2^-74
    constexpr float F4 = (float)(6.283185307179586476925 / 18446744073709551616.0);     // 2 pi 2^-64
    const float xr = fmaf(__uint2float_rn((unsigned)pr & 0x7fffffffu), F1,
                          fmaf(__int2float_rn(D), F2, fmaf(__uint2float_rn(lo << 10), F3, __fmul_rn(dt, F4))));
    const float xh = __fmul_rn(__int2float_rn(X >> 8), 4.656612873077393e-10f);                // exact, 2^-31
    const float xl = fmaf(__int2float_rn(X & 255), 1.8189894035458565e-12f, xr);               // 2^-39
    const float hx = __fmul_rn(0.5f, xh);
    const float uh = __fmul_rn(hx, xh);
    const float ul = fmaf(uh, __fmul_rn(uh, -1.f / 6.f), fmaf(xh, xl, fmaf(hx, xh, -uh)));
    const float ys = fmaf(-uh, xl, fmaf(xh, __fmul_rn(uh, fmaf(uh, 1.f / 30.f, -1.f / 3.f)), xr));
    const float ch = __int2float_rn(chi), sn = __int2float_rn(shi);  // units of 2^-23
    const float uhs = __fmul_rn(uh, 2.3283064365386963e-10f);
    const float xhs = __fmul_rn(__fadd_rn(xh, xl), 2.3283064365386963e-10f);
    const float cl = __uint2float_rn(e.x), sl = __uint2float_rn(e.z);  // units of 2^-55
    constexpr float M = 192.f;
    // what is taken off cos: C u + S ys + Sl x; off sin: S u - C ys - Cl x
    auto rest = [&](float a, float al, float b, float bl) {
        const float g1 = fmaf(a, uh, M), r1 = fmaf(a, uh, __fsub_rn(M, g1));
        const float g2 = fmaf(b, ys, g1), r2 = fmaf(b, ys, __fsub_rn(g1, g2));
        const float g3 = fmaf(bl, xhs, g2), r3 = fmaf(bl, xhs, __fsub_rn(g2, g3));
        const float f = __fadd_rn(__fadd_rn(fmaf(al, uhs, fmaf(a, ul, r1)), r2), r3);
        const int lo55 = __float_as_int(fmaf(f, 4294967296.f, 12582912.f)) - 0x4B400000;
        return ((i64)(__float_as_int(g3) - __float_as_int(M)) << 16) + lo55;
    };
    zi r;
    r.x = (i64)(((unsigned long long)e.y << 32) | e.x) - (wide(shi, X, 0) >> 7) - rest(ch, cl, sn, sl);
    r.y = (i64)(((unsigned long long)e.w << 32) | e.z) + (wide(chi, X, 0) >> 7) - rest(sn, sl, -ch, -cl);
    return r;
}

// The same outside the fixed-point range, in FP64 as the FP64 kernels evaluate it.
__device__ __noinline__ zi fp64_sincos(float x, float y, float z, const double* __restrict__ q, bool& poison) {
    const double p = __dadd_rn(__dadd_rn(__dmul_rn((double)x, q[0]), __dmul_rn((double)y, q[1])),
                               __dmul_rn((double)z, q[2]));
    double s, c;
    sincos(p, &s, &c);
    if (!isfinite(p)) poison = true;
    return zi{__double2ll_rn(c * 36028797018963968.0), __double2ll_rn(s * 36028797018963968.0)};
}

template <int LG>
__global__ void __launch_bounds__(kCfxThreads, 1) self_fx_kernel(CorrLaunch a) {
    typedef CfxShape<LG> Sh;
    constexpr int L = Sh::L, C = Sh::C, G = Sh::G, RPL = Sh::RPL, BC = LG - 4;
    extern __shared__ __align__(128) unsigned char smem[];
    const CorrChunk c = a.chunks[blockIdx.x];
    const CorrSystem sys = a.systems[c.system];
    const int nf = sys.nf, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int4* ttab = reinterpret_cast<int4*>(smem + Sh::kTw);  // [p][col]: W_L^{col br16(p)} as split words
    int4* ktab = reinterpret_cast<int4*>(smem + Sh::kK);   // [q][k_b]: K of bin k_b + 16 br(q)
    zi* tile = reinterpret_cast<zi*>(smem + Sh::kTile) + warp * G * Sh::SER;
    double* bins = reinterpret_cast<double*>(smem + Sh::kBins) + warp * L;
    uint4* rec = reinterpret_cast<uint4*>(smem + Sh::kRec) + warp * Sh::NF * 2;
    // K in units of 2^-kk: |K| <= 8 / (NF L)
    const int kk = 58 + LG + (31 - __clz(nf));
    {
        const longlong2* src = reinterpret_cast<const longlong2*>(a.fx_table);
        for (int i = threadIdx.x; i < kFxTable * kCfxCopies; i += kCfxThreads)
            reinterpret_cast<longlong2*>(smem + Sh::kTab)[i] = src[i / kCfxCopies];
        for (int i = threadIdx.x; i < L; i += kCfxThreads) {
            const int p = i / C, m = (i - p * C) * brev16(p);
            const longlong2 t = src[((m & (L - 1)) * (kFxTable / L)) & (kFxTable - 1)];
            // W^m = cos - i sin, 2^-55 to 2^-62, kept below 1
            const i64 lim = (1ll << 62) - 2;
            const i64 wc = min(max(t.x << 7, -lim), lim), ws = min(max(-t.y << 7, -lim), lim);
            ttab[i] = make_int4(w_hi(wc), w_lo(wc), w_hi(ws), w_lo(ws));
            const int q = i >> 4, k = (i & 15) + 16 * (int)(BC ? __brev((unsigned)q) >> (32 - BC) : 0);
            const double2 kv = reinterpret_cast<const double2*>(sys.kbr)[__brev((unsigned)k) >> (32 - LG)];
            const i64 kr = __double2ll_rn(ldexp(kv.x, kk)), ki = __double2ll_rn(ldexp(kv.y, kk));
            // low words around 0, so that the products left out have no bias
            const i64 rh = (kr + 0x80000000ll) >> 32, ih = (ki + 0x80000000ll) >> 32;
            ktab[i] = make_int4((int)rh, (int)(kr - (rh << 32)) >> 2, (int)ih, (int)(ki - (ih << 32)) >> 2);
        }
        for (int i = lane; i < L; i += 32) bins[i] = 0.0;
    }
    __syncthreads();
    const unsigned char* tab = smem + Sh::kTab + lane % kCfxCopies * 16;
    const int g1 = lane / C, col = lane - g1 * C, kb = lane & 15, half = lane >> 4;

    i64 pacc[C], msx = 0, msy = 0;  // sums of powers (2^-PS) and of means (2^-(PS + kk - 64))
    double ms2 = 0.0;               // sum of the means' squared moduli
#pragma unroll
    for (int q = 0; q < C; ++q) pacc[q] = 0;
    double dsx = 0.0, dsy = 0.0, ds2 = 0.0;
    bool poison = false;
    int rounds = 0;
    // the integer sums, times b^2, to FP64: each half warp takes half of the bins
    auto fold = [&](double w2) {
        const double wp = w2 * (2.0 / (double)(1ll << Sh::PS));
#pragma unroll
        for (int q = 0; q < C / 2; ++q) {
            i64 t0 = pacc[q] >> 1, t1 = pacc[q + C / 2] >> 1;  // half: both half warps' sums fit
            t0 += __shfl_xor_sync(0xffffffffu, t0, 16);
            t1 += __shfl_xor_sync(0xffffffffu, t1, 16);
            pacc[q] = pacc[q + C / 2] = 0;
            const int k = kb + 16 * (half ? cfx_brev(q + C / 2, BC) : cfx_brev(q, BC));
            bins[k] = fma(wp, (double)(half ? t1 : t0), bins[k]);
        }
        dsx = fma(w2, (double)msx, dsx);
        dsy = fma(w2, (double)msy, dsy);
        ds2 = fma(w2 * w2, ms2, ds2);
        msx = msy = 0;
        ms2 = 0.0;
        rounds = 0;
    };

    const int v0 = sys.shell_v[c.shell], nd = sys.shell_v[c.shell + 1] - v0;
    const double* bfac = reinterpret_cast<const double*>(sys.bfac) + (size_t)c.shell * sys.na_pad;
    const i64 npair = (i64)(c.v_end - c.v_begin) * nd;
    const i64 pend = npair * (warp + 1) / kCfxWarps;
    i64 pr = npair * warp / kCfxWarps;
    int at = (int)(pr / nd), d0 = (int)(pr - (i64)at * nd);
    while (pr < pend) {
        const int j = c.v_begin + at, dn = (int)min((i64)nd, d0 + (pend - pr));  // directions [d0, dn) of atom j
        const double b = bfac[j], w2 = b * b;
        // the atom's trajectory as fixed-point records: coordinates (offset 2^31) and flag, residuals
        float4 r[L / 64];
        unsigned mx = 0;
#pragma unroll
        for (int i = 0; i < L / 64; ++i) {
            const int t = lane + 32 * i;
            r[i] = t < nf ? sys.xyz[(size_t)t * sys.na_pad + j] : make_float4(0.f, 0.f, 0.f, 0.f);
            mx = max(mx, max(max(__float_as_uint(fabsf(r[i].x)), __float_as_uint(fabsf(r[i].y))),
                             __float_as_uint(fabsf(r[i].z))));
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        const bool bad = mx >= kFxBig;
        const int E = bad ? 0 : max(0, (int)(mx >> 23) - 126);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < L / 64; ++i) {
            const int t = lane + 32 * i;
            if (bad) {
                rec[t * 2] = make_uint4(__float_as_uint(r[i].x), __float_as_uint(r[i].y), __float_as_uint(r[i].z), 0u);
                continue;
            }
            const float sc = __uint_as_float((unsigned)(127 + 31 - E) << 23);
            const float vx = r[i].x * sc, vy = r[i].y * sc, vz = r[i].z * sc;
            const int ix = __float2int_rn(vx), iy = __float2int_rn(vy), iz = __float2int_rn(vz);
            const float ex = vx - (float)ix, ey = vy - (float)iy, ez = vz - (float)iz;
            const bool some = ex != 0.f || ey != 0.f || ez != 0.f;
            rec[t * 2] = make_uint4((unsigned)ix ^ 0x80000000u, (unsigned)iy ^ 0x80000000u, (unsigned)iz ^ 0x80000000u,
                                    some ? 1u : 0u);
            rec[t * 2 + 1] = make_uint4((unsigned)__float2int_rn(ex * 4294967296.f),
                                        (unsigned)__float2int_rn(ey * 4294967296.f),
                                        (unsigned)__float2int_rn(ez * 4294967296.f), 0u);
        }
        __syncwarp();
        for (int d = d0; d < dn; d += G) {
            const bool ok = d + g1 < dn;
            const int v = v0 + (ok ? d + g1 : d);
            const uint4* qw = reinterpret_cast<const uint4*>(sys.qw) + 4 * (size_t)v;
            const bool slow = bad || __any_sync(0xffffffffu, __ldg(qw + 3).x != 0u);
            // the lane's eight points, through its own slots of the tile: a rolled loop (eight copies
            // of the point's code missed the instruction cache)
            longlong2* mine = reinterpret_cast<longlong2*>(tile) + lane;
            __syncwarp();  // the previous round's rows have been read
            if (slow) {
#pragma unroll 1
                for (int bb = 0; bb < 8; ++bb) {
                    const int n = col + C * bb;
                    zi z{0, 0};
                    if (ok && n < nf) {
                        const float4 p = sys.xyz[(size_t)n * sys.na_pad + j];
                        z = fp64_sincos(p.x, p.y, p.z, sys.qv + 3 * (size_t)v, poison);
                    }
                    mine[bb * 32] = make_longlong2(z.x << Sh::UP, z.y << Sh::UP);
                }
            } else {
                FxQ q;
                fx_shift_q(qw, E, q);
#pragma unroll 2
                for (int bb = 0; bb < 8; ++bb) {
                    const int n = col + C * bb;
                    const uint4 R = rec[n * 2];
                    unsigned long long ph = ((unsigned long long)q.hi0 << 32) | q.lo0;
                    ph += (unsigned long long)q.w1[0] * R.x;
                    ph += (unsigned long long)q.w1[1] * R.y;
                    ph += (unsigned long long)q.w1[2] * R.z;
                    unsigned lo = (unsigned)ph;
                    unsigned hi = (unsigned)(ph >> 32) + q.w2[0] * R.x + q.w2[1] * R.y + q.w2[2] * R.z;
                    const float dt = fmaf(q.w0[0], __int2float_rn((int)(R.x ^ 0x80000000u)),
                                          fmaf(q.w0[1], __int2float_rn((int)(R.y ^ 0x80000000u)),
                                               __fmul_rn(q.w0[2], __int2float_rn((int)(R.z ^ 0x80000000u)))));
                    if (R.w) {  // coordinates with bits below the 32-bit grid
                        const uint4 t = rec[n * 2 + 1];
                        const int tt[3] = {(int)t.x, (int)t.y, (int)t.z};
                        unsigned long long p = ((unsigned long long)hi << 32) | lo;
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                            p += (unsigned long long)(((i64)q.w1[k] * tt[k] >> 32) + (i64)(int)q.w2[k] * tt[k]);
                        hi = (unsigned)(p >> 32);
                        lo = (unsigned)p;
                    }
                    const zi z = fx_sincos(hi, lo, dt, tab);
                    const bool in = ok && n < nf;
                    mine[bb * 32] = make_longlong2(in ? z.x << Sh::UP : 0, in ? z.y << Sh::UP : 0);
                }
            }
            zi x[16];
#pragma unroll
            for (int bb = 0; bb < 8; ++bb) {
                const longlong2 t = mine[bb * 32];
                x[bb] = zi{t.x, t.y};
            }
            z_fold(x);
            z_dif<16, 0, 4>(x);
#pragma unroll
            for (int p = 1; p < 16; ++p) {  // times W_L^{col k_b}, k_b = br16(p)
                const int4 w = ttab[p * C + col];
                x[p] = zmul(x[p], w.x, w.y, w.z, w.w);
            }
            __syncwarp();  // every lane has read its points
            z_store<Sh::ROW>(tile + g1 * Sh::SER + col, x);
            __syncwarp();
#pragma unroll
            for (int jj = 0; jj < RPL; ++jj) {
                const zi* row = tile + (half + 2 * jj) * Sh::SER + kb * Sh::ROW;
#pragma unroll
                for (int q = 0; q < C; ++q) {
                    const longlong2 t = *reinterpret_cast<const longlong2*>(row + q);
                    x[jj * C + q] = zi{t.x, t.y};
                }
            }
            z_rows<C, RPL>(x);
            // powers of the lane's bins and each series' sum of P K
            i64 sx[RPL], sy[RPL], tx[RPL], ty[RPL];  // (s + t 2^-8): high and cross products
#pragma unroll
            for (int jj = 0; jj < RPL; ++jj) sx[jj] = sy[jj] = tx[jj] = ty[jj] = 0;
#pragma unroll
            for (int q = 0; q < C; ++q) {
                const int4 kv = ktab[q * 16 + kb];
#pragma unroll
                for (int jj = 0; jj < RPL; ++jj) {
                    const zi z = x[jj * C + q];
                    const int zh = (int)(z.x >> 32), yh = (int)(z.y >> 32);
                    const i64 cross = wide(zh, (int)((unsigned)z.x >> 1), wide(yh, (int)((unsigned)z.y >> 1), 1 << 29));
                    const i64 P = wide(zh, zh, wide(yh, yh, cross >> 30));  // (x^2 + y^2) 2^-64
                    pacc[q] += P;
                    const int ph = (int)(P >> 32), pl = (int)((unsigned)P >> 2);
                    sx[jj] = wide(ph, kv.x, sx[jj]);
                    sy[jj] = wide(ph, kv.z, sy[jj]);
                    tx[jj] += wide(ph, kv.y, wide(pl, kv.x, 0)) >> 22;
                    ty[jj] += wide(ph, kv.w, wide(pl, kv.z, 0)) >> 22;
                }
            }
#pragma unroll
            for (int jj = 0; jj < RPL; ++jj) {
                i64 mx = sx[jj] + (tx[jj] >> 8), my = sy[jj] + (ty[jj] >> 8);
#pragma unroll
                for (int o = 8; o >= 1; o >>= 1) {  // within the half warp: the series' total
                    mx += __shfl_xor_sync(0xffffffffu, mx, o);
                    my += __shfl_xor_sync(0xffffffffu, my, o);
                }
                msx += mx;
                msy += my;
                const double fx = (double)mx, fy = (double)my;
                ms2 = fma(fx, fx, fma(fy, fy, ms2));
            }
            if (++rounds == Sh::FOLD) fold(w2);
        }
        fold(w2);
        pr += dn - d0;
        d0 = 0;
        ++at;
    }

    // the warps' bins, then the chunk's partial slot in bit-reversed order
    double2* red = reinterpret_cast<double2*>(smem + Sh::kRed);
    double* red2 = reinterpret_cast<double*>(red + kCfxWarps);
    const double es = ldexp(1.0, 64 - Sh::PS - kk), e2 = es * es;
    dsx += __shfl_xor_sync(0xffffffffu, dsx, 16);
    dsy += __shfl_xor_sync(0xffffffffu, dsy, 16);
    ds2 += __shfl_xor_sync(0xffffffffu, ds2, 16);
    if (lane == 0) {
        red[warp] = make_double2(dsx * es, dsy * es);
        red2[warp] = ds2 * e2;
    }
    const double nan_or_0 = __syncthreads_or(poison) ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
    const double* all = reinterpret_cast<const double*>(smem + Sh::kBins);
    double* dst = a.ppart + c.part_off;
    for (int k = threadIdx.x; k < L; k += kCfxThreads) {
        double s = nan_or_0;
        for (int w = 0; w < kCfxWarps; ++w) s += all[w * L + k];
        dst[__brev((unsigned)k) >> (32 - LG)] = s;
    }
    if (threadIdx.x == 0) {
        double2 as = make_double2(nan_or_0, nan_or_0);
        double a2 = nan_or_0;
        for (int w = 0; w < kCfxWarps; ++w) {
            as.x += red[w].x;
            as.y += red[w].y;
            a2 += red2[w];
        }
        a.apart[c.slot] = as;
        a.a2part[c.slot] = a2;
    }
}

template <int LG>
cudaError_t launch_lg(const CorrLaunch& a, cudaStream_t st) {
    const int sm = CfxShape<LG>::kBytes;
    cudaError_t e = cudaFuncSetAttribute(self_fx_kernel<LG>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    self_fx_kernel<LG><<<a.nchunks, kCfxThreads, sm, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

bool self_fx_supported(int precision, int dsp, int lg_min, int lg_max) {
    return precision == PREC_FP64 && dsp == DSP_AUTOCORRELATE && lg_min == lg_max && lg_max >= 6 && lg_max <= 8;
}

cudaError_t launch_self_fx(const CorrLaunch& a, cudaStream_t st) {
    if (a.nchunks == 0) return cudaSuccess;
    switch (a.lg_max) {
        case 6: return launch_lg<6>(a, st);
        case 7: return launch_lg<7>(a, st);
        case 8: return launch_lg<8>(a, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace sassgpu
