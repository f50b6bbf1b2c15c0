// Multipole orientational averages (coherent, FP64 form).
//
// Replaces MPSphereScatterDevice and MPCylinderScatterDevice
// (src/scatter_devices/multipole_scatter_device.cpp). Per q and per moment (l, m) the
// reference sums over atoms, for every frame:
//   sphere   A_lm(t) = sum_j 4 pi i^l b_j j_l(|q| r_j) conj(Y_l^m(theta_j, phi_j))   (:428-497)
//   cylinder A_lm(t) = sqrt(2 pi) sum_j b_j exp(i s z_j q_z) c_lm J_n(q_r r_j) T_m(n (phi_j - phi_q))
//            with n = 2l (m = 0, 1: T = cos, sin) or 2l - 1 (m = 2, 3), c = sqrt(1/2) 2 (-1)^l or
//            i sqrt(1/2) 2 (-1)^(l-1), (l, m) = (0, 0): J_0, and s the sign of z q_z  (:900-986)
// then correlates each moment like the vectors devices and scales the sum by 1/(4 pi)
// (sphere, :396-400) or 1/(2 pi) (cylinder, :865-870). Coordinates are in the spherical or
// cylindrical representation the reference stages (coordinate_sets.cpp:359-363), converted
// here on the device from the staged Cartesian frames in FP64 and rounded to float as the
// reference's float staging does (data_stager.cpp:110-114).
//
// GB300 layout.
//   sphere: the sum over atoms is, for one frame and one l, a product of the matrix
//     b_j(q) j_l(|q| r_j) [q x atom] with conj(Y_l^m(j)) [atom x m]. Basis kernels write both
//     factors for a batch of frames to HBM (every Y_l^m with m >= 0 once, not once per q, in
//     fixed point); a contraction kernel sums every (q, m) output of one (frame, l) in integers.
//     Where the amplitudes of a (frame, q) are so small beside the bounds of both factors that the
//     integers' digits do not reach them, the same sums are taken again in FP64 (MpRedo below).
//   cylinder: basis kernels write J_n(q_r r) for every order n <= 2L, X = b exp(i s z q_z), and
//     cos(n phi), sin(n phi) of a batch of frames; a contraction kernel sums X_j J_n cos(n phi_j)
//     and ... sin(n phi_j) over atoms in integers; each moment is formed from them with
//     cos(n phi_q), sin(n phi_q).
// The special functions are this project's own FP64 implementations (Boost, which the
// reference calls, is not used): spherical Bessel functions by power series, upward
// recurrence where stable or Miller's downward recurrence; normalised associated Legendre
// functions by the standard three-term recurrences; cylinder Bessel functions by Hankel's
// asymptotic expansion plus upward recurrence for large arguments, Miller's algorithm
// otherwise. The amplitudes then go through the engine's correlation and average.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "engine.h"
#include "kernels.h"
#include "plan.h"

namespace sassgpu {

namespace {

constexpr int kMpMaxL = 40;  // largest major moment (sphere) / half order (cylinder)

// ---------------------------------------------------------------------------------------
// coordinate representations
// ---------------------------------------------------------------------------------------
// SphericalCoor3D(CartesianCoor3D), coor3d.cpp:168-215 -> (r, phi, theta) as float.
__device__ float4 to_spherical(float xf, float yf, float zf) {
    const double x = xf, y = yf, z = zf;
    const double r = sqrt(x * x + y * y + z * z);  // squares of float values are exact
    double theta = 0, phi = 0;
    if (r != 0) {
        theta = acos(z / r);
        if (x != 0.0) {
            phi = atan(y / x);
            if (x < 0.0) phi += 3.14159265358979323846;
            else if (y < 0.0) phi += 2 * 3.14159265358979323846;
        } else if (y != 0.0) {
            if (y > 0) phi = 1.57079632679489661923;
            if (y < 0) phi = 3 * 1.57079632679489661923;
        }
    }
    return make_float4((float)r, (float)phi, (float)theta, 0.f);
}

// CylinderCoor3D(CartesianCoor3D) of the projected vector, coor3d.cpp:116-141, with the
// reference's float sign() for the x < 0 branch.
__host__ __device__ inline void to_cylinder(double x, double y, double z, double& r, double& phi, double& zz) {
    r = sqrt(x * x + y * y);
    const double kPi = 3.14159265358979323846, kPi2 = 1.57079632679489661923;
    if (x != 0.0) {
        phi = atan(y / x);
        if (x < 0.0) phi = (double)((float)y < 0.0f ? -(float)kPi : (float)kPi) + phi;
    } else if (y != 0.0) {
        phi = (double)((float)y < 0.0f ? -(float)kPi2 : (float)kPi2);
    } else {
        phi = 0.0;
    }
    phi = phi < 0 ? 2 * kPi + phi : phi;
    zz = z;
}

struct MpBase {
    double e[9];  // e_r, e_phi, e_z of CartesianVectorBase(axis), coor3d.cpp:278-295
};

// Spherical (r, phi, theta, class) or cylindrical (r, phi, z, class) of atom j at slot[j] of
// its frame row (padding slots: class -1).
__global__ void mp_convert_kernel(const float4* __restrict__ xyz, int na_pad, int na, int nf, int cylinder,
                                  MpBase b, const int* __restrict__ slot, const int* __restrict__ cls,
                                  float4* __restrict__ out) {
    const size_t n = (size_t)nf * na_pad;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(i % na_pad);
        if (j >= na) {
            out[i] = make_float4(0.f, 0.f, 0.f, -1.f);
            continue;
        }
        const float4 c = xyz[i];
        if (!cylinder) {
            float4 v = to_spherical(c.x, c.y, c.z);
            v.w = (float)cls[j];
            out[(i - j) + slot[j]] = v;
        } else {
            const double x = c.x, y = c.y, z = c.z;
            const double px = x * b.e[0] + y * b.e[1] + z * b.e[2];
            const double py = x * b.e[3] + y * b.e[4] + z * b.e[5];
            const double pz = x * b.e[6] + y * b.e[7] + z * b.e[8];
            double r, phi, zz;
            to_cylinder(px, py, pz, r, phi, zz);
            out[(i - j) + slot[j]] = make_float4((float)r, (float)phi, (float)zz, (float)cls[j]);
        }
    }
}

// ---------------------------------------------------------------------------------------
// special functions (FP64)
// ---------------------------------------------------------------------------------------
// Per CTA in shared memory: 2 n + 1 and 1 / (2 n + 1), 1 / n (a conversion or a division holds the
// FP64 pipe as long as one or a dozen FMAs).
constexpr int kJlTab = kMpMaxL + 48;
struct JlTab {
    double odd[kJlTab], iodd[kJlTab], inv[kJlTab];
};

// b * j_l(x) for l = 0..L written to out[l * stride].
__device__ void sph_bessel_row(int L, double x, double b, double* out, size_t stride, const JlTab& t) {
    if (x == 0) {
        out[0] = b;
        for (int l = 1; l <= L; ++l) out[l * stride] = 0;
        return;
    }
    if (x < 0.5) {  // power series
        double xl = b;
        const double x2 = -0.5 * x * x;
        for (int l = 0; l <= L; ++l) {
            if (l > 0) xl *= x * t.iodd[l];
            double term = 1, sum = 1;
            for (int k = 1; k < 40; ++k) {
                term *= x2 * t.inv[k] * t.iodd[l + k];
                sum += term;
                // below 2^-60 of the sum
                if ((__double2hiint(term) & 0x7fffffff) + (60 << 20) < (__double2hiint(sum) & 0x7fffffff)) break;
            }
            out[l * stride] = xl * sum;
        }
        return;
    }
    const double ix = 1.0 / x;
    double sx, cx;
    sincos(x, &sx, &cx);
    const double j0 = sx * ix, j1 = (sx * ix - cx) * ix;
    if (x > L) {  // upward recurrence, stable for every l < x
        double jm = b * j0, jc = b * j1;
        out[0] = jm;
        if (L >= 1) out[stride] = jc;
        for (int l = 1; l < L; ++l) {
            const double jn = t.odd[l] * ix * jc - jm;
            out[(l + 1) * stride] = jn;
            jm = jc;
            jc = jn;
        }
        return;
    }
    // Miller's downward recurrence, normalised by j_0 or j_1. It starts at the order N where
    // the ratios j_n / j_{n-1} < x / (2 n + 1 - x) (n > L >= x) have multiplied to 2^-32: the
    // square of that is what the start at (1, 0) leaves of the second solution.
    int N = L;
    for (float p = 1.f, xf = (float)x; p > 2.3e-10f && N < L + 32;) {
        ++N;
        p *= __fdividef(xf, (float)(2 * N + 1) - xf);
    }
    double fp = 0, f = 1e-250;
    for (int n = N; n >= 1; --n) {
        const double fm = t.odd[n] * ix * f - fp;
        fp = f;
        f = fm;
        if (n - 1 <= L) out[(n - 1) * stride] = f;
        if ((__double2hiint(f) & 0x7fffffff) > 0x69800000) {  // 2^665
            for (int l = n - 1; l <= L; ++l) out[l * stride] *= 1e-200;
            fp *= 1e-200;
            f *= 1e-200;
        }
    }
    const double scale = b * (fabs(j0) >= fabs(j1) ? j0 / out[0] : j1 / out[stride]);
    for (int l = 0; l <= L; ++l) out[l * stride] *= scale;
}

// The normalised associated Legendre functions as P_l^m = g_lm y_lm with
//   y_lm = al_lm x y_{l-1,m} - y_{l-2,m}, y_mm = P_mm, y_{m+1,m} = x P_mm
// (two FP64 instructions a step instead of three; the factors g_lm, 0.5 to 9, are applied to the
// sums over atoms): from P_l = a_l (x P_{l-1} - b_l P_{l-2}), a = sqrt((4l^2 - 1)/(l^2 - m^2)),
// b = sqrt(((l-1)^2 - m^2)/(4 (l-1)^2 - 1)), g_l = a_l b_l g_{l-2} and al_l = a_l g_{l-1} / g_l.
// Per (l, m) with m <= l, i = (l (l + 1)) / 2 + m: al[i], g[i], and ex[i] with |y_lm| < 2^ex from
// |P_l^m| <= sqrt((2l + 1) / 4 pi); the seeds per m: sd[m] = -sqrt((2m + 1)/(2m)).
struct MpLegendre {
    double *al, *g, *sd;
    int* ex;
};
__host__ __device__ inline size_t legendre_bytes(int L) {
    return (size_t)((L + 1) * (L + 2) + L + 1) * sizeof(double) + (size_t)(L + 1) * (L + 2) / 2 * sizeof(int);
}
__host__ __device__ inline MpLegendre legendre_at(void* p, int L) {
    MpLegendre t;
    const int n = (L + 1) * (L + 2) / 2;
    t.al = static_cast<double*>(p);
    t.g = t.al + n;
    t.sd = t.g + n;
    t.ex = reinterpret_cast<int*>(t.sd + L + 1);
    return t;
}
__global__ void ylm_coeff_kernel(int L, MpLegendre t) {
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m <= L; m += gridDim.x * blockDim.x) {
        t.sd[m] = m > 0 ? -sqrt((2.0 * m + 1) / (2.0 * m)) : 0.0;
        double g2 = 1, g1 = sqrt(2.0 * m + 3);
        for (int l = m; l <= L; ++l) {
            const int i = l * (l + 1) / 2 + m;
            double g = l == m ? 1.0 : g1, al = 1.0;
            if (l >= m + 2) {
                const double a = sqrt((4.0 * l * l - 1) / ((double)l * l - (double)m * m));
                const double b = sqrt((((double)l - 1) * (l - 1) - (double)m * m) / (4.0 * (l - 1) * (l - 1) - 1));
                g = a * b * g2;
                al = a * g1 / g;
                g2 = g1;
                g1 = g;
            }
            t.al[i] = al;
            t.g[i] = g;
            t.ex[i] = (int)ceil(log2(sqrt((2.0 * l + 1) / (4 * 3.14159265358979323846)) / g * 1.0000001));
        }
    }
}

// v in units of 2^(E - 58), |v| < 2^E
__device__ __forceinline__ long long mp_fixed(double v, int E) {
    const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff;
    const unsigned long long m =
        ((((unsigned long long)((hi & 0xfffff) | (e ? 0x100000 : 0))) << 32) | (unsigned)__double2loint(v)) << 5;
    const long long t = (long long)(m >> min(max(E + 1022 - e, 0), 63));
    const long long sg = (long long)(hi >> 31);
    return (t ^ sg) - sg;
}
// Fixed-point numbers of the contractions: v = (h 2^29 + l) 2^(E - 57), l in [-2^28, 2^28). Rounded to
// nearest: cut off, a column of terms of one sign would lose half a unit each.
__device__ __forceinline__ int2 mp_words(double v, int E) {
    const long long t = mp_fixed(v, E);
    const int h = (int)((t + (1ll << 29) + 1) >> 30);
    return make_int2(h, (int)((unsigned)t + 1u - ((unsigned)h << 30)) >> 1);
}
__device__ __forceinline__ int2 mp_split(long long t) {
    const int h = (int)((t + (1ll << 28)) >> 29);
    return make_int2(h, (int)((unsigned)t - ((unsigned)h << 29)));
}
// a b + c. Written out: of the forms of a sum of products this one keeps both integer pipes busy
// (the contraction 1.12 ms; 1.38 as the compiler takes plain C).
__device__ __forceinline__ long long mp_wide(int a, int b, long long c) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
// a b / 2^57
__device__ __forceinline__ long long mp_mul(int2 a, int2 b) {
    return 2 * mp_wide(a.x, b.x, 0) + (mp_wide(a.x, b.y, mp_wide(a.y, b.x, 1ll << 27)) >> 28);
}
// |v| <= 1 (or rounded above it) in units of 2^-57
__device__ __forceinline__ int2 mp_unit(double v) {
    return mp_split(min(max(mp_fixed(v, 1), -(1ll << 57)), 1ll << 57));
}

// conj(Y_l^m(theta, phi)) / g_lm, m >= 0, for the requested pairs (idx[l (L+1) + m] -> pair, or -1)
// written to out[k * stride] as fixed-point words (re, im) or, with FIXED false, as a double2; m
// outer, l inner, so the Legendre recurrence carries two values. e^{i m phi} by rotation (m
// multiplications of e^{i phi}); its products with the Legendre functions are integers (the FP64 pipe
// is the bound here).
template <bool FIXED>
__device__ void conj_ylm_row(int L, double theta, double phi, const int* __restrict__ idx,
                             const MpLegendre& t, int4* out, size_t stride) {
    const double x = cos(theta), s = sqrt((1 - x) * (1 + x));
    double pmm = sqrt(1.0 / (4 * 3.14159265358979323846));
    double s1, c1;
    sincos(phi, &s1, &c1);
    double cm = 1.0, sm = 0.0;
    for (int m = 0; m <= L; ++m) {
        if (m > 0) {
            pmm = t.sd[m] * s * pmm;
            const double cn = cm * c1 - sm * s1;
            sm = sm * c1 + cm * s1;
            cm = cn;
        }
        const int2 ci = mp_unit(cm), si = mp_unit(sm);
        auto emit = [&](int l, double P) {
            const int k = idx[l * (L + 1) + m];
            if (k < 0) return;
            if constexpr (!FIXED) {
                reinterpret_cast<double2*>(out)[k * stride] = make_double2(P * cm, -P * sm);
                return;
            }
            const int2 pi = mp_words(P, t.ex[l * (l + 1) / 2 + m]);
            const int2 re = mp_split(mp_mul(pi, ci)), im = mp_split(-mp_mul(pi, si));
            out[k * stride] = make_int4(re.x, re.y, im.x, im.y);
        };
        emit(m, pmm);
        if (m < L) {
            double p2 = pmm, p1 = x * pmm;
            emit(m + 1, p1);
            for (int l = m + 2; l <= L; ++l) {
                const double p = t.al[l * (l + 1) / 2 + m] * x * p1 - p2;
                emit(l, p);
                p2 = p1;
                p1 = p;
            }
        }
    }
}

// Coefficients of Hankel's expansions: A_k(nu) = prod_{i <= k} (4 nu^2 - (2 i - 1)^2) / (8 i); P has
// (-1)^j A_2j, Q (-1)^j A_2j+1, in powers of 1/x^2. From x = 25 on, twenty terms reach 3e-17.
struct HankelCoef {
    double p[2][10], q[2][10];
    constexpr HankelCoef() : p{}, q{} {
        for (int nu = 0; nu < 2; ++nu) {
            double a = 1;
            for (int k = 0; k < 20; ++k) {
                if (k > 0) a *= (4.0 * nu * nu - (2.0 * k - 1) * (2.0 * k - 1)) / (8.0 * k);
                const double v = (k / 2) % 2 ? -a : a;
                if (k % 2) q[nu][k / 2] = v;
                else p[nu][k / 2] = v;
            }
        }
    }
};
__constant__ HankelCoef kHankel;

// J_0(x), J_1(x) for x >= 25 (cos, sin of x - pi/4 and x - 3 pi/4 formed from cos x, sin x).
__device__ void bessel01_asymptotic(double x, double& j0, double& j1) {
    const double ix = 1.0 / x, i2 = ix * ix;
    double P[2], Q[2];
#pragma unroll
    for (int nu = 0; nu < 2; ++nu) {
        P[nu] = kHankel.p[nu][9];
        Q[nu] = kHankel.q[nu][9];
#pragma unroll
        for (int k = 8; k >= 0; --k) {
            P[nu] = fma(P[nu], i2, kHankel.p[nu][k]);
            Q[nu] = fma(Q[nu], i2, kHankel.q[nu][k]);
        }
        Q[nu] *= ix;
    }
    double s, c;
    sincos(x, &s, &c);
    const double amp = sqrt(ix * (1.0 / 3.14159265358979323846));  // sqrt(2 / (pi x)) sqrt(1/2)
    j0 = amp * (P[0] * (c + s) - Q[0] * (s - c));
    j1 = amp * (P[1] * (s - c) + Q[1] * (s + c));
}

// J_n(x), n = 0..N, written to out[n * stride]; num[n] = n as FP64.
constexpr int kJnExtra = 72, kJnTab = 2 * kMpMaxL + kJnExtra + 2;
__device__ void cyl_bessel_row(int N, double x, double* out, size_t stride, const double* num) {
    if (x == 0) {
        out[0] = 1;
        for (int n = 1; n <= N; ++n) out[n * stride] = 0;
        return;
    }
    if (!(x > 0)) {  // not a number
        for (int n = 0; n <= N; ++n) out[n * stride] = x;
        return;
    }
    const double ix2 = 2.0 / x;
    if (x >= 25 && x > N) {
        double jm, jc;
        bessel01_asymptotic(x, jm, jc);
        out[0] = jm;
        if (N >= 1) out[stride] = jc;
        for (int n = 1; n < N; ++n) {
            const double jn = num[n] * ix2 * jc - jm;
            out[(n + 1) * stride] = jn;
            jm = jc;
            jc = jn;
        }
        return;
    }
    // Miller's downward recurrence from M, normalised by J_0 + 2 sum J_2k = 1. Ratios J_n / J_{n-1}
    // are below x / (n + sqrt(n^2 - x^2)) for n > x; M is where those from x on have multiplied to
    // 2^-58 (the sum's rest) and those above N to 2^-32 (its square: the second solution).
    int M = (int)x;
    const int cap = max(N, M) + kJnExtra;
    for (float pa = 1.f, pb = 1.f, xf = (float)x; M < cap && (M < N || pa > 3e-18f || pb > 2.3e-10f);) {
        ++M;
        const float nf = (float)M, r = fminf(__fdividef(xf, nf + sqrtf(fmaxf(nf * nf - xf * xf, 0.f))), 1.f);
        pa *= r;
        if (M > N) pb *= r;
    }
    M += M & 1;
    double fp = 0, f = 1e-250, norm = 0;
    auto step = [&](int n) {  // f_n to f_{n-1}
        const double fm = num[n] * ix2 * f - fp;
        fp = f;
        f = fm;
        if (n - 1 <= N) out[(n - 1) * stride] = f;
        if ((__double2hiint(f) & 0x7fffffff) > 0x69800000) {  // 2^665
            for (int k = n - 1; k <= N; ++k) out[k * stride] *= 1e-200;
            fp *= 1e-200;
            f *= 1e-200;
            norm *= 1e-200;
        }
    };
    for (int n = M; n > 0; n -= 2) {
        step(n);
        step(n - 1);
        norm += f;
    }
    const double inorm = 1.0 / (2 * norm - f);
    for (int n = 0; n <= N; ++n) out[n * stride] *= inorm;
}

// ---------------------------------------------------------------------------------------
// Sums again in FP64
// ---------------------------------------------------------------------------------------
// The contractions hold a factor in units of 2^-57 of a bound that is common to all atoms of a frame,
// so a product is off by about 2^-57 of the product of the two bounds, whatever its own size. That is
// far below FP64's rounding where the bounds are reached by the same atoms, but not where every product
// is small beside them: harmonics of high m of atoms near the polar axis (theta^m; a column on the axis,
// 500 atoms, the moment (12, 12) alone: 5e-6 of S(q, 0)), a class of factor 0 that holds the large
// Bessel functions, the sine moments of atoms in one half plane. So the amplitudes of each (frame, q),
// over all the moments asked for, are compared with the error expected of them, and where it is more
// than 2^-44 of their norm the frame's angular functions are written as FP64 numbers and the sums taken
// of those. (The expectation takes the bounds as reached and is some eight times what comes out: single
// moments of 100,000 atoms that pass it differ by 1.6e-14 of S(q, 0) from the FP64 sums, all 441 by 1.4e-15.
// At 2^-47 a third of the frames of such a system would be summed again.)
// One cluster of kRedoCtas CTAs a frame tests it and, where needed, does both. Ordinary calls have none: 64 frames, 10 q, 441 moments 2.500 ms without the test, 2.504 so (2.53 with the three steps
// as kernels of their own). Of a column of 5,000 atoms, the 182 moments of |m| >= 8 are all summed again:
// 1.7 ms without, 4.4 so, 5.9 with FP64 sums alone.
constexpr int kRedoCtas = 8;
struct MpRedo {
    unsigned* word;  // [nfb][nq + 1] whether (frame, q) is summed again; last: any q of the frame
    int nq;
    __device__ unsigned* at(int fl, int q) const { return word + (size_t)fl * (nq + 1) + q; }
};

__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 4^e, e kept where it and sums of it are FP64 numbers
__device__ __forceinline__ double mp_pow4(int e) { return __hiloint2double((2 * min(max(e, -500), 500) + 1023) << 20, 0); }

// One warp: the norm of the moments A[k * stride] against their expected error. `err2` is a lane's share of
// the sum over moments of 4^e, 2^e the product of their rows' bounds, of which each atom's term is off by
// 2^-57. Amplitudes that are not finite stay so.
__device__ __forceinline__ void mp_decide(const MpRedo& r, int fl, int q, double err2, const double2* A, size_t stride,
                                         int nmom, int na) {
    const int lane = threadIdx.x & 31;
    double sum2 = 0.0;
#pragma unroll 8
    for (int k = lane; k < nmom; k += 32) {
        const double2 v = A[k * stride];
        sum2 = fma(v.x, v.x, fma(v.y, v.y, sum2));
    }
    for (int o = 16; o; o >>= 1) {
        sum2 += __shfl_xor_sync(0xffffffffu, sum2, o);
        err2 += __shfl_xor_sync(0xffffffffu, err2, o);
    }
    if (lane) return;
    const unsigned redo = err2 * na > 67108864.0 * sum2;  // 4^(57 - 44)
    *r.at(fl, q) = redo;
    if (redo) atomicOr(r.at(fl, r.nq), 1u);
}

// Exponent of a row whose largest magnitude has the upper half `m`; 4096: not finite.
__device__ __forceinline__ int mp_exponent(unsigned m) {
    return m >= 0x7ff00000u ? 4096 : max((int)(m >> 20), 1) - 1022;
}

// ---------------------------------------------------------------------------------------
// sphere: basis and contraction
// ---------------------------------------------------------------------------------------
struct MpSphereBasis {
    const float4* sph;  // [nf][na_pad] (r, phi, theta, class), atoms in order of frame-0 radius
    const double* cf;   // [nq][nclass]
    const double* qlen; // [nq]
    const int* idx;     // [L+1][L+1]: pair (l, m >= 0) or -1
    void* legendre;     // tables of ylm_coeff_kernel
    double* Jb;         // [nfb][nq][L+1][na_pad]  b_j(q) j_l(|q| r_j)
    unsigned* jmax;     // [nfb][nq][L+1] largest |Jb| of the row, its upper half's bits
    int4* Yc;           // [nfb][npair][na_pad]    conj(Y_l^m(j)) / g_lm, m >= 0, in fixed point
    MpRedo redo;
    int na_pad, nclass, nq, L, npair, f0, nfb;
};

// The tables of the Legendre functions, in shared memory at `smem`.
__device__ __forceinline__ MpLegendre mp_tables(void* legendre, int L, void* smem) {
    const MpLegendre from = legendre_at(legendre, L), t = legendre_at(smem, L);
    const int ncf = (L + 1) * (L + 2) / 2;
    for (int i = threadIdx.x; i < ncf; i += blockDim.x) {
        t.al[i] = from.al[i];
        t.ex[i] = from.ex[i];
    }
    for (int i = threadIdx.x; i <= L; i += blockDim.x) t.sd[i] = from.sd[i];
    __syncthreads();
    return t;
}

// conj(Y_l^m) / g_lm of every (frame, atom) of the batch. Also clears jmax and the frames' redo words for
// the kernels that follow.
__global__ void __launch_bounds__(128) mp_ylm_kernel(MpSphereBasis a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const MpLegendre t = mp_tables(a.legendre, a.L, smem);
    const size_t n = (size_t)a.nfb * a.na_pad, n0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    for (size_t i = n0; i < (size_t)a.nfb * a.nq * (a.L + 1); i += (size_t)gridDim.x * blockDim.x) a.jmax[i] = 0u;
    for (size_t i = n0; i < (size_t)a.nfb; i += (size_t)gridDim.x * blockDim.x) *a.redo.at((int)i, a.nq) = 0u;
    for (size_t i = n0; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int fl = (int)(i / a.na_pad), j = (int)(i - (size_t)fl * a.na_pad);
        const float4 c = a.sph[(size_t)(a.f0 + fl) * a.na_pad + j];
        conj_ylm_row<true>(a.L, (double)c.z, (double)c.y, a.idx, t, a.Yc + (size_t)fl * a.npair * a.na_pad + j, a.na_pad);
    }
}

// b_j(q) j_l(|q| r_j) of every (frame, q, atom) of the batch, and each row's largest magnitude.
__global__ void __launch_bounds__(128) mp_jl_kernel(MpSphereBasis a) {
    __shared__ JlTab t;
    for (int i = threadIdx.x; i < kJlTab; i += blockDim.x) {
        t.odd[i] = 2 * i + 1;
        t.iodd[i] = 1.0 / (2 * i + 1);
        t.inv[i] = i ? 1.0 / i : 0.0;
    }
    __syncthreads();
    const size_t n = (size_t)a.nfb * a.nq * a.na_pad;  // na_pad is a multiple of 32: a warp has one row
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t fq = i / a.na_pad;
        const int j = (int)(i - fq * a.na_pad), fl = (int)(fq / a.nq), q = (int)(fq - (size_t)fl * a.nq);
        const float4 c = a.sph[(size_t)(a.f0 + fl) * a.na_pad + j];
        const int cl = (int)c.w;  // atoms sit in radius order; w carries the class (-1: padding)
        const double b = cl >= 0 ? a.cf[(size_t)q * a.nclass + cl] : 0.0;
        double* row = a.Jb + (fq * (a.L + 1)) * a.na_pad + j;
        sph_bessel_row(a.L, a.qlen[q] * (double)c.x, b, row, a.na_pad, t);
        __syncwarp();
        for (int l = 0; l <= a.L; ++l) {
            const unsigned mx =
                __reduce_max_sync(0xffffffffu, (unsigned)__double2hiint(row[(size_t)l * a.na_pad]) & 0x7fffffffu);
            if ((threadIdx.x & 31) == 0) atomicMax(a.jmax + fq * (a.L + 1) + l, mx);
        }
    }
}

struct MpSphereContract {
    const float4* sph;
    const int* idx;
    const double* Jb;
    const unsigned* jmax;
    int4* Yc;
    void* legendre;
    const int4* groups;  // [ngroups] (l, first pair, pairs (at most 8), 0): pairs of one l, consecutive
    const int* pmom;     // [npair + 1] first entry of each pair in pout
    const int* pout;     // moments of the pairs, 2 moment + (m < 0)
    const int* pm;       // [npair] m of the pair
    const int* pl;       // [npair] l
    double2* A;          // [nq][nmom][nf]
    MpRedo redo;
    int na_pad, na, nq, L, nmom, npair, nf, f0;
};

// The amplitudes of a pair's moments from v = sum_j b_j j_l conj(Y_l^m): times i^l, and for -m
// (-1)^m times the conjugate (b_j j_l is real).
__device__ __forceinline__ void mp_sphere_store(const MpSphereContract& a, int pair, int l, int q, int fl, double2 v) {
    for (int i = a.pmom[pair]; i < a.pmom[pair + 1]; ++i) {
        const int out = a.pout[i];
        double2 u = v;
        if (out & 1) u = (a.pm[pair] & 1) ? make_double2(-v.x, v.y) : make_double2(v.x, -v.y);
        double2 w;
        switch (l & 3) {
            case 0: w = make_double2(u.x, u.y); break;
            case 1: w = make_double2(-u.y, u.x); break;
            case 2: w = make_double2(-u.x, -u.y); break;
            default: w = make_double2(u.y, -u.x); break;
        }
        a.A[((size_t)q * a.nmom + (out >> 1)) * a.nf + a.f0 + fl] = w;
    }
}
constexpr double kMp4Pi = 4 * 3.14159265358979323846;

constexpr int kSumWarps = 8, kSumTile = 256;  // atoms of a tile
static_assert(kSumTile == kSumWarps * 32, "a thread converts one atom of a tile");

__device__ __forceinline__ void mp_cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// sum_j b_j(q) j_l(|q| r_j) conj(Y_l^m(j)) of one frame, up to 8 pairs (l, m) and QB q-vectors, in
// integers: the FP64 pipe takes 19 clocks of an SM per warp FMA, a product of 58-bit numbers as
// three 32 x 32 -> 64-bit multiplications about 1.7 each. J gets the exponent of its row's largest
// value, Y that of its bound, so that both keep 57 bits below it; the low halves' product, below
// 2^-58 of the largest, is left out; where that is not enough see MpRedo. Only m >= 0 is summed. A lane is an atom, a warp a pair (or, of fewer pairs than warps, a
// pair and a part of the atoms): Y is read once, straight from memory; the tile's J words are
// shared. QB x 2 sums of two words each stay in registers; before they could overflow (62-bit
// products, 56 atoms a lane) they are added over the lanes by 26-bit pieces and go to FP64.
// 5,000 atoms, 64 frames, 10 q, 441 moments: 6.7 ms before, 1.1 here.
template <int QB>
__global__ void __launch_bounds__(kSumWarps * 32, 2) mp_sphere_sum_kernel(MpSphereContract a) {
    __shared__ int2 Js[QB][kSumTile];
    __shared__ __align__(16) double raw[QB][kSumTile];  // the next tile
    __shared__ int rowe[QB];
    __shared__ double part[kSumWarps][2 * QB];
    asm volatile("griddepcontrol.launch_dependents;");
    const int4 grp = a.groups[blockIdx.x];
    const int l = grp.x, cnt = grp.z, fl = blockIdx.y, q0 = blockIdx.z * QB, nqb = min(QB, a.nq - q0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* jrow = a.Jb + (((size_t)fl * a.nq + q0) * (a.L + 1) + l) * a.na_pad;
    const size_t qstep = (size_t)(a.L + 1) * a.na_pad;
    const int jend = (a.na + 31) & ~31;  // <= na_pad; b_j = 0 past na
    if (threadIdx.x < nqb) {
        rowe[threadIdx.x] = mp_exponent(a.jmax[((size_t)fl * a.nq + q0 + threadIdx.x) * (a.L + 1) + l]);
    }
    auto fetch = [&](int j0) {  // two atoms a thread and row
        for (int i = threadIdx.x; i < nqb * (kSumTile / 2); i += kSumWarps * 32) {
            const int q = i / (kSumTile / 2), j = i % (kSumTile / 2) * 2;
            if (j0 + j < jend) mp_cp_async16(&raw[q][j], jrow + q * qstep + j0 + j);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    // atoms in parts: 8 / cnt warps share a pair
    const int aw = cnt > 4 ? 1 : cnt > 2 ? 2 : cnt > 1 ? 4 : 8;
    const int k = warp % cnt, g = warp / cnt;
    const bool live = g < aw;
    const int4* y = a.Yc + ((size_t)fl * a.npair + grp.y + k) * a.na_pad + g * 32 + lane;
    long long rh[QB], rx[QB], ih[QB], ix[QB];
#pragma unroll
    for (int q = 0; q < QB; ++q) rh[q] = rx[q] = ih[q] = ix[q] = 0;
    double total = 0.0;  // of the output this lane holds: 2 q (+ 1: imaginary part)
    int n = 0;
    auto flush = [&]() {
        int p0 = 0, p1 = 0, p2 = 0;
        auto take = [&](long long h, int o) {
            const int s0 = __reduce_add_sync(0xffffffffu, (int)h & 0x3ffffff);
            const int s1 = __reduce_add_sync(0xffffffffu, (int)(h >> 26) & 0x3ffffff);
            const int s2 = __reduce_add_sync(0xffffffffu, (int)(h >> 52));
            if (lane == o) {
                p0 = s0;
                p1 = s1;
                p2 = s2;
            }
        };
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            take(rh[q] + ((rx[q] + (1 << 28)) >> 29), 2 * q);
            take(ih[q] + ((ix[q] + (1 << 28)) >> 29), 2 * q + 1);
            rh[q] = rx[q] = ih[q] = ix[q] = 0;
        }
        total += fma((double)p2, 4503599627370496.0, fma((double)p1, 67108864.0, (double)p0));
        n = 0;
    };
    const int4 zero = make_int4(0, 0, 0, 0);
    int4 yv = live && g * 32 < jend ? *y : zero;
    for (int j0 = 0; j0 < jend; j0 += kSumTile) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // raw is here; the exponents; the previous tile has been read
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            int2 w = make_int2(0, 0);
            if (q < nqb && j0 + (int)threadIdx.x < jend) w = mp_words(raw[q][threadIdx.x], rowe[q]);
            Js[q][threadIdx.x] = w;
        }
        __syncthreads();
        if (j0 + kSumTile < jend) fetch(j0 + kSumTile);
        if (!live) continue;
        for (int c = g * 32; c < kSumTile && j0 + c < jend; c += aw * 32) {
            const int4 v = yv;
            y += aw * 32;
            yv = j0 + c + aw * 32 < jend ? *y : zero;
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const int2 w = Js[q][c + lane];
                rh[q] += mp_wide(w.x, v.x, 0);
                rx[q] += mp_wide(w.x, v.y, mp_wide(w.y, v.x, 0));
                ih[q] += mp_wide(w.x, v.z, 0);
                ix[q] += mp_wide(w.x, v.w, mp_wide(w.y, v.z, 0));
            }
            ++n;
        }
        if (n > 48) {
            flush();
        } else if (n & 8 || n > 16) {  // the cross products' sums (2^57 each) into the high ones
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                rh[q] += rx[q] >> 29;
                rx[q] &= (1 << 29) - 1;
                ih[q] += ix[q] >> 29;
                ix[q] &= (1 << 29) - 1;
            }
        }
    }
    if (live) {
        flush();
        if (lane < 2 * QB) part[warp][lane] = total;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < cnt * nqb; o += kSumWarps * 32) {
        const int q = o / cnt, kk = o - q * cnt, pair = grp.y + kk;
        double2 v = make_double2(0.0, 0.0);
        for (int w = kk; w < aw * cnt; w += cnt) {
            v.x += part[w][2 * q];
            v.y += part[w][2 * q + 1];
        }
        const double f = rowe[q] == 4096 ? nan("") : kMp4Pi;
        const MpLegendre lt = legendre_at(a.legendre, a.L);
        const int i0 = l * (l + 1) / 2 + a.pm[pair], e = rowe[q] + lt.ex[i0] - 56;
        v = make_double2(f * lt.g[i0] * scalbn(v.x, e), f * lt.g[i0] * scalbn(v.y, e));
        mp_sphere_store(a, pair, l, q0 + q, fl, v);
    }
}

// A frame's amplitudes against their expected error (4 pi g_lm times the bound 2^ex is below
// 2 sqrt(4 pi (2l + 1))) and, where they need it, their sums in FP64: the harmonics as FP64 numbers in
// place of the words, then a warp a pair, 2 FMAs an atom, which the FP64 pipe bounds.
__global__ void __cluster_dims__(kRedoCtas, 1, 1) __launch_bounds__(kSumWarps * 32) mp_sphere_redo_kernel(MpSphereContract a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int fl = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, jend = (a.na + 31) & ~31;
    const int w0 = blockIdx.x * kSumWarps + warp, wn = kRedoCtas * kSumWarps;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int q = w0; q < a.nq; q += wn) {
        const unsigned* mx = a.jmax + ((size_t)fl * a.nq + q) * (a.L + 1);
        double err2 = 0.0;
        for (int k = lane; k < a.npair; k += 32) {
            const int l = a.pl[k], e = mp_exponent(mx[l]) + 3 + (33 - __clz(2 * l + 1)) / 2;
            err2 = fma(mp_pow4(e), (double)(a.pmom[k + 1] - a.pmom[k]), err2);
        }
        mp_decide(a.redo, fl, q, err2, a.A + (size_t)q * a.nmom * a.nf + a.f0 + fl, a.nf, a.nmom, a.na);
    }
    cluster_barrier();
    if (*reinterpret_cast<volatile unsigned*>(a.redo.at(fl, a.nq)) == 0u) return;  // the same for the whole cluster
    int4* Yf = a.Yc + (size_t)fl * a.npair * a.na_pad;
    {
        const MpLegendre t = mp_tables(a.legendre, a.L, smem);
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < jend; j += kRedoCtas * blockDim.x) {
            const float4 c = a.sph[(size_t)(a.f0 + fl) * a.na_pad + j];
            conj_ylm_row<false>(a.L, (double)c.z, (double)c.y, a.idx, t, Yf + j, a.na_pad);
        }
    }
    cluster_barrier();
    const double* g = legendre_at(a.legendre, a.L).g;
    for (int q = 0; q < a.nq; ++q) {
        if (!*a.redo.at(fl, q)) continue;
        for (int k = w0; k < a.npair; k += wn) {
            const int l = a.pl[k];
            const double* J = a.Jb + (((size_t)fl * a.nq + q) * (a.L + 1) + l) * a.na_pad;
            const double2* Y = reinterpret_cast<const double2*>(Yf) + (size_t)k * a.na_pad;
            double2 v = make_double2(0.0, 0.0);
#pragma unroll 4
            for (int j = lane; j < jend; j += 32) {
                const double b = J[j];
                const double2 y = Y[j];
                v.x = fma(b, y.x, v.x);
                v.y = fma(b, y.y, v.y);
            }
            for (int o = 16; o; o >>= 1) {
                v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
                v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
            }
            const double f = kMp4Pi * g[l * (l + 1) / 2 + a.pm[k]];
            if (lane == 0) mp_sphere_store(a, k, l, q, fl, make_double2(f * v.x, f * v.y));
        }
    }
}

template <int QB>
cudaError_t launch_sphere_sum(int qb, const MpSphereContract& a, dim3 grid, cudaStream_t st) {
    if (qb < QB) {
        if constexpr (QB > 1) return launch_sphere_sum<QB - 1>(qb, a, grid, st);
    }
    mp_sphere_sum_kernel<QB><<<grid, kSumWarps * 32, 0, st>>>(a);
    return cudaGetLastError();
}
constexpr int kSumQ = 10;  // q-vectors of a CTA, at most: their sums fill the registers

// ---------------------------------------------------------------------------------------
// cylinder
// ---------------------------------------------------------------------------------------
struct MpCylinder {
    const float4* cyl;   // [nf][na_pad] (r, phi, z, class), atoms in order of frame-0 radius
    const double* cf;    // [nq][nclass]
    const double* qcyl;  // [nq][3] (q_r, phi_q, q_z)
    double* Jb;          // [nfb][nq][N+3][na_pad]: J_n(q_r r), then real and imaginary part of X
    unsigned* jmax;      // [nfb][nq][N+3] largest magnitude of the row, its upper half's bits
    int4* Tc;            // [nfb][nn][na_pad] cos(n phi), sin(n phi) in fixed point
    const int* ns;       // [nn] the orders that the moments need
    const int* nmom0;    // [nn + 1] first entry of each order in nout
    const int* nout;     // [nmom] the moments of the orders
    const int* mom;      // [nmom][2]
    double2* A;          // [nq][nmom][nf]
    MpRedo redo;
    int na_pad, na, nclass, nq, N, nn, nmom, nf, f0, nfb;
};

// cos(n phi), sin(n phi) of one atom by rotation, n ascending, to out[k * na_pad]: fixed-point words or,
// with FIXED false, a double2.
template <bool FIXED>
__device__ void mp_angle_row(const MpCylinder& a, double phi, int4* out) {
    double s1, c1, cp = 1, sp = 0;
    sincos(phi, &s1, &c1);
    for (int k = 0, at = 0; k < a.nn; ++k) {
        for (const int order = a.ns[k]; at < order; ++at) {
            const double cq = cp * c1 - sp * s1;
            sp = sp * c1 + cp * s1;
            cp = cq;
        }
        if constexpr (FIXED) {
            const int2 c = mp_unit(cp), s = mp_unit(sp);
            out[(size_t)k * a.na_pad] = make_int4(c.x, c.y, s.x, s.y);
        } else {
            reinterpret_cast<double2*>(out)[(size_t)k * a.na_pad] = make_double2(cp, sp);
        }
    }
}

// The angles of every (frame, atom) of the batch. Also clears jmax and the frames' redo words for the
// kernels that follow.
__global__ void __launch_bounds__(128) mp_angle_kernel(MpCylinder a) {
    const size_t n = (size_t)a.nfb * a.na_pad, n0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    for (size_t i = n0; i < (size_t)a.nfb * a.nq * (a.N + 3); i += (size_t)gridDim.x * blockDim.x) a.jmax[i] = 0u;
    for (size_t i = n0; i < (size_t)a.nfb; i += (size_t)gridDim.x * blockDim.x) *a.redo.at((int)i, a.nq) = 0u;
    for (size_t i = n0; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int fl = (int)(i / a.na_pad), j = (int)(i - (size_t)fl * a.na_pad);
        mp_angle_row<true>(a, (double)a.cyl[(size_t)(a.f0 + fl) * a.na_pad + j].y, a.Tc + (size_t)fl * a.nn * a.na_pad + j);
    }
}

// J_n(q_r r), n <= N, and X = b e^{i s z q_z} of every (frame, q, atom) of the batch, and each row's
// largest magnitude. Bound by the FP64 pipe: atoms in order of radius, so that a warp takes one
// branch; about 260 FP64 instructions a row of 41 orders.
__global__ void __launch_bounds__(128) mp_jn_kernel(MpCylinder a) {
    __shared__ double num[kJnTab];
    for (int i = threadIdx.x; i < kJnTab; i += blockDim.x) num[i] = i;
    __syncthreads();
    const size_t n = (size_t)a.nfb * a.nq * a.na_pad;  // na_pad is a multiple of 32: a warp has one row
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t fq = i / a.na_pad;
        const int j = (int)(i - fq * a.na_pad), fl = (int)(fq / a.nq), q = (int)(fq - (size_t)fl * a.nq);
        const float4 c = a.cyl[(size_t)(a.f0 + fl) * a.na_pad + j];
        const int cl = (int)c.w;  // atoms sit in radius order; w carries the class (-1: padding)
        const double b = cl >= 0 ? a.cf[(size_t)q * a.nclass + cl] : 0.0;
        const double qr = a.qcyl[3 * q], qz = a.qcyl[3 * q + 2], z = c.z;
        double sgn = 1.0;  // parallel_sign, multipole_scatter_device.cpp:944-948
        if (z != 0 && qz != 0) sgn = (z * qz) / (fabs(z) * fabs(qz));
        double es, ec;
        sincos(sgn * z * qz, &es, &ec);
        double* row = a.Jb + (fq * (a.N + 3)) * a.na_pad + j;
        row[(size_t)(a.N + 1) * a.na_pad] = b * ec;
        row[(size_t)(a.N + 2) * a.na_pad] = b * es;
        cyl_bessel_row(a.N, (double)c.x * qr, row, a.na_pad, num);
        __syncwarp();
        for (int l = 0; l < a.N + 3; ++l) {
            const unsigned mx =
                __reduce_max_sync(0xffffffffu, (unsigned)__double2hiint(row[(size_t)l * a.na_pad]) & 0x7fffffffu);
            if ((threadIdx.x & 31) == 0) atomicMax(a.jmax + fq * (a.N + 3) + l, mx);
        }
    }
}

// The amplitudes of an order's moments from C, S = sqrt(2 pi) sum_j X_j J_n(j) (cos, sin)(n phi_j).
__device__ __forceinline__ void mp_cylinder_store(const MpCylinder& a, int k, int q, int fl, double2 C, double2 S) {
    const double h2 = 0.70710678118654752440;
    double snq, cnq;
    sincos(a.ns[k] * a.qcyl[3 * q + 1], &snq, &cnq);
    for (int u = a.nmom0[k]; u < a.nmom0[k + 1]; ++u) {
        const int mk = a.nout[u], l = a.mom[2 * mk], m = a.mom[2 * mk + 1];
        double2 v;
        if (l == 0 && m == 0) {
            v = C;
        } else {
            double2 w;  // sum_j X_j J_n cos / sin (n (phi_j - phi_q))
            if (m == 0 || m == 2) w = make_double2(cnq * C.x + snq * S.x, cnq * C.y + snq * S.y);
            else w = make_double2(cnq * S.x - snq * C.x, cnq * S.y - snq * C.y);
            if (m < 2) {
                const double c = h2 * 2.0 * ((l & 1) ? -1.0 : 1.0);
                v = make_double2(c * w.x, c * w.y);
            } else {  // times i sqrt(1/2) 2 (-1)^(l-1)
                const double c = h2 * 2.0 * (((l - 1) & 1) ? -1.0 : 1.0);
                v = make_double2(-c * w.y, c * w.x);
            }
        }
        a.A[((size_t)q * a.nmom + mk) * a.nf + a.f0 + fl] = v;
    }
}
constexpr double kMpSqrt2Pi = 2.50662827463100050242;

// sum_j X_j J_n(j) (cos, sin)(n phi_j) of one frame for up to 8 orders n and QB q-vectors, in integers
// as mp_sphere_sum_kernel sums: a lane is an atom, a warp an order (or a part of one's atoms). The
// tile's X words are shared; J and the angles are read once, straight from memory. X J is one
// 58-bit product more, taken before the four sums' (18 of the 32-bit multiplications per J, 12 of
// them in the sums). 5,000 atoms, 64 frames, 10 q, 41 orders: 8.0 ms with the basis before, 2.7 now
// (1.0 here, 1.5 the Bessel rows).
template <int QB>
__global__ void __launch_bounds__(kSumWarps * 32, 2) mp_cylinder_sum_kernel(MpCylinder a) {
    __shared__ int4 Xs[QB][kSumTile];
    __shared__ int jexp[kSumWarps][QB], xexp[QB];
    __shared__ double part[kSumWarps][4 * QB];
    asm volatile("griddepcontrol.launch_dependents;");
    const int fl = blockIdx.y, q0 = blockIdx.z * QB, nqb = min(QB, a.nq - q0);
    const int k0 = blockIdx.x * kSumWarps, cnt = min(kSumWarps, a.nn - k0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t qstep = (size_t)(a.N + 3) * a.na_pad;
    const double* rows = a.Jb + ((size_t)fl * a.nq + q0) * qstep;
    const unsigned* mx = a.jmax + ((size_t)fl * a.nq + q0) * (a.N + 3);
    const int jend = (a.na + 31) & ~31;  // <= na_pad; b_j = 0 past na
    for (int i = threadIdx.x; i < cnt * nqb; i += kSumWarps * 32)
        jexp[i / nqb][i % nqb] = mp_exponent(mx[(size_t)(i % nqb) * (a.N + 3) + a.ns[k0 + i / nqb]]);
    if (threadIdx.x < nqb)
        xexp[threadIdx.x] = mp_exponent(max(mx[(size_t)threadIdx.x * (a.N + 3) + a.N + 1],
                                         mx[(size_t)threadIdx.x * (a.N + 3) + a.N + 2]));
    __syncthreads();
    const int aw = cnt > 4 ? 1 : cnt > 2 ? 2 : cnt > 1 ? 4 : 8;
    const int k = warp % cnt, g = warp / cnt, order = a.ns[k0 + k];
    const bool live = g < aw;
    const int4* t = a.Tc + ((size_t)fl * a.nn + k0 + k) * a.na_pad + g * 32 + lane;
    const double* jn = rows + (size_t)order * a.na_pad + g * 32 + lane;
    int je[QB];
#pragma unroll
    for (int q = 0; q < QB; ++q) je[q] = q < nqb ? jexp[k][q] : 0;
    long long h[QB][4], x[QB][4];
#pragma unroll
    for (int q = 0; q < QB; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) h[q][i] = x[q][i] = 0;
    double total = 0.0;  // of the output this lane holds: 4 q + (re cos, im cos, re sin, im sin)
    int n = 0;
    auto flush = [&]() {
        int p0 = 0, p1 = 0, p2 = 0;
#pragma unroll
        for (int o = 0; o < 4 * QB; ++o) {
            const long long v = h[o / 4][o % 4] + ((x[o / 4][o % 4] + (1 << 28)) >> 29);
            const int s0 = __reduce_add_sync(0xffffffffu, (int)v & 0x3ffffff);
            const int s1 = __reduce_add_sync(0xffffffffu, (int)(v >> 26) & 0x3ffffff);
            const int s2 = __reduce_add_sync(0xffffffffu, (int)(v >> 52));
            if (lane == o) {
                p0 = s0;
                p1 = s1;
                p2 = s2;
            }
            h[o / 4][o % 4] = x[o / 4][o % 4] = 0;
        }
        total += fma((double)p2, 4503599627370496.0, fma((double)p1, 67108864.0, (double)p0));
        n = 0;
    };
    int4 tv = make_int4(0, 0, 0, 0);
    double jv[QB];
    auto load = [&](int j) {
        if (j < jend) {
            tv = *t;
#pragma unroll
            for (int q = 0; q < QB; ++q) jv[q] = q < nqb ? jn[q * qstep] : 0.0;
        }
        t += aw * 32;
        jn += aw * 32;
    };
    if (live) load(g * 32);
    for (int j0 = 0; j0 < jend; j0 += kSumTile) {
        __syncthreads();  // the previous tile has been read
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            const int j = j0 + threadIdx.x;
            int4 w = make_int4(0, 0, 0, 0);
            if (q < nqb && j < jend) {
                const double* p = rows + q * qstep + (size_t)(a.N + 1) * a.na_pad + j;
                const int2 re = mp_words(p[0], xexp[q]), im = mp_words(p[a.na_pad], xexp[q]);
                w = make_int4(re.x, re.y, im.x, im.y);
            }
            Xs[q][threadIdx.x] = w;
        }
        __syncthreads();
        if (!live) continue;
        for (int c = g * 32; c < kSumTile && j0 + c < jend; c += aw * 32) {
            const int4 v = tv;
            int2 jw[QB];
#pragma unroll
            for (int q = 0; q < QB; ++q) jw[q] = mp_words(jv[q], je[q]);
            load(j0 + c + aw * 32);
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const int4 w = Xs[q][c + lane];
                const int2 re = mp_split(mp_mul(jw[q], make_int2(w.x, w.y)));
                const int2 im = mp_split(mp_mul(jw[q], make_int2(w.z, w.w)));
                h[q][0] += mp_wide(re.x, v.x, 0);
                x[q][0] += mp_wide(re.x, v.y, mp_wide(re.y, v.x, 0));
                h[q][1] += mp_wide(im.x, v.x, 0);
                x[q][1] += mp_wide(im.x, v.y, mp_wide(im.y, v.x, 0));
                h[q][2] += mp_wide(re.x, v.z, 0);
                x[q][2] += mp_wide(re.x, v.w, mp_wide(re.y, v.z, 0));
                h[q][3] += mp_wide(im.x, v.z, 0);
                x[q][3] += mp_wide(im.x, v.w, mp_wide(im.y, v.z, 0));
            }
            ++n;
        }
        if (n > 48) {
            flush();
        } else if (n & 8 || n > 16) {  // the cross products' sums (2^57 each) into the high ones
#pragma unroll
            for (int o = 0; o < 4 * QB; ++o) {
                h[o / 4][o % 4] += x[o / 4][o % 4] >> 29;
                x[o / 4][o % 4] &= (1 << 29) - 1;
            }
        }
    }
    if (live) {
        flush();
        if (lane < 4 * QB) part[warp][lane] = total;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < cnt * nqb; i += kSumWarps * 32) {
        const int kk = i / nqb, q = i - kk * nqb;
        double sum[4] = {0.0, 0.0, 0.0, 0.0};
        for (int w = kk; w < aw * cnt; w += cnt)
            for (int o = 0; o < 4; ++o) sum[o] += part[w][4 * q + o];
        const int e = jexp[kk][q] + xexp[q] - 56;
        const double f = jexp[kk][q] == 4096 || xexp[q] == 4096 ? nan("") : kMpSqrt2Pi;
        mp_cylinder_store(a, k0 + kk, q0 + q, fl, make_double2(f * scalbn(sum[0], e), f * scalbn(sum[1], e)),
                          make_double2(f * scalbn(sum[2], e), f * scalbn(sum[3], e)));
    }
}

// As mp_sphere_redo_kernel, a warp an order. A moment is 2 sqrt(pi) (cos C' + sin S'): below 2^2 of the
// sums C', S'.
__global__ void __cluster_dims__(kRedoCtas, 1, 1) __launch_bounds__(kSumWarps * 32) mp_cylinder_redo_kernel(MpCylinder a) {
    const int fl = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, jend = (a.na + 31) & ~31;
    const int w0 = blockIdx.x * kSumWarps + warp, wn = kRedoCtas * kSumWarps;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int q = w0; q < a.nq; q += wn) {
        const unsigned* mx = a.jmax + ((size_t)fl * a.nq + q) * (a.N + 3);
        const int xe = mp_exponent(max(mx[a.N + 1], mx[a.N + 2]));
        double err2 = 0.0;
        for (int k = lane; k < a.nn; k += 32)
            err2 = fma(mp_pow4(mp_exponent(mx[a.ns[k]]) + xe + 2), (double)(a.nmom0[k + 1] - a.nmom0[k]), err2);
        mp_decide(a.redo, fl, q, err2, a.A + (size_t)q * a.nmom * a.nf + a.f0 + fl, a.nf, a.nmom, a.na);
    }
    cluster_barrier();
    if (*reinterpret_cast<volatile unsigned*>(a.redo.at(fl, a.nq)) == 0u) return;  // the same for the whole cluster
    int4* Tf = a.Tc + (size_t)fl * a.nn * a.na_pad;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < jend; j += kRedoCtas * blockDim.x)
        mp_angle_row<false>(a, (double)a.cyl[(size_t)(a.f0 + fl) * a.na_pad + j].y, Tf + j);
    cluster_barrier();
    for (int q = 0; q < a.nq; ++q) {
        if (!*a.redo.at(fl, q)) continue;
        const double* rows = a.Jb + ((size_t)fl * a.nq + q) * (a.N + 3) * a.na_pad;
        const double *xr = rows + (size_t)(a.N + 1) * a.na_pad, *xi = xr + a.na_pad;
        for (int k = w0; k < a.nn; k += wn) {
            const double* J = rows + (size_t)a.ns[k] * a.na_pad;
            const double2* T = reinterpret_cast<const double2*>(Tf) + (size_t)k * a.na_pad;
            double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
            for (int j = lane; j < jend; j += 32) {
                const double2 t = T[j];
                const double c = J[j] * t.x, s = J[j] * t.y;
                v[0] = fma(xr[j], c, v[0]);
                v[1] = fma(xi[j], c, v[1]);
                v[2] = fma(xr[j], s, v[2]);
                v[3] = fma(xi[j], s, v[3]);
            }
            for (int o = 16; o; o >>= 1)
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
            if (lane == 0)
                mp_cylinder_store(a, k, q, fl, make_double2(kMpSqrt2Pi * v[0], kMpSqrt2Pi * v[1]),
                                  make_double2(kMpSqrt2Pi * v[2], kMpSqrt2Pi * v[3]));
        }
    }
}
constexpr int kCylQ = 5;  // q-vectors of a CTA, at most

template <int QB>
cudaError_t launch_cylinder_sum(int qb, const MpCylinder& a, dim3 grid, cudaStream_t st) {
    if (qb < QB) {
        if constexpr (QB > 1) return launch_cylinder_sum<QB - 1>(qb, a, grid, st);
    }
    mp_cylinder_sum_kernel<QB><<<grid, kSumWarps * 32, 0, st>>>(a);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
struct V3 {
    double x, y, z;
};
V3 cross3(V3 a, V3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
double len3(V3 a) { return sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
V3 div3(V3 a, double l) { return {a.x / l, a.y / l, a.z / l}; }

// CartesianVectorBase(axis), coor3d.cpp:278-295
bool axis_base(const double* axis, MpBase& b) {
    V3 a{axis[0], axis[1], axis[2]};
    if (!(len3(a) > 0)) return false;
    V3 ez = div3(a, len3(a));
    V3 ekez = cross3(V3{0, 0, 1}, ez);
    if (len3(ekez) == 0) ekez = cross3(V3{0, 1, 0}, ez);
    V3 er = div3(ekez, len3(ekez));
    V3 ezer = cross3(ez, er);
    V3 ephi = div3(ezer, len3(ezer));
    const V3 e[3] = {er, ephi, ez};
    for (int k = 0; k < 3; ++k) {
        b.e[3 * k] = e[k].x;
        b.e[3 * k + 1] = e[k].y;
        b.e[3 * k + 2] = e[k].z;
    }
    return true;
}

int fail(std::string& m, int code, const std::string& what) {
    m = what;
    return code;
}

// Starts while the contraction's last CTAs run (they signal at their beginning) and waits for its end
// (cylinder of 1,500 atoms, 30 frames, 4 q: 306 -> 299 us a call, 303 without this kernel).
template <class K, class A>
cudaError_t launch_redo(K kernel, const A& a, int nfb, size_t smem, cudaStream_t st) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(kRedoCtas, (unsigned)nfb);
    c.blockDim = dim3(kSumWarps * 32);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, a);
}

}  // namespace

}  // namespace sassgpu

using namespace sassgpu;

extern "C" int sass_multipole_compute(sass_plan* p, int type, size_t nq, const double* qvectors,
                                      const double* class_factors, size_t nmom, const int32_t* moments,
                                      const double* axis, double* fqt, double* fq, double* fq2) {
    if (!p) return SASS_ERR_ARG;
    if (nq == 0) return SASS_OK;
    if (!qvectors || !class_factors || !moments || !fqt || !fq || !fq2 || nmom == 0)
        return fail(p->msg, SASS_ERR_ARG, "NULL argument or no moments");
    if (type != SASS_MULTIPOLE_SPHERE && type != SASS_MULTIPOLE_CYLINDER)
        return fail(p->msg, SASS_ERR_ARG, "multipole type must be sphere or cylinder");
    if (p->d.precision != SASS_PRECISION_FP64 || p->d.scattering != SASS_SCATTERING_ALL)
        return fail(p->msg, SASS_ERR_UNSUPPORTED, "multipole devices need a coherent FP64 plan");
    if (!p->sys.staged || !p->sys.classes_set) return fail(p->msg, SASS_ERR_STATE, "plan not staged");
    const bool cyl = type == SASS_MULTIPOLE_CYLINDER;
    int L = 0;  // largest major moment
    for (size_t k = 0; k < nmom; ++k) {
        const int l = moments[2 * k], m = moments[2 * k + 1];
        // the reference's checks, parameters.cpp:1076-1114
        if (l < 0) return fail(p->msg, SASS_ERR_ARG, "major multipole moment must be >= 0");
        if (!cyl && std::abs(m) > l) return fail(p->msg, SASS_ERR_ARG, "minor multipole moment must be within -major..major");
        if (cyl && (m < 0 || m > 3)) return fail(p->msg, SASS_ERR_ARG, "minor multipole moment must be between 0 and 3");
        if (cyl && l == 0 && m != 0) return fail(p->msg, SASS_ERR_ARG, "minor multipole moment must be 0 for major 0");
        L = std::max(L, l);
    }
    if (L > kMpMaxL) return fail(p->msg, SASS_ERR_UNSUPPORTED, "major multipole moments above 40 are not supported");
    MpBase base{};
    if (cyl && (!axis || !axis_base(axis, base))) return fail(p->msg, SASS_ERR_ARG, "cylinder axis must be a nonzero vector");

    std::string& m = p->msg;
    auto cuda_fail = [&](cudaError_t e, const char* what) {
        cudaGetLastError();
        m = std::string(what) + ": " + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? SASS_ERR_OOM : SASS_ERR_CUDA;
    };
#define MCK(expr)                                  \
    do {                                           \
        cudaError_t e_ = (expr);                   \
        if (e_ != cudaSuccess) return cuda_fail(e_, #expr); \
    } while (0)
    MCK(cudaSetDevice(p->d.device));
    memset(&p->timing, 0, sizeof(p->timing));
    SystemState& s = p->sys;
    const size_t nf = s.nf, na_pad = s.na_pad, nclass = s.nclass;
    cudaStream_t st = p->st;
    size_t launches = 0;

    // per-q inputs: |q| (sphere) or the projected q in cylinder coordinates
    std::vector<double> qin(cyl ? 3 * nq : nq);
    for (size_t i = 0; i < nq; ++i) {
        const double* qv = qvectors + 3 * i;
        if (!cyl) {
            qin[i] = sqrt(qv[0] * qv[0] + qv[1] * qv[1] + qv[2] * qv[2]);  // q.length()
        } else {
            const double px = qv[0] * base.e[0] + qv[1] * base.e[1] + qv[2] * base.e[2];
            const double py = qv[0] * base.e[3] + qv[1] * base.e[4] + qv[2] * base.e[5];
            const double pz = qv[0] * base.e[6] + qv[1] * base.e[7] + qv[2] * base.e[8];
            to_cylinder(px, py, pz, qin[3 * i], qin[3 * i + 1], qin[3 * i + 2]);
        }
    }
    // sphere: the pairs (l, |m|) of the moments, in order of l, each with its moments (2 moment +
    // (m < 0)), and groups of at most 8 pairs of one l
    std::vector<int> idx((size_t)(L + 1) * (L + 1), -1), pmom, pout, pm, pl;
    std::vector<int4> groups;
    if (!cyl) {
        std::vector<std::vector<int>> at((size_t)(L + 1) * (L + 1));
        for (size_t k = 0; k < nmom; ++k) {
            const int l = moments[2 * k], m = moments[2 * k + 1];
            at[(size_t)l * (L + 1) + std::abs(m)].push_back((int)(2 * k) + (m < 0));
        }
        for (int l = 0; l <= L; ++l) {
            const int first = (int)pm.size();
            for (int m = 0; m <= l; ++m) {
                const std::vector<int>& v = at[(size_t)l * (L + 1) + m];
                if (v.empty()) continue;
                idx[l * (L + 1) + m] = (int)pm.size();
                pm.push_back(m);
                pl.push_back(l);
                pmom.push_back((int)pout.size());
                pout.insert(pout.end(), v.begin(), v.end());
            }
            for (int p0 = first; p0 < (int)pm.size(); p0 += 8)
                groups.push_back(make_int4(l, p0, std::min(8, (int)pm.size() - p0), 0));
        }
        pmom.push_back((int)pout.size());
        std::reverse(groups.begin(), groups.end());  // whole groups first
    }
    const size_t npair = pm.size();
    // cylinder: the orders n of the moments, ascending, each with its moments
    std::vector<int> ns, nmom0, nout;
    if (cyl) {
        std::vector<std::vector<int>> at(2 * (size_t)L + 1);
        for (size_t k = 0; k < nmom; ++k)
            at[moments[2 * k + 1] < 2 ? 2 * moments[2 * k] : 2 * moments[2 * k] - 1].push_back((int)k);
        for (int n = 0; n <= 2 * L; ++n) {
            if (at[n].empty()) continue;
            ns.push_back(n);
            nmom0.push_back((int)nout.size());
            nout.insert(nout.end(), at[n].begin(), at[n].end());
        }
        nmom0.push_back((int)nout.size());
    }
    // one packed upload of every small input (16-byte aligned pieces)
    std::vector<unsigned char> blob;
    auto put = [&](const void* h, size_t bytes) {
        const size_t off = (blob.size() + 15) / 16 * 16;
        blob.resize(off + bytes);
        if (bytes) memcpy(blob.data() + off, h, bytes);
        return off;
    };
    const size_t o_qin = put(qin.data(), qin.size() * sizeof(double));
    const size_t o_cf = put(class_factors, nq * nclass * sizeof(double));
    const size_t o_mom = put(moments, nmom * 2 * sizeof(int32_t));
    const size_t o_idx = put(idx.data(), idx.size() * sizeof(int));
    const size_t o_groups = put(groups.data(), groups.size() * sizeof(int4));
    const size_t o_pmom = put(pmom.data(), pmom.size() * sizeof(int));
    const size_t o_pout = put(pout.data(), pout.size() * sizeof(int));
    const size_t o_pm = put(pm.data(), pm.size() * sizeof(int));
    const size_t o_pl = put(pl.data(), pl.size() * sizeof(int));
    const size_t o_ns = put(ns.data(), ns.size() * sizeof(int));
    const size_t o_nmom0 = put(nmom0.data(), nmom0.size() * sizeof(int));
    const size_t o_nout = put(nout.data(), nout.size() * sizeof(int));
    MCK(p->mp_in.ensure(blob.size()));
    MCK(p->mp_amp.ensure(nq * nmom * nf * sizeof(double2)));
    MCK(p->mp_out.ensure(nq * (nf + 2) * sizeof(double2)));
    unsigned char* din = p->mp_in.as<unsigned char>();
    auto dptr = [&](size_t off) { return din + off; };
    MCK(cudaEventRecord(p->ev[4], st));
    MCK(cudaMemcpyAsync(din, blob.data(), blob.size(), cudaMemcpyHostToDevice, st));
    MCK(cudaEventRecord(p->ev[0], st));

    // representation cache (rebuilt after staging or for another device type / axis)
    if (s.mp_type != type || !s.mp_valid || (cyl && memcmp(s.mp_axis, axis, sizeof(s.mp_axis)) != 0)) {
        MCK(s.mp_xyz.ensure(nf * na_pad * sizeof(float4)));
        // Atoms sorted by their frame-0 distance from the axis (cylinder) or the origin
        // (sphere): consecutive atoms then have similar Bessel arguments, so a warp's 32
        // Bessel rows take one branch (Miller's recurrence, Hankel's expansion, the power
        // series, the upward recurrence) with similar trip counts. A warp-wide FP64
        // instruction holds the narrow FP64 pipe whatever its active lanes.
        std::vector<float4> f0(na_pad);
        MCK(cudaMemcpyAsync(f0.data(), s.xyz.p, na_pad * sizeof(float4), cudaMemcpyDeviceToHost, st));
        MCK(cudaStreamSynchronize(st));
        std::vector<double> r2(s.na);
        for (size_t j = 0; j < s.na; ++j) {
            const double x = f0[j].x, y = f0[j].y, z = f0[j].z;
            if (cyl) {
                const double px = x * base.e[0] + y * base.e[1] + z * base.e[2];
                const double py = x * base.e[3] + y * base.e[4] + z * base.e[5];
                r2[j] = px * px + py * py;
            } else {
                r2[j] = x * x + y * y + z * z;
            }
        }
        std::vector<int> order(s.na), pos(s.na);
        for (size_t j = 0; j < s.na; ++j) order[j] = (int)j;
        std::stable_sort(order.begin(), order.end(), [&](int u, int v) { return r2[u] < r2[v]; });
        for (size_t k = 0; k < s.na; ++k) pos[order[k]] = (int)k;
        MCK(p->mp_slot.ensure(s.na * sizeof(int)));
        MCK(cudaMemcpyAsync(p->mp_slot.p, pos.data(), s.na * sizeof(int), cudaMemcpyHostToDevice, st));
        MCK(cudaStreamSynchronize(st));
        const int* slot = p->mp_slot.as<int>();
        const size_t n = nf * na_pad;
        const int blocks = (int)grid_blocks(n, 256, 16);
        mp_convert_kernel<<<std::max(blocks, 1), 256, 0, st>>>(s.xyz.as<float4>(), (int)na_pad, (int)s.na, (int)nf, cyl,
                                                                base, slot, s.cls.as<int>(), s.mp_xyz.as<float4>());
        MCK(cudaGetLastError());
        ++launches;
        s.mp_type = type;
        s.mp_valid = true;
        if (cyl) memcpy(s.mp_axis, axis, sizeof(s.mp_axis));
    }
    const double* d_cf = reinterpret_cast<const double*>(dptr(o_cf));
    // frame batches: basis of up to a quarter of the free memory (at most 16 GB), so that
    // one contraction launch has thousands of CTAs
    size_t free_b = 0, total_b = 0;
    MCK(cudaMemGetInfo(&free_b, &total_b));
    const size_t budget = std::max<size_t>((size_t)1 << 28, std::min<size_t>((size_t)16 << 30, free_b / 4));
    if (!cyl) {
        const size_t per_frame = na_pad * (nq * (L + 1) * sizeof(double) + npair * sizeof(int4));
        const size_t nfb = std::max<size_t>(1, std::min<size_t>({nf, budget / per_frame, (size_t)65535}));  // grid y
        const size_t ysm = legendre_bytes(L);
        const size_t jmax_bytes = nfb * nq * (L + 1) * sizeof(unsigned);
        MCK(p->mp_ycf.ensure((ysm + 15) / 16 * 16 + jmax_bytes + nfb * (nq + 1) * sizeof(unsigned)));
        ylm_coeff_kernel<<<1, 64, 0, st>>>(L, legendre_at(p->mp_ycf.p, L));
        MCK(cudaGetLastError());
        ++launches;
        MCK(p->mp_Jb.ensure(nfb * nq * (L + 1) * na_pad * sizeof(double)));
        MCK(p->mp_Yc.ensure(nfb * npair * na_pad * sizeof(int4)));
        // q-vectors of a CTA: as even as they go
        const size_t nqc = (nq + kSumQ - 1) / kSumQ, qb = (nq + nqc - 1) / nqc;
        for (size_t f0 = 0; f0 < nf; f0 += nfb) {
            const int nb = (int)std::min(nfb, nf - f0);
            MpSphereBasis ba{};
            ba.sph = s.mp_xyz.as<float4>();
            ba.cf = d_cf;
            ba.qlen = reinterpret_cast<const double*>(dptr(o_qin));
            ba.idx = reinterpret_cast<const int*>(dptr(o_idx));
            ba.legendre = p->mp_ycf.p;
            ba.jmax = reinterpret_cast<unsigned*>(p->mp_ycf.as<unsigned char>() + (ysm + 15) / 16 * 16);
            ba.redo = MpRedo{ba.jmax + nfb * nq * (L + 1), (int)nq};
            ba.Jb = p->mp_Jb.as<double>();
            ba.Yc = p->mp_Yc.as<int4>();
            ba.na_pad = (int)na_pad;
            ba.nclass = (int)nclass;
            ba.nq = (int)nq;
            ba.L = L;
            ba.npair = (int)npair;
            ba.f0 = (int)f0;
            ba.nfb = nb;
            const size_t ny = (size_t)nb * na_pad, nj = ny * nq;
            mp_ylm_kernel<<<grid_blocks(ny, 128, 64), 128, ysm, st>>>(ba);
            MCK(cudaGetLastError());
            mp_jl_kernel<<<grid_blocks(nj, 128, 16), 128, 0, st>>>(ba);
            MCK(cudaGetLastError());
            ++launches;
            MpSphereContract ca{};
            ca.sph = ba.sph;
            ca.idx = ba.idx;
            ca.Jb = p->mp_Jb.as<double>();
            ca.jmax = ba.jmax;
            ca.Yc = p->mp_Yc.as<int4>();
            ca.legendre = p->mp_ycf.p;
            ca.groups = reinterpret_cast<const int4*>(dptr(o_groups));
            ca.pmom = reinterpret_cast<const int*>(dptr(o_pmom));
            ca.pout = reinterpret_cast<const int*>(dptr(o_pout));
            ca.pm = reinterpret_cast<const int*>(dptr(o_pm));
            ca.pl = reinterpret_cast<const int*>(dptr(o_pl));
            ca.redo = ba.redo;
            ca.A = p->mp_amp.as<double2>();
            ca.na_pad = (int)na_pad;
            ca.na = (int)s.na;
            ca.nq = (int)nq;
            ca.L = L;
            ca.nmom = (int)nmom;
            ca.npair = (int)npair;
            ca.nf = (int)nf;
            ca.f0 = (int)f0;
            MCK(launch_sphere_sum<kSumQ>((int)qb, ca, dim3((unsigned)groups.size(), (unsigned)nb, (unsigned)nqc), st));
            // where the integers' digits do not reach: again in FP64
            MCK(launch_redo(mp_sphere_redo_kernel, ca, nb, ysm, st));
            launches += 3;
        }
    } else {
        const int N = 2 * L;
        const size_t nn = ns.size();
        // as many q-vectors at a time as the basis of one frame has room for (all, but for very
        // large systems)
        const size_t per_q = na_pad * (N + 3) * sizeof(double), angles = na_pad * nn * sizeof(int4);
        // The basis stays with the plan, so no more of it than fills the GPU: 4 GiB, frames in even parts, each
        // of which costs about 0.2 ms of its kernels' ends (10,000 atoms, 1,024 frames, 20 q, 41 orders: 16 GB
        // 148 ms, 4 GiB 151, 2 GiB 157; as many frames as make whole waves of the contraction's CTAs: no gain)
        const size_t cap = std::min(budget, (size_t)4 << 30);
        const size_t nqm = std::max<size_t>(1, std::min<size_t>(nq, cap > angles ? (cap - angles) / per_q : 1));
        const size_t most = std::max<size_t>(1, std::min<size_t>({nf, cap / (nqm * per_q + angles), (size_t)65535}));  // grid y
        const size_t parts = (nf + most - 1) / most, nfb = (nf + parts - 1) / parts;
        MCK(p->mp_Jb.ensure(nfb * nqm * per_q));
        MCK(p->mp_Yc.ensure(nfb * angles));
        MCK(p->mp_ycf.ensure(nfb * (nqm * (N + 4) + 1) * sizeof(unsigned)));  // jmax and the redo words
        MpCylinder ca{};
        ca.cyl = s.mp_xyz.as<float4>();
        ca.Jb = p->mp_Jb.as<double>();
        ca.jmax = p->mp_ycf.as<unsigned>();
        ca.Tc = p->mp_Yc.as<int4>();
        ca.ns = reinterpret_cast<const int*>(dptr(o_ns));
        ca.nmom0 = reinterpret_cast<const int*>(dptr(o_nmom0));
        ca.nout = reinterpret_cast<const int*>(dptr(o_nout));
        ca.mom = reinterpret_cast<const int*>(dptr(o_mom));
        ca.na_pad = (int)na_pad;
        ca.na = (int)s.na;
        ca.nclass = (int)nclass;
        ca.N = N;
        ca.nn = (int)nn;
        ca.nmom = (int)nmom;
        ca.nf = (int)nf;
        const size_t qparts = (nq + nqm - 1) / nqm, fparts = (nf + nfb - 1) / nfb;
        for (size_t part = 0; part < fparts * qparts; ++part) {
            const size_t f0 = part / qparts * nfb, q0 = part % qparts * nqm;
            const size_t nqn = std::min(nqm, nq - q0), nqc = (nqn + kCylQ - 1) / kCylQ;
            const size_t qb = (nqn + nqc - 1) / nqc;  // as even as they go
            ca.f0 = (int)f0;
            ca.nfb = (int)std::min(nfb, nf - f0);
            ca.nq = (int)nqn;
            ca.redo = MpRedo{ca.jmax + nfb * nqm * (N + 3), (int)nqn};
            ca.cf = d_cf + q0 * nclass;
            ca.qcyl = reinterpret_cast<const double*>(dptr(o_qin)) + 3 * q0;
            ca.A = p->mp_amp.as<double2>() + q0 * nmom * nf;
            const size_t na2 = (size_t)ca.nfb * na_pad;
            mp_angle_kernel<<<grid_blocks(na2, 128, 64), 128, 0, st>>>(ca);
            MCK(cudaGetLastError());
            // several CTAs for each that fits, or the last round of rows is shared by few (2 GiB: 21.4 ms with 16)
            mp_jn_kernel<<<grid_blocks(na2 * nqn, 128, 64), 128, 0, st>>>(ca);
            MCK(cudaGetLastError());
            MCK(launch_cylinder_sum<kCylQ>(
                (int)qb, ca, dim3((unsigned)((nn + kSumWarps - 1) / kSumWarps), (unsigned)ca.nfb, (unsigned)nqc), st));
            MCK(launch_redo(mp_cylinder_redo_kernel, ca, ca.nfb, 0, st));
            launches += 4;
        }
    }
    const size_t phase_launches = launches;
    // correlation and average of the amplitudes: moments play the sub-vectors
    EngineConfig cfg;
    cfg.scattering = p->d.scattering;
    cfg.dsp = p->d.dsp_type;
    cfg.method = p->d.dsp_method;
    cfg.precision = p->d.precision;
    cfg.device = p->d.device;
    std::vector<WorkItem> items(1);
    WorkItem& it = items[0];
    it.sys = &s;
    for (size_t i = 0; i <= nq; ++i) it.offs.push_back(i * nmom);
    it.d_cf = d_cf;
    double2* o = p->mp_out.as<double2>();
    it.d_fqt = o;
    it.d_fq = o + nq * nf;
    it.d_fq2 = o + nq * (nf + 1);
    it.d_amp_given = p->mp_amp.as<double2>();
    it.norm = cyl ? 1.0 / (2 * 3.14159265358979323846) : 1.0 / (4 * 3.14159265358979323846);
    int rc = p->eng.prepare(cfg, items, p->msg);
    if (rc) return rc;
    MCK(cudaEventRecord(p->ev[1], st));
    cudaEvent_t ev[4] = {p->ev[8], p->ev[9], p->ev[2], p->ev[3]};
    rc = p->eng.enqueue(st, p->msg, ev);
    if (rc) return rc;
    launches += p->eng.stats().launches;
    std::vector<double2> host(nq * (nf + 2));
    MCK(cudaEventRecord(p->ev[6], st));
    MCK(cudaMemcpyAsync(host.data(), o, host.size() * sizeof(double2), cudaMemcpyDeviceToHost, st));
    MCK(cudaEventRecord(p->ev[7], st));
    MCK(cudaStreamSynchronize(st));
    unsigned flag = 0;
    MCK(cudaMemcpy(&flag, p->eng.err_word(), sizeof(unsigned), cudaMemcpyDeviceToHost));
    if (flag) return fail(p->msg, SASS_ERR_TIMEOUT, "device error flag " + std::to_string(flag));
    memcpy(fqt, host.data(), nq * nf * sizeof(double2));
    memcpy(fq, host.data() + nq * nf, nq * sizeof(double2));
    memcpy(fq2, host.data() + nq * (nf + 1), nq * sizeof(double2));
    float ms = 0;
    if (cudaEventElapsedTime(&ms, p->ev[0], p->ev[1]) == cudaSuccess) p->timing.phase_ms = ms;
    if (cudaEventElapsedTime(&ms, p->ev[9], p->ev[2]) == cudaSuccess) p->timing.corr_ms = ms;
    if (cudaEventElapsedTime(&ms, p->ev[2], p->ev[3]) == cudaSuccess) p->timing.finalize_ms = ms;
    if (cudaEventElapsedTime(&ms, p->ev[4], p->ev[0]) == cudaSuccess) p->timing.h2d_ms = ms;
    if (cudaEventElapsedTime(&ms, p->ev[6], p->ev[7]) == cudaSuccess) p->timing.d2h_ms = ms;
    if (cudaEventElapsedTime(&ms, p->ev[4], p->ev[7]) == cudaSuccess) p->timing.total_ms = ms;
    p->timing.kernel_launches = launches;
    p->timing.phase_launches = phase_launches;
    p->timing.h2d_bytes = blob.size();
    p->timing.d2h_bytes = host.size() * sizeof(double2);
    cudaGetLastError();
    p->msg.clear();
    return SASS_OK;
#undef MCK
}
