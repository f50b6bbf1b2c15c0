// Gridded phase sum (FP32 form) for shells that share one direction set.
//
// With sub-vectors lam_k u_d (the reference's "file" and "sphere" orientation types,
// init_subvectors, src/scatter_devices/abstract_vectors_scatter_device.cpp:112-130) every
// shell of a direction needs the same projections s_j = u_d . r_j. The atoms are spread once
// per direction and frame onto a one-dimensional grid of spacing h, six points each, and every
// shell is then a short sum over the grid,
//     A_k = 1 / D(lam_k h) sum_g G_g exp(i lam_k h (g - off)),
// so that the cost per atom does not grow with the number of shells, whatever their spacing
// (the shell recurrence takes K + 5.5 units per atom for K equally spaced shells, the direct
// kernel about 4 per shell).
//
// Weights. c_n(z), n = 0..5, for an atom at z in [-1/2, 1/2] from the middle of its six points:
// polynomials of degree 5 fitted by least squares so that sum_n c_n(z) exp(i l (o_n - z)),
// o_n = n - 5/2, equals its mean over z, D(l), for all z and all |l| <= pi / sigma. Relative
// error, rms and largest (checked by tests/test_grid_weights.py):
//   set 0: sigma = 3   5.3e-7, 4.4e-6 (at l = pi / sigma)
//   set 1: sigma = 4   5.4e-8, 5.2e-7
// FP32's rounding of u.r alone shifts a phase of 20 revolutions by about 2e-6. Mirror symmetry,
// c_{5-n}(z) = c_n(-z), makes a pair of weights E(z^2) +- z O(z^2).
//
// The grid holds 32-bit integers: shared memory adds integers in place at one access per 32
// lanes (FP32 adds are a read and a write, whose latency a warp also waits for between atoms), in
// any order with the same result, and without the bias that small weights take when they are
// added to a large FP32 sum. The unit is a power of two above the largest sum a grid can reach over
// 2^31, so no cell overflows; a grid of 4,096 atoms rounds each weight to at most 1.1e-6 of the largest
// factor, whatever that is (1e-6 where it is 1), which leaves 2.1e-6 rms in A per atom and unit of that factor at
// most (1.35e-6 at small shells; tests/test_grid_unit.py). S(q,t) averages it over atoms and
// directions: 3e-7 of a row, where the direct kernel's FP32 phases leave 3e-7 to 1e-6.
//
// Layout. A lane owns one (direction, frame) and a column of the grid in shared memory, [g][lane],
// so the adds have no bank conflicts. The 32 lanes of a tile are 32 directions of one frame, or
// 16 x 2 or 8 x 4 for the directions left over. The four warps of a CTA share the grid: each
// takes every fourth block of 32 atoms, and then its share of the shells' transforms. Issue
// and the shared-memory adds bound it: about 31 instructions, six of them adds, per 32 (atom,
// direction, frame), and the transforms of the grid.
//
// Measured on a GB300 (phase kernel; before: shell recurrence, direct kernel for the batch):
//   100,000 atoms x 16 frames x 100 shells x 250 directions     6.3 -> 0.80 ms
//   8 uneven systems, 5 to 30 unevenly spaced shells            11.6 -> 2.8 ms
//   10,000 atoms x 1,024 frames x 20 shells x 500 directions   15.3 -> 7.8 ms
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace sassgpu {

namespace {

constexpr int kGridWarps = 4;          // per CTA, sharing one grid
constexpr int kGridSmem = 227 * 1024;  // per SM
constexpr int kGridChunk = kGridShellChunk;  // shells per pass of a warp over the grid
constexpr float kGridPeak = 0.53f;  // above the largest weight of an atom (0.527, an atom on a grid point)

// Coefficient of z^k of the weight n < 3: set 0 for sigma = 3, set 1 for sigma = 4.
__host__ __device__ constexpr float grid_coef(int set, int n, int k) {
    constexpr float w[2][3][6] = {
        {{7.171509609e-04f, -5.209810681e-03f, 1.596390869e-02f, -2.560331769e-02f, 2.124790385e-02f, -7.218498455e-03f},
         {7.180459045e-02f, -2.050803921e-01f, 2.020282116e-01f, -3.913341562e-02f, -6.357396375e-02f, 3.663669382e-02f},
         {4.274785231e-01f, -3.586962285e-01f, -2.179966732e-01f, 2.453574099e-01f, 4.233535168e-02f, -7.375196538e-02f}},
        {{7.102752722e-04f, -5.313225436e-03f, 1.607830258e-02f, -2.515488315e-02f, 2.101725367e-02f, -7.710096042e-03f},
         {7.182139691e-02f, -2.046424867e-01f, 2.017494126e-01f, -4.103535315e-02f, -6.301073230e-02f, 3.872346649e-02f},
         {4.274683536e-01f, -3.595044715e-01f, -2.178282111e-01f, 2.488705974e-01f, 4.199472601e-02f, -7.760810932e-02f}}};
    return w[set][n][k];
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One warp's share of the sums over the grid, times the class factors, into the amplitudes: chunks
// warp, warp + 4 .. of the shells. The points g and -g (from the point of projection 0) share cos
// and, up to the sign, sin: one paired FMA per shell and pair of points on (G_g + G_-g,
// G_g - G_-g). The transform table streams through `ring` (2 KB) by asynchronous copies of 16
// points x 8 shells: read straight from L2, its latency took as long as the atoms.
// `add`: later parts of the same tile add to what the first wrote.
__device__ __noinline__ void grid_flush(const int* __restrict__ col, float4* __restrict__ ring, int lane, int warp,
                                        const GridSystem& sys, const float* __restrict__ fac, float unit,
                                        float2* __restrict__ dst, bool store, bool add) {
    const size_t row = (size_t)sys.nd * sys.nf;
    const int nb = (sys.off + 2 + 15) / 16;  // batches of points 0, 1 .. off + 1 (the last has no mirror)
    const int nch = (sys.nq + kGridChunk - 1) / kGridChunk;
    const int total = (nch - warp + kGridWarps - 1) / kGridWarps * nb;
    const int* mid = col + sys.off * 32;
    auto load = [&](int i) {
        const int c = warp + i / nb * kGridWarps;
        const float4* from = reinterpret_cast<const float4*>(sys.tw) + ((size_t)c * nb + i % nb) * 64 + lane;
        float4* to = ring + (i & 1) * 64 + lane;
        cp_async16(to, from);
        cp_async16(to + 32, from + 32);
        cp_async_commit();
    };
    float2 tot[kGridChunk], acc[kGridChunk];
#pragma unroll
    for (int k = 0; k < kGridChunk; ++k) tot[k] = make_float2(0.f, 0.f);
    if (total > 0) load(0);
    int g0 = 0, k0 = warp * kGridChunk;
    for (int i = 0; i < total; ++i) {
        if (i + 1 < total) {
            load(i + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncwarp();
        const float4* t4 = ring + (i & 1) * 64;
        const int ng = min(16, sys.off + 2 - g0);
#pragma unroll
        for (int k = 0; k < kGridChunk; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int g = 0; g < ng; ++g) {
            const int gg = g0 + g, x = mid[gg * 32], y = gg > 0 && gg <= sys.off ? mid[-gg * 32] : 0;
            const float2 xy = make_float2(__int2float_rn(x + y), __int2float_rn(x - y));
#pragma unroll
            for (int k = 0; k < kGridChunk; k += 2) {
                const float4 t = t4[(g * kGridChunk + k) / 2];
                acc[k] = __ffma2_rn(xy, make_float2(t.x, t.y), acc[k]);
                acc[k + 1] = __ffma2_rn(xy, make_float2(t.z, t.w), acc[k + 1]);
            }
        }
#pragma unroll
        for (int k = 0; k < kGridChunk; ++k) tot[k] = __fadd2_rn(tot[k], acc[k]);
        __syncwarp();  // this half of the ring is refilled next
        g0 += 16;
        if (g0 < nb * 16) continue;
        if (store) {
#pragma unroll
            for (int k = 0; k < kGridChunk; ++k) {
                if (k0 + k >= sys.nq) break;
                const float b = fac ? __fmul_rn(unit, __ldg(fac + k0 + k)) : unit;
                float2 v = make_float2(__fmul_rn(b, tot[k].x), __fmul_rn(b, tot[k].y));
                float2* p = dst + (k0 + k) * row;
                if (add) v = __fadd2_rn(*p, v);
                *p = v;
            }
        }
#pragma unroll
        for (int k = 0; k < kGridChunk; ++k) tot[k] = make_float2(0.f, 0.f);
        g0 = 0;
        k0 += kGridWarps * kGridChunk;
    }
}

// Both halves' coefficients [set][weight][power of z], operands from constant memory: in registers
// they took 36, and the loop could not be unrolled as far (8.45 -> 8.25 ms paired alone, 7.83 with these
// and sixteen pairs a turn).
struct GridCoef {
    float2 c[2][3][6];
    constexpr GridCoef() : c{} {
        for (int s = 0; s < 2; ++s)
            for (int n = 0; n < 3; ++n)
                for (int k = 0; k < 6; ++k) c[s][n][k].x = c[s][n][k].y = grid_coef(s, n, k);
    }
};
__constant__ GridCoef kGridCoef;

// Adds two atoms, one in each half of the paired FP32 instructions (33 of them; 26 single and 12
// paired ones an atom at a time): their six weights in grid units, rounded by adding 1.5 2^23,
// whose bits are then taken off as an integer.
template <int SET>
__device__ __forceinline__ void grid_add2(const float4 xy, const float4 zw, float2 ux, float2 uy, float2 uz,
                                          float2 bw, unsigned colbase) {
    const float2 magic = make_float2(12582912.f, 12582912.f);
    // the middle of the six points lies between two of them: the half unit puts it on an integer
    const float2 x = __ffma2_rn(make_float2(zw.x, zw.y), uz,
                                __ffma2_rn(make_float2(xy.z, xy.w), uy,
                                           __ffma2_rn(make_float2(xy.x, xy.y), ux, make_float2(-0.5f, -0.5f))));
    const float2 t = __fadd2_rn(x, magic);  // rounds to the nearest integer
    const float2 r = __fadd2_rn(t, make_float2(-12582912.f, -12582912.f));
    const float2 z = __ffma2_rn(r, make_float2(-1.f, -1.f), x), nz = __ffma2_rn(x, make_float2(-1.f, -1.f), r);
    const float2 wt = __fmul2_rn(make_float2(zw.z, zw.w), bw), z2 = __fmul2_rn(z, z);
    const unsigned p0 = colbase + (__float_as_uint(t.x) << 7), p1 = colbase + (__float_as_uint(t.y) << 7);
    const auto& w = kGridCoef.c[SET];
    float2 v[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float2 e = __ffma2_rn(__ffma2_rn(w[i][4], z2, w[i][2]), z2, w[i][0]);
        const float2 o = __ffma2_rn(__ffma2_rn(w[i][5], z2, w[i][3]), z2, w[i][1]);
        v[i] = __ffma2_rn(wt, __ffma2_rn(z, o, e), magic);
        v[5 - i] = __ffma2_rn(wt, __ffma2_rn(nz, o, e), magic);
    }
#define GRID_ADD(P, i, V)                                                                                     \
    asm volatile("red.shared.add.u32 [%0 + %1], %2;" ::"r"(P), "n"((i) * 128), "r"(__float_as_uint(V) - 0x4B400000u) \
                 : "memory")
    GRID_ADD(p0, 0, v[0].x);
    GRID_ADD(p0, 1, v[1].x);
    GRID_ADD(p0, 2, v[2].x);
    GRID_ADD(p0, 3, v[3].x);
    GRID_ADD(p0, 4, v[4].x);
    GRID_ADD(p0, 5, v[5].x);
    GRID_ADD(p1, 0, v[0].y);
    GRID_ADD(p1, 1, v[1].y);
    GRID_ADD(p1, 2, v[2].y);
    GRID_ADD(p1, 3, v[3].y);
    GRID_ADD(p1, 4, v[4].y);
    GRID_ADD(p1, 5, v[5].y);
#undef GRID_ADD
}

template <int SET>
__global__ void __launch_bounds__(kGridWarps * 32, 4) phase_grid_kernel(const GridLaunch a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned s_unit;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* col = reinterpret_cast<int*>(smem) + lane;
    float4* ring = reinterpret_cast<float4*>(smem + a.grid_bytes + warp * a.ring_bytes);
    auto clear = [&](int points) {
        for (int i = threadIdx.x; i < points * 8; i += kGridWarps * 32)
            reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    };
    clear(a.grid_bytes / 128);

    for (;;) {
        if (threadIdx.x == 0) s_unit = atomicAdd(a.counter, 1u);
        __syncthreads();  // also: the grid is clear
        const unsigned unit = s_unit;
        if (unit >= (unsigned)a.ntiles * 8u) break;
        const GridTileDesc td = a.tiles[unit >> 3];
        const GridSystem& sys = a.systems[td.system];
        const int F = 32 >> td.lgd, fb = td.f0 + (int)(unit & 7) * F;  // frames fb .. fb + F
        const bool live = fb < sys.nf;
        const int dl = lane & ((1 << td.lgd) - 1), fl = lane >> td.lgd;
        const int d = td.d0 + min(dl, td.nd - 1);
        const bool act = dl < td.nd && fb + fl < sys.nf;
        // grid units
        const double* u = sys.dirs + 3 * (size_t)d;
        const float ux = (float)(u[0] * sys.inv_h), uy = (float)(u[1] * sys.inv_h), uz = (float)(u[2] * sys.inv_h);
        const bool konst = *sys.konst != 0;
        const unsigned colbase = smem_u32(col) + (unsigned)(sys.off - 2) * 128u - (0x4B400000u << 7);
        float2* dst = sys.out_f32 + (size_t)td.split * sys.split_stride + (size_t)d * sys.nf + fb + fl;
        const float4* src = sys.xyzw + lane;
        const size_t na = sys.na_rec;
        auto load = [&](int b, int slot) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < F)
                    cp_async16(ring + (slot * F + i) * 32 + lane, src + (size_t)min(fb + i, sys.nf - 1) * na + b * 32);
            cp_async_commit();
        };
        for (int b0 = td.b_begin; live && b0 < td.b_end;) {
            // the blocks up to b1 are summed in one grid: one class, or all where the factors
            // weight the atoms, and at most slice_atoms
            const int cls = __ldg(sys.block_class + b0) & 0xffff, end = min(td.b_end, b0 + sys.slice_atoms / 32);
            int b1 = end;
            if (!konst)
                for (b1 = b0 + 1; b1 < end && (__ldg(sys.block_class + b1) & 0xffff) == cls;) ++b1;
            int b = b0 + warp;
            if (b < b1) load(b, 0);
            for (int slot = 0; b < b1; b += kGridWarps, slot ^= 1) {
                const float bw = __ldg(sys.gw + (__ldg(sys.block_class + b) & 0xffff));
                if (b + kGridWarps < b1) {
                    load(b + kGridWarps, slot ^ 1);
                    cp_async_wait<1>();
                } else {
                    cp_async_wait<0>();
                }
                __syncwarp();
                const float4* at = ring + (slot * F + fl) * 32;
#pragma unroll
                for (int j = 0; j < 32; j += 2)
                    grid_add2<SET>(at[j], at[j + 1], make_float2(ux, ux), make_float2(uy, uy), make_float2(uz, uz),
                                   make_float2(bw, bw), colbase);
                __syncwarp();  // this slot is refilled two blocks on
            }
            __syncthreads();
            grid_flush(col, ring, lane, warp, sys, konst ? nullptr : sys.facs + (size_t)cls * sys.nq, sys.gw[sys.nclass],
                       dst, act, b0 > td.b_begin);
            __syncthreads();
            clear(sys.G);
            b0 = b1;
            if (b0 < td.b_end) __syncthreads();
        }
        __syncthreads();  // s_unit has been read by all
    }
}

// Per system: the transform table exp(i lam_k h g) / D, whether the class factors weight the atoms
// (then a slice is summed once; uniform_factors is the same rule, with its reasons); the atoms'
// weights per class in grid units, the unit itself (gw[nclass]) and the factors per class and shell.
__global__ void grid_tables_kernel(const GridSystem* __restrict__ systems, const double* __restrict__ shells) {
    const GridSystem s = systems[blockIdx.y];
    const int nk = (s.nq + kGridChunk - 1) / kGridChunk * kGridChunk;
    const double* lam = shells + s.shell_off;  // [nq] lam_k h in revolutions, then [nq] 1 / D
    const int np = (s.off + 2 + 15) / 16 * 16;  // points 0 .. off + 1 of the mirrored transform, padded
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nk * np; i += gridDim.x * blockDim.x) {
        const int k0 = i / (kGridChunk * np) * kGridChunk, r = i - k0 * np;
        const int g = r / kGridChunk, k = k0 + r % kGridChunk;
        float2 v = make_float2(0.f, 0.f);
        if (k < s.nq && g < s.off + 2) {
            double rev = lam[k] * (double)g;
            rev -= rint(rev);
            double sn, cs;
            sincospi(2.0 * rev, &sn, &cs);
            const double inv = lam[s.nq + k];
            v = make_float2((float)(cs * inv), (float)(sn * inv));
        }
        s.tw[i] = v;
    }
    if (blockIdx.x == 0) {
        __shared__ int differs;
        __shared__ float lo, hi;       // smallest and largest |factor| of the atoms' classes
        __shared__ double sum, count;  // of their squares over the atoms; atoms
        if (threadIdx.x == 0) differs = 0;
        __syncthreads();
        if (threadIdx.x >= 32) {
            for (int i = threadIdx.x - 32; i < s.nq * s.nclass; i += blockDim.x - 32) {
                const int c = i % s.nclass;
                const float b = (float)s.cf[i], b0 = (float)s.cf[c];
                s.facs[(size_t)c * s.nq + i / s.nclass] = b;
                if (!(b == b0) || isinf(b)) differs = 1;
            }
        } else {
            const double* atoms = lam + 2 * s.nq;
            double sq = 0.0, n = 0.0;
            unsigned mn = 0x7f800000u, mx = 0u;
            for (int c = threadIdx.x; c < s.nclass; c += 32) {
                const double na = atoms[c];
                const float b = na > 0.0 ? fabsf((float)s.cf[c]) : 0.f;
                n += na;
                sq = fma(na, (double)b * (double)b, sq);
                if (b != 0.f) {
                    mn = min(mn, __float_as_uint(b));
                    mx = max(mx, __float_as_uint(b));
                }
            }
            mn = __reduce_min_sync(0xffffffffu, mn);
            mx = __reduce_max_sync(0xffffffffu, mx);
            for (int o = 16; o; o >>= 1) {
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
                n += __shfl_xor_sync(0xffffffffu, n, o);
            }
            if (threadIdx.x == 0) {
                lo = __uint_as_float(mn);
                hi = __uint_as_float(mx);
                sum = sq;
                count = n;
            }
        }
        __syncthreads();
        const float bmax = hi != 0.f ? hi : 1.f;
        const int konst = !differs && (hi == 0.f || (bmax <= 16.f * lo && (double)bmax * (double)bmax * count <= 16.0 * sum));
        // units per weight of 1: no sum of slice_atoms atoms reaches 2^31, no weight 2^22
        // times a power of two, so that the factors' products with it are exact: a rounding of
        // the scale is common to all atoms and counts four times in fq2
        const double most = fmin(2.0e9 / (kGridPeak * s.slice_atoms), 4.0e6 / kGridPeak);
        int ex;
        frexp(most / (konst ? bmax : 1.f), &ex);
        const double scale = ldexp(1.0, ex - 1);
        if (threadIdx.x == 0) {
            *s.konst = konst;
            s.gw[s.nclass] = (float)(1.0 / scale);
        }
        for (int c = threadIdx.x; c < s.nclass; c += blockDim.x)
            s.gw[c] = (float)((konst ? (double)fminf(fmaxf((float)s.cf[c], -bmax), bmax) : 1.0) * scale);
    }
}

}  // namespace

double grid_deconvolution(int set, double l) {
    // D(l) = integral over z of sum_n c_n(z) cos(l (o_n - z)): 16-point Gauss-Legendre on
    // [-1/2, 1/2] (degree 31) is exact far below FP32 for |l| <= 2
    static const double x[8] = {0.0950125098376374402, 0.2816035507792589132, 0.4580167776572273863,
                                0.6178762444026437484, 0.7554044083550030339, 0.8656312023878317439,
                                0.9445750230732325761, 0.9894009349916499326};
    static const double wt[8] = {0.1894506104550684963, 0.1826034150449235889, 0.1691565193950025382,
                                 0.1495959888165767321, 0.1246289712555338721, 0.0951585116824927848,
                                 0.0622535239386478929, 0.0271524594117540949};
    double d = 0;
    for (int i = 0; i < 8; ++i)
        for (int sgn = -1; sgn <= 1; sgn += 2) {
            const double z = 0.5 * sgn * x[i];
            double sum = 0;
            for (int n = 0; n < 3; ++n) {
                double p = 0, m = 0, zk = 1;
                for (int k = 0; k < 6; ++k) {
                    p += grid_coef(set, n, k) * zk;
                    m += (k & 1 ? -1.0 : 1.0) * grid_coef(set, n, k) * zk;
                    zk *= z;
                }
                const double o = n - 2.5;
                sum += p * std::cos(l * (o - z)) + m * std::cos(l * (-o - z));
            }
            d += 0.5 * wt[i] * sum;
        }
    return d;
}

// A warp's ring: two blocks of 32 atoms of every staged frame, or two batches of the transform
// table.
static int grid_ring_bytes(int ring_frames) { return std::max(2048, 2 * ring_frames * 512); }

int grid_ctas(int grid_points, int ring_frames) {
    // 1 KB per CTA is the system's
    return std::min(4, kGridSmem / (grid_points * 128 + kGridWarps * grid_ring_bytes(ring_frames) + 2048));
}

cudaError_t launch_grid_tables(const GridSystem* systems, int nsys, int max_points, const double* shells,
                               cudaStream_t st) {
    if (nsys <= 0) return cudaSuccess;
    const int blocks = std::max(1, std::min(64, (max_points + 255) / 256));
    grid_tables_kernel<<<dim3((unsigned)blocks, (unsigned)nsys), 256, 0, st>>>(systems, shells);
    return cudaGetLastError();
}

cudaError_t launch_phase_grid(GridLaunch a, int grid_points, int ring_frames, cudaStream_t st) {
    if (a.ntiles <= 0) return cudaSuccess;
    const int ctas = grid_ctas(grid_points, ring_frames);
    if (ctas < 1) return cudaErrorInvalidValue;
    a.grid_bytes = grid_points * 128;
    a.ring_bytes = grid_ring_bytes(ring_frames);
    const int bytes = a.grid_bytes + kGridWarps * a.ring_bytes;
    const auto kernel = a.set ? phase_grid_kernel<1> : phase_grid_kernel<0>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    const long long units = (long long)a.ntiles * 8;
    const unsigned grid = (unsigned)std::min<long long>((long long)current_sms() * ctas, units);
    kernel<<<grid, kGridWarps * 32, bytes, st>>>(a);
    return cudaGetLastError();
}

}  // namespace sassgpu
