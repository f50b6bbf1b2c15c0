// Host-side launch interface of the sassena_gb300 kernels (internal, not the C ABI).
//
// Every launch works on lists of descriptors so that one launch can cover many
// systems (trajectories) with different atom counts, frame counts, shells and
// direction sets. A single scatter-device computation is a list with one system.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <vector>

namespace sassgpu {

// SM count of the current device, queried once per device. Grids are sized from it, never
// from a fixed count; 1 if the query fails, so grid-stride loops stay valid (only slower).
inline int current_sms() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    static int cache[64] = {0};
    if (dev >= 0 && dev < 64 && cache[dev] > 0) return cache[dev];
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
    if (dev >= 0 && dev < 64) cache[dev] = n;
    return n;
}

// Blocks of `threads` for a grid-stride loop over n items: enough for every item, at most
// per_sm CTAs per SM of the current device, at least one.
inline unsigned grid_blocks(size_t n, int threads, int per_sm) {
    size_t b = (n + (size_t)threads - 1) / (size_t)threads;
    const size_t cap = (size_t)current_sms() * (size_t)per_sm;
    if (b > cap) b = cap;
    return b < 1 ? 1u : (unsigned)b;
}

enum Precision { PREC_FP64 = 0, PREC_FP32 = 1 };
// Transform arithmetic of the long-series path beyond the two forms: float-float (a value
// as an unevaluated sum of two floats, about 44 significant bits) on the FP32 pipe.
constexpr int PREC_FF = 2;

// Device-side error codes written to the plan's error word (first writer wins).
enum DeviceError : unsigned int {
    DEV_OK = 0,
    DEV_MBAR_TIMEOUT = 1,  // an mbarrier wait exceeded its iteration limit
    DEV_BAD_SHAPE = 2,     // a kernel saw a shape outside what its host check allowed
};

// Atom padding granule: every device coordinate row holds a multiple of this many
// atoms, so every staged tile is whole and 16-byte aligned.
constexpr int kAtomGranule = 128;
// Largest padded FFT length of the correlation kernels (NF <= 4096).
constexpr int kMaxLg = 13;

// ---------------------------------------------------------------------------------------
// Phase sum
// ---------------------------------------------------------------------------------------
// Tile shape: q-vectors per lane, warps (= frames) per CTA, atoms per pipeline stage, and
// (FP32 form) pairs of a lane's q-vectors whose sin/cos are evaluated on the FP32 pipe.
struct PhaseShape {
    int q_per_lane;
    int warps;
    int atoms;
    int poly_pairs;
};

struct PhaseSystem {
    const float4* xyz;     // [nf][na_pad] staged coordinates
    const void* bfac;      // [nshell][na_pad] factors: float (FP32) or double (FP64)
    const double* qv;      // [nv][3] sub-vectors of this system
    double2* out;          // FP64 form: amplitudes [nv][nf], or split partials [nsplit][nv][nf]
    float2* out_f32;       // FP32 amplitudes [nv][nf] (one atom split), or FP32 split partials [nsplit][nv][nf]
    size_t split_stride;   // nv * nf
    int na_pad, nf;
};

struct PhaseTileDesc {
    int system, shell;     // shell index into the system's factor rows
    int v0, nv;            // sub-vectors [v0, v0+nv) of the system, nv <= 32 * q_per_lane
    int f0;                // first frame (one per warp)
    int j_begin, j_end;    // atoms (multiples of the stage size)
    int split;             // atom-split slice written by this tile
};

struct PhaseLaunch {
    int precision;
    PhaseShape shape;
    const PhaseSystem* systems;
    const PhaseTileDesc* tiles;
    int ntiles;
    unsigned int* counter;  // work-queue counter, zero before the launch
    unsigned int* err;
    int max_ctas;           // 0: SMs x resident CTAs per SM
};

bool phase_shape_supported(int precision, PhaseShape t);
std::vector<PhaseShape> phase_shapes(int precision);
cudaError_t launch_phase_sum(const PhaseLaunch& a, cudaStream_t st);
// out[i] = sum_s part[s][i] in split order (FP64), stored as double2 or float2.
cudaError_t launch_split_reduce(const double2* part, int nsplit, size_t n, double2* out,
                                cudaStream_t st);
cudaError_t launch_split_reduce_f32(const float2* part, int nsplit, size_t n, float2* out,
                                    cudaStream_t st);

// ---------------------------------------------------------------------------------------
// Fixed-point phase sum (FP64 form): a warp owns 32 q-vectors of any shells and one frame.
// ---------------------------------------------------------------------------------------
struct FxSystem {
    const float4* xyz;      // [nf][na_pad] staged coordinates
    const int* map;         // [na_rec] atom of each class-sorted slot (-1: padding)
    const int* block_info;  // [na_rec / 32] class | padding atoms << 16 of every 32-atom block
    const double* cf;       // [nshell][nclass] class factors
    const double* qv;       // [nv][3] sub-vectors
    const uint4* qw;        // [nv][4] their fixed-point words (launch_fx_q)
    const int* shell_v;     // [nshell+1] sub-vector offsets of each shell
    double2* out;           // amplitudes [nv][nf], or split partials [nsplit][nv][nf]
    size_t split_stride;    // nv * nf
    int na_pad, nf, nshell, nclass;
};

struct FxTileDesc {
    int system;
    int v0, nv;             // sub-vectors [v0, v0+nv), nv <= 32
    int f0;                 // first of 8 frames, one per warp
    int b_begin, b_end;     // 32-atom blocks of the class-sorted slots
    int split, pad;
};

struct FxLaunch {
    const FxSystem* systems;
    const FxTileDesc* tiles;
    int ntiles;
    const void* table;      // launch_fx_table
    unsigned int* counter;  // work-queue counter, zero before the launch
};

constexpr size_t kFxQBytes = 64;            // fixed-point words of one sub-vector
constexpr size_t kFxTableGlobalBytes = 1024 * 16;
cudaError_t launch_fx_table(void* table, cudaStream_t st);
cudaError_t launch_fx_q(const double* qv, size_t nv, void* qw, cudaStream_t st);
cudaError_t launch_phase_fx(const FxLaunch& a, cudaStream_t st);

// ---------------------------------------------------------------------------------------
// Shell-recurrence phase sum (FP32 form): runs of shells lam_k = lam0 + k dlam along
// shared base vectors, evaluated with a three-term recurrence over k.
// ---------------------------------------------------------------------------------------
constexpr int kRecMaxClass = 32;  // scattering classes the recurrence kernel handles

struct RecGroup {
    int system;            // owning system
    int s0, ks;            // shells [s0, s0+ks) of the system, ks <= K
    int pad;
    double lam0, dlam;     // shell s0+k has sub-vectors (lam0 + k dlam) * dirs[d]
};

struct RecSystem {
    const float4* xyzw;       // class-sorted coordinates [nf][na_rec] in pairs; padding atoms at the origin
    const int* block_class;   // [na_rec / 32] class (low 16 bits) | padding atoms << 16 of every 32-atom block
    const double* cf;         // [nq][nclass] class factors
    const double* dirs;       // [nd][3] base vectors (FP64)
    double2* out;             // unused by the FP32-only recurrence (kept for the descriptor layout)
    float2* out_f32;          // FP32 amplitudes [nv][nf] (one split), or FP32 split partials [nsplit][nv][nf]
    size_t split_stride;      // nv * nf
    int na_rec, nf, nd, nclass;
    int g_begin;              // first group of this system in the launch's group list
    int pad;
};

struct RecTileDesc {
    int system;
    int p0, np;            // (group, direction) pairs [p0, p0+np) of the system, np <= 32
    int f0;                // first frame (one per warp)
    int j_begin, j_end;    // atoms of the class-sorted rows (multiples of 128; may be empty)
    int split;
    int pad;
};

struct RecLaunch {
    int K;                     // shells per lane (a value of rec_shell_counts())
    const RecSystem* systems;
    const RecGroup* groups;
    const RecTileDesc* tiles;
    int ntiles;
    float* bfac;               // [ngroups][kRecMaxClass][K] filled by launch_rec_factors
    unsigned int* counter;     // work-queue counter, zero before the launch
    unsigned int* err;
    int max_ctas;
};

std::vector<int> rec_shell_counts();
bool rec_shells_supported(int K);
cudaError_t launch_rec_factors(const RecLaunch& a, int ngroups, cudaStream_t st);
cudaError_t launch_phase_rec(const RecLaunch& a, cudaStream_t st);
// dst[f][j] = src[f][map[j]] with w = 1, or a zero row entry with w = 0 where map[j] < 0
cudaError_t launch_permute_stage(const float4* src, int na_pad_src, const int* map, int na_dst, int nf,
                                 float4* dst, cudaStream_t st);

// ---------------------------------------------------------------------------------------
// Gridded phase sum (FP32 form): all shells of a direction from one grid of its projections.
// ---------------------------------------------------------------------------------------
struct GridSystem {
    const float4* xyzw;       // class-sorted coordinates [nf][na_rec] in pairs, w = 0 for padding atoms
    const int* block_class;   // [na_rec / 32] class | padding atoms << 16
    const double* cf;         // [nq][nclass] class factors
    const double* dirs;       // [nd][3] base vectors
    float2* out_f32;          // FP32 amplitudes [nv][nf] (one split), or FP32 split partials
    size_t split_stride;      // nv * nf
    double inv_h;             // 1 / grid spacing (along a base vector)
    // filled by launch_grid_tables
    float2* tw;               // [nq / 8 rounded up][off + 2 rounded up to 16][8]
    float* facs;              // [nclass][nq]
    float* gw;                // [nclass + 1]
    int* konst;
    int na_rec, nf, nd, nclass, nq;
    int G, off;               // grid points; the point of projection 0
    int shell_off;            // of the system's [2][nq] shell constants and [nclass] atoms of each class
    int slice_atoms;          // most atoms summed in one grid (a multiple of 32)
};

struct GridTileDesc {
    int system;
    int d0, nd, lgd;          // directions [d0, d0+nd), nd <= 2^lgd (32, 16 or 8)
    int f0;                   // 8 units of 32 / 2^lgd frames
    int b_begin, b_end;       // 32-atom blocks (not empty)
    int split;
};

struct GridLaunch {
    const GridSystem* systems;
    const GridTileDesc* tiles;
    int ntiles;
    unsigned int* counter;    // work-queue counter, zero before the launch
    int set;                  // weights
    int grid_bytes, ring_bytes;  // set by launch_phase_grid
};

constexpr int kGridShellChunk = 8;
// Atoms of one grid: the unit of its integers grows with them (rounding a weight to at most 1.1e-6 of
// the largest factor at 4,096, to 4.4e-6 at 16,384). Slices are made no longer than the first; the
// second is the limit (100,000 atoms, 64 frames, 200 x 2,000: 20 slices of 5,000 atoms 31.5 ms,
// each as two grids 44).
constexpr size_t kGridMaxSlice = 4096, kGridMaxSum = 16384;
constexpr double kGridSigma[2] = {3.0, 4.0};  // grid points per half period at the largest shell, per weight set
// D(l) of the weights `set`; CTAs per SM for that many grid points and staged frames (0: too many)
double grid_deconvolution(int set, double l);
int grid_ctas(int grid_points, int ring_frames);
// shells: per system [nq] lam_k h / 2 pi, then [nq] 1 / D(lam_k h), then [nclass] atoms
cudaError_t launch_grid_tables(const GridSystem* systems, int nsys, int max_points, const double* shells,
                               cudaStream_t st);
cudaError_t launch_phase_grid(GridLaunch a, int grid_points, int ring_frames, cudaStream_t st);

// ---------------------------------------------------------------------------------------
// Correlation, store and orientational average
// ---------------------------------------------------------------------------------------
enum DspType { DSP_AUTOCORRELATE = 0, DSP_SQUARE = 1, DSP_PLAIN = 2 };

// Per-system data of the correlation kernels.
struct CorrSystem {
    const void* A;          // coherent amplitudes [nv][nf]: float2 (FP32) or double2 (FP64)
    const float4* xyz;      // incoherent: staged coordinates [nf][na_pad]
    const void* bfac;       // incoherent: factors [nshell][na_pad]
    const double* qv;       // sub-vectors [nv][3]
    const int* shell_v;     // [nshell+1] sub-vector offsets of each shell
    const void* kbr;        // [L] bit-reversed store kernel: float2 (FP32) or double2 (FP64)
    const float4* qrev;     // FP32 form: sub-vectors in revolutions (q / 2 pi) [nv]
    const uint4* qw;        // fixed-point form: the sub-vectors' words (launch_fx_q)
    double cx, cy, cz;      // frame centre (FP32 form) for the plain-dsp phase restore
    int nf, lg, na_pad;
};

// FP32 form: out[v] = (float)(q[v] / 2 pi) once per call, so that the series kernels read the
// sub-vectors they need per (atom, direction) pair without FP64 conversions.
cudaError_t launch_q_revolutions(const double* qv, size_t nv, float4* out, cudaStream_t st);

// Work unit: series [v_begin, v_end) (coherent) or atoms [v_begin, v_end) with all the
// shell's directions (incoherent) of one shell of one system, into one partial slot.
struct CorrChunk {
    int system, shell, v_begin, v_end;
    size_t part_off;        // offset (in doubles) of this slot's partial spectrum / series
    int slot;               // index into apart / a2part
    int pad;
};

struct CorrLaunch {
    int precision, dsp;
    const CorrSystem* systems;
    const CorrChunk* chunks;
    int nchunks;
    int lg_max;             // largest padded length of the batch (shared memory sizing)
    int lg_min;             // smallest padded length (0: not known)
    int nf_max;
    const void* tw;         // [L_max/2] exp(-2 pi i k / L_max), float2 or double2
    int restore_phase;      // FP32 form with dsp=plain: multiply by exp(i q.c)
    double* ppart;          // partial spectra / series (see CorrChunk::part_off)
    double2* apart;         // [nslot]
    double* a2part;         // [nslot]
    unsigned int* err;
    const void* fx_table;   // fixed-point form: launch_fx_table
};

cudaError_t launch_corr_accumulate(const CorrLaunch& a, cudaStream_t st);  // coherent
cudaError_t launch_self_accumulate(const CorrLaunch& a, cudaStream_t st);  // incoherent
// Incoherent autocorrelation of the FP64 form in fixed point (padded lengths 64 .. 256, one length
// per launch). Few large chunks: a CTA fills an SM.
bool self_fx_supported(int precision, int dsp, int lg_min, int lg_max);
cudaError_t launch_self_fx(const CorrLaunch& a, cudaStream_t st);

// Per-shell finalisation entry.
struct FinalEntry {
    int slot_begin, slot_end;  // partial slots of this shell (consecutive)
    size_t part_off;           // offset of slot_begin's partial; slots are `part_len` apart
    int part_len;              // L (autocorrelate) or 2*nf (square/plain) doubles per slot
    int f32pair;               // partials are FP32 (Kahan sum, compensation) pairs, not doubles
    int nf, lg;
    double inv_nm;
    double2* fqt;              // [nf]
    double2* fq;
    double2* fq2;
};

// The series [nv][nf] of a shell whose last kTailLags lags are summed directly (A and A64 nullptr: they
// come from the transforms like the others).
constexpr int kTailLags = 8;
struct TailEntry {
    const float2* A;
    const double2* A64;  // FP64 form
    size_t nv;
};

struct FinalLaunch {
    int dsp, conj_out;
    const FinalEntry* entries;
    int nentries;
    int lg_max;
    const double* ppart;
    const double2* apart;
    const double* a2part;
    const double2* tw;         // [L_max/2] FP64
    const TailEntry* tails;    // one per entry, or nullptr: none
    int tails64;               // whether they are FP64 series
};
cudaError_t launch_finalize(const FinalLaunch& a, cudaStream_t st);

// Shared memory of the FFT accumulate kernels for padded length 2^lg.
size_t fft_smem_bytes(int precision, int lg, int nf, bool self);
// Whether the autocorrelation kernels of a launch write their power partials as FP32
// (sum, compensation) pairs (FinalEntry::f32pair): the FP32 form's CTA-per-series kernels.
bool corr_writes_f32_pairs(int precision, int dsp, int lg_max);

// ---------------------------------------------------------------------------------------
// Long series (autocorrelation with padded length 2^14 .. 2^20): four-step FFT through HBM,
// L = R x C with C = 2^kLongRowLg and R = L / C. Spectra are kept in (k1, bit-reversed k2)
// order: index k1 * C + bitrev(k2) holds frequency k1 + R k2.
// ---------------------------------------------------------------------------------------
constexpr int kLongRowLg = 12;
constexpr int kLongLgMax = 20;

struct LongArgs {
    int precision, lg, nf;     // precision of the transforms (Y, twiddles, K)
    int amp_f32;               // the series are float2 (else double2)
    const void* A;             // series [nseries][nf]: the batch's first series
    void* Y;                   // [nseries][L] T2 scratch (column-pass output)
    int nseries;
    const void* tw;            // W_L^j for j < L/2 (T2 of the precision)
    const CorrChunk* chunks;   // row pass: chunk series v reads Y[v - v0]
    int nchunks, v0;
    const void* kbr;           // store kernel K in the long order (T2)
    double* ppart;             // power partial slots (chunk.part_off, L doubles per slot)
    double2* mpart;            // [nv][R] row parts of the series means
    void* xout;                // transform mode: conj(X) in the long order (T2)
};
// Float-float copy (16 bytes per complex value) of an FP64 table: the twiddles and the store
// kernel of the long path's float-float transforms.
cudaError_t launch_to_ff2(const double2* src, size_t n, void* dst, cudaStream_t st);
// Column pass over the batch's series; row pass over its chunks (power, means).
cudaError_t launch_long_columns(const LongArgs& a, cudaStream_t st);
cudaError_t launch_long_rows(const LongArgs& a, cudaStream_t st);
// One series' transform (nseries = 1): xout = conj(FFT_L(x)).
cudaError_t launch_long_transform(const LongArgs& a, cudaStream_t st);
// Incoherent long series: G[p - p0][t] = b_j exp(i q_m . r_j(t)) for pairs p = j * nm + m of
// one shell, p in [p0, p0 + nseries).
struct LongSelfArgs {
    int precision, nf, na_pad, nm, p0, nseries;
    const float4* xyz;         // [nf][na_pad]
    const void* bfac;          // the shell's factor row [na_pad] (T)
    const double* qv;          // the shell's q-vectors [nm][3]
    const float4* qrev;        // FP32 form: the same in revolutions [nm]
    void* G;                   // [nseries][nf] T2
};
cudaError_t launch_long_self_series(const LongSelfArgs& a, cudaStream_t st);
// afinal / a2final partials of every long chunk from the row parts of its series means.
cudaError_t launch_long_means(const CorrChunk* chunks, int nchunks, const double2* mpart, int R, double2* apart,
                              double* a2part, cudaStream_t st);

struct LongFinal {
    const FinalEntry* entries;
    int nentries, lg, conj_out;
    const double* ppart;
    const double2* apart;
    const double* a2part;
    const double2* tw;         // W_L^j, j < L/2, FP64
    double2* Z;                // [nentries][L] scratch
    const double2* A;          // coherent FP64: amplitudes [nv][nf] and sub-vector offsets
    const int* shell_v;        //   [nentries+1] for the directly summed last lags (null: none)
};
cudaError_t launch_long_finalize(const LongFinal& a, cudaStream_t st);
// K of a long system: K(k) = sum_{tau<nf} exp(+2 pi i k tau / L) / (nf L (nf - tau)) in the long
// order, FP64 and FP32 copies; scratch holds nf + L double2.
cudaError_t launch_long_store_kernel(const double2* tw64, int lg, int nf, double2* scratch, double2* k64,
                                     float2* k32, cudaStream_t st);

// FFT tables on the device: tw[k] = exp(-2 pi i k / L) (k < L/2) in FP64 and FP32, and
// the store kernel K at bit-reversed positions for (nf, lg).
cudaError_t launch_twiddles(double2* tw64, float2* tw32, int lg, cudaStream_t st);
cudaError_t launch_store_kernel(const double2* tw64, int lg_tw, double2* k64, float2* k32, int nf,
                                int lg, cudaStream_t st);

// Staging: raw frame-major float [nf][na][3] -> float4 [nf][na_pad] (minus centre); with
// xyz_rec, also the class-sorted copy with atom j at rec_inv[j] (x, y, z, 1). `raw` may be
// host memory the device reads in place.
// With `rmax2` (zeroed by the caller) also the largest |r|^2 of the staged frames, as float bits.
cudaError_t launch_stage(const float* raw, int nf, int na, int na_pad, double cx, double cy,
                         double cz, int center, float4* xyz, const int* rec_inv, int na_rec,
                         float4* xyz_rec, unsigned int* rmax2, cudaStream_t st);
// b[s][j] = class_factors[s][cls[j]] (0 for padding atoms), float or double output.
cudaError_t launch_expand_factors(const double* class_factors, int nclass, int nshell,
                                  const int* cls, int na_pad, int precision, void* b,
                                  cudaStream_t st);

}  // namespace sassgpu
