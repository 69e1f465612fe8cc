// Split-precision back-projection kernels (the fast path).
//
// Work unit: one CTA = one tile of 1024 output pixels (256 threads x 4 pixels),
// looping over its pulses in shared-memory chunks.  Precision plan (per pixel p,
// pulse n, tile centre c; the wide-precision work is per tile or per (tile, pulse), in
// two-float FP32 from the FP64 inputs split once into hi + lo):
//
//   d(p,n) = R + L + eps,    R = |c - pos_n| (two-float, per tile-pulse)
//                            L = u . delta_p  (u = (c - pos_n)/R, delta_p = p - c)
//                            eps = |delta_p x u|^2 / (R + L + d)   (<= ~1 cm, FP32)
//   phase turns = frac(K R + phase_n / 2pi)            two-float -> FP32, per tile-pulse
//               + frac(K u . delta_p)                  exact: W_hi . delta_hi
//               + W_hi . delta_lo + W_lo . delta_p     FP32, tiny terms
//               + K eps - K r_p (polar demodulation, per pixel)
//
// with K = k / 2pi, W = K u.  W_hi is a multiple of 2^eW with <= 10 significant
// bits and delta_hi a multiple of 2^ed with <= 12 (2-D) / 11 (3-D) bits, so each
// product and their sum are exact in FP32 and the large linear phase term is
// reduced modulo one turn without rounding.  The reduced phase feeds the
// hardware sin/cos (MUFU) on [-pi, pi).
//
// Lattice tiles go further: delta_p = i s_row + j s_col, so u . delta_p and W . delta_p are
// sums of a row and a column term.  The records carry the two terms per pulse (the phase
// ones split exactly as above), each thread forms range and phase once per pulse at the middle
// of a run of eight rows and steps along the run by their Taylor series: per pixel-pulse
// only two short polynomials, the window gather and the rotation remain.
//
// Range interpolation: for each (tile, pulse) the chunk stages the range bins
// the tile can touch as Horner coefficients of the reference's four-point
// Lagrange cubic (weight folded in), 32 bytes per bin; a pixel-pulse is then
// two 16-byte shared loads and six FMAs.  Bins whose taps leave the row are
// stored as zero, which reproduces the reference's support rule
// (fast_bp/ffbp.py:27).  A pulse whose window would not fit the staged bins, or that lies
// outside the precision envelope, runs through a two-float per-sample fallback instead.
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace sarbp {
namespace {

constexpr int kThreads = kSplitThreads;
constexpr int kPX = 4;
constexpr int kPointPX = kPointTile / kThreads;  // pixels per thread of the points kernel
// Threads of the single-scene merge kernel: four column pairs of parent pixels per thread (more
// gathers in flight per warp than two pairs at 256 threads).
constexpr int kMergeThreads = 128;
constexpr int kMaxRows = kSplitTilePixels >> 2;  // tile_lc >= 2
constexpr int kMaxCols = 32;                     // tile_lc <= 5
constexpr int kColRun = 8;                       // angle columns per run of a polar tile
constexpr int kMaxMids = kMaxCols / kColRun;
constexpr int kMergeRun = 8;                     // parent rows per run of a merge tile
constexpr int kMergeRows = kMaxRows / kMergeRun; // runs per tile column, at most
constexpr int kMaxChunk = 64;      // pulses per chunk of the direct kernels: two warps compute the records
constexpr int kMaxLeafChunk = 32;  // pulses per chunk of the FFBP leaf kernels: one warp computes the records
// Window bytes per CTA: with kMaxChunk records this keeps three CTAs per SM within 227 KB.
constexpr int kWindowBudget = 68 * 1024;
// Lattice tiles (64 registers): four CTAs per SM.  Per CTA, 49 KB of windows, 5 KB of 80-byte
// records, up to 1.25 KB of static shared memory (the batch kernel) and the 1 KB the runtime
// reserves: 4 x 56.25 KB fits the SM's 228 KB.  The packed windows of a 32 x 32 tile at the
// usual geometries need 15-25 bins per pulse, so 64-pulse chunks mostly fit; wider windows
// just fit fewer pulses per chunk (the image does not depend on the chunking).
constexpr int kLatticeWindowBudget = 49 * 1024;
#ifndef SARBP_BULK_WINDOWS
#define SARBP_BULK_WINDOWS 0
#endif
// Bulk-copy window staging (SARBP_BULK_WINDOWS = 1): each pulse's raw samples arrive in shared
// memory by one cp.async.bulk copy (completion on an mbarrier) before the Horner transform,
// instead of the transform's own global loads.  The raw samples need room beside the windows:
// per window bin 8 bytes plus five samples of margin per pulse, so the window budgets shrink to
// keep the same CTAs per SM.
constexpr int kBulkMargin = 5;
__host__ __device__ constexpr int raw_bytes_for(int cap, int chunk) {
    return SARBP_BULK_WINDOWS ? (cap + kBulkMargin * chunk) * 8 + 16 : 0;
}
// K rho^2 / R limits (turns) for the FP32 eps term: direct BP targets 1e-5 relative
// error, FFBP leaves 1e-4.
constexpr double kDirectEnvelope = 8.0;

struct Rec {
    float4 a;  // W_hi.x, W_hi.y, W_lo.x, W_lo.y   (lattice adjoint: B_row hi, lo, B_col hi, lo;
               // lattice forward: B_row / 2 and B_col modulo one turn in 2^-32 turns, integers)
    float4 b;  // u.x, u.y, 2R, frac(Q) - 1/2       (lattice: u.s_row, u.s_col, 2R (forward: R), frac(Q) - 1/2)
    float4 c;  // Phi, window bias bits, window offset bits, window count - 1 bits
               // (lattice forward: Phi' in 2^-32 turns, window byte base, 2 pi frac(B_row), 12.5 e4: see lattice_runs;
               // points: a = W in 2^-16 turns/m and Phi in 2^-32 turns, e = u / dr in 2^-12 bins/m and c.x the
               // middle's place in the window in 2^-28 bins (integers); b = u, 2R; c.y that place, FP32;
               // d = rest of W, rest of u.x / dr; e.w rest of u.y / dr)
    float4 d;  // u.z, W_hi.z, W_lo.z                (polar runs: -2 pi K a.x, -2 pi K a.y with a = pos - origin, the
               // limit of column_run; lattice adjoint: 2 pi frac(m B_row), u.x, u.y, u.z; lattice forward: the start phases
               // of even and odd pixels from Phi', radians)
    float4 e;  // lattice adjoint: the pairs (2R, 2R), (frac(Q) - 1/2, frac(Q) - 1/2) of packed-FP32 operands;
               // lattice forward: (-, window bias bits, window offset bits, window count - 1 bits)
};

// Where the chunk driver keeps a pulse's window placement: c, or e in the lattice forward records.
template <int MODE>
__device__ __forceinline__ float4& rec_window(Rec& r) { return MODE == 1 ? r.e : r.c; }
template <int MODE>
__device__ __forceinline__ const float4& rec_window(const Rec& r) { return MODE == 1 ? r.e : r.c; }

struct Pix {
    float dx, dy, dz;
    float dxh, dyh, dzh;
    float dxl, dyl, dzl;
    float d2, psi;
    float ar, ai;
};

// A point's offset from the tile centre: FP32 plus rest (the fallback's two-float), and as a whole number of
// 2^-16 m plus rest for the phase.
struct PointPix {
    float dx, dy, dz;     // FP32
    float lx, ly, lz;     // offset - dx
    int ix, iy, iz;       // rint(2^16 dx)
    float rx, ry, rz;     // offset - 2^-16 ix
    float d2;
    float ar, ai;
};

struct TileShared {
    double cx, cy, cz;
    float ch[3], cl[3];         // the centre as two-float (hi + lo), for the FP32 records
    float rhof;
    double rho;                 // bound on |delta_p| (m)
    double scale_d, inv_scale_d;
    double sum[4];
    float bnd[3];               // bounds on |delta_x|, |delta_y|, |delta_z| (m)
    float scale_f, inv_scale_f; // FP32 offset quantum of polar merge tiles
    float red[8][8];
    int base[kMaxChunk];        // global bin of window entry 0, per pulse of the chunk
    float wt[kMaxChunk];
    float rest[kMaxChunk];      // points: the z part of the range scale's rest (see points_chunk)
    int nfit;
    int nfit_w[2];              // fitting pulses among each record warp's 32
    unsigned miss_w[2];         // pulses of each record warp that cannot be staged (bit per lane)
    int wsum;                   // window entries of record warp 0's pulses
    float sth[6], stl[6];       // lattice tiles: step_row (0-2) and step_col (3-5) as two-float
    int row_step;               // lattice tiles: rows between a thread's successive pixels
#if SARBP_BULK_WINDOWS
    int roff[kMaxChunk];        // bulk staging: first raw sample of each pulse in shared memory
    long long raw0[kMaxChunk];  // bulk staging: data-array index of that sample
#endif
};

// Row/column tables of a polar tile; aliased onto the window region during set-up.
struct PolarTables {
    double rx[kMaxRows], ry[kMaxRows];
    float rxh[kMaxRows], rxl[kMaxRows], ryh[kMaxRows], ryl[kMaxRows], dg[kMaxRows], psi[kMaxRows];
    double cxd[kMaxCols + kMaxMids], cyd[kMaxCols + kMaxMids];  // the columns, then the middles of their runs
    float cxh[kMaxCols + kMaxMids], cxl[kMaxCols + kMaxMids], cyh[kMaxCols + kMaxMids], cyl[kMaxCols + kMaxMids];
    float dcs[kMaxCols + kMaxMids], duu[kMaxCols + kMaxMids];
    float mid_c[kMaxMids], mid_u[kMaxMids];
};

struct SplitParams {
    PulseInputs in;
    float2* out;           // direct jobs: output image (pulse split s writes out + s * split_stride)
    long long out_stride;
    double K;              // k / 2pi (turns per metre)
    double inv_dr;         // 1 / data_dr
    double scale_w, inv_scale_w;
    float Kf, inv_drf;
    int chunk;             // pulses per chunk (<= kMaxChunk)
    int cap;               // window entries (32 bytes each) available per chunk
    int pulse_split;
    long long split_stride;
    // Precision envelope of the FP32 eps term: the fast path needs K rho^2 / R <= envelope
    // (the FP32 error of eps is ~2.5e-7 * rho^2 / R metres, i.e. ~2.5e-7 * envelope turns).
    double envelope;
    // Two-float (hi + lo) copies for the FP32 fallback of pulses outside the envelope.
    float Kh, Kl, rsh, rsl, idrh, idrl;
};

struct Job {
    PolarDesc g;          // polar grids
    sarbp_lattice lat;    // lattices
    const double* xyz;    // point lists
    const int* index;     // the point at each place of the list's spatial order, or NULL
    int p_begin, p_end;   // the points of the tile (or of a stretch of it)
    int tile_r, tile_u, lc;
    int p0, p1;
};

// (v, v): an operand of the packed FP32 (f32x2) instructions.
__device__ __forceinline__ float2 pair(float v) { return make_float2(v, v); }

// ---- block reductions (256 threads) ---------------------------------------------
template <int N>
__device__ __forceinline__ void block_max(TileShared& S, float v[N]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] = fmaxf(v[i], __shfl_xor_sync(0xffffffffu, v[i], o));
    }
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) S.red[warp][i] = v[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float m = S.red[0][i];
#pragma unroll
        for (int w = 1; w < 8; ++w) m = fmaxf(m, S.red[w][i]);
        v[i] = m;
    }
    __syncthreads();
}

__device__ __forceinline__ void block_sum4(TileShared& S, double v[4]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ double part[8][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) part[warp][i] = v[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i) {
            double s = 0.0;
            for (int w = 0; w < 8; ++w) s += part[w][i];
            S.sum[i] = s;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = S.sum[i];
    __syncthreads();
}

// v as an unevaluated sum h + l of two FP32 numbers.
__device__ __forceinline__ void split2(double v, float& h, float& l) {
    h = (float)v;
    l = (float)(v - (double)h);
}

__device__ __forceinline__ void set_quantum(TileShared& S, float bound, int bits) {
    int e;
    frexp((double)bound, &e);
    S.scale_d = ldexp(1.0, e - bits);
    S.inv_scale_d = ldexp(1.0, bits - e);
}

__device__ __forceinline__ void pixel_from_offsets(const TileShared& S, double ox, double oy, double oz, Pix& P) {
    quantize(ox, S.scale_d, S.inv_scale_d, P.dxh, P.dxl);
    quantize(oy, S.scale_d, S.inv_scale_d, P.dyh, P.dyl);
    quantize(oz, S.scale_d, S.inv_scale_d, P.dzh, P.dzl);
    P.dx = (float)ox;
    P.dy = (float)oy;
    P.dz = (float)oz;
    P.d2 = P.dx * P.dx + P.dy * P.dy + P.dz * P.dz;
}

// ---- per-tile set-up: tile centre, quantum, per-pixel offsets -------------------
// Polar tile: rows/cols of a polar grid window; separable FP64 row and column
// tables give each pixel offset as an exact hi part plus an FP32 remainder.
// The tables and the tile's centre and bounds; RUNS: also the middles of the runs of columns.
template <bool RUNS>
__device__ void polar_tables(const SplitParams& P, const Job& J, TileShared& S, PolarTables& T, bool demodulate) {
    const PolarDesc& g = J.g;
    const int tid = threadIdx.x;
    const int cols_t = 1 << J.lc, rows_t = kSplitTilePixels >> J.lc;
    const double oz = g.oz, side = (double)g.side;
    const int i0 = g.win_r0 + J.tile_r + (rows_t >> 1);
    const int j0 = g.win_u0 + J.tile_u + (cols_t >> 1);
    const double rc = g.r0 + (double)i0 * g.dr;
    const double gc = sqrt(fmax(0.0, rc * rc - oz * oz));
    const double uc = g.u0 + (double)j0 * g.du;
    const double cc = sqrt(fmax(0.0, 1.0 - uc * uc));
    float m[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (tid < rows_t) {
        const double r = g.r0 + (double)(g.win_r0 + J.tile_r + tid) * g.dr;
        const double dg = sqrt(fmax(0.0, r * r - oz * oz)) - gc;
        const double rx = side * dg * cc, ry = dg * uc;
        T.rx[tid] = rx;
        T.ry[tid] = ry;
        T.dg[tid] = (float)dg;
        const double t = -P.K * r;
        T.psi[tid] = demodulate ? (float)(t - rint(t)) : 0.0f;
        m[0] = (float)fabs(rx);
        m[1] = (float)fabs(ry);
        m[2] = (float)fabs(dg);
    }
    if (tid < cols_t) {
        const double u = g.u0 + (double)(g.win_u0 + J.tile_u + tid) * g.du;
        const double dc = sqrt(fmax(0.0, 1.0 - u * u)) - cc, du = u - uc;
        const double cx = side * gc * dc, cy = gc * du;
        T.cxd[tid] = cx;
        T.cyd[tid] = cy;
        T.dcs[tid] = (float)(side * dc);
        T.duu[tid] = (float)du;
        m[3] = (float)fabs(cx);
        m[4] = (float)fabs(cy);
        m[5] = (float)fabs(dc);
        m[6] = (float)fabs(du);
    }
    const int groups = cols_t / kColRun, mid = tid - kMaxCols;
    if (RUNS && mid >= 0 && mid < groups) {
        const double u = g.u0 + ((double)(g.win_u0 + J.tile_u + kColRun * mid) + 0.5 * (kColRun - 1)) * g.du;
        const double c = sqrt(fmax(0.0, 1.0 - u * u)), dc = c - cc;
        T.cxd[tid] = side * gc * dc;
        T.cyd[tid] = gc * (u - uc);
        T.dcs[tid] = (float)(side * dc);
        T.duu[tid] = (float)(u - uc);
        T.mid_c[mid] = (float)c;
        T.mid_u[mid] = (float)u;
    }
    block_max<7>(S, m);
    // Bounds on |delta_x|, |delta_y| (slightly enlarged for the FP32 maxima).
    const float bx = (m[0] + m[3] + m[2] * m[5]) * 1.0001f + 1e-6f;
    const float by = (m[1] + m[4] + m[2] * m[6]) * 1.0001f + 1e-6f;
    if (tid == 0) {
        S.cx = g.ox + side * gc * cc;
        S.cy = g.oy + gc * uc;
        S.cz = 0.0;
        S.rho = sqrt((double)bx * bx + (double)by * by);
        S.bnd[0] = bx;
        S.bnd[1] = by;
        S.bnd[2] = 0.0f;
        set_quantum(S, fmaxf(bx, by), 12);
        if (RUNS) {  // for the records: centre - origin, and bounds of the runs' expansion (see make_record)
            split2(side * gc * cc, S.sth[0], S.stl[0]);
            split2(gc * uc, S.sth[1], S.stl[1]);
            const float um = fabsf((float)uc) + m[6], h = fabsf((float)g.du);
            const float ic = rsqrtf(fmaxf(1.0f - um * um, 0.0f)), hc = h * ic, hcc = hc * ic, u2 = um * um;
            const float e2 = 0.5f * hc * hc * ic, q4 = e2 * 0.25f * hcc * hcc;  // times (1 + 4 u^2): the fourth order
            S.sth[2] = q4 * (um * hcc * (3.0f + 4.0f * u2) * 525.3f +
                             hcc * hcc * 0.5f * (1.0f + 12.0f * u2 + 8.0f * u2 * u2) * 1838.4f);
            S.sth[3] = 3.5f * hc;
            S.sth[4] = 12.25f * e2;
        }
    }
    __syncthreads();
    if (tid < rows_t) {
        quantize(T.rx[tid], S.scale_d, S.inv_scale_d, T.rxh[tid], T.rxl[tid]);
        quantize(T.ry[tid], S.scale_d, S.inv_scale_d, T.ryh[tid], T.ryl[tid]);
    }
    if (tid < cols_t || (RUNS && mid >= 0 && mid < groups)) {
        quantize(T.cxd[tid], S.scale_d, S.inv_scale_d, T.cxh[tid], T.cxl[tid]);
        quantize(T.cyd[tid], S.scale_d, S.inv_scale_d, T.cyh[tid], T.cyl[tid]);
    }
    __syncthreads();
}

__device__ __forceinline__ void polar_pixels(const Job& J, const PolarTables& T, Pix px[kPX]) {
    const int tid = threadIdx.x, cols_t = 1 << J.lc;
#pragma unroll
    for (int k = 0; k < kPX; ++k) {
        const int p = tid + kThreads * k;
        const int row = p >> J.lc, col = p & (cols_t - 1);
        Pix& q = px[k];
        q.dxh = T.rxh[row] + T.cxh[col];  // exact: both multiples of the quantum
        q.dyh = T.ryh[row] + T.cyh[col];
        q.dxl = fmaf(T.dg[row], T.dcs[col], T.rxl[row] + T.cxl[col]);
        q.dyl = fmaf(T.dg[row], T.duu[col], T.ryl[row] + T.cyl[col]);
        q.dzh = q.dzl = q.dz = 0.0f;
        q.dx = q.dxh + q.dxl;
        q.dy = q.dyh + q.dyl;
        q.d2 = q.dx * q.dx + q.dy * q.dy;
        q.psi = T.psi[row];
        q.ar = q.ai = 0.0f;
    }
    __syncthreads();  // the tables alias the window region
}

__device__ void setup_polar(const SplitParams& P, const Job& J, TileShared& S, PolarTables& T, Pix px[kPX],
                            bool demodulate) {
    polar_tables<false>(P, J, S, T, demodulate);
    polar_pixels(J, T, px);
}

// Polar tile set-up from per-node tables of float pairs (FFBP):
// FP32 two-float arithmetic only, no block reductions.  Row i holds three
// float4: (g hi, g lo, psi, 0), (g/r hi, g/r lo, -oz/r hi, -oz/r lo) and
// (2r, frac(Q) - 1/2, floor(Q) bits, 0) with g = sqrt(r^2 - oz^2),
// psi = frac(-K r) and Q = (r - range_start) / data_dr; column j holds
// (c hi, c lo, u hi, u lo) with c = sqrt(1 - u^2).
struct TabF {
    float rxh[kMaxRows], rxl[kMaxRows], ryh[kMaxRows], ryl[kMaxRows], dg[kMaxRows], psi[kMaxRows];
    float cxh[kMaxCols], cxl[kMaxCols], cyh[kMaxCols], cyl[kMaxCols], dcs[kMaxCols], duu[kMaxCols];
};

// (ah + al) * (bh + bl) as an unevaluated pair p + e.
__device__ __forceinline__ void two_prod(float ah, float al, float bh, float bl, float& p, float& e) {
    p = ah * bh;
    e = fmaf(ah, bh, -p);
    e = fmaf(ah, bl, e);
    e = fmaf(al, bh, e);
}

__device__ __forceinline__ void quantize_pair(float& p, float& e, float q, float iq) {
    const float h = rintf(p * iq) * q;  // exact: q is a power of two and |p / q| < 2^14
    e = (p - h) + e;                    // p - h is exact
    p = h;
}

// One row (i) and one column (j) of a merge tile's tables, before quantization; r0v and c0v are
// the tile centre's row and column (i0, j0).
struct TabRow {
    float rxh, rxl, ryh, ryl, dg, psi;
};
struct TabCol {
    float cxh, cxl, cyh, cyl, dcs, duu;
};

__device__ __forceinline__ TabRow tab_row(const PolarDesc& g, const float4* __restrict__ tables, float4 r0v,
                                          float4 c0v, int i) {
    const float4 rv = __ldg(tables + g.rows_off + 3 * (long long)i);
    const float side = (float)g.side;
    const float dh = rv.x - r0v.x, dl = rv.y - r0v.y;  // g values of one node: dh is exact
    TabRow R;
    float p, e;
    two_prod(dh, dl, c0v.x, c0v.y, p, e);
    R.rxh = side * p;
    R.rxl = side * e;
    two_prod(dh, dl, c0v.z, c0v.w, p, e);
    R.ryh = p;
    R.ryl = e;
    R.dg = dh + dl;
    R.psi = rv.z;
    return R;
}

__device__ __forceinline__ TabCol tab_col(const PolarDesc& g, const float4* __restrict__ tables, float4 r0v,
                                          float4 c0v, int j, int j0) {
    const float4 cv = __ldg(tables + g.cols_off + j);
    const float side = (float)g.side;
    const float ch = cv.x - c0v.x, cl = cv.y - c0v.y;  // c in (0, 1] within a factor 2: exact
    // u_j - u_0 = (j - j0) du, formed from the integer offset (no cancellation).
    const float kj = (float)(j - j0);
    const float duh = g.tf[6].x, dul = g.tf[6].y;
    const float uh = kj * duh;
    const float ul = fmaf(kj, duh, -uh) + kj * dul;
    TabCol C;
    float p, e;
    two_prod(r0v.x, r0v.y, ch, cl, p, e);
    C.cxh = side * p;
    C.cxl = side * e;
    two_prod(r0v.x, r0v.y, uh, ul, p, e);
    C.cyh = p;
    C.cyl = e;
    C.dcs = side * (ch + cl);
    C.duu = uh + ul;
    return C;
}

// Tile centre row and column of a merge tile (rows_t x cols_t pixels at (tile_r, tile_u)).
__device__ __forceinline__ void tab_centre(const PolarDesc& g, int lc, int tile_r, int tile_u,
                                           const float4* __restrict__ tables, float4& r0v, float4& c0v, int& j0) {
    const int cols_t = 1 << lc, rows_t = kSplitTilePixels >> lc;
    const int i0 = min(g.win_r0 + tile_r + (rows_t >> 1), g.nr - 1);
    j0 = min(g.win_u0 + tile_u + (cols_t >> 1), g.nu - 1);
    r0v = __ldg(tables + g.rows_off + 3 * (long long)i0);
    c0v = __ldg(tables + g.cols_off + j0);
}

// Power-of-two quantum of a merge tile's pixel offsets, 2^(e - 12) with the bound on |delta_x|,
// |delta_y| = m 2^e, m in [0.5, 1): row terms are monotone in i and column terms extreme at the
// tile edges, so the bound comes from the first and last row and column.  FP32 bit arithmetic;
// computed once per tile in the child-record prologue.
__device__ __forceinline__ void tab_quantum(const PolarDesc& g, int lc, int tile_r, int tile_u,
                                            const float4* __restrict__ tables, float& q, float& iq) {
    const int cols_t = 1 << lc, rows_t = kSplitTilePixels >> lc;
    float4 r0v, c0v;
    int j0;
    tab_centre(g, lc, tile_r, tile_u, tables, r0v, c0v, j0);
    const TabRow ra = tab_row(g, tables, r0v, c0v, min(g.win_r0 + tile_r, g.nr - 1));
    const TabRow rb = tab_row(g, tables, r0v, c0v, min(g.win_r0 + tile_r + rows_t - 1, g.nr - 1));
    const TabCol ca = tab_col(g, tables, r0v, c0v, min(g.win_u0 + tile_u, g.nu - 1), j0);
    const TabCol cb = tab_col(g, tables, r0v, c0v, min(g.win_u0 + tile_u + cols_t - 1, g.nu - 1), j0);
    const float mrx = fmaxf(fabsf(ra.rxh), fabsf(rb.rxh)), mry = fmaxf(fabsf(ra.ryh), fabsf(rb.ryh));
    const float mdg = fmaxf(fabsf(ra.dg), fabsf(rb.dg));
    const float mcx = fmaxf(fabsf(ca.cxh), fabsf(cb.cxh)), mcy = fmaxf(fabsf(ca.cyh), fabsf(cb.cyh));
    const float mdc = fmaxf(fabsf(ca.dcs), fabsf(cb.dcs)), mdu = fmaxf(fabsf(ca.duu), fabsf(cb.duu));
    // The last run of rows may reach past the grid: its middle lies less than half a run beyond the last row.
    const float over = g.run_k > 0.0f && g.win_r0 + tile_r + rows_t > g.nr
                           ? 0.5f * kMergeRun * fabsf(g.tf[4].x) / __ldg(tables + g.rows_off + 3 * (long long)min(g.win_r0 + tile_r, g.nr - 1) + 1).x
                           : 0.0f;
    const float bx = fmaf(fmaf(mdg, mdc, mrx + mcx) + over, 1.0001f, 1e-6f);
    const float by = fmaf(fmaf(mdg, mdu, mry + mcy) + over, 1.0001f, 1e-6f);
    const int e = ((__float_as_int(fmaxf(bx, by)) >> 23) & 0xff) - 126;
    q = __int_as_float((e - 12 + 127) << 23);
    iq = __int_as_float((12 - e + 127) << 23);
}

// Polar merge-tile set-up from per-node tables of float pairs (FFBP): FP32 two-float arithmetic
// only, one barrier.  The offsets are quantized on the tile's quantum (q, iq) from its child
// record, so each table entry is final when it is written.
template <int THREADS>
__device__ void setup_polar_tab(const Job& J, TabF& T, const float4* __restrict__ tables, float q, float iq) {
    const PolarDesc& g = J.g;
    const int tid = threadIdx.x;
    const int cols_t = 1 << J.lc, rows_t = kSplitTilePixels >> J.lc;
    float4 r0v, c0v;
    int j0;
    tab_centre(g, J.lc, J.tile_r, J.tile_u, tables, r0v, c0v, j0);
    // rows_t <= 256: one row per thread, or a loop when the block is narrower.
    const auto row = [&](int t) {
        TabRow R = tab_row(g, tables, r0v, c0v, min(g.win_r0 + J.tile_r + t, g.nr - 1));
        quantize_pair(R.rxh, R.rxl, q, iq);
        quantize_pair(R.ryh, R.ryl, q, iq);
        T.rxh[t] = R.rxh;
        T.rxl[t] = R.rxl;
        T.ryh[t] = R.ryh;
        T.ryl[t] = R.ryl;
        T.dg[t] = R.dg;
        T.psi[t] = R.psi;
    };
    if (THREADS >= kMaxRows) {
        if (tid < rows_t) row(tid);
    } else {
        for (int t = tid; t < rows_t; t += THREADS) row(t);
    }
    if (tid < cols_t) {  // cols_t <= 32
        TabCol C = tab_col(g, tables, r0v, c0v, min(g.win_u0 + J.tile_u + tid, g.nu - 1), j0);
        quantize_pair(C.cxh, C.cxl, q, iq);
        quantize_pair(C.cyh, C.cyl, q, iq);
        T.cxh[tid] = C.cxh;
        T.cxl[tid] = C.cxl;
        T.cyh[tid] = C.cyh;
        T.cyl[tid] = C.cyl;
        T.dcs[tid] = C.dcs;
        T.duu[tid] = C.duu;
    }
    __syncthreads();
}

// Lattice tile set-up for the separable pulse loops: the tile centre, bounds and quantum in FP64, and
// the steps as two-float.
__device__ void setup_lattice_tile(const Job& J, TileShared& S) {
    const sarbp_lattice& L = J.lat;
    const int cols_t = 1 << J.lc, rows_t = kSplitTilePixels >> J.lc;
    const int hr = rows_t >> 1, hc = cols_t >> 1;
    if (threadIdx.x < 32) {
        // Lanes 0 to 2 form a component each: an FP64 instruction takes 64 cycles for one lane or for 32, and on few
        // tiles this chain is a tenth of the call (96 x 128 pixels, 192 pulses: 15.1 us; by components 14.1).
        const int c = threadIdx.x;
        const double i0 = (double)(J.tile_r + hr), j0 = (double)(J.tile_u + hc);
        const double o = c == 0 ? L.origin[0] : c == 1 ? L.origin[1] : L.origin[2];
        const double r = c == 0 ? L.step_row[0] : c == 1 ? L.step_row[1] : L.step_row[2];
        const double q = c == 0 ? L.step_col[0] : c == 1 ? L.step_col[1] : L.step_col[2];
        const double centre = o + i0 * r + j0 * q, bound = hr * fabs(r) + hc * fabs(q);
        float rh, rl, qh, ql;
        split2(r, rh, rl);
        split2(q, qh, ql);
        if (c < 3) {
            (c == 0 ? S.cx : c == 1 ? S.cy : S.cz) = centre;
            S.sth[c] = rh;
            S.stl[c] = rl;
            S.sth[3 + c] = qh;
            S.stl[3 + c] = ql;
            S.bnd[c] = (float)(bound * 1.0001 + 1e-6);
        }
        double b[3];
        for (int k = 0; k < 3; ++k) b[k] = __shfl_sync(0xffffffffu, bound, k);
        if (c == 0) {
            S.rho = sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]) * 1.0001 + 1e-6;
            const bool has_z = L.step_row[2] != 0.0 || L.step_col[2] != 0.0;
            set_quantum(S, (float)(fmax(b[0], fmax(b[1], b[2])) * 1.0001 + 1e-6), has_z ? 11 : 12);
            S.row_step = kThreads >> J.lc;
        }
    }
    __syncthreads();
}

// setup_lattice_tile plus, per pixel, |delta|^2 (FP32).  Thread t holds pixels (row (t >> lc) + k m,
// column t & (cols - 1)), k = 0..3, m = kThreads >> lc (the adjoint's assignment).
__device__ void setup_lattice_sep(const Job& J, TileShared& S, float d2[kPX]) {
    setup_lattice_tile(J, S);
    const int tid = threadIdx.x;
    const int cols_t = 1 << J.lc, rows_t = kSplitTilePixels >> J.lc;
    const int hr = rows_t >> 1, hc = cols_t >> 1;
    const float dj = (float)((tid & (cols_t - 1)) - hc);
#pragma unroll
    for (int k = 0; k < kPX; ++k) {
        const float di = (float)(((tid + kThreads * k) >> J.lc) - hr);
        float v = 0.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float x = fmaf(di, S.sth[c], dj * S.sth[3 + c]);
            v = fmaf(x, x, v);
        }
        d2[k] = v;
    }
}

// Points [J.p_begin, J.p_end) of the list; the tile's other places repeat the first of them.
__device__ void setup_points(const Job& J, TileShared& S, PointPix px[kPointPX]) {
    const int tid = threadIdx.x;
    double p3[kPointPX][3];
    double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < kPointPX; ++k) {
        const int idx = J.tile_r + tid + kThreads * k;
        const bool ok = idx >= J.p_begin && idx < J.p_end;
        int q = ok ? idx : J.p_begin;
        if (J.index) q = J.index[q];
        p3[k][0] = J.xyz[3LL * q];
        p3[k][1] = J.xyz[3LL * q + 1];
        p3[k][2] = J.xyz[3LL * q + 2];
        if (ok) {
            v[0] += p3[k][0];
            v[1] += p3[k][1];
            v[2] += p3[k][2];
            v[3] += 1.0;
        }
    }
    block_sum4(S, v);
    const double cx = v[0] / v[3], cy = v[1] / v[3], cz = v[2] / v[3];
    float m[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < kPointPX; ++k) {
        m[0] = fmaxf(m[0], (float)fabs(p3[k][0] - cx));
        m[1] = fmaxf(m[1], (float)fabs(p3[k][1] - cy));
        m[2] = fmaxf(m[2], (float)fabs(p3[k][2] - cz));
    }
    block_max<3>(S, m);
    if (tid == 0) {
        S.cx = cx;
        S.cy = cy;
        S.cz = cz;
        const double b0 = m[0] * 1.0001 + 1e-6, b1 = m[1] * 1.0001 + 1e-6, b2 = m[2] * 1.0001 + 1e-6;
        S.rho = sqrt(b0 * b0 + b1 * b1 + b2 * b2);
        S.bnd[0] = (float)b0;
        S.bnd[1] = (float)b1;
        S.bnd[2] = (float)b2;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPointPX; ++k) {
        PointPix& q = px[k];
        const auto part = [](double o, float& h, float& l, int& n, float& r) {
            split2(o, h, l);
            n = __float2int_rn(h * 65536.0f);
            r = (h - (float)n * (1.0f / 65536.0f)) + l;  // exact difference within 256 m
        };
        part(p3[k][0] - cx, q.dx, q.lx, q.ix, q.rx);
        part(p3[k][1] - cy, q.dy, q.ly, q.iy, q.ry);
        part(p3[k][2] - cz, q.dz, q.lz, q.iz, q.rz);
        q.d2 = q.dx * q.dx + q.dy * q.dy + q.dz * q.dz;
        q.ar = q.ai = 0.0f;
    }
}

// ---- the pulse loop ---------------------------------------------------------------
// Points: offsets in three dimensions, no demodulation.  The large linear terms of the phase and of
// the range, W . delta and u . delta / dr, are formed in 32-bit integers: with W in whole 2^-16
// turns/m, u / dr in whole 2^-12 bins/m and delta in whole 2^-16 m, the wrapping products and their sums are exact
// modulo one turn (2^-32 turns) and modulo 16 bins (2^-28 bins); taking the nearest bin off leaves
// a fraction of a bin.  What the roundings leave (rests of W, u / dr and delta, below 1e-3 turns or bins) is FP32.
// An FP32 range of ten bins alone would put 3e-7 on the fraction, and through it on the image.  Tiles hold
// 512 points (the range correction, FP32, grows with the square of the tile).  192,384 points, 1024
// pulses: 0.57 ms; with FP32 products of 10- and 11-bit parts 0.51 ms and an error of 3.6e-7 instead of 2.8e-7.
__device__ __forceinline__ void points_chunk(const SplitParams& P, const Rec* __restrict__ rec,
                                             const float4* __restrict__ win, const float* __restrict__ rest, int chn,
                                             PointPix px[kPointPX]) {
    const float inv_dr = P.inv_drf, Kf = P.Kf;
    // The chunk's sum goes to the image at the end: shorter FP32 sums.
    float ar[kPointPX], ai[kPointPX];
#pragma unroll
    for (int k = 0; k < kPointPX; ++k) ar[k] = ai[k] = 0.0f;
#pragma unroll 1
    for (int nl = 0; nl < chn; ++nl) {
        const float4 rb = rec[nl].b, rc = rec[nl].c, rd = rec[nl].d;
        const int4 ri = *reinterpret_cast<const int4*>(&rec[nl].a), re = *reinterpret_cast<const int4*>(&rec[nl].e);
        const float uly = __int_as_float(re.w), ulz = rest[nl];
        const float4* wrow = win + 2 * __float_as_int(rc.z);
#pragma unroll
        for (int k = 0; k < kPointPX; ++k) {
            const PointPix& q = px[k];
            const float L = fmaf(rb.z, q.dz, fmaf(rb.x, q.dx, rb.y * q.dy));
            const float q2 = fmaf(-L, L, q.d2);
            const float B = rcp_approx(fmaf(2.0f, L, rb.w));
            const float e0 = q2 * B;
            const float eps = fmaf(-e0 * e0, B, e0);
            // Nearest bin of the window (see lattice_runs for why it is inside).
            const float tq = fmaf(L + eps, inv_dr, rc.y) + kMagic;
            const unsigned j = (unsigned)(__float_as_int(tq) - kMagicBits);
            const float4 c01 = wrow[2 * j], c23 = wrow[2 * j + 1];
            // u . (rest of delta), in metres, with eps: small terms of the range and of the phase.
            const float er = eps + fmaf(rb.z, q.rz, fmaf(rb.x, q.rx, rb.y * q.ry));
            const int bins = (int)((unsigned)__float_as_int(rc.x) - ((unsigned)__float_as_int(tq) << 28) +
                                   (unsigned)re.x * (unsigned)q.ix + (unsigned)re.y * (unsigned)q.iy +
                                   (unsigned)re.z * (unsigned)q.iz);
            const float s = fmaf(inv_dr, er, fmaf((float)bins, 3.7252902984619141e-09f,
                                                  fmaf(ulz, q.dz, fmaf(uly, q.dy, rd.w * q.dx))));
            const float vr = fmaf(fmaf(fmaf(c23.z, s, c23.x), s, c01.z), s, c01.x);
            const float vi = fmaf(fmaf(fmaf(c23.w, s, c23.y), s, c01.w), s, c01.y);
            const int turns = (int)((unsigned)ri.w + (unsigned)ri.x * (unsigned)q.ix + (unsigned)ri.y * (unsigned)q.iy +
                                    (unsigned)ri.z * (unsigned)q.iz);
            const float tot = fmaf(Kf, er, fmaf((float)turns, 2.3283064365386963e-10f,
                                                fmaf(rd.z, q.dz, fmaf(rd.y, q.dy, rd.x * q.dx))));
            // K eps goes to a few turns, beyond which the hardware sine and cosine lose accuracy.
            const float ang = (tot - round_magic(tot)) * kTwoPiF;
            float sn, cs;
            __sincosf(ang, &sn, &cs);
            ar[k] = fmaf(vr, cs, ar[k]);
            ar[k] = fmaf(-vi, sn, ar[k]);
            ai[k] = fmaf(vr, sn, ai[k]);
            ai[k] = fmaf(vi, cs, ai[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < kPointPX; ++k) {
        px[k].ar += ar[k];
        px[k].ai += ai[k];
    }
}

// 2-D demodulated tiles (polar grids) with the thread's pixels k = 2h, 2h + 1 as packed FP32
// (f32x2) pairs through the range, fraction, window-index and phase steps; the complex cubic
// evaluates (re, im) as one pair and the accumulation stays scalar.  The chain carries -L, -q2,
// -e0 and -eps (negation is exact):
//   -L = (-u) . delta,  -q2 = (-L)^2 - d2,  2L + 2R = -2 (-L) + 2R,  -e0 = -q2 B,
//   -eps = (-e0)^2 B + (-e0),  qp = ((-L) + (-eps)) (-1/dr) + Fm,  sm = -K (-eps) + Phi + ...
__device__ __forceinline__ void polar_chunk(const SplitParams& P, const Rec* __restrict__ rec,
                                            const float4* __restrict__ win, int chn, Pix px[kPX]) {
    static_assert(kPX == 4, "two pixel pairs per thread");
    const float2 ninv = pair(-P.inv_drf), nKf = pair(-P.Kf), mone = pair(-1.0f), mtwo = pair(-2.0f);
    const float2 magic = pair(kMagic), nmagic = pair(-kMagic), twopi = pair(kTwoPiF);
#pragma unroll
    for (int k = 0; k < kPX; ++k) px[k].d2 = -px[k].d2;  // carried as -d2 through the chunk
#pragma unroll 1
    for (int nl = 0; nl < chn; ++nl) {
        const float4 ra = rec[nl].a, rb = rec[nl].b, rc = rec[nl].c;
        const int bias = __float_as_int(rc.y);
        const unsigned last = (unsigned)__float_as_int(rc.w);
        const float4* wrow = win + 2 * __float_as_int(rc.z);
        const float2 nux = pair(-rb.x), nuy = pair(-rb.y), twoR = pair(rb.z), fm = pair(rb.w);
        const float2 Wx = pair(ra.x), Wy = pair(ra.y), Wlx = pair(ra.z), Wly = pair(ra.w), phi = pair(rc.x);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const Pix &pa = px[2 * h], &pb = px[2 * h + 1];
            const float2 dx = make_float2(pa.dx, pb.dx), dy = make_float2(pa.dy, pb.dy);
            const float2 nL = __ffma2_rn(nux, dx, __fmul2_rn(nuy, dy));
            const float2 nq2 = __ffma2_rn(nL, nL, make_float2(pa.d2, pb.d2));
            const float2 den = __ffma2_rn(mtwo, nL, twoR);
            const float2 B = make_float2(rcp_approx(den.x), rcp_approx(den.y));
            const float2 ne0 = __fmul2_rn(nq2, B);
            const float2 neps = __ffma2_rn(__fmul2_rn(ne0, ne0), B, ne0);
            const float2 qp = __ffma2_rn(__fadd2_rn(nL, neps), ninv, fm);
            const float2 tq = __fadd2_rn(qp, magic);
            const float2 sv = __ffma2_rn(__fadd2_rn(tq, nmagic), mone, qp);
            const float2 tb = __ffma2_rn(Wx, make_float2(pa.dxh, pb.dxh), __fmul2_rn(Wy, make_float2(pa.dyh, pb.dyh)));
            float2 sm = __ffma2_rn(nKf, neps, phi);
            sm = __ffma2_rn(Wx, make_float2(pa.dxl, pb.dxl), sm);
            sm = __ffma2_rn(Wy, make_float2(pa.dyl, pb.dyl), sm);
            sm = __ffma2_rn(Wlx, dx, sm);
            sm = __ffma2_rn(Wly, dy, sm);
            sm = __fadd2_rn(sm, make_float2(pa.psi, pb.psi));
            // The reduced large term is in [-1/2, 1/2] turn and |sm| <= 1 + K eps <= 1 + envelope / 2
            // turns, so the angle stays within +-40 rad, which the hardware sin/cos reduce themselves.
            const float2 rtb = __fadd2_rn(__fadd2_rn(tb, magic), nmagic);
            const float2 ang = __fmul2_rn(__fadd2_rn(__ffma2_rn(rtb, mone, tb), sm), twopi);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                Pix& q = px[2 * h + c];
                const unsigned j = min((unsigned)(__float_as_int(c ? tq.y : tq.x) - bias), last);
                const float4 c01 = wrow[2 * j], c23 = wrow[2 * j + 1];
                const float2 ss = pair(c ? sv.y : sv.x);
                const float2 v = __ffma2_rn(
                    __ffma2_rn(__ffma2_rn(make_float2(c23.z, c23.w), ss, make_float2(c23.x, c23.y)), ss,
                               make_float2(c01.z, c01.w)),
                    ss, make_float2(c01.x, c01.y));
                float sn, cs;
                __sincosf(c ? ang.y : ang.x, &sn, &cs);
                q.ar = fmaf(v.x, cs, q.ar);
                q.ar = fmaf(-v.y, sn, q.ar);
                q.ai = fmaf(v.x, sn, q.ai);
                q.ai = fmaf(v.y, cs, q.ai);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kPX; ++k) px[k].d2 = -px[k].d2;
}

// ---- two-float arithmetic (unevaluated sums hi + lo of two FP32 numbers) ----------------
//
// Error-free transformations (Knuth's two-sum, the FMA form of Dekker's product) give about
// 44 significant bits in FP32 arithmetic, which runs at full rate where GB300's FP64 does not.
// They carry pulses that fall outside the split path's precision envelope.
struct FF {
    float h, l;
};

__device__ __forceinline__ FF ff_norm(float s, float e) {  // |s| >= |e|
    const float h = s + e;
    return FF{h, e - (h - s)};
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
    const float s = a.h + b.h;
    const float bb = s - a.h;
    const float e = (a.h - (s - bb)) + (b.h - bb);
    return ff_norm(s, e + (a.l + b.l));
}
__device__ __forceinline__ FF ff_mul(FF a, FF b) {
    const float p = a.h * b.h;
    const float e = fmaf(a.h, b.h, -p);
    return ff_norm(p, fmaf(a.h, b.l, fmaf(a.l, b.h, e)));
}
__device__ __forceinline__ FF ff_sqr(FF a) {
    const float p = a.h * a.h;
    const float e = fmaf(a.h, a.h, -p);
    return ff_norm(p, fmaf(2.0f * a.h, a.l, e));
}
// sqrt by one Newton step on the FP32 root: s + (a - s^2) / (2 s).
__device__ __forceinline__ FF ff_sqrt(FF a) {
    const float s = __fsqrt_rn(a.h);
    const float p = s * s;
    const float e = fmaf(s, s, -p);
    const float r = ((a.h - p) - e) + a.l;
    return ff_norm(s, r * (0.5f / s));
}
__device__ __forceinline__ FF ff_of(float2 v) { return FF{v.x, v.y}; }
__device__ __forceinline__ FF ff_neg(FF a) { return FF{-a.h, -a.l}; }
// 1/a: the FP32 reciprocal refined by one Newton step in two-float.
__device__ __forceinline__ FF ff_rcp(FF a) {
    const float i0 = __frcp_rn(a.h);
    const FF e = ff_mul(a, FF{i0, 0.0f});
    return ff_norm(i0, i0 * ((1.0f - e.h) - e.l));
}
// Splits a two-float value q into floor and centred fraction: q = I + F + 1/2, F in [-1/2, 1/2).
__device__ __forceinline__ float ff_floor_frac(FF q, float& F) {
    float I = floorf(q.h);
    float f = (q.h - I) + q.l;  // q.h - I is exact
    if (f < 0.0f) {
        f += 1.0f;
        I -= 1.0f;
    } else if (f >= 1.0f) {
        f -= 1.0f;
        I += 1.0f;
    }
    F = f - 0.5f;
    return I;
}


// Per (tile, pulse) data of a pulse the fast path cannot stage: the FP64 vector from the
// antenna to the tile centre as two-float components, the pulse phase in turns, the weight.
struct SlowRec {
    float4 a;  // w.x hi, w.x lo, w.y hi, w.y lo
    float4 b;  // w.z hi, w.z lo, phase / 2pi reduced to [-1/2, 1/2], weight
};

// (ar, ai) plus the contributions of pulses c0 + first, c0 + first + step, ... below c0 + n to one pixel, in two-float
// geometry.  Out of line (and the pixel by value) so that the rarely taken fallback does not add registers
// to the kernels' fast path.
__device__ __noinline__ float2 slow_pixel(const SplitParams& P, const SlowRec* srec, int first, int n, int step,
                                          int c0, float dxh, float dxl, float dyh, float dyl, float dzh, float dzl,
                                          float psi, float ar, float ai);

// Dynamic shared memory of the chunk kernels: [records | windows]; the two-float records of
// a chunk that stages no window live at the start of the window space.
__host__ __device__ constexpr size_t window_offset() { return (size_t)kMaxChunk * sizeof(Rec); }

// Range-sample value and its derivative for a pixel at offset delta from the tile centre,
// pulse record sr, in two-float geometry: returns false when the taps leave the row.
struct SlowSample {
    float vr, vi, dvr, dvi;  // sample1 value and d/dq
    float ang;               // phase (radians, reduced)
    float ex, ey, ez;        // unit vector pulse -> pixel
    float d;                 // range (m, FP32)
};

template <bool DERIV>
__device__ __forceinline__ bool slow_sample(const SplitParams& P, const SlowRec& sr, const float2* __restrict__ row,
                                            const Pix& q, float psi, SlowSample& o) {
    const FF vx = ff_add(FF{sr.a.x, sr.a.y}, FF{q.dxh, q.dxl});
    const FF vy = ff_add(FF{sr.a.z, sr.a.w}, FF{q.dyh, q.dyl});
    const FF vz = ff_add(FF{sr.b.x, sr.b.y}, FF{q.dzh, q.dzl});
    const FF d = ff_sqrt(ff_add(ff_add(ff_sqr(vx), ff_sqr(vy)), ff_sqr(vz)));
    const FF t = ff_mul(FF{P.Kh, P.Kl}, d);
    float tot = ((t.h - rintf(t.h)) + t.l) + (sr.b.z + psi);
    tot -= rintf(tot);
    o.ang = tot * kTwoPiF;
    const FF qq = ff_mul(ff_add(d, FF{-P.rsh, -P.rsl}), FF{P.idrh, P.idrl});
    float fl = floorf(qq.h);
    float f = (qq.h - fl) + qq.l;
    if (f < 0.0f) {
        f += 1.0f;
        fl -= 1.0f;
    } else if (f >= 1.0f) {
        f -= 1.0f;
        fl += 1.0f;
    }
    if (!(fl >= 1.0f && fl <= (float)(P.in.samples - 3))) return false;
    const int i = (int)fl;
    const float2 x0 = __ldg(row + i - 1), x1 = __ldg(row + i), x2 = __ldg(row + i + 1), x3 = __ldg(row + i + 2);
    float4 c01, c23;
    cubic_coefficients(x0, x1, x2, x3, 1.0f, c01, c23);
    const float s = f - 0.5f;
    o.vr = fmaf(fmaf(fmaf(c23.z, s, c23.x), s, c01.z), s, c01.x);
    o.vi = fmaf(fmaf(fmaf(c23.w, s, c23.y), s, c01.w), s, c01.y);
    if (DERIV) {
        o.dvr = fmaf(fmaf(3.0f * c23.z, s, 2.0f * c23.x), s, c01.z);
        o.dvi = fmaf(fmaf(3.0f * c23.w, s, 2.0f * c23.y), s, c01.w);
        const float inv = 1.0f / d.h;
        o.ex = (vx.h + vx.l) * inv;
        o.ey = (vy.h + vy.l) * inv;
        o.ez = (vz.h + vz.l) * inv;
        o.d = d.h;
    }
    return true;
}


// Two-float record of a pulse the fast path cannot stage (out of line: it is rare, and its
// FP64 temporaries would otherwise add to the registers of every chunk kernel).
__device__ __noinline__ void slow_record(const SplitParams& P, const TileShared& S, int n, SlowRec* out) {
    const PulseInputs& in = P.in;
    SlowRec sr;
    split2(S.cx - in.pos[3 * n], sr.a.x, sr.a.y);
    split2(S.cy - in.pos[3 * n + 1], sr.a.z, sr.a.w);
    split2(S.cz - in.pos[3 * n + 2], sr.b.x, sr.b.y);
    const double ph = in.phase[n] * kInvTwoPi;
    sr.b.z = (float)(ph - rint(ph));
    sr.b.w = (float)in.weight[n];
    *out = sr;
}

// Per (tile, pulse) record, computed by lane `lane` of the record warps in two-float FP32
// arithmetic (about 44 bits; GB300's FP64 rate would make these records the barrier-bound
// part of every chunk).  Returns the number of window entries the pulse needs (cap + 1 if
// it cannot be staged).
// MODE 0: per-pixel offsets (polar); 1: lattice tiles; 2: lattice tiles, adjoint; 3: points; 4: polar tiles in runs.
template <int MODE>
__device__ __forceinline__ int make_record(const SplitParams& P, TileShared& S, Rec* rec, int lane, int n) {
    const PulseInputs& in = P.in;
    float ph_, pl_;
    split2(in.pos[3 * n], ph_, pl_);
    const FF vx = ff_add(FF{S.ch[0], S.cl[0]}, FF{-ph_, -pl_});
    split2(in.pos[3 * n + 1], ph_, pl_);
    const FF vy = ff_add(FF{S.ch[1], S.cl[1]}, FF{-ph_, -pl_});
    split2(in.pos[3 * n + 2], ph_, pl_);
    const FF vz = ff_add(FF{S.ch[2], S.cl[2]}, FF{-ph_, -pl_});
    const FF R = ff_sqrt(ff_add(ff_add(ff_sqr(vx), ff_sqr(vy)), ff_sqr(vz)));
    // 1/R: the FP32 reciprocal refined by one Newton step in two-float.
    const float i0 = __frcp_rn(R.h);
    const FF e = ff_mul(R, FF{i0, 0.0f});
    const FF iR = ff_norm(i0, i0 * ((1.0f - e.h) - e.l));
    const FF ux = ff_mul(vx, iR), uy = ff_mul(vy, iR), uz = ff_mul(vz, iR);
    const FF Kk{P.Kh, P.Kl};
    const FF t = ff_mul(Kk, R);
    const double ph = in.phase[n] * kInvTwoPi;
    float t1 = ((t.h - rintf(t.h)) + t.l) + (float)(ph - rint(ph));
    t1 -= rintf(t1);
    const FF Q = ff_mul(ff_add(R, FF{-P.rsh, -P.rsl}), FF{P.idrh, P.idrl});
    float I = floorf(Q.h);
    float fq = (Q.h - I) + Q.l;
    if (fq < 0.0f) {
        fq += 1.0f;
        I -= 1.0f;
    } else if (fq >= 1.0f) {
        fq -= 1.0f;
        I += 1.0f;
    }
    const float Fm = fq - 0.5f;
    const float Rf = R.h, uxf = ux.h + ux.l, uyf = uy.h + uy.l, uzf = uz.h + uz.l;
    // |L| <= sum_c |u_c| bound_c and 0 <= eps <= rho^2 / (2 (R - rho)), in bins.
    const float lin = fabsf(uxf) * S.bnd[0] + fabsf(uyf) * S.bnd[1] + fabsf(uzf) * S.bnd[2];
    const float eps = S.rhof * S.rhof / (2.0f * fmaxf(Rf - S.rhof, 1.0f));
    const float hw = (lin + eps) * fabsf(P.inv_drf) + 1e-3f;
    const float lo = floorf(Fm - hw), hi = ceilf(Fm + hw);
    // Runs of columns of a polar grid: the pulse's offset a from the grid's origin, and what the expansion in
    // the column leaves out at the run's ends, in turns (fifth and sixth order of a.x cos, fifth of the root).
    float ax = 0.0f, ay = 0.0f, lim = 0.5f;
    bool runs_ok = true;
    if (MODE == 4) {
        const FF fx = ff_add(FF{S.sth[0], S.stl[0]}, ff_neg(vx)), fy = ff_add(FF{S.sth[1], S.stl[1]}, ff_neg(vy));
        ax = fx.h + fx.l;
        ay = fy.h + fy.l;
        const float turn = S.sth[3] * (fabsf(ax) + fabsf(ay)), y = turn / Rf;
        runs_ok = fabsf(P.Kf) * (fabsf(ax) * S.sth[2] + turn * (y * y) * (y * y)) <= 1e-7f;
        // The sample's cubic leaves out the square of the quadratic term.
        const float x1 = turn * fabsf(P.inv_drf), x2 = fmaf(S.sth[4], fabsf(ax), 0.5f * turn * y) * fabsf(P.inv_drf);
        lim = (3.0f * x1 * x1 + x2) * x2 <= 1e-7f ? 0.5f : -1.0f;
    }
    // Points: the whole numbers of the linear terms stay within 32 bits (offsets in 2^-16 m, W in 2^-16 turns/m,
    // u / dr in 2^-12 bins/m).
    const bool whole_ok = MODE != 3 || (S.rhof < 32000.0f && fabsf(P.Kf) < 32000.0f && fabsf(P.inv_drf) < 5.0e5f);
    // Points: the range series e0 - e0^2 B leaves out up to rho^6 / 16 R^5, which may cost 1e-6 turns and 1e-6 bins (at
    // a tile's corner; the image's error is a few times less).  Near ranges and wide tiles go over that.
    bool third_ok = true;
    if (MODE == 3) {
        const float x = S.rhof / Rf, x2 = x * x;
        third_ok = fmaxf(fabsf(P.Kf), fabsf(P.inv_drf)) * (x2 * x2 * x) * S.rhof <= 1.6e-5f;
    }
    const bool ok = Rf > 0.0f && fabsf(Q.h) < 1.0e7f && hi - lo + 1.0f <= (float)P.cap &&
                    fabsf(P.Kf) * S.rhof * S.rhof <= (float)P.envelope * Rf && S.rhof < 0.25f * Rf && runs_ok && whole_ok &&
                    third_ok;
    const int bo = ok ? (int)lo : 0;
    S.base[lane] = ok ? (int)I + bo : 0;
    S.wt[lane] = (float)in.weight[n];
    Rec r;
    const FF Wx = ff_mul(Kk, ux), Wy = ff_mul(Kk, uy), Wz = ff_mul(Kk, uz);
    if (MODE == 3) {
        const auto whole = [](FF w, float scale, float inv, float& rest) {
            const int n = __float2int_rn(w.h * scale);
            rest = (w.h - (float)n * inv) + w.l;  // exact difference (n has 24 bits or fewer)
            return __int_as_float(n);
        };
        const FF idr{P.idrh, P.idrl};
        r.a.x = whole(Wx, 65536.0f, 1.0f / 65536.0f, r.d.x);
        r.a.y = whole(Wy, 65536.0f, 1.0f / 65536.0f, r.d.y);
        r.a.z = whole(Wz, 65536.0f, 1.0f / 65536.0f, r.d.z);
        r.a.w = __int_as_float(__float2int_rn(t1 * 4294967296.0f));  // |t1| <= 1/2 (saturates at 1/2)
        r.b = make_float4(uxf, uyf, uzf, 2.0f * Rf);
        r.e.x = whole(ff_mul(ux, idr), 4096.0f, 1.0f / 4096.0f, r.d.w);
        r.e.y = whole(ff_mul(uy, idr), 4096.0f, 1.0f / 4096.0f, r.e.w);
        r.e.z = whole(ff_mul(uz, idr), 4096.0f, 1.0f / 4096.0f, S.rest[lane]);
        const int mid = __float2int_rn(Fm * 268435456.0f);  // |Fm| <= 1/2
        r.c.x = __int_as_float((int)((unsigned)mid - ((unsigned)bo << 28)));
        r.c.y = Fm - (float)bo;
    } else if (MODE == 1 || MODE == 2) {
        // Lattice tile: the linear phase W . delta of pixel (i, j) is i B_row + j B_col with
        // B = W . step.  Both are split on one power-of-two quantum with <= 10 significant
        // bits, so i B_row_hi + j B_col_hi is exact in FP32 for |i|, |j| < 2^12.
        const FF Br = ff_add(ff_add(ff_mul(Wx, FF{S.sth[0], S.stl[0]}), ff_mul(Wy, FF{S.sth[1], S.stl[1]})),
                             ff_mul(Wz, FF{S.sth[2], S.stl[2]}));
        const FF Bc = ff_add(ff_add(ff_mul(Wx, FF{S.sth[3], S.stl[3]}), ff_mul(Wy, FF{S.sth[4], S.stl[4]})),
                             ff_mul(Wz, FF{S.sth[5], S.stl[5]}));
        const int e = ((__float_as_int(fmaxf(fmaxf(fabsf(Br.h), fabsf(Bc.h)), 1e-30f)) >> 23) & 0xff) - 126;
        const float q = __int_as_float((e - 10 + 127) << 23), iq = __int_as_float((10 - e + 127) << 23);
        r.a.x = rintf(Br.h * iq) * q;
        r.a.y = (Br.h - r.a.x) + Br.l;
        r.a.z = rintf(Bc.h * iq) * q;
        r.a.w = (Bc.h - r.a.z) + Bc.l;
        // Phase and range steps between a thread's successive pixels: one row (forward), or
        // m = kThreads >> lc rows (adjoint).
        const float m = MODE == 1 ? 1.0f : (float)S.row_step;
        const float mh = m * Br.h;  // exact: m is a power of two
        float turns = rintf(mh), sp = (mh - turns) + m * Br.l;
        const float more = rintf(sp);
        sp -= more;
        turns += more;
        const float Ar = fmaf(uxf, S.sth[0], fmaf(uyf, S.sth[1], uzf * S.sth[2]));
        const float Ac = fmaf(uxf, S.sth[3], fmaf(uyf, S.sth[4], uzf * S.sth[5]));
        const float spr = sp * kTwoPiF;  // the phase step in radians
        if (MODE == 1) {
            // The linear phase per half row and per column, modulo one turn, in 2^-32 turns: the middle of a
            // run is a whole number of half rows and of columns away, so wrapping products are exact.
            const auto wrap = [](FF v) {
                const float n = rintf(v.h);
                return (int)((unsigned)__float2int_rn((v.h - n) * 4294967296.0f) +
                             (unsigned)__float2int_rn(v.l * 4294967296.0f));
            };
            r.a.x = __int_as_float(wrap(FF{0.5f * Br.h, 0.5f * Br.l}));
            r.a.y = __int_as_float(wrap(Bc));
            r.b = make_float4(Ar, Ac, Rf, Fm);
            // Fourth-order range term of a run of rows, e4 k^4 with k^4 ~ 12.5 k^2 - 21.0625 (lattice_runs).
            const float s2 = S.sth[0] * S.sth[0] + S.sth[1] * S.sth[1] + S.sth[2] * S.sth[2];
            const float iRf = 1.0f / Rf;
            const float e4 = 0.125f * (s2 - Ar * Ar) * (5.0f * Ar * Ar - s2) * iRf * iRf * iRf;
            r.c = make_float4(fmaf(-21.0625f * P.Kf, e4, t1), 0.0f, 0.0f, 12.5f * e4);
            // The phase step reduced modulo half a turn, which keeps the angles along a run small: the step is
            // spT + N / 2 with |spT| <= 1/4, and pixel k = 2 g - 3.5 + c adds k N / 2 = (g - 2) N + (2 c + 1) N / 4
            // turns: N / 4 for the even pixels of the run (c = 0) and half of N more for the odd ones.  Half a turn more
            // is a quarter before and a quarter after a middle phase: the angles stay within 10 rad instead of 12, and the
            // two starts are one packed operation (192 pulses onto 96 x 128: error 3.01e-7 -> 2.89e-7 on average over 12
            // scenes, one pixel at a time 2.91e-7; 4096 onto 2048 x 2048: 17.10 -> 16.94 ms).
            const float n2 = rintf(2.0f * sp);
            const float even = 0.25f * (n2 + 2.0f * turns);
            r.c.z = (sp - 0.5f * n2) * kTwoPiF;
            r.c.x += even - rintf(even);
            const float odd = 0.5f * n2, q = 0.5f * fabsf(odd - rintf(odd));
            r.c.x += q;
            r.d.x = -q * kTwoPiF;
            r.d.y = q * kTwoPiF;
            r.d.z = r.d.w = 0.0f;
            r.c.x = __int_as_float(wrap(FF{r.c.x, 0.0f}));
        } else {
            r.b = make_float4(Ar, Ac, 2.0f * Rf, Fm);
            r.d = make_float4(spr, uxf, uyf, uzf);
            r.e = make_float4(2.0f * Rf, 2.0f * Rf, Fm, Fm);
        }
    } else {
        const float sw = (float)P.scale_w, isw = (float)P.inv_scale_w;  // powers of two: exact
        r.a.x = rintf(Wx.h * isw) * sw;
        r.a.z = (Wx.h - r.a.x) + Wx.l;
        r.a.y = rintf(Wy.h * isw) * sw;
        r.a.w = (Wy.h - r.a.y) + Wy.l;
        r.d.y = rintf(Wz.h * isw) * sw;
        r.d.z = (Wz.h - r.d.y) + Wz.l;
        r.b = make_float4(uxf, uyf, 2.0f * Rf, Fm);
        r.d.x = uzf;
        r.d.w = 0.0f;
        r.e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (MODE == 4) r.d = make_float4(-kTwoPiF * P.Kf * ax, -kTwoPiF * P.Kf * ay, lim, 0.0f);
    }
    if (MODE == 0 || MODE == 2 || MODE == 4) r.c.x = t1;
    float4& rw = rec_window<MODE>(r);
    if (MODE != 3) rw.y = __int_as_float(kMagicBits + bo);
    const int count = ok ? (int)(hi - lo) + 1 : P.cap + 1;
    rw.z = 0.0f;
    rw.w = __int_as_float(count - 1);
    if (MODE == 1) rw.x = 0.0f;
    rec[lane] = r;
    return count;
}

__device__ __noinline__ float2 slow_pixel(const SplitParams& P, const SlowRec* srec, int first, int n, int step,
                                          int c0, float dxh, float dxl, float dyh, float dyl, float dzh, float dzl,
                                          float psi, float ar, float ai) {
    Pix q;
    q.dxh = dxh;
    q.dxl = dxl;
    q.dyh = dyh;
    q.dyl = dyl;
    q.dzh = dzh;
    q.dzl = dzl;
    for (int j = first; j < n; j += step) {
        const SlowRec sr = srec[j];
        SlowSample o;
        if (!slow_sample<false>(P, sr, P.in.data + (size_t)(c0 + j) * P.in.samples, q, psi, o)) continue;
        float sn, cs;
        __sincosf(o.ang, &sn, &cs);
        const float a = sr.b.w;
        ar = fmaf(a * o.vr, cs, fmaf(-a * o.vi, sn, ar));
        ai = fmaf(a * o.vr, sn, fmaf(a * o.vi, cs, ai));
    }
    return make_float2(ar, ai);
}

__device__ int g_wait_timeouts;  // bounded waits on asynchronous copies that ran out

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for phase `phase` of the mbarrier at shared address bar, for at most limit_ns of the GPU's
// timer (and at most 2^24 polls); true once the phase completed.
__device__ __forceinline__ bool timed_wait(unsigned bar, unsigned phase, unsigned long long limit_ns) {
    const unsigned long long t0 = global_ns();
    for (int it = 0; it < (1 << 24); ++it) {
        unsigned done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
    return false;
}

// Bounded wait for the phase `phase` of the mbarrier at shared address bar; true once it completed.
__device__ __forceinline__ bool bulk_wait(unsigned bar, unsigned phase) {
    unsigned done = 0;
    for (int it = 0; it < (1 << 22) && !done; ++it)
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
    return done != 0;
}

#if SARBP_BULK_WINDOWS
// Raw samples [b - 1, b + cnt + 2) of each fitting pulse's row (clipped to the row) arrive in
// shared memory by one 1-D cp.async.bulk copy per pulse, issued by warp 0 after lane 0 has set
// the transaction count on the mbarrier; every thread waits for the phase (a bounded wait that
// records a timeout), then the Horner transform reads shared memory.  A copy must start and end
// on 16-byte boundaries of the data array, so the copied range is widened to even elements.
// Returns false (the same in every thread) if the copies did not arrive within the bounded wait;
// the caller then stops staging and waits once more before leaving.
template <int MODE>
__device__ __forceinline__ bool bulk_stage_windows(const SplitParams& P, TileShared& S, const Rec* rec, float4* win,
                                                   float2* raw, unsigned long long& mbar, unsigned phase, int c0,
                                                   int nfit, bool weighted) {
    const PulseInputs& in = P.in;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&mbar);
    if (warp == 0) {
        long long a0[2];
        int len[2];
        int mine = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int nl = lane + 32 * h;
            a0[h] = 0;
            len[h] = 0;
            if (nl < nfit) {
                const long long row0 = (long long)(c0 + nl) * in.samples;
                const long long b0 = S.base[nl];
                const int cnt = __float_as_int(rec_window<MODE>(rec[nl]).w) + 1;
                // [g0, g1) within the row; rows start on even elements (samples is even), so
                // widening to even bounds stays inside the row.
                const long long g0 = min(max(b0 - 1, 0ll), (long long)in.samples);
                const long long g1 = max(min(b0 + cnt + 2, (long long)in.samples), g0);
                const long long e0 = (row0 + g0) & ~1ll, e1 = (row0 + g1 + 1) & ~1ll;
                a0[h] = e0;
                len[h] = (int)max(e1 - e0, 0ll);
                mine += len[h];
            }
        }
        // Exclusive prefix of the raw lengths (even, so every destination stays 16-byte aligned).
        int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        const int total = __shfl_sync(0xffffffffu, inc, 31);
        int off = inc - mine;
        if (lane == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(total * 8)
                         : "memory");
        }
        __syncwarp();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the last chunk's reads precede these writes
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int nl = lane + 32 * h;
            if (nl < nfit) {
                S.roff[nl] = off;
                S.raw0[nl] = a0[h];
                if (len[h] > 0) {
                    const unsigned dst = (unsigned)__cvta_generic_to_shared(raw + off);
                    asm volatile(
                        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                            dst),
                        "l"(in.data + a0[h]), "r"(len[h] * 8), "r"(bar)
                        : "memory");
                }
                off += len[h];
            }
        }
    }
    // Bounded wait for the copies of this chunk's phase.
    const bool done = __syncthreads_and(bulk_wait(bar, phase)) != 0;  // also orders roff / raw0 of warp 0
    if (!done) {
        if (threadIdx.x == 0) atomicAdd(&g_wait_timeouts, 1);
        return false;
    }
    for (int nl = warp; nl < nfit; nl += kThreads / 32) {
        const int woff = __float_as_int(rec_window<MODE>(rec[nl]).z);
        const int cnt = __float_as_int(rec_window<MODE>(rec[nl]).w) + 1;
        const long long b0 = S.base[nl];
        const float a = weighted ? S.wt[nl] : 1.0f;
        const float2* r = raw + S.roff[nl] + ((long long)(c0 + nl) * in.samples - S.raw0[nl]);  // row-relative
        for (int j = lane; j < cnt; j += 32) {
            const long long g = b0 + j;
            float4 c01 = make_float4(0.f, 0.f, 0.f, 0.f), c23 = c01;
            if (g >= 1 && g <= (long long)in.samples - 3)
                cubic_coefficients(r[g - 1], r[g], r[g + 1], r[g + 2], a, c01, c23);
            win[2 * (woff + j)] = c01;
            win[2 * (woff + j) + 1] = c23;
        }
    }
    return true;
}
#endif

// Horner windows of one pulse (cnt entries from bin b0) staged by one warp with one global load
// per lane and step: lane l loads sample b0 + j0 + l - 1, and entry j0 + l (l < 29) takes its four
// taps from lanes l .. l + 3 by shuffles (the FFBP leaves and polar-grid direct BP).
__device__ __forceinline__ void stage_window_shfl(const float2* __restrict__ row, long long samples, long long b0,
                                                  int cnt, float a, float4* __restrict__ wentry, int lane) {
    for (int j0 = 0; j0 < cnt; j0 += 29) {
        const long long gi = b0 + j0 + lane - 1;
        float2 x = make_float2(0.0f, 0.0f);
        if (gi >= 0 && gi < samples) x = __ldg(row + gi);
        float2 x1, x2, x3;
        x1.x = __shfl_down_sync(0xffffffffu, x.x, 1);
        x1.y = __shfl_down_sync(0xffffffffu, x.y, 1);
        x2.x = __shfl_down_sync(0xffffffffu, x.x, 2);
        x2.y = __shfl_down_sync(0xffffffffu, x.y, 2);
        x3.x = __shfl_down_sync(0xffffffffu, x.x, 3);
        x3.y = __shfl_down_sync(0xffffffffu, x.y, 3);
        const int j = j0 + lane;
        if (lane < 29 && j < cnt) {
            const long long g = b0 + j;
            float4 c01 = make_float4(0.f, 0.f, 0.f, 0.f), c23 = c01;
            if (g >= 1 && g <= samples - 3) cubic_coefficients(x, x1, x2, x3, a, c01, c23);
            wentry[2 * j] = c01;
            wentry[2 * j + 1] = c23;
        }
    }
}

// Chunk driver shared by the forward and adjoint kernels: per chunk of up to 64
// pulses, warps 0 and 1 compute the (tile, pulse) records (one pulse per lane, two-float,
// on two SM sub-partitions at once) and pack the pulses' range windows, all warps
// stage the windows (Horner coefficients, times the pulse weight when `weighted`),
// then `body.fast(rec, win, nfit, c0)` consumes them; a pulse whose window cannot be
// staged goes through `body.slow(c0, n, slow)` with its two-float record.
template <class Body>
__device__ void chunk_loop(const SplitParams& P, const Job& J, TileShared& S, char* smem, bool weighted, Body& body) {
    const PulseInputs& in = P.in;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Rec* rec = reinterpret_cast<Rec*>(smem);
    float4* win = reinterpret_cast<float4*>(smem + window_offset());
    SlowRec* slow = reinterpret_cast<SlowRec*>(win);  // a chunk that stages nothing reuses the window space
#if SARBP_BULK_WINDOWS
    float2* raw = reinterpret_cast<float2*>(smem + window_offset() + (size_t)P.cap * 32);
    __shared__ __align__(8) unsigned long long mbar;
    unsigned phase = 0;
    // Bulk copies need 16-byte aligned rows: an even sample count on a 16-byte aligned array.
    const bool bulk = ((reinterpret_cast<uintptr_t>(in.data) & 15) == 0) && (in.samples % 2 == 0);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&mbar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
#endif
    if (threadIdx.x < 3) {  // the tile centre as two-float for the records (ordered by the loop's barrier)
        split2(threadIdx.x == 0 ? S.cx : threadIdx.x == 1 ? S.cy : S.cz, S.ch[threadIdx.x], S.cl[threadIdx.x]);
        if (threadIdx.x == 0) S.rhof = (float)S.rho;
    }
    for (int c0 = J.p0; c0 < J.p1;) {
        const int want = min(P.chunk, J.p1 - c0);
        __syncthreads();  // the previous chunk's records and windows are consumed
        if (warp < 2) {
            const int idx = 32 * warp + lane;
            const int count = idx < want ? make_record<Body::kRecMode>(P, S, rec, idx, c0 + idx) : 0;
            int inc = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (warp == 0 && lane == 31) S.wsum = inc;
            asm volatile("bar.sync 2, 64;" ::: "memory");  // warps 0 and 1 only
            if (warp == 1) inc += S.wsum;
            // Counts are >= 1, so the pulses that fit form a prefix of the chunk.
            const unsigned fits = __ballot_sync(0xffffffffu, idx < want && inc <= P.cap);
            if (idx < want) {
                float4& rw = rec_window<Body::kRecMode>(rec[idx]);
                rw.z = __int_as_float(inc - count);
                // Byte offset in the windows of the entry that index bits 0 would address: bits * 32 plus
                // this wraps to the entry's own offset.
                if (Body::kRecMode == 1)
                    rec[idx].c.y = __int_as_float((int)(32u * ((unsigned)(inc - count) - (unsigned)__float_as_int(rw.y))));
            }
            if (lane == 0) S.nfit_w[warp] = __popc(fits);
        }
        __syncthreads();
        const int nfit = S.nfit_w[0] + S.nfit_w[1];
        if (nfit > 0) {
#if SARBP_BULK_WINDOWS
            if (bulk) {
                if (!bulk_stage_windows<Body::kRecMode>(P, S, rec, win, raw, mbar, phase, c0, nfit, weighted)) {
                    // The copies did not arrive: the tile's image is invalid (g_wait_timeouts counts it).
                    // Wait once more, bounded, for the copies still in flight, then leave.
                    bulk_wait((unsigned)__cvta_generic_to_shared(&mbar), phase);
                    break;
                }
                phase ^= 1u;
            } else
#endif
            for (int nl = warp; nl < nfit; nl += kThreads / 32) {
                const float4& rw = rec_window<Body::kRecMode>(rec[nl]);
                const int off = __float_as_int(rw.z);
                const int cnt = __float_as_int(rw.w) + 1;
                const long long b0 = S.base[nl];
                const float a = weighted ? S.wt[nl] : 1.0f;
                const float2* row = in.data + (size_t)(c0 + nl) * in.samples;
                if (Body::kShflWindows) {
                    stage_window_shfl(row, in.samples, b0, cnt, a, win + 2 * off, lane);
                    continue;
                }
                for (int j = lane; j < cnt; j += 32) {
                    const long long g = b0 + j;
                    float4 c01 = make_float4(0.f, 0.f, 0.f, 0.f), c23 = c01;
                    if (g >= 1 && g <= (long long)in.samples - 3)
                        cubic_coefficients(__ldg(row + g - 1), __ldg(row + g), __ldg(row + g + 1), __ldg(row + g + 2),
                                           a, c01, c23);
                    win[2 * (off + j)] = c01;
                    win[2 * (off + j) + 1] = c23;
                }
            }
            __syncthreads();
            body.fast(rec, win, nfit, c0);
            c0 += nfit;
        } else {
            // The leading pulses that cannot be staged (outside the precision envelope or with
            // windows too wide): two-float geometry per pixel, [c0, c0 + nslow).
            // (the records mark them with a window count of cap + 1)
            if (warp < 2) {
                const int idx = 32 * warp + lane;
                const unsigned misses =
                    __ballot_sync(0xffffffffu,
                                  idx < want && __float_as_int(rec_window<Body::kRecMode>(rec[idx]).w) + 1 > P.cap);
                if (lane == 0) S.miss_w[warp] = misses;
            }
            __syncthreads();
            const unsigned long long m = (unsigned long long)S.miss_w[0] | ((unsigned long long)S.miss_w[1] << 32);
            const int nslow = ~m == 0ull ? kMaxChunk : __ffsll((long long)~m) - 1;
            if (threadIdx.x < nslow) slow_record(P, S, c0 + threadIdx.x, slow + threadIdx.x);
            __syncthreads();
            body.slow(c0, nslow, slow);
            c0 += nslow;
        }
    }
#if SARBP_BULK_WINDOWS
    __syncthreads();  // every wait on the barrier is over: it can be invalidated (and initialised again)
    if (threadIdx.x == 0)
        asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"((unsigned)__cvta_generic_to_shared(&mbar)) : "memory");
#endif
}

// One pulse on a run of eight angle columns whose range changes by less than a bin's width as a rule
// (polar grids): phase P0 + P1 m + ... + P4 m^4 (radians) and place in the window (bins) qp + b1 m + b2 m^2
// at the columns m = -3.5 ... 3.5.  bias, last: byte offset in the window w0 of the entry that index bits 0
// would address, and of the last entry.  The sample along the run is the window entry's cubic, a cubic in m
// as long as the whole run stays within one range bin; when that holds for all the warp's runs (lim = 1/2;
// below 0: never) the run takes one window entry (two 16-byte loads instead of sixteen), and the even and
// odd parts of both polynomials serve the columns +m and -m.  Otherwise each pixel takes its own entry.
// PARTS = 2: the thread forms half of the run's columns, the inner (part 0) or the outer four, by the same
// arithmetic; ar[2 i + c] then belongs to column run_column<2>(part, i, c).
template <int PARTS>
__device__ __forceinline__ int run_column(int part, int i, int c) {
    const int h = (PARTS == 1 ? 0 : part * (kColRun / 2 / PARTS)) + i;
    return c ? kColRun / 2 + h : kColRun / 2 - 1 - h;
}

template <int PARTS>
__device__ __forceinline__ void column_run(int part, float P0, float P1, float P2, float P3, float P4, float qp, float b1, float b2,
                                           float lim, const char* __restrict__ w0, unsigned bias, unsigned last,
                                           float ar[kColRun / PARTS],
                                           float ai[kColRun / PARTS]) {
    const float tq = qp + kMagic;
    const float s = qp - (tq - kMagic);
    const float spread = fmaf(fabsf(b2), 12.25f, fmaf(fabsf(b1), 3.5f, fabsf(s)));
    if (__all_sync(0xffffffffu, spread <= lim)) {
        const float4* w = reinterpret_cast<const float4*>(w0 + min(32u * (unsigned)__float_as_int(tq) + bias, last));
        const float4 c01 = w[0], c23 = w[1];
        float V0[2], V1[2], V2[2], V3[2];
        const float bb = b1 * b1;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float A0 = c ? c01.y : c01.x, A1 = c ? c01.w : c01.z, A2 = c ? c23.y : c23.x, A3 = c ? c23.w : c23.z;
            const float T = A3 * s;
            const float W1 = A2 + T, W2 = fmaf(3.0f, T, A2);
            const float V = fmaf(W1, s, A1);               // the sample is A0 + V s
            const float D = fmaf(A2 + W2, s, A1);         // its derivative
            V0[c] = fmaf(V, s, A0);
            V1[c] = D * b1;
            V2[c] = fmaf(W2, bb, D * b2);
            V3[c] = fmaf(A3, bb, 2.0f * W2 * b2) * b1;
        }
#pragma unroll
        for (int h = 0; h < kColRun / 2 / PARTS; ++h) {
            const float m = (PARTS == 1 ? 0.5f : 0.5f + (float)(part * (kColRun / 2 / PARTS))) + h, mm = m * m;
            const float ae = fmaf(fmaf(P4, mm, P2), mm, P0), ao = fmaf(P3, mm, P1);
            const float re = fmaf(V2[0], mm, V0[0]), ro = fmaf(V3[0], mm, V1[0]);
            const float ie = fmaf(V2[1], mm, V0[1]), io = fmaf(V3[1], mm, V1[1]);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int k = PARTS == 1 ? run_column<1>(0, h, c) : 2 * h + c;
                const float x = c ? m : -m;
                const float vr = fmaf(ro, x, re), vi = fmaf(io, x, ie);
                float sn, cs;
                __sincosf(fmaf(ao, x, ae), &sn, &cs);
                ar[k] = fmaf(vr, cs, ar[k]);
                ar[k] = fmaf(-vi, sn, ar[k]);
                ai[k] = fmaf(vr, sn, ai[k]);
                ai[k] = fmaf(vi, cs, ai[k]);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < kColRun / PARTS; ++k) {
            const float x = (float)(PARTS == 1 ? k : run_column<PARTS>(part, k / 2, k % 2)) - 0.5f * (kColRun - 1);
            const float p = fmaf(fmaf(b2, x, b1), x, qp);
            const float t = p + kMagic, f = p - (t - kMagic);
            const float4* w = reinterpret_cast<const float4*>(w0 + min(32u * (unsigned)__float_as_int(t) + bias, last));
            const float4 c01 = w[0], c23 = w[1];
            const float vr = fmaf(fmaf(fmaf(c23.z, f, c23.x), f, c01.z), f, c01.x);
            const float vi = fmaf(fmaf(fmaf(c23.w, f, c23.y), f, c01.w), f, c01.y);
            float sn, cs;
            __sincosf(fmaf(fmaf(fmaf(fmaf(P4, x, P3), x, P2), x, P1), x, P0), &sn, &cs);
            ar[k] = fmaf(vr, cs, ar[k]);
            ar[k] = fmaf(-vi, sn, ar[k]);
            ai[k] = fmaf(vr, sn, ai[k]);
            ai[k] = fmaf(vi, cs, ai[k]);
        }
    }
}

// Coefficients along a run of columns: at = (ground range) / d, z = 1 / (2 pi K d) at the run's middle and
// T_j the phase's coefficients at unit ground range and distance (radians).  From
//   d(m)^2 = d^2 - 2 g sum_j (a . s_j) m^j   (a the pulse's offset from the grid's origin).
__device__ __forceinline__ void run_phase(float at, float z, float T1, float T2, float T3, float T4, float& P1, float& P2,
                                          float& P3, float& P4) {
    P1 = at * T1;
    const float y1 = z * P1;
    P2 = fmaf(-0.5f * P1, y1, at * T2);
    P3 = fmaf(-y1, P2, at * T3);
    P4 = fmaf(-y1, P3, fmaf(-0.5f * z * P2, P2, at * T4));
}

struct PolarBody {
    static constexpr int kRecMode = 0;
    // Polar grids stage their windows with one load per lane and shuffled neighbours (751 against
    // 744 Gpixel-pulses/s on the 4096-pulse root grid); the lattice loop measured 0.5% slower with it.
    static constexpr bool kShflWindows = true;
    const SplitParams& P;
    Pix* px;
    __device__ void fast(const Rec* rec, const float4* win, int nfit, int) { polar_chunk(P, rec, win, nfit, px); }
    __device__ void slow(int c0, int nslow, const SlowRec* srec) {
#pragma unroll
        for (int k = 0; k < kPX; ++k) {
            const Pix& q = px[k];
            // Pulse by pulse onto the pixel's sum, so that the image does not depend on the chunks.
            const float2 v = slow_pixel(P, srec, 0, nslow, 1, c0, q.dxh, q.dxl, q.dyh, q.dyl, q.dzh, q.dzl, q.psi, q.ar, q.ai);
            px[k].ar = v.x;
            px[k].ai = v.y;
        }
    }
};

struct PointsBody {
    static constexpr int kRecMode = 3;
    static constexpr bool kShflWindows = false;
    const SplitParams& P;
    const TileShared& S;
    PointPix* px;
    __device__ void fast(const Rec* rec, const float4* win, int nfit, int) {
        points_chunk(P, rec, win, S.rest, nfit, px);
    }
    __device__ void slow(int c0, int nslow, const SlowRec* srec) {
#pragma unroll
        for (int k = 0; k < kPointPX; ++k) {
            const PointPix& q = px[k];
            const float2 v = slow_pixel(P, srec, 0, nslow, 1, c0, q.dx, q.lx, q.dy, q.ly, q.dz, q.lz, 0.0f, 0.0f, 0.0f);
            px[k].ar += v.x;
            px[k].ai += v.y;
        }
    }
};

// ---- lattice tiles: runs of eight rows ---------------------------------------------------
//
// On a lattice the pixel offset is delta = i s_row + j s_col, so u . delta and W . delta
// split into row and column terms.  A thread holds a run of eight pixels, rows i0 + k of one
// column, k = -3.5 .. 3.5 about the run's middle.  Per pulse it forms the range D and the
// reduced phase at the middle from the record's terms, with the exact hi products, and then
// steps along the run with the Taylor series of d(k) = |V + k s_row| (V: antenna to middle):
//   d(k) = D + a k + e2 k^2 + e3 k^3 + e4 k^4,   a = V . s_row / D,
//   e2 = (s^2 - a^2) / 2D,  e3 = -a e2 / D,  e4 = (s^2 - a^2)(5 a^2 - s^2) / 8 D^3.
// a = u . s_row + e1 with e1 = (delta . s_row - (D - R) u . s_row) / D small, so the large
// linear phase K k u . s_row stays in the record's exactly reduced step and only K (e1 k +
// e2 k^2 + e3 k^3) is FP32.  e4 is a per-record constant (it varies by 1% over a tile and is
// below 1e-10 m at a kilometre); over the run's four |k| it is folded into the constant and
// the e2 term (k^4 ~ 12.5 k^2 - 21.0625 within 18).  The envelope bounds the rest: K rho^2 <= 8 R
// leaves a residual below 0.004 / (K R) rad.
//
// Per pixel-pulse that leaves five packed operations per pixel pair for the range and the
// phase, the window gather, the cubic and the rotation; the run's own set-up (about 60
// instructions) is shared by eight pixels.
//
// What bounds the loop: the register file feeds two operands a cycle to the FMA pipe (a fused
// multiply-add of three registers takes 1.5 cycles, a packed one 3), so issue sits at 71% with the
// FMA pipe, the shared-memory pipe and issue all at 60-70%, and every instruction removed shows in
// the time.  4096 pulses onto 2048 x 2048: 16.94 ms (1014 Gpixel-pulses/s; 28.9 instructions per
// pixel-pulse), 19.6 ms (876; 31.3) with four pixels per thread and the root-free range chain of the
// adjoint per pixel.  Measured and not kept: runs of 16 (24 warps per SM instead of 32: 16.7 ms, but a larger
// error on small scenes), the range to the middle in integers too (18.3; error 0.68e-6 instead of 0.80), even
// and odd parts of the polynomials with constant multipliers (17.2), scalar cubic (17.5), staging two bins per
// lane (17.15) and three blocks per SM (17.7).
constexpr int kRun = 8;                               // pixels per run
constexpr int kRunThreads = kSplitTilePixels / kRun;  // threads per pulse group

// Forward on lattice tiles.  The block's two halves take alternate pulses of the tile (by the
// parity of the pulse's distance from the range's first, so that the image does not depend on
// the chunks) and their images are added once at the end.
__device__ __forceinline__ void lattice_runs(const SplitParams& P, const Rec* __restrict__ rec,
                                             const char* __restrict__ win, int first, int chn, float di, float dj,
                                             int hi2, int ji, float d2, float ds, float s2, float ar[kRun], float ai[kRun]) {
    const float inv_dr = P.inv_drf, kr = P.Kf * kTwoPiF;
    const float2 magic = pair(kMagic), nmagic = pair(-kMagic), mone = pair(-1.0f);
#pragma unroll 1
    for (int nl = first; nl < chn; nl += 2) {
        const int4 ra = *reinterpret_cast<const int4*>(&rec[nl].a);
        const float4 rb = rec[nl].b, rc = rec[nl].c;
        const float2 rd = *reinterpret_cast<const float2*>(&rec[nl].d);
        const unsigned wbase = (unsigned)__float_as_int(rc.y);
        const float L = fmaf(dj, rb.y, di * rb.x);
        const int turns = (int)((unsigned)__float_as_int(rc.x) + (unsigned)ra.x * (unsigned)hi2 + (unsigned)ra.y * (unsigned)ji);
        const float q2 = fmaf(-L, L, d2);
        const float h = rb.z + L;
        const float B = rcp_approx(h + h);
        const float e0 = q2 * B;
        const float eps = fmaf(-e0 * e0, B, e0);
        const float iD = rcp_approx(h + eps);
        const float Le = L + eps;
        const float e1 = fmaf(-Le, rb.x, ds) * iD;
        const float a = rb.x + e1;
        const float e2 = fmaf(fmaf(-a, a, s2), 0.5f * iD, rc.w);
        const float e3 = -a * e2 * iD;
        float P0 = fmaf(P.Kf, eps, (float)turns * 2.3283064365386963e-10f);
        P0 -= round_magic(P0);
        const float2 p0 = __ffma2_rn(pair(P0), pair(kTwoPiF), rd);
        const float2 p1 = pair(fmaf(kr, e1, rc.z));
        const float2 p2 = pair(kr * e2), p3 = pair(kr * e3);
        const float2 q0 = pair(fmaf(Le, inv_dr, rb.w)), q1 = pair(a * inv_dr), q2k = pair(e2 * inv_dr);
#pragma unroll
        for (int g = 0; g < kRun / 2; ++g) {
            const float2 kk = make_float2(2.0f * g - 3.5f, 2.0f * g - 2.5f);
            const float2 ang = __ffma2_rn(__ffma2_rn(__ffma2_rn(p3, kk, p2), kk, p1), kk, p0);
            const float2 qp = __ffma2_rn(__ffma2_rn(q2k, kk, q1), kk, q0);
            const float2 tq = __fadd2_rn(qp, magic);
            const float2 s = __ffma2_rn(__fadd2_rn(tq, nmagic), mone, qp);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int k = 2 * g + c;
                // The record's window holds every bin a pixel of the tile can round to, with half a bin to
                // spare, so the index needs no clamp.
                const float4* w = reinterpret_cast<const float4*>(
                    win + (32u * (unsigned)__float_as_int(c ? tq.y : tq.x) + wbase));
                const float4 c01 = w[0], c23 = w[1];
                const float2 ss = pair(c ? s.y : s.x);
                const float2 v = __ffma2_rn(
                    __ffma2_rn(__ffma2_rn(make_float2(c23.z, c23.w), ss, make_float2(c23.x, c23.y)), ss,
                               make_float2(c01.z, c01.w)),
                    ss, make_float2(c01.x, c01.y));
                float sn, cs;
                __sincosf(c ? ang.y : ang.x, &sn, &cs);
                ar[k] = fmaf(v.x, cs, ar[k]);
                ar[k] = fmaf(-v.y, sn, ar[k]);
                ai[k] = fmaf(v.x, sn, ai[k]);
                ai[k] = fmaf(v.y, cs, ai[k]);
            }
        }
    }
}

// Pulses the fast path cannot stage, every second one from `first`, on the run's pixels, out of line so that it
// costs the fast path no registers.  The run's first offset in FP64, the others by steps in two-float: in FP64,
// eight pixels a chunk in both halves of the block, the offsets took as long as the pulses.  256 pulses onto
// 512 x 512 pixels of 1, 2 and 5 m (wide tiles): 290, 734 and 1557 us so, 268, 607 and 742 now (four pixels
// per thread, before there were runs: 257, 583 and 908).
__device__ __noinline__ void lattice_run_slow(const SplitParams& P, const TileShared& S, const sarbp_lattice& L, float di,
                                              float dj, int first, int nslow, int c0, const SlowRec* srec,
                                              float2* more) {
    FF X, Y, Z;
    const double i = (double)(di - 3.5f), j = (double)dj;
    split2(i * L.step_row[0] + j * L.step_col[0], X.h, X.l);
    split2(i * L.step_row[1] + j * L.step_col[1], Y.h, Y.l);
    split2(i * L.step_row[2] + j * L.step_col[2], Z.h, Z.l);
#pragma unroll 1
    for (int k = 0; k < kRun; ++k) {
        more[k] = slow_pixel(P, srec, first, nslow, 2, c0, X.h, X.l, Y.h, Y.l, Z.h, Z.l, 0.0f, 0.0f, 0.0f);
        X = ff_add(X, FF{S.sth[0], S.stl[0]});
        Y = ff_add(Y, FF{S.sth[1], S.stl[1]});
        Z = ff_add(Z, FF{S.sth[2], S.stl[2]});
    }
}

struct LatticeBody {
    static constexpr int kRecMode = 1;
    static constexpr bool kShflWindows = false;
    const SplitParams& P;
    const TileShared& S;
    const sarbp_lattice& lat;
    int p0;
    float di, dj, d2, ds, s2;  // the run's middle: offsets (rows, columns), |delta|^2, delta . s_row; |s_row|^2
    float* ar;
    float* ai;
    __device__ int group() const { return threadIdx.x / kRunThreads; }
    __device__ void fast(const Rec* rec, const float4* win, int nfit, int c0) {
        lattice_runs(P, rec, reinterpret_cast<const char*>(win), (c0 - p0 + group()) & 1, nfit, di, dj,
                     (int)(2.0f * di), (int)dj, d2, ds, s2, ar, ai);
    }
    __device__ void slow(int c0, int nslow, const SlowRec* srec) {
        float2 more[kRun];
        lattice_run_slow(P, S, lat, di, dj, (c0 - p0 + group()) & 1, nslow, c0, srec, more);
#pragma unroll
        for (int k = 0; k < kRun; ++k) {
            ar[k] += more[k].x;
            ai[k] += more[k].y;
        }
    }
};

// ---- adjoint (gradients of a real image loss) -------------------------------------------
//
// With G_p = dl/dRe I_p + i dl/dIm I_p and c_pn = w_n v_pn exp(i phi_pn), the
// per-pulse sums U_n = sum_p conj(G_p) v_pn exp(i phi_pn) and
// A_n = sum_p Re(conj(G_p) (v'_pn / data_dr + i k v_pn) exp(i phi_pn)) e_pn
// (e_pn the unit vector from pos_n to pixel p, v' = d sample1 / dq) give
// dl/dpos_n = -w_n A_n, dl/dphase_n = -w_n Im U_n, dl/dweight_n = Re U_n.
// Each CTA recomputes its tile's contributions and writes per-pulse partial
// sums; adjoint_sum_kernel adds the tiles in fixed order.
constexpr int kAdjVals = 5;  // Re U, Im U, A.x, A.y, A.z

template <bool HAS_Z, bool DEMOD>
struct AdjointBody {
    static constexpr int kRecMode = 0;
    static constexpr bool kShflWindows = false;
    const SplitParams& P;
    const TileShared& S;
    Pix* px;
    const float* gre;
    const float* gim;
    float (*red)[kMaxChunk][kAdjVals];  // [warp][pulse][value]
    float* part;                        // this tile's partial sums, [pulse][kAdjVals]
    int pixels;                         // pixels of the tile that exist (the rest have G = 0)

    __device__ void flush(int n0, int cnt) {
        __syncthreads();
        for (int t = threadIdx.x; t < cnt * kAdjVals; t += kThreads) {
            const int nl = t / kAdjVals, v = t - nl * kAdjVals;
            float acc = 0.0f;
#pragma unroll
            for (int w = 0; w < kThreads / 32; ++w) acc += red[w][nl][v];
            part[(size_t)(n0 + nl) * kAdjVals + v] = acc;
        }
    }

    __device__ void fast(const Rec* rec, const float4* win, int nfit, int c0) {
        const float inv_dr = P.inv_drf, Kf = P.Kf, kr = P.Kf * kTwoPiF;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
        for (int nl = 0; nl < nfit; ++nl) {
            // rd.x (the unit vector's z) is needed for the z gradient even on a flat lattice.
            const float4 ra = rec[nl].a, rb = rec[nl].b, rc = rec[nl].c, rd = rec[nl].d;
            const int bias = __float_as_int(rc.y);
            const unsigned last = (unsigned)__float_as_int(rc.w);
            const float4* wrow = win + 2 * __float_as_int(rc.z);
            const float R = 0.5f * rb.z;
            float v5[kAdjVals] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < kPX; ++k) {
                const Pix& q = px[k];
                float L = fmaf(rb.x, q.dx, rb.y * q.dy);
                if (HAS_Z) L = fmaf(rd.x, q.dz, L);
                const float q2 = fmaf(-L, L, q.d2);
                const float B = rcp_approx(fmaf(2.0f, L, rb.z));
                const float e0 = q2 * B;
                const float eps = fmaf(-e0 * e0, B, e0);
                const float qp = fmaf(L + eps, inv_dr, rb.w);
                const float tq = qp + kMagic;
                const float s = qp - (tq - kMagic);
                const unsigned j = min((unsigned)(__float_as_int(tq) - bias), last);
                const float4 c01 = wrow[2 * j], c23 = wrow[2 * j + 1];
                const float vr = fmaf(fmaf(fmaf(c23.z, s, c23.x), s, c01.z), s, c01.x);
                const float vi = fmaf(fmaf(fmaf(c23.w, s, c23.y), s, c01.w), s, c01.y);
                const float dvr = fmaf(fmaf(3.0f * c23.z, s, 2.0f * c23.x), s, c01.z);
                const float dvi = fmaf(fmaf(3.0f * c23.w, s, 2.0f * c23.y), s, c01.w);
                float tb = ra.y * q.dyh;
                if (HAS_Z) tb = fmaf(rd.y, q.dzh, tb);
                tb = fmaf(ra.x, q.dxh, tb);
                float sm = fmaf(Kf, eps, rc.x);
                sm = fmaf(ra.x, q.dxl, sm);
                sm = fmaf(ra.y, q.dyl, sm);
                sm = fmaf(ra.z, q.dx, sm);
                sm = fmaf(ra.w, q.dy, sm);
                if (HAS_Z) {
                    sm = fmaf(rd.y, q.dzl, sm);
                    sm = fmaf(rd.z, q.dz, sm);
                }
                if (DEMOD) sm += q.psi;
                const float tot = (tb - round_magic(tb)) + sm;
                const float ang = (tot - round_magic(tot)) * kTwoPiF;
                float sn, cs;
                __sincosf(ang, &sn, &cs);
                const float gr = gre[k], gi = gim[k];
                const float er = vr * cs - vi * sn, ei = vr * sn + vi * cs;  // v exp(i phi)
                v5[0] = fmaf(gr, er, fmaf(gi, ei, v5[0]));
                v5[1] = fmaf(gr, ei, fmaf(-gi, er, v5[1]));
                const float zr = fmaf(dvr, inv_dr, -kr * vi), zi = fmaf(dvi, inv_dr, kr * vr);
                const float fr = zr * cs - zi * sn, fi = zr * sn + zi * cs;
                const float t = fmaf(gr, fr, gi * fi) * rcp_approx(R + L + eps);
                v5[2] = fmaf(t, fmaf(R, rb.x, q.dx), v5[2]);
                v5[3] = fmaf(t, fmaf(R, rb.y, q.dy), v5[3]);
                v5[4] = fmaf(t, fmaf(R, rd.x, q.dz), v5[4]);
            }
#pragma unroll
            for (int v = 0; v < kAdjVals; ++v) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v5[v] += __shfl_xor_sync(0xffffffffu, v5[v], o);
            }
            if (lane == 0) {
#pragma unroll
                for (int v = 0; v < kAdjVals; ++v) red[warp][nl][v] = v5[v];
            }
        }
        flush(c0, nfit);
    }

    // Pulses the fast path cannot stage: two-float geometry per pixel, FP32 interpolation.
    __device__ void slow(int c0, int nslow, const SlowRec* srec) {
        const PulseInputs& in = P.in;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const float kr = P.Kf * kTwoPiF, inv_dr = P.inv_drf;
#pragma unroll 1
        for (int j = 0; j < nslow; ++j) {
            const SlowRec sr = srec[j];
            const float2* row = in.data + (size_t)(c0 + j) * in.samples;
            float v5[kAdjVals] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < kPX; ++k) {
                SlowSample o;
                if (!slow_sample<true>(P, sr, row, px[k], DEMOD ? px[k].psi : 0.0f, o)) continue;
                float sn, cs;
                __sincosf(o.ang, &sn, &cs);
                const float gr = gre[k], gi = gim[k];
                const float er = o.vr * cs - o.vi * sn, ei = o.vr * sn + o.vi * cs;
                v5[0] = fmaf(gr, er, fmaf(gi, ei, v5[0]));
                v5[1] = fmaf(gr, ei, fmaf(-gi, er, v5[1]));
                const float zr = fmaf(o.dvr, inv_dr, -kr * o.vi), zi = fmaf(o.dvi, inv_dr, kr * o.vr);
                const float fr = zr * cs - zi * sn, fi = zr * sn + zi * cs;
                const float t = fmaf(gr, fr, gi * fi);
                v5[2] = fmaf(t, o.ex, v5[2]);
                v5[3] = fmaf(t, o.ey, v5[3]);
                v5[4] = fmaf(t, o.ez, v5[4]);
            }
#pragma unroll
            for (int v = 0; v < kAdjVals; ++v) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v5[v] += __shfl_xor_sync(0xffffffffu, v5[v], o);
            }
            if (lane == 0) {
#pragma unroll
                for (int v = 0; v < kAdjVals; ++v) red[warp][j][v] = v5[v];
            }
        }
        flush(c0, nslow);
    }
};

// Adjoint on lattice tiles, with the forward's separable row/column terms.  Per pulse a
// thread sums its pixels' t_p = Re(conj(G_p) z_p e^{i phi}) / d_p as T0 = sum t_p and
// S1 = sum kc_p t_p; with delta_p = di_p s_row + dj_p s_col the position sum is
// A = sum t_p (R u + delta_p) = R u T0 + s_row Ti + s_col Tj, Ti = sum t_p di_p = di T0 + m S1,
// Tj = dj T0 (a thread's pixels share the column).  The warps reduce (Re U, Im U, T0, Ti, Tj)
// and the flush turns them into A with the chunk's records.
__device__ __noinline__ void lattice_adjoint_slow(const SplitParams& P, const TileShared& S, const Job& J, float g0,
                                                  float g1, float g2, float g3, float h0, float h1, float h2,
                                                  float h3, float (*red)[kMaxChunk][kAdjVals], float* part, int c0,
                                                  int nslow, const SlowRec* srec) {
    const sarbp_lattice& L = J.lat;
    const int tid = threadIdx.x, cols_t = 1 << J.lc, hr = (kSplitTilePixels >> J.lc) >> 1;
    const double dj = (double)((tid & (cols_t - 1)) - (cols_t >> 1));
    Pix px[kPX];
#pragma unroll
    for (int k = 0; k < kPX; ++k) {
        const double di = (double)(((tid + kThreads * k) >> J.lc) - hr);
        pixel_from_offsets(S, di * L.step_row[0] + dj * L.step_col[0], di * L.step_row[1] + dj * L.step_col[1],
                           di * L.step_row[2] + dj * L.step_col[2], px[k]);
        px[k].psi = 0.0f;
    }
    const float gre[kPX] = {g0, g1, g2, g3}, gim[kPX] = {h0, h1, h2, h3};
    static_assert(AdjointBody<true, false>::kRecMode == 0, "the fallback works from per-pixel offsets");
    AdjointBody<true, false> body{P, S, px, gre, gim, red, part, kSplitTilePixels};
    body.slow(c0, nslow, srec);  // writes A directly
}

// Warp sums of five values in 28 instructions instead of 50: the first two butterfly levels halve
// the values each lane carries (a lane keeps one of each pair and trades the other with its
// partner), the last three are plain.  Lane l ends with the sum of value (l >> 4) + 2 ((l >> 3) & 1)
// of v0..v3 in sq and of v4 in s4.
__device__ __forceinline__ void warp_sum5(float v0, float v1, float v2, float v3, float v4, float& sq, float& s4) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
    float a = h16 ? v1 : v0;
    a += __shfl_xor_sync(full, h16 ? v0 : v1, 16);
    float b = h16 ? v3 : v2;
    b += __shfl_xor_sync(full, h16 ? v2 : v3, 16);
    float e = v4 + __shfl_xor_sync(full, v4, 16);
    float c = h8 ? b : a;
    c += __shfl_xor_sync(full, h8 ? a : b, 8);
    e += __shfl_xor_sync(full, e, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        c += __shfl_xor_sync(full, c, o);
        e += __shfl_xor_sync(full, e, o);
    }
    sq = c;
    s4 = e;
}

struct LatticeAdjointBody {
    static constexpr int kRecMode = 2;
    static constexpr bool kShflWindows = false;
    const SplitParams& P;
    const TileShared& S;
    const Job& J;
    const float* d2;
    const float* gre;
    const float* gim;
    float (*red)[kMaxChunk][kAdjVals];
    float* part;

    __device__ void flush(int n0, int cnt, const Rec* rec) {
        __syncthreads();
        for (int nl = threadIdx.x; nl < cnt; nl += kThreads) {
            float v[kAdjVals];
#pragma unroll
            for (int c = 0; c < kAdjVals; ++c) {
                float acc = 0.0f;
#pragma unroll
                for (int w = 0; w < kThreads / 32; ++w) acc += red[w][nl][c];
                v[c] = acc;
            }
            const float4 rd = rec[nl].d;
            const float R = 0.5f * rec[nl].b.z, t0 = v[2], ti = v[3], tj = v[4];
            const float u[3] = {rd.y, rd.z, rd.w};
            float* out = part + (size_t)(n0 + nl) * kAdjVals;
            out[0] = v[0];
            out[1] = v[1];
#pragma unroll
            for (int c = 0; c < 3; ++c) out[2 + c] = fmaf(R * u[c], t0, fmaf(S.sth[c], ti, S.sth[3 + c] * tj));
        }
    }

    __device__ void fast(const Rec* rec, const float4* win, int nfit, int c0) {
        const float inv_dr = P.inv_drf, kr = P.Kf * kTwoPiF;
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lc = J.lc;
        const int m = kThreads >> lc, hr = (kSplitTilePixels >> lc) >> 1, cols_t = 1 << lc;
        const float di = (float)((tid >> lc) + 2 * m - hr);
        const float dj = (float)((tid & (cols_t - 1)) - (cols_t >> 1));
        const float mf = (float)m;
        // Pixel pairs as f32x2 lanes: -L, -q2, -e0 and -eps are carried (negation is exact), plus R + (L + eps).
        const float2 nd2[2] = {make_float2(-d2[0], -d2[1]), make_float2(-d2[2], -d2[3])};
        const float2 kcs[2] = {make_float2(-2.0f, -1.0f), make_float2(0.0f, 1.0f)};
        const float2 ninv = pair(-inv_dr), nkr = pair(-kr), magic = pair(kMagic), nmagic = pair(-kMagic);
        const float2 mone = pair(-1.0f), mtwo = pair(-2.0f), half = pair(0.5f);
#pragma unroll 1
        for (int nl = 0; nl < nfit; ++nl) {
            const float4 ra = rec[nl].a, rb = rec[nl].b, rc = rec[nl].c, rd = rec[nl].d, re = rec[nl].e;
            const int bias = __float_as_int(rc.y);
            const unsigned last = (unsigned)__float_as_int(rc.w);
            const float4* wrow = win + 2 * __float_as_int(rc.z);
            const float nL0 = fmaf(-dj, rb.y, -di * rb.x), nmA = -(mf * rb.x);  // -L0, -m u.s_row: exact
            const float t = fmaf(dj, ra.z, di * ra.x);                           // exact
            const float r0 = ((t - round_magic(t)) + fmaf(dj, ra.w, fmaf(di, ra.y, rc.x))) * kTwoPiF;
            const float2 twoR = make_float2(re.x, re.y), fm = make_float2(re.z, re.w);
            const float2 R2 = __fmul2_rn(twoR, half);
            const float2 nL02 = pair(nL0), nstep = pair(nmA), sp = pair(rd.x), r02 = pair(r0);
            float u0 = 0.f, u1 = 0.f, t0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 nL = __ffma2_rn(kcs[h], nstep, nL02);
                const float2 nq2 = __ffma2_rn(nL, nL, nd2[h]);
                const float2 den = __ffma2_rn(mtwo, nL, twoR);
                const float2 B = make_float2(rcp_approx(den.x), rcp_approx(den.y));
                const float2 ne0 = __fmul2_rn(nq2, B);
                const float2 neps = __ffma2_rn(__fmul2_rn(ne0, ne0), B, ne0);
                const float2 nLe = __fadd2_rn(nL, neps);  // -(L + eps)
                const float2 qp = __ffma2_rn(nLe, ninv, fm);
                const float2 tq = __fadd2_rn(qp, magic);
                const float2 s = __ffma2_rn(__fadd2_rn(tq, nmagic), mone, qp);
                const float2 ang = __ffma2_rn(nkr, neps, __ffma2_rn(kcs[h], sp, r02));
                const float2 dist = __ffma2_rn(nLe, mone, R2);  // R + (L + eps)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int k = 2 * h + c;
                    const float kc = (float)(k - 2);
                    const float tqc = c ? tq.y : tq.x;
                    const unsigned j = min((unsigned)(__float_as_int(tqc) - bias), last);
                    const float4 c01 = wrow[2 * j], c23 = wrow[2 * j + 1];
                    // Horner for the value as (re, im) pairs; the derivative c1 + 2 c2 s + 3 c3 s^2 =
                    // p2 + s (p1 + c3 s) reuses its partial results p1 = c3 s + c2, p2 = p1 s + c1.
                    const float2 ss = pair(c ? s.y : s.x), c3 = make_float2(c23.z, c23.w);
                    const float2 p1 = __ffma2_rn(c3, ss, make_float2(c23.x, c23.y));
                    const float2 p2 = __ffma2_rn(p1, ss, make_float2(c01.z, c01.w));
                    const float2 v = __ffma2_rn(p2, ss, make_float2(c01.x, c01.y));
                    const float2 dv = __ffma2_rn(ss, __ffma2_rn(c3, ss, p1), p2);
                    float sn, cs;
                    __sincosf(c ? ang.y : ang.x, &sn, &cs);
                    // h = conj(G) exp(i phi): U += v h, and the position weight
                    // Re(conj(G) (v'/dr + i k v) exp(i phi)) / d = (Re(v' h) / dr - k Im(v h)) / d.
                    const float gr = gre[k], gi = gim[k];
                    const float hr = fmaf(gr, cs, gi * sn), hi = fmaf(gr, sn, -gi * cs);
                    u0 = fmaf(v.x, hr, fmaf(-v.y, hi, u0));
                    const float w1 = fmaf(v.x, hi, v.y * hr);
                    u1 += w1;
                    const float q = fmaf(dv.x, hr, -dv.y * hi);
                    const float tt = fmaf(q, inv_dr, -kr * w1) * rcp_approx(c ? dist.y : dist.x);
                    t0 += tt;
                    s1 = fmaf(kc, tt, s1);
                }
            }
            float sq, s4;
            warp_sum5(u0, u1, t0, fmaf(di, t0, mf * s1), dj * t0, sq, s4);
            if ((lane & 7) == 0) red[warp][nl][(lane >> 4) | ((lane >> 2) & 2)] = sq;
            if (lane == 0) red[warp][nl][4] = s4;
        }
        flush(c0, nfit, rec);
    }

    __device__ void slow(int c0, int nslow, const SlowRec* srec) {
        lattice_adjoint_slow(P, S, J, gre[0], gre[1], gre[2], gre[3], gim[0], gim[1], gim[2], gim[3], red, part, c0,
                             nslow, srec);
    }
};

// ---- output ----------------------------------------------------------------------
__device__ __forceinline__ void store_window(const Job& J, int win_nr, int win_nu, const Pix px[kPX], float2* out,
                                             long long stride) {
    const int cols_t = 1 << J.lc;
#pragma unroll
    for (int k = 0; k < kPX; ++k) {
        const int p = threadIdx.x + kThreads * k;
        const int wr = J.tile_r + (p >> J.lc), wu = J.tile_u + (p & (cols_t - 1));
        if (wr < win_nr && wu < win_nu) out[(long long)wr * stride + wu] = make_float2(px[k].ar, px[k].ai);
    }
}

__device__ __forceinline__ void split_range(int p0, int p1, int parts, int part, int& b, int& e) {
    const long long len = (long long)p1 - p0;
    b = p0 + (int)(len * part / parts);
    e = p0 + (int)(len * (part + 1) / parts);
}

__device__ __forceinline__ void tile_of(int index, int win_nu, int lc, int& tile_r, int& tile_u) {
    const int cols_t = 1 << lc, rows_t = kSplitTilePixels >> lc;
    const int tiles_u = (win_nu + cols_t - 1) / cols_t;
    tile_r = (index / tiles_u) * rows_t;
    tile_u = (index % tiles_u) * cols_t;
}

// ---- direct BP kernels --------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 3) split_polar_kernel(SplitParams P, PolarDesc g) {
    extern __shared__ __align__(16) char smem[];
    __shared__ TileShared S;
    Job J;
    J.g = g;
    J.lc = g.tile_lc;
    tile_of(blockIdx.x, g.win_nu, J.lc, J.tile_r, J.tile_u);
    split_range(g.a, g.b, P.pulse_split, blockIdx.y, J.p0, J.p1);
    Pix px[kPX];
    PolarTables& T = *reinterpret_cast<PolarTables*>(smem + window_offset());
    setup_polar(P, J, S, T, px, true);
    PolarBody body{P, px};
    chunk_loop(P, J, S, smem, true, body);
    store_window(J, g.win_nr, g.win_nu, px, P.out + blockIdx.y * P.split_stride, P.out_stride);
}

// Add the two halves' images of a tile in runs of eight pixels: each half passes on four pixels of every run
// through shared memory and finishes the other four (store(k, value)).
template <class Store>
__device__ __forceinline__ void add_halves(float2* ex, int half, int slot, const float ar[kRun], const float ai[kRun],
                                           Store store) {
    __syncthreads();  // the last chunk's windows are consumed
#pragma unroll
    for (int k = 0; k < kRun / 2; ++k)
        ex[(kRun / 2 * half + k) * kRunThreads + slot] =
            half ? make_float2(ar[k], ai[k]) : make_float2(ar[k + kRun / 2], ai[k + kRun / 2]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRun / 2; ++k) {
        const float2 o = ex[(kRun / 2 * (1 - half) + k) * kRunThreads + slot];
        store(kRun / 2 * half + k, half ? make_float2(o.x + ar[k + kRun / 2], o.y + ai[k + kRun / 2])
                                        : make_float2(ar[k] + o.x, ai[k] + o.y));
    }
}

// Polar tile in runs of eight columns: a run's middle and what the expansion along it needs.
struct PolarRun {
    float dx, dy, dxh, dyh, dxl, dyl, d2, psi;  // the middle's offset from the tile centre, -K r modulo a turn
    float g;                                    // ground range of the row
    float s1, s2, s3, s4, h;                    // s = side sqrt(1 - u^2): s^(j)(u) du^j / j!; du
};

__device__ __forceinline__ void polar_run(const Job& J, const TileShared& S, const PolarTables& T, int row, int group,
                                          PolarRun& q) {
    const int m = kMaxCols + group;
    q.dxh = T.rxh[row] + T.cxh[m];  // exact: both multiples of the quantum
    q.dyh = T.ryh[row] + T.cyh[m];
    q.dxl = fmaf(T.dg[row], T.dcs[m], T.rxl[row] + T.cxl[m]);
    q.dyl = fmaf(T.dg[row], T.duu[m], T.ryl[row] + T.cyl[m]);
    q.dx = q.dxh + q.dxl;
    q.dy = q.dyh + q.dyl;
    q.d2 = q.dx * q.dx + q.dy * q.dy;
    q.psi = T.psi[row];
    q.g = T.dg[row] + sqrtf(S.sth[0] * S.sth[0] + S.sth[1] * S.sth[1]);
    const float u = T.mid_u[group], ic = 1.0f / T.mid_c[group];
    q.h = (float)J.g.du;
    const float hc = q.h * ic, hcc = hc * ic;
    q.s1 = (float)J.g.side * -u * hc;
    q.s2 = (float)J.g.side * -0.5f * hc * hc * ic;
    q.s3 = q.s2 * u * hcc;
    q.s4 = q.s2 * 0.25f * (1.0f + 4.0f * u * u) * hcc * hcc;
    __syncthreads();  // the tables alias the window region
}

// Pulses the fast path cannot stage on a run's pixels, every second one from `first`: offsets in two-float
// from FP64 (rare, and out of line so that it costs the fast path no registers).
__device__ __noinline__ void polar_run_slow(const SplitParams& P, const TileShared& S, const PolarDesc& g, int i, int j0,
                                            int first, int nslow, int c0, const SlowRec* srec, float2* sum) {
    const double r = g.r0 + (double)i * g.dr, gr = sqrt(fmax(0.0, r * r - g.oz * g.oz)), t = -P.K * r;
#pragma unroll 1
    for (int k = 0; k < kColRun; ++k) {
        const double u = g.u0 + (double)(j0 + k) * g.du;
        Pix q;
        pixel_from_offsets(S, g.ox + (double)g.side * gr * sqrt(fmax(0.0, 1.0 - u * u)) - S.cx, g.oy + gr * u - S.cy, 0.0,
                           q);
        // Pulse by pulse onto the run's sums, so that the image does not depend on the chunks.
        for (int j = first; j < nslow; j += 2) {
            const float2 v = slow_pixel(P, srec, j, j + 1, 1, c0, q.dxh, q.dxl, q.dyh, q.dyl, q.dzh, q.dzl,
                                        (float)(t - rint(t)), 0.0f, 0.0f);
            sum[k].x += v.x;
            sum[k].y += v.y;
        }
    }
}

// Direct BP on a polar tile in runs of eight columns; the block's halves take alternate pulses as the
// lattice tiles' do.  Range, phase and window place are worked out once per run (split arithmetic at its
// middle, as polar_chunk does per pixel) and expanded along it from the polar geometry (run_phase).
// What bounds it: instruction issue (77% of the cycles, 248 instructions per warp and pulse) and the last of
// few waves.  1024 pulses onto 720 x 1600: 1.27 ms, pixel by pixel (polar_chunk) 1.76; with every pixel on its
// own window entry 1.66, with 64 registers and four blocks per SM 1.35, with shuffled staging 1.31.
struct PolarRunBody {
    static constexpr int kRecMode = 4;
    static constexpr bool kShflWindows = false;
    const SplitParams& P;
    const TileShared& S;
    const PolarDesc& g;
    int p0;
    const PolarRun& q;
    int i, j0;
    float* ar;
    float* ai;
    __device__ int group() const { return threadIdx.x / kRunThreads; }
    __device__ void fast(const Rec* rec, const float4* win, int nfit, int c0) {
        const float inv_dr = P.inv_drf, Kf = P.Kf, kz = 1.0f / (kTwoPiF * Kf), kd = inv_dr * kz;
#pragma unroll 1
        for (int nl = (c0 - p0 + group()) & 1; nl < nfit; nl += 2) {
            const float4 ra = rec[nl].a, rb = rec[nl].b, rc = rec[nl].c, rd = rec[nl].d;
            const float L = fmaf(rb.x, q.dx, rb.y * q.dy);
            const float q2 = fmaf(-L, L, q.d2);
            const float B = rcp_approx(fmaf(2.0f, L, rb.z));
            const float e0 = q2 * B;
            const float eps = fmaf(-e0 * e0, B, e0);
            const float Le = L + eps;
            const float iR = rcp_approx(fmaf(0.5f, rb.z, Le));
            const float tb = fmaf(ra.x, q.dxh, ra.y * q.dyh);
            float sm = fmaf(Kf, eps, rc.x);
            sm = fmaf(ra.x, q.dxl, sm);
            sm = fmaf(ra.y, q.dyl, sm);
            sm = fmaf(ra.z, q.dx, sm);
            sm = fmaf(ra.w, q.dy, sm);
            const float P0 = ((tb - round_magic(tb)) + (sm + q.psi)) * kTwoPiF;
            float P1, P2, P3, P4;
            run_phase(q.g * iR, iR * kz, fmaf(rd.x, q.s1, rd.y * q.h), rd.x * q.s2, rd.x * q.s3, rd.x * q.s4, P1, P2, P3,
                      P4);
            column_run<1>(0, P0, P1, P2, P3, P4, fmaf(Le, inv_dr, rb.w), P1 * kd, P2 * kd, rd.z,
                       reinterpret_cast<const char*>(win + 2 * __float_as_int(rc.z)), 0u - 32u * (unsigned)__float_as_int(rc.y),
                       32u * (unsigned)__float_as_int(rc.w), ar, ai);
        }
    }
    __device__ void slow(int c0, int nslow, const SlowRec* srec) {
        float2 sum[kColRun];
#pragma unroll
        for (int k = 0; k < kColRun; ++k) sum[k] = make_float2(ar[k], ai[k]);
        polar_run_slow(P, S, g, i, j0, (c0 - p0 + group()) & 1, nslow, c0, srec, sum);
#pragma unroll
        for (int k = 0; k < kColRun; ++k) {
            ar[k] = sum[k].x;
            ai[k] = sum[k].y;
        }
    }
};

// Whether a polar tile is formed in runs, from 32 pulses spread over its range: they have to fit the fast path
// and the runs' expansion, and the range has to change by less than kRunSpread bins on average from a run's middle to
// its ends, so that runs of 32 neighbouring rows mostly stay within a bin.  Fully sampled apertures are at 0.006 (9.6 GHz,
// 0.83 m bins); coarser angle steps and longer waves go pixel by pixel.  256 pulses onto 720 x 512, rows of 0.72 bins,
// changes of 0.011, 0.016 and 0.021 bins: runs 181, 204 and 217 us, pixels 200, 212 and 211; rows of a bin: 160 (0.011)
// and 167 (0.021), pixels 212 and 217.  Tiles too wide for the fast path: runs 1400 to 2050 us, pixels 1020 to 1070
// (890 to 940 in split_polar_kernel, which has their code alone).
constexpr float kRunSpread = 0.02f;
__device__ __forceinline__ bool polar_in_runs(const SplitParams& P, const Job& J, TileShared& S) {
    __shared__ int runs;
    if (threadIdx.x < 32) {
        const double* p = P.in.pos + 3LL * (J.p0 + (J.p1 - 1 - J.p0) * (long long)threadIdx.x / 31);
        const float vx = (float)(S.cx - p[0]), vy = (float)(S.cy - p[1]), vz = (float)(S.cz - p[2]), rho = (float)S.rho;
        const float ax = S.sth[0] - vx, ay = S.sth[1] - vy, g2 = S.sth[0] * S.sth[0] + S.sth[1] * S.sth[1];
        const float R = sqrtf(fmaf(vx, vx, fmaf(vy, vy, vz * vz))), iR = 1.0f / R;
        const float du = (float)fabs(J.g.du), per_m = fabsf(P.inv_drf);
        float spread = 3.5f * du * per_m * sqrtf(g2) * iR * fabsf(ay - ax * S.sth[1] / S.sth[0]);
        const float turn = S.sth[3] * (fabsf(ax) + fabsf(ay)), y = turn * iR;
        const bool fits = fabsf(P.Kf) * rho * rho <= (float)P.envelope * R && rho < 0.25f * R &&
                          2.0f * rho * per_m + 4.0f <= (float)(kWindowBudget / 32) &&
                          fabsf(P.Kf) * (fabsf(ax) * S.sth[2] + turn * (y * y) * (y * y)) <= 1e-7f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) spread += __shfl_xor_sync(0xffffffffu, spread, o);
        const bool all = __all_sync(0xffffffffu, fits);
        if (threadIdx.x == 0) runs = all && spread <= 32.0f * kRunSpread;
    }
    __syncthreads();
    return runs != 0;
}

__global__ void __launch_bounds__(kThreads, 3) split_polar_runs_kernel(SplitParams P, PolarDesc g) {
    extern __shared__ __align__(16) char smem[];
    __shared__ TileShared S;
    Job J;
    J.g = g;
    J.lc = g.tile_lc;  // 3 to 5: whole runs, and a warp's 32 rows in one run of columns
    tile_of(blockIdx.x, g.win_nu, J.lc, J.tile_r, J.tile_u);
    split_range(g.a, g.b, P.pulse_split, blockIdx.y, J.p0, J.p1);
    PolarTables& T = *reinterpret_cast<PolarTables*>(smem + window_offset());
    polar_tables<true>(P, J, S, T, true);
    float2* out = P.out + blockIdx.y * P.split_stride;
    if (!polar_in_runs(P, J, S)) {
        Pix px[kPX];
        polar_pixels(J, T, px);
        PolarBody body{P, px};
        chunk_loop(P, J, S, smem, true, body);
        store_window(J, g.win_nr, g.win_nu, px, out, P.out_stride);
        return;
    }
    const int rows_t = kSplitTilePixels >> J.lc, slot = threadIdx.x & (kRunThreads - 1);
    const int row = slot & (rows_t - 1), col = kColRun * (slot / rows_t);
    PolarRun q;
    polar_run(J, S, T, row, col / kColRun, q);
    float ar[kColRun], ai[kColRun];
#pragma unroll
    for (int k = 0; k < kColRun; ++k) ar[k] = ai[k] = 0.0f;
    PolarRunBody body{P, S, g, J.p0, q, g.win_r0 + J.tile_r + row, g.win_u0 + J.tile_u + col, ar, ai};
    chunk_loop(P, J, S, smem, true, body);
    add_halves(reinterpret_cast<float2*>(smem + window_offset()), body.group(), slot, ar, ai, [&](int k, float2 v) {
        const int wr = J.tile_r + row, wu = J.tile_u + col + k;
        if (wr < g.win_nr && wu < g.win_nu) out[(long long)wr * P.out_stride + wu] = v;
    });
}

// One lattice tile over pulses [p0, p1): the per-item body shared by the one-tile-per-CTA
// kernel and the persistent batch kernel.
__device__ __forceinline__ void lattice_tile(const SplitParams& P, const sarbp_lattice& lat, int lc, int tile_r,
                                             int tile_u, int p0, int p1, float2* out, TileShared& S, char* smem) {
    Job J;
    J.lat = lat;
    J.lc = lc;
    J.tile_r = tile_r;
    J.tile_u = tile_u;
    J.p0 = p0;
    J.p1 = p1;
    setup_lattice_tile(J, S);
    const int cols_t = 1 << lc, hr = (kSplitTilePixels >> lc) >> 1;
    const int slot = threadIdx.x & (kRunThreads - 1), col = slot & (cols_t - 1), row0 = kRun * (slot >> lc);
    const float di = (float)(row0 - hr) + 3.5f, dj = (float)(col - (cols_t >> 1));
    float d2 = 0.0f, ds = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float x = fmaf(di, S.sth[c], dj * S.sth[3 + c]);
        d2 = fmaf(x, x, d2);
        ds = fmaf(x, S.sth[c], ds);
        s2 = fmaf(S.sth[c], S.sth[c], s2);
    }
    float ar[kRun], ai[kRun];
#pragma unroll
    for (int k = 0; k < kRun; ++k) ar[k] = ai[k] = 0.0f;
    LatticeBody body{P, S, lat, p0, di, dj, d2, ds, s2, ar, ai};
    chunk_loop(P, J, S, smem, true, body);
    add_halves(reinterpret_cast<float2*>(smem + window_offset()), body.group(), slot, ar, ai, [&](int k, float2 v) {
        const int wr = tile_r + row0 + k, wu = tile_u + col;
        if (wr < lat.rows && wu < lat.cols) out[(long long)wr * lat.cols + wu] = v;
    });
}

__global__ void __launch_bounds__(kThreads, 4) split_lattice_kernel(SplitParams P, sarbp_lattice lat, int lc) {
    extern __shared__ __align__(16) char smem[];
    __shared__ TileShared S;
    int tile_r, tile_u, p0, p1;
    tile_of(blockIdx.x, lat.cols, lc, tile_r, tile_u);
    split_range(0, P.in.pulses, P.pulse_split, blockIdx.y, p0, p1);
    lattice_tile(P, lat, lc, tile_r, tile_u, p0, p1, P.out + blockIdx.y * P.split_stride, S, smem);
}

__global__ void __launch_bounds__(kThreads, 3) split_points_kernel(SplitParams P, const double* __restrict__ xyz,
                                                                   int npts, const PointOrder* __restrict__ order,
                                                                   const int* __restrict__ index) {
    extern __shared__ __align__(16) char smem[];
    __shared__ TileShared S;
    Job J;
    J.xyz = xyz;
    J.index = order && !order->narrow ? index : nullptr;
    J.lc = 0;
    J.tile_r = blockIdx.x * kPointTile;
    J.tile_u = 0;
    split_range(0, P.in.pulses, P.pulse_split, blockIdx.y, J.p0, J.p1);
    const int end = min(npts, J.tile_r + kPointTile);
    // A tile too wide for the fast path whose list jumps (a spatial order leaves and re-enters the points' outline,
    // targets follow each other) is formed stretch by stretch: whole, on the two-float fallback, it would take as long
    // as seven others and hold up the launch's end.  Lists that jump all the time stay whole.
    __shared__ unsigned jumps[kPointTile / 32];
    __shared__ float limit;
    float2* out = P.out + blockIdx.y * P.split_stride;
    J.p_begin = J.tile_r;
    J.p_end = end;
    int njumps = -1;  // not looked for yet
    while (J.p_begin < end) {
        PointPix px[kPointPX];
        setup_points(J, S, px);
        if (njumps < 0) {
            if (threadIdx.x < 32) {  // lanes 0 to 2: the range to the tile's first, middle and last pulse
                const double* p = P.in.pos + 3LL * (J.p0 + (J.p1 - 1 - J.p0) * (long long)min(threadIdx.x, 2) / 2);
                const float dx = (float)(S.cx - p[0]), dy = (float)(S.cy - p[1]), dz = (float)(S.cz - p[2]);
                float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                r2 = fminf(r2, fminf(__shfl_sync(0xffffffffu, r2, 1), __shfl_sync(0xffffffffu, r2, 2)));
                if (threadIdx.x == 0) limit = points_radius(P.Kf, P.inv_drf, (float)P.cap, sqrtf(r2));
            }
            __syncthreads();
            njumps = 0;
            if ((float)S.rho > limit) {
                const float far = 0.7f * limit;
#pragma unroll
                for (int k = 0; k < kPointPX; ++k) {
                    const int at = J.tile_r + threadIdx.x + kThreads * k;
                    bool jump = false;
                    if (at > J.tile_r && at < end) {
                        const double* a = xyz + 3LL * (J.index ? J.index[at] : at);
                        const double* b = xyz + 3LL * (J.index ? J.index[at - 1] : at - 1);
                        const float dx = (float)a[0] - (float)b[0], dy = (float)a[1] - (float)b[1], dz = (float)a[2] - (float)b[2];
                        jump = dx * dx + dy * dy + dz * dz > far * far;
                    }
                    const unsigned w = __ballot_sync(0xffffffffu, jump);
                    if ((threadIdx.x & 31) == 0) jumps[(threadIdx.x + kThreads * k) >> 5] = w;
                }
                __syncthreads();
                for (int w = 0; w < kPointTile / 32; ++w) njumps += __popc(jumps[w]);
                if (njumps > 4) njumps = 0;
                if (njumps > 0) J.p_end = J.tile_r;  // start over, with the first stretch
            }
        }
        if (J.p_end > J.p_begin) {
            PointsBody body{P, S, px};
            chunk_loop(P, J, S, smem, true, body);
#pragma unroll
            for (int k = 0; k < kPointPX; ++k) {
                const int idx = J.tile_r + threadIdx.x + kThreads * k;
                if (idx >= J.p_begin && idx < J.p_end) out[J.index ? J.index[idx] : idx] = make_float2(px[k].ar, px[k].ai);
            }
        }
        __syncthreads();  // the next stretch's set-up
        J.p_begin = J.p_end;
        J.p_end = end;
        if (njumps > 0)
            for (int w = (J.p_begin + 1 - J.tile_r) >> 5, from = (J.p_begin + 1 - J.tile_r) & 31; w < kPointTile / 32;
                 ++w, from = 0) {
                const unsigned rest = jumps[w] & (0xffffffffu << from);
                if (rest) {
                    J.p_end = J.tile_r + 32 * w + __ffs(rest) - 1;
                    break;
                }
            }
    }
}

// ---- adjoint kernels ----------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 3) split_lattice_adjoint_kernel(SplitParams P, sarbp_lattice lat, int lc,
                                                                            const float2* __restrict__ grad,
                                                                            float* __restrict__ partials) {
    extern __shared__ __align__(16) char smem[];
    __shared__ TileShared S;
    __shared__ float red[kThreads / 32][kMaxChunk][kAdjVals];
    Job J;
    J.lat = lat;
    J.lc = lc;
    tile_of(blockIdx.x, lat.cols, lc, J.tile_r, J.tile_u);
    split_range(0, P.in.pulses, gridDim.y, blockIdx.y, J.p0, J.p1);  // the splits write disjoint partials
    float d2[kPX], gre[kPX], gim[kPX];
    setup_lattice_sep(J, S, d2);
    const int cols_t = 1 << lc;
#pragma unroll
    for (int k = 0; k < kPX; ++k) {
        const int p = threadIdx.x + kThreads * k;
        const int i = J.tile_r + (p >> lc), j = J.tile_u + (p & (cols_t - 1));
        float2 g = make_float2(0.0f, 0.0f);
        if (i < lat.rows && j < lat.cols) g = grad[(size_t)i * lat.cols + j];
        gre[k] = g.x;
        gim[k] = g.y;
    }
    LatticeAdjointBody body{P, S, J, d2, gre, gim, red, partials + (size_t)blockIdx.x * P.in.pulses * kAdjVals};
    chunk_loop(P, J, S, smem, false, body);
}

// Per-pulse gradients from the tiles' partial sums, in a fixed order (deterministic): each
// block takes 32 pulses; its 8 thread groups sum every 8th tile (coalesced: for one tile the
// 32 pulses' values are contiguous), then the 8 group sums are added in group order.
constexpr int kSumPulses = 32, kSumGroups = kThreads / kSumPulses;

__global__ void __launch_bounds__(kThreads) adjoint_sum_kernel(const float* __restrict__ partials, int ntiles,
                                                               int pulses, const double* __restrict__ weight,
                                                               double* grad_pos, double* grad_phase,
                                                               double* grad_weight) {
    __shared__ double part[kSumGroups][kSumPulses][kAdjVals];
    const int pl = threadIdx.x % kSumPulses, grp = threadIdx.x / kSumPulses;
    const int n = blockIdx.x * kSumPulses + pl;
    double acc[kAdjVals] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (n < pulses) {
        for (int t = grp; t < ntiles; t += kSumGroups) {
            const float* p = partials + ((size_t)t * pulses + n) * kAdjVals;
#pragma unroll
            for (int v = 0; v < kAdjVals; ++v) acc[v] += (double)p[v];
        }
    }
#pragma unroll
    for (int v = 0; v < kAdjVals; ++v) part[grp][pl][v] = acc[v];
    __syncthreads();
    if (grp != 0 || n >= pulses) return;
#pragma unroll
    for (int v = 0; v < kAdjVals; ++v) {
        double s = part[0][pl][v];
        for (int g = 1; g < kSumGroups; ++g) s += part[g][pl][v];
        acc[v] = s;
    }
    const double w = weight[n];
    if (grad_pos) {
        grad_pos[3 * n] = -w * acc[2];
        grad_pos[3 * n + 1] = -w * acc[3];
        grad_pos[3 * n + 2] = -w * acc[4];
    }
    if (grad_phase) grad_phase[n] = -w * acc[1];
    if (grad_weight) grad_weight[n] = acc[0];
}

// ---- FFBP: per-node tables and per-pulse leaf records (prologue kernels) ------------------
// Two-float constants of the table entries: K (turns/m), range_start, 1 / data_dr.
struct TableConsts {
    float Kh, Kl, rsh, rsl, idrh, idrl;
};

__host__ __device__ inline TableConsts table_consts(const SplitParams& P) {
    return TableConsts{P.Kh, P.Kl, P.rsh, P.rsl, P.idrh, P.idrl};
}

__device__ __forceinline__ FF ff_sqrt0(FF a) { return a.h > 0.0f ? ff_sqrt(a) : FF{0.0f, 0.0f}; }

// Row t and column t of node g's tables in two-float FP32 arithmetic from the node geometry
// split on the host (PolarDesc::tf).
__device__ __forceinline__ void table_entries(const TableConsts& C, const PolarDesc& g, int t,
                                              float4* __restrict__ tables) {
    const FF ft{(float)t, 0.0f};  // exact: node dimensions are far below 2^24
    if (t < g.nr) {
        const FF r = ff_add(ff_of(g.tf[3]), ff_mul(ft, ff_of(g.tf[4])));
        const FF oz = ff_of(g.tf[2]);
        const FF gg = ff_sqrt0(ff_add(ff_sqr(r), ff_neg(ff_sqr(oz))));
        const FF ph = ff_mul(FF{-C.Kh, -C.Kl}, r);
        float psi = (ph.h - rintf(ph.h)) + ph.l;
        psi -= rintf(psi);
        const FF ir = ff_rcp(r);
        const FF gr = ff_mul(gg, ir), ez = ff_mul(ff_neg(oz), ir);
        float F;
        const float I = fminf(fmaxf(ff_floor_frac(ff_mul(ff_add(r, FF{-C.rsh, -C.rsl}), FF{C.idrh, C.idrl}), F),
                                    -1.0e9f), 1.0e9f);
        float4* row = tables + g.rows_off + 3 * (long long)t;
        row[0] = make_float4(gg.h, gg.l, psi, 0.0f);
        row[1] = make_float4(gr.h, gr.l, ez.h, ez.l);
        row[2] = make_float4(2.0f * (r.h + r.l), F, __int_as_float((int)I), 0.0f);
    }
    if (t < g.nu) {
        const FF u = ff_add(ff_of(g.tf[5]), ff_mul(ft, ff_of(g.tf[6])));
        const FF c = ff_sqrt0(ff_add(FF{1.0f, 0.0f}, ff_neg(ff_sqr(u))));
        tables[g.cols_off + t] = make_float4(c.h, c.l, u.h, u.l);
    }
}

__global__ void ffbp_tables_kernel(TableConsts C, const PolarDesc* __restrict__ nodes, float4* __restrict__ tables) {
    table_entries(C, nodes[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x, tables);
}

// Leaf pulses relative to the leaf's phase centre O (origin formulation).
// A = -K (pos - O) is split into a multiple of a per-leaf power-of-two
// quantum with <= 10 significant bits plus an FP32 remainder.
struct PulseRec {
    float4 a;  // A_hi.x, A_hi.y, A_hi.z, frac(phase / 2pi)
    float4 b;  // A_lo.x, A_lo.y, A_lo.z, |pos - O|^2
    float4 c;  // (pos - O).x, .y, .z, weight
    float4 d;  // the leaf's A quantum (a power of two), its inverse, its largest |A| component and |A.x|
};

__device__ __forceinline__ void leaf_pulses(double K, const double* __restrict__ pos, const double* __restrict__ weight,
                                            const double* __restrict__ phase, const PolarDesc& g,
                                            PulseRec* __restrict__ recs, int amax[2]) {
    if (threadIdx.x < 2) amax[threadIdx.x] = 0;
    __syncthreads();
    float m = 0.0f, mx = 0.0f;
    for (int n = g.a + threadIdx.x; n < g.b; n += blockDim.x) {
        const double ax = pos[3 * n] - g.ox, ay = pos[3 * n + 1] - g.oy, az = pos[3 * n + 2] - g.oz;
        m = fmaxf(m, (float)(fabs(K) * fmax(fabs(ax), fmax(fabs(ay), fabs(az)))));
        mx = fmaxf(mx, (float)(fabs(K) * fabs(ax)));
    }
    atomicMax(amax, __float_as_int(m));  // non-negative floats order like their bit patterns
    atomicMax(amax + 1, __float_as_int(mx));
    __syncthreads();
    int e = 0;
    frexp((double)__int_as_float(amax[0]) * 1.0001 + 1e-30, &e);
    const double scale = ldexp(1.0, e - 10), inv_scale = ldexp(1.0, 10 - e);
    for (int n = g.a + threadIdx.x; n < g.b; n += blockDim.x) {
        const double ax = pos[3 * n] - g.ox, ay = pos[3 * n + 1] - g.oy, az = pos[3 * n + 2] - g.oz;
        PulseRec r;
        quantize(-K * ax, scale, inv_scale, r.a.x, r.b.x);
        quantize(-K * ay, scale, inv_scale, r.a.y, r.b.y);
        quantize(-K * az, scale, inv_scale, r.a.z, r.b.z);
        const double t = phase[n] * kInvTwoPi;
        r.a.w = (float)(t - rint(t));
        r.b.w = (float)(ax * ax + ay * ay + az * az);
        r.c = make_float4((float)ax, (float)ay, (float)az, (float)weight[n]);
        r.d = make_float4((float)scale, (float)inv_scale, __int_as_float(amax[0]), __int_as_float(amax[1]));
        recs[n] = r;
    }
}

__global__ void ffbp_leaf_pulses_kernel(double K, const double* __restrict__ pos, const double* __restrict__ weight,
                                        const double* __restrict__ phase, const PolarDesc* __restrict__ nodes,
                                        const int* __restrict__ leaves, PulseRec* __restrict__ recs) {
    __shared__ int amax[2];
    leaf_pulses(K, pos, weight, phase, nodes[leaves[blockIdx.x]], recs, amax);
}

// ---- FFBP: leaves (origin formulation) ---------------------------------------------------
//
// With O the leaf's phase centre and a = pos_n - O (|a| ~ the leaf aperture),
// a pixel at slant range r from O in unit direction e satisfies exactly
//   d = |r e - a| = r - L + eps,  L = e . a,  eps = (|a|^2 - L^2) / (2 (r - L) + eps),
// so the demodulated phase k (d - r) + phase_n is -K e . a + K eps + phase_n / 2pi
// (turns): no large term, no per-tile FP64.  On a polar grid e = (alpha s, alpha u, beta) with
// alpha = g / r and beta = -oz / r per row and s = side sqrt(1 - u^2), u per column, so
//   e . a = alpha C + beta a.z,       C = s a.x + u a.y,
//   -K e . a = alpha D + beta A.z,    D = s A.x + u A.y   (A = -K a),
// with C and D once per (pulse, tile column).  The phase's large part alpha_hi D_hi + beta_hi
// A_hi.z is exact in FP32: alpha_hi and beta_hi are multiples of 2^-11 (11 bits), D_hi and
// A_hi.z multiples of the leaf's A quantum below 2^10.5 quanta, so each product has at most 22
// bits and their sum 23.
//
// A thread's pixels are a run of eight columns of one tile row.  Along a run the range hardly
// changes (the angle step is chosen so that the phase turns by a fraction of a turn per column:
// millimetres), so everything but the rotation is worked out once per pulse for the run's middle,
// half-way between its fourth and fifth column, with the derivatives in the column offset
// m = -3.5 ... 3.5:
//   C(m) = C + C_1 m + ... + C_4 m^4 (s(u) expanded at the middle; D_j likewise, in radians),
//   d(m)^2 = r^2 + |a|^2 - 2 r (alpha C(m) + beta a.z),   so with t = r / d and z = 1 / (2 pi K d)
//   P_1 = t alpha D_1,  P_2 = t alpha D_2 - z P_1^2 / 2,  P_3 = t alpha D_3 - z P_1 P_2,
//   P_4 = t alpha D_4 - z (P_1 P_3 + P_2^2 / 2)            are the phase's coefficients (radians).
// The pulse's sample along the run is the window entry's cubic in d, a cubic in m as long as the
// whole run stays within one range bin; when that holds for all 32 rows of the warp the run takes
// one window entry (two 16-byte loads instead of sixteen) and the even and odd parts of both
// polynomials serve the columns +m and -m.  Otherwise each pixel takes its own entry.
// What bounds it: instruction issue (74% of the cycles; 295 instructions per warp and pulse, a quarter of
// them windows and records).  4096 pulses in 256 leaves of 16 (1.46 G pixel-pulses): 1.68 ms, with a pixel
// pair per thread and step 2.47; with every pixel on its own window entry 2.15.  Six blocks per SM (80
// registers): with five, seven and eight 1.70, 1.73 and 1.82 ms.
struct LeafRec {
    float4 p0;  // a.z, -|a|^2, A_hi.z, A_lo.z
    float4 p1;  // Phi, and as bits: window byte bias, byte offset of the window, of its last entry in it
};

// One pulse at the middle of one run of columns.
struct LeafCol {
    float4 p0;  // C, D_hi, D_lo, D
    float4 p1;  // 2 pi D_1 ... 2 pi D_4
};

// The middle of a run of columns: (s, u) as float pairs, s's derivatives s_j = s^(j)(u) du^j / j!.
struct LeafMid {
    float4 cv;
    float s1, s2, s3, s4;
    float du;
    float lim;  // half a bin, or below 0: the run's pixels take their own window entries
    int runs;   // the expansion holds for the leaf's pulses
    int first;  // floor(Q) of the tile's first row
};

constexpr int kLeafRun = kColRun;                             // columns per thread
constexpr int kLeafThreads = kSplitTilePixels / kLeafRun;
constexpr int kLeafGroups = kMaxCols / kLeafRun;              // runs per tile row, at most
constexpr int kLeafCtas = 6;                                  // per SM, by registers and by the window budget
constexpr int kLeafWindowBudget = 35 * 1024;
__host__ __device__ constexpr size_t leaf_col_offset() { return (size_t)kMaxLeafChunk * sizeof(LeafRec); }
__host__ __device__ constexpr size_t leaf_mid_offset() {
    return leaf_col_offset() + (size_t)kMaxLeafChunk * kLeafGroups * sizeof(LeafCol);
}
__host__ __device__ constexpr size_t leaf_window_offset() { return leaf_mid_offset() + kLeafGroups * sizeof(LeafMid); }

constexpr float kUnitQ = 1.0f / 2048.0f;  // quantum of unit-vector components (11 bits)

__device__ __forceinline__ void unit_split(float p, float e, float& h, float& l, float& full) {
    h = rintf(p * 2048.0f) * kUnitQ;
    l = (p - h) + e;
    full = p + e;
}

// The values of one pixel row i (tables: (g/r, -oz/r) as float pairs, (2r, frac(Q) - 1/2, floor(Q))).
struct LeafRow {
    float a, b;    // alpha, beta
    float ah, al;  // alpha = ah + al, ah a multiple of 2^-11
    float bh, bl;  // beta = bh + bl
    float r2, fm;  // 2 r, frac(Q) - 1/2 with Q = (r - range_start) / data_dr
    int o;         // floor(Q) - I_first
};

__device__ __forceinline__ LeafRow leaf_row(const PolarDesc& g, const float4* __restrict__ tables, int i, int I_first) {
    const float4 r1 = __ldg(tables + g.rows_off + 3 * (long long)i + 1);
    const float4 rq = __ldg(tables + g.rows_off + 3 * (long long)i + 2);
    LeafRow q;
    unit_split(r1.x, r1.y, q.ah, q.al, q.a);
    unit_split(r1.z, r1.w, q.bh, q.bl, q.b);
    q.r2 = rq.x;
    q.fm = rq.y;
    q.o = __float_as_int(rq.z) - I_first;
    return q;
}

// C and D of one (pulse, column) from the pulse record and the column's (c, u) pairs: D in
// two-float, split on the leaf's A quantum.
__device__ __forceinline__ float4 leaf_col(const PulseRec& pr, float4 cv, float side) {
    const float sh = side * cv.x, sl = side * cv.y, uh = cv.z, ul = cv.w;
    const float C = fmaf(sh, pr.c.x, uh * pr.c.y);
    const float p1 = sh * pr.a.x, e1 = fmaf(sh, pr.a.x, -p1);
    const float p2 = uh * pr.a.y, e2 = fmaf(uh, pr.a.y, -p2);
    const float S = p1 + p2, bb = S - p1;
    float rest = (p1 - (S - bb)) + (p2 - bb);
    rest += e1 + e2;
    rest = fmaf(sh, pr.b.x, rest);
    rest = fmaf(sl, pr.a.x, rest);
    rest = fmaf(uh, pr.b.y, rest);
    rest = fmaf(ul, pr.a.y, rest);
    const float Dh = rintf(S * pr.d.y) * pr.d.x;  // the A quantum is a power of two: exact
    const float Dl = (S - Dh) + rest;             // S - Dh is exact (|S - Dh| <= quantum / 2)
    return make_float4(C, Dh, Dl, S + rest);
}

// The run of columns from column j0 (window columns; the middle is j0 + 3.5), for pulses with
// largest |A| component amax and |A.x| axmax (turns) at ranges from r_min.
__device__ __forceinline__ LeafMid leaf_mid(const SplitParams& P, const PolarDesc& g, int j0, float r_min, float amax,
                                            float axmax) {
    const FF u = ff_add(ff_of(g.tf[5]), ff_mul(FF{(float)j0 + 0.5f * (kLeafRun - 1), 0.0f}, ff_of(g.tf[6])));
    const FF c = ff_sqrt0(ff_add(FF{1.0f, 0.0f}, ff_neg(ff_sqr(u))));
    const float h = g.tf[6].x + g.tf[6].y, uf = u.h, ic = 1.0f / c.h, hc = h * ic, u2 = uf * uf;
    LeafMid M;
    M.cv = make_float4(c.h, c.l, u.h, u.l);
    const float side = (float)g.side;
    // c = sqrt(1 - u^2): c' = -u / c, c'' = -1 / c^3, c''' = -3 u / c^5, c'''' = -3 (1 + 4 u^2) / c^7.
    M.s1 = side * -uf * hc;
    M.s2 = side * -0.5f * hc * hc * ic;
    M.s3 = M.s2 * uf * hc * ic;
    M.s4 = M.s2 * 0.25f * (1.0f + 4.0f * u2) * (hc * ic) * (hc * ic);
    M.du = h;
    // Orders five to seven go into the lower ones: over the run's four |m|, m^5 ~ 15.5 m^3 - 47.3125 m within 26.25,
    // m^6 ~ 16.396 m^4 - 55.051 m^2 within 52.25 and m^7 ~ 203.44 m^3 - 809.47 m within 544.7 (m^5 itself goes to 525).
    const float w = hc * ic, d4 = 1.0f / (1.0f + 4.0f * u2), s5 = M.s4 * uf * w * (3.0f + 4.0f * u2) * d4;
    const float s6 = M.s4 * w * w * 0.5f * (1.0f + 12.0f * u2 + 8.0f * u2 * u2) * d4;
    const float s7 = M.s4 * uf * w * w * w * 0.5f * (5.0f + 20.0f * u2 + 8.0f * u2 * u2) * d4;
    M.s1 += fmaf(-47.3125f, s5, -809.46875f * s7);
    M.s2 = fmaf(-55.050652f, s6, M.s2);
    M.s3 += fmaf(15.5f, s5, 203.4375f * s7);
    M.s4 = fmaf(16.395735f, s6, M.s4);
    // What that leaves, and the fifth order of the root.
    const float m = 0.5f * (kLeafRun - 1), m2 = m * m;
    const float ir = 1.0f / r_min, turn = m * hc * 1.5f * amax, y = turn * ir / fabsf(P.Kf);
    const float rest = axmax * (26.25f * fabsf(s5) + 52.25f * fabsf(s6) + 544.7f * fabsf(s7)) + turn * (y * y) * (y * y);
    M.runs = rest <= 5e-8f && fabsf(P.Kf) > 1e-3f ? 1 : 0;
    // The sample's cubic in m leaves out the square of the quadratic term.
    const float kb = fabsf(P.inv_drf / P.Kf);
    const float x1 = turn * kb, x2 = m2 * (axmax * fabsf(M.s2)) * kb + 0.5f * turn * y * kb;
    M.lim = (3.0f * x1 * x1 + x2) * x2 <= 1e-7f ? 0.5f : -1.0f;
    M.first = 0;
    return M;
}

// The pulses of a chunk on one run (or its part).
template <int PARTS>
__device__ __forceinline__ void leaf_runs(int part, const SplitParams& P, const LeafRec* __restrict__ rec,
                                          const LeafCol* __restrict__ cols, const char* __restrict__ win, int n,
                                          const LeafRow& q, float lim, float ar[kLeafRun / PARTS], float ai[kLeafRun / PARTS]) {
    const float inv_dr = P.inv_drf, Kf = P.Kf;
    const float kz = 1.0f / (kTwoPiF * Kf), kd = inv_dr * kz;
#pragma unroll 1
    for (int nl = 0; nl < n; ++nl) {
        const float4 ra = rec[nl].p0, rb = rec[nl].p1;
        const float4 ca = cols[nl * kLeafGroups].p0, cb = cols[nl * kLeafGroups].p1;
        const float L = fmaf(q.a, ca.x, q.b * ra.x);
        const float nq2 = fmaf(L, L, ra.y);                 // -(|a|^2 - L^2)
        const float B = rcp_approx(fmaf(-2.0f, L, q.r2));   // 1 / (2 (r - L))
        const float ne0 = nq2 * B;
        const float neps = fmaf(ne0 * ne0, B, ne0);
        const float dd = -L - neps;                          // d - r
        const float iR = rcp_approx(fmaf(0.5f, q.r2, dd));
        const float at = q.a * fmaf(-dd, iR, 1.0f);          // alpha r / d
        // Phase at the middle (turns): the exact part, then the small terms.
        const float tb = fmaf(q.ah, ca.y, q.bh * ra.z);
        float sm = fmaf(-Kf, neps, rb.x);
        sm = fmaf(q.ah, ca.z, sm);
        sm = fmaf(q.al, ca.w, sm);
        sm = fmaf(q.bh, ra.w, sm);
        sm = fmaf(q.bl, ra.z + ra.w, sm);
        const float P0 = ((tb - round_magic(tb)) + sm) * kTwoPiF;
        const float z = iR * kz;
        float P1, P2, P3, P4;
        run_phase(at, z, cb.x, cb.y, cb.z, cb.w, P1, P2, P3, P4);
        column_run<PARTS>(part, P0, P1, P2, P3, P4, fmaf(dd, inv_dr, q.fm), P1 * kd, P2 * kd, lim, win + __float_as_int(rb.z),
                   32u * (unsigned)q.o + (unsigned)__float_as_int(rb.y), (unsigned)__float_as_int(rb.w), ar, ai);
    }
}

// n pulses from c0 on the run's pixels one by one, with the taps from the pulse rows: pulses whose
// window does not fit (rare, hence out of line).
__device__ __noinline__ void leaf_direct(const SplitParams& P, const PolarDesc* __restrict__ node,
                                         const float4* __restrict__ tables, const PulseRec* __restrict__ precs, int i, int j0, int c0, int n,
                                         float2* __restrict__ more) {
    const PolarDesc& g = *node;
    const float side = (float)g.side;
    const LeafRow q = leaf_row(g, tables, i, 0);
#pragma unroll 1
    for (int k = 0; k < kLeafRun; ++k) {
        const float4 cv = __ldg(tables + g.cols_off + min(j0 + k, g.nu - 1));
        float sr = 0.0f, si = 0.0f;
#pragma unroll 1
        for (int nl = c0; nl < c0 + n; ++nl) {
            const PulseRec pr = precs[nl];
            const float4 cd = leaf_col(pr, cv, side);
            const float L = fmaf(q.a, cd.x, q.b * pr.c.z);
            const float nq2 = fmaf(L, L, -pr.b.w);
            const float B = rcp_approx(fmaf(-2.0f, L, q.r2));
            const float ne0 = nq2 * B;
            const float neps = fmaf(ne0 * ne0, B, ne0);
            const float qp = fmaf(-L - neps, P.inv_drf, q.fm);
            const float t = qp + kMagic, f = qp - (t - kMagic);
            const long long gb = (long long)(__float_as_int(t) - kMagicBits) + q.o;
            if (!(gb >= 1 && gb <= (long long)P.in.samples - 3)) continue;
            const float2* row = P.in.data + (size_t)nl * P.in.samples + gb - 1;
            float w[4], vr = 0.0f, vi = 0.0f;
            lagrange_centred(f, w);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const float2 x = __ldg(row + b);
                vr = fmaf(w[b], x.x, vr);
                vi = fmaf(w[b], x.y, vi);
            }
            vr *= pr.c.w;
            vi *= pr.c.w;
            const float tb = fmaf(q.ah, cd.y, q.bh * pr.a.z);
            float sm = fmaf(-P.Kf, neps, pr.a.w);
            sm = fmaf(q.ah, cd.z, sm);
            sm = fmaf(q.al, cd.w, sm);
            sm = fmaf(q.bh, pr.b.z, sm);
            sm = fmaf(q.bl, pr.a.z + pr.b.z, sm);
            float sn, cs;
            __sincosf(((tb - round_magic(tb)) + sm) * kTwoPiF, &sn, &cs);
            sr = fmaf(vr, cs, sr);
            sr = fmaf(-vi, sn, sr);
            si = fmaf(vr, sn, si);
            si = fmaf(vi, cs, si);
        }
        more[k] = make_float2(sr, si);
    }
}

// The n pulses of a chunk onto the run's pixels one by one, in tiles with a run whose expansion does not hold (coarse
// angle steps at squint): staged windows as in leaf_runs, C and D per column.  A warp's lanes form those of eight
// columns and some pulses at a time in its part of the columns' shared memory.  n = 0: pulse c0 alone, whose
// window does not fit (leaf_direct).  Out of line, two columns at a time, which leaves leaf_runs its registers (4096
// pulses in 256 leaves: with eight at a time the whole image takes 8.05 ms instead of 7.91).  1024 pulses in 64 leaves
// at 435 MHz and u = 0.5, whole image: 142 us, with the taps from the pulse rows (leaf_direct) 198, a pixel pair per thread,
// before there were runs, 131; 256 leaves of 4 at 9.6 GHz and u = 0.7: 430, 493 and 417.
template <int PARTS>
__device__ __noinline__ void leaf_pixels(const SplitParams& P, const PolarDesc* __restrict__ node,
                                         const float4* __restrict__ tables, const PulseRec* __restrict__ precs, int i, int j0,
                                         int c0, int n, float2* __restrict__ sum) {
    extern __shared__ __align__(16) char smem[];
    const LeafRec* rec = reinterpret_cast<const LeafRec*>(smem);
    float4* cols = reinterpret_cast<float4*>(smem + leaf_col_offset());
    const char* win = smem + leaf_window_offset();
    const int part = threadIdx.x / kLeafThreads;
    if (n == 0) {
        float2 all[kLeafRun];
        leaf_direct(P, node, tables, precs, i, j0, c0, 1, all);
#pragma unroll
        for (int k = 0; k < kLeafRun / PARTS; ++k) {
            const float2 v = all[PARTS == 1 ? k : run_column<PARTS>(part, k / 2, k % 2)];
            sum[k].x += v.x;
            sum[k].y += v.y;
        }
        return;
    }
    const int I_first = reinterpret_cast<const LeafMid*>(smem + leaf_mid_offset())->first;
    constexpr int kWarps = kLeafThreads * PARTS / 32, kPulses = kMaxLeafChunk * kLeafGroups * (int)sizeof(LeafCol) /
                                                                (kWarps * kLeafRun * (int)sizeof(float4));
    static_assert(kPulses * kLeafRun % 32 == 0, "whole warps of (pulse, column)");
    const PolarDesc& g = *node;
    const int lane = threadIdx.x & 31;
    float4* mine = cols + (threadIdx.x >> 5) * (kPulses * kLeafRun);
    const LeafRow q = leaf_row(g, tables, i, I_first);
    const float4 cv = __ldg(tables + g.cols_off + min(j0 + (lane & (kLeafRun - 1)), g.nu - 1));
    const float side = (float)g.side;
    for (int b = 0; b < n; b += kPulses) {
        __syncwarp();
#pragma unroll 1
        for (int e = lane; e < kPulses * kLeafRun; e += 32)
            if (b + e / kLeafRun < n) mine[e] = leaf_col(precs[c0 + b + e / kLeafRun], cv, side);
        __syncwarp();
#pragma unroll 1
        for (int k = 0; k < kLeafRun / PARTS; k += 2) {
            float ar[2], ai[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                ar[h] = sum[k + h].x;
                ai[h] = sum[k + h].y;
            }
#pragma unroll 1
            for (int nl = b; nl < min(b + kPulses, n); ++nl) {
                const float4 ra = rec[nl].p0, rb = rec[nl].p1;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 cd = mine[(nl - b) * kLeafRun + (PARTS == 1 ? k + h : run_column<PARTS>(part, (k + h) / 2, (k + h) % 2))];
                    const float L = fmaf(q.a, cd.x, q.b * ra.x);
                    const float nq2 = fmaf(L, L, ra.y);
                    const float B = rcp_approx(fmaf(-2.0f, L, q.r2));
                    const float ne0 = nq2 * B;
                    const float neps = fmaf(ne0 * ne0, B, ne0);
                    const float qp = fmaf(-L - neps, P.inv_drf, q.fm);
                    const float t = qp + kMagic, f = qp - (t - kMagic);
                    const float4* w = reinterpret_cast<const float4*>(
                        win + __float_as_int(rb.z) +
                        min(32u * (unsigned)(__float_as_int(t) + q.o) + (unsigned)__float_as_int(rb.y), (unsigned)__float_as_int(rb.w)));
                    const float4 c01 = w[0], c23 = w[1];
                    const float vr = fmaf(fmaf(fmaf(c23.z, f, c23.x), f, c01.z), f, c01.x);
                    const float vi = fmaf(fmaf(fmaf(c23.w, f, c23.y), f, c01.w), f, c01.y);
                    const float tb = fmaf(q.ah, cd.y, q.bh * ra.z);
                    float sm = fmaf(-P.Kf, neps, rb.x);
                    sm = fmaf(q.ah, cd.z, sm);
                    sm = fmaf(q.al, cd.w, sm);
                    sm = fmaf(q.bh, ra.w, sm);
                    sm = fmaf(q.bl, ra.z + ra.w, sm);
                    float sn, cs;
                    __sincosf(((tb - round_magic(tb)) + sm) * kTwoPiF, &sn, &cs);
                    ar[h] = fmaf(vr, cs, ar[h]);
                    ar[h] = fmaf(-vi, sn, ar[h]);
                    ai[h] = fmaf(vr, sn, ai[h]);
                    ai[h] = fmaf(vi, cs, ai[h]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) sum[k + h] = make_float2(ar[h], ai[h]);
        }
    }
}

// One leaf tile: the per-item body of the leaf kernels.  precs holds the pulse records of
// the leaf's scene (indexed by pulse); a node with a destination pointer writes there.  PARTS = 2: two threads
// per run, for launches of few tiles.
template <int PARTS>
__device__ __forceinline__ void leaf_tile(const SplitParams& P, const PolarDesc* __restrict__ nodes, const TileItem it,
                                          const float4* __restrict__ tables, const PulseRec* __restrict__ precs,
                                          float2* __restrict__ arena, float2* root_out, int root, char* smem,
                                          int* s_base, float* s_wt, int& s_nfit) {
    const PolarDesc g = nodes[it.node];
    const int lc = g.tile_lc, rows_t = kSplitTilePixels >> lc;  // 32 rows or more: a warp has one run of columns
    const int groups = (1 << lc) / kLeafRun;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kThr = kLeafThreads * PARTS;
    const int slot = tid & (kLeafThreads - 1), part = tid / kLeafThreads;
    const int row = slot & (rows_t - 1), group = slot / rows_t;
    const int ifirst = min(g.win_r0 + it.tile_r, g.nr - 1);
    const int ilast = min(g.win_r0 + it.tile_r + rows_t - 1, g.nr - 1);
    const float4 rfirst = __ldg(tables + g.rows_off + 3 * (long long)ifirst + 2);
    const int I_first = __float_as_int(rfirst.z);
    const int I_span = __float_as_int(__ldg(tables + g.rows_off + 3 * (long long)ilast + 2).z) - I_first;
    const float r_min = 0.5f * rfirst.x;
    const int ipix = min(g.win_r0 + it.tile_r + row, g.nr - 1);
    const int jpix = g.win_u0 + it.tile_u + kLeafRun * group;
    const LeafRow q = leaf_row(g, tables, ipix, I_first);
    float ar[kLeafRun / PARTS], ai[kLeafRun / PARTS];
#pragma unroll
    for (int k = 0; k < kLeafRun / PARTS; ++k) ar[k] = ai[k] = 0.0f;
    LeafRec* rec = reinterpret_cast<LeafRec*>(smem);
    LeafCol* cols = reinterpret_cast<LeafCol*>(smem + leaf_col_offset());
    LeafMid* mids = reinterpret_cast<LeafMid*>(smem + leaf_mid_offset());
    float4* win = reinterpret_cast<float4*>(smem + leaf_window_offset());
    const PulseInputs& in = P.in;
    const float side = (float)g.side;
    for (int c0 = g.a; c0 < g.b;) {
        const int want = min(P.chunk, g.b - c0);
        __syncthreads();  // the last chunk's windows are consumed (and a persistent block's last tile's middles)
        // The runs' middles, one per lane of the second warp, while the first makes the first chunk's records.
        if (c0 == g.a && warp == 1 && lane < groups) {
            const float4 pd = precs[g.a].d;
            const int j = it.tile_u + kLeafRun * lane;
            LeafMid M = leaf_mid(P, g, g.win_u0 + j, r_min, pd.z, pd.w);
            if (j >= g.win_nu) M.runs = 1;  // past the window: nothing to be exact about
            M.first = I_first;
            mids[lane] = M;
        }
        if (warp == 0) {
            int count = 0;
            if (lane < want) {
                const PulseRec pr = precs[c0 + lane];
                const float amag = sqrtf(pr.b.w);
                const float eps_max = pr.b.w / (2.0f * fmaxf(r_min - amag, 1.0f));
                const float hw = (amag + eps_max) * fabsf(P.inv_drf) + 1e-3f;
                const int bo = (int)floorf(-0.5f - hw), top = (int)ceilf(0.5f + hw);
                const long long cnt = (long long)I_span + top - bo + 1;
                count = hw < 1e6f && cnt <= P.cap ? (int)cnt : P.cap + 1;
                s_base[lane] = I_first + bo;
                s_wt[lane] = pr.c.w;
                LeafRec r;
                r.p0 = make_float4(pr.c.z, -pr.b.w, pr.a.z, pr.b.z);
                r.p1 = make_float4(pr.a.w, __int_as_float((int)(0u - 32u * (unsigned)(kMagicBits + bo))), 0.0f,
                                   __int_as_float(32 * (count - 1)));
                rec[lane] = r;
            }
            int inc = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            const unsigned fits = __ballot_sync(0xffffffffu, lane < want && inc <= P.cap);
            if (lane < want) rec[lane].p1.z = __int_as_float(32 * (inc - count));
            if (lane == 0) s_nfit = __popc(fits);
        }
        __syncthreads();
        const int nfit = s_nfit;
        const int chn = nfit > 0 ? nfit : 1;
        bool runs = true;  // all of the tile's
        for (int gi = 0; gi < groups; ++gi) runs = runs && mids[gi].runs != 0;
        for (int e = tid; e < nfit * groups && runs; e += kThr) {  // one (pulse, run of columns) each
            const int nl = e / groups, gi = e - nl * groups;
            const LeafMid& m = mids[gi];
            const PulseRec pr = precs[c0 + nl];
            const float Ax = (pr.a.x + pr.b.x) * kTwoPiF, Ay = (pr.a.y + pr.b.y) * kTwoPiF;
            LeafCol& o = cols[nl * kLeafGroups + gi];
            o.p0 = leaf_col(pr, m.cv, side);
            o.p1 = make_float4(fmaf(Ax, m.s1, Ay * m.du), Ax * m.s2, Ax * m.s3, Ax * m.s4);
        }
        for (int nl = warp; nl < nfit; nl += kThr / 32) {
            const float2* drow = in.data + (size_t)(c0 + nl) * in.samples;
            stage_window_shfl(drow, in.samples, s_base[nl], __float_as_int(rec[nl].p1.w) / 32 + 1, s_wt[nl],
                              win + __float_as_int(rec[nl].p1.z) / 16, lane);
        }
        __syncthreads();
        if (runs && nfit > 0) {
            leaf_runs<PARTS>(part, P, rec, cols + group, reinterpret_cast<const char*>(win), nfit, q, mids[group].lim, ar, ai);
        } else {
            float2 sum[kLeafRun / PARTS];
#pragma unroll
            for (int k = 0; k < kLeafRun / PARTS; ++k) sum[k] = make_float2(ar[k], ai[k]);
            leaf_pixels<PARTS>(P, nodes + it.node, tables, precs, ipix, jpix, c0, nfit, sum);
#pragma unroll
            for (int k = 0; k < kLeafRun / PARTS; ++k) {
                ar[k] = sum[k].x;
                ai[k] = sum[k].y;
            }
        }
        c0 += chn;
    }
    // Each warp holds 32 rows of eight columns: 64 bytes of a row per thread, as float4 where the
    // image's rows are 16-byte aligned.
    float2* dst = g.dst ? g.dst : (it.node == root ? root_out : arena + g.out_offset);
    const int wr = it.tile_r + row, wu = it.tile_u + kLeafRun * group;
    if (wr < g.win_nr && wu < g.win_nu) {
        float2* p = dst + (long long)wr * g.out_stride + wu;
        if (PARTS == 1 && wu + kLeafRun <= g.win_nu && (reinterpret_cast<unsigned long long>(p) & 15) == 0) {
#pragma unroll
            for (int k = 0; k < kLeafRun / PARTS; k += 2)
                reinterpret_cast<float4*>(p)[k / 2] = make_float4(ar[k], ai[k], ar[k + 1], ai[k + 1]);
        } else {
#pragma unroll
            for (int k = 0; k < kLeafRun / PARTS; ++k) {
                const int j = PARTS == 1 ? k : run_column<PARTS>(part, k / 2, k % 2);
                if (wu + j < g.win_nu) p[j] = make_float2(ar[k], ai[k]);
            }
        }
    }
}

template <int PARTS>
__global__ void __launch_bounds__(kLeafThreads * PARTS, PARTS == 1 ? kLeafCtas : 2) split_leaf_kernel(SplitParams P, const PolarDesc* __restrict__ nodes,
                                                                 const TileItem* __restrict__ items,
                                                                 const float4* __restrict__ tables,
                                                                 const PulseRec* __restrict__ precs,
                                                                 float2* __restrict__ arena, float2* root_out,
                                                                 int root) {
    extern __shared__ __align__(16) char smem[];
    __shared__ int s_base[kMaxLeafChunk];
    __shared__ float s_wt[kMaxLeafChunk];
    __shared__ int s_nfit;
    leaf_tile<PARTS>(P, nodes, items[blockIdx.x], tables, precs, arena, root_out, root, smem, s_base, s_wt, s_nfit);
}

// ---- FFBP: merges (both child regrids of one parent tile) --------------------------------
struct ChildRec {
    float4 a;  // W_hi.x, W_hi.y, W_lo.x, W_lo.y
    float4 b;  // u.x, u.y, 2 RR, frac(Qr) - 1/2
    float4 c;  // Phi, h.x, h.y, 2 G
    float4 d;  // G, frac(Qu) - 1/2
    float4 e;  // merge tiles: parent's origin - child's (x, y), r_c - RR
    float inv_sdr, inv_sdu;
    int ir0, iu0, snr, snu;
    const float2* img;
    int sstr;           // row stride of the child image (elements)
    int br0, bu0;       // staged footprint: first row and (even) first column in the child image
    int bh, bw;         // footprint rows and columns; bw == 0: not staged
    const void* tmap;   // TMA tensor map of the child image (staged footprints only)
};

// Record of a polar image c seen from the ground point (px, py, 0), in two-float FP32
// arithmetic from the node geometry split on the host (PolarDesc::tf): the FP32 quantities
// child_value needs for points near it (a parent tile, or a lattice tile).  K in turns/m.
__device__ __forceinline__ ChildRec child_rec_at(FF K, float scale_w, float inv_scale_w, const PolarDesc& c, FF px,
                                                 FF py, const float2* img) {
    const FF vx = ff_add(px, ff_neg(ff_of(c.tf[0])));
    const FF vy = ff_add(py, ff_neg(ff_of(c.tf[1])));
    const FF vz = ff_neg(ff_of(c.tf[2]));
    const FF g2 = ff_add(ff_sqr(vx), ff_sqr(vy));
    const FF G = ff_sqrt(g2);
    const FF RR = ff_sqrt(ff_add(g2, ff_sqr(vz)));
    const FF iR = ff_rcp(RR), iG = ff_rcp(G);
    const FF ux = ff_mul(vx, iR), uy = ff_mul(vy, iR);
    const FF hy = ff_mul(vy, iG);
    const FF t = ff_mul(K, RR);
    float phi = (t.h - rintf(t.h)) + t.l;
    phi -= rintf(phi);
    float fr, fu;
    const FF Qr = ff_mul(ff_add(RR, ff_neg(ff_of(c.tf[3]))), ff_of(c.tf[7]));
    const FF Qu = ff_mul(ff_add(hy, ff_neg(ff_of(c.tf[5]))), ff_of(c.tf[8]));
    const float ir = ff_floor_frac(Qr, fr), iu = ff_floor_frac(Qu, fu);
    const FF Wx = ff_mul(K, ux), Wy = ff_mul(K, uy);
    ChildRec R;
    R.a.x = rintf(Wx.h * inv_scale_w) * scale_w;  // scale_w is a power of two: exact
    R.a.z = (Wx.h - R.a.x) + Wx.l;
    R.a.y = rintf(Wy.h * inv_scale_w) * scale_w;
    R.a.w = (Wy.h - R.a.y) + Wy.l;
    const float Gf = G.h + G.l;
    R.b = make_float4(ux.h + ux.l, uy.h + uy.l, 2.0f * (RR.h + RR.l), fr);
    R.c = make_float4(phi, ff_mul(vx, iG).h, hy.h + hy.l, 2.0f * Gf);
    R.d = make_float4(Gf, fu, 0.0f, 0.0f);
    R.e = make_float4(RR.h, RR.l, 0.0f, 0.0f);
    R.inv_sdr = c.tf[7].x;
    R.inv_sdu = c.tf[8].x;
    const bool ok = fabsf(Qr.h) < 1.0e7f && fabsf(Qu.h) < 1.0e7f && G.h > 0.0f;  // false for NaN
    R.ir0 = ok ? (int)ir : -(1 << 30);
    R.iu0 = ok ? (int)iu : -(1 << 30);
    R.snr = c.nr;
    R.snu = c.nu;
    R.img = img;
    R.sstr = (int)c.out_stride;
    R.br0 = R.bu0 = R.bh = R.bw = 0;
    R.tmap = nullptr;
    return R;
}

// One thread per (merge tile, child).  The tile centre is the centre pixel's position from
// the node's row and column tables (two-float g and c, u), the same point setup_polar_tab
// measures the pixel offsets from.  With tensor maps (tmaps != NULL) a child whose node has a
// footprint box gets the box's origin in its image: box_r rows and box_u columns (rounded down
// to an even column, the TMA's 16-byte rule for 8-byte elements) before the centre's bin.
__device__ __forceinline__ void child_record(FF K, float scale_w, float inv_scale_w,
                                             const PolarDesc* __restrict__ nodes, const float4* __restrict__ tables,
                                             const TileItem it, int t, float2* __restrict__ arena,
                                             const void* tmaps, ChildRec* __restrict__ out) {
    const PolarDesc& g = nodes[it.node];
    const int ci = (t & 1) ? g.right : g.left;
    const PolarDesc& c = nodes[ci];
    const int cols_t = 1 << g.tile_lc, rows_t = kSplitTilePixels >> g.tile_lc;
    const int i0 = min(g.win_r0 + it.tile_r + (rows_t >> 1), g.nr - 1);
    const int j0 = min(g.win_u0 + it.tile_u + (cols_t >> 1), g.nu - 1);
    const float4 rv = __ldg(tables + g.rows_off + 3 * (long long)i0);
    const float4 cv = __ldg(tables + g.cols_off + j0);
    const FF g0{rv.x, rv.y};
    const FF gc = ff_mul(g0, FF{cv.x, cv.y});
    const FF px = ff_add(ff_of(g.tf[0]), g.side < 0 ? ff_neg(gc) : gc);
    const FF py = ff_add(ff_of(g.tf[1]), ff_mul(g0, FF{cv.z, cv.w}));
    ChildRec R = child_rec_at(K, scale_w, inv_scale_w, c, px, py, arena + c.out_offset);
    if (!(t & 1)) tab_quantum(g, g.tile_lc, it.tile_r, it.tile_u, tables, R.d.z, R.d.w);
    const FF r = ff_add(ff_of(g.tf[3]), ff_mul(FF{(float)i0, 0.0f}, ff_of(g.tf[4])));
    const FF off = ff_add(r, FF{-R.e.x, -R.e.y});
    const FF dx = ff_add(ff_of(g.tf[0]), ff_neg(ff_of(c.tf[0]))), dy = ff_add(ff_of(g.tf[1]), ff_neg(ff_of(c.tf[1])));
    R.e = make_float4(dx.h + dx.l, dy.h + dy.l, off.h + off.l, 0.0f);
    if (tmaps != nullptr && c.box_w > 0 && R.ir0 > -(1 << 30)) {
        R.br0 = R.ir0 - c.box_r;
        R.bu0 = (R.iu0 - c.box_u) & ~1;
        R.bh = c.box_h;
        R.bw = c.box_w;
        R.tmap = static_cast<const char*>(tmaps) + kTensorMapBytes * (size_t)ci;
    }
    out[t] = R;
}

__global__ void ffbp_child_records_kernel(float Kh, float Kl, float scale_w, float inv_scale_w,
                                          const PolarDesc* __restrict__ nodes, const float4* __restrict__ tables,
                                          const TileItem* __restrict__ items, int n_items,
                                          float2* __restrict__ arena, const void* tmaps, ChildRec* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * n_items) return;
    child_record(FF{Kh, Kl}, scale_w, inv_scale_w, nodes, tables, items[t >> 1], t, arena, tmaps, out);
}

// Child-image coordinates of a parent pixel: bin indices (ir, iu), centred fractions
// (sr, su) and the second-order range term eps.  ok: the 4x4 stencil lies inside the child.
struct ChildCoord {
    int ir, iu;
    float sr, su, eps;
    bool ok;
};

__device__ __forceinline__ ChildCoord child_coords(const ChildRec& R, const Pix& q) {
    ChildCoord c;
    const float L = fmaf(R.b.x, q.dx, R.b.y * q.dy);
    const float q2 = fmaf(-L, L, q.d2);
    const float B = rcp_approx(fmaf(2.0f, L, R.b.z));
    const float e0 = q2 * B;
    c.eps = fmaf(-e0 * e0, B, e0);
    const float qr = fmaf(L + c.eps, R.inv_sdr, R.b.w);
    const float tr = qr + kMagic;
    c.sr = qr - (tr - kMagic);
    c.ir = R.ir0 + (__float_as_int(tr) - kMagicBits);
    const float Lh = fmaf(R.c.y, q.dx, R.c.z * q.dy);
    const float q2h = fmaf(-Lh, Lh, q.d2);
    const float Bh = rcp_approx(fmaf(2.0f, Lh, R.c.w));
    const float eh = q2h * Bh;
    const float dG = Lh + fmaf(-eh * eh, Bh, eh);
    const float gp = R.d.x + dG;
    const float duu = fmaf(-R.c.z, dG, q.dy) * rcp_approx(gp);
    const float qu = fmaf(duu, R.inv_sdu, R.d.y);
    const float tu = qu + kMagic;
    c.su = qu - (tu - kMagic);
    c.iu = R.iu0 + (__float_as_int(tu) - kMagicBits);
    c.ok = c.ir >= 1 && c.ir <= R.snr - 3 && c.iu >= 1 && c.iu <= R.snu - 3 && gp > 0.0f;
    return c;
}

__device__ __forceinline__ float2 child_value(float Kf, const ChildRec& R, const Pix& q) {
    const ChildCoord c = child_coords(R, q);
    float vr = 0.0f, vi = 0.0f;
    if (c.ok) {
        float wr[4], wu[4];
        lagrange_centred(c.sr, wr);
        lagrange_centred(c.su, wu);
        const float2* base = R.img + (size_t)(c.ir - 1) * R.sstr + (c.iu - 1);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const float2* row = base + (size_t)a * R.sstr;
            const float2 x0 = __ldg(row), x1 = __ldg(row + 1), x2 = __ldg(row + 2), x3 = __ldg(row + 3);
            float rr = wu[0] * x0.x, ri = wu[0] * x0.y;
            rr = fmaf(wu[1], x1.x, rr);
            ri = fmaf(wu[1], x1.y, ri);
            rr = fmaf(wu[2], x2.x, rr);
            ri = fmaf(wu[2], x2.y, ri);
            rr = fmaf(wu[3], x3.x, rr);
            ri = fmaf(wu[3], x3.y, ri);
            vr = fmaf(wr[a], rr, vr);
            vi = fmaf(wr[a], ri, vi);
        }
    }
    const float tb = fmaf(R.a.x, q.dxh, R.a.y * q.dyh);
    float sm = fmaf(Kf, c.eps, R.c.x);
    sm = fmaf(R.a.x, q.dxl, sm);
    sm = fmaf(R.a.y, q.dyl, sm);
    sm = fmaf(R.a.z, q.dx, sm);
    sm = fmaf(R.a.w, q.dy, sm);
    const float tot = (tb - round_magic(tb)) + (sm + q.psi);
    const float ang = (tot - round_magic(tot)) * kTwoPiF;
    float sn, cs;
    __sincosf(ang, &sn, &cs);
    return make_float2(vr * cs - vi * sn, vr * sn + vi * cs);
}

// Child records of a merge tile for the packed merge: every field of one child as a duplicated
// (x, x) pair, so that a chain over two parent pixels (the two lanes of f32x2 operations) takes
// each operand with one 8-byte shared load.  Negated copies stand in for the scalar code's
// subtractions (negation is exact), so every lane equals child_value's arithmetic bit for bit.
struct __align__(16) ChildDup {
    float2 nbx, nby;   // -u.x, -u.y
    float2 bz, bw;     // 2 RR, frac(Qr) - 1/2
    float2 ncy, ncz;   // -h.x, -h.y
    float2 cz, cw;     // h.y, 2 G
    float2 dx, dy;     // G, frac(Qu) - 1/2
    float2 nisr, isu;  // -1/sdr, 1/sdu
    float2 ax, ay;     // W_hi.x, W_hi.y
    float2 az, aw;     // W_lo.x, W_lo.y
    float2 cx;         // Phi
    int ir0, iu0, snr, snu;
    const float2* img;
    int sstr;          // row stride of the child image
    int xr0, xu0, xh, xw;  // staged footprint: first row, first column, rows, columns (xw == 0: not staged)
};

__device__ __forceinline__ void child_dup_store(const ChildRec& R, ChildDup& P) {
    P.nbx = pair(-R.b.x);
    P.nby = pair(-R.b.y);
    P.bz = pair(R.b.z);
    P.bw = pair(R.b.w);
    P.ncy = pair(-R.c.y);
    P.ncz = pair(-R.c.z);
    P.cz = pair(R.c.z);
    P.cw = pair(R.c.w);
    P.dx = pair(R.d.x);
    P.dy = pair(R.d.y);
    P.nisr = pair(-R.inv_sdr);
    P.isu = pair(R.inv_sdu);
    P.ax = pair(R.a.x);
    P.ay = pair(R.a.y);
    P.az = pair(R.a.z);
    P.aw = pair(R.a.w);
    P.cx = pair(R.c.x);
    P.ir0 = R.ir0;
    P.iu0 = R.iu0;
    P.snr = R.snr;
    P.snu = R.snu;
    P.img = R.img;
    P.sstr = R.sstr;
    P.xr0 = R.br0;
    P.xu0 = R.bu0;
    P.xh = R.bh;
    P.xw = R.bw;
}

// Offsets of the parent pixels (row, col) and (row + 1, col) from the tile centre as (upper,
// lower) lane pairs, row even: tab_pixel's arithmetic lane by lane, with d2 negated (exact).
struct VPix {
    float2 dx, dy, dxh, dyh, dxl, dyl, nd2, psi;
};

__device__ __forceinline__ float2 ld_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }

__device__ __forceinline__ VPix tab_vpair(const TabF& T, int row, int col) {
    VPix v;
    v.dxh = __fadd2_rn(ld_pair(T.rxh + row), pair(T.cxh[col]));  // exact: both multiples of the quantum
    v.dyh = __fadd2_rn(ld_pair(T.ryh + row), pair(T.cyh[col]));
    const float2 dg = ld_pair(T.dg + row);
    v.dxl = __ffma2_rn(dg, pair(T.dcs[col]), __fadd2_rn(ld_pair(T.rxl + row), pair(T.cxl[col])));
    v.dyl = __ffma2_rn(dg, pair(T.duu[col]), __fadd2_rn(ld_pair(T.ryl + row), pair(T.cyl[col])));
    v.dx = __fadd2_rn(v.dxh, v.dxl);
    v.dy = __fadd2_rn(v.dyh, v.dyl);
    v.nd2 = __fmul2_rn(__ffma2_rn(v.dx, v.dx, __fmul2_rn(v.dy, v.dy)), pair(-1.0f));
    v.psi = ld_pair(T.psi + row);
    return v;
}

// lagrange_centred for two fractions at once (the lanes of f32x2 operations), per lane the same
// operations and roundings: -a/6, -c2 and -s are the scalar code's a/6, c2 and s negated (exact).
__device__ __forceinline__ void lagrange_centred2(float2 s, float2 w[4]) {
    const float2 a = __ffma2_rn(s, s, pair(-0.25f));
    const float2 na6 = __fmul2_rn(a, pair(-1.0f / 6.0f));
    const float2 b2 = __ffma2_rn(a, pair(0.5f), pair(-1.0f));
    const float2 c1 = __fmul2_rn(pair(-1.5f), na6);
    const float2 nc2 = __fmul2_rn(pair(-0.5f), b2);
    const float2 ns = __fmul2_rn(s, pair(-1.0f));
    w[0] = __ffma2_rn(na6, s, c1);
    w[3] = __ffma2_rn(na6, ns, c1);
    w[1] = __ffma2_rn(b2, s, nc2);
    w[2] = __ffma2_rn(b2, ns, nc2);
}

// Where a stencil's taps come from: the child image through the read-only path (kLdg), the
// child image with weak coherent loads (kCoherent: the merge queue, whose child images were
// written by other CTAs of the same launch; L1-cached, ordered by the acquire that made the
// node ready), or the tile's staged footprint in shared memory (kShared).
enum TapSource { kLdg = 0, kCoherent = 1, kShared = 2 };

// The coherent asm has no memory clobber, so the compiler schedules it as freely as __ldg; its
// address comes from values read after the CTA barrier that follows the acquire.
template <int SRC>
__device__ __forceinline__ void ld_child_row(const float2* p, float2& x0, float2& x1, float2& x2, float2& x3) {
    if (SRC == kCoherent) {
        asm("ld.global.v2.f32 {%0, %1}, [%8];\n\t"
            "ld.global.v2.f32 {%2, %3}, [%8+8];\n\t"
            "ld.global.v2.f32 {%4, %5}, [%8+16];\n\t"
            "ld.global.v2.f32 {%6, %7}, [%8+24];"
            : "=f"(x0.x), "=f"(x0.y), "=f"(x1.x), "=f"(x1.y), "=f"(x2.x), "=f"(x2.y), "=f"(x3.x), "=f"(x3.y)
            : "l"(p));
    } else if (SRC == kShared) {
        x0 = p[0];
        x1 = p[1];
        x2 = p[2];
        x3 = p[3];
    } else {
        x0 = __ldg(p);
        x1 = __ldg(p + 1);
        x2 = __ldg(p + 2);
        x3 = __ldg(p + 3);
    }
}

// 4x4 Lagrange stencil whose first tap is base (rows `stride` elements apart) with weights wr
// (range) and wu (angle); (re, im) run as one f32x2 pair.
template <int SRC>
__device__ __forceinline__ float2 child_stencil(const float2* base, int stride, const float wr[4], const float wu[4]) {
    float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        float2 x0, x1, x2, x3;
        ld_child_row<SRC>(base + (size_t)a * stride, x0, x1, x2, x3);
        float2 r = __fmul2_rn(pair(wu[0]), x0);
        r = __ffma2_rn(pair(wu[1]), x1, r);
        r = __ffma2_rn(pair(wu[2]), x2, r);
        r = __ffma2_rn(pair(wu[3]), x3, r);
        v = __ffma2_rn(pair(wr[a]), r, v);
    }
    return v;
}

// The two stencils of a vertical pair that share three rows: one 5x4 block from row (base),
// the upper pixel's stencil in rows 0-3, the lower one's in rows 1-4 (the same sums as
// child_stencil per pixel).
template <int SRC>
__device__ __forceinline__ void child_pair_block(const float2* base, int stride, const float wrA[4],
                                                 const float wuA[4], const float wrB[4], const float wuB[4],
                                                 float2& vA, float2& vB) {
#pragma unroll
    for (int a = 0; a < 5; ++a) {
        float2 x0, x1, x2, x3;
        ld_child_row<SRC>(base + (size_t)a * stride, x0, x1, x2, x3);
        if (a < 4) {
            float2 r = __fmul2_rn(pair(wuA[0]), x0);
            r = __ffma2_rn(pair(wuA[1]), x1, r);
            r = __ffma2_rn(pair(wuA[2]), x2, r);
            r = __ffma2_rn(pair(wuA[3]), x3, r);
            vA = __ffma2_rn(pair(wrA[a]), r, vA);
        }
        if (a > 0) {
            float2 r = __fmul2_rn(pair(wuB[0]), x0);
            r = __ffma2_rn(pair(wuB[1]), x1, r);
            r = __ffma2_rn(pair(wuB[2]), x2, r);
            r = __ffma2_rn(pair(wuB[3]), x3, r);
            vB = __ffma2_rn(pair(wrB[a - 1]), r, vB);
        }
    }
}

// Child C at the column pair q (lanes: the upper and the lower parent pixel), rotated: per lane
// child_value's arithmetic (the Lagrange weights, the stencil's sum order and the rotation are
// the same).  Two vertically adjacent parent pixels nearly always fall one child range bin apart
// in the same angle column (a parent range step is one child range step, shortened by the
// cosine of the angle between the two phase centres' lines of sight), so their 4x4 stencils
// share three rows: when that holds for every lane of the warp, the pair gathers one 5x4 block
// (20 loads instead of 32).  Otherwise each pixel gathers its own stencil.
// sbox (STAGED, not NULL): the child's footprint staged in shared memory (C.xh x C.xw elements
// from row C.xr0, column C.xu0); a warp whose pairs all share a block inside it reads the blocks
// from shared memory, any other warp gathers each pixel's stencil from the child image (staged
// kernels have no other paths: fewer code paths keep their loop in the instruction cache).  The
// taps are the same values either way.
template <bool COHERENT, bool STAGED>
__device__ __forceinline__ void child_vpair(float Kf, const ChildDup& C, const VPix& q, float2& oA, float2& oB,
                                            const float2* sbox) {
    constexpr int SRC = COHERENT ? kCoherent : kLdg;
    const float2 magic = pair(kMagic), nmagic = pair(-kMagic), mone = pair(-1.0f);
    const float2 nL = __ffma2_rn(C.nbx, q.dx, __fmul2_rn(C.nby, q.dy));
    const float2 nq2 = __ffma2_rn(nL, nL, q.nd2);
    const float2 den = __ffma2_rn(pair(-2.0f), nL, C.bz);
    const float2 B = make_float2(rcp_approx(den.x), rcp_approx(den.y));
    const float2 ne0 = __fmul2_rn(nq2, B);
    const float2 neps = __ffma2_rn(__fmul2_rn(ne0, ne0), B, ne0);
    const float2 tb = __ffma2_rn(C.ax, q.dxh, __fmul2_rn(C.ay, q.dyh));
    float2 sm = __ffma2_rn(pair(-Kf), neps, C.cx);
    sm = __ffma2_rn(C.ax, q.dxl, sm);
    sm = __ffma2_rn(C.ay, q.dyl, sm);
    sm = __ffma2_rn(C.az, q.dx, sm);
    sm = __ffma2_rn(C.aw, q.dy, sm);
    const float2 rtb = __fadd2_rn(__fadd2_rn(tb, magic), nmagic);
    const float2 tot = __fadd2_rn(__ffma2_rn(rtb, mone, tb), __fadd2_rn(sm, q.psi));
    const float2 rtot = __fadd2_rn(__fadd2_rn(tot, magic), nmagic);
    const float2 ang = __fmul2_rn(__ffma2_rn(rtot, mone, tot), pair(kTwoPiF));
    float snA, csA, snB, csB;
    __sincosf(ang.x, &snA, &csA);
    __sincosf(ang.y, &snB, &csB);
    const float2 qr = __ffma2_rn(__fadd2_rn(nL, neps), C.nisr, C.bw);
    const float2 tr = __fadd2_rn(qr, magic);
    const float2 sr = __ffma2_rn(__fadd2_rn(tr, nmagic), mone, qr);
    const float2 nLh = __ffma2_rn(C.ncy, q.dx, __fmul2_rn(C.ncz, q.dy));
    const float2 nq2h = __ffma2_rn(nLh, nLh, q.nd2);
    const float2 denh = __ffma2_rn(pair(-2.0f), nLh, C.cw);
    const float2 Bh = make_float2(rcp_approx(denh.x), rcp_approx(denh.y));
    const float2 neh = __fmul2_rn(nq2h, Bh);
    const float2 ndG = __fadd2_rn(nLh, __ffma2_rn(__fmul2_rn(neh, neh), Bh, neh));
    const float2 gp = __ffma2_rn(ndG, mone, C.dx);
    const float2 num = __ffma2_rn(C.cz, ndG, q.dy);
    const float2 duu = __fmul2_rn(num, make_float2(rcp_approx(gp.x), rcp_approx(gp.y)));
    const float2 qu = __ffma2_rn(duu, C.isu, C.dy);
    const float2 tu = __fadd2_rn(qu, magic);
    const float2 su = __ffma2_rn(__fadd2_rn(tu, nmagic), mone, qu);
    const int irA = C.ir0 + (__float_as_int(tr.x) - kMagicBits), irB = C.ir0 + (__float_as_int(tr.y) - kMagicBits);
    const int iuA = C.iu0 + (__float_as_int(tu.x) - kMagicBits), iuB = C.iu0 + (__float_as_int(tu.y) - kMagicBits);
    const bool okA = irA >= 1 && irA <= C.snr - 3 && iuA >= 1 && iuA <= C.snu - 3 && gp.x > 0.0f;
    const bool okB = irB >= 1 && irB <= C.snr - 3 && iuB >= 1 && iuB <= C.snu - 3 && gp.y > 0.0f;
    const bool share = okA && okB && irB == irA + 1 && iuB == iuA;
    float2 vA = make_float2(0.0f, 0.0f), vB = vA;
    // The pair's block origin relative to the staged footprint (at least 8 x 8 elements when staged).
    const int rA = irA - 1 - C.xr0, uA = iuA - 1 - C.xu0;
    if (STAGED && sbox != nullptr && __all_sync(0xffffffffu, share && (unsigned)rA <= (unsigned)(C.xh - 5) &&
                                              (unsigned)uA <= (unsigned)(C.xw - 4))) {
        float wrA[4], wuA[4], wrB[4], wuB[4];
        float2 wr2[4], wu2[4];
        lagrange_centred2(sr, wr2);  // both pixels' weights as lane pairs
        lagrange_centred2(su, wu2);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            wrA[k] = wr2[k].x;
            wrB[k] = wr2[k].y;
            wuA[k] = wu2[k].x;
            wuB[k] = wu2[k].y;
        }
        child_pair_block<kShared>(sbox + rA * C.xw + uA, C.xw, wrA, wuA, wrB, wuB, vA, vB);
    } else if (!STAGED && __all_sync(0xffffffffu, share)) {
        float wrA[4], wuA[4], wrB[4], wuB[4];
        lagrange_centred(sr.x, wrA);
        lagrange_centred(su.x, wuA);
        lagrange_centred(sr.y, wrB);
        lagrange_centred(su.y, wuB);
        child_pair_block<SRC>(C.img + (size_t)(irA - 1) * C.sstr + (iuA - 1), C.sstr, wrA, wuA, wrB, wuB, vA, vB);
    } else {
        if (okA) {
            float wr[4], wu[4];
            lagrange_centred(sr.x, wr);
            lagrange_centred(su.x, wu);
            vA = child_stencil<SRC>(C.img + (size_t)(irA - 1) * C.sstr + (iuA - 1), C.sstr, wr, wu);
        }
        if (okB) {
            float wr[4], wu[4];
            lagrange_centred(sr.y, wr);
            lagrange_centred(su.y, wu);
            vB = child_stencil<SRC>(C.img + (size_t)(irB - 1) * C.sstr + (iuB - 1), C.sstr, wr, wu);
        }
    }
    // (vr cs - vi sn, vr sn + vi cs)
    oA = __ffma2_rn(pair(vA.x), make_float2(csA, snA), __fmul2_rn(pair(vA.y), make_float2(-snA, csA)));
    oB = __ffma2_rn(pair(vB.x), make_float2(csB, snB), __fmul2_rn(pair(vB.y), make_float2(-snB, csB)));
}

// ---- merge tiles in runs of rows --------------------------------------------------------------
//
// A thread forms a run of eight parent rows in one column.  Along a run the child's range and angle and
// the demodulated phase K (d - r) are smooth, so they are worked out once per (run, child) at the
// run's middle (half-way between its fourth and fifth row, m = 0), in the split arithmetic that child_value uses per
// pixel, and expanded in the row offset m = -3.5 ... 3.5.  With the parent's ground direction e = (side c, u),
// its ground range g(m) (g^2 = r^2 - z^2, r = r_0 + m h), q = e . (O - C) the offset of its origin from the
// child's along e, and d the child's range (d^2 = r^2 + 2 q g + const):
//   D_1 = d_1 - h = (h (r - d) + q g_1) / d          (no cancellation of the row step)
//   d_2 = (2 q g_2 - D_1 (2 h + D_1)) / 2 d,  d_3 = (q g_3 - d_1 d_2) / d
// and with G the child's ground range, cos = (g + q) / G, a = e_y - u' cos, n_j = g_j / G the child's angle is
//   u'_1 = a n_1,  u'_2 = a n_2 - (a cos + u' sin^2 / 2) n_1^2,  u'_3 = a n_3 + ...
// (the Legendre expansion of 1 / G(m)).  g_j per row: h r / g, -h^2 z^2 / 2 g^3, h^3 z^2 r / 2 g^5.
// The third orders go into the slopes with 9.25, the linear fit of m^3 over the run.
// split_merge_run_limit says for which nodes all this holds; the others go pair by pair (child_vpair).
// What bounds it: instruction issue (211 instructions per warp, pair of rows and child; 280 pair by pair).  4096
// pulses, levels of 81 to 82 thousand tiles: 0.67 ms each, pair by pair 0.83; six blocks per SM (80 registers),
// with seven and eight the whole image takes 0.08 and 0.06 ms more.
struct MergeRow {
    float4 o;  // R_hi.x, R_hi.y, R_lo.x, R_lo.y: (g - g_c) (side c, u) at the tile centre's column
    float4 p;  // g - g_c, psi = -K r modulo a turn, r - r_c, g
    float4 w;  // g_1, g_2, g_3, -
};
struct MergeCol {
    float4 o;  // C_hi.x, C_hi.y, C_lo.x, C_lo.y: g_c (side (c - c_c), u - u_c)
    float4 p;  // side (c - c_c), u - u_c, side c, u
};

struct MergeTab {
    MergeRow row[kMergeRows];
    MergeCol col[kMaxCols];
};

// A tile's child: its record, and the bins (relative to the record's) at which a pixel's stencil lies
// inside the child image and, when staged, inside the staged footprint.
struct __align__(16) MergeChild {
    ChildRec r;
    float2 bins;  // child range bins per turn of phase, as a float pair
    int box;      // staged: the footprint's offset in shared memory (elements)
    float lo_r, hi_r, lo_u, hi_u;
};

__device__ __forceinline__ void merge_child(FF K, const PolarDesc& c, const ChildRec& r, int box, MergeChild& C) {
    int r0 = 1, r1 = r.snr - 3, u0 = 1, u1 = r.snu - 3;
    if (r.bw > 0) {
        r0 = max(r0, r.br0 + 1);
        r1 = min(r1, r.br0 + r.bh - 3);
        u0 = max(u0, r.bu0 + 1);
        u1 = min(u1, r.bu0 + r.bw - 3);
    }
    C.r = r;
    const FF b = ff_mul(ff_of(c.tf[7]), ff_rcp(K));
    C.bins = make_float2(b.h, b.l);
    C.box = box;
    const bool ok = r.ir0 > -(1 << 30);
    C.lo_r = ok ? (float)(r0 - r.ir0) : 1.0f;
    C.hi_r = ok ? (float)(r1 - r.ir0) : -1.0f;
    C.lo_u = ok ? (float)(u0 - r.iu0) : 1.0f;
    C.hi_u = ok ? (float)(u1 - r.iu0) : -1.0f;
}

// Row `row` (a whole number, or half-way between two) of node g, `off` rows from the tile's centre row.
__device__ __forceinline__ MergeRow merge_row(FF K, const PolarDesc& g, float4 r0v, float4 c0v, float row, float off,
                                              float q, float iq) {
    const float side = (float)g.side;
    const FF r = ff_add(ff_of(g.tf[3]), ff_mul(FF{row, 0.0f}, ff_of(g.tf[4])));
    const FF z = ff_of(g.tf[2]);
    const FF gg = ff_sqrt0(ff_add(ff_sqr(r), ff_neg(ff_sqr(z))));
    const FF ph = ff_mul(ff_neg(K), r);
    float psi = (ph.h - rintf(ph.h)) + ph.l;
    psi -= rintf(psi);
    const float dh = gg.h - r0v.x, dl = gg.l - r0v.y;  // nearby values: dh is exact
    MergeRow R;
    float p, e;
    two_prod(dh, dl, c0v.x, c0v.y, p, e);
    R.o.x = side * p;
    R.o.z = side * e;
    two_prod(dh, dl, c0v.z, c0v.w, p, e);
    R.o.y = p;
    R.o.w = e;
    quantize_pair(R.o.x, R.o.z, q, iq);
    quantize_pair(R.o.y, R.o.w, q, iq);
    const float h = g.tf[4].x, gf = gg.h, ig = 1.0f / gf, zh = z.h * h * ig;
    R.p = make_float4(dh + dl, psi, off * h, gf);
    R.w.x = h * r.h * ig;
    R.w.y = -0.5f * zh * zh * ig;
    R.w.z = -R.w.y * R.w.x * ig;
    R.w.w = 0.0f;
    return R;
}

// The tables of a merge tile: its runs' middles and its columns, in FP32 two-float arithmetic from the node's
// geometry and column table, with the offsets quantized on the tile's quantum (q, iq).
template <int THREADS>
__device__ __forceinline__ void setup_merge(FF K, const Job& J, MergeTab& T, const float4* __restrict__ tables, float q,
                                            float iq) {
    const PolarDesc& g = J.g;
    const int tid = threadIdx.x;
    const int cols_t = 1 << J.lc, rows_t = kSplitTilePixels >> J.lc;
    float4 r0v, c0v;
    int j0;
    tab_centre(g, J.lc, J.tile_r, J.tile_u, tables, r0v, c0v, j0);
    const float side = (float)g.side;
    static_assert(kMergeRows + kMaxCols <= THREADS, "one run's middle or column per thread");
    if (tid < rows_t / kMergeRun) {
        const int i0 = min(g.win_r0 + J.tile_r + (rows_t >> 1), g.nr - 1), i = g.win_r0 + J.tile_r + kMergeRun * tid;
        T.row[tid] = merge_row(K, g, r0v, c0v, (float)i + 0.5f * (kMergeRun - 1),
                               (float)(i - i0) + 0.5f * (kMergeRun - 1), q, iq);
    }
    const int c = tid - kMergeRows;
    if (c >= 0 && c < cols_t) {
        const int j = min(g.win_u0 + J.tile_u + c, g.nu - 1);
        TabCol C = tab_col(g, tables, r0v, c0v, j, j0);
        quantize_pair(C.cxh, C.cxl, q, iq);
        quantize_pair(C.cyh, C.cyl, q, iq);
        const float4 cv = __ldg(tables + g.cols_off + j);
        T.col[c].o = make_float4(C.cxh, C.cyh, C.cxl, C.cyl);
        T.col[c].p = make_float4(C.dcs, C.duu, side * (cv.x + cv.y), cv.z + cv.w);
    }
    __syncthreads();
}

// The middle of a run: its offset from the tile centre and its row's and column's values.
struct MergeRun {
    Pix x;  // dx, dy, their parts, d2, psi
    float rho, g, g1, g2, g3, ex, ey;
};

__device__ __forceinline__ MergeRun merge_run(const MergeRow& R, const MergeCol& C) {
    const float4 ro = R.o, rp = R.p, rw = R.w, co = C.o, cp = C.p;
    MergeRun m;
    m.x.dxh = ro.x + co.x;  // exact: both multiples of the quantum
    m.x.dyh = ro.y + co.y;
    m.x.dxl = fmaf(rp.x, cp.x, ro.z + co.z);
    m.x.dyl = fmaf(rp.x, cp.y, ro.w + co.w);
    m.x.dx = m.x.dxh + m.x.dxl;
    m.x.dy = m.x.dyh + m.x.dyl;
    m.x.d2 = fmaf(m.x.dx, m.x.dx, m.x.dy * m.x.dy);
    m.x.psi = rp.y;
    m.rho = rp.z;
    m.g = rp.w;
    m.g1 = rw.x;
    m.g2 = rw.y;
    m.g3 = rw.z;
    m.ex = cp.z;
    m.ey = cp.w;
    return m;
}

// A child along a run: range place ir + m + 1/2 + (r0 + r1 m + r2 m^2) and angle place iu + (u0 + u1 m + ...), in
// bins from the record's, and the phase (radians), as polynomials in m.
struct ChildRun {
    int ir, iu;
    float r0, r1, r2;
    float u0, u1, u2;
    float p0, p1, p2;
    int at, row;  // staged: index in the footprint that the bits of the rounded places add to, and the row length
    bool inside;  // every stencil of the run lies where the child's bounds say
    bool ahead;   // the run lies in front of the child's origin
};

__device__ __forceinline__ ChildRun child_run(FF K, float h, const MergeChild& C, const MergeRun& m) {
    const ChildRec& R = C.r;
    ChildRun o;
    const float4 ra = R.a, rb = R.b, rc = R.c, re = R.e;
    const float2 rd = make_float2(R.d.x, R.d.y);
    // K L = tb + tl turns with tb exact, and so the range place below: an FP32 L would be off by 1e-6 bins.
    const float L = fmaf(rb.x, m.x.dx, rb.y * m.x.dy);
    const float q2 = fmaf(-L, L, m.x.d2);
    const float B = rcp_approx(fmaf(2.0f, L, rb.z));
    const float e0 = q2 * B;
    const float eps = fmaf(-e0 * e0, B, e0);
    const float Le = L + eps;
    const float tb = fmaf(ra.x, m.x.dxh, ra.y * m.x.dyh);
    float tl = fmaf(ra.x, m.x.dxl, ra.y * m.x.dyl);
    tl = fmaf(ra.z, m.x.dx, tl);
    tl = fmaf(ra.w, m.x.dy, tl);
    const float tot = (tb - round_magic(tb)) + ((fmaf(K.h, eps, rc.x) + tl) + m.x.psi);
    o.p0 = (tot - round_magic(tot)) * kTwoPiF;
    const float iR = rcp_approx(fmaf(0.5f, rb.z, Le));
    const float q = fmaf(m.ex, re.x, m.ey * re.y);
    const float d1 = fmaf(h, (re.z + m.rho) - Le, q * m.g1) * iR;
    const float r1 = h + d1;
    const float r2 = fmaf(-d1, h + r1, 2.0f * q * m.g2) * (0.5f * iR);
    const float r3 = fmaf(-r1, r2, q * m.g3) * iR;
    const float k2 = K.h * kTwoPiF;
    o.p1 = k2 * fmaf(9.25f, r3, d1);
    o.p2 = k2 * r2;
    const float pb = tb * C.bins.x, pr = round_magic(pb);
    float fr = (pb - pr) + fmaf(tb, C.bins.x, -pb);
    fr = fmaf(tb, C.bins.y, fr);
    fr = fmaf(tl, C.bins.x, fr);
    fr = fmaf(eps, R.inv_sdr, fr) + rb.w;
    o.ir = (int)pr;
    o.r0 = fr - 0.5f;
    o.r1 = fmaf(d1, R.inv_sdr, fmaf(h, R.inv_sdr, -1.0f));
    o.r2 = r2 * R.inv_sdr;
    const float Lg = fmaf(rc.y, m.x.dx, rc.z * m.x.dy);
    const float q2h = fmaf(-Lg, Lg, m.x.d2);
    const float Bh = rcp_approx(fmaf(2.0f, Lg, rc.w));
    const float eh = q2h * Bh;
    const float dG = Lg + fmaf(-eh * eh, Bh, eh);
    const float gp = rd.x + dG;
    const float iG = rcp_approx(gp);
    const float duu = fmaf(-rc.z, dG, m.x.dy) * iG;
    const float pu = fmaf(duu, R.inv_sdu, rd.y), ur = round_magic(pu);
    o.iu = (int)ur;
    o.u0 = pu - ur;
    const float cs = (m.g + q) * iG, up = rc.z + duu;
    const float a = fmaf(-up, cs, m.ey), us = up * fmaf(-cs, cs, 1.0f);
    const float n1 = m.g1 * iG, n2 = m.g2 * iG, n3 = m.g3 * iG;
    const float a2 = -fmaf(cs, a, 0.5f * us), a3 = fmaf(fmaf(1.5f * cs, cs, -0.5f), a, us * cs);
    const float as = a * R.inv_sdu;
    const float u3 = fmaf(fmaf(a3, n1 * n1, 2.0f * a2 * n2) * R.inv_sdu, n1, as * n3);
    o.u1 = fmaf(9.25f, u3, as * n1);
    o.u2 = fmaf(a2 * R.inv_sdu, n1 * n1, as * n2);
    const float wr = fmaf(12.25f, fabsf(o.r2), 3.5f * fabsf(o.r1 + 1.0f));
    const float wu = fmaf(12.25f, fabsf(o.u2), 3.5f * fabsf(o.u1));
    // The first tap of the run's upper pixel, less the places' rounding constant (wrapping arithmetic).
    o.row = R.bw;
    o.at = (int)((unsigned)R.bw * (unsigned)(o.ir + R.ir0 - kMergeRun / 2 - R.br0 - kMagicBits) +
                 (unsigned)(o.iu + R.iu0 - 1 - R.bu0 - kMagicBits)) + C.box;
    o.ahead = gp > 0.0f;
    o.inside = o.ahead && pr + fr - wr >= C.lo_r && pr + fr + wr <= C.hi_r && pu - wu >= C.lo_u && pu + wu <= C.hi_u;
    return o;
}

// The child image at bins (ir, iu) and fractions (sr, su); 0 where the stencil leaves it.
template <int SRC>
__device__ __forceinline__ float2 child_gather(const ChildRec& R, int ir, int iu, float sr, float su, bool ahead) {
    if (!(ir >= 1 && ir <= R.snr - 3 && iu >= 1 && iu <= R.snu - 3 && ahead)) return make_float2(0.0f, 0.0f);
    float wr[4], wu[4];
    lagrange_centred(sr, wr);
    lagrange_centred(su, wu);
    return child_stencil<SRC>(R.img + (size_t)(ir - 1) * R.sstr + (iu - 1), R.sstr, wr, wu);
}

// Child C at the parent rows m and m + 1 of a run (the two lanes of f32x2 operations), rotated, with the weights,
// the sum order and the shared 5x4 blocks of child_vpair.  boxes (STAGED): the staged footprints; a warp
// whose runs lie inside the child's (`inside`, for all its lanes) reads shared memory, any other warp the child
// image.  The taps are the same values either way.
template <bool COHERENT, bool STAGED>
__device__ __forceinline__ void child_pair(const MergeChild& C, const ChildRun& t, bool inside, int k, float m, float2& oA,
                                           float2& oB, const float2* boxes) {
    constexpr int SRC = COHERENT ? kCoherent : kLdg;
    const float2 magic = pair(kMagic), nmagic = pair(-kMagic), mone = pair(-1.0f);
    const float n = m + 1.0f;
    const float2 qr = make_float2(fmaf(fmaf(t.r2, m, t.r1), m, t.r0), fmaf(fmaf(t.r2, n, t.r1), n, t.r0));
    const float2 qu = make_float2(fmaf(fmaf(t.u2, m, t.u1), m, t.u0), fmaf(fmaf(t.u2, n, t.u1), n, t.u0));
    const float2 tr = __fadd2_rn(qr, magic), tu = __fadd2_rn(qu, magic);
    const float2 sr = __ffma2_rn(__fadd2_rn(tr, nmagic), mone, qr);
    const float2 su = __ffma2_rn(__fadd2_rn(tu, nmagic), mone, qu);
    float snA, csA, snB, csB;
    __sincosf(fmaf(fmaf(t.p2, m, t.p1), m, t.p0), &snA, &csA);
    __sincosf(fmaf(fmaf(t.p2, n, t.p1), n, t.p0), &snB, &csB);
    float2 vA = make_float2(0.0f, 0.0f), vB = vA;
    const bool share = __float_as_int(tr.y) == __float_as_int(tr.x) && __float_as_int(tu.y) == __float_as_int(tu.x);
    const bool block = inside && __all_sync(0xffffffffu, share);
    if (block) {
        float wrA[4], wuA[4], wrB[4], wuB[4];
        float2 wr2[4], wu2[4];
        lagrange_centred2(sr, wr2);  // both pixels' weights as lane pairs
        lagrange_centred2(su, wu2);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            wrA[k] = wr2[k].x;
            wrB[k] = wr2[k].y;
            wuA[k] = wu2[k].x;
            wuB[k] = wu2[k].y;
        }
        if (STAGED) {
            const int at = (int)((unsigned)(__float_as_int(tr.x) + 2 * k) * (unsigned)t.row + (unsigned)__float_as_int(tu.x)) + t.at;
            child_pair_block<kShared>(boxes + at, t.row, wrA, wuA, wrB, wuB, vA, vB);
        } else {
            const int ir = __float_as_int(tr.x) + t.ir + C.r.ir0 + 2 * k - kMergeRun / 2 - kMagicBits;
            const int iu = __float_as_int(tu.x) + t.iu + C.r.iu0 - 1 - kMagicBits;
            child_pair_block<SRC>(C.r.img + (size_t)ir * C.r.sstr + iu, C.r.sstr, wrA, wuA, wrB, wuB, vA, vB);
        }
    } else if (STAGED && inside) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float wr[4], wu[4];
            lagrange_centred(c ? sr.y : sr.x, wr);
            lagrange_centred(c ? su.y : su.x, wu);
            const int at = (int)((unsigned)(__float_as_int(c ? tr.y : tr.x) + 2 * k + c) * (unsigned)t.row +
                                 (unsigned)__float_as_int(c ? tu.y : tu.x)) + t.at;
            (c ? vB : vA) = child_stencil<kShared>(boxes + at, t.row, wr, wu);
        }
    } else {
    const int ir0 = t.ir + C.r.ir0 + 2 * k - (kMergeRun / 2 - 1) - kMagicBits, iu0 = t.iu + C.r.iu0 - kMagicBits;  // of the upper pixel
#pragma unroll
        for (int c = 0; c < 2; ++c)
            (c ? vB : vA) = child_gather<SRC>(C.r, __float_as_int(c ? tr.y : tr.x) + ir0 + c, __float_as_int(c ? tu.y : tu.x) + iu0,
                                              c ? sr.y : sr.x, c ? su.y : su.x, t.ahead);
    }
    // (vr cs - vi sn, vr sn + vi cs)
    oA = __ffma2_rn(pair(vA.x), make_float2(csA, snA), __fmul2_rn(pair(vA.y), make_float2(-snA, csA)));
    oB = __ffma2_rn(pair(vB.x), make_float2(csB, snB), __fmul2_rn(pair(vB.y), make_float2(-snB, csB)));
}

// Bytes of a merge tile's tables in dynamic shared memory (the staged footprints follow them).
constexpr int kTabBytes = (int)((sizeof(TabF) + 127) / 128 * 128);
static_assert(sizeof(MergeTab) <= sizeof(TabF), "either kind of tables");

// Staged merge tiles: one thread starts the TMA copies of both children's footprints (2-D tiles
// of the child images, the box's first column even so that it starts on a 16-byte boundary;
// rows or columns outside the image arrive as zeros and are never read, since such stencils
// fail the bounds test) with completion on one mbarrier.  Child 1's footprint follows child 0's
// at the next 128-byte boundary.  withhold: bytes declared on the mbarrier beyond those the copies
// deliver (0; 16 in tests of the wait limit, whose phase then never completes).
__device__ __forceinline__ void stage_children(const ChildRec* __restrict__ crec, unsigned box0, unsigned bar,
                                               unsigned withhold) {
    const int bw0 = crec[0].bw, bw1 = crec[1].bw;
    const unsigned b0 = bw0 > 0 ? (unsigned)(crec[0].bh * bw0 * 8) : 0u;
    const unsigned b1 = bw1 > 0 ? (unsigned)(crec[1].bh * bw1 * 8) : 0u;
    if (b0 + b1 == 0) return;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(b0 + b1 + withhold)
                 : "memory");
    if (b0)
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            ::"r"(box0), "l"(crec[0].tmap), "r"(crec[0].bu0), "r"(crec[0].br0), "r"(bar)
            : "memory");
    if (b1)
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            ::"r"(box0 + (b0 + 127u) / 128u * 128u), "l"(crec[1].tmap), "r"(crec[1].bu0), "r"(crec[1].br0), "r"(bar)
            : "memory");
}

// One merge tile: both children regridded onto the parent tile, each rounded to complex64,
// then added (the reference's rounding points).  crec points at the tile's two child records.
// Thread t of kMergeThreads forms the column pairs (rows 2 m and 2 m + 1 of column t mod cols) for
// m = t / cols + i kMergeThreads / cols; its offsets come back from the shared tables per pair, which
// keeps the live state small.
// STAGED: smem is 128-byte aligned and holds [tables | child 0's footprint | child 1's], which
// stage_children's copies fill (completion on the mbarrier at shared address bar).  Each warp
// waits for them, at most wait_ns; a warp whose wait runs out counts a timeout and gathers from
// the child images instead (the same values), and waits once more, as long, before the CTA ends,
// so that no copy into its shared memory is still in flight when it exits.
template <bool COHERENT, bool STAGED>
__device__ __forceinline__ void merge_tile_pairs(float Kf, const PolarDesc& g, const TileItem it,
                                           const float4* __restrict__ tables, const ChildRec* __restrict__ crec,
                                           ChildDup* C, float2* __restrict__ arena, float2* root_out, int root,
                                           char* smem, unsigned bar, unsigned long long wait_ns) {
    Job J;
    J.g = g;
    J.lc = J.g.tile_lc;
    J.tile_r = it.tile_r;
    J.tile_u = it.tile_u;
    if (threadIdx.x < 2) child_dup_store(crec[threadIdx.x], C[threadIdx.x]);
    const float4 d0 = __ldg(&crec[0].d);  // (G, frac(Qu) - 1/2, tile quantum, its inverse)
    TabF& T = *reinterpret_cast<TabF*>(smem);
    setup_polar_tab<kMergeThreads>(J, T, tables, d0.z, d0.w);
    const float2* sbox[2] = {nullptr, nullptr};
    bool waited = true;
    if (STAGED && (C[0].xw > 0 || C[1].xw > 0)) {
        waited = __all_sync(0xffffffffu, timed_wait(bar, 0, wait_ns));
        if (!waited) {
            if ((threadIdx.x & 31) == 0) atomicAdd(&g_wait_timeouts, 1);
        } else {
            const float2* b0 = reinterpret_cast<const float2*>(smem + kTabBytes);
            if (C[0].xw > 0) sbox[0] = b0;
            if (C[1].xw > 0)
                sbox[1] = b0 + (C[0].xw > 0 ? (int)split_box_bytes(C[0].xh, C[0].xw) / 8 : 0);
        }
    }
    float2* dst = J.g.dst ? J.g.dst : (it.node == root ? root_out : arena + J.g.out_offset);
    const int col = threadIdx.x & ((1 << J.lc) - 1), wu = J.tile_u + col;
    constexpr int kPairs = kSplitTilePixels / (2 * kMergeThreads);  // column pairs per thread
    float2 m[2 * kPairs];
    // Gathering tiles keep all their pairs' gathers in flight (unrolled); staged tiles read shared
    // memory with short latency, and the smaller loop body keeps their instruction cache warm.
    constexpr int kUnroll = STAGED ? 1 : kPairs;
#pragma unroll kUnroll
    for (int k = 0; k < kPairs; ++k) {
        const int row = 2 * ((threadIdx.x >> J.lc) + (kMergeThreads >> J.lc) * k);
        const VPix v = tab_vpair(T, row, col);
        float2 a0, b0, a1, b1;
        child_vpair<COHERENT, STAGED>(Kf, C[0], v, a0, b0, sbox[0]);
        child_vpair<COHERENT, STAGED>(Kf, C[1], v, a1, b1, sbox[1]);
        const float2 mA = __fadd2_rn(a0, a1), mB = __fadd2_rn(b0, b1);
        if (!COHERENT) {
            const int wr = J.tile_r + row;
            if (wu < J.g.win_nu) {
                if (wr < J.g.win_nr) dst[(long long)wr * J.g.out_stride + wu] = mA;
                if (wr + 1 < J.g.win_nr) dst[(long long)(wr + 1) * J.g.out_stride + wu] = mB;
            }
        } else {
            // Coherent child loads may not pass this thread's earlier image stores, so the
            // results are stored after the last gather.
            m[2 * k] = mA;
            m[2 * k + 1] = mB;
        }
    }
    if (COHERENT) {
#pragma unroll
        for (int k = 0; k < kPairs; ++k) {
            const int wr = J.tile_r + 2 * ((threadIdx.x >> J.lc) + (kMergeThreads >> J.lc) * k);
            if (wu < J.g.win_nu) {
                if (wr < J.g.win_nr) dst[(long long)wr * J.g.out_stride + wu] = m[2 * k];
                if (wr + 1 < J.g.win_nr) dst[(long long)(wr + 1) * J.g.out_stride + wu] = m[2 * k + 1];
            }
        }
    }
    if (STAGED && !waited) timed_wait(bar, 0, wait_ns);  // the copies may still land: not past the CTA's end
}

// The same in runs of rows: thread t forms rows 8 m ... 8 m + 7 of column t mod cols for m = t / cols, in pairs.
template <bool COHERENT, bool STAGED>
__device__ __forceinline__ void merge_tile_runs(FF K, const PolarDesc* __restrict__ nodes, const PolarDesc& g,
                                                const TileItem it, const float4* __restrict__ tables,
                                                const ChildRec* __restrict__ crec, MergeChild* C,
                                                float2* __restrict__ arena, float2* root_out, int root, char* smem,
                                                unsigned bar, unsigned long long wait_ns) {
    Job J;
    J.g = g;
    J.lc = J.g.tile_lc;
    J.tile_r = it.tile_r;
    J.tile_u = it.tile_u;
    if (threadIdx.x < 2)
        merge_child(K, nodes[threadIdx.x ? g.right : g.left], crec[threadIdx.x],
                    STAGED && threadIdx.x && crec[0].bw > 0 ? (int)split_box_bytes(crec[0].bh, crec[0].bw) / 8 : 0,
                    C[threadIdx.x]);
    const float4 d0 = __ldg(&crec[0].d);  // (G, frac(Qu) - 1/2, tile quantum, its inverse)
    MergeTab& T = *reinterpret_cast<MergeTab*>(smem);
    setup_merge<kMergeThreads>(K, J, T, tables, d0.z, d0.w);
    // Staged: the footprints, and the second one's offset (elements) when both are there.
    const float2* boxes = reinterpret_cast<const float2*>(smem + kTabBytes);
    bool waited = true;
    if (STAGED && (C[0].r.bw > 0 || C[1].r.bw > 0)) {
        waited = __all_sync(0xffffffffu, timed_wait(bar, 0, wait_ns));
        if (!waited && (threadIdx.x & 31) == 0) atomicAdd(&g_wait_timeouts, 1);
    }
    float2* dst = J.g.dst ? J.g.dst : (it.node == root ? root_out : arena + J.g.out_offset);
    const int col = threadIdx.x & ((1 << J.lc) - 1), run = threadIdx.x >> J.lc;
    const int wu = J.tile_u + col, wr = J.tile_r + kMergeRun * run;
    const int rows = wu < J.g.win_nu ? J.g.win_nr - wr : 0;  // of the run, in the window
    float2* px = dst + (long long)wr * J.g.out_stride + wu;
    float2 v[kMergeRun];
    const float h = J.g.tf[4].x;
    const ChildRun t0 = child_run(K, h, C[0], merge_run(T.row[run], T.col[col]));
    asm volatile("" ::: "memory");
    const ChildRun t1 = child_run(K, h, C[1], merge_run(T.row[run], T.col[col]));
    const bool in0 = __all_sync(0xffffffffu, t0.inside && (!STAGED || (waited && C[0].r.bw > 0)));
    const bool in1 = __all_sync(0xffffffffu, t1.inside && (!STAGED || (waited && C[1].r.bw > 0)));
    // A small loop body keeps the instruction cache warm; coherent tiles keep their results in registers.
    constexpr int kPairs = kMergeRun / 2, kUnroll = COHERENT ? kPairs : 1;
    float x = -0.5f * (kMergeRun - 1);
#pragma unroll kUnroll
    for (int k = 0; k < kPairs; ++k, x += 2.0f) {
        float2 a0, b0, a1, b1;
        child_pair<COHERENT, STAGED>(C[0], t0, in0, k, x, a0, b0, boxes);
        child_pair<COHERENT, STAGED>(C[1], t1, in1, k, x, a1, b1, boxes);
        const float2 mA = __fadd2_rn(a0, a1), mB = __fadd2_rn(b0, b1);
        if (!COHERENT) {
            if (2 * k < rows) px[0] = mA;
            if (2 * k + 1 < rows) px[J.g.out_stride] = mB;
            px += 2 * J.g.out_stride;
        } else {
            // Coherent child loads may not pass this thread's earlier image stores, so the
            // results are stored after the last gather.
            v[2 * k] = mA;
            v[2 * k + 1] = mB;
        }
    }
    if (COHERENT) {
#pragma unroll
        for (int k = 0; k < kMergeRun; ++k)
            if (k < rows) px[k * J.g.out_stride] = v[k];
    }
    if (STAGED && !waited) timed_wait(bar, 0, wait_ns);  // the copies may still land: not past the CTA's end
}

// The children of a merge tile in shared memory, for either kind.
union MergeChildren {
    __device__ MergeChildren() {}
    ChildDup dup[2];
    MergeChild run[2];
};

enum MergeKind { kMergeEither, kMergeRuns, kMergePairs };

// One merge tile; KIND: kMergeRuns or kMergePairs where the caller knows that the node merges so.
template <bool COHERENT = false, bool STAGED = false, int KIND = kMergeEither>
__device__ __forceinline__ void merge_tile(FF K, const PolarDesc* __restrict__ nodes, const TileItem it,
                                           const float4* __restrict__ tables, const ChildRec* __restrict__ crec,
                                           MergeChildren& C, float2* __restrict__ arena, float2* root_out, int root,
                                           char* smem, unsigned bar = 0, unsigned long long wait_ns = 0) {
    const PolarDesc& g = nodes[it.node];
    if (KIND == kMergeRuns || (KIND == kMergeEither && merges_in_runs(g, K.h)))
        merge_tile_runs<COHERENT, STAGED>(K, nodes, g, it, tables, crec, C.run, arena, root_out, root, smem, bar, wait_ns);
    else
        merge_tile_pairs<COHERENT, STAGED>(K.h, g, it, tables, crec, C.dup, arena, root_out, root, smem, bar, wait_ns);
}

__global__ void __launch_bounds__(kMergeThreads, 8) split_merge_kernel(SplitParams P, const PolarDesc* __restrict__ nodes,
                                                                  const TileItem* __restrict__ items,
                                                                  const float4* __restrict__ tables,
                                                                  const ChildRec* __restrict__ crecs,
                                                                  float2* __restrict__ arena, float2* root_out,
                                                                  int root) {
    extern __shared__ __align__(16) char smem[];
    __shared__ MergeChildren C;
    merge_tile<false>(FF{P.Kh, P.Kl}, nodes, items[blockIdx.x], tables, crecs + 2 * (long long)blockIdx.x, C, arena,
                                     root_out, root, smem);
}

// The merge with both children's footprints staged in shared memory by TMA (tiles whose child
// records carry tensor maps; any other child gathers from its image as in split_merge_kernel).
// The dynamic shared memory is 128 bytes of alignment slack, the tables and the footprints.
template <int KIND>
__global__ void __launch_bounds__(kMergeThreads, KIND == kMergeRuns ? 6 : 8) split_merge_staged_kernel(SplitParams P,
                                                                         const PolarDesc* __restrict__ nodes,
                                                                         const TileItem* __restrict__ items,
                                                                         const float4* __restrict__ tables,
                                                                         const ChildRec* __restrict__ crecs,
                                                                         float2* __restrict__ arena,
                                                                         float2* root_out, int root,
                                                                         unsigned long long wait_ns, int withheld) {
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ MergeChildren C;
    __shared__ __align__(8) unsigned long long mbar;
    const unsigned raw = (unsigned)__cvta_generic_to_shared(smem_raw);
    char* smem = smem_raw + (((raw + 127u) & ~127u) - raw);
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&mbar);
    const ChildRec* crec = crecs + 2 * (long long)blockIdx.x;
    const TileItem it = items[blockIdx.x];
    if (threadIdx.x == 0)
        stage_children(crec, (unsigned)__cvta_generic_to_shared(smem + kTabBytes), bar, it.node == withheld ? 16u : 0u);
    merge_tile<false, true, KIND>(FF{P.Kh, P.Kl}, nodes, it, tables, crec, C, arena, root_out, root, smem, bar, wait_ns);
}

// All merge levels in one persistent launch.  Items are in height order; a CTA claims the next
// item and waits (bounded) until the item's node has no unfinished merge children.  Every
// dependency of an item has a lower index, so it is held by a running CTA (or finished) and the
// wait ends.  A finished tile counts down its node's tiles; the node's last tile counts down its
// parent's pending children.  A wait that runs out sets *status and every CTA stops.
__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}


__global__ void __launch_bounds__(kMergeThreads, 6) split_merge_queue_kernel(SplitParams P, const PolarDesc* __restrict__ nodes,
                                                                        const TileItem* __restrict__ items, int nitems,
                                                                        const float4* __restrict__ tables,
                                                                        const ChildRec* __restrict__ crecs,
                                                                        float2* arena, float2* root_out, int root,
                                                                        MergeQueue Q) {
    extern __shared__ __align__(16) char smem[];
    __shared__ MergeChildren C;
    __shared__ int s_item, s_ok;
    for (;;) {
        if (threadIdx.x == 0) {
            const int idx = atomicAdd(Q.next, 1);
            int ok = 1;
            if (idx < nitems) {
                const int node = items[idx].node;
                const unsigned long long t0 = global_ns();
                while (ld_acquire_gpu(Q.pending + node) > 0) {
                    if (ld_acquire_gpu(Q.status) != 0) {  // another CTA gave up: stop too
                        ok = 0;
                        break;
                    }
                    if (global_ns() - t0 > Q.limit_ns) {
                        atomicExch(Q.status, 1);
                        ok = 0;
                        break;
                    }
                    __nanosleep(200);
                }
            }
            s_item = idx;
            s_ok = ok;
        }
        __syncthreads();
        const int idx = s_item;
        if (idx >= nitems || !s_ok) return;
        const TileItem it = items[idx];
        merge_tile<true>(FF{P.Kh, P.Kl}, nodes, it, tables, crecs + 2 * (long long)idx, C, arena, root_out, root, smem);
        __syncthreads();  // every thread's writes of this tile are issued
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicSub(Q.remaining + it.node, 1) == 1) {
                __threadfence();
                const int parent = Q.parent[it.node];
                if (parent >= 0) atomicSub(Q.pending + parent, 1);
            }
        }
    }
}

SplitParams make_params(const PulseInputs& in, int chunk, int cap, int pulse_split) {
    SplitParams P;
    P.in = in;
    P.out = nullptr;
    P.out_stride = 0;
    P.K = in.k * kInvTwoPi;
    P.inv_dr = in.data_dr != 0.0 ? 1.0 / in.data_dr : 0.0;
    int e = 0;
    frexp(fabs(P.K) > 0.0 ? fabs(P.K) : 1e-30, &e);
    P.scale_w = ldexp(1.0, e - 10);
    P.inv_scale_w = ldexp(1.0, 10 - e);
    P.Kf = (float)P.K;
    P.inv_drf = (float)P.inv_dr;
    P.chunk = chunk < 1 ? 1 : (chunk > kMaxChunk ? kMaxChunk : chunk);
    P.cap = cap < 64 ? 64 : cap;  // >= kMaxChunk two-float records (32 bytes each) fit the window space
    P.pulse_split = pulse_split;
    P.split_stride = 0;
    P.envelope = kDirectEnvelope;
    P.Kh = (float)P.K;
    P.Kl = (float)(P.K - (double)P.Kh);
    P.rsh = (float)in.range_start;
    P.rsl = (float)(in.range_start - (double)P.rsh);
    P.idrh = (float)P.inv_dr;
    P.idrl = (float)(P.inv_dr - (double)P.idrh);
    return P;
}

size_t merge_smem() { return sizeof(TabF); }

size_t dynamic_smem(int cap, bool polar) {
    size_t win = (size_t)cap * 32;
    if (polar && win < sizeof(PolarTables)) win = sizeof(PolarTables);
    return window_offset() + win + raw_bytes_for(cap, kMaxChunk);
}

template <class K>
int prepare(K kernel, size_t smem) {
    return allow_shared(reinterpret_cast<const void*>(kernel), smem);
}

// Pulse split that fills the GPU's CTA slots best: the fewest waves ceil(tiles s / slots) / s over
// s <= 8 (and <= pulses), ties to the smaller split.  A tile's pulse ranges are independent
// work, so a small image with few tiles still keeps every SM busy to the end.
template <class K>
int best_pulse_split(K kernel, int threads, size_t smem, long long tiles, int pulses) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm <= 0 ||
        sms <= 0 || tiles <= 0) {
        cudaGetLastError();
        return 1;
    }
    const long long slots = (long long)sms * per_sm;
    int best = 1;
    double best_waves = 1e300;
    for (int sp = 1; sp <= 8 && sp <= pulses; ++sp) {
        const double waves = (double)((tiles * sp + slots - 1) / slots) / sp;
        if (waves < best_waves - 1e-9) {
            best_waves = waves;
            best = sp;
        }
    }
    return best;
}

int tiles_of(int nr, int nu, int lc) {
    const int cols_t = 1 << lc, rows_t = kSplitTilePixels >> lc;
    return ((nr + rows_t - 1) / rows_t) * ((nu + cols_t - 1) / cols_t);
}

// Window entries for one chunk: `chunk` pulses whose windows span at most
// `window_bins` bins each (the kernel packs the actual, usually smaller, windows).
int capacity_for(int chunk, int window_bins, int budget_bytes = kWindowBudget) {
    long long cap = (long long)chunk * window_bins;
    // With bulk staging a window bin also needs 8 bytes of raw samples (plus a fixed margin).
    // (2 KB more are left for the bulk path's larger static shared memory.)
    const long long budget =
        SARBP_BULK_WINDOWS ? (budget_bytes - raw_bytes_for(0, kMaxChunk) - 2048) / 40 : budget_bytes / 32;
    return (int)(cap > budget ? budget : cap);
}

// Lattice tiles: at least room for the block halves' exchange of their images (half a tile's pixels each).
int lattice_capacity(int chunk, int window_bins) {
    return std::max(capacity_for(chunk, window_bins, kLatticeWindowBudget),
                    kSplitTilePixels * (int)sizeof(float2) / 32);
}

// Leaf window entries: the windows share the CTA's shared memory with the chunk's pulse and
// (pulse, column) records, within the same per-CTA total as the direct kernels' windows.
int leaf_capacity(int chunk, int window_bins) {
    return capacity_for(chunk, window_bins, kLeafWindowBudget - (int)leaf_window_offset());
}

}  // namespace

int split_window_bins(double radius, double data_dr) {
    // Worst case: the pixel offset lies along the line of sight; eps <= radius^2/(2(R - radius)) is
    // small at any range used here (R >= 100 m gives the bound below).
    const double wing = (radius + radius * radius / 200.0) / fabs(data_dr) + 0.01;
    return (int)ceil(2.0 * wing) + 4;
}

int split_chunk_for(int window_bins, int requested, bool leaf) {
    const int most = leaf ? kMaxLeafChunk : kMaxChunk;
    int ch = requested > 0 ? requested : most;
    if (ch > most) ch = most;
    const int fit = kWindowBudget / (window_bins * 32 > 0 ? window_bins * 32 : 32);
    if (ch > fit) ch = fit;
    return ch < 1 ? 1 : ch;
}

int split_polar_tile_lc(const PolarDesc& g, double* radius) { return split_polar_tile_lc_slack(g, 1.0, radius); }

int split_polar_tile_lc_slack(const PolarDesc& g, double slack, double* radius) {
    // Ground displacement per range row <= dr * r / g; per angle column <= du * g / sqrt(1 - u^2).
    const double rmin = g.r0 + g.win_r0 * g.dr, rmax = g.r0 + (g.win_r0 + g.win_nr - 1) * g.dr;
    const double gmin = sqrt(fmax(1e-6, rmin * rmin - g.oz * g.oz));
    const double gmax = sqrt(fmax(1e-6, rmax * rmax - g.oz * g.oz));
    const double ua = fabs(g.u0 + g.win_u0 * g.du), ub = fabs(g.u0 + (g.win_u0 + g.win_nu - 1) * g.du);
    const double cmin = sqrt(fmax(1e-6, 1.0 - fmax(ua, ub) * fmax(ua, ub)));
    const double per_row = fabs(g.dr) * fmax(rmin, rmax) / gmin;
    const double per_col = fabs(g.du) * gmax / cmin;
    double rads[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int best = 5;
    double best_r = 1e300;
    for (int lc = 2; lc <= 5; ++lc) {
        const double er = (kSplitTilePixels >> lc) * per_row, eu = (1 << lc) * per_col;
        rads[lc] = 0.5 * sqrt(er * er + eu * eu) * 1.05;
        if (rads[lc] < best_r) {
            best_r = rads[lc];
            best = lc;
        }
    }
    // The widest shape within `slack` of the smallest radius (wider tiles keep a warp's pixels in
    // fewer rows).
    for (int lc = 5; lc > best; --lc)
        if (rads[lc] <= slack * best_r) {
            best = lc;
            break;
        }
    if (radius) *radius = rads[best];
    return best;
}

float split_merge_run_limit(const PolarDesc& g, const PolarDesc* children[2]) {
    // Nearest and farthest rows, widest column of the window (its last tiles' overhang included).
    const int rows_t = kSplitTilePixels >> g.tile_lc, cols_t = 1 << g.tile_lc;
    const double ra = g.r0 + g.win_r0 * g.dr, rb = ra + (g.win_nr - 1 + rows_t) * g.dr, z = fabs(g.oz);
    const double r0 = fmin(ra, rb), r1 = fmax(ra, rb), h = fabs(g.dr);
    const double ua = fabs(g.u0 + g.win_u0 * g.du), ub = fabs(g.u0 + (g.win_u0 + g.win_nu - 1) * g.du);
    const double um = fmax(ua, ub), cm = sqrt(fmax(1e-12, 1.0 - um * um)), m = 0.5 * (kMergeRun - 1), m4 = m * m * m * m;
    if (!(r0 - 8.0 * h > z) || !(um < 1.0)) return 0.0f;
    const double gn = sqrt((r0 - 8.0 * h) * (r0 - 8.0 * h) - z * z), gf = sqrt(r1 * r1 - z * z), ig = 1.0 / gn;
    // K at which the FP32 rounding of eps (1e-8 of K rho^2 / R) stays below 6e-8 turns.
    const double er = 0.5 * rows_t * h * r0 * ig, eu = 0.5 * cols_t * fabs(g.du) * gf / cm, rho2 = er * er + eu * eu;
    double limit = 6.0 * r0 / rho2;
    for (int k = 0; k < 2; ++k) {
        const PolarDesc& c = *children[k];
        const double dx = g.ox - c.ox, dy = g.oy - c.oy, dz = fabs(g.oz - c.oz), off = sqrt(dx * dx + dy * dy);
        const double q = fabs(dx) + um * fabs(dy);
        if (!(gn > 4.0 * off) || !(r0 > 4.0 * (off + dz))) return 0.0f;
        // What child_run leaves out at a run's ends: of the phase and of the angle place the fourth order and the
        // third beyond its linear fit (10.5 of m^3), of the range place the third.
        const double id = 1.0 / (r0 - off - dz), iG = 1.0 / (gn - off);
        const double x = h * r0 * ig, y2 = h * h * z * z * ig * ig;  // the step of g; g_2 = y2 / 2 g
        const double f2 = q * y2 * ig, f3 = f2 * x * ig, f4 = 1.25 * f3 * x * ig;
        const double d1 = h * (off + dz + q * r0 * ig) * id, r2 = (f2 + 3.0 * h * d1) * id, r3 = (f3 + 2.0 * h * r2) * id;
        const double turns = 10.5 * r3 + m4 * (f4 + 2.0 * h * r3 + r2 * r2) * id;  // per K
        const double n1 = x * iG, n2 = 0.5 * y2 * ig * iG, n3 = n2 * x * ig;
        const double angle = 2.0 * off * iG / fabs(c.du) *
                             (10.5 * (n3 + 2.0 * n1 * n2 + n1 * n1 * n1) +
                              m4 * (1.25 * n3 * x * ig + 2.0 * n1 * n3 + n2 * n2 + 3.0 * n1 * n1 * n2 + n1 * n1 * n1 * n1));
        if (!(m * m * m * r3 / fabs(c.dr) <= 2e-6) || !(angle <= 2e-6)) return 0.0f;
        limit = fmin(limit, 3e-7 / fmax(turns, 1e-30));
    }
    return (float)limit;
}

int launch_split_polar(const PulseInputs& in, const PolarDesc& g, int pulse_split, int chunk, int window_bins,
                       float2* out, long long out_stride, long long split_stride, cudaStream_t s) {
    // Runs of columns need tiles at least a run wide and an angle step at which the expansion holds for any
    // pulse the grid resolves (K |a| du below half a turn: 0.5 du^4 turns at fifth order).
    const double ua = fabs(g.u0 + g.win_u0 * g.du), ub = fabs(g.u0 + (g.win_u0 + g.win_nu - 1) * g.du);
    const bool runs = g.tile_lc >= 3 && fabs(in.k) > 1e-2 && fabs(g.du) <= 0.002 * (1.0 - fmax(ua, ub) * fmax(ua, ub));
    int cap = capacity_for(chunk, window_bins);
    if (runs) cap = std::max(cap, kSplitTilePixels * (int)sizeof(float2) / 32);  // the halves' exchange
    SplitParams P = make_params(in, chunk, cap, pulse_split);
    P.out = out;
    P.out_stride = out_stride;
    P.split_stride = split_stride;
    const size_t smem = dynamic_smem(P.cap, true);
    dim3 grid(tiles_of(g.win_nr, g.win_nu, g.tile_lc), pulse_split);
    if (runs) {
        if (int st = prepare(split_polar_runs_kernel, smem)) return st;
        split_polar_runs_kernel<<<grid, kThreads, smem, s>>>(P, g);
    } else {
        if (int st = prepare(split_polar_kernel, smem)) return st;
        split_polar_kernel<<<grid, kThreads, smem, s>>>(P, g);
    }
    note_launches(1);
    return check_launch("split_polar");
}

int split_wait_timeouts(int* count) {
    const cudaError_t e = cudaMemcpyFromSymbol(count, g_wait_timeouts, sizeof(int));
    if (e != cudaSuccess) return fail(SARBP_ERR_CUDA, "wait timeouts: %s", cudaGetErrorString(e));
    return SARBP_OK;
}

// The pulse split of a direct lattice launch that asks for the automatic one: sized for the
// largest window budget, so that it depends on the lattice only and the workspace query and the
// launch agree (fewer pulses only lower it).
int split_lattice_auto_split(const sarbp_lattice& lat, int pulses) {
    const size_t smem = dynamic_smem(capacity_for(kMaxChunk, 1 << 20, kLatticeWindowBudget), false);
    if (prepare(split_lattice_kernel, smem) != SARBP_OK) return 1;
    return best_pulse_split(split_lattice_kernel, kThreads, smem, tiles_of(lat.rows, lat.cols, 5), pulses);
}

int launch_split_lattice(const PulseInputs& in, const sarbp_lattice& lat, int pulse_split, int chunk, int window_bins,
                         float2* out, long long split_stride, cudaStream_t s) {
    SplitParams P = make_params(in, chunk, lattice_capacity(chunk, window_bins), pulse_split);
    P.out = out;
    P.split_stride = split_stride;
    const int lc = 5;
    const size_t smem = dynamic_smem(P.cap, false);
    dim3 grid(tiles_of(lat.rows, lat.cols, lc), pulse_split);
    if (int st = prepare(split_lattice_kernel, smem)) return st;
    split_lattice_kernel<<<grid, kThreads, smem, s>>>(P, lat, lc);
    note_launches(1);
    return check_launch("split_lattice");
}

int split_points_auto_split(int npts, int pulses) {
    const size_t smem = dynamic_smem(capacity_for(kMaxChunk, 1 << 20), false);
    int dev = 0, sms = 0, per_sm = 0;
    if (prepare(split_points_kernel, smem) != SARBP_OK || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, split_points_kernel, kThreads, smem) != cudaSuccess ||
        per_sm <= 0 || sms <= 0) {
        cudaGetLastError();
        return 1;
    }
    // In pulses of a block: the blocks' work spread over the slots, each with its tile's set-up, which costs as much as
    // 40 pulses, and one block more at the end (tiles of a list take unevenly long).  Parts also cost memory and a pass
    // that adds them, hence a twentieth at least.  One pass, best of 2 .. 8 and this choice, us: 8,000 points x 512 pulses 182,
    // 71 and 71; 192,384 x 1024 900, 610 and 623; 300,000 x 2000 2854, 1688 and 1694; a million x 256 735, 790 and 735.
    const double waves = (double)((npts + (long long)kPointTile - 1) / kPointTile) / ((double)sms * per_sm);
    const auto cost = [&](int sp) { return waves * (pulses + 40.0 * sp) + (double)pulses / sp + 40.0; };
    int best = 1;
    for (int sp = 2; sp <= 8 && sp <= pulses; ++sp)
        if (cost(sp) < 0.95 * cost(1) && cost(sp) < cost(best)) best = sp;
    return best;
}

int split_points_capacity(int chunk, int window_bins) { return capacity_for(chunk, window_bins); }

int launch_split_points(const PulseInputs& in, const double* xyz, int npts, const PointOrder* order, const int* index,
                        int pulse_split, int chunk, int window_bins, float2* out, long long split_stride,
                        cudaStream_t s) {
    SplitParams P = make_params(in, chunk, capacity_for(chunk, window_bins), pulse_split);
    P.out = out;
    P.split_stride = split_stride;
    const size_t smem = dynamic_smem(P.cap, false);
    if (int st = prepare(split_points_kernel, smem)) return st;
    dim3 grid((npts + kPointTile - 1) / kPointTile, pulse_split);
    split_points_kernel<<<grid, kThreads, smem, s>>>(P, xyz, npts, order, index);
    note_launches(1);
    return check_launch("split_points");
}

size_t split_adjoint_workspace(const sarbp_lattice& lat, int pulses) {
    return (size_t)tiles_of(lat.rows, lat.cols, 5) * (size_t)pulses * kAdjVals * sizeof(float);
}

int launch_split_lattice_adjoint(const PulseInputs& in, const sarbp_lattice& lat, int chunk, int window_bins,
                                 const float2* grad, float* partials, double* grad_pos, double* grad_phase,
                                 double* grad_weight, cudaStream_t s) {
    SplitParams P = make_params(in, chunk, capacity_for(chunk, window_bins, kLatticeWindowBudget), 1);
    const int lc = 5;
    const size_t smem = dynamic_smem(P.cap, false);
    const int ntiles = tiles_of(lat.rows, lat.cols, lc);
    if (int st = prepare(split_lattice_adjoint_kernel, smem)) return st;
    const dim3 grid(ntiles, best_pulse_split(split_lattice_adjoint_kernel, kThreads, smem, ntiles, in.pulses));
    split_lattice_adjoint_kernel<<<grid, kThreads, smem, s>>>(P, lat, lc, grad, partials);
    note_launches(1);
    if (int st = check_launch("split_lattice_adjoint")) return st;
    adjoint_sum_kernel<<<grid_blocks(in.pulses, kSumPulses), kThreads, 0, s>>>(partials, ntiles, in.pulses, in.weight,
                                                                              grad_pos, grad_phase, grad_weight);
    note_launches(1);
    return check_launch("adjoint_sum");
}

int launch_split_ffbp_tables(const PulseInputs& in, const PolarDesc* nodes, int n_nodes, int max_dim,
                             float4* tables, cudaStream_t s) {
    if (n_nodes <= 0) return SARBP_OK;
    dim3 grid((max_dim + kThreads - 1) / kThreads, n_nodes);
    ffbp_tables_kernel<<<grid, kThreads, 0, s>>>(table_consts(make_params(in, 1, 4, 1)), nodes, tables);
    note_launches(1);
    return check_launch("split_ffbp_tables");
}

int launch_split_ffbp_leaf_pulses(const PulseInputs& in, const PolarDesc* nodes, const int* leaves, int n_leaves,
                                  void* recs, cudaStream_t s) {
    if (n_leaves <= 0) return SARBP_OK;
    ffbp_leaf_pulses_kernel<<<n_leaves, 128, 0, s>>>(in.k * kInvTwoPi, in.pos, in.weight, in.phase, nodes, leaves,
                                                     reinterpret_cast<PulseRec*>(recs));
    note_launches(1);
    return check_launch("split_ffbp_leaf_pulses");
}

int launch_split_ffbp_child_records(double k, const PolarDesc* nodes, const float4* tables, const TileItem* items,
                                    int n_items, float2* arena, const void* tmaps, void* recs, cudaStream_t s) {
    if (n_items <= 0) return SARBP_OK;
    PulseInputs none{};
    none.k = k;
    none.data_dr = 1.0;
    const SplitParams P = make_params(none, 1, 4, 1);
    ffbp_child_records_kernel<<<grid_blocks(2LL * n_items, kThreads), kThreads, 0, s>>>(
        P.Kh, P.Kl, (float)P.scale_w, (float)P.inv_scale_w, nodes, tables, items, n_items, arena, tmaps,
        reinterpret_cast<ChildRec*>(recs));
    note_launches(1);
    return check_launch("split_ffbp_child_records");
}

size_t split_ffbp_pulse_record_bytes() { return sizeof(PulseRec); }
size_t split_ffbp_child_record_bytes() { return sizeof(ChildRec); }

int launch_split_ffbp_leaves(const PulseInputs& in, const PolarDesc* nodes, const TileItem* items, int nitems,
                             int chunk, int window_bins, const float4* tables, const void* precs, float2* arena,
                             float2* root_out, int root, cudaStream_t s) {
    if (nitems <= 0) return SARBP_OK;
    SplitParams P = make_params(in, chunk, leaf_capacity(chunk, window_bins), 1);
    const size_t smem = leaf_window_offset() + (size_t)P.cap * 32;
    // With up to two tiles per SM a sub-partition has only one or two of their warps, and a tile's latency
    // counts: two threads per run (the same image).  32 pulses, 150 tiles: 16.3 us, one thread per run 20.8;
    // 240 tiles 22.3 and 24.4; 160 tiles of 64 pulses 36.6 and 37.3; four threads per run 17.7, 32.6 and 55.0.
    const bool few = nitems <= 2 * sm_count();
    const auto kernel = few ? split_leaf_kernel<2> : split_leaf_kernel<1>;
    if (int st = prepare(kernel, smem)) return st;
    kernel<<<nitems, kLeafThreads * (few ? 2 : 1), smem, s>>>(P, nodes, items, tables,
                                                              reinterpret_cast<const PulseRec*>(precs), arena, root_out, root);
    note_launches(1);
    return check_launch("split_ffbp_leaves");
}

int launch_split_ffbp_merges(double k, const PolarDesc* nodes, const TileItem* items, int nitems,
                             const float4* tables, const void* crecs, float2* arena, float2* root_out, int root,
                             size_t box_bytes, unsigned long long wait_ns, int withheld, bool runs, cudaStream_t s) {
    if (nitems <= 0) return SARBP_OK;
    PulseInputs none{};
    none.k = k;
    none.data_dr = 1.0;
    SplitParams P = make_params(none, 1, 4, 1);
    if (box_bytes > 0) {
        const size_t smem = 128 + kTabBytes + box_bytes;
        const auto kernel = runs ? split_merge_staged_kernel<kMergeRuns> : split_merge_staged_kernel<kMergePairs>;
        if (int st = prepare(kernel, smem)) return st;
        kernel<<<nitems, kMergeThreads, smem, s>>>(
            P, nodes, items, tables, reinterpret_cast<const ChildRec*>(crecs), arena, root_out, root, wait_ns, withheld);
        note_launches(1);
        return check_launch("split_ffbp_merges (staged)");
    }
    const size_t smem = merge_smem();
    if (int st = prepare(split_merge_kernel, smem)) return st;
    split_merge_kernel<<<nitems, kMergeThreads, smem, s>>>(P, nodes, items, tables, reinterpret_cast<const ChildRec*>(crecs),
                                                      arena, root_out, root);
    note_launches(1);
    return check_launch("split_ffbp_merges");
}

int launch_split_ffbp_merge_queue(double k, const PolarDesc* nodes, const TileItem* items, int nitems,
                                  const float4* tables, const void* crecs, float2* arena, float2* root_out, int root,
                                  const MergeQueue& Q, cudaStream_t s) {
    if (nitems <= 0) return SARBP_OK;
    PulseInputs none{};
    none.k = k;
    none.data_dr = 1.0;
    SplitParams P = make_params(none, 1, 4, 1);
    const size_t smem = merge_smem();
    if (int st = prepare(split_merge_queue_kernel, smem)) return st;
    int dev = 0, sms = 1, per_sm = 1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, split_merge_queue_kernel, kMergeThreads, smem);
    if (e != cudaSuccess) return fail(SARBP_ERR_CUDA, "merge queue: %s", cudaGetErrorString(e));
    const int blocks = std::max(1, std::min(nitems, sms * std::max(1, per_sm)));
    split_merge_queue_kernel<<<blocks, kMergeThreads, smem, s>>>(P, nodes, items, nitems, tables,
                                                            reinterpret_cast<const ChildRec*>(crecs), arena,
                                                            root_out, root, Q);
    note_launches(1);
    return check_launch("split_ffbp_merge_queue");
}

// ---- polar image -> ground lattice (evaluate_image on a lattice, split precision) -----------
//
// A lattice tile is a parent tile whose pixels lie on the ground lattice, and the polar
// image is its only child: one two-float record per tile (child_rec_at at the tile centre),
// then per pixel the merge kernel's FP32 child coordinates, 4x4 stencil and phase.  The
// phase restores exp(j k r) (r: the point's range to the image origin); no demodulation.
// The pixel offsets are two-float products of whole numbers and the steps (split on the host): in FP64 their twenty
// operations per pixel bound the kernel (2048 x 2048 of a 4096-pulse polar image: 184 us, now 100; the image alone takes 91 to read).
struct LatticeSteps {
    FF rx, ry, cx, cy;          // step_row, step_col
    float quantum, inv_quantum;  // of the offsets' hi parts: 12 bits of the largest
};

__device__ __forceinline__ void step_offset(float di, float dj, FF r, FF c, float q, float iq, float& h, float& l) {
    const float p1 = di * r.h, p2 = dj * c.h, s = p1 + p2, b = s - p1;
    float e = (p1 - (s - b)) + (p2 - b);
    e += fmaf(di, r.h, -p1) + fmaf(dj, c.h, -p2);
    e = fmaf(di, r.l, fmaf(dj, c.l, e));
    h = rintf(s * iq) * q;
    l = (s - h) + e;
}

__global__ void __launch_bounds__(kThreads, 5) split_evaluate_lattice_kernel(float Kh, float Kl, float scale_w,
                                                                             float inv_scale_w, PolarDesc c,
                                                                             const float2* __restrict__ img,
                                                                             sarbp_lattice lat, LatticeSteps L, int lc,
                                                                             float2* __restrict__ out) {
    __shared__ ChildRec C;
    Job J;
    tile_of(blockIdx.x, lat.cols, lc, J.tile_r, J.tile_u);
    const int hr = (kSplitTilePixels >> lc) >> 1, hc = (1 << lc) >> 1;
    if (threadIdx.x < 32) {  // lanes 0 and 1 form the centre's x and y
        const bool y = threadIdx.x == 1;
        FF v;
        split2((y ? lat.origin[1] : lat.origin[0]) + (double)(J.tile_r + hr) * (y ? lat.step_row[1] : lat.step_row[0]) +
                   (double)(J.tile_u + hc) * (y ? lat.step_col[1] : lat.step_col[0]),
               v.h, v.l);
        const FF w{__shfl_sync(0xffffffffu, v.h, 1), __shfl_sync(0xffffffffu, v.l, 1)};
        if (threadIdx.x == 0) C = child_rec_at(FF{Kh, Kl}, scale_w, inv_scale_w, c, v, w, img);
    }
    Pix px[kPX];
#pragma unroll
    for (int k = 0; k < kPX; ++k) {
        const int p = threadIdx.x + kThreads * k;
        const float di = (float)((p >> lc) - hr), dj = (float)((p & ((1 << lc) - 1)) - hc);
        Pix& q = px[k];
        step_offset(di, dj, L.rx, L.cx, L.quantum, L.inv_quantum, q.dxh, q.dxl);
        step_offset(di, dj, L.ry, L.cy, L.quantum, L.inv_quantum, q.dyh, q.dyl);
        q.dx = q.dxh + q.dxl;
        q.dy = q.dyh + q.dyl;
        q.d2 = q.dx * q.dx + q.dy * q.dy;
        q.psi = 0.0f;
    }
    __syncthreads();
    const float Kf = Kh;
    const int cols_t = 1 << lc;
#pragma unroll
    for (int k = 0; k < kPX; ++k) {
        const float2 v = child_value(Kf, C, px[k]);
        const int p = threadIdx.x + kThreads * k;
        const int wr = J.tile_r + (p >> lc), wu = J.tile_u + (p & (cols_t - 1));
        if (wr < lat.rows && wu < lat.cols) out[(long long)wr * lat.cols + wu] = v;
    }
}

// ---- batched scenes: persistent work-queue kernels ------------------------------------------
//
// Many independent scenes (direct lattice images and FFBP trees) run as one work list.
// Each scene's parameters live in a device array; tile items carry their scene in
// TileItem::pad and FFBP nodes in PolarDesc::pad.  The BP kernel is persistent: every
// CTA takes the next item from a global counter until the list is exhausted, so scenes
// of very different sizes share the GPU without per-scene launches or idle tails.  Items
// are independent (no item waits for another), so the persistent grid needs no
// co-residency guarantee.  Merge levels run as one persistent launch per tree height
// over the nodes of that height in every FFBP scene.
namespace {

struct BatchScene {
    SplitParams P;          // pulse inputs, constants, chunk / window capacity; P.out = direct output
    sarbp_lattice lat;      // direct scenes
    int kind;               // 0 direct lattice, 1 FFBP
    int lc;                 // direct: log2 of tile columns
    int pad[2];
    long long prec_offset;  // FFBP: first pulse record of the scene
};

// Completion time of an item for the scene's trace slot (max over the scene's items): the
// GPU's nanosecond global timer, after every thread of the block is done with the item.
__device__ __forceinline__ void trace_item(unsigned long long* trace, int scene) {
    if (!trace) return;  // uniform
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        atomicMax(trace + scene, t);
    }
}

__global__ void batch_trace_start_kernel(unsigned long long* t0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    *t0 = t;
}

__device__ __forceinline__ int next_item(int* counter, int& s_item) {
    __syncthreads();  // every thread is done with the previous item's shared state
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    return s_item;
}

template <int THREADS>
__device__ __forceinline__ void load_scene(const BatchScene* __restrict__ scenes, int scene, BatchScene& sc) {
    const int* src = reinterpret_cast<const int*>(scenes + scene);
    int* dst = reinterpret_cast<int*>(&sc);
    for (int w = threadIdx.x; w < (int)(sizeof(BatchScene) / sizeof(int)); w += THREADS) dst[w] = src[w];
    __syncthreads();
}

// Direct tiles of every direct scene (flat lattices only, checked when the batch is created).
__global__ void __launch_bounds__(kThreads, 4) batch_direct_kernel(const BatchScene* __restrict__ scenes,
                                                                   const TileItem* __restrict__ items, int nitems,
                                                                   int* counter, unsigned long long* trace) {
    extern __shared__ __align__(16) char smem[];
    __shared__ TileShared S;
    __shared__ int s_item, s_scene;
    __shared__ __align__(16) BatchScene sc;
    if (threadIdx.x == 0) s_scene = -1;
    // The leaf tiles of the batch do not depend on these: their kernel may take the SMs that run dry.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (;;) {
        const int idx = next_item(counter, s_item);
        if (idx >= nitems) return;
        const TileItem it = items[idx];
        if (it.pad != s_scene) {  // uniform across the block
            load_scene<kThreads>(scenes, it.pad, sc);
            if (threadIdx.x == 0) s_scene = it.pad;
        }
        lattice_tile(sc.P, sc.lat, sc.lc, it.tile_r, it.tile_u, 0, sc.P.in.pulses, sc.P.out, S, smem);
        trace_item(trace, it.pad);
    }
}

// Leaf tiles of every FFBP scene.
__global__ void __launch_bounds__(kLeafThreads, kLeafCtas) batch_leaf_kernel(const BatchScene* __restrict__ scenes,
                                                                 const PolarDesc* __restrict__ nodes,
                                                                 const TileItem* __restrict__ items, int nitems,
                                                                 const float4* __restrict__ tables,
                                                                 const PulseRec* __restrict__ precs,
                                                                 float2* __restrict__ arena, int* counter,
                                                                 unsigned long long* trace) {
    extern __shared__ __align__(16) char smem[];
    __shared__ int s_base[kMaxLeafChunk];
    __shared__ float s_wt[kMaxLeafChunk];
    __shared__ int s_nfit, s_item, s_scene;
    __shared__ __align__(16) BatchScene sc;
    if (threadIdx.x == 0) s_scene = -1;
    for (;;) {
        const int idx = next_item(counter, s_item);
        if (idx >= nitems) {
            // Started early (launch_split_batch_leaves): whoever waits for this grid waits for the one before, too.
            asm volatile("griddepcontrol.wait;" ::: "memory");
            return;
        }
        const TileItem it = items[idx];
        if (it.pad != s_scene) {
            load_scene<kLeafThreads>(scenes, it.pad, sc);
            if (threadIdx.x == 0) s_scene = it.pad;
        }
        leaf_tile<1>(sc.P, nodes, it, tables, precs + sc.prec_offset, arena, nullptr, -1, smem, s_base, s_wt, s_nfit);
        trace_item(trace, it.pad);
    }
}

__global__ void __launch_bounds__(kMergeThreads, 8) batch_merge_kernel(const BatchScene* __restrict__ scenes,
                                                                  const PolarDesc* __restrict__ nodes,
                                                                  const TileItem* __restrict__ items, int nitems,
                                                                  const float4* __restrict__ tables,
                                                                  const ChildRec* __restrict__ crecs,
                                                                  float2* __restrict__ arena, int* counter,
                                                                  unsigned long long* trace) {
    extern __shared__ __align__(16) char smem[];
    __shared__ MergeChildren C;
    __shared__ int s_item;
    for (;;) {
        const int idx = next_item(counter, s_item);
        if (idx >= nitems) return;
        const TileItem it = items[idx];
        const SplitParams& P = scenes[it.pad].P;
        merge_tile<false>(FF{P.Kh, P.Kl}, nodes, it, tables, crecs + 2 * (long long)idx, C, arena,
                                         nullptr, -1, smem);
        trace_item(trace, it.pad);
    }
}

__global__ void batch_tables_kernel(const BatchScene* __restrict__ scenes, const PolarDesc* __restrict__ nodes,
                                    float4* __restrict__ tables) {
    const PolarDesc& g = nodes[blockIdx.y];
    const SplitParams& P = scenes[g.pad].P;
    table_entries(table_consts(P), g, blockIdx.x * blockDim.x + threadIdx.x, tables);
}

__global__ void batch_leaf_pulses_kernel(const BatchScene* __restrict__ scenes, const PolarDesc* __restrict__ nodes,
                                         const int* __restrict__ leaves, PulseRec* __restrict__ recs) {
    __shared__ int amax[2];
    const PolarDesc& g = nodes[leaves[blockIdx.x]];
    const BatchScene& sc = scenes[g.pad];
    leaf_pulses(sc.P.K, sc.P.in.pos, sc.P.in.weight, sc.P.in.phase, g, recs + sc.prec_offset, amax);
}

__global__ void batch_child_records_kernel(const BatchScene* __restrict__ scenes, const PolarDesc* __restrict__ nodes,
                                           const float4* __restrict__ tables, const TileItem* __restrict__ items,
                                           int n_items, float2* __restrict__ arena, ChildRec* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * n_items) return;
    const TileItem it = items[t >> 1];
    const SplitParams& P = scenes[it.pad].P;
    child_record(FF{P.Kh, P.Kl}, (float)P.scale_w, (float)P.inv_scale_w, nodes, tables, it, t, arena, nullptr, out);
}

}  // namespace

size_t split_batch_scene_bytes() { return sizeof(BatchScene); }

size_t split_batch_pack_scene(const BatchSceneDesc& d, void* dst) {
    BatchScene b{};
    b.P = make_params(d.in, d.chunk,
                      d.kind == 0 ? lattice_capacity(d.chunk, d.window_bins)
                                  : leaf_capacity(d.chunk, d.window_bins),
                      1);
    b.P.out = d.out;
    b.lat = d.lat;
    b.kind = d.kind;
    b.lc = d.lc;
    b.prec_offset = d.prec_offset;
    memcpy(dst, &b, sizeof(b));
    return (d.kind == 0 ? window_offset() + raw_bytes_for(b.P.cap, kMaxChunk) : leaf_window_offset()) +
           (size_t)b.P.cap * 32;
}

int split_batch_occupancy(size_t direct_smem, size_t leaf_smem, int* direct_per_sm, int* leaf_per_sm,
                          int* merge_per_sm) {
    if (int st = prepare(batch_direct_kernel, direct_smem)) return st;
    if (int st = prepare(batch_leaf_kernel, leaf_smem)) return st;
    if (int st = prepare(batch_merge_kernel, merge_smem())) return st;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(direct_per_sm, batch_direct_kernel, kThreads,
                                                                  direct_smem);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(leaf_per_sm, batch_leaf_kernel, kLeafThreads, leaf_smem);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(merge_per_sm, batch_merge_kernel, kMergeThreads, merge_smem());
    if (e != cudaSuccess) return fail(SARBP_ERR_CUDA, "occupancy query: %s", cudaGetErrorString(e));
    return SARBP_OK;
}

int launch_split_batch_prologue(const void* scenes, const PolarDesc* nodes, int n_nodes, int max_dim,
                                const int* leaves, int n_leaves, const TileItem* merge_items, int n_merge_items,
                                float4* tables, void* precs, void* crecs, float2* arena, cudaStream_t s) {
    const BatchScene* sc = reinterpret_cast<const BatchScene*>(scenes);
    if (n_nodes > 0) {
        dim3 grid((max_dim + kThreads - 1) / kThreads, n_nodes);
        batch_tables_kernel<<<grid, kThreads, 0, s>>>(sc, nodes, tables);
        note_launches(1);
        if (int st = check_launch("batch_tables")) return st;
    }
    if (n_leaves > 0) {
        batch_leaf_pulses_kernel<<<n_leaves, 128, 0, s>>>(sc, nodes, leaves, reinterpret_cast<PulseRec*>(precs));
        note_launches(1);
        if (int st = check_launch("batch_leaf_pulses")) return st;
    }
    if (n_merge_items > 0) {
        batch_child_records_kernel<<<grid_blocks(2LL * n_merge_items, kThreads), kThreads, 0, s>>>(
            sc, nodes, tables, merge_items, n_merge_items, arena, reinterpret_cast<ChildRec*>(crecs));
        note_launches(1);
        if (int st = check_launch("batch_child_records")) return st;
    }
    return SARBP_OK;
}

int launch_split_batch_trace_start(unsigned long long* t0, cudaStream_t s) {
    batch_trace_start_kernel<<<1, 1, 0, s>>>(t0);
    note_launches(1);
    return check_launch("batch_trace_start");
}

int launch_split_batch_direct(const void* scenes, const TileItem* items, int nitems, int* counter, int blocks,
                              size_t smem, unsigned long long* trace, cudaStream_t s) {
    if (nitems <= 0) return SARBP_OK;
    if (int st = prepare(batch_direct_kernel, smem)) return st;
    batch_direct_kernel<<<blocks, kThreads, smem, s>>>(reinterpret_cast<const BatchScene*>(scenes), items, nitems,
                                                       counter, trace);
    note_launches(1);
    return check_launch("batch_direct");
}

int launch_split_batch_leaves(const void* scenes, const PolarDesc* nodes, const TileItem* items, int nitems,
                              const float4* tables, const void* precs, float2* arena, int* counter, int blocks,
                              size_t smem, unsigned long long* trace, bool after_direct, cudaStream_t s) {
    if (nitems <= 0) return SARBP_OK;
    if (int st = prepare(batch_leaf_kernel, smem)) return st;
    // Behind the direct tiles on the same stream the leaves may start while the last of those run: the direct
    // tiles' pulses differ from scene to scene, so that blocks run dry over a quarter of the launch (24 scenes of
    // 128 to 384 pixels a side, 256 to 640 pulses: 0.853 -> 0.799 ms).
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(kLeafThreads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &early;
    c.numAttrs = after_direct ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&c, batch_leaf_kernel, reinterpret_cast<const BatchScene*>(scenes), nodes,
                                             items, nitems, tables, reinterpret_cast<const PulseRec*>(precs), arena,
                                             counter, trace);
    if (e != cudaSuccess) return fail(SARBP_ERR_CUDA, "batch_leaves: %s", cudaGetErrorString(e));
    note_launches(1);
    return check_launch("batch_leaves");
}

int launch_split_batch_merges(const void* scenes, const PolarDesc* nodes, const TileItem* items, int nitems,
                              const float4* tables, const void* crecs, float2* arena, int* counter, int blocks,
                              unsigned long long* trace, cudaStream_t s) {
    if (nitems <= 0) return SARBP_OK;
    if (int st = prepare(batch_merge_kernel, merge_smem())) return st;
    batch_merge_kernel<<<blocks, kMergeThreads, merge_smem(), s>>>(reinterpret_cast<const BatchScene*>(scenes), nodes,
                                                              items, nitems, tables,
                                                              reinterpret_cast<const ChildRec*>(crecs), arena,
                                                              counter, trace);
    note_launches(1);
    return check_launch("batch_merges");
}

int launch_split_evaluate_lattice(const float2* image, const PolarDesc& grid, const sarbp_lattice& lattice, double k,
                                  float2* out, cudaStream_t s) {
    PulseInputs none{};
    none.k = k;
    none.data_dr = 1.0;
    const SplitParams P = make_params(none, 1, 4, 1);
    sarbp_lattice flat = lattice;  // ground points: z is not used
    flat.origin[2] = flat.step_row[2] = flat.step_col[2] = 0.0;
    const int lc = 5;
    const auto two = [](double v) {
        const float h = (float)v;
        return FF{h, (float)(v - (double)h)};
    };
    double most = 0.0;
    for (int c = 0; c < 2; ++c)
        most = fmax(most, 0.5 * ((kSplitTilePixels >> lc) * fabs(lattice.step_row[c]) + (1 << lc) * fabs(lattice.step_col[c])));
    int e;
    frexp(most * 1.0001 + 1e-6, &e);
    const LatticeSteps L{two(lattice.step_row[0]), two(lattice.step_row[1]), two(lattice.step_col[0]),
                         two(lattice.step_col[1]), ldexpf(1.0f, e - 12),     ldexpf(1.0f, 12 - e)};
    split_evaluate_lattice_kernel<<<tiles_of(lattice.rows, lattice.cols, lc), kThreads, 0, s>>>(
        P.Kh, P.Kl, (float)P.scale_w, (float)P.inv_scale_w, grid, image, flat, L, lc, out);
    note_launches(1);
    return check_launch("split_evaluate_lattice");
}

}  // namespace sarbp
