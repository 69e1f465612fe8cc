// Range compression: the FFT matched filter that turns raw LFM echoes into the
// range-compressed pulses the back-projection kernels consume (sar_io.range_compress,
// fast_bp/sar_io.py:116-139).  The FFTs are library calls (cuFFT through the host);
// these kernels are the memory-bound steps around them:
//   rc_prepare  - remove each pulse's mean and zero-pad it to the FFT length,
//   rc_filter   - multiply by the filter response and, when oversampling, place the
//                 product in the longer spectrum (Fourier interpolation with the
//                 Nyquist bin split in half, as scipy.signal.resample does),
//   rc_crop     - cut the exact-lag window out of the correlation and scale it.
// Each is one pass over its data: grid-stride loops, coalesced complex64 accesses.
// Without oversampling the whole chain is one kernel of its own (rc_blocks_kernel): the result is
// a linear correlation, which overlap-save blocks in shared memory form in one pass over the pulses.
// decode_iq turns raw capture frames (int16 I/Q after a header) into complex64 pulses.
#include "common.cuh"

namespace sarbp {
namespace {

constexpr int kRowThreads = 256;

// One block per pulse: the row's mean (FP32 partial sums per thread, FP64 across threads),
// then the centred, zero-padded row.  Rows are read as float4 pairs when 16-byte aligned.
__global__ void rc_prepare_kernel(const float2* __restrict__ raw, int samples, int nfft, float2* __restrict__ out) {
    const int row = blockIdx.x;
    const float2* x = raw + (size_t)row * samples;
    float pr = 0.0f, pi = 0.0f;
    const bool vec = ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const int pairs = vec ? samples / 2 : 0;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    for (int j = threadIdx.x; j < pairs; j += kRowThreads) {
        const float4 v = x4[j];
        pr += v.x + v.z;
        pi += v.y + v.w;
    }
    for (int j = 2 * pairs + threadIdx.x; j < samples; j += kRowThreads) {
        const float2 v = x[j];
        pr += v.x;
        pi += v.y;
    }
    double sr = pr, si = pi;
    __shared__ double red[2][kRowThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        red[0][warp] = sr;
        red[1][warp] = si;
    }
    __syncthreads();
    double tr = 0.0, ti = 0.0;
    for (int w = 0; w < kRowThreads / 32; ++w) {
        tr += red[0][w];
        ti += red[1][w];
    }
    const float mr = (float)(tr / samples), mi = (float)(ti / samples);  // complex64 mean, as the reference
    float2* y = out + (size_t)row * nfft;
    for (int j = threadIdx.x; j < nfft; j += kRowThreads) {
        float2 v = make_float2(0.0f, 0.0f);
        if (j < samples) {
            const float2 a = x[j];
            v = make_float2(a.x - mr, a.y - mi);
        }
        y[j] = v;
    }
}

// The same computation with the row held in registers between the mean and the write (one HBM
// read instead of two): P float4 (two samples each) per thread, rows of an even number of up to
// 2 * 256 * P samples starting on a 16-byte boundary.  Partial sums, their order and the FP64
// reduction are those of rc_prepare_kernel, so the output is bit-identical.
template <int P>
__global__ void __launch_bounds__(kRowThreads) rc_prepare_reg_kernel(const float2* __restrict__ raw, int samples,
                                                                     int nfft, float2* __restrict__ out) {
    const int row = blockIdx.x;
    const float2* x = raw + (size_t)row * samples;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const int pairs = samples / 2;
    float4 v[P];
    float pr = 0.0f, pi = 0.0f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int j = threadIdx.x + kRowThreads * i;
        v[i] = j < pairs ? x4[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < pairs) {
            pr += v[i].x + v[i].z;
            pi += v[i].y + v[i].w;
        }
    }
    double sr = pr, si = pi;
    __shared__ double red[2][kRowThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        red[0][warp] = sr;
        red[1][warp] = si;
    }
    __syncthreads();
    double tr = 0.0, ti = 0.0;
    for (int w = 0; w < kRowThreads / 32; ++w) {
        tr += red[0][w];
        ti += red[1][w];
    }
    const float mr = (float)(tr / samples), mi = (float)(ti / samples);  // complex64 mean, as the reference
    float2* y = out + (size_t)row * nfft;
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int j = threadIdx.x + kRowThreads * i;
        if (j < pairs) {
            y[2 * j] = make_float2(v[i].x - mr, v[i].y - mi);
            y[2 * j + 1] = make_float2(v[i].z - mr, v[i].w - mi);
        }
    }
    for (int j = samples + threadIdx.x; j < nfft; j += kRowThreads) y[j] = make_float2(0.0f, 0.0f);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// out[p, m] for m in [0, length): length == nfft multiplies in place order; a longer
// length places bins [0, nfft/2] at the front and the negative frequencies at the back,
// halving the positive Nyquist bin and copying it to the negative one (even nfft).
// spec and out may be the same array (length == nfft): no __restrict__ on either.
__global__ void rc_filter_kernel(const float2* spec, const float2* __restrict__ response, int pulses, int nfft,
                                 int length, float2* out) {
    const long long total = (long long)pulses * length;
    const int half = nfft / 2, nyq = nfft / 2 + 1;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(t / length);
        const int m = (int)(t - (long long)p * length);
        const float2* s = spec + (size_t)p * nfft;
        float2 v = make_float2(0.0f, 0.0f);
        if (length == nfft) {
            v = cmul(s[m], response[m]);
        } else if (m < nyq) {
            v = cmul(s[m], response[m]);
            if ((nfft & 1) == 0 && m == half) v = make_float2(0.5f * v.x, 0.5f * v.y);
        } else if (m >= length - (nfft - nyq)) {
            const int k = m - length + nfft;  // negative frequency bin of the short spectrum
            v = cmul(s[k], response[k]);
        } else if ((nfft & 1) == 0 && m == length - half) {
            v = cmul(s[half], response[half]);
            v = make_float2(0.5f * v.x, 0.5f * v.y);
        }
        out[t] = v;
    }
}

// Row-per-blockIdx.y forms of the filter and the crop: column index from the x grid, no 64-bit
// division per element (grids with up to 65535 rows).
__global__ void rc_filter_rows_kernel(const float2* spec, const float2* __restrict__ response, int nfft, int length,
                                      float2* out) {
    const int p = blockIdx.y;
    const int half = nfft / 2, nyq = nfft / 2 + 1;
    const float2* s = spec + (size_t)p * nfft;
    float2* o = out + (size_t)p * length;
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < length; m += gridDim.x * blockDim.x) {
        float2 v = make_float2(0.0f, 0.0f);
        if (length == nfft) {
            v = cmul(s[m], response[m]);
        } else if (m < nyq) {
            v = cmul(s[m], response[m]);
            if ((nfft & 1) == 0 && m == half) v = make_float2(0.5f * v.x, 0.5f * v.y);
        } else if (m >= length - (nfft - nyq)) {
            const int k = m - length + nfft;  // negative frequency bin of the short spectrum
            v = cmul(s[k], response[k]);
        } else if ((nfft & 1) == 0 && m == length - half) {
            v = cmul(s[half], response[half]);
            v = make_float2(0.5f * v.x, 0.5f * v.y);
        }
        o[m] = v;
    }
}

__global__ void rc_crop_rows_kernel(const float2* __restrict__ corr, int length, int offset, int samples, float scale,
                                    float2* __restrict__ out) {
    const int p = blockIdx.y;
    const float2* c = corr + (size_t)p * length + offset;
    float2* o = out + (size_t)p * samples;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < samples; j += gridDim.x * blockDim.x) {
        const float2 v = c[j];
        o[j] = make_float2(v.x * scale, v.y * scale);
    }
}

// Columns per block of the row kernels: enough blocks for every SM, a few columns per thread.
dim3 row_grid(int rows, int cols) {
    int bx = (cols + 4 * kRowThreads - 1) / (4 * kRowThreads);
    return dim3(bx > 0 ? bx : 1, rows);
}

__global__ void rc_crop_kernel(const float2* __restrict__ corr, int pulses, int length, int offset, int samples,
                               float scale, float2* __restrict__ out) {
    const long long total = (long long)pulses * samples;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(t / samples);
        const int j = (int)(t - (long long)p * samples);
        const float2 v = corr[(size_t)p * length + offset + j];
        out[t] = make_float2(v.x * scale, v.y * scale);
    }
}

// Raw frames -> complex64: frame i's I/Q pairs start iq_offset bytes into the frame.
__global__ void decode_iq_kernel(const unsigned char* __restrict__ frames, int n, long long frame_size, int iq_offset,
                                 int nr, float2* __restrict__ out) {
    const long long total = (long long)n * nr;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long i = t / nr, j = t - i * nr;
        const short2 v = *reinterpret_cast<const short2*>(frames + i * frame_size + iq_offset + 4 * j);
        out[t] = make_float2((float)v.x, (float)v.y);
    }
}

__global__ void decode_iq_rows_kernel(const unsigned char* __restrict__ frames, long long frame_size, int iq_offset,
                                      int nr, float2* __restrict__ out) {
    const long long i = blockIdx.y;
    const unsigned char* f = frames + i * frame_size + iq_offset;
    float2* o = out + i * nr;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nr; j += gridDim.x * blockDim.x) {
        const short2 v = *reinterpret_cast<const short2*>(f + 4 * (long long)j);
        o[j] = make_float2((float)v.x, (float)v.y);
    }
}

// ---- the whole matched filter in one pass (no oversampling) ------------------------------------
//
// A block of threads holds one pulse in shared memory (one HBM read), takes its mean off and correlates
// it with the n-tap filter by overlap-save: transforms of kBlockFft samples in registers and shared
// memory, of which each gives kBlockFft - n + 1 outputs.  Two groups of 128 threads transform different
// blocks of the pulse; a thread holds 16 samples.  The length is 16 x 16 x 8: the forward transform
// decimates in frequency, the inverse in time, so the spectrum is never reordered, and a thread's 30
// twiddle factors stay in its registers for every block and pulse (persistent blocks over the pulses).
// The shared-memory layouts between the passes are padded so that every access takes the two wavefronts
// that 32 complex values need.  Bound: instruction issue and the barriers between the passes at 16 warps
// per SM (the HBM floor of 4096 pulses of 8192 samples is 79 us).  Those take 234 us; the five passes
// (prepare, cuFFT, filter, inverse cuFFT, crop over 8640 points) took 800 us, with an error against
// FP64 of 1.6e-7 instead of 3.8e-7.
constexpr int kBlockFft = 2048;
constexpr int kBlockGroup = 128, kBlockGroups = 2;
constexpr int kBlockThreads = kBlockGroup * kBlockGroups;
constexpr int kPadA = kBlockGroup + 8;         // row stride of the (k1, t) layout
constexpr int kPadB = kBlockFft / 8 + 4;       // row stride of the (t2, k2, k1) layout
constexpr int kBlockWork = 16 * kPadA;         // complex values of a group's exchange buffer
static_assert(8 * kPadB <= kBlockWork, "both layouts fit the exchange buffer");

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * b, or a * conj(b).
template <bool CONJ>
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
    return CONJ ? make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -(a.x * b.y)))
                : make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.y, b.x, a.x * b.y));
}
// a * (-i) forward, a * i inverse.
template <bool INV>
__device__ __forceinline__ float2 crot(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
    const float2 s0 = cadd(a, c), d0 = csub(a, c), s1 = cadd(b, d), d1 = crot<INV>(csub(b, d));
    a = cadd(s0, s1);
    b = cadd(d0, d1);
    c = csub(s0, s1);
    d = csub(d0, d1);
}

// Natural order in and out.
template <bool INV>
__device__ __forceinline__ void dft16(float2 v[16]) {
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
#pragma unroll
    for (int b = 0; b < 4; ++b) dft4<INV>(v[b], v[4 + b], v[8 + b], v[12 + b]);  // v[4 k + b]: k-th of column b
    const float2 w1 = make_float2(c1, -s1), w2 = make_float2(h, -h), w3 = make_float2(s1, -c1);
    v[5] = cmulc<INV>(v[5], w1);
    v[6] = cmulc<INV>(v[6], w2);
    v[7] = cmulc<INV>(v[7], w3);
    v[9] = cmulc<INV>(v[9], w2);
    v[10] = crot<INV>(v[10]);
    v[11] = cmulc<INV>(v[11], make_float2(-h, -h));
    v[13] = cmulc<INV>(v[13], w3);
    v[14] = cmulc<INV>(v[14], make_float2(-h, -h));
    v[15] = cmulc<INV>(v[15], make_float2(-c1, s1));
#pragma unroll
    for (int k = 0; k < 4; ++k) dft4<INV>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    // v[4 k + m] is output k + 4 m: transpose.
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int m = k + 1; m < 4; ++m) {
            const float2 t = v[4 * k + m];
            v[4 * k + m] = v[4 * m + k];
            v[4 * m + k] = t;
        }
}

// v[0..7] in place, natural order.
template <bool INV>
__device__ __forceinline__ void dft8(float2 v[8]) {
    const float h = 0.70710678118654752440f;
    dft4<INV>(v[0], v[2], v[4], v[6]);
    dft4<INV>(v[1], v[3], v[5], v[7]);
    const float2 e[4] = {v[0], v[2], v[4], v[6]};
    const float2 o[4] = {v[1], cmulc<INV>(v[3], make_float2(h, -h)), crot<INV>(v[5]),
                         cmulc<INV>(v[7], make_float2(-h, -h))};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = cadd(e[k], o[k]);
        v[k + 4] = csub(e[k], o[k]);
    }
}

__device__ __forceinline__ void group_sync(int group) {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kBlockGroup) : "memory");
}

// s + v as an unevaluated sum (s, e): Knuth's two-sum with the running error.
__device__ __forceinline__ void sum_into(float& s, float& e, float v, float ve) {
    const float t = s + v, b = t - s;
    e += ((s - (t - b)) + (v - b)) + ve;
    s = t;
}

// (s + e) / n, rounded once (but for ties); inv: 1 / n.
__device__ __forceinline__ float mean_of(float s, float e, float n, float inv) {
    const float q = s * inv;
    return fmaf(fmaf(-q, n, s) + e, inv, q);
}

// out[p, k] = sum_m h[m] (x - mean x)[k + taps - 1 - taps / 2 - m]; response: the taps' transform of
// kBlockFft points divided by kBlockFft; inv: 1 / samples.
__global__ void __launch_bounds__(kBlockThreads, 2) rc_blocks_kernel(const float2* __restrict__ raw, int pulses,
                                                                     int samples, int taps, float inv,
                                                                     const float2* __restrict__ response,
                                                                     float2* __restrict__ out) {
    extern __shared__ __align__(16) float2 sm[];
    __shared__ float4 part[kBlockThreads / 32];
    float2* work = sm + (threadIdx.x / kBlockGroup) * kBlockWork;
    float2* x = sm + kBlockGroups * kBlockWork;  // the pulse
    const int group = threadIdx.x / kBlockGroup, t = threadIdx.x % kBlockGroup;
    const int k1 = t >> 3, t2 = t & 7;
    float2 tw1[16], tw2[16];  // exp(-2 pi i t k / 2048), exp(-2 pi i t2 k / 128)
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        sincospif((float)(t * k) * (2.0f / kBlockFft), &tw1[k].y, &tw1[k].x);
        sincospif((float)(t2 * k) * (2.0f / 128.0f), &tw2[k].y, &tw2[k].x);
        tw1[k].y = -tw1[k].y;
        tw2[k].y = -tw2[k].y;
    }
    const int step = kBlockFft - taps + 1, nblocks = (samples + step - 1) / step;
    for (int p = blockIdx.x; p < pulses; p += gridDim.x) {
        const float2* row = raw + (size_t)p * samples;
        // The pulse into shared memory, and its mean: FP32 per thread, then two-float sums.
        float sr = 0.0f, si = 0.0f;
        const int head = (int)((reinterpret_cast<uintptr_t>(row) >> 3) & 1);  // 16-byte loads from here on
        const int pairs = (samples - head) >> 1;
        const float4* r4 = reinterpret_cast<const float4*>(row + head);
#pragma unroll 8
        for (int j = threadIdx.x; j < pairs; j += kBlockThreads) {
            const float4 v = __ldg(r4 + j);
            x[head + 2 * j] = make_float2(v.x, v.y);
            x[head + 2 * j + 1] = make_float2(v.z, v.w);
            sr += v.x + v.z;
            si += v.y + v.w;
        }
        if (threadIdx.x < 2) {  // the samples before and after the pairs
            const int j = threadIdx.x ? samples - 1 : 0;
            if (threadIdx.x ? head + 2 * pairs < samples : head != 0) {
                const float2 v = __ldg(row + j);
                x[j] = v;
                sr += v.x;
                si += v.y;
            }
        }
        float er = 0.0f, ei = 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float vr = __shfl_xor_sync(0xffffffffu, sr, o), wr = __shfl_xor_sync(0xffffffffu, er, o);
            const float vi = __shfl_xor_sync(0xffffffffu, si, o), wi = __shfl_xor_sync(0xffffffffu, ei, o);
            sum_into(sr, er, vr, wr);
            sum_into(si, ei, vi, wi);
        }
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = make_float4(sr, er, si, ei);
        __syncthreads();
        sr = er = si = ei = 0.0f;
#pragma unroll
        for (int w = 0; w < kBlockThreads / 32; ++w) {
            const float4 v = part[w];
            sum_into(sr, er, v.x, v.y);
            sum_into(si, ei, v.z, v.w);
        }
        // complex64, as the reference: the two-float sums divided with the remainder (a sum rounded first would
        // put every second mean of a large offset a last bit off).
        const float count = (float)samples;
        const float mr = mean_of(sr, er, count, inv), mi = mean_of(si, ei, count, inv);
        for (int b = group; b < nblocks; b += kBlockGroups) {
            const int k0 = b * step, first = k0 - taps / 2;  // the block's first output and input sample
            float2 v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int i = first + t + kBlockGroup * j;
                v[j] = make_float2(0.0f, 0.0f);
                if (i >= 0 && i < samples) v[j] = make_float2(x[i].x - mr, x[i].y - mi);
            }
            dft16<false>(v);
#pragma unroll
            for (int k = 0; k < 16; ++k) work[k * kPadA + t] = k ? cmulc<false>(v[k], tw1[k]) : v[k];
            group_sync(group);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = work[k1 * kPadA + t2 + 8 * j];
            dft16<false>(v);
            group_sync(group);
#pragma unroll
            for (int k = 0; k < 16; ++k) work[t2 * kPadB + 16 * k + k1] = k ? cmulc<false>(v[k], tw2[k]) : v[k];
            group_sync(group);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int q = t + kBlockGroup * h;
                float2 u[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) u[j] = work[j * kPadB + q];
                dft8<false>(u);
#pragma unroll
                for (int k = 0; k < 8; ++k) u[k] = cmulc<false>(u[k], __ldg(response + q + 256 * k));
                dft8<true>(u);
#pragma unroll
                for (int j = 0; j < 8; ++j) work[j * kPadB + q] = u[j];  // the places it was read from
            }
            group_sync(group);
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                v[k] = work[t2 * kPadB + 16 * k + k1];
                if (k) v[k] = cmulc<true>(v[k], tw2[k]);
            }
            dft16<true>(v);
            group_sync(group);
#pragma unroll
            for (int j = 0; j < 16; ++j) work[k1 * kPadA + t2 + 8 * j] = v[j];
            group_sync(group);
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                v[k] = work[k * kPadA + t];
                if (k) v[k] = cmulc<true>(v[k], tw1[k]);
            }
            dft16<true>(v);
            float2* o = out + (size_t)p * samples;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int i = t + kBlockGroup * j - (taps - 1), k = k0 + i;
                if (i >= 0 && k < samples) o[k] = v[j];
            }
            group_sync(group);  // the next block's first exchange
        }
        __syncthreads();  // the next pulse replaces this one
    }
}

size_t blocks_smem(int samples) { return (size_t)(kBlockGroups * kBlockWork + samples) * sizeof(float2); }

int stream_grid(long long n) {
    int dev = 0, sms = 152;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long blocks = (n + kRowThreads - 1) / kRowThreads;
    return (int)(blocks < 8LL * sms ? (blocks > 0 ? blocks : 1) : 8LL * sms);
}

}  // namespace

int launch_rc_prepare(const float2* raw, int pulses, int samples, int nfft, float2* out, cudaStream_t s) {
    const long long pairs = samples / 2;
    const bool aligned = (reinterpret_cast<uintptr_t>(raw) & 15) == 0 && (samples & 1) == 0;
    if (aligned && pairs <= 4LL * kRowThreads)
        rc_prepare_reg_kernel<4><<<pulses, kRowThreads, 0, s>>>(raw, samples, nfft, out);
    else if (aligned && pairs <= 8LL * kRowThreads)
        rc_prepare_reg_kernel<8><<<pulses, kRowThreads, 0, s>>>(raw, samples, nfft, out);
    else if (aligned && pairs <= 16LL * kRowThreads)
        rc_prepare_reg_kernel<16><<<pulses, kRowThreads, 0, s>>>(raw, samples, nfft, out);
    else
        rc_prepare_kernel<<<pulses, kRowThreads, 0, s>>>(raw, samples, nfft, out);
    note_launches(1);
    return check_launch("rc_prepare");
}

int rc_blocks_points() { return kBlockFft; }

// The pulse and the exchange buffers fit a block's shared memory, and at least half of every transform
// is output.
bool rc_blocks_fit(int samples, int taps) {
    return samples >= 1 && taps >= 1 && taps <= kBlockFft / 2 + 1 && samples <= 24576 && blocks_smem(samples) <= 227 * 1024;
}

int launch_rc_blocks(const float2* raw, int pulses, int samples, int taps, const float2* response, float2* out,
                     cudaStream_t s) {
    const size_t smem = blocks_smem(samples);
    if (int st = allow_shared(reinterpret_cast<const void*>(rc_blocks_kernel), smem)) return st;
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rc_blocks_kernel, kBlockThreads, smem);
    if (e != cudaSuccess || per_sm < 1) return fail(SARBP_ERR_CUDA, "rc_blocks: %s", cudaGetErrorString(e));
    const long long slots = (long long)sms * per_sm;
    rc_blocks_kernel<<<(int)(pulses < slots ? pulses : slots), kBlockThreads, smem, s>>>(
        raw, pulses, samples, taps, 1.0f / (float)samples, response, out);
    note_launches(1);
    return check_launch("rc_blocks");
}

int launch_rc_filter(const float2* spec, const float2* response, int pulses, int nfft, int length, float2* out,
                     cudaStream_t s) {
    if (pulses <= 65535)
        rc_filter_rows_kernel<<<row_grid(pulses, length), kRowThreads, 0, s>>>(spec, response, nfft, length, out);
    else
        rc_filter_kernel<<<stream_grid((long long)pulses * length), kRowThreads, 0, s>>>(spec, response, pulses, nfft,
                                                                                        length, out);
    note_launches(1);
    return check_launch("rc_filter");
}

int launch_decode_iq(const unsigned char* frames, int n, long long frame_size, int iq_offset, int nr, float2* out,
                     cudaStream_t s) {
    if (n <= 65535)
        decode_iq_rows_kernel<<<row_grid(n, nr), kRowThreads, 0, s>>>(frames, frame_size, iq_offset, nr, out);
    else
        decode_iq_kernel<<<stream_grid((long long)n * nr), kRowThreads, 0, s>>>(frames, n, frame_size, iq_offset, nr,
                                                                               out);
    note_launches(1);
    return check_launch("decode_iq");
}

int launch_rc_crop(const float2* corr, int pulses, int length, int offset, int samples, float scale, float2* out,
                   cudaStream_t s) {
    if (pulses <= 65535)
        rc_crop_rows_kernel<<<row_grid(pulses, samples), kRowThreads, 0, s>>>(corr, length, offset, samples, scale,
                                                                               out);
    else
        rc_crop_kernel<<<stream_grid((long long)pulses * samples), kRowThreads, 0, s>>>(corr, pulses, length, offset,
                                                                                       samples, scale, out);
    note_launches(1);
    return check_launch("rc_crop");
}

}  // namespace sarbp
