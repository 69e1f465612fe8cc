// Trajectory update of the phase-gradient autofocus (fast_bp/autofocus.py:40-79) from the smoothed target
// histories: per pulse, the phase gradients of all targets give a horizontal velocity error by
// robust weighted least squares; the velocity errors are summed to positions, detrended and smoothed.
//
// FP64 throughout.  An FP64 instruction occupies a GB300 sub-partition for 64 cycles, so what is not
// arithmetic stays off that unit: medians rank the values' bit patterns as integers, sums over
// targets are one warp per sum, and nothing is formed twice.  144 targets x 2048 pulses: 0.21 ms in six
// launches (the pulses 0.12), 2.3 ms as some 80 tensor operations and four reads by the host.
//
//   pga_targets_kernel  per target: power, coherence
//   pga_weights_kernel  one block: the targets' weight factors, the median coherence
//   pga_pulses_kernel   one block per pulse: gradients, three reweighted solutions
//   pga_track_kernel    one block: running sums, least-squares line taken off
//   pga_smooth_kernel   Savitzky-Golay smoothing by rows of the projection matrix
//   pga_finish_kernel   one block: limit to 1 m, statistics
#include "common.cuh"

namespace sarbp {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxTargets = 1024;

__device__ __forceinline__ double shfl_add(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the block (every thread gets it); part: 33 doubles of shared memory.  One warp adds the warps'
// sums: every warp doing so would cost as many FP64 instructions again as it has warps.
__device__ __forceinline__ double block_add(double v, double* part) {
    v = shfl_add(v);
    __syncthreads();  // the last sum is read
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        const double s = shfl_add(threadIdx.x < blockDim.x / 32 ? part[threadIdx.x] : 0.0);
        if (threadIdx.x == 0) part[32] = s;
    }
    __syncthreads();
    return part[32];
}

// cross = a conj(b)
__device__ __forceinline__ double2 cross_of(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -(a.x * b.y)));
}

__global__ void __launch_bounds__(kThreads) pga_targets_kernel(const double2* __restrict__ smooth, int pulses,
                                                               double* __restrict__ power,
                                                               double* __restrict__ coherence) {
    __shared__ double part[33];
    const double2* s = smooth + (size_t)blockIdx.x * pulses;
    double amp = 0.0, cr = 0.0, ci = 0.0;
    for (int n = threadIdx.x; n < pulses - 1; n += kThreads) {
        const double2 c = cross_of(s[n + 1], s[n]);
        amp += sqrt(fma(c.x, c.x, c.y * c.y));
        cr += c.x;
        ci += c.y;
    }
    amp = block_add(amp, part);
    cr = block_add(cr, part);
    ci = block_add(ci, part);
    if (threadIdx.x == 0) {
        power[blockIdx.x] = amp / (double)(pulses - 1);
        coherence[blockIdx.x] = sqrt(fma(cr, cr, ci * ci)) / amp;
    }
}

// No number, of either sign (the GPU's own has the sign bit set), by integer operations.
__device__ __forceinline__ bool no_number(long long bits) { return ((unsigned long long)bits << 1) > 0xffe0000000000000ull; }

// Order of doubles as signed integers, what is no number above everything.
__device__ __forceinline__ long long order_bits(double v) {
    const long long b = __double_as_longlong(v);
    return no_number(b) ? 0x7fffffffffffffffll : b ^ ((b >> 63) & 0x7fffffffffffffffll);
}

// numpy's median of v[0 .. n) (the two middle values' mean for even n): the values by rank, ties by index.
// One value per thread; mid: two doubles of shared memory.  keys: n of shared memory.
__device__ __forceinline__ double block_median(double v, int n, long long* keys, double* mid) {
    const int t = threadIdx.x;
    __syncthreads();
    if (t < n) keys[t] = order_bits(v);
    __syncthreads();
    if (t < n) {
        const long long k = order_bits(v);
        int rank = 0;
        for (int j = 0; j < n; ++j) rank += keys[j] < k || (keys[j] == k && j < t);
        if (rank == n / 2) mid[1] = v;
        if (rank == (n - 1) / 2) mid[0] = v;
    }
    __syncthreads();
    return n & 1 ? mid[1] : (mid[0] + mid[1]) / 2.0;
}

// scale[t] and factor: w = min(amp scale, 4) with scale = strength coherence^2 / (power + 1e-12).
__global__ void __launch_bounds__(kMaxTargets) pga_weights_kernel(const double* __restrict__ power,
                                                                  const double* __restrict__ coherence, int targets,
                                                                  double* __restrict__ scale,
                                                                  double* __restrict__ stats) {
    __shared__ long long keys[kMaxTargets];
    __shared__ double mid[2];
    const int t = threadIdx.x;
    const double p = t < targets ? power[t] : 0.0, c = t < targets ? coherence[t] : 0.0;
    const double median = block_median(p, targets, keys, mid);
    if (t < targets) {
        double strength = sqrt(p / median);
        if (strength > 3.0) strength = 3.0;
        double cc = c;  // clamped to [0, 1]; no number stays none
        if (cc < 0.0) cc = 0.0;
        if (cc > 1.0) cc = 1.0;
        scale[t] = strength / (p + 1e-12) * (cc * cc);
    }
    const double mc = block_median(c, targets, keys, mid);
    if (t == 0) stats[0] = mc;
}

// One block per pulse n = blockIdx.x + 1; blockDim.x >= targets.
__global__ void pga_pulses_kernel(const double2* __restrict__ smooth, int targets, int pulses,
                                  const double* __restrict__ pos, const double* __restrict__ xyz, double inv_k,
                                  const double* __restrict__ scale, double2* __restrict__ rate) {
    extern __shared__ double sm[];
    double* terms = sm;                                              // [5][blockDim.x]
    long long* keys = reinterpret_cast<long long*>(sm + 5 * blockDim.x);
    __shared__ double sums[5], mid[2], sol[2];
    const int n = blockIdx.x + 1, t = threadIdx.x, warp = t >> 5, lane = t & 31;
    double w = 0.0, ux = 0.0, uy = 0.0, rhs = 0.0;
    if (t < targets) {
        const double2* s = smooth + (size_t)t * pulses + n;
        const double2 c = cross_of(s[0], s[-1]);
        w = sqrt(fma(c.x, c.x, c.y * c.y)) * scale[t];
        if (w > 4.0) w = 4.0;
        rhs = atan2(c.y, c.x) * inv_k;
        const double vx = xyz[3 * t] - pos[3 * n], vy = xyz[3 * t + 1] - pos[3 * n + 1],
                     vz = xyz[3 * t + 2] - pos[3 * n + 2];
        const double inv = 1.0 / sqrt(fma(vx, vx, fma(vy, vy, vz * vz)));
        ux = vx * inv;
        uy = vy * inv;
    }
    const int warps = blockDim.x >> 5;
    for (int it = 0; it < 3; ++it) {
        const double wx = w * ux, wy = w * uy;
        terms[t] = wx * ux;
        terms[blockDim.x + t] = wx * uy;
        terms[2 * blockDim.x + t] = wy * uy;
        terms[3 * blockDim.x + t] = wx * rhs;
        terms[4 * blockDim.x + t] = wy * rhs;
        __syncthreads();
        for (int v = warp; v < 5; v += warps) {
            double s = 0.0;
            for (int j = lane; j < targets; j += 32) s += terms[v * blockDim.x + j];
            s = shfl_add(s);
            if (lane == 0) sums[v] = s;
        }
        __syncthreads();
        if (t == 0) {
            const double a = sums[0], b = sums[1], d = sums[2], ex = sums[3], ey = sums[4];
            const double reg = 0.002 * (a + d), ar = a + reg, dr = d + reg;
            double det = fma(ar, dr, -(b * b));
            if (det < 1e-12) det = 1e-12;
            sol[0] = fma(ex, dr, -(ey * b)) / det;
            sol[1] = fma(ey, ar, -(ex * b)) / det;
        }
        __syncthreads();
        if (it == 2) break;
        const double res = fabs(rhs - ux * sol[0] - uy * sol[1]);
        const double spread = fma(1.4826, block_median(res, targets, keys, mid), 1e-6);
        double f = 2.5 * spread / (res + 1e-12);
        if (f > 1.0) f = 1.0;
        w *= f;
    }
    if (t == 0) rate[n - 1] = make_double2(sol[0], sol[1]);
}

// Positions by running sums of the rates (0 at the first pulse), least-squares line taken off.
constexpr int kTrackThreads = 256;

__global__ void __launch_bounds__(kTrackThreads) pga_track_kernel(const double2* __restrict__ rate, int pulses,
                                                                  double2* __restrict__ xy) {
    __shared__ double part[33];
    __shared__ double2 ends[kTrackThreads];
    const int t = threadIdx.x, per = (pulses + kTrackThreads - 1) / kTrackThreads;
    const int b = min(pulses, t * per), e = min(pulses, b + per);
    double2 s = make_double2(0.0, 0.0);
    for (int n = b; n < e; ++n) {
        if (n > 0) {
            s.x += rate[n - 1].x;
            s.y += rate[n - 1].y;
        }
        xy[n] = s;
    }
    ends[t] = s;
    __syncthreads();
    for (int o = 1; o < kTrackThreads; o <<= 1) {  // inclusive sums of the stretches
        double2 v = ends[t];
        if (t >= o) {
            v.x += ends[t - o].x;
            v.y += ends[t - o].y;
        }
        __syncthreads();
        ends[t] = v;
        __syncthreads();
    }
    const double2 before = t > 0 ? ends[t - 1] : make_double2(0.0, 0.0);
    const double mid = 0.5 * (double)(pulses - 1);
    double sx = 0.0, sy = 0.0;
    for (int n = b; n < e; ++n) {
        xy[n].x += before.x;
        xy[n].y += before.y;
        sx += xy[n].x;
        sy += xy[n].y;
    }
    sx = block_add(sx, part) / (double)pulses;
    sy = block_add(sy, part) / (double)pulses;
    double tx = 0.0, ty = 0.0, tt = 0.0;
    for (int n = b; n < e; ++n) {
        const double u = (double)n - mid;
        tx = fma(u, xy[n].x - sx, tx);
        ty = fma(u, xy[n].y - sy, ty);
        tt = fma(u, u, tt);
    }
    tx = block_add(tx, part);
    ty = block_add(ty, part);
    tt = block_add(tt, part);
    tx /= tt;
    ty /= tt;
    for (int n = b; n < e; ++n) {
        const double u = (double)n - mid;
        xy[n] = make_double2(xy[n].x - sx - u * tx, xy[n].y - sy - u * ty);
    }
}

// out[n] = row . xy[window of n]: the middle row of the projection inside, its first and last rows at the ends.
// One warp per pulse.
__global__ void __launch_bounds__(kThreads) pga_smooth_kernel(const double2* __restrict__ xy, int pulses, int window,
                                                              const double* __restrict__ centre,
                                                              const double* __restrict__ left,
                                                              const double* __restrict__ right,
                                                              double2* __restrict__ out) {
    const int n = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31, half = window / 2;
    if (n >= pulses) return;
    const double* row = centre;
    int first = n - half;
    if (n < half) {
        row = left + (size_t)n * window;
        first = 0;
    } else if (n >= pulses - half) {
        row = right + (size_t)(n - (pulses - half)) * window;
        first = pulses - window;
    }
    double2 s = make_double2(0.0, 0.0);
    for (int j = lane; j < window; j += 32) {
        const double c = row[j];
        const double2 v = xy[first + j];
        s.x = fma(c, v.x, s.x);
        s.y = fma(c, v.y, s.y);
    }
    s.x = shfl_add(s.x);
    s.y = shfl_add(s.y);
    if (lane == 0) out[n] = s;
}

// delta [pulses, 3] = (x, y, 0), scaled down to 1 m at most; stats[1..3] its root mean squares, [4..6] largest sizes.
__global__ void __launch_bounds__(kTrackThreads) pga_finish_kernel(const double2* __restrict__ xy, int pulses,
                                                                   double* __restrict__ delta,
                                                                   double* __restrict__ stats) {
    __shared__ double part[33];
    __shared__ long long top[33];
    // Largest of sizes by their bit patterns (integers; what is no number is above everything: tested apart, since the
    // mask may be compiled to an absolute value, which keeps that one's sign).
    const auto size_bits = [](double v) {
        const long long b = __double_as_longlong(v);
        return no_number(b) ? 0x7fffffffffffffffll : b & 0x7fffffffffffffffll;
    };
    const auto block_max = [&](long long v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
        __syncthreads();
        if ((threadIdx.x & 31) == 0) top[threadIdx.x >> 5] = v;
        __syncthreads();
        long long s = top[0];
        for (int w = 1; w < kTrackThreads / 32; ++w) s = max(s, top[w]);
        return __longlong_as_double(s);
    };
    long long n2 = 0, bx = 0, by = 0;
    double sx = 0.0, sy = 0.0;
    for (int n = threadIdx.x; n < pulses; n += kTrackThreads) {
        const double2 v = xy[n];
        const double xx = v.x * v.x, yy = v.y * v.y;
        n2 = max(n2, size_bits(xx + yy));
        bx = max(bx, size_bits(v.x));
        by = max(by, size_bits(v.y));
        sx += xx;
        sy += yy;
    }
    const double norm = sqrt(block_max(n2)), mx = block_max(bx), my = block_max(by);
    sx = block_add(sx, part);
    sy = block_add(sy, part);
    const double div = norm > 1.0 ? norm : 1.0;
    for (int n = threadIdx.x; n < pulses; n += kTrackThreads) {
        const double2 v = xy[n];
        delta[3 * n] = div > 1.0 ? v.x / div : v.x;
        delta[3 * n + 1] = div > 1.0 ? v.y / div : v.y;
        delta[3 * n + 2] = 0.0;
    }
    if (threadIdx.x == 0) {
        stats[1] = sqrt(sx / (double)pulses) / div;
        stats[2] = sqrt(sy / (double)pulses) / div;
        stats[3] = 0.0;
        stats[4] = mx / div;
        stats[5] = my / div;
        stats[6] = 0.0;
    }
}

}  // namespace

int pga_max_targets() { return kMaxTargets; }

size_t pga_update_workspace(int targets, int pulses) {
    return sizeof(double) * (3 * (size_t)targets + 6 * (size_t)pulses);
}

int launch_pga_update(const double2* smooth, int targets, int pulses, const double* pos, const double* xyz, double k,
                      const double* centre, const double* left, const double* right, int window, double* delta,
                      double* stats, void* ws, cudaStream_t s) {
    double2* rate = static_cast<double2*>(ws);
    double2 *xy = rate + pulses, *smoothed = xy + pulses;
    double *power = reinterpret_cast<double*>(smoothed + pulses), *coherence = power + targets, *scale = coherence + targets;
    const int block = (targets + 31) / 32 * 32;
    const size_t smem = 6 * sizeof(double) * (size_t)block;
    if (int st = allow_shared(reinterpret_cast<const void*>(pga_pulses_kernel), smem)) return st;
    pga_targets_kernel<<<targets, kThreads, 0, s>>>(smooth, pulses, power, coherence);
    pga_weights_kernel<<<1, block, 0, s>>>(power, coherence, targets, scale, stats);
    pga_pulses_kernel<<<pulses - 1, block, smem, s>>>(smooth, targets, pulses, pos, xyz, 1.0 / k, scale, rate);
    pga_track_kernel<<<1, kTrackThreads, 0, s>>>(rate, pulses, xy);
    pga_smooth_kernel<<<(pulses + kThreads / 32 - 1) / (kThreads / 32), kThreads, 0, s>>>(xy, pulses, window, centre,
                                                                                        left, right, smoothed);
    pga_finish_kernel<<<1, kTrackThreads, 0, s>>>(smoothed, pulses, delta, stats);
    note_launches(6);
    return check_launch("pga_update");
}

}  // namespace sarbp
