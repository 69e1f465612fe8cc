// Spatial order of a point list for split-precision direct BP.
//
// The points kernel forms tiles of 512 consecutive points; its fast path needs tiles of a limited
// radius (points_radius: 22 m at 4 km and 9.6 GHz), while a raster of terrain points puts a tile on a strip of
// hundreds of metres and every pulse on the two-float fallback.  These kernels order a list by the Hilbert curve of a 256 x 256
// raster over its bounding square: two stable 8-bit counting passes, so the order (and with it the
// image) is the same on every run.  Nothing is ordered when no tile is wide: the kernels
// then return at once, and the points kernel takes the list as it is.
// 192,384 terrain points in raster order (501 to a row, half a metre apart), 1024 pulses: 2.50 ms as they
// come, 0.61 ms ordered, of which the ordering is about 0.05; error against FP64 2.7e-7 as they come, 2.3e-7 ordered.
#include "common.cuh"

namespace sarbp {
namespace {

constexpr int kThreads = 256;
constexpr int kTilePoints = kPointTile;  // points per tile of the points kernel
// Lists of wider tiles (m; 16 m and the tenth that is added to a box's half diagonal) are ordered even where the fast path takes
// them as they are: what it rounds grows with a tile's radius.  68 x 266 points of 0.25 m at 30 km x 826 pulses, tiles
// of 33 m radius as they come: error 3.6e-7 and 92 us, ordered 1.1e-7 and 107.
constexpr float kCompactRadius = 17.6f;
constexpr int kDigits = 256;

// FP32 as an unsigned of the same order.
__device__ __forceinline__ unsigned ordered(float v) {
    const unsigned b = __float_as_uint(v);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float unordered(unsigned u) {
    return __uint_as_float(u & 0x80000000u ? u ^ 0x80000000u : ~u);
}

// Bounds of each tile: the list's bounding box, and whether any tile is wide (above kCompactRadius or the radius that the fast
// path takes, seen from the first, middle or last pulse; a tile's own radius is about its points' mean and may be a
// little larger than its box's).  One block per tile.
__global__ void __launch_bounds__(kThreads) points_extent_kernel(PulseInputs in, float K, float inv_dr, float cap,
                                                                 const double* __restrict__ xyz, int npts,
                                                                 PointOrder* __restrict__ h) {
    const float inf = __int_as_float(0x7f800000);
    float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
    const int end = min(npts, (blockIdx.x + 1) * kTilePoints);
    for (int i = blockIdx.x * kTilePoints + threadIdx.x; i < end; i += kThreads)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float v = (float)xyz[3LL * i + c];
            lo[c] = fminf(lo[c], v);
            hi[c] = fmaxf(hi[c], v);
        }
    __shared__ float part[kThreads / 32][6];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
            hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
        }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            part[threadIdx.x >> 5][c] = lo[c];
            part[threadIdx.x >> 5][3 + c] = hi[c];
        }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < kThreads / 32; ++w)
        for (int c = 0; c < 3; ++c) {
            lo[c] = fminf(lo[c], part[w][c]);
            hi[c] = fmaxf(hi[c], part[w][3 + c]);
        }
    float d2 = 0.0f, R2 = inf;
    for (int c = 0; c < 3; ++c) d2 += (hi[c] - lo[c]) * (hi[c] - lo[c]);
    for (int k = 0; k < 3; ++k) {
        const double* p = in.pos + 3LL * ((in.pulses - 1) * (long long)k / 2);
        float r2 = 0.0f;
        for (int c = 0; c < 3; ++c) {
            const float d = (float)(p[c] - 0.5 * ((double)lo[c] + (double)hi[c]));
            r2 = fmaf(d, d, r2);
        }
        R2 = fminf(R2, r2);
    }
    const float limit = fminf(points_radius(K, inv_dr, cap, sqrtf(R2)), kCompactRadius), radius = 1.1f * 0.5f * sqrtf(d2);
    for (int c = 0; c < 2; ++c) {
        atomicMin(&h->low[c], ordered(lo[c]));
        atomicMin(&h->high[c], ~ordered(hi[c]));
    }
    atomicMin(&h->narrow, radius <= limit ? 1u : 0u);
}

// Place of cell (x, y) along the Hilbert curve of a 256 x 256 raster: level by level from the top, the
// quadrant's two bits, then the quadrant's own orientation (swap, and mirror in the fourth).  Its steps
// go to neighbouring cells, so any stretch of it is compact (the Z-curve's jumps left a third of the tiles
// wide).
__device__ __forceinline__ unsigned hilbert(unsigned x, unsigned y) {
    unsigned key = 0;
#pragma unroll
    for (unsigned bit = 128; bit; bit >>= 1) {
        const unsigned rx = (x & bit) ? 1u : 0u, ry = (y & bit) ? 1u : 0u;
        key = 4 * key + ((3u * rx) ^ ry);
        if (!ry) {
            if (rx) {
                x = 255u - x;
                y = 255u - y;
            }
            const unsigned t = x;
            x = y;
            y = t;
        }
    }
    return key;
}

// Counts of each digit in each block's keys, digit-major: counts[digit * blocks + block].  FIRST: the keys
// are made from the points.
template <bool FIRST>
__global__ void __launch_bounds__(kThreads) points_count_kernel(const double* __restrict__ xyz, int npts, int per,
                                                                const PointOrder* __restrict__ h,
                                                                unsigned short* __restrict__ keys,
                                                                int* __restrict__ counts) {
    if (h->narrow) return;
    __shared__ int hist[kDigits];
    hist[threadIdx.x] = 0;
    __syncthreads();
    const float x0 = unordered(h->low[0]), y0 = unordered(h->low[1]);
    const float span = fmaxf(unordered(~h->high[0]) - x0, unordered(~h->high[1]) - y0);
    const float scale = 255.99f / fmaxf(span, 1e-6f);
    const int end = min(npts, (int)(blockIdx.x + 1) * per);
    for (int i = blockIdx.x * per + threadIdx.x; i < end; i += kThreads) {
        unsigned key;
        if (FIRST) {
            // Cells outside 0 .. 255 (no numbers, overflow) go to the edge cells.
            const unsigned qx = (unsigned)fminf(fmaxf(((float)xyz[3LL * i] - x0) * scale, 0.0f), 255.0f);
            const unsigned qy = (unsigned)fminf(fmaxf(((float)xyz[3LL * i + 1] - y0) * scale, 0.0f), 255.0f);
            key = hilbert(qx, qy);
            keys[i] = (unsigned short)key;
        } else {
            key = keys[i];
        }
        atomicAdd(&hist[FIRST ? key & 255u : key >> 8], 1);
    }
    __syncthreads();
    counts[threadIdx.x * gridDim.x + blockIdx.x] = hist[threadIdx.x];
}

// Exclusive prefix sum of n counts in place (one block, n a multiple of 4, counts 16-byte aligned): rounds of
// four counts per thread, the next round's load in flight.  (48,128 counts, from 188 blocks: 10 us, with a stretch of
// them per thread 41.)
__global__ void __launch_bounds__(1024) points_scan_kernel(const PointOrder* __restrict__ h, int* __restrict__ counts,
                                                           int n) {
    if (h->narrow) return;
    __shared__ int warps[2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int4* c = reinterpret_cast<int4*>(counts);
    const int quads = n / 4;
    int4 next = (int)threadIdx.x < quads ? c[threadIdx.x] : make_int4(0, 0, 0, 0);
    int carry = 0;
    for (int q0 = 0, round = 0; q0 < quads; q0 += 1024, round ^= 1) {
        const int q = q0 + threadIdx.x;
        const int4 v = next;
        next = q + 1024 < quads ? c[q + 1024] : make_int4(0, 0, 0, 0);
        const int sum = v.x + v.y + v.z + v.w;
        int inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) warps[round][warp] = inc;
        __syncthreads();  // rounds use the two rows in turn, so one barrier each is enough
        int w = warps[round][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        const int before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
        int at = carry + inc - sum + (warp ? before : 0);
        carry += __shfl_sync(0xffffffffu, w, 31);
        if (q < quads) c[q] = make_int4(at, at + v.x, at + v.x + v.y, at + v.x + v.y + v.z);
    }
}

// Stable scatter of one pass: a round of 256 keys at a time, ranked by warp (lanes with the same digit) and
// over the warps.  FIRST: the payload is the point's index.
template <bool FIRST>
__global__ void __launch_bounds__(kThreads) points_scatter_kernel(int npts, int per, const PointOrder* __restrict__ h,
                                                                  const unsigned short* __restrict__ keys,
                                                                  const int* __restrict__ index,
                                                                  const int* __restrict__ counts,
                                                                  unsigned short* __restrict__ keys_out,
                                                                  int* __restrict__ index_out) {
    if (h->narrow) return;
    __shared__ int base[kDigits];
    __shared__ int seen[kThreads / 32][kDigits];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    base[threadIdx.x] = counts[threadIdx.x * gridDim.x + blockIdx.x];
    const int begin = blockIdx.x * per, end = min(npts, begin + per);
    for (int r = begin; r < end; r += kThreads) {
        for (int w = 0; w < kThreads / 32; ++w) seen[w][threadIdx.x] = 0;
        __syncthreads();
        const int i = r + threadIdx.x;
        const unsigned key = i < end ? keys[i] : 0u;
        const unsigned digit = i < end ? (FIRST ? key & 255u : key >> 8) : kDigits;
        const unsigned same = __match_any_sync(0xffffffffu, digit);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (i < end && rank == 0) seen[warp][digit] = __popc(same);
        __syncthreads();
        int at = base[threadIdx.x];  // thread t: digit t
        for (int w = 0; w < kThreads / 32; ++w) {
            const int v = seen[w][threadIdx.x];
            seen[w][threadIdx.x] = at;
            at += v;
        }
        base[threadIdx.x] = at;
        __syncthreads();
        if (i < end) {
            const int to = seen[warp][digit] + rank;
            index_out[to] = FIRST ? i : index[i];
            if (FIRST) keys_out[to] = (unsigned short)key;
        }
        __syncthreads();
    }
}

size_t align_up(size_t v) { return (v + 255) / 256 * 256; }

// Blocks of a counting pass: one per SM at most (the scan of their counts is the cost of more), each on a whole number
// of rounds of kThreads keys.  192,384 points x 1024 pulses, all in all: 94 blocks 599 us, 152 (one per SM) 598, 188 601,
// 376 611; six million points x 4 pulses 1131, 974, 935 and 855.
int keys_per_block(int npts) {
    const long long round = (long long)kThreads * sm_count();
    return (int)(kThreads * ((npts + round - 1) / round));
}
int order_blocks(int npts) { return (int)(((long long)npts + keys_per_block(npts) - 1) / keys_per_block(npts)); }

}  // namespace

size_t points_order_bytes(int npts) {
    return align_up(sizeof(PointOrder)) + 2 * align_up(sizeof(unsigned short) * (size_t)npts) +
           2 * align_up(sizeof(int) * (size_t)npts) + align_up(sizeof(int) * (size_t)kDigits * order_blocks(npts));
}

// Orders the list in `ws` (points_order_bytes, 256-byte aligned); *order, *index: what the points kernel takes.
int launch_points_order(const PulseInputs& in, int cap, const double* xyz, int npts, void* ws, const PointOrder** order,
                        const int** index, cudaStream_t s) {
    char* p = static_cast<char*>(ws);
    const auto take = [&p](size_t bytes) {
        char* at = p;
        p += align_up(bytes);
        return at;
    };
    auto* h = reinterpret_cast<PointOrder*>(take(sizeof(PointOrder)));
    auto* keys = reinterpret_cast<unsigned short*>(take(sizeof(unsigned short) * (size_t)npts));
    auto* keys1 = reinterpret_cast<unsigned short*>(take(sizeof(unsigned short) * (size_t)npts));
    auto* index1 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)npts));
    auto* index2 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)npts));
    const int blocks = order_blocks(npts), per = keys_per_block(npts);
    auto* counts = reinterpret_cast<int*>(take(sizeof(int) * (size_t)kDigits * blocks));
    const cudaError_t e = cudaMemsetAsync(h, 0xff, sizeof(PointOrder), s);
    if (e != cudaSuccess) return fail(SARBP_ERR_CUDA, "points order: %s", cudaGetErrorString(e));
    points_extent_kernel<<<(npts + kTilePoints - 1) / kTilePoints, kThreads, 0, s>>>(
        in, (float)(in.k * kInvTwoPi), (float)(1.0 / in.data_dr), (float)cap, xyz, npts, h);
    points_count_kernel<true><<<blocks, kThreads, 0, s>>>(xyz, npts, per, h, keys, counts);
    points_scan_kernel<<<1, 1024, 0, s>>>(h, counts, kDigits * blocks);
    points_scatter_kernel<true><<<blocks, kThreads, 0, s>>>(npts, per, h, keys, nullptr, counts, keys1, index1);
    points_count_kernel<false><<<blocks, kThreads, 0, s>>>(xyz, npts, per, h, keys1, counts);
    points_scan_kernel<<<1, 1024, 0, s>>>(h, counts, kDigits * blocks);
    points_scatter_kernel<false><<<blocks, kThreads, 0, s>>>(npts, per, h, keys1, index1, counts, nullptr, index2);
    note_launches(7);
    *order = h;
    *index = index2;
    return check_launch("points_order");
}

}  // namespace sarbp
