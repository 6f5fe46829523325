// Environment importance table for NEE built on the device: the reference's
// build_environment_alias_table (threedgrut/model/aliastable.py:244-297) with its Vose alias
// construction (aliastable.py:49-116), which the reference runs in a host Python loop.
//
//   1. weights  per cell: equirect maps are area-averaged to the table size (cube maps, H == 6W,
//               are used as they are); Rec.709 luminance of the finite positive RGB times the
//               cell's solid angle (float32; solid angles evaluated in float64)
//   2. total    float64 sum of the weights (fixed order); all-zero or non-finite totals fall back
//               to the solid angles as weights, as the reference does
//   3. pdf      weight / (total * solid angle), per steradian
//   4. alias    scaled = w * n / total in float64; the small (< 1) and large (>= 1) lists in index
//               order, then Vose's pairing popping from the ends. The pairing is sequential by construction
//               and fixes the table; one thread walks it as a chain of one float64 value, with everything
//               that does not depend on that value done by the other threads before and after (k_env_alias)
#include <cmath>
#include <cstdint>

#include "../../include/ptir_b200.h"

namespace ptir {

namespace {

constexpr int kEnvThreads = 1024;

__device__ double solid_angle_equirect(int row, int h, int w) {
    const double pi = 3.14159265358979323846;
    const double e0 = ((double)row / h - 0.5) * pi, e1 = ((double)(row + 1) / h - 0.5) * pi;
    return fmax((2.0 * pi / w) * (sin(e1) - sin(e0)), 0.0);
}

__device__ double solid_angle_cube(int u, int v, int fs) {
    auto area = [](double x, double y) { return atan2(x * y, sqrt(x * x + y * y + 1.0)); };
    const double u0 = -1.0 + 2.0 * u / fs, u1 = -1.0 + 2.0 * (u + 1) / fs;
    const double v0 = -1.0 + 2.0 * v / fs, v1 = -1.0 + 2.0 * (v + 1) / fs;
    return fmax(area(u1, v1) - area(u0, v1) - area(u1, v0) + area(u0, v0), 0.0);
}

// cell weights (float32, as the reference's float tensor) and solid angles
__global__ void k_env_weights(const float* __restrict__ env, int H, int W, int C, int th, int tw, int cube,
                              bool texels4, float* __restrict__ weight, float* __restrict__ solid) {
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= th * tw) return;
    const int oy = cell / tw, ox = cell - oy * tw;
    float rgb[3] = {0.0f, 0.0f, 0.0f};
    if (cube || (th == H && tw == W)) {
        const float* t = env + ((size_t)oy * W + ox) * C;
        rgb[0] = t[0];
        rgb[1] = t[1];
        rgb[2] = t[2];
    } else {
        // area average over the input rows [y0, y1) and columns [x0, x1) covered by the cell
        const int y0 = (int)(((long long)oy * H) / th), y1 = (int)((((long long)oy + 1) * H + th - 1) / th);
        const int x0 = (int)(((long long)ox * W) / tw), x1 = (int)((((long long)ox + 1) * W + tw - 1) / tw);
        float s[3] = {0.0f, 0.0f, 0.0f};
        for (int y = y0; y < y1; ++y) {
            const float* row = env + (size_t)y * W * C;
            if (texels4) {
                // the sums stay in texel order; only the loads are one a texel and run ahead of them
#pragma unroll 8
                for (int x = x0; x < x1; ++x) {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(row) + x);
                    s[0] += t.x;
                    s[1] += t.y;
                    s[2] += t.z;
                }
            } else {
                for (int x = x0; x < x1; ++x) {
                    const float* t = row + (size_t)x * C;
                    s[0] += t[0];
                    s[1] += t[1];
                    s[2] += t[2];
                }
            }
        }
        const float inv = 1.0f / (float)((y1 - y0) * (x1 - x0));
        rgb[0] = s[0] * inv;
        rgb[1] = s[1] * inv;
        rgb[2] = s[2] * inv;
    }
    for (int k = 0; k < 3; ++k) rgb[k] = (isfinite(rgb[k]) && rgb[k] > 0.0f) ? rgb[k] : 0.0f;
    const float lum = rgb[0] * 0.2126f + rgb[1] * 0.7152f + rgb[2] * 0.0722f;
    const double sa = cube ? solid_angle_cube(ox, oy % tw, tw) : solid_angle_equirect(oy, th, tw);
    solid[cell] = (float)sa;
    weight[cell] = lum * (float)sa;
}

// block-wide float64 sum in a fixed order
__device__ double block_sum(double v, double* red) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
    __syncthreads();
    if (threadIdx.x == 0) red[0] = t;
    __syncthreads();
    t = red[0];
    __syncthreads();
    return t;
}

// exclusive scan of one count per thread (block order), returns this thread's offset and the total
__device__ int block_scan(int v, int* warp_sums, int& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sums[w] = inc;
    __syncthreads();
    if (w == 0) {
        int t = warp_sums[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (lane >= o) t += y;
        }
        warp_sums[lane] = t;
    }
    __syncthreads();
    total = warp_sums[kEnvThreads / 32 - 1];
    const int before = w > 0 ? warp_sums[w - 1] : 0;
    __syncthreads();
    return before + inc - v;
}

// One block: pdf, then the alias table. scratch: scaled [n] float64, small / large [n] int32.
//
// The pairing. Vose pops a small cell s and a large cell g, sets s's probability and alias, and leaves g with
// v = scaled[g] - (1 - scaled[s]): at 1 or above g stays on top of the large list, below it goes on top of the small
// list, to be the next cell popped. So there is one value v in flight, of a large cell that takes the next
// small one (v >= 1) or of a cell that has become small and goes to the next large one (v < 1):
//   v >= 1:  v = v - (1 - small[i]),   alias of small[i] = the large cell
//   v <  1:  v = large[j] - (1 - v),   probability of the cell = v, its alias = large[j]
// The small cells' probabilities and 1 - small[i] do not depend on the chain. One thread walks it over windows of
// both lists in shared memory and logs v before every step; the block loads the windows and writes the table, where
// a scan over the log tells which cells each step popped. The float64 operations are those of the list form, in its
// order, so the table is bit for bit the same. Bound by the chain's latency, two float64 adds and a select a
// cell: a step computes both outcomes and picks one, compares v with 1 by its upper word, and has the next entry
// of both lists at hand. For the 64x128 table of a 512x1024 map the whole build took 1210 us with the lists and the
// scaled weights read and written in global memory on the way, 671 us with a branch and the table's values in
// the loop, and 213 us this way (13,824 cells of a cube map: 2271 -> 346 us).
constexpr int kPairWindow = 1280;  // the windows and the log stay within the 48 KB of static shared memory

struct PairWindows {
    double small[kPairWindow + 2];  // 1 - scaled of the small cells, in popping order
    double large[kPairWindow + 2];  // scaled of the large cells, in popping order
    double log[2 * kPairWindow];    // v before each step
};

// v >= 1 (v is not negative: a large cell's scaled weight is at least 1, and 1 - scaled at most 1)
__device__ __forceinline__ bool takes_small(double v) { return __double2hiint(v) >= 0x3FF00000; }

__global__ void __launch_bounds__(kEnvThreads) k_env_alias(int n, float* __restrict__ weight,
                                                           const float* __restrict__ solid, double* __restrict__ scaled,
                                                           int* __restrict__ small, int* __restrict__ large,
                                                           float* __restrict__ out) {
    __shared__ PairWindows win;
    __shared__ double red[kEnvThreads / 32];
    __shared__ int scan[kEnvThreads / 32];
    __shared__ int at[2];       // smalls and larges popped
    __shared__ int steps;       // of the window
    __shared__ bool finished;
    float* prob = out;
    float* alias = out + n;
    float* pdf = out + 2 * n;
    // contiguous chunk of cells per thread, so that lists come out in index order
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int first = min(n, (int)threadIdx.x * per), last = min(n, first + per);

    double t = 0.0;
    for (int i = first; i < last; ++i) t += (double)weight[i];
    double total = block_sum(t, red);
    // float32 total as the reference's float tensor sum; fall back to the solid angles
    const bool fallback = !(isfinite((float)total) && (float)total > 0.0f);
    if (fallback) {
        for (int i = first; i < last; ++i) weight[i] = solid[i];
        __syncthreads();
        t = 0.0;
        for (int i = first; i < last; ++i) t += (double)weight[i];
        total = block_sum(t, red);
    }
    const float total_f = (float)total;
    // Vose (aliastable.py:49-116): float64 scaled weights, index-ordered lists
    int ns = 0, nl = 0;
    for (int i = first; i < last; ++i) {
        const float w = weight[i], s = solid[i];
        pdf[i] = s > 0.0f ? w / fmaxf(total_f * s, 1.17549435e-38f) : 0.0f;
        const double v = (isfinite(w) && w > 0.0f) ? (double)w * ((double)n / total) : 0.0;
        scaled[i] = v;
        prob[i] = 1.0f;
        alias[i] = (float)i;
        if (total <= 0.0) continue;
        if (v < 1.0) ++ns; else ++nl;
    }
    int n_small = 0, n_large = 0;
    int so = block_scan(ns, scan, n_small);
    int lo = block_scan(nl, scan, n_large);
    if (total > 0.0) {
        // in popping order: the cells with the highest index first
        for (int i = first; i < last; ++i) {
            if (scaled[i] < 1.0) small[n_small - 1 - so++] = i; else large[n_large - 1 - lo++] = i;
        }
    }
    if (threadIdx.x == 0) {
        at[0] = at[1] = 0;
        finished = total <= 0.0 || n_small == 0 || n_large == 0;
    }
    __syncthreads();
    double v = 0.0;  // thread 0's
    while (!finished) {
        const int i0 = at[0], j0 = at[1];
        const int si = min(kPairWindow, n_small - i0), lj = min(kPairWindow, n_large - j0);
        for (int k = threadIdx.x; k < si; k += blockDim.x) win.small[k] = 1.0 - scaled[small[i0 + k]];
        for (int k = threadIdx.x; k < lj; k += blockDim.x) win.large[k] = scaled[large[j0 + k]];
        __syncthreads();
        const bool start = i0 == 0 && j0 == 0;  // the first pair
        if (threadIdx.x == 0) {
            int i = 0, j = 0, k = 0;
            if (start) {
                v = win.large[0] - win.small[0];
                i = j = 1;
            }
            double s0 = win.small[i], s1 = win.small[i + 1], l0 = win.large[j], l1 = win.large[j + 1];
            auto step = [&]() {
                const bool small_next = takes_small(v);
                win.log[k++] = v;
                const double a = v - s0, b = l0 - (1.0 - v);
                v = small_next ? a : b;
                s0 = small_next ? s1 : s0;
                l0 = small_next ? l0 : l1;
                i += small_next ? 1 : 0;
                j += small_next ? 0 : 1;
                s1 = win.small[i + 1];
                l1 = win.large[j + 1];
            };
            // as many steps as neither list can run out in, then step by step to the window's end
            for (int m = min(si - i, lj - j); m >= 8; m = min(si - i, lj - j)) {
#pragma unroll 4
                for (int x = 0; x < m; ++x) step();
            }
            while (takes_small(v) ? i < si : j < lj) step();
            at[0] = i0 + i;
            at[1] = j0 + j;
            steps = k;
            finished = takes_small(v) ? i0 + i >= n_small : j0 + j >= n_large;
        }
        __syncthreads();
        int i1 = i0 + (start ? 1 : 0), j1 = j0 + (start ? 1 : 0);  // popped before the steps
        if (start && threadIdx.x == 0) {
            const int s = small[0];
            prob[s] = (float)fmin(fmax(scaled[s], 0.0), 1.0);
            alias[s] = (float)large[0];
        }
        for (int k0 = 0; k0 < steps; k0 += kEnvThreads) {
            const int k = k0 + (int)threadIdx.x;
            const bool live = k < steps;
            const double vk = live ? win.log[k] : 0.0;
            const bool small_next = live && takes_small(vk);
            int smalls = 0;
            const int before = block_scan(small_next ? 1 : 0, scan, smalls);
            const int i = i1 + before, j = j1 + (k - k0) - before;  // popped before step k
            if (small_next) {
                const int s = small[i];
                prob[s] = (float)fmin(fmax(scaled[s], 0.0), 1.0);
                alias[s] = (float)large[j - 1];
            } else if (live) {
                const int g = large[j - 1];
                prob[g] = (float)fmin(fmax(vk, 0.0), 1.0);
                alias[g] = (float)large[j];
            }
            i1 += smalls;
            j1 += min(kEnvThreads, steps - k0) - smalls;
        }
        __syncthreads();
    }
    // leftovers keep probability 1 and alias themselves (set above)
}

}  // namespace

}  // namespace ptir

extern "C" size_t ptir_env_table_scratch_bytes(int32_t cells) {
    return cells <= 0 ? 0 : (size_t)cells * (sizeof(double) + 2 * sizeof(int) + 2 * sizeof(float)) + 256;
}

extern "C" int ptir_build_env_table(const float* environment, int32_t env_h, int32_t env_w, int32_t channels,
                                    int32_t table_h, int32_t table_w, float* table_out, void* scratch,
                                    size_t scratch_bytes, void* stream) {
    if (!environment || !table_out || env_h <= 0 || env_w <= 0 || channels < 3) return PTIR_EINVAL;
    const bool cube = env_h == 6 * env_w;
    const int th = cube ? env_h : table_h, tw = cube ? env_w : table_w;
    if (th <= 0 || tw <= 0) return PTIR_EINVAL;
    const long long cells = (long long)th * tw;
    if (cells > (1ll << 30) || scratch_bytes < ptir_env_table_scratch_bytes((int32_t)cells) || !scratch)
        return PTIR_EINVAL;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    char* p = static_cast<char*>(scratch);
    p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 15u) & ~uintptr_t(15));
    double* scaled = reinterpret_cast<double*>(p);
    int* small = reinterpret_cast<int*>(scaled + cells);
    int* large = small + cells;
    float* weight = reinterpret_cast<float*>(large + cells);
    float* solid = weight + cells;
    const int block = 64;  // a table has few cells: blocks for all SMs
    const bool texels4 = channels == 4 && (reinterpret_cast<uintptr_t>(environment) & 15u) == 0;
    ptir::k_env_weights<<<(unsigned)((cells + block - 1) / block), block, 0, s>>>(
        environment, env_h, env_w, channels, th, tw, cube ? 1 : 0, texels4, weight, solid);
    ptir::k_env_alias<<<1, ptir::kEnvThreads, 0, s>>>((int)cells, weight, solid, scaled, small, large, table_out);
    return cudaGetLastError() == cudaSuccess ? PTIR_OK : PTIR_ECUDA;
}
