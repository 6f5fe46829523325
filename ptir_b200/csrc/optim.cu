// Fused selective Adam step (the reference's SelectiveAdam, threedgrut/optimizers/optimizers.cu:49-76
// and __init__.py:45-125): for every element of a Gaussian whose visibility flag is set,
//   m = b1 m + (1 - b1) g,  v = b2 v + (1 - b2) g^2,  p -= lr m / (sqrt(v) + eps)
// with no bias correction; elements of hidden Gaussians keep their parameter and moments.
// Square root and division are IEEE round-to-nearest whatever the compile flags.
#include <cstdint>

#include "../../include/ptir_b200.h"

namespace ptir {

namespace {

// One element: the moments and the parameter of a visible row.
__device__ __forceinline__ void adam_element(float g, float& p, float& m, float& v, float lr, float b1, float b2, float eps) {
    const float mi = b1 * m + (1.0f - b1) * g;
    const float vi = b2 * v + (1.0f - b2) * g * g;
    p += __fdiv_rn(-lr * mi, __fadd_rn(__fsqrt_rn(vi), eps));
    m = mi;
    v = vi;
}

// One thread per four consecutive elements, read and written as 16 bytes each, whatever the row length: the four
// may belong to two or more rows; of a four that spans a hidden row's border only the visible row's elements are
// written. Nothing is read of a hidden four but its rows' flags. The up to three elements after the last four
// are a thread each. Bound by HBM (28 bytes an element of a visible row); with one element a thread a
// 64-bit division by the row length each stood before the loads: 300,000 rows of 48, 60 % of them visible, took
// 80.2 us and take 56.7 (242 MB, 4.3 TB/s). Index: unsigned while the elements fit.
template <class Index>
__global__ void __launch_bounds__(256) k_selective_adam4(float4* __restrict__ param, const float4* __restrict__ grad,
                                                         float4* __restrict__ m, float4* __restrict__ v,
                                                         const uint8_t* __restrict__ visible, Index total, Index row,
                                                         float lr, float b1, float b2, float eps) {
    const Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x, fours = total / 4;
    if (i >= fours) {
        const Index e = 3 * fours + i;  // 4 fours + (i - fours)
        if (e < total && (!visible || visible[e / row]))
            adam_element(reinterpret_cast<const float*>(grad)[e], reinterpret_cast<float*>(param)[e],
                         reinterpret_cast<float*>(m)[e], reinterpret_cast<float*>(v)[e], lr, b1, b2, eps);
        return;
    }
    bool on[4] = {true, true, true, true};
    if (visible) {
        const Index first = 4 * i;
        Index r = first / row, left = (r + 1) * row - first;  // elements of row r from here on
        bool f = visible[r] != 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (left == 0) {
                f = visible[++r] != 0;
                left = row;
            }
            on[k] = f;
            --left;
        }
        if (!(on[0] || on[1] || on[2] || on[3])) return;
    }
    float4 p4 = param[i], m4 = m[i], v4 = v[i];
    const float4 g4 = grad[i];
    if (on[0]) adam_element(g4.x, p4.x, m4.x, v4.x, lr, b1, b2, eps);
    if (on[1]) adam_element(g4.y, p4.y, m4.y, v4.y, lr, b1, b2, eps);
    if (on[2]) adam_element(g4.z, p4.z, m4.z, v4.z, lr, b1, b2, eps);
    if (on[3]) adam_element(g4.w, p4.w, m4.w, v4.w, lr, b1, b2, eps);
    if (on[0] && on[1] && on[2] && on[3]) {
        param[i] = p4;
        m[i] = m4;
        v[i] = v4;
        return;
    }
    // a row's border: the hidden elements may be another step's (of other rows, on another stream) and are not written
    float *pe = reinterpret_cast<float*>(param + i), *me = reinterpret_cast<float*>(m + i), *ve = reinterpret_cast<float*>(v + i);
    const float pa[4] = {p4.x, p4.y, p4.z, p4.w}, ma[4] = {m4.x, m4.y, m4.z, m4.w}, va[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!on[k]) continue;
        pe[k] = pa[k];
        me[k] = ma[k];
        ve[k] = va[k];
    }
}

// One element per thread, for buffers that are not 16-byte aligned. With the index in 32 bits where it fits, a million
// rows of 48, a twentieth of them visible, take 78 us (88 us with a 64-bit division an element).
template <class Index>
__global__ void __launch_bounds__(256) k_selective_adam(float* __restrict__ param, const float* __restrict__ grad,
                                                        float* __restrict__ m, float* __restrict__ v,
                                                        const uint8_t* __restrict__ visible, Index total, Index row,
                                                        float lr, float b1, float b2, float eps) {
    for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (Index)gridDim.x * blockDim.x) {
        if (visible && !visible[i / row]) continue;
        adam_element(grad[i], param[i], m[i], v[i], lr, b1, b2, eps);
    }
}

__global__ void k_fold(float* __restrict__ out, const float* __restrict__ comp, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] += comp[i];
}

}  // namespace

// out[i] += comp[i]: the compensation terms of Kahan-pair gradient sums folded into the sums
cudaError_t launch_fold(float* out, const float* comp, long long n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const long long blocks = (n + 255) / 256;
    k_fold<<<(unsigned)(blocks < 148LL * 32 ? blocks : 148LL * 32), 256, 0, s>>>(out, comp, n);
    return cudaGetLastError();
}

}  // namespace ptir

extern "C" int ptir_selective_adam(float* param, const float* grad, float* exp_avg, float* exp_avg_sq,
                                   const uint8_t* visible, int64_t n_rows, int32_t row, float lr, float beta1,
                                   float beta2, float eps, void* stream) {
    if (n_rows < 0 || row <= 0) return PTIR_EINVAL;
    if (n_rows == 0) return PTIR_OK;
    if (!param || !grad || !exp_avg || !exp_avg_sq) return PTIR_EINVAL;
    const long long total = n_rows * (long long)row;
    const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int block = 256;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(param) | reinterpret_cast<uintptr_t>(grad) |
                           reinterpret_cast<uintptr_t>(exp_avg) | reinterpret_cast<uintptr_t>(exp_avg_sq);
    const bool fours = (bits & 15u) == 0;
    long long grid = ((fours ? total / 4 + total % 4 : total) + block - 1) / block;
    if (!fours) grid = grid < 148LL * 64 ? grid : 148LL * 64;
    if (grid > 0x7FFFFFFFll) return PTIR_EINVAL;
    const auto launch = [&](auto index) {
        using Index = decltype(index);
        const Index n = (Index)total, r = (Index)row;
        if (fours) {
            const auto as4 = [](float* p) { return reinterpret_cast<float4*>(p); };
            ptir::k_selective_adam4<Index><<<(unsigned)grid, block, 0, s>>>(
                as4(param), reinterpret_cast<const float4*>(grad), as4(exp_avg), as4(exp_avg_sq), visible, n, r, lr, beta1,
                beta2, eps);
        } else {
            ptir::k_selective_adam<Index><<<(unsigned)grid, block, 0, s>>>(param, grad, exp_avg, exp_avg_sq, visible, n, r,
                                                                           lr, beta1, beta2, eps);
        }
    };
    if (total + row < (1ll << 31)) launch(0u);
    else launch(0ll);
    return cudaGetLastError() == cudaSuccess ? PTIR_OK : PTIR_ECUDA;
}
