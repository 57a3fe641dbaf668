// Parameters and epilogues shared by the general GEMM kernels (gemm_tiled.cu, gemm_tc.cu).
#pragma once
#include "common.cuh"

namespace zl {

struct GemmP {
    const void* x;
    const void* w;
    void* y;
    const float* gate;
    long long ldx, xb, ldw, wb, ldy, yb, ldg, gb;
    int M, N, K;
    const float* bias = nullptr;      // (batch, N) fp32, added before the epilogue
    long long bb = 0;
    const int32_t* grp_off = nullptr; // grouped mode: rows grp_off[b] .. grp_off[b+1] of the sorted list belong to problem b
    const int32_t* x_rows = nullptr;  // sorted index -> row of x (identity when null)
    const int32_t* y_rows = nullptr;  // sorted index -> row of y (identity when null)
    int act_tanh = 0;                 // few-rows kernel without the gated unit: tanh of the (biased) sum
    float limit = 0.f, alpha = 1.f, beta = 0.f;   // gated unit: g = min(gate, limit), u = clamp(up, +-limit), g sigmoid(alpha g) (u + beta)
                                      // soft cap: limit * tanh(v / limit)
    int pair_fn = ZL_GEMM_EPI_GLU_CLAMP;   // few-rows kernel with a gated unit: which of the pair epilogues
    int act_gelu_mul = 0;             // few-rows kernel without the gated unit: gelu_tanh of the (biased) sum times gate[m][n]
    const void* bias_t = nullptr;     // (N) in the input type, instead of `bias` (tensor-core kernel)
    int act_relu2 = 0;                // few-rows kernel without the gated unit: max(sum, 0)^2
};

__host__ __device__ constexpr bool epi_pairs(int epi) { return epi == ZL_GEMM_EPI_GLU_CLAMP || epi == ZL_GEMM_EPI_GEGLU_TANH || epi == ZL_GEMM_EPI_REGLU; }


// rows of problem b and the place of its first row in the sorted list
__device__ __forceinline__ void gemm_rows_of(const GemmP& p, int b, int& rows, int& first) {
    if (p.grp_off) {
        first = p.grp_off[b];
        rows = p.grp_off[b + 1] - first;
    } else {
        first = 0;
        rows = p.M;
    }
}
__device__ __forceinline__ float glu_clamp(float gate, float up, const GemmP& p) {
    const float g = fminf(gate, p.limit), u = fminf(fmaxf(up, -p.limit), p.limit);
    return g * (1.0f / (1.0f + expf(-p.alpha * g))) * (u + p.beta);
}

template <int EPI>
__device__ __forceinline__ float pair_unit(float gate, float up, const GemmP& p) {
    if constexpr (EPI == ZL_GEMM_EPI_GEGLU_TANH) return gelu_f(gate) * up;
    else if constexpr (EPI == ZL_GEMM_EPI_REGLU) return fmaxf(gate, 0.f) * up;
    else return glu_clamp(gate, up, p);
}

template <int EPI>
__device__ __forceinline__ float gemm_epilogue(float v, const GemmP& p, int b, int m, int n) {
    if constexpr (EPI == ZL_GEMM_EPI_RELU2) {
        const float r = fmaxf(v, 0.f);
        return r * r;
    } else if constexpr (EPI == ZL_GEMM_EPI_SIGMOID_GATE) {
        const float g = p.gate[(size_t)b * p.gb + (size_t)m * p.ldg + n];
        return v * (1.0f / (1.0f + expf(-g)));
    } else if constexpr (EPI == ZL_GEMM_EPI_TANH) {
        return tanhf(v);
    } else if constexpr (EPI == ZL_GEMM_EPI_GELU_TANH_MUL) {
        return gelu_f(v) * p.gate[(size_t)b * p.gb + (size_t)m * p.ldg + n];
    } else if constexpr (EPI == ZL_GEMM_EPI_SOFTCAP) {
        return p.limit * tanhf(v / p.limit);
    } else {
        return v;
    }
}

// tcgen05 kernel for 16-bit inputs (gemm_tc.cu): whether it is the faster one for the call, and its launch.  cudaErrorNotSupported:
// nothing was launched, since no tensor map of these pitches could be made; the kernels it stands beside take any.
bool gemm_tc_route(const GemmP& p, int batch, int in_dtype);
// whether gemm_tiled.cu's tile kernel is faster at that
bool gemm_tile_faster(int M, int N, int K, int batch);
cudaError_t launch_gemm_tc(const GemmP& p, int batch, int in_dtype, int out_dtype, int epilogue, bool pdl, cudaStream_t stream);

}  // namespace zl
