// W8A8 Linear for decode-sized M: SmoothQuant INT8 (Int8Linear, src/nn/linear/linear.cpp:432-636) and
// per-tensor FP8 e4m3 (Fp8Linear, linear.cpp:1612-1695).
//
// The reference runs three launches per INT8 Linear -- quant_calc_scale (int8/quant_kernel.cu:15-47), an s32
// cuBLASLt GEMM with M padded to 32 (linear.cpp:591-616) and quant_scale_back (quant_kernel.cu:231-246) -- with an
// int32 (M,N) round trip through HBM, and three per FP8 Linear (segmented_max_reduction + T_KERNEL_cvt_half_fp8 +
// cuBLASLt fp8, fp8/fp8_util.cu:58-228).  Here: one activation-quant kernel (per token / per tensor, optionally
// fused with RMSNorm like layernorm_quant, quant_kernel.cu:106-227) and ONE GEMM kernel that streams the 8-bit
// weights once from HBM straight into mma.sync fragments (m16n8k32, s8*s8->s32 or e4m3*e4m3->f32) and applies the
// scale-back (+bias) in its epilogue.  HBM-bound: N*K bytes per call.
//
// Layout trick (same as dense_gemm.cu): the sum over k is order-free, so lane (g,t) loads 16 CONTIGUOUS bytes of
// weight row g (and g+8) per 64-k step and the activation fragment uses the same k permutation -- every global
// load is a full 16-byte vector, no shared-memory staging of the weights at all.
// Small N is covered by splitting K across the warps of a CTA (int32 partial sums add exactly).
#include "common.cuh"

#include <cstdlib>

namespace zl {
// the same products on pairs of SMs (gemm_tc.cu)
template <typename T, bool FP8>
cudaError_t launch_w8_gemm_tc(const uint8_t* xq, const float* sx, const uint8_t* w, const void* sw, int sw_mode, const T* bias, T* y, int M, int N, int K,
                              bool pdl, cudaStream_t stream);
}  // namespace zl

#include <cuda_fp8.h>

namespace zl {

constexpr int kW8Warps = 8;
constexpr int kW8Unroll = 4;    // 64-k steps in flight per warp (4 x 2 x 16 B per lane)

__device__ __forceinline__ void imma_s8s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void qmma_e4m3(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool FP8>
struct W8Acc {
    using type = int;
};
template <>
struct W8Acc<true> {
    using type = float;
};

// ---------------------------------------------------------------------------------------------
// activation quantisation
// ---------------------------------------------------------------------------------------------
template <typename V>
__device__ __forceinline__ V block_reduce(V v, V* sh, bool is_max) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = is_max ? warp_max(v) : warp_sum(v);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    V r = sh[0];
    for (int i = 1; i < nw; ++i) r = is_max ? fmaxf(r, sh[i]) : r + sh[i];
    __syncthreads();
    return r;
}

// quant_calc_scale (quant_kernel.cu:15-47): scale = absmax/127, q = int8(nearbyint(x * (127/absmax))).
// Bound by latency (24 x 8192: 0.6 MB): with NC > 0 a thread holds its NC chunks of 8 values in registers, all loads on their way at
// once and the row read one time; rows longer than 8 chunks per thread (K > 16384) are read twice, chunk after chunk.
// 24 x 8192 fp16: 6.2 -> 3.8 us.
template <typename T, int NC>
__global__ void __launch_bounds__(256) k_int8_quant_per_token(const T* __restrict__ x, int ldx, int8_t* __restrict__ q,
                                                              float* __restrict__ scale, int K, int early) {
    __shared__ float sh[8];
    pdl_start(early);
    pdl_wait();
    const T* row = x + (size_t)blockIdx.x * ldx;
    float amax = 0.f;
    auto take_max = [&](const uint4& raw) {
        float v[8];
        unpack8<T>(raw, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
    };
    uint4 held[NC > 0 ? NC : 1];
    if constexpr (NC > 0) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int i = (threadIdx.x + c * 256) * 8;
            held[c] = i < K ? ld_cg_u4(row + i) : make_uint4(0, 0, 0, 0);   // zeros leave the maximum as it is
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) take_max(held[c]);
    } else {
        for (int i = threadIdx.x * 8; i < K; i += 256 * 8) take_max(ld_cg_u4(row + i));
    }
    amax = block_reduce(amax, sh, true);
    const float bs = __fdiv_rn(127.f, amax);
    auto convert = [&](const uint4& raw, int i) {
        float v[8];
        unpack8<T>(raw, v);
        uint32_t w[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            // absmax == 0 gives 0 * inf = NaN, which the reference's float->int8 conversion turns into 0
            const float r = nearbyintf(__fmul_rn(v[j], bs));
            const int qi = (r == r) ? (int)r : 0;
            w[j >> 2] |= (uint32_t)(qi & 0xff) << (8 * (j & 3));
        }
        *reinterpret_cast<uint2*>(q + (size_t)blockIdx.x * K + i) = make_uint2(w[0], w[1]);
    };
    if constexpr (NC > 0) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int i = (threadIdx.x + c * 256) * 8;
            if (i < K) convert(held[c], i);
        }
    } else {
        for (int i = threadIdx.x * 8; i < K; i += 256 * 8) convert(ld_cg_u4(row + i), i);
    }
    if (threadIdx.x == 0) scale[blockIdx.x] = __fdiv_rn(amax, 127.f);
}

// layernorm_quant (quant_kernel.cu:106-227): RMSNorm output in T plus its int8 twin.  The twin quantises
// v = x*w/scale (without rsqrt) and folds rsqrt into the scale; absmax is rounded through T (blockReduceMax<T>).
template <typename T>
__global__ void __launch_bounds__(256)
k_rmsnorm_quant(const T* __restrict__ x, const T* __restrict__ weight, T* __restrict__ y, int8_t* __restrict__ q,
                float* __restrict__ qscale, int D, float eps, float scale) {
    __shared__ float sh[8];
    pdl_trigger();
    pdl_wait();
    const T* row = x + (size_t)blockIdx.x * D;
    float sq = 0.f, amax = 0.f;
    for (int i = threadIdx.x * 8; i < D; i += blockDim.x * 8) {
        float v[8], w[8];
        unpack8<T>(ld_cg_u4(row + i), v);
        unpack8<T>(*reinterpret_cast<const uint4*>(weight + i), w);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            sq = fmaf(v[j], v[j], sq);
            amax = fmaxf(amax, fabsf(__fmul_rn(v[j], w[j])));
        }
    }
    sq = block_reduce(sq, sh, false);
    amax = block_reduce(amax, sh, true);
    amax = to_f32<T>(from_f32<T>(amax));
    const float rs = rsqrtf(sq / (float)D + eps);
    const float bs = (float)(127.0 / (double)amax);
    for (int i = threadIdx.x * 8; i < D; i += blockDim.x * 8) {
        float v[8], w[8], o[8];
        unpack8<T>(ld_cg_u4(row + i), v);
        unpack8<T>(*reinterpret_cast<const uint4*>(weight + i), w);
        uint32_t qw[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float vw = __fdiv_rn(__fmul_rn(v[j], w[j]), scale);
            o[j] = __fmul_rn(vw, rs);
            const float r = nearbyintf(__fmul_rn(vw, bs));
            const int qi = (r == r) ? (int)r : 0;
            qw[j >> 2] |= (uint32_t)(qi & 0xff) << (8 * (j & 3));
        }
        *reinterpret_cast<uint4*>(y + (size_t)blockIdx.x * D + i) = pack8<T>(o);
        *reinterpret_cast<uint2*>(q + (size_t)blockIdx.x * D + i) = make_uint2(qw[0], qw[1]);
    }
    if (threadIdx.x == 0) qscale[blockIdx.x] = (float)((double)__fmul_rn(amax, rs) / 127.);
}

// fp8 per-tensor dynamic quant (fp8_util.cu:110-228): scale = absmax / 448, q = e4m3(x / scale).
template <typename T>
__device__ __forceinline__ float fp8_absmax8(const T* p) {
    float v[8], m = 0.f;
    unpack8<T>(ld_cg_u4(p), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(v[j]));
    return m;
}
template <typename T>
__device__ __forceinline__ void fp8_convert8(const T* p, uint8_t* q, float inv) {
    float v[8];
    unpack8<T>(ld_cg_u4(p), v);
    uint32_t w[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        __half2 h2;
        if constexpr (std::is_same<T, __half>::value) {
            // fp16 input: the product is rounded in fp16 (__hmul2 with half(1/scale)), fp8_util.cu:77-80
            h2 = __hmul2(__floats2half2_rn(v[j], v[j + 1]), __float2half2_rn(inv));
        } else {
            h2 = __floats2half2_rn(__fmul_rn(inv, v[j]), __fmul_rn(inv, v[j + 1]));   // fp8_util.cu:74-76
        }
        const __nv_fp8x2_storage_t c = __nv_cvt_halfraw2_to_fp8x2(*reinterpret_cast<__half2_raw*>(&h2), __NV_SATFINITE, __NV_E4M3);
        w[j >> 2] |= (uint32_t)c << (16 * ((j >> 1) & 1));
    }
    *reinterpret_cast<uint2*>(q) = make_uint2(w[0], w[1]);
}

// Decode-sized inputs: one launch, every CTA takes the absmax of the whole (tiny) input itself, so there is no grid-wide
// dependency.  Bound by the latency of that walk: about 0.42 us per round of the CTA's loads.
constexpr int kFp8SmallThreads = 1024;
template <typename T>
__global__ void __launch_bounds__(kFp8SmallThreads)
k_fp8_quant_per_tensor(const T* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale, size_t n, int early) {
    __shared__ float sh[kFp8SmallThreads / 32];
    pdl_start(early);
    pdl_wait();
    float amax = 0.f;
    for (size_t i = (size_t)threadIdx.x * 8; i < n; i += (size_t)blockDim.x * 8) amax = fmaxf(amax, fp8_absmax8(x + i));
    amax = block_reduce(amax, sh, true);
    const float sc = __fdiv_rn(amax, 448.f);
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale = sc;
    const float inv = __fdiv_rn(1.f, sc);
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (size_t)gridDim.x * blockDim.x * 8)
        fp8_convert8(x + i, q + i, inv);
}

// Prompt-sized inputs: the scale word is zeroed, the CTAs raise it to the largest absmax / 448 of their shares, a second kernel
// converts.  Division by a constant is monotone, so the largest rounded quotient is the rounded quotient of the largest value:
// the same scale as above, and non-negative floats order like their bits.  500 x 4096 bf16: 429 us when every CTA walked the
// whole input, 12 us so.
__global__ void __launch_bounds__(32) k_fp8_zero(float* scale, int early) {
    pdl_start(early);
    pdl_wait();
    if (threadIdx.x == 0) *scale = 0.f;
}
template <typename T>
__global__ void __launch_bounds__(256) k_fp8_scale(const T* __restrict__ x, float* __restrict__ scale, size_t n) {
    __shared__ float sh[8];
    pdl_trigger();
    pdl_wait();
    float amax = 0.f;
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (size_t)gridDim.x * blockDim.x * 8)
        amax = fmaxf(amax, fp8_absmax8(x + i));
    amax = block_reduce(amax, sh, true);
    if (threadIdx.x == 0) atomicMax(reinterpret_cast<int*>(scale), __float_as_int(__fdiv_rn(amax, 448.f)));
}
template <typename T>
__global__ void __launch_bounds__(256) k_fp8_convert(const T* __restrict__ x, uint8_t* __restrict__ q, const float* __restrict__ scale,
                                                     size_t n) {
    pdl_trigger();
    pdl_wait();
    const float inv = __fdiv_rn(1.f, __ldcg(scale));
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (size_t)gridDim.x * blockDim.x * 8)
        fp8_convert8(x + i, q + i, inv);
}

// Above this many values (eight rounds of a 1024-thread CTA) the walk of the whole input by every CTA costs more than two more launches.  The
// word is zeroed by a kernel and not by a memset so that a chain of dependents holds.  kPdlBehind against ordinary launches,
// k_int8_quant_per_token too: a whole fp8 Linear of 500 x 4096 -> 14336 43.2 -> 41.1 us in a row of calls, an int8 one of 24 x 8192 -> 8192 20.6 -> 19.9.
constexpr size_t kFp8OneLaunchMax = 65536;

template <typename T>
static cudaError_t launch_fp8_quant(const T* x, uint8_t* q, float* scale, size_t n, int pdl, cudaStream_t st) {
    const size_t vecs = n / 8;
    const bool dependent = pdl != kPdlNone;
    const int early = pdl != kPdlBehind;
    if (n <= kFp8OneLaunchMax)
        return launch(k_fp8_quant_per_tensor<T>, dim3((unsigned)((vecs + kFp8SmallThreads - 1) / kFp8SmallThreads)), dim3(kFp8SmallThreads), 0,
                      st, dependent, x, q, scale, n, early);
    const size_t most = 8 * (size_t)device_sm_count();
    const unsigned ctas = (unsigned)((vecs + 255) / 256 < most ? (vecs + 255) / 256 : most);
    cudaError_t e = launch(k_fp8_zero, dim3(1), dim3(32), 0, st, dependent, scale, early);
    if (e == cudaSuccess) e = launch(k_fp8_scale<T>, dim3(ctas), dim3(256), 0, st, dependent, x, scale, n);
    if (e == cudaSuccess) e = launch(k_fp8_convert<T>, dim3(ctas), dim3(256), 0, st, dependent, x, q, (const float*)scale, n);
    return e;
}

// quant_scale_back (quant_kernel.cu:231-246) for callers that still hold an int32 accumulator
template <typename T>
__global__ void k_int8_scale_back(const int32_t* __restrict__ acc, const float* __restrict__ sx, const void* __restrict__ sw,
                                  int sw_f32, T* __restrict__ y, int N) {
    const int r = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    const float s_w = sw_f32 ? static_cast<const float*>(sw)[c] : to_f32<T>(static_cast<const T*>(sw)[c]);
    y[(size_t)r * N + c] = from_f32<T>(__fmul_rn(__fmul_rn((float)acc[(size_t)r * N + c], sx[r]), s_w));
}

// ---------------------------------------------------------------------------------------------
// GEMM: y(M,N) = scale-back( xq(M,K) . wq(N,K)^T )
// ---------------------------------------------------------------------------------------------
// One CTA = kW8Warps warps = (kW8Warps / KS) row tiles of 16 weight rows, each split KS ways along K.
template <typename T, bool FP8, int NT, int KS>
__global__ void __launch_bounds__(kW8Warps * 32)
k_w8a8_skinny(const uint8_t* __restrict__ xq, const float* __restrict__ sx, const uint8_t* __restrict__ w,
              const void* __restrict__ sw, int sw_f32, const T* __restrict__ bias, T* __restrict__ y, int mc, int N,
              int K) {
    using Acc = typename W8Acc<FP8>::type;
    constexpr int TPC = kW8Warps / KS;   // tiles per CTA
    __shared__ Acc red[KS > 1 ? kW8Warps : 1][NT][4][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int tile = blockIdx.x * TPC + warp / KS;
    const int ks = warp % KS;
    const int row0 = tile * 16;
    const bool live = row0 < N;
    pdl_trigger();

    const int steps = K / 64;
    const int s_lo = (int)((long long)steps * ks / KS), s_hi = (int)((long long)steps * (ks + 1) / KS);
    const int ra = min(row0 + g, N - 1), rb = min(row0 + g + 8, N - 1);
    const uint8_t* wa = w + (size_t)ra * K + t * 16;
    const uint8_t* wb = w + (size_t)rb * K + t * 16;

    uint4 na[kW8Unroll], nb[kW8Unroll];
    if (live) {
#pragma unroll
        for (int u = 0; u < kW8Unroll; ++u)
            if (s_lo + u < s_hi) {
                na[u] = ld_nc_na_u4(wa + (size_t)(s_lo + u) * 64);
                nb[u] = ld_nc_na_u4(wb + (size_t)(s_lo + u) * 64);
            }
    }
    pdl_wait();

    Acc acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[nt][c] = 0;

    if (live) {
        for (int s0 = s_lo; s0 < s_hi; s0 += kW8Unroll) {
            uint4 ca[kW8Unroll], cb[kW8Unroll], xb[kW8Unroll][NT];
#pragma unroll
            for (int u = 0; u < kW8Unroll; ++u) {
                ca[u] = na[u];
                cb[u] = nb[u];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const int tok = nt * 8 + g;
                    xb[u][nt] = (tok < mc && s0 + u < s_hi) ? ld_cg_u4(xq + (size_t)tok * K + (size_t)(s0 + u) * 64 + t * 16)
                                                            : make_uint4(0, 0, 0, 0);
                }
            }
#pragma unroll
            for (int u = 0; u < kW8Unroll; ++u) {
                const int sn = s0 + kW8Unroll + u;
                if (sn < s_hi) {
                    na[u] = ld_nc_na_u4(wa + (size_t)sn * 64);
                    nb[u] = ld_nc_na_u4(wb + (size_t)sn * 64);
                }
            }
#pragma unroll
            for (int u = 0; u < kW8Unroll; ++u) {
                if (s0 + u < s_hi) {
                    const uint32_t a0[4] = {ca[u].x, cb[u].x, ca[u].y, cb[u].y};
                    const uint32_t a1[4] = {ca[u].z, cb[u].z, ca[u].w, cb[u].w};
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        if constexpr (FP8) {
                            qmma_e4m3(acc[nt], a0, xb[u][nt].x, xb[u][nt].y);
                            qmma_e4m3(acc[nt], a1, xb[u][nt].z, xb[u][nt].w);
                        } else {
                            imma_s8s8(acc[nt], a0, xb[u][nt].x, xb[u][nt].y);
                            imma_s8s8(acc[nt], a1, xb[u][nt].z, xb[u][nt].w);
                        }
                    }
                }
            }
        }
    }

    if constexpr (KS > 1) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) red[warp][nt][c][lane] = acc[nt][c];
        __syncthreads();
        if (ks != 0) return;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                Acc s = acc[nt][c];
#pragma unroll
                for (int k2 = 1; k2 < KS; ++k2) s += red[warp + k2][nt][c][lane];
                acc[nt][c] = s;
            }
    }
    if (!live) return;

#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int tok = nt * 8 + 2 * t + (c & 1);
            const int row = row0 + g + ((c >> 1) ? 8 : 0);
            if (tok < mc && row < N) {
                float v;
                if constexpr (FP8) {
                    // cuBLASLt fp8: D = (scaleA * scaleB) * acc (+ bias), functions::Gemm with A/B scales
                    // sw_f32 == 2: one scale per output row (several per-tensor-scaled projections fused along N)
                    const float s_w = sw_f32 == 2 ? static_cast<const float*>(sw)[row] : *static_cast<const float*>(sw);
                    v = acc[nt][c] * (sx[0] * s_w);
                    if (bias) v += to_f32<T>(bias[row]);
                } else {
                    // quant_scale_back (quant_kernel.cu:231-246): T(float(acc) * sx[m] * sw[n]) then add_bias in T
                    const float s_w = sw_f32 ? static_cast<const float*>(sw)[row] : to_f32<T>(static_cast<const T*>(sw)[row]);
                    v = __fmul_rn(__fmul_rn((float)acc[nt][c], sx[tok]), s_w);
                    if (bias) v = to_f32<T>(from_f32<T>(v)) + to_f32<T>(bias[row]);
                }
                y[(size_t)tok * N + row] = from_f32<T>(v);
            }
        }
    }
}

template <typename T, bool FP8, int NT>
static cudaError_t launch_w8_ks(const uint8_t* xq, const float* sx, const uint8_t* w, const void* sw, int sw_f32,
                                const T* bias, T* y, int mc, int N, int K, bool pdl, cudaStream_t st) {
    const int tiles = cdiv(N, 16);
    // enough warps to keep ~13 MB of loads in flight chip-wide: aim for >= 16 warps per SM
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int steps = K / 64;
    int ks = 1;
    while (ks < kW8Warps && tiles * ks < sms * 16 && steps / (ks * 2) >= kW8Unroll) ks *= 2;
    dim3 block(kW8Warps * 32);
#define ZL_W8_LAUNCH(KS_)                                                                                          \
    return launch(k_w8a8_skinny<T, FP8, NT, KS_>, dim3(cdiv(tiles, kW8Warps / KS_)), block, 0, st, pdl, xq, sx, w, \
                  sw, sw_f32, bias, y, mc, N, K)
    if (ks == 1) ZL_W8_LAUNCH(1);
    if (ks == 2) ZL_W8_LAUNCH(2);
    if (ks == 4) ZL_W8_LAUNCH(4);
    ZL_W8_LAUNCH(8);
#undef ZL_W8_LAUNCH
}

template <typename T, bool FP8>
static cudaError_t launch_w8(const uint8_t* xq, const float* sx, const uint8_t* w, const void* sw, int sw_f32,
                             const T* bias, T* y, int mc, int N, int K, bool pdl, cudaStream_t st) {
    if (mc <= 8) return launch_w8_ks<T, FP8, 1>(xq, sx, w, sw, sw_f32, bias, y, mc, N, K, pdl, st);
    if (mc <= 16) return launch_w8_ks<T, FP8, 2>(xq, sx, w, sw, sw_f32, bias, y, mc, N, K, pdl, st);
    return launch_w8_ks<T, FP8, 4>(xq, sx, w, sw, sw_f32, bias, y, mc, N, K, pdl, st);
}

constexpr int kSmBytes = 228 * 1024;   // shared memory of an SM
template <typename T>
static cudaError_t launch_int8_quant(const T* x, int ldx, int8_t* q, float* scale, int M, int K, int pdl, cudaStream_t stream) {
    const int chunks = cdiv(K, 256 * 8);
    auto kernel = chunks <= 1 ? k_int8_quant_per_token<T, 1> : chunks <= 2 ? k_int8_quant_per_token<T, 2>
                  : chunks <= 4 ? k_int8_quant_per_token<T, 4> : chunks <= 8 ? k_int8_quant_per_token<T, 8> : k_int8_quant_per_token<T, 0>;
    // Where it comes under the end of whatever was before, its CTAs ask for the shared memory that spreads them over the SMs: beside a GEMM that still runs they were placed in
    // sixes.  With the GEMM behind it, in a graph, ordinary launches / dependents / dependents so: 100 rows of 4096 x 4096 11.5 / 12.7 / 11.5 us, 64 of 8192 x 8192 14.6 / 16.1 / 14.3, 160 of
    // 6144 x 4096 13.2 / 14.7 / 12.7, 32 of 28672 x 4096 26.3 / 28.6 / 26.2.
    const int per_sm = cdiv(M, device_sm_count()), smem = pdl != kPdlBehind || per_sm > 6 ? 0 : kSmBytes / (per_sm + 1);
    if (smem > 48 * 1024) {
        static bool set[64][5] = {};
        const int at = chunks <= 1 ? 0 : chunks <= 2 ? 1 : chunks <= 4 ? 2 : chunks <= 8 ? 3 : 4;
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 0 || dev >= 64 || !set[dev][at]) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmBytes / 2);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) set[dev][at] = true;
        }
    }
    return launch(kernel, dim3(M), dim3(256), (size_t)smem, stream, pdl != kPdlNone, x, ldx, q, scale, K, (int)(pdl != kPdlBehind));
}

}  // namespace zl

using namespace zl;

extern "C" int zl_int8_quant_per_token(const void* x, int ldx, void* q, float* scale, int M, int K, int dtype, int pdl,
                                       zl_stream_t stream) {
    ZL_CHECK_ARG(x && q && scale && M > 0 && K > 0);
    ZL_CHECK_ARG(dtype == ZL_F16 || dtype == ZL_BF16);
    ZL_CHECK_SUPPORTED(K % 8 == 0 && ldx % 8 == 0 && ldx >= K);
    ZL_CHECK_ARG((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0);
    const cudaError_t e = dtype == ZL_F16 ? launch_int8_quant(static_cast<const __half*>(x), ldx, static_cast<int8_t*>(q), scale, M, K, pdl, stream)
                                          : launch_int8_quant(static_cast<const __nv_bfloat16*>(x), ldx, static_cast<int8_t*>(q), scale, M, K, pdl, stream);
    ZL_CHECK_CUDA(e);
    return ZL_OK;
}

extern "C" int zl_rmsnorm_quant(const void* x, const void* weight, void* y, void* q, float* qscale, int T_, int D,
                                float eps, float scale, int dtype, int pdl, zl_stream_t stream) {
    ZL_CHECK_ARG(x && weight && y && q && qscale && T_ > 0 && D > 0);
    ZL_CHECK_ARG(dtype == ZL_F16 || dtype == ZL_BF16);
    ZL_CHECK_SUPPORTED(D % 8 == 0);
    cudaError_t e;
    if (dtype == ZL_F16)
        e = launch(k_rmsnorm_quant<__half>, dim3(T_), dim3(256), 0, stream, pdl != 0, static_cast<const __half*>(x),
                   static_cast<const __half*>(weight), static_cast<__half*>(y), static_cast<int8_t*>(q), qscale, D, eps,
                   scale);
    else
        e = launch(k_rmsnorm_quant<__nv_bfloat16>, dim3(T_), dim3(256), 0, stream, pdl != 0,
                   static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(weight),
                   static_cast<__nv_bfloat16*>(y), static_cast<int8_t*>(q), qscale, D, eps, scale);
    ZL_CHECK_CUDA(e);
    return ZL_OK;
}

extern "C" int zl_fp8_quant_per_tensor(const void* x, void* q, float* scale, size_t n, int dtype, int pdl,
                                       zl_stream_t stream) {
    ZL_CHECK_ARG(x && q && scale && n > 0);
    ZL_CHECK_ARG(dtype == ZL_F16 || dtype == ZL_BF16);
    ZL_CHECK_SUPPORTED(n % 8 == 0);
    ZL_CHECK_SUPPORTED(n <= ((size_t)1 << 22));   // the range this entry point has always had; the kernels below know no such limit
    const cudaError_t e = dtype == ZL_F16 ? launch_fp8_quant(static_cast<const __half*>(x), static_cast<uint8_t*>(q), scale, n, pdl, stream)
                                          : launch_fp8_quant(static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), scale, n, pdl, stream);
    ZL_CHECK_CUDA(e);
    return ZL_OK;
}

extern "C" int zl_int8_scale_back(const int32_t* acc, const float* x_scale, const void* w_scale, int w_scale_dtype,
                                  void* y, int M, int N, int dtype, zl_stream_t stream) {
    ZL_CHECK_ARG(acc && x_scale && w_scale && y && M > 0 && N > 0);
    ZL_CHECK_ARG(dtype == ZL_F16 || dtype == ZL_BF16);
    ZL_CHECK_ARG(w_scale_dtype == ZL_F32 || w_scale_dtype == dtype);
    dim3 grid(cdiv(N, 256), M);
    if (dtype == ZL_F16)
        k_int8_scale_back<__half><<<grid, 256, 0, stream>>>(acc, x_scale, w_scale, w_scale_dtype == ZL_F32,
                                                            static_cast<__half*>(y), N);
    else
        k_int8_scale_back<__nv_bfloat16><<<grid, 256, 0, stream>>>(acc, x_scale, w_scale, w_scale_dtype == ZL_F32,
                                                                   static_cast<__nv_bfloat16*>(y), N);
    ZL_CHECK_LAUNCH();
    return ZL_OK;
}

// Whether M rows go to the kernel on pairs of SMs (gemm_tc.cu), which costs the same from 1 row to 32 and has few, large tiles, whose K up to four
// pairs share; the mma.sync kernel reads its activations once per 16 weight rows and takes half as long again from 8 rows to 9 and from 16 to 17, fp8
// more than int8.  So the lines are weights per step of rows, and below 17 rows N as well: few tiles read the weights through few SMs.  us of a whole
// Linear in a row of calls, quantisation included, mma.sync / here, when the lines were drawn; of 1112 measured points (46 sizes from 1024 x 1024 to 28672 x 8192) none was sent here
// that took longer here, and what stayed cost 1.7 % on average:
//   int8, 32 rows   4096 x 4096 11.9 / 11.8; 6144 x 4096 20.0 / 12.6; 8192 x 8192 36.0 / 19.3; 1024 x 8192 17.0 / 11.5
//         16        4096 x 4096 8.9 / 11.8; 6144 x 4096 14.5 / 12.5; 4096 x 8192 13.9 / 14.8; 4096 x 14336 21.7 / 19.1
//          8        8192 x 8192 19.1 / 18.8; 8192 x 5120 14.7 / 15.0; 10240 x 4096 17.1 / 14.2; 28672 x 8192 59.9 / 43.8
//   fp8,  32 rows   2048 x 4096 14.4 / 15.8; 4096 x 4096 20.5 / 17.8; 8192 x 8192 49.9 / 24.8
//         16        2048 x 8192 16.4 / 18.4; 4096 x 4096 14.8 / 12.3; 8192 x 8192 39.6 / 25.0
//          8        8192 x 5120 16.7 / 14.7; 14336 x 4096 20.7 / 16.4; 4096 x 14336 22.7 / 24.6
// From 33 rows on it is here at every size (1088 x 512 6.0 against 6.7 / 6.0 for the kernel that served it before).
// This kernel has become faster since.  With both as they are now, 450 points in graphs (25 sizes, 1 .. 32 rows): still none is sent here that takes longer here, and the 180
// that stay cost 4.4 % on average, up to 49 %: fp8, 32 rows of 3072 x 3072 14.4 / 9.7, 8 rows of 8192 x 8192 19.0 / 13.6; int8, 32 rows of 4096 x 4096 11.0 / 9.6.
static bool w8_tc_route(int M, int N, int K, bool fp8) {
    constexpr long long kMi = 1 << 20;
    const long long weights = (long long)N * K;
    if (M > 32 || weights >= 128 * kMi) return true;
    if (M > 16) return fp8 ? weights >= 12 * kMi : weights >= 20 * kMi || (K >= 8192 && weights >= 4 * kMi);
    if (M > 8) return fp8 ? weights >= 12 * kMi && N >= 3072 : weights >= 24 * kMi && (N >= 5120 || weights >= 43 * kMi);
    return weights >= 40 * kMi && (N >= 9472 || (weights >= 66 * kMi && N >= 3584));
}
extern "C" int zl_w8_pairs_route(int M, int N, int K, int kind) {
    return M > 0 && N > 0 && K > 0 && w8_tc_route(M, N, K, kind != ZL_W8_INT8) ? 1 : 0;
}

extern "C" int zl_w8a8_gemm(const void* xq, const float* x_scale, const void* w, const void* w_scale,
                            int w_scale_dtype, const void* bias, void* y, int M, int N, int K, int kind, int dtype,
                            int pdl, zl_stream_t stream) {
    ZL_CHECK_WAITS();
    ZL_CHECK_ARG(xq && x_scale && w && w_scale && y && M > 0 && N > 0 && K > 0);
    ZL_CHECK_ARG(dtype == ZL_F16 || dtype == ZL_BF16);
    ZL_CHECK_ARG(kind == ZL_W8_INT8 || kind == ZL_W8_FP8 || kind == ZL_W8_FP8_ROWS);
    ZL_CHECK_ARG(w_scale_dtype == ZL_F32 || w_scale_dtype == dtype);
    ZL_CHECK_ARG(kind == ZL_W8_INT8 || w_scale_dtype == ZL_F32);
    ZL_CHECK_SUPPORTED(K % 64 == 0);
    ZL_CHECK_ARG((reinterpret_cast<uintptr_t>(xq) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0);
    const uint8_t* xq8 = static_cast<const uint8_t*>(xq);
    const uint8_t* w8 = static_cast<const uint8_t*>(w);
    const int sw_f32 = kind == ZL_W8_FP8_ROWS ? 2 : (w_scale_dtype == ZL_F32 ? 1 : 0);
    const bool fp8 = kind != ZL_W8_INT8;
    if (w8_tc_route(M, N, K, fp8)) {
        const int sw_mode = fp8 ? (kind == ZL_W8_FP8_ROWS ? 2 : 3) : sw_f32;
        cudaError_t e;
#define ZL_W8_TC(TT, F8)                                                                                                              \
    e = launch_w8_gemm_tc<TT, F8>(xq8, x_scale, w8, w_scale, sw_mode, static_cast<const TT*>(bias), static_cast<TT*>(y), M, N, K, pdl != 0, \
                                  stream)
        if (dtype == ZL_F16) {
            if (fp8) ZL_W8_TC(__half, true);
            else ZL_W8_TC(__half, false);
        } else {
            if (fp8) ZL_W8_TC(__nv_bfloat16, true);
            else ZL_W8_TC(__nv_bfloat16, false);
        }
#undef ZL_W8_TC
        if (e != cudaErrorNotSupported) {   // else: nothing launched, no tensor map could be made
            ZL_CHECK_CUDA(e);
            return ZL_OK;
        }
    }
    for (int m0 = 0; m0 < M; m0 += 32) {
        const int mc = (M - m0) < 32 ? (M - m0) : 32;
        const bool p = pdl != 0 && m0 == 0;
        const float* sx = kind == ZL_W8_INT8 ? x_scale + m0 : x_scale;
        cudaError_t e;
#define ZL_W8_GO(TT, F8)                                                                                           \
    e = launch_w8<TT, F8>(xq8 + (size_t)m0 * K, sx, w8, w_scale, sw_f32, static_cast<const TT*>(bias),              \
                          static_cast<TT*>(y) + (size_t)m0 * N, mc, N, K, p, stream)
        if (dtype == ZL_F16) {
            if (kind != ZL_W8_INT8) ZL_W8_GO(__half, true);
            else ZL_W8_GO(__half, false);
        } else {
            if (kind != ZL_W8_INT8) ZL_W8_GO(__nv_bfloat16, true);
            else ZL_W8_GO(__nv_bfloat16, false);
        }
#undef ZL_W8_GO
        ZL_CHECK_CUDA(e);
    }
    return ZL_OK;
}
