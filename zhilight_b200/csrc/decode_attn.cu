// Batch decode attention over per-task ragged KV buffers (GQA/MQA), split-KV with LSE combine.
//
// Replaces nn::multi_query_attention_rag_buffer and its kernels KERNEL_mqa_rag_buffer1 /
// KERNEL_mqa_rag_buffer_split_kv / KERNEL_mqa_combine / the wmma KERNEL_mqa_rag_buffer
// (reference src/nn/attention/attention_kernel.cu:674-725, 730-923, 926-1017, 1252-1457).
//
// One CTA = (kv-split, kv-head, task x query).  The whole GQA group (<= 8 q-heads per pass) shares
// every K/V byte: K is read ONCE per kv-head straight into tensor-core A fragments (16 keys x 16 dims),
// Q is the B operand (16 dims x 8 heads), so S = K.Q^T needs no shuffles; softmax is the reference's
// exact two-pass fp32 form inside the split (mask ? scale*s : -inf, max seeded -1e20, sum seeded 1e-20);
// P.V runs in fp32 on the CUDA cores with 16-byte coalesced V loads (each V element feeds all heads).
// Splits are merged with the reference's LSE rule (attention_kernel.cu:881-923).
#include "common.cuh"
#include "decode_attn_short.cuh"
#include "decode_attn_warp.cuh"
#include "prompt_attn.cuh"

#include <cstdlib>
#include <type_traits>

namespace zl {

constexpr int kAttnThreads = 128;
constexpr int kAttnWarps = 4;
constexpr int kAttnMaxRange = 1024;            // keys per CTA; logits live in shared memory
constexpr int kAttnRowStride = kAttnMaxRange + 4;
constexpr int kAttnMaxSplits = 64;

// PER_SM: CTAs of an SM at least, by registers: for D = 128 3 or 4, for D = 64 4, 5 or 0 (attn_per_sm)
template <typename T, int D, bool PV_FP32, int PER_SM>
__global__ void __launch_bounds__(kAttnThreads, PER_SM)
k_decode_attn(const T* __restrict__ q, const int32_t* __restrict__ buf_lens, T* const* __restrict__ k_addrs,
              T* const* __restrict__ v_addrs, const int8_t* __restrict__ mask, float scale,
              T* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_m,
              float* __restrict__ part_l, int len_q, int num_heads, int num_kv_heads, int m_query,
              int num_splits, int bshd, const uint8_t* __restrict__ pf_ptr, unsigned long long pf_bytes, const __grid_constant__ AttnAddrs inl) {
    constexpr int NI = D / 32;                 // 16-byte chunks per lane per key row
    constexpr int DC = D / 8;                  // threads covering one V row
    constexpr int NSUB = kAttnThreads / DC;    // key subsets in the PV phase
    __shared__ __align__(16) float s_logit[8 * kAttnRowStride];
    __shared__ float s_m[8], s_l[8];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int hgroups = (m_query + 7) / 8;
    const int split = blockIdx.x;
    const int hk = blockIdx.y / hgroups, hg = blockIdx.y % hgroups;
    const int bq = blockIdx.z, b = bq / len_q, qi = bq % len_q;
    const int mq0 = hg * 8;
    const int mq = min(8, m_query - mq0);
    const int head0 = hk * m_query + mq0;

    pdl_start(!inl.behind);
    // attention barely touches HBM at small batch: use the time to pull a later GEMM's weights into L2
    if (pf_ptr) {
        const int n_cta = gridDim.x * gridDim.y * gridDim.z;
        const int cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
        const int wpc = blockDim.x >> 5;
        l2_prefetch_lines(pf_ptr, (size_t)pf_bytes, cta * wpc + warp, n_cta * wpc, lane);
    }
    pdl_wait();

    const int len_buf = buf_lens[b];
    const int chunk = attn_round16((len_buf + num_splits - 1) / num_splits);
    const int k0 = split * chunk;
    const int k1 = min(len_buf, k0 + chunk);
    const int n = max(0, k1 - k0);

    const size_t stride = bshd ? (size_t)num_kv_heads * D : (size_t)D;
    const size_t base = bshd ? (size_t)hk * D : (size_t)hk * len_buf * D;
    const T* kbase = attn_addr(inl, k_addrs, b, false) + base;
    const T* vbase = attn_addr(inl, v_addrs, b, true) + base;

    const int8_t* mrow = nullptr;
    if (mask) {
        size_t len_off = 0;
        for (int j = 0; j < b; ++j) len_off += buf_lens[j];
        mrow = mask + (size_t)len_q * len_off + (size_t)qi * len_buf;
    }

    // ---- phase 1: S = K.Q^T on tensor cores ----
    uint4 qf[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        qf[i] = (g < mq) ? ld_cg_u4(q + ((size_t)bq * num_heads + head0 + g) * D + i * 32 + t * 8)
                         : make_uint4(0, 0, 0, 0);
    }
    const int ntiles = (n + 15) >> 4;
    for (int tile = warp; tile < ntiles; tile += kAttnWarps) {
        const int ka_i = k0 + tile * 16 + g, kb_i = ka_i + 8;
        const T* pa = kbase + (size_t)min(ka_i, k1 - 1) * stride + t * 8;
        const T* pb = kbase + (size_t)min(kb_i, k1 - 1) * stride + t * 8;
        uint4 ka[NI], kb[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            ka[i] = ld_cg_u4(pa + i * 32);
            kb[i] = ld_cg_u4(pb + i * 32);
        }
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const uint32_t a0[4] = {ka[i].x, kb[i].x, ka[i].y, kb[i].y};
            const uint32_t a1[4] = {ka[i].z, kb[i].z, ka[i].w, kb[i].w};
            mma_attn<T>(acc, a0, qf[i].x, qf[i].y);
            mma_attn<T>(acc, a1, qf[i].z, qf[i].w);
        }
        const bool va = ka_i < k1 && (!mrow || mrow[ka_i] != 0);
        const bool vb = kb_i < k1 && (!mrow || mrow[kb_i] != 0);
        const int la = tile * 16 + g;
        const float ninf = -INFINITY;
        if (2 * t < mq) {
            s_logit[(2 * t) * kAttnRowStride + la] = va ? acc[0] * scale : ninf;
            s_logit[(2 * t) * kAttnRowStride + la + 8] = vb ? acc[2] * scale : ninf;
        }
        if (2 * t + 1 < mq) {
            s_logit[(2 * t + 1) * kAttnRowStride + la] = va ? acc[1] * scale : ninf;
            s_logit[(2 * t + 1) * kAttnRowStride + la + 8] = vb ? acc[3] * scale : ninf;
        }
    }
    __syncthreads();

    // ---- phase 2: masked softmax statistics per head (attention_kernel.cu:434-489) ----
    for (int h = warp; h < mq; h += kAttnWarps) {
        float* row = s_logit + h * kAttnRowStride;
        float mx = -1e20f;
        for (int i = lane; i < n; i += 32) mx = fmaxf(mx, row[i]);
        mx = warp_max(mx);
        float sum = 0.f;
        for (int i = lane; i < n; i += 32) {
            const float e = expf(row[i] - mx);
            row[i] = e;
            sum += e;
        }
        sum = warp_sum(sum) + 1e-20f;
        if (lane == 0) {
            s_m[h] = mx;
            s_l[h] = sum;
        }
    }
    __syncthreads();

    // ---- phase 3: O = P.V on the tensor cores (mma.sync m16n8k16, fp32 accumulate); ZL_ATTN_PV_FP32=1 keeps the CUDA-core
    // loop of the first version (every V element times every head in fp32) for A/B measurements ----
    // A = P [head (8 of 16 rows) x 16 keys]: fp16 models carry p * 2^10 in fp16 (11 significant bits, no subnormals); bf16
    // models carry p as bf16 hi + lo (two MMAs), so that the product keeps ~16 bits of p.  B = V [16 keys x 8 columns]: a B
    // register holds TWO KEYS of one column while V is key-major, so lane (g, t) loads D/8 contiguous elements (columns
    // NJ g ..) of its four keys 2t, 2t+1, 2t+8, 2t+9 and interleaves row pairs with PRMT; n-tile j column c stands for column
    // d = NJ c + j of V (a permutation of the columns, undone when the accumulators are written out).
    constexpr int NJ = D / 8;                 // n-tiles = V columns per lane and key row
    constexpr int NW = NJ / 2;                // 32-bit words of a lane's column chunk (2 elements each)
    constexpr bool kHalf = sizeof(T) == 2 && std::is_same<T, __half>::value;
    float* s_red = s_logit;                   // [warp][h][D], valid after the barrier below
    if constexpr (!PV_FP32) {
        float o[NJ][4];
#pragma unroll
        for (int j = 0; j < NJ; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
        for (int tile = warp; tile < ntiles; tile += kAttnWarps) {
            const int kb = tile * 16;
            uint32_t vw[4][NW];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int kk = kb + 2 * t + (r & 1) + (r >> 1) * 8;
#pragma unroll
                for (int w = 0; w < NW; ++w) vw[r][w] = 0u;
                if (kk < n) {
                    const T* src = vbase + (size_t)(k0 + kk) * stride + g * NJ;
#pragma unroll
                    for (int w4 = 0; w4 < NW / 4; ++w4) {
                        const uint4 v = ld_cg_u4(src + w4 * 8);
                        vw[r][w4 * 4 + 0] = v.x, vw[r][w4 * 4 + 1] = v.y, vw[r][w4 * 4 + 2] = v.z, vw[r][w4 * 4 + 3] = v.w;
                    }
                }
            }
            uint32_t af[4] = {0u, 0u, 0u, 0u}, al[4] = {0u, 0u, 0u, 0u};
            if (g < mq) {
                const float* pr = s_logit + g * kAttnRowStride + kb + 2 * t;
                const float2 p0 = *reinterpret_cast<const float2*>(pr), p1 = *reinterpret_cast<const float2*>(pr + 8);
                const float q0 = kb + 2 * t < n ? p0.x : 0.f, q1 = kb + 2 * t + 1 < n ? p0.y : 0.f;
                const float q2 = kb + 2 * t + 8 < n ? p1.x : 0.f, q3 = kb + 2 * t + 9 < n ? p1.y : 0.f;
                if constexpr (kHalf) {
                    const __half2 h0 = __floats2half2_rn(q0 * 1024.f, q1 * 1024.f), h1 = __floats2half2_rn(q2 * 1024.f, q3 * 1024.f);
                    af[0] = *reinterpret_cast<const uint32_t*>(&h0);
                    af[2] = *reinterpret_cast<const uint32_t*>(&h1);
                } else {
                    const __nv_bfloat162 h0 = __floats2bfloat162_rn(q0, q1), h1 = __floats2bfloat162_rn(q2, q3);
                    const float2 f0 = __bfloat1622float2(h0), f1 = __bfloat1622float2(h1);
                    const __nv_bfloat162 l0 = __floats2bfloat162_rn(q0 - f0.x, q1 - f0.y), l1 = __floats2bfloat162_rn(q2 - f1.x, q3 - f1.y);
                    af[0] = *reinterpret_cast<const uint32_t*>(&h0);
                    af[2] = *reinterpret_cast<const uint32_t*>(&h1);
                    al[0] = *reinterpret_cast<const uint32_t*>(&l0);
                    al[2] = *reinterpret_cast<const uint32_t*>(&l1);
                }
            }
#pragma unroll
            for (int w = 0; w < NW; ++w) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {            // element 2 w + e of the chunk = n-tile j
                    const uint32_t sel = e ? 0x7632u : 0x5410u;
                    const uint32_t b0 = __byte_perm(vw[0][w], vw[1][w], sel), b1 = __byte_perm(vw[2][w], vw[3][w], sel);
                    mma_attn<T>(o[2 * w + e], af, b0, b1);
                    if constexpr (!kHalf) mma_attn<T>(o[2 * w + e], al, b0, b1);
                }
            }
        }
        __syncthreads();   // everyone is done reading probabilities; reuse s_logit as the reduction buffer
        if (g < mq) {
            const float sc = kHalf ? (1.f / 1024.f) : 1.f;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                s_red[(warp * 8 + g) * D + NJ * (2 * t) + j] = o[j][0] * sc;
                s_red[(warp * 8 + g) * D + NJ * (2 * t + 1) + j] = o[j][1] * sc;
            }
        }
    } else {
        const int dc = tid % DC, sub = tid / DC;
        float o[8][8];
#pragma unroll
        for (int h = 0; h < 8; ++h)
#pragma unroll
            for (int i = 0; i < 8; ++i) o[h][i] = 0.f;
        const T* vp = vbase + (size_t)k0 * stride + dc * 8;
        constexpr int U = 4;
        for (int key = sub; key < n; key += NSUB * U) {
            uint4 vv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int kk = key + u * NSUB;
                if (kk < n) vv[u] = ld_cg_u4(vp + (size_t)kk * stride);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int kk = key + u * NSUB;
                if (kk < n) {
                    float vf[8];
                    unpack8<T>(vv[u], vf);
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        if (h < mq) {
                            const float p = s_logit[h * kAttnRowStride + kk];
#pragma unroll
                            for (int i = 0; i < 8; ++i) o[h][i] = fmaf(p, vf[i], o[h][i]);
                        }
                    }
                }
            }
        }
        // reduce key subsets: inside the warp first (lanes with equal dc), then across warps via smem
#pragma unroll
        for (int h = 0; h < 8; ++h)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float v = o[h][i];
#pragma unroll
                for (int off = DC; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                o[h][i] = v;
            }
        __syncthreads();   // everyone is done reading probabilities; reuse s_logit as the reduction buffer
        if (lane < DC) {
#pragma unroll
            for (int h = 0; h < 8; ++h)
                if (h < mq) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) s_red[(warp * 8 + h) * D + lane * 8 + i] = o[h][i];
                }
        }
    }
    __syncthreads();
    float* s_all = s_red + kAttnWarps * 8 * D;   // the CTA's results, for the others of a cluster
    static_assert((kAttnWarps + 1) * 8 * D <= 8 * kAttnRowStride, "shared memory");
    for (int e = tid; e < mq * D; e += kAttnThreads) {
        const int h = e / D, d = e % D;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) v += s_red[(w * 8 + h) * D + d];
        v = v / s_l[h];
        const size_t vh = (size_t)bq * num_heads + head0 + h;
        if (num_splits == 1) {
            out[vh * D + d] = from_f32<T>(v);
        } else if (!part_o) {
            s_all[e] = v;
        } else {
            part_o[(vh * num_splits + split) * D + d] = v;
            if (d == 0) {
                part_m[vh * num_splits + split] = s_m[h];
                part_l[vh * num_splits + split] = s_l[h];
            }
        }
    }
    if (num_splits > 1 && !part_o)   // the splits are a cluster
        attn_merge_cluster<T, D, kAttnThreads>(s_all, s_m, s_l, num_splits, split, mq, out + ((size_t)bq * num_heads + head0) * D);
}


// ---------------------------------------------------------------------------------------------------------
// Latency-optimised variant for the small-batch / short-context regime (B200: 148 SMs, a B=1 decode step has
// 8 kv-heads of work): 512 threads, at most 256 keys per CTA, and EVERY global load of the CTA (q, its K tile,
// its V rows) is issued before the first dependent instruction, so the whole CTA costs one memory round trip
// instead of one per loop iteration.  Same math and split/combine contract as k_decode_attn.
// ---------------------------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(kShortThreads)
k_decode_attn_short(const T* __restrict__ q, const int32_t* __restrict__ buf_lens, T* const* __restrict__ k_addrs,
                    T* const* __restrict__ v_addrs, const int8_t* __restrict__ mask, float scale,
                    T* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_m,
                    float* __restrict__ part_l, int len_q, int num_heads, int num_kv_heads, int m_query,
                    int num_splits, int bshd, const uint8_t* __restrict__ pf_ptr, unsigned long long pf_bytes) {
    extern __shared__ __align__(16) float s_dyn[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_trigger();
    // attention barely touches HBM at small batch: use the time to pull a later GEMM's weights into L2
    if (pf_ptr) {
        const int n_cta = gridDim.x * gridDim.y * gridDim.z;
        const int cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
        const int wpc = blockDim.x >> 5;
        l2_prefetch_lines(pf_ptr, (size_t)pf_bytes, cta * wpc + warp, n_cta * wpc, lane);
    }
    pdl_wait();
    attn_short_item<T, D>(q, buf_lens, k_addrs, v_addrs, mask, scale, out, part_o, part_m, part_l, len_q, num_heads,
                          num_kv_heads, m_query, num_splits, bshd, (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z,
                          s_dyn);
}


// grid (B*len_q*num_heads), block D
template <typename T>
__global__ void k_attn_combine(const float* __restrict__ part_o, const float* __restrict__ part_m,
                               const float* __restrict__ part_l, T* __restrict__ out, int num_splits) {
    const int vh = blockIdx.x, D = blockDim.x, d = threadIdx.x;
    pdl_trigger();
    pdl_wait();
    const float* pm = part_m + (size_t)vh * num_splits;
    const float* pl = part_l + (size_t)vh * num_splits;
    float gm = -1e20f;
    for (int i = 0; i < num_splits; ++i) gm = fmaxf(gm, pm[i]);
    float gs = 0.f;
    for (int i = 0; i < num_splits; ++i) gs += pl[i] * expf(pm[i] - gm);
    float res = 0.f;
    for (int i = 0; i < num_splits; ++i) {
        const float w = pl[i] / gs * expf(pm[i] - gm);
        res += part_o[((size_t)vh * num_splits + i) * D + d] * w;
    }
    out[(size_t)vh * D + d] = from_f32<T>(res);
}

// grid.x, the key splits of a head group, as a cluster or not
template <typename... KArgs, typename... Args>
static cudaError_t launch_splits(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl, bool cluster, Args... args) {
    if (!cluster) return launch(kernel, grid, block, smem, stream, pdl, args...);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = grid.x;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    zl_count_launch();
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// CTAs of an SM.  The lengths of the sequences are on the device, so a choice has to hold for all of them.  us, caches all of one length, random ones from half of it on, an
// even spread down to a quarter, every fourth one whole beside eighths; 32 heads on 8, in a graph.
//   D = 128, up to three CTAs per SM: three, whose registers hold more loads.  fp16, four / three: 24 x 2048 42.8 / 41.1, 38.7 / 37.1, 36.7 / 35.6, 21.2 / 20.3.
//   fp16, more: four, 128 registers; a wave of four is two of three: 16 x 4096 50.7 / 69.9, 45.8 / 60.9, 41.1 / 40.7, 31.7 / 30.0; 64 x 1000 50.7 / 67.6, 43.3 / 52.2, 40.0 / 36.4,
//   26.1 / 28.6: only the spread gains by three, where the places of short sequences are taken again.
//   bf16, more: four have too few registers (24 bytes are spilled), so three, unless that is a wave more, beyond the first one of four: 32 x 4096 108 / 114, 93.4 / 95.8,
//   71.9 / 75.8, 59.5 / 58.4; against it 40 x 4096 138 / 126, 111 / 108, 92.8 / 87.5, 73.3 / 68.3; 24 x 4096 90.2 / 84.0, 74.1 / 71.0, 57.1 / 55.8, 54.5 / 49.1.  Within the first one
//   what the lengths are decides, 64 x 1000 55.7 / 71.0, 47.6 / 54.8, 43.2 / 37.6, 27.8 / 29.6, and it stays at three.
//   D = 64: five (96 registers), for bf16 four (100) where these are all: 16 x 4096, five / four, 36.3 / 34.0, 33.2 / 31.6, 22.5 / 21.2, 19.5 / 19.0.  Six hold a fifth more CTAs in a
//   wave, but spill: fp16 24 x 4096, five / six, 61.5 / 60.2, 46.9 / 52.7, 33.4 / 43.8, 19.6 / 21.5.
//   Six without a word to the compiler, 80 registers and no spill, where the rows of a prompt, all of one length, are one wave of them: 48 rows on 148 keys, 16 heads on 16, fp16 9.8 -> 7.9.
static int attn_per_sm(int dim_head, bool fp16, bool one_length, long long ctas) {
    const long long sms = device_sm_count();
    auto waves = [&](int per) { return (ctas + per * sms - 1) / (per * sms); };
    if (dim_head == 64) return one_length && waves(6) < waves(5) ? 6 : fp16 || ctas > 4 * sms ? 5 : 4;
    if (ctas <= 3 * sms) return 3;
    return fp16 || (ctas > 4 * sms && waves(4) < waves(3)) ? 4 : 3;
}
// The splits of a head group as a cluster, which merges their results (attn_merge_cluster), or through the workspace and a second launch.  us, launch / cluster, fp16, D = 128.
// 256-key CTAs are a cluster where the device has room for all clusters with one CTA per SM: 8 x 500 9.9 / 8.7, 4 x 1000 10.6 / 8.8, 2 x 1500 11.1 / 8.9 (96 CTAs by six), 13 x 2000, 8 heads on 1,
// 11.5 / 9.1 (104 by eight); where it has not, some SMs work twice as long: 6 x 760 10.9 / 15.9 (144 CTAs by three), 18 x 1000, 8 on 2, 11.0 / 16.0 (144 by four), 2 x 2000 11.8 / 16.9 (128
// by eight).
// 1024-key CTAs: two or four splits in one wave, 16 x 4096 55.1 / 50.7, 20 x 1500 32.4 / 31.0; in more where each split is long, 32 x 4096 101 / 97.9, against it 32 x 1100 (16 heads on
// 16, every fourth one whole) 29.4 / 30.6.  Three find their places badly: 18 x 3000 46.7 / 67.8; 2048 CTAs gain nothing: 32 x 4096 (16 on 16, D = 64) 108 / 109.
static bool attn_cluster(bool use_short, int splits, long long ctas, int max_len_buf, int dim_head, int per_sm) {
    const long long sms = device_sm_count();
    if (use_short) {
        static ClustersFit fit;
        return splits <= kAttnClusterSplits && ctas / splits <= clusters_at_once(k_decode_attn_warp<__half, 128>, kWarpAttnWarps * 32, 160 * 1024, splits, fit);
    }
    if (splits != 2 && splits != 4) return false;
    return ctas <= per_sm * sms || (!(dim_head == 128 && per_sm == 3) && ctas <= 8 * sms && max_len_buf >= 800 * splits);
}

static int attn_num_splits(int B, int len_q, int num_kv_heads, int m_query, int max_len_buf) {
    const int hgroups = (m_query + 7) / 8;
    const int base = B * len_q * num_kv_heads * hgroups;
    const int min_splits = cdiv(max_len_buf, kAttnMaxRange);
    const int want = cdiv(2 * 148, base);
    const int max_useful = cdiv(max_len_buf, 256) > 0 ? cdiv(max_len_buf, 256) : 1;   // >= 256 keys per split
    int s = want < max_useful ? want : max_useful;
    if (s > kAttnMaxSplits) s = kAttnMaxSplits;
    if (s < min_splits) s = min_splits;
    if (s < 1) s = 1;
    return s;
}

}  // namespace zl

using namespace zl;

// one-shot prefetch hint consumed by the next zl_decode_attention call on this thread (set by the decode driver)
static thread_local const uint8_t* g_attn_pf_ptr = nullptr;
static thread_local unsigned long long g_attn_pf_bytes = 0;
extern "C" int zl_decode_attention_set_prefetch(const void* ptr, size_t bytes) {
    g_attn_pf_ptr = static_cast<const uint8_t*>(ptr);
    g_attn_pf_bytes = bytes;
    return ZL_OK;
}
// one-shot as well: the layers of a prompt's portion share its mask, whose bits the first one's call has left in the workspace
static thread_local bool g_attn_mask_ready = false;
extern "C" int zl_decode_attention_same_mask(void) {
    g_attn_mask_ready = true;
    return ZL_OK;
}

extern "C" size_t zl_decode_attention_workspace_bytes(int B, int len_q, int num_heads, int dim_head,
                                                      int max_len_buf) {
    if (B <= 0 || len_q <= 0 || num_heads <= 0 || dim_head <= 0) return 0;
    int splits = cdiv(max_len_buf > 0 ? max_len_buf : 1, kAttnMaxRange);
    if (splits < kAttnMaxSplits) splits = kAttnMaxSplits;
    return (size_t)B * len_q * num_heads * splits * (dim_head + 2) * sizeof(float);
}

// Splits of a call on len_q = 1 and how they run: the kernel of 256-key CTAs, or that of 1024-key ones and its CTAs of an SM.
struct AttnPlan {
    int splits, per_sm;   // per_sm 0: 256-key CTAs
    long long ctas;
};
static AttnPlan attn_plan(int B, int len_q, int num_kv_heads, int m_query, int dim_head, int max_len_buf, bool fp16) {
    const long long groups = (long long)B * len_q * num_kv_heads * cdiv(m_query, 8);
    // latency regime: few CTAs of work -> 256-key CTAs that issue all their loads up front
    const int short_splits = cdiv(max_len_buf, kShortRange);
    if (short_splits <= kAttnMaxSplits && groups * short_splits <= 4 * 148) return AttnPlan{short_splits, 0, groups * short_splits};
    const int splits = attn_num_splits(B, len_q, num_kv_heads, m_query, max_len_buf);
    return AttnPlan{splits, attn_per_sm(dim_head, fp16, B == 1 && len_q > 1, groups * splits), groups * splits};
}
extern "C" int zl_decode_attention_plan(int B, int num_heads, int num_kv_heads, int dim_head, int max_len_buf, int dtype, int* splits, int* per_sm) {
    ZL_CHECK_ARG(B > 0 && num_heads > 0 && num_kv_heads > 0 && num_heads % num_kv_heads == 0 && max_len_buf > 0 && splits && per_sm);
    ZL_CHECK_SUPPORTED((dim_head == 64 || dim_head == 128) && (dtype == ZL_F16 || dtype == ZL_BF16));
    const AttnPlan plan = attn_plan(B, 1, num_kv_heads, num_heads / num_kv_heads, dim_head, max_len_buf, dtype == ZL_F16);
    *splits = plan.splits;
    *per_sm = plan.per_sm;
    return plan.splits > 1 && attn_cluster(plan.per_sm == 0, plan.splits, plan.ctas, max_len_buf, dim_head, plan.per_sm) ? 1 : 0;
}

extern "C" unsigned zl_prompt_attention_watchdog(void) {
    cudaDeviceSynchronize();
    const unsigned* words = wait_words();
    return words ? words[kWaitAttnPrompt] : 0u;
}

extern "C" int zl_prompt_attention_ranges(int B, int len_q, int num_heads, int num_kv_heads, int max_len_buf) {
    if (B <= 0 || len_q <= 0 || num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads || max_len_buf <= 0) return 0;
    const long long groups = (long long)cdiv(len_q * (num_heads / num_kv_heads), kPaRows) * num_kv_heads * B;
    return prompt_attn_splits(groups, cdiv(max_len_buf, kPaKeys), prompt_attn_fit(8));
}
extern "C" int zl_prompt_attention_smem_bytes(int dim_head) {
    return dim_head == 64 ? PaCfg<64>::kBytes : dim_head == 128 ? PaCfg<128>::kBytes : 0;
}

// Workspace of the prompt kernel: the mask's bits, then the last visible keys.
static size_t prompt_head_bytes(int B, int len_q, int max_len_buf, const int8_t* mask) {
    const size_t q_rows = (size_t)B * len_q;
    return mask ? (q_rows * cdiv(max_len_buf, kPaKeys) * 8 + 15) / 16 * 16 + (q_rows * 4 + 15) / 16 * 16 : 0;
}
// Which kernel serves several query rows.  The decode kernels read K and V once per query row and stay at their latency while these reads
// fit one wave; the prompt kernel reads them once per 128 (query, head) rows and has a mask pass and a longer chain.  Measured in 256-key
// CTAs of the decode kernels, all launches of a call, decode against prompt kernel in us, D = 128, 1100 keys: 32 heads on 8, 80 CTAs 12.1
// against 15.3, 160 CTAs 18.0 against 15.6; 64 on 8, 160 CTAs 21.4 against 15.6; 16 on 8, 160 CTAs 17.0 against 15.6; 8 on 8, 360 CTAs
// 22.7 against 15.6; 300 keys, 144 CTAs 11.6 against 14.8.  D = 64 halves the reads but not the chain: 32 on 8, 160 CTAs 12.3
// against 12.6, 256 CTAs (32 rows alone) 6.0 against 8.0, 360 CTAs 16.2 against 12.8; 12 on 4, 320 CTAs 15.6 against 12.7; one head per
// kv head: 16 on 16, 720 CTAs 13.7 against 15.0, 1024 CTAs 8.2 against 8.4, 1280 CTAs 17.4 against 15.2.  The mask's bits live in the
// workspace, so a masked call without room for them keeps the decode kernels.
static bool prompt_route(int len_q, int m_query, int dim_head, int B, int num_kv_heads, const int8_t* mask, int max_len_buf, const void* out,
                         const void* workspace, size_t workspace_bytes) {
    if (len_q < 2 || num_kv_heads > 65535 || B > 65535 / 16) return false;
    const long long ctas = (long long)B * len_q * num_kv_heads * cdiv(m_query, 8) * cdiv(max_len_buf, 256);
    const long long line = dim_head == 128 ? 150 : m_query > 1 ? 300 : 1000;
    if (ctas < line) return false;
    if ((reinterpret_cast<uintptr_t>(out) & 3) || (reinterpret_cast<uintptr_t>(workspace) & 15)) return false;
    return !mask || (workspace && prompt_head_bytes(B, len_q, max_len_buf, mask) <= workspace_bytes && len_q <= 65535);
}

// Addresses of the caches that a caller holds on the host: B of K, then B of V; table: room for them on the device.
struct HostAddrs {
    const void* addrs;   // null: the tables are the caller's
    void* table;
};
// They travel with the call's first kernel, `ctas` of them, which is then a programmatic dependent behind everything earlier, or a launch before it writes the table,
// behind everything earlier as well, so that the attention may start under its end.  Up to one CTA per SM the launch of 1.3 us is saved: us in a row of calls, table /
// inline, 32 heads on 8: 4 x 300 9.2 / 8.3, 2 x 17 8.2 / 6.1, a portion of 33 behind 567 14.4 / 13.7 (in a graph).  More CTAs come while the kernel before ends are placed where it
// ends first, several on an SM, and stay there: 16 x 4096 with heads of 64 21.6 / 27.2, 500 behind 1000 32.9 / 33.5; as plain launches 32.9 / 34.6.
static int attn_addresses(const HostAddrs& host, int B, long long ctas, bool only_tables, AttnAddrs& inl, void* const*& k_addrs, void* const*& v_addrs, int& pdl,
                          zl_stream_t stream) {
    if (!host.addrs) return ZL_OK;
    pdl = 1;
    if (B <= kAttnInline && ctas <= device_sm_count() && !only_tables) {
        for (int i = 0; i < 2 * B; ++i) inl.p[i] = static_cast<const void* const*>(host.addrs)[i];
        inl.n = B;
        inl.behind = 1;
        return ZL_OK;
    }
    k_addrs = static_cast<void* const*>(host.table);
    v_addrs = k_addrs + B;
    return zl_write_pointers(host.table, host.addrs, 2 * B, stream);
}

template <typename T, int D>
static int prompt_attention(const void* q, const int32_t* buf_lens, void* const* k_addrs, void* const* v_addrs, const int8_t* mask, float scale,
                            int max_len_buf, void* out, int B, int len_q, int num_heads, int num_kv_heads, int bshd, void* workspace,
                            size_t workspace_bytes, int pdl, bool mask_ready, const HostAddrs& host, zl_stream_t stream) {
    const int m_query = num_heads / num_kv_heads;
    const int blocks = cdiv(len_q * m_query, kPaRows), tiles = cdiv(max_len_buf, kPaKeys);
    const long long groups = (long long)blocks * num_kv_heads * B;
    const int splits = prompt_attn_splits(groups, tiles, prompt_attn_fit(8));
    const size_t q_rows = (size_t)B * len_q;
    uint64_t* bits = mask ? static_cast<uint64_t*>(workspace) : nullptr;
    int32_t* last = mask ? reinterpret_cast<int32_t*>(static_cast<uint8_t*>(workspace) + (q_rows * tiles * 8 + 15) / 16 * 16) : nullptr;
    ZL_CHECK_WAITS();
    unsigned* words = wait_words();
    ZL_CHECK_CUDA(words ? cudaSuccess : cudaErrorMemoryAllocation);
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        ZL_CHECK_CUDA(cudaFuncSetAttribute(k_attn_prompt<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, PaCfg<D>::kAloneBytes));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const bool mask_pass = mask && !mask_ready;
    AttnAddrs inl = {};
    const int rc = attn_addresses(host, B, mask_pass ? (long long)len_q * B : groups * splits, false, inl, k_addrs, v_addrs, pdl, stream);
    if (rc) return rc;
    if (mask_pass)
        ZL_CHECK_CUDA(launch(k_mask_bits, dim3(len_q, B), dim3(256), 0, stream, pdl != 0, mask, buf_lens, bits, last, len_q, tiles, inl.behind));
    AttnAddrs own = inl;
    own.behind = inl.behind && !mask_pass;
    const int aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    // behind the mask's kernel the attention may start early whatever the caller's chain allows: it waits for that kernel to end
    ZL_CHECK_CUDA((launch_attn_prompt<T, D>(dim3(blocks, num_kv_heads, B * splits), splits, groups <= prompt_attn_fit(splits), stream, pdl != 0 || mask_pass, (const T*)q, buf_lens,
                                            (T* const*)k_addrs, (T* const*)v_addrs, (const uint64_t*)bits, (const int32_t*)last, tiles, scale,
                                            (T*)out, len_q, num_heads, num_kv_heads, m_query, splits, bshd, aligned, words + kWaitAttnPrompt, own)));
    g_attn_pf_ptr = nullptr;
    g_attn_pf_bytes = 0;
    return ZL_OK;
}

static int attention(const void* q, const int32_t* buf_lens, void* const* k_addrs, void* const* v_addrs, const HostAddrs& host, const int8_t* mask, float scale,
                     int max_len_buf, void* out, int B, int len_q, int num_heads, int num_kv_heads, int dim_head, int bshd, void* workspace,
                     size_t workspace_bytes, int dtype, int pdl, zl_stream_t stream) {
    const bool mask_ready = g_attn_mask_ready;
    g_attn_mask_ready = false;
    ZL_CHECK_ARG(q && buf_lens && (host.addrs || (k_addrs && v_addrs)) && out && B > 0 && len_q > 0 && max_len_buf > 0);
    ZL_CHECK_ARG(num_heads > 0 && num_kv_heads > 0 && num_heads % num_kv_heads == 0);
    ZL_CHECK_SUPPORTED(dim_head == 64 || dim_head == 128);
    ZL_CHECK_SUPPORTED(dtype == ZL_F16 || dtype == ZL_BF16);
    const int m_query = num_heads / num_kv_heads;
    if (prompt_route(len_q, m_query, dim_head, B, num_kv_heads, mask, max_len_buf, out, workspace, workspace_bytes)) {
        if (dtype == ZL_F16)
            return dim_head == 128 ? prompt_attention<__half, 128>(q, buf_lens, k_addrs, v_addrs, mask, scale, max_len_buf, out, B, len_q, num_heads,
                                                                   num_kv_heads, bshd, workspace, workspace_bytes, pdl, mask_ready, host, stream)
                                   : prompt_attention<__half, 64>(q, buf_lens, k_addrs, v_addrs, mask, scale, max_len_buf, out, B, len_q, num_heads,
                                                                  num_kv_heads, bshd, workspace, workspace_bytes, pdl, mask_ready, host, stream);
        return dim_head == 128 ? prompt_attention<__nv_bfloat16, 128>(q, buf_lens, k_addrs, v_addrs, mask, scale, max_len_buf, out, B, len_q,
                                                                      num_heads, num_kv_heads, bshd, workspace, workspace_bytes, pdl, mask_ready, host, stream)
                               : prompt_attention<__nv_bfloat16, 64>(q, buf_lens, k_addrs, v_addrs, mask, scale, max_len_buf, out, B, len_q,
                                                                     num_heads, num_kv_heads, bshd, workspace, workspace_bytes, pdl, mask_ready, host, stream);
    }
    const AttnPlan plan = attn_plan(B, len_q, num_kv_heads, m_query, dim_head, max_len_buf, dtype == ZL_F16);
    const int splits = plan.splits, per_sm = plan.per_sm;
    const bool use_short = per_sm == 0;
    const size_t vheads = (size_t)B * len_q * num_heads;
    float* part_o = nullptr;
    float* part_m = nullptr;
    float* part_l = nullptr;
    if (splits > 1) {
        const size_t need = vheads * splits * (dim_head + 2) * sizeof(float);
        ZL_CHECK_ARG(workspace != nullptr && workspace_bytes >= need);
    }
    static const bool old_short = getenv("ZL_ATTN_OLD_SHORT") != nullptr;
    static const bool pv_fp32 = getenv("ZL_ATTN_PV_FP32") != nullptr;
    const bool cluster = splits > 1 && !(use_short && old_short) && attn_cluster(use_short, splits, plan.ctas, max_len_buf, dim_head, per_sm);
    AttnAddrs inl = {};
    const int rc = attn_addresses(host, B, plan.ctas, use_short && old_short, inl, k_addrs, v_addrs, pdl, stream);
    if (rc) return rc;
    if (splits > 1 && !cluster) {
        part_o = static_cast<float*>(workspace);
        part_m = part_o + vheads * splits * dim_head;
        part_l = part_m + vheads * splits;
    }
    const int hgroups = (m_query + 7) / 8;
    dim3 grid(splits, num_kv_heads * hgroups, B * len_q), block(kAttnThreads);
    // default for the latency regime: the warp-per-32-keys kernel (one __syncthreads per CTA); ZL_ATTN_OLD_SHORT=1 keeps the
    // previous 512-thread short kernel for A/B measurements
    const bool use_warp = use_short && !old_short;
#define ZL_ATTN_LAUNCH(TT, DD)                                                                                  \
    if (use_warp) {                                                                                             \
        ZL_CHECK_CUDA(launch_splits(k_decode_attn_warp<TT, DD>, grid, dim3(kWarpAttnWarps * 32),                \
                             (size_t)warp_attn_smem_floats<DD>() * sizeof(float), stream, pdl != 0, cluster, (const TT*)q, \
                             buf_lens, (TT* const*)k_addrs, (TT* const*)v_addrs, mask, scale, (TT*)out, part_o, \
                             part_m, part_l, len_q, num_heads, num_kv_heads, m_query, splits, bshd, inl));       \
    } else if (use_short) {                                                                                     \
        static bool attr_set = false;                                                                           \
        if (!attr_set) {                                                                                        \
            ZL_CHECK_CUDA(cudaFuncSetAttribute(k_decode_attn_short<TT, DD>,                                     \
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,                     \
                                               short_smem_bytes<DD>()));                                        \
            attr_set = true;                                                                                    \
        }                                                                                                       \
        ZL_CHECK_CUDA(launch(k_decode_attn_short<TT, DD>, grid, dim3(kShortThreads), short_smem_bytes<DD>(),    \
                             stream, pdl != 0, (const TT*)q, buf_lens, (TT* const*)k_addrs,                     \
                             (TT* const*)v_addrs, mask, scale, (TT*)out, part_o, part_m, part_l, len_q,         \
                             num_heads, num_kv_heads, m_query, splits, bshd, g_attn_pf_ptr, g_attn_pf_bytes));                                  \
    } else                                                                                                      \
    if (pv_fp32) {                                                                                              \
        ZL_CHECK_CUDA(launch_splits(k_decode_attn<TT, DD, true, 4>, grid, block, 0, stream, pdl != 0, cluster, (const TT*)q, buf_lens, \
                             (TT* const*)k_addrs, (TT* const*)v_addrs, mask, scale, (TT*)out, part_o, part_m,   \
                             part_l, len_q, num_heads, num_kv_heads, m_query, splits, bshd, g_attn_pf_ptr,      \
                             g_attn_pf_bytes, inl));                                                            \
    } else                                                                                                      \
    ZL_CHECK_CUDA(launch_splits(per_sm == 6 ? k_decode_attn<TT, DD, false, DD == 64 ? 0 : 4> : per_sm == 4 ? k_decode_attn<TT, DD, false, 4> : k_decode_attn<TT, DD, false, DD == 128 ? 3 : 5>, grid, block, 0, stream, pdl != 0, cluster, (const TT*)q, buf_lens, \
                         (TT* const*)k_addrs, (TT* const*)v_addrs, mask, scale, (TT*)out, part_o, part_m,       \
                         part_l, len_q, num_heads, num_kv_heads, m_query, splits, bshd, g_attn_pf_ptr, g_attn_pf_bytes, inl)); \
    if (part_o)                                                                                                 \
        ZL_CHECK_CUDA(launch(k_attn_combine<TT>, dim3((unsigned)vheads), dim3(DD), 0, stream, pdl != 0,         \
                             (const float*)part_o, (const float*)part_m, (const float*)part_l, (TT*)out, splits));
    if (dtype == ZL_F16) {
        if (dim_head == 128) { ZL_ATTN_LAUNCH(__half, 128) } else { ZL_ATTN_LAUNCH(__half, 64) }
    } else {
        if (dim_head == 128) { ZL_ATTN_LAUNCH(__nv_bfloat16, 128) } else { ZL_ATTN_LAUNCH(__nv_bfloat16, 64) }
    }
#undef ZL_ATTN_LAUNCH
    g_attn_pf_ptr = nullptr;
    g_attn_pf_bytes = 0;
    return ZL_OK;
}

extern "C" int zl_decode_attention(const void* q, const int32_t* buf_lens, void* const* k_addrs, void* const* v_addrs, const int8_t* mask, float scale,
                                   int max_len_buf, void* out, int B, int len_q, int num_heads, int num_kv_heads, int dim_head, int bshd,
                                   void* workspace, size_t workspace_bytes, int dtype, int pdl, zl_stream_t stream) {
    return attention(q, buf_lens, k_addrs, v_addrs, HostAddrs{}, mask, scale, max_len_buf, out, B, len_q, num_heads, num_kv_heads, dim_head, bshd, workspace,
                     workspace_bytes, dtype, pdl, stream);
}

extern "C" int zl_decode_attention_host(const void* q, const int32_t* buf_lens, const void* addrs, void* table, const int8_t* mask, float scale, int max_len_buf,
                                        void* out, int B, int len_q, int num_heads, int num_kv_heads, int dim_head, int bshd, void* workspace,
                                        size_t workspace_bytes, int dtype, zl_stream_t stream) {
    ZL_CHECK_ARG(addrs && table);
    return attention(q, buf_lens, nullptr, nullptr, HostAddrs{addrs, table}, mask, scale, max_len_buf, out, B, len_q, num_heads, num_kv_heads, dim_head, bshd,
                     workspace, workspace_bytes, dtype, 1, stream);
}
