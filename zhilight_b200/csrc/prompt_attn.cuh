// Attention of several query rows per task (portions of a prompt, beam and tree rows) over per-task ragged KV buffers: the
// counterpart of the decode kernels for len_q > 1.  Replaces nn::multi_query_attention_rag_buffer with len_q > 1
// (reference src/nn/attention/attention_kernel.cu:1252-1457), same softmax: mask ? scale * s : -inf, maximum from -1e20, sum
// from 1e-20, so a row that sees nothing gives zeros.
//
// The decode kernels give every query row a CTA of its own, which reads the task's whole K and V again: 512 rows behind 588
// bf16 positions, 32 heads on 8, take 306 us so and 58 us here (fp16: 287 and 45).  A CTA owns 64 (query, head) rows of one kv
// head -- all heads of the group share the tile -- and walks the keys 64 at a time with running maxima: 16 rows per warp,
// S = Q K^T and O += P V on mma.sync, K and V tiles double-buffered in shared memory through cp.async.  fp16 models carry
// p * 2^10 in fp16, bf16 models p as bf16 hi + lo (two MMAs), as the decode kernels do.  Bound by the mma.sync rate (64-key tile
// and warp: 64 MMAs for S, 64 or 128 for O, one per 8 cycles and scheduler).
//
// An int8 mask is turned into bits first (k_mask_bits), once for all kv heads, together with each row's last visible key: tiles
// behind the last key any row of the block sees are never loaded, which halves a causal prompt's work.
#pragma once
#include "common.cuh"

#include <type_traits>

namespace zl {

constexpr int kPaRows = 64, kPaKeys = 64, kPaThreads = 128;

template <int D>
constexpr int prompt_attn_smem_bytes() { return 2 * 2 * kPaKeys * D * 2; }   // two stages of K and V

// mask rows -> bits.  grid (len_q, B), 256 threads; bits [B][len_q][pitch64] with zero words behind len_buf, last [B][len_q]: index
// of the last visible key, -1 for none
__global__ void __launch_bounds__(256) k_mask_bits(const int8_t* __restrict__ mask, const int32_t* __restrict__ buf_lens, uint64_t* bits,
                                                   int32_t* last, int len_q, int pitch64) {
    __shared__ int s_last[8];
    pdl_trigger();
    pdl_wait();
    const int qi = blockIdx.x, b = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    size_t off = 0;
    for (int j = 0; j < b; ++j) off += buf_lens[j];
    const int n = buf_lens[b];
    const int8_t* row = mask + (size_t)len_q * off + (size_t)qi * n;
    uint32_t* dst = reinterpret_cast<uint32_t*>(bits + ((size_t)b * len_q + qi) * pitch64);
    int mine = -1;
    const int words = pitch64 * 2;
    for (int w0 = warp * 4; w0 < words; w0 += 32) {   // four loads in flight per lane
        int8_t v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = (w0 + u) * 32 + lane;
            v[u] = i < n ? row[i] : (int8_t)0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t m = __ballot_sync(0xffffffffu, v[u] != 0);
            if (m && w0 + u < words) mine = (w0 + u) * 32 + 31 - __clz((int)m);
            if (lane == 0 && w0 + u < words) dst[w0 + u] = m;
        }
    }
    if (lane == 0) s_last[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) mine = max(mine, s_last[w]);
        last[(size_t)b * len_q + qi] = mine;
    }
}

template <typename T>
__device__ __forceinline__ void pa_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if constexpr (std::is_same<T, __half>::value) mma_16816_f16(d, a, b0, b1, d);
    else mma_16816_bf16(d, a, b0, b1, d);
}
// 16-byte chunk c of row r of a tile with D / 8 chunks per row: xor by the row keeps ldmatrix free of bank conflicts
template <int D>
__device__ __forceinline__ uint32_t pa_off(int r, int c) { return (uint32_t)(r * (D * 2) + ((c ^ (r & 7)) << 4)); }
__device__ __forceinline__ void pa_cp16(uint32_t dst, const void* src, bool in) {
    const int bytes = in ? 16 : 0;   // 0: zero fill, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pa_ldm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void pa_ldm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
template <typename T>
__device__ __forceinline__ void pa_pack(float x, float y, uint32_t& hi, uint32_t& lo) {
    if constexpr (std::is_same<T, __half>::value) {
        const __half2 h = __floats2half2_rn(x * 1024.f, y * 1024.f);
        hi = *reinterpret_cast<const uint32_t*>(&h);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        const float2 f = __bfloat1622float2(h);
        const __nv_bfloat162 l = __floats2bfloat162_rn(x - f.x, y - f.y);
        hi = *reinterpret_cast<const uint32_t*>(&h);
        lo = *reinterpret_cast<const uint32_t*>(&l);
    }
}

// grid (row blocks, kv heads, B * splits); the last row blocks, which see the most keys of a causal prompt, start first
template <typename T, int D>
__global__ void __launch_bounds__(kPaThreads, 2)
k_attn_prompt(const T* __restrict__ q, const int32_t* __restrict__ buf_lens, T* const* __restrict__ k_addrs, T* const* __restrict__ v_addrs,
              const uint64_t* __restrict__ bits, const int32_t* __restrict__ last, int pitch64, float scale, T* __restrict__ out,
              float* __restrict__ part_o, float* __restrict__ part_m, float* __restrict__ part_l, int len_q, int num_heads, int num_kv_heads,
              int m_query, int splits, int bshd) {
    constexpr int KS = D / 16, NJ = D / 8, CH = D / 8;   // k-steps of S, n-tiles of O, 16-byte chunks per row
    constexpr bool kHalf = std::is_same<T, __half>::value;
    extern __shared__ __align__(128) uint8_t pa_smem[];
    __shared__ int s_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int rb = (int)gridDim.x - 1 - (int)blockIdx.x, hk = blockIdx.y, b = blockIdx.z / splits, split = blockIdx.z % splits;
    const int rows = len_q * m_query, row0 = rb * kPaRows;
    pdl_trigger();
    pdl_wait();
    const int len_buf = buf_lens[b];
    const size_t stride = bshd ? (size_t)num_kv_heads * D : (size_t)D;
    const size_t base = bshd ? (size_t)hk * D : (size_t)hk * len_buf * D;
    const T* kbase = k_addrs[b] + base;
    const T* vbase = v_addrs[b] + base;

    // keys this block can see
    int n = len_buf;
    if (bits) {
        if (tid == 0) s_last = -1;
        __syncthreads();
        const int q_lo = row0 / m_query, q_hi = (min(row0 + kPaRows, rows) - 1) / m_query;
        for (int i = q_lo + tid; i <= q_hi; i += kPaThreads) atomicMax(&s_last, last[(size_t)b * len_q + i]);
        __syncthreads();
        n = s_last + 1;
    }
    const int tiles = cdiv(n, kPaKeys);
    const int t0 = (int)((long long)tiles * split / splits), t1 = (int)((long long)tiles * (split + 1) / splits);

    // this lane's two rows (g and g + 8 of the warp's 16): out of range rows compute on row 0's query and are not stored
    int qi[2], hd[2];
    bool live[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = row0 + warp * 16 + g + i * 8;
        live[i] = r < rows;
        qi[i] = live[i] ? r / m_query : 0;
        hd[i] = hk * m_query + (live[i] ? r % m_query : 0);
    }
    uint32_t qf[KS][4];
    {
        const T* q0 = q + (((size_t)b * len_q + qi[0]) * num_heads + hd[0]) * D + 2 * t;
        const T* q1 = q + (((size_t)b * len_q + qi[1]) * num_heads + hd[1]) * D + 2 * t;
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            qf[k][0] = *reinterpret_cast<const uint32_t*>(q0 + k * 16);
            qf[k][1] = *reinterpret_cast<const uint32_t*>(q1 + k * 16);
            qf[k][2] = *reinterpret_cast<const uint32_t*>(q0 + k * 16 + 8);
            qf[k][3] = *reinterpret_cast<const uint32_t*>(q1 + k * 16 + 8);
        }
    }
    const uint64_t* brow[2] = {nullptr, nullptr};
    if (bits) {
#pragma unroll
        for (int i = 0; i < 2; ++i) brow[i] = bits + ((size_t)b * len_q + qi[i]) * pitch64;
    }

    const uint32_t sm = smem_u32(pa_smem);
    constexpr uint32_t kTile = kPaKeys * D * 2;
    auto load_tile = [&](int tile, int st) {
        const int k0 = tile * kPaKeys;
#pragma unroll
        for (int i = 0; i < kPaKeys * CH / kPaThreads; ++i) {
            const int e = tid + i * kPaThreads, r = e / CH, c = e % CH;
            const bool in = k0 + r < n;
            const size_t src = (size_t)(in ? k0 + r : 0) * stride + c * 8;
            pa_cp16(sm + st * 2 * kTile + pa_off<D>(r, c), kbase + src, in);
            pa_cp16(sm + st * 2 * kTile + kTile + pa_off<D>(r, c), vbase + src, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float o[NJ][4], mx[2] = {-1e20f, -1e20f}, sum[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < NJ; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    uint64_t vis_next[2] = {~0ull, ~0ull};
    if (t0 < t1) {
        load_tile(t0, 0);
        if (bits) vis_next[0] = brow[0][t0], vis_next[1] = brow[1][t0];
    }
    for (int tile = t0; tile < t1; ++tile) {
        const int st = (tile - t0) & 1;
        uint64_t vis[2] = {vis_next[0], vis_next[1]};
        if (tile + 1 < t1) {
            load_tile(tile + 1, st ^ 1);
            if (bits) vis_next[0] = brow[0][tile + 1], vis_next[1] = brow[1][tile + 1];
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const int left = n - tile * kPaKeys;
        if (left < kPaKeys) {
            const uint64_t keep = (1ull << left) - 1;
            vis[0] &= keep, vis[1] &= keep;
        }
        // a tile none of the warp's rows sees (the diagonal of a causal prompt) costs nothing
        if (__any_sync(0xffffffffu, (live[0] && vis[0]) || (live[1] && vis[1]))) {
            const uint32_t sk = sm + st * 2 * kTile, sv = sk + kTile;
            float s[8][4];
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    uint32_t kb[4];
                    pa_ldm4(kb, sk + pa_off<D>(jj * 16 + (lane & 7) + (lane >> 4) * 8, k * 2 + ((lane >> 3) & 1)));
                    pa_mma<T>(s[2 * jj], qf[k], kb[0], kb[1]);
                    pa_mma<T>(s[2 * jj + 1], qf[k], kb[2], kb[3]);
                }
            const uint32_t v0[2] = {(uint32_t)vis[0], (uint32_t)(vis[0] >> 32)}, v1[2] = {(uint32_t)vis[1], (uint32_t)(vis[1] >> 32)};
            float m0 = mx[0], m1 = mx[1];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int sh = (j & 3) * 8 + 2 * t;
                const uint32_t w0 = v0[j >> 2] >> sh, w1 = v1[j >> 2] >> sh;
                s[j][0] = (w0 & 1) ? s[j][0] * scale : -INFINITY;
                s[j][1] = (w0 & 2) ? s[j][1] * scale : -INFINITY;
                s[j][2] = (w1 & 1) ? s[j][2] * scale : -INFINITY;
                s[j][3] = (w1 & 2) ? s[j][3] * scale : -INFINITY;
                m0 = fmaxf(m0, fmaxf(s[j][0], s[j][1]));
                m1 = fmaxf(m1, fmaxf(s[j][2], s[j][3]));
            }
#pragma unroll
            for (int x = 1; x < 4; x <<= 1) {
                m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, x));
                m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, x));
            }
            constexpr float kLog2e = 1.4426950408889634f;
            const float c0 = exp2f((mx[0] - m0) * kLog2e), c1 = exp2f((mx[1] - m1) * kLog2e);
            mx[0] = m0, mx[1] = m1;
            float l0 = 0.f, l1 = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                s[j][0] = exp2f((s[j][0] - m0) * kLog2e);
                s[j][1] = exp2f((s[j][1] - m0) * kLog2e);
                s[j][2] = exp2f((s[j][2] - m1) * kLog2e);
                s[j][3] = exp2f((s[j][3] - m1) * kLog2e);
                l0 += s[j][0] + s[j][1];
                l1 += s[j][2] + s[j][3];
            }
            sum[0] = fmaf(sum[0], c0, l0);
            sum[1] = fmaf(sum[1], c1, l1);
#pragma unroll
            for (int j = 0; j < NJ; ++j) o[j][0] *= c0, o[j][1] *= c0, o[j][2] *= c1, o[j][3] *= c1;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint32_t ah[4], al[4];
                pa_pack<T>(s[2 * kk][0], s[2 * kk][1], ah[0], al[0]);
                pa_pack<T>(s[2 * kk][2], s[2 * kk][3], ah[1], al[1]);
                pa_pack<T>(s[2 * kk + 1][0], s[2 * kk + 1][1], ah[2], al[2]);
                pa_pack<T>(s[2 * kk + 1][2], s[2 * kk + 1][3], ah[3], al[3]);
#pragma unroll
                for (int jj = 0; jj < NJ / 2; ++jj) {
                    uint32_t vb[4];
                    pa_ldm4t(vb, sv + pa_off<D>(kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, jj * 2 + (lane >> 4)));
                    pa_mma<T>(o[2 * jj], ah, vb[0], vb[1]);
                    pa_mma<T>(o[2 * jj + 1], ah, vb[2], vb[3]);
                    if constexpr (!kHalf) {
                        pa_mma<T>(o[2 * jj], al, vb[0], vb[1]);
                        pa_mma<T>(o[2 * jj + 1], al, vb[2], vb[3]);
                    }
                }
            }
        }
        __syncthreads();   // everyone is done with this stage: the next iteration refills it
    }

#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float l = sum[i];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        l += 1e-20f;
        if (!live[i]) continue;
        const float inv = (kHalf ? 1.f / 1024.f : 1.f) / l;
        const size_t vh = ((size_t)b * len_q + qi[i]) * num_heads + hd[i];
        if (splits == 1) {
            T* dst = out + vh * D + 2 * t;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                T pr[2] = {from_f32<T>(o[j][2 * i] * inv), from_f32<T>(o[j][2 * i + 1] * inv)};
                *reinterpret_cast<uint32_t*>(dst + j * 8) = *reinterpret_cast<const uint32_t*>(pr);
            }
        } else {
            float* dst = part_o + (vh * splits + split) * D + 2 * t;
#pragma unroll
            for (int j = 0; j < NJ; ++j) *reinterpret_cast<float2*>(dst + j * 8) = make_float2(o[j][2 * i] * inv, o[j][2 * i + 1] * inv);
            if (t == 0) {
                part_m[vh * splits + split] = mx[i];
                part_l[vh * splits + split] = l;
            }
        }
    }
}

// Key splits of a launch of `ctas` row blocks over up to `tiles` key tiles: a tile costs a CTA about 0.8 us, the merge of the splits
// 5 us, so keys are only split where that shortens the longest chain.
inline int prompt_attn_splits(long long ctas, int tiles) {
    const long long slots = 2ll * device_sm_count();
    int s = (int)(slots / (ctas > 0 ? ctas : 1));
    if (s > tiles / 4) s = tiles / 4;
    if (s > 16) s = 16;
    if (s < 2 || (tiles - tiles / s) * 8 < 60) return 1;
    return s;
}

}  // namespace zl
