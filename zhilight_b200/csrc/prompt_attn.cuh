// Attention of several query rows per task (portions of a prompt, beam and tree rows) over per-task ragged KV buffers: the
// counterpart of the decode kernels for len_q > 1.  Replaces nn::multi_query_attention_rag_buffer with len_q > 1
// (reference src/nn/attention/attention_kernel.cu:1252-1457), same softmax: mask ? scale * s : -inf, maximum from -1e20, sum
// from 1e-20, so a row that sees nothing gives zeros.
//
// The decode kernels give every query row a CTA of its own, which reads the task's whole K and V again: 512 rows behind 588 bf16 positions,
// 32 heads on 8, took 306 us so.  A CTA owns 128 (query, head) rows of one kv head -- all heads of the group share the tile -- and walks the
// keys 64 at a time:
//
//   warps 0-3  softmax : thread = row = lane of tensor memory; running maximum and sum in fp32; the probabilities go back over the scores
//   warp 4     S = Q K^T by tcgen05.mma, Q and K in shared memory (128-byte swizzle); two buffers of scores in tensor memory
//   warp 5     O += P V, P from tensor memory, V as it lies (rows of keys: the B operand along n), O in tensor memory; TMEM allocation
//   warps 6-7  K and V tiles by 16-byte cp.async into the swizzled layout (the buffers' addresses are known to the device only), K a tile ahead
//
// Probabilities are carried as a 16-bit value and the rest of it as another (two MMAs), fp16 models' times 2^10.  A row's reference maximum only
// follows the true one once that has grown by 2^5 (fp16) or 2^8, so that O is seldom rescaled (the conditional rescaling published with
// FlashAttention-4); with one fp16 value that would cost precision (the largest probability is no power of two any more: 2.8e-4 from 64 bits against
// 2.55e-4), with two it is 2.1e-4, all of it the output's rounding.
//
// Two CTAs share an SM (256 columns each): one's MMAs run under the other's softmax.  Bound by the chain S -> softmax -> P of a tile: 512 rows over 4096
// keys, 64 heads on 8, take 114 us alone, 3700 cycles for a tile of each of the SM's two CTAs, whose MMAs take 2060 (each: 450 of S, whose operands come
// at 128 bytes a cycle, and 580 of P V); at 500 rows behind 1000 positions, 32 on 8, 33 us, the tensor pipe is busy for 20 % of the time and 30 % of the
// issue slots are taken: of 52000 cycles 5000 until the first tile, 31000 of tiles, 15500 of the merge before its columns were shared out.  One buffer of scores and
// one of probabilities, so that the next scores come under the softmax, is slower (34.7 against 33.5 us): P V then waits behind them.  500 rows behind 1000
// positions, bf16, all launches of the call: 65 us on mma.sync with 64-row blocks, 33 here; 512 x 1500 with 64 heads on 8: 120 -> 48.
//
// An int8 mask is turned into bits first (k_mask_bits), once for all kv heads, together with each row's last visible key: tiles behind the last
// key any row of the block sees are never loaded, which halves a causal prompt's work.  Few blocks are cut along their keys: the CTAs of a
// cluster take a range each and push their O, maximum and sum into the shared memory of the CTAs that finish these columns.
//
// Nothing waits for ever: see tc2_common.cuh.  The waits begin behind the launch dependency.
#pragma once
#include "decode_attn_short.cuh"
#include "tc2_common.cuh"

#include <type_traits>

namespace zl {

constexpr int kPaRows = 128, kPaKeys = 64;
constexpr int kPaWarpS = 4, kPaWarpO = 5, kPaWarpLoad = 6, kPaLoaders = 64, kPaThreads = kPaWarpLoad * 32 + kPaLoaders;

// mask rows -> bits.  grid (len_q, B), 256 threads; bits [B][len_q][pitch64] with zero words behind len_buf, last [B][len_q]: index
// of the last visible key, -1 for none
__global__ void __launch_bounds__(256) k_mask_bits(const int8_t* __restrict__ mask, const int32_t* __restrict__ buf_lens, uint64_t* bits,
                                                   int32_t* last, int len_q, int pitch64, int behind) {
    __shared__ int s_last[8];
    pdl_start(!behind);
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

// ---- PTX wrappers (one CTA, cta_group::1) ---------------------------------------------------------------------------------------
__device__ __forceinline__ void pa_alloc(uint32_t* s_tmem) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "n"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void pa_dealloc(uint32_t tmem) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(256));
}
__device__ __forceinline__ void pa_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
}
__device__ __forceinline__ void pa_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
}
// fp32 accumulators, 128 x n x 16; b_mn: B's rows run along n (V), not along k
__host__ __device__ constexpr uint32_t pa_idesc(bool bf16, int n, bool b_mn) {
    return (1u << 4) | (bf16 ? (1u << 7) | (1u << 10) : 0u) | (b_mn ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kPaRows >> 4) << 24);
}
// B as [64 columns of n][k][128 bytes], 128-byte swizzle: 1024 bytes from 8 rows of k to the next, `block` bytes from 64 columns to the next
__device__ __forceinline__ uint64_t pa_desc_mn(uint32_t saddr, uint32_t block) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)(block >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ void pa_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,"
        "%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void pa_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// two fp32 lanes of a 64-bit register pair at a time: half the instructions of the scalar forms
__device__ __forceinline__ uint64_t pa_two(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void pa_split(uint64_t v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ uint64_t pa_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t pa_add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float pa_max3(float x, float y, float z) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
    return r;
}
__device__ __forceinline__ float pa_exp2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void pa_cp16(uint32_t dst, const void* src, bool in) {
    const int bytes = in ? 16 : 0;   // 0: zero fill, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pa_landed(uint64_t* bar) {   // one arrival once this thread's copies so far are there
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void pa_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void pa_st_cluster4(uint32_t addr, uint4 v) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void pa_st_cluster2(uint32_t addr, float2 v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}

template <int D>
struct PaCfg {
    static constexpr int kAtoms = D / 64;                        // 128-byte columns of a row
    static constexpr int kQ = kAtoms * kPaRows * 128;            // [64 of d][128 rows][128 B]
    static constexpr int kTile = kAtoms * kPaKeys * 128;         // K or V: [64 of d][64 keys][128 B]
    static constexpr int kKOff = kQ, kVOff = kQ + 2 * kTile;
    static constexpr int kStaged = kQ + 4 * kTile;
    static constexpr int kMl = kStaged;                          // merge: {maximum, sum}, then weight, of the rows of up to 8 key ranges
    static constexpr int kUsed = kMl + 8 * kPaRows * 8 + 1024;   // + slack for the manual 1024-byte alignment
    static constexpr int kBytes = kHalfTmemSmem;                 // more than it uses, for the sake of tensor memory
    static constexpr int kAloneBytes = 120 * 1024;               // no SM takes two of them
    static_assert(2 * kAloneBytes > kSmSmem, "an SM each");
    static_assert(kUsed <= kBytes, "shared memory");
    static_assert(kPaRows * (D + 8 * 4) * 4 <= kStaged, "merge: [key range][row][D / ranges + 4] floats, where Q, K and V were");
    static constexpr int kS = 128;                               // TMEM columns: O 0 .. D - 1, S / P 128 .. 255 (two buffers of 64)
};

// grid (row blocks, kv heads, B * splits), clusters of `splits` CTAs along z; the last row blocks, which see the most keys of a causal
// prompt, start first
template <typename T, int D>
__global__ void __launch_bounds__(kPaThreads, 2)
k_attn_prompt(const T* __restrict__ q, const int32_t* __restrict__ buf_lens, T* const* __restrict__ k_addrs, T* const* __restrict__ v_addrs,
              const uint64_t* __restrict__ bits, const int32_t* __restrict__ last, int pitch64, float scale, T* __restrict__ out, int len_q,
              int num_heads, int num_kv_heads, int m_query, int splits, int bshd, int aligned, unsigned* err, const __grid_constant__ AttnAddrs inl) {
    using C = PaCfg<D>;
    constexpr bool kHalf = std::is_same<T, __half>::value;
    constexpr int CH = D / 8;                                    // 16-byte chunks per row
    extern __shared__ uint8_t pa_smem[];
    uint8_t* smem = pa_smem + ((1024u - (smem_u32(pa_smem) & 1023u)) & 1023u);
    __shared__ uint64_t k_full[2], v_full[2];
    __shared__ uint64_t s_full[2];    // scores of a tile are there, and its K is done with
    __shared__ uint64_t p_full[2];
    __shared__ uint64_t o_done[2];    // P V of a tile has been added: its V and its scores' columns are done with
    __shared__ uint32_t s_tmem;
    __shared__ int s_gave_up;
    volatile int* s_abort = &s_gave_up;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rb = (int)gridDim.x - 1 - (int)blockIdx.x, hk = blockIdx.y, b = blockIdx.z / splits, split = blockIdx.z % splits;
    const int rows = len_q * m_query, row0 = rb * kPaRows;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], kPaLoaders);
            mbar_init(&v_full[i], kPaLoaders);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);
            mbar_init(&o_done[i], 1);
        }
        s_gave_up = 0;
        mbar_fence_init();
    }
    if (warp == kPaWarpO) pa_alloc(&s_tmem);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (splits > 1) cluster_arrive();   // waited for ahead of the merge's first store into another CTA, which must have started by then
    pdl_start(!inl.behind);   // behind the allocation: a dependent that takes all of TMEM cannot keep this block waiting for it
    pdl_wait();
    const uint32_t tmem = s_tmem;
    const int len_buf = buf_lens[b];
    const T *kp = attn_addr(inl, k_addrs, b, false), *vp = attn_addr(inl, v_addrs, b, true);

    // keys this block can see; every warp finds out by itself, the loaders go ahead of the rows of q
    int n = len_buf;
    if (bits) {
        const int q_lo = row0 / m_query, q_hi = (min(row0 + kPaRows, rows) - 1) / m_query;
        int mine = -1;
        for (int i = q_lo + lane; i <= q_hi; i += 32) mine = max(mine, last[(size_t)b * len_q + i]);
        asm volatile("" ::"l"(kp), "l"(vp));   // fetched by now, beside the line above: the loaders' next step
        n = __reduce_max_sync(0xffffffffu, mine) + 1;
    }
    if (warp < kPaWarpLoad) {
        // rows of q: [64 of d][row][128 B], chunks xor the row; rows behind the last one are zeros and are not stored
        constexpr int kStep = kPaWarpLoad * 32 / CH;
        const int c = tid % CH, dq = kStep / m_query, dh = kStep % m_query;
        int r = tid / CH, h = row0 + r;
        unsigned at = (unsigned)h / (unsigned)m_query;           // its query, then the place of its (query, head) row
        h -= at * m_query;
        at = at * num_heads + h;
        const T* q0 = q + ((size_t)b * len_q * num_heads + hk * m_query) * D + c * 8;
        const uint32_t dst0 = smem_u32(smem) + (uint32_t)((c >> 3) * (kPaRows * 128));
#pragma unroll
        for (int i = 0; i < (kPaRows + kStep - 1) / kStep; ++i, r += kStep) {
            const bool in = row0 + r < rows;
            const T* src = q0 + (size_t)(in ? at : 0u) * D;
            const uint32_t dst = dst0 + (uint32_t)(r * 128 + (((c & 7) ^ (r & 7)) << 4));
            if (r < kPaRows) {
                if (aligned) {
                    pa_cp16(dst, src, in);
                } else {
                    const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
                    *reinterpret_cast<uint4*>(smem + (dst - smem_u32(smem))) = in ? make_uint4(w[0], w[1], w[2], w[3]) : make_uint4(0, 0, 0, 0);
                }
            }
            h += dh;
            at += dq * num_heads + dh;
            if (h >= m_query) h -= m_query, at += num_heads - m_query;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        pa_fence_async();
        asm volatile("bar.sync 1, %0;" ::"n"(kPaWarpLoad * 32) : "memory");
    }
    const int tiles = cdiv(n, kPaKeys);
    const int t0 = (int)((long long)tiles * split / splits), t1 = (int)((long long)tiles * (split + 1) / splits), count = t1 - t0;

    float l = 0.f, m_ref = -1.4426950e20f;                       // of this thread's row; base-2 logarithms
    if (warp == kPaWarpS) {
        const uint32_t id = pa_idesc(!kHalf, kPaKeys, false);
        const uint64_t qd = tc_desc_sw128(smem_u32(smem));
        for (int j = 0; j < count; ++j) {
            const int st = j & 1;
            const uint32_t ph = (uint32_t)(j >> 1) & 1u;
            if (!tc2_wait(&k_full[st], ph, s_abort, err, 0x4100 + st)) break;
            pa_fence_async();
            if (j > 1 && !tc2_wait(&o_done[st], ph ^ 1u, s_abort, err, 0x4180 + st)) break;
            tc_fence_after();
            if (tc_elect_one()) {
                const uint64_t kd = tc_desc_sw128(smem_u32(smem + C::kKOff + st * C::kTile));
#pragma unroll
                for (int k = 0; k < D / 16; ++k)
                    pa_mma_ss(tmem + (uint32_t)(C::kS + st * 64), qd + (uint64_t)((k >> 2) * (kPaRows * 128 / 16) + (k & 3) * 2),
                              kd + (uint64_t)((k >> 2) * (kPaKeys * 128 / 16) + (k & 3) * 2), id, k > 0 ? 1u : 0u);
                tc_commit(&s_full[st]);
            }
            __syncwarp();
        }
    } else if (warp == kPaWarpO) {
        const uint32_t id = pa_idesc(!kHalf, D, true);
        for (int j = 0; j < count; ++j) {
            const int st = j & 1;
            const uint32_t ph = (uint32_t)(j >> 1) & 1u;
            if (!tc2_wait(&v_full[st], ph, s_abort, err, 0x4200 + st)) break;
            pa_fence_async();
            if (!tc2_wait(&p_full[st], ph, s_abort, err, 0x4300 + st)) break;
            tc_fence_after();
            if (tc_elect_one()) {
                const uint64_t vd = pa_desc_mn(smem_u32(smem + C::kVOff + st * C::kTile), kPaKeys * 128);
                const uint32_t p = tmem + (uint32_t)(C::kS + st * 64);
#pragma unroll
                for (int h = 0; h < 2; ++h)                      // the probabilities' upper halves, then the lower ones
#pragma unroll
                    for (int k = 0; k < kPaKeys / 16; ++k)
                        pa_mma_ts(tmem, p + (uint32_t)(h * 32 + k * 8), vd + (uint64_t)(k * (16 * 128 / 16)), id, (j > 0 || h > 0 || k > 0) ? 1u : 0u);
                tc_commit(&o_done[st]);
            }
            __syncwarp();
        }
    } else if (warp >= kPaWarpLoad) {
        const int t = tid - kPaWarpLoad * 32, c = t % CH;
        const size_t stride = bshd ? (size_t)num_kv_heads * D : (size_t)D;
        const size_t base = (bshd ? (size_t)hk * D : (size_t)hk * len_buf * D) + c * 8;
        const T* kbase = kp + base;
        const T* vbase = vp + base;
        const uint32_t at = smem_u32(smem) + (uint32_t)((c >> 3) * (kPaKeys * 128));
        auto load = [&](const T* from, uint32_t to, int k0) {
#pragma unroll
            for (int i = 0; i < kPaKeys * CH / kPaLoaders; ++i) {
                const int r = t / CH + i * (kPaLoaders / CH);
                const bool in = k0 + r < n;
                pa_cp16(to + (uint32_t)(r * 128 + (((c & 7) ^ (r & 7)) << 4)), from + (size_t)(in ? k0 + r : 0) * stride, in);
            }
        };
        // K runs a tile ahead of V
        for (int i = 0; i < 2 * count; ++i) {
            const int is_v = i > 0 && (i == 2 * count - 1 || !(i & 1)), j = is_v ? (i - 1) >> 1 : (i + 1) >> 1, st = j & 1;
            if (j > 1 && !tc2_wait(is_v ? &o_done[st] : &s_full[st], ((uint32_t)(j >> 1) & 1u) ^ 1u, s_abort, err, 0x4400 + 2 * is_v + st)) break;
            load(is_v ? vbase : kbase, at + (uint32_t)((is_v ? C::kVOff : C::kKOff) + st * C::kTile), (t0 + j) * kPaKeys);
            pa_landed(is_v ? &v_full[st] : &k_full[st]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // warp = quadrant of TMEM lanes, thread = row
        const int r = row0 + tid;
        const uint64_t* vis_row = bits ? bits + ((size_t)b * len_q + (r < rows ? r / m_query : 0)) * pitch64 : nullptr;
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
        constexpr float kLog2e = 1.4426950408889634f;
        constexpr float kTau = kHalf ? 5.f : 8.f;                // p * 2^10 of fp16 stays below 2^15
        constexpr float kUp = kHalf ? 10.f : 0.f;
        uint64_t vis_next = bits && count > 0 ? vis_row[t0] : ~0ull;
        for (int j = 0; j < count; ++j) {
            const int st = j & 1;
            uint64_t vis = vis_next;
            if (bits && j + 1 < count) vis_next = vis_row[t0 + j + 1];
            const int left = n - (t0 + j) * kPaKeys;
            if (left < kPaKeys) vis &= (1ull << left) - 1;
            if (!tc2_wait(&s_full[st], (uint32_t)(j >> 1) & 1u, s_abort, err, 0x4600 + st)) break;
            tc_fence_after();
            const uint32_t ts = taddr + (uint32_t)(C::kS + st * 64);
            uint32_t raw[64];
            pa_ld32(ts, raw);
            pa_ld32(ts + 32, raw + 32);
            pa_wait_ld();
            float c = scale * kLog2e;
            if (!(scale > 0.f) || !__all_sync(0xffffffffu, vis == ~0ull)) {   // some keys are hidden from some row
                const uint32_t lo = (uint32_t)vis, hi = (uint32_t)(vis >> 32);
#pragma unroll
                for (int i = 0; i < 64; ++i) raw[i] = __float_as_uint(((i < 32 ? lo : hi) >> (i & 31) & 1) ? __uint_as_float(raw[i]) * c : -INFINITY);
                c = 1.f;
            }
            float mx[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) mx[i] = __uint_as_float(raw[i]);
#pragma unroll
            for (int i = 4; i < 60; i += 8)
#pragma unroll
                for (int u = 0; u < 4; ++u) mx[u] = pa_max3(mx[u], __uint_as_float(raw[i + 2 * u]), __uint_as_float(raw[i + 2 * u + 1]));
            mx[0] = pa_max3(mx[0], __uint_as_float(raw[60]), __uint_as_float(raw[61]));
            mx[1] = pa_max3(mx[1], __uint_as_float(raw[62]), __uint_as_float(raw[63]));
            const float m_tile = pa_max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]) * c;
            // The reference maximum of a row only follows where the true one has left it by a factor of 2^kTau: any reference gives the
            // same quotient, and rescaling O costs a round trip through the registers.
            const bool up = m_tile > m_ref + kTau;
            if (__any_sync(0xffffffffu, up)) {
                const float f = up ? pa_exp2(m_ref - m_tile) : 1.f;
                if (up) m_ref = m_tile;
                l *= f;
                if (j > 0) {
                    if (!tc2_wait(&o_done[st ^ 1], (uint32_t)((j - 1) >> 1) & 1u, s_abort, err, 0x4700)) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int d0 = 0; d0 < D; d0 += 16) {
                        float v[16];
                        uint32_t w[16];
                        tc_ld16(taddr + (uint32_t)d0, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(v[i] * f);
                        tc_st16(taddr + (uint32_t)d0, w);
                    }
                }
            }
            const uint64_t c2 = pa_two(c, c), m2 = pa_two(kUp - m_ref, kUp - m_ref);
            const uint64_t minus = pa_two(-1.f, -1.f);
            uint64_t sum = 0;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float x, y;
                    pa_split(pa_fma2(pa_two(__uint_as_float(raw[half * 32 + 2 * i]), __uint_as_float(raw[half * 32 + 2 * i + 1])), c2, m2), x, y);
                    x = pa_exp2(x);
                    y = pa_exp2(y);
                    sum = pa_add2(sum, pa_two(x, y));
                    if constexpr (kHalf) {
                        const __half2 h = __floats2half2_rn(x, y);
                        hi[i] = *reinterpret_cast<const uint32_t*>(&h);
                        const float2 f = __half22float2(h);
                        pa_split(pa_fma2(pa_two(f.x, f.y), minus, pa_two(x, y)), x, y);
                        const __half2 e = __floats2half2_rn(x, y);
                        lo[i] = *reinterpret_cast<const uint32_t*>(&e);
                    } else {
                        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
                        hi[i] = *reinterpret_cast<const uint32_t*>(&h);
                        pa_split(pa_fma2(pa_two(__uint_as_float(hi[i] << 16), __uint_as_float(hi[i] & 0xffff0000u)), minus, pa_two(x, y)), x, y);
                        const __nv_bfloat162 e = __floats2bfloat162_rn(x, y);
                        lo[i] = *reinterpret_cast<const uint32_t*>(&e);
                    }
                }
                tc_st16(ts + (uint32_t)(half * 16), hi);
                tc_st16(ts + (uint32_t)(32 + half * 16), lo);
            }
            float s0, s1;
            pa_split(sum, s0, s1);
            l += s0 + s1;
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[st]);
        }
        if (count > 0) tc2_wait(&o_done[(count - 1) & 1], (uint32_t)((count - 1) >> 1) & 1u, s_abort, err, 0x4800);
        tc_fence_after();
        l += kHalf ? 1024.f * 1e-20f : 1e-20f;
        if (splits == 1) {
            T* dst = out + (((size_t)b * len_q + r / m_query) * num_heads + hk * m_query + r % m_query) * D;
            const float inv = 1.f / l;
#pragma unroll 1
            for (int d0 = 0; d0 < D; d0 += 16) {
                float v[16];
                tc_ld16(taddr + (uint32_t)d0, v);
                if (r < rows) {
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        T two[2] = {from_f32<T>(count > 0 ? v[2 * i] * inv : 0.f), from_f32<T>(count > 0 ? v[2 * i + 1] * inv : 0.f)};
                        w[i] = *reinterpret_cast<const uint32_t*>(two);
                    }
                    if (aligned) {
                        *reinterpret_cast<uint4*>(dst + d0) = make_uint4(w[0], w[1], w[2], w[3]);
                        *reinterpret_cast<uint4*>(dst + d0 + 8) = make_uint4(w[4], w[5], w[6], w[7]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) reinterpret_cast<uint32_t*>(dst + d0)[i] = w[i];
                    }
                }
            }
        }
    }
    __syncwarp();
    tc2_drain(s_abort);
    if (splits > 1) {
        cluster_wait();   // every CTA of the cluster runs: one without a key to look at is here before another one has started
        // Each CTA of the cluster finishes its columns of all rows, thread = row as before: 128 threads each add what they hold in tensor memory to what the
        // others sent.  Rows shared out instead, all columns through shared memory, took 10000 cycles behind the first barrier: 500 rows behind 1000 positions 36.8 us,
        // 35.0 so; and with each CTA beginning at another one of the cluster 76 x 1100 (four ranges) 19.6 -> 17.7.
        const int cols = D / splits, sh = 31 - __clz(cols), pitch = cols + 4;   // splits: a power of two; pitch: 16-byte chunks of eight lanes on eight bank groups
        const uint32_t ml = smem_u32(smem) + C::kMl + tid * 8;
        if (warp < kPaWarpS)
            for (int s = 0; s < splits; ++s) pa_st_cluster2(cluster_map(ml + split * (kPaRows * 8), s), make_float2(m_ref, l));
        cluster_sync_all();               // nobody's Q, K and V are needed any more: their place takes the sums
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
        float2* const mine = reinterpret_cast<float2*>(smem + C::kMl) + tid;
        const uint32_t place = smem_u32(smem) + (split * kPaRows + tid) * pitch * 4;
        if (warp < kPaWarpS) {
            tc_fence_after();
            const int first = ((split + 1) << sh) & ~31;          // each CTA begins with another one's columns
#pragma unroll 1
            for (int d = 0; d < D; d += 64) {
                uint32_t v[64];
                const int d1 = (first + d) & (D - 1), d2 = (first + d + 32) & (D - 1);
                pa_ld32(taddr + (uint32_t)d1, v);
                pa_ld32(taddr + (uint32_t)d2, v + 32);
                pa_wait_ld();
#pragma unroll
                for (int i = 0; i < 64; i += 4) {
                    const int at = (i < 32 ? d1 : d2) + (i & 31), to = at >> sh;
                    if (to != split)
                        pa_st_cluster4(cluster_map(place + (at & (cols - 1)) * 4, to),
                                       count > 0 ? make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]) : make_uint4(0u, 0u, 0u, 0u));
                }
                if (cols == 64 && D == 128) break;               // of two CTAs the other half is this one's own
            }
            // weights of the row's parts, in place of their maxima
            float m = -INFINITY, sum = 0.f;
            for (int s = 0; s < splits; ++s) m = fmaxf(m, mine[s * kPaRows].x);
            for (int s = 0; s < splits; ++s) {
                const float f = pa_exp2(mine[s * kPaRows].x - m);
                sum = fmaf(mine[s * kPaRows].y, f, sum);
                mine[s * kPaRows].x = f;
            }
            const float inv = 1.f / sum;
            for (int s = 0; s < splits; ++s) mine[s * kPaRows].x *= inv;
        }
        cluster_sync_all();
        if (warp < kPaWarpS) {
            const int r = row0 + tid;
            T* dst = out + (((size_t)b * len_q + r / m_query) * num_heads + hk * m_query + r % m_query) * D + split * cols;
            for (int c0 = 0; c0 < cols; c0 += 16) {
                float own[16], o[16] = {};
                tc_ld16(taddr + (uint32_t)(split * cols + c0), own);   // of 8 columns the first half
#pragma unroll 2
                for (int s = 0; s < splits; ++s) {
                    const float f = mine[s * kPaRows].x;
                    const float4* from = reinterpret_cast<const float4*>(smem + ((s * kPaRows + tid) * pitch + c0) * 4);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float4 v = s != split ? from[u] : count > 0 ? make_float4(own[4 * u], own[4 * u + 1], own[4 * u + 2], own[4 * u + 3]) : float4{};
                        o[4 * u] = fmaf(v.x, f, o[4 * u]), o[4 * u + 1] = fmaf(v.y, f, o[4 * u + 1]);
                        o[4 * u + 2] = fmaf(v.z, f, o[4 * u + 2]), o[4 * u + 3] = fmaf(v.w, f, o[4 * u + 3]);
                    }
                }
#pragma unroll
                for (int h = 0; h < 16; h += 8) {
                    if (r >= rows || c0 + h >= cols) continue;
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        T two[2] = {from_f32<T>(o[h + 2 * i]), from_f32<T>(o[h + 2 * i + 1])};
                        w[i] = *reinterpret_cast<const uint32_t*>(two);
                    }
                    if (aligned) {
                        *reinterpret_cast<uint4*>(dst + c0 + h) = make_uint4(w[0], w[1], w[2], w[3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) reinterpret_cast<uint32_t*>(dst + c0 + h)[i] = w[i];
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kPaWarpO) {
        tc_fence_after();
        pa_dealloc(tmem);
    }
}

// Key splits (CTAs of a cluster) of a launch of `ctas` row blocks over up to `tiles` key tiles.  A tile is about 1 us of a CTA's chain, being a
// cluster 2 us, so few tiles stay whole (256 x 256, 32 heads on 8: 12.1 against 12.5 us in two), more of them where two CTAs would share an SM (512 x 512 17.2 / 18.9,
// against it 512 x 1024 27.3 / 25.4), and further ones are cut down to two a CTA: 76 x 1100 28.7 us whole, 21.3 in two, 17.7 in four; 200 x 900, 8 on 1, 15.6 in four,
// 14.1 in eight.  Beyond one CTA per SM only pairs (256 x 1300, 16 heads on 4: 18.3 us in four, 23.3 in eight; 128 x 600, 64 on 8: 16.8 in two, 20.7 in four).
// Where some SM has to take two of clusters of eight, they have to save that: us, four / eight, 14 clusters, which find an SM per CTA, 16 tiles 16.4 / 15.0, 64 tiles 38.6 / 28.5 (22.9 as below); 16, which
// do not, 16 tiles 15.2 / 18.1, 41 tiles 29.2 / 25.4; 18 of 41 tiles 27.5 / 26.6, of 24 20.3 / 21.4.
// fit: of clusters of eight, see prompt_attn_fit
inline int prompt_attn_splits(long long ctas, int tiles, int fit) {
    const int sms = device_sm_count();
    int s = 1;
    if (tiles >= (ctas * 2 <= sms ? 8 : 12) && ctas * 2 <= 2ll * sms) s = 2;
    if (s == 2 && tiles >= 8 && ctas * 4 <= sms) s = 4;
    if (s == 4 && (ctas <= fit ? tiles >= 12 : tiles >= 40 && ctas * 8 <= sms)) s = 8;
    return s;
}

// Clusters of `splits` CTAs that find an SM for every CTA at once.  Such a launch takes the shared memory that keeps its CTAs on an SM each: some came in twos on the SMs that the
// mask's kernel had left empty.  107 rows on 2600 keys, 8 heads on 1, 23.8 -> 18.1 us; 91 on 2600, 64 on 8, 45.6 -> 36.6.
inline int prompt_attn_fit(int splits) {
    static ClustersFit fit;
    return splits == 1 ? device_sm_count() : clusters_at_once(k_attn_prompt<__half, 128>, kPaThreads, PaCfg<128>::kAloneBytes, splits, fit);
}

template <typename T, int D, typename... Args>
inline cudaError_t launch_attn_prompt(dim3 grid, int splits, bool alone, cudaStream_t stream, bool pdl, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kPaThreads);
    cfg.dynamicSmemBytes = alone ? PaCfg<D>::kAloneBytes : PaCfg<D>::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = splits;
    }
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    zl_count_launch();
    return cudaLaunchKernelEx(&cfg, k_attn_prompt<T, D>, args...);
}

}  // namespace zl
