// Building blocks of the kernels that run one tcgen05.mma over a pair of SMs (cta_group::2): a cluster of two CTAs, of which rank 0
// (the leader) issues the MMAs for both.  Each CTA holds 128 of the 256 A rows and half of the B rows in its own shared memory, and
// the accumulators of its own 128 rows in its own TMEM.  Waits give up after about a second (a word in host memory is set, every role
// leaves its loop, TMEM is freed and the kernel returns): a fault in the protocol must not hang the GPU.  What is left of the output is
// unwritten then; zl_check_waits() makes it an error of the next synchronisation of a decoder, or of the next call of one of these kernels.
#pragma once
#include "tc_common.cuh"

#include <atomic>

namespace zl {

constexpr int kTc2Rows = 256;                 // A rows of a tile (both CTAs)

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    cluster_arrive();
    cluster_wait();
}
// address of this CTA's shared-memory word `addr` in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Arrives on a barrier of any CTA of the cluster.  What it hands over lies in TMEM or has been read from there (ordered by
// tcgen05.fence), was written by the async proxy, or was made visible to it by fence.proxy.async: no thread of the other CTA reads it
// (a release at cluster scope, which that would take, costs the handing-over warp about a microsecond)
__device__ __forceinline__ void mbar_arrive_at(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// For a whole warp, one lane polls; false: gave up (this wait or another one of the CTA's) and the caller leaves its loop.
__device__ __forceinline__ bool tc2_wait(uint64_t* bar, uint32_t parity, volatile int* s_abort, unsigned* err, unsigned code) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) {
        ok = mbar_try_wait(bar, parity);
        if (!ok) {
            const long long t0 = clock64();
            unsigned spins = 0;
            while (!(ok = mbar_try_wait(bar, parity))) {
                if ((++spins & 1023u) == 0 && (*s_abort || clock64() - t0 > 2000000000ll)) {
                    if (!*s_abort) *reinterpret_cast<volatile unsigned*>(err) = code;   // host memory: there when the kernel has ended
                    *s_abort = 1;
                    break;
                }
            }
        }
    }
    return __all_sync(0xffffffffu, ok);
}
// The same for one thread (an elected lane that runs its warp's whole loop).
__device__ __forceinline__ bool tc2_wait1(uint64_t* bar, uint32_t parity, volatile int* s_abort, unsigned* err, unsigned code) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    unsigned spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++spins & 1023u) == 0 && (*s_abort || clock64() - t0 > 2000000000ll)) {
            if (!*s_abort) *reinterpret_cast<volatile unsigned*>(err) = code;
            *s_abort = 1;
            return false;
        }
    }
    return true;
}
// whether a phase has ended, without waiting for it
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// after an abort: give copies and MMAs in flight time to land before shared memory and TMEM go away
__device__ __forceinline__ void tc2_drain(volatile int* s_abort) {
    if (!*s_abort) return;
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000ll) {}
}

// loads whose completion is counted on a barrier of the leader: `bar` is a cluster address
__device__ __forceinline__ void tma2_load_3d(void* smem_dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(smem_dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc2_alloc(uint32_t* s_tmem) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "n"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
}
__device__ __forceinline__ void tc2_dealloc(uint32_t tmem) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512));
}
// arrives on the barrier at this offset in both CTAs of the pair (lead: the leader's rank in its cluster) once the MMAs issued so far have completed
__device__ __forceinline__ void tc2_commit(uint64_t* bar, uint32_t lead = 0) {
    const uint16_t both = (uint16_t)(3u << lead);
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"(both)
                 : "memory");
}
// kind::f16, fp32 accumulators, 256 x n x 16; bf16 or fp16 operands, both K-major
__host__ __device__ constexpr uint32_t tc2_idesc(bool bf16, int n) {
    return (1u << 4) | (bf16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTc2Rows >> 4) << 24);
}
__device__ __forceinline__ void tc2_mma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}
// 8-bit operands, 256 x n x 32: kind::i8 (s8 x s8 -> s32) or kind::f8f6f4 (e4m3 x e4m3 -> f32)
__host__ __device__ constexpr uint32_t tc2_idesc8(bool fp8, int n) {
    return (fp8 ? (1u << 4) : ((2u << 4) | (1u << 7) | (1u << 10))) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTc2Rows >> 4) << 24);
}
template <bool FP8>
__device__ __forceinline__ void tc2_mma_ss8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    if constexpr (FP8)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
            : "memory");
}
__device__ __forceinline__ void tc2_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}

// ---- a tile whose K is split over the pairs of one cluster ------------------------------------------------------------------------------
// A few tiles leave most pairs idle.  So `splits` pairs (a cluster of 2 x splits CTAs) take a range of k each, and each finishes every
// splits-th chunk of 16 tokens: the others push their sums of it into its shared memory, where the ring was.
__device__ __forceinline__ void tc2_st_cluster4(uint32_t addr, float a, float b, float c, float d) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// place of the sums that pair `from` has of 16-token chunk `c` (of the owner's rows): [from][c / splits][4 tokens][128 rows] float4
__device__ __forceinline__ uint32_t tc2_split_at(int from, int c, int splits, int chunks, int row) {
    return (uint32_t)((((from * ((chunks + splits - 1) / splits) + c / splits) * 4) * 128 + row) * 16);
}
__device__ __forceinline__ void tc2_split_push(uint32_t smem, int rank, int mine, int c, int splits, int chunks, int row, const float (&v)[16]) {
    const uint32_t dst = cluster_map(smem + tc2_split_at(mine, c, splits, chunks, row), (uint32_t)(2 * (c % splits) + rank));
#pragma unroll
    for (int u = 0; u < 4; ++u) tc2_st_cluster4(dst + u * 2048, v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
}
// adds the other pairs' sums to this one's, in the order of k; INT: v are the bits of s32 sums
template <bool INT>
__device__ __forceinline__ void tc2_split_sum(const uint8_t* smem, int mine, int c, int splits, int chunks, int row, float (&v)[16]) {
    float own[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) own[i] = v[i], v[i] = 0.f;
    auto add = [](float& a, float b) { a = INT ? __int_as_float(__float_as_int(a) + __float_as_int(b)) : a + b; };
    for (int s = 0; s < splits; ++s) {
        const float4* part = reinterpret_cast<const float4*>(smem + tc2_split_at(s, c, splits, chunks, row));
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float4 w = s == mine ? make_float4(own[4 * u], own[4 * u + 1], own[4 * u + 2], own[4 * u + 3]) : part[u * 128];
            add(v[4 * u], w.x), add(v[4 * u + 1], w.y), add(v[4 * u + 2], w.z), add(v[4 * u + 3], w.w);
        }
    }
}

// launch of a grid of CTA pairs, `splits` of them in a cluster
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pairs(void (*kernel)(KArgs...), int pairs, int splits, dim3 block, size_t smem, cudaStream_t stream, bool pdl, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    zl_count_launch();
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// clusters of `size` CTAs of a kernel, one CTA per SM by shared memory, that the current device holds at a time, 0: none; the caller keeps what was asked before
struct ClustersFit {
    std::atomic<int> known[64][9] = {};   // count + 1
};
template <typename... KArgs>
inline int clusters_at_once(void (*kernel)(KArgs...), int threads, int smem, int size, ClustersFit& fit) {
    int dev = 0;
    cudaGetDevice(&dev);
    const bool cached = dev >= 0 && dev < 64 && size < 9;
    int n = cached ? fit.known[dev][size].load(std::memory_order_relaxed) - 1 : -1;
    if (n >= 0) return n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((device_sm_count() / size + 1) * size);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    if (cached) fit.known[dev][size].store(n + 1, std::memory_order_relaxed);
    return n;
}
// clusters of `splits` pairs
typedef ClustersFit PairsFit;
template <typename... KArgs>
inline int pairs_clusters(void (*kernel)(KArgs...), int threads, int smem, int splits, PairsFit& fit) {
    return clusters_at_once(kernel, threads, smem, 2 * splits, fit);
}

// (K, rows, batch) tensor, row pitch ld and batch pitch in elements; box = 128 bytes of k x box_rows rows, 128-byte swizzle
inline bool tc2_map_3d(CUtensorMap* map, const void* base, CUtensorMapDataType dt, uint64_t k, uint64_t rows, uint64_t batch, uint64_t ld,
                       uint64_t batch_ld, uint32_t box_rows) {
    const uint64_t elem = dt == CU_TENSOR_MAP_DATA_TYPE_UINT8 ? 1 : 2;
    const uint64_t dims[3] = {k, rows, batch}, strides[2] = {ld * elem, (batch > 1 ? batch_ld : ld * rows) * elem};
    const uint32_t box[3] = {(uint32_t)(128 / elem), box_rows, 1};
    return tc_make_map_nd(map, base, dt, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace zl
