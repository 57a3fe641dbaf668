// What the tcgen05 W4A16 kernels (w4a16_tc.cu, w4a16_tc2.cu) share: parameters, the tensor maps of the packed weights, the epilogues.
#pragma once
#include "common.cuh"
#include "tc_common.cuh"
#include "w4_layout.cuh"
#include "w4_params.h"

namespace zl {

struct alignas(64) W4TcParams {
    CUtensorMap xmap;           // x (M, K) fp16 row-major, box {64, rows of x per load}, 128-byte swizzle; w4a16_tc2.cu: as [K / 64][M][64]
    CUtensorMap wmap;           // ZLW4I nibble words as [N/32][G][32 rows][64 B], box {64 B, 32, 1, 4}, 64-byte swizzle
    CUtensorMap wmap2;          // the same as [N/32][G][16 pairs of rows][128 B], box {128 B, 16, 1, 4}, 128-byte swizzle (w4a16_tc2.cu)
    CUtensorMap tmap;           // the 80-byte scale / zero trailers as [N/32][G][80 B], box {80 B, 1, 4}
    const uint8_t* packed;      // ZLW4I
    const __half* bias;         // indexed by PACKED row
    const __half* residual;
    __half* y;
    int M, N, K, epi;
    int dbg;                    // ZL_TC_DBG timing ablations (results are wrong): 1 no x loads, 2 no dequant, 4 no MMA, 8 no weight loads
    uint2* ws;                  // [2 * CTA + slot][M][128] tagged words {fp32 partial sum, tag}: all zero between launches
    unsigned* err;              // where a wait that gives up leaves its code
    long long* trace;           // ZL_TC_DBG & 16: clock64 stamps of CTA 0, [role][64 stages][8]
    const float* cos;
    const float* sin;
    __half* q_out;
    const int32_t* token_batch;
    const int32_t* placement;
    __half* const* k_addrs;
    __half* const* v_addrs;
    int num_heads, num_kv_heads, dim_head;
    int ntok, tok_tiles;        // w4a16_tc2.cu: rows of x per tile, tiles along them
    int whole, cut;             // w4a16_tc2.cu: tiles from the `whole`-th on come in `cut` pieces of their rows of x
    int early;                  // see pdl_start
    int splits;                 // w4a16_tc2.cu: pairs of a cluster that share a tile's K (then a tile per cluster)
    int wide;                   // two neighbouring values of y may be stored together
};

// ---- epilogue of 16 tokens (c0 .. c0+15) for the weight row owned by this lane -----------------------------------------
// Packed row p = tile * 128 + 32 * quadrant + lane.  Inside a 32-row block, rows (16 tt + g) and (16 tt + g + 8) are
// partners (gate / up, RoPE low / high half): lane and lane + 8.
// the epilogue warps share their schedulers with the dequant warps, which are issue-bound: SiLU through the fast exp / divide
// (2 ulp of fp32, invisible after the fp16 rounding of the product)
__device__ __forceinline__ float tc_silu(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

// Stores of 2 bytes per lane bounded the epilogue of a 256-token tile (10000 cycles for 128 rows), so neighbouring lanes trade the
// values of every other token and store two columns each; where two lanes share an output (gate / up, RoPE partners) each takes every
// other token instead of one doing the work of both.
// residual values of 16 tokens in the layout of the stores: word j = columns (prow & ~1, + 1) of token c0 + 2 j + (lane & 1).  They are a
// round trip to L2 away: the epilogue warps fetch a chunk's words while the one before is processed (wide only).
__device__ __forceinline__ void tc_fetch_residual(const W4TcParams& p, int prow, int lane, int c0, uint32_t (&r)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int tok = c0 + 2 * j + (lane & 1);
        r[j] = tok < p.M ? *reinterpret_cast<const uint32_t*>(p.residual + (size_t)tok * p.N + (prow & ~1)) : 0u;
    }
}
__device__ __forceinline__ uint32_t tc_bits(float x) { return (uint32_t)__half_as_ushort(__float2half_rn(x)); }

// EPI: the epilogue, or -1: p.epi's.  rpre: what tc_fetch_residual got
template <int EPI = -1>
__device__ __forceinline__ void tc_epilogue16(const W4TcParams& p, int prow, int lane, int c0, float (&v)[16], const uint32_t* rpre = nullptr) {
    const int epi = EPI < 0 ? p.epi : EPI;
    const float b = p.bias ? __half2float(p.bias[prow]) : 0.f;
    const bool odd = lane & 1, up = lane & 8;
    if (epi == ZL_EPI_SWIGLU) {
        const int n_out = p.N / 2;
        const int col = (prow >> 5) * 16 + ((lane >> 4) << 3) + (lane & 7);
        uint32_t h[8];   // token 2 j of the gate's lane, 2 j + 1 of the up lane
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float m0 = __half2float(__float2half_rn(v[2 * j] + b)), m1 = __half2float(__float2half_rn(v[2 * j + 1] + b));
            const float other = __shfl_xor_sync(0xffffffffu, up ? m0 : m1, 8);
            h[j] = tc_bits(tc_silu(up ? other : m0) * (up ? m1 : other));
        }
        if (p.wide) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? h[2 * i] : h[2 * i + 1], 1);
                const int tok = c0 + 4 * i + 2 * odd + (up ? 1 : 0);
                if (tok < p.M)
                    *reinterpret_cast<uint32_t*>(p.y + (size_t)tok * n_out + (col & ~1)) = odd ? (other | (h[2 * i + 1] << 16)) : (h[2 * i] | (other << 16));
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int tok = c0 + 2 * j + (up ? 1 : 0);
                if (tok < p.M) p.y[(size_t)tok * n_out + col] = __ushort_as_half((unsigned short)h[j]);
            }
        }
    } else if (epi == ZL_EPI_QKV_ROPE) {
        const int d = p.dim_head, half_dim = d / 2, tiles_per_head = d / 32;
        const int st = prow >> 5, head = st / tiles_per_head, jt = st % tiles_per_head;
        const int c = jt * 16 + ((lane >> 4) << 3) + (lane & 7);
        const bool is_v = head >= p.num_heads + p.num_kv_heads, is_q = head < p.num_heads;
        const int mytok = c0 + (lane & 15);
        __half* mine = nullptr;   // output row of token c0 + (lane & 15)
        if (mytok < p.M) {
            if (is_q) {
                mine = p.q_out + ((size_t)mytok * p.num_heads + head) * d;
            } else {
                const int pl = p.placement[mytok];
                const int hk = is_v ? head - p.num_heads - p.num_kv_heads : head - p.num_heads;
                if (pl >= 0) mine = (is_v ? p.v_addrs : p.k_addrs)[p.token_batch[mytok]] + ((size_t)pl * p.num_kv_heads + hk) * d;
            }
        }
        uint32_t o[8];   // loads first: the stores go through pointers the compiler cannot tell from the tables'
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float m0 = __half2float(__float2half_rn(v[2 * j] + b)), m1 = __half2float(__float2half_rn(v[2 * j + 1] + b));
            const float other = __shfl_xor_sync(0xffffffffu, up ? m0 : m1, 8);
            const float lo = up ? other : m0, hi = up ? m1 : other;
            const int tok = c0 + 2 * j + (up ? 1 : 0);
            float rlo = lo, rhi = hi;
            if (!is_v && tok < p.M) {
                const float* cs = p.cos + (size_t)tok * d;
                const float* sn = p.sin + (size_t)tok * d;
                rlo = lo * cs[c] - hi * sn[c];
                rhi = hi * cs[c + half_dim] + lo * sn[c + half_dim];
            }
            o[j] = tc_bits(rlo) | (tc_bits(rhi) << 16);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            __half* dst = reinterpret_cast<__half*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(mine), 2 * j + (up ? 1 : 0)));
            if (!dst) continue;
            dst[c] = __ushort_as_half((unsigned short)(o[j] & 0xffffu));
            dst[c + half_dim] = __ushort_as_half((unsigned short)(o[j] >> 16));
        }
    } else {
        uint32_t h[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) h[i] = tc_bits(v[i] + b);
        const bool res = epi == ZL_EPI_RESIDUAL;
        if (p.wide) {
            uint32_t rw[8];
            if (res && !rpre) tc_fetch_residual(p, prow, lane, c0, rw);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? h[2 * j] : h[2 * j + 1], 1);
                const int tok = c0 + 2 * j + odd;
                uint32_t w = odd ? (other | (h[2 * j + 1] << 16)) : (h[2 * j] | (other << 16));
                if (res) {
                    const uint32_t r = rpre ? rpre[j] : rw[j];
                    const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&w)), y = __half22float2(*reinterpret_cast<const __half2*>(&r));
                    const __half2 sum = __floats2half2_rn(x.x + y.x, x.y + y.y);
                    w = *reinterpret_cast<const uint32_t*>(&sum);
                }
                if (tok < p.M) *reinterpret_cast<uint32_t*>(p.y + (size_t)tok * p.N + (prow & ~1)) = w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                if (c0 + i >= p.M) continue;
                const size_t at = (size_t)(c0 + i) * p.N + prow;
                __half x = __ushort_as_half((unsigned short)h[i]);
                if (res) x = __float2half_rn(__half2float(x) + __half2float(p.residual[at]));
                p.y[at] = x;
            }
        }
    }
}

// the weight maps of a packed matrix and the epilogue's fields
bool w4_tc_params(W4TcParams& q, const W4Params& p);

}  // namespace zl
