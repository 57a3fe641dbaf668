// W4A16 GEMM for prompt-sized M: tcgen05.mma over pairs of SMs (cta_group::2), the dequantised weights as the A operand in tensor
// memory.  Same arithmetic contract as w4a16_tc.cu (w = (q - z) * s rounded to fp16 once, fp16 x fp16 products, fp32 accumulation
// over all of K) and the same packed weights, maps, conversion and epilogues.
//
// What bounded w4a16_tc.cu at 256 tokens (28672 x 4096: 115 us, 523 TFLOP/s): one accumulator leaves no MMA under an epilogue, and
// cutting the tiles into one range per CTA makes two of a CTA's two or three pieces partial ones that travel through L2 as tagged
// words.  Here
//   * a tile is 256 rows of w by up to 256 tokens over two SMs: each converts its own 128 rows and loads half of the tokens;
//   * tiles are taken whole, in turn by persistent pairs; the token tile's size is chosen so that the last wave is full, or its tiles come in halves;
//   * up to 64 tokens there are two accumulators; with one, the epilogue and the dequant warps shorten the gap together (t2_finish).
// 28672 x 4096 with SwiGLU: 1000 tokens 499 -> 182 us (cuBLAS fp16 178), 256 tokens 128 -> 55; 4096 x 14336 with the residual: 1000 tokens 408 -> 92 us
// (88; 1280 TFLOP/s).  These are 200 calls in a row on a rested GPU; after half a second of them the power limit makes it 211 and 103 (cuBLAS 204 and 100).  Bound by the tensor cores at 256 tokens (1084 cycles per 128-k group, at the clock that the power limit leaves); below 130
// tokens by the conversion (0.31 us of a group, about 600 cycles; 340 when nothing else runs on the SM).
//
// What a stage costs one thread is what bounded small tiles before that (830 cycles): looking at a barrier takes it 120 - 200 cycles even when the
// phase has ended, two TMA instructions and their votes 400.  So the issuing threads are single lanes that run their warp's loop alone and look at
// the next barrier while this stage's work is on its way, a stage is two 128-k groups up to 128 tokens, its x is one box, its weights are two and are issued by two warps in turn, the
// weight boxes have rows of 128 bytes, the ring of weights takes what room there is, and six slots of A fit beside up to 128 tokens' accumulators.
// 4096 x 14336, 256 rows 53.9 -> 45.4 us, 512 rows 55.9 -> 49.2; 28672 x 4096, 64 rows 36 -> 32; 6144 x 4096, 96 rows 22.4 -> 18.9.
// Few tiles: the pairs of a cluster share a tile's K (t2_pick).
//
//   warps 0-7    epilogue : quadrant = warp % 4, 16-token chunks in turns, above 64 tokens shared with the dequant warps
//   warps 8-23   dequant  : four groups of four warps take the 128-k groups in turn, one per slot of A; lane = weight row, quadrant =
//                           warp % 4; their arrivals of both CTAs for a stage meet on the leader's barrier
//   warps 24, 25 weights  : tensor-TMA of the 4 ZLW4I records of a stage and their trailers, this CTA's 128 rows, stages in turn
//   warp 26      x        : this CTA's half of the tokens, counted on the leader's barrier
//   warp 27      MMA      : of the leader, 8 x 256 x ntok x 16 per 128-k group; TMEM allocation
//
// The launch may start while its predecessor still runs, for as long as that takes (an all-reduce waits for its slowest rank).  A wait
// that ends only after x has come would count that time, so no warp enters one before griddepcontrol.wait: the weights of the ring's first
// stages are fetched and each group's first stage is converted ahead of it, neither of which waits for anything but the weights.
#include "tc2_common.cuh"
#include "w4a16_tc.cuh"

namespace zl {

// What tensor memory leaves beside the accumulators: a slot takes 64 columns, an accumulator one per token.
__host__ __device__ constexpr int t2_slots(int ntok) { return ntok > 128 ? 4 : 6; }
__host__ __device__ constexpr int t2_accs(int ntok) { return ntok > 64 ? 1 : 2; }
__host__ __device__ constexpr int t2_x_bytes(int ntok) { return ntok * 128; }   // of a slot and CTA: [64-k atom][ntok / 2 tokens][128 B]

struct T2Cfg {
    static constexpr int kEpiWarps = 8, kDqWarps = 16, kGroupWarps = 4;
    static constexpr int kWarpDq0 = kEpiWarps, kWarpRaw = kWarpDq0 + kDqWarps, kRawWarps = 2, kWarpX = kWarpRaw + kRawWarps, kWarpMma = kWarpX + 1;
    static constexpr int kThreads = (kWarpMma + 1) * 32;
    static constexpr int kGroups = kDqWarps / kGroupWarps;
    static constexpr int kMaxSlots = 6;                                // of A (TMEM, 64 columns each) and x (shared memory)
    static constexpr int kMaxRaw = 16;                                 // stages of packed weights
    static constexpr int kNib = 4 * 2048, kTr = 384;                   // four records' nibbles; their 80-byte trailers, padded
    static constexpr int kRing = 230400;                               // slots of x, then as many of the weights as fit
    static constexpr int kBarOff = kRing;
    static constexpr int kMiscOff = kBarOff + (2 * kMaxRaw + 2 * kMaxSlots + 4) * 8;
    static constexpr int kBytes = kMiscOff + 16 + 1024;                // + slack for the manual 1024-byte alignment
    static_assert(t2_slots(256) * 64 + 256 <= 512 && t2_slots(128) * 64 + 128 <= 512, "TMEM columns");
    static_assert(kBytes <= 232448 && tmem_alone(kBytes), "shared memory");
};
// A weight slot is held while its group converts and is then a round trip to L2 from being full again: more than two per group
__host__ __device__ constexpr int t2_raw_slots(int ntok) {
    const int fit = (T2Cfg::kRing - t2_slots(ntok) * t2_x_bytes(ntok)) / (T2Cfg::kNib + T2Cfg::kTr);
    return fit < T2Cfg::kMaxRaw ? fit : T2Cfg::kMaxRaw;
}
// A wait by parity takes the landing (or the release) before the last one for the one it is meant for, so whoever waits or looks has to know that the
// last but one has been.  The four groups and the two issuing warps run free of each other; what orders them is that group s gets its slot of A once
// group s - slots has been multiplied, and with it all before.
//   A's slot, looked at ahead of group s:   s - 4 had its slot, so s - 4 - slots is multiplied, which has to cover s - 2 slots
//   weights of s + 4, looked at behind the wait for A's slot of s: s - slots is multiplied, which has to cover s + 4 - raw (ahead of that wait only s - 4 -
//                                           slots is: 256 tokens, four slots and 11 weight slots, are one short of it)
//   release of weights s + 2, looked at while s is loaded: s - raw is released, so s - raw - slots is multiplied, which has to cover s + 2 - 2 raw
__host__ __device__ constexpr bool t2_rings_hold(int ntok) {
    return t2_slots(ntok) >= T2Cfg::kGroups && t2_raw_slots(ntok) >= t2_slots(ntok) + T2Cfg::kGroups &&
           t2_raw_slots(ntok) >= t2_slots(ntok) + T2Cfg::kRawWarps;
}
static_assert(t2_rings_hold(32) && t2_rings_hold(64) && t2_rings_hold(96) && t2_rings_hold(128) && t2_rings_hold(160) && t2_rings_hold(192) &&
                  t2_rings_hold(224) && t2_rings_hold(256),
              "a wait by parity could take an earlier phase for its own");

struct T2Tile {
    int n0, t0, ntok;   // first row of w of the pair, first token, tokens (a multiple of 32)
};
__device__ __forceinline__ bool t2_tile(const W4TcParams& p, int i, T2Tile& t) {
    int piece = 0, n = p.ntok;
    if (i >= p.whole) {   // of the last wave
        const int j = i - p.whole;
        i = p.whole + j / p.cut;
        piece = j % p.cut;
        n /= p.cut;
    }
    const int rt = i / p.tok_tiles;
    t.n0 = rt * kTc2Rows;
    t.t0 = (i - rt * p.tok_tiles) * p.ntok + piece * n;
    t.ntok = min(n, (p.M - t.t0 + 31) & ~31);
    return t.n0 < p.N;
}

__device__ __forceinline__ void t2_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// The residual epilogue of tc_epilogue16, eight tokens at a time: what sixteen hold beside the conversion's state does not fit its registers
__device__ __forceinline__ void t2_residual16(const W4TcParams& p, uint32_t taddr, int prow, int lane, int c0) {
    const float b = p.bias ? __half2float(p.bias[prow]) : 0.f;
    const bool odd = lane & 1;
#pragma unroll
    for (int half = 0; half < 2; ++half, c0 += 8, taddr += 8) {
        uint32_t h[8], r[4];
        if (p.wide) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int tok = c0 + 2 * j + odd;
                r[j] = tok < p.M ? *reinterpret_cast<const uint32_t*>(p.residual + (size_t)tok * p.N + (prow & ~1)) : 0u;
            }
        }
        float v[8];
        t2_ld8(taddr, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = tc_bits(v[i] + b);
        if (p.wide) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? h[2 * j] : h[2 * j + 1], 1);
                const int tok = c0 + 2 * j + odd;
                const uint32_t w = odd ? (other | (h[2 * j + 1] << 16)) : (h[2 * j] | (other << 16));
                const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&w)), y = __half22float2(*reinterpret_cast<const __half2*>(&r[j]));
                if (tok < p.M) *reinterpret_cast<__half2*>(p.y + (size_t)tok * p.N + (prow & ~1)) = __floats2half2_rn(x.x + y.x, x.y + y.y);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (c0 + i >= p.M) continue;
                const size_t at = (size_t)(c0 + i) * p.N + prow;
                p.y[at] = __float2half_rn(__half2float(__ushort_as_half((unsigned short)h[i])) + __half2float(p.residual[at]));
            }
        }
    }
}

// The qkv epilogue, eight tokens at a time as well, its loads in the order that hides them: what places a token's row came with the chunk before, the
// rows' addresses, cosines and sines come together ahead of the sums.  at: placement and batch of token c0 + (lane & 15).
__device__ __forceinline__ int2 t2_rope_place(const W4TcParams& p, int tok) {
    return tok < p.M ? make_int2(p.placement[tok], p.token_batch[tok]) : make_int2(-1, 0);
}
__device__ __forceinline__ void t2_rope16(const W4TcParams& p, uint32_t taddr, int prow, int lane, int c0, int2 at) {
    const float b = p.bias ? __half2float(p.bias[prow]) : 0.f;
    const bool up = lane & 8;
    const int d = p.dim_head, half_dim = d / 2, tiles_per_head = d / 32;
    const int st = prow >> 5, head = st / tiles_per_head, jt = st % tiles_per_head;
    const int c = jt * 16 + ((lane >> 4) << 3) + (lane & 7);
    const bool is_v = head >= p.num_heads + p.num_kv_heads, is_q = head < p.num_heads;
    __half* mine = nullptr;   // output row of token c0 + (lane & 15)
    if (is_q) {
        if (c0 + (lane & 15) < p.M) mine = p.q_out + ((size_t)(c0 + (lane & 15)) * p.num_heads + head) * d;
    } else if (at.x >= 0) {
        mine = (is_v ? p.v_addrs : p.k_addrs)[at.y] + ((size_t)at.x * p.num_kv_heads + (is_v ? head - p.num_heads - p.num_kv_heads : head - p.num_heads)) * d;
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        float cl[4], ch[4], sl[4], sh[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int tok = c0 + half * 8 + 2 * j + (up ? 1 : 0);
            const bool turn = !is_v && tok < p.M;
            const float *cs = p.cos + (size_t)tok * d + c, *sn = p.sin + (size_t)tok * d + c;
            cl[j] = turn ? cs[0] : 1.f, sl[j] = turn ? sn[0] : 0.f;
            ch[j] = turn ? cs[half_dim] : 1.f, sh[j] = turn ? sn[half_dim] : 0.f;
        }
        float v[8];
        t2_ld8(taddr + half * 8, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float m0 = __half2float(__float2half_rn(v[2 * j] + b)), m1 = __half2float(__float2half_rn(v[2 * j + 1] + b));
            const float other = __shfl_xor_sync(0xffffffffu, up ? m0 : m1, 8);
            const float lo = up ? other : m0, hi = up ? m1 : other;
            v[2 * j] = is_v ? lo : lo * cl[j] - hi * sl[j];
            v[2 * j + 1] = is_v ? hi : hi * ch[j] + lo * sh[j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            __half* dst = reinterpret_cast<__half*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(mine), half * 8 + 2 * j + (up ? 1 : 0)));
            if (!dst) continue;
            dst[c] = __float2half_rn(v[2 * j]);
            dst[c + half_dim] = __float2half_rn(v[2 * j + 1]);
        }
    }
}

// This warp's part of a finished tile's epilogue, 32 rows of w (TMEM lanes) by the chunks of 16 tokens that are its set's, and its arrival.  Sets 0, 1
// are the epilogue warps, 2 .. 5 the dequant groups.  shared: these help, with a chunk of eight each, the epilogue warps take two (they start
// earlier: a group converts its first stage of the next tile before).
template <int EPI>
__device__ __forceinline__ bool t2_finish(const W4TcParams& p, uint8_t* smem, uint32_t tmem, int tile, int acc, uint32_t phase, bool shared) {
    uint64_t* const acc_full = reinterpret_cast<uint64_t*>(smem + T2Cfg::kBarOff) + 2 * T2Cfg::kMaxRaw + 2 * T2Cfg::kMaxSlots + acc;
    volatile int* const s_abort = reinterpret_cast<volatile int*>(smem + T2Cfg::kMiscOff) + 1;
    const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 3, set = threadIdx.x >> 7;
    const uint32_t rank = cluster_rank();
    T2Tile t;
    t2_tile(p, tile, t);
    const int prow = t.n0 + (int)(rank & 1) * 128 + q * 32 + lane;
    const bool rows = prow < p.N;               // N % 128 == 0: all of the CTA's rows or none
    const int chunks = min(t.ntok, p.M - t.t0 + 15) >> 4;
    int c = set < 2 ? set : set + 2;
    int2 place = EPI == ZL_EPI_QKV_ROPE ? t2_rope_place(p, t.t0 + c * 16 + (lane & 15)) : make_int2(0, 0);
    if (!tc2_wait(acc_full, phase, s_abort, p.err, 0x3800 + acc)) return false;
    tc_fence_after();
    if (rows) {
        while (c < chunks) {
            const int at = c * 16;
            c += !shared || (set < 2 && !(c & 2)) ? 2 : set < 2 ? 6 : 8;
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 64 + at);
            if (EPI == ZL_EPI_RESIDUAL) {
                t2_residual16(p, taddr, prow, lane, t.t0 + at);
            } else if (EPI == ZL_EPI_QKV_ROPE) {
                const int2 now = place;
                place = t2_rope_place(p, t.t0 + c * 16 + (lane & 15));
                t2_rope16(p, taddr, prow, lane, t.t0 + at, now);
            } else {
                float v[16];
                tc_ld16(taddr, v);
                tc_epilogue16<EPI>(p, prow, lane, t.t0 + at, v);
            }
        }
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive_at(cluster_map(smem_u32(acc_full + 2), rank & ~1u));   // the leader's acc_empty
    return true;
}

template <int SUB, int EPI>
__global__ void __launch_bounds__(T2Cfg::kThreads, 1) k_w4a16_tc2(const __grid_constant__ W4TcParams p) {
    using C = T2Cfg;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + C::kBarOff);
    uint64_t* raw_empty = raw_full + C::kMaxRaw;
    uint64_t* a_full = raw_empty + C::kMaxRaw;      // leader's: a dequant group of each CTA, and the x bytes of both
    uint64_t* ax_empty = a_full + C::kMaxSlots;
    uint64_t* acc_full = ax_empty + C::kMaxSlots;
    uint64_t* acc_empty = acc_full + 2;        // leader's: the epilogue warps of both CTAs
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + C::kMiscOff);
    volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = p.splits;
    const uint32_t in_cluster = cluster_rank(), rank = in_cluster & 1, lead = in_cluster & ~1u;   // lead: the pair's leader
    const int part = (int)(in_cluster >> 1), pair = (int)(blockIdx.x >> 1) / splits, pairs = (int)(gridDim.x >> 1) / splits;
    // this pair's 128-k groups of a tile; a group behind K arrives as zeros, as its x does
    const int stages_all = (p.K / kW4GroupK + SUB - 1) / SUB, g_first = stages_all * part / splits * SUB;
    const int G = stages_all * (part + 1) / splits * SUB - g_first;
    const int slots = t2_slots(p.ntok), nacc = t2_accs(p.ntok), xstage = t2_x_bytes(p.ntok), acol0 = 512 - slots * 64;
    const int rslots = t2_raw_slots(p.ntok);
    const bool shared = nacc == 1 && splits == 1;   // a tile's epilogue is everybody's: nothing is multiplied until it has ended
    uint8_t* const nibs = smem + slots * xstage;
    uint8_t* const trs = nibs + rslots * C::kNib;

    if (threadIdx.x == 0) {
        for (int i = 0; i < rslots; ++i) {
            mbar_init(&raw_full[i], 1);
            mbar_init(&raw_empty[i], C::kGroupWarps);
        }
        for (int i = 0; i < slots / SUB; ++i) {
            mbar_init(&a_full[i], 2 * SUB * C::kGroupWarps + 1);
            mbar_init(&ax_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 2 * (C::kEpiWarps + (shared ? C::kDqWarps : 0)));
        }
        *s_abort = 0;
        mbar_fence_init();
    }
    if (warp == C::kWarpMma) tc2_alloc(s_tmem);
    pdl_start(p.early);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers and allocations are in place
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const int q = warp & 3, set = warp >> 2;   // epilogue and dequant warps; with K split a tile's only chunks come behind the exchange below
    T2Tile t;

    if (warp >= C::kWarpRaw && warp < C::kWarpX) {
        // constants: may run ahead of the predecessor kernel (PDL).  The row tiles of one wave are read by several pairs and again
        // by the next token tiles: no evict-first hint here
        if (tc_elect_one()) {
            // the two warps take the stages in turn: issuing the copies of one takes a thread 400 cycles
            int g = warp - C::kWarpRaw, rs = g, st = g;
            uint32_t ph = 0;
            bool ok = true, free = false, early = true;
            for (int i = pair; ok && t2_tile(p, i, t); i += pairs, g -= G) {
                const int rec = (t.n0 + (int)rank * 128) / 32;
                for (; g < G; g += C::kRawWarps, st += C::kRawWarps) {
                    if (early && st >= rslots) {
                        pdl_wait();
                        early = false;
                    }
                    if (!free && !(ok = tc2_wait1(&raw_empty[rs], ph ^ 1u, s_abort, p.err, 0x3100 + rs))) break;
                    uint64_t* const full = &raw_full[rs];
                    const uint32_t nib = smem_u32(nibs + rs * C::kNib), tr = smem_u32(trs + rs * C::kTr), bar = smem_u32(full);
                    rs += C::kRawWarps;
                    if (rs >= rslots) {
                        rs -= rslots;
                        ph ^= 1u;
                    }
                    free = mbar_test(&raw_empty[rs], ph ^ 1u);
                    mbar_expect_tx(full, C::kNib + 4 * 80);
                    asm volatile(
                        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(nib),
                        "l"(reinterpret_cast<uint64_t>(&p.wmap2)), "r"(0), "r"(0), "r"(g_first + g), "r"(rec), "r"(bar)
                        : "memory");
                    asm volatile(
                        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(tr),
                        "l"(reinterpret_cast<uint64_t>(&p.tmap)), "r"(0), "r"(g_first + g), "r"(rec), "r"(bar)
                        : "memory");
                }
            }
        }
        __syncwarp();
    } else if (warp == C::kWarpX) {
        pdl_wait();   // activations: produced by the predecessor kernel
        if (tc_elect_one()) {
            int as = 0;
            uint32_t ph = 0;
            bool ok = true, free = false;
            const int box = p.ntok >> 1;   // rows of a load; a shorter last tile loads rows it does not use
            for (int i = pair; ok && t2_tile(p, i, t); i += pairs) {
                const int tb = t.t0 + (int)rank * (t.ntok >> 1);
                for (int g = 0; g < G; g += SUB) {
                    if (!free && !(ok = tc2_wait1(&ax_empty[as], ph ^ 1u, s_abort, p.err, 0x3200 + as))) break;
                    uint64_t* const full = &a_full[as];
                    uint8_t* dst = smem + as * (SUB * xstage);
                    if (++as == slots / SUB) {
                        as = 0;
                        ph ^= 1u;
                    }
                    free = mbar_test(&ax_empty[as], ph ^ 1u);
                    if (rank == 0) mbar_expect_tx(full, (uint32_t)(4 * SUB * box * 128));
                    const uint32_t bar = cluster_map(smem_u32(full), lead);
                    tma2_load_3d(dst, &p.xmap, 0, tb, (g_first + g) * 2, bar);   // 2 SUB 64-k atoms
                }
            }
        }
        __syncwarp();
    } else if (warp == C::kWarpMma) {
        pdl_wait();
        if (rank == 0 && tc_elect_one()) {
            int as = 0, acc = 0;
            uint32_t ph = 0, acc_ph = 0;
            bool ok = true, ready = false;
            const uint64_t atom = (uint64_t)(((p.ntok >> 1) * 128) >> 4);   // descriptor step from k 0..63 to k 64..127 of a stage
            for (int i = pair; ok && t2_tile(p, i, t); i += pairs) {
                if (!(ok = tc2_wait1(&acc_empty[acc], acc_ph ^ 1u, s_abort, p.err, 0x3300 + acc))) break;
                const uint32_t d = tmem + (uint32_t)(acc * 64), idesc = tc2_idesc(false, t.ntok);
                for (int g = 0; g < G; g += SUB) {
                    if (!ready && !(ok = tc2_wait1(&a_full[as], ph, s_abort, p.err, 0x3400 + as))) break;
                    const uint32_t a = tmem + (uint32_t)(acol0 + as * (64 * SUB));
                    const uint64_t xd = tc_desc_sw128(smem_u32(smem + as * (SUB * xstage)));
                    uint64_t* const used = &ax_empty[as];
                    if (++as == slots / SUB) {
                        as = 0;
                        ph ^= 1u;
                    }
                    ready = mbar_test(&a_full[as], ph);   // looking at a barrier takes 200 cycles: they pass under this stage's MMAs
                    tc_fence_after();
#pragma unroll
                    for (int j = 0; j < 8 * SUB; ++j)
                        tc2_mma_ts(d, a + (uint32_t)(j * 8), xd + (j >> 2) * atom + (uint64_t)((j & 3) * 2), idesc, (g > 0 || j > 0) ? 1u : 0u);
                    tc2_commit(used, lead);
                    if (g == G - SUB) tc2_commit(&acc_full[acc], lead);
                }
                if (++acc == nacc) {
                    acc = 0;
                    acc_ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp >= C::kWarpDq0) {
        const int group = (warp - C::kWarpDq0) >> 2;
        const int tt = lane >> 4, hi = (lane >> 3) & 1, g8 = lane & 7;
        const uint32_t mask = hi ? 0xf0f0f0f0u : 0x0f0f0f0fu;
        const uint32_t magic = hi ? 0x54545454u : 0x64646464u;   // 64 + n / 16 for a high nibble n, 1024 + n for a low one
        const uint32_t sw = (uint32_t)(g8 >> 1);                 // the map's 128-byte swizzle: chunk ^= pair of rows & 7
        const uint32_t tlane = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)acol0;
        int stages = 0;
        for (int i = pair; t2_tile(p, i, t); i += pairs) stages += G;
        int as = group, rs = group;
        uint32_t ph = 0, rph = 0;
        bool raw_ready = false, ok = true;
        // Once a tile is multiplied a group has nothing to convert but what finds a slot beside it (slots stages of the next one): then it takes its
        // part of the epilogue.  28672 x 4096 with SwiGLU, 256 tokens 59.3 -> 55.0 us, 1000 tokens 199 -> 184; 6144 x 4096, 1000
        // tokens 49.2 -> 45.1; 4096 x 4096 with the residual 36.2 -> 32.8.
        int finished = 0;
        auto finish = [&]() {
            const int n = finished++;
            return t2_finish<EPI>(p, smem, tmem, pair + n * pairs, 0, (uint32_t)n & 1u, true);
        };
        for (int st = group; st < stages; st += C::kGroups) {
            if (st >= slots && st < slots + C::kGroups) pdl_wait();
            while (shared && ok && st >= (finished + 1) * G + slots) ok = finish();
            if (!ok) break;
            if (!raw_ready && !tc2_wait(&raw_full[rs], rph, s_abort, p.err, 0x3600 + rs)) break;
            // looking at a barrier takes 200 cycles: they pass under the conversion
            const bool free = mbar_test(&ax_empty[as / SUB], ph ^ 1u);
            const uint8_t* nib = nibs + rs * C::kNib + q * 2048 + (g8 >> 1) * 128;
            const uint8_t* tr = trs + rs * C::kTr + q * 80;
            uint64_t* const used = &raw_empty[rs];
            rs += C::kGroups;
            if (rs >= rslots) {
                rs -= rslots;
                rph ^= 1u;
            }
            bool next = false;
            const __half2 sc2 = *reinterpret_cast<const __half2*>(tr + (tt * 8 + g8) * 4);
            const int zz = tr[64 + tt * 8 + g8];
            const __half2 cz = __float2half2_rn(hi ? (float)(64 + (zz >> 4)) : (float)(1024 + (zz & 0xF)));
            const __half2 s2 = hi ? __half2half2(__high2half(sc2)) : __half2half2(__low2half(sc2));
            const uint32_t taddr = tlane + (uint32_t)(as * 64);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {    // 64 k at a time: 32 columns
                uint4 wv[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    // 16-k chunk kc of the group: k = 32 t + 16 hh + ..., record row (2 tt + hh) * 8 + g, chunk t
                    const int kc = ks * 4 + c, tq = kc >> 1, hh = kc & 1;
                    wv[c] = *reinterpret_cast<const uint4*>(nib + (tt * 2 + hh) * 512 + (((((uint32_t)g8 ^ hh) & 1) << 6) | ((tq ^ sw) << 4)));
                }
                if (ks == 1) {
                    __syncwarp();               // every lane's shared-memory reads of the stage have returned
                    if (lane == 0) mbar_arrive(used);
                }
                uint32_t r[2][16];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint32_t words[4] = {wv[c].x, wv[c].y, wv[c].z, wv[c].w};
#pragma unroll
                    for (int wq = 0; wq < 4; ++wq) {
                        const uint32_t wm = words[wq] & mask;
                        uint32_t a0 = __byte_perm(wm, magic, 0x4140), a1 = __byte_perm(wm, magic, 0x4342);
                        __half2 v0 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&a0), cz), s2);
                        __half2 v1 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&a1), cz), s2);
                        r[c >> 1][(c & 1) * 8 + wq * 2] = *reinterpret_cast<uint32_t*>(&v0);
                        r[c >> 1][(c & 1) * 8 + wq * 2 + 1] = *reinterpret_cast<uint32_t*>(&v1);
                    }
                }
                if (ks == 0) {
                    if (!__all_sync(0xffffffffu, free) && !(ok = tc2_wait(&ax_empty[as / SUB], ph ^ 1u, s_abort, p.err, 0x3700 + as))) break;
                    tc_fence_after();
                    next = mbar_test(&raw_full[rs], rph);   // not before this wait: see t2_rings_hold
                }
                tc_st16(taddr + (uint32_t)(ks * 32), r[0]);
                tc_st16(taddr + (uint32_t)(ks * 32 + 16), r[1]);
            }
            if (!ok) break;
            tc_wait_st();
            tc_fence_before();
            raw_ready = __all_sync(0xffffffffu, next);   // one arrival per warp
            if (lane == 0) mbar_arrive_at(cluster_map(smem_u32(&a_full[as / SUB]), lead));
            as += C::kGroups;
            if (as >= slots) {
                as -= slots;
                ph ^= 1u;
            }
        }
        if (shared) {
            pdl_wait();
            while (ok && finished * G < stages) ok = finish();
        }
    } else {
        int acc = 0;
        uint32_t acc_ph = 0;
        pdl_wait();
        if (splits > 1 && t2_tile(p, pair, t)) tc2_wait(&acc_full[0], 0, s_abort, p.err, 0x3800);   // the rest comes behind the exchange
        for (int i = pair; splits == 1 && t2_tile(p, i, t); i += pairs) {
            if (!t2_finish<EPI>(p, smem, tmem, i, acc, acc_ph, shared)) break;
            if (++acc == nacc) {
                acc = 0;
                acc_ph ^= 1u;
            }
        }
    }
    __syncwarp();
    tc2_drain(s_abort);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // nobody's shared memory or TMEM goes, or takes sums, while another CTA may still use it
    if (splits > 1) {
        tc_fence_after();
        const bool any = t2_tile(p, pair, t);
        const int row = q * 32 + lane, prow = t.n0 + (int)rank * 128 + row;
        const bool epilogue = warp < C::kWarpRaw && any && prow < p.N;   // the dequant warps too
        constexpr int kSets = C::kWarpRaw / 4;
        const int chunks = min(t.ntok, p.M - t.t0 + 15) / 16;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
        if (epilogue)
            for (int c = set; c < chunks; c += kSets) {
                if (c % splits == part) continue;
                float v[16];
                tc_ld16(taddr + (uint32_t)(c * 16), v);
                tc2_split_push(smem_u32(smem), (int)rank, part, c, splits, chunks, row, v);
            }
        cluster_sync_all();
        if (epilogue)
            for (int c = part + set * splits; c < chunks; c += kSets * splits) {
                float v[16];
                tc_ld16(taddr + (uint32_t)(c * 16), v);
                tc2_split_sum<false>(smem, part, c, splits, chunks, row, v);
                tc_epilogue16<EPI>(p, prow, lane, t.t0 + c * 16, v);
            }
        tc_fence_before();
        __syncthreads();
    }
    if (warp == C::kWarpMma) {
        tc_fence_after();
        tc2_dealloc(tmem);
    }
}

// ---- host side --------------------------------------------------------------------------------------------------------
// One instance per epilogue: all of them in one kernel, and the epilogue twice in it, cost instruction fetches that the conversion waits for
typedef void (*T2Kernel)(W4TcParams);
static T2Kernel t2_kernel(int sub, int epi) {
    switch (epi) {
        case ZL_EPI_SWIGLU: return sub == 2 ? k_w4a16_tc2<2, ZL_EPI_SWIGLU> : k_w4a16_tc2<1, ZL_EPI_SWIGLU>;
        case ZL_EPI_RESIDUAL: return sub == 2 ? k_w4a16_tc2<2, ZL_EPI_RESIDUAL> : k_w4a16_tc2<1, ZL_EPI_RESIDUAL>;
        case ZL_EPI_QKV_ROPE: return sub == 2 ? k_w4a16_tc2<2, ZL_EPI_QKV_ROPE> : k_w4a16_tc2<1, ZL_EPI_QKV_ROPE>;
        default: return sub == 2 ? k_w4a16_tc2<2, ZL_EPI_NONE> : k_w4a16_tc2<1, ZL_EPI_NONE>;
    }
}
cudaError_t prepare_w4_tc2() {
    cudaError_t e = cudaSuccess;
    for (int epi = ZL_EPI_NONE; epi <= ZL_EPI_QKV_ROPE && e == cudaSuccess; ++epi)
        for (int sub = 1; sub <= 2 && e == cudaSuccess; ++sub)
            e = cudaFuncSetAttribute(t2_kernel(sub, epi), cudaFuncAttributeMaxDynamicSharedMemorySize, T2Cfg::kBytes);
    return e;
}

// 128-k groups of a stage.  Handing a stage over costs the MMA warp 460 cycles whatever is in it, which is what bounded up to 128 tokens; of
// two groups per stage 300 a group are left beside the conversion (28672 x 4096, 32 tokens: 33 -> 30.4 us; 4096 x 14336 45 -> 43).  Above,
// the MMAs are the longer and four slots of A are too few to pair.
static int t2_sub(int ntok) { return ntok <= 128 ? 2 : 1; }

// Tokens per tile, and how many pairs share a tile's K: with few tiles the pairs of a cluster (the device holds t2_clusters(s) clusters of s pairs
// at a time: 33, 22, 15 of 2, 3, 4) take a part each and exchange their sums.  Microseconds, fitted to the times below: a 128-k group costs its
// conversion (0.31) or its MMAs (0.0022 per token; above 128 tokens the two get into each other's way), a tile's start and end 8.8 + 0.03 per
// token, a further wave less than that, since two accumulators (up to 64 tokens) or only the next tile's first groups hide the epilogue.
// Measured, one pair / two / three, N x K, us: 4096 x 14336, 32 tokens 43 / 27 / 22.7, 96 tokens 45 / 31 / 24.7, 256 tokens 46.5 / 33 / -;
// 4096 x 4096, 96 tokens 18.8 / 16.5 / 16.5, 128 tokens 19.7 / 16.5 / 18.2; 6144 x 4096, 64 tokens 19.0 / 16.5 / -; 8192 x 3584, 128 tokens
// 19.7 / 18.6 / -.  These are the times from before every warp helped with the epilogue; up to 256 rows they stand, since the line to the stream-k kernel
// rests on them (see w4_tc2_route for what that costs).  Beyond, fitted again to 56 sizes and their tiles (M = 320 .. 1000 of eight matrices; within 5 % where power is no limit): a group 0.35, or 0.08 +
// 0.0021 per token above 128, start and end 9 + 0.01 per token, a further wave's end 1.5 + 0.01 per token (hidden up to 64).  There a last wave of few tiles
// may also be cut in halves along its tokens: 28672 x 4096 is 448 tiles of 256 tokens at M = 1000, six waves and four tiles: 192 -> 184 us; M = 512 110 -> 103 (224
// tiles, three waves and two); 16384 x 2048, M = 1000 67.8 -> 61.7.  Quarters: 184, 102 and 73, the conversion (0.4 a group) is the same for 64 tokens.
struct T2Pick {
    int ntok, splits, cut;   // cut: 2: tiles of the last wave come in halves
    double us;
};
static int t2_clusters(int splits) {
    static PairsFit fit;
    return pairs_clusters(k_w4a16_tc2<1, ZL_EPI_NONE>, T2Cfg::kThreads, T2Cfg::kBytes, splits, fit);
}
static T2Pick t2_pick(int M, int row_tiles, int G) {
    const int pairs = device_sm_count() / 2;
    T2Pick best{32, 1, 1, 1e30};
    for (int n = 32; n <= 256; n += 32) {
        const long long tiles = (long long)row_tiles * cdiv(M, n), waves = (tiles + pairs - 1) / pairs;
        for (int s = 1; s <= 4; ++s) {
            const int sub = t2_sub(n), mine = cdiv(cdiv(G, sub), s) * sub;
            if (s > 1 && (cdiv(G, sub) < 2 * s || tiles * s > pairs || tiles > t2_clusters(s))) break;
            const double exchange = s > 1 ? 1.2 + 0.01 * n : 0.0;
            if (M <= 256) {
                const double group = n <= 128 ? fmax(0.31, 0.0022 * n) : fmax(0.00223 * n, 0.21 + 0.00137 * n);
                const double further = (double)(waves - 1) * (n <= 64 ? 0.3 : n <= 128 ? 3.0 + 0.03 * n : 0.0074 * n);
                const double us = 8.8 + 0.03 * n + (double)waves * mine * group + further + exchange;
                if (us < best.us - 1e-9) best = T2Pick{n, s, 1, us};
                continue;
            }
            const long long whole = tiles / pairs, left = tiles % pairs;
            auto group = [](int n) { return n <= 128 ? 0.35 : 0.08 + 0.0021 * n; };
            const double wave = mine * group(n), end = n <= 64 ? 0.0 : 1.5 + 0.01 * n, us = 9.0 + 0.01 * n + exchange + (double)waves * wave + (double)(waves - 1) * end;
            if (us < best.us - 1e-9) best = T2Pick{n, s, 1, us};
            // the last wave's tiles in halves: one wave of them as well, none of them empty
            if (s == 1 && whole > 0 && left > 0 && left * 2 <= pairs && n % 64 == 0 && (M - 1) % n + 1 > n / 2) {
                const double shorter = us - wave + mine * fmax(0.4, group(n / 2));
                if (shorter < best.us - 1e-9) best = T2Pick{n, 1, 2, shorter};
            }
        }
        if (n >= M) break;
    }
    return best;
}

// Whether M tokens are this kernel's.  Beyond 256 w4a16_tc.cu would need several passes; below, tiles on few pairs stand against its ranges
// over all SMs and their exchange: 10 us + 4.2 ns per token and million weights, a quarter more where it works on 128 or 256 tokens for fewer.
// Where its ranges are down to eight groups every tile is cut, and what is exchanged grows with M.
// Measured in a row of calls, N x K, there / here, us: 4096 x 14336 at M = 32 / 64 / 128 / 256 21 / 23 / 36 / 59 and 21 / 22 / 25 / 31; 28672 x 4096 31 / 37 /
// 54 / 105 and 28 / 29 / 37 / 61; 6144 x 4096 15 / 19 / 28 / 49 and 14 / 15 / 17 / 20; 2304 x 1152 at M = 33 / 256 16 / 49 and 10 / 10; 512 x 14336 18 / 34 and
// 18 / 18; 4096 x 4096 at M = 33 / 64 13.1 / 13.7 and 14.1 / 14.3; 10240 x 8192 at M = 17 / 48 24 / 27 and 27 / 28.  The estimates are older than that.  With
// both kernels as they are now, 284 points in graphs (22 sizes from 2048 x 2048 to 27648 x 5120, 17 .. 256 rows): none is sent here that takes longer here (among 95 further points 64 rows of
// 9472 x 8192 are, 27.8 / 22.5, half of the pairs work, and 17 of 18944 x 4096 where the weights come from HBM, 18.8 / 18.4); of the 77 that stay 52 would be the faster ones here by more than 2 %, 10 % on average over the 77: 64 rows of 6144 x 4096 12.7 / 17.8 (here / there), 96 of 2048 x 4096
// 12.0 / 16.3, 128 of 1024 x 8192 12.6 / 16.7 (and 256 of 512 x 14336 18 / 34).  In a feed-forward of 4096 and 14336 at 32 rows both products there take 55.6 us,
// both here 54.6, one of each 55.4 to 57.4; as programmatic dependents in a graph 47.2, 43.8, and 45.0 to 48.1.
bool w4_tc2_route(int M, int N, int K) {
    if (M <= 16 || N % kTcRows || K % kW4GroupK) return false;
    if (M > 256) return true;
    const int G = K / kW4GroupK;
    // Both as they are since each starts under its predecessor's end: here 5.8 us, 0.34 a group of a wave and 1.5 for sums that meet; there 10 us and 0.156 (up to
    // 32 rows) or 11.5 and 0.17 per million weights.  Measured in a row of calls, there / here, 32 and 40 rows, N x K: 14336 x 4096 19.6 / 16.7 and 21.8 / 17.4; 8192 x 8192
    // 19.7 / 18.2 and 23.1 / 18.7; 8192 x 4096 14.8 / 12.9 and 18.0 / 13.4; 5120 x 5120 16.7 / 14.2 and 17.8 / 14.8; 16384 x 2048 15.8 / 11.5 and 17.7 / 12.1; a feed-forward of
    // 2048 and 8192 35.5 / 28.4 and 35.4 / 27.7; not 10240 x 8192 23.4 / 28.0 and 25.9 / 28.8 (40 pairs of 74 work), 22016 x 4096 24.2 / 27.3 and 27.0 / 28.1 (a second
    // wave of 12).  Where they are closer, and below 26 million weights, the older estimates below decide.
    const double weights = 1e-6 * N * K;
    if (M <= 64 && weights >= 26.0) {
        const T2Pick pick = t2_pick(M, cdiv(N, kTc2Rows), G);
        const int pairs = device_sm_count() / 2, sub = t2_sub(pick.ntok), mine = cdiv(cdiv(G, sub), pick.splits) * sub;
        const double here = 5.8 + 0.34 * mine * cdiv(cdiv(N, kTc2Rows) * cdiv(M, pick.ntok), pairs) + (pick.splits > 1 ? 1.5 : 0.0);
        if (M <= 32 ? here < 0.9 * (10.0 + 0.156 * weights) : here < 0.85 * (11.5 + 0.17 * weights)) return true;
    }
    const double there = (10.0 + 4.2e-9 * M * (double)N * K) * (M > 64 && N >= 4096 ? 1.25 : 1.0);
    const bool cut = M > 32 && (long long)(N / kTcRows) * G < 8 * device_sm_count();
    return t2_pick(M, cdiv(N, kTc2Rows), G).us < there + (!cut ? 0.0 : K < 4096 ? 0.1 * M : N >= 1024 ? 0.015 * M : 0.0);
}

// all M tokens in one launch
cudaError_t launch_w4_tc2(const W4Params& p, bool pdl, cudaStream_t stream) {
    const int row_tiles = cdiv(p.N, kTc2Rows), G = p.K / kW4GroupK, max_pairs = device_sm_count() / 2;
    W4TcParams q;
    unsigned* words = wait_words();
    if (!words) return cudaErrorMemoryAllocation;
    if (!w4_tc_params(q, p)) return cudaErrorInvalidValue;
    q.err = words + kWaitW4Pairs;
    const T2Pick pick = t2_pick(p.mc, row_tiles, G);
    const int sub = t2_sub(pick.ntok);
    q.ntok = pick.ntok;
    q.splits = pick.splits;
    q.tok_tiles = cdiv(p.mc, q.ntok);
    int tiles = row_tiles * q.tok_tiles;
    q.cut = pick.cut;
    q.whole = pick.cut > 1 ? tiles / max_pairs * max_pairs : tiles;
    tiles = q.whole + (tiles - q.whole) * q.cut;
    {   // x as [K / 64][M][64]: a stage's atoms of half the tokens are one box
        const uint64_t dims[3] = {64, (uint64_t)p.mc, (uint64_t)p.K / 64}, strides[2] = {(uint64_t)p.ldx * 2, 128};
        const uint32_t box[3] = {64, (uint32_t)q.ntok / 2, (uint32_t)(2 * sub)};
        if (!tc_make_map_nd(&q.xmap, p.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return cudaErrorInvalidValue;
    }
    return launch_pairs(t2_kernel(sub, p.epi), (tiles < max_pairs ? tiles : max_pairs) * q.splits, q.splits, dim3(T2Cfg::kThreads),
                        (size_t)T2Cfg::kBytes, stream, pdl, q);
}

}  // namespace zl

extern "C" int zl_w4_pairs_rings(int ntok, int* slots, int* raw_slots) {
    ZL_CHECK_ARG(ntok >= 32 && ntok <= 256 && ntok % 32 == 0 && slots && raw_slots);
    *slots = zl::t2_slots(ntok);
    *raw_slots = zl::t2_raw_slots(ntok);
    return ZL_OK;
}

extern "C" int zl_w4_pairs_splits(int M, int N, int K) {
    return zl_w4_pairs_route(M, N, K) ? zl::t2_pick(M, zl::cdiv(N, zl::kTc2Rows), K / zl::kW4GroupK).splits : 0;
}

extern "C" int zl_w4_pairs_pieces(int M, int N, int K) {
    return zl_w4_pairs_route(M, N, K) ? zl::t2_pick(M, zl::cdiv(N, zl::kTc2Rows), K / zl::kW4GroupK).cut : 0;
}

extern "C" unsigned zl_w4_tc2_watchdog(void) {
    cudaDeviceSynchronize();
    const unsigned* words = zl::wait_words();
    return words ? words[zl::kWaitW4Pairs] : 0u;
}
