// General GEMM y[b](M, N) = epi(x[b](M, K) @ w[b](N, K)^T + bias) of 16-bit inputs on the 5th-generation tensor cores, for prompt-sized
// M: the counterpart of gemm_tiled.cu's mma.sync kernel and of dense_gemm.cu's 32-row passes, same epilogues, same fp32
// accumulation, and the grouped form of a mixture of experts.
//
// A tile is 256 rows of w (tcgen05.mma's A operand, 128 per CTA of the pair) by up to 256 rows of x (the B operand, half per CTA):
// per 64-k stage each SM loads 16 KB of w and 16 KB of x for 512 cycles of MMA, where 64 x 64 tiles on mma.sync load 16 KB for 64
// cycles' worth.  Operands through tensor-TMA in six stages of 128-byte swizzled rows, two accumulators in TMEM so that a tile's
// epilogue runs under the next tile's MMAs, persistent pairs of CTAs that take the tiles in turn.  bf16, 14336 x 4096: M = 2048
// 970 -> 171 us (1410 TFLOP/s), M = 512 268 -> 55 us, M = 64 69 -> 30 us; 8192 x 2048, M = 1024: 154 -> 34 us.  Bound by the tensor
// cores from about 1000 rows on, below by the loads of w and by tiles that do not fill the pairs: 4096 x 14336 has 16 of them for 74 pairs at M <= 256
// (200 us on mma.sync, 42.6 with a pair each, 37.2 where two share one).
//
//   warp 0       producer  : w and x boxes, one lane
//   warp 1       MMA       : of the leader, one lane, 4 x 256 x ntok x 16 per 64-k block
//   warp 2       TMEM allocation
//   warps 4-11   epilogue  : quadrant = warp % 4, 16-row chunks of x in turns; lane = row of w = column of y; of the last tile all warps
//   warps 12-15  grouped   : rows of x through their index lists, by 16-byte cp.async into the swizzled layout that the boxes have;
//                            a stage's barrier counts the copies as they land, warp 3 hands the stage to the MMAs
//
// The issuing lanes look at their next barrier while this stage's work is on its way (a look costs 120 - 200 cycles, a warp's vote with it
// more): bf16 4096 x 4096, 512 rows 27.0 -> 21.8 us; 14336 x 4096, 777 rows 85 -> 75; int8 8192 x 8192, 24 rows 22.8 -> 19.4; 16 experts of 2048 x 2048,
// 2048 rows 85.6 + 49.6 -> 79 + 47.  Few tiles over a long K: the pairs of a cluster share a tile's K (gt_pick).
//
// The 8-bit Linears (zl_w8a8_gemm: Int8Linear, Fp8Linear) run on the same kernel: a stage is 128 bytes of k whatever the type, only the MMA
// (kind::i8 with s32 accumulators, kind::f8f6f4) and the epilogue (scale-back, bias) are theirs.
#include "gemm_common.cuh"
#include "tc2_common.cuh"

#include <type_traits>

namespace zl {

constexpr int kGtThreads = 16 * 32, kGtRowWarps = 4, kGtEpiWarps = 8, kGtSets = 4;   // sets of four warps, one per quadrant of TMEM lanes
// The ring is cut into as many stages as fit, of blocks of 16 KB of w and 128 bytes per row of a CTA's half tile of x.
constexpr int kGtRing = 204800, kGtMaxStages = 12, kGtAStage = 128 * 128;
constexpr int kGtBarOff = kGtRing;
constexpr int kGtMiscOff = kGtBarOff + (3 * kGtMaxStages + 5) * 8;
constexpr int kGtMaxGroups = 1024;
constexpr int kGtCumOff = kGtMiscOff + 16;                       // grouped: tiles before each group
constexpr int kGtBytes = kGtCumOff + (kGtMaxGroups + 1) * 4 + 1024;   // + slack for the manual 1024-byte alignment
static_assert(kGtBytes <= 232448 && tmem_alone(kGtBytes), "shared memory");
enum { kGt16 = 0, kGtInt8 = 1, kGtFp8 = 2 };

struct alignas(64) GemmTcP {
    CUtensorMap wmap;           // w (K, N, batch), box 64 x 128
    CUtensorMap xmap;           // x (K, rows, batch), box 64 x box_rows; not grouped
    GemmP g;
    int epi, groups;            // groups: batch, or the number of groups
    int row_tiles, tok_tiles;   // tok_tiles: not grouped
    int splits;                 // pairs of a cluster that share a tile's K (then a tile per cluster); not grouped
    int ntok, box_rows;         // not grouped: rows of x of a tile, and of a box (a CTA's half of them)
    int wide;                   // two neighbouring values of y may be stored together
    int stages, sub;            // stages of `sub` blocks: 128 bytes of k of w (16 KB) and of x
    int block_bytes;
    const float* sx;            // 8-bit: scales of the rows of x (int8) or one (fp8)
    const void* sw;             // 8-bit: scales of the rows of w, or one
    int sw_mode;                // 0: per row in y's type, 1 / 2: per row fp32, 3: one fp32
    unsigned* err;              // wait_words()[kWaitGemmTc]
    int behind;                 // dependents may start once everything before this kernel has ended
};

struct GtTile {
    int b, n0, t0, ntok, M, first;
};

// tile `i` of the launch; false behind the last one.  Row tiles of a group follow each other with the rows of x innermost, so that
// the pairs working at one time share their rows of w
template <bool GROUPED>
__device__ __forceinline__ bool gt_tile(const GemmTcP& p, const int* s_cum, int i, int& hint, GtTile& t) {
    if constexpr (GROUPED) {
        if (i >= s_cum[p.groups]) return false;
        while (i >= s_cum[hint + 1]) ++hint;
        t.b = hint;
        t.first = p.g.grp_off[hint];
        t.M = p.g.grp_off[hint + 1] - t.first;
        const int tt = (t.M + 255) >> 8, j = i - s_cum[hint];
        t.n0 = (j / tt) * kTc2Rows;
        t.t0 = (j % tt) * 256;
        t.ntok = min(256, (t.M - t.t0 + 31) & ~31);
    } else {
        const int per = p.row_tiles * p.tok_tiles;
        if (i >= per * p.groups) return false;
        t.b = i / per;
        const int j = i - t.b * per;
        t.n0 = (j / p.tok_tiles) * kTc2Rows;
        t.t0 = (j % p.tok_tiles) * p.ntok;
        t.M = p.g.M;
        t.first = 0;
        t.ntok = min(p.ntok, (t.M - t.t0 + 31) & ~31);
    }
    return true;
}

// two values of a 16-bit type, the first one below
template <typename TO>
__device__ __forceinline__ uint32_t gt_pack2(float a, float b) {
    if constexpr (std::is_same<TO, __half>::value) {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
}
// own: two rows of y of this lane's column, other: of the neighbour's; the first row of both for the lane of the lower column, the second for the other's
__device__ __forceinline__ uint32_t gt_trade(uint32_t own, uint32_t other, bool upper) { return __byte_perm(own, other, upper ? 0x3276 : 0x5410); }

// 16 rows of y, column n of this lane; mine: row of y of token c0 + lane (grouped).  Two columns of every other token per lane (wide): half the stores, twice
// as wide.  16-bit values travel in pairs and the last rows alone are looked at one by one: the instructions are what a tile's end takes, 1250 cycles a
// chunk with a look, a conversion and a product of addresses for each value.
template <typename TO>
__device__ __forceinline__ void gt_put16(const GemmTcP& p, const GtTile& t, TO* y, int mine, int n, int c0, const float (&v)[16], int lane) {
    const GemmP& g = p.g;
    const int odd = lane & 1;
    if (sizeof(TO) == 2 && p.wide) {
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t own = gt_pack2<TO>(v[2 * j], v[2 * j + 1]);
            w[j] = gt_trade(own, __shfl_xor_sync(0xffffffffu, own, 1), odd);
        }
        const int first = t.t0 + c0 + odd, left = n < g.N ? t.M - first : 0;   // N is even
        TO* at = y + (n & ~1);
        if (g.grp_off) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int row = __shfl_sync(0xffffffffu, mine, 2 * j + odd);
                if (2 * j < left) *reinterpret_cast<uint32_t*>(at + (size_t)row * g.ldy) = w[j];
            }
        } else {
            at += (size_t)first * g.ldy;
            const size_t step = 2 * (size_t)g.ldy;
            if (left >= 15) {
#pragma unroll
                for (int j = 0; j < 8; ++j, at += step) *reinterpret_cast<uint32_t*>(at) = w[j];
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j, at += step)
                    if (2 * j < left) *reinterpret_cast<uint32_t*>(at) = w[j];
            }
        }
    } else if (p.wide) {
        const int first = t.t0 + c0 + odd, left = n < g.N ? t.M - first : 0;   // N is even
        struct alignas(2 * sizeof(TO)) Two {
            TO a, b;
        };
        auto two = [&](int j) {
            const float other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * j] : v[2 * j + 1], 1);
            return Two{from_f32<TO>(odd ? other : v[2 * j]), from_f32<TO>(odd ? v[2 * j + 1] : other)};
        };
        TO* at = y + (n & ~1);
        if (g.grp_off) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const Two w = two(j);
                const int row = __shfl_sync(0xffffffffu, mine, 2 * j + odd);
                if (2 * j < left) *reinterpret_cast<Two*>(at + (size_t)row * g.ldy) = w;
            }
        } else {
            at += (size_t)first * g.ldy;
            const size_t step = 2 * (size_t)g.ldy;
#pragma unroll
            for (int j = 0; j < 8; ++j, at += step) {
                const Two w = two(j);
                if (2 * j < left) *reinterpret_cast<Two*>(at) = w;
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int m = t.t0 + c0 + i;
            const int row = g.grp_off ? __shfl_sync(0xffffffffu, mine, i) : m;
            if (n < g.N && m < t.M) y[(size_t)row * g.ldy + n] = from_f32<TO>(v[i]);
        }
    }
}

template <typename T, typename TO, int EPI>
__device__ __forceinline__ void gt_store16(const GemmTcP& p, const GtTile& t, int n, int c0, float (&v)[16], float bias, int lane) {
    const GemmP& g = p.g;
    TO* y = static_cast<TO*>(g.y) + (size_t)t.b * (g.grp_off ? 0 : g.yb);
    int mine = 0;   // row of y of token c0 + lane
    if (g.grp_off) {
        const int m = t.t0 + c0 + (lane & 15);
        mine = m < t.M ? (g.y_rows ? g.y_rows[t.first + m] : t.first + m) : 0;
    }
    const int odd = lane & 1;
    if constexpr (epi_pairs(EPI)) {
        // gate and up of an output sit in neighbouring lanes: the even lane takes the tokens 0, 2, ..., the odd one 1, 3, ...
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float a0 = v[2 * j] + bias, a1 = v[2 * j + 1] + bias;
            const float other = __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 1);
            v[j] = pair_unit<EPI>(odd ? other : a0, odd ? a1 : other, g);
        }
        if (sizeof(TO) == 2 && p.wide) {   // two columns of every other one of its tokens per lane
            const bool up = lane & 2;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t own = gt_pack2<TO>(v[2 * i], v[2 * i + 1]), w = gt_trade(own, __shfl_xor_sync(0xffffffffu, own, 2), up);
                const int at = 4 * i + 2 * up + odd, m = t.t0 + c0 + at;
                const int row = g.grp_off ? __shfl_sync(0xffffffffu, mine, at) : m;
                if (n < g.N && m < t.M) *reinterpret_cast<uint32_t*>(y + (size_t)row * g.ldy + ((n >> 1) & ~1)) = w;   // N % 4 == 0
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int m = t.t0 + c0 + 2 * j + odd;
                const int row = g.grp_off ? __shfl_sync(0xffffffffu, mine, 2 * j + odd) : m;
                if ((n | 1) < g.N && m < t.M) y[(size_t)row * g.ldy + (n >> 1)] = from_f32<TO>(v[j]);
            }
        }
    } else {
        // results first, stores behind them: the compiler cannot tell y from the gate's values
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int m = t.t0 + c0 + i;
            constexpr bool kReads = EPI == ZL_GEMM_EPI_SIGMOID_GATE || EPI == ZL_GEMM_EPI_GELU_TANH_MUL;
            v[i] = !kReads || (m < t.M && n < g.N) ? gemm_epilogue<EPI>(v[i] + bias, g, t.b, m, n) : 0.f;
        }
        gt_put16<TO>(p, t, y, mine, n, c0, v, lane);
    }
}

// 8-bit: v are the raw accumulators (s32 bits or f32)
template <typename TO, int KIND>
__device__ __forceinline__ void gt_store16_8bit(const GemmTcP& p, const GtTile& t, int n, int c0, float (&v)[16], float s_w, float bias, bool has_bias,
                                                int lane) {
    const int mt = t.t0 + c0 + (lane & 15);
    const float scales = KIND == kGtFp8 ? p.sx[0] * s_w : (mt < t.M ? p.sx[mt] : 0.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if constexpr (KIND == kGtFp8) {
            v[i] *= scales;                                       // cuBLASLt fp8: D = (scaleA * scaleB) * acc (+ bias)
            if (has_bias) v[i] += bias;
        } else {
            // quant_scale_back (quant_kernel.cu:231-246): T(float(acc) * sx[m] * sw[n]), then add_bias in T
            v[i] = __fmul_rn(__fmul_rn((float)__float_as_int(v[i]), __shfl_sync(0xffffffffu, scales, i)), s_w);
            if (has_bias) v[i] = to_f32<TO>(from_f32<TO>(v[i])) + bias;
        }
    }
    gt_put16<TO>(p, t, static_cast<TO*>(p.g.y), 0, n, c0, v, lane);
}

template <typename T, typename TO, bool GROUPED, int KIND, int SUB>
__global__ void __launch_bounds__(kGtThreads, 1) k_gemm_tc(const __grid_constant__ GemmTcP p) {
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kGtBarOff);
    uint64_t* empty = full + kGtMaxStages;
    uint64_t* acc_full = empty + kGtMaxStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* last_full = acc_empty + 2;       // the pair's last tile
    uint64_t* rows_full = last_full + 1;       // grouped: this CTA's rows of a stage have landed
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + kGtMiscOff);
    volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
    int* s_cum = reinterpret_cast<int*>(smem + kGtCumOff);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = GROUPED ? 1 : p.splits;
    const uint32_t in_cluster = cluster_rank(), rank = in_cluster & 1, lead = in_cluster & ~1u;   // lead: the pair's leader
    const int part = (int)(in_cluster >> 1);
    const int pair = (int)(blockIdx.x >> 1) / splits, pairs = (int)(gridDim.x >> 1) / splits;
    constexpr int kBlockK = KIND == kGt16 ? 64 : 128;   // 128 bytes
    constexpr int sub = SUB;
    const int stages = p.stages, block_bytes = p.block_bytes, stage_bytes = sub * block_bytes;
    const int ks_all = (p.g.K + kBlockK * sub - 1) / (kBlockK * sub);
    const int k_first = (int)((long long)ks_all * part / splits), ks = (int)((long long)ks_all * (part + 1) / splits) - k_first;

    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; ++i) {
            mbar_init(&full[i], GROUPED ? 3 : 1);
            mbar_init(&empty[i], 1);
            mbar_init(&rows_full[i], kGtRowWarps * 32);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 2 * kGtEpiWarps);
        }
        mbar_init(last_full, 1);
        *s_abort = 0;
        mbar_fence_init();
    }
    if (warp == 2) tc2_alloc(s_tmem);
    if (!p.behind) pdl_trigger();
    if (KIND == kGt16) pdl_wait();   // 8-bit: below; the weights do not wait for the rows' quantisation (8192 x 8192, 24 rows: 1 us)
    if (p.behind) pdl_trigger();
    if (GROUPED && warp == 3) {   // tiles before each group: a running sum over the groups' sizes
        int base = 0;
        for (int g0 = 0; g0 < p.groups; g0 += 32) {
            const int g = g0 + lane;
            int c = 0;
            if (g < p.groups) c = ((p.g.grp_off[g + 1] - p.g.grp_off[g] + 255) >> 8) * p.row_tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, c, o);
                if (lane >= o) c += u;
            }
            if (g < p.groups) s_cum[g + 1] = base + c;
            base += __shfl_sync(0xffffffffu, c, 31);
        }
        if (lane == 0) s_cum[0] = 0;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers and allocations are in place
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const int total = GROUPED ? s_cum[p.groups] : p.row_tiles * p.tok_tiles * p.groups;

    // The three loops below are one lane's each: a vote or a look at a barrier costs the warp 100 - 200 cycles a stage, so each looks at its next
    // barrier while this stage's copies or MMAs are on their way
    if (warp == 0) {
        if (tc_elect_one()) {
            int st = 0, hint = 0;
            uint32_t ph = 0;
            GtTile t;
            bool ok = true, free = false;
            const uint32_t bytes = 2u * sub * (kGtAStage + (GROUPED ? 0 : p.box_rows * 128));
            auto weights = [&](int at, int k) {   // the stage's bytes and this CTA's half of its weight rows
                const uint32_t bar = cluster_map(smem_u32(&full[at]), lead);
                if (rank == 0) mbar_expect_tx(&full[at], bytes);
#pragma unroll
                for (int u = 0; u < sub; ++u)     // a block behind K arrives as zeros
                    tma2_load_3d(smem + at * stage_bytes + u * block_bytes, &p.wmap, ((k_first + k) * sub + u) * kBlockK, t.n0 + (int)rank * 128, t.b, bar);
            };
            int ahead = 0;                        // stages of the first tile whose weights are on their way already
            if (KIND != kGt16) {
                if (gt_tile<GROUPED>(p, s_cum, pair, hint, t)) ahead = min(stages, ks);
                for (int k = 0; k < ahead; ++k) weights(k, k);
                pdl_wait();
            }
            for (int i = pair; ok && gt_tile<GROUPED>(p, s_cum, i, hint, t); i += pairs) {
                const int tb = t.t0 + (int)rank * (t.ntok >> 1);
                for (int k = 0; k < ks; ++k) {
                    if (!free && !(ok = tc2_wait1(&empty[st], ph ^ 1u, s_abort, p.err, 0x2100 + st))) break;
                    const int at = st;
                    if (++st == stages) {
                        st = 0;
                        ph ^= 1u;
                    }
                    free = mbar_test(&empty[st], ph ^ 1u);
                    if (KIND == kGt16 || ahead <= 0) weights(at, k);
                    if (!GROUPED) {
                        const uint32_t bar = cluster_map(smem_u32(&full[at]), lead);
#pragma unroll
                        for (int u = 0; u < sub; ++u)
                            tma2_load_3d(smem + at * stage_bytes + u * block_bytes + kGtAStage, &p.xmap, ((k_first + k) * sub + u) * kBlockK, tb, t.b, bar);
                    }
                    --ahead;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1 && rank == 0) {
        if (KIND != kGt16) pdl_wait();       // nothing of use arrives before, and the bounded waits start here
        if (tc_elect_one()) {
            int st = 0, acc = 0, hint = 0;
            uint32_t ph = 0, acc_ph = 0;
            GtTile t;
            bool ok = true, ready = false;
            for (int i = pair; ok && gt_tile<GROUPED>(p, s_cum, i, hint, t); i += pairs) {
                if (!(ok = tc2_wait1(&acc_empty[acc], acc_ph ^ 1u, s_abort, p.err, 0x2300 + acc))) break;
                const uint32_t d = tmem + (uint32_t)(acc * 256);
                const uint32_t idesc = KIND == kGt16 ? tc2_idesc(std::is_same<T, __nv_bfloat16>::value, t.ntok) : tc2_idesc8(KIND == kGtFp8, t.ntok);
                for (int k = 0; k < ks; ++k) {
                    if (!ready && !(ok = tc2_wait1(&full[st], ph, s_abort, p.err, 0x2400 + st))) break;
                    const uint32_t base = smem_u32(smem + st * stage_bytes);
                    uint64_t* const used = &empty[st];
                    if (++st == stages) {
                        st = 0;
                        ph ^= 1u;
                    }
                    ready = mbar_test(&full[st], ph);
                    tc_fence_after();
#pragma unroll
                    for (int u = 0; u < sub; ++u) {
                        const uint64_t ad = tc_desc_sw128(base + u * block_bytes), bd = tc_desc_sw128(base + u * block_bytes + kGtAStage);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {   // 32 bytes of k per MMA
                            const uint64_t a = ad + (uint64_t)(j * 2), b = bd + (uint64_t)(j * 2);
                            const uint32_t accum = (k > 0 || u > 0 || j > 0) ? 1u : 0u;
                            if constexpr (KIND == kGt16) tc2_mma_ss(d, a, b, idesc, accum);
                            else tc2_mma_ss8<KIND == kGtFp8>(d, a, b, idesc, accum);
                        }
                    }
                    tc2_commit(used, lead);
                    if (k == ks - 1) tc2_commit(i + pairs < total ? &acc_full[acc] : last_full, lead);
                }
                if (++acc == 2) {
                    acc = 0;
                    acc_ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (GROUPED && warp == 3) {
        // rows that have landed become visible to the proxy the MMAs read through, then count as arrived at the leader
        if (tc_elect_one()) {
            int st = 0, hint = 0;
            uint32_t ph = 0;
            GtTile t;
            bool ok = true, ready = false;
            for (int i = pair; ok && gt_tile<GROUPED>(p, s_cum, i, hint, t); i += pairs)
                for (int k = 0; k < ks; ++k) {
                    if (!ready && !(ok = tc2_wait1(&rows_full[st], ph, s_abort, p.err, 0x2500 + st))) break;
                    const uint32_t to = cluster_map(smem_u32(&full[st]), lead);
                    if (++st == stages) {
                        st = 0;
                        ph ^= 1u;
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_arrive_at(to);
                    ready = mbar_test(&rows_full[st], ph);
                }
        }
        __syncwarp();
    } else if (GROUPED && warp >= 4 + kGtEpiWarps) {
        // thread: 16-byte chunk c of rows j, j + 16, ... of the CTA's half
        const int tid = threadIdx.x - 12 * 32, c = tid & 7, j = tid >> 3;
        const uint32_t sm = smem_u32(smem) + kGtAStage + (uint32_t)(j * 128 + ((c ^ (j & 7)) << 4));
        int st = 0, hint = 0;
        uint32_t ph = 0;
        GtTile t;
        bool ok = true, free = false;
        for (int i = pair; ok && gt_tile<GROUPED>(p, s_cum, i, hint, t); i += pairs) {
            const int half = t.ntok >> 1, tb = t.t0 + (int)rank * half;
            const T* row[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {   // rows behind the group's end load its first row and are not stored
                const int m = tb + j + u * 16, e = t.first + (m < t.M ? m : 0);
                row[u] = static_cast<const T*>(p.g.x) + (size_t)(p.g.x_rows ? p.g.x_rows[e] : e) * p.g.ldx + c * 8;
            }
            for (int k = 0; k < ks; ++k) {
                if (!__all_sync(0xffffffffu, free) && !(ok = tc2_wait(&empty[st], ph ^ 1u, s_abort, p.err, 0x2200 + st))) break;
                free = st + 1 < stages ? mbar_test(&empty[st + 1], ph ^ 1u) : mbar_test(&empty[0], ph);
#pragma unroll
                for (int u2 = 0; u2 < sub; ++u2) {
                    const int k0 = (k * sub + u2) * 64;
                    const bool in = k0 + c * 8 < p.g.K;
                    const int bytes = in ? 16 : 0;   // 0: zeros, nothing is read
                    const uint32_t dst = sm + (uint32_t)(st * stage_bytes + u2 * block_bytes);
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (u * 16 < half)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(u * 2048)),
                                         "l"(in ? row[u] + k0 : row[u] - c * 8), "r"(bytes)
                                         : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&rows_full[st])) : "memory");
                if (++st == stages) {
                    st = 0;
                    ph ^= 1u;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    // The epilogue warps' tiles.  The last one is everybody's: nothing is left to hide its end, and the other warps have nothing else to do.  With the shorter
    // chunks of gt_put16, in a row of calls: bf16 8192 x 2048, 777 rows 31.3 -> 29.0 us; 16 experts of 2048 x 2048, 512 rows in four each: 127.5 -> 121.8;
    // fp8 14336 x 4096, 500 rows 41.1 -> 39.6.  With K split a tile's only chunks come behind the exchange below.
    const int q = warp & 3, set = ((warp >> 2) + kGtSets - 1) % kGtSets;   // 0, 1: the epilogue warps
    float bias = 0.f, s_w = 0.f;
    auto row_values = [&](const GtTile& t, int n) {
        bias = s_w = 0.f;
        if (n < p.g.N) {
            if (KIND != kGt16)
                s_w = p.sw_mode == 0 ? to_f32<T>(static_cast<const T*>(p.sw)[n]) : static_cast<const float*>(p.sw)[p.sw_mode == 3 ? 0 : n];
            if (p.g.bias) bias = p.g.bias[(size_t)t.b * p.g.bb + n];
            else if (p.g.bias_t) bias = to_f32<T>(static_cast<const T*>(p.g.bias_t)[n]);
        }
    };
    auto put = [&](const GtTile& t, int n, int c0, float (&v)[16]) {
        if constexpr (KIND != kGt16) {
            gt_store16_8bit<TO, KIND>(p, t, n, c0, v, s_w, bias, p.g.bias_t != nullptr, lane);
        } else {
            switch (p.epi) {
#define ZL_GT_EPI(E) case E: gt_store16<T, TO, E>(p, t, n, c0, v, bias, lane); break;
                ZL_GT_EPI(ZL_GEMM_EPI_RELU2)
                ZL_GT_EPI(ZL_GEMM_EPI_SIGMOID_GATE)
                ZL_GT_EPI(ZL_GEMM_EPI_TANH)
                ZL_GT_EPI(ZL_GEMM_EPI_GLU_CLAMP)
                ZL_GT_EPI(ZL_GEMM_EPI_GEGLU_TANH)
                ZL_GT_EPI(ZL_GEMM_EPI_GELU_TANH_MUL)
                ZL_GT_EPI(ZL_GEMM_EPI_SOFTCAP)
                ZL_GT_EPI(ZL_GEMM_EPI_REGLU)
                default: gt_store16<T, TO, ZL_GEMM_EPI_NONE>(p, t, n, c0, v, bias, lane);
#undef ZL_GT_EPI
            }
        }
    };
    {
        if (KIND != kGt16) pdl_wait();
        const int tiles = pair < total ? (total - pair + pairs - 1) / pairs : 0;
        // The helpers sleep at a barrier of the SM until the first set has seen the last tile: eight more warps that poll would take issue slots from the
        // lanes that load and multiply (4096 x 4096, 40 rows: 10.9 -> 10.4 us; int8 8192 x 8192, 24 rows, with the scales ahead of the exchange, 19.7 -> 18.4)
        constexpr int kMeet = (kGtSets - 1) * 128;
        const bool helps = set >= 2, meet = tiles > 0 && splits == 1;
        bool told = false;
        int hint = 0;
        GtTile t;
        for (int j = helps ? tiles - 1 : 0; j >= 0 && j < tiles && !(helps && !meet); ++j) {
            const int acc = j & 1;
            const bool last = j == tiles - 1;
            // which tile, its bias and its scales ahead of the wait
            if (GROUPED && helps) {   // whose group lies anywhere: a walk from the first of 64 groups on took as long as the tile's end, 1.2 us
                int end = p.groups;
                while (end - hint > 1) {
                    const int mid = (hint + end) >> 1;
                    (s_cum[mid] <= pair + j * pairs ? hint : end) = mid;
                }
            }
            gt_tile<GROUPED>(p, s_cum, pair + j * pairs, hint, t);
            const int n = t.n0 + (int)rank * 128 + q * 32 + lane, step = last ? 16 * kGtSets : 32;
            if (splits == 1) row_values(t, n);
            if (helps) asm volatile("bar.sync 2, %0;" ::"n"(kMeet) : "memory");
            const bool ok = helps ? !*s_abort : tc2_wait(last ? last_full : &acc_full[acc], last ? 0u : (uint32_t)(j >> 1) & 1u, s_abort, p.err, 0x2800 + acc);
            if (last && set == 0 && meet) {
                asm volatile("bar.arrive 2, %0;" ::"n"(kMeet) : "memory");
                told = true;
            }
            if (!ok) break;
            tc_fence_after();
            if (splits > 1) break;
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 256);
            for (int c0 = set * 16; c0 < t.ntok && t.t0 + c0 < t.M; c0 += step) {
                float v[16];
                tc_ld16(taddr + (uint32_t)c0, v);
                put(t, n, c0, v);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && !last) mbar_arrive_at(cluster_map(smem_u32(&acc_empty[acc]), lead));
        }
        if (set == 0 && meet && !told) asm volatile("bar.arrive 2, %0;" ::"n"(kMeet) : "memory");   // gave up on an earlier tile
    }
    GtTile t;
    int at = 0;
    const bool any = !GROUPED && splits > 1 && gt_tile<GROUPED>(p, s_cum, pair, at, t);
    const int row = q * 32 + lane, n = any ? t.n0 + (int)rank * 128 + row : 0;
    if (any) row_values(t, n);   // their round trip ahead of the exchange: int8 8192 x 2048, 40 rows 12.1 -> 11.3 us
    __syncwarp();
    tc2_drain(s_abort);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // nobody's shared memory or TMEM goes, or takes sums, while another CTA may still use it
    if (!GROUPED && splits > 1) {
        tc_fence_after();
        const int chunks = any ? min(t.ntok, t.M - t.t0 + 15) / 16 : 0;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
        for (int c = set; c < chunks; c += kGtSets) {
            if (c % splits == part) continue;
            float v[16];
            tc_ld16(taddr + (uint32_t)(c * 16), v);
            tc2_split_push(smem_u32(smem), (int)rank, part, c, splits, chunks, row, v);
        }
        cluster_sync_all();
        for (int c = part + set * splits; c < chunks; c += kGtSets * splits) {
            float v[16];
            tc_ld16(taddr + (uint32_t)(c * 16), v);
            tc2_split_sum<KIND == kGtInt8>(smem, part, c, splits, chunks, row, v);
            put(t, n, c * 16, v);
        }
        tc_fence_before();
        __syncthreads();
    }
    if (warp == 2) {
        tc_fence_after();
        tc2_dealloc(tmem);
    }
}

// Rows of x per tile, and how many pairs share a tile's K, for `blocks` 128-byte blocks of k: with few tiles the pairs of a cluster (the device holds
// fit[0] clusters of two pairs at a time, fit[1] of four) take a part each and exchange their sums.  In cycles, fitted to the times below, which are from before all
// warps took part in the exchange and in the last tile's end: a block 190 + 1.4 per row of x, the exchange 2850 + 42 per row.  Measured, one pair / two, us, N x K: bf16 4096 x 14336, 65 rows 39.3 / 31.2, 256 rows
// 42.6 / 37.2; 1024 x 8192, 65 rows 23.3 / 17.2 and 14.9 with four; int8 8192 x 8192, 24 rows 20.3 / 18.9; against it bf16 4096 x 4096, 512 rows
// 22.5 / 25.4; 8192 x 2048, 256 rows 16.9 / 20.9.
struct GtPick {
    int ntok, splits;
};
static GtPick gt_pick(int M, long long rows, int pairs, int blocks, const int (&fit)[2]) {
    GtPick best{32, 1};
    double best_cost = 1e30;
    for (int n = 32; n <= 256; n += 32) {
        const long long tiles = rows * cdiv(M, n), waves = (tiles + pairs - 1) / pairs;
        for (int s = 1; s <= 4; s *= 2) {
            if (s > 1 && (tiles > fit[s / 4] || blocks < 8 * s)) continue;
            const double cost = (double)waves * cdiv(blocks, s) * (190.0 + 1.4 * n) + (s > 1 ? 2850.0 + 42.0 * n : 0.0);
            if (cost < best_cost - 1e-9) {
                best_cost = cost;
                best = GtPick{n, s};
            }
        }
        if (n >= M) break;
    }
    return best;
}

// A short K and few tiles are the tile kernel's: a launch of it costs 2.9 us and 1 us per 100 of k, here the pair's allocation, barriers and
// hand-overs cost 4 us and k a sixth of that.  Both times in us per call of a row of calls in a graph, where this kernel starts under the end of the one
// before it, fitted to 1488 measured shapes (M = 33 .. 512, N = 128 .. 4096, K = 64 .. 1024, 1 .. 48 matrices; above K = 256 this kernel was the
// faster one at all of them): the tile kernel's first wave of 64 x 64 blocks and what each further block's rows cost; here the tile's rows and what a
// further wave of pairs costs.  Measured, tile kernel / here, M x N x K: 33 x 128 x 64 2.8 / 4.0; 256 x 512 x 256 5.5 / 4.4; 384 x 2048 x 256 7.8 / 5.6;
// 16 matrices of 33 x 512 x 128 3.7 / 4.8, of 256 x 128 x 64 3.6 / 5.6; 48 of 200 x 256 x 128 12.4 / 8.9, of 33 x 4096 x 256 37.8 / 25.6.  The estimates err by 6 and 5 %
// on average, so half a microsecond counts as even and stays there.  This kernel has become faster since, the estimates are those of then.  With both as they are now, 768 shapes
// (M = 33 .. 512, N = 128 .. 4096, K = 64 .. 256, 1 .. 48 matrices): this kernel still serves none that the other one would serve faster by more than 2 %, and what stays
// costs up to 94 %, 4 % on average over all: 48 matrices of 200 x 512 x 64 8.0 / 15.6 us (here / there), of 33 x 2048 x 192 10.8 / 17.7, one of 512 x 4096 x 64 5.8 / 8.4.
bool gemm_tile_faster(int M, int N, int K, int batch) {
    if (K > 256) return false;
    const int sms = device_sm_count(), pairs = sms / 2;
    const long long blocks = (long long)batch * cdiv(M, 64) * cdiv(N, 64), rows = (long long)batch * cdiv(N, kTc2Rows);
    const double further = blocks > sms ? (double)(blocks - sms) * M / (64.0 * cdiv(M, 64)) : 0.0;
    const int n = gt_pick(M, rows, pairs, cdiv(K, 64), {0, 0}).ntok;   // too short a K for any pairs to share
    const double waves = (double)((rows * cdiv(M, n) + pairs - 1) / pairs - 1);
    const double tile = 2.9 + 0.0102 * K + further * (0.0086 + 3.1e-5 * K);
    const double here = 3.3 + 0.0017 * K + 0.028 * n + waves * (0.2 + 0.0204 * n + 0.003 * K);
    return tile < here + 0.45;
}

bool gemm_tc_route(const GemmP& p, int batch, int in_dtype) {
    if (in_dtype != ZL_F16 && in_dtype != ZL_BF16) return false;
    // 16-byte aligned bases and pitches (tensor-TMA, cp.async), extents below 2^31
    if ((reinterpret_cast<uintptr_t>(p.x) & 15) || (reinterpret_cast<uintptr_t>(p.w) & 15) || p.ldx % 8 || p.ldw % 8) return false;
    // a batch whose matrices share one x or w (pitch 0) stays with the tile kernel: a tensor map has no zero pitch
    if (batch > 1 && (p.wb % 8 || p.wb <= 0 || (!p.grp_off && (p.xb % 8 || p.xb <= 0)))) return false;
    if (p.N < 128 || p.K < 64) return false;
    // groups: few rows through small matrices are the tile kernel's (32 groups of 1024 x 768: 36 list entries 22 against 27 us, 256
    // entries 30 against 28; 16 of 4096 x 2048: 36 entries 75 against 69 us, 2048 entries 202 against 86)
    if (p.grp_off) return batch <= kGtMaxGroups && p.K % 8 == 0 && (p.M >= 128 || (p.M > 8 && (long long)batch * p.N * p.K >= (64ll << 20)));
    return p.M > 32 && (long long)cdiv(p.N, kTc2Rows) * cdiv(p.M, 32) * batch < (1ll << 30);
}

template <typename T, typename TO, bool GROUPED, int KIND, int SUB>
static cudaError_t launch_gt_sub(const GemmTcP& q, int pairs, bool pdl, cudaStream_t stream) {
    static bool set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(k_gemm_tc<T, TO, GROUPED, KIND, SUB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGtBytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) set[dev] = true;
    }
    return launch_pairs(k_gemm_tc<T, TO, GROUPED, KIND, SUB>, pairs, q.splits, dim3(kGtThreads), (size_t)kGtBytes, stream, pdl, q);
}
template <typename T, typename TO, bool GROUPED, int KIND>
static cudaError_t launch_gt(const GemmTcP& q, int pairs, bool pdl, cudaStream_t stream) {
    if constexpr (!GROUPED)
        if (q.sub == 2) return launch_gt_sub<T, TO, GROUPED, KIND, 2>(q, pairs, pdl, stream);
    return launch_gt_sub<T, TO, GROUPED, KIND, 1>(q, pairs, pdl, stream);
}
template <typename T, typename TO>
static cudaError_t launch_gt16(const GemmTcP& q, bool grouped, int pairs, bool pdl, cudaStream_t stream) {
    return grouped ? launch_gt<T, TO, true, kGt16>(q, pairs, pdl, stream) : launch_gt<T, TO, false, kGt16>(q, pairs, pdl, stream);
}

// clusters of two and of four pairs that the current device holds at a time; 0: none
static void gt_clusters(int (&fit)[2]) {
    static PairsFit known;
    for (int i = 0; i < 2; ++i) fit[i] = pairs_clusters(k_gemm_tc<__half, __half, false, kGt16, 1>, kGtThreads, kGtBytes, 2 << i, known);
}

// tiles, maps and stages of a call; returns the number of pairs, 0 without a map
static int gt_plan(GemmTcP& q, CUtensorMapDataType dt, int batch, int out_bytes) {
    const GemmP& p = q.g;
    const bool grouped = p.grp_off != nullptr;
    int pairs = device_sm_count() / 2;
    unsigned* words = wait_words();
    if (!words) return 0;
    q.err = words + kWaitGemmTc;
    q.groups = batch;
    q.row_tiles = cdiv(p.N, kTc2Rows);
    q.tok_tiles = 0;
    q.ntok = 256;
    q.splits = 1;
    q.wide = p.N % (epi_pairs(q.epi) ? 4 : 2) == 0 && p.ldy % 2 == 0 && p.yb % 2 == 0 && reinterpret_cast<uintptr_t>(p.y) % (2 * out_bytes) == 0;
    if (!tc2_map_3d(&q.wmap, p.w, dt, p.K, p.N, batch, p.ldw, p.wb, 128)) return 0;
    if (!grouped) {
        int fit[2];
        gt_clusters(fit);
        const int block_k = dt == CU_TENSOR_MAP_DATA_TYPE_UINT8 ? 128 : 64;
        const GtPick pick = gt_pick(p.M, (long long)q.row_tiles * batch, pairs, cdiv(p.K, block_k), fit);
        q.ntok = pick.ntok;
        q.splits = pick.splits;
        q.tok_tiles = cdiv(p.M, q.ntok);
        const long long tiles = (long long)q.row_tiles * q.tok_tiles * batch * q.splits;
        if (tiles < pairs) pairs = (int)tiles;
        if (!tc2_map_3d(&q.xmap, p.x, dt, p.K, p.M, batch, p.ldx, p.xb, q.ntok / 2)) return 0;
    }
    q.box_rows = q.ntok / 2;
    q.block_bytes = kGtAStage + q.box_rows * 128;
    // handing a stage over costs the MMA warp more than a small block's MMAs (2 cycles per row of x): small tiles take two blocks per stage
    // (not grouped rows, whose copies come to too few stages then: 87 -> 95 us)
    q.sub = q.ntok <= 128 && !grouped ? 2 : 1;
    const int fit = kGtRing / (q.sub * q.block_bytes);
    q.stages = fit < kGtMaxStages ? fit : kGtMaxStages;
    return pairs;
}

cudaError_t launch_gemm_tc(const GemmP& p, int batch, int in_dtype, int out_dtype, int epilogue, bool pdl, cudaStream_t stream) {
    const bool bf16 = in_dtype == ZL_BF16, grouped = p.grp_off != nullptr;
    GemmTcP q{};
    q.g = p;
    q.epi = epilogue;
    const int pairs = gt_plan(q, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, batch, out_dtype == ZL_F32 ? 4 : 2);
    if (pairs <= 0) return cudaErrorNotSupported;
    // The 16-bit kernel touches nothing of its predecessor's before it has waited for it, so its allocation, barriers and cluster launch run under the
    // predecessor's end whatever the caller's chain allows.  A caller that did not ask for that may have a dependent which reads what was written
    // before this kernel without waiting: it starts behind the wait.  In a row of calls: bf16 8192 x 2048, 777 rows 32.8 -> 30.6 us; 1280 -> 8288,
    // 164 rows 12.4 -> 10.0; both products of 16 experts 129 -> 123.
    q.behind = !pdl;
    pdl = true;
    if (bf16) return out_dtype == ZL_F32 ? launch_gt16<__nv_bfloat16, float>(q, grouped, pairs, pdl, stream)
                                         : launch_gt16<__nv_bfloat16, __nv_bfloat16>(q, grouped, pairs, pdl, stream);
    return out_dtype == ZL_F32 ? launch_gt16<__half, float>(q, grouped, pairs, pdl, stream) : launch_gt16<__half, __half>(q, grouped, pairs, pdl, stream);
}

template <typename T, bool FP8>
cudaError_t launch_w8_gemm_tc(const uint8_t* xq, const float* sx, const uint8_t* w, const void* sw, int sw_mode, const T* bias, T* y, int M, int N, int K,
                              bool pdl, cudaStream_t stream) {
    GemmTcP q{};
    q.g = GemmP{xq, w, y, nullptr, K, 0, K, 0, N, 0, 0, 0, M, N, K};
    q.g.bias_t = bias;
    q.sx = sx;
    q.sw = sw;
    q.sw_mode = sw_mode;
    const int pairs = gt_plan(q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 2);
    if (pairs <= 0) return cudaErrorNotSupported;
    return launch_gt<T, T, false, FP8 ? kGtFp8 : kGtInt8>(q, pairs, pdl, stream);
}
#define ZL_W8_TC(T, F8)                                                                                                                    \
    template cudaError_t launch_w8_gemm_tc<T, F8>(const uint8_t*, const float*, const uint8_t*, const void*, int, const T*, T*, int, int, int, bool, \
                                                  cudaStream_t);
ZL_W8_TC(__half, false)
ZL_W8_TC(__half, true)
ZL_W8_TC(__nv_bfloat16, false)
ZL_W8_TC(__nv_bfloat16, true)
#undef ZL_W8_TC

}  // namespace zl

extern "C" int zl_gemm_pairs_splits(int M, int N, int K, int batch, int elem_bytes) {
    if (M <= 0 || N <= 0 || K <= 0 || batch <= 0 || (elem_bytes != 1 && elem_bytes != 2)) return 0;
    int fit[2];
    zl::gt_clusters(fit);
    return zl::gt_pick(M, (long long)zl::cdiv(N, zl::kTc2Rows) * batch, zl::device_sm_count() / 2, zl::cdiv(K, 128 / elem_bytes), fit).splits;
}

extern "C" unsigned zl_gemm_tc_watchdog(void) {
    cudaDeviceSynchronize();
    const unsigned* words = zl::wait_words();
    return words ? words[zl::kWaitGemmTc] : 0u;
}
