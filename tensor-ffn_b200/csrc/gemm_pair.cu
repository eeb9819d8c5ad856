// Tensor-core GEMM of prompts and training batches: the products of gemm_tc.cu where there are enough rows to fill the
// chip with 256-row tiles.
//     out[t, n] = epilogue( sum_k X[t,k] * W[n,k] )
// Two CTAs (a cluster, two neighbouring SMs) share one 256-token x BN-weight-row tile as one tcgen05.mma.cta_group::2:
// each stages its 128 tokens and half of the weight rows, so a stage's 32 KB feed twice the products of a single CTA's.
// Persistent: a pair walks over tiles (token tiles first, so that a weight row is fetched from HBM once), and the
// accumulator alternates between two TMEM regions so that a tile's epilogue runs under the next tile's products.
//   warp 0    TMA producer (both CTAs; completions of both are counted by the leader's barrier)
//   warp 1    TMEM allocation; in the leader also tcgen05.mma
//   warps 2-9 epilogue: lane = token, registers = consecutive output columns (gate beside up, a rotary pair beside each
//             other), transposed 32 x 32 through shared memory so that global accesses are 64 to 128 bytes of a row
// Here the tokens are the MMA's rows (gemm_tc.cu has the weights there, which suits few tokens).
// Tiles that would be a last wave on less than half of the pairs are split along K where that pays (pair_split): every part leaves its
// fp32 sums in scratch memory, and per warp the last part to finish (a ticket, no waiting) adds all of them in order and finishes the tile.
// Two operand pairs of different scale (base and expert down projections) take both TMEM regions as accumulators; their K
// extent is long, so the exposed epilogue weighs little.
#include "kernels.h"
#include "ptx.cuh"
#include "launch.h"
#include <cstring>

namespace tffn {

namespace {

constexpr int kPairTokens = 256, kHalf = 128, BK = 64;
constexpr int kEpiWarps = 8, kPairThreads = 64 + 32 * kEpiWarps;
constexpr int kStageRow = 128;  // bytes of a row in a warp's transposition buffer: 32 fp32 columns

template <int BN>
struct PairCfg {
    static constexpr int A_BYTES = kHalf * BK * 2;
    static constexpr int B_BYTES = (BN / 2) * BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = 196608 / STAGE_BYTES;  // 192 KB in flight per SM
    static constexpr int EPI_BYTES = kEpiWarps * 32 * kStageRow;
    static constexpr int SMEM = STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*align*/ + 256 /*barriers*/;
    static constexpr int TMEM_COLS = 2 * BN;
};

struct PairDev {
    CUtensorMap tmW[4];  // [problem * 2 + operand pair]; GEMM_SWIGLU: gate, up
    CUtensorMap tmX[4];
    int kblocks[2];
    int N, T, m_tiles, n_tiles, nprob;
    float alpha, out_scale;
    void* out[2];
    long long ldo;
    int* status;
    GemmQkvEpilogue qkv;
    unsigned long long* tl;
    unsigned long long* trace;  // 64 phase stamps per CTA, as those of gemm_tc.cu
    int batch, out_batch;
    int whole, splits;  // PAIR_SPLIT: tiles worked on as one, the first ones; parts of each of the others
    float* partials;    // [split tile][part][rank][epilogue warp][column][row]
    int* tickets;       // [split tile][rank][epilogue warp], zero
    const GroupTile* grp;
};
#define TFFN_TRACE(slot)                                                       \
    do {                                                                       \
        if (p.trace) p.trace[(size_t)blockIdx.x * 64 + (slot)] = gtime_ns();   \
    } while (0)

// ------------------------------------------------------------------------------------------- cta_group::2 forms
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D (both CTAs' TMEM) (+)= A (128 rows of each CTA) * B (half of the columns from each CTA); one elected lane of a uniform warp
__device__ __forceinline__ void umma2_bf16_elect(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on the barrier at this offset in both CTAs once the MMAs issued so far have completed
__device__ __forceinline__ void umma2_commit_elect(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b16 m;\n\t"
        "mov.b16 m, 3;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(smem_u32(bar))
        : "memory");
}
// TMA loads into this CTA's shared memory whose completion is counted by a barrier of either CTA of the pair
__device__ __forceinline__ void tma2_load_2d_elect(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}" ::"r"(dst),
        "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma2_load_3d_elect(uint32_t dst, const void* tmap, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n\t}" ::"r"(dst),
        "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
        "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
          "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// ------------------------------------------------------------------------------------------- epilogue
// lane = row with 32 consecutive columns -> shared memory, 16-byte pieces swizzled by the row (conflict-free both ways)
__device__ __forceinline__ void park(float* buf, int lane, const float (&v)[32]) {
    __syncwarp();  // the previous piece has been read
#pragma unroll
    for (int j = 0; j < 8; ++j)
        *(float4*)(buf + lane * 32 + 4 * (j ^ (lane & 7))) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    __syncwarp();
}
// row 4 * i + lane / 8, columns 4 * (lane % 8) ..
__device__ __forceinline__ float4 parked(const float* buf, int lane, int i) {
    const int row = 4 * i + (lane >> 3);
    return *(const float4*)(buf + row * 32 + 4 * ((lane & 7) ^ (row & 7)));
}
__device__ __forceinline__ uint2 pack4(float a, float b, float c, float d) {
    return make_uint2((uint32_t)bf16_bits(a) | ((uint32_t)bf16_bits(b) << 16), (uint32_t)bf16_bits(c) | ((uint32_t)bf16_bits(d) << 16));
}

// the parked piece: columns n .. n + 3 (n = column of this lane) of rows t0 + 4 i + lane / 8. vec: all four columns exist and
// can be moved as one; old: the values a residual product is added to
template <int MODE>
__device__ __forceinline__ void store_piece(const PairDev& p, void* out, const float* buf, int lane, int t0, int t_end, int n, const uint2 (&old)[8],
                                            bool vec) {
    if (n >= p.N) return;
    const int row0 = lane >> 3;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (t0 + 4 * i + row0 >= t_end) break;
        float4 v = parked(buf, lane, i);
        const size_t o = (size_t)(t0 + 4 * i + row0) * (size_t)p.ldo + n;
        if (MODE == GEMM_STORE_F32) v = make_float4(v.x * p.out_scale, v.y * p.out_scale, v.z * p.out_scale, v.w * p.out_scale);
        if (MODE == GEMM_RELU2) {
            v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
            v = make_float4(v.x * v.x, v.y * v.y, v.z * v.z, v.w * v.w);
        }
        if (vec) {
            if (MODE == GEMM_RESIDUAL) v = make_float4(v.x + bf16_lo(old[i].x), v.y + bf16_hi(old[i].x), v.z + bf16_lo(old[i].y), v.w + bf16_hi(old[i].y));
            if (MODE == GEMM_STORE_F32) *(float4*)((float*)out + o) = v;
            else *(uint2*)((bf16*)out + o) = pack4(v.x, v.y, v.z, v.w);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n + j >= p.N) continue;
                float f = j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
                bf16* dst = (bf16*)out + o + j;
                if (MODE == GEMM_RESIDUAL) f += __uint_as_float((uint32_t)__ldcg((const unsigned short*)dst) << 16);
                if (MODE == GEMM_STORE_F32) ((float*)out)[o + j] = f;
                else *dst = __float2bfloat16_rn(f);
            }
        }
    }
}

// GEMM_QKV: the position and page of this lane's token (page -1: bad)
__device__ __forceinline__ void qkv_token(const PairDev& p, int t, int t_end, int& pos, int& pg) {
    const GemmQkvEpilogue& e = p.qkv;
    pos = pg = -1;
    if (t >= t_end) return;
    pos = __ldcg(e.tok_pos + t);
    if (pos < 0 || pos >= e.max_pos) {
        pos = -1;
        dev_fail(p.status, DEV_ERR_BOUNDS);
        return;
    }
    const int seq = __ldcg(e.tok_seq + t);
    const int page = __ldcg(e.kv.block_table + (size_t)seq * e.kv.max_pages_per_seq + pos / kPageTokens);
    pg = page >= 0 && page < e.kv.num_pages ? page : -1;
}

// GEMM_QKV, columns c .. c + 31 (a) and their rotary partners (b): round to bf16, add the bias in bf16 (k_add_bias,
// inference/src/model/qwen.cu:223-226), rotate q and k in fp32 (k_rope, qwen.cu:232-244); q stays fp32, k and v go to the
// token's page as bf16 (qwen.cu:339-346)
__device__ __forceinline__ void qkv_pair(const PairDev& p, float* buf, int lane, int t0, int t_end, int n, int pos, int pg, float (&a)[32], float (&b)[32]) {
    const GemmQkvEpilogue& e = p.qkv;
    const int hd = e.kv.hd, half = hd >> 1, nq = e.nh * hd, nk = e.kv.nkv * hd;
    const int kind = n < nq ? 0 : n < nq + nk ? 1 : 2;
    const bool biased = e.bias != nullptr;
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
        uint32_t ba = 0, bb = 0;
        if (biased) {
            ba = *(const uint32_t*)(e.bias + n + j);
            bb = *(const uint32_t*)(e.bias + n + half + j);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            a[j + k] = bf16_round(a[j + k]);
            b[j + k] = bf16_round(b[j + k]);
            if (biased) {
                a[j + k] = bf16_round(a[j + k] + (k ? bf16_hi(ba) : bf16_lo(ba)));
                b[j + k] = bf16_round(b[j + k] + (k ? bf16_hi(bb) : bf16_lo(bb)));
            }
        }
    }
    if (kind != 2 && pos >= 0) {
        const size_t at = (size_t)pos * half + n % hd;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 cs = *(const float4*)(e.rope_cos + at + j), sn = *(const float4*)(e.rope_sin + at + j);
            const float c4[4] = {cs.x, cs.y, cs.z, cs.w}, s4[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float u = a[j + k], v = b[j + k];
                a[j + k] = u * c4[k] - v * s4[k];
                b[j + k] = u * s4[k] + v * c4[k];
            }
        }
    }
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        if (part == 0) park(buf, lane, a);
        else park(buf, lane, b);
        const int col = n + part * half + 4 * (lane & 7);
        if (kind == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int t = t0 + 4 * i + (lane >> 3);
                if (t < t_end) *(float4*)(e.q_out + (size_t)t * nq + col) = parked(buf, lane, i);
            }
            continue;
        }
        const int head = (col - nq - (kind == 2 ? nk : 0)) / hd;
        bf16* pool = (kind == 1 ? e.kv.k_pool : e.kv.v_pool) + (size_t)e.layer * e.kv.layer_stride + (size_t)head * kPageTokens * hd + col % hd;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = 4 * i + (lane >> 3);
            const int ps = __shfl_sync(0xffffffffu, pos, row), page = __shfl_sync(0xffffffffu, pg, row);
            if (t0 + row >= t_end || ps < 0) continue;
            if (page < 0) {
                dev_fail(p.status, DEV_ERR_BOUNDS);
                continue;
            }
            const float4 v = parked(buf, lane, i);
            *(uint2*)(pool + ((size_t)page * e.kv.nkv * kPageTokens + ps % kPageTokens) * hd) = pack4(v.x, v.y, v.z, v.w);
        }
    }
}

// a wait whose outcome is the same in every lane (the loops around it elect lanes and must stay uniform)
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int* status, int code) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, status, code));
}

// What a launch's tiles are: tiles of one or two problems, of a batch or of groups; of several layers (GemmCall::layers: a problem is a
// layer, tmW is 3-D: column, layer, row); with the last ones in parts. The issuing loops of the first kind carry none of what the others need: a test per k-block there cost a
// prompt's products 2 to 3 %.
enum PairKind { PAIR_TILES, PAIR_LAYERS, PAIR_SPLIT };
template <int BN, int MODE, int KIND>
__global__ void __launch_bounds__(kPairThreads, 1) k_gemm_pair(const __grid_constant__ PairDev p) {
    using Cfg = PairCfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* epi = smem + Cfg::STAGES * Cfg::STAGE_BYTES;
    uint64_t* full = (uint64_t*)(epi + Cfg::EPI_BYTES);
    uint64_t* empty = full + Cfg::STAGES;
    uint64_t* acc_full = empty + Cfg::STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    int* used_slot = (int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    if (threadIdx.x == 0) {
        TFFN_TRACE(0);
        tl_mark(p.tl, 0);
        for (int s = 0; s < Cfg::STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * kEpiWarps);
        }
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc2(tmem_slot, Cfg::TMEM_COLS);
    int m_tiles = p.m_tiles;
    if (p.grp) {  // an earlier kernel wrote the table; its unused entries are at the end
        pdl_wait();
        if (warp == 0) {
            if (lane == 0) {
                TFFN_TRACE(2);
                tl_mark(p.tl, 1);
            }
            int used = 0;
            for (int i = lane; i < p.m_tiles; i += 32) used += __ldcg(&p.grp[i].group) >= 0 ? 1 : 0;
            for (int o = 16; o > 0; o >>= 1) used += __shfl_xor_sync(0xffffffffu, used, o);
            if (lane == 0) *used_slot = used;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // barriers and TMEM of both CTAs are ready
    tc_fence_after();
    if (p.grp) m_tiles = *used_slot;
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    const int tiles = m_tiles * p.n_tiles * p.nprob, stride = (int)gridDim.x >> 1, first = (int)blockIdx.x >> 1;
    const int total_kb = p.kblocks[0] + p.kblocks[1];
    constexpr bool halves = MODE == GEMM_SWIGLU;
    const bool dual = p.kblocks[1] > 0;
    constexpr int tile_n = halves ? BN / 2 : BN;
    struct Tile {
        int m, n0, prob, t0, t_end, w_row0;
        int kb0, kb1;       // k-blocks of this unit
        int split, part;    // number of the split tile (-1: a whole one), part of it
    };
    constexpr bool SPLIT = KIND == PAIR_SPLIT, LAYERED = KIND == PAIR_LAYERS;
    // the u-th tile, or part of one, of this pair (false: there are no more)
    auto tile_at = [&](int u, Tile& x) {
        int i = first + u * stride;
        x.kb0 = 0;
        x.kb1 = total_kb;
        x.split = -1;
        x.part = 0;
        if (SPLIT && i >= p.whole) {
            x.split = (i - p.whole) / p.splits;
            x.part = (i - p.whole) % p.splits;
            x.kb0 = (int)((long long)x.part * total_kb / p.splits);
            x.kb1 = (int)((long long)(x.part + 1) * total_kb / p.splits);
            i = p.whole + x.split;
        }
        if (i >= tiles) return false;
        x.m = i % m_tiles;
        const int r = i / m_tiles;
        x.n0 = (r % p.n_tiles) * tile_n;
        x.prob = r / p.n_tiles;
        x.t0 = x.m * kPairTokens;
        x.t_end = p.T;
        x.w_row0 = x.n0;
        if (p.grp) {
            const int4 g = __ldcg((const int4*)(p.grp + x.m));
            x.t0 = g.y;
            x.t_end = min(g.z, g.y + kPairTokens);
            x.w_row0 = g.x * p.N + x.n0;
        } else if (p.batch > 1) {
            x.w_row0 = x.prob * p.N + x.n0;
        }
        return true;
    };

    // The two issuing warps pace the pipeline (a k-block's products take 0.13 to 0.27 us), so their loops carry stage, phase
    // and addresses along instead of computing them. Every lane runs them (uniform), one is elected per instruction.
    if (warp == 0) {
        const uint32_t a_0 = smem_u32(smem), full_0 = smem_u32(full), lead_0 = map_shared_rank(full_0, 0);
        int s = 0, issued = 0;
        uint32_t ph = 1;  // a fresh barrier passes a wait for the phase before its first
        bool waited = p.grp != nullptr, ok = true;
        Tile x;
        for (int u = 0; ok && tile_at(u, x); ++u) {
            const int map = p.batch > 1 || LAYERED ? 0 : x.prob * 2;
            const int t = x.t0 + rank * kHalf + (LAYERED ? x.prob * p.T : 0), wr = halves ? x.w_row0 : x.w_row0 + rank * (BN / 2);
            auto load_w = [&](const CUtensorMap* tm, int k, int st) {
                if (LAYERED) tma2_load_3d_elect(a_0 + st * Cfg::STAGE_BYTES + Cfg::A_BYTES, tm, k, x.prob, wr, lead_0 + st * 8);
                else tma2_load_2d_elect(a_0 + st * Cfg::STAGE_BYTES + Cfg::A_BYTES, tm, k, wr, lead_0 + st * 8);
            };
            auto load_x = [&](const CUtensorMap* tm, int k, int st) {
                if (p.batch > 1) tma2_load_3d_elect(a_0 + st * Cfg::STAGE_BYTES, tm, k, x.prob, t, lead_0 + st * 8);
                else tma2_load_2d_elect(a_0 + st * Cfg::STAGE_BYTES, tm, k, t, lead_0 + st * 8);
            };
            const CUtensorMap* const w_map[2] = {&p.tmW[map + (halves ? rank : 0)], &p.tmW[map + 1]};
            int ahead = 0;
            if (!waited) {  // weights do not depend on the previous kernel: the first ring is requested ahead of the wait
                const int kb0 = SPLIT ? x.kb0 : 0, n = SPLIT ? x.kb1 - x.kb0 : total_kb;
                ahead = n < Cfg::STAGES ? n : Cfg::STAGES;
                for (int st = 0; st < ahead; ++st) {
                    const int kb = kb0 + st, seg = kb >= p.kblocks[0] ? 1 : 0;
                    if (rank == 0) mbar_arrive_expect_tx_elect(full_0 + st * 8, 2 * Cfg::STAGE_BYTES);
                    load_w(w_map[seg], (kb - seg * p.kblocks[0]) * BK, st);
                }
                ahead += kb0;
                if (lane == 0) TFFN_TRACE(1);
                pdl_wait();
                if (lane == 0) {
                    TFFN_TRACE(2);
                    tl_mark(p.tl, 1);
                }
                __syncwarp();
                waited = true;
            }
            int kb = SPLIT ? x.kb0 : 0;
            for (int seg = 0; seg < 2 && ok; ++seg) {
                const CUtensorMap *const tw = w_map[seg], *const tx = &p.tmX[map + seg];
                const int seg0 = seg ? p.kblocks[0] : 0;
                const int k_end = SPLIT ? (min(x.kb1, seg0 + p.kblocks[seg]) - seg0) * BK : p.kblocks[seg] * BK;
                for (int k = SPLIT ? (kb - seg0) * BK : 0; k < k_end; k += BK, ++kb) {
                    if (!(ok = warp_wait(&empty[s], ph, p.status, DEV_ERR_EMPTY_WAIT))) break;
                    if (kb >= ahead) {
                        if (rank == 0) mbar_arrive_expect_tx_elect(full_0 + s * 8, 2 * Cfg::STAGE_BYTES);
                        load_w(tw, k, s);
                    }
                    load_x(tx, k, s);
                    ++issued;
                    if (++s == Cfg::STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
        if (!waited) pdl_wait();
        // the leader's last arrivals land here: leave only after them
        for (int j = 0; j < Cfg::STAGES && ok; ++j) {
            if (issued > j) ok = warp_wait(&empty[(s + Cfg::STAGES - 1 - j) % Cfg::STAGES], j < s ? ph ^ 1 : ph, p.status, DEV_ERR_EMPTY_WAIT);
        }
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr uint32_t idesc = umma_idesc_bf16(kPairTokens, BN);
            const uint64_t a_0 = umma_desc_k128(smem_u32(smem)), b_0 = umma_desc_k128(smem_u32(smem) + Cfg::A_BYTES);
            int s = 0, n = 0;
            uint32_t ph = 0;
            bool ok = true;
            Tile x;
            for (int i = first; ok && (SPLIT ? tile_at(n, x) : i < tiles); i += stride, ++n) {
                const int buf = dual ? 0 : n & 1, use = dual ? n : n >> 1;
                if (!(ok = warp_wait(&acc_empty[buf], (uint32_t)(use & 1) ^ 1u, p.status, DEV_ERR_ACC_WAIT))) break;
                for (int seg = 0; seg < 2 && ok; ++seg) {
                    const uint32_t d = tmem_base + (uint32_t)((dual ? seg : buf) * BN);
                    const int seg0 = seg ? p.kblocks[0] : 0;
                    const int kb_first = SPLIT ? max(x.kb0, seg0) : 0, kb_end = SPLIT ? min(x.kb1, seg0 + p.kblocks[seg]) : p.kblocks[seg];
                    for (int kb = kb_first; kb < kb_end; ++kb) {
                        if (!(ok = warp_wait(&full[s], ph, p.status, DEV_ERR_FULL_WAIT))) break;
                        tc_fence_after();
                        const uint64_t at = (uint64_t)(uint32_t)(s * (Cfg::STAGE_BYTES >> 4));
                        const uint64_t ad = a_0 + at, bd = b_0 + at;
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) umma2_bf16_elect(d, ad + 2 * k, bd + 2 * k, idesc, ((SPLIT ? kb - kb_first : kb) | k) ? 1u : 0u);
                        umma2_commit_elect(&empty[s]);
                        if (++s == Cfg::STAGES) {
                            s = 0;
                            ph ^= 1;
                        }
                    }
                }
                umma2_commit_elect(&acc_full[buf]);
            }
            if (lane == 0) TFFN_TRACE(3);
        }
    } else {
        pdl_wait();
        const int q = warp & 3, part = (warp - 2) >> 2;  // TMEM lane quarter, which half of the columns
        float* buf32 = (float*)(epi + (warp - 2) * 32 * kStageRow);
        int n = 0;
        Tile x;
        for (; tile_at(n, x); ++n) {
            const int buf = dual ? 0 : n & 1, use = dual ? n : n >> 1;
            const int t0 = x.t0 + rank * kHalf + q * 32;
            int pos = -1, pg = -1;
            if (MODE == GEMM_QKV) qkv_token(p, t0 + lane, x.t_end, pos, pg);
            if (!warp_wait(&acc_full[buf], (uint32_t)use & 1u, p.status, DEV_ERR_ACC_WAIT)) break;
            if (threadIdx.x == 64 && n == 0) TFFN_TRACE(4);
            __syncwarp();
            tc_fence_after();
            const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(dual ? 0 : buf * BN);
            if (t0 < x.t_end) {
                if (MODE == GEMM_QKV) {
                    const int hd = p.qkv.kv.hd, half = hd >> 1, per_head = half / 32;
                    for (int pr = part; pr < BN / 64; pr += 2) {
                        const int c = (pr / per_head) * hd + (pr % per_head) * 32;
                        if (x.n0 + c >= p.N) break;
                        float a[32], b[32];
                        tmem_ld32(acc + (uint32_t)c, a);
                        tmem_ld32(acc + (uint32_t)(c + half), b);
                        tc_wait_ld();
                        qkv_pair(p, buf32, lane, t0, x.t_end, x.n0 + c, pos, pg, a, b);
                    }
                } else {
                    const bool one_out = p.batch > 1 || LAYERED;
                    void* out = p.out[one_out ? 0 : x.prob];
                    if (one_out) {
                        const size_t at = (size_t)x.prob * (p.batch > 1 ? (size_t)p.out_batch : (size_t)p.T * (size_t)p.ldo);
                        if (MODE == GEMM_STORE_F32) out = (float*)out + at;
                        else out = (bf16*)out + at;
                    }
                    const int cols = tile_n / 2;  // of this warp
                    // a part's sums: a warp's block of the scratch memory, [column][row]
                    const size_t block = (size_t)cols * 32, slot = (size_t)2 * kEpiWarps * block;
                    float* const sums = SPLIT && x.split >= 0 ? p.partials + (size_t)x.split * p.splits * slot + ((size_t)rank * kEpiWarps + (warp - 2)) * block : nullptr;
                    bool finish = true;
                    if (SPLIT && x.split >= 0) {
                        const bool has0 = x.kb0 < p.kblocks[0], has1 = x.kb1 > p.kblocks[0];
                        float* mine = sums + x.part * slot;
#pragma unroll 1
                        for (int c = 0; c < cols; c += 32) {
                            float v[32];
                            if (dual) {
                                float w[32];
                                tmem_ld32(acc + (uint32_t)(part * cols + c), v);
                                tmem_ld32(acc + (uint32_t)(part * cols + c + BN), w);
                                tc_wait_ld();
#pragma unroll
                                for (int j = 0; j < 32; ++j) v[j] = (has0 ? v[j] : 0.f) + (has1 ? p.alpha * w[j] : 0.f);
                            } else {
                                tmem_ld32(acc + (uint32_t)(part * cols + c), v);
                                tc_wait_ld();
                            }
#pragma unroll
                            for (int j = 0; j < 32; ++j) mine[(c + j) * 32 + lane] = v[j];
                        }
                        __threadfence();
                        __syncwarp();
                        int* ticket = p.tickets + (x.split * 2 + rank) * kEpiWarps + (warp - 2);
                        int before = 0;
                        if (lane == 0) before = atomicAdd(ticket, 1);
                        finish = __shfl_sync(0xffffffffu, before, 0) == p.splits - 1;
                        if (finish) {
                            if (lane == 0) *ticket = 0;
                            __threadfence();
                        }
                    }
#pragma unroll 1
                    for (int c = part * cols; finish && c < (part + 1) * cols; c += 32) {
                        if (x.n0 + c >= p.N) break;
                        const int col = x.n0 + c + 4 * (lane & 7);
                        const bool vec = col + 3 < p.N && ((p.ldo | p.out_batch) & 3) == 0;
                        uint2 old[8];
                        if (MODE == GEMM_RESIDUAL && vec) {
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const int t = t0 + 4 * k + (lane >> 3);
                                if (t < x.t_end) old[k] = __ldcg((const uint2*)((const bf16*)out + (size_t)t * (size_t)p.ldo + col));
                            }
                        }
                        float v[32];
                        if (SPLIT && x.split >= 0) {
                            const float* from = sums + (size_t)(c - part * cols) * 32 + lane;
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = __ldcg(from + j * 32);
                            for (int z = 1; z < p.splits; ++z) {
                                from += slot;
#pragma unroll
                                for (int j = 0; j < 32; ++j) v[j] += __ldcg(from + j * 32);
                            }
                            park(buf32, lane, v);
                            store_piece<MODE>(p, out, buf32, lane, t0, x.t_end, col, old, vec);
                            continue;
                        }
                        tmem_ld32(acc + (uint32_t)c, v);
                        if (halves || dual) {
                            float w[32];
                            tmem_ld32(acc + (uint32_t)(c + (halves ? BN / 2 : BN)), w);
                            tc_wait_ld();
                            if (halves) {
#pragma unroll
                                for (int j = 0; j < 32; ++j) v[j] = silu_mul_bf16(v[j], w[j]);
                            } else {
#pragma unroll
                                for (int j = 0; j < 32; ++j) v[j] = v[j] + p.alpha * w[j];
                            }
                        } else {
                            tc_wait_ld();
                        }
                        park(buf32, lane, v);
                        store_piece<MODE>(p, out, buf32, lane, t0, x.t_end, col, old, vec);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(map_shared_rank(smem_u32(&acc_empty[buf]), 0));
        }
        if (threadIdx.x == 64) TFFN_TRACE(5);
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // no barrier or operand of the peer is needed any more
    if (threadIdx.x == 64) {
        TFFN_TRACE(8);
        tl_mark(p.tl, 2);
    }
    __syncwarp();
    if (warp == 1) tmem_dealloc2(tmem_base, Cfg::TMEM_COLS);
}

template <int BN>
int launch_pair(const GemmCall& c, const GemmWorkspace& ws, cudaStream_t stream) {
    PairDev p;
    memset(&p, 0, sizeof p);
    const bool halves = c.mode == GEMM_SWIGLU, batched = c.batch > 1, layered = c.layers > 1;
    if (layered && ((c.mode != GEMM_SWIGLU && c.mode != GEMM_STORE_F32) || batched || c.grp || c.out2 || c.w_layer % 8 || c.w_layer >> 32 || (!halves && c.op[1].K > 0)))
        return (int)cudaErrorInvalidValue;
    const int maps = c.out2 ? 2 : 1;
    for (int pr = 0; pr < maps; ++pr)
        for (int i = 0; i < 2; ++i) {
            const GemmOperand& o = pr ? c.op2[i] : c.op[i];
            if (pr == 0) p.kblocks[i] = o.K > 0 ? (o.K + BK - 1) / BK : 0;
            if (o.K <= 0) continue;
            const uint64_t w_rows = (uint64_t)c.N * (c.grp ? c.grp_count : batched ? c.batch : 1);
            if (!make_tmap_2d(ws.tmaps, &p.tmW[pr * 2 + i], o.W, w_rows, (uint64_t)o.K, (uint64_t)o.ldw, BN / 2, layered ? (uint32_t)c.layers : 1u,
                              (uint32_t)c.w_layer))
                return -1000;
            if (!make_tmap_2d(ws.tmaps, &p.tmX[pr * 2 + i], o.X, (uint64_t)(c.x_rows_alloc > c.T ? c.x_rows_alloc : c.T), (uint64_t)o.K,
                              (uint64_t)o.ldx, kHalf, batched ? (uint32_t)c.batch : 1u, (uint32_t)c.x_batch))
                return -1000;
        }
    if (halves) p.kblocks[1] = 0;  // gate and up are the two halves of one accumulator
    for (int i = 1; i < 4; ++i)  // keep unused maps valid
        if (i >= maps * 2 || (p.kblocks[i & 1] == 0 && !halves)) {
            p.tmW[i] = p.tmW[0];
            p.tmX[i] = p.tmX[0];
        }
    const int tile_n = halves ? BN / 2 : BN;
    p.batch = batched ? c.batch : 1;
    p.out_batch = batched ? c.out_batch : 0;
    p.nprob = batched ? c.batch : layered ? c.layers : maps;
    p.N = c.N;
    p.T = c.T;
    p.m_tiles = c.grp ? c.grp_tiles : (c.T + kPairTokens - 1) / kPairTokens;
    p.n_tiles = (c.N + tile_n - 1) / tile_n;
    p.alpha = c.alpha;
    p.out_scale = c.out_scale == 0.f ? 1.f : c.out_scale;
    p.out[0] = c.out;
    p.out[1] = c.out2 ? c.out2 : c.out;
    p.ldo = c.ldo;
    p.status = ws.status;
    p.tl = c.tl;
    p.grp = c.grp;
    if (c.mode == GEMM_QKV) p.qkv = *c.qkv;
    const long long tiles = (long long)p.m_tiles * p.n_tiles * p.nprob;
    int pairs = (int)(tiles < ws.num_sms / 2 ? tiles : ws.num_sms / 2);
    bool split = false;
    if (!c.grp && !layered && ws.partials && (c.mode == GEMM_STORE_F32 || c.mode == GEMM_STORE_BF16 || c.mode == GEMM_RESIDUAL)) {
        const PairSplit s = pair_split(tiles, p.kblocks[0] + p.kblocks[1], BN, ws.num_sms);
        split = s.splits > 1 && (size_t)s.tail * s.splits * kPairTokens * BN <= ws.partial_floats && (long long)s.tail * 2 * kEpiWarps <= ws.num_counters;
        if (split) {
            p.whole = (int)(tiles - s.tail);
            p.splits = s.splits;
            p.partials = ws.partials;
            p.tickets = ws.counters;
            const long long units = p.whole + (long long)s.tail * s.splits;
            pairs = (int)(units < ws.num_sms / 2 ? units : ws.num_sms / 2);
        }
    }
    p.trace = 2 * pairs <= c.trace_ctas ? c.trace : nullptr;
    auto go = [&](auto kern) { return (int)launch_k_cluster(kern, dim3(2 * pairs), dim3(kPairThreads), dim3(2, 1, 1), PairCfg<BN>::SMEM, stream, c.pdl, p); };
    if (layered) return halves ? go(k_gemm_pair<BN, GEMM_SWIGLU, PAIR_LAYERS>) : go(k_gemm_pair<BN, GEMM_STORE_F32, PAIR_LAYERS>);
    switch (c.mode) {
        case GEMM_STORE_F32: return split ? go(k_gemm_pair<BN, GEMM_STORE_F32, PAIR_SPLIT>) : go(k_gemm_pair<BN, GEMM_STORE_F32, PAIR_TILES>);
        case GEMM_STORE_BF16: return split ? go(k_gemm_pair<BN, GEMM_STORE_BF16, PAIR_SPLIT>) : go(k_gemm_pair<BN, GEMM_STORE_BF16, PAIR_TILES>);
        case GEMM_RESIDUAL: return split ? go(k_gemm_pair<BN, GEMM_RESIDUAL, PAIR_SPLIT>) : go(k_gemm_pair<BN, GEMM_RESIDUAL, PAIR_TILES>);
        case GEMM_SWIGLU: return go(k_gemm_pair<BN, GEMM_SWIGLU, PAIR_TILES>);
        case GEMM_RELU2: return go(k_gemm_pair<BN, GEMM_RELU2, PAIR_TILES>);
        case GEMM_QKV: return go(k_gemm_pair<BN, GEMM_QKV, PAIR_TILES>);
    }
    return (int)cudaErrorInvalidValue;
}

template <int BN>
cudaError_t prepare_pair() {
    cudaError_t e = cudaSuccess;
    auto prep = [&](auto kern) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<BN>::SMEM);
        if (e == cudaSuccess) e = prefer_max_shared(kern);
    };
    prep(k_gemm_pair<BN, GEMM_STORE_F32, PAIR_TILES>);
    prep(k_gemm_pair<BN, GEMM_STORE_BF16, PAIR_TILES>);
    prep(k_gemm_pair<BN, GEMM_RESIDUAL, PAIR_TILES>);
    prep(k_gemm_pair<BN, GEMM_SWIGLU, PAIR_TILES>);
    prep(k_gemm_pair<BN, GEMM_RELU2, PAIR_TILES>);
    prep(k_gemm_pair<BN, GEMM_QKV, PAIR_TILES>);
    prep(k_gemm_pair<BN, GEMM_SWIGLU, PAIR_LAYERS>);
    prep(k_gemm_pair<BN, GEMM_STORE_F32, PAIR_LAYERS>);
    prep(k_gemm_pair<BN, GEMM_STORE_F32, PAIR_SPLIT>);
    prep(k_gemm_pair<BN, GEMM_STORE_BF16, PAIR_SPLIT>);
    prep(k_gemm_pair<BN, GEMM_RESIDUAL, PAIR_SPLIT>);
    return e;
}

}  // namespace

// A k-block costs a pair 0.34 us with 128 weight rows and 0.42 with 256 (0.34 while it has the chip to itself), a tile about 1 us
// around them; whole waves of 74 pairs count. The tiles of the last wave can be split along K, if it is at most half full: a part's
// sums cost about 3 us to leave behind and the last part 1.6 us for each of them to add up (4 096 tokens, K 17920 of two operand
// pairs, N 1536: 96 tiles, the last 22 in three parts, 235 -> 179 us). Shares of equal length for all pairs, across tile borders, were
// slower than whole tiles (262): the pairs no longer read the same columns at about the same time.
PairSplit pair_split(long long tiles, int kb, int bn, int num_sms) {
    const int pairs = num_sms / 2, tail = (int)(tiles % pairs);
    const double us = bn == 128 || tiles < pairs ? 0.34 : 0.42;
    const double whole = (double)((tiles + pairs - 1) / pairs) * (kb * us + 1.0);
    PairSplit best{tail, 1, whole, whole};
    for (int s = 2; tail > 0 && s * tail <= pairs && s <= 8 && kb >= 8 * s; ++s) {
        const double cost = (double)(tiles / pairs) * (kb * us + 1.0) + (double)kb / s * us + 1.0 + 3.0 + 1.6 * s;
        if (cost < best.us) best = PairSplit{tail, s, cost, whole};
    }
    return best;
}

int gemm_pair_prepare() {
    const cudaError_t e = prepare_pair<128>();
    return (int)(e == cudaSuccess ? prepare_pair<256>() : e);
}

int launch_gemm_pair(const GemmCall& c, const GemmWorkspace& ws, cudaStream_t stream, int bn) {
    return bn == 128 ? launch_pair<128>(c, ws, stream) : launch_pair<256>(c, ws, stream);
}

}  // namespace tffn
