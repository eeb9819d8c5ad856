// Tensor-core GEMM of the batched path (prefill and decode with more than one token):
//     out[t, n] = epilogue( sum_k X[t,k] * W[n,k] )
// "swap-AB": the weight rows fill the MMA's M = 128 dimension and the tokens are the MMA's N
// (16..256), so a decode step with a few dozen tokens wastes no tensor-core rows and each
// weight byte is streamed from HBM exactly once per token tile.
//
// One CTA = one 128-row x BN-token output tile (optionally one K split of it), 6 warps:
//   warp 0   TMA producer: 128x64 weight box + BNx64 activation box per stage, 128-byte swizzle
//   warp 1   allocates TMEM, issues tcgen05.mma (one elected lane), commits stages back to the producer
//   warps 2-5 epilogue: tcgen05.ld the fp32 accumulators (lane = weight row, column = token),
//            apply the epilogue and store. With split-K the splits of a tile are one thread-block
//            cluster: partial tiles stay in shared memory and are summed across the cluster over
//            distributed shared memory in rank order, so the result does not depend on
//            scheduling and no partial sum touches HBM.
// Two operand pairs can be accumulated into two TMEM regions (gate|up for the SwiGLU epilogue,
// base|expert for the down projection) and are combined in fp32 in the epilogue.
// It replaces the reference's cublasGemmEx wrappers (inference/src/backend/cuda_ops.cu:18-43)
// and the element-wise kernels around them (silu_mul :58-69, add :152-157,
// k_add_fp32_to_bf16 inference/src/model/qwen.cu:282-285).
#include "kernels.h"
#include "ptx.cuh"
#include "launch.h"
#include <cstdio>
#include <cstring>
#include <functional>
#include <mutex>
#include <unordered_map>

namespace tffn {

namespace {

constexpr int BM = 128;  // weight rows per tile
constexpr int BK = 64;   // K elements per stage (128 bytes of bf16)
constexpr int kGemmThreads = 192;
constexpr int kMaxSmem = 227 * 1024;  // dynamic shared memory a CTA may claim on sm_100
constexpr int kMaxSplits = 16;  // cluster size; above 8 needs the non-portable opt-in (gemm_prepare)

struct GemmDev {
    CUtensorMap tmW[4];  // [problem * 2 + operand pair]
    CUtensorMap tmX[4];
    int kblocks[2];
    int N, T, splits, mode, t_tiles, stages;
    int tile_n;          // output indices per tile: 128, or 64 for GEMM_SWIGLU (64 gate rows + 64 up rows per tile)
    int tiles_1;         // with a product beside it (launch_gemm_beside): tiles blockIdx.x >= tiles_1 are its, a GEMM_SWIGLU's, else 0
    int N_2;
    long long ldo_2;
    float alpha, out_scale;
    void* out[2];        // per problem
    long long ldo;
    int* status;
    GemmQkvEpilogue qkv;  // GEMM_QKV only
    unsigned long long* trace;  // optional: 64 timestamps (ns) per CTA, see GemmCall::trace
    unsigned long long* tl;     // optional: step timeline of this launch
    int batch, out_batch;       // batched launch (GemmCall::batch): X is a 3-D map (column, problem, row)
    const int* bins;            // grouped launch over bins: GemmCall::bin_counts
    int bin, bin_groups, bin_ahead;
    const GroupTile* grp;       // grouped launch: one entry per token tile (blockIdx.y), see GemmCall::grp
    const bf16* norm_w;         // GemmCall::norm_w and what follows
    bf16* norm_out;
    float* norm_ssq;
    const float* rms_ssq;
    int rms_tiles, rms_n;
    float rms_eps;
    float* amax_val;            // GEMM_STORE_F32: per (token, tile) maximum and its index, or nullptr
    int* amax_idx;
};

#define TFFN_TRACE(slot)                                                                                            \
    do {                                                                                                            \
        if (p.trace) p.trace[(size_t)((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * 64 + (slot)] = gtime_ns(); \
    } while (0)

// what a CTA writes: the launch's product, or the one beside it
struct OutView {
    int N, mode;
    long long ldo;
};

template <int BN>
struct GemmCfg {
    static constexpr int A_BYTES = BM * BK * 2;
    static constexpr int B_BYTES = BN * BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    // The ring depth is chosen at launch. A grid of at most one CTA per SM gets the deepest ring
    // that fits (about 190 KB in flight per SM: the HBM latency under load is several microseconds,
    // so the bytes in flight bound the stream); a larger grid of decode-sized tiles gets 4 stages
    // so that two CTAs share an SM.
    static constexpr int MAX_STAGES = (196 * 1024 / STAGE_BYTES) > 10 ? 10 : (196 * 1024 / STAGE_BYTES);
    static constexpr int SHARED_STAGES = (BN <= 64) ? 4 : MAX_STAGES;
    // the epilogue parks one fp32 plane [BN][128] in the (by then idle) stage memory
    static_assert(BN * BM * 4 + BN * 8 <= SHARED_STAGES * STAGE_BYTES, "plane (+ per-token maxima) must fit the smallest ring");
    static constexpr int smem_bytes(int stages) { return stages * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/ + BN * 4 /*factors of the rows*/; }
    static constexpr int TMEM_COLS = (2 * BN < 32) ? 32 : 2 * BN;  // two accumulators, power of two
};

// ---------------------------------------------------------------------------------------------
// Finalisation of 4 consecutive rows (n .. n+3) of one token column: the epilogues of all modes.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint2 pack_bf16x4(float a, float b, float c, float d) {
    return make_uint2((uint32_t)bf16_bits(a) | ((uint32_t)bf16_bits(b) << 16),
                      (uint32_t)bf16_bits(c) | ((uint32_t)bf16_bits(d) << 16));
}

// What a finalisation reads from global memory besides the accumulators. None of it depends on this
// kernel's own arithmetic, so with split-K (where a warp finishes at most two columns) the epilogue warps
// fetch it while the MMAs still run, instead of paying two or three dependent L2 round trips per column
// after the reduction.
struct FinalizePre {
    bool valid;      // the fields below were fetched
    uint2 residual;  // GEMM_RESIDUAL: the four old bf16 values
    int pos, pg;     // GEMM_QKV: position and page of the token (pg = -1: bad page or position)
    float4 cs, sn;   // GEMM_QKV: the RoPE table entries of this lane's rows
};

// GEMM_QKV: position of token t, its page, and the RoPE entries for rows n .. n+3
__device__ __forceinline__ void prefetch_qkv(const GemmDev& p, int n, int t, FinalizePre& f) {
    const GemmQkvEpilogue& e = p.qkv;
    const int hd = e.kv.hd, half = hd >> 1;
    f.valid = true;
    f.pos = __ldcg(e.tok_pos + t);
    f.pg = -1;
    f.cs = f.sn = make_float4(0.f, 0.f, 0.f, 0.f);
    if (f.pos < 0 || f.pos >= e.max_pos || n >= p.N) return;
    const int seq = __ldcg(e.tok_seq + t);
    const int pg = __ldcg(e.kv.block_table + (size_t)seq * e.kv.max_pages_per_seq + f.pos / kPageTokens);
    f.pg = (pg >= 0 && pg < e.kv.num_pages) ? pg : -1;
    if (n < (e.nh + e.kv.nkv) * hd) {  // q and k rows are rotated
        const int i = (n % hd) % half;
        f.cs = *(const float4*)(e.rope_cos + (size_t)f.pos * half + i);
        f.sn = *(const float4*)(e.rope_sin + (size_t)f.pos * half + i);
    }
}

// GEMM_QKV: round to bf16, add the bias in bf16 (k_add_bias, inference/src/model/qwen.cu:223-226),
// rotate q and k in fp32 at the token's position (k_rope, qwen.cu:232-244) — the RoPE partner rows
// (i <-> i + hd/2) sit hd/8 lanes away in the same warp, because a warp holds all 128 rows of a
// column — keep q in fp32, write k (rounded after the rotation) and v as bf16 into the
// sequence's page (qwen.cu:339-346). Every lane of the warp must call it (shuffles).
__device__ __forceinline__ void finalize_qkv(const GemmDev& p, int n, int t, float4 v, FinalizePre f) {
    const GemmQkvEpilogue& e = p.qkv;
    const int hd = e.kv.hd, half = hd >> 1;
    const int d = n % hd;  // tiles start at multiples of 128 and hd divides 128
    const bool in_range = n < p.N;
    float x[4] = {bf16_round(v.x), bf16_round(v.y), bf16_round(v.z), bf16_round(v.w)};
    if (e.bias && in_range) {
        const uint2 b = *(const uint2*)(e.bias + n);
        x[0] = bf16_round(x[0] + bf16_lo(b.x));
        x[1] = bf16_round(x[1] + bf16_hi(b.x));
        x[2] = bf16_round(x[2] + bf16_lo(b.y));
        x[3] = bf16_round(x[3] + bf16_hi(b.y));
    }
    float xp[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) xp[j] = __shfl_xor_sync(0xffffffffu, x[j], hd >> 3);
    if (!in_range) return;
    if (!f.valid) prefetch_qkv(p, n, t, f);
    if (f.pos < 0 || f.pos >= e.max_pos) {
        dev_fail(p.status, DEV_ERR_BOUNDS);
        return;
    }
    const int nq = e.nh * hd, nk = e.kv.nkv * hd;
    const int kind = n < nq ? 0 : (n < nq + nk ? 1 : 2);
    float o[4] = {x[0], x[1], x[2], x[3]};
    if (kind != 2) {
        const float cs[4] = {f.cs.x, f.cs.y, f.cs.z, f.cs.w}, sn[4] = {f.sn.x, f.sn.y, f.sn.z, f.sn.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = d < half ? x[j] * cs[j] - xp[j] * sn[j] : xp[j] * sn[j] + x[j] * cs[j];
    }
    if (kind == 0) {
        *(float4*)(e.q_out + (size_t)t * nq + n) = make_float4(o[0], o[1], o[2], o[3]);
        return;
    }
    if (f.pg < 0) {
        dev_fail(p.status, DEV_ERR_BOUNDS);
        return;
    }
    const int head = kind == 1 ? (n - nq) / hd : (n - nq - nk) / hd;
    bf16* pool = (kind == 1 ? e.kv.k_pool : e.kv.v_pool) + (size_t)e.layer * e.kv.layer_stride;
    bf16* dst = pool + (((size_t)f.pg * e.kv.nkv + head) * kPageTokens + f.pos % kPageTokens) * hd + d;
    *(uint2*)dst = pack_bf16x4(o[0], o[1], o[2], o[3]);
}

__device__ __forceinline__ bool plain_is_vector(const GemmDev& p, const OutView& w, int n) { return (n + 3 < w.N) && (((w.ldo | p.out_batch) & 3) == 0); }

// GEMM_RESIDUAL: the old values of rows n .. n+3 of token t (read through L2)
__device__ __forceinline__ void prefetch_residual(const GemmDev& p, const OutView& w, const void* out, int n, int t, FinalizePre& f) {
    f.valid = n < w.N && plain_is_vector(p, w, n);
    if (f.valid) f.residual = __ldcg((const uint2*)((const bf16*)out + (size_t)t * (size_t)w.ldo + n));
}

// GEMM_RESIDUAL with norm_w: h = bf16(float(h) + sum), the normed row up to its factor, and this tile's share of the factor. The
// whole warp calls it.
__device__ __forceinline__ void finalize_residual_norm(const GemmDev& p, void* out, int n, int t, float4 v, const FinalizePre& pre, uint2 nw, int lane) {
    const size_t o = (size_t)t * (size_t)p.ldo + n;
    bf16* h = (bf16*)out;
    const uint2 old = pre.valid ? pre.residual : __ldcg((const uint2*)(h + o));
    const uint2 now = pack_bf16x4(bf16_lo(old.x) + v.x, bf16_hi(old.x) + v.y, bf16_lo(old.y) + v.z, bf16_hi(old.y) + v.w);
    *(uint2*)(h + o) = now;
    const float a = bf16_lo(now.x), b = bf16_hi(now.x), c = bf16_lo(now.y), d = bf16_hi(now.y);
    *(uint2*)(p.norm_out + o) = pack_bf16x4(a * bf16_lo(nw.x), b * bf16_hi(nw.x), c * bf16_lo(nw.y), d * bf16_hi(nw.y));
    float ss = (a * a + b * b) + (c * c + d * d);
    ss = warp_sum(ss);
    if (lane == 0) p.norm_ssq[(size_t)t * gridDim.x + blockIdx.x] = ss;
}

// STORE / RESIDUAL / SWIGLU (the SwiGLU value was formed before the call)
__device__ __forceinline__ void finalize_plain(const GemmDev& p, const OutView& w, void* out, int n, int t, float4 v, FinalizePre pre) {
    if (n >= w.N) return;
    const size_t o = (size_t)t * (size_t)w.ldo + n;
    const bool vec = plain_is_vector(p, w, n);
    const float f[4] = {v.x, v.y, v.z, v.w};
    switch (w.mode) {
        case GEMM_STORE_F32:
            if (!out) break;  // only the fused arg-max was asked for
            if (vec) {
                *(float4*)((float*)out + o) = make_float4(p.out_scale * v.x, p.out_scale * v.y, p.out_scale * v.z, p.out_scale * v.w);
            } else {
                for (int j = 0; j < 4 && n + j < w.N; ++j) ((float*)out)[o + j] = p.out_scale * f[j];
            }
            break;
        case GEMM_RESIDUAL: {
            // h = bf16(float(h) + sum) (k_add_fp32_to_bf16, qwen.cu:282-285); h is read through L2
            bf16* h = (bf16*)out;
            if (vec) {
                const uint2 old = pre.valid ? pre.residual : __ldcg((const uint2*)(h + o));
                *(uint2*)(h + o) = pack_bf16x4(bf16_lo(old.x) + f[0], bf16_hi(old.x) + f[1], bf16_lo(old.y) + f[2],
                                               bf16_hi(old.y) + f[3]);
            } else {
                for (int j = 0; j < 4 && n + j < w.N; ++j) {
                    const float old = __uint_as_float((uint32_t)__ldcg((const unsigned short*)(h + o + j)) << 16);
                    h[o + j] = __float2bfloat16_rn(old + f[j]);
                }
            }
            break;
        }
        default:  // GEMM_STORE_BF16, GEMM_SWIGLU, GEMM_RELU2
            if (w.mode == GEMM_RELU2) {
                float r[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float a = fmaxf(f[j], 0.f);
                    r[j] = a * a;
                }
                if (vec) {
                    *(uint2*)((bf16*)out + o) = pack_bf16x4(r[0], r[1], r[2], r[3]);
                } else {
                    for (int j = 0; j < 4 && n + j < w.N; ++j) ((bf16*)out)[o + j] = __float2bfloat16_rn(r[j]);
                }
                break;
            }
            if (vec) {
                *(uint2*)((bf16*)out + o) = pack_bf16x4(f[0], f[1], f[2], f[3]);
            } else {
                for (int j = 0; j < 4 && n + j < w.N; ++j) ((bf16*)out)[o + j] = __float2bfloat16_rn(f[j]);
            }
            break;
    }
}

// Fused greedy pick (GEMM_STORE_F32): all 32 lanes of the warp that finished tile column t hold rows
// n .. n+3 of it; the tile's maximum and its index (lowest index among equal maxima: sample(),
// inference/src/main.cpp:45-51) go to amax_val / amax_idx [t][tile].
__device__ __forceinline__ void warp_amax(const GemmDev& p, int n, float4 v, float& best, int& bi) {
    const float f[4] = {v.x, v.y, v.z, v.w};
    best = -INFINITY;
    bi = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (n + j < p.N && (f[j] > best || (f[j] == best && n + j < bi))) { best = f[j]; bi = n + j; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
}
__device__ __forceinline__ void publish_amax(const GemmDev& p, int n, int t, float4 v, int lane) {
    if (!p.amax_val) return;
    float best;
    int bi;
    warp_amax(p, n, v, best, bi);
    if (lane == 0) {
        p.amax_val[(size_t)t * gridDim.x + blockIdx.x] = best;
        p.amax_idx[(size_t)t * gridDim.x + blockIdx.x] = bi;
    }
}
__device__ __forceinline__ float4 ld_shared_cluster_v4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void add4(float4& a, const float4& b) {
    a.x += b.x;
    a.y += b.y;
    a.z += b.z;
    a.w += b.w;
}

// What a launch can be beyond tiles of one or two problems, of a batch or of groups: TC_FOLD passes a norm on or takes one
// (GemmCall::norm_w, rms_ssq), TC_MIXED finds its rows in bins or has another product's tiles behind its own. The tests for the latter on the
// way to the first load cost every launch 0.2 us (a step of 97 products 687 -> 706 us), but the steps that have such launches run all of
// theirs as one kind (GemmCall::mixed): a kernel of its own for some of them was not in the SMs' instruction caches when its turn came
// (16 sequences, parallel blocks, first products 6.5 -> 7.8 us, step 322 -> 342).
enum TcKind { TC_PLAIN, TC_FOLD, TC_MIXED };
template <int BN, int KIND>
__global__ void __launch_bounds__(kGemmThreads, (BN <= 64) ? 2 : 1) k_gemm_tc(const __grid_constant__ GemmDev p) {
    using Cfg = GemmCfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int STAGES = p.stages;
    uint64_t* full = (uint64_t*)(smem + STAGES * Cfg::STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
    int* tile_end = (int*)(tmem_slot + 1);  // bins: for the warps that do not read the count themselves
    float* row_factor = (float*)(smem + STAGES * Cfg::STAGE_BYTES + 256);  // per token of the tile, with rms_ssq

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    int prob = blockIdx.y / p.t_tiles;  // independent problems (base / expert gate-up) share a launch
    constexpr bool FOLD = KIND == TC_FOLD;
    const bool bins = KIND == TC_MIXED && p.bins, beside = KIND == TC_MIXED && p.tiles_1 > 0 && (int)blockIdx.x >= p.tiles_1;
    const OutView view = beside ? OutView{p.N_2, GEMM_SWIGLU, p.ldo_2} : OutView{p.N, p.mode, p.ldo};
    const int n0 = beside ? ((int)blockIdx.x - p.tiles_1) * (BM / 2) : (int)blockIdx.x * p.tile_n;
    int t0 = (blockIdx.y % p.t_tiles) * BN, t_end = p.T, w_row0 = n0;
    if (p.grp) {
        // grouped launch: which group's weights and which rows this tile covers was written by an earlier kernel, so
        // nothing can be requested ahead of the wait; unused tiles (the grid is sized for the worst case) leave
        // together, all CTAs of a cluster alike
        pdl_wait();
        const int4 g = __ldcg((const int4*)(p.grp + blockIdx.y));
        if (g.x < 0) return;
        t0 = g.y;
        t_end = min(g.z, g.y + BN);
        w_row0 = g.x * p.N + n0;
    }
    // bins: which weights this CTA needs does not depend on the counts, only how many rows there are
    // (the groups' first tiles come first: the others are mostly empty and would hold their places)
    const int group = bins ? (int)blockIdx.y % p.bin_groups : 0, bin0 = group * p.bin;
    auto bin_end = [&] { return min(bin0 + min(p.bin, __ldcg(p.bins + group)), t0 + BN); };
    bool count_later = false;
    if (bins) {
        t0 = bin0 + (int)blockIdx.y / p.bin_groups * BN;
        w_row0 = group * p.N + n0;
        prob = 0;
        count_later = p.bin_ahead && t0 == bin0;
        if (!count_later) {
            pdl_wait();
            t_end = bin_end();
            if (t_end <= t0) return;  // an empty tile: all CTAs of a cluster alike
        }
    }
    const bool batched = p.batch > 1;
    const int prob_b = prob;
    if (batched) {  // the problems share operand maps and output
        w_row0 = prob_b * p.N + n0;
        prob = 0;
    }
    if (beside) prob = 1;
    const bool halves = view.mode == GEMM_SWIGLU;  // A tile = 64 gate rows over 64 up rows, one accumulator
    void* out = p.out[prob];
    if (batched) {
        if (p.mode == GEMM_STORE_F32) out = (float*)out + (size_t)prob_b * p.out_batch;
        else out = (bf16*)out + (size_t)prob_b * p.out_batch;
    }
    const int total_kb = p.kblocks[0] + p.kblocks[1];
    const int kb_begin = (int)(((long long)blockIdx.z * total_kb) / p.splits);
    const int kb_end = (int)(((long long)(blockIdx.z + 1) * total_kb) / p.splits);
    const int n_iters = kb_end - kb_begin;
    const bool has0 = kb_begin < p.kblocks[0] && n_iters > 0;
    const bool has1 = kb_end > p.kblocks[0] && p.kblocks[1] > 0 && n_iters > 0;
    constexpr uint32_t tmem_cols = Cfg::TMEM_COLS;

    if (threadIdx.x == 0) {
        TFFN_TRACE(0);
        tl_mark(p.tl, 0);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    const uint2 norm_w4 = FOLD && p.norm_w && warp >= 2 ? __ldg((const uint2*)(p.norm_w + n0 + lane * 4)) : make_uint2(0u, 0u);
    FinalizePre pre[2];  // epilogue warps, split-K: operands of the columns they will finish
    pre[0].valid = pre[1].valid = false;

    // The two issuing warps pace a CTA's stream, so every lane runs their loops (uniform control flow and operands, stage and
    // phase carried along) and one is elected per instruction: from a branch of a single lane each costs several times as much.
    // Inside a decode step: down projections of base and expert, K 2 x 4 864, N 896, 64 tokens 12.0 -> 10.3 us, 13 tokens
    // 8.7 -> 6.5; q|k|v and gate|up on average 13.0 -> 12.2 (64 tokens, LM head included), 8.5 -> 7.7 (13 tokens).
    if (warp == 0) {
        const CUtensorMap *const tw = &p.tmW[prob * 2], *const tx = &p.tmX[batched ? 0 : prob * 2];
        const uint32_t ring = smem_u32(smem), full_0 = smem_u32(full);
        if (lane == 0) {
            prefetch_tmap(tw);
            prefetch_tmap(tx);
        }
        __syncwarp();
        auto load_w = [&](int i, int s) {
            const int seg = i >= p.kblocks[0] ? 1 : 0, x = (seg ? i - p.kblocks[0] : i) * BK;
            const uint32_t a = ring + s * Cfg::STAGE_BYTES, bar = full_0 + s * 8;
            mbar_arrive_expect_tx_elect(bar, Cfg::STAGE_BYTES);
            if (halves) {
                tma_load_2d_elect(a, tw, x, w_row0, bar);
                tma_load_2d_elect(a + Cfg::A_BYTES / 2, tw + 1, x, w_row0, bar);
            } else {
                tma_load_2d_elect(a, tw + seg, x, w_row0, bar);
            }
        };
        auto load_x = [&](int i, int s) {
            const int seg = i >= p.kblocks[0] ? 1 : 0, x = (seg ? i - p.kblocks[0] : i) * BK;
            const uint32_t b = ring + s * Cfg::STAGE_BYTES + Cfg::A_BYTES, bar = full_0 + s * 8;
            if (batched) tma_load_3d_elect(b, tx, x, prob_b, t0, bar);
            else tma_load_2d_elect(b, tx + seg, x, t0, bar);
        };
        // Weights do not depend on the previous kernel: the first ring of weight boxes is
        // requested before griddepcontrol.wait, the activation boxes after it.
        const int pre = n_iters < STAGES ? n_iters : STAGES;
        for (int it = 0; it < pre; ++it) load_w(kb_begin + it, it);
        if (lane == 0) TFFN_TRACE(1);
        pdl_wait();
        if (lane == 0) {
            TFFN_TRACE(2);
            tl_mark(p.tl, 1);
        }
        __syncwarp();
        for (int it = 0; it < pre; ++it) load_x(kb_begin + it, it);
        int s = 0;
        uint32_t ph = 0;
        for (int it = pre; it < n_iters; ++it) {
            if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ph, p.status, DEV_ERR_EMPTY_WAIT))) break;
            load_w(kb_begin + it, s);
            load_x(kb_begin + it, s);
            if (++s == STAGES) {
                s = 0;
                ph ^= 1;
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc_bf16(BM, BN);
        const uint64_t a_0 = umma_desc_k128(smem_u32(smem)), b_0 = umma_desc_k128(smem_u32(smem) + Cfg::A_BYTES);
        int s = 0;
        uint32_t ph = 0;
        for (int it = 0; it < n_iters; ++it) {
            if (!__all_sync(0xffffffffu, mbar_wait(&full[s], ph, p.status, DEV_ERR_FULL_WAIT))) break;
            if (lane == 0 && it < 12) TFFN_TRACE(16 + it);
            __syncwarp();
            tc_fence_after();
            const int seg = (kb_begin + it) >= p.kblocks[0] ? 1 : 0;
            const bool more = it > 0 && kb_begin + it != p.kblocks[0];  // not the first of its accumulator
            const uint64_t at = (uint64_t)(uint32_t)(s * (Cfg::STAGE_BYTES >> 4));
            const uint32_t d = tmem_base + (uint32_t)(seg * BN);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) umma_bf16_elect(d, a_0 + at + 2 * k, b_0 + at + 2 * k, idesc, (more || k > 0) ? 1u : 0u);
            umma_commit_elect(&empty[s]);
            if (++s == STAGES) {
                s = 0;
                ph ^= 1;
            }
        }
        if (lane == 0) TFFN_TRACE(3);
        __syncwarp();
        umma_commit_elect(acc_full);  // arrives when every MMA above has finished (also on the error path)
    } else {
        // Epilogue warps 2..5 own TMEM lane quarter (warp % 4): thread = one weight row. They combine
        // the two operand pairs (base + alpha * expert) and park ONE fp32 plane [column][row] in the
        // idle stage memory.
        const int q = warp & 3;
        const int row = q * 32 + lane;
        pdl_wait();  // later phases read and write buffers of earlier kernels
        if (count_later) {
            t_end = bin_end();
            if (threadIdx.x == 64) *tile_end = t_end;
        }
        // the row factors: 128 / BN neighbouring lanes per token. Their loads are requested here and used behind the requests below.
        constexpr int L = (kGemmThreads - 64) / BN < 1 ? 1 : (kGemmThreads - 64) / BN;
        const int rj = ((int)threadIdx.x - 64) / L, sub = (int)threadIdx.x % L;
        const float* from = p.rms_ssq + (size_t)(t0 + rj) * p.rms_tiles;
        float part[4] = {0.f, 0.f, 0.f, 0.f};
        if (FOLD && p.rms_ssq && t0 + rj < t_end) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (sub + u * L < p.rms_tiles) part[u] = __ldcg(from + sub + u * L);
        }
        if (p.splits > 1) {
            // split-K: the (at most two) columns this warp will finish are known; fetch their operands now
            const int S = p.splits, cps = BN / S, rank = (int)cluster_ctarank();
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int jj = (warp - 2) + 4 * u, t = t0 + jj * S + rank;
                if (cps <= 8 && jj < cps && t < t_end) {
                    if (p.mode == GEMM_QKV) prefetch_qkv(p, n0 + lane * 4, t, pre[u]);
                    else if (p.mode == GEMM_RESIDUAL) prefetch_residual(p, view, out, n0 + lane * 4, t, pre[u]);
                }
            }
        }
        if (FOLD && p.rms_ssq) {
            float ss = (part[0] + part[1]) + (part[2] + part[3]);
            for (int i0 = sub + 4 * L; i0 < p.rms_tiles && t0 + rj < t_end; i0 += 4 * L) {
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = i0 + u * L < p.rms_tiles ? __ldcg(from + i0 + u * L) : 0.f;
                ss += (v[0] + v[1]) + (v[2] + v[3]);
            }
#pragma unroll
            for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (sub == 0) row_factor[rj] = rsqrtf(ss / (float)p.rms_n + p.rms_eps);
        }
        // every lane waits (acquire); the outcome is made warp-uniform because tcgen05.ld is .aligned
        bool ok = mbar_wait(acc_full, 0, p.status, DEV_ERR_ACC_WAIT);
        ok = __all_sync(0xffffffffu, ok);
        if (threadIdx.x == 64) TFFN_TRACE(4);
        tc_fence_after();
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const bool dual = p.kblocks[1] > 0;
        const bool live = ok && n_iters > 0;
        float* plane = (float*)smem;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            if (t0 + c0 >= t_end) break;
            uint32_t v0[16], v1[16];
            if (live && has0) tmem_ld16(lane_addr + (uint32_t)c0, v0);
            if (live && has1) tmem_ld16(lane_addr + (uint32_t)(BN + c0), v1);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float a0 = (live && has0) ? __uint_as_float(v0[j]) : 0.f;
                const float a1 = (live && has1) ? __uint_as_float(v1[j]) : 0.f;
                plane[(size_t)(c0 + j) * BM + row] = dual ? a0 + p.alpha * a1 : a0;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (count_later && warp < 2) t_end = *tile_end;
    if (threadIdx.x == 64) TFFN_TRACE(5);
    // Finalisation is vectorised the other way round from the TMEM layout: a warp takes one column, a
    // lane 4 consecutive rows, so every global access is 8 or 16 bytes per lane and the RoPE partner of
    // a row sits in the same warp. With split-K the splits of one output tile form a thread-block
    // cluster (1,1,splits): after a cluster barrier each rank finalises the columns it owns
    // (column % splits == rank), adding up the parked planes of all ranks in rank order over
    // distributed shared memory (the result does not depend on scheduling). A second cluster barrier
    // keeps every plane alive until its peers have read it; a thread arrives at it as soon as its own
    // remote reads are done and waits only before it leaves, so the barrier's latency hides behind the
    // global stores. (Measured alternatives, both slower per launch: pushing the partial columns into the
    // owners' shared memory with 4-byte remote stores, +3 us; exchanging the planes through an L2
    // workspace, +1 us.)
    if (p.splits > 1) {
        cluster_sync_all();
        if (threadIdx.x == 64) TFFN_TRACE(6);
        if (warp < 2) cluster_arrive();
    }
    constexpr int kWarps = kGemmThreads / 32;
    if (n_iters > 0 && p.splits == 1 && p.mode != GEMM_QKV) {
        // Unsplit tile: every column comes from this CTA's own plane, nothing to wait for, so all six
        // warps (the copy and MMA warps are idle by now) take columns, four in flight per warp.
        const int w = warp;
        const int ncols = min(BN, t_end - t0);
        const float* plane = (const float*)smem;
        if (threadIdx.x == 64) TFFN_TRACE(9);
        if (halves) {
            // rows 0..63 of the tile hold gate, rows 64..127 up, for the same 64 output indices;
            // lane l finishes indices n0 + 2l and n0 + 2l + 1
            bf16* o = (bf16*)out;
            const int nn = n0 + 2 * lane;
            const bool pair = nn + 1 < view.N && (view.ldo & 1) == 0;
#pragma unroll 4
            for (int c = w; c < ncols; c += kWarps) {
                const float2 g = *(const float2*)(plane + (size_t)c * BM + 2 * lane);
                const float2 u = *(const float2*)(plane + (size_t)c * BM + 64 + 2 * lane);
                const float f = FOLD && p.rms_ssq ? row_factor[c] : 1.f;
                const float a0 = silu_mul_bf16(g.x * f, u.x * f), a1 = silu_mul_bf16(g.y * f, u.y * f);
                bf16* dst = o + (size_t)(t0 + c) * (size_t)view.ldo + nn;
                if (pair) {
                    *(uint32_t*)dst = (uint32_t)bf16_bits(a0) | ((uint32_t)bf16_bits(a1) << 16);
                } else {
                    if (nn < view.N) dst[0] = __float2bfloat16_rn(a0);
                    if (nn + 1 < view.N) dst[1] = __float2bfloat16_rn(a1);
                }
            }
        } else {
            const int n = n0 + lane * 4;
            FinalizePre none;
            none.valid = false;
            if (FOLD && p.norm_w) {
                if (warp >= 2)
#pragma unroll 2
                    for (int c = w - 2; c < ncols; c += kWarps - 2)
                        finalize_residual_norm(p, out, n, t0 + c, *(const float4*)(plane + (size_t)c * BM + lane * 4), none, norm_w4, lane);
            } else if (!p.amax_val) {
#pragma unroll 4
                for (int c = w; c < ncols; c += kWarps)
                    finalize_plain(p, view, out, n, t0 + c, *(const float4*)(plane + (size_t)c * BM + lane * 4), none);
            } else if (warp < 2) {
                // Fused greedy pick: thread = token column, a plain scan down the 128 parked rows (a warp
                // reduction per column would put 64 shuffle chains into every CTA's epilogue). The scan
                // starts at a row that depends on the column so that the lanes hit different banks; the
                // lowest index among equal maxima wins whatever the order.
                for (int c = (int)threadIdx.x; c < ncols; c += 64) {
                    float best = -INFINITY;
                    int bi = 0x7fffffff;
#pragma unroll 8
                    for (int j = 0; j < BM / 4; ++j) {
                        const int r = ((j + c) & (BM / 4 - 1)) * 4;
                        const float4 v = *(const float4*)(plane + (size_t)c * BM + r);
                        const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int q4 = 0; q4 < 4; ++q4) {
                            const int idx = n0 + r + q4;
                            if (idx < p.N && (f[q4] > best || (f[q4] == best && idx < bi))) { best = f[q4]; bi = idx; }
                        }
                    }
                    p.amax_val[(size_t)(t0 + c) * gridDim.x + blockIdx.x] = best;
                    p.amax_idx[(size_t)(t0 + c) * gridDim.x + blockIdx.x] = bi;
                }
            } else if (out) {
#pragma unroll 4
                for (int c = w - 2; c < ncols; c += kWarps - 2)
                    finalize_plain(p, view, out, n, t0 + c, *(const float4*)(plane + (size_t)c * BM + lane * 4), none);
            }
        }
    } else if (warp >= 2) {
        const int w = warp - 2;
        const int r4 = lane * 4;
        const int n = n0 + r4;
        const int S = p.splits, cps = BN / S;
        const uint32_t rank = S > 1 ? cluster_ctarank() : 0u;
        const uint32_t plane_local = smem_u32(smem);
        if (threadIdx.x == 64) TFFN_TRACE(9);
        // sum over the ranks' planes of rows row_off .. row_off+3 of tile column c
        auto column_sum = [&](int c, int row_off) {
            const uint32_t off = (uint32_t)(((size_t)c * BM + row_off) * 4);
            if (S == 1) return *(const float4*)(smem + off);
            float4 acc = ld_shared_cluster_v4(map_shared_rank(plane_local + off, 0u));
#pragma unroll 4
            for (int z = 1; z < S; ++z) add4(acc, ld_shared_cluster_v4(map_shared_rank(plane_local + off, (uint32_t)z)));
            return acc;
        };
        auto finish = [&](int t, float4 acc, float4 up, const FinalizePre& f) {
            if (FOLD && p.rms_ssq) {
                const float r = row_factor[t - t0];
                acc = make_float4(acc.x * r, acc.y * r, acc.z * r, acc.w * r);
                up = make_float4(up.x * r, up.y * r, up.z * r, up.w * r);
            }
            if (FOLD && p.norm_w) {
                finalize_residual_norm(p, out, n, t, acc, f, norm_w4, lane);
            } else if (p.mode == GEMM_QKV) {
                finalize_qkv(p, n, t, acc, f);
            } else if (halves) {
                // rows 0..63 of the tile hold gate, rows 64..127 up, for the same 64 output indices
                if (lane < 16)
                    finalize_plain(p, view, out, n, t,
                                   make_float4(silu_mul_bf16(acc.x, up.x), silu_mul_bf16(acc.y, up.y), silu_mul_bf16(acc.z, up.z),
                                               silu_mul_bf16(acc.w, up.w)), f);
            } else {
                finalize_plain(p, view, out, n, t, acc, f);
                publish_amax(p, n, t, acc, lane);
            }
        };
        const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (S > 1 && cps <= 8) {
            // at most two columns per warp: all remote reads first, then the arrival, then the stores
            float4 acc[2], up[2];
            bool have[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int jj = w + 4 * u, c = jj * S + (int)rank;
                have[u] = n_iters > 0 && jj < cps && t0 + c < t_end;  // warp-uniform
                acc[u] = have[u] ? column_sum(c, r4) : zero4;
                up[u] = (have[u] && halves && lane < 16) ? column_sum(c, r4 + 64) : zero4;
            }
            cluster_arrive();
            if (threadIdx.x == 64) TFFN_TRACE(10);
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (have[u]) finish(t0 + (w + 4 * u) * S + (int)rank, acc[u], up[u], pre[u]);
        } else {
            FinalizePre none;
            none.valid = false;
            for (int jj = w; jj < cps && n_iters > 0; jj += 4) {
                const int c = jj * S + (int)rank;
                if (t0 + c >= t_end) break;  // warp-uniform
                const float4 acc = column_sum(c, r4);
                const float4 up = (halves && lane < 16) ? column_sum(c, r4 + 64) : zero4;
                finish(t0 + c, acc, up, none);
            }
            if (S > 1) cluster_arrive();
        }
        if (threadIdx.x == 64) TFFN_TRACE(7);
    }
    if (p.splits > 1) cluster_wait();  // every peer has finished reading this CTA's plane
    if (threadIdx.x == 64) {
        TFFN_TRACE(8);
        tl_mark(p.tl, 2);
    }
    if (warp == 1) tmem_dealloc(tmem_base, tmem_cols);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

struct TmapKey {
    const void* ptr;
    uint64_t rows, cols, ld;
    uint32_t box_rows;
    uint32_t batch, batch_ld;
    bool operator==(const TmapKey& o) const {
        return ptr == o.ptr && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows && batch == o.batch && batch_ld == o.batch_ld;
    }
};
struct TmapKeyHash {
    size_t operator()(const TmapKey& k) const {
        return std::hash<const void*>()(k.ptr) ^ (k.rows * 1000003u) ^ (k.cols * 7919u) ^ (k.ld << 20) ^ k.box_rows ^ ((size_t)k.batch * 104729u);
    }
};

// bf16 tensor [rows, cols] with a row stride, box = box_rows x 64 columns, 128-byte swizzle. batch > 1: `batch` such
// tensors interleaved in a row, batch_ld elements apart; 3-D (column, problem, row), a box of one problem
bool encode_tmap(CUtensorMap* tm, const bf16* ptr, uint64_t rows, uint64_t cols, uint64_t ld_elems, uint32_t box_rows, uint32_t batch,
                 uint32_t batch_ld) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return false;
    const bool b = batch > 1;
    cuuint64_t dims[3] = {cols, b ? batch : rows, rows};
    cuuint64_t strides[2] = {(b ? batch_ld : ld_elems) * 2, ld_elems * 2};
    cuuint32_t box[3] = {(cuuint32_t)BK, b ? 1u : box_rows, box_rows};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, b ? 3 : 2, (void*)ptr, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

}  // namespace

struct TmapCache {
    std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> maps;
};
TmapCache* tmap_cache_create() { return new TmapCache(); }
void tmap_cache_free(TmapCache* c) { delete c; }

namespace {

bool make_tmap(TmapCache* cache, CUtensorMap* tm, const bf16* ptr, uint64_t rows, uint64_t cols, uint64_t ld_elems, uint32_t box_rows,
               uint32_t batch = 1, uint32_t batch_ld = 0) {
    if (!cache) return encode_tmap(tm, ptr, rows, cols, ld_elems, box_rows, batch, batch_ld);
    TmapKey key{ptr, rows, cols, ld_elems, box_rows, batch, batch_ld};
    auto it = cache->maps.find(key);
    if (it != cache->maps.end()) {
        *tm = it->second;
        return true;
    }
    if (!encode_tmap(tm, ptr, rows, cols, ld_elems, box_rows, batch, batch_ld)) return false;
    cache->maps.emplace(key, *tm);
    return true;
}

// clusters of `splits` CTAs of k_gemm_tc<BN> with `stages` ring stages that can be resident at once on the
// current device (cudaOccupancyMaxActiveClusters; remembered per configuration)
template <int BN>
int max_active_clusters(const cudaLaunchConfig_t& cfg, int stages, int splits) {
    static std::mutex mu;
    static std::unordered_map<long long, int> seen;
    int dev = 0;
    cudaGetDevice(&dev);
    const long long key = ((long long)dev << 32) | ((long long)stages << 8) | splits;
    std::lock_guard<std::mutex> lock(mu);
    auto it = seen.find(key);
    if (it != seen.end()) return it->second;
    int n = 0;
    cudaLaunchConfig_t q = cfg;
    q.dynamicSmemBytes = GemmCfg<BN>::smem_bytes(stages);
    if (cudaOccupancyMaxActiveClusters(&n, k_gemm_tc<BN, TC_PLAIN>, &q) != cudaSuccess) {
        cudaGetLastError();
        n = 1 << 30;  // unknown: keep the configuration
    }
    seen.emplace(key, n);
    return n;
}

// beside: an independent GEMM_SWIGLU of the same rows and K whose tiles follow those of c, or nullptr
template <int BN>
int launch_bn(const GemmCall& c, const GemmWorkspace& ws, cudaStream_t stream, int force_splits, const GemmCall* beside = nullptr) {
    using Cfg = GemmCfg<BN>;
    GemmDev p;
    memset(&p, 0, sizeof p);
    const bool batched = c.batch > 1;
    const int maps = c.out2 ? 2 : 1, nprob = batched ? c.batch : maps;
    const bool halves = c.mode == GEMM_SWIGLU;
    p.tile_n = halves ? BM / 2 : BM;
    if (halves && (c.op[0].K != c.op[1].K || c.op[0].X != c.op[1].X)) return (int)cudaErrorInvalidValue;
    if (batched && (c.out2 || c.grp || c.op[1].K > 0 || c.x_batch % 8 || (c.mode != GEMM_STORE_F32 && c.mode != GEMM_STORE_BF16) || c.amax_val))
        return (int)cudaErrorInvalidValue;
    for (int pr = 0; pr < maps; ++pr)
        for (int i = 0; i < 2; ++i) {
            const GemmOperand& o = pr ? c.op2[i] : c.op[i];
            if (pr == 0) p.kblocks[i] = o.K > 0 ? (o.K + BK - 1) / BK : 0;
            if (o.K <= 0) continue;
            if (pr == 1 && (o.K + BK - 1) / BK != p.kblocks[i]) return (int)cudaErrorInvalidValue;
            const uint64_t w_rows = (uint64_t)c.N * (c.grp || c.bin_counts ? c.grp_count : batched ? c.batch : 1);
            if (!make_tmap(ws.tmaps, &p.tmW[pr * 2 + i], o.W, w_rows, (uint64_t)o.K, (uint64_t)o.ldw, halves ? BM / 2 : BM)) return -1000;
            if (!make_tmap(ws.tmaps, &p.tmX[pr * 2 + i], o.X, (uint64_t)(c.x_rows_alloc > c.T ? c.x_rows_alloc : c.T), (uint64_t)o.K,
                           (uint64_t)o.ldx, BN, batched ? (uint32_t)c.batch : 1u, (uint32_t)c.x_batch))
                return -1000;
        }
    if (halves) p.kblocks[1] = 0;  // gate and up rows share one accumulator and one pass over K
    if (beside) {
        if (batched || c.grp || c.bin_counts || c.out2 || halves || c.op[1].K > 0 || c.mode == GEMM_QKV || c.norm_w || beside->mode != GEMM_SWIGLU || beside->T != c.T ||
            beside->op[0].K != c.op[0].K || beside->op[1].K != c.op[0].K || beside->op[1].X != beside->op[0].X || beside->out2 || beside->rms_ssq)
            return (int)cudaErrorInvalidValue;
        for (int i = 0; i < 2; ++i) {
            const GemmOperand& o = beside->op[i];
            if (!make_tmap(ws.tmaps, &p.tmW[2 + i], o.W, (uint64_t)beside->N, (uint64_t)o.K, (uint64_t)o.ldw, BM / 2)) return -1000;
            if (!make_tmap(ws.tmaps, &p.tmX[2 + i], o.X, (uint64_t)(beside->x_rows_alloc > c.T ? beside->x_rows_alloc : c.T), (uint64_t)o.K, (uint64_t)o.ldx, BN))
                return -1000;
        }
    }
    for (int i = 1; i < 4; ++i)  // keep unused maps valid
        if ((!beside || i < 2) && (i >= maps * 2 || (p.kblocks[i & 1] == 0 && !halves))) {
            p.tmW[i] = p.tmW[0];
            p.tmX[i] = p.tmX[0];
        }
    p.batch = batched ? c.batch : 1;
    p.out_batch = batched ? c.out_batch : 0;
    p.N = c.N;
    p.T = c.T;
    p.mode = c.mode;
    p.alpha = c.alpha;
    p.out_scale = c.out_scale == 0.f ? 1.f : c.out_scale;
    p.out[0] = c.out;
    p.out[1] = beside ? beside->out : c.out2 ? c.out2 : c.out;
    p.N_2 = beside ? beside->N : 0;
    p.ldo_2 = beside ? beside->ldo : 0;
    p.ldo = c.ldo;
    p.status = ws.status;
    p.trace = c.trace;
    p.tl = c.tl;
    if ((c.norm_w && (c.mode != GEMM_RESIDUAL || !c.norm_out || !c.norm_ssq || c.N % BM || c.ldo % 4)) ||
        (c.rms_ssq && ((c.mode != GEMM_QKV && c.mode != GEMM_SWIGLU) || c.rms_tiles < 1 || c.rms_n < 1)) ||
        ((c.norm_w || c.rms_ssq) && (c.T > kFoldTokens || batched || c.grp || c.bin_counts)))
        return (int)cudaErrorInvalidValue;
    p.norm_w = c.norm_w;
    p.norm_out = c.norm_out;
    p.norm_ssq = c.norm_ssq;
    p.rms_ssq = c.rms_ssq;
    p.rms_tiles = c.rms_tiles;
    p.rms_n = c.rms_n;
    p.rms_eps = c.rms_eps;
    p.amax_val = c.mode == GEMM_STORE_F32 ? c.amax_val : nullptr;
    p.amax_idx = c.amax_idx;
    if (!c.out && !(c.mode == GEMM_STORE_F32 && c.amax_val && c.amax_idx) && c.mode != GEMM_QKV) return (int)cudaErrorInvalidValue;
    if (c.mode == GEMM_QKV) {
        if (!c.qkv || c.op[1].K > 0 || c.out2 || (c.qkv->kv.hd != 64 && c.qkv->kv.hd != 128)) return (int)cudaErrorInvalidValue;
        p.qkv = *c.qkv;
    }
    p.tiles_1 = beside ? (c.N + BM - 1) / BM : 0;
    const int n_tiles = (c.N + p.tile_n - 1) / p.tile_n + (beside ? (beside->N + BM / 2 - 1) / (BM / 2) : 0),
              bin_tiles = (c.bin + BN - 1) / BN, t_tiles = c.bin_counts ? c.grp_count * bin_tiles : c.grp ? c.grp_tiles : (c.T + BN - 1) / BN;
    if (c.bin_counts && (c.grp || batched || c.grp_bn != BN || BN > 64 || c.op[1].K > 0 || c.out2 || halves || c.mode == GEMM_QKV || c.bin < 1 || c.grp_count < 1))
        return (int)cudaErrorInvalidValue;
    p.bins = c.bin_counts;
    p.bin = c.bin;
    p.bin_groups = c.grp_count;
    p.bin_ahead = c.bin_ahead ? 1 : 0;
    if (c.grp && (c.grp_bn != BN || c.op[1].K > 0 || c.out2 || halves || c.mode == GEMM_QKV || c.grp_tiles < 1 || c.grp_count < 1))
        return (int)cudaErrorInvalidValue;
    p.grp = c.grp;
    const int total_kb = p.kblocks[0] + p.kblocks[1];
    // grouped: the grid has room for the worst case, the split policy goes by one tile per group that can have rows
    const int tiles = (c.grp || c.bin_counts) && c.grp_rows_hint > 0 ? n_tiles * c.grp_rows_hint : n_tiles * t_tiles * nprob;
    p.t_tiles = t_tiles;
    // K splits = cluster size (1, 2, 4, 8 or 16). A CTA's stream is bound by the latency of its stages (about 50 GB/s per SM,
    // all SMs together about 7 TB/s), so a weight-streaming launch needs about as many CTAs as there are SMs: tiles are split
    // along K until the grid fills the SMs.
    int splits = 1;
    if (force_splits > 0) {
        splits = force_splits;
    } else {
        while (splits < kMaxSplits && tiles * splits * 2 <= ws.num_sms + ws.num_sms / 8 && total_kb / (splits * 2) >= 1) splits *= 2;
        // A long K extent: two CTAs per SM stream twice as much as one until HBM is the limit; keep splitting while every CTA
        // still gets eight k-blocks and the grid fits two per SM (measured at 16 tokens, N 2048, K 22016:
        // 8 splits 49.5 us, half of the 8-CTA clusters waiting for a second wave; 16 splits 18.0 us).
        // A grouped launch cannot request weights ahead of its dependency wait (the tile table comes from the kernel
        // before), so its k-loop is all exposed and shorter splits pay.
        const int min_kb = c.grp || (c.bin_counts && !c.bin_ahead) ? 3 : 8;
        // From 32 to 64 tokens a stage's products weigh more and a second CTA on a third of the SMs is as far as it pays (us a step of
        // four layers, K 22016, N 2048: 32 tokens 381 with 16 splits, 364 with 8; 64 tokens in 32-wide tiles 462, in 64-wide ones 428
        // and 406; K 17920, N 1536: 64 tokens 390, 352, 352).
        const int most = (BN != 32 && BN != 64) || c.grp || c.bin_counts ? 2 * ws.num_sms : ws.num_sms + ws.num_sms / 3;
        // Tiles that the loop above left whole, up to four fifths of the SMs (84 to 118 of 148), stay whole: their halves would be two
        // to an SM here and one there, and need clusters. Back to back with early starts, us a launch whole and in halves, 84 and 118
        // tiles: 16 tokens, K 512 4.5, 6.7 and 5.3, 7.0; K 2048 10.9, 12.3 and 12.5, 15.7; K 17920 62.4, 65.0 and 80.0, 101.8; 64
        // tokens, K 2048 12.0, 15.5 and 14.0, 17.2; K 17920 67.5, 72.4 and 84.7, 87.9; 100 tokens, K 2048 13.5, 29.8 and 15.2, 31.2; K
        // 17920 75.0, 98.8 and 90.3, 107.2. A step of one sequence, 8 layers 2 048 wide, first products of 96 and 113 tiles: 450 -> 430.
        const bool whole = !c.grp && !c.bin_counts && splits == 1 && tiles * 10 < ws.num_sms * 8;
        while (!whole && splits < kMaxSplits && tiles * splits * 2 <= most && total_kb / (splits * 2) >= min_kb) splits *= 2;
    }
    if (splits != 1 && splits != 2 && splits != 4 && splits != 8 && splits != 16) return (int)cudaErrorInvalidValue;
    if (splits > total_kb) return (int)cudaErrorInvalidValue;
    const bool shared_sm = tiles * splits > ws.num_sms;  // more than one CTA per SM
    p.stages = shared_sm ? Cfg::SHARED_STAGES : Cfg::MAX_STAGES;
    // Many short tiles per SM (the LM head of a small model: 1 187 tiles of 14 k-blocks): what limits such a
    // launch is the set-up and epilogue of every tile, which the other CTAs of the SM have to cover. Three
    // CTAs per SM with 3-stage rings do that better than two with 4 stages (measured inside a decode step,
    // 0.5B shape, 64 tokens: 61 -> 50 us for the 272 MB LM head = 5.4 TB/s).
    if (shared_sm && BN == 64 && splits == 1 && total_kb <= 16 && tiles >= 4 * ws.num_sms) p.stages = 3;
    {
        // No deeper than the k-blocks a CTA streams (but deep enough to park the epilogue plane): the
        // shared memory a CTA does not claim lets CTAs of the next kernel of the stream become resident
        // early under programmatic dependent launch and fetch their weights ahead of their grid wait.
        const int iters = (total_kb + splits - 1) / splits;
        const int plane_stages = (BN * BM * 4 + BN * 8 /* per-token maxima of the fused pick */ + Cfg::STAGE_BYTES - 1) / Cfg::STAGE_BYTES;
        const int want = iters > plane_stages ? iters : plane_stages;
        if (p.stages > want) p.stages = want;
    }
    p.splits = splits;
    cudaLaunchConfig_t cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(n_tiles, t_tiles * nprob, splits);
    if ((long long)n_tiles * t_tiles * nprob * splits > c.trace_ctas) p.trace = nullptr;
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = Cfg::smem_bytes(p.stages);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (splits > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 1;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = splits;
        ++na;
    }
    if (c.pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    if (splits > 1 && !shared_sm) {
        // A cluster lives inside one GPC. With deep rings (one CTA per SM) a GPC of 18 SMs holds two clusters
        // of 8 and leaves two SMs empty, so that 18 clusters need a second wave (seen on the 7B shape over two
        // ranks: q|k|v, 18 clusters of 8 with 7-stage rings, 2 clusters started 14 us late). Ask how many
        // clusters of this launch can be resident at once and, if they are fewer than the grid has, give up
        // ring depth (not below three stages or what the epilogue plane needs) until they all fit. Grids of
        // more CTAs than SMs already run their shallow shared-SM rings and are left alone.
        const int clusters = n_tiles * t_tiles * nprob;
        const int iters = (total_kb + splits - 1) / splits;
        const int plane_stages = (BN * BM * 4 + BN * 8 + Cfg::STAGE_BYTES - 1) / Cfg::STAGE_BYTES;
        const int want_stages = iters < 3 ? iters : 3;
        const int floor_stages = plane_stages > want_stages ? plane_stages : want_stages;  // never below the parked plane
        while (p.stages > floor_stages && max_active_clusters<BN>(cfg, p.stages, splits) < clusters) {
            --p.stages;
            cfg.dynamicSmemBytes = Cfg::smem_bytes(p.stages);
        }
    }
    if constexpr (BN <= kFoldTokens) {
        if (p.norm_w || p.rms_ssq) return (int)cudaLaunchKernelEx(&cfg, k_gemm_tc<BN, TC_FOLD>, p);
        if (p.bins || beside || c.mixed) return (int)cudaLaunchKernelEx(&cfg, k_gemm_tc<BN, TC_MIXED>, p);
    }
    return (int)cudaLaunchKernelEx(&cfg, k_gemm_tc<BN, TC_PLAIN>, p);
}

}  // namespace

bool make_tmap_2d(TmapCache* cache, CUtensorMap* tm, const bf16* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t batch,
                  uint32_t batch_ld) {
    return make_tmap(cache, tm, ptr, rows, cols, ld, box_rows, batch, batch_ld);
}

int gemm_prepare() {
    cudaError_t e;
#define TFFN_PREP(BN, KIND)                                                                                                 \
    e = cudaFuncSetAttribute(k_gemm_tc<BN, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem); \
    if (e != cudaSuccess) return (int)e;                                                                             \
    e = cudaFuncSetAttribute(k_gemm_tc<BN, KIND>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);                     \
    if (e != cudaSuccess) return (int)e;                                                                             \
    e = prefer_max_shared(k_gemm_tc<BN, KIND>);                                                                            \
    if (e != cudaSuccess) return (int)e;
    TFFN_PREP(16, TC_PLAIN) TFFN_PREP(32, TC_PLAIN) TFFN_PREP(64, TC_PLAIN) TFFN_PREP(128, TC_PLAIN) TFFN_PREP(256, TC_PLAIN)
    TFFN_PREP(16, TC_FOLD) TFFN_PREP(32, TC_FOLD) TFFN_PREP(64, TC_FOLD)
    TFFN_PREP(16, TC_MIXED) TFFN_PREP(32, TC_MIXED) TFFN_PREP(64, TC_MIXED)
#undef TFFN_PREP
    return gemm_pair_prepare();
}

// Groups differ in size: a tile of the average size would leave the larger half of the groups a second, nearly
// empty tile and their weights would be streamed twice, so the tile has room for twice the average.
int gemm_group_tile(int rows) {
    int bn = 16;
    while (bn < 256 && bn < 2 * rows) bn *= 2;
    return bn;
}

int cheaper_width(long long narrow, long long wide, int kb, int num_sms, bool can_split) {
    auto us = [&](long long tiles, int bn) {
        const PairSplit s = pair_split(tiles, kb, bn, num_sms);
        return can_split ? s.us : s.whole_us;
    };
    return us(narrow, 128) <= us(wide, 256) ? 128 : 256;
}
// Which launches take the two-CTA tiles of gemm_pair.cu, and how wide (0: none). Measured back to back on one B200 against
// the tiles of this file (us, here -> there): 4 096 tokens, K 896: q|k|v N 1152 87 -> 23, N 4864 gate|up of base and expert
// 277 -> 118 (1.21 PFLOP/s); 2 048 tokens, K 3584, N 18944: 1 235 -> 726 (1.53 PFLOP/s).
//  * gate|up from 65 tokens on (K 896, N 4864: 28 -> 13); other products from 129 on where K is short enough that splitting
//    it cannot make up for the wider tile (N 4608, K 3584: 160 tokens 50 -> 28, 128 tokens 25 -> 28); very short ones from 65.
//  * A long K extent with few tiles is split over clusters here: 14 wide tiles of 152 k-blocks 14 -> 50. The wide tiles win
//    once they are about a quarter of the k-blocks in number, or nearly fill the chip (K 4864, N 896: 768 tokens 39 -> 29,
//    512 tokens 21 -> 29; two pairs of that K: 1 000 tokens 49 -> 54, 2 048 tokens 80 -> 56), or, where they can be split too, from
//    2 700 narrow tiles' k-blocks on (with 6 us of launch: K 11008, N 2048: 130 tokens 55 -> 43, 512 tokens 81 -> 44; K 17920 of two
//    pairs, N 1536: 130 tokens 46 -> 49, 512 tokens 70 -> 50, 1 000 tokens 109 -> 60; K 37888, N 3584: 130 tokens 95 -> 80; below:
//    K 9728, N 896: 384 tokens 39 -> 41, 256 tokens 25 -> 30).
//  * One narrow row tile (a router) needs many tokens (K 896: 4 096 tokens 14 -> 8; K 2048: 768 tokens 9 -> 13).
int pair_width(const GemmCall& c, const GemmWorkspace& ws) {
    if (c.amax_val || c.norm_w || c.rms_ssq || c.bin_counts || (!c.out && c.mode != GEMM_QKV) || (c.grp && c.grp_bn != 256)) return 0;
    const bool halves = c.mode == GEMM_SWIGLU, batched = c.batch > 1;
    // what launch_bn refuses stays with it
    if (halves && (c.op[0].K != c.op[1].K || c.op[0].X != c.op[1].X)) return 0;
    if (batched && (c.out2 || c.grp || c.op[1].K > 0 || c.x_batch % 8 || (c.mode != GEMM_STORE_F32 && c.mode != GEMM_STORE_BF16))) return 0;
    if (c.grp && (c.op[1].K > 0 || c.out2 || halves || c.mode == GEMM_QKV || c.grp_tiles < 1 || c.grp_count < 1)) return 0;
    if (c.out2 && (c.op2[0].K != c.op[0].K || c.op2[1].K != c.op[1].K)) return 0;
    if (c.mode == GEMM_QKV && (!c.qkv || c.op[1].K > 0 || c.out2 || (c.qkv->kv.hd != 64 && c.qkv->kv.hd != 128))) return 0;
    const int kb = (c.op[0].K + BK - 1) / BK + (c.op[1].K > 0 && !halves ? (c.op[1].K + BK - 1) / BK : 0);
    const long long rows = (c.grp ? (c.grp_rows_hint > 0 ? c.grp_rows_hint : c.grp_tiles) : (c.T + 255) / 256) * (batched ? (long long)c.batch : c.out2 ? 2 : 1);
    const long long wide = rows * ((c.N + (halves ? 127 : 255)) / (halves ? 128 : 256)), narrow = rows * ((c.N + (halves ? 63 : 127)) / (halves ? 64 : 128));
    const bool can_split = !c.grp && ws.partials && (c.mode == GEMM_STORE_F32 || c.mode == GEMM_STORE_BF16 || c.mode == GEMM_RESIDUAL);
    if (!c.grp) {
        if (c.N <= BM && !batched && !halves) {
            if (c.T < 2048) return 0;
        } else if (c.T <= (halves || kb <= 8 ? 64 : 128)) {
            return 0;
        } else if (!halves && kb > 56 && narrow * 4 < (kb < 240 ? kb : 240) && (!can_split || narrow * kb < 2700)) {
            return 0;
        }
    }
    return cheaper_width(narrow, wide, kb, ws.num_sms, can_split);
}

int launch_gemm_layers(const GemmCall& c, const GemmWorkspace& ws, cudaStream_t stream) {
    const bool halves = c.mode == GEMM_SWIGLU;
    if (c.T <= 0 || c.N <= 0 || c.op[0].K <= 0 || !c.out || (halves && (c.op[0].K != c.op[1].K || c.op[0].X != c.op[1].X))) return (int)cudaErrorInvalidValue;
    const long long rows = (long long)((c.T + 255) / 256) * (c.layers > 1 ? c.layers : 1);
    const int wide_n = halves ? 128 : 256;
    const int bn = cheaper_width(rows * ((c.N + wide_n / 2 - 1) / (wide_n / 2)), rows * ((c.N + wide_n - 1) / wide_n), (c.op[0].K + BK - 1) / BK, ws.num_sms, false);
    return launch_gemm_pair(c, ws, stream, bn);
}

int launch_gemm(const GemmCall& c, const GemmWorkspace& ws, cudaStream_t stream, int force_splits) {
    if (c.T <= 0 || c.N <= 0 || c.op[0].K <= 0) return (int)cudaErrorInvalidValue;
    if (force_splits == 0)
        if (const int bn = pair_width(c, ws)) return launch_gemm_pair(c, ws, stream, bn);
    if (c.grp || c.bin_counts) {
        switch (c.grp_bn) {
            case 16: return launch_bn<16>(c, ws, stream, force_splits);
            case 32: return launch_bn<32>(c, ws, stream, force_splits);
            case 64: return launch_bn<64>(c, ws, stream, force_splits);
            case 128: return launch_bn<128>(c, ws, stream, force_splits);
            case 256: return launch_bn<256>(c, ws, stream, force_splits);
            default: return (int)cudaErrorInvalidValue;
        }
    }
    // A short K extent with few output tiles (the attention projections of a small model): the grid is
    // filled by splitting K, and the cost of such a launch is the exchange of the partial tiles (measured:
    // 28 KB per CTA over distributed shared memory take 2 to 3.6 us). Halving the token tile (two token
    // tiles, the same split factor, twice the CTAs) halves the plane a CTA parks and the exchange: 14 KB per
    // CTA; the weights are then read twice, the second time from L2 (measured on the 0.5B shape at 64
    // tokens: q|k|v 8.5 -> 7.2 us, o_proj 8.0 -> 7.2 us per launch inside a step).
    {
        const int total_kb = (c.op[0].K + BK - 1) / BK + (c.op[1].K > 0 ? (c.op[1].K + BK - 1) / BK : 0);
        const int n_tiles = (c.N + BM - 1) / BM;
        if (force_splits == 0 && c.mode != GEMM_SWIGLU && !c.out2 && c.T > 32 && c.T <= 64 && total_kb <= 16 &&
            n_tiles * 8 <= ws.num_sms)
            return launch_bn<32>(c, ws, stream, force_splits);
        // A long K extent with as few tiles (the down projection of the narrowest model): the largest cluster, 16 splits, is
        // not enough to fill the SMs with 64-token tiles; with 32-token tiles twice as many CTAs (two per SM)
        // stream half as many k-blocks each (measured: 12.6 -> 11.6 us per launch inside a step), as long as the SMs hold them all.
        if (force_splits == 0 && c.mode != GEMM_SWIGLU && !c.out2 && c.T > 32 && c.T <= 64 && total_kb >= 64 && n_tiles * kMaxSplits <= ws.num_sms)
            return launch_bn<32>(c, ws, stream, kMaxSplits);
    }
    // One row tile (a router): with wide token tiles a handful of CTAs would carry the whole launch and split it along
    // K, exchanging planes that are mostly padding; narrow token tiles spread it over the SMs instead.
    if (c.N <= BM && c.T > 64 && c.mode == GEMM_STORE_F32 && !c.out2 && c.op[1].K <= 0) return launch_bn<64>(c, ws, stream, force_splits);
    // Many tiles of a short K extent (prompts): the set-up and epilogue of a tile weigh as much as its products, and three
    // CTAs of 64 tokens per SM cover them better than one of 256 (4 096 tokens, K 64 to 896: 5 to 30 % less time per launch).
    {
        const int total_kb = (c.op[0].K + BK - 1) / BK + (c.op[1].K > 0 && c.mode != GEMM_SWIGLU ? (c.op[1].K + BK - 1) / BK : 0);
        const long long tiles = (long long)((c.N + BM - 1) / BM) * ((c.T + 63) / 64) * (c.batch > 1 ? c.batch : 1) * (c.mode == GEMM_SWIGLU ? 2 : 1);
        if (force_splits == 0 && c.T > 64 && total_kb <= 14 && tiles >= 4ll * ws.num_sms) return launch_bn<64>(c, ws, stream, force_splits);
    }
    if (c.T <= 16) return launch_bn<16>(c, ws, stream, force_splits);
    if (c.T <= 32) return launch_bn<32>(c, ws, stream, force_splits);
    if (c.T <= 64) return launch_bn<64>(c, ws, stream, force_splits);
    if (c.T <= 128) return launch_bn<128>(c, ws, stream, force_splits);
    return launch_bn<256>(c, ws, stream, force_splits);
}

int launch_gemm_beside(const GemmCall& a, const GemmCall& b, const GemmWorkspace& ws, cudaStream_t stream) {
    const bool one = a.T > 0 && a.T <= 64 && b.T == a.T && a.N > 0 && b.N > 0 && a.out && b.out && a.op[0].K > 0 && a.op[0].K == b.op[0].K && b.mode == GEMM_SWIGLU &&
                     !pair_width(a, ws) && !pair_width(b, ws);
    if (!one) {
        const int rc = launch_gemm(a, ws, stream);
        return rc ? rc : launch_gemm(b, ws, stream);
    }
    if (a.T <= 16) return launch_bn<16>(a, ws, stream, 0, &b);
    return a.T <= 32 ? launch_bn<32>(a, ws, stream, 0, &b) : launch_bn<64>(a, ws, stream, 0, &b);
}

}  // namespace tffn
