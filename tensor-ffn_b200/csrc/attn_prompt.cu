// Grouped-query attention of prompt rows over the paged bf16 cache on the tensor cores (arithmetic as in attn.cu:
// inference/src/model/qwen.cu:349-412). The query heads of a kv head at up to 128 / G consecutive tokens of a sequence are the
// 128 rows of one tile, so that a tile's causal edge is a few tokens wide whatever G is, and a page is read once for all of them:
//   S[row, key] = Q[row, :] . K[key, :]    tcgen05.mma, Q and K in shared memory (both K-major)
//   O[row, :]  += P[row, :] . V[key, :]    tcgen05.mma, P in tensor memory, V read the other way round (N-major)
// q and P are fp32 in the reference; each enters its product as a bf16 pair (hi + lo, 16 mantissa bits).
//
// One CTA = one tile, 6 warps, two CTAs per SM (one's softmax runs under the other's products):
//   warps 0-3  Q into shared memory; then thread = row: S out of tensor memory, online softmax in fp32, P back into the
//              columns S came from, and the output row at the end
//   warp 4     TMA producer: 64 keys (two pages) per stage, K and V in rings of their own
//   warp 5     tensor memory and the products: S of the next tile is issued before P V of this one
// The reference maximum of a row moves only when it would be exceeded by more than 2^8, so O is rarely rescaled.
//
// What bounds it: a tile step is the softmax's instructions at 64 columns (64 exponentials and their split per row) and the
// products' operand reads as well at 128; short prompts are bound by the chain wait, Q, S, softmax, P V, output (about 6 us).
// Measured inside a request, per layer and 4 096 tokens, against the warp-level mma.sync kernel it replaced (eight tokens per
// CTA): 8 x 512 tokens of 14 heads of 64 82 -> 30 us; 2 x 2 048 of 12 heads of 128 350 -> 56 us; 4 001 of 16 heads of 128
// 646 -> 106 us; 128 tokens 7.5 -> 7.9 us (fewer rows run as a block per token: attention_prompt_as_rows).
#include "kernels.h"
#include "ptx.cuh"
#include "launch.h"
#include <cmath>
#include <cstring>

namespace tffn {

namespace {

constexpr int TK = 64, kRows = 128, kThreads = 192;
constexpr float kNeg = -1e30f;

template <int HD>
struct PromptCfg {
    static constexpr int BLOCKS = HD / 64;                 // column blocks of 64 (128 swizzled bytes)
    static constexpr int Q_BLOCK = kRows * 128, K_BLOCK = TK * 128;
    static constexpr int Q_BYTES = 2 * BLOCKS * Q_BLOCK;   // hi, lo
    static constexpr int TILE_BYTES = BLOCKS * K_BLOCK;    // K or V of a stage
    // 112 KB at 128 columns is what two CTAs per SM leave: the V ring is one deep there, since V is needed a softmax later than K
    static constexpr int KST = HD == 64 ? 3 : 2, VST = HD == 64 ? 3 : 1;
    static constexpr int BAR_OFF = Q_BYTES + (KST + VST) * TILE_BYTES;
    static constexpr int SMEM = BAR_OFF + 256;
    static constexpr int COL_O = 2 * TK;                   // S / P twice, then O
    static constexpr int TMEM_COLS = 256;
};

struct PromptDev {
    CUtensorMap tmK, tmV;  // [pages * nkv * kPageTokens][hd or vd] of this layer, boxes of 64 columns x one page
    const float* q;        // [T][nh][kd]
    const int* block_table;
    int max_pages_per_seq, num_pages, nkv;
    const int *tok_seq, *tok_pos, *grp_first, *grp_count;
    bf16* ctx;
    long long ctx_ld;
    int nh, G, part_heads, parts;  // query heads per kv head; heads of a tile; parts of at most kRows heads
    int kd, vdim, chunk, vec;      // vec: output rows can be written 16 bytes at a time
    int warm;
    float scale_log2;
    int* status;
    unsigned long long* tl;
};

template <int HD>
__global__ void __launch_bounds__(kThreads, 2) k_attn_prompt(const __grid_constant__ PromptDev p) {
    using C = PromptCfg<HD>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *const q_s = smem, *const k_s = smem + C::Q_BYTES, *const v_s = k_s + C::KST * C::TILE_BYTES;
    uint64_t* const k_full = (uint64_t*)(smem + C::BAR_OFF);
    uint64_t *const k_empty = k_full + 3, *const v_full = k_empty + 3, *const v_empty = v_full + 3;
    uint64_t *const s_full = v_empty + 3, *const p_full = s_full + 2, *const q_full = p_full + 2, *const pv_done = q_full + 1;
    uint32_t* const tmem_slot = (uint32_t*)(pv_done + 1);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (tid == 0) {
        tl_mark(p.tl, 0);
        for (int i = 0; i < 3; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], kRows);
        }
        mbar_init(q_full, kRows);
        mbar_init(pv_done, 1);
        fence_mbar_init();
    }
    if (warp == 5) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();  // behind the allocation: a dependent kernel's must not get ahead of it
    const int unit = blockIdx.x, part = unit % p.parts, kvh = unit / p.parts % p.nkv;
    const int group = gridDim.x / (p.parts * p.nkv) - 1 - unit / p.parts / p.nkv;  // later groups see more keys: first
    // groups, slots, positions and block tables are older than the step's first kernel (a full dependency of the stream)
    const int t0 = __ldcg(p.grp_first + group), ntok = __ldcg(p.grp_count + group);
    const int seq = __ldcg(p.tok_seq + t0);
    const int first_pos = __ldcg(p.tok_pos + t0), len = first_pos + ntok;  // consecutive positions
    const int key0 = p.chunk > 0 ? first_pos / p.chunk * p.chunk / kPageTokens * kPageTokens : 0;  // first visible key, rounded to a page
    const bool len_ok = first_pos >= 0 && (len + kPageTokens - 1) / kPageTokens <= p.max_pages_per_seq;
    if (!len_ok && tid == 0) dev_fail(p.status, DEV_ERR_BOUNDS);
    const int tiles = len_ok ? (len - key0 + TK - 1) / TK : 0;
    const int head0 = part * p.part_heads, nheads = min(p.part_heads, p.G - head0);

    if (warp == 4) {
        if (lane == 0) {
            prefetch_tmap(&p.tmK);
            prefetch_tmap(&p.tmV);
        }
        __syncwarp();
        const int* bt = p.block_table + (size_t)seq * p.max_pages_per_seq;
        const int page0 = key0 / kPageTokens, last_page = (len - 1) / kPageTokens;
        const uint32_t k_a = smem_u32(k_s), v_a = smem_u32(v_s), kf = smem_u32(k_full), vf = smem_u32(v_full);
        auto pages = [&](int j) {  // ids of 32 pages (lane = page); those past the end are replaced by the last one, whose keys are masked
            int id = __ldg(bt + min(page0 + j * 2 + lane, last_page));
            if (id < 0 || id >= p.num_pages) {
                dev_fail(p.status, DEV_ERR_BOUNDS);
                id = 0;
            }
            return id;
        };
        int ids[2] = {0, 0};  // of K's and of V's current tiles
        if (tiles > 0) ids[0] = ids[1] = pages(0);
        pdl_wait();  // the keys and values of these very tokens
        if (lane == 0) tl_mark(p.tl, 1);
        auto load = [&](const CUtensorMap* tm, int which, int j, uint32_t dst, uint32_t bar) {
            if (j > 0 && j * 2 % 32 == 0) ids[which] = pages(j);
            mbar_arrive_expect_tx_elect(bar, C::TILE_BYTES);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = (__shfl_sync(0xffffffffu, ids[which], (j * 2 + h) % 32) * p.nkv + kvh) * kPageTokens;
#pragma unroll
                for (int b = 0; b < C::BLOCKS; ++b) tma_load_2d_elect(dst + b * C::K_BLOCK + h * kPageTokens * 128, tm, b * 64, row, bar);
            }
        };
        bool ok = true;
        // K runs a tile ahead of V: its buffer is free once S of an earlier tile is there, V's only after a P V
        for (int j = 0; j <= tiles && ok; ++j) {
            if (j < tiles) {
                const int st = j % C::KST;
                if (j >= C::KST) ok = __all_sync(0xffffffffu, mbar_wait(&k_empty[st], (uint32_t)(j / C::KST - 1) & 1u, p.status, DEV_ERR_EMPTY_WAIT));
                if (ok) load(&p.tmK, 0, j, k_a + st * C::TILE_BYTES, kf + st * 8);
            }
            if (j > 0 && ok) {
                const int i = j - 1, st = i % C::VST;
                if (i >= C::VST) ok = __all_sync(0xffffffffu, mbar_wait(&v_empty[st], (uint32_t)(i / C::VST - 1) & 1u, p.status, DEV_ERR_EMPTY_WAIT));
                if (ok) load(&p.tmV, 1, i, v_a + st * C::TILE_BYTES, vf + st * 8);
            }
        }
    } else if (warp == 5) {
        constexpr uint32_t idesc_s = umma_idesc_bf16(kRows, TK), idesc_o = umma_idesc_bf16(kRows, HD) | (1u << 16);  // V: its K extent in rows
        const uint64_t q_d = umma_desc_k128(smem_u32(q_s)), k_d = umma_desc_k128(smem_u32(k_s)), v_d = umma_desc_n128(smem_u32(v_s), C::K_BLOCK);
        auto wait = [&](uint64_t* bar, uint32_t parity, int code) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, code)); };
        auto scores = [&](int j) {
            const int st = j % C::KST;
            if (!wait(&k_full[st], (uint32_t)(j / C::KST) & 1u, DEV_ERR_FULL_WAIT)) return false;
            tc_fence_after();
            const uint32_t d = tmem + (j & 1) * TK;
            const uint64_t kd = k_d + (uint64_t)(uint32_t)(st * (C::TILE_BYTES >> 4));
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int b = 0; b < C::BLOCKS; ++b)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        umma_bf16_elect(d, q_d + (half * C::BLOCKS + b) * (C::Q_BLOCK >> 4) + 2 * i, kd + b * (C::K_BLOCK >> 4) + 2 * i, idesc_s,
                                        half > 0 || b > 0 || i > 0);
            umma_commit_elect(&s_full[j & 1]);
            umma_commit_elect(&k_empty[st]);
            return true;
        };
        pdl_wait();
        bool ok = tiles > 0 && wait(q_full, 0, DEV_ERR_FULL_WAIT) && scores(0);
        if (ok && tiles > 1) ok = scores(1);
        for (int j = 0; j < tiles && ok; ++j) {
            const int st = j % C::VST;
            ok = wait(&v_full[st], (uint32_t)(j / C::VST) & 1u, DEV_ERR_FULL_WAIT) && wait(&p_full[j & 1], (uint32_t)(j >> 1) & 1u, DEV_ERR_ACC_WAIT);
            if (!ok) break;
            tc_fence_after();
            const uint64_t vd = v_d + (uint64_t)(uint32_t)(st * (C::TILE_BYTES >> 4));
#pragma unroll
            for (int half = 0; half < 2; ++half)  // P hi, P lo
#pragma unroll
                for (int kk = 0; kk < TK / 16; ++kk)
                    umma_bf16_ts(tmem + C::COL_O, tmem + (j & 1) * TK + half * (TK / 2) + kk * 8, vd + kk * 128, idesc_o, j > 0 || half > 0 || kk > 0);
            umma_commit_elect(&v_empty[st]);
            umma_commit_elect(pv_done);
            if (j + 2 < tiles) ok = scores(j + 2);  // behind P V, whose P lies where this S goes
        }
    } else {
        // Rows t * part_heads + head; rows without a query and columns past the head are zero. A thread copies 8 columns of
        // every 16th (8th) row, the loads of eight rows in flight together.
        constexpr int PIECES = HD / 8, STEP = kRows / PIECES, BATCH = 8;
        const int c = tid % PIECES * 8;
        const float* q_row[kRows / STEP];
#pragma unroll
        for (int i = 0; i < kRows / STEP; ++i) {
            const int r = tid / PIECES + i * STEP, qt = r / p.part_heads, h = r % p.part_heads;
            q_row[i] = qt < ntok && h < nheads && c < p.kd ? p.q + ((size_t)(t0 + qt) * p.nh + kvh * p.G + head0 + h) * p.kd + c : nullptr;
        }
        const int tok = tid / p.part_heads, head = tid % p.part_heads;
        const bool active = tok < ntok && head < nheads;
        const int pos = first_pos + tok;
        const int end = active ? pos + 1 - key0 : 0, begin = active && p.chunk > 0 ? pos / p.chunk * p.chunk - key0 : 0;  // visible keys, from key0
        const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
        bool ok = true;
        // A small grid finds its instructions in no SM's cache. With one CTA per SM at most, the time until the previous kernel
        // is done goes into a rehearsal: the softmax warps take one tile of whatever tensor memory holds through their code,
        // without a barrier and without an output (128 tokens, 24 layers: 9.7 -> 7.9 us per launch).
#pragma unroll 1
        for (int pass = p.warm ? 0 : 1; pass < 2 && ok; ++pass) {
            const bool real = pass == 1;
            if (real) pdl_wait();
#pragma unroll
            for (int i0 = 0; i0 < kRows / STEP; i0 += BATCH) {
                float4 a[BATCH], b[BATCH];
#pragma unroll
                for (int i = 0; i < BATCH; ++i) {
                    a[i] = b[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (q_row[i0 + i]) {
                        a[i] = __ldcg((const float4*)q_row[i0 + i]);
                        b[i] = __ldcg((const float4*)q_row[i0 + i] + 1);
                    }
                }
#pragma unroll
                for (int i = 0; i < BATCH; ++i) {
                    const int r = tid / PIECES + (i0 + i) * STEP;
                    uint4 hi, lo;
                    split_bf16x2(a[i].x, a[i].y, hi.x, lo.x);
                    split_bf16x2(a[i].z, a[i].w, hi.y, lo.y);
                    split_bf16x2(b[i].x, b[i].y, hi.z, lo.z);
                    split_bf16x2(b[i].z, b[i].w, hi.w, lo.w);
                    uint8_t* dst = q_s + (c >> 6) * C::Q_BLOCK + r * 128 + ((((c & 63) >> 3) ^ (r & 7)) << 4);
                    *(uint4*)dst = hi;
                    *(uint4*)(dst + C::BLOCKS * C::Q_BLOCK) = lo;
                }
            }
            fence_proxy_async_smem();
            tc_fence_before();
            if (real) mbar_arrive(q_full);
            float m_ref = kNeg, l_sum = 0.f;
            const int n = real ? tiles : 1;
            for (int j = 0; j < n && ok; ++j) {
                if (real) ok = __all_sync(0xffffffffu, mbar_wait(&s_full[j & 1], (uint32_t)(j >> 1) & 1u, p.status, DEV_ERR_ACC_WAIT));
                if (!ok) break;
                tc_fence_after();
                const uint32_t buf = lane_addr + (j & 1) * TK;
                uint32_t s[TK / 16][16];
#pragma unroll
                for (int k = 0; k < TK / 16; ++k) tmem_ld16(buf + k * 16, s[k]);
                tc_wait_ld();
                float mx = kNeg;
                if (__all_sync(0xffffffffu, begin <= j * TK && end >= j * TK + TK)) {
#pragma unroll
                    for (int i = 0; i < TK; ++i) {
                        const float v = __uint_as_float(s[i >> 4][i & 15]) * p.scale_log2;
                        s[i >> 4][i & 15] = __float_as_uint(v);
                        mx = fmaxf(mx, v);
                    }
                } else {
                    const int lo = begin - j * TK, hi = end - j * TK;
#pragma unroll
                    for (int i = 0; i < TK; ++i) {
                        const float v = i >= lo && i < hi ? __uint_as_float(s[i >> 4][i & 15]) * p.scale_log2 : kNeg;
                        s[i >> 4][i & 15] = __float_as_uint(v);
                        mx = fmaxf(mx, v);
                    }
                }
                float corr = 1.f;
                bool moved = false;
                if (j == 0) {
                    m_ref = mx;
                } else if (mx > m_ref + 8.f) {
                    corr = exp2_fast(m_ref - mx);
                    m_ref = mx;
                    moved = true;
                }
                l_sum *= corr;
                const float m_sub = m_ref == kNeg ? 0.f : m_ref;  // nothing visible yet: all weights are zero
                uint32_t hi[TK / 32][16], lo[TK / 32][16];
#pragma unroll
                for (int i = 0; i < TK; i += 2) {
                    const float a = exp2_fast(__uint_as_float(s[i >> 4][i & 15]) - m_sub), b = exp2_fast(__uint_as_float(s[i >> 4][(i & 15) + 1]) - m_sub);
                    l_sum += a + b;
                    const __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
                    const uint32_t h = *(const uint32_t*)&h2;
                    const __nv_bfloat162 l2 = __floats2bfloat162_rn(a - bf16_lo(h), b - bf16_hi(h));
                    hi[i >> 5][(i & 31) >> 1] = h;
                    lo[i >> 5][(i & 31) >> 1] = *(const uint32_t*)&l2;
                }
                // O is still; every phase of the barrier is waited for, so that none is mistaken for the one before
                if (j > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(pv_done, (uint32_t)(j - 1) & 1u, p.status, DEV_ERR_ACC_WAIT));
                    if (!ok) break;
                    tc_fence_after();
                }
                if (__any_sync(0xffffffffu, moved)) {  // never with j == 0
#pragma unroll 1
                    for (int k = 0; k < HD / 16; ++k) {
                        uint32_t o[16];
                        tmem_ld16(lane_addr + C::COL_O + k * 16, o);
                        tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                        tmem_st16(lane_addr + C::COL_O + k * 16, o);
                    }
                }
#pragma unroll
                for (int k = 0; k < TK / 32; ++k) {
                    tmem_st16(buf + k * 16, hi[k]);
                    tmem_st16(buf + TK / 2 + k * 16, lo[k]);
                }
                tc_wait_st();
                if (real && j == tiles - 1 && (len - key0) % TK != 0) {
                    // rows of V past the end weigh zero, but what an earlier request left there may not be finite
                    const int st = j % C::VST, rows0 = (len - key0) % TK;
                    ok = __all_sync(0xffffffffu, mbar_wait(&v_full[st], (uint32_t)(j / C::VST) & 1u, p.status, DEV_ERR_FULL_WAIT));
                    if (!ok) break;
                    for (int r = rows0 + (tid >> 3); r < TK; r += kRows / 8)
#pragma unroll
                        for (int b = 0; b < C::BLOCKS; ++b)
                            *(uint4*)(v_s + st * C::TILE_BYTES + b * C::K_BLOCK + r * 128 + (tid & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                    fence_proxy_async_smem();
                }
                tc_fence_before();
                if (real) mbar_arrive(&p_full[j & 1]);
            }
            if (n > 0 && ok) {
                if (real) ok = __all_sync(0xffffffffu, mbar_wait(pv_done, (uint32_t)(tiles - 1) & 1u, p.status, DEV_ERR_ACC_WAIT));
                tc_fence_after();
                const bool out = active && real;
                const float inv = active ? 1.f / l_sum : 0.f;
                bf16* dst = p.ctx + (size_t)(t0 + (active ? tok : 0)) * (size_t)p.ctx_ld + (size_t)(kvh * p.G + head0 + head) * p.vdim;
                for (int k = 0; k < (p.vdim + 15) / 16 && ok; ++k) {
                    uint32_t o[16];
                    tmem_ld16(lane_addr + C::COL_O + k * 16, o);
                    tc_wait_ld();
                    if (out && p.vec) {
#pragma unroll
                        for (int i = 0; i < 16; i += 8) {
                            uint32_t w[4];
#pragma unroll
                            for (int x = 0; x < 4; ++x)
                                w[x] = (uint32_t)bf16_bits(__uint_as_float(o[i + 2 * x]) * inv) | ((uint32_t)bf16_bits(__uint_as_float(o[i + 2 * x + 1]) * inv) << 16);
                            if (k * 16 + i < p.vdim) *(uint4*)(dst + k * 16 + i) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    } else if (out) {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (k * 16 + i < p.vdim) dst[k * 16 + i] = __float2bfloat16_rn(__uint_as_float(o[i]) * inv);
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) tmem_dealloc(tmem, C::TMEM_COLS);
    if (tid == 0) tl_mark(p.tl, 2);
}

template <int HD>
cudaError_t prompt_attrs() {
    const cudaError_t e = cudaFuncSetAttribute(k_attn_prompt<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, PromptCfg<HD>::SMEM);
    return e == cudaSuccess ? prefer_max_shared(k_attn_prompt<HD>) : e;
}

}  // namespace

int attn_prompt_prepare() {
    const cudaError_t e = prompt_attrs<64>();
    return (int)(e == cudaSuccess ? prompt_attrs<128>() : e);
}

int launch_attention_prefill(const float* q, KvView kv, int layer, const int* tok_seq, const int* tok_pos, const int* grp_first,
                             const int* grp_count, int n_groups, bf16* ctx, int nh, int num_sms, int* status, TmapCache* tmaps, cudaStream_t s, bool pdl,
                             unsigned long long* tl, const AttnOptions& options, int key_spread) {
    const AttnOptions opt = resolve_attn_options(options, kv, nh);
    PromptDev p;
    memset(&p, 0, sizeof p);
    const uint64_t rows = (uint64_t)kv.num_pages * kv.nkv * kPageTokens;
    if (!make_tmap_2d(tmaps, &p.tmK, kv.k_pool + (size_t)layer * kv.layer_stride, rows, kv.hd, kv.hd, kPageTokens)) return -1000;
    if (!make_tmap_2d(tmaps, &p.tmV, kv.v_pool + (size_t)layer * kv.layer_stride, rows, kv.vd, kv.vd, kPageTokens)) return -1000;
    p.q = q;
    p.block_table = kv.block_table;
    p.max_pages_per_seq = kv.max_pages_per_seq;
    p.num_pages = kv.num_pages;
    p.nkv = kv.nkv;
    p.tok_seq = tok_seq;
    p.tok_pos = tok_pos;
    p.grp_first = grp_first;
    p.grp_count = grp_count;
    p.ctx = ctx;
    p.ctx_ld = opt.ctx_ld;
    p.nh = nh;
    p.G = nh / kv.nkv;
    p.part_heads = p.G < kRows ? p.G : kRows;
    p.parts = (p.G + p.part_heads - 1) / p.part_heads;
    p.kd = kv.hd;
    p.vdim = opt.vdim;
    p.chunk = opt.chunk;
    p.vec = opt.vdim % 8 == 0 && opt.ctx_ld % 8 == 0 && (uintptr_t)ctx % 16 == 0;
    p.scale_log2 = opt.scale * 1.4426950408889634f;
    p.status = status;
    p.tl = tl;
    const dim3 grid((unsigned)n_groups * kv.nkv * p.parts), block(kThreads);
    if (attention_prompt_waits(grid.x, num_sms, key_spread)) pdl = false;
    p.warm = pdl && grid.x <= (unsigned)num_sms;
    if (kv.hd <= 64 && kv.vd <= 64) return (int)launch_k(k_attn_prompt<64>, grid, block, (size_t)PromptCfg<64>::SMEM, s, pdl, p);
    if (kv.hd <= 128 && kv.vd <= 128) return (int)launch_k(k_attn_prompt<128>, grid, block, (size_t)PromptCfg<128>::SMEM, s, pdl, p);
    return (int)cudaErrorInvalidValue;
}

}  // namespace tffn
