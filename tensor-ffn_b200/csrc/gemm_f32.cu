// The batched path's matrix products in true fp32: out[t, n] = epilogue(sum_k X[t,k] * W[n,k]) with fp32 activations,
// bf16 weights widened exactly, fp32 FMA on the CUDA cores, the same call structure as the tensor-core GEMM
// (gemm_tc.cu) so that a session that computes in fp32 runs the same sequence of steps. Two kernels:
//
// k_gemm_f32_rows, up to eight tokens, bound by streaming the weights: the threads of a block divide K (16 bytes of a weight
//   row each) for up to eight rows, and the sums meet in shuffles and shared memory. Blocks walk over groups of rows; the weights
//   of the next pieces are on their way into shared memory, the first ones requested ahead of the dependency wait.
// k_gemm_f32, more tokens: one CTA = 64 tokens x 64 weight rows, 8 x 8 outputs per thread (four 16-byte
//   shared loads and eight splats per 32 packed FMA, which bound it: the products of a prompt of 450 rows, 8 layers 896 wide, run at 18.5
//   TFLOP/s where a stream of FMA sustains 46 to 68); the four 64-thread groups of a CTA take a quarter of every K slice each, so that one tile
//   fills an SM's schedulers. Slices are double-buffered through registers. Where the tiles are fewer than the SMs, K is also
//   split over a thread-block cluster whose CTAs add their tiles through distributed shared memory in rank order.
#include "kernels.h"
#include "ptx.cuh"
#include "launch.h"
#include <cstring>

namespace tffn {

namespace {

constexpr int TB = kGemmF32Tile, NB = 64, KB = 32;
constexpr int kThreads = 256, kGroups = 4, kGroupK = KB / kGroups;
constexpr int kLd = 68;       // floats of a slice's row in shared memory (64 and a pad; 16-byte aligned)
constexpr int kMaxSplits = 8; // portable cluster size
constexpr int kRowTokens = 8;
constexpr int rows_per_thread(int tokens) { return tokens > 2 ? 4 : 8; }  // 32 sums at most

struct F32Dev {
    const float* X[2];
    const bf16* W[2];
    float* out[2];
    long long ldx[2], ldw[2], ldo;
    int N, T, K[2], mode, batch, x_batch, out_batch;
    float out_scale, alpha;
    const GroupTile* grp;
    int splits;   // k_gemm_f32: CTAs of a cluster
    int lanes;    // k_gemm_f32_rows: threads that divide K
    unsigned long long* tl;
};

// where a block works: tokens [t0, t_end), its rows of W, its columns of X
struct Place {
    int t0, t_end, op0, b;
    long long w_row0;
    float* out;
};
__device__ __forceinline__ bool place(const F32Dev& p, int tile, int prob, Place& x) {
    x.t0 = tile * TB;
    x.t_end = min(p.T, x.t0 + TB);
    x.w_row0 = 0;
    if (p.grp) {
        const int4 g = __ldcg((const int4*)(p.grp + tile));
        if (g.x < 0) return false;
        x.t0 = g.y;
        x.t_end = min(g.z, g.y + TB);
        x.w_row0 = (long long)g.x * p.N;
    }
    x.b = p.batch > 1 ? prob : 0;  // batched: the problems share their operands
    if (x.b > 0) x.w_row0 = (long long)x.b * p.N;
    x.op0 = p.batch > 1 ? 0 : prob;
    x.out = p.batch > 1 ? p.out[0] + (size_t)x.b * p.out_batch : p.out[prob];
    return true;
}
__device__ __forceinline__ float finish(const F32Dev& p, float first, float v) {
    if (p.K[1] > 0) v = p.mode == GEMM_SWIGLU ? first / (1.f + expf(-first)) * v : first + p.alpha * v;
    v *= p.out_scale;
    if (p.mode == GEMM_RELU2) {
        v = fmaxf(v, 0.f);
        v *= v;
    }
    return v;
}

// ------------------------------------------------------------------------------------------- few tokens
// the first `live` of a word's two bf16 values, the others zero
__device__ __forceinline__ uint32_t keep_low(uint32_t u, int live) { return live >= 2 ? u : live == 1 ? u & 0xffffu : 0u; }

// Sums of v[0 .. COUNT) (COUNT a power of two, at most 32) over the warp by halving exchange: lane l returns that of value l % COUNT.
template <int COUNT>
__device__ __forceinline__ float warp_sums(float (&v)[COUNT], int lane) {
#pragma unroll
    for (int o = 16, n = COUNT; o > 0; o >>= 1) {
        if (n > 1) {
            // the lanes with bit (n / 2) of their number keep the upper half of the values, their partners the lower
            n >>= 1;
            const int x = n;  // exchange distance: the values left are those of lane % n
#pragma unroll
            for (int i = 0; i < COUNT / 2; ++i) {
                if (i >= n) break;
                const bool up = lane & x;
                const float give = up ? v[i] : v[i + n];
                v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, give, x);
            }
        }
    }
    float r = v[0];
#pragma unroll
    for (int o = 16; o >= COUNT; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}

// p.lanes threads (8 .. 256, a power of two) divide K in pieces of 8; the block's kThreads / lanes teams take
// rows_per_thread weight rows each. TT tokens at a time (the rows' weights are read again, from L2, for the next TT).
// A thread's next DEPTH pieces are on their way into shared memory of its own (no barrier), 96 KB a block: the bytes in flight bound
// it, and one piece ahead in registers was too few. ONE: K is one piece of every thread and both pairs read the same X, which then
// stays in registers for all row groups. Inside a step of three sequences, 8 layers 896 wide, us: gate|up 16.8 -> 9.4, out and down
// 12.5 -> 7.7, LM head (32 768 rows) 41 -> 23; the step 633 -> 375.
constexpr int rows_depth(int tokens) { return 24 / rows_per_thread(tokens); }
constexpr size_t rows_smem(int tokens) { return (size_t)rows_depth(tokens) * rows_per_thread(tokens) * kThreads * 16; }
template <int TT, bool ONE>
__global__ void __launch_bounds__(kThreads, 2) k_gemm_f32_rows(const F32Dev p) {
    constexpr int R = rows_per_thread(TT), SUMS = R * TT, DEPTH = rows_depth(TT);
    extern __shared__ __align__(16) uint8_t ring_raw[];  // [DEPTH][R][kThreads] pieces of 16 bytes
    __shared__ float part[2][kThreads / 32][SUMS];  // per warp; a sum's readers are done before the one after next is written
    if (threadIdx.x == 0) tl_mark(p.tl, 0);
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, team = tid / p.lanes, kl = tid % p.lanes, teams = kThreads / p.lanes;
    const int group_rows = teams * R, groups = (p.N + group_rows - 1) / group_rows, pairs = p.K[1] > 0 ? 2 : 1;
    const int steps_of[2] = {(p.K[0] + p.lanes * 8 - 1) / (p.lanes * 8), (p.K[1] + p.lanes * 8 - 1) / (p.lanes * 8)};
    uint4* const ring = (uint4*)ring_raw + tid;
    Place at{};
    // what a block works through: row groups, operand pairs, pieces of K
    struct Piece {
        int group, pair, step;
    };
    const Piece start{(int)blockIdx.x, 0, 0};
    auto next = [&](Piece x) {
        if (++x.step < (x.pair ? steps_of[1] : steps_of[0])) return x;
        x.step = 0;
        if (++x.pair < pairs) return x;
        x.pair = 0;
        x.group += gridDim.x;
        return x;
    };
    auto request = [&](const Piece& x, int slot) {  // rows and columns that do not exist become zeros
        const int k = (x.step * p.lanes + kl) * 8, n0 = x.group * group_rows + team * R, op = at.op0 + x.pair;
        const bool k_on = x.group < groups && k < p.K[x.pair];
        const bf16* W = p.W[op] + (size_t)(at.w_row0 + n0) * p.ldw[op] + k;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool on = k_on && n0 + r < p.N;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(ring + (slot * R + r) * kThreads)),
                         "l"(on ? W + (size_t)r * p.ldw[op] : p.W[op]), "r"(on ? 16 : 0)
                         : "memory");
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    Piece ahead = start;
    auto fill = [&] {
        ahead = start;
        for (int i = 0; i < DEPTH; ++i) {
            request(ahead, i);
            commit();
            ahead = next(ahead);
        }
    };
    // ungrouped weights are older than the previous kernel, and so are all but its own outputs
    if (!p.grp) {
        place(p, blockIdx.y, blockIdx.z, at);
        fill();
    }
    pdl_wait();
    if (tid == 0) tl_mark(p.tl, 1);
    if (p.grp) {
        if (!place(p, blockIdx.y, blockIdx.z, at)) return;
        fill();
    }
    int half = 0;
    for (int t0 = at.t0; t0 < at.t_end; t0 += TT) {
        if (t0 > at.t0) fill();  // the next tokens start over
        float acc[SUMS], first = 0.f;
#pragma unroll
        for (int i = 0; i < SUMS; ++i) acc[i] = 0.f;
        // columns k .. k + 7 of token t0 + t; what a row's padding holds counts as zero
        auto load_x = [&](int op, int t, int k, int live, float (&v)[8]) {
            const float* xp = p.X[op] + (size_t)at.b * p.x_batch + k + (size_t)min(t0 + t, at.t_end - 1) * p.ldx[op];
            *(float4*)v = live > 0 ? __ldcg((const float4*)xp) : make_float4(0.f, 0.f, 0.f, 0.f);
            *(float4*)(v + 4) = live > 4 ? __ldcg((const float4*)(xp + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (live < 8) {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = j < live ? v[j] : 0.f;
            }
        };
        float kept[ONE ? TT : 1][8];
        if constexpr (ONE) {
#pragma unroll
            for (int t = 0; t < TT; ++t) load_x(at.op0, t, kl * 8, p.K[0] - kl * 8, kept[t]);
        }
        int slot = 0;
        for (Piece x = start; x.group < groups; x = next(x)) {
            const int K = p.K[x.pair], k = (x.step * p.lanes + kl) * 8, live = K - k;  // columns of this piece
            asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
            if (live > 0) {
                uint4 w[R];
#pragma unroll
                for (int r = 0; r < R; ++r) w[r] = ring[(slot * R + r) * kThreads];
                if (live < 8) {  // what a row's padding holds counts as zero
#pragma unroll
                    for (int r = 0; r < R; ++r) w[r] = make_uint4(keep_low(w[r].x, live), keep_low(w[r].y, live - 2), keep_low(w[r].z, live - 4), keep_low(w[r].w, live - 6));
                }
#pragma unroll
                for (int t = 0; t < TT; ++t) {
                    float xv[8];
                    if constexpr (ONE) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) xv[j] = kept[t][j];
                    } else {
                        load_x(at.op0 + x.pair, t, k, live, xv);
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const uint32_t u[4] = {w[r].x, w[r].y, w[r].z, w[r].w};
                        float a = acc[r * TT + t];
#pragma unroll
                        for (int j = 0; j < 4; ++j) a = fmaf(xv[2 * j + 1], bf16_hi(u[j]), fmaf(xv[2 * j], bf16_lo(u[j]), a));
                        acc[r * TT + t] = a;
                    }
                }
            }
            request(ahead, slot);
            commit();
            ahead = next(ahead);
            if (++slot == DEPTH) slot = 0;
            if (x.step + 1 == (x.pair ? steps_of[1] : steps_of[0])) {  // the pair's sums
                const int n0 = x.group * group_rows + team * R;
                auto store = [&](int i, float v) {
                    const int n = n0 + i / TT, t = t0 + i % TT;
                    if (n < p.N && t < at.t_end) at.out[(size_t)t * p.ldo + n] = finish(p, first, v);
                };
                if (p.lanes < 32) {  // one pair: every lane of the team gets the sums
                    for (int o = p.lanes >> 1; o > 0; o >>= 1)
#pragma unroll
                        for (int i = 0; i < SUMS; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
#pragma unroll
                    for (int i = 0; i < SUMS; ++i)
                        if (i % p.lanes == kl) store(i, acc[i]);
                } else {
                    const float mine = warp_sums<SUMS>(acc, lane);
                    half ^= 1;
                    if (lane < SUMS) part[half][tid >> 5][lane] = mine;
                    __syncthreads();
                    if (kl < SUMS) {
                        const int warp0 = team * (p.lanes / 32);
                        float v = 0.f;
                        for (int q = 0; q < p.lanes / 32; ++q) v += part[half][warp0 + q][kl];
                        if (x.pair + 1 < pairs) first = v;
                        else store(kl, v);
                    }
                }
#pragma unroll
                for (int i = 0; i < SUMS; ++i) acc[i] = 0.f;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    if (tid == 0) tl_mark(p.tl, 2);
}

// ------------------------------------------------------------------------------------------- more tokens
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 splat2(float x) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
// VEC: 16-byte copies (rows of X and W aligned, see launch_gemm_f32); else element by element.
template <bool VEC>
__global__ void __launch_bounds__(kThreads) k_gemm_f32(const F32Dev p) {
    __shared__ __align__(16) float smem[2 * 2 * KB * kLd];  // two slices of X and W, transposed; then the tile [64][kLd]
    if (threadIdx.x == 0) tl_mark(p.tl, 0);
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x == 0) tl_mark(p.tl, 1);
    const int tid = threadIdx.x;
    const int rank = (int)blockIdx.x % p.splits, n0 = (int)blockIdx.x / p.splits * NB;
    Place at;
    if (!place(p, blockIdx.y, blockIdx.z, at)) return;  // the whole cluster
    const int grp = tid >> 6, g = tid & 63, tx = g & 7, ty = g >> 3;  // tx: weight rows 4 tx and 32 + 4 tx .., ty: tokens alike
    const int cr = tid >> 2, ck = (tid & 3) * 8;                      // copies: row, first of 8 columns
    float first[16];
    const int pairs = p.K[1] > 0 ? 2 : 1;
    for (int pair = 0; pair < pairs; ++pair) {
        const int op = at.op0 + pair, K = p.K[pair];
        const bool t_on = at.t0 + cr < at.t_end, n_on = n0 + cr < p.N;
        const float* X = p.X[op] + (size_t)at.b * p.x_batch + (size_t)(t_on ? at.t0 + cr : at.t0) * p.ldx[op];
        const bf16* W = p.W[op] + (size_t)(at.w_row0 + (n_on ? n0 + cr : 0)) * p.ldw[op];
        const int slices = (K + KB - 1) / KB, per = (slices + p.splits - 1) / p.splits;
        const int s0 = rank * per, s1 = min(slices, s0 + per);
        float xr[8], wr[8];
        auto fetch = [&](int s) {
            const int k = s * KB + ck;
            if (VEC && k + 8 <= K) {
                const float4 a = t_on ? __ldcg((const float4*)(X + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 b = t_on ? __ldcg((const float4*)(X + k + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
                const uint4 u = n_on ? __ldg((const uint4*)(W + k)) : make_uint4(0, 0, 0, 0);
                xr[0] = a.x; xr[1] = a.y; xr[2] = a.z; xr[3] = a.w;
                xr[4] = b.x; xr[5] = b.y; xr[6] = b.z; xr[7] = b.w;
                const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) { wr[2 * j] = bf16_lo(w[j]); wr[2 * j + 1] = bf16_hi(w[j]); }
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    xr[j] = t_on && k + j < K ? __ldcg(X + k + j) : 0.f;
                    wr[j] = n_on && k + j < K ? __bfloat162float(W[k + j]) : 0.f;
                }
            }
        };
        f32x2 acc[8][4];  // pairs of neighbouring weight rows: packed FMA
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
        if (s0 < s1) fetch(s0);
        for (int s = s0; s < s1; ++s) {
            float* sx = smem + ((s - s0) & 1) * (2 * KB * kLd);
            float* sw = sx + KB * kLd;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                sx[(ck + j) * kLd + cr] = xr[j];
                sw[(ck + j) * kLd + cr] = wr[j];
            }
            __syncthreads();  // one barrier per slice: the buffer of slice s - 1 is written again only behind the next one
            if (s + 1 < s1) fetch(s + 1);
#pragma unroll
            for (int kk = 0; kk < kGroupK; ++kk) {
                const float* xk = sx + (grp * kGroupK + kk) * kLd;
                const float* wk = sw + (grp * kGroupK + kk) * kLd;
                float a[8];
                *(float4*)a = *(const float4*)(xk + 4 * ty);
                *(float4*)(a + 4) = *(const float4*)(xk + 32 + 4 * ty);
                const ulonglong2 b0 = *(const ulonglong2*)(wk + 4 * tx), b1 = *(const ulonglong2*)(wk + 32 + 4 * tx);
                const f32x2 b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const f32x2 aa = splat2(a[i]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fma2(aa, b[j], acc[i][j]);
                }
            }
        }
        // the groups' quarters, in order, then the cluster's parts
#pragma unroll 1
        for (int q = 0; q < kGroups; ++q) {
            __syncthreads();
            if (grp != q) continue;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float4* dst = (float4*)(smem + ((i >> 2) * 32 + 4 * ty + (i & 3)) * kLd + h * 32 + 4 * tx);
                    const float2 lo = unpack2(acc[i][2 * h]), hi = unpack2(acc[i][2 * h + 1]);
                    float4 v = make_float4(lo.x, lo.y, hi.x, hi.y);
                    if (q > 0) {
                        const float4 o = *dst;
                        v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
                    }
                    *dst = v;
                }
        }
        if (p.splits > 1) cluster_sync_all();
        else __syncthreads();
        // thread: 4 columns from 4 (tid % 16) of rows tid / 16 + 16 i; of a cluster's tile every CTA finishes some rows
        const uint32_t plane = smem_u32(smem);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = (tid >> 4) + 16 * i, c = 4 * (tid & 15), t = at.t0 + row;
            if (row % p.splits != rank || t >= at.t_end) continue;
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (p.splits == 1) {
                *(float4*)v = *(const float4*)(smem + row * kLd + c);
            } else {
                for (int z = 0; z < p.splits; ++z) {
                    const uint32_t src = map_shared_rank(plane + (uint32_t)(row * kLd + c) * 4, (uint32_t)z);
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] += ld_shared_cluster_f32(src + 4 * j);
                }
            }
            if (pair == 0 && pairs == 2) {
#pragma unroll
                for (int j = 0; j < 4; ++j) first[4 * i + j] = v[j];
                continue;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n0 + c + j < p.N) at.out[(size_t)t * p.ldo + n0 + c + j] = finish(p, pairs == 2 ? first[4 * i + j] : 0.f, v[j]);
        }
        if (p.splits > 1) cluster_sync_all();  // the peers have read this CTA's tile
        else __syncthreads();
    }
    if (tid == 0) tl_mark(p.tl, 2);
}

}  // namespace

int gemm_f32_prepare() {
    cudaError_t e = cudaSuccess;
    auto prep = [&](auto kern, int tokens) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_smem(tokens));
        if (e == cudaSuccess) e = prefer_max_shared(kern);
    };
    prep(k_gemm_f32_rows<1, true>, 1), prep(k_gemm_f32_rows<2, true>, 2), prep(k_gemm_f32_rows<4, true>, 4);
    prep(k_gemm_f32_rows<1, false>, 1), prep(k_gemm_f32_rows<2, false>, 2), prep(k_gemm_f32_rows<4, false>, 4), prep(k_gemm_f32_rows<8, false>, 8);
    return (int)e;
}

int launch_gemm_f32(const GemmCall& c, const GemmWorkspace& ws, cudaStream_t stream) {
    if (c.T <= 0 || c.N <= 0 || c.op[0].K <= 0 || !c.out) return (int)cudaErrorInvalidValue;
    if (c.mode != GEMM_STORE_F32 && c.mode != GEMM_STORE_BF16 && c.mode != GEMM_RELU2 && c.mode != GEMM_SWIGLU) return (int)cudaErrorInvalidValue;
    if (c.mode == GEMM_SWIGLU ? c.op[1].K != c.op[0].K : c.mode == GEMM_RELU2 && c.op[1].K > 0) return (int)cudaErrorInvalidValue;
    if (c.op[1].K > 0 && (c.out2 || c.grp || c.batch > 1)) return (int)cudaErrorInvalidValue;
    if (c.batch > 1 && (c.out2 || c.grp || (c.mode != GEMM_STORE_F32 && c.mode != GEMM_STORE_BF16))) return (int)cudaErrorInvalidValue;
    if (c.out2 && (c.op2[0].K != c.op[0].K || c.op2[1].K > 0 || c.grp)) return (int)cudaErrorInvalidValue;
    if (c.grp && (c.grp_bn != TB || c.grp_tiles < 1)) return (int)cudaErrorInvalidValue;
    F32Dev p;
    memset(&p, 0, sizeof p);
    p.X[0] = (const float*)c.op[0].X;
    p.W[0] = c.op[0].W;
    p.ldx[0] = c.op[0].ldx;
    p.ldw[0] = c.op[0].ldw;
    p.out[0] = (float*)c.out;
    if (c.op[1].K > 0) {
        p.X[1] = (const float*)c.op[1].X;
        p.W[1] = c.op[1].W;
        p.ldx[1] = c.op[1].ldx;
        p.ldw[1] = c.op[1].ldw;
    }
    if (c.out2) {
        p.X[1] = (const float*)c.op2[0].X;
        p.W[1] = c.op2[0].W;
        p.ldx[1] = c.op2[0].ldx;
        p.ldw[1] = c.op2[0].ldw;
        p.out[1] = (float*)c.out2;
    }
    p.ldo = c.ldo;
    p.N = c.N;
    p.T = c.T;
    p.K[0] = c.op[0].K;
    p.K[1] = c.op[1].K;
    p.alpha = c.alpha;
    p.batch = c.batch > 1 ? c.batch : 1;
    p.x_batch = c.x_batch;
    p.out_batch = c.out_batch;
    p.mode = c.mode;
    p.out_scale = c.out_scale == 0.f ? 1.f : c.out_scale;
    p.grp = c.grp;
    p.tl = c.tl;
    // 16-byte copies need every row of X and W to start on a 16-byte boundary
    bool vec = c.x_batch % 4 == 0;
    for (int i = 0; i < 2; ++i)
        if (p.X[i] && ((uintptr_t)p.X[i] % 16 || (uintptr_t)p.W[i] % 16 || p.ldx[i] % 4 || p.ldw[i] % 8)) vec = false;
    const int probs = c.out2 ? 2 : p.batch, t_tiles = c.grp ? c.grp_tiles : (c.T + TB - 1) / TB;
    // A tile of 64 tokens costs the same for one as for 64; streaming the rows costs as much again for every eight. Groups go by
    // their average, rounded up to leave room (a group of more rows reads its weights again,
    // from L2). 16 experts, 896 x 1 792, four a token, us a launch: 4 pairs 13 -> 7, 8 pairs 41 -> 11; in tiles of 64: 16 pairs 110 -> 18.
    const int live_tiles = !c.grp ? t_tiles : c.grp_rows_hint > 0 && c.grp_rows_hint < t_tiles ? c.grp_rows_hint : t_tiles;
    const int avg = c.grp ? (c.T + live_tiles - 1) / live_tiles : c.T, at_once = c.grp && avg < c.T ? 2 * avg : avg;
    if (vec && at_once <= kRowTokens) {
        const int K = p.K[0] > p.K[1] ? p.K[0] : p.K[1], tokens = at_once <= 2 ? at_once : at_once <= 4 ? 4 : kRowTokens;
        p.lanes = p.K[1] > 0 ? 32 : 8;
        while (p.lanes < kThreads && p.lanes * 8 < K) p.lanes *= 2;
        const int rows = kThreads / p.lanes * rows_per_thread(tokens), groups = (c.N + rows - 1) / rows;
        // two blocks per SM; more groups than that are walked over, so that their weights are requested ahead
        const int most = (2 * ws.num_sms + live_tiles * probs - 1) / (live_tiles * probs);
        const dim3 grid(groups <= most ? groups : most, t_tiles, probs);
        auto go = [&](auto kern) { return (int)launch_k(kern, grid, dim3(kThreads), rows_smem(tokens), stream, c.pdl, p); };
        if (K <= p.lanes * 8 && (p.K[1] <= 0 || (p.K[1] == p.K[0] && p.X[1] == p.X[0] && p.ldx[1] == p.ldx[0])) && tokens <= 4)
            return tokens == 1 ? go(k_gemm_f32_rows<1, true>) : tokens == 2 ? go(k_gemm_f32_rows<2, true>) : go(k_gemm_f32_rows<4, true>);
        return tokens == 1 ? go(k_gemm_f32_rows<1, false>) : tokens == 2 ? go(k_gemm_f32_rows<2, false>) : tokens == 4 ? go(k_gemm_f32_rows<4, false>) : go(k_gemm_f32_rows<8, false>);
    }
    // splits until the chip is full once, at least four slices each
    const long long tiles = (long long)((c.N + NB - 1) / NB) * t_tiles * probs;
    const int slices = (p.K[0] + KB - 1) / KB;
    p.splits = 1;
    while (p.splits < kMaxSplits && tiles * p.splits * 2 <= 2 * ws.num_sms && slices >= 8 * p.splits) p.splits *= 2;
    const dim3 grid((c.N + NB - 1) / NB * p.splits, t_tiles, probs);
    auto go = [&](auto kern) { return (int)launch_k_cluster(kern, grid, dim3(kThreads), dim3(p.splits, 1, 1), 0, stream, c.pdl, p); };
    return vec ? go(k_gemm_f32<true>) : go(k_gemm_f32<false>);
}

}  // namespace tffn
