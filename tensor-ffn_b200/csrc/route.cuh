// The choice of experts for one token by one warp, shared by the stand-alone router kernel and the row kernel that
// routes in the same pass.
#pragma once
#include "act.cuh"
#include "ptx.cuh"
#include <cfloat>

namespace tffn {

// s[0 .. n): the token's logits in shared memory, n = experts + identity (overwritten with the softmax scores);
// choice[0 .. n): scratch, with bins afterwards the rows of the pairs. The lanes own strided entries.
__device__ __forceinline__ void route_token(const MoeRoute& a, int t, float* s, float* choice, int lane) {
    const int n = a.experts + a.identity;
    float mx = -INFINITY;
    for (int i = lane; i < n; i += 32) mx = fmaxf(mx, s[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
    for (int i = lane; i < n; i += 32) {
        const float e = expf(s[i] - mx);
        s[i] = e;
        sum += e;
    }
    const float inv = 1.f / warp_sum(sum);
    auto put = [&](int j, int bi) {  // place within the expert; the choices' atomics are in flight together
        int2 p = make_int2(-1, 0);
        if (bi < a.experts) p = make_int2(bi, atomicAdd(a.counts + bi, 1));
        a.pair[(size_t)t * a.top + j] = p;
        a.pair_w[(size_t)t * a.top + j] = s[bi];
        if (a.bin > 0) {
            const int row = p.x < 0 ? -1 : p.x * a.bin + p.y;
            a.pair_row[(size_t)t * a.top + j] = row;
            ((int*)choice)[j] = row;
        }
    };
    // What can be chosen is at least -FLT_MAX (a correction of -inf retires an entry; NaN inputs), what has been chosen is -inf: a token
    // never chooses an entry twice, so an expert has at most T rows, as many as a bin holds.
    auto score = [&](int i) { return fmaxf(s[i] + __ldg(a.correction + i), -FLT_MAX); };
    if (n <= 32) {
        // a lane per entry: its rank is the number of entries chosen before it (larger, or equal and earlier)
        float c = -INFINITY;
        if (lane < n) {
            s[lane] *= inv;
            c = score(lane);
        }
        int rank = 0;
        for (int j = 0; j < n; ++j) {
            const float o = __shfl_sync(0xffffffffu, c, j);
            rank += o > c || (o == c && j < lane) ? 1 : 0;
        }
        __syncwarp();
        if (lane < n && rank < a.top) put(rank, lane);
        return;
    }
    for (int i = lane; i < n; i += 32) {
        s[i] *= inv;
        choice[i] = score(i);
    }
    int mine[2] = {-1, -1};  // lane j keeps choices j and 32 + j (top <= 64)
    for (int j = 0; j < a.top; ++j) {
        float best = -INFINITY;
        int bi = 0x7fffffff;
        for (int i = lane; i < n; i += 32)
            if (choice[i] > best) { best = choice[i]; bi = i; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if ((bi & 31) == lane) choice[bi] = -INFINITY;
        if ((j & 31) == lane) mine[j >> 5] = bi;
    }
    __syncwarp();  // every lane's scores are visible
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int j = k * 32 + lane;
        if (j < a.top) put(j, mine[k]);
    }
}

}  // namespace tffn
