// Softmax attention of head size 64 on CUDA cores, a 64 x 64 tile at a time: the kernels of attention_simt.cu, and what attention_split.cu falls
// back to where a result is not finite.
#pragma once
#include "device_utils.cuh"
#include "kernels.cuh"

// ---- head size 64: tiles of 64 queries x 64 keys ----
// One block per tile of queries (or keys) of a (batch, head), 256 threads, 4 x 4 results of every 64 x 64 x 64 product per
// thread.  Tiles sit in shared memory as FP32 rows of 65 words: a thread's four rows and four columns are 16 apart, so any
// product of two tiles, over the rows or the columns of either, reads without bank conflicts and no tile is kept twice.
// Shared-memory reads bound it (eight words per sixteen multiply-adds).  The row-per-warp kernels of attention_simt.cu read every key row
// from L2 for every query: FP32, 8 x 4 heads x 256 tokens, forward 210 -> 39 us, backward 513 -> 108 us.
constexpr int Side = 64, Pitch = 65, SideThreads = 256;
using SideTile = float[Side][Pitch];
template <class T> __device__ __forceinline__ void load_side(SideTile &tile, const T *rows, int64_t ld, int valid) {
    for (int i = threadIdx.x; i < Side * Side / 8; i += SideThreads) {
        const int r = i / 8, c = i % 8 * 8;
        float v[8] = {};
        if (r < valid)
            load8(rows + r * ld + c, v);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            tile[r][c + j] = v[j];
    }
}
// acc[i][j] += sum_k A(row i, k) B(row j, k); a tile read transposed gives A(row, k) = tile[k][row].  Diagonal: A holds
// queries x keys of the same 64 positions; its zeros above the diagonal are left out, since what they would multiply may be
// infinite.
template <bool TransposeA, bool TransposeB, bool Diagonal = false>
__device__ __forceinline__ void multiply_side(float (&acc)[4][4], const SideTile &a, const SideTile &b, int tx, int ty) {
#pragma unroll 8
    for (int k = 0; k < Side; ++k) {
        float av[4], bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            av[i] = TransposeA ? a[k][ty + 16 * i] : a[ty + 16 * i][k];
            bv[i] = TransposeB ? b[k][tx + 16 * i] : b[tx + 16 * i][k];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (!Diagonal || (TransposeA ? k >= ty + 16 * i : k <= ty + 16 * i))
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
}
__device__ __forceinline__ float row_max(float x) { // over the 16 threads that share rows
#pragma unroll
    for (int k = 8; k; k >>= 1)
        x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, k));
    return x;
}
__device__ __forceinline__ float row_sum(float x) {
#pragma unroll
    for (int k = 8; k; k >>= 1)
        x += __shfl_xor_sync(0xffffffffu, x, k);
    return x;
}
struct SideBlock { // which tile of which (batch, head) a block works on
    int tile, head, tx, ty;
    int64_t base, statistics; // first token of the sequence; first element of the (batch, head)'s row statistics
    __device__ __forceinline__ SideBlock(int index, int batch, int heads, int context)
        : tile(index / (batch * heads)), head(index % heads), tx(threadIdx.x % 16), ty(threadIdx.x / 16) {
        const int pair = index % (batch * heads);
        base = int64_t(pair / heads) * context, statistics = int64_t(pair) * context;
    }
};
template <class T> __device__ void side_forward(const SoftmaxAttentionArgs &a, SideTile *side_tiles, const SideBlock &block) { // four tiles
    SideTile &q = side_tiles[0], &k = side_tiles[1], &v = side_tiles[2], &p = side_tiles[3];
    const int tx = block.tx, ty = block.ty, q0 = block.tile * Side;
    const int64_t ld = 3 * a.width;
    const T *qkv = (const T *)a.qkv + block.base * ld + block.head * Side;
    load_side(q, qkv + q0 * ld, ld, a.context - q0);
    float high[4], sum[4] = {}, out[4][4] = {};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        high[i] = -CUDART_INF_F;
    for (int k0 = 0; k0 <= q0; k0 += Side) {
        __syncthreads();
        load_side(k, qkv + a.width + k0 * ld, ld, a.context - k0);
        load_side(v, qkv + 2 * a.width + k0 * ld, ld, a.context - k0);
        __syncthreads();
        float s[4][4] = {};
        multiply_side<false, false>(s, q, k, tx, ty);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float top = -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = k0 + tx + 16 * j <= q0 + ty + 16 * i ? s[i][j] * .125f : -CUDART_INF_F;
                top = fmaxf(top, s[i][j]);
            }
            top = fmaxf(high[i], row_max(top)); // finite: the tile's first key is at or before every query
            const float correction = expf(high[i] - top);
            high[i] = top;
            float part = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = expf(s[i][j] - top);
                part += e;
                p[ty + 16 * i][tx + 16 * j] = e;
                out[i][j] *= correction;
            }
            sum[i] = sum[i] * correction + row_sum(part);
        }
        __syncwarp(); // a warp's rows of p are its own
        if (k0 == q0)
            multiply_side<false, true, true>(out, p, v, tx, ty);
        else
            multiply_side<false, true>(out, p, v, tx, ty);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int query = q0 + ty + 16 * i;
        if (query >= a.context)
            break;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            ((T *)a.out)[(block.base + query) * a.width + block.head * Side + tx + 16 * j] = from_float<T>(out[i][j] / sum[i]);
        if (tx == 0)
            a.lse[block.statistics + query] = high[i] + logf(sum[i]);
    }
}
// Queries == true: dq of a tile of queries, over the keys at or before it; false: dk and dv of a tile of keys, over the
// queries at or after it.  P = exp(S - lse), dS = P (dO V^T - delta) / sqrt(d).  Bounded: lse may come from scores of other bits than these, and an
// exponential above one from their difference is one.
template <class T, bool Queries, bool Bounded = false>
__device__ void side_backward(const SoftmaxAttentionBackwardArgs &a, SideTile *side_tiles, const SideBlock &block) { // five tiles for queries, else six
    SideTile &q = side_tiles[0], &k = side_tiles[1], &v = side_tiles[2], &dy = side_tiles[3], &ds = side_tiles[4], &p = side_tiles[5];
    const int tx = block.tx, ty = block.ty, fixed = block.tile * Side;
    const int64_t ld = 3 * a.width;
    const T *qkv = (const T *)a.qkv + block.base * ld + block.head * Side, *dout = (const T *)a.dout + block.base * a.width + block.head * Side;
    auto load_queries = [&](int q0) {
        load_side(q, qkv + q0 * ld, ld, a.context - q0);
        load_side(dy, dout + int64_t(q0) * a.width, a.width, a.context - q0);
    };
    auto load_keys = [&](int k0) {
        load_side(k, qkv + a.width + k0 * ld, ld, a.context - k0);
        load_side(v, qkv + 2 * a.width + k0 * ld, ld, a.context - k0);
    };
    if (Queries)
        load_queries(fixed);
    else
        load_keys(fixed);
    float first[4][4] = {}, second[4][4] = {}; // dq, or dk and dv
    for (int moving = Queries ? 0 : fixed; Queries ? moving <= fixed : moving < a.context; moving += Side) {
        const int q0 = Queries ? fixed : moving, k0 = Queries ? moving : fixed;
        __syncthreads();
        if (Queries)
            load_keys(k0);
        else
            load_queries(q0);
        __syncthreads();
        float s[4][4] = {}, dp[4][4] = {};
        multiply_side<false, false>(s, q, k, tx, ty);
        multiply_side<false, false>(dp, dy, v, tx, ty);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int query = q0 + ty + 16 * i;
            const float lse = query < a.context ? a.lse[block.statistics + query] : 0.f, delta = query < a.context ? a.delta[block.statistics + query] : 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool seen = k0 + tx + 16 * j <= query && query < a.context;
                const float x = s[i][j] * .125f - lse, e = seen ? expf(Bounded && x > 0.f ? 0.f : x) : 0.f;
                ds[ty + 16 * i][tx + 16 * j] = seen ? e * (dp[i][j] - delta) * .125f : 0.f;
                if (!Queries)
                    p[ty + 16 * i][tx + 16 * j] = e;
            }
        }
        if (Queries) {
            __syncwarp();
            if (k0 == q0)
                multiply_side<false, true, true>(first, ds, k, tx, ty); // dq += ds k
            else
                multiply_side<false, true>(first, ds, k, tx, ty);
        } else {
            __syncthreads();
            if (k0 == q0) {
                multiply_side<true, true, true>(first, ds, q, tx, ty);  // dk += ds^T q
                multiply_side<true, true, true>(second, p, dy, tx, ty); // dv += p^T dy
            } else {
                multiply_side<true, true>(first, ds, q, tx, ty);
                multiply_side<true, true>(second, p, dy, tx, ty);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int token = fixed + ty + 16 * i;
        if (token >= a.context)
            break;
        T *out = (T *)a.dqkv + (block.base + token) * ld + block.head * Side + tx;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (Queries)
                out[16 * j] = from_float<T>(first[i][j]);
            else
                out[a.width + 16 * j] = from_float<T>(first[i][j]), out[2 * a.width + 16 * j] = from_float<T>(second[i][j]);
        }
    }
}
