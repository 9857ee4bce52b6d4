// Causal softmax attention of FP32 engines, head size 64, on the tensor cores: FP32 products as products of BF16 parts.
//
// Every operand is split into three BF16 parts and the six products of parts above 2^-24 are formed (see gemm_split.cu); the leading parts' sums
// never run over more than 32 terms before they are added in FP32.  Probabilities and their gradients are split in registers: the
// accumulator fragment of one m16n8k16 product is, packed, the operand fragment of the next.  (mma.sync and not tcgen05: the 16 x 32 pieces
// that a warp carries from product to product would each pass through tensor memory, and a sequence of 256 has four steps.)
//
// A block takes a tile of 64 queries (dK and dV: keys) and walks the other side in tiles of 64.  Eight warps: warp w owns rows
// 16 (w % 4) ... of the tile and half w / 4 of every other-side tile, with sums of its own, so that nothing but the tiles' loads is
// shared until the two halves are added at the end.
//
// What bounds it: the chain of a step (loads, split, 96 to 192 products a warp one after another, exponentials).  8 x 4 heads x 256 tokens,
// the CUDA cores' kernels and these: forward 34 -> 16.5 us, backward 8 + 69 + 55 -> 41 in one launch (beside weight gradients).
//
// A tile with a result that is not finite is computed once more by the CUDA cores' code: products of parts of an infinity are NaN, and a
// masked zero must not meet one.
#include "attention_side.cuh"
#include "sm100.cuh"

using namespace sm100;

namespace {
constexpr int PartBytes = Side * Side * 2, TileBytes = 3 * PartBytes; // [part][row][64 columns], 16-byte pieces swizzled by row
constexpr int Rows = 16, Half = Side / 2, Frags = Half / 8;           // of a warp: rows, columns of the other side, 8-column fragments
constexpr int PartialPitch = Side + 4;
constexpr int StatisticsAt = 4 * TileBytes, SplitShared = 6 * int(sizeof(SideTile)); // q, k, v, dO tiles; lse and delta of a query tile
static_assert(StatisticsAt + 2 * Side * 4 <= SplitShared && 2 * 4 * Rows * PartialPitch * 4 <= StatisticsAt, "");

using Fragment = float[4];

struct Loaded { // a thread's share of a 64 x 64 tile on its way
    float4 v[4];
    __device__ __forceinline__ void load(const float *rows, int64_t ld, int valid) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = threadIdx.x + SideThreads * c, row = i / 16;
            v[c] = row < valid ? *reinterpret_cast<const float4 *>(rows + row * ld + i % 16 * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ void split(uint32_t tile) const {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = threadIdx.x + SideThreads * c, row = i / 16, quad = i % 16;
            const uint32_t at = tile + row * 128 + ((quad / 2 ^ (row & 7)) << 4) + quad % 2 * 8;
            uint64_t rest[2] = {float_pair(v[c].x, v[c].y), float_pair(v[c].z, v[c].w)};
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                uint32_t packed[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float lo, hi;
                    split_pair(rest[j], lo, hi);
                    packed[j] = pack_bf16(lo, hi);
                    rest[j] = fma_pair(float_pair(__uint_as_float(packed[j] << 16), __uint_as_float(packed[j] & 0xffff0000u)), float_pair(-1.f, -1.f), rest[j]);
                }
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + part * PartBytes), "r"(packed[0]), "r"(packed[1]) : "memory");
            }
        }
    }
};

__device__ __forceinline__ void load_matrices(uint32_t address, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address) : "memory");
}
__device__ __forceinline__ void load_matrices_transposed(uint32_t address, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address) : "memory");
}
__device__ __forceinline__ uint32_t piece(uint32_t tile, int row, int column16) { return tile + row * 128 + ((column16 ^ (row & 7)) << 4); }

// Six products of parts into the leading parts' sums and the others'.  Mirrored: in the order that gives the bits of the transposed product.
template <bool Mirrored = false>
__device__ __forceinline__ void multiply_parts(Fragment &lead, Fragment &rest, const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int n) {
    auto multiply = [&](Fragment &d, int i, int j) {
        if (Mirrored)
            mma_bf16(d[0], d[1], d[2], d[3], a[j], b[i][2 * n], b[i][2 * n + 1]);
        else
            mma_bf16(d[0], d[1], d[2], d[3], a[i], b[j][2 * n], b[j][2 * n + 1]);
    };
    multiply(lead, 0, 0);
    multiply(rest, 0, 1);
    multiply(rest, 1, 0);
    multiply(rest, 1, 1);
    multiply(rest, 0, 2);
    multiply(rest, 2, 0);
}
// out[16 rows x 32] = A's rows from `row` on times B's rows from `column` on, transposed, over the 64 columns of both.
template <bool Mirrored = false> __device__ __forceinline__ void multiply_rows(Fragment (&out)[Frags], uint32_t a_tile, int row, uint32_t b_tile, int column, int lane) {
#pragma unroll
    for (int n = 0; n < Frags / 2; ++n) {
        Fragment lead[2][2] = {}, rest[2] = {}; // of either half of K; of both
#pragma unroll
        for (int k = 0; k < Side / 16; ++k) {
            uint32_t a[3][4], b[3][4];
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                load_matrices(piece(a_tile + part * PartBytes, row + ((lane >> 3) & 1) * 8 + (lane & 7), k * 2 + (lane >> 4)), a[part]);
                load_matrices(piece(b_tile + part * PartBytes, column + n * 16 + (lane >> 4) * 8 + (lane & 7), k * 2 + ((lane >> 3) & 1)), b[part]);
            }
            multiply_parts<Mirrored>(lead[k / 2][0], rest[0], a, b, 0);
            multiply_parts<Mirrored>(lead[k / 2][1], rest[1], a, b, 1);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                out[2 * n + h][i] = (lead[0][h][i] + lead[1][h][i]) + rest[h][i];
    }
}
// 16 rows x 32 columns as they leave a product or a function of it, split, as the left operand of two 16-deep steps.
struct Left {
    uint32_t a[2][3][4];
    __device__ __forceinline__ explicit Left(const Fragment (&v)[Frags]) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) { // rows g and g + 8 of one fragment, then of the next
                uint64_t rest = float_pair(v[2 * k + i / 2][i % 2 * 2], v[2 * k + i / 2][i % 2 * 2 + 1]);
#pragma unroll
                for (int part = 0; part < 3; ++part) {
                    float lo, hi;
                    split_pair(rest, lo, hi);
                    const uint32_t packed = a[k][part][i] = pack_bf16(lo, hi);
                    rest = fma_pair(float_pair(__uint_as_float(packed << 16), __uint_as_float(packed & 0xffff0000u)), float_pair(-1.f, -1.f), rest);
                }
            }
    }
};
// out[16 x 64] += left times the 32 rows of B from `row` on.
__device__ __forceinline__ void multiply_columns(Fragment (&out)[Side / 8], const Left &left, uint32_t b_tile, int row, int lane) {
#pragma unroll
    for (int n = 0; n < Side / 16; ++n) {
        Fragment lead[2] = {}, rest[2] = {};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            uint32_t b[3][4];
#pragma unroll
            for (int part = 0; part < 3; ++part)
                load_matrices_transposed(piece(b_tile + part * PartBytes, row + k * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), n * 2 + (lane >> 4)), b[part]);
            multiply_parts(lead[0], rest[0], left.a[k], b, 0);
            multiply_parts(lead[1], rest[1], left.a[k], b, 1);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                out[2 * n + h][i] += lead[h][i] + rest[h][i];
    }
}
__device__ __forceinline__ float quad_max(float x) {
    x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
    return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
__device__ __forceinline__ float quad_sum(float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x + __shfl_xor_sync(0xffffffffu, x, 2);
}
// A warp's 16 x 64 sums to or from the memory that its counterpart of the other half reads.
__device__ __forceinline__ float2 *partial_at(float *partial, int own, int row, int f, int t) {
    return reinterpret_cast<float2 *>(partial + (own * Rows + row) * PartialPitch + f * 8 + 2 * t);
}
__device__ __forceinline__ void put_partial(float *partial, int own, const Fragment (&v)[Side / 8], int g, int t) {
#pragma unroll
    for (int f = 0; f < Side / 8; ++f)
#pragma unroll
        for (int r = 0; r < 2; ++r)
            *partial_at(partial, own, g + 8 * r, f, t) = make_float2(v[f][2 * r], v[f][2 * r + 1]);
}

__global__ void __launch_bounds__(SideThreads, 1) attention_split_forward_kernel(SoftmaxAttentionArgs a) {
    extern __shared__ __align__(1024) uint8_t shared[];
    const SideBlock block(gridDim.x - 1 - blockIdx.x, a.batch, a.heads, a.context); // the longest first
    const uint32_t q_tile = smem_address(shared), k_tile = q_tile + TileBytes, v_tile = k_tile + TileBytes;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, t = lane % 4, own = warp % 4, half = warp / 4;
    const int q0 = block.tile * Side, query = q0 + own * Rows + g; // and eight further
    const int64_t ld = 3 * a.width;
    const float *qkv = (const float *)a.qkv + block.base * ld + block.head * Side;
    Loaded x, y;
    x.load(qkv + q0 * ld, ld, a.context - q0);
    x.split(q_tile);
    Fragment out[Side / 8] = {};
    float high[2] = {-CUDART_INF_F, -CUDART_INF_F}, sum[2] = {0.f, 0.f};
    for (int k0 = 0; k0 <= q0; k0 += Side) {
        x.load(qkv + a.width + k0 * ld, ld, a.context - k0);
        y.load(qkv + 2 * a.width + k0 * ld, ld, a.context - k0);
        __syncthreads(); // the tiles before these have been read
        x.split(k_tile);
        y.split(v_tile);
        __syncthreads();
        Fragment s[Frags];
        multiply_rows(s, q_tile, own * Rows, k_tile, half * Half, lane);
        float top[2] = {high[0], high[1]};
#pragma unroll
        for (int f = 0; f < Frags; ++f)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int key = k0 + half * Half + f * 8 + 2 * t + i % 2;
                s[f][i] = key <= query + i / 2 * 8 ? s[f][i] * .125f : -CUDART_INF_F;
                top[i / 2] = fmaxf(top[i / 2], s[f][i]);
            }
        float part[2] = {0.f, 0.f}, correction[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            top[r] = quad_max(top[r]);
            const float base = top[r] == -CUDART_INF_F ? 0.f : top[r]; // the row may have no key in this half yet
            correction[r] = expf(high[r] - base);
            high[r] = top[r];
            top[r] = base;
        }
#pragma unroll
        for (int f = 0; f < Frags; ++f)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[f][i] = expf(s[f][i] - top[i / 2]);
                part[i / 2] += s[f][i];
            }
#pragma unroll
        for (int r = 0; r < 2; ++r)
            sum[r] = sum[r] * correction[r] + quad_sum(part[r]);
#pragma unroll
        for (int f = 0; f < Side / 8; ++f)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                out[f][i] *= correction[i / 2];
        multiply_columns(out, Left(s), v_tile, half * Half, lane);
    }
    __syncthreads(); // the tiles become the other half's sums
    float *partial = reinterpret_cast<float *>(shared);
    float2 *rows = reinterpret_cast<float2 *>(shared + StatisticsAt); // maximum and sum of a row
    if (half) {
        put_partial(partial, own, out, g, t);
        if (t == 0)
#pragma unroll
            for (int r = 0; r < 2; ++r)
                rows[own * Rows + g + 8 * r] = make_float2(high[r], sum[r]);
    }
    __syncthreads();
    bool finite = true;
    if (!half) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int at = query + 8 * r;
            if (at >= a.context)
                continue;
            const float2 other = rows[own * Rows + g + 8 * r];
            const float top = fmaxf(high[r], other.x), mine = expf(high[r] - top), theirs = expf(other.x - top);
            const float total = sum[r] * mine + other.y * theirs;
            float *row = (float *)a.out + (block.base + at) * a.width + block.head * Side;
#pragma unroll
            for (int f = 0; f < Side / 8; ++f) {
                const float2 o = *partial_at(partial, own, g + 8 * r, f, t);
                const float2 v = make_float2((out[f][2 * r] * mine + o.x * theirs) / total, (out[f][2 * r + 1] * mine + o.y * theirs) / total);
                finite = finite && isfinite(v.x) && isfinite(v.y);
                *reinterpret_cast<float2 *>(row + f * 8 + 2 * t) = v;
            }
            const float lse = top + logf(total);
            finite = finite && isfinite(lse);
            if (t == 0)
                a.lse[block.statistics + at] = lse;
        }
    }
    if (!__syncthreads_and(finite))
        side_forward<float>(a, reinterpret_cast<SideTile *>(shared), block);
}

// dq of a tile of queries, or dk and dv of a tile of keys.
template <bool Queries> __device__ __forceinline__ void split_backward(const SoftmaxAttentionBackwardArgs &a, uint8_t *shared, const SideBlock &block) {
    const uint32_t q_tile = smem_address(shared), k_tile = q_tile + TileBytes, v_tile = k_tile + TileBytes, dy_tile = v_tile + TileBytes;
    float *lse_of = reinterpret_cast<float *>(shared + StatisticsAt), *delta_of = lse_of + Side; // of the query tile in shared memory
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, t = lane % 4, own = warp % 4, half = warp / 4;
    const int fixed = block.tile * Side;
    const int64_t ld = 3 * a.width;
    const float *qkv = (const float *)a.qkv + block.base * ld + block.head * Side, *dout = (const float *)a.dout + block.base * a.width + block.head * Side,
                *out = (const float *)a.out + block.base * a.width + block.head * Side;
    Loaded x, y;
    float delta, lse;
    auto load_queries = [&](int q0) {
        x.load(qkv + q0 * ld, ld, a.context - q0);
        y.load(dout + int64_t(q0) * a.width, a.width, a.context - q0);
        // delta = sum of dO O: four threads a row
        const int row = threadIdx.x / 4;
        delta = lse = 0.f;
        if (q0 + row < a.context) {
            const int64_t at = int64_t(q0 + row) * a.width + threadIdx.x % 4 * 16;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float4 d = *reinterpret_cast<const float4 *>(dout + at + 4 * c), o = *reinterpret_cast<const float4 *>(out + at + 4 * c);
                delta += (d.x * o.x + d.y * o.y) + (d.z * o.z + d.w * o.w);
            }
            lse = a.lse[block.statistics + q0 + row];
        }
        delta = quad_sum(delta);
    };
    auto load_keys = [&](int k0) {
        x.load(qkv + a.width + k0 * ld, ld, a.context - k0);
        y.load(qkv + 2 * a.width + k0 * ld, ld, a.context - k0);
    };
    auto put_queries = [&] {
        x.split(q_tile);
        y.split(dy_tile);
        if (threadIdx.x % 4 == 0)
            lse_of[threadIdx.x / 4] = lse, delta_of[threadIdx.x / 4] = delta;
    };
    auto put_keys = [&] {
        x.split(k_tile);
        y.split(v_tile);
    };
    if (Queries) {
        load_queries(fixed);
        put_queries();
    } else {
        load_keys(fixed);
        put_keys();
    }
    Fragment first[Side / 8] = {}, second[Queries ? 1 : Side / 8] = {}; // dq, or dk and dv
    for (int moving = Queries ? 0 : fixed; Queries ? moving <= fixed : moving < a.context; moving += Side) {
        if (Queries)
            load_keys(moving);
        else
            load_queries(moving);
        __syncthreads();
        if (Queries)
            put_keys();
        else
            put_queries();
        __syncthreads();
        const int q0 = Queries ? fixed : moving, k0 = Queries ? moving : fixed;
        Fragment s[Frags], dp[Frags]; // rows: the tile's own; columns: the other side's
        // The scores to the bit of the forward pass: where their last place is large, exp(s - lse) is one for the same bits only.
        multiply_rows<!Queries>(s, Queries ? q_tile : k_tile, own * Rows, Queries ? k_tile : q_tile, half * Half, lane);
        multiply_rows(dp, Queries ? dy_tile : v_tile, own * Rows, Queries ? v_tile : dy_tile, half * Half, lane);
#pragma unroll
        for (int f = 0; f < Frags; ++f)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = own * Rows + g + i / 2 * 8, column = half * Half + f * 8 + 2 * t + i % 2;
                const int in_queries = Queries ? row : column, query = q0 + in_queries, key = k0 + (Queries ? column : row);
                const bool seen = key <= query && query < a.context;
                const float e = seen ? expf(s[f][i] * .125f - lse_of[in_queries]) : 0.f;
                dp[f][i] = seen ? e * (dp[f][i] - delta_of[in_queries]) * .125f : 0.f;
                s[f][i] = e;
            }
        multiply_columns(first, Left(dp), Queries ? k_tile : q_tile, half * Half, lane);
        if constexpr (!Queries)
            multiply_columns(second, Left(s), dy_tile, half * Half, lane);
    }
    __syncthreads(); // the tiles become the other half's sums
    float *partial = reinterpret_cast<float *>(shared), *partial2 = partial + 4 * Rows * PartialPitch;
    if (half) {
        put_partial(partial, own, first, g, t);
        if constexpr (!Queries)
            put_partial(partial2, own, second, g, t);
    }
    __syncthreads();
    bool finite = true;
    if (!half) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int token = fixed + own * Rows + g + 8 * r;
            if (token >= a.context)
                continue;
            float *row = (float *)a.dqkv + (block.base + token) * ld + block.head * Side + 2 * t;
            auto store = [&](const Fragment &mine, const float2 &theirs, float *to) {
                const float2 v = make_float2(mine[2 * r] + theirs.x, mine[2 * r + 1] + theirs.y);
                finite = finite && isfinite(v.x) && isfinite(v.y);
                *reinterpret_cast<float2 *>(to) = v;
            };
#pragma unroll
            for (int f = 0; f < Side / 8; ++f) {
                store(first[f], *partial_at(partial, own, g + 8 * r, f, t), row + (Queries ? 0 : a.width) + f * 8);
                if constexpr (!Queries)
                    store(second[f], *partial_at(partial2, own, g + 8 * r, f, t), row + 2 * a.width + f * 8);
            }
        }
    }
    if (__syncthreads_and(finite))
        return;
    // delta as the CUDA cores' code wants it: of every query it will read.  Whole warps go round: a query's four lanes add up through a shuffle of all 32.
    for (int first = 0; first < a.context; first += SideThreads / 4) {
        const int i = first + threadIdx.x / 4;
        float total = 0.f;
        for (int c = threadIdx.x % 4; i < a.context && c < Side; c += 4)
            total += dout[int64_t(i) * a.width + c] * out[int64_t(i) * a.width + c];
        total = quad_sum(total);
        if (i < a.context && threadIdx.x % 4 == 0)
            a.delta[block.statistics + i] = total; // the same value from every block that comes here
    }
    __syncthreads();
    side_backward<float, Queries, true>(a, reinterpret_cast<SideTile *>(shared), block);
}
// Blocks of either kind in turn, the longest first.
__global__ void __launch_bounds__(SideThreads, 1) attention_split_backward_kernel(SoftmaxAttentionBackwardArgs a) {
    extern __shared__ __align__(1024) uint8_t shared[];
    const int tiles = gridDim.x / 2, index = blockIdx.x / 2;
    if (blockIdx.x % 2)
        split_backward<true>(a, shared, SideBlock(tiles - 1 - index, a.batch, a.heads, a.context));
    else
        split_backward<false>(a, shared, SideBlock(index, a.batch, a.heads, a.context));
}

template <class Args> void launch(void (*kernel)(Args), const Args &a, int passes, cudaStream_t s) {
    CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitShared));
    kernel<<<passes * a.batch * a.heads * ((a.context + Side - 1) / Side), SideThreads, SplitShared, s>>>(a);
}
} // namespace

bool attention_split_supported(int width, int heads) { return width == heads * Side; }
void launch_attention_split_forward(const SoftmaxAttentionArgs &a, cudaStream_t s) { launch(attention_split_forward_kernel, a, 1, s); }
void launch_attention_split_backward(const SoftmaxAttentionBackwardArgs &a, cudaStream_t s) { launch(attention_split_backward_kernel, a, 2, s); }
