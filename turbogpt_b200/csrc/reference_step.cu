// Forward and backward pass of the reference architecture (width 16, four arg-max heads of size 4, SwiGLU 48,
// RMSNorm, untied 256-way head; reference cuda/model.cuh:7-99) in one kernel per step.
//
// What bounds it: a token's whole step is 52 k multiply-adds over matrices of 16 columns, so as separate
// kernels (one per operator, ~150 launches) a step is launch latency and half-empty tiles: 1.43 ms at depth 4,
// context 4, batch 2880, and 0.86 ms at batch 16 (now 49 and 30 us with reduction and update: the latency of the chain of
// dependent products).  Here a block takes whole sequences (up to 128 tokens) through
// every layer and back: each warp keeps its 16 tokens' residual stream in registers, the weights sit in shared
// memory once, and only k and v (forward) and the attention gradients (backward) pass between warps.
//
// Matrix products are mma.sync m16n8k16: K is 16 or 48 and a warp's accumulator fragment of one product is,
// packed to BF16, the operand fragment of the next, so a chain of products never leaves the registers.
// (A tcgen05 product would send each 16-wide intermediate through tensor memory and back.)  The rows of the
// qkv matrix and the columns of the attention projection are permuted when they are copied to shared memory, so that
// the lane which holds row r, fragment column t holds head t's four dimensions: attention is per-lane work.
//
// Activations kept for backward: x, middle (as fragments), the winning key and score of every (token, head);
// everything else is recomputed from them with the forward's roundings.  Weight gradients: the warps stage dy and x of
// a layer in shared memory, then share the layer's 16 x 16 gradient tiles, each summed over the block's tokens by one
// warp; a block's sums go to its own row of `partial`, and reduce_gradients_kernel adds the rows in block order.  All
// sums have a fixed order: the same bits on every run.
#include "device_utils.cuh"
#include "kernels.cuh"
#include "sm100.cuh"
#include <algorithm>

using namespace sm100;

namespace {
constexpr int Width = 16, Heads = 4, Hidden = 48;
constexpr int StepWarps = 16, StepThreads = StepWarps * 32;
constexpr int HeadTiles = Vocabulary / 16 / StepWarps; // 16-column groups of logits per warp
constexpr int MaxRows = 128, MaxRowTiles = MaxRows / 16; // tokens of one block's tile: 16 per warp
constexpr int LayerParameters = 4 * Width * Width + 3 * Hidden * Width + 2 * Width;
constexpr int OffQkv = Width, OffAttention = OffQkv + 3 * Width * Width, OffMlpNorm = OffAttention + Width * Width,
              OffGate = OffMlpNorm + Width, OffDown = OffGate + 2 * Hidden * Width; // inside a layer; gate and up are adjacent
constexpr int Layer0 = Vocabulary * Width;   // after the embedding

// Shared memory.  Weights are panels of 16 columns (32-byte rows, the two 16-byte halves swapped in every second
// group of four rows so that ldmatrix, plain or transposed, is free of bank conflicts); staged tensors have
// pitches of an odd number of 16-byte units for the same reason.
constexpr int RowsQkv = 0, RowsAttention = 48, RowsWide = 64, RowsDown = 160, LayerRows = 208; // down: 3 panels of 16 rows
constexpr int PitchWide = 208, PitchHidden = 112, PitchQkv = 112, PitchWidth = 48, PitchLogits = 528;
constexpr int StageBytesPerRow = PitchWide + PitchHidden + PitchQkv + 5 * PitchWidth;
constexpr int MaxShared = 232448;
constexpr int TeamRows = 48; // rows of the largest tile whose owners have helpers: see below
struct StepShared {
    int weights, scales, rope, bytes, saved_x, saved_middle, saved_top, selected, exchange, dy, dt_gate, norm_sums, row_sums, stage, total;
    bool overlap; // two stages: a layer's weight gradients are taken by the warps without rows while the others are at the next layer
    __host__ __device__ StepShared(int depth, int rows, int context) {
        int at = 0;
        auto take = [&](int n) {
            const int here = at;
            at += (n + 15) / 16 * 16;
            return here;
        };
        weights = take((depth * LayerRows + Vocabulary) * 32);
        scales = take((2 * depth + 1) * Width * 4);
        rope = take(context * 8);
        bytes = take(2 * rows);
        saved_x = take(depth * rows * 32);
        saved_middle = take(depth * rows * 32);
        saved_top = take(depth * rows * Heads * 4);
        selected = take(depth * rows * Heads);
        exchange = take(rows * PitchQkv);
        dy = take(rows * 32);
        dt_gate = take(rows * Heads * 8);
        norm_sums = take(StepWarps * 2 * Width * 4); // of every second layer in its second half: at most eight warps own rows
        row_sums = take(rows * StepWarps * 8);
        stage = take(rows * StageBytesPerRow);
        // up to three row tiles seven warps or more have no part in them
        overlap = rows <= TeamRows && at + rows * StageBytesPerRow <= MaxShared;
        if (overlap)
            take(rows * StageBytesPerRow);
        total = at;
    }
};

struct StepParams {
    const uint8_t *data; // resident corpus to sample from, or nullptr: x and y hold the batch
    int64_t data_size;
    uint64_t seed;
    const uint8_t *x, *y;
    const StepCounters *counters;
    const bf16 *weight_high;
    const uint16_t *weight_low;
    const float2 *rope; // [context] cos and sin of the position in radians
    float *partial;     // [blocks][partial_stride]
    float *token_losses;
    int64_t partial_stride;
    int batch, context, depth, sequences, rows, tiles;
    float gradient_scale;
    ReferenceActivations saved;
};

__device__ __forceinline__ void load_matrices(uint32_t address, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address) : "memory");
}
__device__ __forceinline__ void load_matrices_transposed(uint32_t address, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address) : "memory");
}
template <int Bytes> __device__ __forceinline__ void copy_async(uint32_t to, const void *from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(from), "n"(Bytes) : "memory");
}
__device__ __forceinline__ uint32_t panel_address(uint32_t base, int row, int half) {
    return base + row * 32 + ((half ^ ((row >> 2) & 1)) << 4);
}

// A warp's 16 tokens x 16 columns: lane (g = lane / 4, t = lane % 4) holds rows g and g + 8, columns 2t, 2t+1, 8+2t, 9+2t,
// as the two m16n8 accumulators of a product: v[0..1] row g, v[2..3] row g + 8 (columns 2t), v[4..7] likewise (8 + 2t).
using Tile = float[8];
__device__ __forceinline__ void pack_tile(const Tile &v, uint32_t (&a)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        a[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
}
__device__ __forceinline__ void unpack_tile(const uint4 &u, Tile &v) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        v[2 * i] = __uint_as_float(w[i] << 16), v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
}
// Both values of a pair as BF16 stores them: one conversion and two bit operations.
__device__ __forceinline__ void round_pair(float &a, float &b) {
    const uint32_t u = pack_bf16(a, b);
    a = __uint_as_float(u << 16), b = __uint_as_float(u & 0xffff0000u);
}
__device__ __forceinline__ void round_tile(Tile &v) {
#pragma unroll
    for (int i = 0; i < 8; i += 2)
        round_pair(v[i], v[i + 1]);
}
// 1 / (1 + e^-x) without the exact division's branches, which cost the step a third of its time (37 -> 48 us at 64 tokens,
// 52 -> 61 at 11520): e^-|x| keeps the denominator in [1, 2], where the reciprocal instruction (1 ulp) and one Newton-Raphson
// step serve.  Over all BF16 x the error is 1.3 x 2^-23 at most (1.1 with the division), and x / (1 + e^-x) rounds to the
// same BF16 value from -80 on (below -88.7 the division underflows to 0, this does not).
__device__ __forceinline__ float fast_sigmoid(float x) {
    const float e = expf(-fabsf(x)), denominator = 1.f + e;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(denominator));
    r = fmaf(r, fmaf(-denominator, r, 1.f), r);
    return x < 0.f ? e * r : r;
}
// The residual stream after a branch: both rounded, as a product's own rounding and the sum's.
__device__ __forceinline__ void add_branch(Tile &x, Tile &branch) {
    round_tile(branch);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        x[i] += branch[i];
    round_tile(x);
}
// y (+)= a W^T for sixteen rows of W starting at `row` of the panel (K = 16).
__device__ __forceinline__ void multiply(Tile &y, const uint32_t (&a)[4], uint32_t panel, int row, int lane) {
    uint32_t b[4];
    load_matrices(panel_address(panel, row + (lane >> 4) * 8 + (lane & 7), (lane >> 3) & 1), b);
    mma_bf16(y[0], y[1], y[2], y[3], a, b[0], b[1]);
    mma_bf16(y[4], y[5], y[6], y[7], a, b[2], b[3]);
}
// y (+)= a W for sixteen rows of W (the contraction) starting at `row`: the sixteen columns of the panel come out.
__device__ __forceinline__ void multiply_transposed(Tile &y, const uint32_t (&a)[4], uint32_t panel, int row, int lane) {
    uint32_t b[4];
    load_matrices_transposed(panel_address(panel, row + ((lane >> 3) & 1) * 8 + (lane & 7), lane >> 4), b);
    mma_bf16(y[0], y[1], y[2], y[3], a, b[0], b[1]);
    mma_bf16(y[4], y[5], y[6], y[7], a, b[2], b[3]);
}
__device__ __forceinline__ float quad_sum(float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x + __shfl_xor_sync(0xffffffffu, x, 2);
}
__device__ __forceinline__ float quad_max(float x) {
    x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
    return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
struct Scale { // the lane's four columns of a norm's FP32 scale
    float w[4];
    __device__ __forceinline__ Scale(const float *s, int t) {
        const float2 a = *reinterpret_cast<const float2 *>(s + 2 * t), b = *reinterpret_cast<const float2 *>(s + 8 + 2 * t);
        w[0] = a.x, w[1] = a.y, w[2] = b.x, w[3] = b.y;
    }
    __device__ __forceinline__ float of(int i) const { return w[(i >> 2) * 2 + (i & 1)]; }
};
__device__ __forceinline__ void inverse_rms(const Tile &x, float (&inv)[2]) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float s = (x[2 * r] * x[2 * r] + x[2 * r + 1] * x[2 * r + 1]) + (x[4 + 2 * r] * x[4 + 2 * r] + x[5 + 2 * r] * x[5 + 2 * r]);
        inv[r] = rsqrtf(quad_sum(s) / Width + 1e-6f);
    }
}
__device__ __forceinline__ void rms_norm(const Tile &x, const Scale &scale, Tile &y) {
    float inv[2];
    inverse_rms(x, inv);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        y[i] = x[i] * inv[(i >> 1) & 1] * scale.of(i);
    round_tile(y);
}
// dx = round(norm'(dy)), plus `residual` and another rounding when given; the column sums of dy z over the warp's tokens
// go to sums[16] (rows past the end hold zero gradients).
__device__ __forceinline__ void rms_norm_backward(const Tile &x, const Tile &dy, const Scale &scale, const Tile *residual, Tile &dx,
                                                  float *sums, int lane) {
    float inv[2], dot[2] = {0.f, 0.f}, column[4];
    inverse_rms(x, inv);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        dot[(i >> 1) & 1] += dy[i] * scale.of(i) * (x[i] * inv[(i >> 1) & 1]);
#pragma unroll
    for (int r = 0; r < 2; ++r)
        dot[r] = quad_sum(dot[r]) / Width;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int i = (c >> 1) * 4 + (c & 1);
        column[c] = dy[i] * (x[i] * inv[0]) + dy[i + 2] * (x[i + 2] * inv[1]);
    }
#pragma unroll
    for (int k = 4; k < 32; k *= 2)
#pragma unroll
        for (int c = 0; c < 4; ++c)
            column[c] += __shfl_xor_sync(0xffffffffu, column[c], k);
    if (lane < 4)
#pragma unroll
        for (int c = 0; c < 4; ++c)
            sums[(c >> 1) * 8 + 2 * lane + (c & 1)] = column[c];
    Tile value;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = (i >> 1) & 1;
        value[i] = (dy[i] * scale.of(i) - x[i] * inv[r] * dot[r]) * inv[r];
    }
    round_tile(value);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        dx[i] = residual ? (*residual)[i] + value[i] : value[i];
    if (residual)
        round_tile(dx);
}
// Fragment columns to a [row][column] array in memory (shared or global), natural column order.
__device__ __forceinline__ void put_tile(void *rows, int64_t pitch, const Tile &v, int g, int t) {
    char *p = static_cast<char *>(rows) + g * pitch + 4 * t;
    *reinterpret_cast<uint32_t *>(p) = pack_bf16(v[0], v[1]);
    *reinterpret_cast<uint32_t *>(p + 8 * pitch) = pack_bf16(v[2], v[3]);
    *reinterpret_cast<uint32_t *>(p + 16) = pack_bf16(v[4], v[5]);
    *reinterpret_cast<uint32_t *>(p + 8 * pitch + 16) = pack_bf16(v[6], v[7]);
}
__device__ __forceinline__ void get_tile(const void *rows, int64_t pitch, Tile &v, int g, int t) {
    const char *p = static_cast<const char *>(rows) + g * pitch + 4 * t;
    unpack_tile(make_uint4(*reinterpret_cast<const uint32_t *>(p), *reinterpret_cast<const uint32_t *>(p + 8 * pitch),
                           *reinterpret_cast<const uint32_t *>(p + 16), *reinterpret_cast<const uint32_t *>(p + 8 * pitch + 16)), v);
}
// The same for a tile whose lane holds columns 4t .. 4t+3 (a head): v[0], v[1], v[4], v[5] of row g.
__device__ __forceinline__ void put_heads(void *rows, int64_t pitch, const Tile &v, int g, int t) {
    char *p = static_cast<char *>(rows) + g * pitch + 8 * t;
    *reinterpret_cast<uint2 *>(p) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[4], v[5]));
    *reinterpret_cast<uint2 *>(p + 8 * pitch) = make_uint2(pack_bf16(v[2], v[3]), pack_bf16(v[6], v[7]));
}
// Tokens past the end of the batch are not written to global memory.
__device__ __forceinline__ void save_tile(void *base, int columns, int first_column, bool heads, const Tile &v, int64_t token, int valid,
                                          int g, int t) {
    bf16 *p = static_cast<bf16 *>(base) + token * columns + first_column;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (g + 8 * r >= valid)
            continue;
        bf16 *row = p + int64_t(g + 8 * r) * columns;
        *reinterpret_cast<uint32_t *>(row + (heads ? 4 * t : 2 * t)) = pack_bf16(v[2 * r], v[2 * r + 1]);
        *reinterpret_cast<uint32_t *>(row + (heads ? 4 * t + 2 : 8 + 2 * t)) = pack_bf16(v[4 + 2 * r], v[5 + 2 * r]);
    }
}
struct Four {
    float v[4];
};
// From shared memory.  Written out so that a load never waits for a condition on its use: as plain loads the compiler put them
// behind the condition, and the gradients' gather loop took 1730 clocks instead of 950 (680 in pairs).
__device__ __forceinline__ Four load_four(const void *p) {
    uint2 u;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(u.x), "=r"(u.y) : "r"(smem_address(p)) : "memory");
    return {{__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u)}};
}
__device__ __forceinline__ float2 load_pair(const void *p) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(smem_address(p)) : "memory");
    return v;
}
__device__ __forceinline__ int load_byte(const void *p) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(smem_address(p)) : "memory");
    return int(v);
}
__device__ __forceinline__ float dot_four(const Four &a, const Four &b) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        s += a.v[c] * b.v[c];
    return s;
}
// The first two dimensions of every head turn `position` radians; products unfused (see rope_kernel).
__device__ __forceinline__ void rotate(float &x, float &y, float2 cs) {
    const float a = x, b = y;
    x = __fsub_rn(__fmul_rn(a, cs.x), __fmul_rn(b, cs.y));
    y = __fadd_rn(__fmul_rn(a, cs.y), __fmul_rn(b, cs.x));
    round_pair(x, y);
}

// A 16 x 16 block of gradient sums to memory, rows of `columns` floats.
__device__ __forceinline__ void add_gradient(float *out, int columns, const Tile &acc, bool accumulate, int lane) {
    out += lane / 4 * columns + lane % 4 * 2;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 *p = reinterpret_cast<float2 *>(out + i % 2 * 8 * columns + i / 2 * 8);
        float2 v = make_float2(acc[2 * i], acc[2 * i + 1]);
        if (accumulate)
            v.x += p->x, v.y += p->y;
        *p = v;
    }
}
// SwiGLU with the forward's roundings: gate and up projections in, the activation in `up`.
__device__ __forceinline__ void activate(Tile &gate, Tile &up) {
    round_tile(gate);
    round_tile(up);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        gate[i] *= fast_sigmoid(gate[i]);
    round_tile(gate);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        up[i] *= gate[i];
    round_tile(up);
}
// Its gradient (see swiglu_backward_kernel): gate and up become their gradients, not yet rounded; the activation is recomputed.
__device__ __forceinline__ void activate_backward(Tile &gate, Tile &up, Tile &dout, Tile &activated) {
    round_tile(gate);
    round_tile(up);
    round_tile(dout);
    Tile silu, da, sig;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        sig[i] = fast_sigmoid(gate[i]), silu[i] = gate[i] * sig[i], da[i] = dout[i] * up[i];
    round_tile(silu);
    round_tile(da);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        activated[i] = silu[i] * up[i];
        gate[i] = da[i] * sig[i] * (1.f + gate[i] * (1.f - sig[i]));
        up[i] = dout[i] * silu[i];
    }
}

// out[16, 16] (+)= dy^T x over the block's rows: two staged [row][column] arrays, from their columns `dy` and `x` on.
__device__ __forceinline__ void weight_gradient(float *out, int columns, uint32_t dy, int dy_pitch, uint32_t x, int x_pitch, int rows,
                                                bool accumulate, int lane) {
    Tile acc = {};
    dy += ((lane >> 4) * 8 + (lane & 7)) * dy_pitch + ((lane >> 3) & 1) * 16;
    x += (((lane >> 3) & 1) * 8 + (lane & 7)) * x_pitch + (lane >> 4) * 16;
#pragma unroll 2
    for (int k = 0; k < rows; k += 16) {
        uint32_t a[4], b[4];
        load_matrices_transposed(dy + k * dy_pitch, a);
        load_matrices_transposed(x + k * x_pitch, b);
        mma_bf16(acc[0], acc[1], acc[2], acc[3], a, b[0], b[1]);
        mma_bf16(acc[4], acc[5], acc[6], acc[7], a, b[2], b[3]);
    }
    add_gradient(out, columns, acc, accumulate, lane);
}

// A tile's 16 rows belong to one warp, its owner.  In tiles of up to TeamRows rows two other warps help each owner and take a third
// of its products each (of the MLP's columns, of q, k and v), which otherwise follow one another in one warp, a chain of dependent
// instructions that leaves the SM idle; the warps that are left take the weight gradients of a layer beside the next one, where a
// second stage fits (1184 sequences of 4 tokens 37.2 and 36.0 us, 600 of 8 at depth 8 62.1 and 59.8).  Where the
// line lies, us a step without and with: 16 rows, depth 4 35.8 and 30.9; 32 rows, context 4 40.2 and 36.4, depth 16 239 and 214;
// 48 rows, context 4 41.3 and 39.2, depth 8 64.2 and 60.2; 64 rows, context 16 47.3 and 48.1, context 64 68.1 and 71.1; 80 rows,
// where one warp is left for the gradients, 49.5 and 60.8.
// What a helper hands over are factors, never a part of a sum: the owner multiplies them into its one accumulator in the order of
// the columns, so that no bit depends on the tile.
struct Share { // [from, to) of the three 16-column groups that a warp takes: of the MLP, and of q, k and v going forward
    int from, to;
};
// Of q, k and v when they are recomputed going back, while the owner is at the norm and the attention projection.
__device__ __forceinline__ Share qkv_back_share_of(int member) { return member == 0 ? Share{0, 0} : member == 1 ? Share{0, 2} : Share{2, 3}; }

// The kernel's code is kept short (loops are rolled, one call site for the weight gradients): a block's warps run it once
// per layer with little to overlap, and unrolled it was bound by instruction fetch (4.4 of 9 cycles per instruction).
// Sixteen warps although eight own rows at most: the head and the weight gradients are shared by all, the layers by teams.
// Save: also write the activations to p.saved.  Teams: see TeamRows.
template <bool Save, bool Teams>
__global__ void __launch_bounds__(StepThreads, 1) reference_step_kernel(const __grid_constant__ StepParams p) {
    extern __shared__ __align__(16) uint8_t shared[];
    const StepShared at(p.depth, p.rows, p.context);
    const uint32_t base = smem_address(shared), weights = base + at.weights, stage_base = base + at.stage;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
    float *scales = reinterpret_cast<float *>(shared + at.scales);
    const float2 *rope = reinterpret_cast<const float2 *>(shared + at.rope);
    uint8_t *xs = shared + at.bytes, *ys = xs + p.rows;
    float2 *dt_gate = reinterpret_cast<float2 *>(shared + at.dt_gate);
    float *norm_sums = reinterpret_cast<float *>(shared + at.norm_sums); // [layer's parity][row tile][two norms][16]
    float2 *row_sums = reinterpret_cast<float2 *>(shared + at.row_sums); // [row][warp]: maximum, sum of exponentials
    uint8_t *stage = shared + at.stage;
    const int s_wide = 0, s_hidden = s_wide + p.rows * PitchWide, s_qkv = s_hidden + p.rows * PitchHidden,
              s_dh = s_qkv + p.rows * PitchQkv, s_dh2 = s_dh + p.rows * PitchWidth, s_attended = s_dh2 + p.rows * PitchWidth,
              s_normed1 = s_attended + p.rows * PitchWidth, s_normed2 = s_normed1 + p.rows * PitchWidth;
    const int s_logits = 0, s_final = p.rows * PitchLogits; // the head's use of the same bytes
    float *partial = p.partial + int64_t(blockIdx.x) * p.partial_stride;

    grid_launch_dependents();
    for (int i = threadIdx.x; i < p.context; i += StepThreads)
        reinterpret_cast<float2 *>(shared + at.rope)[i] = p.rope[i];

    // ---- a tile's bytes, one thread per row; then the embeddings of its tokens, into the attention gradients' memory ----
    auto fetch_bytes = [&](int tile) {
        const int r = threadIdx.x, first_sequence = tile * p.sequences, valid = min(p.sequences, p.batch - first_sequence) * p.context;
        int x = -1, y = 0;
        if (r < valid && r < p.rows) {
            if (p.data) { // endpoint = lo + hash(seed + step * batch + sequence) % (size - lo), see sample_kernel
                const int64_t lo = p.context > 8 ? p.context : 8;
                const uint64_t seed = p.seed + __ldcg(&p.counters->step) * uint64_t(p.batch) + uint64_t(first_sequence + r / p.context);
                const uint8_t *source = p.data + lo + (long long)(hash_u64(seed) % uint64_t(p.data_size - lo)) - p.context + r % p.context;
                x = source[0], y = source[1];
            } else {
                x = p.x[int64_t(first_sequence) * p.context + r], y = p.y[int64_t(first_sequence) * p.context + r];
            }
        }
        if (r < p.rows)
            xs[r] = uint8_t(max(x, 0)), ys[r] = uint8_t(y);
        return x;
    };
    auto fetch_embeddings = [&](int x) {
        if (x >= 0)
#pragma unroll
            for (int half = 0; half < 2; ++half)
                copy_async<16>(base + at.dy + threadIdx.x * 32 + half * 16, p.weight_high + x * Width + half * 8);
    };
    // The bytes are found while the update before this step runs: the step's number is counted up by the reduction before that update, which has ended
    // when the update lets this kernel start.
    const int first_byte = fetch_bytes(blockIdx.x);
    grid_dependency_wait(); // the weights of the update before this step
    fetch_embeddings(first_byte);

    // ---- weights to shared memory; they are awaited before the first product ----
    const int final_norm = Layer0 + p.depth * LayerParameters, head = final_norm + Width, head_rows = p.depth * LayerRows;
    auto row_half = [&](int row, int half) { return weights + row * 32 + ((half ^ ((row >> 2) & 1)) << 4); };
#pragma unroll 1
    for (int i = threadIdx.x; i < LayerRows * 2; i += StepThreads) { // one 16-byte half row, of every layer
        const int row = i / 2, half = i % 2, r = row % 16;
        // row 2t + j of a group of 16 qkv rows is the matrix's row 4t + j, row 8 + 2t + j its row 4t + 2 + j
        int from = OffQkv + (row - r + (r % 8) / 2 * 4 + r / 8 * 2 + r % 2) * Width + half * 8;
        if (row >= RowsDown)
            from = OffDown + r * Hidden + (row - RowsDown) / 16 * 16 + half * 8;
        else if (row >= RowsWide)
            from = OffGate + (row - RowsWide) * Width + half * 8;
        uint32_t to = row_half(row, half);
        const bf16 *source = p.weight_high + Layer0 + from;
        if (row >= RowsAttention && row < RowsWide) { // columns permuted like qkv's rows
            source = p.weight_high + Layer0 + OffAttention + r * Width + 2 * half;
#pragma unroll 1
            for (int l = 0; l < p.depth; ++l, to += LayerRows * 32, source += LayerParameters)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    copy_async<4>(to + 4 * c, source + 4 * c);
        } else {
#pragma unroll 1
            for (int l = 0; l < p.depth; ++l, to += LayerRows * 32, source += LayerParameters)
                copy_async<16>(to, source);
        }
    }
#pragma unroll
    for (int i = threadIdx.x; i < Vocabulary * 2; i += StepThreads)
        copy_async<16>(row_half(head_rows + i / 2, i % 2), p.weight_high + head + i / 2 * Width + i % 2 * 8);
#pragma unroll 1
    for (int i = threadIdx.x; i < (2 * p.depth + 1) * Width; i += StepThreads) {
        const int norm = i / Width;
        const int from = norm == 2 * p.depth ? final_norm : Layer0 + norm / 2 * LayerParameters + (norm % 2 ? OffMlpNorm : 0);
        scales[i] = join_weight(p.weight_high[from + i % Width], p.weight_low[from + i % Width]);
    }

    constexpr int Team = Teams ? 3 : 1;
    const int row_tiles = p.rows / 16;
    int own = Teams ? warp % row_tiles : warp, member = Teams ? warp / row_tiles : 0; // the warp's 16 rows, its place in the team at them
    asm volatile("" : "+r"(own), "+r"(member));                                       // kept, not divided out again at every use
    const int row0 = own * 16;
    const bool mine = Teams ? member == 0 : own < row_tiles, active = Teams ? member < Team : mine; // owns the rows; has a share in them
    const Share share = Teams ? Share{member, member + 1} : Share{0, 3}, qkv_back_share = Teams ? qkv_back_share_of(member) : share;
    auto team_barrier = [&] {
        if constexpr (Teams)
            asm volatile("bar.sync %0, %1;" ::"r"(1 + own), "n"(32 * Team) : "memory");
    };
    // The owner's rows as the helpers read them, after it has put them there.
    auto as_kept = [&](const uint4 *slot, const Tile &owners, Tile &v) {
        if constexpr (Teams) {
            unpack_tile(*slot, v);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = owners[i];
        }
    };
    // 32 bytes per lane and helper in the memory of the head's row sums: two packed tiles, the helper's or, going back, first the
    // owner's gradient for it
    auto helper_slot = [&](int helper) { return reinterpret_cast<uint4 *>(shared + at.row_sums + ((own * 2 + helper - 1) * 32 + lane) * 32); };
    auto hand_in = [&](int which, const uint32_t (&v)[4]) { helper_slot(member)[which] = make_uint4(v[0], v[1], v[2], v[3]); };
    auto handed_in = [&](int helper, int which, uint32_t (&v)[4]) {
        const uint4 u = helper_slot(helper)[which];
        v[0] = u.x, v[1] = u.y, v[2] = u.z, v[3] = u.w;
    };
    auto hand_out = [&](const Tile &v) { // the owner's rows, rounded
        if constexpr (Teams) {
            uint32_t packed[4];
            pack_tile(v, packed);
#pragma unroll
            for (int helper = 1; helper < Team; ++helper)
                helper_slot(helper)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        }
    };
    // rows g and g + 8: position inside the sequence and the sequence's first row
    int start[2], position[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        position[r] = (row0 + g + 8 * r) % p.context;
        start[r] = row0 + g + 8 * r - position[r];
    }
    const int longest = max(position[0], position[1]), furthest = p.context - min(position[0], position[1]);

    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
        const bool accumulate = tile != int(blockIdx.x);
        const int first_sequence = tile * p.sequences, count = min(p.sequences, p.batch - first_sequence);
        const int valid = count * p.context; // rows of the tile that hold tokens
        const int64_t token0 = int64_t(first_sequence) * p.context;
        if (accumulate) {
            __syncthreads(); // the previous tile has been read
            fetch_embeddings(fetch_bytes(tile));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();

        Tile x = {}; // residual stream, then its gradient
        if (mine) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (row0 + g + 8 * r >= valid) // stays zero: an infinite weight that no token reads must not reach the sums
                    continue;
                const uint32_t *row = reinterpret_cast<const uint32_t *>(shared + at.dy + (row0 + g + 8 * r) * 32);
                const uint32_t a = row[t], b = row[4 + t];
                x[2 * r] = __uint_as_float(a << 16), x[2 * r + 1] = __uint_as_float(a & 0xffff0000u);
                x[4 + 2 * r] = __uint_as_float(b << 16), x[5 + 2 * r] = __uint_as_float(b & 0xffff0000u);
            }
        }
        auto saved_slot = [&](int offset, int l) { return reinterpret_cast<uint4 *>(shared + offset) + (l * row_tiles + own) * 32 + lane; };
        auto top_slot = [&](int l) { return reinterpret_cast<float2 *>(shared + at.saved_top) + (l * row_tiles + own) * 32 + lane; };
        auto keep = [&](int offset, int l, const Tile &v) {
            uint32_t packed[4];
            pack_tile(v, packed);
            *saved_slot(offset, l) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        };
        auto save = [&](void *to, int columns, int column, bool heads, const Tile &v) {
            if constexpr (Save)
                save_tile(to, columns, column, heads, v, token0 + row0, valid - row0, g, t);
        };
        // normed1 of a layer and its rotated q, k, v (those in `share`) from its input, the latter to `buffer` [row][48]
        auto project_qkv = [&](int l, uint32_t panel, const Tile &input, Tile &normed, uint8_t *buffer, const Share &share) {
            rms_norm(input, Scale(scales + 2 * l * Width, t), normed);
            uint32_t a[4];
            pack_tile(normed, a);
#pragma unroll 1
            for (int m = share.from; m < share.to; ++m) {
                Tile y = {};
                multiply(y, a, panel, RowsQkv + 16 * m, lane);
                round_tile(y);
                if (m < 2)
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        rotate(y[2 * r], y[2 * r + 1], rope[position[r]]);
                put_heads(buffer + row0 * PitchQkv + 32 * m, PitchQkv, y, g, t);
                save(p.saved.layer[l].qkv, 3 * Width, 16 * m, true, y); // (backward writes the same values again)
            }
        };

        // ---- forward ----
        for (int l = 0; l < p.depth; ++l) {
            // k and v of consecutive layers alternate between two buffers: one barrier a layer (the second lies in the stage)
            uint8_t *buffer = l % 2 ? stage : shared + at.exchange;
            const uint32_t panel = weights + l * LayerRows * 32;
            if (mine)
                keep(at.saved_x, l, x);
            if (active) {
                team_barrier();
                Tile input, normed;
                as_kept(saved_slot(at.saved_x, l), x, input);
                project_qkv(l, panel, input, normed, buffer, share);
                if (mine) {
                    save(p.saved.layer[l].x, Width, 0, false, x);
                    save(p.saved.layer[l].normed1, Width, 0, false, normed);
                }
            }
            __syncthreads();
            if (!active)
                continue;
            uint32_t a[4];
            if (mine) {
                Tile attended;
                Four q[2];
                float top[2];
                int best[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    q[r] = load_four(buffer + (row0 + g + 8 * r) * PitchQkv + 8 * t);
                    top[r] = -CUDART_INF_F, best[r] = start[r];
                }
#pragma unroll 1
                for (int j = 0; j <= longest; j += 2) {
                    Four k[2][2];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int r = 0; r < 2; ++r) // the row's own key again once past it: no change
                            k[u][r] = load_four(buffer + (start[r] + min(j + u, position[r])) * PitchQkv + 32 + 8 * t);
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const float score = dot_four(q[r], k[u][r]);
                            if (score > top[r]) // the first key wins ties
                                top[r] = score, best[r] = start[r] + min(j + u, position[r]);
                        }
                }
                const Four v[2] = {load_four(buffer + best[0] * PitchQkv + 64 + 8 * t), load_four(buffer + best[1] * PitchQkv + 64 + 8 * t)};
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float gate = gelu(top[r]);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        attended[(c >> 1) * 4 + 2 * r + (c & 1)] = v[r].v[c] * gate; // rounded when packed
                    shared[at.selected + (l * p.rows + row0 + g + 8 * r) * Heads + t] = uint8_t(best[r]);
                }
                *top_slot(l) = make_float2(top[0], top[1]);
                pack_tile(attended, a);
                Tile branch = {};
                multiply(branch, a, panel, RowsAttention, lane);
                add_branch(x, branch); // middle
                keep(at.saved_middle, l, x);
                save(p.saved.layer[l].attended, Width, 0, true, attended);
                save(p.saved.layer[l].middle, Width, 0, false, x);
            }
            team_barrier();
            Tile middle, normed, down = {};
            as_kept(saved_slot(at.saved_middle, l), x, middle);
            rms_norm(middle, Scale(scales + (2 * l + 1) * Width, t), normed);
            if (mine)
                save(p.saved.layer[l].normed2, Width, 0, false, normed);
            pack_tile(normed, a);
#pragma unroll 1
            for (int m = share.from; m < share.to; ++m) {
                Tile gate = {}, up = {};
                multiply(gate, a, panel, RowsWide + 16 * m, lane);
                multiply(up, a, panel, RowsWide + Hidden + 16 * m, lane);
                activate(gate, up);
                save(p.saved.layer[l].activated, Hidden, 16 * m, false, up);
                uint32_t h[4];
                pack_tile(up, h);
                if (mine)
                    multiply(down, h, panel, RowsDown + 16 * m, lane);
                else
                    hand_in(0, h);
            }
            team_barrier();
            if (mine) {
#pragma unroll
                for (int helper = 1; helper < Team; ++helper) {
                    uint32_t h[4];
                    handed_in(helper, 0, h);
                    multiply(down, h, panel, RowsDown + 16 * helper, lane);
                }
                add_branch(x, down);
            }
        }

        // ---- head and loss: every warp takes its share of the 256 columns, for all rows ----
        __syncthreads(); // the last layers' k and v buffers become the stage
        const Scale final_scale(scales + 2 * p.depth * Width, t);
        if (mine) {
            Tile normed;
            rms_norm(x, final_scale, normed);
            save(p.saved.final_x, Width, 0, false, x);
            save(p.saved.final_normed, Width, 0, false, normed);
            put_tile(stage + s_final + row0 * PitchWidth, PitchWidth, normed, g, t);
        }
        __syncthreads();
        // a 16 x 16 block of a staged array as the left operand
        auto left_operand = [&](int offset, int pitch, uint32_t (&a)[4]) {
            load_matrices(stage_base + offset + (((lane >> 3) & 1) * 8 + (lane & 7)) * pitch + (lane >> 4) * 16, a);
        };
#pragma unroll 1
        for (int row_tile = 0; row_tile < row_tiles; ++row_tile) {
            uint32_t a[4];
            left_operand(s_final + row_tile * 16 * PitchWidth, PitchWidth, a);
            Tile y[HeadTiles] = {};
#pragma unroll
            for (int m = 0; m < HeadTiles; ++m) {
                multiply(y[m], a, weights, head_rows + 16 * (HeadTiles * warp + m), lane);
                round_tile(y[m]); // logits are BF16 values, as in calls that return them
                put_tile(stage + s_logits + row_tile * 16 * PitchLogits + 32 * (HeadTiles * warp + m), PitchLogits, y[m], g, t);
            }
            float high[2] = {-CUDART_INF_F, -CUDART_INF_F}, sum[2] = {0.f, 0.f};
#pragma unroll
            for (int m = 0; m < HeadTiles; ++m)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    high[i >> 1 & 1] = fmaxf(high[i >> 1 & 1], y[m][i]);
#pragma unroll
            for (int r = 0; r < 2; ++r)
                high[r] = quad_max(high[r]);
#pragma unroll
            for (int m = 0; m < HeadTiles; ++m)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    sum[i >> 1 & 1] += expf(y[m][i] - high[i >> 1 & 1]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                sum[r] = quad_sum(sum[r]);
                if (t == 0)
                    row_sums[(row_tile * 16 + g + 8 * r) * StepWarps + warp] = make_float2(high[r], sum[r]);
            }
        }
        __syncthreads();
        for (int row = threadIdx.x; row < p.rows; row += StepThreads) { // a row's maximum, sum and loss, once
            const float4 *sums = reinterpret_cast<const float4 *>(row_sums + row * StepWarps);
            float high = -CUDART_INF_F, sum = 0.f;
            float4 pair[StepWarps / 2];
#pragma unroll
            for (int k = 0; k < StepWarps / 2; ++k) {
                pair[k] = sums[k];
                high = fmaxf(high, fmaxf(pair[k].x, pair[k].z));
            }
#pragma unroll
            for (int k = 0; k < StepWarps / 2; ++k)
                sum += pair[k].y * expf(pair[k].x - high) + pair[k].w * expf(pair[k].z - high);
            if (row < valid)
                p.token_losses[token0 + row] =
                    high + logf(sum) - __bfloat162float(*reinterpret_cast<const bf16 *>(stage + s_logits + row * PitchLogits + 2 * ys[row]));
            row_sums[row * StepWarps] = make_float2(high, 1.f / sum);
        }
        __syncthreads();
#pragma unroll 1
        for (int row_tile = 0; row_tile < row_tiles; ++row_tile)
#pragma unroll
            for (int m = 0; m < HeadTiles; ++m) {
                uint8_t *block = stage + s_logits + row_tile * 16 * PitchLogits + 32 * (HeadTiles * warp + m);
                Tile y;
                get_tile(block, PitchLogits, y, g, t);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int row = row_tile * 16 + g + 8 * r;
                    const float2 total = row_sums[row * StepWarps];
                    const float scaled = row < valid ? p.gradient_scale : 0.f; // rows past the end carry no gradient
                    const int target = int(ys[row]) - 16 * (HeadTiles * warp + m) - 2 * t; // as an offset from the lane's first column
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float &v = y[e / 2 * 4 + 2 * r + e % 2];
                        v = (expf(v - total.x) * total.y - (target == e / 2 * 8 + e % 2 ? 1.f : 0.f)) * scaled;
                    }
                }
                put_tile(block, PitchLogits, y, g, t);
            }
        __syncthreads();
        if (mine) {
            Tile dnormed = {};
#pragma unroll 4
            for (int m = 0; m < 16; ++m) {
                uint32_t a[4];
                left_operand(s_logits + row0 * PitchLogits + 32 * m, PitchLogits, a);
                multiply_transposed(dnormed, a, weights, head_rows + 16 * m, lane);
            }
            round_tile(dnormed);
            rms_norm_backward(x, dnormed, final_scale, nullptr, x, norm_sums + (p.depth % 2 * MaxRowTiles + own) * 2 * Width, lane);
        }
        auto sum_norm = [&](int half, int which, int offset) { // 16 lanes: a norm's scale gradient over the warps, in order
            float total = 0.f;
            for (int w = 0; w < row_tiles; ++w)
                total += norm_sums[((half * MaxRowTiles + w) * 2 + which) * Width + lane];
            partial[offset + lane] = accumulate ? partial[offset + lane] + total : total;
        };
#pragma unroll 1
        for (int job = warp; job < 16; job += StepWarps)
            weight_gradient(partial + head + 16 * job * Width, Width, stage_base + s_logits + 32 * job, PitchLogits, stage_base + s_final,
                            PitchWidth, p.rows, accumulate, lane);
        if (mine)
            hand_out(x); // the row sums have been read
        __syncthreads();
        if (warp == StepWarps - 1 && lane < Width)
            sum_norm(p.depth % 2, 0, final_norm);

        // ---- backward ----
        const bool overlap = Teams && at.overlap;
        const int first_free = overlap ? Team * row_tiles : 0, stage_apart = overlap ? p.rows * StageBytesPerRow : 0;
        for (int l = p.depth - 1; l >= -1; --l) {
            // the 13 weight-gradient tiles of 16 x 16 and two norm scales of the layer that has just been staged
            if (l + 1 < p.depth && warp >= first_free) {
                const int layer0 = Layer0 + (l + 1) * LayerParameters;
                const uint32_t from = stage_base + (l + 1) % 2 * stage_apart;
#pragma unroll 1
                for (int job = warp - first_free; job < 15; job += StepWarps - first_free) {
                    if (job >= 13) {
                        if (lane < Width)
                            sum_norm((l + 1) % 2, job - 13, layer0 + (job == 13 ? 0 : OffMlpNorm));
                        continue;
                    }
                    int to = OffGate + 16 * job * Width, columns = Width, dy_at = s_wide + 32 * job, dy_pitch = PitchWide, x_at = s_normed2,
                        x_pitch = PitchWidth;
                    if (job >= 6) // down: columns 16 (job - 6) of [16][48]
                        to = OffDown + 16 * (job - 6), columns = Hidden, dy_at = s_dh, dy_pitch = PitchWidth, x_at = s_hidden + 32 * (job - 6),
                        x_pitch = PitchHidden;
                    if (job >= 9)
                        to = OffQkv + 16 * (job - 9) * Width, columns = Width, dy_at = s_qkv + 32 * (job - 9), dy_pitch = PitchQkv, x_at = s_normed1,
                        x_pitch = PitchWidth;
                    if (job == 12)
                        to = OffAttention, dy_at = s_dh2, dy_pitch = PitchWidth, x_at = s_attended;
                    weight_gradient(partial + layer0 + to, columns, from + dy_at, dy_pitch, from + x_at, x_pitch, p.rows, accumulate, lane);
                }
            }
            if (!overlap && l + 1 < p.depth)
                __syncthreads();
            if (l < 0)
                break;
            uint8_t *const stage = shared + at.stage + l % 2 * stage_apart, *exchange = shared + at.exchange;
            const uint8_t *selected = shared + at.selected + l * p.rows * Heads;
            const uint32_t panel = weights + l * LayerRows * 32;
            Tile input, dq;
            Four dy[2];
            if (active) {
                Tile middle, normed;
                uint32_t a[4], dh[4];
                unpack_tile(*saved_slot(at.saved_middle, l), middle);
                const Scale scale(scales + (2 * l + 1) * Width, t);
                rms_norm(middle, scale, normed);
                pack_tile(normed, a);
                if (mine) {
                    put_tile(stage + s_normed2 + row0 * PitchWidth, PitchWidth, normed, g, t);
                    put_tile(stage + s_dh + row0 * PitchWidth, PitchWidth, x, g, t);
                    pack_tile(x, dh);
                } else {
                    handed_in(member, 0, dh);
                }
                Tile branch = {};
                auto into_branch = [&](int m, const uint32_t (&dgate)[4], const uint32_t (&dup)[4]) {
                    multiply_transposed(branch, dgate, panel, RowsWide + 16 * m, lane);
                    multiply_transposed(branch, dup, panel, RowsWide + Hidden + 16 * m, lane);
                };
#pragma unroll 1
                for (int m = share.from; m < share.to; ++m) {
                    Tile gate = {}, up = {}, dout = {};
                    multiply(gate, a, panel, RowsWide + 16 * m, lane);
                    multiply(up, a, panel, RowsWide + Hidden + 16 * m, lane);
                    multiply_transposed(dout, dh, panel, RowsDown + 16 * m, lane);
                    Tile activated;
                    activate_backward(gate, up, dout, activated);
                    put_tile(stage + s_hidden + row0 * PitchHidden + 32 * m, PitchHidden, activated, g, t);
                    put_tile(stage + s_wide + row0 * PitchWide + 32 * m, PitchWide, gate, g, t);
                    put_tile(stage + s_wide + row0 * PitchWide + 2 * Hidden + 32 * m, PitchWide, up, g, t);
                    uint32_t dgate[4], dup[4];
                    pack_tile(gate, dgate);
                    pack_tile(up, dup);
                    if (mine)
                        into_branch(m, dgate, dup);
                    else
                        hand_in(0, dgate), hand_in(1, dup);
                }
                team_barrier();
                if (mine) {
#pragma unroll
                    for (int helper = 1; helper < Team; ++helper) {
                        uint32_t dgate[4], dup[4];
                        handed_in(helper, 0, dgate);
                        handed_in(helper, 1, dup);
                        into_branch(helper, dgate, dup);
                    }
                    round_tile(branch);
                    rms_norm_backward(middle, branch, scale, &x, x, norm_sums + ((l % 2 * MaxRowTiles + own) * 2 + 1) * Width, lane);
                    put_tile(stage + s_dh2 + row0 * PitchWidth, PitchWidth, x, g, t);
                    // gradient of the attended values: the lane's head t of rows g and g + 8
                    pack_tile(x, a);
                    Tile dattended = {};
                    multiply_transposed(dattended, a, panel, RowsAttention, lane);
                    round_tile(dattended);
                    put_heads(shared + at.dy + row0 * 32, 32, dattended, g, t);
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        dy[r] = {{dattended[2 * r], dattended[2 * r + 1], dattended[4 + 2 * r], dattended[5 + 2 * r]}};
                }
                unpack_tile(*saved_slot(at.saved_x, l), input);
                if (qkv_back_share.to) {
                    project_qkv(l, panel, input, normed, exchange, qkv_back_share);
                    if (qkv_back_share.from == 0)
                        put_tile(stage + s_normed1 + row0 * PitchWidth, PitchWidth, normed, g, t);
                }
            }
            __syncthreads();
            if (mine) {
                const float2 top = load_pair(top_slot(l));
                Tile attended;
                Four k[2], v[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint8_t *key = exchange + load_byte(selected + (row0 + g + 8 * r) * Heads + t) * PitchQkv + 8 * t;
                    k[r] = load_four(key + 32), v[r] = load_four(key + 64);
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float score = r ? top.y : top.x, gate = gelu(score);
                    const float dt = dot_four(dy[r], v[r]) * gelu_derivative(score);
                    dt_gate[(row0 + g + 8 * r) * Heads + t] = make_float2(dt, gate);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int i = (c >> 1) * 4 + 2 * r + (c & 1);
                        attended[i] = v[r].v[c] * gate;
                        dq[i] = dt * k[r].v[c];
                    }
                }
                round_tile(dq);
                put_heads(stage + s_attended + row0 * PitchWidth, PitchWidth, attended, g, t);
            }
            __syncthreads();
            if (mine) {
                Tile dk = {}, dv = {};
#pragma unroll 1
                for (int j = 0; j < furthest; j += 2) { // a key gathers from the queries that selected it; of the others it takes zeros
                    // (every load of the pair is issued before the first is used)
                    Four q[2][2], d[2][2];
                    float2 w[2][2];
                    bool chosen[2][2];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const int row = row0 + g + 8 * r, last = min(row + p.context - 1 - position[r], p.rows - 1), query = min(row + j + u, last);
                            q[u][r] = load_four(exchange + query * PitchQkv + 8 * t), d[u][r] = load_four(shared + at.dy + query * 32 + 8 * t);
                            w[u][r] = load_pair(dt_gate + query * Heads + t);
                            chosen[u][r] = (row + j + u <= last) & (load_byte(selected + query * Heads + t) == row);
                        }
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const float dt = chosen[u][r] ? w[u][r].x : 0.f, gate = chosen[u][r] ? w[u][r].y : 0.f;
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                const int i = (c >> 1) * 4 + 2 * r + (c & 1);
                                dk[i] += dt * (chosen[u][r] ? q[u][r].v[c] : 0.f), dv[i] += (chosen[u][r] ? d[u][r].v[c] : 0.f) * gate;
                            }
                        }
                }
                round_tile(dk);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 cs = rope[position[r]], back = make_float2(cs.x, -cs.y);
                    rotate(dq[2 * r], dq[2 * r + 1], back);
                    rotate(dk[2 * r], dk[2 * r + 1], back);
                }
                Tile branch = {};
                uint32_t a[4];
                uint8_t *rows = stage + s_qkv + row0 * PitchQkv;
                put_heads(rows, PitchQkv, dq, g, t);
                put_heads(rows + 32, PitchQkv, dk, g, t);
                put_heads(rows + 64, PitchQkv, dv, g, t);
                pack_tile(dq, a);
                multiply_transposed(branch, a, panel, RowsQkv, lane);
                pack_tile(dk, a);
                multiply_transposed(branch, a, panel, RowsQkv + 16, lane);
                pack_tile(dv, a);
                multiply_transposed(branch, a, panel, RowsQkv + 32, lane);
                round_tile(branch);
                rms_norm_backward(input, branch, Scale(scales + 2 * l * Width, t), &x, x, norm_sums + (l % 2 * MaxRowTiles + own) * 2 * Width, lane);
                hand_out(x);
            }
            __syncthreads();
        }

        // ---- embedding gradient: one-hot(x)^T dh, the one-hot operand built in registers ----
        bool finite = true;
        if (mine) { // (the first layer's stage may still be read)
            put_tile(stage + stage_apart + s_dh + row0 * PitchWidth, PitchWidth, x, g, t);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                finite = finite && isfinite(x[i]);
        }
        if (!__syncthreads_and(finite)) { // the product's zeros would carry one token's NaN to every byte value
#pragma unroll 1
            for (int i = threadIdx.x; i < Vocabulary * Width; i += StepThreads) {
                float total = 0.f;
#pragma unroll 1
                for (int r = 0; r < valid; ++r)
                    if (xs[r] == i / Width)
                        total += __bfloat162float(reinterpret_cast<const bf16 *>(stage + stage_apart + s_dh + r * PitchWidth)[i % Width]);
                partial[i] = accumulate ? partial[i] + total : total;
            }
            continue;
        }
        const uint32_t b_lane = stage_base + stage_apart + s_dh + (((lane >> 3) & 1) * 8 + (lane & 7)) * PitchWidth + (lane >> 4) * 16;
#pragma unroll 1
        for (int job = warp; job < 16; job += StepWarps) {
            Tile acc = {};
            const int value = 16 * job + g;
#pragma unroll 1
            for (int k = 0; k < p.rows; k += 16) {
                uint32_t a[4], b[4];
                const int b0 = xs[k + 2 * t], b1 = xs[k + 2 * t + 1], b2 = xs[k + 8 + 2 * t], b3 = xs[k + 9 + 2 * t];
#pragma unroll
                for (int r = 0; r < 2; ++r) { // 0x3f80 is 1.0
                    a[r] = (b0 == value + 8 * r ? 0x3f80u : 0u) | (b1 == value + 8 * r ? 0x3f800000u : 0u);
                    a[2 + r] = (b2 == value + 8 * r ? 0x3f80u : 0u) | (b3 == value + 8 * r ? 0x3f800000u : 0u);
                }
                load_matrices_transposed(b_lane + k * PitchWidth, b);
                mma_bf16(acc[0], acc[1], acc[2], acc[3], a, b[0], b[1]);
                mma_bf16(acc[4], acc[5], acc[6], acc[7], a, b[2], b[3]);
            }
            add_gradient(partial + 16 * job * Width, Width, acc, accumulate, lane);
        }
    }
}

// Blocks 0 .. gradient_blocks-1: 64 parameters each, the rows of `partial` added in a fixed order (sixteen interleaved
// groups of rows, then the groups), and the block's sum of squares for the clip norm.  The blocks after them: the mean
// loss of one position over the batch, summed in double (see loss_history_kernel; one thread per position took 120 us
// at batch 2880).
constexpr int ReduceParameters = 64, ReduceGroups = 16;
struct ReduceParams {
    const float *partial;
    int64_t stride;
    int parts, count, gradient_blocks;
    float *gradient, *norm_partial;
    const float *token_losses;
    float *history;
    StepCounters *counters;
    int batch, context;
};
__global__ void __launch_bounds__(256) reduce_gradients_kernel(const __grid_constant__ ReduceParams p) {
    __shared__ float4 sums[ReduceGroups][ReduceParameters / 4];
    __shared__ double loss_sums[8];
    grid_launch_dependents();
    grid_dependency_wait();
    // The step's number is read by the step kernel, which has ended, and by the update, which knows that it has been counted up; the update in turn
    // counts the rows of losses, which only this kernel reads.  (The update's last block counted both by a ticket, a microsecond at its end, and the bytes'
    // chain of loads began after it: 64 tokens 31.5 -> 30.2 us a step, 11520 tokens 50.6 -> 49.5.  More of the rows below at a time: 1.4 us slower, the code
    // being fetched anew for every step.)
    if (blockIdx.x == 0 && threadIdx.x == 255)
        p.counters->step += 1;
    if (int(blockIdx.x) >= p.gradient_blocks) {
        const int position = blockIdx.x - p.gradient_blocks;
        double total = 0;
        for (int b = threadIdx.x; b < p.batch; b += 256)
            total += p.token_losses[int64_t(b) * p.context + position];
#pragma unroll
        for (int k = 16; k; k >>= 1)
            total += __shfl_xor_sync(0xffffffffu, total, k);
        if (threadIdx.x % 32 == 0)
            loss_sums[threadIdx.x / 32] = total;
        __syncthreads();
        if (threadIdx.x == 0) {
            total = 0;
            for (int w = 0; w < 8; ++w)
                total += loss_sums[w];
            p.history[int64_t(p.counters->iteration) * p.context + position] = float(total / p.batch);
        }
        return;
    }
    const int quad = threadIdx.x % (ReduceParameters / 4), group = threadIdx.x / (ReduceParameters / 4);
    const int at = blockIdx.x * ReduceParameters + quad * 4; // the rows of `partial` are padded to whole blocks
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int part = group; part < p.parts; part += ReduceGroups) {
        const float4 v = *reinterpret_cast<const float4 *>(p.partial + part * p.stride + at);
        sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
    }
    sums[group][quad] = sum;
    __syncthreads();
    if (threadIdx.x < 32) {
        float square = 0.f;
        for (int i = threadIdx.x; i < ReduceParameters; i += 32) {
            float total = 0.f;
            for (int k = 0; k < ReduceGroups; ++k)
                total += reinterpret_cast<const float *>(sums[k])[i];
            const int index = blockIdx.x * ReduceParameters + i;
            if (index < p.count) {
                p.gradient[index] = total;
                square += total * total;
            }
        }
        square = warp_sum(square);
        if (threadIdx.x == 0)
            p.norm_partial[blockIdx.x] = square;
    }
}

int tile_rows_that_fit(int depth, int context) {
    for (int rows = MaxRows; rows >= 16; rows -= 16)
        if (StepShared(depth, rows, context).total <= MaxShared)
            return rows;
    return 0;
}
} // namespace

// The kernel takes any batch; a sequence must fit a block's tile beside the weights (depth 4: 128 tokens, depth 8: 96,
// depth 16: 48).
bool reference_step_supported(const TgConfigEx &c) {
    return c.width == Width && c.heads == Heads && c.hidden == Hidden && c.norm == TG_NORM_RMS && c.attention == TG_ATTENTION_ARGMAX &&
           c.mlp == TG_MLP_SWIGLU && !c.tied && c.rope == TG_ROPE_PARTIAL && c.hidden_optimizer == TG_HIDDEN_MUON &&
           c.precision == TG_PRECISION_BF16 && c.base.depth <= ReferenceMaxDepth &&
           c.base.context <= tile_rows_that_fit(c.base.depth, c.base.context);
}

// As many sequences per tile as spread the batch evenly over the SMs in the fewest rounds, but at least one warp's
// 16 tokens: a smaller tile would pay the same latency for padding.
ReferenceStepPlan reference_step_plan(const TgConfigEx &c, int sms) {
    const int most = tile_rows_that_fit(c.base.depth, c.base.context) / c.base.context, batch = c.base.batch;
    const int rounds = ((batch + most - 1) / most + sms - 1) / sms;
    ReferenceStepPlan plan;
    plan.sequences = std::min(most, std::max((batch + rounds * sms - 1) / (rounds * sms), 16 / c.base.context));
    plan.rows = (plan.sequences * c.base.context + 15) / 16 * 16;
    plan.tiles = (batch + plan.sequences - 1) / plan.sequences;
    plan.blocks = std::min(plan.tiles, sms);
    const int count = Layer0 + c.base.depth * LayerParameters + Width + Vocabulary * Width;
    plan.gradient_blocks = (count + ReduceParameters - 1) / ReduceParameters;
    plan.partial_stride = int64_t(plan.gradient_blocks) * ReduceParameters;
    plan.helpers = plan.rows <= TeamRows;
    plan.overlap = StepShared(c.base.depth, plan.rows, c.base.context).overlap;
    return plan;
}

void launch_reference_step(const ReferenceStepArgs &a, const ReferenceStepPlan &plan, cudaStream_t s) {
    StepParams p{};
    p.data = a.data, p.data_size = a.data_size, p.seed = a.seed, p.x = a.x, p.y = a.y, p.counters = a.counters;
    p.weight_high = a.weight_high, p.weight_low = a.weight_low, p.rope = a.rope, p.partial = a.partial, p.token_losses = a.token_losses;
    p.partial_stride = plan.partial_stride;
    p.batch = a.batch, p.context = a.context, p.depth = a.depth;
    p.sequences = plan.sequences, p.rows = plan.rows, p.tiles = plan.tiles;
    p.gradient_scale = 1.f / (float(a.batch) * float(a.context));
    if (a.save)
        p.saved = *a.save;
    const int shared = StepShared(a.depth, plan.rows, a.context).total;
    auto *kernel = plan.helpers ? a.save ? reference_step_kernel<true, true> : reference_step_kernel<false, true>
                                : a.save ? reference_step_kernel<true, false> : reference_step_kernel<false, false>;
    CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MaxShared));
    // Launched programmatically: each kernel's set-up overlaps the tail of the one before it.
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(plan.blocks), config.blockDim = dim3(StepThreads), config.dynamicSmemBytes = shared, config.stream = s;
    config.attrs = &attribute, config.numAttrs = 1;
    CHECK_CUDA(cudaLaunchKernelEx(&config, kernel, p));
    const int count = Layer0 + a.depth * LayerParameters + Width + Vocabulary * Width;
    ReduceParams r{a.partial, plan.partial_stride, plan.blocks, count, plan.gradient_blocks, a.gradient, a.norm_partial, a.token_losses,
                   a.history, a.counters, a.batch, a.context};
    config.gridDim = dim3(plan.gradient_blocks + a.context), config.blockDim = dim3(256), config.dynamicSmemBytes = 0;
    CHECK_CUDA(cudaLaunchKernelEx(&config, reduce_gradients_kernel, r));
}
