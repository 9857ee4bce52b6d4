// Optimizer kernels (reference cuda/optim.cuh).  One fused pass over the flat parameter arena
// applies "mantissa" AdamW: FP32 masters are kept as a BF16 high half (the compute weight) and
// the 16 low mantissa bits, so updates below one BF16 ulp are retained.  Muon's elementwise
// stages sit either side of Newton-Schulz GEMMs issued by the host.
#include "device_utils.cuh"
#include "kernels.cuh"
#include "sm100.cuh"
#include <algorithm>

// Fixed-order partial sums of squares: block b covers a contiguous slice.
__global__ void __launch_bounds__(256) sum_squares_kernel(const float *gradient, int64_t count, float *partial) {
    __shared__ float scratch[32];
    sm100::grid_dependency_wait();
    sm100::grid_launch_dependents(); // after the wait: what starts now may read all that was written before this kernel
    int64_t per = (count + gridDim.x - 1) / gridDim.x;
    per = (per + 3) / 4 * 4;
    int64_t begin = blockIdx.x * per, end = begin + per < count ? begin + per : count;
    float sum = 0;
    int64_t i = begin + threadIdx.x * 4;
    for (; i + 3 * 1024 + 4 <= end; i += 4 * 1024) { // four independent 128-bit loads in flight per thread
        float4 g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            g[u] = *reinterpret_cast<const float4 *>(gradient + i + u * 1024);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            sum += g[u].x * g[u].x + g[u].y * g[u].y + g[u].z * g[u].z + g[u].w * g[u].w;
    }
    for (; i < end; i += 256 * 4) {
        if (i + 4 <= end) {
            float4 g = *reinterpret_cast<const float4 *>(gradient + i);
            sum += g.x * g.x + g.y * g.y + g.z * g.z + g.w * g.w;
        } else {
            for (int64_t j = i; j < end; ++j)
                sum += gradient[j] * gradient[j];
        }
    }
    sum = block_sum(sum, scratch);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = sum;
}
void launch_sum_squares(const float *gradient, int64_t count, float *partial, int blocks, cudaStream_t s) {
    sm100::launch_overlapping(sum_squares_kernel, blocks, 256, 0, s, gradient, count, partial);
}

// clip = min(1, clip / (|g| + 1e-6)) from the per-block sums, same order in every block.
__device__ __forceinline__ float clip_factor(const float *norm_partial, int norm_blocks, float clip,
                                             float *scratch) {
    if (!(clip > 0))
        return 1.f;
    float local = 0;
    for (int b = threadIdx.x; b < norm_blocks; b += blockDim.x)
        local += norm_partial[b];
    float norm = block_sum(local, scratch);
    return fminf(1.f, clip / (sqrtf(norm) + 1e-6f));
}

// What every AdamW thread needs of the step: its own schedule point (reference cuda/optim.cuh:82-89), and bias
// correction with the current, possibly cycled, beta1 as torch.optim.AdamW does.
struct AdamRates {
    float clip = 1.f, lr, beta1, step_size, inv_sqrt_bc2;
    __device__ __forceinline__ AdamRates(const AdamArgs &a, unsigned long long step) {
        float multiplier = 1;
        beta1 = a.beta1;
        if (a.schedule) {
            TgStepRates rates = a.schedule[step];
            multiplier = rates.multiplier;
            beta1 = rates.momentum;
        }
        lr = a.learning_rate * multiplier;
        step_size = lr / (1 - powf(beta1, float(step + 1)));
        inv_sqrt_bc2 = 1.f / sqrtf(1 - powf(a.beta2, float(step + 1)));
    }
};
// Eight consecutive parameters and their state, fetched before the rates are known.
struct AdamGroup {
    int mode = 0;
    float g[8], m[8], v[8];
    uint4 high, low;
    __device__ __forceinline__ AdamGroup() {}
    __device__ __forceinline__ AdamGroup(const AdamArgs &a, int64_t group) : mode(a.mode[group]) {
        if (mode == 0) // Muon's
            return;
        const int64_t i = group * 8;
        load8(a.gradient + i, g);
        load8(a.momentum + i, m);
        load8(a.variance + i, v);
        high = *reinterpret_cast<const uint4 *>(a.weight_high + i);
        low = *reinterpret_cast<const uint4 *>(a.weight_low + i);
    }
    // Of the second moment's two products one is rounded before it is added: written out, so that each kernel keeps the one it has (DecayedRounded: the
    // old moment's) whatever stands around it.
    template <bool DecayedRounded> __device__ __forceinline__ void update(const AdamArgs &a, const AdamRates &rates, int64_t group) {
        if (mode == 0)
            return;
        const int64_t i = group * 8;
        const float decay = 1 - rates.lr * (mode == 2 ? a.weight_decay : 0.f);
        float w[8];
        const unsigned hw[4] = {high.x, high.y, high.z, high.w}, lw[4] = {low.x, low.y, low.z, low.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            w[2 * j] = __uint_as_float((hw[j] << 16) | (lw[j] & 0xffffu));
            w[2 * j + 1] = __uint_as_float((hw[j] & 0xffff0000u) | (lw[j] >> 16));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float gj = g[j] * rates.clip;
            m[j] = m[j] + (1 - rates.beta1) * (gj - m[j]);
            v[j] = DecayedRounded ? fmaf((1 - a.beta2) * gj, gj, a.beta2 * v[j]) : fmaf(a.beta2, v[j], (1 - a.beta2) * gj * gj);
            w[j] = w[j] * decay - rates.step_size * m[j] / (sqrtf(v[j]) * rates.inv_sqrt_bc2 + a.epsilon);
        }
        store8(a.momentum + i, m);
        store8(a.variance + i, v);
        unsigned ho[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            unsigned b0 = __float_as_uint(w[2 * j]), b1 = __float_as_uint(w[2 * j + 1]);
            ho[j] = (b0 >> 16) | (b1 & 0xffff0000u);
            lo[j] = (b0 & 0xffffu) | (b1 << 16);
        }
        *reinterpret_cast<uint4 *>(a.weight_high + i) = make_uint4(ho[0], ho[1], ho[2], ho[3]);
        *reinterpret_cast<uint4 *>(a.weight_low + i) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        if (a.weight_fp32)
            store8(a.weight_fp32 + i, w);
    }
};
// Starts while the sums of squares are taken, and has the step's rates by then.  (Fetching the first group of parameters meanwhile takes 82 registers
// or more instead of 64: 4 layers d 256 17 -> 25 us.)
__global__ void __launch_bounds__(256) adamw_kernel(AdamArgs a) {
    __shared__ float scratch[32];
    sm100::grid_launch_dependents();
    const int64_t groups = a.count / 8;
    AdamRates rates(a, a.counters->step);
    sm100::grid_dependency_wait();
    rates.clip = clip_factor(a.norm_partial, a.norm_blocks, a.clip, scratch);
    for (int64_t group = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; group < groups;
         group += int64_t(gridDim.x) * blockDim.x)
        AdamGroup(a, group).update<true>(a, rates, group);
    if (!a.advance)
        return;
    __syncthreads(); // every thread has read the step before the block's arrival is counted
    if (threadIdx.x == 0 && atomicInc(a.ticket, gridDim.x - 1) == gridDim.x - 1) {
        a.advance->step += 1;
        a.advance->iteration += 1;
    }
}
void launch_adamw(const AdamArgs &a, int sms, cudaStream_t s) {
    int64_t groups = a.count / 8;
    int64_t blocks = (groups + 255) / 256;
    if (blocks > int64_t(sms) * 8)
        blocks = int64_t(sms) * 8;
    sm100::launch_overlapping(adamw_kernel, int(blocks < 1 ? 1 : blocks), 256, 0, s, a);
}

// ---- Muon (reference cuda/optim.cuh:16-65) ----

__device__ __forceinline__ void finish_block(const MuonPrepareArgs &a, int matrix, float squares) { // one thread
    a.sumsq[matrix * MuonBlocks + blockIdx.x] = squares;
    if (a.progress && blockIdx.x == 0)
        a.progress[matrix] = 0;
}

__global__ void __launch_bounds__(256) muon_prepare_kernel(MuonPrepareArgs a) {
    __shared__ float scratch[32];
    const float clip = clip_factor(a.norm_partial, a.norm_blocks, a.clip, scratch);
    float mu = a.momentum_rate;
    if (a.schedule)
        mu = a.schedule[a.counters->step].momentum;
    const int matrix = blockIdx.y;
    const int64_t size = int64_t(a.rows) * a.cols, base = matrix * a.stride;
    const bool transpose = a.rows > a.cols;
    float squares = 0;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < size;
         i += int64_t(gridDim.x) * blockDim.x) {
        float g = a.gradient[base + i] * clip;
        float m = a.momentum[base + i] + (1 - mu) * (g - a.momentum[base + i]);
        a.momentum[base + i] = m;
        bf16 u = __float2bfloat16_rn(g + mu * (m - g));
        int64_t index = transpose ? (i % a.cols) * a.rows + i / a.cols : i;
        a.x[matrix * size + index] = u;
        squares += __bfloat162float(u) * __bfloat162float(u);
    }
    squares = block_sum(squares, scratch);
    if (threadIdx.x == 0)
        finish_block(a, matrix, squares);
}
// The same stage, 128-bit: eight consecutive elements per thread (matrices stored in the orientation the
// iterations use, rows <= cols).
__global__ void __launch_bounds__(256) muon_prepare_vector_kernel(MuonPrepareArgs a) {
    __shared__ float scratch[32];
    const float clip = clip_factor(a.norm_partial, a.norm_blocks, a.clip, scratch);
    float mu = a.momentum_rate;
    if (a.schedule)
        mu = a.schedule[a.counters->step].momentum;
    const int matrix = blockIdx.y;
    const int64_t size = int64_t(a.rows) * a.cols, base = matrix * a.stride;
    float squares = 0;
    // Three groups of eight are fetched before the first is worked on: one at a time, each waits for memory on its own (six 384 x 1536 matrices
    // beside the other families 36 -> 15 us).
    constexpr int Ahead = 3;
    const int64_t apart = int64_t(gridDim.x) * blockDim.x * 8;
    for (int64_t first = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) * 8; first < size; first += Ahead * apart) {
        float g[Ahead][8], m[Ahead][8], u[8];
#pragma unroll
        for (int k = 0; k < Ahead; ++k)
            if (first + k * apart < size) {
                load8(a.gradient + base + first + k * apart, g[k]);
                load8(a.momentum + base + first + k * apart, m[k]);
            }
#pragma unroll
        for (int k = 0; k < Ahead; ++k) {
            const int64_t i = first + k * apart;
            if (i >= size)
                break;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                g[k][j] *= clip;
                m[k][j] += (1 - mu) * (g[k][j] - m[k][j]);
                u[j] = rounded<bf16>(g[k][j] + mu * (m[k][j] - g[k][j]));
                squares += u[j] * u[j];
            }
            store8(a.momentum + base + i, m[k]);
            store8(a.x + matrix * size + i, u);
        }
    }
    squares = block_sum(squares, scratch);
    if (threadIdx.x == 0)
        finish_block(a, matrix, squares);
}
// Tall matrices (rows > cols) are orthogonalised transposed.  64 x 64 tiles go through shared memory so
// that gradient and momentum are read, and the transposed BF16 matrix written, in whole 128-byte lines.
constexpr int MuonTile = 64, MuonTilePitch = 66; // BF16 elements per tile row in shared memory (33 words: spreads the banks)
__global__ void __launch_bounds__(256) muon_prepare_transpose_kernel(MuonPrepareArgs a) {
    __shared__ float scratch[32];
    __shared__ __align__(16) bf16 tile[MuonTile * MuonTilePitch]; // [column][row]
    const float clip = clip_factor(a.norm_partial, a.norm_blocks, a.clip, scratch);
    float mu = a.momentum_rate;
    if (a.schedule)
        mu = a.schedule[a.counters->step].momentum;
    const int matrix = blockIdx.y;
    const int64_t size = int64_t(a.rows) * a.cols, base = matrix * a.stride;
    const int tiles_across = a.cols / MuonTile, tiles = (a.rows / MuonTile) * tiles_across;
    float squares = 0;
    // A thread's two groups of eight columns of a tile (rows 32 apart) are fetched while the tile before is worked on: as plain
    // loads, each waiting for the stores before it, a tile cost two round trips to memory.
    constexpr int Items = MuonTile * 8 / 256;
    const int rr = threadIdx.x / 8, chunk = threadIdx.x % 8;
    float next_g[Items][8], next_m[Items][8];
    auto place = [&](int t, int i) { return base + int64_t(t / tiles_across * MuonTile + rr + 32 * i) * a.cols + t % tiles_across * MuonTile + chunk * 8; };
    auto fetch = [&](int t) {
#pragma unroll
        for (int i = 0; i < Items; ++i) {
            load8(a.gradient + place(t, i), next_g[i]);
            load8(a.momentum + place(t, i), next_m[i]);
        }
    };
    if (int(blockIdx.x) < tiles)
        fetch(blockIdx.x);
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int r0 = t / tiles_across * MuonTile, c0 = t % tiles_across * MuonTile;
        float g[Items][8], m[Items][8];
#pragma unroll
        for (int i = 0; i < Items; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                g[i][j] = next_g[i][j], m[i][j] = next_m[i][j];
        if (t + int(gridDim.x) < tiles)
            fetch(t + gridDim.x);
#pragma unroll
        for (int i = 0; i < Items; ++i) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                g[i][j] *= clip;
                m[i][j] += (1 - mu) * (g[i][j] - m[i][j]);
                const bf16 u = __float2bfloat16_rn(g[i][j] + mu * (m[i][j] - g[i][j]));
                tile[(chunk * 8 + j) * MuonTilePitch + rr + 32 * i] = u;
                squares += __bfloat162float(u) * __bfloat162float(u);
            }
            store8(a.momentum + place(t, i), m[i]);
        }
        __syncthreads();
        for (int item = threadIdx.x; item < MuonTile * 8; item += blockDim.x) { // (column, group of 8 rows)
            const int cc = item / 8, chunk = item % 8;
            const uint32_t *source = reinterpret_cast<const uint32_t *>(tile + cc * MuonTilePitch + chunk * 8);
            *reinterpret_cast<uint4 *>(a.x + matrix * size + int64_t(c0 + cc) * a.rows + r0 + chunk * 8) =
                make_uint4(source[0], source[1], source[2], source[3]);
        }
        __syncthreads();
    }
    squares = block_sum(squares, scratch);
    if (threadIdx.x == 0)
        finish_block(a, matrix, squares);
}
void launch_muon_prepare(const MuonPrepareArgs &a, cudaStream_t s) {
    const dim3 grid(MuonBlocks, a.batch);
    const bool aligned = a.stride % 8 == 0 && reinterpret_cast<uintptr_t>(a.gradient) % 32 == 0 &&
                         reinterpret_cast<uintptr_t>(a.momentum) % 32 == 0;
    if (aligned && a.rows > a.cols && a.rows % MuonTile == 0 && a.cols % MuonTile == 0)
        muon_prepare_transpose_kernel<<<grid, 256, 0, s>>>(a);
    else if (aligned && a.rows <= a.cols && (int64_t(a.rows) * a.cols) % 8 == 0)
        muon_prepare_vector_kernel<<<grid, 256, 0, s>>>(a);
    else
        muon_prepare_kernel<<<grid, 256, 0, s>>>(a);
}
// x /= max(bf16(|x|_F), bf16(1e-7)), rounded to BF16.
__global__ void __launch_bounds__(256) muon_normalize_kernel(bf16 *x, const float *sumsq, int64_t per_matrix) {
    const int matrix = blockIdx.y;
    float total = 0;
    for (int b = 0; b < MuonBlocks; ++b)
        total += sumsq[matrix * MuonBlocks + b];
    const float norm = fmaxf(__bfloat162float(__float2bfloat16_rn(sqrtf(total))),
                             __bfloat162float(__float2bfloat16_rn(1e-7f)));
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < per_matrix;
         i += int64_t(gridDim.x) * blockDim.x)
        x[matrix * per_matrix + i] = __float2bfloat16_rn(__bfloat162float(x[matrix * per_matrix + i]) / norm);
}
__global__ void __launch_bounds__(256) muon_normalize_vector_kernel(bf16 *x, const float *sumsq, int64_t per_matrix) {
    const int matrix = blockIdx.y;
    float total = 0;
    for (int b = 0; b < MuonBlocks; ++b)
        total += sumsq[matrix * MuonBlocks + b];
    const float norm = fmaxf(__bfloat162float(__float2bfloat16_rn(sqrtf(total))),
                             __bfloat162float(__float2bfloat16_rn(1e-7f)));
    for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) * 8; i < per_matrix;
         i += int64_t(gridDim.x) * blockDim.x * 8) {
        float v[8];
        load8(x + matrix * per_matrix + i, v);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            v[j] /= norm;
        store8(x + matrix * per_matrix + i, v);
    }
}
// All Newton-Schulz iterations of one small matrix (the reference architecture's 16 x 16 .. 16 x 48) in one
// block's shared memory, with the roundings of the three-GEMM form: BF16 operands, FP32 sums over ascending k,
// A = X X^T, B = 2.0315 A A - 4.775 A and X' = B X + 3.4445 X each rounded to BF16 (reference
// cuda/optim.cuh:60-106).  One launch instead of three per iteration.
__global__ void __launch_bounds__(256) muon_newton_schulz_small_kernel(bf16 *x_all, int r, int n, int steps) {
    extern __shared__ float shared[];
    float *x = shared, *a = x + r * n, *b = a + r * r, *next = b + r * r;
    bf16 *matrix = x_all + int64_t(blockIdx.x) * r * n;
    for (int i = threadIdx.x; i < r * n; i += blockDim.x)
        x[i] = __bfloat162float(matrix[i]);
    __syncthreads();
    for (int step = 0; step < steps; ++step) {
        for (int i = threadIdx.x; i < r * r; i += blockDim.x) {
            const float *p = x + (i / r) * n, *q = x + (i % r) * n;
            float sum = 0.f;
            for (int k = 0; k < n; ++k)
                sum = fmaf(p[k], q[k], sum);
            a[i] = rounded<bf16>(sum);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < r * r; i += blockDim.x) {
            const float *p = a + (i / r) * r;
            const int column = i % r;
            float sum = 0.f;
            for (int k = 0; k < r; ++k)
                sum = fmaf(p[k], a[k * r + column], sum);
            b[i] = rounded<bf16>(2.0315f * sum + -4.775f * a[i]);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < r * n; i += blockDim.x) {
            const float *p = b + (i / n) * r;
            const int column = i % n;
            float sum = 0.f;
            for (int k = 0; k < r; ++k)
                sum = fmaf(p[k], x[k * n + column], sum);
            next[i] = rounded<bf16>(1.f * sum + 3.4445f * x[i]);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < r * n; i += blockDim.x)
            x[i] = next[i];
        __syncthreads();
    }
    for (int i = threadIdx.x; i < r * n; i += blockDim.x)
        matrix[i] = __float2bfloat16(x[i]);
}
bool muon_newton_schulz_small_supported(int r, int n) { return r <= 32 && n <= 128; }
void launch_muon_newton_schulz_small(bf16 *x, int r, int n, int steps, int matrices, cudaStream_t s) {
    const size_t bytes = size_t(2 * r * n + 2 * r * r) * sizeof(float); // at most 40 KB
    muon_newton_schulz_small_kernel<<<matrices, 256, bytes, s>>>(x, r, n, steps);
}

// w = w * (1 - lr * wd) - lr * sqrt(max(1, rows/cols)) * x, x transposed back when rows > cols.
__global__ void __launch_bounds__(256) muon_apply_kernel(MuonApplyArgs a) {
    float multiplier = 1;
    if (a.schedule)
        multiplier = a.schedule[a.counters->step].multiplier;
    const float lr = a.muon_lr * multiplier;
    const float adjusted = lr * sqrtf(fmaxf(1.f, float(a.rows) / a.cols));
    const int matrix = blockIdx.y;
    const int64_t size = int64_t(a.rows) * a.cols, base = matrix * a.stride;
    const bool transpose = a.rows > a.cols;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < size;
         i += int64_t(gridDim.x) * blockDim.x) {
        int64_t index = transpose ? (i % a.cols) * a.rows + i / a.cols : i;
        float w = join_weight(a.weight_high[base + i], a.weight_low[base + i]) * (1 - lr * a.weight_decay);
        w -= adjusted * __bfloat162float(a.x[matrix * size + index]);
        unsigned bits = __float_as_uint(w);
        a.weight_high[base + i] = __ushort_as_bfloat16((unsigned short)(bits >> 16));
        a.weight_low[base + i] = uint16_t(bits);
        if (a.weight_fp32)
            a.weight_fp32[base + i] = w;
    }
}
// Eight consecutive weights per thread: both 16-bit halves of the FP32 masters as 128-bit accesses.
__device__ __forceinline__ void muon_update8(const MuonApplyArgs &a, int64_t at, const float (&x)[8], float keep,
                                             float adjusted) {
    const uint4 high = *reinterpret_cast<const uint4 *>(a.weight_high + at);
    const uint4 low = *reinterpret_cast<const uint4 *>(a.weight_low + at);
    const unsigned h[4] = {high.x, high.y, high.z, high.w}, l[4] = {low.x, low.y, low.z, low.w};
    unsigned ho[4], lo[4];
    float w[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        w[2 * j] = __uint_as_float((h[j] << 16) | (l[j] & 0xffffu));
        w[2 * j + 1] = __uint_as_float((h[j] & 0xffff0000u) | (l[j] >> 16));
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        w[j] *= keep;
        w[j] -= adjusted * x[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const unsigned b0 = __float_as_uint(w[2 * j]), b1 = __float_as_uint(w[2 * j + 1]);
        ho[j] = (b0 >> 16) | (b1 & 0xffff0000u);
        lo[j] = (b0 & 0xffffu) | (b1 << 16);
    }
    *reinterpret_cast<uint4 *>(a.weight_high + at) = make_uint4(ho[0], ho[1], ho[2], ho[3]);
    *reinterpret_cast<uint4 *>(a.weight_low + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    if (a.weight_fp32)
        store8(a.weight_fp32 + at, w);
}
__global__ void __launch_bounds__(256) muon_apply_vector_kernel(MuonApplyArgs a) {
    float multiplier = 1;
    if (a.schedule)
        multiplier = a.schedule[a.counters->step].multiplier;
    const float lr = a.muon_lr * multiplier;
    const float adjusted = lr * sqrtf(fmaxf(1.f, float(a.rows) / a.cols)), keep = 1 - lr * a.weight_decay;
    const int matrix = blockIdx.y;
    const int64_t size = int64_t(a.rows) * a.cols, base = matrix * a.stride;
    for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) * 8; i < size;
         i += int64_t(gridDim.x) * blockDim.x * 8) {
        float x[8];
        load8(a.x + matrix * size + i, x);
        muon_update8(a, base + i, x, keep, adjusted);
    }
}
__global__ void __launch_bounds__(256) muon_apply_transpose_kernel(MuonApplyArgs a) {
    __shared__ __align__(16) bf16 tile[MuonTile * MuonTilePitch]; // [column][row], as stored
    float multiplier = 1;
    if (a.schedule)
        multiplier = a.schedule[a.counters->step].multiplier;
    const float lr = a.muon_lr * multiplier;
    const float adjusted = lr * sqrtf(fmaxf(1.f, float(a.rows) / a.cols)), keep = 1 - lr * a.weight_decay;
    const int matrix = blockIdx.y;
    const int64_t size = int64_t(a.rows) * a.cols, base = matrix * a.stride;
    const int tiles_across = a.cols / MuonTile, tiles = (a.rows / MuonTile) * tiles_across;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int r0 = t / tiles_across * MuonTile, c0 = t % tiles_across * MuonTile;
        for (int item = threadIdx.x; item < MuonTile * 8; item += blockDim.x) { // (column, group of 8 rows)
            const int cc = item / 8, chunk = item % 8;
            const uint4 v = *reinterpret_cast<const uint4 *>(a.x + matrix * size + int64_t(c0 + cc) * a.rows + r0 + chunk * 8);
            uint32_t *target = reinterpret_cast<uint32_t *>(tile + cc * MuonTilePitch + chunk * 8);
            target[0] = v.x, target[1] = v.y, target[2] = v.z, target[3] = v.w;
        }
        __syncthreads();
        for (int item = threadIdx.x; item < MuonTile * 8; item += blockDim.x) { // (row, group of 8 columns)
            const int rr = item / 8, chunk = item % 8;
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                x[j] = __bfloat162float(tile[(chunk * 8 + j) * MuonTilePitch + rr]);
            muon_update8(a, base + int64_t(r0 + rr) * a.cols + c0 + chunk * 8, x, keep, adjusted);
        }
        __syncthreads();
    }
}
// Blocks per matrix of a stage that leaves no partial sums: eight per SM over all matrices, as far as there are 64 x 64 tiles (four
// thousand elements) for them.  With MuonBlocks of them a block of six 1536 x 384 matrices took four tiles one after another: eight
// optimizer steps of 8 layers d 512 7.17 -> 6.74 ms, 4 layers d 1024 16.6 -> 15.7, 6 layers d 384 level.
static int muon_blocks(int64_t size, int batch, int sms) {
    return int(std::max<int64_t>(1, std::min<int64_t>(size / (MuonTile * MuonTile), std::max(sms * 8 / batch, MuonBlocks))));
}
void launch_muon_normalize(bf16 *x, const float *sumsq, int64_t per_matrix, int batch, int sms, cudaStream_t s) {
    const dim3 grid(muon_blocks(per_matrix, batch, sms), batch);
    if (per_matrix % 8 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0)
        muon_normalize_vector_kernel<<<grid, 256, 0, s>>>(x, sumsq, per_matrix);
    else
        muon_normalize_kernel<<<grid, 256, 0, s>>>(x, sumsq, per_matrix);
}
void launch_muon_apply(const MuonApplyArgs &a, int sms, cudaStream_t s) {
    const dim3 grid(muon_blocks(int64_t(a.rows) * a.cols, a.batch, sms), a.batch);
    const bool aligned = a.stride % 8 == 0 && reinterpret_cast<uintptr_t>(a.weight_high) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(a.weight_low) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(a.weight_fp32) % 32 == 0 && reinterpret_cast<uintptr_t>(a.x) % 16 == 0;
    if (aligned && a.rows > a.cols && a.rows % MuonTile == 0 && a.cols % MuonTile == 0)
        muon_apply_transpose_kernel<<<grid, 256, 0, s>>>(a);
    else if (aligned && a.rows <= a.cols && (int64_t(a.rows) * a.cols) % 8 == 0)
        muon_apply_vector_kernel<<<grid, 256, 0, s>>>(a);
    else
        muon_apply_kernel<<<grid, 256, 0, s>>>(a);
}

__global__ void advance_kernel(StepCounters *counters) {
    counters->step += 1;
    counters->iteration += 1;
}
void launch_advance(StepCounters *counters, cudaStream_t s) {
    advance_kernel<<<1, 1, 0, s>>>(counters);
}

// ------------------------------------------------------------------------------------------
// Whole update of a model of 16-wide matrices.  As separate kernels it was 5 x (prepare, normalise, Newton-Schulz in
// shared memory, apply), AdamW and the counter: 22 launches and 0.2 ms, all latency (now 5 us).  One warp takes one matrix: X
// (16 x n, n = 16 or 48, the wide orientation) lives in registers as m16n8k16 operand fragments, and an iteration is
// n/8 + 2 + n/8 products per 16-deep step with the roundings of muon_newton_schulz_small_kernel:
//   A = X X^T     X's fragments are both operands
//   B = 2.0315 A A - 4.775 A,  X' = B X + 3.4445 X     the right operands are 8 x 8 blocks transposed in registers
// ------------------------------------------------------------------------------------------
constexpr int SmallWarps = 4; // matrices per block
__device__ __forceinline__ uint32_t transposed_block(uint32_t block) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(block));
    return r;
}
__device__ __forceinline__ float low_half(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float high_half(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

template <int Steps> struct SmallMuon { // Steps: columns of X / 16
    SmallMatrix matrix;
    int g, t;
    float mu, multiplier;
    float grad[Steps][4][2], momentum[Steps][4][2];
    bf16 high[Steps][4][2];
    uint16_t low[Steps][4][2];

    // register i of step k, half j: row g + 8 (i % 2), column 16 k + 8 (i / 2) + 2 t + j of X
    __device__ __forceinline__ int index(int k, int i, int j) const {
        const int row = g + 8 * (i % 2), column = 16 * k + 8 * (i / 2) + 2 * t + j;
        return matrix.offset + (matrix.rows > matrix.cols ? column * matrix.cols + row : row * matrix.cols + column);
    }
    template <class F> __device__ __forceinline__ void each(F &&f) const {
#pragma unroll
        for (int k = 0; k < Steps; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    f(k, i, j);
    }
    // Every load is issued before the clip norm is awaited and before the first store (they may alias as far as the
    // compiler knows: interleaved, each of the 24 elements paid a round trip to L2).
    __device__ __forceinline__ SmallMuon(const SmallOptimizerArgs &a, const SmallMatrix &matrix, int lane)
        : matrix(matrix), g(lane / 4), t(lane % 4), mu(a.momentum_rate), multiplier(1.f) {
        each([&](int k, int i, int j) {
            const int at = index(k, i, j);
            grad[k][i][j] = a.adam.gradient[at], momentum[k][i][j] = a.adam.momentum[at];
            high[k][i][j] = a.adam.weight_high[at], low[k][i][j] = a.adam.weight_low[at];
        });
        if (a.adam.schedule) {
            const TgStepRates rates = a.adam.schedule[a.counters->step - 1];
            mu = rates.momentum, multiplier = rates.multiplier;
        }
    }
    __device__ __forceinline__ void update(const SmallOptimizerArgs &a, float clip) {
        uint32_t x[Steps][4];
        float squares = 0;
#pragma unroll
        for (int k = 0; k < Steps; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float u[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float d = grad[k][i][j] * clip, m = momentum[k][i][j] + (1 - mu) * (d - momentum[k][i][j]);
                    a.adam.momentum[index(k, i, j)] = m;
                    u[j] = rounded<bf16>(d + mu * (m - d));
                    squares += u[j] * u[j];
                }
                x[k][i] = pack_bf16(u[0], u[1]);
            }
        const float inverse = 1.f / fmaxf(rounded<bf16>(sqrtf(warp_sum(squares))), rounded<bf16>(1e-7f));
#pragma unroll
        for (int k = 0; k < Steps; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                x[k][i] = pack_bf16(low_half(x[k][i]) * inverse, high_half(x[k][i]) * inverse);
        for (int step = 0; step < a.ns_steps; ++step) {
            float acc[8] = {};
#pragma unroll
            for (int k = 0; k < Steps; ++k) {
                mma_bf16(acc[0], acc[1], acc[2], acc[3], x[k], x[k][0], x[k][2]);
                mma_bf16(acc[4], acc[5], acc[6], acc[7], x[k], x[k][1], x[k][3]);
            }
            uint32_t square[4], b[4]; // A, then B, as left operands
#pragma unroll
            for (int i = 0; i < 4; ++i)
                square[i] = pack_bf16(acc[2 * i], acc[2 * i + 1]), acc[2 * i] = acc[2 * i + 1] = 0.f;
            mma_bf16(acc[0], acc[1], acc[2], acc[3], square, transposed_block(square[0]), transposed_block(square[1]));
            mma_bf16(acc[4], acc[5], acc[6], acc[7], square, transposed_block(square[2]), transposed_block(square[3]));
#pragma unroll
            for (int i = 0; i < 4; ++i)
                b[i] = pack_bf16(2.0315f * acc[2 * i] - 4.775f * low_half(square[i]), 2.0315f * acc[2 * i + 1] - 4.775f * high_half(square[i]));
#pragma unroll
            for (int k = 0; k < Steps; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h) { // eight columns
                    float y[4] = {};
                    mma_bf16(y[0], y[1], y[2], y[3], b, transposed_block(x[k][2 * h]), transposed_block(x[k][2 * h + 1]));
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        x[k][2 * h + r] =
                            pack_bf16(y[2 * r] + 3.4445f * low_half(x[k][2 * h + r]), y[2 * r + 1] + 3.4445f * high_half(x[k][2 * h + r]));
                }
        }
        const float lr = a.muon_lr * multiplier, keep = 1 - lr * a.adam.weight_decay;
        const float adjusted = lr * sqrtf(fmaxf(1.f, float(matrix.rows) / matrix.cols));
        each([&](int k, int i, int j) {
            const int at = index(k, i, j);
            float w = join_weight(high[k][i][j], low[k][i][j]) * keep;
            w -= adjusted * (j ? high_half(x[k][i]) : low_half(x[k][i]));
            const unsigned bits = __float_as_uint(w);
            a.adam.weight_high[at] = __ushort_as_bfloat16((unsigned short)(bits >> 16));
            a.adam.weight_low[at] = uint16_t(bits);
        });
    }
};
// clip_factor for one warp on its own: a few hundred partial sums, the same order in every warp.
__device__ __forceinline__ float clip_of_warp(const AdamArgs &a) {
    if (!(a.clip > 0))
        return 1.f;
    float local = 0;
#pragma unroll 4
    for (int b = threadIdx.x % 32; b < a.norm_blocks; b += 32)
        local += a.norm_partial[b];
    return fminf(1.f, a.clip / (sqrtf(warp_sum(local)) + 1e-6f));
}
__global__ void __launch_bounds__(SmallWarps * 32) small_optimizer_kernel(const __grid_constant__ SmallOptimizerArgs a, int matrix_blocks) {
    const int index = blockIdx.x * SmallWarps + threadIdx.x / 32;
    SmallMatrix matrix{0, 16, 16};
    if (index < a.matrix_count)
        matrix = a.matrices[index];
    sm100::grid_dependency_wait();
    sm100::grid_launch_dependents(); // the next step's kernel reads the step's number, which is this one's and has been counted up by now
    if (int(blockIdx.x) >= matrix_blocks) {
        const int64_t group = int64_t(blockIdx.x - matrix_blocks) * blockDim.x + threadIdx.x;
        AdamGroup parameters;
        if (group < a.adam.count / 8)
            parameters = AdamGroup(a.adam, group);
        AdamRates rates(a.adam, a.counters->step - 1);
        rates.clip = clip_of_warp(a.adam);
        parameters.update<false>(a.adam, rates, group);
    } else {
        if (max(matrix.rows, matrix.cols) == 48) {
            SmallMuon<3> muon(a, matrix, threadIdx.x % 32);
            muon.update(a, clip_of_warp(a.adam));
        } else if (index < a.matrix_count) {
            SmallMuon<1> muon(a, matrix, threadIdx.x % 32);
            muon.update(a, clip_of_warp(a.adam));
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        a.counters->iteration += 1; // its readers have ended
}
void launch_small_optimizer(const SmallOptimizerArgs &a, cudaStream_t s) {
    const int matrix_blocks = (a.matrix_count + SmallWarps - 1) / SmallWarps, per_block = SmallWarps * 32;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(matrix_blocks + unsigned((a.adam.count / 8 + per_block - 1) / per_block));
    config.blockDim = dim3(per_block), config.stream = s, config.attrs = &attribute, config.numAttrs = 1;
    CHECK_CUDA(cudaLaunchKernelEx(&config, small_optimizer_kernel, a, matrix_blocks));
}
