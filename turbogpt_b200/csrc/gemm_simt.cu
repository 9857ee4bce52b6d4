// GEMM on CUDA cores: C[m,n] = sum_k A[m,k] * B[n,k] with arbitrary element strides, BF16 or
// FP32 operands, FP32 accumulation.  It serves the shapes the tensor-core kernels do not take
// (the reference architecture's 16/48-wide matrices) and engines without tensor cores, and is the on-device
// cross-check of the tcgen05 kernels.  Two kernels: gemm_simt_kernel takes any strides, sizes and
// alignments (64x64 output tile, 16-deep shared-memory slices, 4x4 outputs per thread, scalar loads);
// gemm_simt_wide_kernel (BF16 operands) and gemm_fp32_kernel (FP32) take what 16-byte pieces can reach and every shape of
// a real model (see there).
#include "epilogue_ops.cuh"
#include <algorithm>
#include <type_traits>

constexpr int TileM = 64, TileN = 64, TileK = 16;

// `partials` == nullptr: blockIdx.z is the batch index and the block walks all of K.  Otherwise (batch 1)
// blockIdx.z is a slice of K, `slice_k` elements long, and the block writes its FP32 partial tile to
// partials[slice][m][n]; gemm_simt_reduce_kernel adds the slices in order.
template <class In, class Out>
__global__ void __launch_bounds__(256) gemm_simt_kernel(GemmArgs g, float *partials, int slice_k) {
    __shared__ float as[TileK][TileM + 4], bs[TileK][TileN + 4];
    const int z = partials ? 0 : blockIdx.z;
    const In *a = (const In *)g.a + z * g.a_batch, *b = (const In *)g.b + z * g.b_batch;
    const int m0 = blockIdx.y * TileM, n0 = blockIdx.x * TileN;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int k_begin = partials ? blockIdx.z * slice_k : 0;
    const int k_end = partials ? min(g.k, k_begin + slice_k) : g.k;
    float acc[4][4] = {};
    for (int k0 = k_begin; k0 < k_end; k0 += TileK) {
        // 64x16 elements per operand, 4 per thread.  Thread order follows the unit stride.
        for (int i = threadIdx.x; i < TileM * TileK; i += 256) {
            int mm, kk;
            if (g.a_col == 1) {
                kk = i % TileK, mm = i / TileK;
            } else {
                mm = i % TileM, kk = i / TileM;
            }
            int m = m0 + mm, k = k0 + kk;
            as[kk][mm] = (m < g.m && k < k_end) ? to_float(a[m * g.a_row + k * g.a_col]) : 0.f;
        }
        for (int i = threadIdx.x; i < TileN * TileK; i += 256) {
            int nn, kk;
            if (g.b_col == 1) {
                kk = i % TileK, nn = i / TileK;
            } else {
                nn = i % TileN, kk = i / TileN;
            }
            int n = n0 + nn, k = k0 + kk;
            bs[kk][nn] = (n < g.n && k < k_end) ? to_float(b[n * g.b_row + k * g.b_col]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TileK; ++kk) {
            float av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                av[i] = as[kk][ty * 4 + i];
                bv[i] = bs[kk][tx * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    acc[i][j] += av[i] * bv[j];
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
            if (m < g.m && n < g.n) {
                if (partials)
                    partials[(int64_t(blockIdx.z) * g.m + m) * g.n + n] = acc[i][j];
                else
                    EpilogueOps<Out>::apply(g, acc[i][j], int64_t(m) * g.ldc + n, int64_t(m) * g.ldr + n, z);
            }
        }
}

// The same product for aligned BF16 operands.  FP32 multiply-adds bound it (128 per clock and SM, 72 TFLOP/s), so the rest has to
// stay out of their way: 8 x TN outputs per thread (12 or 16 shared-memory words per 32 or 64 multiply-adds), operands
// as 64-bit loads that are issued a slice ahead and land in the other of two shared-memory buffers, one barrier a slice.
// TN = 8: 128 x 128 tiles, 256 threads; TN = 4: 64 x 64 tiles, 128 threads, for outputs of too few large tiles.
struct Quad {
    uint2 v;
    __device__ __forceinline__ float at(int i) const {
        const unsigned w = i < 2 ? v.x : v.y;
        return __uint_as_float(i % 2 ? w & 0xffff0000u : w << 16);
    }
};
// Rows x TileK elements of an operand, four at a time along its unit stride, through registers into [k][row].
template <int Rows, int Threads> struct SliceLoader {
    static constexpr int Count = Rows * TileK / 4 / Threads;
    Quad quad[Count];
    __device__ __forceinline__ void fetch(const bf16 *base, int64_t row_stride, int64_t k_stride, int first_row, int rows, int k0, int k_end) {
#pragma unroll
        for (int c = 0; c < Count; ++c) {
            const int i = threadIdx.x + c * Threads;
            const bool k_major = k_stride == 1;
            const int row = first_row + (k_major ? i / (TileK / 4) : i % (Rows / 4) * 4), k = k0 + (k_major ? i % (TileK / 4) * 4 : i / (Rows / 4));
            quad[c] = {};
            if (row < rows && k < k_end)
                quad[c].v = *reinterpret_cast<const uint2 *>(base + row * row_stride + k * k_stride);
        }
    }
    __device__ __forceinline__ void put(float (*tile)[Rows + 4], int64_t k_stride) const {
#pragma unroll
        for (int c = 0; c < Count; ++c) {
            const int i = threadIdx.x + c * Threads;
            if (k_stride == 1) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    tile[i % (TileK / 4) * 4 + e][i / (TileK / 4)] = quad[c].at(e);
            } else {
                *reinterpret_cast<float4 *>(&tile[i / (Rows / 4)][i % (Rows / 4) * 4]) = make_float4(quad[c].at(0), quad[c].at(1), quad[c].at(2), quad[c].at(3));
            }
        }
    }
};
template <class Out, int TN>
__global__ void __launch_bounds__(TN == 8 ? 256 : 128) gemm_simt_wide_kernel(GemmArgs g, float *partials, int slice_k) {
    constexpr int Side = TN == 8 ? 128 : 64, Threads = TN == 8 ? 256 : 128;
    __shared__ __align__(16) float as[2][TileK][Side + 4], bs[2][TileK][Side + 4];
    const int z = partials ? 0 : blockIdx.z;
    const bf16 *a = (const bf16 *)g.a + z * g.a_batch, *b = (const bf16 *)g.b + z * g.b_batch;
    const int m0 = blockIdx.y * Side, n0 = blockIdx.x * Side;
    const int k_begin = partials ? blockIdx.z * slice_k : 0, k_end = partials ? min(g.k, k_begin + slice_k) : g.k;
    // a warp covers 64 x 32 (TN = 8) or 64 x 16 outputs: 8 threads down, 4 across; a thread's rows and columns come in
    // runs of four, 32 rows and 4 TN / 2 columns apart, so that its reads are whole 16-byte words without conflicts
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int row = (TN == 8 ? warp % 2 * 64 : 0) + lane / 4 * 4, column = (TN == 8 ? warp / 2 * 32 : warp * 16) + lane % 4 * 4;
    float acc[8][TN] = {};
    SliceLoader<Side, Threads> next_a, next_b;
    next_a.fetch(a, g.a_row, g.a_col, m0, g.m, k_begin, k_end);
    next_b.fetch(b, g.b_row, g.b_col, n0, g.n, k_begin, k_end);
    next_a.put(as[0], g.a_col);
    next_b.put(bs[0], g.b_col);
    __syncthreads();
    for (int k0 = k_begin, buffer = 0; k0 < k_end; k0 += TileK, buffer ^= 1) {
        const bool more = k0 + TileK < k_end;
        if (more) {
            next_a.fetch(a, g.a_row, g.a_col, m0, g.m, k0 + TileK, k_end);
            next_b.fetch(b, g.b_row, g.b_col, n0, g.n, k0 + TileK, k_end);
        }
#pragma unroll
        for (int k = 0; k < TileK; ++k) {
            float av[8], bv[TN];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float4 *>(av + 4 * h) = *reinterpret_cast<const float4 *>(&as[buffer][k][row + 32 * h]);
#pragma unroll
            for (int h = 0; h < TN / 4; ++h)
                *reinterpret_cast<float4 *>(bv + 4 * h) = *reinterpret_cast<const float4 *>(&bs[buffer][k][column + 16 * h]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        if (more) {
            next_a.put(as[buffer ^ 1], g.a_col);
            next_b.put(bs[buffer ^ 1], g.b_col);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + row + i / 4 * 32 + i % 4;
        if (m >= g.m)
            break;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int n = n0 + column + j / 4 * 16;
            if (n >= g.n)
                continue;
            if (partials) // n is a multiple of 4 here
                *reinterpret_cast<float4 *>(partials + (int64_t(blockIdx.z) * g.m + m) * g.n + n) =
                    make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    EpilogueOps<Out>::apply(g, acc[i][j + e], int64_t(m) * g.ldc + n + e, int64_t(m) * g.ldr + n + e, z);
        }
    }
}

// FP32 operands of the same alignment.  128 multiply-adds per clock and SM bound it; next come the operand reads from shared
// memory: they return 128 bytes per clock, so with 8 x 4 outputs per thread (12 words for 32 multiply-adds) they take half as
// long again as the multiply-adds, with 8 x 8 (16 for 64) exactly as long.  What is left is how well the two overlap and the last
// round of tiles: 2048 x 768 x 256 is 384 tiles for the 296 that fit at once.  64 x 64 tiles of 64 threads are two warps, too few to hide their own
// latencies on an SM that holds one to four tiles, so FP32Groups groups of 64 threads each take every fourth slice of K, with
// buffers and a barrier of their own, and their sums are added through shared memory in group order.
// Against the kernel for BF16 operands, which took these before: the 51 products of 4 layers d 256 over 2048 tokens 2230 -> 1720 us
// (that evaluation 2.52 -> 2.37 ms), 6 layers d 512 over 4096 tokens 19.9 -> 16.3 ms; eight groups in one block per SM instead of two
// blocks of four measured 5 % slower.  128 registers for two blocks spill 56 bytes (activations) and 96 (input gradients); one block
// without spills is 2 to 3 % slower from 2000 tokens on (steps of 2 layers d 1024, 16384 tokens 70.9 and 73.2 ms), 4 to 6 % faster where
// the tiles are fewer than the SMs (4 layers d 256, one sequence of 256 tokens 428 and 402 us).  Sums are shorter too: gradients 1.7 to 2.3e-7 from 64 bits instead of 3.0 to 4.6e-7.
// Slices come by cp.async as they lie in memory: [row][k] where K is the unit stride (read as pairs of k), else [k][row].
constexpr int FP32Side = 64, FP32Groups = 4, FP32Stages = 2, FP32PitchK = TileK + 4, FP32PitchRow = FP32Side + 4;
constexpr int FP32Slice = FP32Side * FP32PitchK; // floats of one operand's slice; the [k][row] form needs less
constexpr int FP32Shared = FP32Groups * FP32Stages * 2 * FP32Slice * int(sizeof(float));
static_assert(TileK * FP32PitchRow <= FP32Slice && FP32Groups * FP32Side * FP32PitchRow * int(sizeof(float)) <= FP32Shared, "");

// Outside the operand nothing is read; the address given is then its first one.
__device__ __forceinline__ void copy16_or_zeros(float *to, const float *from, const float *operand, bool inside) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(to))), "l"(inside ? from : operand), "r"(inside ? 16 : 0)
                 : "memory");
}
// The 16-byte pieces of an operand's slices that one of 64 threads copies: four a slice, sixteen rows (K-major) or four k apart.
template <bool KMajor> struct SliceCopier {
    static constexpr int Pieces = FP32Side * TileK / 4 / 64;
    const float *operand, *source; // the operand; the first piece of the next slice
    int64_t apart, advance;
    int row, k, rows_left, shared_at; // of the first piece
    __device__ __forceinline__ SliceCopier(const float *base, int64_t row_stride, int64_t k_stride, int first_row, int rows, int first_k, int thread)
        : operand(base) {
        row = KMajor ? thread / (TileK / 4) : thread % (FP32Side / 4) * 4;
        const int in_slice = KMajor ? thread % (TileK / 4) * 4 : thread / (FP32Side / 4);
        k = first_k + in_slice, rows_left = rows - first_row - row;
        source = base + (first_row + row) * row_stride + k * k_stride;
        apart = KMajor ? 16 * row_stride : 4 * k_stride;
        advance = TileK * FP32Groups * k_stride;
        shared_at = KMajor ? row * FP32PitchK + in_slice : in_slice * FP32PitchRow + row;
    }
    __device__ __forceinline__ void copy(float *slice, int k_end) {
        const float *from = source;
#pragma unroll
        for (int c = 0; c < Pieces; ++c, from += apart)
            copy16_or_zeros(slice + shared_at + c * (KMajor ? 16 * FP32PitchK : 4 * FP32PitchRow), from, operand,
                            KMajor ? 16 * c < rows_left && k < k_end : rows_left > 0 && k + 4 * c < k_end);
        source += advance, k += TileK * FP32Groups;
    }
};
// A thread's eight rows (or columns) of a tile, by its place 0..7: as the reads want them, without bank conflicts.
template <bool KMajor> __device__ __forceinline__ int fp32_row(int place, int i) {
    return KMajor ? place + 8 * i : i / 4 * 32 + place * 4 + i % 4;
}
template <bool KMajor> __device__ __forceinline__ void read_pair(const float *slice, int place, int k, float (&v)[2][8]) { // k and k + 1
    if constexpr (KMajor) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 u = *reinterpret_cast<const float2 *>(slice + fp32_row<true>(place, i) * FP32PitchK + k);
            v[0][i] = u.x, v[1][i] = u.y;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float4 *>(v[e] + 4 * h) = *reinterpret_cast<const float4 *>(slice + (k + e) * FP32PitchRow + h * 32 + place * 4);
    }
}
template <bool AK, bool BK>
__global__ void __launch_bounds__(64 * FP32Groups, 2) gemm_fp32_kernel(GemmArgs g, float *partials, int slice_k) {
    extern __shared__ __align__(16) float shared[];
    const int z = partials ? 0 : blockIdx.z;
    const float *a = (const float *)g.a + z * g.a_batch, *b = (const float *)g.b + z * g.b_batch;
    const int m0 = blockIdx.y * FP32Side, n0 = blockIdx.x * FP32Side;
    const int k_begin = partials ? blockIdx.z * slice_k : 0, k_end = partials ? min(g.k, k_begin + slice_k) : g.k;
    const int group = threadIdx.x / 64, thread = threadIdx.x % 64;
    const int down = thread % 32 / 4, across = thread / 32 * 4 + thread % 4; // 8 x 8 threads, a warp 8 x 4
    float *buffers = shared + group * FP32Stages * 2 * FP32Slice;
    const int slices = (k_end - k_begin + TileK - 1) / TileK;
    SliceCopier<AK> copy_a(a, g.a_row, g.a_col, m0, g.m, k_begin + group * TileK, thread);
    SliceCopier<BK> copy_b(b, g.b_row, g.b_col, n0, g.n, k_begin + group * TileK, thread);
    auto fetch = [&](int stage) { // the group's next slice
        float *to = buffers + stage * 2 * FP32Slice;
        copy_a.copy(to, k_end);
        copy_b.copy(to + FP32Slice, k_end);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[8][8] = {};
    if (group < slices)
        fetch(0);
    for (int s = group, stage = 0; s < slices; s += FP32Groups, stage ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("bar.sync %0, 64;" ::"r"(1 + group) : "memory"); // the slice has landed, and the other stage has been read
        if (s + FP32Groups < slices)
            fetch(stage ^ 1);
        const float *as = buffers + stage * 2 * FP32Slice, *bs = as + FP32Slice;
#pragma unroll
        for (int k = 0; k < TileK; k += 2) {
            float av[2][8], bv[2][8];
            read_pair<AK>(as, down, k, av);
            read_pair<BK>(bs, across, k, bv);
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        acc[i][j] = fmaf(av[e][i], bv[e][j], acc[i][j]);
        }
    }
    __syncthreads(); // every group's buffers have been read: they now take the sums
    float *sums = shared + group * FP32Side * FP32PitchRow;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            sums[fp32_row<AK>(down, i) * FP32PitchRow + fp32_row<BK>(across, j)] = acc[i][j];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < FP32Side * FP32Side / 4 / (64 * FP32Groups); ++c) {
        const int i = threadIdx.x + c * 64 * FP32Groups, row = i / (FP32Side / 4), column = i % (FP32Side / 4) * 4;
        const int m = m0 + row, n = n0 + column;
        if (m >= g.m || n >= g.n) // n is a multiple of 4 here
            continue;
        float v[4] = {};
#pragma unroll
        for (int k = 0; k < FP32Groups; ++k) {
            const float4 u = *reinterpret_cast<const float4 *>(shared + (k * FP32Side + row) * FP32PitchRow + column);
            v[0] += u.x, v[1] += u.y, v[2] += u.z, v[3] += u.w;
        }
        if (partials)
            *reinterpret_cast<float4 *>(partials + (int64_t(blockIdx.z) * g.m + m) * g.n + n) = make_float4(v[0], v[1], v[2], v[3]);
        else
#pragma unroll
            for (int e = 0; e < 4; ++e)
                EpilogueOps<float>::apply(g, v[e], int64_t(m) * g.ldc + n + e, int64_t(m) * g.ldr + n + e, z);
    }
}

// C = the K slices' partial tiles added in slice order (the same bits on every run).
template <class Out> __global__ void gemm_simt_reduce_kernel(GemmArgs g, const float *partials, int slices) {
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x, count = int64_t(g.m) * g.n;
    if (i >= count)
        return;
    float sum = 0.f;
    for (int slice = 0; slice < slices; ++slice)
        sum += partials[slice * count + i];
    const int64_t m = i / g.n, n = i % g.n;
    EpilogueOps<Out>::apply(g, sum, m * g.ldc + n, m * g.ldr + n, 0);
}

// What the vector loads need: unit stride in one dimension of each operand, the other stride, the extent along the unit
// stride and the base a multiple of four elements; n a multiple of 4.  Below a 64-wide output most of a tile is padding.  The
// FP32 kernel has the three layouts that a layer needs: activations, input gradients, weight gradients.
static bool wide_supported(const GemmArgs &g) {
    const size_t bytes = 4 * dtype_size(g.in);
    auto operand = [&](const void *p, int64_t row, int64_t col, int rows, int64_t batch) {
        const bool k_major = col == 1;
        return (k_major || row == 1) && (k_major ? row : col) % 4 == 0 && (k_major ? g.k : rows) % 4 == 0 && batch % 4 == 0 &&
               reinterpret_cast<uintptr_t>(p) % bytes == 0;
    };
    if (g.in == Dtype::FP32 && g.a_col != 1 && g.b_col == 1)
        return false;
    return g.m >= 64 && g.n >= 64 && g.k >= 16 && g.n % 4 == 0 && operand(g.a, g.a_row, g.a_col, g.m, g.a_batch) &&
           operand(g.b, g.b_row, g.b_col, g.n, g.b_batch);
}
struct SimtPlan {
    bool wide = false, large = false; // gemm_simt_wide_kernel (FP32: gemm_fp32_kernel), with 128 x 128 tiles
    int slices = 1;
};
// BF16: the smaller tile costs a quarter more shared-memory reads per product, the larger leaves SMs idle when there are fewer
// than one per SM.  K is cut where the tiles would not give every SM two blocks (the partial tiles then cost one more pass
// over the output each), in slices of at least 256 (wide) or 64.
static SimtPlan simt_plan(const GemmArgs &g) {
    auto tiles = [&](int side) { return int64_t((g.n + side - 1) / side) * ((g.m + side - 1) / side); };
    SimtPlan plan;
    plan.wide = wide_supported(g);
    plan.large = plan.wide && g.in == Dtype::BF16 && tiles(128) * g.batch >= 148;
    const int64_t count = tiles(plan.large ? 128 : 64);
    if (g.batch != 1)
        return plan;
    if (plan.wide) {
        if (!plan.large && g.k >= 512)
            plan.slices = int(std::clamp<int64_t>(296 / count, 1, g.k / 256));
    } else if (count <= 32 && g.k >= 2048) {
        // A weight gradient of the reference architecture is a 16..96-wide output over tens of thousands of tokens: one or
        // two tiles that would each walk all of K alone.
        plan.slices = int(std::min<int64_t>((296 + count - 1) / count, g.k / 64)); // at least four 16-deep steps per slice
    }
    return plan;
}
size_t gemm_simt_scratch_bytes(const GemmArgs &g) {
    const int slices = simt_plan(g).slices;
    return slices > 1 ? size_t(slices) * g.m * g.n * sizeof(float) : 0;
}

static void launch_fp32(const GemmArgs &g, dim3 grid, float *partials, int slice_k, cudaStream_t s) {
    auto launch = [&](auto kernel) {
        CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FP32Shared));
        kernel<<<grid, 64 * FP32Groups, FP32Shared, s>>>(g, partials, slice_k);
    };
    if (g.a_col != 1)
        launch(gemm_fp32_kernel<false, false>);
    else if (g.b_col != 1)
        launch(gemm_fp32_kernel<true, false>);
    else
        launch(gemm_fp32_kernel<true, true>);
}
template <class In, class Out> static void launch_simt(const GemmArgs &g, const SimtPlan &plan, float *scratch, cudaStream_t s) {
    const int slices = scratch ? plan.slices : 1, side = plan.large ? 128 : 64;
    float *partials = slices > 1 ? scratch : nullptr;
    const int slice_k = slices > 1 ? ((g.k + slices - 1) / slices + TileK - 1) / TileK * TileK : 0;
    const int used = slices > 1 ? (g.k + slice_k - 1) / slice_k : 1;
    const dim3 grid((g.n + side - 1) / side, (g.m + side - 1) / side, slices > 1 ? used : g.batch);
    if (!plan.wide)
        gemm_simt_kernel<In, Out><<<grid, 256, 0, s>>>(g, partials, slice_k);
    else if constexpr (std::is_same_v<In, float>)
        launch_fp32(g, grid, partials, slice_k, s);
    else if (plan.large)
        gemm_simt_wide_kernel<Out, 8><<<grid, 256, 0, s>>>(g, partials, slice_k);
    else
        gemm_simt_wide_kernel<Out, 4><<<grid, 128, 0, s>>>(g, partials, slice_k);
    if (partials)
        gemm_simt_reduce_kernel<Out><<<unsigned((int64_t(g.m) * g.n + 255) / 256), 256, 0, s>>>(g, partials, used);
}
void launch_gemm_slices(const GemmArgs &g, const float *partials, int slices, cudaStream_t s) {
    gemm_simt_reduce_kernel<float><<<unsigned((int64_t(g.m) * g.n + 255) / 256), 256, 0, s>>>(g, partials, slices);
}
void launch_gemm_simt(const GemmArgs &g, cudaStream_t s, float *scratch) {
    if (g.epilogue == Epilogue::Gelu || g.epilogue == Epilogue::CrossEntropy)
        throw std::runtime_error("This epilogue runs on the tensor cores");
    const SimtPlan plan = simt_plan(g);
    if (g.in == Dtype::BF16 && g.out == Dtype::BF16)
        launch_simt<bf16, bf16>(g, plan, scratch, s);
    else if (g.in == Dtype::BF16 && g.out == Dtype::FP32)
        launch_simt<bf16, float>(g, plan, scratch, s);
    else if (g.in == Dtype::FP32 && g.out == Dtype::FP32)
        launch_simt<float, float>(g, plan, scratch, s);
    else
        throw std::runtime_error("GEMM: FP32 operands with BF16 output are not used");
}
