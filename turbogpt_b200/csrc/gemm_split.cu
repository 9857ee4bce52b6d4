// FP32 products on the tensor cores: C[m,n] = sum_k A[m,k] * B[n,k] with FP32 operands, for the FP32 check mode.
//
// Every operand value is the sum of three BF16 parts, x = h + m + l, each the rounded rest of what the parts before it leave (24 bits of
// significand in three times eight).  Of the nine products of parts the six above 2^-24 of x y are formed, exact in FP32: h h into one
// accumulator, h m, m h, m m, h l and l h into another.  The tensor core cuts its sums off instead of rounding them (1.2e-8 of the
// result for every step, 4.4e-6 after 256), so the first accumulator only ever holds 32 of K, two steps, and is added to FP32 registers; the second is
// 2^-8 of the result and holds 2048 (all of K: a weight gradient's error grew with its tokens, 262144 of them 2.7e-6, now 1.0e-6; CUDA cores 2.9e-6).
// Against 64 bits (N(0,1) operands, K 64 to 8192) 0.5 to 2.2e-7, where the CUDA cores' sums have 0.8 to 8.1e-7; what is cut off has the result's sign, 1 to 5e-8 of it.
// BF16 ends at 2^-133: a result all of whose terms have an operand below 2^-112 has fewer bits (2^-116 2e-6, 2^-120 4e-5).
//
// What bounds it: 24 products of 128 x BN x 16 a block read their operands from shared memory, 6 (4 + BN / 32) KB each, at 128 B/clk, beside the
// 48 + 3/8 BN KB that the split operands are written with: 1560 clocks a 128 x 128 x 64 block where the CUDA cores take 8192 for the
// multiply-adds alone.  (Measured 1.25 us a block beside 9 of start and end, 0.78 and 6 for 64 columns.)  2048 x 768 x 256 33 -> 14 us, 2048 x
// 256 x 1024 45 -> 18, 4096 x 2048 x 512 245 -> 72, dW 1024 x 256 x 2048 35 -> 17; an evaluation with gradients of 4 layers d 256, 2048 tokens
// 2.15 -> 1.47 ms, of 4 layers d 512, 4096 tokens 10.7 -> 4.9.  A CTA computes one 128 x BN tile of one slice of K: sixteen warps load the next block into registers, split what they
// loaded before into one of two shared-memory stages (the layouts of the BF16 product kernel, so that no operand is transposed) and add
// the finished block's sums to their registers; one thread issues the products.
//
// A result that is not finite is computed once more with FP32 multiply-adds: an infinity, or a value that rounds to one as BF16, has
// parts whose products are NaN.  Few of a tile by one thread each, many by the whole block as on CUDA cores (a tile of NaN in the first form took
// 3 to 73 times the CUDA-core kernel, now 1.6 to 2.1 times: 4 layers d 512, 4096 tokens, everything NaN 329 -> 19 ms where the CUDA cores take 11.8).
#include "epilogue_ops.cuh"
#include "sm100.cuh"
#include <algorithm>

using namespace sm100;

namespace {
constexpr int BM = 128, Block = 64; // rows of a tile, K elements of a block
constexpr int RestBlocks = 32;      // that the second accumulator holds
constexpr int Workers = 16, Threads = 32 * (Workers + 1), WorkerThreads = 32 * Workers;
constexpr int RowBytes = Block * 2; // of a K-major part; an MN-major one has 128 bytes (64 rows) per k
constexpr int ControlBytes = 64;
constexpr int part_bytes(int rows) { return rows * RowBytes; }
constexpr int stage_bytes(int bn) { return 3 * (part_bytes(BM) + part_bytes(bn)); }
constexpr int shared_bytes(int bn) { return 2 * stage_bytes(bn) + ControlBytes + 1024; }

// A worker's pieces of four values of a 64-deep block of an operand: along K where that is the unit stride, else along the rows.
template <int Rows, bool KMajor> struct Pieces {
    static constexpr int Count = Rows * Block / 4 / WorkerThreads;
    static constexpr int Apart = KMajor ? WorkerThreads / (Block / 4) : WorkerThreads / (Rows / 4); // rows, or k, between a thread's pieces
    float4 v[Count];
    const float *source; // of the first piece in the next block
    int64_t apart, advance;
    int k, rows_left, offset; // offset: in a part
    __device__ __forceinline__ Pieces(const float *base, int64_t row_stride, int64_t k_stride, int first_row, int rows, int first_k, int thread) {
        const int row = KMajor ? thread / (Block / 4) : thread % (Rows / 4) * 4, in_block = KMajor ? thread % (Block / 4) * 4 : thread / (Rows / 4);
        k = first_k + in_block, rows_left = rows - first_row - row;
        source = base + (first_row + row) * row_stride + k * k_stride;
        apart = Apart * (KMajor ? row_stride : k_stride);
        advance = Block * k_stride;
        const int line = KMajor ? row : in_block, unit = KMajor ? in_block : row % 64; // 128-byte line, element in it
        offset = (KMajor ? 0 : row / 64 * 64 * RowBytes) + line * RowBytes + ((unit / 8 ^ line % 8) << 4) + unit % 8 * 2;
    }
    __device__ __forceinline__ void load(int k_end) {
        const float *from = source;
#pragma unroll
        for (int c = 0; c < Count; ++c, from += apart) {
            const bool inside = KMajor ? Apart * c < rows_left && k < k_end : rows_left > 0 && k + Apart * c < k_end;
            v[c] = inside ? *reinterpret_cast<const float4 *>(from) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        source += advance, k += Block;
    }
    __device__ __forceinline__ void split(uint32_t parts) const {
#pragma unroll
        for (int c = 0; c < Count; ++c) {
            const uint32_t at = parts + offset + c * Apart * RowBytes; // Apart is a multiple of 8: the same place in its line
            uint64_t rest[2] = {float_pair(v[c].x, v[c].y), float_pair(v[c].z, v[c].w)};
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                uint32_t packed[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float lo, hi;
                    split_pair(rest[i], lo, hi);
                    packed[i] = pack_bf16(lo, hi);
                    const uint64_t value = float_pair(__uint_as_float(packed[i] << 16), __uint_as_float(packed[i] & 0xffff0000u));
                    rest[i] = fma_pair(value, float_pair(-1.f, -1.f), rest[i]); // exact
                }
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + part * part_bytes(Rows)), "r"(packed[0]), "r"(packed[1]) : "memory");
            }
        }
    }
};

__device__ __noinline__ float direct_product(const GemmArgs &g, int m, int n, int k_begin, int k_end) {
    const float *a = (const float *)g.a + m * g.a_row, *b = (const float *)g.b + n * g.b_row;
    float sum = 0.f;
    for (int k = k_begin; k < k_end; ++k)
        sum = fmaf(a[k * g.a_col], b[k * g.b_col], sum);
    return sum;
}

// Replaces what is not finite in a tile of sums (rows of BN + 4 in shared memory, behind which there is room) by the sums of FP32 multiply-adds in the order of K.
template <int BN, bool AK, bool BK>
__device__ __noinline__ void recompute(const GemmArgs &g, float *tile, int m0, int n0, int k_begin, int k_end) {
    constexpr int Pitch = BN + 4, Deep = 32, PitchA = BM + 4, Rows = BM / Workers, Columns = BN / 32; // of a thread: consecutive rows, columns 32 apart
    constexpr int FetchA = BM * Deep / WorkerThreads, FetchB = BN * Deep / WorkerThreads;
    static_assert((BM * Pitch + Deep * (PitchA + Pitch)) * int(sizeof(float)) <= 2 * stage_bytes(BN), "");
    const bool worker = threadIdx.x < WorkerThreads;
    const int valid_m = min(BM, g.m - m0), valid_n = min(BN, g.n - n0);
    int bad = 0;
    for (int i = threadIdx.x; worker && i < BM * BN; i += WorkerThreads) {
        const int m = i / BN, n = i % BN;
        bad += m < valid_m && n < valid_n && !isfinite(tile[m * Pitch + n]);
    }
    if (!__syncthreads_or(bad > 2)) {
        for (int i = threadIdx.x; worker && bad && i < BM * BN; i += WorkerThreads) {
            const int m = i / BN, n = i % BN;
            if (m < valid_m && n < valid_n && !isfinite(tile[m * Pitch + n]))
                tile[m * Pitch + n] = direct_product(g, m0 + m, n0 + n, k_begin, k_end);
        }
        __syncthreads();
        return;
    }
    float *sa = tile + BM * Pitch, *sb = sa + Deep * PitchA; // [k][row], [k][column]
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    float fa[FetchA], fb[FetchB], acc[Rows][Columns] = {};
    auto place = [&](int i, int rows, bool k_major, int &row, int &k) { row = k_major ? i / Deep : i % rows, k = k_major ? i % Deep : i / rows; };
    auto fetch = [&](int k0) {
        int row, k;
#pragma unroll
        for (int c = 0; c < FetchA; ++c) {
            place(threadIdx.x + c * WorkerThreads, BM, AK, row, k);
            fa[c] = row < valid_m && k0 + k < k_end ? ((const float *)g.a)[(m0 + row) * g.a_row + (k0 + k) * g.a_col] : 0.f;
        }
#pragma unroll
        for (int c = 0; c < FetchB; ++c) {
            place(threadIdx.x + c * WorkerThreads, BN, BK, row, k);
            fb[c] = row < valid_n && k0 + k < k_end ? ((const float *)g.b)[(n0 + row) * g.b_row + (k0 + k) * g.b_col] : 0.f;
        }
    };
    if (worker)
        fetch(k_begin);
    for (int k0 = k_begin; k0 < k_end; k0 += Deep) {
        if (worker) {
            int row, k;
#pragma unroll
            for (int c = 0; c < FetchA; ++c) {
                place(threadIdx.x + c * WorkerThreads, BM, AK, row, k);
                sa[k * PitchA + row] = fa[c];
            }
#pragma unroll
            for (int c = 0; c < FetchB; ++c) {
                place(threadIdx.x + c * WorkerThreads, BN, BK, row, k);
                sb[k * Pitch + row] = fb[c];
            }
        }
        __syncthreads();
        if (worker) {
            if (k0 + Deep < k_end)
                fetch(k0 + Deep);
#pragma unroll 4
            for (int k = 0; k < Deep; ++k) {
                float av[Rows], bv[Columns];
#pragma unroll
                for (int i = 0; i < Rows; i += 4)
                    *reinterpret_cast<float4 *>(av + i) = *reinterpret_cast<const float4 *>(sa + k * PitchA + warp * Rows + i);
#pragma unroll
                for (int j = 0; j < Columns; ++j)
                    bv[j] = sb[k * Pitch + lane + 32 * j];
#pragma unroll
                for (int i = 0; i < Rows; ++i)
#pragma unroll
                    for (int j = 0; j < Columns; ++j)
                        acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < Rows; ++i)
#pragma unroll
        for (int j = 0; j < Columns; ++j) {
            float *sum = tile + (warp * Rows + i) * Pitch + lane + 32 * j;
            if (worker && !isfinite(*sum))
                *sum = acc[i][j];
        }
    __syncthreads();
}

// `partials`: as in gemm_simt_kernel.
template <int BN, bool AK, bool BK>
__global__ void __launch_bounds__(Threads, 1) gemm_split_kernel(const __grid_constant__ GemmArgs g, float *partials, int slice_k, StepCounters *counters) {
    extern __shared__ uint8_t raw_shared[];
    const uint32_t base = (smem_address(raw_shared) + 1023u) & ~1023u;
    uint8_t *aligned = raw_shared + (base - smem_address(raw_shared));
    uint64_t *barriers = reinterpret_cast<uint64_t *>(aligned + 2 * stage_bytes(BN));
    const uint32_t full0 = smem_address(barriers), done0 = full0 + 16, added = done0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(barriers + 5);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    constexpr int Columns = BN == 128 ? 512 : 256; // of tensor memory: an accumulator of h h for either half of a block, one of the rest
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbarrier_init(full0 + 8 * s, Workers);
            mbarrier_init(done0 + 8 * s, 1);
        }
        mbarrier_init(added, Workers);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == Workers) {
        tmem_alloc(smem_address(tmem_slot), Columns);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_launch_dependents();
    grid_dependency_wait();

    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int k_begin = partials ? blockIdx.z * slice_k : 0, k_end = partials ? min(g.k, k_begin + slice_k) : g.k;
    const int blocks = (k_end - k_begin + Block - 1) / Block;
    constexpr int Share = BN / 4; // columns that a worker adds up, of its 32 rows
    const int quarter = warp % 4, first_column = warp / 4 * Share;
    float sums[Share];
    bool ok = true;
    if (warp == Workers) {
        if (elect_one()) {
            const uint32_t instruction = instruction_descriptor(BM, BN, !AK, !BK);
            constexpr uint32_t a_step = AK ? 32 : 16 * RowBytes, b_step = BK ? 32 : 16 * RowBytes;
            const uint64_t a_desc = smem_descriptor(base, AK ? 16 : 64 * RowBytes, 1024),
                           b_desc = smem_descriptor(base + 3 * part_bytes(BM), BK ? 16 : 64 * RowBytes, 1024);
            for (int b = 0; b < blocks && ok; ++b) {
                const int s = b % 2;
                ok = mbarrier_wait(full0 + 8 * s, b / 2 & 1, abort_flag, counters, 411); // the block is there
                if (!ok)
                    break;
                const uint64_t da = descriptor_at(a_desc, s * stage_bytes(BN)), db = descriptor_at(b_desc, s * stage_bytes(BN));
                const bool emptied = b % RestBlocks == 0; // the second accumulator, with the block before
                auto block_before_added = [&] { return b == 0 || (ok = mbarrier_wait(added, (b - 1) & 1, abort_flag, counters, 413)); };
                if (emptied && !block_before_added())
                    break;
                tcgen05_fence_after();
                auto multiply = [&](uint32_t accumulator, int a_part, int b_part, int ks, bool add) {
                    tcgen05_mma_bf16(accumulator, descriptor_at(da, a_part * part_bytes(BM) + ks * a_step),
                                     descriptor_at(db, b_part * part_bytes(BN) + ks * b_step), instruction, add);
                };
#pragma unroll
                for (int ks = 0; ks < Block / 16; ++ks) {
                    multiply(tmem_base + 2 * BN, 0, 1, ks, !emptied || ks > 0);
                    multiply(tmem_base + 2 * BN, 1, 0, ks, true);
                    multiply(tmem_base + 2 * BN, 1, 1, ks, true);
                    multiply(tmem_base + 2 * BN, 0, 2, ks, true);
                    multiply(tmem_base + 2 * BN, 2, 0, ks, true);
                }
                if (!emptied && !block_before_added())
                    break;
                tcgen05_fence_after();
#pragma unroll
                for (int ks = 0; ks < Block / 16; ++ks)
                    multiply(tmem_base + ks / 2 * BN, 0, 0, ks, ks % 2);
                tcgen05_commit(done0 + 8 * s);
            }
        }
        __syncwarp();
    } else {
        Pieces<BM, AK> a((const float *)g.a, g.a_row, g.a_col, m0, g.m, k_begin, threadIdx.x);
        Pieces<BN, BK> b((const float *)g.b, g.b_row, g.b_col, n0, g.n, k_begin, threadIdx.x);
#pragma unroll
        for (int j = 0; j < Share; ++j)
            sums[j] = 0.f;
        const uint32_t accumulators = tmem_base + (uint32_t(quarter * 32) << 16) + first_column;
        auto finish = [&](int block) {
            if (!mbarrier_wait(done0 + 8 * (block % 2), block / 2 & 1, abort_flag, counters, 412))
                return false;
            tcgen05_fence_after();
#pragma unroll
            for (int c = 0; c < Share; c += 8) { // more columns at a time spill
                uint32_t v[8], w[8];
                tmem_load_32x8_async(accumulators + c, v);
                tmem_load_32x8_async(accumulators + BN + c, w);
                tmem_wait_load(v);
                tmem_wait_load(w);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    sums[c + j] += __uint_as_float(v[j]) + __uint_as_float(w[j]);
            }
            if (block == blocks - 1 || block % RestBlocks == RestBlocks - 1) {
#pragma unroll
                for (int c = 0; c < Share; c += 16) {
                    uint32_t v[16];
                    tmem_load_32x16_async(accumulators + 2 * BN + c, v);
                    tmem_wait_load(v);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        sums[c + j] += __uint_as_float(v[j]);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0)
                mbarrier_arrive(added);
            return true;
        };
        a.load(k_end);
        b.load(k_end);
        for (int i = 0; i < blocks; ++i) {
            const uint32_t stage = base + i % 2 * stage_bytes(BN); // read by the products of block i - 2, which have been added up
            a.split(stage);
            b.split(stage + 3 * part_bytes(BM));
            fence_async_proxy();
            __syncwarp();
            if (lane == 0)
                mbarrier_arrive(full0 + 8 * (i % 2));
            if (i + 1 < blocks) {
                a.load(k_end);
                b.load(k_end);
            }
            if (i > 0 && !(ok = finish(i - 1)))
                break;
        }
        ok = ok && finish(blocks - 1);
    }
    ok = __syncthreads_and(ok); // every product is done: the stages take the sums
    constexpr int Pitch = BN + 4;
    float *tile = reinterpret_cast<float *>(aligned);
    bool finite = true;
    if (ok && warp < Workers) {
        const int row = quarter * 32 + lane;
#pragma unroll
        for (int j = 0; j < Share; ++j)
            finite = finite && isfinite(sums[j]);
#pragma unroll
        for (int j = 0; j < Share; j += 4)
            *reinterpret_cast<float4 *>(tile + row * Pitch + first_column + j) = make_float4(sums[j], sums[j + 1], sums[j + 2], sums[j + 3]);
    }
    tcgen05_fence_before();
    finite = __syncthreads_and(finite);
    if (warp == Workers)
        tmem_dealloc(tmem_base, Columns);
    if (!ok)
        return;
    if (!finite)
        recompute<BN, AK, BK>(g, tile, m0, n0, k_begin, k_end);
    const int n = n0 + threadIdx.x % BN;
    for (int row = threadIdx.x / BN; warp < Workers && row < BM; row += WorkerThreads / BN) {
        const int m = m0 + row;
        if (m >= g.m || n >= g.n)
            break;
        const float v = tile[row * Pitch + threadIdx.x % BN];
        if (partials)
            partials[(int64_t(blockIdx.z) * g.m + m) * g.n + n] = v;
        else
            EpilogueOps<float>::apply(g, v, int64_t(m) * g.ldc + n, int64_t(m) * g.ldr + n, 0);
    }
}

struct Plan {
    int bn = 0, slices = 1, slice_k = 0;
};
// Tile width and K slices by the time they take, in us: a 64-deep block, a tile's start and end, and the slices' partial tiles with the kernel that
// adds them.  Weight gradients run beside the chain of input gradients, in whose way more blocks are: their slices are charged twice
// that (6 layers d 320, 999 tokens 2.13 and 1.95 ms a step).
Plan split_plan(const GemmArgs &g, int sms) {
    Plan best;
    const double slicing = g.a_col == 1 ? 4. : 8.;
    double best_time = 0;
    const int blocks = (g.k + Block - 1) / Block;
    for (int bn : {128, 64}) {
        const int64_t tiles = int64_t((g.m + BM - 1) / BM) * ((g.n + bn - 1) / bn);
        for (int slices = 1; slices <= blocks && slices <= 32; ++slices) {
            const int per = (blocks + slices - 1) / slices;
            if ((blocks + per - 1) / per != slices || (slices > 1 && size_t(slices) * g.m * g.n * sizeof(float) > SplitScratchBytes))
                continue;
            const int64_t rounds = (tiles * slices + sms - 1) / sms;
            const double time = rounds * (bn == 128 ? per * 1.25 + 9. : per * .78 + 6.) + (slices > 1 ? slicing + slices * double(g.m) * g.n * 2e-6 : 0.);
            if (!best.bn || time < best_time)
                best = {bn, slices, per * Block}, best_time = time;
        }
    }
    return best;
}
} // namespace

// Unit stride in one dimension of each operand, everything else in pieces of four values; the three layouts that a layer needs.
bool gemm_split_supported(const GemmArgs &g) {
    auto operand = [&](const void *p, int64_t row, int64_t col, int rows) {
        const bool k_major = col == 1;
        return (k_major || row == 1) && (k_major ? row : col) % 4 == 0 && (k_major ? g.k : rows) % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0;
    };
    return g.in == Dtype::FP32 && g.out == Dtype::FP32 && g.batch == 1 && g.epilogue != Epilogue::Gelu && g.epilogue != Epilogue::CrossEntropy &&
           (g.a_col == 1 || g.b_col != 1) && g.m >= 64 && g.n >= 64 && g.k >= 16 && operand(g.a, g.a_row, g.a_col, g.m) &&
           operand(g.b, g.b_row, g.b_col, g.n);
}
void launch_gemm_split(const GemmArgs &g, int sms, StepCounters *counters, cudaStream_t s, float *scratch) {
    Plan plan = split_plan(g, sms);
    if (plan.slices > 1 && !scratch)
        plan.slices = 1;
    float *partials = plan.slices > 1 ? scratch : nullptr;
    const dim3 grid((g.n + plan.bn - 1) / plan.bn, (g.m + BM - 1) / BM, plan.slices);
    auto launch = [&](auto kernel) {
        const int shared = shared_bytes(plan.bn);
        CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shared));
        cudaLaunchConfig_t config{};
        config.gridDim = grid, config.blockDim = dim3(Threads), config.dynamicSmemBytes = shared, config.stream = s;
        cudaLaunchAttribute attribute{};
        attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attribute.val.programmaticStreamSerializationAllowed = 1;
        config.attrs = &attribute, config.numAttrs = 1;
        CHECK_CUDA(cudaLaunchKernelEx(&config, kernel, g, partials, plan.slice_k, counters));
    };
    auto launch_width = [&](auto bn) {
        constexpr int BN = decltype(bn)::value;
        if (g.a_col != 1)
            launch(gemm_split_kernel<BN, false, false>);
        else if (g.b_col != 1)
            launch(gemm_split_kernel<BN, true, false>);
        else
            launch(gemm_split_kernel<BN, true, true>);
    };
    if (plan.bn == 128)
        launch_width(std::integral_constant<int, 128>());
    else
        launch_width(std::integral_constant<int, 64>());
    if (partials)
        launch_gemm_slices(g, partials, plan.slices, s);
}
