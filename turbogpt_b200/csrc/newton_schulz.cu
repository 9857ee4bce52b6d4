// Muon's Newton-Schulz iterations of whole families of matrices in one persistent launch (reference cuda/optim.cuh:60-106):
//   A = X X^T,   B = 2.0315 A A - 4.775 A,   X' = B X + 3.4445 X,   each rounded to BF16, products accumulated in FP32.
//
// What bounds it: as launches of their own the fifteen dependent products of a step take 5 to 9 us each however small they are (launch,
// first loads, last stores), and a family's tiles fill the last wave badly.  Here the tiles of every product of every matrix are items of one
// list, iteration by iteration, product by product; CTA c takes items c, c + grid, ...  A matrix's product starts when the product
// before it is complete for that matrix alone: finished tiles are counted in global memory and the producer thread of a
// later item waits for the count.  The launch is cooperative, so every CTA is resident, and the list is ordered, so the first unfinished item can
// always run.  What is left is a tile's latency: 1.1 us from the count to the first operands, its products, 0.4 until they are in tensor memory, 0.8 to
// 2.5 of epilogue, 1.1 until its stores are everywhere and counted, 0.4 until that is seen.  Per iteration, launches of the product kernel (the
// families beside each other on four lanes up to 5 layers d 512) and this: 3 layers d 64 29.7 -> 4 us, 4 layers d 256 35.6 -> 16, 6 layers d 384
// 41.8 -> 27, 5 layers d 512 50 -> 37, 3 layers d 1024 168 -> 128, 12 layers d 768 277 -> 235; the same bits.
//
// A and B are symmetric: only tiles on and above the diagonal are computed, in groups of `square` rows and columns.  What lies below is read
// from the transposed place: a K block of an operand comes as rows (K-major) where it is stored, else as columns (MN-major) of its
// mirror image; the tensor core takes either.  The products of a mirrored element are the same numbers added in the same order:
// the same bits as from the full matrix.
#include "device_utils.cuh"
#include "sm100.cuh"
#include "tile_rows.cuh"
#include <algorithm>

using namespace sm100;

namespace {
constexpr int BM = 128, BK = 64, MaxBN = 256, MaxStages = 8;
constexpr int ReadyRing = 16; // items: the producer is at most a ring of one-block items and two accumulators ahead of the epilogue
constexpr int StoredRing = 4; // items whose stores are on their way
constexpr int StageABytes = BM * BK * 2;
constexpr int EpilogueWarps = 16, Threads = 96 + 32 * EpilogueWarps; // warp 0 loads, warp 1 multiplies, the last one reports finished tiles
constexpr int ControlBytes = 512;
constexpr int MaxShared = 232448 - 1024;
constexpr int MaxFamilies = 5;
enum Product { Gram, Square, Update, Products }; // A, B and X'

struct Maps {
    CUtensorMap x_rows[2], x_columns[2], a_rows, a_columns, b_rows, b_columns; // boxes of 128 rows x 64 K elements; 64 K rows x 64 columns
    CUtensorMap x_short[2], a_short; // 64 rows x 64 K elements
};
struct Family {
    bf16 *x[2], *a, *b;
    long long per_matrix, per_square; // elements
    int r, n;
    int row_tiles, square;            // tiles of 128 rows; A and B are stored in blocks of square x square
    int bn[Products];                 // columns of a tile
    int tiles[Products];              // per matrix
    int first[Products];              // item of the product's list at which the family begins
    int matrix0;                      // its first matrix in `progress`
    int aligned32;                    // rows are 32-byte aligned: 256-bit epilogue accesses
};
struct Params {
    Maps maps[MaxFamilies];
    Family family[MaxFamilies];
    int families, steps, stages, stage_bytes;
    int items[Products], per_step;
    float alpha[Products], beta[Products];
    unsigned *progress; // per matrix: finished tiles since the step began
    StepCounters *counters;
};

struct Item {
    int product, family, z, mt, nt, bn, k_blocks, step;
    int left_columns, right_columns; // K blocks before these are read as columns of K rows
    unsigned needed; // of the matrix's progress before it may be read
};
// A and B: column groups of `square` one after another, group j holds the row tiles up to its own end, each in square / bn tiles.
__device__ __forceinline__ Item locate(const Params &p, const Family *families, int work) {
    Item i;
    i.step = work / p.per_step;
    int at = work - i.step * p.per_step;
    i.product = Gram;
    while (at >= p.items[i.product])
        at -= p.items[i.product++];
    i.family = 0;
    while (i.family + 1 < p.families && at >= families[i.family + 1].first[i.product])
        ++i.family;
    const Family &f = families[i.family];
    at -= f.first[i.product];
    i.z = at / f.tiles[i.product];
    at -= i.z * f.tiles[i.product];
    const int per_matrix = f.tiles[Gram] + f.tiles[Square] + f.tiles[Update];
    int before = i.step * per_matrix;
    i.bn = f.bn[i.product];
    if (i.product == Update) {
        i.nt = at / f.row_tiles; // the row tiles of a column block follow one another: they share its X
        i.mt = at - i.nt * f.row_tiles;
        before += f.tiles[Gram] + f.tiles[Square];
    } else {
        const int split = f.square / i.bn;
        int group = 0;
        for (int here = min(f.row_tiles, f.square / BM) * split; at >= here; here = min(f.row_tiles, (group + 1) * (f.square / BM)) * split)
            at -= here, ++group;
        i.mt = at / split;
        i.nt = group * split + at - i.mt * split;
        before += i.product == Square ? f.tiles[Gram] : 0;
    }
    i.k_blocks = ((i.product == Gram ? f.n : f.r) + BK - 1) / BK;
    i.needed = unsigned(before);
    const int square_blocks = f.square / BK; // A block (k, j) of squares is stored where k <= j
    i.left_columns = i.product == Gram ? 0 : i.mt / (f.square / BM) * square_blocks;
    i.right_columns = i.product == Gram ? 0 : i.product == Square ? (i.nt * i.bn / f.square + 1) * square_blocks : i.k_blocks;
    return i;
}

__device__ __forceinline__ unsigned load_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void count_up(unsigned *p) { asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory"); }
__device__ __forceinline__ void fence_proxies() { asm volatile("fence.proxy.async;" ::: "memory"); } // generic writes before, copy-engine reads after

// Bounded like every wait (see mbarrier_wait).
__device__ __forceinline__ bool wait_for_progress(const unsigned *progress, unsigned needed, volatile int *abort_flag, StepCounters *counters) {
    if (load_acquire(progress) >= needed)
        return true;
    const unsigned long long start = global_timer();
    for (unsigned spins = 1;; ++spins) {
        if (load_acquire(progress) >= needed)
            return true;
        if ((spins & 0xff) == 0) {
            if (*abort_flag)
                return false;
            if (global_timer() - start > WaitLimitNs) {
                *abort_flag = 1;
                if (counters)
                    atomicCAS(&counters->error, 0, 401);
                return false;
            }
        }
    }
}

__global__ void __launch_bounds__(Threads, 1) newton_schulz_kernel(const __grid_constant__ Params p) {
    extern __shared__ uint8_t raw_shared[];
    const uint32_t base = (smem_address(raw_shared) + 1023u) & ~1023u;
    uint8_t *aligned = raw_shared + (base - smem_address(raw_shared));
    uint64_t *barriers = reinterpret_cast<uint64_t *>(aligned + p.stages * p.stage_bytes);
    const uint32_t full0 = smem_address(barriers), empty0 = full0 + 8 * MaxStages, tfull0 = empty0 + 8 * MaxStages, tempty0 = tfull0 + 16,
                   ready0 = tempty0 + 16, stored0 = ready0 + 8 * ReadyRing, reported0 = stored0 + 8 * StoredRing;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(barriers + 2 * MaxStages + 4 + ReadyRing + 2 * StoredRing);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    // The families' sizes in shared memory: through a run-time index the parameters are loads of hundreds of clocks.
    __shared__ Family families[MaxFamilies];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int i = threadIdx.x; i < int(sizeof(families) / 4); i += Threads)
        reinterpret_cast<uint32_t *>(families)[i] = reinterpret_cast<const uint32_t *>(p.family)[i];
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbarrier_init(full0 + 8 * s, 1);
            mbarrier_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbarrier_init(tfull0 + 8 * b, 1);
            mbarrier_init(tempty0 + 8 * b, EpilogueWarps);
        }
        for (int i = 0; i < ReadyRing; ++i)
            mbarrier_init(ready0 + 8 * i, 1);
        for (int i = 0; i < StoredRing; ++i) {
            mbarrier_init(stored0 + 8 * i, EpilogueWarps);
            mbarrier_init(reported0 + 8 * i, 1);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_address(tmem_slot), 2 * MaxBN);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int work_items = p.per_step * p.steps, first_item = blockIdx.x, item_stride = gridDim.x;

    if (warp == 0) {
        // ---------------- producer: waits for the item's matrix, then streams its operands ----------------
        if (elect_one()) {
            int stage = 0, count = 0;
            uint32_t phase = 0;
            for (int w = first_item; w < work_items; w += item_stride, ++count) {
                const Item item = locate(p, families, w);
                const Family &f = families[item.family];
                const Maps *maps = p.maps + item.family;
                const int m_first = item.mt * BM, n_first = item.nt * item.bn, z = item.z;
                const CUtensorMap *x_rows = maps->x_rows + item.step % 2, *x_columns = maps->x_columns + item.step % 2;
                const CUtensorMap *left_rows = item.product == Gram ? x_rows : item.product == Square ? &maps->a_rows : &maps->b_rows,
                                  *left_columns = item.product == Square ? &maps->a_columns : &maps->b_columns;
                const CUtensorMap *right_rows = item.product == Gram ? maps->x_short + item.step % 2 : &maps->a_short,
                                  *right_columns = item.product == Square ? &maps->a_columns : x_columns;
                prefetch_map(left_rows), prefetch_map(right_rows);
                prefetch_map(left_columns), prefetch_map(right_columns);
                if (item.needed && !wait_for_progress(p.progress + f.matrix0 + item.z, item.needed, abort_flag, p.counters))
                    break;
                mbarrier_arrive(ready0 + 8 * (count % ReadyRing)); // the epilogue may read the second tensor
                fence_proxies();
                bool ok = true;
                for (int kb = 0; kb < item.k_blocks; ++kb) {
                    ok = mbarrier_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, p.counters, 402);
                    if (!ok)
                        break;
                    const uint32_t sa = base + stage * p.stage_bytes, sb = sa + StageABytes, bar = full0 + 8 * stage;
                    mbarrier_expect_tx(bar, StageABytes + item.bn * BK * 2);
                    const int k = kb * BK;
                    if (kb < item.left_columns) {
                        tma_load_3d(sa, left_columns, m_first, k, z, bar);
                        tma_load_3d(sa + 64 * BK * 2, left_columns, m_first + 64, k, z, bar);
                    } else {
                        tma_load_3d(sa, left_rows, k, m_first, z, bar);
                    }
                    if (kb < item.right_columns) {
                        for (int j = 0; j < item.bn / 64; ++j)
                            tma_load_3d(sb + j * 64 * BK * 2, right_columns, n_first + j * 64, k, z, bar);
                    } else {
                        for (int j = 0; j < item.bn / 64; ++j)
                            tma_load_3d(sb + j * 64 * BK * 2, right_rows, k, n_first + j * 64, z, bar);
                    }
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok)
                    break;
            }
        }
    } else if (warp == 1) {
        // ---------------- products ----------------
        if (elect_one()) {
            // the first stage's descriptors, by rows and by columns
            const uint64_t a_rows = smem_descriptor(base, 16, 1024), a_columns = smem_descriptor(base, 64 * BK * 2, 1024);
            const uint64_t b_rows = smem_descriptor(base + StageABytes, 16, 1024), b_columns = smem_descriptor(base + StageABytes, 64 * BK * 2, 1024);
            int stage = 0, buffer = 0;
            uint32_t phase = 0, buffer_phase = 0;
            for (int w = first_item; w < work_items; w += item_stride) {
                const Item item = locate(p, families, w);
                if (!mbarrier_wait(tempty0 + 8 * buffer, buffer_phase ^ 1, abort_flag, p.counters, 403))
                    break;
                tcgen05_fence_after();
                const uint32_t accumulator = tmem_base + buffer * MaxBN, shape = instruction_descriptor(BM, item.bn, 0, 0);
                bool ok = true;
                for (int kb = 0; kb < item.k_blocks; ++kb) {
                    const bool left = kb < item.left_columns, right = kb < item.right_columns;
                    const uint32_t instruction = shape | instruction_descriptor(0, 0, left, right);
                    const uint32_t a_step = left ? 16 * 128 : 32, b_step = right ? 16 * 128 : 32;
                    const uint64_t da = descriptor_at(left ? a_columns : a_rows, stage * p.stage_bytes),
                                   db = descriptor_at(right ? b_columns : b_rows, stage * p.stage_bytes);
                    ok = mbarrier_wait(full0 + 8 * stage, phase, abort_flag, p.counters, 404);
                    if (!ok)
                        break;
                    tcgen05_fence_after();
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks)
                        tcgen05_mma_bf16(accumulator, descriptor_at(da, ks * a_step), descriptor_at(db, ks * b_step), instruction, kb > 0 || ks > 0);
                    tcgen05_commit(empty0 + 8 * stage);
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok)
                    break;
                tcgen05_commit(tfull0 + 8 * buffer);
                if (++buffer == 2) {
                    buffer = 0;
                    buffer_phase ^= 1;
                }
            }
        }
    } else if (warp == Threads / 32 - 1) {
        // ---------------- reports a tile when its stores have left: the wait for them, a microsecond or two, is no epilogue warp's ----------------
        if (elect_one()) {
            int count = 0;
            for (int w = first_item; w < work_items; w += item_stride, ++count) {
                const Item item = locate(p, families, w);
                const int slot = count % StoredRing;
                if (!mbarrier_wait(stored0 + 8 * slot, count / StoredRing & 1, abort_flag, p.counters, 407))
                    break;
                __threadfence(); // the epilogue's stores, which the barrier has shown to this thread, before the count
                count_up(p.progress + families[item.family].matrix0 + item.z);
                mbarrier_arrive(reported0 + 8 * slot);
            }
        }
    } else {
        // ---------------- epilogue: four warps per quarter of tensor memory take every fourth 32-column chunk ----------------
        constexpr int Shares = EpilogueWarps / 4;
        const int quarter = warp % 4, share = (warp - 2) / 4;
        const bool odd = lane & 1;
        int buffer = 0, count = 0;
        uint32_t buffer_phase = 0;
        for (int w = first_item; w < work_items; w += item_stride, ++count) {
            const Item item = locate(p, families, w);
            const Family &f = families[item.family];
            const int pitch = item.product == Update ? f.n : f.r; // of the output and of the second tensor
            const int columns = min(item.bn, pitch - item.nt * item.bn);
            const long long matrix = item.z * (item.product == Update ? f.per_matrix : f.per_square);
            bf16 *out = (item.product == Gram ? f.a : item.product == Square ? f.b : f.x[(item.step + 1) % 2]) + matrix;
            const bf16 *second = (item.product == Square ? f.a : f.x[item.step % 2]) + matrix;
            const int row = item.mt * BM + quarter * 32 + (lane & ~1); // the pair's first row
            const bool combine = item.product != Gram;
            const float alpha = p.alpha[item.product], beta = p.beta[item.product];
            uint32_t rv[2][8];
            auto fetch_second = [&](int c) {
                const int column = item.nt * item.bn + c * 32 + (odd ? 16 : 0);
                if (!combine || column >= pitch)
                    return;
#pragma unroll
                for (int g = 0; g < 2; ++g)
                    if (row + g < f.r)
                        load_global32(second + (long long)(row + g) * pitch + column, rv[g], f.aligned32 && column + 16 <= pitch, column + 8 < pitch);
            };
            if (combine) {
                if (!mbarrier_wait(ready0 + 8 * (count % ReadyRing), count / ReadyRing & 1, abort_flag, p.counters, 405))
                    break;
                fetch_second(share);
            }
            if (!mbarrier_wait(tfull0 + 8 * buffer, buffer_phase, abort_flag, p.counters, 406))
                break;
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + buffer * MaxBN;
            auto release = [&] {
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbarrier_arrive(tempty0 + 8 * buffer);
            };
            const int chunks = (columns + 31) / 32;
            for (int c = share; c < chunks; c += Shares) {
                uint32_t v[16];
                if (combine)
                    exchange_rows(rv[0], rv[1], odd); // to lane = row
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t acc[16];
                    tmem_load_32x16_async(taddr + c * 32 + half * 16, acc);
                    tmem_wait_load(acc);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float s0 = __uint_as_float(acc[2 * j]), s1 = __uint_as_float(acc[2 * j + 1]);
                        v[half * 8 + j] = combine ? pack_bf16(alpha * s0 + beta * __uint_as_float(rv[half][j] << 16),
                                                              alpha * s1 + beta * __uint_as_float(rv[half][j] & 0xffff0000u))
                                                  : pack_bf16(s0, s1);
                    }
                }
                if (c + Shares >= chunks)
                    release();
                else
                    fetch_second(c + Shares);
                exchange_rows(v, v + 8, odd);
                const int column = item.nt * item.bn + c * 32 + (odd ? 16 : 0);
#pragma unroll
                for (int g = 0; g < 2; ++g)
                    if (row + g < f.r && column < pitch)
                        store_global32(out + (long long)(row + g) * pitch + column, v + g * 8, f.aligned32 && column + 16 <= pitch, column + 8 < pitch);
            }
            if (share >= chunks)
                release();
            const int slot = count % StoredRing;
            if (!mbarrier_wait(reported0 + 8 * slot, (count / StoredRing & 1) ^ 1, abort_flag, p.counters, 408)) // of the item StoredRing before
                break;
            __syncwarp();
            if (lane == 0)
                mbarrier_arrive(stored0 + 8 * slot);
            if (++buffer == 2) {
                buffer = 0;
                buffer_phase ^= 1;
            }
        }
    }

    // Teardown, as in the product kernel.
    __syncthreads();
    if (*abort_flag)
        __nanosleep(2000000);
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1)
        tmem_dealloc(tmem_base, 2 * MaxBN);
}

// Tiles of a symmetric r x r matrix in whose block of `square` x `square` something lies on or above the diagonal.
int symmetric_tiles(int r, int square, int bn) {
    const int row_tiles = (r + BM - 1) / BM;
    int tiles = 0;
    for (int group = 0; group * square < r; ++group)
        tiles += std::min(row_tiles, (group + 1) * (square / BM));
    return tiles * (square / bn);
}
} // namespace

bool newton_schulz_supported(int rows, int cols, const void *x) {
    const int r = std::min(rows, cols), n = std::max(rows, cols);
    return r >= 64 && r % 8 == 0 && n % 8 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0;
}

bool launch_newton_schulz(const NewtonSchulzArgs &a, int sms, cudaStream_t s) {
    if (a.count < 1 || a.count > MaxFamilies || a.steps < 1)
        throw std::runtime_error("Newton-Schulz: one to five families, at least one step");
    static_assert(sizeof(Params) <= 32764, "the most a kernel's parameters may take");
    static thread_local Params p;
    p = Params{};
    int order[MaxFamilies]; // the longest products first: what follows them fills the gaps
    for (int i = 0; i < a.count; ++i)
        order[i] = i;
    auto side = [&](int i) { return std::max(a.family[i].rows, a.family[i].cols); };
    std::stable_sort(order, order + a.count, [&](int i, int j) { return side(i) > side(j); });
    // Tile widths.  A narrow tile is done sooner (its epilogue is as long as its stores, and what follows waits for all of a matrix's tiles),
    // a wide one loads less for its products: 64 columns where that makes at most one tile per SM, 128 up to just under two, else
    // 256.  Over 18 models of 2 to 12 layers, d 64 to 1024, every combination timed, this is 1.0 % from the best of each (at worst 5 %);
    // ten iterations of 6 layers d 384 with 128, 128 and 256 columns for A, B and X' 361 us, with 64 throughout 648, 256 throughout 405; 4 layers d
    // 256 with 64, 64 and 128 196 us, with 256 throughout 267.
    auto tiles_of = [&](Product product, int i, int bn) {
        const int r = std::min(a.family[i].rows, a.family[i].cols);
        return product == Update ? (r + BM - 1) / BM * ((side(i) + bn - 1) / bn) : symmetric_tiles(r, std::max(bn, BM), bn);
    };
    auto width = [&](Product product) {
        auto tiles = [&](int bn) {
            long long all = 0;
            for (int i = 0; i < a.count; ++i)
                all += (long long)a.batch * tiles_of(product, i, bn);
            return all;
        };
        return tiles(64) <= sms ? 64 : tiles(128) * 10 <= 19ll * sms ? 128 : 256;
    };
    const int bn[Products] = {width(Gram), width(Square), width(Update)};
    const int square = std::max({bn[Gram], bn[Square], BM}); // both are read by it
    p.families = a.count, p.steps = a.steps, p.progress = a.progress, p.counters = a.counters;
    p.stage_bytes = StageABytes + std::max({bn[Gram], bn[Square], bn[Update]}) * BK * 2;
    p.stages = std::min(MaxStages, (MaxShared - 1024 - ControlBytes) / p.stage_bytes);
    p.alpha[Gram] = 1.f, p.beta[Gram] = 0.f, p.alpha[Square] = 2.0315f, p.beta[Square] = -4.775f, p.alpha[Update] = 1.f, p.beta[Update] = 3.4445f;
    for (int i = 0; i < a.count; ++i) {
        const NewtonSchulzArgs::Family &from = a.family[order[i]];
        Family &f = p.family[i];
        const int r = f.r = std::min(from.rows, from.cols), n = f.n = std::max(from.rows, from.cols);
        f.per_matrix = (long long)r * n, f.per_square = (long long)r * r;
        f.row_tiles = (r + BM - 1) / BM, f.square = square;
        for (int product = Gram; product < Products; ++product)
            f.bn[product] = bn[product];
        f.tiles[Gram] = symmetric_tiles(r, square, bn[Gram]), f.tiles[Square] = symmetric_tiles(r, square, bn[Square]);
        f.tiles[Update] = tiles_of(Update, order[i], bn[Update]);
        f.matrix0 = order[i] * a.batch;
        f.x[0] = from.x[0], f.x[1] = from.x[1], f.a = from.a, f.b = from.b;
        f.aligned32 = r % 16 == 0 && n % 16 == 0;
        for (const bf16 *pointer : {from.x[0], from.x[1], from.a, from.b})
            f.aligned32 &= reinterpret_cast<uintptr_t>(pointer) % 32 == 0;
        Maps &maps = p.maps[i];
        for (int j = 0; j < 2; ++j) {
            maps.x_rows[j] = make_map_bf16(from.x[j], n, r, a.batch, n, f.per_matrix, BK, BM);
            maps.x_columns[j] = make_map_bf16(from.x[j], n, r, a.batch, n, f.per_matrix, 64, BK);
        }
        for (int j = 0; j < 2; ++j)
            maps.x_short[j] = make_map_bf16(from.x[j], n, r, a.batch, n, f.per_matrix, BK, 64);
        maps.a_short = make_map_bf16(from.a, r, r, a.batch, r, f.per_square, BK, 64);
        maps.a_rows = make_map_bf16(from.a, r, r, a.batch, r, f.per_square, BK, BM);
        maps.a_columns = make_map_bf16(from.a, r, r, a.batch, r, f.per_square, 64, BK);
        maps.b_rows = make_map_bf16(from.b, r, r, a.batch, r, f.per_square, BK, BM);
        maps.b_columns = make_map_bf16(from.b, r, r, a.batch, r, f.per_square, 64, BK);
        for (int product = Gram; product < Products; ++product)
            f.first[product] = p.items[product], p.items[product] += f.tiles[product] * a.batch;
    }
    p.per_step = p.items[Gram] + p.items[Square] + p.items[Update];
    if ((long long)p.per_step * a.steps > (1 << 30))
        return false;
    const int shared = p.stages * p.stage_bytes + ControlBytes + 1024;
    CHECK_CUDA(cudaFuncSetAttribute(newton_schulz_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MaxShared));
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(std::min(sms, p.per_step)), config.blockDim = dim3(Threads), config.dynamicSmemBytes = shared, config.stream = s;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeCooperative; // every CTA is resident: they wait for one another
    attribute.val.cooperative = 1;
    config.attrs = &attribute, config.numAttrs = 1;
    const cudaError_t status = cudaLaunchKernelEx(&config, newton_schulz_kernel, p);
    if (status == cudaErrorCooperativeLaunchTooLarge) {
        (void)cudaGetLastError();
        return false;
    }
    CHECK_CUDA(status);
    return true;
}
